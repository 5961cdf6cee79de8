"""Dslash with boundary phases alone (GEN_PHASES): phases in any set of
directions, odd numbers of right-hand sides, partly filled blocks, against
the CPU oracle; dslashDir with the same phases keeps the general path.
Tolerances: test_dslash_gpu.py's."""
import numpy as np
import pytest

from helpers import TOL, make_setup, rel_l2
from qphix_b200 import fields as F

pytestmark = pytest.mark.gpu

PHASES = [[np.exp(0.3j), None, None, None], [None, np.exp(-0.7j), np.exp(0.2j), None],
          [np.exp(0.3j), np.exp(-0.7j), np.exp(0.4j), np.exp(1.1j)]]


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (6, 4, 2, 6)])
@pytest.mark.parametrize("prec", ["f64", "f32", "f16", "q16f32"])
@pytest.mark.parametrize("recon", [18, 12])
def test_boundary_phases(oracle, dims, prec, recon):
    from qphix_b200 import api
    s = make_setup(dims, seed=41, mass=0.1)
    lat = api.Lattice(dims)
    u = lat.gauge(prec, recon).upload(s["gauge"])
    psi, chi = (np.stack([F.gaussian_spinor(dims, k + i) for i in range(3)]) for k in (7, 17))
    gp, gc, gr = lat.spinor(prec, 3).upload(psi), lat.spinor(prec, 3).upload(chi), lat.spinor(prec, 3)
    A, Ai = (lat.clover(prec).upload(s[k][1]) for k in ("clov", "invclov"))
    for ph in PHASES:
        use = [p is not None for p in ph]
        phases = [(p.real, p.imag) if p is not None else (1.0, 0.0) for p in ph]
        L = oracle.make_lattice(dims, -1.0, 0.8, 1.1, tbc=ph)
        W, D = api.Dslash(lat, -1.0, 0.8, 1.1, use, phases), api.ClovDslash(lat, -1.0, 0.8, 1.1, use, phases)
        for sign in (1, -1):
            def same(want):
                got = gr.download()
                for i in range(3):
                    assert rel_l2(got[i], want(psi[i], chi[i])) < TOL[prec]

            W.dslash(gr, gp, u, sign, 1)
            same(lambda p, c: oracle.dslash(L, p, s["gauge"], sign, 1))
            W.dslashAChiMinusBDPsi(gr, gp, gc, u, 0.7, 0.3, sign, 1)
            same(lambda p, c: oracle.dslash_achimbdpsi(L, p, c, s["gauge"], 0.7, 0.3, sign, 1))
            D.dslash(gr, gp, u, Ai, sign, 1)
            same(lambda p, c: oracle.clov_dslash(L, p, s["gauge"], s["invclov"][1], sign, 1))
            D.dslashAChiMinusBDPsi(gr, gp, gc, u, A, 0.25, sign, 1)
            same(lambda p, c: oracle.clov_achimbdpsi(L, p, c, s["gauge"], s["clov"][1], 0.25, 0.0, sign, 1))
        for d in range(8):
            W.dslashDir(gr, gp, u, 1, d)
            same(lambda p, c: oracle.dslash_dir(L, p, s["gauge"], 1, d))


@pytest.mark.parametrize("prec", ["f64", "f32", "f16", "bf16", "q16", "q16f32"])
@pytest.mark.parametrize("recon", [18, 12])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 4])
def test_untimed_shapes(oracle, prec, recon, nrhs):
    """the autotuner off, reductions included: the rule's shape for a lattice
    of few blocks (its others: test_shapes_gpu.py)"""
    from qphix_b200 import api
    dims = (6, 4, 2, 6)
    s = make_setup(dims, seed=47, mass=0.1)
    lat = api.Lattice(dims)
    u = lat.gauge(prec, recon).upload(s["gauge"])
    psi, chi = (np.stack([F.gaussian_spinor(dims, k + i) for i in range(nrhs)]) for k in (7, 17))
    gp, gc, gr = (lat.spinor(prec, nrhs).upload(v) for v in (psi, chi, psi))
    A = lat.clover(prec).upload(s["clov"][1])
    D = api.ClovDslash(lat, -1.0, 1.0, 1.0)
    L = oracle.make_lattice(dims, -1.0, 1.0, 1.0)
    api.tune_enable(False)
    try:
        red = D.dslashAChiMinusBDPsiNorms(gr, gp, gc, u, A, 0.25, 1, 1)
    finally:
        api.tune_enable(True)
    assert lat.dslash_shape() == (1, 1)
    got = gr.download().reshape(nrhs, -1, 4, 3)
    for i in range(nrhs):
        want = oracle.clov_achimbdpsi(L, psi[i], chi[i], s["gauge"], s["clov"][1], 0.25, 0.0, 1, 1)
        assert rel_l2(got[i], want) < TOL[prec]
        assert abs(red[i, 0] - np.vdot(want, want).real) < 4 * TOL[prec] * np.vdot(want, want).real
