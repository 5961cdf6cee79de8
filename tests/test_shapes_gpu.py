"""Which launch shape a Dslash takes: the rule for configurations that were not
timed, on both sides of its line (296 blocks at two sites or right-hand sides
per thread, 148 for BF16), with the autotuner off and inside a solver's captured iteration.
Shapes read (right-hand sides, sites) per thread, lanes (2, 0)."""
import numpy as np
import pytest

from helpers import TOL, rel_l2
from qphix_b200 import fields as F

pytestmark = pytest.mark.gpu

DIMS = (16, 16, 16, 18)  # 288 blocks of 128 sites a right-hand side


def rule(prec, recon, nrhs):
    pairs = recon == 12 and nrhs % 2 == 0
    if prec == "f64" or 288 * nrhs // 2 < (148 if prec == "bf16" else 296):
        return 1, 1
    if pairs:
        return (2, 1) if prec == "f32" else (2, 0)
    return (1, 2) if prec == "bf16" else (1, 1)


@pytest.fixture(scope="module")
def gauge():
    return F.make_gauge(DIMS, 3, "weak")


@pytest.mark.parametrize("prec", ["f64", "f32", "f16", "bf16", "q16", "q16f32"])
@pytest.mark.parametrize("recon", [12, 18])
def test_rule_with_tuning_off(gauge, prec, recon, monkeypatch):
    """the shape, and its result and reductions against one site and one
    right-hand side per thread"""
    from qphix_b200 import api
    lat = api.Lattice(DIMS)
    u = lat.gauge(prec, recon).upload(gauge)
    A = api.clover_build(lat.clover("f64"), lat.gauge("f64", 18).upload(gauge), 1, 0.1, 1.0)
    if prec != "f64":
        A = api.clover_convert(lat.clover(prec), A)
    D = api.ClovDslash(lat, -1.0, 1.0, 1.0)
    for nrhs in (1, 2, 3, 4):
        x, c = (lat.spinor(prec, nrhs).upload(np.stack([F.gaussian_spinor(DIMS, s + i) for i in range(nrhs)]))
                for s in (5, 15))
        y = lat.spinor(prec, nrhs)
        api.tune_enable(False)
        try:
            red = D.dslashAChiMinusBDPsiNorms(y, x, c, u, A, 0.25, 1, 1)
        finally:
            api.tune_enable(True)
        assert lat.dslash_shape() == rule(prec, recon, nrhs)
        got = y.download()
        with monkeypatch.context() as m:
            m.setenv("QPHIX_GPU_RHS_TILE", "1")
            m.setenv("QPHIX_GPU_SITES_PER_THREAD", "1")
            want = D.dslashAChiMinusBDPsiNorms(y, x, c, u, A, 0.25, 1, 1)
        assert lat.dslash_shape() == (1, 1)
        assert rel_l2(got, y.download()) < TOL[prec]
        assert np.all(np.abs(red - want) < 4 * TOL[prec] * want[:, :1])


@pytest.mark.parametrize("prec", ["f64", "f32", "f16", "bf16"])
@pytest.mark.parametrize("recon", [12, 18])
def test_captured_iteration_keeps_the_rule(gauge, prec, recon):
    """A solver's captured iteration reduces in its last Dslash, which nothing
    has timed: its shape, and with it the number of partials, must not follow
    what this process happened to time (here the operator's own launches)."""
    from qphix_b200 import api
    lat = api.Lattice(DIMS)
    M = api.EvenOddWilsonOperator(0.2, lat.gauge(prec, recon).upload(gauge))
    for nrhs in (1, 2, 3, 4):
        x, b = lat.spinor(prec, nrhs), lat.spinor(prec, nrhs)
        b.upload(np.stack([F.gaussian_spinor(DIMS, 5 + i) for i in range(nrhs)]))
        M(x, b)
        api.zero(x)
        api.InvBiCGStab(M, 3)(x, b, 1e-3)
        assert lat.dslash_shape(captured=True) == rule(prec, recon, nrhs), nrhs


@pytest.mark.parametrize("prec", ["f64", "f32", "f16"])
def test_forced_shapes(prec, monkeypatch):
    """the variables, one at a time and together"""
    from qphix_b200 import api
    lat = api.Lattice((4, 4, 4, 4))
    u = lat.gauge(prec, 12)
    x, y = lat.spinor(prec, 2), lat.spinor(prec, 2)
    D = api.Dslash(lat, -1.0, 1.0, 1.0)
    one = {"f64": (1, 1)}
    for tile, sites, lanes, want in (("1", None, None, one.get(prec, (1, 2))), ("2", None, None, one.get(prec, (2, 1))),
                                     (None, "1", None, (1, 1)), (None, "2", None, one.get(prec, (1, 2))),
                                     ("1", "1", None, (1, 1)), ("1", "2", None, one.get(prec, (1, 2))),
                                     ("2", "1", None, one.get(prec, (2, 1))), (None, None, "1", one.get(prec, (2, 0)))):
        with monkeypatch.context() as m:
            for name, v in (("RHS_TILE", tile), ("SITES_PER_THREAD", sites), ("RHS_LANES", lanes)):
                if v:
                    m.setenv("QPHIX_GPU_" + name, v)
            D.dslash(y, x, u, 1, 0)
        assert lat.dslash_shape() == want, (tile, sites, lanes)
