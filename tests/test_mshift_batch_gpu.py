"""Multishift CG's batched shift updates (mshift_update_kernel): iterates at
every remainder of a batch, at odd site counts and shift counts, against the
oracle's (include/qphix/minvcg.h:279-384).

The FP64 iterates follow the same recurrences on the same values, so after k
iterations they differ from the oracle's by k roundings of the operator and
its reductions, amplified by the recurrence: 1e-11 relative covers 20
iterations of a well-conditioned system (each ~1e-15, factor ~10 apiece at
most for the first ones); FP32 the same with 6e-8 in place of 1e-16.
"""
import numpy as np
import pytest

from helpers import make_setup, rel_l2
from qphix_b200 import fields as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_iters", [1, 2, 3, 8, 9, 10, 16, 17, 18, 400])
@pytest.mark.parametrize("ns,dims", [(1, (4, 4, 4, 8)), (3, (6, 4, 2, 6)), (5, (4, 4, 4, 8)), (32, (6, 2, 4, 4))])
def test_iterates(oracle, max_iters, ns, dims):
    from qphix_b200 import api
    s = make_setup(dims, seed=31, gauge_kind="weak", mass=0.2)
    lat = api.Lattice(dims)
    M = api.EvenOddWilsonOperator(s["mass"], lat.gauge("f64", 12).upload(s["gauge"]))
    O = oracle.OracleOp("wilson", oracle.make_lattice(dims, -1.0, 1.0, 1.0), s["gauge"], mass=s["mass"])
    b = F.gaussian_spinor(dims, 33)
    shifts = np.logspace(-3, 0.5, ns)
    tol = np.logspace(-9, -4, ns)  # the shifts converge in different iterations
    gb = lat.spinor("f64").upload(b)
    xs = [lat.spinor("f64") for _ in shifts]
    solve = api.MInvCG(M, max_iters)
    xo, io, _, _ = oracle.minvcg(O, b, shifts, tol, max_iters)
    for _ in range(2):  # the second solve replays the captured batch
        try:
            it, _, _ = solve(xs, gb, shifts, tol)
            assert it == io
        except RuntimeError as e:
            assert "converge" in str(e) and max_iters < 400
        for k in range(ns):
            assert rel_l2(xs[k].download(), xo[k]) < 1e-11, (k, shifts[k])


@pytest.mark.parametrize("prec,bound", [("f32", 1e-5), ("f16", 2e-2)])
def test_low_precision(oracle, prec, bound):
    """FP32 (chunks) and FP16 (whole sites): every shift within the storage's
    reach of the oracle's solution."""
    from qphix_b200 import api
    dims = (6, 4, 2, 6)
    s = make_setup(dims, seed=35, gauge_kind="weak", mass=0.2)
    lat = api.Lattice(dims)
    M = api.EvenOddWilsonOperator(s["mass"], lat.gauge(prec, 12).upload(s["gauge"]))
    O = oracle.OracleOp("wilson", oracle.make_lattice(dims, -1.0, 1.0, 1.0), s["gauge"], mass=s["mass"])
    b = F.gaussian_spinor(dims, 36)
    shifts, tol = [0.01, 0.1, 1.0, 2.0, 3.0], [1e-3 if prec == "f16" else 1e-6] * 5
    gb = lat.spinor(prec).upload(b)
    xs = [lat.spinor(prec) for _ in shifts]
    api.MInvCG(M, 200)(xs, gb, shifts, tol)
    xo, _, _, _ = oracle.minvcg(O, b, shifts, [1e-10] * 5, 400)
    for x, xr in zip(xs, xo):
        assert rel_l2(x.download(), xr) < bound
