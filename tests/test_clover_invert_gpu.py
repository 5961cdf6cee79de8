"""Clover inverses where the pivot is not the diagonal, and the clover build,
at site counts that leave a block of 32 partly filled.

The blocks are U diag(l) U^+ with |l| in [0.5, 2] of both signs, so the
condition is at most 4 (4.5 with the twist) and an FP64 elimination of six
steps stays within 6 x 4 x 1e-16 x a growth factor below 10: 1e-13.  Stored
in FP32 / FP16 the result is one rounding off.
"""
import numpy as np
import pytest

from helpers import rel_l2
from qphix_b200 import fields as F

pytestmark = pytest.mark.gpu

DIMS = [(6, 4, 2, 6), (2, 2, 2, 2), (4, 4, 2, 4), (10, 2, 6, 4)]  # 144, 8, 64 and 240 sites a checkerboard


def _blocks(dims, seed):
    """indefinite Hermitian blocks, some with a zero first row up to the last entry"""
    rng = np.random.default_rng(seed)
    n = F.vh(dims)
    m = rng.standard_normal((n, 2, 6, 6)) + 1j * rng.standard_normal((n, 2, 6, 6))
    q, _ = np.linalg.qr(m)
    lam = rng.uniform(0.5, 2.0, (n, 2, 6)) * rng.choice((-1.0, 1.0), (n, 2, 6))
    a = np.einsum("nbij,nbj,nbkj->nbik", q, lam, q.conj())
    a[::3] = 0
    flip = np.arange(5, -1, -1)
    a[::3, :, np.arange(6), flip] = np.array([1.5, -0.7, 1.0, 1.0, -0.7, 1.5])
    return (a + a.conj().swapaxes(-1, -2)) / 2


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("prec,bound", [("f64", 1e-13), ("f32", 1e-7), ("f16", 6e-4)])
def test_pivoted_inverses(dims, prec, bound):
    from qphix_b200 import api
    a = _blocks(dims, 3)
    lat = api.Lattice(dims)
    A = lat.clover("f64").upload(F.blocks_to_packed(a))
    got = api.clover_invert(lat.clover(prec), A).download().reshape(-1, 2, 36)
    assert rel_l2(got, F.blocks_to_packed(np.linalg.inv(a))) < bound
    mu, eps = 0.3, 0.2
    g5 = np.array([1.0, -1.0])[None, :, None, None] * np.eye(6)

    def full(f):
        d = f.download().reshape(-1, 2, 6, 6, 2)
        return d[..., 0] + 1j * d[..., 1]

    fp, fm = api.clover_invert_twisted(lat.full_clover(prec), lat.full_clover(prec), A, mu)
    assert rel_l2(full(fp), np.linalg.inv(a + 1j * mu * g5)) < bound
    assert rel_l2(full(fm), np.linalg.inv(a - 1j * mu * g5)) < bound
    up, dn, od = api.clover_invert_ndtm(lat.full_clover(prec), lat.full_clover(prec), lat.clover(prec), A, mu, eps)
    q = np.linalg.inv(a @ a + (mu * mu - eps * eps) * np.eye(6))
    assert rel_l2(full(up), q @ (a - 1j * mu * g5)) < 5 * bound  # the condition enters squared
    assert rel_l2(full(dn), q @ (a + 1j * mu * g5)) < 5 * bound
    assert rel_l2(od.download().reshape(-1, 2, 36), F.blocks_to_packed(eps * q)) < 5 * bound


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("recon", [18, 12])
@pytest.mark.parametrize("prec,bound", [("f64", 1e-14), ("f32", 1e-7), ("bf16", 5e-3)])
def test_build(dims, recon, prec, bound):
    from qphix_b200 import api
    g = F.make_gauge(dims, 5, "gaussian")
    ref = F.make_clover(dims, g, 0.1, 1.3, 0.8)
    lat = api.Lattice(dims)
    u = lat.gauge("f64", recon).upload(g)
    for cb in (0, 1):
        got = api.clover_build(lat.clover(prec), u, cb, 0.1, 1.3, 0.8).download()
        assert rel_l2(got.reshape(ref[cb].shape), ref[cb]) < bound
