"""Multishift CG's residual buffers: smaller batches (QPHIX_GPU_MSHIFT_BATCH,
or what a device that is nearly full leaves) give the same bits, the solve
needs no more memory than its smallest batch does, leaves half of what was
free, and gives its buffers back where the lattice needs the memory."""
import numpy as np
import pytest

from qphix_b200 import fields as F

pytestmark = pytest.mark.gpu

NS = 5
SHIFTS, RSD = np.logspace(-3, 0.5, NS), np.logspace(-9, -4, NS)


def _system(api, dims, prec="f64"):
    lat = api.Lattice(dims)
    b = lat.spinor(prec).upload(F.gaussian_spinor(dims, 1))
    M = api.EvenOddWilsonOperator(0.2, lat.gauge(prec, 18).upload(F.make_gauge(dims, 3, "weak")))
    return lat, M, b, [lat.spinor(prec) for _ in range(NS)]


@pytest.mark.parametrize("max_iters", [1, 3, 9, 400])
@pytest.mark.parametrize("prec", ["f64", "f32", "f16"])
def test_batches_give_the_same_bits(max_iters, prec, monkeypatch):
    """every power of two up to the largest batch; other values round down.
    16-bit storage rounds the vectors once a batch, so there the bits of the
    batches differ and the iteration count is what has to agree."""
    from qphix_b200 import api
    rsd = RSD if prec == "f64" else np.maximum(RSD, 1e-5 if prec == "f32" else 1e-2)
    found = {}
    for batch in ("1", "2", "3", "4", "8", None):
        with monkeypatch.context() as m:
            if batch:
                m.setenv("QPHIX_GPU_MSHIFT_BATCH", batch)
            lat, M, b, xs = _system(api, (6, 4, 2, 6), prec)
            try:
                it = api.MInvCG(M, max_iters)(xs, b, SHIFTS, rsd)[0]
            except RuntimeError as e:
                assert "converge" in str(e) and max_iters < 400
                it = -1
            found[batch] = it, np.stack([x.download() for x in xs])
    for batch in found:
        assert found[batch][0] == found["1"][0]
        if prec != "f16":
            assert np.array_equal(found[batch][1], found["1"][1]), batch
    assert np.array_equal(found["3"][1], found["2"][1])


def _round(n):
    return -(-n // (2 << 20)) * (2 << 20)  # cudaMalloc's granularity


@pytest.fixture
def fill():
    """fill(left): take the device's free memory but `left` bytes"""
    import torch
    held = []

    def take(left):
        torch.cuda.synchronize()
        n = torch.cuda.mem_get_info()[0] - left
        if n > 0:
            held.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
    yield take
    held.clear()
    torch.cuda.empty_cache()


def test_nearly_full_device(fill):
    """Memory for the solve's own vectors (p0, two products, NS directions, a
    residual, the operator's temporary) and three spinors more."""
    import torch

    from qphix_b200 import api
    dims = (16, 16, 16, 32)
    want = {}
    for full in (False, True):
        lat, M, b, xs = _system(api, dims)
        spinor = _round(lat.vh * 24 * 8)
        lat.sync()
        if full:
            fill((3 + NS + 1 + 1 + 3) * spinor)
        it = api.MInvCG(M, 400)(xs, b, SHIFTS, RSD)[0]
        if full:
            # of the three spinors at most half went into buffers
            assert torch.cuda.mem_get_info()[0] >= 1.5 * spinor - (2 << 20)
        want[full] = it, np.stack([x.download() for x in xs])
        del lat, M, b, xs
    assert want[True][0] == want[False][0]
    assert np.array_equal(want[True][1], want[False][1])


def test_buffers_are_given_back(fill):
    """a field that does not fit beside the solver's idle temporaries gets
    their memory, and the next solve takes new ones"""
    from qphix_b200 import api
    lat, M, b, xs = _system(api, (16, 16, 16, 32))
    solve = api.MInvCG(M, 400)
    it = solve(xs, b, SHIFTS, RSD)[0]
    want = np.stack([x.download() for x in xs])
    spinor = _round(lat.vh * 24 * 8)
    fill(2 * spinor)
    extra = lat.spinor("f64", 4)
    extra.close()
    assert solve(xs, b, SHIFTS, RSD)[0] == it
    assert np.array_equal(np.stack([x.download() for x in xs]), want)
