"""The fold of block partials (fold_kernel) on both sides of the line where it
takes two partials a load: even and odd block counts, at three and four loads
a lane, against numpy's sum of the downloaded values.

FP64 sums of n positive terms in any two orders differ by at most 2 n eps
relatively, in practice by a few eps; 1e-13 is the repository's FP64 bound.
"""
import numpy as np
import pytest

from qphix_b200 import fields as F

pytestmark = pytest.mark.gpu


# sites of a checkerboard / 128: 124 (3 loads a lane with 32 values), 128 and
# 130 (4, in pairs; the second with a remainder), 129 (odd); 4096 with one value
@pytest.mark.parametrize("dims,nrhs", [((4, 4, 32, 62), 32), ((4, 8, 16, 64), 32), ((4, 8, 16, 65), 32),
                                       ((4, 4, 48, 43), 32), ((4, 8, 16, 65), 9), ((32, 32, 32, 32), 1)])
def test_norm_and_product(dims, nrhs):
    from qphix_b200 import api
    lat = api.Lattice(dims)
    rng = np.random.default_rng(3)
    v = F.gaussian_complex(rng, (2, nrhs, lat.vh, 4, 3))
    x, y = (lat.spinor("f64", nrhs).upload(a) for a in v)
    a, b = v.reshape(2, nrhs, -1)
    nn, ip = api.norm2(x), api.inner_product(x, y)
    for _ in range(2):
        assert np.array_equal(nn, api.norm2(x))  # the order of every addition is fixed
    want = np.einsum("ij,ij->i", a.conj(), a).real
    assert np.all(np.abs(nn - want) < 1e-13 * want)
    assert np.all(np.abs(ip - np.einsum("ij,ij->i", a.conj(), b)) < 1e-13 * want)
