"""The far field of long, low planes, whose rows are summed in parts, and of
many directions of a small plane in one pass, against the oracle's sum: the
same float64 terms in another order, relative 1e-11 of the peak (some n^1/2
roundings of 1e-16 with n cells)."""
import numpy as np
import pytest

import fdtd_oracle as O
from fdtdsarsim_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('ny,nx,nthetas,nphis,dtype', [
    (3, 511, 2, 1, np.complex64), (3, 513, 2, 1, np.complex64), (3, 9473, 4, 1, np.complex64),
    (11, 577, 16, 1, np.complex128), (255, 513, 1, 1, np.complex64), (259, 513, 1, 1, np.complex64),
    (21, 601, 65, 2, np.complex128), (3, 3, 9000, 2, np.complex64), (19, 19, 331, 7, np.complex128)])
def test_parts_and_passes(ny, nx, nthetas, nphis, dtype):
    rng = np.random.default_rng(ny * nx)
    planes = [(rng.standard_normal((ny, nx)) + 1j * rng.standard_normal((ny, nx))).astype(dtype)
              for _ in range(4)]
    thetas, phis = np.linspace(-75.0, 80.0, nthetas), np.linspace(0.0, 170.0, nphis)
    got = _native.near2far(*planes, nx, ny, 21, 0.0021, 2.0e3, thetas, phis, 5.4e9)
    ref = O.near2far(*planes, nx, ny, 21, 0.0021, 2.0e3, thetas, phis, 5.4e9)
    for k in ('E_theta', 'E_phi', 'H_theta', 'H_phi'):
        r = np.asarray(ref[k]).reshape(nphis, nthetas)
        assert np.max(np.abs(got[k] - r)) <= 1e-11 * np.max(np.abs(r)), k
