"""The far field's matrix product at the edges of its tiles (64 directions, 64
columns of 4 per plane row, 16 cells of x) and of its passes (1024
directions), against the oracle's sum. Both sum the same float64 terms in
another order: with n cells the difference is some n^1/2 roundings of 1e-16
of the peak, far below 1e-11."""
import numpy as np
import pytest

import fdtd_oracle as O
from fdtdsarsim_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('ny,nx,nthetas,nphis,dtype', [
    (3, 3, 1, 1, np.complex64), (15, 17, 63, 1, np.complex128), (17, 31, 65, 1, np.complex64),
    (33, 15, 5, 26, np.complex128), (5, 7, 345, 3, np.complex64)])
def test_tile_and_pass_edges(ny, nx, nthetas, nphis, dtype):
    rng = np.random.default_rng(ny * nx)
    planes = [(rng.standard_normal((ny, nx)) + 1j * rng.standard_normal((ny, nx))).astype(dtype)
              for _ in range(4)]
    thetas, phis = np.linspace(-75.0, 80.0, nthetas), np.linspace(0.0, 170.0, nphis)
    got = _native.near2far(*planes, nx, ny, 21, 0.0021, 2.0e3, thetas, phis, 5.4e9)
    ref = O.near2far(*planes, nx, ny, 21, 0.0021, 2.0e3, thetas, phis, 5.4e9)
    for k in ('E_theta', 'E_phi', 'H_theta', 'H_phi'):
        r = np.asarray(ref[k]).reshape(nphis, nthetas)
        assert np.max(np.abs(got[k] - r)) <= 1e-11 * np.max(np.abs(r)), k
