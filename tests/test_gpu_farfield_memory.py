"""The far field where little device memory is left: 1024 directions of a
741 x 741 plane take 91 MB at once; with less they go in smaller passes, with
the same bits (a direction's sums do not depend on the pass)."""
import numpy as np
import pytest

from fdtdsarsim_b200 import _native
from helpers import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', [np.complex64, np.complex128])
def test_far_field_with_80_mb_left(dtype):
    import torch
    n = 741 if dtype == np.complex64 else 523   # planes of 18 MB either way
    rng = np.random.default_rng(n)
    planes = [(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))).astype(dtype) for _ in range(4)]
    args = (n, n, 21, 0.0021, 2.0e3, np.linspace(-80.0, 80.0, 128), np.linspace(0.0, 170.0, 8), 5.4e9)
    want = _native.near2far(*planes, *args)
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (80 << 20), dtype=torch.uint8, device='cuda')
    got = _native.near2far(*planes, *args)
    del filler
    torch.cuda.empty_cache()
    assert all(bits_equal(got[k], want[k]) for k in want) and np.any(want['E_theta'])
