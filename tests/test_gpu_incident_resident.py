"""The incident run in one resident launch against the split passes, bit for
bit: recorded planes and incident phasors, with one cell and with vectors per
thread, odd and even step counts (the last odd step updates H in place), a
source that ends before the run and one that does not."""
import numpy as np
import pytest

from helpers import bits_equal, make_params
from fdtdsarsim_b200 import _native
from fdtdsarsim_b200.absorbers import packed_profiles
from fdtdsarsim_b200.gpu.main_sim import native_geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', ['float32', 'float64'])
@pytest.mark.parametrize('nx,ny,nz,nt,npulse', [(27, 25, 31, 9, 4), (33, 23, 30, 8, 8), (29, 31, 28, 2, 2),
                                                (61, 67, 43, 7, 5), (71, 57, 44, 6, 6)])
def test_resident_incident_run_equals_split(dtype, nx, ny, nz, nt, npulse):
    pc = make_params(nx, ny, nz, nz // 2, nt, 0, dtype=dtype, cell_wl=0.05)
    rng = np.random.default_rng(nx)
    src = rng.standard_normal((2, npulse, ny, nx)).astype(dtype)
    out = []
    for opts in ({_native.OPT_MULTISTEP: _native.MULTI_RESIDENT}, {_native.OPT_MULTISTEP: _native.MULTI_OFF},
                 {_native.OPT_KERNEL: _native.FDTD_KERNEL_SPLIT}):
        inc = _native.NativeIncident(native_geometry(pc), npulse, 0)
        inc.set_absorbers(packed_profiles(pc))
        for k, v in opts.items():
            inc.set_option(k, v)
        inc.set_excitation(src[0], src[1])
        inc.run()
        inc.run()   # a second run starts afresh
        out.append({**inc.get_planes(), **inc.get_phasors()})
        inc.close()
    if nt > 5:   # the source is four planes from the read-out
        assert any(np.any(v) for v in out[2].values())
    for other in out[:2]:
        for k, v in out[2].items():
            assert bits_equal(other[k], v), k
