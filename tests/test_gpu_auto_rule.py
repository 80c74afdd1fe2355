"""FDTD_MULTI_AUTO leaves grids alone on which several steps per launch are
slower: thin ones for pairs, wide ones at the edge of L2 for resident steps
(single steps were measured 6 % to 28 % faster there); it keeps them on grids of
the same sizes in other shapes, and in double."""
import numpy as np
import pytest

from fdtdsarsim_b200 import _native
from fdtdsarsim_b200.absorbers import packed_profiles
from fdtdsarsim_b200.gpu.main_sim import native_geometry
from helpers import bits_equal, make_params, native_for

pytestmark = pytest.mark.gpu

SINGLE, RESIDENT, PAIR = _native.PATH_SINGLE, _native.PATH_RESIDENT, _native.PATH_PAIR


@pytest.mark.parametrize('nz,ny,nx,dtype,want', [
    (800, 34, 200, 'float32', SINGLE), (26, 939, 177, 'float32', SINGLE), (724, 33, 175, 'float32', SINGLE),
    (232, 51, 367, 'float32', SINGLE), (975, 33, 251, 'float32', SINGLE), (332, 32, 637, 'float32', SINGLE),
    (137, 123, 479, 'float32', PAIR), (43, 600, 165, 'float32', PAIR), (137, 328, 254, 'float32', PAIR),
    (54, 320, 257, 'float32', PAIR), (63, 266, 377, 'float32', PAIR), (25, 598, 643, 'float32', PAIR),
    (52, 85, 670, 'float32', SINGLE), (38, 90, 725, 'float32', SINGLE), (62, 168, 283, 'float32', SINGLE),
    (55, 133, 133, 'float32', RESIDENT), (45, 383, 74, 'float32', RESIDENT), (24, 24, 1500, 'float32', RESIDENT),
    (621, 46, 75, 'float32', RESIDENT), (700, 34, 70, 'float64', PAIR), (24, 260, 260, 'float64', PAIR),
    (47, 87, 107, 'float64', RESIDENT)])
def test_auto_takes_the_faster_path(nz, ny, nx, dtype, want):
    pc = make_params(nx, ny, nz, max(12, nz // 2), 4, 0, dtype=dtype)
    sim = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), shell=_native.SHELL_SPLIT)
    sim.set_option(_native.OPT_MULTISTEP, _native.MULTI_AUTO)
    sim.set_materials(np.ones((nz, ny, nx), dtype), np.ones((nz, ny, nx), dtype))
    sim.run(4)
    sim.synchronize()
    taken = sim.get_option(_native.OPT_STEP_PATH)
    sim.close()
    assert taken == want


@pytest.mark.parametrize('nz,ny,nx', [(52, 85, 670), (45, 383, 74)])
def test_incident_run_by_the_same_rule_equals_split(nz, ny, nx):
    """Single steps on the first grid (resident 5.4 ms per 60 steps, single
    4.7), resident ones on the second."""
    nt = 8
    pc = make_params(nx, ny, nz, nz // 2, nt, 0, cell_wl=0.05)
    src = np.random.default_rng(nx).standard_normal((2, nt, ny, nx)).astype('float32')
    out = []
    for opts in ({}, {_native.OPT_KERNEL: _native.FDTD_KERNEL_SPLIT}):
        inc = _native.NativeIncident(native_geometry(pc), nt, 0)
        inc.set_absorbers(packed_profiles(pc))
        for k, v in opts.items():
            inc.set_option(k, v)
        inc.set_excitation(src[0], src[1])
        inc.run()
        out.append({**inc.get_planes(), **inc.get_phasors()})
        inc.close()
    assert all(bits_equal(out[0][k], out[1][k]) and np.any(out[1][k]) for k in out[1])
