"""A fused tile that the fused step does not take is refused whatever the path
of the run, as it is without several steps per launch."""
import numpy as np
import pytest

from fdtdsarsim_b200 import _native
from fdtdsarsim_b200.absorbers import packed_profiles
from fdtdsarsim_b200.gpu.main_sim import native_geometry
from helpers import make_params, native_for, random_problem

pytestmark = pytest.mark.gpu

TILES = [(32, 5), (64, 4)]


def _refused(call):
    with pytest.raises(_native.FdtdError) as ei:
        call()
    assert ei.value.code == _native.FDTD_ERR_INVALID and 'tile' in str(ei.value)


@pytest.mark.parametrize('tile', TILES)
@pytest.mark.parametrize('mode', [_native.MULTI_OFF, _native.MULTI_AUTO, _native.MULTI_RESIDENT, _native.MULTI_PAIR])
def test_unsupported_tile_is_refused_on_every_path(mode, tile):
    pc = make_params(101, 53, 35, 17, 8, 8)
    _, _, ca, cb, inc = random_problem(pc, 1)
    sim = native_for(pc, _native.FDTD_KERNEL_FUSED, tile, shell=_native.SHELL_SPLIT)
    sim.set_option(_native.OPT_MULTISTEP, mode)
    sim.set_materials(ca, cb)
    sim.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
    for chunk in (0, 2):
        sim.set_option(_native.OPT_GRAPH_CHUNK, chunk)
        _refused(lambda: sim.run(8))
    _refused(lambda: sim.grad_forward(4))
    sim.set_option(_native.OPT_TILE_X, 32)
    sim.set_option(_native.OPT_TILE_Y, 4)
    sim.reset()
    sim.run(8)
    assert np.any(sim.get_field('ex'))
    sim.close()


@pytest.mark.parametrize('mode', [_native.MULTI_OFF, _native.MULTI_AUTO])
def test_unsupported_tile_is_refused_by_the_incident_run(mode):
    pc = make_params(27, 25, 31, 15, 9, 0, cell_wl=0.05)
    inc = _native.NativeIncident(native_geometry(pc), 4, 0)
    inc.set_absorbers(packed_profiles(pc))
    inc.set_excitation(*np.ones((2, 4, 25, 27), np.float32))
    inc.set_option(_native.OPT_MULTISTEP, mode)
    inc.set_option(_native.OPT_TILE_Y, 5)
    _refused(inc.run)
    inc.set_option(_native.OPT_TILE_Y, 4)
    inc.run()
    inc.close()
