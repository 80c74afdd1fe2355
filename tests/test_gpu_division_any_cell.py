"""The float division by the cell size at cells of every scale, for every
float input: from 2 m on (no power of two) a subnormal quotient can lie on a
rounding boundary, where the product with a rounded reciprocal may fall on
either side; powers of two, the smallest and the largest cells."""
import numpy as np
import pytest

from fdtdsarsim_b200 import _native
from helpers import LAM, bits_equal, make_params, native_for, oracle_for, random_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('cell_size', [2.5, 3.0, 6.1, 47.3, 1.1e3, 1.7e6, 3.3e30, 3.4e38, 0.25, 8.0, 0.1, 1e-10,
                                       2e-38, 1e-42])
def test_float_division_is_exact_for_every_input(cell_size):
    tested, bad = _native.check_cell_division('float32', cell_size)
    assert tested == 2 ** 32
    assert bad == 0


@pytest.mark.parametrize('mode,path', [(_native.MULTI_OFF, _native.PATH_SINGLE),
                                       (_native.MULTI_RESIDENT, _native.PATH_RESIDENT),
                                       (_native.MULTI_PAIR, _native.PATH_PAIR)])
@pytest.mark.parametrize('cell_size', [0.0011, 0.7, 4.0, 2.61, 1.7e6])
def test_faint_fields_match_oracle_at_any_cell(cell_size, mode, path):
    """Fields whose CPML terms are subnormal; several steps per launch leave the
    cells with boundary quotients to the single step."""
    pc = make_params(101, 53, 35, 17, 6, 6, cell_wl=cell_size / LAM)
    assert np.float32(pc.geom_params.cell_size) == np.float32(cell_size)
    _, _, ca, cb, inc = random_problem(pc, 8)
    for k in inc:
        inc[k] *= np.float32(1e-38)
    orc = oracle_for(pc)
    orc.run(ca, cb, inc, 6)
    sim = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), shell=_native.SHELL_SPLIT)
    sim.set_option(_native.OPT_MULTISTEP, mode)
    sim.set_materials(ca, cb)
    sim.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
    sim.run(6)
    sim.synchronize()
    boundary = cell_size in (2.61, 1.7e6)
    assert sim.get_option(_native.OPT_STEP_PATH) == (_native.PATH_SINGLE if boundary else path)
    assert all(bits_equal(sim.get_field(c), getattr(orc, c)) for c in _native.FIELD_NAMES)
    assert np.any(orc.ex)
    sim.close()
