"""Several time steps per pass (FDTD_OPT_MULTISTEP) against the oracle, bit
for bit: the arithmetic of every cell is the single step's, so fields and
phasors must be equal in every bit."""
import numpy as np
import pytest

from fdtdsarsim_b200 import _native
from helpers import bits_equal, make_params, native_for, oracle_for, random_problem

pytestmark = pytest.mark.gpu

# nx, ny, nz, npml, tfsf_z, steps run, dtype
PAIR = [
    # column widths around one and two tiles of 120 cells, rows around 13,
    # partial last tiles, the injection plane in and beside the z faces
    (148, 39, 26, 10, 12, 5, 'float32'),
    (156, 38, 30, 10, 9, 4, 'float32'),
    (261, 45, 30, 10, 19, 5, 'float32'),
    (300, 70, 40, 10, 10, 4, 'float32'),
    (173, 53, 40, 10, 28, 4, 'float32'),
    (70, 61, 37, 10, 36, 4, 'float32'),
    (140, 45, 200, 10, 100, 3, 'float32'),
    (77, 41, 24, 7, 14, 6, 'float32'),
    (93, 64, 31, 3, 1, 4, 'float32'),
    # doubles: tiles of 60 cells
    (140, 33, 26, 10, 12, 4, 'float64'),
    (85, 50, 37, 10, 27, 5, 'float64'),
    (150, 61, 30, 5, 2, 3, 'float64'),
]


# grids down to the smallest, rows of every unit width, odd and even runs
RESIDENT = [
    (27, 25, 23, 10, 12, 7, 'float32'),
    (7, 8, 9, 2, 4, 6, 'float32'),
    (150, 33, 26, 10, 20, 4, 'float32'),
    (64, 70, 31, 7, 14, 5, 'float32'),
    (33, 23, 25, 10, 12, 6, 'float64'),
    (45, 41, 29, 10, 24, 5, 'float64'),
]


def _multi(pc, ca, cb, inc, mode, phasor_mode=0):
    sim = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), phasor_mode, shell=_native.SHELL_SPLIT)
    sim.set_option(_native.OPT_MULTISTEP, mode)
    sim.set_materials(ca, cb)
    sim.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
    return sim


def _assert_matches(orc, sim):
    for c in _native.FIELD_NAMES:
        assert bits_equal(sim.get_field(c), getattr(orc, c)), c
    for k, name in enumerate(_native.PHASOR_NAMES):
        assert bits_equal(sim.get_phasor(k), orc.ph[name]), name


@pytest.mark.parametrize('case,mode', [(c, _native.MULTI_PAIR) for c in PAIR]
                         + [(c, _native.MULTI_RESIDENT) for c in RESIDENT],
                         ids=lambda c: 'x'.join(map(str, c)) if isinstance(c, tuple) else
                         {_native.MULTI_PAIR: 'pair', _native.MULTI_RESIDENT: 'resident'}[c])
def test_multi_step_matches_oracle(case, mode):
    """A run, then a second one from the field set that the first left;
    between them odd and even counts, injection ending inside the first."""
    nx, ny, nz, npml, tfsf, nt, dtype = case
    pc = make_params(nx, ny, nz, tfsf, nt + 3, nt - 1, dtype=dtype, npml=npml)
    _, _, ca, cb, inc = random_problem(pc, nx + ny)
    orc = oracle_for(pc)
    sim = _multi(pc, ca, cb, inc, mode)
    try:
        for n in (nt, 3):
            orc.run(ca, cb, inc, n)
            sim.run(n)
            sim.synchronize()
            _assert_matches(orc, sim)
    finally:
        sim.close()
