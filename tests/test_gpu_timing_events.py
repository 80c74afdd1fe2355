"""FDTD_OPT_TIMING keeps at most 4096 groups of events waiting, whatever the
step path: the process does not grow with the number of timed runs (12288
more groups would hold 36864 events, some 22 MB), and every step is counted."""
import pytest

from fdtdsarsim_b200 import _native
from helpers import make_params, native_for, random_problem

pytestmark = pytest.mark.gpu


def _resident_mb():
    with open('/proc/self/statm') as f:
        return int(f.read().split()[1]) * 4096 / 1e6


@pytest.mark.parametrize('mode', [_native.MULTI_RESIDENT, _native.MULTI_OFF])
def test_timed_runs_do_not_grow_the_process(mode):
    runs = 4 * 4096
    pc = make_params(27, 25, 23, 12, 2 * runs, 2)
    _, _, ca, cb, inc = random_problem(pc, 5)
    sim = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), shell=_native.SHELL_SPLIT)
    sim.set_option(_native.OPT_MULTISTEP, mode)
    sim.set_materials(ca, cb)
    sim.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
    sim.set_option(_native.OPT_TIMING, 1)
    for k in range(runs):
        if k == 4096:
            before = _resident_mb()
        sim.run(2)
    grown = _resident_mb() - before
    ms, steps = sim.kernel_time(_native.TIME_STEP)
    sim.close()
    assert steps == 2 * runs and ms > 0
    assert grown < 8
