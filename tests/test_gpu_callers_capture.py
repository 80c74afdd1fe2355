"""fdtd_run captured by its caller on a stream of the caller's own: with
several steps per launch as with single ones, without a run before it."""
import pytest

from fdtdsarsim_b200 import _native
from helpers import bits_equal, make_params, native_for, random_problem

pytestmark = pytest.mark.gpu


def _sim(pc, mode):
    _, _, ca, cb, inc = random_problem(pc, 2)
    s = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), shell=_native.SHELL_SPLIT)
    s.set_option(_native.OPT_MULTISTEP, mode)
    s.set_materials(ca, cb)
    s.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
    return s


@pytest.mark.parametrize('warm', [False, True])
@pytest.mark.parametrize('mode', [_native.MULTI_OFF, _native.MULTI_RESIDENT, _native.MULTI_PAIR])
def test_first_run_can_be_captured(mode, warm):
    import torch
    pc = make_params(101, 53, 35, 17, 12, 12)
    sim, ref = _sim(pc, mode), _sim(pc, _native.MULTI_OFF)
    stream = torch.cuda.Stream()
    if warm:
        sim.run(2)
        sim.reset()
    sim.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sim.run(5)
    taken = sim.get_option(_native.OPT_STEP_PATH)
    with torch.cuda.stream(stream):
        graph.replay()
    sim.run(7)
    ref.run(12)
    sim.synchronize()
    assert all(bits_equal(sim.get_field(c), ref.get_field(c)) for c in _native.FIELD_NAMES)
    got, want = sim.get_phasors(), ref.get_phasors()
    assert all(bits_equal(got[k], want[k]) for k in want)
    pair = _native.PATH_PAIR | _native.PATH_SINGLE   # five and seven steps: one is left over
    assert taken == {_native.MULTI_OFF: _native.PATH_SINGLE, _native.MULTI_RESIDENT: _native.PATH_RESIDENT,
                     _native.MULTI_PAIR: pair if warm else _native.PATH_SINGLE}[mode]
    assert sim.get_option(_native.OPT_STEP_PATH) == {_native.MULTI_OFF: _native.PATH_SINGLE,
                                                     _native.MULTI_RESIDENT: _native.PATH_RESIDENT,
                                                     _native.MULTI_PAIR: pair}[mode]
    del graph
    sim.set_stream(0)
    sim.close()
    ref.close()
