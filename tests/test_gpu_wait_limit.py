"""A wait inside a step kernel that runs out (FDTD_OPT_WAIT_LIMIT_US, here 0:
the resident step's grid barrier gives up where a block is not there yet; no
copy is in flight and every block leaves) is an error of every call that hands
out what the run left, until a reset; the run after it is whole again."""
import numpy as np
import pytest

from fdtdsarsim_b200 import _native
from fdtdsarsim_b200.absorbers import packed_profiles
from fdtdsarsim_b200.gpu.main_sim import native_geometry
from helpers import bits_equal, make_params, native_for, random_problem

pytestmark = pytest.mark.gpu

NT = 40


def _sim(pc, mode):
    _, _, ca, cb, inc = random_problem(pc, 11)
    sim = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), shell=_native.SHELL_SPLIT)
    sim.set_option(_native.OPT_MULTISTEP, mode)
    sim.set_materials(ca, cb)
    sim.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
    return sim


def _fails(call, code=_native.FDTD_ERR_CUDA, word='wait'):
    with pytest.raises(_native.FdtdError) as ei:
        call()
    assert ei.value.code == code and word in str(ei.value)


@pytest.mark.parametrize('chunk', [0, 8])
def test_every_read_reports_a_wait_that_ran_out(chunk):
    pc = make_params(64, 57, 41, 20, NT, NT)
    sim = _sim(pc, _native.MULTI_RESIDENT)
    sim.set_option(_native.OPT_GRAPH_CHUNK, chunk)
    sim.set_option(_native.OPT_WAIT_LIMIT_US, 0)
    assert sim.get_option(_native.OPT_WAIT_LIMIT_US) == 0
    sim.run(NT)
    w = np.ones(sim.ny_ph + sim.nx_ph + sim.nz_ph - 1)
    ph = {f'{c}_inc_phasor': np.zeros((sim.ny_ph, sim.nx_ph), np.complex64) for c in ('ex', 'ey', 'hx', 'hy')}
    for _ in range(2):
        for read in (sim.synchronize, lambda: sim.get_phasor(4), sim.get_phasors, lambda: sim.get_field('ex'),
                     lambda: sim.near_field_power(ph, 5, w)):
            _fails(read)
    _fails(lambda: sim.grad_forward(10))
    zero = np.zeros((4, sim.ny_ph, sim.nx_ph))
    _fails(lambda: sim.grad_backward(zero, zero, 5), _native.FDTD_ERR_STATE, 'grad_forward')
    sim.set_option(_native.OPT_WAIT_LIMIT_US, 2000000)
    sim.reset()
    sim.run(NT)
    sim.synchronize()
    ref = _sim(pc, _native.MULTI_OFF)
    ref.run(NT)
    assert all(bits_equal(sim.get_field(c), ref.get_field(c)) for c in _native.FIELD_NAMES)
    got, want = sim.get_phasors(), ref.get_phasors()
    assert all(bits_equal(got[k], want[k]) for k in want) and np.any(want['ex_ph_u'])
    sim.close()
    ref.close()


def test_a_batch_reports_its_members_wait():
    pc = make_params(64, 57, 41, 20, NT, NT)
    sim = _sim(pc, _native.MULTI_RESIDENT)
    sim.set_option(_native.OPT_WAIT_LIMIT_US, 0)
    batch = _native.Batch([sim], mode=_native.BATCH_STREAMS)   # one member: its own step path
    batch.run(NT)
    for _ in range(2):
        _fails(batch.synchronize)
    batch.close()
    _fails(sim.synchronize)
    sim.close()


def test_an_incident_run_hands_out_nothing_after_it():
    pc = make_params(61, 67, 43, 21, NT, 0, cell_wl=0.05)
    rng = np.random.default_rng(1)
    inc = _native.NativeIncident(native_geometry(pc), 9, 0)
    inc.set_absorbers(packed_profiles(pc))
    inc.set_excitation(*rng.standard_normal((2, 9, 67, 61)).astype('float32'))
    inc.run()
    want = inc.get_planes()
    inc.set_option(_native.OPT_WAIT_LIMIT_US, 0)
    _fails(inc.run)
    for read in (inc.get_planes, inc.get_phasors):
        _fails(read, _native.FDTD_ERR_STATE, 'not done')
    inc.set_option(_native.OPT_WAIT_LIMIT_US, 2000000)
    inc.run()
    got = inc.get_planes()
    inc.close()
    assert all(bits_equal(got[k], want[k]) for k in want) and any(np.any(v) for v in want.values())


@pytest.mark.parametrize('value', [-1, 10000001])
def test_limits_out_of_range_are_refused(value):
    sim = native_for(make_params(27, 25, 23, 14, 4, 4))
    _fails(lambda: sim.set_option(_native.OPT_WAIT_LIMIT_US, value), _native.FDTD_ERR_INVALID, 'wait limit')
    sim.close()


def test_a_callers_graph_reports_a_wait_of_any_replay():
    import torch
    pc = make_params(64, 57, 41, 20, 3 * NT, 3 * NT)
    sim = _sim(pc, _native.MULTI_RESIDENT)
    stream = torch.cuda.Stream()
    sim.set_stream(stream.cuda_stream)
    sim.set_option(_native.OPT_WAIT_LIMIT_US, 0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sim.run(NT)
    sim.synchronize()   # nothing has run
    for _ in range(2):
        with torch.cuda.stream(stream):
            graph.replay()
        _fails(sim.synchronize)
        _fails(sim.get_phasors)
        sim.reset()
        sim.synchronize()
    del graph
    sim.set_stream(0)
    sim.close()
