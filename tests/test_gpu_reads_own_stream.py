"""Reading results back waits for the handle's stream only: not for work on
the legacy default stream or any other stream of the process."""
import pytest

from fdtdsarsim_b200 import _native
from helpers import make_params, native_for, random_problem

pytestmark = pytest.mark.gpu

READS = {'synchronize': lambda s: s.synchronize(), 'phasor': lambda s: s.get_phasor(4),
         'phasors': lambda s: s.get_phasors(), 'field': lambda s: s.get_field('ex')}


@pytest.mark.parametrize('read', READS)
@pytest.mark.parametrize('mode', [_native.MULTI_OFF, _native.MULTI_RESIDENT, _native.MULTI_PAIR])
def test_a_read_does_not_wait_for_the_default_stream(mode, read):
    import torch
    pc = make_params(148, 39, 26, 12, 4, 4)
    _, _, ca, cb, inc = random_problem(pc, 5)
    sim = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), shell=_native.SHELL_SPLIT)
    sim.set_option(_native.OPT_MULTISTEP, mode)
    sim.set_materials(ca, cb)
    sim.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
    torch.cuda._sleep(1000)   # loads the kernel
    torch.cuda.synchronize()
    sim.run(4)
    torch.cuda.ExternalStream(sim.stream()).synchronize()
    torch.cuda._sleep(1 << 31)   # about a second, on the default stream
    done = torch.cuda.Event()
    done.record()
    READS[read](sim)
    waited = done.query()
    torch.cuda.synchronize()
    sim.close()
    assert not waited
