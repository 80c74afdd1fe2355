"""A resident run leaves the device to others between its launches of about two
milliseconds: work of another stream, and another simulation, finish while a
long run is still going."""
import pytest

from fdtdsarsim_b200 import _native
from fdtdsarsim_b200.absorbers import packed_profiles
from fdtdsarsim_b200.gpu.main_sim import native_geometry
from helpers import bits_equal, make_params, native_for, random_problem

pytestmark = pytest.mark.gpu


def _sim(nx, ny, nz, nt, mode):
    pc = make_params(nx, ny, nz, nz // 2, nt, 4)
    _, _, ca, cb, inc = random_problem(pc, nx)
    s = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), shell=_native.SHELL_SPLIT)
    s.set_option(_native.OPT_MULTISTEP, mode)
    s.set_materials(ca, cb)
    s.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
    return s


@pytest.mark.parametrize('mode', [_native.MULTI_AUTO, _native.MULTI_OFF], ids=['resident', 'single'])
@pytest.mark.parametrize('other', ['kernel', 'simulation'])
def test_others_finish_during_a_long_run(mode, other):
    import torch
    nt = 12000   # 0.2 s or more
    a = _sim(61, 67, 43, nt, mode)
    b = _sim(45, 41, 33, 12, mode)
    x = torch.zeros(1 << 16, device='cuda')
    stream = torch.cuda.Stream()
    run = torch.cuda.ExternalStream(a.stream())
    b.run(2)
    b.reset()
    x += 1
    torch.cuda.synchronize()
    a.run(nt)
    if other == 'kernel':
        with torch.cuda.stream(stream):
            x += 1
        stream.synchronize()
    else:
        b.run(12)
        b.synchronize()
    during = not run.query()
    a.synchronize()
    want = _native.PATH_RESIDENT if mode == _native.MULTI_AUTO else _native.PATH_SINGLE
    assert a.get_option(_native.OPT_STEP_PATH) == want
    assert during
    a.close()
    b.close()


@pytest.mark.parametrize('dtype', ['float32', 'float64'])
@pytest.mark.parametrize('nx,ny,nz,runs', [(29, 31, 27, (301, 2, 140)), (61, 67, 43, (101, 90, 1)),
                                           (131, 90, 61, (47, 30, 3))])
def test_runs_of_several_launches_equal_single_steps(dtype, nx, ny, nz, runs):
    """Odd and even counts on either side of a launch's steps."""
    nt = sum(runs)
    pc = make_params(nx, ny, nz, nz // 2, nt, nt, dtype=dtype)
    _, _, ca, cb, inc = random_problem(pc, nx)
    for k in inc:   # a beam that vanishes on the plane's edges: long runs stay finite
        inc[k][:, [0, -1], :] = 0
        inc[k][:, :, [0, -1]] = 0
    sims = []
    for mode in (_native.MULTI_RESIDENT, _native.MULTI_OFF):
        s = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), shell=_native.SHELL_SPLIT)
        s.set_option(_native.OPT_MULTISTEP, mode)
        s.set_materials(ca, cb)
        s.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
        sims.append(s)
    for n in runs:
        for s in sims:
            s.run(n)
        assert all(bits_equal(sims[0].get_field(c), sims[1].get_field(c)) for c in _native.FIELD_NAMES)
        got, want = (s.get_phasors() for s in sims)
        assert all(bits_equal(got[k], want[k]) for k in want)
    for s in sims:
        s.close()


@pytest.mark.parametrize('nx,ny,nz,nt', [(27, 25, 31, 301), (61, 67, 43, 100)])
def test_incident_runs_of_several_launches_equal_split(nx, ny, nz, nt):
    import numpy as np
    pc = make_params(nx, ny, nz, nz // 2, nt, 0, cell_wl=0.05)
    src = np.random.default_rng(nx).standard_normal((2, 40, ny, nx)).astype('float32')
    out = []
    for opt, value in ((_native.OPT_MULTISTEP, _native.MULTI_RESIDENT),
                       (_native.OPT_KERNEL, _native.FDTD_KERNEL_SPLIT)):
        inc = _native.NativeIncident(native_geometry(pc), 40, 0)
        inc.set_absorbers(packed_profiles(pc))
        inc.set_option(opt, value)
        inc.set_excitation(src[0], src[1])
        inc.run()
        out.append({**inc.get_planes(), **inc.get_phasors()})
        inc.close()
    assert all(bits_equal(out[0][k], out[1][k]) and np.any(out[1][k]) for k in out[1])
