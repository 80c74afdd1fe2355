"""A captured step graph belongs to where it was captured: a member's resident
graph is not replayed among a batch's streams, nor a batch's single steps when
the member runs alone."""
import pytest

from fdtdsarsim_b200 import _native
from helpers import bits_equal, make_params, native_for, random_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('first', ['alone', 'batch'])
@pytest.mark.parametrize('mode,alone,side', [
    (_native.MULTI_RESIDENT, _native.PATH_RESIDENT, _native.PATH_SINGLE),
    (_native.MULTI_AUTO, _native.PATH_RESIDENT, _native.PATH_SINGLE),
    (_native.MULTI_PAIR, _native.PATH_PAIR, _native.PATH_PAIR)])
def test_member_graphs_follow_where_they_run(mode, alone, side, first):
    sims, refs = [], []
    for k in range(2):
        pc = make_params(101, 53 - 4 * k, 35, 17, 48, 48)
        _, _, ca, cb, inc = random_problem(pc, k)
        for out, m in ((sims, mode), (refs, _native.MULTI_OFF)):
            s = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), shell=_native.SHELL_SPLIT)
            s.set_option(_native.OPT_MULTISTEP, m)
            s.set_materials(ca, cb)
            s.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
            out.append(s)
    for s in sims:
        s.set_option(_native.OPT_GRAPH_CHUNK, 4)
    batch = _native.Batch(sims, streams=True)
    for turn in range(4):
        if (turn % 2 == 0) == (first == 'alone'):
            for s in sims:
                s.run(12)
                s.synchronize()
        else:
            batch.run(12)
            batch.synchronize()
        want = alone if (turn % 2 == 0) == (first == 'alone') else side
        assert [s.get_option(_native.OPT_STEP_PATH) for s in sims] == [want, want]
    for a, b in zip(sims, refs):
        b.run(48)
        assert all(bits_equal(a.get_field(c), b.get_field(c)) for c in _native.FIELD_NAMES)
        got, want = a.get_phasors(), b.get_phasors()
        assert all(bits_equal(got[k], want[k]) for k in want)
    batch.close()
    for s in sims + refs:
        s.close()
