"""The autotuner's decisions, on a stand-in for the device handle that
reports given times and paths."""
import pytest

from fdtdsarsim_b200 import _native, tuning
from fdtdsarsim_b200.gpu.main_sim import native_geometry
from helpers import make_params

SPLIT, FUSED = _native.FDTD_KERNEL_SPLIT, _native.FDTD_KERNEL_FUSED
PATHS = {_native.MULTI_OFF: _native.PATH_SINGLE, _native.MULTI_RESIDENT: _native.PATH_RESIDENT,
         _native.MULTI_PAIR: _native.PATH_PAIR}


class FakeSim:
    """times: (kernel, tile_y, slab, shell, multi) -> (step ms, phasor ms) of a
    step; other candidates take 9 and 1. narrow: no pairs."""
    times = {}
    narrow = False

    def __init__(self, geom, device=0):
        self.opt = {_native.OPT_MULTISTEP: _native.MULTI_OFF}
        self.steps = 0

    def set_option(self, opt, value):
        self.opt[opt] = value

    def get_option(self, opt):
        if opt != _native.OPT_STEP_PATH:
            return self.opt[opt]
        multi = self.opt[_native.OPT_MULTISTEP] if self.opt[_native.OPT_KERNEL] == FUSED else 0
        return _native.PATH_SINGLE if self.narrow and multi == _native.MULTI_PAIR else PATHS[multi]

    def kernel_time(self, kind):
        o = self.opt
        key = tuple(o.get(k) for k in (_native.OPT_KERNEL, _native.OPT_TILE_Y, _native.OPT_FUSED_SLAB,
                                       _native.OPT_SHELL, _native.OPT_MULTISTEP))
        t = self.times.get(key, (9.0, 1.0))
        return t[0 if kind == _native.TIME_STEP else 1] * self.steps, self.steps

    def clear_kernel_time(self):
        self.steps = 0

    def run(self, n):
        self.steps += n

    def set_absorbers(self, *a):
        pass

    set_materials = reset = synchronize = close = set_absorbers


@pytest.fixture
def tune(tmp_path, monkeypatch):
    monkeypatch.setenv('FDTDSARSIM_B200_TUNING', str(tmp_path / 'tune.json'))
    geom = native_geometry(make_params(41, 37, 35, 16, 9, 9))

    def run(times, narrow=False):
        fake = type('Sim', (FakeSim,), {'times': times, 'narrow': narrow})
        monkeypatch.setattr(tuning._native, 'NativeSim', fake)
        best, timings = tuning.autotune(geom)
        assert len(timings) == len(tuning.CANDIDATES)
        assert tuning.choose(geom) == best
        return best
    return run


FUSED4 = (FUSED, 4, 0, _native.SHELL_SPLIT)
RES, PAIR = FUSED4 + (_native.MULTI_RESIDENT,), FUSED4 + (_native.MULTI_PAIR,)


@pytest.mark.parametrize('times,want', [
    # resident times hold their phasors, the others' come beside
    ({RES: (0.076, 0.0), PAIR: (0.070, 0.013)}, _native.MULTI_RESIDENT),
    ({RES: (0.076, 0.0), PAIR: (0.060, 0.013)}, _native.MULTI_PAIR),
    ({RES: (0.076, 0.0), FUSED4 + (0,): (0.075, 0.011)}, _native.MULTI_RESIDENT)])
def test_candidates_are_compared_by_the_whole_step(tune, times, want):
    assert tune(times)['multi'] == want


def test_a_candidate_that_fell_back_is_not_taken_for_its_name(tune):
    times = {PAIR: (0.080, 0.01), FUSED4 + (0,): (0.081, 0.01)}
    assert tune(times)['multi'] == _native.MULTI_PAIR
    assert tune(times, narrow=True)['multi'] == _native.MULTI_OFF


@pytest.mark.parametrize('multi', [RES, PAIR])
def test_several_steps_per_pass_keep_the_fastest_single_step_beside_them(tune, multi):
    fast = (FUSED, 8, 0, _native.SHELL_MARCH)
    best = tune({multi: (0.05, 0.0), fast + (0,): (0.07, 0.01), FUSED4 + (0,): (0.08, 0.01)})
    assert best == {'kernel': FUSED, 'tile_x': 32, 'tile_y': 8, 'zchunk': 0, 'slab': 0,
                    'shell': _native.SHELL_MARCH, 'multi': multi[-1]}
