"""The tuner measures several steps per pass beside the single-step kernels,
keeps what it measured in its cache, and choose() hands it on; a run with the
tuned choice equals the split kernel's bit for bit."""
import numpy as np
import pytest

from fdtdsarsim_b200 import _native, tuning
from fdtdsarsim_b200.gpu.main_sim import native_geometry
from helpers import make_params, native_for, random_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('multi', [_native.MULTI_OFF, _native.MULTI_RESIDENT, _native.MULTI_PAIR])
def test_tuned_choice_round_trips_and_runs(tmp_path, monkeypatch, multi):
    monkeypatch.setenv('FDTDSARSIM_B200_TUNING', str(tmp_path / 'tune.json'))
    pc = make_params(41, 37, 35, 16, 9, 9)
    geom = native_geometry(pc)
    cands = [c for c in tuning.CANDIDATES if (c[5] if len(c) > 5 else _native.MULTI_OFF) == multi]
    best, timings = tuning.autotune(geom, candidates=cands)
    assert len(timings) == len(cands) and all(ms > 0 for ms, _ in timings)
    choice = tuning.choose(geom)
    assert choice == best and choice['multi'] == multi
    eps, sig, _, _, inc = random_problem(pc, 3)
    fields = []
    for c in (choice, dict(choice, kernel=_native.FDTD_KERNEL_SPLIT)):
        sim = native_for(pc)
        tuning.apply(sim, c)
        sim.set_materials_eps_sigma(eps, sig)
        sim.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
        sim.run(9)
        fields.append({**sim.get_fields(), **sim.get_phasors()})
        sim.close()
    assert all(np.array_equal(fields[0][k], fields[1][k]) for k in fields[0])
