"""The multi-step paths that a solve takes by default, on the grids the bench
line is measured on, against the C oracle bit for bit: the first 16 steps of
plain_16x16 and the first 200 of plain_8x8 as pairs (the latter also in odd
runs), plain_2x2 and plain_4x4 whole as resident steps."""
import numpy as np
import pytest

from fdtdsarsim_b200 import _native, tuning
from fdtdsarsim_b200.absorbers import packed_profiles
from fdtdsarsim_b200.gpu.main_sim import native_geometry
from helpers import bits_equal
from test_gpu_bench_configs import _bench, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('workload,runs,path', [
    ('plain_16x16', (16,), _native.PATH_PAIR),
    ('plain_8x8', (101, 98, 1), _native.PATH_PAIR),
    ('adjoint_4x4', None, _native.PATH_RESIDENT),
    ('plain_2x2', None, _native.PATH_RESIDENT)])
def test_default_choice_is_bit_exact(workload, runs, path):
    pc, ca, cb, inc = _bench().build_workload(workload, 'float32', sum(runs) + 1 if runs else 10 ** 6)
    geom = native_geometry(pc)
    runs = runs or (pc.geom_params.size_t,)
    orc = _oracle(pc)
    orc.run(ca, cb, inc, sum(runs))
    sim = _native.NativeSim(geom, 0)
    try:
        sim.set_absorbers(packed_profiles(pc))
        tuning.apply(sim, tuning.choose(geom, use_cache=False))
        sim.set_materials(ca, cb)
        sim.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
        taken = 0
        for n in runs:
            sim.run(n)
            taken |= sim.get_option(_native.OPT_STEP_PATH)
        sim.synchronize()
        assert taken & path
        for c in _native.FIELD_NAMES:
            assert bits_equal(sim.get_field(c), getattr(orc, c)), c
        got = sim.get_phasors()
        for name in _native.PHASOR_NAMES:
            assert bits_equal(got[name], orc.ph[name]), name
        assert np.any(orc.ex) and np.any(orc.hz)
    finally:
        sim.close()
