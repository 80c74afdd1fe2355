"""The multi-step paths where FDTD_OPT_MULTISTEP's own tests do not reach:
every case asserts the path that ran (FDTD_OPT_STEP_PATH), and every result is
the single step's or the oracle's, bit for bit.

The resident step holds one cell per thread up to 160000 cells and 16-byte
vectors above; the pair step needs a plain box of 32 columns and 8 rows."""
import numpy as np
import pytest

from fdtdsarsim_b200 import _native, tuning
from fdtdsarsim_b200.gpu.main_sim import native_geometry
from helpers import bits_equal, make_params, native_for, oracle_for, random_problem
from test_gpu_multistep import PAIR

pytestmark = pytest.mark.gpu

OFF, AUTO, RESIDENT = _native.MULTI_OFF, _native.MULTI_AUTO, _native.MULTI_RESIDENT
TWO = _native.MULTI_PAIR
SINGLE = _native.PATH_SINGLE
PATH = {OFF: SINGLE, RESIDENT: _native.PATH_RESIDENT, TWO: _native.PATH_PAIR}

# nx, ny, nz, npml, tfsf_z, steps run, dtype
CASES = [
    # resident with vectors: nx mod 4 (mod 2 for doubles) of every kind, partial
    # 16-cell units and rows, injection in, beside and between the z faces
    (RESIDENT, (61, 67, 43, 10, 21, 7, 'float32')),
    (RESIDENT, (62, 57, 47, 10, 9, 6, 'float32')),
    (RESIDENT, (71, 59, 41, 10, 40, 5, 'float32')),
    (RESIDENT, (80, 63, 33, 10, 23, 4, 'float32')),
    (RESIDENT, (27, 121, 53, 10, 10, 5, 'float32')),
    (RESIDENT, (93, 49, 37, 3, 2, 4, 'float32')),
    (RESIDENT, (61, 63, 43, 10, 30, 6, 'float64')),
    (RESIDENT, (74, 57, 41, 10, 11, 5, 'float64')),
    # pairs with the injection on the last plane, beside it and on the first
    (TWO, (100, 61, 37, 10, 36, 4, 'float32')),
    (TWO, (101, 44, 31, 10, 30, 5, 'float32')),
    (TWO, (124, 41, 29, 10, 0, 4, 'float32')),
    (TWO, (97, 51, 24, 10, 23, 5, 'float64')),
]


def _sim(pc, ca, cb, inc, mode, phasor_mode=0):
    sim = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), phasor_mode, shell=_native.SHELL_SPLIT)
    sim.set_option(_native.OPT_MULTISTEP, mode)
    sim.set_materials(ca, cb)
    if inc is not None:
        sim.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
    return sim


def _path(sim):
    return sim.get_option(_native.OPT_STEP_PATH)


def _same(a, b):
    for c in _native.FIELD_NAMES:
        assert bits_equal(a.get_field(c), b.get_field(c)), c
    got, want = a.get_phasors(), b.get_phasors()
    for k in want:
        assert bits_equal(got[k], want[k]), k
    assert np.any(want['ex_ph_u'])


def _ids(v):
    return 'x'.join(map(str, v)) if isinstance(v, tuple) else \
        {OFF: 'single', RESIDENT: 'resident', TWO: 'pair'}.get(v)


@pytest.mark.parametrize('mode,case', CASES, ids=_ids)
def test_path_taken_matches_oracle(mode, case):
    nx, ny, nz, npml, tfsf, nt, dtype = case
    pc = make_params(nx, ny, nz, tfsf, nt + 3, nt - 1, dtype=dtype, npml=npml)
    _, _, ca, cb, inc = random_problem(pc, nx + ny)
    orc = oracle_for(pc)
    sim = _sim(pc, ca, cb, inc, mode)
    try:
        for n in (nt, 3):
            orc.run(ca, cb, inc, n)
            sim.run(n)
            sim.synchronize()
            assert _path(sim) == PATH[mode] | (SINGLE if mode == TWO and n % 2 else 0)
            for c in _native.FIELD_NAMES:
                assert bits_equal(sim.get_field(c), getattr(orc, c)), c
            for k, name in enumerate(_native.PHASOR_NAMES):
                assert bits_equal(sim.get_phasor(k), orc.ph[name]), name
    finally:
        sim.close()


@pytest.mark.parametrize('case', [c for c in PAIR if c[0] != 70], ids=_ids)
def test_pair_cases_run_pairs(case):
    nx, ny, nz, npml, tfsf, _, dtype = case
    pc = make_params(nx, ny, nz, tfsf, 2, 2, dtype=dtype, npml=npml)
    _, _, ca, cb, inc = random_problem(pc, 1)
    sim = _sim(pc, ca, cb, inc, TWO)
    sim.run(2)
    sim.synchronize()
    assert _path(sim) == _native.PATH_PAIR
    sim.close()


@pytest.mark.parametrize('dtype', ['float32', 'float64'])
@pytest.mark.parametrize('mode', [RESIDENT, TWO], ids=_ids)
class TestOptions:
    """Options beside a multi-step path, against the single step under the
    same option."""
    nx, ny, nz = 101, 53, 35

    def _problem(self, dtype, nt=24):
        pc = make_params(self.nx, self.ny, self.nz, 17, nt, nt, dtype=dtype)
        return (pc,) + random_problem(pc, 9)[2:]

    def test_kahan_phasors(self, mode, dtype):
        pc, ca, cb, inc = self._problem(dtype)
        a = _sim(pc, ca, cb, inc, mode, _native.FDTD_PHASOR_KAHAN)
        b = _sim(pc, ca, cb, inc, OFF, _native.FDTD_PHASOR_KAHAN)
        for n in (7, 12, 5):
            a.run(n)
            b.run(n)
        assert _path(a) & PATH[mode] and _path(b) == SINGLE
        _same(a, b)
        a.close()
        b.close()

    @pytest.mark.parametrize('chunk', [1, 2, 3, 4, 5])
    def test_graph_chunks(self, mode, dtype, chunk):
        pc, ca, cb, inc = self._problem(dtype)
        a, b = _sim(pc, ca, cb, inc, mode), _sim(pc, ca, cb, inc, OFF)
        a.set_option(_native.OPT_GRAPH_CHUNK, chunk)
        for n in (11, 1, 12):
            a.run(n)
            b.run(n)
        assert bool(_path(a) & PATH[mode]) == (chunk > 1)
        _same(a, b)
        a.close()
        b.close()

    def test_streamed_planes(self, mode, dtype):
        pc, ca, cb, inc = self._problem(dtype)
        a, b = _sim(pc, ca, cb, None, mode), _sim(pc, ca, cb, inc, OFF)
        for n in (21, 3):
            a.run_streamed(n, inc['ex'], inc['ey'], inc['hx'], inc['hy'])
            assert _path(a) & PATH[mode]
            b.run(n)
        _same(a, b)
        a.close()
        b.close()

    def test_non_finite_check_takes_single_steps(self, mode, dtype):
        pc, ca, cb, inc = self._problem(dtype)
        a, b = _sim(pc, ca, cb, inc, mode), _sim(pc, ca, cb, inc, OFF)
        a.set_option(_native.OPT_CHECK_EVERY, 4)
        a.run(9)
        a.synchronize()
        assert _path(a) == SINGLE
        a.set_option(_native.OPT_CHECK_EVERY, 0)
        a.run(8)
        assert _path(a) == PATH[mode]
        b.run(17)
        _same(a, b)
        a.close()
        b.close()

    def test_gradient(self, mode, dtype):
        """The forward accumulates the upper plane's phasors only."""
        pc, ca, cb, inc = self._problem(dtype)
        out = []
        rng = np.random.default_rng(4)
        shape = (2, 4, self.ny - 20, self.nx - 20)
        re, im = rng.standard_normal(shape)
        for m in (mode, OFF):
            sim = _sim(pc, ca, cb, inc, m)
            sim.grad_forward(7)
            assert _path(sim) & PATH[m]
            ph = [sim.get_phasor(k) for k in range(4, 8)]
            out.append(ph + list(sim.grad_backward(re, im, self.nz)))
            sim.close()
        assert all(bits_equal(x, y) and np.any(y) for x, y in zip(*out))

    def test_batch_streams(self, mode, dtype):
        """Members side by side take pairs, but nothing resident."""
        sims, refs = [], []
        for k, (nx, ny) in enumerate([(101, 53), (97, 41), (85, 45)]):
            pc = make_params(nx, ny, self.nz, 17, 20, 20, dtype=dtype)
            _, _, ca, cb, inc = random_problem(pc, 20 + k)
            sims.append(_sim(pc, ca, cb, inc, mode))
            refs.append(_sim(pc, ca, cb, inc, OFF))
        batch = _native.Batch(sims, streams=True)
        for n in (9, 11):
            batch.run(n)
        batch.synchronize()
        want = SINGLE if mode == RESIDENT else _native.PATH_PAIR | SINGLE
        for a, b in zip(sims, refs):
            assert _path(a) == want
            b.run(20)
            _same(a, b)
        batch.close()
        for s in sims + refs:
            s.close()


def test_auto_takes_each_path():
    """FDTD_MULTI_AUTO's rule by bytes, cells and width, one grid of each."""
    for (nx, ny, nz, dtype), want in (((55, 53, 41, 'float32'), _native.PATH_RESIDENT),
                                      ((200, 220, 100, 'float32'), _native.PATH_PAIR),
                                      ((100, 220, 200, 'float32'), SINGLE),
                                      ((150, 120, 100, 'float64'), _native.PATH_PAIR)):
        pc = make_params(nx, ny, nz, 20, 4, 0, dtype=dtype)
        shape = (nz, ny, nx)
        sim = _sim(pc, np.ones(shape, dtype), np.ones(shape, dtype), None, AUTO)
        sim.run(4)
        sim.synchronize()
        assert _path(sim) == want, (nx, ny, nz, dtype)
        with pytest.raises(_native.FdtdError):
            sim.set_option(_native.OPT_STEP_PATH, 1)
        sim.close()


def test_a_tuned_pair_choice_runs_pairs(tmp_path, monkeypatch):
    """On a grid whose plain box is wide enough (41 columns are not)."""
    monkeypatch.setenv('FDTDSARSIM_B200_TUNING', str(tmp_path / 'tune.json'))
    pc = make_params(101, 53, 35, 16, 9, 9)
    geom = native_geometry(pc)
    best, _ = tuning.autotune(geom, candidates=[c for c in tuning.CANDIDATES if c[5:] == (TWO,)])
    assert tuning.choose(geom) == best and best['multi'] == TWO
    _, _, ca, cb, inc = random_problem(pc, 3)
    a, b = _sim(pc, ca, cb, inc, OFF), _sim(pc, ca, cb, inc, OFF)
    tuning.apply(a, best)
    for s in (a, b):
        s.run(9)
    assert _path(a) == _native.PATH_PAIR | SINGLE
    _same(a, b)
    a.close()
    b.close()
