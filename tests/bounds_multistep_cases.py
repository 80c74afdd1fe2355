"""Cases for the bounds-checked build (run by test_gpu_bounds_multistep.py in
a child process with FDTDSARSIM_B200_LIBRARY=check): the pair and the resident
step, the resident incident run, each compared bit for bit with the oracle or
the split passes. Prints one JSON line."""
import json
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
for p in (HERE, os.path.join(ROOT, 'sar-pixel-simulator_b200'), os.path.join(ROOT, 'oracle')):
    if p not in sys.path:
        sys.path.insert(0, p)

import numpy as np  # noqa: E402

from bounds_cases import problem, same  # noqa: E402
from fdtdsarsim_b200 import _native  # noqa: E402
from fdtdsarsim_b200.absorbers import packed_profiles  # noqa: E402
from fdtdsarsim_b200.gpu.main_sim import native_geometry  # noqa: E402
from helpers import bits_equal, make_params, native_for  # noqa: E402

PAIR, RESIDENT = _native.MULTI_PAIR, _native.MULTI_RESIDENT
PATH = {PAIR: _native.PATH_PAIR, RESIDENT: _native.PATH_RESIDENT}

# nx, ny, nz, tfsf_z, nt, ntp, dtype
GRIDS = [
    (PAIR, (84, 33, 24, 12, 7, 6, 'float32')),       # one column tile, few rows, the lowest grid
    (PAIR, (149, 39, 31, 30, 6, 6, 'float32')),      # odd width, injection on the last plane
    (PAIR, (261, 45, 75, 10, 5, 4, 'float32')),      # several tiles and z chunks
    (PAIR, (93, 53, 33, 21, 6, 6, 'float64')),
    (RESIDENT, (23, 23, 23, 12, 7, 6, 'float32')),   # the smallest grid npml 10 allows
    (RESIDENT, (133, 27, 29, 14, 6, 6, 'float32')),
    (RESIDENT, (61, 67, 43, 42, 5, 4, 'float32')),   # vectors, odd width
    (RESIDENT, (33, 23, 25, 12, 6, 5, 'float64')),
    (RESIDENT, (75, 57, 41, 30, 5, 5, 'float64')),
]
# nx, ny, nz, nt, pulse, dtype
BEAMS = [(27, 25, 31, 9, 4, 'float32'), (61, 67, 43, 7, 5, 'float32'), (61, 67, 43, 6, 6, 'float64')]


def beam(case, opt, value):
    nx, ny, nz, nt, pulse, dtype = case
    pc = make_params(nx, ny, nz, nz // 2, nt, 0, dtype=dtype, cell_wl=0.05)
    src = np.random.default_rng(nx).standard_normal((2, pulse, ny, nx)).astype(dtype)
    inc = _native.NativeIncident(native_geometry(pc), pulse, 0)
    inc.set_absorbers(packed_profiles(pc))
    inc.set_option(opt, value)
    inc.set_excitation(src[0], src[1])
    inc.run()
    out = {**inc.get_planes(), **inc.get_phasors()}
    inc.close()
    return out


def main():
    out = {'library': _native.LIB_NAME, 'checked': _native.bounds_check_enabled(), 'runs': []}
    for k, (mode, case) in enumerate(GRIDS):
        pc, ca, cb, inc, orc = problem(case, 940 + k)
        sim = native_for(pc, _native.FDTD_KERNEL_FUSED, (32, 4), shell=_native.SHELL_SPLIT)
        rec = {'grid': list(case[:4]), 'dtype': case[6], 'mode': mode, 'error': None, 'bit_exact': False}
        try:
            sim.set_option(_native.OPT_MULTISTEP, mode)
            sim.set_materials(ca, cb)
            sim.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
            sim.run(case[4])
            rec['path'] = bool(sim.get_option(_native.OPT_STEP_PATH) & PATH[mode])
            sim.synchronize()
            rec['bit_exact'] = same(orc, sim)
        except _native.FdtdError as e:
            rec['error'] = f'{e.code}: {e}'
        sim.close()
        out['runs'].append(rec)
    probe = native_for(make_params(23, 23, 23, 12, 4, 4))   # its synchronize reports the beams' violations
    for case in BEAMS:
        rec = {'beam': list(case[:5]), 'dtype': case[5], 'error': None, 'bit_exact': False, 'path': True}
        try:
            a = beam(case, _native.OPT_MULTISTEP, RESIDENT)
            b = beam(case, _native.OPT_KERNEL, _native.FDTD_KERNEL_SPLIT)
            probe.synchronize()
            rec['bit_exact'] = all(bits_equal(a[k], b[k]) for k in b)
        except _native.FdtdError as e:
            rec['error'] = f'{e.code}: {e}'
        out['runs'].append(rec)
    probe.close()
    print(json.dumps(out))


if __name__ == '__main__':
    main()
