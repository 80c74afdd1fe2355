"""The bounds-checked build (libfdtd_b200_check.so) on the multi-step paths:
pairs, resident steps and the resident incident run on tiny and ragged grids,
every global access of their kernels but the pair step's plane copies (whose
tensor maps bound them) checked against the library's live allocations. No
violation, and the oracle's bits. Runs in a child process, which loads the
checked library instead of the normal one."""
import json
import os
import subprocess
import sys

import pytest

from test_gpu_bounds import CHECK_LIB, HERE

pytestmark = pytest.mark.gpu


def test_checked_build_of_the_multi_step_paths():
    assert os.path.exists(CHECK_LIB), 'build it: python sar-pixel-simulator_b200/build.py --bounds-check'
    env = dict(os.environ, FDTDSARSIM_B200_LIBRARY='check')
    out = subprocess.run([sys.executable, os.path.join(HERE, 'bounds_multistep_cases.py')], env=env,
                         capture_output=True, text=True, timeout=900)
    assert out.returncode == 0, out.stderr[-3000:]
    res = json.loads(out.stdout.strip().splitlines()[-1])
    assert res['library'] == 'libfdtd_b200_check.so' and res['checked'] is True
    bad = [r for r in res['runs'] if r['error'] is not None or not r['bit_exact'] or not r['path']]
    assert not bad, bad
    assert len(res['runs']) == 12
