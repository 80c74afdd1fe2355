"""A gradient whose device has no room for the staged material block makes Ca
and Cb on the host; other errors pass."""
import numpy as np
import pytest

from fdtdsarsim_b200 import _native
from fdtdsarsim_b200.adjoint import BackscatterGradient
from helpers import make_params, random_problem


class Sim:
    def __init__(self, code):
        self.code = code

    def set_materials_eps_sigma(self, eps, sig):
        raise _native.FdtdError(self.code, 'injected')

    def set_materials(self, ca, cb):
        self.got = ca, cb


@pytest.mark.parametrize('dtype', ['float32', 'float64'])
def test_materials_without_room_for_staging(dtype):
    pc = make_params(27, 25, 23, 14, 4, 4, dtype=dtype)
    eps, sig, ca, cb, _ = random_problem(pc, 1)
    run = object.__new__(BackscatterGradient)
    run.params, run.sim = pc, Sim(_native.FDTD_ERR_NOMEM)
    run._set_materials(eps, sig)
    assert np.array_equal(run.sim.got[0], ca) and np.array_equal(run.sim.got[1], cb)
    run.sim = Sim(_native.FDTD_ERR_CUDA)
    with pytest.raises(_native.FdtdError):
        run._set_materials(eps, sig)
