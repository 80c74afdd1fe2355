"""The gradient with respect to eps_r and sigma made on the device
(fdtd_grad_backward_eps_sigma) against the host's closed form applied to
dJ/dCa, dJ/dCb: the same float64 operations in the same order, so equal."""
import numpy as np
import pytest

from fdtdsarsim_b200.adjoint import ca_cb_partials
from helpers import make_params, native_for, random_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype,nx', [('float32', 33), ('float64', 37)])
def test_device_material_gradient_equals_host_closed_form(dtype, nx):
    pc = make_params(nx, 31, 29, 15, 12, 9, dtype=dtype, nz_mat=13)
    eps, sig, _, _, inc = random_problem(pc, nx)
    g = pc.geom_params
    sim = native_for(pc)
    try:
        sim.set_materials_eps_sigma(eps, sig)
        sim.set_incident(inc['ex'], inc['ey'], inc['hx'], inc['hy'])
        rng = np.random.default_rng(2)
        re, im = rng.standard_normal((2, 4, sim.ny_ph, sim.nx_ph))
        sim.grad_forward(5)
        gca, gcb = sim.grad_backward(re, im, 13)
        sim.grad_forward(5)
        ge, gs = sim.grad_backward_eps_sigma(re, im, eps, sig)
    finally:
        sim.close()
    a, b, c, d = ca_cb_partials(eps, sig, g.timestep, g.cell_size)
    assert np.array_equal(ge, gca * a + gcb * c)
    assert np.array_equal(gs, gca * b + gcb * d)
    assert np.any(ge) and np.any(gs)
