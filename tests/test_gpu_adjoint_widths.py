"""The adjoint sweep at widths where its two-cell vectors straddle the x
faces and the domain edge (nx is odd; the narrowest grids the CPML
allows), against the float64 numpy adjoint. The device sums the same products
in another order: relative 1e-9 as float64 leaves after 24 steps."""
import numpy as np
import pytest

from adjoint_ref import AdjointRef
from fdtdsarsim_b200 import synthetic
from fdtdsarsim_b200.absorbers import cpml_profiles
from fdtdsarsim_b200.adjoint import BackscatterGradient, power_and_phasor_grad
from fdtdsarsim_b200.materials import MaterialModel, compute_material_arrays
from helpers import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nx,ny', [(23, 25), (25, 23), (27, 23), (33, 25), (35, 23), (65, 23)])
def test_adjoint_matches_numpy_adjoint_at_any_width(nx, ny):
    nt = 24
    pc = make_params(nx, ny, 27, 14, nt, 30, dtype='float64')
    pc.inc_beam_params.polarization = 'HH'
    g = pc.geom_params
    rng = np.random.default_rng(nx)
    shape = (g.size_z_material, g.size_y, g.size_x)
    eps, sig = rng.uniform(2.0, 12.0, size=shape), rng.uniform(0.0, 0.1, size=shape)
    inc = synthetic.plane_wave_incident(pc, g.size_t_inc, 'float64')
    ref = AdjointRef(g.size_x, g.size_y, g.size_z, g.size_pml, g.tfsf_z, g.cell_size, g.timestep,
                     pc.inc_beam_params.frequency, cpml_profiles(pc), theta_deg=-20.0, phi_deg=0.0)
    ca, cb = compute_material_arrays(pc, MaterialModel(eps, sig, g.cell_size))
    _, gca_ref, gcb_ref = ref.grad(ca, cb, inc, nt)
    run = BackscatterGradient(pc, inc, checkpoint_every=5)
    run._set_materials(eps, sig)
    run.sim.grad_forward(5)
    _, g_re, g_im = power_and_phasor_grad(run._upper_phasors(), run.a, run.b, run.sign)
    gca, gcb = run.sim.grad_backward(g_re, g_im, g.size_z)
    run.close()
    for got, want in ((gca, gca_ref), (gcb, gcb_ref)):
        assert np.linalg.norm(got - want) <= 1e-9 * np.linalg.norm(want)
