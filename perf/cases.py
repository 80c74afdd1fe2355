"""The work this framework is used for, as cases that can be timed and compared.

Every case goes through the entry points that a user's program calls:
MainSimGpu (a model solve), _native.Batch (a sweep over models of uneven
sizes), BackscatterGradient (forward and backward), IncidentSimGpu (the beam
of a new geometry) and FarFieldTransform (the post-processing of a solve).
Sizes are grids of cells (z, y, x) with a 10-cell absorber; the named ones are
the repository's own configurations. ``exact`` is the same computation in 64
bits with plain torch.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                'sar-pixel-simulator_b200'))

C0 = 299792458.0
MU0 = 1.25663706127e-06
E0 = 8.8541878188e-12          # the update's constant
E0_MATERIAL = 8.8541878128e-12   # the material code's constant
ETA0 = 376.730313668
FREQ = 5.4e9
LAM = C0 / FREQ
NPML = 10
RADIUS = 2.0e3
DEV = 'cuda'
PLANES = ('ex_ph_d', 'ey_ph_d', 'hx_ph_d', 'hy_ph_d', 'ex_ph_u', 'ey_ph_u', 'hx_ph_u', 'hy_ph_u',
          'ey_ph_l', 'ez_ph_l', 'hy_ph_l', 'hz_ph_l', 'ey_ph_r', 'ez_ph_r', 'hy_ph_r', 'hz_ph_r',
          'ex_ph_f', 'ez_ph_f', 'hx_ph_f', 'hz_ph_f', 'ex_ph_b', 'ez_ph_b', 'hx_ph_b', 'hz_ph_b')


def _grid(kind, nz, nzm, ny, nx, nt, cell, dtype='float32', pol='HH', theta=20.0, **more):
    return dict(kind=kind, nz=nz, nzm=nzm, ny=ny, nx=nx, nt=nt, cell=cell, dtype=dtype, pol=pol,
                theta=theta, **more)


def listed():
    return [
        # one model solved as run_experiment solves it (material block up, all
        # steps, phasors back), 2 x 2 wavelengths: the smallest geometry in use
        dict(_grid('solve', 31, 9, 39, 39, 720, 0.05), name='solve_2x2'),
        # the same for the 4 x 4 wavelength geometry
        dict(_grid('solve', 55, 33, 133, 133, 1200, 0.03), name='solve_4x4'),
        # the same in double precision, on an uneven grid
        dict(_grid('solve', 47, 28, 87, 107, 600, 0.035, dtype='float64', pol='VV'), name='solve_f64'),
        # the time loop of an 8 x 8 wavelength model (material resident)
        dict(_grid('steps', 101, 71, 381, 381, 286, 0.021), name='steps_8x8'),
        # the time loop of the full-size 16 x 16 wavelength model, VV
        dict(_grid('steps', 203, 142, 761, 761, 120, 0.021, pol='VV'), name='steps_16x16'),
        # an accuracy run: 8 x 8 wavelengths in double precision
        dict(_grid('steps', 101, 71, 381, 381, 100, 0.021, dtype='float64'), name='steps_8x8_f64'),
        # a long narrow footprint (ragged: odd sizes, a short y side)
        dict(_grid('steps', 137, 96, 123, 479, 300, 0.025), name='steps_strip'),
        # a sweep over models of uneven extents, one launch per pass
        dict(kind='batch', members=32, layout=7, nt=100, cell=0.03, dtype='float32', streams=False,
             name='batch_32'),
        # a smaller sweep as run_experiment_batched runs it
        dict(kind='batch', members=10, layout=3, nt=150, cell=0.03, dtype='float32', streams=True,
             name='batch_streams_10'),
        # backscatter power and its gradient for every cell: forward and backward
        dict(_grid('gradient', 55, 33, 133, 133, 800, 0.03, every=64), name='gradient_4x4'),
        # the incident beam of a new 4 x 4 wavelength geometry
        dict(kind='beam', ny=133, nx=133, nt=480, npulse=400, cell=0.03, dtype='float32', pol='HH',
             width=4.0, name='beam_4x4'),
        # the far field of a full-size solve over the angles that post-processing takes
        dict(kind='farfield', ny=741, nx=741, nz=183, cell=0.021, dtype='float32', thetas=161, phis=1,
             name='farfield_16x16'),
    ]


def _odd(v):
    return int(v) // 2 * 2 + 1


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(('solve', 'solve', 'steps', 'steps', 'steps', 'batch', 'gradient', 'beam', 'farfield'))
    dtype = rng.choice(('float32', 'float32', 'float64'))
    if kind == 'farfield':
        n = _odd(_log(rng, 19, 741))
        return dict(kind=kind, ny=n, nx=_odd(_log(rng, 19, 741)), nz=_odd(_log(rng, 11, 183)),
                    cell=round(rng.uniform(0.02, 0.05), 4), dtype=dtype, thetas=rng.choice((1, 37, 161)),
                    phis=1)
    if kind == 'beam':
        ny, nx = _odd(_log(rng, 31, 160)), _odd(_log(rng, 31, 160))
        nt = rng.randint(120, 480)
        return dict(kind=kind, ny=ny, nx=nx, nt=nt, npulse=int(nt / 1.2), cell=round(rng.uniform(0.03, 0.06), 4),
                    dtype=dtype, pol=rng.choice(('HH', 'VV')), width=4.0)
    if kind == 'batch':
        return dict(kind=kind, members=rng.randint(2, 24), layout=rng.randint(0, 10 ** 6), nt=rng.randint(40, 120),
                    cell=0.03, dtype=dtype, streams=rng.random() < 0.5)
    # a grid of log-uniform volume, its sides within a factor of about four
    top = {'solve': 2.5e6, 'steps': 1.1e8, 'gradient': 1.0e6}[kind] / (2 if dtype == 'float64' else 1)
    low = {'solve': 4.0e4, 'steps': 1.0e6, 'gradient': 4.0e4}[kind]
    vol = _log(rng, low, top)
    a, b = _log(rng, 1.0, 4.0), _log(rng, 0.6, 1.6)
    nz = max(31, (vol / (a * a * b)) ** (1.0 / 3.0))
    ny = max(33, math.sqrt(vol / nz / b))
    nx = max(33, vol / nz / ny)
    nz, ny, nx = _odd(nz), _odd(ny), _odd(nx)
    cell = round(_log(rng, 0.021, 0.05), 4)
    while nz - 2 * NPML - int(0.3 / cell) < 4:   # the injection plane stays below the upper planes
        nz += 2
    nzm = max(2, min(int(rng.uniform(0.3, 0.7) * nz), nz - NPML - 3 - int(0.3 / cell)))
    cells = nz * ny * nx * (2 if dtype == 'float64' else 1)
    nt = int({'solve': min(1200, 1.2e9 / cells), 'steps': max(24, min(600, 1.2e10 / cells)),
              'gradient': min(700, 7e8 / cells)}[kind])
    more = {'every': rng.choice((16, 40, 64))} if kind == 'gradient' else {}
    return _grid(kind, nz, nzm, ny, nx, nt, cell, dtype=dtype, pol=rng.choice(('HH', 'VV')),
                 theta=float(rng.randint(0, 45)), **more)


# ---------------------------------------------------------------------------
# inputs, made from the seed alone
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _torch_dtype(case):
    return torch.float32 if case['dtype'] == 'float32' else torch.float64


def _surface(ny, nx, gen):
    """A rough surface (ny, nx) in cells, a few cells rms."""
    k = min(9, ny // 4, nx // 4)
    n = torch.randn((1, 1, k, k), generator=gen, device=DEV, dtype=torch.float64)
    return 1.5 * torch.nn.functional.interpolate(n, size=(ny, nx), mode='bicubic', align_corners=True)[0, 0]


def _material(case, seed):
    """eps_r, sigma of the block (nzm, ny, nx): scatterers (ice, wood) in air
    over rough soil with a spread of permittivities per cell."""
    gen = _gen(seed)
    nzm, ny, nx = case['nzm'], case['ny'], case['nx']
    dt = _torch_dtype(case)
    z = torch.arange(nzm, device=DEV, dtype=torch.float64)[:, None, None]
    soil = z <= nzm * 0.5 + _surface(ny, nx, gen)[None]
    noise = torch.randn((nzm, ny, nx), generator=gen, device=DEV, dtype=torch.float32)
    eps = torch.where(soil, 8.0 * torch.exp(0.05 * noise), torch.ones_like(noise))
    sig = torch.where(soil, torch.full_like(noise, 0.02), torch.zeros_like(noise))
    blobs = torch.rand((1, 1, max(1, nzm // 3), max(1, ny // 3), max(1, nx // 3)), generator=gen, device=DEV)
    blobs = torch.nn.functional.interpolate(blobs, size=(nzm, ny, nx), mode='nearest')[0, 0]
    ice = ~soil & (blobs > 0.8)
    eps = torch.where(ice, torch.full_like(eps, 3.15), eps)
    return eps.to(dt), sig.to(dt)


def _incident(case, seed):
    """Incident planes (nt, ny, nx) of a tapered plane wave that ramps up over
    three periods; its tangential components vanish on the plane's edges, as
    the package's own beam does."""
    r = random.Random(int(seed) * 31 + 5)
    amp, shift = r.uniform(0.7, 1.4), r.uniform(0.0, 1.0)
    nt, ny, nx = case['nt'], case['ny'], case['nx']
    dx = LAM * case['cell']
    dt = dx * 0.5 / C0
    th = math.radians(case['theta'])
    f64 = dict(device=DEV, dtype=torch.float64)
    x = (torch.arange(nx, **f64) - (nx - 1) / 2.0) * dx
    y = (torch.arange(ny, **f64) - (ny - 1) / 2.0) * dx
    tau = torch.arange(nt, **f64)[:, None] * dt - x[None, :] * math.sin(th) / C0
    ramp = 0.5 * (1.0 - torch.cos(math.pi * torch.clamp(tau * FREQ / 3.0 + 0.2 * shift, 0.0, 1.0)))
    carrier = amp * torch.sin(2 * math.pi * (FREQ * tau + shift)) * ramp
    taper = torch.exp(-(y[:, None] / (0.4 * ny * dx)) ** 2 - (x[None, :] / (0.4 * nx * dx)) ** 2)
    e = (carrier[:, None, :] * taper[None]).to(_torch_dtype(case))
    zero = torch.zeros_like(e)
    if case['pol'] == 'VV':
        out = {'ex': e * math.cos(th), 'ey': zero, 'hx': zero.clone(), 'hy': e / ETA0}
    else:
        out = {'ex': zero, 'ey': e, 'hx': -e * math.cos(th) / ETA0, 'hy': zero.clone()}
    for k in ('ey', 'hx'):
        out[k][:, :, 0] = 0
        out[k][:, :, -1] = 0
    for k in ('ex', 'hy'):
        out[k][:, 0, :] = 0
        out[k][:, -1, :] = 0
    return out


def _tfsf(case):
    return case['nzm'] + int(0.3 / case['cell'])


def _params(case):
    """The ParameterCollection of a grid case."""
    from fdtdsarsim_b200.parameters import ParameterCollection
    pc = ParameterCollection()
    pc.processing_params.processing_type = 'gpu'
    pc.processing_params.datatype = case['dtype']
    b = pc.inc_beam_params
    b.frequency, b.polarization, b.theta_angle, b.phi_angle = FREQ, case['pol'], case['theta'], 0.0
    b.duration, b.illumination_width = 10.0, case['nx'] * case['cell']
    g = pc.geom_params
    g.courant, g.size_pml = 0.5, NPML
    g.cell_size = LAM * case['cell']
    g.timestep = g.cell_size * 0.5 / C0
    g.size_x, g.size_y, g.size_z, g.size_z_material = case['nx'], case['ny'], case['nz'], case['nzm']
    g.tfsf_z = _tfsf(case)
    g.size_t = g.size_t_inc = case['nt']
    g.size_t_pulse = int(case['nt'] / 1.2)
    g.simulation_duration = case['nt'] * g.timestep * FREQ
    return pc


def _members(case):
    """The members of a sweep: x-y 67 to 267 cells, z 43 to 95."""
    r = random.Random(case['layout'])
    out = []
    for k in range(case['members']):
        ny, nx = _odd(r.uniform(67, 267)), _odd(r.uniform(67, 267))
        nz = _odd(r.uniform(43, 95))
        out.append(_grid('steps', nz, int(0.6 * nz) - 3, ny, nx, case['nt'], case['cell'], dtype=case['dtype'],
                         pol='HH' if k % 2 else 'VV'))
    return out


def _host(t):
    return t.cpu().numpy()


def _simulator(case, seed):
    """A MainSimGpu with its incident beam, its model resident."""
    from fdtdsarsim_b200.gpu.main_sim import MainSimGpu
    sim = MainSimGpu(_params(case))
    inc = _incident(case, seed)
    sim.load_incident(*[_host(inc[k]) for k in ('ex', 'ey', 'hx', 'hy')])
    del inc
    eps, sig = _material(case, seed)
    return sim, _host(eps), _host(sig)


def _pinned(sim):
    """A page-locked buffer for the 24 phasor planes, as the package's benchmark keeps one."""
    cdt = torch.complex64 if sim.cdtype == np.complex64 else torch.complex128
    return torch.empty(sim.phasors_size(), dtype=cdt).pin_memory().numpy()


def _pulse(case, seed):
    r = random.Random(int(seed) * 13 + 1)
    return dict(theta=r.uniform(5.0, 40.0), phi=r.uniform(-20.0, 20.0), duration=r.uniform(8.0, 10.0))


def _beam_params(case, seed):
    p = _params(dict(case, nz=31, nzm=9, theta=0.0))
    q = _pulse(case, seed)
    b = p.inc_beam_params
    b.theta_angle, b.phi_angle, b.duration, b.illumination_width = q['theta'], q['phi'], q['duration'], case['width']
    p.geom_params.size_t_pulse = case['npulse']
    return p


def _plane_phasors(case, seed):
    """Upper phasor planes ex, ey, hx, hy (ny, nx): a few plane waves and speckle."""
    gen = _gen(seed)
    ny, nx = case['ny'], case['nx']
    f64 = dict(device=DEV, dtype=torch.float64)
    k = 2 * math.pi * case['cell']
    x, y = torch.arange(nx, **f64) * k, torch.arange(ny, **f64) * k
    out = {}
    for name in ('ex_ph_u', 'ey_ph_u', 'hx_ph_u', 'hy_ph_u'):
        p = 0.1 * torch.complex(torch.randn((ny, nx), generator=gen, **f64), torch.randn((ny, nx), generator=gen, **f64))
        for a, b, c in torch.rand((4, 3), generator=gen, **f64).tolist():
            arg = (2 * a - 1) * x[None, :] + (b - 0.5) * y[:, None] + 6.0 * c
            p += torch.complex(torch.cos(arg), torch.sin(arg))
        p *= torch.exp(-((x - x.mean())[None, :] / (0.5 * k * nx)) ** 2 - ((y - y.mean())[:, None] / (0.5 * k * ny)) ** 2)
        if name[0] == 'h':
            p /= ETA0
        out[name] = p.to(torch.complex64 if case['dtype'] == 'float32' else torch.complex128)
    return out


def _angles(case):
    thetas = np.linspace(-80.0, 80.0, case['thetas']) if case['thetas'] > 1 else np.array([-20.0])
    return thetas, np.linspace(0.0, 30.0, case['phis'])


def prepare(case, seed):
    kind = case['kind']
    if kind in ('solve', 'steps'):
        sim, eps, sig = _simulator(case, seed)
        if kind == 'solve':
            return dict(kind=kind, sim=sim, eps=eps, sig=sig)
        sim.native.set_materials_eps_sigma(eps, sig)
        return dict(kind=kind, sim=sim, nt=case['nt'], out=_pinned(sim.native))
    if kind == 'batch':
        from fdtdsarsim_b200 import _native
        sims = []
        for k, m in enumerate(_members(case)):
            sim, eps, sig = _simulator(m, seed * 100 + k)
            sim.native.set_materials_eps_sigma(eps, sig)
            sims.append(sim)
        batch = _native.Batch([s.native for s in sims], streams=case['streams'])
        return dict(kind=kind, sims=sims, batch=batch, nt=case['nt'], outs=[_pinned(s.native) for s in sims])
    if kind == 'gradient':
        from fdtdsarsim_b200.adjoint import BackscatterGradient
        inc = {k: _host(v) for k, v in _incident(case, seed).items()}
        eps, sig = _material(case, seed)
        return dict(kind=kind, runner=BackscatterGradient(_params(case), inc, checkpoint_every=case['every']),
                    eps=_host(eps), sig=_host(sig))
    if kind == 'beam':
        from fdtdsarsim_b200.incident import IncidentSimGpu, create_pulse
        p = _beam_params(case, seed)
        _, _, fft, freqs = create_pulse(p)
        return dict(kind=kind, sim=IncidentSimGpu(p), fft=fft, freqs=freqs)
    from fdtdsarsim_b200.near2far import FarFieldTransform
    planes = {k: _host(v) for k, v in _plane_phasors(case, seed).items()}
    return dict(kind=kind, transform=FarFieldTransform(), planes=planes, angles=_angles(case), case=case)


def run(state):
    kind = state['kind']
    if kind == 'solve':
        state['sim'].simulate_eps_sigma(state['eps'], state['sig'])
        return state['sim'].phasors()
    if kind == 'steps':
        sim = state['sim']
        sim.reset()
        sim.step(state['nt'])
        return sim.native.get_phasors(state['out'])
    if kind == 'batch':
        for s in state['sims']:
            s.reset()
        state['batch'].run(state['nt'])
        for s, out in zip(state['sims'], state['outs']):
            s.native.get_phasors(out)
        return state['outs']
    if kind == 'gradient':
        return state['runner'].value_and_grad(state['eps'], state['sig'])
    if kind == 'beam':
        sim = state['sim']
        sim.make_excitation(state['fft'], state['freqs'])
        sim.run()
        return dict(planes=sim.planes(), phasors=sim.phasors())
    c = state['case']
    return state['transform'](state['planes'], c['nx'], c['ny'], c['nz'], LAM * c['cell'], RADIUS, *state['angles'], FREQ)


def work(case):
    """Bytes and operations of one pass. A time step reads and writes the six
    field components and reads the two coefficients of every cell (14 values,
    33 operations); the absorber's, incident and phasor planes are small
    beside that and left out."""
    size = 4 if case['dtype'] == 'float32' else 8
    kind = case['kind']
    if kind == 'farfield':
        n, a = case['nx'] * case['ny'], case['thetas'] * case['phis']
        return dict(bytes=8 * size * n + 64 * a, flops=32 * n * a)   # four complex sums per direction
    if kind == 'batch':
        steps = sum(m['nz'] * m['ny'] * m['nx'] for m in _members(case)) * case['nt']
        return dict(bytes=14 * size * steps, flops=33 * steps)
    if kind == 'beam':
        n = case['nx'] * case['ny']
        steps = int(3.0 / case['cell']) * n * case['nt']
        return dict(bytes=12 * size * steps + 4 * size * n * case['nt'], flops=33 * steps)
    steps = case['nz'] * case['ny'] * case['nx'] * case['nt']
    if kind == 'gradient':
        # forward, and backward: adjoint fields in and out, forward fields and
        # coefficients in, two double gradients in and out (material planes)
        back = 20 * size + 32 * case['nzm'] / case['nz']
        return dict(bytes=(14 * size + back) * steps, flops=33 * steps * 2.5)
    return dict(bytes=14 * size * steps, flops=33 * steps)


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _profiles(dx, dt):
    """CPML profiles of the low and high faces (Taflove ch. 7.9): {'e': (b, c)
    low, high, 'h': ...}, kappa 1, sigma graded cubically, alpha linearly."""
    n = torch.arange(NPML, dtype=torch.float64, device=DEV)
    dec, span = NPML - 1 - n, NPML - 1.0
    smax, amax, tiny = 0.8 * 4 / (ETA0 * dx), 0.2, 1e-30

    def bc(sig, alp):
        b = torch.exp(-(sig + alp) * dt / E0_MATERIAL)
        return b, (sig + tiny) * (b - 1) / (sig + alp + tiny)

    def s3(v):
        return smax * (v / span) ** 3

    return {('e', 0): bc(s3(dec), amax * n / span), ('h', 0): bc(s3(dec - 0.5), amax * (n + 0.5) / span),
            ('e', 1): bc(s3(n), amax * dec / span),
            ('h', 1): bc(s3(n + 0.5), torch.clamp(amax * (dec - 0.5) / span, min=0.0))}


class _Yee64:
    """The Yee grid of a solve in float64: H and E half steps with the CPML of
    the six faces; ``functional`` keeps autograd able to look back."""

    def __init__(self, nz, ny, nx, dx, ca, cb, functional=False):
        self.n, self.dx, self.ca, self.cb, self.fn = (nz, ny, nx), dx, ca, cb, functional
        self.dt = dx * 0.5 / C0
        self.prof = _profiles(dx, self.dt)
        f64 = dict(dtype=torch.float64, device=DEV)
        self.f = {c: torch.zeros(self.n, **f64) for c in ('ex', 'ey', 'ez', 'hx', 'hy', 'hz')}
        self.psi = {}
        for kind in 'eh':
            for ax in range(3):
                shape = [v - 1 for v in self.n]
                shape[ax] = NPML - 1
                for side in (0, 1):
                    for k in (0, 1):
                        self.psi[kind, ax, side, k] = torch.zeros(shape, **f64)

    def state(self):
        return list(self.f.values()) + list(self.psi.values())

    def load(self, tensors):
        tensors = list(tensors)
        self.f = dict(zip(self.f, tensors[:6]))
        self.psi = dict(zip(self.psi, tensors[6:]))

    def _cpml(self, kind, target, ax, k, diff, scale):
        """target += scale * psi on both faces of axis ax, psi driven by diff
        (the difference along ax on the box, cells 0 .. n - 2 of each axis)."""
        m, n = NPML, self.n[ax]
        for side in (0, 1):
            low = (1 if kind == 'e' else 0) if side == 0 else n - m
            q0 = 1 if (kind, side) == ('e', 0) else 0
            b, c = (p[q0:q0 + m - 1].reshape([-1 if a == ax else 1 for a in range(3)]) for p in self.prof[kind, side])
            at = [slice(0, v - 1) for v in self.n]
            at[ax] = slice(low, low + m - 1)
            at = tuple(at)
            psi = b * self.psi[kind, ax, side, k] + c * diff.narrow(ax, low, m - 1) / self.dx
            self.psi[kind, ax, side, k] = psi
            target[at] += (scale[at] if torch.is_tensor(scale) else scale) * psi

    def h_half(self):
        f = {c: v.clone() if self.fn and c[0] == 'h' else v for c, v in self.f.items()}
        ex, ey, ez, hx, hy, hz = f.values()
        db, dtm0 = self.dt / (MU0 * self.dx), self.dt / MU0
        lo = (slice(0, -1),) * 3
        up = [tuple(slice(1, None) if a == ax else slice(0, -1) for a in range(3)) for ax in range(3)]
        dey_z, dez_y, dex_z = ey[up[0]] - ey[lo], ez[up[1]] - ez[lo], ex[up[0]] - ex[lo]
        dez_x, dex_y, dey_x = ez[up[2]] - ez[lo], ex[up[1]] - ex[lo], ey[up[2]] - ey[lo]
        hx[:-1, :-1, 1:-1] -= db * (dez_y - dey_z)[:, :, 1:]
        hy[:-1, 1:-1, :-1] -= db * (dex_z - dez_x)[:, 1:, :]
        hz[1:-1, :-1, :-1] -= db * (dey_x - dex_y)[1:]
        self._cpml('h', hy, 0, 0, dex_z, -dtm0)
        self._cpml('h', hx, 0, 1, dey_z, dtm0)
        self._cpml('h', hz, 2, 0, dey_x, -dtm0)
        self._cpml('h', hy, 2, 1, dez_x, dtm0)
        self._cpml('h', hx, 1, 0, dez_y, -dtm0)
        self._cpml('h', hz, 1, 1, dex_y, dtm0)
        self.f = f

    def e_half(self):
        old = self.f
        f = {c: v.clone() if self.fn and c[0] == 'e' else v for c, v in old.items()}
        ex, ey, ez, hx, hy, hz = f.values()
        ca, cb = self.ca, self.cb
        cbdx = cb * self.dx

        def back(h, ax):   # h - h one cell lower, on the box; the first cell is never read
            d = h[:-1, :-1, :-1]
            return d - torch.roll(d, 1, ax)

        dhz_y, dhy_z, dhx_z = back(hz, 1), back(hy, 0), back(hx, 0)
        dhz_x, dhx_y, dhy_x = back(hz, 2), back(hx, 1), back(hy, 2)
        r = (slice(1, -1), slice(1, -1), slice(0, -1))
        ex[r] = old['ex'][r] * ca[r] + cb[r] * (dhz_y - dhy_z)[1:, 1:, :]
        r = (slice(1, -1), slice(0, -1), slice(1, -1))
        ey[r] = old['ey'][r] * ca[r] + cb[r] * (dhx_z - dhz_x)[1:, :, 1:]
        r = (slice(0, -1), slice(1, -1), slice(1, -1))
        ez[r] = old['ez'][r] * ca[r] + cb[r] * (dhy_x - dhx_y)[:, 1:, 1:]
        self._cpml('e', ey, 0, 0, dhx_z, cbdx)
        self._cpml('e', ex, 0, 1, dhy_z, -cbdx)
        self._cpml('e', ez, 2, 0, dhy_x, cbdx)
        self._cpml('e', ey, 2, 1, dhz_x, -cbdx)
        self._cpml('e', ex, 1, 0, dhz_y, cbdx)
        self._cpml('e', ez, 1, 1, dhx_y, -cbdx)
        self.f = f

    def step(self, inc, t, plane):
        """One time step with the incident planes added on z = plane."""
        db, de = self.dt / (MU0 * self.dx), self.dt / (E0 * self.dx)
        self.h_half()
        self.f['hx'][plane] += db * inc['ey'][t]
        self.f['hy'][plane] -= db * inc['ex'][t]
        self.e_half()
        self.f['ey'][plane] += de * inc['hx'][t]
        self.f['ex'][plane] -= de * inc['hy'][t]

    def phase(self, t):
        return complex(math.cos(-2 * math.pi * FREQ * t * self.dt), math.sin(-2 * math.pi * FREQ * t * self.dt))

    def plane_means(self, group):
        """Field means of a phasor plane group (d, u, l, r, f, b): E, E, H, H
        at the plane's cells (first row and column left out)."""
        m = NPML
        ax = {'d': 0, 'u': 0, 'l': 2, 'r': 2, 'f': 1, 'b': 1}[group]
        p = m + 1 if group in 'dlf' else self.n[ax] - m - 1

        def at(c, *back):   # the component on the plane, one cell lower along the axes in back
            s = [slice(m + 1 - (a in back), v - m - (a in back)) for a, v in enumerate(self.n)]
            s[ax] = p - (ax in back)
            return self.f[c][tuple(s)]

        def mean(c, *axes):
            if len(axes) == 1:
                return 0.5 * (at(c) + at(c, axes[0]))
            return 0.25 * (at(c) + at(c, axes[0]) + at(c, axes[1]) + at(c, *axes))

        if ax == 0:
            return mean('ex', 2), mean('ey', 1), mean('hx', 1, 0), mean('hy', 2, 0)
        if ax == 2:
            return mean('ey', 1), mean('ez', 0), mean('hy', 2, 0), mean('hz', 2, 1)
        return mean('ex', 2), mean('ez', 0), mean('hx', 1, 0), mean('hz', 1, 2)


def _coefficients(case, eps, sig):
    """Ca, Cb of the grid: the block, vacuum above it."""
    dx = LAM * case['cell']
    dt = dx * 0.5 / C0
    shape = (case['nz'] - case['nzm'], case['ny'], case['nx'])
    eps = torch.cat([eps, torch.ones(shape, dtype=eps.dtype, device=DEV)]) * E0_MATERIAL
    x = torch.cat([sig, torch.zeros(shape, dtype=sig.dtype, device=DEV)]) * dt / (2 * eps)
    return (1 - x) / (1 + x), dt / (eps * dx) / (1 + x)


def _solve64(case, seed):
    """The 24 phasor planes of a solve, complex128, by name."""
    eps, sig = (v.double() for v in _material(case, seed))
    ca, cb = _coefficients(case, eps, sig)
    del eps, sig
    inc = {k: v.double() for k, v in _incident(case, seed).items()}
    y = _Yee64(case['nz'], case['ny'], case['nx'], LAM * case['cell'], ca, cb)
    n = [v - 2 * NPML for v in y.n]
    shapes = {g: [v for a, v in enumerate(n) if a != ax] for g, ax in zip('dulrfb', (0, 0, 2, 2, 1, 1))}
    out = {k: torch.zeros(shapes[k[-1]], dtype=torch.complex128, device=DEV) for k in PLANES}
    names = {g: [k for k in PLANES if k[-1] == g] for g in 'dulrfb'}
    for t in range(case['nt']):
        y.step(inc, t, _tfsf(case))
        pe, ph = y.phase(t), y.phase(t - 0.5)
        for g in 'dulrfb':
            for k, v in zip(names[g], y.plane_means(g)):
                out[k][1:, 1:] += (pe if k[0] == 'e' else ph) * v
    return out


def _exact_gradient(case, seed):
    """Backscatter power and its derivatives by torch's own reverse mode, the
    steps recomputed in segments."""
    eps, sig = (v.double().requires_grad_() for v in _material(case, seed))
    ca0, cb0 = _coefficients(case, eps, sig)
    ca, cb = ca0.detach().requires_grad_(), cb0.detach().requires_grad_()
    inc = {k: v.double() for k, v in _incident(case, seed).items()}
    y = _Yee64(case['nz'], case['ny'], case['nx'], LAM * case['cell'], ca, cb, functional=True)
    nt, seg, plane = case['nt'], 25, _tfsf(case)
    ny, nx = case['ny'] - 2 * NPML, case['nx'] - 2 * NPML
    f64 = dict(dtype=torch.float64, device=DEV)

    def segment(state, t0):
        """State after steps t0 .. t0 + seg - 1 and their part of the phasors."""
        y.load(state)
        ph = torch.zeros((2, 4, ny - 1, nx - 1), **f64)
        for t in range(t0, min(nt, t0 + seg)):
            y.step(inc, t, plane)
            pe, p_h = y.phase(t), y.phase(t - 0.5)
            for j, v in enumerate(y.plane_means('u')):
                p = pe if j < 2 else p_h
                ph = ph + torch.stack([p.real * v, p.imag * v])[:, None] * torch.eye(4, **f64)[j][None, :, None, None]
        return y.state(), ph

    marks, total = [], torch.zeros((2, 4, ny - 1, nx - 1), **f64)
    with torch.no_grad():
        state = y.state()
        for t0 in range(0, nt, seg):
            marks.append(state)
            state, ph = segment(state, t0)
            total += ph
    total.requires_grad_()
    # the far field in the backscatter direction (theta = -theta_inc, phi = 0)
    dx, k, th = LAM * case['cell'], 2 * math.pi * FREQ / C0, math.radians(-case['theta'])

    def simpson(n):
        w = torch.ones(n, **f64)
        w[1:-1:2], w[2:-1:2] = 4.0, 2.0
        return w * dx / 3.0

    x = (torch.arange(nx, **f64) - (nx - 1) // 2) * dx
    z = ((case['nz'] - 2 * NPML - 1) // 2) * dx
    arg = k * (x[None, :] * math.sin(th) + z * math.cos(th)).expand(ny, nx)
    w = (torch.outer(simpson(ny), simpson(nx)) * torch.complex(torch.cos(arg), torch.sin(arg)))[1:, 1:]
    ex, ey, hx, hy = torch.complex(total[0], total[1])
    ct = math.cos(th)
    n_t, n_p, l_t, l_p = (-ct * w * hy).sum(), (w * hx).sum(), (ct * w * ey).sum(), (-w * ex).sum()
    ff = 1j * k * complex(math.cos(k * RADIUS), -math.sin(k * RADIUS)) / (4 * math.pi * RADIUS)
    if case['pol'] == 'HH':
        power = 0.5 * torch.real(-ff * (l_t - ETA0 * n_p) * torch.conj(ff * (n_p - l_t / ETA0)))
    else:
        power = 0.5 * torch.real(ff * (-l_p - ETA0 * n_t) * torch.conj(ff * (-n_t - l_p / ETA0)))
    (g_ph,) = torch.autograd.grad(power, total)
    lam = [torch.zeros_like(v) for v in state]
    g_ca, g_cb = torch.zeros_like(ca), torch.zeros_like(cb)
    for t0 in reversed(range(0, nt, seg)):
        start = [v.detach().requires_grad_() for v in marks.pop()]
        end, ph = segment(start, t0)
        got = torch.autograd.grad(end + [ph], start + [ca, cb], lam + [g_ph], allow_unused=True)
        lam = [torch.zeros_like(v) if g is None else g for g, v in zip(got, start)]
        g_ca, g_cb = g_ca + got[-2], g_cb + got[-1]
        del end, ph, got
    ge, gs = torch.autograd.grad([ca0, cb0], [eps, sig], [g_ca, g_cb])
    return float(power), ge, gs


def _exact_beam(case, seed):
    """The recorded planes and phasors of the vacuum beam run, from Braunisch's
    tapered wave per pulse frequency (excitation normalised to a peak of 10)."""
    q = _pulse(case, seed)
    ny, nx, nt = case['ny'], case['nx'], case['nt']
    dx = LAM * case['cell']
    dt = dx * 0.5 / C0
    c128 = dict(dtype=torch.complex128, device=DEV)
    tv = np.linspace(0.0, dt * (nt - 1), num=nt)
    sig = q['duration'] / FREQ / (2.0 * math.sqrt(2.0 * math.log(10.0)))
    pulse = np.exp(-(tv - dt * case['npulse'] / 2) ** 2 / sig ** 2) * np.exp(2j * math.pi * FREQ * tv)
    spectrum, freqs = np.fft.fft(pulse), np.fft.fftfreq(nt, dt)
    radius = case['width'] * LAM / (2.0 * math.sqrt(2.0 * math.log(10.0)))
    kx = torch.fft.fftfreq(nx, dx, dtype=torch.float64, device=DEV)[None, :].expand(ny, nx) * 2 * math.pi
    ky = torch.fft.fftfreq(ny, dx, dtype=torch.float64, device=DEV)[:, None].expand(ny, nx) * 2 * math.pi
    kp = torch.hypot(kx, ky)
    pos = kp > 0
    safe = torch.where(pos, kp, torch.ones_like(kp))
    th, ph = math.radians(q['theta']), math.radians(q['phi'])
    eh_, ev_ = {'HH': (1.0, 0.0), 'VV': (0.0, 1.0)}[case['pol']]
    horx = torch.where(pos, ky / safe, torch.full_like(kp, math.sin(ph)))
    hory = torch.where(pos, -kx / safe, torch.full_like(kp, -math.cos(ph)))
    exc = torch.zeros((2, nt, ny, nx), **c128)
    for i, f in enumerate(freqs):
        k = 2 * math.pi * f / C0
        if k == 0.0:
            continue
        kz = torch.conj(torch.sqrt((k * k - kp * kp).to(torch.complex128)))
        kix, kiy = k * math.sin(th) * math.cos(ph), k * math.sin(th) * math.sin(ph)
        kip = math.hypot(kix, kiy)
        kiz = math.sqrt(k * k - kip * kip)
        gauss = radius ** 2 / (4 * math.pi) * torch.exp(-radius ** 2 * ((kx - kix) ** 2 + (ky - kiy) ** 2) / 4)
        verx = torch.where(pos, kz * kx / (k * safe), torch.full_like(kz, math.cos(ph)))
        very = torch.where(pos, kz * ky / (k * safe), torch.full_like(kz, math.sin(ph)))
        verz = torch.where(pos, kp / k, torch.zeros_like(kp))
        hix, hiy = kiy / kip, -kix / kip
        vix, viy, viz = kiz * kix / (k * kip), kiz * kiy / (k * kip), kip / k
        eh = eh_ * (hix * horx + hiy * hory) + ev_ * (vix * horx + viy * hory)
        ev = eh_ * (hix * verx + hiy * very) + ev_ * (vix * verx + viy * very + viz * verz)
        for c, (h, v) in enumerate(((horx, verx), (hory, very))):
            exc[c, i] = complex(spectrum[i]) * torch.fft.fftshift(torch.fft.fft2(gauss * (eh * h + ev * v)))
    exc = torch.fft.ifft(exc, dim=1)
    exc = (exc * (10.0 / exc.abs().max())).imag[:, :case['npulse']].contiguous()
    nz = int(3.0 * LAM / dx)
    cb = dt / (E0 * dx) * torch.ones((nz, ny, nx), dtype=torch.float64, device=DEV)
    y = _Yee64(nz, ny, nx, dx, torch.ones_like(cb), cb)
    z, feed = nz // 2, nz // 2 + 4
    comps = ('ex', 'ey', 'hx', 'hy')
    planes = {c: torch.zeros((nt, ny, nx), dtype=torch.float64, device=DEV) for c in comps}
    out = {f'{c}_inc_phasor': torch.zeros((ny - 2 * NPML, nx - 2 * NPML), **c128) for c in comps}
    m = NPML
    for t in range(nt):
        y.e_half()
        if t < case['npulse']:
            y.f['ex'][feed, 1:-1, :-1] = exc[0, t, 1:-1, :-1]
            y.f['ey'][feed, 1:-1, :-1] = exc[1, t, 1:-1, :-1]
        y.h_half()
        for c in comps:
            planes[c][t] = y.f[c][z]

        def at(c, dz, dy, dx_):
            return y.f[c][z - dz, m + 1 - dy:ny - m - dy, m + 1 - dx_:nx - m - dx_]

        pe, p_h = y.phase(t - 0.5), y.phase(t)
        out['ex_inc_phasor'][1:, 1:] += pe * 0.5 * (at('ex', 0, 0, 0) + at('ex', 0, 0, 1))
        out['ey_inc_phasor'][1:, 1:] += pe * 0.5 * (at('ey', 0, 0, 0) + at('ey', 0, 1, 0))
        out['hx_inc_phasor'][1:, 1:] += p_h * 0.25 * (at('hx', 0, 0, 0) + at('hx', 0, 1, 0) + at('hx', 1, 0, 0)
                                                      + at('hx', 1, 1, 0))
        out['hy_inc_phasor'][1:, 1:] += p_h * 0.25 * (at('hy', 0, 0, 0) + at('hy', 0, 0, 1) + at('hy', 1, 0, 0)
                                                      + at('hy', 1, 0, 1))
    return dict(planes=planes, phasors=out)


def _exact_farfield(case, seed):
    p = {k: v.to(torch.complex128) for k, v in _plane_phasors(case, seed).items()}
    thetas, phis = (np.radians(v) for v in _angles(case))
    ny, nx = case['ny'], case['nx']
    dx, k = LAM * case['cell'], 2 * math.pi * FREQ / C0
    f64 = dict(dtype=torch.float64, device=DEV)

    def simpson(n):
        w = torch.ones(n, **f64)
        w[1:-1:2], w[2:-1:2] = 4.0, 2.0
        return w * dx / 3.0

    x, y = (torch.arange(nx, **f64) - nx // 2) * dx, (torch.arange(ny, **f64) - ny // 2) * dx
    z = ((case['nz'] - 1) // 2) * dx
    w = torch.outer(simpson(ny), simpson(nx))
    ff = 1j * k * complex(math.cos(k * RADIUS), -math.sin(k * RADIUS)) / (4 * math.pi * RADIUS)
    out = {n: np.zeros((len(phis), len(thetas)), np.complex128) for n in ('E_theta', 'E_phi', 'H_theta', 'H_phi')}
    for i, ph in enumerate(phis):
        for j, th in enumerate(thetas):
            ct, st, cp, sp = math.cos(th), math.sin(th), math.cos(ph), math.sin(ph)
            arg = k * (x[None, :] * st * cp + y[:, None] * st * sp + z * ct)
            e = w * torch.complex(torch.cos(arg), torch.sin(arg))
            ix, iy, jx, jy = (complex((e * p[n]).sum()) for n in ('ex_ph_u', 'ey_ph_u', 'hx_ph_u', 'hy_ph_u'))
            n_t, n_p = ct * (-jy * cp + jx * sp), jy * sp + jx * cp
            l_t, l_p = ct * (iy * cp - ix * sp), -iy * sp - ix * cp
            out['E_theta'][i, j] = ff * (-l_p - ETA0 * n_t)
            out['E_phi'][i, j] = ff * (l_t - ETA0 * n_p)
            out['H_theta'][i, j] = ff * (n_p - l_t / ETA0)
            out['H_phi'][i, j] = ff * (-n_t - l_p / ETA0)
    return {n: np.squeeze(v) for n, v in out.items()}


def exact(case, seed):
    kind = case['kind']
    if kind == 'farfield':
        return _exact_farfield(case, seed)
    if kind == 'beam':
        return _exact_beam(case, seed)
    if kind == 'gradient':
        return _exact_gradient(case, seed)
    with torch.no_grad():
        if kind == 'batch':
            members = _members(case)
            if sum(m['nz'] * m['ny'] * m['nx'] for m in members) * case['nt'] > 6e9:
                members = members[:6]   # the rest would take too long
            got = [torch.cat([v.reshape(-1) for v in _solve64(m, seed * 100 + k).values()])
                   for k, m in enumerate(members)]
            return got + [None] * (case['members'] - len(got))
        out = _solve64(case, seed)
    # a plane that the wave has not reached in this many steps holds no value
    # above the noise of its precursors
    top = {c: max(float(v.abs().max()) for k, v in out.items() if k[0] == c) for c in 'eh'}
    return {k: v if float(v.abs().max()) > 1e-6 * top[k[0]] else None for k, v in out.items()}
