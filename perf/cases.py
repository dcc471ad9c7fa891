"""The work users have this package do, as timed cases: 2D E_z and H_z runs from small to the 8192 x 8192 roofline grid,
scattering runs with a plane-wave box, dispersive media, field maps and probes, 3D runs, an adjoint gradient and a
served stream of jobs.  Every case goes through the public entry points (Simulation, EMPhysics3D, FluxAdjoint2D,
ServingLoop) and returns what the run computed: monitor spectra, maps, probe series, fields, gradients.

A case with "resume" continues a long run from fields already on the grid (each pass is its next stretch of steps);
the others run whole simulations from rest, as a parameter sweep does.  ``exact`` restates the same physics in float64
torch: full-grid Yee updates with CPML psi terms as row vectors that are zero outside the layers.
"""
import math

import numpy as np
import torch

import opensol_b200 as ob
from opensol_b200 import serving
from opensol_b200.adjoint import FluxAdjoint2D
from opensol_b200.domain3d import BoundaryConfig3D, Domain3D
from opensol_b200.physics3d import EMPhysics3D

C0, EPS0, MU0 = 299792458.0, 8.8541878128e-12, 1.2566370614e-6
ETA0 = math.sqrt(MU0 / EPS0)
DX = 20e-9
WAVELENGTH, BANDWIDTH = 1550e-9, 0.5


# ---- the cases -------------------------------------------------------------------------------------------------------
def _case2d(name, kind, nx, ny, steps, npml=15, boundaries='pml', shapes=12, freqs=4, lines=2, lossy=False,
            resume=False, tfsf=False, poles=False, maps=0, probes=0):
    case = dict(kind=kind, nx=nx, ny=ny, steps=steps, npml=npml, boundaries=boundaries, shapes=shapes, freqs=freqs,
                lines=lines, lossy=lossy, resume=resume, tfsf=tfsf, poles=poles, maps=maps, probes=probes)
    return dict(case, name=name) if name else case


def _case3d(name, nx, ny, nz, steps, npml=12, faces='pml', shapes=40, freqs=8, resume=False):
    case = dict(kind='em3d', nx=nx, ny=ny, nz=nz, steps=steps, npml=npml, faces=faces, shapes=shapes, freqs=freqs,
                resume=resume)
    return dict(case, name=name) if name else case


def _adjoint(name, n, design, steps, every=256):
    case = dict(kind='adjoint', nx=n, ny=n, npml=20, design=design, steps=steps, every=every)
    return dict(case, name=name) if name else case


def _serving(name, jobs, side_lo, side_hi, steps_lo, steps_hi):
    case = dict(kind='serving', jobs=jobs, side_lo=side_lo, side_hi=side_hi, steps_lo=steps_lo, steps_hi=steps_hi)
    return dict(case, name=name) if name else case


def listed():
    return [
        # a slab on a 240 x 120 window, periodic in y, as a script or a test runs it: the smallest simulation
        _case2d('ez_slab_240x120', 'ez', 240, 120, 1370, boundaries='periodic_y', shapes=1, freqs=2, lines=1),
        # an absorber and dielectrics in an all-CPML box with odd rows, flux lines and time-domain probes
        _case2d('ez_lossy_421x373', 'ez', 421, 373, 1200, npml=10, lossy=True, probes=2),
        # an ordinary device simulation, row length not a multiple of 4
        _case2d('ez_device_1045', 'ez', 1045, 1045, 1500, shapes=30),
        # a plane wave on dispersive scatterers: scattered-field lines, a field map and a probe
        _case2d('ez_scatter_drude_600x480', 'ez', 600, 480, 900, npml=12, shapes=4, tfsf=True, poles=True, maps=2,
                probes=1),
        # the roofline grid: a stretch of a long run on 8192 x 8192 with four 16-frequency lines
        _case2d('ez_roofline_8192', 'ez', 8152, 8152, 3000, npml=20, shapes=2000, freqs=16, lines=4, resume=True),
        # the H_z polarisation: a lossy device with a dispersive part and a field map
        _case2d('hz_metal_360x280', 'hz', 360, 280, 900, npml=12, lossy=True, poles=True, maps=3),
        # an ordinary H_z device simulation
        _case2d('hz_device_900x700', 'hz', 900, 700, 1500, shapes=30),
        # a stretch of a long H_z run on a grid far beyond the cache
        _case2d('hz_large_4096', 'hz', 4056, 4056, 1200, npml=20, shapes=500, freqs=8, lines=4, resume=True),
        # a periodic unit cell between CPML ends, odd sizes
        _case3d('em3d_unit_cell_75x75x141', 75, 75, 141, 500, faces='periodic_xy', shapes=6),
        # a stretch of a 3D run on 384^3 with a closed 8-frequency flux box
        _case3d('em3d_384', 360, 360, 360, 250, shapes=200, resume=True),
        # one optimisation step of an inverse design: objective and its gradient on a design box
        _adjoint('adjoint_640', 600, 160, 1600),
        # a stream of mixed jobs, all queued at once
        _serving('serving_16_jobs', 16, 256, 900, 1200, 2400),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['ez', 'ez', 'ez', 'hz', 'hz', 'em3d', 'adjoint', 'serving'])
    if kind == 'adjoint':
        n = _log(rng, 300, 900)
        steps = int(1.2 * n) + rng.randint(600, 900)   # the pulse has reached the monitor
        return _adjoint(None, n, rng.randint(n // 8, n // 3), steps, rng.choice([128, 256]))
    if kind == 'serving':
        lo = rng.randint(200, 500)
        hi = lo + rng.randint(100, 500)
        steps = int(1.4 * hi)   # long enough for the wave to reach every monitor
        return _serving(None, rng.randint(6, 16), lo, hi, steps, steps + rng.randint(200, 900))
    if kind == 'em3d':
        faces = rng.choice(['pml', 'periodic_xy'])
        nx, ny = _log(rng, 50, 280), _log(rng, 50, 280)
        return _case3d(None, nx, ny, _log(rng, 60, 300), rng.randint(100, 300), npml=rng.choice([8, 12]), faces=faces,
                       shapes=rng.randint(3, 60), resume=rng.random() < 0.3)
    nx = _log(rng, 150, 4000)
    ny = max(100, min(4000, int(nx * rng.uniform(0.5, 1.6))))
    steps = max(300, min(1500, int(4e9 / (nx * ny))))
    large = nx * ny > 2_000_000
    tfsf = kind == 'ez' and not large and rng.random() < 0.25
    return _case2d(None, kind, nx, ny, steps, npml=rng.choice([10, 12, 15, 20]),
                   boundaries='pml' if tfsf else rng.choice(['pml', 'pml', 'periodic_y', 'periodic_x']),
                   shapes=rng.randint(1, 40), freqs=rng.randint(1, 8), lines=rng.randint(1, 4),
                   lossy=rng.random() < 0.3, resume=large, tfsf=tfsf, poles=not large and rng.random() < 0.25,
                   maps=rng.choice([0, 0, 0, 2, 4]), probes=rng.choice([0, 0, 1, 3]))


# ---- inputs from the seed --------------------------------------------------------------------------------------------
def _faces2d(boundaries):
    """(CPML in x, CPML in y)"""
    return boundaries in ('pml', 'periodic_y'), boundaries in ('pml', 'periodic_x')


def _shape2d(case):
    open_x, open_y = _faces2d(case.get('boundaries', 'pml'))
    pad = 2 * case['npml']
    return case['nx'] + pad * open_x, case['ny'] + pad * open_y


def _paint(rng, shape, lo, hi, count, radius):
    """float32 eps_r (1 outside) with `count` discs or balls of eps_r U(2, 12) inside the box lo..hi."""
    eps = np.ones(shape, np.float32)
    for _ in range(count):
        r = rng.uniform(*radius)
        centre = [rng.uniform(a + r, max(a + r + 1, b - r)) for a, b in zip(lo, hi)]
        box = tuple(slice(max(0, int(c - r)), min(n, int(c + r) + 2)) for c, n in zip(centre, shape))
        dist = sum((np.arange(s.start, s.stop).reshape([-1 if k == a else 1 for k in range(len(shape))]) - c) ** 2
                   for a, (s, c) in enumerate(zip(box, centre)))
        eps[box][dist <= r * r] = np.float32(rng.uniform(2.0, 12.0))
    return eps


def _geometry2d(case, seed):
    """eps_r, sigma_e (or None) and the Drude / Lorentz rectangles of a 2D case, in grid cells."""
    rng = np.random.default_rng(seed)
    shape = _shape2d(case)
    open_x, open_y = _faces2d(case['boundaries'])
    lo = [case['npml'] * open_x + 0.3 * case['nx'], case['npml'] * open_y + 0.25 * case['ny']]
    hi = [case['npml'] * open_x + 0.7 * case['nx'], case['npml'] * open_y + 0.75 * case['ny']]
    if case['shapes'] > 100:
        lo = [case['npml'] + 0.15 * n for n in (case['nx'], case['ny'])]
        hi = [case['npml'] + 0.85 * n for n in (case['nx'], case['ny'])]
    size = 0.25 * min(case['nx'], case['ny'])
    eps = _paint(rng, shape, lo, hi, case['shapes'], (2.5, 10.0) if case['shapes'] > 100 else (4.0, max(5.0, size)))
    sigma = None
    if case['lossy']:
        sigma = np.zeros(shape, np.float32)
        a, b = (slice(int(l), int(l + 0.1 * (h - l)) + 2) for l, h in zip(lo, hi))
        sigma[a, b] = np.float32(rng.uniform(1e4, 6e4))
    poles = []
    if case['poles']:
        for kind in ('drude', 'lorentz'):
            at = 0.35 if kind == 'drude' else 0.6
            box = tuple(slice(int(l + at * (h - l)), int(l + (at + rng.uniform(0.1, 0.2)) * (h - l)) + 2)
                        for l, h in zip(lo, hi))
            w = 2 * np.pi * C0 / WAVELENGTH
            poles.append((kind, box, tuple(float(np.float32(v)) for v in
                                           ((rng.uniform(1.5, 3.0) * w, rng.uniform(0.02, 0.1) * w) if kind == 'drude'
                                            else (rng.uniform(0.5, 2.0), rng.uniform(1.5, 2.5) * w, 0.05 * w)))))
    return eps, sigma, poles


def _plane_waves(shape, rng, axes, amplitude=1.0):
    """sum of plane waves (wavelength 24..60 cells) travelling in the plane of two axes, and the same weighted by the
    two direction cosines; float32 numpy, `shape` broadcast over the other axes."""
    device = 'cuda' if torch.cuda.is_available() else 'cpu'
    u, v = (torch.arange(shape[a], device=device, dtype=torch.float32) for a in axes)
    total, along_u, along_v = (torch.zeros(len(u), len(v), device=device) for _ in range(3))
    for _ in range(5):
        angle, k, phase = rng.uniform(0, 2 * np.pi), 2 * np.pi / rng.uniform(24, 60), rng.uniform(0, 2 * np.pi)
        wave = amplitude * torch.cos(k * (math.cos(angle) * u[:, None] + math.sin(angle) * v[None, :]) + phase)
        total += wave
        along_u += math.cos(angle) * wave
        along_v += math.sin(angle) * wave
    return total, along_u, along_v


def _fields2d(case, seed):
    """The fields a resumed run starts from: travelling waves over the whole grid."""
    shape = _shape2d(case)
    wave, cx, cy = _plane_waves(shape, np.random.default_rng(seed + 10_000), (0, 1))
    if case['kind'] == 'ez':
        out = {'ez': wave, 'hx': cy / ETA0, 'hy': -cx / ETA0}
    else:
        out = {'hz': wave / ETA0, 'ex': -cy, 'ey': cx}
    return {k: v.cpu().numpy() for k, v in out.items()}


def _fields3d(shape, seed):
    rng = np.random.default_rng(seed + 10_000)
    wave, cx, cy = _plane_waves(shape, rng, (0, 1))
    other, dy, dz = _plane_waves(shape, rng, (1, 2))
    xy, yz = (lambda a: a[:, :, None].expand(shape)), (lambda a: a[None].expand(shape))
    out = {'ex': yz(other), 'ey': 0 * yz(other), 'ez': xy(wave), 'hx': xy(cy) / ETA0,
           'hy': -xy(cx) / ETA0 + yz(dz) / ETA0, 'hz': -yz(dy) / ETA0}
    return {k: np.ascontiguousarray(v.cpu().numpy()) for k, v in out.items()}


def _setup2d(case):
    """Window cells of the line source, the flux lines (axis, cell), the plane-wave box, the map box and the probes."""
    nx, ny = case['nx'], case['ny']
    open_x, open_y = _faces2d(case['boundaries'])
    along_y = open_x          # the source line lies across the axis with CPML
    source = ('y', int(0.15 * nx)) if along_y else ('x', int(0.15 * ny))
    lines = [('y', int(0.9 * nx)), ('x', int(0.9 * ny)), ('y', int(0.08 * nx)), ('x', int(0.08 * ny))]
    if not along_y:
        lines = [lines[1], lines[0], lines[3], lines[2]]
    lines = lines[:case['lines']]
    box = (int(0.2 * nx), int(0.2 * ny), int(0.8 * nx), int(0.8 * ny))
    probes = [(int(0.5 * nx) + 3 * k, int(0.5 * ny) - 2 * k) for k in range(case['probes'])]
    freqs = np.linspace(0.8, 1.2, case['freqs']) * (C0 / WAVELENGTH)
    return source, lines, box, probes, freqs


def _at(cell):
    return (cell + 0.5) * DX


# ---- what a user's program has in hand before the call ---------------------------------------------------------------
def _prepare2d(case, seed):
    sim = ob.Simulation(case['nx'] * DX, case['ny'] * DX, DX, npml=case['npml'], boundaries=case['boundaries'],
                        polarization=case['kind'], verbose=False)
    eps, sigma, poles = _geometry2d(case, seed)
    if sim.domain.materials.array('eps_r').shape != eps.shape:
        raise ValueError(f"grid {sim.domain.materials.array('eps_r').shape}, expected {eps.shape}")
    names = ('eps_r',) if case['kind'] == 'ez' else ('eps_xx', 'eps_yy')
    for name in names:
        sim.domain.materials.array(name)[...] = eps
    if sigma is not None:
        sim.domain.materials.array('sigma_e')[...] = sigma
    sim.em.materials_changed(names + ('sigma_e',))
    for kind, box, args in poles:
        mask = np.zeros(eps.shape, bool)
        mask[box] = True
        sim.add_dispersive(ob.DrudePole(*args) if kind == 'drude' else ob.LorentzPole(*args), mask)
    source, lines, box, probes, freqs = _setup2d(case)
    if case['tfsf']:
        sim.add_tfsf(*(_at(c) for c in box), wavelength=WAVELENGTH, bandwidth=BANDWIDTH)
    else:
        sim.add_line_source(source[0], _at(source[1]), wavelength=WAVELENGTH, bandwidth=BANDWIDTH)
    out = {}
    for k, (axis, cell) in enumerate(lines):
        span = (case['ny'] if axis == 'y' else case['nx']) * DX
        out[f'flux{k}'] = sim.add_flux_monitor(axis, _at(cell), (0.0, span), frequencies=freqs.tolist()).spectra
    if case['maps']:
        monitor = sim.add_dft_monitor(*(_at(c) for c in box), frequencies=[C0 / WAVELENGTH], downsample=case['maps'])
        maps = ('ez_dft',) if case['kind'] == 'ez' else ('hz_dft', 'ex_dft', 'ey_dft')
        out.update({name: (lambda m=monitor, n=name: getattr(m, n)) for name in maps})
    for k, (i, j) in enumerate(probes):
        probe = sim.add_field_probe(_at(i), _at(j))
        out[f'probe{k}'] = lambda p=probe: p.get_data()[1]
    sim.finalize()
    engine = sim.em.engine
    if case['resume']:
        for name, values in _fields2d(case, seed).items():
            engine.write_field(name, values)
    for name in engine.FIELDS:
        out[name] = lambda n=name: engine.read_field(n)
    return {'case': case, 'sim': sim, 'out': out}


def _domain3d(case):
    faces = {} if case['faces'] == 'pml' else {f'{a}_{s}': 'periodic' for a in 'xy' for s in ('lo', 'hi')}
    config = BoundaryConfig3D(faces, npml=case['npml'])
    return Domain3D.uniform(case['nx'] * DX, case['ny'] * DX, case['nz'] * DX, DX, npml_sides=config.npml_sides,
                            boundary_config=config)


def _geometry3d(case, seed):
    """(eps_r, grid offset of the window, flux box in window cells, source cell)"""
    pads = [case['npml'] * (case['faces'] == 'pml' or a == 2) for a in range(3)]
    window = [case['nx'], case['ny'], case['nz']]
    shape = tuple(n + 2 * p for n, p in zip(window, pads))
    small = 0.25 * min(window)
    eps = _paint(np.random.default_rng(seed), shape, [p + 0.2 * n for p, n in zip(pads, window)],
                 [p + 0.8 * n for p, n in zip(pads, window)], case['shapes'], (2.0, min(14.0, small)))
    box = [(int(0.2 * n), int(0.8 * n)) for n in window]
    return eps, pads, box, tuple(n // 2 for n in window)


def _prepare3d(case, seed):
    physics = EMPhysics3D(_domain3d(case))
    eps, _, box, source = _geometry3d(case, seed)
    physics.domain.materials.array('eps_r')[...] = eps
    physics.materials_changed(('eps_r',))
    physics.add_dipole(_at(source[0]), _at(source[1]), source[2] * DX, orientation='z', dipole_moment=1e-12,
                       wavelength=WAVELENGTH, bandwidth=BANDWIDTH)
    freqs = np.linspace(0.8, 1.2, case['freqs']) * (C0 / WAVELENGTH)
    monitor = physics.add_flux_box(*zip(*[(a * DX, b * DX) for a, b in box]), frequencies=freqs.tolist())
    physics.finalize()
    if case['resume']:
        for name, values in _fields3d(eps.shape, seed).items():
            physics.engine.write_field(name, values)
    return {'case': case, 'physics': physics, 'box': monitor}


def _design(case, seed):
    """(eps_r of the design box, its cells, the source and the monitor column in window cells)"""
    n = case['nx'] + 2 * case['npml']
    i0 = (n - case['design']) // 2
    eps = np.random.default_rng(seed).uniform(1.0, 12.1, (case['design'],) * 2).astype(np.float32)
    return eps, (i0, i0 + case['design'], i0, i0 + case['design']), int(0.15 * case['nx']), int(0.85 * case['nx'])


def _prepare_adjoint(case, seed):
    sim = ob.Simulation(case['nx'] * DX, case['ny'] * DX, DX, npml=case['npml'], verbose=False)
    eps, box, source, line = _design(case, seed)
    sim.domain.materials.array('eps_r')[box[0]:box[1], box[2]:box[3]] = eps
    sim.add_line_source('y', _at(source), wavelength=WAVELENGTH, bandwidth=BANDWIDTH)
    monitor = sim.add_flux_monitor('y', _at(line), (0.0, case['ny'] * DX), wavelengths=[WAVELENGTH])
    sim.finalize()
    return {'case': case, 'adjoint': FluxAdjoint2D(sim, monitor, 0, box, case['steps'], case['every']), 'eps': eps}


def _specs(case, seed):
    return serving.make_job_specs(n_jobs=case['jobs'], rate=0.0, seed=seed, side_range=(case['side_lo'], case['side_hi']),
                                  steps_range=(case['steps_lo'], case['steps_hi']))


def prepare(case, seed):
    if case['kind'] == 'em3d':
        return _prepare3d(case, seed)
    if case['kind'] == 'adjoint':
        return _prepare_adjoint(case, seed)
    if case['kind'] == 'serving':
        return {'case': case, 'loop': serving.ServingLoop(), 'specs': _specs(case, seed)}
    return _prepare2d(case, seed)


# ---- one pass --------------------------------------------------------------------------------------------------------
def run(state):
    case = state['case']
    if case['kind'] == 'serving':
        results = state['loop'].run(state['specs'], realtime=False)
        return [r.fluxes for r in sorted(results, key=lambda r: r.job_id)]
    if case['kind'] == 'adjoint':
        value = state['adjoint'].forward(state['eps'])
        return {'value': value, 'gradient': state['adjoint'].backward()}
    if case['kind'] == 'em3d':
        physics = state['physics']
        if not case['resume']:
            physics.engine.reset()
        physics.run(case['steps'])
        spectra = [plane.spectra() for plane in state['box'].planes()]
        return {'spectra': spectra, 'ez': physics.engine.read_field('ez'), 'hx': physics.engine.read_field('hx')}
    sim = state['sim']
    if not case['resume']:
        sim.em.engine.reset()
    sim.run(n_steps=case['steps'], verbose=False)
    return {name: read() for name, read in state['out'].items()}


def work(case):
    """Bytes: the fields and the material word read once and the fields written once (a gradient: the two sweeps);
    operations: those of the plain Yee update per cell and step, without layers, sources and monitors."""
    if case['kind'] == 'serving':
        # the means of the drawn sides and steps
        a, b = case['side_lo'] + 30, case['side_hi'] + 30
        cells, steps = case['jobs'] * (a * a + a * b + b * b) / 3, (case['steps_lo'] + case['steps_hi']) / 2
        return {'bytes': 28.0 * cells, 'flops': 15.0 * cells * steps}
    if case['kind'] == 'em3d':
        pads = [2 * case['npml'] * (case['faces'] == 'pml' or a == 2) for a in range(3)]
        cells = (case['nx'] + pads[0]) * (case['ny'] + pads[1]) * (case['nz'] + pads[2])
        return {'bytes': 50.0 * cells, 'flops': 36.0 * cells * case['steps']}
    nx, ny = _shape2d(case)
    if case['kind'] == 'adjoint':   # the forward sweep, its recomputation and the transposed sweep
        return {'bytes': 56.0 * nx * ny, 'flops': 45.0 * nx * ny * case['steps']}
    return {'bytes': (28.0 if case['kind'] == 'ez' else 32.0) * nx * ny, 'flops': 15.0 * nx * ny * case['steps']}


def tolerance(case):
    """float32 fields over hundreds to thousands of steps: another order of the sums in a step moves the results by a
    few 1e-6 (the distance to float64 that `exact` shows, up to 8e-6)."""
    return {'rel': 2e-5}


# ---- the same in float64 ---------------------------------------------------------------------------------------------
def _f32(x):
    return np.asarray(np.float32(x), dtype=np.float64)


def _rows(n, npml, cpml, periodic, dt, device):
    """Per axis: inverse spacings of the cell centres and hi faces (kappa folded in) and the CPML recursion b and gain
    of both, zero outside the layers, as float64 vectors."""
    dx = float(np.float32(DX))
    out = {}
    for kind, shift in (('e', 0.0), ('h', 0.5)):
        sigma, kappa = np.zeros(n), np.ones(n)
        if cpml:
            for rows, depth in ((slice(1 if kind == 'e' else 0, npml + (kind == 'e')),
                                 (np.arange(npml - 1, -1, -1) + shift) / npml),
                                (slice(n - npml - 1, n - 1), (np.arange(npml) + shift) / npml)):
                sigma[rows] = 4.0 / (150.0 * np.pi * dx) * depth ** 3
                kappa[rows] = 1.0 + 14.0 * depth ** 3
        b = _f32(np.exp(-(sigma / kappa) * dt / EPS0))
        a = _f32(np.divide(sigma * (b - 1.0), sigma * kappa, out=np.zeros(n), where=sigma > 0))
        inv = _f32(_f32(1.0 / dx) / _f32(kappa))
        if kind == 'h' and not periodic:
            inv[-1] = 0.0
        out[kind] = tuple(torch.as_tensor(v, device=device) for v in (inv, np.where(sigma > 0, b, 0.0), a * _f32(1.0 / dx)))
    return out


class _Axis:
    """Differences along one axis of float64 arrays, with the axis's spacings and CPML recursion."""

    def __init__(self, axis, ndim, n, npml, cpml, periodic, dt, device):
        view = [-1 if a == axis else 1 for a in range(ndim)]
        self.axis, self.cpml = axis, cpml
        rows = _rows(n, npml, cpml, periodic, dt, device)
        self.e, self.h = (tuple(v.reshape(view) for v in rows[kind]) for kind in ('e', 'h'))
        keep = torch.ones(n, dtype=torch.float64, device=device)
        keep[0] = 1.0 if periodic else 0.0
        self.keep = keep.reshape(view)

    def up(self, f, psi):
        """(f[k + 1] - f[k]) / spacing + psi, and the new psi"""
        return self._curl(torch.roll(f, -1, self.axis) - f, self.h, psi)

    def down(self, f, psi):
        return self._curl(f - torch.roll(f, 1, self.axis) * self.keep, self.e, psi)

    def _curl(self, d, rows, psi):
        inv, b, gain = rows
        if not self.cpml:
            return d * inv, psi
        psi = b * psi + gain * d
        return d * inv + psi, psi


def _time_step(axes):
    return float(np.float32(0.99 / (C0 * np.sqrt(axes / (DX if axes == 2 else float(np.float32(DX))) ** 2))))


def _pulse(t, scale=1.0):
    f0 = C0 / WAVELENGTH
    tau = 1.0 / (BANDWIDTH * f0 * np.pi)
    d = t - 4.5 * tau
    return scale * math.exp(-(d / tau) ** 2) * math.sin(2 * math.pi * f0 * d)


def _interval(dt, freqs):
    return max(1, int(np.floor(1.0 / ((C0 / WAVELENGTH * (1 + 3.72 * BANDWIDTH) + float(np.max(freqs))) * dt))))


def _admittance(eps, dt):
    """launch factor of a sheet current on cells of permittivity eps (complex)"""
    omega = 2 * np.pi * C0 / WAVELENGTH
    half = float(DX) * math.sin(0.5 * omega * dt) / (C0 * dt)
    return np.abs(np.sqrt(eps) * np.sqrt(1.0 - eps * half ** 2))


class _Yee2D:
    """The plain float64 step of both polarisations: `f` the out-of-plane field, (a, b) the in-plane pair (x, y)."""

    def __init__(self, case, eps, sigma, device):
        self.ez = case.get('kind') != 'hz'
        nx, ny = eps.shape
        open_x, open_y = _faces2d(case.get('boundaries', 'pml'))
        self.dt = _time_step(2)
        self.x = _Axis(0, 2, nx, case['npml'], open_x, not open_x, self.dt, device)
        self.y = _Axis(1, 2, ny, case['npml'], open_y, not open_y, self.dt, device)
        zeros = lambda: torch.zeros(nx, ny, dtype=torch.float64, device=device)   # noqa: E731
        self.f, self.a, self.b = zeros(), zeros(), zeros()
        self.psi = [zeros() for _ in range(4)]
        eps = torch.as_tensor(eps, dtype=torch.float64, device=device)
        sigma = None if sigma is None else torch.as_tensor(sigma, dtype=torch.float64, device=device)
        self.mu = self.dt / MU0
        if self.ez:
            self.ca, self.cb = self._coefficients(eps, sigma)
        else:
            self.cx = self._coefficients(*(self._face(v, 1, not open_y) for v in (eps, sigma)))
            self.cy = self._coefficients(*(self._face(v, 0, not open_x) for v in (eps, sigma)))

    def _coefficients(self, eps, sigma):
        loss = 0.0 if sigma is None else sigma * self.dt / (2 * eps * EPS0)
        return (1.0 - loss) / (1.0 + loss), self.dt / (eps * EPS0) / (1.0 + loss)

    @staticmethod
    def _face(v, axis, periodic):
        if v is None:
            return None
        nxt = torch.roll(v, -1, axis)
        if not periodic:
            last = [slice(None)] * 2
            last[axis] = slice(-1, None)
            nxt[tuple(last)] = v[tuple(last)]
        return 0.5 * (v + nxt)

    def first_half(self):
        p = self.psi
        if self.ez:
            dy, p[0] = self.y.up(self.f, p[0])
            dx, p[1] = self.x.up(self.f, p[1])
            self.a, self.b = self.a - self.mu * dy, self.b + self.mu * dx
        else:
            dy, p[0] = self.y.down(self.a, p[0])
            dx, p[1] = self.x.down(self.b, p[1])
            self.f = self.f + self.mu * (dy - dx)

    def second_half(self):
        p = self.psi
        if self.ez:
            dx, p[2] = self.x.down(self.b, p[2])
            dy, p[3] = self.y.down(self.a, p[3])
            self.f = self.ca * self.f + self.cb * (dx - dy)
        else:
            dy, p[2] = self.y.up(self.f, p[2])
            dx, p[3] = self.x.up(self.f, p[3])
            self.a = self.cx[0] * self.a + self.cx[1] * dy
            self.b = self.cy[0] * self.b - self.cy[1] * dx


class _PlaneWaveBox:
    """The +x plane-wave box of an E_z run on its 1D incident line."""

    def __init__(self, y, box, npml, device):
        self.y = y
        self.x0, self.y0 = box[0] + npml, box[1] + npml
        self.x1, self.y1 = box[2] + npml + 1, box[3] + npml + 1
        n = self.x1 - self.x0 + 40
        self.e, self.h = (torch.zeros(n, dtype=torch.float64, device=device) for _ in range(2))
        self.ch, self.ce = y.dt / (MU0 * float(np.float32(DX))), y.dt / (EPS0 * float(np.float32(DX)))
        courant = C0 * y.dt / float(np.float32(DX))
        half = 0.5 * (2 * np.pi * C0 / WAVELENGTH) * y.dt
        cos_k = math.sqrt(1.0 - (math.sin(half) / courant) ** 2)
        mur = courant * cos_k / math.cos(half)
        self.scale, self.mur = 2.0 * courant * cos_k, (mur - 1.0) / (mur + 1.0)

    def after_h(self):
        y, e, m = self.y, self.e, 20
        y.b[self.x0 - 1, self.y0:self.y1] -= self.ch * e[m]
        y.b[self.x1 - 1, self.y0:self.y1] += self.ch * e[m + self.x1 - 1 - self.x0]
        inside = e[m:m + self.x1 - self.x0]
        y.a[self.x0:self.x1, self.y0 - 1] += self.ch * inside
        y.a[self.x0:self.x1, self.y1 - 1] -= self.ch * inside
        self.h[:-1] += self.ch * (e[1:] - e[:-1])

    def after_e(self, t_half):
        y, e, h, m = self.y, self.e, self.h, 20
        y.f[self.x0, self.y0:self.y1] -= self.ce * h[m - 1]
        y.f[self.x1 - 1, self.y0:self.y1] += self.ce * h[m + self.x1 - 1 - self.x0]
        old = e[[0, 1, -2, -1]].clone()
        e[1:-1] += self.ce * (h[1:-1] - h[:-2])
        e[10] += _pulse(t_half, self.scale)
        e[0] = old[1] + self.mur * (e[1] - old[0])
        e[-1] = old[2] + self.mur * (e[-2] - old[3])


class _Pole64:
    """One Drude or Lorentz medium on (weighted) samples of one field array."""

    def __init__(self, kind, args, weight, dt):
        self.kind, self.weight = kind, weight
        self.a, self.b = torch.zeros_like(weight), torch.zeros_like(weight)
        gamma = args[1] if kind == 'drude' else args[2]
        denom = 1.0 + gamma * dt / 2.0
        self.damping = -gamma * dt / denom
        if kind == 'drude':
            self.drive = EPS0 * args[0] ** 2 * dt / denom
        else:
            self.restoring = (args[1] * dt) ** 2 / denom
            self.drive = EPS0 * args[0] * self.restoring
        self.dt = dt

    def update(self, field):
        if self.kind == 'drude':
            self.a = self.a + self.damping * self.a + self.drive * self.weight * field
        else:
            self.b = self.b + self.damping * self.b - self.restoring * self.a + self.drive * self.weight * field
            self.a = self.a + self.b

    def current(self):
        return self.a if self.kind == 'drude' else self.b / self.dt


def _run2d(case, eps, sigma, poles, steps, start, source, lines, freqs, box=None, probes=(), device='cuda',
           record=None):
    """The float64 run: {'flux<k>': (E, H), ..., maps, probe series, fields}."""
    y = _Yee2D(case, eps, sigma, device)
    ez, npml = y.ez, case['npml']
    open_x, open_y = _faces2d(case.get('boundaries', 'pml'))
    ox, oy = npml * open_x, npml * open_y
    if start:
        y.f, y.a, y.b = (torch.as_tensor(start[k], dtype=torch.float64, device=device)
                         for k in (('ez', 'hx', 'hy') if ez else ('hz', 'ex', 'ey')))
    if record is not None:
        y.cb = record(y.cb)
    tfsf = _PlaneWaveBox(y, box, npml, device) if case.get('tfsf') else None
    media = []
    for kind, where, args in poles:
        mask = torch.zeros(eps.shape, dtype=torch.float64, device=device)
        mask[where] = 1.0
        if ez:
            media.append((_Pole64(kind, args, mask, y.dt), 'f'))
        else:
            media.append((_Pole64(kind, args, y._face(mask, 1, not open_y), y.dt), 'a'))
            media.append((_Pole64(kind, args, y._face(mask, 0, not open_x), y.dt), 'b'))
    # the source line: cb x launch factor x 2 / (eta0 dx) on its cells (E_z) or hi faces (H_z)
    at = source[1] + (ox if source[0] == 'y' else oy)
    row = (lambda v, k=0: v[at + k] if source[0] == 'y' else v[:, at + k])
    omega = 2 * np.pi * C0 / WAVELENGTH
    loss = np.zeros(eps.shape, np.float32) if sigma is None else sigma
    line_eps = row(eps).astype(np.complex128) - 1j * row(loss).astype(np.float64) / (omega * EPS0)
    if not ez:
        above = row(eps, 1).astype(np.complex128) - 1j * row(loss, 1).astype(np.float64) / (omega * EPS0)
        line_eps = 0.5 * (line_eps + above)
    factor = torch.as_tensor(_admittance(line_eps, y.dt) * 2.0 / (ETA0 * DX), device=device)
    target = 'f' if ez else ('a' if source[0] == 'x' else 'b')
    coefficient = y.cb if ez else (y.cx[1] if source[0] == 'x' else y.cy[1])
    profile = row(coefficient.detach()) * factor
    picks = []
    for axis, cell in lines:
        if axis == 'y':
            where, h, e = (cell + ox, slice(oy, oy + case['ny'])), 'b', 'f'
        else:
            where, h, e = (slice(ox, ox + case['nx']), cell + oy), 'a', 'f'
        picks.append((where, (e, h) if ez else (h, e)))
    monitored = lines or case.get('maps')
    m = _interval(y.dt, freqs if lines else [C0 / WAVELENGTH]) if monitored else 0
    if lines and case.get('maps'):
        m = _interval(y.dt, list(freqs) + [C0 / WAVELENGTH])
    sums = [[None, None] for _ in picks]
    map_sums = None
    if case.get('maps'):
        s = case['maps']
        cut = tuple(slice(lo + off + min(s, hi + 1 - lo) // 2, hi + 1 + off, s)
                    for lo, hi, off in ((box[0], box[2], ox), (box[1], box[3], oy)))
        map_sums = [0, 0, 0] if not ez else [0]
    series = [[] for _ in probes]
    t = 0.0
    for n in range(1, steps + 1):
        t_half, t = t + 0.5 * y.dt, t + y.dt
        old = (y.f, y.a, y.b)
        y.first_half()
        if tfsf:
            tfsf.after_h()
        for pole, name in media:
            pole.update(dict(zip('fab', old))[name])
        y.second_half()
        for pole, name in media:
            cb = y.cb if ez else (y.cx[1] if name == 'a' else y.cy[1])
            setattr(y, name, getattr(y, name) - cb * pole.current())
        if tfsf:
            tfsf.after_e(t_half)
        else:
            value = _pulse(t_half)
            field = getattr(y, target)
            if source[0] == 'y':
                field[at] += value * profile
            else:
                field[:, at] += value * profile
        for k, (i, j) in enumerate(probes):
            series[k].append(y.f[i + ox, j + oy])
        if m and n % m == 0:
            for k, (where, names) in enumerate(picks):
                phase = torch.as_tensor(np.exp(-2j * np.pi * np.asarray(freqs) * t) * m * y.dt, device=device)
                for q, name in enumerate(names):
                    term = phase[:, None] * getattr(y, name)[where][None].to(torch.complex128)
                    sums[k][q] = term if sums[k][q] is None else sums[k][q] + term
            if map_sums is not None:
                w = 2 * np.pi * C0 / WAVELENGTH
                scale = m * y.dt
                if ez:
                    map_sums[0] = map_sums[0] + y.f[cut] * (np.exp(-1j * w * t) * scale)
                else:
                    ex, ey = (0.5 * (v + torch.roll(v, 1, ax)) for v, ax in ((y.a, 1), (y.b, 0)))
                    map_sums[0] = map_sums[0] + y.f[cut] * (np.exp(-1j * w * (t - 0.5 * y.dt)) * scale)
                    map_sums[1] = map_sums[1] + ex[cut] * (np.exp(-1j * w * t) * scale)
                    map_sums[2] = map_sums[2] + ey[cut] * (np.exp(-1j * w * t) * scale)
    out = {f'flux{k}': tuple(s) for k, s in enumerate(sums)}
    if map_sums is not None:
        out.update(zip(('ez_dft',) if ez else ('hz_dft', 'ex_dft', 'ey_dft'), (v[None] for v in map_sums)))
    out.update({f'probe{k}': torch.stack(s) for k, s in enumerate(series)})
    out.update(zip(('ez', 'hx', 'hy') if ez else ('hz', 'ex', 'ey'), (y.f, y.a, y.b)))
    return out, y.dt


def _flux64(spectra, sign, freqs, dt):
    """Power through a line, as FluxMonitor.flux() defines it."""
    e, h = spectra
    freqs = torch.as_tensor(np.asarray(freqs), device=e.device)
    h = h * torch.exp(1j * math.pi * freqs * dt)[:, None]
    return sign * torch.cos(math.pi * freqs * dt) * (e * h.conj()).real.sum(1) * DX


def _host(out):
    """numpy values in the same layout"""
    if isinstance(out, dict):
        return {k: _host(v) for k, v in out.items()}
    if isinstance(out, (list, tuple)):
        return [_host(v) for v in out]
    return out.detach().cpu().numpy() if isinstance(out, torch.Tensor) else out


def _exact2d(case, seed, device):
    eps, sigma, poles = _geometry2d(case, seed)
    source, lines, box, probes, freqs = _setup2d(case)
    start = _fields2d(case, seed) if case['resume'] else None
    out, _ = _run2d(case, eps, sigma, poles, case['steps'], start, source, lines, freqs, box, probes, device)
    return _host(out)


def _exact_adjoint(case, seed, device):
    eps_box, box, source, line = _design(case, seed)
    n = case['nx'] + 2 * case['npml']
    cells = (slice(box[0], box[1]), slice(box[2], box[3]))
    eps = np.ones((n, n), np.float32)
    eps[cells] = eps_box
    variable = torch.as_tensor(eps_box, dtype=torch.float64, device=device).requires_grad_(True)

    def record(cb):
        cb = cb.clone()
        cb[cells] = _time_step(2) / (variable * EPS0)
        return cb
    full = dict(case, kind='ez', boundaries='pml')
    out, dt = _run2d(full, eps, None, (), case['steps'], None, ('y', source), [('y', line)], [C0 / WAVELENGTH],
                     device=device, record=record)
    value = _flux64(out['flux0'], -1.0, [C0 / WAVELENGTH], dt)[0]
    value.backward()
    return _host({'value': value, 'gradient': variable.grad})


def _exact_serving(case, seed, device):
    results = []
    for spec in _specs(case, seed):
        window, n, npml = spec.side * DX, spec.side + 2 * spec.npml, spec.npml
        eps = np.ones((n, n), np.float32)
        centre = (0.5 * ((np.arange(n) - npml) * DX + (np.arange(1, n + 1) - npml) * DX)).astype(np.float32)
        for x0, y0, x1, y1, value in spec.rectangles:
            sx, sy = ((centre >= a * window) & (centre < b * window) for a, b in ((x0, x1), (y0, y1)))
            eps[np.ix_(sx, sy)] = np.float32(value)
        results.append(_job64(spec, eps, window, device))
    return results


def _job64(spec, eps, window, device):
    """Fluxes of one served job: its own wavelength, so its own pulse and sample interval."""
    global WAVELENGTH
    held, WAVELENGTH = WAVELENGTH, spec.wavelength
    try:
        freqs = np.linspace(0.8, 1.2, spec.n_freqs) * (C0 / spec.wavelength)
        cell = (lambda f: min(spec.side - 1, int(math.floor(f * window / DX + 1e-9))))
        case = dict(kind='ez', npml=spec.npml, nx=spec.side, ny=spec.side)
        lines = [('y', cell(0.05)), ('y', cell(0.9))]
        out, dt = _run2d(case, eps, None, (), spec.steps, None, ('y', cell(0.1)), lines, freqs, device=device)
        return [_host(_flux64(out[f'flux{k}'], -1.0, freqs, dt)) for k in range(2)]
    finally:
        WAVELENGTH = held


def _exact3d(case, seed, device):
    eps, pads, box, source = _geometry3d(case, seed)
    shape, dt = eps.shape, _time_step(3)
    axes = [_Axis(a, 3, shape[a], case['npml'], pads[a] > 0, pads[a] == 0, dt, device) for a in range(3)]
    eps = torch.as_tensor(eps, dtype=torch.float64, device=device)
    cb = []
    for a in range(3):
        nxt = torch.roll(eps, -1, a)
        if pads[a]:
            nxt.select(a, -1).copy_(eps.select(a, -1))
        cb.append(dt / (0.5 * (eps + nxt) * EPS0))
    zeros = lambda: torch.zeros(shape, dtype=torch.float64, device=device)   # noqa: E731
    e, h = [zeros() for _ in range(3)], [zeros() for _ in range(3)]
    if case['resume']:
        start = _fields3d(shape, seed)
        e = [torch.as_tensor(start['e' + a], dtype=torch.float64, device=device) for a in 'xyz']
        h = [torch.as_tensor(start['h' + a], dtype=torch.float64, device=device) for a in 'xyz']
    psi_e, psi_h = ([[zeros() if pads[a] else None for a in range(3)] for _ in range(3)] for _ in range(2))
    cell = [c + p for c, p in zip(source, pads)]
    # the dipole sits on the E_z face at the lower edge of its cell: the hi face of the cell below
    cell[2] -= 1
    weight = float(cb[2][tuple(cell)]) * 1e-12 / float(np.float32(DX)) ** 3
    freqs = np.linspace(0.8, 1.2, case['freqs']) * (C0 / WAVELENGTH)
    m = _interval(dt, freqs)
    edges = [(lo + p, hi + p) for (lo, hi), p in zip(box, pads)]
    sums = {}
    t = 0.0
    for n in range(1, case['steps'] + 1):
        t_half, t = t + 0.5 * dt, t + dt
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3
            d1, psi_h[c][u] = axes[u].up(e[v], psi_h[c][u])
            d2, psi_h[c][v] = axes[v].up(e[u], psi_h[c][v])
            h[c] = h[c] - dt / MU0 * (d1 - d2)
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3
            d1, psi_e[c][u] = axes[u].down(h[v], psi_e[c][u])
            d2, psi_e[c][v] = axes[v].down(h[u], psi_e[c][v])
            e[c] = e[c] + cb[c] * (d1 - d2)
        e[2][tuple(cell)] += weight * _pulse(t_half)
        if n % m:
            continue
        phase = torch.as_tensor(np.exp(-2j * np.pi * freqs * t) * m * dt, device=device)
        for a in range(3):
            for side in (0, 1):
                edge = edges[a][side]
                for k, (ea, ha) in enumerate((((a + 1) % 3, (a + 2) % 3), ((a + 2) % 3, (a + 1) % 3))):
                    cut = [None] * 3
                    cut[ea] = slice(max(edges[ea][0], 1) - 1, edges[ea][1])
                    cut[ha] = slice(edges[ha][0], edges[ha][1])
                    low, high = list(cut), list(cut)
                    low[a], high[a] = edge - 1, edge
                    for q, value in enumerate((0.5 * (e[ea][tuple(low)] + e[ea][tuple(high)]), h[ha][tuple(low)])):
                        term = phase[:, None, None] * value[None].to(torch.complex128)
                        key = (a, side, k, q)
                        sums[key] = term if key not in sums else sums[key] + term
    spectra = [[(sums[a, side, k, 0], sums[a, side, k, 1]) for k in range(2)] for a in range(3) for side in (0, 1)]
    return _host({'spectra': spectra, 'ez': e[2], 'hx': h[0]})


def exact(case, seed):
    device = 'cuda' if torch.cuda.is_available() else 'cpu'
    if case['kind'] == 'serving':
        return _exact_serving(case, seed, device)
    if case['kind'] == 'adjoint':
        return _exact_adjoint(case, seed, device)
    if case['kind'] == 'em3d':
        cells = (case['nx'] + 24) * (case['ny'] + 24) * (case['nz'] + 24)
        return None if cells * case['steps'] > 8e9 else _exact3d(case, seed, device)
    nx, ny = _shape2d(case)
    return None if nx * ny * case['steps'] > 3e10 else _exact2d(case, seed, device)
