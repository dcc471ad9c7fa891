"""The resident form of the 2D step (a whole chunk in one launch, fields in registers; what a new engine runs where
the grid fits) against the per-half-step kernels (variant 0), which the oracle and open_sol's fixtures pin: fields,
spectra, maps and probe series bit for bit, on strips of one row and of many, every boundary preset, odd rows, lossy
and magnetic cells, plane-wave boxes, poles, chunk ends on and off DFT samples, and switches between the forms."""
import ctypes

import numpy as np
import pytest

import opensol_b200 as ob
from opensol_b200 import _native

pytestmark = pytest.mark.gpu
DX = 20e-9


def _sim(pol, nx, ny, boundaries, npml, seed, lossy=False, magnetic=False, tfsf=0, poles=(), maps=(), probes=0,
         lines=('y', 'x')):
    rng = np.random.default_rng(seed)
    sim = ob.Simulation(nx * DX, ny * DX, DX, npml=npml, boundaries=boundaries, polarization=pol, verbose=False)
    shape = (sim.grid.nx, sim.grid.ny)
    materials = sim.domain.materials
    for name in (('eps_r',) if pol == 'ez' else ('eps_xx', 'eps_yy')):
        materials.array(name)[...] = rng.uniform(2.0, 6.0, shape)   # above the poles' stability term
    if lossy:
        materials.array('sigma_e')[...] = rng.uniform(0, 4e4, shape) * (rng.random(shape) < 0.3)
    if magnetic:
        materials.array('mu_r')[...] = rng.uniform(1.0, 2.0, shape)
        materials.array('sigma_m')[...] = rng.uniform(0, 1e3, shape)
    sim.em.materials_changed(('eps_r', 'eps_xx', 'eps_yy', 'sigma_e', 'mu_r', 'sigma_m'))
    at = lambda cell: (cell + 0.5) * DX   # noqa: E731
    for k, pole in enumerate(poles):
        mask = np.zeros(shape, bool)
        a, b = int(shape[0] * (0.3 + 0.1 * k)), int(shape[1] * 0.3)
        mask[a:a + shape[0] // 4 + 1, b:b + shape[1] // 3 + 1] = rng.random((shape[0] // 4 + 1, shape[1] // 3 + 1)) < 0.8
        sim.add_dispersive(pole, mask)
    for k, axis in enumerate(lines):
        n_across, n_along = (nx, ny) if axis == 'y' else (ny, nx)
        span = None if k == 0 else (at(n_along // 5), at(4 * n_along // 5))
        sim.add_line_source(axis, at(int(0.3 * n_across)), wavelength=700e-9, bandwidth=0.8, amplitude=1.0 + k,
                            span=span)
    for k in range(tfsf):
        sim.add_tfsf(at(4 + k), at(5 + k), at(nx - 6), at(ny - 5 - k), wavelength=800e-9, bandwidth=0.5)
    freqs = [3.5e14, 4.2e14, 5e14]
    out = [sim.add_flux_monitor('y', at(int(f * nx)), (0.0, ny * DX), frequencies=freqs).spectra for f in (0.1, 0.8)]
    out.append(sim.add_flux_monitor('x', at(int(0.7 * ny)), (at(1), at(nx - 2)), frequencies=freqs[:1]).spectra)
    for ds in maps:
        monitor = sim.add_dft_monitor(0.0, at(1), nx * DX, at(ny - 2), frequencies=freqs[:2], downsample=ds)
        out.append(lambda m=monitor: m._maps())
    components = ('ez', 'hx', 'hy') if pol == 'ez' else ('hz', 'ex', 'ey')
    for k in range(probes):
        probe = sim.add_field_probe(at(int((0.2 + 0.29 * k) * nx)), at(int((0.8 - 0.3 * k) * ny)), components[k % 3])
        out.append(lambda p=probe: p.get_data()[1])
    sim.finalize()
    start = np.random.default_rng(seed + 1)
    for name in sim.em.engine.FIELDS:
        scale = 1.0 if name[0] == 'e' else 2.7e-3
        sim.em.engine.write_field(name, (scale * start.standard_normal(shape)).astype(np.float32))
    return sim, out


def _outputs(sim, out):
    engine = sim.em.engine
    got = [engine.read_field(name) for name in engine.FIELDS]
    for read in out:
        value = read()
        got.extend(value if isinstance(value, tuple) else [value])
    return got


def _compare(args, chunks, switch=None, resident=None):
    """chunks of steps in the resident form and in variant 0 from the same seeded fields; `switch`: after that chunk the
    resident engine continues with the blocked kernels and then goes back; `resident`: which chunks run resident (all)."""
    sim, out = _sim(**args)
    ref, ref_out = _sim(**args)
    ref.em.engine.configure(variant=0)
    for k, n in enumerate(chunks):
        if switch is not None and k in (switch, switch + 1):
            sim.em.engine.configure(variant=1 if k == switch else 3)
        sim.em.engine.advance(n)
        launches = sim.em.engine.launch_count()
        if resident is not None and not resident[k]:
            assert launches != 1   # the flux lines' folds aside, a resident chunk is one launch
        elif switch is None or k != switch:
            assert launches <= 1 + 3   # one resident launch, one fold per flux line
        ref.em.engine.advance(n)
    for a, b in zip(_outputs(sim, out), _outputs(ref, ref_out)):
        np.testing.assert_array_equal(a, b)
        assert np.isfinite(np.asarray(b)).all()
    assert np.abs(_outputs(sim, out)[0]).max() > 0


DRUDE, LORENTZ = ob.DrudePole(6e15, 2e14), ob.LorentzPole(1.5, 5e15, 3e14)
CASES = [
    dict(nx=120, ny=75, boundaries='pml', npml=10),
    dict(nx=127, ny=64, boundaries='pml', npml=10, lossy=True, probes=3),            # 147 strips of one row
    dict(nx=129, ny=33, boundaries='pml', npml=10, magnetic=True, probes=2),         # 149 rows: strips of one and two
    dict(nx=300, ny=1200, boundaries='pml', npml=15, maps=(3,)),                     # blocks of 640 threads
    dict(nx=777, ny=129, boundaries='periodic_y', npml=15, maps=(1,), probes=1),
    dict(nx=150, ny=131, boundaries='periodic_x', npml=8, lines=('x', 'y'), maps=(2,)),
    dict(nx=149, ny=90, boundaries='periodic', npml=15, lossy=True, magnetic=True),
    dict(nx=160, ny=140, boundaries='pml', npml=12, tfsf=1, lines=(), poles=(DRUDE, LORENTZ), probes=1),
    dict(nx=90, ny=141, boundaries='periodic_y', npml=9, poles=(DRUDE, DRUDE, LORENTZ), lossy=True, maps=(2,)),
    dict(nx=330, ny=77, boundaries='periodic_x', npml=9, lines=('x',), poles=(LORENTZ,), tfsf=2),
]


@pytest.mark.parametrize('pol', ['ez', 'hz'])
@pytest.mark.parametrize('case', range(len(CASES)))
def test_resident_equals_per_step(pol, case):
    args = dict(CASES[case], pol=pol, seed=100 + case)
    _compare(args, (41, 1, 2, 36))


@pytest.mark.parametrize('pol', ['ez', 'hz'])
def test_resident_among_the_other_forms(pol):
    """Chunks in the resident form, then blocked, then resident again continue one run."""
    _compare(dict(pol=pol, nx=200, ny=164, boundaries='pml', npml=10, seed=7, maps=(3,), probes=2), (20, 31, 25), 1)


@pytest.mark.parametrize('pol', ['ez', 'hz'])
@pytest.mark.parametrize('chunks', [(1,) * 60, (2,) * 30, (1, 2, 3, 30, 1)])
def test_plane_wave_in_short_launches(pol, chunks):
    """A plane wave's line is read by every strip and written by one: launches of fewer steps than there are strips, on
    148 of them, the box reaching from the first strips to the last."""
    _compare(dict(pol=pol, nx=320, ny=60, boundaries='pml', npml=6, tfsf=2, lines=(), seed=21), chunks)


# One set of grids per kernel shape (columns a thread, rows a strip, threads) of the launch table; cells a side with the
# CPML, so that the columns leave 1, 2 and 3 over whole threads.
SHAPES = {
    (2, 8, 640): [dict(nx=1100, ny=1131, boundaries='pml'), dict(nx=700, ny=1050, boundaries='periodic_y', lossy=True),
                  dict(nx=1020, ny=1203, boundaries='periodic_x', maps=(7,), probes=2)],
    (2, 16, 384): [dict(nx=2300, ny=301, boundaries='pml', probes=3), dict(nx=1330, ny=90, boundaries='periodic', lossy=True),
                   dict(nx=1900, ny=203, boundaries='periodic_y', maps=(30,)), dict(nx=1500, ny=77, boundaries='pml', tfsf=2,
                                                                                   lines=())],
    (2, 24, 256): [dict(nx=2900, ny=121, boundaries='pml'), dict(nx=2700, ny=63, boundaries='periodic_y', probes=1),
                   dict(nx=2800, ny=130, boundaries='pml', tfsf=1, lines=())],
    (4, 4, 640): [dict(nx=560, ny=1501, boundaries='pml', tfsf=1, lines=(), poles=('drude', 'lorentz'), probes=2),
                  dict(nx=300, ny=1402, boundaries='periodic_y', poles=('lorentz',), lossy=True, maps=(6,)),
                  dict(nx=420, ny=1999, boundaries='periodic_x', poles=('drude', 'drude'), lines=('x', 'y'))],
    (4, 8, 512): [dict(nx=760, ny=1501, boundaries='pml', tfsf=1, lines=(), poles=('drude', 'lorentz')),
                  dict(nx=700, ny=1402, boundaries='periodic_y', poles=('lorentz',), magnetic=True),
                  dict(nx=1000, ny=1299, boundaries='periodic', poles=('drude',), maps=(9,))],
    (4, 10, 384): [dict(nx=1400, ny=901, boundaries='pml', tfsf=2, lines=(), probes=2),
                   dict(nx=1450, ny=1002, boundaries='pml', tfsf=1, lines=('y',), maps=(8,)),
                   dict(nx=1350, ny=1503, boundaries='periodic_y', tfsf=1)],
    (4, 16, 256): [dict(nx=2200, ny=801, boundaries='pml', tfsf=1, lines=()),
                   dict(nx=1650, ny=1002, boundaries='periodic_y', tfsf=2, maps=(9,)),
                   dict(nx=1580, ny=903, boundaries='periodic_x', tfsf=1, lossy=True, lines=('x',))],
}


@pytest.mark.parametrize('pol', ['ez', 'hz'])
@pytest.mark.parametrize('shape, case', [(shape, k) for shape in SHAPES for k in range(len(SHAPES[shape]))])
def test_every_kernel_shape(pol, shape, case):
    args = dict(SHAPES[shape][case], pol=pol, seed=50 + case, npml=7)
    for axis, n in (('x', 'nx'), ('y', 'ny')):
        if args['boundaries'] not in ('periodic', f'periodic_{axis}'):
            args[n] -= 14
    args['poles'] = tuple({'drude': DRUDE, 'lorentz': LORENTZ}[p] for p in args.get('poles', ()))
    _compare(args, (24, 20, 25))
    # the shapes before this one in the table do not fit, so the launch used it
    tall, wide = -(-SHAPES[shape][case]['nx'] // 148), SHAPES[shape][case]['ny']
    table = [(2, 4, 640), (2, 8, 512), (2, 8, 640), (4, 4, 640), (2, 16, 384), (4, 8, 512), (2, 24, 256), (4, 10, 384),
             (4, 16, 256)]
    fits = [s for s in table if tall <= s[1] and -(-wide // s[0]) <= s[2]
            and (s[0] == 2 or args['poles'] or args.get('tfsf'))]
    assert fits[0] == shape


# rows a strip, steps of the shortest resident chunk (E_z, H_z), features
RULE = [(4, 1, 2, {}), (5, 3, 3, {}), (8, 4, 4, {}), (13, 7, 7, {}), (17, 9, 9, {}), (20, 20, 20, {}),
        (6, 2, 2, dict(probes=1)), (7, 4, 4, dict(probes=1)), (6, 2, 2, dict(maps=(5,))), (8, 4, 4, dict(maps=(5,)))]


@pytest.mark.parametrize('pol', ['ez', 'hz'])
@pytest.mark.parametrize('rows, ez_steps, hz_steps, features', RULE)
def test_short_chunks_take_the_quicker_form(pol, rows, ez_steps, hz_steps, features):
    """A chunk runs resident from the length at which its launch pays for reading and writing the strips' state; chunks
    on both sides of the line continue one run."""
    least = hz_steps if pol == 'hz' else ez_steps
    args = dict(pol=pol, nx=148 * rows - 12 - 2 * rows, ny=36, boundaries='pml', npml=6, seed=rows, **features)
    chunks = [n for n in (least, least - 1, least + 1, max(1, least - 1)) if n]
    _compare(args, chunks, resident=[n >= least for n in chunks])


# polarisation, features, rows a strip up to which they run resident, columns
TALL = [('ez', {}, 20, 64), ('hz', {}, 22, 64), ('hz', dict(lossy=True), 5, 1040), ('ez', dict(tfsf=1, lines=()), 12, 60),
        ('hz', dict(lossy=True), 9, 60), ('ez', dict(lossy=True), 17, 60), ('hz', dict(magnetic=True), 9, 60),
        ('ez', dict(magnetic=True), 9, 60), ('ez', dict(magnetic=True), 17, 302), ('hz', dict(maps=(40,)), 16, 60),
        ('ez', dict(maps=(3,)), 17, 60), ('ez', dict(poles=(DRUDE,)), 14, 60), ('hz', dict(poles=(DRUDE,)), 12, 60),
        ('ez', dict(poles=(LORENTZ,)), 12, 820), ('hz', dict(poles=(LORENTZ,)), 8, 1340)]


@pytest.mark.parametrize('pol, features, rows, ny', TALL)
def test_tall_strips_take_the_quicker_form(pol, features, rows, ny):
    for r in (rows, rows + 1):
        args = dict(pol=pol, nx=148 * r - 12 - 2 * r, ny=ny - 12, boundaries='pml', npml=6, seed=r, **features)
        _compare(args, (45, 2 * rows + 2), resident=[r == rows] * 2)


@pytest.mark.parametrize('pol, rows, maps, resident', [
    ('ez', 8, (1, 1, 1), True), ('ez', 8, (1, 1, 1, 1), False), ('ez', 3, (1, 1, 1, 1), True), ('ez', 14, (1,), True),
    ('ez', 14, (1, 1), False), ('hz', 3, (1, 1, 1, 1), True), ('hz', 4, (1, 1, 1, 1), False), ('hz', 8, (2,), True),
    ('hz', 8, (1,), False), ('hz', 12, (9,), False), ('hz', 12, (13,), True)])
def test_maps_with_many_terms_take_the_quicker_form(pol, rows, maps, resident):
    args = dict(pol=pol, nx=148 * rows - 12 - 2 * rows, ny=48, boundaries='pml', npml=6, seed=rows, maps=maps)
    sim, _out = _sim(**args)
    assert sim.em.engine.sample_interval == 9   # two frequencies a map: 2 x 2 x rows / 9 terms a thread and step, H_z 3 times
    _compare(args, (40, 31), resident=[resident] * 2)


def test_resident_chunk_past_the_staged_samples():
    """A chunk with more DFT samples than one launch stages (every step sampled) runs in several launches."""
    got = []
    for variant in (3, 0):
        sim, out = _sim('ez', 30, 1200, 'pml', 10, seed=9)
        sim.em.engine.configure(variant=variant)
        sim.em.engine.set_sample_interval(1)
        sim.em.engine.advance(4000)
        if variant == 3:
            assert sim.em.engine.launch_count() == 2 * (1 + 3)
        got.append(_outputs(sim, out))
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


def test_resident_two_rows():
    """The smallest strips: a periodic grid of 2 x 40 cells, and of 3 rows."""
    for nx in (2, 3):
        sim, out = {}, {}
        for variant in (3, 0):
            s = ob.Simulation(nx * DX, 40 * DX, DX, boundaries='periodic', verbose=False)
            s.add_line_source('x', 10.5 * DX, wavelength=700e-9)
            s.em.engine.configure(variant=variant)
            s.run(n_steps=55, verbose=False)
            sim[variant], out[variant] = s, [s.em.engine.read_field(n) for n in ('ez', 'hx', 'hy')]
        for a, b in zip(out[3], out[0]):
            np.testing.assert_array_equal(a, b)
        assert np.abs(out[0][0]).max() > 0


def test_resident_engines_share_the_device():
    """Engines on streams of their own advanced from the host in turn: each launch needs the whole chip, and every
    result is that of the engine alone."""
    args = [dict(pol=p, nx=180, ny=100, boundaries='pml', npml=10, seed=s) for p, s in (('ez', 1), ('hz', 2), ('ez', 3))]
    together = [_sim(**a) for a in args]
    for _ in range(3):
        for sim, _out in together:
            sim.em.engine.advance(40)
    for a, (sim, out) in zip(args, together):
        alone, alone_out = _sim(**a)
        for _ in range(3):
            alone.em.engine.advance(40)
        for x, y in zip(_outputs(sim, out), _outputs(alone, alone_out)):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize('pol', ['ez', 'hz'])
def test_resident_passes_repeat(pol):
    """Whole passes from rest on one engine, with other engines' passes queued between: every pass gives the same bits,
    those of the per-step kernels."""
    runs = [dict(nx=250, ny=131, boundaries='pml', npml=8, lossy=True, probes=2, maps=(3,)),
            dict(nx=300, ny=90, boundaries='pml', npml=8, tfsf=1, lines=(), poles=(DRUDE, LORENTZ), maps=(2,)),
            dict(nx=900, ny=203, boundaries='periodic_y', npml=8, probes=1),
            dict(nx=700, ny=1300, boundaries='pml', npml=8, poles=(LORENTZ,))]
    sims = [_sim(pol=pol, seed=30 + k, **args) for k, args in enumerate(runs)]
    first = [None] * len(runs)
    for repeat in range(3):
        for sim, _out in sims:
            sim.em.engine.reset()
            for n in (60, 31):
                sim.em.engine.advance(n)
        for k, (sim, out) in enumerate(sims):
            got = [np.array(a) for a in _outputs(sim, out)]
            if repeat == 0:
                ref, ref_out = _sim(pol=pol, seed=30 + k, **runs[k])
                ref.em.engine.configure(variant=0)
                ref.em.engine.reset()
                for n in (60, 31):
                    ref.em.engine.advance(n)
                first[k] = [np.array(a) for a in _outputs(ref, ref_out)]
            for a, b in zip(got, first[k]):
                np.testing.assert_array_equal(a, b)


def test_resident_bounded_wait():
    """A boundary row that never arrives (the test hook: one strip sends none for 1 ms and leaves) ends the launch with
    the error status; the engine runs again after a reset."""
    args = dict(pol='ez', nx=150, ny=100, boundaries='pml', npml=10, seed=4)
    sim, out = _sim(**args)
    engine = sim.em.engine
    engine.set_stall_probe(1_000_000)
    engine.advance(30)
    with pytest.raises(RuntimeError, match='bounded wait'):
        engine.synchronize()
    engine.set_stall_probe(0)
    engine.reset()
    engine.advance(30)
    engine.synchronize()
    clean, clean_out = _sim(**args)
    clean.em.engine.reset()
    clean.em.engine.advance(30)
    for a, b in zip(_outputs(sim, out), _outputs(clean, clean_out)):
        np.testing.assert_array_equal(a, b)


def test_variant_range_is_refused():
    sim, _ = _sim(pol='ez', nx=40, ny=40, boundaries='pml', npml=8, seed=1)
    for variant in (-1, 4):
        with pytest.raises(ValueError):
            _native.check(_native.load().os_fdtd2d_configure(sim.em.engine.handle, ctypes.c_int32(variant), 3, 0))
