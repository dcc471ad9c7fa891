"""Large reads (4 MB and more, which several threads fetch) hold what the work queued before them leaves, whatever the
caller's stream, and the same values as reads of an engine on its own stream."""
import numpy as np
import pytest

import opensol_b200 as ob
from opensol_b200 import workloads

pytestmark = pytest.mark.gpu
PER_THREAD = 2   # cudaStreamPerThread: a handle that names another stream in every thread
CELLS = 1100     # 4.84 MB a field
STEPS = 600


def _sim():
    sim = ob.Simulation(**workloads.roofline_2d_sim_args(total_cells=CELLS), verbose=False)
    workloads.apply(sim, workloads.roofline_2d_ops(total_cells=CELLS, n_cylinders=30, seed=5))
    sim.em.finalize()
    return sim


def _streams():
    import torch
    return [PER_THREAD, torch.cuda.Stream().cuda_stream]


def _fields(engine):
    return [engine.read_field(name) for name in ('ez', 'hx', 'hy')]


@pytest.mark.parametrize('variant', [1, 3])
@pytest.mark.parametrize('which', [0, 1])
def test_read_on_a_callers_stream(variant, which):
    got = []
    for stream in (None, _streams()[which]):
        sim = _sim()
        engine = sim.em.engine
        engine.configure(variant=variant)
        engine.set_stream(stream)
        engine.advance(STEPS)
        got.append(_fields(engine))
        engine.set_stream(None)
        engine.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
    assert np.abs(got[0][0]).max() > 0


@pytest.mark.parametrize('cells', [1000, 1030, 1100, 2540])
def test_read_into_fresh_and_used_memory(cells):
    """Destinations whose pages are there and whose are not take different ways (from 4 and 24 MB: 1000 and 1030, 2540
    cells a side lie around them): the same values."""
    import mmap
    from opensol_b200 import _native
    sim = ob.Simulation(**workloads.roofline_2d_sim_args(total_cells=cells), verbose=False)
    sim.em.finalize()
    engine = sim.em.engine
    want = np.random.default_rng(cells).standard_normal((engine.nx, engine.ny)).astype(np.float32)
    engine.write_field('hx', want)
    lib = _native.load()
    for used in (False, True):
        out = np.frombuffer(mmap.mmap(-1, want.nbytes + 4), np.float32)[1:].reshape(want.shape)
        if used:
            out[...] = np.nan
        _native.check(lib.os_fdtd2d_read_field(engine.handle, 1, _native.fptr(out)))
        np.testing.assert_array_equal(out, want)


def test_read_into_page_locked_memory():
    """A page-locked destination takes one direct copy: the same values."""
    import ctypes
    from opensol_b200 import _native
    sim = _sim()
    engine = sim.em.engine
    engine.advance(STEPS)
    want = _fields(engine)
    lib, p = _native.load(), ctypes.c_void_p()
    _native.check(lib.os_fdtd_host_alloc(want[0].nbytes, ctypes.byref(p)))
    try:
        out = np.frombuffer((ctypes.c_char * want[0].nbytes).from_address(p.value), np.float32).reshape(want[0].shape)
        for component, field in enumerate(want):
            out[...] = np.nan
            _native.check(lib.os_fdtd2d_read_field(engine.handle, component, _native.fptr(out)))
            np.testing.assert_array_equal(out, field)
    finally:
        _native.check(lib.os_fdtd_host_free(p))
