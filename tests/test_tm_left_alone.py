"""What the TE tiles leave of the components they do not step (E_z, H_x, H_y and their CPML psi): after
an odd number of launches, which leaves the other copies current, the general kernels find them at zero
whatever the memory held before and whatever ran on the context earlier."""
import ctypes as C

import numpy as np
import pytest

from photonoxide_b200.batch import Batch
from photonoxide_b200.engine import Engine
from photonoxide_b200.fdtd import Simulation, library
from photonoxide_b200.types import (INF, Axis, Boundaries, Boxes, Cpml, Field, Grid3d, Periodic, Pml,
                                    Source, Waveform)
from scenarios import noise

pytestmark = pytest.mark.gpu

EDGES = Boundaries(Pml(6, 5), Pml(4, 6), Periodic(), Cpml(kappa=2.0, alpha=0.3))
# the tiles' shape (None: the run alone), precision, and steps that are an odd number of launches
ROUTES = [(None, 32, 40), (None, 64, 40), ((112, 16), 32, 40), ((112, 16), 64, 40), ((120, 40), 32, 36),
          ((120, 24), 64, 36), ((64, 8), 32, 41)]


def grid(precision, n=(130, 45)):
    return Simulation(Grid3d.centred((n[0], n[1], 1), 0.05),
                      Boxes(1.0).add((-0.4, -0.2, -INF), (0.3, 0.25, INF), 9.0), EDGES, 0.9,
                      precision=precision)


def te_fields(s):
    r = np.arange(s.grid.cells())
    for c in range(3):
        zero = np.zeros(r.size)
        s.set_field(Field.E, c, 0.01 * noise(r + 17 * c) if c < 2 else zero)
        s.set_field(Field.H, c, 0.01 * noise(r + 50_000) if c == 2 else zero)


def all_fields(s):
    return [s.e(c) for c in range(3)] + [s.h(c) for c in range(3)]


def silent_ez(s):
    """A source of no amplitude on E_z: the general kernels step the run."""
    s.add_source(Source(Field.E, Axis.Z, (9, 9, 0), Waveform.continuous(1.0, 0.0, 0.0)))


def take(s, tile, steps):
    if tile is None:
        s.run(steps)
    else:
        Batch([s], tile=tile).run(steps)


class Dirty:
    """Device memory in the default pool filled with a pattern that is no zero in either type, freed and
    kept in the pool, where the next allocations come from."""

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        self.rt = C.CDLL("libcudart.so.12")
        self.pool, self.old = C.c_void_p(), C.c_uint64()
        keep = C.c_uint64(1 << 40)
        assert self.rt.cudaDeviceGetDefaultMemPool(C.byref(self.pool), 0) == 0
        assert self.rt.cudaMemPoolGetAttribute(self.pool, 4, C.byref(self.old)) == 0
        assert self.rt.cudaMemPoolSetAttribute(self.pool, 4, C.byref(keep)) == 0
        return self

    def fill(self):
        size, p = C.c_size_t(256 << 20), C.c_void_p()
        assert self.rt.cudaMallocAsync(C.byref(p), size, None) == 0
        assert self.rt.cudaMemsetAsync(p, 0x3e, size, None) == 0
        assert self.rt.cudaFreeAsync(p, None) == 0
        assert self.rt.cudaDeviceSynchronize() == 0

    def __exit__(self, *_):
        self.rt.cudaMemPoolSetAttribute(self.pool, 4, C.byref(self.old))


@pytest.mark.parametrize("tile,precision,steps", ROUTES)
def test_psi_of_e_whatever_the_memory_held(tile, precision, steps):
    with Dirty() as dirty:
        a, o = grid(precision), grid(precision)
        for s in (a, o):
            te_fields(s)
            s.run(1)
        dirty.fill()
        take(a, tile, steps)
        silent_ez(o)
        o.run(steps)
        silent_ez(a)
        for s in (a, o):
            s.run(6)
    for x, y in zip(all_fields(a), all_fields(o)):
        assert np.array_equal(x, y)
    for q in (a.e(2), a.h(0), a.h(1)):
        assert not q.any()


@pytest.mark.parametrize("tile,precision,steps", ROUTES)
def test_psi_of_h_of_an_earlier_tm_run(tile, precision, steps):
    a, o = grid(precision), grid(precision)
    r = np.arange(a.grid.cells())
    for c in range(3):
        a.set_field(Field.E, c, noise(r + c))
        a.set_field(Field.H, c, noise(r + 90 + c))
    a.run(7)
    for s in (a, o):
        te_fields(s)  # the upload starts psi anew
    take(a, tile, steps)
    silent_ez(o)
    o.run(steps)
    silent_ez(a)
    for s in (a, o):
        s.run(6)
    for x, y in zip(all_fields(a), all_fields(o)):
        assert np.array_equal(x, y)
    for q in (a.e(2), a.h(0), a.h(1)):
        assert not q.any()


class Waveform_(C.Structure):
    _fields_ = [("kind", C.c_int32), ("p", C.c_double * 5)]


class Injection(C.Structure):
    _fields_ = [("field", C.c_int32), ("component", C.c_int32), ("r", C.c_int64), ("a_re", C.c_double),
                ("a_im", C.c_double), ("emitter", C.c_int32), ("point", C.c_int32)]


def test_a_te_run_after_tm_steps_through_the_complex_entry(monkeypatch):
    """One context: TE steps, steps with an E_z source through fdtd_bloch_run, TE sources again. The
    fields are no longer TE, and every component goes on."""
    x = library()
    out = []
    for kernel in (None, "quad"):
        if kernel:
            monkeypatch.setenv("PHOTONOXIDE_FDTD_KERNEL", kernel)
        re, im = grid(32), grid(32)
        for s in (re, im):
            te_fields(s)
            s.run(20)
        a, b = Engine(re.engine()), Engine(im.engine())
        wave = Waveform_(2, (C.c_double * 5)(1.0, 1.0, 0.0, 0.0, 0.0))
        ez = Injection(0, 2, 20 * 130 + 60, 1.0, 0.0, 0, 1)
        assert x.fdtd_set_sources(C.c_void_p(a.ctx), 1, C.byref(wave), C.c_int64(1), C.byref(ez)) == 0
        assert x.fdtd_bloch_run(C.c_void_p(a.ctx), C.c_void_p(b.ctx), 0, None, C.c_int64(20), C.c_int64(20)) == 0
        assert x.fdtd_set_sources(C.c_void_p(a.ctx), 0, None, C.c_int64(0), None) == 0
        a.run(24, 40)
        n = 3 * re.grid.cells()
        e, h = np.empty(n), np.empty(n)
        a.download_fields(e, h)
        out.append((e, h))
        assert e[2 * n // 3:].any()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_fields_that_are_not_te_are_looked_at_once(monkeypatch):
    """A run of fields on E_z without sources: the first run's look at the fields is not repeated (a
    kernel, and a wait that fdtd_run_async would make its caller pay on every run)."""
    counts = []
    for kernel in (None, "quad"):
        if kernel:
            monkeypatch.setenv("PHOTONOXIDE_FDTD_KERNEL", kernel)
        s = grid(32)
        r = np.arange(s.grid.cells())
        s.set_field(Field.E, 2, noise(r))
        s.run(40)
        e = Engine(s.engine())
        first = e.launches()
        e.run(40, 40)
        counts.append((first, e.launches(), s.e(2)))
    (a1, a2, a), (o1, o2, o) = counts
    assert a1 == o1 + 1 and a2 == o2
    assert np.array_equal(a, o)


def test_a_caller_captures_te_steps():
    """Steps of a TE run enqueued while the caller captures the context's stream: they are captured (on the
    general kernels, which need no look at the fields and no tables), and replayed they are the same steps."""
    rt = C.CDLL("libcudart.so.12")
    out = []
    for captured in (False, True):
        s = grid(32)
        te_fields(s)
        s.run(2)  # an even number of steps, before and within: a replay finds the same copies current
        e = Engine(s.engine())
        stream = C.c_void_p(e.stream())
        for first in (2, 22):
            if captured and first == 2:
                graph, exec_ = C.c_void_p(), C.c_void_p()
                assert rt.cudaStreamBeginCapture(stream, 1) == 0
                e.run_async(20, first)
                assert rt.cudaStreamEndCapture(stream, C.byref(graph)) == 0
                assert rt.cudaGraphInstantiate(C.byref(exec_), graph, C.c_ulonglong(0)) == 0
            if captured:
                assert rt.cudaGraphLaunch(exec_, stream) == 0
            else:
                e.run_async(20, first)
        e.synchronize()
        if captured:
            assert rt.cudaGraphExecDestroy(exec_) == 0 and rt.cudaGraphDestroy(graph) == 0
        n = 3 * s.grid.cells()
        E, H = np.empty(n), np.empty(n)
        e.download_fields(E, H)
        out.append((E, H))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
