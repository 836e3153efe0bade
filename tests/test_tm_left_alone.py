"""What the TE tiles leave of the components they do not step (E_z, H_x, H_y and their CPML psi): after
an odd number of launches, which leaves the other copies current, the general kernels find them at zero
whatever the memory held before and whatever ran on the context earlier."""
import ctypes as C

import numpy as np
import pytest

from photonoxide_b200.batch import Batch
from photonoxide_b200.fdtd import Simulation
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
