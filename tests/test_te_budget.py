"""What a 2D TE run's tables take counts against the context's HBM budget, and gives way to anything else
the context needs."""
import ctypes as C
import gc

import numpy as np
import pytest

from photonoxide_b200.engine import Engine
from photonoxide_b200.fdtd import Simulation
from photonoxide_b200.types import Axis, Boundaries, Boxes, Field, Grid3d, Source, Waveform

pytestmark = pytest.mark.gpu

MB = 1 << 20


def pool_bytes():
    """The device's default pool's memory in use."""
    import torch
    torch.cuda.synchronize()
    rt = C.CDLL("libcudart.so.12")
    pool, used = C.c_void_p(), C.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, C.byref(used)) == 0
    return used.value


def make(budget):
    s = Simulation(Grid3d.centred((400, 300, 1), 0.04), Boxes(2.0), Boundaries.cpml_2d(8), 0.7,
                   hbm_budget=budget)
    s.add_source(Source(Field.H, Axis.Z, (200, 150, 0), Waveform.pulse(1.0, 0.6)))
    s.add_dft((0, 0, 0), (399, 299, 0), [0.9])
    for q in range(500):
        s.add_probe(Field.E, Axis.X, (30 + q % 300, 40 + q // 300, 0))
    return s


def test_the_tables_count_and_give_way(monkeypatch):
    monkeypatch.setenv("PHOTONOXIDE_FDTD_KERNEL", "quad")
    gc.collect()
    before = pool_bytes()
    o = make(0)
    o.run(40)
    general = pool_bytes() - before  # the engine's own, on the general kernels
    o.run(25_000)
    want, probe = o.transforms(), o.probe(499)
    record = 25_040 * 500 * 8
    del o
    gc.collect()
    monkeypatch.delenv("PHOTONOXIDE_FDTD_KERNEL")
    # room for the tables or for the record of the second run's probes, not for both in full; and for the
    # record alone
    for budget in (general + record + 40 * MB, general + record + 2 * MB):
        before = pool_bytes()
        s = make(budget)
        s.run(40)
        assert pool_bytes() - before <= budget
        s.run(25_000)
        assert pool_bytes() - before <= budget
        assert np.array_equal(s.transforms(), want) and np.array_equal(s.probe(499), probe)
        del s
        gc.collect()


def test_short_rings_and_chunks_of_half_the_length(monkeypatch):
    """Transforms whose ring the engine's 1 GB cuts to 8 rows (the tiles' chunks are of 16 steps: half of
    the plane's values stay zero in a TE run): the general kernels' bits."""
    def big():
        s = Simulation(Grid3d.centred((1001, 1500, 1), 0.04), Boxes(2.0), Boundaries.cpml_2d(8), 0.7, precision=64)
        s.add_source(Source(Field.H, Axis.Z, (200, 150, 0), Waveform.pulse(1.0, 0.6)))
        s.add_dft((0, 0, 0), (1000, 1499, 0), [0.9])
        for steps in (40, 8992, 51):  # the tables wait for a thousandth of the 9 million values' steps
            s.run(steps)
            counts.append(Engine(s.engine()).launches() / steps)
        return s.h(2), s.transforms()

    counts = []
    a = big()
    monkeypatch.setenv("PHOTONOXIDE_FDTD_KERNEL", "quad")
    b = big()
    general, tiles = counts[0], counts[2]
    assert tiles < 0.7 * general and counts[5] > 0.9 * general  # (a launch a step, and the recording's)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
