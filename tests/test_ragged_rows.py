"""Grids whose rows are not whole vectors of four on the quad kernel, psi's padded rows carried out
and in again, and short runs of planes on grids with few tiles: in f64 the oracle's bits, in f32 the
bits of the row kernel, which takes any width."""
import numpy as np
import pytest

from photonoxide_b200.fdtd import Simulation
from photonoxide_b200.types import (Axis, Boundaries, Boxes, Cpml, Dispersive, Field, Grid3d,
                                    Periodic, Pml, Pole)
from scenarios import busy, noise

pytestmark = pytest.mark.gpu


def stirred(make, n, edges, lossy=False, media=False):
    s = make(Grid3d.centred(n, 0.04), Boxes(2.0).add((-0.2, -0.1, -1.0), (0.25, 0.15, 1.0), 9.0),
             Boundaries(*edges, Cpml(kappa=2.5, alpha=0.25)), 0.8)
    if lossy:
        s.with_conductivity(Boxes(0.3))
    if media:
        s.with_medium(Dispersive(2.25, [Pole.lorentz(1.0, 0.5, 0.01), Pole.drude(0.4, 0.02)]),
                      Boxes(0.0).add((-0.3, -0.2, -1.0), (0.1, 0.3, 1.0), 1.0))
    r = np.arange(s.grid.cells())
    for c in range(3):
        s.set_field(Field.E, Axis(c), noise(r + 11 * c))
        s.set_field(Field.H, Axis(c), noise(r + 13 * c + 7_000))
    return s


def fields(s):
    return [s.e(c) for c in range(3)] + [s.h(c) for c in range(3)]


W, L = Pml(0, 0), Pml(3, 4)
CASES = [((1, 9, 5), (W, L, W)), ((2, 9, 12), (Pml(0, 1), W, L)), ((3, 17, 5), (Pml(1, 0), Periodic(), W)),
         ((3, 9, 5), (W, W, W)), ((7, 9, 5), (W, W, W)), ((33, 9, 6), (L, L, W)), ((123, 8, 9), (L, Periodic(), L)),
         ((125, 15, 4), (L, W, Periodic())), ((126, 8, 9), (W, L, L)), ((249, 14, 3), (L, L, Periodic())),
         ((45, 30, 1), (Pml(20, 17), L, Periodic())), ((37, 21, 19), (L, L, L))]


@pytest.mark.parametrize("n,edges", CASES)
@pytest.mark.parametrize("lossy,media", [(False, False), (True, False), (True, True)])
def test_ragged_rows(monkeypatch, n, edges, lossy, media):
    from pyoracle import OracleSimulation
    d = stirred(lambda *q: Simulation(*q, precision=64), n, edges, lossy, media)  # the kernel it gets
    d.run(12)
    monkeypatch.setenv("PHOTONOXIDE_FDTD_KERNEL", "quad")
    a = stirred(lambda *q: Simulation(*q, precision=64), n, edges, lossy, media)
    o = stirred(lambda *q: OracleSimulation(*q, precision=64), n, edges, lossy, media)
    f = stirred(lambda *q: Simulation(*q, precision=32), n, edges, lossy, media)
    f.run(12)
    a.run(12)
    monkeypatch.setenv("PHOTONOXIDE_FDTD_KERNEL", "row")
    g = stirred(lambda *q: Simulation(*q, precision=32), n, edges, lossy, media)
    g.run(12)
    o.run(12)
    for x, y, z in zip(fields(a), fields(o), fields(d)):
        assert np.array_equal(x, y) and np.array_equal(z, y)
    for x, y in zip(fields(f), fields(g)):
        assert np.array_equal(x, y)


def test_sources_and_monitors_on_ragged_rows():
    """The busy scenario (sources, currents, a dipole, monitors) on rows of 37 and 131 places."""
    from pyoracle import OracleSimulation
    for n in ((37, 21, 19), (131, 24, 17)):
        a = busy(lambda *q: Simulation(*q, precision=64), False, n=n)
        o = busy(lambda *q: OracleSimulation(*q, precision=64), False, n=n)
        for s in (a, o):
            s.run(70)
        for x, y in zip(fields(a), fields(o)):
            assert np.array_equal(x, y)
        assert np.array_equal(a.transforms(), o.transforms())
        assert np.array_equal(a.probe(2), o.probe(2))
