"""Many sources on a row: currents over whole rows and tile edges, two on the same values, as a
plane wave's box or a Bloch side gives them. The quad kernel, and the row kernel (rows that are no whole
vectors, narrow or wrapped), take a row's values a lane each, more than 32 in turn; in f64 every value is the oracle's bits, in f32 within the reference's GPU tolerance
(2e-5 of the largest value, src/fdtd/gpu/tests.rs:51-66)."""
import numpy as np
import pytest

from photonoxide_b200.fdtd import Simulation
from photonoxide_b200.types import (Axis, Boundaries, Boxes, Cpml, Current, Field, Grid3d, Periodic,
                                    Pml, Waveform)

pytestmark = pytest.mark.gpu


def problem(make, n, periodic, lossy):
    b = Boundaries(Periodic() if periodic else Pml(3, 4), Periodic() if periodic else Pml(3, 3),
                   Pml(2, 2), Cpml(kappa=2.0, alpha=0.1))
    s = make(Grid3d.centred(n, 0.05), Boxes(2.25), b, 0.8)
    if lossy:
        s.with_conductivity(Boxes(0.5))
    w = Waveform.pulse(1.0, 0.8)
    nx, ny, nz = n
    rows = [(c, (i, j, k)) for c in range(3) for j in (0, 6, 7, ny - 1) for k in (0, nz // 2)
            for i in range(nx)]
    for field in (Field.E, Field.H):
        for scale in (1.0, -0.4):
            s.add_current(Current(field, [(Axis(c), at, complex(scale * (1 + 0.01 * q), 0.2))
                                          for q, (c, at) in enumerate(rows)], w))
    return s


@pytest.mark.parametrize("n", [(4, 8, 5), (128, 15, 6), (252, 9, 5), (27, 15, 6), (131, 9, 5)])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("precision,lossy", [(64, False), (64, True), (32, False), (32, True)])
def test_rows_of_sources_match_the_oracle(n, periodic, precision, lossy):
    from pyoracle import OracleSimulation
    if n[0] == 4 and not periodic:
        n = (12, 8, 5)  # room for the CPMLs
    a = problem(lambda *q: Simulation(*q, precision=precision), n, periodic, lossy)
    b = problem(lambda *q: OracleSimulation(*q, precision=64), n, periodic, lossy)
    a.run(25)
    b.run(25)
    for f in ("e", "h"):
        for c in range(3):
            x, y = getattr(a, f)(c), getattr(b, f)(c)
            if precision == 64:
                assert np.array_equal(x, y)
            else:
                assert np.max(np.abs(x - y)) <= 2e-5 * np.max(np.abs(y))
