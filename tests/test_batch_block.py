"""The batch's tiles of several steps a launch (112 x 16 of eight; 120 x 40 in f32 and 120 x 24 in f64
of four): every grid has the bits it has alone, at the tiles' edges, on grids that wrap within one tile's halo, with runs
that end within a launch, and through the adjoint's recomputed curls (tests/test_adjoint.py)."""
import numpy as np
import pytest

from photonoxide_b200.batch import Batch
from photonoxide_b200.fdtd import Simulation
from photonoxide_b200.types import Axis, Boundaries, Cpml, Field, Periodic, Pml
from test_batch import CASES, CASES4, general, same, te_busy

pytestmark = pytest.mark.gpu

P, C = Periodic(), Cpml(kappa=2.0, alpha=0.3)
EDGES = [
    ((33, 17), Boundaries(P, P, P, C)),                       # wraps several times in a region
    ((32, 16), Boundaries(P, Pml(3, 3), P, C)),
    ((112, 16), Boundaries(Pml(4, 4), P, P, C)),
    ((120, 24), Boundaries(Pml(9, 3), Pml(3, 5), P, C)),
    ((121, 25), Boundaries(Pml(5, 5), Pml(5, 5), P, C)),
    ((241, 49), Boundaries(P, P, P, C)),
    ((224, 33), Boundaries(Pml(0, 0), Pml(0, 0), P, C)),
    ((260, 48), Boundaries(Pml(30, 20), Pml(12, 20), P, C)),  # CPMLs wider than a halo
]


@pytest.mark.parametrize("tile,precision", [((112, 16), 32), ((120, 40), 32), ((112, 16), 64),
                                            ((120, 24), 64)])
def test_block_tiles_give_each_grids_own_bits(tile, precision):
    cases = CASES + CASES4 + EDGES
    a = [te_busy(Simulation, n, b, 11 * i, precision) for i, (n, b) in enumerate(cases)]
    o = [te_busy(general, n, b, 11 * i, precision) for i, (n, b) in enumerate(cases)]
    B = Batch(a, tile=tile)
    assert B.tile == tile
    for steps in (1, 7, 77, 64, 3):  # remainders of one to eight steps, odd numbers of launches
        B.run(steps)
    for s in o:
        s.run(152)
    for x, y in zip(a, o):
        same(x, y)


def test_a_grid_alone_between_batch_runs():
    a = [te_busy(Simulation, n, b, 3 * i, 32) for i, (n, b) in enumerate(EDGES[:4])]
    o = [te_busy(general, n, b, 3 * i, 32) for i, (n, b) in enumerate(EDGES[:4])]
    B = Batch(a, tile=(112, 16))
    B.run(40)  # five launches: the other copies are current when the grids step alone
    for s in a:
        s.run(6)
    B.run(41)
    for s in o:
        s.run(87)
    for x, y in zip(a, o):
        same(x, y)
    assert np.all(np.isfinite(a[0].e(0)))


@pytest.mark.parametrize("edges,precision", [(4, 32), (6, 32), (6, 64), (4, 64)])  # the last: too few cells
def test_a_te_run_alone_takes_the_same_tiles(edges, precision):
    """Simulation.run of a 2D TE grid, in runs long and short (16 steps on go to the tiles), fields
    set by the caller in between, against the general kernels."""
    n, b = EDGES[edges]
    a, o = te_busy(Simulation, n, b, 5, precision), te_busy(general, n, b, 5, precision)
    for steps in (40, 3, 17, 70):
        a.run(steps)
        o.run(steps)
    same(a, o)
    for s in (a, o):
        s.set_field(Field.E, Axis.Z, np.full(n[0] * n[1], 0.01))  # no longer TE
        s.run(40)
    same(a, o)


@pytest.mark.parametrize("precision", [32, 64])
def test_many_small_grids_time_the_shapes(precision):
    """Grids that fill a third of a tile, too many for the tiles to be few: the first run of 320 steps or
    more times every shape on steps of its own, with probes and transforms; a shorter one takes a shape
    by the sizes. The bits of each grid alone."""
    n, b = EDGES[0]
    for steps in (330, 40):
        a = [te_busy(Simulation, n, b, 5 * i, precision) for i in range(200)]
        B = Batch(a)
        B.run(steps)
        B.run(21)
        for i in (0, 77, 199):
            o = te_busy(general, n, b, 5 * i, precision)
            o.run(steps + 21)
            same(a[i], o)
