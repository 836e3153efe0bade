"""2D TE grids whose CPML reaches past the middle, along x and along y: a place belongs to the CPML
whose ends hold it, wherever the grid's middle is. The engine alone, the batch on every tile shape and
the adjoint against the oracle."""
import math

import numpy as np
import pytest
import torch

from photonoxide_b200.adjoint import Design2d, TeFlux, TeProblem, central_differences
from photonoxide_b200.batch import Batch
from photonoxide_b200.fdtd import Simulation, average
from photonoxide_b200.types import (INF, Axis, Boundaries, Boxes, Cpml, Current, Field, FluxPlane,
                                    Grid3d, Periodic, Pml, Source, Waveform)
from pyoracle import OracleSimulation
from scenarios import noise, pulse

pytestmark = pytest.mark.gpu

P = Periodic()
CASES = [((60, 40), Pml(35, 5), Pml(4, 4)), ((40, 60), Pml(4, 4), Pml(35, 5)),
         ((20, 33), Pml(12, 0), P), ((33, 20), P, Pml(12, 0)),
         ((20, 21), Pml(0, 12), Pml(11, 5)), ((21, 20), Pml(11, 5), Pml(0, 12)),
         ((260, 50), Pml(150, 20), Pml(3, 30))]
STEPS = 45


def te(make, case, precision):
    n, x, y = case
    s = make(Grid3d.centred((n[0], n[1], 1), 0.05), Boxes(1.0).add((-0.4, -0.2, -INF), (0.3, 0.25, INF), 9.0),
             Boundaries(x, y, P, Cpml(kappa=2.0, alpha=0.3)), 0.9, precision=precision)
    r = np.arange(s.grid.cells())
    s.set_field(Field.E, 0, 0.01 * noise(r + 5))
    s.set_field(Field.E, 1, 0.01 * noise(r + 17))
    s.set_field(Field.H, 2, 0.01 * noise(r + 50_000))
    s.add_source(Source(Field.H, Axis.Z, (n[0] // 2, n[1] // 2, 0), pulse()))
    return s


def fields(s):
    return [s.e(0), s.e(1), s.h(2)]


@pytest.fixture(scope="module")
def oracles():
    out = {}
    for precision in (32, 64):
        for q, case in enumerate(CASES):
            o = te(OracleSimulation, case, precision)
            o.run(STEPS)
            out[precision, q] = fields(o)
    return out


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("q", range(len(CASES)))
def test_a_run_alone(oracles, q, precision):
    s = te(Simulation, CASES[q], precision)
    s.run(STEPS)
    for x, y in zip(fields(s), oracles[precision, q]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("tile,precision", [(t, 32) for t in ((32, 8), (64, 8), (128, 4), (124, 7),
                                                              (112, 16), (120, 40))]
                         + [((64, 4), 64), ((124, 7), 64), ((112, 16), 64), ((120, 24), 64)])
def test_a_batch(oracles, tile, precision):
    sims = [te(Simulation, case, precision) for case in CASES]
    Batch(sims, tile=tile).run(STEPS)
    for q, s in enumerate(sims):
        for x, y in zip(fields(s), oracles[precision, q]):
            assert np.array_equal(x, y)


def design(steps, segment, cls=None):
    """An 8 x 8 design between a source and a flux plane, the x CPML 35 of 60 places from the left and
    the y CPML 24 of 44 from the top; a transform of the whole plane, whose sums the objective leaves
    alone."""
    h = 0.02
    g = Grid3d.centred((60, 44, 1), h)
    background = average(g, Boxes(2.25))

    def build(eps, precision):
        s = (cls or Simulation)(g, eps, Boundaries(Pml(35, 5), Pml(6, 24), P, Cpml()), 0.5, precision=precision)
        s.add_current(Current(Field.E, [(Axis.Y, (37, j, 0), complex(math.exp(-((j - 13) / 5.0) ** 2)))
                                        for j in range(8, 19)], Waveform.pulse(2.0, 1.5)))
        s.add_flux(FluxPlane(Axis.X, 51, ((7, 18), None)), [2.0])
        s.add_dft((0, 0, 0), (59, 43, 0), [2.0])
        return s

    return TeProblem(g, background, Design2d(40, 9, 8, 8), build, steps, precision=64, segment=segment)


def gradient(p, eps):
    e = torch.tensor(eps, requires_grad=True)
    flux = TeFlux.apply(e, p)
    flux[0].backward()
    return float(flux[0].detach()), e.grad.numpy().copy()


def test_the_adjoint():
    eps = 2.25 + np.random.default_rng(2).uniform(0.0, 4.0, (8, 8))
    steps = 900
    J, g = gradient(design(steps, 200), eps)
    o = design(steps, 200, OracleSimulation)

    def objective(e):
        s = o.simulation(e)
        s.run(steps)
        return float(s.flux(0)[0])

    assert J == objective(eps)
    pixels = np.random.default_rng(7).choice(64, 4, replace=False)
    fd = central_differences(objective, eps, pixels, 1e-3)
    ga = g.reshape(-1)[pixels]
    # as in the adjoint's other check by central differences
    assert np.linalg.norm(ga - fd) <= 1e-3 * np.linalg.norm(fd), (ga, fd)


def test_the_reverse_by_tiles_and_step_by_step():
    """A segment whose amounts take more than the tiles' 256 MB (7920 transform values and the flux
    plane's, 8 bytes, 4600 steps) goes back step by step: the same bits."""
    eps = 2.25 + np.random.default_rng(3).uniform(0.0, 4.0, (8, 8))
    _, a = gradient(design(4600, 100), eps)
    _, b = gradient(design(4600, 4600), eps)
    assert np.array_equal(a, b)
