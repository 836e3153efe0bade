"""Transforms read again and again, through plain memory at first and page-locked chunks once the reads come
to 8 MiB in all: the same sums as read once, but for the order of a few additions."""
import numpy as np
import pytest

from photonoxide_b200.fdtd import Simulation
from photonoxide_b200.types import Axis, Boundaries, Boxes, Field, Grid3d, Source, Waveform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(60, 50, 1), (301, 300, 1)])  # 36 000 doubles a read, and more than two chunks
def test_reads_come_to_the_same_sums(n):
    def make():
        s = Simulation(Grid3d.centred(n, 0.04), Boxes(2.0), Boundaries.cpml_2d(6), 0.7)
        s.add_source(Source(Field.H, Axis.Z, (n[0] // 2, n[1] // 2, 0), Waveform.pulse(1.0, 0.6)))
        s.add_dft((0, 0, 0), (n[0] - 1, n[1] - 1, 0), [0.9])
        return s

    a, b = make(), make()
    reads = 40
    for _ in range(reads):
        a.run(5)
        sums = a.transforms()
    b.run(5 * reads)
    want = b.transforms()
    assert np.any(want != 0)
    # each value's 200 terms in two groupings: at most 200 roundings of the sums' magnitudes
    assert np.max(np.abs(sums - want)) <= 200 * 2.0 ** -53 * 2 * np.max(np.abs(want)) * reads
