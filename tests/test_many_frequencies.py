"""A transform of more frequencies than a launch has rows for (65 535 times eight): every frequency's sums,
on the general kernels and on the TE tiles."""
import numpy as np
import pytest

from photonoxide_b200.fdtd import Simulation
from photonoxide_b200.types import Axis, Boundaries, Boxes, Field, Grid3d, Source, Waveform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["tiles", "quad"])
def test_half_a_million_frequencies(monkeypatch, kernel):
    if kernel == "quad":
        monkeypatch.setenv("PHOTONOXIDE_FDTD_KERNEL", "quad")
    count = 65535 * 8 + 11
    freqs = np.linspace(0.5, 2.0, count)

    def make(f):
        s = Simulation(Grid3d.centred((40, 30, 1), 0.04), Boxes(2.0), Boundaries.cpml_2d(6), 0.7)
        s.add_source(Source(Field.H, Axis.Z, (20, 15, 0), Waveform.pulse(1.0, 0.6)))
        s.add_dft((22, 15, 0), (22, 15, 0), list(f))
        s.run(40)
        return s.transforms().reshape(6, -1)

    some = np.r_[0:9, count // 2, count - 20:count]
    all_of, few = make(freqs), make(freqs[some])
    assert np.any(few != 0)
    assert np.array_equal(all_of[:, some], few)
