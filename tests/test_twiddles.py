"""The built table of stage rotations (cuopo_b200/build.py, csrc/fft.cuh): the
rotation of each entry, undone quarter turns added back, is W^{jk} to FP64
rounding (tan and sin correctly rounded up to one ulp: 2.5e-16 each, their
combination below 1e-15)."""
import numpy as np

from cuopo_b200 import build


def test_rotations_are_the_stage_twiddles():
    rows = np.array(build.twiddle_rows()).reshape(build.TW_NS, 6, 2)
    k = np.arange(build.TW_NS)
    assert np.all(np.abs(rows) <= 1.0)          # every angle within [-pi/2, pi/2]
    for j, mult in enumerate((1, 2, 3, 4, 8, 12)):
        quarter = 0 if j < 4 else 1 if j == 4 else np.where(2 * k < build.TW_NS, 1, 2)
        t, s = rows[:, j, 0], rows[:, j, 1]
        cos = 1.0 - t * s                       # the shears' first column: (1 - t s, s)
        got = (cos + 1j * s) * 1j ** quarter
        want = np.exp(2j * np.pi * ((mult * k) % (16 * build.TW_NS)) / (16 * build.TW_NS))
        assert np.max(np.abs(got - want)) < 1e-15
