"""The VTI survey call on a device with room for the shots' fields but not for a copy of the model beside them:
the same records bit for bit, apertures over the model's edges included."""
import numpy as np
import pytest

from conftest import bits_equal
from seismic_code_github_b200 import seisfd as S
from test_out_of_memory_gpu import Hog
from test_vti_gpu import model

pytestmark = pytest.mark.gpu


def test_windows_without_a_copy_of_the_model():
    vz, eps, de = model(3000, 1500, seed=8)  # 52 MB in three arrays
    shots = [(x, 1, 1, x - 150, x + 149) for x in (20, 1400, 2990)]
    args = (5.0, 5.0, 5e-4, 30.0, 20, (20, 20, 6, 20))
    want, t = S.vti_forward(vz, eps, de, *args, shots, exact=True)
    assert t["h2d_bytes"] == 12 * vz.size and np.abs(want).max() > 0
    pitch, rows = 416, 1524  # 338 columns: six tiles of 64 and margins; rows with the stencil's
    slab = 4 * 7 * pitch * (rows + 10)
    hog = Hog(3 * slab + (12 << 20) + 4 * 3 * (14 * 40 * rows + 8 * 340 * 26))
    try:
        got, t = S.vti_forward(vz, eps, de, *args, shots, exact=True)
    finally:
        hog.release()
    assert t["h2d_bytes"] < 12 * vz.size  # the shots' columns only
    assert bits_equal(got, want)
