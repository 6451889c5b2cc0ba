"""The viscoacoustic adjoint forms its products T1, T4 from the stress and memory adjoints with the residuals
already added (one rounding of the sum, as the transposed update is written): the gradient of a small case
equals, bit for bit, tests/golden/q_gradient_88x70.f32 -- d misfit / d vp, then d misfit / d (1/Q), from a
kernel that formed T1 and T4 where it differentiated them.  In both modes: the gradient does not depend on
SFD_EXACT."""
import os

import numpy as np
import pytest

from conftest import GOLDEN, bits_equal
from seismic_code_github_b200 import seisfd as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, S.EXACT], ids=["default", "exact"])
def test_gradient_bits(flags):
    rng = np.random.default_rng(3)
    nx, nz, npx, dt, f0 = 70, 52, 9, 5e-4, 20.0
    vp = S.pad_model((2000.0 + 40.0 * rng.standard_normal((nx, nz))).astype(np.float32), npx, npx, npx, npx)
    rho = S.pad_model((2100 + 100 * rng.random((nx, nz))).astype(np.float32), npx, npx, npx, npx)
    q = S.pad_model((30.0 + 50.0 * rng.random((nx, nz))).astype(np.float32), npx, npx, npx, npx)
    rx = np.arange(npx, vp.shape[0] - npx, dtype=np.int32)
    rz = np.full_like(rx, npx + 2)
    with S.Engine(S.VISCOAC_2D, vp.shape[0], vp.shape[1], 10.0, 10.0, dt, npx, order=10, f0=f0, flags=flags) as e:
        e.set_model(vp, rho, q)
        e.set_shots([S.ShotSpec(npx + 15 + 12 * i, npx + 3, rx, rz, S.wavelet(S.WAVELET_Q, 220 - 40 * i, dt, f0))
                     for i in range(2)])
        obs = (1e-6 * rng.standard_normal(e.record_size())).astype(np.float32)
        _, g, gq = e.gradient(obs, want_invq=True)
    want = np.fromfile(os.path.join(GOLDEN, "q_gradient_88x70.f32"), "<f4").reshape(2, *vp.shape)
    assert np.abs(want).max() > 0
    assert bits_equal(g, want[0]) and bits_equal(gq, want[1])
