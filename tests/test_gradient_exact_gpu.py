"""The gradient of an SFD_EXACT acoustic context.  Its forwards run the reference's rounding order, its
gradient the default kernels, so misfit, gradient and wavelet gradient equal those of a default context
bit for bit: constant and variable density, equal and unequal spacings, every schedule of the step
kernels, host, device and per-shot calls, and again after a model update."""
import numpy as np
import pytest

from conftest import bits_equal, rel_l2
from seismic_code_github_b200 import seisfd as S
from test_gradient_device_gpu import device_gradient

pytestmark = pytest.mark.gpu


def gradients(flags, vp, den, dz, order, shots, obs):
    out = []
    with S.Engine(S.ACOUSTIC_2D, vp.shape[0], vp.shape[1], 10.0, dz, 1e-3, 10, order=order, flags=flags) as e:
        e.set_model(vp, den)
        e.set_shots(shots)
        e.set_checkpoint_interval(13)
        for scale in (1.0, 1.01):  # the second pass after an update of the model in place
            e.set_model((vp * scale).astype(np.float32), None if den is None else (den * scale).astype(np.float32))
            out.append(e.gradient(obs)[:2] + (e.wavelet_gradient(0),))
            out.append(e.gradient(obs, per_shot=True)[:2] + (e.wavelet_gradient(0),))
            out.append(device_gradient(e, obs, vp.shape)[:2] + (e.wavelet_gradient(0),))
    return out


@pytest.mark.parametrize("switch", [{}, {"SFD_FMA_STAGES": "1"}, {"SFD_FMA_STAGES": "2"}, {"SFD_MARCH_SEG": "128"}],
                         ids=["default", "tile", "persistent", "march"])
@pytest.mark.parametrize("order,nx,nz,dz,varden", [(16, 131, 70, 10.0, True), (8, 67, 97, 12.0, True),
                                                   (16, 90, 65, 12.0, False)])
def test_gradient_of_an_exact_context(monkeypatch, switch, order, nx, nz, dz, varden):
    for k in ("SFD_FMA_STAGES", "SFD_MARCH_SEG"):
        monkeypatch.delenv(k, raising=False)
    for k, v in switch.items():
        monkeypatch.setenv(k, v)
    rng = np.random.default_rng(nx)
    vp = (2000.0 + 600.0 * rng.random((nx, nz))).astype(np.float32)
    den = (1900.0 + 400.0 * rng.random((nx, nz))).astype(np.float32) if varden else None
    w = S.wavelet(S.WAVELET_RIC, 60, 1e-3, 25.0, 25)
    rx, rz = np.arange(10, nx - 10, dtype=np.int32), np.full(nx - 20, 13, np.int32)
    shots = [S.ShotSpec(nx // 2, nz // 2, rx, rz, w), S.ShotSpec(nx // 3, 14, rx[:30], rz[:30], w[:47])]
    obs = rng.standard_normal(len(rx) * 60 + 30 * 47).astype(np.float32)
    got, want = (gradients(f, vp, den, dz, order, shots, obs) for f in (S.EXACT, 0))
    for (j, g, wg), (j0, g0, wg0) in zip(got, want):
        assert np.abs(g0).max() > 0 and np.abs(wg0).max() > 0
        assert rel_l2(j, j0) <= 1e-6  # the misfit's double sum is formed in any order
        assert bits_equal(g, g0) and bits_equal(wg, wg0)
