"""Which step kernels a 2-D acoustic call launches, counted with the CUDA activity of torch's profiler."""
import numpy as np
import pytest

from conftest import bits_equal
from seismic_code_github_b200 import seisfd as S

pytestmark = pytest.mark.gpu


def launched(call):
    """Step kernels launched by call(), by kernel name: {"small" | "tile" | "march": launches}."""
    import torch
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        call()
        torch.cuda.synchronize()
    out = {}
    for ev in prof.events():
        for key, name in (("small", "acoustic2d_small_kernel"), ("tile", "acoustic2d_step_fma_kernel"),
                          ("march", "acoustic2d_march_kernel")):
            if name in ev.name:
                out[key] = out.get(key, 0) + 1
    return out


def engine(nx, nz, order, nshot, nt, varden=False):
    rng = np.random.default_rng(nx)
    vp = (2000.0 + 600.0 * rng.random((nx, nz))).astype(np.float32)
    den = (1900.0 + 300.0 * rng.random((nx, nz))).astype(np.float32) if varden else None
    rx, rz = np.arange(10, nx - 10, dtype=np.int32), np.full(nx - 20, 12, np.int32)
    w = S.wavelet(S.WAVELET_RIC, nt, 1e-3, 25.0, 20)
    e = S.Engine(S.ACOUSTIC_2D, nx, nz, 10.0, 10.0, 1e-3, 10, order=order)
    e.set_model(vp, den)
    e.set_shots([S.ShotSpec(nx // 2 + 3 * i, 14, rx, rz, w) for i in range(nshot)])
    return e, vp


@pytest.fixture(autouse=True)
def no_switches(monkeypatch):
    for k in ("SFD_FMA_STAGES", "SFD_MARCH_SEG"):
        monkeypatch.delenv(k, raising=False)


def test_schedules_are_timed_once_per_shot_set():
    """A caller that only takes gradients: the candidate kernels are timed on the first call, not on the
    second, not after a model update; the gradients agree bit for bit."""
    nt = 30
    e, vp = engine(500, 400, 16, 4, nt)  # 8 x 7 tiles a shot
    with e:
        obs = np.zeros(e.record_size(), np.float32)
        e.set_checkpoint_interval(nt)
        grads, counts = [], []
        for scale in (1.0, 1.0, 1.01):
            if scale != 1.0:
                e.set_model((vp * scale).astype(np.float32))
            counts.append(launched(lambda: grads.append(e.gradient(obs)[1])))
        n = [sum(c.values()) for c in counts]
        assert bits_equal(grads[0], grads[1]) and not bits_equal(grads[1], grads[2])
    assert n[0] > n[1] == n[2]
    assert 2 * nt <= n[1] <= 3 * nt  # forward, adjoint, and the recomputation of what is not kept


@pytest.mark.parametrize("order,varden", [(16, False), (8, True)])
def test_small_tiles_run_untimed_in_one_wave_only(monkeypatch, order, varden):
    """Up to one wave of its CTAs (92 tiles of 64 x 64 on 148 SMs) the small-tile kernel runs alone, forward
    and gradient; beyond it (110 and 143 tiles) it is one candidate among those that are timed.  The
    records equal those of a pinned schedule, which never runs it, bit for bit."""
    nt = 20
    for tx, tz in ((10, 9), (11, 10), (13, 11)):
        recs = []
        for pin in (None, "2"):
            monkeypatch.delenv("SFD_FMA_STAGES", raising=False)
            if pin:
                monkeypatch.setenv("SFD_FMA_STAGES", pin)
            e, _ = engine(64 * tx - 3, 64 * tz, order, 1, nt, varden)
            with e:
                first = launched(lambda: recs.append(e.forward().copy()))
                grad = launched(lambda: e.gradient(np.zeros(e.record_size(), np.float32)))
            if pin:
                assert first == {"tile": nt} and set(grad) == {"tile"}
            elif tx * tz <= 92:
                assert first == {"small": nt} and set(grad) == {"small"}
            else:
                assert first["small"] >= 20 and first["tile"] >= 40
        assert np.abs(recs[0]).max() > 0 and bits_equal(recs[0], recs[1])
