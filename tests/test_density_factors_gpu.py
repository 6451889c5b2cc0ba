"""3-D variable density without memory for the factors dt / (d den): the model, the shots and the gradient that
fit without them are accepted, the step divides by the density itself, and records and gradients are the
same bit for bit (the gradient's schedule is fixed by the memory limit)."""
import numpy as np
import pytest

from conftest import bits_equal
from seismic_code_github_b200 import seisfd as S
from test_out_of_memory_gpu import Hog

pytestmark = pytest.mark.gpu

N, NT, PML = (280, 256, 240), 24, 8
SLAB = 4 * N[0] * N[1] * N[2]  # 66 MB: more than the driver may have left over in blocks it already holds


def divides(call):
    """Whether the 3-D steps that call() launches divide by the density (template argument kDivide = 2)."""
    import torch
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        call()
        torch.cuda.synchronize()
    names = {ev.name.split("acoustic3d_step_kernel<")[1].split(">")[0] for ev in prof.events()
             if "acoustic3d_step_kernel<" in ev.name}
    kinds = {n.split(",")[1].strip()[-1] for n in names}
    assert len(kinds) == 1 and kinds <= {"1", "2"}, names
    return kinds == {"2"}


@pytest.mark.parametrize("order,dy", [(8, 10.0), (4, 12.0)])
def test_steps_without_the_factors(order, dy):
    rng = np.random.default_rng(order)
    vp = (2000.0 + 300.0 * rng.random(N)).astype(np.float32)
    den = (1900.0 + 300.0 * rng.random(N)).astype(np.float32)
    rx = np.arange(20, 250, dtype=np.int32)
    w = S.wavelet(S.WAVELET_RIC, NT, 1e-3, 25.0, 12)
    shots = [S.ShotSpec(80 + 4 * i, PML + 4, rx, np.full(rx.size, PML + 4, np.int32), w, sy=70,
                        rec_y=np.full(rx.size, 70, np.int32)) for i in range(2)]
    out = []
    for short in (None, "model", "shots"):
        with S.Engine(S.ACOUSTIC_3D, N[0], N[2], 10.0, 10.0, 1e-3, PML, order=order, ny=N[1], dy=dy) as e:
            hog = Hog(2 * SLAB + SLAB // 2) if short == "model" else None  # vp and den
            try:
                e.set_model(vp, den)
            finally:
                if hog:
                    hog.release()
            hog = Hog(8 * 2 * SLAB - SLAB // 2) if short == "shots" else None  # eight slabs a shot
            try:
                e.set_shots(shots)
            finally:
                if hog:
                    hog.release()
            rec = e.forward().copy()
            # one shot a group, one level of checkpoints: 19 + 6 + 4 * 4 slabs, and the fixed buffers
            e.set_checkpoint_interval(6)
            e.set_memory_limit(41 * SLAB + SLAB // 2 + 8 * (SLAB // 4) + 16 * e.record_size() + 4 * 2 * NT)
            obs = np.zeros(e.record_size(), np.float32)
            kept = not divides(lambda: e.forward())
            assert kept == (short is None)
            out.append((rec, e.gradient(obs)[1].copy()))
    for rec, g in out[1:]:
        assert np.abs(rec).max() > 0 and np.abs(g).max() > 0
        assert bits_equal(rec, out[0][0]) and bits_equal(g, out[0][1])
