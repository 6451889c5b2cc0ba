"""The 2-D gradients when memory is short: with no room for kept derivatives every segment is recomputed from
its checkpoint, and misfit and gradients equal those with everything kept bit for bit -- with a last
segment shorter than the others too; the viscoacoustic checkpoints hold the eight fields of the reference's
state (sigma is formed from them)."""
import numpy as np
import pytest

from conftest import bits_equal, rel_l2
from seismic_code_github_b200 import seisfd as S

pytestmark = pytest.mark.gpu


def engine(kind, nx, nz, pml, nts, flags=0):
    rng = np.random.default_rng(nx)
    vp = (2000.0 + 300.0 * rng.random((nx, nz))).astype(np.float32)
    den = (1900.0 + 300.0 * rng.random((nx, nz))).astype(np.float32)
    q = (30.0 + 60.0 * rng.random((nx, nz))).astype(np.float32)
    visco = kind == "visco"
    dt = 5e-4 if visco else 1e-3
    e = S.Engine(S.VISCOAC_2D if visco else S.ACOUSTIC_2D, nx, nz, 10.0, 10.0, dt, pml, order=10, flags=flags, f0=20.0)
    e.set_model(vp, den, q if visco else None)
    rx, rz = np.arange(pml, nx - pml, dtype=np.int32), np.full(nx - 2 * pml, pml + 3, np.int32)
    e.set_shots([S.ShotSpec(nx // 2 - 5 * i, pml + 5, rx, rz,
                            S.wavelet(S.WAVELET_Q, nt, dt, 20.0) if visco else S.wavelet(S.WAVELET_RIC, nt, dt, 25.0, 20))
                 for i, nt in enumerate(nts)])
    return e


@pytest.mark.parametrize("kind,flags", [("acoustic", 0), ("visco", 0), ("visco", S.EXACT)])
@pytest.mark.parametrize("interval", [7, 12, 17, 60])
def test_recomputed_segments_equal_kept_ones(kind, flags, interval):
    visco = kind == "visco"
    out = []
    for limit in (0, 1):
        with engine(kind, 90, 70, 8, (60, 41, 52), flags) as e:
            e.set_memory_limit(limit)
            obs = np.zeros(e.record_size(), np.float32)
            e.set_checkpoint_interval(interval)
            for per_shot in (False, True):
                out.append(e.gradient(obs, want_invq=visco, per_shot=per_shot) + (e.timing()["point_updates"],))
    assert out[2][3] > out[0][3]  # recomputed
    for j, g, gq, _ in out[1:]:
        assert np.abs(g).max() > 0 and rel_l2(j, out[0][0]) <= 1e-6 and bits_equal(g, out[0][1])
        assert not visco or bits_equal(gq, out[0][2])


def test_viscoacoustic_checkpoints_hold_eight_fields():
    import torch
    nx = nz = 300
    nt, nshot = 64, 8
    with engine("visco", nx, nz, 8, (nt,) * nshot, S.EXACT) as e:
        e.set_memory_limit(1)
        e.forward()
        obs = np.zeros(e.record_size(), np.float32)
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info()[0]
        e.gradient(obs)
        used = free0 - torch.cuda.mem_get_info()[0]
    # slabs of the 64 x 64 tiles with margins of 8 columns and 8 rows, rows rounded to 32 floats: eight
    # checkpoints, 12 adjoint fields, two imaging sums in float and double, two derivatives per step of a segment
    slab = 4 * nshot * (8 + 320 + 8) * 352
    assert used <= (8 * 8 + 12 + 2 + 4 + 2 * 8) * slab + (16 << 20)
