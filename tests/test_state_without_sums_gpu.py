"""The split schemes on a device without memory for the slabs of the sums that their kernels stage: a batch
whose split parts fit is accepted, its kernels sum the parts themselves, and records, wavefields, snapshots
and (viscoacoustic) gradients equal those with the slabs bit for bit."""
import numpy as np
import pytest

from conftest import bits_equal
from seismic_code_github_b200 import seisfd as S
from test_out_of_memory_gpu import Hog

pytestmark = pytest.mark.gpu

SLABS = {"visco": (8, 9), "viscoel": (22, 27), "elastic": (10, 15), "elastic_abc": (10, 15)}  # without, with
NX, NZ, PML, NSHOT, NT = 250, 190, 10, 256, 24


def prepare(kind):
    rng = np.random.default_rng(3)
    vp = (2000.0 + 300.0 * rng.random((NX, NZ))).astype(np.float32)
    den = (1900.0 + 300.0 * rng.random((NX, NZ))).astype(np.float32)
    q = (30.0 + 60.0 * rng.random((NX, NZ))).astype(np.float32)
    scheme = {"visco": S.VISCOAC_2D, "viscoel": S.VISCOEL_2D}.get(kind, S.ELASTIC_2D)
    e = S.Engine(scheme, NX, NZ, 5.0, 5.0, 5e-4, PML, order=10, flags=S.EXACT if kind == "visco" else 0, f0=20.0)
    if kind.startswith("elastic"):
        e.set_gauss_radius(6)
        if kind == "elastic":
            e.set_free_surface(PML)
            e.set_topography((PML + 4 + np.round(3 * np.sin(np.arange(NX) / 20))).astype(np.int32))
    if kind == "visco":
        e.set_model(vp, den, q)
    else:
        e.set_model_elastic(vp, vp / np.float32(1.8), den, *((q, q) if kind == "viscoel" else ()))
    rx = np.arange(PML, NX - PML, dtype=np.int32)
    rz = np.full(rx.size, PML + 9, np.int32)
    w = S.wavelet(S.WAVELET_Q, NT, 5e-4, 20.0)
    return e, [S.ShotSpec(PML + 20 + i % 200, PML + 12, rx, rz, w[:NT - i % 7]) for i in range(NSHOT)]


def results(e, kind):
    e.set_snapshots(0, S.FIELD_VX, 7, 8, 2)
    out = [e.forward().copy(), e.snapshots(0, 5).copy(), e.wavefield(1, S.FIELD_P), e.wavefield(2, S.FIELD_VZ)]
    if kind == "viscoel":
        out.append(e.records(S.FIELD_P).copy())
    if kind.startswith("elastic"):
        out.append(e.records(S.FIELD_VZ).copy())
    e.set_snapshots(0, S.FIELD_VX, 0, 1, 0)
    return out


def sums_kept(call):
    """Whether the step kernels that call() launches stage the slabs of the sums (their last template argument)."""
    import torch
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        call()
        torch.cuda.synchronize()
    names = {ev.name for ev in prof.events() if "velocity_kernel<" in ev.name}
    assert len(names) == 1
    return names.pop().split("velocity_kernel<")[1].split(">")[0].endswith("true")


@pytest.mark.parametrize("kind", list(SLABS))
def test_batch_of_the_split_parts(kind):
    slab = 4 * NSHOT * (8 + 256 + 8) * 224
    few, many = SLABS[kind]
    out = []
    for short in (False, True):
        e, shots = prepare(kind)
        with e:
            if short:  # memory for the records and half of the sums' slabs
                rec = 4 * NSHOT * (NX - 2 * PML) * NT
                hog = Hog((few + many) * slab // 2 + rec * (2 if kind == "visco" else 4))
            try:
                e.set_shots(shots)
            finally:
                if short:
                    hog.release()
            assert sums_kept(e.forward) == (not short)
            out.append(results(e, kind))
            if kind == "visco":
                e.set_memory_limit(1 if short else 0)  # short: every segment recomputed from its checkpoint
                out[-1] += list(e.gradient(np.zeros(e.record_size(), np.float32), want_invq=True)[1:])
    assert len(out[0]) == len(out[1])
    for a, b in zip(*out):
        assert np.abs(b).max() > 0 and bits_equal(a, b)
