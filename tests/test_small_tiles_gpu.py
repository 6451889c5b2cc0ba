"""The small-tile step kernel (16 x 32 tiles), which every launch with fewer 64 x 64 tiles than SMs runs,
gives the tile kernel's bits, forward and gradient: every order, constant and variable density, widths and
depths around the multiples of its tile, apertures, a source next to the rim, shared receiver cells; and
the records stay within the tolerance of test_acoustic_gpu against the FP64 oracle."""
import numpy as np
import pytest

import oracle_lib as ol
from conftest import bits_equal, rel_l2
from seismic_code_github_b200 import seisfd as S

pytestmark = pytest.mark.gpu


def run(monkeypatch, stages, vp, den, pml, shots, order):
    monkeypatch.delenv("SFD_MARCH_SEG", raising=False)
    if stages:
        monkeypatch.setenv("SFD_FMA_STAGES", stages)
    else:
        monkeypatch.delenv("SFD_FMA_STAGES", raising=False)
    with S.Engine(S.ACOUSTIC_2D, vp.shape[0], vp.shape[1], 10.0, 12.0, 1e-3, pml, order=order) as e:
        e.set_model(vp, den)
        e.set_shots(shots)
        e.set_snapshots(0, S.FIELD_P, 20, 30, 2)
        rec = e.forward().copy()
        snap = e.snapshots(0, 0).copy()
        v = [e.wavefield(0, f) for f in (S.FIELD_P, S.FIELD_VX, S.FIELD_VZ)]
        e.set_snapshots(0, S.FIELD_P, 0, 1, 0)
        e.set_model((vp * 1.01).astype(np.float32), den)
        e.set_checkpoint_interval(17)
        J, g, _ = e.gradient(rec)
        wg = e.wavelet_gradient(0)
    return rec, snap, v, J, g, wg


@pytest.mark.parametrize("order,nx,nz,varden", [(16, 47, 64, False), (16, 65, 33, True), (10, 49, 97, True),
                                                (8, 80, 96, False), (8, 63, 95, True), (4, 33, 31, True),
                                                (2, 129, 40, False)])
def test_small_tiles_equal_the_tile_kernel(monkeypatch, order, nx, nz, varden):
    pml, nt = 10, 70
    rng = np.random.default_rng(nx)
    vp = (2000.0 + 800.0 * rng.random((nx, nz))).astype(np.float32)
    den = (1900.0 + 400.0 * rng.random((nx, nz))).astype(np.float32) if varden else None
    R = order // 2
    w = S.wavelet(S.WAVELET_RIC, nt, 1e-3, 25.0, 25)
    rx = np.r_[np.arange(nx), [nx // 2, nx // 2]].astype(np.int32)
    rz = np.r_[np.full(nx, min(nz - 1, 12)), [nz // 2, nz // 2]].astype(np.int32)  # two receivers share a cell
    ap = max(2 * pml + 1, 2 * R + 1, nx - 7)
    shots = [S.ShotSpec(nx // 2, nz // 2, rx, rz, w),
             S.ShotSpec(min(R, ap - 1), min(R, nz - 1), rx[:ap], rz[:ap], w[:50], ap_x0=nx - ap, ap_nx=ap)]
    a = run(monkeypatch, None, vp, den, pml, shots, order)
    b = run(monkeypatch, "1", vp, den, pml, shots, order)
    assert np.abs(b[0]).max() > 0 and np.abs(b[4]).max() > 0
    assert bits_equal(a[0], b[0]) and bits_equal(a[1], b[1])
    for x, y in zip(a[2], b[2]):
        assert bits_equal(x, y)
    assert a[3] == b[3] and bits_equal(a[5], b[5])
    assert rel_l2(a[4], b[4]) <= 1e-6  # the residuals of a shared receiver cell add in either order
    d = den if varden else np.full_like(vp, 2400.0)
    ref, _, _ = ol.afd_forward(nx, nz, pml, nt, 10.0, 12.0, 1e-3, vp, d, w, nx // 2, nz // 2, rx, rz, radius=R)
    assert rel_l2(a[0][:len(rx) * nt].reshape(len(rx), nt), ref) <= 1e-5


@pytest.mark.parametrize("order,nx,nz,varden", [(16, 47, 64, True), (16, 65, 33, False), (10, 49, 97, True),
                                                (8, 80, 31, True), (4, 33, 95, False), (2, 129, 40, True)])
def test_reference_order_tile_edges(order, nx, nz, varden):
    """SFD_EXACT on the same tiles, and the same kernel reading a caller's unpadded model
    (sfd_forward_noalloc), bit for bit against the oracle."""
    import ctypes
    import torch
    pml, nt = 8, 60
    rng = np.random.default_rng(order + nx)
    vp = (2000.0 + 800.0 * rng.random((nx, nz))).astype(np.float32)
    den = (1900.0 + 400.0 * rng.random((nx, nz))).astype(np.float32) if varden else None
    w = S.wavelet(S.WAVELET_RIC, nt, 1e-3, 25.0, 25)
    rx, rz = np.arange(nx, dtype=np.int32), np.full(nx, min(nz - 1, 13), np.int32)
    ref, _, _ = ol.afd_forward(nx, nz, pml, nt, 10.0, 12.0, 1e-3, vp, den if varden else np.full_like(vp, 2400.0), w,
                               nx // 2, nz // 2, rx, rz, radius=order // 2)
    with S.Engine(S.ACOUSTIC_2D, nx, nz, 10.0, 12.0, 1e-3, pml, order=order, flags=S.EXACT) as e:
        e.set_model(vp, den)
        e.set_shots([S.ShotSpec(nx // 2, nz // 2, rx, rz, w)])
        rec = e.forward().reshape(nx, nt)
    assert np.abs(ref).max() > 0 and bits_equal(rec, ref)
    g = S.Grid(S.ACOUSTIC_2D, nx, 1, nz, pml, 10.0, 0.0, 12.0, 1e-3, order, S.EXACT, 0.0)
    dev = [None if a is None else torch.from_numpy(a).cuda() for a in (vp, den, w)]
    out = torch.zeros(nx * nt, device="cuda")
    torch.cuda.synchronize()
    rc = S.load().sfd_forward_noalloc(ctypes.byref(g), dev[0].data_ptr(), None if den is None else dev[1].data_ptr(),
                                      dev[2].data_ptr(), nt, nx // 2, nz // 2, nx, S._ip(rx), S._ip(rz), out.data_ptr(), None)
    assert rc == 0 and bits_equal(out.cpu().numpy().reshape(nx, nt), ref)
