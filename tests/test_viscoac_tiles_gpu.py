"""The reference-order viscoacoustic kernels and their adjoint work on tiles of 64 rows by 8 columns, two
cells per thread: padded widths and depths around their multiples, the forward bit for bit against the
FP32 restatement, the gradient (with receivers that share a cell in a sponge corner) against the FP64
adjoint oracle within the tolerance of test_q_gradient_gpu."""
import numpy as np
import pytest

import oracle_lib as ol
from conftest import bits_equal, rel_l2
from test_q_gradient_gpu import DT, NPX, TOL_GRAD, engine, model, observed, oracle
from test_viscoac_gpu import TOL_FAST, qmodel, run_gpu
from seismic_code_github_b200 import seisfd as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(28, 44), (29, 45), (35, 43), (31, 107), (36, 108)])
def test_forward_tile_edges(nx, nz):
    vp, rho, q = qmodel(nx=nx, nz=nz, seed=nx)
    npx, f0, dt, dx, nt = 10, 20.0, 5e-4, 10.0, 90
    decay = ol.q_decay(f0, dt)
    a, b = npx + nx // 2, npx + nz // 2
    recs, _ = run_gpu(vp, rho, q, npx, f0, dt, dx, [(a, b, nt + decay, 2)])
    ref, _, _ = ol.q_forward(vp, vp * 0, rho, q, q, dx, dx, dt, f0, nt, npx, npx, a, b, nrz0=2)
    assert np.abs(ref).max() > 0 and bits_equal(recs[0][:, decay:], ref)


@pytest.mark.parametrize("nx,nz", [(40 - 2 * NPX + 1, 64 - 2 * NPX), (48 - 2 * NPX, 66 - 2 * NPX + 63)])
def test_gradient_tile_edges(nx, nz):
    vp, rho, q = model(nx, nx=nx, nz=nz)
    rx = np.r_[np.arange(vp.shape[0]), [2, 2]].astype(np.int32)
    rz = np.r_[np.full(vp.shape[0], NPX + 1), [2, 2]].astype(np.int32)
    w = S.wavelet(S.WAVELET_Q, 120, DT, 20.0)
    shots = [S.ShotSpec(vp.shape[0] // 2, NPX + 4, rx, rz, w)]
    obs = observed((vp * 1.02).astype(np.float32), rho, (q * 0.8).astype(np.float32), shots)
    with engine(vp, rho, q) as e:
        e.set_shots(shots)
        e.set_checkpoint_interval(13)
        J, gv, gq = e.gradient(obs, want_invq=True)
        obs_list = e.split_records(obs)
    Jo, gvo, gqo = oracle(vp, rho, q, shots, obs_list)
    assert np.abs(gqo).max() > 0 and abs(J - Jo) <= 1e-4 * Jo
    assert rel_l2(gv, gvo) <= TOL_GRAD and rel_l2(gq, gqo) <= TOL_GRAD


@pytest.mark.parametrize("nx,nz", [(28, 44), (29, 45), (27, 41), (43, 107), (45, 110)])
def test_default_step_tile_edges(nx, nz):
    """The default step's tiles of 64 rows by 16 columns, four rows and four or two columns per thread:
    the final stress everywhere on padded grids around those multiples, against the FP64 restatement."""
    vp, rho, q = qmodel(seed=nz, nx=nx, nz=nz)
    npx, f0, dt, dx, nt = 10, 20.0, 5e-4, 10.0, 110
    decay = ol.q_decay(f0, dt)
    a, b = npx + nx - 3, npx + nz // 2
    vpp, rhop, qp = (S.pad_model(m, npx, npx, npx, npx) for m in (vp, rho, q))
    with S.Engine(S.VISCOAC_2D, vpp.shape[0], vpp.shape[1], dx, dx, dt, npx, order=10, f0=f0) as e:
        e.set_model(vpp, rhop, qp)
        rx = np.arange(vpp.shape[0], dtype=np.int32)
        e.set_shots([S.ShotSpec(a - 1, b - 1, rx, np.full_like(rx, b - 1),
                                S.wavelet(S.WAVELET_Q, nt + decay, dt, f0))])
        rec = e.split_records(e.forward())[0]
        p = e.wavefield(0, S.FIELD_P)
    _, _, fin = ol.q_forward(vp, vp * 0, rho, q, q, dx, dx, dt, f0, nt, npx, npx, a, b, fp64=True, want_final=True)
    assert np.abs(fin).max() > 0 and rel_l2(p, fin) <= TOL_FAST
    assert bits_equal(rec[:, -1].ravel(), p[:, b - 1].ravel())
