"""The visco-elastic kernels work on tiles of 64 rows by 4 columns: padded widths and depths around
their multiples, with receivers on every column, bit for bit against the FP32 restatement."""
import numpy as np
import pytest

import oracle_lib as ol
from conftest import bits_equal
from test_viscoel_gpu import emodel, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(24, 44), (25, 45), (30, 43), (35, 107), (41, 108)])
def test_tile_edges(nx, nz):
    model = emodel(seed=nx, nx=nx, nz=nz)
    npx, f0, dt, dx, nt = 10, 20.0, 5e-4, 10.0, 90
    decay = ol.q_decay(f0, dt)
    a, b = npx + nx // 2, npx + nz // 2
    r1, r2, _, e = run_gpu(model, npx, f0, dt, dx, [(a, b, nt + decay, 2)])
    e.close()
    o1, o2, _ = ol.q_forward(*model, dx, dx, dt, f0, nt, npx, npx, a, b, nrz0=2)
    assert np.abs(o1).max() > 0
    assert bits_equal(r1[0][:, decay:], o1) and bits_equal(r2[0][:, decay:], o2)
