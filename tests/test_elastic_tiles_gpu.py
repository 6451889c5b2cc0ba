"""The elastic kernels work on tiles of 64 rows by 8 columns, one vector of four cells per thread:
padded widths and depths around the multiples of 8 and 64, a last vector of one to four cells, and
surfaces that cross a tile row, in both boundary modes, bit for bit against the FP32 restatement."""
import numpy as np
import pytest

import oracle_lib as ol
from conftest import bits_equal
from test_elastic_gpu import imodel, run_fs, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(24, 44), (25, 45), (31, 46), (37, 47), (40, 108)])
def test_absorbing_tile_edges(nx, nz):
    model = imodel(seed=nx, nx=nx, nz=nz)
    npx, f0, dt, dx, nt, idecay = 10, 20.0, 5e-4, 10.0, 90, 30
    a, b = npx + nx // 2, npx + nz // 2
    r1, r2, _, e = run_gpu(model, npx, f0, dt, dx, [(a, b, nt + idecay, 2, idecay)], rgau=7)
    e.close()
    o1, o2, _ = ol.iso_forward(*model, dx, dx, dt, f0, nt, npx, npx, a, b, nrz0=2, idecay=idecay, rgau=7)
    assert np.abs(o1).max() > 0
    assert bits_equal(r1[0][:, idecay:], o1) and bits_equal(r2[0][:, idecay:], o2)


@pytest.mark.parametrize("nx,nz,top", [(24, 52, 2), (29, 118, 60), (36, 55, 63), (41, 121, 66)])
def test_free_surface_tile_edges(nx, nz, top):
    model = imodel(seed=nz, nx=nx, nz=nz)
    npx, f0, dt, dx, nt, idecay = 10, 20.0, 5e-4, 10.0, 90, 30
    a, b = npx + nx // 2, top + 4
    r1, r2, _, vx = run_fs(model, npx, top, f0, dt, dx, [(a, b, nt + idecay, 1, idecay)])
    o1, o2, fin = ol.iso_forward(*model, dx, dx, dt, f0, nt, npx, npx, a, b, nrz0=1, idecay=idecay, rgau=20, fsbc=True,
                                 npz_top=top, want_final=True)
    assert np.abs(o2).max() > 0
    assert bits_equal(r1[0][:, idecay:], o1) and bits_equal(r2[0][:, idecay:], o2) and bits_equal(vx, fin)
