"""The default mode of the VTI modeller is no further from a 64-bit run than the reference's own rounding order
is, with PML strips on all four sides (whose recurrences amplify an error that repeats at every step)."""
import numpy as np
import pytest

import oracle_lib as ol
from conftest import rel_l2
from seismic_code_github_b200 import seisfd as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxv,nzv,bound,top,nt", [(120, 100, 20, 20, 500), (120, 100, 30, 12, 500),
                                                  (150, 110, 24, 25, 500), (100, 120, 16, 30, 600)])
def test_default_mode_against_64_bits(nxv, nzv, bound, top, nt):
    rng = np.random.default_rng(top)
    z = np.arange(nzv)
    vz = np.tile(np.linspace(1600.0, 3000.0, nzv), (nxv, 1)).astype(np.float32)
    vz += (40.0 * rng.standard_normal(vz.shape)).astype(np.float32)
    eps = np.tile(np.where(z < 45, 0.12, 0.22), (nxv, 1)).astype(np.float32)
    delta = np.tile(np.where(z < 45, 0.04, 0.09), (nxv, 1)).astype(np.float32)
    args, shot = (5.0, 5.0, 5e-4, 30.0, nt, (bound, bound, top, bound)), (nxv // 2, 2, 2, 0, nxv - 1)
    ref64 = ol.vti_forward(vz, eps, delta, *args, *shot, fp64=True)
    ref32 = ol.vti_forward(vz, eps, delta, *args, *shot)
    rec, _ = S.vti_forward(vz, eps, delta, *args, [shot])
    assert np.abs(ref64).max() > 0
    assert rel_l2(rec[0], ref64) <= rel_l2(ref32, ref64)
