"""The VTI step works on tiles of 64 x 2 cells and builds the shot windows on the device: grid widths
and depths around the tile's multiples, no left or top PML, apertures that reach over both model edges,
and zeroed epsilon / delta rows, against the FP32 restatement (bit for bit with SFD_EXACT) and, in the
default mode, within the tolerance of test_vti_gpu."""
import numpy as np
import pytest

import oracle_lib as ol
from conftest import rel_l2
from seismic_code_github_b200 import seisfd as S
from test_vti_gpu import model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxv,nzv,bounds,shot", [
    (40, 31, (12, 14, 0, 10), (20, 1, 1, 0, 39)),       # nx 64
    (44, 30, (0, 15, 6, 9), (20, 3, 2, 0, 43)),         # no left PML
    (60, 41, (33, 34, 0, 12), (30, 2, 1, -10, 69)),     # nx 145, aperture over both edges
    (25, 22, (20, 2, 3, 2), (12, 5, 4, 3, 22)),         # two-cell PML on the right and below
])
def test_tile_and_window_edges(nxv, nzv, bounds, shot):
    vz, eps, de = model(nxv, nzv, seed=nxv)
    nt = 260
    ref = ol.vti_forward(vz, eps, de, 5.0, 5.0, 5e-4, 30.0, nt, bounds, *shot)
    rec, _ = S.vti_forward(vz, eps, de, 5.0, 5.0, 5e-4, 30.0, nt, bounds, [shot], exact=True)
    assert np.abs(ref).max() > 0
    assert np.array_equal(rec[0].view(np.uint32), ref.view(np.uint32))
    fast, _ = S.vti_forward(vz, eps, de, 5.0, 5.0, 5e-4, 30.0, nt, bounds, [shot])
    assert rel_l2(fast[0], ref) <= 1e-5


def test_bad_model_values_outside_the_windows_are_accepted():
    """Only values that enter a shot's window are checked: a bad one outside its columns, or an epsilon
    in the rows that the modeller zeroes, is accepted as before; inside it is refused."""
    vz, eps, de = model(60, 40, seed=3)
    args = (5.0, 5.0, 5e-4, 30.0, 12, (10, 10, 0, 10))
    shot = (20, 1, 1, 5, 34)
    far, inside = vz.copy(), vz.copy()
    far[50, 3] = -1.0
    inside[20, 3] = np.nan
    shallow, deep = eps.copy(), eps.copy()
    shallow[20, 6] = np.nan  # row nsz0 + 6: zeroed
    deep[20, 7] = np.nan
    S.vti_forward(far, eps, de, *args, [shot])
    S.vti_forward(vz, shallow, de, *args, [shot])
    for m, e in ((inside, eps), (vz, deep)):
        with pytest.raises(S.SfdError) as err:
            S.vti_forward(m, e, de, *args, [shot])
        assert err.value.status == 1


@pytest.mark.parametrize("nzv,row", [(65600, 65560), (131200, 131130), (262300, 262190)])
def test_grids_of_many_rows(nzv, row):
    """More rows than one launch's grid.y holds (65535 rows of the window kernel, 131070 of the step), the
    source and the receivers among the last of them."""
    vz, eps, de = model(24, nzv, seed=4)
    args = (100.0, 100.0, 1e-2, 12.0, 14, (8, 9, 0, 10))
    shot = (12, row, row + 8, 0, 23)
    ref = ol.vti_forward(vz, eps, de, *args, *shot)
    assert np.abs(ref).max() > 0
    rec, t = S.vti_forward(vz, eps, de, *args, [shot], exact=True)
    assert np.array_equal(rec[0].view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("exact", [True, False], ids=["exact", "default"])
def test_slab_of_more_than_2_to_the_32_floats(exact):
    """A shot whose fields take more than 2^32 floats: near the left and bottom PML, whose split fields lie
    past that offset, it records what a grid of the same left part does (nothing returns from the right
    edge of either within the record), bit for bit."""
    vz, eps, de = model(1, 200000, seed=6)  # one model column, replicated over the aperture
    args = (100.0, 100.0, 1e-2, 12.0, 8, (10, 10, 0, 10))
    recs = []
    for width in (200, 2990):
        shot = (6, 199985, 199990, 0, width - 1)
        rec, _ = S.vti_forward(vz, eps, de, *args, [shot], exact=exact)
        recs.append(rec[0][:60].copy())
    assert np.abs(recs[0]).max() > 0
    assert np.array_equal(recs[0].view(np.uint32), recs[1].view(np.uint32))
