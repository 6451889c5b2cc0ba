"""The 3-D step splits the x march into segments when a launch has fewer columns than the chip has
CTA slots.  Short grids give a last segment of one or a few planes and segments shorter than the
2R - 1 planes they fill their Vx ring with; every case against the FP64 restatement (the tolerance
of test_acoustic3d_gpu)."""
import pytest

from test_acoustic3d_gpu import check_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,order,varden", [(9, 8, False), (13, 8, True), (23, 8, False), (42, 4, True), (75, 8, True)])
def test_segment_edges(nx, order, varden):
    check_case(nx, 37, 66, 3, 60, (nx // 2, 18, 30), seed=nx, order=order, varden=varden)


def test_unequal_spacing_with_variable_density():
    """Each axis has its own precomputed dt / (d den)."""
    import numpy as np
    import oracle_lib as ol
    from conftest import rel_l2
    from seismic_code_github_b200 import seisfd as S
    from test_acoustic3d_gpu import TOL, model3d, receivers
    nx, ny, nz, pml, nt = 30, 37, 41, 5, 60
    vp, den = model3d(nx, ny, nz, 8, varden=True)
    rx, ry, rz = receivers(nx, ny, nz, 8)
    w = S.wavelet(S.WAVELET_RIC, nt, 1e-3, 25.0, 25)
    with S.Engine(S.ACOUSTIC_3D, nx, nz, 10.0, 9.0, 1e-3, pml, order=8, ny=ny, dy=12.0) as e:
        e.set_model(vp, den)
        e.set_shots([S.ShotSpec(14, 20, rx, rz, w, sy=18, rec_y=ry)])
        rec = e.forward().reshape(len(rx), nt)
    ref, _ = ol.afd3d_forward(vp, den, w, (14, 18, 20), rx, ry, rz, pml, 10.0, 12.0, 9.0, 1e-3, radius=4)
    assert np.abs(ref).max() > 0 and rel_l2(rec, ref) <= TOL
