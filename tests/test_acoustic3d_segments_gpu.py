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
