"""Very long lines.  A shot near the right end of one records what it records on a line of 400 columns with
the same right end, bit for bit: the models vary with depth only, and nothing returns from the left edge
of either within the record.  The viscoacoustic gradient likewise, near that end."""
import numpy as np
import pytest

from conftest import bits_equal, rel_l2
from seismic_code_github_b200 import seisfd as S

pytestmark = pytest.mark.gpu

NZ, PML, NT = 32, 6, 8
COLUMNS = {"viscoel": 4, "visco_exact": 8, "visco_gradient": 8, "elastic": 8, "visco": 16}  # per tile


def run(kind, nx):
    scheme = {"viscoel": S.VISCOEL_2D, "elastic": S.ELASTIC_2D}.get(kind, S.VISCOAC_2D)
    rng = np.random.default_rng(5)

    def line(lo, hi):
        return np.ascontiguousarray(np.broadcast_to((lo + (hi - lo) * rng.random(NZ)).astype(np.float32), (nx, NZ)))

    vp, den, q = line(2000.0, 2600.0), line(1800.0, 2300.0), line(30.0, 90.0)
    rx = nx - 1 - np.arange(8, 60, dtype=np.int32)
    rz = np.full(rx.size, PML + 5, np.int32)
    w = S.wavelet(S.WAVELET_Q, NT, 5e-4, 20.0)
    with S.Engine(scheme, nx, NZ, 5.0, 5.0, 5e-4, PML, order=10, flags=S.EXACT if kind == "visco_exact" else 0,
                  f0=20.0) as e:
        if kind == "elastic":
            e.set_gauss_radius(8)
            e.set_free_surface(PML)
        if kind in ("elastic", "viscoel"):
            e.set_model_elastic(vp, vp / np.float32(1.8), den, *((q, q) if kind == "viscoel" else ()))
        else:
            e.set_model(vp, den, q)
        e.set_shots([S.ShotSpec(nx - 30, PML + 8, rx, rz, w)])
        if kind == "visco_gradient":
            e.set_checkpoint_interval(3)
            _, g, gq = e.gradient(np.zeros(rx.size * NT, np.float32), want_invq=True)
            return [g[-60:].copy(), gq[-60:].copy()], [e.wavelet_gradient(0)], e.timing()["launches"]
        out = [e.forward().copy()]
        if kind == "viscoel":
            out.append(e.records(S.FIELD_P).copy())
        if kind == "elastic":
            out.append(e.records(S.FIELD_VZ).copy())
        return out, [], e.timing()["launches"]


def compare(kind, nx):
    want, want_sum, n = run(kind, 400 if nx % 2 == 0 else 401)  # the stamp's centre depends on the parity
    got, got_sum, n_wide = run(kind, nx)
    for a, b in zip(got, want):
        assert np.abs(b).max() > 0 and bits_equal(a, b)
    for a, b in zip(got_sum, want_sum):  # partial sums of several tiles, added in any order
        assert np.abs(b).max() > 0 and rel_l2(a, b) <= 1e-5
    return n, n_wide


@pytest.mark.parametrize("kind", ["viscoel", "visco_exact", "visco"])
def test_source_stamp_of_a_long_line(kind):
    """The squared distances of the Gaussian stamp's normalising sum exceed 31 bits."""
    compare(kind, 100000)


@pytest.mark.parametrize("kind", list(COLUMNS))
def test_more_tile_columns_than_a_grid_holds(kind):
    """More tile columns than one launch's grid.y holds (65535): a step takes several launches."""
    n, n_wide = compare(kind, 65535 * COLUMNS[kind] + 100)
    assert n_wide > n
