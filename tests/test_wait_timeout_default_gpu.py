"""sfd_test_wait_timeout on a context whose schedule is not forced and whose launches are small: the hook's
step reports SFD_ERR_TIMEOUT from the forward, the per-shot forward and the gradient, and after its removal
the context gives the records and the gradient of a fresh one bit for bit."""
import numpy as np
import pytest

from conftest import bits_equal
from seismic_code_github_b200 import seisfd as S
from test_wait_timeout_gpu import engine_case

pytestmark = pytest.mark.gpu


def test_hook_on_small_launches(monkeypatch):
    for k in ("SFD_FMA_STAGES", "SFD_MARCH_SEG"):
        monkeypatch.delenv(k, raising=False)
    case, shots = engine_case()
    out = []
    for hook in (False, True):
        with S.Engine(S.ACOUSTIC_2D, case.Nx, case.Nz, case.dx, case.dz, case.dt, case.PML, order=16) as e:
            e.set_model(case.vp, case.den)
            e.set_shots(shots)
            obs = np.zeros(e.record_size(), np.float32)
            if hook:
                e.test_wait_timeout(0, 37, 1e-4)
                for call in (e.forward, e.forward_per_shot, lambda: e.gradient(obs)):
                    with pytest.raises(S.SfdError) as ei:
                        call()
                    assert ei.value.status == S.ERR_TIMEOUT
                e.test_wait_timeout(-1, 0)
            out.append((e.forward().copy(), e.gradient(obs)[1].copy()))
    assert np.abs(out[0][0]).max() > 0 and np.abs(out[0][1]).max() > 0
    assert bits_equal(out[0][0], out[1][0]) and bits_equal(out[0][1], out[1][1])
