"""A model or shot set that replaces another is what the next call uses: host data reach the device in the
order of the context's stream, on which the kernels that read them run.  On the CPU: no host-to-device
copy of the library runs outside a stream.  On the GPU: many updates in a row, each followed at once by a
gradient, equal the gradients of contexts that never held another model, bit for bit."""
import os
import re

import numpy as np
import pytest

from conftest import ROOT, bits_equal
from seismic_code_github_b200 import seisfd as S

CSRC = os.path.join(ROOT, "seismic_code_github_b200", "csrc")


def test_host_copies_are_stream_ordered():
    found = 0
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        for m in re.finditer(r"(cudaMemcpy\w*)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            if "cudaMemcpyHostToDevice" in text[m.end():i]:
                found += 1
                assert m.group(1).endswith("Async"), f"{name}: {text[m.start():i]}"
        assert not re.search(r"\bcudaMemset\s*\(", text), name
    assert found >= 4


@pytest.mark.gpu
@pytest.mark.parametrize("order,varden", [(16, True), (8, False)])
def test_updates_are_seen_by_the_next_gradient(order, varden):
    nx, nz, nt = 131, 70, 40
    rng = np.random.default_rng(order)
    vp = (2000.0 + 600.0 * rng.random((nx, nz))).astype(np.float32)
    den = (1900.0 + 400.0 * rng.random((nx, nz))).astype(np.float32) if varden else None
    w = S.wavelet(S.WAVELET_RIC, nt, 1e-3, 25.0, 20)
    rx, rz = np.arange(10, nx - 10, dtype=np.int32), np.full(nx - 20, 13, np.int32)
    obs = rng.standard_normal(len(rx) * nt).astype(np.float32)
    models = [((vp * s).astype(np.float32), None if den is None else (den * s).astype(np.float32))
              for s in (1.0, 1.02, 1.05)]

    def engine():
        return S.Engine(S.ACOUSTIC_2D, nx, nz, 10.0, 10.0, 1e-3, 10, order=order)

    want = []
    for m in models:
        with engine() as e:
            e.set_model(*m)
            e.set_shots([S.ShotSpec(nx // 2, nz // 2, rx, rz, w)])
            e.forward()
            want.append(e.gradient(obs)[1])
    assert not bits_equal(want[0], want[1])
    with engine() as e:
        e.set_model(*models[0])
        e.set_shots([S.ShotSpec(nx // 2, nz // 2, rx, rz, w)])
        for k in range(30):
            e.set_model(*models[k % 3])
            assert bits_equal(e.gradient(obs)[1], want[k % 3]), k
