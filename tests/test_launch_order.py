"""Order between kernels that are programmatic dependents, read from the sources: a race there need not show
in a run.  acquire() of a kernel waits for its direct predecessor only, so what a kernel reads before its
acquire() must be written before the chain of programmatic dependents begins."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "seismic_code_github_b200", "csrc")


def source(name):
    return open(os.path.join(CSRC, name)).read()


def test_vti_chain_starts_with_a_plain_launch():
    """vti_step_kernel reads the shot windows before acquire(), so the first kernel after vti_window_kernel,
    which writes them, is launched without the programmatic attribute."""
    text = source("vti2d.cu")
    kernel = text[text.index("vti_step_kernel(const __grid_constant__"):]
    assert kernel.index("P[o.vz + g]") < kernel.index("acquire()")
    launches = text[text.index("vti_window_kernel<<<"):]
    first = re.search(r"tile::launch\(([^;]*)\);", launches).group(1)
    assert "vti_inject_kernel" in first and first.endswith(", it > 1")
