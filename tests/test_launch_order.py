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


def test_read_only_loads_of_constant_data_only():
    """__ldg promises that nothing writes the data while the kernel runs, and the compiler may move it above
    acquire(); a programmatic dependent may start before its predecessor's stores.  So the step kernels read
    through __ldg only what no kernel of the chain writes."""
    constant = {"vp", "den", "bxm", "bym", "bzm", "busg", "p1", "p2", "q1", "q2", "q3", "m1", "m2", "m3", "b2e", "b1e",
                "lm2", "lam", "mue", "itopo", "wavelets", "stamps", "spg", "tile_order"}
    local = {"trp", "tn", "tp", "re"}          # receiver lists and sponge tables by local names
    helpers = ("model4", "ldg4", "ld_model")
    wrapped = {"f", "p", "base", "reinterpret_cast"}  # parameters of helpers, whose calls are checked below
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", source(name))
        for m in re.finditer(r"__ldg\(((?:[^()]|\((?:[^()]|\([^()]*\))*\))*)\)", text):
            arg = m.group(1)
            members = set(re.findall(r"\ba\.(\w+)", arg)) - {"mpitch", "nx_model", "spg_stride", "L", "step", "pml"}
            if members:
                assert members <= constant, f"{name}: __ldg({arg})"
            else:
                assert set(re.findall(r"^(?:at4\()?(\w+)", arg)) <= local | wrapped, f"{name}: __ldg({arg})"
                if set(re.findall(r"^(?:at4\()?(\w+)", arg)) <= wrapped:  # inside one of the helpers
                    defs = re.findall(r"auto (\w+) = \[|float4 (\w+)\(const float\* p\)", text[:m.start()])
                    assert "".join(defs[-1]) in helpers, f"{name}: __ldg({arg}) in {defs[-1]}"
        for helper in helpers + ("model_at",):
            for m in re.finditer(helper + r"\(((?:[^()]|\([^()]*\))*)\)", text):
                members = set(re.findall(r"\ba\.(\w+)", m.group(1)))
                assert members <= constant, f"{name}: {m.group(0)}"
