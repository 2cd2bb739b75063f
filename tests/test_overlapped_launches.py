"""Kernels that may start while the kernel before them still runs (previous_done() in common.cuh): what that one writes must
not be read through the read-only path, which requires data that nothing changes while the kernel runs. Read off the
sources; on the GPU the mistake would show as a race."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "gridnet_b200", "csrc")
# tensors of the caller that no kernel of the library writes ahead of a reader
CALLERS = {"p.scale", "w"}


def early_kernels():
    found = {}
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for part in re.split(r"\b__global__\b", text)[1:]:
            body = part[:part.index("\n}\n")]
            if "previous_done()" in body:
                kernel = re.search(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\([^;{]*?\)\s*(?=\w)", "", body, count=1)).group(1)
                found[kernel] = body
    return found


def test_early_kernels_do_not_read_through_the_read_only_path():
    kernels = early_kernels()
    assert {"step_fwd_quad", "quad_reverse_k", "quad_wgrad_k", "norm_finalize_k", "from_il4_k"} <= set(kernels), sorted(kernels)
    for kernel, body in kernels.items():
        for source in re.findall(r"__ldg\(\s*([\w.]+)", body):
            assert source in CALLERS, f"{kernel}: __ldg({source})"
        head = body[:body.index("{")]
        for name in re.findall(r"const \w+ \*__restrict__ (\w+)", head):
            if re.search(r"(?<![\w(])" + name + r"\s*\[", body) and name not in CALLERS:
                raise AssertionError(f"{kernel}: {name} may be read through the read-only path")
    with open(os.path.join(CSRC, "quad_geo.cuh")) as f:
        assert "__ldg(" not in f.read(), "device functions shared by the kernels above"
