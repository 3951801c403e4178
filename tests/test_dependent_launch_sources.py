"""Kernels that may start before the one in front of them is complete wait for it (griddepcontrol.wait) and then read what it
wrote.  Invariant loads -- __ldg, or plain ones through const __restrict__ parameters -- may be moved above that wait by a
compiler, and no run shows that reliably; so the sources are checked: such a kernel reads its inputs in other ways."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "slimkernels_b200", "csrc")
WAITS = ("grid_dep_wait();", "act_wait_for_inputs();")


def _code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _kernels(code):
    """(name, parameter list, body) of every __global__ function."""
    for m in re.finditer(r"__global__", code):
        head = re.compile(r"(\w+)\s*\(").search(code, m.end())
        while head.group(1) in ("__launch_bounds__",):             # skip its arguments
            depth, i = 1, head.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(code[i], 0)
                i += 1
            head = re.compile(r"(\w+)\s*\(").search(code, i)
        end = code.index(")", head.end())
        start = code.index("{", end)
        depth, i = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(code[i], 0)
            i += 1
        yield head.group(1), code[head.end():end], code[start:i]


def test_inputs_are_read_behind_the_wait():
    seen = set()
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        for kernel, params, body in _kernels(_code(name)):
            if not any(w in body for w in WAITS):
                continue
            seen.add(kernel)
            assert not re.search(r"const[^,]*__restrict__", params), f"{kernel}: invariant loads of its inputs"
            assert "__ldg(p.x_scale" not in body, f"{kernel}: invariant loads of the token scales"
            if kernel == "w2a8_umma_kernel":                       # reads the group scales behind the wait, too
                assert "__ldg(" not in body, kernel
    assert {"w2a8_direct_kernel", "w2a8_umma_kernel", "w2a8_decode_kernel", "w2a8_stream_kernel", "quantize_activation_kernel",
            "silu_mul_quantize_cluster_kernel", "silu_mul_quantize_twopass_kernel"} <= seen
