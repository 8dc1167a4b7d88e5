"""Kernels that wait for their predecessor (programmatic dependent launch) read with ordinary loads, on the CPU."""
import os
import re

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "..", "cmblensing_b200", "csrc")


def _kernels():
    """name -> (parameters, body) of every __global__ function, and of the device functions that integrate a lens."""
    out = {}
    for name in ("lf_kernels.cuh", "lf_cluster.cuh"):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(SRC, name)).read())
        for m in re.finditer(r"(?:__global__ void __launch_bounds__\((?:[^()]|\([^()]*\))*\)|__device__ __forceinline__ void)"
                             r"\s+(k_\w+|cl_integrate)\(([^)]*)\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            out[m.group(1)] = (m.group(2), text[m.end():i])
    return out


def test_no_noncoherent_loads_behind_the_wait():
    """A non-coherent load needs memory that is constant for the kernel's whole life and may move ahead of
    griddepcontrol.wait: neither __ldg nor a __restrict__ parameter in a kernel that waits.  The p planes are constant
    from before the lens's first kernel started, and so in the stage kernels that follow it."""
    kernels = _kernels()
    waiting = {k: v for k, v in kernels.items() if "pdl_wait()" in v[1]}
    assert {"k_col", "k_row", "k_row_pair", "k_row_pair_adj", "k_row_rows"} <= set(waiting)
    for name, (params, body) in waiting.items():
        assert "__restrict__" not in params and "ld.global.nc" not in body, name
        if name in ("k_row_pair", "k_row_pair_adj"):
            body = body.replace("__ldg(pq + ", "")
        if name == "k_row_rows":
            body = re.sub(r"INIT \? pq\[([^]]*)\] : __ldg\(pq \+ \1\)", "", body)
        assert "__ldg" not in body, name
