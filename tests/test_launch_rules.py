"""Rules of the kernels that may start while the kernel before them still runs
(pdl_wait in pic_internal.cuh), read off the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "msc-thesis_gb300", "csrc")
TABLES = ("SegBlock", "EnsRun")  # written between steps only


def dependent_kernels():
    """(name, parameters) of every kernel whose body calls pdl_wait."""
    for f in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, f)).read() if f.endswith((".cu", ".cuh")) else ""
        for m in re.finditer(r"__global__ void\s+(?:__cluster_dims__\([^)]*\)\s*)?"
                             r"(?:__launch_bounds__\([^)]*(?:\([^)]*\))?[^)]*\)\s*)?(\w+)\(([^)]*)\)\s*\{(.*?)\n\}",
                             text, re.S):
            if "pdl_wait()" in m[3]:
                yield m[1], m[2]


def test_no_read_only_arguments_that_earlier_kernels_write():
    found = dict(dependent_kernels())
    assert {"push_kernel", "ens_push_kernel", "convert_kernel", "kspace_kernel", "adj_kick_kernel",
            "ens_adj_kick_kernel", "spec_cols_kernel", "ntc_list_kernel", "compat_push_kernel"} <= set(found)
    for name, params in found.items():
        for p in params.split(","):
            if "const" in p and "__restrict__" in p:
                assert any(t in p for t in TABLES), f"{name}: {p.strip()}"
