"""A chained kernel exists while the kernel before it still writes, so it may
not read lattice state through the read-only path: no __ldg in the code that the
chained kernels are made of, and no const __restrict__ source, which would
let the compiler choose that path."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imexlbm_gb300", "csrc")
# headers whose device code runs in chained kernels only, or in them too
SHARED = ["kernels_common.cuh", "flat_lowp.cuh", "moments_fixed.cuh", "conserved.cuh", "minmax.cuh", "rows_lowp.cuh",
          "two_f32.cuh", "two_f32.cu"]
# chained kernels by file; the row-staged and the two-step kernels read lattices by bulk and tensor copies alone
KERNELS = {"conserved.cuh": ["k_conserved"], "minmax.cuh": ["k_extremes", "k_pick"], "kernels_lowp.cu": ["k_flat_lowp"],
           "kernels_fx.cu": ["k_step_fxs"], "two_f32.cu": ["k_edge_f32", "k_two_f32"], "rows_lowp.cuh": ["k_rows_lowp"],
           "batch.cu": ["k_batch_rows", "k_batch_pairs"]}


def source(name):
    with open(os.path.join(CSRC, name)) as fp:
        return re.sub(r"//[^\n]*", "", fp.read())


def definition(text, kernel):
    """A kernel's parameters and body."""
    at = re.search(r"__global__[^;{]*?\b" + kernel + r"\s*\(", text).end()
    begin = text.index("{", at)
    depth, end = 1, begin + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[at:begin], text[begin:end]


def test_every_chained_kernel_is_listed():
    launched = set()
    for name in os.listdir(CSRC):
        if name.endswith((".cu", ".cuh")):
            text = source(name)
            launched |= set(re.findall(r"launch_chained\([^;]*?\b(?:rowslp::)?(k_\w+)", text)) | set(re.findall(r"\bgo\((k_\w+)", text))
    assert launched == {k for ks in KERNELS.values() for k in ks}


def test_no_read_only_loads():
    for name in SHARED:
        assert "__ldg" not in source(name), name
    for name, kernels in KERNELS.items():
        for kernel in kernels:
            params, body = definition(source(name), kernel)
            assert "__ldg" not in body, kernel
            if kernel not in ("k_two_f32", "k_rows_lowp"):
                assert not re.search(r"const[^,]*__restrict__ src\b", params), kernel

