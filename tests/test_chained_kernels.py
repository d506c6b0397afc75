"""Kernels that programmatic dependent launch may start early (they call grid_dep_wait or grid_dep_sync) read what
other kernels are still writing, so none of it may come through the read-only path: no __ldg, and no __restrict__ on
anything but a layer's constants.  A compiler that moved such a load above the wait would show as rare wrong routing on
a GPU and nowhere else, so the sources are checked."""
import glob
import os
import re

from conftest import ROOT

CONSTANT = {"bias"}   # written by moe_load_layer, which waits


def kernels():
    for path in sorted(glob.glob(os.path.join(ROOT, "gpt-oss_b200", "csrc", "*.cu"))):
        for part in open(path).read().split("__global__")[1:]:
            head, body = part.split(") {", 1)
            name = re.search(r"(\w+)\(", re.sub(r"__\w+__\([^)]*\)", "", head)).group(1)
            yield name, head, body.split("\n}\n", 1)[0]


def test_chained_kernels_read_with_ordinary_loads():
    chained = {n: (h, b) for n, h, b in kernels() if "grid_dep_" in b}
    assert {"router_kernel", "topk_softmax_kernel", "build_index_kernel", "quantize_rows_kernel",
            "quantize_few_rows_kernel", "expert_gemm_kernel", "combine_kernel", "rmsnorm_rows_kernel"} <= set(chained)
    for name, (head, body) in chained.items():
        restricted = set(re.findall(r"__restrict__ (\w+)", head + body))
        assert restricted <= CONSTANT, (name, restricted - CONSTANT)
        assert "__ldg(" not in body, name
