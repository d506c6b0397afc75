"""Orderings that only a memory model shows: a compiler or a GPU that used the freedom would give rare wrong results and
nothing a GPU test could be relied on to see, so the sources are checked.

Kernels that programmatic dependent launch may start early (they call grid_dep_wait or grid_dep_sync) read what
other kernels are still writing, so none of it may come through the read-only path: no __ldg, and no __restrict__ on
anything but a layer's constants.

The warp that counts finished MLP1 items publishes rows that sixteen other warps wrote: acquire in every lane, warp
barrier, fence in every lane, then the counts.

What one CTA of a pair hands to the other needs cluster scope: copies complete on the even CTA's barrier by themselves,
and arrivals there name their scope."""
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


def test_counts_are_published_behind_all_epilogue_warps():
    body = {n: b for n, _, b in kernels()}["expert_gemm_kernel"]
    part = body[body.index("warp == kDoneWarp"):]
    steps = ["ld_acquire_cta(", "__syncwarp();", "__threadfence();", "atomicAdd(f.tile_done + pa.work"]
    at = [part.index(x) for x in steps]
    assert at == sorted(at)


def test_no_bounded_wait_starts_before_the_predecessor_is_done():
    """The ~1 s limit of a wait must not run while a kernel only waits for its turn: every role of the kernels with
    bounded waits passes the grid wait first."""
    body = {n: b for n, _, b in kernels()}
    gemm = body["expert_gemm_kernel"]
    assert gemm.index("grid_dep_sync();") < gemm.index("mbar_wait_warp")
    router = body["router_kernel"]
    roles = re.split(r"(?:if|else if) \(warp (?:==|<) \d\) \{", router[router.index("grid_dep_release();"):])
    roles = [r for r in roles[1:] if "mbar_wait_warp" in r]
    assert len(roles) == 3
    for r in roles:
        assert "grid_dep_wait();" in r and r.index("grid_dep_wait();") < r.index("mbar_wait_warp")


def test_hand_overs_of_a_cta_pair_have_cluster_scope():
    body = {n: b for n, _, b in kernels()}["expert_gemm_kernel"]
    ptx = open(os.path.join(ROOT, "gpt-oss_b200", "csrc", "sm100_ptx.cuh")).read()
    for arrive in re.findall(r"mbarrier\.arrive[\w.:]*shared::cluster", ptx):
        assert ".cluster.shared::cluster" in arrive, arrive
    assert not re.search(r"\b(tma_load_\dd|tma_load_\dd_hint|bulk_load\w*)\(", body)    # only loads of the pair
    waits = re.findall(r"mbar_wait_warp(<Wait::k(?:Cluster|ClusterRelaxed)>)?\((\w+)_bar", body)
    assert {bar for _, bar in waits} == {"full", "empty", "dfull", "dempty"}
    assert all(scope for scope, _ in waits) and ("<Wait::kCluster>", "full") in waits
    assert "fence.acquire.sync_restrict::shared::cluster.cluster" in ptx
