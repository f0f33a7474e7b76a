"""Barriers of the cluster kernels and of the block kernels with a role per warp, checked on their
source: a fault here would be undefined behaviour on the device, not a wrong value."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "edge_to_b200", "csrc")


def source(name):
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", src, flags=re.S)


def body(src, name):
    """The text between the braces of the definition of `name`."""
    m = re.search(r"\b%s\s*\([^;{]*\)\s*\{" % name, src)
    assert m, name
    depth, k = 1, m.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(src[k], 0)
        k += 1
    return src[m.end():k - 1]


def test_peer_shared_memory_is_addressed_behind_a_cluster_barrier():
    """A block of a cluster may be addressed through map_shared_rank only once it has started, which a
    cluster barrier establishes: every use in a kernel comes after one."""
    uses = {f: source(f).count("map_shared_rank") for f in os.listdir(CSRC)}
    assert {f: n for f, n in uses.items() if n} == {"fields.cu": 1, "batch_ops.cuh": 1, "batch.cu": 1}
    oc = body(source("fields.cu"), "oc_team")
    assert oc.count("map_shared_rank") == 1
    first = re.search(r"barrier_wait\(\)|this_cluster\(\)\.sync\(\)", oc)
    assert first and first.start() < oc.index("map_shared_rank") < oc.index("team_sum(v)")
    # the batched solve: the queue's barrier comes before the first read of a peer and before the solve,
    # whose sums (TeamSum::run) write to peers; the one-launch cycle sums nothing
    kern = body(source("batch.cu"), "k_batch_pcg")
    assert kern.count("map_shared_rank") == 1
    assert kern.index("TM::sync()") < kern.index("map_shared_rank") < kern.index("b_pcg_problem")
    assert "TeamSum" not in source("vtail.cu")


def test_stencil_warps_meet_at_one_barrier():
    """k_st3_apply_d gives its warps different work; __syncthreads() is defined only where every thread of
    the block reaches the same one, so none may stand inside a branch."""
    b = body(source("coarse.cuh"), "k_st3_apply_d")
    assert b.count("__syncthreads()") == 1
    before = b[:b.index("__syncthreads()")]
    assert before.count("{") == before.count("}")
