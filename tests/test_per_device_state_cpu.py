"""Function attributes (dynamic shared memory above 48 KB, cluster sizes above 8) belong to a device's
context.  A flag that the process has set one would leave them unset on a second device, or after a
device reset, where the launches would then be refused."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "edge_to_b200", "csrc")


def test_function_attributes_are_not_kept_per_process():
    seen = 0
    for f in os.listdir(CSRC):
        src = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(CSRC, f)).read(), flags=re.S)
        seen += src.count("cudaFuncSetAttribute")
        # a function-local flag or once-guard ahead of the call, within the same function
        for m in re.finditer(r"cudaFuncSetAttribute", src):
            start = src.rfind("\n}\n", 0, m.start())
            head = src[max(start, 0):m.start()]
            assert not re.search(r"\bstatic\s+(std::atomic\w*(<[^>]*>)?|bool|int|std::once_flag)\s+\w+\s*[{=;]", head), \
                (f, head[-200:])
    assert seen >= 8


def test_oc_update_does_not_need_a_cluster_of_sixteen():
    """Sixteen blocks of one cluster need a GPC of 16 SMs, which a slice of a GPU may not have: a refused
    launch must leave the passes over the whole grid, which take any size, to do the update."""
    src = open(os.path.join(CSRC, "fields.cu")).read()
    body = src[src.index("\nint oc_launch("):]
    body = body[:body.index("\n}\n")]
    cluster = body[body.index("if (n <= OC_CLUSTER_MAX)"):]
    guarded = re.search(r"if \(cudaFuncSetAttribute\(k_oc_cluster.*?cudaLaunchKernelEx\(&cfg, k_oc_cluster.*?==\s*cudaSuccess\)"
                        r"\s*return 1;\s*cudaGetLastError\(\);", cluster, flags=re.S)
    assert guarded and "return 0" not in body
    assert "k_oc_bisect" in cluster[guarded.end():]
