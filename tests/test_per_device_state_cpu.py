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
