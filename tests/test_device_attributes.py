"""Kernels that use more than 48 KB of dynamic shared memory must be allowed to on every device: the
attribute belongs to the current device, so it is set where a context's device is prepared
(preload_kernels, once per device), never once per process."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "2d-treecodes_b200", "csrc")
FILES = {os.path.basename(p): open(p).read()
         for p in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.h"))}


def body(src, head):
    """Text of the function whose definition starts with `head`."""
    at = src.index("{", src.index(head))
    depth = 0
    for i in range(at, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[at:i + 1]
    raise AssertionError(head)


def test_no_attribute_is_set_once_per_process():
    for name, src in FILES.items():
        assert not re.search(r"static\s+const\s+cudaError_t", src), name


def prepare_bodies(src):
    return {fn: body(src, f"int {fn}() {{") for fn in re.findall(r"^int (prepare_\w+)\(\) \{", src, re.M)}


def test_every_attribute_is_set_per_device():
    preload = body(FILES["capi.cu"], "static int preload_kernels(int device)")
    found = 0
    for name, src in FILES.items():
        if name == "tc_internal.h":   # (allow_shared itself)
            src = src.replace(body(src, "inline int allow_shared("), "")
        for fn, text in prepare_bodies(src).items():
            assert fn + "()" in preload, fn
            src = src.replace(text, "")
            found += 1
        assert "cudaFuncSetAttribute" not in src, name
    assert found == 4


def test_every_kernel_with_dynamic_shared_memory_is_prepared():
    found = set()
    for name, src in FILES.items():
        prepared = "".join(prepare_bodies(src).values())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(", src):
            if "extern __shared__" in body(src, m.group(0)):
                assert re.search(r"\b%s\b" % m.group(1), prepared), (name, m.group(1))
                found.add(m.group(1))
    assert found == {"k_sort_small", "k_sort_small_targets", "k_leaf_p2e", "k_potential_eval"}
