"""Loads written as inline assembly: one that the compiler may move (not
volatile) is a pure function of its address, so it may only read records that
no kernel writes; what the kernel before wrote is read by volatile loads, which
stay behind the wait for that kernel."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ccfd_b200", "csrc")

# mesh records, written by the upload only
MESH_RECORDS = ("gw + k", "T.f_nl + id", "T.f_bb + id", "T.f_gp + id")


def test_movable_loads_read_mesh_records_only():
    with open(os.path.join(CSRC, "stage_impl.cuh")) as f:
        text = f.read()
    # functions holding a movable load
    movable = set()
    for m in re.finditer(r'asm\("ld\.', text):
        movable.add(re.findall(r"__device__ __forceinline__ \S+ (\w+)\(", text[:m.start()])[-1])
    assert movable == {"ld32", "ld32_once"}
    for name in movable:
        for m in re.finditer(rf"(?<!\w){name}\(([^()]*(?:\([^()]*\))?[^()]*)\)", text):
            arg = m.group(1)
            assert arg in MESH_RECORDS or arg == "const double4* p", (name, arg)
