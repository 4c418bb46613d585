"""clast_search_noalloc promises no device, stream-ordered or pinned allocation:
none stands in the functions that its search runs through (a context's first
search included), read from the source.  Kernel launchers take their scratch
from the workspace, which is the fixed block there."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "clast_b200", "csrc")
ALLOCATES = re.compile(r"cuda(Malloc|Free|HostAlloc|HostRegister)\w*\s*\(|\.alloc\s*\(|\bstage\s*\(")


def body(text, head):
    """The text of the function whose definition starts with `head`, without comments."""
    at = text.index(head)
    start = text.index("{\n", at)
    depth, i = 0, start
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return re.sub(r"//[^\n]*", "", text[start:i])


@pytest.mark.parametrize("name,head", [
    ("clast_engine.cu", "const GroupCtl& read_ctl("), ("clast_engine.cu", "int64_t search_group("),
    ("clast_engine.cu", 'extern "C" int clast_search_noalloc('), ("clast_workspace.h", "void* arena_get("),
    ("clast_kernels.cu", "int radix_sort_u64("), ("clast_kernels.cu", "DpBuckets dp_bucket_count("),
    ("clast_kernels.cu", "long long launch_dp_mode("), ("clast_kernels.cu", "void scan_1pass("),
    ("clast_kernels.cu", "void seed_filter("), ("clast_kernels.cu", "void final_order(")])
def test_search_allocates_nothing(name, head):
    text = body(open(os.path.join(CSRC, name)).read(), head)
    assert len(text) > 60
    found = ALLOCATES.search(text)
    assert found is None, found.group(0)
