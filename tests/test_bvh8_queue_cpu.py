"""The BVH8 collapse is over when as many items are finished as allocated.  That
may not be found early: a warp counts an item only behind the atomic that
allocated its children, and looks at the finished count before the allocated
one."""
import re

import pytest

from tests.test_launch_order_cpu import CSRC, block

WIDE = (CSRC / "wide.cu").read_text()


def test_the_finished_count_is_read_before_the_allocated_one():
    body = block(WIDE, WIDE.index("struct FinishedItems"))
    look = block(body, body.index("bool all()"))
    first, second = look.index("kBvh8Finished"), look.index("kBvh8Alloc + (finished >> 31)")
    assert first < second


@pytest.mark.parametrize("kernel", ["bvh8_kernel", "bvh8_group_kernel"])
def test_items_are_counted_behind_their_childrens_allocation(kernel):
    body = block(WIDE, re.search(r"void %s\(" % kernel, WIDE).end())
    alloc = body.index("bases = atomicAdd(")
    result = re.search(r"bases = __shfl_sync\(kFullMask, bases, \d+\);", body)
    assert alloc < result.start() < body.index("items.add(done)")
    assert body.count("items.add(") == 1
    stores = [m.start() for m in re.finditer(r"st_relaxed_u64\(pairs", body)]
    assert stores and result.end() < min(stores)
