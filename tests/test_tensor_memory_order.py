"""The order in which kernels take tensor memory and let the kernel behind them start, read from their source.

`tcgen05.alloc` waits until the SM has the columns.  A kernel that lets the one behind start (`pdl_launch_dependents`) before its
own blocks have theirs can meet a successor that takes columns ahead of its own wait (the products do): the successor then waits
for this grid to end, and this grid for the successor's columns.  So the permission comes after the allocation, in the warp that
allocated or behind a block-wide barrier; and attention, which may run right behind a library product whose order is not known,
allocates after its own wait for the kernel in front."""

import glob
import os
import re

import pytest

from paged_llm_b200.csrc import build


def kernels():
    """(file, name, body) of every kernel that takes tensor memory."""
    found = []
    for path in sorted(glob.glob(os.path.join(build.HERE, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for part in re.split(r"(?=__global__ )", text)[1:]:
            body = part[:part.index("\n}\n")]
            if "tcgen05.alloc" in body:
                found.append((os.path.basename(path), re.search(r"(\w+)\(", body.split("__launch_bounds__")[1].split(")", 1)[1]).group(1), body))
    return found


FOUND = kernels()


def test_the_kernels_are_found():
    assert {name for _, name, _ in FOUND} >= {"attn_tc_kernel", "attn_tc2_kernel", "gemm_mid_kernel", "gemm_tc_duo_kernel"}


@pytest.mark.parametrize("file,name,body", FOUND, ids=[name for _, name, _ in FOUND])
def test_the_kernel_behind_starts_after_the_allocation(file, name, body):
    alloc, release = body.index("tcgen05.alloc"), body.index("pdl_launch_dependents")
    assert alloc < release, f"{file}: {name} lets the next kernel start before it has its tensor memory"
    between = body[alloc:release]
    assert "__syncthreads" in between or "}" not in between, f"{file}: {name}: threads that did not allocate may let it start"


@pytest.mark.parametrize("file,name,body", [f for f in FOUND if f[1].startswith("attn")], ids=[f[1] for f in FOUND if f[1].startswith("attn")])
def test_attention_allocates_after_its_wait(file, name, body):
    assert body.rindex("pdl_wait") < body.index("tcgen05.alloc"), f"{file}: {name}"
