"""What the sources of the tensor-memory kernels have to keep to, read from the text: a CTA lets the next kernel start
(talos_pdl) only once it holds its tensor memory, i.e. behind the block barrier that follows the allocation.  The other way
round two dependent kernels could wait in their allocations at the same time, the later one served first and waiting for
the earlier one."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "talos-xii_b200", "csrc")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_next_kernel_starts_behind_the_allocation(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    for m in re.finditer(r"\btmem_alloc2?\(tmem_slot", text):
        body = text[m.end():]
        assert body.index("__syncthreads()") < body.index("talos_pdl("), name
        start = text.rindex("extern __shared__", 0, m.start())
        assert "talos_pdl(" not in text[start:m.start()], name


def test_the_allocating_kernels_are_seen():
    seen = [f for f in os.listdir(CSRC) if f.endswith(".cu") and re.search(r"\btmem_alloc2?\(tmem_slot", open(os.path.join(CSRC, f)).read())]
    assert sorted(seen) == ["attention_tc.cu", "gemm_tcgen05.cu", "gemm_tcgen05_2cta.cu"]
