"""What the two CTAs of a pair owe each other: the order the source sets up a pair in (CPU)."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "primus_turbo_b200" / "csrc"


def _source():
    text = "".join(p.read_text() for p in sorted(CSRC.glob("ptb_gemm*.cu*")))
    return re.sub(r"//[^\n]*", "", text)


def test_a_pair_meets_before_it_allocates_tensor_memory():
    """The two-CTA allocation is made by both CTAs together: it comes after a cluster barrier, and that after the mbarriers."""
    text = _source()
    kernel = text[text.index("fp8_gemm_kernel(const __grid_constant__") :]
    init, alloc = kernel.index("fence.mbarrier_init"), kernel.index("tcgen05.alloc.cta_group::2")
    assert init < kernel.find("cluster_sync()") < alloc < kernel.index("grid_dep_begin()")
