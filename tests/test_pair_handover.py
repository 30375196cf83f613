"""What one CTA of a pair hands to the other: which barrier operations the source uses for it (CPU), and the unpadded
variable-K groups whose last block is cleared in both CTAs before the MMA reads it (GPU)."""

import re
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "primus_turbo_b200" / "csrc"


def _source():
    text = "".join(p.read_text() for p in sorted(CSRC.glob("ptb_gemm*.cu*")))
    return re.sub(r"//[^\n]*", "", text)


def test_relaxed_arrivals_hand_over_tensor_memory_only():
    """A relaxed arrival publishes no write, so none may signal that shared memory is ready for the other CTA."""
    text = _source()
    relaxed = [m for m in re.finditer(r"void (\w+)\(uint32_t \w+\) \{\s*asm volatile\(\"mbarrier\.arrive\.relaxed\.cluster", text)]
    assert len(relaxed) == 1
    calls = re.findall(rf"(?<!void ){relaxed[0].group(1)}\(([^;]*)\);", text)
    assert calls and all("tmem_empty" in c for c in calls)


def test_one_cta_clears_both_halves_before_it_completes_the_stage():
    """The rows are cleared, fenced and reported by a warp of the CTA whose MMA reads them; the other CTA signals no `full`."""
    text = _source()
    warp3 = text[text.index("else if (CTAS == 2 && warp == 3)") :]
    order = ["while (leader &&", "mbar_wait(smem_u32(&ctl->cut[s])", "clear_tail_rows_pair<", "__syncwarp()", "mbar_arrive(smem_u32(&ctl->full[s]))"]
    assert sorted(map(warp3.index, order)) == list(map(warp3.index, order))
    clear = text[text.index("void clear_tail_rows_pair(") :]
    assert clear.index("st_zero16_cluster(") < clear.index("fence.proxy.async;")


def test_a_pair_meets_before_it_allocates_tensor_memory():
    """The two-CTA allocation is made by both CTAs together: it comes after a cluster barrier, and that after the mbarriers."""
    text = _source()
    kernel = text[text.index("fp8_gemm_kernel(const __grid_constant__") :]
    init, alloc = kernel.index("fence.mbarrier_init"), kernel.index("tcgen05.alloc.cta_group::2")
    assert init < kernel.find("cluster_sync()") < alloc < kernel.index("grid_dep_begin()")


@pytest.mark.gpu
@pytest.mark.parametrize("gran", ["TENSORWISE", "ROWWISE"])
def test_rows_of_neighbouring_groups_never_reach_the_product(gran):
    """Every second group holds FP8 NaN bytes only; the groups between them, whose last block reaches into those rows, come
    out finite, right, and the same in every launch.  fp32 outputs: only the summation order may differ (5e-6)."""
    from oracle import fp8_oracle as O
    from primus_turbo_b200 import _lib
    from primus_turbo_b200.pytorch.core.low_precision import ScalingGranularity
    from primus_turbo_b200.pytorch.kernels.gemm_impl import grouped_gemm_fp8_variable_k_impl
    from tests.gpu_util import DEV, E4, gen, randn

    g = gen(5)
    lens = torch.tensor([1, 3, 127, 9, 129, 1, 255, 40, 300, 7] * 4)
    offs = O.group_offs_from_lens(lens)
    m, n, k = int(offs[-1]) + 50, 272, 400
    quant = (lambda t: O.quant_rowwise(t, E4, -2)) if gran == "ROWWISE" else (lambda t: O.quant_tensorwise(t, E4))
    (xq, xs), (gq, gs) = quant(randn(g, m, k)), quant(randn(g, m, n, scale=1e-3))
    xb, gb = xq.view(torch.uint8).clone(), gq.view(torch.uint8).clone()
    for i in range(1, len(lens), 2):
        xb[offs[i] : offs[i + 1]], gb[offs[i] : offs[i + 1]] = 0x7F, 0xFF
    xb[offs[-1] :], gb[offs[-1] :] = 0xFF, 0x7F
    args = [t.to(DEV) for t in (xb.view(E4), gb.view(E4), xs, gs, lens, offs)]
    outs = [grouped_gemm_fp8_variable_k_impl(*args, True, False, True, torch.float32, ScalingGranularity[gran].value)[::2] for _ in range(20)]
    assert _lib.gemm_status() == 0
    assert all(torch.equal(o, outs[0]) for o in outs)
    for i, o in zip(range(0, len(lens), 2), outs[0].cpu()):
        lo, hi = int(offs[i]), int(offs[i + 1])
        ref = (gq[lo:hi].float().t() @ xq[lo:hi].float()) * (gs.view(-1, 1) if gran == "ROWWISE" else gs) * xs.view(1, -1)
        assert bool(torch.isfinite(o).all()) and O.rel_frobenius(ref, o) <= 5e-6
