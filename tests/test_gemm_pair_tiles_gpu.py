"""GPU: the two-CTA (256-row) tiles of the tensorwise / rowwise GEMM where they can go wrong -- row counts around the halves of
a tile, a second half without rows, column edges, odd grids, ragged row groups whose last tile fills one half only --
against dequantise-then-matmul in fp32 on identical inputs.  fp32 outputs: only the summation order may differ (5e-6)."""

import pytest
import torch

from oracle import fp8_oracle as O
from tests.gpu_util import DEV, E4, gen, randn

pytestmark = pytest.mark.gpu

from primus_turbo_b200 import _lib  # noqa: E402
from primus_turbo_b200.pytorch.core.low_precision import ScalingGranularity as G  # noqa: E402
from primus_turbo_b200.pytorch.kernels.gemm_impl import gemm_fp8_impl, grouped_gemm_fp8_impl  # noqa: E402


def _quant(x, gran, axis):
    return O.quant_rowwise(x, E4, axis) if gran == G.ROWWISE else O.quant_tensorwise(x, E4)


@pytest.mark.parametrize("gran", [G.TENSORWISE, G.ROWWISE])
@pytest.mark.parametrize("m", [1, 127, 128, 129, 255, 257, 385])
@pytest.mark.parametrize("n,k,num_sms", [(16, 128, 0), (272, 400, 3), (640, 1040, 2)])
def test_dense(gran, m, n, k, num_sms):
    g = gen(m + n)
    a, b = randn(g, m, k), randn(g, n, k, scale=0.02)
    qa, sa = _quant(a, gran, -1)
    qb, sb = _quant(b, gran, -1)
    for dt, tol in ((torch.float32, 5e-6), (torch.bfloat16, 2**-8)):
        out = gemm_fp8_impl(qa.to(DEV), sa.to(DEV), False, qb.to(DEV), sb.to(DEV), True, dt, False, gran.value, num_sms=num_sms)
        ref = (qa.float() * sa) @ (qb.float() * sb).t()
        assert _lib.gemm_status() == 0
        assert O.rel_frobenius(ref, out.float().cpu()) <= tol


@pytest.mark.parametrize("gran", [G.TENSORWISE, G.ROWWISE])
@pytest.mark.parametrize("trans_b", [True, False])
@pytest.mark.parametrize("lens", [[5, 0, 900, 257, 1500], [384, 385, 513, 640, 127], [2049]])
def test_row_groups(gran, trans_b, lens):
    n, k, tail = 272, 400, 37
    g = gen(sum(lens))
    offs = O.group_offs_from_lens(torch.tensor(lens))
    m = int(offs[-1]) + tail
    a = randn(g, m, k)
    w = randn(g, len(lens), n, k, scale=0.02) if trans_b else randn(g, len(lens), k, n, scale=0.02)
    qa, sa = _quant(a, gran, -1)
    qw, sw = _quant(w, gran, -1 if trans_b else -2)
    out = grouped_gemm_fp8_impl(qa.to(DEV), qw.to(DEV), sa.to(DEV), sw.to(DEV), torch.tensor(lens).to(DEV), offs.to(DEV), False, trans_b,
                                torch.float32, gran.value)
    assert _lib.gemm_status() == 0
    ref = O.grouped_gemm_rowwise(qa, sa, qw, sw, offs, trans_b, torch.float32)
    assert O.rel_frobenius(ref, out.cpu()) <= 5e-6
    assert bool((out[m - tail:] == 0).all())
