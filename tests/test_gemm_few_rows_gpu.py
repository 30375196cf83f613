"""Few rows against a K-major weight: the swapped-operand kernel against the general one on the same rows (the terms of
a product and their order are the same, so are the bits), at the edges of its 32 / 64 / 128-row tiles, with ragged
widths and depths, uneven and empty groups, and rows past the last group."""

import pytest
import torch

from primus_turbo_b200.pytorch.core.low_precision import Float8QuantConfig, Format, ScaleDtype, ScalingGranularity
from primus_turbo_b200.pytorch.ops import gemm_fp8, grouped_gemm_fp8

pytestmark = pytest.mark.gpu
GRANS = [ScalingGranularity.TENSORWISE, ScalingGranularity.ROWWISE, ScalingGranularity.BLOCKWISE]


def _config(gran):
    return Float8QuantConfig(format=Format.E4M3, granularity=gran, scale_dtype=ScaleDtype.FP32,
                             block_size=128 if gran == ScalingGranularity.BLOCKWISE else None)


@pytest.mark.parametrize("gran", GRANS)
@pytest.mark.parametrize("n,k", [(128, 128), (16, 16), (1040, 1200), (19200, 640)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_dense_rows_equal_the_general_kernel(gran, n, k, dtype):
    torch.manual_seed(n + k)
    x = torch.randn(300, k, device="cuda", dtype=dtype)
    x[0, 0] = 16.0  # the tensorwise scale is the same for every number of rows
    w = torch.randn(n, k, device="cuda", dtype=dtype)
    full = gemm_fp8(x, w, trans_b=True, config=_config(gran))
    for m in (1, 31, 32, 33, 64, 65, 127, 128, 129):
        assert torch.equal(gemm_fp8(x[:m], w, trans_b=True, config=_config(gran)), full[:m]), m


@pytest.mark.parametrize("gran", GRANS)
@pytest.mark.parametrize("lens", [[8] * 12, [0, 65, 1, 0, 40, 0], [0, 0, 96, 0], [32, 33, 31, 0, 0],
                                  [0] * 9 + [33, 0, 1, 65, 32] + [0] * 6, [5, 0, 33, 1, 0, 0]])
@pytest.mark.parametrize("tail", [0, 7])
def test_groups_equal_the_general_kernel(gran, lens, tail):
    torch.manual_seed(len(lens))
    g, n, k = len(lens), 528, 1168
    rows = sum(lens) + tail
    x = torch.randn(rows, k, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(g, n, k, device="cuda", dtype=torch.bfloat16)
    out = grouped_gemm_fp8(x, w, torch.tensor(lens, device="cuda"), config=_config(gran))
    # the same rows with enough others past the last group to leave the rule's range (zeros are written there)
    more = torch.zeros(33 * g + rows, k, device="cuda", dtype=torch.bfloat16)
    more[:rows] = x
    want = grouped_gemm_fp8(more, w, torch.tensor(lens, device="cuda"), config=_config(gran))
    assert torch.equal(out[: sum(lens)], want[: sum(lens)])
    assert not out[sum(lens) :].any() and not want[sum(lens) :].any()


def _grads(op, x, w, gy):
    x, w = x.detach().requires_grad_(), w.detach().requires_grad_()
    return torch.autograd.grad(op(x, w), (x, w), gy)


@pytest.mark.parametrize("gran", GRANS)
@pytest.mark.parametrize("n,k", [(128, 256), (1040, 1200)])
def test_dense_backward_of_few_rows_with_mixed_formats(gran, n, k):
    """The gradient against a [K, N] weight is a product with a K-major weight: e5m2 rows, e4m3 weight."""
    cfg = _config(gran)
    cfg.format = Format.HYBRID
    torch.manual_seed(n)
    x, gy = torch.randn(300, k, device="cuda", dtype=torch.bfloat16), torch.randn(300, n, device="cuda", dtype=torch.bfloat16)
    x[0, 0], gy[0, 0] = 16.0, 16.0  # the tensorwise scales are the same for every number of rows
    w = torch.randn(k, n, device="cuda", dtype=torch.bfloat16)
    op = lambda a, b: gemm_fp8(a, b, config=cfg)  # noqa: E731
    full = _grads(op, x, w, gy)[0]
    for m in (1, 31, 33, 64, 65, 128, 129):
        assert torch.equal(_grads(op, x[:m], w, gy[:m])[0], full[:m]), m


@pytest.mark.parametrize("gran", GRANS)
@pytest.mark.parametrize("lens", [[8] * 12, [0, 65, 1, 0, 40, 0], [0, 0, 96, 0], [32, 33, 31, 0, 0], [0, 0, 0, 130, 0, 3, 0, 0],
                                  [0] * 9 + [33, 0, 1, 65, 32] + [0] * 6, [5, 0, 6, 1, 0, 0]])
def test_group_backward_of_few_rows_with_mixed_formats(gran, lens):
    cfg = _config(gran)
    cfg.format = Format.HYBRID
    torch.manual_seed(len(lens))
    g, n, k = len(lens), 528, 1168
    rows, more = sum(lens), 33 * len(lens) + sum(lens)
    x, gy = torch.randn(rows, k, device="cuda", dtype=torch.bfloat16), torch.randn(rows, n, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(g, k, n, device="cuda", dtype=torch.bfloat16)
    op = lambda a, b: grouped_gemm_fp8(a, b, torch.tensor(lens, device="cuda"), trans_b=False, config=cfg)  # noqa: E731
    got = _grads(op, x, w, gy)[0]
    pad = lambda t: torch.cat([t, t.new_zeros(more - rows, t.shape[1])])  # noqa: E731
    want = _grads(op, pad(x), w, pad(gy))[0]
    assert torch.equal(got, want[:rows])
