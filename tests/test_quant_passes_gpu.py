"""The streaming passes of the quantise family at the sizes where their loops end: unrolled bodies and remainders, rows
held in registers and rows that are not, vector and element forms of dequantise, and the FP8-to-FP8 requantise."""

import pytest
import torch

from primus_turbo_b200 import _lib
from primus_turbo_b200._lib import dtype_code, ptr, stream_of
from primus_turbo_b200.pytorch.core.low_precision import ScalingGranularity, float8_e4m3, float8_e5m2
from primus_turbo_b200.pytorch.ops import dequantize_fp8, quantize_fp8

pytestmark = pytest.mark.gpu
FMAX = {float8_e4m3: 448.0, float8_e5m2: 57344.0}


def _rows_ref(x, fp8, dim):
    """fp32 restatement: scale = fmax / max(amax, 1e-12); bytes and scales have one right value."""
    amax = x.float().abs().amax(dim, keepdim=True).clamp(min=1e-12)
    scale = torch.full_like(amax, FMAX[fp8]) / amax
    q = (x.float() * scale).clamp(-FMAX[fp8], FMAX[fp8]).to(fp8)
    return q.view(torch.uint8), torch.ones_like(scale) / scale


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n", [8, 4096 * 8, 262144 - 8, 262144, 262144 + 8, 4 * 592 * 512 * 8 - 8, 4 * 592 * 512 * 8 + 24, 4 * 592 * 512 * 8 + 5])
def test_tensorwise_pass_ends(dtype, n):
    x = torch.randn(n, device="cuda").to(dtype)
    x[-1] = 40.0  # the maximum sits in the last vector or in the element tail
    q, s = quantize_fp8(x, float8_e4m3, ScalingGranularity.TENSORWISE)
    ref, inv = _rows_ref(x.view(1, -1), float8_e4m3, 1)
    assert torch.equal(q.view(torch.uint8), ref.view(-1)) and torch.equal(s.view(1), inv.view(1))
    y = dequantize_fp8(q, dtype, ScalingGranularity.TENSORWISE, scale_inv=s)
    assert torch.equal(y, (q.float() * s).to(dtype))


@pytest.mark.parametrize("fp8", [float8_e4m3, float8_e5m2])
@pytest.mark.parametrize("cols", [8, 2048, 2056, 8184, 8192, 8200, 1001])
def test_inner_rows(fp8, cols):
    x = torch.randn(5, cols, device="cuda", dtype=torch.bfloat16)
    x[:, -1] = 9.0
    q, s = quantize_fp8(x, fp8, ScalingGranularity.ROWWISE, axis=1)
    ref, inv = _rows_ref(x, fp8, 1)
    assert torch.equal(q.view(torch.uint8), ref) and torch.equal(s.view(-1), inv.view(-1))


@pytest.mark.parametrize("out", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(1, 8), (37, 264), (300, 1032), (129, 333)])
@pytest.mark.parametrize("axis", [0, 1])
def test_dequantise_rows_and_columns(out, shape, axis):
    q = torch.randn(shape, device="cuda").to(float8_e4m3)
    s = torch.rand((1, shape[1]) if axis == 0 else (shape[0], 1), device="cuda") + 0.5
    y = dequantize_fp8(q, out, ScalingGranularity.ROWWISE, axis=axis, scale_inv=s)
    assert torch.equal(y, (q.float() * s).to(out))
    nb = (shape[axis] + 127) // 128
    s = torch.rand((nb, shape[1]) if axis == 0 else (shape[0], nb), device="cuda") + 0.5
    y = dequantize_fp8(q, out, ScalingGranularity.BLOCKWISE, block_size=128, axis=axis, scale_inv=s)
    full = s.repeat_interleave(128, axis).narrow(axis, 0, shape[axis])
    assert torch.equal(y, (q.float() * full).to(out))


@pytest.mark.parametrize("fp8", [float8_e4m3, float8_e5m2])
@pytest.mark.parametrize("hp", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(1, 1, 8), (1, 31, 264), (1, 300, 2056), (3, 129, 72), (2, 257, 333)])
def test_requantise_is_dequantise_then_quantise(fp8, hp, shape):
    B, M, N = shape
    x = torch.randn(shape, device="cuda").to(hp)
    x[0, 0, 0] = 0.0
    q, s = quantize_fp8(x, fp8, ScalingGranularity.ROWWISE, axis=2)
    want_q, want_s = quantize_fp8(
        dequantize_fp8(q, hp, ScalingGranularity.ROWWISE, axis=2, scale_inv=s), fp8, ScalingGranularity.ROWWISE, axis=1
    )
    got_q, got_s = torch.empty_like(q), torch.empty((B, 1, N), device="cuda")
    ws = torch.full((B * N,), float("nan"), device="cuda")
    _lib.call("ptb_requant_fp8_rowwise", ptr(q), dtype_code(fp8), ptr(s), dtype_code(hp), B, M, N, ptr(got_q), ptr(got_s),
              ptr(ws), stream_of(q))
    assert torch.equal(got_q.view(torch.uint8), want_q.view(torch.uint8)) and torch.equal(got_s, want_s.view_as(got_s))
