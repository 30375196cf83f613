"""GPU: the native host path of ``gemm_fp8`` / ``grouped_gemm_fp8`` gives what the Python path gives, bit for bit -- forward
alone, with one gradient wanted and with both, raw and cached weights, transposed and non-contiguous operands.  The
Python path is what runs while per-kernel times are recorded."""

import pytest
import torch

from primus_turbo_b200 import _lib
from primus_turbo_b200.pytorch.core.low_precision import Float8QuantConfig, Format, ScaleDtype
from primus_turbo_b200.pytorch.core.low_precision import ScalingGranularity as G
from primus_turbo_b200.pytorch.core.quantized_tensor import create_quantized_weight
from primus_turbo_b200.pytorch.ops import gemm_fp8, grouped_gemm_fp8

pytestmark = pytest.mark.gpu
DEV = "cuda"
GRANS = [G.TENSORWISE, G.ROWWISE, G.BLOCKWISE, G.MX_BLOCKWISE]


def _config(gran, fmt=Format.HYBRID):
    block = {G.BLOCKWISE: 128, G.MX_BLOCKWISE: 32}.get(gran)
    scale = ScaleDtype.E8M0 if gran == G.MX_BLOCKWISE else ScaleDtype.FP32
    return Float8QuantConfig(format=fmt, granularity=gran, block_size=block, scale_dtype=scale)


def _both_ways(op, a, b, wanted, gy):
    a, b = a.detach().requires_grad_("a" in wanted), b.detach().requires_grad_("b" in wanted)

    def once():
        out = op(a, b)
        leaves = [t for t in (a, b) if t.requires_grad]
        return [out.detach(), *(torch.autograd.grad(out, leaves, gy) if leaves else ())]

    before = _lib.launch_count
    native = once()
    assert _lib.launch_count > before
    with _lib.record_kernel_times():
        python = once()
    assert len(native) == len(python)
    for x, y in zip(native, python):
        assert x.shape == y.shape and x.dtype == y.dtype and torch.equal(x, y)


@pytest.mark.parametrize("gran", GRANS)
@pytest.mark.parametrize("wanted", ["", "a", "b", "ab"])
@pytest.mark.parametrize("trans_b", [True, False])
def test_dense(gran, wanted, trans_b):
    if gran == G.MX_BLOCKWISE and not trans_b:
        pytest.skip("MX takes transposed weights only")
    m, n, k = 193, 288, 416
    g = torch.Generator(DEV).manual_seed(m)
    a = torch.randn(k, m, device=DEV, generator=g, dtype=torch.bfloat16).t()  # not contiguous
    b = torch.randn((n, k) if trans_b else (k, n), device=DEV, generator=g, dtype=torch.bfloat16)
    gy = torch.randn(m, n, device=DEV, generator=g, dtype=torch.bfloat16)
    cfg = _config(gran)
    _both_ways(lambda x, w: gemm_fp8(x, w, trans_b=trans_b, config=cfg), a, b, wanted, gy)


@pytest.mark.parametrize("gran", GRANS)
@pytest.mark.parametrize("wanted", ["", "a", "b", "ab"])
@pytest.mark.parametrize("tail", [0, 9])
def test_grouped(gran, wanted, tail):
    lens = torch.tensor([5, 0, 130, 1, 256], device=DEV)
    m, n, k = 392 + tail, 256, 384
    g = torch.Generator(DEV).manual_seed(m)
    a = torch.randn(m, k, device=DEV, generator=g, dtype=torch.bfloat16)
    b = torch.randn(5, n, k, device=DEV, generator=g, dtype=torch.bfloat16)
    gy = torch.randn(m, n, device=DEV, generator=g, dtype=torch.bfloat16)
    cfg = _config(gran)
    _both_ways(lambda x, w: grouped_gemm_fp8(x, w, lens, config=cfg), a, b, wanted, gy)


@pytest.mark.parametrize("gran", GRANS)
def test_cached_weight_in_inference(gran):
    g = torch.Generator(DEV).manual_seed(3)
    a = torch.randn(70, 384, device=DEV, generator=g, dtype=torch.bfloat16)
    w = torch.randn(2, 256, 384, device=DEV, generator=g, dtype=torch.bfloat16)
    lens = torch.tensor([33, 37], device=DEV)
    cfg = _config(gran, Format.E4M3)
    qw, _ = create_quantized_weight(w, torch.float8_e4m3fn, cfg)
    q0, _ = create_quantized_weight(w[0].contiguous(), torch.float8_e4m3fn, cfg)
    with torch.no_grad():
        assert torch.equal(grouped_gemm_fp8(a, qw, lens, config=cfg), grouped_gemm_fp8(a, w, lens, config=cfg))
        assert torch.equal(gemm_fp8(a, q0, trans_b=True, config=cfg), gemm_fp8(a, w[0], trans_b=True, config=cfg))
