"""GPU: the native host path of ``gemm_fp8`` / ``grouped_gemm_fp8`` gives what the Python path gives, bit for bit -- forward
alone, with one gradient wanted and with both, raw and cached weights, transposed and non-contiguous operands.  The
Python path is what runs while per-kernel times are recorded."""

import pytest
import torch

from primus_turbo_b200 import _lib, _native
from primus_turbo_b200.pytorch.core.low_precision import Float8QuantConfig, Format, ScaleDtype
from primus_turbo_b200.pytorch.core.low_precision import ScalingGranularity as G
from primus_turbo_b200.pytorch.core.quantized_tensor import create_quantized_weight
from primus_turbo_b200.pytorch.ops import dequantize_fp8, gemm_fp8, grouped_gemm_fp8, quantize_fp8, quantize_fp8_with_trans

pytestmark = pytest.mark.gpu
DEV = "cuda"
GRANS = [G.TENSORWISE, G.ROWWISE, G.BLOCKWISE, G.MX_BLOCKWISE]


def _config(gran, fmt=Format.HYBRID):
    block = {G.BLOCKWISE: 128, G.MX_BLOCKWISE: 32}.get(gran)
    scale = ScaleDtype.E8M0 if gran == G.MX_BLOCKWISE else ScaleDtype.FP32
    return Float8QuantConfig(format=fmt, granularity=gran, block_size=block, scale_dtype=scale)


@pytest.fixture
def path(monkeypatch):
    """``path(f)`` -> what ``f()`` gives and which host path its library calls were made on."""
    python = []
    call = _lib.call
    monkeypatch.setattr(_lib, "call", lambda name, *a: (python.append(name), call(name, *a))[1])

    def run(f):
        del python[:]
        before = _native.ext.calls()
        out = f()
        native = _native.ext.calls() - before
        assert native or python
        return out, "mixed" if native and python else "native" if native else "python"

    return run


def _both_ways(path, op, a, b, wanted, gy):
    a, b = a.detach().requires_grad_("a" in wanted), b.detach().requires_grad_("b" in wanted)

    def once():
        out = op(a, b)
        leaves = [t for t in (a, b) if t.requires_grad]
        return [out.detach(), *(torch.autograd.grad(out, leaves, gy) if leaves else ())]

    native, how = path(once)
    assert how == "native"
    with _lib.record_kernel_times():
        python, how = path(once)
    assert how == "python"
    assert len(native) == len(python)
    for x, y in zip(native, python):
        assert x.shape == y.shape and x.dtype == y.dtype and torch.equal(x, y)


@pytest.mark.parametrize("gran", GRANS)
@pytest.mark.parametrize("wanted", ["", "a", "b", "ab"])
@pytest.mark.parametrize("trans_b", [True, False])
def test_dense(path, gran, wanted, trans_b):
    if gran == G.MX_BLOCKWISE and not trans_b:
        pytest.skip("MX takes transposed weights only")
    m, n, k = 193, 288, 416
    g = torch.Generator(DEV).manual_seed(m)
    a = torch.randn(k, m, device=DEV, generator=g, dtype=torch.bfloat16).t()  # not contiguous
    b = torch.randn((n, k) if trans_b else (k, n), device=DEV, generator=g, dtype=torch.bfloat16)
    gy = torch.randn(m, n, device=DEV, generator=g, dtype=torch.bfloat16)
    cfg = _config(gran)
    _both_ways(path, lambda x, w: gemm_fp8(x, w, trans_b=trans_b, config=cfg), a, b, wanted, gy)


@pytest.mark.parametrize("gran", GRANS)
@pytest.mark.parametrize("wanted", ["", "a", "b", "ab"])
@pytest.mark.parametrize("tail", [0, 9])
def test_grouped(path, gran, wanted, tail):
    lens = torch.tensor([5, 0, 130, 1, 256], device=DEV)
    m, n, k = 392 + tail, 256, 384
    g = torch.Generator(DEV).manual_seed(m)
    a = torch.randn(m, k, device=DEV, generator=g, dtype=torch.bfloat16)
    b = torch.randn(5, n, k, device=DEV, generator=g, dtype=torch.bfloat16)
    gy = torch.randn(m, n, device=DEV, generator=g, dtype=torch.bfloat16)
    cfg = _config(gran)
    _both_ways(path, lambda x, w: grouped_gemm_fp8(x, w, lens, config=cfg), a, b, wanted, gy)


@pytest.mark.parametrize("gran", GRANS)
def test_cached_weight_in_inference(path, gran):
    g = torch.Generator(DEV).manual_seed(3)
    a = torch.randn(70, 384, device=DEV, generator=g, dtype=torch.bfloat16)
    w = torch.randn(2, 256, 384, device=DEV, generator=g, dtype=torch.bfloat16)
    lens = torch.tensor([33, 37], device=DEV)
    cfg = _config(gran, Format.E4M3)
    qw, _ = create_quantized_weight(w, torch.float8_e4m3fn, cfg)
    q0, _ = create_quantized_weight(w[0].contiguous(), torch.float8_e4m3fn, cfg)
    with torch.no_grad():
        for cached, raw in ((lambda: grouped_gemm_fp8(a, qw, lens, config=cfg), lambda: grouped_gemm_fp8(a, w, lens, config=cfg)),
                            (lambda: gemm_fp8(a, q0, trans_b=True, config=cfg), lambda: gemm_fp8(a, w[0], trans_b=True, config=cfg))):
            out, how = path(cached)
            assert how == "native"
            with _lib.record_kernel_times():
                want, how = path(cached)
            assert how == "python" and torch.equal(out, want) and torch.equal(out, raw())


@pytest.mark.parametrize("gran", GRANS)
@pytest.mark.parametrize("axis", [0, 1])
def test_quantise_and_dequantise(path, gran, axis):
    x = torch.randn(200, 416, device=DEV, dtype=torch.bfloat16, generator=torch.Generator(DEV).manual_seed(9))
    kw = dict(block_size=_config(gran).block_size, axis=None if gran == G.TENSORWISE else axis)

    def there_and_back():
        q, s = quantize_fp8(x, torch.float8_e4m3fn, gran, **kw)
        both = ()
        if gran in (G.BLOCKWISE, G.MX_BLOCKWISE):
            both = quantize_fp8_with_trans(x, torch.float8_e5m2, gran, block_size=kw["block_size"])
        return [q, s, *both, dequantize_fp8(q, torch.bfloat16, gran, scale_inv=s, **kw)]

    native, how = path(there_and_back)
    assert how == "native"
    with _lib.record_kernel_times():
        python, how = path(there_and_back)
    assert how == "python" and len(native) == len(python)
    for a, b in zip(native, python):
        assert a.shape == b.shape and a.dtype == b.dtype
        view = torch.int32 if a.dtype == torch.float32 else torch.int16 if a.dtype == torch.bfloat16 else torch.uint8
        assert torch.equal(a.view(view), b.view(view))
