"""GPU: chains of small calls enqueued without a host synchronisation.  Their kernels start while the one before them ends, so
what is read too early -- a scale, an FP8 copy, a workspace -- shows here and not in tests that wait after every GEMM:
the outputs have to be those of the same calls made one at a time."""

import pytest
import torch

from primus_turbo_b200 import _lib, _native
from primus_turbo_b200.pytorch.core.low_precision import Float8QuantConfig, Format, ScaleDtype
from primus_turbo_b200.pytorch.core.low_precision import ScalingGranularity as G
from primus_turbo_b200.pytorch.core.quantized_tensor import create_quantized_weight
from primus_turbo_b200.pytorch.ops import dequantize_fp8, gemm_fp8, grouped_gemm_fp8, quantize_fp8

pytestmark = pytest.mark.gpu
DEV = "cuda"
GRANS = [G.TENSORWISE, G.ROWWISE, G.BLOCKWISE, G.MX_BLOCKWISE]
ROUNDS = 12


@pytest.fixture
def no_status_wait(monkeypatch):
    """The wait for the device after every GEMM, off on both host paths."""
    before = _lib._DEBUG_STATUS
    monkeypatch.setattr(_lib, "_DEBUG_STATUS", False)
    _native.ext.set_check_status(False)
    yield
    _native.ext.set_check_status(before)


def _config(gran):
    block = {G.BLOCKWISE: 128, G.MX_BLOCKWISE: 32}.get(gran)
    scale = ScaleDtype.E8M0 if gran == G.MX_BLOCKWISE else ScaleDtype.FP32
    return Float8QuantConfig(format=Format.HYBRID, granularity=gran, block_size=block, scale_dtype=scale)


def _steps(gran):
    """(activation rows, K, step of the activation buffer): forward, forward and backward, decode rows, row groups, a cached
    weight, and a quantise that reads what a GEMM wrote."""
    g = torch.Generator(DEV).manual_seed(11)
    rand = lambda *s: torch.randn(*s, device=DEV, dtype=torch.bfloat16, generator=g)  # noqa: E731
    cfg = _config(gran)
    w, wg, gy = rand(384, 256), rand(4, 384, 256), rand(320, 384)
    lens = torch.tensor([100, 0, 37, 183], device=DEV)
    few = torch.tensor([3, 0, 1, 4], device=DEV)
    cached, _ = create_quantized_weight(w, torch.float8_e4m3fn, cfg)
    quant = dict(block_size=cfg.block_size, axis=None if gran == G.TENSORWISE else 1)

    def train(op, x, weight):
        x, weight = x.detach().requires_grad_(), weight.detach().requires_grad_()
        out = op(x, weight)
        return [out.detach(), *torch.autograd.grad(out, (x, weight), gy)]

    @torch.no_grad()
    def chain(x):
        """The second product reads the first one's output."""
        y = gemm_fp8(x, w, trans_b=True, config=cfg)
        q, s = quantize_fp8(y, torch.float8_e4m3fn, gran, **quant)
        return [y, gemm_fp8(y[:, :256].contiguous(), w, trans_b=True, config=cfg), dequantize_fp8(q, torch.bfloat16, gran, scale_inv=s, **quant)]

    def infer(op):
        def step(x):
            with torch.no_grad():
                return [op(x)]
        return step

    return [
        (320, infer(lambda x: gemm_fp8(x, w, trans_b=True, config=cfg))),
        (320, lambda x: train(lambda a, b: gemm_fp8(a, b, trans_b=True, config=cfg), x, w)),
        (8, infer(lambda x: gemm_fp8(x, cached, trans_b=True, config=cfg))),
        (320, lambda x: train(lambda a, b: grouped_gemm_fp8(a, b, lens, config=cfg), x, wg)),
        (8, infer(lambda x: grouped_gemm_fp8(x, wg, few, config=cfg))),
        (320, chain),
    ]


@pytest.mark.parametrize("grans", [[g] for g in GRANS] + [GRANS])
def test_a_chain_without_waits_gives_what_single_calls_give(no_status_wait, grans):
    steps = [s for gran in grans for s in _steps(gran)]
    g = torch.Generator(DEV).manual_seed(12)
    inputs = [torch.randn(320, 256, device=DEV, dtype=torch.bfloat16, generator=g) * (1.0 + 3.0 * i) for i in range(ROUNDS)]
    want = []
    for x in inputs:
        for rows, step in steps:
            torch.cuda.synchronize()
            want.append(step(x[:rows]))
    torch.cuda.synchronize()
    assert _lib.gemm_status() == 0
    for _ in range(3):
        buffer = torch.empty_like(inputs[0])  # one buffer for all: a late read would see the next round's values
        got = []
        for x in inputs:
            buffer.copy_(x)
            for rows, step in steps:
                got.append(step(buffer[:rows]))
        torch.cuda.synchronize()
        assert _lib.gemm_status() == 0
        for i, (a, b) in enumerate(zip(got, want)):
            assert all(torch.equal(x, y) for x, y in zip(a, b)), (i // len(steps), i % len(steps))
