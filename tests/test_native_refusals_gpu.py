"""GPU: calls that the native host path leaves to the Python form -- because only that refuses them, can be recorded, or
reads what the call brings along -- and what the native path must not lose when it does take a call."""

import pytest
import torch
import torch.autograd.forward_ad as fwAD

from primus_turbo_b200 import _lib
from primus_turbo_b200.pytorch.core.low_precision import Float8QuantConfig, Format, ScaleDtype
from primus_turbo_b200.pytorch.core.low_precision import ScalingGranularity as G
from primus_turbo_b200.pytorch.core.quantized_tensor import QuantizedTensor, QuantizedTensorPair, create_quantized_weight
from primus_turbo_b200.pytorch.ops import dequantize_fp8, gemm_fp8, grouped_gemm_fp8, quantize_fp8

pytestmark = pytest.mark.gpu
DEV = "cuda"
E4 = torch.float8_e4m3fn
GRANS = [G.TENSORWISE, G.ROWWISE, G.BLOCKWISE, G.MX_BLOCKWISE]


def _config(gran, fmt=Format.E4M3):
    block = {G.BLOCKWISE: 128, G.MX_BLOCKWISE: 32}.get(gran)
    scale = ScaleDtype.E8M0 if gran == G.MX_BLOCKWISE else ScaleDtype.FP32
    return Float8QuantConfig(format=fmt, granularity=gran, block_size=block, scale_dtype=scale)


def _rand(*shape, seed=1):
    return torch.randn(*shape, device=DEV, dtype=torch.bfloat16, generator=torch.Generator(DEV).manual_seed(seed))


LENS = [33, 0, 67]


def _op(grouped, gran, fmt=Format.E4M3):
    """(op of activation and weight, activation, weight)"""
    cfg = _config(gran, fmt)
    if grouped:
        lens = torch.tensor(LENS, device=DEV)
        return lambda a, w: grouped_gemm_fp8(a, w, lens, config=cfg), _rand(100, 256), _rand(3, 384, 256, seed=2)
    return lambda a, w: gemm_fp8(a, w, trans_b=True, config=cfg), _rand(100, 256), _rand(384, 256, seed=2)


# ---- forward-mode differentiation -----------------------------------------------------------------------------
@pytest.mark.parametrize("gran", GRANS)
@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("dual", ["a", "w", "a, cached w"])
@pytest.mark.parametrize("grad_mode", [True, False])
def test_a_forward_mode_tangent_is_refused(gran, grouped, dual, grad_mode):
    """The ops have no forward-mode derivative: a tangent raises, it is not dropped."""
    op, a, w = _op(grouped, gran)
    with fwAD.dual_level(), torch.set_grad_enabled(grad_mode):
        if dual == "w":
            w = fwAD.make_dual(w, torch.ones_like(w))
        else:
            a = fwAD.make_dual(a, torch.ones_like(a))
        if "cached" in dual:
            w, _ = create_quantized_weight(w, E4, _config(gran))
        with pytest.raises((NotImplementedError, RuntimeError), match="(?i)jvp|forward mode|forward AD" if "cached" not in dual else None):
            op(a, w)


# ---- torch.jit.trace --------------------------------------------------------------------------------------------
@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("gran", GRANS)
def test_a_traced_call_runs_again_on_new_inputs(gran, grouped):
    op, a, w = _op(grouped, gran)
    other = _rand(100, 256, seed=7)
    if gran == G.MX_BLOCKWISE:  # torch cannot record the byte views of the MX form: an error, not a constant
        with pytest.raises(RuntimeError):
            torch.jit.trace(lambda x: op(x, w), (a,), check_trace=False)
        return
    traced = torch.jit.trace(lambda x: op(x, w), (a,), check_trace=False)
    assert torch.equal(traced(other), op(other, w))
    assert torch.equal(traced(a), op(a, w))


# ---- per-kernel times -------------------------------------------------------------------------------------------
@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("gran", GRANS)
def test_kernel_times_of_a_backward_whose_forward_ran_before(gran, grouped):
    op, a, w = _op(grouped, gran)
    a.requires_grad_(), w.requires_grad_()

    def log_of(forward_inside):
        with _lib.record_kernel_times() if forward_inside else torch.enable_grad():
            out = op(a, w)
        with _lib.record_kernel_times() as rec:
            torch.autograd.grad(out, (a, w), torch.ones_like(out))
        times = rec.durations_ms()
        assert all(t >= 0 for v in times.values() for t in v)
        # (the Python form of a grouped backward pass derives the group offsets once more)
        return {name: len(v) for name, v in times.items() if name != "ptb_group_offs"}

    native, python = log_of(False), log_of(True)
    assert native == python and any("gemm" in name for name in native)
    with _lib.record_kernel_times() as rec:
        pass
    out = op(a, w)  # and nothing is logged once recording has ended
    assert rec.log == {}


# ---- kernel counts ----------------------------------------------------------------------------------------------
@pytest.mark.parametrize("recorded", [False, True])
@pytest.mark.parametrize("n,offset,dtype,kernels", [
    (262144, 0, torch.bfloat16, 1), (8, 0, torch.float16, 1), (262152, 0, torch.bfloat16, 2), (262140, 0, torch.bfloat16, 2),
    (4096, 1, torch.bfloat16, 2), (4096, 0, torch.float32, 2),
])
def test_tensorwise_quantise_counts_the_kernels_it_launches(recorded, n, offset, dtype, kernels):
    """One kernel for at most 262144 16-bit elements in whole aligned vectors, else a maximum and a conversion pass."""
    x = torch.randn(n + offset, device=DEV).to(dtype)[offset:]
    before = _lib.launch_count
    with _lib.record_kernel_times() if recorded else torch.enable_grad():
        quantize_fp8(x, E4, G.TENSORWISE)
    assert _lib.launch_count - before == kernels


@pytest.mark.parametrize("recorded", [False, True])
def test_rowwise_quantise_counts_the_kernels_it_launches(recorded):
    x = _rand(64, 256)
    for axis, kernels in ((1, 1), (0, 2)):
        before = _lib.launch_count
        with _lib.record_kernel_times() if recorded else torch.enable_grad():
            quantize_fp8(x, E4, G.ROWWISE, axis=axis)
        assert _lib.launch_count - before == kernels


# ---- weights quantised ahead of time ----------------------------------------------------------------------------
def _with_scale(q, scale):
    return QuantizedTensor(q.qdata, scale, shape=q.shape, orig_dtype=q.dtype, dest_dtype=q.real_dtype, granularity=q.granularity,
                           block_size=q.block_size, scaling_recipe=q.scaling_recipe, quantized_axis=-1)


@pytest.mark.parametrize("grouped", [False, True])
def test_a_cached_weight_whose_scales_do_not_fit_is_refused(grouped):
    """A reshaped weight keeps its scales (``QuantizedTensor.view``): fewer than the product has columns is an error."""
    op, _, w = _op(grouped, G.ROWWISE)
    q, _ = create_quantized_weight(w, E4, _config(G.ROWWISE))
    wider = q.view(*w.shape[:-2], w.shape[-2] * 2, w.shape[-1] // 2)
    with torch.no_grad(), pytest.raises((AssertionError, RuntimeError)):
        op(_rand(100, 128), wider)


@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("gran", [G.TENSORWISE, G.ROWWISE, G.BLOCKWISE])
def test_a_cached_weight_with_wider_scales_is_still_taken(gran, grouped):
    op, a, w = _op(grouped, gran)
    q, _ = create_quantized_weight(w, E4, _config(gran))
    with torch.no_grad():
        assert torch.equal(op(a, _with_scale(q, q.scale_inv.double())), op(a, q))


# ---- operands that come as a pair ------------------------------------------------------------------------------------
@pytest.mark.parametrize("gran", [G.ROWWISE, G.MX_BLOCKWISE])
@pytest.mark.parametrize("grouped", [False, True])
def test_a_companion_that_does_not_fit_is_refused(gran, grouped):
    """The backward-direction copy of a pair is checked in inference as well, as the Python form does."""
    op, a, w = _op(grouped, gran)
    q, q_t = create_quantized_weight(w, E4, _config(gran), need_weight_transpose_cache=True)
    with torch.no_grad():
        assert torch.equal(op(a, QuantizedTensorPair(q, q_t)), op(a, q))
        with pytest.raises((AssertionError, AttributeError)):
            op(a, QuantizedTensorPair(q, w))
        if gran == G.MX_BLOCKWISE:
            with pytest.raises(AssertionError):
                op(a, QuantizedTensorPair(q, q))


@pytest.mark.parametrize("which", ["a", "w"])
def test_a_companion_beside_a_raw_operand_is_used(which):
    """ROWWISE: the copy handed in for the backward pass is the one the gradient is made from."""
    op, a, w = _op(False, G.ROWWISE)
    a.requires_grad_(), w.requires_grad_()
    a_t = QuantizedTensor.quantize(torch.zeros_like(a), E4, G.ROWWISE, axis=-2)
    w_t = QuantizedTensor.quantize(torch.zeros_like(w), E4, G.ROWWISE, axis=-2)
    pair = (QuantizedTensorPair(a, a_t), w) if which == "a" else (a, QuantizedTensorPair(w, w_t))
    out = op(*pair)
    ga, gw = torch.autograd.grad(out, (a, w), torch.ones_like(out))
    zero, other = (gw, ga) if which == "a" else (ga, gw)
    assert not zero.any() and other.any()


# ---- the SM cap ------------------------------------------------------------------------------------------------------
def test_num_cu_may_be_any_number():
    a, w, lens = _rand(100, 256), _rand(3, 384, 256, seed=2), torch.tensor(LENS, device=DEV)
    with torch.no_grad():
        assert torch.equal(grouped_gemm_fp8(a, w, lens, num_cu=8.0), grouped_gemm_fp8(a, w, lens, num_cu=8))


# ---- dequantise -------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("axis", [0, 1])
def test_mx_scales_of_another_byte_type_are_refused(axis):
    q, s = quantize_fp8(_rand(128, 256), E4, G.MX_BLOCKWISE, block_size=32, axis=axis)
    kw = dict(block_size=32, axis=axis)
    y = dequantize_fp8(q, torch.bfloat16, G.MX_BLOCKWISE, scale_inv=s, **kw)
    assert torch.equal(dequantize_fp8(q, torch.bfloat16, G.MX_BLOCKWISE, scale_inv=s.view(torch.uint8), **kw), y)
    for other in (torch.int8, E4, torch.float8_e5m2):
        with pytest.raises(AssertionError, match="e8m0"):
            dequantize_fp8(q, torch.bfloat16, G.MX_BLOCKWISE, scale_inv=s.view(other), **kw)
