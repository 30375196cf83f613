"""GPU: NaN in MXFP8 blocks.  A block maximum passes over NaN, in both directions: the scale byte of a block is that of its other
values, and that of an empty maximum (0; 127 in the grouped form) where all 32 are NaN; the payload of a NaN is NaN."""

import pytest
import torch

from primus_turbo_b200.pytorch.kernels.quantization_impl import grouped_quantize_mxfp8_impl, quantize_mxfp8_impl

pytestmark = pytest.mark.gpu
FP8 = [torch.float8_e4m3fn, torch.float8_e5m2]


def _input(dtype):
    x = torch.randn(96, 256, generator=torch.Generator().manual_seed(3)).to(dtype).cuda()
    x[3, 32:64] = float("nan")  # one whole block of a row
    x[32:64, 70] = float("nan")  # one whole block of a column
    x[64:96, 128:160] = float("nan")  # a whole tile
    x[10, 5:30], x[50, 200] = float("nan"), float("nan")  # parts of blocks
    return x


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("fp8", FP8)
@pytest.mark.parametrize("tiles", [False, True])
def test_scale_bytes_pass_over_nan(dtype, fp8, tiles):
    x = _input(dtype)
    nan = x.isnan()
    want = quantize_mxfp8_impl(x.nan_to_num(nan=0.0), fp8, None, 32, True, tiles, tiles)
    got = quantize_mxfp8_impl(x, fp8, None, 32, True, tiles, tiles)
    for s in (1, 3):
        assert torch.equal(got[s].view(torch.uint8), want[s].view(torch.uint8))
    for q, where in ((0, nan), (2, nan.t())):
        g, w = got[q][:, : where.shape[1]], want[q][:, : where.shape[1]]
        assert torch.equal(g.float().isnan(), where)
        assert torch.equal(g.view(torch.uint8)[~where], w.view(torch.uint8)[~where])


@pytest.mark.parametrize("fp8", FP8)
def test_grouped_scale_bytes_pass_over_nan(fp8):
    x = _input(torch.bfloat16)
    lens = torch.tensor([40, 0, 56], device="cuda")
    offs = torch.tensor([0, 40, 40, 96], device="cuda")
    got = grouped_quantize_mxfp8_impl(x, fp8, 32, lens, offs, row_align=1)
    want = grouped_quantize_mxfp8_impl(x.nan_to_num(nan=0.0), fp8, 32, lens, offs, row_align=1)
    assert torch.equal(got[1].view(torch.uint8)[:96], want[1].view(torch.uint8)[:96])
    assert int(got[1].view(torch.uint8)[3, 1]) == 127
    assert torch.equal(got[3].view(torch.uint8), want[3].view(torch.uint8))
    assert torch.equal(got[0][:96].float().isnan(), x.isnan())
