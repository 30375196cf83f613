"""MoE row movement and the activation at the sizes where their kernels change form: expert counts around the 64-expert
tile, token counts around the 256-token block, widths around the vector slices, more rows than are routed, and every
number of warps per activation row."""

import pytest
import torch

from primus_turbo_b200.pytorch.ops.activation import swiglu_with_probs
from primus_turbo_b200.pytorch.ops.moe import token_permute, token_unpermute

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T,E", [(1, 1), (255, 17), (256, 64), (257, 65), (700, 130), (40, 1024)])
@pytest.mark.parametrize("H", [8, 24, 520, 1032])
@pytest.mark.parametrize("merge", [False, True])
def test_rows_there_and_back(T, E, H, merge):
    torch.manual_seed(T + E + H)
    mask = torch.rand(T, E, device=DEV) < min(1.0, 4 / E)
    n, extra = int(mask.sum()), 3
    x = torch.randn(T, H, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    probs = (torch.rand(T, E, device=DEV) * mask).requires_grad_(True)
    rows, pp, idx, counts = token_permute(x, n + extra, probs=probs, routing_map=mask)
    order = mask.t().nonzero()  # expert-major, tokens in order
    assert torch.equal(counts, mask.sum(0)) and torch.equal(idx[:n], order[:, 1]) and bool((idx[n:] == -1).all())
    assert torch.equal(rows[:n], x[order[:, 1]]) and not rows[n:].any()
    assert torch.equal(pp[:n], probs[order[:, 1], order[:, 0]]) and not pp[n:].any()
    gpp = torch.randn(n + extra, device=DEV)
    (gp,) = torch.autograd.grad(pp, probs, gpp, retain_graph=True)
    want = torch.zeros_like(probs)
    want[order[:, 1], order[:, 0]] = gpp[:n]
    assert torch.equal(gp, want)

    y = torch.randn(n + extra, H, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    out = token_unpermute(y, idx, merging_probs=probs if merge else None, restore_shape=(T, H), routing_map=mask)
    acc = torch.zeros(T, H, device=DEV)
    for e in range(E):  # one addition per copy, experts in order
        sel = order[:, 0] == e
        p = probs[order[sel, 1], e].unsqueeze(1) if merge else 1.0
        acc[order[sel, 1]] += y[:n][sel].float() * p
    assert torch.equal(out, acc.to(torch.bfloat16))
    g = torch.randn(T, H, device=DEV, dtype=torch.bfloat16)
    grads = torch.autograd.grad(out, (y, probs) if merge else (y,), g)
    scale = probs[order[:, 1], order[:, 0]].unsqueeze(1) if merge else 1.0
    assert torch.equal(grads[0][:n], (g[order[:, 1]].float() * scale).to(torch.bfloat16)) and not grads[0][n:].any()
    if merge:
        dot = (g[order[:, 1]].double() * y[:n].double()).sum(1)
        size = (g[order[:, 1]].double() * y[:n].double()).abs().sum(1)
        # H products added in fp32, at most H / 32 + 13 additions in a row, each within 2^-24 of its partial sum
        assert bool(((grads[1][order[:, 1], order[:, 0]] - dot).abs() <= size * (H / 32 + 16) * 2.0**-24).all())
        assert not grads[1][~mask].any()


@pytest.mark.parametrize("rows", [1, 7, 9])
@pytest.mark.parametrize("h", [8, 1024, 1032, 2048, 2056, 4096, 4104, 8200])
def test_activation_row_warps(rows, h):
    torch.manual_seed(h)
    x = torch.randn(rows, 2 * h, device=DEV, dtype=torch.float16, requires_grad=True)
    p = torch.rand(rows, device=DEV, requires_grad=True)
    g = torch.randn(rows, h, device=DEV, dtype=torch.float16)
    out = swiglu_with_probs(x, p)
    gx, gp = torch.autograd.grad(out, (x, p), g)
    xd, pd = x.detach().double().requires_grad_(True), p.detach().double().requires_grad_(True)
    ref = torch.nn.functional.silu(xd[:, :h]) * xd[:, h:] * pd[:, None]
    rx, rp = torch.autograd.grad(ref, (xd, pd), g.double())
    # one rounding to fp16 (2^-11) and a few fp32 operations; fp16 is subnormal below 6e-5
    torch.testing.assert_close(out.double(), ref, rtol=2.0**-10, atol=1e-6)
    torch.testing.assert_close(gx.double(), rx, rtol=2.0**-10, atol=2e-6)
    size = (g.double() * (ref / pd[:, None]).detach()).abs().sum(1)
    assert bool(((gp - rp).abs() <= size * (h / 256 + 40) * 2.0**-23).all())
