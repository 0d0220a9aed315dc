"""RMSNorm and head-norm + RoPE backward at row counts around their row groups and at every width that a row may keep in
registers, against 64-bit autograd."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

# gradients are rounded to bf16 once (2^-9 per entry at most); weight gradients are fp32 sums
DX_TOL, DW_TOL = 2.0 ** -8, 1e-4


def _bf(g, *shape, scale=1.0):
    return (scale * torch.randn(*shape, device="cuda", generator=g)).to(torch.bfloat16)


def _close(a, r, tol):
    assert (a.double() - r).norm() <= tol * r.norm() + 1e-6, float((a.double() - r).norm() / r.norm())


def _shapes(small, above):
    """Every small shape, and the shapes above one resident wave (148 SMs x 2 - 3 blocks of 8 warps), whose warps walk
    several row groups, the last one with a remainder."""
    return [s for group in small for s in group] + above


@pytest.mark.parametrize("D,rows", _shapes(
    [[(D, r) for r in (1, 3, 9, 70, 1000)] for D in (64, 128, 256, 512, 768, 1024, 1280)],
    [(64, 120_003), (256, 40_961), (768, 9_001), (1024, 9_001), (1024, 40_961)]))
@pytest.mark.parametrize("resid", [False, True])
def test_add_rmsnorm_backward(D, rows, resid):
    from cverl_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(D + rows)
    x, r, w = _bf(g, rows, D).requires_grad_(True), _bf(g, rows, D), _bf(g, D, scale=0.2).requires_grad_(True)
    w.main_grad = torch.zeros(D, device="cuda")
    dy, dh = _bf(g, rows, D), _bf(g, rows, D)
    y, h = ops.add_rmsnorm(x, r if resid else None, w, 1e-6, 1.0)
    torch.autograd.backward([y, h] if resid else [y], [dy, dh] if resid else [dy])
    hd = h.detach().double().requires_grad_(True)
    wd = w.detach().double().requires_grad_(True)
    want = hd * torch.rsqrt((hd * hd).mean(-1, keepdim=True) + 1e-6) * (1 + wd)
    dx, dw = torch.autograd.grad(want, (hd, wd), dy.double())
    _close(x.grad, dx + (dh.double() if resid else 0), DX_TOL)
    _close(w.main_grad, dw, DW_TOL)


@pytest.mark.parametrize("D,tokens,heads", _shapes([[(D, *s) for s in ((1, 1), (5, 3), (67, 16))]
                                                    for D in (64, 128, 256, 512, 768, 1024)],
                                                   [(128, 6_667, 3), (256, 2_501, 4), (768, 3_001, 3), (1024, 3_001, 3)]))
def test_gated_rmsnorm_backward(D, tokens, heads):
    from cverl_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(D + tokens)
    x, w = _bf(g, tokens, heads, D).requires_grad_(True), _bf(g, D).requires_grad_(True)
    wide = _bf(g, tokens, heads * D + 16).requires_grad_(True)      # the gate is a column range of a wider tensor
    dy = _bf(g, tokens, heads, D)
    ops.gated_rmsnorm(x, wide[:, :heads * D], w, 1e-6).backward(dy)
    xd, wd, zd = (t.detach().double().requires_grad_(True) for t in (x, w, wide))
    want = xd * torch.rsqrt((xd * xd).mean(-1, keepdim=True) + 1e-6) * wd * F.silu(zd[:, :heads * D].reshape(tokens, heads, D))
    want.backward(dy.double())
    for a, r in ((x.grad, xd.grad), (wide.grad, zd.grad), (w.grad, wd.grad)):
        _close(a, r, DX_TOL)


@pytest.mark.parametrize("D,rot,tokens,heads", _shapes([[(*d, *s) for s in ((1, 1), (3, 5), (130, 8))]
                                                        for d in ((64, 16), (128, 128), (256, 64))],
                                                       [(64, 16, 13_337, 9), (128, 128, 6_667, 6), (256, 64, 6_667, 3)]))
@pytest.mark.parametrize("use_norm", [True, False])
def test_headnorm_rope_backward(D, rot, tokens, heads, use_norm):
    from cverl_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(D + tokens)
    wide = _bf(g, tokens, heads, 2 * D).requires_grad_(True)         # strided heads, as in the fused projection
    w = _bf(g, D, scale=0.2).requires_grad_(True)
    w.main_grad = torch.zeros(D, device="cuda")
    cos, sin = ops.rope_tables(tokens + 3, rot, 1e4, wide.device)
    pos = torch.randperm(tokens + 3, device="cuda", generator=g)[:tokens].to(torch.int32)
    dy = _bf(g, tokens, heads, D)
    ops.headnorm_rope(wide[..., :D], w, cos, sin, pos, rot, 1e-6, 1.0, use_norm).backward(dy)
    xd, wd = wide.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    n = xd[..., :D]
    if use_norm:
        n = n * torch.rsqrt((n * n).mean(-1, keepdim=True) + 1e-6) * (1 + wd)
    c, s = (t[pos.long()].double().unsqueeze(1) for t in (cos, sin))
    a, b, rest = n.split([rot // 2, rot // 2, D - rot], -1)
    torch.cat([a * c - b * s, b * c + a * s, rest], -1).backward(dy.double())
    _close(wide.grad, xd.grad, DX_TOL)
    if use_norm:
        _close(w.main_grad, wd.grad, DW_TOL)
