"""The fused expert block against a plain fp32 loop over the experts."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _oracle(x, ids, w, gate_up, down):
    out, norms = torch.zeros_like(x), torch.zeros(w.shape, device=w.device)
    for e in range(gate_up.shape[0]):
        tok, slot = (ids == e).nonzero(as_tuple=True)
        if tok.numel():
            a, u = (x[tok] @ gate_up[e].t()).chunk(2, -1)
            y = (F.silu(a) * u) @ down[e].t()
            norms[tok, slot] = y.detach().norm(dim=-1)
            out = out.index_add(0, tok, y * w[tok, slot].unsqueeze(-1))
    return out, norms


@pytest.mark.parametrize("T,E,k,H,inter,one", [(1, 4, 1, 64, 64, False), (5, 8, 3, 72, 40, False), (129, 4, 2, 2056, 96, False),
                                               (300, 16, 8, 256, 128, False), (260, 6, 1, 128, 64, True)])
@pytest.mark.parametrize("main_grad", [False, True])
def test_expert_block_matches_a_loop_over_experts(T, E, k, H, inter, one, main_grad):
    from cverl_b200 import _native as nv
    from cverl_b200.ops.moe import moe_experts, supported
    g = torch.Generator(device="cuda").manual_seed(T + E)

    def bf(*s, scale=1.0):
        return (scale * torch.randn(*s, device="cuda", generator=g)).to(torch.bfloat16)
    x, gu, dn = bf(T, H), bf(E, 2 * inter, H, scale=H ** -0.5), bf(E, H, inter, scale=inter ** -0.5)
    ids = torch.rand(T, E, device="cuda", generator=g).topk(k, -1).indices
    if one:
        ids = torch.full((T, 1), 2, device="cuda")              # one expert takes every token, the others none
    w = torch.softmax(torch.randn(T, k, device="cuda", generator=g), -1)
    dy = bf(T, H)
    ref = [t.float().requires_grad_(True) for t in (x, w, gu, dn)]
    want, norms = _oracle(ref[0], ids, *ref[1:])
    want.backward(dy.float())
    got = [t.detach().clone().requires_grad_(True) for t in (x, w, gu, dn)]
    if main_grad:
        for p in got[2:]:
            p.main_grad = torch.ones(p.shape, device="cuda")
    assert supported(got[0], got[2], got[3], k)
    y = moe_experts(got[0], ids, *got[1:])
    y.backward(dy)
    nv.check_status()
    # five bf16 roundings in a row (gate|up, activation, expert output, result; as many backward): 2^-9 each
    tol = 5 * 2.0 ** -9
    assert (y.float() - want).norm() <= tol * want.norm()
    for a, r in zip(got, ref):
        ga = a.main_grad - 1 if main_grad and a.dim() == 3 else a.grad
        # a routing weight's gradient is <dy, y> and may cancel: its error is relative to |dy| |y|, not to the result
        size = (dy.float().norm(dim=-1, keepdim=True) * norms).norm() if r is ref[1] else r.grad.norm()
        assert (ga.float() - r.grad).norm() <= tol * size + 1e-6 * r.grad.numel() ** 0.5


@pytest.mark.parametrize("layout", ["strided", "misaligned"])
def test_expert_block_copies_rows_that_cannot_be_read_in_place(layout):
    """Token rows and output gradients with a row stride, or 2 bytes off a 16-byte boundary: the result of packed ones."""
    from cverl_b200 import _native as nv
    from cverl_b200.ops.moe import moe_experts, supported
    g = torch.Generator(device="cuda").manual_seed(3)
    T, E, k, H, inter = 130, 4, 2, 136, 64

    def bf(*s, scale=1.0):
        return (scale * torch.randn(*s, device="cuda", generator=g)).to(torch.bfloat16)

    def odd(t):
        if layout == "strided":
            return torch.stack([t, t], 1)[:, 0]
        buf = torch.empty(t.numel() + 8, device="cuda", dtype=t.dtype)
        return buf[1:1 + t.numel()].view(t.shape).copy_(t)
    x, dy, gu, dn = bf(T, H), bf(T, H), bf(E, 2 * inter, H, scale=H ** -0.5), bf(E, H, inter, scale=inter ** -0.5)
    ids = torch.rand(T, E, device="cuda", generator=g).topk(k, -1).indices
    w = torch.softmax(torch.randn(T, k, device="cuda", generator=g), -1)
    res = []
    for make in (lambda t: t, odd):
        a, b = make(x).detach().requires_grad_(True), w.clone().requires_grad_(True)
        assert supported(a, gu, dn, k)
        y = moe_experts(a, ids, b, gu, dn)
        res.append((y.detach(),) + torch.autograd.grad(y, (a, b), make(dy)))
    nv.check_status()
    for p, q in zip(*res):
        assert torch.equal(p, q)
