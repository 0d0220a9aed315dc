"""Attention kernels at the edges of their query tiles and key blocks, against a 64-bit statement."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(B, Sq, Skv, Hq, Hkv, D, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(B, s, h, D, device="cuda", generator=g).to(torch.bfloat16)
            for s, h in ((Sq, Hq), (Skv, Hkv), (Skv, Hkv))]


def _ref(q, k, v, scale, causal, q0, k0):
    n = q.shape[2] // k.shape[2]
    q, k, v = (t.double() if not t.requires_grad else t for t in (q, k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", q, k.repeat_interleave(n, 2)) * scale
    if causal:
        hidden = (torch.arange(k.shape[1], device=q.device) + k0)[None, :] > (torch.arange(q.shape[1], device=q.device)
                                                                              + q0)[:, None]
        s = s.masked_fill(hidden, float("-inf"))
    lse = torch.logsumexp(s, -1)
    p = torch.exp(s - torch.where(torch.isinf(lse), torch.zeros_like(lse), lse)[..., None])
    return torch.einsum("bhqk,bkhd->bqhd", p, v.repeat_interleave(n, 2)), lse


@pytest.mark.parametrize("D,Hq,Hkv", [(128, 4, 1), (256, 2, 2)])
@pytest.mark.parametrize("Sq,Skv,causal,q0,k0", [
    (1, 1, True, 0, 0), (63, 63, True, 0, 0), (128, 128, True, 0, 0), (129, 129, True, 0, 0), (257, 257, True, 0, 0),
    (640, 640, True, 0, 0), (1001, 1001, True, 0, 0),
    (128, 64, False, 0, 0), (200, 333, False, 0, 0), (384, 384, True, 0, 100), (256, 128, True, 500, 0),
    (130, 130, True, 0, 1000)])
def test_forward_edges(D, Hq, Hkv, Sq, Skv, causal, q0, k0):
    from cverl_b200 import _native as nv
    from cverl_b200.ops import attention_native as an
    q, k, v = _inputs(2, Sq, Skv, Hq, Hkv, D, Sq + Skv)
    scale = 1 / math.sqrt(D)
    out, lse = an._fwd(q, k, v, scale, causal, q0, k0)
    nv.check_status()
    want, lse_want = _ref(q, k, v, scale, causal, q0, k0)
    # P and O are rounded to bf16 (2^-9 each, the first averaged over the row); rows that see no key give zero
    assert (out.double() - want).norm() <= 2.0 ** -8 * want.norm()
    assert torch.equal(torch.isinf(lse), torch.isinf(lse_want))
    seen = ~torch.isinf(lse_want)
    assert bool((out[(~seen).transpose(1, 2)] == 0).all())
    assert (lse.double() - lse_want)[seen].abs().max() < 1e-4 if bool(seen.any()) else True


def test_forward_scores_that_grow_along_the_keys():
    """Every key block raises the row maximum by more than the rescale threshold, so O is rescaled each time."""
    from cverl_b200.ops import attention_native as an
    for D in (128, 256):
        q, k, v = _inputs(1, 512, 512, 2, 1, D, 7)
        k = (k.float() * torch.linspace(0.5, 12, 512, device="cuda")[None, :, None, None]).to(torch.bfloat16)
        out, _ = an._fwd(q, k, v, 1.0 / math.sqrt(D), True, 0, 0)
        want, _ = _ref(q, k, v, 1.0 / math.sqrt(D), True, 0, 0)
        assert (out.double() - want).norm() <= 2.0 ** -8 * want.norm()


@pytest.mark.parametrize("D", [128, 256])
@pytest.mark.parametrize("S", [640, 1500])
def test_forward_scores_that_grow_now_and_then(D, S):
    """Wide scores: a row's maximum passes the rescale bound at irregular blocks, with blocks in between that do not."""
    from cverl_b200.ops import attention_native as an
    q, k, v = _inputs(2, S, S, 2, 1, D, 11)
    q = (q.float() * 12).to(torch.bfloat16)
    out, lse = an._fwd(q, k, v, 1.0 / math.sqrt(D), True, 0, 0)
    want, lse_want = _ref(q, k, v, 1.0 / math.sqrt(D), True, 0, 0)
    assert (out.double() - want).norm() <= 2.0 ** -8 * want.norm()
    assert (lse.double() - lse_want).abs().max() < 1e-3      # |score| up to 60: 2^-24 relative in fp32, with margin


@pytest.mark.parametrize("D,Hq,Hkv", [(128, 4, 1), (128, 2, 2), (256, 2, 2), (256, 4, 1)])
@pytest.mark.parametrize("Sq,Skv,causal,q0,k0", [
    (1, 1, True, 0, 0), (63, 63, True, 0, 0), (65, 65, True, 0, 0), (128, 128, True, 0, 0), (129, 129, True, 0, 0),
    (640, 640, True, 0, 0), (1001, 1001, True, 0, 0),
    (200, 333, False, 0, 0), (384, 384, True, 0, 100), (256, 128, True, 500, 0), (130, 130, True, 0, 1000)])
def test_backward_edges(D, Hq, Hkv, Sq, Skv, causal, q0, k0):
    from cverl_b200 import _native as nv
    from cverl_b200.ops import attention_native as an
    q, k, v = _inputs(2, Sq, Skv, Hq, Hkv, D, Sq + Skv + 1)
    do = _inputs(2, Sq, Skv, Hq, Hkv, D, 99)[0]
    scale = 1 / math.sqrt(D)
    out, lse = an._fwd(q, k, v, scale, causal, q0, k0)
    got = an._bwd(q, k, v, out, lse, do, scale, causal, q0, k0)
    again = an._bwd(q, k, v, out, lse, do, scale, causal, q0, k0)
    nv.check_status()
    leaves = [t.double().requires_grad_(True) for t in (q, k, v)]
    want, _ = _ref(*leaves, scale, causal, q0, k0)
    grads = torch.autograd.grad(want, leaves, do.double())
    for name, a, b, r in zip("qkv", got, again, grads):
        assert torch.equal(a, b), name           # no sums across CTAs: the order is fixed
        # P, dS, the saved output behind Delta and the result are rounded to bf16, 2^-9 each; with one visible key
        # dq and dk cancel to zero, and what is left is the rounding of dP - Delta, of the size of |dO| |V| scale
        floor = 2.0 ** -8 * scale * float(do.double().norm()) * D ** 0.5 if Skv < 8 and name != "v" else 0.0
        assert (a.double() - r).norm() <= 4 * 2.0 ** -9 * r.norm() + floor + 1e-9, name
