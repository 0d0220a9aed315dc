"""Which calls of ``causal_attention`` run on the kernels, and that the kernels give at ragged lengths what the general
path gives."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seq", [1, 63, 127, 130, 255, 333])
@pytest.mark.parametrize("layout", ["packed", "strided", "misaligned"])
def test_ragged_head_dim_256_matches_the_library(seq, layout):
    from cverl_b200.ops import attention, attention_native
    g = torch.Generator(device="cuda").manual_seed(seq)
    B, Hq, Hkv, D = 2, 4, 2, 256

    def make(h):
        n = B * seq * h * D
        if layout == "strided":
            return torch.randn(B * seq, 2, h, D, device="cuda", generator=g).to(torch.bfloat16)[:, 1]
        flat = torch.randn(n + 8, device="cuda", generator=g).to(torch.bfloat16)
        off = 1 if layout == "misaligned" else 0
        return flat[off:off + n].view(B * seq, h, D)
    base = [make(h) for h in (Hq, Hkv, Hkv)]
    do = make(Hq)
    got_in = [t.detach().requires_grad_(True) for t in base]
    out = attention_native.causal_attention(*got_in, B, seq)
    got = (out,) + torch.autograd.grad(out, got_in, do)
    ref_in = [t.detach().double().requires_grad_(True) for t in base]
    q, k, v = (t.view(B, seq, -1, D).transpose(1, 2) for t in ref_in)
    s = (q @ k.repeat_interleave(2, 1).transpose(-1, -2)) / math.sqrt(D)
    s = s.masked_fill(torch.ones(seq, seq, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    want_o = (torch.softmax(s, -1) @ v.repeat_interleave(2, 1)).transpose(1, 2).reshape(B * seq, Hq, D)
    want = (want_o,) + torch.autograd.grad(want_o, ref_in, do.double())
    # the library's kernel needs 16-byte boundaries and does not check them: it gets aligned copies
    lib_in = [t.detach().clone(memory_format=torch.contiguous_format).requires_grad_(True) for t in base]
    lib_o = attention._sdpa(*lib_in, B, seq, None)
    lib = (lib_o,) + torch.autograd.grad(lib_o, lib_in, do.clone(memory_format=torch.contiguous_format))
    for a, r, b in zip(got, want, lib):
        assert a.shape == b.shape and a.dtype == b.dtype
        # bf16 results of either path; one visible key: dq and dk are zero up to rounding
        err, other = (a.double() - r).norm(), (b.double() - r).norm()
        assert err <= 4 * 2.0 ** -9 * r.norm() or err <= 2 * other + 1e-9, (float(err), float(other))


def _qk(batch, seq, d=256, hq=4, hkv=2, seed=5):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(batch * seq, h, d, device="cuda", generator=g).to(torch.bfloat16) for h in (hq, hkv)]


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("seq", [100, 128, 1001, 1024])
def test_the_route_depends_on_the_length_alone(d, seq):
    """A sequence takes the same path, and with it the same roundings, in a small batch and in a large one."""
    from cverl_b200.ops import attention, attention_native as an
    from cverl_b200.utils import fallbacks
    for batch in (1, 3, 40):
        q, k = _qk(batch, seq, d)
        assert an.supported(q, k, k, seq) == (seq % 128 == 0)
        fallbacks.reset()
        attention.causal_attention(q, k, k, batch, seq)
        assert fallbacks.total() == (seq % 128 != 0)
    assert not an.supported(q.float(), k.float(), k.float(), seq)
    empty = torch.empty(0, 2, d, device="cuda", dtype=torch.bfloat16)
    assert an.causal_attention(empty, empty, empty, 0, 100).shape == (0, 2, d)
    fallbacks.reset()


def test_ragged_calls_keep_the_transforms_of_the_general_path():
    """Function transforms run, a second derivative is refused instead of left out."""
    from cverl_b200.ops import attention
    (q, k), seq = _qk(3, 1001), 1001
    one = attention.causal_attention(q, k, k, 3, seq)
    two = torch.func.vmap(lambda a, b: attention.causal_attention(a, b, b, 3, seq))(torch.stack([q, q]),
                                                                                     torch.stack([k, k]))
    # bf16 results of the same sums, in another order if the library splits the larger batch differently
    assert (two.float() - one.float()).norm() <= 2 ** 0.5 * 2.0 ** -8 * one.float().norm()
    dq = torch.func.grad(lambda a: attention.causal_attention(a, k, k, 3, seq).float().sum())(q)
    a = q.detach().requires_grad_(True)
    (want,) = torch.autograd.grad(attention.causal_attention(a, k, k, 3, seq).float().sum(), a, create_graph=True)
    assert (dq.float() - want.float()).norm() <= 2.0 ** -8 * want.detach().float().norm()
    with pytest.raises(RuntimeError):
        torch.autograd.grad(want.float().pow(2).sum(), a)
