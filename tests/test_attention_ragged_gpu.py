"""Which calls of ``causal_attention`` run on the kernels, and that ragged ones give what the general path gives."""
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


def test_calls_that_stay_on_the_general_path():
    from cverl_b200.ops import attention_native as an
    q = torch.randn(100, 2, 128, device="cuda").to(torch.bfloat16)
    assert not an.supported(q, q, q, 100)                              # head dim 128, ragged
    assert an.supported(q, q, q, 128)
    small = torch.randn(100, 2, 256, device="cuda").to(torch.bfloat16)
    assert not an.supported(small, small, small, 100)                  # 20,000 scores: the host's side decides
    empty = torch.empty(0, 2, 256, device="cuda", dtype=torch.bfloat16)
    assert an.causal_attention(empty, empty, empty, 0, 100).shape == (0, 2, 256)


def test_large_ragged_call_runs_on_the_kernels():
    """3 sequences of 1001 with 4 / 2 heads: the smallest length that this many heads send to the kernels is 1000."""
    from cverl_b200.ops import attention, attention_native as an
    from cverl_b200.utils import fallbacks
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k = (torch.randn(3 * 1001, h, 256, device="cuda", generator=g).to(torch.bfloat16) for h in (4, 2))
    assert an.supported(q, k, k, 1001) and not an.supported(q.float(), k.float(), k.float(), 1001)
    fallbacks.reset()
    out = attention.causal_attention(q, k, k, 3, 1001)
    assert fallbacks.total() == 0
    ref = attention._sdpa(q, k, k, 3, 1001, None)
    # two bf16 results of the same sums: half a unit in the last place each, and the rounded weights
    assert (out.float() - ref.float()).norm() <= 2.0 ** -8 * ref.float().norm()
    attention.causal_attention(q[:999 * 3], k[:999 * 3], k[:999 * 3], 3, 999)
    assert fallbacks.total() == 1
    fallbacks.reset()
