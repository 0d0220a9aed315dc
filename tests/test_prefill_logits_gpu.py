"""Logits of the last prompt position: fp32 arithmetic, contiguous at any vocabulary size."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,vocab", [(1, 512), (4, 4099), (33, 1001)])
def test_prefill_logits_are_fp32_sums(batch, vocab):
    from cverl_b200.models import decode
    g = torch.Generator(device="cuda").manual_seed(vocab)
    hidden, w = (torch.randn(n, 1024, device="cuda", generator=g).to(torch.bfloat16) for n in (batch, vocab))
    model = SimpleNamespace(lm_head_weight=lambda: w, ctx=SimpleNamespace(tp_size=1))
    got = decode._full_logits(model, hidden)
    assert got.dtype == torch.float32 and got.shape == (batch, vocab) and got.is_contiguous()
    want = hidden.double() @ w.double().t()
    # products of bf16 are exact in fp32; 1024 additions rounded to nearest add sqrt(1024) errors of 2^-25 / sqrt(3) of a
    # partial sum, which is 1 / sqrt(2) of the result on average: 4e-7
    assert (got.double() - want).norm() <= 4e-7 * want.norm()
