"""Epilogues that turn their chunk in shared memory, at the edges of rows, columns and chunks."""
import pytest
import torch

from cverl_b200 import ops

pytestmark = pytest.mark.gpu


def _bf(*shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (scale * torch.randn(*shape, device="cuda", generator=g)).to(torch.bfloat16)


@pytest.mark.parametrize("M", [1, 31, 129, 290])
@pytest.mark.parametrize("N", [8, 36, 100, 256, 264, 600])
def test_fp32_store_and_accumulate(M, N):
    K = 192
    a, b = _bf(M, K, seed=1), _bf(N, K, seed=2)
    want = a.double() @ b.double().t()
    # fp32 accumulation of K bf16 products: K rounding steps of 2^-24 on a sum of magnitude sqrt(K)
    tol = K * 2.0 ** -24 * K ** 0.5 * 4
    got = ops.gemm_nt(a, b, out_dtype=torch.float32)
    assert (got.double() - want).abs().max() <= tol
    N4 = (N + 3) // 4 * 4
    pad = torch.full((M + 2, N4 + 8), 3.0, device="cuda")
    acc = pad[:M, :N]
    at = torch.zeros(K, (M + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
    bt = torch.zeros(K, (N + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
    at[:, :M], bt[:, :N] = a.t(), b.t()
    ops.gemm_tn_acc(at[:, :M], bt[:, :N], acc)
    assert (acc.double() - 3 - want).abs().max() <= tol + 2.0 ** -20
    assert bool((pad[M:] == 3).all()) and bool((pad[:, N4:] == 3).all())     # nothing outside the result


@pytest.mark.parametrize("rows", [1, 45, 130])
@pytest.mark.parametrize("vocab", [64, 328, 1032])
def test_head_logprob_and_softmax_gradient(rows, vocab):
    H = 128
    h, e = _bf(rows, H, seed=3).requires_grad_(True), _bf(vocab, H, seed=4, scale=0.1).requires_grad_(True)
    t = torch.randint(0, vocab, (rows,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    d = torch.randn(rows, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6))
    lp = ops.lmhead_logprob(h, e, t)
    lp.backward(d)
    h64, e64 = h.detach().double().requires_grad_(True), e.detach().double().requires_grad_(True)
    want = torch.log_softmax(h64 @ e64.t(), -1).gather(1, t[:, None])[:, 0]
    want.backward(d.double())
    assert (lp.double() - want).abs().max() < 2e-5
    # the softmax gradient travels as bf16 (2^-9 per entry) and both results are stored as bf16
    for got, ref in ((h.grad, h64.grad), (e.grad, e64.grad)):
        assert (got.double() - ref).norm() <= 4 * 2.0 ** -9 * ref.norm()
