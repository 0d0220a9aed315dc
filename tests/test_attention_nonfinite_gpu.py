"""A value that is not finite shows in every attention result that depends on it and in no other sequence or head group."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(t):
    """Which (sequence, row, head) of [B, S, H, D] hold a NaN."""
    return t.isnan().any(-1)


@pytest.mark.parametrize("D", [128, 256])
@pytest.mark.parametrize("S", [256, 300])
def test_nan_reaches_what_sees_it(D, S):
    from cverl_b200 import _native as nv
    from cverl_b200.ops import attention_native as an
    g = torch.Generator(device="cuda").manual_seed(D + S)
    B, Hq, Hkv, at = 2, 4, 2, 200
    q, k, v, do = (torch.randn(B, S, h, D, device="cuda", generator=g).to(torch.bfloat16) for h in (Hq, Hkv, Hkv, Hq))
    idx = torch.arange(S, device="cuda")

    def run(q, k, v):
        out, lse = an._fwd(q, k, v, D ** -0.5, True, 0, 0)
        grads = an._bwd(q, k, v, out, lse, do, D ** -0.5, True, 0, 0)
        nv.check_status()
        for t in (out,) + grads:
            assert torch.isfinite(t[1].float()).all()            # the other sequence
            assert torch.isfinite(t[0, :, t.shape[2] // 2:].float()).all()   # the other kv head and its queries
        return out, grads
    bad = q.clone()
    bad[0, at, 0, 5] = float("nan")                               # one query of head 0
    out, (dq, dk, dv) = run(bad, k, v)
    assert torch.equal(_rows(out)[0, :, 0], idx == at) and not _rows(out)[0, :, 1].any()
    assert torch.equal(_rows(dq)[0, :, 0], idx == at) and not _rows(dq)[0, :, 1].any()
    assert torch.equal(_rows(dv)[0, :, 0], idx <= at)             # every key that the query sees
    assert bool(_rows(dk)[0, :at + 1, 0].all())
    bad = k.clone()
    bad[0, at, 0, 5] = float("nan")                               # one key of kv head 0: every query from it on
    out, (dq, dk, dv) = run(q, bad, v)
    for h in (0, 1):
        assert torch.equal(_rows(out)[0, :, h], idx >= at)
        assert bool(_rows(dq)[0, at:, h].all())
    assert bool(_rows(dv)[0, at, 0]) and bool(_rows(dk)[0, :, 0].any())
    bad = v.clone()
    bad[0, at, 0, 5] = float("inf")                               # one value: the queries from it on, in that column
    out, _ = an._fwd(q, k, bad, D ** -0.5, True, 0, 0)
    nv.check_status()
    assert not torch.isfinite(out[0, at:, :2, 5].float()).any() and torch.isfinite(out[0, :, :2, 6].float()).all()
    assert torch.isfinite(out[0, :at // 128 * 128].float()).all() and torch.isfinite(out[1].float()).all()
