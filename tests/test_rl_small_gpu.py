"""One-launch loss and advantage kernels: the sizes around their limit and the layouts of rows and groups, against the
plain statements in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (rows, cols): one token, fewer rows than warps, more rows than warps, odd widths, at and above the one-launch limit
SHAPES = [(1, 1), (3, 5), (64, 512), (127, 33), (129, 31), (1000, 100), (128, 256), (129, 256), (256, 128), (257, 100),
          (2048, 16), (2049, 17)]


def _data(rows, cols, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    lens = torch.randint(0, cols + 1, (rows, 1), device="cuda", generator=g)        # some rows are empty
    lens[0] = cols
    mask = (torch.arange(cols, device="cuda")[None] < lens).float()
    lp, old, ref, adv = (0.3 * torch.randn(rows, cols, device="cuda", generator=g) for _ in range(4))
    return lp, old, ref, adv, mask, g


@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("agg", [0, 1, 2])
def test_loss_matches_the_plain_statement(rows, cols, agg):
    from cverl_b200.ops import rl
    lp, old, ref, adv, mask, _ = _data(rows, cols, rows + cols + agg)
    metrics, grad = rl.fused_ppo_loss(old, lp, adv, mask, ref, kl_coef=0.05, kl_penalty_kind="k3", agg=agg, loss_scale=0.5)
    x = lp.double().requires_grad_(True)
    res = rl.ppo_clipped_loss(old.double(), x, adv.double(), mask.double(), agg=agg)
    kl = rl.masked_mean(rl.kl_penalty(x, ref.double(), "k3"), mask.double())
    (want,) = torch.autograd.grad((res.pg_loss + 0.05 * kl) * 0.5, x)
    ref_m = torch.stack([res.pg_loss, res.pg_clipfrac, res.ppo_kl, res.pg_clipfrac_lower, kl, mask.double().sum()]).detach()
    # fp32 per token (2^-24, a few operations), sums in 64 bits; a ratio within 2^-22 of the clip may fall either way
    assert (metrics.double() - ref_m)[[0, 2, 4, 5]].abs().max() <= 2e-6 * (1 + ref_m.abs().max())
    assert (metrics.double() - ref_m)[[1, 3]].abs().max() <= 2.0 / float(mask.sum())
    assert (grad.double() - want).norm() <= 1e-5 * want.norm() + 1e-12


@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("norm", [False, True])
def test_advantage_matches_the_plain_statement(rows, cols, norm):
    from cverl_b200.ops import rl
    _, _, _, rewards, mask, g = _data(rows, cols, rows)
    groups = torch.randint(0, max(1, rows // 4), (rows,), device="cuda", generator=g)      # unsorted, some of one row
    got, _ = rl.fused_grpo_advantage(rewards, mask, groups, norm_adv_by_std=norm)
    want, _ = rl.grpo_outcome_advantage(rewards.double(), mask.double(), groups, norm_adv_by_std=norm)
    # a row sum of `cols` fp32 terms, then a difference that may cancel: relative to the scores' size
    assert (got.double() - want).abs().max() <= 2e-5 * (1 + want.abs().max())
