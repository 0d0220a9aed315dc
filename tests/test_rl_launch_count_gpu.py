"""The launch counter on either side of the one-launch limits of the loss and the advantage."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,loss,adv", [(64, 512, 1, 1), (128, 256, 1, 1), (129, 256, 3, 3), (257, 100, 1, 3),
                                                (256, 128, 1, 1), (1, 1, 1, 1), (2049, 17, 3, 3)])
def test_counted_launches(rows, cols, loss, adv):
    from cverl_b200 import ops
    from cverl_b200.ops import rl
    x, mask = torch.randn(rows, cols, device="cuda"), torch.ones(rows, cols, device="cuda")
    groups = torch.arange(rows, device="cuda") // 4
    for fn, want in ((lambda: rl.fused_ppo_loss(x, x, x, mask), loss),
                     (lambda: rl.fused_grpo_advantage(x, mask, groups), adv)):
        n = ops.launch_counter["n"]
        fn()
        assert ops.launch_counter["n"] - n == want
