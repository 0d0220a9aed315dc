"""A strong decay at one token leaves every earlier output of the Gated-DeltaNet core as it was, bit for bit."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gate", [-20.0, -1e4, -1e6])
@pytest.mark.parametrize("token", [1, 33, 34, 63, 65, 127])
def test_a_later_gate_does_not_reach_earlier_outputs(gate, token):
    from cverl_b200.ops import gdn
    gen = torch.Generator(device="cuda").manual_seed(token)
    B, S, H = 2, 128, 3
    mixed = F.silu(torch.randn(B, S, 3 * H * 128, device="cuda", generator=gen)).to(torch.bfloat16)
    beta = torch.sigmoid(torch.randn(B, S, H, device="cuda", generator=gen))
    g = -0.05 * torch.rand(B, S, H, device="cuda", generator=gen)
    out = []
    for x in (-0.01, gate):
        g[:, token] = x
        out.append(gdn.gated_delta_rule_packed(mixed, beta, g, scale=128 ** -0.5, heads=H)[0])
    assert torch.isfinite(out[1].float()).all()
    assert torch.equal(out[0][:, :token], out[1][:, :token])
    assert not torch.equal(out[0][:, token:], out[1][:, token:])
