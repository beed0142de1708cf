"""An empty batch is refused by the network's forward and backward pass, and leaves
the weights as they are."""
import pytest

pytestmark = pytest.mark.gpu


def test_empty_batch_is_refused():
    import torch
    from ps_claude_opt_b200 import native, screen

    net = screen.Mlp(sizes=(16, 32, 1), seed=1)
    x = torch.randn((20, 16), generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    y = torch.zeros(20, device="cuda")
    net.train_step(x, y)  # moments that a step on nothing would apply
    before = [t.clone() for t in net.W + net.b + net.mW + net.vW]
    with pytest.raises(native.PsError):
        net.forward(x[:0])
    with pytest.raises(native.PsError):
        net.backward(y[:0])
    with pytest.raises(native.PsError):
        net.train_step(x[:0], y[:0])
    assert net.steps == 1
    for a, b in zip(before, net.W + net.b + net.mW + net.vW):
        assert torch.equal(a, b)
