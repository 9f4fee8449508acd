"""The per-layer allocation that is enqueued at the start of the last backward against the one at its end."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def steps(early, kind, monkeypatch):
    import actnn_b200 as actnn
    from actnn_b200.conf import QuantizationConfig, config
    config.__dict__.update(QuantizationConfig().__dict__)
    actnn.set_optimization_level("L3")
    actnn.QScheme.layers, actnn.QBNScheme.layers, actnn.QScheme.prev_layer = [], [], None
    torch.manual_seed(1)
    torch.cuda.manual_seed(1)
    if kind == "conv":
        net = torch.nn.Sequential(actnn.QConv2d(3, 8, 3), actnn.QBatchNorm2d(8), actnn.QReLU(), actnn.QConv2d(8, 4, 3)).cuda()
        x = torch.randn(12, 3, 16, 16, device="cuda")
    else:
        net = torch.nn.Sequential(actnn.QLinear(300, 64), actnn.QReLU(), actnn.QLinear(64, 10)).cuda()
        x = torch.randn(12, 300, device="cuda")
    if kind == "frozen":                                     # the step ends at the first layer that trains
        net[0].weight.requires_grad_(False)
        net[0].bias.requires_grad_(False)
        x.requires_grad_(True)
    seen = []
    if not early:
        monkeypatch.setattr(actnn.QScheme, "start_allocation", lambda self: None)
    for _ in range(3):
        y = net(x)
        y.square().mean().backward()
        seen.append([float(s.bits) for s in actnn.QScheme.layers + actnn.QBNScheme.layers])
        assert all(s._started is None for s in actnn.QScheme.layers)
    monkeypatch.undo()
    config.__dict__.update(QuantizationConfig().__dict__)
    return seen, [p.grad for p in net.parameters() if p.grad is not None]


@pytest.mark.parametrize("kind", ["conv", "linear", "frozen"])
def test_widths_are_those_of_an_allocation_at_the_end(kind, monkeypatch):
    a, ga = steps(True, kind, monkeypatch)
    b, gb = steps(False, kind, monkeypatch)
    assert a == b and a[0] != [2.0] * len(a[0])
    assert all(torch.allclose(s, t, rtol=1e-3, atol=1e-5) for s, t in zip(ga, gb))
