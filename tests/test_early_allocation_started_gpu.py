"""That the widths' allocation does start before the last backward, and what follows where one group cannot."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def train(early, bits, monkeypatch):
    import actnn_b200 as actnn
    from actnn_b200.conf import QuantizationConfig, config
    config.__dict__.update(QuantizationConfig().__dict__)
    actnn.set_optimization_level("L3")
    config.activation_compression_bits = bits
    actnn.QScheme.layers, actnn.QBNScheme.layers, actnn.QScheme.prev_layer = [], [], None
    torch.manual_seed(1)
    torch.cuda.manual_seed(1)
    net = torch.nn.Sequential(actnn.QLinear(300, 64), actnn.QReLU(), actnn.QLinear(64, 64), actnn.QReLU(),
                              actnn.QLinear(64, 32, group=1), actnn.QReLU(), actnn.QLinear(32, 10, group=1)).cuda()
    x = torch.randn(12, 300, device="cuda")
    starts, widths, start = [], [], actnn.QScheme.start_perlayer
    monkeypatch.setattr(actnn.QScheme, "start_perlayer", staticmethod(lambda: (starts.append(start()), starts[-1])[1]))
    if not early:
        monkeypatch.setattr(actnn.QScheme, "start_allocation", lambda self: None)
    for _ in range(3):
        net(x).square().mean().backward()
        widths.append([float(s.bits) for s in actnn.QScheme.layers])
    monkeypatch.undo()
    config.__dict__.update(QuantizationConfig().__dict__)
    return starts, widths


# two groups of layers; the second one at the widths it began with, which is no allocation, so none starts early
@pytest.mark.parametrize("bits,groups", [([2, 3], 2), ([2, 8], None)])
def test_one_start_a_step(bits, groups, monkeypatch):
    starts, widths = train(True, bits, monkeypatch)
    assert len(starts) == 3
    assert all(s is None if groups is None else len(s) == groups for s in starts)
    none, later = train(False, bits, monkeypatch)
    assert not none and widths == later
    assert widths[0][:2] != [float(bits[0])] * 2
    if groups is None:
        assert all(w[2:] == [8.0, 8.0] for w in widths)
