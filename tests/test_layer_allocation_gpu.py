"""The one-launch allocation over layers x samples against the general kernel and the oracle's heap."""
import pytest
import torch

import actnn_oracle as O

pytestmark = pytest.mark.gpu


# one sample; layers that end inside a warp; one, two and eight blocks of the cluster; several samples a thread; the limit
@pytest.mark.parametrize("layers,n", [(1, 1), (3, 7), (5, 32), (1, 1024), (7, 256), (54, 256), (64, 512), (256, 128)])
@pytest.mark.parametrize("kind", ["random", "ties", "zero", "wide"])
def test_sums_of_widths(layers, n, kind):
    from actnn_b200.cpp_extension import calc_precision as cp
    g = torch.Generator().manual_seed(layers * n)
    C = torch.rand(layers, n, generator=g)
    if kind == "ties":
        C = torch.randint(1, 4, (layers, n), generator=g).float()
    elif kind == "zero":
        C = torch.zeros(layers, n)
    elif kind == "wide":
        C = torch.exp(torch.randn(layers, n, generator=g) * 12)
    dims = torch.randint(1, 2 ** 22, (layers,), generator=g).tolist()
    Cd = C.cuda()
    w = torch.tensor(dims, dtype=torch.int32).repeat_interleave(n).cuda()
    weight = float(sum(dims) * n)
    for target in (2.0 * weight, 3.3 * weight, weight, 0.0, 8.0 * weight, 1.001 * weight):
        sums = cp.allocate_layers([Cd[i].contiguous() for i in range(layers)], dims, 8, target)
        bits, _ = cp.allocate_bits(Cd.view(-1), 8, target, w)
        assert torch.equal(sums.long(), bits.view(layers, n).sum(1)), target
    if layers * n <= 2000:
        target = 2.0 * weight
        ref = O.calc_precision(torch.full((layers * n,), 8, dtype=torch.int32), C.view(-1), w.cpu(), target)
        sums = cp.allocate_layers([Cd[i].contiguous() for i in range(layers)], dims, 8, target)
        assert torch.equal(sums.cpu().long(), ref.view(layers, n).sum(1))


def test_what_does_not_fit_is_left_to_the_general_path():
    from actnn_b200.cpp_extension import calc_precision as cp
    C = [torch.rand(256, device="cuda") for _ in range(129)]
    assert cp.allocate_layers(C, [5] * 129, 8, 100.0) is None                       # 33024 samples
    assert cp.allocate_layers([C[0], C[1][:100]], [5, 5], 8, 100.0) is None          # unequal batches
    assert cp.allocate_layers([C[0].double()], [5], 8, 100.0) is None
