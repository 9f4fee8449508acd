"""The mean of the per-sample squared norms is that of the sums, rounded once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 256, 512, 513, 1024])
def test_mean_is_rounded_once(n):
    from actnn_b200.cpp_extension import calc_precision as cp
    for seed in range(20):
        torch.manual_seed(seed)
        g = torch.randn(n, 24, device="cuda") * torch.exp(0.5 * torch.randn(n, 1, device="cuda"))
        want = cp.sample_sumsq(g).double().mean()
        # half a unit in the last place; the float64 sums' own roundings are 2^-29 of it each
        assert abs(float((cp.mean_sample_sumsq(g).double() - want) / want)) <= 2 ** -24 * (1 + 2 ** -12)
