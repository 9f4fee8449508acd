"""The mean of the per-sample squared norms from the launch of the sums: rounded once, and up to how many samples."""
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


@pytest.mark.parametrize("n", [1024, 1025])
def test_many_samples_take_a_launch_of_their_own(n, monkeypatch):
    from actnn_b200.cpp_extension import calc_precision as cp
    g = torch.randn(n, 24, device="cuda")
    sums, calls = cp.sample_sumsq(g), []
    monkeypatch.setattr(cp, "sample_sumsq", lambda grad: (calls.append(grad), sums)[1])
    mean = cp.mean_sample_sumsq(g)
    assert len(calls) == (n > 1024)
    assert mean.shape == () and abs(float(mean.double() / sums.double().mean()) - 1) <= 24 * 2 ** -24
