"""Mean of the per-sample squared norms from the launch that computes them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,f", [(1, 5), (3, 1001), (512, 64), (513, 7), (1500, 33), (64, 4096)])
def test_mean_of_the_sums(n, f, dtype):
    from actnn_b200 import _lib
    from actnn_b200.cpp_extension import calc_precision as cp
    torch.manual_seed(n + f)
    g = torch.randn(n, f, device="cuda").to(dtype)
    sums = cp.sample_sumsq(g)
    for _ in range(3):                                       # the ticket is left at zero
        mean = cp.mean_sample_sumsq(g)
        assert mean.shape == () and mean.dtype == torch.float32
        # positive terms, chains of at most n / 512 + 16 additions: a rounding of the result each, and one of the division
        assert abs(float(mean.double() / sums.double().mean()) - 1) <= (n / 512 + 22) * 2 ** -24
        assert int(_lib.ticket(g.device)[:4].view(torch.int32)) == 0
    assert torch.equal(mean, cp.mean_sample_sumsq(g))
    strided = g.t().contiguous().t()
    assert torch.equal(cp.mean_sample_sumsq(strided), mean)
    g[0, 0] = float("nan")
    assert torch.isnan(cp.mean_sample_sumsq(g))
