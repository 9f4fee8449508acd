"""Strips of several rows in the packed pooling kernels, both ways, to the bit: what a thread carries from row to row."""
import pytest
import torch

import actnn_oracle as O
from test_max_pool_packed_gpu import reference

pytestmark = pytest.mark.gpu


# On 148 multiprocessors and maps 64 wide, strips of four rows and pairs, of two output rows, and of two pairs; the
# last strip of a map is shorter.  Output rows are whole octets with (2, 0) and (3, 1) only; the others take one a thread.
@pytest.mark.parametrize("planes", [6144, 3072, 1536])
@pytest.mark.parametrize("h", [100, 101])
@pytest.mark.parametrize("k,p", [(2, 0), (2, 1), (3, 0), (3, 1)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_values_codes_and_gradients(k, p, h, planes, dtype):
    from actnn_b200.cpp_extension import quantization as q
    torch.manual_seed(h + k)
    some = torch.randint(-3, 4, (1, 13, h, 64)).to(dtype)                  # many ties; every plane is one of these
    some[0, 1] = torch.randn(h, 64).to(dtype)
    some[0, 2] = torch.tensor([-0.0, 0.0])[torch.randint(2, (h, 64))].to(dtype)
    which = torch.arange(planes, device="cuda") % 13
    geom = ((k, k), (2, 2), (p, p), (1, 1))
    ry, ridx = O.max_pool2d_forward(some, *geom)
    y, idx = q.max_pool2d_forward(some.cuda()[0, which].view(planes // 96, 96, h, 64), *geom)
    assert torch.equal(y.view(planes, *ry.shape[2:]).view(torch.int16), ry.cuda()[0, which].view(torch.int16))
    assert torch.equal(idx.view(planes, *ry.shape[2:]), ridx.cuda()[0, which])
    gy = (torch.randn(ry.shape) * 2.0 ** torch.randint(-26, 15, ry.shape).float()).to(dtype)     # subnormals to overflow
    want = reference(gy, ridx, some.shape, k, p).cuda()[0, which].view(torch.int16)
    gx = q.max_pool2d_backward(gy.cuda()[0, which].view(y.shape), idx, (planes // 96, 96, h, 64), *geom)
    gx, nan = gx.view(want.shape).view(torch.int16), torch.isnan(want.view(dtype))
    assert torch.equal(torch.isnan(gx.view(dtype)), nan)
    assert torch.equal(gx[~nan], want[~nan])
