"""How the mask-saving layers behave as autograd nodes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, grad):
        return None


@pytest.mark.parametrize("name", ["relu", "relu_minmax", "dropout", "max_pool"])
def test_no_gradient_from_above_counts_as_zeros(name):
    from actnn_b200.cpp_extension import quantization as q
    layer = {"relu": q.act_quantized_relu, "relu_minmax": q.act_quantized_relu_with_minmax,
             "dropout": lambda x: q.act_quantized_dropout(x, 0.5),
             "max_pool": lambda x: q.act_quantized_max_pool2d(x, (2, 2), (2, 2), (0, 0), (1, 1), False, False)}[name]
    x = torch.randn(4, 8, 8, 8, device="cuda", dtype=torch.float16, requires_grad=True)
    (g,) = torch.autograd.grad(NoGradient.apply(layer(x)).sum(), x)
    assert g.shape == x.shape and g.dtype == x.dtype and not g.any()
