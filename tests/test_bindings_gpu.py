"""The two halves of the binding, C++ and Python, make the same calls: equal results to the bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _grads(layer, x):
    x = x.clone().requires_grad_()
    y = layer(x)
    wanted = [x] + list(getattr(layer, "parameters", list)())
    gy = torch.randn(y.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).to(y.dtype)
    return [y.detach(), *torch.autograd.grad(y, wanted, gy)]


def _codec(shape, level, dtype):
    import actnn_b200 as actnn
    from actnn_b200 import ops
    actnn.set_optimization_level(level)
    x = torch.randn(shape, device="cuda").to(dtype)
    quantized = ops.quantize_activation(x, actnn.QConv2d(shape[1], 4, 3).scheme)
    return [t for t in quantized if isinstance(t, torch.Tensor)] + [ops.dequantize_activation(quantized, x.shape, dtype)]


def _batch_norm(shape, dtype, **kw):
    import actnn_b200 as actnn
    layer = actnn.QBatchNorm2d(shape[1], **kw).cuda()
    out = _grads(layer, (torch.randn(shape, device="cuda") * 2 + 1).to(dtype))
    return out + [layer.running_mean, layer.running_var]


def _ranges_of_a_relu(dtype):
    from actnn_b200 import ops
    from actnn_b200.cpp_extension import quantization as q
    import actnn_b200 as actnn
    y = q.act_quantized_relu_with_minmax(torch.randn(6, 16, 16, 8, device="cuda").to(dtype))
    mn, mx, _ = y.actnn_minmax
    return [mn, mx] + [t for t in ops.quantize_activation(y, actnn.QConv2d(16, 4, 3).scheme, minmax=(mn, mx))]


def _mask_layers(dtype):
    from actnn_b200.cpp_extension import quantization as q
    x = torch.randn(5, 6, 15, 24, device="cuda").to(dtype)
    whole = torch.randn(6, 16, 16, 8, device="cuda").to(dtype)
    return (_grads(q.act_quantized_relu, x) + _grads(lambda t: q.act_quantized_relu_with_minmax(t), whole)
            + _grads(lambda t: q.act_quantized_dropout(t, 0.3), x)
            + _grads(lambda t: q.act_quantized_max_pool2d(t, (3, 3), (2, 2), (1, 1), (1, 1), False, False), x)
            + _grads(lambda t: q.act_quantized_max_pool2d(t, (3, 2), (1, 3), (1, 0), (2, 1), False, False), x))


def _helpers(dtype):
    from actnn_b200.cpp_extension import backward_func as bf
    from actnn_b200.cpp_extension import calc_precision as cp
    x = torch.randn(5, 24, 7, 9, device="cuda").to(dtype)
    out = [cp.sample_sumsq(x), cp.sample_sumsq(x.transpose(1, 3))]
    if dtype != torch.float32:
        last = bf.to_channels_last(x)
        assert last.is_contiguous(memory_format=torch.channels_last) and torch.equal(last, x)
        out += [last.permute(0, 2, 3, 1).contiguous(), bf.to_planes(last)]
    return out


CASES = {
    "ragged adaptive": lambda dt: _codec((9, 5, 11, 7), "L3", dt), "whole adaptive": lambda dt: _codec((9, 16, 16, 8), "L3", dt),
    "ragged uniform": lambda dt: _codec((9, 5, 11, 7), "L2", dt), "whole uniform": lambda dt: _codec((9, 16, 16, 8), "L2", dt),
    "batch norm 14": lambda dt: _batch_norm((10, 24, 14, 14), dt), "batch norm 16": lambda dt: _batch_norm((10, 24, 16, 16), dt),
    "batch norm 2": lambda dt: _batch_norm((10, 24, 2, 2), dt),
    "batch norm, cumulative average": lambda dt: _batch_norm((10, 24, 5, 5), dt, momentum=None),
    "ranges of a ReLU": _ranges_of_a_relu, "mask layers": _mask_layers, "helpers": _helpers,
}


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("name", list(CASES))
def test_native_and_python_calls_agree(name, dtype, monkeypatch):
    import actnn_b200 as actnn
    from actnn_b200 import _lib
    results = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(_lib, "_native", False)
        assert bool(_lib.native()) == native
        actnn.QScheme.layers.clear()
        actnn.QBNScheme.layers.clear()
        torch.manual_seed(11)
        results.append(CASES[name](dtype))
    assert len(results[0]) == len(results[1])
    for a, b in zip(*results):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)
