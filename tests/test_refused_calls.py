"""Calls with arguments that make no sense end with an exception, never with the process (no GPU needed)."""
import pytest
import torch

GEOMETRY = {"kernel_size": (2, 2), "stride": (2, 2), "padding": (0, 0), "dilation": (1, 1)}


@pytest.mark.parametrize("name,value", [("stride", (0, 0)), ("stride", (2, 0)), ("stride", (-1, 2)), ("stride", (2 ** 32 + 2, 2)),
                                        ("kernel_size", (0, 2)), ("dilation", (1, 0)), ("padding", (-1, 0)),
                                        ("padding", (0, 2 ** 31))])
def test_max_pool_geometry(name, value):
    from actnn_b200 import _lib
    from actnn_b200.cpp_extension import quantization as q
    geom = dict(GEOMETRY, **{name: value})
    with pytest.raises(RuntimeError, match=name):
        q._pool_args(**geom)
    # the C++ half on its own: refused before it looks at the tensor's device or divides
    with pytest.raises(RuntimeError, match="must be positive"):
        _lib.native().max_pool2d(torch.zeros(1, 1, 4, 4), [v for pair in geom.values() for v in pair])


def test_max_pool_geometry_that_is_taken():
    from actnn_b200.cpp_extension import quantization as q
    assert q._pool_args(**GEOMETRY) == [2, 2, 2, 2, 0, 0, 1, 1]
    assert q._pool_args([3, 3], [1, 2 ** 31 - 1], [1, 1], [2, 1]) == [3, 3, 1, 2 ** 31 - 1, 1, 1, 2, 1]
