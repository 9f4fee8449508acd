"""The kept ticket of the allocation kernels, and stream capture."""
import pytest
import torch


def test_a_capture_gets_a_ticket_of_its_own(monkeypatch):
    """Host logic only: tensors on the CPU stand in for the device's."""
    from actnn_b200 import _lib
    capturing = False
    monkeypatch.setattr(_lib, "_tickets", {})
    monkeypatch.setattr(_lib, "stream_of_index", lambda idx: 77)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
    dev = torch.device("cpu")
    capturing = True
    first = _lib.ticket(dev)
    assert not _lib._tickets and first.numel() == 256 and not first.any()
    capturing = False
    kept = _lib.ticket(dev)
    assert _lib.ticket(dev) is kept and kept is not first
    capturing = True
    assert _lib.ticket(dev) is not kept


@pytest.mark.gpu
def test_batch_norm_forward_captured_before_it_ran_eagerly():
    """On a stream without a ticket: capture, then the eager call on that stream, then replays on another one."""
    from actnn_b200.cpp_extension import backward_func as bf
    n, c, hw = 40, 24, 49
    x = torch.randn(n, c, hw, device="cuda", dtype=torch.float16)
    weight, bias = torch.rand(c, device="cuda") + 0.5, torch.randn(c, device="cuda")

    def forward():
        y, quantized, mean, invstd = bf.batch_norm_codes_forward(x, weight, bias, None, None, 0.1, 1e-5, 2 * n, 8, 0.5, False)
        return (y, *quantized, mean, invstd)

    ref = forward()
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        captured = forward()
    with torch.cuda.stream(stream):
        eager = forward()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(eager, ref))
    for _ in range(2):
        for t in captured:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(captured, ref))
