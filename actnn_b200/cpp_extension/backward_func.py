"""Backward operators under the names the reference re-exports
(actnn/actnn/cpp_extension/backward_func.cc:81-91).

PyTorch 2.x dropped ``cudnn_convolution_backward`` / ``cudnn_convolution_transpose_backward``
in favour of ``convolution_backward``; the two names are kept here with the reference's
argument order and are routed to that operator: the dense convolution math stays in cuDNN.

``cudnn_batch_norm`` / ``cudnn_batch_norm_backward`` keep the reference's names, arguments
and return values, but the training-mode work is done by this package's own kernels
(``actnn_batch_norm_forward`` / ``actnn_batch_norm_backward`` of the C ABI), which spread a
channel over many blocks instead of cuDNN's one block per channel.  ``batch_norm_stats``,
``batch_norm_elemt``, ``batch_norm_backward_reduce`` and ``batch_norm_backward_elemt`` are
the same kernels under the names of the ATen operators the reference's synchronised batch
norm calls (ops.py:515-603)."""
import ctypes
import functools

import torch

from .. import _lib
from . import quantization

aten = torch.ops.aten


class _cudnn_benchmark:
    """``torch.backends.cudnn.benchmark = flag`` for the duration of a call; the global is only
    touched when it differs (the usual case, one setting for a whole run, costs nothing)."""

    def __init__(self, flag):
        self.flag = bool(flag)
        self.prev = None

    def __enter__(self):
        cur = torch.backends.cudnn.benchmark
        if cur != self.flag:
            self.prev = cur
            torch.backends.cudnn.benchmark = self.flag

    def __exit__(self, *exc):
        if self.prev is not None:
            torch.backends.cudnn.benchmark = self.prev
        return False


def cudnn_convolution_backward(input, grad_output, weight, padding, stride, dilation, groups,
                               benchmark, deterministic, allow_tf32, output_mask):
    with _cudnn_benchmark(benchmark):
        gi, gw, _ = aten.convolution_backward(
            grad_output, input, weight, None, list(stride), list(padding), list(dilation), False,
            [0] * len(stride), groups, [bool(output_mask[0]), bool(output_mask[1]), False])
    return gi, gw


def cudnn_convolution_transpose_backward(input, grad_output, weight, padding, output_padding, stride,
                                         dilation, groups, benchmark, deterministic, allow_tf32,
                                         output_mask):
    with _cudnn_benchmark(benchmark):
        gi, gw, _ = aten.convolution_backward(
            grad_output, input, weight, None, list(stride), list(padding), list(dilation), True,
            list(output_padding), groups, [bool(output_mask[0]), bool(output_mask[1]), False])
    return gi, gw


# ---------------------------------------------------------------------------------------
# channels-last around the convolution library
# ---------------------------------------------------------------------------------------
CHANNELS_LAST_ELEMENTS = 1 << 24          # smallest input that is converted, see channels_last_pays


def channels_last_pays(input, weight, groups) -> bool:
    """Whether a 2-D convolution of contiguous NCHW tensors is computed on channels-last copies.

    cuDNN has only NHWC kernels for 16-bit convolutions with more than one tap on this GPU, so for
    NCHW operands it converts each of them in every call (in a backward pass the gradient twice).  Measured on a
    B200, float16, forward + backward: 3x3, 256 x 64 x 56 x 56: 742 us on NCHW, 230 on NHWC operands, 31
    per converted tensor; 256 x 256 x 28 x 28: 920 against 509.  1x1 convolutions are matrix products in
    either layout (188 against 157, less than the conversions cost) and stay; so do channel counts that
    NHWC kernels cannot read in 16-byte vectors, and grouped convolutions.  float32 stays because the transpose is written
    for 16-bit elements and no case calls for another: its convolutions are converted by cuDNN, too, but in the classifier of
    32 x 32 images that is 122 of 1019 us on the GPU in a step of 2446 that waits for the host.  Small layers are paced
    by the host, to which the library's own conversions are cheaper than seven calls: convolution + ReLU, forward +
    backward, 128 x 64 x 28 x 28 (6.4 M elements) 265 us on NCHW against 288, 12.8 M elements 277 against 285;
    from 25 M elements on the conversions are GPU time (bottleneck block at batch 256: 253 us of cuDNN's against 93)."""
    return (input.dim() == 4 and input.is_cuda and input.dtype in (torch.float16, torch.bfloat16)
            and weight.dtype == input.dtype and groups == 1 and weight.shape[2] * weight.shape[3] > 1
            and weight.shape[0] % 8 == 0 and weight.shape[1] % 8 == 0 and input.shape[1] == weight.shape[1]
            and input.numel() >= CHANNELS_LAST_ELEMENTS and input.shape[2] * input.shape[3] > 1
            and input.is_contiguous() and weight.is_contiguous()
            and torch.backends.cudnn.enabled)


def to_channels_last(x):
    """A channels-last copy of a contiguous 16-bit NCHW tensor."""
    nat = _lib.native()
    if nat:
        return nat.transpose16(x, True)
    n, c, h, w = x.shape
    out = torch.empty(x.shape, dtype=x.dtype, device=x.device, memory_format=torch.channels_last)
    _lib.call("actnn_transpose16", x, x.data_ptr(), out.data_ptr(), n, c, h * w, _lib.stream_of(x))
    return out


def to_planes(x):
    """The contiguous NCHW form of a 16-bit tensor that came back channels-last."""
    if x.is_contiguous() or not x.is_contiguous(memory_format=torch.channels_last):
        return x.contiguous()
    nat = _lib.native()
    if nat:
        return nat.transpose16(x, False)
    n, c, h, w = x.shape
    out = torch.empty(x.shape, dtype=x.dtype, device=x.device)
    _lib.call("actnn_transpose16", x, x.data_ptr(), out.data_ptr(), n, h * w, c, _lib.stream_of(x))
    return out


def _as_f32(t):
    return None if t is None else (t if t.dtype == torch.float32 else t.float()).contiguous()


def _bn_dims(input):
    if input.dim() < 2:
        raise RuntimeError("batch_norm: expected an input of at least 2 dimensions, got %d" % input.dim())
    N, C = input.shape[0], input.shape[1]
    HW = input.numel() // (N * C) if N * C else 0
    return N, C, HW


def _bn_workspace(N, C, HW, device):
    """Scratch of the batch-norm kernels (they clear what must start at zero themselves), taken
    from the per-stream scratch buffer instead of the allocator."""
    nbytes = _lib.load().actnn_batch_norm_workspace(N, C, HW)
    return _lib.scratch(device, max(nbytes, 16)), nbytes


def cudnn_batch_norm(input, weight, bias, running_mean, running_var, training, exponential_average_factor,
                     epsilon):
    """Returns ``(output, save_mean, save_invstd, reserve)`` like ``at::cudnn_batch_norm``
    (reference call site: ops.py:457-458).  ``reserve`` is an empty byte tensor."""
    if not training:
        return aten.cudnn_batch_norm(input, weight, bias, running_mean, running_var, training,
                                     exponential_average_factor, epsilon)
    if not input.is_cuda:
        raise RuntimeError("cudnn_batch_norm: the input must be a CUDA tensor")
    x = input.contiguous()
    N, C, HW = _bn_dims(x)
    w32, b32 = _as_f32(weight), _as_f32(bias)
    for name, t in (("running_mean", running_mean), ("running_var", running_var)):
        if t is not None and (t.dtype != torch.float32 or not t.is_contiguous()):
            raise RuntimeError("cudnn_batch_norm: %s must be a contiguous float32 tensor" % name)
    y = torch.empty_like(x)
    save_mean = torch.empty(C, dtype=torch.float32, device=x.device)
    save_invstd = torch.empty(C, dtype=torch.float32, device=x.device)
    ws, nbytes = _bn_workspace(N, C, HW, x.device)
    _lib.call("actnn_batch_norm_forward", x, _lib.ptr(x), _lib.ptr(w32), _lib.ptr(b32), _lib.ptr(running_mean),
              _lib.ptr(running_var), _lib.ptr(y), _lib.ptr(save_mean), _lib.ptr(save_invstd), N, C, HW,
              float(exponential_average_factor), float(epsilon), _lib.dtype_id(x.dtype), _lib.ptr(ws), nbytes,
              _lib.stream_of(x))
    return y, save_mean, save_invstd, torch.empty(0, dtype=torch.uint8, device=x.device)


def cudnn_batch_norm_backward(input, grad_output, weight, running_mean, running_var, save_mean, save_var,
                              epsilon, reserve):
    """Returns ``(grad_input, grad_weight, grad_bias)`` like ``at::cudnn_batch_norm_backward``
    (reference call site: ops.py:492-493); ``save_var`` is the inverse standard deviation the
    forward saved."""
    if not input.is_cuda:
        raise RuntimeError("cudnn_batch_norm_backward: the input must be a CUDA tensor")
    x = input.contiguous()
    dy = grad_output.contiguous()
    if dy.dtype != x.dtype:
        dy = dy.to(x.dtype)
    N, C, HW = _bn_dims(x)
    w32 = _as_f32(weight)
    dx = torch.empty_like(x)
    dweight = torch.empty(C, dtype=torch.float32, device=x.device)
    dbias = torch.empty(C, dtype=torch.float32, device=x.device)
    ws, nbytes = _bn_workspace(N, C, HW, x.device)
    _lib.call("actnn_batch_norm_backward", x, _lib.ptr(x), _lib.ptr(dy), _lib.ptr(w32), _lib.ptr(save_mean),
              _lib.ptr(save_var), _lib.ptr(dx), _lib.ptr(dweight), _lib.ptr(dbias), N, C, HW,
              _lib.dtype_id(x.dtype), _lib.ptr(ws), nbytes, _lib.stream_of(x))
    if weight is not None and weight.dtype != torch.float32:
        dweight, dbias = dweight.to(weight.dtype), dbias.to(weight.dtype)
    return dx, dweight, dbias


@functools.lru_cache(maxsize=4096)
def _codes_workspace(N, C, HW, dtype_id, device_index):
    """Scratch bytes of ``actnn_batch_norm_codes_backward``; ``None``: a geometry it does not cover."""
    nbytes = ctypes.c_int64(0)
    with torch.cuda.device(device_index):
        status = _lib.load().actnn_batch_norm_codes_workspace(N, C, HW, dtype_id, ctypes.addressof(nbytes))
    return None if status else nbytes.value


def batch_norm_codes_forward(x, weight, bias, running_mean, running_var, momentum, eps, target_bits, initial_bits,
                             range_factor, stochastic, stats=None):
    """Training-mode batch norm of a contiguous ``x`` and its compressed copy in one native call:
    ``(y, (packed, bits, scale, min), mean, invstd)``, or ``None`` when the geometry is not covered (nothing
    has been drawn or written then).  ``stats``: what ``batch_norm_stats_minimax`` returned for ``x``, when it was
    called (and has updated the running statistics).  The same codes as ``compress_mixed_precision`` with the next Philox offset."""
    if x.dim() < 2 or x.dtype not in (torch.float16, torch.bfloat16, torch.float32) or x.numel() == 0:
        return None
    for t in (running_mean, running_var):
        if t is not None and (t.dtype != torch.float32 or not t.is_contiguous()):
            return None
    nat = _lib.native()
    if nat:
        out = nat.batch_norm_forward(x, weight, bias, running_mean, running_var, momentum, eps, int(target_bits),
                                     initial_bits, range_factor, bool(stochastic), *(stats or (None,) * 4),
                                     _lib.ticket(x.device))
        if out is None:
            return None
        y, packed, bits, scale, mn, mean, invstd, offsets = out
        packed.word_offsets = bits.word_offsets = offsets
        bits.total_bits = min(initial_bits * x.shape[0], max(int(target_bits), x.shape[0]))
        return y, (packed, bits, scale, mn), mean, invstd
    N, C, HW = _bn_dims(x)
    dev, dt = x.device, _lib.dtype_id(x.dtype)
    nbytes = _codes_workspace(N, C, HW, dt, dev.index)
    if nbytes is None:
        return None
    stat = torch.bfloat16 if x.dtype == torch.float32 else x.dtype
    G = (C * HW + 255) // 256
    total = min(initial_bits * N, max(int(target_bits), N))        # what the greedy ends with
    w32, b32 = _as_f32(weight), _as_f32(bias)
    y = torch.empty_like(x)
    packed = torch.empty(total * G * 8, dtype=torch.int32, device=dev)
    scale = torch.empty((N, G, 1), dtype=stat, device=dev)
    mn = torch.empty((N, G, 1), dtype=stat, device=dev)
    bits = torch.empty(N, dtype=torch.int32, device=dev)
    offsets = torch.empty(N + 1, dtype=torch.int64, device=dev)
    if stats is None:
        floats = torch.empty(2 * C + N, dtype=torch.float32, device=dev)      # mean, invstd, sensitivities
        gmn = gmx = None
        mean, invstd, sens = floats[:C], floats[C:2 * C], floats.data_ptr() + 8 * C
    else:
        gmn, gmx, mean, invstd = stats
        floats = torch.empty(N, dtype=torch.float32, device=dev)
        sens = floats.data_ptr()
    seed, offset = _lib.next_philox(dev) if stochastic else (0, 0)
    ws = _lib.scratch(dev, nbytes)
    _lib.call("actnn_batch_norm_codes_forward", x, x.data_ptr(), _lib.ptr(gmn), _lib.ptr(gmx), _lib.ptr(w32),
              _lib.ptr(b32), _lib.ptr(running_mean), _lib.ptr(running_var), y.data_ptr(), mean.data_ptr(),
              invstd.data_ptr(), packed.data_ptr(), scale.data_ptr(), mn.data_ptr(), bits.data_ptr(),
              offsets.data_ptr(), sens, N, C, HW, float(momentum), float(eps), dt,
              _lib.dtype_id(stat), float(range_factor), int(initial_bits), float(target_bits), int(bool(stochastic)),
              seed, offset, _lib.ticket(dev).data_ptr(), ws.data_ptr(), nbytes, _lib.stream_of(x))
    packed.word_offsets = bits.word_offsets = offsets
    bits.total_bits = total
    return y, (packed, bits, scale, mn), mean, invstd


def batch_norm_codes_backward(quantized, shape, dtype, grad_output, weight, save_mean, save_invstd):
    """Backward of a training-mode batch norm from the compressed input: what ``dequantize_activation``
    followed by ``cudnn_batch_norm_backward`` computes (ops.py:470-493), with the decoded input in
    registers only.  ``quantized``: ``(packed, bits, scale, min)`` of the mixed stream, on the device.
    Returns ``(grad_input, grad_weight, grad_bias)``, or ``None`` when the geometry is not covered."""
    packed, bits, scale, mn = quantized
    if len(shape) < 2 or not packed.is_cuda or dtype not in (torch.float16, torch.bfloat16, torch.float32) \
            or scale.dtype != (torch.bfloat16 if dtype == torch.float32 else dtype):
        return None
    N, C = shape[0], shape[1]
    F = 1
    for d in shape[1:]:
        F *= d
    if N * F == 0 or tuple(scale.shape) != (N, (F + 255) // 256, 1) or bits.numel() != N:
        return None
    HW = F // C
    word_offsets = getattr(packed, "word_offsets", None)
    if word_offsets is None:
        word_offsets = quantization.bits_prefix(bits, scale.shape[1], 256)
    nat = _lib.native()
    if nat:
        out = nat.batch_norm_backward(packed, bits, word_offsets, scale, mn, shape, grad_output,
                                      dtype == torch.float32, weight, save_mean, save_invstd)
        if out is not None and weight is not None and weight.dtype != torch.float32:
            out = out[0], out[1].to(weight.dtype), out[2].to(weight.dtype)
        return out
    dt = _lib.dtype_id(dtype)
    nbytes = _codes_workspace(N, C, HW, dt, packed.device.index)
    if nbytes is None:
        return None
    dy = grad_output.contiguous()
    if dy.dtype != dtype:
        dy = dy.to(dtype)
    w32 = _as_f32(weight)
    dx = torch.empty(shape, dtype=dtype, device=packed.device)
    dweight = torch.empty(C, dtype=torch.float32, device=packed.device)
    dbias = torch.empty(C, dtype=torch.float32, device=packed.device)
    ws = _lib.scratch(packed.device, nbytes)
    _lib.call("actnn_batch_norm_codes_backward", packed, packed.data_ptr(), bits.data_ptr(), word_offsets.data_ptr(),
              scale.data_ptr(), mn.data_ptr(), dy.data_ptr(), _lib.ptr(w32), save_mean.data_ptr(),
              save_invstd.data_ptr(), dx.data_ptr(), dweight.data_ptr(), dbias.data_ptr(), N, C, HW, dt,
              _lib.dtype_id(scale.dtype), ws.data_ptr(), nbytes, _lib.stream_of(packed))
    if weight is not None and weight.dtype != torch.float32:
        dweight, dbias = dweight.to(weight.dtype), dbias.to(weight.dtype)
    return dx, dweight, dbias


def batch_norm_stats(input, eps, out=None):
    """``torch.batch_norm_stats``: per-channel ``(mean, invstd)`` of this rank's batch
    (reference call site: ops.py:515).  ``out``: an optional contiguous float32 buffer of at
    least ``2 * C`` elements that receives mean then invstd (the message a synchronised batch
    norm gathers), so that no concatenation is needed."""
    x = input.contiguous()
    N, C, HW = _bn_dims(x)
    if out is None:
        out = torch.empty(2 * C, dtype=torch.float32, device=x.device)
    elif out.dtype != torch.float32 or not out.is_contiguous() or out.numel() < 2 * C or out.device != x.device:
        raise RuntimeError("batch_norm_stats: out must be a contiguous float32 tensor of >= 2*C elements")
    ws, nbytes = _bn_workspace(N, C, HW, x.device)
    _lib.call("actnn_batch_norm_stats", x, _lib.ptr(x), out.data_ptr(), out.data_ptr() + 4 * C, N, C, HW, float(eps),
              _lib.dtype_id(x.dtype), _lib.ptr(ws), nbytes, _lib.stream_of(x))
    flat = out.view(-1)
    return flat[:C], flat[C:2 * C]


def batch_norm_stats_minimax(input, weight, bias, running_mean, running_var, momentum, eps, out=None):
    """Batch-norm statistics AND the codec's per-group min / max from one read of ``input``
    (the reference reads it once for each: ops.py:456-458 / :515 and qbnscheme.py:28-40).

    Returns ``(mn, mx, mean, invstd)`` -- ``mn`` / ``mx`` shaped ``[N, G, 1]`` in the input's
    dtype, ``mean`` / ``invstd`` float32 ``[C]`` -- or ``None`` when the geometry is not covered
    (then the caller takes the two-read path).  ``running_mean`` / ``running_var`` are updated
    when given; ``out``: optional float32 buffer of >= 2 * C elements for mean then invstd.
    ``weight`` and ``bias`` are not looked at (they are in the calls programs have)."""
    if not input.is_cuda or not input.is_contiguous() or input.dim() < 2:
        return None
    for t in (running_mean, running_var):
        if t is not None and (t.dtype != torch.float32 or not t.is_contiguous()):
            return None
    nat = _lib.native()
    if nat:
        return nat.batch_norm_stats_minimax(input, running_mean, running_var, momentum, eps, out)
    N, C, HW = _bn_dims(input)
    dev = input.device
    nbytes = _lib.load().actnn_batch_norm_stats_minimax_workspace(N, C, HW)
    if nbytes < 0:
        return None
    if out is not None and (out.dtype != torch.float32 or not out.is_contiguous() or out.numel() < 2 * C or out.device != dev):
        raise RuntimeError("batch_norm_stats_minimax: out must be a contiguous float32 tensor of >= 2*C elements")
    G = C * HW // 256
    mn = torch.empty((N, G, 1), dtype=input.dtype, device=dev)
    mx = torch.empty((N, G, 1), dtype=input.dtype, device=dev)
    if out is None:
        out = torch.empty(2 * C, dtype=torch.float32, device=dev)
    ws = _lib.scratch(dev, nbytes)
    _lib.call("actnn_batch_norm_stats_minimax", input, _lib.ptr(input), mn.data_ptr(), mx.data_ptr(), 0, 0,
              _lib.ptr(running_mean), _lib.ptr(running_var), out.data_ptr(), out.data_ptr() + 4 * C,
              N, C, HW, float(momentum), float(eps), _lib.dtype_id(input.dtype), ws.data_ptr(), nbytes,
              _lib.stream_of(input))
    flat = out.view(-1)
    return mn, mx, flat[:C], flat[C:2 * C]


def batch_norm_elemt(input, weight, bias, mean, invstd, eps):
    """``torch.batch_norm_elemt``: normalise with given statistics (ops.py:554)."""
    x = input.contiguous()
    N, C, HW = _bn_dims(x)
    y = torch.empty_like(x)
    ws = _lib.scratch(x.device, max(16 * C, 16))
    # the converted copies must outlive the call: a pointer taken from a temporary would dangle
    w32, b32, m32, i32 = _as_f32(weight), _as_f32(bias), _as_f32(mean), _as_f32(invstd)
    _lib.call("actnn_batch_norm_elemt", x, _lib.ptr(x), _lib.ptr(w32), _lib.ptr(b32), _lib.ptr(m32), _lib.ptr(i32),
              _lib.ptr(y), N, C, HW, _lib.dtype_id(x.dtype), _lib.ptr(ws), 16 * C, _lib.stream_of(x))
    return y


def batch_norm_backward_reduce(grad_out, input, mean, invstd, weight, input_g, weight_g, bias_g, out=None):
    """``torch.batch_norm_backward_reduce``: ``(sum_dy, sum_dy_xmu, grad_weight, grad_bias)`` of this
    rank (ops.py:570-577).  ``out``: optional contiguous float32 ``[2 * C]`` buffer that receives
    sum_dy then sum_dy_xmu (the message a synchronised batch norm all-reduces)."""
    x = input.contiguous()
    dy = grad_out.contiguous()
    if dy.dtype != x.dtype:
        dy = dy.to(x.dtype)
    N, C, HW = _bn_dims(x)
    if out is None:
        out = torch.empty(2 * C, dtype=torch.float32, device=x.device)
    elif out.dtype != torch.float32 or not out.is_contiguous() or out.numel() < 2 * C or out.device != x.device:
        raise RuntimeError("batch_norm_backward_reduce: out must be a contiguous float32 tensor of >= 2*C elements")
    grad_weight = torch.empty(C, dtype=torch.float32, device=x.device)
    ws, nbytes = _bn_workspace(N, C, HW, x.device)
    w32, m32, i32 = _as_f32(weight), _as_f32(mean), _as_f32(invstd)       # kept alive across the call
    _lib.call("actnn_batch_norm_backward_reduce", x, _lib.ptr(x), _lib.ptr(dy), _lib.ptr(w32),
              _lib.ptr(m32), _lib.ptr(i32), out.data_ptr(), out.data_ptr() + 4 * C,
              _lib.ptr(grad_weight), N, C, HW, _lib.dtype_id(x.dtype), _lib.ptr(ws), nbytes, _lib.stream_of(x))
    flat = out.view(-1)
    sum_dy, sum_dy_xmu = flat[:C], flat[C:2 * C]
    grad_bias = sum_dy.clone() if bias_g else None             # the message buffer is all-reduced in place later
    if weight is not None and weight.dtype != torch.float32:
        grad_weight = grad_weight.to(weight.dtype)
        grad_bias = None if grad_bias is None else grad_bias.to(weight.dtype)
    return sum_dy, sum_dy_xmu, (grad_weight if weight_g else None), grad_bias


def batch_norm_backward_elemt(grad_out, input, mean, invstd, weight, sum_dy, sum_dy_xmu, count):
    """``torch.batch_norm_backward_elemt``: the input gradient from sums over all ranks; ``count``
    holds every rank's elements per channel and stays on the device (ops.py:594-603)."""
    x = input.contiguous()
    dy = grad_out.contiguous()
    if dy.dtype != x.dtype:
        dy = dy.to(x.dtype)
    N, C, HW = _bn_dims(x)
    counts = count.reshape(-1).to(torch.float32).contiguous()
    dx = torch.empty_like(x)
    ws = _lib.scratch(x.device, max(16 * C, 16))
    w32, m32, i32 = _as_f32(weight), _as_f32(mean), _as_f32(invstd)       # kept alive across the call
    sdy, sdx = _as_f32(sum_dy), _as_f32(sum_dy_xmu)
    _lib.call("actnn_batch_norm_backward_elemt", x, _lib.ptr(x), _lib.ptr(dy), _lib.ptr(w32),
              _lib.ptr(m32), _lib.ptr(i32), _lib.ptr(sdy),
              _lib.ptr(sdx), _lib.ptr(counts), counts.numel(), _lib.ptr(dx), N, C, HW,
              _lib.dtype_id(x.dtype), _lib.ptr(ws), 16 * C, _lib.stream_of(x))
    return dx


def native_batch_norm(input, weight, bias, running_mean, running_var, training, momentum, eps):
    return aten.native_batch_norm(input, weight, bias, running_mean, running_var, training, momentum, eps)


def native_batch_norm_backward(grad_out, input, weight, running_mean, running_var, save_mean, save_invstd,
                               train, eps, output_mask):
    return aten.native_batch_norm_backward(grad_out, input, weight, running_mean, running_var, save_mean,
                                           save_invstd, train, eps, list(output_mask))
