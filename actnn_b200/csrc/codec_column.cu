// The mixed-precision codec on [N, F] activations whose samples are not whole groups of 256, or not
// a multiple of four groups: min / max, pack and unpack on the column mapping (column.cuh), reading
// and writing the activation where it is.  Large activations are packed in the order of the stream instead
// (codec_ragged.cu).  (The reference pads every sample with a concatenation and strips the padding with a copy,
// actnn/actnn/qscheme.py:61-71 and ops.py:137-139.)
//
// Bound by HBM at large sizes and by launches at small ones.  float16, compress and decompress of
// 100 x 192 x 35 x 35 (918.75 groups a sample): 127.1 -> 60.6 us, of which the padded copy was 18 and the
// cut-out copy 49 (52.1 with the pack in the order of the stream); 8 x 16 x 14 x 14: 81.1 -> 46.4 us (seven kernels -> four).
#include "column.cuh"

namespace actnn {
namespace {

// min / max of every group.  `clear_word` (optional) is set to zero: the ticket of the next kernel.
// Samples are walked from the last to the first, the order that leaves what the pack reads first
// in the L2.
template <typename T, bool EDGE>
__global__ void __launch_bounds__(kColThreads)
column_minimax_kernel(const T* __restrict__ data, ColumnShape sh, T* __restrict__ mn, T* __restrict__ mx,
                      unsigned* __restrict__ clear_word) {
  const int lane = threadIdx.x & 31;
  if (clear_word && blockIdx.x == 0 && threadIdx.x == 0) *clear_word = 0u;
  const ColumnTask t = column_task(sh);
  if (!t.valid) return;
  const ColumnOctets<EDGE> oct(sh, t, lane);
  Oct<T> next[kBundle];
  oct.template load<T>(data + (int64_t)(t.n1 - 1) * sh.F, next);
  for (int n = t.n1 - 1; n >= t.n0; --n) {
    Oct<T> x[kBundle];
#pragma unroll
    for (int gi = 0; gi < kBundle; ++gi) x[gi] = next[gi];
    if (n > t.n0) oct.template load<T>(data + (int64_t)(n - 1) * sh.F, next);
    float lo = 0.f, hi = 0.f;
    bundle_minmax<T>(x, lane, lo, hi);
    if (lane < t.count) {
      const int64_t q = (int64_t)n * sh.G + t.g0 + lane;
      store_scalar<T>(mn, q, lo);
      store_scalar<T>(mx, q, hi);
    }
  }
}

template <typename T, typename ST, bool PHILOX, bool EDGE>
__global__ void __launch_bounds__(kColThreads, 2)
column_pack_kernel(const T* __restrict__ data, ColumnShape sh, const T* __restrict__ mn, const T* __restrict__ mx,
                   const int32_t* __restrict__ bits, const int64_t* __restrict__ word_offsets,
                   int32_t* __restrict__ packed, ST* __restrict__ scale, ST* __restrict__ mn_out,
                   const T* __restrict__ noise, const NoiseKey key) {
  const int lane = threadIdx.x & 31;
  const ColumnTask t = column_task(sh);
  if (!t.valid) return;
  const ColumnOctets<EDGE> oct(sh, t, lane);
  pack_column<T, ST, PHILOX>(data, sh, t, oct, mn, mx, bits, word_offsets, packed, scale, mn_out, noise, key, lane, false,
                             [](int, const Oct<T> (&)[kBundle]) {});
}

template <typename T, typename ST, bool EDGE>
__global__ void __launch_bounds__(kColThreads, 3)
column_unpack_kernel(const int32_t* __restrict__ packed, const int32_t* __restrict__ bits,
                     const int64_t* __restrict__ word_offsets, const ST* __restrict__ scale,
                     const ST* __restrict__ mn, ColumnShape sh, T* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const ColumnTask t = column_task(sh);
  if (!t.valid) return;
  const ColumnOctets<EDGE> oct(sh, t, lane);
  const TransposePlan plan = make_transpose_plan(lane);
  const WordOrder<T> order(lane);
  for (int nb = t.n0; nb < t.n1; nb += 32) {
    const int nl = min(32, t.n1 - nb);
    ColumnStream st;
    st.open(t, nb + lane, lane < nl, bits, word_offsets);
    BundleWords next = st.fetch<T, ST>(t, order, sh.G, nb, 0, packed, scale, mn, lane);
    for (int i = 0; i < nl; ++i) {
      const BundleWords cur = next;
      if (i + 1 < nl) next = st.fetch<T, ST>(t, order, sh.G, nb + i + 1, i + 1, packed, scale, mn, lane);
      T* sample = out + (int64_t)(nb + i) * sh.F;
      decode_column<T>(cur, t.count, plan, lane,
                       [&](int gi, const Oct<T>& x) { oct.template store<T>(sample, gi, x); });
    }
  }
}

constexpr int kPackWarps = 16, kUnpackWarps = 24, kMinimaxWarps = 32;     // resident warps per SM the grids are sized for

template <typename T>
int launch_minimax(const void* data, void* mn, void* mx, int64_t N, int64_t F, unsigned* clear_word, cudaStream_t s) {
  const int al = octet_alignment(data, F, sizeof(T));
  const ColumnShape sh = column_shape(N, F, al, kMinimaxWarps);
  const bool edge = al != kOct || F % kGroup != 0;
  auto kernel = edge ? column_minimax_kernel<T, true> : column_minimax_kernel<T, false>;
  kernel<<<column_grid(sh), kColThreads, 0, s>>>((const T*)data, sh, (T*)mn, (T*)mx, clear_word);
  return check_launch();
}

template <typename T, typename ST>
int launch_pack(const void* data, const void* mn, const void* mx, const int32_t* bits, const int64_t* word_offsets,
                int32_t* packed, void* scale, void* mn_out, int64_t N, int64_t F, int stochastic, const void* noise,
                uint64_t seed, uint64_t offset, cudaStream_t s) {
  const int al = octet_alignment(data, F, sizeof(T));
  const ColumnShape sh = column_shape(N, F, al, kPackWarps);
  const bool edge = al != kOct || F % kGroup != 0;
  const bool philox = stochastic && !noise;
  const NoiseKey key = make_noise_key(seed, offset);
  auto kernel = philox ? (edge ? column_pack_kernel<T, ST, true, true> : column_pack_kernel<T, ST, true, false>)
                       : (edge ? column_pack_kernel<T, ST, false, true> : column_pack_kernel<T, ST, false, false>);
  kernel<<<column_grid(sh), kColThreads, 0, s>>>((const T*)data, sh, (const T*)mn, (const T*)mx, bits, word_offsets,
                                                 packed, (ST*)scale, (ST*)mn_out,
                                                 (const T*)(stochastic ? noise : nullptr), key);
  return check_launch();
}

template <typename T, typename ST>
int launch_unpack(const int32_t* packed, const int32_t* bits, const int64_t* word_offsets, const void* scale,
                  const void* mn, void* out, int64_t N, int64_t F, cudaStream_t s) {
  const int al = octet_alignment(out, F, sizeof(T));
  const ColumnShape sh = column_shape(N, F, al, kUnpackWarps);
  const bool edge = al != kOct || F % kGroup != 0;
  auto kernel = edge ? column_unpack_kernel<T, ST, true> : column_unpack_kernel<T, ST, false>;
  kernel<<<column_grid(sh), kColThreads, 0, s>>>(packed, bits, word_offsets, (const ST*)scale, (const ST*)mn, sh,
                                                 (T*)out);
  return check_launch();
}

}  // namespace

int column_minimax(const void* data, void* mn, void* mx, int64_t N, int64_t F, int dtype, unsigned* clear_word,
                   cudaStream_t s) {
  if (!column_supported(N, F)) return ACTNN_ERR_SHAPE;
  switch (dtype) {
    case ACTNN_F32: return launch_minimax<float>(data, mn, mx, N, F, clear_word, s);
    case ACTNN_F16: return launch_minimax<__half>(data, mn, mx, N, F, clear_word, s);
    case ACTNN_BF16: return launch_minimax<__nv_bfloat16>(data, mn, mx, N, F, clear_word, s);
    default: return ACTNN_ERR_DTYPE;
  }
}

int column_pack(const void* data, const void* mn, const void* mx, const int32_t* bits, const int64_t* word_offsets,
                int32_t* packed, void* scale, void* mn_out, int64_t N, int64_t F, int dtype, int stat_dtype,
                int stochastic, const void* noise, uint64_t seed, uint64_t offset, double width, cudaStream_t s) {
  if (!column_supported(N, F)) return ACTNN_ERR_SHAPE;
  if (stochastic && noise && !aligned(noise, dtype == ACTNN_F32 ? 32 : 16)) return ACTNN_ERR_ALIGN;
  if (ragged_pays(N, F, dtype, width))
    return ragged_pack(data, mn, mx, bits, word_offsets, packed, scale, mn_out, N, F, dtype, stat_dtype, stochastic,
                       noise, seed, offset, s);
#define ACTNN_PACK(T, ST)                                                                                         \
  return launch_pack<T, ST>(data, mn, mx, bits, word_offsets, packed, scale, mn_out, N, F, stochastic, noise, seed, \
                            offset, s)
  switch (dtype) {
    case ACTNN_F16: ACTNN_PACK(__half, __half);
    case ACTNN_BF16: ACTNN_PACK(__nv_bfloat16, __nv_bfloat16);
    default:
      if (stat_dtype == ACTNN_BF16) ACTNN_PACK(float, __nv_bfloat16);
      ACTNN_PACK(float, float);
  }
#undef ACTNN_PACK
}

int column_unpack(const int32_t* packed, const int32_t* bits, const int64_t* word_offsets, const void* scale,
                  const void* mn, void* out, int64_t N, int64_t F, int dtype, int stat_dtype, cudaStream_t s) {
  if (!column_supported(N, F)) return ACTNN_ERR_SHAPE;
#define ACTNN_UNPACK(T, ST) return launch_unpack<T, ST>(packed, bits, word_offsets, scale, mn, out, N, F, s)
  switch (dtype) {
    case ACTNN_F16: ACTNN_UNPACK(__half, __half);
    case ACTNN_BF16: ACTNN_UNPACK(__nv_bfloat16, __nv_bfloat16);
    default:
      if (stat_dtype == ACTNN_BF16) ACTNN_UNPACK(float, __nv_bfloat16);
      ACTNN_UNPACK(float, float);
  }
#undef ACTNN_UNPACK
}
}  // namespace actnn

using namespace actnn;

extern "C" int actnn_unpack_mixed_samples(const int32_t* packed, const int32_t* bits, const int64_t* word_offsets,
                                          const void* scale, const void* mn, void* out, int64_t N, int64_t F,
                                          int dtype, int stat_dtype, actnn_stream_t stream) {
  if (N < 0 || F < 0) return ACTNN_ERR_SHAPE;
  if (dtype < ACTNN_F32 || dtype > ACTNN_BF16) return ACTNN_ERR_DTYPE;
  if (!(stat_dtype == dtype || (dtype == ACTNN_F32 && stat_dtype == ACTNN_BF16))) return ACTNN_ERR_DTYPE;
  if (N == 0 || F == 0) return ACTNN_OK;
  if (!packed || !bits || !word_offsets || !scale || !mn || !out) return ACTNN_ERR_NULL;
  if (!aligned(out, dtype_size(dtype)) || !aligned(packed, 4)) return ACTNN_ERR_ALIGN;
  return column_unpack(packed, bits, word_offsets, scale, mn, out, N, F, dtype, stat_dtype, (cudaStream_t)stream);
}
