// Batched transpose of 16-bit matrices: [rows, cols] -> [cols, rows] for every sample, i.e. NCHW <-> NHWC.
//
// The convolution library computes in NHWC on this GPU and converts NCHW operands on every call: twice the
// input gradient's operands in a backward pass, for instance.  Converting each tensor once with this kernel
// and handing the library NHWC tensors leaves its conversions out (actnn/actnn/ops.py:163-220 is where the
// reference calls it).  Bound by HBM: one read and one write.  A block moves a tile of 64 x 64 elements
// through shared memory: vectors along the columns in, vectors along the rows out, pairs of columns per
// 32-bit word, rows padded to 33 words (stores conflict-free, reads two-way).
#include "common.cuh"

namespace actnn {
namespace {

constexpr int kTile = 64;
constexpr int kLayoutThreads = 256;

template <int V> struct Vec16;
template <> struct Vec16<8> { using type = uint4; };
template <> struct Vec16<4> { using type = uint2; };
template <> struct Vec16<2> { using type = uint32_t; };
template <> struct Vec16<1> { using type = uint16_t; };

// VL / VS: elements per load / store; cols % VL == 0, rows % VS == 0 and the pointers are aligned to them.
template <int VL, int VS>
__global__ void __launch_bounds__(kLayoutThreads)
transpose16_kernel(const uint16_t* __restrict__ in, uint16_t* __restrict__ out, int rows, int cols, uint32_t row_tiles,
                   uint32_t col_tiles) {
  __shared__ uint32_t tile[kTile][kTile / 2 + 1];
  const uint32_t per = row_tiles * col_tiles;
  const uint32_t b = blockIdx.x / per, t = blockIdx.x - b * per;
  const int r0 = (int)(t / col_tiles) * kTile, c0 = (int)(t % col_tiles) * kTile;
  const int64_t base = (int64_t)b * rows * cols;
  constexpr int kLoads = kTile * kTile / VL / kLayoutThreads;
  using L = typename Vec16<VL>::type;
  L v[kLoads];
#pragma unroll
  for (int k = 0; k < kLoads; ++k) {
    const int i = k * kLayoutThreads + threadIdx.x, r = r0 + i / (kTile / VL), c = c0 + i % (kTile / VL) * VL;
    if (r < rows && c < cols) v[k] = __ldg(reinterpret_cast<const L*>(in + base + (int64_t)r * cols + c));
  }
#pragma unroll
  for (int k = 0; k < kLoads; ++k) {
    const int i = k * kLayoutThreads + threadIdx.x, r = i / (kTile / VL), c = i % (kTile / VL) * VL;
    if constexpr (VL == 1) {
      reinterpret_cast<uint16_t*>(tile[r])[c] = v[k];
    } else {
      const uint32_t* w = reinterpret_cast<const uint32_t*>(&v[k]);
#pragma unroll
      for (int j = 0; j < VL / 2; ++j) tile[r][c / 2 + j] = w[j];
    }
  }
  __syncthreads();
  using S = typename Vec16<VS>::type;
  constexpr int kGroups = kTile / VS;                          // stores along a row of the output
#pragma unroll
  for (int i = threadIdx.x; i < kGroups * kTile / 2; i += kLayoutThreads) {
    const int g = i % kGroups, pair = i / kGroups;
    const int r = r0 + g * VS, c = c0 + 2 * pair;
    if (r >= rows || c >= cols) continue;
    uint16_t lo[VS], hi[VS];
#pragma unroll
    for (int j = 0; j < VS; ++j) {
      const uint32_t w = tile[g * VS + j][pair];
      lo[j] = (uint16_t)w;
      hi[j] = (uint16_t)(w >> 16);
    }
    S a, z;
    __builtin_memcpy(&a, lo, sizeof(S));
    __builtin_memcpy(&z, hi, sizeof(S));
    uint16_t* o = out + base + (int64_t)c * rows + r;
    *reinterpret_cast<S*>(o) = a;
    if (c + 1 < cols) *reinterpret_cast<S*>(o + rows) = z;
  }
}

template <int VL, int VS>
int launch(const void* in, void* out, int64_t batch, int64_t rows, int64_t cols, cudaStream_t s) {
  const int64_t rt = (rows + kTile - 1) / kTile, ct = (cols + kTile - 1) / kTile;
  if (batch * rt * ct > 0x7fffffff) return ACTNN_ERR_SHAPE;
  transpose16_kernel<VL, VS><<<(unsigned)(batch * rt * ct), kLayoutThreads, 0, s>>>(
      (const uint16_t*)in, (uint16_t*)out, (int)rows, (int)cols, (uint32_t)rt, (uint32_t)ct);
  return check_launch();
}

int vector_width(const void* p, int64_t extent) {
  int v = 8;
  while (v > 1 && (extent % v != 0 || !aligned(p, 2 * v))) v >>= 1;
  return v;
}

}  // namespace
}  // namespace actnn

using namespace actnn;

extern "C" int actnn_transpose16(const void* in, void* out, int64_t batch, int64_t rows, int64_t cols,
                                 actnn_stream_t stream) {
  if (batch < 0 || rows < 0 || cols < 0 || rows > 0x7fffff00 || cols > 0x7fffff00) return ACTNN_ERR_SHAPE;
  if (batch == 0 || rows == 0 || cols == 0) return ACTNN_OK;
  if (!in || !out) return ACTNN_ERR_NULL;
  if (!aligned(in, 2) || !aligned(out, 2)) return ACTNN_ERR_ALIGN;
  cudaStream_t s = (cudaStream_t)stream;
  const int vl = vector_width(in, cols), vs = vector_width(out, rows);
  // one side is the channels in practice, a multiple of eight; the other is whatever the maps are
  if (vs == 8) {
    switch (vl) {
      case 8: return launch<8, 8>(in, out, batch, rows, cols, s);
      case 4: return launch<4, 8>(in, out, batch, rows, cols, s);
      case 2: return launch<2, 8>(in, out, batch, rows, cols, s);
      default: return launch<1, 8>(in, out, batch, rows, cols, s);
    }
  }
  if (vl == 8) {
    switch (vs) {
      case 4: return launch<8, 4>(in, out, batch, rows, cols, s);
      case 2: return launch<8, 2>(in, out, batch, rows, cols, s);
      default: return launch<8, 1>(in, out, batch, rows, cols, s);
    }
  }
  return launch<1, 1>(in, out, batch, rows, cols, s);
}
