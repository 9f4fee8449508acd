// Pack of [N, F] activations whose samples are not whole groups of 256, or not a multiple of four groups, in the
// order of the stream: samples of many groups.  (Samples of few groups: the column kernels, codec_column.cu.)
//
// The bundles are the aligned groups 4k .. 4k+3 of the flat [N * G] list, as in the kernels for whole groups, so that a
// call of the noise generator serves each (columns of an odd G need two), and a bundle inside a sample is
// addressed and packed as there: only the sample's offset differs.  What is special happens in one bundle or two a
// sample, those that hold its last, partial group or groups of two samples; they are taken group by group.  A warp
// prepares up to 32 groups at a time, a group a lane.
// What bounds it: instruction issue (the generator, rounding); it runs at the pace of the pack of whole groups.
#include "flat_runs.cuh"

namespace actnn {
namespace {

constexpr int kThreads = 256;

struct RaggedShape {
  int64_t Q, G, F;            // groups in all, groups per sample, elements per sample
  int align;                  // elements that octets of the activation are aligned to
  int64_t pad;                // elements missing in the last group of a sample
};

// The bundles in tasks of up to eight, all of the same length or one less and as many for every warp; the warps take
// them in turn.  So the warps of a block are on neighbouring groups, mostly of one sample and one width, and share its
// code in the instruction caches, and every warp meets all parts of the activation.  (One run of consecutive bundles a
// warp had the warps of a block on different samples, and was slower than the columns where widths are many: float16
// compress of 512 x 785 groups, columns / runs / tasks in turn, 2 bits on average 120 / 103 / 96 us, 4 bits 128 / 147 /
// 113, 6 bits 136 / 158 / 129; float32 170 / 162 / 157, 178 / 211 / 165, 185 / 210 / 171.)
// FROM_END: the last task first, for float32: 200 x 900 groups 79.9 -> 74.0 us; float16 49.4 -> 49.0, 512 x 785 95.0 -> 97.1.
template <bool FROM_END> struct BundleTasks {
  int64_t next, stride, tasks, base, rem;
  ACTNN_DEV BundleTasks(int64_t Q) {
    const int64_t total = (Q + kFlatBundle - 1) / kFlatBundle;
    constexpr int kMost = kFlatGroups / kFlatBundle;
    next = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
    stride = ((int64_t)gridDim.x * kThreads) >> 5;
    tasks = min((total + stride * kMost - 1) / (stride * kMost) * stride, total);
    base = total / tasks;
    rem = total - base * tasks;
  }
  // Bundles of the next task, which begins with group q0; zero: no more.
  ACTNN_DEV int take(int64_t& q0) {
    if (next >= tasks) return 0;
    const int64_t t = FROM_END ? tasks - 1 - next : next;
    q0 = (t * base + min(t, rem)) * kFlatBundle;
    next += stride;
    return (int)(base + (t < rem ? 1 : 0));
  }
};

// The lane's group: its sample and place in it (-1: past the share or the activation), and the bundles of the share that
// are four whole groups of one sample (bit 4k: bundle k).
struct LaneGroup {
  int n, r;
  unsigned inner;
  ACTNN_DEV LaneGroup(const RaggedShape& sh, int64_t q0, int bundles, int lane) {
    const int64_t q = q0 + lane;
    n = r = -1;
    if (lane < bundles * kFlatBundle && q < sh.Q) {
      int64_t n64, r64;
      split_group_index(q, sh.G, n64, r64);
      n = (int)n64;
      r = (int)r64;
    }
    const int last_n = __shfl_sync(kFull, n, lane | 3), last_r = __shfl_sync(kFull, r, lane | 3);
    inner = __ballot_sync(kFull, (lane & 3) == 0 && n >= 0 && last_n == n && last_r < (int)sh.G - 1);
  }
  // Bundles k, k+1, ... (all inner) of the sample of bundle k.
  ACTNN_DEV int run(int k, int lane) const {
    const int first = k * kFlatBundle;
    const unsigned same = (__ballot_sync(kFull, n == __shfl_sync(kFull, n, first)) & inner) >> first;
    const unsigned other = ~same & 0x11111111u;
    return other ? (__ffs((int)other) - 1) >> 2 : kFlatGroups / kFlatBundle;
  }
};
ACTNN_DEV int64_t shfl64(int64_t v, int src) {
  const uint32_t lo = __shfl_sync(kFull, (uint32_t)v, src), hi = __shfl_sync(kFull, (uint32_t)((uint64_t)v >> 32), src);
  return (int64_t)(((uint64_t)hi << 32) | lo);
}
ACTNN_DEV int elements_left(const RaggedShape& sh, int r, int lane) {      // of the lane's octet in group r
  return (int)max((int64_t)0, min((int64_t)kOct, sh.F - ((int64_t)r * kGroup + lane * kOct)));
}

// ------------------------------------------------------------------ pack
template <typename T, int B>
ACTNN_DEV void pack_group(const Oct<T>& x, const Oct<T>& nz, const QP<T>& qp, int32_t* __restrict__ out,
                          const TransposePlan& plan, int lane) {
  uint32_t lo, hi;
  row_from_magic<T, B>(quantize_oct<T, false, B>(x, nz, qp), lo, hi);
  const uint32_t a = warp_transpose32(lo, plan);
  if (lane < 8 * B) out[lane] = (int32_t)a;
  if constexpr (B > 4) {
    const uint32_t b = warp_transpose32(hi, plan);
    if (lane < 8 * B - 32) out[32 + lane] = (int32_t)b;
  }
}

template <typename T, typename ST, int MODE, bool ALIGNED>
__global__ void __launch_bounds__(kThreads, 2)
pack_ragged_kernel(const T* __restrict__ data, const T* __restrict__ mn, const T* __restrict__ mx,
                   const int32_t* __restrict__ bits, const int64_t* __restrict__ word_offsets,
                   int32_t* __restrict__ packed, ST* __restrict__ scale, ST* __restrict__ mn_out, RaggedShape sh,
                   const T* __restrict__ noise, const NoiseKey key) {
  constexpr bool PREFETCH = sizeof(T) == 2;
  const int lane = threadIdx.x & 31;
  const TransposePlan plan = make_transpose_plan(lane);
  Oct<T> bufA[kFlatBundle], bufB[kFlatBundle];                  // bufB stays unused without PREFETCH
  BundleTasks<sizeof(T) == 4> tasks(sh.Q);
  int64_t q0;
  while (const int bundles = tasks.take(q0)) {
    const LaneGroup g(sh, q0, bundles, lane);
    int b_l = 0;
    int64_t off_l = 0;
    LaneParams<T> mine = {0u, 0u};
    if (g.n >= 0) {
      const int64_t q = q0 + lane;
      b_l = __ldg(bits + g.n);
      if (b_l < 1 || b_l > 8) b_l = 0;                          // not a width: nothing written
      off_l = __ldg(word_offsets + g.n) + (int64_t)g.r * (8 * b_l);
      const float gmn = load_scalar<T>(mn, q), gmx = load_scalar<T>(mx, q);
      const GroupParams gp = prepare_group<T>(gmn, gmx, b_l);
      store_scalar<ST>(scale, q, gp.scale);
      store_scalar<ST>(mn_out, q, gmn);
      mine = lane_params<T>(gp);
    }
    int k = 0;
    while (k < bundles) {
      const int first = k * kFlatBundle;
      if ((g.inner >> first) & 1u) {
        const int k1 = k + g.run(k, lane);
        const int n = __shfl_sync(kFull, g.n, first), b = __shfl_sync(kFull, b_l, first);
        int32_t* out = packed + shfl64(off_l, first);
        const T* from = data - (int64_t)n * sh.pad;
#pragma unroll
        for (int gi = 0; gi < kFlatBundle; ++gi)
          bufA[gi] = load_octet<T, !ALIGNED>(from + (q0 + first + gi) * kGroup + lane * kOct, kOct, sh.align);
#define ACTNN_CASE(B)                                                                                              \
        case B:                                                                                                    \
          pack_flat_run<T, B, MODE, false, PREFETCH, ALIGNED>(bufA, bufB, k, k1, q0, from, mine, out, noise, key,  \
                                                              plan, lane, sh.align);                               \
          break;
        switch (b) {
          ACTNN_CASE(1) ACTNN_CASE(2) ACTNN_CASE(3) ACTNN_CASE(4) ACTNN_CASE(5) ACTNN_CASE(6) ACTNN_CASE(7)
          ACTNN_CASE(8)
          default: break;
        }
#undef ACTNN_CASE
        k = k1;
      } else {
        // all octets and their noise first, so that the loads travel together; then group by group over one copy of the code
        Oct<T> nz[kFlatBundle];
#pragma unroll
        for (int gi = 0; gi < kFlatBundle; ++gi) {
          const int n = __shfl_sync(kFull, g.n, first + gi), r = __shfl_sync(kFull, g.r, first + gi);
          bufA[gi] = load_octet<T, true>(data + (int64_t)n * sh.F + (int64_t)r * kGroup + lane * kOct,
                                         n < 0 ? 0 : elements_left(sh, r, lane), sh.align);
          if constexpr (MODE == kNoiseTensor)
            nz[gi] = n < 0 ? zero_oct<T>() : load_oct<T>(noise + (q0 + first + gi) * kGroup + lane * kOct);
          else nz[gi] = zero_oct<T>();
        }
        if constexpr (MODE == kNoisePhilox) noise_bundle<T>(key, q0 + first, lane, nz);
#pragma unroll 1
        for (int gi = 0; gi < kFlatBundle; ++gi) {
          const int b = __shfl_sync(kFull, b_l, first + gi);    // zero past the activation
          int32_t* out = packed + shfl64(off_l, first + gi);
          const QP<T> qp = fetch_lane_params<T>(mine, first + gi);
#define ACTNN_CASE(B) case B: pack_group<T, B>(bufA[0], nz[0], qp, out, plan, lane); break;
          switch (b) {
            ACTNN_CASE(1) ACTNN_CASE(2) ACTNN_CASE(3) ACTNN_CASE(4) ACTNN_CASE(5) ACTNN_CASE(6) ACTNN_CASE(7)
            ACTNN_CASE(8)
            default: break;
          }
#undef ACTNN_CASE
#pragma unroll
          for (int i = 0; i + 1 < kFlatBundle; ++i) {
            bufA[i] = bufA[i + 1];
            nz[i] = nz[i + 1];
          }
        }
        ++k;
      }
    }
  }
}

// ------------------------------------------------------------------ host side
RaggedShape ragged_shape(const void* data, int64_t N, int64_t F, int elem_size) {
  RaggedShape sh;
  sh.F = F;
  sh.G = (F + kGroup - 1) / kGroup;
  sh.Q = N * sh.G;
  sh.align = octet_alignment(data, F, elem_size);
  sh.pad = sh.G * kGroup - F;
  return sh;
}

template <typename T, typename ST>
int launch_pack(const void* data, const void* mn, const void* mx, const int32_t* bits, const int64_t* word_offsets,
                int32_t* packed, void* scale, void* mn_out, int64_t N, int64_t F, int stochastic, const void* noise,
                uint64_t seed, uint64_t offset, cudaStream_t s) {
  const RaggedShape sh = ragged_shape(data, N, F, sizeof(T));
  const NoiseKey key = make_noise_key(seed, offset);
  const int64_t bundles = (sh.Q + kFlatBundle - 1) / kFlatBundle;
#define ACTNN_LAUNCH(MODE, ALIGNED)                                                                                   \
  {                                                                                                                   \
    auto kernel = pack_ragged_kernel<T, ST, MODE, ALIGNED>;                                                           \
    kernel<<<persistent_grid(kernel, kThreads, bundles), kThreads, 0, s>>>(                                           \
        (const T*)data, (const T*)mn, (const T*)mx, bits, word_offsets, packed, (ST*)scale, (ST*)mn_out, sh,          \
        (const T*)noise, key);                                                                                        \
  }
#define ACTNN_MODE(MODE)                                \
  if (sh.align == kOct) ACTNN_LAUNCH(MODE, true)        \
  else ACTNN_LAUNCH(MODE, false)
  if (!stochastic) { ACTNN_MODE(kNoiseNone) }
  else if (noise) { ACTNN_MODE(kNoiseTensor) }
  else { ACTNN_MODE(kNoisePhilox) }
#undef ACTNN_MODE
#undef ACTNN_LAUNCH
  return check_launch();
}

}  // namespace

// Where the bundles inside a sample outweigh its last one or two, and every warp gets a few of them.  How many groups a
// sample that takes depends on how many widths the warps of a block meet, of which the host knows the average (`width`; 1:
// all the same): the columns keep all warps on one sample.  us of a compress, columns / this, float16 except where noted;
// the samples' scales spread as exp(0.7 randn):
//   2 bits   160 x 256 groups 20.3 / 19.7, 200 x 259 24.8 / 22.1, 400 x 300 39.3 / 39.5, 512 x 257 48.9 / 42.9, 1024 x 257 91.3 /
//            83.3, 50 x 919 22.3 / 20.1, 100 x 919 33.6 / 28.1, 16 x 7442 46.5 / 35.8; but 300 x 130 23.4 / 23.2, 1000 x 130 53.3 / 55.1
//   3 bits   200 x 259 25.4 / 23.9, 300 x 400 41.6 / 39.7, 400 x 440 54.5 / 53.3, 512 x 401 72.9 / 62.6; but 256 x 256 27.0 / 29.5,
//            400 x 300 40.8 / 43.3; float32 400 x 440 82.9 / 78.0, 400 x 300 59.2 / 59.2
//   4 bits   256 x 515 50.0 / 43.4, 512 x 401 72.3 / 69.4, 400 x 440 56.9 / 57.9, 2000 x 401 555 / 560 (spread as exp(0.3 randn) 55.7 /
//            53.2 and 551 / 508); but 200 x 300 26.6 / 29.1, 400 x 300 41.8 / 46.3; float32 400 x 440 85.4 / 81.1, 400 x 300 61.0 / 62.9
//   6 bits   64 x 641 23.4 / 21.5, 512 x 785 136 / 129; but 512 x 401 77.8 / 75.5, 400 x 440 60.2 / 67.4, 1024 x 513 180 / 188; float32
//            512 x 401 105.9 / 96.9, 400 x 440 89.5 / 85.0
//   all of 8 200 x 259 25.4 / 23.1, 512 x 785 135 / 113, 400 x 300 42.4 / 41.8
// (The unpack has no generator to save and stays with the columns: 13.3 against 17.5, 100 x 919.)
bool ragged_pays(int64_t N, int64_t F, int dtype, double width) {
  const int64_t G = (F + kGroup - 1) / kGroup;
  int64_t least = 256;
  if (width > 2 && (width > 3 || N > 200)) least = 384;
  if (width > 4 && dtype != ACTNN_F32) least = 640;
  return G >= least && N * G >= 40960 && N * G < ((int64_t)1 << 31);
}

int ragged_pack(const void* data, const void* mn, const void* mx, const int32_t* bits, const int64_t* word_offsets,
                int32_t* packed, void* scale, void* mn_out, int64_t N, int64_t F, int dtype, int stat_dtype,
                int stochastic, const void* noise, uint64_t seed, uint64_t offset, cudaStream_t s) {
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

}  // namespace actnn
