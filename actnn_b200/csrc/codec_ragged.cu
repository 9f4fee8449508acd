// Pack of [N, F] activations whose samples are not whole groups of 256, or not a multiple of four groups, in the
// order of the stream: samples of many groups.  (Samples of few groups: the column kernels, codec_column.cu.)
//
// The bundles are the aligned groups 4k .. 4k+3 of the flat [N * G] list, as in the kernels for whole groups, so that a
// call of the noise generator serves each (columns of an odd G need two), and a bundle inside a sample is
// addressed and packed as there: only the sample's offset differs.  What is special happens in one bundle or two a
// sample, those that hold its last, partial group or groups of two samples; they are taken group by group.  Every warp
// gets an equal share of consecutive bundles and prepares up to 32 groups at a time, a group a lane.
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

// The warp's share of the bundles, up to eight at a time.
struct BundleShare {
  int64_t next, left;
  ACTNN_DEV BundleShare(int64_t Q) {
    const int64_t warp = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * kThreads) >> 5;
    const int64_t total = (Q + kFlatBundle - 1) / kFlatBundle;
    const int64_t base = total / nwarps, rem = total - base * nwarps;
    next = warp * base + min(warp, rem);
    left = base + (warp < rem ? 1 : 0);
  }
  ACTNN_DEV int take(int64_t& q0) {
    const int n = (int)min(left, (int64_t)(kFlatGroups / kFlatBundle));
    q0 = next * kFlatBundle;
    next += n;
    left -= n;
    return n;
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
  BundleShare share(sh.Q);
  while (share.left > 0) {
    int64_t q0;
    const int bundles = share.take(q0);
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

// Where the bundles inside a sample outweigh its last one or two, and every warp gets a few of them.  us, columns against
// this, widths around 2 bits, whole octets: float16 100 x 919 groups 20.0 / 14.5, 50 x 919 11.1 / 9.2, 30 x 919 7.7 / 7.9, 200 x 259
// 13.0 / 10.0, 300 x 919 (octets on 4 elements) 61.9 / 43.2, 16 x 7442 24.3 / 16.7; 200 x 130 7.3 / 7.9, 1000 x 130 26.4 / 23.7
// but 28.5 / 35.5 around 4 bits, 4000 x 33 30.2 / 32.5; float32 100 x 919 24.9 / 21.7, 200 x 259 15.6 / 12.7, 30 x 919 9.2 / 8.9.
// (The unpack has no generator to save and stays with the columns: 13.3 against 17.5, 100 x 919.)
bool ragged_pays(int64_t N, int64_t F) {
  const int64_t G = (F + kGroup - 1) / kGroup;
  return G >= 256 && N * G >= 40960 && N * G < ((int64_t)1 << 31);
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
