// Mixed-precision stream: per-sample bit widths, int32 words.
//
// Layout (reference: quantization_cuda_kernel.cu:51-79).  For 256-element groups the
// reference formula "bit i of element d goes to word (d*b+i) % W, bit (d*b+i) / W,
// W = 8b" reads, with d = 8t + j:  word j*b + i, bit t.  Word w of a group is therefore
// the 32-lane ballot of bit w of each lane's "row" (its eight b-bit codes laid end to
// end), and a group's 8b words are the bit-matrix transpose of the 32 rows.
//
// A warp owns a bundle of four consecutive groups of one sample.  Each lane concatenates
// the rows of the four groups into a 32b-bit string S[0..b-1]; transposing word k of that
// string across the warp yields output words 32k .. 32k+31 of the bundle, lane w holding
// word 32k + w, so every store is one fully coalesced 128-byte line.  No shared memory,
// no atomics, no block-level synchronisation.
#include "flat_runs.cuh"

namespace actnn {
namespace {

constexpr int kThreads = 256;

struct BundleCoord {
  int64_t n, q0;                      // sample, first flat group
  int g0, count;                      // first group within the sample, groups in this bundle
};

// Walks the (sample, bundle-in-sample) pairs a warp owns without 64-bit divisions: the
// stride between a warp's tasks is split once into whole samples and a remainder.
struct BundleWalker {
  int64_t n, N, G;
  int r, bps, step_n, step_r, gpb;
  ACTNN_DEV BundleWalker(int64_t warp, int64_t nwarps, int64_t N_, int64_t G_, int gpb_ = kBundle)
      : N(N_), G(G_), gpb(gpb_) {
    bps = (int)((G_ + gpb - 1) / gpb);
    n = warp / bps;
    r = (int)(warp - n * bps);
    step_n = (int)(nwarps / bps);
    step_r = (int)(nwarps - (int64_t)step_n * bps);
  }
  ACTNN_DEV bool valid() const { return n < N; }
  ACTNN_DEV BundleCoord coord() const {
    BundleCoord c;
    c.n = n;
    c.g0 = r * gpb;
    c.count = (int)min((int64_t)gpb, G - c.g0);
    c.q0 = n * G + c.g0;
    return c;
  }
  ACTNN_DEV void next() {
    n += step_n;
    r += step_r;
    if (r >= bps) { r -= bps; ++n; }
  }
};

// Device counter of bundles whose width was outside 1..8 (nothing is written for them).
__device__ unsigned g_bad_width_bundles;

// ---------------------------------------------------------------------------- pack
// Groups per pack bundle: eight octets per lane for 16-bit types, four for float32.
template <typename T> struct PackShape { static constexpr int GPB = sizeof(T) == 2 ? 8 : 4; };

// PHILOX (whole bundles): the noise is known at compile time to come from the generator, so
// the body has no branch on `stochastic` / `noise` and the generator's dependent chain can be
// interleaved with the arithmetic of neighbouring groups.
template <typename T, typename ST, int B, bool FULL, bool PHILOX>
ACTNN_DEV void pack_bundle(const Oct<T> (&x)[PackShape<T>::GPB], const BundleCoord& c, const T* __restrict__ mn,
                           const T* __restrict__ mx, ST* __restrict__ scale, ST* __restrict__ mn_out,
                           int32_t* __restrict__ out, const T* __restrict__ noise, int stochastic,
                           NoiseGen<T>& gen, const TransposePlan& plan, int lane) {
  constexpr int GPB = PackShape<T>::GPB;
  constexpr int W = GPB * 8 * B / 32;                    // words per lane string = transposes
  const int count = FULL ? GPB : c.count;
  // lane g (< count) prepares group g, then ships (mn', scale) to everyone
  ParamWords mine = {0u, 0u};
  if (lane < count) {
    const float gmn = load_scalar<T>(mn, c.q0 + lane), gmx = load_scalar<T>(mx, c.q0 + lane);
    const GroupParams gp = prepare_group<T>(gmn, gmx, B);
    store_scalar<ST>(scale, c.q0 + lane, gp.scale);
    if (mn_out) store_scalar<ST>(mn_out, c.q0 + lane, gmn);
    mine = pack_params<T>(gp);
  }
  uint32_t S[W];
#pragma unroll
  for (int k = 0; k < W; ++k) S[k] = 0u;
  Oct<T> nzb[NoiseShape<T>::GPC];                     // one call's worth of noise octets
#pragma unroll
  for (int gi = 0; gi < GPB; ++gi) {
    const QP<T> qp = fetch_params<T>(mine, gi);
    if (FULL || gi < count) {
      Oct<T> nz;
      if constexpr (PHILOX) {
        if (gi % NoiseShape<T>::GPC == 0) noise_block<T>(gen.key, (uint64_t)(c.q0 + gi), lane, nzb);
        nz = nzb[gi % NoiseShape<T>::GPC];
      } else if (!stochastic) nz = zero_oct<T>();
      else if (noise) nz = load_oct<T>(noise + (c.q0 + gi) * kGroup + lane * kOct);
      else if (!FULL) nz = gen.get((uint64_t)(c.q0 + gi));
      else {                                          // FULL: q0 is a multiple of the groups per call
        if (gi % NoiseShape<T>::GPC == 0) noise_block<T>(gen.key, (uint64_t)(c.q0 + gi), lane, nzb);
        nz = nzb[gi % NoiseShape<T>::GPC];
      }
      uint32_t lo, hi;
      row_from_magic<T, B>(quantize_oct<T, true, B>(x[gi], nz, qp), lo, hi);
      if (gi == 0) put_row<B, 0 * 8 * B>(S, lo, hi);
      if (gi == 1) put_row<B, 1 * 8 * B>(S, lo, hi);
      if (gi == 2) put_row<B, 2 * 8 * B>(S, lo, hi);
      if (gi == 3) put_row<B, 3 * 8 * B>(S, lo, hi);
      if constexpr (GPB > 4) {
        if (gi == 4) put_row<B, 4 * 8 * B>(S, lo, hi);
        if (gi == 5) put_row<B, 5 * 8 * B>(S, lo, hi);
        if (gi == 6) put_row<B, 6 * 8 * B>(S, lo, hi);
        if (gi == 7) put_row<B, 7 * 8 * B>(S, lo, hi);
      }
    }
  }
  const int words = count * 8 * B;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const uint32_t y = warp_transpose32(S[k], plan);
    const int o = k * 32 + lane;
    if (FULL || o < words) out[o] = (int32_t)y;
  }
}

template <typename T, typename ST, bool FULL, bool PHILOX = false>
__global__ void __launch_bounds__(kThreads, (MagicInfo<T>::paired && !PHILOX) ? 3 : 2)
pack_mixed_kernel(const T* __restrict__ data, const T* __restrict__ mn, const T* __restrict__ mx,
                  const int32_t* __restrict__ bits, const int64_t* __restrict__ word_offsets,
                  int32_t* __restrict__ packed, ST* __restrict__ scale, ST* __restrict__ mn_out,
                  int64_t N, int64_t G, const T* __restrict__ noise, int stochastic, const NoiseKey key) {
  constexpr int GPB = PackShape<T>::GPB;
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * kThreads) >> 5;
  const TransposePlan plan = make_transpose_plan(lane);
  NoiseGen<T> gen(key, lane);

  for (BundleWalker walk(warp, nwarps, N, G, GPB); walk.valid(); walk.next()) {
    const BundleCoord c = walk.coord();
    Oct<T> x[GPB];
#pragma unroll
    for (int gi = 0; gi < GPB; ++gi)
      x[gi] = (FULL || gi < c.count) ? load_oct<T>(data + (c.q0 + gi) * kGroup + lane * kOct) : zero_oct<T>();
    const int b = __ldg(bits + c.n);
    int32_t* out = packed + (__ldg(word_offsets + c.n) + (int64_t)c.g0 * 8 * b);
#define ACTNN_CASE(B)                                                                                     \
    case B:                                                                                               \
      pack_bundle<T, ST, B, FULL, PHILOX>(x, c, mn, mx, scale, mn_out, out, noise, stochastic, gen, plan, lane); \
      break;
    switch (b) {
      ACTNN_CASE(1) ACTNN_CASE(2) ACTNN_CASE(3) ACTNN_CASE(4) ACTNN_CASE(5) ACTNN_CASE(6) ACTNN_CASE(7)
      ACTNN_CASE(8)
      default:            // widths outside 1..8: nothing is written, the bundle is counted
        if (lane == 0) atomicAdd(&g_bad_width_bundles, 1u);
        break;
    }
#undef ACTNN_CASE
  }
}

// ---------------------------------------------------------------------------- pack, flat tasks
// Fast path for G % 4 == 0 and G >= 32 (every layer of the usual networks).  A warp task is
// 32 consecutive groups of the flattened [N * G] list:
//   * lane l prepares group q0 + l: its sample, width and stream position, one coalesced load
//     of min / max, ONE division, coalesced stores of scale / min.  All 32 lanes work, so the
//     per-group cost is a quarter of what a four-group bundle with four active lanes pays;
//   * the task is then worked off as eight bundles of four groups (one generator call per
//     lane, `B` transposes, `B` coalesced 128-byte stores).  A bundle never straddles two
//     samples because G % 4 == 0, so its width is warp-uniform;
//   * the octets of the next bundle (also across the task boundary) are requested before the
//     current one is quantized: a warp always has loads in flight.
#ifndef ACTNN_FLAT_BLOCKS
#define ACTNN_FLAT_BLOCKS 2
#endif
#ifndef ACTNN_FLAT_UNPACK_BLOCKS
#define ACTNN_FLAT_UNPACK_BLOCKS 3   // 85 registers, nothing spilled: measured 3-4 % faster than 4 blocks (64 registers, spills)
#endif
constexpr int kFlatUnpackBlocks = ACTNN_FLAT_UNPACK_BLOCKS;
constexpr int kFlatBlocks16 = ACTNN_FLAT_BLOCKS;   // resident blocks per SM the flat kernels are compiled for (16-bit types)

template <typename T, typename ST, int MODE, bool CLAMP_LOW>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 2 ? kFlatBlocks16 : 2)
pack_mixed_flat_kernel(const T* __restrict__ data, const T* __restrict__ mn, const T* __restrict__ mx,
                       const int32_t* __restrict__ bits, const int64_t* __restrict__ word_offsets,
                       int32_t* __restrict__ packed, ST* __restrict__ scale, ST* __restrict__ mn_out,
                       int64_t Q, int64_t G, const T* __restrict__ noise, const NoiseKey key) {
  constexpr bool PREFETCH = sizeof(T) == 2;
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * kThreads) >> 5;
  const TransposePlan plan = make_transpose_plan(lane);
  const int64_t tasks = (Q + kFlatGroups - 1) / kFlatGroups;
  if (warp >= tasks) return;

  // (sample, group) of the task's first group, advanced without divisions inside the loop
  int64_t q0 = warp * kFlatGroups;
  int64_t n0 = q0 / G;
  int64_t r0 = q0 - n0 * G;
  const int64_t stride = nwarps * kFlatGroups;
  const int64_t step_n = stride / G, step_r = stride - step_n * G;

  Oct<T> bufA[kFlatBundle], bufB[kFlatBundle];                  // bufB stays unused without PREFETCH
  for (; q0 < Q; q0 += stride) {
    // the octets of the task's first bundle are requested before anything else, so that they
    // travel while the lanes prepare their groups
#pragma unroll
    for (int gi = 0; gi < kFlatBundle; ++gi) bufA[gi] = load_oct<T>(data + (q0 + gi) * kGroup + lane * kOct);
    // ---- this lane's group
    const int64_t q = q0 + lane;
    int64_t n = n0, r = r0 + lane;
    if (r >= G) { r -= G; ++n; }                              // G >= 32: at most one wrap
    int b_l = -1;                                             // past the end of the activation
    int64_t off_l = 0;
    LaneParams<T> mine = {0u, 0u};
    if (q < Q) {
      b_l = __ldg(bits + n);
      if (b_l < 1 || b_l > 8) b_l = 0;                        // not a width: counted, nothing written
      off_l = __ldg(word_offsets + n) + r * (8 * b_l);
      const float gmn = load_scalar<T>(mn, q), gmx = load_scalar<T>(mx, q);
      const GroupParams gp = prepare_group<T>(gmn, gmx, b_l);
      store_scalar<ST>(scale, q, gp.scale);
      if (mn_out) store_scalar<ST>(mn_out, q, gmn);
      mine = lane_params<T>(gp);
    }
    // ---- runs of bundles of one width (the lanes past the end close the last run)
    int k = 0;
    while (k < kFlatGroups / kFlatBundle) {
      const int first = k * kFlatBundle;
      const int b = __shfl_sync(kFull, b_l, first);
      if (b < 0) break;
      const unsigned same = __ballot_sync(kFull, b_l == b) >> first;          // bit i: lane first + i
      const int run_lanes = same == 0xffffffffu >> first ? 32 - first : __ffs((int)~same) - 1;
      const int k1 = k + run_lanes / kFlatBundle;
      const uint32_t olo = __shfl_sync(kFull, (uint32_t)off_l, first);
      const uint32_t ohi = __shfl_sync(kFull, (uint32_t)((uint64_t)off_l >> 32), first);
      int32_t* out = packed + (int64_t)(((uint64_t)ohi << 32) | olo);
      if (k > 0) {
#pragma unroll
        for (int gi = 0; gi < kFlatBundle; ++gi)
          bufA[gi] = load_oct<T>(data + (q0 + first + gi) * kGroup + lane * kOct);
      }
#define ACTNN_CASE(B)                                                                                          \
      case B:                                                                                                  \
        pack_flat_run<T, B, MODE, CLAMP_LOW, PREFETCH>(bufA, bufB, k, k1, q0, data, mine, out, noise, key, plan, lane); \
        break;
      switch (b) {
        ACTNN_CASE(1) ACTNN_CASE(2) ACTNN_CASE(3) ACTNN_CASE(4) ACTNN_CASE(5) ACTNN_CASE(6) ACTNN_CASE(7)
        ACTNN_CASE(8)
        default:
          if (lane == 0) atomicAdd(&g_bad_width_bundles, (unsigned)(k1 - k));
          break;
      }
#undef ACTNN_CASE
      k = k1;
    }
    n0 += step_n;
    r0 += step_r;
    if (r0 >= G) { r0 -= G; ++n0; }
  }
}

// ---------------------------------------------------------------------------- unpack
// Decoding a group needs only 2^B distinct outputs, code / scale + min for code = 0..2^B-1.
// Lanes compute those once (one IEEE division per lane for up to four groups at a time)
// and the elements look theirs up: for 16-bit types up to 3 bits by byte permutes (mixed_bundle.cuh); otherwise a warp
// shuffle fetches the entry; from 6 bits on the division is done per element.
// Unpack of whole groups whose count per sample is no multiple of four, or below 32: a warp task is a bundle of four
// groups (the last one of a sample may be shorter), in the order of the stream, so that the bundles of a wide sample
// are spread over the warps.  The column kernel, which writes the same values, leaves them to one block, and samples
// of 8 and of 1 bits (what equal sensitivities give, as before the first gradient) make that block the last:
// 512 x 130 groups of float32 16.7 us against 36.1; with widths near the average of 2 bits 14.2 against 13.9, 256 x 130
// 8.7 against 9.4; all at 8 bits, 16 x 7442, 65.2 against 89.5; float16 7.1 against 7.6 and 26.3 against 27.9.
// Narrow widths of 16-bit types bring their words in the order of the nibble decode in a branch of their own: its arithmetic
// before every load had all widths pay.  float16 512 x 781 groups at 2 / 4 / 8 bits, words in the order of the stream 47.5 /
// 64.9 / 84.2 us, in the nibbles' without the branch 48.5 / 68.8 / 94.2, with it 44.7 / 64.6 / 85.5; 300 x 130 groups 6.5 / 8.4 /
// 10.0, 6.9 / 9.1 / 10.5, 6.5 / 8.5 / 10.2.
template <typename T, typename ST>
__global__ void __launch_bounds__(kThreads, 4)
unpack_mixed_kernel(const int32_t* __restrict__ packed, const int32_t* __restrict__ bits,
                    const int64_t* __restrict__ word_offsets, const ST* __restrict__ scale,
                    const ST* __restrict__ mn, T* __restrict__ out, int64_t N, int64_t G) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * kThreads) >> 5;
  const TransposePlan plan = make_transpose_plan(lane);

  // A bundle's input is only b * 128 bytes per warp: issue the loads of DEPTH bundles before
  // decoding the first, so that enough bytes are in flight to cover the memory latency.
  constexpr int DEPTH = 2;
  BundleWalker walk(warp, nwarps, N, G);
  while (walk.valid()) {
    BundleCoord t_c[DEPTH];
    int t_b[DEPTH];
    bool t_ok[DEPTH];
    uint32_t t_w[DEPTH][8];
    float t_sc[DEPTH], t_m[DEPTH];
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) {
      t_ok[d] = walk.valid();
      t_b[d] = 0;                                         // not a width: nothing was written
      t_sc[d] = 1.f;
      t_m[d] = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) t_w[d][k] = 0u;
      if (t_ok[d]) {
        t_c[d] = walk.coord();
        const BundleCoord& c = t_c[d];
        const int b = __ldg(bits + c.n);
        if (b >= 1 && b <= 8) t_b[d] = b;
        const int32_t* in = packed + (__ldg(word_offsets + c.n) + (int64_t)c.g0 * 8 * t_b[d]);
        const int words = c.count * 8 * t_b[d];
        if (kNibbles<T, 3> && t_b[d] <= 3) {                  // warp-uniform
          const WordOrder<T> order(lane);
          const int base = order.base(t_b[d]), step = order.step(t_b[d]);
#pragma unroll
          for (int k = 0; k < 3; ++k)
            if (k < t_b[d] && base + k * step < words) t_w[d][k] = (uint32_t)__ldg(in + base + k * step);
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k * 32 + lane < words) t_w[d][k] = (uint32_t)__ldg(in + k * 32 + lane);
        }
        if (lane < c.count) {
          t_sc[d] = load_scalar<ST>(scale, c.q0 + lane);
          t_m[d] = load_scalar<ST>(mn, c.q0 + lane);
        }
        walk.next();
      }
    }
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) {
      if (!t_ok[d]) break;                                // warp-uniform
      const int count = t_c[d].count;
      T* dst = out + t_c[d].q0 * kGroup + lane * kOct;
      auto store = [&](int gi, const Oct<T>& x) { if (gi < count) store_oct_streaming<T>(dst + gi * kGroup, x); };
#define ACTNN_CASE(B)                                                                \
      case B: {                                                                      \
        uint32_t w[B];                                                               \
        _Pragma("unroll") for (int k = 0; k < B; ++k) w[k] = t_w[d][k];              \
        decode_bundle<T, B>(w, t_sc[d], t_m[d], plan, lane, store);                  \
        break;                                                                       \
      }
      switch (t_b[d]) {
        ACTNN_CASE(1) ACTNN_CASE(2) ACTNN_CASE(3) ACTNN_CASE(4) ACTNN_CASE(5) ACTNN_CASE(6) ACTNN_CASE(7)
        ACTNN_CASE(8)
        default: break;
      }
#undef ACTNN_CASE
    }
  }
}

// How the flat unpack kernel deals out its tasks (32 consecutive groups each).  Block b owns tasks
// b, b + gridDim.x, b + 2 gridDim.x, ... -- a sample is 20 to 30 consecutive tasks, so every block
// meets every width in the proportion of the whole activation -- and its warps claim them one at
// a time from a counter in shared memory: a warp that met wider (slower) samples simply takes
// fewer tasks.  The last `split` tasks of a block are claimed as halves of 16 groups, which
// shortens the ragged end of the launch (an activation is only a few tasks per resident warp).
// Nothing is shared between blocks or launches.
#ifndef ACTNN_UNPACK_SPLIT
#define ACTNN_UNPACK_SPLIT 8
#endif
struct FlatClaim { int64_t task; int kb, ke; };            // bundles kb .. ke-1 of the task
struct FlatPool {
  unsigned* counters;                                      // [0] whole tasks claimed, [1] halves claimed
  unsigned whole, halves;
  bool in_halves;
  ACTNN_DEV void init(unsigned* smem2, int64_t tasks, int split_tasks) {
    counters = smem2;
    const int64_t mine = tasks > blockIdx.x ? (tasks - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    const int64_t split = mine < split_tasks ? mine : split_tasks;
    whole = (unsigned)(mine - split);
    halves = (unsigned)(2 * split);
    in_halves = false;
    if (threadIdx.x < 2) counters[threadIdx.x] = 0u;
    __syncthreads();
  }
  ACTNN_DEV int64_t task_of(unsigned i) const { return blockIdx.x + (int64_t)i * gridDim.x; }
  ACTNN_DEV bool claim(int lane, FlatClaim& c) {
    unsigned i = 0u;
    if (!in_halves) {
      if (lane == 0) i = atomicAdd(&counters[0], 1u);
      i = __shfl_sync(kFull, i, 0);
      if (i < whole) { c.task = task_of(i); c.kb = 0; c.ke = kFlatGroups / kFlatBundle; return true; }
      in_halves = true;
    }
    if (lane == 0) i = atomicAdd(&counters[1], 1u);
    i = __shfl_sync(kFull, i, 0);
    if (i >= halves) return false;
    constexpr int kHalfBundles = kFlatGroups / kFlatBundle / 2;
    c.task = task_of(whole + (i >> 1));
    c.kb = (int)(i & 1u) * kHalfBundles;
    c.ke = c.kb + kHalfBundles;
    return true;
  }
};
// ---------------------------------------------------------------------------- unpack, flat tasks
// Same task shape as the flat pack: lane l owns group q0 + l of a task of 32 groups (its
// sample, width, stream position, scale and min come from coalesced loads), and eight bundles
// of four groups are decoded with the words of the next bundle already requested.  For 16-bit
// outputs of up to 3 bits the lane also computes the 2^B decoded values of its own group once
// per task (their low and high bytes in two registers, four at 3 bits); a bundle then fetches them with a shuffle each.
#ifndef ACTNN_UNPACK_DIRECT_FROM
#define ACTNN_UNPACK_DIRECT_FROM 6
#endif
template <typename T, int B, bool FASTDIV>
ACTNN_DEV void unpack_flat_bundle(const uint32_t (&words)[B], float sc_l, float m_l, int first,
                                  int64_t q, T* __restrict__ out, const TransposePlan& plan, int lane) {
  // from kDirect bits on every element is computed (a table of 2^B entries no longer fits a warp,
  // or costs more shuffles than the arithmetic)
  constexpr int kDirect = FASTDIV ? ACTNN_UNPACK_DIRECT_FROM : 6;
  constexpr int E = 1 << (B < kDirect ? B : 5);        // table entries per group
  constexpr int GPC = (32 / E) < kFlatBundle ? (32 / E) : kFlatBundle;   // groups served by one table
  uint32_t S[B];
#pragma unroll
  for (int k = 0; k < B; ++k) S[k] = warp_transpose32(words[k], plan);
  uint32_t entry = 0u;
#pragma unroll
  for (int gi = 0; gi < kFlatBundle; ++gi) {
    if constexpr (B < kDirect) {
      if (gi % GPC == 0) {                               // (re)build the table for groups gi .. gi+GPC-1
        const int g = first + ((gi + lane / E) & (kFlatBundle - 1));
        const float sc = __shfl_sync(kFull, sc_l, g), m = __shfl_sync(kFull, m_l, g);
        entry = dequant_bits<T>((float)(lane % E), sc, m);
      }
    }
    uint32_t lo = 0u, hi = 0u;                           // this group's row
    if (gi == 0) { lo = get_bits<0 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<0 * 8 * B + 32, 8 * B - 32>(S); }
    if (gi == 1) { lo = get_bits<1 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<1 * 8 * B + 32, 8 * B - 32>(S); }
    if (gi == 2) { lo = get_bits<2 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<2 * 8 * B + 32, 8 * B - 32>(S); }
    if (gi == 3) { lo = get_bits<3 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<3 * 8 * B + 32, 8 * B - 32>(S); }
    Oct<T> o;
    uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
    uint32_t v[8];
    const uint32_t S2[2] = {lo, hi};
    uint32_t code[8];
    get_codes<B, 0>(S2, code);
    if constexpr (B < kDirect) {
      const int base = (gi % GPC) * E;
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __shfl_sync(kFull, entry, base + (int)code[j]);
    } else {
      const float sc = __shfl_sync(kFull, sc_l, first + gi), m = __shfl_sync(kFull, m_l, first + gi);
      float y = 0.f;
      if (FASTDIV && group_reciprocal(sc, y)) {                 // warp-uniform: one scale per group
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = dequant_bits_recip<T>((float)code[j], sc, y, m);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = dequant_bits<T>((float)code[j], sc, m);
      }
    }
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int j = 0; j < 8; ++j) ow[j] = v[j];
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) ow[k] = v[2 * k] | (v[2 * k + 1] << 16);
    }
    store_oct_streaming<T>(out + (q + gi) * kGroup + lane * kOct, o);
  }
}

// The bytes of the values of codes 0..7 (2^b are used) of one group.
template <typename T> ACTNN_DEV ByteTable byte_table(int b, float sc, float m) {
  float y = 0.f;
  const bool fast = group_reciprocal(sc, y);
  auto pair = [&](int c) {
    const uint32_t v0 = fast ? dequant_bits_recip<T>((float)c, sc, y, m) : dequant_bits<T>((float)c, sc, m);
    const uint32_t v1 = fast ? dequant_bits_recip<T>((float)(c + 1), sc, y, m) : dequant_bits<T>((float)(c + 1), sc, m);
    return v0 | (v1 << 16);
  };
  ByteTable t = {0u, 0u, 0u, 0u};
  const uint32_t p01 = pair(0), p23 = pair(2);
  t.lo0 = select_bytes(p01, p23, 0x6420u);
  t.hi0 = select_bytes(p01, p23, 0x7531u);
  if (b == 3) {
    const uint32_t p45 = pair(4), p67 = pair(6);
    t.lo1 = select_bytes(p45, p67, 0x6420u);
    t.hi1 = select_bytes(p45, p67, 0x7531u);
  }
  return t;
}

// A run of bundles k0 .. k1-1 of one width B (see pack_flat_run), `in` its first word; a bundle is 32 * B words.
// Widths whose codes the transpose leaves in nibbles: two bundles at a time are decoded as straight-line code
// (four, at 1 and 2 bits: 37.5 against 37.1 us, 512 x 784 groups of bfloat16; four at 3 bits, too: 43.1; four blocks an
// SM instead of three: 41.0).
// The words of the next ones are requested before, the transposes of a pass are issued together, and only the
// stores are predicated, so the scheduler always has independent work.  A run of an odd number of bundles transposes
// a few zero words.
template <typename T, int B>
ACTNN_DEV void unpack_flat_nibbles(int k0, int k1, int64_t q0, const int32_t* __restrict__ in,
                                   const WordOrder<T>& order, const ByteTable& mine, T* __restrict__ out,
                                   const TransposePlan& plan) {
  constexpr int PER = 2, kBundles = kFlatGroups / kFlatBundle;
  const int lane = order.lane, step = order.step(B);
  in += order.base(B);
  uint32_t S[PER][B], next[PER][B];
  auto load = [&](uint32_t (&w)[PER][B], int k) {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
#pragma unroll
      for (int kk = 0; kk < B; ++kk) w[i][kk] = k + i < k1 ? (uint32_t)__ldg(in + (k - k0 + i) * (32 * B) + kk * step) : 0u;
    }
  };
  load(S, k0);
  // kept rolled: the straight-line body of one pass is long, and the instruction cache is shared by all widths
#pragma unroll 1
  for (int kb = k0; kb < k1; kb += PER) {
    load(next, kb + PER);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
#pragma unroll
      for (int kk = 0; kk < B; ++kk) S[i][kk] = warp_transpose32(S[i][kk], plan);
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const bool live = kb + i < k1;
      const int first = (kb + i < kBundles ? kb + i : kBundles - 1) * kFlatBundle;      // a lane of this warp in any case
#pragma unroll
      for (int gi = 0; gi < kFlatBundle; ++gi) {
        ByteTable t;
        t.lo0 = t.lo1 = __shfl_sync(kFull, mine.lo0, first + gi);
        t.hi0 = t.hi1 = __shfl_sync(kFull, mine.hi0, first + gi);
        if constexpr (B == 3) {
          t.lo1 = __shfl_sync(kFull, mine.lo1, first + gi);
          t.hi1 = __shfl_sync(kFull, mine.hi1, first + gi);
        }
        const Oct<T> o = decode_nibbles<T>(group_nibbles<B>(S[i], gi), t);
        if (live) store_oct_streaming<T>(out + (q0 + (kb + i) * kFlatBundle + gi) * kGroup + lane * kOct, o);
      }
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
#pragma unroll
      for (int kk = 0; kk < B; ++kk) S[i][kk] = next[i][kk];
    }
  }
}

// Other widths and float32: the B words per lane of bundle k+1 are requested before bundle k is decoded.
template <typename T, int B, bool FASTDIV>
ACTNN_DEV void unpack_flat_run(int k0, int k1, int64_t q0, const int32_t* __restrict__ in, float sc_l, float m_l,
                               T* __restrict__ out, const TransposePlan& plan, int lane) {
  auto load = [&](uint32_t (&w)[B], const int32_t* p) {
#pragma unroll
    for (int kk = 0; kk < B; ++kk) w[kk] = (uint32_t)__ldg(p + kk * 32);
  };
  in += lane;
  uint32_t wa[B], wb[B];
  load(wa, in);
  for (int k = k0; k < k1; k += 2) {
    if (k + 1 < k1) load(wb, in + 32 * B);
    unpack_flat_bundle<T, B, FASTDIV>(wa, sc_l, m_l, k * kFlatBundle, q0 + k * kFlatBundle, out, plan, lane);
    if (k + 1 >= k1) break;
    if (k + 2 < k1) load(wa, in + 64 * B);
    unpack_flat_bundle<T, B, FASTDIV>(wb, sc_l, m_l, (k + 1) * kFlatBundle, q0 + (k + 1) * kFlatBundle, out, plan, lane);
    in += 64 * B;
  }
}

template <typename T, typename ST>
__global__ void __launch_bounds__(kThreads, kFlatUnpackBlocks)
unpack_mixed_flat_kernel(const int32_t* __restrict__ packed, const int32_t* __restrict__ bits,
                         const int64_t* __restrict__ word_offsets, const ST* __restrict__ scale,
                         const ST* __restrict__ mn, T* __restrict__ out, int64_t Q, int64_t G) {
  const int lane = threadIdx.x & 31;
  const TransposePlan plan = make_transpose_plan(lane);
  const WordOrder<T> order(lane);
  __shared__ unsigned pool_counters[2];
  FlatPool pool;
  pool.init(pool_counters, (Q + kFlatGroups - 1) / kFlatGroups, ACTNN_UNPACK_SPLIT);

  FlatClaim claim;
  while (pool.claim(lane, claim)) {
    const int64_t q0 = claim.task * kFlatGroups;
    const int64_t q = q0 + lane;
    int b_l = -1;                                             // past the end of the activation
    int64_t off_l = 0;
    float sc_l = 1.f, m_l = 0.f;
    ByteTable mine = {0u, 0u, 0u, 0u};
    if (q < Q) {
      int64_t n, r;
      split_group_index(q, G, n, r);
      b_l = __ldg(bits + n);
      if (b_l < 1 || b_l > 8) b_l = 0;                        // not a width: the pack kernel wrote nothing either
      off_l = __ldg(word_offsets + n) + r * (8 * b_l);
      sc_l = load_scalar<ST>(scale, q);
      m_l = load_scalar<ST>(mn, q);
      if (sizeof(T) == 2 && b_l >= 1 && b_l <= 3) mine = byte_table<T>(b_l, sc_l, m_l);
    }
    int k = claim.kb;
    while (k < claim.ke) {
      const int first = k * kFlatBundle;
      const int b = __shfl_sync(kFull, b_l, first);
      if (b < 0) break;
      const unsigned same = __ballot_sync(kFull, b_l == b) >> first;          // bit i: lane first + i
      const int run_lanes = same == 0xffffffffu >> first ? 32 - first : __ffs((int)~same) - 1;
      const int k1 = min(k + run_lanes / kFlatBundle, claim.ke);
      const uint32_t olo = __shfl_sync(kFull, (uint32_t)off_l, first);
      const uint32_t ohi = __shfl_sync(kFull, (uint32_t)((uint64_t)off_l >> 32), first);
      const int32_t* in = packed + (int64_t)(((uint64_t)ohi << 32) | olo);
#define ACTNN_CASE(B)                                                                                             \
      case B:                                                                                                     \
        if constexpr (kNibbles<T, B>) unpack_flat_nibbles<T, B>(k, k1, q0, in, order, mine, out, plan);           \
        else unpack_flat_run<T, B, sizeof(ST) == 2>(k, k1, q0, in, sc_l, m_l, out, plan, lane);                   \
        break;
      switch (b) {
        ACTNN_CASE(1) ACTNN_CASE(2) ACTNN_CASE(3) ACTNN_CASE(4) ACTNN_CASE(5) ACTNN_CASE(6) ACTNN_CASE(7)
        ACTNN_CASE(8)
        default: break;
      }
#undef ACTNN_CASE
      k = k1;
    }
  }
}

// ---------------------------------------------------------------------------- prefix
// word_offsets[n] = (G * gs / 32) * sum_{m < n} bits[m]; one block, chunked scan.
__global__ void __launch_bounds__(1024)
bits_prefix_kernel(const int32_t* __restrict__ bits, int64_t N, int64_t words_per_bit,
                   int64_t* __restrict__ word_offsets) {
  __shared__ int64_t warp_sums[32];
  __shared__ int64_t carry;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t start = 0; start < N; start += 1024) {
    const int64_t i = start + threadIdx.x;
    const int64_t v = i < N ? (int64_t)bits[i] : 0;
    int64_t incl = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const int64_t t = __shfl_up_sync(kFull, incl, s);
      if (lane >= s) incl += t;
    }
    if (lane == 31) warp_sums[wid] = incl;
    __syncthreads();
    if (wid == 0) {
      int64_t ws = warp_sums[lane], wincl = ws;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const int64_t t = __shfl_up_sync(kFull, wincl, s);
        if (lane >= s) wincl += t;
      }
      warp_sums[lane] = wincl - ws;          // exclusive over warps
    }
    __syncthreads();
    const int64_t excl = carry + warp_sums[wid] + incl - v;
    if (i < N) word_offsets[i] = excl * words_per_bit;
    __syncthreads();
    if (threadIdx.x == 1023) carry = excl + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) word_offsets[N] = carry * words_per_bit;
}

template <typename T, typename ST, int MODE, bool CLAMP_LOW>
void launch_pack_flat(const void* data, const void* mn, const void* mx, const int32_t* bits,
                      const int64_t* word_offsets, int32_t* packed, void* scale, void* mn_out, int64_t N,
                      int64_t G, const void* noise, const NoiseKey& key, cudaStream_t stream) {
  auto kernel = pack_mixed_flat_kernel<T, ST, MODE, CLAMP_LOW>;
  const int64_t tasks = (N * G + kFlatGroups - 1) / kFlatGroups;
  kernel<<<persistent_grid(kernel, kThreads, tasks), kThreads, 0, stream>>>(
      (const T*)data, (const T*)mn, (const T*)mx, bits, word_offsets, packed, (ST*)scale, (ST*)mn_out, N * G, G,
      (const T*)noise, key);
}

template <typename T, typename ST>
int launch_pack(const void* data, const void* mn, const void* mx, const int32_t* bits,
                const int64_t* word_offsets, int32_t* packed, void* scale, void* mn_out, int64_t N,
                int64_t G, int stochastic, const void* noise, uint64_t seed, uint64_t offset,
                bool min_is_exact, cudaStream_t stream) {
  constexpr int GPB = PackShape<T>::GPB;
  const int64_t tasks = N * ((G + GPB - 1) / GPB);
  const NoiseKey key = make_noise_key(seed, offset);
  if (G % kFlatBundle == 0 && G >= kFlatGroups) {
#define ACTNN_FLAT(MODE)                                                                                     \
    if (min_is_exact)                                                                                        \
      launch_pack_flat<T, ST, MODE, false>(data, mn, mx, bits, word_offsets, packed, scale, mn_out, N, G, noise, \
                                           key, stream);                                                     \
    else                                                                                                     \
      launch_pack_flat<T, ST, MODE, true>(data, mn, mx, bits, word_offsets, packed, scale, mn_out, N, G, noise, \
                                          key, stream);
    if (!stochastic) { ACTNN_FLAT(kNoiseNone) }
    else if (noise) { ACTNN_FLAT(kNoiseTensor) }
    else { ACTNN_FLAT(kNoisePhilox) }
#undef ACTNN_FLAT
    return check_launch();
  }
  if (G % GPB == 0 && stochastic && !noise)
    pack_mixed_kernel<T, ST, true, true><<<persistent_grid(pack_mixed_kernel<T, ST, true, true>, kThreads, tasks),
                                           kThreads, 0, stream>>>(
        (const T*)data, (const T*)mn, (const T*)mx, bits, word_offsets, packed, (ST*)scale, (ST*)mn_out, N, G,
        (const T*)noise, stochastic, key);
  else if (G % GPB == 0)
    pack_mixed_kernel<T, ST, true><<<persistent_grid(pack_mixed_kernel<T, ST, true>, kThreads, tasks), kThreads, 0,
                                     stream>>>(
        (const T*)data, (const T*)mn, (const T*)mx, bits, word_offsets, packed, (ST*)scale, (ST*)mn_out, N, G,
        (const T*)noise, stochastic, key);
  else
    pack_mixed_kernel<T, ST, false><<<persistent_grid(pack_mixed_kernel<T, ST, false>, kThreads, tasks), kThreads, 0,
                                      stream>>>(
        (const T*)data, (const T*)mn, (const T*)mx, bits, word_offsets, packed, (ST*)scale, (ST*)mn_out, N, G,
        (const T*)noise, stochastic, key);
  return check_launch();
}

template <typename T, typename ST>
int launch_unpack(const int32_t* packed, const int32_t* bits, const int64_t* word_offsets,
                  const void* scale, const void* mn, void* out, int64_t N, int64_t G, cudaStream_t stream) {
  if (G % kFlatBundle == 0 && G >= kFlatGroups) {
    auto kernel = unpack_mixed_flat_kernel<T, ST>;
    const int64_t flat_tasks = (N * G + kFlatGroups - 1) / kFlatGroups;
    // sized by half tasks: a small activation spreads over twice the warps (see FlatPool)
    kernel<<<persistent_grid(kernel, kThreads, 2 * flat_tasks), kThreads, 0, stream>>>(
        packed, bits, word_offsets, (const ST*)scale, (const ST*)mn, (T*)out, N * G, G);
    return check_launch();
  }
  const int64_t tasks = N * ((G + kBundle - 1) / kBundle);
  auto kernel = unpack_mixed_kernel<T, ST>;
  kernel<<<persistent_grid(kernel, kThreads, tasks), kThreads, 0, stream>>>(
      packed, bits, word_offsets, (const ST*)scale, (const ST*)mn, (T*)out, N, G);
  return check_launch();
}

int check_common(int64_t N, int64_t G, int64_t group_size, int dtype, int stat_dtype) {
  if (N < 0 || G < 0) return ACTNN_ERR_SHAPE;
  if (group_size != kGroup && !generic_group_ok(group_size)) return ACTNN_ERR_SHAPE;
  if (dtype < ACTNN_F32 || dtype > ACTNN_BF16) return ACTNN_ERR_DTYPE;
  if (!(stat_dtype == dtype || (dtype == ACTNN_F32 && stat_dtype == ACTNN_BF16))) return ACTNN_ERR_DTYPE;
  if (N > (int64_t)1 << 40 || G > (int64_t)1 << 40 || (G && N > ((int64_t)1 << 52) / G)) return ACTNN_ERR_SHAPE;
  return ACTNN_OK;
}

}  // namespace
}  // namespace actnn

using namespace actnn;

extern "C" int actnn_bits_prefix(const int32_t* bits, int64_t N, int64_t G, int64_t group_size,
                                 int64_t* word_offsets, actnn_stream_t stream) {
  if (!word_offsets || (N > 0 && !bits)) return ACTNN_ERR_NULL;
  if (N < 0 || G < 0 || group_size <= 0 || group_size % 32 != 0 || N > (1 << 20)) return ACTNN_ERR_SHAPE;
  bits_prefix_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(bits, N, G * group_size / 32, word_offsets);
  return check_launch();
}

namespace actnn {
// `min_is_exact`: every `mn[q]` is the true minimum of its group (then the rounding itself maps
// the smallest values to code 0 and the lower clamp is dropped).
int pack_mixed_impl(const void* data, const void* mn, const void* mx, const int32_t* bits,
                    const int64_t* word_offsets, int32_t* packed, void* scale, void* mn_out, int64_t N, int64_t G,
                    int64_t group_size, int dtype, int stat_dtype, int stochastic, const void* noise, uint64_t seed,
                    uint64_t offset, bool min_is_exact, double width, cudaStream_t s) {
  if (int st = check_common(N, G, group_size, dtype, stat_dtype)) return st;
  if (N == 0 || G == 0) return ACTNN_OK;
  if (!data || !mn || !mx || !bits || !word_offsets || !packed || !scale) return ACTNN_ERR_NULL;
  if (group_size != kGroup)
    return pack_mixed_generic(data, mn, mx, bits, word_offsets, packed, scale, mn_out, N, G, group_size, dtype,
                              stat_dtype, stochastic, noise, seed, offset, s);
  const size_t al = dtype == ACTNN_F32 ? 32 : 16;
  if (!aligned(data, al) || (noise && !aligned(noise, al)) || !aligned(packed, 4)) return ACTNN_ERR_ALIGN;
  // the flat tasks need whole bundles and at most one sample boundary in 32 groups; other group counts
  // take the column kernels, which the step-by-step entry (min not known to be exact) does not have
  if (min_is_exact && mn_out && (G % kFlatBundle != 0 || G < kFlatGroups))
    return column_pack(data, mn, mx, bits, word_offsets, packed, scale, mn_out, N, G * kGroup, dtype, stat_dtype,
                       stochastic, noise, seed, offset, width, s);
  switch (dtype) {
    case ACTNN_F16:
      return launch_pack<__half, __half>(data, mn, mx, bits, word_offsets, packed, scale, mn_out, N, G,
                                         stochastic, noise, seed, offset, min_is_exact, s);
    case ACTNN_BF16:
      return launch_pack<__nv_bfloat16, __nv_bfloat16>(data, mn, mx, bits, word_offsets, packed, scale, mn_out,
                                                       N, G, stochastic, noise, seed, offset, min_is_exact, s);
    default:
      if (stat_dtype == ACTNN_BF16)
        return launch_pack<float, __nv_bfloat16>(data, mn, mx, bits, word_offsets, packed, scale, mn_out, N, G,
                                                 stochastic, noise, seed, offset, min_is_exact, s);
      return launch_pack<float, float>(data, mn, mx, bits, word_offsets, packed, scale, mn_out, N, G,
                                       stochastic, noise, seed, offset, min_is_exact, s);
  }
}
}  // namespace actnn

extern "C" int actnn_pack_mixed(const void* data, const void* mn, const void* mx, const int32_t* bits,
                                const int64_t* word_offsets, int32_t* packed, void* scale, void* mn_out,
                                int64_t N, int64_t G, int64_t group_size, int dtype, int stat_dtype,
                                int stochastic, const void* noise, uint64_t seed, uint64_t offset,
                                actnn_stream_t stream) {
  return pack_mixed_impl(data, mn, mx, bits, word_offsets, packed, scale, mn_out, N, G, group_size, dtype,
                         stat_dtype, stochastic, noise, seed, offset, false, 8.0, (cudaStream_t)stream);
}

extern "C" int actnn_bad_width_bundles(uint32_t* count) {
  if (!count) return ACTNN_ERR_NULL;
  return cudaMemcpyFromSymbol(count, g_bad_width_bundles, sizeof(unsigned)) == cudaSuccess ? ACTNN_OK
                                                                                           : ACTNN_ERR_LAUNCH;
}

extern "C" int actnn_unpack_mixed(const int32_t* packed, const int32_t* bits, const int64_t* word_offsets,
                                  const void* scale, const void* mn, void* out, int64_t N, int64_t G,
                                  int64_t group_size, int dtype, int stat_dtype, actnn_stream_t stream) {
  if (int st = check_common(N, G, group_size, dtype, stat_dtype)) return st;
  if (N == 0 || G == 0) return ACTNN_OK;
  if (!packed || !bits || !word_offsets || !scale || !mn || !out) return ACTNN_ERR_NULL;
  cudaStream_t s = (cudaStream_t)stream;
  if (group_size != kGroup)
    return unpack_mixed_generic(packed, bits, word_offsets, scale, mn, out, N, G, group_size, dtype, stat_dtype, s);
  if (!aligned(out, dtype == ACTNN_F32 ? 32 : 16) || !aligned(packed, 4)) return ACTNN_ERR_ALIGN;
  switch (dtype) {
    case ACTNN_F16: return launch_unpack<__half, __half>(packed, bits, word_offsets, scale, mn, out, N, G, s);
    case ACTNN_BF16:
      return launch_unpack<__nv_bfloat16, __nv_bfloat16>(packed, bits, word_offsets, scale, mn, out, N, G, s);
    default:
      if (stat_dtype == ACTNN_BF16)
        return launch_unpack<float, __nv_bfloat16>(packed, bits, word_offsets, scale, mn, out, N, G, s);
      return launch_unpack<float, float>(packed, bits, word_offsets, scale, mn, out, N, G, s);
  }
}
