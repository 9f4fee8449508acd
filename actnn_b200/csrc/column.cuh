// The column mapping of the mixed-precision codec: a warp owns one bundle of four consecutive groups
// POSITION (a "column" of the [sample, group] grid) and walks down the samples of a split with it.
//
// Against tasks of consecutive groups this buys three things.  The position inside the sample is
// fixed for the whole kernel, so what depends on it -- the channel of each element, the channel's
// coefficients, how many elements of the last octet exist -- is worked out once per warp instead
// of once per octet.  Per-channel sums live in registers across all samples of the split.  And a
// sample needs no particular length: [N, F] is addressed as it is, elements past F read as zero
// (what the reference's padding holds, actnn/actnn/qscheme.py:61-71) and are never written.
#pragma once

#include "mixed_bundle.cuh"

namespace actnn {
namespace {

constexpr int kColThreads = 256;

struct ColumnShape {
  int64_t F;          // elements per sample
  int N, G;           // samples, groups per sample (the last one may be partial)
  int P, S, spp;      // columns, splits of the samples, samples per split
  int align;          // elements (1, 2, 4, 8) that octets of the activation are aligned to
};

// Splits of the samples: a warp per (column, split).  The resident warps should all be busy and the
// last wave should not be nearly empty, so the candidates are one to four waves' worth of warps and
// the one with the fewest bundles on the critical path (plus a bundle's worth of start-up) is taken.
struct SampleSplits { int S, spp; };
inline SampleSplits split_samples(int64_t N, int64_t P, int warps_per_sm) {
  const int64_t resident = (int64_t)device_info().sm_count * warps_per_sm;
  SampleSplits r = {1, (int)N};
  int64_t best = -1;
  for (int k = 1; k <= 4; ++k) {
    int64_t S = resident * k / P;
    S = S < 1 ? 1 : S > N ? N : S;
    const int64_t spp = (N + S - 1) / S;
    S = (N + spp - 1) / spp;
    const int64_t cost = (P * S + resident - 1) / resident * (spp + 1);
    if (best < 0 || cost < best) { best = cost; r.S = (int)S; r.spp = (int)spp; }
  }
  return r;
}
inline ColumnShape column_shape(int64_t N, int64_t F, int align, int warps_per_sm) {
  ColumnShape sh;
  sh.F = F;
  sh.N = (int)N;
  sh.G = (int)((F + kGroup - 1) / kGroup);
  sh.P = (sh.G + kBundle - 1) / kBundle;
  sh.align = align;
  const SampleSplits splits = split_samples(N, sh.P, warps_per_sm);
  sh.S = splits.S;
  sh.spp = splits.spp;
  return sh;
}
inline int column_grid(const ColumnShape& sh) {
  return (int)(((int64_t)sh.P * sh.S + kColThreads / 32 - 1) / (kColThreads / 32));
}
inline bool column_supported(int64_t N, int64_t F) {
  if (N <= 0 || F <= 0 || N > 0x7fffffff || F > ((int64_t)1 << 38)) return false;
  const int64_t P = (F + kBundle * kGroup - 1) / (kBundle * kGroup);
  return N * P < ((int64_t)1 << 31);
}
// Alignment, in elements, of every octet of a [N, F] activation at `p`.
inline int octet_alignment(const void* p, int64_t F, int elem_size) {
  int a = kOct;
  while (a > 1 && (F % a != 0 || !aligned(p, (size_t)a * elem_size))) a >>= 1;
  return a;
}

// This warp's column and split.
struct ColumnTask {
  int p, g0, count;   // column, its first group, its groups (1..4)
  int n0, n1;         // samples
  bool valid;
};
ACTNN_DEV ColumnTask column_task(const ColumnShape& sh) {
  ColumnTask t;
  const uint32_t warp = blockIdx.x * (kColThreads / 32) + (threadIdx.x >> 5);
  const uint32_t s = warp / (uint32_t)sh.P;
  t.p = (int)(warp - s * (uint32_t)sh.P);
  t.g0 = t.p * kBundle;
  t.count = min(kBundle, sh.G - t.g0);
  t.n0 = (int)s * sh.spp;
  t.n1 = min(sh.N, t.n0 + sh.spp);
  t.valid = (int)s < sh.S;
  return t;
}

// ------------------------------------------------------------------ octets at any alignment
template <int BYTES> struct WordOf;
template <> struct WordOf<16> { using type = uint4; };
template <> struct WordOf<8> { using type = uint2; };
template <> struct WordOf<4> { using type = uint32_t; };
template <> struct WordOf<2> { using type = uint16_t; };

template <typename T, int A> ACTNN_DEV void load_pieces(const T* p, Oct<T>& o) {
  using W = typename WordOf<A * sizeof(T)>::type;
  W* dst = reinterpret_cast<W*>(&o);
#pragma unroll
  for (int i = 0; i < kOct / A; ++i) dst[i] = __ldg(reinterpret_cast<const W*>(p) + i);
}
template <typename T, int A> ACTNN_DEV void store_pieces(T* p, const Oct<T>& o) {
  using W = typename WordOf<A * sizeof(T)>::type;
  const W* src = reinterpret_cast<const W*>(&o);
#pragma unroll
  for (int i = 0; i < kOct / A; ++i) reinterpret_cast<W*>(p)[i] = src[i];
}
// The octet at `p`, of which the first `valid` elements exist; the others read as zero.
// EDGE = false: a whole octet on its natural alignment.
template <typename T, bool EDGE> ACTNN_DEV Oct<T> load_octet(const T* p, int valid, int align) {
  if constexpr (!EDGE) return load_oct<T>(p);
  Oct<T> o = zero_oct<T>();
  if (valid >= kOct) {
    if (align == 8) o = load_oct<T>(p);
    else if (align == 4) load_pieces<T, 4>(p, o);
    else if (align == 2) load_pieces<T, 2>(p, o);
    else load_pieces<T, 1>(p, o);
  } else if (valid > 0) {
    T* e = reinterpret_cast<T*>(&o);
#pragma unroll
    for (int j = 0; j < kOct - 1; ++j)
      if (j < valid) e[j] = p[j];
  }
  return o;
}
template <typename T, bool EDGE> ACTNN_DEV void store_octet(T* p, const Oct<T>& o, int valid, int align) {
  if constexpr (!EDGE) {
    store_oct_streaming<T>(p, o);
  } else if (valid >= kOct) {
    if (align == 8) store_oct_streaming<T>(p, o);
    else if (align == 4) store_pieces<T, 4>(p, o);
    else if (align == 2) store_pieces<T, 2>(p, o);
    else store_pieces<T, 1>(p, o);
  } else if (valid > 0) {
    const T* e = reinterpret_cast<const T*>(&o);
#pragma unroll
    for (int j = 0; j < kOct - 1; ++j)
      if (j < valid) p[j] = e[j];
  }
}

// The four octets of this lane in sample n: element offsets inside the sample and how many exist.
template <bool EDGE> struct ColumnOctets {
  int64_t first;              // offset of the lane's octet of group 0 of the column
  int valid[EDGE ? kBundle : 1];
  int count, align;
  ACTNN_DEV ColumnOctets(const ColumnShape& sh, const ColumnTask& t, int lane) {
    first = (int64_t)t.g0 * kGroup + lane * kOct;
    count = t.count;
    align = sh.align;
    if constexpr (EDGE) {
#pragma unroll
      for (int gi = 0; gi < kBundle; ++gi)
        valid[gi] = (int)max((int64_t)0, min((int64_t)kOct, sh.F - (first + gi * kGroup)));
    }
  }
  template <typename T> ACTNN_DEV void load(const T* sample, Oct<T> (&x)[kBundle]) const {
#pragma unroll
    for (int gi = 0; gi < kBundle; ++gi) {
      if constexpr (EDGE) x[gi] = load_octet<T, true>(sample + first + gi * kGroup, valid[gi], align);
      else x[gi] = gi < count ? load_oct<T>(sample + first + gi * kGroup) : zero_oct<T>();
    }
  }
  // The column's part of a sample into the L2; one lane asks for all of it.
  template <typename T> ACTNN_DEV void prefetch(const T* sample, const ColumnShape& sh, int lane) const {
    if (lane != 0 || (EDGE && align != kOct)) return;
    l2_prefetch(sample + first, (uint32_t)(min((int64_t)(kBundle * kGroup), sh.F - first) * (int64_t)sizeof(T)));
  }
  template <typename T> ACTNN_DEV void store(T* sample, int gi, const Oct<T>& x) const {
    if constexpr (EDGE) store_octet<T, true>(sample + first + gi * kGroup, x, valid[gi], align);
    else if (gi < count) store_oct_streaming<T>(sample + first + gi * kGroup, x);
  }
};

// ------------------------------------------------------------------ group min / max of a bundle
// Lane gi (< COUNT) ends with the extrema of group gi.
template <typename T, int COUNT = kBundle>
ACTNN_DEV void bundle_minmax(const Oct<T> (&x)[kBundle], int lane, float& mn, float& mx) {
#pragma unroll
  for (int gi = 0; gi < COUNT; ++gi) {
    float lo, hi;
    oct_minmax<T>(x[gi], lo, hi);
    lo = warp_min(lo);
    hi = warp_max(hi);
    if (lane == gi) { mn = lo; mx = hi; }
  }
}

// ------------------------------------------------------------------ noise of four consecutive groups
// Groups q .. q+3 of the activation; generator calls serve aligned blocks of GPC groups (see
// quant_math.cuh), so an unaligned q needs one call more.
template <typename T>
ACTNN_DEV void noise_bundle(const NoiseKey& key, int64_t q, int lane, Oct<T> (&nz)[kBundle]) {
  constexpr int GPC = NoiseShape<T>::GPC;
  const int r = (int)(q % GPC);
  if (r == 0) {
#pragma unroll
    for (int gi = 0; gi < kBundle; gi += GPC) {
      const NoiseWords w = expand_call(noise_call(key, (uint64_t)((q + gi) / GPC) * 32ull + (uint64_t)lane));
#pragma unroll
      for (int h = 0; h < GPC; ++h) nz[gi + h] = noise_oct<T>(w, h);
    }
    return;
  }
  NoiseWords w = expand_call(noise_call(key, (uint64_t)(q / GPC) * 32ull + (uint64_t)lane));
#pragma unroll
  for (int gi = 0; gi < kBundle; ++gi) {
    const int slot = (r + gi) % GPC;
    if (gi > 0 && slot == 0) w = expand_call(noise_call(key, (uint64_t)((q + gi) / GPC) * 32ull + (uint64_t)lane));
    nz[gi] = noise_oct<T>(w, slot);
  }
}

// ------------------------------------------------------------------ pack one bundle of width B
template <typename T, int B>
ACTNN_DEV void pack_column_bundle(const Oct<T> (&x)[kBundle], const Oct<T> (&nz)[kBundle], const LaneParams<T>& mine,
                                  int first_lane, int count, int32_t* __restrict__ out, const TransposePlan& plan,
                                  int lane) {
  uint32_t S[B];
#pragma unroll
  for (int k = 0; k < B; ++k) S[k] = 0u;
#pragma unroll
  for (int gi = 0; gi < kBundle; ++gi) {
    const QP<T> qp = fetch_lane_params<T>(mine, first_lane + gi);
    uint32_t lo, hi;
    row_from_magic<T, B>(quantize_oct<T, false, B>(x[gi], nz[gi], qp), lo, hi);
    if (gi == 0) put_row<B, 0 * 8 * B>(S, lo, hi);
    if (gi == 1) put_row<B, 1 * 8 * B>(S, lo, hi);
    if (gi == 2) put_row<B, 2 * 8 * B>(S, lo, hi);
    if (gi == 3) put_row<B, 3 * 8 * B>(S, lo, hi);
  }
  const int words = count * 8 * B;                       // groups past the sample's last one have no words
#pragma unroll
  for (int k = 0; k < B; ++k) {
    const uint32_t w = warp_transpose32(S[k], plan);
    if (k * 32 + lane < words) out[k * 32 + lane] = (int32_t)w;
  }
}

// Scale, stochastic rounding and pack of a column; each(n, octets) sees every sample's octets on the way.  `ahead`: the
// octets of the sample after the one being loaded are requested into the L2.
// Eight samples at a time: lane 4i + g prepares group g of the i-th of them (one division per lane for eight
// bundles).  The noise octets are formed before the dispatch on the width, so the eight width variants stay short.
template <typename T, typename ST, bool PHILOX, bool EDGE, typename Each>
ACTNN_DEV void pack_column(const T* __restrict__ data, const ColumnShape& sh, const ColumnTask& t,
                           const ColumnOctets<EDGE>& oct, const T* __restrict__ mn, const T* __restrict__ mx,
                           const int32_t* __restrict__ bits, const int64_t* __restrict__ word_offsets,
                           int32_t* __restrict__ packed, ST* __restrict__ scale, ST* __restrict__ mn_out,
                           const T* __restrict__ noise, const NoiseKey& key, int lane, bool ahead, Each each) {
  const TransposePlan plan = make_transpose_plan(lane);
  Oct<T> next[kBundle];
  oct.template load<T>(data + (int64_t)t.n0 * sh.F, next);
  for (int nb = t.n0; nb < t.n1; nb += 8) {
    const int n_l = nb + (lane >> 2), g_l = lane & 3;
    int b_l = 0;
    int64_t off_l = 0;
    LaneParams<T> mine = {0u, 0u};
    if (n_l < t.n1 && g_l < t.count) {
      b_l = __ldg(bits + n_l);
      if (b_l < 1 || b_l > 8) b_l = 0;                   // not a width: nothing written
      off_l = __ldg(word_offsets + n_l) + (int64_t)t.g0 * 8 * b_l;
      const int64_t q = (int64_t)n_l * sh.G + t.g0 + g_l;
      const float gmn = load_scalar<T>(mn, q), gmx = load_scalar<T>(mx, q);
      const GroupParams gp = prepare_group<T>(gmn, gmx, b_l);
      store_scalar<ST>(scale, q, gp.scale);
      store_scalar<ST>(mn_out, q, gmn);
      mine = lane_params<T>(gp);
    }
    const int cnt = min(8, t.n1 - nb);
    for (int i = 0; i < cnt; ++i) {
      const int n = nb + i;
      Oct<T> x[kBundle], nz[kBundle];
#pragma unroll
      for (int gi = 0; gi < kBundle; ++gi) x[gi] = next[gi];
      if (n + 1 < t.n1) oct.template load<T>(data + (int64_t)(n + 1) * sh.F, next);
      if (ahead && n + 2 < t.n1) oct.template prefetch<T>(data + (int64_t)(n + 2) * sh.F, sh, lane);
      const int64_t q0 = (int64_t)n * sh.G + t.g0;
      if constexpr (PHILOX) {
        noise_bundle<T>(key, q0, lane, nz);
      } else {                                           // an injected tensor shaped [N, G, 256], or none
#pragma unroll
        for (int gi = 0; gi < kBundle; ++gi)
          nz[gi] = noise && gi < t.count ? load_oct<T>(noise + (q0 + gi) * kGroup + lane * kOct) : zero_oct<T>();
      }
      each(n, x);
      const int b = __shfl_sync(kFull, b_l, 4 * i);
      const uint32_t olo = __shfl_sync(kFull, (uint32_t)off_l, 4 * i);
      const uint32_t ohi = __shfl_sync(kFull, (uint32_t)((uint64_t)off_l >> 32), 4 * i);
      int32_t* out = packed + (int64_t)(((uint64_t)ohi << 32) | olo);
#define ACTNN_CASE(B) \
      case B: pack_column_bundle<T, B>(x, nz, mine, 4 * i, t.count, out, plan, lane); break;
      switch (b) {
        ACTNN_CASE(1) ACTNN_CASE(2) ACTNN_CASE(3) ACTNN_CASE(4) ACTNN_CASE(5) ACTNN_CASE(6) ACTNN_CASE(7)
        ACTNN_CASE(8)
        default: break;
      }
#undef ACTNN_CASE
    }
  }
}

// ------------------------------------------------------------------ the stream of a column, read ahead
// Of a block of 32 samples, lane l knows the width and the stream position of the l-th; the first words
// and the statistics (lane gi < 4: group gi) of one bundle are requested a sample ahead of their use.
// Four words a lane are a bundle of up to 4 bits, nearly all there is at an average of 2; wider
// bundles load the rest when they are decoded, which keeps four registers free in the common case.
constexpr int kAhead = 4;
struct BundleWords {
  uint32_t w[kAhead];
  float sc, m;                // statistics of group `lane`
  const int32_t* in;          // the bundle's first word
  int b;                      // 0: not a width, nothing was written
};
struct ColumnStream {
  int b_l;                    // width of the lane's sample
  int64_t off_l;              // first word of that sample's bundle
  ACTNN_DEV void open(const ColumnTask& t, int n_l, bool active, const int32_t* __restrict__ bits,
                      const int64_t* __restrict__ word_offsets) {
    b_l = 0;
    off_l = 0;
    if (active) {
      b_l = __ldg(bits + n_l);
      if (b_l < 1 || b_l > 8) b_l = 0;
      off_l = __ldg(word_offsets + n_l) + (int64_t)t.g0 * 8 * b_l;
    }
  }
  // sample n, which is lane i's
  template <typename T, typename ST>
  ACTNN_DEV BundleWords fetch(const ColumnTask& t, const WordOrder<T>& order, int G, int n, int i,
                              const int32_t* __restrict__ packed, const ST* __restrict__ scale,
                              const ST* __restrict__ mn, int lane) const {
    BundleWords r;
    r.b = __shfl_sync(kFull, b_l, i);
    const uint32_t olo = __shfl_sync(kFull, (uint32_t)off_l, i);
    const uint32_t ohi = __shfl_sync(kFull, (uint32_t)((uint64_t)off_l >> 32), i);
    r.in = packed + (int64_t)(((uint64_t)ohi << 32) | olo);
    const int words = t.count * 8 * r.b;
    // one set of loads for all widths: with a branch for the narrow ones, unpack of 512 x 784 groups less 8 elements of float16 at 2 /
    // 4 / 6 bits 49.3 / 76.6 / 105 us, so 47.9 / 75.0 / 101
    const int base = order.base(r.b), step = order.step(r.b);
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const int w = base + k * step;
      r.w[k] = k < r.b && w < words ? (uint32_t)__ldg(r.in + w) : 0u;
    }
    r.sc = 1.f;
    r.m = 0.f;
    if (lane < t.count) {
      const int64_t q = (int64_t)n * G + t.g0 + lane;
      r.sc = load_scalar<ST>(scale, q);
      r.m = load_scalar<ST>(mn, q);
    }
    return r;
  }
};
template <typename T, int B, typename Use>
ACTNN_DEV void decode_words(const BundleWords& r, int count, const TransposePlan& plan, int lane, Use use) {
  uint32_t w[B];
#pragma unroll
  for (int k = 0; k < B; ++k)
    w[k] = k < kAhead ? r.w[k < kAhead ? k : 0] : k * 32 + lane < count * 8 * B ? (uint32_t)__ldg(r.in + k * 32 + lane) : 0u;
  decode_bundle<T, B>(w, r.sc, r.m, plan, lane, use);
}
template <typename T, typename Use>
ACTNN_DEV void decode_column(const BundleWords& r, int count, const TransposePlan& plan, int lane, Use use) {
  switch (r.b) {
    case 1: decode_words<T, 1>(r, count, plan, lane, use); break;
    case 2: decode_words<T, 2>(r, count, plan, lane, use); break;
    case 3: decode_words<T, 3>(r, count, plan, lane, use); break;
    case 4: decode_words<T, 4>(r, count, plan, lane, use); break;
    case 5: decode_words<T, 5>(r, count, plan, lane, use); break;
    case 6: decode_words<T, 6>(r, count, plan, lane, use); break;
    case 7: decode_words<T, 7>(r, count, plan, lane, use); break;
    case 8: decode_words<T, 8>(r, count, plan, lane, use); break;
    default: break;
  }
}

}  // namespace
}  // namespace actnn
