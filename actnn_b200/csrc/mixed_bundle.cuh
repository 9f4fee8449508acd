// Four groups of the mixed-precision stream, one warp: the pieces that the flat and the column
// kernels share.  Lane t owns elements 8t .. 8t+7 of each group (see codec_mixed.cu for the layout).
#pragma once

#include "quant_math.cuh"

namespace actnn {
namespace {

constexpr int kBundle = 4;            // groups per bundle

enum NoiseMode { kNoisePhilox = 0, kNoiseTensor = 1, kNoiseNone = 2 };

// (mn', scale) of the lane's own group in the form the quantizer consumes.
template <typename T> struct LaneParams { uint32_t a, b; };
template <typename T> ACTNN_DEV LaneParams<T> lane_params(const GroupParams& gp) {
  LaneParams<T> p;
  if constexpr (sizeof(T) == 4) {
    p.a = __float_as_uint(gp.mn1);
    p.b = __float_as_uint(gp.scale);
  } else {
    p.a = bits_of<T>(gp.mn1) * 0x00010001u;
    p.b = bits_of<T>(gp.scale) * 0x00010001u;
  }
  return p;
}
template <typename T> ACTNN_DEV QP<T> fetch_lane_params(const LaneParams<T>& mine, int src_lane) {
  const uint32_t a = __shfl_sync(kFull, mine.a, src_lane), b = __shfl_sync(kFull, mine.b, src_lane);
  QP<T> q;
  if constexpr (sizeof(T) == 4) {
    q.mn1 = __uint_as_float(a);
    q.scale = __uint_as_float(b);
  } else {
    q.mn2 = *reinterpret_cast<const decltype(q.mn2)*>(&a);
    q.sc2 = *reinterpret_cast<const decltype(q.sc2)*>(&b);
  }
  return q;
}

// ------------------------------------------------------------------ codes as byte-permute selectors
// A group of a 16-bit type at up to 3 bits has at most eight different values: their low bytes fill two registers,
// their high bytes two more, and one byte permute picks four bytes by four codes -- if each code sits in a nibble
// of its own.  The transpose can leave them there for nothing: which word of the bundle a lane brings to it decides
// which bit of the string holds what, so lane i (nibble n = i / 4, bit r = i % 4) takes, as its k-th word,
//   1 bit:   word n of group r;                                  string 0: bit r of nibble n = code n of group r
//   2 bits:  word 2n + r % 2 of group 2k + r / 2;                string k: bits 2h, 2h + 1 of nibble n = code n of group 2k + h
//   3 bits:  r < 3: word 3n + r of group k; r = 3: word 3n + k of group 3;
//                                                                string k: bits 0..2 = code n of group k, bit 3 = bit k of group 3's
// instead of word 32k + i (the same 128-byte lines).  Two instructions for the selector of eight elements and eight
// permutes decode them, where spreading the codes of a row took 24 for 2 bits, and a shuffle an element at 3.
template <typename T, int B> constexpr bool kNibbles = sizeof(T) == 2 && B <= 3;

// The lane's k-th word of a bundle of width b is base(b) + k * step(b).
template <typename T> struct WordOrder {
  uint32_t packed;                     // bytes: base(1), base(2), base(3), step(3)
  int lane;
  ACTNN_DEV explicit WordOrder(int lane_) : lane(lane_) {
    const uint32_t n = (uint32_t)lane >> 2, r = (uint32_t)lane & 3u;
    const uint32_t b1 = 8 * r + n, b2 = 16 * (r >> 1) + 2 * n + (r & 1u), b3 = r < 3 ? 3 * n + r : 72 + 3 * n;
    packed = b1 | (b2 << 8) | (b3 << 16) | ((r < 3 ? 24u : 1u) << 24);
  }
  ACTNN_DEV int base(int b) const {
    if (sizeof(T) != 2) return lane;
    return b <= 3 ? (int)((packed >> ((8 * b - 8) & 31)) & 0xffu) : lane;
  }
  ACTNN_DEV int step(int b) const { return sizeof(T) == 2 && b == 3 ? (int)(packed >> 24) : 32; }
};

ACTNN_DEV uint32_t select_bytes(uint32_t a, uint32_t b, uint32_t sel) {     // sel: nibbles 0..7 in its low half
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
// Codes of group gi, one in each nibble.
template <int B> ACTNN_DEV uint32_t group_nibbles(const uint32_t (&S)[B], int gi) {
  if constexpr (B == 1) return (S[0] >> gi) & 0x11111111u;
  if constexpr (B == 2) return (S[gi >> 1] >> (2 * (gi & 1))) & 0x33333333u;
  if constexpr (B == 3) {
    if (gi < 3) return S[gi < 3 ? gi : 0] & 0x77777777u;
    return ((S[0] >> 3) & 0x11111111u) | ((S[1] >> 2) & 0x22222222u) | ((S[2] >> 1) & 0x44444444u);
  }
}
// Low and high bytes of the values of codes 0..3 and (3 bits) 4..7.
struct ByteTable { uint32_t lo0, hi0, lo1, hi1; };
template <typename T> ACTNN_DEV Oct<T> decode_nibbles(uint32_t sel, const ByteTable& t) {
  Oct<T> x;
  uint32_t* w = reinterpret_cast<uint32_t*>(&x);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t lo = select_bytes(t.lo0, t.lo1, sel), hi = select_bytes(t.hi0, t.hi1, sel);
    w[2 * h] = select_bytes(lo, hi, 0x5140u);
    w[2 * h + 1] = select_bytes(lo, hi, 0x7362u);
    sel >>= 16;
  }
  return x;
}

// decode_bundle for the widths whose codes the transpose leaves in nibbles.
template <typename T, int B, typename Use>
ACTNN_DEV void decode_bundle_nibbles(const uint32_t (&S)[B], float stat_scale, float stat_mn, int lane, Use use) {
  constexpr int E = 1 << B;
  const int g = (lane / E) & (kBundle - 1);
  const float sc = __shfl_sync(kFull, stat_scale, g), m = __shfl_sync(kFull, stat_mn, g);
  const uint32_t entry = dequant_bits<T>((float)(lane % E), sc, m);
  const uint32_t pair = entry | (__shfl_down_sync(kFull, entry, 1) << 16);
  uint32_t lo_l, hi_l = 0u;                            // bytes of this lane's value and the next three
  if constexpr (B == 1) {
    lo_l = select_bytes(pair, pair, 0x3120u);
  } else {
    const uint32_t pair2 = __shfl_down_sync(kFull, pair, 2);
    lo_l = select_bytes(pair, pair2, 0x6420u);
    hi_l = select_bytes(pair, pair2, 0x7531u);
  }
#pragma unroll
  for (int gi = 0; gi < kBundle; ++gi) {
    ByteTable t;
    t.lo0 = __shfl_sync(kFull, lo_l, gi * E);
    if constexpr (B == 1) t.hi0 = t.lo0 >> 16;
    else t.hi0 = __shfl_sync(kFull, hi_l, gi * E);
    t.lo1 = t.lo0;
    t.hi1 = t.hi0;
    if constexpr (B == 3) {
      t.lo1 = __shfl_sync(kFull, lo_l, gi * E + 4);
      t.hi1 = __shfl_sync(kFull, hi_l, gi * E + 4);
    }
    use(gi, decode_nibbles<T>(group_nibbles<B>(S, gi), t));
  }
}

// decode_bundle from rows, the codes of a group end to end: a shuffle fetches the value of each, from 6 bits on it is
// computed.
template <typename T, int B, typename Use>
ACTNN_DEV void decode_bundle_rows(const uint32_t (&S)[B], float stat_scale, float stat_mn, int lane, Use use) {
  constexpr int E = 1 << (B < 6 ? B : 5);              // table entries per group
  constexpr int GPC = (32 / E) < kBundle ? (32 / E) : kBundle;   // groups served by one table computation
  uint32_t entry = 0u;
#pragma unroll
  for (int gi = 0; gi < kBundle; ++gi) {
    if constexpr (B < 6) {
      if (gi % GPC == 0) {                               // (re)build the table for groups gi .. gi+GPC-1
        const int g = (gi + lane / E) & (kBundle - 1);
        const float sc = __shfl_sync(kFull, stat_scale, g), m = __shfl_sync(kFull, stat_mn, g);
        entry = dequant_bits<T>((float)(lane % E), sc, m);
      }
    }
    uint32_t lo = 0u, hi = 0u;                           // this group's row
    if (gi == 0) { lo = get_bits<0 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<0 * 8 * B + 32, 8 * B - 32>(S); }
    if (gi == 1) { lo = get_bits<1 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<1 * 8 * B + 32, 8 * B - 32>(S); }
    if (gi == 2) { lo = get_bits<2 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<2 * 8 * B + 32, 8 * B - 32>(S); }
    if (gi == 3) { lo = get_bits<3 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<3 * 8 * B + 32, 8 * B - 32>(S); }
    Oct<T> x;
    uint32_t* ow = reinterpret_cast<uint32_t*>(&x);
    uint32_t v[8];
    const uint32_t S2[2] = {lo, hi};
    uint32_t code[8];
    get_codes<B, 0>(S2, code);
    if constexpr (B < 6) {
      const int base = (gi % GPC) * E;
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __shfl_sync(kFull, entry, base + (int)code[j]);
    } else {
      const float sc = __shfl_sync(kFull, stat_scale, gi), m = __shfl_sync(kFull, stat_mn, gi);
      float y = 0.f;
      if (sizeof(T) == 2 && group_reciprocal(sc, y)) {           // 16-bit statistics; warp-uniform
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
    use(gi, x);
  }
}

// Decodes the four groups of a bundle of width B and hands them on one by one, use(group, octet): only
// one decoded octet per lane is live.  `words[k]` is the lane's k-th word (WordOrder) of the bundle, zero past its
// end; lane g < 4 holds the statistics of group g in (stat_scale, stat_mn).
template <typename T, int B, typename Use>
ACTNN_DEV void decode_bundle(const uint32_t (&words)[B], float stat_scale, float stat_mn, const TransposePlan& plan,
                             int lane, Use use) {
  uint32_t S[B];
#pragma unroll
  for (int k = 0; k < B; ++k) S[k] = warp_transpose32(words[k], plan);
  if constexpr (kNibbles<T, B>) decode_bundle_nibbles<T, B>(S, stat_scale, stat_mn, lane, use);
  else decode_bundle_rows<T, B>(S, stat_scale, stat_mn, lane, use);
}

}  // namespace
}  // namespace actnn
