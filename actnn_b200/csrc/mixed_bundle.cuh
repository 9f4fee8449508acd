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

template <int B> ACTNN_DEV uint32_t spread_codes_to_bytes(uint32_t r) {   // four B-bit codes -> one per byte
  if constexpr (B == 2) {
    uint32_t t = (r | (r << 12)) & 0x000f000fu;
    return (t | (t << 6)) & 0x03030303u;
  } else {
    uint32_t t = (r | (r << 14)) & 0x00030003u;
    return (t | (t << 7)) & 0x01010101u;
  }
}

// Decodes the four groups of a bundle of width B and hands them on one by one, use(group, octet): only
// one decoded octet per lane is live.  `words[k]` is word 32k + lane of the bundle (zero past its end);
// lane g < 4 holds the statistics of group g in (stat_scale, stat_mn).
template <typename T, int B, typename Use>
ACTNN_DEV void decode_bundle(const uint32_t (&words)[B], float stat_scale, float stat_mn, const TransposePlan& plan,
                             int lane, Use use) {
  constexpr int E = 1 << (B < 6 ? B : 5);              // table entries per group
  constexpr int GPC = (32 / E) < kBundle ? (32 / E) : kBundle;   // groups served by one table computation
  uint32_t S[B];
#pragma unroll
  for (int k = 0; k < B; ++k) S[k] = warp_transpose32(words[k], plan);
  uint32_t entry = 0u, pairs = 0u;
#pragma unroll
  for (int gi = 0; gi < kBundle; ++gi) {
    if constexpr (B < 6) {
      if (gi % GPC == 0) {                               // (re)build the table for groups gi .. gi+GPC-1
        const int g = (gi + lane / E) & (kBundle - 1);
        const float sc = __shfl_sync(kFull, stat_scale, g), m = __shfl_sync(kFull, stat_mn, g);
        entry = dequant_bits<T>((float)(lane % E), sc, m);
        if constexpr (sizeof(T) == 2 && B <= 2)
          pairs = entry | (__shfl_down_sync(kFull, entry, 1) << 16);
      }
    }
    uint32_t lo = 0u, hi = 0u;                           // this group's row
    if (gi == 0) { lo = get_bits<0 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<0 * 8 * B + 32, 8 * B - 32>(S); }
    if (gi == 1) { lo = get_bits<1 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<1 * 8 * B + 32, 8 * B - 32>(S); }
    if (gi == 2) { lo = get_bits<2 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<2 * 8 * B + 32, 8 * B - 32>(S); }
    if (gi == 3) { lo = get_bits<3 * 8 * B, (8 * B < 32 ? 8 * B : 32)>(S); if constexpr (8 * B > 32) hi = get_bits<3 * 8 * B + 32, 8 * B - 32>(S); }
    Oct<T> x;
    uint32_t* ow = reinterpret_cast<uint32_t*>(&x);
    if constexpr (sizeof(T) == 2 && B <= 2) {
      const int base = (gi % GPC) * E;
      const uint32_t t01 = __shfl_sync(kFull, pairs, base);
      const uint32_t t23 = B == 2 ? __shfl_sync(kFull, pairs, base + 2) : t01;
#pragma unroll
      for (int h = 0; h < 2; ++h) {                      // four elements per step
        const uint32_t y = spread_codes_to_bytes<B>((lo >> (4 * B * h)) & ((1u << (4 * B)) - 1u));
        const uint32_t sel = y * 0x22u + 0x10101010u;    // byte pair (2c, 2c+1) per element
        ow[2 * h] = __byte_perm(t01, t23, sel);
        ow[2 * h + 1] = __byte_perm(t01, t23, sel >> 16);
      }
    } else {
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
    }
    use(gi, x);
  }
}

}  // namespace
}  // namespace actnn
