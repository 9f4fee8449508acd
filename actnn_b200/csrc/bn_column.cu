// Batch-norm passes fused with the compression of their input, on the column mapping (column.cuh).
//
// Forward: one read of x gives the statistics and the group ranges, the second packs AND normalises:
//   stats   min / max of the bundle's groups, sums of (x - shift) and its square per octet in registers;
//   finish  one warp per channel: mean, inverse deviation, running statistics, coefficients;
//           (maps of a group and more: both from the pass of bn_stats_minimax_kernel, called before)
//   (allocation of the widths, stats.cu)
//   pack    codes and y from the same registers.
// 4 + b/8 + 2 bytes an element for 16-bit types; statistics, pack and normalisation as passes of their own read x
// three times.  float16 256 x 64 x 56 x 56: pack 28.1 + coefficients 1.6 + normalise 32.4 us -> 37.6 us (6.1 TB/s would be
// 36); 128 x 256 x 14 x 14, seven launches 34 us -> four 24.6 us.
//
// Backward: both passes decode the saved codes in registers, so the decoded activation is never
// written to memory (the reference decodes it, ops.py:470-476, and cuDNN reads it back, ops.py:490-493):
//   reduce  reads the codes and dy; sum(dy) and sum(dy * (x - mean)) of the lane's octets stay in
//           registers across the samples of the split, because an octet position has one channel;
//   finish  one warp per channel adds the columns' and splits' sums in a fixed order;
//   apply   reads the codes and dy again and writes dx, walking the samples backwards so that it
//           starts with what the reduce left in the L2.
// Per element of a 16-bit activation that is 2 + b/8 bytes for the reduce and 4 + b/8 for the apply,
// against 2 (decode) + 4 + 6.  The apply moves 0.83 of the copy rate, the reduce 0.53.  With 16 warps an SM it issues 57 % of
// the time, and nothing tried moved that: a ring of bulk copies for dy and the words 42.0 / 40.6 us (reduce / apply),
// a ring of per-lane asynchronous copies without barriers 35.0 - 36.0 / 39.3 - 39.9, dy requested into the L2 ahead
// 35.1 / 37.7, a third block an SM 36.2 / 47.6, a decode of half the instructions 32.5 / 39.4 against 32.7 / 39.5.
// float16, 256 x 64 x 56 x 56: decode 24.9 + reduce 40.9 + apply 40.5 us -> 32.5 + 2.6 + 39.4.
#include "column.cuh"

namespace actnn {
namespace {

// Elements 8t .. 8t+7 touch one channel (SUB = 8: HW % 8 == 0), one channel per half (SUB = 4: HW % 4 == 0) or change
// channel at any element (SUB = 1).  HW >= 8, so there are at most two.
template <int SUB> struct Slots { static constexpr int N = SUB == 8 ? 1 : 2; };

struct BnColumns { int C, HW, kmax; };       // kmax: channels a column can touch

// Channels of the lane's octets; a channel number >= C marks elements past the end of the sample.
template <int SUB> struct ColumnChannels {
  static constexpr int NS = Slots<SUB>::N;
  int ch[kBundle][NS];
  int first_of_next[SUB == 1 ? kBundle : 1];      // SUB = 1: first element of slot 1
  int c_lo, nch;                                  // channels of the whole column
  ACTNN_DEV ColumnChannels(const ColumnShape& sh, const BnColumns& bn, const ColumnTask& t, int lane) {
    const uint32_t hw = (uint32_t)bn.HW;
    const uint32_t e0 = (uint32_t)t.p * (kBundle * kGroup);
    const uint32_t last = (uint32_t)min((int64_t)e0 + kBundle * kGroup, sh.F) - 1u;
    c_lo = (int)(e0 / hw);
    nch = (int)(last / hw) - c_lo + 1;
#pragma unroll
    for (int gi = 0; gi < kBundle; ++gi) {
      const uint32_t e = e0 + gi * kGroup + lane * kOct;
      ch[gi][0] = (int)(e / hw);
      if constexpr (SUB == 4) ch[gi][1] = (int)((e + 4) / hw);
      if constexpr (SUB == 1) {
        ch[gi][1] = ch[gi][0] + 1;
        first_of_next[gi] = (int)min(8u, (uint32_t)ch[gi][1] * hw - e);
      }
    }
  }
  ACTNN_DEV bool second(int gi, int j) const {     // element j of octet gi belongs to slot 1
    if constexpr (SUB == 8) return false;
    else if constexpr (SUB == 4) return j >= 4;
    else return j >= first_of_next[gi];
  }
};

// Two float32 operations per instruction (sm_100).
ACTNN_DEV float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 c, a, b;\n\t"
      "mov.b64 {%0, %1}, c;\n\t}" : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
ACTNN_DEV float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
ACTNN_DEV float2 both(float v) { return make_float2(v, v); }

// Elements 2k, 2k+1 of an octet.
template <typename T> ACTNN_DEV float2 octet_pair(const Oct<T>& o, int k) {
  if constexpr (sizeof(T) == 4) return make_float2(o.f[2 * k], o.f[2 * k + 1]);
  else if constexpr (DType<T>::id == ACTNN_F16) return __half22float2(*reinterpret_cast<const __half2*>(&o.r[k]));
  else return make_float2(__uint_as_float(o.r[k] << 16), __uint_as_float(o.r[k] & 0xffff0000u));
}
// Elements 2k, 2k+1 plus (a, b): for the 16-bit types the mixed-precision add of sm_100, no conversion.
template <typename T> ACTNN_DEV float2 octet_pair_plus(const Oct<T>& o, int k, float a, float b) {
  if constexpr (sizeof(T) == 4) {
    return add2(make_float2(o.f[2 * k], o.f[2 * k + 1]), make_float2(a, b));
  } else {
    float2 r;
    const uint16_t lo = (uint16_t)o.r[k], hi = (uint16_t)(o.r[k] >> 16);
    if constexpr (DType<T>::id == ACTNN_F16) {
      asm("add.rn.f32.f16 %0, %1, %2;" : "=f"(r.x) : "h"(lo), "f"(a));
      asm("add.rn.f32.f16 %0, %1, %2;" : "=f"(r.y) : "h"(hi), "f"(b));
    } else {
      asm("add.rn.f32.bf16 %0, %1, %2;" : "=f"(r.x) : "h"(lo), "f"(a));
      asm("add.rn.f32.bf16 %0, %1, %2;" : "=f"(r.y) : "h"(hi), "f"(b));
    }
    return r;
  }
}
// Element e plus a, likewise.
template <typename T> ACTNN_DEV float octet_plus(const Oct<T>& o, int e, float a) {
  if constexpr (sizeof(T) == 4) return o.f[e] + a;
  else return e % 2 ? octet_pair_plus<T>(o, e / 2, 0.f, a).y : octet_pair_plus<T>(o, e / 2, a, 0.f).x;
}
template <typename T> ACTNN_DEV void set_octet_pair(Oct<T>& o, int k, float2 v) {
  if constexpr (sizeof(T) == 4) {
    o.f[2 * k] = v.x;
    o.f[2 * k + 1] = v.y;
  } else if constexpr (DType<T>::id == ACTNN_F16) {
    const __half2 h = __floats2half2_rn(v.x, v.y);
    o.r[k] = *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
    o.r[k] = *reinterpret_cast<const uint32_t*>(&h);
  }
}

// Sums of two quantities per channel of the column, from per-lane sums per octet and slot; partial sum k
// of the column is channel c_lo + k's.
template <int SUB>
ACTNN_DEV void write_partials(const ColumnChannels<SUB>& cc, const float2 (&a)[kBundle][Slots<SUB>::N],
                              const float2 (&b)[kBundle][Slots<SUB>::N], float2* __restrict__ dst, int lane) {
  for (int k = 0; k < cc.nch; ++k) {
    float sa = 0.f, sb = 0.f;
#pragma unroll
    for (int gi = 0; gi < kBundle; ++gi) {
#pragma unroll
      for (int s = 0; s < Slots<SUB>::N; ++s) {
        if (cc.ch[gi][s] == cc.c_lo + k) { sa += a[gi][s].x + a[gi][s].y; sb += b[gi][s].x + b[gi][s].y; }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sa += __shfl_xor_sync(kFull, sa, o);
      sb += __shfl_xor_sync(kFull, sb, o);
    }
    if (lane == 0) dst[k] = make_float2(sa, sb);
  }
}

// Channel c's sums over all columns and splits, in a fixed order; one warp, the result in every lane.
ACTNN_DEV float2 collect_partials(const ColumnShape& sh, const BnColumns& bn, const float2* __restrict__ partial, int c,
                                  int lane) {
  const uint32_t span = kBundle * kGroup;
  const uint32_t first = (uint32_t)c * (uint32_t)bn.HW, last = first + (uint32_t)bn.HW - 1u;
  const int p_lo = (int)(first / span), np = (int)(last / span) - p_lo + 1;
  float a = 0.f, b = 0.f;
  for (int i = lane; i < np * sh.S; i += 32) {
    const int s = i / np, p = p_lo + (i - s * np);
    const int k = c - (int)((uint32_t)p * span / (uint32_t)bn.HW);
    const float2 v = __ldg(partial + ((int64_t)s * sh.P + p) * bn.kmax + k);
    a += v.x;
    b += v.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(kFull, a, o);
    b += __shfl_xor_sync(kFull, b, o);
  }
  return make_float2(a, b);
}

constexpr int kBnBlocks = 2;     // resident blocks per SM: 128 registers and no spills beat 3 blocks with them (40.1 against 41.3 us, apply)

constexpr int bn_stats_blocks(int elem_size, int sub) { return elem_size == 2 && sub == 8 ? 3 : 2; }

// ------------------------------------------------------------------ forward
template <typename T, int SUB, bool EDGE>
__global__ void __launch_bounds__(kColThreads, bn_stats_blocks(sizeof(T), SUB))
bn_column_stats_kernel(const T* __restrict__ x, ColumnShape sh, BnColumns bn, T* __restrict__ mn, T* __restrict__ mx,
                       float2* __restrict__ partial) {
  constexpr int NS = Slots<SUB>::N;
  const int lane = threadIdx.x & 31;
  const ColumnTask t = column_task(sh);
  if (!t.valid) return;
  const ColumnOctets<EDGE> oct(sh, t, lane);
  const ColumnChannels<SUB> cc(sh, bn, t, lane);
  float neg_shift[kBundle][NS];                        // shift: the channel's first element
  float2 sum[kBundle][NS], sq[kBundle][NS];
#pragma unroll
  for (int gi = 0; gi < kBundle; ++gi) {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      neg_shift[gi][s] = cc.ch[gi][s] < bn.C ? -load_scalar<T>(x, (int64_t)cc.ch[gi][s] * bn.HW) : 0.f;
      sum[gi][s] = sq[gi][s] = both(0.f);
    }
  }
  // the samples from the last to the first: the pack starts with what is read here last
  Oct<T> next[kBundle];
  oct.template load<T>(x + (int64_t)(t.n1 - 1) * sh.F, next);
  for (int n = t.n1 - 1; n >= t.n0; --n) {
    Oct<T> v[kBundle];
#pragma unroll
    for (int gi = 0; gi < kBundle; ++gi) v[gi] = next[gi];
    if (n > t.n0) oct.template load<T>(x + (int64_t)(n - 1) * sh.F, next);
    float lo = 0.f, hi = 0.f;
    bundle_minmax<T>(v, lane, lo, hi);
    if (lane < t.count) {
      const int64_t q = (int64_t)n * sh.G + t.g0 + lane;
      store_scalar<T>(mn, q, lo);
      store_scalar<T>(mx, q, hi);
    }
#pragma unroll
    for (int gi = 0; gi < kBundle; ++gi) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if constexpr (SUB != 1) {
          const int s = SUB == 8 ? 0 : k / 2;
          const float2 d = octet_pair_plus<T>(v[gi], k, neg_shift[gi][s], neg_shift[gi][s]);
          sum[gi][s] = add2(sum[gi][s], d);
          sq[gi][s] = fma2(d, d, sq[gi][s]);
        } else {
          const bool s0 = cc.second(gi, 2 * k), s1 = cc.second(gi, 2 * k + 1);
          const float2 d = octet_pair_plus<T>(v[gi], k, neg_shift[gi][s0 ? 1 : 0], neg_shift[gi][s1 ? 1 : 0]);
          sum[gi][0].x += s0 ? 0.f : d.x; sum[gi][0].y += s1 ? 0.f : d.y;
          sum[gi][1].x += s0 ? d.x : 0.f; sum[gi][1].y += s1 ? d.y : 0.f;
          sq[gi][0].x += s0 ? 0.f : d.x * d.x; sq[gi][0].y += s1 ? 0.f : d.y * d.y;
          sq[gi][1].x += s0 ? d.x * d.x : 0.f; sq[gi][1].y += s1 ? d.y * d.y : 0.f;
        }
      }
    }
  }
  const int split = t.n0 / sh.spp;
  write_partials<SUB>(cc, sum, sq, partial + ((int64_t)split * sh.P + t.p) * bn.kmax, lane);
}

// Statistics of channel c from the sums of its (x - shift) and their squares.
template <typename T>
ACTNN_DEV void finish_channel(float2 tot, int N, int HW, int c, const T* __restrict__ x, float* __restrict__ running_mean,
                              float* __restrict__ running_var, float* __restrict__ save_mean,
                              float* __restrict__ save_invstd, float momentum, float eps) {
  const float M = (float)N * (float)HW;
  const float m_s = tot.x / M;
  const float var = fmaxf(tot.y / M - m_s * m_s, 0.f);
  const float mean = load_scalar<T>(x, (int64_t)c * HW) + m_s;
  const float invstd = 1.0f / sqrtf(var + eps);
  save_mean[c] = mean;
  save_invstd[c] = invstd;
  if (running_mean) running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * mean;
  if (running_var) {
    const float unbiased = M > 1.f ? var * (M / (M - 1.f)) : var;
    running_var[c] = (1.f - momentum) * running_var[c] + momentum * unbiased;
  }
}

// One warp per channel.
template <typename T>
__global__ void __launch_bounds__(kColThreads)
bn_column_stats_finish_kernel(const float2* __restrict__ partial, ColumnShape sh, BnColumns bn, const T* __restrict__ x,
                              float* __restrict__ running_mean, float* __restrict__ running_var,
                              float* __restrict__ save_mean, float* __restrict__ save_invstd, float momentum,
                              float eps) {
  const int lane = threadIdx.x & 31;
  const int c = (int)(blockIdx.x * (kColThreads / 32) + (threadIdx.x >> 5));
  if (c >= bn.C) return;
  const float2 tot = collect_partials(sh, bn, partial, c, lane);
  if (lane == 0)
    finish_channel<T>(tot, sh.N, bn.HW, c, x, running_mean, running_var, save_mean, save_invstd, momentum, eps);
}

// ------------------------------------------------------------------ statistics by themselves
// Statistics and group ranges for the entry point that returns only these: maps of at least a group, whole octets and
// samples of whole groups.  The work of a warp is the same R = min(8, HW / 256) consecutive groups of every sample of
// its split: no more than two channels, and which of them an element belongs to does not change from sample to
// sample.  Sums are closed once a sample: eight elements of a row, the rows, the lanes, then a partial sum per
// channel, added up below in a fixed order.  So no chain of additions grows with the number of elements a warp
// happens to get, and the result does not depend on the number of SMs.  (Accumulators carried down all samples of a
// split, as in the kernel above, cost the variance of 1024 x 256 x 56 x 56 a root mean square error of 8.5e-7, against 2.1e-7.)
// Bound by instruction issue (69 instructions a group and warp at R = 8, 87 at R = 3).  us, both launches, float16: tasks
// strided over by persistent warps, both channels' sums kept for every octet -> this; in brackets sums down the samples:
// 256 x 64 x 56 x 56 29.2 -> 28.0 (25.3), 256 x 512 x 28 x 28 71.0 -> 52.3 (41.3), 256 x 128 x 28 x 28 24.9 -> 19.9 (16.9),
// 128 x 256 x 16 x 16 18.7 -> 12.8 (12.6); one task of one group a warp there: 20.8.
struct StatShape {
  int N, C, HW, G;
  int R, T;           // groups per task, tasks per sample
  int M, U;           // tasks a warp takes together, units of that per sample
  int step;           // groups loaded at a time
  int S, spp;         // splits of the samples, samples per split
};

constexpr int kStatRowsMax = 8;

// M: four tasks of a group, two of two groups, or one of more; STEP: groups loaded at a time, three or four.
template <typename T, int M, int STEP>
__global__ void __launch_bounds__(kColThreads, sizeof(T) == 2 ? 3 : 2)
bn_stats_minimax_kernel(const T* __restrict__ x, StatShape sh, T* __restrict__ mn, T* __restrict__ mx,
                        float4* __restrict__ partial) {
  const int lane = threadIdx.x & 31;
  const uint32_t warp = blockIdx.x * (kColThreads / 32) + __shfl_sync(kFull, threadIdx.x >> 5, 0);
  const int split = (int)(warp / (uint32_t)sh.U), u = (int)(warp - (uint32_t)split * (uint32_t)sh.U);
  if (split >= sh.S) return;
  const int n0 = split * sh.spp, n1 = min(sh.N, n0 + sh.spp);
  const int row0 = u * (M * sh.R), rows = min(M * sh.R, sh.G - row0);
  const int64_t F = (int64_t)sh.G * kGroup;
  int other[M];                    // the lane's rows of the task from which on its elements are the second channel's
  float neg0[M], neg1[M];          // shifts: the channels' first elements
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const uint32_t e0 = (uint32_t)(row0 + m * sh.R) * kGroup, c0 = e0 / (uint32_t)sh.HW;
    const int left = (int)min((c0 + 1) * (int64_t)sh.HW - e0, (int64_t)kStatRowsMax * kGroup);
    other[m] = (left - lane * kOct + kGroup - 1) / kGroup;                       // HW % 8 == 0: whole octets
    neg0[m] = c0 < (uint32_t)sh.C ? -load_scalar<T>(x, (int64_t)c0 * sh.HW) : 0.f;
    neg1[m] = c0 + 1 < (uint32_t)sh.C ? -load_scalar<T>(x, (int64_t)(c0 + 1) * sh.HW) : 0.f;
  }
  auto task = [](int i) { return i * M / kBundle; };                             // of row i of a bundle
  auto second = [&](int r0, int i) { return (M == 1 ? r0 + i : i % (kBundle / M)) >= other[task(i)]; };
  // a row past the end reads as zeros with a shift of zero and adds nothing
  auto shift = [&](int r0, int i) { return r0 + i >= rows ? 0.f : second(r0, i) ? neg1[task(i)] : neg0[task(i)]; };
  auto load = [&](Oct<T> (&v)[kBundle], const T* p, int r0) {
#pragma unroll
    for (int i = 0; i < STEP; ++i) v[i] = r0 + i < rows ? load_oct<T>(p + (r0 + i) * kGroup) : zero_oct<T>();
  };
  // the samples from the last to the first: the pack starts with what is read here last
  const T* p = x + (n1 - 1) * F + (int64_t)row0 * kGroup + lane * kOct;
  int64_t q0 = (int64_t)(n1 - 1) * sh.G + row0 + lane;
  float* dst = reinterpret_cast<float*>(partial + (int64_t)(n1 - 1) * sh.T + u * M) + (lane >> 3);
  Oct<T> next[kBundle];
#pragma unroll
  for (int i = 0; i < kBundle; ++i) next[i] = zero_oct<T>();
  load(next, p, 0);
  for (int n = n1 - 1; n >= n0; --n) {
    float2 a0[M], a1[M];           // (sum, sum of squares) of a task's two channels
#pragma unroll
    for (int m = 0; m < M; ++m) a0[m] = a1[m] = both(0.f);
    for (int r0 = 0; r0 < rows; r0 += STEP) {
      Oct<T> v[kBundle];
#pragma unroll
      for (int i = 0; i < kBundle; ++i) v[i] = next[i];
      if (M == 1 && r0 + STEP < rows) {
        load(next, p, r0 + STEP);
      } else if (n > n0) {
        p -= F;
        load(next, p, 0);
      }
      float lo = 0.f, hi = 0.f;
      bundle_minmax<T, STEP>(v, lane, lo, hi);
      if (lane < min(STEP, rows - r0)) {
        store_scalar<T>(mn, q0 + r0, lo);
        store_scalar<T>(mx, q0 + r0, hi);
      }
      auto add_row = [&](int i, float2 row) {
        const bool other_channel = second(r0, i);
        a0[task(i)] = add2(a0[task(i)], other_channel ? both(0.f) : row);
        a1[task(i)] = add2(a1[task(i)], other_channel ? row : both(0.f));
      };
#pragma unroll
      for (int i = 0; i + 1 < STEP; i += 2) {                   // two rows, one in each half of a pair
        const float na = shift(r0, i), nb = shift(r0, i + 1);
        float2 s = both(0.f), q = both(0.f);
#pragma unroll
        for (int e = 0; e < kOct; ++e) {
          const float2 d = make_float2(octet_plus<T>(v[i], e, na), octet_plus<T>(v[i + 1], e, nb));
          s = add2(s, d);
          q = fma2(d, d, q);
        }
        add_row(i, make_float2(s.x, q.x));
        add_row(i + 1, make_float2(s.y, q.y));
      }
      if constexpr (STEP % 2) {
        const float na = shift(r0, STEP - 1);
        float s = 0.f, q = 0.f;
#pragma unroll
        for (int e = 0; e < kOct; ++e) {
          const float d = octet_plus<T>(v[STEP - 1], e, na);
          s += d;
          q = fmaf(d, d, q);
        }
        add_row(STEP - 1, make_float2(s, q));
      }
    }
    // the four sums over the warp: halves of it specialise on a channel, then quarters on sum or sum of squares;
    // lanes 0, 8, 16, 24 end with them
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const bool hi16 = lane & 16, hi8 = lane & 8;
      const float2 keep = hi16 ? a1[m] : a0[m], give = hi16 ? a0[m] : a1[m];
      const float a = keep.x + __shfl_xor_sync(kFull, give.x, 16);
      const float b = keep.y + __shfl_xor_sync(kFull, give.y, 16);
      float t = (hi8 ? b : a) + __shfl_xor_sync(kFull, hi8 ? a : b, 8);
      t += __shfl_xor_sync(kFull, t, 4);
      t += __shfl_xor_sync(kFull, t, 2);
      t += __shfl_xor_sync(kFull, t, 1);
      if ((lane & 7) == 0 && (M == 1 || m * sh.R < rows)) dst[4 * m] = t;
    }
    q0 -= sh.G;
    dst -= 4 * (int64_t)sh.T;
  }
}

// One block per channel: adds the partial sums of every task that touches it, sample after sample and task after task.
template <typename T>
__global__ void __launch_bounds__(kColThreads)
bn_stats_finish_kernel(const float4* __restrict__ partial, StatShape sh, const T* __restrict__ x,
                       float* __restrict__ running_mean, float* __restrict__ running_var, float* __restrict__ save_mean,
                       float* __restrict__ save_invstd, float momentum, float eps) {
  const int c = blockIdx.x;
  const uint32_t span = (uint32_t)sh.R * kGroup, hw = (uint32_t)sh.HW;
  const uint32_t first = (uint32_t)c * hw, last = first + hw - 1;
  const int j_lo = (int)(first / span), j_hi = min((int)(last / span), sh.T - 1);
  const int lo_is_second = (uint32_t)j_lo * span < first;       // only the first task can begin in the channel before
  float sum = 0.f, sq = 0.f;
  for (int n = threadIdx.x; n < sh.N; n += kColThreads) {
    for (int j = j_lo; j <= j_hi; ++j) {
      const float4 p = __ldg(partial + (int64_t)n * sh.T + j);
      const bool second = j == j_lo && lo_is_second;
      sum += second ? p.z : p.x;
      sq += second ? p.w : p.y;
    }
  }
  const float2 tot = block_sum2<kColThreads>(sum, sq);
  if (threadIdx.x == 0)
    finish_channel<T>(tot, sh.N, sh.HW, c, x, running_mean, running_var, save_mean, save_invstd, momentum, eps);
}

// ------------------------------------------------------------------ pack and normalise
template <typename T, typename ST, int SUB, bool PHILOX, bool EDGE>
__global__ void __launch_bounds__(kColThreads, kBnBlocks)
bn_column_pack_kernel(const T* __restrict__ x, ColumnShape sh, BnColumns bn, const T* __restrict__ mn,
                      const T* __restrict__ mx, const int32_t* __restrict__ bits,
                      const int64_t* __restrict__ word_offsets, int32_t* __restrict__ packed, ST* __restrict__ scale,
                      ST* __restrict__ mn_out, const NoiseKey key, const float* __restrict__ mean,
                      const float* __restrict__ invstd, const float* __restrict__ weight,
                      const float* __restrict__ bias, T* __restrict__ y, bool ahead) {
  constexpr int NS = Slots<SUB>::N;
  const int lane = threadIdx.x & 31;
  const ColumnTask t = column_task(sh);
  if (!t.valid) return;
  const ColumnOctets<EDGE> oct(sh, t, lane);
  const ColumnChannels<SUB> cc(sh, bn, t, lane);
  float neg_mean[kBundle][NS], slope[kBundle][NS], shift[kBundle][NS];
#pragma unroll
  for (int gi = 0; gi < kBundle; ++gi) {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const int c = min(cc.ch[gi][s], bn.C - 1);       // elements past the sample are never stored
      neg_mean[gi][s] = -__ldg(mean + c);
      slope[gi][s] = __ldg(invstd + c) * (weight ? __ldg(weight + c) : 1.f);
      shift[gi][s] = bias ? __ldg(bias + c) : 0.f;
    }
  }
  pack_column<T, ST, PHILOX>(
      x, sh, t, oct, mn, mx, bits, word_offsets, packed, scale, mn_out, (const T*)nullptr, key, lane,
      PHILOX && sizeof(T) == 2 && ahead,
      [&](int n, const Oct<T> (&v)[kBundle]) {
        T* sample = y + (int64_t)n * sh.F;
#pragma unroll
        for (int gi = 0; gi < kBundle; ++gi) {
          Oct<T> r;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if constexpr (SUB != 1) {
              const int s = SUB == 8 ? 0 : k / 2;
              const float2 d = octet_pair_plus<T>(v[gi], k, neg_mean[gi][s], neg_mean[gi][s]);
              set_octet_pair<T>(r, k, fma2(d, both(slope[gi][s]), both(shift[gi][s])));
            } else {
              const int a = cc.second(gi, 2 * k) ? 1 : 0, b = cc.second(gi, 2 * k + 1) ? 1 : 0;
              const float2 d = octet_pair_plus<T>(v[gi], k, a ? neg_mean[gi][1] : neg_mean[gi][0], b ? neg_mean[gi][1] : neg_mean[gi][0]);
              set_octet_pair<T>(r, k, make_float2(fmaf(d.x, a ? slope[gi][1] : slope[gi][0], a ? shift[gi][1] : shift[gi][0]),
                                                  fmaf(d.y, b ? slope[gi][1] : slope[gi][0], b ? shift[gi][1] : shift[gi][0])));
            }
          }
          oct.template store<T>(sample, gi, r);
        }
      });
}

// ------------------------------------------------------------------ backward
// EDGE: samples that are not whole groups, or octets off their natural alignment.
template <typename T, typename ST, int SUB, bool EDGE>
__global__ void __launch_bounds__(kColThreads, kBnBlocks)
bn_codes_reduce_kernel(const int32_t* __restrict__ packed, const int32_t* __restrict__ bits,
                       const int64_t* __restrict__ word_offsets, const ST* __restrict__ scale,
                       const ST* __restrict__ mn, const T* __restrict__ dy, ColumnShape sh, BnColumns bn,
                       const float* __restrict__ save_mean, float2* __restrict__ partial) {
  constexpr int NS = Slots<SUB>::N;
  const int lane = threadIdx.x & 31;
  const ColumnTask t = column_task(sh);
  if (!t.valid) return;
  const ColumnChannels<SUB> cc(sh, bn, t, lane);
  const TransposePlan plan = make_transpose_plan(lane);
  const WordOrder<T> order(lane);
  float neg_mean[kBundle][NS];
  float2 sg[kBundle][NS], sgx[kBundle][NS];
#pragma unroll
  for (int gi = 0; gi < kBundle; ++gi) {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      neg_mean[gi][s] = cc.ch[gi][s] < bn.C ? -__ldg(save_mean + cc.ch[gi][s]) : 0.f;
      sg[gi][s] = sgx[gi][s] = both(0.f);
    }
  }
  auto add = [&](int gi, const Oct<T>& x, const Oct<T>& g) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 vg = octet_pair<T>(g, k);
      if constexpr (SUB != 1) {
        const int s = SUB == 8 ? 0 : k / 2;
        sg[gi][s] = add2(sg[gi][s], vg);
        sgx[gi][s] = fma2(vg, octet_pair_plus<T>(x, k, neg_mean[gi][s], neg_mean[gi][s]), sgx[gi][s]);
      } else {
        const bool s0 = cc.second(gi, 2 * k), s1 = cc.second(gi, 2 * k + 1);
        const float2 d = octet_pair_plus<T>(x, k, neg_mean[gi][s0 ? 1 : 0], neg_mean[gi][s1 ? 1 : 0]);
        const float p0 = vg.x * d.x, p1 = vg.y * d.y;
        sg[gi][0].x += s0 ? 0.f : vg.x; sg[gi][0].y += s1 ? 0.f : vg.y;
        sg[gi][1].x += s0 ? vg.x : 0.f; sg[gi][1].y += s1 ? vg.y : 0.f;
        sgx[gi][0].x += s0 ? 0.f : p0; sgx[gi][0].y += s1 ? 0.f : p1;
        sgx[gi][1].x += s0 ? p0 : 0.f; sgx[gi][1].y += s1 ? p1 : 0.f;
      }
    }
  };
  const ColumnOctets<EDGE> oct(sh, t, lane);
  for (int nb = t.n0; nb < t.n1; nb += 32) {
    const int nl = min(32, t.n1 - nb);
    ColumnStream st;
    st.open(t, nb + lane, lane < nl, bits, word_offsets);
    BundleWords next = st.fetch<T, ST>(t, order, sh.G, nb, 0, packed, scale, mn, lane);
    for (int i = 0; i < nl; ++i) {
      const BundleWords cur = next;
      Oct<T> g[kBundle];
      oct.template load<T>(dy + (int64_t)(nb + i) * sh.F, g);
      if (i + 1 < nl) next = st.fetch<T, ST>(t, order, sh.G, nb + i + 1, i + 1, packed, scale, mn, lane);
      decode_column<T>(cur, t.count, plan, lane, [&](int gi, const Oct<T>& x) { add(gi, x, g[gi]); });
    }
  }
  const int split = t.n0 / sh.spp;
  write_partials<SUB>(cc, sg, sgx, partial + ((int64_t)split * sh.P + t.p) * bn.kmax, lane);
}

// coef[c]: (mean, weight * invstd, sum_dy / M, sum_dy_xmu * invstd^2 / M); one warp per channel.
__global__ void __launch_bounds__(kColThreads)
bn_codes_finish_kernel(const float2* __restrict__ partial, ColumnShape sh, BnColumns bn,
                       const float* __restrict__ weight, const float* __restrict__ save_mean,
                       const float* __restrict__ save_invstd, float* __restrict__ dweight, float* __restrict__ dbias,
                       float4* __restrict__ coef) {
  const int lane = threadIdx.x & 31;
  const int c = (int)(blockIdx.x * (kColThreads / 32) + (threadIdx.x >> 5));
  if (c >= bn.C) return;
  const float2 tot = collect_partials(sh, bn, partial, c, lane);
  if (lane != 0) return;
  const float M = (float)sh.N * (float)bn.HW, invstd = save_invstd[c];
  if (dbias) dbias[c] = tot.x;
  if (dweight) dweight[c] = tot.y * invstd;
  coef[c] = make_float4(save_mean[c], (weight ? weight[c] : 1.f) * invstd, tot.x / M, tot.y * invstd * invstd / M);
}

template <typename T, typename ST, int SUB, bool EDGE>
__global__ void __launch_bounds__(kColThreads, kBnBlocks)
bn_codes_apply_kernel(const int32_t* __restrict__ packed, const int32_t* __restrict__ bits,
                      const int64_t* __restrict__ word_offsets, const ST* __restrict__ scale,
                      const ST* __restrict__ mn, const T* __restrict__ dy, T* __restrict__ dx, ColumnShape sh,
                      BnColumns bn, const float4* __restrict__ coef) {
  constexpr int NS = Slots<SUB>::N;
  const int lane = threadIdx.x & 31;
  const ColumnTask t = column_task(sh);
  if (!t.valid) return;
  const ColumnOctets<EDGE> oct(sh, t, lane);
  const ColumnChannels<SUB> cc(sh, bn, t, lane);
  const TransposePlan plan = make_transpose_plan(lane);
  const WordOrder<T> order(lane);
  float4 kf[kBundle][NS];                              // (-mean, weight * invstd, -mean_dy, -q)
#pragma unroll
  for (int gi = 0; gi < kBundle; ++gi) {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const float4 k = cc.ch[gi][s] < bn.C ? __ldg(coef + cc.ch[gi][s]) : make_float4(0.f, 0.f, 0.f, 0.f);
      kf[gi][s] = make_float4(-k.x, k.y, -k.z, -k.w);
    }
  }
  auto gradient = [&](int gi, const Oct<T>& x, const Oct<T>& g) {
    Oct<T> r;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if constexpr (SUB != 1) {
        const float4 c = kf[gi][SUB == 8 ? 0 : k / 2];
        const float2 d = fma2(octet_pair_plus<T>(x, k, c.x, c.x), both(c.w), octet_pair_plus<T>(g, k, c.z, c.z));
        set_octet_pair<T>(r, k, make_float2(c.y * d.x, c.y * d.y));
      } else {
        const float4 c0 = cc.second(gi, 2 * k) ? kf[gi][1] : kf[gi][0];
        const float4 c1 = cc.second(gi, 2 * k + 1) ? kf[gi][1] : kf[gi][0];
        const float2 vx = octet_pair_plus<T>(x, k, c0.x, c1.x), vg = octet_pair_plus<T>(g, k, c0.z, c1.z);
        set_octet_pair<T>(r, k, make_float2(c0.y * fmaf(vx.x, c0.w, vg.x), c1.y * fmaf(vx.y, c1.w, vg.y)));
      }
    }
    return r;
  };
  // the samples from the last to the first: what the reduce read last is still in the L2
  const int total = t.n1 - t.n0;
  for (int kb = 0; kb < total; kb += 32) {
    const int nl = min(32, total - kb);
    const int top = t.n1 - 1 - kb;
    ColumnStream st;
    st.open(t, top - lane, lane < nl, bits, word_offsets);
    BundleWords next = st.fetch<T, ST>(t, order, sh.G, top, 0, packed, scale, mn, lane);
    for (int i = 0; i < nl; ++i) {
      const BundleWords cur = next;
      Oct<T> g[kBundle];
      oct.template load<T>(dy + (int64_t)(top - i) * sh.F, g);
      if (i + 1 < nl) next = st.fetch<T, ST>(t, order, sh.G, top - i - 1, i + 1, packed, scale, mn, lane);
      T* sample = dx + (int64_t)(top - i) * sh.F;
      decode_column<T>(cur, t.count, plan, lane,
                       [&](int gi, const Oct<T>& x) { oct.template store<T>(sample, gi, gradient(gi, x, g[gi])); });
    }
  }
}

// ------------------------------------------------------------------ host side
bool bn_columns_supported(int64_t N, int64_t C, int64_t HW) {
  if (N <= 0 || C <= 0 || HW < kOct || C > 0x7fffffff || HW > 0x7fffffff) return false;
  return C * HW < ((int64_t)1 << 31) - kBundle * kGroup && column_supported(N, C * HW);
}
BnColumns bn_columns(int64_t C, int64_t HW) {
  BnColumns bn;
  bn.C = (int)C;
  bn.HW = (int)HW;
  bn.kmax = (int)((kBundle * kGroup - 1) / HW + 2);
  return bn;
}
constexpr int kBnWarps = kBnBlocks * kColThreads / 32;       // resident warps per SM
int64_t bn_partial_bytes(const ColumnShape& sh, const BnColumns& bn) {
  return ((int64_t)sh.P * sh.S * bn.kmax * (int64_t)sizeof(float2) + 255) / 256 * 256;
}
int64_t bn_coef_bytes(int64_t C) { return (C * (int64_t)sizeof(float4) + 255) / 256 * 256; }

ColumnShape bn_stats_shape(int64_t N, int64_t C, int64_t HW, int align, int elem_size) {
  return column_shape(N, C * HW, align, bn_stats_blocks(elem_size, HW % 8 == 0 ? 8 : 4) * kColThreads / 32);
}
struct BnForward {
  const void *group_mn, *group_mx;
  unsigned* ticket;
  const float *weight, *bias;
  float *running_mean, *running_var, *save_mean, *save_invstd;
  int32_t *packed, *bits;
  void *scale, *mn_out;
  int64_t* word_offsets;
  float* C;
  float momentum, eps, range_factor;
  int initial_bits, stochastic;
  double target;
  uint64_t seed, offset;
};
int64_t bn_range_bytes(int64_t N, int64_t F, int elem_size) {
  return (N * ((F + kGroup - 1) / kGroup) * elem_size + 255) / 256 * 256;
}

template <typename T, int SUB, bool EDGE>
int launch_stats(const T* x, T* mn, T* mx, float* running_mean, float* running_var, float* save_mean, float* save_invstd,
                 float momentum, float eps, const ColumnShape& sh, const BnColumns& bn, float2* partial, cudaStream_t s) {
  bn_column_stats_kernel<T, SUB, EDGE><<<column_grid(sh), kColThreads, 0, s>>>(x, sh, bn, mn, mx, partial);
  if (int st = check_launch()) return st;
  bn_column_stats_finish_kernel<T><<<(bn.C + kColThreads / 32 - 1) / (kColThreads / 32), kColThreads, 0, s>>>(
      partial, sh, bn, x, running_mean, running_var, save_mean, save_invstd, momentum, eps);
  return check_launch();
}

template <typename T, typename ST, int SUB, bool EDGE>
int launch_forward(const void* x, void* y, const BnForward& f, const ColumnShape& stats, const ColumnShape& sh,
                   const BnColumns& bn, void* workspace, cudaStream_t s) {
  const T *mn = (const T*)f.group_mn, *mx = (const T*)f.group_mx;
  if (!mn) {                                           // else ranges and statistics come from a pass before this call
    T* own_mn = (T*)((char*)workspace + bn_partial_bytes(stats, bn));
    T* own_mx = (T*)((char*)own_mn + bn_range_bytes(sh.N, sh.F, sizeof(T)));
    if (int st = launch_stats<T, SUB, EDGE>((const T*)x, own_mn, own_mx, f.running_mean, f.running_var, f.save_mean,
                                            f.save_invstd, f.momentum, f.eps, stats, bn, (float2*)workspace, s))
      return st;
    mn = own_mn;
    mx = own_mx;
  }
  if (range_greedy_supported(sh.N, f.initial_bits)) {
    if (int st = range_greedy_impl(mn, mx, sh.N, sh.G, DType<T>::id, f.range_factor, 1.f, nullptr, f.C, f.ticket,
                                   f.initial_bits, f.target, f.bits, f.word_offsets, kGroup, s))
      return st;
  } else {
    if (int st = actnn_range_sqr(mn, mx, sh.N, sh.G, DType<T>::id, f.range_factor, 1.f, nullptr, f.C, s)) return st;
    if (int st = actnn_calc_precision(f.C, nullptr, sh.N, f.initial_bits, f.target, f.bits, f.word_offsets, sh.G, kGroup,
                                      nullptr, 0, s))
      return st;
  }
  auto pack = f.stochastic ? bn_column_pack_kernel<T, ST, SUB, true, EDGE> : bn_column_pack_kernel<T, ST, SUB, false, EDGE>;
  // Large 16-bit activations: requested into the L2 a sample ahead of the loads, while y goes out.  The line lies between
  // the sizes that were measured, 15 MB and 40 MB.  The kernels of float32 and of rounding to nearest are compiled without it:
  // its branch alone cost 512 x 256 x 28 x 28 of float32 240 -> 250 us (whole pass), and rounding to nearest 123.7 -> 126.5.
  // float16 256 x 64 x 56 x 56 41.5 -> 37.6 us (two samples ahead 38.0, three 38.3), 256 x 128 x 28 x 28 21.8 -> 19.8, 200 x
  // 64 x 40 x 40 18.1 -> 16.8; at 15 MB (64 x 100 x 35 x 35) 19.3 -> 19.6, and float32 pays: 76.5 -> 80.
  const bool ahead = sizeof(T) == 2 && (int64_t)sh.N * sh.F >= ((int64_t)16 << 20);
  pack<<<column_grid(sh), kColThreads, 0, s>>>((const T*)x, sh, bn, mn, mx, f.bits, f.word_offsets, f.packed,
                                               (ST*)f.scale, (ST*)f.mn_out, make_noise_key(f.seed, f.offset), f.save_mean,
                                               f.save_invstd, f.weight, f.bias, (T*)y, ahead);
  return check_launch();
}

template <typename T, typename ST, int SUB, bool EDGE>
int launch_backward(const int32_t* packed, const int32_t* bits, const int64_t* word_offsets, const void* scale,
                    const void* mn, const void* dy, const float* weight, const float* save_mean,
                    const float* save_invstd, void* dx, float* dweight, float* dbias, const ColumnShape& sh,
                    const BnColumns& bn, void* workspace, cudaStream_t s) {
  float4* coef = (float4*)workspace;
  float2* partial = (float2*)((char*)workspace + bn_coef_bytes(bn.C));
  bn_codes_reduce_kernel<T, ST, SUB, EDGE><<<column_grid(sh), kColThreads, 0, s>>>(
      packed, bits, word_offsets, (const ST*)scale, (const ST*)mn, (const T*)dy, sh, bn, save_mean, partial);
  if (int st = check_launch()) return st;
  bn_codes_finish_kernel<<<(bn.C + kColThreads / 32 - 1) / (kColThreads / 32), kColThreads, 0, s>>>(
      partial, sh, bn, weight, save_mean, save_invstd, dweight, dbias, coef);
  if (int st = check_launch()) return st;
  bn_codes_apply_kernel<T, ST, SUB, EDGE><<<column_grid(sh), kColThreads, 0, s>>>(
      packed, bits, word_offsets, (const ST*)scale, (const ST*)mn, (const T*)dy, (T*)dx, sh, bn, coef);
  return check_launch();
}

}  // namespace
}  // namespace actnn

using namespace actnn;

extern "C" int actnn_batch_norm_codes_workspace(int64_t N, int64_t C, int64_t HW, int dtype, int64_t* bytes) {
  if (!bytes) return ACTNN_ERR_NULL;
  if (dtype < ACTNN_F32 || dtype > ACTNN_BF16) return ACTNN_ERR_DTYPE;
  if (!bn_columns_supported(N, C, HW)) return ACTNN_ERR_SHAPE;
  const ColumnShape sh = column_shape(N, C * HW, kOct, kBnWarps);
  const BnColumns bn = bn_columns(C, HW);
  const ColumnShape stats = bn_stats_shape(N, C, HW, kOct, dtype_size(dtype));
  *bytes = bn_coef_bytes(C) + max(bn_partial_bytes(sh, bn), bn_partial_bytes(stats, bn)) +
           2 * bn_range_bytes(N, C * HW, dtype_size(dtype));                       // ranges: forward only
  return ACTNN_OK;
}

// The statistics pass by itself.
static bool stats_minimax_shape(int64_t N, int64_t C, int64_t HW, StatShape& sh) {
  constexpr int64_t k31 = (int64_t)1 << 31;
  if (N <= 0 || C <= 0 || N >= k31 || C >= k31 || HW >= k31 || HW < kGroup || HW % kOct != 0 || N * C >= k31 ||
      N * C * HW >= ((int64_t)1 << 40) || C * HW % kGroup != 0 || C * HW >= 2 * k31 - kStatRowsMax * kGroup)
    return false;
  sh.N = (int)N;
  sh.C = (int)C;
  sh.HW = (int)HW;
  sh.G = (int)(C * HW / kGroup);
  sh.R = (int)min((int64_t)kStatRowsMax, HW / kGroup);
  sh.T = (sh.G + sh.R - 1) / sh.R;
  sh.M = sh.R <= 2 ? kBundle / sh.R : 1;
  sh.U = (sh.T + sh.M - 1) / sh.M;
  const int rows = sh.M * sh.R, steps = (rows + kBundle - 1) / kBundle;
  sh.step = (rows + steps - 1) / steps;
  return true;
}
static int64_t stats_minimax_bytes(const StatShape& sh) {
  return ((int64_t)sh.N * sh.T * (int64_t)sizeof(float4) + 255) / 256 * 256;
}

extern "C" int64_t actnn_batch_norm_stats_minimax_workspace(int64_t N, int64_t C, int64_t HW) {
  StatShape sh;
  return stats_minimax_shape(N, C, HW, sh) ? stats_minimax_bytes(sh) : -1;
}

extern "C" int actnn_batch_norm_stats_minimax(const void* x, void* mn, void* mx, const float* weight, const float* bias,
                                              float* running_mean, float* running_var, float* save_mean,
                                              float* save_invstd, int64_t N, int64_t C, int64_t HW, double momentum,
                                              double eps, int dtype, void* workspace, int64_t workspace_bytes,
                                              actnn_stream_t stream) {
  (void)weight;
  (void)bias;
  if (dtype < ACTNN_F32 || dtype > ACTNN_BF16) return ACTNN_ERR_DTYPE;
  StatShape sh;
  if (!stats_minimax_shape(N, C, HW, sh)) return ACTNN_ERR_SHAPE;
  if (!x || !mn || !mx || !save_mean || !save_invstd || !workspace) return ACTNN_ERR_NULL;
  if (workspace_bytes < stats_minimax_bytes(sh)) return ACTNN_ERR_CAPACITY;
  if (!aligned(x, dtype == ACTNN_F32 ? 32 : 16) || !aligned(workspace, 16)) return ACTNN_ERR_ALIGN;
  const SampleSplits splits = split_samples(N, sh.U, (dtype == ACTNN_F32 ? 2 : 3) * kColThreads / 32);
  sh.S = splits.S;
  sh.spp = splits.spp;
  const int grid = (int)(((int64_t)sh.U * sh.S + kColThreads / 32 - 1) / (kColThreads / 32));
  cudaStream_t s = (cudaStream_t)stream;
#define ACTNN_STATS(T)                                                                                              \
  {                                                                                                                 \
    auto kernel = sh.M == 4 ? bn_stats_minimax_kernel<T, 4, 4>                                                      \
                            : sh.M == 2 ? bn_stats_minimax_kernel<T, 2, 4>                                          \
                                        : sh.step == 4 ? bn_stats_minimax_kernel<T, 1, 4>                           \
                                                       : bn_stats_minimax_kernel<T, 1, 3>;                          \
    kernel<<<grid, kColThreads, 0, s>>>((const T*)x, sh, (T*)mn, (T*)mx, (float4*)workspace);                       \
    if (int st = check_launch()) return st;                                                                         \
    bn_stats_finish_kernel<T><<<sh.C, kColThreads, 0, s>>>((const float4*)workspace, sh, (const T*)x, running_mean, \
                                                           running_var, save_mean, save_invstd, (float)momentum,    \
                                                           (float)eps);                                             \
    return check_launch();                                                                                          \
  }
  switch (dtype) {
    case ACTNN_F32: ACTNN_STATS(float)
    case ACTNN_F16: ACTNN_STATS(__half)
    default: ACTNN_STATS(__nv_bfloat16)
  }
#undef ACTNN_STATS
}

extern "C" int actnn_batch_norm_codes_forward(const void* x, const void* group_mn, const void* group_mx,
                                              const float* weight, const float* bias, float* running_mean, float* running_var,
                                              void* y, float* save_mean,
                                              float* save_invstd, int32_t* packed, void* scale, void* mn_out,
                                              int32_t* bits_out, int64_t* word_offsets_out, float* C_out, int64_t N,
                                              int64_t C, int64_t HW, double momentum, double eps, int dtype,
                                              int stat_dtype, float range_factor, int initial_bits, double target,
                                              int stochastic, uint64_t seed, uint64_t offset, void* ticket,
                                              void* workspace, int64_t workspace_bytes, actnn_stream_t stream) {
  if (dtype < ACTNN_F32 || dtype > ACTNN_BF16) return ACTNN_ERR_DTYPE;
  if (stat_dtype != (dtype == ACTNN_F32 ? ACTNN_BF16 : dtype)) return ACTNN_ERR_DTYPE;
  if (initial_bits < 1 || initial_bits > 8) return ACTNN_ERR_BITS;
  if (!(target == target)) return ACTNN_ERR_ARG;
  if (!bn_columns_supported(N, C, HW)) return ACTNN_ERR_SHAPE;
  if (!x || !y || !save_mean || !save_invstd || !packed || !scale || !mn_out || !bits_out || !word_offsets_out ||
      !C_out || !ticket || !workspace || (!group_mn != !group_mx))
    return ACTNN_ERR_NULL;
  const int es = dtype_size(dtype);
  const int64_t F = C * HW;
  // whole groups want vector alignment, as in the codec's own entries
  if (!aligned(x, F % kGroup == 0 ? es * kOct : es) || !aligned(y, es) || !aligned(packed, 4) || !aligned(workspace, 256))
    return ACTNN_ERR_ALIGN;
  const int al = min(octet_alignment(x, F, es), octet_alignment(y, F, es));
  const ColumnShape sh = column_shape(N, F, al, kBnWarps);
  const BnColumns bn = bn_columns(C, HW);
  const ColumnShape stats = bn_stats_shape(N, C, HW, al, es);
  if (!group_mn && workspace_bytes < bn_partial_bytes(stats, bn) + 2 * bn_range_bytes(N, F, es))
    return ACTNN_ERR_CAPACITY;
  const BnForward f{group_mn, group_mx, (unsigned*)ticket, weight, bias, running_mean, running_var, save_mean,
                    save_invstd, packed, bits_out, scale, mn_out, word_offsets_out, C_out, (float)momentum, (float)eps,
                    range_factor, initial_bits, stochastic, target, seed, offset};
  cudaStream_t s = (cudaStream_t)stream;
  const bool edge = al != kOct || F % kGroup != 0;
#define ACTNN_FWD(T, ST, SUB, EDGE) return launch_forward<T, ST, SUB, EDGE>(x, y, f, stats, sh, bn, workspace, s)
#define ACTNN_FWD_T(T, ST)                                  \
  {                                                         \
    if (HW % 8 == 0) {                                      \
      if (edge) ACTNN_FWD(T, ST, 8, true);                  \
      ACTNN_FWD(T, ST, 8, false);                           \
    }                                                       \
    if (HW % 4 == 0) {                                      \
      if (edge) ACTNN_FWD(T, ST, 4, true);                  \
      ACTNN_FWD(T, ST, 4, false);                           \
    }                                                       \
    ACTNN_FWD(T, ST, 1, true);                              \
  }
  switch (dtype) {
    case ACTNN_F16: ACTNN_FWD_T(__half, __half)
    case ACTNN_BF16: ACTNN_FWD_T(__nv_bfloat16, __nv_bfloat16)
    default: ACTNN_FWD_T(float, __nv_bfloat16)
  }
#undef ACTNN_FWD_T
#undef ACTNN_FWD
}

extern "C" int actnn_batch_norm_codes_backward(const int32_t* packed, const int32_t* bits, const int64_t* word_offsets,
                                               const void* scale, const void* mn, const void* grad_out,
                                               const float* weight, const float* save_mean, const float* save_invstd,
                                               void* grad_in, float* grad_weight, float* grad_bias, int64_t N,
                                               int64_t C, int64_t HW, int dtype, int stat_dtype, void* workspace,
                                               int64_t workspace_bytes, actnn_stream_t stream) {
  if (dtype < ACTNN_F32 || dtype > ACTNN_BF16) return ACTNN_ERR_DTYPE;
  if (stat_dtype != (dtype == ACTNN_F32 ? ACTNN_BF16 : dtype)) return ACTNN_ERR_DTYPE;
  if (!bn_columns_supported(N, C, HW)) return ACTNN_ERR_SHAPE;
  if (!packed || !bits || !word_offsets || !scale || !mn || !grad_out || !save_mean || !save_invstd || !grad_in ||
      !workspace)
    return ACTNN_ERR_NULL;
  const int es = dtype_size(dtype);
  const int64_t F = C * HW;
  const int al = min(octet_alignment(grad_out, F, es), octet_alignment(grad_in, F, es));
  if (!aligned(grad_out, es) || !aligned(grad_in, es) || !aligned(packed, 4) || !aligned(workspace, 16))
    return ACTNN_ERR_ALIGN;
  const ColumnShape sh = column_shape(N, F, al, kBnWarps);
  const BnColumns bn = bn_columns(C, HW);
  if (workspace_bytes < bn_coef_bytes(C) + bn_partial_bytes(sh, bn)) return ACTNN_ERR_CAPACITY;
  cudaStream_t s = (cudaStream_t)stream;
  const bool edge = al != kOct || F % kGroup != 0;
#define ACTNN_BWD(T, ST, SUB, EDGE)                                                                                 \
  return launch_backward<T, ST, SUB, EDGE>(packed, bits, word_offsets, scale, mn, grad_out, weight, save_mean,      \
                                           save_invstd, grad_in, grad_weight, grad_bias, sh, bn, workspace, s)
#define ACTNN_BWD_T(T, ST)                                  \
  {                                                         \
    if (HW % 8 == 0) {                                      \
      if (edge) ACTNN_BWD(T, ST, 8, true);                  \
      ACTNN_BWD(T, ST, 8, false);                           \
    }                                                       \
    if (HW % 4 == 0) {                                      \
      if (edge) ACTNN_BWD(T, ST, 4, true);                  \
      ACTNN_BWD(T, ST, 4, false);                           \
    }                                                       \
    ACTNN_BWD(T, ST, 1, true);                              \
  }
  switch (dtype) {
    case ACTNN_F16: ACTNN_BWD_T(__half, __half)
    case ACTNN_BF16: ACTNN_BWD_T(__nv_bfloat16, __nv_bfloat16)
    default: ACTNN_BWD_T(float, __nv_bfloat16)
  }
#undef ACTNN_BWD_T
#undef ACTNN_BWD
}
