// Packing runs of four-group bundles in the order of the stream (flat tasks): what the kernels for whole groups and for
// samples of any length share.  A task is up to 32 consecutive groups of the activation, lane l prepares group l of it.
#pragma once

#include "column.cuh"

namespace actnn {
namespace {

constexpr int kFlatGroups = 32;       // groups per task
constexpr int kFlatBundle = 4;        // groups per bundle

// (sample, group) of group q; one 32-bit division where the activation allows it
ACTNN_DEV void split_group_index(int64_t q, int64_t G, int64_t& n, int64_t& r) {
  if (((uint64_t)q | (uint64_t)G) >> 32) { n = q / G; } else { n = (int64_t)((uint32_t)q / (uint32_t)G); }
  r = q - n * G;
}

template <typename T, int B, int MODE, bool CLAMP_LOW>
ACTNN_DEV void pack_flat_bundle(const Oct<T> (&x)[kFlatBundle], const LaneParams<T>& mine, int first_lane,
                                int64_t q, int32_t* __restrict__ out, const T* __restrict__ noise,
                                const NoiseKey& key, const TransposePlan& plan, int lane) {
  constexpr int GPC = NoiseShape<T>::GPC;
  uint32_t S[B];
#pragma unroll
  for (int k = 0; k < B; ++k) S[k] = 0u;
  Oct<T> nzb[GPC];
#pragma unroll
  for (int gi = 0; gi < kFlatBundle; ++gi) {
    const QP<T> qp = fetch_lane_params<T>(mine, first_lane + gi);
    Oct<T> nz;
    if constexpr (MODE == kNoisePhilox) {
      if (gi % GPC == 0) noise_block<T>(key, (uint64_t)(q + gi), lane, nzb);
      nz = nzb[gi % GPC];
    } else if constexpr (MODE == kNoiseTensor) {
      nz = load_oct<T>(noise + (q + gi) * kGroup + lane * kOct);
    } else {
      nz = zero_oct<T>();
    }
    uint32_t lo, hi;
    row_from_magic<T, B>(quantize_oct<T, CLAMP_LOW, B>(x[gi], nz, qp), lo, hi);
    if (gi == 0) put_row<B, 0 * 8 * B>(S, lo, hi);
    if (gi == 1) put_row<B, 1 * 8 * B>(S, lo, hi);
    if (gi == 2) put_row<B, 2 * 8 * B>(S, lo, hi);
    if (gi == 3) put_row<B, 3 * 8 * B>(S, lo, hi);
  }
#pragma unroll
  for (int k = 0; k < B; ++k) out[k * 32 + lane] = (int32_t)warp_transpose32(S[k], plan);
}

// A run: bundles k0 .. k1-1 of a task, all of the same width B (a run ends where the next
// sample has another width).  The width is a template argument here, so the loop over the
// bundles has no dispatch in it and the octets of bundle k+1 are requested before bundle k is
// quantized (two register buffers used alternately; nothing is copied).  `a` already holds the
// octets of bundle k0.  ALIGNED: octets on their natural alignment, else on `align` elements.
template <typename T, int B, int MODE, bool CLAMP_LOW, bool PREFETCH, bool ALIGNED = true>
ACTNN_DEV void pack_flat_run(Oct<T> (&a)[kFlatBundle], Oct<T> (&b)[kFlatBundle], int k0, int k1, int64_t q0,
                             const T* __restrict__ data, const LaneParams<T>& mine, int32_t* __restrict__ out,
                             const T* __restrict__ noise, const NoiseKey& key, const TransposePlan& plan, int lane,
                             int align = kOct) {
  auto load = [&](Oct<T> (&dst)[kFlatBundle], int k) {
#pragma unroll
    for (int gi = 0; gi < kFlatBundle; ++gi)
      dst[gi] = load_octet<T, !ALIGNED>(data + (q0 + k * kFlatBundle + gi) * kGroup + lane * kOct, kOct, align);
  };
  if constexpr (!PREFETCH) {
    for (int k = k0; k < k1; ++k) {
      if (k > k0) load(a, k);
      pack_flat_bundle<T, B, MODE, CLAMP_LOW>(a, mine, k * kFlatBundle, q0 + k * kFlatBundle, out, noise, key, plan,
                                              lane);
      out += 32 * B;                                           // consecutive groups are consecutive in the stream
    }
  } else {
    for (int k = k0; k < k1; k += 2) {
      if (k + 1 < k1) load(b, k + 1);
      pack_flat_bundle<T, B, MODE, CLAMP_LOW>(a, mine, k * kFlatBundle, q0 + k * kFlatBundle, out, noise, key, plan,
                                              lane);
      out += 32 * B;
      if (k + 1 >= k1) break;
      if (k + 2 < k1) load(a, k + 2);
      pack_flat_bundle<T, B, MODE, CLAMP_LOW>(b, mine, (k + 1) * kFlatBundle, q0 + (k + 1) * kFlatBundle, out,
                                              noise, key, plan, lane);
      out += 32 * B;
    }
  }
}

}  // namespace
}  // namespace actnn
