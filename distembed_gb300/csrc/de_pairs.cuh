// The pairs of a work item with its rows' addresses held by the warp's lanes, shared by
// the FP32 plain, SpMM, sparse embedding and BF16 attractive kernels.
#pragma once
#include <cuda_runtime.h>

#include "de_device.cuh"
#include "de_internal.h"

namespace de {
namespace dev {

// Layout of a pair: LP lanes hold a row, C components each, G pairs a warp step and S
// steps' rows in flight.  Lane gl of a pair holds components [4 gl, 4 gl + 4) and, with
// C = 8, [D/2 + 4 gl, D/2 + 4 gl + 4): 128-bit loads, each contiguous over the lanes.
// Below dim 128 a row is too short for a warp; at dim 128 two pairs a step measured
// slower than one (R-MAT of 2^20 vertices, B = 4096: 18.3 against 15.0 us a
// minibatch, at dim 64 11.9 against 12.6, dim 32 9.2 against 11.7).
template <int D>
struct Lay {
  static constexpr int LP = D >= 128 ? 32 : D / 8, G = 32 / LP, C = D / LP;
  static constexpr int S = D == 128 ? 8 : D == 256 ? 4 : 2;
};
// A lane's components of a row.
template <int N>
struct LaneVec {
  float v[N];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int t = 0; t < N; ++t) v[t] = 0.f;
  }
};
template <int D>
using LaneRow = LaneVec<Lay<D>::C>;

// How a row is read: kFinal, rows that no launch in flight writes (read-only path);
// kStaged, rows of minibatch j-1 written by the launch before (L2); kShared, shared
// memory or kFinal rows through generic addresses.
enum RowRead { kFinal, kStaged, kShared };
template <int D, RowRead kRead>
__device__ __forceinline__ void load_lanes(LaneRow<D> &f, const float *row, int gl) {
  const float4 *p = reinterpret_cast<const float4 *>(row) + gl;
#pragma unroll
  for (int h = 0; h < Lay<D>::C / 4; ++h, p += D / 8) {
    const float4 t = kRead == kFinal ? __ldg(p) : kRead == kStaged ? __ldcg(p) : *p;
    f.v[4 * h] = t.x; f.v[4 * h + 1] = t.y; f.v[4 * h + 2] = t.z; f.v[4 * h + 3] = t.w;
  }
}

// Stores of lanes [0, LP), which hold a whole row.
template <int D, bool kCg>
__device__ __forceinline__ void store_lanes(const LaneRow<D> &f, float *row, int lane) {
  if (lane >= Lay<D>::LP) return;
  float4 *p = reinterpret_cast<float4 *>(row) + lane;
#pragma unroll
  for (int h = 0; h < Lay<D>::C / 4; ++h, p += D / 8) {
    const float4 t = make_float4(f.v[4 * h], f.v[4 * h + 1], f.v[4 * h + 2], f.v[4 * h + 3]);
    if constexpr (kCg) __stcg(p, t);
    else *p = t;
  }
}

// The sums of a row's lane groups of LP added up (fixed order), on every lane.
template <int LP, int C>
__device__ __forceinline__ void sum_lane_groups(LaneVec<C> &acc) {
#pragma unroll
  for (int m = LP; m < 32; m <<= 1)
#pragma unroll
    for (int t = 0; t < C; ++t) acc.v[t] += __shfl_xor_sync(kFull, acc.v[t], m);
}
template <int D>
__device__ __forceinline__ void sum_groups(LaneRow<D> &acc) {
  sum_lane_groups<Lay<D>::LP>(acc);
}

// What the pair loops need to know of the rows: the layout above, how a lane's share of
// a row is loaded and kept until it is used (Raw), and how it becomes FP32.
template <int D, RowRead kRead>
struct F32Rows {
  static constexpr int LP = Lay<D>::LP, G = Lay<D>::G, C = Lay<D>::C, S = Lay<D>::S;
  typedef LaneRow<D> Raw;
  static __device__ __forceinline__ void load(Raw &x, const void *row, int gl) {
    load_lanes<D, kRead>(x, static_cast<const float *>(row), gl);
  }
  static __device__ __forceinline__ const LaneVec<C> &unpack(const Raw &x) { return x; }
};
// BF16 rows: 16 bytes (8 components in order) a lane.
template <int D, int kSteps>
struct B16Rows {
  static constexpr int LP = D / 8, G = 32 / LP, C = 8, S = kSteps;
  typedef uint4 Raw;
  static __device__ __forceinline__ void load(Raw &x, const void *row, int gl) {
    x = __ldg(static_cast<const uint4 *>(row) + gl);
  }
  static __device__ __forceinline__ LaneVec<C> unpack(const Raw &x) {
    LaneVec<C> f;
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f.v[2 * i] = __uint_as_float(w[i] << 16);
      f.v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
    return f;
  }
};

// What an item's pairs share.
struct PairCtx {
  float lr, bound, clip_r;
  bool want_loss;
  __device__ __forceinline__ PairCtx(float rate, float max_bound, bool loss)
      : lr(rate), bound(max_bound), want_loss(loss) {
    // |c (x_d - n_d)| <= |c| sqrt(r): 2 sqrt(r) / (1 + r) <= 1 for attraction, less
    // than 2 / sqrt(r) for repulsion.  So the clip (algo.hpp:65-72) is the identity at
    // bound >= 1 and r >= clip_r = 4 / bound^2 (and 3 % more for rounding).
    clip_r = bound >= 1.0f ? 4.12f / (bound * bound) : __int_as_float(0x7f800000);
  }
};

// S steps of pairs [k0, k0 + S G) of a window of 32: lane k of `rows` holds pair k's
// other row.  Bit k of vm: pair k counts, of rm: it counts and repels.  The row of a
// pair that does not count is x_i's own, whose (attractive) force is exactly 0.
// Attractive: c = -2/(1+r); repulsive: c = 2/((r+1e-6)(1+r)) (algo.hpp:573, 626/641).
template <class R, int S>
__device__ __forceinline__ void pair_steps(LaneVec<R::C> &acc, const LaneVec<R::C> &xi, const void *rows, unsigned vm,
                                           unsigned rm, int k0, const PairCtx &c, float &loss, int lane) {
  constexpr int LP = R::LP, G = R::G, C = R::C;
  const int q = G > 1 ? lane / LP : 0, gl = G > 1 ? lane % LP : lane;
  typename R::Raw raw[S];
#pragma unroll
  for (int s = 0; s < S; ++s)
    R::load(raw[s], reinterpret_cast<const void *>(
                        __shfl_sync(kFull, reinterpret_cast<unsigned long long>(rows), k0 + s * G + q)), gl);
  LaneVec<C> x[S];  // x_i - the row
  float r[S];
#pragma unroll
  for (int s = 0; s < S; ++s) {
    x[s] = R::unpack(raw[s]);
    float2 p = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = 0; t < C; t += 2) {
      const float2 d = sub2(make_float2(xi.v[t], xi.v[t + 1]), make_float2(x[s].v[t], x[s].v[t + 1]));
      x[s].v[t] = d.x;
      x[s].v[t + 1] = d.y;
      p = __ffma2_rn(d, d, p);
    }
    r[s] = p.x + p.y;
  }
  bool may_clip = false;
  // coefficient and loss term of pair k at squared distance rr; the term is added on
  // one lane of the pair
  auto coefficient = [&](float rr, int k, bool adds) -> float {
    const bool at = !((rm >> k) & 1u);
    const float one = 1.0f + rr, eps = rr + 1e-6f;
    may_clip |= rr < c.clip_r && (!at || c.bound < 1.0f);
    if (c.want_loss && adds && ((vm >> k) & 1u)) loss += at ? log1pf(rr) : logf(one / eps);
    return __fdividef(at ? -2.0f : 2.0f, at ? one : eps * one);
  };
  float cf[S];
  if constexpr (G == 1) {
    // S sums over the whole warp at once; lane group v holds pair v's
    constexpr int L = Log2<S>::value;
    const float rr = multi_warp_sum<S>(r, lane);
    const int v = (lane >> (5 - L)) & (S - 1);
    const float cv = coefficient(rr, k0 + v, (lane & ((32 >> L) - 1)) == 0);
#pragma unroll
    for (int s = 0; s < S; ++s) cf[s] = __shfl_sync(kFull, cv, s << (5 - L));
  } else {
#pragma unroll
    for (int m = LP / 2; m >= 1; m >>= 1)
#pragma unroll
      for (int s = 0; s < S; ++s) r[s] += __shfl_xor_sync(kFull, r[s], m);
#pragma unroll
    for (int s = 0; s < S; ++s) cf[s] = coefficient(r[s], k0 + s * G + q, gl == 0);
  }
  if (!__any_sync(kFull, may_clip)) {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const float lc = c.lr * cf[s];
#pragma unroll
      for (int t = 0; t < C; t += 2) {
        const float2 o = __ffma2_rn(make_float2(lc, lc), make_float2(x[s].v[t], x[s].v[t + 1]),
                                    make_float2(acc.v[t], acc.v[t + 1]));
        acc.v[t] = o.x;
        acc.v[t + 1] = o.y;
      }
    }
  } else {
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
      for (int t = 0; t < C; ++t) acc.v[t] = fmaf(c.lr, clip(x[s].v[t] * cf[s], c.bound), acc.v[t]);
  }
}

// Every pair of a window of 32, S steps at a time and half as many at its end.
template <class R, int S = R::S>
__device__ __forceinline__ void pair_window(LaneVec<R::C> &acc, const LaneVec<R::C> &xi, const void *rows, unsigned vm,
                                            unsigned rm, const PairCtx &c, float &loss, int lane) {
  constexpr int kChunk = S * R::G;
  const int end = 32 - __clz(vm);
  for (int k = 0; k < end; k += kChunk) {
    if (((vm >> k) & (kFull >> (32 - kChunk))) == 0) continue;
    if (end - k > kChunk / 2) pair_steps<R, S>(acc, xi, rows, vm, rm, k, c, loss, lane);
    else pair_steps<R, S / 2>(acc, xi, rows, vm, rm, k, c, loss, lane);
  }
}

// Split rows: two-level, fixed-order combine of the parts; the partial is in slot
// it.first_slot + it.part.  True on the warp that ends up with the row's sum, in acc.
template <int D>
__device__ __forceinline__ bool combine_parts(Frag<D> &acc, const WorkItem &it, float *slots, int32_t *counters,
                                              int lane) {
  const int P = it.nparts;
  const int g = it.part / kCombineGroup;
  const int ng = (P + kCombineGroup - 1) / kCombineGroup;
  const int gsize = min(kCombineGroup, P - g * kCombineGroup);
  bool owner = arrive_last(counters + it.counter + g, gsize, lane);
  if (owner) {
    sum_slots(acc, slots + size_t(it.first_slot + g * kCombineGroup) * D, gsize, lane);
    if (ng > 1) {
      store<D, true>(acc, slots + size_t(it.first_slot + P + g) * D, lane);
      owner = arrive_last(counters + it.counter + ng, ng, lane);
      if (owner) sum_slots(acc, slots + size_t(it.first_slot + P) * D, ng, lane);
    }
  }
  return owner;
}

}  // namespace dev
}  // namespace de
