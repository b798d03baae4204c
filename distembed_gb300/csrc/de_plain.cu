// FP32 plain form of the force-model SGD minibatch step (sm_103a).
//
// One launch per minibatch.  A warp owns one work item (a row, or an edge-capped
// piece of a high-degree row); items are sorted by decreasing cost so the block
// scheduler hands out the long ones first.  The pairs of an item are its CSR entries
// (cpp/algo/algo.hpp:531-582) and then, on a row's first piece, the minibatch's shared
// negatives (algo.hpp:594-647): one sequence, each lane holding one pair's other row.
// At dim 128 and 256 a warp holds a row, eight or four rows are in flight, their
// squared distances are reduced together, each lane turns one of them into the
// t-distribution coefficient and the coefficients are broadcast back; below, a pair is
// computed by dim/8 lanes and a warp takes four or eight pairs a step.  The update
// (algo.hpp:651-666) is fused into the same pass.
//
// Within a minibatch the reference reads only pre-minibatch values (the update
// is applied after both passes), and minibatch j+1 must see minibatch j's update
// (algo.hpp:164-192).  Here the new rows of minibatch j go to a staging buffer
// S[j % 4]; launch j+1 copies them back into X, and until that copy is known to
// be complete (two launches later) readers take those rows from S.  Launch j
// runs in two phases around griddepcontrol.wait (programmatic dependent launch):
// before the wait it does every force whose other row is not in minibatch j-1
// (those rows are final), overlapping launch j-1; after the wait it does the
// few forces into minibatch j-1, combines split rows and stores.  A row without such
// forces is stored without waiting.  Launch j+1 is released once minibatch j-1 is
// complete (the CTAs that copy it back wait for that first), so at most two minibatches
// are in flight and launch j+1's early phase only ever reads rows that are final; and a
// fourth staging buffer keeps launch j's early stores away from the two that launch j-1
// still reads.
#include <cuda_runtime.h>

#include "de_async.cuh"
#include "de_device.cuh"
#include "de_internal.h"
#include "de_pairs.cuh"

namespace de {
namespace {

using namespace dev;

__device__ __forceinline__ int epoch_of(const PlainBatchArgs &a) { return a.epoch_at >= 0 ? a.epoch_at : a.epoch[0]; }
__device__ __forceinline__ int first_epoch_of(const PlainBatchArgs &a) {
  return a.epoch_at >= 0 ? a.first_epoch_at : a.epoch[1];
}
__device__ __forceinline__ float rate_of(const PlainBatchArgs &a, int epoch) {
  return a.epoch_at >= 0 ? a.lr_at : a.lr[epoch];
}

__device__ __forceinline__ bool in_prev(const PlainBatchArgs &a, int n) {
  return unsigned(n - a.prev_base) < unsigned(a.prev_rows);
}

// Row n before the wait (n is not in minibatch j-1): minibatch j-2's rows are
// read from their staging buffer (their copy-back may be in flight), every
// other row is final in X.  After the wait only rows of minibatch j-1 are read,
// from their staging buffer.
template <bool kAfterWait>
__device__ __forceinline__ const float *row_ptr(const PlainBatchArgs &a, int n, int D) {
  if (kAfterWait) return a.S_prev + size_t(n - a.prev_base) * D;
  const unsigned off = unsigned(n - a.prev2_base);
  return off < unsigned(a.prev2_rows) ? a.S_prev2 + size_t(off) * D : a.X + size_t(n) * D;
}

// Resident CTAs per SM the registers are held to.  One warp an item: 64 registers
// spill at dim 128 (measured against 72, R-MAT of 2^20 vertices, B = 4096: 14.5 against
// 13.6 us a minibatch) and pay below (dim 64: 10.5 against 11.0).  Several warps an
// item do not fill the GPU, so they take 80.
template <int D>
constexpr int kMinBlocks = D >= 256 ? 4 : D == 128 ? 7 : 8;
template <int D>
constexpr int kTeamMinBlocks = D >= 256 ? 4 : 6;

// The item's update: a whole row's new value staged (algo.hpp:651-666), or the part
// combined with the row's others and the row staged by the last of them.
template <int D>
__device__ __forceinline__ void finish_item(const PlainBatchArgs &a, const WorkItem &it, const LaneRow<D> &xi,
                                            LaneRow<D> &acc, int lane) {
  float *out = a.S_cur + size_t(it.row) * D;
  if (it.nparts <= 1) {
#pragma unroll
    for (int t = 0; t < Lay<D>::C; ++t) acc.v[t] = xi.v[t] + acc.v[t];
    store_lanes<D, false>(acc, out, lane);
    return;
  }
  store_lanes<D, true>(acc, a.P + size_t(it.first_slot + it.part) * D, lane);
  Frag<D> sum, x;
  if (!combine_parts<D>(sum, it, a.P, a.counters, lane)) return;
  load_nc(x, a.X + size_t(a.base + it.row) * D, lane);
#pragma unroll
  for (int t = 0; t < Frag<D>::N; ++t) sum.v[t] = x.v[t] + sum.v[t];
  store<D, false>(sum, out, lane);
}

// Rows of minibatch j-1: staging buffer -> X.  Until the next launch passes
// its wait, every reader takes these rows from the staging buffer.
constexpr int kCopyRows = 4;  // rows in flight of a warp that only copies
template <int D, int K>
__device__ __forceinline__ void copy_back(const PlainBatchArgs &a, int lane, int gw, int total_w) {
  for (int r0 = gw; r0 < a.prev_rows; r0 += K * total_w) {
    Frag<D> t[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (r0 + k * total_w < a.prev_rows) load_cg(t[k], a.S_prev + size_t(r0 + k * total_w) * D, lane);
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (r0 + k * total_w < a.prev_rows) store<D, false>(t[k], a.X + size_t(a.prev_base + r0 + k * total_w) * D, lane);
  }
}

template <int D>
__global__ void __launch_bounds__(kPlainWarps * 32, kMinBlocks<D>)
    plain_batch_kernel(const PlainBatchArgs a) {
  extern __shared__ __align__(16) float negsm[];  // stage_negs: [ns, D] rows of the minibatch's draws
  __shared__ __align__(8) uint64_t negbar;
  __shared__ int negerr;
  const int lane = threadIdx.x & 31;
  const int gw = blockIdx.x * kPlainWarps + (threadIdx.x >> 5);

  // The last CTAs copy minibatch j-1 back into X.  They release launch j+1 after their
  // wait, that is, with minibatch j-1 complete; the others release it at once.
  const int item_ctas = (a.n_items + kPlainWarps - 1) / kPlainWarps;
  if (int(blockIdx.x) >= item_ctas) {
    pdl_wait();
    pdl_trigger();
    copy_back<D, kCopyRows>(a, lane, gw - item_ctas * kPlainWarps, (gridDim.x - item_ctas) * kPlainWarps);
    return;
  }
  // An epoch's first minibatch reads what the launch before it writes.  The work item is
  // loaded after the wait, and every row's address comes out of it: a read-only load
  // whose address were known before could be moved ahead of the wait.
  if (a.first) pdl_wait();
  pdl_trigger();
  const bool has_item = gw < a.n_items;
  WorkItem it{};
  if (has_item) it = a.items[gw];
  const int epoch = epoch_of(a);
  const PairCtx c(rate_of(a, epoch), a.bound, a.compute_loss != 0);
  const int skip = a.skip_last ? a.n - 1 : -1;  // edges into n-1 are dropped (algo.hpp:399-405, 538)
  const int cnt = it.e_end - it.e_begin;
  // the repulsive pass of a row is done by its part 0
  const int rep_rows = (a.quirks && epoch + first_epoch_of(a) > 0) ? a.last_batch_size : a.rows;
  const int total = cnt + (has_item && it.part == 0 && it.row < rep_rows ? a.ns : 0);
  const int32_t *negs = a.negs + (size_t(epoch) * a.batches + a.batch_id) * a.ns;
  // the other row of the item's pair k0 + lane: its CSR entries, then the draws; -1 = none
  auto fetch = [&](int k0) -> int {
    const int k = k0 + lane;
    int id = -1;
    if (k < cnt) {
      id = __ldg(a.col + it.e_begin + k);
      if (id == skip) id = -1;
    } else if (k < total) {
      id = __ldg(negs + k - cnt);
      if (id >= a.n) id = -1;  // a draw equal to n contributes nothing
    }
    return id;
  };

  // Staged negatives: bit k of `staged`: draw k is a vertex outside minibatch j-1
  // (final before the wait), copied by one thread of the CTA into row k of negsm
  // with bulk asynchronous copies; the CTA waits (bounded) on one barrier.
  if (a.stage_negs) {
    unsigned staged = 0;
    for (int k = 0; k < a.ns; ++k) {
      const int nid = __ldg(negs + k);
      if (nid >= 0 && nid < a.n && !in_prev(a, nid)) staged |= 1u << k;
    }
    const uint32_t bar = smem_u32(&negbar);
    if (threadIdx.x == 0) {
      negerr = 0;
      mbar_init(bar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      mbar_expect_tx(bar, uint32_t(__popc(staged)) * D * 4u);
      for (int k = 0; k < a.ns; ++k)
        if ((staged >> k) & 1u)
          bulk_g2s(smem_u32(negsm + k * D), row_ptr<false>(a, __ldg(negs + k), D), D * 4u, bar);
    }
    __syncthreads();
    // after a timeout the results of this launch are invalid; the host reports the error
    if (!mbar_wait(bar, 0, &negerr) && lane == 0) atomicExch(a.err, 1);
  }

  float loss = 0.f;  // this item's loss terms (FP32); the epoch sum is FP64
  const float *const own = a.X + size_t(a.base + it.row) * D;
  LaneRow<D> xi, acc;
  acc.zero();
  int ids = fetch(0);
  if (has_item) load_lanes<D, kFinal>(xi, own, lane % Lay<D>::LP);
  // ---- before the wait: forces whose other row is final
  for (int k0 = 0; k0 < total; k0 += 32) {
    if (k0 > 0) ids = fetch(k0);
    const bool now = ids >= 0 && !in_prev(a, ids);
    const bool repels = now && k0 + lane >= cnt;
    const unsigned vm = __ballot_sync(kFull, now), rm = __ballot_sync(kFull, repels);
    const float *row = now ? row_ptr<false>(a, ids, D) : own;
    if (a.stage_negs) {
      if (repels) row = negsm + (k0 + lane - cnt) * D;
      pair_window<F32Rows<D, kShared>>(acc, xi, row, vm, rm, c, loss, lane);
    } else {
      pair_window<F32Rows<D, kFinal>>(acc, xi, row, vm, rm, c, loss, lane);
    }
  }
  // A whole row without a pair in minibatch j-1 is done: its staging slot is the one of
  // minibatch j-4, which no launch in flight reads.  Its warp need not hold its place
  // until minibatch j-1 is complete, so the later items of a launch of more than one
  // wave are not held up either (R-MAT of 2^20 vertices, B = 4096, dim 64 / 128 / 256:
  // 10.5 / 13.6 / 24.5 -> 9.6 / 12.2 / 22.8 us a minibatch).
  if (!has_item) return;
  if (it.nparts > 1 || total > 32 || __any_sync(kFull, ids >= 0 && in_prev(a, ids))) {
    pdl_wait();
    // ---- after the wait: forces into minibatch j-1
    for (int k0 = 0; a.prev_rows > 0 && k0 < total; k0 += 32) {
      if (total > 32) ids = fetch(k0);
      const bool late = ids >= 0 && in_prev(a, ids);
      const unsigned vm = __ballot_sync(kFull, late), rm = __ballot_sync(kFull, late && k0 + lane >= cnt);
      if (vm) pair_window<F32Rows<D, kStaged>>(acc, xi, late ? row_ptr<true>(a, ids, D) : own, vm, rm, c, loss, lane);
    }
  }
  sum_groups<D>(acc);
  finish_item<D>(a, it, xi, acc, lane);
  if (c.want_loss) {
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) loss += __shfl_xor_sync(kFull, loss, m);
    if (lane == 0) a.loss_partial[a.loss_off + gw] = double(loss);
  }
}

// ---------------------------------------------------------------- small minibatches
//
// The same step with W warps to a work item.  A minibatch that does not fill the
// GPU takes as long as the longest chain in it, and a warp alone goes through a
// row's pairs chunk after chunk (a load, a reduction, a divide: about 0.6 us).  Here
// an item's pairs are cut into groups of 8 (4 at dim 256), group q on warp q % W, so a
// row of 32 entries and its draws is two rounds at W = 4 instead of five; the warps'
// sums are added in warp order through shared memory.  Phases, staging ring and split
// rows as in plain_batch_kernel.  Measured, microseconds a minibatch at one / two / four
// warps an item: 20,000-vertex kNN graph, dim 128: B = 256 5.0 / 4.0 / 3.9, 1100 6.5 /
// 5.5 / 6.8; dim 256, B = 256 6.7 / 5.1 / 4.1; R-MAT of 100,003 vertices, dim 64, B = 512
// 5.1 / 4.5 / 5.0.  Eight warps an item, or groups of half the size, gained at most 6 %
// below 100 items and lost above 300.
template <int D, int W>
__global__ void __launch_bounds__(kPlainWarps * 32, kTeamMinBlocks<D>)
    plain_team_kernel(const PlainBatchArgs a) {
  constexpr int kTeams = kPlainWarps / W;      // items of a CTA
  constexpr int kPairs = D >= 256 ? 4 : 8;     // pairs of a group
  constexpr int kSteps = kPairs / Lay<D>::G;
  constexpr int kGroups = 32 / kPairs;         // groups of a warp whose ids its lanes hold at once
  __shared__ __align__(16) float s_acc[kTeams][W - 1][D];  // rows, 16 bytes at a time
  __shared__ float s_loss[kTeams][W - 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int team = warp / W, tw = warp % W;
  const int item = blockIdx.x * kTeams + team;
  if (a.first) {  // as in plain_batch_kernel
    pdl_wait();
    pdl_trigger();
  }
  const bool has_item = item < a.n_items;
  WorkItem it{};
  if (has_item) it = a.items[item];
  const int epoch = epoch_of(a);
  const PairCtx c(rate_of(a, epoch), a.bound, a.compute_loss != 0);
  const int skip = a.skip_last ? a.n - 1 : -1;  // edges into n-1 are dropped (algo.hpp:399-405, 538)
  const int cnt = it.e_end - it.e_begin;
  // the repulsive pass of a row is done by its part 0
  const int rep_rows = (a.quirks && epoch + first_epoch_of(a) > 0) ? a.last_batch_size : a.rows;
  const int total = cnt + (has_item && it.part == 0 && it.row < rep_rows ? a.ns : 0);
  const int32_t *negs = a.negs + (size_t(epoch) * a.batches + a.batch_id) * a.ns;
  const int groups = (total + kPairs - 1) / kPairs;
  const int mine = groups > tw ? (groups - tw + W - 1) / W : 0;  // this warp's groups
  // entry lane % kPairs of this warp's group s + lane / kPairs: its index among the
  // item's pairs, and its other row (-1 = none)
  auto entry = [&](int s) -> int { return ((s + lane / kPairs) * W + tw) * kPairs + lane % kPairs; };
  auto fetch = [&](int k) -> int {
    int id = -1;
    if (k < cnt) {
      id = __ldg(a.col + it.e_begin + k);
      if (id == skip) id = -1;
    } else if (k < total) {
      id = __ldg(negs + k - cnt);
      if (id >= a.n) id = -1;  // a draw equal to n contributes nothing
    }
    return id;
  };
  float loss = 0.f;
  const float *const own = a.X + size_t(a.base + it.row) * D;
  LaneRow<D> xi, acc;
  acc.zero();
  int ids = mine > 0 ? fetch(entry(0)) : -1;
  if (has_item) load_lanes<D, kFinal>(xi, own, lane % Lay<D>::LP);
  // ---- before the wait: forces whose other row is final
  for (int s = 0; s < mine; s += kGroups) {
    if (s > 0) ids = fetch(entry(s));
    const bool now = ids >= 0 && !in_prev(a, ids);
    const unsigned vm = __ballot_sync(kFull, now), rm = __ballot_sync(kFull, now && entry(s) >= cnt);
    const float *row = now ? row_ptr<false>(a, ids, D) : own;
    for (int r = 0; r < kGroups && s + r < mine; ++r)
      if ((vm >> (r * kPairs)) & ((1u << kPairs) - 1))
        pair_steps<F32Rows<D, kFinal>, kSteps>(acc, xi, row, vm, rm, r * kPairs, c, loss, lane);
  }
  pdl_wait();
  pdl_trigger();
  // ---- after the wait: forces into minibatch j-1
  for (int s = 0; a.prev_rows > 0 && s < mine; s += kGroups) {
    if (mine > kGroups) ids = fetch(entry(s));
    const bool late = ids >= 0 && in_prev(a, ids);
    const unsigned vm = __ballot_sync(kFull, late), rm = __ballot_sync(kFull, late && entry(s) >= cnt);
    const float *row = late ? row_ptr<true>(a, ids, D) : own;
    for (int r = 0; vm != 0 && r < kGroups && s + r < mine; ++r)
      if ((vm >> (r * kPairs)) & ((1u << kPairs) - 1))
        pair_steps<F32Rows<D, kStaged>, kSteps>(acc, xi, row, vm, rm, r * kPairs, c, loss, lane);
  }
  sum_groups<D>(acc);
  if (c.want_loss) {
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) loss += __shfl_xor_sync(kFull, loss, m);
  }
  copy_back<D, 1>(a, lane, blockIdx.x * kPlainWarps + warp, gridDim.x * kPlainWarps);
  if (tw > 0) {
    store_lanes<D, false>(acc, s_acc[team][tw - 1], lane);
    if (lane == 0) s_loss[team][tw - 1] = loss;
  }
  __syncthreads();
  if (tw > 0 || !has_item) return;
#pragma unroll
  for (int w = 0; w < W - 1; ++w) {
    LaneRow<D> t;
    load_lanes<D, kShared>(t, s_acc[team][w], lane % Lay<D>::LP);
#pragma unroll
    for (int k = 0; k < Lay<D>::C; ++k) acc.v[k] += t.v[k];
    loss += s_loss[team][w];
  }
  finish_item<D>(a, it, xi, acc, lane);
  if (c.want_loss && lane == 0) a.loss_partial[a.loss_off + item] = double(loss);
}

// SpMMAlgo::algo_spmm's step at one rank (cpp/algo/spmm.hpp:54-159):
// y[i] = sum over the CSR entries of row i of lr * x[col] (spmm.hpp:358-392), from the
// unchanged input x into the output y (spmm.hpp:397-412).  The reference goes
// minibatch by minibatch; the rows do not depend on one another, so every work item
// runs in one launch.  One warp per work item; the lanes hold the addresses of the
// item's rows, S steps of G rows are in flight (Lay), and a window in which every row
// counts loads them without a test.  Split rows are combined in piece order as in
// plain_batch_kernel.
// Bound by the rows' way from L2 to the SMs (17.3 GB gathered at R-MAT s20, dim 128,
// 4.1 GB of it from HBM): 1.49 ms as one row a load with a test each -> 1.28 ms, 13.5
// TB/s of gathered rows.
template <int D>
constexpr int kSpmmSteps = D == 128 ? 8 : D == 256 ? 4 : 2;
// Resident CTAs per SM the registers are held to: warps in flight count for more than
// the few spilled words (R-MAT of 2^20 vertices, ms a pass: dim 128 at 10 / 12 / 14
// CTAs 1.42 / 1.34 / 1.28; dim 64 at 8 / 12 / 16 1.08 / 0.88 / 0.87; dim 32 0.84 /
// 0.76 / 0.70; dim 256 at 5 / 6 / 7 3.07 / 2.81 / 2.71).
template <int D>
constexpr int kSpmmMinBlocks = D == 128 ? 14 : D == 256 ? 7 : 16;

template <int D, int S, bool kAll>
__device__ __forceinline__ void spmm_steps(LaneRow<D> &acc, const float *rows, int k0, float lr, int lane) {
  constexpr int LP = Lay<D>::LP, G = Lay<D>::G, C = Lay<D>::C;
  const int q = G > 1 ? lane / LP : 0, gl = G > 1 ? lane % LP : lane;
  LaneRow<D> x[S];
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const float *row = reinterpret_cast<const float *>(
        __shfl_sync(kFull, reinterpret_cast<unsigned long long>(rows), k0 + s * G + q));
    if (kAll || row) load_lanes<D, kFinal>(x[s], row, gl);
    else x[s].zero();
  }
#pragma unroll
  for (int s = 0; s < S; ++s)
#pragma unroll
    for (int t = 0; t < C; t += 2) {
      const float2 o = __ffma2_rn(make_float2(lr, lr), make_float2(x[s].v[t], x[s].v[t + 1]),
                                  make_float2(acc.v[t], acc.v[t + 1]));
      acc.v[t] = o.x;
      acc.v[t + 1] = o.y;
    }
}

template <int D>
__global__ void __launch_bounds__(kPlainWarps * 32, kSpmmMinBlocks<D>)
    spmm_kernel(const SpmmArgs a) {
  constexpr int S = kSpmmSteps<D>, kChunk = S * Lay<D>::G;
  const int lane = threadIdx.x & 31;
  const int64_t gw = blockIdx.x * int64_t(kPlainWarps) + (threadIdx.x >> 5);
  if (gw >= a.n_items) return;
  const WorkItem it = a.items[gw];
  const float *row = nullptr;
  if (lane < it.e_end - it.e_begin) {
    const int id = __ldg(a.col + it.e_begin + lane);
    if (id != a.skip) row = a.X + size_t(id) * D;  // edges into n-1 (spmm.hpp:260-265, 365)
  }
  const unsigned vm = __ballot_sync(kFull, row != nullptr);
  const int end = 32 - __clz(vm);
  LaneRow<D> acc;
  acc.zero();
  for (int k = 0; k < end; k += kChunk) {
    constexpr unsigned kMask = kFull >> (32 - kChunk);
    if (((vm >> k) & kMask) == kMask) spmm_steps<D, S, true>(acc, row, k, a.lr, lane);
    else if (end - k > kChunk / 2) spmm_steps<D, S, false>(acc, row, k, a.lr, lane);
    else spmm_steps<D, S / 2, false>(acc, row, k, a.lr, lane);
  }
  sum_groups<D>(acc);
  float *const out = a.Y + (size_t(it.batch) * a.batch + it.row) * D;
  if (it.nparts <= 1) {
    store_lanes<D, false>(acc, out, lane);
    return;
  }
  float *const P = a.P + size_t(__ldg(a.slot_off + it.batch)) * D;
  store_lanes<D, true>(acc, P + size_t(it.first_slot + it.part) * D, lane);
  Frag<D> sum;
  if (combine_parts<D>(sum, it, P, a.counters + __ldg(a.counter_off + it.batch), lane))
    store<D, false>(sum, out, lane);
}

// v[0] + ... + v[n - 1] by a CTA of 256 threads in a fixed order; on thread 0.
__device__ __forceinline__ double block_sum(const double *v, int64_t n, double *red) {
  double s = 0.0;
  int64_t i = threadIdx.x;
  for (; i + 7 * 256 < n; i += 8 * 256) {  // eight loads in flight, added in order
    double t[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) t[u] = __ldcg(v + i + u * 256);
#pragma unroll
    for (int u = 0; u < 8; ++u) s += t[u];
  }
  for (; i < n; i += 256) s += __ldcg(v + i);
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) s += __shfl_xor_sync(kFull, s, m);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  s = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < 8; ++w) s += red[w];
  return s;
}

// End of an epoch: write back the last minibatch, reduce the epoch's loss
// partials in a fixed order (each CTA a fixed chunk, then the last CTA to
// finish sums the chunk sums in order), advance the epoch counter.
template <int D>
__global__ void __launch_bounds__(256) flush_kernel(const FlushArgs a) {
  const int lane = threadIdx.x & 31;
  const int gw = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int total_w = gridDim.x * 8;
  pdl_wait();
  pdl_trigger();
  for (int r = gw; r < a.last_rows; r += total_w) {
    Frag<D> t;
    load_cg(t, a.S_last + size_t(r) * D, lane);  // written by the launch before
    store<D, false>(t, a.X + size_t(a.last_base + r) * D, lane);
  }
  if (!a.compute_loss) {
    // every reader of the epoch counter was in the launches before this one
    if (blockIdx.x == 0 && threadIdx.x == 0) a.epoch[0] += 1;
    return;
  }
  // The loss: kFlushChunk partials a CTA (or more, where the grid is too small), so
  // a small job's sum needs no second step across CTAs.
  const int64_t chunk = flush_chunk(a.n_partials);
  const int parts = flush_parts(a.n_partials);
  if (int(blockIdx.x) >= parts) return;
  __shared__ double red[8];
  __shared__ bool last;
  const int64_t lo = blockIdx.x * chunk;
  double s = block_sum(a.loss_partial + lo, min(a.n_partials - lo, chunk), red);
  if (parts > 1) {
    if (threadIdx.x == 0) {
      a.block_sums[blockIdx.x] = s;
      __threadfence();
      last = atomicAdd(a.done, 1) == parts - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s = block_sum(a.block_sums, parts, red);
  }
  if (threadIdx.x == 0) {
    const int e = a.epoch[0];
    a.loss[e] = s;
    a.epoch[0] = e + 1;
    *a.done = 0;
  }
}

// Losses of epochs (blockIdx.x) whose items' losses lie one epoch after another: with
// one part (blockIdx.y) the sum, else the parts' sums for epoch_parts_kernel; in
// flush_kernel's order.
__global__ void __launch_bounds__(256) epoch_losses_kernel(const double *partial, int64_t n_items, double *out) {
  __shared__ double red[8];
  const int64_t chunk = flush_chunk(n_items), lo = blockIdx.y * chunk;
  const double s = block_sum(partial + int64_t(blockIdx.x) * n_items + lo, min(n_items - lo, chunk), red);
  if (threadIdx.x == 0) out[int64_t(blockIdx.x) * gridDim.y + blockIdx.y] = s;
}
__global__ void __launch_bounds__(256) epoch_parts_kernel(const double *sums, int parts, double *loss) {
  __shared__ double red[8];
  const double s = block_sum(sums + int64_t(blockIdx.x) * parts, parts, red);
  if (threadIdx.x == 0) loss[blockIdx.x] = s;
}

__global__ void f64_to_f32_kernel(const double *__restrict__ s, float *__restrict__ d, int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    d[i] = float(s[i]);
}

__global__ void f32_to_f64_kernel(const float *__restrict__ s, double *__restrict__ d, int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    d[i] = double(s[i]);
}

template <typename Args>
cudaError_t launch(void (*k)(Args), int grid, int block, const Args &a, bool pdl, cudaStream_t s, size_t smem = 0) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, a);
}

}  // namespace

cudaError_t launch_plain_batch(int dim, const PlainBatchArgs &a, bool teams, bool pdl, cudaStream_t s) {
  const int block = kPlainWarps * 32;
  if (a.stage_negs && a.ns > kStageNegMax) return cudaErrorInvalidValue;
  const size_t smem = a.stage_negs ? size_t(a.ns) * dim * sizeof(float) : 0;
  const int w = teams ? plain_team_warps(dim, a.n_items) : 1;
  const int team_grid = (a.n_items * w + kPlainWarps - 1) / kPlainWarps;
  if (w == 4) {
    switch (dim) {
      case 64: return launch(plain_team_kernel<64, 4>, team_grid, block, a, pdl, s);
      case 128: return launch(plain_team_kernel<128, 4>, team_grid, block, a, pdl, s);
      case 256: return launch(plain_team_kernel<256, 4>, team_grid, block, a, pdl, s);
      default: return cudaErrorInvalidValue;
    }
  }
  if (w == 2) {
    switch (dim) {
      case 32: return launch(plain_team_kernel<32, 2>, team_grid, block, a, pdl, s);
      case 64: return launch(plain_team_kernel<64, 2>, team_grid, block, a, pdl, s);
      case 128: return launch(plain_team_kernel<128, 2>, team_grid, block, a, pdl, s);
      case 256: return launch(plain_team_kernel<256, 2>, team_grid, block, a, pdl, s);
      default: return cudaErrorInvalidValue;
    }
  }
  // CTAs of their own copy minibatch j-1 back
  const int per = kPlainWarps * kCopyRows;
  const int grid = (a.n_items + kPlainWarps - 1) / kPlainWarps + (a.prev_rows + per - 1) / per;
  switch (dim) {
    case 32: return launch(plain_batch_kernel<32>, grid, block, a, pdl, s, smem);
    case 64: return launch(plain_batch_kernel<64>, grid, block, a, pdl, s, smem);
    case 128: return launch(plain_batch_kernel<128>, grid, block, a, pdl, s, smem);
    case 256: return launch(plain_batch_kernel<256>, grid, block, a, pdl, s, smem);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_epoch_losses(const double *partial, int64_t n_items, int epochs, double *block_sums, double *loss,
                                cudaStream_t s) {
  const int parts = flush_parts(n_items);
  epoch_losses_kernel<<<dim3(epochs, parts), 256, 0, s>>>(partial, n_items, parts > 1 ? block_sums : loss);
  if (parts > 1) epoch_parts_kernel<<<epochs, 256, 0, s>>>(block_sums, parts, loss);
  return cudaGetLastError();
}

cudaError_t launch_spmm(int dim, const SpmmArgs &a, cudaStream_t s) {
  const int64_t grid = (a.n_items + kPlainWarps - 1) / kPlainWarps;
  if (grid == 0) return cudaSuccess;
  if (grid >= (int64_t(1) << 31)) return cudaErrorInvalidValue;
  switch (dim) {
    case 32: spmm_kernel<32><<<unsigned(grid), kPlainWarps * 32, 0, s>>>(a); break;
    case 64: spmm_kernel<64><<<unsigned(grid), kPlainWarps * 32, 0, s>>>(a); break;
    case 128: spmm_kernel<128><<<unsigned(grid), kPlainWarps * 32, 0, s>>>(a); break;
    case 256: spmm_kernel<256><<<unsigned(grid), kPlainWarps * 32, 0, s>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_flush(int dim, const FlushArgs &a, bool pdl, cudaStream_t s) {
  switch (dim) {
    case 32: return launch(flush_kernel<32>, kFlushBlocks, 256, a, pdl, s);
    case 64: return launch(flush_kernel<64>, kFlushBlocks, 256, a, pdl, s);
    case 128: return launch(flush_kernel<128>, kFlushBlocks, 256, a, pdl, s);
    case 256: return launch(flush_kernel<256>, kFlushBlocks, 256, a, pdl, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_f64_to_f32(const double *src, float *dst, int64_t count, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  const int grid = int(count / 256 + 1 < 152 * 8 ? count / 256 + 1 : 152 * 8);
  f64_to_f32_kernel<<<grid, 256, 0, s>>>(src, dst, count);
  return cudaGetLastError();
}

cudaError_t launch_f32_to_f64(const float *src, double *dst, int64_t count, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  const int grid = int(count / 256 + 1 < 152 * 8 ? count / 256 + 1 : 152 * 8);
  f32_to_f64_kernel<<<grid, 256, 0, s>>>(src, dst, count);
  return cudaGetLastError();
}

}  // namespace de
