// Batched form, register kernel: a warp runs vertices_per_warp work items at once
// on 32 / vertices_per_warp lanes each, neighbour rows loaded into registers.  A
// team is one CTA, or the CTAs of a cluster where the graphs alone would leave SMs
// idle (register_ctas in de_batched.cu); a graph's results do not depend on which.
#include "de_batched.cuh"

namespace de {
namespace batched {
namespace {

// One group of L = 32 / VPW lanes works on one item; lane j of the group holds
// components [j*P, j*P + P) of a row, P = D / L.
template <int D, int VPW>
struct Row {
  static constexpr int L = 32 / VPW;
  static constexpr int P = D / L;
  float v[P];
};

template <int D, int VPW, bool kBF16>
__device__ __forceinline__ void load_row(Row<D, VPW> &r, const BatchedArgs &a, int64_t vertex, int gl) {
  constexpr int P = Row<D, VPW>::P;
  const int64_t base = vertex * D + int64_t(gl) * P;
  // widest loads the lane's P components allow (rows and lane offsets are P-aligned)
  if constexpr (kBF16) {
    constexpr int K = P % 8 == 0 ? 4 : P % 4 == 0 ? 2 : 1;  // 32-bit words per load
    const uint32_t *p = reinterpret_cast<const uint32_t *>(a.xb + base);
#pragma unroll
    for (int i = 0; i < P / 2; i += K) {
      uint32_t w[K];
      if constexpr (K == 4) {
        const uint4 u = *reinterpret_cast<const uint4 *>(p + i);
        w[0] = u.x, w[1] = u.y, w[2] = u.z, w[3] = u.w;
      } else if constexpr (K == 2) {
        const uint2 u = *reinterpret_cast<const uint2 *>(p + i);
        w[0] = u.x, w[1] = u.y;
      } else {
        w[0] = p[i];
      }
#pragma unroll
      for (int k = 0; k < K; ++k) {
        r.v[2 * (i + k)] = __uint_as_float(w[k] << 16);
        r.v[2 * (i + k) + 1] = __uint_as_float(w[k] & 0xffff0000u);
      }
    }
  } else if constexpr (P % 4 == 0) {
    const float4 *p = reinterpret_cast<const float4 *>(a.xm + base);
#pragma unroll
    for (int i = 0; i < P / 4; ++i) {
      const float4 f = __ldcg(p + i);
      r.v[4 * i] = f.x, r.v[4 * i + 1] = f.y, r.v[4 * i + 2] = f.z, r.v[4 * i + 3] = f.w;
    }
  } else {
    const float2 *p = reinterpret_cast<const float2 *>(a.xm + base);
#pragma unroll
    for (int i = 0; i < P / 2; ++i) {
      const float2 f = __ldcg(p + i);
      r.v[2 * i] = f.x, r.v[2 * i + 1] = f.y;
    }
  }
}

template <int L>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int m = L / 2; m >= 1; m >>= 1) v += __shfl_xor_sync(kAll, v, m);
  return v;
}

// Rows in flight per group.  Eight take more registers, and at most shapes a resident CTA
// with them (dim 32, vertices_per_warp 4, 8 warps, 1,000 graphs: 2.52 ms against 1.55 with
// four).  They pay where they do not and a cluster's short chains are what bounds a
// minibatch: dim 32, FP32, 24 and 64 graphs on clusters of eight 4-7 % (BF16 loses 4 %).
template <int D, int VPW, int WARPS, bool kBF16, bool kCluster>
constexpr int kInFlight = kCluster && !kBF16 && D == 32 && VPW == 4 && (WARPS == 8 || WARPS == 16) ? 8 : 4;

// Resident CTAs the registers are held to where the compiler alone takes one too many for
// the fourth (0: its own choice).  400 graphs, dim 64: 16.0 ms at 160 registers, 14.1 before.
template <int D, int VPW, int WARPS>
constexpr int kMinCtas = D == 64 && VPW == 2 && WARPS == 4 ? 4 : 0;

// Whether a chunk's column ids are loaded a chunk ahead.  At dim 128, FP32, a row to a
// warp of sixteen the registers for it are not there: 400 graphs 9.6 ms so, 8.5 without.
template <int D, int VPW, int WARPS, bool kBF16, bool kCluster>
constexpr bool kIdsAhead = kCluster || kBF16 || D != 128 || VPW != 1 || WARPS != 16;

// Forces of up to U rows named by lanes [k, k + U) of the group (ids < 0: none),
// all groups of the warp in step (the caller keeps the warp converged).  xi is the
// row's FP32 master value.  In the BF16 form the rows are read as BF16; a pair
// whose squared distance from those reads is below a.near_r is read again from
// the FP32 master and recomputed, so that the rounding of the copy does not bias
// close pairs (their distance is then comparable with the BF16 rounding step).
template <int D, int VPW, int U, bool kBF16, bool kAttract>
__device__ __forceinline__ void group_forces(const BatchedArgs &a, Row<D, VPW> &acc, const Row<D, VPW> &xi,
                                             int64_t voff, int ids, int k, int gbase, int gl, float lr,
                                             float &loss, bool want) {
  constexpr int L = Row<D, VPW>::L, P = Row<D, VPW>::P;
  Row<D, VPW> xn[U];
  int nid[U];
  float r[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    int n = __shfl_sync(kAll, ids, gbase + k + u);
    nid[u] = n;
    if (n >= 0) load_row<D, VPW, kBF16>(xn[u], a, voff + n, gl);
    else xn[u] = xi;
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    float p = 0.f;
#pragma unroll
    for (int t = 0; t < P; ++t) {
      const float d = xi.v[t] - xn[u].v[t];
      p = fmaf(d, d, p);
    }
    r[u] = group_sum<L>(p);
  }
  if constexpr (kBF16) {
    bool near[U], any = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      near[u] = nid[u] >= 0 && r[u] < a.near_r;
      any |= near[u];
    }
    if (__any_sync(kAll, any)) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (near[u]) load_row<D, VPW, false>(xn[u], a, voff + nid[u], gl);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float p = 0.f;
#pragma unroll
        for (int t = 0; t < P; ++t) {
          const float d = xi.v[t] - xn[u].v[t];
          p = fmaf(d, d, p);
        }
        p = group_sum<L>(p);
        if (near[u]) r[u] = p;
      }
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    float c = kAttract ? -2.0f / (1.0f + r[u]) : 2.0f / ((r[u] + 1e-6f) * (1.0f + r[u]));
    if (nid[u] < 0) c = 0.f;
#pragma unroll
    for (int t = 0; t < P; ++t) acc.v[t] = fmaf(lr, bclip((xi.v[t] - xn[u].v[t]) * c, a.bound), acc.v[t]);
    if (want && nid[u] >= 0 && gl == 0) loss += kAttract ? log1pf(r[u]) : logf((1.0f + r[u]) / (r[u] + 1e-6f));
  }
}

// kCluster: a team is the CTAs of the cluster that the kernel is launched in, else one CTA
// (a kernel of its own: the cluster's run-time size takes up to 45 registers).
template <int D, int VPW, int WARPS, bool kBF16, bool kCluster>
__global__ void __launch_bounds__(WARPS * 32, kMinCtas<D, VPW, WARPS>) batched_kernel(const BatchedArgs a) {
  constexpr int L = Row<D, VPW>::L, P = Row<D, VPW>::P, U = kInFlight<D, VPW, WARPS, kBF16, kCluster>;
  static_assert(P % 2 == 0, "components per lane must be even");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grp = lane / L, gl = lane % L, gbase = grp * L;
  __shared__ int sh_graph;
  // team: nct CTAs (those of the cluster), this one its rank-th
  const int nct = kCluster ? cluster_ctas() : 1, rank = kCluster ? cluster_rank() : 0;
  const int team = blockIdx.x / nct, tw = rank * WARPS + warp, TW = nct * WARPS;
  auto team_sync = [&]() {
    if (kCluster) cluster_sync();
    else __syncthreads();
  };
  float *stage = a.stage + size_t(team) * a.stage_rows * D;
  float *slots = a.slots + size_t(team) * a.slot_stride * D;
  float *item_loss = a.item_loss + size_t(team) * a.item_stride;
  const int skip_last = a.quirks;

  for (;;) {
    int g;
    if (threadIdx.x == 0 && rank == 0) {
      const int i = atomicAdd(a.next_graph, 1);
      g = i < a.n_graphs ? a.order[i] : -1;
      if (kCluster) *reinterpret_cast<volatile int *>(a.cluster_slot + team) = g;
      else sh_graph = g;
    }
    team_sync();
    g = kCluster ? __ldcg(a.cluster_slot + team) : sh_graph;
    team_sync();  // the slot is rewritten only after every thread has read it
    if (g < 0) return;
    if (a.trace && threadIdx.x == 0 && rank == 0) {
      a.trace[3 * g] = globaltimer();
      a.trace[3 * g + 2] = blockIdx.x;
    }
    const GraphInfo G = a.graphs[g];
    const int skip = skip_last ? G.n - 1 : -1;  // edges into n-1 are dropped (algo.hpp:399-405, 538)
    for (int e = 0; e < a.epochs; ++e) {
      const float lr = a.lr[e];
      const bool want = a.compute_loss && e >= a.loss_from;
      double eloss = 0.0;  // rank 0, warp 0: the epoch's loss, minibatch by minibatch
      for (int j = 0; j < G.batches; ++j) {
        const int64_t bi = G.batch_off + j;
        const int64_t it0 = a.batch_item_off[bi];
        const int n_items = int(a.batch_item_off[bi + 1] - a.batch_item_off[bi]);
        const int base = j * a.batch;
        const int rows = min(a.batch, G.n - base);
        const int rep_rows = (a.quirks && e > 0) ? G.last_batch_size : rows;  // algo.hpp:167-169, 594
        const int32_t *negs = a.negs + G.neg_off + (size_t(e) * G.batches + j) * a.ns;
        // ---- 1. items, VPW per warp at a time
        for (int i0 = tw * VPW; i0 < n_items; i0 += TW * VPW) {
          const int my = i0 + grp;
          const bool has = my < n_items;
          WorkItem it{};
          if (has) it = a.items[it0 + my];
          Row<D, VPW> xi, acc;
#pragma unroll
          for (int t = 0; t < P; ++t) acc.v[t] = 0.f;
          if (has) load_row<D, VPW, false>(xi, a, G.voff + base + it.row, gl);
          else
#pragma unroll
            for (int t = 0; t < P; ++t) xi.v[t] = 0.f;
          float loss = 0.f;
          const int cnt = has ? it.e_end - it.e_begin : 0;
          const int32_t *cols = a.col + G.eoff + it.e_begin;
          int maxcnt = cnt;
#pragma unroll
          for (int m = 16; m >= L; m >>= 1) maxcnt = max(maxcnt, __shfl_xor_sync(kAll, maxcnt, m));
          constexpr bool kAhead = kIdsAhead<D, VPW, WARPS, kBF16, kCluster>;
          int next = kAhead && gl < cnt ? __ldg(cols + gl) : -1;
          for (int c0 = 0; c0 < maxcnt; c0 += L) {
            if constexpr (!kAhead) next = gl < cnt - c0 ? __ldg(cols + c0 + gl) : -1;
            const int ids = next == skip ? -1 : next;
            if constexpr (kAhead) next = gl < cnt - c0 - L ? __ldg(cols + c0 + L + gl) : -1;
            for (int k = 0; k < L && c0 + k < maxcnt; k += U)
              group_forces<D, VPW, U, kBF16, true>(a, acc, xi, G.voff, ids, k, gbase, gl, lr, loss, want);
          }
          const bool repulse = has && it.part == 0 && it.row < rep_rows;
          const bool any_rep = __any_sync(kAll, repulse);
          for (int k0 = 0; any_rep && k0 < a.ns; k0 += L) {
            int ids = -1;
            if (repulse && gl < a.ns - k0) {
              ids = __ldg(negs + k0 + gl);
              if (ids >= G.n) ids = -1;  // a draw equal to n contributes nothing
            }
            for (int k = 0; k < L && k0 + k < a.ns; k += U)
              group_forces<D, VPW, U, kBF16, false>(a, acc, xi, G.voff, ids, k, gbase, gl, lr, loss, want);
          }
          if (has) {
            float *dst = it.nparts > 1 ? slots + size_t(it.first_slot + it.part) * D : stage + size_t(it.row) * D;
#pragma unroll
            for (int t = 0; t < P; t += 2) *reinterpret_cast<float2 *>(dst + gl * P + t) = make_float2(acc.v[t], acc.v[t + 1]);
            if (want && gl == 0) item_loss[my] = loss;
          }
        }
        team_sync();
        // ---- 2. split rows: pieces in piece order
        const int s0 = a.batch_split_off[bi], s1 = a.batch_split_off[bi + 1];
        combine_split_rows<D>(a, slots, stage, s0, s1, tw, TW, lane);
        // the minibatch's loss in item order, whatever team made it
        if (want && tw == 0) eloss += minibatch_loss(item_loss, n_items, lane);
        if (s1 > s0) team_sync();
        // ---- 3. update (algo.hpp:651-666)
        update_rows<kBF16>(a.xm, a.xb, stage, (G.voff + base) * D, rows * D, rank * WARPS * 32 + threadIdx.x,
                           TW * 32);
        team_sync();
      }
      if (tw == 0 && lane == 0 && a.compute_loss) a.loss[size_t(g) * a.epochs + e] = eloss;
    }
    if (a.trace && threadIdx.x == 0 && rank == 0) a.trace[3 * g + 1] = globaltimer();
  }
}


// A team shape exists when every lane of a group holds an even number of components.
template <int D, int V>
constexpr bool kShapeOk = (D / (32 / V)) % 2 == 0;

template <int D, bool kBF16, int V, int W>
BatchedKernel pick_team(bool cluster) {
  return cluster ? batched_kernel<D, V, W, kBF16, true> : batched_kernel<D, V, W, kBF16, false>;
}

template <int D, bool kBF16, int V>
BatchedKernel pick_warps(int warps, bool cluster) {
  if constexpr (kShapeOk<D, V>) {
    switch (warps) {
      case 4: return pick_team<D, kBF16, V, 4>(cluster);
      case 8: return pick_team<D, kBF16, V, 8>(cluster);
      case 16: return pick_team<D, kBF16, V, 16>(cluster);
      case 32: return pick_team<D, kBF16, V, 32>(cluster);
    }
  }
  return nullptr;
}

template <int D, bool kBF16>
BatchedKernel pick(int vpw, int warps, bool cluster) {
  switch (vpw) {
    case 1: return pick_warps<D, kBF16, 1>(warps, cluster);
    case 2: return pick_warps<D, kBF16, 2>(warps, cluster);
    case 4: return pick_warps<D, kBF16, 4>(warps, cluster);
  }
  return nullptr;
}

}  // namespace

BatchedKernel pick_register(int dim, bool bf16, int vpw, int warps, bool cluster) {
  switch (dim) {
    case 32: return bf16 ? pick<32, true>(vpw, warps, cluster) : pick<32, false>(vpw, warps, cluster);
    case 64: return bf16 ? pick<64, true>(vpw, warps, cluster) : pick<64, false>(vpw, warps, cluster);
    case 128: return bf16 ? pick<128, true>(vpw, warps, cluster) : pick<128, false>(vpw, warps, cluster);
  }
  return nullptr;
}


}  // namespace batched
}  // namespace de
