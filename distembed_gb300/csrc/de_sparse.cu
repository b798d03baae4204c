// Sparse embedding (SparseEmbedding::algo_sparse_embedding at one rank,
// cpp/algo/sparse_embedding.hpp:78-194).  An embedding row is a dense FP64
// vector in which INT_MIN marks an absent entry (the reference's dense
// collector, cpp/core/sparse_mat.hpp:367-377, 492-505).  The pair term walks
// the union of the two rows' present entries (sparse_embedding.hpp:380-427,
// 548-598): value x_i - x_j, x_i or -x_j, r = sum of value^2, an update on
// every union entry.  With absent entries read as 0 this is the dense pair
// term: a dim absent from both rows adds 0 to r and 0 to the update.  So the
// kernels read an FP32 mirror of the rows that holds 0 for absent entries and
// reuse the dense pair arithmetic (dev::pair_forces); the FP64 rows keep the
// reference's values, and the top-k pruning compares them exactly.
#include <cuda_runtime.h>

#include <cstdint>

#include "de_device.cuh"
#include "de_internal.h"
#include "de_pairs.cuh"

namespace de {
namespace {

using dev::Frag;
using dev::kFull;

constexpr uint64_t kAbsent64 = 0xC1E0000000000000ull;  // bits of (double)INT_MIN
int elementwise_grid(int64_t count) { return int(count / 256 + 1 < 152 * 8 ? count / 256 + 1 : 152 * 8); }

// The attractive pass of every minibatch of one iteration in one launch (the
// one-rank branch never merges its updates, so no row changes during the
// iteration): one warp per work item, split rows combined in piece order.  Row i's
// update goes to Y[i] (FP32, from zero).  The launch is hundreds of thousands of warps,
// so resident warps hide the gather's latency, and the registers are held down for
// them.  The sums keep the order of whole-warp rows at every dim (the collector adds
// the updates up in 64 bits): from dim 128 on that is dev::pair_window's, below it is
// dev::pair_forces'.  R-MAT of 131,072 vertices, dim 64 / 128 / 256: 187 / 231 / 610 us
// an iteration -> 160 / 198 / 344 (four rows in flight; eight, or eight resident CTAs,
// were slower at dim 128: 423 and 222).
template <int D>
constexpr int kAttractMinBlocks = D >= 256 ? 7 : D == 128 ? 12 : 8;

template <int D>
__global__ void __launch_bounds__(kPlainWarps * 32, kAttractMinBlocks<D>) sparse_attract_kernel(const SpmmArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = blockIdx.x * int64_t(kPlainWarps) + (threadIdx.x >> 5);
  if (gw >= a.n_items) return;
  const WorkItem it = a.items[gw];
  const int64_t row = int64_t(it.batch) * a.batch + it.row;
  const float *const own = a.X + size_t(row) * D;
  const int cnt = it.e_end - it.e_begin;  // at most 32
  const int id = lane < cnt ? __ldg(a.col + it.e_begin + lane) : -1;
  float unused_loss = 0.f;
  Frag<D> acc;
  if constexpr (D >= 128) {
    static_assert(dev::Lay<D>::LP == 32, "a whole warp holds a row");
    const dev::PairCtx c(a.lr, a.bound, false);
    dev::LaneRow<D> xi, sum;
    dev::load_lanes<D, dev::kFinal>(xi, own, lane);
    sum.zero();
    dev::pair_window<dev::F32Rows<D, dev::kFinal>, 4>(sum, xi, id >= 0 ? a.X + size_t(id) * D : own, __ballot_sync(kFull, id >= 0), 0u,
                                     c, unused_loss, lane);
#pragma unroll
    for (int t = 0; t < Frag<D>::N; ++t) acc.v[t] = sum.v[t];
  } else {
    constexpr int U = 8;
    Frag<D> xi;
    dev::load_nc(xi, own, lane);
    acc.zero();
    for (int k = 0; k < cnt; k += U) {
      Frag<D> xn[U];
      unsigned valid = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int nb = __shfl_sync(kFull, id, (k + u) & 31);
        if (k + u < cnt) {
          dev::load_nc(xn[u], a.X + size_t(nb) * D, lane);
          valid |= 1u << u;
        } else {
          xn[u] = xi;
        }
      }
      dev::pair_forces<D, U, true>(acc, xi, xn, valid, a.lr, a.bound, false, unused_loss, lane);
    }
  }
  bool owner = true;
  if (it.nparts > 1) {
    float *const P = a.P + size_t(__ldg(a.slot_off + it.batch)) * D;
    dev::store<D, true>(acc, P + size_t(it.first_slot + it.part) * D, lane);
    owner = dev::combine_parts<D>(acc, it, P, a.counters + __ldg(a.counter_off + it.batch), lane);
  }
  if (owner) dev::store<D, false>(acc, a.Y + size_t(row) * D, lane);
}

// Batch collector: slot r of minibatch j holds row jB + r, and the one-rank
// branch adds every minibatch into the same slots without clearing them
// (sparse_embedding.hpp:452-455, 380-386): coll[r] += Y[r] + Y[B + r] + ..., in
// minibatch order.  The terms are FP32 (the rows' updates); their running sum is
// kept as an unevaluated FP32 pair hi + lo (Knuth's TwoSum adds each term with
// its rounding error carried in lo, about 44 bits of precision), then added to
// the FP64 collector once: two FP64 operations per slot instead of two per term
// on the GPU's narrow FP64 pipe.
__global__ void __launch_bounds__(256)
    sparse_collect_kernel(const float *__restrict__ y, double *__restrict__ coll, int64_t n, int32_t batch,
                          int32_t dim) {
  const int64_t slots = int64_t(batch) * dim;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < slots; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t r = e / dim;
    const float *yp = y + r * dim + (e - r * dim);
    const int64_t stride = int64_t(batch) * dim;
    const int64_t rows = (n - r + batch - 1) / batch;  // rows r, r + B, ... below n
    float hi = 0.f, lo = 0.f;
    auto add = [&](float v) {
      const float s = __fadd_rn(hi, v);
      const float bv = __fsub_rn(s, hi);
      const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bv)), __fsub_rn(v, bv));
      hi = s;
      lo = __fadd_rn(lo, err);
    };
    int64_t q = 0;
    for (; q + 8 <= rows; q += 8) {  // eight loads in flight, added in order
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldg(yp + (q + u) * stride);
#pragma unroll
      for (int u = 0; u < 8; ++u) add(v[u]);
    }
    for (; q < rows; ++q) add(__ldg(yp + q * stride));
    coll[e] = coll[e] + (double(hi) + double(lo));
  }
}

// FP32 mirror: 0 for an absent entry, the value rounded to FP32 otherwise.
__global__ void __launch_bounds__(256) sparse_mirror_kernel(const double *__restrict__ x64, float *__restrict__ x32,
                                                            int64_t count) {
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < count; e += int64_t(gridDim.x) * blockDim.x) {
    const double v = x64[e];
    x32[e] = __double_as_longlong(v) == int64_t(kAbsent64) ? 0.f : float(v);
  }
}

// Rows in: x64 = src and its mirror x32 in one pass over src (device memory, or
// pinned host memory read over the host link); two entries per thread step.
__global__ void __launch_bounds__(256) sparse_load_kernel(const double2 *__restrict__ src, double2 *__restrict__ x64,
                                                          float2 *__restrict__ x32, int64_t pairs) {
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < pairs; e += int64_t(gridDim.x) * blockDim.x) {
    const double2 v = src[e];
    x64[e] = v;
    x32[e] = make_float2(__double_as_longlong(v.x) == int64_t(kAbsent64) ? 0.f : float(v.x),
                         __double_as_longlong(v.y) == int64_t(kAbsent64) ? 0.f : float(v.y));
  }
}

// Rows out: dst = src, two entries per thread step (dst: pinned host memory).
__global__ void __launch_bounds__(256) sparse_store_kernel(const double2 *__restrict__ src, double2 *__restrict__ dst,
                                                           int64_t pairs) {
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < pairs; e += int64_t(gridDim.x) * blockDim.x)
    dst[e] = src[e];
}

// Present entries (value != INT_MIN) of the FP64 rows, added to *present.
__global__ void __launch_bounds__(256) sparse_count_kernel(const double *__restrict__ x64, int64_t count,
                                                           unsigned long long *present) {
  unsigned long long c = 0;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < count; e += int64_t(gridDim.x) * blockDim.x)
    c += __double_as_longlong(x64[e]) != int64_t(kAbsent64);
  for (int m = 16; m >= 1; m >>= 1) c += __shfl_xor_sync(kFull, c, m);
  __shared__ unsigned long long part[8];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < int(blockDim.x >> 5); ++w) t += part[w];
    atomicAdd(present, t);
  }
}

// Order-preserving integer keys: a < b as floating-point values (with -0 = +0)
// iff key(a) < key(b).  INT_MIN, the absent marker, orders below every value
// of an embedding.
__device__ __forceinline__ uint64_t order_key(double v) {
  uint64_t b = uint64_t(__double_as_longlong(v));
  if (b == 0x8000000000000000ull) b = 0;  // -0 -> +0
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ uint64_t order_key(float v) {
  uint32_t b = __float_as_uint(v);
  if (b == 0x80000000u) b = 0;
  return uint64_t((b >> 31) ? ~b : (b | 0x80000000u)) << 32;
}

// Top-k pruning (preserveHighestK, sparse_embedding.hpp:745-767): in every row
// the dim - keep smallest values become absent; at equal values the lower dim
// goes first.  One warp per row, lane l holding dims [lN, lN + N).  The boundary
// between the two sets is found bit by bit from the highest bit in which the row's
// keys differ: a bit of the threshold is set when fewer than dim - keep keys lie
// below it, and the search ends as soon as exactly that many do, which for distinct
// values takes about as many bits as tell the two middle ones apart (a sorting
// network takes its 22 to 28 stages over all keys; with the count before it, 131,072
// rows at density 0.5: dim 128 289 -> 176 us, dim 256 922 -> 315 us).  Only when keys
// are equal at the boundary does it come to the last bit, and the lowest of those dims are dropped.
// T = double: the FP64 rows (absent = INT_MIN) and their mirror; T = float: the
// mirror alone.  With `present` set the rows are pruned only when
// floor(present / n) > keep (sparse_embedding.hpp:172-181), decided
// here so that the host need not wait.
template <int N, typename T>
__device__ __forceinline__ void load_values(T (&v)[N], const T *p) {
  constexpr int W = int(16 / sizeof(T)) < N ? int(16 / sizeof(T)) : N;  // values of a load
  struct alignas(W * sizeof(T)) Pack { T x[W]; };
#pragma unroll
  for (int i = 0; i < N; i += W) {
    const Pack t = *reinterpret_cast<const Pack *>(p + i);
#pragma unroll
    for (int k = 0; k < W; ++k) v[i + k] = t.x[k];
  }
}
template <int N, typename T>
__device__ __forceinline__ void store_values(T *p, const T (&v)[N]) {
  constexpr int W = int(16 / sizeof(T)) < N ? int(16 / sizeof(T)) : N;
  struct alignas(W * sizeof(T)) Pack { T x[W]; };
#pragma unroll
  for (int i = 0; i < N; i += W) {
    Pack t;
#pragma unroll
    for (int k = 0; k < W; ++k) t.x[k] = v[i + k];
    *reinterpret_cast<Pack *>(p + i) = t;
  }
}

// The warp's words w[t] with in(t): the largest *bound with at most `want` of them
// below it; returns how many lie below and stops early at exactly `want`.  Starts at
// the highest bit, or with kAll (every word is in) at the highest in which they differ.
template <int N, bool kAll, typename In>
__device__ __forceinline__ int boundary(const uint32_t (&w)[N], int want, uint32_t *bound, In in) {
  int bit = 31;
  uint32_t b = 0;
  if constexpr (kAll) {
    const uint32_t first = __shfl_sync(kFull, w[0], 0);
    uint32_t diff = 0;
#pragma unroll
    for (int t = 0; t < N; ++t) diff |= w[t] ^ first;
    diff = __reduce_or_sync(kFull, diff);
    bit = 31 - __clz(int(diff));  // -1: all the same
    b = bit == 31 ? 0u : bit < 0 ? first : first & ~((2u << bit) - 1);
  }
  int below = 0;
  for (; bit >= 0; --bit) {
    const uint32_t cand = b | (1u << bit);
    int c = 0;
#pragma unroll
    for (int t = 0; t < N; ++t) c += in(t) && w[t] < cand;
    c = __reduce_add_sync(kFull, c);
    if (c > want) continue;
    b = cand;
    below = c;
    if (c == want) break;
  }
  *bound = b;
  return below;
}

template <int D, typename T>
__global__ void __launch_bounds__(256) sparse_prune_kernel(T *xs, float *x32, int64_t n, int32_t keep,
                                                           const unsigned long long *present) {
  constexpr int N = D / 32;
  if (present && static_cast<int>(double(*present) / double(n)) <= keep) return;
  const int lane = threadIdx.x & 31;
  const int nullify = D - keep;
  if (nullify <= 0) return;
  for (int64_t row = blockIdx.x * int64_t(blockDim.x >> 5) + (threadIdx.x >> 5); row < n;
       row += int64_t(gridDim.x) * (blockDim.x >> 5)) {
    T *xr = xs + row * D + lane * N;
    T val[N];
    load_values<N>(val, xr);
    uint64_t key[N];
#pragma unroll
    for (int t = 0; t < N; ++t) key[t] = order_key(val[t]);
    // keys below `bound` are dropped, and the first `ties` of those equal to it: the
    // high words first, the low ones only among keys equal in the high word
    uint64_t bound = ~uint64_t(0);
    int ties = D;
    if (nullify < D) {
      uint32_t hi[N];
#pragma unroll
      for (int t = 0; t < N; ++t) hi[t] = uint32_t(key[t] >> 32);
      int want = nullify;
      uint32_t bhi = 0, blo = 0;
      want -= boundary<N, true>(hi, want, &bhi, [](int) { return true; });
      if (want > 0) {
        uint32_t lo[N];
#pragma unroll
        for (int t = 0; t < N; ++t) lo[t] = uint32_t(key[t]);
        want -= boundary<N, false>(lo, want, &blo, [&](int t) { return hi[t] == bhi; });
      }
      bound = (uint64_t(bhi) << 32) | blo;
      ties = want;
    }
    int rank = 0;  // keys equal to `bound` in lower dims
    if (ties > 0) {
      int own = 0;
#pragma unroll
      for (int t = 0; t < N; ++t) own += key[t] == bound;
      rank = own;
#pragma unroll
      for (int m = 1; m < 32; m <<= 1) {
        const int up = __shfl_up_sync(kFull, rank, m);
        if (lane >= m) rank += up;
      }
      rank -= own;
    }
    float mirror[N];
#pragma unroll
    for (int t = 0; t < N; ++t) {
      const bool drop = key[t] < bound || (key[t] == bound && rank++ < ties);
      if constexpr (sizeof(T) == 8) {
        mirror[t] = drop || __double_as_longlong(val[t]) == int64_t(kAbsent64) ? 0.f : float(val[t]);
        if (drop) val[t] = __longlong_as_double(int64_t(kAbsent64));
      } else if (drop) {
        val[t] = 0.f;  // xs is the mirror itself
      }
    }
    store_values<N>(xr, val);
    if constexpr (sizeof(T) == 8) store_values<N>(x32 + row * D + lane * N, mirror);
  }
}

// After the last iteration absent entries become 0 (the final CSR build with
// clear_dense_collector, cpp/core/distributed_mat.hpp:63-91).
// Two entries per thread step; a pair is written back only when it held one.
__global__ void __launch_bounds__(256) sparse_finalize_kernel(double2 *__restrict__ x64, int64_t pairs) {
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < pairs; e += int64_t(gridDim.x) * blockDim.x) {
    double2 v = x64[e];
    const bool ax = __double_as_longlong(v.x) == int64_t(kAbsent64);
    const bool ay = __double_as_longlong(v.y) == int64_t(kAbsent64);
    if (ax) v.x = 0.0;
    if (ay) v.y = 0.0;
    if (ax || ay) x64[e] = v;
  }
}

template <typename T>
cudaError_t prune_dispatch(int dim, T *xs, float *x32, int64_t n, int32_t keep, const unsigned long long *present,
                           cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int grid = int(n / 8 + 1 < 152 * 16 ? n / 8 + 1 : 152 * 16);
  switch (dim) {
    case 32: sparse_prune_kernel<32, T><<<grid, 256, 0, s>>>(xs, x32, n, keep, present); break;
    case 64: sparse_prune_kernel<64, T><<<grid, 256, 0, s>>>(xs, x32, n, keep, present); break;
    case 128: sparse_prune_kernel<128, T><<<grid, 256, 0, s>>>(xs, x32, n, keep, present); break;
    case 256: sparse_prune_kernel<256, T><<<grid, 256, 0, s>>>(xs, x32, n, keep, present); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_sparse_attract(int dim, const SpmmArgs &a, cudaStream_t s) {
  const int64_t grid = (a.n_items + kPlainWarps - 1) / kPlainWarps;
  if (grid == 0) return cudaSuccess;
  if (grid >= (int64_t(1) << 31)) return cudaErrorInvalidValue;
  switch (dim) {
    case 32: sparse_attract_kernel<32><<<unsigned(grid), kPlainWarps * 32, 0, s>>>(a); break;
    case 64: sparse_attract_kernel<64><<<unsigned(grid), kPlainWarps * 32, 0, s>>>(a); break;
    case 128: sparse_attract_kernel<128><<<unsigned(grid), kPlainWarps * 32, 0, s>>>(a); break;
    case 256: sparse_attract_kernel<256><<<unsigned(grid), kPlainWarps * 32, 0, s>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_sparse_collect(const float *y, double *coll, int64_t n, int32_t batch, int32_t dim,
                                  cudaStream_t s) {
  const int64_t slots = int64_t(batch) * dim;
  if (slots <= 0) return cudaSuccess;
  sparse_collect_kernel<<<elementwise_grid(slots), 256, 0, s>>>(y, coll, n, batch, dim);
  return cudaGetLastError();
}

cudaError_t launch_sparse_mirror(const double *x64, float *x32, int64_t count, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  sparse_mirror_kernel<<<elementwise_grid(count), 256, 0, s>>>(x64, x32, count);
  return cudaGetLastError();
}

cudaError_t launch_sparse_load(const double *src, double *x64, float *x32, int64_t count, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  if ((count & 1) || (reinterpret_cast<uintptr_t>(src) & 15)) return cudaErrorInvalidValue;
  sparse_load_kernel<<<elementwise_grid(count / 2), 256, 0, s>>>(
      reinterpret_cast<const double2 *>(src), reinterpret_cast<double2 *>(x64), reinterpret_cast<float2 *>(x32),
      count / 2);
  return cudaGetLastError();
}

cudaError_t launch_sparse_store(const double *src, double *dst, int64_t count, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  if ((count & 1) || (reinterpret_cast<uintptr_t>(dst) & 15)) return cudaErrorInvalidValue;
  sparse_store_kernel<<<elementwise_grid(count / 2), 256, 0, s>>>(reinterpret_cast<const double2 *>(src),
                                                                  reinterpret_cast<double2 *>(dst), count / 2);
  return cudaGetLastError();
}

cudaError_t launch_sparse_count(const double *x64, int64_t count, unsigned long long *present, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  sparse_count_kernel<<<elementwise_grid(count), 256, 0, s>>>(x64, count, present);
  return cudaGetLastError();
}

cudaError_t launch_sparse_prune_f64(int dim, double *x64, float *x32, int64_t n, int32_t keep,
                                    const unsigned long long *present, cudaStream_t s) {
  return prune_dispatch<double>(dim, x64, x32, n, keep, present, s);
}

cudaError_t launch_sparse_prune_f32(int dim, float *x32, int64_t n, int32_t keep, cudaStream_t s) {
  return prune_dispatch<float>(dim, x32, x32, n, keep, nullptr, s);
}

cudaError_t launch_sparse_finalize(double *x64, int64_t count, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  if (count & 1) return cudaErrorInvalidValue;  // n x dim with dim a multiple of 32
  sparse_finalize_kernel<<<elementwise_grid(count / 2), 256, 0, s>>>(reinterpret_cast<double2 *>(x64), count / 2);
  return cudaGetLastError();
}

}  // namespace de
