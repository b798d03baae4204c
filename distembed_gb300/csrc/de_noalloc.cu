// One minibatch of the FP32 plain embedding step on caller-owned device memory,
// with no device allocation at all.
//
// Who needs this: code that is not allowed to call cudaMalloc / cudaFree.  A host
// framework that owns the whole device heap through its own pool allocator
// (an inference server, another training framework calling this as a plug-in
// operator) cannot let a library allocate behind its back: the memory would be
// invisible to its accounting and fragment its pool.  A latency-bound request
// loop cannot afford the implicit device-wide synchronisation that cudaMalloc
// and cudaFree bring.  Those callers allocate every input and output themselves
// and call this entry point, which only launches kernels.
//
// The only working memory is the file-scope device array below, of a fixed size
// that every GPU loading the library holds until the process exits.  It keeps the
// staged rows of one minibatch (at most kNoAllocMaxRowFloats floats, i.e.
// batch_size * dim <= 1,048,576) and one FP64 loss partial per row.  Both are
// fully rewritten by every call before they are read, so nothing has to start at
// zero; every call shares them, so two calls that overlap on the GPU (different
// streams, or different host threads without ordering) race and corrupt each
// other.
//
// A row's attractive pass in CSR order and its repulsive pass over the minibatch's
// negatives (cpp/algo/algo.hpp:521-584, 586-649) are spread over the warps of one
// CTA, the result is staged and committed to x by a second launch
// (algo.hpp:651-666), so every read in the first launch sees the pre-minibatch
// values as the reference's does.
#include <cuda_runtime.h>

#include <string>

#include "../../include/distembed_gb300.h"
#include "de_device.cuh"

namespace de {
void set_thread_error(const std::string &msg);  // de_runtime.cpp
}

namespace {

constexpr int64_t kNoAllocMaxRowFloats = int64_t(1) << 20;  // 4 MiB of staged rows
constexpr int64_t kNoAllocMaxRows = 65536;                  // loss partials (FP64)
constexpr size_t kNoAllocBytes = size_t(kNoAllocMaxRowFloats) * sizeof(float) + size_t(kNoAllocMaxRows) * sizeof(double);

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr unsigned kFullMask = 0xffffffffu;

struct NoAllocArgs {
  int32_t n;
  const int32_t *rowptr;
  const int32_t *col;
  float *x;
  int32_t base, rows, rep_rows;
  const int32_t *negs;
  int32_t ns;
  int32_t skip;  // column to drop (n - 1 when reproducing the reference), else -1
  float lr, bound;
  float *staged;    // [rows, dim] inside the scratch array
  double *partial;  // [rows] inside the scratch array
  double *loss;     // nullable: this minibatch's loss
};

__device__ __forceinline__ float nclip(float v, float b) { return v > b ? b : (v < -b ? -b : v); }

// Components of a row held by a lane: with wide loads (x 16-byte aligned, so every
// row is) dev::Frag's, else l, l + 32, ... by 4-byte loads.  Ordinary loads, here and
// for the graph and the draws: the launch before may have written any of them, and a
// load through the read-only path may be moved ahead of the wait for it.
template <int D, bool kWide>
__device__ __forceinline__ void nload(de::dev::Frag<D> &f, const float *row, int lane) {
  constexpr int N = D / 32;
  if constexpr (kWide && N == 2) {
    const float2 t = reinterpret_cast<const float2 *>(row)[lane];
    f.v[0] = t.x; f.v[1] = t.y;
  } else if constexpr (kWide && N >= 4) {
#pragma unroll
    for (int h = 0; h < N / 4; ++h) {
      const float4 t = reinterpret_cast<const float4 *>(row)[32 * h + lane];
      f.v[4 * h] = t.x; f.v[4 * h + 1] = t.y; f.v[4 * h + 2] = t.z; f.v[4 * h + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int t = 0; t < N; ++t) f.v[t] = row[lane + 32 * t];
  }
}

// The pairs of x_i with up to U rows (lane u of `ids`: row u, -1 = none), all
// loads issued before the first is used; the U squared distances are reduced
// together (multi_warp_sum), so a lane divides for one pair.
template <int D, int U, bool kWide, bool kAttract>
__device__ __forceinline__ void nforces(const NoAllocArgs &a, de::dev::Frag<D> &acc, const de::dev::Frag<D> &xi,
                                        int ids, bool want_loss, double &loss, int lane) {
  constexpr int N = D / 32, L = de::dev::Log2<U>::value;
  de::dev::Frag<D> xn[U];
  unsigned mask = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int nb = __shfl_sync(kFullMask, ids, u);
    if (nb >= 0) {
      nload<D, kWide>(xn[u], a.x + size_t(nb) * D, lane);
      mask |= 1u << u;
    } else {
      xn[u] = xi;
    }
  }
  if (mask == 0) return;
  float p[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    p[u] = 0.f;
#pragma unroll
    for (int t = 0; t < N; ++t) {
      xn[u].v[t] = xi.v[t] - xn[u].v[t];
      p[u] = fmaf(xn[u].v[t], xn[u].v[t], p[u]);
    }
  }
  const float r = de::dev::multi_warp_sum<U>(p, lane);
  const int v = (lane >> (5 - L)) & (U - 1);
  float c = kAttract ? -2.0f / (1.0f + r) : 2.0f / ((r + 1e-6f) * (1.0f + r));
  if (!((mask >> v) & 1u)) c = 0.f;
  else if (want_loss && (lane & ((32 >> L) - 1)) == 0)
    loss += kAttract ? double(log1pf(r)) : double(logf((1.0f + r) / (r + 1e-6f)));
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const float cu = __shfl_sync(kFullMask, c, u << (5 - L));
#pragma unroll
    for (int t = 0; t < N; ++t) acc.v[t] = fmaf(a.lr, nclip(xn[u].v[t] * cu, a.bound), acc.v[t]);
  }
}

// One row per CTA of W warps: the row's CSR entries and then its negatives in
// groups of U, group q on warp q % W; the warps' sums are added in warp order.
// A minibatch is too small to fill the GPU with bytes, so a call takes as long as
// the longest chain of dependent loads.  Here a row of up to U W pairs is one
// round: row pointer, column ids, rows.  Measured on the epoch of a 2,000-vertex
// kNN graph (8 calls of 256 rows of about 14 neighbours, dim 64, 5 negatives):
// 305 us with a warp per row and one neighbour in flight, 56 us so (7 us a call, both
// launches in it).
template <int D, int U, int W, bool kWide>
__global__ void __launch_bounds__(W * 32) noalloc_rows_kernel(const NoAllocArgs a) {
  constexpr int N = D / 32;
  __shared__ float sums[W][D];
  __shared__ double losses[W];
  de::dev::pdl_wait();
  de::dev::pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.x, row = a.base + r;
  const int e0 = a.rowptr[row], deg = max(a.rowptr[row + 1] - e0, 0);  // a pointer that falls: no entries
  de::dev::Frag<D> xi, acc;
  nload<D, kWide>(xi, a.x + size_t(row) * D, lane);
  acc.zero();
  const bool want_loss = a.loss != nullptr;
  double loss = 0.0;
  const int ge = (deg + U - 1) / U;
  const int groups = ge + (r < a.rep_rows ? (a.ns + U - 1) / U : 0);
  for (int q = warp; q < groups; q += W) {
    if (q < ge) {
      const int k = q * U + lane;
      int id = lane < U && k < deg ? a.col[e0 + k] : -1;
      if (id == a.skip) id = -1;
      nforces<D, U, kWide, true>(a, acc, xi, id, want_loss, loss, lane);
    } else {
      const int k = (q - ge) * U + lane;
      int id = lane < U && k < a.ns ? a.negs[k] : -1;
      if (id >= a.n) id = -1;  // a draw equal to n contributes nothing
      nforces<D, U, kWide, false>(a, acc, xi, id, want_loss, loss, lane);
    }
  }
#pragma unroll
  for (int t = 0; t < N; ++t) sums[warp][t * 32 + lane] = acc.v[t];
  if (want_loss) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(kFullMask, loss, o);
    if (lane == 0) losses[warp] = loss;
  }
  __syncthreads();
  if (warp != 0) return;
  acc.zero();
#pragma unroll
  for (int w = 0; w < W; ++w)
#pragma unroll
    for (int t = 0; t < N; ++t) acc.v[t] += sums[w][t * 32 + lane];
#pragma unroll
  for (int t = 0; t < N; ++t) acc.v[t] = xi.v[t] + acc.v[t];
  if constexpr (kWide) {
    de::dev::store<D, false>(acc, a.staged + size_t(r) * D, lane);
  } else {
#pragma unroll
    for (int t = 0; t < N; ++t) a.staged[size_t(r) * D + lane + 32 * t] = acc.v[t];
  }
  if (want_loss && lane == 0) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < W; ++w) s += losses[w];
    a.partial[r] = s;
  }
}

// x rows = staged rows, and the minibatch's loss.  Bound by its launch: 64 KB at
// 256 rows, dim 64.
template <bool kWide>
__global__ void __launch_bounds__(256) noalloc_commit_kernel(const NoAllocArgs a, int64_t total, int64_t first) {
  de::dev::pdl_trigger();
  de::dev::pdl_wait();
  const int64_t i0 = blockIdx.x * int64_t(blockDim.x) + threadIdx.x, step = int64_t(gridDim.x) * blockDim.x;
  if constexpr (kWide) {
    for (int64_t i = i0; i < total / 4; i += step)
      reinterpret_cast<float4 *>(a.x + first)[i] = reinterpret_cast<const float4 *>(a.staged)[i];
  } else {
    for (int64_t i = i0; i < total; i += step) a.x[first + i] = a.staged[i];
  }
  if (blockIdx.x != 0 || a.loss == nullptr) return;
  __shared__ double red[256];
  double s = 0.0;
  for (int i = threadIdx.x; i < a.rows; i += 256) s += a.partial[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *a.loss = red[0];
}

// Both kernels are launched with a programmatic dependency on the kernel before
// them in the stream: each waits for that kernel's end before it reads anything
// (griddepcontrol.wait comes first), so only its launch overlaps.
template <typename... P, typename... A>
cudaError_t nlaunch(void (*k)(P...), int grid, int block, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

// Eight warps a row, so that the longest rows finish sooner, where every row's CTA then
// still is resident (the registers of 256 threads: six CTAs an SM at dim 32, five at 64,
// three at 128 and 256); four warps beyond.  Time of a call with four warps over that with
// eight, rows of about 14 / 40 entries: dim 256, 128 rows 1.00 / 1.23, 456 1.01 / 1.21, 912
// 0.93 / 0.93, 1216 0.93 / 0.96; dim 128, 456 rows 0.99 / 1.03, 912 0.92 / 0.91, 1216 0.82 /
// 0.96, 2432 0.70 / 0.89; dim 64, 760 rows 1.01 / 0.99, 1216 0.96 / 0.96, 2432 0.82 / 0.96;
// dim 32, 912 rows 0.99 / 1.03, 1216 0.98 / 0.90, 2432 0.88 / 0.97.
template <int D>
constexpr int kWideTeamRows = 152 * (D == 32 ? 6 : D == 64 ? 5 : 3);

template <int D, bool kWide>
cudaError_t nrun(const NoAllocArgs &a, cudaStream_t s) {
  constexpr int U = D == 256 ? 4 : 8;
  cudaError_t e = a.rows <= kWideTeamRows<D> ? nlaunch(noalloc_rows_kernel<D, U, 8, kWide>, a.rows, 256, s, a)
                                          : nlaunch(noalloc_rows_kernel<D, U, 4, kWide>, a.rows, 128, s, a);
  if (e != cudaSuccess) return e;
  const int64_t total = int64_t(a.rows) * D, per = 256 * (kWide ? 4 : 1);
  const int grid = int((total + per - 1) / per < 152 * 4 ? (total + per - 1) / per : 152 * 4);
  return nlaunch(noalloc_commit_kernel<kWide>, grid, 256, s, a, total, int64_t(a.base) * D);
}

// Device address of the scratch array in the current device's context.  It is
// looked up on every call (a lookup allocates nothing): after a device reset, or
// under another context on the same device, the module is loaded again at a new
// address, and a cached address would point at memory of the old context.
int scratch_for_current_device(void **out) {
  void *ptr = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
  if (e != cudaSuccess) {
    de::set_thread_error(std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    return DE_ERR_CUDA;
  }
  *out = ptr;
  return DE_OK;
}

}  // namespace

extern "C" int de_minibatch_noalloc(int64_t n, const int32_t *rowptr, const int32_t *col, int32_t dim, float *x,
                                    int32_t batch_id, int32_t batch_size, const int32_t *negs, int32_t ns,
                                    int32_t rep_rows, int32_t skip_last_vertex, float lr, float max_bound,
                                    double *loss, void *stream) {
  if (n <= 0 || n >= (int64_t(1) << 31) - 1 || !rowptr || !col || !x || batch_size <= 0 || batch_id < 0 ||
      ns < 0 || (ns > 0 && !negs) || !(max_bound > 0)) {
    de::set_thread_error("de_minibatch_noalloc: bad argument");
    return DE_ERR_INVALID;
  }
  if (dim != 32 && dim != 64 && dim != 128 && dim != 256) {
    de::set_thread_error("de_minibatch_noalloc: dim must be 32, 64, 128 or 256");
    return DE_ERR_INVALID;
  }
  const int64_t base = int64_t(batch_id) * batch_size;
  if (base >= n) {
    de::set_thread_error("de_minibatch_noalloc: batch_id beyond the last minibatch");
    return DE_ERR_INVALID;
  }
  const int64_t rows = (n - base < batch_size) ? n - base : batch_size;
  if (rows * dim > kNoAllocMaxRowFloats || rows > kNoAllocMaxRows) {
    de::set_thread_error("de_minibatch_noalloc: minibatch too large for the fixed scratch: rows * dim must be "
                         "<= 1048576 (e.g. 8192 rows at dim 128)");
    return DE_ERR_INVALID;
  }
  void *scratch = nullptr;
  if (int rc = scratch_for_current_device(&scratch)) return rc;
  NoAllocArgs a{};
  a.n = int32_t(n);
  a.rowptr = rowptr;
  a.col = col;
  a.x = x;
  a.base = int32_t(base);
  a.rows = int32_t(rows);
  a.rep_rows = rep_rows < 0 ? 0 : (rep_rows > rows ? int32_t(rows) : rep_rows);
  a.negs = negs;
  a.ns = ns;
  a.skip = skip_last_vertex ? int32_t(n - 1) : -1;
  a.lr = lr;
  a.bound = max_bound;
  a.staged = static_cast<float *>(scratch);
  a.partial = reinterpret_cast<double *>(static_cast<unsigned char *>(scratch) + kNoAllocMaxRowFloats * sizeof(float));
  a.loss = loss;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // wide loads and stores need x on a 16-byte boundary; a caller's x need not be
  const bool wide = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  cudaError_t e = cudaSuccess;
  switch (dim) {
    case 32: e = wide ? nrun<32, true>(a, s) : nrun<32, false>(a, s); break;
    case 64: e = wide ? nrun<64, true>(a, s) : nrun<64, false>(a, s); break;
    case 128: e = wide ? nrun<128, true>(a, s) : nrun<128, false>(a, s); break;
    default: e = wide ? nrun<256, true>(a, s) : nrun<256, false>(a, s); break;
  }
  if (e != cudaSuccess) {
    de::set_thread_error(std::string("de_minibatch_noalloc launch: ") + cudaGetErrorString(e));
    return DE_ERR_CUDA;
  }
  return DE_OK;
}
