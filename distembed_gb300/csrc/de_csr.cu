// COO -> CSR on the GPU: the CSR the host reader builds (cpp/io/parrallel_IO.hpp:31-88
// and the COO -> CSR of cpp/core/csr_local.hpp:37-125 at one rank, with columns
// ascending within a row), from keys row * cols + col: radix sort of the keys,
// merge of equal keys, then per row the first key of the row by binary search
// (row pointers) and per key its column.  The parse of a MatrixMarket file stays
// on the host (de_io.cpp); the sort, which dominates the host reader on large
// graphs, runs here.  COO entries are checked and turned into keys here as well,
// and the CSR stays on the GPU until it is copied out: 2.4 M entries mirrored to a
// CSR of 4.2 M took 13 ms when the host built the keys one by one and the result
// went through a host copy (see de_coo_to_csr for what it takes so).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/distembed_gb300.h"
#include "de_internal.h"

// rowptr[rows + 1] and col[nnz] on GPU `device`; without entries nothing is
// allocated and every row pointer is 0.
struct de_csr {
  int64_t rows = 0, cols = 0, nnz = 0;
  int32_t device = 0;
  int64_t *d_rowptr = nullptr, *d_col = nullptr;  // one allocation, d_rowptr first
  cudaStream_t st = nullptr;                      // the one it was built on, for its copies out
};

namespace de {

void set_thread_error(const std::string &msg);  // de_runtime.cpp
int parse_mm(const char *path, int64_t *rows, int64_t *cols, std::vector<int64_t> &key);  // de_io.cpp

namespace {

int csr_fail(int rc, const std::string &m) {
  set_thread_error(m);
  return rc;
}

// rowptr[r] = first position of a key >= r * cols (r = 0 .. rows).
__global__ void row_pointers_kernel(const uint64_t *__restrict__ key, int64_t m, int64_t rows, int64_t cols,
                                    int64_t *__restrict__ rowptr) {
  for (int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r <= rows; r += int64_t(gridDim.x) * blockDim.x) {
    const uint64_t target = uint64_t(r) * uint64_t(cols);
    int64_t lo = 0, hi = m;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (key[mid] < target) lo = mid + 1;
      else hi = mid;
    }
    rowptr[r] = lo;
  }
}

__global__ void columns_kernel(const uint64_t *__restrict__ key, int64_t m, int64_t cols, int64_t *__restrict__ col) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < m; i += int64_t(gridDim.x) * blockDim.x)
    col[i] = int64_t(key[i] % uint64_t(cols));
}

// Keys of COO entries: key[e] = row * cols + col and, mirrored, key[m + e] = col *
// cols + row (a diagonal entry gives its own key twice, which the merge removes).
// An entry outside the matrix writes key 0 and lowers *bad to 2 e (the entry
// itself) or 2 e + 1 (only its mirror image).
__global__ void coo_keys_kernel(const int64_t *__restrict__ row, const int64_t *__restrict__ col, int64_t m,
                                int64_t rows, int64_t cols, int mirror, uint64_t *__restrict__ key,
                                unsigned long long *bad) {
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < m; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = row[e], j = col[e];
    uint64_t k = 0, t = 0;
    if (i < 0 || j < 0 || i >= rows || j >= cols) {
      atomicMin(bad, 2ull * uint64_t(e));
    } else {
      k = uint64_t(i) * uint64_t(cols) + uint64_t(j);
      t = k;
      if (mirror && i != j) {
        if (j >= rows || i >= cols) atomicMin(bad, 2ull * uint64_t(e) + 1);
        else t = uint64_t(j) * uint64_t(cols) + uint64_t(i);
      }
    }
    key[e] = k;
    if (mirror) key[m + e] = t;
  }
}

// dst = src as int32; counters[0] counts the columns outside [0, n), counters[1] those
// equal to n - 1.
__global__ void __launch_bounds__(256) check_columns_kernel(const int64_t *__restrict__ src, int32_t *__restrict__ dst,
                                                            int64_t count, int64_t n, unsigned long long *counters) {
  unsigned bad = 0, last = 0;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < count; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t c = src[i];
    dst[i] = int32_t(c);
    bad += c < 0 || c >= n;
    last += c == n - 1;
  }
  bad = __reduce_add_sync(0xffffffffu, bad);
  last = __reduce_add_sync(0xffffffffu, last);
  if ((threadIdx.x & 31) == 0) {
    if (bad) atomicAdd(counters, static_cast<unsigned long long>(bad));
    if (last) atomicAdd(counters + 1, static_cast<unsigned long long>(last));
  }
}

int grid_for(int64_t n) { return int(std::min<int64_t>((n + 255) / 256 + 1, 152 * 16)); }

struct DeviceBuffers {
  void *block = nullptr, *result = nullptr;
  cudaStream_t st = nullptr;
  ~DeviceBuffers() {
    if (st) cudaStreamSynchronize(st);
    if (block) cudaFree(block);
    if (result) cudaFree(result);
    if (st) cudaStreamDestroy(st);
  }
};

#define CSR_CUDA(call)                                                              \
  do {                                                                              \
    const cudaError_t e_ = (call);                                                  \
    if (e_ != cudaSuccess) return csr_fail(DE_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// The entries of a matrix on the host: keys, or (keys null) coordinates.
struct Entries {
  const int64_t *keys = nullptr;
  const int64_t *row = nullptr, *col = nullptr;
  int64_t count = 0;
  bool mirror = false;
};

int entry_error(bool mirrored) {
  return csr_fail(DE_ERR_INVALID, mirrored ? "mirrored entry outside the matrix" : "COO entry outside the matrix");
}

// The first entry outside the matrix, as coo_keys_kernel finds it, on the host.
int check_entries(const Entries &in, int64_t rows, int64_t cols) {
  for (int64_t e = 0; !in.keys && e < in.count; ++e) {
    const int64_t i = in.row[e], j = in.col[e];
    if (i < 0 || j < 0 || i >= rows || j >= cols) return entry_error(false);
    if (in.mirror && i != j && (j >= rows || i >= cols)) return entry_error(true);
  }
  return DE_OK;
}

// Entries -> CSR in `out`.
int build_on_gpu(int32_t device, int64_t rows, int64_t cols, const Entries &in, de_csr *out) {
  out->rows = rows;
  out->cols = cols;
  out->device = device;
  if (in.count == 0) return DE_OK;
  const int64_t n = in.count * (in.mirror ? 2 : 1);  // keys
  if (n >= (int64_t(1) << 31)) return csr_fail(DE_ERR_UNSUPPORTED, "at most 2^31 - 1 entries");
  if (const cudaError_t e = cudaSetDevice(device); e != cudaSuccess) {
    if (int rc = check_entries(in, rows, cols)) return rc;
    return csr_fail(DE_ERR_CUDA, std::string("cudaSetDevice: ") + cudaGetErrorString(e));
  }
  DeviceBuffers b;
  CSR_CUDA(cudaStreamCreateWithFlags(&b.st, cudaStreamNonBlocking));
  // bits of the largest key rows * cols - 1
  const uint64_t top = uint64_t(rows) * uint64_t(cols) - 1;
  int end_bit = 1;
  while (end_bit < 64 && (top >> end_bit) != 0) ++end_bit;
  size_t sort_bytes = 0, uniq_bytes = 0;
  uint64_t *nil = nullptr;
  int64_t *num_nil = nullptr;
  CSR_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, sort_bytes, nil, nil, n, 0, end_bit, b.st));
  CSR_CUDA(cub::DeviceSelect::Unique(nullptr, uniq_bytes, nil, nil, num_nil, n, b.st));
  // one allocation: keys, sorted keys (before them the coordinates), the two
  // counters and the temporary storage
  const size_t nb = size_t(n) * sizeof(uint64_t), sorted = std::max(nb, in.keys ? nb : 2 * size_t(in.count) * 8);
  auto round = [](size_t v) { return (v + 255) & ~size_t(255); };
  const size_t off_sorted = round(nb), off_count = off_sorted + round(sorted), off_temp = off_count + 256;
  CSR_CUDA(cudaMalloc(&b.block, off_temp + std::max(sort_bytes, uniq_bytes)));
  char *base = static_cast<char *>(b.block);
  uint64_t *d_key = reinterpret_cast<uint64_t *>(base), *d_sorted = reinterpret_cast<uint64_t *>(base + off_sorted);
  int64_t *d_count = reinterpret_cast<int64_t *>(base + off_count);
  unsigned long long *d_bad = reinterpret_cast<unsigned long long *>(d_count + 1);
  void *temp = base + off_temp;
  CSR_CUDA(cudaMemsetAsync(d_count, 0xff, 2 * sizeof(int64_t), b.st));
  if (in.keys) {
    CSR_CUDA(cudaMemcpyAsync(d_key, in.keys, nb, cudaMemcpyHostToDevice, b.st));
  } else {
    int64_t *d_row = reinterpret_cast<int64_t *>(d_sorted), *d_colin = d_row + in.count;
    CSR_CUDA(cudaMemcpyAsync(d_row, in.row, size_t(in.count) * 8, cudaMemcpyHostToDevice, b.st));
    CSR_CUDA(cudaMemcpyAsync(d_colin, in.col, size_t(in.count) * 8, cudaMemcpyHostToDevice, b.st));
    coo_keys_kernel<<<grid_for(in.count), 256, 0, b.st>>>(d_row, d_colin, in.count, rows, cols, in.mirror ? 1 : 0,
                                                          d_key, d_bad);
    CSR_CUDA(cudaGetLastError());
  }
  CSR_CUDA(cub::DeviceRadixSort::SortKeys(temp, sort_bytes, d_key, d_sorted, n, 0, end_bit, b.st));
  CSR_CUDA(cub::DeviceSelect::Unique(temp, uniq_bytes, d_sorted, d_key, d_count, n, b.st));
  int64_t found[2] = {0, 0};  // merged keys; first bad entry, all ones when none
  CSR_CUDA(cudaMemcpyAsync(found, d_count, sizeof(found), cudaMemcpyDeviceToHost, b.st));
  CSR_CUDA(cudaStreamSynchronize(b.st));
  if (found[1] != -1) return entry_error(found[1] & 1);
  const int64_t m = found[0];
  CSR_CUDA(cudaMalloc(&b.result, size_t(rows + 1 + m) * sizeof(int64_t)));
  int64_t *d_rowptr = static_cast<int64_t *>(b.result), *d_col = d_rowptr + rows + 1;
  row_pointers_kernel<<<grid_for(rows + 1), 256, 0, b.st>>>(d_key, m, rows, cols, d_rowptr);
  CSR_CUDA(cudaGetLastError());
  columns_kernel<<<grid_for(m), 256, 0, b.st>>>(d_key, m, cols, d_col);
  CSR_CUDA(cudaGetLastError());
  CSR_CUDA(cudaStreamSynchronize(b.st));
  out->nnz = m;
  out->d_rowptr = d_rowptr;
  out->d_col = d_col;
  out->st = b.st;
  b.result = nullptr;  // the CSR's now, with the stream
  b.st = nullptr;
  return DE_OK;
}

// Touches the pages of a destination of the caller's on several host threads: a
// copy from the GPU into fresh memory otherwise takes their page faults one by one
// (36 MB: 2.4 to 5 ms against 0.2 ms into memory that was written before).
void touch_pages(void *p, size_t bytes) {
  constexpr size_t kPage = 4096;
  char *c = static_cast<char *>(p);
  const int64_t pages = int64_t((bytes + kPage - 1) / kPage);
  parallel_indices(pages, 256, [&](int64_t i) { *reinterpret_cast<volatile char *>(c + size_t(i) * kPage) = 0; });
}

}  // namespace

cudaError_t launch_columns(const int64_t *src, int32_t *dst, int64_t count, int64_t n, unsigned long long *counters,
                           cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  check_columns_kernel<<<grid_for(count), 256, 0, s>>>(src, dst, count, n, counters);
  return cudaGetLastError();
}

}  // namespace de

extern "C" {

// 2.4 M entries with their mirror images to a CSR of 4.2 M (262,144 rows), from host
// arrays to fresh host arrays: 13.3 -> 3.5 ms, 0.35 ms of it in the kernels (five
// radix passes 0.25 ms); the rest is the copies, the allocations and the page faults
// of the result.
int de_coo_to_csr(int64_t rows, int64_t cols, const int64_t *row_idx, const int64_t *col_idx, int64_t nnz,
                  int32_t mirror, int32_t device, de_csr **out) {
  if (!out) return de::csr_fail(DE_ERR_INVALID, "out is NULL");
  *out = nullptr;
  if (rows <= 0 || cols <= 0 || nnz < 0 || (nnz > 0 && (!row_idx || !col_idx)) || rows >= (int64_t(1) << 31) ||
      cols >= (int64_t(1) << 31))
    return de::csr_fail(DE_ERR_INVALID, "bad COO arguments");
  de::Entries in;
  in.row = row_idx;
  in.col = col_idx;
  in.count = nnz;
  in.mirror = mirror != 0;
  // The GPU gives a diagonal entry two keys.  Where that alone would pass the limit
  // on keys, the host builds them.
  std::vector<int64_t> keys;
  if (in.mirror && nnz >= (int64_t(1) << 30)) {
    if (int rc = de::check_entries(in, rows, cols)) return rc;
    for (int64_t e = 0; e < nnz; ++e) {
      keys.push_back(row_idx[e] * cols + col_idx[e]);
      if (row_idx[e] != col_idx[e]) keys.push_back(col_idx[e] * cols + row_idx[e]);
    }
    in = de::Entries{};
    in.keys = keys.data();
    in.count = int64_t(keys.size());
  } else if (nnz >= (int64_t(1) << 31)) {
    if (int rc = de::check_entries(in, rows, cols)) return rc;
  }
  auto c = new de_csr;
  if (int rc = de::build_on_gpu(device, rows, cols, in, c)) {
    delete c;
    return rc;
  }
  *out = c;
  return DE_OK;
}

int de_mm_read_gpu(const char *path, int32_t device, de_csr **out) {
  if (!path || !out) return de::csr_fail(DE_ERR_INVALID, "NULL argument");
  *out = nullptr;
  int64_t rows = 0, cols = 0;
  std::vector<int64_t> keys;
  if (int rc = de::parse_mm(path, &rows, &cols, keys)) return rc;
  de::Entries in;
  in.keys = keys.data();
  in.count = int64_t(keys.size());
  auto c = new de_csr;
  if (int rc = de::build_on_gpu(device, rows, cols, in, c)) {
    delete c;
    return rc;
  }
  *out = c;
  return DE_OK;
}

int de_csr_info(const de_csr *c, int64_t *rows, int64_t *cols, int64_t *nnz) {
  if (!c || !rows || !cols || !nnz) return DE_ERR_INVALID;
  *rows = c->rows;
  *cols = c->cols;
  *nnz = c->nnz;
  return DE_OK;
}

int de_csr_copy(const de_csr *c, int64_t *rowptr, int64_t *col) {
  if (!c || !rowptr || (!col && c->nnz > 0)) return DE_ERR_INVALID;
  if (c->nnz == 0) {
    std::memset(rowptr, 0, size_t(c->rows + 1) * sizeof(int64_t));
    return DE_OK;
  }
  int before = 0;
  if (cudaGetDevice(&before) != cudaSuccess || cudaSetDevice(c->device) != cudaSuccess)
    return de::csr_fail(DE_ERR_CUDA, "CSR copy: no device");
  de::touch_pages(col, size_t(c->nnz) * sizeof(int64_t));
  de::touch_pages(rowptr, size_t(c->rows + 1) * sizeof(int64_t));
  cudaError_t e = cudaMemcpyAsync(col, c->d_col, size_t(c->nnz) * sizeof(int64_t), cudaMemcpyDeviceToHost, c->st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(rowptr, c->d_rowptr, size_t(c->rows + 1) * sizeof(int64_t), cudaMemcpyDeviceToHost, c->st);
  const cudaError_t e2 = cudaStreamSynchronize(c->st);
  if (e == cudaSuccess) e = e2;
  cudaSetDevice(before);
  if (e != cudaSuccess) return de::csr_fail(DE_ERR_CUDA, std::string("CSR copy: ") + cudaGetErrorString(e));
  return DE_OK;
}

void de_csr_free(de_csr *c) {
  if (!c) return;
  if (c->d_rowptr) {
    int before = 0;
    const bool known = cudaGetDevice(&before) == cudaSuccess;
    cudaSetDevice(c->device);
    cudaFree(c->d_rowptr);
    cudaStreamDestroy(c->st);
    if (known) cudaSetDevice(before);
  }
  delete c;
}

}  // extern "C"
