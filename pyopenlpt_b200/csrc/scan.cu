// Device-wide exclusive scan (tile sums, then every tile scanned from its predecessors' sums) and
// the CSR builder declared in olpt_scan.cuh.
#include "olpt_scan.cuh"

namespace olpt {
namespace {


constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;  // per thread per block tile
constexpr int kScanTile = kScanThreads * kScanItems;

// Sum over the block's threads, in every thread.
__device__ __forceinline__ int block_sum(int x, int* warp_tot) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  x = __reduce_add_sync(0xffffffffu, x);
  if (lane == 0) warp_tot[wid] = x;
  __syncthreads();
  x = __reduce_add_sync(0xffffffffu, warp_tot[lane]);
  __syncthreads();
  return x;
}

// Phase 1: tile totals.
__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(const int* in, int n, int* sums) {
  __shared__ int warp_tot[32];
  const int base = blockIdx.x * kScanTile + threadIdx.x;
  int t = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j)
    if (base + j * kScanThreads < n) t += in[base + j * kScanThreads];
  t = block_sum(t, warp_tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = t;
}

// Phase 2: every block adds up the totals of the tiles before its own (a few loads a thread
// up to millions of entries) and scans its tile; the last one writes out[n] = total.  Two
// launches, no block waits for another.
__global__ void __launch_bounds__(kScanThreads) scan_tiles_kernel(const int* in, int n, int* out,
                                                                  const int* sums) {
  __shared__ int warp_tot[32];
  int before = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += kScanThreads) before += sums[b];
  before = block_sum(before, warp_tot);
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int v[kScanItems];
  int t = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    v[j] = (base + j < n) ? in[base + j] : 0;
    t += v[j];
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int incl = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int w = warp_tot[lane];
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += y;
    }
    warp_tot[lane] = wi - w;
  }
  __syncthreads();
  int run = before + warp_tot[wid] + incl - t;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    if (base + j < n) out[base + j] = run;
    run += v[j];
    if (base + j == n - 1) out[n] = run;
  }
}

}  // namespace

void exclusive_scan(const int* in, int n, int* out, DevBuf& tmp, cudaStream_t s, int most) {
  if (n > most) require_scan(n);
  if (n <= 0) {
    OLPT_CUDA(cudaMemsetAsync(out, 0, sizeof(int), s));
    return;
  }
  const int n_tiles = (n + kScanTile - 1) / kScanTile;
  tmp.ensure((size_t)(n_tiles + 1) * sizeof(int), s);
  if (n_tiles > 1) scan_sums_kernel<<<OLPT_G(n_tiles), kScanThreads, 0, s>>>(in, n, tmp.as<int>());
  scan_tiles_kernel<<<OLPT_G(n_tiles), kScanThreads, 0, s>>>(in, n, out, tmp.as<int>());
  OLPT_CUDA(cudaGetLastError());
}

namespace {

// CSR scatter: items with key >= 0 go to bucket `key`; `counts` (the buckets' sizes) end at 0.
__global__ void csr_scatter_kernel(const int* key, int n, const int* start, int* counts,
                                   int* items) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = key[i];
  if (k < 0) return;
  items[start[k] + atomicSub(&counts[k], 1) - 1] = i;
}

__global__ void csr_count_kernel(const int* key, int n, int* counts) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = key[i];
  if (k >= 0) atomicAdd(&counts[k], 1);
}

}  // namespace

void Csr::build(const int* key, int n, int n_buckets, cudaStream_t s) {
  start.ensure((n_buckets + 1) * sizeof(int), s);
  cursor.ensure((n_buckets + 1) * sizeof(int), s);
  items.ensure((n + 1) * sizeof(int), s);
  OLPT_CUDA(cudaMemsetAsync(cursor.p, 0, n_buckets * sizeof(int), s));
  if (n > 0) csr_count_kernel<<<OLPT_G((n + 255) / 256), 256, 0, s>>>(key, n, cursor.as<int>());
  exclusive_scan(cursor.as<int>(), n_buckets, start.as<int>(), tmp, s);
  if (n > 0)
    csr_scatter_kernel<<<OLPT_G((n + 255) / 256), 256, 0, s>>>(key, n, start.as<int>(),
                                                               cursor.as<int>(), items.as<int>());
  OLPT_CUDA(cudaGetLastError());
}

}  // namespace olpt
