// Device half of the candidate ordering and of StereoMatch::pruneMatch
// (src/srcSTB/StereoMatch.cpp:153-156, 631-980).
//
// The candidates of checkMatch stay on the device:
//  1. sort by ids (lexicographic, camera 0 first; -1 < any id) with a stable LSD
//     radix sort of packed 64-bit keys;
//  2. every candidate's 2D points (global point index per active camera, camera
//     order) and the point -> candidate lists (CSR, in any order);
//  3. per 2D point (one warp): the percentile of every candidate in the point's pool.
//     The reference stable-sorts the pool with a tolerance comparator (rtol 1e-9,
//     atol 1e-12) and averages ranks over runs of tolerance-equal e_check.  When the
//     runs are tolerance-equal end to end (checked here), the comparator is a strict
//     weak ordering on the pool, the runs are the tolerance classes, and every rank
//     follows from the class boundaries of the exactly sorted pool;
//  4. per candidate: the mean percentile over its points, summed in point order;
//  5. the greedy order by (percentile, e_check, index) of the candidates the greedy
//     can take: tolerance classes of the percentiles, then of e_check inside every
//     percentile class (computed and checked the same way over the sorted values),
//     and a radix sort by class;
//  6. the greedy: parallel rounds of the in-order greedy independent set, checked
//     against the replacement rule; the sequential loop on the host when a
//     replacement would fire.
// Everything is enqueued without a look at a count: candidates that drop out of a list
// sort to its end under the largest key, and the kernels read the counts on the device.
// Whenever a check fails (a tolerance class wider than the tolerance) the caller falls
// back to the host implementation, which keeps the reference's std::stable_sort.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "olpt_ctx.cuh"
#include "olpt_prune.h"
#include "olpt_scan.cuh"

namespace olpt {
namespace {

inline int nblk(int64_t n, int t = 256) { return (int)((n + t - 1) / t); }

// ---------------------------------------------------------------- radix sort
// Stable LSD sort by 8-bit digits, two launches a digit: the tiles' digit counts, and the
// scatter, whose blocks add up the counts of the tiles before theirs themselves (5 launches
// with a device-wide scan of the counts in between; 30,000 keys of 64 bits: 72 us instead of
// 200).  Those sums grow with the square of the tiles, so above kRsSumTiles the counts lie by
// digit and are scanned.  Counts, scan and scatter of a digit at 2, 8 and 16 million keys: 61,
// 403 and 1,293 us with sums in every block, 40, 118 and 221 us with the scan.  A warp owns
// 256 consecutive items of the tile and ranks them without block barriers.
constexpr int kRsThreads = 512;
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRsItems = 8;
constexpr int kRsTile = kRsThreads * kRsItems;
// 0.5 and 1 million keys, a digit: 23 and 30 us with the sums, 25 and 29 us with the scan
constexpr int kRsSumTiles = 256;

// counts by tile, or (SCANNED) by digit
template <bool SCANNED>
__global__ void __launch_bounds__(kRsThreads) rs_hist_kernel(const uint64_t* key, int n, int shift,
                                                             int* hist) {
  __shared__ int h[256];
  if (threadIdx.x < 256) h[threadIdx.x] = 0;
  __syncthreads();
  const int tile = blockIdx.x * kRsTile + threadIdx.x;
#pragma unroll
  for (int k = 0; k < kRsItems; ++k) {
    const int i = tile + k * kRsThreads;
    if (i < n) atomicAdd(&h[(int)((key[i] >> shift) & 255u)], 1);
  }
  __syncthreads();
  if (threadIdx.x < 256)
    hist[SCANNED ? threadIdx.x * gridDim.x + blockIdx.x : blockIdx.x * 256 + threadIdx.x] =
        h[threadIdx.x];
}

// Exclusive prefix sums of the first 256 threads' values.
__device__ __forceinline__ int scan256(int x, int* wsum) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (w < 8 && lane == 31) wsum[w] = incl;
  __syncthreads();
  int before = 0;
  for (int k = 0; k < 8; ++k) before += k < w ? wsum[k] : 0;
  return before + incl - x;
}

// hist: the tiles' counts, or (SCANNED) the first position of every digit and tile
template <bool SCANNED>
__global__ void __launch_bounds__(kRsThreads) rs_scatter_kernel(const uint64_t* key, const int* val,
                                                                int n, int shift, const int* hist,
                                                                int n_blocks, uint64_t* key_out,
                                                                int* val_out) {
  __shared__ int cnt[kRsWarps][256];
  __shared__ int half_all[256], half_before[256], wsum[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int d = threadIdx.x & 255, half = threadIdx.x >> 8;
  for (int q = threadIdx.x; q < kRsWarps * 256; q += kRsThreads) (&cnt[0][0])[q] = 0;
  int base = 0;
  if constexpr (SCANNED) {
    if (!half) base = hist[d * n_blocks + blockIdx.x];
    __syncthreads();
  } else {
    // this digit's count in all tiles and in the tiles before, over every second tile
    int all = 0, before = 0;
#pragma unroll 8
    for (int b = half; b < n_blocks; b += 2) {
      const int x = hist[b * 256 + d];
      all += x;
      before += b < (int)blockIdx.x ? x : 0;
    }
    if (half) {
      half_all[d] = all;
      half_before[d] = before;
    }
    __syncthreads();
    if (!half) {
      all += half_all[d];
      before += half_before[d];
    }
    base = scan256(half ? 0 : all, wsum) + before;
  }
  const int i0 = blockIdx.x * kRsTile + w * (32 * kRsItems) + lane;
  uint64_t kk[kRsItems];
  int vv[kRsItems];
#pragma unroll
  for (int k = 0; k < kRsItems; ++k) {
    const int i = i0 + 32 * k;
    kk[k] = i < n ? key[i] : 0ull;
    vv[k] = i < n ? val[i] : 0;
    if (i < n) atomicAdd(&cnt[w][(int)((kk[k] >> shift) & 255u)], 1);
  }
  __syncthreads();
  if (!half)
    for (int q = 0; q < kRsWarps; ++q) {
      const int t = cnt[q][d];
      cnt[q][d] = base;
      base += t;
    }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kRsItems; ++k) {
    const bool ok = i0 + 32 * k < n;
    const int dig = ok ? (int)((kk[k] >> shift) & 255u) : 256 + lane;  // invalid: unique per lane
    const unsigned peers = __match_any_sync(0xffffffffu, dig);
    int pos = 0;
    if (ok) pos = cnt[w][dig] + __popc(peers & ((1u << lane) - 1u));
    __syncwarp();
    if (ok && lane == __ffs(peers) - 1) cnt[w][dig] += __popc(peers);
    __syncwarp();
    if (ok) {
      key_out[pos] = kk[k];
      val_out[pos] = vv[k];
    }
  }
}

// Short lists: one block runs all digits in shared memory (4,096 keys of 64 bits: 16 us).
constexpr int kSmallSort = 4096;
constexpr int kSmallThreads = 1024, kSmallWarps = kSmallThreads / 32;
constexpr size_t kSmallSmem =
    2 * kSmallSort * (sizeof(uint64_t) + sizeof(int)) + kSmallWarps * 256 * sizeof(int);

__global__ void __launch_bounds__(kSmallThreads) small_sort_kernel(const uint64_t* key,
                                                                   const int* val, int n, int bits,
                                                                   uint64_t* key_out,
                                                                   int* val_out) {
  extern __shared__ __align__(16) unsigned char sort_smem[];
  __shared__ int wsum[8];
  uint64_t* ka = reinterpret_cast<uint64_t*>(sort_smem);
  uint64_t* kb = ka + kSmallSort;
  int* va = reinterpret_cast<int*>(kb + kSmallSort);
  int* vb = va + kSmallSort;
  int* cnt = vb + kSmallSort;  // [warp][256]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < n; i += kSmallThreads) {
    ka[i] = key[i];
    va[i] = val[i];
  }
  const int per = (n + kSmallThreads - 1) / kSmallThreads * 32;  // consecutive items a warp
  for (int shift = 0; shift < bits; shift += 8) {
    for (int q = threadIdx.x; q < kSmallWarps * 256; q += kSmallThreads) cnt[q] = 0;
    __syncthreads();
    for (int k = lane; k < per; k += 32) {
      const int i = w * per + k;
      if (i < n) atomicAdd(&cnt[w * 256 + (int)((ka[i] >> shift) & 255u)], 1);
    }
    __syncthreads();
    int all = 0;
    if (threadIdx.x < 256)
      for (int q = 0; q < kSmallWarps; ++q) all += cnt[q * 256 + threadIdx.x];
    int base = scan256(all, wsum);
    if (threadIdx.x < 256)
      for (int q = 0; q < kSmallWarps; ++q) {
        const int t = cnt[q * 256 + threadIdx.x];
        cnt[q * 256 + threadIdx.x] = base;
        base += t;
      }
    __syncthreads();
    for (int k = lane; k < per; k += 32) {
      const int i = w * per + k;
      const bool ok = i < n;
      const uint64_t kk = ok ? ka[i] : 0ull;
      const int dig = ok ? (int)((kk >> shift) & 255u) : 256 + lane;
      const unsigned peers = __match_any_sync(0xffffffffu, dig);
      int pos = 0;
      if (ok) pos = cnt[w * 256 + dig] + __popc(peers & ((1u << lane) - 1u));
      __syncwarp();
      if (ok && lane == __ffs(peers) - 1) cnt[w * 256 + dig] += __popc(peers);
      __syncwarp();
      if (ok) {
        kb[pos] = kk;
        vb[pos] = va[i];
      }
    }
    __syncthreads();
    uint64_t* tk = ka;
    ka = kb;
    kb = tk;
    int* tv = va;
    va = vb;
    vb = tv;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kSmallThreads) {
    key_out[i] = ka[i];
    val_out[i] = va[i];
  }
}

// Lists of a middle length: a cluster of 16 blocks runs all digits with the items in its
// shared memories, position p at block p / per.  A block counts its items' digits by warp,
// adds up the other blocks' totals and scatters through distributed shared memory: two cluster
// barriers a digit instead of two launches whose few tiles of 4,096 leave the chip idle: the
// four sorts of 60,000 candidates took 50 launches and 420 us and take 4 and 170 us.  Bound
// by the ranking's chain through the warps' counters (items ordered by digit in the block
// first, for neighbouring remote stores: 229 us); the limit is what 16 blocks' shared memories
// hold.
constexpr int kClBlocks = 16;
constexpr int kClCap = 7168;  // items a block
constexpr int kClSort = kClBlocks * kClCap;
constexpr size_t kClSmem =
    2 * kClCap * (sizeof(uint64_t) + sizeof(int)) + kSmallWarps * 256 * sizeof(int);

__global__ void __launch_bounds__(kSmallThreads) cluster_sort_kernel(const uint64_t* key,
                                                                     const int* val, int n,
                                                                     int bits, int per,
                                                                     uint64_t* key_out,
                                                                     int* val_out) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char sort_smem[];
  __shared__ int wsum[8], tot[256], start[256], quarter[4][256], quarter_before[4][256];
  cg::cluster_group cluster = cg::this_cluster();
  uint64_t* ka = reinterpret_cast<uint64_t*>(sort_smem);
  uint64_t* kb = ka + kClCap;
  int* va = reinterpret_cast<int*>(kb + kClCap);
  int* vb = va + kClCap;
  int* cnt = vb + kClCap;  // [warp][256]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int me = (int)cluster.block_rank();
  const int m = max(0, min(per, n - me * per));  // items here
  for (int i = threadIdx.x; i < m; i += kSmallThreads) {
    ka[i] = key[me * per + i];
    va[i] = val[me * per + i];
  }
  const int chunk = (m + kSmallThreads - 1) / kSmallThreads * 32;  // consecutive items a warp
  const int d = threadIdx.x & 255, part = threadIdx.x >> 8;
  for (int shift = 0; shift < bits; shift += 8) {
    for (int q = threadIdx.x; q < kSmallWarps * 256; q += kSmallThreads) cnt[q] = 0;
    __syncthreads();
    for (int k = lane; k < chunk; k += 32) {
      const int i = w * chunk + k;
      if (i < m) atomicAdd(&cnt[w * 256 + (int)((ka[i] >> shift) & 255u)], 1);
    }
    __syncthreads();
    if (part == 0) {
      int t = 0;
#pragma unroll 8
      for (int q = 0; q < kSmallWarps; ++q) {
        const int x = cnt[q * 256 + d];
        cnt[q * 256 + d] = t;  // of the warps before
        t += x;
      }
      tot[d] = t;
    }
    cluster.sync();
    int all = 0, before = 0;
#pragma unroll
    for (int b = 4 * part; b < 4 * part + 4; ++b) {
      const int x = *cluster.map_shared_rank(&tot[d], b);
      all += x;
      before += b < me ? x : 0;
    }
    quarter[part][d] = all;
    quarter_before[part][d] = before;
    __syncthreads();
    if (part == 0)
      for (int q = 1; q < 4; ++q) {
        all += quarter[q][d];
        before += quarter_before[q][d];
      }
    const int first = scan256(part == 0 ? all : 0, wsum) + before;
    if (part == 0) start[d] = first;
    __syncthreads();
    for (int k = lane; k < chunk; k += 32) {
      const int i = w * chunk + k;
      const bool ok = i < m;
      const uint64_t kk = ok ? ka[i] : 0ull;
      const int dig = ok ? (int)((kk >> shift) & 255u) : 256 + lane;
      const unsigned peers = __match_any_sync(0xffffffffu, dig);
      int pos = 0;
      if (ok) pos = start[dig] + cnt[w * 256 + dig] + __popc(peers & ((1u << lane) - 1u));
      __syncwarp();
      if (ok && lane == __ffs(peers) - 1) cnt[w * 256 + dig] += __popc(peers);
      __syncwarp();
      if (ok) {
        const int b = pos / per, at = pos - b * per;
        *cluster.map_shared_rank(kb + at, b) = kk;
        *cluster.map_shared_rank(vb + at, b) = va[i];
      }
    }
    cluster.sync();  // the blocks' items are in place; none reads tot any more
    uint64_t* tk = ka;
    ka = kb;
    kb = tk;
    int* tv = va;
    va = vb;
    vb = tv;
  }
  for (int i = threadIdx.x; i < m; i += kSmallThreads) {
    key_out[me * per + i] = ka[i];
    val_out[me * per + i] = va[i];
  }
}

// ---------------------------------------------------------------- candidates
__device__ __forceinline__ bool eq_eps(double a, double b) {
  const double s = fmax(fabs(a), fabs(b));
  return fabs(a - b) <= (s * 1e-9 + 1e-12);
}

__global__ void id_keys_kernel(const int* ids, int M, int n, int bits, uint64_t* key, int* val) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= M) return;
  uint64_t k = 0;
  for (int c = 0; c < n; ++c) k = (k << bits) | (uint64_t)(uint32_t)(ids[(int64_t)j * n + c] + 1);
  key[j] = k;
  val[j] = j;
}

// Word w of the candidates' id keys, for a lexicographic sort in several 64-bit
// passes: the ids of cameras [w * per, (w + 1) * per) of candidate perm[i] (i when perm
// is null), packed most significant first; val[i] = the candidate.
__global__ void word_keys_kernel(const int* ids, int M, int n, int bits, int per, int w,
                                 const int* perm, uint64_t* key, int* val) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= M) return;
  const int j = perm ? perm[i] : i;
  const int c1 = min(n, (w + 1) * per);
  uint64_t k = 0;
  for (int c = w * per; c < c1; ++c)
    k = (k << bits) | (uint64_t)(uint32_t)(ids[(int64_t)j * n + c] + 1);
  key[i] = k;
  val[i] = j;
}

__global__ void gather_cand_kernel(const int* perm, int M, int n, const int* ids, const double* e,
                                   const double* X, int* ids_s, double* e_s, double* X_s) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= M) return;
  const int j = perm[i];
  for (int c = 0; c < n; ++c) ids_s[(int64_t)i * n + c] = ids[(int64_t)j * n + c];
  e_s[i] = e[j];
  for (int d = 0; d < 3; ++d) X_s[3 * (int64_t)i + d] = X[3 * (int64_t)j + d];
}

// The candidate's 2D points (global index, camera order) in slots j*n .. j*n+n-1.
__global__ void flat_kernel(const int* ids, int M, int n, PruneView pv, int* fl, int* key,
                            uint8_t* fcnt) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= M) return;
  int k = 0;
  for (int c = 0; c < n; ++c) {
    const int pid = ids[(int64_t)j * n + c];
    if (!pv.active[c] || pid < 0 || pid >= pv.count[c]) continue;
    const int f = pv.offset[c] + pid;
    fl[(int64_t)j * n + k] = f;
    key[(int64_t)j * n + k] = f;
    ++k;
  }
  for (int q = k; q < n; ++q) {
    fl[(int64_t)j * n + q] = -1;
    key[(int64_t)j * n + q] = -1;
  }
  fcnt[j] = (uint8_t)k;
}

// Per 2D point, one warp: percentile of each candidate of the point's pool.  Pools of up to 32
// candidates stay in registers, larger ones of up to kPoolMax in shared memory, the rest in
// the global scratch (indexed by their position in the point -> candidate list).  Bound by the
// latency of the gathers, so by the warps in flight: shared memory for pools of 512 in every
// warp left room for 16 of them an SM (2.5 million points, 850 -> 420 us; 200,000 points with
// pools of dozens, 175 -> 110 us).
constexpr int kPctWarps = 4;
constexpr int kPoolMax = 128;
struct PoolSmem {
  double e[kPoolMax];
  int j[kPoolMax];
  int slot[kPoolMax];
  int ord[kPoolMax];
  int cls[kPoolMax];
  int start[kPoolMax];
};
struct PoolScratch {  // global, one entry per (point, candidate) pair
  double* e;
  int *j, *slot, *ord, *cls, *start;
};

__global__ void __launch_bounds__(kPctWarps * 32) pct_kernel(const int* pstart, const int* items,
                                                             int n_points, int n, const double* e,
                                                             PoolScratch gs, double* slot_pct,
                                                             uint8_t* slot_used, int* flag) {
  extern __shared__ __align__(16) unsigned char pool_raw[];
  PoolSmem& S = reinterpret_cast<PoolSmem*>(pool_raw)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int f = blockIdx.x * kPctWarps + (threadIdx.x >> 5);
  if (f >= n_points) return;
  const int b = pstart[f], end = pstart[f + 1];
  const unsigned lt = (1u << lane) - 1u;
  if (end - b <= 32) {
    if (end == b) return;
    const int slot = items[min(b + lane, end - 1)];
    const int j = slot / n;
    const double ev = e[j];
    const bool fin = b + lane < end && isfinite(ev);
    const unsigned m = __ballot_sync(0xffffffffu, fin);
    const int np = __popc(m);
    if (np <= 1) {
      if (fin) {
        slot_pct[slot] = 0.0;
        slot_used[slot] = 1;
      }
      return;
    }
    // exact order by (e, j)
    int r = 0;
    for (unsigned k = m; k; k &= k - 1) {
      const double ek = __shfl_sync(0xffffffffu, ev, __ffs(k) - 1);
      const int jk = __shfl_sync(0xffffffffu, j, __ffs(k) - 1);
      r += ek < ev || (ek == ev && jk < j) ? 1 : 0;
    }
    if (fin) {
      S.e[r] = ev;
      S.slot[r] = slot;
    }
    __syncwarp();
    // tolerance classes over the sorted values: lane p is the p-th
    const bool valid = lane < np;
    const double mine = S.e[valid ? lane : 0];
    const unsigned starts = __ballot_sync(
        0xffffffffu, valid && (lane == 0 || !eq_eps(S.e[valid && lane ? lane - 1 : 0], mine)));
    const int s0 = 31 - __clz(starts & (lt | (1u << lane)));
    const unsigned above = starts & ~(lt | (1u << lane));
    const int s1 = above ? __ffs(above) - 2 : np - 1;
    bool bad = false;
    if (valid) {
      bad = !eq_eps(S.e[s0], mine);
      const double avg_rank = 0.5 * (double)(s0 + s1);
      slot_pct[S.slot[lane]] = avg_rank / (double)(np - 1);
      slot_used[S.slot[lane]] = 1;
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(flag, 2);
    return;
  }
  int np = 0;
  for (int base = b; base < end; base += 32) {
    const int q = base + lane;
    const bool fin = q < end && isfinite(e[items[q] / n]);
    np += __popc(__ballot_sync(0xffffffffu, fin));
  }
  if (np == 0) return;
  const bool big = np > kPoolMax;
  double* pe = big ? gs.e + b : S.e;
  int* pj = big ? gs.j + b : S.j;
  int* pslot = big ? gs.slot + b : S.slot;
  int* pord = big ? gs.ord + b : S.ord;
  int* pcls = big ? gs.cls + b : S.cls;
  int* pstart2 = big ? gs.start + b : S.start;
  int cnt = 0;
  for (int base = b; base < end; base += 32) {
    const int q = base + lane;
    const bool valid = q < end;
    const int slot = valid ? items[q] : 0;
    const int j = slot / n;
    const double ev = valid ? e[j] : 0.0;
    const bool fin = valid && isfinite(ev);
    const unsigned m = __ballot_sync(0xffffffffu, fin);
    const int pos = cnt + __popc(m & lt);
    if (fin) {
      pe[pos] = ev;
      pj[pos] = j;
      pslot[pos] = slot;
    }
    cnt += __popc(m);
  }
  __syncwarp();
  if (np == 1) {
    if (lane == 0) {
      slot_pct[pslot[0]] = 0.0;
      slot_used[pslot[0]] = 1;
    }
    return;
  }
  // exact order by (e, j)
  for (int i = lane; i < np; i += 32) {
    const double ei = pe[i];
    const int ji = pj[i];
    int r = 0;
    for (int k = 0; k < np; ++k) r += (pe[k] < ei || (pe[k] == ei && pj[k] < ji)) ? 1 : 0;
    pord[r] = i;
  }
  __syncwarp();
  // tolerance classes over the sorted values
  int run = -1;
  for (int p0 = 0; p0 < np; p0 += 32) {
    const int p = p0 + lane;
    const bool valid = p < np;
    const bool newc = valid && (p == 0 || !eq_eps(pe[pord[p - 1]], pe[pord[p]]));
    const unsigned m = __ballot_sync(0xffffffffu, newc);
    const int cid = run + __popc(m & (lt | (1u << lane)));
    if (valid) pcls[p] = cid;
    if (newc) pstart2[cid] = p;
    run += __popc(m);
  }
  __syncwarp();
  const int n_cls = run + 1;
  bool bad = false;
  for (int p = lane; p < np; p += 32) {
    const int c = pcls[p];
    const int s0 = pstart2[c];
    const int s1 = (c + 1 < n_cls) ? pstart2[c + 1] - 1 : np - 1;
    if (!eq_eps(pe[pord[s0]], pe[pord[p]])) bad = true;
    const double avg_rank = 0.5 * (double)(s0 + s1);
    const double pct = avg_rank / (double)(np - 1);
    const int slot = pslot[pord[p]];
    slot_pct[slot] = pct;
    slot_used[slot] = 1;
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(flag, 2);
}

__device__ __forceinline__ uint64_t ordered_bits(double v) {
  if (v == 0.0) v = 0.0;
  const uint64_t b = (uint64_t)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | (1ull << 63));
}

// Mean percentile of every candidate, summed in point order; the key of the percentile sort
// (a candidate without one goes last) and the counts of both candidate sets.
__global__ void pct_score_kernel(const uint8_t* fcnt, int M, int n, const double* slot_pct,
                                 const uint8_t* slot_used, const double* e, double* pct_score,
                                 uint64_t* key, int* val, int* counts) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  bool a = false, b = false;
  if (j < M) {
    double sum = 0.0;
    int cnt = 0;
    for (int k = 0; k < fcnt[j]; ++k) {
      const int64_t s = (int64_t)j * n + k;
      if (slot_used[s]) {
        sum += slot_pct[s];
        ++cnt;
      }
    }
    const double p = cnt > 0 ? sum / (double)cnt : __longlong_as_double(0x7ff0000000000000LL);
    pct_score[j] = p;
    a = isfinite(p);
    b = a && isfinite(e[j]);
    key[j] = a ? ordered_bits(p) : ~0ull;
    val[j] = j;
  }
  const unsigned ma = __ballot_sync(0xffffffffu, a), mb = __ballot_sync(0xffffffffu, b);
  if ((threadIdx.x & 31) == 0) {
    if (ma) atomicAdd(&counts[PC_PCT], __popc(ma));
    if (mb) atomicAdd(&counts[PC_BOTH], __popc(mb));
  }
}

// keys of the e_check sort over the candidates the greedy can take (the others go last)
__global__ void e_keys_kernel(const double* pct, const double* e, int M, uint64_t* key, int* val) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= M) return;
  key[j] = isfinite(pct[j]) && isfinite(e[j]) ? ordered_bits(e[j]) : ~0ull;
  val[j] = j;
}

// keys of the sort by percentile class; positions past the count keep the end
__global__ void group_keys_kernel(const int* idx, int M, const int* counts, const int* grp,
                                  uint64_t last, uint64_t* key) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= M) return;
  key[p] = p < counts[PC_BOTH] ? (uint64_t)grp[idx[p]] : last;
}

// Tolerance classes over sorted values: a class starts where the value leaves the tolerance
// of its predecessor, or where the group (the percentile class, when given) changes.  First
// launch: class starts per tile and the tile's last one; second: every block adds up the tiles
// before its own, numbers the classes, and checks every member against its class's start.
constexpr int kClsTile = 1024;

__device__ __forceinline__ bool class_starts(const int* idx, int p, const double* val,
                                             const int* grp) {
  return p == 0 || (grp && grp[idx[p - 1]] != grp[idx[p]]) || !eq_eps(val[idx[p - 1]], val[idx[p]]);
}

__global__ void __launch_bounds__(kClsTile) class_count_kernel(const int* idx, const int* m_ptr,
                                                               const double* val, const int* grp,
                                                               int2* tiles) {
  __shared__ int s_n[32], s_l[32];
  const int p = blockIdx.x * kClsTile + threadIdx.x, m = *m_ptr;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned b = __ballot_sync(0xffffffffu, p < m && class_starts(idx, p, val, grp));
  if (lane == 0) {
    s_n[w] = __popc(b);
    s_l[w] = b ? p + 31 - __clz(b) : -1;
  }
  __syncthreads();
  if (w == 0) {
    const int n = __reduce_add_sync(0xffffffffu, s_n[lane]);
    const int l = __reduce_max_sync(0xffffffffu, s_l[lane]);
    if (lane == 0) tiles[blockIdx.x] = make_int2(n, l);
  }
}

__global__ void __launch_bounds__(kClsTile) class_assign_kernel(const int* idx, const int* m_ptr,
                                                                const double* val, const int* grp,
                                                                const int2* tiles, int* cls,
                                                                int* start, int* mixed,
                                                                int* counts, int n_word, int bad) {
  __shared__ int s_n[32], s_l[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int m = *m_ptr;
  if ((int)blockIdx.x * kClsTile >= m && blockIdx.x > 0) return;
  // classes before the tile and the last start before it
  int nb = 0, lb = -1;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += kClsTile) {
    const int2 t = tiles[b];
    nb += t.x;
    lb = max(lb, t.y);
  }
  nb = __reduce_add_sync(0xffffffffu, nb);
  lb = __reduce_max_sync(0xffffffffu, lb);
  if (lane == 0) {
    s_n[w] = nb;
    s_l[w] = lb;
  }
  __syncthreads();
  nb = __reduce_add_sync(0xffffffffu, s_n[lane]);
  lb = __reduce_max_sync(0xffffffffu, s_l[lane]);
  __syncthreads();
  const int p = blockIdx.x * kClsTile + threadIdx.x;
  const bool first = p < m && class_starts(idx, p, val, grp);
  const unsigned b = __ballot_sync(0xffffffffu, first);
  if (lane == 0) {
    s_n[w] = __popc(b);
    s_l[w] = b ? p + 31 - __clz(b) : -1;
  }
  __syncthreads();
  for (int k = 0; k < w; ++k) {
    nb += s_n[k];
    lb = max(lb, s_l[k]);
  }
  const unsigned le = b & (0xffffffffu >> (31 - lane));
  const int c = nb + __popc(le) - 1;
  const int sp = le ? p - lane + 31 - __clz(le) : lb;
  if (p < m) {
    if (!eq_eps(val[idx[sp]], val[idx[p]])) atomicOr(&counts[PC_FLAG], bad);
    cls[idx[p]] = c;
    if (first) start[c] = p;
    // members that differ in value: the class needs its members re-sorted by index
    if (mixed && !first && val[idx[p - 1]] != val[idx[p]]) {
      mixed[c] = 1;
      counts[PC_MIXED] = 1;
    }
    if (p == m - 1) counts[n_word] = c + 1;
  }
}

// The (percentile class, e_check) order has the members of an e_check class sorted by
// e_check value, then index; the greedy wants them by index.  Only classes whose members
// differ in value need it.
__global__ void class_index_sort_kernel(int* idx, const int* start, const int* counts,
                                        const int* mixed) {
  if (!counts[PC_MIXED]) return;
  const int c = blockIdx.x * blockDim.x + threadIdx.x, n_cls = counts[PC_ECLS];
  if (c >= n_cls || !mixed[c]) return;
  const int b = start[c], e = c + 1 < n_cls ? start[c + 1] : counts[PC_BOTH];
  for (int i = b + 1; i < e; ++i) {
    const int v = idx[i];
    int j = i - 1;
    while (j >= b && idx[j] > v) {
      idx[j + 1] = idx[j];
      --j;
    }
    idx[j + 1] = v;
  }
}

__global__ void gather_greedy_kernel(const int* order, const int* counts, int n, const int* fl,
                                     const uint8_t* fcnt, const double* pct, const double* e,
                                     int* g_pts, uint8_t* g_cnt, double* g_pct, double* g_e) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= counts[PC_BOTH]) return;
  const int j = order[i];
  for (int k = 0; k < n; ++k) g_pts[(int64_t)i * n + k] = fl[(int64_t)j * n + k];
  g_cnt[i] = fcnt[j];
  g_pct[i] = pct[j];
  g_e[i] = e[j];
}

// ---------------------------------------------------------------- greedy
// The greedy of pruneMatch over candidates in greedy order.  Without replacements it
// is the in-order greedy independent set (a candidate is taken iff no earlier taken
// candidate shares one of its points), which these rounds compute in parallel: a
// candidate is rejected once a taken one shares a point (it came earlier: while it was
// undecided it was the first on that point), and taken once it is the earliest undecided
// candidate on every one of its points.  Then every rejected candidate evaluates the
// replacement rule against its owners (the taken candidates before it on its points)
// exactly as the sequential loop would; if any would replace, the caller runs the
// sequential loop instead.  One cooperative launch with one grid barrier a round: a thread
// decides its candidates from the round's minima over their points, and enters those that stay
// undecided into the next round's at once.  The rounds' minima alternate between two arrays,
// and hold the round's complement above the candidate, so that a later round's replace an
// earlier one's without clearing.  (A candidate whose owner was taken in the same round enters
// the next one's minima; it would also with a barrier in between.)  Bound by the barriers and
// the rounds' dependent reads: 240 -> 195 us at 200,000 points with two barriers -> one.
constexpr uint8_t kUndecided = 0, kTaken = 1, kRejected = 2, kSkipped = 3;
constexpr int kGreedyThreads = 512;

// StereoMatch::pruneMatch replacement rule (StereoMatch.cpp:930-975) for a rejected
// candidate against the owners of its points, averaged in point order.
__device__ bool replaces(const int* g_pts, int cnt, int i, int n, const int* owner,
                         const double* g_pct, const double* g_e) {
  int S[OLPT_MAX_CAM];
  int ns = 0;
  double avg_pct = 0.0, avg_err = 0.0;
  for (int k = 0; k < cnt; ++k) {
    const int o = owner[g_pts[(int64_t)i * n + k]];
    if (o < 0 || o >= i) continue;
    bool seen = false;
    for (int t = 0; t < ns; ++t) seen |= (S[t] == o);
    if (seen) continue;
    S[ns++] = o;
    avg_pct += g_pct[o];
    avg_err += g_e[o];
  }
  if (ns == 0) return true;  // cannot happen for a rejected candidate
  avg_pct /= (double)ns;
  avg_err /= (double)ns;
  const double pj = g_pct[i], ej = g_e[i];
  const bool better_pct = (!eq_eps(pj, avg_pct)) && ((pj + 1e-12) < avg_pct);
  const bool tie_better = eq_eps(pj, avg_pct) && (!eq_eps(ej, avg_err)) && ((ej + 1e-12) < avg_err);
  return better_pct || tie_better;
}

__global__ void __launch_bounds__(kGreedyThreads) greedy_kernel(
    int* counts, const int* g_pts, const uint8_t* g_cnt, int n, uint8_t* state,
    unsigned long long* first, int n_points, int* owner, const int* order, const double* g_pct,
    const double* g_e, uint8_t* sel, int* scnt) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  const int G = counts[PC_BOTH];
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  auto enter = [&](int i, unsigned round) {
    const unsigned long long mark = (unsigned long long)(0xffffffffu - round) << 32 | (unsigned)i;
    unsigned long long* f = first + (round & 1u) * (size_t)n_points;
    for (int k = 0; k < g_cnt[i]; ++k) atomicMin(&f[g_pts[(int64_t)i * n + k]], mark);
  };
  // candidates without a point are passed over by the loop (neither kept nor owners)
  for (int i = t0; i < G; i += step) {
    state[i] = g_cnt[i] == 0 ? kSkipped : kUndecided;
    enter(i, 0);
  }
  grid.sync();
  // every round decides at least the earliest undecided candidate
  for (unsigned round = 0; round <= (unsigned)G; ++round) {
    // three flags: the next round's is cleared while nobody reads or sets it
    int* left = counts + PC_LEFT + round % 3;
    if (t0 == 0) counts[PC_LEFT + (round + 1) % 3] = 0;
    const unsigned long long hi = (unsigned long long)(0xffffffffu - round) << 32;
    const unsigned long long* now = first + (round & 1u) * (size_t)n_points;
    bool und = false;
    for (int i = t0; i < G; i += step) {
      if (state[i] != kUndecided) continue;
      bool all_first = true, blocked = false;
      for (int k = 0; k < g_cnt[i]; ++k) {
        const int f = g_pts[(int64_t)i * n + k];
        blocked = blocked || __ldcg(owner + f) >= 0;
        all_first = all_first && __ldcg(now + f) == (hi | (unsigned)i);
      }
      if (blocked) {
        state[i] = kRejected;
      } else if (all_first) {
        state[i] = kTaken;
        for (int k = 0; k < g_cnt[i]; ++k) __stcg(owner + g_pts[(int64_t)i * n + k], i);
      } else {
        enter(i, round + 1);
        und = true;
      }
    }
    if (__syncthreads_or(und) && threadIdx.x == 0) atomicOr(left, 1);
    grid.sync();
    if (__ldcg(left) == 0) break;
  }
  for (int i = t0; i < G; i += step) {
    const uint8_t st = state[i];
    if (st == kTaken) {
      sel[order[i]] = 1;
      scnt[order[i]] = 1;
    } else if (st == kRejected && replaces(g_pts, g_cnt[i], i, n, owner, g_pct, g_e)) {
      atomicOr(&counts[PC_REPLACE], 1);
    }
  }
}

__global__ void sel_count_kernel(const uint8_t* sel, int M, int* f) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < M) f[i] = sel[i] ? 1 : 0;
}

int bit_width(uint64_t x) {
  int b = 0;
  while (x) {
    ++b;
    x >>= 1;
  }
  return b;
}

}  // namespace

// Stable LSD radix sort of (key, val) pairs on the low `bits` bits, rounded up to whole
// digits; result in (key, val), scratch in (key2, val2).
static void radix_sort_device(PruneWork& W, int n, int bits, cudaStream_t s) {
  if (n <= 1 || bits <= 0) return;
  W.key2.ensure((size_t)(n + 1) * sizeof(uint64_t), s);
  W.val2.ensure((size_t)(n + 1) * sizeof(int), s);
  if (n <= kSmallSort) {
    OLPT_CUDA(cudaFuncSetAttribute(small_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kSmallSmem));
    small_sort_kernel<<<OLPT_G(1), kSmallThreads, kSmallSmem, s>>>(
        W.key.as<uint64_t>(), W.val.as<int>(), n, bits, W.key2.as<uint64_t>(), W.val2.as<int>());
    OLPT_CUDA(cudaGetLastError());
    std::swap(W.key, W.key2);
    std::swap(W.val, W.val2);
    return;
  }
  if (n <= kClSort && W.cluster != 0) {
    OLPT_CUDA(cudaFuncSetAttribute(cluster_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kClSmem));
    OLPT_CUDA(cudaFuncSetAttribute(cluster_sort_kernel,
                                   cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kClBlocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kClBlocks);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = kClSmem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (W.cluster < 0) {  // a partition of the device may have no 16 SMs side by side
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, cluster_sort_kernel, &cfg) != cudaSuccess)
        cudaGetLastError();
      W.cluster = clusters > 0;
    }
    if (W.cluster) {
      const int per = ((n + kClBlocks - 1) / kClBlocks + 31) / 32 * 32;
      cfg.gridDim = dim3(OLPT_G(kClBlocks));
      OLPT_CUDA(cudaLaunchKernelEx(&cfg, cluster_sort_kernel,
                                   (const uint64_t*)W.key.as<uint64_t>(),
                                   (const int*)W.val.as<int>(), n, bits, per,
                                   W.key2.as<uint64_t>(), W.val2.as<int>()));
      std::swap(W.key, W.key2);
      std::swap(W.val, W.val2);
      return;
    }
  }
  const int n_blocks = (n + kRsTile - 1) / kRsTile;
  const bool scanned = n_blocks > kRsSumTiles;
  auto hist = scanned ? rs_hist_kernel<true> : rs_hist_kernel<false>;
  auto scatter = scanned ? rs_scatter_kernel<true> : rs_scatter_kernel<false>;
  W.hist.ensure((size_t)256 * n_blocks * sizeof(int), s);
  if (scanned) W.hist2.ensure(((size_t)256 * n_blocks + 1) * sizeof(int), s);
  for (int shift = 0; shift < bits; shift += 8) {
    hist<<<OLPT_G(n_blocks), kRsThreads, 0, s>>>(W.key.as<uint64_t>(), n, shift, W.hist.as<int>());
    if (scanned)
      exclusive_scan(W.hist.as<int>(), 256 * n_blocks, W.hist2.as<int>(), W.scan_tmp, s);
    scatter<<<OLPT_G(n_blocks), kRsThreads, 0, s>>>(
        W.key.as<uint64_t>(), W.val.as<int>(), n, shift, (scanned ? W.hist2 : W.hist).as<int>(),
        n_blocks, W.key2.as<uint64_t>(), W.val2.as<int>());
    std::swap(W.key, W.key2);
    std::swap(W.val, W.val2);
  }
  OLPT_CUDA(cudaGetLastError());
}

// Sort the device candidates (ids, e, X) by ids into the `_s` buffers.  The ids of all
// cameras form one lexicographic key; when it does not fit in 64 bits it is split into
// words sorted least significant first, each pass stable, so the order is the same.
bool sort_candidates_device(PruneWork& W, const int* ids, const double* e, const double* X, int M,
                            int n, int max_id, cudaStream_t s) {
  const int bits = bit_width((uint64_t)(max_id + 1));
  if (bits > 32) return false;
  W.key.ensure((size_t)(M + 1) * sizeof(uint64_t), s);
  W.val.ensure((size_t)(M + 1) * sizeof(int), s);
  W.key2.ensure((size_t)(M + 1) * sizeof(uint64_t), s);
  W.val2.ensure((size_t)(M + 1) * sizeof(int), s);
  W.ids_s.ensure((size_t)(M + 1) * n * sizeof(int), s);
  W.e_s.ensure((size_t)(M + 1) * sizeof(double), s);
  W.X_s.ensure((size_t)(M + 1) * 3 * sizeof(double), s);
  if (M == 0) return true;
  if (bits * n <= 64) {
    id_keys_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(ids, M, n, bits, W.key.as<uint64_t>(),
                                                  W.val.as<int>());
    radix_sort_device(W, M, bits * n, s);
  } else {
    const int per = 64 / bits;
    const int words = (n + per - 1) / per;
    for (int w = words - 1; w >= 0; --w) {
      const bool first = w == words - 1;
      word_keys_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(
          ids, M, n, bits, per, w, first ? nullptr : W.val.as<int>(), W.key2.as<uint64_t>(),
          W.val2.as<int>());
      std::swap(W.key, W.key2);
      std::swap(W.val, W.val2);
      const int in_word = std::min(n, (w + 1) * per) - w * per;
      radix_sort_device(W, M, bits * in_word, s);
    }
  }
  gather_cand_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(W.val.as<int>(), M, n, ids, e, X,
                                                    W.ids_s.as<int>(), W.e_s.as<double>(),
                                                    W.X_s.as<double>());
  OLPT_CUDA(cudaGetLastError());
  return true;
}

// Steps 2-6 on the sorted candidates (W.ids_s, W.e_s).
void prune_device(PruneWork& W, const PruneView& pv, int M, int n, int64_t total_points,
                  cudaStream_t s) {
  require_scan(M);
  if (M > 0) require_scan(total_points);
  W.counts.ensure(PC_N * sizeof(int), s);
  W.sel.ensure((size_t)M + 16, s);
  W.scnt.ensure((size_t)(M + 1) * sizeof(int), s);
  W.spos.ensure((size_t)(M + 1) * sizeof(int), s);
  OLPT_CUDA(cudaMemsetAsync(W.counts.p, 0, PC_N * sizeof(int), s));
  OLPT_CUDA(cudaMemsetAsync(W.sel.p, 0, (size_t)M + 1, s));
  OLPT_CUDA(cudaMemsetAsync(W.scnt.p, 0, (size_t)(M + 1) * sizeof(int), s));
  if (M > 0) {
    const size_t slots = (size_t)M * n;
    const size_t pts = (size_t)std::max<int64_t>(total_points, 1);
    W.fl.ensure((slots + 1) * sizeof(int), s);
    W.slot_key.ensure((slots + 1) * sizeof(int), s);
    W.fcnt.ensure(M + 16, s);
    W.slot_pct.ensure((slots + 1) * sizeof(double), s);
    W.slot_used.ensure(slots + 16, s);
    for (DevBuf* b : {&W.pct, &W.g_pct, &W.g_e}) b->ensure((size_t)(M + 1) * sizeof(double), s);
    for (DevBuf* b : {&W.key, &W.key2}) b->ensure((size_t)(M + 1) * sizeof(uint64_t), s);
    for (DevBuf* b : {&W.val, &W.val2, &W.pcls, &W.ecls, &W.cstart, &W.mixed})
      b->ensure((size_t)(M + 1) * sizeof(int), s);
    const int n_tile = nblk(M, kClsTile);
    W.tiles.ensure((size_t)n_tile * sizeof(int2), s);
    int* counts = W.counts.as<int>();
    OLPT_CUDA(cudaMemsetAsync(W.slot_used.p, 0, slots, s));
    flat_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(W.ids_s.as<int>(), M, n, pv, W.fl.as<int>(),
                                               W.slot_key.as<int>(), W.fcnt.as<uint8_t>());
    W.points.build(W.slot_key.as<int>(), (int)slots, (int)total_points, s);
    const size_t smem = kPctWarps * sizeof(PoolSmem);
    OLPT_CUDA(cudaFuncSetAttribute(pct_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
    W.pool_e.ensure((slots + 1) * sizeof(double), s);
    W.pool_i.ensure((slots + 1) * 5 * sizeof(int), s);
    PoolScratch gs;
    gs.e = W.pool_e.as<double>();
    gs.j = W.pool_i.as<int>();
    gs.slot = gs.j + slots;
    gs.ord = gs.slot + slots;
    gs.cls = gs.ord + slots;
    gs.start = gs.cls + slots;
    if (total_points > 0)
      pct_kernel<<<OLPT_G(nblk(total_points, kPctWarps)), kPctWarps * 32, smem, s>>>(
          W.points.start.as<int>(), W.points.items.as<int>(), (int)total_points, n,
          W.e_s.as<double>(), gs, W.slot_pct.as<double>(), W.slot_used.as<uint8_t>(),
          counts + PC_FLAG);
    pct_score_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(
        W.fcnt.as<uint8_t>(), M, n, W.slot_pct.as<double>(), W.slot_used.as<uint8_t>(),
        W.e_s.as<double>(), W.pct.as<double>(), W.key.as<uint64_t>(), W.val.as<int>(), counts);
    auto classes = [&](const int* m, const double* val, const int* grp, int* cls, int* mixed,
                       int n_word, int bad) {
      class_count_kernel<<<OLPT_G(n_tile), kClsTile, 0, s>>>(W.val.as<int>(), m, val, grp,
                                                            W.tiles.as<int2>());
      class_assign_kernel<<<OLPT_G(n_tile), kClsTile, 0, s>>>(
          W.val.as<int>(), m, val, grp, W.tiles.as<int2>(), cls, W.cstart.as<int>(), mixed, counts,
          n_word, bad);
    };
    // percentile classes over all candidates with a finite percentile
    radix_sort_device(W, M, 64, s);
    classes(counts + PC_PCT, W.pct.as<double>(), nullptr, W.pcls.as<int>(), nullptr, PC_PCLS, 4);
    // e_check classes inside every percentile class (the reference compares e_check
    // only between candidates of equal percentile), over the candidates the greedy
    // takes: sorted by (percentile class, e_check, index)
    e_keys_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(W.pct.as<double>(), W.e_s.as<double>(), M,
                                                 W.key.as<uint64_t>(), W.val.as<int>());
    radix_sort_device(W, M, 64, s);
    const int bits = bit_width((uint64_t)M);
    group_keys_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(W.val.as<int>(), M, counts,
                                                     W.pcls.as<int>(), (1ull << bits) - 1,
                                                     W.key.as<uint64_t>());
    radix_sort_device(W, M, bits, s);
    OLPT_CUDA(cudaMemsetAsync(W.mixed.p, 0, (size_t)(M + 1) * sizeof(int), s));
    classes(counts + PC_BOTH, W.e_s.as<double>(), W.pcls.as<int>(), W.ecls.as<int>(),
            W.mixed.as<int>(), PC_ECLS, 8);
    // greedy order: e_check class ids already increase with the percentile class, so
    // (class, index) is (percentile class, e_check class, index)
    class_index_sort_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(W.val.as<int>(), W.cstart.as<int>(),
                                                           counts, W.mixed.as<int>());
    W.g_pts.ensure((slots + n) * sizeof(int), s);
    W.g_cnt.ensure(M + 16, s);
    gather_greedy_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(
        W.val.as<int>(), counts, n, W.fl.as<int>(), W.fcnt.as<uint8_t>(), W.pct.as<double>(),
        W.e_s.as<double>(), W.g_pts.as<int>(), W.g_cnt.as<uint8_t>(), W.g_pct.as<double>(),
        W.g_e.as<double>());
    OLPT_CUDA(cudaGetLastError());
    W.gstate.ensure(M + 16, s);
    W.gfirst.ensure(2 * pts * sizeof(unsigned long long), s);
    W.gowner.ensure(pts * sizeof(int), s);
    OLPT_CUDA(cudaMemsetAsync(W.gfirst.p, 0xff, 2 * pts * sizeof(unsigned long long), s));
    OLPT_CUDA(cudaMemsetAsync(W.gowner.p, 0xff, pts * sizeof(int), s));
    const int* a_pts = W.g_pts.as<int>();
    const uint8_t* a_cnt = W.g_cnt.as<uint8_t>();
    uint8_t* a_state = W.gstate.as<uint8_t>();
    unsigned long long* a_first = W.gfirst.as<unsigned long long>();
    int* a_owner = W.gowner.as<int>();
    const int* a_order = W.val.as<int>();
    const double *a_pct = W.g_pct.as<double>(), *a_e = W.g_e.as<double>();
    uint8_t* a_sel = W.sel.as<uint8_t>();
    int* a_scnt = W.scnt.as<int>();
    int n_first = (int)pts;
    void* args[] = {&counts, &a_pts, &a_cnt, &n, &a_state, &a_first, &n_first, &a_owner, &a_order,
                    &a_pct, &a_e, &a_sel, &a_scnt};
    // at most one block an SM: they have to be resident together
    int dev = 0, sms = 1;
    OLPT_CUDA(cudaGetDevice(&dev));
    OLPT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int blocks = std::max(1, std::min(nblk(M, kGreedyThreads), sms));
    OLPT_CUDA(cudaLaunchCooperativeKernel((const void*)greedy_kernel, dim3(OLPT_G(blocks)),
                                          dim3(kGreedyThreads), args, 0, s));
  }
  exclusive_scan(W.scnt.as<int>(), M, W.spos.as<int>(), W.scan_tmp, s);
}

void count_selected(PruneWork& W, int M, cudaStream_t s) {
  if (M > 0)
    sel_count_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(W.sel.as<uint8_t>(), M, W.scnt.as<int>());
  exclusive_scan(W.scnt.as<int>(), M, W.spos.as<int>(), W.scan_tmp, s);
  OLPT_CUDA(cudaGetLastError());
}

}  // namespace olpt
