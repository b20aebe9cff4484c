// Device-wide exclusive prefix sum of int32 counts and a CSR builder
// (count -> scan -> scatter; the order inside a bucket is arbitrary), shared by the
// stereo grid and prune, the shake tile bins and the 3D hash grids.  Implementation: scan.cu.
#pragma once
#include <cuda_runtime.h>

#include "olpt_ctx.cuh"

namespace olpt {

// Entries that lists and grids may have (OLPT_ERR_UNSUPPORTED above).
constexpr int kScanMax = 1 << 24;
inline void require_scan(int64_t n) {
  OLPT_REQUIRE(n <= kScanMax, OLPT_ERR_UNSUPPORTED, "scan longer than 16M entries");
}

// out[0..n] = exclusive scan of in[0..n), out[n] = total.  `tmp` is scratch.  n: up to kScanMax,
// or `most` where several lists that each keep to it are scanned as one.
void exclusive_scan(const int* in, int n, int* out, DevBuf& tmp, cudaStream_t s,
                    int most = kScanMax);

}  // namespace olpt
