// Device candidate ordering and prune (prune.cu); the sequential greedy
// (greedy_select, stereo_host.cpp) remains the fallback.
#pragma once
#include <cuda_runtime.h>

#include "olpt_ctx.cuh"

namespace olpt {

// words of PruneWork::counts
enum PruneCount : int {
  PC_PCT = 0,    // candidates with a finite percentile
  PC_BOTH,       // and a finite e_check: those the greedy can take
  PC_PCLS,       // percentile classes
  PC_ECLS,       // e_check classes
  PC_MIXED,      // some e_check class has members that differ in value
  PC_FLAG,       // a comparator sort must run on the host (a class is not transitive)
  PC_REPLACE,    // the greedy's replacement rule would fire
  PC_LEFT,       // greedy rounds: candidates left undecided (three words)
  PC_N = PC_LEFT + 3
};

bool sort_candidates_device(PruneWork& W, const int* ids, const double* e, const double* X, int M,
                            int n, int max_id, cudaStream_t s);
// Order and greedy of M candidates enqueued on s (nothing waits): kept flags in W.sel, their
// prefix counts in W.spos (total in W.spos[M]); W.counts tells whether they stand.
void prune_device(PruneWork& W, const PruneView& pv, int M, int n, int64_t total_points,
                  cudaStream_t s);
// prefix counts of the kept flags in W.sel -> W.spos
void count_selected(PruneWork& W, int M, cudaStream_t s);

}  // namespace olpt
