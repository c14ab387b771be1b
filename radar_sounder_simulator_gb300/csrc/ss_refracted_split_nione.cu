// Split refracted kernels (fast pass and fix-up) for the sequential solve
// of a single crossing.
#include "ss_refracted_split.cuh"

namespace ss {

int split_launch_one(RefArgs &a, const RefSplitConsts &k, const Plan &p,
                     size_t smem, cudaStream_t st) {
  return launch_split_r<kOneNI>(a, k, p, smem, st);
}

int refracted_batch_launch_nione(const RefBatchJob *jobs, int n_jobs,
                               long long n_items, long long n_words,
                               unsigned long long *counter, int rough_kind,
                               bool plain, int ctas, size_t smem,
                               size_t fix_smem, cudaStream_t st) {
  return ref_batch_launch_r<kOneNI>(jobs, n_jobs, n_items, n_words, counter,
                               rough_kind, plain, ctas, smem, fix_smem, st);
}

int refracted_batch_occupancy_nione(int rough_kind, bool plain, size_t smem) {
  return ref_batch_occupancy<kOneNI>(rough_kind, plain, smem);
}

}  // namespace ss
