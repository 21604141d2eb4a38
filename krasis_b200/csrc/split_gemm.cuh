// Host side of split_gemm.cu: how a product with few rows is cut.
#pragma once
#include <cuda_runtime.h>

namespace kb2 {

// 64-wide K blocks per accumulator of an fp32 result.  The tensor core truncates when it adds to an accumulator: the error of a sum grows by
// 1.0e-9 per K (2.1e-6 at K = 2048, 4.4e-6 at 4096, in the 2-norm).  Sums of 512 products meet in fp32 round-to-nearest instead: 4.8e-7 at
// any K measured, what sequential fp32 FMAs have.
constexpr int kSplitChunk = 8;

struct SplitPlan {
  int nt = 0;       // rows of X per tile (a multiple of 16, at most 256)
  int ks = 1;       // CTAs of a cluster that share a tile along K
  int stages = 0;   // depth of the TMA ring
  int chunk = kSplitChunk;   // K blocks per accumulator
};

// false: the 128 x 256 tiles of dense_gemm.cu are the better cut of this product
bool split_gemm_plan(int M, int N, int K, bool out_f32, int num_sms, SplitPlan* out);

// binned rows (one weight matrix per row tile): a CTA per tile and 128 columns, K uncut
SplitPlan split_gemm_binned_plan(int N, int K, bool out_f32, int tile_rows);

cudaError_t launch_split_gemm(const void* x, const void* w, void* out, const float* bias, int M, int N, int K, long long ldo, bool out_f32,
                              const SplitPlan& plan, const int* tile_group, const int* n_tiles_dev, int groups, cudaStream_t s);

}  // namespace kb2
