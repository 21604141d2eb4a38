// Host side of split_gemm.cu: how a product with few rows, or with fp32 operands, is cut.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace kb2 {

// 64-wide K blocks per accumulator of sums in chunks.  The tensor core truncates when it adds to an accumulator: the error of a sum grows by
// 9.3e-10 per K (2.1e-6 at K = 2048, 4.4e-6 at 4096, in the 2-norm).  Sums of 512 products meet in fp32 round-to-nearest instead: 4.8e-7 at
// any K measured, where sequential fp32 FMAs are 8.1e-7 off at K = 2048 and 1.6e-6 at 8192.  Up to K = 512, where those are 2.0e-7 (K 128)
// to 4.1e-7 (K 512) off, sums of 256: 2.4e-7.
constexpr int kSplitChunk = 8, kSplitChunkShort = 4;
// Products of fewer rows sum in chunks where an fp32 result is asked for (kb2_linear_bf16).
constexpr int kWholeSumRows = 256;

// Shared memory that a CTA of a cluster takes at least when it allocates `cols` columns of tensor memory.  A CTA that waits for tensor memory may have
// cluster peers that others wait for in turn, so CTAs of clusters (of any kernel, on any stream) that share an SM must never ask for more than its 512
// columns together: at 430 bytes per column (1 KB of it is the system's) the 228 KB of an SM hold fewer than 544, and columns come in multiples of 32.
constexpr int tmem_smem(int cols) { return cols * 430 - 1024; }

struct SplitPlan {
  int mt = 0;       // rows of X per tile (a multiple of 16)
  int ks = 1;       // CTAs of a cluster that share a tile along K
  int stages = 0;   // depth of the TMA ring
  int chunk = 0;    // K blocks per accumulator (all of a CTA's: one sum)
  bool pair = false; // three parts of x on pairs of CTAs: tiles of mt rows (a multiple of 32), K in ks segments whose sums meet in a workspace
};

// x [M][K] and w [groups][N][K] as bf16 arrays, or as three bf16 parts of fp32 arrays laid out by launch_split_parts.
struct SplitGemm {
  const void* x = nullptr;
  const void* w = nullptr;
  void* out = nullptr;
  const float* bias = nullptr;
  int M = 0, N = 0, K = 0;
  long long ldo = 0;
  bool out_f32 = false;
  int xparts = 1, wparts = 1;               // 1 or 3; three parts of w only with three of x
  int groups = 1;
  const int* tile_group = nullptr;          // binned rows: matrix of each row tile, and the number of row tiles (device)
  const int* n_tiles_dev = nullptr;
  bool batched = false;                     // every group has M rows of its own: out row m of group g at g * out_group + m * ldo
  long long out_group = 0;
  // the operands the parts were made of (three parts only): an output that is not a number is computed again from them, since parts of an
  // infinity times a zero part are not what the product is
  const float* x_raw = nullptr;
  long long x_ld = 0, x_group = 0;
  const void* w_raw = nullptr;              // fp32 when wparts is 3, else bf16; rows of K
  // W is [gate ; up] of N / 2 rows each and the output [M][N / 2] their gated unit (glu_value, seq_act.cuh) in bf16; both are rounded to bf16 first, as
  // a product and an activation pass would
  bool glu = false;
  int glu_kind = 0;
  float glu_limit = 0.f, glu_alpha = 0.f;
  float* partial = nullptr;                 // pairs with several segments: parts_partial_bytes of workspace
  const uint8_t* w_low = nullptr;           // wparts 3: what launch_split_weights says about the low parts
};

// K blocks for which launch_split_weights says together whether the low parts of 128 rows hold anything: at most 32 such spans, four blocks each where that
// leaves it enough to share out, fewer for small matrices (9 rows, fp32 weights, N 512, K 2048: 18.7 us with four, 13.8 with one).
inline int split_low_span(int N, int K, int groups) {
  const int nkb = K / 64, least = (nkb + 31) / 32;
  int span = 4;
  while (span > 1 && (long long)groups * ((N + 127) / 128) * ((nkb + span - 1) / span) < 512) span /= 2;
  return span > least ? span : least;
}

// The segments' sums of a product on pairs; calls that would take more of them than kPartialMost stay with split_gemm_kernel.
constexpr size_t kPartialMost = 256u << 20;
inline size_t parts_partial_bytes(int M, int N, int groups, int ks) { return ks > 1 ? (size_t)ks * groups * M * N * 4 : 0; }

// One accumulator over all of K, K block by K block: the sums of dense_gemm.cu, bit for bit.  false: not estimated to take less than `us`.
bool split_gemm_plan_whole(int M, int N, int K, int num_sms, float us, SplitPlan* out);
// Whether launch_dense_gemm runs a product on these tiles, and how.
bool dense_gemm_is_split(int M, int N, int K, int num_sms, SplitPlan* out);
// The form launch_dense_gemm runs a product in: -1 these tiles, 0 one CTA per 128 x 256 tile, else the columns of a pair of CTAs; smem: shared memory
// of a CTA of such a pair (0 for the others).
int dense_gemm_form(int M, int N, int K, int num_sms, int* smem);
// Sums in chunks, in an order that depends on N, K, the parts and the groups, not on M.  false: sizes not taken.
bool split_gemm_plan(int M, int N, int K, int num_sms, int xparts, int wparts, int groups, SplitPlan* out);
// binned rows (one weight matrix per row tile): a CTA per tile and 128 columns, K uncut
SplitPlan split_gemm_binned_plan(int K, int tile_rows);

cudaError_t launch_split_gemm(const SplitGemm& g, const SplitPlan& plan, cudaStream_t s);

// fp32 [groups][rows][K] (row stride ld, group stride group_stride) -> bf16 parts hi, mid, lo with hi + mid + lo = value (24 bits), laid out
// [groups][tiles][3][mt][K] with zero rows behind the last one
cudaError_t launch_split_parts(const float* x, long long ld, long long group_stride, int rows, int K, int mt, int groups, void* parts, int num_sms,
                               cudaStream_t s);

// fp32 weights [groups][N][K] -> [3][groups * N][K]; low [groups][tiles of 128 rows][spans]: whether parts two and three of those rows and K blocks
// hold anything.  If not, they are not written.
cudaError_t launch_split_weights(const float* w, int N, int K, int groups, void* parts, uint8_t* low, cudaStream_t s);

}  // namespace kb2
