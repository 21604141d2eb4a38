// Ragged-batch sequence operators: the kernels a decoder needs when one step carries portions of several prompts next to single
// decoded tokens.  Every kernel works on a flat token axis [T] with per-token (sequence, position) and per-sequence
// (first row, state slot, page list) metadata, so prefill, chunked prefill, decode and any mixture run the same code.
//
//   embed_scale            x = table[token] * scale                                   (fp32 residual stream)
//   gemm_nt / gemv_nt      C = A B^T for any M, N, K; fp32 or bf16 operands, fp32 accumulation in a fixed K order per output
//   residual_norm          x += norm(y) (+ x0);  h = layer_norm(x)                    (residual update fused with the next norm)
//   residual_scale_rms     x += m y;  h = x / rms(x) * (shift + w)                    (the same for RMS norms and a residual multiplier)
//   residual_post_rms      z = c1 y1 + c2 y2 + b;  x += m z / rms(z) * w;  h = x or x / rms(x) * wh   (norm on the sublayer's output only)
//   act_mul                gelu_tanh(a) * b                                           (gated feed-forward)
//   side_gate              gelu_tanh(g) * per-layer slice of a token table            (per-layer token input)
//   latent_prep            RMS-normed latent + rotated shared key -> paged cache, rotary on the query's rotated part (any frequency
//                          table); the latent columns follow the queries or come from a buffer of their own
//   latent_window_attn     absorbed-form latent attention over the page list: sliding window, softmax with an optional per-head sink,
//                          optional sigmoid gate per head on the result
//   conv_silu (+ state)    short causal convolution per channel over time with a carried tail, optional bias ahead of the taps or on
//                          their result (or both), then SiLU or nothing; conv_run reads every input once on long steps
//   delta_rule             gated delta rule S <- g S; u = beta (v - S^T k); S += k u^T; o = S^T q, state in fp32 slots,
//                          unit-norm q / k, per-head RMS norm of o with a SiLU or sigmoid gate; g is one decay per head, or one
//                          per head and key channel (it then multiplies the rows of S)
//
// Precision: the residual stream, every norm, softmax, the rotary angles, decays, gates and the recurrent state are fp32 (angles
// are reduced in fp64).  `dt` codes: 0 = float32, 1 = bfloat16.
#include "ptx.cuh"
#include "seq_common.cuh"

namespace kb2seq {

thread_local char g_err[512] = "";
long long g_launches = 0;

// ------------------------------------------------------------------------------------------------ embedding
template <typename T>
__global__ void embed_scale_kernel(const T* __restrict__ table, const int* __restrict__ tokens, float* __restrict__ x, int W,
                                   float scale) {
  kb2::pdl_enter(table, tokens, x);
  const long long t = blockIdx.x;
  const long long row = tokens[t];
  for (int d = threadIdx.x; d < W; d += blockDim.x) x[t * W + d] = ldf(table, row * W + d) * scale;
}
// bf16 tables whose rows start on 16 bytes: eight columns per thread, so that a row's cold loads are all in flight at once
// (4 tokens of 2048 columns took 9.5 us with eight rounds of loads)
__global__ void __launch_bounds__(256) embed_scale_vec_kernel(const bf16* __restrict__ table, const int* __restrict__ tokens, float* __restrict__ x, int W,
                                                              float scale) {
  kb2::pdl_enter(table, tokens, x);
  const long long t = blockIdx.x, row = tokens[t];
  for (int d = threadIdx.x * 8; d < W; d += 256 * 8) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(table + row * W + d), f);
    float4* o = reinterpret_cast<float4*>(x + t * W + d);
    o[0] = make_float4(f[0] * scale, f[1] * scale, f[2] * scale, f[3] * scale);
    o[1] = make_float4(f[4] * scale, f[5] * scale, f[6] * scale, f[7] * scale);
  }
}

// ------------------------------------------------------------------------------------------------ GEMM
// C[M,N] = A[M,K] * B[N,K]^T.  64x64 tile, 16-wide K steps, 4x4 outputs per thread, fp32 FMA.  Each output sums its K products
// in the same order whatever M and N are, so a row's result does not depend on which other rows share the launch.
template <typename TA, typename TB, typename TC>
__global__ void __launch_bounds__(256) gemm_nt_kernel(const TA* __restrict__ A, long long lda, const TB* __restrict__ B, long long ldb,
                                                      TC* __restrict__ C, long long ldc, int M, int N, int K, long long sA,
                                                      long long sB, long long sC) {
  kb2::pdl_enter(A, B, C);
  constexpr int BM = 64, BN = 64, BK = 16;
  __shared__ float As[BK][BM + 4], Bs[BK][BN + 4];
  A += (long long)blockIdx.z * sA;
  B += (long long)blockIdx.z * sB;
  C += (long long)blockIdx.z * sC;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int i = tid + it * 256, r = i >> 4, c = i & 15;
      const int m = m0 + r, n = n0 + r, k = k0 + c;
      As[c][r] = (m < M && k < K) ? ldf(A, (long long)m * lda + k) : 0.f;
      Bs[c][r] = (n < N && k < K) ? ldf(B, (long long)n * ldb + k) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) stf(C, (long long)m * ldc + n, acc[i][j]);
    }
  }
}

// Few rows (decode): one warp per output column, all M <= MR rows at once, so the weight matrix is read once at full width.
template <typename TA, typename TB, typename TC, int MR>
__global__ void __launch_bounds__(256) gemv_nt_kernel(const TA* __restrict__ A, long long lda, const TB* __restrict__ B, long long ldb,
                                                      TC* __restrict__ C, long long ldc, int M, int N, int K, long long sA,
                                                      long long sB, long long sC) {
  kb2::pdl_enter(A, B, C);
  A += (long long)blockIdx.z * sA;
  B += (long long)blockIdx.z * sB;
  C += (long long)blockIdx.z * sC;
  const int lane = threadIdx.x & 31;
  const int n = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (n >= N) return;
  float acc[MR];
#pragma unroll
  for (int m = 0; m < MR; ++m) acc[m] = 0.f;
  const TB* b = B + (long long)n * ldb;
  // eight loads of a row ahead of their sums, which stay in their order (left to the compiler they go out one by one: N 16384, K 2048 in fp32 at one row
  // 64 us instead of 25)
  int k = lane;
  for (; k + 7 * 32 < K; k += 8 * 32) {
    float w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = ldf(b, k + 32 * i);
#pragma unroll
    for (int m = 0; m < MR; ++m) {
      if (m >= M) break;
      float a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = ldf(A, (long long)m * lda + k + 32 * i);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[m] = fmaf(a[i], w[i], acc[m]);
    }
  }
  for (; k < K; k += 32) {
    const float w = ldf(b, k);
#pragma unroll
    for (int m = 0; m < MR; ++m)
      if (m < M) acc[m] = fmaf(ldf(A, (long long)m * lda + k), w, acc[m]);
  }
#pragma unroll
  for (int m = 0; m < MR; ++m) {
    const float v = warp_sum(acc[m]);
    if (lane == 0 && m < M) stf(C, (long long)m * ldc + n, v);
  }
}

template <typename TA> __device__ __forceinline__ void load8(const TA* p, float* f);
template <> __device__ __forceinline__ void load8<float>(const float* p, float* f) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
template <> __device__ __forceinline__ void load8<bf16>(const bf16* p, float* f) { unpack8(*reinterpret_cast<const uint4*>(p), f); }

// fp32 rows and few columns: KS warps of a block share a column.
template <typename TC, int MR, int KS>
__global__ void __launch_bounds__(256) gemv_nt_vec_kernel(const float* __restrict__ A, long long lda, const bf16* __restrict__ B, long long ldb,
                                                          TC* __restrict__ C, long long ldc, int M, int N, int K, long long sA, long long sB,
                                                          long long sC) {
  kb2::pdl_enter(A, B, C);
  A += (long long)blockIdx.z * sA;
  B += (long long)blockIdx.z * sB;
  C += (long long)blockIdx.z * sC;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kpart = warp % KS;
  const int n = (blockIdx.x * (blockDim.x >> 5) + warp) / KS;
  float acc[MR];
#pragma unroll
  for (int m = 0; m < MR; ++m) acc[m] = 0.f;
  // the warps take interleaved pieces of 256; the weights of the next piece are requested before the current ones are used
  const int kstep = 256 * KS;
  int k = (kpart * 32 + lane) * 8;
  const auto weights = [&](int k) { return k < K && n < N ? ld_stream16(B + (long long)n * ldb + k) : make_uint4(0, 0, 0, 0); };
  uint4 wv = weights(k);
  for (; k < K; k += kstep) {
    const uint4 wn = weights(k + kstep);
#pragma unroll
    for (int m = 0; m < MR; ++m)
      if (m < M) {
        float a[8], w[8];
        load8<float>(A + (long long)m * lda + k, a);
        unpack8(wv, w);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[m] = fmaf(a[i], w[i], acc[m]);
      }
    wv = wn;
  }
  __shared__ float red[8][MR];
#pragma unroll
  for (int m = 0; m < MR; ++m) {
    const float v = warp_sum(acc[m]);
    if (lane == 0) red[warp][m] = v;
  }
  __syncthreads();
  if (kpart == 0 && lane < MR) {
    float v = 0.f;
    for (int p = 0; p < KS; ++p) v += red[warp + p][lane];
    if (lane < M && n < N) stf(C, (long long)lane * ldc + n, v);
  }
}

template <typename TC>
static bool launch_gemv_vec(const float* A, long long lda, const bf16* B, long long ldb, TC* C, long long ldc, int M, int N, int K, int batch, long long sA,
                            long long sB, long long sC, cudaStream_t s) {
  if (K % 8 || ldb % 8 || sB % 8 || ((uintptr_t)B & 15) || ((uintptr_t)A & 15) || lda % 4 || sA % 4) return false;
  const dim3 grid((N + 1) / 2, 1, batch);
  auto kern = M <= 4 ? gemv_nt_vec_kernel<TC, 4, 4> : gemv_nt_vec_kernel<TC, 8, 4>;
  kb2::launch_pdl(kern, grid, 256, 0, s, A, lda, B, ldb, C, ldc, M, N, K, sA, sB, sC);
  return true;
}

// ---- few rows against bfloat16 weights, on the warp-level tensor instructions
// Bound: the weights' way from HBM; the arithmetic has to stay out of the way (fp32 FMAs on unpacked values took 200 instructions per KB of
// weights at 4 rows).  A warp owns 16 weight rows (the 16-row side of mma.m16n8k16) and up to 8 rows of A (its 8-column side).  A product
// does not care about the order along K, so a lane takes 16 neighbouring bytes of its weight row and the same 16 of its row of A, and word
// pairs of the two go into two instructions as they are: no shuffles, 64-byte runs per quad and load.  The copies of the steps ahead are on their way
// into a ring of the warp in shared memory, from which every lane reads what it copied itself, so that bytes in flight cost no registers (with the next
// piece in registers: fp32 rows, N 32768, K 2048 42 us instead of 28.5, eight warps on an SM; bf16 rows, N 2048, K 2048 4.0 instead of 3.4).  KS warps of
// a block share the rows and take pieces of 128 numbers in turn.  Each instruction
// pair starts from zero, its 32 products join a compensated running sum, and the warps' sums meet pairwise: the error is that of the FMA form
// (8e-8) or less.  From HBM at 4 rows, us before (gemv_nt_vec) and now: N 16384, K 2048 32.3 -> 13.7 (floor 10.3);
// N 2048, K 8192 19.8 -> 8.2 (5.1); N 32768, K 2048 44.4 -> 24.7 (20.5); N 2048, K 2048 7.3 -> 3.4.
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// the same without an addend
__device__ __forceinline__ void mma16816_new(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// fp32 rows are three bf16 parts, exactly (the leading 8 bits, of what is left the next 8, the rest): the products with the first part go into one
// accumulator, those with the others into a second, and both join the running sum.  The later parts are taken 2^16 times as large: bf16 ends at 2^-133,
// and parts of the smallest numbers lie below; above 2^119 they overflow, and the sum is made again like others that are not finite.  The parts are made
// by every warp for itself, numbers in pairs; so that they serve more weights, its pieces are 32 rows of 64 numbers.  fp32 rows, us before
// (gemv_nt_vec) at 1 / 2 / 4 / 8 rows and now at one and eight: N 65536, K 2048 47.4 / 52.3 / 76.8 / 149, 56.8 / 58; N 32768 27.4 / 30.2 / 40.4 / 79.9,
// 29.4 / 29.6; N 16384 17.7 / 19.5 / 29.6 / 48.6, 17.0 / 17.2; N 2048 5.2 / 6.0 / 8.3 / 12.7, 4.6 / 5.3; N 512, K 512 2.6 /
// 2.8 / 3.5 / 5.8, 1.9; error 1.6e-7 before, 6e-8 to 8e-8 now.  A sum that is not finite is made again in plain fp32 (the parts of an infinity are not
// numbers).
template <bool kFp32, int kTiles> struct GemvPiece {
  static constexpr int kRows = 16 * kTiles;                                    // weight rows of a warp
  static constexpr int kSteps = kFp32 ? 2 : 4, kLen = 32 * kSteps;             // of K, 32 a step
  // warps of a block: few of them share a group's sums, so that the SMs get the same number of warps (N 65536: 14 at most instead of 16)
  static constexpr int warps(int ks) { return kFp32 ? (ks < 2 ? 2 : ks) : ks > 8 ? 16 : 8; }
  static constexpr int kLoads = 2 * kTiles + (kFp32 ? 2 : 1);                  // 16-byte copies of a lane and step, the weights' first
  static constexpr int kStages = kLoads > 4 ? 4 : kFp32 ? 6 : 8, kRing = kStages * kLoads * 512;  // bytes of a warp's ring
};

// Two fp32 numbers that go through the arithmetic together.
struct Pair {
  uint64_t v;
  __device__ __forceinline__ static Pair of(uint32_t a, uint32_t b) {
    Pair p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "r"(a), "r"(b));
    return p;
  }
  __device__ __forceinline__ static Pair of(float a, float b) { return of(__float_as_uint(a), __float_as_uint(b)); }
  __device__ __forceinline__ void get(uint32_t& a, uint32_t& b) const { asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v)); }
};
__device__ __forceinline__ Pair add2(Pair a, Pair b) {
  Pair p;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(p.v) : "l"(a.v), "l"(b.v));
  return p;
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
  Pair p;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p.v) : "l"(a.v), "l"(b.v));
  return p;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
  Pair p;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return p;
}

// {the bf16 that leads the first, the one that leads the second}; what is left of them
__device__ __forceinline__ uint32_t lead_pair(Pair& f) {
  uint32_t a, b;
  f.get(a, b);
  f = fma2(Pair::of(a & 0xffff0000u, b & 0xffff0000u), Pair::of(-1.f, -1.f), f);
  return __byte_perm(a, b, 0x7632);
}

// A product in plain fp32 by a warp; K a multiple of 8, both rows 16-byte aligned.
__device__ __noinline__ float row_product(const float* a, const bf16* b, int K, int lane) {
  float v = 0.f;
  for (int k = lane * 8; k < K; k += 256) {
    float x[8], w[8];
    load8(a + k, x);
    load8(b + k, w);
#pragma unroll
    for (int i = 0; i < 8; ++i) v = fmaf(x[i], w[i], v);
  }
  return warp_sum(v);
}

// kShare: the blocks of a cluster along y share the pieces
template <typename TA, typename TC, int KS, int kTiles, bool kShare>
__global__ void __launch_bounds__(32 * GemvPiece<sizeof(TA) == 4, kTiles>::warps(KS))
    gemv_mma_kernel(const TA* __restrict__ A, long long lda, const bf16* __restrict__ B, long long ldb, TC* __restrict__ C, long long ldc, int M, int N, int K,
                    long long sA, long long sB, long long sC) {
  constexpr bool kFp32 = sizeof(TA) == 4;
  using P = GemvPiece<kFp32, kTiles>;
  constexpr int kRows = P::kRows, kWarps = P::warps(KS), kGroups = kWarps / KS, kW = 2 * kTiles;
  kb2::pdl_enter(A, B, C);
  extern __shared__ __align__(16) uint8_t gemv_ring[];
  __shared__ float red[kWarps][8][kRows + 1];            // [warp][row of A][weight row], odd pitch
  A += (long long)blockIdx.z * sA;
  B += (long long)blockIdx.z * sB;
  C += (long long)blockIdx.z * sC;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quad = lane >> 2, t8 = (lane & 3) * 8;
  const int n0 = (blockIdx.x * kGroups + warp / KS) * kRows;
  // rows beyond the last one are read as the last one and not written
  const bf16* w[kW];
#pragma unroll
  for (int i = 0; i < kW; ++i) w[i] = B + (long long)min(n0 + quad + 8 * i, N - 1) * ldb + t8;
  const TA* x = A + (long long)min(quad, M - 1) * lda + t8;
  const bool row = quad < M;
  uint8_t* ring = gemv_ring + warp * P::kRing + lane * 16;     // a lane reads what it copied itself: no barrier
  const int parts = kShare ? KS * gridDim.y : KS, part = kShare ? warp % KS + KS * blockIdx.y : warp % KS;
  const int pieces = (K + P::kLen - 1) / P::kLen, steps = n0 < N ? (pieces - part + parts - 1) / parts * P::kSteps : 0;
  auto fetch = [&](int i) {
    if (i < steps) {
      const int k = ((i / P::kSteps) * parts + part) * P::kLen + i % P::kSteps * 32;
      const uint32_t to = kb2::smem_u32(ring + i % P::kStages * (P::kLoads * 512));
      const bool in = k + t8 < K;
      const int at = in ? k : 0;                           // the step's address from one base (fp32) or from two: each the faster for its rows, by 4 %
#pragma unroll
      for (int r = 0; r < kW; ++r) cp_async16_stream(to + r * 512, kFp32 ? w[r] + at : in ? w[r] + k : w[r], in);
#pragma unroll
      for (int h = 0; h < P::kLoads - kW; ++h) cp_async16(to + (kW + h) * 512, kFp32 ? x + at + 4 * h : in ? x + k : x, in && row);
    }
    kb2::cp_async_commit();
  };
  float sum[kTiles][4] = {}, lost[kTiles][4] = {};
  Pair total[kTiles][2], kept[kTiles][2];                // fp32 rows: sums, and what their last additions rounded off
#pragma unroll
  for (int t = 0; t < kTiles; ++t) total[t][0] = total[t][1] = kept[t][0] = kept[t][1] = Pair::of(0.f, 0.f);
  auto join = [&](int t, int i, float add) {             // compensated: what the addition rounds off goes into the next one
    const float s = sum[t][i] + add;
    // an infinity stays one: inf - inf must not reach the next addition
    lost[t][i] = isfinite(s) ? (s - sum[t][i]) - add : 0.f;
    sum[t][i] = s;
  };
#pragma unroll
  for (int i = 0; i < P::kStages - 1; ++i) fetch(i);
#pragma unroll 1
  for (int i = 0; i < steps; ++i) {
    kb2::cp_async_wait<P::kStages - 2>();
    const uint4* at = reinterpret_cast<const uint4*>(ring + i % P::kStages * (P::kLoads * 512));
    uint4 v[P::kLoads];
#pragma unroll
    for (int r = 0; r < P::kLoads; ++r) v[r] = at[r * 32];
    if constexpr (kFp32) {
      const uint4 x0 = v[kW], x1 = v[kW + 1];
      Pair f[4] = {Pair::of(x0.x, x0.y), Pair::of(x0.z, x0.w), Pair::of(x1.x, x1.y), Pair::of(x1.z, x1.w)};
      uint32_t part[3][4];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          part[q][i] = lead_pair(f[i]);
          if (q == 0) f[i] = mul2(f[i], Pair::of(65536.f, 65536.f));
        }
      }
#pragma unroll
      for (int t = 0; t < kTiles; ++t) {
        const uint4 a = v[2 * t], c = v[2 * t + 1];
        float d[4], e[4];
        mma16816_new(e, a.x, c.x, a.y, c.y, part[2][0], part[2][1]);
        mma16816(e, a.z, c.z, a.w, c.w, part[2][2], part[2][3]);
        mma16816(e, a.x, c.x, a.y, c.y, part[1][0], part[1][1]);
        mma16816(e, a.z, c.z, a.w, c.w, part[1][2], part[1][3]);
        mma16816_new(d, a.x, c.x, a.y, c.y, part[0][0], part[0][1]);
        mma16816(d, a.z, c.z, a.w, c.w, part[0][2], part[0][3]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const Pair add = add2(Pair::of(d[2 * i], d[2 * i + 1]), fma2(Pair::of(e[2 * i], e[2 * i + 1]), Pair::of(1.f / 65536.f, 1.f / 65536.f), kept[t][i]));
          const Pair s = add2(total[t][i], add);
          kept[t][i] = add2(fma2(s, Pair::of(-1.f, -1.f), total[t][i]), add);
          total[t][i] = s;
        }
      }
    } else {
      const uint4 a = v[0], c = v[1];
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      mma16816(d, a.x, c.x, a.y, c.y, v[2].x, v[2].y);
      mma16816(d, a.z, c.z, a.w, c.w, v[2].z, v[2].w);
#pragma unroll
      for (int i = 0; i < 4; ++i) join(0, i, d[i] - lost[0][i]);
    }
    fetch(i + P::kStages - 1);
  }
  if constexpr (kFp32)
#pragma unroll
    for (int t = 0; t < kTiles; ++t)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t a, b;
        total[t][i].get(a, b);
        sum[t][2 * i] = __uint_as_float(a);
        sum[t][2 * i + 1] = __uint_as_float(b);
      }
  // of a tile sum[0], [1]: weight row quad, rows 2 (lane & 3) and + 1 of A; [2], [3]: weight row quad + 8
  const int m = (lane & 3) * 2;
#pragma unroll
  for (int t = 0; t < kTiles; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) red[warp][m + (i & 1)][16 * t + quad + (i >> 1) * 8] = sum[t][i];
  __syncthreads();
  constexpr int kOut = kGroups * 8 * kRows;
  auto total_of = [&](int i) {
    const int g = i / (8 * kRows), mm = i / kRows % 8, r = i % kRows;
    float v[KS];
#pragma unroll
    for (int p = 0; p < KS; ++p) v[p] = red[g * KS + p][mm][r];
#pragma unroll
    for (int o = KS / 2; o > 0; o >>= 1)
#pragma unroll
      for (int p = 0; p < o; ++p) v[p] += v[p + o];
    return v[0];
  };
  auto finish = [&](int i, float v) {
    const int g = i / (8 * kRows), mm = i / kRows % 8, r = i % kRows, n = (blockIdx.x * kGroups + g) * kRows + r;
    const bool in = mm < M && n < N;
    if constexpr (kFp32) {
      for (unsigned again = __ballot_sync(0xffffffffu, in && !isfinite(v)); again; again &= again - 1) {      // the whole warp for one output after the other
        const int src = __ffs(again) - 1;
        const float t = row_product(A + (long long)__shfl_sync(0xffffffffu, mm, src) * lda, B + (long long)__shfl_sync(0xffffffffu, n, src) * ldb, K, lane);
        if (lane == src) v = t;
      }
    }
    if (in) stf(C, (long long)mm * ldc + n, v);
  };
  if constexpr (kShare) {
    static_assert(kOut <= kWarps * 32, "an output per thread");
    __shared__ float whole[kOut];
    const int i = threadIdx.x;
    if (i < kOut) whole[i] = total_of(i);
    kb2::cluster_sync_all();
    if (blockIdx.y == 0 && i < kOut) {                     // whole warps
      float v = whole[i];
      for (unsigned b = 1; b < gridDim.y; ++b) {
        float of;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(of) : "r"(kb2::cluster_addr(whole + i, b)) : "memory");
        v += of;
      }
      finish(i, v);
    }
    kb2::cluster_sync_all();                               // nobody leaves while its sums are read
  } else {
    for (int i = threadIdx.x; i < kOut; i += kWarps * 32) finish(i, total_of(i));
  }
}

template <typename TA, typename TC, int kTiles>
static void launch_gemv_tiles(const void* A, long long lda, const void* B, long long ldb, void* C, long long ldc, int M, int N, int K,
                            int batch, long long sA, long long sB, long long sC, cudaStream_t s) {
  using Piece = GemvPiece<sizeof(TA) == 4, kTiles>;
  const int groups = (N + Piece::kRows - 1) / Piece::kRows;
  int ks = 1;                                  // about 2048 warps, in one wave of two blocks per SM, as long as each has a piece of K
  while (ks < 16 && (long long)groups * batch * 2 * ks <= 2368 && K > Piece::kLen * ks) ks *= 2;
  const int warps = Piece::warps(ks), per = warps / ks;
  // few columns and a long K: up to four blocks along K where SMs stand idle, as long as a warp has more than four steps of fp32 rows to share out, eight
  // of bf16 (us without and with them, four rows: fp32, K 8192, N 288 10.2 / 5.9, N 512 10.3 / 6.3, N 1024 10.5 / 8.4, N 300, K 16384 18.2 / 8.1; bf16
  // 7.2 / 5.0, 7.2 / 5.4, 7.5 / 7.0, 12.7 / 6.4; below the line, fp32, N 1024, K 2048 3.8 / 4.5, bf16, N 512, K 4096 4.5 / 4.9)
  unsigned blocks = 1;
  if (ks == 16 && K > 32 * ks * (sizeof(TA) == 4 ? 4 : 8))
    while (blocks < 4 && (long long)groups * batch * 2 * blocks <= kb2::current_sms() && K > 128 * ks * (int)blocks) blocks *= 2;
  const dim3 grid((groups + per - 1) / per, blocks, batch);
  const size_t smem = (size_t)warps * Piece::kRing;
#define KB2_GEMV(KSV, SHARE)                                                                                                                     \
  do {                                                                                                                                           \
    kb2::allow_smem<gemv_mma_kernel<TA, TC, KSV, kTiles, SHARE>>(Piece::warps(KSV) * Piece::kRing);                                              \
    kb2::launch_pdl_clusters(gemv_mma_kernel<TA, TC, KSV, kTiles, SHARE>, grid, 32 * warps, smem, s, dim3(1, blocks, 1), (const TA*)A, lda, (const bf16*)B,  \
                             ldb, (TC*)C, ldc, M, N, K, sA, sB, sC);                                                                             \
  } while (0)
  if (blocks > 1) KB2_GEMV(16, true);
  else if (ks == 16) KB2_GEMV(16, false);
  else if (ks == 8) KB2_GEMV(8, false);
  else if (ks == 4) KB2_GEMV(4, false);
  else if (ks == 2) KB2_GEMV(2, false);
  else KB2_GEMV(1, false);
#undef KB2_GEMV
}

template <typename TA, typename TC>
static bool launch_gemv_mma(const void* A, long long lda, const void* B, long long ldb, void* C, long long ldc, int M, int N, int K,
                            int batch, long long sA, long long sB, long long sC, cudaStream_t s) {
  constexpr int kA16 = 16 / sizeof(TA);
  if (K % 8 || ldb % 8 || sB % 8 || ((uintptr_t)B & 15) || ((uintptr_t)A & 15) || lda % kA16 || sA % kA16) return false;
  // at any number of rows, so that a row's sums do not depend on the rows beside it; bf16 rows, gemv_nt_vec, us at 1 / 2 / 4 / 8 rows and here at any:
  // N 512, K 1024 2.7 / 3.5 / 5.3 / 9.7, 2.1; N 4096, K 224 2.3 / 2.7 / 3.4 / 5.2, 2.2; N 256, K 2048 2.2 / 2.6 / 3.5 / 5.6, 2.7; N 128, K 8192
  // 3.9 / 5.6 / 9.2 / 17, 4.8
  if constexpr (sizeof(TA) == 4) {             // 32 weight rows a warp where that still gives every SM a block (N 2048, K 8192: 15.9 us, with 16 rows 11.2)
    if ((long long)((N + 31) / 32) * batch >= kb2::current_sms()) {
      launch_gemv_tiles<TA, TC, 2>(A, lda, B, ldb, C, ldc, M, N, K, batch, sA, sB, sC, s);
      return true;
    }
  }
  launch_gemv_tiles<TA, TC, 1>(A, lda, B, ldb, C, ldc, M, N, K, batch, sA, sB, sC, s);
  return true;
}

template <typename TA, typename TB, typename TC>
static void launch_gemm(const void* A, long long lda, const void* B, long long ldb, void* C, long long ldc, int M, int N, int K,
                        int batch, long long sA, long long sB, long long sC, cudaStream_t s) {
  if (M <= 8) {
    if constexpr (sizeof(TB) == 2) {
      // fp32 rows, few columns and a long K: sixteen rows a block would leave the weights to a handful of SMs, and with one row the FMAs are few (us at
      // 1 / 2 / 4 / 8 rows, N 256, K 2048 2.2 / 2.6 / 3.5 / 5.5 here, 3.5 at any on the tensor cores; N 128, K 8192 5.5 / 6.6 / 9.9 / 17.6, 10.4 there with
      // all of K in one block.  With K shared by four blocks N 288 takes 5.8 / 5.8 / 5.9 / 6.6 there: from two rows on this line lies too high for long K)
      if constexpr (sizeof(TA) == 4) {
        if ((long long)N * batch <= 256 && K >= 2048 && launch_gemv_vec((const float*)A, lda, (const bf16*)B, ldb, (TC*)C, ldc, M, N, K, batch, sA, sB, sC, s)) return;
      }
      if (launch_gemv_mma<TA, TC>(A, lda, B, ldb, C, ldc, M, N, K, batch, sA, sB, sC, s)) return;
    }
    dim3 grid((N + 7) / 8, 1, batch);
    kb2::launch_pdl(gemv_nt_kernel<TA, TB, TC, 8>, grid, 256, 0, s, (const TA*)A, lda, (const TB*)B, ldb, (TC*)C, ldc, M, N, K, sA, sB, sC);
  } else {
    dim3 grid((N + 63) / 64, (M + 63) / 64, batch);
    kb2::launch_pdl(gemm_nt_kernel<TA, TB, TC>, grid, 256, 0, s, (const TA*)A, lda, (const TB*)B, ldb, (TC*)C, ldc, M, N, K, sA, sB, sC);
  }
}

// ------------------------------------------------------------------------------------------------ residual update + norm
// One block per token row.  x (fp32) += norm_a(y) where norm_a is a layer norm (y_mode 1: weight wa, bias ba), an RMS norm
// (y_mode 2: weight wa), the plain sum y + y2 (y_mode 3: two sublayers that read the same normed input; y2 may be null) or absent
// (y == nullptr); x += x0 if given; then h = layer_norm(x; wb, bb) if h is given (bb == nullptr: no bias).
// Variances are means of squared deviations (two passes over the row held in shared memory).
__global__ void __launch_bounds__(256) residual_norm_kernel(float* __restrict__ x, const float* __restrict__ y, int y_mode,
                                                            const float* __restrict__ wa, const float* __restrict__ ba,
                                                            const float* __restrict__ x0, const float* __restrict__ wb,
                                                            const float* __restrict__ bb, void* __restrict__ h, int dt_h, int W,
                                                            float eps, const float* __restrict__ y2) {
  kb2::pdl_enter(x, y, wa, ba, x0, wb, bb, h, y2);
  extern __shared__ float rowbuf[];
  __shared__ float red[32];
  const long long row = blockIdx.x;
  float* xr = x + row * W;
  const float inv_w = 1.f / (float)W;
  if (y != nullptr) {
    const float* yr = y + row * W;
    float s = 0.f;
    for (int d = threadIdx.x; d < W; d += blockDim.x) {
      const float v = yr[d];
      rowbuf[d] = v;
      s += y_mode == 1 ? v : v * v;
    }
    s = block_sum(s, red);
    float mean = 0.f, rstd;
    if (y_mode == 3) {
      for (int d = threadIdx.x; d < W; d += blockDim.x) {
        float v = rowbuf[d];
        if (y2 != nullptr) v += y2[row * W + d];
        v += xr[d];
        if (x0 != nullptr) v += x0[row * W + d];
        xr[d] = v;
        rowbuf[d] = v;
      }
      rstd = 0.f;
    } else if (y_mode == 1) {
      mean = s * inv_w;
      float q = 0.f;
      for (int d = threadIdx.x; d < W; d += blockDim.x) {
        const float c = rowbuf[d] - mean;
        q += c * c;
      }
      q = block_sum(q, red);
      rstd = 1.f / sqrtf(q * inv_w + eps);
    } else {
      rstd = 1.f / sqrtf(s * inv_w + eps);
    }
    for (int d = threadIdx.x; y_mode != 3 && d < W; d += blockDim.x) {
      float v = (rowbuf[d] - mean) * rstd * wa[d];
      if (y_mode == 1) v += ba[d];
      v += xr[d];
      if (x0 != nullptr) v += x0[row * W + d];
      xr[d] = v;
      rowbuf[d] = v;
    }
  } else {
    for (int d = threadIdx.x; d < W; d += blockDim.x) {
      float v = xr[d];
      if (x0 != nullptr) {
        v += x0[row * W + d];
        xr[d] = v;
      }
      rowbuf[d] = v;
    }
  }
  if (h == nullptr) return;
  float s = 0.f;
  for (int d = threadIdx.x; d < W; d += blockDim.x) s += rowbuf[d];
  const float mean = block_sum(s, red) * inv_w;
  float q = 0.f;
  for (int d = threadIdx.x; d < W; d += blockDim.x) {
    const float c = rowbuf[d] - mean;
    q += c * c;
  }
  q = block_sum(q, red);
  const float rstd = 1.f / sqrtf(q * inv_w + eps);
  for (int d = threadIdx.x; d < W; d += blockDim.x) st_dt(h, dt_h, row * W + d, (rowbuf[d] - mean) * rstd * wb[d] + (bb != nullptr ? bb[d] : 0.f));
}

// The same for widths that are multiples of 4 up to 1024 NV: a thread keeps its 4 NV columns in registers and asks for everything the row
// needs before the first sum, and a sum over the block costs one barrier.  Bound by traffic on long steps, by the chain of (up to) four sums
// on short ones: 4 rows of 2048 7.5 -> 2.7 us.
template <int NV>
__global__ void __launch_bounds__(256) residual_norm_vec_kernel(float* __restrict__ x, const float* __restrict__ y, int y_mode,
                                                                const float* __restrict__ wa, const float* __restrict__ ba,
                                                                const float* __restrict__ x0, const float* __restrict__ wb,
                                                                const float* __restrict__ bb, void* __restrict__ h, int dt_h, int W, float eps,
                                                                const float* __restrict__ y2) {
  kb2::pdl_enter(x, y, wa, ba, x0, wb, bb, h, y2);
  kb2::pdl_trigger();
  __shared__ float red[4][8];
  const long long base = (long long)blockIdx.x * W;
  const int tid = threadIdx.x;
  const float inv_w = 1.f / (float)W;
  int turn = 0;
  auto row_sum = [&](float v) {                // four sums at most, each in a row of `red` of its own
    v = warp_sum(v);
    float* r = red[turn++ & 3];
    if ((tid & 31) == 0) r[tid >> 5] = v;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += r[i];
    return t;
  };
  auto at = [&](int i) { return (i * 256 + tid) * 4; };
  auto load = [&](const float* p, int i) {
    return p != nullptr && at(i) < W ? *reinterpret_cast<const float4*>(p + at(i)) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  auto row = [&](const float* p) { return p != nullptr ? p + base : nullptr; };
  float4 v[NV], yv[NV], av[NV], cv[NV], gv[NV], bv[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    v[i] = load(row(x), i);
    yv[i] = load(row(y), i);
    av[i] = load(row(x0), i);
    cv[i] = load(row(y2), i);
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    gv[i] = load(y != nullptr && y_mode != 3 ? wa : nullptr, i);
    bv[i] = load(y != nullptr && y_mode == 1 ? ba : nullptr, i);
  }
  auto sum4 = [](const float4& q) { return (q.x + q.y) + (q.z + q.w); };
  auto sq4 = [](const float4& q, float m) {
    const float a = q.x - m, b = q.y - m, c = q.z - m, d = q.w - m;
    return (a * a + b * b) + (c * c + d * d);
  };
  auto squares = [&](const float4 (&q)[NV], float m) {      // columns beyond the row do not count
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) t += at(i) < W ? sq4(q[i], m) : 0.f;
    return t;
  };
  if (y != nullptr && y_mode != 3) {
    float mean = 0.f;
    if (y_mode == 1) {
      float t = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) t += sum4(yv[i]);
      mean = row_sum(t) * inv_w;
    }
    const float rstd = 1.f / sqrtf(row_sum(squares(yv, mean)) * inv_w + eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      v[i].x += fmaf((yv[i].x - mean) * rstd, gv[i].x, bv[i].x);
      v[i].y += fmaf((yv[i].y - mean) * rstd, gv[i].y, bv[i].y);
      v[i].z += fmaf((yv[i].z - mean) * rstd, gv[i].z, bv[i].z);
      v[i].w += fmaf((yv[i].w - mean) * rstd, gv[i].w, bv[i].w);
    }
  } else {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      v[i].x += yv[i].x + cv[i].x;
      v[i].y += yv[i].y + cv[i].y;
      v[i].z += yv[i].z + cv[i].z;
      v[i].w += yv[i].w + cv[i].w;
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    v[i].x += av[i].x;
    v[i].y += av[i].y;
    v[i].z += av[i].z;
    v[i].w += av[i].w;
    if ((y != nullptr || x0 != nullptr) && at(i) < W) *reinterpret_cast<float4*>(x + base + at(i)) = v[i];
    gv[i] = load(h != nullptr ? wb : nullptr, i);
    bv[i] = load(h != nullptr ? bb : nullptr, i);
  }
  if (h == nullptr) return;
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) t += sum4(v[i]);
  const float mean = row_sum(t) * inv_w;
  const float rstd = 1.f / sqrtf(row_sum(squares(v, mean)) * inv_w + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (at(i) >= W) continue;
    const float4 o = make_float4(fmaf((v[i].x - mean) * rstd, gv[i].x, bv[i].x), fmaf((v[i].y - mean) * rstd, gv[i].y, bv[i].y),
                                 fmaf((v[i].z - mean) * rstd, gv[i].z, bv[i].z), fmaf((v[i].w - mean) * rstd, gv[i].w, bv[i].w));
    if (dt_h == 0) {
      *reinterpret_cast<float4*>((float*)h + base + at(i)) = o;
    } else {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(o.x, o.y), hi = __floats2bfloat162_rn(o.z, o.w);
      *reinterpret_cast<uint2*>((bf16*)h + base + at(i)) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  }
}

static int launch_residual_norm(float* x, const float* y, int y_mode, const float* wa, const float* ba, const float* x0, const float* wb,
                                const float* bb, void* h, int dt_h, int T, int W, float eps, const float* y2, cudaStream_t s) {
  const uintptr_t all = (uintptr_t)x | (uintptr_t)y | (uintptr_t)wa | (uintptr_t)ba | (uintptr_t)x0 | (uintptr_t)wb | (uintptr_t)bb | (uintptr_t)h | (uintptr_t)y2;
  if (W % 4 == 0 && W <= 8192 && !(all & 15)) {
#define KB2_RN(NVV) kb2::launch_pdl(residual_norm_vec_kernel<NVV>, T, 256, 0, s, x, y, y_mode, wa, ba, x0, wb, bb, h, dt_h, W, eps, y2)
    if (W <= 1024) KB2_RN(1); else if (W <= 2048) KB2_RN(2); else if (W <= 4096) KB2_RN(4); else KB2_RN(8);
#undef KB2_RN
  } else {
    const size_t smem = (size_t)W * 4;
    if (smem > 48 * 1024) SEQ_CUDA(cudaFuncSetAttribute(residual_norm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kb2::launch_pdl(residual_norm_kernel, T, 256, smem, s, x, y, y_mode, wa, ba, x0, wb, bb, h, dt_h, W, eps, y2);
  }
  SEQ_LAUNCHED();
  return KB2SEQ_OK;
}

// One block per token row.  x (fp32) += y_mult * y (y may be null); then h = x / sqrt(mean(x^2) + eps) * (w_shift + w) if h is given
// (w_shift 1: w holds the offset from one).  h may be x itself when y is null and dt_h is fp32 (a norm in place).
__global__ void __launch_bounds__(256) residual_scale_rms_kernel(float* x, const float* __restrict__ y, float y_mult,
                                                                 const float* __restrict__ w, float w_shift, void* h, int dt_h, int W,
                                                                 float eps) {
  kb2::pdl_enter(x, y, w, h);
  extern __shared__ float rowbuf[];
  __shared__ float red[32];
  const long long row = blockIdx.x;
  float* xr = x + row * W;
  float s = 0.f;
  for (int d = threadIdx.x; d < W; d += blockDim.x) {
    float v = xr[d];
    if (y != nullptr) {
      v = fmaf(y_mult, y[row * W + d], v);
      xr[d] = v;
    }
    rowbuf[d] = v;
    s = fmaf(v, v, s);
  }
  if (h == nullptr) return;
  s = block_sum(s, red);
  const float rstd = 1.f / sqrtf(s / (float)W + eps);
  for (int d = threadIdx.x; d < W; d += blockDim.x) st_dt(h, dt_h, row * W + d, rowbuf[d] * rstd * (w_shift + w[d]));
}

// Norm on the sublayer's output only; the next sublayer reads the residual stream as it is.  One block per token row:
// z = c1 y1 + c2 y2 + bias (y2, bias may be null), x (fp32) += mult * z / sqrt(mean(z^2) + eps) * w; then, if h is given, h = x in dt_h, or
// with wh x / sqrt(mean(x^2) + eps) * wh (the norm ahead of the head).  y1 == nullptr: x is left as it is.  V columns per access.
template <int V>
__global__ void __launch_bounds__(256) residual_post_rms_kernel(float* __restrict__ x, const float* __restrict__ y1, float c1,
                                                                const float* __restrict__ y2, float c2, const float* __restrict__ bias,
                                                                float mult, const float* __restrict__ w, const float* __restrict__ wh,
                                                                void* __restrict__ h, int dt_h, int W, float eps) {
  kb2::pdl_enter(x, y1, y2, bias, w, wh, h);
  extern __shared__ __align__(16) float rowbuf[];
  __shared__ float red[32];
  const long long base = (long long)blockIdx.x * W;
  auto load = [](const float* p, float* v) {
    if constexpr (V == 4) {
      const float4 f = *reinterpret_cast<const float4*>(p);
      v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else {
      v[0] = p[0];
    }
  };
  auto store = [](float* p, const float* v) {
    if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else p[0] = v[0];
  };
  auto store_h = [&](int d, const float* v) {
    if (dt_h == 0) {
      store((float*)h + base + d, v);
    } else if constexpr (V == 4) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
      uint2 o;
      o.x = *reinterpret_cast<const uint32_t*>(&lo);
      o.y = *reinterpret_cast<const uint32_t*>(&hi);
      *reinterpret_cast<uint2*>((bf16*)h + base + d) = o;
    } else {
      ((bf16*)h)[base + d] = __float2bfloat16_rn(v[0]);
    }
  };
  float ss = 0.f, rstd = 0.f;
  if (y1 != nullptr) {
    for (int d = threadIdx.x * V; d < W; d += blockDim.x * V) {
      float z[V];
      load(y1 + base + d, z);
#pragma unroll
      for (int i = 0; i < V; ++i) z[i] *= c1;
      if (y2 != nullptr) {
        float t[V];
        load(y2 + base + d, t);
#pragma unroll
        for (int i = 0; i < V; ++i) z[i] = fmaf(c2, t[i], z[i]);
      }
      if (bias != nullptr) {
        float t[V];
        load(bias + d, t);
#pragma unroll
        for (int i = 0; i < V; ++i) z[i] += t[i];
      }
      store(rowbuf + d, z);
#pragma unroll
      for (int i = 0; i < V; ++i) ss = fmaf(z[i], z[i], ss);
    }
    rstd = mult / sqrtf(block_sum(ss, red) / (float)W + eps);
    ss = 0.f;
  }
  for (int d = threadIdx.x * V; d < W; d += blockDim.x * V) {        // a thread reads back the columns it wrote
    float xv[V];
    load(x + base + d, xv);
    if (y1 != nullptr) {
      float z[V], wv[V];
      load(rowbuf + d, z);
      load(w + d, wv);
#pragma unroll
      for (int i = 0; i < V; ++i) xv[i] = fmaf(z[i] * rstd, wv[i], xv[i]);
      store(x + base + d, xv);
    }
    if (wh != nullptr) {
      store(rowbuf + d, xv);
#pragma unroll
      for (int i = 0; i < V; ++i) ss = fmaf(xv[i], xv[i], ss);
    } else if (h != nullptr) {
      store_h(d, xv);
    }
  }
  if (wh == nullptr || h == nullptr) return;
  rstd = 1.f / sqrtf(block_sum(ss, red) / (float)W + eps);
  for (int d = threadIdx.x * V; d < W; d += blockDim.x * V) {
    float xv[V], wv[V];
    load(rowbuf + d, xv);
    load(wh + d, wv);
#pragma unroll
    for (int i = 0; i < V; ++i) xv[i] = xv[i] * rstd * wv[i];
    store_h(d, xv);
  }
}

// ------------------------------------------------------------------------------------------------ elementwise
__global__ void act_mul_kernel(const void* __restrict__ in, int dt_in, void* __restrict__ out, int dt_out, long long T, int F) {
  kb2::pdl_enter(in, out);
  const long long t = blockIdx.y;
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= F) return;
  const float a = ld_dt(in, dt_in, t * 2 * F + f), b = ld_dt(in, dt_in, t * 2 * F + F + f);
  st_dt(out, dt_out, t * F + f, gelu_tanh(a) * b);
}
// fp32 in and out, F a multiple of 4: 16-byte accesses (512 rows of 8192: 16.9 -> 7.9 us, 50 MB)
__global__ void __launch_bounds__(256) act_mul_f32x4_kernel(const float* __restrict__ in, float* __restrict__ out, int F) {
  kb2::pdl_enter(in, out);
  const long long t = blockIdx.y;
  const int f = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (f >= F) return;
  const float4 a = *reinterpret_cast<const float4*>(in + t * 2 * F + f), b = *reinterpret_cast<const float4*>(in + t * 2 * F + F + f);
  *reinterpret_cast<float4*>(out + t * F + f) = make_float4(gelu_tanh(a.x) * b.x, gelu_tanh(a.y) * b.y, gelu_tanh(a.z) * b.z, gelu_tanh(a.w) * b.w);
}
// bf16 in and out, F a multiple of 8: 16-byte accesses
__global__ void act_mul_bf16x8_kernel(const bf16* __restrict__ in, bf16* __restrict__ out, int F) {
  kb2::pdl_enter(in, out);
  kb2::pdl_trigger();
  const long long t = blockIdx.y;
  const int f = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (f >= F) return;
  float a[8], b[8];
  unpack8(*reinterpret_cast<const uint4*>(in + t * 2 * F + f), a);
  unpack8(*reinterpret_cast<const uint4*>(in + t * 2 * F + F + f), b);
  uint4 o;
  __nv_bfloat162* po = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) po[i] = __floats2bfloat162_rn(gelu_tanh(a[2 * i]) * b[2 * i], gelu_tanh(a[2 * i + 1]) * b[2 * i + 1]);
  *reinterpret_cast<uint4*>(out + t * F + f) = o;
}

__global__ void side_gate_kernel(const float* __restrict__ g, const void* __restrict__ table, int dt_table, long long table_ld,
                                 const int* __restrict__ tokens, int col0, int dim, long long T, void* __restrict__ out, int dt_out) {
  kb2::pdl_enter(g, table, tokens, out);
  kb2::pdl_trigger();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * dim) return;
  const long long t = i / dim;
  const int d = (int)(i - t * dim);
  const float e = ld_dt(table, dt_table, (long long)tokens[t] * table_ld + col0 + d);
  st_dt(out, dt_out, i, gelu_tanh(g[i]) * e);
}

// ------------------------------------------------------------------------------------------------ latent attention
// proj [T, ldp] fp32 = [q (H x (dn + dr)) | latent (r) | shared rotated key (dr)].  Per token: RMS-normed latent and rotated key part
// go to the page the token's position maps to; the query's rotated parts are rotated in place.
__global__ void __launch_bounds__(512) latent_prep_kernel(float* __restrict__ proj, long long ldp, int H, int dn, int dr, int r,
                                                          const float* __restrict__ cw, float eps, const double* __restrict__ freq,
                                                          int rot_dims, float amp, const int* __restrict__ positions,
                                                          const int* __restrict__ seq_of, const int* __restrict__ pages, int max_pages,
                                                          int page_size, void* __restrict__ ckv, void* __restrict__ kr, int dt_cache,
                                                          const float* __restrict__ lat_rows, long long ldl) {
  kb2::pdl_enter(proj, cw, freq, positions, seq_of, pages, ckv, kr, lat_rows);
  __shared__ float red[32];
  const long long t = blockIdx.x;
  const int pos = positions[t];
  float* p = proj + t * ldp;
  const long long slot = (long long)pages[(long long)seq_of[t] * max_pages + pos / page_size] * page_size + pos % page_size;
  const float* lat = lat_rows != nullptr ? lat_rows + t * ldl : p + (long long)H * (dn + dr);
  float ss = 0.f;
  if (threadIdx.x < 128)                     // the first four warps' sum, whatever else the block has
    for (int d = threadIdx.x; d < r; d += 128) ss += lat[d] * lat[d];
  ss = block_sum(ss, red);
  const float rstd = 1.f / sqrtf(ss / (float)r + eps);
  for (int d = threadIdx.x; d < r; d += blockDim.x) st_dt(ckv, dt_cache, slot * r + d, lat[d] * rstd * cw[d]);
  const int half = rot_dims / 2;
  // (H + 1) vectors of dr: the heads' query parts (in place) and the shared key part (to the cache)
  for (int i = threadIdx.x; i < (H + 1) * half; i += blockDim.x) {
    const int hh = i / half, j = i - hh * half;
    float c, s;
    rot_cs(pos, freq[j], amp, &c, &s);
    if (hh < H) {
      float* q = p + (long long)hh * (dn + dr) + dn;
      const float u = q[2 * j], v = q[2 * j + 1];
      q[2 * j] = u * c - v * s;
      q[2 * j + 1] = v * c + u * s;
    } else {
      const float* k = lat + r;
      const float u = k[2 * j], v = k[2 * j + 1];
      st_dt(kr, dt_cache, slot * dr + 2 * j, u * c - v * s);
      st_dt(kr, dt_cache, slot * dr + 2 * j + 1, v * c + u * s);
    }
  }
  for (int d = rot_dims + threadIdx.x; d < dr; d += blockDim.x) st_dt(kr, dt_cache, slot * dr + d, lat[r + d]);
}

// Absorbed form: score(t, h, j) = (q_abs[t,h] . c_j + q_rot[t,h] . kr_j) * scale over the keys j of the token's sequence with
// 0 <= pos - j < window; the softmax denominator also holds exp(sink_h) (a key with no value: running max starts at the sink,
// running sum at 1).  Output: sum_j p_j c_j (the value up-projection follows as a per-head GEMM).
// One block per (token, group of HG heads, piece of the key range); keys in tiles of 32, in shared memory as fp32 rows whose pitch is an
// odd number of 16-byte units, so that a lane per key reads 16 bytes without bank conflicts.
//   scores    every warp takes an eighth of the dimensions for all HG heads: one 16-byte read of a key row serves HG dot products, whose
//             pieces meet in shared memory
//   values    a thread owns NC columns for all HG heads: one read of a latent element serves HG sums
// Bound where few tokens decode: latency, a chain of position, page, key rows and four phases on them.  Loads of a phase go out together, and the key range is
// cut into pieces of 8 keys and more, so that short contexts reach all SMs, too (4 tokens x 16 heads, 116 keys, from HBM: pieces of 32 18.6 us, now 11.4).
// Where many do: instructions.  A thread finds its next unit of a row by addition, and the lanes' step through the scores is a constant in two forms of the loop or
// three: a layer of 16 heads, 127 tokens after 1000 keys, with a division per unit and a variable step 434 us (bf16) and 1443 (fp32, 4 bytes a load), now 362 and 458.
// gate [T, ldg] (may be null): head h's output is multiplied by sigmoid(gate[t, h]); it commutes with the value up-projection.
constexpr int kAttnThreads = 256, kAttnAcc = 16, kAttnKT = 32, kAttnWarps = kAttnThreads / 32;
constexpr int kAttnPiece = 8;              // keys of a piece are a multiple of this
__device__ __forceinline__ float head_gate(const float* __restrict__ gate, long long ldg, long long t, int h) {
  return gate != nullptr ? 1.f / (1.f + expf(-gate[t * ldg + h])) : 1.f;
}
__host__ __device__ inline int attn_q_pitch(int D) { return (D + 3) / 4 * 4; }
__host__ __device__ inline int attn_k_pitch(int D) { return attn_q_pitch(D) / 4 % 2 ? attn_q_pitch(D) : attn_q_pitch(D) + 4; }
__host__ __device__ inline size_t attn_smem_floats(int HG, int D) {
  return 2 * kAttnKT + (size_t)HG * attn_q_pitch(D) + (size_t)kAttnKT * attn_k_pitch(D) + (size_t)kAttnWarps * HG * kAttnKT + (size_t)kAttnKT * HG + 3 * HG;
}
template <int HG, int NC>
__global__ void __launch_bounds__(kAttnThreads, 2) latent_window_attn_kernel(
    const float* __restrict__ q_abs, const float* __restrict__ proj, long long ldp, int H, int dn, int dr, int r,
    const void* __restrict__ ckv, const void* __restrict__ kr, int dt_cache, const int* __restrict__ positions,
    const int* __restrict__ seq_of, const int* __restrict__ pages, int max_pages, int page_size, const float* __restrict__ sinks,
    float scale, int window, float* __restrict__ out, const int* __restrict__ cu, int skip_from, int nsplit,
    float* __restrict__ part_acc, float* __restrict__ part_ml, const float* __restrict__ gate, long long ldg, bool vec_q, bool vec_k) {
  kb2::pdl_enter(q_abs, proj, ckv, kr, positions, seq_of, pages, sinks, out, cu, part_acc, part_ml, gate);
  static_assert(HG <= kAttnWarps, "a warp per head runs the softmax");
  constexpr int KT = kAttnKT;
  extern __shared__ __align__(16) float sm[];
  if (cu != nullptr) {                    // sequences whose portion has skip_from tokens or more are served by another kernel
    const int sq = seq_of[blockIdx.x];
    if (cu[sq + 1] - cu[sq] >= skip_from) return;
  }
  const int D = r + dr, QP = attn_q_pitch(D), DP = attn_k_pitch(D), n4 = QP >> 2;
  long long* krow = (long long*)sm;       // [KT] cache rows of the tile's keys
  float* qs = sm + 2 * KT;                // [HG][QP], zeros beyond the head's D numbers and beyond the last head
  float* kt = qs + HG * QP;               // [KT][DP]
  float* sp = kt + KT * DP;               // [warps][HG][KT] pieces of the scores
  float* pr = sp + kAttnWarps * HG * KT;  // [KT][HG] weights
  float* m_run = pr + KT * HG;            // [HG]
  float* l_run = m_run + HG;              // [HG]
  float* alpha = l_run + HG;              // [HG]
  const long long t = blockIdx.x;
  const int h0 = blockIdx.y * HG;
  const int nh = min(HG, H - h0);
  const int pos = positions[t], seq = seq_of[t];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // nsplit > 1: block z takes the z-th piece of the token's key range and leaves an unnormalised partial result (running max, sum,
  // weighted latents) for latent_attn_combine_kernel; the sink belongs to piece 0
  const int z = blockIdx.z;
  const int j_lo = max(0, pos - window + 1);
  int j_begin = j_lo, j_end = pos;
  if (nsplit > 1) {
    const int piece = (((pos - j_lo + 1) + nsplit - 1) / nsplit + kAttnPiece - 1) / kAttnPiece * kAttnPiece;
    j_begin = j_lo + z * piece;
    j_end = min(pos, j_begin + piece - 1);
  }
  if (j_begin > j_end) {                  // no keys: the join takes the pieces ahead of the first empty one (a whole range always has its own position)
    if (tid < nh) {
      part_ml[((t * nsplit + z) * H + h0 + tid) * 2] = -INFINITY;
      part_ml[((t * nsplit + z) * H + h0 + tid) * 2 + 1] = 0.f;
    }
    return;
  }
  const auto row_of = [&](int j) { return (long long)pages[(long long)seq * max_pages + j / page_size] * page_size + j % page_size; };
  if (tid < KT && j_begin + tid <= j_end) krow[tid] = row_of(j_begin + tid);      // of the first tile, under way together with the query
  if (vec_q) {                            // sizes, strides and pointers in units of four numbers: five loads of a thread in flight
    constexpr int kAhead = 5;
    for (int base = tid; base < HG * n4; base += kAhead * kAttnThreads) {
      float4 v[kAhead];
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        const int u = base + i * kAttnThreads, hh = u / n4, d = (u - hh * n4) * 4;
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (hh < nh)
          v[i] = *reinterpret_cast<const float4*>(d < r ? q_abs + (t * H + h0 + hh) * r + d : proj + t * ldp + (long long)(h0 + hh) * (dn + dr) + dn + (d - r));
      }
#pragma unroll
      for (int i = 0; i < kAhead; ++i)
        if (base + i * kAttnThreads < HG * n4) reinterpret_cast<float4*>(qs)[base + i * kAttnThreads] = v[i];
    }
  } else {
    for (int i = tid; i < HG * QP; i += kAttnThreads) {
      const int hh = i / QP, d = i - hh * QP;
      float v = 0.f;
      if (hh < nh && d < D) v = d < r ? q_abs[(t * H + h0 + hh) * r + d] : proj[t * ldp + (long long)(h0 + hh) * (dn + dr) + dn + (d - r)];
      qs[i] = v;
    }
  }
  for (int i = tid; i < KT * (DP - D); i += kAttnThreads) {      // the rows' padding stays zero: tiles write D numbers per row only
    const int k = i / (DP - D);
    kt[k * DP + D + i - k * (DP - D)] = 0.f;
  }
  if (tid < HG) {
    const bool sk = z == 0 && sinks != nullptr && tid < nh;       // no sinks: an ordinary softmax over the keys
    m_run[tid] = sk ? sinks[h0 + tid] : -INFINITY;
    l_run[tid] = sk ? 1.f : 0.f;
  }
  float acc[NC][HG];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int hh = 0; hh < HG; ++hh) acc[c][hh] = 0.f;
  // numbers of 16 bytes of a cache row, and such units a row (0: rows that are not made of them)
  const int unit = dt_cache ? 8 : 4, units = vec_k ? D / unit : 0;
  const int first_k = units ? tid / units : 0, first_d = tid - first_k * units, ahead_k = units ? kAttnThreads / units : 0, ahead_d = kAttnThreads - ahead_k * units;
  const int seg = (n4 + kAttnWarps - 1) / kAttnWarps, u_lo = min(n4, warp * seg), u_hi = min(n4, u_lo + seg);
  for (int j0 = j_begin; j0 <= j_end; j0 += KT) {
    const int nk = min(KT, j_end - j0 + 1);
    __syncthreads();
    if (j0 > j_begin) {
      if (tid < nk) krow[tid] = row_of(j0 + tid);
      __syncthreads();
    }
    if (units) {
      // 16 bytes at a time, three loads of a thread in flight; a thread's next unit is ahead_k rows and ahead_d units on
      for (int k = first_k, d = first_d; k < nk;) {
        constexpr int kAhead = 3;
        uint4 v[kAhead];
        int at[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
          const int c = d * unit;
          at[j] = k < nk ? k * DP + c : -1;
          if (k < nk) {
            const long long row = krow[k];
            v[j] = *reinterpret_cast<const uint4*>((const char*)(c < r ? ckv : kr) + ((c < r ? row * r + c : row * dr + (c - r)) << (dt_cache ? 1 : 2)));
          }
          k += ahead_k;
          d += ahead_d;
          if (d >= units) {
            d -= units;
            ++k;
          }
        }
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
          if (at[j] < 0) continue;
          if (dt_cache) {
            float f[8];
            unpack8(v[j], f);
            *reinterpret_cast<float4*>(kt + at[j]) = make_float4(f[0], f[1], f[2], f[3]);
            *reinterpret_cast<float4*>(kt + at[j] + 4) = make_float4(f[4], f[5], f[6], f[7]);
          } else {
            *reinterpret_cast<uint4*>(kt + at[j]) = v[j];
          }
        }
      }
    } else {
      for (int i = tid; i < nk * D; i += kAttnThreads) {
        const int k = i / D, d = i - k * D;
        kt[k * DP + d] = d < r ? ld_dt(ckv, dt_cache, krow[k] * r + d) : ld_dt(kr, dt_cache, krow[k] * dr + (d - r));
      }
    }
    __syncthreads();
    // scores: a lane per key, a piece of the dimensions per warp, all heads of the group; of up to 8 or 16 keys four or two lanes share one
    const auto scores = [&](auto lanes) {
      constexpr int kKeys = decltype(lanes)::value, kStep = 32 / kKeys;
      const int key = lane & (kKeys - 1);
      float s[HG];
#pragma unroll
      for (int hh = 0; hh < HG; ++hh) s[hh] = 0.f;
      if (key < nk) {
        const float4* kk = reinterpret_cast<const float4*>(kt + key * DP);
        const float4* qq = reinterpret_cast<const float4*>(qs);
#pragma unroll(kKeys == 32 ? 2 : 1)
        for (int u = u_lo + lane / kKeys; u < u_hi; u += kStep) {
          const float4 kv = kk[u];
#pragma unroll
          for (int hh = 0; hh < HG; ++hh) {
            const float4 qv = qq[hh * n4 + u];
            s[hh] = fmaf(qv.x, kv.x, s[hh]);
            s[hh] = fmaf(qv.y, kv.y, s[hh]);
            s[hh] = fmaf(qv.z, kv.z, s[hh]);
            s[hh] = fmaf(qv.w, kv.w, s[hh]);
          }
        }
      }
#pragma unroll
      for (int o = kKeys; o < 32; o <<= 1)
#pragma unroll
        for (int hh = 0; hh < HG; ++hh) s[hh] += __shfl_xor_sync(0xffffffffu, s[hh], o);
#pragma unroll
      for (int hh = 0; hh < HG; ++hh) sp[(warp * HG + hh) * KT + lane] = s[hh];
    };
    if (nk > 16) scores(std::integral_constant<int, 32>{});
    else if (nk > 8) scores(std::integral_constant<int, 16>{});
    else scores(std::integral_constant<int, 8>{});
    __syncthreads();
    // running softmax: warp hh serves head hh
    if (warp < HG) {
      float p = 0.f;
      if (warp < nh) {
        const float m_old = m_run[warp];
        float sc = -INFINITY;
        if (lane < nk) {
          float dot = 0.f;
#pragma unroll
          for (int w = 0; w < kAttnWarps; ++w) dot += sp[(w * HG + warp) * KT + lane];
          sc = dot * scale;
        }
        const float m_new = fmaxf(m_old, warp_max(sc));
        if (lane < nk) p = expf(sc - m_new);
        const float lsum = warp_sum(p);
        if (lane == 0) {
          const float al = m_old == -INFINITY ? 0.f : expf(m_old - m_new);
          alpha[warp] = al;
          l_run[warp] = l_run[warp] * al + lsum;
          m_run[warp] = m_new;
        }
      } else if (lane == 0) {
        alpha[warp] = 0.f;
      }
      pr[lane * HG + warp] = p;
    }
    __syncthreads();
    {
#pragma unroll
      for (int hh = 0; hh < HG; ++hh) {
        const float al = alpha[hh];
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[c][hh] *= al;
      }
      for (int k = 0; k < nk; ++k) {
        float p[HG];
        if constexpr (HG % 4 == 0) {
#pragma unroll
          for (int q = 0; q < HG / 4; ++q) {
            const float4 f = *reinterpret_cast<const float4*>(pr + k * HG + 4 * q);
            p[4 * q] = f.x; p[4 * q + 1] = f.y; p[4 * q + 2] = f.z; p[4 * q + 3] = f.w;
          }
        } else {
#pragma unroll
          for (int hh = 0; hh < HG; ++hh) p[hh] = pr[k * HG + hh];
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int d = tid + c * kAttnThreads;
          if (d < r) {
            const float v = kt[k * DP + d];
#pragma unroll
            for (int hh = 0; hh < HG; ++hh) acc[c][hh] = fmaf(p[hh], v, acc[c][hh]);
          }
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int hh = 0; hh < HG; ++hh) {
    if (hh >= nh) continue;
    const float f = nsplit > 1 ? 1.f : head_gate(gate, ldg, t, h0 + hh);
    const float l = l_run[hh];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int d = tid + c * kAttnThreads;
      if (d < r) {
        if (nsplit > 1) part_acc[((t * nsplit + z) * H + h0 + hh) * r + d] = acc[c][hh];
        else out[(t * H + h0 + hh) * r + d] = acc[c][hh] / l * f;
      }
    }
  }
  if (nsplit > 1 && tid < nh) {
    part_ml[((t * nsplit + z) * H + h0 + tid) * 2] = m_run[tid];
    part_ml[((t * nsplit + z) * H + h0 + tid) * 2 + 1] = l_run[tid];
  }
}

// out[t, h, :] = sum_z w_z acc_z / sum_z w_z l_z with w_z = exp(m_z - max_z m_z); pieces without keys come last and have l_z = 0
__global__ void __launch_bounds__(512) latent_attn_combine_kernel(const float* __restrict__ part_acc, const float* __restrict__ part_ml,
                                                                  int H, int r, int nsplit, float* __restrict__ out,
                                                                  const int* __restrict__ seq_of, const int* __restrict__ cu, int skip_from,
                                                                  const float* __restrict__ gate, long long ldg) {
  kb2::pdl_enter(part_acc, part_ml, out, seq_of, cu, gate);
  kb2::pdl_trigger();
  extern __shared__ float wz[];           // [nsplit]
  __shared__ float red[32];
  const long long t = blockIdx.x;
  const int h = blockIdx.y;
  if (cu != nullptr) {
    const int sq = seq_of[t];
    if (cu[sq + 1] - cu[sq] >= skip_from) return;
  }
  auto ml = [&](int z) { return *reinterpret_cast<const float2*>(part_ml + ((t * nsplit + z) * H + h) * 2); };
  float M = -INFINITY;
  int there = 0;
  for (int z0 = 0; z0 < nsplit; z0 += blockDim.x) {
    const int z = z0 + threadIdx.x;
    const float2 v = z < nsplit ? ml(z) : make_float2(0.f, 0.f);
    if (v.y > 0.f) M = fmaxf(M, v.x);
    there += __syncthreads_count(v.y > 0.f);
  }
  M = warp_max(M);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = M;
  __syncthreads();
  for (int w = 0; w < (int)blockDim.x >> 5; ++w) M = fmaxf(M, red[w]);
  float L = 0.f;
  for (int z = threadIdx.x; z < nsplit; z += blockDim.x) {
    const float2 v = ml(z);
    const float w = v.y > 0.f ? expf(v.x - M) : 0.f;
    wz[z] = w;
    L = fmaf(w, v.y, L);
  }
  L = block_sum(L, red);
  const float f = head_gate(gate, ldg, t, h) / L;
  const float* pa = part_acc + (t * nsplit * H + h) * r;
  const long long step = (long long)H * r;
  for (int d = threadIdx.x; d < r; d += blockDim.x) {
    float v = 0.f;
#pragma unroll 8
    for (int z = 0; z < there; ++z) v = fmaf(wz[z], pa[z * step + d], v);
    out[(t * H + h) * r + d] = v * f;
  }
}

// ------------------------------------------------------------------------------------------------ short convolution + delta rule
// y[t, c] = act(bias_out[c] + sum_j taps[c, j] * x[i - (K - 1) + j, c]) with i the token's index in its portion and x = proj + bias (either
// bias may be null); act 1: silu, 0: none.  Inputs before the portion come from the sequence's carried tail (the last K - 1 inputs of earlier portions,
// bias included; zeros at the start of a sequence).
__global__ void conv_silu_kernel(const float* __restrict__ proj, long long ldp, int C, int K, const float* __restrict__ taps,
                                 const float* __restrict__ tail, const int* __restrict__ seq_of, const int* __restrict__ cu,
                                 const int* __restrict__ slots, long long T, float* __restrict__ out, const float* __restrict__ bias,
                                 int act, const float* __restrict__ bias_out) {
  kb2::pdl_enter(proj, taps, tail, seq_of, cu, slots, out, bias, bias_out);
  const long long t = blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const long long idx = t * C + c;
  const int s = seq_of[t];
  const int i = (int)(t - cu[s]);
  const float* tl = tail + ((long long)slots[s] * C + c) * (K - 1);
  const float b = bias != nullptr ? bias[c] : 0.f;
  float acc = bias_out != nullptr ? bias_out[c] : 0.f;
  for (int j = 0; j < K; ++j) {
    const int src = i - (K - 1) + j;
    const float xv = src >= 0 ? proj[(t - i + src) * ldp + c] + b : tl[(K - 1) + src];
    acc = fmaf(taps[(long long)c * K + j], xv, acc);
  }
  out[idx] = act ? silu(acc) : acc;
}

// The same for long steps and K <= kConvMaxTaps: a thread owns a channel over kConvRun consecutive rows and keeps the last K inputs in
// registers, so that every input is read once (plus K - 1 rows of overlap per run) instead of K times.
constexpr int kConvMaxTaps = 8, kConvRun = 16;
__global__ void __launch_bounds__(256) conv_run_kernel(const float* __restrict__ proj, long long ldp, int C, int K,
                                                       const float* __restrict__ taps, const float* __restrict__ tail,
                                                       const int* __restrict__ seq_of, const int* __restrict__ cu,
                                                       const int* __restrict__ slots, long long T, float* __restrict__ out,
                                                       const float* __restrict__ bias, int act, const float* __restrict__ bias_out) {
  kb2::pdl_enter(proj, taps, tail, seq_of, cu, slots, out, bias, bias_out);
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const long long r0 = (long long)blockIdx.y * kConvRun, r1 = min(T, r0 + kConvRun);
  float w[kConvMaxTaps], x[kConvMaxTaps] = {};     // x[j]: the input K - 1 - j rows back, x[K - 1] the current one
#pragma unroll
  for (int j = 0; j < kConvMaxTaps; ++j) w[j] = j < K ? taps[(long long)c * K + j] : 0.f;
  const float b = bias != nullptr ? bias[c] : 0.f, b_out = bias_out != nullptr ? bias_out[c] : 0.f;
  int s = -1;
  for (long long t = r0; t < r1; ++t) {
    const int st = seq_of[t];
    if (st != s || t == r0) {                        // first row of this run, or of another sequence: fetch the K - 1 earlier inputs
      s = st;
      const int i = (int)(t - cu[s]);
      const float* tl = tail + ((long long)slots[s] * C + c) * (K - 1);
#pragma unroll
      for (int j = 0; j < kConvMaxTaps - 1; ++j)
        if (j < K - 1) {
          const int src = i - (K - 1) + j;
          x[j + 1] = src >= 0 ? proj[(t - i + src) * ldp + c] + b : tl[(K - 1) + src];
        }
    }
#pragma unroll
    for (int j = 0; j < kConvMaxTaps - 1; ++j) x[j] = x[j + 1];
    // after the shift x[0 .. K - 2] hold the K - 1 earlier inputs; the current one goes to x[K - 1]
    const float cur = proj[t * ldp + c] + b;
    float acc = b_out;
#pragma unroll
    for (int j = 0; j < kConvMaxTaps; ++j) {
      if (j == K - 1) x[j] = cur;
      if (j < K) acc = fmaf(w[j], x[j], acc);
    }
    out[t * C + c] = act ? silu(acc) : acc;
  }
}

// The same for 2 to 4 taps and channels in groups of four: a thread takes four channels over kConvRun rows, all of which it asks for before the first is used
// (each thread reads back what it copied itself, so nothing but its own groups is waited for).  Bound by traffic: each input read once, plus K - 1 rows per run,
// mostly from L2; each output written once.  With four rows in
// flight per thread and a branch in every quotient of silu: 100 / 1000 / 4000 tokens x 8192 channels 10.6 / 24.6 / 88.0 us; without the branches 80 (4096), and
// with all rows ahead 6.3 / 16.5 / 54.4 (4.8 TB/s).
constexpr int kConvThreads = 128;
template <int K> constexpr int kConvSmem = (kConvRun + K - 1) * kConvThreads * 16;
template <int K>
__global__ void __launch_bounds__(kConvThreads, 5) conv_run_vec_kernel(const float* __restrict__ proj, long long ldp, int C, const float* __restrict__ taps,
                                                                      const float* __restrict__ tail, const int* __restrict__ seq_of, const int* __restrict__ cu,
                                                                      const int* __restrict__ slots, long long T, float* __restrict__ out,
                                                                      const float* __restrict__ bias, int act, const float* __restrict__ bias_out) {
  kb2::pdl_enter(proj, taps, tail, seq_of, cu, slots, out, bias, bias_out);
  extern __shared__ __align__(16) float4 conv_rows[];    // [K - 1 rows ahead of the run, the run][thread]
  const int c = (blockIdx.x * kConvThreads + threadIdx.x) * 4;
  if (c >= C) return;
  const long long r0 = (long long)blockIdx.y * kConvRun, r1 = min(T, r0 + kConvRun);
  float4* mine = conv_rows + threadIdx.x;
#pragma unroll
  for (int i = 1 - K; i < kConvRun; ++i) {
    if (i >= 0 ? r0 + i < r1 : r0 > 0) kb2::cp_async16(mine + (i + K - 1) * kConvThreads, proj + (r0 + i) * ldp + c);
    if (i >= 0 && i % 4 == 3) kb2::cp_async_commit();
  }
  int s = seq_of[r0];
  const bool one = seq_of[r1 - 1] == s && r1 - r0 == kConvRun;
  const long long first = cu[s];
  float w[4][K], x[K - 1][4], b[4], bo[4];               // x[j]: the input K - 1 - j rows back
#pragma unroll
  for (int e = 0; e < 4; ++e) {
#pragma unroll
    for (int j = 0; j < K; ++j) w[e][j] = taps[(long long)(c + e) * K + j];
    b[e] = bias != nullptr ? bias[c + e] : 0.f;
    bo[e] = bias_out != nullptr ? bias_out[c + e] : 0.f;
  }
  auto before = [&](long long t, int at) {               // the K - 1 inputs ahead of row t, which is number `at` of sequence s
#pragma unroll
    for (int j = 0; j < K - 1; ++j) {
      const int src = at - (K - 1) + j;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        x[j][e] = src >= 0 ? proj[(t - at + src) * ldp + c + e] + b[e] : tail[((long long)slots[s] * C + c + e) * (K - 1) + (K - 1) + src];
    }
  };
  auto row = [&](long long t) {
    const float4 in = mine[(t - r0 + K - 1) * kConvThreads];
    const float cur[4] = {in.x + b[0], in.y + b[1], in.z + b[2], in.w + b[3]};
    float acc[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      acc[e] = bo[e];
#pragma unroll
      for (int j = 0; j < K - 1; ++j) acc[e] = fmaf(w[e][j], x[j][e], acc[e]);
      acc[e] = fmaf(w[e][K - 1], cur[e], acc[e]);
#pragma unroll
      for (int j = 0; j < K - 2; ++j) x[j][e] = x[j + 1][e];
      x[K - 2][e] = cur[e];
      if (act) acc[e] = silu(acc[e]);
    }
    *reinterpret_cast<float4*>(out + t * C + c) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  };
  if (!one) {                                            // a sequence begins in the run, or the step ends in it
    kb2::cp_async_wait<0>();
    s = -1;
#pragma unroll 1
    for (long long t = r0; t < r1; ++t) {
      if (const int q = seq_of[t]; q != s) {
        s = q;
        before(t, (int)(t - cu[s]));
      }
      row(t);
    }
    return;
  }
  kb2::cp_async_wait<3>();
  if (r0 - first >= K - 1) {
#pragma unroll
    for (int j = 0; j < K - 1; ++j) {
      const float4 in = mine[j * kConvThreads];
      x[j][0] = in.x + b[0]; x[j][1] = in.y + b[1]; x[j][2] = in.z + b[2]; x[j][3] = in.w + b[3];
    }
  } else {
    before(r0, (int)(r0 - first));
  }
  auto four = [&](int i0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) row(r0 + i0 + i);
  };
  static_assert(kConvRun == 16, "a group of four rows per wait");
  four(0);
  kb2::cp_async_wait<2>();
  four(4);
  kb2::cp_async_wait<1>();
  four(8);
  kb2::cp_async_wait<0>();
  four(12);
}

// after the convolution: the tail becomes the last K - 1 inputs seen so far (one thread per (sequence, channel), ascending order)
__global__ void conv_tail_kernel(const float* __restrict__ proj, long long ldp, int C, int K, float* __restrict__ tail,
                                 const int* __restrict__ cu, const int* __restrict__ slots, int S, const float* __restrict__ bias) {
  kb2::pdl_enter(proj, tail, cu, slots, bias);
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)S * C) return;
  const int s = (int)(idx / C), c = (int)(idx - (long long)s * C);
  const int t0 = cu[s], n = cu[s + 1] - cu[s];
  float* tl = tail + ((long long)slots[s] * C + c) * (K - 1);
  const float b = bias != nullptr ? bias[c] : 0.f;
  for (int j = 0; j < K - 1; ++j) {
    const int src = n - (K - 1) + j;         // index in the portion of the input that lands in tail[j]
    tl[j] = src >= 0 ? proj[(long long)(t0 + src) * ldp + c] + b : tl[j + n];
  }
}

// One block per (sequence, head); thread j owns column j of the head's state S [dk][dv] (kept in shared memory for the portion).
// conv [T, C] = silu(conv(q | k | v)); proj holds the gate (g_off), the decay input (a_off) and the write-strength input (b_off).
// ch 0: one decay per (token, head), from a[t, h] and dt_bias[h].  ch 1: one per (token, head, key channel), from a[t, h dk + i] and
// dt_bias[h dk + i]; it multiplies the rows of the state.  gate_act 0: silu(gate), 1: sigmoid(gate).
constexpr int kDeltaTile = 16;
__global__ void __launch_bounds__(1024) delta_rule_kernel(const float* __restrict__ conv, int C, const float* __restrict__ bproj,
                                                          long long ldb, const float* __restrict__ aproj, long long lda, int ch,
                                                          const float* __restrict__ gproj, long long ldg, int gate_act, int H, int Hk,
                                                          int dk, int dv, const float* __restrict__ A_log,
                                                          const float* __restrict__ dt_bias, const float* __restrict__ norm_w, float eps,
                                                          float* __restrict__ state, const int* __restrict__ cu,
                                                          const int* __restrict__ slots, void* __restrict__ out, int dt_out, int dvb,
                                                          float* __restrict__ o_raw) {
  kb2::pdl_enter(conv, bproj, aproj, gproj, A_log, dt_bias, norm_w, state, cu, slots, out, o_raw);
  // dvb = value columns of this block (the columns of the state do not meet in the recurrence).  dvb < dv: blockIdx.z picks the slice,
  // the raw read-out goes to o_raw [T, H, dv] and the norm and gate are left to delta_out_kernel.
  extern __shared__ float sm[];
  float* S = sm;                                  // [dk][dvb]
  float* qn = S + (long long)dk * dvb;            // [tile][dk]
  float* kn = qn + kDeltaTile * dk;               // [tile][dk]
  float* ob = kn + kDeltaTile * dk;               // [tile][dvb]
  float* beta = ob + kDeltaTile * dvb;            // [tile]
  float* dec = beta + kDeltaTile;                 // [tile] or [tile][dk]
  const int dstr = ch ? dk : 1;
  const int s = blockIdx.x, h = blockIdx.y, hk = h / (H / Hk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int t0 = cu[s], n = cu[s + 1] - cu[s];
  const int col0 = blockIdx.z * dvb, nc = min(dvb, dv - col0);
  float* Sg = state + ((long long)slots[s] * H + h) * dk * dv + col0;
  for (int i = tid; i < dk * nc; i += blockDim.x) S[(i / nc) * dvb + i % nc] = Sg[(long long)(i / nc) * dv + i % nc];
  const double rate_h = exp((double)A_log[h]);
  const float qscale = 1.f / sqrtf((float)dk);
  const int q_col = hk * dk, k_col = Hk * dk + hk * dk, v_col = 2 * Hk * dk + h * dv;
  for (int b0 = 0; b0 < n; b0 += kDeltaTile) {
    const int nt = min(kDeltaTile, n - b0);
    __syncthreads();
    for (int tt = warp; tt < nt; tt += nw) {
      const float* row = conv + (long long)(t0 + b0 + tt) * C;
      float sq = 0.f, sk = 0.f;
      for (int i = lane; i < dk; i += 32) {
        const float qv = row[q_col + i], kv = row[k_col + i];
        sq += qv * qv;
        sk += kv * kv;
      }
      sq = warp_sum(sq);
      sk = warp_sum(sk);
      const float rq = qscale / sqrtf(sq + 1e-6f), rk = 1.f / sqrtf(sk + 1e-6f);
      for (int i = lane; i < dk; i += 32) {
        qn[tt * dk + i] = row[q_col + i] * rq;
        kn[tt * dk + i] = row[k_col + i] * rk;
      }
      const float* ar = aproj + (long long)(t0 + b0 + tt) * lda + (long long)h * dstr;
      for (int i = lane; i < dstr; i += 32) dec[tt * dstr + i] = decay_from_rate(rate_h, ar[i], dt_bias[h * dstr + i]);
      if (lane == 0) beta[tt] = 1.f / (1.f + expf(-bproj[(long long)(t0 + b0 + tt) * ldb + h]));
    }
    __syncthreads();
    if (tid < nc) {
      for (int tt = 0; tt < nt; ++tt) {
        const float* gg = dec + tt * dstr;
        const float* kk = kn + tt * dk;
        const float* qq = qn + tt * dk;
        float sk = 0.f;
        for (int i = 0; i < dk; ++i) {
          const float sv = S[i * dvb + tid] * gg[ch ? i : 0];
          S[i * dvb + tid] = sv;
          sk = fmaf(sv, kk[i], sk);
        }
        const float u = beta[tt] * (conv[(long long)(t0 + b0 + tt) * C + v_col + col0 + tid] - sk);
        float o = 0.f;
        for (int i = 0; i < dk; ++i) {
          const float sv = fmaf(kk[i], u, S[i * dvb + tid]);
          S[i * dvb + tid] = sv;
          o = fmaf(sv, qq[i], o);
        }
        if (o_raw != nullptr) o_raw[((long long)(t0 + b0 + tt) * H + h) * dv + col0 + tid] = o;
        else ob[tt * dvb + tid] = o;
      }
    }
    __syncthreads();
    for (int tt = warp; o_raw == nullptr && tt < nt; tt += nw) {
      float ss = 0.f;
      for (int j = lane; j < dv; j += 32) ss += ob[tt * dv + j] * ob[tt * dv + j];
      ss = warp_sum(ss);
      const float rstd = 1.f / sqrtf(ss / (float)dv + eps);
      const long long t = t0 + b0 + tt;
      for (int j = lane; j < dv; j += 32) {
        const float gz = gproj[t * ldg + h * dv + j];
        st_dt(out, dt_out, (t * H + h) * dv + j, ob[tt * dv + j] * rstd * norm_w[j] * gate_value(gz, gate_act));
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < dk * nc; i += blockDim.x) Sg[(long long)(i / nc) * dv + i % nc] = S[(i / nc) * dvb + i % nc];
}


// ---- the same recurrence for key sizes 32 / 64 / 128 and value sizes that are multiples of 32: state in registers.
// delta_prep: unit-norm q (times dk^-1/2) and k per (token, key head), write strength and decay per (token, head), all tokens in
// parallel.  delta_rule_reg: one block per (sequence, head, 32 value columns); lane = column, warp p holds rows [p DK/8, (p+1) DK/8) of
// the state in registers, so the k and q values a warp needs are the same for all its lanes (one shared-memory transaction per 16
// bytes); the pieces of S^T k meet through shared memory and one block barrier per token, those of S^T q once per 8 tokens; q / k / v /
// gates of the next 8 tokens stream into shared memory with cp.async while the current 8 are processed.  delta_out: per-head RMS norm and SiLU gate.
__global__ void __launch_bounds__(256) delta_prep_kernel(const float* __restrict__ conv, int C, const float* __restrict__ bproj,
                                                         long long ldb, const float* __restrict__ aproj, long long lda, int ch, int H,
                                                         int Hk, int dk, const float* __restrict__ A_log,
                                                         const float* __restrict__ dt_bias, long long T, float* __restrict__ qn,
                                                         float* __restrict__ kn, float* __restrict__ beta, float* __restrict__ dec) {
  kb2::pdl_enter(conv, bproj, aproj, A_log, dt_bias, qn, kn, beta, dec);
  const long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= T * Hk) return;
  const long long t = w / Hk;
  const int hk = (int)(w - t * Hk);
  const float* row = conv + t * C;
  const int q_col = hk * dk, k_col = Hk * dk + hk * dk;
  float sq = 0.f, sk = 0.f;
  for (int i = lane; i < dk; i += 32) {
    const float qv = row[q_col + i], kv = row[k_col + i];
    sq += qv * qv;
    sk += kv * kv;
  }
  sq = warp_sum(sq);
  sk = warp_sum(sk);
  const float rq = (1.f / sqrtf((float)dk)) / sqrtf(sq + 1e-6f), rk = 1.f / sqrtf(sk + 1e-6f);
  for (int i = lane; i < dk; i += 32) {
    qn[w * dk + i] = row[q_col + i] * rq;
    kn[w * dk + i] = row[k_col + i] * rk;
  }
  const int rep = H / Hk;
  for (int j = lane; j < rep; j += 32) {
    const int h = hk * rep + j;
    beta[t * H + h] = 1.f / (1.f + expf(-bproj[t * ldb + h]));
    if (!ch) dec[t * H + h] = decay_of(A_log[h], aproj[t * lda + h], dt_bias[h]);
  }
  if (ch)                                    // one decay per key channel of each of this key head's heads: dec [T][H][dk]
    for (int j = 0; j < rep; ++j) {
      const int h = hk * rep + j;
      const double rate = exp((double)A_log[h]);
      for (int i = lane; i < dk; i += 32) {
        const long long c = (long long)h * dk + i;
        dec[t * H * dk + c] = decay_from_rate(rate, aproj[t * lda + c], dt_bias[c]);
      }
    }
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

constexpr int kRegTile = 8;
constexpr int kRegPieces = 8;                // warps of a block (the sum of the pieces below is written for 8): warp p holds rows [p DK/8, (p+1) DK/8) of 32 state columns
template <int DK, bool CH>
__global__ void __launch_bounds__(32 * kRegPieces) delta_rule_reg_kernel(const float* __restrict__ qn, const float* __restrict__ kn,
                                                                         const float* __restrict__ conv, int C, int v_col0,
                                                                         const float* __restrict__ beta, const float* __restrict__ dec,
                                                                         int H, int Hk, int dv, float* __restrict__ state,
                                                                         const int* __restrict__ cu, const int* __restrict__ slots,
                                                                         float* __restrict__ o_out) {
  kb2::pdl_enter(qn, kn, conv, beta, dec, state, cu, slots, o_out);
  constexpr int P = kRegPieces, NT = 32 * P;
  constexpr int Q = DK / P;                 // state rows per thread
  __shared__ __align__(16) float ks[2][kRegTile][DK];
  __shared__ __align__(16) float qs[2][kRegTile][DK];
  __shared__ __align__(16) float vs[2][kRegTile][32];
  __shared__ float bs[2][kRegTile], gs[2][kRegTile];
  __shared__ __align__(16) float gc[CH ? 2 : 1][CH ? kRegTile : 1][CH ? DK : 4];   // per-channel decays of the tile's tokens
  __shared__ float part[2][P][32];          // per token: the pieces of S^T k, summed by every warp after one barrier
  __shared__ float os_part[kRegTile][P][32];   // pieces of S^T q, summed once per tile
  const int s = blockIdx.x, h = blockIdx.y, j0 = blockIdx.z * 32;
  const int hk = h / (H / Hk);
  const int tid = threadIdx.x, lane = tid & 31, piece = tid >> 5;
  const int t0 = cu[s], n = cu[s + 1] - cu[s];
  float* Sg = state + ((long long)slots[s] * H + h) * DK * dv;
  float S[Q];
#pragma unroll
  for (int ii = 0; ii < Q; ++ii) S[ii] = Sg[(long long)(piece * Q + ii) * dv + j0 + lane];

  auto load_tile = [&](int buf, int b0) {
    const int nt = min(kRegTile, n - b0);
    for (int c = tid; c < nt * (DK / 4); c += NT) {                  // 16-byte chunks of the q and k rows
      const int tt = c / (DK / 4), cc = c - tt * (DK / 4);
      const long long src = ((long long)(t0 + b0 + tt) * Hk + hk) * DK + cc * 4;
      cp_async16(&ks[buf][tt][cc * 4], kn + src);
      cp_async16(&qs[buf][tt][cc * 4], qn + src);
      if (CH) cp_async16(&gc[CH ? buf : 0][CH ? tt : 0][cc * 4], dec + ((long long)(t0 + b0 + tt) * H + h) * DK + cc * 4);
    }
    for (int c = tid; c < nt * 8; c += NT) {
      const int tt = c >> 3, cc = c & 7;
      cp_async16(&vs[buf][tt][cc * 4], conv + (long long)(t0 + b0 + tt) * C + v_col0 + h * dv + j0 + cc * 4);
    }
    if (tid < nt) {
      cp_async4(&bs[buf][tid], beta + (long long)(t0 + b0 + tid) * H + h);
      if (!CH) cp_async4(&gs[buf][tid], dec + (long long)(t0 + b0 + tid) * H + h);
    }
    cp_async_commit();
  };

  load_tile(0, 0);
  int buf = 0;
  for (int b0 = 0; b0 < n; b0 += kRegTile, buf ^= 1) {
    const int nt = min(kRegTile, n - b0);
    cp_async_wait_all();
    __syncthreads();                                  // tile `buf` is in place; everyone is done with the other buffer and with os_part
    if (b0 + kRegTile < n) load_tile(buf ^ 1, b0 + kRegTile);
    for (int tt = 0; tt < nt; ++tt) {
      const float g = CH ? 1.f : gs[buf][tt], b = bs[buf][tt];
      // the same address for every lane: one shared-memory transaction per 16 bytes.  All of the token's k and q values are fetched
      // up front (the loads are in flight together, none has to wait behind the barrier below)
      const float4* k4 = reinterpret_cast<const float4*>(&ks[buf][tt][piece * Q]);
      const float4* q4 = reinterpret_cast<const float4*>(&qs[buf][tt][piece * Q]);
      float4 kr[Q / 4], qr[Q / 4];
#pragma unroll
      for (int ii = 0; ii < Q / 4; ++ii) kr[ii] = k4[ii];
#pragma unroll
      for (int ii = 0; ii < Q / 4; ++ii) qr[ii] = q4[ii];
      const float vv = vs[buf][tt][lane];
      float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
      if (CH) {                               // the rows of the state decay each by its own factor before anything reads them
        const float4* g4 = reinterpret_cast<const float4*>(&gc[CH ? buf : 0][CH ? tt : 0][piece * Q]);
#pragma unroll
        for (int ii = 0; ii < Q / 4; ++ii) {
          const float4 gr = g4[ii];
          S[4 * ii] *= gr.x;
          S[4 * ii + 1] *= gr.y;
          S[4 * ii + 2] *= gr.z;
          S[4 * ii + 3] *= gr.w;
        }
      }
#pragma unroll
      for (int ii = 0; ii < Q / 4; ++ii) {
        a0 = fmaf(S[4 * ii], kr[ii].x, a0);
        a1 = fmaf(S[4 * ii + 1], kr[ii].y, a1);
        a2 = fmaf(S[4 * ii + 2], kr[ii].z, a2);
        a3 = fmaf(S[4 * ii + 3], kr[ii].w, a3);
      }
      part[tt & 1][piece][lane] = (a0 + a1) + (a2 + a3);
      __syncthreads();
      float pp[P];
#pragma unroll
      for (int p = 0; p < P; ++p) pp[p] = part[tt & 1][p][lane];
      const float sk = ((pp[0] + pp[1]) + (pp[2] + pp[3])) + ((pp[4] + pp[5]) + (pp[6] + pp[7]));
      const float u = b * (vv - g * sk);
      a0 = a1 = a2 = a3 = 0.f;
#pragma unroll
      for (int ii = 0; ii < Q / 4; ++ii) {
        S[4 * ii] = fmaf(kr[ii].x, u, g * S[4 * ii]);
        S[4 * ii + 1] = fmaf(kr[ii].y, u, g * S[4 * ii + 1]);
        S[4 * ii + 2] = fmaf(kr[ii].z, u, g * S[4 * ii + 2]);
        S[4 * ii + 3] = fmaf(kr[ii].w, u, g * S[4 * ii + 3]);
        a0 = fmaf(S[4 * ii], qr[ii].x, a0);
        a1 = fmaf(S[4 * ii + 1], qr[ii].y, a1);
        a2 = fmaf(S[4 * ii + 2], qr[ii].z, a2);
        a3 = fmaf(S[4 * ii + 3], qr[ii].w, a3);
      }
      os_part[tt][piece][lane] = (a0 + a1) + (a2 + a3);
    }
    __syncthreads();
    for (int i = tid; i < nt * 32; i += NT) {
      const int tt = i >> 5, c = i & 31;
      float o = 0.f;
#pragma unroll
      for (int p = 0; p < P; ++p) o += os_part[tt][p][c];
      o_out[((long long)(t0 + b0 + tt) * H + h) * dv + j0 + c] = o;
    }
  }
#pragma unroll
  for (int ii = 0; ii < Q; ++ii) Sg[(long long)(piece * Q + ii) * dv + j0 + lane] = S[ii];
}

// ---- the recurrence with one decay per head, sixteen tokens at a time on the warp-level tensor instructions (long portions).
// With S0 the state ahead of a tile, G_i = g_0 .. g_i and D_ij = g_(j+1) .. g_i, the token-by-token rule is
//   u_i = beta_i (v_i - G_i S0^T k_i - sum_(j<i) D_ij (k_i . k_j) u_j),   o_i = G_i S0^T q_i + sum_(j<=i) D_ij (q_i . k_j) u_j,
//   S = G_15 S0 + sum_j D_15,j k_j u_j^T.
// The u_i solve (I + L) u = diag(beta) (V - diag(G) K S0) with L_ij = beta_i D_ij (k_i . k_j) below the diagonal, and T = (I + L)^-1 needs no
// state: delta_tile_prep makes V' = T diag(beta) V and W = T diag(beta G) K for all tiles at once, which leaves u = V' - W S0 for the chain of
// tiles (the WY form of a product of Householder-like factors: Bischof and Van Loan 1987; for this rule Yang et al. 2024, "Parallelizing Linear
// Transformers with the Delta Rule over Sequence Length").  No entry of T exceeds 1, since T_ij is made of products of the contractions
// I - beta k k^T.  Everything stays at fp32 grade: the operands of the products go in as three bf16 parts each (24 bits; six of nine products,
// the rest is below 2^-26), tensor sums run over 32 rows or 16 tokens and start from zero, and the state is updated by fp32 multiply-adds.
// A token's numbers never meet those of a later one, not even times zero: the sums of the prep stop at the diagonal, rows of a tensor product
// do not mix, and the read-out takes what is not finite out of its product and adds it to the later tokens by hand.
//
// A block has 32 value columns of a (sequence, head) as two groups of 16 columns.  A group has DK / 32 warps with 32 rows of the state each, as
// accumulator fragments that are the operand fragments of the next tile's product as they stand, and a warp for the read-outs, which are off the
// chain.  k, q and W arrive as ready images (bulk copies by a warp of their own, three tiles ahead) and enter through ldmatrix, plain for S0^T w
// and transposed for k u^T; the partial sums of a group's warps meet in shared memory in fragment order, so nothing is moved between lanes.
// The largest of the six products of an update and of a read-out goes eight tokens at a time, each to a sum of its own: the tensor cores cut off
// what they add, and with sixteen at a time states were 1 % further off (6.6e-7 instead of 6.5e-7).
// Bound: 1270 cycles of the tensor pipe and 1370 of shared memory per tile, of 2210 (counters at 2048 tokens; 4096 tokens, 32 / 16 heads x 128: 310 us, the prep 98); left
// is the chain split - W - exchange - u - update.  The next tile is waited for and its W fetched between the instructions of the update and the use of their sums,
// and the read-out's buffer at its first store: with all three at the head of a tile 338 us (q fetched ahead of W's sums as well: 364).
// With eight tokens per tile, where each warp solved for u itself, the phases were shorter and as dependent, and the whole took 642 + 56 us.
constexpr int kDT = 16, kDTStages = 4;
// what couples the tokens of a (tile, head): G[16] | D_15,j [16] | G_15 and padding to 48 floats | D_ij q_i . k_j as three bf16 parts [i][24]
constexpr int kDTG = 0, kDTEnd = 16, kDTAll = 32, kDTQK = 48, kDTQKPitch = 24, kDTQKPart = kDT * kDTQKPitch;
constexpr int kDTScalars = kDTQK + 3 * kDTQKPart / 2;      // floats
template <int NI> struct DeltaTile {
  static constexpr int DK = 32 * NI, kPitch = DK + 8;      // bf16 row pitch: 16 bytes more, so that the eight rows of an ldmatrix do not collide
  static constexpr int kWPart = kDT * kPitch, kPart = 2 * kWPart;      // bf16 of one part: of W; of k rows, then q rows
  static constexpr int kImage = 3 * kPart, kWImage = 3 * kWPart;       // bf16 of a (tile, key head) and of a (tile, head): hi, mid, lo
  static constexpr int kImageBytes = kImage * 2, kWBytes = kWImage * 2, kScalarBytes = kDTScalars * 4, kVBytes = kDT * 32 * 4;
  static constexpr int kStageBytes = kImageBytes + kWBytes + kVBytes + kScalarBytes;
  static constexpr int kRedFloats = 2 * 2 * NI * 4 * 128;  // [buffer][column group][row piece][W tokens 0..7, 8..15, q 0..7, 8..15][lane][4]
  static constexpr int kUFloats = 2 * 2 * 256;             // [buffer][column group][lane][8]
  static constexpr int kSmem = kDTStages * kStageBytes + (kRedFloats + kUFloats) * 4 + (2 * kDTStages + 12) * 8;
  static constexpr int kThreads = 64 * NI + 96;
  // image, then v of a pair's second head | k | q, then v of the first head | k.k and q.k in two halves | per head of a pair L, T beta G, T beta | gates
  static constexpr int prep_image(int vb) { return kImageBytes > kDT * 32 * vb * 4 ? kImageBytes : kDT * 32 * vb * 4; }
  static constexpr int prep_rows(int vb) { return kDT * DK + kDT * (DK > 32 * vb ? DK : 32 * vb); }
  static constexpr int prep_smem(int vb, int rep) { return prep_image(vb) + (prep_rows(vb) + 10 * kDT * 20 + 2 * kDT * rep) * 4; }
  static_assert(kImageBytes % 16 == 0 && kWBytes % 16 == 0 && kScalarBytes % 16 == 0 && kStageBytes % 16 == 0, "bulk copies");
  static_assert(kSmem <= 227 * 1024, "shared memory");
};

// fp32 pair -> three words of bf16 pairs whose sums they are, exact to 24 bits (the largest finite numbers too: their first part stops at the
// largest bf16 number instead of rounding to infinity; an infinity becomes NaN, as in the recurrence it does one token later)
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&p)[3]) {
  asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(p[0]) : "f"(y), "f"(x));
  const float rx = x - __uint_as_float(p[0] << 16), ry = y - __uint_as_float(p[0] & 0xFFFF0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p[1]) : "f"(ry), "f"(rx));
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p[2]) : "f"(ry - __uint_as_float(p[1] & 0xFFFF0000u)), "f"(rx - __uint_as_float(p[1] << 16)));
}
// eight tokens of the sixteen
__device__ __forceinline__ void mma1688_new(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0), "f"(0.f));
}
template <bool kTrans> __device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const void* row) {
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(row);
  if constexpr (kTrans)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
// The six products of two numbers in three parts that are worth having: the parts that go into product m (the largest, m = 0, has a sum of its own).
__device__ __forceinline__ constexpr int part_a(int m) { return 0x120100 >> (4 * m) & 15; }
__device__ __forceinline__ constexpr int part_b(int m) { return 0x102010 >> (4 * m) & 15; }

struct DeltaPrep {
  const float* conv;               // [T][C]: q | k | v
  long long C, ldp;
  const float *bproj, *aproj, *A_log, *dt_bias;
  int H, Hk, dv, S;
  const int* cu;
  long long f0, f1;                // the slice of the step's tiles that is worked on: images lie from tile f0 on
  bool whole;                      // the slice is all of them
  bf16 *image, *wimage;
  float *vimage, *sc;
};

// The tile's rows t0 .. t0 + nt - 1 of kWidth neighbouring channels from c on, to shared memory [16][kWidth], zeros behind the last one.
template <int kWidth>
__device__ __forceinline__ void delta_fetch(const DeltaPrep& p, int t0, int nt, int c, float* to) {
  for (int i = threadIdx.x; i < kDT * kWidth / 4; i += 256) {
    const int t = i / (kWidth / 4), e = i % (kWidth / 4) * 4;
    if (t < nt) kb2::cp_async16(to + t * kWidth + e, p.conv + (long long)(t0 + t) * p.C + c + e);
    else *reinterpret_cast<float4*>(to + t * kWidth + e) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// A block of eight warps per (tile, key head).  Mostly traffic: at 4096 tokens, 32 / 16 heads x 128, 134 MB of k, q and v come
// in and 304 MB go out in 98 us, 0.68 of the copy rate; the rest is the chain of a tile's products, half of whose phases keep two or four of the warps busy.
// Four blocks share an SM since the values lie where q and the image were (three: 111 us).  All loops are rolled as far as registers allow: with everything unrolled and a warp for each part the block took 35 KB of
// instructions once, and waiting for them was most of its time.
// image [tiles][Hk] | W [tiles][H] | V' [tiles][H][dv / 16][lane][8], in the order in which a lane of delta_tile_kernel takes them | scalars [tiles][H]
template <int NI, int VB>
__global__ void __launch_bounds__(256, 4) delta_tile_prep_kernel(const DeltaPrep p) {
  kb2::pdl_wait();
  using D = DeltaTile<NI>;
  constexpr int DK = D::DK, kCols = 32 * VB;          // value columns of a pass
  extern __shared__ __align__(128) uint8_t tsm[];
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = tid & 31;
  const long long flat = blockIdx.x / p.Hk;
  const int hk = (int)(blockIdx.x - flat * p.Hk), H = p.H, rep = H / p.Hk;
  long long tile = p.f0 + flat;
  int sq = 0, t0 = 0, n = 0;                          // the tile's sequence: tiles are counted sequence by sequence
  for (; sq < p.S; ++sq) {
    t0 = p.cu[sq];
    n = p.cu[sq + 1] - t0;
    const int nt = (n + kDT - 1) / kDT;
    if (tile < nt) break;
    tile -= nt;
  }
  if (sq == p.S) return;
  t0 += (int)tile * kDT;
  const int nt = min(kDT, n - (int)tile * kDT);
  bf16* img = reinterpret_cast<bf16*>(tsm);
  float* rows = reinterpret_cast<float*>(tsm + D::prep_image(VB));     // k [16][DK] | q [16][DK]
  float* const vrow[2] = {rows + kDT * DK, reinterpret_cast<float*>(tsm)};      // of a pair's heads [16][kCols], where q and the image were
  float* pairs = rows + D::prep_rows(VB);             // [k.k, q.k][half of the sum][16][20]
  float* Lb = pairs + 4 * kDT * 20;                   // [head of the pair][16][20], as T beta G and T beta
  float* Tw = Lb + 2 * kDT * 20;
  float* Tv = Tw + 2 * kDT * 20;
  float* gates = Tv + 2 * kDT * 20;                   // [decay, strength][head of the key head][16]

  delta_fetch<DK>(p, t0, nt, p.Hk * DK + hk * DK, rows);
  delta_fetch<DK>(p, t0, nt, hk * DK, rows + kDT * DK);
  kb2::cp_async_commit();
  auto fetch_values = [&](int hh, int r0, int j0) {
    if (r0 + hh < rep) delta_fetch<kCols>(p, t0, nt, 2 * p.Hk * DK + (hk * rep + r0 + hh) * p.dv + j0, vrow[hh]);
    kb2::cp_async_commit();
  };
  // decays and write strengths of the block's heads, under the wait for the rows (fp64 exponentials: a few hundred dependent instructions)
  for (int i = tid; i < 2 * rep * kDT; i += 256) {
    const int which = i / (rep * kDT), h = hk * rep + i % (rep * kDT) / kDT, t = i % kDT;
    const long long row = (long long)(t0 + t) * p.ldp + h;
    gates[i] = t >= nt ? (which ? 0.f : 1.f) : which ? 1.f / (1.f + expf(-p.bproj[row])) : decay_of(p.A_log[h], p.aproj[row], p.dt_bias[h]);
  }
  kb2::cp_async_wait<0>();
  __syncthreads();

  auto store = [&](bf16* to, int part, const float (&v)[NI]) {       // the three parts of a row, `part` numbers apart
    if constexpr (NI == 1) {
      const float other = __shfl_down_sync(0xffffffffu, v[0], 1);
      uint32_t q[3];
      split_pair(v[0], other, q);
      if (!(lane & 1))
#pragma unroll
        for (int c = 0; c < 3; ++c) *reinterpret_cast<uint32_t*>(to + c * part + lane) = q[c];
    } else {
      uint32_t q[NI / 2][3];
#pragma unroll
      for (int i = 0; i < NI; i += 2) split_pair(v[i], v[i + 1], q[i / 2]);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if constexpr (NI == 4) *reinterpret_cast<uint2*>(to + c * part + lane * 4) = make_uint2(q[0][c], q[1][c]);
        else *reinterpret_cast<uint32_t*>(to + c * part + lane * 2) = q[0][c];
      }
    }
  };
  auto take = [&](const float* from, auto& v) {       // a lane's neighbouring numbers of a row
    constexpr int N = sizeof(v) / sizeof(float);
    if constexpr (N == 4) {
      const float4 f = *reinterpret_cast<const float4*>(from + lane * 4);
      v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = from[lane * N + i];
    }
  };
#pragma unroll
  for (int r = 0; r < 4; ++r) {                       // unit rows: 16 of k, then 16 of q
    const int t = warp * 4 + r;
    float v[NI], a = 0.f;
    take(rows + t * DK, v);
#pragma unroll
    for (int i = 0; i < NI; ++i) a += v[i] * v[i];
    a = warp_sum(a);
    const float s = warp < 4 ? 1.f / sqrtf(a + 1e-6f) : (1.f / sqrtf((float)DK)) / sqrtf(a + 1e-6f);
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      v[i] *= s;
      rows[t * DK + lane * NI + i] = v[i];
    }
    store(img + t * D::kPitch, D::kPart, v);
  }
  kb2::fence_proxy_async_smem();
  __syncthreads();
  if (tid == 128) {
    kb2::bulk_s2g(p.image + (flat * p.Hk + hk) * D::kImage, img, D::kImageBytes);
    kb2::bulk_commit_group();
  }
  fetch_values(0, 0, 0);
  if (tid == 128) kb2::bulk_wait_group_read0();       // the image has left shared memory
  if (warp < 4) {                                     // k_i . k_j (warps 0, 1: halves of the sum) and q_i . k_j (2, 3)
    float s[2][4] = {};
    const bf16* row = img + ((lane >> 4) * 8 + (lane & 7)) * D::kPitch + ((lane >> 3) & 1) * 8;
    const int mine = warp < 2 ? 0 : D::kWPart;
#pragma unroll 1
    for (int k0 = (warp & 1) * 32; k0 < DK; k0 += 64) {
      float big[2][2][4], small[2][4];                // [16 numbers][columns 0..7, 8..15]
#pragma unroll
      for (int kb = 0; kb < 2; ++kb) {
        uint32_t x[3][4], y[3][4];                    // tokens 0..7: numbers 0..7, 8..15; tokens 8..15 the same
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          ldmatrix4<false>(x[c], row + c * D::kPart + k0 + kb * 16);
          ldmatrix4<false>(y[c], row + c * D::kPart + mine + k0 + kb * 16);
        }
#pragma unroll
        for (int m = 0; m < 6; ++m)
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            float(&d)[4] = m ? small[b] : big[kb][b];
            const uint32_t(&ya)[4] = y[part_a(m)];
            const uint32_t(&xb)[4] = x[part_b(m)];
            if (m == 0 || (kb == 0 && m == 1)) mma16816_new(d, ya[0], ya[2], ya[1], ya[3], xb[2 * b], xb[2 * b + 1]);
            else mma16816(d, ya[0], ya[2], ya[1], ya[3], xb[2 * b], xb[2 * b + 1]);
          }
      }
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[b][e] += (big[0][b][e] + big[1][b][e]) + small[b][e];
    }
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        *reinterpret_cast<float2*>(pairs + warp * kDT * 20 + ((lane >> 2) + e * 8) * 20 + b * 8 + (lane & 3) * 2) = make_float2(s[b][2 * e], s[b][2 * e + 1]);
  }
  __syncthreads();
  fetch_values(1, 0, 0);
#pragma unroll 1
  for (int r0 = 0; r0 < rep; r0 += 2) {
    if (warp < 2) {                                   // a lane per (head of the pair, token): what couples the tokens
      const int me = lane & 15, half = lane >> 4, h = hk * rep + r0 + half;
      const bool head = r0 + half < rep, in = me < nt;
      float gs[kDT], up = 1.f, d = 1.f, row[kDT];     // d: D_me,j for the j at hand, from j = 15 down
#pragma unroll
      for (int t = 0; t < kDT; ++t) gs[t] = head ? gates[(r0 + half) * kDT + t] : 1.f;      // 1 behind the last token
#pragma unroll
      for (int t = 0; t < kDT; ++t)
        if (t <= me) up *= gs[t];
      const float* mine = pairs + (warp ? 0 : 2 * kDT * 20) + me * 20;
#pragma unroll
      for (int j4 = kDT - 4; j4 >= 0; j4 -= 4) {
        const float4 a = *reinterpret_cast<const float4*>(mine + j4), b = *reinterpret_cast<const float4*>(mine + kDT * 20 + j4);
        const float av[4] = {a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w};
#pragma unroll
        for (int e = 3; e >= 0; --e) {
          const int j = j4 + e;
          row[j] = j < me + !warp ? d * av[e] : 0.f;  // below the diagonal; q . k with it
          if (j <= me) d *= gs[j];
        }
      }
      if (warp == 0) {                                // what the chain and the read-out take as numbers; tokens behind the last one take no part
        float down = 1.f, all = 1.f;
#pragma unroll
        for (int t = 0; t < kDT; ++t) {
          all *= gs[t];
          if (t > me) down *= gs[t];
        }
        if (head) {
          float* o = p.sc + (flat * H + h) * kDTScalars;
          o[kDTG + me] = in ? up : 0.f;
          o[kDTEnd + me] = in ? down : 0.f;
          o[kDTAll + me] = me == 0 ? all : 0.f;
          uint32_t q[kDT / 2][3];
#pragma unroll
          for (int j = 0; j < kDT; j += 2) split_pair(in ? row[j] : 0.f, in ? row[j + 1] : 0.f, q[j / 2]);
          bf16* parts = reinterpret_cast<bf16*>(o + kDTQK) + me * kDTQKPitch;
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int j = 0; j < 2; ++j)
              *reinterpret_cast<uint4*>(parts + c * kDTQKPart + j * 8) = make_uint4(q[4 * j][c], q[4 * j + 1][c], q[4 * j + 2][c], q[4 * j + 3][c]);
        }
      } else {
        const float beta = head ? gates[(rep + r0 + half) * kDT + me] : 0.f;
        float* L = Lb + half * kDT * 20;
#pragma unroll
        for (int j = 0; j < kDT; j += 4)
          *reinterpret_cast<float4*>(L + me * 20 + j) = make_float4(beta * row[j], beta * row[j + 1], beta * row[j + 2], beta * row[j + 3]);
        __syncwarp();
        float x[kDT];                                 // column `me` of T
#pragma unroll
        for (int i = 0; i < kDT; ++i) {
          float a = i == me ? 1.f : 0.f;
#pragma unroll
          for (int j4 = 0; j4 < i; j4 += 4) {
            const float4 l = *reinterpret_cast<const float4*>(L + i * 20 + j4);
            const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (j4 + e < i) a = fmaf(-lv[e], x[j4 + e], a);
          }
          x[i] = a;
        }
#pragma unroll
        for (int i = 0; i < kDT; ++i) {
          Tv[half * kDT * 20 + i * 20 + me] = x[i] * beta;
          Tw[half * kDT * 20 + i * 20 + me] = x[i] * beta * up;
        }
      }
    }
    const int hh = (warp >> 1) & 1, hv = hk * rep + r0 + hh, b0 = warp & 1;      // two warps per product with T: rows 0..3, 8..11 and 4..7, 12..15
    const bool there = r0 + hh < rep;
#pragma unroll 1
    for (int j0 = 0; j0 < p.dv; j0 += kCols) {
      kb2::cp_async_wait<0>();
      __syncthreads();
      // four rows of a product with T: no column behind a row's own
      auto four = [&](const float* T, const float* x, int width, int ib, auto& acc) {
        constexpr int N = sizeof(acc[0]) / sizeof(float);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int m = 0; m < N; ++m) acc[i][m] = 0.f;
        auto block = [&](int jb, bool whole) {
          float xr[4][N];
#pragma unroll
          for (int j = 0; j < 4; ++j) take(x + (jb * 4 + j) * width, xr[j]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 c = *reinterpret_cast<const float4*>(T + (ib * 4 + i) * 20 + jb * 4);
            const float cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (whole || j <= i)
#pragma unroll
                for (int m = 0; m < N; ++m) acc[i][m] = fmaf(cv[j], xr[j][m], acc[i][m]);
          }
        };
#pragma unroll 1
        for (int jb = 0; jb < ib; ++jb) block(jb, true);
        block(ib, false);
      };
      if (warp < 4) {
        if (j0 == 0 && there) {
          bf16* wi = p.wimage + (flat * H + hv) * D::kWImage;
#pragma unroll 1
          for (int ib = b0; ib < 4; ib += 2) {
            float a[4][NI];
            four(Tw + hh * kDT * 20, rows, DK, ib, a);
#pragma unroll
            for (int i = 0; i < 4; ++i) store(wi + (ib * 4 + i) * D::kPitch, D::kWPart, a[i]);
          }
        }
      } else if (there) {
        float a[4][VB], c[4][VB];
        const float* T = Tv + hh * kDT * 20;
        const float* x = vrow[hh];
        four(T, x, kCols, b0, a);
        four(T, x, kCols, b0 + 2, c);
        float* vi = p.vimage + (flat * H + hv) * kDT * p.dv;
#pragma unroll
        for (int m = 0; m < VB; ++m) {
          const int col = j0 + lane * VB + m;
#pragma unroll
          for (int i = 0; i < 4; i += 2)
            *reinterpret_cast<float4*>(vi + (col >> 4) * 256 + (col & 7) * 32 + (b0 * 2 + i / 2) * 8 + ((col >> 3) & 1) * 4) =
                make_float4(a[i][m], a[i + 1][m], c[i][m], c[i + 1][m]);
        }
      }
      if (j0 + kCols < p.dv || r0 + 2 < rep) {
        __syncthreads();
        const bool more = j0 + kCols < p.dv;
        for (int v = 0; v < 2; ++v) fetch_values(v, more ? r0 : r0 + 2, more ? j0 + kCols : 0);
      }
    }
  }
  if (tid == 128) kb2::bulk_wait_group0();
}

template <int NI>
__global__ void __launch_bounds__(DeltaTile<NI>::kThreads, 1)
    delta_tile_kernel(const bf16* __restrict__ image, const bf16* __restrict__ wimage, const float* __restrict__ vimage, const float* __restrict__ sc,
                      int H, int Hk, int dv, float* __restrict__ state, const int* __restrict__ cu, const int* __restrict__ slots,
                      float* __restrict__ o_out, long long f0, long long f1, bool whole) {
  kb2::pdl_enter(image, wimage, vimage, sc, state, cu, slots, o_out);
  using D = DeltaTile<NI>;
  extern __shared__ __align__(128) uint8_t tsm[];
  float* red = reinterpret_cast<float*>(tsm + kDTStages * D::kStageBytes);
  float* ubuf = red + D::kRedFloats;
  uint64_t* full = reinterpret_cast<uint64_t*>(ubuf + D::kUFloats);
  uint64_t* empty = full + kDTStages;
  uint64_t* w_there = empty + kDTStages;           // [buffer][column group]: all pieces of W S0
  uint64_t* o_there = w_there + 4;                 // all pieces of q S0, and u
  uint64_t* o_free = o_there + 4;                  // the read-out has taken them
  const int s = blockIdx.x, h = blockIdx.y, j0 = blockIdx.z * 32, hk = h / (H / Hk);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int n_all = cu[s + 1] - cu[s];
  long long first = 0;                             // the sequence's tiles come after those of the sequences before it
  if (!whole || warp == 2 * NI + 2)
    for (int i = 0; i < s; ++i) first += (cu[i + 1] - cu[i] + kDT - 1) / kDT;
  int skip = 0, tiles = (n_all + kDT - 1) / kDT;   // tiles of the sequence ahead of the slice, and in it
  if (!whole) {
    const long long all = first + tiles;
    skip = (int)(min(max(f0, first), all) - first);
    tiles = (int)(min(max(f1, first), all) - first) - skip;
  }
  if (tiles == 0) return;
  const int t0 = cu[s] + skip * kDT, n = n_all - skip * kDT;      // tokens from the slice on
  if (threadIdx.x == 0) {
    for (int i = 0; i < kDTStages; ++i) {
      kb2::mbar_init(&full[i], 1);
      kb2::mbar_init(&empty[i], 2 * NI + 2);
    }
    for (int i = 0; i < 4; ++i) {
      kb2::mbar_init(&w_there[i], NI);
      kb2::mbar_init(&o_there[i], NI);
      kb2::mbar_init(&o_free[i], 1);
    }
    kb2::fence_mbar_init();
  }
  __syncthreads();
  const int quad = lane >> 2, pair = (lane & 3) * 2;      // fragment: columns quad, quad + 8; rows or tokens pair, pair + 1
  if (warp == 2 * NI + 2) {                        // ---- the tiles' way into shared memory
    for (int i = 0; i < tiles; ++i) {
      const int st = i % kDTStages;
      uint8_t* b = tsm + st * D::kStageBytes;
      kb2::mbar_wait(&empty[st], (uint32_t)(i / kDTStages & 1) ^ 1u);
      if (lane == 0) kb2::mbar_arrive_expect_tx(&full[st], (uint32_t)D::kStageBytes);
      __syncwarp();
      const long long flat = first + skip + i - f0;
      if (lane == 0) kb2::bulk_g2s(b, image + (flat * Hk + hk) * D::kImage, D::kImageBytes, &full[st]);
      else if (lane == 1) kb2::bulk_g2s(b + D::kImageBytes, wimage + (flat * H + h) * D::kWImage, D::kWBytes, &full[st]);
      else if (lane == 2) kb2::bulk_g2s(b + D::kImageBytes + D::kWBytes, vimage + (flat * H + h) * kDT * dv + j0 * kDT, D::kVBytes, &full[st]);
      else if (lane == 3) kb2::bulk_g2s(b + D::kImageBytes + D::kWBytes + D::kVBytes, sc + (flat * H + h) * kDTScalars, D::kScalarBytes, &full[st]);
    }
    return;
  }
  auto one = [](float (&d)[4], bool first, const uint32_t (&a)[3][4], const uint32_t (&b)[3][4], int at, int m) {      // product m of the six
    const int p = part_a(m), r = part_b(m);
    if (first) mma16816_new(d, a[p][0], a[p][1], a[p][2], a[p][3], b[r][at], b[r][at + 1]);
    else mma16816(d, a[p][0], a[p][1], a[p][2], a[p][3], b[r][at], b[r][at + 1]);
  };
  if (warp >= 2 * NI) {                            // ---- the read-outs of a column group
    const int cg = warp - 2 * NI;
    for (int i = 0; i < tiles; ++i) {
      const int st = i % kDTStages, buf = (i & 1) * 2 + cg;
      const float* ss = reinterpret_cast<const float*>(tsm + st * D::kStageBytes + D::kImageBytes + D::kWBytes + D::kVBytes);
      const bf16* qk = reinterpret_cast<const bf16*>(ss + kDTQK);
      kb2::mbar_wait(&full[st], (uint32_t)(i / kDTStages & 1));
      uint32_t b[3][4];                            // tokens 0..7 by j 0..7, j 8..15; tokens 8..15 the same
#pragma unroll
      for (int c = 0; c < 3; ++c)
        ldmatrix4<false>(b[c], qk + c * kDTQKPart + ((lane >> 4) * 8 + (lane & 7)) * kDTQKPitch + ((lane >> 3) & 1) * 8);
      kb2::mbar_wait(&o_there[buf], (uint32_t)(i >> 1) & 1u);
      float u[8], qs[8] = {};
      {
        const float4 x = *reinterpret_cast<const float4*>(ubuf + buf * 256 + lane * 8), y = *reinterpret_cast<const float4*>(ubuf + buf * 256 + lane * 8 + 4);
        u[0] = x.x; u[1] = x.y; u[2] = x.z; u[3] = x.w; u[4] = y.x; u[5] = y.y; u[6] = y.z; u[7] = y.w;
      }
#pragma unroll
      for (int pc = 0; pc < NI; ++pc)
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
          const float4 x = *reinterpret_cast<const float4*>(red + ((buf * NI + pc) * 4 + 2 + nb) * 128 + lane * 4);
          qs[nb * 4] += x.x; qs[nb * 4 + 1] += x.y; qs[nb * 4 + 2] += x.z; qs[nb * 4 + 3] += x.w;
        }
      bool odd = false;
      uint32_t a[3][4];
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        const bool f0 = isfinite(u[e]), f1 = isfinite(u[e + 1]);
        odd |= !f0 | !f1;
        uint32_t p[3];
        split_pair(f0 ? u[e] : 0.f, f1 ? u[e + 1] : 0.f, p);
#pragma unroll
        for (int c = 0; c < 3; ++c) a[c][e / 2] = p[c];
      }
      float big[2][2][4], small[2][4];
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
        mma1688_new(big[0][nb], a[0][0], a[0][1], b[0][2 * nb]);
        mma1688_new(big[1][nb], a[0][2], a[0][3], b[0][2 * nb + 1]);
      }
#pragma unroll
      for (int m = 1; m < 6; ++m)
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) one(small[nb], m < 2, a, b, 2 * nb, m);
      float o[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int t = (e >> 2) * 8 + pair + (e & 1);
        o[e] = fmaf(ss[kDTG + t], qs[e], (big[0][e >> 2][e & 3] + big[1][e >> 2][e & 3]) + small[e >> 2][e & 3]);
      }
      if (__any_sync(0xffffffffu, odd)) {          // what is not finite joins its own and later tokens
#pragma unroll 1
        for (int j = 0; j < kDT; ++j) {
          const float* from = ubuf + buf * 256 + (quad * 4 + ((j & 7) >> 1)) * 8 + (j >> 3) * 4 + (j & 1);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int t = (e >> 2) * 8 + pair + (e & 1);
            const float uj = from[((e >> 1) & 1) * 2];
            const bf16* c = qk + t * kDTQKPitch + j;
            if (j <= t && !isfinite(uj)) o[e] += uj * (__bfloat162float(c[0]) + (__bfloat162float(c[kDTQKPart]) + __bfloat162float(c[2 * kDTQKPart])));
          }
        }
      }
      __syncwarp();
      if (lane == 0) {
        kb2::mbar_arrive(&o_free[buf]);
        kb2::mbar_arrive(&empty[st]);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int t = (e >> 2) * 8 + pair + (e & 1);
        if (i * kDT + t < n) o_out[((t0 + (long long)i * kDT + t) * H + h) * dv + j0 + cg * 16 + quad + ((e >> 1) & 1) * 8] = o[e];
      }
    }
    return;
  }
  const int cg = warp / NI, piece = warp % NI;     // ---- the chain
  float* Sg = state + ((long long)slots[s] * H + h) * D::DK * dv + (long long)piece * 32 * dv + j0 + cg * 16;
  float S[4][4];                                   // [eight rows][column quad: 2 rows, column quad + 8: 2 rows]
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int e = 0; e < 4; ++e) S[r][e] = Sg[(long long)(r * 8 + pair + (e & 1)) * dv + quad + (e >> 1) * 8];
  // ldmatrix rows: tokens along the lanes' eights, plain and transposed
  const int plain = ((lane >> 4) * 8 + (lane & 7)) * D::kPitch + piece * 32 + ((lane >> 3) & 1) * 8;
  const int turned = (((lane >> 3) & 1) * 8 + (lane & 7)) * D::kPitch + piece * 32 + (lane >> 4) * 8;
  // operand fragments of 16 tokens: [16 rows][part]
  auto fetch = [&](const bf16* rows, int part, uint32_t (&x)[2][3][4]) {
#pragma unroll
    for (int kb = 0; kb < 2; ++kb)
#pragma unroll
      for (int c = 0; c < 3; ++c) ldmatrix4<false>(x[kb][c], rows + c * part + plain + kb * 16);
  };
  uint32_t w[2][3][4];
  auto enter = [&](int i) {                        // tile i is there, and W as operand: looked for under the update of the tile before it
    kb2::mbar_wait(&full[i % kDTStages], (uint32_t)(i / kDTStages & 1));
    fetch(reinterpret_cast<const bf16*>(tsm + i % kDTStages * D::kStageBytes + D::kImageBytes), D::kWPart, w);
  };
  enter(0);
  for (int i = 0; i < tiles; ++i) {
    const int st = i % kDTStages, buf = (i & 1) * 2 + cg;
    const uint32_t turn = (uint32_t)(i >> 1) & 1u;
    const uint8_t* b = tsm + st * D::kStageBytes;
    const bf16* img = reinterpret_cast<const bf16*>(b);
    const float* vs = reinterpret_cast<const float*>(b + D::kImageBytes + D::kWBytes) + cg * 256 + lane * 8;
    const float* ss = reinterpret_cast<const float*>(b + D::kImageBytes + D::kWBytes + D::kVBytes);
    float* mine = red + (buf * NI + piece) * 512 + lane * 4;
    uint32_t sp[2][3][4];                          // S0^T as operand: [16 rows][part]
#pragma unroll
    for (int kb = 0; kb < 2; ++kb)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint32_t p[3];
        split_pair(S[2 * kb + (e >> 1)][(e & 1) * 2], S[2 * kb + (e >> 1)][(e & 1) * 2 + 1], p);
#pragma unroll
        for (int c = 0; c < 3; ++c) sp[kb][c][e] = p[c];
      }
    // S0^T [16 columns x 32 rows] times 16 tokens, in three sums of up to six instructions, each of which waits for the one before
    auto product = [&](const uint32_t (&x)[2][3][4], float (&sum)[3][2][4]) {
#pragma unroll
      for (int kb = 0; kb < 2; ++kb)
#pragma unroll
        for (int m = 0; m < 6; ++m)
#pragma unroll
          for (int nb = 0; nb < 2; ++nb) one(sum[m ? 1 + (m & 1) : 0][nb], kb == 0 && m < 3, sp[kb], x[kb], 2 * nb, m);
    };
    auto keep = [&](float* to, const float (&sum)[3][2][4]) {
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = sum[0][nb][e] + (sum[1][nb][e] + sum[2][nb][e]);
        *reinterpret_cast<float4*>(to + nb * 128) = make_float4(v[0], v[1], v[2], v[3]);
      }
    };
    uint32_t q[2][3][4];
    {
      float ws[3][2][4];
      product(w, ws);
      kb2::mbar_wait(&o_free[buf], turn ^ 1u);
      keep(mine, ws);
    }
    __syncwarp();
    if (lane == 0) kb2::mbar_arrive(&w_there[buf]);
    float qs[3][2][4];                             // q, under the wait for the other pieces; put away when there is time
    fetch(img + D::kWPart, D::kPart, q);
    product(q, qs);
    uint32_t kt[2][3][4];                          // k transposed: [16 rows][part]
#pragma unroll
    for (int rr = 0; rr < 2; ++rr)
#pragma unroll
      for (int c = 0; c < 3; ++c) ldmatrix4<true>(kt[rr][c], img + c * D::kPart + turned + rr * 16);
    float u[8];
    {
      const float4 x = *reinterpret_cast<const float4*>(vs), y = *reinterpret_cast<const float4*>(vs + 4);
      u[0] = x.x; u[1] = x.y; u[4] = x.z; u[5] = x.w; u[2] = y.x; u[3] = y.y; u[6] = y.z; u[7] = y.w;
    }
    const float2 e0 = *reinterpret_cast<const float2*>(ss + kDTEnd + pair), e1 = *reinterpret_cast<const float2*>(ss + kDTEnd + 8 + pair);
    const float total = ss[kDTAll];
    kb2::mbar_wait(&w_there[buf], turn);
    float ws[8] = {};
#pragma unroll
    for (int pc = 0; pc < NI; ++pc)
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
        const float4 x = *reinterpret_cast<const float4*>(red + (buf * NI + pc) * 512 + nb * 128 + lane * 4);
        ws[nb * 4] += x.x; ws[nb * 4 + 1] += x.y; ws[nb * 4 + 2] += x.z; ws[nb * 4 + 3] += x.w;
      }
#pragma unroll
    for (int e = 0; e < 8; ++e) u[e] -= ws[e];
    if (piece == 0) {
      *reinterpret_cast<float4*>(ubuf + buf * 256 + lane * 8) = make_float4(u[0], u[1], u[2], u[3]);
      *reinterpret_cast<float4*>(ubuf + buf * 256 + lane * 8 + 4) = make_float4(u[4], u[5], u[6], u[7]);
    }
    uint32_t up[3][4];                             // D_15,j u_j
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      uint32_t p[3];
      split_pair(u[e] * (e < 4 ? e0.x : e1.x), u[e + 1] * (e < 4 ? e0.y : e1.y), p);
#pragma unroll
      for (int c = 0; c < 3; ++c) up[c][e / 2] = p[c];
    }
    float big[2][4][4], small[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      mma1688_new(big[0][r], up[0][0], up[0][1], kt[r >> 1][0][(r & 1) * 2]);
      mma1688_new(big[1][r], up[0][2], up[0][3], kt[r >> 1][0][(r & 1) * 2 + 1]);
    }
#pragma unroll
    for (int m = 1; m < 6; ++m)
#pragma unroll
      for (int r = 0; r < 4; ++r) one(small[r], m < 2, up, kt[r >> 1], (r & 1) * 2, m);
    if (i + 1 < tiles) enter(i + 1);
    keep(mine + 256, qs);
    __syncwarp();
    if (lane == 0) {
      kb2::mbar_arrive(&o_there[buf]);
      kb2::mbar_arrive(&empty[st]);                // everything of the tile is in registers
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[r][e] = fmaf(S[r][e], total, (big[0][r][e] + big[1][r][e]) + small[r][e]);
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int e = 0; e < 4; ++e) Sg[(long long)(r * 8 + pair + (e & 1)) * dv + quad + (e >> 1) * 8] = S[r][e];
}

// delta_out for long steps with 128 value columns: a warp takes four (token, head) rows, whose loads are in flight together (4096 tokens x 32
// heads: 52 -> 44 us; a row per warp leaves too few bytes under way).
__global__ void __launch_bounds__(256) delta_out_rows_kernel(const float* __restrict__ o, const float* __restrict__ gproj, long long ldg, int gate_act, int H,
                                                             const float* __restrict__ norm_w, float eps, long long rows, void* __restrict__ out, int dt_out) {
  kb2::pdl_enter_global(o, gproj, norm_w, out);
  const long long w = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * 4;
  const int j = (threadIdx.x & 31) * 4;
  float4 f[4], g[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const long long r = min(w + i, rows - 1);
    f[i] = *reinterpret_cast<const float4*>(o + r * 128 + j);
    g[i] = *reinterpret_cast<const float4*>(gproj + r / H * ldg + r % H * 128 + j);
  }
  const float4 nw = *reinterpret_cast<const float4*>(norm_w + j);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float ss = warp_sum((f[i].x * f[i].x + f[i].y * f[i].y) + (f[i].z * f[i].z + f[i].w * f[i].w));
    const float rstd = 1.f / sqrtf(ss / 128.f + eps);
    auto finish = [&](float v, float gz, float n) { return v * rstd * n * gate_value(gz, gate_act); };
    const float4 r = make_float4(finish(f[i].x, g[i].x, nw.x), finish(f[i].y, g[i].y, nw.y), finish(f[i].z, g[i].z, nw.z), finish(f[i].w, g[i].w, nw.w));
    if (w + i >= rows) return;
    if (dt_out == 0) {
      *reinterpret_cast<float4*>((float*)out + (w + i) * 128 + j) = r;
    } else {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(r.x, r.y), hi = __floats2bfloat162_rn(r.z, r.w);
      *reinterpret_cast<uint2*>((bf16*)out + (w + i) * 128 + j) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  }
}

// out[t, h, :] = o / rms(o) * norm_w * silu(gate) (gate_act 1: sigmoid(gate)); a warp per (token, head).  V numbers per access: 4 where sizes
// and pointers allow (a row of 128 is then one 16-byte read per lane).
template <int V>
__global__ void __launch_bounds__(256) delta_out_kernel(const float* __restrict__ o, const float* __restrict__ gproj, long long ldg,
                                                        int gate_act, int H, int dv, const float* __restrict__ norm_w, float eps,
                                                        long long T, void* __restrict__ out, int dt_out) {
  kb2::pdl_enter(o, gproj, norm_w, out);
  const long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= T * H) return;
  const long long t = w / H;
  const int h = (int)(w - t * H);
  const float* row = o + w * dv;
  const float* gate = gproj + t * ldg + (long long)h * dv;
  auto finish = [&](float v, float gz, float nw, float rstd) { return v * rstd * nw * gate_value(gz, gate_act); };
  float ss = 0.f;
  if constexpr (V == 4) {
    for (int j = lane * 4; j < dv; j += 128) {
      const float4 f = *reinterpret_cast<const float4*>(row + j);
      ss += (f.x * f.x + f.y * f.y) + (f.z * f.z + f.w * f.w);
    }
    ss = warp_sum(ss);
    const float rstd = 1.f / sqrtf(ss / (float)dv + eps);
    for (int j = lane * 4; j < dv; j += 128) {
      const float4 f = *reinterpret_cast<const float4*>(row + j), g = *reinterpret_cast<const float4*>(gate + j), nw = *reinterpret_cast<const float4*>(norm_w + j);
      const float4 r = make_float4(finish(f.x, g.x, nw.x, rstd), finish(f.y, g.y, nw.y, rstd), finish(f.z, g.z, nw.z, rstd), finish(f.w, g.w, nw.w, rstd));
      if (dt_out == 0) {
        *reinterpret_cast<float4*>((float*)out + w * dv + j) = r;
      } else {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(r.x, r.y), hi = __floats2bfloat162_rn(r.z, r.w);
        *reinterpret_cast<uint2*>((bf16*)out + w * dv + j) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      }
    }
  } else {
    for (int j = lane; j < dv; j += 32) ss += row[j] * row[j];
    ss = warp_sum(ss);
    const float rstd = 1.f / sqrtf(ss / (float)dv + eps);
    for (int j = lane; j < dv; j += 32) st_dt(out, dt_out, w * dv + j, finish(row[j], gate[j], norm_w[j], rstd));
  }
}

// ---- a step in which every sequence has one token, 128 key and 128 value channels: convolution, its tail, unit rows, gates, the recurrence and the read-out in
// one launch.  Bound: latency (a block per (token, head) takes its state of 64 KB in and out, and six short phases follow one another); as five launches
// (conv_silu, conv_tail, delta_prep, delta_rule_reg, delta_out) most of the time was theirs: 4 tokens x 32 / 16 heads 18.2 -> 6.9 us.  All sums in the order of
// those, so that a token's numbers do not depend on what else is in its step.  A warp has a piece of 16 rows of the state, a lane four neighbouring columns.  The
// heads of a key head are a cluster: each convolves q and k for itself, and the first one moves their tail on when all have read it.
struct DeltaStep {
  const float* proj;               // [T][ldp]: q | k | v ahead of the convolution, gates from g_off, decay and strength inputs from a_off and b_off
  long long ldp;
  int g_off, a_off, b_off, H, Hk;
  const float *taps, *A_log, *dt_bias, *norm_w;
  float eps;
  float *tail, *state;             // [slots][channels][K - 1], [slots][H][128][128]
  const int* slots;                // of token t's sequence
  void* out;
  int dt_out;
};
template <int K>
__global__ void __launch_bounds__(256, 2) delta_step_kernel(const DeltaStep p) {
  kb2::pdl_wait();
  kb2::pdl_trigger();
  constexpr int D = 128, Q = D / kRegPieces;
  __shared__ __align__(16) float qk[2 * D], vs[D], part[kRegPieces][D], os[kRegPieces][D];
  __shared__ float gates[2];       // decay, strength
  const long long t = blockIdx.y;
  const int h = blockIdx.x, rep = p.H / p.Hk, hk = h / rep;
  const int tid = threadIdx.x, lane = tid & 31, piece = tid >> 5;
  const float* row = p.proj + t * p.ldp;
  const long long slot = p.slots[t], C = 2ll * p.Hk * D + (long long)p.H * D;
  // a channel of q or k per thread, and one of v for the first half
  const long long c_qk = tid < D ? hk * D + tid : p.Hk * D + hk * D + (tid - D), c_v = 2ll * p.Hk * D + (long long)h * D + (tid & (D - 1));
  float x[2][K], w[2][K];
  const auto fetch = [&](long long c, float (&x)[K], float (&w)[K]) {
    const float* tl = p.tail + (slot * C + c) * (K - 1);
#pragma unroll
    for (int j = 0; j < K - 1; ++j) x[j] = tl[j];
    x[K - 1] = row[c] + 0.f;
#pragma unroll
    for (int j = 0; j < K; ++j) w[j] = p.taps[c * K + j];
  };
  fetch(c_qk, x[0], w[0]);
  if (tid < D) fetch(c_v, x[1], w[1]);
  float4* Sg = reinterpret_cast<float4*>(p.state + ((slot * p.H + h) * D + piece * Q) * D) + lane;
  float4 S[Q], gz, nw;
#pragma unroll
  for (int i = 0; i < Q; ++i) S[i] = Sg[i * (D / 4)];
  if (piece == 0) {
    gz = *reinterpret_cast<const float4*>(row + p.g_off + (long long)h * D + lane * 4);
    nw = *reinterpret_cast<const float4*>(p.norm_w + lane * 4);
  }
  const auto filtered = [&](const float (&x)[K], const float (&w)[K]) {
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < K; ++j) acc = fmaf(w[j], x[j], acc);
    return silu(acc);
  };
  const auto move_on = [&](long long c, const float (&x)[K]) {
    float* tl = p.tail + (slot * C + c) * (K - 1);
#pragma unroll
    for (int j = 0; j < K - 1; ++j) tl[j] = x[j + 1];
  };
  qk[tid] = filtered(x[0], w[0]);
  if (tid < D) {
    vs[tid] = filtered(x[1], w[1]);
    move_on(c_v, x[1]);
  }
  if (piece == kRegPieces - 1 && lane < 2)
    gates[lane] = lane ? 1.f / (1.f + expf(-row[p.b_off + h])) : decay_of(p.A_log[h], row[p.a_off + h], p.dt_bias[h]);
  if (rep > 1) kb2::cluster_sync_all();      // every head has read the tails of q and k
  else __syncthreads();
  if (h == hk * rep) move_on(c_qk, x[0]);
  if (piece < 2) {                 // unit rows
    float *r = qk + piece * D, a = 0.f;
#pragma unroll
    for (int i = 0; i < D / 32; ++i) a += r[lane + 32 * i] * r[lane + 32 * i];
    a = warp_sum(a);
    const float f = piece ? 1.f / sqrtf(a + 1e-6f) : (1.f / sqrtf((float)D)) / sqrtf(a + 1e-6f);
#pragma unroll
    for (int i = 0; i < D / 32; ++i) r[lane + 32 * i] *= f;
  }
  __syncthreads();
  const float g = gates[0], b = gates[1];
  const float4 *q4 = reinterpret_cast<const float4*>(qk + piece * Q), *k4 = reinterpret_cast<const float4*>(qk + D + piece * Q);
  // the sums over a piece's rows i = 0, 4, 8, ..; 1, 5, ..; 2, ..; 3, .. of S times a row's number, for the lane's four columns
  const auto dot = [](const float4 (&S)[Q], const float4* f4) {
    float4 a[4] = {};
#pragma unroll
    for (int i = 0; i < Q / 4; ++i) {
      const float4 f = f4[i];
      const float fv[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a[e].x = fmaf(S[4 * i + e].x, fv[e], a[e].x);
        a[e].y = fmaf(S[4 * i + e].y, fv[e], a[e].y);
        a[e].z = fmaf(S[4 * i + e].z, fv[e], a[e].z);
        a[e].w = fmaf(S[4 * i + e].w, fv[e], a[e].w);
      }
    }
    return make_float4((a[0].x + a[1].x) + (a[2].x + a[3].x), (a[0].y + a[1].y) + (a[2].y + a[3].y), (a[0].z + a[1].z) + (a[2].z + a[3].z),
                       (a[0].w + a[1].w) + (a[2].w + a[3].w));
  };
  *reinterpret_cast<float4*>(&part[piece][lane * 4]) = dot(S, k4);
  __syncthreads();
  float4 u;
  {
    float4 pp[kRegPieces];
#pragma unroll
    for (int i = 0; i < kRegPieces; ++i) pp[i] = *reinterpret_cast<const float4*>(&part[i][lane * 4]);
    const float4 v = *reinterpret_cast<const float4*>(&vs[lane * 4]);
    const auto strength = [&](float p0, float p1, float p2, float p3, float p4, float p5, float p6, float p7, float vv) {
      const float sk = ((p0 + p1) + (p2 + p3)) + ((p4 + p5) + (p6 + p7));
      return b * (vv - g * sk);
    };
    u = make_float4(strength(pp[0].x, pp[1].x, pp[2].x, pp[3].x, pp[4].x, pp[5].x, pp[6].x, pp[7].x, v.x),
                    strength(pp[0].y, pp[1].y, pp[2].y, pp[3].y, pp[4].y, pp[5].y, pp[6].y, pp[7].y, v.y),
                    strength(pp[0].z, pp[1].z, pp[2].z, pp[3].z, pp[4].z, pp[5].z, pp[6].z, pp[7].z, v.z),
                    strength(pp[0].w, pp[1].w, pp[2].w, pp[3].w, pp[4].w, pp[5].w, pp[6].w, pp[7].w, v.w));
  }
#pragma unroll
  for (int i = 0; i < Q / 4; ++i) {
    const float4 f = k4[i];
    const float fv[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float4& s = S[4 * i + e];
      s = make_float4(fmaf(fv[e], u.x, g * s.x), fmaf(fv[e], u.y, g * s.y), fmaf(fv[e], u.z, g * s.z), fmaf(fv[e], u.w, g * s.w));
      Sg[(4 * i + e) * (D / 4)] = s;
    }
  }
  *reinterpret_cast<float4*>(&os[piece][lane * 4]) = dot(S, q4);
  __syncthreads();
  if (piece == 0) {
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kRegPieces; ++i) {
      const float4 f = *reinterpret_cast<const float4*>(&os[i][lane * 4]);
      o.x += f.x; o.y += f.y; o.z += f.z; o.w += f.w;
    }
    const float rstd = 1.f / sqrtf(warp_sum((o.x * o.x + o.y * o.y) + (o.z * o.z + o.w * o.w)) / (float)D + p.eps);
    const auto finish = [&](float v, float z, float n) { return v * rstd * n * silu(z); };
    const float4 r = make_float4(finish(o.x, gz.x, nw.x), finish(o.y, gz.y, nw.y), finish(o.z, gz.z, nw.z), finish(o.w, gz.w, nw.w));
    const long long at = (t * p.H + h) * D + lane * 4;
    if (p.dt_out == 0) {
      *reinterpret_cast<float4*>((float*)p.out + at) = r;
    } else {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(r.x, r.y), hi = __floats2bfloat162_rn(r.z, r.w);
      *reinterpret_cast<uint2*>((bf16*)p.out + at) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  }
}

}  // namespace kb2seq

using namespace kb2seq;

extern "C" {

KB2SEQ_API const char* kb2_seq_last_error(void) { return g_err; }
KB2SEQ_API int kb2_seq_wait_timeouts(int device, int put, int* up) {
  if (!up) return failf(KB2SEQ_ERR_VALUE, "wait_timeouts: bad argument");
  SEQ_CUDA(kb2::exchange_wait_flags(device, put, up));
  return KB2SEQ_OK;
}
KB2SEQ_API long long kb2_seq_total_launches(void) { return g_launches; }

KB2SEQ_API int kb2_seq_embed(const void* table, int dt, const int* tokens, float* x, int T, int W, float scale, void* stream) {
  if (!table || !tokens || !x || T <= 0 || W <= 0 || bad_dt(dt)) return failf(KB2SEQ_ERR_VALUE, "embed: bad argument");
  if (dt && W % 8 == 0 && !((uintptr_t)table & 15) && !((uintptr_t)x & 15))
    kb2::launch_pdl(embed_scale_vec_kernel, T, 256, 0, (cudaStream_t)stream, (const bf16*)table, tokens, x, W, scale);
  else if (dt) kb2::launch_pdl(embed_scale_kernel<bf16>, T, 128, 0, (cudaStream_t)stream, (const bf16*)table, tokens, x, W, scale);
  else kb2::launch_pdl(embed_scale_kernel<float>, T, 128, 0, (cudaStream_t)stream, (const float*)table, tokens, x, W, scale);
  SEQ_LAUNCHED();
  return KB2SEQ_OK;
}

KB2SEQ_API int kb2_seq_gemm(const void* A, int dtA, long long lda, const void* B, int dtB, long long ldb, void* C, int dtC,
                            long long ldc, int M, int N, int K, int batch, long long sA, long long sB, long long sC, void* stream) {
  if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0 || batch <= 0 || batch > 65535 || bad_dt(dtA) || bad_dt(dtB) || bad_dt(dtC))
    return failf(KB2SEQ_ERR_VALUE, "gemm: bad argument (M=%d N=%d K=%d batch=%d)", M, N, K, batch);
  cudaStream_t s = (cudaStream_t)stream;
  const int code = dtA * 4 + dtB * 2 + dtC;
#define G(TA, TB, TC) launch_gemm<TA, TB, TC>(A, lda, B, ldb, C, ldc, M, N, K, batch, sA, sB, sC, s)
  switch (code) {
    case 0: G(float, float, float); break;
    case 1: G(float, float, bf16); break;
    case 2: G(float, bf16, float); break;
    case 3: G(float, bf16, bf16); break;
    case 4: G(bf16, float, float); break;
    case 5: G(bf16, float, bf16); break;
    case 6: G(bf16, bf16, float); break;
    default: G(bf16, bf16, bf16); break;
  }
#undef G
  SEQ_LAUNCHED();
  return KB2SEQ_OK;
}

KB2SEQ_API int kb2_seq_residual_norm(float* x, const float* y, int y_mode, const float* wa, const float* ba, const float* x0,
                                     const float* wb, const float* bb, void* h, int dt_h, int T, int W, float eps, void* stream) {
  if (!x || T <= 0 || W <= 0 || bad_dt(dt_h)) return failf(KB2SEQ_ERR_VALUE, "residual_norm: bad argument");
  if (y && (y_mode < 1 || y_mode > 2 || !wa || (y_mode == 1 && !ba))) return failf(KB2SEQ_ERR_VALUE, "residual_norm: norm of y needs its weights");
  if (h && (!wb || !bb)) return failf(KB2SEQ_ERR_VALUE, "residual_norm: output norm needs weight and bias");
  const size_t smem = (size_t)W * 4;
  if (smem > 200 * 1024) return failf(KB2SEQ_ERR_VALUE, "residual_norm: width %d too large", W);
  return launch_residual_norm(x, y, y_mode, wa, ba, x0, wb, bb, h, dt_h, T, W, eps, nullptr, (cudaStream_t)stream);
}

KB2SEQ_API int kb2_seq_residual_add_norm(float* x, const float* y, const float* y2, const float* wb, const float* bb, void* h, int dt_h,
                                         int T, int W, float eps, void* stream) {
  if (!x || T <= 0 || W <= 0 || bad_dt(dt_h) || (y2 && !y)) return failf(KB2SEQ_ERR_VALUE, "residual_add_norm: bad argument");
  if (h && !wb) return failf(KB2SEQ_ERR_VALUE, "residual_add_norm: output norm needs its weight");
  const size_t smem = (size_t)W * 4;
  if (smem > 200 * 1024) return failf(KB2SEQ_ERR_VALUE, "residual_add_norm: width %d too large", W);
  return launch_residual_norm(x, y, 3, nullptr, nullptr, nullptr, wb, bb, h, dt_h, T, W, eps, y2, (cudaStream_t)stream);
}

KB2SEQ_API int kb2_seq_act_mul(const void* in, int dt_in, void* out, int dt_out, int T, int F, void* stream) {
  if (!in || !out || T <= 0 || F <= 0 || bad_dt(dt_in) || bad_dt(dt_out)) return failf(KB2SEQ_ERR_VALUE, "act_mul: bad argument");
  if (T > 65535) return failf(KB2SEQ_ERR_VALUE, "act_mul: more than 65535 rows in one step");
  if (dt_in == 1 && dt_out == 1 && F % 8 == 0 && !((uintptr_t)in & 15) && !((uintptr_t)out & 15))
    kb2::launch_pdl(act_mul_bf16x8_kernel, dim3((F / 8 + 127) / 128, T), 128, 0, (cudaStream_t)stream, (const bf16*)in, (bf16*)out, F);
  else if (dt_in == 0 && dt_out == 0 && F % 4 == 0 && !((uintptr_t)in & 15) && !((uintptr_t)out & 15))
    kb2::launch_pdl(act_mul_f32x4_kernel, dim3((F / 4 + 255) / 256, T), 256, 0, (cudaStream_t)stream, (const float*)in, (float*)out, F);
  else
    kb2::launch_pdl(act_mul_kernel, dim3((F + 255) / 256, T), 256, 0, (cudaStream_t)stream, in, dt_in, out, dt_out, T, F);
  SEQ_LAUNCHED();
  return KB2SEQ_OK;
}

KB2SEQ_API int kb2_seq_side_gate(const float* g, const void* table, int dt_table, long long table_ld, const int* tokens, int col0,
                                 int dim, int T, void* out, int dt_out, void* stream) {
  if (!g || !table || !tokens || !out || T <= 0 || dim <= 0 || col0 < 0 || bad_dt(dt_table) || bad_dt(dt_out))
    return failf(KB2SEQ_ERR_VALUE, "side_gate: bad argument");
  const long long n = (long long)T * dim;
  kb2::launch_pdl(side_gate_kernel, (unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream, g, table, dt_table, table_ld, tokens, col0, dim, T, out,
                                                                                  dt_out);
  SEQ_LAUNCHED();
  return KB2SEQ_OK;
}

KB2SEQ_API int kb2_seq_latent_prep(float* proj, long long ldp, int T, int H, int dn, int dr, int r, const float* cw, float eps,
                                   const double* freq, int rot_dims, float amp, const int* positions, const int* seq_of,
                                   const int* pages, int max_pages, int page_size, void* ckv, void* kr, int dt_cache, const float* lat,
                                   long long ldl, void* stream) {
  if (!proj || !cw || !freq || !positions || !seq_of || !pages || !ckv || !kr || T <= 0 || H <= 0 || dn < 0 || dr < 0 || r <= 0 ||
      rot_dims < 0 || rot_dims > dr || (rot_dims & 1) || page_size <= 0 || max_pages <= 0 || bad_dt(dt_cache))
    return failf(KB2SEQ_ERR_VALUE, "latent_prep: bad argument");
  kb2::launch_pdl(latent_prep_kernel, T, 512, 0, (cudaStream_t)stream, proj, ldp, H, dn, dr, r, cw, eps, freq, rot_dims, amp, positions, seq_of, pages,
                                                          max_pages, page_size, ckv, kr, dt_cache, lat, ldl);
  SEQ_LAUNCHED();
  return KB2SEQ_OK;
}

KB2SEQ_API int kb2_seq_latent_window_attn(const float* q_abs, const float* proj, long long ldp, int T, int H, int dn, int dr, int r,
                                          const void* ckv, const void* kr, int dt_cache, const int* positions, const int* seq_of,
                                          const int* pages, int max_pages, int page_size, const float* sinks, float scale, int window,
                                          float* out, const int* cu, int skip_from, int nsplit, float* part_acc, float* part_ml,
                                          const float* gate, long long ldg, void* stream) {
  if (!q_abs || !proj || !ckv || !kr || !positions || !seq_of || !pages || !out || T <= 0 || H <= 0 || r <= 0 || dr < 0 ||
      window <= 0 || bad_dt(dt_cache))
    return failf(KB2SEQ_ERR_VALUE, "latent_window_attn: bad argument");
  if (r > kAttnThreads * kAttnAcc) return failf(KB2SEQ_ERR_VALUE, "latent_window_attn: latent size %d > %d", r, kAttnThreads * kAttnAcc);
  const int D = r + dr;
  int NC = 1;                              // latent columns per thread: a power of two
  while (NC * kAttnThreads < r) NC <<= 1;
  int HG = 8;                              // heads per block: a power of two, HG x NC sums per thread
  while (HG > 1 && (HG > H || HG * NC > kAttnAcc || attn_smem_floats(HG, D) * 4 > 200 * 1024)) HG >>= 1;
  if (nsplit < 1 || nsplit > 1024 || (nsplit > 1 && (!part_acc || !part_ml))) return failf(KB2SEQ_ERR_VALUE, "latent_window_attn: bad key split");
  const size_t smem = attn_smem_floats(HG, D) * 4;
  if (smem > 200 * 1024) return failf(KB2SEQ_ERR_VALUE, "latent_window_attn: latent + rotated size %d too large", D);
  const dim3 grid(T, (H + HG - 1) / HG, nsplit);
  const int unit = dt_cache ? 8 : 4;
  const bool vec_k = r % unit == 0 && dr % unit == 0 && !(((uintptr_t)ckv | (uintptr_t)kr) & 15);
  const bool vec_q = r % 4 == 0 && dr % 4 == 0 && dn % 4 == 0 && ldp % 4 == 0 && !(((uintptr_t)q_abs | (uintptr_t)proj) & 15);
#define KB2_LA(HGV, NCV)                                                                                                                      \
  case HGV * 32 + NCV: {                                                                                                                      \
    if (smem > 48 * 1024)                                                                                                                     \
      SEQ_CUDA(cudaFuncSetAttribute(latent_window_attn_kernel<HGV, NCV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));            \
    kb2::launch_pdl(latent_window_attn_kernel<HGV, NCV>, grid, kAttnThreads, smem, (cudaStream_t)stream,                                                    \
        q_abs, proj, ldp, H, dn, dr, r, ckv, kr, dt_cache, positions, seq_of, pages, max_pages, page_size, sinks, scale, window, out, cu,     \
        skip_from, nsplit, part_acc, part_ml, gate, ldg, vec_q, vec_k);                                                                              \
    break;                                                                                                                                    \
  }
  switch (HG * 32 + NC) {
    KB2_LA(8, 1) KB2_LA(8, 2) KB2_LA(4, 1) KB2_LA(4, 2) KB2_LA(4, 4) KB2_LA(2, 1) KB2_LA(2, 2) KB2_LA(2, 4) KB2_LA(2, 8)
    KB2_LA(1, 1) KB2_LA(1, 2) KB2_LA(1, 4) KB2_LA(1, 8) KB2_LA(1, 16)
    default: return failf(KB2SEQ_ERR_VALUE, "latent_window_attn: no kernel for %d heads x %d columns", HG, NC);
  }
#undef KB2_LA
  SEQ_LAUNCHED();
  if (nsplit > 1) {
    kb2::launch_pdl(latent_attn_combine_kernel, dim3(T, H), r >= 512 ? 512 : (r + 31) / 32 * 32, (size_t)nsplit * 4, (cudaStream_t)stream, part_acc, part_ml, H, r, nsplit, out, seq_of, cu, skip_from,
                                                                                               gate, ldg);
    SEQ_LAUNCHED();
  }
  return KB2SEQ_OK;
}

KB2SEQ_API int kb2_seq_conv(const float* proj, long long ldp, int T, int S, int C, int K, const float* taps, const float* bias,
                            const float* bias_out, int act, float* tail, const int* seq_of, const int* cu, const int* slots, float* out,
                            void* stream) {
  if (!proj || !taps || !tail || !seq_of || !cu || !slots || !out || T <= 0 || S <= 0 || C <= 0 || K <= 0 || act < 0 || act > 1)
    return failf(KB2SEQ_ERR_VALUE, "conv: bad argument");
  if (T > 65535) return failf(KB2SEQ_ERR_VALUE, "conv: more than 65535 rows in one step");
  const bool vec = C % 4 == 0 && ldp % 4 == 0 && !(((uintptr_t)proj | (uintptr_t)out) & 15);
  const dim3 vgrid((C / 4 + kConvThreads - 1) / kConvThreads, (T + kConvRun - 1) / kConvRun);
#define KB2_CONV(KV)                                                                                                                                        \
  SEQ_CUDA(kb2::allow_smem<conv_run_vec_kernel<KV>>(kConvSmem<KV>));                                                                                        \
  kb2::launch_pdl(conv_run_vec_kernel<KV>, vgrid, kConvThreads, kConvSmem<KV>, (cudaStream_t)stream, proj, ldp, C, taps, tail, seq_of, cu, slots, T, out, bias, act, bias_out)
  if (T >= 4 * kConvRun && vec && K >= 2 && K <= 4) {
    if (K == 2) { KB2_CONV(2); } else if (K == 3) { KB2_CONV(3); } else { KB2_CONV(4); }
  } else if (T >= 4 * kConvRun && K <= kConvMaxTaps)
    kb2::launch_pdl(conv_run_kernel, dim3((C + 255) / 256, (T + kConvRun - 1) / kConvRun), 256, 0, (cudaStream_t)stream, proj, ldp, C, K, taps, tail, seq_of,
                                                                                                          cu, slots, T, out, bias, act, bias_out);
  else
    kb2::launch_pdl(conv_silu_kernel, dim3((C + 255) / 256, T), 256, 0, (cudaStream_t)stream, proj, ldp, C, K, taps, tail, seq_of, cu, slots, T, out, bias,
                                                                                 act, bias_out);
#undef KB2_CONV
  SEQ_LAUNCHED();
  if (K > 1) {
    const long long m = (long long)S * C;
    kb2::launch_pdl(conv_tail_kernel, (unsigned)((m + 255) / 256), 256, 0, (cudaStream_t)stream, proj, ldp, C, K, tail, cu, slots, S, bias);
    SEQ_LAUNCHED();
  }
  return KB2SEQ_OK;
}

KB2SEQ_API int kb2_seq_conv_silu(const float* proj, long long ldp, int T, int S, int C, int K, const float* taps, float* tail,
                                 const int* seq_of, const int* cu, const int* slots, float* out, void* stream) {
  return kb2_seq_conv(proj, ldp, T, S, C, K, taps, nullptr, nullptr, 1, tail, seq_of, cu, slots, out, stream);
}

KB2SEQ_API int kb2_seq_residual_scale_rms(float* x, const float* y, float y_mult, const float* w, float w_shift, void* h, int dt_h, int T,
                                          int W, float eps, void* stream) {
  if (!x || T <= 0 || W <= 0 || bad_dt(dt_h) || (h && !w)) return failf(KB2SEQ_ERR_VALUE, "residual_scale_rms: bad argument");
  if (h == (void*)x && (y || dt_h != 0)) return failf(KB2SEQ_ERR_VALUE, "residual_scale_rms: a norm in place takes no addend and is fp32");
  const size_t smem = (size_t)W * 4;
  if (smem > 200 * 1024) return failf(KB2SEQ_ERR_VALUE, "residual_scale_rms: width %d too large", W);
  if (smem > 48 * 1024) SEQ_CUDA(cudaFuncSetAttribute(residual_scale_rms_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kb2::launch_pdl(residual_scale_rms_kernel, T, 256, smem, (cudaStream_t)stream, x, y, y_mult, w, w_shift, h, dt_h, W, eps);
  SEQ_LAUNCHED();
  return KB2SEQ_OK;
}

KB2SEQ_API int kb2_seq_residual_post_rms(float* x, const float* y1, float c1, const float* y2, float c2, const float* bias, float mult,
                                         const float* w, const float* wh, void* h, int dt_h, int T, int W, float eps, void* stream) {
  if (!x || T <= 0 || W <= 0 || bad_dt(dt_h) || (y1 && !w) || (!y1 && (y2 || !h)) || (wh && !h) || h == (void*)x)
    return failf(KB2SEQ_ERR_VALUE, "residual_post_rms: bad argument");
  const size_t smem = (size_t)W * 4;
  if (smem > 200 * 1024) return failf(KB2SEQ_ERR_VALUE, "residual_post_rms: width %d too large", W);
  const uintptr_t all = (uintptr_t)x | (uintptr_t)y1 | (uintptr_t)y2 | (uintptr_t)bias | (uintptr_t)w | (uintptr_t)wh | (uintptr_t)h;
  if (W % 4 == 0 && !(all & 15)) {
    if (smem > 40 * 1024) SEQ_CUDA(cudaFuncSetAttribute(residual_post_rms_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kb2::launch_pdl(residual_post_rms_kernel<4>, T, 256, smem, (cudaStream_t)stream, x, y1, c1, y2, c2, bias, mult, w, wh, h, dt_h, W, eps);
  } else {
    if (smem > 40 * 1024) SEQ_CUDA(cudaFuncSetAttribute(residual_post_rms_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kb2::launch_pdl(residual_post_rms_kernel<1>, T, 256, smem, (cudaStream_t)stream, x, y1, c1, y2, c2, bias, mult, w, wh, h, dt_h, W, eps);
  }
  SEQ_LAUNCHED();
  return KB2SEQ_OK;
}

static int delta_out_launch(const float* o, const float* gproj, long long ldg, int gate_act, int H, int dv, const float* norm_w, float eps, int T,
                            void* out, int dt_out, cudaStream_t st) {
  const unsigned blocks = (unsigned)(((long long)T * H + 7) / 8);
  const bool vec = dv % 4 == 0 && ldg % 4 == 0 && !(((uintptr_t)o | (uintptr_t)gproj | (uintptr_t)norm_w | (uintptr_t)out) & 15);
  if (vec && dv == 128 && blocks >= kb2::current_sms() * 16u)         // from two full rounds of resident blocks on
    kb2::launch_pdl(delta_out_rows_kernel, (blocks + 3) / 4, 256, 0, st, o, gproj, ldg, gate_act, H, norm_w, eps, (long long)T * H, out, dt_out);
  else if (vec)
    kb2::launch_pdl(delta_out_kernel<4>, blocks, 256, 0, st, o, gproj, ldg, gate_act, H, dv, norm_w, eps, T, out, dt_out);
  else
    kb2::launch_pdl(delta_out_kernel<1>, blocks, 256, 0, st, o, gproj, ldg, gate_act, H, dv, norm_w, eps, T, out, dt_out);
  SEQ_LAUNCHED();
  return KB2SEQ_OK;
}

static int delta_rule_launch(const float* conv, int C, const float* bproj, long long ldb, const float* aproj, long long lda, int ch,
                             const float* gproj, long long ldg, int gate_act, int T, int S, int H, int Hk, int dk, int dv,
                             const float* A_log, const float* dt_bias, const float* norm_w, float eps, float* state, const int* cu,
                             const int* slots, float* scratch, void* out, int dt_out, void* stream) {
  if (!conv || !bproj || !aproj || !gproj || !A_log || !dt_bias || !norm_w || !state || !cu || !slots || !out || S <= 0 || H <= 0 ||
      Hk <= 0 || H % Hk || dk <= 0 || dv <= 0 || bad_dt(dt_out))
    return failf(KB2SEQ_ERR_VALUE, "delta_rule: bad argument");
  if (scratch && (dk == 32 || dk == 64 || dk == 128) && dv % 32 == 0 && C % 4 == 0 && ((2 * Hk * dk) % 4) == 0) {
    // scratch: qn [T, Hk, dk] | kn [T, Hk, dk] | beta [T, H] | dec [T, H] or [T, H, dk] | o [T, H, dv]   (fp32)
    cudaStream_t st = (cudaStream_t)stream;
    float* qn = scratch;
    float* kn = qn + (long long)T * Hk * dk;
    float* be = kn + (long long)T * Hk * dk;
    float* de = be + (long long)T * H;
    if (ch) de = (float*)(((uintptr_t)de + 15) & ~(uintptr_t)15);
    float* ob = de + (long long)T * H * (ch ? dk : 1);
    ob = (float*)(((uintptr_t)ob + 15) & ~(uintptr_t)15);
    const long long nw = (long long)T * Hk;
    kb2::launch_pdl(delta_prep_kernel, (unsigned)((nw + 7) / 8), 256, 0, st, conv, C, bproj, ldb, aproj, lda, ch, H, Hk, dk, A_log, dt_bias, T, qn, kn, be, de);
    SEQ_LAUNCHED();
    dim3 grid(S, H, dv / 32);
    const int v_col0 = 2 * Hk * dk;
#define R(DK, CHV) kb2::launch_pdl(delta_rule_reg_kernel<DK, CHV>, grid, 32 * kRegPieces, 0, st, qn, kn, conv, C, v_col0, be, de, H, Hk, dv, state, cu, slots, ob)
    if (ch) {
      if (dk == 32) R(32, true); else if (dk == 64) R(64, true); else R(128, true);
    } else {
      if (dk == 32) R(32, false); else if (dk == 64) R(64, false); else R(128, false);
    }
#undef R
    SEQ_LAUNCHED();
    return delta_out_launch(ob, gproj, ldg, gate_act, H, dv, norm_w, eps, T, out, dt_out, st);
  }
  auto smem_of = [&](int cols) { return ((size_t)dk * cols + (size_t)kDeltaTile * (2 * dk + cols + 1 + (ch ? dk : 1))) * 4; };
  int dvb = dv;                                // a state too large for one block's shared memory is cut into slices of value columns
  if (dv > 1024 || smem_of(dv) > 220 * 1024) {
    dvb = dv < 1024 ? dv / 32 * 32 : 1024;
    while (dvb > 32 && smem_of(dvb) > 220 * 1024) dvb -= 32;
    if (dvb < 32 || smem_of(dvb) > 220 * 1024)
      return failf(KB2SEQ_ERR_VALUE, "delta_rule: %d key channels do not fit one block's shared memory", dk);
    if (!scratch) return failf(KB2SEQ_ERR_VALUE, "delta_rule: a %d x %d state needs the scratch buffer (T H dv floats)", dk, dv);
  }
  const size_t smem = smem_of(dvb);
  if (smem > 48 * 1024) SEQ_CUDA(cudaFuncSetAttribute(delta_rule_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int threads = (dvb + 31) / 32 * 32;
  if (threads < 128) threads = 128;
  const bool cut = dvb < dv;
  dim3 grid(S, H, (dv + dvb - 1) / dvb);
  kb2::launch_pdl(delta_rule_kernel, grid, threads, smem, (cudaStream_t)stream, conv, C, bproj, ldb, aproj, lda, ch, gproj, ldg, gate_act, H, Hk, dk, dv, A_log,
                                                                  dt_bias, norm_w, eps, state, cu, slots, out, dt_out, dvb,
                                                                  cut ? scratch : nullptr);
  SEQ_LAUNCHED();
  if (cut) return delta_out_launch(scratch, gproj, ldg, gate_act, H, dv, norm_w, eps, T, out, dt_out, (cudaStream_t)stream);
  return KB2SEQ_OK;
}

// scratch: images of k and q [slice][Hk] | of W [slice][H] | V' [slice][H][16 dv] | scalars [slice][H] | o [T, H, dv].  At most T / 16 + S tiles, a
// partial one per sequence.  What belongs to tiles (74 KB per token with 32 / 16 heads x 128, twice that of tiles of eight, which had no W and no V') is
// made and used a slice of tiles at a time, so that it stays below kDeltaSliceBytes: 8192 tokens take 435 MB in all instead of 704, in 2 % more time.
// Slices of 96 MB cost 5 to 7 % (4096 tokens 488 -> 524 us) and 20 % with several sequences, whose chains no longer run side by side.
constexpr long long kDeltaSliceBytes = 320ll << 20;
struct DeltaScratch {
  long long tiles, slice, image, wimage, floats;      // floats of an image, of W, of everything
  DeltaScratch(int T, int S, int H, int Hk, int dk, int dv) : tiles((long long)T / kDT + S) {
    image = dk == 32 ? DeltaTile<1>::kImage / 2 : dk == 64 ? DeltaTile<2>::kImage / 2 : DeltaTile<4>::kImage / 2;
    wimage = image / 2;
    const long long per = Hk * image + H * (wimage + (long long)kDT * dv + kDTScalars), most = std::max(1ll, kDeltaSliceBytes / 4 / per);
    const long long slices = (tiles + most - 1) / most;
    slice = (tiles + slices - 1) / slices;
    floats = slice * per + (long long)T * H * dv;
  }
};
KB2SEQ_API long long kb2_seq_delta_tiles_scratch(int T, int S, int H, int Hk, int dk, int dv) {
  if (T <= 0 || S <= 0 || H <= 0 || Hk <= 0 || H % Hk || (dk != 32 && dk != 64 && dk != 128) || dv <= 0 || dv % 32) return 0;
  return DeltaScratch(T, S, H, Hk, dk, dv).floats;
}

extern "C++" {
template <int NI, int VB>
static int launch_delta_tiles(const DeltaScratch& z, DeltaPrep p, float* state, const int* slots, float* scratch, float** o, cudaStream_t st) {
  using D = DeltaTile<NI>;
  p.image = (bf16*)scratch;
  p.wimage = (bf16*)(scratch + z.slice * p.Hk * z.image);
  p.vimage = scratch + z.slice * (p.Hk * z.image + p.H * z.wimage);
  p.sc = p.vimage + z.slice * p.H * kDT * p.dv;
  *o = p.sc + z.slice * p.H * kDTScalars;
  p.whole = z.slice == z.tiles;
  const int prep_smem = D::prep_smem(VB, p.H / p.Hk);
  if (prep_smem > 227 * 1024) return failf(KB2SEQ_ERR_VALUE, "delta_tiles: %d heads per key head are too many", p.H / p.Hk);
  SEQ_CUDA((kb2::allow_smem<delta_tile_prep_kernel<NI, VB>>(227 * 1024)));
  SEQ_CUDA((kb2::allow_smem<delta_tile_kernel<NI>>(D::kSmem)));
  for (p.f0 = 0; p.f0 < z.tiles; p.f0 += z.slice) {
    p.f1 = std::min(p.f0 + z.slice, z.tiles);
    kb2::launch_pdl(delta_tile_prep_kernel<NI, VB>, (unsigned)((p.f1 - p.f0) * p.Hk), 256, prep_smem, st, p);
    SEQ_LAUNCHED();
    kb2::launch_pdl(delta_tile_kernel<NI>, dim3(p.S, p.H, p.dv / 32), D::kThreads, D::kSmem, st, p.image, p.wimage, p.vimage, p.sc, p.H, p.Hk, p.dv, state,
                    p.cu, slots, *o, p.f0, p.f1, p.whole);
    SEQ_LAUNCHED();
  }
  return KB2SEQ_OK;
}
}  // extern "C++"

KB2SEQ_API int kb2_seq_delta_tiles(const float* conv, int C, const float* proj, long long ldp, int g_off, int a_off, int b_off, int T, int S, int H,
                                   int Hk, int dk, int dv, const float* A_log, const float* dt_bias, const float* norm_w, float eps, float* state,
                                   const int* cu, const int* slots, float* scratch, long long scratch_floats, void* out, int dt_out, void* stream) {
  const long long need = kb2_seq_delta_tiles_scratch(T, S, H, Hk, dk, dv);
  if (!conv || !proj || !A_log || !dt_bias || !norm_w || !state || !cu || !slots || !scratch || !out || bad_dt(dt_out) || !need ||
      scratch_floats < need || ((uintptr_t)scratch & 15) || ((uintptr_t)conv & 15) || C % 4 || C < 2 * Hk * dk + H * dv)
    return failf(KB2SEQ_ERR_VALUE, "delta_tiles: bad argument");
  cudaStream_t st = (cudaStream_t)stream;
  const DeltaScratch z(T, S, H, Hk, dk, dv);
  DeltaPrep p{};
  p.conv = conv; p.C = C; p.ldp = ldp; p.bproj = proj + b_off; p.aproj = proj + a_off; p.A_log = A_log; p.dt_bias = dt_bias;
  p.H = H; p.Hk = Hk; p.dv = dv; p.S = S; p.cu = cu;
  float* ob = nullptr;
  // values in passes of 128 columns, 64 or 32 (32 portions of 64 tokens, 8 heads of 64: 32 columns a pass made the step slower than its eight-token form)
#define KB2_DT1(NIV, VBV) launch_delta_tiles<NIV, VBV>(z, p, state, slots, scratch, &ob, st)
#define KB2_DT(NIV) (dv % 128 == 0 ? KB2_DT1(NIV, 4) : dv % 64 == 0 ? KB2_DT1(NIV, 2) : KB2_DT1(NIV, 1))
  const int rc = dk == 32 ? KB2_DT(1) : dk == 64 ? KB2_DT(2) : KB2_DT(4);
#undef KB2_DT
#undef KB2_DT1
  if (rc != KB2SEQ_OK) return rc;
  return delta_out_launch(ob, proj + g_off, ldp, 0, H, dv, norm_w, eps, T, out, dt_out, st);
}

KB2SEQ_API int kb2_seq_delta_rule(const float* conv, int C, const float* proj, long long ldp, int g_off, int a_off, int b_off, int T,
                                  int S, int H, int Hk, int dk, int dv, const float* A_log, const float* dt_bias, const float* norm_w,
                                  float eps, float* state, const int* cu, const int* slots, float* scratch, void* out, int dt_out,
                                  void* stream) {
  if (!proj) return failf(KB2SEQ_ERR_VALUE, "delta_rule: bad argument");
  return delta_rule_launch(conv, C, proj + b_off, ldp, proj + a_off, ldp, 0, proj + g_off, ldp, 0, T, S, H, Hk, dk, dv, A_log, dt_bias, norm_w,
                           eps, state, cu, slots, scratch, out, dt_out, stream);
}

KB2SEQ_API int kb2_seq_delta_rule_ch(const float* conv, int C, const float* beta_in, long long ldb, const float* decay_in, long long lda,
                                     const float* gate_in, long long ldg, int gate_act, int T, int S, int H, int Hk, int dk, int dv,
                                     const float* A_log, const float* dt_bias, const float* norm_w, float eps, float* state, const int* cu,
                                     const int* slots, float* scratch, void* out, int dt_out, void* stream) {
  if (gate_act < 0 || gate_act > 1) return failf(KB2SEQ_ERR_VALUE, "delta_rule_ch: bad argument");
  return delta_rule_launch(conv, C, beta_in, ldb, decay_in, lda, 1, gate_in, ldg, gate_act, T, S, H, Hk, dk, dv, A_log, dt_bias, norm_w, eps,
                           state, cu, slots, scratch, out, dt_out, stream);
}

KB2SEQ_API int kb2_seq_delta_step(const float* proj, long long ldp, int g_off, int a_off, int b_off, int T, int H, int Hk, int dk, int dv, int K,
                                  const float* taps, float* tail, const float* A_log, const float* dt_bias, const float* norm_w, float eps, float* state,
                                  const int* slots, void* out, int dt_out, void* stream) {
  if (!proj || !taps || !tail || !A_log || !dt_bias || !norm_w || !state || !slots || !out || T <= 0 || H <= 0 || Hk <= 0 || H % Hk || bad_dt(dt_out))
    return failf(KB2SEQ_ERR_VALUE, "delta_step: bad argument");
  if (dk != 128 || dv != 128 || K < 2 || K > 4 || H / Hk > 8 || T > 65535 || ldp % 4 || g_off % 4 || (((uintptr_t)proj | (uintptr_t)norm_w | (uintptr_t)state | (uintptr_t)out) & 15))
    return failf(KB2SEQ_ERR_VALUE, "delta_step: 128 key and value channels, at most 8 heads per key head, 2 to 4 taps and 16-byte aligned rows");
  const DeltaStep p{proj, ldp, g_off, a_off, b_off, H, Hk, taps, A_log, dt_bias, norm_w, eps, tail, state, slots, out, dt_out};
  auto kern = K == 2 ? delta_step_kernel<2> : K == 3 ? delta_step_kernel<3> : delta_step_kernel<4>;
  kb2::launch_pdl_clusters(kern, dim3(H, T), 256, 0, (cudaStream_t)stream, dim3(H / Hk, 1, 1), p);
  SEQ_LAUNCHED();
  return KB2SEQ_OK;
}

}  // extern "C"
