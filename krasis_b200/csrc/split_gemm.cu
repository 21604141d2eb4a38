// Dense BF16 product for few rows:  Y[M,N] = X[M,K] (bf16) x W[N,K]^T (bf16), fp32 accumulation in TMEM, BF16 or FP32 output.
//
// Bound: the weights.  Up to a few hundred rows the time is N * K * 2 bytes from HBM, and dense_gemm.cu's 128 x 256 tiles leave most SMs
// without a tile (N = 2048: 8 tiles per 128 rows).  So the roles of the operands are swapped — 128 weight rows are the UMMA's M side, the
// rows of X (any multiple of 16 up to 256) its N side, which costs no padding to 128 rows — and K is cut over the CTAs of a cluster
// (1, 2, 4 or 8).  A CTA has one tile: its TMA ring streams the weights while two CTAs share an SM, so that one fills its ring while the
// other drains.  The partial tiles of a cluster meet in shared memory (one [row][128] fp32 image per CTA, read through distributed shared
// memory); every output is summed in rank order, so a result does not depend on timing.
//
// Grouped form: row tile i of X multiplies matrix tile_group[i] (routed experts on binned rows); only the first n_tiles_dev[0] row tiles
// exist, the CTAs of the others return at once.
#include <cuda.h>

#include <algorithm>

#include "moe_common.cuh"
#include "prof.cuh"
#include "ptx.cuh"
#include "split_gemm.cuh"

namespace kb2 {

constexpr int kSThreads = 128;
constexpr int kSRows = 128;                        // weight rows per tile
constexpr int kSWBytes = kSRows * kBlockK * 2;     // 16 KB of weights per stage
constexpr int kSMaxStages = 12;

struct SplitArgs {
  void* out;
  const float* bias;
  long long ldo;
  int M, N, n_kblocks, nt, stages, chunk, tmem_cols;
  const int* tile_group;
  const int* n_tiles_dev;
};

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_dsmem_f4(uint32_t local_addr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

// KS CTAs of a cluster share one output tile along K.
template <bool kOutF32, int KS>
__global__ void __launch_bounds__(kSThreads)
    split_gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const SplitArgs p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int row_tile = blockIdx.x / KS, rank = blockIdx.x % KS;
  if (p.n_tiles_dev != nullptr && row_tile >= p.n_tiles_dev[0]) return;      // the same decision in every CTA of the cluster
  const int stage_bytes = kSWBytes + p.nt * 128;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + p.stages * stage_bytes);
  uint64_t* empty = full + kSMaxStages;
  uint64_t* done = empty + kSMaxStages;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(done + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int m0 = row_tile * p.nt, n0 = blockIdx.y * kSRows;
  const int w0 = n0 + (p.tile_group != nullptr ? p.tile_group[row_tile] * p.N : 0);        // row of W
  const int kb0 = (int)((long long)p.n_kblocks * rank / KS), kb1 = (int)((long long)p.n_kblocks * (rank + 1) / KS);

  if (threadIdx.x == 32) {
    if (smem_u32(smem) & 1023u) __trap();
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(done, 1);
    fence_mbar_init();
  }
  if (threadIdx.x == 64) {
    prefetch_tmap(&tmap_x);
    prefetch_tmap(&tmap_w);
  }
  if (warp == 0) tmem_alloc(tmem_ptr_smem, p.tmem_cols);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;

  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      mbar_wait(&empty[stage], phase ^ 1);
      uint8_t* a = smem + stage * stage_bytes;
      if (elect_one()) {
        mbar_arrive_expect_tx(&full[stage], stage_bytes);
        tma_load_2d(a, &tmap_w, kb * kBlockK, w0, &full[stage]);
        tma_load_2d(a + kSWBytes, &tmap_x, kb * kBlockK, m0, &full[stage]);
      }
      __syncwarp();
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    int stage = 0;
    uint32_t phase = 0;
    const uint32_t idesc = umma_idesc_bf16_m128(p.nt);
    uint32_t acc = tmem_base;
    int in_chunk = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      mbar_wait(&full[stage], phase);
      tc_fence_after_sync();
      const uint32_t a_addr = smem_u32(smem + stage * stage_bytes);
      const uint64_t ad = umma_desc_k_sw128(a_addr);
      const uint64_t bd = umma_desc_k_sw128(a_addr + kSWBytes);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(acc, ad + 2 * k, bd + 2 * k, idesc, (in_chunk > 0 || k > 0) ? 1u : 0u);
        umma_commit(&empty[stage]);
      }
      __syncwarp();
      if (++in_chunk == p.chunk) { in_chunk = 0; acc += p.nt; }
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
    if (elect_one()) umma_commit(done);
    __syncwarp();
  }
  __syncwarp();
  mbar_wait(done, 0);                              // every load has been consumed: the ring's memory is free
  tc_fence_after_sync();
  float* part = reinterpret_cast<float*>(smem);    // [nt][128]
  const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16);
  const int n_acc = (kb1 - kb0 + p.chunk - 1) / p.chunk;
  for (int c0 = 0; c0 < p.nt; c0 += 16) {
    float v[16];
    uint32_t r[16];
    tmem_ld16(taddr + c0, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
    for (int a = 1; a < n_acc; ++a) {
      tmem_ld16(taddr + a * p.nt + c0, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(r[j]);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) part[(c0 + j) * kSRows + warp * 32 + lane] = v[j];
  }
  tc_fence_before_sync();
  if constexpr (KS > 1) cluster_sync_all(); else __syncthreads();
  // the cluster's CTAs take the tile's rows in turn; a warp writes one row of 128 columns, four per lane
  const int n = n0 + lane * 4;
  if (n < p.N) {                                   // N % 16 == 0 is required by the launcher
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.bias != nullptr) b = make_float4(p.bias[n], p.bias[n + 1], p.bias[n + 2], p.bias[n + 3]);
    const int rows = min(p.nt, p.M - m0);
#pragma unroll 2
    for (int c = rank + KS * warp; c < rows; c += KS * 4) {
      const uint32_t at = smem_u32(part + c * kSRows + lane * 4);
      float4 v[KS];
#pragma unroll
      for (int i = 0; i < KS; ++i) {
        if constexpr (KS > 1) v[i] = ld_dsmem_f4(at, i);
        else v[i] = *reinterpret_cast<const float4*>(part + c * kSRows + lane * 4);
      }
      float4 s = v[0];
#pragma unroll
      for (int i = 1; i < KS; ++i) { s.x += v[i].x; s.y += v[i].y; s.z += v[i].z; s.w += v[i].w; }
      s.x += b.x; s.y += b.y; s.z += b.z; s.w += b.w;
      if constexpr (kOutF32) {
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + (long long)(m0 + c) * p.ldo + n) = s;
      } else {
        uint2 o;
        o.x = bf16x2_bits_rn(s.y, s.x);
        o.y = bf16x2_bits_rn(s.w, s.z);
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + (long long)(m0 + c) * p.ldo + n) = o;
      }
    }
  }
  if constexpr (KS > 1) cluster_sync_all(); else __syncthreads();      // nobody's image goes while a peer still reads it
  if (warp == 0) tmem_dealloc(tmem_base, p.tmem_cols);
}

cudaError_t make_tmap_bf16_rows(void* out_tmap, const void* base, long long rows, long long cols, int box_rows);

template <bool F32, int KS>
static cudaError_t launch_one_split(const CUtensorMap& tx, const CUtensorMap& tw, const SplitArgs& p, dim3 grid, int smem, cudaStream_t s) {
  auto kern = split_gemm_kernel<F32, KS>;
  static PerDeviceOnce once;
  if (const int dev = once.pending(); dev >= 0) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    once.mark(dev);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kSThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = KS;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = KS > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, tx, tw, p);
}

static int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// Depth of the ring: two CTAs share an SM where there are more tiles than SMs and the tile is narrow enough for four stages in half the
// shared memory (nt <= 64); wider tiles run faster alone with a deep ring (N 16384, K 2048, 256 rows in tiles of 128: 25 us with seven
// stages, 32 us with two CTAs of three).
static int ring_stages(int nt, int kb, bool share) {
  const int stage = kSWBytes + nt * 128, room = (share && nt <= 64 ? 113 : 226) * 1024 - 256;
  return std::max(std::min({kSMaxStages, room / stage, kb}), ceil_div((long long)nt * kSRows * 4, stage));
}

// The plan with the least estimated time (us), and whether that beats the 128 x 256 tiles of dense_gemm.cu.  Constants fitted to 700
// timings of M 4..2048 x 14 weight shapes from HBM (the chosen plan is 5 % slower than the best one on average, 20 % at most): an SM takes in
// 190 KB/us, HBM 5.76 MB/us, a 64-wide K block costs 0.135 us of latency at least, reading out a row 0.05 us + 1.2 ns per accumulator, a
// launch 1.9 us.  The 128 x 256 tiles take 0.355 us per K block and 5 us around it.  Measured on both sides of the line: M 1000, N 2048, K 2048
// 12.1 against 18.3 us; M 2048 at the same shape 23.2 against 18.7; M 256, N 12352 21.7 against 23.0; M 515 39.5 against 39.0.
bool split_gemm_plan(int M, int N, int K, bool out_f32, int num_sms, SplitPlan* out) {
  if (M > 2048 || K % kBlockK || N % 16) return false;
  const int nkb = K / kBlockK, nb = ceil_div(N, kSRows);
  static const float kShare[4] = {0.f, 0.45f, 0.55f, 1.0f};
  float best = 0.355f * nkb * ceil_div((long long)ceil_div(M, 128) * ceil_div(N, 256), num_sms) + 5.f;
  bool found = false;
  int last_nt = 0;
  for (int t = ceil_div(M, 256), tries = 0; tries < 8; ++t, ++tries) {
    const int nt = ceil_div(ceil_div(M, t), 16) * 16;
    if (nt == last_nt || (nt < 32 && M > 32)) continue;
    last_nt = nt;
    for (int i = 0; i < 4; ++i) {
      const int ks = 1 << i;
      if (ks > 1 && nkb < 2 * ks) break;
      const int kb = ceil_div(nkb, ks), n_acc = out_f32 ? ceil_div(kb, kSplitChunk) : 1;
      if (n_acc * nt > 512) continue;
      const long long ctas = (long long)ceil_div(M, nt) * nb * ks;
      const int per_sm = ceil_div(ctas, num_sms);
      const float load = (float)per_sm * kb * (kSWBytes + 128 * nt) / 190e3f, hbm = (float)N * K * 2.f / 5.76e6f;
      const float time = std::max({load, hbm, 0.135f * kb}) + nt * (0.05f + 0.0012f * n_acc) * ceil_div(per_sm, 2) +
                         kShare[i] * ceil_div(per_sm, 2) + 1.9f;
      if (time >= best) continue;
      best = time;
      found = true;
      out->nt = nt;
      out->ks = ks;
      out->stages = ring_stages(nt, kb, ctas > num_sms);
      out->chunk = out_f32 ? kSplitChunk : kb;
    }
  }
  return found;
}

SplitPlan split_gemm_binned_plan(int N, int K, bool out_f32, int tile_rows) {
  SplitPlan p;
  p.nt = tile_rows;
  int n_acc = out_f32 ? ceil_div(K / kBlockK, kSplitChunk) : 1;
  while (n_acc > 1 && n_acc * tile_rows > 256) n_acc = ceil_div(n_acc, 2);         // half of the tensor memory, so that two CTAs share an SM
  p.chunk = ceil_div(K / kBlockK, n_acc);
  p.stages = ring_stages(tile_rows, K / kBlockK, true);
  return p;
}

cudaError_t launch_split_gemm(const void* x, const void* w, void* out, const float* bias, int M, int N, int K, long long ldo, bool out_f32,
                              const SplitPlan& plan, const int* tile_group, const int* n_tiles_dev, int groups, cudaStream_t s) {
  KernelSpan span(K_DENSE_BF16, s);
  if (K % kBlockK || N % 16 || M <= 0 || plan.nt < 16 || plan.nt > 256 || plan.nt % 16 || K / kBlockK < plan.ks) return cudaErrorInvalidValue;
  alignas(64) CUtensorMap tx, tw;
  cudaError_t e = make_tmap_bf16_rows(&tx, x, M, K, plan.nt);
  if (e != cudaSuccess) return e;
  e = make_tmap_bf16_rows(&tw, w, (long long)groups * N, K, kSRows);
  if (e != cudaSuccess) return e;
  SplitArgs p{};
  p.out = out;
  p.bias = bias;
  p.ldo = ldo;
  p.M = M;
  p.N = N;
  p.n_kblocks = K / kBlockK;
  p.nt = plan.nt;
  p.stages = plan.stages;
  p.chunk = plan.chunk;
  const int n_acc = plan.chunk > 0 ? ((p.n_kblocks + plan.ks - 1) / plan.ks + plan.chunk - 1) / plan.chunk : 0;
  p.tmem_cols = 32;
  while (p.tmem_cols < n_acc * plan.nt) p.tmem_cols *= 2;
  if (n_acc < 1 || p.tmem_cols > 512) return cudaErrorInvalidValue;
  p.tile_group = tile_group;
  p.n_tiles_dev = n_tiles_dev;
  const int ring = plan.stages * (kSWBytes + plan.nt * 128);
  // a CTA that waits for tensor memory may have cluster peers that others wait for in turn, so co-resident CTAs must never ask for more
  // than the 512 columns together: each takes at least 430 bytes of shared memory per column (1 KB of it is the system's); of 228 KB that
  // leaves fewer than 544 columns, and columns come in multiples of 32
  const int smem = std::max(ring + 2 * kSMaxStages * 8 + 16, p.tmem_cols * 430 - 1024);
  if (plan.stages < 1 || plan.stages > kSMaxStages || ring < plan.nt * kSRows * 4 || smem > 227 * 1024) return cudaErrorInvalidValue;
  const int row_tiles = (M + plan.nt - 1) / plan.nt;
  const dim3 grid(row_tiles * plan.ks, (N + kSRows - 1) / kSRows);
#define KB2_SPLIT(KSV)                                                                  \
  (out_f32 ? launch_one_split<true, KSV>(tx, tw, p, grid, smem, s) : launch_one_split<false, KSV>(tx, tw, p, grid, smem, s))
  switch (plan.ks) {
    case 1: return KB2_SPLIT(1);
    case 2: return KB2_SPLIT(2);
    case 4: return KB2_SPLIT(4);
    case 8: return KB2_SPLIT(8);
    default: return cudaErrorInvalidValue;
  }
#undef KB2_SPLIT
}

}  // namespace kb2
