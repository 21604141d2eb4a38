// Dense product for few rows:  Y[M,N] = X[M,K] x W[N,K]^T with bf16 operands, fp32 accumulation in TMEM, BF16 or FP32 output; and the same for
// fp32 operands, as exact bf16 parts.
//
// Bound: the weights.  Up to a few hundred rows the time is N * K * 2 bytes from HBM, and dense_gemm.cu's 128 x 256 tiles leave most SMs
// without a tile (N = 2048: 8 tiles per 128 rows).  So the roles of the operands are swapped — 128 weight rows are the UMMA's M side, the
// rows of X (any multiple of 16 up to 256) its N side, which costs no padding to 128 rows — and K is cut over the CTAs of a cluster
// (1, 2, 4 or 8).  A CTA has one tile: its TMA ring streams the weights while two CTAs share an SM, so that one fills its ring while the
// other drains.  The partial tiles of a cluster meet in shared memory (one [row][128] fp32 image per CTA, read through distributed shared
// memory); every output is summed in rank order, so a result does not depend on timing, and the plans (below) keep it from depending on the number
// of rows.  From HBM, 77 rows: N 16384, K 2048 15.0 us (11.1 us
// of traffic), N 2048, K 8192 12.6 us (5.4 us), where fp32-FMA tiles took 697 and 449 us.
//
// Grouped form: row tile i of X multiplies matrix tile_group[i] (routed experts on binned rows); only the first n_tiles_dev[0] row tiles
// exist, the CTAs of the others return at once.  Batched form: group g has M rows and a matrix of its own (per-head products).
//
// Gated units: W is [gate ; up], and a tile's 128 weight rows are 64 of each, so a CTA has both numbers of an output and writes the unit itself: the
// pass over a product of 2 F columns and its launch go away (F 8192, K 2048: 9 rows 16.2 -> 14.4 us, 77 rows 17.7 -> 15.7, 255 rows 28.1 -> 26.2).
//
// fp32 operands: x = x1 + x2 + x3 with bf16 parts of 8 bits each, exactly (Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial
// Intelligence Datatype For Higher-Precision Computations", ARITH 2019).  The parts of a tile's rows lie side by side on the N side, so one
// weight tile serves all of them: w x1 goes to the main accumulators, w x2 and w x3 to two small ones.  With fp32 weights in three parts
// too, w1 [x1 x2 x3], w2 [x1 x2] and w3 [x1] are added in: six of the nine products, the other three are below 2^-26 of the result.  512 rows,
// N 16384, K 2048: 222 us (on pairs of CTAs, below; 263 without), 2-norm error 4.7e-7; fp32-FMA tiles 1494 us, 8.1e-7.  Where w2 and w3 are zeros (the fp32 form of a bf16 checkpoint),
// the pass that makes the parts says so per 128 rows x 256 columns; they are then neither written nor loaded nor multiplied: the same sums to
// the last bit, 138 us (175 without pairs; weights of 134 MB among them: 4 bytes of each read, 2 written).
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "moe_common.cuh"
#include "prof.cuh"
#include "ptx.cuh"
#include "seq_act.cuh"
#include "split_gemm.cuh"

namespace kb2 {

// one warp issues copies, one products; all read the accumulators back and write the rows (with four of them 255 rows, N 16384, K 2048 took 24.7 us
// instead of 23.4, and gated units 34.2 instead of 26.2)
constexpr int kSWarps = 8, kSThreads = 32 * kSWarps;
constexpr int kSRows = 128;                        // weight rows per tile
constexpr int kSWBytes = kSRows * kBlockK * 2;     // 16 KB of weights per stage
constexpr int kSMaxStages = 12;

struct SplitArgs {
  void* out;
  const float* bias;
  long long ldo, out_group, w_part_rows;
  int M, N, n_kblocks, mt, xparts, wparts, stages, chunk, tmem_cols, tiles_per_group;
  const uint8_t* w_low;      // wparts 3: [group][tile of 128 rows][low_spans], whether w2 and w3 hold anything in low_span K blocks
  int low_span, low_spans;
  const int* tile_group;
  const int* n_tiles_dev;
  const float* x_raw;
  long long x_ld, x_group;
  const void* w_raw;
  int glu_kind;
  float glu_limit, glu_alpha;
};

__device__ __forceinline__ float4 ld_dsmem_f4(uint32_t local_addr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

// One output from the fp32 operands themselves (see SplitGemm::x_raw).
__device__ __noinline__ float product_again(const float* x, const void* w, long long w0, bool w_f32, int K) {
  float acc = 0.f;
  for (int k = 0; k < K; ++k)
    acc = fmaf(x[k], w_f32 ? reinterpret_cast<const float*>(w)[w0 + k] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w)[w0 + k]), acc);
  return acc;
}

// KS CTAs of a cluster share one output tile along K.
template <bool kOutF32, int KS, bool kGlu>
__global__ void __launch_bounds__(kSThreads)
    split_gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const SplitArgs p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int row_tile = blockIdx.x / KS, rank = blockIdx.x % KS;
  const int nt = p.xparts * p.mt, ring_bytes = p.stages * (p.wparts * kSWBytes + nt * 128);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + ring_bytes);
  uint64_t* empty = full + kSMaxStages;
  uint64_t* done = empty + kSMaxStages;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(done + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  constexpr int kTileCols = kGlu ? kSRows / 2 : kSRows;      // output columns of a tile
  const int n0 = blockIdx.y * kTileCols;
  const int m0 = (p.tiles_per_group > 0 ? row_tile % p.tiles_per_group : row_tile) * p.mt;     // row of the output (of its group)
  const int kb0 = (int)((long long)p.n_kblocks * rank / KS), kb1 = (int)((long long)p.n_kblocks * (rank + 1) / KS);

  if (threadIdx.x == 32) {
    if (smem_u32(smem) & 1023u) __trap();
    for (int i = 0; i < kSMaxStages; ++i) {
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
  pdl_wait();
  if (p.n_tiles_dev != nullptr && row_tile >= p.n_tiles_dev[0]) {            // the same decision in every CTA of the cluster
    if (warp == 0) tmem_dealloc(tmem_base, p.tmem_cols);
    return;
  }
  const int group = p.tile_group != nullptr ? p.tile_group[row_tile] : p.tiles_per_group > 0 ? row_tile / p.tiles_per_group : 0;
  const int w0 = n0 + group * p.N;                                                             // row of W
  // spans of K blocks in which w2 and w3 take part; none: stages without room for them
  uint32_t low = 0;
  if (p.wparts > 1) {
    const uint8_t* said = p.w_low + (long long)(group * gridDim.y + blockIdx.y) * p.low_spans;
    const bool mine = lane >= kb0 / p.low_span && lane <= (kb1 - 1) / p.low_span;
    low = __ballot_sync(0xffffffffu, mine && said[lane] != 0);
  }
  const int w_bytes = low ? 3 * kSWBytes : kSWBytes, stage_bytes = w_bytes + nt * 128, stages = min(kSMaxStages, ring_bytes / stage_bytes);

  int span = low ? kb0 / p.low_span : 0, span_left = (span + 1) * p.low_span - kb0;      // of the K block at hand
  auto next_block = [&]() {
    if (--span_left == 0) {
      ++span;
      span_left = p.low_span;
    }
  };

  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb, next_block()) {
      mbar_wait(&empty[stage], phase ^ 1);
      uint8_t* a = smem + stage * stage_bytes;
      if (elect_one()) {
        const int w_parts = low >> span & 1 ? 3 : 1;
        mbar_arrive_expect_tx(&full[stage], w_parts * kSWBytes + nt * 128);
        if constexpr (kGlu) {
          tma_load_2d(a, &tmap_w, kb * kBlockK, w0, &full[stage]);
          tma_load_2d(a + kSWBytes / 2, &tmap_w, kb * kBlockK, w0 + p.N / 2, &full[stage]);
        } else {
          for (int q = 0; q < w_parts; ++q) tma_load_2d(a + q * kSWBytes, &tmap_w, kb * kBlockK, w0 + (int)(q * p.w_part_rows), &full[stage]);
        }
        tma_load_2d(a + w_bytes, &tmap_x, kb * kBlockK, row_tile * nt, &full[stage]);
      }
      __syncwarp();
      if (++stage == stages) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    int stage = 0;
    uint32_t phase = 0;
    const uint32_t idesc1 = umma_idesc_bf16_m128(p.mt), idesc2 = umma_idesc_bf16_m128(2 * p.mt);
    const uint32_t small = tmem_base;                                        // w x2, w x3 and what the further parts of w bring
    uint32_t acc = tmem_base + (p.xparts > 1 ? 2 * p.mt : 0);                // w x1, a set of columns per chunk
    int in_chunk = 0;
    for (int kb = kb0; kb < kb1; ++kb, next_block()) {
      mbar_wait(&full[stage], phase);
      tc_fence_after_sync();
      const uint32_t a_addr = smem_u32(smem + stage * stage_bytes);
      const uint64_t ad = umma_desc_k_sw128(a_addr);
      const uint64_t bd = umma_desc_k_sw128(a_addr + w_bytes);               // x1; x2 and x3 follow mt rows apart
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(acc, ad + 2 * k, bd + 2 * k, idesc1, (in_chunk > 0 || k > 0) ? 1u : 0u);
        if (p.xparts > 1) {
          const uint64_t bd2 = umma_desc_k_sw128(a_addr + w_bytes + p.mt * 128);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16(small, ad + 2 * k, bd2 + 2 * k, idesc2, (kb > kb0 || k > 0) ? 1u : 0u);
          if (low >> span & 1) {
            const uint64_t ad2 = umma_desc_k_sw128(a_addr + kSWBytes), ad3 = umma_desc_k_sw128(a_addr + 2 * kSWBytes);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_bf16(small, ad2 + 2 * k, bd + 2 * k, idesc2, 1u);             // w2 [x1 x2]
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_bf16(small + p.mt, ad3 + 2 * k, bd + 2 * k, idesc1, 1u);      // w3 x1
          }
        }
        umma_commit(&empty[stage]);
      }
      __syncwarp();
      if (++in_chunk == p.chunk) { in_chunk = 0; acc += p.mt; }
      if (++stage == stages) { stage = 0; phase ^= 1; }
    }
    if (elect_one()) umma_commit(done);
    __syncwarp();
  }
  __syncwarp();
  mbar_wait(done, 0);                              // every load has been consumed: the ring's memory is free
  tc_fence_after_sync();
  float* part = reinterpret_cast<float*>(smem);    // [mt][128]
  const int lanes = warp % 4 * 32;                 // of the tensor memory that this warp can read
  const uint32_t taddr = tmem_base + ((uint32_t)lanes << 16);
  const int n_small = p.xparts > 1 ? 2 : 0, n_sets = (kb1 - kb0 + p.chunk - 1) / p.chunk + n_small;      // the small ones come first
  for (int c0 = warp / 4 * 16; c0 < p.mt; c0 += kSWarps * 4) {
    float v[16];
    uint32_t r[16];
    tmem_ld16(taddr + n_small * p.mt + c0, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
    for (int a = n_small + 1; a < n_sets; ++a) {
      tmem_ld16(taddr + a * p.mt + c0, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(r[j]);
    }
    if (n_small) {                                 // their sum goes in last, as pairs of CTAs add it (parts_pair_kernel)
      uint32_t t[16];
      tmem_ld16(taddr + c0, r);
      tmem_ld16(taddr + p.mt + c0, t);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(r[j]) + __uint_as_float(t[j]);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) part[(c0 + j) * kSRows + lanes + lane] = v[j];
  }
  tc_fence_before_sync();
  if constexpr (KS > 1) cluster_sync_all(); else __syncthreads();
  auto whole = [&](int c, int col) {               // four columns of a row, summed over the cluster's images
    float4 v[KS];
#pragma unroll
    for (int i = 0; i < KS; ++i) {
      if constexpr (KS > 1) v[i] = ld_dsmem_f4(smem_u32(part + c * kSRows + col), i);
      else v[i] = *reinterpret_cast<const float4*>(part + c * kSRows + col);
    }
    float4 s = v[0];
#pragma unroll
    for (int i = 1; i < KS; ++i) { s.x += v[i].x; s.y += v[i].y; s.z += v[i].z; s.w += v[i].w; }
    return s;
  };
  if constexpr (kGlu) {                            // half a warp per row of 64 columns
    const int n = n0 + (lane & 15) * 4, rows = n < p.N / 2 ? min(p.mt, p.M - m0) : 0;
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out) + group * p.out_group + (long long)m0 * p.ldo + n;
    auto write = [&](auto kind) {
      auto unit = [&](float g, float u) { return kb2act::glu_value(bf16_round_rn(g), bf16_round_rn(u), decltype(kind)::value, p.glu_limit, p.glu_alpha); };
#pragma unroll 2
      for (int c = (rank + KS * warp) * 2 + (lane >> 4); c < rows; c += KS * kSWarps * 2) {
        const float4 g = whole(c, (lane & 15) * 4), u = whole(c, 64 + (lane & 15) * 4);
        *reinterpret_cast<uint2*>(out + c * p.ldo) = make_uint2(bf16x2_bits_rn(unit(g.y, u.y), unit(g.x, u.x)), bf16x2_bits_rn(unit(g.w, u.w), unit(g.z, u.z)));
      }
    };
    if (p.glu_kind == 0) write(std::integral_constant<int, 0>{});
    else if (p.glu_kind == 1) write(std::integral_constant<int, 1>{});
    else write(std::integral_constant<int, 2>{});
  } else {
    // the cluster's CTAs take the tile's rows in turn; a warp writes one row of 128 columns, four per lane
    const int n = n0 + lane * 4;
    if (n < p.N) {                                   // N % 16 == 0 is required by the launcher
      float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.bias != nullptr) b = make_float4(p.bias[n], p.bias[n + 1], p.bias[n + 2], p.bias[n + 3]);
      const int rows = min(p.mt, p.M - m0);
      const long long out0 = group * p.out_group + (long long)m0 * p.ldo + n;
#pragma unroll 2
      for (int c = rank + KS * warp; c < rows; c += KS * kSWarps) {
        float4 s = whole(c, lane * 4);
        if (p.x_raw != nullptr && (isnan(s.x) || isnan(s.y) || isnan(s.z) || isnan(s.w))) {
          const float* xr = p.x_raw + group * p.x_group + (long long)(m0 + c) * p.x_ld;
          const int K = p.n_kblocks * kBlockK;
          const long long wr = ((long long)group * p.N + n) * K;
          s.x = product_again(xr, p.w_raw, wr, p.wparts > 1, K);
          s.y = product_again(xr, p.w_raw, wr + K, p.wparts > 1, K);
          s.z = product_again(xr, p.w_raw, wr + 2 * K, p.wparts > 1, K);
          s.w = product_again(xr, p.w_raw, wr + 3 * K, p.wparts > 1, K);
        }
        s.x += b.x; s.y += b.y; s.z += b.z; s.w += b.w;
        if constexpr (kOutF32) {
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + out0 + c * p.ldo) = s;
        } else {
          uint2 o;
          o.x = bf16x2_bits_rn(s.y, s.x);
          o.y = bf16x2_bits_rn(s.w, s.z);
          *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + out0 + c * p.ldo) = o;
        }
      }
    }
  }
  if constexpr (KS > 1) cluster_sync_all(); else __syncthreads();      // nobody's image goes while a peer still reads it
  if (warp == 0) tmem_dealloc(tmem_base, p.tmem_cols);
}

// ---- fp32 operands in parts on pairs of CTAs, for steps that fill the chip
// A tile of split_gemm_kernel holds 80 rows at most (three parts of them are one operand, every chunk has an accumulator), its CTA can neither load
// nor multiply while it reads its accumulators out, and 512 rows x 8192 columns were 448 such tiles on 148 SMs: four rounds for three.  Here a pair of
// CTAs has 256 weight rows and up to 128 rows of X, each CTA half of either, and goes through its tiles one after the other: eight warps take every
// chunk's accumulator (two in turn) into registers while the next chunk runs, so a tile needs four accumulators whatever K is.  The largest products,
// those with x2 and those with x3 go to accumulators of their own, as there; where CTAs of a cluster share K there, tiles are cut into the same segments here, and
// parts_reduce_kernel adds these in the same order: the same sums, bit for bit.
// 512 rows, N 8192, K 2048 in three products: 61 -> 43 us (1.2 PFLOP/s; 128 tiles of 128 rows on 74 pairs are two rounds for 1.73, and under this load the clock
// is that of a cuBLAS product at 1.64 PFLOP/s); N 2048, K 8192 69 -> 42 us and 5 for the segments' sums.
// Per K block of 64 a CTA takes in 16 KB of weights and 24 KB of x for 768 cycles of MMAs (128 rows): [w1 | its half of x1 | x2 (the first CTA) or
// x3], so that one MMA of twice the columns multiplies x2 and x3 (512 rows, N 8192, K 2048: the tensor pipe is active in 0.63 of the cycles, 768 a K block).  Where w2 and w3 hold anything, a second stage [w2 | w3 | halves of x1 | of x2] follows.
constexpr int kPTThreads = 384, kPTWarps = 8, kPTMaxStages = 8, kPTRing = 216 * 1024, kPTSmem = kPTRing + (2 * kPTMaxStages + 6) * 8 + 8;
static_assert(kPTSmem >= tmem_smem(512) && kPTSmem <= 227 * 1024, "what a CTA of a cluster takes for 512 columns");

struct PartsArgs {
  void* out;
  long long ldo, out_group, w_part_rows;
  int M, N, n_kblocks, nt, wparts, chunk, segments, row_tiles, tiles_per_group, w_tiles;
  const uint8_t* w_low;      // [group][tile of 128 rows][low_spans]
  int low_span, low_spans;
  const float* x_raw;
  long long x_ld, x_group;
  const void* w_raw;
  float* partial;            // [segment][group * M + row][N] where there are several, else null
  long long partial_rows;
};

template <bool kOutF32>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPTThreads, 1)
    parts_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const PartsArgs p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kPTRing);        // of the first CTA: both CTAs' loads
  uint64_t* empty = full + kPTMaxStages;
  uint64_t* acc_full = empty + kPTMaxStages;       // [2] a chunk, [2] the two small ones
  uint64_t* acc_empty = acc_full + 3;              // of the first CTA: both CTAs' read-outs
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(acc_empty + 3);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  if (threadIdx.x == 32) {
    if (smem_u32(smem) & 1023u) __trap();
    for (int i = 0; i < kPTMaxStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 3; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 2 * kPTWarps);
    }
    fence_mbar_init();
  }
  if (threadIdx.x == 64) {
    prefetch_tmap(&tmap_x);
    prefetch_tmap(&tmap_w);
  }
  if (warp == 0) tmem_alloc_pair(tmem_ptr_smem, 512);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                              // the other CTA's barriers are there
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  pdl_wait();
  // a unit is a segment of K of a tile: row tiles first, so that neighbours share the weights
  const int tiles = p.w_tiles * p.row_tiles, total = tiles * p.segments, first = blockIdx.x >> 1, step = gridDim.x >> 1;
  const int nt = p.nt, half = nt / 2, tiles128 = (p.N + kSRows - 1) / kSRows;
  // what launch_split_weights says about a span of the K blocks of the 128 rows that CTA r has of tile t
  const auto said = [&](int unit, int r, int span) {
    const int t = unit % tiles, wt = t / p.row_tiles * 2 + r;
    return wt < tiles128 && p.w_low[(long long)(t % p.row_tiles / p.tiles_per_group * tiles128 + wt) * p.low_spans + span] != 0;
  };
  bool any_low = false;                            // of all tiles of the pair: stages then have room for three parts of the weights
  if (p.wparts > 1) {
    for (int i = threadIdx.x; i < (total - first + step - 1) / step * 2 * p.low_spans; i += kPTThreads)
      any_low |= said(first + i / (2 * p.low_spans) * step, i / p.low_spans & 1, i % p.low_spans);
    // broadcasts: what addresses and branches of the MMA loop follow from has to be uniform for the compiler, too
    any_low = __shfl_sync(0xffffffffu, (int)__syncthreads_or(any_low), 0);
  }
  const auto low_of = [&](int t, int r) {
    return any_low ? __shfl_sync(0xffffffffu, __ballot_sync(0xffffffffu, lane < p.low_spans && said(t, r, lane)), 0) : 0u;
  };
  const int bytes1 = kSWBytes + 3 * half * 128, bytes2 = 2 * kSWBytes + 2 * half * 128;
  const int stage_bytes = any_low ? max(bytes1, bytes2) : bytes1, stages = min(kPTMaxStages, kPTRing / stage_bytes);
  const auto seg_begin = [&](int s) { return (int)((long long)p.n_kblocks * s / p.segments); };

  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0;
    for (int unit = first; unit < total; unit += step) {
      const int t = unit % tiles, rt = t % p.row_tiles, group = rt / p.tiles_per_group;
      const int w0 = t / p.row_tiles * 2 * kSRows + (int)rank * kSRows + group * p.N, x0 = rt * 3 * nt;
      const uint32_t own = low_of(unit, rank), both = own | low_of(unit, rank ^ 1);
      for (int kb = seg_begin(unit / tiles), kb1 = seg_begin(unit / tiles + 1); kb < kb1; ++kb) {
        const int span = kb / p.low_span;
        for (int low = 0; low <= (int)(both >> span & 1); ++low) {
          mbar_wait(&empty[stage], phase ^ 1);
          uint8_t* a = smem + stage * stage_bytes;
          if (elect_one()) {
            const uint32_t bar = cluster_addr(&full[stage], 0);
            if (rank == 0) mbar_arrive_expect_tx(&full[stage], 2 * (low ? bytes2 : bytes1));
            if (low == 0) {
              tma_load_2d_pair(a, &tmap_w, kb * kBlockK, w0, bar);
              a += kSWBytes;
              tma_load_2d_pair(a, &tmap_x, kb * kBlockK, x0 + (int)rank * half, bar);
              for (int i = 0; i < 2; ++i) tma_load_2d_pair(a + (1 + i) * half * 128, &tmap_x, kb * kBlockK, x0 + (1 + (int)rank) * nt + i * half, bar);
            } else {
              // parts that are zeros were not written: rows behind the last one read as zeros
              for (int q = 1; q < 3; ++q, a += kSWBytes)
                tma_load_2d_pair(a, &tmap_w, kb * kBlockK, own >> span & 1 ? w0 + (int)(q * p.w_part_rows) : (int)(3 * p.w_part_rows), bar);
              for (int q = 0; q < 2; ++q, a += half * 128) tma_load_2d_pair(a, &tmap_x, kb * kBlockK, x0 + q * nt + (int)rank * half, bar);
            }
          }
          __syncwarp();
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
      }
    }
    for (int i = 0; i < stages; ++i) {             // the last reports of freed stages have arrived, too
      mbar_wait(&empty[stage], phase ^ 1);
      if (++stage == stages) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1 && rank == 0) {
    int stage = 0, b = 0;
    uint32_t phase = 0, taken = 0;                 // a bit per accumulator: the parity of its turn
    const uint32_t idesc = umma_idesc_bf16_m128(nt) + ((128u >> 4) << 24), idesc2 = umma_idesc_bf16_m128(2 * nt) + ((128u >> 4) << 24);      // M = 256
    const uint32_t small = tmem_base + 2 * nt;
    for (int unit = first; unit < total; unit += step) {
      const uint32_t low = low_of(unit, 0) | low_of(unit, 1);
      const int kb0 = seg_begin(unit / tiles), kb1 = seg_begin(unit / tiles + 1);
      for (int kb = kb0, in_chunk = 0; kb < kb1; ++kb) {
        if (in_chunk == 0) {
          mbar_wait(&acc_empty[b], (taken >> b & 1) ^ 1);
          taken ^= 1u << b;
        }
        mbar_wait(&full[stage], phase);
        tc_fence_after_sync();
        const uint32_t a_addr = smem_u32(smem + stage * stage_bytes);
        const uint64_t w1 = umma_desc_k_sw128(a_addr), x1 = umma_desc_k_sw128(a_addr + kSWBytes), x23 = umma_desc_k_sw128(a_addr + kSWBytes + half * 128);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_pair(tmem_base + b * nt, w1 + 2 * k, x1 + 2 * k, idesc, (in_chunk > 0 || k > 0) ? 1u : 0u);
        }
        __syncwarp();
        if (kb == kb0) {
          mbar_wait(&acc_empty[2], (taken >> 2 & 1) ^ 1);
          taken ^= 4u;
          tc_fence_after_sync();
        }
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_pair(small, w1 + 2 * k, x23 + 2 * k, idesc2, (kb > kb0 || k > 0) ? 1u : 0u);
          umma_commit_pair(&empty[stage]);
        }
        __syncwarp();
        if (++stage == stages) { stage = 0; phase ^= 1; }
        if (low >> (kb / p.low_span) & 1) {
          mbar_wait(&full[stage], phase);
          tc_fence_after_sync();
          const uint32_t l_addr = smem_u32(smem + stage * stage_bytes);
          const uint64_t w2 = umma_desc_k_sw128(l_addr), w3 = umma_desc_k_sw128(l_addr + kSWBytes), y1 = umma_desc_k_sw128(l_addr + 2 * kSWBytes),
                         y2 = umma_desc_k_sw128(l_addr + 2 * kSWBytes + half * 128);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_bf16_pair(small, w2 + 2 * k, y1 + 2 * k, idesc, 1u);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_bf16_pair(small + nt, w2 + 2 * k, y2 + 2 * k, idesc, 1u);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_bf16_pair(small + nt, w3 + 2 * k, y1 + 2 * k, idesc, 1u);
            umma_commit_pair(&empty[stage]);
          }
          __syncwarp();
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
        if (elect_one()) {
          if (kb + 1 == kb1) umma_commit_pair(&acc_full[2]);
          if (in_chunk + 1 == p.chunk || kb + 1 == kb1) umma_commit_pair(&acc_full[b]);
        }
        __syncwarp();
        if (++in_chunk == p.chunk || kb + 1 == kb1) {
          in_chunk = 0;
          b ^= 1;
        }
      }
    }
  } else if (warp >= 4) {
    // lane = weight row; the two warps of a quarter of the rows have half the columns (rows of X) each
    constexpr int kCols = 64;
    const int q = warp & 3, c0 = (warp - 4) / 4 * half;
    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + c0;
    uint32_t turns = 0;
    int b = 0;
    const auto take = [&](uint32_t at, int c, uint32_t (&r)[16]) {
      tmem_ld16(at + c, r);
      tmem_ld_wait();
    };
    const auto leave = [&](int which) {            // the accumulator may be written again
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[which], 0));
    };
    for (int unit = first; unit < total; unit += step) {
      const int seg = unit / tiles, t = unit % tiles, blocks = seg_begin(seg + 1) - seg_begin(seg);
      float acc[kCols];
      for (int k = 0; k < blocks; k += p.chunk) {
        mbar_wait(&acc_full[b], turns >> b & 1);
        turns ^= 1u << b;
        tc_fence_after_sync();
#pragma unroll
        for (int c = 0; c < kCols; c += 16)
          if (c < half) {
            uint32_t r[16];
            take(taddr + b * nt, c, r);
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[c + j] = k == 0 ? __uint_as_float(r[j]) : acc[c + j] + __uint_as_float(r[j]);
          }
        leave(b);
        b ^= 1;
      }
      mbar_wait(&acc_full[2], turns >> 2 & 1);
      turns ^= 4u;
      tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < kCols; c += 16)
        if (c < half) {
          uint32_t r[16], u[16];
          tmem_ld16(taddr + 2 * nt + c, r);
          take(taddr + 3 * nt, c, u);
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(r[j]) + __uint_as_float(u[j]);
        }
      leave(2);
      const int rt = t % p.row_tiles, group = rt / p.tiles_per_group, m0 = rt % p.tiles_per_group * nt + c0;
      const int n = t / p.row_tiles * 2 * kSRows + (int)rank * kSRows + q * 32 + lane;
      const int rows = n < p.N ? min(half, p.M - m0) : 0;
      if (p.partial != nullptr) {
        float* to = p.partial + (seg * p.partial_rows + (long long)group * p.M + m0) * p.N + n;
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          if (c >= rows) break;
          to[(long long)c * p.N] = acc[c];
        }
      } else {
        const long long at = group * p.out_group + (long long)m0 * p.ldo + n;
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          if (c >= rows) break;
          if (isnan(acc[c]))
            acc[c] = product_again(p.x_raw + group * p.x_group + (long long)(m0 + c) * p.x_ld, p.w_raw, ((long long)group * p.N + n) * p.n_kblocks * kBlockK,
                                   p.wparts > 1, p.n_kblocks * kBlockK);
          if constexpr (kOutF32) reinterpret_cast<float*>(p.out)[at + c * p.ldo] = acc[c];
          else reinterpret_cast<__nv_bfloat16*>(p.out)[at + c * p.ldo] = __float2bfloat16_rn(acc[c]);
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                              // nobody leaves while the other may still report to its barriers
  tc_fence_after_sync();
  if (warp == 0) tmem_dealloc_pair(tmem_base, 512);
}

// The segments' sums, added in order; four neighbouring columns per thread (N % 16 == 0).  Bound by traffic, from L2.
template <bool kOutF32>
__global__ void __launch_bounds__(256) parts_reduce_kernel(const PartsArgs p) {
  pdl_wait();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x, step = p.partial_rows * p.N;
  const int n4 = p.N / 4, n = (int)(i % n4) * 4;
  const long long r = i / n4;
  if (r >= p.partial_rows) return;
  const float* from = p.partial + r * p.N + n;
  float4 v = *reinterpret_cast<const float4*>(from);
  for (int s = 1; s < p.segments; ++s) {
    const float4 f = *reinterpret_cast<const float4*>(from + s * step);
    v.x += f.x; v.y += f.y; v.z += f.z; v.w += f.w;
  }
  const int group = (int)(r / p.M), K = p.n_kblocks * kBlockK;
  const long long m = r - (long long)group * p.M, at = group * p.out_group + m * p.ldo + n, w0 = ((long long)group * p.N + n) * K;
  const float* x = p.x_raw + group * p.x_group + m * p.x_ld;
  if (isnan(v.x)) v.x = product_again(x, p.w_raw, w0, p.wparts > 1, K);
  if (isnan(v.y)) v.y = product_again(x, p.w_raw, w0 + K, p.wparts > 1, K);
  if (isnan(v.z)) v.z = product_again(x, p.w_raw, w0 + 2 * K, p.wparts > 1, K);
  if (isnan(v.w)) v.w = product_again(x, p.w_raw, w0 + 3 * K, p.wparts > 1, K);
  if constexpr (kOutF32) *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + at) = v;
  else *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + at) = make_uint2(bf16x2_bits_rn(v.y, v.x), bf16x2_bits_rn(v.w, v.z));
}

cudaError_t make_tmap_bf16_rows(void* out_tmap, const void* base, long long rows, long long cols, int box_rows);

template <bool F32, int KS, bool kGlu>
static cudaError_t launch_one_split(const CUtensorMap& tx, const CUtensorMap& tw, const SplitArgs& p, dim3 grid, int smem, cudaStream_t s) {
  auto kern = split_gemm_kernel<F32, KS, kGlu>;
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
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = KS;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = KS > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, tx, tw, p);
}

static int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// Depth of the ring: two CTAs share an SM where there are more tiles than SMs and a stage is small enough for four of them in half the
// shared memory; larger tiles run faster alone with a deep ring (N 16384, K 2048, 256 rows in tiles of 128: 25 us with seven stages,
// 32 us with two CTAs of three).
static int ring_stages(int stage, int mt, int kb, bool share) {
  const int room = (share && 4 * stage <= 112 * 1024 ? 113 : 226) * 1024 - 256;
  return std::max(std::min({kSMaxStages, room / stage, kb}), ceil_div((long long)mt * kSRows * 4, stage));
}

// The plan with the least estimated time (us) among those that cut K over ks CTAs (0: over 1, 2, 4 or 8); false: none fits.  Constants fitted to 700
// timings of M 4..2048 x 14 weight shapes from HBM (the chosen plan is 5 % slower than the best one on average, 20 % at most): an SM takes in
// 190 KB/us, HBM 5.76 MB/us, a 64-wide K block costs 0.135 us of latency at least, reading out a row 0.05 us + 1.2 ns per accumulator, a
// launch 1.9 us.
static bool cheapest(int M, int N, int K, bool whole, int num_sms, int xparts, int wparts, int groups, int ks_only, float* best, SplitPlan* out) {
  const int nkb = K / kBlockK, nb = ceil_div(N, kSRows);
  static const float kShare[4] = {0.f, 0.45f, 0.55f, 1.0f};
  bool found = false;
  for (int i = 0; i < 4; ++i) {
    const int ks = 1 << i;
    if (ks_only ? ks != ks_only : ks > 1 && (whole || nkb < 2 * ks)) continue;
    const int kb = ceil_div(nkb, ks);
    const int chunk = whole ? kb : std::max(nkb <= kSplitChunk ? kSplitChunkShort : kSplitChunk, ceil_div(kb, 30));      // tensor memory holds 32 of 16 rows
    const int sets = ceil_div(kb, chunk) + (xparts > 1 ? 2 : 0);
    const int most = std::min(256 / xparts, 512 / sets) / 16 * 16;
    int last = 0;
    for (int t = ceil_div(M, most), tries = 0; tries < 8; ++t, ++tries) {
      const int mt = ceil_div(ceil_div(M, t), 16) * 16;
      if (mt == last || (mt < 32 && most >= 32 && M > 32 && xparts == 1)) continue;
      last = mt;
      const int stage = wparts * kSWBytes + xparts * mt * 128;
      if (ceil_div((long long)mt * kSRows * 4, stage) * stage > 226 * 1024 - 256) continue;
      const long long ctas = (long long)ceil_div(M, mt) * groups * nb * ks;
      const int per_sm = ceil_div(ctas, num_sms), cols = mt * (xparts == 1 ? 1 : wparts == 1 ? 3 : 6);
      const float load = (float)per_sm * kb * stage / 190e3f, math = (float)per_sm * kb * cols * (2.f / 1700.f);
      const float hbm = (float)N * K * 2.f * wparts * groups / 5.76e6f;
      const float time = std::max({load, math, hbm, 0.135f * kb}) + mt * (0.05f + 0.0012f * sets) * ceil_div(per_sm, 2) +
                         kShare[i] * ceil_div(per_sm, 2) + 1.9f;
      if (time >= *best) continue;
      *best = time;
      found = true;
      out->mt = mt;
      out->ks = ks;
      out->chunk = chunk;
      out->stages = ring_stages(stage, mt, kb, ctas > num_sms);
    }
  }
  return found;
}

// Taken only where the wide tiles of dense_gemm.cu are estimated to take longer (us).  Launches that wait for one another, on both sides of the line (this /
// wide): M 1000, N 2048, K 2048 14.0 / 14.4 us; M 2000 at the same shape 25.2 / 18.2; M 515, N 12288 26.6 / 32.1; M 700 32.2 / 32.0.
bool split_gemm_plan_whole(int M, int N, int K, int num_sms, float us, SplitPlan* out) {
  if (M <= 0 || M > 2048 || K % kBlockK || N % 16) return false;
  // the estimates of `cheapest` are of launches that wait for one another, `us` is of launches in a stream: both fitted at 323 shapes
  float best = (us + 2.1f) / 0.948f;
  return cheapest(M, N, K, true, num_sms, 1, 1, 1, 1, &best, out);
}

// Products of fp32 rows on pairs, cut along K as `out` says, where that is estimated to take less than the plan that is there.  Both estimates (us) are fitted to
// 270 timings of M 33..2048 x 7 weight shapes, bf16 and fp32 weights, from HBM: the chosen form is within 0.8 % of the better one on average.  On both sides of
// the line (tiles of 80 rows / pairs, bf16 weights): N 16384, K 2048: 160 rows 39.9 / 44.5, 200 rows 63.4 / 46.6, 512 rows 109 / 82, 2048 rows 399 / 282; N 2048,
// K 8192: 300 rows 44.0 / 55.8, 400 rows 83.5 / 59.8, 2048 rows 335 / 190; N 4096, K 512: 512 rows 18.4 / 16.9.  Fewer rows than 128 never gained.
static void parts_pair_plan(int M, int N, int K, int num_sms, int wparts, int groups, SplitPlan* out) {
  const int nkb = K / kBlockK, kb = ceil_div(nkb, out->ks);
  const int chunk = nkb <= kSplitChunk ? kSplitChunkShort : std::max(kSplitChunk, ceil_div(kb, 30));
  const size_t partial = parts_partial_bytes(M, N, groups, out->ks);
  if (M < 128 || chunk != out->chunk || partial > kPartialMost) return;
  const int per_sm = ceil_div((long long)ceil_div(M, out->mt) * groups * ceil_div(N, kSRows) * out->ks, num_sms);
  const bool share = per_sm > 1 && 4 * (wparts * kSWBytes + 3 * out->mt * 128) <= 112 * 1024;
  float us = 0.97f * (4.f + per_sm * (share ? 0.75f : 1.f) * (3.5f + 0.41f * kb * (out->mt > 64 ? 1.2f : 1.f)));
  const float hbm = (float)N * K * 2.f * groups / 5.76e6f;
  for (int nt = 128; nt >= 64; nt -= 32) {                     // fewer rows take as long as 64
    const long long units = (long long)ceil_div(N, 2 * kSRows) * ceil_div(M, nt) * groups * out->ks;
    const float rounds = (float)((units + num_sms / 2 - 1) / (num_sms / 2));
    const float block = 4.f * (std::max(89.f, nt * 0.5f) + std::max(89.f, (float)nt)) / 1550.f;      // the two MMAs of a step; what fits the timings
    const float time = 11.5f + std::max(hbm, rounds * (1.5f + kb * block)) + (partial ? 3.f + 2.f * partial / 8e6f : 0.f);
    if (time >= us) continue;
    us = time;
    out->pair = true;
    out->mt = nt;
  }
}

// K is cut as for a step of 64 rows (128 with operands in parts), whatever M is, so that a row's sums do not depend on the rows beside it.  By the
// estimate above that costs nothing at 9..255 rows of 14 weight shapes (at most 4 % but for two of 112 cases), and 3 % on average with parts
// at 9..2048 rows (50 % in the worst case, N 1024, K 2048 at 2048 rows).
bool split_gemm_plan(int M, int N, int K, int num_sms, int xparts, int wparts, int groups, SplitPlan* out) {
  if (M <= 0 || K <= 0 || K % kBlockK || N % 16) return false;
  float best = 1e30f;
  if (!cheapest(xparts > 1 ? 128 : 64, N, K, false, num_sms, xparts, wparts, groups, 0, &best, out)) return false;
  const int ks = out->ks;
  best = 1e30f;
  if (!cheapest(M, N, K, false, num_sms, xparts, wparts, groups, ks, &best, out)) return false;
  if (xparts > 1) parts_pair_plan(M, N, K, num_sms, wparts, groups, out);
  return true;
}

// Tiles of 16 rows sum in chunks, as the products of 9 to 255 rows do; larger ones in one accumulator, as the tiles of 128 rows do: which tile
// of these a run gets changes nothing in its rows.
SplitPlan split_gemm_binned_plan(int K, int tile_rows) {
  const int nkb = K / kBlockK;
  SplitPlan p;
  p.mt = tile_rows;
  p.chunk = tile_rows > 16 ? nkb : std::max(nkb <= kSplitChunk ? kSplitChunkShort : kSplitChunk, ceil_div(nkb, 512 / 16));
  p.stages = ring_stages(kSWBytes + tile_rows * 128, tile_rows, nkb, true);
  return p;
}

static cudaError_t launch_parts_pair(const SplitGemm& g, const SplitPlan& plan, cudaStream_t s) {
  const int tiles = ceil_div(g.M, plan.mt), row_tiles = tiles * g.groups;
  if (g.xparts != 3 || !g.batched || g.tile_group || g.bias || g.glu || !g.x_raw || !g.w_raw || plan.mt % 32 || plan.mt > 128 || plan.chunk < 1 || plan.ks < 1 ||
      (plan.ks > 1 && !g.partial) || (g.wparts != 1 && (g.wparts != 3 || !g.w_low)))
    return cudaErrorInvalidValue;
  alignas(64) CUtensorMap tx, tw;
  cudaError_t e = make_tmap_bf16_rows(&tx, g.x, (long long)row_tiles * 3 * plan.mt, g.K, plan.mt / 2);
  if (e != cudaSuccess) return e;
  e = make_tmap_bf16_rows(&tw, g.w, (long long)g.wparts * g.groups * g.N, g.K, kSRows);
  if (e != cudaSuccess) return e;
  PartsArgs p{};
  p.out = g.out;
  p.ldo = g.ldo;
  p.out_group = g.out_group;
  p.w_part_rows = (long long)g.groups * g.N;
  p.M = g.M;
  p.N = g.N;
  p.n_kblocks = g.K / kBlockK;
  p.nt = plan.mt;
  p.wparts = g.wparts;
  p.chunk = plan.chunk;
  p.segments = plan.ks;
  p.row_tiles = row_tiles;
  p.tiles_per_group = tiles;
  p.w_tiles = ceil_div(g.N, 2 * kSRows);
  p.w_low = g.w_low;
  p.low_span = split_low_span(g.N, g.K, g.groups);
  p.low_spans = ceil_div(p.n_kblocks, p.low_span);
  p.x_raw = g.x_raw;
  p.x_ld = g.x_ld;
  p.x_group = g.x_group;
  p.w_raw = g.w_raw;
  p.partial = plan.ks > 1 ? g.partial : nullptr;
  p.partial_rows = (long long)g.groups * g.M;
  const int pairs = (int)std::min<long long>((long long)p.w_tiles * row_tiles * plan.ks, current_sms() / 2);
  const unsigned blocks = (unsigned)((p.partial_rows * (g.N / 4) + 255) / 256);
  const auto run = [&](auto f32) {
    constexpr bool kF32 = decltype(f32)::value;
    cudaError_t r = allow_smem<parts_pair_kernel<kF32>>(kPTSmem);
    if (r == cudaSuccess) r = launch_pdl(parts_pair_kernel<kF32>, dim3(2 * pairs), dim3(kPTThreads), kPTSmem, s, tx, tw, p);
    if (r == cudaSuccess && plan.ks > 1) r = launch_pdl(parts_reduce_kernel<kF32>, blocks, 256, 0, s, p);
    return r;
  };
  return g.out_f32 ? run(std::true_type{}) : run(std::false_type{});
}

cudaError_t launch_split_gemm(const SplitGemm& g, const SplitPlan& plan, cudaStream_t s) {
  KernelSpan span(K_DENSE_BF16, s);
  const int nkb = g.K / kBlockK, nt = g.xparts * plan.mt;
  if (g.K % kBlockK || g.N % 16 || g.M <= 0 || g.groups <= 0) return cudaErrorInvalidValue;
  if (plan.pair) return launch_parts_pair(g, plan, s);
  if (plan.mt < 16 || nt > 256 || plan.mt % 16 || plan.ks < 1 || nkb < plan.ks ||
      plan.chunk < 1 || (g.xparts != 1 && g.xparts != 3) || (g.wparts != 1 && g.wparts != g.xparts))
    return cudaErrorInvalidValue;
  const int tiles = ceil_div(g.M, plan.mt), row_tiles = g.batched ? tiles * g.groups : tiles;
  alignas(64) CUtensorMap tx, tw;
  // three parts: whole tiles of zero-padded rows; else the caller's M rows (rows beyond them read as zeros)
  cudaError_t e = make_tmap_bf16_rows(&tx, g.x, g.xparts > 1 ? (long long)row_tiles * nt : (long long)g.M, g.K, nt);
  if (e != cudaSuccess) return e;
  e = make_tmap_bf16_rows(&tw, g.w, (long long)g.wparts * g.groups * g.N, g.K, g.glu ? kSRows / 2 : kSRows);
  if (e != cudaSuccess) return e;
  SplitArgs p{};
  p.out = g.out;
  p.bias = g.bias;
  p.ldo = g.ldo;
  p.out_group = g.batched ? g.out_group : 0;
  p.w_part_rows = (long long)g.groups * g.N;
  p.M = g.M;
  p.N = g.N;
  p.n_kblocks = nkb;
  p.mt = plan.mt;
  p.xparts = g.xparts;
  p.wparts = g.wparts;
  p.stages = plan.stages;
  p.chunk = plan.chunk;
  const int sets = ceil_div(ceil_div(nkb, plan.ks), plan.chunk) + (g.xparts > 1 ? 2 : 0);
  p.tmem_cols = 32;
  while (p.tmem_cols < sets * plan.mt) p.tmem_cols *= 2;
  if (p.tmem_cols > 512) return cudaErrorInvalidValue;
  p.tiles_per_group = g.batched ? tiles : 0;
  p.tile_group = g.tile_group;
  p.n_tiles_dev = g.n_tiles_dev;
  p.x_raw = g.xparts > 1 ? g.x_raw : nullptr;
  p.x_ld = g.x_ld;
  p.x_group = g.x_group;
  p.w_raw = g.w_raw;
  p.w_low = g.w_low;
  p.glu_kind = g.glu_kind;
  p.glu_limit = g.glu_limit;
  p.glu_alpha = g.glu_alpha;
  if (g.glu && (g.out_f32 || g.xparts != 1 || g.bias != nullptr || g.N % 32)) return cudaErrorInvalidValue;
  p.low_span = split_low_span(g.N, g.K, g.groups);
  p.low_spans = ceil_div(nkb, p.low_span);
  if (g.wparts > 1 && g.w_low == nullptr) return cudaErrorInvalidValue;
  const int ring = plan.stages * (g.wparts * kSWBytes + nt * 128);
  const int smem = std::max(ring + 2 * kSMaxStages * 8 + 16, tmem_smem(p.tmem_cols));
  if (plan.stages < 1 || plan.stages > kSMaxStages || ring < plan.mt * kSRows * 4 || smem > 227 * 1024) return cudaErrorInvalidValue;
  const dim3 grid(row_tiles * plan.ks, ceil_div(g.glu ? g.N / 2 : g.N, g.glu ? kSRows / 2 : kSRows));
#define KB2_SPLIT(KSV)                                                                                                                                \
  (g.glu ? launch_one_split<false, KSV, true>(tx, tw, p, grid, smem, s) : g.out_f32 ? launch_one_split<true, KSV, false>(tx, tw, p, grid, smem, s) \
                                                                                   : launch_one_split<false, KSV, false>(tx, tw, p, grid, smem, s))
  switch (plan.ks) {
    case 1: return KB2_SPLIT(1);
    case 2: return KB2_SPLIT(2);
    case 4: return KB2_SPLIT(4);
    case 8: return KB2_SPLIT(8);
    default: return cudaErrorInvalidValue;
  }
#undef KB2_SPLIT
}

// ------------------------------------------------------------------------------------------------ fp32 -> three bf16 parts
// hi = bf16(v), mid = bf16(v - hi), lo = v - hi - mid: nearest rounding leaves 9 + 9 bits behind, so 24 bits are carried exactly (a value next
// to the largest fp32 number is truncated instead of rounded to infinity; what is not finite goes into hi alone).  bf16 numbers end at 2^-133: below 1e-33 the low parts miss up to 2^-134.
__device__ __forceinline__ void split3(float v, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const uint32_t bits = __float_as_uint(v), e = bits & 0x7F800000u;
  hi = bf16_bits_rn(v);
  if (e != 0x7F800000u && (hi & 0x7F80u) == 0x7F80u) hi = bits >> 16;
  float r = v - __uint_as_float(hi << 16);
  if (e == 0x7F800000u) r = 0.f;
  mid = bf16_bits_rn(r);
  lo = bf16_bits_rn(r - __uint_as_float(mid << 16));
}

// Bound by traffic (4 bytes in, 6 out); a thread takes eight neighbouring columns.
template <bool kVec>
__global__ void __launch_bounds__(256) split_parts_kernel(const float* __restrict__ x, long long ld, long long group_stride, int rows, int K, int mt,
                                                          int tiles, long long total, __nv_bfloat16* __restrict__ parts) {
  pdl_enter(x, parts);
  const int k8 = K >> 3;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
    const long long r = i / k8;                      // row of the padded [groups][tiles][mt] order
    const int c = (int)(i - r * k8) * 8;
    const long long tile = r / mt;
    const int in = (int)(r - tile * mt), group = (int)(tile / tiles), row = (int)(tile - (long long)group * tiles) * mt + in;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.f;
    if (row < rows) {
      const float* src = x + group * group_stride + (long long)row * ld + c;
      if constexpr (kVec) {
        const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = src[j];
      }
    }
    uint32_t o[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t a[3], b[3];
      split3(v[2 * j], a[0], a[1], a[2]);
      split3(v[2 * j + 1], b[0], b[1], b[2]);
#pragma unroll
      for (int q = 0; q < 3; ++q) o[q][j] = a[q] | (b[q] << 16);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q)
      *reinterpret_cast<uint4*>(parts + ((tile * 3 + q) * mt + in) * K + c) = make_uint4(o[q][0], o[q][1], o[q][2], o[q][3]);
  }
}

// The parts of weights, [3][groups * N][K].  A block makes those of 128 rows x `cols` columns; it writes the low ones only if one of them is not
// zero (usually seen in its first round, or else in a second pass over what it has just read) and says so in `low`.
template <bool kVec>
__global__ void __launch_bounds__(512) split_weight_parts_kernel(const float* __restrict__ w, int N, int K, long long all_rows, int tiles, int cols, int spans,
                                                                 __nv_bfloat16* __restrict__ parts, uint8_t* __restrict__ low) {
  pdl_enter(w, parts, low);
  const int span = blockIdx.x % spans, gt = blockIdx.x / spans, group = gt / tiles, n0 = gt % tiles * 128, c0 = span * cols;
  const int k8 = min(cols, K - c0) >> 3, total = min(128, N - n0) * k8;
  const long long first = (long long)group * N + n0;
  bool any = false, write = false;
  for (int pass = 0; pass < 2; ++pass) {
    for (int base = 0; base < total; base += 512) {
      const int i = base + threadIdx.x;
      const long long at = (first + i / k8) * K + c0 + i % k8 * 8;
      float v[8];
      uint32_t o[3][4];
      if (i < total) {
        const float* src = w + at;
        if constexpr (kVec) {
          const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
          v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = src[j];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t a[3], b[3];
          split3(v[2 * j], a[0], a[1], a[2]);
          split3(v[2 * j + 1], b[0], b[1], b[2]);
#pragma unroll
          for (int q = 0; q < 3; ++q) o[q][j] = a[q] | (b[q] << 16);
          any |= (o[1][j] | o[2][j]) != 0;
        }
        if (pass == 0) *reinterpret_cast<uint4*>(parts + at) = make_uint4(o[0][0], o[0][1], o[0][2], o[0][3]);
      }
      if (pass == 0 && base == 0) write = __syncthreads_or(any);
      if (write && i < total)
#pragma unroll
        for (int q = 1; q < 3; ++q) *reinterpret_cast<uint4*>(parts + q * all_rows * K + at) = make_uint4(o[q][0], o[q][1], o[q][2], o[q][3]);
    }
    if (write || !__syncthreads_or(any)) break;
    write = true;                                    // seen later on: once more for the low parts
  }
  if (threadIdx.x == 0) low[blockIdx.x] = write;
}

cudaError_t launch_split_weights(const float* w, int N, int K, int groups, void* parts, uint8_t* low, cudaStream_t s) {
  KernelSpan span(K_DENSE_BF16, s);
  const int tiles = ceil_div(N, kSRows), cols = split_low_span(N, K, groups) * kBlockK, spans = ceil_div(K, cols);
  const unsigned blocks = (unsigned)groups * tiles * spans;
  auto kern = (uintptr_t)w & 15 ? split_weight_parts_kernel<false> : split_weight_parts_kernel<true>;
  return launch_pdl(kern, blocks, 512, 0, s, w, N, K, (long long)groups * N, tiles, cols, spans, (__nv_bfloat16*)parts, low);
}

cudaError_t launch_split_parts(const float* x, long long ld, long long group_stride, int rows, int K, int mt, int groups, void* parts,
                               int num_sms, cudaStream_t s) {
  KernelSpan span(K_DENSE_BF16, s);
  const int tiles = ceil_div(rows, mt);
  const long long total = (long long)groups * tiles * mt * (K / 8);
  const unsigned blocks = (unsigned)std::min<long long>((total + 255) / 256, num_sms * 16);
  const bool vec = !((uintptr_t)x & 15) && ld % 4 == 0 && group_stride % 4 == 0;
  if (vec) launch_pdl(split_parts_kernel<true>, blocks, 256, 0, s, x, ld, group_stride, rows, K, mt, tiles, total, (__nv_bfloat16*)parts);
  else launch_pdl(split_parts_kernel<false>, blocks, 256, 0, s, x, ld, group_stride, rows, K, mt, tiles, total, (__nv_bfloat16*)parts);
  return cudaGetLastError();
}

}  // namespace kb2
