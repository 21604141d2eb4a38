// Programmatic dependent launches: a kernel's blocks come up as the last blocks of the kernel ahead of it in the stream leave, do what needs no
// input (barriers, tensor memory, descriptors) and wait for it to have ended and written everything, before they touch anything it may have
// written.  Between plain launches the chip stands idle for 1 to 2 us; small steps are chains of dozens of them.  us per call, plain launches
// and these: 3 tokens through 8 of 256 experts (6 launches) 55.8 / 43, a latent-attention layer of 1000 tokens (6) 79.3 / 68.7, 128 tokens
// through routed bf16 experts (11) 211 / 188, a captured decode step of 4 requests (46) 254 / 244.
// Some kernels let the next one come up when their own wait is over (pdl_trigger): those of few registers and next to no shared memory that many short steps run
// (residual norms, gates, the join of latent attention's pieces), and the delta rule's decode step (256 threads of 128 registers, 10 KB, a block per token and head:
// what it leaves of an SM is room for the next): a serving run of 4 requests 4880 -> 4765 us.  The others do not: with that at the start of
// every kernel waiting blocks took slots for whole kernels, and 8192 tokens through routed experts took 734 us instead of 720, 389 tokens 144 instead of
// 137, the decode step 262.  Bringing the waiting products' weights into L2 meanwhile gained nothing (4720; all of a product's weights at once 4880).
// Rules that keep this safe:
//   - a kernel launched with launch_pdl calls pdl_enter (or pdl_wait) in every block, ahead of its first access to global memory.  So when it
//     ends, everything ahead of it in the stream has ended too, and a wait for the neighbour is a wait for all;
//   - nothing is read ahead of the wait, not even weights: the kernel ahead may be the one that writes them;
//   - a block that waits for tensor memory waits for a block of the kernel ahead, which waits for nobody behind it: the blocks of a kernel
//     come up only when all blocks of the one ahead have theirs.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace kb2 {

// Waits for the kernel ahead in the stream.  Returns zero, in a way that the compiler cannot see.
__device__ __forceinline__ long long pdl_wait() {
  long long zero;
  asm volatile("griddepcontrol.wait;\n\tmov.u64 %0, 0;" : "=l"(zero)::"memory");
  return zero;
}
// Lets the next kernel in the stream come up now, as soon as every block of this one has said so or left.  Behind the kernel's own wait.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// pdl_wait for a kernel with the pointers p: loads through a __restrict__ pointer may otherwise move ahead of the wait, so each of them gets the
// wait's zero added.
template <typename... P>
__device__ __forceinline__ void pdl_enter(P&... p) {
  const long long zero = pdl_wait();
  ((p = (P)((const char*)p + zero)), ...);
}
// The same for kernels that the compiler would otherwise address through generic pointers; in exchange it no longer knows that they are __restrict__.
// Whichever is faster (us with plain pointers, with pdl_enter, with this: moe_gemv 26.6 / 30.3 / 26.5, attn_finish 40.6 / 47.2 / 39.6, gla_reg 102 / 104 /
// 100, delta_out_rows 23.4 / 24.1 / 21.7; but rmsnorm_warp 10.5 / 10.4 / 15.3, scatter 19.4 / 19.3 / 23.3).  Either takes registers for pointers that plain
// ones read from the constant bank: gqa_prep went from 32 to 48 of them, five blocks on an SM instead of eight, 27.5 -> 34 us until its launch bounds said so.
template <typename... P>
__device__ __forceinline__ void pdl_enter_global(P&... p) {
  const size_t zero = (size_t)pdl_wait();
  ((p = (P)__cvta_global_to_generic(__cvta_generic_to_global((const void*)p) + zero)), ...);
}

// The kernel in clusters of `cluster` blocks.
template <typename... P, typename... A>
inline cudaError_t launch_pdl_clusters(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, dim3 cluster, A&&... args) {
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster.x;
  at[1].val.clusterDim.y = cluster.y;
  at[1].val.clusterDim.z = cluster.z;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = cluster.x * cluster.y * cluster.z > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  return launch_pdl_clusters(kernel, grid, block, smem, s, dim3(1, 1, 1), std::forward<A>(args)...);
}

}  // namespace kb2
