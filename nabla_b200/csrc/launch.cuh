// Launches that follow each other closely. A kernel that starts with follow_grid() and is launched by launch_following() is
// resident, with its set-up done, before the launch ahead of it in the stream has ended: its blocks take the SMs as that
// one's leave them, and the start of a grid lies under the last blocks ahead of it. Captured steps, us before and after: a
// transformer block of 2 x 1001 x 512 199 and 184, four layers of 4 x 333 x 512 257 and 241, two small layers and their Adam
// 61.5 and 55.9, three attention kernels of 8 x 12 heads x 777 209 and 200; from a tape: an adapter's step at 2048 141 and 130.
//
// Rules that keep this the order of the stream:
//  - nothing in global memory is read or written before follow_grid() (nor loaded into shared memory); it returns when every
//    grid ahead has ended and its writes are visible. All blocks call it, on every path out of the kernel.
//  - pointers that a kernel takes as parameters and reads through go in as arguments of follow_grid(). What lies behind a `const T*
//    __restrict__` counts as constant for the whole kernel, so the compiler may read it ahead of the wait, and by the load for constants,
//    whose lines the wait need not drop; the pointers that come back from it are no longer known to be those. (Members of a
//    struct parameter never were.) They are still known to point to global memory: as pointers to anywhere, their loads were not moved ahead of
//    stores to shared memory, and of 220 convolutions and filter gradients each in chains those took 1.07 and 1.18 times as long
//    (16 x 7 x 7 x 24 -> 64, 3 x 3, 13.4 us and 18.9).
//  - only then does it let the next launch begin, so no more than two grids of a stream are on the chip. A kernel that takes
//    tensor memory has it by then: a waiting block may wait for the tensor memory of a running one, never the other way.
//  - a kernel without follow_grid() is launched with <<< >>> and waits for the end of all that is ahead of it, as before.
// Two exceptions, and what they rest on:
//  - kernels with bounded waits look at the device's status word while they set up, half a microsecond that a launch would otherwise
//    pay behind its wait. They see it as of then: the launch right behind one whose wait ran out may still start, and meets the limits
//    of its own waits; the one behind it leaves. Nothing else follows from the word on the device.
//  - attn_bwd_dq_kernel, unless it reads a mask of a row per query, works and lets the next launch begin before it has waited. The kernel ahead of it, dK / dV,
//    writes nothing that it reads and reads nothing that it writes, and begins it only behind its own wait, so all that came before is
//    complete; what it reads goes past L1; and its blocks wait before they end, so whoever waits for it has dK and dV too. Three grids
//    are on the chip then. A second kernel of this kind directly behind it would not have that ground to stand on.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace nb {

__device__ __forceinline__ void wait_for_previous_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_grid_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename Pointer>
__device__ __forceinline__ void as_of_now(Pointer& p) {
  size_t global = __cvta_generic_to_global(p);
  asm volatile("" : "+l"(global) : : "memory");
  p = static_cast<Pointer>(__cvta_global_to_generic(global));
}
// `early` false, for every block of a grid: the next launch begins as these blocks end, which counts as much as saying so. Thousands of small blocks
// spend up to a third of their time on saying so. us in chains, before launches followed each other, with every block saying so, and by ending:
// layer norm of 40000 x 64 fp32 9.0, 11.2, 8.4; 11368 rows of 256 fp32 from a table 8.2, 13.1, 7.2; gradient of the cross-entropy of 6410 x 100 bf16 5.8, 8.0, 5.4.
constexpr unsigned MANY_BLOCKS = 2048;
template <typename... Pointers>
__device__ __forceinline__ void follow_grid_when(bool early, Pointers&... read) {
  wait_for_previous_grid();
  if (early) let_next_grid_start();
  (as_of_now(read), ...);
}
template <typename... Pointers>
__device__ __forceinline__ void follow_grid(Pointers&... read) { follow_grid_when(true, read...); }

// Adds the attribute to a launch whose attribute array has room for one more.
inline void set_following(cudaLaunchConfig_t& cfg) {
  cudaLaunchAttribute& a = cfg.attrs[cfg.numAttrs++];
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
}

// A kernel with follow_grid() may also be launched behind all that is ahead of it (`following` false). Blocks that start in the room that running ones
// leave are not spread evenly: where a grid is less than the SMs could hold, some of them get several blocks and others none, and a
// kernel that runs for long then pays more than the start of a launch.
template <typename... Params, typename... Args>
inline cudaError_t launch_when(bool following, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  if (following) set_following(cfg);
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
template <typename... Params, typename... Args>
inline cudaError_t launch_following(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  return launch_when(true, kernel, grid, block, smem, stream, std::forward<Args>(args)...);
}

}  // namespace nb
