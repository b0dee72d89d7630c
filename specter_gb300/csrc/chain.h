// Launches that the GPU prepares while the kernel before them in the stream still runs (programmatic
// dependent launch): their blocks start as its last ones end, and what a kernel does before chain_wait()
// overlaps the flush of its predecessor's writes.  For chains of short kernels: six launches of a 32 x 32 x 58
// transform 19.5 -> 15.7 us, a channel step at 64 x 64 x 90 1.5 % faster.  (Letting the next kernel's blocks in
// before the previous one's end costs 3 % at 256^2 x 257: blocks that wait hold the room of blocks that work.)
#pragma once

#include <utility>

#include <cuda_runtime.h>

namespace sg {

// The first thing of a chained kernel that touches what earlier kernels read or wrote: returns when they have
// completed and their writes are visible.  Every thread of every block executes it, so a kernel's end
// implies its predecessor's.
__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

constexpr unsigned kSMs = 152;

// Only launches of one wave gain; larger ones measured the same or up to 3 % slower (128^2 x 154 to physical
// space, 126 -> 129 us), so they are ordinary launches.
constexpr unsigned long long kChainBlocks = 3 * kSMs;

template <typename... P, typename... A>
void chain(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    c.attrs = &at;
    c.numAttrs = 1ull * grid.x * grid.y * grid.z <= kChainBlocks;
    cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);  // errors surface at the caller's check_launch
}

}  // namespace sg
