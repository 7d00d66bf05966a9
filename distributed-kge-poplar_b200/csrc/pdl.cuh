// Programmatic dependent launch for the kernels of a training step.
//
// A step is a chain of short kernels, each a few microseconds long, so the time between the end
// of one kernel and the first instruction of the next is a large part of the step.  Launched with
// the programmatic-serialisation attribute, a kernel's blocks may become resident (parameters
// loaded, shared memory carved, barriers initialised) while the predecessor in the stream still
// runs.  The kernel then calls grid_dependency_sync() before it touches global memory: that waits
// for the predecessor to complete with its writes visible, and then lets this kernel's own
// successor begin to launch, so at most one successor is resident and waiting at any time.
// Before that call a kernel may read what was written by the kernels ahead of its predecessor: all
// of the predecessor's blocks have passed their own wait by then, so those are complete.  (k_loss
// reads its labels and k_lookup its index streams there; prefetches into L2 are open too.)
//
// Every kernel launched with the attribute must call grid_dependency_sync() in every block that
// does not return at once: completion of kernel N then implies completion of kernel N-1, which is
// what makes a chain of such launches behave like plain stream order.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

namespace kge {

#ifdef __CUDACC__
__device__ __forceinline__ void grid_dependency_sync() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

// State that CUDA keeps per device (function attributes, occupancy answers) is cached per device:
// the slot of the current device, or -1 when it cannot be cached (then the caller asks CUDA again).
constexpr int kMaxDeviceOrdinals = 64;
inline int current_device_slot() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDeviceOrdinals) return -1;
    return device;
}

// Process-wide switch (on by default; KGE_NO_DEPENDENT_LAUNCH=1 in the environment turns it off).
bool dependent_launch_enabled();

// kernel<<<grid, block, smem, stream>>>(args...) with the attribute when enabled; cluster_z > 1
// also makes every cluster_z blocks that are neighbours in z one thread-block cluster.
template <typename... Params, typename... Args>
inline cudaError_t launch_dependent_cluster(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                            unsigned cluster_z, Args&&... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    unsigned n = 0;
    if (dependent_launch_enabled()) {
        attribute[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attribute[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    if (cluster_z > 1) {
        attribute[n].id = cudaLaunchAttributeClusterDimension;
        attribute[n].val.clusterDim.x = 1;
        attribute[n].val.clusterDim.y = 1;
        attribute[n].val.clusterDim.z = cluster_z;
        ++n;
    }
    config.attrs = attribute;
    config.numAttrs = n;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

template <typename... Params, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                    Args&&... args) {
    return launch_dependent_cluster(kernel, grid, block, smem, stream, 1u, static_cast<Args&&>(args)...);
}

// A launch whose blocks are spread evenly over the SMs.  A dependent kernel's blocks are placed while its predecessor still
// runs, on whatever SM has room for them first, and where an SM has room for eight a grid of 512 small blocks ends up on
// half of the SMs.  Unused shared memory leaves each SM room for its share of the blocks and no more.  (The loss and the
// lookups of a step launched this way: RotatE with features 88.2 to 86.1 us a step, ComplEx 76.4 to 74.6.  Kernels whose
// blocks are long enough to be dealt out as others end, as the pair gradients, gained nothing or lost.)
constexpr int kSmCount = 148;
template <auto Kernel, typename... Args>
inline cudaError_t launch_spread(dim3 grid, dim3 block, cudaStream_t stream, Args&&... args) {
    // The blocks of an SM without the unused memory (high half, 0: not asked yet) and a block's static memory, in one word:
    // engines on several threads ask and answer here.
    static std::atomic<uint64_t> known[kMaxDeviceOrdinals] = {};
    const int slot = current_device_slot();
    uint64_t answer = slot >= 0 ? known[slot].load() : 0;
    if (answer == 0) {
        cudaFuncAttributes attributes;
        int blocks = 0;
        cudaError_t err = cudaFuncGetAttributes(&attributes, Kernel);
        if (err == cudaSuccess) err = cudaFuncSetAttribute(Kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (err == cudaSuccess) err = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - (int)attributes.sharedSizeBytes);
        if (err == cudaSuccess) err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, Kernel, (int)(block.x * block.y * block.z), 0);
        if (err != cudaSuccess) return err;
        answer = (uint64_t)blocks << 32 | (uint32_t)attributes.sharedSizeBytes;
        if (slot >= 0) known[slot].store(answer);
    }
    const int natural = (int)(answer >> 32), static_bytes = (int)(uint32_t)answer;
    const int share = (int)(((long long)grid.x * grid.y * grid.z + kSmCount - 1) / kSmCount);
    // a block takes its memory and 1 KB of the SM's 228: so much that share + 1 blocks do not fit (an empty grid is CUDA's to refuse)
    int unused = 0;
    if (share > 0 && share < natural) unused = std::min(228 * 1024 / (share + 1) + 128, 228 * 1024 / share) - 1024 - static_bytes;
    unused = std::max(0, std::min(unused, 227 * 1024 - static_bytes)) / 128 * 128;
    return launch_dependent(Kernel, grid, block, (size_t)unused, stream, static_cast<Args&&>(args)...);
}
// That memory keeps kernels of other streams off the SM too: the lookups and the loss of shards that run side by side, each on
// a stream, are not spread (us a step, spread -> not: four shards of 256 x 320 x 10 L1 scores 60 -> 55, of 64 columns 62 -> 57).
// In the step of separate kernels the loss of one shard is spread for TransH alone (512 x 768 x 50: 137, 150 without), not in
// front of L1 gradients, whose blocks stay where its blocks have left room (512 x 768 x 63: 76 -> 74; its lookups not spread, 87).
template <auto Kernel, typename... Args>
inline cudaError_t launch_spread_if(bool spread, dim3 grid, dim3 block, cudaStream_t stream, Args&&... args) {
    if (!spread) return launch_dependent(Kernel, grid, block, 0, stream, static_cast<Args&&>(args)...);
    return launch_spread<Kernel>(grid, block, stream, static_cast<Args&&>(args)...);
}

}  // namespace kge
