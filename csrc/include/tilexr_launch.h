// Kernel launch service of the core runtime, used by every operator library.
//
// A kernel is described by a KernelEntry with two entry points compiled from the same device
// body: `single` takes the argument struct by value and runs one rank; `emulated` takes a
// device array of argument structs, one per rank, and runs rank blockIdx.y, so that a whole
// emulated world (several ranks on ONE GPU) is a single cooperative launch.  Kernels whose
// blocks wait for one another, or for peers, are launched cooperatively: the launch fails
// with an error instead of deadlocking when the grid cannot be co-resident.
//
// (The reference registers device binaries and launches them by signature,
// src/collectives/host/collective_kernel.cpp:97-223; on CUDA the function pointer is enough.)
#ifndef TILEXR_LAUNCH_H
#define TILEXR_LAUNCH_H

#include <stddef.h>
#include <stdint.h>
#ifdef __cplusplus
#include <functional>
#endif

#include "tilexr_api.h"

namespace TileXR {

constexpr int EMULATED_INLINE_RANKS = 8;
constexpr size_t EMULATED_HEADER_BYTES = 16;

struct KernelEntry {
    const void *single;
    const void *emulated;
    size_t argBytes;
    const char *name;
    // How `emulated` takes its argument structs: up to this many ranks inside the launch's parameters (EmulatedArgs), zero: always a
    // device array, which every launch allocates, uploads and frees.
    int inlineRanks = 0;
};

struct LaunchConfig {
    unsigned grid;        // blocks per rank
    unsigned block;       // threads per block
    size_t smemBytes;     // dynamic shared memory
    bool cooperative;     // blocks of the grid wait on one another
    bool overlap = false; // the kernel calls StreamWait (device/tilexr_platform.cuh): it may start before its predecessor has ended
};

// Launches `kernel` for `comm`'s rank on `stream`.  On an emulated communicator the call is
// recorded and issued by TileXRGroupEnd together with the other ranks' calls.
int LaunchKernel(TileXRCommPtr comm, const KernelEntry &kernel, const void *args, const LaunchConfig &cfg,
                 TileXRStream stream);

// An ordinary launch of a kernel that calls StreamWait: its blocks are brought up (barriers, tensor memory, descriptors) while the kernel
// before it in the stream ends, one or two microseconds per launch (17 x 7168 x 2048 in a row 12.3 -> 10.3 us, 1000 x 4104 x 2056 24.2 -> 22.4).
// `cluster` blocks to a cluster (0: none, or as the kernel says).  Returns a cudaError_t.
int LaunchOverlapped(const void *kernel, unsigned gridX, unsigned gridY, unsigned block, size_t smemBytes, unsigned cluster, void **params,
                     TileXRStream stream);

// Number of kernels this library launched since the process started (all communicators).
uint64_t LaunchCount();
// Called by code that launches a kernel directly (local ops without a communicator).
void NoteLaunch();

// Largest grid of `kernel` that can be co-resident on the communicator's device.
// Host work (typically a small follow-up kernel launch) that has to come after the launch that `comm` issued last.  On a
// real communicator that launch is already in its stream and `fn` runs at once; a communicator of an emulated world only
// queues its launches until the group closes, and `fn` runs right after that queued launch has been issued.
int RunAfterLaunch(TileXRCommPtr comm, std::function<int()> fn);

int MaxCooperativeGrid(TileXRCommPtr comm, const KernelEntry &kernel, unsigned block, size_t smemBytes, int ranksPerDevice,
                       unsigned *maxGrid);

} // namespace TileXR

#if defined(__CUDACC__)
namespace TileXR {
// The parameter of an emulated kernel.  The argument structs of up to EMULATED_INLINE_RANKS ranks travel with the launch: an
// allocation, a copy and a release per launch cost 15 us of host time, and where the stream-ordered pool had returned its memory
// to the driver, several hundred.  More ranks than that come as a device array.
template <typename ARGS> struct EmulatedArgs {
    static_assert(alignof(ARGS) <= EMULATED_HEADER_BYTES, "the structs start behind the header");
    union {
        const ARGS *array;            // null: `rank` holds them
        char header[EMULATED_HEADER_BYTES];
    };
    ARGS rank[EMULATED_INLINE_RANKS];
};
} // namespace TileXR

// Defines NAME_single / NAME_emulated around a device body `BODY(const ARGS &)` and a
// KernelEntry named NAME##Entry.
#define TILEXR_DEFINE_KERNEL(NAME, ARGS, BODY, MAX_THREADS) TILEXR_DEFINE_KERNEL_OCC(NAME, ARGS, BODY, MAX_THREADS, 1)
// Same, asking the compiler to keep MIN_BLOCKS blocks of MAX_THREADS threads resident per SM.
#define TILEXR_DEFINE_KERNEL_OCC(NAME, ARGS, BODY, MAX_THREADS, MIN_BLOCKS)                            \
    __global__ void __launch_bounds__(MAX_THREADS, MIN_BLOCKS) NAME##_single(const ARGS a) { BODY(a); } \
    __global__ void __launch_bounds__(MAX_THREADS, MIN_BLOCKS)                                         \
    NAME##_emulated(const __grid_constant__ TileXR::EmulatedArgs<ARGS> perRank)                        \
    {                                                                                                  \
        const ARGS a = perRank.array != nullptr ? perRank.array[blockIdx.y] : perRank.rank[blockIdx.y]; \
        BODY(a);                                                                                       \
    }                                                                                                  \
    static const TileXR::KernelEntry NAME##Entry = {reinterpret_cast<const void *>(&NAME##_single),    \
                                                    reinterpret_cast<const void *>(&NAME##_emulated),  \
                                                    sizeof(ARGS), #NAME, TileXR::EMULATED_INLINE_RANKS};
#endif

#endif // TILEXR_LAUNCH_H
