#include "tilexr_launch.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include <cuda_runtime_api.h>

#include "comm.h"
#include "tilexr_log.h"

namespace TileXR {

namespace {

struct PendingLaunch {
    TileXRComm *comm;
    const KernelEntry *kernel;
    std::vector<uint8_t> args;
    LaunchConfig cfg;
    cudaStream_t stream;
    std::vector<std::function<int()>> after;     // host work to run once the launch has been issued (RunAfterLaunch)
};

struct GroupState {
    int depth = 0;
    std::vector<PendingLaunch> pending;
};

thread_local GroupState g_group;
std::atomic<uint64_t> g_launches{0};

int SetSmemLimit(const void *fn, size_t smemBytes)
{
    if (smemBytes > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smemBytes));
        if (e != cudaSuccess) {
            TILEXR_LOG(ERROR) << "cudaFuncSetAttribute(smem=" << smemBytes << "): " << cudaGetErrorString(e);
            return TILEXR_ERROR_RUNTIME;
        }
    }
    return TILEXR_SUCCESS;
}

// Resident blocks per SM of a kernel at a block size and an amount of shared memory, and the SMs of the device: the same for every
// launch, asked of the driver once (three calls, 4 us of a launch's host time).
int OccupancyOf(const void *fn, unsigned block, size_t smemBytes, int device, int *perSm, int *sms)
{
    static std::mutex mutex;
    static std::map<std::tuple<const void *, unsigned, size_t, int>, std::pair<int, int>> known;
    const auto key = std::make_tuple(fn, block, smemBytes, device);
    {
        std::lock_guard<std::mutex> lock(mutex);
        const auto it = known.find(key);
        if (it != known.end()) {
            *perSm = it->second.first;
            *sms = it->second.second;
            return TILEXR_SUCCESS;
        }
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(perSm, fn, static_cast<int>(block), smemBytes) != cudaSuccess) {
        cudaGetLastError();
        return TILEXR_ERROR_RUNTIME;
    }
    if (cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return TILEXR_ERROR_RUNTIME;
    std::lock_guard<std::mutex> lock(mutex);
    known[key] = {*perSm, *sms};
    return TILEXR_SUCCESS;
}

int IssueWorldLaunch(EmulatedWorld *world, std::vector<PendingLaunch *> &perRank)
{
    const PendingLaunch &first = *perRank[0];
    const int ranks = world->rankSize;
    for (int r = 0; r < ranks; ++r) {
        const PendingLaunch &p = *perRank[r];
        if (p.kernel != first.kernel || p.cfg.grid != first.cfg.grid || p.cfg.block != first.cfg.block ||
            p.cfg.smemBytes != first.cfg.smemBytes) {
            TILEXR_LOG(ERROR) << "emulated world: rank " << r << " queued " << p.kernel->name << " grid " << p.cfg.grid
                              << " but rank 0 queued " << first.kernel->name << " grid " << first.cfg.grid;
            return TILEXR_ERROR_PARA_CHECK_FAIL;
        }
    }
    if (cudaSetDevice(world->device) != cudaSuccess) return TILEXR_ERROR_RUNTIME;
    const size_t argBytes = first.kernel->argBytes;
    const int inlineRanks = first.kernel->inlineRanks;
    // EmulatedArgs<ARGS>: a pointer in a header, then `inlineRanks` argument structs; without room for any, the pointer alone
    std::vector<uint8_t> packed(EMULATED_HEADER_BYTES + argBytes * std::max(ranks, inlineRanks));
    for (int r = 0; r < ranks; ++r) std::memcpy(packed.data() + EMULATED_HEADER_BYTES + r * argBytes, perRank[r]->args.data(), argBytes);
    void *devArgs = nullptr;
    if (ranks > inlineRanks) {
        // stream-ordered scratch: freed after the kernel on the same stream
        if (cudaMallocAsync(&devArgs, argBytes * ranks, first.stream) != cudaSuccess) return TILEXR_ERROR_RUNTIME;
        if (cudaMemcpyAsync(devArgs, packed.data() + EMULATED_HEADER_BYTES, argBytes * ranks, cudaMemcpyHostToDevice, first.stream) != cudaSuccess) {
            return TILEXR_ERROR_RUNTIME;
        }
        // pageable source: the copy is staged before the call returns, `packed` may go away
    }
    std::memcpy(packed.data(), &devArgs, sizeof(devArgs));
    int ret = SetSmemLimit(first.kernel->emulated, first.cfg.smemBytes);
    if (ret != TILEXR_SUCCESS) return ret;
    void *params[] = {packed.data()};
    const dim3 grid(first.cfg.grid, ranks, 1);
    const dim3 block(first.cfg.block, 1, 1);
    cudaError_t e = cudaLaunchCooperativeKernel(first.kernel->emulated, grid, block, params, first.cfg.smemBytes,
                                                first.stream);
    if (devArgs != nullptr) cudaFreeAsync(devArgs, first.stream);
    if (e != cudaSuccess) {
        TILEXR_LOG(ERROR) << "cooperative launch of " << first.kernel->name << " for " << ranks << " emulated ranks x "
                          << first.cfg.grid << " blocks failed: " << cudaGetErrorString(e);
        cudaGetLastError();
        return TILEXR_ERROR_RUNTIME;
    }
    g_launches.fetch_add(1);
    return TILEXR_SUCCESS;
}

} // namespace

int LaunchOverlapped(const void *kernel, unsigned gridX, unsigned gridY, unsigned block, size_t smemBytes, unsigned cluster, void **params,
                     TileXRStream stream)
{
    cudaLaunchAttribute attrs[2];
    unsigned n = 0;
    attrs[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[n++].val.programmaticStreamSerializationAllowed = 1;
    if (cluster > 0) {
        attrs[n].id = cudaLaunchAttributeClusterDimension;
        attrs[n].val.clusterDim.x = cluster;
        attrs[n].val.clusterDim.y = 1;
        attrs[n++].val.clusterDim.z = 1;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gridX, gridY, 1);
    cfg.blockDim = dim3(block, 1, 1);
    cfg.dynamicSmemBytes = smemBytes;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cfg.attrs = attrs;
    cfg.numAttrs = n;
    return static_cast<int>(cudaLaunchKernelExC(&cfg, kernel, params));
}

uint64_t LaunchCount() { return g_launches.load(); }
void NoteLaunch() { g_launches.fetch_add(1); }

int LaunchKernel(TileXRCommPtr commPtr, const KernelEntry &kernel, const void *args, const LaunchConfig &cfg,
                 TileXRStream streamPtr)
{
    TileXRComm *comm = static_cast<TileXRComm *>(commPtr);
    cudaStream_t stream = static_cast<cudaStream_t>(streamPtr);
    if (comm == nullptr || !comm->initialized()) return TILEXR_ERROR_NOT_INITIALIZED;
    if (comm->isHostMemory()) return TILEXR_ERROR_NOT_SUPPORT;
    if (comm->isEmulated()) {
        if (g_group.depth == 0) {
            TILEXR_LOG(ERROR) << kernel.name << ": a communicator of an emulated world launches only inside "
                              << "TileXRGroupStart/TileXRGroupEnd";
            return TILEXR_ERROR_NOT_SUPPORT;
        }
        PendingLaunch p;
        p.comm = comm;
        p.kernel = &kernel;
        p.args.assign(static_cast<const uint8_t *>(args), static_cast<const uint8_t *>(args) + kernel.argBytes);
        p.cfg = cfg;
        p.stream = stream;
        g_group.pending.push_back(std::move(p));
        return TILEXR_SUCCESS;
    }
    int ret = SetSmemLimit(kernel.single, cfg.smemBytes);
    if (ret != TILEXR_SUCCESS) return ret;
    void *params[] = {const_cast<void *>(args)};
    cudaError_t e;
    if (cfg.cooperative) {
        e = cudaLaunchCooperativeKernel(kernel.single, dim3(cfg.grid), dim3(cfg.block), params, cfg.smemBytes, stream);
    } else if (cfg.overlap) {
        e = static_cast<cudaError_t>(LaunchOverlapped(kernel.single, cfg.grid, 1, cfg.block, cfg.smemBytes, 0, params, stream));
    } else {
        e = cudaLaunchKernel(kernel.single, dim3(cfg.grid), dim3(cfg.block), params, cfg.smemBytes, stream);
    }
    if (e != cudaSuccess) {
        TILEXR_LOG(ERROR) << "launch of " << kernel.name << " grid " << cfg.grid << " block " << cfg.block << " smem "
                          << cfg.smemBytes << " failed: " << cudaGetErrorString(e);
        cudaGetLastError();
        return TILEXR_ERROR_RUNTIME;
    }
    g_launches.fetch_add(1);
    return TILEXR_SUCCESS;
}

int RunAfterLaunch(TileXRCommPtr commPtr, std::function<int()> fn)
{
    TileXRComm *comm = static_cast<TileXRComm *>(commPtr);
    if (comm != nullptr && comm->isEmulated() && g_group.depth > 0) {
        for (auto it = g_group.pending.rbegin(); it != g_group.pending.rend(); ++it) {
            if (it->comm == comm) {
                it->after.push_back(std::move(fn));
                return TILEXR_SUCCESS;
            }
        }
    }
    return fn();
}

int MaxCooperativeGrid(TileXRCommPtr commPtr, const KernelEntry &kernel, unsigned block, size_t smemBytes,
                       int ranksPerDevice, unsigned *maxGrid)
{
    TileXRComm *comm = static_cast<TileXRComm *>(commPtr);
    if (comm == nullptr || !comm->initialized() || comm->isHostMemory()) return TILEXR_ERROR_NOT_INITIALIZED;
    const void *fn = comm->isEmulated() ? kernel.emulated : kernel.single;
    int ret = SetSmemLimit(fn, smemBytes);
    if (ret != TILEXR_SUCCESS) return ret;
    int perSm = 0, sms = 0;
    ret = OccupancyOf(fn, block, smemBytes, comm->device(), &perSm, &sms);
    if (ret != TILEXR_SUCCESS) return ret;
    const int total = perSm * sms;
    *maxGrid = static_cast<unsigned>(total / (ranksPerDevice > 0 ? ranksPerDevice : 1));
    return TILEXR_SUCCESS;
}

extern "C" int TileXRGroupStart(void)
{
    g_group.depth += 1;
    return TILEXR_SUCCESS;
}

extern "C" int TileXRGroupEnd(void)
{
    if (g_group.depth == 0) return TILEXR_ERROR_PARA_CHECK_FAIL;
    g_group.depth -= 1;
    if (g_group.depth > 0) return TILEXR_SUCCESS;
    std::vector<PendingLaunch> pending;
    pending.swap(g_group.pending);
    // The k-th call of every rank of a world forms the k-th launch of that world.
    std::map<EmulatedWorld *, std::vector<std::vector<PendingLaunch *>>> byWorld;
    for (PendingLaunch &p : pending) {
        EmulatedWorld *w = p.comm->world();
        std::vector<std::vector<PendingLaunch *>> &perRank = byWorld[w];
        if (perRank.empty()) perRank.resize(w->rankSize);
        perRank[p.comm->rank()].push_back(&p);
    }
    int result = TILEXR_SUCCESS;
    for (auto &kv : byWorld) {
        EmulatedWorld *w = kv.first;
        const size_t calls = kv.second[0].size();
        for (int r = 0; r < w->rankSize; ++r) {
            if (kv.second[r].size() != calls) {
                TILEXR_LOG(ERROR) << "emulated world: rank " << r << " queued " << kv.second[r].size()
                                  << " launches, rank 0 queued " << calls;
                return TILEXR_ERROR_PARA_CHECK_FAIL;
            }
        }
        for (size_t k = 0; k < calls; ++k) {
            std::vector<PendingLaunch *> row(w->rankSize);
            for (int r = 0; r < w->rankSize; ++r) row[r] = kv.second[r][k];
            int ret = IssueWorldLaunch(w, row);
            if (ret != TILEXR_SUCCESS) result = ret;
            for (PendingLaunch *p : row) {
                for (auto &fn : p->after) {
                    ret = fn();
                    if (ret != TILEXR_SUCCESS) result = ret;
                }
            }
        }
    }
    return result;
}

} // namespace TileXR
