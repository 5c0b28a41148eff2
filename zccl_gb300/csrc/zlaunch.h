/*
 * zlaunch.h -- host side of a launch: what a kernel's grid and shared memory
 * are on the current device, and its shared-memory limit.
 */
#ifndef ZCCL_GB300_ZLAUNCH_H
#define ZCCL_GB300_ZLAUNCH_H

#include <cuda_runtime_api.h>
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>

#include <mutex>
#include <vector>

/* Launch-shape queries, remembered per device and kernel: the occupancy
 * calculator and the shared-memory attribute cost host time on every
 * launch, and a pipelined host-buffer call launches a hundred kernels. */
struct LaunchCache {
    struct Occ {
        const void *fn;
        int dev, threads, per;
        size_t smem;
    };
    struct Attr {
        const void *fn;
        int dev;
        size_t smem;
    };
    struct Dev {
        int nsm, smem_sm, smem_rsv; /* 0: not asked yet */
    };
    std::mutex mu; /* every access below */
    std::vector<Occ> occ;
    std::vector<Attr> attr;
    std::vector<Dev> dev;
};

static inline LaunchCache &launch_cache()
{
    static LaunchCache c;
    return c;
}

/* Blocks of fn per SM at this block size and shared memory (at least 1). */
static inline int blocks_per_sm(const void *fn, int threads, size_t smem)
{
    LaunchCache &c = launch_cache();
    int dev = 0;
    cudaGetDevice(&dev);
    {
        std::lock_guard<std::mutex> lk(c.mu);
        for (const LaunchCache::Occ &o : c.occ)
            if (o.fn == fn && o.dev == dev && o.threads == threads && o.smem == smem) return o.per;
    }
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        per = 0;
    }
    if (per < 1) per = 1;
    std::lock_guard<std::mutex> lk(c.mu);
    try {
        c.occ.push_back({fn, dev, threads, per, smem});
    } catch (...) { /* no memory: asked again next time */
    }
    return per;
}

/* The current device's SMs, and the shared memory of one and of a block's
 * reserve in it; all 1, 0, 0 where the device does not tell. */
static inline LaunchCache::Dev device_shape()
{
    LaunchCache &c = launch_cache();
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(c.mu);
    if (dev >= 0 && (size_t)dev < c.dev.size() && c.dev[dev].nsm > 0) return c.dev[dev];
    LaunchCache::Dev d = {0, 0, 0};
    if (cudaDeviceGetAttribute(&d.nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || d.nsm < 1 ||
        cudaDeviceGetAttribute(&d.smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&d.smem_rsv, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess) {
        cudaGetLastError();
        return {d.nsm > 0 ? d.nsm : 1, 0, 0};
    }
    try {
        if ((size_t)dev >= c.dev.size()) c.dev.resize((size_t)dev + 1, LaunchCache::Dev{0, 0, 0});
        c.dev[dev] = d;
    } catch (...) {
    }
    return d;
}

/* SMs of the current device. */
static inline int sm_count() { return device_shape().nsm; }

/* cudaFuncSetAttribute(fn, MaxDynamicSharedMemorySize, smem), skipped when
 * an equal or larger value is already set for fn on this device.  Every
 * kernel's limit goes through here, so no call lowers one that another
 * thread's launch counts on. */
static inline cudaError_t set_max_smem(const void *fn, size_t smem)
{
    LaunchCache &c = launch_cache();
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(c.mu); /* held while setting: a call that wants less must not undo one that wants more */
    size_t i = 0;
    while (i < c.attr.size() && !(c.attr[i].fn == fn && c.attr[i].dev == dev)) i++;
    if (i < c.attr.size() && c.attr[i].smem >= smem) return cudaSuccess;
    if (i == c.attr.size()) {
        try {
            c.attr.push_back({fn, dev, 0});
        } catch (...) { /* never set without a record */
            return cudaErrorMemoryAllocation;
        }
    }
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) c.attr[i].smem = smem;
    return e;
}

/* Ring bytes of a kernel that runs `per_sm` CTAs per SM and needs `fixed`
 * other bytes of shared memory: at least `least` (one worst-case tile), and
 * up to the CTA's share of the SM's shared memory less a kilobyte of margin.
 * The longer the ring, the longer a tile may wait there for its place
 * before the compute warps run out of room. */
static inline uint32_t ring_bytes(uint32_t per_sm, uint32_t fixed, uint32_t least)
{
    const LaunchCache::Dev d = device_shape();
    if (!d.smem_sm) return least;
    const int share = d.smem_sm / (int)per_sm - d.smem_rsv - 1024 - (int)fixed;
    return share > (int)least ? (uint32_t)share & ~15u : least;
}

static inline unsigned persistent_grid(const void *fn, int threads, size_t smem, uint64_t ntiles)
{
    const uint64_t g = (uint64_t)sm_count() * (uint64_t)blocks_per_sm(fn, threads, smem);
    return (unsigned)(g < ntiles ? g : ntiles);
}

/* Grid of a kernel whose tiles' places come from the scanning CTA: `want`
 * working CTAs (0: as many as fit, at most one per tile) and, with more than
 * one tile, the scanner (none where only one CTA fits).  Test hook:
 * ZCCL_GPU_TEST_ONE_CTA=1 in the environment launches a single CTA. */
static inline unsigned scanned_grid(const void *fn, int threads, size_t smem, uint64_t ntiles, unsigned want)
{
    const char *one = getenv("ZCCL_GPU_TEST_ONE_CTA");
    if (ntiles == 1 || (one && one[0] == '1' && !one[1])) return 1;
    const unsigned g = persistent_grid(fn, threads, smem, ntiles + 1);
    return want && want + 1 < g ? want + 1 : g;
}

#endif
