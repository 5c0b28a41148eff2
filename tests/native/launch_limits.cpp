/*
 * Test helper: zlaunch.h over a fake runtime of 16 devices.  Threads ask for
 * random shared-memory limits of 200 kernels; prints how often a kernel's limit
 * was lowered, how often it was below what a call had just asked for, and how
 * often a device's SM count was wrong.  Built and run by
 * tests/test_launch_limits.py.
 */
#include "zlaunch.h"

#include <atomic>
#include <cstdio>
#include <random>
#include <thread>

constexpr int NDEV = 16, NFN = 200;
static std::atomic<int> limit[NDEV][NFN];
static std::atomic<long> lowered{0};
static char fns[NFN];
static thread_local int cur = 0;

extern "C" {
cudaError_t cudaGetDevice(int *d)
{
    *d = cur;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int dev)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 100 + dev : a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 233472 : 1024;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *per, const void *, int threads, size_t)
{
    *per = 2048 / threads;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *fn, cudaFuncAttribute, int v)
{
    std::atomic<int> &l = limit[cur][(const char *)fn - fns];
    if (l.exchange(v) > v) lowered++;
    return cudaSuccess;
}
}

int main()
{
    std::atomic<long> below{0}, wrong{0};
    std::vector<std::thread> th;
    for (int t = 0; t < 8; t++)
        th.emplace_back([&, t] {
            std::mt19937 r(t);
            for (int i = 0; i < 2000; i++) {
                cur = (int)(r() % NDEV);
                const int f = (int)(r() % NFN), want = 1024 * (1 + (int)(r() % 200));
                if (set_max_smem(fns + f, want) != cudaSuccess || limit[cur][f] < want) below++;
                if (sm_count() != 100 + cur || blocks_per_sm(fns + f, 256, want) != 8) wrong++;
            }
        });
    for (auto &t : th) t.join();
    std::printf("%ld %ld %ld\n", lowered.load(), below.load(), wrong.load());
}
