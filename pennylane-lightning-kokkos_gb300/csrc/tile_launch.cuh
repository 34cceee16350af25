// tile_launch.cuh — launch shapes of the tile kernels.
#pragma once

#include <atomic>

#include "tile_kernels.cuh"

namespace plk {
namespace tile {

// register bits, CTA threads (2^(largest T - R)) and CTAs per SM
constexpr int kRegsC64Fwd = 4, kThreadsC64Fwd = 512, kCtasC64Fwd = 2;
constexpr int kRegsC64Bwd = 4, kThreadsC64Bwd = 256, kCtasC64Bwd = 2;
constexpr int kRegsC128Fwd = 4, kThreadsC128Fwd = 256, kCtasC128Fwd = 2;
constexpr int kRegsC128Bwd = 3, kThreadsC128Bwd = 256, kCtasC128Bwd = 2;
constexpr size_t kMaxBlob = 20480;

constexpr size_t smem_bytes(int amp_bytes, bool bwd, int T, size_t blob, int nacc, int threads) {
    return ((size_t)amp_bytes << T) * (bwd ? 2 : 1) + blob + (bwd ? (size_t)nacc * (threads / 32) * 8 : 0);
}

template <class A, int R, bool BWD, int THREADS, int CTAS>
int launch(const Args &a, dim3 grid, int threads, size_t smem, cudaStream_t st) {
    // more than 48 KiB of dynamic shared memory needs an opt-in, once per device
    static std::atomic<unsigned long long> opted{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(opted.load() & bit)) {
        int T = R;
        while ((1 << (T - R)) < THREADS) T++;
        PLK_CUDA(cudaFuncSetAttribute(k_tile<A, R, BWD, THREADS, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem_bytes(A::kBytes, BWD, T, kMaxBlob, 2 * kMaxAcc, THREADS)));
        opted.fetch_or(bit);
    }
    k_tile<A, R, BWD, THREADS, CTAS><<<grid, threads, smem, st>>>(a);
    PLK_CHECK_LAUNCH();
    return PLK_OK;
}

int launch_c64(bool bwd, const Args &a, dim3 grid, int threads, size_t smem, cudaStream_t st);
int launch_c128_fwd(const Args &a, dim3 grid, int threads, size_t smem, cudaStream_t st);
int launch_c128_bwd(const Args &a, dim3 grid, int threads, size_t smem, cudaStream_t st);

} // namespace tile
} // namespace plk
