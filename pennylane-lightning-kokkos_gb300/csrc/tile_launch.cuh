// tile_launch.cuh — launch shapes of the tile kernels.
#pragma once

#include <atomic>

#include "tile_kernels.cuh"

namespace plk {
namespace tile {

// Register bits, CTA threads (2^(largest T - R)) and CTAs per SM.  All shapes
// fill the register file; smaller CTAs drift apart, so that one's memory phase
// runs under another's arithmetic, larger ones need fewer passes.  Measured
// (27-qubit QAOA, complex64 forward): 512 x 2 9.78 ms, 256 x 4 9.54, 128 x 8
// 9.18.  26-qubit gradient, complex64 backward: 256 x 2 41.9 ms, 128 x 4 40.0,
// R = 3 512 x 2 44.7.  25-qubit circuit, complex128 forward: 256 x 2 8.23 ms,
// 128 x 4 8.16, 64 x 8 8.81, R = 3 512 x 2 8.65.  20-qubit Jacobian, complex128
// backward: R = 3 256 x 2 32.8 ms, 128 x 4 36.9; R = 4 (its code overflows the
// instruction cache) 128 x 2 36.0, 64 x 4 35.3.
constexpr int kRegsC64Fwd = 4, kThreadsC64Fwd = 128, kCtasC64Fwd = 8;
constexpr int kRegsC64Bwd = 4, kThreadsC64Bwd = 128, kCtasC64Bwd = 4;
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
