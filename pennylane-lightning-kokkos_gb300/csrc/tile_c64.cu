// tile_c64.cu — complex64 tile sweeps (kernel in tile_kernels.cuh).
#include "tile_launch.cuh"

namespace plk {
namespace tile {

int launch_c64(bool bwd, const Args &a, dim3 grid, int threads, size_t smem, cudaStream_t st) {
    return bwd ? launch<AmpC64, kRegsC64Bwd, true, kThreadsC64Bwd, kCtasC64Bwd>(a, grid, threads, smem, st)
               : launch<AmpC64, kRegsC64Fwd, false, kThreadsC64Fwd, kCtasC64Fwd>(a, grid, threads, smem, st);
}

} // namespace tile
} // namespace plk
