// tile_c128_bwd.cu — complex128 tile sweeps, backward (kernel in
// tile_kernels.cuh; one translation unit per direction, compiled in parallel).
#include "tile_launch.cuh"

namespace plk {
namespace tile {

int launch_c128_bwd(const Args &a, dim3 grid, int threads, size_t smem, cudaStream_t st) {
    return launch<AmpC128, kRegsC128Bwd, true, kThreadsC128Bwd, kCtasC128Bwd>(a, grid, threads, smem, st);
}

} // namespace tile
} // namespace plk
