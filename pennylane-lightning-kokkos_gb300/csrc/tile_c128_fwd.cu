// tile_c128_fwd.cu — complex128 tile sweeps, forward (kernel in
// tile_kernels.cuh; one translation unit per direction, compiled in parallel).
#include "tile_launch.cuh"

namespace plk {
namespace tile {

int launch_c128_fwd(const Args &a, dim3 grid, int threads, size_t smem, cudaStream_t st) {
    return launch<AmpC128, kRegsC128Fwd, false, kThreadsC128Fwd, kCtasC128Fwd>(a, grid, threads, smem, st);
}

} // namespace tile
} // namespace plk
