// tile_filter_kernel<float> (k_tile.cuh).
#include "k_tile.cuh"

namespace clv {
template cudaError_t setup_tile_filter<float>(size_t, int, int *);
template cudaError_t launch_tile_filter<float>(const LaunchTileFilter &, cudaStream_t);
}  // namespace clv
