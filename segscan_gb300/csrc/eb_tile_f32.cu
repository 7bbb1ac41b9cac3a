// FP32 instantiations of the tile walk.
#include "eb_tile.cuh"

namespace ss {
void *tile_kernel_f32(int G, int V, int NV, bool addc) { return tile_ptr<float, float>(G, V, NV, addc); }
}  // namespace ss
