// FP16 values and B, FP32 C: instantiations of the tile walk.
#include "eb_tile.cuh"

namespace ss {
void *tile_kernel_f16_f32(int G, int V, int NV, bool addc) { return tile_ptr<__half, float>(G, V, NV, addc); }
}  // namespace ss
