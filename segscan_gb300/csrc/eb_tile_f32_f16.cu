// FP32 values and B, FP16 C: instantiations of the tile walk.
#include "eb_tile.cuh"

namespace ss {
void *tile_kernel_f32_f16(int G, int V, int NV, bool addc) { return tile_ptr<float, __half>(G, V, NV, addc); }
}  // namespace ss
