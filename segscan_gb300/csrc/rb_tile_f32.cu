// Instantiations of the staged rbsr: FP32.
#include "rb_tile.cuh"

namespace ss {
void *rb_tile_kernel_f32(int G, int V, int NV, bool addc) { return rb_tile_ptr<float, float>(G, V, NV, addc); }
}  // namespace ss
