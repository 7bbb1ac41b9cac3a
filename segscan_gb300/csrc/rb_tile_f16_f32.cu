// Instantiations of the staged rbsr: FP16, FP32 C.
#include "rb_tile.cuh"

namespace ss {
void *rb_tile_kernel_f16_f32(int G, int V, int NV, bool addc) { return rb_tile_ptr<__half, float>(G, V, NV, addc); }
}  // namespace ss
