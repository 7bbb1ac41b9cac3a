// Instantiations of the staged rbsr: BF16, FP32 C.
#include "rb_tile.cuh"

namespace ss {
void *rb_tile_kernel_bf16_f32(int G, int V, int NV, bool addc) { return rb_tile_ptr<__nv_bfloat16, float>(G, V, NV, addc); }
}  // namespace ss
