// BF16 values and B, FP32 C: instantiations of the tile walk.
#include "eb_tile.cuh"

namespace ss {
void *tile_kernel_bf16_f32(int G, int V, int NV, bool addc) { return tile_ptr<__nv_bfloat16, float>(G, V, NV, addc); }
}  // namespace ss
