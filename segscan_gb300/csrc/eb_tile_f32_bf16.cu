// FP32 values and B, BF16 C: instantiations of the tile walk.
#include "eb_tile.cuh"

namespace ss {
void *tile_kernel_f32_bf16(int G, int V, int NV, bool addc) { return tile_ptr<float, __nv_bfloat16>(G, V, NV, addc); }
}  // namespace ss
