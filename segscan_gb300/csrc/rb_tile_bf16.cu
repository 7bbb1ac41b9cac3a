// Instantiations of the staged rbsr: BF16.
#include "rb_tile.cuh"

namespace ss {
void *rb_tile_kernel_bf16(int G, int V, int NV, bool addc) { return rb_tile_ptr<__nv_bfloat16, __nv_bfloat16>(G, V, NV, addc); }
}  // namespace ss
