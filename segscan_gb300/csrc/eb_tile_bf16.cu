// BF16 instantiations of the tile walk.
#include "eb_tile.cuh"

namespace ss {
void *tile_kernel_bf16(int G, int V, int NV, bool addc) { return tile_ptr<__nv_bfloat16, __nv_bfloat16>(G, V, NV, addc); }
}  // namespace ss
