// BF16 instantiations of the segment tile walk.
#include "seg_tile.cuh"

namespace ss {
void *seg_tile_kernel_bf16(int G, int V, int NV, bool addc) { return seg_tile_ptr<__nv_bfloat16>(G, V, NV, addc); }
}  // namespace ss
