// FP32 instantiations of the segment tile walk.
#include "seg_tile.cuh"

namespace ss {
void *seg_tile_kernel_f32(int G, int V, int NV, bool addc) { return seg_tile_ptr<float>(G, V, NV, addc); }
}  // namespace ss
