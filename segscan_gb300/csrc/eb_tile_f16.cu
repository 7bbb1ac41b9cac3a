// FP16 instantiations of the tile walk.
#include "eb_tile.cuh"

namespace ss {
void *tile_kernel_f16(int G, int V, int NV, bool addc) { return tile_ptr<__half, __half>(G, V, NV, addc); }
}  // namespace ss
