// Instantiations of the staged rbsr: FP16.
#include "rb_tile.cuh"

namespace ss {
void *rb_tile_kernel_f16(int G, int V, int NV, bool addc) { return rb_tile_ptr<__half, __half>(G, V, NV, addc); }
}  // namespace ss
