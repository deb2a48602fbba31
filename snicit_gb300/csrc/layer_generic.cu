// Layer kernel instances (T rows per tile, smem row stride, groups per warp).
// The kernel itself lives in layer_kernel.cuh.
#include <vector>
#include "layer_kernel.cuh"

namespace sdnn {

SDNN_CHUNK_INSTANCE(1, 0, 16, false)
SDNN_CHUNK_INSTANCE(1, 0, 16, true)

void register_layer_generic(std::vector<LayerInstance>& v) {
  SDNN_ROWS_INSTANCES(v, 1, 0, false);
  SDNN_ROWS_INSTANCES(v, 1, 0, true);
  SDNN_ROWS_INSTANCES(v, 2, 0, false);
  SDNN_ROWS_INSTANCES(v, 2, 0, true);
  SDNN_ROWS_INSTANCES(v, 4, 0, false);
  SDNN_ROWS_INSTANCES(v, 8, 0, false);
  v.push_back({1, 0, 16, false, false, (const void*)&layer_chunk_kernel<1, 0, 16, false>});
  v.push_back({1, 0, 16, true, false, (const void*)&layer_chunk_kernel<1, 0, 16, true>});
}

}  // namespace sdnn
