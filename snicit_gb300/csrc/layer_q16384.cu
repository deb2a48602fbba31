// Layer kernel instances (T rows per tile, smem row stride, groups per warp).
// The kernel itself lives in layer_kernel.cuh.
#include <vector>
#include "layer_kernel.cuh"

namespace sdnn {

SDNN_CHUNK_INSTANCE(1, 16416, 16, false)
SDNN_CHUNK_INSTANCE(1, 16416, 16, true)
SDNN_CHUNK_INSTANCE(2, 16416, 16, false)
SDNN_CHUNK_INSTANCE(2, 16416, 16, true)
SDNN_CHUNK_INSTANCE(3, 16416, 16, false)
SDNN_CHUNK_INSTANCE(3, 16416, 16, true)
SDNN_CHUNK_INSTANCE(1, 16416, 8, false)
SDNN_CHUNK_INSTANCE(1, 16416, 8, true)
SDNN_CHUNK_INSTANCE(2, 16416, 8, false)
SDNN_CHUNK_INSTANCE(2, 16416, 8, true)
SDNN_CHUNK_INSTANCE(3, 16416, 8, false)
SDNN_CHUNK_INSTANCE(3, 16416, 8, true)
SDNN_CHUNK_INSTANCE(1, 32800, 16, false)
SDNN_CHUNK_INSTANCE(1, 32800, 16, true)

void register_layer_q16384(std::vector<LayerInstance>& v) {
  SDNN_ROWS_INSTANCES(v, 1, 16416, false);
  SDNN_ROWS_INSTANCES(v, 2, 16416, false);
  SDNN_ROWS_INSTANCES(v, 2, 16416, true);
  SDNN_ROWS_INSTANCES(v, 3, 16416, false);
  v.push_back({1, 16416, 16, false, false, (const void*)&layer_chunk_kernel<1, 16416, 16, false>});
  v.push_back({1, 16416, 16, true, false, (const void*)&layer_chunk_kernel<1, 16416, 16, true>});
  v.push_back({2, 16416, 16, false, false, (const void*)&layer_chunk_kernel<2, 16416, 16, false>});
  v.push_back({2, 16416, 16, true, false, (const void*)&layer_chunk_kernel<2, 16416, 16, true>});
  v.push_back({3, 16416, 16, false, false, (const void*)&layer_chunk_kernel<3, 16416, 16, false>});
  v.push_back({3, 16416, 16, true, false, (const void*)&layer_chunk_kernel<3, 16416, 16, true>});
  v.push_back({1, 16416, 8, false, false, (const void*)&layer_chunk_kernel<1, 16416, 8, false>});
  v.push_back({1, 16416, 8, true, false, (const void*)&layer_chunk_kernel<1, 16416, 8, true>});
  v.push_back({2, 16416, 8, false, false, (const void*)&layer_chunk_kernel<2, 16416, 8, false>});
  v.push_back({2, 16416, 8, true, false, (const void*)&layer_chunk_kernel<2, 16416, 8, true>});
  v.push_back({3, 16416, 8, false, false, (const void*)&layer_chunk_kernel<3, 16416, 8, false>});
  v.push_back({3, 16416, 8, true, false, (const void*)&layer_chunk_kernel<3, 16416, 8, true>});
  v.push_back({1, 32800, 16, false, false, (const void*)&layer_chunk_kernel<1, 32800, 16, false>});
  v.push_back({1, 32800, 16, true, false, (const void*)&layer_chunk_kernel<1, 32800, 16, true>});
}

}  // namespace sdnn
