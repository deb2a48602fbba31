// Layer kernel instances (T rows per tile, smem row stride, groups per warp).
// The kernel itself lives in layer_kernel.cuh.
#include <vector>
#include "layer_kernel.cuh"

namespace sdnn {

SDNN_ROWS_INSTANCE(2, 4128, false)
SDNN_ROWS_INSTANCE(2, 4128, true)
SDNN_ROWS_INSTANCE(3, 4128, false)
SDNN_ROWS_INSTANCE(3, 4128, true)
SDNN_ROWS_INSTANCE(4, 4128, false)
SDNN_ROWS_INSTANCE(4, 4128, true)
SDNN_ROWS_INSTANCE(5, 4128, false)
SDNN_ROWS_INSTANCE(5, 4128, true)
SDNN_ROWS_INSTANCE(6, 4128, false)
SDNN_ROWS_INSTANCE(6, 4128, true)

void register_layer_q4096(std::vector<LayerInstance>& v) {
  v.push_back({2, 4128, 1, false, (const void*)&layer_rows_kernel<2, 4128, false>});
  v.push_back({2, 4128, 1, true, (const void*)&layer_rows_kernel<2, 4128, true>});
  v.push_back({3, 4128, 1, false, (const void*)&layer_rows_kernel<3, 4128, false>});
  v.push_back({3, 4128, 1, true, (const void*)&layer_rows_kernel<3, 4128, true>});
  v.push_back({4, 4128, 1, false, (const void*)&layer_rows_kernel<4, 4128, false>});
  v.push_back({4, 4128, 1, true, (const void*)&layer_rows_kernel<4, 4128, true>});
  v.push_back({5, 4128, 1, false, (const void*)&layer_rows_kernel<5, 4128, false>});
  v.push_back({5, 4128, 1, true, (const void*)&layer_rows_kernel<5, 4128, true>});
  v.push_back({6, 4128, 1, false, (const void*)&layer_rows_kernel<6, 4128, false>});
  v.push_back({6, 4128, 1, true, (const void*)&layer_rows_kernel<6, 4128, true>});
}

}  // namespace sdnn
