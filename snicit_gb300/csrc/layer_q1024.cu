// Layer kernel instances (T rows per tile, smem row stride, groups per warp).
// The kernel itself lives in layer_kernel.cuh.
#include <vector>
#include "layer_kernel.cuh"

namespace sdnn {

SDNN_ROWS_INSTANCE(8, 1056, false)
SDNN_ROWS_INSTANCE(8, 1056, true)
SDNN_ROWS_INSTANCE(12, 1056, false)
SDNN_ROWS_INSTANCE(12, 1056, true)
SDNN_ROWS_INSTANCE(16, 1056, false)
SDNN_ROWS_INSTANCE(16, 1056, true)
SDNN_ROWS_INSTANCE(24, 1056, false)
SDNN_ROWS_INSTANCE(24, 1056, true)

void register_layer_q1024(std::vector<LayerInstance>& v) {
  v.push_back({8, 1056, 1, false, (const void*)&layer_rows_kernel<8, 1056, false>});
  v.push_back({8, 1056, 1, true, (const void*)&layer_rows_kernel<8, 1056, true>});
  v.push_back({12, 1056, 1, false, (const void*)&layer_rows_kernel<12, 1056, false>});
  v.push_back({12, 1056, 1, true, (const void*)&layer_rows_kernel<12, 1056, true>});
  v.push_back({16, 1056, 1, false, (const void*)&layer_rows_kernel<16, 1056, false>});
  v.push_back({16, 1056, 1, true, (const void*)&layer_rows_kernel<16, 1056, true>});
  v.push_back({24, 1056, 1, false, (const void*)&layer_rows_kernel<24, 1056, false>});
  v.push_back({24, 1056, 1, true, (const void*)&layer_rows_kernel<24, 1056, true>});
}

}  // namespace sdnn
