// Layer kernel instances (T rows per tile, smem row stride, groups per warp).
// The kernel itself lives in layer_kernel.cuh.
#include <vector>
#include "layer_kernel.cuh"

namespace sdnn {

void register_layer_q1024(std::vector<LayerInstance>& v) {
  SDNN_ROWS_INSTANCES(v, 8, 1056, false);
  SDNN_ROWS_INSTANCES(v, 12, 1056, false);
  SDNN_ROWS_INSTANCES(v, 16, 1056, false);
  SDNN_ROWS_INSTANCES(v, 24, 1056, false);
}

}  // namespace sdnn
