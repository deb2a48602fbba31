// Layer kernel instances (T rows per tile, smem row stride, groups per warp).
// The kernel itself lives in layer_kernel.cuh.
#include <vector>
#include "layer_kernel.cuh"

namespace sdnn {

void register_layer_q4096(std::vector<LayerInstance>& v) {
  SDNN_ROWS_INSTANCES(v, 2, 4128, false);
  SDNN_ROWS_INSTANCES(v, 3, 4128, false);
  SDNN_ROWS_INSTANCES(v, 4, 4128, false);
  SDNN_ROWS_INSTANCES(v, 5, 4128, false);
  SDNN_ROWS_INSTANCES(v, 6, 4128, false);
}

}  // namespace sdnn
