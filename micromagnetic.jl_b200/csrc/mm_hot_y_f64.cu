// mm_hot_y_f64.cu -- run-time-length y passes of 3-D meshes, FP64 form.
#define MM_HOT_IMPL
#include "mm_hotpass.cuh"

namespace mm {
MM_HOT_Y(, double)
}  // namespace mm
