// mm_hot_y_f32.cu -- run-time-length y passes of 3-D meshes, FP32 form.
#define MM_HOT_IMPL
#include "mm_hotpass.cuh"

namespace mm {
MM_HOT_Y(, float)
}  // namespace mm
