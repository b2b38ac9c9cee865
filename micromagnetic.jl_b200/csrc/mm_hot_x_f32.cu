// mm_hot_x_f32.cu -- run-time-length x passes, FP32 form.
#define MM_HOT_IMPL
#include "mm_hotpass.cuh"

namespace mm {
MM_HOT_X(, float)
}  // namespace mm
