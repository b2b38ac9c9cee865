// mm_hot_yc_f32.cu -- run-time-length fused film columns, FP32 form.
#define MM_HOT_IMPL
#include "mm_hotpass.cuh"

namespace mm {
MM_HOT_YC(, float)
}  // namespace mm
