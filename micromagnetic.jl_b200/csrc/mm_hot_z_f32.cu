// mm_hot_z_f32.cu -- run-time-length z convolutions, FP32 form.
#define MM_HOT_IMPL
#include "mm_hotpass.cuh"

namespace mm {
MM_HOT_Z(, float)
}  // namespace mm
