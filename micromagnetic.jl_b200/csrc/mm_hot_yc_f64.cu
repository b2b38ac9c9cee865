// mm_hot_yc_f64.cu -- run-time-length fused film columns, FP64 form.
#define MM_HOT_IMPL
#include "mm_hotpass.cuh"

namespace mm {
MM_HOT_YC(, double)
}  // namespace mm
