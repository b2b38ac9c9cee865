// mm_hot_x_f64.cu -- run-time-length x passes, FP64 form.
#define MM_HOT_IMPL
#include "mm_hotpass.cuh"

namespace mm {
MM_HOT_X(, double)
}  // namespace mm
