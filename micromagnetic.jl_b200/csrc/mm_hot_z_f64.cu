// mm_hot_z_f64.cu -- run-time-length z convolutions, FP64 form.
#define MM_HOT_IMPL
#include "mm_hotpass.cuh"

namespace mm {
MM_HOT_Z(, double)
}  // namespace mm
