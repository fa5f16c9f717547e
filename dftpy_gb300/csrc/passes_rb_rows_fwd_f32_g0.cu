// Register-blocked forward rows: FP32 lengths without kernels of their own.
#define GB_RB_GROUP 0
#include "passes_rb.cuh"

GB_RB_DEFINE_FWD(float, f32)
