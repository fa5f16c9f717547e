// Register-blocked WGC columns: FP32 lengths without kernels of their own.
#define GB_RB_GROUP 0
#include "passes_rb.cuh"

GB_RB_DEFINE_WGC(float, f32)
