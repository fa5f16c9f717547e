// Register-blocked LWT rows and columns: FP32 lengths without kernels of their own.
#define GB_RB_GROUP 0
#include "passes_rb.cuh"

GB_RB_DEFINE_LWT(float, f32)
