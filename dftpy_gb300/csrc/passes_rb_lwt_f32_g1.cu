// Register-blocked LWT rows and columns: FP32 lengths of group 1.
#define GB_RB_GROUP 1
#include "passes_rb.cuh"

GB_RB_DEFINE_LWT(float, f32)
