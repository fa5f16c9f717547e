// Register-blocked LWT rows and columns: FP32 lengths of group 2.
#define GB_RB_GROUP 2
#include "passes_rb.cuh"

GB_RB_DEFINE_LWT(float, f32)
