// Register-blocked inverse rows: FP32 lengths of group 4.
#define GB_RB_GROUP 4
#include "passes_rb.cuh"

GB_RB_DEFINE_INV(float, f32)
