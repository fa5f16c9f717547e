// Register-blocked forward rows: FP64.
#define GB_RB_GROUP 0
#include "passes_rb.cuh"

GB_RB_DEFINE_FWD(double, f64)
