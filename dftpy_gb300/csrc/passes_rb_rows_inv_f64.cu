// Register-blocked inverse rows: FP64.
#define GB_RB_GROUP 0
#include "passes_rb.cuh"

GB_RB_DEFINE_INV(double, f64)
