// Register-blocked columns: FP64.
#define GB_RB_GROUP 0
#include "passes_rb.cuh"

GB_RB_DEFINE_COLS(double, f64)
