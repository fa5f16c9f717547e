// Register-blocked LWT rows and columns: FP64.
#define GB_RB_GROUP 0
#include "passes_rb.cuh"

GB_RB_DEFINE_LWT(double, f64)
