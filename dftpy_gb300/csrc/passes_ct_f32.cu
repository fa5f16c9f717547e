// The FP32 plane pipeline: row passes of compile-time length, plane convolution.
#include "passes_ct.cuh"

GB_CT_DEFINE_PLANE()
