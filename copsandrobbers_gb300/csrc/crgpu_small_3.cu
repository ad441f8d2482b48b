// The small solve's kernel for k = 3 (see crgpu_small.cu).
#define CR_SMALL_K 3
#include "crgpu_small_run.cuh"
