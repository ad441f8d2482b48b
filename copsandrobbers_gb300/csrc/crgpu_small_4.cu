// The small solve's kernel for k = 4 (see crgpu_small.cu).
#define CR_SMALL_K 4
#include "crgpu_small_run.cuh"
