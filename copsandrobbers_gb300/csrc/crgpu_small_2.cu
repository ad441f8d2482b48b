// The small solve's kernel for k = 2 (see crgpu_small.cu).
#define CR_SMALL_K 2
#include "crgpu_small_run.cuh"
