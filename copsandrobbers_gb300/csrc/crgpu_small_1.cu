// The small solve's kernel for k = 1 (see crgpu_small.cu).
#define CR_SMALL_K 1
#include "crgpu_small_run.cuh"
