// resident_m1.cu -- the resident kernel for M = 1 (see resident_m.cuh).
#define FOMO_RESIDENT_M 1
#include "resident_m.cuh"
