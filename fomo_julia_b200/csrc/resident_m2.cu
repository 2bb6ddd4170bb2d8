// resident_m2.cu -- the resident kernel for M = 2 (see resident_m.cuh).
#define FOMO_RESIDENT_M 2
#include "resident_m.cuh"
