// resident_m3.cu -- the resident kernel for M = 3 (see resident_m.cuh).
#define FOMO_RESIDENT_M 3
#include "resident_m.cuh"
