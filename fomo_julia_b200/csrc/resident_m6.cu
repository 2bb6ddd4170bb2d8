// resident_m6.cu -- the resident kernel for M = 6 (see resident_m.cuh).
#define FOMO_RESIDENT_M 6
#include "resident_m.cuh"
