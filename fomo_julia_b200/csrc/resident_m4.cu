// resident_m4.cu -- the resident kernel for M = 4 (see resident_m.cuh).
#define FOMO_RESIDENT_M 4
#include "resident_m.cuh"
