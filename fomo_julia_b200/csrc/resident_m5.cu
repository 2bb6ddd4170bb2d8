// resident_m5.cu -- the resident kernel for M = 5 (see resident_m.cuh).
#define FOMO_RESIDENT_M 5
#include "resident_m.cuh"
