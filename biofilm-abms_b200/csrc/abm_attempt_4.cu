// The attempt kernels of the 4-stage tableaux.
#define ABM_STAGES 4
#include "abm_attempt.cuh"
