// The attempt kernels of the 2-stage tableaux.
#define ABM_STAGES 2
#include "abm_attempt.cuh"
