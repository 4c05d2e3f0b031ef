// The attempt kernels of the 6-stage tableaux.
#define ABM_STAGES 6
#include "abm_attempt.cuh"
