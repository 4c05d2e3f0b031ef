// The attempt kernels of the 7-stage tableaux.
#define ABM_STAGES 7
#include "abm_attempt.cuh"
