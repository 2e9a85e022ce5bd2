// Compiled instances: LES y and z passes in gradient form, float arithmetic.
#include "sc_dispatch.cuh"
#define LES_T float
SC_DEFINE_LES(float)
