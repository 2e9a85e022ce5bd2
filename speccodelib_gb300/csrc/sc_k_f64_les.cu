// Compiled instances: LES y and z passes in gradient form, double arithmetic.
#include "sc_dispatch.cuh"
#define LES_T double
SC_DEFINE_LES(double)
