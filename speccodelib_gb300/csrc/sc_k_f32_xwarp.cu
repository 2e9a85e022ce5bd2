// Compiled instances: x-pass, float arithmetic: lane groups for M = 16, 32,
// 64, a warp per row for M = 128, 256.
#include "sc_dispatch.cuh"
SC_DEFINE_XWARP(float,
                SC_XGROUP_CASE(float, 4) SC_XGROUP_CASE(float, 5) SC_XGROUP_CASE(float, 6)
                SC_XWARP_CASE(float, 7) SC_XWARP_CASE(float, 8),
                SC_XGUMAX_CASE(float, 4) SC_XGUMAX_CASE(float, 5) SC_XGUMAX_CASE(float, 6)
                SC_XUMAX_CASE(float, 7) SC_XUMAX_CASE(float, 8))
