// Compiled instances: lane-group x-pass, double arithmetic (M = 16 .. 256).
#include "sc_dispatch.cuh"
SC_DEFINE_XWARP(double,
                SC_XGROUP_CASE(double, 4) SC_XGROUP_CASE(double, 5) SC_XGROUP_CASE(double, 6)
                SC_XGROUP_CASE(double, 7) SC_XGROUP_CASE(double, 8),
                SC_XGUMAX_CASE(double, 4) SC_XGUMAX_CASE(double, 5) SC_XGUMAX_CASE(double, 6)
                SC_XGUMAX_CASE(double, 7) SC_XGUMAX_CASE(double, 8))
