#define KB_TC_KIND KUDNN_B200_F16
#include "tc_wide_inst.cuh"
