#define KB_TC_KIND KUDNN_B200_S8
#include "tc_wide_inst.cuh"
