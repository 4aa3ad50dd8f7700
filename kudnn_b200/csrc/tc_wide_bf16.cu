#define KB_TC_KIND KUDNN_B200_BF16
#include "tc_wide_inst.cuh"
