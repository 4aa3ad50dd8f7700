#define KB_TC_KIND KUDNN_B200_F32
#include "tc_inst.cuh"
