/* conv_mxr_k: one input item a stage. */
#include "conv_tcr.cuh"

const conv_r_fn umx_conv_r_one[6] = UMX_R_FORM(false, 0, false);
