/* conv_mxr_k: scale windows gathered by the scale warp. */
#include "conv_tcr.cuh"

const conv_r_fn umx_conv_r_gather[6] = UMX_R_FORM(false, 1, false);
