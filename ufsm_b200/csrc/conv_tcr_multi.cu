/* conv_mxr_k: several input items a stage. */
#include "conv_tcr.cuh"

const conv_r_fn umx_conv_r_multi[6] = UMX_R_FORM(false, 0, true);
