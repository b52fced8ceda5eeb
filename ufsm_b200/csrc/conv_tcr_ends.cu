/* conv_mxr_k: scale windows gathered by the scale warp from a tensor that ends inside a word. */
#include "conv_tcr.cuh"

const conv_r_fn umx_conv_r_ends[6] = UMX_R_FORM(false, 2, false);
