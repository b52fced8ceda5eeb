/* conv_mxr_k: InstanceNorm sums in the epilogue. */
#include "conv_tcr.cuh"

const conv_r_fn umx_conv_r_stats[6] = UMX_R_FORM(true, 0, false);

/* after a bounded wait gave up, blocks may have left without drawing their ticket: the counters start from zero again */
void umx_conv_r_tickets_reset(void) { void *p = nullptr; if (cudaGetSymbolAddress(&p, g_conv_tickets) == cudaSuccess && p) cudaMemset(p, 0, sizeof(unsigned) * 64); }
