/* Weight preparation of the 27-tap convs: fp32 weights [co][ci][27] -> the shared-memory images of the general kernel (UMX_CONV3, UMX_CONV3S2) and
   of the z-marching ones (conv_tcr.cu, conv_s2.cu), quantised per (row, tap, 32 input channels) as the reference's prep_w8_k / prep_w4_k
   (src/lp_f8fwd.cu:54-71, src/lp_f4fwd.cu:53-66).

   A warp owns one (output row, K item of 32 or 64 input channels): its weights are one contiguous run of 27 floats a channel, which comes into
   shared memory coalesced, and lane t < 27 then quantises tap t (27 is odd: no bank conflicts).  Callers that change their weights
   between calls pay for this pass on every call, so it is bound by the memory rate and not by its access pattern: 256 -> 256 in MX-fp4 (7 MB)
   took 24 us with a thread a row reading 4 bytes every 108 (and one thread writing the bias), 7.3 us in this form with nine loads in flight and about 1 us less
   with all of them (32 -> 64 channels 0.6 us less). */
#include "conv_epi.cuh"

namespace {

struct RImage { uint8_t *wr; int nt, w_bytes, w_codes, nquad, gt, goff1, goff2; };      /* the z-marching kernel's image (prep_wr layout), wr NULL: none */

template <int BITS>
__global__ void __launch_bounds__(128) prep_w27_k(const PrepArgs p, const RImage r) {
    pdl_trigger(); pdl_wait();
    constexpr int CI = BITS == 8 ? 32 : 64, RUN = CI * 27;
    __shared__ float sm[4][RUN];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.x, ki = blockIdx.y * 4 + warp;
    if (blockIdx.y == 0 && threadIdx.x == 0 && p.bias_p) p.bias_p[row] = (p.bias && row < p.co) ? ld_dep(p.bias + row) : 0.f;
    const int nitem = (p.ci + CI - 1) / CI;                   /* K items a tap */
    if (ki >= nitem) return;
    float *s = sm[warp];
    const int have = row < p.co ? min(CI, p.ci - ki * CI) * 27 : 0;
    const float *src = p.w + ((size_t)row * p.ci + (size_t)ki * CI) * 27;
    /* all of a warp's loads in flight at once; the caller's weights may come from the kernel just ahead */
    float t[RUN / 32];
#pragma unroll
    for (int k = 0; k < RUN / 32; k++) t[k] = 32 * k + lane < have ? ld_dep(src + 32 * k + lane) : 0.f;
#pragma unroll
    for (int k = 0; k < RUN / 32; k++) s[32 * k + lane] = t[k];
    __syncwarp();
    if (lane >= 27) return;
    const int tap = lane;
    unsigned w[8], sb[2] = {127u, 127u};
    float v[32];
#pragma unroll
    for (int k = 0; k < 32; k++) v[k] = s[k * 27 + tap];
    sb[0] = mx_encode_row32<BITS>(v, w);
    if (BITS == 4) {
#pragma unroll
        for (int k = 0; k < 32; k++) v[k] = s[(32 + k) * 27 + tap];
        sb[1] = mx_encode_row32<4>(v, w + 4);
    }
    if (p.wpk) {
        int st, j;
        if (p.kind == UMX_CONV3) { st = 3 * ki + tap / 9; j = tap % 9; }
        else { const int it = tap * nitem + ki; st = it >> 2; j = it & 3; }
        const int ntile = row / p.nt, rl = row - ntile * p.nt;
        uint8_t *stg = p.wpk + ((size_t)ntile * p.nst + st) * p.w_stage_bytes;
        *(uint4 *)(stg + ((size_t)(j * 2) * p.nt + rl) * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        *(uint4 *)(stg + ((size_t)(j * 2 + 1) * p.nt + rl) * 16) = make_uint4(w[4], w[5], w[6], w[7]);
        uint8_t *sf = stg + (size_t)p.items_max * p.nt * 32;
        const int q = j / p.ipq, l = rl & 31, c = rl >> 5;
        if (BITS == 8) sf[q * 512 + l * 16 + c * 4 + (j & 3)] = (uint8_t)sb[0];
        else *(unsigned short *)(sf + q * 512 + l * 16 + c * 4 + (j & 1) * 2) = (unsigned short)(sb[0] | (sb[1] << 8));
    }
    if (r.wr) {
        const int nt = r.nt, R3 = 3 * nt, ct = row / nt, cl = row - ct * nt, dz = tap / 9, j = tap % 9;
        /* the rows of a tap in the order dz = 0, 1, 2, with scale images from each of them on; stride 2: dz = 0, 2, 1, with images of (0, 2), 2 and 1 */
        const bool s2 = p.kind == UMX_CONV3S2;
        const int rw = (s2 ? (3 - dz) % 3 : dz) * nt + cl;
        uint8_t *wr = r.wr + (size_t)ct * r.w_bytes, *base = wr + (size_t)(ki * 9 + j) * 2 * R3 * 16;
        *(uint4 *)(base + (size_t)rw * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        *(uint4 *)(base + (size_t)(R3 + rw) * 16) = make_uint4(w[4], w[5], w[6], w[7]);
        for (int d = s2 && dz == 1 ? 2 : 0; d <= (s2 ? (3 - dz) % 3 : dz); d++) {
            const int rr = rw - d * nt, g = rr >> 7, col = (rr & 127) >> 5, l = rr & 31, gb = d == 0 ? 0 : d == 1 ? r.goff1 : r.goff2;
            if (BITS == 8) wr[r.w_codes + ((ki * r.nquad + (j >> 2)) * r.gt + gb + g) * 512 + l * 16 + col * 4 + (j & 3)] = (uint8_t)sb[0];
            else *(unsigned short *)(wr + r.w_codes + ((ki * r.nquad + (j >> 1)) * r.gt + gb + g) * 512 + l * 16 + col * 4 + (j & 1) * 2) = (unsigned short)(sb[0] | (sb[1] << 8));
        }
    }
}

}   // namespace

/* p.wpk: the general kernel's image or NULL; wr: the z-marching kernel's or NULL; p.bias_p: the padded bias or NULL */
void umx_prep_w27(const PrepArgs &p, uint8_t *wr, int nt, int w_bytes, int w_codes, int gt, int goff1, int goff2) {
    const RImage r = {wr, nt, w_bytes, w_codes, p.bits == 8 ? 3 : 5, gt, goff1, goff2};      /* scale quads of nine taps */
    const int nitem = (p.ci + (p.bits == 8 ? 31 : 63)) / (p.bits == 8 ? 32 : 64);
    const dim3 grid((unsigned)p.cop, (unsigned)((nitem + 3) / 4));
    if (p.bits == 8) umx_launch(prep_w27_k<8>, grid, dim3(128), 0, p, r); else umx_launch(prep_w27_k<4>, grid, dim3(128), 0, p, r);
    g_umx_launches++;
}
