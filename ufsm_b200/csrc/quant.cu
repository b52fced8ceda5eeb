/* MX quantiser and inverse: plane-major fp32 / fp16 <-> channel-blocked MX-fp8 / MX-fp4 tensors.

   HBM-bound passes.  A thread owns one (n, block, voxel) row, so the amax that defines the row's scale is local: consecutive
   lanes own consecutive voxels, every channel plane is read in full sectors (32 lanes x 2 or 4 bytes), and a warp writes one
   contiguous run of rows (32 x 32 B or 32 x 16 B) plus 32 contiguous scale bytes.  Algorithmic bytes per element: read 4 or 2,
   write 1 + 1/32 (fp8) or 1/2 + 1/32 (fp4).  Semantics: src/lp_mx_cvt.cu:9-19, src/lp_mxops.cuh:46-68 of the reference. */
#include "mx_common.cuh"
#include <cuda_bf16.h>

__host__ __device__ static inline int mxbw(int C, int force) { return force > 0 ? force : C <= 8 ? 8 : C <= 16 ? 16 : 32; }

template <typename T> __device__ __forceinline__ float ld_as_f32(const T *p);
template <> __device__ __forceinline__ float ld_as_f32<float>(const float *p) { return ld_dep(p); }
template <> __device__ __forceinline__ float ld_as_f32<__half>(const __half *p) { return __half2float(ld_dep(p)); }
template <> __device__ __forceinline__ float ld_as_f32<__nv_bfloat16>(const __nv_bfloat16 *p) { return __uint_as_float((unsigned)ld_dep((const unsigned short *)p) << 16); }

/* grid = (voxel chunks, blocks, samples): no index division per row; consecutive threads take consecutive voxels, so the plane-major
   reads and the row writes are both coalesced.  Channels from c2 on come from a second tensor x2 of C - c2 channels (a conv's concat
   input, split_t.x2 / c_split of the reference: the 32-channel blocks run over the concatenated index); c2 = C without one. */
template <int BITS, typename TI, bool CAT>
__global__ void __launch_bounds__(256) pm_to_mx_k(const TI *x, uint8_t *__restrict__ y, int N, int C, size_t S, int bw, int split, const TI *x2, int c2) {
    pdl_trigger(); pdl_wait();
    const int nb = gridDim.y, blk = blockIdx.y, n = blockIdx.z, rb = bw * BITS / 8;
    const size_t rows = (size_t)N * nb * S, row0 = ((size_t)n * nb + blk) * S;
    uint8_t *sc = y + rows * rb;
    const TI *xb = x + ((size_t)n * c2 + (size_t)blk * bw) * S;                       /* channel k of the block: xb + k S while blk bw + k < c2 */
    const TI *xb2 = CAT ? x2 + ((ptrdiff_t)n * (C - c2) + (ptrdiff_t)blk * bw - c2) * (ptrdiff_t)S : nullptr;   /* and xb2 + k S from there on */
    const int nch = min(bw, C - blk * bw), k2 = c2 - blk * bw;
    for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < S; v += (size_t)gridDim.x * blockDim.x) {
        const size_t i = row0 + v;
        unsigned w[8]; unsigned sb;
        if (nch == 1) {
            /* a block with one real channel (a one-channel stem): the same bytes as the general path, without the 31 zero lanes */
            const float x0 = ld_as_f32((!CAT || 0 < k2 ? xb : xb2) + v);
            const int e = mx_exp(__uint_as_float(__float_as_uint(x0) & 0x7fffffffu), BITS == 4 ? 1.f / 6.f : 1.f / 448.f);
            const float m = exp2i(-e);
            sb = (unsigned)(e + 127) & 0xffu;
            const float z = 0.f * m;                     /* 0, or NaN for an inf / NaN block (scale byte 0xFF), as the general path gives */
            const unsigned zc = BITS == 8 ? cvt_e4m3x4(z, z, z, z) : cvt_e2m1x8((const float[8]){z, z, z, z, z, z, z, z}, 1.f);
#pragma unroll
            for (int k = 1; k < 8; k++) w[k] = zc;
            w[0] = BITS == 8 ? cvt_e4m3x4(x0 * m, z, z, z) : ((zc & ~0xfu) | (cvt_e2m1x2(x0 * m, z) & 0xfu));
        } else {
            float r[32];
            if (nch == 32 && (!CAT || k2 >= 32 || k2 <= 0)) {       /* a whole block of one tensor: 32 loads in flight */
                const TI *xp = (!CAT || k2 >= 32 ? xb : xb2) + v;
#pragma unroll
                for (int k = 0; k < 32; k++) { r[k] = ld_as_f32(xp); xp += S; }
            } else
#pragma unroll
            for (int k = 0; k < 32; k++) {
                if (CAT) r[k] = k < nch ? ld_as_f32((k < k2 ? xb : xb2) + (ptrdiff_t)k * (ptrdiff_t)S + v) : 0.f;
                else r[k] = k < nch ? ld_as_f32(xb + (size_t)k * S + v) : 0.f;
            }
            sb = mx_encode_row32<BITS>(r, w);
        }
        uint8_t *p = y + i * rb;
        if (BITS == 8) {
            if (bw == 32 && split) {   /* two 16-byte planes per block: [n][blk][half][voxel][16 B] */
                const size_t hp = ((size_t)n * nb + blk) * 2;
                *(uint4 *)(y + (hp * S + v) * 16) = make_uint4(w[0], w[1], w[2], w[3]); *(uint4 *)(y + ((hp + 1) * S + v) * 16) = make_uint4(w[4], w[5], w[6], w[7]);
            } else if (bw == 32) { ((uint4 *)p)[0] = make_uint4(w[0], w[1], w[2], w[3]); ((uint4 *)p)[1] = make_uint4(w[4], w[5], w[6], w[7]); }
            else if (bw == 16) ((uint4 *)p)[0] = make_uint4(w[0], w[1], w[2], w[3]);
            else ((uint2 *)p)[0] = make_uint2(w[0], w[1]);
        } else {
            if (bw == 32) ((uint4 *)p)[0] = make_uint4(w[0], w[1], w[2], w[3]);
            else if (bw == 16) ((uint2 *)p)[0] = make_uint2(w[0], w[1]);
            else ((unsigned *)p)[0] = w[0];
        }
        sc[i] = (uint8_t)sb;
    }
}
/* Whole 32-channel blocks of one fp16 tensor, two neighbouring voxels a thread: a plane's pair is one 4-byte load (a warp reads 128 contiguous
   bytes), and the two rows are measured, scaled and converted together on packed halves, which is exact while both block scales are normal
   fp16 numbers (below 2^-14 a scaled value rounds to zero either way); other rows take the fp32 path.  Bytes as mx_encode_row32 of the
   values converted to fp32.  Bound by latency and the memory rate: 32 channels x 64^3 into MX-fp8 16.4 us at one voxel and 32 predicated
   2-byte loads a thread, 5.6 us in this form. */
template <int BITS>
__global__ void __launch_bounds__(128) h16_to_mx_pair_k(const __half *x, uint8_t *__restrict__ y, int N, int C, size_t S, int split) {
    pdl_trigger(); pdl_wait();
    const int nb = gridDim.y, blk = blockIdx.y, n = blockIdx.z;
    constexpr int RB = 32 * BITS / 8;
    const size_t row0 = ((size_t)n * nb + blk) * S, S2 = S >> 1;
    const unsigned *xb = (const unsigned *)(x + ((size_t)n * C + (size_t)blk * 32) * S);
    uint8_t *sc = y + (size_t)N * nb * S * RB;
    for (size_t v2 = blockIdx.x * (size_t)128 + threadIdx.x; v2 < S2; v2 += (size_t)gridDim.x * 128) {
        unsigned raw[32];
#pragma unroll
        for (int k = 0; k < 32; k++) raw[k] = ld_dep(xb + (size_t)k * S2 + v2);
        const __half2 *h = (const __half2 *)raw;
        __half2 a2 = __habs2(h[0]);
#pragma unroll
        for (int k = 1; k < 32; k++) a2 = __hmax2_nan(a2, __habs2(h[k]));
        const float2 am = __half22float2(a2);
        const mx_sb q0 = mx_scale_of(am.x, BITS == 4 ? 1.f / 6.f : 1.f / 448.f), q1 = mx_scale_of(am.y, BITS == 4 ? 1.f / 6.f : 1.f / 448.f);
        unsigned w0[8], w1[8];
        if (q0.sb - 112u <= 29u && q1.sb - 112u <= 29u) {          /* -15 <= e <= 14 */
            const unsigned mm = ((142u - q0.sb) << 10) | ((142u - q1.sb) << 26);
            const __half2 m2 = *(const __half2 *)&mm;
#pragma unroll
            for (int j = 0; j < 32 * BITS / 32; j++) {              /* one word of codes a row */
                constexpr int CW = 32 / BITS;                       /* channels a word */
                unsigned s[CW];
#pragma unroll
                for (int k = 0; k < CW; k++) { const __half2 t = __hmul2(h[CW * j + k], m2); s[k] = *(const unsigned *)&t; }
                if (BITS == 8) {
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const unsigned p0 = __byte_perm(s[0], s[1], u ? 0x7632 : 0x5410), p1 = __byte_perm(s[2], s[3], u ? 0x7632 : 0x5410);
                        unsigned short c0, c1;
                        asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(c0) : "r"(p0));
                        asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(c1) : "r"(p1));
                        const unsigned w = (unsigned)c0 | ((unsigned)c1 << 16);
                        if (u) w1[j] = w; else w0[j] = w;
                    }
                } else {
                    float2 f[CW];
#pragma unroll
                    for (int k = 0; k < CW; k++) f[k] = __half22float2(*(const __half2 *)&s[k]);
                    w0[j] = cvt_e2m1_word(f[0].x, f[1].x, f[2].x, f[3].x, f[4 % CW].x, f[5 % CW].x, f[6 % CW].x, f[7 % CW].x);
                    w1[j] = cvt_e2m1_word(f[0].y, f[1].y, f[2].y, f[3].y, f[4 % CW].y, f[5 % CW].y, f[6 % CW].y, f[7 % CW].y);
                }
            }
        } else {
            float r[32];
#pragma unroll
            for (int k = 0; k < 32; k++) r[k] = __low2float(h[k]);
            mx_encode_row32<BITS>(r, w0);
#pragma unroll
            for (int k = 0; k < 32; k++) r[k] = __high2float(h[k]);
            mx_encode_row32<BITS>(r, w1);
        }
        const size_t v = 2 * v2;
        if (BITS == 8 && split) {
            uint4 *p = (uint4 *)(y + (row0 * 2 + v) * 16), *ph = (uint4 *)(y + (row0 * 2 + S + v) * 16);
            p[0] = make_uint4(w0[0], w0[1], w0[2], w0[3]); p[1] = make_uint4(w1[0], w1[1], w1[2], w1[3]);
            ph[0] = make_uint4(w0[4], w0[5], w0[6], w0[7]); ph[1] = make_uint4(w1[4], w1[5], w1[6], w1[7]);
        } else if (BITS == 8) {
            uint4 *p = (uint4 *)(y + (row0 + v) * 32);
            p[0] = make_uint4(w0[0], w0[1], w0[2], w0[3]); p[1] = make_uint4(w0[4], w0[5], w0[6], w0[7]);
            p[2] = make_uint4(w1[0], w1[1], w1[2], w1[3]); p[3] = make_uint4(w1[4], w1[5], w1[6], w1[7]);
        } else {
            uint4 *p = (uint4 *)(y + (row0 + v) * 16);
            p[0] = make_uint4(w0[0], w0[1], w0[2], w0[3]); p[1] = make_uint4(w1[0], w1[1], w1[2], w1[3]);
        }
        *(unsigned short *)(sc + row0 + v) = (unsigned short)(q0.sb | (q1.sb << 8));
    }
}

/* One 32-wide row a thread: its codes in 16-byte loads, decoded by the hardware conversion to halves (exact), each channel's plane written 128
   bytes a warp.  grid (voxels, blocks, samples).  Rows of 8 or 16 channels take mx_to_pm_k.  64 channels x 48^3 15.0 us with a decode in integer
   arithmetic and three index divisions a row, 5.3 us in this form. */
template <int BITS>
__global__ void __launch_bounds__(128) mx32_to_pm_k(const uint8_t *x, float *__restrict__ y, int N, int C, size_t S, int split) {
    pdl_trigger(); pdl_wait();
    const int nb = gridDim.y, blk = blockIdx.y, n = blockIdx.z;
    constexpr int RB = 32 * BITS / 8;
    const size_t row0 = ((size_t)n * nb + blk) * S;
    const uint8_t *sc = x + (size_t)N * nb * S * RB;
    float *yb = y + ((size_t)n * C + (size_t)blk * 32) * S;
    const int nch = min(32, C - blk * 32);
    for (size_t v = blockIdx.x * (size_t)128 + threadIdx.x; v < S; v += (size_t)gridDim.x * 128) {
        uint4 q[RB / 16];
#pragma unroll
        for (int h = 0; h < RB / 16; h++) q[h] = ld_dep((const uint4 *)(x + (BITS == 8 && split ? (row0 * 2 + h * S + v) * 16 : (row0 + v) * RB + h * 16)));
        const float s = mx_scale(ld_dep(sc + row0 + v));
        const unsigned *w = (const unsigned *)q;
        float e[32];
#pragma unroll
        for (int j = 0; j < RB / 4; j++) { if (BITS == 8) dec_e4m3x4(w[j], e + 4 * j); else dec_e2m1x8(w[j], e + 8 * (j & 3)); }
        float *p = yb + v;
        if (nch == 32) {
#pragma unroll
            for (int k = 0; k < 32; k++) { *p = e[k] * s; p += S; }
        } else {
#pragma unroll
            for (int k = 0; k < 32; k++) if (k < nch) { *p = e[k] * s; p += S; }
        }
    }
}
template <int BITS>
__global__ void __launch_bounds__(256) mx_to_pm_k(const uint8_t *__restrict__ x, float *__restrict__ y, int N, int C, size_t S, int bw, int split) {
    const int nb = (C + bw - 1) / bw, rb = bw * BITS / 8;
    const size_t rows = (size_t)N * nb * S;
    const uint8_t *sc = x + rows * rb;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < rows; i += (size_t)gridDim.x * blockDim.x) {
        const size_t v = i % S; const int blk = (int)((i / S) % nb), n = (int)(i / (S * nb));
        const float s = mx_scale(sc[i]);
        const uint8_t *p = x + i * rb;
        for (int k = 0; k < bw; k++) {
            const int c = blk * bw + k; if (c >= C) break;
            const float e = BITS == 8 ? dec_e4m3(split ? x[(((i / S) * 2 + (k >> 4)) * S + v) * 16 + (k & 15)] : p[k]) : dec_e2m1((p[k >> 1] >> ((k & 1) * 4)) & 15u);
            y[((size_t)n * C + c) * S + v] = e * s;
        }
    }
}
__global__ void __launch_bounds__(256) h16b_to_pm_k(const __half *__restrict__ x, float *__restrict__ y, int N, int C, size_t S) {
    const int nb = (C + 31) / 32;
    const size_t rows = (size_t)N * nb * S;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < rows; i += (size_t)gridDim.x * blockDim.x) {
        const size_t v = i % S; const int blk = (int)((i / S) % nb), n = (int)(i / (S * nb));
        for (int k = 0; k < 32; k++) { const int c = blk * 32 + k; if (c >= C) break; y[((size_t)n * C + c) * S + v] = __half2float(x[i * 32 + k]); }
    }
}

static unsigned grid_for(size_t rows) { size_t g = (rows + 255) / 256; return (unsigned)(g > 148u * 64u ? 148u * 64u : g ? g : 1); }

static void to_mx(const void *x, int dt, int N, int C, size_t S, void *y, int bits, int bwf, const char *who, int split = 0, const void *x2 = nullptr, int c2 = 0) {
    if (!umx_ready(who)) return;
    if (dt != 0 && dt != 1 && dt != 2) { fprintf(stderr, "%s: source type %d is not built (fp32, bf16 and fp16 only)\n", who, dt); abort(); }
    if (!x2) c2 = C;
    const int bw = mxbw(C, bwf);
    const int nb = (C + bw - 1) / bw;
    if (!S || !N) return;
    /* blocks per (block, sample): 16 per multiprocessor; a tensor of one channel (2 bytes read per 33 written: the network input) runs a
       third faster with two (measured: 31 against 42 us for 128^3) */
    if (dt == 2 && !x2 && bw == 32 && !(C & 31) && !(S & 1) && !((size_t)x & 3) && !((size_t)y & 15)) {      /* pairs of voxels are aligned in every plane */
        size_t gp = (S / 2 + 127) / 128; if (gp > 148u * 64u) gp = 148u * 64u;
        const dim3 g2((unsigned)gp, (unsigned)nb, (unsigned)N);
        if (bits == 8) umx_launch(h16_to_mx_pair_k<8>, g2, dim3(128), 0, (const __half *)x, (uint8_t *)y, N, C, S, split);
        else umx_launch(h16_to_mx_pair_k<4>, g2, dim3(128), 0, (const __half *)x, (uint8_t *)y, N, C, S, split);
        g_umx_launches++;
        UMX_CK(who);
        return;
    }
    const size_t cap = C == 1 ? 148u * 2u : 148u * 16u;
    size_t gx = (S + 255) / 256; if (gx > cap) gx = cap;
    const dim3 g((unsigned)gx, (unsigned)nb, (unsigned)N);
#define UMX_Q(B, T) do { if (x2) umx_launch(pm_to_mx_k<B, T, true>, g, dim3(256), 0, (const T *)x, (uint8_t *)y, N, C, S, bw, split, (const T *)x2, c2); \
                         else umx_launch(pm_to_mx_k<B, T, false>, g, dim3(256), 0, (const T *)x, (uint8_t *)y, N, C, S, bw, split, (const T *)x2, c2); } while (0)
    if (bits == 8) { if (dt == 2) UMX_Q(8, __half); else if (dt == 1) UMX_Q(8, __nv_bfloat16); else UMX_Q(8, float); }
    else { if (dt == 2) UMX_Q(4, __half); else if (dt == 1) UMX_Q(4, __nv_bfloat16); else UMX_Q(4, float); }
#undef UMX_Q
    g_umx_launches++;
    UMX_CK(who);
}
static void from_mx(const void *x, int N, int C, size_t S, float *y, int bits, int bwf, const char *who, int split = 0) {
    if (!umx_ready(who)) return;
    const int bw = mxbw(C, bwf);
    const size_t rows = (size_t)N * ((C + bw - 1) / bw) * S;
    if (!rows) return;
    if (bw == 32 && N <= 65535 && C <= 65535 * 32 && !((size_t)x & 15)) {
        size_t gx = (S + 127) / 128; if (gx > 148u * 64u) gx = 148u * 64u;
        const dim3 g2((unsigned)gx, (unsigned)((C + 31) / 32), (unsigned)N);
        if (bits == 8) umx_launch(mx32_to_pm_k<8>, g2, dim3(128), 0, (const uint8_t *)x, y, N, C, S, split);
        else umx_launch(mx32_to_pm_k<4>, g2, dim3(128), 0, (const uint8_t *)x, y, N, C, S, split);
        g_umx_launches++;
        UMX_CK(who);
        return;
    }
    if (bits == 8) mx_to_pm_k<8><<<grid_for(rows), 256>>>((const uint8_t *)x, y, N, C, S, bw, split);
    else mx_to_pm_k<4><<<grid_for(rows), 256>>>((const uint8_t *)x, y, N, C, S, bw, split);
    g_umx_launches++;
    UMX_CK(who);
}
extern "C" size_t lp_mx8_bytes(int N, int C, size_t S) { const int bw = mxbw(C, 0); return (size_t)N * ((C + bw - 1) / bw) * S * (bw + 1); }
extern "C" size_t lp_mx4_bytes(int N, int C, size_t S) { const int bw = mxbw(C, 0); return (size_t)N * ((C + bw - 1) / bw) * S * (bw / 2 + 1); }
extern "C" size_t umx_mx_bytes32(int bits, int N, int C, size_t S) { return (size_t)N * ((C + 31) / 32) * S * (32 * bits / 8 + 1); }
extern "C" void lp_f32_to_mx8(const float *x, int N, int C, size_t S, void *y) { to_mx(x, 0, N, C, S, y, 8, 0, "lp_f32_to_mx8"); }
extern "C" void lp_f32_to_mx4(const float *x, int N, int C, size_t S, void *y) { to_mx(x, 0, N, C, S, y, 4, 0, "lp_f32_to_mx4"); }
extern "C" void lp_h16_to_mx8(const void *x, int dt, int N, int C, size_t S, void *y) { to_mx(x, dt, N, C, S, y, 8, 0, "lp_h16_to_mx8"); }
extern "C" void lp_h16_to_mx4(const void *x, int dt, int N, int C, size_t S, void *y) { to_mx(x, dt, N, C, S, y, 4, 0, "lp_h16_to_mx4"); }
extern "C" void lp_mx8_to_f32(const void *x, int N, int C, size_t S, float *y) { from_mx(x, N, C, S, y, 8, 0, "lp_mx8_to_f32"); }
extern "C" void lp_mx4_to_f32(const void *x, int N, int C, size_t S, float *y) { from_mx(x, N, C, S, y, 4, 0, "lp_mx4_to_f32"); }
extern "C" void umx_pm_to_mx32(const void *x, int dt, int N, int C, size_t S, void *y, int bits, int layout) { to_mx(x, dt, N, C, S, y, bits, 32, "umx_pm_to_mx32", layout == UMX_LAYOUT_SPLIT && bits == 8); }
/* the same from two tensors: channels [0, c2) of the C from x, the rest from x2 */
extern "C" void umx_pm_to_mx32_cat(const void *x, const void *x2, int c2, int dt, int N, int C, size_t S, void *y, int bits, int layout) {
    if (x2 && (c2 < 1 || c2 >= C)) { fprintf(stderr, "umx_pm_to_mx32_cat: split at channel %d of %d\n", c2, C); abort(); }
    to_mx(x, dt, N, C, S, y, bits, 32, "umx_pm_to_mx32_cat", layout == UMX_LAYOUT_SPLIT && bits == 8, x2, c2);
}
extern "C" void umx_mx32_to_f32(const void *x, int bits, int N, int C, size_t S, float *y, int layout) { from_mx(x, N, C, S, y, bits, 32, "umx_mx32_to_f32", layout == UMX_LAYOUT_SPLIT && bits == 8); }
extern "C" void umx_h16b_to_f32(const void *x, int N, int C, size_t S, float *y) {
    if (!umx_ready("umx_h16b_to_f32")) return;
    h16b_to_pm_k<<<grid_for((size_t)N * ((C + 31) / 32) * S), 256>>>((const __half *)x, y, N, C, S);
    g_umx_launches++;
    UMX_CK("umx_h16b_to_f32");
}

/* MX-fp8 codes between the reference layout [n][blk][voxel][32 B] and the split layout [n][blk][half][voxel][16 B].  grid (voxels, blocks of all
   samples): a thread moves half rows 2 v + h of its block, consecutive threads consecutive 16-byte pieces of the reference layout */
__global__ void __launch_bounds__(256) relayout8_k(const uint4 *src, uint4 *__restrict__ dst, size_t blocks, size_t S, int to_split) {
    pdl_trigger(); pdl_wait();
    for (size_t b = blockIdx.y; b < blocks; b += gridDim.y) {
        const uint4 *s = src + b * 2 * S; uint4 *d = dst + b * 2 * S;
        for (size_t i = blockIdx.x * (size_t)1024 + threadIdx.x; i < 2 * S; i += (size_t)gridDim.x * 1024) {
            uint4 t[4];
#pragma unroll
            for (int k = 0; k < 4; k++) { const size_t j = i + 256 * k; if (j < 2 * S) t[k] = ld_dep(s + (to_split ? j : (j & 1) * S + (j >> 1))); }
#pragma unroll
            for (int k = 0; k < 4; k++) { const size_t j = i + 256 * k; if (j < 2 * S) d[to_split ? (j & 1) * S + (j >> 1) : j] = t[k]; }
        }
    }
}
static void relayout8(const void *src, void *dst, size_t blocks, size_t S, int to_split) {
    size_t gx = (2 * S + 1023) / 1024; if (gx > 148u * 16u) gx = 148u * 16u;
    umx_launch(relayout8_k, dim3((unsigned)gx, (unsigned)(blocks < 65535 ? blocks : 65535)), dim3(256), 0, (const uint4 *)src, (uint4 *)dst, blocks, S, to_split);
    g_umx_launches++;
}
/* the codes alone, into the split layout (a conv's MX-fp8 operand of the reference interface) */
void umx_mx_codes_to_split(const void *x, size_t blocks, size_t S, void *y) {
    if (!blocks || !S) return;
    relayout8(x, y, blocks, S, 1);
    UMX_CK("umx_mx_codes_to_split");
}
extern "C" void umx_mx_relayout(const void *src, int bits, int N, int C, size_t S, void *dst, int to_layout) {
    if (!umx_ready("umx_mx_relayout")) return;
    const size_t blocks = (size_t)N * ((C + 31) / 32), rows = blocks * S, rb = bits == 8 ? 32 : 16;
    if (!rows) return;
    if (bits == 8) relayout8(src, dst, blocks, S, to_layout == UMX_LAYOUT_SPLIT);
    else cudaMemcpyAsync(dst, src, rows * rb, cudaMemcpyDeviceToDevice, 0);
    cudaMemcpyAsync((uint8_t *)dst + rows * rb, (const uint8_t *)src + rows * rb, rows, cudaMemcpyDeviceToDevice, 0);
    UMX_CK("umx_mx_relayout");
}
/* blocks of an MX tensor (32-wide rows, reference layout, nb_src blocks a sample) to blocks [b0, b0 + nb_src) of one of nb_dst blocks, codes and scale
   bytes in one launch; to_split: MX-fp8 codes into the split layout.  The part of a conv's concat input that needs no transform. */
template <int RB>
__global__ void __launch_bounds__(256) mx_blocks_put_k(const uint8_t *src, uint8_t *__restrict__ dst, int N, int nb_src, int nb_dst, int b0, size_t S, int to_split) {
    pdl_trigger(); pdl_wait();
    const int blk = blockIdx.y, n = blockIdx.z;
    const size_t sb = (size_t)n * nb_src + blk, db = (size_t)n * nb_dst + b0 + blk;
    const uint8_t *ss = src + (size_t)N * nb_src * S * RB + sb * S; uint8_t *ds = dst + (size_t)N * nb_dst * S * RB + db * S;
    const uint4 *s = (const uint4 *)(src + sb * S * RB); uint4 *d = (uint4 *)(dst + db * S * RB);
    for (size_t v = blockIdx.x * (size_t)256 + threadIdx.x; v < S; v += (size_t)gridDim.x * 256) {
        const uint4 a = ld_dep(s + v * (RB / 16)), b = RB == 32 ? ld_dep(s + v * 2 + 1) : a;
        const uint8_t e = ld_dep(ss + v);
        if (RB == 32 && to_split) { d[v] = a; d[S + v] = b; }
        else if (RB == 32) { d[2 * v] = a; d[2 * v + 1] = b; }
        else d[v] = a;
        ds[v] = e;
    }
}
void umx_mx_blocks_put(const void *src, int bits, int N, int nb_src, size_t S, void *dst, int nb_dst, int b0, int to_split) {
    if (!N || !nb_src || !S) return;
    size_t gx = (S + 255) / 256; if (gx > 148u * 16u) gx = 148u * 16u;
    const dim3 g((unsigned)gx, (unsigned)nb_src, (unsigned)N);
    if (bits == 8) umx_launch(mx_blocks_put_k<32>, g, dim3(256), 0, (const uint8_t *)src, (uint8_t *)dst, N, nb_src, nb_dst, b0, S, to_split);
    else umx_launch(mx_blocks_put_k<16>, g, dim3(256), 0, (const uint8_t *)src, (uint8_t *)dst, N, nb_src, nb_dst, b0, S, to_split);
    g_umx_launches++;
    UMX_CK("umx_mx_blocks_put");
}

/* MX tensors of 16 channels or fewer keep rows of 8 or 16 channels in the reference's storage (src/lp_common.cuh:132-134).  Such a row
   and the 32-wide row holding the same channels followed by zeros have the same amax, hence the same scale byte and the same codes:
   widening and narrowing are copies.  One thread per row. */
__global__ void __launch_bounds__(256) mx_rewidth_k(const uint8_t *src, uint8_t *__restrict__ dst, size_t rows, int rb_src, int rb_dst) {
    pdl_trigger(); pdl_wait();
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < rows; i += (size_t)gridDim.x * blockDim.x) {
        const unsigned *s = (const unsigned *)(src + i * rb_src); unsigned *d = (unsigned *)(dst + i * rb_dst);
        for (int k = 0; k < rb_dst / 4; k++) d[k] = k < rb_src / 4 ? ld_dep(s + k) : 0u;
        dst[rows * rb_dst + i] = ld_dep(src + rows * rb_src + i);
    }
}
/* x: an MX tensor of C <= 16 channels (one block of 8 or 16 a voxel) -> y: the same tensor with 32-wide rows (to_wide), or back */
extern "C" void umx_mx_rewidth(const void *x, int bits, int N, int C, size_t S, void *y, int to_wide) {
    if (!umx_ready("umx_mx_rewidth")) return;
    if (C < 1 || C > 16 || (bits != 8 && bits != 4)) { fprintf(stderr, "umx_mx_rewidth: %d channels, %d bits\n", C, bits); abort(); }
    const int bw = mxbw(C, 0), rn = bw * bits / 8, r32 = 32 * bits / 8;
    const size_t rows = (size_t)N * S;
    if (!rows) return;
    umx_launch(mx_rewidth_k, dim3(grid_for(rows)), dim3(256), 0, (const uint8_t *)x, (uint8_t *)y, rows, to_wide ? rn : r32, to_wide ? r32 : rn);
    g_umx_launches++;
    UMX_CK("umx_mx_rewidth");
}

/* lp_pred_input_mx (src/nn_lp.h:164-165, src/lp_mx_cvt.cu:20-57): the network input of the reference's predict for window planes
   [z0, z0 + nz) of a W x W x depth CT window: channel 0 the z-scored CT byte, 1 zero, 2 and 3 the unit direction away from the scroll
   axis (dy, dx) (axis 0: zeros; -1 flips it), each rounded to the 16-bit input type (hd 2 fp16, 1 bf16, 0 none), stored as MX rows of
   one 8-channel block.  The radius is sqrt(fma(dy, dy, dx dx)) + 1e-6: the contraction a compiler picks for dy dy + dx dx, spelled out. */
template <int HD> __device__ __forceinline__ float round16(float v) {
    if (HD == 2) return __half2float(__float2half_rn(v));
    if (HD == 1) return __bfloat162float(__float2bfloat16_rn(v));
    return v;
}
template <int HD> __device__ __forceinline__ float2 round16x2(float a, float b) {
    if (HD == 2) return __half22float2(__floats2half2_rn(a, b));
    return make_float2(round16<HD>(a), round16<HD>(b));
}
/* grid (runs of 1024 voxels of a plane, groups of planes): a warp takes 128 consecutive voxels of the plane, four a lane 32 apart, so loads and
   stores are coalesced, and a lane works its coordinates out once for all planes of its group.  The row has three channels that are not
   zero by construction, so only those are measured and encoded.  Bound by instruction issue, a third of it the IEEE square root and division
   a voxel: 192^3 50.8 us with a 32-channel encode and 64-bit index divisions a voxel, 25 us in this form (1 B read, 9 B written). */
template <int BITS, int HD>
__global__ void __launch_bounds__(256) pred_input_k(const uint8_t *ct, int W, float mean, float isd, const float *dyo, const float *dxo,
                                                    int axis, int z0, int nz, uint8_t *__restrict__ y) {
    pdl_trigger(); pdl_wait();
    const unsigned plane = (unsigned)W * (unsigned)W;
    const unsigned p0 = blockIdx.x * 1024u + (threadIdx.x >> 5) * 128u + (threadIdx.x & 31u);
    if (p0 >= plane) return;
    float fy[4], fx[4];
    {
        int yy = (int)(p0 / (unsigned)W), xx = (int)(p0 - (unsigned)yy * (unsigned)W);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            fy[k] = (float)yy; fx[k] = (float)xx;
            xx += 32;
            while (xx >= W) { xx -= W; yy++; }
        }
    }
    const float fa = (float)axis;
    const uint8_t *cp = ct + (size_t)(z0 + (int)blockIdx.y) * plane + p0;
    uint8_t *yp = y + ((size_t)blockIdx.y * plane + p0) * BITS, *sp = y + (size_t)nz * plane * BITS + (size_t)blockIdx.y * plane + p0;   /* a row is BITS bytes: eight channels */
    const size_t step = (size_t)gridDim.y * plane;
    for (int zl = blockIdx.y; zl < nz; zl += gridDim.y, cp += step, yp += step * BITS, sp += step) {
        const float oy = ld_dep(dyo + z0 + zl), ox = ld_dep(dxo + z0 + zl);
        unsigned cv[4];
#pragma unroll
        for (int k = 0; k < 4; k++) cv[k] = p0 + 32 * k < plane ? ld_dep(cp + 32 * k) : 0u;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float dy = __fadd_rn(oy, fy[k]), dx = __fadd_rn(ox, fx[k]);
            const float inv = axis ? __fdiv_rn(fa, __fadd_rn(__fsqrt_rn(__fmaf_rn(dy, dy, __fmul_rn(dx, dx))), 1e-6f)) : 0.f;
            /* the byte as a float without the conversion unit (2^23 + byte, minus 2^23) */
            const float r0 = round16<HD>(__fmul_rn(__fsub_rn(__fsub_rn(__uint_as_float(0x4b000000u | cv[k]), 8388608.f), mean), isd));
            const float2 r23 = round16x2<HD>(__fmul_rn(dy, inv), __fmul_rn(dx, inv));
            const int e = mx_exp(__uint_as_float(amax_u(amax_u(amax_u(0u, r0), r23.x), r23.y)), BITS == 4 ? 1.f / 6.f : 1.f / 448.f);
            const float m = exp2i(-e);
            unsigned c01, c23, z2 = 0u;                               /* codes of channels 0 and 1, 2 and 3, and of a pair of zero channels */
            if (BITS == 8) { c01 = cvt_e4m3x4(r0 * m, 0.f * m, r23.x * m, r23.y * m); c23 = c01 >> 16; c01 &= 0xffffu; if (e == 128) z2 = cvt_e4m3x4(0.f * m, 0.f * m, 0.f * m, 0.f * m); }
            else { c01 = cvt_e2m1x2(r0 * m, 0.f * m); c23 = cvt_e2m1x2(r23.x * m, r23.y * m); if (e == 128) z2 = cvt_e2m1x2(0.f * m, 0.f * m); }   /* an inf / NaN row: 0 times its scale is NaN, as the 32-channel encode gives */
            if (p0 + 32 * k < plane) {
                if (BITS == 8) *(uint2 *)(yp + 32 * k * 8) = make_uint2(c01 | (c23 << 16), z2);
                else *(unsigned *)(yp + 32 * k * 4) = c01 | (c23 << 8) | (z2 << 16) | (z2 << 24);
                sp[32 * k] = (uint8_t)(e + 127);
            }
        }
    }
}
extern "C" void lp_pred_input_mx(const uint8_t *ct, int W, float mean, float isd, const float *dyo, const float *dxo, int axis, int z0, int nz, void *y, int hd, int bits) {
    if (!umx_ready("lp_pred_input_mx")) return;
    if ((bits != 8 && bits != 4) || hd < 0 || hd > 2) { fprintf(stderr, "lp_pred_input_mx: %d bits, 16-bit type %d\n", bits, hd); abort(); }
    const size_t S = (size_t)(nz > 0 ? nz : 0) * W * W;
    if (!S) return;
    if (W > 46340) { fprintf(stderr, "lp_pred_input_mx: planes of %d x %d voxels\n", W, W); abort(); }
    /* groups of planes: one wave of the six blocks that a multiprocessor holds, at most one group a plane */
    const unsigned gx = (unsigned)(((size_t)W * W + 1023) / 1024), gy = 148u * 6u / gx < 1 ? 1 : 148u * 6u / gx;
    const dim3 g(gx, gy < (unsigned)nz ? gy : (unsigned)nz);
#define UMX_PI(B, H) umx_launch(pred_input_k<B, H>, g, dim3(256), 0, ct, W, mean, isd, dyo, dxo, axis, z0, nz, (uint8_t *)y)
    if (bits == 8) { if (hd == 2) UMX_PI(8, 2); else if (hd == 1) UMX_PI(8, 1); else UMX_PI(8, 0); }
    else { if (hd == 2) UMX_PI(4, 2); else if (hd == 1) UMX_PI(4, 1); else UMX_PI(4, 0); }
#undef UMX_PI
    g_umx_launches++;
    UMX_CK("lp_pred_input_mx");
}
extern "C" void lp_pred_input_mx8(const uint8_t *ct, int W, float mean, float isd, const float *dyo, const float *dxo, int axis, int z0, int nz, void *y, int hd) {
    lp_pred_input_mx(ct, W, mean, isd, dyo, dxo, axis, z0, nz, y, hd, 8);
}
