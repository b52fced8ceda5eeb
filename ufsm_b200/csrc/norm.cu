/* InstanceNorm coefficients from the conv epilogue's partial sums, and the fused apply: y = fp16(LeakyReLU(x a + b)) requantised
   to MX for the next conv.  HBM-bound: the apply reads 2 B and writes 1 + 1/32 B (fp8) or 1/2 + 1/32 B (fp4) per element (twice
   that when the space-to-depth copy for a down conv is also written).  Semantics: k_in_coef and k_inq of the reference
   (src/nn_xnet.cu:1565-1570, 1577-1620) with 32-channel UE8M0 blocks. */
#include "mx_common.cuh"
#include "tc_ptx.cuh"
#include <string.h>

/* mean and variance of S values to the coefficients (a, b) of an affine map (k_in_coef, src/nn_xnet.cu:1565-1570) */
__device__ __forceinline__ float2 coef_of(double sum, double sq, double S, float eps, const float *gamma, const float *beta, int c) {
    const double m = sum / S, v = fmax(sq / S - m * m, 0.0);
    const float rs = (float)(1.0 / sqrt(v + (double)eps)), ca = __fmul_rn(rs, gamma ? gamma[c] : 1.f);
    return make_float2(ca, __fmaf_rn(-(float)m, ca, beta ? beta[c] : 0.f));
}

/* partial sums: part[((n * T + t) * Cop + c) * 2 + {0, 1}], T voxel chunks, Cop = C rounded up to 32.  One block per (c, n); the
   chunk sums are added in a fixed order (strided per thread, then a fixed tree), so the result does not depend on scheduling. */
__global__ void __launch_bounds__(256) in_coef_k(const double *__restrict__ part, int C, int Cop, int T, double S, const float *gamma, const float *beta, float eps, float *coef) {
    const int c = blockIdx.x, n = blockIdx.y;
    double s = 0.0, q = 0.0;
    for (int t = threadIdx.x; t < T; t += 256) { const double *p = part + (((size_t)n * T + t) * Cop + c) * 2; s += p[0]; q += p[1]; }
    __shared__ double ss[256], sq[256];
    ss[threadIdx.x] = s; sq[threadIdx.x] = q;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) { if ((int)threadIdx.x < o) { ss[threadIdx.x] += ss[threadIdx.x + o]; sq[threadIdx.x] += sq[threadIdx.x + o]; } __syncthreads(); }
    if (threadIdx.x == 0) {
        const float2 ab = coef_of(ss[0], sq[0], S, eps, gamma, beta, c);
        coef[2 * ((size_t)n * C + c)] = ab.x;
        coef[2 * ((size_t)n * C + c) + 1] = ab.y;
    }
}
extern "C" void umx_in_coef(const double *part, int N, int C, int D, int H, int W, const float *gamma, const float *beta, float eps, float *coef);
/* voxel chunks per (sample, channel) of the partial sums: about 1024 voxels each, at most 444 (three blocks on each of 148 multiprocessors), a
   multiple of 111 where there are that many, so that two or four channel blocks or samples make whole waves too */
int umx_stats_chunks(int D, int H, int W) { const size_t S = (size_t)D * H * W; const size_t t = S / 1024; return t < 1 ? 1 : t >= 444 ? 444 : t >= 111 ? (int)t / 111 * 111 : (int)t; }

/* fp16 values to fp64 sums and sums of squares: exact to the last bits whatever the order */
struct StatAcc { double s[8], q[8]; };
__device__ __forceinline__ void stat_zero(StatAcc &a) {
#pragma unroll
    for (int k = 0; k < 8; k++) { a.s[k] = 0.0; a.q[k] = 0.0; }
}
__device__ __forceinline__ void stat_add(StatAcc &a, const uint4 &r) {
    const __half2 *h = (const __half2 *)&r;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float2 f = __half22float2(h[k]);
        const double d0 = (double)f.x, d1 = (double)f.y;
        a.s[2 * k] += d0; a.q[2 * k] = fma(d0, d0, a.q[2 * k]); a.s[2 * k + 1] += d1; a.q[2 * k + 1] = fma(d1, d1, a.q[2 * k + 1]);
    }
}
/* partial sums of chunk t of block blk of sample n of a blocked fp16 tensor: part[((n * T + t) * Cop + c) * 2 + {0, 1}].  A thread owns
   eight channels (one 16-byte load) of every 64th voxel of the chunk, eight loads in flight, so a warp reads 512 contiguous bytes per
   load; the 64 phases are added in a fixed order.  fp64 throughout: sums of fp16 values and of their squares are then exact to the
   last bits whatever the order.  HBM-bound: reads 2 B per element. */
/* tickets of the fused finalise: one counter per (sample, block); the block that draws the last ticket finalises and resets it */
__device__ unsigned g_stat_tickets[8192];

template <bool FINAL>
__global__ void __launch_bounds__(256, 3) in_part_k(const uint4 *y, size_t S, int T, double *__restrict__ part,
                                                 int C, const float *gamma, const float *beta, float eps, float *coef) {
    pdl_trigger(); pdl_wait();
    const int t = blockIdx.x, blk = blockIdx.y, n = blockIdx.z, nb = gridDim.y, Cop = nb * 32;
    const int qd = threadIdx.x & 3, ph = threadIdx.x >> 2;
    const uint4 *p = y + ((size_t)n * nb + blk) * S * 4 + qd;
    StatAcc acc;
    stat_zero(acc);
    auto add = [&](const uint4 &r) { stat_add(acc, r); };
    /* all blocks sweep the tensor together, 256 voxels a block and trip, from its end to its start: the conv before left its end in L2, and this pass
       leaves its start there for the apply (32 channels x 128^3: 35 us, and 37 instead of 41 for the apply; 37 with a contiguous piece a block in ascending order) */
    const size_t sweep = (size_t)T * 256;
    size_t k = (S + sweep - 1) / sweep;
    auto at = [&](size_t trip, int u) { const size_t v = trip * sweep + (size_t)t * 256 + 64 * u + ph; return v < S ? ld_dep(p + v * 4) : make_uint4(0u, 0u, 0u, 0u); };      /* rows past the end add zeros */
    for (; k >= 2; k -= 2) {      /* eight loads in flight */
        const uint4 r0 = at(k - 1, 0), r1 = at(k - 1, 1), r2 = at(k - 1, 2), r3 = at(k - 1, 3), r4 = at(k - 2, 0), r5 = at(k - 2, 1), r6 = at(k - 2, 2), r7 = at(k - 2, 3);
        add(r0); add(r1); add(r2); add(r3); add(r4); add(r5); add(r6); add(r7);
    }
    if (k) { const uint4 r0 = at(0, 0), r1 = at(0, 1), r2 = at(0, 2), r3 = at(0, 3); add(r0); add(r1); add(r2); add(r3); }
    __shared__ double ss[64][33], sq[64][33];
#pragma unroll
    for (int k = 0; k < 8; k++) { ss[ph][qd * 8 + k] = acc.s[k]; sq[ph][qd * 8 + k] = acc.q[k]; }
    __syncthreads();
    {
        /* the 64 phases of 32 channels and two sums: 256 threads add 16 each, then 64 threads the four quarters in order */
        const int c = threadIdx.x & 31, which = (threadIdx.x >> 5) & 1, g = threadIdx.x >> 6; double (*src)[33] = which ? sq : ss;
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < 16; k++) t += src[g * 16 + k][c];
        __syncthreads();
        src[g][c] = t;
        __syncthreads();
        if (threadIdx.x < 64) part[(((size_t)n * T + blockIdx.x) * Cop + blk * 32 + c) * 2 + which] = ((src[0][c] + src[1][c]) + src[2][c]) + src[3][c];
    }
    if (!FINAL) return;
    /* the last block of this (sample, block) to finish turns the partial sums into coefficients: eight threads a channel add
       every eighth chunk, then the eight in order; the result does not depend on which block came last */
    __shared__ unsigned last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) { const unsigned tk = atomicAdd(&g_stat_tickets[n * nb + blk], 1u); last = tk == (unsigned)T - 1u; if (last) g_stat_tickets[n * nb + blk] = 0u; }
    __syncthreads();
    if (!last) return;
    __threadfence();
    {
        const int c = threadIdx.x & 31, g8 = threadIdx.x >> 5;
        double a0 = 0.0, a1 = 0.0;
        const double2 *pb = (const double2 *)part + ((size_t)n * T) * Cop + blk * 32 + c;
        int k = g8;
        for (; k < T; k += 128) {          /* sixteen loads in flight; the order of the additions is fixed */
            double2 pv[16];
#pragma unroll
            for (int j = 0; j < 16; j++) pv[j] = k + 8 * j < T ? __ldcg(pb + (size_t)(k + 8 * j) * Cop) : make_double2(0.0, 0.0);
#pragma unroll
            for (int j = 0; j < 16; j++) { a0 += pv[j].x; a1 += pv[j].y; }
        }
        __syncthreads();
        ss[g8][c] = a0; sq[g8][c] = a1;
        __syncthreads();
        if (g8 == 0 && blk * 32 + c < C) {
            for (int k = 1; k < 8; k++) { a0 += ss[k][c]; a1 += sq[k][c]; }
            const int ch = blk * 32 + c;
            const float2 ab = coef_of(a0, a1, (double)S, eps, gamma, beta, ch);
            coef[2 * ((size_t)n * C + ch)] = ab.x;
            coef[2 * ((size_t)n * C + ch) + 1] = ab.y;
        }
    }
}
void umx_stat_tickets_reset(void) { void *p = nullptr; if (cudaGetSymbolAddress(&p, g_stat_tickets) == cudaSuccess && p) cudaMemset(p, 0, sizeof(unsigned) * 8192); }
/* InstanceNorm partial sums of a stored blocked-fp16 conv output (what umx_conv_fwd runs after the conv when it is given `part`) */
void umx_in_part(const void *y, int N, int C, int D, int H, int W, double *part) {
    if (!umx_ready("umx_in_part")) return;
    const int T = umx_stats_chunks(D, H, W);
    umx_launch(in_part_k<false>, dim3(T, (C + 31) / 32, N), dim3(256), 0, (const uint4 *)y, (size_t)D * H * W, T, part, C, (const float *)nullptr, (const float *)nullptr, 0.f, (float *)nullptr);
    g_umx_launches++;
    UMX_CK("umx_in_part");
}
/* statistics and coefficients of a stored blocked-fp16 tensor in one launch (part: scratch of umx_stats_doubles doubles).  Launches of
   this function on one device must not overlap (they share the ticket counters); on one stream they never do. */
extern "C" void umx_in_stats_coef(const void *y, int N, int C, int D, int H, int W, const float *gamma, const float *beta, float eps, double *part, float *coef) {
    if (!umx_ready("umx_in_stats_coef")) return;
    const int T = umx_stats_chunks(D, H, W), nb = (C + 31) / 32;
    if ((size_t)N * nb > 8192) { umx_in_part(y, N, C, D, H, W, part); umx_in_coef(part, N, C, D, H, W, gamma, beta, eps, coef); return; }
    umx_launch(in_part_k<true>, dim3(T, nb, N), dim3(256), 0, (const uint4 *)y, (size_t)D * H * W, T, part, C, gamma, beta, eps, coef);
    g_umx_launches++;
    UMX_CK("umx_in_stats_coef");
}
extern "C" void umx_in_coef(const double *part, int N, int C, int D, int H, int W, const float *gamma, const float *beta, float eps, float *coef) {
    if (!umx_ready("umx_in_coef")) return;
    const int T = umx_stats_chunks(D, H, W), Cop = (C + 31) / 32 * 32;
    in_coef_k<<<dim3(C, N), 256>>>(part, C, Cop, T, (double)D * H * W, gamma, beta, eps, coef);
    g_umx_launches++;
    UMX_CK("umx_in_coef");
}


/* Four lanes a row, eight channels a lane, four rows together: affine map, LeakyReLU, fp16 rounding (o), MX codes (w0, w1).  Returns the scale byte of row
   qd: the four rows' maxima are reduced so that each lane of the quad ends up with one row's, works that row's scale out and hands it to the other three.
   Instruction issue bounds the passes that call this where
   they are not DRAM bound (rows one at a time, each lane working out each scale: with the space-to-depth copy 59 us for 32 channels x 128^3, 52 this way;
   64^3 x 64 in one launch 20.9, 19.4).
   LeakyReLU is max(g, slope g) for 0 < slope <= 1; rounding to fp16 is monotonic, so the maximum is taken of the rounded pairs.  mask: channels that are
   real (FULL: all).  All 32 lanes call it together. */
template <int BITS, bool COEF, bool FULL>
__device__ __forceinline__ unsigned apply4(const uint4 *raw, const float2 *ca, const float2 *cb, float slope, const unsigned *mask, int qd, uint4 *o, unsigned *w0, unsigned *w1) {
    const float2 sl = make_float2(slope, slope);
    __half2 am[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const __half2 *hp = (const __half2 *)(raw + u);
        __half2 *op = (__half2 *)(o + u);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float2 g = __half22float2(hp[k]);
            if (COEF) g = __ffma2_rn(g, ca[k], cb[k]);
            const float2 l = __fmul2_rn(sl, g);
            op[k] = __hmax2(__floats2half2_rn(g.x, g.y), __floats2half2_rn(l.x, l.y));
            if (!FULL) *(unsigned *)(op + k) &= mask[k];
        }
        /* amax of the stored fp16 values, NaN-propagating, taken on the halves (exact: the conversion to fp32 is monotonic) */
        am[u] = __hmax2_nan(__hmax2_nan(__habs2(op[0]), __habs2(op[1])), __hmax2_nan(__habs2(op[2]), __habs2(op[3])));
    }
    const __half2 p01 = __hmax2_nan(__lows2half2(am[0], am[1]), __highs2half2(am[0], am[1])), p23 = __hmax2_nan(__lows2half2(am[2], am[3]), __highs2half2(am[2], am[3]));
    const unsigned b01 = *(const unsigned *)&p01, b23 = *(const unsigned *)&p23;
    unsigned own = qd & 2 ? b23 : b01, t = __shfl_xor_sync(0xffffffffu, qd & 2 ? b01 : b23, 2);
    __half2 m = __hmax2_nan(*(const __half2 *)&own, *(const __half2 *)&t);
    own = *(const unsigned *)&m; t = __shfl_xor_sync(0xffffffffu, own, 1);
    m = __hmax2_nan(m, *(const __half2 *)&t);
    const float a1 = __half2float(qd & 1 ? __high2half(m) : __low2half(m));
    const mx_sb mq = mx_scale_of(__uint_as_float(__float_as_uint(a1) & 0x7fffffffu), BITS == 4 ? 1.f / 6.f : 1.f / 448.f);
    /* what the row's codes need: the factor 2^-e as fp16 where it is a normal one (0: it is not) and the scale byte */
    const unsigned pack = (mq.sb - 112u <= 29u ? (142u - mq.sb) << 10 : 0u) | (mq.sb << 16);
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const unsigned f = __shfl_sync(0xffffffffu, pack, u, 4);
        const __half2 *op = (const __half2 *)(o + u);
        w1[u] = 0u;
        if (BITS == 8 && (f & 0xffffu)) {
            /* scale the halves (exact, or below 2^-14 where E4M3 rounds to zero either way) and convert pairs */
            const unsigned m2 = __byte_perm(f, f, 0x1010);
            const __half2 mm = *(const __half2 *)&m2;
            unsigned short c0, c1, c2, c3;
            const __half2 s0 = __hmul2(op[0], mm), s1 = __hmul2(op[1], mm), s2 = __hmul2(op[2], mm), s3 = __hmul2(op[3], mm);
            asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(c0) : "r"(*(const unsigned *)&s0));
            asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(c1) : "r"(*(const unsigned *)&s1));
            asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(c2) : "r"(*(const unsigned *)&s2));
            asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(c3) : "r"(*(const unsigned *)&s3));
            w0[u] = (unsigned)c0 | ((unsigned)c1 << 16); w1[u] = (unsigned)c2 | ((unsigned)c3 << 16);
        } else {
            float v[8];
#pragma unroll
            for (int k = 0; k < 4; k++) { const float2 r = __half22float2(op[k]); v[2 * k] = r.x; v[2 * k + 1] = r.y; }
            const float fm = __uint_as_float((254u - (f >> 16)) << 23);
            if (BITS == 8) { w0[u] = cvt_e4m3x4(v[0] * fm, v[1] * fm, v[2] * fm, v[3] * fm); w1[u] = cvt_e4m3x4(v[4] * fm, v[5] * fm, v[6] * fm, v[7] * fm); }
            else w0[u] = cvt_e2m1x8(v, fm);
        }
    }
    return mq.sb;
}
/* where a voxel lies in the space-to-depth copy: tap << 28 | coarse voxel (fewer than 2^28 of them); wsh >= 0: W and H are powers of two */
__device__ __forceinline__ unsigned s2d_where(unsigned v, int H, int W, int wsh, int hsh) {
    unsigned xx, yy, zz;
    if (wsh >= 0) { xx = v & ((1u << wsh) - 1u); const unsigned t1 = v >> wsh; yy = t1 & ((1u << hsh) - 1u); zz = t1 >> hsh; }
    else { const unsigned t1 = v / (unsigned)W; xx = v - t1 * (unsigned)W; zz = t1 / (unsigned)H; yy = t1 - zz * (unsigned)H; }
    const unsigned tap = ((zz & 1) * 2 + (yy & 1)) * 2 + (xx & 1);
    return tap << 28 | (((zz >> 1) * (unsigned)(H >> 1) + (yy >> 1)) * (unsigned)(W >> 1) + (xx >> 1));
}
/* one (sample, block)'s destinations: codes of the plain tensor and of the space-to-depth copy (block tap * nb + blk at the coarse voxel), each with this lane's
   offset in a row, and the scale planes; put4 stores four rows, of which row u is voxel v[u], and the scale byte of voxel vo (any of them S or more: not there) */
template <int BITS, bool S2D>
struct MxDst {
    uint8_t *qb, *qsc, *q2, *q2sc; int qs, q2s, H, W, wsh, hsh; size_t tstep, tsc;
    __device__ __forceinline__ MxDst(uint8_t *q, uint8_t *qd2, int N, int nb, int n, int blk, int nb_dst, int b0, size_t S, int H_, int W_, int split, int qd) : H(H_), W(W_) {
        constexpr int RB = 32 * BITS / 8;
        const size_t drow = (size_t)n * nb_dst + b0 + blk, Sc = S / 8, ro = (size_t)n * 8 * nb + blk;
        const int half = BITS == 8 && split;
        qs = half ? 16 : RB;
        qb = q ? q + (half ? (drow * 2 + (qd >> 1)) * S * 16 + (qd & 1) * 8 : drow * S * RB + qd * (RB / 4)) : nullptr;
        qsc = q ? q + (size_t)N * nb_dst * S * RB + drow * S : nullptr;
        if (S2D) {
            const int pow2 = !(W & (W - 1)) && !(H & (H - 1));
            wsh = pow2 ? __ffs(W) - 1 : -1; hsh = pow2 ? __ffs(H) - 1 : 0;
            q2s = qs; tstep = (size_t)nb * Sc * RB; tsc = (size_t)nb * Sc;
            q2 = qd2 + (half ? (ro * 2 + (qd >> 1)) * Sc * 16 + (qd & 1) * 8 : ro * Sc * RB + qd * (RB / 4));
            q2sc = qd2 + (size_t)N * 8 * nb * Sc * RB + ro * Sc;
        }
    }
    __device__ __forceinline__ void put4(const unsigned *v, unsigned vo, unsigned S, const unsigned *w0, const unsigned *w1, unsigned sb) const {
        unsigned wo = 0u;
        if (S2D) { wo = vo < S ? s2d_where(vo, H, W, wsh, hsh) : 0u; if (vo < S) q2sc[(size_t)(wo >> 28) * tsc + (wo & 0x0fffffffu)] = (uint8_t)sb; }
        if (qb && vo < S) qsc[vo] = (uint8_t)sb;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            unsigned wu = 0u;
            if (S2D) wu = __shfl_sync(0xffffffffu, wo, u, 4);
            if (v[u] < S) {
                if (qb) { if (BITS == 8) *(uint2 *)(qb + (size_t)v[u] * qs) = make_uint2(w0[u], w1[u]); else *(unsigned *)(qb + (size_t)v[u] * qs) = w0[u]; }
                if (S2D) {
                    uint8_t *d = q2 + (size_t)(wu >> 28) * tstep + (size_t)(wu & 0x0fffffffu) * q2s;
                    if (BITS == 8) *(uint2 *)d = make_uint2(w0[u], w1[u]); else *(unsigned *)d = w0[u];
                }
            }
        }
    }
};

/* Four threads per voxel row, eight channels (one 16-byte load) each; a block walks a run of voxels of one (sample, block), so the
   sixteen coefficients a thread needs stay in registers.  The row's amax is combined with two shuffles.  grid = (voxel chunks,
   blocks, samples).  This pass is bound by instruction issue (see apply4) and, at three blocks a multiprocessor, by latency (32 channels x 128^3 36.5 us, 33.3 at
   four; the 64-channel MX-fp4 pass with its copy on 96^3 47 and 39), so the variants are compiled apart: COEF (affine map present), FULL (all 32
   channels of every block are real), S2D (second, space-to-depth destination). */
template <int BITS, bool COEF, bool FULL, bool S2D>
__global__ void __launch_bounds__(256, 4) in_apply_k(const uint4 *x, const float2 *coef, int C, int D, int H, int W, int act,
                                                  uint8_t *__restrict__ q, int nb_dst, int b0, uint8_t *__restrict__ q2, uint4 *__restrict__ hout, int split, int T) {
    pdl_trigger(); pdl_wait();
    const int N = gridDim.z, nb = gridDim.y, blk = blockIdx.y, n = blockIdx.z;
    const size_t S = (size_t)D * H * W;
    const int qd = threadIdx.x & 3, ph = threadIdx.x >> 2;
    float2 ca[4], cb[4]; unsigned mask[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int c = blk * 32 + qd * 8 + 2 * k;
        float2 p = make_float2(1.f, 0.f), r = p;
        if (COEF) { if (FULL || c < C) p = ld_dep(coef + (size_t)n * C + c); if (FULL || c + 1 < C) r = ld_dep(coef + (size_t)n * C + c + 1); }
        ca[k] = make_float2(p.x, r.x); cb[k] = make_float2(p.y, r.y);
        mask[k] = FULL ? 0xffffffffu : (c < C ? 0xffffu : 0u) | (c + 1 < C ? 0xffff0000u : 0u);
    }
    const float slope = act == 2 ? 0.01f : 1.f;           /* LeakyReLU as max(g, slope g); slope 1 leaves g as it is */
    const unsigned v0 = (unsigned)(S * blockIdx.x / T), v1 = (unsigned)(S * (blockIdx.x + 1) / T);      /* S < 2^31: 32-bit voxel indices in the loop */
    const uint4 *xp = x + ((size_t)n * nb + blk) * S * 4 + qd;
    uint4 *hp_out = hout ? hout + ((size_t)n * nb + blk) * S * 4 + qd : nullptr;
    const MxDst<BITS, S2D> dst(q, q2, N, nb, n, blk, nb_dst, b0, S, H, W, split, qd);
    for (unsigned vb = v0; vb < v1; vb += 256) {
        /* four rows a thread per trip, their loads issued together */
        uint4 raws[4], o[4]; unsigned v[4], w0[4], w1[4];
#pragma unroll
        for (int u = 0; u < 4; u++) { v[u] = vb + u * 64 + ph; raws[u] = v[u] < v1 ? __ldcs(xp + (size_t)v[u] * 4) : make_uint4(0u, 0u, 0u, 0u); }      /* the last use of x */
        const unsigned sb = apply4<BITS, COEF, FULL>(raws, ca, cb, slope, mask, qd, o, w0, w1);
        if (hp_out) {
#pragma unroll
            for (int u = 0; u < 4; u++) if (v[u] < v1) hp_out[(size_t)v[u] * 4] = o[u];
        }
        dst.put4(v, vb + (unsigned)qd * 64 + ph, v1, w0, w1, sb);
    }
}
template <int BITS, bool COEF, bool FULL>
static void in_apply_launch(dim3 grid, const void *x, const float *coef, int C, int D, int H, int W, int act, void *q, int nb_dst, int b0, void *q_s2d, void *h, int split, int T) {
    if (q_s2d) umx_launch(in_apply_k<BITS, COEF, FULL, true>, grid, dim3(256), 0, (const uint4 *)x, (const float2 *)coef, C, D, H, W, act, (uint8_t *)q, nb_dst, b0, (uint8_t *)q_s2d, (uint4 *)h, split, T);
    else umx_launch(in_apply_k<BITS, COEF, FULL, false>, grid, dim3(256), 0, (const uint4 *)x, (const float2 *)coef, C, D, H, W, act, (uint8_t *)q, nb_dst, b0, (uint8_t *)nullptr, (uint4 *)h, split, T);
}
extern "C" void umx_in_apply(const void *x, const float *coef, int N, int C, int D, int H, int W, int act, void *q, int bits, int nb_dst, int b0, void *q_s2d, void *h, int layout) {
    if (!umx_ready("umx_in_apply")) return;
    if (q_s2d && ((D | H | W) & 1)) { fprintf(stderr, "umx_in_apply: the space-to-depth copy needs even D, H, W\n"); abort(); }
    const int nb = (C + 31) / 32; if (!nb_dst) { nb_dst = nb; b0 = 0; }
    const size_t S = (size_t)D * H * W;
    if (S >= ((size_t)1 << 31)) { fprintf(stderr, "umx_in_apply: more than 2^31 voxels per sample\n"); abort(); }
    if (!S || !N) return;
    /* runs of about 1024 voxels, enough blocks to fill the machine */
    size_t T = (S + 1023) / 1024; if (T > 65535) T = 65535;
    const dim3 grid((unsigned)T, (unsigned)nb, (unsigned)N);
    const int split = layout == UMX_LAYOUT_SPLIT, full = (C & 31) == 0;
#define UMX_APPLY(B, CO, FU) in_apply_launch<B, CO, FU>(grid, x, coef, C, D, H, W, act, q, nb_dst, b0, q_s2d, h, split, (int)T)
    if (bits == 8) { if (coef) { if (full) UMX_APPLY(8, true, true); else UMX_APPLY(8, true, false); } else { if (full) UMX_APPLY(8, false, true); else UMX_APPLY(8, false, false); } }
    else { if (coef) { if (full) UMX_APPLY(4, true, true); else UMX_APPLY(4, true, false); } else { if (full) UMX_APPLY(4, false, true); else UMX_APPLY(4, false, false); } }
#undef UMX_APPLY
    g_umx_launches++;
    UMX_CK("umx_in_apply");
}

/* ---- statistics, coefficients and apply in one launch: what a conv of the U-Net is followed by.  B blocks share a (sample, 32-channel block).
   A block adds up its share of the voxels, the blocks' sums meet (small tensors: a cluster, through distributed shared memory; others: through
   global memory and a counter), and the values are transformed where they are, in registers (ROWS rows a thread).  Tensors too large for that
   take two launches (32 channels x 128^3 66.8 us); read again in one launch they were no faster (87 us against 79 for two at the time).
   Two launches are each a chain of a load, a reduction and a store behind a device-wide wait, which is what bounds them on the deep levels and on
   small patches: 8^3 x 320 channels 10.7 us, 16^3 x 256 11.0, 32^3 x 128 14.3, with the space-to-depth copy 16.5; in one launch 5.9, 5.7, 8.0 and 9.0.
   A launch has at most one block a multiprocessor, so its blocks are resident together once the kernels before them have drained, and the wait at the
   counter is short.  Nothing rests on that (another process may hold part of the device): a block that has waited for kNormWait leaves its rows to
   whichever block of its group arrives last, which by then waits for nobody, and ends.  Every block therefore ends, and the result is the same
   either way.  (A cooperative launch, which guarantees residency, cannot overlap the end of its predecessor: 4 us for the four of the 32^3
   three-level network, 19 for the eight of the 96^3 four-level one, where this form costs nothing.  Clusters do not give it: of 36 clusters of
   eight that the occupancy query allows, 32 were scheduled.)  Sums are fp64 in a fixed order: rows of a thread, row phases, shares.  The shares are those of
   a launch with one sample, whatever the batch (norm_plan), so a sample's bytes are its own: a block of a launch with several samples does several shares one
   after the other (MULTI), and a batch that is too much for one launch takes the same sums in a launch of their own (in_share_k) and in_apply_k. ---- */
namespace {
/* blocks of a launch that meet through the counter, at most; shares of a (sample, block), for which part has room and for the coefficients; shares of a block, for which shared memory has; (sample,
   block) pairs that meet */
constexpr int kNormBlocks = 1024, kNormPart = 511, kNormPer = 4, kNormPairs = 4096;
constexpr long long kNormWait = 200000;                      /* clock cycles (0.1 ms) */
/* per (sample, block): blocks that have left their sums | blocks that have left their rows << 16; blocks that need neither word any more (the last one clears both) */
__device__ unsigned g_norm_count[2 * kNormPairs];
__device__ unsigned g_norm_left[kNormBlocks];                /* per (sample, block): 1 + rank of the blocks that have left their rows, zero between launches */
/* ranks: shares of a (sample, block), of which a block takes rank, rank + B, ...; vp: voxels of a share's trip, NT / 4 to NT; step: of all shares' together; trips: of
   a share at most; cl: blocks of a cluster, all B of them, or 1 */
struct NormArgs { const uint4 *x; int N, H, W; unsigned S; float eps; int act; uint8_t *q; int nb_dst, b0; uint8_t *q2; int split; int cl, ranks; unsigned vp, step, trips; long long wait; double *part; int *err; };

/* The trips of a block, NT voxels (four rows a thread) each: those of its first share, of the next, ...  Trip k of share r begins at voxel k step + r vp; trips past
   the end of the tensor are not there (they come last in a share, and every share has a first one). */
constexpr unsigned kNoTrip = 0x80000000u;
struct NormTrips {
    unsigned v, k, r;                                        /* first voxel of the trip, kNoTrip when there are no more; number in its share; share */
    __device__ __forceinline__ NormTrips(const NormArgs &a, unsigned rank) : v(rank * a.vp), k(0u), r(rank) {}
    __device__ __forceinline__ void next(const NormArgs &a, unsigned B) {
        k++;
        v += a.step;
        if (k == a.trips || v >= a.S) { k = 0u; r += B; v = r < (unsigned)a.ranks ? r * a.vp : kNoTrip; }
    }
};
/* A warp's sums of one share into shared memory, as [sum or sum of squares][channel].  The lanes that hold the same channels halve what they hold three
   times, each keeping one half and adding what the other held of it: no barrier, and a sixteenth of the shared memory traffic of 16 doubles a thread.  With it
   and shares of 512 voxels or more 32 channels x 32^3 take 6.8 us (8.2 before), 64 x 64^3 17.8 (18.7), and a second share a block costs 32 x 64^3 x 2 samples
   0.8 us of 19.5; with a barrier and the wide form it cost 4. */
__device__ __forceinline__ void warp_sums(const StatAcc &acc, double *to) {
    const int lane = threadIdx.x & 31;
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) { const bool up = lane & 16; const double o = __shfl_xor_sync(0xffffffffu, up ? acc.s[k] : acc.q[k], 16); v[k] = (up ? acc.q[k] : acc.s[k]) + o; }
#pragma unroll
    for (int k = 0; k < 4; k++) { const bool up = lane & 8; const double o = __shfl_xor_sync(0xffffffffu, up ? v[k] : v[k + 4], 8); v[k] = (up ? v[k + 4] : v[k]) + o; }
#pragma unroll
    for (int k = 0; k < 2; k++) { const bool up = lane & 4; const double o = __shfl_xor_sync(0xffffffffu, up ? v[k] : v[k + 2], 4); v[k] = (up ? v[k + 2] : v[k]) + o; }
    *(double2 *)&to[((lane >> 4) << 5) + (lane & 3) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2] = make_double2(v[0], v[1]);
}
/* the n rows of place threadIdx.x & 63, added in order */
template <int N> __device__ __forceinline__ double rows_sum(const double (*red)[64]) {
    double t = red[0][threadIdx.x & 63];
#pragma unroll
    for (int k = 1; k < N; k++) t += red[k][threadIdx.x & 63];
    return t;
}
/* the sums of all shares, on the first 64 threads */
template <int NT> __device__ __forceinline__ double shares_sum(const double *part, int ranks, double (*red)[64]) {
    double t = 0.0;
#pragma unroll 4
    for (int k = threadIdx.x >> 6; k < ranks; k += NT / 64) t += __ldcg(part + k * 64 + (threadIdx.x & 63));
    red[threadIdx.x >> 6][threadIdx.x & 63] = t;
    __syncthreads();
    return threadIdx.x < 64 ? rows_sum<NT / 64>(red) : 0.0;
}
template <int BITS, bool S2D, int ROWS, int NT, bool STASH, bool MULTI>
__global__ void __launch_bounds__(NT) in_norm_k(const NormArgs a) {
    pdl_trigger();
    constexpr int PH = NT / 4, NW = NT / 32;
    __shared__ __align__(16) double red[MULTI ? kNormPer : 1][NW][64];
    __shared__ double mine[64];
    __shared__ float2 sc[32];
    extern __shared__ __align__(16) uint8_t stash_raw[];
    uint4 *stash = (uint4 *)stash_raw + threadIdx.x;           /* STASH: [row of a thread][thread] */
    const int nb = gridDim.y, blk = blockIdx.y, n = blockIdx.z, B = gridDim.x, rank = blockIdx.x, CL = a.cl;
    const int qd = threadIdx.x & 3, ph = threadIdx.x >> 2, warp = threadIdx.x >> 5;
    const unsigned S = a.S, g = blockIdx.z * (unsigned)nb + (unsigned)blk;
    const uint4 *xp = a.x + ((size_t)n * nb + blk) * S * 4 + qd;
    double *part = a.part + (size_t)(n * nb + blk) * a.ranks * 64;
    unsigned left = 0;                                       /* blocks of the group whose rows are this block's to do as well */
    StatAcc acc;
    stat_zero(acc);
    pdl_wait();
    uint4 raw[ROWS];
    unsigned at[ROWS / 4];                                   /* where the trips in raw begin */
    bool turn[ROWS / 4];                                     /* MULTI: the trip begins another share */
    NormTrips tr(a, (unsigned)rank);
    unsigned kept = 0;                                       /* rows of a thread that wait in shared memory: those before the ones in registers */
    int cur = 0;                                             /* the block's share that is being added up */
    /* voxel of this thread's row u of the trip that begins at v; S or more: none */
    auto vox = [&](unsigned v, int u) { return NT == 512 || (unsigned)(PH * u) < a.vp ? v + (unsigned)(PH * u + ph) : S; };
    auto load4 = [&](uint4 *r, unsigned v) {
#pragma unroll
        for (int u = 0; u < 4; u++) { const unsigned w = vox(v, u); r[u] = w < S ? ld_dep(xp + (size_t)w * 4) : make_uint4(0u, 0u, 0u, 0u); }      /* rows past the end add zeros */
    };
    auto load = [&]() {
#pragma unroll
        for (int k = 0; k < ROWS / 4; k++) {
            at[k] = tr.v; turn[k] = MULTI && !tr.k && tr.v != kNoTrip && kept + k;
            load4(raw + 4 * k, tr.v);
            if (tr.v != kNoTrip) tr.next(a, (unsigned)B);
        }
    };
    load();
    if (STASH) while (tr.v != kNoTrip) {
#pragma unroll
        for (int u = 0; u < ROWS; u++) {
            if (MULTI && !(u & 3) && turn[u / 4]) { warp_sums(acc, red[cur++][warp]); stat_zero(acc); }
            stat_add(acc, raw[u]);
            stash[(size_t)(kept + u) * NT] = raw[u];
        }
        kept += ROWS;
        load();
    }
#pragma unroll
    for (int u = 0; u < ROWS; u++) {
        if (MULTI && !(u & 3) && turn[u / 4]) { warp_sums(acc, red[cur++][warp]); stat_zero(acc); }
        stat_add(acc, raw[u]);
    }
    warp_sums(acc, red[cur][warp]);
    __syncthreads();
    double tot = 0.0;                                        /* of the first 64 threads: over all shares */
    if (CL > 1) {                                            /* the blocks are a cluster */
        if (threadIdx.x < 64) mine[threadIdx.x] = rows_sum<NW>(red[0]);
        cluster_sync_all();
        if (threadIdx.x < 64) {
            const uint32_t at0 = smem_u32(mine) + threadIdx.x * 8;
            for (int r = 0; r < CL; r++) tot += cluster_ldd(cluster_addr(at0, (uint32_t)r));
        }
        cluster_arrive();                                    /* no block's memory is read after this; everyone waits for everyone before leaving */
    } else if (B > 1) {
        const int j = threadIdx.x >> 6;                      /* 64 threads a share */
        if (j <= cur) { __stcg(part + (rank + j * B) * 64 + (threadIdx.x & 63), rows_sum<NW>(red[j])); __threadfence(); }
        __shared__ unsigned others;
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            unsigned *cnt = &g_norm_count[2 * g], w = atomicAdd(cnt, 1u) + 1u, rest = 0u;
            if ((w & 0xffffu) == (unsigned)B) rest = w >> 16;         /* the last to arrive: nobody leaves rows behind after this */
            else {
                const long long t0 = clock64();
                for (;;) {
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(w) : "l"(cnt) : "memory");
                    if ((w & 0xffffu) == (unsigned)B) break;
                    if (clock64() - t0 < a.wait) continue;
                    if (atomicCAS(cnt, w, w + 0x10000u) == w) {       /* not all here: the rows are the last block's */
                        asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(&g_norm_left[g * B + (w >> 16)]), "r"((unsigned)rank + 1u) : "memory");
                        rest = ~0u;
                        break;
                    }
                }
            }
            __threadfence();
            if (atomicAdd(&cnt[1], 1u) == (unsigned)B - 1u) { cnt[0] = 0u; cnt[1] = 0u; }
            others = rest;
        }
        __syncthreads();
        left = others;
        if (left == ~0u) return;
        tot = shares_sum<NT>(part, a.ranks, red[0]);
    } else if (threadIdx.x < 64) tot = rows_sum<NW>(red[0]);
    if (threadIdx.x < 64) red[0][0][threadIdx.x] = tot;
    __syncthreads();
    if (threadIdx.x < 32) sc[threadIdx.x] = coef_of(red[0][0][threadIdx.x], red[0][0][32 + threadIdx.x], (double)S, a.eps, nullptr, nullptr, 0);
    __syncthreads();
    float2 ca[4], cb[4]; unsigned mask[4];
#pragma unroll
    for (int k = 0; k < 4; k++) { const float2 p = sc[qd * 8 + 2 * k], r = sc[qd * 8 + 2 * k + 1]; ca[k] = make_float2(p.x, r.x); cb[k] = make_float2(p.y, r.y); mask[k] = 0xffffffffu; }
    const float slope = a.act == 2 ? 0.01f : 1.f;
    const MxDst<BITS, S2D> dst(a.q, a.q2, a.N, nb, n, blk, a.nb_dst, a.b0, S, a.H, a.W, a.split, qd);
    auto put = [&](const uint4 *r, unsigned w) {             /* the four rows of the trip that begins at w */
        uint4 o[4]; unsigned v[4], w0[4], w1[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = vox(w, u);
        const unsigned sb = apply4<BITS, true, true>(r, ca, cb, slope, mask, qd, o, w0, w1);
        dst.put4(v, vox(w, qd), S, w0, w1, sb);
    };
#pragma unroll
    for (int k = 0; k < ROWS / 4; k++) if (at[k] != kNoTrip) put(raw + 4 * k, at[k]);
    if (STASH) {
        NormTrips w(a, (unsigned)rank);
        for (unsigned k = 0; k < kept; k += 4) {
            uint4 r[4];
#pragma unroll
            for (int u = 0; u < 4; u++) r[u] = stash[(size_t)(k + u) * NT];
            put(r, w.v);
            w.next(a, (unsigned)B);
        }
    }
    if (CL > 1) cluster_wait();
    for (unsigned i = 0; i < left; i++) {                    /* rows of blocks that could not wait; read again */
        __shared__ unsigned whose;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned r = 0u;                                 /* the block has announced itself and writes its rank next */
            const long long t0 = clock64();
            while (!r && clock64() - t0 < 4000000000ll) asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(r) : "l"(&g_norm_left[g * B + i]) : "memory");
            if (!r && atomicCAS(a.err, 0, 10) == 0) { a.err[1] = (int)blockIdx.x; a.err[2] = (int)i; }
            g_norm_left[g * B + i] = 0u;
            whose = r;
        }
        __syncthreads();
        if (!whose) continue;
        for (NormTrips w(a, whose - 1u); w.v != kNoTrip; w.next(a, (unsigned)B)) {
            uint4 r[4];
            load4(r, w.v);
            put(r, w.v);
        }
    }
}
/* The statistics alone, for a batch that is more than one launch holds: a block a share, the sums and their order those of in_norm_k; the block of a (sample,
   block) that comes last makes the coefficients.  The last sample comes first: it is what the conv before left in L2.  With the apply 64 channels x 64^3 x 2
   samples take 32.0 us, 35.5 with in_part_k, 40.4 in one launch a sample. */
__global__ void __launch_bounds__(512, 2) in_share_k(const NormArgs a, float2 *coef) {
    pdl_trigger();
    __shared__ __align__(16) double red[16][64];
    __shared__ unsigned last;
    const int nb = gridDim.y, blk = blockIdx.y, n = gridDim.z - 1 - blockIdx.z, rank = blockIdx.x, qd = threadIdx.x & 3, ph = threadIdx.x >> 2;
    const unsigned S = a.S, g = (unsigned)(n * nb + blk);
    const uint4 *xp = a.x + (size_t)g * S * 4 + qd;
    double *part = a.part + (size_t)g * a.ranks * 64;
    StatAcc acc;
    stat_zero(acc);
    pdl_wait();
    for (NormTrips tr(a, (unsigned)rank); tr.v != kNoTrip; tr.next(a, (unsigned)a.ranks)) {
        uint4 r[4];
#pragma unroll
        for (int u = 0; u < 4; u++) { const unsigned v = tr.v + 128u * u + (unsigned)ph; r[u] = v < S ? ld_dep(xp + (size_t)v * 4) : make_uint4(0u, 0u, 0u, 0u); }
#pragma unroll
        for (int u = 0; u < 4; u++) stat_add(acc, r[u]);
    }
    warp_sums(acc, red[threadIdx.x >> 5]);
    __syncthreads();
    if (threadIdx.x < 64) { __stcg(part + rank * 64 + threadIdx.x, rows_sum<16>(red)); __threadfence(); }
    __syncthreads();
    if (threadIdx.x == 0) { last = atomicAdd(&g_norm_count[2 * g], 1u) == (unsigned)a.ranks - 1u; if (last) g_norm_count[2 * g] = 0u; __threadfence(); }
    __syncthreads();
    if (!last) return;
    const double tot = shares_sum<512>(part, a.ranks, red);
    if (threadIdx.x < 64) red[0][threadIdx.x] = tot;
    __syncthreads();
    if (threadIdx.x < 32) coef[(size_t)g * 32 + threadIdx.x] = coef_of(red[0][threadIdx.x], red[0][32 + threadIdx.x], (double)S, a.eps, nullptr, nullptr, 0);
}
/* whether clusters of 16 blocks of a variant can be launched, looked up once per device */
template <int BITS, bool S2D, int ROWS, int NT> bool norm_sixteen() {
    static int have[16];
    int d = 0; cudaGetDevice(&d); d &= 15;
    if (!have[d]) {
        const void *k = (const void *)in_norm_k<BITS, S2D, ROWS, NT, false, false>;
        cudaLaunchConfig_t cfg; memset(&cfg, 0, sizeof cfg);
        cudaLaunchAttribute at; memset(&at, 0, sizeof at);
        at.id = cudaLaunchAttributeClusterDimension; at.val.clusterDim.x = 16; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
        cfg.gridDim = dim3(16); cfg.blockDim = dim3(NT); cfg.attrs = &at; cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) n = 0;
        cudaGetLastError();
        have[d] = n > 0 ? 1 : -1;
    }
    return have[d] > 0;
}
/* one block a multiprocessor that keeps eight rows a thread in registers and up to kStashTrips x 4 more in shared memory (they come to 226 KB with the sums) */
constexpr int kStashTrips = 6;
/* How a tensor is dealt out.  ranks, vp and trips (of a share, at most), which fix the order of the sums, follow from one sample; per (shares of a block, at
   most), blocks and all (trips of a block, at most) from the batch.  held 0: not in this form, 1: in one launch, 2: one sample would be, the batch takes
   in_share_k and in_apply_k */
struct NormPlan { int held, blocks, cl, ranks, per, vp, trips, all; };
NormPlan norm_plan(size_t S, int nb, int N, int sms, bool sixteen) {
    NormPlan p = {1, 1, 1, 1, 1, 256, 1, 1};
    if (S <= 4096) {                                         /* a block, or a cluster while a thread of it has at most four (eight) rows */
        p.blocks = p.cl = p.ranks = S <= 256 ? 1 : S <= 1024 || !sixteen ? 8 : 16;
        if ((size_t)p.ranks * 256 > S) p.vp = (int)((S + p.ranks * 64 - 1) / (size_t)(p.ranks * 64)) * 64;
        p.trips = (int)((S + (size_t)p.ranks * p.vp - 1) / ((size_t)p.ranks * p.vp));
        p.all = p.trips;
        return p;
    }
    /* one block a multiprocessor, dealt to the (sample, block) pairs, each of at most 1024 voxels in registers and 3072 in shared memory */
    if (sms > kNormBlocks) sms = kNormBlocks;
    long long r = sms / nb;
    if (r > kNormPart) r = kNormPart;
    if (r < 1 || (size_t)r * (2 + kStashTrips) * 512 < S) { p.held = 0; return p; }
    p.vp = 512;
    p.trips = (int)((S + (size_t)r * 512 - 1) / ((size_t)r * 512));
    /* no share without a voxel; a multiple of four where that does not cost a trip (it deals out well to two and four samples) */
    p.ranks = p.trips == 1 ? (int)((S + 511) / 512) : (size_t)(r & ~3ll) * 512 * p.trips >= S ? (int)(r & ~3ll) : (int)r;
    /* trips of the first block, which has most: of a share all but the last, and that one where it begins before the end */
    const int fit = (int)(sms / ((long long)nb * N));
    p.held = 2;
    if (fit < 1) return p;
    p.per = (p.ranks + fit - 1) / fit; p.blocks = (p.ranks + p.per - 1) / p.per; p.all = 0;
    for (int s = 0; s < p.ranks; s += p.blocks) p.all += p.trips - (((long long)(p.trips - 1) * p.ranks + s) * 512 >= (long long)S);
    if (p.per <= kNormPer && p.all <= 2 + kStashTrips) p.held = 1;
    return p;
}
template <int BITS, bool S2D, int ROWS, int NT> void norm_go(const NormArgs &a, int B, int nb) {
    umx_launch_cluster(in_norm_k<BITS, S2D, ROWS, NT, false, false>, dim3((unsigned)B, (unsigned)nb, (unsigned)a.N), dim3((unsigned)a.cl, 1, 1), dim3(NT), 0, a);
}
template <int BITS, bool S2D, bool MULTI> bool norm_go_wide(const NormArgs &a, const NormPlan &p, int nb) {
    const dim3 grid((unsigned)p.blocks, (unsigned)nb, (unsigned)a.N);
    const int kept = (p.all - 1) / 2 * 2;                     /* trips in shared memory, two in registers */
    if (!kept) { umx_launch(in_norm_k<BITS, S2D, 8, 512, false, MULTI>, grid, dim3(512), 0, a); return true; }
    static int set[16];
    int d = 0; cudaGetDevice(&d); d &= 15;
    if (!set[d]) set[d] = cudaFuncSetAttribute((const void *)in_norm_k<BITS, S2D, 8, 512, true, MULTI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStashTrips * 4 * 512 * 16) == cudaSuccess ? 1 : -1;
    if (set[d] < 0) { cudaGetLastError(); return false; }
    umx_launch(in_norm_k<BITS, S2D, 8, 512, true, MULTI>, grid, dim3(512), (size_t)kept * 4 * 512 * 16, a);
    return true;
}
/* 1: in one launch; 2: the caller launches in_share_k and the apply; 0: not this tensor */
template <int BITS, bool S2D> int norm_pick(NormArgs &a, int nb, int sms) {
    const NormPlan p = norm_plan(a.S, nb, a.N, sms, a.S > 1024 && a.S <= 4096 && norm_sixteen<BITS, S2D, 4, 256>());
    a.cl = p.cl; a.ranks = p.ranks; a.vp = (unsigned)p.vp; a.step = (unsigned)(p.ranks * p.vp); a.trips = (unsigned)p.trips;
    if (p.held != 1) return p.held;
    if (a.S <= 4096) { if (p.trips == 1) norm_go<BITS, S2D, 4, 256>(a, p.blocks, nb); else norm_go<BITS, S2D, 8, 256>(a, p.blocks, nb); return 1; }
    if (p.all == 1) { norm_go<BITS, S2D, 4, 512>(a, p.blocks, nb); return 1; }
    return p.per > 1 ? norm_go_wide<BITS, S2D, true>(a, p, nb) : norm_go_wide<BITS, S2D, false>(a, p, nb);
}
}   // namespace
/* the plan of a tensor: held, blocks, cluster, shares, shares a block, voxels a trip, trips a share, trips a block */
extern "C" void umx_norm_plan(size_t S, int nb, int N, int sms, int sixteen, int *out) { const NormPlan p = norm_plan(S, nb, N, sms, sixteen != 0); memcpy(out, &p, sizeof p); }
/* umx_in_norm_apply dealt out for sms multiprocessors, its blocks waiting for one another for `wait` clock cycles */
extern "C" int umx_in_norm_apply_on(const void *x, int N, int C, int D, int H, int W, float eps, int act, double *part, void *q, int bits, int nb_dst, int b0, void *q_s2d, int layout, int sms, long long wait) {
    const size_t S = (size_t)D * H * W;
    if (!umx_ready("umx_in_norm_apply") || !S || !N || (C & 31) || S >= (size_t)1 << 31 || !q || (q_s2d && ((D | H | W) & 1)) || C / 32 > kNormPairs) return 1;
    NormArgs a; memset(&a, 0, sizeof a);
    a.x = (const uint4 *)x; a.N = N; a.H = H; a.W = W; a.S = (unsigned)S; a.eps = eps; a.act = act; a.q = (uint8_t *)q; a.nb_dst = nb_dst ? nb_dst : C / 32; a.b0 = nb_dst ? b0 : 0;
    a.q2 = (uint8_t *)q_s2d; a.split = layout == UMX_LAYOUT_SPLIT; a.wait = wait; a.part = part; a.err = umx_errflag();
    if (!a.err) return -1;
    const int form = bits == 8 ? (q_s2d ? norm_pick<8, true>(a, C / 32, sms) : norm_pick<8, false>(a, C / 32, sms)) : (q_s2d ? norm_pick<4, true>(a, C / 32, sms) : norm_pick<4, false>(a, C / 32, sms));
    if (!form) return 1;
    if (form == 2) {
        float2 *coef = (float2 *)(part + (size_t)N * (C / 32) * a.ranks * 64);      /* behind the sums: a place of 64 doubles a (sample, block) is left */
        const int nb = C / 32, most = kNormPairs / nb;        /* samples a launch: a counter a (sample, block) */
        for (int n = 0; n < N; n += most) {
            NormArgs b = a;
            b.x += (size_t)n * nb * S * 4; b.part += (size_t)n * nb * a.ranks * 64;
            umx_launch(in_share_k, dim3((unsigned)a.ranks, (unsigned)nb, (unsigned)(N - n < most ? N - n : most)), dim3(512), 0, b, coef + (size_t)n * C);
        }
        umx_in_apply(x, (const float *)coef, N, C, D, H, W, act, q, bits, nb_dst, b0, q_s2d, nullptr, layout);      /* counts itself */
    }
    g_umx_launches++;
    UMX_CK("umx_in_norm_apply");
    return 0;
}
/* statistics, coefficients (gamma 1, beta 0) and apply of a blocked fp16 tensor of a multiple of 32 channels in one launch; part: scratch of
   umx_stats_doubles doubles.  Launches on one device must not overlap (they share the counters).  1: not this tensor; the caller takes
   umx_in_stats_coef and umx_in_apply. */
extern "C" int umx_in_norm_apply(const void *x, int N, int C, int D, int H, int W, float eps, int act, double *part, void *q, int bits, int nb_dst, int b0, void *q_s2d, int layout) {
    static int sms_of[16];
    int d = 0; cudaGetDevice(&d); d &= 15;
    if (!sms_of[d]) { int v = 1; cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d); sms_of[d] = v; }
    return umx_in_norm_apply_on(x, N, C, D, H, W, eps, act, part, q, bits, nb_dst, b0, q_s2d, layout, sms_of[d], kNormWait);
}
void umx_norm_counts_reset(void) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_norm_count) == cudaSuccess && p) cudaMemset(p, 0, sizeof(unsigned) * 2 * kNormPairs);
    if (cudaGetSymbolAddress(&p, g_norm_left) == cudaSuccess && p) cudaMemset(p, 0, sizeof(unsigned) * kNormBlocks);
}
