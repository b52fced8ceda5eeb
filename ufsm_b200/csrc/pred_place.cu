/* The back end of the reference's predict on the device (src/nn.h:871-885, src/nn_elem.cu:1096-1178): one head's logits of a
   D x W x W window become probability bytes, the window's halo is cropped, and what is left of the interior inside the output shard
   is written at its place in a device shard buffer.  byte = trunc(255 / (1 + exp(-logit)) + 0.5) where the CT voxel is material
   (CT >= iso, or its bit in a mask built from the CT beforehand), 0 elsewhere.

   Geometry (place_isect of the reference): window voxel (z, y, x) sits at shard coordinate (oz + z, oy + y, ox + x); it is written when
   it is interior (z in [hz, D - hz), y and x in [halo, W - halo)) and inside the shard's extent ([0, ez) x [0, ey) x [0, ex)).  The box of
   such voxels is worked out on the host and a thread takes eight consecutive x of one box row, so a warp reads and writes runs of 256
   voxels of a row or of neighbouring rows. */
#include "mx_common.cuh"

namespace {

struct PlaceBox { int z0, y0, x0, nz, ny, nx; };
PlaceBox place_box_of(int D, int W, int hz, int halo, int oz, int oy, int ox, int ez, int ey, int ex) {
    PlaceBox b;
    b.z0 = hz > -oz ? hz : -oz; b.y0 = halo > -oy ? halo : -oy; b.x0 = halo > -ox ? halo : -ox;
    const int z1 = D - hz < ez - oz ? D - hz : ez - oz, y1 = W - halo < ey - oy ? W - halo : ey - oy, x1 = W - halo < ex - ox ? W - halo : ex - ox;
    b.nz = z1 > b.z0 ? z1 - b.z0 : 0; b.ny = y1 > b.y0 ? y1 - b.y0 : 0; b.nx = x1 > b.x0 ? x1 - b.x0 : 0;
    return b;
}
/* trunc(255 / (1 + exp(-l)) + 0.5), a NaN as 0; the truncation as an addition of 2^23 rounded down, which keeps the conversion unit free for the
   two approximations */
__device__ __forceinline__ unsigned prob255(float l) { return __float_as_uint(__fadd_rd(fmaxf(__fdividef(255.f, 1.f + __expf(-l)) + 0.5f, 0.f), 8388608.f)) & 0xffu; }
template <typename LT> __device__ __forceinline__ float logit_at(const LT *lg, size_t k);
template <> __device__ __forceinline__ float logit_at<float>(const float *lg, size_t k) { return ld_dep(lg + k); }
template <> __device__ __forceinline__ float logit_at<__half>(const __half *lg, size_t k) { return __half2float(ld_dep(lg + k)); }

/* MASK 0: material where ct[k] >= iso; 1: where bit k of `bits` is set.  zoff: the window is held from its plane zoff on (a half of a split window).
   A block takes R = 256 / nq whole rows of the box at a time (nq groups of eight x a row), so a thread works out its place once and needs
   one 32-bit division a trip; eight voxels go with one load of their logits, one of their mask bits and one store where these are aligned.
   Bound by latency and issue: 160^3 of a 192^3 window 12.4 us with 64-bit index divisions every four voxels, 7.6 us in this form. */
template <typename LT, int MASK>
__global__ void __launch_bounds__(256) pred_place_k(const LT *lg, const uint8_t *ct, const uint32_t *bits, PlaceBox B, int W, int zoff,
                                                    int oz, int oy, int ox, int shard, uint8_t *__restrict__ dsh, int iso) {
    pdl_trigger(); pdl_wait();
    const int nq = (B.nx + 7) >> 3, R = nq < 256 ? 256 / nq : 1, tr = (int)threadIdx.x / nq;
    const unsigned rows = (unsigned)B.nz * (unsigned)B.ny;
    if (R > 1 && tr >= R) return;
    for (unsigned row = blockIdx.x * (unsigned)R + (R > 1 ? tr : 0); row < rows; row += gridDim.x * (unsigned)R) {
        const int zz = (int)(row / (unsigned)B.ny), y = B.y0 + (int)(row - (unsigned)zz * (unsigned)B.ny), z = B.z0 + zz;
        const size_t kr = ((size_t)(z - zoff) * W + y) * W;
        uint8_t *orow = dsh + ((size_t)(oz + z) * shard + (oy + y)) * shard + ox;
        for (int q = R > 1 ? (int)threadIdx.x - tr * nq : (int)threadIdx.x; q < nq; q += 256) {
            const int xa = B.x0 + 8 * q, n = min(8, B.x0 + B.nx - xa);
            const size_t k = kr + xa;
            uint8_t *o = orow + xa;
            float l[8]; unsigned on = 0u;
            if (n == 8 && !((size_t)(lg + k) & 15)) {
                if (sizeof(LT) == 2) {
                    const uint4 r = ld_dep((const uint4 *)(lg + k)); const __half2 *h = (const __half2 *)&r;
#pragma unroll
                    for (int j = 0; j < 4; j++) { const float2 f = __half22float2(h[j]); l[2 * j] = f.x; l[2 * j + 1] = f.y; }
                } else {
                    const float4 r = ld_dep((const float4 *)(lg + k)), t = ld_dep((const float4 *)(lg + k) + 1);
                    l[0] = r.x; l[1] = r.y; l[2] = r.z; l[3] = r.w; l[4] = t.x; l[5] = t.y; l[6] = t.z; l[7] = t.w;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++) l[j] = j < n ? logit_at<LT>(lg, k + j) : 0.f;
            }
            if (MASK) {
                const unsigned sh = (unsigned)(k & 31);
                on = ld_dep(bits + (k >> 5)) >> sh;
                if (sh + n > 32) on |= ld_dep(bits + (k >> 5) + 1) << (32 - sh);
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++) if (j < n && (int)ld_dep(ct + k + j) >= iso) on |= 1u << j;
            }
            unsigned v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) { const unsigned t = prob255(l[j]); v[j] = (on >> j) & 1u ? t : 0u; }
            if (n == 8 && !((size_t)o & 7)) *(uint2 *)o = make_uint2(v[0] | (v[1] << 8) | (v[2] << 16) | (v[3] << 24), v[4] | (v[5] << 8) | (v[6] << 16) | (v[7] << 24));
            else for (int j = 0; j < n; j++) o[j] = (uint8_t)v[j];
        }
    }
}
__global__ void __launch_bounds__(256) pred_out_k(const void *lg, int h16, const uint8_t *ct, size_t n, uint8_t *__restrict__ out) {
    pdl_trigger(); pdl_wait();
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = ld_dep(ct + i) ? (uint8_t)prob255(h16 ? logit_at<__half>((const __half *)lg, i) : logit_at<float>((const float *)lg, i)) : (uint8_t)0;
}
/* one 32-voxel word a thread: two 16-byte loads where the bytes are there and aligned, byte compares four at a time */
__global__ void __launch_bounds__(256) ctmask_k(const uint8_t *ct, size_t n, uint32_t *__restrict__ bits, int t) {
    pdl_trigger(); pdl_wait();
    const size_t w = blockIdx.x * (size_t)blockDim.x + threadIdx.x, i0 = w * 32;
    if (i0 >= n) return;
    uint32_t m = 0;
    if (t > 255) { bits[w] = 0u; return; }
    if (i0 + 32 <= n && !((size_t)(ct + i0) & 15)) {
        const uint4 u0 = ld_dep((const uint4 *)(ct + i0)), u1 = ld_dep((const uint4 *)(ct + i0) + 1);
        const uint32_t v[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w}, tt = (uint32_t)t * 0x01010101u;
#pragma unroll
        for (int j = 0; j < 8; j++) m |= ((((__vcmpgeu4(v[j], tt) & 0x01010101u) * 0x01020408u) >> 24) & 15u) << (4 * j);
    } else {
        const int cnt = (int)min((size_t)32, n - i0);
        for (int j = 0; j < cnt; j++) m |= (uint32_t)((int)ld_dep(ct + i0 + j) >= t) << j;
    }
    bits[w] = m;
}

/* ---- seam feather (the blend of src/predict.c:282-333, which the reference runs on host threads over downloaded windows) ----
   Windows lie on a grid with interior S per axis; each window's prediction E covers its interior and B voxels of its upper halo per axis
   (E = S + B).  The output over the interior is E itself except in the lower shell (a coordinate below B), where the upper spills of the
   windows before it are blended in: the window shifted back by delta in {0, 1}^3 (bit 0 x, 1 y, 2 z) has the weight
   prod_axis (delta ? 1 - u(v) : u(v)), u(j) = sin^2(pi / 2 (j + 0.5) / B) for v < B (1 / 0 above), normalised over the windows present.
   A neighbour's spill is its z slab [B][E][E] when it lies a window back in z, else its y slab [S][B][E] when back in y, else its x slab
   [S][S][B] (fe_val).  fp32 products and sums in the reference's order, without contraction. */
struct FeatherArgs { int S, B, E, osh; int oo[3], on[3]; const uint8_t *e; const uint8_t *nb[8]; const float *u; uint8_t *out; };
/* the row (z, y) of window d's spill, addressed with this window's x: byte x of the row is its value at (z, y, x) */
__device__ __forceinline__ const uint8_t *fe_row(const FeatherArgs &f, int d, int z, int y) {
    if (!d) return f.e + ((size_t)z * f.E + y) * f.E;
    const uint8_t *p = f.nb[d];
    const int uy = y + ((d & 2) ? f.S : 0), ux = (d & 1) ? f.S : 0;
    if (d & 4) return p + ((size_t)z * f.E + uy) * f.E + ux;
    if (d & 2) return p + ((size_t)z * f.B + y) * f.E + ux;
    return p + ((size_t)z * f.S + y) * f.B;
}
/* four bytes of a row from x on (n of them real) */
__device__ __forceinline__ unsigned fe_four(const uint8_t *r, int x, int n) {
    const uint8_t *p = r + x;
    if (n == 4 && !((size_t)p & 3)) return ld_dep((const uint32_t *)p);
    unsigned v = 0u;
    for (int j = 0; j < n; j++) v |= (unsigned)ld_dep(p + j) << (8 * j);
    return v;
}
/* The output box in up to eight parts by which axes lie in the lower shell (bit 0 x, 1 y, 2 z), so that the windows that reach a voxel are the
   part's subsets and every warp runs the sum its part needs and no more.  Blocks [first, next first) of the grid work on a part. */
struct FeatherPart { int z0, y0, x0, nz, ny, nx; unsigned first; };
struct FeatherParts { FeatherPart p[8]; };
/* byte j of v as a float (2^23 + byte, minus 2^23: no conversion unit) */
__device__ __forceinline__ float byte_f(unsigned v, int j) { return __fsub_rn(__uint_as_float(__byte_perm(v, 0x4b000000u, 0x7440u | j)), 8388608.f); }
/* the four bytes of part M at (z, y, x .. x + n): the weighted mean over the windows d within M that are present, in ascending d */
template <int M> __device__ __forceinline__ unsigned fe_mean(const FeatherArgs &f, int z, int y, int x, int n) {
    const unsigned own = fe_four(fe_row(f, 0, z, y), x, n);
    if (M == 0) return own;
    const int B = f.B;
    unsigned b[8]; bool have[8];
#pragma unroll
    for (int d = 0; d < 8; d++) {
        have[d] = d == 0; b[d] = own;
        if (d && (d & ~M) == 0) { have[d] = f.nb[d] != nullptr; if (have[d]) b[d] = fe_four(fe_row(f, d, z, y), x, n); }
    }
    float wz[2] = {1.f, 1.f}, wy[2] = {1.f, 1.f};
#pragma unroll
    for (int k = 0; k < 2; k++) { if (M & 4) wz[k] = ld_dep(f.u + k * B + z); if (M & 2) wy[k] = ld_dep(f.u + k * B + y); }
    unsigned v = 0u;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        float wx[2] = {1.f, 1.f};
        if ((M & 1) && j < n) { wx[0] = ld_dep(f.u + x + j); wx[1] = ld_dep(f.u + B + x + j); }
        float s = 0.f, w = 0.f;
#pragma unroll
        for (int d = 0; d < 8; d++) {
            if ((d & ~M) || !have[d]) continue;
            const float wi = __fmul_rn(__fmul_rn(wz[d >> 2], wy[(d >> 1) & 1]), wx[d & 1]);
            s = __fadd_rn(s, __fmul_rn(wi, byte_f(b[d], j)));
            w = __fadd_rn(w, wi);
        }
        v |= (w > 0.f ? (unsigned)fminf(255.f, __fadd_rn(__fdiv_rn(s, w), 0.5f)) : 0u) << (8 * j);
    }
    return v;
}
template <int M> __device__ __forceinline__ void fe_part(const FeatherArgs &f, const FeatherPart &pt, unsigned nblk) {
    const int nq = (pt.nx + 3) >> 2, R = nq < 256 ? 256 / nq : 1, tr = (int)threadIdx.x / nq;
    const unsigned rows = (unsigned)pt.nz * (unsigned)pt.ny;
    if (R > 1 && tr >= R) return;
    for (unsigned row = (blockIdx.x - pt.first) * (unsigned)R + (R > 1 ? tr : 0); row < rows; row += nblk * (unsigned)R) {
        const int rz = (int)(row / (unsigned)pt.ny), z = pt.z0 + rz, y = pt.y0 + (int)(row - (unsigned)rz * (unsigned)pt.ny);
        for (int q = R > 1 ? (int)threadIdx.x - tr * nq : (int)threadIdx.x; q < nq; q += 256) {
            const int x = pt.x0 + 4 * q, n = min(4, pt.nx - 4 * q);
            uint8_t *o = f.out + ((size_t)(z - f.oo[0]) * f.osh + (y - f.oo[1])) * f.osh + (x - f.oo[2]);
            const unsigned v = fe_mean<M>(f, z, y, x, n);
            if (n == 4 && !((size_t)o & 3)) *(uint32_t *)o = v;
            else for (int j = 0; j < n; j++) o[j] = (uint8_t)(v >> (8 * j));
        }
    }
}
/* A thread takes four x of a row of its part (a block R = 256 / nq whole rows of nq such groups); their bytes come as one word a window where rows
   are aligned, all loads ahead of the sums.  Bound by instruction issue in the shell: 144^3 with seven neighbours 24.5 us at one thread and
   three 64-bit divisions a voxel with the eight windows tested for each, 9.7 us in this form. */
__global__ void __launch_bounds__(256) feather_k(const FeatherArgs f, const FeatherParts parts) {
    pdl_trigger(); pdl_wait();
    int pi = 0;
#pragma unroll
    for (int k = 1; k < 8; k++) if (blockIdx.x >= parts.p[k].first) pi = k;
    const FeatherPart pt = parts.p[pi];
    const unsigned nblk = (pi < 7 ? parts.p[pi + 1].first : gridDim.x) - pt.first;
    switch (7 - pi) {                                         /* the shell first: its blocks take longest */
    case 0: fe_part<0>(f, pt, nblk); break;
    case 1: fe_part<1>(f, pt, nblk); break;
    case 2: fe_part<2>(f, pt, nblk); break;
    case 3: fe_part<3>(f, pt, nblk); break;
    case 4: fe_part<4>(f, pt, nblk); break;
    case 5: fe_part<5>(f, pt, nblk); break;
    case 6: fe_part<6>(f, pt, nblk); break;
    default: fe_part<7>(f, pt, nblk); break;
    }
}
/* a window's upper slabs, kept for the windows after it (feather_keep, src/predict.c:362-376): one T (byte or four-byte word) a thread, indices of type I */
template <typename T, typename I>
__global__ void __launch_bounds__(256) feather_keep_k(const T *e, I S, I B, I SX, I BX, T *__restrict__ zs, T *__restrict__ ys, T *__restrict__ xs) {
    pdl_trigger(); pdl_wait();
    /* S, B, E in voxels; SX, BX, EX along x in units of T */
    const I E = S + B, EX = SX + BX, nz = B * E * EX, ny = S * B * EX, nx = S * S * BX;
    for (I i = blockIdx.x * (I)blockDim.x + threadIdx.x; i < nz + ny + nx; i += (I)gridDim.x * blockDim.x) {
        if (i < nz) zs[i] = ld_dep(e + S * E * EX + i);
        else if (i < nz + ny) { const I k = i - nz, r = k / EX, x = k - r * EX, z = r / B, y = r - z * B; ys[k] = ld_dep(e + (z * E + S + y) * EX + x); }
        else { const I k = i - nz - ny, r = k / BX, x = k - r * BX, z = r / S, y = r - z * S; xs[k] = ld_dep(e + (z * E + y) * EX + SX + x); }
    }
}

int g_logits_h16[16], g_iso[16];
int cur_dev() { int d = 0; cudaGetDevice(&d); return d & 15; }
unsigned grid_of(size_t n) { const size_t g = (n + 255) / 256; return (unsigned)(g < 1 ? 1 : g > 148 * 32 ? 148 * 32 : g); }

template <int MASK>
void place(const char *fn, const void *lg, const uint8_t *ct, const uint32_t *bits, PlaceBox B, int W, int zoff, int oz, int oy, int ox, int shard, uint8_t *dsh) {
    if (!umx_ready(fn)) return;
    const size_t n = (size_t)B.nz * B.ny * ((B.nx + 7) >> 3);
    if (!n) return;
    if ((size_t)B.nz * B.ny >= (size_t)1 << 31) { fprintf(stderr, "%s: 2^31 rows or more\n", fn); abort(); }
    const int d = cur_dev(), iso = g_iso[d] < 1 ? 1 : g_iso[d];
    if (g_logits_h16[d]) umx_launch(pred_place_k<__half, MASK>, dim3(grid_of(n)), dim3(256), 0, (const __half *)lg, ct, bits, B, W, zoff, oz, oy, ox, shard, dsh, iso);
    else umx_launch(pred_place_k<float, MASK>, dim3(grid_of(n)), dim3(256), 0, (const float *)lg, ct, bits, B, W, zoff, oz, oy, ox, shard, dsh, iso);
    g_umx_launches++;
    UMX_CK(fn);
}

}   // namespace

/* src/nn.h:385: the prediction readers take fp16 logits (per device, as the reference's flag is per process with one device a thread) */
extern "C" void nn_set_logits_h16(int on) { g_logits_h16[cur_dev()] = on != 0; }
/* src/nn_elem.cu:1104-1106: outputs only where CT >= t (1: CT > 0) */
extern "C" void nn_set_pred_iso(int t) { g_iso[cur_dev()] = t < 1 ? 1 : t; }
extern "C" int nn_get_pred_iso(void) { const int v = g_iso[cur_dev()]; return v < 1 ? 1 : v; }
/* src/nn_elem.cu:1098-1103: every voxel of a window, no crop; material where CT != 0 */
extern "C" void nn_pred_output(const float *lg, const uint8_t *ct, size_t n, uint8_t *out) {
    if (!umx_ready("nn_pred_output") || !n) return;
    umx_launch(pred_out_k, dim3(grid_of(n)), dim3(256), 0, (const void *)lg, g_logits_h16[cur_dev()], ct, n, out);
    g_umx_launches++;
    UMX_CK("nn_pred_output");
}
/* src/nn_elem.cu:1125-1132 */
extern "C" void nn_pred_place_d(const float *lg, const uint8_t *ct, int D, int W, int hz, int halo, int oz, int oy, int ox, int ez, int ey, int ex, int shard, uint8_t *dsh) {
    place<0>("nn_pred_place_d", lg, ct, nullptr, place_box_of(D, W, hz, halo, oz, oy, ox, ez, ey, ex), W, 0, oz, oy, ox, shard, dsh);
}
extern "C" void nn_pred_place(const float *lg, const uint8_t *ct, int W, int halo, int oz, int oy, int ox, int ez, int ey, int ex, int shard, uint8_t *dsh) {
    nn_pred_place_d(lg, ct, W, W, halo, halo, oz, oy, ox, ez, ey, ex, shard, dsh);
}
/* src/nn_elem.cu:1133-1144: the CT window's material voxels as bits (word k >> 5, bit k & 31) */
extern "C" void nn_pred_ctmask_t(const uint8_t *ct, size_t n, uint32_t *bits, int t) {
    if (!umx_ready("nn_pred_ctmask") || !n) return;
    const size_t words = (n + 31) / 32;
    umx_launch(ctmask_k, dim3((unsigned)((words + 255) / 256)), dim3(256), 0, ct, n, bits, t < 1 ? 1 : t > 255 ? 256 : t);
    g_umx_launches++;
    UMX_CK("nn_pred_ctmask");
}
extern "C" void nn_pred_ctmask(const uint8_t *ct, size_t n, uint32_t *bits) { nn_pred_ctmask_t(ct, n, bits, 1); }
/* src/nn_elem.cu:1145-1160: the same place with the mask bits */
extern "C" void nn_pred_place_m_d(const float *lg, const uint32_t *bits, int D, int W, int hz, int halo, int oz, int oy, int ox, int ez, int ey, int ex, int shard, uint8_t *dsh) {
    place<1>("nn_pred_place_m_d", lg, nullptr, bits, place_box_of(D, W, hz, halo, oz, oy, ox, ez, ey, ex), W, 0, oz, oy, ox, shard, dsh);
}
extern "C" void nn_pred_place_m(const float *lg, const uint32_t *bits, int W, int halo, int oz, int oy, int ox, int ez, int ey, int ex, int shard, uint8_t *dsh) {
    nn_pred_place_m_d(lg, bits, W, W, halo, halo, oz, oy, ox, ez, ey, ex, shard, dsh);
}
/* src/nn_elem.cu:1161-1178: a window held as planes [zoff, zoff + D) (one half of a split window): its planes [zlo, zhi) that lie in the interior */
extern "C" void nn_pred_place_mz(const float *lg, const uint32_t *bits, int W, int halo, int zlo, int zhi, int zoff, int oz, int oy, int ox, int ez, int ey, int ex, int shard, uint8_t *dsh) {
    if (zlo < halo) zlo = halo;
    if (zhi > W - halo) zhi = W - halo;
    if (zhi <= zlo) return;
    PlaceBox B = place_box_of(W, W, halo, halo, oz, oy, ox, ez, ey, ex);
    const int z0 = B.z0 > zlo ? B.z0 : zlo, z1 = B.z0 + B.nz < zhi ? B.z0 + B.nz : zhi;
    B.z0 = z0; B.nz = z1 > z0 ? z1 - z0 : 0;
    place<1>("nn_pred_place_mz", lg, nullptr, bits, B, W, zoff, oz, oy, ox, shard, dsh);
}

/* The seam feather's blend on the device (the arithmetic of fe_blend / fe_rows, src/predict.c:305-333): f->e, f->nb[1..7] (NULL: no such
   window), f->out are device pointers; the interior voxels [oo, oo + on) per axis of this window go to out[(lz osh + ly) osh + lx].
   The weight table of a band width is built on the host (double sin, as feather_init) and kept on the device. */
extern "C" int umx_feather_blend(const umx_feather_t *h) {
    if (!umx_ready("umx_feather_blend")) return -1;
    if (!h || h->S < 1 || h->B < 1 || h->B > 1024 || h->B > h->S || !h->e || !h->out) { umx_latch_msg("umx_feather_blend: bad arguments"); return -1; }
    for (int d = 0; d < 3; d++) if (h->oo[d] < 0 || h->on[d] < 0 || h->oo[d] + h->on[d] > h->S || h->on[d] > h->osh) { umx_latch_msg("umx_feather_blend: output box outside the interior or the shard"); return -1; }
    static float *utab[16]; static int ub[16];
    const int dv = cur_dev();
    if (!utab[dv] || ub[dv] != h->B) {
        float hu[2048];
        for (int j = 0; j < h->B; j++) { const double s = sin(3.14159265358979323846 / 2 * (j + 0.5) / h->B); hu[j] = (float)(s * s); hu[h->B + j] = (float)(1 - s * s); }
        cudaDeviceSynchronize();
        if (!utab[dv]) utab[dv] = (float *)nn_malloc(2048 * sizeof(float));
        if (!utab[dv]) return -1;
        nn_h2d(utab[dv], hu, (size_t)2 * h->B * sizeof(float));
        ub[dv] = h->B;
    }
    FeatherArgs f; memset(&f, 0, sizeof f);
    f.S = h->S; f.B = h->B; f.E = h->S + h->B; f.osh = h->osh; f.e = h->e; f.u = utab[dv]; f.out = h->out;
    for (int d = 0; d < 3; d++) { f.oo[d] = h->oo[d]; f.on[d] = h->on[d]; }
    for (int d = 1; d < 8; d++) f.nb[d] = h->nb[d];
    const size_t n = (size_t)f.on[0] * f.on[1] * f.on[2];
    if (!n) return 0;
    if ((size_t)f.on[0] * f.on[1] >= (size_t)1 << 31) { umx_latch_msg("umx_feather_blend: 2^31 rows or more"); return -1; }
    FeatherParts parts; memset(&parts, 0, sizeof parts);
    int lo[3]; unsigned blocks = 0;
    for (int d = 0; d < 3; d++) lo[d] = f.oo[d] < h->B ? (h->B < f.oo[d] + f.on[d] ? h->B - f.oo[d] : f.on[d]) : 0;      /* voxels of the box below B, per axis */
    for (int k = 0; k < 8; k++) {
        FeatherPart &pt = parts.p[k];
        const int m = 7 - k, bit[3] = {m >> 2 & 1, m >> 1 & 1, m & 1};
        int o[3], n[3];
        for (int d = 0; d < 3; d++) { o[d] = bit[d] ? f.oo[d] : f.oo[d] + lo[d]; n[d] = bit[d] ? lo[d] : f.on[d] - lo[d]; }
        pt = {o[0], o[1], o[2], n[0], n[1], n[2], blocks};
        const size_t rows = (size_t)n[0] * n[1];
        if (!rows || !n[2]) continue;                          /* an empty part gets no block */
        const size_t nq = ((size_t)n[2] + 3) >> 2, per = nq < 256 ? 256 / nq : 1, g = (rows + per - 1) / per;
        blocks += (unsigned)(g < 148 * 32 ? g : 148 * 32);
    }
    umx_launch(feather_k, dim3(blocks), dim3(256), 0, f, parts);
    g_umx_launches++;
    UMX_CK("umx_feather_blend");
    return 0;
}
extern "C" void umx_feather_keep(const uint8_t *e, int S, int B, uint8_t *zslab, uint8_t *yslab, uint8_t *xslab) {
    if (!umx_ready("umx_feather_keep") || S < 1 || B < 1) return;
    const size_t E = (size_t)S + B, n = B * E * E + (size_t)S * B * E + (size_t)S * S * B;
    /* words where every row starts on one; 32-bit indices while the window has fewer than 2^32 bytes */
    const bool words = !((S | B) & 3) && !(((size_t)e | (size_t)zslab | (size_t)yslab | (size_t)xslab) & 3);
    if (E * E * E >= (size_t)1 << 32) umx_launch(feather_keep_k<uint8_t, size_t>, dim3(grid_of(n)), dim3(256), 0, e, S, B, S, B, zslab, yslab, xslab);
    else if (words) umx_launch(feather_keep_k<uint32_t, unsigned>, dim3(grid_of(n / 4)), dim3(256), 0, (const uint32_t *)e, S, B, S / 4, B / 4, (uint32_t *)zslab, (uint32_t *)yslab, (uint32_t *)xslab);
    else umx_launch(feather_keep_k<uint8_t, unsigned>, dim3(grid_of(n)), dim3(256), 0, e, S, B, S, B, zslab, yslab, xslab);
    g_umx_launches++;
    UMX_CK("umx_feather_keep");
}
