/* Host side of the z-marching 3^3 kernel (conv_tcr.cuh): geometry, choice, launch. */
#include "conv_tcr.cuh"

/* Self-test of the bounded wait and of its report: one block waits, for `limit_clocks` at most, on a barrier that nobody arrives on, gives
   up, and leaves the same record a conv role would (role code 1, stage 123).  Returns 0 when the kernel ran; lp_check() then holds the
   "bounded wait gave up" message.  The context stays usable. */
__global__ void wait_selftest_k(ConvRArgs a, long long limit) {
    __shared__ uint64_t bar; __shared__ int abort_s;
    if (threadIdx.x == 0) { mbar_init(smem_u32(&bar), 1); abort_s = 0; fence_barrier_init(); }
    __syncthreads();
    if (threadIdx.x == 0 && !mbar_wait(smem_u32(&bar), 0, &abort_s, limit)) raise_r(a, &abort_s, 1, 123, 0, 0);
}
extern "C" int umx_wait_selftest(long long limit_clocks) {
    if (!umx_ready("umx_wait_selftest")) return -1;
    if (limit_clocks < 1 || limit_clocks > 2000000000ll) limit_clocks = 2000000;
    ConvRArgs a; memset(&a, 0, sizeof a);
    a.err = umx_errflag(); if (!a.err) return -1;
    wait_selftest_k<<<1, 32>>>(a, limit_clocks);
    g_umx_launches++;
    UMX_CK("umx_wait_selftest");
    return 0;
}

/* geometry of the weight image; 0 when the z-marching kernel cannot run this conv (3^3 only; a column tile's codes + scales resident in shared memory,
   its B scales resident in TMEM beside at least four accumulator slots) */
struct RGeo { int nt, ncol, w_codes, w_bytes, gt, goff1, goff2, tmem_cols, nslot, sfa_base, sfa_cols, sfb_base; };
static int r_geometry_nt(const umx_conv *c, int nt, RGeo *g) {
    if (c->cop % nt) return 0;
    g->nt = nt; g->ncol = c->cop / nt;
    const int g0 = (3 * nt + 127) / 128, g1 = (2 * nt + 127) / 128, g2 = (nt + 127) / 128;
    g->goff1 = g0; g->goff2 = g0 + g1; g->gt = g0 + g1 + g2;
    g->w_codes = c->nki * 9 * 2 * 3 * nt * 16;
    g->w_bytes = g->w_codes + c->nki * c->nquad * g->gt * 512;
    if (g->w_bytes > 136 * 1024) return 0;
    g->sfa_cols = c->nquad * 4;
    const int fixed = 2 * g->sfa_cols + c->nki * c->nquad * g->gt * 4;
    /* 256 columns (two blocks a multiprocessor) when that leaves four slots, else the whole 512 */
    g->tmem_cols = (256 - fixed) / nt >= 4 ? 256 : 512;
    g->nslot = (g->tmem_cols - fixed) / nt;
    if (g->nslot > kMaxSlots) g->nslot = kMaxSlots;
    if (g->nslot < 4) return 0;
    g->sfa_base = g->nslot * nt; g->sfb_base = g->sfa_base + 2 * g->sfa_cols;
    return 1;
}
/* the widest column tile (64 or 32 channels) whose weight image fits; wider layers run as several column tiles, each on its own
   share of the blocks (the input is then read once per column tile, from L2 when it fits there) */
static int r_geometry(const umx_conv *c, RGeo *g) {
    if (c->kind != UMX_CONV3) return 0;
    if (c->cop <= 64 && r_geometry_nt(c, c->cop, g)) return 1;
    if (r_geometry_nt(c, 64, g)) return 1;
    return r_geometry_nt(c, 32, g);
}
/* upper bound on the blocks per column tile (0: as many as the device holds): lets a small grid be cut into the multi-run pieces, wrapped
   slot windows and several-planes-a-block regime that otherwise only volumes with thousands of tile planes reach */
static int g_r_block_cap = 0;
extern "C" void umx_conv_r_block_cap(int cap) { g_r_block_cap = cap > 0 ? cap : 0; }
int umx_conv_r_cap(void) { return g_r_block_cap; }                /* the stride-2 kernel's too */
/* Weight image of the z-marching kernel (made by umx_prep_w27): codes [input item][dy dx][k half][dz * nt + channel][16 B], then the B scale
   bytes in the TMEM scale layout per (input item, tap quad, first dz of the MMA, 128-row group): byte (lane, column, id) = row 128 g + 32
   column + lane counted from that dz's first row, tap 4 q + id (fp8) or tap 2 q + id / 2, block id % 2 (fp4).  A block-scaled MMA wants its
   scale address on a 4-column boundary of TMEM (a one-column offset faults with "misaligned address"), hence one re-based image per
   starting dz.  0 when the kernel cannot run this conv. */
int umx_conv_r_image(const umx_conv *c, RImageGeo *o) {
    RGeo g;
    if (!r_geometry(c, &g)) return 0;
    o->nt = g.nt; o->ncol = g.ncol; o->w_bytes = g.w_bytes; o->w_codes = g.w_codes; o->gt = g.gt; o->goff1 = g.goff1; o->goff2 = g.goff2;
    return 1;
}
int umx_conv_ksplit(const umx_conv *c, int D, int H, int W, int sms);       /* conv_tc.cu */
/* the launch of this geometry, everything but the operands; 0 when the kernel does not apply */
static int r_plan(const umx_conv *c, const uint8_t *x_sc, int N, int D, int H, int W, const EpiArgs &e, int want_coef, const double *part, ConvRArgs &a, int *grid) {
    memset(&a, 0, sizeof a);
    RGeo g;
    if (!r_geometry(c, &g)) return 0;
    a.gather = (W & 15) || ((size_t)x_sc & 15);      /* TMA takes the scale plane only in rows that are multiples of 16 bytes */
    a.w_codes = g.w_codes; a.w_bytes = g.w_bytes; a.gt = g.gt; a.goff1 = g.goff1 * 4; a.goff2 = g.goff2 * 4;   /* TMEM column offsets of the dz >= 1, 2 images */
    a.tmem_cols = g.tmem_cols; a.nslot = g.nslot; a.sfa_base = g.sfa_base; a.sfa_cols = g.sfa_cols; a.sfb_base = g.sfb_base;
    a.N = N; a.D = D; a.H = H; a.W = W; a.nkb = c->nkb; a.nki = c->nki; a.bits = c->bits; a.nt = g.nt; a.ncol = g.ncol;
    a.tiles_x = (W + 7) / 8; a.tiles = a.tiles_x * ((H + 15) / 16);
    a.units = (long long)N * a.tiles * D;
    a.nquad = c->nquad;
    a.fast_h16 = e.out_mode == UMX_OUT_H16B && !e.tconv && (want_coef || !((size_t)e.y & 31));      /* stores of 32 bytes */
    a.fast_pm16 = e.out_mode == UMX_OUT_PM16 && !e.tconv && !((size_t)e.y & 15) && !(W & 7);        /* tile rows are aligned and whole */
    if (want_coef && (!a.fast_h16 || !part || g.ncol > 64 || a.gather)) return 0;
    a.cop = c->cop;
    /* the codes and the scale window are TMA destinations (128-byte aligned) */
    a.offSW = 5888; a.offSFA = a.offSW + (c->bits == 8 ? 640 : 1152);
    a.item_bytes = a.offSFA + c->nquad * 512;                          /* a multiple of 128 */
    a.stage_bytes = (a.item_bytes + 1023) & ~1023;
    a.off_rec = 1024; a.off_bias = a.off_rec + 12 * 64; a.off_stage = 2048; a.off_red = a.off_stage; a.off_w = a.off_stage + (want_coef ? 8192 * (g.nt == 32 ? 1 : 2) : a.fast_pm16 ? 8192 : 0); a.off_ring = (a.off_w + a.w_bytes + 1023) & ~1023;
    int dev = 0, sms = 148; cudaGetDevice(&dev);
    { static int sms_of[16]; if (!sms_of[dev & 15]) { int v = 148; cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev); sms_of[dev & 15] = v; } sms = sms_of[dev & 15]; }   /* looked up once per device */
    /* two blocks a multiprocessor when shared memory (113 KB each) and TMEM (256 columns each) allow */
    const int two = g.tmem_cols == 256 && a.off_ring + 4 * a.stage_bytes <= 113 * 1024;
    const int room = (two ? 113 : 227) * 1024 - a.off_ring;
    long long slots = (long long)sms * (two ? 2 : 1) / g.ncol;      /* blocks per column tile */
    if (slots < 1) return 0;
    if (g_r_block_cap && slots > g_r_block_cap) slots = g_r_block_cap;
    /* Input items of a stage: what the MMA warp does once a stage (its barrier, record and commit, some 380 clocks) is as much as half of an item's MMAs, so a stage takes as many items
       of its plane as leave three stages, at most four, where a block has four planes or more (with fewer, the first MMAs wait for more bytes than that is worth: 64 -> 64 on 32^3
       12.7 us, 13.6 with two).  With one item and this way, us, 128 -> 64 on 64^3 63.9 and 56.9, 96 -> 32 on 64^3 31.8 and 30.2, 64 -> 32 on 128^3 115.6 and 112.1; MX-fp4 128 -> 64 on
       64^3 31.3 and 30.3. */
    a.ips = 1;
    if (!a.gather && !want_coef && a.units >= 4 * slots) for (int k = 2; k <= 4 && k <= a.nki; k++) if (3 * k * a.item_bytes <= room) a.ips = k;
    if (a.ips > 1) a.stage_bytes = a.ips * a.item_bytes;
    a.ring = room / a.stage_bytes; if (a.ring > 12) a.ring = 12;
    if (a.ring < 3) return 0;
    /* What the general kernel does with the call.  In MX-fp4, or with one input item, it adds in this kernel's order (a dz at a time, the items within it) unless it splits K, which it does by
       one sample's geometry: the bits are the same, and the choice follows all samples' planes.  Otherwise it follows from one sample's, so that the result does not depend on the batch; and the
       layers of a network (blocked halves) stay with the order that they have at that size: the last bit of the sums decides codes next to a rounding boundary, which the layers behind make
       0.05 (three levels) to 0.07 (four) of the logits, relative L2. */
    const long long units1 = (long long)a.tiles * D;
    const bool same = (c->bits == 4 || c->nki == 1) && umx_conv_ksplit(c, D, H, W, sms) == 1, keep = !same && e.out_mode == UMX_OUT_H16B;
    const long long planes = same ? a.units : units1;
    /* A block here pays two halo planes a run and loads its weights first, so with several column tiles and fewer than eight planes a block the general kernel is faster while one wave of
       its blocks, two a multiprocessor, holds the call, and slower once it takes a second.  General kernel and this one, us, fp8 / fp4: 32 -> 128 on 32^3 (256 of its blocks) 9.2 and 11.3 /
       9.4 and 10.6, two samples (512) 16.7 and 15.7 / 17.7 and 14.3; 64 -> 256 on 24 x 20 x 32 (384) 19.4 and 15.4 / 16.5 and 12.6; 32 -> 96 on 32^3 (256) 8.2 and 9.0, two samples 15.0 and
       11.6 / 16.3 and 11.5; 128 -> 128 on 24 x 20 x 32, two samples, fp4 22.3 and 14.6.  Volumes with fewer planes than blocks are left here: nothing to gain either way. */
    if (g.ncol > 1 && units1 >= slots && units1 < 8 * slots && (keep || planes * ((c->cop + 127) / 128) <= 2 * sms)) return 0;
    /* The scale warp that gathers costs 3 to 8 % in MX-fp8 and 6 to 27 in MX-fp4 against the TMA window, and a piece's start, so few planes, and a column tile that re-reads the
       input, are the general kernel's.  General kernel and this one, us: 32 -> 32 fp4 on 33 x 31 x 30 (264 planes) 6.9 and 9.0, on 36^3 (540) 14.5 and 11.6, on 63 x 61 x 66 45 and
       17; fp8 64 -> 32 on 80 x 80 x 84 112 and 43; 64 columns, fp4 128 -> 64 plane-major on 36^3 23.0 and 24.6, on 40 x 35 x 42 (720) 33.0 and 29.0; two column tiles, fp8 32 -> 128 on
       63 x 61 x 66 91 and 124. */
    if (a.gather && (keep || g.ncol > 1 || 2 * planes < (g.nt == 32 ? 7ll : 9ll) * (slots < sms ? slots : sms))) return 0;
    a.gcol = (int)(a.units < slots ? a.units : slots); if (a.gcol > 512) a.gcol = 512;
    *grid = a.gcol * g.ncol;
    return 1;
}
/* would umx_conv_fwd_r take this conv (its weight image aside)? */
int umx_conv_r_takes(const umx_conv *c, const uint8_t *x_sc, int N, int D, int H, int W, const EpiArgs &e) {
    ConvRArgs a; int grid;
    return r_plan(c, x_sc, N, D, H, W, e, 0, nullptr, a, &grid);
}
/* x_sc: the MX tensor's scale plane; m0: tensor map over its codes (fp8 in the split layout; ref: in the reference's); enc: the driver's tensor-map encoder (for the scale plane).
   Returns 1 when this kernel does not apply to the geometry (the caller then takes the general kernel), 0 after a launch, -1 on error. */
/* coef != NULL (only with the blocked fp16 output): InstanceNorm coefficients are produced by the same launch; part then holds N x (blocks per
   column tile, at most 512) x cop x 2 doubles of scratch */
int umx_conv_fwd_r(const umx_conv *c, const uint8_t *x_sc, const CUtensorMap *m0, int ref, void *enc_v, int N, int D, int H, int W, const EpiArgs &e,
                   double *part, const float *gamma, const float *beta, float eps, float *coef) {
    typedef CUresult (*encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    ConvRArgs a; int grid;
    if (!c->wr || !r_plan(c, x_sc, N, D, H, W, e, coef != nullptr, part, a, &grid)) return 1;
    a.part = part; a.coef = coef; a.gamma = gamma; a.beta = beta; a.eps = eps;
    int dev = 0; cudaGetDevice(&dev);
    const size_t S = (size_t)D * H * W;
    CUtensorMap ms; memset(&ms, 0, sizeof ms);
    if (!a.gather) {
        /* MX-fp4: samples as a dimension of their own, so that the second block of an item past the last one reads the fill, not the next sample's scales (whose NaN would come through the
           zero weights); MX-fp8 reads one block at a time, over all samples' blocks in a row */
        const bool f8 = c->bits == 8;
        const cuuint64_t gd[5] = {(cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D, (cuuint64_t)c->nkb * (f8 ? N : 1), (cuuint64_t)N};
        const cuuint64_t gs[4] = {(cuuint64_t)W, (cuuint64_t)W * H, (cuuint64_t)S, (cuuint64_t)S * c->nkb};
        const cuuint32_t box[5] = {32, 18, 1, f8 ? 1u : 2u, 1}, es[5] = {1, 1, 1, 1, 1};
        const CUresult r0 = ((encode_fn)enc_v)(&ms, CU_TENSOR_MAP_DATA_TYPE_UINT8, f8 ? 4 : 5, (void *)x_sc, gd, gs, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r0 != CUDA_SUCCESS) return 1;                        /* e.g. a scale plane that is not 16-byte aligned: take the general kernel */
    }
    a.wr = c->wr; a.x_sc = x_sc; a.w_dep = c->w_src != nullptr; a.e = e; a.err = umx_errflag();
    if (!a.err) return -1;
    const size_t smem = (size_t)a.off_ring + (size_t)a.ring * a.stage_bytes;
    static const conv_r_fn *const ks[5] = {umx_conv_r_one, umx_conv_r_stats, umx_conv_r_gather, umx_conv_r_multi, umx_conv_r_ends};
    const int form = coef ? 1 : a.gather ? (gather_ends(N, c->nkb, D, H, W) ? 4 : 2) : a.ips > 1 ? 3 : 0, variant = (ref ? 4 : c->bits == 8 ? 0 : 2) | (a.nt == 32 ? 0 : 1);
    /* the attribute loads the form's kernels (1.3 ms) the first time: only when one is launched */
    static unsigned attr_set[16];
    const unsigned bit = 1u << (6 * form + variant);
    if (!(attr_set[dev & 15] & bit)) {
        const cudaError_t er = cudaFuncSetAttribute((const void *)ks[form][variant], cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (er != cudaSuccess) { umx_latch("umx_conv_fwd: shared memory attribute", er); return -1; }
        __atomic_fetch_or(&attr_set[dev & 15], bit, __ATOMIC_RELAXED);
    }
    umx_launch(ks[form][variant], dim3(grid), dim3(kThreadsR), smem, *m0, ms, a);
    return 0;
}
