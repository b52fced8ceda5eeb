/* 3^3 stride-2 pad-1 MX conv forward, persistent and z-marching, for layers whose prepared weights fit in shared memory (MX-fp8 up to 64 input channels with 64
   outputs a column tile, up to 160 with 32; MX-fp4 twice that).

   Output voxel v reads the input voxels 2 v + tap - 1: per axis an even input coordinate belongs to one tap (1), an odd one to two (2 of the voxel below it, 0 of the
   voxel above it).  So an input plane comes into shared memory as its four (y, x) parity classes, each through its own TMA map with a traversal stride of two voxels: even
   rows and columns 16 x 8 of them, odd ones one more.  Every one of the nine (dy, dx) taps is then a view of one class, at most a row and a column further on, in
   the canonical K-major operand form (8 voxels x 16 B core matrices, row groups 128 or 144 bytes apart).  An odd input plane feeds two output planes: their weights (dz =
   0 for the plane above, dz = 2 for the one below) are stacked along N, and the accumulators of consecutive output planes sit in consecutive TMEM slots, newest first.
   A block marches along z: two input planes an output plane, each read once, where a tile of its own for every tap (the general kernel's form, conv_tc.cu) moves 27
   tiles of 128 voxels an output tile: 110 KB through the L2 where this form moves 36, and the weights once a block instead of once a tile.  The input is read as it
   is, in the reference's layout (16 bytes of every second 32-byte row) or the split one: no relayout pass.

   32 -> 64 channels on 96^3 take about 13 us, 39 in the general kernel behind 9 us of relayout; figures and the rule are at umx_conv_s2_takes.

   Roles (320 threads): warp 0 producer (stage records, weights, TMA), warp 1 TMEM, scale copies and MMA issue, warps 2-5 scale gather (a thread a GEMM row, two stages ahead),
   warps 6-9 epilogue.  A stage is one input plane of one K item (32 fp8 or 64 fp4 channels).  All waits are bounded as in conv_mx_k. */
#include "conv_epi.cuh"
#include "tc_ptx.cuh"
#include <stdlib.h>
#include <string.h>

namespace {

constexpr int kThreadsS = 320;
constexpr int kMaxSlotsS = 8, kMaxRingS = 8;
constexpr long long kWaitLimitS = 4000000000ll;
/* the parity classes of a stage: [even y even x][even y odd x][odd y even x][odd y odd x], each [k half][row][voxel][16 B]; a half is a TMA destination of its own
   (128-byte aligned) */
constexpr int kOffEO = 2 * 2048, kOffOE = kOffEO + 2 * 2304, kOffOO = kOffOE + 2 * 2176, kCodesS = kOffOO + 2 * 2560;
constexpr uint32_t kTxS = 2u * (16 * 8 + 16 * 9 + 17 * 8 + 17 * 9) * 16u;

struct ConvSArgs {
    int N, D, H, W, Di, Hi, Wi;                  /* output and input grid */
    int nbi, nki, nt;                            /* 32-channel blocks of the input, K items, column tile */
    int tiles_x, tiles, gcol;                    /* blocks per column tile */
    long long units;                             /* N x tiles x D output planes of one tile, split evenly over the blocks */
    int ring, stage_bytes, nquad, nslot, tmem_cols, sfa_base, sfa_cols, sfb_base, w_bytes, w_codes;
    int off_w, off_ring;
    int c_half, p_blk, p_half;                   /* TMA coordinates of half h of block b: byte c_half h of a row, plane p_blk b + p_half h */
    int w_dep;                                   /* the weights and the bias were written by a kernel just ahead in the stream */
    const uint8_t *x_sc, *wr;
    EpiArgs e;
    int *err;
};
/* first group: accumulator, instruction descriptor with N, B descriptor of tap 0, B scales; second group when the two slots of an odd plane wrap around the slot ring;
   accumulator-empty barrier to pass first (address | parity << 31), accumulator-full barrier to commit to, last stage of the block */
struct RecS { uint32_t d1, idn1, bb1, sfb1, d2, idn2, bb2, sfb2, wait, commit, last, pad; };
static_assert(sizeof(RecS) == 48, "stage record is 48 bytes");

__device__ __forceinline__ void raise_s(const ConvSArgs &a, volatile int *abort_flag, int code, int stage, uint32_t bar_off = 0, uint32_t parity = 0) {
    if (atomicCAS(a.err, 0, code) == 0) { a.err[1] = (int)blockIdx.x; a.err[2] = stage; a.err[3] = (int)threadIdx.x; __threadfence(); }
    if (((volatile int *)a.err)[1] == (int)blockIdx.x && code < 8) { int *d = a.err + 16 + 4 * code; d[0] = stage; d[1] = (int)bar_off; d[2] = (int)parity; d[3] = 1; }
    *abort_flag = 1;
    __threadfence_block();
}
/* the block's piece of the list of output planes, u = (sample * tiles + tile) * D + z, cut into runs along z */
struct RunS { int n, txy, zb, ze; };
struct PieceS {
    long long u, u1;
    __device__ __forceinline__ explicit PieceS(const ConvSArgs &a) { const long long b = (long long)(blockIdx.x % a.gcol); u = a.units * b / a.gcol; u1 = a.units * (b + 1) / a.gcol; }
    __device__ __forceinline__ bool more() const { return u < u1; }
    __device__ __forceinline__ RunS next(const ConvSArgs &a) {
        const long long col = u / a.D; RunS r;
        r.zb = (int)(u - col * a.D); r.ze = (int)min((long long)a.D, (long long)r.zb + (u1 - u));
        r.n = (int)(col / a.tiles); r.txy = (int)(col - (long long)r.n * a.tiles);
        u += r.ze - r.zb;
        return r;
    }
};
/* the nine (dy, dx) MMAs of a group: the view of tap j is a constant away from the stage's base, its row pitch that of its class */
template <int BITS, int NT>
__device__ __forceinline__ void s2_group(uint32_t d, uint32_t idn, uint32_t bb, uint32_t sfb, uint32_t a_lo, uint32_t sfa, uint32_t lead) {
    constexpr int IPQ = BITS == 8 ? 4 : 2;
#pragma unroll
    for (int j = 0; j < 9; j++) {
        const int dy = j / 3, dx = j % 3, oddy = dy != 1, oddx = dx != 1;
        const uint32_t half = oddy ? (oddx ? 2560u : 2176u) : (oddx ? 2304u : 2048u), pitch = oddx ? 144u : 128u;
        const uint32_t off = (oddy ? (oddx ? kOffOO : kOffOE) : (oddx ? kOffEO : 0)) + (dy == 2 ? pitch : 0u) + (dx == 2 ? 16u : 0u);
        const uint64_t ad = desc_make(a_lo + ((off >> 4) | ((half >> 4) << 16)), desc_hi(pitch)), bd = desc_make(bb + (uint32_t)j * (2u * 3u * NT), desc_hi(128));
        const int q = j / IPQ, id = (j % IPQ) * (4 / IPQ);
        const uint32_t idesc = idn | ((uint32_t)id << 4) | ((uint32_t)id << 29);
        if (BITS == 8) umma_mxf8(d, ad, bd, idesc, 1u, sfa + 4 * q, sfb + 12 * q, lead);
        else umma_mxf4(d, ad, bd, idesc, 1u, sfa + 4 * q, sfb + 12 * q, lead);
    }
}

template <int BITS, int NCH>
__global__ void __launch_bounds__(kThreadsS, 1) conv_s2_k(const __grid_constant__ CUtensorMap mee, const __grid_constant__ CUtensorMap meo, const __grid_constant__ CUtensorMap moe,
                                                          const __grid_constant__ CUtensorMap moo, const ConvSArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    constexpr int NT = 32 * NCH, NQ = BITS == 8 ? 3 : 5, NB = BITS == 8 ? 9 : 18;
    uint64_t *bars = (uint64_t *)smem_raw;
    uint32_t *tmem_slot = (uint32_t *)(smem_raw + 512);
    volatile int *abort_flag = (volatile int *)(smem_raw + 516);
    RecS *recs = (RecS *)(smem_raw + 640);
    float *bias_s = (float *)(smem_raw + 640 + kMaxRingS * sizeof(RecS));
    uint8_t *wsm = smem_raw + a.off_w, *stages = smem_raw + a.off_ring;
    const int warp = (int)uni(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int R = a.ring, NS = a.nslot;
    /* barriers: codes landed, A scales laid out, stage consumed; accumulator full / empty per slot; weights */
    const uint32_t bar_tma = smem_u32(bars), bar_sf = bar_tma + 8 * kMaxRingS, bar_empty = bar_sf + 8 * kMaxRingS, bar_accf = bar_empty + 8 * kMaxRingS, bar_acce = bar_accf + 8 * kMaxSlotsS, bar_w = bar_acce + 8 * kMaxSlotsS;
    if (threadIdx.x == 0) {
        for (int i = 0; i < R; i++) { mbar_init(bar_tma + 8 * i, 1); mbar_init(bar_sf + 8 * i, 4); mbar_init(bar_empty + 8 * i, 1); }
        for (int i = 0; i < NS; i++) { mbar_init(bar_accf + 8 * i, 1); mbar_init(bar_acce + 8 * i, 4); }
        mbar_init(bar_w, 1);
        *abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), (uint32_t)a.tmem_cols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();                               /* the next kernel cannot take this block's tensor memory any more */
    const uint32_t tmem = uni(*tmem_slot);
    const int ctile = (int)blockIdx.x / a.gcol;
    PieceS piece(a);

    if (warp == 0) {
        /* ---------------- producer ---------------- */
        const uint32_t lead = elect_one();
        if (lead) { tma_prefetch_desc(&mee); tma_prefetch_desc(&meo); tma_prefetch_desc(&moe); tma_prefetch_desc(&moo); }
        if (a.w_dep) pdl_wait();                /* else the weights are constants of the layer and load while the kernel before is still running */
        if (lead) {
            mbar_expect_tx(bar_w, (uint32_t)a.w_bytes);
            for (int o = 0; o < a.w_bytes; o += 32768) bulk_g2s(smem_u32(wsm + o), a.wr + (size_t)ctile * a.w_bytes + o, (uint32_t)min(32768, a.w_bytes - o), bar_w);
        }
        if (!a.w_dep) pdl_wait();
        const uint32_t b_lo0 = desc_lo(smem_u32(wsm), 3u * NT * 16u), bstep9 = 9u * 2u * 3u * NT;
        const uint32_t idesc_b = BITS == 8 ? idesc_mxf8(0, 0, 0) : idesc_mxf4(0, 0, 0), ntn = (uint32_t)(NT >> 3) << 17;
        const uint32_t sfb_t0 = tmem + (uint32_t)a.sfb_base;
        int s = 0, ph = 0, it = 0; bool ok = true;
        int pos = NS - 1; uint32_t wp = 1u;     /* ring position and wrap parity of the newest output plane started so far */
        while (piece.more() && ok) {
            const RunS rn = piece.next(a);
            const bool last_run = !piece.more();
            const int x0 = (rn.txy % a.tiles_x) * 16, y0 = (rn.txy / a.tiles_x) * 32;      /* input coordinates of the tile */
            const int zlo = max(0, 2 * rn.zb - 1), zhi = min(a.Di - 1, 2 * rn.ze - 1);
            for (int zi = zlo; zi <= zhi && ok; zi++) {
                const bool odd = zi & 1, up = odd && (zi + 1) / 2 < rn.ze, down = odd && (zi - 1) / 2 >= rn.zb;     /* dz = 0 of the plane above, dz = 2 of the plane below */
                uint32_t w0 = 0u, done = 0u;
                if (up || zi == 0) {
                    if (++pos == NS) { pos = 0; wp ^= 1u; }
                    w0 = (bar_acce + 8u * (uint32_t)(NS - 1 - pos)) | (wp << 31);
                }
                const int slot = NS - 1 - pos, older = slot + 1 < NS ? slot + 1 : 0;
                if (down) done = bar_accf + 8u * (uint32_t)(up ? older : slot);
                else if (!odd && zi == a.Di - 1) done = bar_accf + 8u * (uint32_t)slot;
                const bool both = up && down, wrap = both && older == 0;
                const uint32_t row = odd ? (up ? 0u : (uint32_t)NT) : 2u * NT, img = odd ? (up ? 0u : 4u) : 8u;
                for (int ki = 0; ki < a.nki; ki++) {
                    if (!__all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, kWaitLimitS))) { if (lane == 0) raise_s(a, abort_flag, 1, it, bar_empty + 8 * s - bar_tma, ph ^ 1); ok = false; break; }
                    const uint32_t bar = bar_tma + 8 * s, sb = smem_u32(stages + (size_t)s * a.stage_bytes);
                    const bool kl = ki == a.nki - 1;
                    if (lead) {
                        const uint32_t bk = b_lo0 + (uint32_t)ki * bstep9, sk = sfb_t0 + (uint32_t)(ki * NQ * 12);
                        uint4 *r = (uint4 *)(recs + s);
                        r[0] = make_uint4(tmem + (uint32_t)(slot * NT), idesc_b | (both && !wrap ? 2u * ntn : ntn), bk + row, sk + img);
                        r[1] = make_uint4(tmem, wrap ? idesc_b | ntn : 0u, bk + NT, sk + 4u);
                        r[2] = make_uint4(ki == 0 ? w0 : 0u, kl ? done : 0u, last_run && zi == zhi && kl, 0u);
                        mbar_expect_tx(bar, kTxS);
                    }
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int c = a.c_half * h, p = (rn.n * a.nbi + (BITS == 8 ? ki : 2 * ki)) * a.p_blk + a.p_half * h;
                        tma_load_5d(sb + h * 2048, &mee, bar, c, x0, y0, zi, p, lead);
                        tma_load_5d(sb + kOffEO + h * 2304, &meo, bar, c, x0 - 1, y0, zi, p, lead);
                        tma_load_5d(sb + kOffOE + h * 2176, &moe, bar, c, x0, y0 - 1, zi, p, lead);
                        tma_load_5d(sb + kOffOO + h * 2560, &moo, bar, c, x0 - 1, y0 - 1, zi, p, lead);
                    }
                    it++; if (++s == R) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        /* ---------------- MMA issue: the warp runs the loop on uniform values, one lane issues ---------------- */
        const uint32_t lead = elect_one(), sf_hi = desc_hi(128);
        bool ok = __all_sync(0xffffffffu, mbar_wait(bar_w, 0, abort_flag, kWaitLimitS));
        if (!ok && lane == 0) raise_s(a, abort_flag, 6, 0);
        tc_fence_after();
        const uint32_t wbase = smem_u32(wsm);
        if (ok) for (int i = 0; i < a.nki * NQ * 3; i++) utccp_32x128b(tmem + a.sfb_base + i * 4, desc_make(desc_lo(wbase + a.w_codes + i * 512, 0), sf_hi), lead);
        const uint32_t a_lo0 = desc_lo(smem_u32(stages), 0), a_step = (uint32_t)a.stage_bytes >> 4;
        int s = 0, ph = 0, it = 0;
        while (ok) {
            if (!__all_sync(0xffffffffu, mbar_wait(bar_sf + 8 * s, ph, abort_flag, kWaitLimitS))) { if (lane == 0) raise_s(a, abort_flag, 3, it, bar_sf + 8 * s - bar_tma, ph); break; }
            if (!__all_sync(0xffffffffu, mbar_wait(bar_tma + 8 * s, ph, abort_flag, kWaitLimitS))) { if (lane == 0) raise_s(a, abort_flag, 2, it, 8 * s, ph); break; }
            /* the record goes to registers before anything is committed: the commit of `empty` hands it back to the producer */
            const uint4 *r = (const uint4 *)(recs + s);
            const uint4 g1 = uni(r[0]), g2 = uni(r[1]), c = uni(r[2]);
            if (c.x && !__all_sync(0xffffffffu, mbar_wait(c.x & 0x7fffffffu, c.x >> 31, abort_flag, kWaitLimitS))) { if (lane == 0) raise_s(a, abort_flag, 7, it, (c.x & 0x7fffffffu) - bar_tma, c.x >> 31); break; }
            tc_fence_after();
            const uint32_t a_lo = a_lo0 + (uint32_t)s * a_step, sfa_t = tmem + (uint32_t)a.sfa_base + ((uint32_t)it & 1u) * (uint32_t)a.sfa_cols;
            /* copies and MMAs of one thread run in issue order: a buffer is overwritten after the MMAs that read it two stages ago */
#pragma unroll
            for (int q = 0; q < NQ; q++) utccp_32x128b(sfa_t + 4 * q, desc_make(a_lo + (kCodesS >> 4) + 32u * q, sf_hi), lead);
            s2_group<BITS, NT>(g1.x, g1.y, g1.z, g1.w, a_lo, sfa_t, lead);
            if (g2.y) s2_group<BITS, NT>(g2.x, g2.y, g2.z, g2.w, a_lo, sfa_t, lead);
            umma_commit(bar_empty + 8 * s, lead);
            if (c.y) umma_commit(c.y, lead);
            it++; if (++s == R) { s = 0; ph ^= 1; }
            if (c.z) break;
        }
    } else if (warp < 6) {
        /* ---------------- A scales: a thread owns a GEMM row and fetches the scale bytes of its nine taps from the scale plane, two stages ahead of their use ---------------- */
        const int q4 = warp & 3, r = q4 * 32 + lane, ry = r >> 3, rx = r & 7;
        const size_t hwi = (size_t)a.Hi * a.Wi;
        pdl_wait();
        struct Cur { RunS rn; int zi, zhi, ki, off; unsigned inm; bool live; };
        PieceS pc = piece;
        Cur c; c.live = false; c.zi = 1; c.zhi = 0; c.ki = 0;
        auto open = [&]() {                      /* the next run */
            c.live = pc.more();
            if (!c.live) return;
            c.rn = pc.next(a);
            c.zi = max(0, 2 * c.rn.zb - 1); c.zhi = min(a.Di - 1, 2 * c.rn.ze - 1); c.ki = 0;
            const int iy = 2 * ((c.rn.txy / a.tiles_x) * 16 + ry) - 1, ix = 2 * ((c.rn.txy % a.tiles_x) * 8 + rx) - 1;
            c.off = iy * a.Wi + ix; c.inm = 0u;
#pragma unroll
            for (int j = 0; j < 9; j++) { const int yy = iy + j / 3, xx = ix + j % 3; if (yy >= 0 && yy < a.Hi && xx >= 0 && xx < a.Wi) c.inm |= 1u << j; }
        };
        auto fetch = [&](unsigned *raw) {        /* the stage at the cursor, then on to the next; voxels outside the grid have zero codes and scale 1 */
            if (!c.live) return;
            const int blk = BITS == 8 ? c.ki : 2 * c.ki;
            const uint8_t *p = a.x_sc + (((size_t)c.rn.n * a.nbi + blk) * a.Di + c.zi) * hwi + c.off;
            const bool two = BITS == 4 && blk + 1 < a.nbi;
#pragma unroll
            for (int j = 0; j < 9; j++) {
                const bool in = (c.inm >> j) & 1u;
                const int o = (j / 3) * a.Wi + j % 3;
                raw[j] = in ? ld_dep(p + o) : 127u;
                if (BITS == 4) raw[9 + j] = in && two ? ld_dep(p + (size_t)a.Di * hwi + o) : 127u;
            }
            if (++c.ki == a.nki) { c.ki = 0; if (++c.zi > c.zhi) open(); }
        };
        unsigned r0[NB], r1[NB];
        int s = 0, ph = 0, it = 0; bool ok = true;
        auto lay = [&](const unsigned *raw) {
            uint32_t wq[5] = {0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu};
#pragma unroll
            for (int j = 0; j < 9; j++) {
                if (BITS == 8) wq[j >> 2] = (wq[j >> 2] & ~(0xffu << (8 * (j & 3)))) | (raw[j] << (8 * (j & 3)));
                else wq[j >> 1] = (wq[j >> 1] & ~(0xffffu << (16 * (j & 1)))) | ((raw[j] | (raw[BITS == 4 ? 9 + j : 0] << 8)) << (16 * (j & 1)));
            }
            if (!__all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, kWaitLimitS))) { if (lane == 0) raise_s(a, abort_flag, 4, it, bar_empty + 8 * s - bar_tma, ph ^ 1); ok = false; return; }
            uint32_t *sfa = (uint32_t *)(stages + (size_t)s * a.stage_bytes + kCodesS);
            /* quad q: word (lane, column) = row 32 * column + lane */
#pragma unroll
            for (int q = 0; q < NQ; q++) sfa[q * 128 + lane * 4 + q4] = wq[q];
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_sf + 8 * s);
            it++; if (++s == R) { s = 0; ph ^= 1; }
        };
        open();
        bool l0 = c.live; fetch(r0);
        bool l1 = c.live; fetch(r1);
        while (ok) {
            if (!l0) break;
            lay(r0); l0 = c.live; fetch(r0);
            if (!ok || !l1) break;
            lay(r1); l1 = c.live; fetch(r1);
        }
    } else {
        /* ---------------- epilogue: one output plane of one tile at a time ---------------- */
        const int q4 = warp & 3, r = q4 * 32 + lane, ry = r >> 3, rx = r & 7;
        const uint32_t tlane = tmem + ((uint32_t)(q4 * 32) << 16);
        for (int sl = 0; sl < NS; sl++)
#pragma unroll
            for (int jc = 0; jc < NCH; jc++) tmem_zero32(tlane + (uint32_t)(sl * NT + jc * 32));
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) for (int sl = 0; sl < NS; sl++) mbar_arrive(bar_acce + 8 * sl);
        if (a.w_dep) pdl_wait();
        float *bw = bias_s + (warp - 6) * NT;    /* a copy a warp: no barrier among the four */
#pragma unroll
        for (int jc = 0; jc < NCH; jc++) bw[jc * 32 + lane] = ld_dep(a.e.bias + ctile * NT + jc * 32 + lane);
        __syncwarp();
        int pcm = 0, pph = 0, pc = 0; bool dead = false;
        while (piece.more() && !dead) {
            const RunS rn = piece.next(a);
            const int ox = (rn.txy % a.tiles_x) * 8 + rx, oy = (rn.txy / a.tiles_x) * 16 + ry;
            const bool row_ok = oy < a.H && ox < a.W;
            for (int z = rn.zb; z < rn.ze; z++, pc++) {
                const int slot = NS - 1 - pcm;
                if (!__all_sync(0xffffffffu, mbar_wait(bar_accf + 8 * slot, (uint32_t)pph, abort_flag, kWaitLimitS))) { if (lane == 0) raise_s(a, abort_flag, 5, pc, bar_accf + 8 * slot - bar_tma, pph); dead = true; break; }
                tc_fence_after();
                uint32_t rr[NCH][32];
                const uint32_t tcol = tlane + (uint32_t)(slot * NT);
#pragma unroll
                for (int jc = 0; jc < NCH; jc++) tmem_ld32(tcol + jc * 32, rr[jc]);
                tmem_ld_wait();
#pragma unroll
                for (int jc = 0; jc < NCH; jc++) tmem_zero32(tcol + jc * 32);      /* every MMA accumulates */
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_acce + 8 * slot);
#pragma unroll
                for (int jc = 0; jc < NCH; jc++) {
                    float v[32];
#pragma unroll
                    for (int k = 0; k < 32; k++) v[k] = __uint_as_float(rr[jc][k]);
                    epi_chunk<true>(a.e, rn.n, z, oy, ox, row_ok, ctile * NCH + jc, v, bw + jc * 32);
                }
                if (++pcm == NS) { pcm = 0; pph ^= 1; }
            }
        }
    }
    /* ---------------- teardown ---------------- */
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && warp == 0 && lane == 0) {
        /* after a give-up: let this thread's own copies in flight land (bounded) before the block's shared memory is released */
        for (int s = 0; s < R; s++) { const long long t0 = clock64(); while (!mbar_try(bar_tma + 8 * s, 0) && !mbar_try(bar_tma + 8 * s, 1) && clock64() - t0 < 20000000ll) { } }
        { const long long t0 = clock64(); while (!mbar_try(bar_w, 0) && clock64() - t0 < 20000000ll) { } }
    }
    if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem, (uint32_t)a.tmem_cols); }
}

/* column tile, image and TMEM of a layer; 0 when its weights do not fit */
struct SGeo { int nt, ncol, w_codes, w_bytes, nslot, tmem_cols, sfa_base, sfa_cols, sfb_base, off_w, off_ring, stage_bytes, ring; };
int s2_geometry(const umx_conv *c, SGeo *g) {
    if (c->kind != UMX_CONV3S2) return 0;
    const int nki = c->nki / 27, nq = c->bits == 8 ? 3 : 5;
    for (int nt = c->cop % 64 ? 32 : 64; nt >= 32; nt -= 32) {
        g->nt = nt; g->ncol = c->cop / nt;
        g->w_codes = nki * 9 * 2 * 3 * nt * 16; g->w_bytes = g->w_codes + nki * nq * 3 * 512;
        g->stage_bytes = kCodesS + nq * 512;                     /* multiples of 128 */
        g->off_w = 2048; g->off_ring = (g->off_w + g->w_bytes + 1023) & ~1023;
        g->ring = (227 * 1024 - g->off_ring) / g->stage_bytes; if (g->ring > kMaxRingS) g->ring = kMaxRingS;
        g->sfa_cols = nq * 4;
        const int fixed = 2 * g->sfa_cols + nki * nq * 12;
        g->tmem_cols = 512;
        g->nslot = (512 - fixed) / nt; if (g->nslot > kMaxSlotsS) g->nslot = kMaxSlotsS;
        g->sfa_base = g->nslot * nt; g->sfb_base = g->sfa_base + 2 * g->sfa_cols;
        if (g->ring >= 3 && g->nslot >= 3) return 1;
    }
    return 0;
}

}   // namespace

/* The weight image: codes [K item][dy dx][k half][row][16 B] with the rows of dz = 0, 2, 1 behind one another, then the B scale bytes in the TMEM scale layout per (K item, tap
   quad) three times: rows of dz = 0 and 2, of dz = 2, of dz = 1 (a block-scaled MMA wants its scales on a 4-column boundary) */
int umx_conv_s2_image(const umx_conv *c, RImageGeo *o) {
    SGeo g;
    if (!s2_geometry(c, &g)) return 0;
    o->nt = g.nt; o->ncol = g.ncol; o->w_bytes = g.w_bytes; o->w_codes = g.w_codes; o->gt = 3; o->goff1 = 1; o->goff2 = 2;
    return 1;
}
int umx_conv_r_cap(void);
static int s2_sms() {
    static int sms_of[16];
    int d = 0; cudaGetDevice(&d); d &= 15;
    if (!sms_of[d]) { int v = 148; cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d); sms_of[d] = v; }
    return sms_of[d];
}
/* Whether this kernel takes the conv: wherever the weights fit, on every grid.  A call of lp_conv_fwd_s2_f8 (weight preparation, and the relayout of an MX-fp8 tensor ahead of the
   general kernel), general kernel and this one, us: MX-fp8 32 -> 64 on 8^3 18.9 and 10.7, on 96^3 55.3 and 19.7, 64 -> 64 on 110 x 100 x 90 136 and 36, 128 -> 256 on 16^3 23.8 and
   15.0, on 48^3 57.4 and 54.9 (the least of 96 shapes); MX-fp4 32 -> 64 on 8^3 17.8 and 9.2, 256 -> 320 on 32^3 54.3 and 41.5.  96^3 moves 43 MB, 7 us at the rate of a copy;
   what is left is the preparation (5 us), the fill and the end of a piece of six planes a block. */
int umx_conv_s2_takes(const umx_conv *c) {
    SGeo g;
    return s2_geometry(c, &g) && g.ncol <= s2_sms();
}
/* x: the MX tensor (split: fp8 codes in the split layout).  0 after a launch, 1 when the tensor cannot be mapped (the caller takes the general kernel), -1 on error. */
int umx_conv_fwd_s2(const umx_conv *c, const void *x, int split, const uint8_t *x_sc, void *enc_v, int N, int Di, int Hi, int Wi, const EpiArgs &e) {
    typedef CUresult (*encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    SGeo g; ConvSArgs a; memset(&a, 0, sizeof a);
    if (!c->wr || !s2_geometry(c, &g)) return 1;
    a.N = N; a.D = e.D; a.H = e.H; a.W = e.W; a.Di = Di; a.Hi = Hi; a.Wi = Wi;
    a.nbi = (c->ci + 31) / 32; a.nki = c->nki / 27; a.nt = g.nt;
    a.tiles_x = (e.W + 7) / 8; a.tiles = a.tiles_x * ((e.H + 15) / 16); a.units = (long long)N * a.tiles * e.D;
    a.ring = g.ring; a.stage_bytes = g.stage_bytes; a.nslot = g.nslot; a.tmem_cols = g.tmem_cols; a.sfa_base = g.sfa_base; a.sfa_cols = g.sfa_cols; a.sfb_base = g.sfb_base;
    a.w_bytes = g.w_bytes; a.w_codes = g.w_codes; a.off_w = g.off_w; a.off_ring = g.off_ring;
    a.w_dep = c->w_src != nullptr; a.x_sc = x_sc; a.wr = c->wr; a.e = e;
    const size_t S = (size_t)Di * Hi * Wi;
    const bool ref8 = c->bits == 8 && !split;
    const int rb = ref8 ? 32 : 16;
    a.c_half = ref8 ? 16 : 0; a.p_blk = c->bits == 8 && split ? 2 : 1; a.p_half = ref8 ? 0 : 1;
    CUtensorMap m[4]; memset(m, 0, sizeof m);
    for (int i = 0; i < 4; i++) {
        /* every second voxel along x and y: a box of 2 k positions delivers k of them */
        const cuuint64_t gd[5] = {(cuuint64_t)rb, (cuuint64_t)Wi, (cuuint64_t)Hi, (cuuint64_t)Di, (cuuint64_t)N * a.nbi * a.p_blk};
        const cuuint64_t gs[4] = {(cuuint64_t)rb, (cuuint64_t)Wi * rb, (cuuint64_t)Wi * Hi * rb, (cuuint64_t)S * rb};
        const cuuint32_t box[5] = {16, (cuuint32_t)(i & 1 ? 18 : 16), (cuuint32_t)(i & 2 ? 34 : 32), 1, 1}, es[5] = {1, 2, 2, 1, 1};
        if (((encode_fn)enc_v)(&m[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, (void *)x, gd, gs, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return 1;
    }
    a.err = umx_errflag(); if (!a.err) return -1;
    int dev = 0; cudaGetDevice(&dev); dev &= 15;
    typedef void (*kernel_fn)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const ConvSArgs);
    static const kernel_fn ks[4] = {conv_s2_k<8, 1>, conv_s2_k<8, 2>, conv_s2_k<4, 1>, conv_s2_k<4, 2>};
    const int variant = (c->bits == 8 ? 0 : 2) | (g.nt == 32 ? 0 : 1);
    static unsigned attr_set[16];                       /* a bit a kernel: the attribute loads it */
    if (!(attr_set[dev] >> variant & 1)) {
        const cudaError_t er = cudaFuncSetAttribute((const void *)ks[variant], cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (er != cudaSuccess) { umx_latch("umx_conv_fwd: shared memory attribute", er); return -1; }
        __atomic_fetch_or(&attr_set[dev], 1u << variant, __ATOMIC_RELAXED);
    }
    long long slots = s2_sms() / g.ncol;
    if (umx_conv_r_cap() && slots > umx_conv_r_cap()) slots = umx_conv_r_cap();
    a.gcol = (int)(a.units < slots ? a.units : slots);
    const dim3 grid((unsigned)(a.gcol * g.ncol));
    const size_t smem = (size_t)g.off_ring + (size_t)g.ring * g.stage_bytes;
    umx_launch(ks[variant], grid, dim3(kThreadsS), smem, m[0], m[1], m[2], m[3], a);
    return 0;
}
