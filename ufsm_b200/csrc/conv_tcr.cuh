/* 3^3 MX conv forward, persistent z-marching kernel for layers whose prepared weights fit in shared memory (up to 64 output
   channels: the 32- and 64-channel levels, which hold most of the network's voxels).

   A block keeps the whole weight image (all taps, all input blocks) in shared memory and the B scale factors in TMEM, and owns a
   contiguous piece of the list of (sample, y-x tile, z) output planes; a piece is one to three runs along z.  Inside a run the
   block marches along z.  Each input plane (one TMA halo load of the codes and one of the scale bytes per input block) is the A
   operand of nine MMAs, one per (dy, dx); the three dz taps that use the same shifted view are stacked along N: B rows are
   (dz, channel), and the accumulators of the three output planes z + 1, z, z - 1 sit in consecutive TMEM slots (slot = ring
   position of the plane, descending), so one MMA of N = 3 x channels updates all three.  When that window wraps around the slot
   ring a stage issues two groups of MMAs.


   What bounds this kernel.  An M = 128, N = 96, K = 32 MMA occupies the tensor pipe for 56 clocks (48 of arithmetic; its 4 KB A tile and
   3 KB B tile exceed what shared memory delivers in 48).  One warp runs the MMA loop with uniform values and one elected lane issues: issued by
   a lone thread, with operands moved to uniform registers one by one, a stage of nine MMAs took 1190 clocks on 128 -> 64 channels, 64^3 (80.7 us
   the conv, 60.0 now).  A commit costs its issuer another 60 clocks, so there is one per stage, and every role's per-stage program is kept short: (1) the
   producer tracks slots and parities incrementally (no division) and hands the MMA warp a record with everything
   precomputed: TMEM addresses, the N field of the instruction descriptor, B descriptor and B scale addresses, the barriers to wait
   for; (2) the MMA warp's stage is three PTX blocks of three MMAs whose operands are a record field plus an immediate; (3)
   accumulators are never "fresh": the epilogue zeroes a slot after reading it, so every MMA accumulates; (4) the A scale factors are
   laid out from a window in shared memory (voxels outside the volume are zero codes with scale byte 0 in it): staged by TMA, or, where TMA does not take the
   scale plane's rows, fetched by the scale warp itself with the bytes outside the volume masked (GATHER), as far ahead of the MMAs as the ring is deep, and copied to TMEM by the MMA warp (copies and MMAs of one thread run in issue order,
   so nothing guards the two buffers; copied by the gathering warps, which had to wait for the MMAs of two stages back, 64 -> 64 on 64^3 took
   26.8 us, 25.8 this way); (5) the MMA warp's single commit per stage lands on the stage's `empty` barrier; a relay passes the completion of
   output planes on to the epilogue's accumulator-full barriers; (6) two blocks share a multiprocessor when the weights are small enough: one
   block's waits are the other's issue time.

   Roles (256 threads): warp 0 producer (records + TMA), warp 1 scale copies and MMA issue (and TMEM), warp 2 scale layout, warp 3 completion
   relay, warps 4-7 epilogue.  All waits are bounded as in conv_mx_k. */
#pragma once
#include "conv_epi.cuh"
#include "tc_ptx.cuh"
#include "gather_win.cuh"
#include <stdlib.h>
#include <string.h>
#include <type_traits>


#define UMX_STR_(x) #x
#define UMX_STR(x) UMX_STR_(x)
/* operand numbers of the PTX blocks below: the five immediates of a tap follow one another */
#define UMX_ADD1(o) UMX_CAT(UMX_N1_, o)
#define UMX_ADD2(o) UMX_CAT(UMX_N2_, o)
#define UMX_ADD3(o) UMX_CAT(UMX_N3_, o)
#define UMX_ADD4(o) UMX_CAT(UMX_N4_, o)
#define UMX_CAT_(a, b) a##b
#define UMX_CAT(a, b) UMX_CAT_(a, b)
#define UMX_N1_8 9
#define UMX_N2_8 10
#define UMX_N3_8 11
#define UMX_N4_8 12
#define UMX_N1_13 14
#define UMX_N2_13 15
#define UMX_N3_13 16
#define UMX_N4_13 17
#define UMX_N1_18 19
#define UMX_N2_18 20
#define UMX_N3_18 21
#define UMX_N4_18 22

struct ConvRArgs {
    int N, D, H, W, nkb, nki, bits, nt;
    int tiles_x, tiles, ncol, gcol;              /* column tiles of nt channels; blocks per column tile */
    long long units;                             /* N x tiles x D output planes of one tile, split evenly over the grid */
    int ring, stage_bytes, offSW, offSFA;
    int ips, item_bytes;                         /* input items of a stage (one plane's; the last stage of a plane may have fewer), bytes of one's codes, window and scales */
    int w_bytes, w_codes, nquad, gt, goff1, goff2, nslot;
    int tmem_cols, sfa_base, sfa_cols, sfb_base; /* TMEM: accumulator slots from 0, two A scale buffers, B scales */
    int off_rec, off_bias, off_stage, off_w, off_ring;   /* off_stage (with statistics or a plane-major output): 2 KB per epilogue warp (and 32-channel chunk), the fp16 rows on their way to wide stores */
    int fast_h16, fast_pm16;                     /* output is the fp16 blocked tensor of a plain conv, or plane-major fp16: the short epilogues */
    /* InstanceNorm statistics taken in that epilogue (coef != NULL): fp64 sums of the stored fp16 values and of their squares, written once per
       sample and block into part [n][gcol][cop][2]; the last block of a column tile to finish adds the blocks' entries in block order and
       turns them into coefficients (a, b) per (sample, channel) */
    double *part; float *coef; const float *gamma, *beta; float eps; int cop, off_red;
    const uint8_t *wr, *x_sc;
    int gather, w_dep;                           /* see GATHER; the weights and the bias were written by a kernel just ahead in the stream */
    EpiArgs e;
    int *err;
};
/* The instances come in five forms, each in a source file of its own with a table of six: MX-fp8 and MX-fp4 with 32- and 64-channel column tiles, MX-fp8 in the reference's layout with
   either.  A process loads a source file's kernels as a whole, unpacked, when it first launches one of them, and should not pay for forms it does not use: with all (24 then) in one
   the first 3^3 conv of a process took 10.6 ms and the first forward of the network on 128^3 17 ms; 1.5 (and 1.3 where it meets a second form) and 8.9 this way. */
typedef void (*conv_r_fn)(const CUtensorMap, const CUtensorMap, const ConvRArgs);
extern const conv_r_fn umx_conv_r_one[6], umx_conv_r_stats[6], umx_conv_r_gather[6], umx_conv_r_ends[6], umx_conv_r_multi[6];
#define UMX_R_FORM(ST, GA, MU) {conv_mxr_k<8, 1, ST, GA, MU>, conv_mxr_k<8, 2, ST, GA, MU>, conv_mxr_k<4, 1, ST, GA, MU>, conv_mxr_k<4, 2, ST, GA, MU>, conv_mxr_k<8, 1, ST, GA, MU, true>, conv_mxr_k<8, 2, ST, GA, MU, true>}

namespace {

constexpr int kThreadsR = 256;
constexpr int kMaxSlots = 12;
constexpr long long kWaitLimitR = 4000000000ll;

/* what the MMA warp does for one stage; written by the producer */
struct StageRec {
    uint32_t d1, idn1, bb1, sfb1;      /* first group: TMEM accumulator address, instruction descriptor with N, B descriptor low word of tap 0, B scale address */
    uint32_t d2, idn2, bb2, sfb2;      /* second group when the window wraps (idn2 = 0: none) */
    uint32_t wait0, wait1;             /* accumulator-empty barriers to pass first: address | parity << 31 (0: none) */
    uint32_t items, pad0;              /* input items of the stage */
    uint32_t last, pad[3];
};
static_assert(sizeof(StageRec) == 64, "stage record is 64 bytes");

/* a wait gave up (its own limit, or another role's abort flag): the first to get here names the block; every role of that block then leaves
   where it stood (stage, barrier, parity), which the host prints */
__device__ __forceinline__ void raise_r(const ConvRArgs &a, volatile int *abort_flag, int code, int stage, uint32_t bar_off = 0, uint32_t parity = 0) {
    if (atomicCAS(a.err, 0, code) == 0) { a.err[1] = (int)blockIdx.x; a.err[2] = stage; a.err[3] = (int)threadIdx.x; __threadfence(); }
    if (((volatile int *)a.err)[1] == (int)blockIdx.x && code < 8) { int *d = a.err + 16 + 4 * code; d[0] = stage; d[1] = (int)bar_off; d[2] = (int)parity; d[3] = 1; }
    *abort_flag = 1;
    __threadfence_block();
}
/* Three of the nine (dy, dx) MMAs of a group in one PTX block: tap j reads the A view a_lo + (j / 3) * 10 + j % 3 and the B image
   b_lo + j * BSTEP; the scale sets come in quads of four (fp8) or two (fp4) taps.  Everything that depends on the tap is an immediate, so
   between two MMAs the warp runs a handful of independent uniform instructions that the assembler is free to hoist; `lead` is 1 in the lane that issues. */
template <int BITS, int BSTEP, int SFBQ, int J0>
__device__ __forceinline__ void mma3(uint32_t d, uint32_t idn, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t sfa, uint32_t sfb, uint32_t lead) {
    constexpr int IPQ = BITS == 8 ? 4 : 2;
#define UMX_TAP(j) "n"(((j) / 3) * 10 + (j) % 3), "n"((j) * BSTEP), "n"(((((j) % IPQ) * (4 / IPQ)) << 4) | ((((j) % IPQ) * (4 / IPQ)) << 29)), "n"(4 * ((j) / IPQ)), "n"(((j) / IPQ) * SFBQ)
#define UMX_MMA_TEXT(KIND, o)                                                                                        \
    "add.u32 ta, %2, %" #o ";\n\tmov.b64 da, {ta, %3};\n\t"                                                         \
    "add.u32 tb, %4, %" UMX_STR(UMX_ADD1(o)) ";\n\tmov.b64 db, {tb, %5};\n\t"                                      \
    "or.b32 ti, %1, %" UMX_STR(UMX_ADD2(o)) ";\n\t"                                                                   \
    "add.u32 sa, %6, %" UMX_STR(UMX_ADD3(o)) ";\n\tadd.u32 sb, %7, %" UMX_STR(UMX_ADD4(o)) ";\n\t"                  \
    "@pl tcgen05.mma.cta_group::1.kind::" KIND " [%0], da, db, ti, [sa], [sb], p;\n\t"
    if constexpr (BITS == 8) {
        asm volatile("{\n\t.reg .pred p, pl;\n\t.reg .b32 ta, tb, ti, sa, sb;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %1, 0;\n\tsetp.ne.b32 pl, %23, 0;\n\t"
                     UMX_MMA_TEXT("mxf8f6f4.block_scale", 8) UMX_MMA_TEXT("mxf8f6f4.block_scale", 13) UMX_MMA_TEXT("mxf8f6f4.block_scale", 18) "}"
                     ::"r"(d), "r"(idn), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(sfa), "r"(sfb), UMX_TAP(J0), UMX_TAP(J0 + 1), UMX_TAP(J0 + 2), "r"(lead) : "memory");
    } else {
        asm volatile("{\n\t.reg .pred p, pl;\n\t.reg .b32 ta, tb, ti, sa, sb;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %1, 0;\n\tsetp.ne.b32 pl, %23, 0;\n\t"
                     UMX_MMA_TEXT("mxf4.block_scale.scale_vec::2X", 8) UMX_MMA_TEXT("mxf4.block_scale.scale_vec::2X", 13) UMX_MMA_TEXT("mxf4.block_scale.scale_vec::2X", 18) "}"
                     ::"r"(d), "r"(idn), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(sfa), "r"(sfb), UMX_TAP(J0), UMX_TAP(J0 + 1), UMX_TAP(J0 + 2), "r"(lead) : "memory");
    }
#undef UMX_TAP
#undef UMX_MMA_TEXT
}
/* the nine (dy, dx) MMAs of one group into the accumulator window at d (idn: the instruction descriptor with the window's N) */
template <int BITS, int NT> __device__ __forceinline__ void issue_group(uint32_t d, uint32_t idn, uint32_t bb, uint32_t sfb, uint32_t a_lo, uint32_t a_hi, uint32_t b_hi, uint32_t sfa_t, uint32_t lead) {
    constexpr int BSTEP = 2 * 3 * NT, SFBQ = 4 * ((3 * NT + 127) / 128 + (2 * NT + 127) / 128 + (NT + 127) / 128);
    mma3<BITS, BSTEP, SFBQ, 0>(d, idn, a_lo, a_hi, bb, b_hi, sfa_t, sfb, lead);
    mma3<BITS, BSTEP, SFBQ, 3>(d, idn, a_lo, a_hi, bb, b_hi, sfa_t, sfb, lead);
    mma3<BITS, BSTEP, SFBQ, 6>(d, idn, a_lo, a_hi, bb, b_hi, sfa_t, sfb, lead);
}
/* the block's piece of the plane list, u in [u0, u1) with u = (sample * tiles + tile) * D + z, cut into runs along z */
struct Piece { long long u, u1; };
__device__ __forceinline__ Piece piece_of_block(const ConvRArgs &a) {
    const long long b = (long long)(blockIdx.x % a.gcol);      /* blocks [k gcol, (k + 1) gcol) share column tile k and split the plane list */
    Piece p; p.u = a.units * b / (long long)a.gcol; p.u1 = a.units * (b + 1) / (long long)a.gcol; return p;
}
struct Run { int n, txy, zb, ze; };
__device__ __forceinline__ Run next_run(const ConvRArgs &a, Piece &p) {
    const long long col = p.u / a.D; Run r;
    r.zb = (int)(p.u - col * a.D); r.ze = (int)min((long long)a.D, (long long)r.zb + (p.u1 - p.u));
    r.n = (int)(col / a.tiles); r.txy = (int)(col - (long long)r.n * a.tiles);
    p.u += r.ze - r.zb;
    return r;
}

/* ---- InstanceNorm sums in the epilogue.  They are taken in fp64 where the warp re-reads its staged fp16 rows for the coalesced store:
   there a lane holds eight channels of the four voxels of one x, and it keeps one (sum, sum of squares) pair per channel for the whole
   sample.  A stored fp16 value and its square are exact in fp64 and so are their sums over a sample of any realistic size, so neither
   the order of the planes nor their partition over blocks changes a bit, and the coefficients equal those of the separate fp64 pass
   (in_part_k).  Per sample and block the eight lanes that hold the same channels are added with shuffles, then the four warps, then (by
   the block that finishes last, in block order) the blocks. ---- */
/* the sum over the eight lanes x = 0..7 that hold this lane's channels (partners p4, p2, p1: the lanes at x ^ 4, x ^ 2, x ^ 1) */
__device__ __forceinline__ double lanes8_sum(double v, int p4, int p2, int p1) {
    v += __shfl_sync(0xffffffffu, v, p4);
    v += __shfl_sync(0xffffffffu, v, p2);
    return v + __shfl_sync(0xffffffffu, v, p1);
}

__device__ unsigned g_conv_tickets[64];      /* one per column tile; the block that draws the last ticket finalises and resets it */

/* NCH: 32-channel chunks of the column tile (1: two blocks per multiprocessor and at most 128 registers; 2: one block, more registers);
   STATS: the epilogue also takes the InstanceNorm sums; GATHER: the scale warp fetches its window of scale bytes itself, for scale planes whose rows TMA does not
   take (W not a multiple of 16), 2: of a tensor that ends inside a word (gather_win.cuh); MULTI: a stage holds up to a.ips input items of its plane (see r_plan), else one; REF:
   MX-fp8 codes in the reference's layout (32-byte rows): a half of a row a load, the halves 2944 bytes apart in a stage (as a branch on an argument it cost the split layout 1.3 % on
   32 -> 32, 64^3) */
template <int BITS, int NCH, bool STATS, int GATHER, bool MULTI, bool REF = false>
__global__ void __launch_bounds__(kThreadsR, NCH == 1 ? 2 : 1) conv_mxr_k(const __grid_constant__ CUtensorMap map0, const __grid_constant__ CUtensorMap maps, const ConvRArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint64_t *bars = (uint64_t *)smem_raw;
    uint32_t *tmem_slot = (uint32_t *)(smem_raw + 768);
    volatile int *abort_flag = (volatile int *)(smem_raw + 772);
    StageRec *recs = (StageRec *)(smem_raw + a.off_rec);
    float *bias_s = (float *)(smem_raw + a.off_bias);
    uint8_t *wsm = smem_raw + a.off_w, *stages = smem_raw + a.off_ring;
    const int warp = (int)uni(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int R = a.ring, NS = a.nslot, ips = MULTI ? a.ips : 1;
    /* barriers: tma[R] (codes + scale window landed), sf[R] (A scales laid out), empty[R], accumulator full / empty per slot, weights */
    const uint32_t bar_tma = smem_u32(bars), bar_sf = bar_tma + 8 * R, bar_empty = bar_tma + 16 * R, bar_accf = bar_tma + 24 * R, bar_acce = bar_accf + 8 * kMaxSlots, bar_w = bar_acce + 8 * kMaxSlots, bar_red = bar_w + 8;
    constexpr int NQ = BITS == 8 ? 3 : 5;                  /* A scale quads per stage */
    constexpr int GB = BITS == 8 ? 54 : 108, GN = (GB + 31) / 32;          /* words of the gathered scale window, of a lane */
    auto win_at = [](int i) { return i / 54 * 576 + (i % 54) / 3 * 32 + i % 3 * 4; };      /* where word i lies in the stage's window */
    constexpr uint32_t TX = 5760u + (GATHER ? 0u : BITS == 8 ? 576u : 1152u);

    if (threadIdx.x == 0) {
        for (int i = 0; i < R; i++) { mbar_init(bar_tma + 8 * i, 1); mbar_init(bar_sf + 8 * i, 1); mbar_init(bar_empty + 8 * i, 1); }
        for (int i = 0; i < kMaxSlots; i++) { mbar_init(bar_accf + 8 * i, 1); mbar_init(bar_acce + 8 * i, 4); }
        mbar_init(bar_w, 1); mbar_init(bar_red, 128);
        *abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    const int ctile = (int)blockIdx.x / a.gcol;
    if (!a.w_dep && (int)threadIdx.x < a.nt) bias_s[threadIdx.x] = a.e.bias[ctile * a.nt + threadIdx.x];
    auto load_weights = [&]() {
        mbar_expect_tx(bar_w, (uint32_t)a.w_bytes);
        for (int o = 0; o < a.w_bytes; o += 32768) bulk_g2s(smem_u32(wsm + o), a.wr + (size_t)ctile * a.w_bytes + o, (uint32_t)min(32768, a.w_bytes - o), bar_w);
    };
    if (!a.w_dep && threadIdx.x == 0) load_weights();      /* the weight image of a prepared layer is a constant: it may load while the previous kernel of the stream is still running */
    if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), (uint32_t)a.tmem_cols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();                               /* the next kernel cannot take this block's tensor memory any more */
    const uint32_t tmem = uni(*tmem_slot);
    Piece piece = piece_of_block(a);

    if (warp == 0) {
        /* ---------------- producer: stage records and TMA ---------------- */
        {
            const uint32_t lead = elect_one();
            if (lead) { tma_prefetch_desc(&map0); tma_prefetch_desc(&maps); }
            pdl_wait();      /* a prepared layer: the only role that reads what an earlier kernel wrote (GATHER: the scale warp reads the scale plane, behind a wait of its own); every
                                other role's data comes through this warp's loads, so the weight load, the B scale copies and the zeroing of the accumulators overlap the previous
                                kernel.  Weights that a kernel just ahead wrote (w_dep) load behind this wait, and the epilogue reads their bias behind its own */
            if (a.w_dep && lead) load_weights();
            const uint32_t nt = (uint32_t)a.nt, bstep9 = 9u * 2u * 3u * nt;            /* B descriptor step of one input block: nine taps of two halves of 3 nt rows */
            const uint32_t b_lo0 = desc_lo(smem_u32(wsm), 3u * nt * 16u);
            const uint32_t idesc_b = (BITS == 8 ? idesc_mxf8(0, 0, 0) : idesc_mxf4(0, 0, 0)), ntn = (nt >> 3) << 17;
            const uint32_t sfb_t0 = tmem + (uint32_t)a.sfb_base, sfb_per_ki = (uint32_t)(a.nquad * a.gt * 4);
            int s = 0, ph = 0, it = 0; bool ok = true;
            int pos = NS - 1; uint32_t wp = 1u;           /* ring position and wrap parity of the newest plane started so far */
            while (piece.u < piece.u1 && ok) {
                const Run rn = next_run(a, piece);
                const bool last_run = piece.u >= piece.u1;
                const int x0 = (rn.txy % a.tiles_x) * 8, y0 = (rn.txy / a.tiles_x) * 16;
                const int zb = rn.zb, ze = rn.ze, zlo = max(0, zb - 1), zhi = min(a.D - 1, ze);
                const int xa = ((x0 - 1) >> 4) << 4;             /* 16-aligned start of the 32-byte scale window (x0 = 0: -16, read as zeros) */
                const int cx = (x0 - 1) * 16, cy = y0 - 1;
                const int pl0 = BITS == 8 ? rn.n * a.nkb * 2 : rn.n * a.nkb, pls = rn.n * a.nkb;
                for (int zi = zlo; zi <= zhi && ok; zi++) {
                    /* output planes fed by input plane zi: z = zi + 1 - dz, newest first */
                    const int newest = min(zi + 1, ze - 1), oldest = max(zi - 1, zb), cnt = newest - oldest + 1, dzf = zi + 1 - newest;
                    const int nfresh = zi == zlo ? cnt : (newest == zi + 1 ? 1 : 0);
                    uint32_t w0 = 0, w1 = 0;
                    for (int f = 0; f < nfresh; f++) {
                        if (++pos == NS) { pos = 0; wp ^= 1u; }
                        const uint32_t wf = (bar_acce + 8u * (uint32_t)(NS - 1 - pos)) | (wp << 31);
                        if (f == 0) w0 = wf; else w1 = wf;
                    }
                    const int slot = NS - 1 - pos, n1 = min(cnt, NS - slot), n2 = cnt - n1;
                    const uint32_t g1 = (uint32_t)(dzf == 0 ? 0 : dzf == 1 ? a.goff1 : a.goff2), g2 = (uint32_t)(dzf + n1 == 1 ? a.goff1 : a.goff2);
                    for (int ki = 0; ki < a.nki; ki += ips) {
                        if (!__all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, kWaitLimitR))) { if (lane == 0) raise_r(a, abort_flag, 1, it, bar_empty + 8 * s - bar_tma, ph ^ 1); ok = false; break; }
                        const int nit = MULTI ? min(ips, a.nki - ki) : 1;
                        const bool kl = ki + nit == a.nki;
                        const uint32_t bk = b_lo0 + (uint32_t)ki * bstep9, sk = sfb_t0 + (uint32_t)ki * sfb_per_ki;
                        if (lead) {
                            uint4 *r = (uint4 *)(recs + s);
                            r[0] = make_uint4(tmem + (uint32_t)slot * nt, idesc_b | (uint32_t)n1 * ntn, bk + (uint32_t)dzf * nt, sk + g1);
                            r[1] = make_uint4(tmem, n2 ? (idesc_b | (uint32_t)n2 * ntn) : 0u, bk + (uint32_t)(dzf + n1) * nt, sk + g2);
                            r[2] = make_uint4(ki == 0 ? w0 : 0u, ki == 0 ? w1 : 0u, (uint32_t)nit, 0u);
                            r[3] = make_uint4((last_run && zi == zhi && kl) ? 1u : 0u, 0u, 0u, 0u);
                            mbar_expect_tx(bar_tma + 8 * s, TX * (uint32_t)nit);
                        }
                        uint32_t sb = smem_u32(stages + (size_t)s * a.stage_bytes); const uint32_t bar = bar_tma + 8 * s;
                        /* codes: two 16-byte-wide planes (fp8: the halves of block ki; fp4: blocks 2 ki and 2 ki + 1), 18 rows of 10 voxels;
                           scale bytes: 18 rows of a 32-byte window per block */
                        for (int k = ki; k < ki + (MULTI ? nit : 1); k++, sb += (uint32_t)a.item_bytes) {
                            if (REF) { tma_load_5d(sb, &map0, bar, 0, x0 - 1, cy, zi, pls + k, lead); tma_load_5d(sb + 2944, &map0, bar, 16, x0 - 1, cy, zi, pls + k, lead); }
                            else tma_load_4d(sb, &map0, bar, cx, cy, zi, pl0 + 2 * k, lead);
                            if (!GATHER && BITS == 8) tma_load_4d(sb + a.offSW, &maps, bar, xa, cy, zi, pls + k, lead);
                            if (!GATHER && BITS == 4) tma_load_5d(sb + a.offSW, &maps, bar, xa, cy, zi, 2 * k, rn.n, lead);
                        }
                        it++; if (++s == R) { s = 0; ph ^= 1; }
                    }
                }
            }
        }
    } else if (warp == 1) {
        /* ---------------- MMA issue: one warp follows the records; a stage is straight-line code.  The whole warp runs the loop and one lane issues:
           a record passes through a shuffle, so that the operands of an MMA are known to be the same in every lane and its address arithmetic stays in
           the uniform registers that the instruction reads, instead of being moved there operand by operand ---------------- */
        {
            const uint32_t lead = elect_one();
            bool ok = mbar_wait(bar_w, 0, abort_flag, kWaitLimitR);
            if (!ok && lane == 0) raise_r(a, abort_flag, 6, 0);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            const uint32_t wbase = smem_u32(wsm);
            const uint32_t a_hi = desc_hi(160), b_hi = desc_hi(128);
            const uint32_t sf_hi = desc_hi(128);                     /* scale blocks: 32 rows of 16 bytes, 8-row groups 128 bytes apart */
            if (ok) {
                /* the B scale factors of every (input block, tap quad, image, 128-row group): copied to TMEM once */
                const int nsf = a.nki * a.nquad * a.gt;
                for (int i = 0; i < nsf; i++) utccp_32x128b(tmem + a.sfb_base + i * 4, desc_make(desc_lo(wbase + a.w_codes + i * 512, 0), sf_hi), lead);
            }
            const uint32_t a_lo0 = desc_lo(smem_u32(stages), REF ? 2944u : 2880u), a_step = (uint32_t)a.stage_bytes >> 4, sfa_off = (uint32_t)a.offSFA >> 4;
            const uint32_t sfa_t0 = tmem + (uint32_t)a.sfa_base, sfa_cols = (uint32_t)a.sfa_cols;
            const uint32_t i_step = (uint32_t)a.item_bytes >> 4, bstep9 = 9u * 2u * 3u * 32u * NCH, sfb_step = (uint32_t)(a.nquad * a.gt * 4);
            uint32_t item = 0;
            int s = 0, ph = 0, it = 0;
            while (ok) {
                /* the stage's A scales are laid out; the scale warp passed the stage's load barrier before, so the codes have landed too */
                if (!__all_sync(0xffffffffu, mbar_wait(bar_sf + 8 * s, ph, abort_flag, kWaitLimitR))) { if (lane == 0) raise_r(a, abort_flag, 3, it, bar_sf + 8 * s - bar_tma, ph); break; }
                /* the whole record goes to registers before anything is committed: committing `empty` hands the stage, record included, back to the producer */
                const uint4 *r = (const uint4 *)(recs + s);
                const uint4 g1 = uni(r[0]), g2 = uni(r[1]), wc = uni(r[2]); const uint32_t last = uni(r[3].x);
                if (wc.x) {   /* a plane that starts here: its slot must have been read out and zeroed by the epilogue */
                    bool got = mbar_wait(wc.x & 0x7fffffffu, wc.x >> 31, abort_flag, kWaitLimitR);
                    if (got && wc.y) got = mbar_wait(wc.y & 0x7fffffffu, wc.y >> 31, abort_flag, kWaitLimitR);
                    if (!__all_sync(0xffffffffu, got)) { if (lane == 0) raise_r(a, abort_flag, 7, it, (wc.x & 0x7fffffffu) - bar_tma, wc.x >> 31); break; }
                }
                tc_fence_after();
                /* copies and MMAs of one thread run in issue order, so a buffer is overwritten after the MMAs that read it two items ago */
                if (!MULTI) {
                    const uint32_t a_lo = a_lo0 + (uint32_t)s * a_step, sfa_t = sfa_t0 + ((uint32_t)it & 1u) * sfa_cols;
#pragma unroll
                    for (int q = 0; q < NQ; q++) utccp_32x128b(sfa_t + 4 * q, desc_make((a_lo & 0xffffu) + sfa_off + 32u * q, sf_hi), lead);
                    issue_group<BITS, 32 * NCH>(g1.x, g1.y, g1.z, g1.w, a_lo, a_hi, b_hi, sfa_t, lead);
                    if (g2.y) issue_group<BITS, 32 * NCH>(g2.x, g2.y, g2.z, g2.w, a_lo, a_hi, b_hi, sfa_t, lead);
                } else {
                    uint32_t a_lo = a_lo0 + (uint32_t)s * a_step, bb1 = g1.z, sf1 = g1.w, bb2 = g2.z, sf2 = g2.w;
                    for (uint32_t i = 0; i < wc.z; i++) {
                        const uint32_t sfa_t = sfa_t0 + (item & 1u) * sfa_cols;
                        item++;
#pragma unroll
                        for (int q = 0; q < NQ; q++) utccp_32x128b(sfa_t + 4 * q, desc_make((a_lo & 0xffffu) + sfa_off + 32u * q, sf_hi), lead);
                        issue_group<BITS, 32 * NCH>(g1.x, g1.y, bb1, sf1, a_lo, a_hi, b_hi, sfa_t, lead);
                        if (g2.y) issue_group<BITS, 32 * NCH>(g2.x, g2.y, bb2, sf2, a_lo, a_hi, b_hi, sfa_t, lead);
                        a_lo += i_step; bb1 += bstep9; bb2 += bstep9; sf1 += sfb_step; sf2 += sfb_step;
                    }
                }
                /* the one commit of a stage: "stage s has been consumed".  The producer reuses the ring slot on it, and the relay passes the news that output
                   planes are complete on to the epilogue */
                umma_commit(bar_empty + 8 * s, lead);
                it++; if (++s == R) { s = 0; ph ^= 1; }
                if (last) break;
            }
        }
    } else if (warp == 2) {
        /* ---------------- A scales ----------------
           The TMA left 18 rows of a 32-byte window of scale bytes (two windows for fp4); row r of the tile needs, for tap (dy, dx), the
           byte at window row r / 8 + dy, column r % 8 + dx + (x0 - 1 - xa).  Four rows per lane (one per TMEM column of the quad); the three
           dx of a row are neighbours, so two words and a funnel shift fetch them.  The warp lays the nine shifted scale sets out in shared
           memory in the tcgen05.cp layout, as far ahead of the MMAs as the ring is deep. */
        int it = 0, s = 0, ph = 0; bool ok = true;
        /* one stage: window -> scale sets; off: this lane's first byte of the window, gw: the window's bytes (GATHER) */
        auto lay = [&](int off, int nit, const unsigned *gw) {
            if (!__all_sync(0xffffffffu, mbar_wait(bar_tma + 8 * s, ph, abort_flag, kWaitLimitR))) { if (lane == 0) raise_r(a, abort_flag, 4, it, 8 * s, ph); ok = false; return; }
            uint8_t *stg = stages + (size_t)s * a.stage_bytes;
            for (int i = 0; i < (MULTI ? nit : 1); i++, stg += a.item_bytes) {
            if (GATHER) {
#pragma unroll
                for (int k = 0; k < GN; k++) {
                    const int i = 32 * k + lane;
                    if (i < GB) *(unsigned *)(stg + a.offSW + win_at(i)) = __funnelshift_r(gw[4 * k], gw[4 * k + 1], gw[4 * k + 2]) & gw[4 * k + 3];
                }
                __syncwarp();
            }
            const int sh = (off & 3) * 8;
            const uint32_t *sw = (const uint32_t *)(stg + a.offSW + (off & ~3));
            uint32_t *sfa = (uint32_t *)(stg + a.offSFA);
            uint32_t wq[4][5];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                uint32_t t[3], u[3];          /* bytes 0..2: the scales of dx = 0, 1, 2 */
#pragma unroll
                for (int dy = 0; dy < 3; dy++) {
                    const uint32_t *p = sw + q * 32 + dy * 8;
                    t[dy] = __funnelshift_r(p[0], p[1], sh);
                    if (BITS == 4) u[dy] = __funnelshift_r(p[144], p[145], sh);
                }
                if (BITS == 8) {              /* taps 0-3, 4-7, 8 */
                    wq[q][0] = __byte_perm(t[0], t[1], 0x4210); wq[q][1] = __byte_perm(t[1], t[2], 0x5421); wq[q][2] = (t[2] >> 16) & 0xffu;
                } else {                      /* pairs (block 2 ki, block 2 ki + 1) of taps 0 1, 2 3, 4 5, 6 7, 8 */
                    wq[q][0] = __byte_perm(t[0], u[0], 0x5140); wq[q][1] = __byte_perm(__byte_perm(t[0], u[0], 0x0062), __byte_perm(t[1], u[1], 0x0040), 0x5410);
                    wq[q][2] = __byte_perm(t[1], u[1], 0x6251); wq[q][3] = __byte_perm(t[2], u[2], 0x5140); wq[q][4] = __byte_perm(t[2], u[2], 0x0062) & 0xffffu;
                }
            }
            /* quad qd: word (lane, column) = row 32 * column + lane; a lane's four columns are 16 contiguous bytes: one store */
#pragma unroll
            for (int qd = 0; qd < NQ; qd++) *(uint4 *)(sfa + qd * 128 + lane * 4) = make_uint4(wq[0][qd], wq[1][qd], wq[2][qd], wq[3][qd]);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_sf + 8 * s);
            it++; if (++s == R) { s = 0; ph ^= 1; }
        };
        const int off0 = (lane >> 3) * 32 + (lane & 7);
        if (!GATHER) {
            while (piece.u < piece.u1 && ok) {
                const Run rn = next_run(a, piece);
                const int x0 = (rn.txy % a.tiles_x) * 8;
                const int zlo = max(0, rn.zb - 1), zhi = min(a.D - 1, rn.ze);
                const int off = off0 + (x0 - 1) - (((x0 - 1) >> 4) << 4);
                for (int zi = zlo; zi <= zhi && ok; zi++)
                    for (int ki = 0; ki < a.nki && ok; ki += ips) lay(off, MULTI ? min(ips, a.nki - ki) : 1, nullptr);
            }
        } else {
            /* The window (gather_win.cuh): every word is put together from the two aligned words it lies in, and bytes outside the volume are cleared (scale byte 0, under zero
               codes).  A lane has GN words and asks for them two stages ahead of their use.  Byte by byte
               this warp was the slowest role in the 64-channel MX-fp4 tiles. */
            pdl_wait();
            Run rn; int zi = 1, zhi = 0, ki = 0; bool live = false; const uint8_t *base = nullptr;
            unsigned keep[GN];                   /* the bytes of word k that are wanted */
            int offs[GN];
            const uint8_t *end = a.x_sc + (size_t)a.N * a.nkb * a.D * a.H * a.W;
            int tail_z = 0;
            const size_t S = (size_t)a.D * a.H * a.W;
#pragma unroll
            for (int k = 0; k < GN; k++) { const int i = (32 * k + lane) % 54; offs[k] = (i / 3) * a.W + i % 3 * 4; }
            auto open = [&]() {
                live = piece.u < piece.u1;
                if (!live) return;
                rn = next_run(a, piece);
                zi = max(0, rn.zb - 1); zhi = min(a.D - 1, rn.ze); ki = 0;
                const int x0 = (rn.txy % a.tiles_x) * 8 - 1, y0 = (rn.txy / a.tiles_x) * 16 - 1;
                base = a.x_sc + (ptrdiff_t)y0 * a.W + x0;
                if (GATHER == 2) tail_z = gather_tail(rn.n, a.N, a.D, a.H, a.W);
#pragma unroll
                for (int k = 0; k < GN; k++) keep[k] = 32 * k + lane < GB ? gather_keep((32 * k + lane) % 54, x0, y0, a.W, a.H) : 0u;
            };
            auto fetch = [&](unsigned *g) {
                if (!live) return;
                const uint8_t *p = base + ((size_t)rn.n * a.nkb + (BITS == 8 ? ki : 2 * ki)) * S + (size_t)zi * a.H * a.W;
                const bool two = BITS == 4 && 2 * ki + 1 < a.nkb;
                /* fp4: words of the item's second block, which may not be there (zero weights); put together in lay, when they have come */
                auto words = [&](auto tail) {
#pragma unroll
                    for (int k = 0; k < GN; k++) {
                        const bool second = 32 * k + lane >= 54;
                        gather_word<decltype(tail)::value>(p + (second ? S : 0) + offs[k], !second || two ? keep[k] : 0u, end, g + 4 * k, [](auto *q) { return ld_dep(q); });
                    }
                };
                if (GATHER == 1 || zi < tail_z) words(std::false_type()); else words(std::true_type());
                if (++ki == a.nki) { ki = 0; if (++zi > zhi) open(); }
            };
            unsigned g0[4 * GN], g1[4 * GN];
            open();
            bool l0 = live; fetch(g0);
            bool l1 = live; fetch(g1);
            while (ok && l0) {
                lay(off0, 1, g0); l0 = live; fetch(g0);
                if (!ok || !l1) break;
                lay(off0, 1, g1); l1 = live; fetch(g1);
            }
        }
    } else if (warp == 3) {
        /* ---------------- completion relay ----------------
           The MMA warp commits once per stage, on the stage's `empty` barrier.  This thread passes every one of them in order, knows which
           output planes a stage completes (the plane below the input plane, and the volume's last plane with it) and arrives on their
           accumulator-full barriers, which the epilogue waits on. */
        if (lane == 0) {
            int it = 0, s = 0, ph = 0, fs = NS - 1; bool ok = true;      /* fs: accumulator slot of the oldest plane not yet complete */
            while (piece.u < piece.u1 && ok) {
                const Run rn = next_run(a, piece);
                const int zlo = max(0, rn.zb - 1), zhi = min(a.D - 1, rn.ze);
                for (int zi = zlo; zi <= zhi && ok; zi++) {
                    for (int ki = 0; ki < a.nki; ki += ips) {
                        if (!mbar_wait(bar_empty + 8 * s, ph, abort_flag, kWaitLimitR)) { raise_r(a, abort_flag, 2, it, bar_empty + 8 * s - bar_tma, ph); ok = false; break; }
                        it++; if (++s == R) { s = 0; ph ^= 1; }
                    }
                    const int nc = (zi - 1 >= rn.zb ? 1 : 0) + ((zi == a.D - 1 && rn.ze == a.D) ? 1 : 0);
                    for (int k = 0; k < nc && ok; k++) { mbar_arrive(bar_accf + 8 * fs); fs = fs == 0 ? NS - 1 : fs - 1; }
                }
            }
        }
    } else {
        /* ---------------- epilogue: one output plane of one tile at a time ---------------- */
        const int q4 = warp & 3, r = q4 * 32 + lane, ry = r >> 3, rx = r & 7;
        constexpr int nchunk = NCH;
        const uint32_t tlane = tmem + ((uint32_t)(q4 * 32) << 16);
        /* every slot starts zeroed and released */
        for (int sl = 0; sl < NS; sl++) {
            for (int jc = 0; jc < nchunk; jc++) tmem_zero32(tlane + (uint32_t)(sl * a.nt + jc * 32));
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) for (int sl = 0; sl < NS; sl++) mbar_arrive(bar_acce + 8 * sl);     /* one arrival per warp: arrivals on one barrier serialise */
        if (a.w_dep) {                                          /* every warp writes the same values */
            pdl_wait();
#pragma unroll
            for (int jc = 0; jc < NCH; jc++) bias_s[jc * 32 + lane] = ld_dep(a.e.bias + ctile * a.nt + jc * 32 + lane);
            __syncwarp();
        }
        int pcm = 0, pph = 0, pc = 0; bool dead = false;        /* pcm = plane count mod slots, pph = its wrap parity */
        const size_t S = (size_t)a.D * a.H * a.W;
        constexpr bool stats = STATS;
        const int et = (int)threadIdx.x - 128, bcol = (int)blockIdx.x % a.gcol;
        const int cl = (lane & 3) ^ ((lane >> 3) & 3);          /* the 16-byte chunk of a staged row this lane finds when it re-reads the rows for the coalesced store (see below) */
        /* statistics: x of this lane's voxels, the lanes that hold the same channels at x ^ 4, x ^ 2, x ^ 1, and the channel (of a 32-channel
           chunk) whose unit sum this lane ends up with */
        const int sx = lane >> 2;
        const int sp4 = 4 * (sx ^ 4) + (cl ^ (((sx ^ 4) >> 1) & 3)), sp2 = 4 * (sx ^ 2) + (cl ^ (((sx ^ 2) >> 1) & 3)), sp1 = 4 * (sx ^ 1) + (cl ^ (((sx ^ 1) >> 1) & 3));
        const int sch = 8 * cl + sx;                            /* the channel (of a 32-channel chunk) whose lane-group sum this lane writes out */
        /* this lane's channels 8 cl .. 8 cl + 7 of each chunk: sums and sums of squares of the sample in progress */
        double dsum[STATS ? NCH : 1][8], dsq[STATS ? NCH : 1][8];
        if (STATS) {
#pragma unroll
            for (int k = 0; k < NCH; k++)
#pragma unroll
                for (int t = 0; t < 8; t++) { dsum[k][t] = 0.0; dsq[k][t] = 0.0; }
        }
        double *red = (double *)(smem_raw + a.off_red);        /* [4 warps][nt][2] */
        uint32_t red_ph = 0;
        /* the 128 epilogue threads meet on an mbarrier (a bounded wait, unlike bar.sync: after a give-up nobody is left waiting for good) */
        auto esync = [&]() { mbar_arrive(bar_red); if (!mbar_wait(bar_red, red_ph, abort_flag, kWaitLimitR)) { raise_r(a, abort_flag, 8, pc); dead = true; } red_ph ^= 1u; };
        /* writes this block's sums of sample n (or zeros): (sum, sum of squares) per channel */
        auto flush = [&](int n, bool have) {
            esync();                                            /* every warp is done with the staging buffers the exchange area overlays */
            if (STATS && have) {
#pragma unroll
                for (int k = 0; k < NCH; k++) {
                    double ws = 0.0, wq = 0.0;
#pragma unroll
                    for (int t = 0; t < 8; t++) {
                        const double a8 = lanes8_sum(dsum[k][t], sp4, sp2, sp1), q8 = lanes8_sum(dsq[k][t], sp4, sp2, sp1);
                        if (t == sx) { ws = a8; wq = q8; }
                        dsum[k][t] = 0.0; dsq[k][t] = 0.0;
                    }
                    double *d = red + ((size_t)(q4 * a.nt + k * 32 + sch)) * 2;
                    d[0] = ws; d[1] = wq;
                }
            }
            esync();
            if (et < a.nt) {
                double ss = 0.0, qq = 0.0;
                if (have) for (int w4 = 0; w4 < 4; w4++) { const double *r2 = red + ((size_t)(w4 * a.nt + et)) * 2; ss += r2[0]; qq += r2[1]; }
                double *d = a.part + (((size_t)n * a.gcol + bcol) * a.cop + ctile * a.nt + et) * 2;
                d[0] = ss; d[1] = qq;
            }
            esync();
        };
        /* fp16 rows on their way out: a thread converts one voxel (64 bytes per 32 channels), the warp's 32 rows pass through 2 KB of shared
           memory (16-byte chunk c of row r at chunk c ^ (r / 2 % 4): no bank conflicts either way) and leave as four stores of 512 contiguous
           bytes each (the eight voxels of one tile row) instead of 32 scattered 16-byte pieces per store */
        uint8_t *stg = smem_raw + a.off_stage + q4 * (2048 * NCH);
        uint8_t *stg_w = stg + lane * 64; const int swz = (lane >> 1) & 3;
        const uint8_t *stg_r = stg + (lane >> 2) * 64 + (lane & 3) * 16;
        const size_t plane_b = (size_t)a.H * a.W * 64, row_b = (size_t)a.W * 64;
        /* sample being accumulated and the first sample this block has planes of.  Nothing is written to `part` before the block has taken a plane
           out of TMEM: this kernel may have been started while its predecessor in the stream, which can be a conv that shares `part`, was still
           running, and of a prepared layer only the producer waits for the predecessor; a plane in TMEM means that wait is over.  So the zero entries of the
           samples this block has no planes of are written at the end. */
        int n_cur = -1, n_first = -1;
        while (piece.u < piece.u1 && !dead) {
            const Run rn = next_run(a, piece);
            const int x0t = (rn.txy % a.tiles_x) * 8, y0t = (rn.txy / a.tiles_x) * 16;
            const int ox = x0t + rx, oy = y0t + ry;
            const bool row_ok = oy < a.H && ox < a.W;
            const int sy = y0t + q4 * 4;                        /* first of the four tile rows this warp stores */
            uint8_t *run_dst = (uint8_t *)a.e.y + (((size_t)rn.n * a.e.nb_dst + a.e.b0 + ctile * NCH) * S + (size_t)sy * a.W + x0t + (lane >> 2)) * 64 + cl * 16;
            if (stats && rn.n != n_cur) {
                if (n_cur >= 0) flush(n_cur, true); else n_first = rn.n;
                n_cur = rn.n;
            }
            for (int z = rn.zb; z < rn.ze && !dead; z++, pc++) {
                const int slot = NS - 1 - pcm;
                if (!mbar_wait(bar_accf + 8 * slot, (uint32_t)pph, abort_flag, kWaitLimitR)) { raise_r(a, abort_flag, 5, pc, bar_accf + 8 * slot - bar_tma, pph); dead = true; break; }
                tc_fence_after();
                uint32_t rr[NCH][32];
                const uint32_t tcol = tlane + (uint32_t)(slot * a.nt);
                tmem_ld32(tcol, rr[0]);
                if (NCH > 1) tmem_ld32(tcol + 32, rr[NCH - 1]);
                tmem_ld_wait();
                tmem_zero32(tcol);
                if (NCH > 1) tmem_zero32(tcol + 32);
                if (a.fast_h16 && !STATS) {
                    /* fp16 blocked output [n][block][voxel][32]: bias, one rounding.  A thread has a whole row of 64 bytes and stores it as two full sectors: passing
                       the rows through shared memory for 512-byte runs took a tenth of its bandwidth, which the MMA operands need (64 -> 64 MX-fp4 on 64^3 20.9 us,
                       18.5 this way; 32 -> 32 MX-fp8 on 128^3 68.9 and 68.0) */
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_acce + 8 * slot);          /* the slot is free once it is in registers and zeroed */
                    uint8_t *pv = (uint8_t *)a.e.y + (((size_t)rn.n * a.e.nb_dst + a.e.b0 + ctile * NCH) * S + ((size_t)z * a.H + oy) * a.W + ox) * 64;
#pragma unroll
                    for (int jc = 0; jc < NCH; jc++) {
                        const float4 *bs = (const float4 *)(bias_s + jc * 32);
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            uint32_t h[8];
#pragma unroll
                            for (int t = 0; t < 4; t++) {
                                const float4 b0 = bs[4 * k + t];
                                const __half2 x0 = __floats2half2_rn(__fadd_rn(__uint_as_float(rr[jc][16 * k + 4 * t]), b0.x), __fadd_rn(__uint_as_float(rr[jc][16 * k + 4 * t + 1]), b0.y));
                                const __half2 x1 = __floats2half2_rn(__fadd_rn(__uint_as_float(rr[jc][16 * k + 4 * t + 2]), b0.z), __fadd_rn(__uint_as_float(rr[jc][16 * k + 4 * t + 3]), b0.w));
                                h[2 * t] = *(const uint32_t *)&x0; h[2 * t + 1] = *(const uint32_t *)&x1;
                            }
                            if (row_ok) st_32b(pv + (size_t)jc * S * 64 + k * 32, h[0], h[1], h[2], h[3], h[4], h[5], h[6], h[7]);
                        }
                    }
                } else if (a.fast_h16) {
                    /* the same with the statistics, which are taken where a warp re-reads its rows; the zeroing of the slot completes meanwhile */
                    __syncwarp();                               /* the previous plane's rows have been read out of the staging buffer */
#pragma unroll
                    for (int jc = 0; jc < NCH; jc++) {
                        const float4 *bs = (const float4 *)(bias_s + jc * 32);
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const float4 b0 = bs[2 * k], b1 = bs[2 * k + 1];
                            __half2 h[4];
                            h[0] = __floats2half2_rn(__fadd_rn(__uint_as_float(rr[jc][8 * k + 0]), b0.x), __fadd_rn(__uint_as_float(rr[jc][8 * k + 1]), b0.y));
                            h[1] = __floats2half2_rn(__fadd_rn(__uint_as_float(rr[jc][8 * k + 2]), b0.z), __fadd_rn(__uint_as_float(rr[jc][8 * k + 3]), b0.w));
                            h[2] = __floats2half2_rn(__fadd_rn(__uint_as_float(rr[jc][8 * k + 4]), b1.x), __fadd_rn(__uint_as_float(rr[jc][8 * k + 5]), b1.y));
                            h[3] = __floats2half2_rn(__fadd_rn(__uint_as_float(rr[jc][8 * k + 6]), b1.z), __fadd_rn(__uint_as_float(rr[jc][8 * k + 7]), b1.w));
                            *(uint4 *)(stg_w + jc * 2048 + ((k ^ swz) << 4)) = make_uint4(*(const uint32_t *)&h[0], *(const uint32_t *)&h[1], *(const uint32_t *)&h[2], *(const uint32_t *)&h[3]);
                        }
                    }
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_acce + 8 * slot);          /* the slot is free once it is in registers and zeroed */
                    uint8_t *pz = run_dst + (size_t)z * plane_b;
#pragma unroll
                    for (int jc = 0; jc < NCH; jc++) {
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const uint4 v = *(const uint4 *)(stg_r + jc * 2048 + i * 512);
                            const bool in = sy + i < a.H;
                            if (in) *(uint4 *)(pz + (size_t)jc * S * 64 + (size_t)i * row_b) = v;
                            if (in) {
                                const __half2 *hp = (const __half2 *)&v;
#pragma unroll
                                for (int t = 0; t < 4; t++) {
                                    const float2 f = __half22float2(hp[t]);
                                    const double p0 = (double)f.x, p1 = (double)f.y;
                                    dsum[jc][2 * t] += p0; dsq[jc][2 * t] = fma(p0, p0, dsq[jc][2 * t]);
                                    dsum[jc][2 * t + 1] += p1; dsq[jc][2 * t + 1] = fma(p1, p1, dsq[jc][2 * t + 1]);
                                }
                            }
                        }
                    }
                } else if (!STATS && a.fast_pm16) {
                    /* plane-major fp16: a tile row is 16 bytes of a plane.  The warp's 32 voxels pass through shared memory as [channel pair][voxel], so that a lane
                       stores whole tile rows instead of a 2-byte piece a channel (32 -> 32 on 64^3 20.7 us, 17.1 this way; 64 -> 64 51.4 and 30.4).  On volumes far
                       beyond L2 half-written sectors bound it (128^3 233 us) */
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_acce + 8 * slot);
                    uint32_t *sp = (uint32_t *)(smem_raw + a.off_stage + q4 * 2048);
#pragma unroll
                    for (int jc = 0; jc < NCH; jc++) {
                        const float4 *bs = (const float4 *)(bias_s + jc * 32);
                        __syncwarp();                       /* the rows before have been read */
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            const float4 b0 = bs[k];
                            const __half2 x0 = __floats2half2_rn(__fadd_rn(__uint_as_float(rr[jc][4 * k]), b0.x), __fadd_rn(__uint_as_float(rr[jc][4 * k + 1]), b0.y));
                            const __half2 x1 = __floats2half2_rn(__fadd_rn(__uint_as_float(rr[jc][4 * k + 2]), b0.z), __fadd_rn(__uint_as_float(rr[jc][4 * k + 3]), b0.w));
                            sp[2 * k * 32 + lane] = *(const uint32_t *)&x0; sp[(2 * k + 1) * 32 + lane] = *(const uint32_t *)&x1;
                        }
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            const int q = i * 32 + lane, pair = q >> 2, y = sy + (q & 3), c = (ctile * NCH + jc) * 32 + 2 * pair;
                            const uint4 u = *(const uint4 *)(sp + pair * 32 + (q & 3) * 8), v = *(const uint4 *)(sp + pair * 32 + (q & 3) * 8 + 4);
                            __half *d = (__half *)a.e.y + ((size_t)rn.n * a.e.co_real + c) * S + ((size_t)z * a.H + y) * a.W + x0t;
                            if (y < a.H && c < a.e.co_real) *(uint4 *)d = make_uint4(__byte_perm(u.x, u.y, 0x5410), __byte_perm(u.z, u.w, 0x5410), __byte_perm(v.x, v.y, 0x5410), __byte_perm(v.z, v.w, 0x5410));
                            if (y < a.H && c + 1 < a.e.co_real) *(uint4 *)(d + S) = make_uint4(__byte_perm(u.x, u.y, 0x7632), __byte_perm(u.z, u.w, 0x7632), __byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x7632));
                        }
                    }
                } else {
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_acce + 8 * slot);
#pragma unroll
                    for (int jc = 0; jc < NCH; jc++) {
                        float v[32];
#pragma unroll
                        for (int k = 0; k < 32; k++) v[k] = __uint_as_float(rr[jc][k]);
                        epi_chunk<true>(a.e, rn.n, z, oy, ox, row_ok, ctile * NCH + jc, v, bias_s + jc * 32);
                    }
                }
                if (++pcm == NS) { pcm = 0; pph ^= 1; }
            }
        }
        if (stats && !dead) {
            if (n_cur >= 0) flush(n_cur, true);
            for (int n = 0; n < a.N; n++) if (n_cur < 0 || n < n_first || n > n_cur) flush(n, false);
            /* the last block of this column tile to get here turns the partial sums into coefficients; the order of the additions is
               fixed (block 0, 1, ...), so the result does not depend on which block came last */
            volatile unsigned &last = *(volatile unsigned *)(smem_raw + 776);
            __threadfence();
            esync();
            if (et == 0) { const unsigned tk = atomicAdd(&g_conv_tickets[ctile], 1u); last = tk == (unsigned)a.gcol - 1u; if (last) g_conv_tickets[ctile] = 0u; }
            esync();
            if (last) {
                __threadfence();
                for (int i = et; i < a.N * a.nt; i += 128) {
                    const int n = i / a.nt, c = ctile * a.nt + i % a.nt;
                    if (c >= a.e.co_real) continue;
                    double s0 = 0.0, q0 = 0.0;
                    const double *pp = a.part + ((size_t)n * a.gcol * a.cop + c) * 2;
                    for (int t = 0; t < a.gcol; t++) { s0 += __ldcg(pp + (size_t)t * a.cop * 2); q0 += __ldcg(pp + (size_t)t * a.cop * 2 + 1); }
                    const double m = s0 / (double)S, v = fmax(q0 / (double)S - m * m, 0.0);
                    const float rs = (float)(1.0 / sqrt(v + (double)a.eps)), ca = __fmul_rn(rs, a.gamma ? a.gamma[c] : 1.f);
                    a.coef[2 * ((size_t)n * a.e.co_real + c)] = ca;
                    a.coef[2 * ((size_t)n * a.e.co_real + c) + 1] = __fmaf_rn(-(float)m, ca, a.beta ? a.beta[c] : 0.f);
                }
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

}   // namespace
