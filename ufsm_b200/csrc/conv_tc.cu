/* MX block-scaled implicit-GEMM 3-D convolution forward on the sm_100a tensor cores (tcgen05, TMEM accumulators, TMA staging).

   GEMM view.  M = 128 output voxels of one tile (8 along x by 16 along y of one z plane), N = up to 128 output channels,
   K = taps x input channels in steps of one MX block pair: 32 E4M3 bytes (kind::mxf8f6f4, one UE8M0 scale per row) or 64 E2M1
   nibbles (kind::mxf4, two scales per row) per tcgen05.mma.  The activation tensor is the reference's channel-blocked MX
   storage (src/lp_common.cuh:100-106), so one voxel's K step is 32 contiguous bytes (fp8) or two 16-byte rows of adjacent
   blocks (fp4).

   Operand staging.  A 3^3 conv loads, per (input block, dz), one halo plane of 18 x 10 voxels with TMA (out-of-range voxels are
   zero-filled: that is the padding) as two 16-byte-wide planes [k half][y][x][16 B].  In that layout the canonical K-major
   no-swizzle UMMA operand (8 rows x 16 B core matrices; stride 160 B between the 16 y groups, 2880 B between the K halves) of
   every (dy, dx) tap is the same tile at a start address shifted by (dy * 10 + dx) * 16 bytes (2944 B where each half is a load of its own, so
   that its TMA destination is 128-byte aligned), so nine MMAs reuse one load.
   Weights are prepared once into the exact shared-memory image of a stage ([tap][k half][row][16 B] + scale bytes in the
   TMEM scale layout) and arrive with one bulk copy.  1^3 convs (head, the 2^3 stride-2 down conv on a space-to-depth copy, the
   transposed conv as a GEMM to 8 Cout columns) run the same pipeline with one tap and four K items a stage.

   Scale factors.  tcgen05 block-scaled MMAs read scales from TMEM: row r of a 128-row operand at lane r % 32, column r / 32,
   byte = scale id.  The scale of an A row depends on the tap (it is the shifted voxel's), so four epilogue warps gather, per
   stage, the nine shifted scale sets from the scale plane into that layout in shared memory, and the MMA warp copies them to
   TMEM with tcgen05.cp before issuing the stage's MMAs.  Out-of-range voxels get scale 1 (their codes are zero).

   Roles (192 threads): warp 0 = TMA producer; warp 1 = TMEM allocation, scale copies and MMA issue; warps 2-5 = scale gather, then the epilogue
   (tcgen05.ld of 32 channels per voxel = one MX block per thread: bias, fp16 store or MX requantisation;
   InstanceNorm partial sums are taken by a separate pass over the stored output).  Every wait is bounded; a wait that gives up records (code, block, stage) in a device
   flag, raises a block-wide abort flag and the block tears down normally. */
#include "conv_epi.cuh"
#include "tc_ptx.cuh"
#include <stdlib.h>
#include <string.h>

namespace {

constexpr int kThreads = 192;
constexpr int kTmemCols = 256;
constexpr int kSfBase = 128;        /* TMEM columns: [0, 128) accumulators, then two scale buffers of 40 (A 20 | B 20) */
constexpr long long kWaitLimit = 4000000000ll;   /* clock cycles (about two seconds) */

struct ConvArgs {
    int N, D, H, W;                 /* the grid of GEMM rows */
    int nkb;                        /* 32-channel blocks of the activation tensor */
    int nki;                        /* K items per tap: nkb (fp8) or ceil(nkb / 2) (fp4) */
    int taps, bits;
    int cop, nt, ntiles_n;          /* GEMM columns (padded to 32), column tile, column tiles */
    int tiles_x, tiles_y;
    int ring;                       /* pipeline depth */
    int stage_bytes, offW, offSFB, offA, offSFA;
    int w_stage_bytes, nst;         /* packed weight bytes per stage, stages per column tile */
    int items_max, ipq, nquad;      /* K items per stage, items per scale quad (4 fp8 / 2 fp4), quads per stage */
    const uint8_t *x_sc;
    const uint8_t *wpk;
    /* K split: the ksplit blocks of an output tile are a cluster; each takes a contiguous range of the stages and keeps its fp32 accumulators in shared
       memory, where the blocks add them up chunk by chunk in split order */
    int ksplit;
    int first_n;                        /* first sample of this launch */
    /* 3^3 stride-2 pad-1 conv: K item = (tap, input block), each item's A tile is its own strided TMA load from the input grid Di x Hi x Wi */
    int s2, nbi, nit, Di, Hi, Wi;       /* stride-2 conv: blocks of the input tensor, K items per tap, input grid */
    int ref, half;                      /* 3^3 on MX-fp8 codes in the reference's layout (32-byte rows): a half of a row a load; bytes between the halves of a stage's A */
    EpiArgs e;
    int *err;
};


__device__ __forceinline__ void raise(const ConvArgs &a, volatile int *abort_flag, int code, int stage) {
    if (atomicCAS(a.err, 0, code) == 0) { a.err[1] = (int)(blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)); a.err[2] = stage; a.err[3] = (int)threadIdx.x; }
    *abort_flag = 1;
    __threadfence_block();
}

/* WDEP: the weights and the bias were written by a kernel just ahead in the stream */
template <int BITS, bool WDEP>
__global__ void __launch_bounds__(kThreads, 2) conv_mx_k(const __grid_constant__ CUtensorMap map0, const ConvArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    /* control block, then the stage ring at the next 1024-byte boundary */
    uint64_t *bars = (uint64_t *)smem_raw;                       /* ring each: tma full, scales laid out, empty; then accumulator full */
    uint32_t *tmem_slot = (uint32_t *)(smem_raw + 512);
    volatile int *abort_flag = (volatile int *)(smem_raw + 516);
    uint8_t *stages = smem_raw + 1024;
    const int warp = (int)uni(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int R = a.ring;
    const uint32_t bar_tma = smem_u32(bars), bar_sf = bar_tma + 8 * R, bar_empty = bar_tma + 16 * R, bar_acc = bar_tma + 24 * R;

    const int txy = blockIdx.x, tx = txy % a.tiles_x, ty = txy / a.tiles_x;
    const int z = blockIdx.y;
    const int sp = (int)blockIdx.z % a.ksplit, bz = (int)blockIdx.z / a.ksplit;
    const int n = a.first_n + bz / a.ntiles_n, ntile = bz % a.ntiles_n;
    const int x0 = tx * 8, y0 = ty * 16;
    const int n0 = ntile * a.nt, n_cur = min(a.nt, a.cop - n0);
    /* this block's stages: all of them, or its share (whole input items of a 3^3 conv, so that every share has a live stage) */
    int st_lo = 0, st_hi = a.nst;
    if (a.ksplit > 1) {
        if (a.taps == 27) { st_lo = 3 * (a.nki * sp / a.ksplit); st_hi = 3 * (a.nki * (sp + 1) / a.ksplit); }
        else { st_lo = a.nst * sp / a.ksplit; st_hi = a.nst * (sp + 1) / a.ksplit; }
    }

    if (threadIdx.x == 0) {
        for (int i = 0; i < R; i++) { mbar_init(bar_tma + 8 * i, 1); mbar_init(bar_sf + 8 * i, 4); mbar_init(bar_empty + 8 * i, 1); }
        mbar_init(bar_acc, 1);
        *abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), kTmemCols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();                               /* the next kernel cannot take this block's tensor memory any more */
    const uint32_t tmem = uni(*tmem_slot);
    /* The order of a 3^3 block's stages (each the nine (dy, dx) of an input item and a dz): in MX-fp4 dz outermost, which is the z-marching kernel's order, so that the two give the same bits
       and the choice between them may follow the batch; in MX-fp8 the items outermost.  A conv of one item has the two orders in one.  (MX-fp4 sums are exact in fp32 over many octaves of
       scales, so its order seldom shows; in MX-fp8 it shows in the last bit, and a network of convs makes 3 to 7 % of that in its logits: codes next to a rounding boundary.) */
    const int first_dz = a.taps == 27 && z == 0, last_dz = a.taps == 27 ? (z == a.D - 1 ? 1 : 2) : 0;       /* stages whose input plane lies outside the volume would add zeros: left out */
    const int nshare = st_hi - st_lo, st_step = a.taps == 27 ? 3 : 1, st_first = st_lo + first_dz;
    const int nlive = a.taps == 27 ? nshare / 3 * (last_dz - first_dz + 1) : nshare;
    auto next_stage = [&](int st) -> int {
        if (BITS == 8) return a.taps == 27 && st % 3 == last_dz ? st + 3 - (last_dz - first_dz) : st + 1;
        st += st_step; return st < st_hi ? st : st - nshare + 1;
    };
    auto stage_items = [&](int st) -> int { return a.taps == 27 ? 9 : min(4, a.nki - 4 * st); };

    /* a stage's A and B scales from shared memory to TMEM buffer buf.  Copies and MMAs of one thread run in issue order, so two buffers are enough and no
       barrier guards them; with uniform operands a copy costs the warp a few clocks (as a role of its own it cost a barrier round trip a stage: 128 -> 128 on
       32^3 18.0 us against 16.6, 256 -> 128 28.4 against 26.1) */
    auto copy_scales = [&](int st, uint32_t so, int buf, uint32_t lead) {
        const uint32_t sf_hi = desc_hi(128), sb0 = smem_u32(stages), sfa_lo = desc_lo(sb0 + a.offSFA, 0) + so, sfb_lo = desc_lo(sb0 + a.offSFB, 0) + so;
        const uint32_t sfa_t = tmem + kSfBase + buf * 40, sfb_t = sfa_t + 20;
        const int nq = a.taps == 27 ? a.nquad : (stage_items(st) + a.ipq - 1) / a.ipq;
        for (int q = 0; q < nq; q++) {
            utccp_32x128b(sfa_t + 4 * q, desc_make(sfa_lo + 32u * q, sf_hi), lead);
            utccp_32x128b(sfb_t + 4 * q, desc_make(sfb_lo + 32u * q, sf_hi), lead);
        }
    };

    if (warp == 0) {
        /* ---------------- TMA producer ---------------- */
        {
            const uint32_t lead = elect_one();
            if (lead) tma_prefetch_desc(&map0);
            const uint8_t *wbase = a.wpk + (size_t)ntile * a.nst * a.w_stage_bytes;
            auto put_weights = [&](int st, int s) {
                const uint32_t bar = bar_tma + 8 * s;
                const int abytes = a.taps == 27 ? 5760 : stage_items(st) * 4096;
                if (!lead) return;
                mbar_expect_tx(bar, (uint32_t)(abytes + a.w_stage_bytes));
                bulk_g2s(smem_u32(stages + (size_t)s * a.stage_bytes + a.offW), wbase + (size_t)st * a.w_stage_bytes, (uint32_t)a.w_stage_bytes, bar);
            };
            /* the weights of the first ring's stages are constants of a prepared layer: they load while the previous kernel of the stream is still running */
            int early = 0;
            if (!WDEP) for (int st = st_first; early < min(nlive, R); st = next_stage(st)) put_weights(st, early++);
            pdl_wait();                          /* from here on this thread touches activations */
            int s = 0, ph = 0;
            for (int it = 0, st = st_first; it < nlive; it++, st = next_stage(st)) {
                uint8_t *sb = stages + (size_t)s * a.stage_bytes;
                const uint32_t bar = bar_tma + 8 * s;
                const int items = stage_items(st);
                if (it >= early) {
                    if (!__all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, kWaitLimit))) { if (lane == 0) raise(a, abort_flag, 1, st); break; }
                    put_weights(st, s);
                }
                /* two 16-byte-wide planes per K item (fp8: the halves of block ki; fp4: blocks 2 ki and 2 ki + 1) */
                if (a.taps == 27) {
                    const int ki = st / 3, zi = z + st % 3 - 1;
                    if (BITS == 8 && a.ref) { tma_load_5d(smem_u32(sb + a.offA), &map0, bar, 0, x0 - 1, y0 - 1, zi, n * a.nkb + ki, lead); tma_load_5d(smem_u32(sb + a.offA) + 2944, &map0, bar, 16, x0 - 1, y0 - 1, zi, n * a.nkb + ki, lead); }
                    else tma_load_4d(smem_u32(sb + a.offA), &map0, bar, (x0 - 1) * 16, y0 - 1, zi, BITS == 8 ? (n * a.nkb + ki) * 2 : n * a.nkb + 2 * ki, lead);
                } else {
                    for (int j = 0; j < items; j++) {
                        const int ki = 4 * st + j;
                        if (a.s2) {   /* every second voxel of the input, starting at 2 v + tap - 1 (voxels outside the grid arrive as zeros: the padding) */
                            /* K item ki = tap * a.nit + i: fp8: block i (its two half planes); fp4: blocks 2 i and 2 i + 1 (the second may lie past the
                               sample's last block: its weights are zero and its scale is read as 1) */
                            const int tap = ki / a.nit, blk = ki - tap * a.nit;
                            tma_load_5d(smem_u32(sb + a.offA + j * 4096), &map0, bar, 0, 2 * x0 + tap % 3 - 1, 2 * y0 + (tap / 3) % 3 - 1, 2 * z + tap / 9 - 1, BITS == 8 ? (n * a.nbi + blk) * 2 : n * a.nbi + 2 * blk, lead);
                        } else
                        tma_load_4d(smem_u32(sb + a.offA + j * 4096), &map0, bar, x0 * 16, y0, z, BITS == 8 ? (n * a.nkb + ki) * 2 : n * a.nkb + 2 * ki, lead);
                    }
                }
                if (++s == R) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        /* ---------------- MMA issue: one warp, of which one lane issues; everything that does not change with the stage is worked out before the loop ---------------- */
        {
            const uint32_t lead = elect_one();
            int s = 0, ph = 0; bool ok = true;
            const uint32_t sb0 = smem_u32(stages), sstep = (uint32_t)a.stage_bytes >> 4;
            const uint32_t b_hi = desc_hi(128), a_hi = a.taps == 27 ? desc_hi(160) : desc_hi(128);
            const uint32_t a_lo0 = desc_lo(sb0 + a.offA, (uint32_t)a.half), b_lo0 = desc_lo(sb0 + a.offW, (uint32_t)a.nt * 16);
            const uint32_t idesc0 = BITS == 8 ? idesc_mxf8(n_cur, 0, 0) : idesc_mxf4(n_cur, 0, 0);
            const uint32_t bstep = (uint32_t)a.nt * 2;
            int buf = 0;
            for (int it = 0, st = st_first; it < nlive && ok; it++, st = next_stage(st)) {
                const uint32_t so = (uint32_t)s * sstep;
                const uint32_t sfa_t = tmem + kSfBase + buf * 40, sfb_t = sfa_t + 20;
                if (!__all_sync(0xffffffffu, mbar_wait(bar_sf + 8 * s, ph, abort_flag, kWaitLimit))) { if (lane == 0) raise(a, abort_flag, 3, st); ok = false; break; }
                if (!__all_sync(0xffffffffu, mbar_wait(bar_tma + 8 * s, ph, abort_flag, kWaitLimit))) { if (lane == 0) raise(a, abort_flag, 2, st); ok = false; break; }
                tc_fence_after();
                copy_scales(st, so, buf, lead);
                if (a.taps == 27) issue_items<BITS, 9, true>(tmem, a_lo0 + so, a_hi, b_lo0 + so, b_hi, bstep, 0, idesc0, sfa_t, sfb_t, it == 0, 9, lead);
                else issue_items<BITS, 4, false>(tmem, a_lo0 + so, a_hi, b_lo0 + so, b_hi, bstep, 256, idesc0, sfa_t, sfb_t, it == 0, stage_items(st), lead);
                umma_commit(bar_empty + 8 * s, lead);
                if (++s == R) { s = 0; ph ^= 1; }
                buf ^= 1;
            }
            umma_commit(bar_acc, lead);   /* also after a give-up: the epilogue must not wait for its full limit */
        }
    } else {
        /* ---------------- scale gather, then epilogue ---------------- */
        const int q4 = warp & 3, r = q4 * 32 + lane;             /* TMEM lane quarter of this warp; GEMM row of this thread */
        const int ry = r >> 3, rx = r & 7;
        const int oy = y0 + ry, ox = x0 + rx;
        const bool row_ok = oy < a.H && ox < a.W;
        const size_t S = (size_t)a.D * a.H * a.W;
        pdl_wait();
        /* The scale bytes of a stage come straight from the scale plane, an L2 round trip.  They are asked for a stage ahead of their use, so that the
           trip of one stage overlaps the packing of the one before: without that the gather was the pipeline's slowest role (a stage of the
           320 -> 320 conv on 8^3 1650 clocks). */
        constexpr int NB = 9 * (BITS == 8 ? 1 : 2);
        unsigned raw[NB];
        unsigned inm = 0u;                                       /* 3^3: the taps of this row that lie inside the plane */
        int toff[3];                                             /* and the offsets of its three tap rows */
        if (a.taps == 27) {
#pragma unroll
            for (int j = 0; j < 9; j++) { const int iy = oy + j / 3 - 1, ix = ox + j % 3 - 1; if (iy >= 0 && iy < a.H && ix >= 0 && ix < a.W) inm |= 1u << j; }
#pragma unroll
            for (int k = 0; k < 3; k++) toff[k] = (oy + k - 1) * a.W + ox - 1;
        }
        auto load_scales = [&](int st) {
            if (a.taps == 27) {
                const int ki = st / 3, zi = z + st % 3 - 1;
                const uint8_t *p = a.x_sc + ((size_t)n * a.nkb + (BITS == 8 ? ki : 2 * ki)) * S + (size_t)zi * a.H * a.W;
                const bool two = BITS == 4 && 2 * ki + 1 < a.nkb;
#pragma unroll
                for (int j = 0; j < 9; j++) {
                    const bool in = (inm >> j) & 1u;
                    raw[j] = in ? ld_dep(p + toff[j / 3] + j % 3) : 127u;
                    if (BITS == 4) raw[9 + j] = in && two ? ld_dep(p + S + toff[j / 3] + j % 3) : 127u;
                }
            } else {
                const int items = stage_items(st);
                const size_t vox = ((size_t)z * a.H + oy) * a.W + ox;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    raw[j] = 127u; if (BITS == 4) raw[9 + j] = 127u;
                    if (j >= items) continue;
                    const int ki = 4 * st + j;
                    if (a.s2) {
                        const int tap = ki / a.nit, blk = ki - tap * a.nit;
                        const int iz = 2 * z + tap / 9 - 1, iy = 2 * oy + (tap / 3) % 3 - 1, ix = 2 * ox + tap % 3 - 1;
                        const bool in = row_ok && iz >= 0 && iz < a.Di && iy >= 0 && iy < a.Hi && ix >= 0 && ix < a.Wi;
                        const size_t Si = (size_t)a.Di * a.Hi * a.Wi, vi = ((size_t)iz * a.Hi + iy) * a.Wi + ix;
                        const uint8_t *p = a.x_sc + ((size_t)n * a.nbi + (BITS == 8 ? blk : 2 * blk)) * Si + vi;
                        if (in) raw[j] = ld_dep(p);
                        if (BITS == 4 && in && 2 * blk + 1 < a.nbi) raw[9 + j] = ld_dep(p + Si);
                    } else {
                        const uint8_t *p = a.x_sc + ((size_t)n * a.nkb + (BITS == 8 ? ki : 2 * ki)) * S + vox;
                        if (row_ok) raw[j] = ld_dep(p);
                        if (BITS == 4 && row_ok && 2 * ki + 1 < a.nkb) raw[9 + j] = ld_dep(p + S);
                    }
                }
            }
        };
        load_scales(st_first);
        for (int it = 0, st = st_first, nxt; it < nlive; it++, st = nxt) {
            const int s = it % R, ph = (it / R) & 1;
            nxt = next_stage(st);
            uint32_t wq[5] = {0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu};
            const int nj = a.taps == 27 ? 9 : 4;
#pragma unroll
            for (int j = 0; j < 9; j++) {
                if (j >= nj) break;
                if (BITS == 8) wq[j >> 2] = (wq[j >> 2] & ~(0xffu << (8 * (j & 3)))) | (raw[j] << (8 * (j & 3)));
                else wq[j >> 1] = (wq[j >> 1] & ~(0xffffu << (16 * (j & 1)))) | ((raw[j] | (raw[9 + j] << 8)) << (16 * (j & 1)));
            }
            if (it + 1 < nlive) load_scales(nxt);
            if (!mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, kWaitLimit)) { raise(a, abort_flag, 4, st); break; }
            uint32_t *sfa = (uint32_t *)(stages + (size_t)s * a.stage_bytes + a.offSFA);
            /* quad q: word (lane, column) = row 32 * column + lane -> this thread's word is at lane * 4 + quarter */
#pragma unroll
            for (int q = 0; q < 5; q++) if (q < a.nquad) sfa[q * 128 + lane * 4 + q4] = wq[q];
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_sf + 8 * s);        /* one arrival a warp: arrivals on one barrier serialise */
        }
        /* ---- epilogue ---- */
        if (!mbar_wait(bar_acc, 0, abort_flag, kWaitLimit)) raise(a, abort_flag, 5, 0);
        tc_fence_after();
        const int nchunk = n_cur >> 5;
        if (!*abort_flag && a.ksplit > 1) {
            /* this block's part of the sums, [32-column chunk][column quad][row][4], into the now idle stage ring */
            float4 *mine = (float4 *)stages + r;
            for (int jc = 0; jc < nchunk; jc++) {
                uint32_t rr[32];
                tmem_ld32(tmem + ((uint32_t)(q4 * 32) << 16) + (uint32_t)(jc * 32), rr);
                tmem_ld_wait();
#pragma unroll
                for (int k = 0; k < 8; k++) mine[jc * 1024 + k * 128] = make_float4(__uint_as_float(rr[4 * k]), __uint_as_float(rr[4 * k + 1]), __uint_as_float(rr[4 * k + 2]), __uint_as_float(rr[4 * k + 3]));
            }
        } else if (!*abort_flag) {
            for (int jc = 0; jc < nchunk; jc++) {
                uint32_t rr[32];
                tmem_ld32(tmem + ((uint32_t)(q4 * 32) << 16) + (uint32_t)(jc * 32), rr);
                tmem_ld_wait();
                float v[32];
#pragma unroll
                for (int k = 0; k < 32; k++) v[k] = __uint_as_float(rr[k]);
                epi_chunk<WDEP>(a.e, n, z, oy, ox, row_ok, (n0 >> 5) + jc, v, a.e.bias + n0 + jc * 32);
            }
        }
    }
    if (a.ksplit > 1) {
        /* K split: the blocks of a tile are a cluster.  Each takes every ksplit-th 32-column chunk, adds the parts of all of them in split order (the order
           is fixed: results do not depend on scheduling) straight from their shared memory, and runs the chunk's epilogue.  Leaving the parts
           in global memory for the block that came last cost 5 to 6 us a launch.  Every thread passes both cluster barriers, also after a
           give-up. */
        __syncwarp();
        cluster_sync_all();
        if (warp >= 2 && warp < 6) {
            const int q4 = warp & 3, r = q4 * 32 + lane, oy = y0 + (r >> 3), ox = x0 + (r & 7), nchunk = n_cur >> 5;
            const bool row_ok = oy < a.H && ox < a.W;
            const uint32_t base = smem_u32(stages) + (uint32_t)r * 16u;
            for (int jc = sp; jc < nchunk && !*abort_flag; jc += a.ksplit) {
                const uint32_t cb = base + (uint32_t)jc * 16384u;
                float4 t[8], nx[8];
                float v[32];
                auto fetch = [&](int s2) { const uint32_t ra = cluster_addr(cb, (uint32_t)s2);
#pragma unroll
                    for (int k = 0; k < 8; k++) nx[k] = cluster_ld4(ra + (uint32_t)k * 2048u); };
                fetch(0);
#pragma unroll
                for (int k = 0; k < 8; k++) t[k] = nx[k];
                fetch(1);
#pragma unroll
                for (int k = 0; k < 8; k++) { v[4 * k] = t[k].x; v[4 * k + 1] = t[k].y; v[4 * k + 2] = t[k].z; v[4 * k + 3] = t[k].w; }
                for (int s2 = 1; s2 < a.ksplit; s2++) {
#pragma unroll
                    for (int k = 0; k < 8; k++) t[k] = nx[k];
                    if (s2 + 1 < a.ksplit) fetch(s2 + 1);
#pragma unroll
                    for (int k = 0; k < 8; k++) { v[4 * k] += t[k].x; v[4 * k + 1] += t[k].y; v[4 * k + 2] += t[k].z; v[4 * k + 3] += t[k].w; }
                }
                epi_chunk<WDEP>(a.e, n, z, oy, ox, row_ok, (n0 >> 5) + jc, v, a.e.bias + n0 + jc * 32);
            }
        }
        __syncwarp();
        cluster_sync_all();                                  /* no block leaves while another may still read its part */
    }
    /* ---------------- teardown ---------------- */
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && warp == 0 && lane == 0) {
        /* after a give-up: let this thread's own copies in flight land (bounded) before the block's shared memory is released */
        for (int s = 0; s < R; s++) { const long long t0 = clock64(); while (!mbar_try(bar_tma + 8 * s, 0) && !mbar_try(bar_tma + 8 * s, 1) && clock64() - t0 < 20000000ll) { } }
    }
    if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem, kTmemCols); }
}

/* ---- weight preparation of the one-tap convs: fp32 weights -> the shared-memory image of every (column tile, stage): items x [k half][row][16 B]
   codes, then the scale bytes in the TMEM scale layout (quad, lane, column, byte).  One thread per (column tile, stage, item, row).
   Quantisation per (row, tap, 32 input channels) as the reference's prep_w8_k / prep_w4_k (src/lp_f8fwd.cu:54-71,
   src/lp_f4fwd.cu:53-66). ---- */
__global__ void __launch_bounds__(128) prep_w_k(const PrepArgs p) {
    const size_t total = (size_t)p.ntiles_n * p.nst * p.items_max * p.nt;
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < (size_t)p.cop && p.bias_p) {
        const int c = (int)i, o = p.kind == UMX_TCONV2 ? c % (32 * p.cob_t) : c;
        p.bias_p[c] = (p.bias && o < p.co) ? p.bias[o] : 0.f;
    }
    if (i >= total) return;
    const int rl = (int)(i % p.nt), j = (int)((i / p.nt) % p.items_max), st = (int)((i / ((size_t)p.nt * p.items_max)) % p.nst), ntile = (int)(i / ((size_t)p.nt * p.items_max * p.nst));
    const int row = ntile * p.nt + rl;
    const int tap = 0, ki = 4 * st + j;
    uint8_t *stg = p.wpk + ((size_t)ntile * p.nst + st) * p.w_stage_bytes;
    const bool live = row < p.cop && ki < p.nki;
    unsigned w[8]; unsigned sb[2] = {127u, 127u};
    float v[32];
    if (p.bits == 8) {
#pragma unroll
        for (int k = 0; k < 32; k++) v[k] = live ? prep_src(p, row, tap, ki, k) : 0.f;
        sb[0] = mx_encode_row32<8>(v, w);
    } else {
        unsigned w4[4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
#pragma unroll
            for (int k = 0; k < 32; k++) v[k] = live ? prep_src(p, row, tap, 2 * ki + h, k) : 0.f;
            sb[h] = mx_encode_row32<4>(v, w4);
#pragma unroll
            for (int t = 0; t < 4; t++) w[4 * h + t] = w4[t];
        }
    }
    if (!live) { sb[0] = 127u; sb[1] = 127u; }
    uint4 *d0 = (uint4 *)(stg + ((size_t)(j * 2 + 0) * p.nt + rl) * 16), *d1 = (uint4 *)(stg + ((size_t)(j * 2 + 1) * p.nt + rl) * 16);
    *d0 = make_uint4(w[0], w[1], w[2], w[3]); *d1 = make_uint4(w[4], w[5], w[6], w[7]);
    uint8_t *sf = stg + (size_t)p.items_max * p.nt * 32;
    const int q = j / p.ipq, l = rl & 31, c = rl >> 5;
    if (p.bits == 8) sf[q * 512 + l * 16 + c * 4 + (j & 3)] = (uint8_t)sb[0];
    else { sf[q * 512 + l * 16 + c * 4 + (j & 1) * 2] = (uint8_t)sb[0]; sf[q * 512 + l * 16 + c * 4 + (j & 1) * 2 + 1] = (uint8_t)sb[1]; }
}

typedef CUresult (*encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
encode_fn get_encode() {
    static encode_fn fn = nullptr;
    if (!fn) {
        void *p = nullptr; cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) != cudaSuccess || qr != cudaDriverEntryPointSuccess) { umx_latch_msg("cuTensorMapEncodeTiled is not available from the driver"); return nullptr; }
        fn = (encode_fn)p;
    }
    return fn;
}
int ceil_div(int a, int b) { return (a + b - 1) / b; }

}   // namespace

int umx_conv_r_takes(const umx_conv *c, const uint8_t *x_sc, int N, int D, int H, int W, const EpiArgs &e);

int umx_conv_fwd_r(const umx_conv *c, const uint8_t *x_sc, const CUtensorMap *m0, int ref, void *enc, int N, int D, int H, int W, const EpiArgs &e,
                   double *part, const float *gamma, const float *beta, float eps, float *coef);
extern "C" void umx_in_stats_coef(const void *y, int N, int C, int D, int H, int W, const float *gamma, const float *beta, float eps, double *part, float *coef);
void umx_in_part(const void *y, int N, int C, int D, int H, int W, double *part);
uint8_t *umx_conv_p_prepare(const umx_conv *c, const float *w_dev);
uint8_t *umx_conv_stem_prepare(const umx_conv *c, const float *w_dev);
int umx_conv_fwd_stem(const umx_conv *c, const void *x, int src8, int N, int D, int H, int W, void *y);
int umx_conv_fwd_p(const umx_conv *c, const void *x, const uint8_t *x_sc, void *enc, int N, int D, int H, int W, const EpiArgs &e);
const uint8_t *umx_prob_table(void);
void umx_mx_codes_to_split(const void *x, size_t blocks, size_t S, void *y);
int umx_conv_s2_takes(const umx_conv *c);
int umx_conv_fwd_s2(const umx_conv *c, const void *x, int split, const uint8_t *x_sc, void *enc, int N, int Di, int Hi, int Wi, const EpiArgs &e);
/* the z-marching image of either kind */
static int march_image(const umx_conv *c, RImageGeo *o) { return c->kind == UMX_CONV3S2 ? umx_conv_s2_image(c, o) : umx_conv_r_image(c, o); }


/* the fields of a conv that follow from its kind and sizes */
static void conv_geometry(umx_conv *c, int kind, int co, int ci, int bits) {
    memset(c, 0, sizeof *c);
    c->kind = kind; c->co = co; c->ci = ci; c->bits = bits;
    c->taps = kind == UMX_CONV3 ? 27 : 1;
    const int nbi = ceil_div(ci, 32);
    /* K blocks of the GEMM: (sub-voxel or tap) x input blocks; the MX-fp4 stride-2 conv pads the blocks of a tap to an even count, so that a
       K item of two blocks never spans two taps (two different shifts of the input) */
    c->nkb = kind == UMX_DOWN2 ? 8 * nbi : kind == UMX_CONV3S2 ? 27 * (bits == 4 ? 2 * ceil_div(nbi, 2) : nbi) : nbi;
    c->nki = bits == 8 ? c->nkb : ceil_div(c->nkb, 2);
    c->cob_t = ceil_div(co, 32);
    c->cop = (kind == UMX_TCONV2 ? 8 : 1) * c->cob_t * 32;
    c->nt = c->cop >= 128 ? 128 : c->cop;               /* 32, 64, 96 or 128 */
    c->ntiles_n = ceil_div(c->cop, c->nt);
    c->items_max = c->taps == 27 ? 9 : 4;
    c->ipq = bits == 8 ? 4 : 2;
    c->nquad = ceil_div(c->items_max, c->ipq);
    c->nst = c->taps == 27 ? 3 * c->nki : ceil_div(c->nki, 4);
    c->w_stage_bytes = c->items_max * c->nt * 32 + c->nquad * 512;
}
static size_t wpk_bytes(const umx_conv *c) { return (size_t)c->ntiles_n * c->nst * c->w_stage_bytes; }
static PrepArgs prep_args(const umx_conv *c, const float *w_dev, const float *bias_dev) {
    PrepArgs p; memset(&p, 0, sizeof p);
    p.w = w_dev; p.wpk = c->wpk; p.bias = bias_dev; p.bias_p = c->bias_p; p.kind = c->kind; p.co = c->co; p.ci = c->ci; p.bits = c->bits; p.cop = c->cop; p.cob_t = c->cob_t;
    p.nkb = c->nkb; p.nki = c->nki; p.taps = c->taps; p.nt = c->nt; p.ntiles_n = c->ntiles_n; p.nst = c->nst; p.items_max = c->items_max; p.ipq = c->ipq; p.nquad = c->nquad; p.w_stage_bytes = c->w_stage_bytes;
    return p;
}
static umx_conv *conv_build(int kind, const float *w_dev, const float *bias_dev, int co, int ci, int bits) {
    if (!umx_ready("umx_conv_create")) return nullptr;
    if ((bits != 8 && bits != 4) || kind < 0 || kind > 4 || co < 1 || ci < 1 ) { fprintf(stderr, "umx_conv_create: bad arguments (kind %d, co %d, ci %d, bits %d)\n", kind, co, ci, bits); abort(); }
    umx_conv *c = (umx_conv *)malloc(sizeof *c);
    conv_geometry(c, kind, co, ci, bits);
    const size_t wb = wpk_bytes(c);
    c->wpk = (uint8_t *)nn_malloc(wb); c->bias_p = (float *)nn_malloc((size_t)c->cop * 4);
    if (!c->wpk || !c->bias_p) { umx_conv_free(c); return nullptr; }
    cudaMemset(c->wpk, 127, wb);   /* unused scale slots read as 1 */
    const PrepArgs p = prep_args(c, w_dev, bias_dev);
    if (kind == UMX_CONV3 || kind == UMX_CONV3S2) {
        RImageGeo g; memset(&g, 0, sizeof g);
        if (march_image(c, &g)) {
            c->wr = (uint8_t *)nn_malloc((size_t)g.w_bytes * g.ncol);
            if (!c->wr) { umx_conv_free(c); return nullptr; }
            cudaMemset(c->wr, 127, (size_t)g.w_bytes * g.ncol);
        }
        umx_prep_w27(p, c->wr, g.nt, g.w_bytes, g.w_codes, g.gt, g.goff1, g.goff2);
        c->wstem = umx_conv_stem_prepare(c, w_dev);
    } else {
        const size_t total = (size_t)c->ntiles_n * c->nst * c->items_max * c->nt;
        prep_w_k<<<(unsigned)((total + 127) / 128), 128>>>(p);
        g_umx_launches++;
        c->wp = umx_conv_p_prepare(c, w_dev);
    }
    UMX_CK("umx_conv_create");
    /* the conv kernels read the prepared weights and the bias before their griddepcontrol.wait (they are layer constants that may load while
       the previous kernel still runs), so the preparation kernels must have finished before a conv can be launched behind them */
    cudaStreamSynchronize(0);
    return c;
}
/* A conv for one call on weights that may change before the next one: c is the caller's, its images live in scratch and are made by the first
   kernel that asks for them (image_for_call), in stream order; nothing is allocated, copied or waited for once the scratch has its size.  The
   caller keeps other users of that scratch out (lp_entry.cu's lock) and leaves no pointer to c behind. */
void umx_conv_per_call(umx_conv *c, int kind, const float *w_dev, const float *bias_dev, int co, int ci, int bits) {
    conv_geometry(c, kind, co, ci, bits);
    c->w_src = w_dev; c->b_src = bias_dev;
}
/* which 0: the general kernel's image, 1: the z-marching kernel's; true when it is there.  A kernel that follows one made here reads weights and bias behind its
   dependency wait (w_dep); launched without the programmatic attribute instead it took 2.5 to 3.6 us longer (256 -> 256 in MX-fp4 on
   15 x 18 x 20 27.2 us, 24.7 this way; 32 -> 32 on 64^3 20.7 and 17.0). */
static bool image_for_call(umx_conv *c, int which) {
    if (which ? c->wr != nullptr : c->wpk != nullptr) return true;
    if (!c->w_src) return false;
    c->bias_p = (float *)umx_ws(15, (size_t)c->cop * 4);
    RImageGeo g; memset(&g, 0, sizeof g);
    if (which) { if (!march_image(c, &g)) return false; c->wr = (uint8_t *)umx_ws(14, (size_t)g.w_bytes * g.ncol); }
    else c->wpk = (uint8_t *)umx_ws(13, wpk_bytes(c));
    if (!c->bias_p || (which ? !c->wr : !c->wpk)) return false;
    PrepArgs p = prep_args(c, c->w_src, c->b_src);
    if (which) p.wpk = nullptr;
    umx_prep_w27(p, which ? c->wr : nullptr, g.nt, g.w_bytes, g.w_codes, g.gt, g.goff1, g.goff2);
    return true;
}
extern "C" umx_conv *umx_conv_create_dev(int kind, const float *w_dev, const float *bias_dev, int co, int ci, int bits) { return conv_build(kind, w_dev, bias_dev, co, ci, bits); }
extern "C" umx_conv *umx_conv_create(int kind, const float *w, const float *bias, int co, int ci, int bits) {
    if (!umx_ready("umx_conv_create")) return nullptr;
    const size_t nw = (size_t)co * ci * ((kind == UMX_CONV3 || kind == UMX_CONV3S2) ? 27 : kind == UMX_CONV1 ? 1 : 8);
    float *wd = (float *)nn_malloc(nw * 4), *bd = bias ? (float *)nn_malloc((size_t)co * 4) : nullptr;
    if (!wd || (bias && !bd)) { nn_free(wd); nn_free(bd); return nullptr; }
    nn_h2d(wd, w, nw * 4); if (bias) nn_h2d(bd, bias, (size_t)co * 4);
    umx_conv *c = conv_build(kind, wd, bd, co, ci, bits);
    cudaDeviceSynchronize();
    nn_free(wd); nn_free(bd);
    return c;
}
extern "C" void umx_conv_free(umx_conv *c) { if (!c) return; nn_free(c->wpk); nn_free(c->bias_p); nn_free(c->wr); nn_free(c->wp); nn_free(c->wstem); free(c); }
int umx_stats_chunks(int D, int H, int W);
/* room for 512 partial sums of two doubles per (sample, channel): the statistics pass uses up to that many voxel chunks, the conv epilogue
   one entry per block */
extern "C" size_t umx_stats_doubles(int N, int co, int D, int H, int W) { (void)D; (void)H; (void)W; return (size_t)N * 512 * (size_t)(ceil_div(co, 32) * 32) * 2; }

static int up128(int v) { return (v + 127) & ~127; }
/* bytes of the general kernel's stage: weights and their scales, A, A scales */
static int stage_layout(const umx_conv *c, int *offA, int *offSFA) {
    *offA = up128(c->w_stage_bytes);
    *offSFA = *offA + up128(c->taps == 27 ? 2944 + 2880 : 4 * 4096);
    return (*offSFA + c->nquad * 512 + 1023) & ~1023;
}
/* K split of the general kernel for the layers with fewer tiles than multiprocessors (the deep levels); chosen from one sample's geometry (the grid of GEMM rows) and nothing else, so that
   a sample's result does not depend on the batch it is in */
int umx_conv_ksplit(const umx_conv *c, int D, int H, int W, int sms) {
    static int no_split = -1;
    if (no_split < 0) { const char *ev = getenv("UMX_KSPLIT"); no_split = ev && *ev == '0'; }
    int offA, offSFA;
    const int stage_bytes = stage_layout(c, &offA, &offSFA);
    const long long blocks1 = (long long)ceil_div(W, 8) * ceil_div(H, 16) * D * c->ntiles_n;
    const int units = c->taps == 27 ? c->nki : c->nst;
    long long ks = blocks1 > 0 ? sms / blocks1 : 1;
    if (ks > units) ks = units;
    if (ks > c->nst / 6) ks = c->nst / 6;              /* at least six stages a share: shorter shares cost more in the reduction than they save */
    /* at most as many parts as 16 KB pieces fit the shallow ring, whatever ring this launch has, so that the split does not change with the batch
       (never more than six, a portable cluster) */
    int rs = 100 * 1024 / stage_bytes; if (rs > 8) rs = 8; if (rs < 2) rs = 2;
    const long long cap = (long long)rs * stage_bytes / 16384; if (ks > cap) ks = cap;
    return !no_split && ks >= 2 && ks <= 8 ? (int)ks : 1;
}

static int g_last_kernel = -1;
extern "C" int umx_conv_last_kernel(void) { return g_last_kernel; }
struct NormArgs { const float *gamma, *beta; float eps; float *coef; };
static int conv_fwd_impl(const umx_conv *c, const void *x, int N, int D, int H, int W, void *y, int out_mode, int out_bits, int nb_dst, int b0, double *part, int flags, const NormArgs *nrm) {
    if (!umx_ready("umx_conv_fwd")) return -1;
    if (!c) { umx_latch_msg("umx_conv_fwd: no conv"); return -1; }
    if (part && (out_mode != UMX_OUT_H16B || c->kind == UMX_TCONV2)) { fprintf(stderr, "umx_conv_fwd: partial sums only with a blocked fp16 output of a plain conv\n"); abort(); }
    if (out_mode == UMX_OUT_PROB8 && (!c || c->kind != UMX_CONV1 || part || nb_dst)) { fprintf(stderr, "umx_conv_fwd: probability bytes only from a 1^3 conv into a tensor of its own\n"); abort(); }
    if ((out_mode == UMX_OUT_MX || out_mode == UMX_OUT_MXRAW) && out_bits != 8 && out_bits != 4) { fprintf(stderr, "umx_conv_fwd: MX output needs out_bits 8 or 4\n"); abort(); }
    if (flags & (UMX_X_H16 | UMX_X_U8)) {
        /* x is the fp16 tensor [N][ci][D][H][W] itself.  The tap-packed kernel takes the one-channel 3^3 case as it is; everything else is
           quantised into scratch first and goes the usual way. */
        if (c->kind != UMX_CONV3 && c->kind != UMX_CONV1) { fprintf(stderr, "umx_conv_fwd: an fp16 input only for the 3^3 and 1^3 convs\n"); abort(); }
        /* UMX_STEM=0 in the environment (read at every such call): always quantise first.  That path adds the taps of a one-channel conv one
           by one in ascending order, as a sequential fp32 loop does; the tap-packed tile adds them inside one MMA. */
        const char *env = getenv("UMX_STEM");
        const bool stem_on = !(env && *env == '0');
        if (stem_on && c->wstem && out_mode == UMX_OUT_H16B && !nb_dst) {
            const int r = umx_conv_fwd_stem(c, x, (flags & UMX_X_U8) != 0, N, D, H, W, y);
            if (r < 0) return -1;
            if (r == 0) {
                g_last_kernel = 3;
                if (nrm) umx_in_stats_coef(y, N, c->co, D, H, W, nrm->gamma, nrm->beta, nrm->eps, part, nrm->coef);
                else if (part) umx_in_part(y, N, c->co, D, H, W, part);
                return 0;
            }
        }
        if (flags & UMX_X_U8) {                             /* bytes -> fp16 in scratch */
            const size_t nx = (size_t)N * c->ci * D * H * W;
            void *h = umx_ws(12, nx * 2);
            if (!h) return -1;
            umx_u8_to_h16((const uint8_t *)x, nx, h);
            x = h;
        }
        void *ws = umx_ws(1, umx_mx_bytes32(c->bits, N, c->ci, (size_t)D * H * W));
        if (!ws) return -1;
        umx_pm_to_mx32(x, UMX_F16, N, c->ci, (size_t)D * H * W, ws, c->bits, UMX_LAYOUT_SPLIT);
        x = ws; flags = (flags & ~(UMX_X_H16 | UMX_X_U8)) | UMX_X_SPLIT;
    }
    encode_fn enc = get_encode(); if (!enc) return -1;
    ConvArgs a; memset(&a, 0, sizeof a);
    /* the stride-2 3^3 conv is given its input grid; its GEMM rows are the output grid ceil(D / 2) x ceil(H / 2) x ceil(W / 2) */
    const bool s2 = c->kind == UMX_CONV3S2;
    const int Dx = D, Hx = H, Wx = W, nbx = s2 ? ceil_div(c->ci, 32) : c->nkb;  /* grid and 32-channel blocks of the tensor x */
    const size_t Sx = (size_t)Dx * Hx * Wx;
    if (s2) { D = (D + 1) / 2; H = (H + 1) / 2; W = (W + 1) / 2; a.s2 = 1; a.nbi = nbx; a.nit = c->nki / 27; a.Di = Dx; a.Hi = Hx; a.Wi = Wx; }
    a.N = N; a.D = D; a.H = H; a.W = W; a.nkb = c->nkb; a.nki = c->nki; a.taps = c->taps; a.bits = c->bits;
    a.cop = c->cop; a.nt = c->nt; a.ntiles_n = c->ntiles_n; a.tiles_x = ceil_div(W, 8); a.tiles_y = ceil_div(H, 16);
    a.w_stage_bytes = c->w_stage_bytes; a.nst = c->nst; a.items_max = c->items_max; a.ipq = c->ipq; a.nquad = c->nquad;
    a.offW = 0; a.offSFB = c->items_max * c->nt * 32;
    a.stage_bytes = stage_layout(c, &a.offA, &a.offSFA);
    static int sms_of[16];                                  /* multiprocessors, looked up once per device */
    int d0 = 0; cudaGetDevice(&d0); d0 &= 15;
    if (!sms_of[d0]) { int v = 148; cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d0); sms_of[d0] = v; }
    const int sms = sms_of[d0];
    /* two blocks a multiprocessor (two issuing threads keep the tensor pipe busier than one) for the narrow tiles, and for the wide ones when
       there are more blocks than multiprocessors; a deep ring for one block otherwise */
    const long long blocks_all = (long long)a.tiles_x * a.tiles_y * D * N * a.ntiles_n;
    const int budget = (c->nt > 64 && blocks_all <= sms) ? 200 * 1024 : 100 * 1024;
    a.ring = budget / a.stage_bytes; if (a.ring > 8) a.ring = 8; if (a.ring < 2) a.ring = 2;
    const size_t S = (size_t)D * H * W;
    const int rb = c->bits == 8 ? 32 : 16;
    a.x_sc = (const uint8_t *)x + (size_t)N * nbx * Sx * rb;
    a.e.N = N; a.e.D = D; a.e.H = H; a.e.W = W; a.e.cop = c->cop;
    a.e.out_mode = out_mode; a.e.out_bits = out_bits; a.e.tconv = c->kind == UMX_TCONV2; a.e.co_real = c->co; a.e.cob_t = c->cob_t;
    a.e.nb_dst = nb_dst ? nb_dst : c->cob_t; a.e.b0 = nb_dst ? b0 : 0;
    a.e.y = y; a.e.y_split = (flags & UMX_Y_SPLIT) != 0; a.err = umx_errflag();
    if (out_mode == UMX_OUT_PROB8) { a.e.ptab = umx_prob_table(); if (!a.e.ptab) return -1; }
    if (!a.err) return -1;
    /* algorithmic work: 2 x output voxels x real input channels x real output channels x taps (no credit for padding) */
    const double flops = 2.0 * (double)N * S * (c->kind == UMX_DOWN2 ? 8.0 : 1.0) * c->ci * (double)c->co * (c->kind == UMX_TCONV2 ? 8.0 : 1.0) * ((c->taps == 27 || s2) ? 27.0 : 1.0);
    static int force_v1 = -1;
    if (force_v1 < 0) { const char *ev = getenv("UMX_CONV_V1"); force_v1 = ev && *ev && *ev != '0'; }
    if (s2 && !force_v1 && umx_conv_s2_takes(c) && image_for_call((umx_conv *)c, 1)) {
        a.e.bias = c->bias_p;
        const int pid = umx_prof_open(flops);
        const int rc = umx_conv_fwd_s2(c, x, c->bits == 8 && (flags & UMX_X_SPLIT), a.x_sc, (void *)enc, N, Dx, Hx, Wx, a.e);
        if (rc <= 0) {
            umx_prof_close(pid);
            g_umx_launches++; g_last_kernel = 4;
            UMX_CK("umx_conv_fwd");
            if (rc == 0 && nrm) umx_in_stats_coef(y, N, c->co, D, H, W, nrm->gamma, nrm->beta, nrm->eps, part, nrm->coef);
            else if (rc == 0 && part) umx_in_part(y, N, c->co, D, H, W, part);
            return rc;
        }
    }
    /* tensor map over the activation codes seen as 16-byte-wide planes [plane][z][y][x * 16 B]: fp8 in the split layout has two planes a
       block, fp4 one.  A box is (10 or 8 voxels) x (18 or 16 rows) x 1 plane of z x 2 planes; voxels outside the volume read as zero. */
    /* MX-fp8 in the reference's layout: a 3^3 conv loads the two halves of the 32-byte rows apart; a one-tap conv has its codes re-laid into scratch first.  32 -> 32 on
       7 x 9 x 11 11.1 us with a relayout pass ahead, 7.0 this way, on 64^3 17.4 and 13.3, on 128^3 88 and 63; 256 -> 256 on 15 x 18 x 20 26.7 and 24.5: pieces of 16 bytes hold neither kernel up. */
    a.ref = c->bits == 8 && !(flags & UMX_X_SPLIT) && c->taps == 27;
    a.half = a.ref ? 2944 : c->taps == 27 ? 2880 : 2048;
    if (c->bits == 8 && !(flags & UMX_X_SPLIT) && !a.ref) {
        void *ws = umx_ws(1, umx_mx_bytes32(8, N, nbx * 32, Sx));
        if (!ws) return -1;
        umx_mx_codes_to_split(x, (size_t)N * nbx, Sx, ws);         /* the scale plane stays where it is */
        x = ws;
    }
    CUtensorMap m0; memset(&m0, 0, sizeof m0);
    if (s2) {
        /* [plane][z][y][x][16 B] with a traversal stride of two voxels along x and y: a box of 16 x 32 voxel positions delivers 8 x 16 voxels */
        const cuuint64_t gd[5] = {16, (cuuint64_t)Wx, (cuuint64_t)Hx, (cuuint64_t)Dx, (cuuint64_t)N * nbx * (c->bits == 8 ? 2 : 1)};
        const cuuint64_t gs[4] = {16, (cuuint64_t)Wx * 16, (cuuint64_t)Wx * Hx * 16, (cuuint64_t)Sx * 16};
        const cuuint32_t box[5] = {16, 16, 32, 1, 2}, es[5] = {1, 2, 2, 1, 1};
        const CUresult r0 = enc(&m0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, (void *)x, gd, gs, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r0 != CUDA_SUCCESS) { char b[160]; snprintf(b, sizeof b, "umx_conv_fwd: cuTensorMapEncodeTiled failed (%d) for the stride-2 map of %d x %d x %d x %d, %d blocks", (int)r0, N, Dx, Hx, Wx, nbx); umx_latch_msg(b); return -1; }
    } else if (a.ref) {
        const cuuint64_t gd[5] = {32, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D, (cuuint64_t)N * c->nkb}, gs[4] = {32, (cuuint64_t)W * 32, (cuuint64_t)W * H * 32, (cuuint64_t)S * 32};
        const cuuint32_t box[5] = {16, 10, 18, 1, 1}, es[5] = {1, 1, 1, 1, 1};
        const CUresult r0 = enc(&m0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, (void *)x, gd, gs, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r0 != CUDA_SUCCESS) { char b[160]; snprintf(b, sizeof b, "umx_conv_fwd: cuTensorMapEncodeTiled failed (%d) for %d x %d x %d x %d, %d blocks of 32-byte rows", (int)r0, N, D, H, W, c->nkb); umx_latch_msg(b); return -1; }
    } else {
        const cuuint32_t bx = c->taps == 27 ? 10 : 8, by = c->taps == 27 ? 18 : 16;
        const cuuint64_t gd[4] = {(cuuint64_t)W * 16, (cuuint64_t)H, (cuuint64_t)D, (cuuint64_t)N * c->nkb * (c->bits == 8 ? 2 : 1)};
        const cuuint64_t gs[3] = {(cuuint64_t)W * 16, (cuuint64_t)W * H * 16, (cuuint64_t)S * 16};
        const cuuint32_t box[4] = {bx * 16, by, 1, 2}, es[4] = {1, 1, 1, 1};
        const CUresult r0 = enc(&m0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void *)x, gd, gs, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r0 != CUDA_SUCCESS) { char b[160]; snprintf(b, sizeof b, "umx_conv_fwd: cuTensorMapEncodeTiled failed (%d) for %d x %d x %d x %d, %d blocks", (int)r0, N, D, H, W, c->nkb); umx_latch_msg(b); return -1; }
    }
    /* InstanceNorm statistics are a separate pass over the stored output (umx_in_part below) */
    if (!force_v1 && c->kind == UMX_CONV3 && (c->wr || (c->w_src && umx_conv_r_takes(c, a.x_sc, N, D, H, W, a.e) && image_for_call((umx_conv *)c, 1)))) {   /* resident weights: the persistent z-marching kernel, when the geometry allows */
        const int pid = umx_prof_open(flops);
        a.e.bias = c->bias_p;
        int rc = (nrm && (flags & UMX_STATS_EPILOGUE)) ? umx_conv_fwd_r(c, a.x_sc, &m0, a.ref, (void *)enc, N, D, H, W, a.e, part, nrm->gamma, nrm->beta, nrm->eps, nrm->coef) : 1;
        const bool fused = rc == 0;
        if (rc > 0) rc = umx_conv_fwd_r(c, a.x_sc, &m0, a.ref, (void *)enc, N, D, H, W, a.e, nullptr, nullptr, nullptr, 0.f, nullptr);
        if (rc <= 0) {
            umx_prof_close(pid);
            g_umx_launches++; g_last_kernel = 1;
            UMX_CK("umx_conv_fwd");
            if (rc == 0 && nrm && !fused) umx_in_stats_coef(y, N, c->co, D, H, W, nrm->gamma, nrm->beta, nrm->eps, part, nrm->coef);
            else if (rc == 0 && part && !nrm) umx_in_part(y, N, c->co, D, H, W, part);
            return rc;
        }
    }
    a.e.bias = c->bias_p;
    if (!force_v1 && c->wp) {   /* one tap, resident weights: the streaming kernel */
        const int pid = umx_prof_open(flops);
        const int rc = umx_conv_fwd_p(c, x, a.x_sc, (void *)enc, N, D, H, W, a.e);
        if (rc <= 0) {
            umx_prof_close(pid);
            g_umx_launches++; g_last_kernel = 2;
            UMX_CK("umx_conv_fwd");
            if (rc == 0 && nrm) umx_in_stats_coef(y, N, c->co, D, H, W, nrm->gamma, nrm->beta, nrm->eps, part, nrm->coef);
            else if (rc == 0 && part) umx_in_part(y, N, c->co, D, H, W, part);
            return rc;
        }
    }
    if (out_mode == UMX_OUT_PROB8) {
        /* not the head's shape: fp16 plane-major logits into scratch, then the probability pass (the same bytes) */
        const size_t ny = (size_t)N * c->co * S;
        void *t = umx_ws(12, ny * 2);
        if (!t) return -1;
        const int rc = conv_fwd_impl(c, x, N, D, H, W, t, UMX_OUT_PM16, 0, 0, 0, nullptr, flags | (c->bits == 8 ? UMX_X_SPLIT : 0), nullptr);
        if (rc == 0) umx_h16_to_prob_u8(t, ny, (uint8_t *)y);
        return rc;
    }
    if (!image_for_call((umx_conv *)c, 0)) return -1;
    a.wpk = c->wpk; a.e.bias = c->bias_p;
    const size_t smem = 1024 + (size_t)a.ring * a.stage_bytes;
    static size_t smem_set[16];
    int dev = 0; cudaGetDevice(&dev); dev &= 15;
    if (smem_set[dev] < smem) {
        const void *ks[4] = {(const void *)conv_mx_k<8, false>, (const void *)conv_mx_k<4, false>, (const void *)conv_mx_k<8, true>, (const void *)conv_mx_k<4, true>};
        cudaError_t e = cudaSuccess;
        for (int i = 0; i < 4 && e == cudaSuccess; i++) e = cudaFuncSetAttribute(ks[i], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(227 * 1024));
        if (e != cudaSuccess) { umx_latch("umx_conv_fwd: shared memory attribute", e); return -1; }
        smem_set[dev] = 227 * 1024;
    }
    a.ksplit = umx_conv_ksplit(c, D, H, W, sms);
    const int per_n = a.ntiles_n * a.ksplit, n_max = per_n < 65535 ? 65535 / per_n : 1;      /* a grid has at most 65535 blocks along z: a larger batch goes in several launches */
    const int pid = umx_prof_open(flops);
    /* the parts need 16 KB a 32-column chunk of the ring */
    auto go = [&](auto k) {
        for (a.first_n = 0; a.first_n < N; a.first_n += n_max) {
            const dim3 grid(a.tiles_x * a.tiles_y, D, (unsigned)((N - a.first_n < n_max ? N - a.first_n : n_max) * per_n));
            if (a.ksplit > 1) umx_launch_cluster(k, grid, dim3(1, 1, (unsigned)a.ksplit), dim3(kThreads), smem, m0, a); else umx_launch(k, grid, dim3(kThreads), smem, m0, a);
            g_umx_launches++;
        }
    };
    if (c->w_src) { if (c->bits == 8) go(conv_mx_k<8, true>); else go(conv_mx_k<4, true>); }
    else if (c->bits == 8) go(conv_mx_k<8, false>); else go(conv_mx_k<4, false>);
    umx_prof_close(pid);
    g_last_kernel = 0;
    UMX_CK("umx_conv_fwd");
    if (nrm) umx_in_stats_coef(y, N, c->co, D, H, W, nrm->gamma, nrm->beta, nrm->eps, part, nrm->coef);
    else if (part) umx_in_part(y, N, c->co, D, H, W, part);
    return 0;
}
extern "C" int umx_conv_fwd(const umx_conv *c, const void *x, int N, int D, int H, int W, void *y, int out_mode, int out_bits, int nb_dst, int b0, double *part, int flags) {
    return conv_fwd_impl(c, x, N, D, H, W, y, out_mode, out_bits, nb_dst, b0, part, flags, nullptr);
}
/* conv -> blocked fp16 y, and the InstanceNorm coefficients (a, b) per (sample, channel) of that stored tensor; part: scratch of
   umx_stats_doubles doubles.  The resident-weight kernel takes the sums in its epilogue (fp32 inside 32-voxel units, exact above them);
   only under UMX_STATS_EPILOGUE; otherwise, and for the other kernels, the conv is followed by the statistics pass.  gamma / beta: device arrays or NULL (1 / 0). */
extern "C" int umx_conv_fwd_norm(const umx_conv *c, const void *x, int N, int D, int H, int W, void *y, double *part, const float *gamma, const float *beta, float eps, float *coef, int flags) {
    if (!part || !coef) { fprintf(stderr, "umx_conv_fwd_norm: part and coef are required\n"); abort(); }
    if (c && c->kind == UMX_TCONV2) { fprintf(stderr, "umx_conv_fwd_norm: not for the transposed conv\n"); abort(); }
    const NormArgs nrm = {gamma, beta, eps, coef};
    return conv_fwd_impl(c, x, N, D, H, W, y, UMX_OUT_H16B, 0, 0, 0, part, flags, &nrm);
}
