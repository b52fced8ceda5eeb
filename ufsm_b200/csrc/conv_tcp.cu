/* One-tap MX convs as a streaming GEMM: the 1^3 head, the 2^3 stride-2 down conv on a space-to-depth copy (K = 8 Cin) and the
   transposed conv (N = 8 Cout sub-voxel columns), for layers whose prepared weights fit in shared memory.  These layers move
   far more bytes than they compute, so the kernel is built around latency: persistent blocks (two a multiprocessor when shared
   memory allows), weights and B scale factors loaded once per block, and per job only what changes.

   GEMM rows are 128 consecutive voxels of the sample's linear voxel order.  In the split MX layout [plane][voxel][16 B] that is
   one contiguous 2 KB run per 16-byte-wide plane, so the A operand of a K item (32 fp8 or 64 fp4 channels) is one TMA box of
   256 x 2 eight-byte elements: [k half][128 rows][16 B], the canonical K-major no-swizzle operand (core matrices 128 B apart,
   halves 2 KB apart).  Rows past the end of the sample arrive as zeros.  The scale bytes of the same rows arrive as a second
   box (128 bytes x the stage's blocks) and one warp lays them out for tcgen05.cp.

   A job is (row tile, column tile of up to 64 GEMM columns); a stage is up to four K items of a job.  Jobs of a row tile are
   consecutive, so the tile is re-read from L2, not from HBM.  Accumulators alternate between TMEM slots; the epilogue is the
   generic one (bias, fp16 / MX / plane-major output, the transposed conv's scatter).

   Roles (384 threads): warp 0 producer and warp 1 MMA issue (the warp runs the loop, an elected lane issues; warp 1 also allocates TMEM), warp 2 scale
   layout, warp 3 idle, warps 4-11 epilogue (two groups, jobs in turn).  All waits are bounded as in conv_mx_k. */
#include "conv_epi.cuh"
#include "tc_ptx.cuh"
#include <stdlib.h>
#include <string.h>


namespace {

constexpr int kThreadsP = 384;
constexpr int kMaxSlotsP = 8;
constexpr long long kWaitLimitP = 4000000000ll;

struct ConvPArgs {
    int N, nkb, nki, bits, cop, ntp, ntiles, ngroups;
    long long S, rtiles_per_n, jobs;             /* voxels per sample, row tiles per sample, (row tile, column tile) jobs */
    int HW, W;
    unsigned hw_mul, w_mul; int hw_shift, w_shift;      /* reciprocals of H W and W (fast_div) */
    int ring, stage_bytes, offSW, offSFA, sw_rows;
    int w_bytes, w_codes, nquad, nslot;
    int tmem_cols, sfa_base, sfb_base;
    int off_w, off_ring;
    const uint8_t *wp;
    EpiArgs e;
    int *err;
};

/* a wait gave up (its own limit, or another role's abort flag): the first to get here names the block; every role of that block then leaves
   where it stood (stage, barrier, parity), which the host prints */
__device__ __forceinline__ void raise_p(const ConvPArgs &a, volatile int *abort_flag, int code, int stage, uint32_t bar_off = 0, uint32_t parity = 0) {
    if (atomicCAS(a.err, 0, code) == 0) { a.err[1] = (int)blockIdx.x; a.err[2] = stage; a.err[3] = (int)threadIdx.x; __threadfence(); }
    if (((volatile int *)a.err)[1] == (int)blockIdx.x && code < 8) { int *d = a.err + 16 + 4 * code; d[0] = stage; d[1] = (int)bar_off; d[2] = (int)parity; d[3] = 1; }
    *abort_flag = 1;
    __threadfence_block();
}

/* n / d for n < 2^31: mul = ceil(2^(31 + l) / d), shift = l - 1 with l = ceil(log2 d) (Granlund and Montgomery, "Division by invariant integers using
   multiplication"); mul = 0 stands for d = 1 */
__device__ __forceinline__ unsigned fast_div(unsigned n, unsigned mul, int shift) { return mul ? __umulhi(n, mul) >> shift : n; }
/* EPI: the output mode known at compile time (0: any, read from the arguments; 1: plane-major fp32; 2: plane-major fp16; 3: MX-fp8 split
   layout; 4: the same through the transposed conv's scatter; 5, 6: MX-fp4 likewise), so that the epilogue's code is only what that mode needs */
template <int BITS, int EPI>
__global__ void __launch_bounds__(kThreadsP, 2) conv_mxp_k(const __grid_constant__ CUtensorMap map0, const __grid_constant__ CUtensorMap maps, const ConvPArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint64_t *bars = (uint64_t *)smem_raw;
    uint32_t *tmem_slot = (uint32_t *)(smem_raw + 768);
    volatile int *abort_flag = (volatile int *)(smem_raw + 772);
    uint8_t *wsm = smem_raw + a.off_w, *stages = smem_raw + a.off_ring;
    const int warp = (int)uni(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int R = a.ring, NS = a.nslot;
    const uint32_t bar_tma = smem_u32(bars), bar_sf = bar_tma + 8 * R, bar_empty = bar_tma + 16 * R, bar_accf = bar_tma + 24 * R, bar_acce = bar_accf + 8 * kMaxSlotsP, bar_w = bar_acce + 8 * kMaxSlotsP;
    constexpr int IPQ = BITS == 8 ? 4 : 2, NQ = 4 / IPQ;      /* K items a scale quad, quads a stage */

    if (threadIdx.x == 0) {
        for (int i = 0; i < R; i++) { mbar_init(bar_tma + 8 * i, 1); mbar_init(bar_sf + 8 * i, 1); mbar_init(bar_empty + 8 * i, 1); }
        for (int i = 0; i < kMaxSlotsP; i++) { mbar_init(bar_accf + 8 * i, 1); mbar_init(bar_acce + 8 * i, 4); }
        mbar_init(bar_w, 1);
        *abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (threadIdx.x == 0) {
        /* the weight image is a constant of the layer: it may load while the previous kernel of the stream is still running */
        mbar_expect_tx(bar_w, (uint32_t)a.w_bytes);
        for (int o = 0; o < a.w_bytes; o += 32768) bulk_g2s(smem_u32(wsm + o), a.wp + o, (uint32_t)min(32768, a.w_bytes - o), bar_w);
    }
    if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), (uint32_t)a.tmem_cols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();                               /* the next kernel cannot take this block's tensor memory any more */
    const uint32_t tmem = uni(*tmem_slot);
    const long long j0 = a.jobs * (long long)blockIdx.x / (long long)gridDim.x, j1 = a.jobs * ((long long)blockIdx.x + 1) / (long long)gridDim.x;

    if (warp == 0) {
        /* ---------------- producer: the whole warp runs the loop on uniform values, one lane issues ---------------- */
        const uint32_t lead = elect_one();
        if (lead) { tma_prefetch_desc(&map0); tma_prefetch_desc(&maps); }
        pdl_wait();      /* the only role that reads activations from global memory; every other role's data comes through these loads, so the weight load and the B scale copies
                            overlap the previous kernel */
        int s = 0, ph = 0, it = 0; bool ok = true;
        /* job = (row tile, column tile), column tile fastest; the indices advance incrementally (no division per job) */
        int ntile = (int)(j0 % a.ntiles), n = (int)((j0 / a.ntiles) / a.rtiles_per_n), tin = (int)((j0 / a.ntiles) % a.rtiles_per_n);
        for (long long job = j0; job < j1 && ok; job++) {
            const int cx = tin * 256, pl0 = BITS == 8 ? n * a.nkb * 2 : n * a.nkb, cs = tin * 128;
            for (int g = 0; g < a.ngroups; g++) {
                if (!__all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, kWaitLimitP))) { if (lane == 0) raise_p(a, abort_flag, 1, it); ok = false; break; }
                const int items = min(4, a.nki - 4 * g);
                const uint32_t sb = smem_u32(stages + (size_t)s * a.stage_bytes), bar = bar_tma + 8 * s;
                if (lead) mbar_expect_tx(bar, (uint32_t)(items * 4096 + a.sw_rows * 128));
                for (int j = 0; j < items; j++) tma_load_2d(sb + j * 4096, &map0, bar, cx, pl0 + 2 * (4 * g + j), lead);
                tma_load_3d(sb + a.offSW, &maps, bar, cs, a.sw_rows * g, n, lead);
                it++; if (++s == R) { s = 0; ph ^= 1; }
            }
            if (++ntile == a.ntiles) { ntile = 0; if (++tin == (int)a.rtiles_per_n) { tin = 0; n++; } }
        }
    } else if (warp == 1) {
        /* ---------------- MMA issue (the warp runs the loop, one lane issues) ---------------- */
        {
            const uint32_t lead = elect_one();
            const bool ok0 = mbar_wait(bar_w, 0, abort_flag, kWaitLimitP);
            bool ok = __all_sync(0xffffffffu, ok0);
            if (!ok && lane == 0) raise_p(a, abort_flag, 6, 0);
            tc_fence_after();
            const uint32_t wbase = smem_u32(wsm), sf_hi = desc_hi(128), a_hi = desc_hi(128), b_hi = desc_hi(128);
            const uint32_t idesc_b = (BITS == 8 ? idesc_mxf8(0, 0, 0) : idesc_mxf4(0, 0, 0));
            if (ok) {
                const int nsf = a.ntiles * a.ngroups * NQ;
                for (int i = 0; i < nsf; i++) utccp_32x128b(tmem + a.sfb_base + i * 4, desc_make(desc_lo(wbase + a.w_codes + i * 512, 0), sf_hi), lead);
            }
            const uint32_t a_lo0 = desc_lo(smem_u32(stages), 2048), a_step = (uint32_t)a.stage_bytes >> 4, sfa_off = (uint32_t)a.offSFA >> 4;
            const uint32_t b_lo0 = desc_lo(wbase, (uint32_t)a.ntp * 16), b_item = 2u * (uint32_t)a.ntp, b_tile = (uint32_t)a.nki * b_item;
            int s = 0, ph = 0, it = 0, slot = 0, sph = 0;
            long long job = j0; int ntile = (int)(j0 % a.ntiles);
            while (ok && job < j1) {
                const int n_cur = min(a.ntp, a.cop - ntile * a.ntp);
                const uint32_t idn = idesc_b | ((uint32_t)(n_cur >> 3) << 17), d = tmem + (uint32_t)(slot * a.ntp);
                if (!__all_sync(0xffffffffu, mbar_wait(bar_acce + 8 * slot, (uint32_t)(sph ^ 1), abort_flag, kWaitLimitP))) { if (lane == 0) raise_p(a, abort_flag, 7, it); break; }
                for (int g = 0; g < a.ngroups; g++) {
                    if (!__all_sync(0xffffffffu, mbar_wait(bar_sf + 8 * s, ph, abort_flag, kWaitLimitP))) { if (lane == 0) raise_p(a, abort_flag, 3, it); ok = false; break; }
                    tc_fence_after();                            /* the scale warp passed the stage's load barrier before: the codes have landed too */
                    const uint32_t a_lo = a_lo0 + (uint32_t)s * a_step, sfa_t = tmem + (uint32_t)a.sfa_base + ((uint32_t)it & 1u) * 8u;
                    const uint32_t sfb_t = tmem + (uint32_t)a.sfb_base + (uint32_t)((ntile * a.ngroups + g) * NQ * 4);
                    const uint32_t bb = b_lo0 + (uint32_t)ntile * b_tile + (uint32_t)(4 * g) * b_item;
                    const int items = min(4, a.nki - 4 * g);
#pragma unroll
                    for (int q = 0; q < NQ; q++) utccp_32x128b(sfa_t + 4 * q, desc_make((a_lo & 0xffffu) + sfa_off + 32u * q, sf_hi), lead);
#pragma unroll
                    for (int j = 0; j < 4; j++) if (j < items) {
                        const int q = j / IPQ, id = (j % IPQ) * (4 / IPQ);
                        const uint32_t idesc = idn | ((uint32_t)id << 4) | ((uint32_t)id << 29), acc = (g == 0 && j == 0) ? 0u : 1u;
                        const uint64_t ad = desc_make(a_lo + (uint32_t)j * 256u, a_hi), bd = desc_make(bb + (uint32_t)j * b_item, b_hi);
                        if (BITS == 8) umma_mxf8(d, ad, bd, idesc, acc, sfa_t + 4 * q, sfb_t + 4 * q, lead); else umma_mxf4(d, ad, bd, idesc, acc, sfa_t + 4 * q, sfb_t + 4 * q, lead);
                    }
                    /* one commit a stage: a second one right behind it costs this warp 135 clocks.  The last stage of a job completes its accumulators, and the epilogue, which waits for
                       those, passes the stage back to the producer */
                    umma_commit(g == a.ngroups - 1 ? bar_accf + 8 * slot : bar_empty + 8 * s, lead);
                    it++; if (++s == R) { s = 0; ph ^= 1; }
                }
                if (++slot == NS) { slot = 0; sph ^= 1; }
                job++; if (++ntile == a.ntiles) ntile = 0;
            }
        }
    } else if (warp == 2) {
        /* ---------------- A scale layout: the window holds, per block of the stage, the scale bytes of the 128 rows ---------------- */
        int s = 0, ph = 0, it = 0; bool ok = true;
        const long long nst = (j1 - j0) * a.ngroups;
        for (long long i = 0; i < nst && ok; i++) {
            if (!mbar_wait(bar_tma + 8 * s, ph, abort_flag, kWaitLimitP)) { if (lane == 0) raise_p(a, abort_flag, 4, it); ok = false; break; }
            uint8_t *stg = stages + (size_t)s * a.stage_bytes;
            const uint8_t *sw = stg + a.offSW;
            uint32_t *sfa = (uint32_t *)(stg + a.offSFA);
#pragma unroll
            for (int q = 0; q < NQ; q++) {
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const uint8_t *p = sw + (q * 4) * 128 + c * 32 + lane;
                    sfa[q * 128 + lane * 4 + c] = (uint32_t)p[0] | ((uint32_t)p[128] << 8) | ((uint32_t)p[256] << 16) | ((uint32_t)p[384] << 24);
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_sf + 8 * s);
            it++; if (++s == R) { s = 0; ph ^= 1; }
        }
    } else if (warp >= 4) {
        /* ---------------- epilogue: two groups of four warps; jobs alternate between them, and so do the accumulator slots (their number is even, so a
           group sees every phase of its slots' barriers).  A thread has the whole GEMM row of one voxel.  What bounds the MX modes is the instructions of this
           part (64 -> 32 transposed conv on 64^3: 416 a row of 32 values with two divisions, 64-bit index products and a store of 16 bytes for each
           half row, 44.4 us; 31.7 us this way): coordinates come from multiplications by host-made reciprocals, bases are worked out once a job,
           biases are added in pairs, and a transposed conv's two x neighbours, which share sectors, belong to one job and leave in one store. ---------------- */
        const int q4 = warp & 3, eg = (warp - 4) >> 2, r = q4 * 32 + lane;
        const uint32_t tlane = tmem + ((uint32_t)(q4 * 32) << 16);
        int slot = eg, sph = 0; bool dead = false;
        const unsigned Su = (unsigned)a.S;
        int last_s = ((eg + 1) * a.ngroups - 1) % R;                 /* ring slot of the last stage of this group's job */
        long long job = j0 + eg;
        int ntile = (int)(job % a.ntiles), n = (int)((job / a.ntiles) / a.rtiles_per_n), tin = (int)((job / a.ntiles) % a.rtiles_per_n);
        for (; job < j1 && !dead; job += 2) {
            const int n_cur = min(a.ntp, a.cop - ntile * a.ntp), nchunk = n_cur >> 5, cb = ntile * (a.ntp >> 5);
            if (!mbar_wait(bar_accf + 8 * slot, (uint32_t)sph, abort_flag, kWaitLimitP)) { raise_p(a, abort_flag, 5, (int)(job - j0)); dead = true; break; }
            if (q4 == 0 && lane == 0) mbar_arrive(bar_empty + 8 * last_s);
            for (last_s += 2 * a.ngroups; last_s >= R;) last_s -= R;
            tc_fence_after();
            const uint32_t tcol = tlane + (uint32_t)(slot * a.ntp);
            const unsigned vo = (unsigned)tin * 128u + (unsigned)r;
            const bool row_ok = vo < Su;
            auto release = [&]() { tc_fence_before(); __syncwarp(); if (lane == 0) mbar_arrive(bar_acce + 8 * slot); };     /* one arrival per warp: arrivals on one barrier serialise */
            if (EPI == 7 || ((EPI == 1 || EPI == 2) && a.e.co_real <= 8)) {
                /* a plane-major output of at most eight channels (the head): only those accumulator columns leave TMEM; a warp's 32 voxels are consecutive
                   in every plane.  7: probability bytes, the byte of fp16(acc + bias) from the table of all 65536 fp16 values */
                uint32_t r8[8];
                tmem_ld8(tcol, r8); tmem_ld_wait();
                release();
                if (row_ok) {
                    const size_t o = (size_t)n * a.e.co_real * Su + vo;
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        if (k < a.e.co_real) {
                            const float v = __fadd_rn(__uint_as_float(r8[k]), __ldg(a.e.bias + k));
                            if (EPI == 1) ((float *)a.e.y)[o + (size_t)k * Su] = v;
                            else if (EPI == 2) ((__half *)a.e.y)[o + (size_t)k * Su] = __float2half_rn(v);
                            else ((uint8_t *)a.e.y)[o + (size_t)k * Su] = __ldg(a.e.ptab + __half_as_ushort(__float2half_rn(v)));
                        }
                    }
                }
            } else if (EPI >= 3) {
                /* MX rows.  Column blocks of a transposed conv come as (dz, dy, block, dx): the two chunks of a job are the voxels 2 x and 2 x + 1 of one
                   output row (neighbours in the 16-byte-wide planes); without one they are two blocks of the same voxel */
                constexpr bool T = EPI == 4 || EPI == 6, O8 = EPI == 3 || EPI == 4;
                constexpr int NW = O8 ? 8 : 4;
                const size_t So = T ? (size_t)Su * 8 : (size_t)Su;
                int ob = cb; size_t vx = vo;
                if (T) {
                    const int pair = cb >> 1, zy = a.e.cob_t == 1 ? pair : pair / a.e.cob_t;
                    ob = a.e.cob_t == 1 ? 0 : pair - zy * a.e.cob_t;
                    const unsigned z = fast_div(vo, a.hw_mul, a.hw_shift), rem = vo - z * (unsigned)a.HW, oy = fast_div(rem, a.w_mul, a.w_shift), ox = rem - oy * (unsigned)a.W;
                    vx = ((size_t)(2 * z + (unsigned)(zy >> 1)) * (unsigned)(2 * a.e.H) + (2 * oy + (unsigned)(zy & 1))) * (unsigned)(2 * a.W) + 2 * ox;
                }
                const size_t blk = (size_t)n * a.e.nb_dst + a.e.b0 + ob;
                uint8_t *pc = (uint8_t *)a.e.y + (O8 ? (2 * blk * So + vx) * 16 : (blk * So + vx) * 16);
                uint8_t *ps = (uint8_t *)a.e.y + (size_t)a.N * a.e.nb_dst * So * (O8 ? 32 : 16) + blk * So + vx;
                unsigned w[2][NW], sb[2];
#pragma unroll
                for (int jc = 0; jc < 2; jc++) {
                    if (jc < nchunk) {
                        uint32_t rr[32];
                        tmem_ld32(tcol + (uint32_t)(jc * 32), rr); tmem_ld_wait();
                        if (jc == nchunk - 1) release();
                        const float4 *bp = (const float4 *)(a.e.bias + (T ? ob : cb + jc) * 32);
                        __half2 h[16];
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            const float4 b = __ldg(bp + k);
                            const float2 s0 = __fadd2_rn(make_float2(__uint_as_float(rr[4 * k]), __uint_as_float(rr[4 * k + 1])), make_float2(b.x, b.y));
                            const float2 s1 = __fadd2_rn(make_float2(__uint_as_float(rr[4 * k + 2]), __uint_as_float(rr[4 * k + 3])), make_float2(b.z, b.w));
                            h[2 * k] = __floats2half2_rn(s0.x, s0.y); h[2 * k + 1] = __floats2half2_rn(s1.x, s1.y);
                        }
                        if (O8) sb[jc] = mx_encode_row32_h8(h, w[jc]);
                        else {
                            float v[32];
#pragma unroll
                            for (int k = 0; k < 16; k++) { const float2 f = __half22float2(h[k]); v[2 * k] = f.x; v[2 * k + 1] = f.y; }
                            sb[jc] = mx_encode_row32<4>(v, w[jc]);
                        }
                        if (!T && row_ok) {
                            *(uint4 *)pc = make_uint4(w[jc][0], w[jc][1], w[jc][2], w[jc][3]);
                            if (O8) *(uint4 *)(pc + So * 16) = make_uint4(w[jc][4 % NW], w[jc][5 % NW], w[jc][6 % NW], w[jc][7 % NW]);
                            *ps = (uint8_t)sb[jc];
                            pc += So * (O8 ? 32 : 16); ps += So;
                        }
                    }
                }
                if (T && row_ok) {
                    st_32b(pc, w[0][0], w[0][1], w[0][2], w[0][3], w[1][0], w[1][1], w[1][2], w[1][3]);
                    if (O8) st_32b(pc + So * 16, w[0][4 % NW], w[0][5 % NW], w[0][6 % NW], w[0][7 % NW], w[1][4 % NW], w[1][5 % NW], w[1][6 % NW], w[1][7 % NW]);
                    *(unsigned short *)ps = (unsigned short)(sb[0] | (sb[1] << 8));
                }
            } else {
                const unsigned z = fast_div(vo, a.hw_mul, a.hw_shift), rem = vo - z * (unsigned)a.HW, oy = fast_div(rem, a.w_mul, a.w_shift);
                for (int jc = 0; jc < nchunk; jc++) {
                    uint32_t rr[32];
                    tmem_ld32(tcol + (uint32_t)(jc * 32), rr); tmem_ld_wait();
                    if (jc == nchunk - 1) release();
                    float v[32];
#pragma unroll
                    for (int k = 0; k < 32; k++) v[k] = __uint_as_float(rr[k]);
                    EpiArgs e = a.e;
                    if (EPI == 1) { e.out_mode = UMX_OUT_PM32; e.tconv = 0; }
                    if (EPI == 2) { e.out_mode = UMX_OUT_PM16; e.tconv = 0; }
                    /* the caller's order of a transposed conv's column blocks is (dz, dy, dx, block) */
                    const int pair = cb >> 1;
                    epi_chunk(e, n, (int)z, (int)oy, (int)(rem - oy * (unsigned)a.W), row_ok, e.tconv ? (2 * (pair / e.cob_t) + jc) * e.cob_t + pair % e.cob_t : cb + jc, v);
                }
            }
            slot += 2; if (slot >= NS) { slot = eg; sph ^= 1; }
            ntile += 2; while (ntile >= a.ntiles) { ntile -= a.ntiles; if (++tin == (int)a.rtiles_per_n) { tin = 0; n++; } }
        }
    }
    /* ---------------- teardown ---------------- */
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && warp == 0 && lane == 0) {
        for (int s = 0; s < R; s++) { const long long t0 = clock64(); while (!mbar_try(bar_tma + 8 * s, 0) && !mbar_try(bar_tma + 8 * s, 1) && clock64() - t0 < 20000000ll) { } }
        { const long long t0 = clock64(); while (!mbar_try(bar_w, 0) && clock64() - t0 < 20000000ll) { } }
    }
    if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem, (uint32_t)a.tmem_cols); }
}

/* Weight image of the streaming kernel: codes [column tile][K item][k half][row of the tile][16 B], then the B scale bytes in the TMEM
   scale layout per (column tile, stage of four K items, scale quad): byte (lane, column, id) = row 32 column + lane, K item 4 g + id
   (fp8) or item 4 g + 2 q + id / 2, block id % 2 (fp4).  Quantisation per (row, 32 input channels) as the reference's prep_w8_k /
   prep_w4_k (src/lp_f8fwd.cu:54-71, src/lp_f4fwd.cu:53-66).  One thread per (column tile, K item, row). */
__global__ void __launch_bounds__(128) prep_wp_k(const PrepArgs p, uint8_t *wp, int ntp, int ntiles, int ngroups, int w_codes) {
    const int total = ntiles * p.nki * ntp, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int rl = i % ntp, ki = (i / ntp) % p.nki, nt_i = i / (ntp * p.nki), row = nt_i * ntp + rl;
    const bool live = row < p.cop;
    /* a transposed conv's column blocks in the order (dz, dy, block, dx): see the epilogue */
    int src = row;
    if (p.kind == UMX_TCONV2) { const int pair = row >> 6, zy = pair / p.cob_t; src = ((2 * zy + ((row >> 5) & 1)) * p.cob_t + pair % p.cob_t) * 32 + (row & 31); }
    unsigned w[8]; unsigned sb[2] = {127u, 127u};
    float v[32];
    if (p.bits == 8) {
#pragma unroll
        for (int k = 0; k < 32; k++) v[k] = live ? prep_src(p, src, 0, ki, k) : 0.f;
        sb[0] = mx_encode_row32<8>(v, w);
    } else {
        unsigned w4[4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
#pragma unroll
            for (int k = 0; k < 32; k++) v[k] = live ? prep_src(p, src, 0, 2 * ki + h, k) : 0.f;
            sb[h] = mx_encode_row32<4>(v, w4);
#pragma unroll
            for (int t = 0; t < 4; t++) w[4 * h + t] = w4[t];
        }
    }
    if (!live) { sb[0] = 127u; sb[1] = 127u; }
    uint8_t *base = wp + ((size_t)(nt_i * p.nki + ki) * 2) * ntp * 16;
    *(uint4 *)(base + (size_t)rl * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    *(uint4 *)(base + (size_t)(ntp + rl) * 16) = make_uint4(w[4], w[5], w[6], w[7]);
    const int g = ki >> 2, j = ki & 3, l = rl & 31, c = rl >> 5, nq = p.bits == 8 ? 1 : 2;
    if (p.bits == 8) wp[w_codes + (size_t)((nt_i * ngroups + g) * nq) * 512 + l * 16 + c * 4 + j] = (uint8_t)sb[0];
    else { uint8_t *q = wp + w_codes + (size_t)((nt_i * ngroups + g) * nq + (j >> 1)) * 512 + l * 16 + c * 4 + (j & 1) * 2; q[0] = (uint8_t)sb[0]; q[1] = (uint8_t)sb[1]; }
}

}   // namespace

struct PGeo { int ntp, ntiles, ngroups, nq, w_codes, w_bytes; };
static int p_geometry(const umx_conv *c, PGeo *g) {
    if (c->kind == UMX_CONV3 || c->kind == UMX_CONV3S2) return 0;
    g->ntp = c->cop >= 64 ? 64 : 32; g->ntiles = (c->cop + g->ntp - 1) / g->ntp; g->ngroups = (c->nki + 3) / 4; g->nq = c->bits == 8 ? 1 : 2;
    g->w_codes = g->ntiles * c->nki * 2 * g->ntp * 16;
    g->w_bytes = g->w_codes + g->ntiles * g->ngroups * g->nq * 512;
    if (g->w_bytes > 150 * 1024) return 0;
    if (16 + g->ntiles * g->ngroups * g->nq * 4 + 2 * g->ntp > 512) return 0;
    return 1;
}
static void recip(unsigned d, unsigned *mul, int *shift) {
    int l = 0; while ((1ull << l) < d) l++;
    *mul = l ? (unsigned)(((1ull << (31 + l)) + d - 1) / d) : 0u; *shift = l - 1;
}
/* builds the weight image of the streaming kernel from device fp32 weights; NULL when the conv does not qualify */
uint8_t *umx_conv_p_prepare(const umx_conv *c, const float *w_dev) {
    PGeo g;
    if (!p_geometry(c, &g)) return nullptr;
    uint8_t *wp = (uint8_t *)nn_malloc((size_t)g.w_bytes);
    if (!wp) return nullptr;
    cudaMemset(wp, 127, (size_t)g.w_bytes);
    PrepArgs p; memset(&p, 0, sizeof p);
    p.w = w_dev; p.kind = c->kind; p.co = c->co; p.ci = c->ci; p.bits = c->bits; p.cop = c->cop; p.cob_t = c->cob_t; p.nkb = c->nkb; p.nki = c->nki; p.taps = 1;
    const int total = g.ntiles * c->nki * g.ntp;
    prep_wp_k<<<(total + 127) / 128, 128>>>(p, wp, g.ntp, g.ntiles, g.ngroups, g.w_codes);
    g_umx_launches++;
    return wp;
}
/* x: MX tensor (fp8 in the split layout).  Returns 1 when this kernel does not apply (the caller takes the general kernel), 0 after a
   launch, -1 on error. */
int umx_conv_fwd_p(const umx_conv *c, const void *x, const uint8_t *x_sc, void *enc_v, int N, int D, int H, int W, const EpiArgs &e) {
    typedef CUresult (*encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    PGeo g; ConvPArgs a; memset(&a, 0, sizeof a);
    const size_t S = (size_t)D * H * W;
    if (!c->wp || !p_geometry(c, &g) || (S & 15) || S > (size_t)1 << 30) return 1;
    if (e.out_mode == UMX_OUT_PROB8 && (e.co_real > 8 || g.ntiles != 1 || e.tconv || !e.ptab)) return 1;     /* the probability epilogue is the head's: one column tile, at most eight channels */       /* the scale plane's rows must be multiples of 16 bytes */
    a.N = N; a.nkb = c->nkb; a.nki = c->nki; a.bits = c->bits; a.cop = c->cop; a.ntp = g.ntp; a.ntiles = g.ntiles; a.ngroups = g.ngroups;
    a.S = (long long)S; a.rtiles_per_n = (long long)((S + 127) / 128); a.jobs = (long long)N * a.rtiles_per_n * g.ntiles; a.HW = H * W; a.W = W;
    recip((unsigned)(H * W), &a.hw_mul, &a.hw_shift); recip((unsigned)W, &a.w_mul, &a.w_shift);
    a.w_codes = g.w_codes; a.w_bytes = g.w_bytes; a.nquad = g.nq;
    a.sw_rows = c->bits == 8 ? 4 : 8;
    a.offSW = 4 * 4096; a.offSFA = a.offSW + 1024; a.stage_bytes = (a.offSFA + g.nq * 512 + 1023) & ~1023;
    a.off_w = 1024; a.off_ring = (a.off_w + a.w_bytes + 1023) & ~1023;
    const int sfb_cols = g.ntiles * g.ngroups * g.nq * 4;
    const int two = a.off_ring + 3 * a.stage_bytes <= 113 * 1024 && (256 - 16 - sfb_cols) / g.ntp >= 2;
    a.tmem_cols = two ? 256 : 512;
    a.nslot = (a.tmem_cols - 16 - sfb_cols) / g.ntp; if (a.nslot > kMaxSlotsP) a.nslot = kMaxSlotsP;
    a.nslot &= ~1;
    if (a.nslot < 2) return 1;
    a.sfa_base = a.nslot * g.ntp; a.sfb_base = a.sfa_base + 16;
    a.ring = ((two ? 113 : 227) * 1024 - a.off_ring) / a.stage_bytes; if (a.ring > 8) a.ring = 8;
    if (a.ring < 2) return 1;
    CUtensorMap m0, ms; memset(&m0, 0, sizeof m0); memset(&ms, 0, sizeof ms);
    const int planes = N * c->nkb * (c->bits == 8 ? 2 : 1);
    {
        const cuuint64_t gd[2] = {(cuuint64_t)S * 2, (cuuint64_t)planes}, gs[1] = {(cuuint64_t)S * 16};
        const cuuint32_t box[2] = {256, 2}, es[2] = {1, 1};
        if (((encode_fn)enc_v)(&m0, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, (void *)x, gd, gs, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return 1;
        /* samples as a dimension of their own: an MX-fp4 item's second block past the last one reads the fill, not the next sample's scales (whose NaN would come through the zero weights) */
        const cuuint64_t gd2[3] = {(cuuint64_t)S, (cuuint64_t)c->nkb, (cuuint64_t)N}, gs2[2] = {(cuuint64_t)S, (cuuint64_t)S * c->nkb};
        const cuuint32_t box2[3] = {128, (cuuint32_t)a.sw_rows, 1}, es2[3] = {1, 1, 1};
        if (((encode_fn)enc_v)(&ms, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, (void *)x_sc, gd2, gs2, box2, es2, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return 1;
    }
    a.wp = c->wp; a.e = e; a.err = umx_errflag();
    if (!a.err) return -1;
    int dev = 0, sms = 148; cudaGetDevice(&dev);
    { static int sms_of[16]; if (!sms_of[dev & 15]) { int v = 148; cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev); sms_of[dev & 15] = v; } sms = sms_of[dev & 15]; }   /* looked up once per device */
    static int attr_set[16];
    if (!attr_set[dev & 15]) {
        cudaError_t er = cudaSuccess;
#define UMX_P_ATTR(B, E) if (er == cudaSuccess) er = cudaFuncSetAttribute(conv_mxp_k<B, E>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024)
        UMX_P_ATTR(8, 0); UMX_P_ATTR(8, 1); UMX_P_ATTR(8, 2); UMX_P_ATTR(8, 3); UMX_P_ATTR(8, 4); UMX_P_ATTR(8, 5); UMX_P_ATTR(8, 6); UMX_P_ATTR(8, 7);
        UMX_P_ATTR(4, 0); UMX_P_ATTR(4, 1); UMX_P_ATTR(4, 2); UMX_P_ATTR(4, 3); UMX_P_ATTR(4, 4); UMX_P_ATTR(4, 5); UMX_P_ATTR(4, 6); UMX_P_ATTR(4, 7);
#undef UMX_P_ATTR
        if (er != cudaSuccess) { umx_latch("umx_conv_fwd: shared memory attribute", er); return -1; }
        attr_set[dev & 15] = 1;
    }
    const long long slots = (long long)sms * (two ? 2 : 1);
    const int grid = (int)(a.jobs < slots ? a.jobs : slots);
    const size_t smem = (size_t)a.off_ring + (size_t)a.ring * a.stage_bytes;
    int epi = 0;
    if (e.out_mode == UMX_OUT_PM32 && !e.tconv) epi = 1;
    else if (e.out_mode == UMX_OUT_PM16 && !e.tconv) epi = 2;
    /* the pair stores of the transposed conv want a 32-byte aligned tensor (its planes are multiples of 128 voxels); the scale plane then starts on an even address */
    else if (e.out_mode == UMX_OUT_MX && e.tconv && ((size_t)e.y & 31)) epi = 0;
    else if (e.out_mode == UMX_OUT_MX && e.out_bits == 8 && e.y_split) epi = e.tconv ? 4 : 3;
    else if (e.out_mode == UMX_OUT_MX && e.out_bits == 4) epi = e.tconv ? 6 : 5;
    else if (e.out_mode == UMX_OUT_PROB8) epi = 7;
#define UMX_P_GO(B, E) umx_launch(conv_mxp_k<B, E>, dim3(grid), dim3(kThreadsP), smem, m0, ms, a)
    if (c->bits == 8) { switch (epi) { case 1: UMX_P_GO(8, 1); break; case 2: UMX_P_GO(8, 2); break; case 3: UMX_P_GO(8, 3); break; case 4: UMX_P_GO(8, 4); break; case 5: UMX_P_GO(8, 5); break; case 6: UMX_P_GO(8, 6); break; case 7: UMX_P_GO(8, 7); break; default: UMX_P_GO(8, 0); } }
    else { switch (epi) { case 1: UMX_P_GO(4, 1); break; case 2: UMX_P_GO(4, 2); break; case 3: UMX_P_GO(4, 3); break; case 4: UMX_P_GO(4, 4); break; case 5: UMX_P_GO(4, 5); break; case 6: UMX_P_GO(4, 6); break; case 7: UMX_P_GO(4, 7); break; default: UMX_P_GO(4, 0); } }
#undef UMX_P_GO
    return 0;
}
