/* The window of scale bytes that a stage of the z-marching conv gathers where TMA does not take the scale plane (rows that are no multiple of 16 bytes): 18 rows of 10 bytes of a
   block's plane, of each the three words that begin at its first byte, word i = 3 row + third; MX-fp4 has a second window (words 54 to 107) for the item's second block.  A word is put
   together from the two aligned words it lies in.  Also compiled by a host compiler, so that the addresses can be checked without a GPU.

   The scale bytes of all samples and blocks end where the tensor ends: unless their number is a multiple of four, the aligned word around the last one to three of them reaches behind
   it and is read byte by byte, in instances of their own (ENDS), in the planes where it may come up.  Anything more in the scale warp's program costs a launch: 32 -> 32 in MX-fp4 on
   63 x 61 x 66 (which ends inside a word) 14.4 us without care for the end, 15.3 this way, 16.2 with the bytes loaded ahead and put in, 17.1 with every word checked. */
#pragma once
#include <stddef.h>
#include <stdint.h>
#ifdef __CUDACC__
#define UMX_HD __host__ __device__ __forceinline__
#else
#define UMX_HD inline
#endif

/* whether the scale bytes end inside a word */
UMX_HD bool gather_ends(int N, int nkb, int D, int H, int W) { return (unsigned)N * (unsigned)nkb * (unsigned)D * (unsigned)H * (unsigned)W & 3u; }
/* the first z plane of sample n with a word that may reach behind the end of all scale bytes (D: none has): the last sample's last plane, or more of them where a plane or a block has fewer
   than three bytes */
UMX_HD int gather_tail(int n, int N, int D, int H, int W) {
    if ((size_t)D * H * W < 3) return 0;
    return n < N - 1 ? D : (size_t)H * W < 3 ? 0 : D - 1;
}
/* the bytes of word i (of one window, 0 to 53) that are wanted: inside the volume and the window's ten columns; (x0, y0): the window's first column and row */
UMX_HD uint32_t gather_keep(int i, int x0, int y0, int W, int H) {
    const int y = y0 + i / 3, x = x0 + i % 3 * 4;
    uint32_t keep = 0u;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int t = 0; t < 4; t++) if (x + t >= 0 && x + t < W && i % 3 * 4 + t < 10) keep |= 0xffu << (8 * t);
    return y < 0 || y >= H ? 0u : keep;
}
/* the four bytes at q, masked: an aligned word is read only where it has a byte of m, and byte by byte where it ends behind `end` (TAIL; otherwise none does).  The value is
   __funnelshift_r(w[0], w[1], w[2]) & w[3] once they have come. */
template <bool TAIL, class Load>
UMX_HD void gather_word(const uint8_t *q, uint32_t m, const uint8_t *end, uint32_t *w, Load load) {
    const uint32_t sh = (uint32_t)(size_t)q & 3u;
    const uint8_t *p = q - sh;
    auto aligned = [&](const uint8_t *a) -> uint32_t {
        if (!TAIL || a + 4 <= end) return load((const uint32_t *)a);
        uint32_t v = 0u;
#ifdef __CUDACC__
#pragma unroll 1
#endif
        for (int t = 0; t < 3; t++) if (a + t < end) v |= (uint32_t)load(a + t) << (8 * t);
        return v;
    };
    w[0] = m << (8 * sh) ? aligned(p) : 0u; w[1] = sh && m >> (32 - 8 * sh) ? aligned(p + 4) : 0u;
    w[2] = 8 * sh; w[3] = m;
}
