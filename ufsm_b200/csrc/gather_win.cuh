/* The window of scale bytes that a stage of the z-marching conv gathers where TMA does not take the scale plane (rows that are no multiple of 16 bytes): 18 rows of 10 bytes of a
   block's plane, of each the three words that begin at its first byte, word i = 3 row + third; MX-fp4 has a second window (words 54 to 107) for the item's second block.  A word is put
   together from the two aligned words it lies in.  Also compiled by a host compiler, so that the addresses can be checked without a GPU.

   The scale bytes of all samples and blocks end where the tensor ends, at any address: an aligned word around the last one to three of them would reach behind it.  Those bytes come once,
   at the kernel's start, and the stage they belong to (the last sample's last block and plane) leaves them out of its words and puts them in on its own. */
#pragma once
#include <stddef.h>
#include <stdint.h>
#ifdef __CUDACC__
#define UMX_HD __host__ __device__ __forceinline__
#else
#define UMX_HD inline
#endif

/* how many of the bytes lie in a word that ends behind the last one */
UMX_HD int gather_rest(int N, int nkb, int D, int H, int W) { return (int)((unsigned)N * (unsigned)nkb * (unsigned)D * (unsigned)H * (unsigned)W & 3u); }
/* the bytes of word i (of one window, 0 to 53) that are wanted: inside the volume and the window's ten columns, of voxels (y W + x) before `limit`; (x0, y0): the window's first column and
   row */
UMX_HD uint32_t gather_keep(int i, int x0, int y0, int W, int H, int limit) {
    const int y = y0 + i / 3, x = x0 + i % 3 * 4, most = limit - y * W;
    const int hi = most < W ? most : W;
    uint32_t keep = 0u;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int t = 0; t < 4; t++) if (x + t >= 0 && x + t < hi && i % 3 * 4 + t < 10) keep |= 0xffu << (8 * t);
    return y < 0 || y >= H ? 0u : keep;
}
/* the four bytes at q, masked: an aligned word is read only where it has a byte of m.  The value is __funnelshift_r(w[0], w[1], w[2]) & w[3] once they have come. */
template <class Load>
UMX_HD void gather_word(const uint8_t *q, uint32_t m, uint32_t *w, Load load) {
    const uint32_t sh = (uint32_t)(size_t)q & 3u;
    const uint32_t *p = (const uint32_t *)(q - sh);
    w[0] = m << (8 * sh) ? load(p) : 0u; w[1] = sh && m >> (32 - 8 * sh) ? load(p + 1) : 0u;
    w[2] = 8 * sh; w[3] = m;
}
/* word i's share of the last `rest` bytes (`bytes`, the first in bits 0 to 7): the word's bytes with them in their places; *has: it has any */
UMX_HD uint32_t gather_last(int i, int x0, int y0, int W, int H, int rest, uint32_t bytes, bool *has) {
    const int first = H * W - rest;
    const uint32_t m = gather_keep(i, x0, y0, W, H, H * W) & ~gather_keep(i, x0, y0, W, H, first);
    const int at = first - ((y0 + i / 3) * W + x0 + i % 3 * 4);      /* place of the first of them, counted from the word's first byte */
    *has = m != 0u;
    return (at >= 0 ? bytes << (8 * (at & 3)) : bytes >> (8 * (-at & 3))) & m;
}
