/* The window of scale bytes that a stage of the z-marching conv gathers where TMA does not take the scale plane (rows that are no multiple of 16 bytes): 18 rows of 10 bytes of a
   block's plane, of each the three words that begin at its first byte, word i = 3 row + third; MX-fp4 has a second window (words 54 to 107) for the item's second block.  Also
   compiled by a host compiler, so that the addresses can be checked without a GPU. */
#pragma once
#include <stddef.h>
#include <stdint.h>
#ifdef __CUDACC__
#define UMX_HD __host__ __device__ __forceinline__
#else
#define UMX_HD inline
#endif

/* the bytes of word i (of one window, 0 to 53) that are wanted: inside the volume and the window's ten columns; (x0, y0): the window's first column and row */
UMX_HD uint32_t gather_keep(int i, int x0, int y0, int W, int H) {
    const int y = y0 + i / 3, x = x0 + i % 3 * 4;
    uint32_t keep = 0u;
    for (int t = 0; t < 4; t++) if (x + t >= 0 && x + t < W && i % 3 * 4 + t < 10) keep |= 0xffu << (8 * t);
    return y < 0 || y >= H ? 0u : keep;
}
/* the four bytes at q lie in two aligned words; one is read only where it has a wanted byte (mask m), and the last word of a plane that ends inside it byte by byte, so that nothing
   behind `end` is read.  The value is __funnelshift_r(w[0], w[1], w[2]) & w[3] once they have come.  load(const uint32_t *) and load(const uint8_t *) return the value. */
template <class Load>
UMX_HD void gather_word(const uint8_t *q, uint32_t m, const uint8_t *end, uint32_t *w, Load load) {
    const uint32_t sh = (uint32_t)(size_t)q & 3u;
    const uint8_t *p = q - sh;
    auto aligned = [&](const uint8_t *a) -> uint32_t {
        if (a + 4 <= end) return load((const uint32_t *)a);
        uint32_t v = 0u;
        for (int t = 0; t < 3; t++) if (a + t < end) v |= (uint32_t)load(a + t) << (8 * t);
        return v;
    };
    w[0] = m << (8 * sh) ? aligned(p) : 0u; w[1] = sh && m >> (32 - 8 * sh) ? aligned(p + 4) : 0u;
    w[2] = 8 * sh; w[3] = m;
}
