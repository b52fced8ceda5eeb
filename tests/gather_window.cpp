/* Every tile's gathered scale window of small volumes, word by word as the kernel's lanes do it, against a plane that ends at its last byte: the bytes are the plane's (0 outside the
   volume), and no load leaves the plane. */
#include "gather_win.cuh"
#include <stdio.h>
#include <stdlib.h>
#include <vector>

static const uint8_t *lo, *hi;
static long bad;
struct Load {
    uint32_t operator()(const uint32_t *p) const {
        const uint8_t *b = (const uint8_t *)p;
        if (b < lo || b + 4 > hi || ((size_t)b & 3)) { bad++; return 0; }
        return (uint32_t)b[0] | (uint32_t)b[1] << 8 | (uint32_t)b[2] << 16 | (uint32_t)b[3] << 24;
    }
    uint8_t operator()(const uint8_t *p) const { if (p < lo || p >= hi) { bad++; return 0; } return *p; }
};

int main() {
    long words = 0, wrong = 0;
    const int widths[] = {1, 2, 3, 5, 7, 8, 9, 11, 13, 17, 18, 21, 30, 31, 33}, heights[] = {1, 2, 3, 5, 16, 17, 18, 31};
    for (int W : widths) for (int H : heights) for (int D = 1; D <= 5; D += 2) for (int blocks = 1; blocks <= 3; blocks++) {
        const size_t S = (size_t)D * H * W, n = S * blocks;
        std::vector<uint32_t> room(n / 4 + 2);                    /* word-aligned, as the codes before it make it */
        uint8_t *sc = (uint8_t *)room.data();
        for (size_t i = 0; i < n; i++) sc[i] = (uint8_t)(1 + rand() % 255);
        lo = sc; hi = sc + n;
        for (int per = 1; per <= blocks; per++) if (blocks % per == 0)      /* blocks a sample */
        for (int b = 0; b < blocks; b++) for (int z = 0; z < D; z++)
            for (int y0 = -1; y0 < H; y0 += 16) for (int x0 = -1; x0 < W; x0 += 8) for (int i = 0; i < 54; i++) {
                const uint32_t m = gather_keep(i, x0, y0, W, H);
                uint32_t w[4];
                const uint8_t *q = sc + (ptrdiff_t)b * S + (ptrdiff_t)z * H * W + (ptrdiff_t)(y0 + i / 3) * W + x0 + i % 3 * 4;
                if (!gather_ends(blocks / per, per, D, H, W) || z < gather_tail(b / per, blocks / per, D, H, W)) gather_word<false>(q, m, hi, w, Load()); else gather_word<true>(q, m, hi, w, Load());
                const uint32_t v = (uint32_t)(((uint64_t)w[1] << 32 | w[0]) >> w[2]) & w[3];
                for (int t = 0; t < 4; t++) {
                    const int x = x0 + i % 3 * 4 + t, y = y0 + i / 3;
                    const bool in = x >= 0 && x < W && y >= 0 && y < H && i % 3 * 4 + t < 10;
                    const uint8_t want = in ? sc[b * S + ((size_t)z * H + y) * W + x] : 0;
                    if ((uint8_t)(v >> (8 * t)) != want) wrong++;
                }
                words++;
            }
    }
    printf("%ld words, %ld wrong bytes, %ld loads outside the plane\n", words, wrong, bad);
    return wrong || bad || !words;
}
