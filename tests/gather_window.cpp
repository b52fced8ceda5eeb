/* Every tile's gathered scale window of small volumes, lane by lane as the scale warp does it, against scale planes that end at their last byte: the bytes are the planes' (0 outside the
   volume), no load leaves them, and a lane has at most one word with bytes that come apart.  Planes of fewer
   than four voxels do not take this path. */
#include "gather_win.cuh"
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <vector>

static const uint8_t *lo, *hi;
static long bad;
struct Load {
    uint32_t operator()(const uint32_t *p) const {
        const uint8_t *b = (const uint8_t *)p;
        if (b < lo || b + 4 > hi || ((size_t)b & 3)) { bad++; return 0; }
        uint32_t v; memcpy(&v, b, 4);
        return v;
    }
    uint8_t operator()(const uint8_t *p) const { if (p < lo || p >= hi) { bad++; return 0; } return *p; }
};

int main() {
    long words = 0, wrong = 0, twice = 0, patched = 0;
    const int widths[] = {1, 2, 3, 5, 7, 8, 9, 11, 13, 17, 18, 21, 30, 31, 33}, heights[] = {1, 2, 3, 5, 16, 17, 18, 31};
    for (int W : widths) for (int H : heights) for (int D = 1; D <= 5; D += 2) for (int N = 1; N <= 3; N++) for (int nkb = 1; nkb <= 3; nkb++) for (int windows = 1; windows <= 2; windows++) {
        if (H * W < 4) continue;
        const size_t S = (size_t)D * H * W, n_all = S * N * nkb;
        std::vector<uint32_t> room(n_all / 4 + 2);                    /* word-aligned, as the codes before it make it */
        uint8_t *sc = (uint8_t *)room.data();
        for (size_t i = 0; i < n_all; i++) sc[i] = (uint8_t)(1 + rand() % 255);
        lo = sc; hi = sc + n_all;
        for (int n = 0; n < N; n++) for (int b = 0; b < nkb; b += windows) for (int z = 0; z < D; z++) {
            const int rest = gather_rest(N, nkb, D, H, W);
            uint32_t rest_b = 0;
            for (int t = 0; t < rest; t++) rest_b |= (uint32_t)hi[t - rest] << (8 * t);
            const bool two = windows == 2 && b + 1 < nkb, last = rest && n == N - 1 && z == D - 1 && b + windows >= nkb;
            const int w_last = windows == 2 && !(nkb & 1) ? 54 : 0;
            for (int y0 = -1; y0 < H; y0 += 16) for (int x0 = -1; x0 < W; x0 += 8) for (int lane = 0; lane < 32; lane++) {
                int patches = 0;
                for (int i = lane; i < 54 * windows; i += 32) {
                    const int j = i % 54;
                    const bool second = i >= 54;
                    const ptrdiff_t at = ((ptrdiff_t)n * nkb + b + second) * (ptrdiff_t)S + (ptrdiff_t)z * H * W + (ptrdiff_t)(y0 + j / 3) * W + x0 + j % 3 * 4;
                    const bool l = last && i / 54 * 54 == w_last;
                    const uint32_t m = gather_keep(j, x0, y0, W, H, l ? H * W - rest : H * W);
                    uint32_t w[4];
                    gather_word(sc + at, !second || two ? m : 0u, w, Load());
                    uint32_t v = (uint32_t)(((uint64_t)w[1] << 32 | w[0]) >> w[2]) & w[3];
                    bool has = false;
                    if (l) v |= gather_last(j, x0, y0, W, H, rest, rest_b, &has);
                    if (has) { patches++; patched++; }
                    for (int t = 0; t < 4; t++) {
                        const int x = x0 + j % 3 * 4 + t, y = y0 + j / 3;
                        const bool in = x >= 0 && x < W && y >= 0 && y < H && j % 3 * 4 + t < 10 && (!second || two);
                        if ((uint8_t)(v >> (8 * t)) != (in ? sc[at + t] : 0)) wrong++;
                    }
                    words++;
                }
                if (patches > 1) twice++;
            }
        }
    }
    printf("%ld words, %ld of them patched, %ld wrong bytes, %ld loads outside the planes, %ld lanes with several patches\n", words, patched, wrong, bad, twice);
    return wrong || bad || twice || !words || !patched;
}
