// Replays the per-lane row rings of the vertical cross-aggregation kernel
// (k_vert_views) on the host with the kernel's own constants (rts_vert_ring.h)
// and index arithmetic.  For every arm length of the fused path (0..23), strip
// start, strip height and image end, with the longest and with random arms, it
// checks that every slot read is inside the ring and holds the row it stands
// for, and that a walk covers every row of the arm within 64 mask bits.
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <random>
#include <vector>

#include "rts_vert_ring.h"

using namespace rts;

static int fail(const char *what, int L, int y0, int nrows, int tail, int y) {
    printf("FAIL %s: L=%d y0=%d rows=%d tail=%d y=%d\n", what, L, y0, nrows, tail, y);
    return 1;
}

int main() {
    std::mt19937 rng(7);
    for (int L = 0; L <= 23; L++) {
        const int DEP = vert_lane_depth(L), S = kVertStep;
        if (DEP % 4) return fail("depth", L, 0, 0, 0, 0);
        for (int y0 = 0; y0 <= L + 5; y0++)
            for (int nrows = 1; nrows <= 61; nrows += 6)
                for (int tail = 0; tail <= L + 2; tail += 1 + tail / 3)
                    for (int full = 0; full < 2; full++) {
                        const int y1 = y0 + nrows, H = y1 + tail;
                        const int ra = std::max(0, y0 - L), rb = std::min(H, y1 + L), n = rb - ra;
                        std::vector<int> held(DEP, -1000);  // row (from ra) in each slot
                        held[DEP - 1] = -1;                 // the running count before row ra
                        int ts = 0;
                        auto ingest = [&](int i) {
                            for (int k = 0; k < S; k++) held[ts + k] = S * i + k;
                            ts += S;
                            if (ts == DEP) ts = 0;
                        };
                        const int T0 = vert_lane_first(y0, ra, L);
                        int i = 0;
                        for (; i < T0 - 1; i++) ingest(i);
                        int sy = y0 - ra;
                        if (sy >= DEP) return fail("first slot", L, y0, nrows, tail, y0);
                        for (int s = 0; s < (nrows + S - 1) / S; s++, i++) {
                            ingest(i);
                            const int yr = y0 - ra + S * s, nj = std::min(S, nrows - S * s);
                            int t[4], b[4], lo = yr, hi = yr;
                            for (int j = 0; j < S; j++) {
                                const int y = y0 + S * s + j;
                                // rows past the image entered with empty arms
                                const int tm = yr + j < n ? std::min(L, y) : 0;
                                const int bm = yr + j < n ? std::min(L, H - 1 - y) : 0;
                                t[j] = full ? tm : (int)(rng() % (tm + 1));
                                b[j] = full ? bm : (int)(rng() % (bm + 1));
                                if (j < nj) {
                                    lo = std::min(lo, yr + j - (full ? tm : std::min(tm, t[j] + (int)(rng() % 3))));
                                    hi = std::max(hi, yr + j + (full ? bm : std::min(bm, b[j] + (int)(rng() % 3))));
                                }
                                int sl = sy + j;
                                sl = sl >= DEP ? sl - DEP : sl;
                                const uint32_t end = DEP * 32u, at = sl * 32u;
                                const uint32_t up = at + 32u * b[j], dn = at - 32u * t[j] - 32u;
                                const uint32_t oh = std::min(up, up - end), ol = std::min(dn, dn + end);
                                if (sl >= DEP || oh >= end || ol >= end) return fail("slot range", L, y0, nrows, tail, y);
                                if (j >= nj) continue;
                                if (held[sl] != yr + j) return fail("own row", L, y0, nrows, tail, y);
                                if (held[oh / 32] != yr + j + b[j]) return fail("bottom row", L, y0, nrows, tail, y);
                                if (held[ol / 32] != yr + j - t[j] - 1) return fail("row before", L, y0, nrows, tail, y);
                            }
                            const int base = lo & ~3;
                            if (base < 0) return fail("base", L, y0, nrows, tail, yr);
                            int g = sy - (yr - base);
                            g = (g < 0 ? g + DEP : g) >> 2;
                            const int ng = ((hi - base) >> 2) + 1;
                            if (ng > 16) return fail("walk above 64 rows", L, y0, nrows, tail, yr);
                            uint64_t seen[4] = {0, 0, 0, 0}, want[4] = {0, 0, 0, 0};
                            for (int q = 0; q < ng; q++) {
                                if (g < 0 || g >= DEP / 4) return fail("group range", L, y0, nrows, tail, yr);
                                for (int k = 0; k < 4; k++)
                                    for (int j = 0; j < nj; j++)
                                        if (held[4 * g + k] == base + 4 * q + k) seen[j] |= 1ull << (4 * q + k);
                                if (++g == DEP / 4) g = 0;
                            }
                            for (int j = 0; j < nj; j++) {
                                for (int r = yr + j - t[j]; r <= yr + j + b[j]; r++) want[j] |= 1ull << (r - base);
                                if ((seen[j] & want[j]) != want[j]) return fail("arm row", L, y0, nrows, tail, yr + j);
                            }
                            sy += S;
                            if (sy >= DEP) sy -= DEP;
                        }
                    }
        printf("L=%d depth=%d\n", L, DEP);
    }
    printf("ok\n");
    return 0;
}
