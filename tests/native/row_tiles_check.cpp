// CPU check of csrc/row_tiles.hpp: the cuts of a launch with more tiles than SMs, over row counts, weight tiles and formats.
#include <algorithm>
#include <cstdio>

#include "row_tiles.hpp"

using namespace rsv;

static int bad = 0;
static void fail(const char* what, int R, int mt, int fmt, const RowTiles& c) {
    if (++bad <= 20) std::printf("%s: %d rows, %d weight tiles, format %d -> %d tiles of %d rows\n", what, R, mt, fmt, c.n, c.rt);
}

int main() {
    for (int sms : {148, 132})
        for (int fmt : {RL_F16, RL_I8, RL_I8G})
            for (int mt : {1, 4, 8, 16, 20, 32, 48, 66, 80, 100, 112, 128, 147, 148, 149, 200, 512})
                for (int R = 1; R <= 2300; ++R) {
                    const int most = fmt == RL_F16 ? kRlMaxRowsF : fmt == RL_I8 ? kRlMaxRows : kRlMaxRowsG;
                    const RowTiles wide = cut_rows(R, (R + most - 1) / most);
                    auto turns = [&](const RowTiles& c) { return (mt * c.n + sms - 1) / sms; };
                    for (int k = 0; k < 4; ++k) {  // the two base cuts of a step (wide and narrow layers), one segment or one per row
                        const int before = k & 2 ? 2 * R : R + 1;
                        const RowTiles t = row_tiles(R, fmt == RL_I8G, (k & 1) || fmt == RL_I8), c = fit_turns(t, mt, 16, fmt, sms, before);
                        // every row in one tile, no empty tile, tiles the kernel has room for
                        if (c.R != R || (c.n - 1) * c.rt >= R || c.n * c.rt < R || c.rt > most || c.rt < 1) fail("not a cut", R, mt, fmt, c);
                        if (c.nt8 < 4 * c.rt || c.nt16 < 2 * c.rt || c.nt8 % 16 || c.nt16 % 16 || c.nt(fmt) > 256) fail("operand columns", R, mt, fmt, c);
                        if (!c.turns) {
                            if (c.n != t.n || c.rt != t.rt) fail("cut again for another kernel", R, mt, fmt, c);
                            continue;
                        }
                        if (fmt == RL_I8G || mt * t.n <= sms) fail("no turns to cut for", R, mt, fmt, c);
                        if (turns(c) > turns(wide)) fail("more turns than the widest tiles need", R, mt, fmt, c);
                        if (c.nt(fmt) > wide.nt(fmt)) fail("wider than the widest", R, mt, fmt, c);
                        if (turns(c) == 1 && 4 * mt * c.n < 3 * sms && 4 * before <= 5 * sms) fail("one turn, and SMs without a tile", R, mt, fmt, c);
                        // as narrow as the turns allow
                        for (int n = c.n + 1; mt * n <= sms * turns(wide); ++n)
                            if (cut_rows(R, n).nt(fmt) < c.nt(fmt)) {
                                fail("a narrower cut has as many turns", R, mt, fmt, c);
                                break;
                            }
                    }
                    if (fit_turns(row_tiles(R, false, true), mt, 15, fmt, sms, 1).turns) fail("short K", R, mt, fmt, wide);
                }
    if (bad) {
        std::printf("%d failures\n", bad);
        return 1;
    }
    std::puts("row tiles ok");
    return 0;
}
