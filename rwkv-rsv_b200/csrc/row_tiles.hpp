// How the activation rows of a step are cut into tiles for the tensor-core linear layers (rows_linear.cuh).  Host arithmetic only, so that it can be checked on
// the CPU.
#pragma once
#include <cstddef>

namespace rsv {

enum RlFmt : int { RL_F16 = 0, RL_I8 = 1, RL_I8G = 2 };  // fp16; int8 with one (scale, zero) per row; int8 with one per row and group of 128
constexpr int kRlDigits = 4;
// columns an activation row takes in an operand tile
constexpr int rl_cols(int fmt) { return fmt == RL_F16 ? 2 : kRlDigits; }
// K elements in a 128-byte block
constexpr int rl_kelems(int fmt) { return fmt == RL_F16 ? 64 : 128; }

constexpr int kRlMaxRows = 64;    // activation rows of a tile with int8 weights, or few rows
constexpr int kRlMaxRowsF = 128;  // the same for fp16 weights and many rows (256 columns of operand either way)
constexpr int kRlMaxRowsG = 32;   // the same for per-group weights: two accumulators are in use, and fp32 sums in registers

// Row tiles of a step, of equal size: at most 64 activation rows each (32 with per-group int8 weights).  With fp16 weights alone and more
// than 128 rows a tile has up to 128: its two columns per row then fill the matrix instruction as four per row of 64 do, and the
// weights pass through L2 half as often.
struct RowTiles {
    int R = 0, rt = 0, n = 0, nt8 = 0, nt16 = 0;
    bool turns = false;  // cut for the persistent kernel (fit_turns): K is not split
    int nt(int fmt) const { return fmt == RL_F16 ? nt16 : nt8; }
    std::size_t image_bytes(int fmt, int K) const { return (std::size_t)n * ((K + rl_kelems(fmt) - 1) / rl_kelems(fmt)) * nt(fmt) * 128; }
};
inline RowTiles cut_rows(int R, int n) {
    RowTiles t;
    t.R = R;
    t.rt = (R + n - 1) / n;
    t.n = (R + t.rt - 1) / t.rt;
    t.nt8 = (t.rt * rl_cols(RL_I8) + 15) / 16 * 16;
    t.nt16 = (t.rt * rl_cols(RL_F16) + 15) / 16 * 16;
    return t;
}
inline RowTiles row_tiles(int R, bool per_group, bool int8) {
    const int most = per_group ? kRlMaxRowsG : int8 || R <= kRlMaxRowsF ? kRlMaxRows : kRlMaxRowsF;
    return cut_rows(R, (R + most - 1) / most);
}
// The row tiles of a launch with more tiles than SMs, which the persistent kernel takes in turns: `mt` weight tiles, at least `kb` blocks of K, fmt the format
// of most of them.  The widest tiles need the fewest turns; the cut with the fewest operand columns among those that need no more turns is taken, and the
// fewest tiles among equals.  A turn costs its K blocks' copies, less with narrower tiles, but the weight tiles' part of them and a tile's epilogue
// whatever its width: a turn more was never made up for by narrower ones.  Measured (2560 channels, exclusive time in the step):
//   512 int8 rows, att.output and ffn.value: 160 tiles of 64 rows in two turns 20.5 and 55 us, 260 of 40 in two 17 and 48, 300 of 35 in three 22 and 67;
//   1024 int8 rows, r, k, v and rank projections: 1056 tiles of 64 rows in eight turns 73 us, 1320 of 52 in nine 77;
//   512 fp16 rows, ffn.value: 80 tiles of 128 rows in one turn 60 us, 140 of 74 in one 50, 160 of 64 in two 88 (a CTA per tile: 85).
// Where one turn is enough but leaves more than a quarter of the SMs without a tile (ffn.key of 65 to 128 fp16 rows: 80 of 148), what counts is the neighbours, for
// whose CTAs two 64-row tiles per SM leave room in another way: ffn.value starts later behind the persistent kernel (128 rows 26 us instead of 24), a
// LayerNorm that does not fit beside the waiting CTAs of ffn.key any more starts earlier (13 us or 8).  A layer of a prompt of 97 and 128 rows takes 138 and 152 us
// with the persistent kernel and 137 and 150 without, one of 112 and 128 sessions 149.5 and 154 with and 152.5 and 157 without, 80 sessions the same.  So
// the wide tiles need a LayerNorm of more than 5 CTAs per 4 SMs (`before`: the CTAs of the kernel before, one per row and one per segment).
inline RowTiles fit_turns(const RowTiles& t, int mt, int kb, int fmt, int sms, int before) {
    if (t.n < 2 || fmt == RL_I8G || mt * t.n <= sms || kb < 16) return t;
    const int most = fmt == RL_F16 ? kRlMaxRowsF : kRlMaxRows, widest = (t.R + most - 1) / most;
    const int turns = (mt * widest + sms - 1) / sms;
    RowTiles best = cut_rows(t.R, widest);
    for (int n = widest + 1; mt * n <= turns * sms; ++n) {
        const RowTiles c = cut_rows(t.R, n);
        if (c.nt(fmt) < best.nt(fmt)) best = c;
    }
    if (turns == 1 && 4 * mt * best.n < 3 * sms && 4 * before <= 5 * sms) return t;
    best.turns = true;
    return best;
}

}  // namespace rsv
