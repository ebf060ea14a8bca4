// Which form of a many-row kernel a launch takes, where two forms give the same bits: plain functions of sizes, so that a host can check the lines.
// Figures: us a launch with events between the launches, 148 multiprocessors.
#pragma once

// The combine of a call's ranks (sz_moe_rows.cuh): a warp a (row, 128 outputs), or a warp a rank for 512 outputs of a row.  The first one adds
// eleven ranks in three rounds of four, one after the other; the second has them side by side and meets in shared memory.  Only
// where the rounds are full and the outputs many, or some but all of them at work at once (two blocks a multiprocessor), is the first one sooner (second / first, 10
// experts a row of 2,048: 504 rows 41.9 / 37.1, 256 26.6 / 24.6, 208 23.8 / 23.0, 192 22.5 / 24.1, 160 20.5 / 22.5, 136 20.4 / 18.5, 80 the same 16.4, 8 - whose
// sums are cut over many blocks' parts - 12.3 / 18.4; of 1,024: 504 28.7 / 25.6, 352 23.4 / 24.6, 288 20.5 / 19.3, 136 13.0 / 16.5).  With 8 experts a row its third
// round is a single rank: 504 rows 30.8 / 34.9, 136 16.5 / 18.3.
static inline bool sz_rows_combine_by_warp(int live, int hidden, int top_k, int sms) {
    const int items = live * (hidden / 512);         // pieces of 512 outputs; two a block of the first form
    return top_k >= 10 && (items >= 832 || (items >= 480 && items / 2 <= 2 * sms));
}

// The router over more than 128 rows: the pass's kernel with a block row for 8 rows (its last blocks choose), or the logits as tiles on the f64 tensor
// instructions and a kernel that chooses - in tiles of 16 x 16, for 1,025 .. 2,048 columns also 32 x 32 or 32 x 64 (router rows x rows; up
// to 1,024 the larger ones were sooner nowhere: 513 router rows, 504 rows: 37 each; beyond 2,048 they do not fit shared memory).  Up to 128 rows the
// pass's.  Each form's time in tenths of us, from runs of all of them at 17 .. 1,001 router rows x 136 .. 504 rows x 512 .. 4,096 columns; an estimate is
// within a tenth of its measurement.
//   pass  by how many groups of 4 router rows a block takes one after the other (wider than 2,048 columns, by its blocks: a group a block)
//   tiles by waves of a block a multiprocessor, and 8 us of the kernel that chooses
// (2,048 columns, 513 router rows, pass / best tiles: 136 rows 37 / 31 + 8, 200 47 / 32 + 8, 256 57 / 38 + 8, 504 98 / 59 + 8; 129 router rows: 136 20 / 20 + 8, 504 35 /
// 27 + 8; 17: 504 17 / 21 + 8; 1,024 columns, 513: 136 31 / 18 + 8, 504 76 / 37 + 8; 4,096 columns, 17: 136 28 / 44 + 8, 256 36 / 45 + 8; 129: 256 80 / 46 + 8.)
enum { SZ_ROUTE_PASS, SZ_ROUTE_16x16, SZ_ROUTE_32x32, SZ_ROUTE_32x64 };
// blocks of the pass's kernel that share the router rows of 8 rows: about one a multiprocessor over all of them (wider rows do not stay in registers as f64: a block a group)
static inline int sz_route_pass_blocks(int groups, int chunks, int hidden, int sms) {
    const int gx = sms / chunks < 1 ? 1 : sms / chunks;
    return hidden > 2048 || gx > groups ? groups : gx;
}
static inline int sz_route_rows_form(int route_rows, int rows, int live, int hidden, int sms) {
    if (live <= 128) return SZ_ROUTE_PASS;
    auto waves = [&](int e, int r) { return ((route_rows + e - 1) / e * ((live + r - 1) / r) + sms - 1) / sms; };
    const int groups = (route_rows + 3) / 4, chunks = rows / 8, gx = sz_route_pass_blocks(groups, chunks, hidden, sms), in_turn = (groups + gx - 1) / gx;
    const int w = waves(16, 16);
    int pass, small, mid = 1 << 30, large = 1 << 30;
    if (hidden <= 1024) { pass = 130 + 19 * in_turn / 2; small = 85 + 37 * w; }
    else if (hidden <= 2048) {      // (three blocks of the smallest tiles a multiprocessor)
        pass = 140 + 132 * in_turn / 10; small = 225 * ((w - 1) / 3) + (w % 3 == 1 ? 205 : w % 3 == 2 ? 265 : 315); mid = 60 + 320 * waves(32, 32); large = 50 + 540 * waves(32, 64);
    } else { pass = 240 + (int)(groups * chunks * 148ll / sms / 2); small = 150 + 293 * w; }
    const int best = small <= mid && small <= large ? small : mid <= large ? mid : large;
    return best + 80 >= pass ? SZ_ROUTE_PASS : best == small ? SZ_ROUTE_16x16 : best == mid ? SZ_ROUTE_32x32 : SZ_ROUTE_32x64;
}

// Attention of a step's groups of two query tiles, heads of 256 (sz_attn2_kernel), by the blocks that have positions: blocks of four warps, two a multiprocessor, or of eight, one a
// multiprocessor.  Four win where blocks queue; where each has a multiprocessor of its own, eight do it sooner (eight / four: 1 sequence of 4 rows at 24,000
// positions, 128 blocks, 30.8 / 36.8; 2, 256 blocks, 55 / 47; at 8,000 2 of them, 128 blocks, 24.4 / 28.6; 3, 192 blocks, 41 / 34; 32 at 200, 128 blocks,
// 17.4 / 20.4) - a step of few sequences, and the last rows of a prompt.
static inline bool sz_attn_four_warps(int blocks, int sms) { return blocks > sms; }

// The Q8_0 projections over many rows (sz_dense_rows_q8_kernel): units of 16 matrix rows -> warps a block (a unit each), groups of 8 rows a block, blocks
// that share the columns.  Blocks of 8 units and 32 rows where they are as many as the multiprocessors; else of 4 and 16, or of 4 and 8 where those, too, are
// fewer than the multiprocessors.  As long as three of them fit a multiprocessor two share the columns, or four (us a launch from memory, blocks of 16 rows alone / in
// two, of 8 rows in two / in four: 2,048 x 4,096, 80 rows 37 / 29, 42 / 41; 24 rows 29 / 21, 21 / 17; 8 rows 29 / 21, 19 / 13).  Where blocks of 8 rows in two would be
// more than that, those of 16 share (9,216 x 2,048, 16 rows: 18.9 / 16.9, 20.7 / 26.4; 4,096 x 1,024, 32 rows 12.7 / 12.8, 14.8 / 16.9).  Of 512 columns, four
// stages, only blocks that are few do (1,024 rows, 32 rows: 10.7 / 9.5, 8.7 / 8.7; 8,192, 8 rows: 8.8 / 10.7, 10.7 / 10.7).
struct SzDenseRowsForm { int warps, groups, share; };
static inline SzDenseRowsForm sz_dense_rows_form(int units, int rows, int cols, int sms) {
    auto blocks = [&](int nw, int ng) { return (units + nw - 1) / nw * ((rows + 8 * ng - 1) / (8 * ng)); };
    if (blocks(8, 4) >= sms) return {8, 4, 1};
    if (blocks(4, 2) > sms * 3 / 2 || (cols <= 512 && blocks(4, 1) * 4 > sms * 2)) return {4, 2, 1};
    if (blocks(4, 2) >= sms || blocks(4, 1) * 2 > sms * 3) return {4, 2, 2};      // (a part of the columns has to be whole stages: cols is a multiple of 256)
    if (cols % 512 || blocks(4, 1) * 4 > sms * 3) return {4, 1, 2};
    return {4, 1, 4};
}
