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
