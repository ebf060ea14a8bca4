// The MoE sublayer over MANY rows (a prompt chunk, or the verify rows of many sequences): what sz_moe_verify computes for up to 8
// rows, for up to SZ_ROWS_CAP, with every expert's matrices decoded ONCE for (almost) all the rows that chose it.  The role of the
// reference's grouped experts of a long prompt (device planner plan_scan_w / plan_fill_w, kernels/forward.cu:3234-3319; mma_grouped*,
// kernels/matvec.cu:1190-1260; EXL3 exl3_mma, kernels/exl3.cu:500-590) with this library's exact arithmetic.
//
//   route     sz_route_kernel with a second grid dimension, 8 rows a block row, or sz_route_rows_kernel and sz_route_topk_kernel: a verify pass's logits and choice
//   plan      sz_rows_plan_kernel: every expert's pairs in ascending row order side by side (a pair's place is its SLOT), cut into
//             groups of up to 16; the shared expert's groups (16 consecutive rows each) are spread evenly among them
//   gate/up   sz_rows_gateup_kernel: a persistent launch over all groups
//   act       sz_rows_act_kernel: SwiGLU of every pair, left as the down product's operand fragments
//   down      sz_rows_down_kernel: as gate/up, over those fragments
//   combine   sz_rows_combine_ranks_kernel, sz_rows_combine_kernel: an output's ranks' terms in rank order, as sz_x3_combine_kernel adds them
// A pair's numbers do not depend on which rows share its group (every row of a group is a column of its own in the tensor-core
// product, the sums over column blocks are integer): a row's output is bit for bit what sz_moe_verify gives for it.
//
// What bounds the expert kernels is the trellis decode (some 60 cycles a tile of 256 weights and scheduler, sz_xw_afrag), so a group
// takes up to 16 rows: the second eight cost two more tensor-core instructions a tile, a group of their own the whole decode.  256
// rows of the benchmark's layer (512 experts, top 10) are some 540 groups.  Units - (group, matrix, 512 outputs, 128 inputs) - are
// shared out contiguously over one block a multiprocessor, by what they cost (sz_rows_weight), whatever the routing, with the inputs fastest: a consumer
// warp adds the units of one ITEM (the same group and outputs) up in 64-bit registers and stores the finished f32 sums; only where a
// block's share begins or ends inside an item do its parts go to a side buffer, as integers, for the reader to add - no atomics and
// nothing to clear.  (The form before it launched a window of 80 groups as a block row of the verify pass's kernels: 3 units a block
// where 2.7 would have been even, 1.35 of 2 in the down matrices, 63 M atomics into sums that had to be zeroed first, and launches
// of their own for the shared expert.)
#pragma once
#include "sz_moe.cuh"
#include "sz_moe_exl3w.cuh"

#define SZ_ROWS_MAX 256           // rows a call of sz_moe_rows (a multiple of 8)
#define SZ_ROWS_CAP 512           // rows the plan holds (a prompt's chunk inside a session)
#define SZ_ROWS_G 16              // rows a group
#define SZ_ROWS_MAXG (SZ_MAX_EXPERTS + SZ_ROWS_CAP * SZ_MAX_TOPK / SZ_ROWS_G + SZ_ROWS_CAP / SZ_ROWS_G)
#define SZ_ROWS_MAXB 256          // blocks of the expert kernels (one a multiprocessor)
#define SZ_ROWS_PAIRS (SZ_ROWS_CAP * (SZ_MAX_TOPK + 1))

struct SzRowsPlan {
    int32_t n_groups, overflow, pad[2];
    int32_t first[SZ_ROWS_MAXG];        // the group's first slot
    int16_t expert[SZ_ROWS_MAXG];       // -1: the shared expert
    int16_t count[SZ_ROWS_MAXG];
    int16_t row[SZ_ROWS_PAIRS];         // slot -> input row
    int32_t group[SZ_ROWS_PAIRS];       // slot -> its group
    int32_t pair_loc[SZ_ROWS_PAIRS];    // pair (row * top_k + rank; then the rows of the shared expert) -> slot
    // the blocks' shares of the gate / up units [0] and of the down units [1]: block b works on [start[b], start[b + 1]); and for every
    // item the first and the last block that works on it (low and high half)
    int32_t start[2][SZ_ROWS_MAXB + 1];
    u32 gu_blocks[SZ_ROWS_MAXG][2], dn_blocks[SZ_ROWS_MAXG][8];
};
// What a unit of a group of n rows costs: the decode, a row's fragments, the second eight rows' products.  Least squares over the blocks of gate / up
// launches of 8 .. 256 rows (cycles; 2,048 x 512, 512 experts): 2 bits 4,707 + 22.7 a row up to eight, 5,848 + 18.9 beyond; 3 bits 4,696 + 26.2 and
// 5,901 + 15.2; 4 bits 4,679 + 25.7 and 5,902 + 17.8 (0.5 % rms of a block); 4,096 x 512, 64 experts, 3 bits: 4,774 + 23.0 and 5,853 + 18.6; 2,048 x 256, whose
// units are half as large, 2,995 + 23.0 and 3,687 + 15.7 - the same proportions, which is all that counts.  Down's rows are copied, not made: 4,937 + 4.6 and 5,899 + 6.1
// (3 bits), so a group beyond eight is 1.20 of a small one where the weights say 1.27: its blocks end within 96 - 98 % of the last one's time on average, gate /
// up's within 98; weights of its own (1.17) changed down by -3 .. +2 %, none (no term a row) by under 1 %.
__device__ __forceinline__ int sz_rows_weight(int n) { return n <= 8 ? 172 + n : 218 + n / 2; }

// ---- plan: one block of 1024 threads ---------------------------------------------------------------------------------------------------
// Every (row, rank) pair marks its row in its expert's row mask; an expert's pairs in ascending row order are then the set bits of
// its mask, and a pair's place among them the number of set bits below its row: no sorting, no order of arrival.  Slots and groups
// are prefix sums over the experts, one a thread.  Dynamic shared memory: the masks, and the set bits before every word of them, a word an entry of
// padding behind an expert's (sz_rows_plan_smem).
// One block whose 32 warps wait for shared memory most of the time, so what counts is how often they go there one after the other: a pair's place
// is one count and one word (counting its expert's words one by one, two banks for all experts, took 20,600 of 51,000 cycles at 504 rows), and the
// block that an item falls to is guessed from its weight and put right (two binary searches an item: 16,400).  With the events around it, 512 experts: 504 rows 33 -> 25 us,
// 256 25 -> 19, 96 18 -> 14, 8 12 -> 10.  (The loops over a thread's pairs end with the call's: all of them made a division each, 2 us where pairs are few.)
#define SZ_ROWS_MW (SZ_ROWS_CAP / 32 + 1)       // words of an expert's mask (odd: experts in different banks)
static inline size_t sz_rows_plan_smem(int experts) { return (size_t)experts * SZ_ROWS_MW * 6; }
__global__ void __launch_bounds__(1024)
sz_rows_plan_kernel(const int32_t* __restrict__ ridx, int R, int k, int ne, int has_shared, int upg_gu, int ns, int upg_dn, int kb, int grid,
                    SzRowsPlan* __restrict__ P, u32* __restrict__ err) {
    extern __shared__ u32 mask[];
    u16* pre = (u16*)(mask + (size_t)ne * SZ_ROWS_MW);
    __shared__ int slot_of[SZ_MAX_EXPERTS], grp_of[SZ_MAX_EXPERTS];
    __shared__ int wsum[2][32];
    __shared__ int before[SZ_ROWS_MAXG + 1];        // a group's weight, then the weights before it
    __shared__ int bs[2][SZ_ROWS_MAXB + 1];
    constexpr int MW = SZ_ROWS_MW, NP = SZ_ROWS_CAP * SZ_MAX_TOPK / 1024;      // pairs a thread, at most
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, pairs = R * k;
    const int words = (R + 31) / 32;
    for (int i = t; i < ne * MW; i += 1024) mask[i] = 0u;
    sz_pdl_wait();
    sz_pdl_trigger();
    int pe[NP];                 // the pairs' experts, asked for at once
#pragma unroll
    for (int i = 0; i < NP; i++) pe[i] = t + 1024 * i < pairs ? __ldcg(ridx + t + 1024 * i) : -1;
    if (t == 0) P->overflow = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NP; i++) {
        if (1024 * i >= pairs) break;
        const int row = (t + 1024 * i) / k;
        if ((unsigned)pe[i] >= (unsigned)ne) continue;     // (a routing that was never written: caught below, nothing is touched)
        atomicOr(&mask[pe[i] * MW + (row >> 5)], 1u << (row & 31));
    }
    __syncthreads();
    int c = 0;
    if (t < ne)
        for (int q = 0; q < words; q++) { pre[t * MW + q] = (u16)c; c += __popc(mask[t * MW + q]); }
    const int ng = (c + SZ_ROWS_G - 1) / SZ_ROWS_G;
    int sc = c, sg = ng;                                // inclusive sums over the warp, then over the warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, sc, o), b = __shfl_up_sync(0xffffffffu, sg, o);
        if (lane >= o) { sc += a; sg += b; }
    }
    if (lane == 31) { wsum[0][warp] = sc; wsum[1][warp] = sg; }
    __syncthreads();
    if (warp == 0) {
        int a = wsum[0][lane], b = wsum[1][lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) { a += x; b += y; }
        }
        wsum[0][lane] = a; wsum[1][lane] = b;
    }
    __syncthreads();
    const int shg = has_shared ? (R + SZ_ROWS_G - 1) / SZ_ROWS_G : 0;
    const int s0 = sc - c + (warp ? wsum[0][warp - 1] : 0), g0 = sg - ng + (warp ? wsum[1][warp - 1] : 0), total = wsum[1][31];
    // a full group costs more than an expert's few rows: one of the shared expert's before every `every` others, so that the blocks'
    // equal shares of the groups are equal work (in front of the others they made four blocks of 148 a seventh late)
    const int every = shg > 0 ? (total / shg > 1 ? total / shg : 1) : 1;
    auto place = [&](int q) { return q + (shg > 0 ? (q / every + 1 < shg ? q / every + 1 : shg) : 0); };
    if (t < ne) {
        slot_of[t] = s0; grp_of[t] = g0;
        for (int q = 0; q < ng; q++) {
            const int at = place(g0 + q);
            P->first[at] = s0 + q * SZ_ROWS_G;
            P->expert[at] = (int16_t)t;
            const int n = c - q * SZ_ROWS_G < SZ_ROWS_G ? c - q * SZ_ROWS_G : SZ_ROWS_G;
            P->count[at] = (int16_t)n;
            before[at] = sz_rows_weight(n);
        }
    }
    if (t == 0) P->n_groups = shg + total;
    // the shared expert's group j comes before the others' group j * every (after all of them where those are fewer)
    auto place_sh = [&](int j) { return j * every < total ? j * (every + 1) : total + j; };
    if (has_shared) {   // the rows in order, after the pairs' slots
        for (int j = t; j < shg; j += 1024) {
            const int g = place_sh(j);
            P->first[g] = pairs + j * SZ_ROWS_G;
            P->expert[g] = -1;
            const int n = R - j * SZ_ROWS_G < SZ_ROWS_G ? R - j * SZ_ROWS_G : SZ_ROWS_G;
            P->count[g] = (int16_t)n;
            before[g] = sz_rows_weight(n);
        }
        for (int r = t; r < R; r += 1024) { P->row[pairs + r] = (int16_t)r; P->group[pairs + r] = place_sh(r / SZ_ROWS_G); P->pair_loc[pairs + r] = pairs + r; }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NP; i++) {
        const int p = t + 1024 * i, e = pe[i];
        if (p >= pairs) break;
        const int row = p / k;
        if ((unsigned)e >= (unsigned)ne) { P->pair_loc[p] = 0; P->overflow = 4; atomicOr(err, 4u); continue; }   // an expert id out of range: the call is reported as failed (the flag is this call's, the word stays)
        const int n = pre[e * MW + (row >> 5)] + __popc(mask[e * MW + (row >> 5)] & ((1u << (row & 31)) - 1u));
        const int slot = slot_of[e] + n;
        P->row[slot] = (int16_t)row;
        P->group[slot] = place(grp_of[e] + n / SZ_ROWS_G);
        P->pair_loc[p] = slot;
    }
    // ---- the blocks' shares: equal weights
    const int NG = shg + total;
    const int w0 = 2 * t < NG ? before[2 * t] : 0, w1 = 2 * t + 1 < NG ? before[2 * t + 1] : 0;   // (2,048 threads' worth: SZ_ROWS_MAXG fits)
    int ws = w0 + w1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int a = __shfl_up_sync(0xffffffffu, ws, o); if (lane >= o) ws += a; }
    __syncthreads();
    if (lane == 31) wsum[0][warp] = ws;
    __syncthreads();
    if (warp == 0) {
        int a = wsum[0][lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int b = __shfl_up_sync(0xffffffffu, a, o); if (lane >= o) a += b; }
        wsum[0][lane] = a;
    }
    __syncthreads();
    ws += (warp ? wsum[0][warp - 1] : 0) - w0 - w1;
    if (2 * t <= NG) before[2 * t] = ws;
    if (2 * t + 1 <= NG) before[2 * t + 1] = ws + w0;
    __syncthreads();
    for (int i = t; i < 2 * (grid + 1); i += 1024) {
        const int b = i >> 1, upg = (i & 1) ? upg_dn : upg_gu;
        const long long T = (long long)before[NG] * upg * b / grid;      // weight before the block's share
        int lo = 0, hi = NG;                                             // the group it falls in: before[lo] * upg <= T
        while (lo + 1 < hi) { const int mid = (lo + hi) >> 1; if ((long long)before[mid] * upg <= T) lo = mid; else hi = mid; }
        int u = b == grid ? NG * upg : 0;
        if (b < grid && NG > 0) u = lo * upg + (int)((T - (long long)before[lo] * upg) / (before[lo + 1] - before[lo]));
        bs[i & 1][b] = u;
        P->start[i & 1][b] = u;
    }
    __syncthreads();
    // the last block that starts at or before unit u, the `r`-th of group g: about the share that the weight before it is of all
    const float per = before[NG] > 0 ? (float)grid / (float)before[NG] : 0.f;
    auto block_of = [&](const int* st, float inv, int g, int r, int u) {
        int b = (int)(((float)before[g] + (float)(before[g + 1] - before[g]) * (float)r * inv) * per);
        b = b < 0 ? 0 : (b > grid - 1 ? grid - 1 : b);
        while (b > 0 && st[b] > u) b--;
        while (b + 1 < grid && st[b + 1] <= u) b++;
        return (u32)b;
    };
    const int nc = upg_dn / kb, per_g = 2 + nc;
    const float inv_gu = 1.f / (float)upg_gu, inv_dn = 1.f / (float)upg_dn;
    for (int i = t; i < NG * per_g; i += 1024) {
        const int g = i / per_g, q = i - g * per_g;
        if (q < 2) { const int r = q * ns, u = g * upg_gu + r; P->gu_blocks[g][q] = block_of(bs[0], inv_gu, g, r, u) | (block_of(bs[0], inv_gu, g, r + ns - 1, u + ns - 1) << 16); }
        else { const int r = (q - 2) * kb, u = g * upg_dn + r; P->dn_blocks[g][q - 2] = block_of(bs[1], inv_dn, g, r, u) | (block_of(bs[1], inv_dn, g, r + kb - 1, u + kb - 1) << 16); }
    }
}

// A block's groups, staged once: it works on a contiguous range of units, so on a few consecutive groups.
#define SZ_ROWS_STAGED 64
struct SzRowsGroups {
    int32_t first[SZ_ROWS_STAGED];
    int16_t expert[SZ_ROWS_STAGED], count[SZ_ROWS_STAGED];
    int16_t row[SZ_ROWS_STAGED][SZ_ROWS_G];
};
__device__ __forceinline__ void sz_rows_stage_groups(const SzRowsPlan* __restrict__ P, int g_lo, int g_hi, SzRowsGroups* S) {
    for (int i = threadIdx.x; i < (g_hi - g_lo) * SZ_ROWS_G; i += blockDim.x) {
        const int g = i / SZ_ROWS_G, t = i % SZ_ROWS_G;
        const int first = __ldcg(&P->first[g_lo + g]), n = __ldcg(&P->count[g_lo + g]);
        if (t == 0) { S->first[g] = first; S->expert[g] = __ldcg(&P->expert[g_lo + g]); S->count[g] = (int16_t)n; }
        S->row[g][t] = t < n ? __ldcg(&P->row[first + t]) : (int16_t)0;
    }
}

// One staged unit for up to 8 NB rows: 8 tile rows x TW tile columns a warp; c[nt][tc] as sz_xw_compute's.  The second eight rows'
// fragments follow the first's.  trow: bytes from one staged tile row to the next.
template <int K, int TW, int NB>
__device__ __forceinline__ void sz_rows_compute_n(const u8* wbase, int trow, const uint4* fl, const SzXWLane<K>& S, float (*c)[TW][4]) {
#pragma unroll
    for (int nt = 0; nt < NB; nt++)
#pragma unroll
        for (int tc = 0; tc < TW; tc++) { c[nt][tc][0] = 0.f; c[nt][tc][1] = 0.f; c[nt][tc][2] = 0.f; c[nt][tc][3] = 0.f; }
#pragma unroll
    for (int kr = 0; kr < 8; kr++) {
        uint4 b[NB];
#pragma unroll
        for (int nt = 0; nt < NB; nt++) b[nt] = fl[nt * 256 + kr * 32];
#pragma unroll
        for (int tc = 0; tc < TW; tc++) {
            u32 a[4];
            sz_xw_afrag<K>((const u32*)(wbase + kr * trow + tc * (32 * K)), S, a);
#pragma unroll
            for (int nt = 0; nt < NB; nt++) {
                sz_mma16816(c[nt][tc], a, b[nt].x, b[nt].y);
                sz_mma16816(c[nt][tc], a, b[nt].z, b[nt].w);
            }
        }
    }
}
// .. and its partial sums, rounded to fixed point as every unit's are, into the warp's running sums
template <int TW, int NB>
__device__ __forceinline__ void sz_rows_add(long long (*a)[TW][4], const float (*c)[TW][4]) {
#pragma unroll
    for (int nt = 0; nt < NB; nt++)
#pragma unroll
        for (int tc = 0; tc < TW; tc++)
#pragma unroll
            for (int i = 0; i < 4; i++) a[nt][tc][i] += __float2ll_rn(c[nt][tc][i] * SZ_FIX_SCALE);
}
// (two bodies: with the second eight rows' instructions merely predicated off, a group of eight paid their issue slots).  `done`: the
// warp has read the stage.
template <int K, int TW, typename Done>
__device__ __forceinline__ void sz_rows_unit(const u8* wbase, int trow, const uint4* fl, int n, const SzXWLane<K>& S, long long (*a)[TW][4], Done done) {
    if (n > 8) {
        float c[2][TW][4];
        sz_rows_compute_n<K, TW, 2>(wbase, trow, fl, S, c);
        done();
        sz_rows_add<TW, 2>(a, c);
    } else {
        float c[1][TW][4];
        sz_rows_compute_n<K, TW, 1>(wbase, trow, fl, S, c);
        done();
        sz_rows_add<TW, 1>(a, c);
    }
}
// An item's sums to their place: rows t < n of the group, the warp's TW tile columns from column col0 on - finished (f32, dst + t *
// stride) or, where another block has the rest of the item, as integers (part + t * 512).
template <int TW>
__device__ __forceinline__ void sz_rows_store(bool whole, float* dst, size_t stride, long long* part, int n, int col0, int lane, long long (*a)[TW][4]) {
    const int q = lane & 3, g8 = lane >> 2;
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int tt = 0; tt < 2; tt++) {
            const int t = nt * 8 + 2 * q + tt;
            if (t < n) {
#pragma unroll
                for (int tc = 0; tc < TW; tc++) {
                    const long long lo = a[nt][tc][tt], hi = a[nt][tc][2 + tt];
                    const int at = col0 + tc * 16 + g8;
                    if (whole) { float* d = dst + (size_t)t * stride + at; d[0] = (float)((double)lo * SZ_FIX_INV); d[8] = (float)((double)hi * SZ_FIX_INV); }
                    else { long long* d = part + t * 512 + at; d[0] = lo; d[8] = hi; }
                }
            }
        }
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int tc = 0; tc < TW; tc++)
#pragma unroll
            for (int i = 0; i < 4; i++) a[nt][tc][i] = 0;
}
// A reader's side: an item that one block worked on is finished at its place; of several (blocks: first and last) the parts are added.
// A block's first item, begun by another block, is its part 0; its last item, left unfinished, its part 1.
__device__ __forceinline__ long long* sz_rows_part(long long* parts, int b, bool begun_before) { return parts + ((size_t)b * 2 + (begun_before ? 0 : 1)) * (SZ_ROWS_G * 512); }
// .. four values (columns col + 32 e) of row t of the item
__device__ __forceinline__ void sz_rows_read(const float* done, const long long* parts, u32 blocks, const int32_t* start, int t, int col, float* v) {
    const int b0 = (int)(blocks & 0xffffu), b1 = (int)(blocks >> 16);
    if (b0 == b1) {
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] = __ldcg(done + 32 * e);
        return;
    }
    long long a[4] = {0, 0, 0, 0};
    for (int b = b0; b <= b1; b++) {
        if (__ldcg(start + b) == __ldcg(start + b + 1)) continue;     // (fewer units than blocks: this one has none)
        const long long* p = sz_rows_part(const_cast<long long*>(parts), b, b > b0) + t * 512 + col;
#pragma unroll
        for (int e = 0; e < 4; e++) a[e] += __ldcg(p + 32 * e);
    }
#pragma unroll
    for (int e = 0; e < 4; e++) v[e] = (float)((double)a[e] * SZ_FIX_INV);
}

#define SZ_ROWS_CW 16             // consumer warps
#define SZ_ROWS_PW 4              // gate / up: warps that make the fragments (rows p, p + 4, .. of a group; warp 0 of them copies, too)
template <int K, int TW>
struct SzRowsX {
    static constexpr int TILE_BYTES = 32 * K;
    static constexpr int FRAG_BYTES = 2 * 8 * 32 * 16;        // fragments of 16 rows x 128 inputs
    static constexpr int STAGE_BYTES = 8 * SZ_ROWS_CW * TW * TILE_BYTES;   // the trellis words of 8 tile rows x 16 TW tile columns
    static constexpr int FIT = 200 * 1024 / (STAGE_BYTES + FRAG_BYTES);
    static constexpr int STAGES = FIT > 6 ? 6 : FIT;          // gate / up: trellis and fragments a stage
    static constexpr int GU_SMEM = STAGES * (STAGE_BYTES + FRAG_BYTES) + 2 * STAGES * 8;
    static constexpr int DFIT = (200 * 1024 - 4 * FRAG_BYTES) / STAGE_BYTES;
    static constexpr int DSTAGES = DFIT > 6 ? 6 : DFIT;       // down: the fragments of a group's (up to) four input blocks apart
    static constexpr int DN_SMEM = DSTAGES * STAGE_BYTES + 4 * FRAG_BYTES + 2 * (DSTAGES + 4) * 8;
};

// ---- gate / up: gu[slot][2][FF] = the pairs' sums -------------------------------------------------------------------------------------
// unit = (group * 2 + matrix) * NS + input block; FF = 256 TW outputs (or 128, TW = 1: half of the consumers idle)
template <int K, int TW>
__global__ void __launch_bounds__(32 * (SZ_ROWS_CW + SZ_ROWS_PW), 1)
sz_rows_gateup_kernel(const SzRowsPlan* __restrict__ P, const u8* __restrict__ gate, u64 gstride, const u8* __restrict__ up, u64 ustride,
                      const u8* __restrict__ sh_gate, const u8* __restrict__ sh_up, const float* __restrict__ x, int H, int FF,
                      float* __restrict__ gu, long long* __restrict__ parts, u32* __restrict__ err) {
    using X = SzRowsX<K, TW>;
    constexpr int S = X::STAGES;
    extern __shared__ __align__(128) u8 smem[];
    u8* stages = smem;
    uint4* frags = (uint4*)(smem + S * X::STAGE_BYTES);
    u64 *full = (u64*)(smem + S * (X::STAGE_BYTES + X::FRAG_BYTES)), *empty = full + S;
    __shared__ SzRowsGroups G;
    __shared__ __align__(16) float buf[SZ_ROWS_PW][128];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; i++) { sz_mbar_init(&full[i], 1 + SZ_ROWS_PW); sz_mbar_init(&empty[i], SZ_ROWS_CW); }
        sz_mbar_fence_init();
    }
    sz_pdl_wait();
    sz_pdl_trigger();
    const int NS = H / 128, upg = 2 * NS;
    const int u0 = __ldcg(&P->start[0][blockIdx.x]), u1 = __ldcg(&P->start[0][blockIdx.x + 1]), count = u1 - u0;
    if (count <= 0) return;
    const int g0 = u0 / upg;
    sz_rows_stage_groups(P, g0, (u1 - 1) / upg + 1, &G);
    __syncthreads();
    // the unit's (group, matrix, input block): divided out once, then stepped
    int g = 0, mat, s;
    { const int rem = u0 - g0 * upg; mat = rem / NS; s = rem - mat * NS; }
    auto step = [&]() { if (++s == NS) { s = 0; if (++mat == 2) { mat = 0; g++; } } };
    int failed = 0;
    if (warp >= SZ_ROWS_CW) {
        const int p = warp - SZ_ROWS_CW;
        const size_t hdr = 2 * (size_t)H + 2 * (size_t)FF + 4;
        const u32 mrow = (u32)(FF / 16) * X::TILE_BYTES;    // bytes of one tile row of the matrix
        auto blob_of = [&]() -> const u8* {
            const int e = G.expert[g];
            return e < 0 ? (mat ? sh_up : sh_gate) : (mat ? up + (u64)e * ustride : gate + (u64)e * gstride);
        };
        // a unit's values and scales are requested when the unit before it has been handed over, and used after the wait for its stage
        float v[4][4], sc[4];
        auto load = [&]() {
            const u16* suh = (const u16*)blob_of() + s * 128;
            const int n = G.count[g];
#pragma unroll
            for (int e = 0; e < 4; e++) sc[e] = sz_f16_to_f32(__ldg(suh + lane + 32 * e));
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (p + SZ_ROWS_PW * i < n) {
                    const float* xr = x + (size_t)G.row[g][p + SZ_ROWS_PW * i] * H + s * 128 + lane;
#pragma unroll
                    for (int e = 0; e < 4; e++) v[i][e] = __ldcg(xr + 32 * e);
                }
        };
        load();
        for (int i = 0; i < count; i++) {
            const int st = i % S;
            if (i >= S && !sz_mbar_wait(&empty[st], ((i / S) - 1) & 1)) { failed = 1; break; }
            const int n = G.count[g];
            if (p == 0 && lane == 0) {    // the unit is contiguous: every tile column of 8 tile rows
                sz_mbar_expect_tx(&full[st], 8 * mrow);
                sz_bulk_g2s(stages + (size_t)st * X::STAGE_BYTES, blob_of() + hdr + (size_t)s * 8 * mrow, 8 * mrow, &full[st]);
            }
            uint4* frag = frags + st * (X::FRAG_BYTES / 16) + (lane >> 2) * 32 + (lane & 3);
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int t = p + SZ_ROWS_PW * r;
                if (t < n) {
#pragma unroll
                    for (int e = 0; e < 4; e++) v[r][e] *= sc[e];
                    frag[(t >> 3) * 256 + 4 * (t & 7)] = sz_xw_piece(v[r], buf[p], lane);
                }
            }
            __syncwarp();
            if (lane == 0) sz_mbar_arrive(&full[st]);   // (release: the warp's fragment stores are ordered before it by the __syncwarp)
            step();
            if (i + 1 < count) load();
        }
    } else {
        const SzXWLane<K> LS = sz_xw_lane<K>(lane);
        const bool on = warp * TW * 16 < FF;
        const int trow = FF / 16 * X::TILE_BYTES;
        long long a[2][TW][4];
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
            for (int tc = 0; tc < TW; tc++)
#pragma unroll
                for (int i = 0; i < 4; i++) a[nt][tc][i] = 0;
        bool whole = s == 0;       // the item at hand began here
        for (int i = 0; i < count; i++) {
            const int st = i % S, n = G.count[g];
            if (!sz_mbar_wait(&full[st], (i / S) & 1)) { failed = 1; break; }
            auto done = [&]() {
                __syncwarp();
                if (lane == 0) sz_mbar_arrive(&empty[st]);
            };
            if (on) {
                sz_rows_unit<K, TW>(stages + (size_t)st * X::STAGE_BYTES + (size_t)(warp * TW) * X::TILE_BYTES, trow, frags + st * (X::FRAG_BYTES / 16) + lane, n, LS, a, done);
                if (s == NS - 1 || i == count - 1)
                    sz_rows_store<TW>(whole && s == NS - 1, gu + ((size_t)G.first[g] * 2 + mat) * FF, (size_t)2 * FF, sz_rows_part(parts, blockIdx.x, !whole), n, warp * TW * 16, lane, a);
            } else {
                done();
            }
            if (s == NS - 1) whole = true;
            step();
        }
    }
    if (failed && lane == 0) atomicExch(err, 1u);
}

// ---- act: SwiGLU of every pair, a warp a (slot, block of 128) ------------------------------------------------------------------------
// Rotate back (H), scale by svh, silu(g) * u, then into the down trellis' basis (suh, H): the row's pieces of the down product's
// fragments, [group][input block][16 rows] in fragment order.
__global__ void __launch_bounds__(256)
sz_rows_act_kernel(const SzRowsPlan* __restrict__ P, const u8* __restrict__ gate, u64 gstride, const u8* __restrict__ up, u64 ustride,
                   const u8* __restrict__ down, u64 dstride, const u8* __restrict__ sh_gate, const u8* __restrict__ sh_up, const u8* __restrict__ sh_down,
                   int H, int FF, int slots, const float* __restrict__ gu, const long long* __restrict__ parts, uint4* __restrict__ frags) {
    __shared__ __align__(16) float buf[8][128];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, KB = FF / 128;
    const int item = blockIdx.x * 8 + warp;
    const int slot = item / KB, kb = item - slot * KB;
    sz_pdl_wait();
    sz_pdl_trigger();
    if (item >= slots * KB) return;
    const int g = __ldcg(&P->group[slot]);
    const int t = slot - __ldcg(&P->first[g]), e_ = __ldcg(&P->expert[g]);
    const u8* bg = e_ < 0 ? sh_gate : gate + (u64)e_ * gstride;
    const u8* bu = e_ < 0 ? sh_up : up + (u64)e_ * ustride;
    const u8* bd = e_ < 0 ? sh_down : down + (u64)e_ * dstride;
    const u16* svg = (const u16*)(bg + 2 * (size_t)H) + kb * 128 + lane;
    const u16* svu = (const u16*)(bu + 2 * (size_t)H) + kb * 128 + lane;
    const u16* suh = (const u16*)bd + kb * 128 + lane;
    float gg[4], uu[4], v[4], sc[12];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        sc[e] = sz_f16_to_f32(__ldg(svg + 32 * e));
        sc[4 + e] = sz_f16_to_f32(__ldg(svu + 32 * e));
        sc[8 + e] = sz_f16_to_f32(__ldg(suh + 32 * e));
    }
    const float* done = gu + (size_t)slot * 2 * FF + kb * 128 + lane;
    sz_rows_read(done, parts, __ldcg(&P->gu_blocks[g][0]), P->start[0], t, kb * 128 + lane, gg);
    sz_rows_read(done + FF, parts, __ldcg(&P->gu_blocks[g][1]), P->start[0], t, kb * 128 + lane, uu);
    sz_wht128_warp(gg, lane);
    sz_wht128_warp(uu, lane);
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float gv = (gg[e] * SZ_RSQRT128) * sc[e], uv = (uu[e] * SZ_RSQRT128) * sc[4 + e];
        v[e] = (sz_silu(gv) * uv) * sc[8 + e];
    }
    frags[((size_t)g * KB + kb) * 512 + (t >> 3) * 256 + (lane >> 2) * 32 + 4 * (t & 7) + (lane & 3)] = sz_xw_piece(v, buf[warp], lane);
}

// ---- down: dn[slot][H] = the pairs' sums -------------------------------------------------------------------------------------------------
// unit = (group * NC + chunk of 512 outputs) * KB + input block.  The trellis goes through a ring of stages, the group's fragments
// through a buffer an input block: copied when the group's first unit of that block comes up, kept for the group's other chunks.
template <int K>
__global__ void __launch_bounds__(32 * (SZ_ROWS_CW + 1), 1)
sz_rows_down_kernel(const SzRowsPlan* __restrict__ P, const u8* __restrict__ down, u64 dstride, const u8* __restrict__ sh_down, int H, int FF,
                    const uint4* __restrict__ gfrags, float* __restrict__ dn, long long* __restrict__ parts, u32* __restrict__ err) {
    constexpr int TW = 2;
    using X = SzRowsX<K, TW>;
    constexpr int S = X::DSTAGES, ROW_BYTES = X::STAGE_BYTES / 8;
    extern __shared__ __align__(128) u8 smem[];
    u8* stages = smem;
    uint4* frags = (uint4*)(smem + S * X::STAGE_BYTES);
    u64 *full = (u64*)(smem + S * X::STAGE_BYTES + 4 * X::FRAG_BYTES), *empty = full + S, *ffull = empty + S, *fempty = ffull + 4;
    __shared__ SzRowsGroups G;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; i++) { sz_mbar_init(&full[i], 1); sz_mbar_init(&empty[i], SZ_ROWS_CW); }
        for (int i = 0; i < 4; i++) { sz_mbar_init(&ffull[i], 1); sz_mbar_init(&fempty[i], SZ_ROWS_CW); }
        sz_mbar_fence_init();
    }
    // the plan was finished three kernels ago (each of them waited for the one before it): read ahead of the wait, as the trellis is
    const int KB = FF / 128, NC = H / 512, upg = NC * KB;
    const int u0 = __ldcg(&P->start[1][blockIdx.x]), u1 = __ldcg(&P->start[1][blockIdx.x + 1]), count = u1 - u0;
    const int g0 = u0 / upg;
    if (count > 0) sz_rows_stage_groups(P, g0, (u1 - 1) / upg + 1, &G);
    __syncthreads();
    if (count <= 0) { sz_pdl_wait(); sz_pdl_trigger(); return; }
    int g = 0, c, kb;
    { const int rem = u0 - g0 * upg; c = rem / KB; kb = rem - c * KB; }
    auto step = [&]() { if (++kb == KB) { kb = 0; if (++c == NC) { c = 0; g++; } } };
    u32 seen = 0, gen = 0;      // bit kb: this group's fragments of the block were asked for; how often so far, a byte a block (fewer than 255 groups a block)
    int failed = 0;
    if (warp == SZ_ROWS_CW) {
        if (lane == 0) {
            const size_t hdr = 2 * (size_t)FF + 2 * (size_t)H + 4;
            const u64 mrow = (u64)(H / 16) * X::TILE_BYTES;
            int pg = 0, pc = c, pkb = kb;             // the unit whose trellis is requested next, ahead of the fragments' (g, c, kb)
            auto issue = [&](int at) {
                const int e = G.expert[pg];
                const u8* src = (e < 0 ? sh_down : down + (u64)e * dstride) + hdr + (size_t)pkb * 8 * mrow + (size_t)pc * ROW_BYTES;
                u8* dst = stages + (size_t)(at % S) * X::STAGE_BYTES;
                sz_mbar_expect_tx(&full[at % S], X::STAGE_BYTES);
#pragma unroll
                for (int kr = 0; kr < 8; kr++) sz_bulk_g2s(dst + kr * ROW_BYTES, src + kr * mrow, ROW_BYTES, &full[at % S]);
                if (++pkb == KB) { pkb = 0; if (++pc == NC) { pc = 0; pg++; } }
            };
            // the unit's fragments, if no unit of the group asked for them before: after the group before it is done with the buffer
            auto ask = [&]() -> bool {
                if (!((seen >> kb) & 1u)) {
                    const u32 n_ = (gen >> (8 * kb)) & 0xffu;
                    if (n_ > 0 && !sz_mbar_wait(&fempty[kb], (n_ - 1) & 1)) return false;
                    const u32 bytes = G.count[g] > 8 ? X::FRAG_BYTES : X::FRAG_BYTES / 2;
                    sz_mbar_expect_tx(&ffull[kb], bytes);
                    sz_bulk_g2s(frags + kb * (X::FRAG_BYTES / 16), gfrags + ((size_t)(g0 + g) * KB + kb) * 512, bytes, &ffull[kb]);
                    seen |= 1u << kb;
                    gen += 1u << (8 * kb);
                }
                const int gw = g;
                step();
                if (g != gw) seen = 0;
                return true;
            };
            const int pre = count < S ? count : S;
            for (int i = 0; i < pre; i++) issue(i);
            sz_pdl_wait();
            sz_pdl_trigger();
            for (int i = 0; i < pre && !failed; i++) failed = !ask();
            for (int i = pre; i < count && !failed; i++) {
                if (!sz_mbar_wait(&empty[i % S], ((i / S) - 1) & 1)) { failed = 1; break; }
                issue(i);
                failed = !ask();
            }
        } else {
            sz_pdl_wait();
            sz_pdl_trigger();
        }
    } else {
        sz_pdl_wait();
        sz_pdl_trigger();
        const SzXWLane<K> LS = sz_xw_lane<K>(lane);
        long long a[2][TW][4];
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
            for (int tc = 0; tc < TW; tc++)
#pragma unroll
                for (int i = 0; i < 4; i++) a[nt][tc][i] = 0;
        bool whole = kb == 0;
        for (int i = 0; i < count; i++) {
            const int st = i % S, n = G.count[g];
            if (!((seen >> kb) & 1u)) { seen |= 1u << kb; gen += 1u << (8 * kb); }
            if (!sz_mbar_wait(&ffull[kb], (((gen >> (8 * kb)) & 0xffu) - 1) & 1) || !sz_mbar_wait(&full[st], (i / S) & 1)) { failed = 1; break; }
            const bool last = i + KB >= count || c == NC - 1;    // the group's last unit of this input block here
            sz_rows_unit<K, TW>(stages + (size_t)st * X::STAGE_BYTES + (size_t)(warp * TW) * X::TILE_BYTES, ROW_BYTES, frags + kb * (X::FRAG_BYTES / 16) + lane, n, LS, a, [&]() {
                __syncwarp();
                if (lane == 0) { sz_mbar_arrive(&empty[st]); if (last) sz_mbar_arrive(&fempty[kb]); }
            });
            if (kb == KB - 1 || i == count - 1)
                sz_rows_store<TW>(whole && kb == KB - 1, dn + (size_t)G.first[g] * H + c * 512, (size_t)H, sz_rows_part(parts, blockIdx.x, !whole), n, warp * TW * 16, lane, a);
            if (kb == KB - 1) whole = true;
            const int gw = g;
            step();
            if (g != gw) seen = 0;
        }
    }
    if (failed && lane == 0) atomicExch(err, 1u);
}

// ---- combine: two forms (which: sz_rows_combine_by_warp) ---------------------------------------------------------------------------------
// y[j] = sum over ranks of w * (H eo * svh) + sigmoid(shared gate logit) * (H so * svh_shared), term by term as sz_x3_combine_kernel: the ranks'
// terms are finished and added in rank order in f64.  dn, parts: the down kernel's sums.
// A warp a rank for 512 outputs of a row: warp t finishes rank t's term (warp top_k: the shared expert's), then a thread adds an output's terms.
// A block takes the 512 outputs of one of its items, so that the way to the sums - expert, slot, group, blocks: four trips to memory one after
// the other - is gone once for 16 values a lane (a block per 128 outputs: 504 rows 55 -> 43 us), and the ranks go it side by side: few rows' sums, which
// lie in many blocks' parts, are added by all warps at once (1 row of 10 experts 12 us, the form below 24).
// grid (rows * H / 512), block (top_k + 1) warps
__global__ void __launch_bounds__((SZ_MAX_TOPK + 1) * 32)
sz_rows_combine_ranks_kernel(const float* __restrict__ dn, const long long* __restrict__ parts, const SzRowsPlan* __restrict__ P, const int32_t* __restrict__ ridx, const double* __restrict__ rw,
                       const u8* __restrict__ down, u64 dstride, const u8* __restrict__ sh_down, const float* __restrict__ logits, int ne, int top_k,
                       int rows, int H, int FF, int SF, int has_shared, float* __restrict__ y) {
    __shared__ float part[SZ_MAX_TOPK + 1][512];
    __shared__ double rws[SZ_MAX_TOPK];
    sz_pdl_wait();
    sz_pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nb = H / 512;
    const int j = blockIdx.x / nb, b = blockIdx.x % nb;
    if (warp < top_k || has_shared) {
        const bool routed = warp < top_k;
        const int pair = routed ? j * top_k + warp : rows * top_k + j;
        int e = routed ? __ldcg(ridx + pair) : 0;
        const int loc = __ldcg(&P->pair_loc[pair]), g = __ldcg(&P->group[loc]);
        e = (unsigned)e < (unsigned)ne ? e : 0;
        const u16* svh = (const u16*)(routed ? down + (u64)e * dstride + 2 * (size_t)FF : sh_down + 2 * (size_t)SF) + b * 512 + lane;
        u16 sv[16];
#pragma unroll
        for (int i = 0; i < 16; i++) sv[i] = __ldg(svh + 32 * i);
        const float sg = routed ? 1.f : sz_sigmoid(__ldcg(logits + (size_t)j * (ne + 1) + ne));
        const double wt = routed && lane == 0 ? __ldcg(rw + pair) : 0.0;
        const u32 blocks = __ldcg(&P->dn_blocks[g][b]);
        const int t = loc - __ldcg(&P->first[g]), b0 = (int)(blocks & 0xffffu), b1 = (int)(blocks >> 16);
        float v[16];
        if (b0 == b1) {
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = __ldcg(dn + (size_t)loc * H + b * 512 + lane + 32 * i);
        } else {
            long long a[16] = {};
            for (int q = b0; q <= b1; q++) {
                if (__ldcg(P->start[1] + q) == __ldcg(P->start[1] + q + 1)) continue;     // (fewer units than blocks: this one has none)
                const long long* p = sz_rows_part(const_cast<long long*>(parts), q, q > b0) + t * 512 + lane;
#pragma unroll
                for (int i = 0; i < 16; i++) a[i] += __ldcg(p + 32 * i);
            }
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = (float)((double)a[i] * SZ_FIX_INV);
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
            sz_wht128_warp(v + 4 * c, lane);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float x = (v[4 * c + q] * SZ_RSQRT128) * sz_f16_to_f32(sv[4 * c + q]);
                part[warp][128 * c + lane + 32 * q] = routed ? x : sg * x;
            }
        }
        if (routed && lane == 0) rws[warp] = wt;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 512; i += blockDim.x) {
        double a = 0.0;
        for (int t = 0; t < top_k; t++) a += rws[t] * (double)part[t][i];
        if (has_shared) a += (double)part[top_k][i];
        y[(size_t)j * H + b * 512 + i] = (float)a;
    }
}

// .. and a warp a (row, 128 outputs), for many rows of many ranks.
// What bounds it is the way to the sums - slot, group, blocks: three trips to memory one after the other - and then their 4 bytes an output and rank.
// So the ranks go that way side by side, a lane each; the sums are asked for by their slots, without waiting for the blocks that say whether
// they are finished there (of those that are not - one block's share ended inside - the parts are added instead), four ranks at a time; and one warp has all
// ranks of its outputs, so nothing meets in shared memory.  (10 experts a row of 2,048: 504 rows 42 -> 37 us, 256 27 -> 25.)  Shuffles and f64 conversions of eleven rotations an output are the most of it now.
// grid (ceil(rows * H / 1024)), block 256
__global__ void __launch_bounds__(256)
sz_rows_combine_kernel(const float* __restrict__ dn, const long long* __restrict__ parts, const SzRowsPlan* __restrict__ P, const int32_t* __restrict__ ridx, const double* __restrict__ rw,
                       const u8* __restrict__ down, u64 dstride, const u8* __restrict__ sh_down, const float* __restrict__ logits, int ne, int top_k,
                       int rows, int H, int FF, int SF, int has_shared, float* __restrict__ y) {
    constexpr int RB = 4;               // ranks at a time
    sz_pdl_wait();
    sz_pdl_trigger();
    const int lane = threadIdx.x & 31, nb = H / 128, item = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int j = item / nb, b = item - j * nb, n = top_k + (has_shared ? 1 : 0);
    if (j >= rows) return;
    // lane t: rank t's expert, slot, weight (rank top_k: the shared expert's)
    int e = 0, loc = 0;
    double wt = 0.0;
    float sg = 1.f;
    if (lane < n) {
        const bool routed = lane < top_k;
        loc = __ldcg(&P->pair_loc[routed ? j * top_k + lane : rows * top_k + j]);
        if (routed) {
            e = __ldcg(ridx + j * top_k + lane);
            e = (unsigned)e < (unsigned)ne ? e : 0;
            wt = __ldcg(rw + j * top_k + lane);
        } else sg = __ldcg(logits + (size_t)j * (ne + 1) + ne);
    }
    float v[2][RB][4];
    u16 sv[2][RB][4];
    auto fetch = [&](int t0, float (*d)[4], u16 (*s)[4]) {
#pragma unroll
        for (int r = 0; r < RB; r++) {
            const int t = t0 + r;
            const int l = __shfl_sync(0xffffffffu, loc, t), ex = __shfl_sync(0xffffffffu, e, t);
            if (t >= n) continue;
            const u16* svh = (const u16*)(t < top_k ? down + (u64)ex * dstride + 2 * (size_t)FF : sh_down + 2 * (size_t)SF) + b * 128 + lane;
#pragma unroll
            for (int i = 0; i < 4; i++) { d[r][i] = __ldcg(dn + (size_t)l * H + b * 128 + lane + 32 * i); s[r][i] = __ldg(svh + 32 * i); }
        }
    };
    fetch(0, v[0], sv[0]);
    u32 blocks = 0;
    int row = 0;                        // the pair's row of its group
    if (lane < n) {
        const int g = __ldcg(&P->group[loc]);
        blocks = __ldcg(&P->dn_blocks[g][b >> 2]);
        row = loc - __ldcg(&P->first[g]);
    }
    if (has_shared) sg = sz_sigmoid(__shfl_sync(0xffffffffu, sg, top_k));
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    auto add = [&](int t0, float (*d)[4], u16 (*s)[4]) {
#pragma unroll
        for (int r = 0; r < RB; r++) {
            const int t = t0 + r;
            const u32 bl = __shfl_sync(0xffffffffu, blocks, t);
            const int tr = __shfl_sync(0xffffffffu, row, t), b0 = (int)(bl & 0xffffu), b1 = (int)(bl >> 16);
            const double w = __shfl_sync(0xffffffffu, wt, t);
            if (t >= n) continue;
            if (b0 != b1) {
                long long p[4] = {0, 0, 0, 0};
                for (int q = b0; q <= b1; q++) {
                    if (__ldcg(P->start[1] + q) == __ldcg(P->start[1] + q + 1)) continue;     // (fewer units than blocks: this one has none)
                    const long long* at = sz_rows_part(const_cast<long long*>(parts), q, q > b0) + tr * 512 + (b & 3) * 128 + lane;
#pragma unroll
                    for (int i = 0; i < 4; i++) p[i] += __ldcg(at + 32 * i);
                }
#pragma unroll
                for (int i = 0; i < 4; i++) d[r][i] = (float)((double)p[i] * SZ_FIX_INV);
            }
            sz_wht128_warp(d[r], lane);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float x = (d[r][i] * SZ_RSQRT128) * sz_f16_to_f32(s[r][i]);
                if (t < top_k) a[i] += w * (double)x;
                else a[i] += (double)(sg * x);
            }
        }
    };
    for (int t0 = 0; t0 < n; t0 += 2 * RB) {
        if (t0 + RB < n) fetch(t0 + RB, v[1], sv[1]);
        add(t0, v[0], sv[0]);
        if (t0 + 2 * RB < n) fetch(t0 + 2 * RB, v[0], sv[0]);
        if (t0 + RB < n) add(t0 + RB, v[1], sv[1]);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) y[(size_t)j * H + b * 128 + lane + 32 * i] = (float)a[i];
}
