// EXL3 expert FFN for a verify pass, warp-specialised streaming form.
//
// Same units, same arithmetic and same fixed-point partial sums as the kernels of sz_moe_exl3.cuh (bit-identical results), another
// division of labour.  One block a multiprocessor: twenty-four DECODE warps do nothing but decode trellis tiles, issue tensor-core
// instructions and add the sums, four PRODUCER warps keep a ring of shared-memory stages full (cp.async.bulk) and prepare the units'
// activation fragments.  The two sides meet only at mbarriers: a `full` barrier a stage (the copy's bytes have landed and the
// fragments are written) and an `empty` barrier a stage (its items are decoded).
//
// A unit is cut into 8 items of TW tile columns; a decode warp that is free takes the block's next item from a counter.  Three blocks of
// eight decode warps a multiprocessor, each with units of its own, keep as many warps but do not end together: the oldest block's warps
// win the issue slots, so its units took 3.4 us where the youngest one's took 14, and the last block's last units ran alone.  Measured (us a
// layer, 2048 x 512, 512 experts, top 10; three blocks -> this): 4 rows 59.5 -> 56.0, 8 rows 107 -> 89.5, 1 row 31.8 -> 30.9.  What bounds it: the
// decode, 60 - 66 cycles a tile and scheduler with six warps (at 8 rows 51 of the 70 us of both launches), then what is not overlapped with
// it: from the wait to the first full stage 3 - 4.5 us a launch (plan, copies, fragments), and an item's sums (some 0.9 us of its 6.7).
// One launch for both (units drawn from a counter of the launch, the down units' fragments waiting for their group's gate / up units) was
// measured, too: 57.8 us at 4 rows, 94.3 at 8 - SwiGLU beside the decode takes 3 us a row, and the ring waits for it.
#pragma once

#include "sz_moe_exl3.cuh"

#define SZ_XW_DECODE 24
#define SZ_XW_PRODUCE 4
#define SZ_XW_THREADS (32 * (SZ_XW_DECODE + SZ_XW_PRODUCE))
#define SZ_XW_ITEMS 8        // items a unit

// A unit: 8 tile rows (one 128-input block) x 8 TW tile columns (TW an item).
template <int K, int TW>
struct SzXW {
    static constexpr int TILE_BYTES = 32 * K;
    static constexpr int ROW_BYTES = SZ_XW_ITEMS * TW * TILE_BYTES;   // one tile row of the unit
    static constexpr int STAGE_BYTES = 8 * ROW_BYTES;                 // the unit's trellis bytes
    static constexpr int FRAG_BYTES = 8 * 32 * 16;                    // the unit's activation fragments: [8 tile rows][32 lanes] uint4
    static constexpr int FIT = 200 * 1024 / (STAGE_BYTES + FRAG_BYTES);
    static constexpr int STAGES = FIT > 8 ? 8 : FIT;
    static constexpr int SMEM_BYTES = STAGES * (STAGE_BYTES + FRAG_BYTES) + STAGES * (2 * 8 + 4);
};

// Two-word form of SzExl3Tile<K>::states_pre: valid when the lane's span (16 + 7 K bits) starting at its bit offset inside the
// first word never crosses into a third word.  sb = first bit of window 0 = ((8 L + 1) K - 16) mod 256 K; for K = 2, 3, 4 the
// offsets sb mod 32 are {2, 18}, {3, 11, 19, 27} and {20}, and offset + span is at most 48, 64 and 64.
template <int K>
struct SzExl3Two {
    static_assert(K == 2 || K == 3 || K == 4, "the span of a lane's windows fits two words for 2, 3 and 4 bits a weight");
    static constexpr int WORDS = 8 * K, RING = 256 * K;
    struct Lane { int w0, w1, off; };
    __device__ __forceinline__ static Lane lane_setup(int lane) {
        Lane L;
        const int sb = ((8 * lane + 1) * K - 16 + RING) % RING;
        L.w0 = sb >> 5;
        L.w1 = L.w0 + 1 >= WORDS ? 0 : L.w0 + 1;
        L.off = sb & 31;
        return L;
    }
    __device__ __forceinline__ static void states(const u32* tile, const Lane& L, u32* st) {
        const u32 w0 = tile[L.w0], w1 = tile[L.w1];
        const u32 a0 = __funnelshift_l(w1, w0, L.off);   // the span from its first bit: 32 bits, then the rest
        const u32 a1 = w1 << L.off;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int pos = j * K;
            if (pos == 0) st[j] = a0 >> 16;
            else if (pos <= 16) { u32 p; asm("mul.lo.u32 %0, %1, %2;" : "=r"(p) : "r"(a0), "r"(1u << pos)); st[j] = p >> 16; }
            else st[j] = __funnelshift_l(a1, a0, pos) >> 16;
        }
    }
};

// The decode's instructions are spread over the pipes.  Measured from shared memory alone, 16 warps a multiprocessor, in cycles a tile
// and scheduler: windows by shift and mask with the byte sums on the integer tensor pipe 63.1 (the ALU pipe, at two cycles an
// instruction, has 21 of the tile's 48); byte sums by dp4a 60.9; windows of the first word by a multiplication that puts them on top
// and one shift, too, 59.8, in 52 registers instead of 83.  In the many-row gate / up kernel 400 -> 369 us.
template <int K>
struct SzXWLane {
    typename SzExl3Two<K>::Lane L;
};
template <int K>
__device__ __forceinline__ SzXWLane<K> sz_xw_lane(int lane) {
    SzXWLane<K> s;
    s.L = SzExl3Two<K>::lane_setup(lane);
    return s;
}

// The lane's 8 weights of a tile as the A fragment of m16n8k16 (the same values, bit for bit, as sz_exl3_afrag).
template <int K>
__device__ __forceinline__ void sz_xw_afrag(const u32* tile, const SzXWLane<K>& S, u32* a) {
    u32 st[8];
    SzExl3Two<K>::states(tile, S.L, st);
    const __half2 kinv = __halves2half2(__ushort_as_half((u16)0x1eee), __ushort_as_half((u16)0x1eee));
    const __half2 kbias = __halves2half2(__ushort_as_half((u16)0xc931), __ushort_as_half((u16)0xc931));
    u32 x[8];
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = st[i] * 0x83DCD12Du;
    u32 c[8];
#pragma unroll
    for (int i = 0; i < 8; i++) c[i] = __dp4a(x[i], 0x01010101u, 0x6400u);
    u32 p[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const u32 packed = __byte_perm(c[2 * i], c[2 * i + 1], 0x5410);
        const __half2 h = __hfma2(*(const __half2*)&packed, kinv, kbias);
        p[i] = *(const u32*)&h;
    }
    a[0] = p[0]; a[1] = p[2]; a[2] = p[1]; a[3] = p[3];
}

// Decodes and multiplies one staged unit (8 tile rows x 8 NTC tile columns): warp w takes tile columns w NTC .. w NTC + NTC - 1.
// c[tc] = outputs (w NTC + tc) 16 + {g, g + 8} for rows 2 q, 2 q + 1.
// The decode loop is fully unrolled: rolled over the tile rows it ran 6% slower.
template <int K, int TW>
__device__ __forceinline__ void sz_xw_compute(const u8* stage, const uint4* frag, int warp, int lane, const SzXWLane<K>& S, float (*c)[4]) {
#pragma unroll
    for (int tc = 0; tc < TW; tc++) { c[tc][0] = 0.f; c[tc][1] = 0.f; c[tc][2] = 0.f; c[tc][3] = 0.f; }
    const u8* wbase = stage + (size_t)(warp * TW) * (32 * K);
    const uint4* fl = frag + lane;
#pragma unroll
    for (int kr = 0; kr < 8; kr++) {
        const uint4 b = fl[kr * 32];
#pragma unroll
        for (int tc = 0; tc < TW; tc++) {
            const u32* tile = (const u32*)(wbase + (size_t)(kr * 8 * TW + tc) * (32 * K));
            u32 a[4];
            sz_xw_afrag<K>(tile, S, a);
            sz_mma16816(c[tc], a, b.x, b.y);
            sz_mma16816(c[tc], a, b.z, b.w);
        }
    }
}

// A row's 128 values (k = lane + 32 e on entry), rotated, as its share of the B fragments.  In the fragment order a row owns 32 whole 16-byte
// pieces - (tile row kr, quad q): values 16 kr + 2 q, + 1 and + 8, + 9 as f16 high parts, then the low parts - so the values change lanes
// through `buf` (128 floats of the warp's own) and every lane makes the piece (lane / 4, lane % 4).
__device__ __forceinline__ uint4 sz_xw_piece(float* v, float* buf, int lane) {
    sz_wht128_warp(v, lane);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 4; e++) buf[lane + 32 * e] = v[e] * SZ_RSQRT128;
    __syncwarp();
    const int at = 16 * (lane >> 2) + 2 * (lane & 3);
    const float2 x0 = *(const float2*)(buf + at), x1 = *(const float2*)(buf + at + 8);
    const __half2 h0 = __floats2half2_rn(x0.x, x0.y), h1 = __floats2half2_rn(x1.x, x1.y);
    const __half2 l0 = __floats2half2_rn(x0.x - __low2float(h0), x0.y - __high2float(h0)), l1 = __floats2half2_rn(x1.x - __low2float(h1), x1.y - __high2float(h1));
    return make_uint4(*(const u32*)&h0, *(const u32*)&h1, *(const u32*)&l0, *(const u32*)&l1);
}

// What the two sides of both kernels share: the stage ring, its barriers and whose turn a stage is.  A wait for a phase looks at its parity, so
// it is sound only where the barrier is at most one phase behind, and the ring alone does not see to that: gate / up's producers fill units
// out of order (and with 5 or 7 stages a stage's next unit is another producer's), a decode warp takes an item of whatever unit comes
// next, and one that is late with a stage does not keep the others from the units after it.  Without the turns a producer refilled
// stages that were still being read (4 bits, 6 rows, five stages: the launch failed), and a decode warp could read a stage a fill early.
// So a stage's word says which unit it was last given to, and from a stage's second fill on whoever needs it waits for that word before the
// barrier (in the first fill no phase can be mistaken; asking there, too, cost 0.5 us a layer, all warps polling while the first units arrive).
// Down's producers go through all units in order and each has arrived for a stage's unit before it waits for the next: theirs needs no word.
template <int K, int TW>
struct SzXWRing {
    using X = SzXW<K, TW>;
    u8* stages;
    uint4* frags;
    u64 *full, *empty;
    int* turn;
    __device__ __forceinline__ void init(u8* smem, int arrivals) {
        stages = smem;
        frags = (uint4*)(smem + X::STAGES * X::STAGE_BYTES);
        full = (u64*)(smem + X::STAGES * (X::STAGE_BYTES + X::FRAG_BYTES));
        empty = full + X::STAGES;
        turn = (int*)(empty + X::STAGES);
        if (threadIdx.x == 0) {
            for (int i = 0; i < X::STAGES; i++) { sz_mbar_init(&full[i], arrivals); sz_mbar_init(&empty[i], SZ_XW_ITEMS); turn[i] = -1; }
            sz_mbar_fence_init();
        }
    }
    // one warp: unit i has its stage (bounded; the lanes leave together)
    __device__ __forceinline__ bool given(int i, int lane) const {
        bool ok = lane != 0;
        if (lane == 0) {
            for (u32 n = 0; n < 20000000u && !ok; n++) {
                int v;
                asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(sz_smem_addr(turn + i % X::STAGES)) : "memory");
                ok = v == i;
            }
        }
        ok = __all_sync(0xffffffffu, ok);
        __syncwarp();
        return ok;
    }
    // .. is given it (by one lane, once the unit before it has been decoded)
    __device__ __forceinline__ void give(int i) {
        asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"(sz_smem_addr(turn + i % X::STAGES)), "r"(i) : "memory");
    }
    // one warp: the unit's 8 tile rows, `row_stride` bytes apart in the matrix, into stage st (a lane a row: one lane after the other took 60 ns each)
    __device__ __forceinline__ void issue(int st, const u8* src, u64 row_stride, int lane) {
        u8* dst = stages + (size_t)st * X::STAGE_BYTES;
        if (lane == 0) sz_mbar_expect_tx(&full[st], X::STAGE_BYTES);
        __syncwarp();
        if (row_stride == (u64)X::ROW_BYTES) {
            if (lane == 0) sz_bulk_g2s(dst, src, X::STAGE_BYTES, &full[st]);
        } else if (lane < 8) {
            sz_bulk_g2s(dst + lane * X::ROW_BYTES, src + lane * row_stride, X::ROW_BYTES, &full[st]);
        }
    }
};

// A decode warp: items of the block's `count` units until there are none.  unit[st] = (group, which of the two sums of a pair, first output
// column, -); a pair's sums are `stride` values, of which the second kind follows `second` after the first.  The sums of an item are added to
// the fixed-point accumulators of the group's pairs after its stage has been handed back.
template <int K, int TW>
__device__ __forceinline__ bool sz_xw_decode(const SzXWRing<K, TW>& R, const int4* unit, u32* next, int count, const SzPlan* plan, int D, int m, int top_k,
                                             long long* base, size_t stride, size_t second, int lane) {
    using X = SzXW<K, TW>;
    const SzXWLane<K> LS = sz_xw_lane<K>(lane);
    u32 item = 0;
    if (lane == 0) item = atomicAdd(next, 1u);
    for (;;) {
        item = __shfl_sync(0xffffffffu, item, 0);
        const int i = (int)(item / SZ_XW_ITEMS), part = (int)(item % SZ_XW_ITEMS), st = i % X::STAGES;
        if (i >= count) return true;
        if ((i >= X::STAGES && !R.given(i, lane)) || !sz_mbar_wait(&R.full[st], (i / X::STAGES) & 1)) return false;
        float c[TW][4];
        sz_xw_compute<K, TW>(R.stages + (size_t)st * X::STAGE_BYTES, R.frags + st * 256, part, lane, LS, c);
        const int4 d = unit[st];
        __syncwarp();
        if (lane == 0) { sz_mbar_arrive(&R.empty[st]); item = atomicAdd(next, 1u); }   // (the next item's number arrives beside the additions)
        const int n = d.x < D ? plan->count[d.x] : m;
        long long* dst0 = base + (d.y ? second : 0) + d.z + part * TW * 16 + (lane >> 2);
#pragma unroll
        for (int tt = 0; tt < 2; tt++) {
            const int t = 2 * (lane & 3) + tt;
            if (t < n) {
                long long* dst = dst0 + (size_t)(d.x < D ? plan->pairs[d.x][t] : m * top_k + t) * stride;
#pragma unroll
                for (int tc = 0; tc < TW; tc++) {
                    sz_fix_add(dst + tc * 16, c[tc][tt]);
                    sz_fix_add(dst + tc * 16 + 8, c[tc][2 + tt]);
                }
            }
        }
    }
}

// ---- gate / up --------------------------------------------------------------------------------------------------------------------
// Units: group x {gate, up} x input block x column chunk (8 TW tile columns of the FF / 16), the chunk fastest, dealt out to the blocks one by
// one (the shared expert's, which have the most rows, come last and so to every block alike); a block's producer warps take its units in turn: copy, fragments.  acc: i64 [pairs][2][FF], zero on entry.
template <int K, int NTC, int TW>
__global__ void __launch_bounds__(SZ_XW_THREADS, 1)
sz_xw_gateup_kernel(const SzPlan* __restrict__ plan, const u8* __restrict__ gate, u64 gstride, const u8* __restrict__ up, u64 ustride,
                    const u8* __restrict__ sh_gate, const u8* __restrict__ sh_up, const float* __restrict__ x, int m, int H, int top_k,
                    long long* __restrict__ acc, u32* __restrict__ ctrl) {
    using X = SzXW<K, TW>;
    constexpr int FF = 128 * NTC, S = X::STAGES, NCH = NTC / TW;
    static_assert(NTC % TW == 0, "column chunks tile the matrix");
    extern __shared__ __align__(128) u8 smem[];
    SzXWRing<K, TW> R;
    R.init(smem, 2);
    __shared__ __align__(16) SzPlan splan;
    __shared__ __align__(16) float buf[SZ_XW_PRODUCE][128];
    __shared__ int4 unit[S];
    __shared__ u32 next;
    if (threadIdx.x == 0) next = 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    sz_pdl_wait();
    sz_pdl_trigger();
    plan = sz_plan_stage(plan, &splan);
    __syncthreads();
    const int D = plan->n_groups, NG = D + (sh_gate ? 1 : 0), NS = H / 128;
    const int U = NG * 2 * NS * NCH, count = (U + (int)gridDim.x - 1 - (int)blockIdx.x) / (int)gridDim.x;   // units blockIdx.x, + gridDim.x, ..
    bool ok = true;
    if (warp >= SZ_XW_DECODE) {
        const int p = warp - SZ_XW_DECODE;
        const size_t hdr = 2 * (size_t)H + 2 * (size_t)FF + 4;
        const u64 mrow = (u64)(8 * NTC) * X::TILE_BYTES;    // bytes of one tile row of the matrix
        for (int i = p; i < count; i += SZ_XW_PRODUCE) {
            const int st = i % S;
            const int u = (int)blockIdx.x + i * (int)gridDim.x, key = u / NCH, ch = u - key * NCH, g = key / (2 * NS), rem = key - g * 2 * NS, mat = rem >= NS, s = rem - (mat ? NS : 0);
            const bool routed = g < D;
            const u64 e = routed ? (u64)plan->expert[g] : 0;
            const u8* blob = routed ? (mat ? up + e * ustride : gate + e * gstride) : (mat ? sh_up : sh_gate);
            const int n = routed ? plan->count[g] : m;
            const u16* suh = (const u16*)blob + s * 128 + lane;
            u16 sc[4];
#pragma unroll
            for (int q = 0; q < 4; q++) sc[q] = __ldg(suh + 32 * q);
            if (i >= S && ((i >= 2 * S && !R.given(i - S, lane)) || !sz_mbar_wait(&R.empty[st], ((i / S) - 1) & 1))) { ok = false; break; }
            if (lane == 0) { unit[st] = make_int4(g, mat, ch * SZ_XW_ITEMS * TW * 16, 0); R.give(i); }
            R.issue(st, blob + hdr + (size_t)s * 8 * mrow + (size_t)ch * X::ROW_BYTES, mrow, lane);
            uint4* frag = R.frags + st * 256 + (lane >> 2) * 32 + (lane & 3);   // (unused rows hold whatever was there: a row is a column of its own in the products)
            for (int t0 = 0; t0 < n; t0 += 4) {
                // four rows' loads are in flight before the first is used (a row at a time would pay the L2 latency once a row)
                float v[4][4];
#pragma unroll
                for (int t = 0; t < 4; t++)
                    if (t0 + t < n) {
                        const float* xr = x + (size_t)(routed ? plan->rows[g][t0 + t] : t0 + t) * H + s * 128 + lane;
#pragma unroll
                        for (int q = 0; q < 4; q++) v[t][q] = __ldg(xr + 32 * q);
                    }
#pragma unroll
                for (int t = 0; t < 4; t++)
                    if (t0 + t < n) {
#pragma unroll
                        for (int q = 0; q < 4; q++) v[t][q] *= sz_f16_to_f32(sc[q]);
                        frag[4 * (t0 + t)] = sz_xw_piece(v[t], buf[p], lane);
                    }
            }
            __syncwarp();
            if (lane == 0) sz_mbar_arrive(&R.full[st]);   // (release: the warp's fragment stores are ordered before it by the __syncwarp)
        }
    } else {
        ok = sz_xw_decode<K, TW>(R, unit, &next, count, plan, D, m, top_k, acc, (size_t)2 * FF, (size_t)FF, lane);
    }
    if (!ok && lane == 0) atomicExch(&ctrl[1], 1u);
}

// ---- down ---------------------------------------------------------------------------------------------------------------------------
// Units: group x input block (128 of FF) x output chunk (8 TW tile columns of the H / 16), the chunk fastest; 8 tile rows, strided.
// The input of a unit is the SwiGLU product of its pairs, finished by the producer warps from the gate / up sums: rotate back (H),
// scale by svh, silu(g) * u, then into the down trellis' basis (suh, H).  The chunks of one (group, input block) follow one another and
// share it: producer p makes the pieces of rows p and p + 4, keeps them in registers and stores them to every stage of the chunks.
// out: i64 [pairs][H], zero on entry.
template <int K, int TW>
__global__ void __launch_bounds__(SZ_XW_THREADS, 1)
sz_xw_down_kernel(const SzPlan* __restrict__ plan, const u8* __restrict__ gate, u64 gstride, const u8* __restrict__ up, u64 ustride,
                  const u8* __restrict__ down, u64 dstride, const u8* __restrict__ sh_gate, const u8* __restrict__ sh_up,
                  const u8* __restrict__ sh_down, int m, int H, int FF, int top_k, const long long* __restrict__ acc,
                  long long* __restrict__ out, u32* __restrict__ ctrl) {
    using X = SzXW<K, TW>;
    constexpr int S = X::STAGES;
    extern __shared__ __align__(128) u8 smem[];
    SzXWRing<K, TW> R;
    R.init(smem, 1 + SZ_XW_PRODUCE);
    __shared__ __align__(16) SzPlan splan;
    __shared__ __align__(16) float buf[SZ_XW_PRODUCE][128];
    __shared__ int4 unit[S];
    __shared__ u32 next;
    if (threadIdx.x == 0) next = 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the plan was finished two kernels ago (the kernel before this one waited for it before it let this one start): it can be read,
    // and the first copies issued, ahead of the wait; only the gate / up sums need the wait
    plan = sz_plan_stage(plan, &splan);
    __syncthreads();
    const int D = plan->n_groups, NG = D + (sh_down ? 1 : 0), KB = FF / 128, NC = H / (128 * TW);
    const u32 U = (u32)(NG * KB * NC), u0 = U * blockIdx.x / gridDim.x, u1 = U * (blockIdx.x + 1) / gridDim.x;
    const int count = (int)(u1 - u0);
    bool ok = true;
    if (warp >= SZ_XW_DECODE) {
        const int p = warp - SZ_XW_DECODE;
        const size_t hdr = 2 * (size_t)FF + 2 * (size_t)H + 4;
        const u64 drow = (u64)(H / 16) * X::TILE_BYTES;  // bytes of one tile row of the down matrix
        // the unit at hand: divided out once, then stepped (the units of a block follow one another)
        int g = u0 / (KB * NC), kb, c;
        { const int rem = u0 - g * KB * NC; kb = rem / NC; c = rem - kb * NC; }
        auto step = [&](int& g_, int& kb_, int& c_) { if (++c_ == NC) { c_ = 0; if (++kb_ == KB) { kb_ = 0; g_++; } } };
        auto issue = [&](int i, int g_, int kb_, int c_) {
            const int st = i % S;
            if (lane == 0) { unit[st] = make_int4(g_, 0, c_ * SZ_XW_ITEMS * TW * 16, 0); R.give(i); }
            R.issue(st, (g_ < D ? down + (u64)plan->expert[g_] * dstride : sh_down) + hdr + (size_t)kb_ * 8 * drow + (size_t)c_ * X::ROW_BYTES, drow, lane);
        };
        const int pre = count < S ? count : S;
        if (p == SZ_XW_PRODUCE - 1) {      // (the warp that has the fewest rows to prepare)
            int g_ = g, kb_ = kb, c_ = c;
            for (int i = 0; i < pre; i++) { issue(i, g_, kb_, c_); step(g_, kb_, c_); }
        }
        // the scales of rows p, p + 4 of the first (group, input block), too
        u16 sc[12];
        auto scales = [&]() {
            const u64 e = g < D ? (u64)plan->expert[g] : 0;
            const u16* svg = (const u16*)((g < D ? gate + e * gstride : sh_gate) + 2 * (size_t)H) + kb * 128 + lane;
            const u16* svu = (const u16*)((g < D ? up + e * ustride : sh_up) + 2 * (size_t)H) + kb * 128 + lane;
            const u16* suh = (const u16*)(g < D ? down + e * dstride : sh_down) + kb * 128 + lane;
#pragma unroll
            for (int q = 0; q < 4; q++) { sc[q] = sz_ldg16b_here(svg + 32 * q); sc[4 + q] = sz_ldg16b_here(svu + 32 * q); sc[8 + q] = sz_ldg16b_here(suh + 32 * q); }
        };
        if (count > 0 && p < (g < D ? plan->count[g] : m)) scales();
        sz_pdl_wait();
        sz_pdl_trigger();
        uint4 piece[2];
        for (int i = 0; i < count; i++) {
            const int st = i % S, n = g < D ? plan->count[g] : m;
            if ((i == 0 || c == 0) && p < n) {
                if (i > 0) scales();
                long long raw[2][8];
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int t = p + SZ_XW_PRODUCE * r;
                    if (t < n) {
                        const long long* a = acc + (size_t)(g < D ? plan->pairs[g][t] : m * top_k + t) * 2 * FF + kb * 128 + lane;
#pragma unroll
                        for (int q = 0; q < 4; q++) { raw[r][q] = __ldcg(a + 32 * q); raw[r][4 + q] = __ldcg(a + FF + 32 * q); }
                    }
                }
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    if (p + SZ_XW_PRODUCE * r < n) {
                        float gg[4], uu[4], v[4];
#pragma unroll
                        for (int q = 0; q < 4; q++) { gg[q] = (float)((double)raw[r][q] * SZ_FIX_INV); uu[q] = (float)((double)raw[r][4 + q] * SZ_FIX_INV); }
                        sz_wht128_warp(gg, lane);
                        sz_wht128_warp(uu, lane);
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const float gv = (gg[q] * SZ_RSQRT128) * sz_f16_to_f32(sc[q]), uv = (uu[q] * SZ_RSQRT128) * sz_f16_to_f32(sc[4 + q]);
                            v[q] = (sz_silu(gv) * uv) * sz_f16_to_f32(sc[8 + q]);
                        }
                        piece[r] = sz_xw_piece(v, buf[p], lane);
                    }
                }
            }
            if (i >= S) {
                if (!sz_mbar_wait(&R.empty[st], ((i / S) - 1) & 1)) { ok = false; break; }
                if (p == SZ_XW_PRODUCE - 1) issue(i, g, kb, c);
            }
            uint4* frag = R.frags + st * 256 + (lane >> 2) * 32 + (lane & 3);
            if (p < n) frag[4 * p] = piece[0];
            if (p + SZ_XW_PRODUCE < n) frag[4 * (p + SZ_XW_PRODUCE)] = piece[1];
            __syncwarp();
            if (lane == 0) sz_mbar_arrive(&R.full[st]);
            step(g, kb, c);
        }
    } else {
        sz_pdl_wait();
        sz_pdl_trigger();
        ok = sz_xw_decode<K, TW>(R, unit, &next, count, plan, D, m, top_k, out, (size_t)H, 0, lane);
    }
    if (!ok && lane == 0) atomicExch(&ctrl[1], 1u);
}
