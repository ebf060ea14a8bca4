// The router over many rows: what sz_route_kernel computes for the rows of a pass, its logits and its choice bit for bit, for the rows of a
// step or a prompt's chunk.  Two kernels: the logits, then a warp a row for top-k and weights.
#pragma once

// ---- logits ------------------------------------------------------------------------------------------------------------------------------
// An f64 product of [router rows] x [rows] whose additions keep the pass's order.  There a thread forms a chain of 4 NCH multiply-adds (its
// float4 pieces), a warp adds its 32 chains as a butterfly (16 apart first, then 8, 4, 2, 1), and the 8 warps' sums are added in order.  Here a
// chain is NCH mma.m8n8k4 in f64 - which are multiply-adds one after the other in the order of k, checked bit for bit - for 64 outputs at once, the
// butterfly is a tree over the chains in registers (sz_rr_tree), and one warp goes through the 8 parts.
// What bounds it is the f64 pipe, 64 multiply-adds a clock and multiprocessor: 29 us for 504 rows x 513 router rows x 2,048, an eighth more for the
// tree's additions, and the conversions, which take it, too.  The f32 operands are staged 128 NCH columns at a time, two stages, and converted
// behind shared memory.  Measured with the events around it: 504 rows 59 us, 248 39 (the pass's kernel with a block row for 8 rows, which adds
// by shuffles and chooses, too: 98 and 57; where it is the sooner one: sz_route_rows_form).  Conversions by integer instructions (504 rows: 76; of the rows alone 67), or once a block into
// f64 stages (69, for want of a second stage): slower.
// A block takes 8 ME WE router rows and 8 NR WR rows of the step: WE x WR warps, a warp 8 ME router rows and 8 NR rows.
template <int NCH, int WE, int WR, int ME, int NR>
struct SzRouteRows {
    static constexpr int E = 8 * ME * WE, R = 8 * NR * WR, NT = 32 * WE * WR;
    static constexpr int STRIDE = 128 * NCH + 4;              // floats between two staged rows (4 (mod 32): the 8 rows x 4 columns a warp reads at once)
    static constexpr int SMEM = 2 * (E + R) * STRIDE * 4;
};
template <int NCH, int ME, int NR>
struct SzRouteAt { const float *w, *x; };      // the lane's element of the warp's first router row and row, chain 0

// The sums of the chains c, c + OFF', .. for the OFF' < OFF still to be added: v[tile][2].
template <int OFF, int NCH, int ME, int NR>
__device__ __forceinline__ void sz_rr_tree(const SzRouteAt<NCH, ME, NR>& at, int c, double (*v)[2]) {
    constexpr int ST = 128 * NCH + 4;
    if constexpr (OFF == 32) {
#pragma unroll
        for (int i = 0; i < ME * NR; i++) { v[i][0] = 0.0; v[i][1] = 0.0; }
#pragma unroll
        for (int u = 0; u < NCH; u++) {
            double a[ME], b[NR];
#pragma unroll
            for (int i = 0; i < ME; i++) a[i] = (double)at.w[i * 8 * ST + 128 * u + 4 * c];
#pragma unroll
            for (int i = 0; i < NR; i++) b[i] = (double)at.x[i * 8 * ST + 128 * u + 4 * c];
#pragma unroll
            for (int i = 0; i < ME; i++)
#pragma unroll
                for (int j = 0; j < NR; j++)
                    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(v[i * NR + j][0]), "+d"(v[i * NR + j][1]) : "d"(a[i]), "d"(b[j]));
        }
    } else {
        sz_rr_tree<2 * OFF, NCH, ME, NR>(at, c, v);
        double b[ME * NR][2];
        sz_rr_tree<2 * OFF, NCH, ME, NR>(at, c + OFF, b);
#pragma unroll
        for (int i = 0; i < ME * NR; i++) { v[i][0] += b[i][0]; v[i][1] += b[i][1]; }
    }
}

// grid (ceil(router rows / E), ceil(rows / R)), block 32 WE WR
template <int NCH, int WE, int WR, int ME, int NR>
__global__ void __launch_bounds__(32 * WE * WR)
sz_route_rows_kernel(const float* __restrict__ x, int H, const float* __restrict__ router, const float* __restrict__ shared_router, int ne, int rows, float* __restrict__ logits) {
    using X = SzRouteRows<NCH, WE, WR, ME, NR>;
    constexpr int E = X::E, R = X::R, ST = X::STRIDE, NT = X::NT;
    extern __shared__ __align__(16) float rr_smem[];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, q = lane & 3;
    const int nrows = ne + (shared_router != nullptr ? 1 : 0), e0 = blockIdx.x * E, r0 = blockIdx.y * R;
    // part p: the columns of the pass's warp p, 128 p + 1024 u + 0 .. 127.  Rows past the last repeat it (nobody keeps their sums), columns past the last are zero.
    auto stage = [&](int p, bool w) {
        float* d = rr_smem + (p & 1) * (E + R) * ST + (w ? 0 : E * ST);
#pragma unroll 4
        for (int i = t; i < (w ? E : R) * 32 * NCH; i += NT) {
            const int r = i / (32 * NCH), c = i % (32 * NCH), col = 128 * p + 1024 * (c >> 5) + 4 * (c & 31);
            const float* src;
            if (w) { const int e = e0 + r < nrows ? e0 + r : nrows - 1; src = e < ne ? router + (size_t)e * H : shared_router; }
            else src = x + (size_t)(r0 + r < rows ? r0 + r : rows - 1) * H;
            if (col < H) sz_cp_async16(d + r * ST + 4 * c, src + col);
            else *(float4*)(d + r * ST + 4 * c) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    stage(0, true);                       // (the router is constant: ahead of the wait)
    sz_pdl_wait();
    sz_pdl_trigger();
    stage(0, false);
    sz_cp_async_commit();
    const int we = warp / WR * 8 * ME, wr = warp % WR * 8 * NR;
    double sum[ME * NR][2];
#pragma unroll
    for (int i = 0; i < ME * NR; i++) { sum[i][0] = 0.0; sum[i][1] = 0.0; }
    for (int p = 0; p < 8; p++) {
        if (p + 1 < 8) { stage(p + 1, true); stage(p + 1, false); }
        sz_cp_async_commit();
        sz_cp_async_wait<1>();
        __syncthreads();
        const float* s = rr_smem + (p & 1) * (E + R) * ST;
        const SzRouteAt<NCH, ME, NR> at = {s + (we + g) * ST + q, s + (E + wr + g) * ST + q};
        double v[ME * NR][2];
        sz_rr_tree<1, NCH, ME, NR>(at, 0, v);
#pragma unroll
        for (int i = 0; i < ME * NR; i++) { sum[i][0] += v[i][0]; sum[i][1] += v[i][1]; }
        __syncthreads();                  // (read before the part after the next one is staged over it)
    }
#pragma unroll
    for (int i = 0; i < ME; i++)
#pragma unroll
        for (int j = 0; j < NR; j++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int e = e0 + we + 8 * i + g, r = r0 + wr + 8 * j + 2 * q + k;
                if (e < nrows && r < rows) logits[(size_t)r * (ne + 1) + e] = (float)sum[i * NR + j][k];
            }
}

// ---- top-k and weights: a warp a row -------------------------------------------------------------------------------------------------------
// As the pass's: a lane owns the experts lane, lane + 32, ..; the k-th best of the lanes' best is a floor under the k-th best logit, the keys at or
// above it (at most k lanes' worth, typically a dozen) are ranked by counting.  Keys are (orderable f32 image of logit - max, ~index).  (The chain
// of one row is 4,500 cycles, hidden here by the other warps; in a pass, where nothing hides it, this form was no faster than all threads on the rows.)
struct SzTopkRow {
    u64 best[32];
    u64 cand[SZ_MAX_TOPK * (SZ_MAX_EXPERTS / 32)];
    double ex[SZ_MAX_TOPK];
    int sel[SZ_MAX_TOPK];
};
#define SZ_RR_TW 4        // rows a block
// NK: experts a lane, at least ne / 32.  grid (ceil(rows / SZ_RR_TW)), block 32 SZ_RR_TW
template <int NK>
__global__ void __launch_bounds__(32 * SZ_RR_TW)
sz_route_topk_kernel(const float* __restrict__ logits, int ne, int k, int rows, int32_t* __restrict__ ridx, double* __restrict__ rw, int32_t* __restrict__ out_idx,
                     double* __restrict__ out_w) {
    __shared__ __align__(16) SzTopkRow tk[SZ_RR_TW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.x * SZ_RR_TW + warp;
    SzTopkRow& S = tk[warp];
    sz_pdl_wait();
    sz_pdl_trigger();
    if (row >= rows) return;
    const float* lg = logits + (size_t)row * (ne + 1);
    float lv[NK];
    float mx = -FLT_MAX;  // f32::MIN, forward.rs:1093
#pragma unroll
    for (int q = 0; q < NK; q++) lv[q] = lane + 32 * q < ne ? __ldcg(lg + lane + 32 * q) : -INFINITY;
#pragma unroll
    for (int q = 0; q < NK; q++) mx = fmaxf(mx, lv[q]);
    mx = sz_fkey_inv(__reduce_max_sync(0xffffffffu, sz_fkey(mx)));
    u64 key[NK], own = 0ull;
#pragma unroll
    for (int q = 0; q < NK; q++) {
        const int e = lane + 32 * q;
        key[q] = e < ne ? (((u64)sz_fkey(lv[q] - mx) << 32) | (u64)(0xffffffffu - (u32)e)) : 0ull;  // in f32, as the reference
        own = key[q] > own ? key[q] : own;
    }
    S.best[lane] = own;
    __syncwarp();
    int rank = 0;
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        const ulonglong2 b = *(const ulonglong2*)&S.best[i];
        rank += (b.x > own) + (b.y > own);
    }
    // the floor: keys are distinct, so exactly one lane with an expert has this rank (k <= experts)
    const u64 fl = __shfl_sync(0xffffffffu, own, __ffs(__ballot_sync(0xffffffffu, own != 0ull && rank == k - 1)) - 1);
    int C = 0;                                           // k <= C <= k * NK
#pragma unroll
    for (int q = 0; q < NK; q++) {
        const bool in = key[q] >= fl && key[q] != 0ull;
        const u32 m = __ballot_sync(0xffffffffu, in);
        if (in) S.cand[C + __popc(m & ((1u << lane) - 1u))] = key[q];
        C += __popc(m);
    }
    __syncwarp();
    for (int i = lane; i < C; i += 32) {
        const u64 c = S.cand[i];
        int r = 0;
#pragma unroll 4
        for (int q = 0; q < C; q++) r += S.cand[q] > c;
        if (r < k) { S.sel[r] = (int)(0xffffffffu - (u32)c); S.ex[r] = exp((double)sz_fkey_inv((u32)(c >> 32))); }
    }
    __syncwarp();
    if (lane >= k) return;
    // the softmax over all experts, the chosen ones renormalised: the full sum cancels (sz_route_kernel)
    double tz = 0.0;
    for (int r = 0; r < k; r++) tz += S.ex[r];
    const double wv = S.ex[lane] / tz;
    const size_t at = (size_t)row * k + lane;
    ridx[at] = S.sel[lane];
    rw[at] = wv;
    if (out_idx) out_idx[at] = S.sel[lane];
    if (out_w) out_w[at] = wv;
}
