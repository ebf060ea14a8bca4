// Many rows of one or several sequences through a layer at once: what the kernels of a pass do for up to 8 rows of one sequence, for
// the rows of a batched step and of a prompt's chunk, from tables of the sequences and of the rows.  A row's results are bit for bit
// those of the passes that would otherwise carry it: the same arithmetic, and attention in the same groups of up to 8 rows.
#pragma once

#include "sz_session_kernels.cuh"

#ifdef __CUDACC__

// grid (rows + sequences): a row's embedding into its residual streams; a sequence's staging block into its session
__global__ void __launch_bounds__(256)
sz_rows_embed_kernel(const SzSeqDev* __restrict__ seqs, const int32_t* __restrict__ ids, int rows, const u8* __restrict__ embd, int type, int H, int C, int vocab,
                     float* __restrict__ r) {
    __shared__ u32 grid[512];
    sz_pdl_wait();
    sz_pdl_trigger();
    if ((int)blockIdx.x >= rows) {
        const SzSeqDev& q = seqs[blockIdx.x - rows];
        if (threadIdx.x < 32) q.ids[threadIdx.x] = q.staged[threadIdx.x];
        return;
    }
    if (type == SZ_TYPE_IQ3_S) {
        for (int i = threadIdx.x; i < 512; i += 256) grid[i] = c_iq3s_grid[i];
        __syncthreads();
    }
    const int j = blockIdx.x;
    int tok = ids[j];
    tok = tok < 0 ? 0 : (tok >= vocab ? vocab - 1 : tok);
    const u8* row = embd + (size_t)tok * sz_dense_row_bytes(type, H);
    for (int e = 4 * threadIdx.x; e < H; e += 1024) {
        float w[4], sc;
        sz_dense_w4(type, row, e, grid, w, sc);
        const float4 v = make_float4(sc * w[0], sc * w[1], sc * w[2], sc * w[3]);
        for (int s = 0; s < C; s++) *(float4*)(r + ((size_t)j * C + s) * H + e) = v;
    }
}

// ---- the read over many rows at the usual shape (rank 256, 4 streams) -------------------------------------------------------------------
// Both halves are matrix products on the FMA pipe whose additions keep the pass's order (sz_hc_down_body, sz_hc_up_body), so what is left
// to choose is how often an operand is loaded.  Measured a launch at 256 rows (hidden 2048): first half 82 -> 68, second half 126 -> 55 us
// (80 rows: 45 -> 25), where the multiply-adds alone take 15 and 14 us of the whole chip; loads from shared memory bound both.
//
// First half.  A block takes 32 rows and 1 / gridDim.x of the C*H columns.  Its rows of rn and, 64 columns at a time in two buffers, the
// matrix sit in shared memory; a thread sums 8 outputs of 4 rows, so that a loaded word feeds four multiply-adds (with a matrix row a
// thread every input was loaded by every thread: the loads took twice the multiply-adds' time).  Per 64 columns the sums are rounded to
// fixed point as the pass's kernel rounds them and added up as integers in shared memory, and the block adds them to the accumulator
// once (128 atomics a value before, now 16).  The last block of a row tile finishes silu(down / C), so the second half reads plain
// f32.  A ninth warp takes the inject rows.  (Clusters that added up over shared memory were tried: eight blocks that must share a GPC
// left the chip in two waves, 127 us at 256 rows.)
#define SZ_HC_K 64        // columns between two roundings
#define SZ_HC_WS 144      // bytes between two staged matrix rows
#define SZ_HC_M 32        // rows a block
#define SZ_HC_TICKET 264  // the accumulator's word that counts a row tile's finished blocks (cleared with it)
static inline size_t sz_hc_down_rows_smem(int part) { return (size_t)SZ_HC_M * (part + 4) * 4 + 2 * 260 * SZ_HC_WS + (size_t)SZ_HC_M * 260 * 8; }
// a rounded to 2^-40 as __double2ll_rn((double)a * 2^40) rounds it: 1.5 * 2^12 puts the last place of the sum there
__device__ __forceinline__ long long sz_hc_fix(float a) {
    if (fabsf(a) < 2048.0f) return __double_as_longlong((double)a + 6144.0) - __double_as_longlong(6144.0);
    return __double2ll_rn((double)a * SZ_HC_FIX);
}
// grid (column parts, ceil(rows / 32)), block 288; hd: f32 [rows][256]; acc: zero on entry
__global__ void __launch_bounds__(288, 1)
sz_hc_down_rows_kernel(const float* __restrict__ rn, const u8* __restrict__ down, const u8* __restrict__ inject, int H, int rows, float* __restrict__ hd,
                       long long* __restrict__ acc) {
    constexpr int C = 4, RANK = 256, OUTS = RANK + C, M = SZ_HC_M, OT = 8, OG = RANK / OT;
    extern __shared__ __align__(128) u8 smem[];
    __shared__ int s_last;
    const int CH = C * H, part = CH / gridDim.x, xst = part + 4, k0 = blockIdx.x * part, row0 = blockIdx.y * M;
    float* xs = (float*)smem;                                               // [M][part + 4]
    u8* ws = smem + (size_t)M * xst * 4;                                    // [2][OUTS][SZ_HC_WS]
    long long* sums = (long long*)(ws + 2 * OUTS * SZ_HC_WS);               // [M][OUTS]
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int nout = inject != nullptr ? OUTS : RANK;
    auto stage = [&](int s, int buf) {      // columns s .. s + 63 of every matrix row
        for (int i = t; i < nout * 8; i += 288) {
            const int o = i >> 3;
            const u8* src = (o < RANK ? down + ((size_t)o * CH + k0 + s) * 2 : inject + ((size_t)(o - RANK) * CH + k0 + s) * 2) + 16 * (i & 7);
            sz_cp_async16(ws + (size_t)(buf * OUTS + o) * SZ_HC_WS + 16 * (i & 7), src);
        }
        sz_cp_async_commit();
    };
    stage(0, 0);                            // (constant data: ahead of the wait)
    for (int i = t; i < M * OUTS; i += 288) sums[i] = 0;
    sz_pdl_wait();
    sz_pdl_trigger();
    for (int i = t; i < M * part / 4; i += 288) {
        const int j = i / (part / 4), c = i - j * (part / 4);
        if (row0 + j < rows) sz_cp_async16(xs + (size_t)j * xst + 4 * c, rn + (size_t)(row0 + j) * CH + k0 + 4 * c);
        else *(float4*)(xs + (size_t)j * xst + 4 * c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    sz_cp_async_commit();
    // a thread's outputs og + 32 i and rows rg + 8 j
    const int og = (warp & 3) * 8 + (lane & 7), rg = (warp >> 2) * 4 + (lane >> 3);
    for (int s = 0, buf = 0; s < part; s += SZ_HC_K, buf ^= 1) {
        sz_cp_async_wait<0>();
        __syncthreads();                    // the buffer at hand has landed, and nobody reads the other any more
        if (s + SZ_HC_K < part) stage(s + SZ_HC_K, buf ^ 1);
        if (warp < 8) {
            float a[OT][4];
#pragma unroll
            for (int i = 0; i < OT; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) a[i][j] = 0.f;
            const u8* w = ws + (size_t)(buf * OUTS + og) * SZ_HC_WS;
            const float* x = xs + (size_t)rg * xst + s;
#pragma unroll 4
            for (int c = 0; c < SZ_HC_K; c += 4) {
                float4 xv[4];
#pragma unroll
                for (int j = 0; j < 4; j++) xv[j] = *(const float4*)(x + (size_t)j * 8 * xst + c);
#pragma unroll
                for (int i = 0; i < OT; i++) {
                    const uint2 q = *(const uint2*)(w + (size_t)i * OG * SZ_HC_WS + 2 * c);
                    const float f0 = __uint_as_float(q.x << 16), f1 = __uint_as_float(q.x & 0xffff0000u), f2 = __uint_as_float(q.y << 16), f3 = __uint_as_float(q.y & 0xffff0000u);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        a[i][j] = fmaf(f0, xv[j].x, a[i][j]);
                        a[i][j] = fmaf(f1, xv[j].y, a[i][j]);
                        a[i][j] = fmaf(f2, xv[j].z, a[i][j]);
                        a[i][j] = fmaf(f3, xv[j].w, a[i][j]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < OT; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) sums[(rg + 8 * j) * OUTS + og + i * OG] += sz_hc_fix(a[i][j]);
        } else if (inject != nullptr) {     // lane: stream lane & 3, rows (lane >> 2) + 8 q
            const int s4 = lane & 3;
            float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (int c = 0; c < SZ_HC_K; c += 4) {
                const uint2 p = *(const uint2*)(ws + (size_t)(buf * OUTS + RANK + s4) * SZ_HC_WS + 2 * c);
                const float f0 = __uint_as_float(p.x << 16), f1 = __uint_as_float(p.x & 0xffff0000u), f2 = __uint_as_float(p.y << 16), f3 = __uint_as_float(p.y & 0xffff0000u);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float4 xv = *(const float4*)(xs + (size_t)((lane >> 2) + 8 * q) * xst + s + c);
                    a[q] = fmaf(f0, xv.x, a[q]);
                    a[q] = fmaf(f1, xv.y, a[q]);
                    a[q] = fmaf(f2, xv.z, a[q]);
                    a[q] = fmaf(f3, xv.w, a[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; q++) sums[((lane >> 2) + 8 * q) * OUTS + RANK + s4] += sz_hc_fix(a[q]);
        }
    }
    __syncthreads();
    const int live = rows - row0 < M ? rows - row0 : M;
    for (int i = t; i < live * OUTS; i += 288) {
        const int j = i / OUTS, o = i - j * OUTS;
        if (o < nout) atomicAdd((unsigned long long*)(acc + (size_t)(row0 + j) * SZ_HC_ACC_ROWS + o), (unsigned long long)sums[i]);
    }
    __threadfence();
    __syncthreads();
    if (t == 0) s_last = atomicAdd((unsigned long long*)(acc + (size_t)row0 * SZ_HC_ACC_ROWS + SZ_HC_TICKET), 1ull) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int i = t; i < live * RANK; i += 288) {
        const int j = i / RANK, o = i - j * RANK;
        const float f = (float)((double)__ldcg(acc + (size_t)(row0 + j) * SZ_HC_ACC_ROWS + o) * SZ_HC_FIX_INV);
        hd[(size_t)(row0 + j) * RANK + o] = sz_silu(f / (float)C);
    }
}

// silu(down / C) from the accumulator, for the first half's block-row form.  grid (rows), block 256
__global__ void __launch_bounds__(256)
sz_hc_rows_act_kernel(const long long* __restrict__ acc, int C, float* __restrict__ hd) {
    sz_pdl_wait();
    sz_pdl_trigger();
    const float v = (float)((double)__ldcg(acc + (size_t)blockIdx.x * SZ_HC_ACC_ROWS + threadIdx.x) * SZ_HC_FIX_INV);
    hd[(size_t)blockIdx.x * 256 + threadIdx.x] = sz_silu(v / (float)C);
}

// Second half.  A block takes 16 hidden positions (the 64 rows of the up matrix that their 4 streams have) and 32 rows of the step; a thread
// one position and 4 rows: 16 dot products, every operand in shared memory read for four of them.  A dot product is the pass's: 32 pieces
// of 8 multiply-adds, added as the butterfly over a row's 32 lanes adds them - pieces 16 apart first, then 8, 4, 2, 1.
#define SZ_HC_UP_ROWS 32
#define SZ_HC_UP_WS 264       // halves between two rows of the staged up matrix (4 (mod 32) words: the 8 rows a warp reads at once)
#define SZ_HC_UP_XS 260       // floats between two staged rows of the step
struct SzHcUpRows { static constexpr int SMEM = 64 * SZ_HC_UP_WS * 2 + SZ_HC_UP_ROWS * SZ_HC_UP_XS * 4; };

struct SzHcUpAt { const u8* w; const float* x; };
// f(4, c) of the tree: pieces c, c + 4, .. c + 28; OFF: the first offset that is added
template <int OFF>
__device__ __forceinline__ void sz_hc_up_tree(const SzHcUpAt& at, int c, float (*v)[4]) {
    if constexpr (OFF == 32) {
        float4 x[4][2];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            x[j][0] = *(const float4*)(at.x + (size_t)j * 8 * SZ_HC_UP_XS + 8 * c);
            x[j][1] = *(const float4*)(at.x + (size_t)j * 8 * SZ_HC_UP_XS + 8 * c + 4);
        }
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const uint4 w = *(const uint4*)(at.w + (size_t)s * 16 * SZ_HC_UP_WS * 2 + 16 * c);
            const u32 ww[4] = {w.x, w.y, w.z, w.w};
            float f[8];
#pragma unroll
            for (int q = 0; q < 4; q++) { f[2 * q] = __uint_as_float(ww[q] << 16); f[2 * q + 1] = __uint_as_float(ww[q] & 0xffff0000u); }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float a = f[0] * x[j][0].x;
                a = fmaf(f[1], x[j][0].y, a); a = fmaf(f[2], x[j][0].z, a); a = fmaf(f[3], x[j][0].w, a);
                a = fmaf(f[4], x[j][1].x, a); a = fmaf(f[5], x[j][1].y, a); a = fmaf(f[6], x[j][1].z, a); a = fmaf(f[7], x[j][1].w, a);
                v[s][j] = a;
            }
        }
    } else {
        sz_hc_up_tree<2 * OFF>(at, c, v);
        float b[4][4];
        sz_hc_up_tree<2 * OFF>(at, c + OFF, b);
#pragma unroll
        for (int s = 0; s < 4; s++)
#pragma unroll
            for (int j = 0; j < 4; j++) v[s][j] += b[s][j];
    }
}
// grid (H / 16, ceil(rows / 32)), block 128
__global__ void __launch_bounds__(128, 3)
sz_hc_up_rows_kernel(const float* __restrict__ hd, const u8* __restrict__ up, const float* __restrict__ rn, int H, int rows, float* __restrict__ u) {
    constexpr int C = 4, RANK = 256;
    extern __shared__ __align__(128) u8 smem[];
    float* xs = (float*)(smem + 64 * SZ_HC_UP_WS * 2);
    const int t = threadIdx.x, h0 = blockIdx.x * 16, row0 = blockIdx.y * SZ_HC_UP_ROWS;
    for (int i = t; i < 64 * 32; i += 128) {      // row s * 16 + hl of the staged matrix, 16-byte piece i & 31
        const int lr = i >> 5;
        sz_cp_async16(smem + (size_t)lr * SZ_HC_UP_WS * 2 + 16 * (i & 31), up + ((size_t)((lr >> 4) * H + h0 + (lr & 15)) * RANK) * 2 + 16 * (i & 31));
    }
    sz_pdl_wait();
    sz_pdl_trigger();
    for (int i = t; i < SZ_HC_UP_ROWS * 64; i += 128) {
        const int j = i >> 6;
        if (row0 + j < rows) sz_cp_async16(xs + (size_t)j * SZ_HC_UP_XS + 4 * (i & 63), hd + (size_t)(row0 + j) * RANK + 4 * (i & 63));
    }
    sz_cp_async_commit();
    // a thread's position and rows: 8 positions and 4 of every 8 rows a warp
    const int warp = t >> 5, lane = t & 31, hl = (warp & 1) * 8 + (lane & 7), rg = (warp >> 1) * 4 + (lane >> 3);
    float rv[4][4];       // rn of the thread's (stream, row)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int s = 0; s < 4; s++) rv[s][j] = row0 + rg + 8 * j < rows ? __ldcg(rn + ((size_t)(row0 + rg + 8 * j) * C + s) * H + h0 + hl) : 0.f;
    sz_cp_async_wait<0>();
    __syncthreads();
    const SzHcUpAt at = {smem + (size_t)hl * SZ_HC_UP_WS * 2, xs + (size_t)rg * SZ_HC_UP_XS};
    float a[4][4] = {}, b[4][4] = {};
#pragma unroll 1
    for (int it = 0; it < 4; it++) {         // f(4, 0), f(4, 2), f(4, 1), f(4, 3)
        float v[4][4];
        sz_hc_up_tree<4>(at, it == 0 ? 0 : (it == 1 ? 2 : (it == 2 ? 1 : 3)), v);
#pragma unroll
        for (int s = 0; s < 4; s++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (it == 0) a[s][j] = v[s][j];
                else if (it == 1) a[s][j] += v[s][j];
                else if (it == 2) b[s][j] = v[s][j];
                else a[s][j] += b[s][j] + v[s][j];
            }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int row = row0 + rg + 8 * j;
        if (row < rows) {
            float m = 0.f;
#pragma unroll
            for (int s = 0; s < 4; s++) m = __fadd_rn(m, __fmul_rn(sz_sigmoid(a[s][j]), rv[s][j]));    // (rounded one by one, as the pass's kernel does)
            u[(size_t)row * H + h0 + hl] = m / (float)C;
        }
    }
}

// The DeltaNet front end over the rows of a step (sz_delta_prep_kernel's arithmetic).  grid (ceil(ch / 256), ceil(rows / SZ_PREP_ROWS)).
// What the scan reads - and a replay, when the sequence's rows may be rejected - goes to the session's buffers, of a prompt's chunk to
// the step's (xc_all, beta_all, decay_all), and a chunk's last row leaves the carried conv rows behind it in the other buffer.
// A thread takes its channel for 4 rows of the step: taps and their conversions once, a projection loaded for its own row serves the three
// after it (a row a block: 504 rows 71 -> 45 us).  K: the taps where they are the usual 4, else 0.
#define SZ_PREP_ROWS 4
template <int K>
__global__ void __launch_bounds__(256)
sz_rows_delta_prep_kernel(const SzSeqDev* __restrict__ seqs, const SzRowDev* __restrict__ rws, int rows, int di, const float* __restrict__ xin, const float* __restrict__ cw,
                          const float* __restrict__ b, const float* __restrict__ a, const float* __restrict__ a_log, const float* __restrict__ dt, int kh, int vh, int d,
                          int kr, float* __restrict__ xc_all, float* __restrict__ beta_all, float* __restrict__ decay_all) {
    constexpr int RB = SZ_PREP_ROWS, KM = K ? K : 8;
    __shared__ double sred[RB][8];
    const int k = K ? K : kr;
    const int r0 = blockIdx.y * RB, nr = min(RB, rows - r0), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kd = kh * d, ch = 2 * kd + vh * d, i = blockIdx.x * 256 + threadIdx.x;
    const bool norms = (int)blockIdx.x * 256 < 2 * kd;      // (d divides 256: a head of q or k is whole warps of one block)
    double taps[KM];
#pragma unroll
    for (int t = 0; t < KM; t++) taps[t] = i < ch && t < k ? (double)__ldg(cw + (size_t)i * k + t) : 0.0;
    sz_pdl_wait();
    sz_pdl_trigger();
    float xw[RB + KM - 1], v[RB];                            // rows r0 - (KM - 1) .. of the step; what is not of a row's sequence is not used
#pragma unroll
    for (int e = 0; e < RB + KM - 1; e++) {
        const int r = r0 - (KM - 1) + e;
        xw[e] = i < ch && r >= 0 && r < rows ? __ldcg(xin + (size_t)r * ch + i) : 0.f;
    }
#pragma unroll
    for (int e = 0; e < RB; e++) {
        v[e] = 0.f;
        if (e < nr && i < ch) {
            const SzSeqDev& q = seqs[rws[r0 + e].seq];
            const int j = rws[r0 + e].j, cur = q.state[1];
            const size_t cl = (size_t)(k - 1) * ch;
            const float* conv = (cur ? q.conv1 : q.conv0) + di * cl;
            const float own = xw[e + KM - 1];
            double last = 0.0, acc;
#pragma unroll
            for (int t = 0; t < KM; t++) if (t == k - 1) last = taps[t];
            acc = last * (double)own;
#pragma unroll
            for (int t = 0; t < KM - 1; t++)
                if (t < k - 1) {
                    const int tau = j - (k - 1) + t;
                    float prev = 0.f;
                    if (K) prev = xw[e + t];
                    else {
#pragma unroll
                        for (int w = 0; w < KM - 1; w++) if (w == KM - k + t) prev = xw[e + w];
                    }
                    if (tau < 0) prev = conv[(size_t)((k - 1) + tau) * ch + i];
                    acc += taps[t] * (double)prev;
                }
            v[e] = sz_silu((float)acc);
            if (!q.all) q.xin[((size_t)di * SZ_MAX_VERIFY + j) * ch + i] = own;
            else if (j == q.m - 1) {
                float* convw = (cur ? q.conv0 : q.conv1) + di * cl;
                const float* x = xin + (size_t)(r0 + e) * ch;
                for (int t = 0; t < k - 1; t++) {
                    const int tau = q.m - (k - 1) + t;
                    convw[(size_t)t * ch + i] = tau >= 0 ? x[(long long)(t - (k - 2)) * ch + i] : conv[(size_t)((k - 1) + tau) * ch + i];
                }
            }
        }
    }
    if (norms) {
#pragma unroll
        for (int e = 0; e < RB; e++) {
            const double sq = sz_warp_sum((double)v[e] * (double)v[e]);
            if (lane == 0) sred[e][warp] = sq;
        }
        __syncthreads();
    }
    for (int e = 0; e < nr; e++) {
        const SzSeqDev& q = seqs[rws[r0 + e].seq];
        const int j = rws[r0 + e].j;
        float out = e == 0 ? v[0] : (e == 1 ? v[1] : (e == 2 ? v[2] : v[3]));
        if (i < ch) {
            if (i < 2 * kd) {
                const int w0 = (threadIdx.x / d) * (d / 32);
                double ss = 0.0;
                for (int t = 0; t < d / 32; t++) ss += sred[e][w0 + t];
                const double n = sz_rsqrt64(ss + 1e-6);
                float t = (float)((double)out * n);
                if (i < kd) t = t / sqrtf((float)d);
                out = t;
            }
            (q.all ? xc_all + (size_t)(r0 + e) * ch : q.xc + ((size_t)di * SZ_MAX_VERIFY + j) * ch)[i] = out;
        }
        if (blockIdx.x == 0) {
            const int r = r0 + e;
            float* beta = q.all ? beta_all + (size_t)r * vh : q.beta + ((size_t)di * SZ_MAX_VERIFY + j) * vh;
            float* decay = q.all ? decay_all + (size_t)r * vh : q.decay + ((size_t)di * SZ_MAX_VERIFY + j) * vh;
            for (int h = threadIdx.x; h < vh; h += 256) {
                beta[h] = sz_sigmoid(b[(size_t)r * vh + h]);
                const float sp_in = a[(size_t)r * vh + h] + dt[h];
                const float sp = sp_in > 20.0f ? sp_in : log1pf(expf(sp_in));
                decay[h] = expf(a_log[h] * sp);
            }
        }
    }
}

// The scans of a layer for the sequences of a step, after sz_rows_delta_prep_kernel.  grid (vh * D / 32, sequences)
template <int D>
__global__ void __cluster_dims__(D / 32, 1, 1) __launch_bounds__(D)
sz_rows_scan_kernel(const SzSeqDev* __restrict__ seqs, int di, const float* __restrict__ xc_all, const float* __restrict__ beta_all, const float* __restrict__ decay_all,
                    const float* __restrict__ z, const float* __restrict__ norm_w, int kh, int vh, float eps, float* __restrict__ og) {
    __shared__ SzScanSeq q;
    if (threadIdx.x == 0) {
        const SzSeqDev& s = seqs[blockIdx.y];
        const int ch = (2 * kh + vh) * D, vd = vh * D;
        const size_t Sl = (size_t)vh * D * D * di, at = (size_t)di * SZ_MAX_VERIFY;
        q.xc = s.all ? xc_all + (size_t)s.off * ch : s.xc + at * ch;
        q.beta = s.all ? beta_all + (size_t)s.off * vh : s.beta + at * vh;
        q.decay = s.all ? decay_all + (size_t)s.off * vh : s.decay + at * vh;
        q.z = z + (size_t)s.off * vd;
        q.S0 = s.S0 + Sl; q.S1 = s.S1 + Sl; q.O0 = s.S0 + Sl; q.O1 = s.S1 + Sl;
        q.state = s.state; q.res = s.res;
        q.og = og + (size_t)s.off * vd;
        q.pp.xin = nullptr;
        q.m = s.m;
    }
    __syncthreads();
    sz_delta_scan_body<D, 32>(q, norm_w, kh, vh, eps, (const SzTree*)nullptr, (float*)nullptr, (int)blockIdx.x / (D / 32), (int)blockIdx.x % (D / 32), 0);
}

// After a step: the sequences whose rows were all kept move on, and what a kernel over all rows raised in the step's error word becomes
// every sequence's own (it stays there until the session is reset; the step's word is ready for whoever has the room next).  One block.
__global__ void sz_rows_commit_kernel(const SzSeqDev* __restrict__ seqs, int n, u32* __restrict__ err) {
    sz_pdl_wait();
    sz_pdl_trigger();
    const int b = threadIdx.x;
    const u32 e = __ldcg(err);
    if (b < n) {
        int32_t* state = const_cast<int32_t*>(seqs[b].state);
        if (e) atomicOr((u32*)state + 2, e);
        if (seqs[b].all) {
            state[0] += seqs[b].m;
            state[1] ^= 1;
        }
    }
    __syncthreads();
    if (b == 0 && e) *err = 0u;
}

#endif
