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
// to choose is how often an operand is loaded.
//
// First half.  A block takes 32 rows and 32 of the 256 outputs over 1 / gridDim.y of the C*H columns; its warps share the columns, 64 at a
// time, each with two buffers of its own (32 columns by asynchronous copies) and no barrier between them: per 64 columns the sums are rounded to fixed
// point as the pass's kernel rounds them, and integers may be added in any order - in registers, at the end over the warps, and over
// gridDim.y blocks by atomics where a launch of few rows needs them to fill the chip.  A thread sums 8 outputs of 4 rows, two outputs an
// instruction (fma.rn.f32x2: each half is the pass's multiply-add).  silu(down / C) is finished here, so the second half reads plain f32.  The
// inject rows are dealt out: block j of a row tile's eight sums those of rows 4 j .. 4 j + 3, a chain a lane.
// Measured (us a launch, events between the launches; 32 rows x all outputs a block over a sixteenth of the columns -> this): 504 rows 118 -> 86,
// 264 68 -> 53; against a thread a matrix row, 8 rows a block and a launch for silu: 80 rows 34 + 6 -> 27.  The multiply-adds alone would take 30 us
// at 504 rows; what bounds it is the loop over them (plain multiply-adds instead of pairs: 99; without rounding 82; with no copies after the
// first the same; 8 warps instead of 12: 91).  More columns a block and atomics between more blocks were tried first: the atomics (2 M of
// them at the end of a launch) cost what the fuller chip gave.
#define SZ_HC_K 64        // columns between two roundings
#define SZ_HC_W 12        // warps a block
#define SZ_HC_S 32        // columns a stage
#define SZ_HC_WS (2 * SZ_HC_S + 16)      // bytes between two staged matrix rows
#define SZ_HC_XS (4 * SZ_HC_S + 16)      // bytes between two staged rows of the step
#define SZ_HC_M 32        // rows a block
#define SZ_HC_N 32        // outputs a block
#define SZ_HC_TICKET 264  // the accumulator's words that count a tile's finished blocks, a word a tile of outputs (cleared with it)
#define SZ_HC_STAGE (SZ_HC_M * SZ_HC_XS + (SZ_HC_N + 4) * SZ_HC_WS)
struct SzHcDownRows { static constexpr int SMEM = SZ_HC_W * 2 * SZ_HC_STAGE; };
__device__ __forceinline__ void sz_fma2(u64& a, u64 f, u64 x) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(f), "l"(x)); }
__device__ __forceinline__ u64 sz_mul2(u64 a, u64 b) { u64 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ u64 sz_add2(u64 a, u64 b) { u64 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ u64 sz_pack2(u32 a, u32 b) { u64 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(a), "r"(b)); return d; }
// grid (8 row tiles, column parts), block 32 SZ_HC_W; hd: f32 [rows][256]; acc: zero on entry
__global__ void __launch_bounds__(32 * SZ_HC_W, 1)
sz_hc_down_rows_kernel(const float* __restrict__ rn, const u8* __restrict__ down, const u8* __restrict__ inject, int H, int rows, float* __restrict__ hd,
                       long long* __restrict__ acc) {
    constexpr int C = 4, RANK = 256, NT = RANK / SZ_HC_N;
    extern __shared__ __align__(128) u8 smem[];
    __shared__ u64 isums[SZ_HC_W][16];
    __shared__ int s_last;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int CH = C * H, NK = CH / SZ_HC_K, P = gridDim.y;
    const int row0 = (int)blockIdx.x / NT * SZ_HC_M, nt = (int)blockIdx.x % NT, n0 = nt * SZ_HC_N;
    const int k0 = NK * (int)blockIdx.y / P, k1 = NK * ((int)blockIdx.y + 1) / P;     // the block's pieces of 64 columns; a warp takes every SZ_HC_W-th
    u8* mine = smem + (size_t)warp * 2 * SZ_HC_STAGE;
    const bool injects = inject != nullptr;
    // a warp's stages: number i is half i & 1 of its piece i >> 1, in buffer i & 1
    const int NI = k0 + warp < k1 ? 2 * ((k1 - k0 - warp + SZ_HC_W - 1) / SZ_HC_W) : 0;
    auto col = [&](int i) { return (k0 + warp + (i >> 1) * SZ_HC_W) * SZ_HC_K + (i & 1) * SZ_HC_S; };
    auto stage_w = [&](int i) {
        u8* d = mine + (i & 1) * SZ_HC_STAGE + SZ_HC_M * SZ_HC_XS;
        const u8* src = down + ((size_t)(n0 + (lane >> 2)) * CH + col(i)) * 2 + 16 * (lane & 3);
#pragma unroll
        for (int q = 0; q < SZ_HC_N / 8; q++) sz_cp_async16(d + (8 * q + (lane >> 2)) * SZ_HC_WS + 16 * (lane & 3), src + (size_t)q * 16 * CH);
        if (injects && lane < 16) sz_cp_async16(d + (SZ_HC_N + (lane >> 2)) * SZ_HC_WS + 16 * (lane & 3), inject + ((size_t)(lane >> 2) * CH + col(i)) * 2 + 16 * (lane & 3));
    };
    auto stage_x = [&](int i) {                     // (rows past the last one repeat it; nobody keeps their sums)
        u8* d = mine + (i & 1) * SZ_HC_STAGE + 16 * (lane & 7);
        const float* src = rn + col(i) + 4 * (lane & 7);
#pragma unroll
        for (int q = 0; q < SZ_HC_M / 4; q++) {
            const int r = 4 * q + (lane >> 3), row = row0 + r < rows ? row0 + r : rows - 1;
            sz_cp_async16(d + r * SZ_HC_XS, src + (size_t)row * CH);
        }
    };
    if (NI) stage_w(0);                             // (constant data: ahead of the wait)
    sz_pdl_wait();
    sz_pdl_trigger();
    if (NI) stage_x(0);
    sz_cp_async_commit();
    // a thread's outputs og + 4 i and rows rg + 8 j; inject row lane & 3 of row 4 nt + (lane >> 2) (lanes 0 .. 15)
    const int og = lane & 3, rg = lane >> 2;
    u64 sum[32], isum = 0, added = 0;               // [4 pairs of outputs][4 rows][2]
#pragma unroll
    for (int i = 0; i < 32; i++) sum[i] = 0;
    u64 a[4][4];
    float b = 0.f;
    for (int i = 0; i < NI; i++) {
        if (i + 1 < NI) { stage_w(i + 1); stage_x(i + 1); }
        sz_cp_async_commit();
        sz_cp_async_wait<1>();
        __syncwarp();
        const u8* st = mine + (i & 1) * SZ_HC_STAGE;
        const u8* x = st + rg * SZ_HC_XS;
        const u8* w = st + SZ_HC_M * SZ_HC_XS + og * SZ_HC_WS;
        if (!(i & 1)) {
#pragma unroll
            for (int p = 0; p < 4; p++)
#pragma unroll
                for (int j = 0; j < 4; j++) a[p][j] = 0ull;
            b = 0.f;
        }
#pragma unroll 4
        for (int c = 0; c < SZ_HC_S; c += 4) {
            uint2 q[8];
            uint4 xv[4];
#pragma unroll
            for (int j = 0; j < 4; j++) xv[j] = *(const uint4*)(x + j * 8 * SZ_HC_XS + 4 * c);
#pragma unroll
            for (int i = 0; i < 8; i++) q[i] = *(const uint2*)(w + i * 4 * SZ_HC_WS + 2 * c);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                u64 f[4], xd[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const u32 lo = e < 2 ? q[2 * i].x : q[2 * i].y, hi = e < 2 ? q[2 * i + 1].x : q[2 * i + 1].y;
                    f[i] = e & 1 ? sz_pack2(lo & 0xffff0000u, hi & 0xffff0000u) : sz_pack2(lo << 16, hi << 16);
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const u32 v = e == 0 ? xv[j].x : (e == 1 ? xv[j].y : (e == 2 ? xv[j].z : xv[j].w));
                    xd[j] = sz_pack2(v, v);
                }
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) sz_fma2(a[i][j], f[i], xd[j]);
            }
        }
        if (injects && lane < 16) {
            const u8* xi = st + (4 * nt + (lane >> 2)) * SZ_HC_XS;
            const u8* wi = st + SZ_HC_M * SZ_HC_XS + (SZ_HC_N + og) * SZ_HC_WS;
#pragma unroll
            for (int c = 0; c < SZ_HC_S; c += 4) {
                const uint2 q = *(const uint2*)(wi + 2 * c);
                const float4 v = *(const float4*)(xi + 4 * c);
                b = fmaf(__uint_as_float(q.x << 16), v.x, b);
                b = fmaf(__uint_as_float(q.x & 0xffff0000u), v.y, b);
                b = fmaf(__uint_as_float(q.y << 16), v.z, b);
                b = fmaf(__uint_as_float(q.y & 0xffff0000u), v.w, b);
            }
        }
        if (i & 1) {
            sz_hc_round<16>(&a[0][0], sum);
            added++;
            isum += sz_hc_fix(b);
        }
        __syncwarp();                               // the buffer is read before the copies after the next ones fill it
    }
    // ---- over the warps: [row][output] of a warp's sums where its buffers were
    sz_cp_async_wait<0>();
    __syncwarp();
    u64* red = (u64*)mine;
#pragma unroll
    for (int i = 0; i < 32; i++) {
        const int o = og + 4 * (2 * (i >> 3) + (i & 1)), r = rg + 8 * ((i >> 1) & 3);
        red[r * (SZ_HC_N + 1) + o] = sum[i] - added * SZ_HC_MAGIC;
    }
    if (lane < 16) isums[warp][lane] = isum;
    __syncthreads();
    if (injects && t < 16 && row0 + 4 * nt + (t >> 2) < rows) {
        u64 v = 0;
#pragma unroll
        for (int q = 0; q < SZ_HC_W; q++) v += isums[q][t];
        atomicAdd((unsigned long long*)(acc + (size_t)(row0 + 4 * nt + (t >> 2)) * SZ_HC_ACC_ROWS + RANK + (t & 3)), (unsigned long long)v);
    }
    const int live = warp < 8 ? rows - row0 : 0;
    // thread: output lane of rows warp, warp + 8, ..
    u64 v[4] = {0, 0, 0, 0};
    if (warp < 8) {
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int q = 0; q < SZ_HC_W; q++) v[j] += *(const u64*)(smem + (size_t)q * 2 * SZ_HC_STAGE + ((warp + 8 * j) * (SZ_HC_N + 1) + lane) * 8);
    }
    long long* at = acc + (size_t)(row0 + warp) * SZ_HC_ACC_ROWS + n0 + lane;
    if (P > 1) {
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (warp + 8 * j < live) atomicAdd((unsigned long long*)(at + (size_t)8 * j * SZ_HC_ACC_ROWS), (unsigned long long)v[j]);
        __threadfence();
        __syncthreads();
        if (t == 0) s_last = atomicAdd((unsigned long long*)(acc + (size_t)row0 * SZ_HC_ACC_ROWS + SZ_HC_TICKET + nt), 1ull) == (unsigned long long)(P - 1);
        __syncthreads();
        if (!s_last) return;
        __threadfence();
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (warp + 8 * j < live) v[j] = (u64)__ldcg(at + (size_t)8 * j * SZ_HC_ACC_ROWS);
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (warp + 8 * j < live) hd[(size_t)(row0 + warp + 8 * j) * RANK + n0 + lane] = sz_silu((float)((double)(long long)v[j] * SZ_HC_FIX_INV) / (float)C);
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
// one position and 4 rows: 16 dot products, two streams an instruction, every operand in shared memory read for four of them (one stream an
// instruction: 504 rows 92 us a launch, now 72; 264 57 -> 45, 80 24.7 -> 22.7; the multiply-adds alone would take 30 us at 504 rows).  A dot product is the pass's: 32 pieces
// of 8 multiply-adds, added as the butterfly over a row's 32 lanes adds them - pieces 16 apart first, then 8, 4, 2, 1.
#define SZ_HC_UP_ROWS 32
#define SZ_HC_UP_WS 264       // halves between two rows of the staged up matrix (4 (mod 32) words: the 8 rows a warp reads at once)
#define SZ_HC_UP_XS 260       // floats between two staged rows of the step
struct SzHcUpRows { static constexpr int SMEM = 64 * SZ_HC_UP_WS * 2 + SZ_HC_UP_ROWS * SZ_HC_UP_XS * 4; };

struct SzHcUpAt { const u8* w; const float* x; };
// f(4, c) of the tree: pieces c, c + 4, .. c + 28; OFF: the first offset that is added.  v[p][j]: streams 2 p and 2 p + 1 of row j, two an instruction.
template <int OFF>
__device__ __forceinline__ void sz_hc_up_tree(const SzHcUpAt& at, int c, u64 (*v)[4]) {
    if constexpr (OFF == 32) {
        uint4 x[4][2];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            x[j][0] = *(const uint4*)(at.x + (size_t)j * 8 * SZ_HC_UP_XS + 8 * c);
            x[j][1] = *(const uint4*)(at.x + (size_t)j * 8 * SZ_HC_UP_XS + 8 * c + 4);
        }
        uint4 w[4];
#pragma unroll
        for (int s = 0; s < 4; s++) w[s] = *(const uint4*)(at.w + (size_t)s * 16 * SZ_HC_UP_WS * 2 + 16 * c);
#pragma unroll
        for (int e = 0; e < 8; e++) {
            u64 f[2], xd[4];
#pragma unroll
            for (int p = 0; p < 2; p++) {
                const u32* lo = (const u32*)&w[2 * p] + (e >> 1);
                const u32* hi = (const u32*)&w[2 * p + 1] + (e >> 1);
                f[p] = e & 1 ? sz_pack2(*lo & 0xffff0000u, *hi & 0xffff0000u) : sz_pack2(*lo << 16, *hi << 16);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const u32 q = *((const u32*)&x[j][e >> 2] + (e & 3));
                xd[j] = sz_pack2(q, q);
            }
#pragma unroll
            for (int p = 0; p < 2; p++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (e == 0) v[p][j] = sz_mul2(f[p], xd[j]);
                    else sz_fma2(v[p][j], f[p], xd[j]);
                }
        }
    } else {
        sz_hc_up_tree<2 * OFF>(at, c, v);
        u64 b[2][4];
        sz_hc_up_tree<2 * OFF>(at, c + OFF, b);
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int j = 0; j < 4; j++) v[p][j] = sz_add2(v[p][j], b[p][j]);
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
    u64 a[2][4] = {}, b[2][4] = {};
#pragma unroll 1
    for (int it = 0; it < 4; it++) {         // f(4, 0), f(4, 2), f(4, 1), f(4, 3)
        u64 v[2][4];
        sz_hc_up_tree<4>(at, it == 0 ? 0 : (it == 1 ? 2 : (it == 2 ? 1 : 3)), v);
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (it == 0) a[p][j] = v[p][j];
                else if (it == 1) a[p][j] = sz_add2(a[p][j], v[p][j]);
                else if (it == 2) b[p][j] = v[p][j];
                else a[p][j] = sz_add2(a[p][j], sz_add2(b[p][j], v[p][j]));
            }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int row = row0 + rg + 8 * j;
        if (row < rows) {
            float m = 0.f;
#pragma unroll
            for (int s = 0; s < 4; s++) m = __fadd_rn(m, __fmul_rn(sz_sigmoid(__uint_as_float((u32)(a[s >> 1][j] >> (32 * (s & 1))))), rv[s][j]));    // (rounded one by one, as the pass's kernel does)
            u[(size_t)row * H + h0 + hl] = m / (float)C;
        }
    }
}

// The DeltaNet front end over the rows of a step (sz_delta_prep_kernel's arithmetic).  grid (ceil(ch / 256), ceil(rows / SZ_PREP_ROWS)).
// What the scan reads goes to the step's buffers (xc_all, beta_all, decay_all), what a replay reads - of rows that may be rejected - to the
// session's, too, and the last row of a prompt's chunk leaves the carried conv rows behind it in the other buffer.
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
            if (j >= q.keep) q.xin[((size_t)di * SZ_MAX_VERIFY + j - q.keep) * ch + i] = own;
            else if (j == q.keep - 1) {
                float* convw = (cur ? q.conv0 : q.conv1) + di * cl;
                const float* x = xin + (size_t)(r0 + e) * ch;
                for (int t = 0; t < k - 1; t++) {
                    const int tau = q.keep - (k - 1) + t;
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
            xc_all[(size_t)(r0 + e) * ch + i] = out;
            if (j >= q.keep) q.xc[((size_t)di * SZ_MAX_VERIFY + j - q.keep) * ch + i] = out;
        }
        if (blockIdx.x == 0) {
            const int r = r0 + e;
            for (int h = threadIdx.x; h < vh; h += 256) {
                const float bt = sz_sigmoid(b[(size_t)r * vh + h]);
                const float sp_in = a[(size_t)r * vh + h] + dt[h];
                const float sp = sp_in > 20.0f ? sp_in : log1pf(expf(sp_in));
                const float dc = expf(a_log[h] * sp);
                beta_all[(size_t)r * vh + h] = bt; decay_all[(size_t)r * vh + h] = dc;
                if (j >= q.keep) {
                    const size_t at = ((size_t)di * SZ_MAX_VERIFY + j - q.keep) * vh + h;
                    q.beta[at] = bt; q.decay[at] = dc;
                }
            }
        }
    }
}

// The scans of a layer for the sequences of a step, after sz_rows_delta_prep_kernel: sz_delta_scan_body's recurrence, its sums in the same
// order, for any number of rows one after the other.  What bounds a lone prompt's launch is the chain of a row (128 blocks, a warp a
// scheduler), so everything that is not the chain is kept off it:
//   - a column's D / 32 threads sit in one warp, 32 of the state's D rows in each, and add their runs by shuffles: no barrier, no trip through
//     shared memory, and the warps of a block go at their own pace;
//   - the two runs of a thread are the halves of packed instructions (mul, fma, add.rn.f32x2: each half rounded as the plain one), which take half
//     the issue slots; the k and q of a row lie interleaved in shared memory, so that a 16-byte read is two operand pairs;
//   - the output products of a row run beside the next row's k products; runs of 8 rows are added up at once, and left unnormed: the gated
//     norm over a head's D outputs is sz_rows_gate_kernel's, not eight f64 chains a stage inside this one;
//   - a fifth warp keeps SZ_RS_STAGES stages of 8 rows' operands on their way.
// Measured (128 x 128 states, 32 heads; us a launch, events between the launches): 504 rows of one prompt 298 -> 164 and 10 for the gate, which
// packs the rows as a launch of 7 did before; 80 rows of 32 sequences 63 -> 47 and 8.  MINB: blocks a multiprocessor that the registers leave room
// for - 2 where no more come (three: 186 for one prompt), 3 for many sequences (two: 57 for the 32).  A row takes some 800 cycles: 300 the products with
// the reads of its operands, 270 the sum (two conversions of 27 cycles, ten f64 operations of 8, two shuffles), 105 the update, 115 a row's share of a
// stage.  The next row's k in registers of its own, its reads in a fixed order, or conversions by integer instructions: 179 - 190 for one prompt.
// grid (vh * D / 32, sequences), block D + 32
#define SZ_RS_STAGES 3
#define SZ_RS_SEG 36          // floats between the 32 k (or q) of one thread of a column and the next one's (32, kept out of each other's banks)
template <int D>
struct SzRowsScan {
    float k[SZ_RS_STAGES][SZ_SCAN_RC][D / 32 * SZ_RS_SEG], q[SZ_RS_STAGES][SZ_SCAN_RC][D / 32 * SZ_RS_SEG], v[SZ_RS_STAGES][SZ_SCAN_RC][32];
    float beta[SZ_RS_STAGES][SZ_SCAN_RC], decay[SZ_RS_STAGES][SZ_SCAN_RC];
    float orun[SZ_SCAN_RC][D / 16][36];          // the outputs' runs (36: a warp writes its columns' of D / 32 runs at once)
    u64 full[SZ_RS_STAGES], empty[SZ_RS_STAGES];
    u64 nz2;                                     // two floats, -0
};
template <int D, int MINB>
__global__ void __launch_bounds__(D + 32, MINB)
sz_rows_scan_kernel(const SzSeqDev* __restrict__ seqs, int di, const float* __restrict__ xc_all, const float* __restrict__ beta_all, const float* __restrict__ decay_all,
                    int kh, int vh, float* __restrict__ og, u32* __restrict__ err) {
    constexpr int NW = D / 32, CW = 32 / NW, RC = SZ_SCAN_RC, ST = SZ_RS_STAGES;     // warps that scan (and threads a column); columns a warp
    __shared__ __align__(16) SzRowsScan<D> sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, hd = blockIdx.x / (D / 32), cb = blockIdx.x % (D / 32);
    const int ch = (2 * kh + vh) * D, vd = vh * D, kx = hd % kh;      // value heads are tiled over the key heads
    if (threadIdx.x == 0) {
        for (int i = 0; i < ST; i++) { sz_mbar_init(&sh.full[i], 1); sz_mbar_init(&sh.empty[i], NW); }
        sz_mbar_fence_init();
        *(volatile u64*)&sh.nz2 = 0x8000000080000000ull;
    }
    const SzSeqDev& sq = seqs[blockIdx.y];
    const int rows = sq.m, off = sq.off, cur = sq.state[1];     // (the buffers change places at the end of a step only)
    const int rq = lane / CW, cl = (warp % NW) * CW + lane % CW;       // the thread's rows 32 rq .. of the state, and its column of the block's 32
    const size_t Sat = ((size_t)di * vh + hd) * D * D + (size_t)(rq * 32) * D + cb * 32 + cl;
    u64 S[16];                   // rows i and 16 + i of the thread's
    if (warp < NW) {
        const float* Sg = (cur ? sq.S1 : sq.S0) + Sat;
#pragma unroll
        for (int i = 0; i < 16; i++) S[i] = sz_pack2(__float_as_uint(sz_ld32_here(Sg + (size_t)i * D)), __float_as_uint(sz_ld32_here(Sg + (size_t)(16 + i) * D)));
    }
    __syncthreads();
    sz_pdl_wait();
    sz_pdl_trigger();
    const int sets = (rows + RC - 1) / RC;
    if (warp == NW) {
        // ---- the operands' warp
        const float* x = xc_all + (size_t)off * ch;
        const float *be = beta_all + (size_t)off * vh + hd, *de = decay_all + (size_t)off * vh + hd;
        float4 qv[RC], kv[RC];
        float vv[RC], bv = 0.f, dv = 0.f;
        auto load = [&](int c0) {
#pragma unroll
            for (int j = 0; j < RC; j++)
                if (c0 + j < rows) {
                    const float* xr = x + (size_t)(c0 + j) * ch;
                    if (lane < D / 4) { qv[j] = __ldcg((const float4*)(xr + kx * D) + lane); kv[j] = __ldcg((const float4*)(xr + (kh + kx) * D) + lane); }
                    vv[j] = __ldcg(xr + 2 * kh * D + hd * D + cb * 32 + lane);
                }
            if (lane < RC && c0 + lane < rows) { bv = __ldcg(be + (size_t)(c0 + lane) * vh); dv = __ldcg(de + (size_t)(c0 + lane) * vh); }
        };
        // element e of piece `lane`: row 4 lane + e, so half (row / 16) & 1 of pair row & 15 of thread row / 32
        const int to = (lane >> 3) * SZ_RS_SEG + 8 * (lane & 3) + ((lane >> 2) & 1);
        load(0);
        for (int c = 0; c < sets; c++) {
            const int st = c % ST;
            if (c >= ST && !sz_mbar_wait_warp(&sh.empty[st], ((c / ST) - 1) & 1)) { if (lane == 0) atomicExch(err, 1u); return; }
#pragma unroll
            for (int j = 0; j < RC; j++)
                if (c * RC + j < rows) {
                    if (lane < D / 4) {
                        const float qe[4] = {qv[j].x, qv[j].y, qv[j].z, qv[j].w}, ke[4] = {kv[j].x, kv[j].y, kv[j].z, kv[j].w};
#pragma unroll
                        for (int e = 0; e < 4; e++) { sh.q[st][j][to + 2 * e] = qe[e]; sh.k[st][j][to + 2 * e] = ke[e]; }
                    }
                    sh.v[st][j][lane] = vv[j];
                }
            if (lane < RC) { sh.beta[st][lane] = bv; sh.decay[st][lane] = dv; }
            __syncwarp();
            if (lane == 0) sz_mbar_arrive(&sh.full[st]);
            if (c + 1 < sets) load((c + 1) * RC);
        }
        return;
    }
    // the state goes to the other buffer; where a pass follows the chunk, the chunk's does - it is the pass's to start from - and the pass's to this one
    auto leave = [&](bool other) {
        float* So = ((cur != 0) == other ? sq.S0 : sq.S1) + Sat;
#pragma unroll
        for (int i = 0; i < 16; i++) { So[(size_t)i * D] = __uint_as_float((u32)S[i]); So[(size_t)(16 + i) * D] = __uint_as_float((u32)(S[i] >> 32)); }
    };
    const int chunk = sq.keep < rows ? sq.keep : 0;
    float* o = og + (size_t)off * vd + hd * D + cb * 32;
    u64 kr[16], qr[16], nz2;
    nz2 = *(volatile u64*)&sh.nz2;
    for (int c = 0; c < sets; c++) {
        const int st = c % ST, nr = rows - c * RC < RC ? rows - c * RC : RC;
        if (!sz_mbar_wait_warp(&sh.full[st], (c / ST) & 1)) { if (lane == 0) atomicExch(err, 1u); return; }
        const float (*ks)[D / 32 * SZ_RS_SEG] = sh.k[st], (*qs)[D / 32 * SZ_RS_SEG] = sh.q[st];
        auto pairs = [&](const float* row, u64* to) {
#pragma unroll
            for (int i = 0; i < 8; i++) { const ulonglong2 p = *(const ulonglong2*)(row + rq * SZ_RS_SEG + 4 * i); to[2 * i] = p.x; to[2 * i + 1] = p.y; }
        };
        pairs(ks[0], kr);
        float dc = sh.decay[st][0], bt = sh.beta[st][0], vj = sh.v[st][0][cl];
        auto keep_runs = [&](int jj, u64 r) {
            sh.orun[jj][2 * rq][cl] = __uint_as_float((u32)r);
            sh.orun[jj][2 * rq + 1][cl] = __uint_as_float((u32)(r >> 32));
        };
        for (int jj = 0; jj < nr; jj++) {
            const u64 dc2 = sz_pack2(__float_as_uint(dc), __float_as_uint(dc));
            u64 r = 0, out = 0;
            if (jj > 0) {                          // with the output products of the row before
#pragma unroll
                for (int i = 0; i < 16; i++) { sz_fma2(out, S[i], qr[i]); S[i] = sz_mul2(S[i], dc2); sz_fma2(r, S[i], kr[i]); }
            } else {
#pragma unroll
                for (int i = 0; i < 16; i++) { S[i] = sz_mul2(S[i], dc2); sz_fma2(r, S[i], kr[i]); }
            }
            const float r0 = __uint_as_float((u32)r), r1 = __uint_as_float((u32)(r >> 32));
            // the column's sum: parts of four runs, each ((0 + r) + r) + r) + r in f64 over two threads, the parts in order
            const double a = (double)(0.f + r0) + (double)r1;      // (an f32 sum with zero is exact)
            const double b = (__shfl_xor_sync(0xffffffffu, a, CW) + (double)r0) + (double)r1;      // the second thread of a part has it
            double tot = 0.0;
#pragma unroll
            for (int p = 0; p < D / 64; p++) tot += __shfl_sync(0xffffffffu, b, (2 * p + 1) * CW + lane % CW);
            if (jj > 0) keep_runs(jj - 1, out);
            pairs(qs[jj], qr);
            const float dl = (float)(((double)vj - tot) * (double)bt);
            const u64 dl2 = sz_pack2(__float_as_uint(dl), __float_as_uint(dl));
#pragma unroll
            for (int i = 0; i < 16; i++) {      // rounded twice, as the CPU reference does (the compiler makes a packed mul and add one instruction, even with .rn; k dl + a -0 that it cannot see, not)
                u64 kd = nz2;
                sz_fma2(kd, kr[i], dl2);
                S[i] = sz_add2(S[i], kd);
            }
            const int nx = jj + 1 < nr ? jj + 1 : jj;
            pairs(ks[nx], kr);
            dc = sh.decay[st][nx]; bt = sh.beta[st][nx]; vj = sh.v[st][nx][cl];
        }
        u64 out = 0;
#pragma unroll
        for (int i = 0; i < 16; i++) sz_fma2(out, S[i], qr[i]);
        keep_runs(nr - 1, out);
        __syncwarp();
        if (lane == 0) sz_mbar_arrive(&sh.empty[st]);
        // the outputs of the warp's columns: a thread adds the runs of every NW-th row
#pragma unroll
        for (int e = 0; e < RC / NW; e++) {
            const int jj = rq + NW * e;
            if (jj < nr) {
                double tot = 0.0;
#pragma unroll
                for (int p = 0; p < D / 64; p++) {
                    double s = 0.0;
#pragma unroll
                    for (int i = 0; i < 4; i++) s += (double)sh.orun[jj][4 * p + i][cl];
                    tot += s;
                }
                o[(size_t)(c * RC + jj) * vd + cl] = (float)tot;
            }
        }
        __syncwarp();            // (read before the next rows' runs are written)
        if ((c + 1) * RC == chunk) leave(true);
    }
    leave(chunk == 0);
}

// The scan's outputs through the gated RMS norm of their head (sz_delta_scan_body's `finish`), a warp a (row, value head): into xh as the
// output projection's f16 high and low parts (sz_dense_rows_pack_kernel's) or, where that takes another form, in place.
// grid (rows * vh / 8), block 256
template <int D>
__global__ void __launch_bounds__(256)
sz_rows_gate_kernel(float* __restrict__ og, const float* __restrict__ z, const float* __restrict__ norm_w, int rows, int vh, float eps, int padded, __half* __restrict__ xh) {
    const int lane = threadIdx.x & 31, item = blockIdx.x * 8 + (threadIdx.x >> 5);
    float nw[D / 32];
#pragma unroll
    for (int i = 0; i < D / 32; i++) nw[i] = __ldg(norm_w + lane + 32 * i);
    sz_pdl_wait();
    sz_pdl_trigger();
    if (item >= rows * vh) return;
    const size_t at = (size_t)item * D + lane;
    float o[D / 32], zv[D / 32];
#pragma unroll
    for (int i = 0; i < D / 32; i++) { o[i] = __ldcg(og + at + 32 * i); zv[i] = __ldcg(z + at + 32 * i); }
    double ss = 0.0;
#pragma unroll
    for (int i = 0; i < D / 32; i++) ss += (double)o[i] * (double)o[i];
    ss = sz_warp_sum(ss);
    const double rr = sz_rsqrt64(ss / (double)D + (double)eps);
#pragma unroll
    for (int i = 0; i < D / 32; i++) {
        const float y = __fmul_rn((float)((double)o[i] * rr) * nw[i], sz_sigmoid(zv[i]));      // (rounded before the high part is taken from it)
        if (xh == nullptr) { og[at + 32 * i] = y; continue; }
        const __half h = __float2half_rn(y);
        xh[at + 32 * i] = h;
        xh[(size_t)padded * vh * D + at + 32 * i] = __float2half_rn(y - __half2float(h));
    }
}

// After a step: the sequences move on by the rows of their chunks, and what a kernel over all rows raised in the step's error word becomes
// every sequence's own (it stays there until the session is reset; the step's word is ready for whoever has the room next).  One block.
__global__ void sz_rows_commit_kernel(const SzSeqDev* __restrict__ seqs, int n, u32* __restrict__ err) {
    sz_pdl_wait();
    sz_pdl_trigger();
    const int b = threadIdx.x;
    const u32 e = __ldcg(err);
    if (b < n) {
        int32_t* state = const_cast<int32_t*>(seqs[b].state);
        if (e) atomicOr((u32*)state + 2, e);
        if (seqs[b].keep) {
            state[0] += seqs[b].keep;
            state[1] ^= 1;
        }
    }
    __syncthreads();
    if (b == 0 && e) *err = 0u;
}

#endif
