// Dense projections of a verify pass: y[j] = W x[j] for the 1..8 rows of the pass, W in any of the stored types.
// The role of the reference's matvec_cols_* family (kernels/matvec.cu:677-756) and multi_cols (crates/shadowzero-cuda/src/session.rs:
// 7346-7398: several projections of one input in a launch).  A warp takes a matrix row, a lane four consecutive weights of every
// 128, the inputs sit in shared memory; f32 accumulate.
#pragma once

#include "sz_formats.cuh"

#define SZ_DENSE_MAX_JOBS 6
#define SZ_EPI_NONE 0
#define SZ_EPI_SILU_DIV 1      // silu(v / div)            (hyper-connection down, forward.rs:803)
#define SZ_EPI_SIGMOID 2       // sigmoid(v)
#define SZ_EPI_SIGMOID2_DIV 3  // 2 * sigmoid(v / div)     (hyper-connection inject, forward.rs:812)

struct SzDenseJob {
    const u8* w;     // matrix, rows contiguous
    float* out;      // out[j * ostride + r]
    int rows;
    int type;
    int ostride;
    int epi;
    float div;
    int row0;        // first global row index of this job (filled by the launcher)
};

struct SzDenseArgs {
    SzDenseJob job[SZ_DENSE_MAX_JOBS];
    int n_jobs;
    int total_rows;
    const float* x;  // [m][xstride]
    int xstride;
    int cols;
    int m;
    u32* err;        // set to 1 when a bounded wait on a copy ran out (null: not reported)
};

#ifdef __CUDACC__

__device__ __forceinline__ size_t sz_dense_row_bytes(int type, int cols) {
    switch (type) {
        case SZ_TYPE_F32: return (size_t)cols * 4;
        case SZ_TYPE_F16: case SZ_TYPE_BF16: return (size_t)cols * 2;
        case SZ_TYPE_Q8_0: return (size_t)(cols / 32) * 34;
        default: return (size_t)(cols / 256) * 110;
    }
}

template <typename T, bool GLOBAL>
__device__ __forceinline__ T sz_ld(const void* p) {
    if (GLOBAL) return __ldg((const T*)p);
    return *(const T*)p;
}

// the lane's four weights at columns e .. e + 3 of `row`, and the scale they share.  GLOBAL: `row` is in global memory (read-only
// path); otherwise any address space (a staged copy in shared memory)
template <bool GLOBAL = true>
__device__ __forceinline__ void sz_dense_w4(int type, const u8* __restrict__ row, int e, const u32* grid, float* w, float& scale) {
    if (type == SZ_TYPE_F32) {
        const float4 v = sz_ld<float4, GLOBAL>(row + (size_t)e * 4);
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w; scale = 1.f;
    } else if (type == SZ_TYPE_BF16) {
        const uint2 v = sz_ld<uint2, GLOBAL>(row + (size_t)e * 2);
        w[0] = __uint_as_float(v.x << 16); w[1] = __uint_as_float(v.x & 0xffff0000u);
        w[2] = __uint_as_float(v.y << 16); w[3] = __uint_as_float(v.y & 0xffff0000u); scale = 1.f;
    } else if (type == SZ_TYPE_F16) {
        const uint2 v = sz_ld<uint2, GLOBAL>(row + (size_t)e * 2);
        w[0] = sz_f16_to_f32((u16)(v.x & 0xffff)); w[1] = sz_f16_to_f32((u16)(v.x >> 16));
        w[2] = sz_f16_to_f32((u16)(v.y & 0xffff)); w[3] = sz_f16_to_f32((u16)(v.y >> 16)); scale = 1.f;
    } else if (type == SZ_TYPE_Q8_0) {
        const u8* blk = row + (e >> 5) * 34;
        const int i = e & 31;
        scale = sz_f16_to_f32(sz_ld<u16, GLOBAL>(blk));
        const u32 q01 = sz_ld<u16, GLOBAL>(blk + 2 + i), q23 = sz_ld<u16, GLOBAL>(blk + 4 + i);
        w[0] = (float)(int8_t)(q01 & 0xff); w[1] = (float)(int8_t)(q01 >> 8);
        w[2] = (float)(int8_t)(q23 & 0xff); w[3] = (float)(int8_t)(q23 >> 8);
    } else {  // IQ3_S
        const u8* blk = row + (e >> 8) * 110;
        const int jj = (e & 255) >> 2;
        const int idx = blk[2 + jj] | (((blk[66 + (jj >> 3)] >> (jj & 7)) & 1) << 8);
        const int g = jj >> 3;
        const int s = (blk[106 + (g >> 1)] >> (4 * (g & 1))) & 15;
        scale = sz_f16_to_f32(sz_ld16(blk)) * (float)(1 + 2 * s);
        const u32 mags = grid[idx];
        const u32 sg = blk[74 + (jj >> 1)] >> (4 * (jj & 1));
        w[0] = (float)(mags & 0xff); w[1] = (float)((mags >> 8) & 0xff); w[2] = (float)((mags >> 16) & 0xff); w[3] = (float)(mags >> 24);
        w[0] = (sg & 1) ? -w[0] : w[0]; w[1] = (sg & 2) ? -w[1] : w[1]; w[2] = (sg & 4) ? -w[2] : w[2]; w[3] = (sg & 8) ? -w[3] : w[3];
    }
}

__device__ __forceinline__ float sz_epilogue(int epi, float v, float div) {
    switch (epi) {
        case SZ_EPI_SILU_DIV: return sz_silu(v / div);
        case SZ_EPI_SIGMOID: return sz_sigmoid(v);
        case SZ_EPI_SIGMOID2_DIV: return 2.0f * sz_sigmoid(v / div);
        default: return v;
    }
}

// grid: any (blocks stride over the rows of all jobs, 8 rows a block at a time); block 256; dynamic shared memory 2048 + mt * cols * 4
// where mt = rows of x handled per sweep (the launcher picks the largest that fits).
template <int MT>
__global__ void __launch_bounds__(256) sz_dense_kernel(const SzDenseArgs a) {
    extern __shared__ __align__(128) u8 smem[];
    u32* grid = (u32*)smem;
    float* xs = (float*)(smem + 2048);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    sz_pdl_wait();
    sz_pdl_trigger();
    for (int i = threadIdx.x; i < 512; i += 256) grid[i] = c_iq3s_grid[i];
    for (int j0 = 0; j0 < a.m; j0 += MT) {
        const int mt = min(MT, a.m - j0);
        __syncthreads();
        for (int j = 0; j < mt; j++) {
            const float4* src = (const float4*)(a.x + (size_t)(j0 + j) * a.xstride);
            float4* dst = (float4*)(xs + (size_t)j * a.cols);
            for (int i = threadIdx.x; i < a.cols / 4; i += 256) dst[i] = __ldcg(src + i);
        }
        __syncthreads();
        for (int r = blockIdx.x * 8 + warp; r < a.total_rows; r += gridDim.x * 8) {
            int ji = 0;
#pragma unroll
            for (int q = 1; q < SZ_DENSE_MAX_JOBS; q++)
                if (q < a.n_jobs && r >= a.job[q].row0) ji = q;
            const SzDenseJob& jb = a.job[ji];
            const int rr = r - jb.row0;
            const u8* row = jb.w + (size_t)rr * sz_dense_row_bytes(jb.type, a.cols);
            float acc[MT];
#pragma unroll
            for (int j = 0; j < MT; j++) acc[j] = 0.f;
            for (int e = 4 * lane; e < a.cols; e += 128) {
                float w[4], scale;
                sz_dense_w4<true>(jb.type, row, e, grid, w, scale);
#pragma unroll
                for (int j = 0; j < MT; j++) {
                    if (j < mt) {
                        const float4 v = *(const float4*)(xs + (size_t)j * a.cols + e);
                        float p = w[0] * v.x;
                        p = fmaf(w[1], v.y, p);
                        p = fmaf(w[2], v.z, p);
                        p = fmaf(w[3], v.w, p);
                        acc[j] = fmaf(scale, p, acc[j]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < MT; j++) {
                if (j < mt) {
                    const float v = sz_warp_sum(acc[j]);
                    if (lane == 0) jb.out[(size_t)(j0 + j) * jb.ostride + rr] = sz_epilogue(jb.epi, v, jb.div);
                }
            }
        }
    }
}

// ---- streaming form -------------------------------------------------------------------------------------------------------------------
// Units of R whole rows (about 32 KB) are copied into a ring of shared-memory stages by the TMA engine (cp.async.bulk) while the
// warps work on the previous ones.  Warp w takes RW rows of the unit (row group w % NG) and one of KP column ranges (w / NG), so an
// x value read from shared memory feeds RW rows: the kernel is bound by the weight stream, not by shared-memory reads of x.
// Column-range partial sums meet in shared memory.  Needs row bytes that are a multiple of 16.
struct SzDense2Cfg {
    int R, RW, KP, NS;       // rows a unit, rows a warp, column parts, stages
    int unit_bytes;          // R * row bytes (the same for every job: one input width, and the jobs of a launch share a type size class)
    int units[SZ_DENSE_MAX_JOBS + 1];  // first unit of each job; units[n_jobs] = total
};

template <int MT, int RW>
__global__ void __launch_bounds__(256) sz_dense2_kernel(const SzDenseArgs a, const SzDense2Cfg c) {
    extern __shared__ __align__(128) u8 smem[];
    u64* bars = (u64*)smem;                               // NS barriers (64 bytes reserved)
    u32* grid = (u32*)(smem + 64);                        // IQ3_S codebook
    float* red = (float*)(smem + 64 + 2048);              // [8 warps][RW][MT]
    float* xs = (float*)(smem + 64 + 2048 + 8 * 4 * 8 * 4);
    u8* stages = smem + 64 + 2048 + 1024 + (size_t)MT * a.cols * 4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int NG = c.R / RW;
    const int grp = warp % NG, kp = warp / NG;
    const int part = a.cols / c.KP;
    const int e0 = kp * part, e1 = e0 + part;
    if (threadIdx.x == 0) {
        for (int i = 0; i < c.NS; i++) sz_mbar_init(&bars[i], 1);
        sz_mbar_fence_init();
    }
    for (int i = threadIdx.x; i < 512; i += 256) grid[i] = c_iq3s_grid[i];
    __syncthreads();
    const int total = c.units[a.n_jobs];
    auto locate = [&](int u, int& ji, int& row0, int& nrows) {
        ji = 0;
#pragma unroll
        for (int q = 1; q < SZ_DENSE_MAX_JOBS; q++)
            if (q < a.n_jobs && u >= c.units[q]) ji = q;
        row0 = (u - c.units[ji]) * c.R;
        nrows = min(c.R, a.job[ji].rows - row0);
    };
    // weights do not depend on the previous kernel: start streaming before waiting for it
    const int first = blockIdx.x, step = gridDim.x;
    const int count = first < total ? (total - first + step - 1) / step : 0;
    auto issue = [&](int local, int gi) {  // local: which of this block's units; gi: running copy index over all sweeps
        int ji, row0, nrows;
        locate(first + local * step, ji, row0, nrows);
        const size_t rb = sz_dense_row_bytes(a.job[ji].type, a.cols);
        u64* bar = &bars[gi % c.NS];
        const u32 bytes = (u32)(nrows * rb);
        sz_mbar_expect_tx(bar, bytes);
        sz_bulk_g2s(stages + (size_t)(gi % c.NS) * c.unit_bytes, a.job[ji].w + (size_t)row0 * rb, bytes, bar);
    };
    int failed = 0;
    for (int j0 = 0; j0 < a.m; j0 += MT) {
        const int mt = min(MT, a.m - j0);
        const int base = (j0 / MT) * count;  // units issued so far (each sweep streams every unit again)
        if (threadIdx.x == 0)
            for (int i = 0; i < c.NS - 1 && i < count; i++) issue(i, base + i);
        if (j0 == 0) { sz_pdl_wait(); sz_pdl_trigger(); }
        __syncthreads();
        for (int j = 0; j < mt; j++) {
            const float4* src = (const float4*)(a.x + (size_t)(j0 + j) * a.xstride);
            float4* dst = (float4*)(xs + (size_t)j * a.cols);
            for (int i = threadIdx.x; i < a.cols / 4; i += 256) dst[i] = __ldcg(src + i);
        }
        __syncthreads();
        for (int i = 0; i < count; i++) {
            const int gi = base + i;
            if (threadIdx.x == 0 && i + c.NS - 1 < count) issue(i + c.NS - 1, gi + c.NS - 1);
            int ji, row0, nrows;
            locate(first + i * step, ji, row0, nrows);
            const SzDenseJob& jb = a.job[ji];
            const size_t rb = sz_dense_row_bytes(jb.type, a.cols);
            if (!sz_mbar_wait(&bars[gi % c.NS], (gi / c.NS) & 1)) failed = 1;
            const u8* st = stages + (size_t)(gi % c.NS) * c.unit_bytes;
            float acc[RW][MT];
#pragma unroll
            for (int r = 0; r < RW; r++)
#pragma unroll
                for (int j = 0; j < MT; j++) acc[r][j] = 0.f;
            if (!failed && kp < c.KP && grp * RW < nrows) {
                for (int e = e0 + 4 * lane; e < e1; e += 128) {
                    float4 xv[MT];
#pragma unroll
                    for (int j = 0; j < MT; j++) xv[j] = j < mt ? *(const float4*)(xs + (size_t)j * a.cols + e) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int r = 0; r < RW; r++) {
                        const int rr = grp * RW + r;
                        if (rr < nrows) {
                            float w[4], scale;
                            sz_dense_w4<false>(jb.type, st + (size_t)rr * rb, e, grid, w, scale);
#pragma unroll
                            for (int j = 0; j < MT; j++) {
                                float p = w[0] * xv[j].x;
                                p = fmaf(w[1], xv[j].y, p);
                                p = fmaf(w[2], xv[j].z, p);
                                p = fmaf(w[3], xv[j].w, p);
                                acc[r][j] = fmaf(scale, p, acc[r][j]);
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < RW; r++)
#pragma unroll
                for (int j = 0; j < MT; j++) {
                    const float v = sz_warp_sum(acc[r][j]);
                    if (lane == 0) red[(warp * RW + r) * MT + j] = v;
                }
            if (__syncthreads_or(failed)) { failed = 1; break; }
            // the column parts of a row meet here: thread t finishes (row rr, input row j)
            for (int t = threadIdx.x; t < nrows * mt; t += 256) {
                const int rr = t / mt, j = t % mt;
                const int g2 = rr / RW, r2 = rr % RW;
                float v = 0.f;
                for (int q = 0; q < c.KP; q++) v += red[((q * NG + g2) * RW + r2) * MT + j];
                jb.out[(size_t)(j0 + j) * jb.ostride + row0 + rr] = sz_epilogue(jb.epi, v, jb.div);
            }
            __syncthreads();
        }
        if (failed) break;
    }
    if (failed && threadIdx.x == 0 && a.err) atomicExch(a.err, 1u);
}

// ---- Q8_0 on the tensor pipe ----------------------------------------------------------------------------------------------------------
// The same streaming skeleton for Q8_0 matrices, with the multiply-adds on mma.sync: a warp owns one eighth of the columns of a
// 16-row unit; per 32-column block it turns each row's 32 int8 codes into f16 exactly (0x6400 | (q ^ 0x80) is the f16 1024 + q + 128),
// multiplies them with the rows of the pass (the B operand, split into f16 high and low parts so the activations keep f32 accuracy)
// into a fresh accumulator and adds that, times the block's scale, to the running sums.  Per weight this is ~2.6 issue slots
// whatever the number of rows, against ~8 for the scalar form at 4 rows, which is what lets the kernel follow the HBM stream.
// Lane (g, q) takes the block's bytes 8 q .. 8 q + 7 of rows g and g + 8; the k slots of the two MMAs are permuted accordingly and
// the B fragments use the same permutation (x columns 8 q .. 8 q + 7 of row-of-the-pass g).
__device__ __forceinline__ void sz_mma16816_z(float* c, const u32* a, u32 b0, u32 b1) {  // c += a * b
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void sz_mma16816_zn(float* c, const u32* a, u32 b0, u32 b1) {  // the same, free to move among its neighbours
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <bool V> struct SzBool { static constexpr bool value = V; };

// two int8 codes (the low 16 bits of p) as an f16 pair
__device__ __forceinline__ u32 sz_q8_pair(u32 p) {
    const u32 t = __byte_perm(p ^ 0x8080u, 0x64646464u, 0x4140);  // 0x64 b1' 0x64 b0' with b' = b ^ 0x80
    const __half2 h = __hsub2(*(const __half2*)&t, __halves2half2(__ushort_as_half((u16)0x6480), __ushort_as_half((u16)0x6480)));  // - 1152
    return *(const u32*)&h;
}

// the four codes of a word as two f16 pairs
__device__ __forceinline__ void sz_q8_quad(u32 w, u32& lo, u32& hi) {
    const u32 x = w ^ 0x80808080u;
    const __half2 k = __halves2half2(__ushort_as_half((u16)0x6480), __ushort_as_half((u16)0x6480));
    const u32 a = __byte_perm(x, 0x64646464u, 0x4140), b = __byte_perm(x, 0x64646464u, 0x4342);
    const __half2 ha = __hsub2(*(const __half2*)&a, k), hb = __hsub2(*(const __half2*)&b, k);
    lo = *(const u32*)&ha; hi = *(const u32*)&hb;
}

// Codes 8 q .. 8 q + 7 of the Q8_0 block at p (of a row that starts at a multiple of 4 bytes; `odd`: the block's number) as the two A
// fragments' registers of one row, and its scale.  In odd blocks the codes start at a multiple of 4, in even ones 2 behind one.
template <bool ODD>
__device__ __forceinline__ void sz_q8_row(const u8* p, int q, u32& a1l, u32& a1h, u32& a2l, u32& a2h, float& d) {
    u32 c01, c23;
    if (ODD) {
        c01 = *(const u32*)(p + 2 + 8 * q); c23 = *(const u32*)(p + 6 + 8 * q);
    } else {
        const u32 w0 = *(const u32*)(p + 8 * q), w1 = *(const u32*)(p + 8 * q + 4), w2 = *(const u32*)(p + 8 * q + 8);   // (an odd block follows: no byte past the row)
        c01 = __funnelshift_r(w0, w1, 16); c23 = __funnelshift_r(w1, w2, 16);
    }
    d = sz_f16_to_f32(*(const u16*)p);
    sz_q8_quad(c01, a1l, a1h);
    sz_q8_quad(c23, a2l, a2h);
}

struct SzDenseQ8Cfg {
    int NS, unit_bytes;
    int rbp;   // bytes between the rows of a staged unit: the row bytes padded so that rows 0..7 start in different banks
    int xsp;   // halves between the staged rows of the pass, padded likewise
    int units[SZ_DENSE_MAX_JOBS + 1];
};

// Shared-memory layout matters more than anything else here: a matrix row is cols / 32 * 34 bytes, a multiple of 128 for the usual
// widths, so eight lanes reading the same block of eight different rows would hit one bank eight times over.  Every row of a unit
// is therefore its own bulk copy to a padded stride (rbp), and the rows of the pass are padded the same way (xsp).
// grid: any; block 256; dynamic shared memory: 64 (barriers) + 4096 (reduction) + 2 * m * xsp * 2 (x as f16 hi | lo) + NS * unit_bytes
static __global__ void __launch_bounds__(256, 2) sz_dense_q8_kernel(const SzDenseArgs a, const SzDenseQ8Cfg c) {
    extern __shared__ __align__(128) u8 smem[];
    u64* bars = (u64*)smem;
    float* red = (float*)(smem + 64);                       // [8 warps][16 rows][8 rows of the pass]
    __half* xhi = (__half*)(smem + 64 + 4096);              // [m][xsp]
    __half* xlo = xhi + (size_t)a.m * c.xsp;
    u8* stages = smem + 64 + 4096 + (size_t)a.m * c.xsp * 4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, q = lane & 3;
    const size_t rb = (size_t)(a.cols / 32) * 34;
    if (threadIdx.x == 0) {
        for (int i = 0; i < c.NS; i++) sz_mbar_init(&bars[i], 1);
        sz_mbar_fence_init();
    }
    __syncthreads();
    const int total = c.units[a.n_jobs];
    auto locate = [&](int u, int& ji, int& row0, int& nrows) {
        ji = 0;
#pragma unroll
        for (int t = 1; t < SZ_DENSE_MAX_JOBS; t++)
            if (t < a.n_jobs && u >= c.units[t]) ji = t;
        row0 = (u - c.units[ji]) * 16;
        nrows = min(16, a.job[ji].rows - row0);
    };
    const int first = blockIdx.x, step = gridDim.x;
    const int count = first < total ? (total - first + step - 1) / step : 0;
    auto issue = [&](int i) {      // warp 0, a lane a row
        int ji, row0, nrows;
        locate(first + i * step, ji, row0, nrows);
        u64* bar = &bars[i % c.NS];
        if (lane == 0) sz_mbar_expect_tx(bar, (u32)(nrows * rb));
        __syncwarp();
        u8* dst = stages + (size_t)(i % c.NS) * c.unit_bytes;
        const u8* src = a.job[ji].w + (size_t)row0 * rb;
        if (lane < nrows) sz_bulk_g2s(dst + (size_t)lane * c.rbp, src + (size_t)lane * rb, (u32)rb, bar);
    };
    if (warp == 0)
        for (int i = 0; i < c.NS - 1 && i < count; i++) issue(i);
    sz_pdl_wait();
    sz_pdl_trigger();
    // the rows' pieces, of up to four rows and two places in flight (a piece after the other paid the way to L2 eight times at 4 rows)
    const int pieces = a.cols / 4;
    for (int c4 = threadIdx.x; c4 < pieces; c4 += 512)
        for (int j0 = 0; j0 < a.m; j0 += 4) {
            float4 v[4][2];
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int e = 0; e < 2; e++)
                    if (j0 + j < a.m && c4 + 256 * e < pieces) v[j][e] = __ldcg((const float4*)(a.x + (size_t)(j0 + j) * a.xstride) + c4 + 256 * e);
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int e = 0; e < 2; e++)
                    if (j0 + j < a.m && c4 + 256 * e < pieces) {
                        const float4 f = v[j][e];
                        const __half2 h0 = __floats2half2_rn(f.x, f.y), h1 = __floats2half2_rn(f.z, f.w);
                        const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
                        const __half2 l0 = __floats2half2_rn(f.x - f0.x, f.y - f0.y), l1 = __floats2half2_rn(f.z - f1.x, f.w - f1.y);
                        const size_t at = (size_t)(j0 + j) * c.xsp + 4 * (c4 + 256 * e);
                        *(uint2*)(xhi + at) = make_uint2(*(const u32*)&h0, *(const u32*)&h1);
                        *(uint2*)(xlo + at) = make_uint2(*(const u32*)&l0, *(const u32*)&l1);
                    }
        }
    __syncthreads();
    const int part = a.cols / 8;          // columns of this warp: [warp * part, (warp + 1) * part), whole 32-column blocks
    const int nblk = part / 32;
    int failed = 0;
    for (int i = 0; i < count; i++) {
        if (warp == 0 && i + c.NS - 1 < count) issue(i + c.NS - 1);
        int ji, row0, nrows;
        locate(first + i * step, ji, row0, nrows);
        const SzDenseJob& jb = a.job[ji];
        if (!sz_mbar_wait(&bars[i % c.NS], (i / c.NS) & 1)) failed = 1;
        const u8* st = stages + (size_t)(i % c.NS) * c.unit_bytes;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};  // rows g, g + 8 x rows of the pass 2 q, 2 q + 1
        if (!failed) {
            const u8* r0 = st + (size_t)(g < nrows ? g : 0) * c.rbp;
            const u8* r1 = st + (size_t)(g + 8 < nrows ? g + 8 : 0) * c.rbp;
            auto block = [&](int blk, auto odd) {
                const int col = blk * 32 + 8 * q;
                uint4 bh = make_uint4(0, 0, 0, 0), bl = make_uint4(0, 0, 0, 0);
                if (g < a.m) {
                    bh = *(const uint4*)(xhi + (size_t)g * c.xsp + col);
                    bl = *(const uint4*)(xlo + (size_t)g * c.xsp + col);
                }
                u32 a1[4], a2[4];
                float d0, d1;
                sz_q8_row<decltype(odd)::value>(r0 + (size_t)blk * 34, q, a1[0], a1[2], a2[0], a2[2], d0);
                sz_q8_row<decltype(odd)::value>(r1 + (size_t)blk * 34, q, a1[1], a1[3], a2[1], a2[3], d1);
                float t[4] = {0.f, 0.f, 0.f, 0.f};
                sz_mma16816_zn(t, a1, bh.x, bh.y);
                sz_mma16816_zn(t, a2, bh.z, bh.w);
                sz_mma16816_zn(t, a1, bl.x, bl.y);
                sz_mma16816_zn(t, a2, bl.z, bl.w);
                acc[0] = fmaf(d0, t[0], acc[0]); acc[1] = fmaf(d0, t[1], acc[1]);
                acc[2] = fmaf(d1, t[2], acc[2]); acc[3] = fmaf(d1, t[3], acc[3]);
            };
            // (the MMAs of a block are a chain of four: two blocks' run side by side; four's gain the tiny model's passes nothing but code)
            if (!(nblk & 1)) {
#pragma unroll 1
                for (int blk = warp * nblk; blk < warp * nblk + nblk; blk += 2) { block(blk, SzBool<false>()); block(blk + 1, SzBool<true>()); }
            } else {
                for (int blk = warp * nblk; blk < warp * nblk + nblk; blk++)
                    if (blk & 1) block(blk, SzBool<true>()); else block(blk, SzBool<false>());
            }
        }
        // the eight column parts of a row meet in shared memory
        red[(warp * 16 + g) * 8 + 2 * q] = acc[0];
        red[(warp * 16 + g) * 8 + 2 * q + 1] = acc[1];
        red[(warp * 16 + g + 8) * 8 + 2 * q] = acc[2];
        red[(warp * 16 + g + 8) * 8 + 2 * q + 1] = acc[3];
        if (__syncthreads_or(failed)) { failed = 1; break; }
        for (int t = threadIdx.x; t < 16 * 8; t += 256) {
            const int rr = t >> 3, j = t & 7;
            if (rr < nrows && j < a.m) {
                float v = 0.f;
#pragma unroll
                for (int w = 0; w < 8; w++) v += red[(w * 16 + rr) * 8 + j];
                jb.out[(size_t)j * jb.ostride + row0 + rr] = sz_epilogue(jb.epi, v, jb.div);
            }
        }
        __syncthreads();
    }
    if (failed && threadIdx.x == 0 && a.err) atomicExch(a.err, 1u);
}

// ---- many-row form of the Q8_0 tensor-pipe kernel ------------------------------------------------------------------------------------
// The projections of a batch or a prompt's chunk: y[j] = W x[j] for tens or hundreds of rows, bit for bit what sz_dense_q8_kernel gives for
// 8 of them.  There a warp owns an eighth of the columns and runs, block of 32 columns after block, four MMAs into a fresh accumulator and
// one multiply-add with the block's scale into its part's running sum; the eight parts' sums are then added in order.  Here a warp runs
// through all columns - the same chains, the parts one after the other, a part's sum added to the total when its last block is done - for
// a unit of 16 matrix rows and 32 rows of the step, so that nothing but the result leaves it.  A thread block's 8 warps stage the slices
// of their units and of the rows (f16 high and low parts, made once by sz_dense_rows_pack_kernel) 128 columns at a time through a ring of
// asynchronous copies; a block of 32 columns decoded into A fragments serves 4 row groups.  Two thread blocks a multiprocessor: with two
// units a warp, which loads the rows' fragments half as often but needs 200 registers, one fitted, and its 8 warps kept the tensor pipe 40 %
// busy (504 rows of 12,352 outputs: 251 -> 199 us; 80 rows 50.8 -> 45.0).
// (The form before it gave a thread block one part and four or eight row groups: a fragment of the rows was loaded from shared memory for
// every unit, and the parts' sums - 98 MB at 256 rows of 12,352 outputs - went through a scratch and a second kernel.  the four MMAs a
// block and group alone are 44 us.)
// Where thread blocks of 8 units and 32 rows would leave multiprocessors idle (80 rows of 2,048 outputs: 48 of them, 49 us, 3,000 cycles for
// 128 columns in which the tensor pipe works 900), the blocks are of 4 units and 16 rows (35 us) or 8.  What such a launch takes is then the chain of its
// stages, so two or four thread blocks share the columns as long as the multiprocessors have room for them: sz_dense_rows_form has the lines and what
// the forms measured.
// A slice of a matrix row starts at a multiple of 8 bytes, not of 16: the copy starts at the 16-byte boundary below it.
struct SzDenseRowsCfg {
    int units[SZ_DENSE_MAX_JOBS + 1];   // 16-row units before each job
    int rows;                           // rows in all (a multiple of 8)
    const __half* xh;                   // high parts [rows][cols], then the low parts
};
#define SZ_DR_COLS 128      // columns a stage
#define SZ_DR_RS 144        // bytes between the staged slices (136 and where they start)
#define SZ_DR_XS 160        // halves between the staged rows (16 (mod 32) words: the eight rows a quarter of a warp reads at once)
// NW: warps a thread block, a unit of 16 matrix rows each; NG: groups of 8 rows of the step; KS: thread blocks of a cluster that share the columns,
// whole parts each.  A part's sums stay where they are made, in shared memory, and once all are there each block adds the parts of its groups in order.
template <int NW, int NG, int KS = 1>
struct SzDenseRows {
    static constexpr int WROWS = NW * 16;                                        // matrix rows a thread block
    static constexpr int STAGE = WROWS * SZ_DR_RS + 2 * 8 * NG * SZ_DR_XS * 2;
    static constexpr int STAGES = NW == 8 ? 2 : (KS > 1 ? 3 : 4);
    static constexpr int PARTS = KS > 1 ? 8 / KS * NG * 4 * 32 * NW * 4 : 0;     // [part][group, value][thread]
    static constexpr int OCC = KS > 1 ? 3 : 2;
    static constexpr int SMEM = STAGES * STAGE + WROWS * 8 + PARTS;
};

// grid (ceil(cols / 1024), rows), block 256: the rows' f16 high and low parts
static __global__ void __launch_bounds__(256) sz_dense_rows_pack_kernel(const float* __restrict__ x, int xstride, int cols, int rows, __half* __restrict__ xh) {
    sz_pdl_wait();
    sz_pdl_trigger();
    const int c4 = blockIdx.x * 256 + threadIdx.x, j = blockIdx.y;
    if (c4 * 4 >= cols) return;
    const float4 v = __ldcg((const float4*)(x + (size_t)j * xstride) + c4);
    const __half2 h0 = __floats2half2_rn(v.x, v.y), h1 = __floats2half2_rn(v.z, v.w);
    const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
    const __half2 l0 = __floats2half2_rn(v.x - f0.x, v.y - f0.y), l1 = __floats2half2_rn(v.z - f1.x, v.w - f1.y);
    *(uint2*)(xh + (size_t)j * cols + 4 * c4) = make_uint2(*(const u32*)&h0, *(const u32*)&h1);
    *(uint2*)(xh + (size_t)(rows + j) * cols + 4 * c4) = make_uint2(*(const u32*)&l0, *(const u32*)&l1);
}

// grid (ceil(units / NW) * KS, ceil(rows / (8 NG))), block 32 NW, cluster KS; KS > 1: cols a multiple of 128 KS
template <int NW, int NG, int KS>
static __global__ void __cluster_dims__(KS, 1, 1) __launch_bounds__(32 * NW, (SzDenseRows<NW, NG, KS>::OCC)) sz_dense_rows_q8_kernel(const SzDenseArgs a, const SzDenseRowsCfg c) {
    using X = SzDenseRows<NW, NG, KS>;
    constexpr int NTH = 32 * NW;
    constexpr int S = X::STAGES;
    extern __shared__ __align__(128) u8 smem[];
    const u8** wrow = (const u8**)(smem + S * X::STAGE);       // where the thread block's matrix rows start
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, q = lane & 3;
    const int total = c.units[a.n_jobs], u0 = (int)blockIdx.x / KS * NW, j0 = blockIdx.y * 8 * NG, kr = (int)blockIdx.x % KS;
    const int ng = (c.rows - j0) / 8 < NG ? (c.rows - j0) / 8 : NG;
    const size_t rb = (size_t)(a.cols / 32) * 34;
    const int nchunk = a.cols / SZ_DR_COLS / KS, k0 = kr * nchunk, nblk = a.cols / 256;      // the block's stages, the first of them; blocks of 32 columns a part
    float* const parts = (float*)(smem + S * X::STAGE + X::WROWS * 8);
    auto locate = [&](int u, int& ji, int& row0, int& nrows) {
        ji = 0;
#pragma unroll
        for (int t = 1; t < SZ_DENSE_MAX_JOBS; t++)
            if (t < a.n_jobs && u >= c.units[t]) ji = t;
        row0 = (u - c.units[ji]) * 16;
        nrows = min(16, a.job[ji].rows - row0);
    };
    for (int r = threadIdx.x; r < X::WROWS; r += NTH) {
        const int u = min(u0 + (r >> 4), total - 1);          // (units past the last: its rows again; nothing of them is kept)
        int ji, row0, nrows;
        locate(u, ji, row0, nrows);
        wrow[r] = a.job[ji].w + (size_t)(row0 + ((r & 15) < nrows ? (r & 15) : 0)) * rb;
    }
    __syncthreads();
    auto stage_w = [&](int ci) {
        u8* st = smem + (size_t)(ci % S) * X::STAGE;
        const int at = (k0 + ci) * 136 & ~15;
#pragma unroll
        for (int i = threadIdx.x; i < X::WROWS * 9; i += NTH) {
            const int r = i / 9, ch = i - r * 9;
            sz_cp_async16(st + r * SZ_DR_RS + ch * 16, wrow[r] + at + ch * 16);
        }
    };
    auto stage_x = [&](int ci) {
        u8* st = smem + (size_t)(ci % S) * X::STAGE + X::WROWS * SZ_DR_RS;
#pragma unroll
        for (int i = threadIdx.x; i < 2 * 8 * NG * 16; i += NTH) {
            const int part = i / (8 * NG * 16), j = (i >> 4) % (8 * NG), ch = i & 15;
            if (j < ng * 8) sz_cp_async16(st + (size_t)(part * 8 * NG + j) * SZ_DR_XS * 2 + ch * 16, c.xh + (size_t)(part * c.rows + j0 + j) * a.cols + (k0 + ci) * SZ_DR_COLS + ch * 8);
        }
    };
    for (int i = 0; i < S - 1 && i < nchunk; i++) stage_w(i);      // (the matrices are constants: on their way before the wait)
    sz_pdl_wait();
    sz_pdl_trigger();
    for (int i = 0; i < S - 1; i++) { if (i < nchunk) stage_x(i); sz_cp_async_commit(); }
    float tot[NG][4], acc[NG][4];
#pragma unroll
    for (int gi = 0; gi < NG; gi++)
#pragma unroll
        for (int e = 0; e < 4; e++) { tot[gi][e] = 0.f; acc[gi][e] = 0.f; }
    int left = nblk, part = 0;             // blocks left of the part at hand, and its number here
    for (int ci = 0; ci < nchunk; ci++) {
        sz_cp_async_wait<S - 2>();
        __syncthreads();                   // stage ci has landed, and everybody is done with the one that is filled next
        if (ci + S - 1 < nchunk) { stage_w(ci + S - 1); stage_x(ci + S - 1); }
        sz_cp_async_commit();
        const u8* st = smem + (size_t)(ci % S) * X::STAGE;
        const u8* wr = st + (size_t)(warp * 16 + g) * SZ_DR_RS + (((k0 + ci) & 1) ? 8 : 0) + 8 * q;
        const __half* xr = (const __half*)(st + X::WROWS * SZ_DR_RS) + (size_t)g * SZ_DR_XS + 8 * q;
#pragma unroll
        for (int b = 0; b < 4; b++) {
            // a block's 34 bytes: scale, 32 codes; the lane's 8 codes start at a multiple of 4 in odd blocks, 2 behind one in even ones
            u32 a1[4], a2[4];
            float d[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const u8* p = wr + (size_t)(8 * h) * SZ_DR_RS + b * 34;
                u32 c01, c23;
                if (b & 1) {
                    c01 = *(const u32*)(p + 2); c23 = *(const u32*)(p + 6);
                } else {
                    const u32 w0 = *(const u32*)p, w1 = *(const u32*)(p + 4), w2 = *(const u32*)(p + 8);
                    c01 = __funnelshift_r(w0, w1, 16); c23 = __funnelshift_r(w1, w2, 16);
                }
                d[h] = sz_f16_to_f32(*(const u16*)(p - 8 * q));
                sz_q8_quad(c01, a1[h], a1[2 + h]);
                sz_q8_quad(c23, a2[h], a2[2 + h]);
            }
#pragma unroll
            // (all groups, whether the step has them or not: a branch around one would keep its MMAs - a chain of four - from running
            // between the others')
            for (int gi = 0; gi < NG; gi++) {
                const uint4 bh = *(const uint4*)(xr + (size_t)gi * 8 * SZ_DR_XS + b * 32);
                const uint4 bl = *(const uint4*)(xr + (size_t)(8 * NG + gi * 8) * SZ_DR_XS + b * 32);
                float t[4] = {0.f, 0.f, 0.f, 0.f};
                sz_mma16816_zn(t, a1, bh.x, bh.y);
                sz_mma16816_zn(t, a2, bh.z, bh.w);
                sz_mma16816_zn(t, a1, bl.x, bl.y);
                sz_mma16816_zn(t, a2, bl.z, bl.w);
                acc[gi][0] = fmaf(d[0], t[0], acc[gi][0]); acc[gi][1] = fmaf(d[0], t[1], acc[gi][1]);
                acc[gi][2] = fmaf(d[1], t[2], acc[gi][2]); acc[gi][3] = fmaf(d[1], t[3], acc[gi][3]);
            }
            if (--left == 0) {             // the part's sum is complete
                left = nblk;
#pragma unroll
                for (int gi = 0; gi < NG; gi++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        if constexpr (KS > 1) parts[((part * NG + gi) * 4 + e) * NTH + threadIdx.x] = acc[gi][e];
                        else tot[gi][e] += acc[gi][e];
                        acc[gi][e] = 0.f;
                    }
                part++;
            }
        }
    }
    if constexpr (KS > 1) {                // all parts of the block's groups, in order
        sz_cluster_sync();
#pragma unroll
        for (int gi = 0; gi < NG; gi++)
            if (gi % KS == kr)
#pragma unroll
                for (int k = 0; k < 8; k++)
#pragma unroll
                    for (int e = 0; e < 4; e++) tot[gi][e] += sz_cluster_ld(&parts[((k % (8 / KS) * NG + gi) * 4 + e) * NTH + threadIdx.x], k / (8 / KS));
        sz_cluster_sync();                 // (no block leaves while another reads its parts)
    }
    const int u = u0 + warp;
    if (u < total) {
        int ji, row0, nrows;
        locate(u, ji, row0, nrows);
        const SzDenseJob& jb = a.job[ji];
#pragma unroll
        for (int gi = 0; gi < NG; gi++) {
            if (gi < ng && (KS == 1 || gi % KS == kr)) {
                float* o = jb.out + (size_t)(j0 + gi * 8 + 2 * q) * jb.ostride + row0 + g;
                if (g < nrows) { o[0] = sz_epilogue(jb.epi, tot[gi][0], jb.div); o[jb.ostride] = sz_epilogue(jb.epi, tot[gi][1], jb.div); }
                if (g + 8 < nrows) { o[8] = sz_epilogue(jb.epi, tot[gi][2], jb.div); o[jb.ostride + 8] = sz_epilogue(jb.epi, tot[gi][3], jb.div); }
            }
        }
    }
}

#endif  // __CUDACC__

// host: launches the jobs of `a` (row0 / total_rows are filled here)
int sz_dense_launch(SzDenseArgs& a, cudaStream_t st, const char* name);
// a.m rows, a multiple of 8 (any number of them), through the many-row form of the Q8_0 tensor-pipe kernel when sz_dense_launch would
// take that kernel for 8 rows of these jobs: *taken = 1 and the rows are computed (bit for bit as 8 at a time); otherwise *taken = 0
// and nothing is launched.  xh: a.m * a.cols * 2 halves of scratch; packed: they hold the rows already.
bool sz_dense_rows_takes(const SzDenseArgs& a);
int sz_dense_rows_launch(SzDenseArgs& a, void* xh, bool packed, cudaStream_t st, const char* name, int* taken);
int sz_dense_check(const sz_tensor* t, const char* what, int64_t rows, int64_t cols);
