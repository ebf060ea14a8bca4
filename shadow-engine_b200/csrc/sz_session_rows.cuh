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

// The DeltaNet front end over the rows of a step (sz_delta_prep_kernel's arithmetic).  grid (ceil(ch / 256), rows).  What the scan
// reads - and a replay, when the sequence's rows may be rejected - goes to the session's buffers, of a prompt's chunk to the step's
// (xc_all, beta_all, decay_all), and a chunk's last row leaves the carried conv rows behind it in the other buffer.
__global__ void __launch_bounds__(256)
sz_rows_delta_prep_kernel(const SzSeqDev* __restrict__ seqs, const SzRowDev* __restrict__ rws, int di, const float* __restrict__ xin, const float* __restrict__ cw,
                          const float* __restrict__ b, const float* __restrict__ a, const float* __restrict__ a_log, const float* __restrict__ dt, int kh, int vh, int d,
                          int k, float* __restrict__ xc_all, float* __restrict__ beta_all, float* __restrict__ decay_all) {
    __shared__ double sred[8];
    const int r = blockIdx.y, j = rws[r].j;
    const SzSeqDev& q = seqs[rws[r].seq];
    const int kd = kh * d, ch = 2 * kd + vh * d, i = blockIdx.x * 256 + threadIdx.x;
    float taps[8];
    for (int t = 0; t < k; t++) taps[t] = i < ch ? __ldg(cw + (size_t)i * k + t) : 0.f;
    sz_pdl_wait();
    sz_pdl_trigger();
    const int cur = q.state[1];
    const size_t cl = (size_t)(k - 1) * ch;
    const float* conv = (cur ? q.conv1 : q.conv0) + di * cl;
    float* convw = (cur ? q.conv0 : q.conv1) + di * cl;
    float* xc = q.all ? xc_all + (size_t)r * ch : q.xc + ((size_t)di * SZ_MAX_VERIFY + j) * ch;
    const float* x = xin + (size_t)r * ch;          // (the rows before it in its sequence are the rows before it in the step)
    float v = 0.f;
    if (i < ch) {
        const float own = x[i];
        double acc = (double)taps[k - 1] * (double)own;
        for (int t = 0; t < k - 1; t++) {
            const int tau = j - (k - 1) + t;
            const float prev = tau >= 0 ? x[(long long)(t - (k - 1)) * ch + i] : conv[(size_t)((k - 1) + tau) * ch + i];
            acc += (double)taps[t] * (double)prev;
        }
        v = sz_silu((float)acc);
        if (!q.all) q.xin[((size_t)di * SZ_MAX_VERIFY + j) * ch + i] = own;
        else if (j == q.m - 1)
            for (int t = 0; t < k - 1; t++) {
                const int tau = q.m - (k - 1) + t;
                convw[(size_t)t * ch + i] = tau >= 0 ? x[(long long)(t - (k - 2)) * ch + i] : conv[(size_t)((k - 1) + tau) * ch + i];
            }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double sq = sz_warp_sum((double)v * (double)v);
    if (lane == 0) sred[warp] = sq;
    __syncthreads();
    if (i < ch) {
        if (i < 2 * kd) {
            const int w0 = (threadIdx.x / d) * (d / 32);
            double ss = 0.0;
            for (int t = 0; t < d / 32; t++) ss += sred[w0 + t];
            const double n = sz_rsqrt64(ss + 1e-6);
            float t = (float)((double)v * n);
            if (i < kd) t = t / sqrtf((float)d);
            v = t;
        }
        xc[i] = v;
    }
    if (blockIdx.x == 0) {
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

// The scans of a layer for the sequences of a step, after sz_rows_delta_prep_kernel.  grid (vh * D / 32, sequences)
template <int D>
__global__ void __cluster_dims__(D / 32, 1, 1) __launch_bounds__(2 * D)
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
    sz_delta_scan_body<D>(q, norm_w, kh, vh, eps, (const SzTree*)nullptr, (float*)nullptr, (int)blockIdx.x / (D / 32), (int)blockIdx.x % (D / 32), 0);
}

// After a step: the sequences whose rows were all kept move on.  One block.
__global__ void sz_rows_commit_kernel(const SzSeqDev* __restrict__ seqs, int n) {
    sz_pdl_wait();
    sz_pdl_trigger();
    const int b = threadIdx.x;
    if (b < n && seqs[b].all) {
        int32_t* state = const_cast<int32_t*>(seqs[b].state);
        state[0] += seqs[b].m;
        state[1] ^= 1;
    }
}

#endif
