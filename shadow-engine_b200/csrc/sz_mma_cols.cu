// Many-row dense projections on the 5th-generation tensor cores (tcgen05 + TMEM): Y[token][row] = sum_k W[row][k] * X[token][k].
//
// This is the prompt / batched form of a dense projection, the one place of the engine where the work is a contraction and not a
// stream: with 64..256 token rows a Q8_0 weight is used a few hundred times once it is decoded.  It replaces the reference's
// tensor-core family for a long prompt's projections, kernels/matvec.cu:758-1260 (`mma_core`, `mma_cols_<type>`, `mma_cols64_<type>`:
// mma.sync m16n8k16, 64 weight rows x 32 or 64 tokens a block), launched by crates/shadowzero-cuda/src/session.rs:7276, and keeps
// its arithmetic: a weight is decoded as the reference decodes it (the float d * q) and rounded to f16, the input is rounded to
// f16, products accumulate in f32; the order of the sum is the tensor core's.  The reference calls this mode inexact and uses it
// for prompts only; so does this build (the verify step's projections stay on the bit-stable kernels).
//
// Shape of the kernel.  A block owns MT x 128 weight rows (the M side of the instruction), one tile of up to 256 tokens (the N side) and,
// with a cluster of `ks` blocks, a part of K; the accumulators D[128 rows][NT tokens] live in tensor memory (MT x 256 columns of 128
// lanes), so no register holds a partial sum until the end.  K advances in steps of 32 columns, one Q8_0 block a row, through a ring of
// four or eight stages:
//   warp 18     raw Q8_0 bytes of the block's rows, 256 columns at a time (272 bytes a row: a multiple of 16, which the 34 bytes of a
//               step are not) as MT tiled TMA copies (cp.async.bulk.tensor.2d over the matrix seen as [rows][row bytes / 2] 16-bit
//               words, box 136 x 128; 128 separate 272-byte bulk copies a piece kept the copy engine, not the tensor core, as the bound).
//   warp 0      the token tile of a step, already in f16 and in the instruction's own shared-memory order (written once by
//               sz_x16_pack_kernel), one bulk copy.
//   warps 1..16 decode, in groups of MT x 128 threads: a thread takes its group's blocks of a weight row's 272 bytes into registers -
//               which frees the buffer for the next piece once the last word is there - and turns them block after block into f16 in the canonical K-major
//               no-swizzle order (8 rows x 16 bytes core matrices), then fence.proxy.async and arrive.  The groups take the steps in turn.
//   warp 17     one thread issues a turn's (one or two steps') 2 MT tcgen05.mma a step (K = 16 each) from shared-memory descriptors and commits
//               them to the turn's "empty" barrier, which frees its stages for the decoders and the copy warp.
// After the last step the decode warps read the accumulators with tcgen05.ld (lane = weight row, column = token) and write Y: for one
// token, the 32 lanes of a warp write 32 consecutive rows.  With ks > 1 a block of the cluster finishes its share of the columns: the
// others store their parts of those into its shared memory (the stages' and the raw bytes', no longer needed), and it adds the parts in
// the order of K.
// What bounds it.  At many tokens L2 (10.8 TB/s): a step of 32 columns moves the token tile and the rows' bytes, so two row tiles share
// a token tile (25 KB per 256 x 256 x 32) where one a block moved 41, and the tensor core, which needs 512 cycles of the step's 625; the
// sums of a unit, which all blocks write at about the same time, are a fifth.  At few tokens latency: the chain decode, fence, barrier,
// instruction.  The issuing thread took 390 cycles a step to make descriptors for 256 cycles of instructions; it makes them once.
// 12,288 x 2,048: 4,093 tokens 281 -> 241 us (sustained, 1.4 GHz under the power cap), 256 tokens 28.8 -> 25.0 -> 22.4;
// 512 x 2,048, one token: 20 -> 11.9 (K in four parts).
// Every wait is bounded; a wait that runs out records where in the error word, and the block still frees its tensor memory.
#include <cuda.h>   // CUtensorMap and its enums; the encoder's entry point is asked of the runtime, nothing links against the driver
#include "sz_common.cuh"
#include "sz_formats.cuh"

namespace {

constexpr int MC_BM = 128;        // weight rows a block
constexpr int MC_KT = 32;         // columns a step
constexpr int MC_PS = 64;         // columns of a unit of the packed tokens' order
constexpr int MC_SS = 256;        // columns a raw copy
constexpr int MC_RAW_ROW = 272;   // bytes of a row's 8 Q8_0 blocks
constexpr int MC_STEPS = MC_SS / MC_KT;   // steps a raw piece: one a Q8_0 block of a row
constexpr int MC_KS_MAX = 4;      // blocks along K at most
constexpr int MC_NT_MAX = 256;    // tokens a tile
constexpr int MC_TILES_MORE = 3;  // token tiles more than the fewest, so that the units fill the chip's last turn
constexpr int MC_DEC = 512;       // decode threads
constexpr int MC_THREADS = MC_DEC + 96;   // copy warp, decode warps, issue warp, raw copy warp
constexpr int MC_A_BYTES = MC_BM * MC_KT * 2;
constexpr int MC_RAW_BYTES = MC_BM * MC_RAW_ROW;
constexpr size_t MC_SMEM_MIN = 116 * 1024;   // one block a multiprocessor: blocks of clusters that wait for tensor memory another holds could wait for each other
constexpr u32 MC_WAIT = 4000000u; // polls before a wait gives up

struct McSmem {
    u64 full[8], empty[8], raw_full, raw_empty, acc_full, acc_empty;
    u32 tmem_base, failed;
};

// One arrival a warp: the arrivals of 32 lanes on one barrier are taken one after the other.  What the other lanes did before it is
// ordered by the __syncwarp (and by their own proxy fence, where the reader is a copy or the tensor core), then by the arrival's release.
__device__ __forceinline__ void mc_arrive_warp(u64* bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sz_smem_addr(bar)) : "memory");
}
// The raw words a warp's lanes have loaded are in registers: the buffer may be refilled.  The refill is a write of the async proxy, and a
// load that was only issued is ordered before it by nothing: released right after its loads, a buffer was at times overwritten under
// one (16 bytes of one weight row wrong for all tokens, seen with four groups and a saturated shared memory).  So the arrival's
// address depends on every word of every lane (`zero` is 0, which only the host knows), and every lane fences its reads.
template <int N>
__device__ __forceinline__ void mc_release_raw(u64* bar, const u32 (&W)[N], u32 zero) {
    u32 any = 0;
#pragma unroll
    for (int i = 0; i < N; i++) any |= W[i];
    any = __reduce_or_sync(0xffffffffu, any);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sz_smem_addr(bar) + (any & zero)) : "memory");
}
// A decode warp's wait, all lanes with one outcome (those that gave up leave together, and nobody waits for them at the next __syncwarp).
// The copy and issue warps wait in one lane: a lane that only waited could fall two phases behind and find its parity come round.
__device__ __forceinline__ bool mc_wait_warp(u64* bar, u32 phase) { return __all_sync(0xffffffffu, sz_mbar_wait(bar, phase, MC_WAIT)); }
__device__ __forceinline__ void mc_fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mc_tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void mc_tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mc_cluster_sync() { asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory"); }

// Shared-memory matrix descriptor, K-major, no swizzle: 8 rows x 16 bytes core matrices; `lbo` = bytes between the two core
// matrices an instruction reads along K, `sbo` = bytes between 8-row groups.  Bits: address >> 4 at 0, lbo >> 4 at 16, sbo >> 4 at
// 32, descriptor version 1 at 46, layout type 0 (none) at 61.
__device__ __forceinline__ u64 mc_desc(u32 smem_addr, u32 lbo, u32 sbo) {
    return (u64)((smem_addr & 0x3ffffu) >> 4) | ((u64)(lbo >> 4) << 16) | ((u64)(sbo >> 4) << 32) | (1ull << 46);
}
// Instruction descriptor, kind::f16: D = f32 (bit 4), A = B = f16 (0), both K-major (0), N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ u32 mc_idesc(int n) { return (1u << 4) | ((u32)(n >> 3) << 17) | ((u32)(MC_BM >> 4) << 24); }

__device__ __forceinline__ void mc_mma(u32 d_tmem, u64 a_desc, u64 b_desc, u32 idesc, u32 accumulate) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
        "  tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mc_commit(u64* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(sz_smem_addr(bar)) : "memory");
}

// A Q8_0 block that starts OFF bytes (even) into W -> 32 f16 weights, stored as the 4 chunks of 8 the block covers (chunk stride 16 * 128
// bytes).  A pair of bytes is always one half of a word.  A weight is d * q rounded once to f16; d is f16 and q an integer below 128, so
// the f16 product (one rounding of the exact product) is that same value.  q as f16: the byte with its sign bit flipped is q + 128, placed
// under exponent 0x64 it reads 1024 + q + 128, and 1152 is subtracted.
template <int OFF>
__device__ __forceinline__ void mc_decode_block(const u32* W, u8* __restrict__ dst) {
    const u32 d2 = __byte_perm(W[OFF / 4], 0, OFF % 4 ? 0x3232 : 0x1010);
    const __half2 dh = *(const __half2*)&d2;
    const u32 bias = 0x64806480u;   // 1152, twice
    const __half2 bh = *(const __half2*)&bias;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        u32 o[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int b = OFF + 2 + 2 * (4 * c + i);                      // first byte of the pair
            const u32 v = __byte_perm(W[b / 4] ^ 0x80808080u, 0x64646464u, b % 4 ? 0x4342 : 0x4140);
            const __half2 w = __hmul2(dh, __hsub2(*(const __half2*)&v, bh));
            o[i] = *(const u32*)&w;
        }
        *(uint4*)(dst + c * 16 * 128) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}
// G: decode groups, which take the steps in turn.  TS: the steps of a turn, which have one pair of barriers and one commit; SLOTS: turns in the ring.
// What the issuing thread does per step besides its instructions (a wait, a commit) is on the path: with one row tile - where shared memory
// has room for eight stages - two steps share it (12,288 x 2,048, 256 tokens 25.0 -> 22.4 us, 1 token 21.8 -> 18.8, 1,024 tokens 74 -> 63; four
// steps a turn 22.1 where two give 21.9 on the same day, eight stages of one step each 28).  mc_deep says where the ring of four stages is better.
template <int MT, bool DEEP> struct McTurn {
    static_assert(!DEEP || MT == 1, "two row tiles leave no room for the deep ring");
    static constexpr int G = MC_DEC / (MT * MC_BM), TS = DEEP ? 2 : 1, STAGES = DEEP ? 8 : 4, SLOTS = STAGES / TS;
};
// The block of a piece that step j takes: the decode groups in turn, each the next of its blocks.
template <int MT>
__device__ __forceinline__ int mc_block(int j) { constexpr int G = MC_DEC / (MT * MC_BM); return j % G * (MC_STEPS / G) + j / G; }
// Group g of G has blocks g * 8 / G on of a row's eight, from the 16 bytes on that its first one starts in: 8 / G blocks, their number I
// known at compile time.
template <int G>
__device__ __forceinline__ int mc_group_start(int g) { return g * (MC_RAW_ROW / G) / 16 * 16; }
template <int G, int I>
__device__ __forceinline__ void mc_decode_of(int g, const u32* W, u8* __restrict__ dst) {
    constexpr int S = MC_RAW_ROW / G;
    if (g == 0) mc_decode_block<34 * I>(W, dst);
    else if (g == 1) mc_decode_block<S % 16 + 34 * I>(W, dst);
    else if (G == 4 && g == 2) mc_decode_block<2 * S % 16 + 34 * I>(W, dst);
    else if (G == 4) mc_decode_block<3 * S % 16 + 34 * I>(W, dst);
}

// The token rows as f16 in the order the instruction reads them from shared memory, so that a step's tile is one contiguous copy:
// out[tile][step][chunk c of 8 columns][token t][8 halves]; tokens past m are zero.  One thread a 16-byte unit.
__global__ void __launch_bounds__(256) sz_x16_pack_kernel(const float* __restrict__ x, long long xs, int m, int cols, int nt, int tiles, uint4* __restrict__ out) {
    const int steps = cols / MC_PS;
    const long long units = (long long)tiles * steps * 8 * nt;
    sz_pdl_wait();
    sz_pdl_trigger();
    for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < units; u += (long long)gridDim.x * blockDim.x) {
        const int t = (int)(u % nt);
        long long r = u / nt;
        const int c = (int)(r % 8); r /= 8;
        const int ks = (int)(r % steps);
        const int tile = (int)(r / steps);
        const int tok = tile * nt + t;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (tok < m) {
            const float4* p = (const float4*)(x + (long long)tok * xs + ks * MC_PS + c * 8);
            const float4 a = __ldg(p), b = __ldg(p + 1);
            __half2 h0 = __floats2half2_rn(a.x, a.y), h1 = __floats2half2_rn(a.z, a.w), h2 = __floats2half2_rn(b.x, b.y), h3 = __floats2half2_rn(b.z, b.w);
            v = make_uint4(*(u32*)&h0, *(u32*)&h1, *(u32*)&h2, *(u32*)&h3);
        }
        out[u] = v;
    }
}

template <int I> struct McInt { static constexpr int value = I; };

struct McArgs {
    const uint4* x16;
    float* y;
    long long ys;
    int rows, cols, m, nt, tiles, ks;   // nt: tokens a tile; ks: blocks of a cluster, the parts of K
    u32* err;
    u32 zero;                             // 0 (mc_release_raw)
};

// grid: ks == 1, up to 148 blocks that take (row tile, token tile) units in turn; else (units * ks), cluster (ks).
template <int MT, bool DEEP>
__global__ void __launch_bounds__(MC_THREADS, 1)
sz_mma_cols_q8_kernel(const __grid_constant__ CUtensorMap wmap, const McArgs a) {
    extern __shared__ __align__(128) u8 smem[];
    const int nt = a.nt, b_bytes = nt * MC_KT * 2;
    u8* raw = smem;                                   // [MT * 128 rows][272]
    u8* sa = raw + MT * MC_RAW_BYTES;                 // [stages][MT][4 chunks][16 row groups][128]
    using R = McTurn<MT, DEEP>;
    constexpr int G = R::G, TS = R::TS, SLOTS = R::SLOTS, STAGES = R::STAGES;
    u8* sb = sa + STAGES * MT * MC_A_BYTES;           // [stages][4 chunks][nt / 8 token groups][128]
    McSmem* S = (McSmem*)(sb + STAGES * b_bytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rtiles = (a.rows + MT * MC_BM - 1) / (MT * MC_BM), units = rtiles * a.tiles;
    const int kr = (int)blockIdx.x % a.ks, u0 = (int)blockIdx.x / a.ks, us = (int)gridDim.x / a.ks;
    const int P = a.cols / MC_SS, p0 = P * kr / a.ks, pieces = P * (kr + 1) / a.ks - p0, steps = pieces * MC_STEPS;
    constexpr int LAST = MC_DEC / 32;                 // the last decode warp

    if (threadIdx.x == 0) {
        for (int i = 0; i < SLOTS; i++) { sz_mbar_init(&S->full[i], TS * MT * MC_BM / 32 + 1); sz_mbar_init(&S->empty[i], 1); }
        sz_mbar_init(&S->raw_full, 1); sz_mbar_init(&S->raw_empty, MC_DEC / 32);
        sz_mbar_init(&S->acc_full, 1); sz_mbar_init(&S->acc_empty, MC_DEC / 32);
        S->failed = 0;
        sz_mbar_fence_init();
    }
    if (warp == 0) {   // tensor memory for the accumulators: MT x 256 columns, the whole warp asks
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sz_smem_addr(&S->tmem_base)), "r"((u32)MT * 256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    mc_tc_fence_before();
    __syncthreads();
    mc_tc_fence_after();
    const u32 tmem = S->tmem_base;
    int failed = 0;

    // A turn's slot is its number % SLOTS; T counts the turns of all units (a piece is whole turns of the ring), n the units.
    if (warp == 0) {
        // ---- token tiles as stages come free (what the pack kernel wrote: after the dependency wait)
        sz_pdl_wait();
        sz_pdl_trigger();
        asm volatile("fence.proxy.async.global;" ::: "memory");   // the pack kernel's stores, visible since the wait, before the copies' reads
        for (int u = lane == 0 ? u0 : units, T = 0; u < units && !failed; u += us) {
            const u8* src = (const u8*)a.x16 + ((size_t)(u / rtiles) * (a.cols / MC_KT) + p0 * MC_STEPS) * b_bytes;
            for (int j = 0; j < steps; j += TS, T++) {
                const int sl = T % SLOTS;
                if (T >= SLOTS && !sz_mbar_wait(&S->empty[sl], (T / SLOTS - 1) & 1, MC_WAIT)) { failed = 1; break; }
                sz_mbar_expect_tx(&S->full[sl], (u32)(TS * b_bytes));
#pragma unroll
                for (int s = 0; s < TS; s++)
                    sz_bulk_g2s(sb + (sl * TS + s) * b_bytes, src + (size_t)((j + s) / MC_STEPS * MC_STEPS + mc_block<MT>((j + s) % MC_STEPS)) * b_bytes, (u32)b_bytes, &S->full[sl]);
            }
        }
        __syncwarp();
    } else if (warp == LAST + 2) {
        // ---- raw weight bytes, a piece as soon as the decoders have the one before it in registers (mc_release_raw)
        for (int u = lane == 0 ? u0 : units, n = 0; u < units && !failed; u += us)
            for (int p = 0; p < pieces; p++, n++) {
                if (n > 0 && !sz_mbar_wait(&S->raw_empty, (n - 1) & 1, MC_WAIT)) { failed = 2; break; }
                // x = 136 * piece words = 272 * piece bytes: a multiple of 16; rows past the matrix arrive as zeros
                sz_mbar_expect_tx(&S->raw_full, (u32)(MT * MC_RAW_BYTES));
#pragma unroll
                for (int mt = 0; mt < MT; mt++)
                    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                                     sz_smem_addr(raw + mt * MC_RAW_BYTES)),
                                 "l"(&wmap), "r"((p0 + p) * (MC_RAW_ROW / 2)), "r"((u % rtiles * MT + mt) * MC_BM), "r"(sz_smem_addr(&S->raw_full))
                                 : "memory");
            }
        __syncwarp();
    } else if (warp == LAST + 1) {
        // ---- issue: one thread, descriptors of the ring's first stage made once (a step is 256 cycles of the tensor core
        // at 256 tokens and MT = 1: what this thread does besides its instructions is on the path)
        if (lane == 0) {
            const u32 idesc = mc_idesc(nt);
            const u64 ad = mc_desc(sz_smem_addr(sa), MC_BM * 16, 128), bd = mc_desc(sz_smem_addr(sb), (u32)nt * 16, 128);
            u32 phase = 0;
            for (int u = u0, n = 0; u < units && !failed; u += us, n++) {
                if (n > 0 && !sz_mbar_wait(&S->acc_empty, (n - 1) & 1, MC_WAIT)) { failed = 7; break; }
                for (int j = 0; j < steps; j += STAGES, phase ^= 1) {
#pragma unroll
                    for (int sl = 0; sl < SLOTS; sl++) {
                        if (!sz_mbar_wait(&S->full[sl], phase, MC_WAIT)) { failed = 5; break; }
                        mc_tc_fence_after();
#pragma unroll
                        for (int st = sl * TS; st < sl * TS + TS; st++)
#pragma unroll
                            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                                for (int q = 0; q < MC_KT / 16; q++)      // (addresses are in 16-byte units, in the low bits)
                                    mc_mma(tmem + mt * 256, ad + (u32)((st * MT + mt) * (MC_A_BYTES / 16) + q * 2 * MC_BM), bd + (u32)(st * (nt * MC_KT / 8) + q * 2 * nt), idesc, (j | st | q) ? 1u : 0u);
                        mc_commit(&S->empty[sl]);
                    }
                    if (failed) break;
                }
                mc_commit(&S->acc_full);      // arrives when every instruction above has finished (also after a failure: nothing pending then)
            }
        }
        __syncwarp();
    } else {
        // ---- decode: thread d has row d % (128 MT) and 8 / G blocks of it; then the accumulators to Y.  A warp reads the 32 lanes of
        // its quadrant (warp % 4), the four warps of a quadrant take every fourth 16 columns.
        constexpr int NW = MC_RAW_ROW / 16 / G + 1;      // 16-byte words of a group's blocks
        const int d = threadIdx.x - 32, g = d / (MT * MC_BM), r = d % (MT * MC_BM), mtd = r >> 7;
        u8* const dst0 = sa + mtd * MC_A_BYTES + ((r & 127) >> 3) * 128 + (r & 7) * 16;
        const int quad = warp & 3, part = (warp - 1) >> 2;
        auto load16 = [&](int mt, int c, u32* v) {
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                         : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                           "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                         : "r"(tmem + ((u32)(quad * 32) << 16) + (u32)(mt * 256 + c)));
        };
        auto loaded16 = [&](u32* v) {     // the registers go through the wait, so that nothing uses them before it
            asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                         "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]) :: "memory");
        };
        auto store16 = [&](int u, int mt, int c, const u32* v) {
            const int row = (u % rtiles * MT + mt) * MC_BM + quad * 32 + lane, tok = u / rtiles * nt + c;
            if (row >= a.rows) return;
            float* y = a.y + (long long)tok * a.ys + row;
            if (tok + 16 <= a.m) {
#pragma unroll
                for (int i = 0; i < 16; i++, y += a.ys) *y = __uint_as_float(v[i]);
            } else {
#pragma unroll
                for (int i = 0; i < 16; i++, y += a.ys)
                    if (tok + i < a.m) *y = __uint_as_float(v[i]);
            }
        };
        int k0 = 0, n = 0, np = 0;
        for (int u = u0; u < units && !failed; u += us, n++) {
            for (int p = 0; p < pieces && !failed; p++, np++, k0 += MC_STEPS) {
                if (!mc_wait_warp(&S->raw_full, np & 1)) { failed = 4; break; }
                u32 W[NW * 4];
                const uint4* rp = (const uint4*)(raw + (size_t)r * MC_RAW_ROW + mc_group_start<G>(g));
#pragma unroll
                for (int i = 0; i < NW; i++) { const uint4 v = rp[i]; W[4 * i] = v.x; W[4 * i + 1] = v.y; W[4 * i + 2] = v.z; W[4 * i + 3] = v.w; }
                mc_release_raw(&S->raw_empty, W, a.zero);
                auto step = [&](auto I) {
                    constexpr int i = decltype(I)::value;
                    const int k = k0 + i * G + g, T = k / TS, sl = T % SLOTS;
                    if (failed) return;
                    if (T >= SLOTS && !mc_wait_warp(&S->empty[sl], (T / SLOTS - 1) & 1)) { failed = 3; return; }
                    mc_decode_of<G, i>(g, W, dst0 + k % STAGES * MT * MC_A_BYTES);
                    mc_fence_async();                 // every lane's stores, before the tensor core reads them through the async proxy:
                    mc_arrive_warp(&S->full[sl]);     // fence, warp, arrival; the issuing thread waits and goes through tcgen05.fence
                };
                step(McInt<0>()); step(McInt<1>());
                if constexpr (G == 2) { step(McInt<2>()); step(McInt<3>()); }
            }
            if (!failed && !mc_wait_warp(&S->acc_full, n & 1)) failed = 6;
            mc_tc_fence_after();
            if (a.ks == 1) {
                if (!failed) {
                    for (int t = part; t < MT * (nt / 16); t += 4) {
                        u32 v[16];
                        const int mt = MT == 2 && t >= nt / 16, c = (t - mt * (nt / 16)) * 16;
                        load16(mt, c, v);
                        loaded16(v);
                        store16(u, mt, c, v);
                    }
                    mc_tc_fence_before();
                    mc_arrive_warp(&S->acc_empty);
                }
                continue;
            }
            // one unit: its sums are the cluster's
            const int nu = nt / 16;
            auto unit0 = [&](int rank) { return nu * rank / a.ks; };   // the 16-column units a block finishes
            mc_cluster_sync();           // every block of the cluster is done with its stages: they take the other blocks' parts
            if (!failed)
                for (int o = 0; o < a.ks; o++) {
                    if (o == kr) continue;
                    const int c0 = unit0(o), cn = unit0(o + 1) - c0, slot = kr < o ? kr : kr - 1;
                    u32 base;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base) : "r"(sz_smem_addr(smem)), "r"(o));
                    for (int t = part; t < MT * cn; t += 4) {
                        u32 v[16];
                        const int mt = t / cn, c = t - mt * cn;
                        load16(mt, (c0 + c) * 16, v);
                        loaded16(v);
                        const u32 at = base + (u32)((((slot * MT + mt) * cn + c) * 16 * 128 + quad * 32 + lane) * 4);
#pragma unroll
                        for (int i = 0; i < 16; i++) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at + (u32)i * 512u), "r"(v[i]) : "memory");
                    }
                }
            mc_cluster_sync();           // .. which are here now
            if (!failed) {
                const int c0 = unit0(kr), cn = unit0(kr + 1) - c0;
                for (int t = part; t < MT * cn; t += 4) {
                    u32 v[16];
                    float s[16];
                    const int mt = t / cn, c = t - mt * cn;
                    load16(mt, (c0 + c) * 16, v);
                    loaded16(v);
                    for (int k = 0; k < a.ks; k++) {        // in the order of K, whoever has the part
                        const float* part_k = (const float*)smem + (size_t)(((k < kr ? k : k - 1) * MT + mt) * cn + c) * 16 * 128 + quad * 32 + lane;
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            const float x = k == kr ? __uint_as_float(v[i]) : part_k[i * 128];
                            s[i] = k == 0 ? x : s[i] + x;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 16; i++) v[i] = __float_as_uint(s[i]);
                    store16(u, mt, (c0 + c) * 16, v);
                }
            }
        }
    }
    if (failed) atomicMax(&S->failed, (u32)failed);
    if (a.ks > 1 && (warp == 0 || warp > LAST)) { mc_cluster_sync(); mc_cluster_sync(); }    // the decoders' two
    mc_tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        mc_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((u32)MT * 256u) : "memory");
    }
    if (threadIdx.x == 0 && S->failed) atomicMax(a.err, S->failed);
}

// What a call takes: 128-row tiles a block (mt), blocks along K (ks), token tiles of nt tokens.  The least of an estimate in microseconds,
// with what was measured put into it: a piece of 256 columns takes a block 1.85 us with one row tile and 3.2 with two at 256 tokens, of
// which 0.35 and 1 go with the tokens (the rest is decoding); L2 gives the blocks that run together 10.8 TB/s; the sums go to memory at
// 6.5 TB/s; a cluster's exchange costs a little for each block of it, and of clusters of 2, 3 and 4 blocks the chip holds 74, 45 and 33 at
// once.  So two row tiles win where the units are many (the tokens cross L2 half as often), parts of K where they are few, and a token
// tile more than the fewest where it fills the last turn.  With one token tile the estimate does not look at its width, so that a token's
// sums are the same however many tokens come with it.
struct McPlan { int mt, ks, nt, tiles; };
McPlan mc_plan(int rows, int cols, int m) {
    const int P = cols / MC_SS, t0 = (m + MC_NT_MAX - 1) / MC_NT_MAX;
    McPlan best = {};
    float least = -1.f;
    for (int tiles = t0; tiles <= t0 + (t0 > 1 && t0 < 8 ? MC_TILES_MORE : 0); tiles++)
        for (int mt = 1; mt <= 2; mt++)
            for (int ks = 1; ks <= MC_KS_MAX && ks <= P; ks++) {
                const int nt = (((m + tiles - 1) / tiles) + 15) & ~15, slots = ks == 1 ? 148 : ks == 2 ? 74 : ks == 3 ? 45 : 33;
                const int units = (rows + mt * MC_BM - 1) / (mt * MC_BM) * tiles, pieces = (P + ks - 1) / ks;
                const float w = tiles == 1 ? 1.f : nt / 256.f;
                auto turn = [&](int n) {      // n units at once
                    const float work = mt == 1 ? 1.5f + 0.35f * w : 2.2f + w, l2 = n * ks * (16.f * w + 4.35f * mt) * 7.6e-4f;
                    return pieces * (work > l2 ? work : l2) + n * mt * w * 0.02f + (ks > 1 ? 1.7f * ks - 1.1f + 1.8f * (mt - 1) : 0.f) + 2.f * (mt - 1);
                };
                const float cost = units / slots * turn(slots) + (units % slots ? turn(units % slots) : 0.f);
                if (least < 0.f || cost < 0.97f * least) { least = cost; best = {mt, ks, nt, tiles}; }
            }
    return best;
}

// Which ring a plan with one row tile a block takes.  The deep one asks for twice as much ahead, which stops paying when many blocks read
// wide token tiles of a large packed matrix at the same time.  Both rings measured at 400 plans (128 .. 12,288 rows, 512 .. 8,192 columns, 1 .. 8,000
// tokens; deep / ring of four): tiles of up to 192 tokens 0.80 .. 1.02, whatever the matrix; wider ones by the matrix and the blocks -
// 512 x 2,048 (128 blocks) 0.98 at 2,900 tokens, 1.10 at 3,870; 128 x 2,048 (32 blocks) 0.96 at 3,870; 512 x 4,096 1.08 at 1,822, 1.14 at 3,102;
// 256 x 8,192 1.05 at 1,822, 1.48 at 3,870; 1,024 x 3,072, K in one part, 0.98 at 2,846, 1.21 at 4,093.  The line below is never more than 2.5 % above the
// better of the two at any of them (0.1 % on average); tiles x parts >= 32, before it, lost up to 21 % against the ring of four.
bool mc_deep(const McPlan& p, int rows, int cols, int m) {
    const long long blocks = (long long)((rows + MC_BM - 1) / MC_BM) * p.tiles * p.ks;
    return p.nt <= 192 || (long long)m * cols + 30000 * (blocks < 148 ? blocks : 148) < 9500000;
}

typedef CUresult (*McEncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
McEncodeTiled mc_encoder() {
    static McEncodeTiled fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess) fn = (McEncodeTiled)p;
    }
    return fn;
}


template <int MT, bool DEEP>
int mc_launch(const CUtensorMap& wmap, const McArgs& a, cudaStream_t st) {
    size_t smem = MT * MC_RAW_BYTES + McTurn<MT, DEEP>::STAGES * (MT * MC_A_BYTES + (size_t)a.nt * MC_KT * 2) + sizeof(McSmem);
    if (smem < MC_SMEM_MIN) smem = MC_SMEM_MIN;
    static bool set = false;
    if (!set) {
        SZ_CUDA(cudaFuncSetAttribute(sz_mma_cols_q8_kernel<MT, DEEP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     MT * MC_RAW_BYTES + McTurn<MT, DEEP>::STAGES * (MT * MC_A_BYTES + MC_NT_MAX * MC_KT * 2) + (int)sizeof(McSmem)));
        set = true;
    }
    cudaLaunchConfig_t cfg = {};
    const int units = (a.rows + MT * MC_BM - 1) / (MT * MC_BM) * a.tiles;
    cfg.gridDim = dim3(a.ks > 1 ? units * a.ks : units < 148 ? units : 148);
    cfg.blockDim = dim3(MC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)a.ks;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.ks > 1 ? 2 : 1;
    SZ_CUDA(cudaLaunchKernelEx(&cfg, sz_mma_cols_q8_kernel<MT, DEEP>, wmap, a));
    sz_trace_mark("mma_cols_q8", st);
    return SZ_OK;
}

}  // namespace

// Bytes of scratch for up to m token rows of `cols` inputs: an error word and the f16 copy of the rows.
extern "C" int sz_mma_cols_scratch_bytes(int cols, int m, int64_t* bytes) {
    if (!bytes || m < 1 || cols < MC_SS || cols % MC_SS) return sz_fail(SZ_E_ARG, "sz_mma_cols_scratch_bytes: m >= 1 and cols a multiple of %d", MC_SS);
    *bytes = 256 + ((int64_t)m + 16 * ((m + MC_NT_MAX - 1) / MC_NT_MAX + MC_TILES_MORE)) * cols * 2;     // whichever tiling a matrix takes
    return SZ_OK;
}

// y[t * ys + r] = sum_k w[r][k] * x[t * xs + k] for t < m, r < w->rows (strides in floats; x rows 16-byte aligned).  w: Q8_0.
extern "C" int sz_mma_cols(const sz_tensor* w, uint64_t x, int64_t xs, uint64_t y, int64_t ys, int m, uint64_t scratch, int64_t scratch_bytes,
                           uint64_t stream) {
    if (!w || !w->data || !x || !y || !scratch) return sz_fail(SZ_E_ARG, "sz_mma_cols: null argument");
    if (w->type != SZ_TYPE_Q8_0) return sz_fail(SZ_E_TYPE, "sz_mma_cols: Q8_0 weights (type %d given)", w->type);
    int64_t need = 0;
    int rc = sz_mma_cols_scratch_bytes((int)w->cols, m, &need);
    if (rc) return rc;
    if (scratch_bytes < need) return sz_fail(SZ_E_SCRATCH, "sz_mma_cols: %lld bytes of scratch given, %lld needed", (long long)scratch_bytes, (long long)need);
    if ((x & 15) || (xs & 3) || (w->data & 15) || (scratch & 255)) return sz_fail(SZ_E_ARG, "sz_mma_cols: x rows and the weights 16-byte aligned, scratch 256-byte aligned");
    if (w->rows < 1) return sz_fail(SZ_E_ARG, "sz_mma_cols: no rows");
    cudaStream_t st = (cudaStream_t)stream;
    const int cols = (int)w->cols, rows = (int)w->rows;
    const McPlan plan = mc_plan(rows, cols, m);
    const int nt = plan.nt, tiles = plan.tiles;
    u32* err = (u32*)scratch;
    uint4* x16 = (uint4*)(scratch + 256);
    McEncodeTiled enc = mc_encoder();
    if (!enc) return sz_fail(SZ_E_CUDA, "sz_mma_cols: the driver has no cuTensorMapEncodeTiled");
    CUtensorMap wmap;
    {   // the matrix as [rows][row bytes / 2] 16-bit words; a box is 272 bytes of 128 rows
        const cuuint64_t row_bytes = (cuuint64_t)(cols / 32) * 34;
        const cuuint64_t gdim[2] = {row_bytes / 2, (cuuint64_t)rows}, gstride[1] = {row_bytes};
        const cuuint32_t box[2] = {MC_RAW_ROW / 2, MC_BM}, es[2] = {1, 1};
        const CUresult r = enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, (void*)w->data, gdim, gstride, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return sz_fail(SZ_E_CUDA, "sz_mma_cols: cuTensorMapEncodeTiled failed (%d)", (int)r);
    }
    const long long units = (long long)tiles * (cols / MC_PS) * 8 * nt;
    SZ_CUDA(sz_launch("x16_pack", sz_x16_pack_kernel, dim3((unsigned)((units + 255) / 256 < 1184 ? (units + 255) / 256 : 1184)), dim3(256), 0, st, true,
                      (const float*)x, (long long)xs, m, cols, nt, tiles, x16));
    McArgs a;
    a.x16 = x16; a.y = (float*)y; a.ys = (long long)ys; a.rows = rows; a.cols = cols; a.m = m; a.nt = nt; a.tiles = tiles; a.ks = plan.ks; a.err = err; a.zero = 0;
    if (plan.mt == 2) return mc_launch<2, false>(wmap, a, st);
    return mc_deep(plan, rows, cols, m) ? mc_launch<1, true>(wmap, a, st) : mc_launch<1, false>(wmap, a, st);
}

// Clears (init != 0) or reads the scratch's error word; reading synchronises the stream.  0: no wait of a kernel ran out.
extern "C" int sz_mma_cols_status(uint64_t scratch, int init, int* code, uint64_t stream) {
    if (!scratch) return sz_fail(SZ_E_ARG, "sz_mma_cols_status: null scratch");
    cudaStream_t st = (cudaStream_t)stream;
    if (init) { SZ_CUDA(cudaMemsetAsync((void*)scratch, 0, 256, st)); return SZ_OK; }
    if (!code) return sz_fail(SZ_E_ARG, "sz_mma_cols_status: null code");
    u32 v = 0;
    SZ_CUDA(cudaMemcpyAsync(&v, (const void*)scratch, 4, cudaMemcpyDeviceToHost, st));
    SZ_CUDA(cudaStreamSynchronize(st));
    *code = (int)v;
    return v ? sz_fail(SZ_E_CUDA, "sz_mma_cols: a bounded wait of the kernel ran out (stage %u)", v) : SZ_OK;
}
