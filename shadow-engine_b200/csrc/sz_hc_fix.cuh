// Fixed point of the hyper-connection reads' sums: 2^-40, 64 bits.  Integers may be added in any order, and a sum that leaves the range comes
// back when what took it out is subtracted again - so everything that is added is unsigned (the bits of two's complement; a signed
// sum may not overflow).  Needs nothing but u32, u64 and the conversions by name, so that a host can run it, too.
#pragma once

#define SZ_HC_FIX 1099511627776.0             // 2^40
#define SZ_HC_FIX_INV (1.0 / 1099511627776.0)

// Many rows round pieces without a conversion: a + 6144 = a + 1.5 * 2^12 has its last place at 2^-40, so the sum's bits are SZ_HC_MAGIC (those of
// 6144) + the rounded piece, ties to even as __double2ll_rn((double)a * 2^40) rounds them, while |a| < 2^11 - which the sum's exponent
// says; beyond it the conversion does it (it saturates).
#define SZ_HC_MAGIC 0x40B8000000000000ull
__device__ __forceinline__ u64 sz_hc_fix(float a) {
    if (fabsf(a) < 2048.0f) return (u64)__double_as_longlong((double)a + 6144.0) - SZ_HC_MAGIC;
    return (u64)__double2ll_rn((double)a * SZ_HC_FIX);
}
// sum[i] += SZ_HC_MAGIC + the rounded half i of the N pairs
template <int N>
__device__ __forceinline__ void sz_hc_round(const u64* a, u64* sum) {
    u32 all = 0xffffffffu, any = 0u;          // of the sums' upper words: one exponent for all, or not
#pragma unroll
    for (int i = 0; i < 2 * N; i++) {
        const u32 hi = (u32)__double2hiint((double)__uint_as_float((u32)(a[i >> 1] >> (32 * (i & 1)))) + 6144.0);
        all &= hi; any |= hi;
    }
    if ((all >> 20) == 0x40Bu && (any >> 20) == 0x40Bu) {
#pragma unroll
        for (int i = 0; i < 2 * N; i++) sum[i] += (u64)__double_as_longlong((double)__uint_as_float((u32)(a[i >> 1] >> (32 * (i & 1)))) + 6144.0);
    } else {
#pragma unroll
        for (int i = 0; i < 2 * N; i++) sum[i] += sz_hc_fix(__uint_as_float((u32)(a[i >> 1] >> (32 * (i & 1))))) + SZ_HC_MAGIC;
    }
}
