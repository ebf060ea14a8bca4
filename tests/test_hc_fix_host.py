"""The many-row reads' rounding to fixed point (csrc/sz_hc_fix.cuh), compiled for the host with the signed-overflow check on: sums of any
number of pieces are those of exact arithmetic modulo 2^64, ties to even, and nothing signed overflows on the way."""
import os
import struct
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from tests.util import ROOT

SHIM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#define __device__
#define __forceinline__ inline
typedef uint32_t u32;
typedef uint64_t u64;
template <class T, class F> static T bits(F f) { T t; memcpy(&t, &f, sizeof t); return t; }
static float __uint_as_float(u32 v) { return bits<float>(v); }
static long long __double_as_longlong(double v) { return bits<long long>(v); }
static int __double2hiint(double v) { return (int)(bits<u64>(v) >> 32); }
static long long __double2ll_rn(double v) {      // saturates; not a number: the least (cvt.rni.s64.f64)
    if (!(v >= -9223372036854775808.0)) return INT64_MIN;
    return v >= 9223372036854775808.0 ? INT64_MAX : llrint(v);
}
#include "sz_hc_fix.cuh"
int main() {                     // pieces of 16 pairs; the sums after each piece, taken back to the pieces' own
    float f[32];
    u64 a[16], sum[32] = {}, added = 0;
    while (fread(f, 4, 32, stdin) == 32) {
        for (int i = 0; i < 16; i++) a[i] = (u64)bits<u32>(f[2 * i]) | (u64)bits<u32>(f[2 * i + 1]) << 32;
        sz_hc_round<16>(a, sum);
        added++;
        for (int i = 0; i < 32; i++) {
            const long long v = (long long)(sum[i] - added * SZ_HC_MAGIC), one = (long long)sz_hc_fix(f[i]);
            fwrite(&v, 8, 1, stdout);
            fwrite(&one, 8, 1, stdout);
        }
    }
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("hc_fix")
    (d / "t.cpp").write_text(SHIM)
    exe = str(d / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wno-unknown-pragmas", "-fsanitize=signed-integer-overflow", "-fno-sanitize-recover=all", "-I",
                    os.path.join(ROOT, "shadow-engine_b200", "csrc"), str(d / "t.cpp"), "-o", exe], check=True)

    def go(pieces):
        p = subprocess.run([exe], input=pieces.astype("<f4").tobytes(), capture_output=True)
        assert p.returncode == 0, p.stderr.decode()[-500:]
        return np.frombuffer(p.stdout, "<i8").reshape(-1, 32, 2)
    return go


def fixed(f):
    """a * 2^40 to the nearest whole number, ties to even, as a saturating conversion has it."""
    if f != f:
        return -2 ** 63
    if f in (float("inf"), float("-inf")):
        return 2 ** 63 - 1 if f > 0 else -2 ** 63
    return max(-2 ** 63, min(2 ** 63 - 1, round(Fraction(f) * 2 ** 40)))


def check(run, pieces):
    pieces = np.asarray(pieces, np.float32)
    got, total = run(pieces), [0] * 32
    assert got.shape[0] == pieces.shape[0]
    for p, row in enumerate(pieces):
        for i, f in enumerate(row):
            one = fixed(float(f))
            total[i] += one
            want = struct.unpack("<q", struct.pack("<Q", total[i] % 2 ** 64))[0]
            assert got[p, i, 1] == one and got[p, i, 0] == want, "piece %d, half %d: %r" % (p, i, float(f))


@pytest.mark.parametrize("scale", [1e-12, 1e-6, 1.0, 300.0, 5e3, 1e9])
def test_sums_of_a_warps_pieces_are_exact(run, scale):
    check(run, np.random.default_rng(3).normal(size=(24, 32)) * scale)


def test_ties_limits_and_what_is_no_number(run):
    tie = np.float32(2.0 ** -41)      # half a place
    a = np.zeros((6, 32), np.float32)
    a[0, :8] = [tie, -tie, 3 * tie, -3 * tie, 5 * tie, 2 * tie, -0.0, np.float32(2.0 ** -149)]
    a[1] = np.nextafter(np.float32(2048), np.float32(0))
    a[2] = 2048.0
    a[3, :4] = [-2048.0, 2047.5, np.float32(8388607.5), np.float32(-8388608.0)]
    a[4, :4] = [np.inf, -np.inf, np.nan, np.float32(3.4e38)]
    a[5, :4] = [np.inf, -np.inf, np.nan, np.float32(3.4e38)]      # a second time: the sums leave 64 bits
    check(run, a)
