"""Integer building blocks of the FP64 factorisations, compiled on the host from
the kernels' own headers: roots, reciprocal roots and quotients in fixed point (csrc/lla_int_math.h),
and the balanced digits, fixed-point values and 64-bit-to-double conversion of
the FP64 trailing update (csrc/lla_oz_digits.h).  The references are the
compiler's long double and integer arithmetic."""
import os
import shutil
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "linfa-linalg_gb300", "csrc")

HARNESS = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "lla_int_math.h"
#include "lla_oz_digits.h"
using namespace lla;
static long long bad = 0;
#define CHECK(c, ...) do { if (!(c) && bad++ < 5) std::printf(__VA_ARGS__); } while (0)
int main() {
    std::mt19937_64 g(7);
    // reciprocal roots: within one unit in the last place, any positive normal argument
    for (long t = 0; t < 2000000; ++t) {
        uint64_t b = g() & 0x7fffffffffffffffull;
        if (t % 5 == 0) b = (b & 0x000fffffffffffffull) | ((1021ull + g() % 5) << 52);
        if (t % 7 == 0) b &= ~0xffffffffffull;             // few mantissa bits
        if (t % 11 == 0) b |= 0x000ffffffffffff0ull;        // mantissa near the top
        if (!im_positive_normal(b)) continue;
        const double d = im_double(b), y = im_rsqrt(d);
        const long double want = 1.0L / sqrtl((long double)d);
        const double w = (double)want;
        const long double ulp = (long double)w - (long double)std::nextafter(w, 0.0);
        CHECK(fabsl((long double)y - want) <= ulp, "rsqrt(%a) = %a\n", d, y);
    }
    for (double d : {0.0, -0.0, -1.0, 5e-324, 2.2250738585072009e-308, HUGE_VAL, -HUGE_VAL, std::nan("")})
        CHECK(!im_positive_normal(im_bits(d)), "normal(%a)\n", d);
    CHECK(im_positive_normal(im_bits(2.2250738585072014e-308)) && im_positive_normal(im_bits(1.7976931348623157e308)), "ends\n");
    // quotients: IEEE division's where they say so, which is nearly always
    long taken = 0, refused = 0;
    for (long t = 0; t < 300000; ++t) {
        uint64_t db = g();
        if (t % 3) db = (db & 0x800fffffffffffffull) | ((1000ull + g() % 40) << 52);
        if (t % 5 == 0) db &= ~0xfffffffffffull;
        if (t % 7 == 0) db |= 0xfffffffffffffull;
        const double d = im_double(db);
        const ImDivisor v = im_divisor(d);
        for (int k = 0; k < 6; ++k) {
            uint64_t ab = g();
            if (k & 1) ab = (ab & 0x800fffffffffffffull) | ((1000ull + g() % 40) << 52);
            if (k == 2) ab = im_bits(im_double((g() & 0x000ffffffff00000ull) | (1023ull << 52)) * d);
            if (k == 4) ab &= 0x8000000000000000ull;
            const double a = im_double(ab);
            bool ok;
            const double q = im_div(a, v, ok);
            CHECK(!ok || im_bits(q) == im_bits(a / d), "%a / %a = %a\n", a, d, q);
            if (k == 3 && t % 3 && im_positive_normal(ab & ~(1ull << 63))) (ok ? taken : refused)++;
        }
    }
    CHECK(refused * 1000 < taken, "refused %ld of %ld\n", refused, taken);
    // roots: IEEE's, and the divisor they become
    for (long t = 0; t < 1000000; ++t) {
        uint64_t b = g() & 0x7fffffffffffffffull;
        if (t % 3 == 0) b = (b & 0x000fffffffffffffull) | ((1000ull + g() % 40) << 52);
        if (t % 5 == 0) b |= 0xfffffffffffffull;
        if (t % 7 == 0) b &= ~0xfffffffffffull;
        if (t % 11 == 0) b = im_bits(im_double((g() & 0x000ffffffc000000ull) | (1023ull << 52)));
        if (t % 13 == 0) b = im_bits(im_double((g() & 0x000fffffffffffffull) | ((1023ull + g() % 2) << 52)));
        if (t % 11 == 0 || t % 13 == 0) b = im_bits(im_double(b) * im_double(b));  // squares
        if (!im_positive_normal(b)) continue;
        ImDivisor v;
        const double d = im_double(b), r = im_sqrt(d, v);
        CHECK(im_bits(r) == im_bits(std::sqrt(d)), "sqrt(%a) = %a\n", d, r);
        const double a = im_double((g() & 0x800fffffffffffffull) | (((uint64_t)(v.e & 0x7ff) / 2 + 512) << 52));
        bool ok;
        const double q = im_div(a, v, ok);
        CHECK(!ok || im_bits(q) == im_bits(a / r), "%a / %a = %a\n", a, r, q);
    }
    // digits: V = nearest multiple of 2^(e-55), its seven balanced digits exact in BF16
    std::uniform_real_distribution<double> U(0.5, 1.0);
    for (long t = 0; t < 400000; ++t) {
        const int e = (int)(g() % 1601) - 800;
        int64_t v[2];
        double a[2];
        for (int u = 0; u < 2; ++u) {
            a[u] = std::ldexp(U(g), e - (int)(g() % 62));
            if (g() & 1) a[u] = -a[u];
            if (t % 101 == u) a[u] = t & 1 ? 0.0 : -0.0;
            if (t % 103 == u) a[u] = std::ldexp(std::nextafter(1.0, 0.0), e);
            v[u] = oz_fixed55((int64_t)im_bits(a[u]), e);
            const long double x = std::ldexp((long double)a[u], 55 - e);
            CHECK(fabsl(x - (long double)v[u]) <= 0.5L, "fixed(%a, %d)\n", a[u], e);
        }
        CHECK(oz_bits_exponent(im_bits(std::fabs(a[0]))) <= e || a[0] == 0, "exponent(%a)\n", a[0]);
        uint32_t q[kOzBal];
        oz_balanced_pair(v[0], v[1], q);
        for (int u = 0; u < 2; ++u) {
            int64_t s = 0;
            for (int p = 0; p < kOzBal; ++p) {
                const uint32_t w = (u ? q[p] & 0xffff0000u : q[p] << 16);
                float f;
                std::memcpy(&f, &w, 4);
                CHECK(std::fabs(f) <= 128.f && f == std::rint(f), "digit %g\n", f);
                s = s * 256 + (int64_t)f;
            }
            CHECK(s == v[u], "digits of %lld\n", (long long)v[u]);
        }
    }
    // the same for FP32 values: multiples of 2^(e-31), four digits
    for (long t = 0; t < 400000; ++t) {
        const int e = (int)(g() % 201) - 100;
        int64_t v[2];
        for (int u = 0; u < 2; ++u) {
            float a = (float)std::ldexp(U(g), e - (int)(g() % 36));
            if (std::fabs(a) >= std::ldexp(1.0, e)) a = std::nextafter((float)std::ldexp(1.0, e), 0.f);
            if (g() & 1) a = -a;
            if (t % 101 == u) a = t & 1 ? 0.f : -0.f;
            if (t % 103 == u) a = std::nextafter((float)std::ldexp(1.0, e), 0.f);
            int32_t b;
            std::memcpy(&b, &a, 4);
            v[u] = oz_fixed31(b, e);
            CHECK(std::fabs(std::ldexp((double)a, 31 - e) - (double)v[u]) <= 0.5, "fixed31(%a, %d)\n", a, e);
        }
        uint32_t q[kOzBal32];
        oz_balanced_pair(v[0], v[1], q);
        for (int u = 0; u < 2; ++u) {
            int64_t s = 0;
            for (int p = 0; p < kOzBal32; ++p) {
                const uint32_t w = (u ? q[p] & 0xffff0000u : q[p] << 16);
                float f;
                std::memcpy(&f, &w, 4);
                CHECK(std::fabs(f) <= 128.f && f == std::rint(f), "digit %g\n", f);
                s = s * 256 + (int64_t)f;
            }
            CHECK(s == v[u], "digits of %lld\n", (long long)v[u]);
        }
    }
    // 64-bit integer times a power of two, rounded to nearest even
    for (long t = 0; t < 1000000; ++t) {
        int64_t T = (int64_t)g() >> (g() % 64);
        if (T == INT64_MIN) T = 0;
        if (t % 3 == 0) T = (T >> 12 << 12) | 0x400;  // ties
        const int s = (int)(g() % 1900) - 1000;
        const double got = oz_scaled_double(T, s), want = (double)std::ldexp((long double)T, s);
        const bool sub = std::fabs(want) < 2.3e-308;   // subnormal results round twice
        CHECK(im_bits(got) == im_bits(want) || (T == 0 && got == 0) || (sub && std::fabs(got - want) <= 5e-324),
              "scaled(%lld, %d) = %a, %a\n", (long long)T, s, got, want);
    }
    std::printf("bad %lld\n", bad);
    return bad != 0;
}
"""


@pytest.mark.parametrize("seed_error", ["0.0f", "-2.4e-7f", "2.4e-7f"])
def test_integer_math_on_host(seed_error):
    """`seed_error`: relative error put on the FP32 seed (the hardware's is below 2^-22)."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        with open(src, "w") as f:
            f.write(HARNESS)
        subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", f"-DIM_SEED_ERROR={seed_error}", "-I", CSRC,
                        src, "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout


DIVISION = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "lla_int_math.h"
using namespace lla;
static float bits(uint32_t b) { float f; std::memcpy(&f, &b, 4); return f; }
static uint32_t ubits(float f) { uint32_t b; std::memcpy(&b, &f, 4); return b; }
int main() {
    std::mt19937_64 g(11);
    long long bad = 0, taken = 0, asked = 0;
    auto check = [&](float a, const FloatDivisor &v, bool want) {
        const float q = float_div(a, v), w = a / v.d;
        const bool ok = float_div_ok(a, q, v);
        if (ok && ubits(q) != ubits(w) && bad++ < 5) std::printf("%a / %a = %a, %a\n", a, v.d, q, w);
        if (want) ++asked, taken += ok;
    };
    for (long t = 0; t < 1500000; ++t) {
        uint32_t db = (uint32_t)g();
        if (t % 2) db = (db & 0x807fffffu) | ((100u + (uint32_t)(g() % 54)) << 23);
        if (t % 5 == 0) db |= 0x7fff00u;            // mantissas near the ends
        if (t % 7 == 0) db &= ~0x7fff00u;
        if (t % 11 == 0) db |= 0x7fffffu;
        const FloatDivisor v = float_divisor(bits(db));
        for (int k = 0; k < 8; ++k) {
            uint32_t ab = (uint32_t)g();
            if (k & 1) ab = (ab & 0x807fffffu) | ((100u + (uint32_t)(g() % 54)) << 23);
            if (k == 1) ab |= 0x7ffff0u;
            if (k == 3) ab &= ~0x7ffff0u;
            // next to a quotient, and next to the midpoint of two quotients
            if (k == 4) ab = ubits(bits((uint32_t)(g() & 0x7fffffu) | 0x3f800000u) * v.d) + (uint32_t)(g() % 3) - 1u;
            if (k == 6) ab = ubits((float)(((double)((g() & 0xffffffu) | 0x800000u) + 0.5) * (double)v.d * 0x1p-23));
            if (k == 2) ab &= 0x80000000u;
            check(bits(ab), v, k == 5 && t % 2);
        }
    }
    // every mantissa by a few divisors
    for (uint32_t db : {0x3f800001u, 0x3fffffffu, 0x3f7fffffu, 0xbfaaaaabu, 0x3fb504f3u})
        for (uint32_t m = 0; m < 1u << 23; ++m) check(bits(0x3f800000u | m), float_divisor(bits(db)), false);
    std::printf("bad %lld, taken %lld of %lld\n", bad, taken, asked);
    return bad != 0 || taken != asked;
}
"""


def test_float_division_on_host():
    """FP32 quotients by Markstein's corrections: IEEE division's wherever they say so, and always
    for exponents well inside the range."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        with open(src, "w") as f:
            f.write(DIVISION)
        subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, src, "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout
