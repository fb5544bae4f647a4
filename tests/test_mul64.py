"""The FP64 product on integer pipes (cf_mul64.cuh, plain C++ here) against the
hardware's, bit for bit: random significands over the exponents it takes and past
them, ties, carries out of the rounding, zeros, subnormals, infinities and NaNs."""
import os
import subprocess

import pytest

SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include "cf_mul64.cuh"
using namespace cf;
static uint64_t bits(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
static double from(uint64_t u) { double d; memcpy(&d, &u, 8); return d; }
static long long bad = 0;
static void check(double a, double b) {
    volatile double x = a, y = b;
    const double want = x * y, got = mul64i(a, b);
    if (std::isnan(want) ? !std::isnan(got) : bits(want) != bits(got)) {
        if (bad++ < 5) printf("%a * %a: %a, not %a\n", a, b, got, want);
    }
}
int main(int, char** argv) {
    std::mt19937_64 g(atoll(argv[1]));
    const uint64_t mant = (1ull << 52) - 1;
    // edges of the significand and of the exponent range, every pair
    const uint64_t ms[] = {0, 1, 2, 3, mant, mant - 1, mant - 2, 1ull << 51, (1ull << 51) - 1, (1ull << 51) + 1,
                           0x5555555555555ull, 0xaaaaaaaaaaaaaull, 0xffffffffull, 0x100000000ull, 0x6a09e667f3bcdull,
                           0x6a09e667f3bccull, 1ull << 26, 1ull << 31};
    const int es[] = {0, 1, 500, 639, 640, 641, 1000, 1022, 1023, 1024, 1150, 1151, 1152, 1500, 2046, 2047};
    for (uint64_t ma : ms)
        for (uint64_t mb : ms)
            for (int ea : es)
                for (int eb : es)
                    for (int s = 0; s < 4; ++s)
                        check(from((uint64_t)(s & 1) << 63 | (uint64_t)ea << 52 | ma),
                              from((uint64_t)(s >> 1) << 63 | (uint64_t)eb << 52 | mb));
    for (int k = 0; k < 3000000; ++k) {
        const uint64_t r = g(), q = g();
        uint64_t ma = r & mant, mb = q & mant;
        // short significands meet ties often
        if (k % 3 == 1) ma &= ~0ull << (g() % 52);
        if (k % 3) mb &= ~0ull << (g() % 52);
        const uint64_t ea = 560 + (r >> 52) % 670, eb = 560 + (q >> 52) % 670;
        check(from((r & 1ull << 63) | ea << 52 | ma), from((q & 1ull << 63) | eb << 52 | mb));
    }
    return bad != 0;
}
"""


@pytest.mark.parametrize("seed", [1, 2])
def test_product_is_the_hardware_one(tmp_path, seed):
    here = os.path.dirname(os.path.abspath(__file__))
    csrc = os.path.join(here, "..", "cajitafluids_gb300", "csrc")
    cpp = tmp_path / "m.cpp"
    cpp.write_text(SRC)
    exe = tmp_path / "m"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", csrc, str(cpp), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), str(seed)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
