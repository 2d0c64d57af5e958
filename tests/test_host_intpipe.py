"""The integer-pipe FP64 arithmetic (csrc/intpipe.cuh) compiled for the host: correctly rounded
products, reciprocals, quotients and square roots must equal the IEEE operations bit for
bit on random, nearly equal and special operands, whatever the reciprocal seeds' last bits are;
x^a lies within 0.55 units in the last place of long double's."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

DRIVER = r'''
#include "intpipe.cuh"
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace cfd2d;
typedef unsigned long long u64;
static double dbl(u64 b) { double x; memcpy(&x, &b, 8); return x; }
static u64 bits(double x) { u64 b; memcpy(&b, &x, 8); return b; }
static bool same(double x, double y) { return bits(x) == bits(y) || (x != x && y != y); }
int main(int argc, char** argv) {
    const long n = atol(argv[1]);
    std::mt19937_64 g(atol(argv[2]));
    const double special[] = {0.0, -0.0, 1.0, -1.0, 0.5, 2.0, 1.0 / 0.0, -1.0 / 0.0, 0.0 / 0.0, 4.9e-324, 2.2e-308,
                              1.7e308, 0x1p-510, 0x1p510, 0x1.fffffffffffffp0, 0x1.0000000000001p0, 0x1p-511, 0x1p511};
    long bad = 0;
    auto rnd = [&](unsigned mode) {
        const int e = mode % 4 == 0 ? 1019 + (int)(g() % 8) : mode % 4 == 1 ? 963 + (int)(g() % 120) : mode % 4 == 2 ? (int)(g() % 2048) : 1023;
        u64 f = g() & 0xfffffffffffffull;
        if (mode % 5 == 1) f &= ~((1ull << (g() % 53)) - 1);
        if (mode % 7 == 2) f |= (1ull << (g() % 52)) - 1;
        return mode % 61 == 0 ? special[g() % 18] : dbl((g() << 63) | ((u64)e << 52) | f);
    };
    for (long i = 0; i < n; i++) {
        const unsigned m = (unsigned)(g() % 100000);
        double a = rnd(m), b = rnd(m / 7);
        if (i % 4 == 1) b = dbl((bits(a) ^ (g() << 63)) + g() % 5 - 2);  // nearly equal
        if (i % 8 == 3) a = rnd(0) * b;                                   // quotients near a double
        ip::seed_ulps() = (int)(g() % 5) - 2;
        const double x = i % 5 == 0 ? b * b : i % 5 == 1 ? dbl(bits(b * b) + g() % 3 - 1) : a;  // roots near a double
        const bool ok = same(ip::mul(a, b), a * b) && ip::less(a, b) == (a < b) && ip::not_negative(a) == (a >= 0) && ip::positive(a) == (a > 0) &&
                        same(ip::rcp(b), 1.0 / b) && same(ip::quot(a, b), a / b) && same(ip::sqrt(x), std::sqrt(x)) &&
                        same(ip::half(a), 0.5 * a) && same(ip::plus_zero(a), 0.0 + a);
        if (!ok && bad++ < 5) printf("%a %a %a\n", a, b, x);
        const double px = dbl((u64)(i % 3 ? 1022 + g() % 2 : 903 + g() % 240) << 52 | (g() & 0xfffffffffffffull));
        const double e = i % 2 ? 1.0 / 7.0 : 2.5, y = ip::pow(px, e);
        const long double t = powl((long double)px, (long double)e);
        if (!((double)fabsl(y - t) <= 0.55 * std::ldexp(1.0, std::ilogb((double)t) - 52)) && bad++ < 5) printf("pow %a %a\n", px, e);
    }
    return bad != 0;
}
'''


@pytest.mark.parametrize("n,seed", [(2_000_000, 1), (2_000_000, 2), (1000, 3)])
def test_matches_ieee_operations(tmp_path, n, seed):
    inc = next((p for p in ("/usr/local/cuda/include", os.path.join(os.environ.get("CUDA_HOME", ""), "include"))
                if os.path.exists(os.path.join(p, "cuda_runtime.h"))), None)
    if inc is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    src = tmp_path / "driver.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "driver"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(PKG, "csrc"), "-isystem", inc,
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(n), str(seed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
