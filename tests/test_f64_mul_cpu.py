"""The integer products of the FP64 collision (csrc/lbm_f64.cuh), built for the
host and compared bit for bit with the host's IEEE multiplication: random
mantissas and exponents over the accepted range, mantissas next to powers of
two and to rounding ties, both signs."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
HEADER = os.path.join(HERE, "..", "cavityflow_cuda_gb300", "csrc", "lbm_f64.cuh")

PROGRAM = r"""
#include <cstdio>
#include "%s"
using namespace lbm::f64;
static uint64_t x = 0x9E3779B97F4A7C15ull;
static uint64_t next() { x ^= x << 13; x ^= x >> 7; x ^= x << 17; return x; }
// a double with exponent field in [1023 - 400, 1023 + 400] and a mantissa of one of several kinds
static double draw()
{
    uint64_t m = next() & 0xfffffffffffffull;
    switch (next() %% 6) {
    case 0: m &= ~0ull << (next() %% 52); break;            // few leading bits
    case 1: m = next() %% 4; break;                          // just above a power of two
    case 2: m = 0xfffffffffffffull - next() %% 4; break;     // just below one
    case 3: m = (1ull << (next() %% 52)) + next() %% 3; break;
    default: break;
    }
    const uint64_t e = 1023 - 400 + next() %% 801;
    uint64_t u = (next() & 1) << 63 | e << 52 | (m & 0xfffffffffffffull);
    double d;
    std::memcpy(&d, &u, 8);
    return d;
}
static int same(double got, double want, const char* what, double a, double b)
{
    if (bits_of(got) == bits_of(want)) return 0;
    printf("%%s %%a %%a: %%a, want %%a\n", what, a, b, got, want);
    return 1;
}
int main()
{
    int bad = 0;
    volatile double three = 3.0, c15 = 1.5, c45 = 4.5;
    const double w[] = {1.0 / 18.0, 1.0 / 36.0, 1.0 / 3.0};
    for (long i = 0; i < 20000000 && bad < 20; ++i) {
        volatile double a = draw(), b = draw();
        bad += !exp_ok(a) || is_zero(a);
        bad += same(mul(a, b), a * b, "mul", a, b);
        bad += same(mul(a, a), a * a, "square", a, a);
        bad += same(mul3(a), three * a, "mul3", a, 3);
        bad += same(mul1_5(a), c15 * a, "mul1_5", a, 1.5);
        bad += same(mul4_5(a), c45 * a, "mul4_5", a, 4.5);
        volatile double c = w[i %% 3];
        bad += same(mul(c, a), c * a, "weight", c, a);
    }
    const double out[] = {0.0, -0.0, 4.9e-324, 1e-310, 1e-200, 1e200, 1.0 / three * 0 + 1e308 * 10, -1e308 * 10};
    for (double a : out) bad += exp_ok(a);
    printf("checked\n");
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not found")
def test_integer_products_match_ieee(tmp_path):
    src = tmp_path / "f64mul.cu"
    src.write_text(PROGRAM % os.path.abspath(HEADER).replace("\\", "/"))
    exe = tmp_path / "f64mul"
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-o", str(exe), str(src)], check=True, capture_output=True,
                   timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("checked"), r.stdout[-2000:]
