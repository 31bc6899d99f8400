"""The iterations' division by sigma (csrc/common.cuh: SigmaDivisor) against the division itself,
on the host: the same operations, each correctly rounded, as on the GPU."""
import subprocess

from saddlepoint_b200 import build

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>
#include "common.cuh"

static bool same(double a, double b) { return (std::isnan(a) && std::isnan(b)) || !memcmp(&a, &b, sizeof a); }
static double with_bits(uint64_t b) { double v; memcpy(&v, &b, sizeof v); return v; }
static uint64_t bits_of(double v) { uint64_t b; memcpy(&b, &v, sizeof b); return b; }

int main() {
    std::mt19937_64 rng(7);
    long pairs = 0, fast = 0, bad = 0;
    auto check = [&](const sp::SigmaDivisor &d, double s, double y) {
        const volatile double sv = s, yv = y;
        ++pairs;
        if (!same(d(y), yv / sv) && ++bad <= 5) printf("%a / %a: %a, not %a\n", y, s, d(y), yv / sv);
    };
    auto around = [](std::vector<double> &v, double x) {  // x and its neighbours, of both signs
        for (double u : {std::nextafter(x, 0.0), x, std::nextafter(x, INFINITY)}) v.insert(v.end(), {u, -u});
    };
    const double top = std::numeric_limits<double>::max(), tiny = std::numeric_limits<double>::denorm_min();
    // the ranges' ends, mantissas at both ends, the excluded ones, zeros, denormals, infinities, NaN
    std::vector<double> ss = {0.0, -0.0, INFINITY, -INFINITY, NAN}, ys = ss;
    for (double e : {0x1p-400, 0x1p400, 1.0, 0x1p-1, 0x1p300}) {
        around(ss, e);
        for (uint64_t m : {0xfffffffffffffull, 0xffffefffffffffull, 0xfffff00000000ull, 0xffffeffffffffull, 0xffffe00000000ull, 1ull})
            ss.push_back(with_bits((bits_of(e) & ~0xfffffffffffffull) | (m & 0xfffffffffffffull)));
    }
    for (double e : {0x1p-500, 0x1p500, 1.0, 0x1p-1022, tiny, top, 0x1p-1000, 0x1p900}) {
        around(ys, e);
        ys.push_back(with_bits(bits_of(e) | 0xfffffffffffffull));
    }
    for (double s : ss)
        for (double y : ys) check(sp::SigmaDivisor(s), s, y);
    // random ones over the whole ranges, and quotients next to a rounding boundary
    std::uniform_real_distribution<double> mant(1.0, 2.0);
    std::uniform_int_distribution<int> es(-401, 400), ey(-501, 500), near(-12, 12);
    for (int k = 0; k < 200000; ++k) {
        const double s = std::ldexp(k % 3 ? mant(rng) : with_bits(bits_of(1.0) | (rng() & 0xfffffffffffffull)), k % 5 ? near(rng) : es(rng));
        const sp::SigmaDivisor d(s);
        fast += d.ok;
        for (int i = 0; i < 40; ++i) {
            const double q = std::ldexp(mant(rng), near(rng));
            check(d, s, std::ldexp(mant(rng), i % 4 ? near(rng) : ey(rng)) * (i & 1 ? 1.0 : -1.0));
            const double p = q * s;  // y near (q + half a unit) * s
            for (double y : {p, std::nextafter(p, INFINITY), std::nextafter(p, 0.0), std::fma(0.5 * (std::nextafter(q, INFINITY) - q), s, p)})
                check(d, s, y);
        }
    }
    printf("%ld pairs, %ld divisors on the short path, %ld differ\n", pairs, fast, bad);
    return bad != 0 || fast < 150000;
}
"""


def test_sigma_divisor_gives_the_quotients_bits(tmp_path):
    src = tmp_path / "sigma.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "sigma"
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-O2", "--fmad=false", "-Xcompiler", "-ffp-contract=off",
                    "-I", build.CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
