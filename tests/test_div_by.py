"""The division by a divisor used many times (div_by, csrc/ensc_cycle.cuh) rounds
as `/` does in the range that its comment states: the function is compiled for
the host from the header's own text and compared over magnitudes and at the
range's edges.  Below the range its remainders underflow, and it differs."""
import os
import re
import subprocess

from enscdynamics_b200 import build

MAIN = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#define __device__
#define __forceinline__ inline
static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
%s
static uint64_t s = 88172645463325252ull;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
// a double of exponent e: a random fraction, or one of few bits or all ones
static double num(int e) {
    uint64_t m = rnd() >> 12;
    const int kind = rnd() %% 8;
    if (kind == 0) m = 0;
    if (kind == 1) m = (1ull << 52) - 1;
    if (kind == 2) m &= 0xFull << 48;
    if (kind == 3) m |= ((1ull << 52) - 1) & ~0xFull;
    double d;
    const uint64_t b = (static_cast<uint64_t>(e + 1023) << 52) | m;
    memcpy(&d, &b, 8);
    return rnd() & 1 ? -d : d;
}
static int uni(int lo, int hi) { return lo + static_cast<int>(rnd() %% static_cast<uint64_t>(hi - lo + 1)); }
int main() {
    long tried = 0, off = 0, below = 0;
    for (long i = 0; i < 4000000; ++i) {
        // exponents spread over the range, one in four near its lower edge
        const int ex = i %% 4 ? uni(-969, 1022) : uni(-969, -960), ec = i %% 8 < 6 ? uni(-1020, 1020) : uni(-70, 70);
        if (ex - ec < -1020 || ex - ec > 1021) continue;
        const double x = num(ex), c = num(ec), r = 1.0 / c;
        ++tried;
        off += div_by(x, c, r) != x / c;
    }
    for (long i = 0; i < 200000; ++i) {
        const double x = num(uni(-1015, -1005)), c = num(uni(-5, 5));
        below += div_by(x, c, 1.0 / c) != x / c;
    }
    const double z = div_by(-0.0, 3.0, 1.0 / 3.0);
    printf("%%ld %%ld %%ld %%d\n", tried, off, below, z == 0.0);
    return 0;
}
"""


def test_rounds_as_the_division_in_its_range(tmp_path):
    with open(os.path.join(build.CSRC, "ensc_cycle.cuh")) as f:
        text = f.read()
    fn = re.search(r"__device__ __forceinline__ double div_by\(.*?\n}\n", text, re.S).group(0)
    assert "2^-969" in text[:text.index(fn)]
    src, exe = str(tmp_path / "div.cpp"), str(tmp_path / "div")
    with open(src, "w") as f:
        f.write(MAIN % fn)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-o", exe, src], check=True)
    tried, off, below, zero = map(int, subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split())
    assert tried > 2_000_000 and off == 0 and below > 0 and zero == 1
