"""The step's quotients by a constant (hb_physics.cuh, divk_raw): one multiply
by the rounded reciprocal and one fused correction give the rounded quotient.
Restated in C with fma: every fp32 significand of both signs, and random and
near-midpoint fp64 dividends, for every constant the step divides by."""
import subprocess

SOURCE = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
static uint64_t mix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull; z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull; return z ^ (z >> 31);
}
int main(void) {
    const double cs[] = {3.0, 9.81, 39.24, 4.905, 313.92, 0.1, 10.0};
    long bad = 0;
    for (int i = 0; i < 7; i++) {
        const float c = (float)cs[i], y = 1.0f / c;
        for (uint32_t m = 0; m < (1u << 24); m++) {
            const uint32_t u = (127u << 23) | (m & 0x7FFFFFu) | (m >> 23 << 31);
            float x; memcpy(&x, &u, 4);
            const float q = x * y;
            bad += fmaf(fmaf(-q, c, x), y, q) != x / c;
        }
        const double d = cs[i], z = 1.0 / d;
        for (uint64_t n = 0; n < 2000000; n++) {
            const uint64_t a = mix(n + 77 * i), ub = (1023ull << 52) | (a & 0xFFFFFFFFFFFFFull);
            double x; memcpy(&x, &ub, 8);
            if (n & 1) x = fma(d, 0x1p-53, fma(d, x, 0.0));   /* about a midpoint of two quotients */
            const double q = x * z;
            bad += fma(fma(-q, d, x), z, q) != x / d;
        }
    }
    printf("%ld\n", bad);
    return bad != 0;
}
"""


def test_quotients_by_constants_are_correctly_rounded(tmp_path):
    src, exe = tmp_path / "q.c", tmp_path / "q"
    src.write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-mfma", "-o", str(exe), str(src), "-lm"], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout.strip() == "0"
