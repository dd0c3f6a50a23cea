"""The device divides by the constants of its Gaussians through their reciprocals (div_const:
an estimate corrected once by its exact remainder) and takes floor() of a bounded value
through a sum rounded down.  Both must be the correctly rounded result.  Shown here for
every f32 wavelength in [380, 780] nm and every width of the colour matching and spectrum
lobes, and for every exponent argument of the polynomial exponential, in C++ with the same
fused operations."""
from __future__ import annotations

import subprocess

import pytest

LOBES = [(501.1, 20.4, 26.2), (599.8, 37.9, 31.0), (442.0, 16.0, 26.7), (530.9, 16.3, 31.1), (568.8, 46.9, 40.5),
         (459.0, 26.0, 13.8), (437.0, 11.8, 36.0), (615.0, 45.0, 65.0), (545.0, 45.0, 45.0), (465.0, 40.0, 45.0)]

SOURCE = r"""
#include <cfenv>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
static float f(uint32_t b) { float v; memcpy(&v, &b, 4); return v; }
static uint32_t u(float v) { uint32_t b; memcpy(&b, &v, 4); return b; }
static float div_const(float a, float c, float rc) { const float q = a * rc; return fmaf(fmaf(-c, q, a), rc, q); }
int main() {
    const float lobes[][3] = {LOBES};
    long bad = 0, n = 0;
    for (auto &l : lobes)
        for (uint32_t b = u(380.0f); b <= u(780.0f); ++b, ++n) {
            const float x = f(b), s = x < l[0] ? l[1] : l[2];
            bad += u(div_const(x - l[0], s, 1.0f / s)) != u((x - l[0]) / s);
        }
    // every argument the clamp of the exponential lets through
    volatile float magic = 12582912.0f;
    for (int sign = 0; sign < 2; ++sign)
        for (uint32_t b = 0; b <= u(sign ? 87.33654f : 88.02875f); ++b, ++n) {
            const float v = fmaf(f(b | (uint32_t)sign << 31), 1.44269504088896340736f, 0.5f);
            fesetround(FE_DOWNWARD);
            volatile float biased = v + magic;
            fesetround(FE_TONEAREST);
            const float whole = biased - magic;
            const int e = (int)floorf(v);
            bad += whole != floorf(v) || ((u(biased) + 127u) << 23) != (uint32_t)(e + 127) << 23;
            if (b > u(1.0f) || b % 64 == 0) continue;
            b += 61;  // below 1 the argument moves v by less than its last bits: a sample is enough
        }
    printf("%ld %ld\n", n, bad);
    return 0;
}
"""


def test_constant_division_and_floor_are_exact(tmp_path):
    rows = ", ".join("{%sf, %sf, %sf}" % t for t in LOBES)
    src, exe = tmp_path / "exact.cpp", tmp_path / "exact"
    src.write_text(SOURCE.replace("{LOBES}", "{" + rows + "}"))
    r = subprocess.run(["g++", "-O1", "-mfma", "-frounding-math", "-ffp-contract=off", "-o", str(exe), str(src)],
                       capture_output=True, text=True)
    if r.returncode != 0:
        pytest.skip("no C++ compiler: " + r.stderr[-200:])
    n, bad = (int(v) for v in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert n > 80_000_000 and bad == 0, (n, bad)
