"""The bidirectional weights' densities (csrc/bpt_density.h) are the reference's
double products rounded to float (diffuseObj.h:22-27, glossyObj.h:25-31), bit
for bit: the header is compiled as the device has it, without contraction, and
compared over every significand and exponent, subnormals, zeros, infinities
and NaN."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "bpt_density.h"
static float f_of(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static uint32_t u_of(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static uint64_t bad;
static void same(float got, float want) { bad += !(u_of(got) == u_of(want) || (got != got && want != want)); }
static void over(float x) { same(wr::over_pi(x), (float)((double)x * 0.31830988618379067153776752674503)); }
static void lobe(float power, float c) {
    same(wr::lobe_density(power, c),
         (float)(((double)power + 1.0) * (double)c * (0.31830988618379067153776752674503 * 0.5)));
}
int main() {
    for (uint32_t m = 0; m < 1u << 23; m++)                        // every significand in [1, 2)
        over(f_of(127u << 23 | m));
    for (uint64_t u = 0; u < 1ull << 32; u += 2003) over(f_of((uint32_t)u));   // every exponent and sign
    printf("over_pi %llu\n", (unsigned long long)bad);
    bad = 0;
    uint32_t r = 12345u;
    auto next = [&]() { return r = r * 1664525u + 1013904223u; };
    const float powers[] = {0.f, 1e-6f, 0.5f, 1.f, 3.f, 10.f, 100.f, 12345.678f, 1e6f, 1e9f, f_of(0x7f800000u)};
    for (float p : powers) {
        for (int k = 0; k < 400000; k++) lobe(p, f_of(next() & 0x7fffffffu));   // any c: also subnormal, infinite, NaN
        for (int k = 0; k < 400000; k++) lobe(p, f_of(u_of(1e-38f) + next() % (u_of(1e-30f) - u_of(1e-38f))));
        for (float c : {0.f, 1.f, f_of(1u), f_of(0x00800000u), f_of(0x7f800000u)}) lobe(p, c);
    }
    printf("lobe_density %llu\n", (unsigned long long)bad);
    return 0;
}
"""


@pytest.fixture(scope="module")
def differing(tmp_path_factory):
    d = tmp_path_factory.mktemp("density")
    src, exe = d / "density.cpp", d / "density"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "walkray_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return {k: int(v) for k, v in (line.split() for line in out.splitlines())}


@pytest.mark.parametrize("density", ["over_pi", "lobe_density"])
def test_density_is_the_double_product_rounded(differing, density):
    assert differing[density] == 0
