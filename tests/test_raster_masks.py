"""The row masks of the raster's records (row_columns and mask_rows of csrc/spl_raster.cuh), compiled for the host by an
optimising compiler that holds them to the language's aliasing rules: every pixel that a record covers is in its mask, no
mask leaves the record's box, and a rectangle's mask reaches no further than its documented widening.  Tiles that the
box crosses, needles at any angle, records that no column bound holds for (axis-aligned A), both rectangle kinds."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HOST = r"""
#include <algorithm>
#include <cfenv>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__
#define __forceinline__ inline
using std::max; using std::memcpy; using std::min;
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
static inline float2 make_float2(float x, float y) { return {x, y}; }
static inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
static inline uint32_t __float_as_uint(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
static inline float as_float(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
static inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t n) {
    return (uint32_t)((((uint64_t)hi << 32 | lo) << (n & 31u)) >> 32);
}
static float directed(float a, float b, int mode) {
    const int was = std::fegetround();
    std::fesetround(mode);
    volatile float x = a, y = b, z = x + y;
    std::fesetround(was);
    return z;
}
static inline float __fadd_ru(float a, float b) { return directed(a, b, FE_UPWARD); }
static inline float __fadd_rd(float a, float b) { return directed(a, b, FE_DOWNWARD); }
static inline float2 add2(float2 a, float2 b) { return {a.x + b.x, a.y + b.y}; }
static inline float2 fma2(float2 a, float2 b, float2 c) { return {std::fmaf(a.x, b.x, c.x), std::fmaf(a.y, b.y, c.y)}; }
constexpr int RASTER_BATCH = 256;
"""

MAIN = r"""
static uint32_t s_pm[8][RASTER_BATCH];

template <bool RECT>
static int check(std::mt19937& gen) {
    auto u = [&](double a, double b) { return (float)std::uniform_real_distribution<double>(a, b)(gen); };
    const float margin = u(0, 1) < 0.5f ? 2.0f : u(0.5, 9.5);
    const int wx0 = 16 * (int)(gen() % 200), ty0 = 16 * (int)(gen() % 120);
    const float cx = wx0 + u(-12, 28), cy = ty0 + u(-12, 28), angle = u(0, 6.2832);
    const float wide = std::exp(u(-1, 4)), thin = gen() % 3 ? std::exp(u(-2, 1)) : wide;
    float a00 = std::cos(angle) / wide, a01 = std::sin(angle) / wide, a10 = -std::sin(angle) / thin, a11 = std::cos(angle) / thin;
    if (gen() % 4 == 0) a01 = a10 = 0.0f;
    const float b0 = -(a00 * cx + a01 * cy), b1 = -(a10 * cx + a11 * cy);
    // the box of the rectangle |tc| <= margin, or one drawn at will (a square's)
    const float det = a00 * a11 - a01 * a10;
    float ex = margin * (std::fabs(a11) + std::fabs(a01)) / std::fabs(det), ey = margin * (std::fabs(a10) + std::fabs(a00)) / std::fabs(det);
    if (!RECT) ex = ey = u(0.2, 20);
    int x0 = max(0, (int)std::floor(cx - ex)), x1 = (int)std::ceil(cx + ex), y0 = max(0, (int)std::floor(cy - ey)), y1 = (int)std::ceil(cy + ey);
    if (x1 < 0 || y1 < 0 || x1 > 65000 || y1 > 65000) return 0;
    if (gen() % 16 == 0) x0 = x1 + 1;  // not drawn
    // only records of this tile are listed
    if (x0 > wx0 + 15 || x1 < wx0 || y0 > ty0 + 15 || y1 < ty0) return 0;
    const float4 r0 = make_float4(a00, a01, b0, a10);
    const float4 r1 = make_float4(a11, b1, 0.5f, as_float((uint32_t)x0 | (uint32_t)y0 << 16));
    const float4 r2 = make_float4(0.5f, 0.5f, 0.5f, as_float((uint32_t)x1 | (uint32_t)y1 << 16));
    const uint32_t slot = gen() % RASTER_BATCH;
    for (int sw = 0; sw < 8; ++sw) s_pm[sw][slot] = 0u;
    mask_rows<RECT>(s_pm, slot, r0, r1, r2, wx0, ty0, margin);
    uint32_t word[8], most = 0;
    for (int sw = 0; sw < 8; ++sw) most |= word[sw] = s_pm[sw][slot];
    int covered = 0;
    for (int row = 0; row < 16; ++row)
        for (int col = 0; col < 16; ++col) {
            const int px = wx0 + col, py = ty0 + row;
            const float X = px + 0.5f, Y = py + 0.5f;
            const float tx = std::fmaf(a01, Y, std::fmaf(a00, X, b0)), ty = std::fmaf(a11, Y, std::fmaf(a10, X, b1));
            const bool box = px >= x0 && px <= x1 && py >= y0 && py <= y1;
            const bool drawn = box && (!RECT || (std::fabs(tx) <= margin && std::fabs(ty) <= margin));
            const bool listed = word[row >> 1] >> (16 * (row & 1) + col) & 1u;
            if (drawn && !listed) return std::printf("a covered pixel is not listed\n"), -1;
            if (listed && (!box || (!RECT && !drawn))) return std::printf("a pixel outside is listed\n"), -1;
            // a listed pixel's centre is within the documented widening of the rectangle (where a row bounds columns at all)
            if (RECT && listed) {
                const double big = 1e-6 * ((std::fabs(a00) + std::fabs(a10)) * (wx0 + 16) + (std::fabs(a01) + std::fabs(a11)) * (ty0 + 16) +
                                           std::fabs(b0) + std::fabs(b1) + margin);
                if ((std::fabs(a00) > 1e-30f && std::fabs(tx) > margin + 4 * big + 2e-3 * std::fabs(a00)) ||
                    (std::fabs(a10) > 1e-30f && std::fabs(ty) > margin + 4 * big + 2e-3 * std::fabs(a10)))
                    return std::printf("a pixel far outside is listed\n"), -1;
            }
            covered += drawn;
        }
    return covered;
}

int main() {
    std::mt19937 gen(1);
    long covered = 0;
    for (int i = 0; i < 400000; ++i) {
        const int n = i & 1 ? check<true>(gen) : check<false>(gen);
        if (n < 0) return std::printf("case %d\n", i), 1;
        covered += n;
    }
    std::printf("%ld pixels\n", covered);
    return covered > 1000000 ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    text = open(os.path.join(ROOT, "splatter_gb300", "csrc", "spl_raster.cuh")).read()
    columns = re.search(r"^__device__ [^\n]*\brow_columns\(.*?^}\n", text, re.M | re.S).group(0)
    rows = re.search(r"^template <bool RECT>\n__device__ [^\n]*\bmask_rows\(.*?^}\n", text, re.M | re.S).group(0)
    path = tmp_path_factory.mktemp("masks")
    (path / "masks.cpp").write_text(HOST + columns + rows + MAIN)
    compiler = shutil.which("g++")
    if compiler is None:
        pytest.skip("no g++")
    run = subprocess.run([compiler, "-std=c++17", "-O3", "-ffp-contract=off", "-frounding-math", "-Wstrict-aliasing=2", "-Werror",
                          str(path / "masks.cpp"), "-o", str(path / "masks")], capture_output=True, text=True)
    return path / "masks", run


def test_words_are_written_by_their_own_type(program):
    assert program[1].returncode == 0, program[1].stderr


def test_masks_hold_the_covered_pixels(program):
    run = subprocess.run([str(program[0])], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
