// Exact float arithmetic of the reference's projection step without the FP64 pipe (host and
// device).  The reference computes p_t = (-div / acc) * OVER_RELAXATION with a float quotient and
// a double constant (project/smokeSimulation.cu:38, :384): q = x / d in float, d = 1..6, then
// float(double(q) * omega): the product rounded to 53 bits and then to 24.  An FP64 product with
// its two conversions costs three passes through GB300's FP64 pipe (a few lanes per clock and SM),
// and the IEEE quotient about ten instructions; here a cell takes five FP32 multiplies and FMAs.
//
//   Quotient: q = fma(x, zh, x * zl) with zh = 1/d rounded toward zero and zl = 1/d - zh rounded
//   (division by a known constant as an unevaluated sum, after Brisebarre, Muller and Raina,
//   "Accelerating correctly rounded floating-point division when the divisor is known in
//   advance", IEEE Trans. Computers 53(8), 2004).  Before the last rounding the error is below
//   2^-46 |x/d|, while x/d for d = 3, 5, 6 is never a midpoint of two floats and keeps a distance
//   of at least 2^-28 |x/d| from every midpoint (d odd: d * midpoint needs 26 bits); d = 1, 2, 4
//   are exact.  So q is the IEEE quotient while x * zl does not underflow.
//
//   Product: with omega = wh + wl, wh rounded toward zero to float (|wl| below its last place) and
//   wl = wl1 + wl2 as two floats,
//     c = fma(q, wl1, q * wl2)   q * wl rounded to float, off by 2^-24 |c| at most,
//     p = fma(q, wh, c)          q * wh + c rounded once.
//   Let omega be the double nearest to n / D, D <= 1000 (every constant of up to three decimals; 1.9 =
//   19 / 10).  q n / D keeps a distance of at least 1 / (2 D) of a place from every midpoint of
//   two floats that it does not equal, far more than the error of c, so p and float(double(q) *
//   omega) are the same neighbour there.  Midpoints it does equal are common (for 1.9 one q in
//   ten): q n / D - q wh is then a multiple of the last place of q * wh and smaller than 2^24 of
//   them, so c is exactly that number, the FMA meets the exact midpoint and rounds to even, as the
//   conversion does provided that the double product is the midpoint itself.  It is when omega's
//   own error is below half a last place of every product: |omega - n / D| < m 2^(e - 54), omega
//   = m 2^e with m in [1, 2) (omega_split checks this).
//   An omega without such n / D has midpoints only by chance: there p is taken where the results
//   with c enlarged and diminished by 2^-21 c agree (Ziv's rounding test; they disagree about
//   once in 2^20 cells), else the FP64 product.
//
// A cell whose |x| is below 2^-96 but not zero (underflow would void the argument; in a fresh
// simulation the passes spread such values, subnormal ones among them, ahead of the first smoke)
// takes the same steps on x * 2^64 and scales the result back, exact where it is normal (pt_scaled).
// Results below 2^-125 lie on the grid of 2^-149: quotient and product are rounded to whole numbers
// of it, each from an estimate corrected by its exact remainder (pt_grid).  What is left (values that
// are not finite, a failed rounding test) takes FP64: the quotient corrected once by its exact
// remainder and rounded (a float or a midpoint that x / d equals is then exact, the others are far
// away), and the double product itself.  Zeros keep their sign: zl has the sign of zh, wl1 and wl2
// that of wh.
#pragma once
#include <math.h>
#include <stdint.h>

#include "kernels.h"

namespace smk {

constexpr float ES_TINY = 0x1p-96f, ES_HUGE = 0x1p120f;

// zh, zl of the divisor d = 1..6 (host: the table of a kernel is filled from these).
struct DivSplit {
    float zh, zl;
};

__host__ __device__ __forceinline__ DivSplit div_split(int d) {
    // 1/d rounded toward zero to 24 bits, and the rest: 1/3 = 0xAAAAAA * 2^-25 + ..., 1/5 =
    // 0xCCCCCC * 2^-26 + ..., 1/6 = 0xAAAAAA * 2^-26 + ...; the rest of 1/d after n/2^k is
    // (2^k - n d) / (d 2^k), here (2/3) 2^-25, (4/5) 2^-26 and (2/3) 2^-26
    DivSplit s;
    switch (d) {
        case 1: s.zh = 1.0f; s.zl = 0.0f; break;
        case 2: s.zh = 0.5f; s.zl = 0.0f; break;
        case 3: s.zh = 11184810.0f * 0x1p-25f; s.zl = (2.0f / 3.0f) * 0x1p-25f; break;
        case 4: s.zh = 0.25f; s.zl = 0.0f; break;
        case 5: s.zh = 13421772.0f * 0x1p-26f; s.zl = (4.0f / 5.0f) * 0x1p-26f; break;
        default: s.zh = 11184810.0f * 0x1p-26f; s.zl = (2.0f / 3.0f) * 0x1p-26f; break;
    }
    return s;
}

// Whether x / d and its product need the FP64 path (a value that is not finite does too).
__host__ __device__ __forceinline__ bool es_rare(float x) {
    const float a = fabsf(x);
    return !(a >= ES_TINY && a <= ES_HUGE) && a != 0.0f;
}

__host__ __device__ __forceinline__ float div_fast(float x, float zh, float zl) { return fmaf(x, zh, x * zl); }

__host__ __device__ __forceinline__ float scale_rest(float q, const OmegaSplit& s) { return fmaf(q, s.wl1, q * s.wl2); }
// Ziv's test of the product for an omega that is no n / D.
__host__ __device__ __forceinline__ bool scale_sure(float q, float c, const OmegaSplit& s) {
    return fmaf(q, s.wh, c * (1.0f + 0x1p-21f)) == fmaf(q, s.wh, c * (1.0f - 0x1p-21f));
}

// x / d rounded to float, through FP64, for any x; d = 1..6 and r = RN(1/d) in double.
__host__ __device__ __forceinline__ float div_exact(float x, double d, double r) {
    const double X = (double)x;
    double y = X * r;
    if (fabsf(x) <= 3.4028234663852886e38f) y = fma(fma(-y, d, X), r, y);
    return x == 0.0f ? x : (float)y;
}

// p_t for 0 < |x| < 2^-96 where the result is normal and safely so; ok says whether it is.
__host__ __device__ __forceinline__ float pt_scaled(float x, float zh, float zl, const OmegaSplit& s, bool& ok) {
    const float q = div_fast(x * 0x1p64f, zh, zl);
    const float c = scale_rest(q, s);
    const float p = fmaf(q, s.wh, c);
    ok = fabsf(p) >= 0x1p-61f && fabsf(q) >= 0x1p-61f && (s.rational || scale_sure(q, c, s));
    return p * 0x1p-64f;
}

// p_t for 0 < |x| < 2^-118 where quotient and product are below 2^-125 (whole numbers of 2^-149, at most 2^24),
// omega n / D; d = 1..6.  ok says whether the operands are such.
__host__ __device__ __forceinline__ float pt_grid(float x, int d, float zh, float zl, const OmegaSplit& s, bool& ok) {
    const float m = fabsf(x) * 0x1p64f * 0x1p85f;  // |x| = m 2^-149, a whole number
    ok = s.rational != 0 && m < 0x1p31f;
    const float mf = ok ? m : 0.0f;
    // k = m / d to the nearest whole number, ties to even: the estimate is within 1 of it
    int k = (int)rintf(div_fast(mf, zh, zl));
    const int rem = 2 * ((int)mf - k * d);
    if (rem > d || (rem == d && (k & 1))) k += 1;
    else if (rem < -d || (rem == -d && (k & 1))) k -= 1;
    // j = k |omega| to the nearest whole number; in the tie case the remainder is exactly 1/2
    const float kf = (float)k;
    const float c = scale_rest(kf, s);
    const float t = fmaf(kf, s.wh, c);
    const float e = rintf(t);
    int j = (int)e;
    if (fabsf(t) < 0x1p23f) {
        const float r = fmaf(kf, s.wh, -e) + c;
        if (r > 0.5f || (r == 0.5f && (j & 1))) j += 1;
        else if (r < -0.5f || (r == -0.5f && (j & 1))) j -= 1;
    }
    ok = ok && k <= (1 << 24) && j <= (1 << 24) && j >= -(1 << 24);
    const float p = (float)(j < 0 ? -j : j) * 0x1p-85f * 0x1p-64f;  // exact
    return (x < 0.0f) != (s.wh < 0.0f) ? -p : p;
}

__host__ __device__ __forceinline__ float scale_exact(float q, double omega) { return (float)((double)q * omega); }

#ifdef __CUDACC__
// A cell that the common path does not decide (es_rare, or the rounding test): zh, zl as in its table
// entry, pt the common path's value, kept where `rare` is not set; ofs holds the cell's six neighbour bits
// (8..13) and its projectable bit (14).  pt_scaled, pt_grid, then FP64
// (exact_scale.cuh; zh + zl stands for 1/acc, whose 2^-48 the correction by the exact remainder makes up
// for).  The FP64 part is one block of PTX: as plain code the compiler evaluates it for every lane
// and selects, which puts the FP64 instructions on every cell.
constexpr unsigned ES_ENTRY_PROJ = 1u << 14;
static __device__ __noinline__ float cell_pt_rare(float pt, bool rare, float x, unsigned ofs, float zh, float zl,
                                             const OmegaSplit& os, double omega) {
    rare = rare && (ofs & ES_ENTRY_PROJ);
    const int acc = max(__popc((ofs >> 8) & 63u), 1);
    bool ok;
    const bool tiny = rare && fabsf(x) < ES_TINY;
    const float ps = pt_scaled(x, zh, zl, os, ok);
    if (tiny && ok) pt = ps;
    rare = rare && !(tiny && ok);
    if (!__any_sync(0xffffffffu, rare)) return pt;
    const float pg = pt_grid(x, acc, zh, zl, os, ok);
    if (rare && ok) pt = pg;
    const bool left = rare && !ok;
    if (!__any_sync(0xffffffffu, left)) return pt;
    asm volatile(
        "{\n\t"
        ".reg .pred mine, fin;\n\t"
        ".reg .f32 ax, r;\n\t"
        ".reg .f64 X, d, i, y, c, e;\n\t"
        "setp.ne.u32 mine, %1, 0;\n\t"
        "cvt.rn.f64.u32 d, %3;\n\t"
        "cvt.f64.f32 i, %5;\n\t"
        "cvt.f64.f32 e, %6;\n\t"
        "add.rn.f64 i, i, e;\n\t"
        "cvt.f64.f32 X, %2;\n\t"
        "mul.rn.f64 y, X, i;\n\t"
        "neg.f64 c, y;\n\t"
        "fma.rn.f64 e, c, d, X;\n\t"
        "fma.rn.f64 c, e, i, y;\n\t"
        "abs.f32 ax, %2;\n\t"
        "setp.lt.f32 fin, ax, 0f7f800000;\n\t"
        "selp.f64 y, c, y, fin;\n\t"
        "cvt.rn.f32.f64 r, y;\n\t"
        "cvt.f64.f32 y, r;\n\t"
        "mul.rn.f64 y, y, %4;\n\t"
        "cvt.rn.f32.f64 r, y;\n\t"
        "selp.f32 %0, r, %0, mine;\n\t"
        "}"
        : "+f"(pt)
        : "r"((unsigned)left), "f"(x), "r"(acc), "d"(omega), "f"(zh), "f"(zl));
    return pt;
}
#endif

}  // namespace smk
