/*
 * b2g_trig.h — sine and cosine of an f32 angle, identical on host and device.
 *
 * The reference builds every rotation with `f32::sin` / `f32::cos`
 * (B2Rot::set, src/b2_math.rs:363-376), which on Linux is the platform libm's
 * sinf/cosf. CUDA's sinf/cosf give different last bits, so this project uses
 * one function of its own on both sides, evaluated in IEEE double and rounded
 * once to f32 (so it is correctly rounded except in astronomically rare ties):
 *
 *   1. Cody–Waite reduction: k = nearest integer to x·2/π, r = x − k·π/2 with
 *      π/2 split into three doubles; the first two carry 33 significant bits so
 *      k·P1 and k·P2 are exact for |k| < 2^20 (|x| < ~1.6e6 rad).
 *   2. Taylor series of sin and cos about 0 on |r| ≤ π/4, through r^19 and
 *      r^18, evaluated by Horner's rule (truncation error < 1e-21).
 *   3. Quadrant selection by k mod 4, then one rounding to f32.
 *
 * Every operation is a separately rounded IEEE double operation. Host code must
 * be compiled with -ffp-contract=off and device code with --fmad=false so that
 * no multiply-add is fused; then host and device results are bit-identical.
 *
 * b2g_sincosf returns exactly the same bits, faster: GB300's FP64 rate is a small fraction of
 * its FP32 rate, so for |x| <= 8192 the value is first computed in floats (hi + lo pairs only where
 * the low part matters, explicit fused multiply-adds for the exact products):
 *   1. the same reduction r = x - k*pi/2 with pi/2 in three floats: x - k*P1 is exact (a multiple of
 *      2^-24 below 1), k*P2 an exact product pair, k*P3 a float;
 *   2. r = j/512 + d with |d| <= 1/1024 and a table of sin(j/512), cos(j/512) as float pairs;
 *   3. sin d = d + d^3 (-1/6 + d^2/120) and cos d - 1 = -d^2/2 + d^4/24: with so small a d a float of
 *      each correction is within 2^-45, so only sin(j/512) + cos(j/512) d and cos(j/512) - sin(j/512) d
 *      are kept as pairs.
 * The result is returned only when adding the error bound to the low part and subtracting it round
 * to the same float (2^-42 relative, above the error of either computation; with k != 0 also 2^-60,
 * the reduction's): then the true value and the double evaluation round to that float too. Otherwise
 * (about one call in 2^17), and for |x| > 8192, inf and NaN, the double routine runs.
 * The solver's position sweeps are chains of these calls (two bodies, two points), so their length is what
 * counts: about 40 dependent operations and 220 cycles a call, 374 for two side by side (double-precision
 * evaluation, which static bodies' zero angles once took, made a colour of the 210-box pyramid's position
 * sweeps 4.0 us; it takes 1.3). tests/trig_check.cpp compares the two routines on floats of the fast range,
 * tests/trig_check_gpu.cu on every one; tests/test_trig_table.py makes the table's rows again. */
#ifndef B2G_TRIG_H
#define B2G_TRIG_H

#include <math.h>
#include <string.h>

#if defined(__CUDACC__)
#define B2G_HD __host__ __device__ __forceinline__
#else
#define B2G_HD inline
#endif

/* π/2 = B2G_PIO2_1 + B2G_PIO2_2 + B2G_PIO2_3 (first two terms: 33 significant bits). */
#define B2G_PIO2_1 0x1.921fb54400000p+0
#define B2G_PIO2_2 0x1.0b4611a600000p-34
#define B2G_PIO2_3 0x1.3198a2e037073p-69
#define B2G_2_OVER_PI 0x1.45f306dc9c883p-1

/* 1/n! rounded to double */
#define B2G_INV_F2 0x1.0000000000000p-1
#define B2G_INV_F3 0x1.5555555555555p-3
#define B2G_INV_F4 0x1.5555555555555p-5
#define B2G_INV_F5 0x1.1111111111111p-7
#define B2G_INV_F6 0x1.6c16c16c16c17p-10
#define B2G_INV_F7 0x1.a01a01a01a01ap-13
#define B2G_INV_F8 0x1.a01a01a01a01ap-16
#define B2G_INV_F9 0x1.71de3a556c734p-19
#define B2G_INV_F10 0x1.27e4fb7789f5cp-22
#define B2G_INV_F11 0x1.ae64567f544e4p-26
#define B2G_INV_F12 0x1.1eed8eff8d898p-29
#define B2G_INV_F13 0x1.6124613a86d09p-33
#define B2G_INV_F14 0x1.93974a8c07c9dp-37
#define B2G_INV_F15 0x1.ae7f3e733b81fp-41
#define B2G_INV_F16 0x1.ae7f3e733b81fp-45
#define B2G_INV_F17 0x1.952c77030ad4ap-49
#define B2G_INV_F18 0x1.6827863b97d97p-53
#define B2G_INV_F19 0x1.2f49b46814157p-57

/* sin(x), cos(x) for f32 x evaluated in double (the definition of the results). NaN/inf inputs
 * give NaN. */
B2G_HD void b2g_sincosf_ref(float x, float* out_s, float* out_c)
{
    const double xd = (double)x;
    if (!(xd - xd == 0.0)) { /* inf or nan */
        const double nan = xd - xd;
        *out_s = (float)nan;
        *out_c = (float)nan;
        return;
    }
    /* nearest integer by the 1.5·2^52 shift (|t| < 2^51 always holds for f32 input / (π/2)) */
    const double shifter = 0x1.8p52;
    const double t = xd * B2G_2_OVER_PI;
    const double kd = (t + shifter) - shifter;
    double r = xd - kd * B2G_PIO2_1;
    r = r - kd * B2G_PIO2_2;
    r = r - kd * B2G_PIO2_3;
    const double z = r * r;
    /* sin r = r + r*z*(-1/3! + z*(1/5! - z*(...))) */
    double ps = -B2G_INV_F19;
    ps = ps * z + B2G_INV_F17;
    ps = ps * z - B2G_INV_F15;
    ps = ps * z + B2G_INV_F13;
    ps = ps * z - B2G_INV_F11;
    ps = ps * z + B2G_INV_F9;
    ps = ps * z - B2G_INV_F7;
    ps = ps * z + B2G_INV_F5;
    ps = ps * z - B2G_INV_F3;
    const double sr = r + (r * z) * ps;
    /* cos r = 1 - z/2 + z*z*(1/4! - z/6! + ... - z^7/18!) */
    double pc = -B2G_INV_F18;
    pc = pc * z + B2G_INV_F16;
    pc = pc * z - B2G_INV_F14;
    pc = pc * z + B2G_INV_F12;
    pc = pc * z - B2G_INV_F10;
    pc = pc * z + B2G_INV_F8;
    pc = pc * z - B2G_INV_F6;
    pc = pc * z + B2G_INV_F4;
    const double cr = (1.0 - z * B2G_INV_F2) + (z * z) * pc;
    /* quadrant: k mod 4 (two's complement of a small integer) */
    const long long k = (long long)kd;
    const int q = (int)(k & 3);
    double s, c;
    if (q == 0) { s = sr; c = cr; }
    else if (q == 1) { s = cr; c = -sr; }
    else if (q == 2) { s = -sr; c = -cr; }
    else { s = -cr; c = sr; }
    *out_s = (float)s;
    *out_c = (float)c;
}

/* ---- the float fast path (see the file comment) ---- */
/* sin(j/512) hi, lo, cos(j/512) hi, lo for j = 0..402 */
constexpr int b2g_sc_rows = 403;
#if defined(__CUDACC__)
__device__ static const float4 b2g_sc_table_dev[b2g_sc_rows] = {
#include "b2g_trig_table.h"
};
#endif
static const float b2g_sc_table_host[b2g_sc_rows * 4] = {
#include "b2g_trig_table.h"
};

B2G_HD float b2g_fmaf_(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    return __fmaf_rn(a, b, c);
#else
    return fmaf(a, b, c);
#endif
}

/* The double routine as the fast path calls it: on the device a function of its own, so that its 150
 * instructions are not in the loops that call b2g_sincosf (the kernel of a small world waited more than
 * half of its cycles an instruction for instruction fetches). */
#if defined(__CUDACC__)
static __device__ __noinline__ float2 b2g_sincosf_slow_dev(float x) {
    float2 r;
    b2g_sincosf_ref(x, &r.x, &r.y);
    return r;
}
#endif
B2G_HD void b2g_sincosf_slow_(float x, float* out_s, float* out_c) {
#if defined(__CUDA_ARCH__)
    const float2 r = b2g_sincosf_slow_dev(x);
    *out_s = r.x;
    *out_c = r.y;
#else
    b2g_sincosf_ref(x, out_s, out_c);
#endif
}

B2G_HD int b2g_f2i_(float v) {
#if defined(__CUDA_ARCH__)
    return __float_as_int(v);
#else
    int i;
    memcpy(&i, &v, 4);
    return i;
#endif
}
B2G_HD float b2g_flip_(float v, int sign_bit) {  /* v with its sign flipped where sign_bit's bit 31 is set */
#if defined(__CUDA_ARCH__)
    return __int_as_float(__float_as_int(v) ^ (sign_bit & (int)0x80000000));
#else
    return sign_bit < 0 ? -v : v;
#endif
}

/* The fast path for any x: whether its results are certain. Without a branch, so that two calls (a
 * constraint's two bodies) run side by side; nearest integers by the 1.5 * 2^23 shift, whose bits are the
 * integer too. */
B2G_HD bool b2g_sincosf_try_(float x, float* out_s, float* out_c)
{
    const float shifter = 0x1.8p23f;
    /* x - k*pi/2 = t + e */
    const float km = b2g_fmaf_(x, 0x1.45f306p-1f, shifter);
    const float kf = km - shifter;
    const float a = b2g_fmaf_(-kf, 0x1.921fb6p+0f, x);
    const float p = kf * -0x1.777a5cp-25f;
    const float pe = b2g_fmaf_(kf, -0x1.777a5cp-25f, -p);
    const float t = a - p;                       /* and the rest exactly (two-sum) */
    const float bb = t - a;
    const float e = b2g_fmaf_(kf, 0x1.ee59dap-50f, ((a - (t - bb)) - (p + bb)) - pe);
    /* t + e = j/512 + (d + e) */
    const float jm = b2g_fmaf_(t, 512.0f, shifter);
    const float jf = jm - shifter;
    const float d = b2g_fmaf_(jf, -0x1.0p-9f, t);  /* exact */
    const int j = b2g_f2i_(jm) - 0x4b400000;
    const unsigned aj = (unsigned)(j < 0 ? -j : j);
    const unsigned at = aj < (unsigned)b2g_sc_rows ? aj : 0u;  /* always so for |x| <= 8192 */
#if defined(__CUDA_ARCH__)
    const float4 row = b2g_sc_table_dev[at];
    const float sth = b2g_flip_(row.x, j), stl = b2g_flip_(row.y, j), cth = row.z, ctl = row.w;
#else
    const float sth = b2g_flip_(b2g_sc_table_host[4 * at], j), stl = b2g_flip_(b2g_sc_table_host[4 * at + 1], j);
    const float cth = b2g_sc_table_host[4 * at + 2], ctl = b2g_sc_table_host[4 * at + 3];
#endif
    const float d2 = d * d;
    /* sin(d + e) = d + sd, cos(d + e) - 1 = m */
    const float sd = b2g_fmaf_(d * d2, b2g_fmaf_(d2, 0x1.111112p-7f, -0x1.555556p-3f), e);
    const float m = b2g_fmaf_(d2 * d2, 0x1.555556p-5f, b2g_fmaf_(-d, e, -0.5f * d2));
    /* sin r = st + ct*sin(d + e) + st*m, cos r = ct - st*sin(d + e) + ct*m */
    const float bh = cth * d, bl = b2g_fmaf_(cth, d, -bh);
    const float sh = sth + bh;                   /* |sth| >= |bh|, or sth = 0 */
    const float sl = (bh - (sh - sth)) + (((stl + bl) + b2g_fmaf_(cth, sd, ctl * d)) + sth * m);
    const float gh = sth * d, gl = b2g_fmaf_(sth, d, -gh);
    const float ch = cth - gh;
    const float cl = ((cth - ch) - gh) + (((ctl - gl) - b2g_fmaf_(sth, sd, stl * d)) + cth * m);
    /* the rounding test */
    const float abs_err = kf != 0.0f ? 0x1.0p-60f : 0.0f;
    const float se = b2g_fmaf_(0x1.0p-42f, sh < 0.0f ? -sh : sh, abs_err);
    const float ce = b2g_fmaf_(0x1.0p-42f, ch, abs_err);
    const float s1 = sh + (sl + se), s2 = sh + (sl - se);
    const float c1 = ch + (cl + ce), c2 = ch + (cl - ce);
    /* quadrant k mod 4 */
    const int q = b2g_f2i_(km);
    *out_s = b2g_flip_((q & 1) ? c1 : s1, q << 30);
    *out_c = b2g_flip_((q & 1) ? s1 : c1, (q + 1) << 30);
    const float ax = x < 0.0f ? -x : x;
    return s1 == s2 && c1 == c2 && ax <= 8192.0f;
}

/* sin(x), cos(x) for f32 x: the same results as b2g_sincosf_ref. */
B2G_HD void b2g_sincosf(float x, float* out_s, float* out_c)
{
    if (!b2g_sincosf_try_(x, out_s, out_c)) b2g_sincosf_slow_(x, out_s, out_c);
}

/* the same of two angles */
B2G_HD void b2g_sincosf2(float x, float y, float* xs, float* xc, float* ys, float* yc)
{
    const bool okx = b2g_sincosf_try_(x, xs, xc), oky = b2g_sincosf_try_(y, ys, yc);
    if (!(okx && oky)) {
        if (!okx) b2g_sincosf_slow_(x, xs, xc);
        if (!oky) b2g_sincosf_slow_(y, ys, yc);
    }
}

#endif /* B2G_TRIG_H */
