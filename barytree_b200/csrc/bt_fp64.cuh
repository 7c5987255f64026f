// bt_fp64.cuh -- FP64 building blocks of the evaluation kernels (internal).
//
// The FP64 kernels are bound by the FP64 pipe (64 lanes per clock and SM), so
// what counts is the number of FP64 instructions per kernel value.  CUDA's
// rsqrt, sqrt, exp and division handle every argument (zero, subnormal,
// infinite) inside their sequences.  Here the arguments that occur take short
// sequences of their own, and an argument outside them makes the value
// non-finite (rsqrt_n); the kernels look at each sum once and form it again
// with the library functions where it is not finite.
#pragma once

#include <cfloat>
#include <cmath>
#include <cstdint>

namespace bt {

// 1/sqrt(x) for normal x > 0: the hardware's estimate y0, whose lower 32 bits
// are zero (so its square is exact), and one Householder step of third order,
// y = y0 (1 + e/2 + 3 e^2 / 8) with e = 1 - x y0^2, which leaves (5/16)|e|^3.
// Five FP64 instructions.  x zero, subnormal, infinite or NaN gives an
// infinity or NaN.
__device__ __forceinline__ double rsqrt_n(double x, double &y0)
{
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(x));
    const double e = fma(-x, y0 * y0, 1.0);
    return fma(y0 * e, fma(e, 0.375, 0.5), y0);
}
__device__ __forceinline__ double rsqrt_n(double x)
{
    double y0;
    return rsqrt_n(x, y0);
}

// y = 1/sqrt(x) and r = sqrt(x): r = x y and one correction by the residual
// x - r^2 over 2 r, 1/(2 r) taken from the estimate with its exponent lowered.
__device__ __forceinline__ double rsqrt_sqrt_n(double x, double &r)
{
    double y0;
    const double y = rsqrt_n(x, y0), r0 = x * y;
    r = fma(fma(-r0, r0, x), __hiloint2double(__double2hiint(y0) - (1 << 20), 0), r0);
    return y;
}

// exp(-kappa r) by a table of 2^(j/64) and a polynomial, the table-driven
// method of P. T. P. Tang ("Table-driven implementation of the exponential
// function in IEEE floating-point arithmetic", ACM TOMS 15, 1989):
// -kappa r = (n + f) ln2 / 64 with the integer n = 64 k + j and |f| <= 1/2, so
// exp = 2^k (2^(j/64) + 2^(j/64) p(f)), p the Taylor polynomial of degree 5 of
// 2^(f/64) - 1 (truncated below 4e-17).  Eleven FP64 instructions; the integer
// pipe adds k to the exponent.
constexpr int EXP64_TAB = 64;
__constant__ const double2 exp64_table[EXP64_TAB] = {      // {2^(j/64) rounded, the rest}
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56},
    {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55}, {0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57},
    {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54}, {0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59},
    {0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54}, {0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55}, {0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55},
    {0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54}, {0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54}, {0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55},
    {0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55}, {0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54},
    {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55}, {0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54},
    {0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54}, {0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56},
    {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55}, {0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58},
    {0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59}, {0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56}, {0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54},
    {0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55}, {0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54},
    {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54}, {0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54},
    {0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54}, {0x1.6623882552225p+0, -0x1.bb60987591c34p-54},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54}, {0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57},
    {0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55}, {0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55}, {0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56},
    {0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54}, {0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54},
    {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54}, {0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55},
    {0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57}, {0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54},
    {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56}, {0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54},
    {0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54}, {0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54}, {0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57},
    {0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56}, {0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55},
    {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55}, {0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54},
    {0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56}, {0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54},
    {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55}, {0x1.da9e603db3285p+0, 0x1.c2300696db532p-54},
    {0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54}, {0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54}, {0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54},
    {0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54}, {0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55}
};

struct Exp64 {
    double chi, clo;        // -kappa * 64 / ln2 in two parts
    int rmax;               // upper half of the largest r that the table serves
    int out;                // upper half of exp beyond it: 0, or (kappa < 0) infinity
    const double2 *tab;     // the table in shared memory
};

// |kappa| < 1e300 (a NaN or more than that: the library functions).
__device__ __forceinline__ bool exp64_takes(double kappa) { return fabs(kappa) < 1.0e300; }
__device__ __forceinline__ Exp64 exp64_make(double kappa, const double2 *tab)
{
    constexpr double hi = 92.33248261689366, lo = 1.3027375194195861e-15;     // 64 / ln2
    Exp64 c;
    c.chi = -kappa * hi;
    c.clo = fma(-kappa, hi, -c.chi) - kappa * lo;
    // exp down to 2^-1021.99 and up to 2^1023.99 (an r whose upper half is rmax
    // lies within 2^-20 of it); kappa 0: infinity
    c.rmax = __double2hiint((kappa < 0.0 ? 1023.99 : 1021.99) * 0.6931471805599453 / fabs(kappa));
    c.out = kappa < 0.0 ? 0x7ff00000 : 0;
    c.tab = tab;
    return c;
}

// r >= 0 (a NaN may give any value).  FAR: r may lie beyond rmax, where the
// result is 0, for an exponential below the normal numbers, or infinity for a
// growing one (kappa < 0), whose sum is then formed again with the library
// functions.  Without FAR no r does (exp64_range).  The selection is written
// out: from a condition the compiler makes a branch around the polynomial, and
// values no longer overlap (300,000 Yukawa particles 36 ms a call, 28.3 ms with
// FAR so, 26.9 ms without FAR; 27.6 ms with r and the exponent cut off, which
// left 2^-1022 where the sum is zero).
template <bool FAR>
__device__ __forceinline__ double exp64(double r, const Exp64 &c)
{
    constexpr double magic = 6755399441055744.0;            // 1.5 * 2^52
    constexpr double c1 = 0.010830424696249145, c2 = 5.86490495505617e-05, c3 = 2.1173137155464776e-07,
                     c4 = 5.732851688640402e-10, c5 = 1.2417843701716925e-12;   // (ln2 / 64)^i / i!
    const double m = fma(r, c.chi, magic), n = m - magic;
    const double f = fma(r, c.clo, fma(r, c.chi, -n));
    const double p = f * fma(f, fma(f, fma(f, fma(f, c5, c4), c3), c2), c1);
    const int lo = __double2loint(m);
    const double2 T = c.tab[lo & (EXP64_TAB - 1)];
    const double v = T.x + fma(T.x, p, T.y);
    int hi = __double2hiint(v) + ((lo & -EXP64_TAB) << 14), low = __double2loint(v);
    if (FAR)
        asm("{\n\t.reg .pred p;\n\t"
            "setp.gt.s32 p, %2, %3;\n\t"
            "selp.b32 %0, %4, %0, p;\n\t"
            "selp.b32 %1, 0, %1, p;\n\t}"
            : "+r"(hi), "+r"(low)
            : "r"(__double2hiint(r)), "r"(c.rmax), "r"(c.out));
    return __hiloint2double(hi, low);
}

}  // namespace bt
