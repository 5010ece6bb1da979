// x^b for positive x in double precision, for the steps of double layouts,
// whose chain is mostly this power: shorter than pow(), which takes any
// arguments (a step of a two-dimensional layout 746 cycles against 1,250), and
// no less exact (4 million arguments, x in 2^-52 .. 2^40, b in 0.3 .. 1.8,
// against 64-bit mantissas: at most 1.01 units in the last place and 0.3235 on
// average, pow() 1.32 and 0.3299).
//
// The method is the table-driven one (Tang, "Table-driven implementation of
// the logarithm function in IEEE floating-point arithmetic", ACM TOMS 1990; of
// the exponential function, 1989): with x = 2^k m and c the middle of m's
// 64th of [1, 2),
//   log2 x = (k + log2 c) + log2(1 + r),   r = m / c - 1, |r| <= 2^-7,
// its first part exact in a double, its second, with the rest of log2 c, a
// polynomial; b log2 x is kept as a double and a remainder, and
//   2^y = 2^(j / 64) 2^f,   |f| <= 2^-7,
// with a polynomial again.  Table: 1 / c to 12 bits, -log2 of that to a multiple
// of 2^-40 and what is left, 2^(j / 64).  Polynomials: interpolation at the
// Chebyshev nodes of the ranges, errors 2^-72 and 2^-69.
#pragma once

#include <cuda_runtime.h>

namespace umapb {

struct alignas(32) PowRow {
    double inv, log_hi, log_lo, exp2;
};

static __device__ const PowRow POW_TABLE[64] = {
    {0x1.fc00000000000p-1, 0x1.72c7ba2100000p-7, -0x1.19b14945cf6bap-44, 0x1.0000000000000p+0},
    {0x1.f440000000000p-1, 0x1.1263289520000p-5, -0x1.0a32f8393f026p-42, 0x1.02c9a3e778061p+0},
    {0x1.ecc0000000000p-1, 0x1.c4eb3635c0000p-5, 0x1.d40c95ee56b05p-42, 0x1.059b0d3158574p+0},
    {0x1.e580000000000p-1, 0x1.3a0cf56a00000p-4, 0x1.b12a90d3a7915p-42, 0x1.0874518759bc8p+0},
    {0x1.de60000000000p-1, 0x1.916a59b810000p-4, -0x1.772b0660d0bf2p-42, 0x1.0b5586cf9890fp+0},
    {0x1.d780000000000p-1, 0x1.e6f50c2da0000p-4, -0x1.15844900583dep-45, 0x1.0e3ec32d3d1a2p+0},
    {0x1.d0c0000000000p-1, 0x1.1e153cd5e0000p-3, -0x1.a7c65f4564fa8p-43, 0x1.11301d0125b51p+0},
    {0x1.ca40000000000p-1, 0x1.47b2c2f8c8000p-3, 0x1.8aab6501f60a2p-42, 0x1.1429aaea92de0p+0},
    {0x1.c400000000000p-1, 0x1.7046031c78000p-3, 0x1.f84be19cb9578p-43, 0x1.172b83c7d517bp+0},
    {0x1.bde0000000000p-1, 0x1.9895d0a730000p-3, 0x1.7cb29f3c8a9ccp-42, 0x1.1a35beb6fcb75p+0},
    {0x1.b7e0000000000p-1, 0x1.c09d645468000p-3, 0x1.aa9dff836f12cp-42, 0x1.1d4873168b9aap+0},
    {0x1.b200000000000p-1, 0x1.e857d3d360000p-3, 0x1.367bde40c5e6dp-43, 0x1.2063b88628cd6p+0},
    {0x1.ac60000000000p-1, 0x1.0771a97670000p-2, -0x1.c43d175e57184p-42, 0x1.2387a6e756238p+0},
    {0x1.a6e0000000000p-1, 0x1.1a88d1009c000p-2, -0x1.336e8e314a0e5p-42, 0x1.26b4565e27cddp+0},
    {0x1.a160000000000p-1, 0x1.2ddff3bc60000p-2, -0x1.b522a65a84991p-42, 0x1.29e9df51fdee1p+0},
    {0x1.9c20000000000p-1, 0x1.409347a934000p-2, 0x1.c8fb873a17a10p-43, 0x1.2d285a6e4030bp+0},
    {0x1.9700000000000p-1, 0x1.530fd08f28000p-2, 0x1.fa709d0b28090p-42, 0x1.306fe0a31b715p+0},
    {0x1.9200000000000p-1, 0x1.6552b49988000p-2, -0x1.d8894dbdff331p-42, 0x1.33c08b26416ffp+0},
    {0x1.8d40000000000p-1, 0x1.76e2065018000p-2, 0x1.d09b889393f3bp-42, 0x1.371a7373aa9cbp+0},
    {0x1.8860000000000p-1, 0x1.891fe20b00000p-2, -0x1.1e88bf60501c5p-44, 0x1.3a7db34e59ff7p+0},
    {0x1.83c0000000000p-1, 0x1.9aa4354228000p-2, 0x1.9a9378be719c7p-49, 0x1.3dea64c123422p+0},
    {0x1.7f40000000000p-1, 0x1.abe2f8ec98000p-2, -0x1.8e2339bc74cdfp-42, 0x1.4160a21f72e2ap+0},
    {0x1.7ae0000000000p-1, 0x1.bcd915bcb8000p-2, -0x1.04e3c679e594cp-42, 0x1.44e086061892dp+0},
    {0x1.7680000000000p-1, 0x1.ce01a12f5c000p-2, 0x1.8d11f5fdec0d4p-42, 0x1.486a2b5c13cd0p+0},
    {0x1.7240000000000p-1, 0x1.dede169c34000p-2, 0x1.d7722e99804bfp-42, 0x1.4bfdad5362a27p+0},
    {0x1.6e20000000000p-1, 0x1.ef6b3d3444000p-2, 0x1.0b35b2d1614fbp-43, 0x1.4f9b2769d2ca7p+0},
    {0x1.6a20000000000p-1, 0x1.ffa5d49cf0000p-2, -0x1.9fda43c3ce9ffp-42, 0x1.5342b569d4f82p+0},
    {0x1.6620000000000p-1, 0x1.080748d542000p-1, 0x1.6e30ede3382b7p-42, 0x1.56f4736b527dap+0},
    {0x1.6240000000000p-1, 0x1.1010826b18000p-1, 0x1.ea3c98a07d258p-43, 0x1.5ab07dd485429p+0},
    {0x1.5e80000000000p-1, 0x1.17ece95560000p-1, -0x1.46fab3fa1a144p-44, 0x1.5e76f15ad2148p+0},
    {0x1.5ac0000000000p-1, 0x1.1fdef5db3a000p-1, 0x1.442de8501d871p-43, 0x1.6247eb03a5585p+0},
    {0x1.5720000000000p-1, 0x1.27a23a05a8000p-1, 0x1.cb0ea30b214a6p-43, 0x1.6623882552225p+0},
    {0x1.53a0000000000p-1, 0x1.2f34fd35e6000p-1, 0x1.054558f1e92fap-42, 0x1.6a09e667f3bcdp+0},
    {0x1.5020000000000p-1, 0x1.36dbd5d54a000p-1, -0x1.c6d0b3aa66b9dp-53, 0x1.6dfb23c651a2fp+0},
    {0x1.4ca0000000000p-1, 0x1.3e972f86d0000p-1, 0x1.7b3058a0c2f3dp-43, 0x1.71f75e8ec5f74p+0},
    {0x1.4960000000000p-1, 0x1.45d7e475de000p-1, 0x1.5941c80ef3110p-43, 0x1.75feb564267c9p+0},
    {0x1.4600000000000p-1, 0x1.4d7380dcc4000p-1, 0x1.1646b761c48dep-44, 0x1.7a11473eb0187p+0},
    {0x1.42e0000000000p-1, 0x1.5490e8d628000p-1, -0x1.988f42809d533p-42, 0x1.7e2f336cf4e62p+0},
    {0x1.3fc0000000000p-1, 0x1.5bc007cc08000p-1, -0x1.21bbcf5d58e5fp-42, 0x1.82589994cce13p+0},
    {0x1.3ca0000000000p-1, 0x1.630136d308000p-1, 0x1.443405bb4531bp-42, 0x1.868d99b4492edp+0},
    {0x1.39a0000000000p-1, 0x1.6a096fbcd4000p-1, -0x1.fc78559a053eap-43, 0x1.8ace5422aa0dbp+0},
    {0x1.36a0000000000p-1, 0x1.7122f642b4000p-1, -0x1.3fedabcd79823p-42, 0x1.8f1ae99157736p+0},
    {0x1.33a0000000000p-1, 0x1.784e205f4c000p-1, 0x1.3acec97897218p-44, 0x1.93737b0cdc5e5p+0},
    {0x1.30e0000000000p-1, 0x1.7ef026ac0a000p-1, 0x1.739ebcd166082p-44, 0x1.97d829fde4e50p+0},
    {0x1.2e00000000000p-1, 0x1.85efd062c6000p-1, 0x1.5b338360c2ae2p-43, 0x1.9c49182a3f090p+0},
    {0x1.2b40000000000p-1, 0x1.8cb19c5f06000p-1, -0x1.5f5cde492c839p-47, 0x1.a0c667b5de565p+0},
    {0x1.2880000000000p-1, 0x1.938360a10a000p-1, 0x1.601ccfac2b557p-45, 0x1.a5503b23e255dp+0},
    {0x1.25e0000000000p-1, 0x1.9a14f63cdc000p-1, 0x1.73bd46553bb31p-44, 0x1.a9e6b5579fdbfp+0},
    {0x1.2340000000000p-1, 0x1.a0b5a267b2000p-1, 0x1.1ace3c5d64cd7p-42, 0x1.ae89f995ad3adp+0},
    {0x1.20c0000000000p-1, 0x1.a713ca5708000p-1, -0x1.ca2b13a9f15fbp-42, 0x1.b33a2b84f15fbp+0},
    {0x1.1e20000000000p-1, 0x1.add2b70698000p-1, 0x1.3c194e00ad5c5p-43, 0x1.b7f76f2fb5e47p+0},
    {0x1.1bc0000000000p-1, 0x1.b3fae09ea6000p-1, -0x1.d1a78f54076dbp-42, 0x1.bcc1e904bc1d2p+0},
    {0x1.1940000000000p-1, 0x1.ba844ffcd6000p-1, 0x1.0d9aaa3b48fe9p-45, 0x1.c199bdd85529cp+0},
    {0x1.16e0000000000p-1, 0x1.c0c7e94752000p-1, 0x1.165be242d4ed5p-42, 0x1.c67f12e57d14bp+0},
    {0x1.1480000000000p-1, 0x1.c71939b5d8000p-1, 0x1.0ac59a41a5281p-42, 0x1.cb720dcef9069p+0},
    {0x1.1240000000000p-1, 0x1.cd2248a6c8000p-1, -0x1.958a73689846ap-42, 0x1.d072d4a07897cp+0},
    {0x1.0fe0000000000p-1, 0x1.d38efdd9e4000p-1, -0x1.26c7b113d38eep-42, 0x1.d5818dcfba487p+0},
    {0x1.0dc0000000000p-1, 0x1.d95acc02d6000p-1, 0x1.21432f3936ee9p-42, 0x1.da9e603db3285p+0},
    {0x1.0b80000000000p-1, 0x1.df8aae0e46000p-1, 0x1.eacede1650abdp-42, 0x1.dfc97337b9b5fp+0},
    {0x1.0960000000000p-1, 0x1.e56ed99fb4000p-1, 0x1.7a4d97228439dp-42, 0x1.e502ee78b3ff6p+0},
    {0x1.0740000000000p-1, 0x1.eb5f254ba8000p-1, 0x1.7e0c6023e66d4p-42, 0x1.ea4afa2a490dap+0},
    {0x1.0520000000000p-1, 0x1.f15bc36374000p-1, -0x1.a0ebd3444a8a3p-43, 0x1.efa1bee615a27p+0},
    {0x1.0300000000000p-1, 0x1.f764e7742c000p-1, -0x1.7b0c4bb41a6c9p-42, 0x1.f50765b6e4540p+0},
    {0x1.0100000000000p-1, 0x1.fd1ec77250000p-1, 0x1.54e22d4990b6ep-42, 0x1.fa7c1819e90d8p+0}};

__device__ __forceinline__ double pow_pos(double x, double b) {
    const int hi = __double2hiint(x);
    const double2* row = reinterpret_cast<const double2*>(&POW_TABLE[(hi >> 14) & 63]);
    const double2 u = __ldg(row);
    const double lo = __ldg(&row[1].x);
    const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(x));
    const double r = fma(m, u.x, -1.0), r2 = r * r;
    const double s = static_cast<double>((hi >> 20) - 1023) + u.y;
    const double p01 = fma(r, -0x1.71547652b82fep-1, 0x1.71547652b82fep+0), p23 = fma(r, -0x1.71547652b8392p-2, 0x1.ec709dc3a04a2p-2);
    const double p45 = fma(r, -0x1.ec709dac8a6dfp-3, 0x1.2776c50226859p-2), p67 = fma(r, -0x1.715db2333300cp-3, 0x1.a621a52e77f31p-3);
    const double t = fma(r, fma(r2 * r2, fma(r2, p67, p45), fma(r2, p23, p01)), lo);
    const double y = b * s, y_lo = fma(b, t, fma(b, s, -y));
    constexpr double SHIFT = 0x1.8p52;
    const double q = fma(y + y_lo, 64.0, SHIFT);
    const int n = __double2loint(q);
    const double f = fma(q - SHIFT, -1.0 / 64, y) + y_lo, f2 = f * f;
    const double e2 = __ldg(&POW_TABLE[n & 63].exp2);
    const double q01 = fma(f, 0x1.ebfbdff82c58fp-3, 0x1.62e42fefa39efp-1), q23 = fma(f, 0x1.3b2ab6fba483bp-7, 0x1.c6b08d7048ec1p-5);
    const double q45 = fma(f, 0x1.430923996e797p-13, 0x1.5d88167636ffap-10);
    const double w = f * fma(f2, fma(f2, q45, q23), q01);
    const double z = fma(e2, w, e2);
    // outside: x not a normal number (or infinite, or a NaN), or a result near the ends of the range
    if (!(x >= 0x1p-1000 && x <= 0x1p1000 && fabs(y) < 1000.0)) return pow(x, b);
    return __hiloint2double(__double2hiint(z) + (n >> 6 << 20), __double2loint(z));
}

}  // namespace umapb
