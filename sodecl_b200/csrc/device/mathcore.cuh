// Elementary functions as straight-line code in FP64, each on the arguments its
// comment names.  Shared, as text, by the NVRTC programs (embedded by the
// build; fastmath.cuh and threefry.cuh build on it) and the statically compiled
// test kernels in aux_kernels.cu.  Self-contained: no includes.
//
// Methods: argument reduction in the manner of Cody and Waite ("Software
// Manual for the Elementary Functions", 1980) with fused multiply-adds, and
// minimax polynomials (Remez exchange) evaluated by Horner's rule.
//  sin: x = n pi + r, |r| <= pi/2, sin x = (-1)^n sin r, sin r = r + r^3 P(r^2)
//       with P of degree 7 (relative error 2^-61.6).  Reducing by pi and not
//       by pi/2 needs two more coefficients and no choice between a sine and
//       a cosine polynomial.  pi is held in two doubles: its tail
//       contributes n 2^-108.
//  cos: x = (k + 1/2) pi + r, cos x = (-1)^(k+1) sin r.
//  exp: x = n ln 2 + r, |r| <= ln 2 / 2, a polynomial of degree 11 whose first
//       coefficients are 1, 1, 1/2 and the rounded 1/6 (relative error
//       2^-57.2), times 2^n, added to the exponent.
//  log: x = m 2^k, m in [sqrt(1/2), sqrt(2)), f = m - 1, s = f / (2 + f), and
//       log m = f - f^2/2 + s (f^2/2 + R(s^2)), the arrangement of fdlibm's
//       log (Sun Microsystems, 1993), R of degree 7 in s^2 (error 2^-59.5).
//  sqrt: the hardware's approximate reciprocal root, one cubic step for it and
//       the root together, and the residual's correction.
// Against quadruple precision: sin and cos within 1.7 ulp (mean 0.33; the
// library's within 1.44, mean 0.30), exp within 0.90 ulp (mean 0.26; the
// library's 0.83, 0.26), log within 0.80 ulp, sqrt correctly rounded on 1.5e6
// arguments.
//
// What bounds them is the FP64 pipe (14 instructions a sine, two cycles each
// per warp and scheduler).  Independent sums of sines, every SM full: 8.9e11
// sines/s against the library's 4.9e11, latency 114 cycles against 241.  The
// coefficients sit in constant memory, which an FP64 instruction reads as an
// operand; as literals, built in registers, those sums run at 6.6e11.
#ifndef SODECL_MATHCORE_CUH
#define SODECL_MATHCORE_CUH

__constant__ double sodecl_sin_poly[8] = {-0x1.5555555555555p-3,  0x1.11111111110c1p-7,  -0x1.a01a01a014878p-13,
                                          0x1.71de3a5285e6ap-19,  -0x1.ae6454ca7583fp-26, 0x1.6123caeee6360p-33,
                                          -0x1.ae430e21eac89p-41, 0x1.8827f95e04f40p-49};
// 1/pi, 1.5 x 2^52 (adding it leaves the nearest integer in the low bits), -pi in two parts
__constant__ double sodecl_sin_red[4] = {0x1.45f306dc9c883p-2, 0x1.8p52, -0x1.921fb54442d18p+1, -0x1.1a62633145c07p-53};
__constant__ double sodecl_exp_poly[10] = {0.5,                   0x1.5555555555555p-3,  0x1.55555555536aep-5,
                                           0x1.11111111195ddp-7,  0x1.6c16c17b75711p-10, 0x1.a01a015a31628p-13,
                                           0x1.a019aee45f929p-16, 0x1.71dee995f714fp-19, 0x1.289c23e2e03a1p-22,
                                           0x1.ada6dcf53a45fp-26};
// 1/ln 2, 1.5 x 2^52, -ln 2 in two parts
__constant__ double sodecl_exp_red[4] = {0x1.71547652b82fep+0, 0x1.8p52, -0x1.62e42fefa39efp-1, -0x1.abc9e3b39803fp-56};

// sin r for |r| <= pi/2 (and a little beyond), which has r's sign, a zero's
// too; the sign bit of `flip` turns it
__device__ __forceinline__ double sodecl_sin_poly_signed(double r, int flip)
{
    const double u = __dmul_rn(r, r);
    double p = sodecl_sin_poly[7];
#pragma unroll
    for (int k = 6; k >= 0; --k) p = __fma_rn(p, u, sodecl_sin_poly[k]);
    const double s = __fma_rn(__dmul_rn(r, u), p, r);
    return __hiloint2double((__double2hiint(s) & 0x7fffffff) | ((__double2hiint(r) ^ flip) & (int)0x80000000),
                            __double2loint(s));
}

// |x| <= 2^30
__device__ __forceinline__ double sodecl_sin_core(double x)
{
    const double t = __fma_rn(x, sodecl_sin_red[0], sodecl_sin_red[1]);
    const double n = __dsub_rn(t, sodecl_sin_red[1]);
    double r = __fma_rn(n, sodecl_sin_red[2], x);
    r = __fma_rn(n, sodecl_sin_red[3], r);
    return sodecl_sin_poly_signed(r, __double2loint(t) << 31);
}

__device__ __forceinline__ double sodecl_cos_core(double x)
{
    const double t = __fma_rd(x, sodecl_sin_red[0], sodecl_sin_red[1]);  // floor(x / pi)
    const double h = __dadd_rn(__dsub_rn(t, sodecl_sin_red[1]), 0.5);
    double r = __fma_rn(h, sodecl_sin_red[2], x);
    r = __fma_rn(h, sodecl_sin_red[3], r);
    return sodecl_sin_poly_signed(r, ~__double2loint(t) << 31);
}

// |x| < 708.  Fine: the reduction's and the last product's rounding errors are
// kept and added (within 0.75 ulp, mean 0.255), for six more instructions.
template <bool Fine>
__device__ __forceinline__ double sodecl_exp_core_of(double x)
{
    const double t = __fma_rn(x, sodecl_exp_red[0], sodecl_exp_red[1]);
    const double n = __dsub_rn(t, sodecl_exp_red[1]);
    const double r1 = __fma_rn(n, sodecl_exp_red[2], x);  // exact
    const double r = __fma_rn(n, sodecl_exp_red[3], r1);
    double p = sodecl_exp_poly[9];
#pragma unroll
    for (int k = 8; k >= 0; --k) p = __fma_rn(p, r, sodecl_exp_poly[k]);
    p = __fma_rn(p, r, 1.0);
    double s = __fma_rn(p, r, 1.0);
    if (Fine) {
        const double low = __fma_rn(n, sodecl_exp_red[3], __dsub_rn(r1, r));
        s = __dadd_rn(s, __dadd_rn(__fma_rn(p, r, __dsub_rn(1.0, s)), low));
    }
    return __hiloint2double(__double2hiint(s) + (__double2loint(t) << 20), __double2loint(s));
}
__device__ __forceinline__ double sodecl_exp_core(double x) { return sodecl_exp_core_of<false>(x); }
__device__ __forceinline__ double sodecl_exp_fine_core(double x) { return sodecl_exp_core_of<true>(x); }

__constant__ double sodecl_log_poly[7] = {0x1.5555555555593p-1, 0x1.999999997fb31p-2, 0x1.2492494217a15p-2,
                                          0x1.c71c51e7f758cp-3, 0x1.7466462c93937p-3, 0x1.39a0f50122a2dp-3,
                                          0x1.2f0d8ea92ff11p-3};
// ln 2 in two parts
__constant__ double sodecl_log_red[2] = {0x1.62e42fefa39efp-1, 0x1.abc9e3b39803fp-56};

// 0 < x < infinity, x normal
__device__ __forceinline__ double sodecl_log_core(double x)
{
    const int hi = __double2hiint(x);
    const int k = (hi - 0x3fe6a09e) >> 20;  // 0x3fe6a09e: the high word of sqrt(1/2)
    const double f = __dsub_rn(__hiloint2double(hi - (k << 20), __double2loint(x)), 1.0);
    const double d = __dadd_rn(f, 2.0);
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = __fma_rn(-d, r, 1.0);
    r = __fma_rn(r, __fma_rn(e, e, e), r);
    const double s = __dmul_rn(f, r), z = __dmul_rn(s, s);
    double p = sodecl_log_poly[6];
#pragma unroll
    for (int q = 5; q >= 0; --q) p = __fma_rn(p, z, sodecl_log_poly[q]);
    const double h = __dmul_rn(__dmul_rn(0.5, f), f), kd = (double)k;
    const double t = __fma_rn(s, __fma_rn(p, z, h), __dmul_rn(kd, sodecl_log_red[1]));
    return __fma_rn(kd, sodecl_log_red[0], __dsub_rn(f, __dsub_rn(h, t)));
}

// 2^-1000 < x < 2^1000
__device__ __forceinline__ double sodecl_sqrt_core(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = __dmul_rn(x, y), h = __dmul_rn(0.5, y);
    const double r = __fma_rn(-g, h, 0.5);
    const double c = __fma_rn(__dmul_rn(r, 1.5), r, r);
    g = __fma_rn(g, c, g);
    h = __fma_rn(h, c, h);
    return __fma_rn(__fma_rn(-g, g, x), h, g);
}

#endif
