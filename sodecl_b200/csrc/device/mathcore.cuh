// Elementary functions as straight-line code in FP64, each on the arguments its
// comment names.  Shared, as text, by the NVRTC programs (embedded by the
// build; fastmath.cuh and threefry.cuh build on it) and the statically compiled
// test kernels in aux_kernels.cu.  Needs fastdiv.cuh before it.
//
// Methods: argument reduction in the manner of Cody and Waite ("Software
// Manual for the Elementary Functions", 1980) with fused multiply-adds, and
// minimax polynomials (Remez exchange) evaluated by Horner's rule.
//  sin, cos: x = n pi/2 + r, |r| <= pi/4, and of sin r = r + r^3 S(r^2) and
//       cos r = 1 + r^2 (-1/2 + r^2 C(r^2)), S and C of degree 5 (relative errors
//       2^-57.6 and 2^-59.6 with rounded coefficients), the one that n's parity
//       names, with n's sign.  Both are evaluated, so that nothing branches and
//       a sine and a cosine of one argument share the work.  pi/2 is held in
//       three doubles, 2^-163 short of it, and |r| is at least 2^-60 for the
//       doubles up to 2^30: r is right to its last bit next to a zero too.
//  exp: x = n ln 2 + r, |r| <= ln 2 / 2, exp r = 1 + r + r^2 P(r) with P of
//       degree 9 (first coefficients 1/2 and the rounded 1/6, relative error
//       2^-57.2), times 2^n, added to the exponent.
//  log: x = m 2^k, m in [sqrt(1/2), sqrt(2)), f = m - 1, s = f / (2 + f), and
//       log m = 2 artanh s = 2 s + s^3 P(s^2), P of degree 7 (relative error
//       2^-61.6), with the rounding errors of s and of 2 s + k ln 2 kept and
//       added.
//  sqrt: the hardware's approximate reciprocal root, one cubic step for it and
//       the root together, and the residual's correction.
// Against quadruple precision: sin and cos within 1.47 ulp (mean 0.296; the
// library's 1.48, 0.297 on the same arguments) up to 2^30 and next to every
// zero, exp within 0.78 ulp (mean 0.255; the library's 0.87, 0.258), log within
// 0.55 ulp (the library's 0.54, both means 0.250), sqrt correctly rounded on 1.5e6 arguments.
//
// What bounds them is the FP64 pipe (20 instructions a sine, two cycles each
// per warp and scheduler).  The coefficients sit in constant memory, which an
// FP64 instruction reads as an operand.  (Reducing by pi takes 14 instructions
// and no choice between two polynomials, but its rounding errors near pi/2 reach
// 1.7 ulp: stochastic Kuramoto of 32 phases, 2^16 orbits x 200 steps, 18.8 ms
// so, 24.9 ms here, 33.2 ms with the library's sine.)
#ifndef SODECL_MATHCORE_CUH
#define SODECL_MATHCORE_CUH

__constant__ double sodecl_sin_poly[6] = {-0x1.5555555555548p-3,  0x1.111111110f703p-7,  -0x1.a01a019bdf0eap-13,
                                          0x1.71de3548ea12ap-19,  -0x1.ae5e3f8b69be0p-26, 0x1.5d8749807c1ebp-33};
__constant__ double sodecl_cos_poly[7] = {-0.5,                   0x1.555555555554bp-5,  -0x1.6c16c16c14f8ap-10,
                                          0x1.a01a019c8390fp-16,  -0x1.27e4f7ea37964p-22, 0x1.1ee9d75291b14p-29,
                                          -0x1.8fa465ee996e4p-37};
// 2/pi, 1.5 x 2^52 (adding it leaves the nearest integer in the low bits), -pi/2 in three parts
__constant__ double sodecl_sin_red[5] = {0x1.45f306dc9c883p-1, 0x1.8p52, -0x1.921fb54442d18p+0, -0x1.1a62633145c07p-54,
                                         0x1.f1976b7ed8fbcp-110};
__constant__ double sodecl_exp_poly[10] = {0.5,                   0x1.5555555555555p-3,  0x1.55555555536aep-5,
                                           0x1.11111111195ddp-7,  0x1.6c16c17b75711p-10, 0x1.a01a015a31628p-13,
                                           0x1.a019aee45f929p-16, 0x1.71dee995f714fp-19, 0x1.289c23e2e03a1p-22,
                                           0x1.ada6dcf53a45fp-26};
// 1/ln 2, 1.5 x 2^52, -ln 2 in two parts
__constant__ double sodecl_exp_red[4] = {0x1.71547652b82fep+0, 0x1.8p52, -0x1.62e42fefa39efp-1, -0x1.abc9e3b39803fp-56};

#ifndef SODECL_APPROXIMATIONS
__device__ __forceinline__ double sodecl_rsqrt_approx(double x)
{
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}
#endif

// x = n pi/2 + r: n's low bits, r's sign bit (and others), sin r and cos r.
// |x| <= 2^30.
struct sodecl_quarter {
    int n, sign;
    double s, c;
};
__device__ __forceinline__ sodecl_quarter sodecl_quarter_of(double x)
{
    sodecl_quarter q;
    const double t = __fma_rn(x, sodecl_sin_red[0], sodecl_sin_red[1]);
    const double n = __dsub_rn(t, sodecl_sin_red[1]);
    q.n = __double2loint(t);
    double r = __fma_rn(n, sodecl_sin_red[2], x);  // exact
    r = __fma_rn(n, sodecl_sin_red[3], r);
    q.sign = __double2hiint(r);  // (the last part, of the other sign, would turn -0 into 0)
    r = __fma_rn(n, sodecl_sin_red[4], r);
    const double u = __dmul_rn(r, r);
    double s = sodecl_sin_poly[5], c = sodecl_cos_poly[6];
#pragma unroll
    for (int k = 4; k >= 0; --k) s = __fma_rn(s, u, sodecl_sin_poly[k]);
#pragma unroll
    for (int k = 5; k >= 0; --k) c = __fma_rn(c, u, sodecl_cos_poly[k]);
    q.s = __fma_rn(__dmul_rn(r, u), s, r);
    q.c = __fma_rn(c, u, 1.0);
    return q;
}

// sin(r + n pi/2).  A sine has r's sign, a zero's too.
__device__ __forceinline__ double sodecl_quarter_sin(const sodecl_quarter &q, int n)
{
    const double v = (n & 1) ? q.c : q.s;
    const int sign = ((n & 1) ? 0 : q.sign) ^ (n << 30);
    return __hiloint2double((__double2hiint(v) & 0x7fffffff) | (sign & (int)0x80000000), __double2loint(v));
}

// |x| <= 2^30
__device__ __forceinline__ double sodecl_sin_core(double x)
{
    const sodecl_quarter q = sodecl_quarter_of(x);
    return sodecl_quarter_sin(q, q.n);
}

__device__ __forceinline__ double sodecl_cos_core(double x)
{
    const sodecl_quarter q = sodecl_quarter_of(x);
    return sodecl_quarter_sin(q, q.n + 1);
}

// |x| < 708.  1 + r is taken in two parts, so that of r's and the sums'
// rounding errors only r's own is left.
__device__ __forceinline__ double sodecl_exp_core(double x)
{
    const double t = __fma_rn(x, sodecl_exp_red[0], sodecl_exp_red[1]);
    const double n = __dsub_rn(t, sodecl_exp_red[1]);
    double r = __fma_rn(n, sodecl_exp_red[2], x);  // exact
    r = __fma_rn(n, sodecl_exp_red[3], r);
    double p = sodecl_exp_poly[9];
#pragma unroll
    for (int k = 8; k >= 0; --k) p = __fma_rn(p, r, sodecl_exp_poly[k]);
    const double h = __dadd_rn(1.0, r), low = __dsub_rn(r, __dsub_rn(h, 1.0));
    const double s = __dadd_rn(h, __fma_rn(__dmul_rn(r, r), p, low));
    return __hiloint2double(__double2hiint(s) + (__double2loint(t) << 20), __double2loint(s));
}

// The same for any argument, each result one that the function can have, and
// whether it is the value (else `outside` is set): code that goes on with it
// until somebody looks must not meet a negative exp or a sine beyond 1.
// For finite |x| >= 2^30 sin and cos are next to 0.  Inf and NaN are inside.
__device__ __forceinline__ bool sodecl_trig_outside(double x)
{
    const unsigned h = (unsigned)__double2hiint(x) << 1;  // 0x83a00000: 2^30, 0xffe00000: infinity
    return h - 0x83a00000u < 0xffe00000u - 0x83a00000u;
}
__device__ __forceinline__ double sodecl_sin_bounded(double x, bool &outside)
{
    const double v = sodecl_sin_core(x);
    outside = sodecl_trig_outside(x);
    return __hiloint2double(outside ? 0 : __double2hiint(v), __double2loint(v));
}
__device__ __forceinline__ double sodecl_cos_bounded(double x, bool &outside)
{
    const double v = sodecl_cos_core(x);
    outside = sodecl_trig_outside(x);
    return __hiloint2double(outside ? 0 : __double2hiint(v), __double2loint(v));
}

__device__ __forceinline__ double sodecl_sincos_bounded(double x, double &cosine, bool &outside)
{
    const sodecl_quarter q = sodecl_quarter_of(x);
    const double s = sodecl_quarter_sin(q, q.n), c = sodecl_quarter_sin(q, q.n + 1);
    outside = sodecl_trig_outside(x);
    cosine = __hiloint2double(outside ? 0 : __double2hiint(c), __double2loint(c));
    return __hiloint2double(outside ? 0 : __double2hiint(s), __double2loint(s));
}

// exp is 0 from -748 down and infinity from 748 up, and outside only between
// them and 708.  The high word as a float is ordered like the number: 4.19140625f
// is that of 708, 4.23046875f that of 748; those of the largest numbers, Inf and
// NaN are Inf or NaN.  As an unsigned number, a NaN's exceeds infinity's.
__device__ __forceinline__ double sodecl_exp_bounded(double x, bool &outside)
{
    const double v = sodecl_exp_core(x);
    const int hi = __double2hiint(x);
    const float m = fabsf(__int_as_float(hi));
    const bool inside = m < 4.19140625f, negative = hi <= (int)0xfff00000;
    outside = m >= 4.19140625f && m < 4.23046875f;
    const int end = negative ? 0 : (int)max((unsigned)hi, 0x7ff00000u);
    return __hiloint2double(inside ? __double2hiint(v) : end, inside ? __double2loint(v) : 0);
}

__constant__ double sodecl_log_poly[8] = {0x1.5555555555555p-1, 0x1.9999999999dfcp-2, 0x1.249249242b70dp-2,
                                          0x1.c71c7258cba33p-3, 0x1.745cde43ad8bap-3, 0x1.3b20a964a1f34p-3,
                                          0x1.0f5cf550b1f53p-3, 0x1.0f61a3beb2042p-3};
// ln 2 in two parts, the first with eleven zeros at its end: its products by k are exact
__constant__ double sodecl_log_red[2] = {0x1.62e42fefa3800p-1, 0x1.ef35793c76730p-45};

// 0 < x < infinity, x normal
__device__ __forceinline__ double sodecl_log_core(double x)
{
    const int hi = __double2hiint(x);
    const int k = (hi - 0x3fe6a09e) >> 20;  // 0x3fe6a09e: the high word of sqrt(1/2)
    const double f = __dsub_rn(__hiloint2double(hi - (k << 20), __double2loint(x)), 1.0);
    const double d = __dadd_rn(f, 2.0), dlow = __dsub_rn(f, __dsub_rn(d, 2.0));
    double r = sodecl_rcp_approx(d);
    const double e = __fma_rn(-d, r, 1.0);
    r = __fma_rn(r, __fma_rn(e, e, e), r);
    const double s = __dmul_rn(f, r), z = __dmul_rn(s, s);
    const double slow = __dmul_rn(__fma_rn(-s, dlow, __fma_rn(-s, d, f)), r);
    double p = sodecl_log_poly[7];
#pragma unroll
    for (int q = 6; q >= 0; --q) p = __fma_rn(p, z, sodecl_log_poly[q]);
    const double kd = (double)k, top = __dmul_rn(kd, sodecl_log_red[0]);
    const double v = __fma_rn(2.0, s, top), vlow = __fma_rn(2.0, s, __dsub_rn(top, v));
    const double rest = __fma_rn(kd, sodecl_log_red[1], __fma_rn(__dmul_rn(s, z), p, __dadd_rn(slow, slow)));
    return __dadd_rn(v, __dadd_rn(vlow, rest));
}

// 2^-1000 < x < 2^1000
__device__ __forceinline__ double sodecl_sqrt_core(double x)
{
    const double y = sodecl_rsqrt_approx(x);
    double g = __dmul_rn(x, y), h = __dmul_rn(0.5, y);
    const double r = __fma_rn(-g, h, 0.5);
    const double c = __fma_rn(__dmul_rn(r, 1.5), r, r);
    g = __fma_rn(g, c, g);
    h = __fma_rn(h, c, h);
    return __fma_rn(__fma_rn(-g, g, x), h, g);
}

#endif
