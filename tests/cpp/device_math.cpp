// The elementary functions and quotients of csrc/device compiled for the host,
// on arrays: the device's rounding intrinsics are the host's (IEEE 754 FMA, one
// rounding each).  The hardware's approximations of 1/x and 1/sqrt(x) come from
// the caller's side as values within 2^-20 (a rounded reciprocal with its low
// bits changed).
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __forceinline__ inline
#define __constant__ static const
#define SODECL_APPROXIMATIONS

static long long __double_as_longlong(double x) { long long b; std::memcpy(&b, &x, 8); return b; }
static double __longlong_as_double(long long b) { double x; std::memcpy(&x, &b, 8); return x; }
static int __float_as_int(float x) { int b; std::memcpy(&b, &x, 4); return b; }
static unsigned max(unsigned a, unsigned b) { return a > b ? a : b; }
static float __int_as_float(int b) { float x; std::memcpy(&x, &b, 4); return x; }
static int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
static int __double2loint(double x) { return (int)(__double_as_longlong(x) & 0xffffffffLL); }
static double __hiloint2double(int hi, int lo)
{
    return __longlong_as_double((long long)(((unsigned long long)(unsigned)hi << 32) | (unsigned)lo));
}
static double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static double __dmul_rn(double a, double b) { volatile double r = a * b; return r; }
static double __dadd_rn(double a, double b) { volatile double r = a + b; return r; }
static double __dsub_rn(double a, double b) { volatile double r = a - b; return r; }
static float __fmul_rn(float a, float b) { volatile float r = a * b; return r; }
// relative errors of up to 2^-20, of either sign, by the argument's bits
static double off(double r, double x)
{
    const long long b = __double_as_longlong(x);
    const double k = (double)((b * 0x9E3779B97F4A7C15LL) >> 44) / 524288.0;  // [-1, 1)
    return std::isfinite(r) ? r + r * k * 0x1p-20 : r;
}
static double sodecl_rcp_approx(double x) { return off(1.0 / x, x); }
static double sodecl_rsqrt_approx(double x) { return off(1.0 / std::sqrt(x), x); }

#include "device/fastdiv.cuh"
#include "device/mathcore.cuh"

extern "C" {
#define VALUES(fn)                                                       \
    void fn##_values(const double *x, double *y, long n)                 \
    {                                                                    \
        for (long i = 0; i < n; ++i) y[i] = sodecl_##fn##_core(x[i]);    \
    }
VALUES(sin)
VALUES(cos)
VALUES(exp)
VALUES(log)
VALUES(sqrt)

#define BOUNDED(fn)                                                               \
    void fn##_bounded(const double *x, double *y, unsigned char *outside, long n) \
    {                                                                             \
        for (long i = 0; i < n; ++i) {                                            \
            bool o;                                                               \
            y[i] = sodecl_##fn##_bounded(x[i], o);                                \
            outside[i] = o;                                                       \
        }                                                                         \
    }
BOUNDED(sin)
BOUNDED(cos)
BOUNDED(exp)

void chain_quotients(const double *a, const double *b, double *q, unsigned char *outside, long n)
{
    for (long i = 0; i < n; ++i) {
        bool bad = false;
        q[i] = sodecl_div_chain(a[i], b[i], bad);
        outside[i] = bad;
    }
}
void straight_quotients(const double *a, const double *b, double *q, unsigned char *outside, long n)
{
    for (long i = 0; i < n; ++i) {
        q[i] = sodecl_div_straight(a[i], b[i], 1.0 / b[i]);
        outside[i] = sodecl_straight_divisor_outside(b[i]) || sodecl_straight_dividend_outside(a[i]);
    }
}
void straight_quotients_f32(const float *a, const float *b, float *q, unsigned char *outside, long n)
{
    for (long i = 0; i < n; ++i) {
        q[i] = sodecl_div_straight(a[i], b[i], 1.0f / b[i]);
        outside[i] = sodecl_straight_divisor_outside(b[i]) || sodecl_straight_dividend_outside(a[i]);
    }
}
}
