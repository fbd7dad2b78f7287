// sin, cos, exp and the quotient for the system files of the explicit and
// stochastic solvers, sin and cos for those of the implicit solvers, the
// quotient for those of the adaptive solver, without branches.
//
// The math library's functions end in a branch to a slow path for rare
// arguments, and so does the reciprocal quotient, so the compiler cannot
// overlap two of them: a Kuramoto row is a chain of 240-cycle sines, one after
// the other.  The functions here are straight-line code on the range they
// cover, and the system file is compiled twice:
//  - the speculative copy (namespace sodecl_spec) calls sodecl_spec_sin and
//    so on, which compute the covered range's result and raise the thread's
//    flag for an argument outside it (a predicated store, no branch).  What the
//    copy computes after that is thrown away, but it runs: so only files whose
//    loops and addresses do not hang on numbers get one (speculable.hpp);
//  - the plain copy calls sodecl_plain_sin and so on, which test the range, and
//    outside it take the library's function and raise the flag too.
// A step whose speculative copy raised the flag counts as the plain copy takes
// it, from the same state (solvers.cuh).  Covered arguments give the same function
// values in both copies, but the compiler may contract the products around them
// differently; since the step's own state decides which copy counts, results do
// not depend on where a run, a launch or a record interval began.  After a plain
// step the next one is tried with the plain copy first; it counts if it raises
// the flag too, else the speculative copy decides again.  So an orbit that stays
// outside pays for the plain copy alone (in FP32 with IEEE division for both: float's
// own quotients raise no flag).
// Programs without speculative steps (the one-thread implicit kernel) call
// sodecl_full_sin and so on, the plain copy's values without the flag.
#ifndef SODECL_FASTMATH_CUH
#define SODECL_FASTMATH_CUH

// One flag per thread of the block, cleared at the kernel's start.  It is
// reached only through these, whose order the compiler keeps among themselves
// and which leave every other value free to move.  (Keeping the largest
// argument in a register instead, free of any order, let the compiler
// interleave more than the registers hold: oculomotor RK4, 2^18 orbits x 1000
// steps, 6.8 against 5.8 ms.)
__shared__ unsigned sodecl_flags[SODECL_BLOCK_MAX];
__device__ __forceinline__ unsigned sodecl_flag_address()
{
    return (unsigned)__cvta_generic_to_shared(sodecl_flags + threadIdx.x);
}
__device__ __forceinline__ void sodecl_raise(bool outside)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.u32 [%1], %0;\n\t}"
                 ::"r"((unsigned)outside), "r"(sodecl_flag_address()));
}
// sodecl_straight_dividend_outside and the raise
__device__ __forceinline__ void sodecl_raise_dividend(double a)
{
    const unsigned hi = (unsigned)__double2hiint(a);
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\tsetp.ge.and.u32 p, %1, 0xe1000000, p;\n\t"
                 "@p st.shared.u32 [%2], %0;\n\t}"
                 ::"r"(hi | (unsigned)__double2loint(a)), "r"((hi << 1) - (123u << 21)), "r"(sodecl_flag_address()));
}
__device__ __forceinline__ void sodecl_raise_dividend(float a)
{
    const unsigned bits = (unsigned)__float_as_int(a);
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\tsetp.ge.and.u32 p, %1, 0xcc000000, p;\n\t"
                 "@p st.shared.u32 [%2], %0;\n\t}"
                 ::"r"(bits), "r"((bits << 1) - (25u << 24)), "r"(sodecl_flag_address()));
}
__device__ __forceinline__ bool sodecl_raised()
{
    unsigned flag;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(flag) : "r"(sodecl_flag_address()));
    return flag != 0u;
}
__device__ __forceinline__ void sodecl_lower()
{
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(sodecl_flag_address()), "r"(0u));
}

// Outside the covered range the speculative copy gets a value that the function
// can have (sodecl_*_bounded), not the polynomial's: the rest of the step runs on
// it.
#define SODECL_MATH_FN(fn, library)                                                                             \
    __device__ __forceinline__ double sodecl_spec_##fn(double x)                                                \
    {                                                                                                           \
        bool outside;                                                                                           \
        const double v = sodecl_##fn##_bounded(x, outside);                                                     \
        sodecl_raise(outside);                                                                                  \
        return v;                                                                                               \
    }                                                                                                           \
    __device__ __forceinline__ double sodecl_plain_##fn(double x)                                               \
    {                                                                                                           \
        bool outside;                                                                                           \
        const double v = sodecl_##fn##_bounded(x, outside);                                                     \
        if (outside) sodecl_raise(true);                                                                        \
        return outside ? library(x) : v;                                                                        \
    }                                                                                                           \
    __device__ __forceinline__ double sodecl_full_##fn(double x)                                                \
    {                                                                                                           \
        bool outside;                                                                                           \
        const double v = sodecl_##fn##_bounded(x, outside);                                                     \
        return outside ? library(x) : v;                                                                        \
    }                                                                                                           \
    SODECL_MATH_OTHER(sodecl_spec_##fn, library)                                                                \
    SODECL_MATH_OTHER(sodecl_plain_##fn, library)                                                               \
    SODECL_MATH_OTHER(sodecl_full_##fn, library)
// the other argument types as the library's own overloads take them: float
// stays float, integers go through double
#if SODECL_FAST_DIV
#define SODECL_MATH_NUM(name) \
    __device__ __forceinline__ sodecl_num name(sodecl_num x) { return sodecl_num(name(x.v)); }
#else
#define SODECL_MATH_NUM(name)
#endif
#define SODECL_MATH_AS_DOUBLE(name, type) \
    __device__ __forceinline__ double name(type x) { return name((double)x); }
#define SODECL_MATH_OTHER(name, library)                                                       \
    __device__ __forceinline__ float name(float x) { return library(x); }                      \
    SODECL_MATH_AS_DOUBLE(name, int)                                                           \
    SODECL_MATH_AS_DOUBLE(name, unsigned)                                                      \
    SODECL_MATH_AS_DOUBLE(name, long)                                                          \
    SODECL_MATH_AS_DOUBLE(name, unsigned long)                                                 \
    SODECL_MATH_AS_DOUBLE(name, long long)                                                     \
    SODECL_MATH_AS_DOUBLE(name, unsigned long long)                                            \
    SODECL_MATH_NUM(name)
// sincos in both its forms (OpenCL's and CUDA's): the values of sin and cos, from
// one reduction and with one test
template <bool Raise, bool Library> __device__ __forceinline__ double sodecl_sincos_of(double x, double *c)
{
    bool outside;
    double cosine;
    const double sine = sodecl_sincos_bounded(x, cosine, outside);
    if (Raise) sodecl_raise(outside);
    const bool library = Library && outside;
    *c = library ? ::cos(x) : cosine;
    return library ? ::sin(x) : sine;
}
template <bool Raise, bool Library> __device__ __forceinline__ float sodecl_sincos_of(float x, float *c)
{
    *c = ::cos(x);
    return ::sin(x);
}
#if SODECL_FAST_DIV
template <bool Raise, bool Library> __device__ __forceinline__ sodecl_num sodecl_sincos_of(sodecl_num x, sodecl_num *c)
{
    return sodecl_num(sodecl_sincos_of<Raise, Library>(x.v, &c->v));
}
#endif
#define SODECL_MATH_SINCOS(name, raise, library)                                               \
    template <class X, class R> __device__ __forceinline__ R name(X x, R *c)                   \
    {                                                                                          \
        return sodecl_sincos_of<raise, library>((R)x, c);                                      \
    }                                                                                          \
    template <class X, class R> __device__ __forceinline__ void name(X x, R *s, R *c)          \
    {                                                                                          \
        *s = sodecl_sincos_of<raise, library>((R)x, c);                                        \
    }

SODECL_MATH_FN(sin, ::sin)
SODECL_MATH_FN(cos, ::cos)
SODECL_MATH_FN(exp, ::exp)
SODECL_MATH_SINCOS(sodecl_spec_sincos, true, false)
SODECL_MATH_SINCOS(sodecl_plain_sincos, true, true)
SODECL_MATH_SINCOS(sodecl_full_sincos, false, true)

#if SODECL_FAST_DIV
// The IEEE quotient's bits.  The divisor's test is a branch of its own: it keeps
// the reciprocal out of the step loop, where the compiler otherwise computes it
// again next to its uses (oculomotor RK4, 2^18 orbits x 1000 steps: 5.8 against
// 8.9 ms).
template <class R> __device__ __forceinline__ R sodecl_div_spec(R a, R b)
{
    const R r = (R)1 / b;
    if (sodecl_straight_divisor_outside(b)) sodecl_raise(true);
    sodecl_raise_dividend(a);
    return sodecl_div_straight(a, b, r);
}
template <class R> __device__ __forceinline__ R sodecl_div_spec_literal(R a, R b)
{
    const R r = (R)1 / b;
    if (sodecl_straight_divisor_outside(b) || sodecl_straight_dividend_outside(a)) sodecl_raise(true);
    return sodecl_div_straight(a, b, r);
}
template <class R> __device__ __forceinline__ R sodecl_div_plain(R a, R b)
{
    const R r = (R)1 / b;
    if (!sodecl_straight_divisor_outside(b) && !sodecl_straight_dividend_outside(a)) return sodecl_div_straight(a, b, r);
    sodecl_raise(true);
    return a / b;
}
// each copy's `/`, declared where the copy stands
#define SODECL_COPY_QUOTIENT(divide)                                                                         \
    __device__ __forceinline__ sodecl_num operator/(sodecl_num a, sodecl_num b)                              \
    {                                                                                                        \
        return sodecl_num(divide(a.v, b.v));                                                                 \
    }                                                                                                        \
    __device__ __forceinline__ sodecl_num &operator/=(sodecl_num &a, sodecl_num b) { return a = a / b; }
// (a dividend of a scalar type is a literal, whose test the compiler takes)
#define SODECL_SPEC_QUOTIENT                                                                                 \
    SODECL_COPY_QUOTIENT(sodecl_div_spec)                                                                    \
    template <class A> __device__ __forceinline__ sodecl_num operator/(A a, sodecl_num b)                    \
    {                                                                                                        \
        return sodecl_num(sodecl_div_spec_literal((sodecl_num_t)a, b.v));                                    \
    }
#define SODECL_PLAIN_QUOTIENT SODECL_COPY_QUOTIENT(sodecl_div_plain)
#else
#define SODECL_SPEC_QUOTIENT
#define SODECL_PLAIN_QUOTIENT
#endif

#endif
