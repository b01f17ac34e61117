// Host build of the double <-> double-float conversions of the generated element kernels
// (df_convert.inl, passed as the header df_convert.h without its string delimiters): prints the
// number of values tried, of those converted to other bits than the FP64 formulas, and of those left
// to the formulas.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#define __device__
#define __forceinline__ inline
template <typename A, typename B>
static A bits(B b)
{
    A a;
    std::memcpy(&a, &b, sizeof a);
    return a;
}
static int __double2hiint(double x) { return (int)(bits<uint64_t>(x) >> 32); }
static int __double2loint(double x) { return (int)bits<uint64_t>(x); }
static unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned s) { return (unsigned)((((uint64_t)hi << 32) | lo) >> s); }
static float __uint_as_float(unsigned u) { return bits<float>(u); }
static unsigned __float_as_uint(float f) { return bits<unsigned>(f); }
static float __int2float_rn(int i) { return (float)i; }
static int __float2int_rn(float f) { return (int)std::nearbyint(f); }
static double __longlong_as_double(long long v) { return bits<double>(v); }
struct symxg_df {
    float hi, lo;
    symxg_df(float h, float l) : hi(h), lo(l) {}
    symxg_df(double x) : hi((float)x), lo((float)(x - (double)(float)x)) {}
};
#include "df_convert.h"

static long long n = 0, bad = 0, refused = 0;
static void check(double x)
{
    bool out = false;
    const symxg_df a = symxg_split(x, out), b(x);
    if (!out) bad += bits<unsigned>(a.hi) != bits<unsigned>(b.hi) || bits<unsigned>(a.lo) != bits<unsigned>(b.lo);
    ++n;
    refused += out;
}
static void check(float hi, float lo)
{
    bool out = false;
    const double a = symxg_join(symxg_df(hi, lo), out);
    if (!out) bad += bits<uint64_t>(a) != bits<uint64_t>((double)hi + (double)lo);
    ++n;
    refused += out;
}
int main()
{
    std::mt19937_64 g(1);
    for (int i = 0; i < 2000000; ++i) {
        const uint64_t u = g(), m = u & 0xfffffffffffffull;
        check(bits<double>(u));  // any bits: zeros, infinities, NaN and denormals below
        const double x = bits<double>(((uint64_t)(1023 - 140 + g() % 300) << 52) | m | (u & (1ull << 63)));
        check(x);
        check(bits<double>(bits<uint64_t>(x) & ~0x1fffffffull));                   // floats
        check(bits<double>((bits<uint64_t>(x) & ~0x1fffffffull) | 0x10000000ull));  // ties
        check(bits<double>(bits<uint64_t>(x) | 0xfffff00000000ull | 0xe0000000ull));  // up to the next power of two
        const symxg_df d(x);
        check(d.hi, d.lo);
        check(d.hi, bits<float>((unsigned)g()));
        check(d.hi, std::ldexp((float)(int)g(), std::ilogb(d.hi) - 55 - (int)(g() % 8)));  // at and above half a unit
        check(bits<float>(bits<unsigned>(d.hi) & 0xff800000u), d.lo);                     // powers of two
        check(bits<float>((unsigned)g()), bits<float>((unsigned)g()));
    }
    for (double x : {0.0, -0.0, (double)INFINITY, -(double)INFINITY, (double)NAN, 5e-324, 1e-310, 1e-45, 3.5e38, 1.0, -1.0}) {
        check(x);
        for (float l : {0.f, -0.f, 1e-45f, -1e-30f, (float)INFINITY, (float)NAN}) check((float)x, l);
    }
    for (double x = 1e-22; x < 1e38; x *= 1.37) {  // what the kernels meet is converted
        bool out = false;
        const symxg_df d = symxg_split(x, out);
        symxg_join(d, out);
        bool z = false;
        symxg_join(symxg_split(0.0, z), z);
        bad += out || z;
    }
    std::printf("%lld %lld %lld\n", n, bad, refused);
    return 0;
}
