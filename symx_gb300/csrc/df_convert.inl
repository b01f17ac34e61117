R"(
// Conversions between double and double-float with integer instructions.  On GB300 an FP64 instruction
// holds a quarter SM's FP64 pipe for 64 clocks per warp, and each conversion needs three (two changes of
// type and a subtraction or an addition): 24 inputs and 13 outputs per tetrahedron took 0.33 ms of the
// pipe for 1.6 M of them.  Same results as the FP64 formulas, or `bad` is set (values near the ends of
// float's exponents): the caller then converts all its values again with the formulas, so the
// instruction stream holds them once.
//
// hi = (float)x, lo = (float)(x - hi)
__device__ __forceinline__ symxg_df symxg_split(double x, bool& bad)
{
    const unsigned u1 = (unsigned)__double2hiint(x), u0 = (unsigned)__double2loint(x);
    const unsigned e = (u1 >> 20) & 0x7ffu, sign = u1 & 0x80000000u;
    const bool zero = ((u1 << 1) | u0) == 0u;
    bad = bad || (e - 949u > 200u && !zero);  // x outside [2^-74, 2^127)
    const unsigned rem = u0 & 0x1fffffffu;    // the 29 bits below float's last one
    const unsigned kept = __funnelshift_r(u0, u1 & 0x7fffffffu, 29) - (896u << 23);
    const unsigned up = rem > 0x10000000u - (kept & 1u) ? 1u : 0u;  // to nearest, ties to even
    const int r = (int)rem - (int)(up << 29);                       // |x| - |hi| in units of 2^(E - 52)
    const float unit = __uint_as_float((e - 948u) << 23);
    const float lo = __int2float_rn(sign ? -r : r) * unit;
    return symxg_df(__uint_as_float(zero ? sign : (kept + up) | sign), zero ? 0.0f : lo);
}
// hi + lo
__device__ __forceinline__ double symxg_join(const symxg_df& a, bool& bad)
{
    const unsigned h = __float_as_uint(a.hi), l = __float_as_uint(a.lo), e = (h >> 23) & 0xffu, sign = h & 0x80000000u;
    const bool zero = ((h | l) << 1) == 0u;
    const float units = a.lo * __uint_as_float((306u - e) << 23);  // lo in units of 2^(E - 52)
    // hi outside [2^-74, 2^127), or lo above half a unit of hi's last place, or hi + lo possibly below
    // hi's power of two
    bad = bad || (!zero && (e - 53u > 200u || !(fabsf(units) <= 268435456.0f) || (h & 0x7fffffu) == 0u));
    const int r = __float2int_rn(sign ? -units : units);
    const unsigned top = ((h & 0x7fffffffu) >> 3) + (896u << 20), low = h << 29;
    const unsigned long long d = (((unsigned long long)top << 32) | low) + (unsigned long long)(long long)r;
    return __longlong_as_double(zero ? (long long)((unsigned long long)(sign & l) << 32)
                                     : (long long)(d | ((unsigned long long)sign << 32)));
}
)"
