// Device pieces shared by the PCG kernels: block-row vectors and float-float sums.
#pragma once

namespace symxg {

// PCG vectors hold one block row as four values (x, y, z, 0): a gathered block column is
// one 16-byte load (float) instead of three 4-byte loads spread over 12 bytes.
template <typename T>
struct Row4 {
    T x, y, z, w;
};
__device__ __forceinline__ Row4<float> ld4(const float* __restrict__ p)
{
    const float4 v = *reinterpret_cast<const float4*>(p);
    return Row4<float>{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ Row4<double> ld4(const double* __restrict__ p)
{
    const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
    return Row4<double>{a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ void st4(float* __restrict__ p, const Row4<float>& v)
{
    *reinterpret_cast<float4*>(p) = make_float4(v.x, v.y, v.z, v.w);
}
__device__ __forceinline__ void st4(double* __restrict__ p, const Row4<double>& v)
{
    reinterpret_cast<double2*>(p)[0] = make_double2(v.x, v.y);
    reinterpret_cast<double2*>(p)[1] = make_double2(v.z, v.w);
}

// ---- float-float (double-single) accumulation for the FP32 PCG's dot products.
// Error-free transformations on the FP32 pipe (TwoSum, FMA-based TwoProd); the __f*_rn
// intrinsics keep the compiler from contracting or reordering them.  Relative accuracy is
// about 2^-44, with no FP64 instruction per vector entry (FP64 is 1/64 rate on this part).
struct FF {
    float hi, lo;
};
__device__ __forceinline__ FF ff_add(FF a, FF b)
{
    const float s = __fadd_rn(a.hi, b.hi);
    const float bb = __fsub_rn(s, a.hi);
    float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));
    e = __fadd_rn(e, __fadd_rn(a.lo, b.lo));
    const float h = __fadd_rn(s, e);
    return FF{h, __fsub_rn(e, __fsub_rn(h, s))};
}
__device__ __forceinline__ FF ff_prod(float x, float y)
{
    const float p = __fmul_rn(x, y);
    return FF{p, fmaf(x, y, -p)};
}
__device__ __forceinline__ FF ff_shfl_down(FF a, int o)
{
    return FF{__shfl_down_sync(0xffffffffu, a.hi, o), __shfl_down_sync(0xffffffffu, a.lo, o)};
}
__device__ __forceinline__ FF ff_shfl_xor(FF a, int o)
{
    return FF{__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)};
}

}  // namespace symxg
