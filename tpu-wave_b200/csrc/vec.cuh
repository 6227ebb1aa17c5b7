// Vectors of 16 bytes (4 FP32 or 2 FP64 values) for the stencil kernels that give a thread adjacent
// columns. FP32 sums and products go two at a time (packed f32x2 instructions: each half is rounded on
// its own, as the scalar instruction).
#pragma once
#include "device_math.cuh"

namespace tw {

namespace {

using u64 = unsigned long long;
using tw::add;   // (the scalar overloads beside the vector ones below)
using tw::mul;

// ---- vectors of 16 bytes
template <class C> struct Vec;
template <> struct Vec<float> {
    static constexpr int N = 4;
    using W = u64;   // a weight, in both halves
    u64 a, b;
};
template <> struct Vec<double> {
    static constexpr int N = 2;
    using W = double;
    double a, b;
};
using VF = Vec<float>;
using VD = Vec<double>;

__device__ __forceinline__ u64 pk(float x, float y)
{
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void unpk(u64 v, float &x, float &y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ u64 mul2(u64 x, u64 y)
{
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return r;
}
__device__ __forceinline__ u64 fma2(u64 x, u64 y, u64 z)
{
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
    return r;
}
__device__ __forceinline__ u64 wt(float s) { return pk(s, s); }
__device__ __forceinline__ double wt(double s) { return s; }
__device__ __forceinline__ VF mul(VF x, VF y) { return {mul2(x.a, y.a), mul2(x.b, y.b)}; }
__device__ __forceinline__ VF mulw(VF x, u64 s) { return {mul2(x.a, s), mul2(x.b, s)}; }
__device__ __forceinline__ VD mul(VD x, VD y) { return {mul(x.a, y.a), mul(x.b, y.b)}; }
__device__ __forceinline__ VD mulw(VD x, double s) { return {mul(x.a, s), mul(x.b, s)}; }
__device__ __forceinline__ VF vzero(float) { return {0ull, 0ull}; }
__device__ __forceinline__ VD vzero(double) { return {0., 0.}; }
__device__ __forceinline__ VF vld(const float *p)
{
    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
    return {v.x, v.y};
}
__device__ __forceinline__ VD vld(const double *p)
{
    const double2 v = *reinterpret_cast<const double2 *>(p);
    return {v.x, v.y};
}
__device__ __forceinline__ VF vldg(const float *p)
{
    const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(p));
    return {v.x, v.y};
}
__device__ __forceinline__ VD vldg(const double *p)
{
    const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
    return {v.x, v.y};
}
__device__ __forceinline__ void vst(float *p, VF v) { *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(v.a, v.b); }
__device__ __forceinline__ void vst(double *p, VD v) { *reinterpret_cast<double2 *>(p) = make_double2(v.a, v.b); }
__device__ __forceinline__ void vget(VF v, float (&e)[4])
{
    unpk(v.a, e[0], e[1]);
    unpk(v.b, e[2], e[3]);
}
__device__ __forceinline__ void vget(VD v, double (&e)[2])
{
    e[0] = v.a;
    e[1] = v.b;
}
__device__ __forceinline__ VF vset(const float (&e)[4]) { return {pk(e[0], e[1]), pk(e[2], e[3])}; }
__device__ __forceinline__ VD vset(const double (&e)[2]) { return {e[0], e[1]}; }

// the stencil weights and the vector sums. A packed FP32 sum is fma(x, 1, y) with a 1 the compiler
// cannot see through (and a difference fma(y, -1, x)): a mul.rn.f32x2 whose result feeds an
// add.rn.f32x2 came out contracted into one rounding, and these cannot be.
template <class C> struct St;
template <>
struct St<float> {
    u64 w[4], one, mone;
    __device__ __forceinline__ St(const float (&st)[4], bool truth)
    {
#pragma unroll
        for (int k = 0; k < 4; k++) w[k] = wt(st[k]);
        one = wt(truth ? 1.f : 2.f);
        mone = wt(truth ? -1.f : 2.f);
    }
    __device__ __forceinline__ VF add(VF x, VF y) const { return {fma2(x.a, one, y.a), fma2(x.b, one, y.b)}; }
    __device__ __forceinline__ VF sub(VF x, VF y) const { return {fma2(y.a, mone, x.a), fma2(y.b, mone, x.b)}; }
};
template <>
struct St<double> {
    double w[4];
    __device__ __forceinline__ St(const double (&st)[4], bool)
    {
#pragma unroll
        for (int k = 0; k < 4; k++) w[k] = st[k];
    }
    __device__ __forceinline__ VD add(VD x, VD y) const { return {tw::add(x.a, y.a), tw::add(x.b, y.b)}; }
    __device__ __forceinline__ VD sub(VD x, VD y) const { return {tw::sub(x.a, y.a), tw::sub(x.b, y.b)}; }
};

// sum of four taps, each a vector (the leading 0 + is left out: see tma_step.cuh)
template <class C>
__device__ __forceinline__ Vec<C> taps(const St<C> &s, Vec<C> t0, Vec<C> t1, Vec<C> t2, Vec<C> t3)
{
    Vec<C> v = mulw(t0, s.w[0]);
    v = s.add(v, mulw(t1, s.w[1]));
    v = s.add(v, mulw(t2, s.w[2]));
    return s.add(v, mulw(t3, s.w[3]));
}

// y derivative of N-type points from the M-type row p (taps c-2 .. c+1); mid: the vector at c
__device__ __forceinline__ VF dyN(const St<float> &s, const float *p, VF mid)
{
    const u64 l = *reinterpret_cast<const u64 *>(p - 2);
    float l0, l1, m0, m1, m2, m3;
    unpk(l, l0, l1);
    unpk(mid.a, m0, m1);
    unpk(mid.b, m2, m3);
    const u64 o0 = pk(l1, m0), o1 = pk(m1, m2), o2 = pk(m3, p[4]);
    return taps<float>(s, {l, mid.a}, {o0, o1}, mid, {o1, o2});
}
__device__ __forceinline__ VD dyN(const St<double> &s, const double *p, VD mid)
{
    const VD l = vld(p - 2);
    const double r = p[2];
    return taps<double>(s, l, {l.b, mid.a}, mid, {mid.b, r});
}
// y derivative of M-type points from the N-type row p (taps c-1 .. c+2)
// (alt: the column after the vector is *z)
__device__ __forceinline__ VF dyM(const St<float> &s, const float *p, VF mid, bool alt, const float *z)
{
    const u64 r = *reinterpret_cast<const u64 *>(p + 4);
    float m0, m1, m2, m3, r0, r1;
    unpk(mid.a, m0, m1);
    unpk(mid.b, m2, m3);
    unpk(r, r0, r1);
    if (alt) r0 = *z;
    const u64 o0 = pk(p[-1], m0), o1 = pk(m1, m2), o2 = pk(m3, r0);
    return taps<float>(s, {o0, o1}, mid, {o1, o2}, {mid.b, pk(r0, r1)});
}
__device__ __forceinline__ VD dyM(const St<double> &s, const double *p, VD mid, bool alt, const double *z)
{
    VD r = vld(p + 2);
    if (alt) r.a = *z;
    const double l = p[-1];
    return taps<double>(s, {l, mid.a}, mid, {mid.b, r.a}, r);
}

}  // namespace

}  // namespace tw
