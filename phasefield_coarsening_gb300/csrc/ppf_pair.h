// ppf_pair.h -- arithmetic on pairs of cells.
#pragma once

#include <cuda_runtime.h>

#include <cstring>

namespace ppf {

// Two cells of one thread evaluated together.  For float this is the
// packed f32x2 arithmetic of sm_100+ (one instruction per pair); for double
// it is plain scalar code.  Each lane is rounded exactly as the scalar
// operation would be.
template <typename T>
struct V2;

template <>
struct V2<float> {
    float2 v;
    __device__ __forceinline__ V2() {}
    __device__ __forceinline__ V2(float a, float b) : v(make_float2(a, b)) {}
    __device__ __forceinline__ explicit V2(float2 w) : v(w) {}
    __device__ __forceinline__ float x() const { return v.x; }
    __device__ __forceinline__ float y() const { return v.y; }
};
__device__ __forceinline__ V2<float> operator+(V2<float> a, V2<float> b) { return V2<float>(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ V2<float> operator*(V2<float> a, V2<float> b) { return V2<float>(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ V2<float> operator-(V2<float> a, V2<float> b) {
    unsigned long long ra, xa, ya;
    memcpy(&xa, &a.v, 8);
    memcpy(&ya, &b.v, 8);
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(ra) : "l"(xa), "l"(ya));
    float2 r;
    memcpy(&r, &ra, 8);
    return V2<float>(r);
}
__device__ __forceinline__ V2<float> fma2(V2<float> a, V2<float> b, V2<float> c) {
    return V2<float>(__ffma2_rn(a.v, b.v, c.v));
}

template <>
struct V2<double> {
    double a, b;
    __device__ __forceinline__ V2() {}
    __device__ __forceinline__ V2(double p, double q) : a(p), b(q) {}
    __device__ __forceinline__ explicit V2(double2 w) : a(w.x), b(w.y) {}
    __device__ __forceinline__ double x() const { return a; }
    __device__ __forceinline__ double y() const { return b; }
};
__device__ __forceinline__ V2<double> operator+(V2<double> p, V2<double> q) { return V2<double>(p.a + q.a, p.b + q.b); }
__device__ __forceinline__ V2<double> operator*(V2<double> p, V2<double> q) { return V2<double>(p.a * q.a, p.b * q.b); }
__device__ __forceinline__ V2<double> operator-(V2<double> p, V2<double> q) { return V2<double>(p.a - q.a, p.b - q.b); }
__device__ __forceinline__ V2<double> fma2(V2<double> p, V2<double> q, V2<double> r) {
    return V2<double>(fma(p.a, q.a, r.a), fma(p.b, q.b, r.b));
}

template <typename T>
__device__ __forceinline__ V2<T> splat(T a) { return V2<T>(a, a); }

// a pair stored as two adjacent elements (one 2-element shared access)
__device__ __forceinline__ V2<float> ld2(const float *p) { return V2<float>(*reinterpret_cast<const float2 *>(p)); }
__device__ __forceinline__ V2<double> ld2(const double *p) { return V2<double>(*reinterpret_cast<const double2 *>(p)); }
__device__ __forceinline__ void st2(float *p, V2<float> v) { *reinterpret_cast<float2 *>(p) = v.v; }
__device__ __forceinline__ void st2(double *p, V2<double> v) { *reinterpret_cast<double2 *>(p) = make_double2(v.a, v.b); }

// sums of pairs of floats carried with their rounding errors (Knuth's TwoSum)
__device__ __forceinline__ V2<float> two_sum(V2<float> a, V2<float> x, V2<float> &err) {
    const V2<float> s = a + x;
    const V2<float> bp = s - a;
    err = (a - (s - bp)) + (x - bp);
    return s;
}

__device__ __forceinline__ float two_sum1(float a, float x, float &err) {
    const float s = a + x;
    const float bp = s - a;
    err = (a - (s - bp)) + (x - bp);
    return s;
}

template <typename T>
struct Sum;   // a pair of running sums, about 48 bits or better
template <>
struct Sum<float> {
    V2<float> hi = splat(0.f), lo = splat(0.f);
    __device__ __forceinline__ void add(V2<float> x) {
        V2<float> e;
        hi = two_sum(hi, x, e);
        lo = lo + e;
    }
    __device__ __forceinline__ double get() const {
        float e;
        const float h = two_sum1(hi.x(), hi.y(), e);
        return (double)h + (double)(lo.x() + lo.y() + e);
    }
};
template <>
struct Sum<double> {
    V2<double> s = splat(0.0);
    __device__ __forceinline__ void add(V2<double> x) { s = s + x; }
    __device__ __forceinline__ double get() const { return s.x() + s.y(); }
};

template <typename T>
struct Mass : Sum<double> {};   // FP64: the plain sum
template <>
struct Mass<float> {            // FP32: three parts
    V2<float> hi = splat(0.f), mid = splat(0.f), lo = splat(0.f);
    __device__ __forceinline__ void add(V2<float> x) {
        V2<float> e, f;
        hi = two_sum(hi, x, e);
        mid = two_sum(mid, e, f);
        lo = lo + f;
    }
    __device__ __forceinline__ double get() const {
        float e, f, q;
        const float h = two_sum1(hi.x(), hi.y(), e);
        const float m = two_sum1(two_sum1(mid.x(), mid.y(), f), e, q);
        return (double)h + ((double)m + (double)(lo.x() + lo.y() + f + q));
    }
};

struct Mass1 {   // Mass<float> of single floats
    float hi = 0.f, mid = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float x) {
        float e, f;
        hi = two_sum1(hi, x, e);
        mid = two_sum1(mid, e, f);
        lo += f;
    }
    __device__ __forceinline__ double get() const { return (double)hi + ((double)mid + (double)lo); }
};

}  // namespace ppf
