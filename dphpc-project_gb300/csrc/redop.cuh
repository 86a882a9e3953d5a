// The arithmetic reduction operators, applied as inout = f(in, inout)
// (gpu_libs/gpu_mpi/operators.cu:216-218), and their fold over one vector.
// Sums and products of floating-point values use the round-to-nearest
// intrinsics, so that nothing is contracted and a fold in rank order has the
// bits of a host fold.
#pragma once

#include <cuda_runtime.h>

namespace gm {

template <class T> struct OMax { __device__ static T f(T a, T b) { return a > b ? a : b; } };
template <class T> struct OMin { __device__ static T f(T a, T b) { return a > b ? b : a; } };
template <class T> struct OSum { __device__ static T f(T a, T b) { return (T)(a + b); } };
template <class T> struct OProd { __device__ static T f(T a, T b) { return (T)(a * b); } };

template <> struct OSum<float> { __device__ static float f(float a, float b) { return __fadd_rn(a, b); } };
template <> struct OSum<double> { __device__ static double f(double a, double b) { return __dadd_rn(a, b); } };
template <> struct OProd<float> { __device__ static float f(float a, float b) { return __fmul_rn(a, b); } };
template <> struct OProd<double> { __device__ static double f(double a, double b) { return __dmul_rn(a, b); } };

// acc[e] = f(x[e], acc[e]) over the T elements of a vector V.
template <class T, class O, class V>
static __device__ __forceinline__ void combine(V& acc, const V& x) {
    T* a = reinterpret_cast<T*>(&acc);
    const T* xe = reinterpret_cast<const T*>(&x);
#pragma unroll
    for (int e = 0; e < (int)(sizeof(V) / sizeof(T)); e++) a[e] = O::f(xe[e], a[e]);
}

}  // namespace gm
