// One-direction forward-mode dual number for the adjoint kernels.
//
// The face physics of afx_device.cuh is templated on its arithmetic type, so
// instantiating it with Dual gives the exact directional derivative next to
// the value, one pass per input direction.  The adjoint kernels use it for the
// ghost states of boundary faces (the flux of a face is reversed by hand).
//
// Branches (entropy fix, limiter cases, characteristic boundary cases, min /
// max) follow the value, so the derivative is the one of the active branch.
#pragma once

#include <cuda_runtime.h>

#include "afx_fp64.cuh"

namespace afx {
namespace dev {

struct Dual {
    double v, d;
    __device__ __forceinline__ Dual() : v(0), d(0) {}
    __device__ __forceinline__ Dual(double x) : v(x), d(0) {}
    __device__ __forceinline__ Dual(double x, double dx) : v(x), d(dx) {}
};

__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return Dual(a.v + b.v, a.d + b.d); }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return Dual(a.v - b.v, a.d - b.d); }
__device__ __forceinline__ Dual operator-(Dual a) { return Dual(-a.v, -a.d); }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) { return Dual(a.v * b.v, a.d * b.v + a.v * b.d); }
__device__ __forceinline__ Dual operator/(Dual a, Dual b) {
    const fp64::Den y = fp64::den(b.v);
    const double r = fp64::quot(a.v, y);
    return Dual(r, fp64::quot(a.d - r * b.d, y));
}
__device__ __forceinline__ Dual& operator+=(Dual& a, Dual b) { return a = a + b; }
__device__ __forceinline__ Dual& operator-=(Dual& a, Dual b) { return a = a - b; }
__device__ __forceinline__ Dual& operator*=(Dual& a, Dual b) { return a = a * b; }
__device__ __forceinline__ bool operator<(Dual a, Dual b) { return a.v < b.v; }
__device__ __forceinline__ bool operator>(Dual a, Dual b) { return a.v > b.v; }
__device__ __forceinline__ bool operator<=(Dual a, Dual b) { return a.v <= b.v; }
__device__ __forceinline__ bool operator>=(Dual a, Dual b) { return a.v >= b.v; }

__device__ __forceinline__ Dual dsqrt(Dual x) {
    const double s = fp64::root(x.v);
    return Dual(s, fp64::quot(x.d, fp64::twice(fp64::den(s))));
}
__device__ __forceinline__ Dual dabs(Dual x) { return x.v < 0 ? -x : x; }

}  // namespace dev
}  // namespace afx
