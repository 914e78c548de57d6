// Device side of the GB300 rans residual path: face physics and the kernels
// of one explicit iteration, templated on the arithmetic type T (double for
// the FP64 path, float for the FP32-mixed path).
//
// Bit parity (FP64): this header is compiled with -fmad=false and every
// expression keeps the operand order and grouping of AeroFLEX's source, so
// each face flux, gradient, limiter and time step equals the reference's
// definition bit for bit.  Per-cell sums visit the cell's faces in the
// reference's edge order (the device layout stores them that way), which
// reproduces the serial edge loops' accumulation order without atomics.
//
// Layout in HBM (N cells, F faces, B boundary faces):
//   cell vectors  q, gx, gy, phi : one 4-vector per cell (32 B FP64 / 16 B FP32)
//   cslot  int4 per cell: its faces (device ids), ascending reference edge id
//   faces  int2 (c0, c1; c1 < 0 marks boundary -(b+1)), and T2 pairs
//          n = (nx, ny), Lg = (length, Green-Gauss weight), d0, d1 = face
//          centre minus cell-0 / cell-1 centroid
#pragma once

#include <cuda_runtime.h>

#include "afx_fp64.cuh"
#include "afx_launch.hpp"

namespace afx {
namespace dev {

struct __align__(32) d4 {
    double x, y, z, w;
};

template <class T> struct V2t;
template <> struct V2t<double> { using type = double2; };
template <> struct V2t<float> { using type = float2; };
template <class T> struct V4t;
template <> struct V4t<double> { using type = d4; };
template <> struct V4t<float> { using type = float4; };
template <class T> using V2 = typename V2t<T>::type;
template <class T> using V4 = typename V4t<T>::type;

// cnbr of an empty slot (a triangle's fourth)
constexpr int NO_NEIGHBOUR = (int)0x80000000;

enum { BT_INTERNAL = 0, BT_FARFIELD = 1, BT_SLIP = 2, BT_WALL = 3, BT_INOUT = 4 };

__device__ __forceinline__ void ld4(const d4* p, double* v) {
    const double2* q = reinterpret_cast<const double2*>(p);
    double2 a = __ldg(q), b = __ldg(q + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void ld4(const float4* p, float* v) {
    float4 a = __ldg(p);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
template <class T>
__device__ __forceinline__ void ld4c(const V4<T>* p, T* v) { ld4(p, v); }
__device__ __forceinline__ d4 ldv4d(const d4* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    double2 a = __ldg(q), b = __ldg(q + 1);
    d4 r;
    r.x = a.x; r.y = a.y; r.z = b.x; r.w = b.y;
    return r;
}
__device__ __forceinline__ float4 ldv4d(const float4* p) { return __ldg(p); }
template <class T>
__device__ __forceinline__ V4<T> ldv4(const V4<T>* p) { return ldv4d(p); }
// load a state stored as S into T registers
__device__ __forceinline__ void ld4s(const d4* p, double* v) { ld4(p, v); }
__device__ __forceinline__ void ld4s(const float4* p, float* v) { ld4(p, v); }
__device__ __forceinline__ void ld4s(const d4* p, float* v) {
    double t[4];
    ld4(p, t);
    for (int k = 0; k < 4; ++k) v[k] = (float)t[k];
}

__device__ __forceinline__ void st4(d4* p, const double* v) {
    double2* q = reinterpret_cast<double2*>(p);
    q[0] = make_double2(v[0], v[1]);
    q[1] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void st4(float4* p, const float* v) { *p = make_float4(v[0], v[1], v[2], v[3]); }
// conversions in integer arithmetic: the instructions hold the FP64 pipe
__device__ __forceinline__ double to_f64(const float x) { return fp64::widen(__float_as_uint(x)); }
__device__ __forceinline__ float to_f32(const double x) {
    uint32_t r;
    if (!fp64::narrow(x, r)) return (float)x;
    return __uint_as_float(r);
}
__device__ __forceinline__ void st4(float4* p, const double* v) {
    *p = make_float4(to_f32(v[0]), to_f32(v[1]), to_f32(v[2]), to_f32(v[3]));
}
// a + b and the error of it, exactly (Knuth's two-sum)
__device__ __forceinline__ float two_sum(const float a, const float b, float& err) {
    const float s = __fadd_rn(a, b), c = __fadd_rn(s, -a);
    err = __fadd_rn(__fadd_rn(a, -__fadd_rn(s, -c)), __fadd_rn(b, -c));
    return s;
}

__device__ __forceinline__ double dsqrt(double x) { return fp64::root(x); }
__device__ __forceinline__ float dsqrt(float x) { return sqrtf(x); }
// quotients: FP64 in integer arithmetic (afx_fp64.cuh), otherwise the type's own;
// Div holds a denominator that several quotients share
template <class T> __device__ __forceinline__ T fdiv(const T a, const T b) { return a / b; }
__device__ __forceinline__ double fdiv(const double a, const double b) { return fp64::div(a, b); }
template <class T> struct Div {
    T y;
    __device__ __forceinline__ explicit Div(const T v) : y(v) {}
    __device__ __forceinline__ T operator()(const T x) const { return x / y; }
};
template <> struct Div<double> {
    fp64::Den d;
    __device__ __forceinline__ explicit Div(const double v) : d(fp64::den(v)) {}
    __device__ __forceinline__ double operator()(const double x) const { return fp64::quot(x, d); }
};
__device__ __forceinline__ double dabs(double x) { return fabs(x); }
__device__ __forceinline__ float dabs(float x) { return fabsf(x); }
// x or -x, without an FP64 instruction and without a branch around the sum it
// goes into (a - b and a + (-b) are the same number; two branches of a sum are
// formed one after the other in a warp whose lanes differ)
__device__ __forceinline__ float flip(const float x, const bool neg) { return neg ? -x : x; }
// a product on the integer lanes, in FP64 (fp64::mul); a unit compiled with
// contraction keeps it on the FP64 pipe, where most products go into a fused
// multiply-add with the sum that follows
#ifdef AFX_CONTRACTED
__device__ __forceinline__ double imul(const double a, const double b) { return a * b; }
#else
__device__ __forceinline__ double imul(const double a, const double b) { return fp64::mul(a, b); }
#endif
template <class T> __device__ __forceinline__ T imul(const T a, const T b) { return a * b; }
__device__ __forceinline__ double flip(const double x, const bool neg) {
    return fp64::of_bits(fp64::bits_of(x) ^ (neg ? 0x8000000000000000ull : 0ull));
}

// std::min / std::max semantics: min(a,b) = (b < a) ? b : a; max(a,b) = (a < b) ? b : a
template <class T> __device__ __forceinline__ T smin(T a, T b) { return (b < a) ? b : a; }
template <class T> __device__ __forceinline__ T smax(T a, T b) { return (a < b) ? b : a; }
__device__ __forceinline__ double smin(double a, double b) { return fp64::less(b, a) ? b : a; }
__device__ __forceinline__ double smax(double a, double b) { return fp64::less(a, b) ? b : a; }

// Kernel view of the mesh and physics.
template <class T>
struct KM {
    int n_cells, n_faces;
    int ahead;  // blocks ahead of the running one whose data is brought into L2 (0: none)
    const int4* __restrict__ cslot;  // +(face+1) if the cell is the face's cell 0, -(face+1) if cell 1, 0 empty
    const int4* __restrict__ cnbr;   // the face's other cell, or -(b+1) for boundary face b
    const T* __restrict__ area;
    const int2* __restrict__ fcell;
    const V2<T>* __restrict__ fn;
    const V2<T>* __restrict__ fLg;
    const V2<T>* __restrict__ fd0;
    const V2<T>* __restrict__ fd1;
    const V2<T>* __restrict__ dsl;  // FP32: the cells' own offsets, slot s of cell i at s * n_cells + i
    const V4<T>* __restrict__ ft;
    const int* __restrict__ btype;
    const V4<T>* __restrict__ bq;
    T gamma, R, mu, kheat, limk, cfl;
    int limiter;
    int lsq;                          // least-squares gradient
    const V2<T>* __restrict__ lsqw;   // 4 per cell: (M d_j) of local edge j
    const int* __restrict__ lsqs;     // per cell: slot of local edge j (2 bits each), edge count << 8
    // Spalart-Allmaras (VISC 2): eddy viscosity of the stage state per cell,
    // and the gas constants of the turbulent heat conductivity
    const T* __restrict__ mut;
    T cp, PrL, PrT;
};

__device__ __forceinline__ bool two_sided(int bt) { return bt == BT_INTERNAL || bt == BT_INOUT; }

// ---------------------------------------------------------------- physics
// sabs and entropy_correction, physics.h:84-86, 133-135
template <class T> __device__ __forceinline__ T sabs(T x) { return dsqrt(x * x + T(1e-4)); }
template <class T> __device__ __forceinline__ T entropy_corr(T l, T d) {
    return l > d ? l : (l * l + d * d) / (T(2) * d);
}

// Central flux + Roe dissipation with Harten's entropy fix, physics.h:168-228.
template <class T>
__device__ __forceinline__ void roe_flux(const T gamma, const T nx, const T ny, const T* qL, const T* qR, T* f) {
    const T rho_L = qL[0], rho_u_L = qL[1], rho_v_L = qL[2], rho_e_L = qL[3];
    const T rho_R = qR[0], rho_u_R = qR[1], rho_v_R = qR[2], rho_e_R = qR[3];
    const T V_L = (rho_u_L * nx + rho_v_L * ny) / rho_L;
    const T V_R = (rho_u_R * nx + rho_v_R * ny) / rho_R;
    const T p_L = (gamma - T(1)) * (rho_e_L - T(0.5) / rho_L * (rho_u_L * rho_u_L + rho_v_L * rho_v_L));
    const T p_R = (gamma - T(1)) * (rho_e_R - T(0.5) / rho_R * (rho_u_R * rho_u_R + rho_v_R * rho_v_R));
    f[0] = (V_L * rho_L + V_R * rho_R) * T(0.5);
    f[1] = (V_L * rho_u_L + p_L * nx + V_R * rho_u_R + p_R * nx) * T(0.5);
    f[2] = (V_L * rho_v_L + p_L * ny + V_R * rho_v_R + p_R * ny) * T(0.5);
    f[3] = (V_L * (rho_e_L + p_L) + V_R * (rho_e_R + p_R)) * T(0.5);
    const T pL = p_L, pR = p_R;
    const T uL = qL[1] / qL[0];
    const T uR = qR[1] / qR[0];
    const T vL = qL[2] / qL[0];
    const T vR = qR[2] / qR[0];
    const T srhoL = dsqrt(qL[0]);
    const T srhoR = dsqrt(qR[0]);
    const T rho = srhoR * srhoL;
    const T u = (uL * srhoL + uR * srhoR) / (srhoL + srhoR);
    const T v = (vL * srhoL + vR * srhoR) / (srhoL + srhoR);
    const T h = ((qL[3] + pL) / qL[0] * srhoL + (qR[3] + pR) / qR[0] * srhoR) / (srhoL + srhoR);
    const T q2 = u * u + v * v;
    const T c = dsqrt((gamma - T(1)) * (h - T(0.5) * q2));
    const T V = u * nx + v * ny;
    const T VR = uR * nx + vR * ny;
    const T VL = uL * nx + vL * ny;
    const T lambda_cm = entropy_corr(sabs(V - c), T(0.05) * c);
    const T lambda_c = entropy_corr(sabs(V), T(0.05) * c);
    const T lambda_cp = entropy_corr(sabs(V + c), T(0.05) * c);
    const T kF1 = lambda_cm * ((pR - pL) - rho * c * (VR - VL)) / (T(2) * c * c);
    const T kF234_0 = lambda_c * ((qR[0] - qL[0]) - (pR - pL) / (c * c));
    const T kF234_1 = lambda_c * rho;
    const T kF5 = lambda_cp * ((pR - pL) + rho * c * (VR - VL)) / (T(2) * c * c);
    f[0] -= T(0.5) * (kF1 + kF234_0 + kF5);
    f[1] -= T(0.5) * (kF1 * (u - c * nx) + kF234_0 * u + kF234_1 * (uR - uL - (VR - VL) * nx) + kF5 * (u + c * nx));
    f[2] -= T(0.5) * (kF1 * (v - c * ny) + kF234_0 * v + kF234_1 * (vR - vL - (VR - VL) * ny) + kF5 * (v + c * ny));
    f[3] -= T(0.5) * (kF1 * (h - c * V) + kF234_0 * q2 * T(0.5) +
                      kF234_1 * (u * (uR - uL) + v * (vR - vL) - V * (VR - VL)) + kF5 * (h + c * V));
}

// The same in FP64, twice the flux (the caller's face length takes the half,
// an exact factor): every quotient, root and compare in integer arithmetic
// with shared denominators, and every factor of two folded into a sum as an
// exact product or into a denominator's exponent, so each result has the bits
// of the expression above.  What would be left on the FP64 pipe are about 135
// sums and products (the compiler's form held it for 18 divisions at 7 and 6
// roots at 7.6 instructions each beside 180 sums and products); 31 of the
// products, and 16 of the reconstruction's, are given to the integer lanes,
// which the quotients alone leave idle half of the time: k_face_flux on 1.57M
// faces 1203 us at first, 630 without the compiler's divisions, 467 so.
__device__ __forceinline__ double entropy_corr64(const double l, const double d, const fp64::Den& d2) {
    return fp64::less(d, l) ? l : fp64::quot(l * l + d * d, d2);
}
__device__ __forceinline__ void roe_flux2(const double gamma, const double nx, const double ny, const double* qL,
                                          const double* qR, double* f) {
    using namespace fp64;
    const Den iL = den(qL[0]), iR = den(qR[0]);
    const double g1 = gamma - 1.0;
    const double V_L = quot(qL[1] * nx + qL[2] * ny, iL);
    const double V_R = quot(qR[1] * nx + qR[2] * ny, iR);
    const double pL = g1 * (qL[3] - quot(0.5, iL) * (qL[1] * qL[1] + qL[2] * qL[2]));
    const double pR = g1 * (qR[3] - quot(0.5, iR) * (qR[1] * qR[1] + qR[2] * qR[2]));
    const double uL = quot(qL[1], iL), uR = quot(qR[1], iR);
    const double vL = quot(qL[2], iL), vR = quot(qR[2], iR);
    const double srhoL = root(qL[0]), srhoR = root(qR[0]);
    const double rho = srhoR * srhoL;
    const Den is = den(srhoL + srhoR);
    const double u = quot(uL * srhoL + uR * srhoR, is);
    const double v = quot(vL * srhoL + vR * srhoR, is);
    const double h = quot(quot(qL[3] + pL, iL) * srhoL + quot(qR[3] + pR, iR) * srhoR, is);
    const double q2 = u * u + v * v;
    const double c = root(g1 * __fma_rn(-0.5, q2, h));
    const double V = u * nx + v * ny;
    const double VR = uR * nx + vR * ny;
    const double VL = uL * nx + vL * ny;
    const double d = 0.05 * c;
    const Den d2 = twice(den(d));
    const double lambda_cm = entropy_corr64(sabs(V - c), d, d2);
    const double lambda_c = entropy_corr64(sabs(V), d, d2);
    const double lambda_cp = entropy_corr64(sabs(V + c), d, d2);
    const Den cc = den(c * c), cc2 = twice(cc);
    const double dp = pR - pL, dV = VR - VL, rcV = rho * c * dV;
    const double kF1 = quot(lambda_cm * (dp - rcV), cc2);
    const double kF234_0 = lambda_c * ((qR[0] - qL[0]) - quot(dp, cc));
    const double kF234_1 = lambda_c * rho;
    const double kF5 = quot(lambda_cp * (dp + rcV), cc2);
    const double cnx = c * nx, cny = c * ny, cV = c * V;
    // the products of these sums on the integer lanes, beside the FP64 pipe
    f[0] = (imul(V_L, qL[0]) + imul(V_R, qR[0])) - (kF1 + kF234_0 + kF5);
    f[1] = (imul(V_L, qL[1]) + imul(pL, nx) + imul(V_R, qR[1]) + imul(pR, nx)) -
           (imul(kF1, u - cnx) + imul(kF234_0, u) + imul(kF234_1, uR - uL - imul(dV, nx)) + imul(kF5, u + cnx));
    f[2] = (imul(V_L, qL[2]) + imul(pL, ny) + imul(V_R, qR[2]) + imul(pR, ny)) -
           (imul(kF1, v - cny) + imul(kF234_0, v) + imul(kF234_1, vR - vL - imul(dV, ny)) + imul(kF5, v + cny));
    f[3] = (imul(V_L, qL[3] + pL) + imul(V_R, qR[3] + pR)) -
           (__fma_rn(0.5, imul(kF234_0, q2), imul(kF1, h - cV)) +
            imul(kF234_1, imul(u, uR - uL) + imul(v, vR - vL) - imul(V, dV)) + imul(kF5, h + cV));
}
__device__ __forceinline__ void roe_flux(const double gamma, const double nx, const double ny, const double* qL,
                                         const double* qR, double* f) {
    roe_flux2(gamma, nx, ny, qL, qR, f);
#pragma unroll
    for (int k = 0; k < 4; ++k) f[k] *= 0.5;
}

// Laminar viscous flux at the mean state, physics.h:230-258 with
// calc_grad_p / calc_grad_temp / calc_grad_u / calc_grad_v (physics.h:33-82).
template <class T>
__device__ __forceinline__ void laminar_flux(const T gamma, const T Rgas, const T mu, const T kheat, const T nx,
                                             const T ny, const T* qL, const T* qR, const T* gx, const T* gy, T* f) {
    T qc[4];
    for (int k = 0; k < 4; ++k) qc[k] = T(0.5) * (qL[k] + qR[k]);
    const Div<T> i1(qc[0]), i2(qc[0] * qc[0]), i3(T(3));
    const T p = (gamma - T(1)) * (qc[3] - i1(T(0.5)) * (qc[1] * qc[1] + qc[2] * qc[2]));
    // (FP64: half of the products on the integer lanes, as in roe_flux2)
    T gp0 = T(2) * gx[3];
    gp0 -= i1(imul(gx[1], qc[1])) + i2(imul(qc[1], imul(gx[1], qc[0]) - gx[0] * qc[1]));
    gp0 -= i1(imul(gx[2], qc[2])) + i2(imul(qc[2], imul(gx[2], qc[0]) - gx[0] * qc[2]));
    gp0 *= T(0.5) * (gamma - T(1));
    T gp1 = T(2) * gy[3];
    gp1 -= i1(imul(gy[1], qc[1])) + i2(imul(qc[1], imul(gy[1], qc[0]) - gy[0] * qc[1]));
    gp1 -= i1(imul(gy[2], qc[2])) + i2(imul(qc[2], imul(gy[2], qc[0]) - gy[0] * qc[2]));
    gp1 *= T(0.5) * (gamma - T(1));
    const T Rinv = fdiv(T(1), Rgas);
    const T gT0 = Rinv * i2(imul(gp0, qc[0]) - gx[0] * p);
    const T gT1 = Rinv * i2(imul(gp1, qc[0]) - gy[0] * p);
    const T gu0 = i2(imul(qc[0], gx[1]) - qc[1] * gx[0]);
    const T gu1 = i2(imul(qc[0], gy[1]) - qc[1] * gy[0]);
    const T gv0 = i2(imul(qc[0], gx[2]) - qc[2] * gx[0]);
    const T gv1 = i2(imul(qc[0], gy[2]) - qc[2] * gy[0]);
    const T div3 = i3(gu0 + gv1);
    const T tau_xx = T(2) * mu * (gu0 - div3);
    const T tau_yy = T(2) * mu * (gv1 - div3);
    const T tau_xy = mu * (gu1 + gv0);
    const T uc = i1(qc[1]), vc = i1(qc[2]);
    const T phi0 = imul(uc, tau_xx) + vc * tau_xy + kheat * gT0;
    const T phi1 = imul(uc, tau_xy) + vc * tau_yy + kheat * gT1;
    f[1] -= imul(nx, tau_xx) + ny * tau_xy;
    f[2] -= imul(nx, tau_xy) + ny * tau_yy;
    f[3] -= imul(nx, phi0) + ny * phi1;
}

// Boundary ghost state from the interior state qL and the stored boundary
// state qbc: slip wall (physics.h:311-339), wall (physics.h:377-405),
// farfield characteristics (physics.h:446-530, with the outside `va` of the
// subsonic outlet, line 524), internal average otherwise (physics.h:267-276).
template <class T>
__device__ __forceinline__ void ghost_state(const int type, const T gamma, const T nx, const T ny, const T* qL,
                                            const T* qbc, T* qR) {
    if (type == BT_SLIP) {
        const T rhoV = qL[1] * nx + qL[2] * ny;
        qR[0] = qL[0];
        qR[1] = qL[1] - T(2) * rhoV * nx;
        qR[2] = qL[2] - T(2) * rhoV * ny;
        qR[3] = qL[3];
        return;
    }
    if (type == BT_WALL) {
        qR[0] = qL[0]; qR[1] = -qL[1]; qR[2] = -qL[2]; qR[3] = qL[3];
        return;
    }
    if (type != BT_FARFIELD) {
        for (int k = 0; k < 4; ++k) qR[k] = (qL[k] + qbc[k]) * T(0.5);
        return;
    }
    const T rho = qL[0], rho_u = qL[1], rho_v = qL[2], rho_e = qL[3];
    const T bc_rho = qbc[0], bc_rhou = qbc[1], bc_rhov = qbc[2], bc_rhoe = qbc[3];
    const Div<T> ib(bc_rho), ii(rho), ig(gamma - T(1));
    const T bc_u = ib(bc_rhou);
    const T bc_v = ib(bc_rhov);
    const T bc_p = (gamma - T(1)) * (bc_rhoe - ib(T(0.5)) * (bc_rhou * bc_rhou + bc_rhov * bc_rhov));
    const T p = (gamma - T(1)) * (rho_e - ii(T(0.5)) * (rho_u * rho_u + rho_v * rho_v));
    const T c = dsqrt(ii(gamma * p));
    const Div<T> irc(rho * c);
    const T mach = irc(dsqrt(rho_u * rho_u + rho_v * rho_v));
    const T inlet_outlet = rho_u * nx + rho_v * ny;
    if (mach > T(1)) {
        if (inlet_outlet < T(0)) {
            qR[0] = bc_rho;
            qR[1] = bc_rho * bc_u;
            qR[2] = bc_rho * bc_v;
            qR[3] = ig(bc_p) + T(0.5) * bc_rho * (bc_u * bc_u + bc_v * bc_v);
        } else {
            qR[0] = rho; qR[1] = rho_u; qR[2] = rho_v; qR[3] = rho_e;
        }
    } else {
        const T pa = bc_p, rhoa = bc_rho, ua = bc_u, va = bc_v;
        const T pd = p, rhod = rho, ud = ii(rho_u), vd = ii(rho_v);
        const T rho0 = rho, c0 = c;
        const Div<T> icc(c0 * c0);
        if (inlet_outlet < T(0)) {
            const T pb = T(0.5) * (pa + pd - rho0 * c0 * (nx * (ua - ud) + ny * (va - vd)));
            qR[0] = rhoa + icc(pb - pa);
            qR[1] = qR[0] * (ua - irc(nx * (pa - pb)));
            qR[2] = qR[0] * (va - irc(ny * (pa - pb)));
            qR[3] = ig(pb) + fdiv(T(0.5), qR[0]) * (qR[1] * qR[1] + qR[2] * qR[2]);
        } else {
            const T pb = pa;
            qR[0] = rhod + icc(pb - pd);
            qR[1] = qR[0] * (ud + irc(nx * (pd - pb)));
            qR[2] = qR[0] * (va + irc(ny * (pd - pb)));
            qR[3] = ig(pb) + fdiv(T(0.5), qR[0]) * (qR[1] * qR[1] + qR[2] * qR[2]);
        }
    }
}

// Face flux F (not yet times length) of the reference's per-face functor:
// internal faces (and frozen-ghost boundaries) with the face gradient for the
// laminar term; wall/farfield faces through their ghost state without
// gradients (physics.h:287-299, 352-364, 417-432).  With zero gradients the
// laminar term is exactly zero, so boundary faces skip it.
// VISC 2 (Spalart-Allmaras): the laminar terms with mu_L + mu_t,f and
// cp (mu_L / Pr_L + mu_t,f / Pr_T), mu_t,f the mean of the face's two cells.
template <class T, int VISC>
__device__ __forceinline__ void face_flux(const KM<T>& m, const int bt, const T nx, const T ny, const T* qL,
                                          const T* qR, const T* fgx, const T* fgy, T* f, const T mut_f = T(0)) {
    if (two_sided(bt)) {
        roe_flux(m.gamma, nx, ny, qL, qR, f);
        if (VISC == 1) laminar_flux(m.gamma, m.R, m.mu, m.kheat, nx, ny, qL, qR, fgx, fgy, f);
        if (VISC == 2)
            laminar_flux(m.gamma, m.R, m.mu + mut_f, m.cp * (fdiv(m.mu, m.PrL) + fdiv(mut_f, m.PrT)), nx, ny, qL, qR, fgx, fgy,
                         f);
    } else {
        // VISC 2: the inviscid part of a no-slip wall takes the slip-wall
        // ghost (pressure only); the caller adds the wall shear
        T qb[4];
        ghost_state(VISC == 2 && bt == BT_WALL ? BT_SLIP : bt, m.gamma, nx, ny, qL, qR, qb);
        roe_flux(m.gamma, nx, ny, qL, qb, f);
    }
}

// Spalart-Allmaras no-slip wall: the wall shear mu_L u_t / delta of the cell
// state q0 (u_t its tangential velocity, delta the distance from its centroid
// to the wall face, d0 = face centre - centroid), added to the face flux F.
template <class T>
__device__ __forceinline__ void sa_wall_shear(const KM<T>& m, const T nx, const T ny, const T d0x, const T d0y,
                                              const T* q0, T* f) {
    const Div<T> delta(dabs(d0x * nx + d0y * ny)), i0(q0[0]);
    const T u = i0(q0[1]), v = i0(q0[2]);
    const T un = u * nx + v * ny;
    f[1] += delta(m.mu * (u - un * nx));
    f[2] += delta(m.mu * (v - un * ny));
}

// Spectral radius (c + |V_n|) of one side, solver.h:329-344.
template <class T>
__device__ __forceinline__ T face_eig(const T gamma, const T nx, const T ny, const T* q) {
    const Div<T> i0(q[0]);
    const T V = i0(q[1] * nx + q[2] * ny);
    const T p = (gamma - T(1)) * (q[3] - i0(T(0.5)) * (q[1] * q[1] + q[2] * q[2]));
    return dsqrt(i0(p * gamma)) + dabs(V);
}

// Venkatakrishnan limiter of one cell-face-variable (solver.h:578-584) and
// the Michalak variant (solver.h:557-576, physics.h:581-592).
template <class T>
__device__ __forceinline__ T limiter_value(const int kind, const T dqg, const T delta_max, const T delta_min,
                                           const T K3a) {
    if (kind == 0) {
        // the side first: one formula for both signs, so a warp whose lanes
        // differ in sign forms it once, not twice
        if (!(dabs(dqg) > T(1e-16))) return T(1);
        const T dm = dqg > T(0) ? delta_max : delta_min;
        return T(1) / dqg * ((dm * dm + K3a) * dqg + T(2) * dqg * dqg * dm) /
               (dm * dm + T(2) * dqg * dqg + dm * dqg + K3a);
    }
    const T dMaxMin2 = (delta_max - delta_min) * (delta_max - delta_min);
    T sig;
    if (dMaxMin2 <= K3a) sig = T(1);
    else if (dMaxMin2 <= T(2) * K3a) {
        const T y = (dMaxMin2 / K3a - T(1));
        sig = T(2) * y * y * y - T(3) * y * y + T(1);
    } else sig = T(0);
    T lim = T(1);
    if (sig < T(1)) {
        T y = T(2);
        bool set = false;
        if (dqg > T(1e-14)) { y = delta_max / dqg; set = true; }
        else if (dqg < T(-1e-14)) { y = delta_min / dqg; set = true; }
        if (set) {
            const T YT = T(2);
            const T a = T(1) / (YT * YT) - T(2) / (YT * YT * YT);
            const T b = -T(3) / T(2) * a * YT - T(0.5) / YT;
            lim = (y >= YT) ? T(1) : a * y * y * y + b * y * y + y;
        }
    }
    return sig + (T(1) - sig) * lim;
}

// The same in FP64 (bits of the expressions above; factors of two as exact
// products of a fused multiply-add, quotients and compares in integers).
__device__ __forceinline__ double limiter_value(const int kind, const double dqg, const double delta_max,
                                                const double delta_min, const double K3a) {
    using namespace fp64;
    const uint64_t u = bits_of(dqg), mag = u & 0x7fffffffffffffffull;
    const bool pos = (u >> 63) == 0;
    if (kind == 0) {
        // |dqg| > 1e-16, false for a NaN
        const bool on = mag > 0x3c9cd2b297d889bcull && mag <= 0x7ff0000000000000ull;
        const double g = on ? dqg : 1.0;
        const double dm = pos ? delta_max : delta_min;
        const double d2 = dm * dm, g2 = g * g;
        const double num = __fma_rn(2.0, g2 * dm, (d2 + K3a) * g);
        const double dn = (__fma_rn(2.0, g2, d2) + dm * g) + K3a;
        const double lim = quot(quot(1.0, den(g)) * num, den(dn));
        return on ? lim : 1.0;
    }
    const double dd = delta_max - delta_min;
    const double dMaxMin2 = dd * dd;
    double sig;
    if (less_equal(dMaxMin2, K3a)) sig = 1.0;
    else if (less_equal(dMaxMin2, 2.0 * K3a)) {
        const double y = div(dMaxMin2, K3a) - 1.0;
        sig = 2.0 * y * y * y - 3.0 * y * y + 1.0;
    } else sig = 0.0;
    double lim = 1.0;
    if (less(sig, 1.0)) {
        // |dqg| > 1e-14, false for a NaN
        const bool on = mag > 0x3d06849b86a12b9bull && mag <= 0x7ff0000000000000ull;
        const double y = on ? div(pos ? delta_max : delta_min, dqg) : 2.0;
        const double YT = 2.0;
        const double a = 1.0 / (YT * YT) - 2.0 / (YT * YT * YT);
        const double b = -3.0 / 2.0 * a * YT - 0.5 / YT;
        lim = less_equal(YT, y) ? 1.0 : a * y * y * y + b * y * y + y;
    }
    return sig + (1.0 - sig) * lim;
}

// F times the face length.  FP64 without a viscous term: twice the flux times
// half the length, an exact factor.
template <class T, int VISC>
__device__ __forceinline__ void face_flux_length(const KM<T>& m, const int bt, const T nx, const T ny, const T* qL,
                                                 const T* qR, const T* fgx, const T* fgy, const T L, T* fl,
                                                 const T mut_f) {
    face_flux<T, VISC>(m, bt, nx, ny, qL, qR, fgx, fgy, fl, mut_f);
#pragma unroll
    for (int k = 0; k < 4; ++k) fl[k] = fl[k] * L;
}
template <>
__device__ __forceinline__ void face_flux_length<double, 0>(const KM<double>& m, const int bt, const double nx,
                                                            const double ny, const double* qL, const double* qR,
                                                            const double*, const double*, const double L, double* fl,
                                                            const double) {
    double qb[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) qb[k] = qR[k];
    if (!two_sided(bt)) ghost_state(bt, m.gamma, nx, ny, qL, qR, qb);
    roe_flux2(m.gamma, nx, ny, qL, qb, fl);
    const double h = 0.5 * L;
#pragma unroll
    for (int k = 0; k < 4; ++k) fl[k] = fl[k] * h;
}

}  // namespace dev
}  // namespace afx
