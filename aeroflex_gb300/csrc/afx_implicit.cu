// Implicit solver of the rans path on the GPU (implicitSolver, solver.h:852-1213,
// driven by multigrid<implicitSolver>::run_solver, multigrid.h:240-293).
//
// Each iteration assembles the reference's linear system
//     (A_i/dt_i I + sum_faces dF/dq L) dQ = -sum_faces F L
// over the real cells (ghost rows are identity with a zero right-hand side in
// the reference, so ghost unknowns stay zero and drop out), solves it with
// restarted GMRES(30) to a relative tolerance of 1e-2 (at most 500 Krylov
// iterations), and updates q += relaxation dQ, followed by up to
// rhs_iterations chord steps with the same matrix.
//
// GB300 form:
//   * face Jacobians J = dF/dq_c0 L, K = dF/dq_c1 L by the reference's
//     one-sided differences (physics.h:533-578: step max(1e-6, 1e-6 |q|)),
//     one thread per face;
//   * block rows, not a general sparse matrix: rows grouped by colour (no
//     two face neighbours share a colour), one 4x4 diagonal block per row and
//     four off-diagonal ELL blocks (K for the face's cell 0, -J for its cell
//     1), interleaved across rows so every warp load is contiguous;
//   * preconditioner: block ILU(0) in that colour ordering (the factor's
//     diagonal blocks formed colour by colour), applied as a forward then a
//     backward sweep over the colours -- a fixed linear operator, so right
//     preconditioned GMRES applies unchanged;
//   * Krylov vectors and matrix blocks in T = double (FP64 path) or float
//     (FP32-mixed path: the right-hand side, the update and the norms stay
//     FP64, so the iteration converges to the FP64 solution);
//   * CGS2 in three fused passes over the basis, 16-byte loads; every
//     reduction is a fixed-order two-level sum (deterministic);
//   * each solve is one CUDA graph whose restart and Arnoldi loops are
//     device-side WHILE nodes (or, with krylov_graph = 0, the same kernels
//     from a host loop);
//   * the adjoint transposes the filled system in place and reuses all of it.
#include <algorithm>
#include <memory>
#include <string>
#include <vector>

#define AFX_CONTRACTED  // this unit is compiled with multiply-add contraction
#include "afx_host.hpp"
#include "afx_kernels_impl.cuh"
#include "afx_pdl.cuh"

namespace afx {
namespace dev {

constexpr int GM_M = 30;       // GMRES restart length (Eigen's default)
constexpr int DOT_THREADS = 256;

struct GmresCtl {
    int stop;    // the current cycle has converged / ended
    int k;       // Arnoldi steps taken in the current cycle
    int iters;   // Krylov iterations of this solve
    int halt;    // no further restart cycle
    int max_iters;
    int graph;   // launched inside the solve graph: set the WHILE conditions
    cudaGraphConditionalHandle hin, hout;  // WHILE conditions: Arnoldi steps, restart cycles
    double tol;  // absolute residual target
    double res;  // current residual estimate
    double H[(GM_M + 1) * GM_M];  // column-major: H[i + (GM_M + 1) * j]
    double g[GM_M + 1], cs[GM_M], sn[GM_M], y[GM_M];
    double hnext;  // h_{j+1,j} of the last step (before rotation)
};

template <class T> struct B4;
template <> struct B4<double> { using type = d4; };
template <> struct B4<float> { using type = float4; };

// Krylov-side vectors in their own precision T: FP32 arithmetic stays in the
// FP32 pipes (a float-to-double conversion per operand would run on GB300's
// FP64 pipe, at ~1/64 of the FP32 rate)
__device__ __forceinline__ void ldt(const d4* p, double* v) {
    const double2* c = reinterpret_cast<const double2*>(p);
    const double2 a = ldw(c), b = ldw(c + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void ldt(const float4* p, float* v) {
    const float4 a = ldw(p);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void stt(d4* p, const double* v) { st4(p, v); }
__device__ __forceinline__ void stt(float4* p, const float* v) { *p = make_float4(v[0], v[1], v[2], v[3]); }

// Row r of a 4x4 block (row-major), one (FP32) or two (FP64) 16-byte chunks
// `stride` chunks apart, and its product with x.
template <class T> struct Row { T a[4]; };
__device__ __forceinline__ Row<float> row_at(const float* __restrict__ chunk, const size_t) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(chunk));
    return Row<float>{{v.x, v.y, v.z, v.w}};
}
__device__ __forceinline__ Row<double> row_at(const double* __restrict__ chunk, const size_t stride) {
    const double2* c = reinterpret_cast<const double2*>(chunk);
    const double2 u = __ldg(c), v = __ldg(c + stride);
    return Row<double>{{u.x, u.y, v.x, v.y}};
}
template <class T>
__device__ __forceinline__ T row_dot(const Row<T>& r, const T* x) {
    T t = 0;
    t += r.a[0] * x[0];
    t += r.a[1] * x[1];
    t += r.a[2] * x[2];
    t += r.a[3] * x[3];
    return t;
}

// Batch: a cell of a case that has stopped takes no part in the linear
// solve (its rows and unknowns are zero), so a case that went non-finite
// cannot spread into the others
__device__ __forceinline__ bool held(const int* case_of, const int* case_done, const int i) {
    return case_done && ((volatile const int*)case_done)[__ldg(&case_of[i])];
}

// A batch case whose diagonal block cannot be inverted stops (status 4)
// instead of failing the whole batch; the first cell to find it stops it.
__device__ __forceinline__ void stop_case(const int* case_of, int* case_done, CaseCtrl* cctrl, Ctrl* ctrl,
                                          const int i) {
    const int c = __ldg(&case_of[i]);
    if (atomicCAS(&case_done[c], 0, 1) == 0) {
        cctrl[c].status = 4;
        cctrl[c].done = 1;
        atomicAdd(&ctrl->ndone, 1);
    }
}

// ------------------------------------------------------------- assembly
// F of face f for the cell states (no reconstruction; the ghost side is the
// stored boundary state), as the reference's flux functor evaluates it.
// Spalart-Allmaras (VISC 2): the eddy viscosity is frozen at its current
// value (mut_f) and the no-slip wall shear of the cell state is included.
template <int VISC>
__device__ __forceinline__ void flux_cells(const KM<double>& m, const int bt, const double nx, const double ny,
                                           const double* qL, const double* qR, const double* fgx, const double* fgy,
                                           double* F, const double mut_f = 0.0, const double2 d0 = double2()) {
    face_flux<double, VISC>(m, bt, nx, ny, qL, qR, fgx, fgy, F, mut_f);
    if (VISC == 2 && bt == BT_WALL) sa_wall_shear(m, nx, ny, d0.x, d0.y, qL, F);
}

// calc_convective_jacobian (physics.h:533-578) times the face length:
// J = dF/dq_L, K = dF/dq_R by one-sided differences with the reference's
// step and its in-place perturb/restore of each component.
template <class T, int VISC>
__global__ void __launch_bounds__(128) k_imp_jac(const KM<double> m, const int n_faces, const d4* __restrict__ q,
                                                 const d4* __restrict__ gx, const d4* __restrict__ gy,
                                                 T* __restrict__ jf, const Ctrl* __restrict__ ctrl) {
    if (ctrl->done) return;
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_faces) return;
    const int2 cc = __ldg(&m.fcell[f]);
    const double2 n = __ldg(&m.fn[f]);
    const double L = __ldg(&m.fLg[f]).x;
    double qL[4], qR[4];
    ld4(&q[cc.x], qL);
    int bt = BT_INTERNAL;
    if (cc.y >= 0) {
        ld4(&q[cc.y], qR);
    } else {
        bt = __ldg(&m.btype[-cc.y - 1]);
        ld4(&m.bq[-cc.y - 1], qR);
    }
    double fgx[4] = {0, 0, 0, 0}, fgy[4] = {0, 0, 0, 0};
    double mut_f = 0.0;
    double2 d0 = make_double2(0.0, 0.0);
    if (VISC == 2) {
        if (two_sided(bt)) mut_f = 0.5 * (__ldg(&m.mut[cc.x]) + __ldg(&m.mut[cc.y]));
        d0 = __ldg(&m.fd0[f]);
    }
    if (VISC >= 1 && two_sided(bt)) {
        double gx0[4], gy0[4], gx1[4] = {0, 0, 0, 0}, gy1[4] = {0, 0, 0, 0};
        ld4(&gx[cc.x], gx0);
        ld4(&gy[cc.x], gy0);
        if (cc.y >= 0) {
            ld4(&gx[cc.y], gx1);
            ld4(&gy[cc.y], gy1);
        }
        face_gradient(qL, qR, gx0, gy0, gx1, gy1, ldv4<double>(&m.ft[f]), fgx, fgy);
    }
    double f0[4];
    flux_cells<VISC>(m, bt, n.x, n.y, qL, qR, fgx, fgy, f0, mut_f, d0);
    T* out = jf + 32 * (size_t)f;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
        const double upd = fmax(1e-6, fabs(qL[c]) * 1e-6);
        qL[c] += upd;
        double fp[4];
        flux_cells<VISC>(m, bt, n.x, n.y, qL, qR, fgx, fgy, fp, mut_f, d0);
        qL[c] -= upd;
#pragma unroll
        for (int r = 0; r < 4; ++r) out[4 * r + c] = (T)((fp[r] - f0[r]) / upd * L);
    }
    if (cc.y >= 0) {
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            const double upd = fmax(1e-6, fabs(qR[c]) * 1e-6);
            qR[c] += upd;
            double fp[4];
            flux_cells<VISC>(m, bt, n.x, n.y, qL, qR, fgx, fgy, fp, mut_f, d0);
            qR[c] -= upd;
#pragma unroll
            for (int r = 0; r < 4; ++r) out[16 + 4 * r + c] = (T)((fp[r] - f0[r]) / upd * L);
        }
    }
}

// Row layout of the linear system.  Rows are grouped by colour (the cells
// of a colour in device order), so a colour of the Gauss-Seidel sweep is a
// contiguous range of rows and every per-row access is coalesced.  A row's
// four off-diagonal blocks (ELL slots: the cell's face slots) carry the sign
// of the cell's side.
struct Ell {
    const int* perm;      // [N] device cell of row p
    const int4* col;      // [N] row of the neighbour in each slot, -1: none
    const int4* face;     // [N] signed face of each slot (cslot convention), 0: none
    const int4* tr;       // [N] ELL index 4 q + s' of the transposed block of each slot
    const int* case_row;  // [N] batch: case of row p, else null
};

// Off-diagonal blocks are interleaved across rows: 16-byte chunk c of slot
// s of row p (c = the block's row for FP32, half-row for FP64) is chunk
// (s * CPB + c) * N + p, so a warp's loads of one chunk are contiguous.
template <class T> struct Ell16 { static constexpr int W = 16 / sizeof(T), CPB = 16 / W; };
template <class T>
__device__ __forceinline__ size_t ell_at(const int N, const int p, const int s, const int k) {
    constexpr int W = Ell16<T>::W, CPB = Ell16<T>::CPB;
    return ((size_t)(s * CPB + k / W) * N + p) * W + (k % W);
}
// row r of the block of slot s of row p
template <class T>
__device__ __forceinline__ Row<T> ell_row(const T* __restrict__ off, const int N, const int p, const int s,
                                          const int r) {
    constexpr int W = Ell16<T>::W, CPB = Ell16<T>::CPB;
    return row_at(off + ((size_t)(s * CPB + r * (CPB / 4)) * N + p) * W, (size_t)N);
}

// Diagonal block A/dt I + sum (own: J, other: -K) of row p and its inverse
// (Gauss-Jordan with partial pivoting, in double), and the row's
// off-diagonal blocks (own: K, other: -J) from the face Jacobians.
template <class T>
__global__ void __launch_bounds__(128) k_imp_assemble(const KM<double> m, const Ell e, const double* __restrict__ dt,
                                                      const T* __restrict__ jf, T* __restrict__ dblk,
                                                      T* __restrict__ dinv, T* __restrict__ off,
                                                      int* __restrict__ singular, Ctrl* __restrict__ ctrl,
                                                      int* __restrict__ case_done, CaseCtrl* __restrict__ cctrl) {
    if (ctrl->done) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= m.n_cells) return;
    const int i = __ldg(&e.perm[p]);
    const int4 fsl = __ldg(&e.face[p]);
    const int4 col = __ldg(&e.col[p]);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int fs = pick(fsl, s);
        if (fs == 0 || pick(col, s) < 0) continue;
        const int f = (fs > 0 ? fs : -fs) - 1;
        const T* B = jf + 32 * (size_t)f + (fs > 0 ? 16 : 0);
#pragma unroll
        for (int k = 0; k < 16; ++k) off[ell_at<T>(m.n_cells, p, s, k)] = fs > 0 ? B[k] : -B[k];
    }
    if (held(e.case_row, case_done, p)) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            dblk[16 * (size_t)p + k] = T((k % 5 == 0) ? 1 : 0);
            dinv[16 * (size_t)p + k] = T((k % 5 == 0) ? 1 : 0);
        }
        return;
    }
    double D[16];
    const double ad = __ldg(&m.area[i]) / __ldg(&dt[i]);
#pragma unroll
    for (int k = 0; k < 16; ++k) D[k] = (k % 5 == 0) ? ad : 0.0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int fs = pick(fsl, s);
        if (fs == 0) continue;
        const int f = (fs > 0 ? fs : -fs) - 1;
        const T* B = jf + 32 * (size_t)f + (fs > 0 ? 0 : 16);
        const double sg = fs > 0 ? 1.0 : -1.0;
#pragma unroll
        for (int k = 0; k < 16; ++k) D[k] += sg * (double)B[k];
    }
    T* Do = dblk + 16 * (size_t)p;
#pragma unroll
    for (int k = 0; k < 16; ++k) Do[k] = (T)D[k];
    double I[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) I[k] = (k % 5 == 0) ? 1.0 : 0.0;
    for (int c = 0; c < 4; ++c) {
        int pv = c;
        double best = fabs(D[4 * c + c]);
        for (int r = c + 1; r < 4; ++r)
            if (fabs(D[4 * r + c]) > best) {
                best = fabs(D[4 * r + c]);
                pv = r;
            }
        if (!(best > 0)) {
            if (case_done) {
                stop_case(e.case_row, case_done, cctrl, ctrl, p);
#pragma unroll
                for (int k = 0; k < 16; ++k) dinv[16 * (size_t)p + k] = T((k % 5 == 0) ? 1 : 0);
            } else {
                *singular = 1;
            }
            return;
        }
        if (pv != c)
            for (int k = 0; k < 4; ++k) {
                double t = D[4 * c + k];
                D[4 * c + k] = D[4 * pv + k];
                D[4 * pv + k] = t;
                t = I[4 * c + k];
                I[4 * c + k] = I[4 * pv + k];
                I[4 * pv + k] = t;
            }
        const double inv = 1.0 / D[4 * c + c];
        for (int k = 0; k < 4; ++k) {
            D[4 * c + k] *= inv;
            I[4 * c + k] *= inv;
        }
        for (int r = 0; r < 4; ++r) {
            if (r == c) continue;
            const double fct = D[4 * r + c];
            for (int k = 0; k < 4; ++k) {
                D[4 * r + k] -= fct * D[4 * c + k];
                I[4 * r + k] -= fct * I[4 * c + k];
            }
        }
    }
    T* Io = dinv + 16 * (size_t)p;
#pragma unroll
    for (int k = 0; k < 16; ++k) Io[k] = (T)I[k];
}

// Block ILU(0) in the colour ordering: for the cells of colour c,
//     D~_i = D_i - sum_{neighbours o of a lower colour} O_io D~_o^-1 O_oi,
// inverted into dinv (colour 0 keeps D^-1).  With these inverses the
// symmetric multicolour Gauss-Seidel sweep below applies the ILU(0) factors
// (D~ + L) D~^-1 (D~ + U) exactly.
__device__ __forceinline__ void inv4(const double* A, double* I, int* singular) {
    double D[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        D[k] = A[k];
        I[k] = (k % 5 == 0) ? 1.0 : 0.0;
    }
    for (int c = 0; c < 4; ++c) {
        int p = c;
        double best = fabs(D[4 * c + c]);
        for (int r = c + 1; r < 4; ++r)
            if (fabs(D[4 * r + c]) > best) {
                best = fabs(D[4 * r + c]);
                p = r;
            }
        if (!(best > 0)) {
            *singular = 1;
            return;
        }
        if (p != c)
            for (int k = 0; k < 4; ++k) {
                double t = D[4 * c + k];
                D[4 * c + k] = D[4 * p + k];
                D[4 * p + k] = t;
                t = I[4 * c + k];
                I[4 * c + k] = I[4 * p + k];
                I[4 * p + k] = t;
            }
        const double inv = 1.0 / D[4 * c + c];
        for (int k = 0; k < 4; ++k) {
            D[4 * c + k] *= inv;
            I[4 * c + k] *= inv;
        }
        for (int r = 0; r < 4; ++r) {
            if (r == c) continue;
            const double fct = D[4 * r + c];
            for (int k = 0; k < 4; ++k) {
                D[4 * r + k] -= fct * D[4 * c + k];
                I[4 * r + k] -= fct * I[4 * c + k];
            }
        }
    }
}

template <class T>
__global__ void __launch_bounds__(128) k_imp_ilu(const Ell e, const int N, const T* __restrict__ dblk,
                                                 const T* __restrict__ off, const int c0, const int n,
                                                 T* __restrict__ dinv,
                                                 int* __restrict__ singular, int* __restrict__ case_done,
                                                 CaseCtrl* __restrict__ cctrl, Ctrl* __restrict__ ctrl) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int p = c0 + t;
    if (held(e.case_row, case_done, p)) return;
    double D[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) D[k] = (double)dblk[16 * (size_t)p + k];
    const int4 col = __ldg(&e.col[p]);
    const int4 tr = __ldg(&e.tr[p]);
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
        const int q = pick(col, s);
        if (q < 0 || q >= c0) continue;  // rows of lower colours precede c0
        const int t2 = pick(tr, s);  // 4 q + s': the block of row q, column p
        double Oio[16], Ooi[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            Oio[k] = (double)off[ell_at<T>(N, p, s, k)];
            Ooi[k] = (double)off[ell_at<T>(N, t2 >> 2, t2 & 3, k)];
        }
        const T* Dinv_o = dinv + 16 * (size_t)q;
        double Y[16];  // D~_q^-1 O_qp
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                double acc = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) acc += (double)Dinv_o[4 * r + k] * Ooi[4 * k + c];
                Y[4 * r + c] = acc;
            }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                double acc = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) acc += Oio[4 * r + k] * Y[4 * k + c];
                D[4 * r + c] -= acc;
            }
    }
    double I[16];
    int sing = 0;
    inv4(D, I, &sing);
    if (sing) {
        if (case_done) {
            stop_case(e.case_row, case_done, cctrl, ctrl, p);
        } else {
            *singular = 1;
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) dinv[16 * (size_t)p + k] = (T)I[k];
}

// --------------------------------------------------------- linear algebra
// RT threads per row, each with NC = 4 / RT rows of its 4x4 blocks.  One
// thread per row (16-byte chunks side by side in a warp's loads) streams best
// when there are rows enough to fill the GPU; a colour of a mesh of tens of
// thousands of cells has only a few thousand, and then four threads per row
// put four times as many warps to work (in FP64 a thread's 80 fused
// multiply-adds alone hold the two FP64 lanes of its SM for microseconds).
// The sums run in the order of the block form either way, so the results do
// not depend on RT.  Bound by latency at these sizes: a colour of 3,300 rows in
// FP64 took 8.0 us with one thread per row in blocks of 256, 3.8 us with four.
// Matrix data is read before pdl_wait() where it fits in registers (AHEAD):
// the next colour's blocks arrive while the previous colour is computed, and
// only the gathers of x remain after the wait.
template <class T, int RT> constexpr bool AHEAD = RT == 4 || sizeof(T) == 4;

template <class T, int RT>
__device__ __forceinline__ void row_load(const T* r, const size_t p, const int c, T* s) {
    if constexpr (RT == 1) ldt(reinterpret_cast<const typename B4<T>::type*>(r) + p, s);
    else s[0] = ldw(r + 4 * p + c);
}
template <class T, int RT>
__device__ __forceinline__ void row_store(T* r, const size_t p, const int c, const T* s) {
    if constexpr (RT == 1) stt(reinterpret_cast<typename B4<T>::type*>(r) + p, s);
    else r[4 * p + c] = s[0];
}

// rows of M x for row p (the diagonal block's rows already in d)
template <class T, int RT>
__device__ __forceinline__ void spmv_row(const int n_rows, const int4 col, const Row<T>* d, const T* __restrict__ off,
                                         const T* x, const int p, const int c, T* y) {
    constexpr int NC = 4 / RT;
    const typename B4<T>::type* x4 = reinterpret_cast<const typename B4<T>::type*>(x);
    T xi[4];
    ldt(&x4[p], xi);
#pragma unroll
    for (int r = 0; r < NC; ++r) y[r] = row_dot<T>(d[r], xi);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int q = pick(col, s);
        if (q < 0) continue;
        T xo[4];
        ldt(&x4[q], xo);
#pragma unroll
        for (int r = 0; r < NC; ++r) y[r] += row_dot<T>(ell_row<T>(off, n_rows, p, s, c + r), xo);
    }
}
template <class T, int RT>
__device__ __forceinline__ void diag_rows(const T* __restrict__ d, const int p, const int c, Row<T>* o) {
#pragma unroll
    for (int r = 0; r < 4 / RT; ++r) o[r] = row_at(d + 16 * (size_t)p + 4 * (c + r), 1);
}

// y = M x over the rows (diagonal block, then the slots in face order)
template <class T>
__global__ void __launch_bounds__(256) k_imp_spmv(const int n_rows, const Ell e, const T* __restrict__ dblk,
                                                  const T* __restrict__ off, const T* x, T* y, const int* stop,
                                                  const int* __restrict__ case_done) {
    pdl_wait();
    if (stop && ldw(stop)) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_rows) return;
    T yr[4] = {0, 0, 0, 0};
    if (!held(e.case_row, case_done, p)) {
        Row<T> d[4];
        diag_rows<T, 1>(dblk, p, 0, d);
        spmv_row<T, 1>(n_rows, __ldg(&e.col[p]), d, off, x, p, 0, yr);
    }
    row_store<T, 1>(y, p, 0, yr);
}

// Rows of D_p^-1 s (its rows in d); with RT = 4 the row's four threads hold one
// component of s each
template <class T, int RT>
__device__ __forceinline__ void dinv_row(const Row<T>* d, const T* s, T* x) {
    T sv[4];
    if constexpr (RT == 1) {
#pragma unroll
        for (int k = 0; k < 4; ++k) sv[k] = s[k];
    } else {
        const unsigned lanes = 0xfu << (threadIdx.x & 28);
#pragma unroll
        for (int k = 0; k < 4; ++k) sv[k] = __shfl_sync(lanes, s[0], k, RT);
    }
#pragma unroll
    for (int r = 0; r < 4 / RT; ++r) x[r] = row_dot<T>(d[r], sv);
}

// One row of a block Gauss-Seidel sweep: x_p = D_p^-1 (r_p - sum O x_q) over
// the slots left in col; its blocks first (`blocks`), the arithmetic after.
template <class T, int RT>
struct GsRow {
    static constexpr int NC = 4 / RT;
    int p, c;
    int4 col;
    Row<T> d[NC], o[4][NC];
    // `top`: slots of rows from there on are left out (the forward sweep reads
    // lower colours only: the higher ones have no value yet)
    __device__ __forceinline__ void at(const Ell& e, const int row, const int comp, const int top) {
        p = row;
        c = comp;
        col = __ldg(&e.col[p]);
        if (col.x >= top) col.x = -1;
        if (col.y >= top) col.y = -1;
        if (col.z >= top) col.z = -1;
        if (col.w >= top) col.w = -1;
    }
    __device__ __forceinline__ void blocks(const T* __restrict__ dinv, const T* __restrict__ off, const int N) {
        diag_rows<T, RT>(dinv, p, c, d);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (pick(col, k) >= 0)
#pragma unroll
                for (int j = 0; j < NC; ++j) o[k][j] = ell_row<T>(off, N, p, k, c + j);
    }
    __device__ __forceinline__ void solve(const T* r, T* x, const bool is_held) const {
        T xr[NC];
        if (is_held) {
#pragma unroll
            for (int k = 0; k < NC; ++k) xr[k] = T(0);
            row_store<T, RT>(x, p, c, xr);
            return;
        }
        T s[NC];
        row_load<T, RT>(r, p, c, s);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int q = pick(col, k);
            if (q < 0) continue;
            T xo[4];
            ldt(reinterpret_cast<const typename B4<T>::type*>(x) + q, xo);
#pragma unroll
            for (int j = 0; j < NC; ++j) s[j] -= row_dot<T>(o[k][j], xo);
        }
        dinv_row<T, RT>(d, s, xr);
        row_store<T, RT>(x, p, c, xr);
    }
};

// One colour (rows c0 .. c0+n-1) of the sweep.  r = rbase + (*rk) * stride
// when rk is given (the current Krylov vector).
template <class T, int RT>
__global__ void __launch_bounds__(128) k_imp_gs(const Ell e, const int N, const T* __restrict__ dinv,
                                                const T* __restrict__ off, const int c0, const int n, const T* rbase,
                                                const int* rk, const long long stride, T* x, const int* stop,
                                                const int* __restrict__ case_done, const bool fwd) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = t < n * RT;
    GsRow<T, RT> row;
    if (in) {
        row.at(e, c0 + t / RT, (4 / RT) * (t % RT), fwd ? c0 : N);
        if (AHEAD<T, RT>) row.blocks(dinv, off, N);
    }
    pdl_wait();
    if (!in || (stop && ldw(stop))) return;
    if (!AHEAD<T, RT>) row.blocks(dinv, off, N);
    row.solve(rbase + (rk ? (long long)ldw(rk) * stride : 0), x, held(e.case_row, case_done, row.p));
}

// The top of the sweep in one block: the last colours of a greedy colouring
// hold a handful of rows (16k quadrilaterals: 6836, 6848, 2140, 554, 6), and
// each cost a launch on the way up and another on the way down.  Stage j does
// n[j] rows: c0[j], c0[j]+1, ... (forward), or list[c0[j]], ... (backward, fwd
// 0): on the way down only rows with a neighbour of a higher colour change, the
// others would be formed again unchanged.
constexpr int GS_TAIL = 6;
struct TailStages {
    int m;
    int c0[GS_TAIL], n[GS_TAIL], fwd[GS_TAIL];
};
template <class T>
__global__ void __launch_bounds__(1024) k_imp_gs_tail(const Ell e, const int N, const T* __restrict__ dinv,
                                                      const T* __restrict__ off, const TailStages st,
                                                      const int* __restrict__ list, const T* rbase, const int* rk,
                                                      const long long stride, T* x, const int* stop,
                                                      const int* __restrict__ case_done) {
    pdl_wait();
    if (stop && ldw(stop)) return;
    constexpr int RT = 4;
    const T* r = rbase + (rk ? (long long)ldw(rk) * stride : 0);
    for (int j = 0; j < st.m; ++j) {
        for (int t = threadIdx.x; t < RT * st.n[j]; t += blockDim.x) {
            const int i = st.c0[j] + t / RT, p = st.fwd[j] ? i : __ldg(&list[i]);
            GsRow<T, RT> row;
            row.at(e, p, t % RT, st.fwd[j] ? st.c0[j] : N);
            row.blocks(dinv, off, N);
            row.solve(r, x, held(e.case_row, case_done, p));
        }
        __syncthreads();  // the stage's rows are visible to the block
    }
}

// The start of Arnoldi step k: the second Gram-Schmidt update of the vector
// the previous step left, v_k = (w - sum_j h2_j v_j) * scale[0] over j < k (step
// 0: v_0 = w * scale[0]), and the first colour of the forward sweep,
// x_p = D_p^-1 v_p, over its n0 rows.  Basis vectors are read DOT_U at a time,
// all loads of a group before its arithmetic: one after the other each would
// wait out its own latency.
constexpr int DOT_U = 8;
static_assert((GM_M + 2) % DOT_U == 0, "whole groups");
template <class T, int RT>
__global__ void __launch_bounds__(128) k_imp_next_vec(const Ell e, const int n_rows, const T* __restrict__ dinv,
                                                      const int n0, const T* w, const double* h2, const double* scale,
                                                      T* vbase, const int* vk, T* x, const int* stop,
                                                      const int* __restrict__ case_done) {
    constexpr int NC = 4 / RT;
    __shared__ T hs[GM_M + 2];
    const int t = blockIdx.x * blockDim.x + threadIdx.x, p = t / RT, c = NC * (t % RT);
    Row<T> d[NC];
    if (p < n0) diag_rows<T, RT>(dinv, p, c, d);
    pdl_wait();
    if (ldw(stop)) return;
    const int k = ldw(vk);
    if (threadIdx.x < GM_M + 2) hs[threadIdx.x] = (int)threadIdx.x < k ? (T)ldw(&h2[threadIdx.x]) : T(0);
    __syncthreads();
    if (p >= n_rows) return;
    const T sc = (T)ldw(scale);
    T s[NC], xr[NC];
    row_load<T, RT>(w, p, c, s);
    for (int j0 = 0; j0 < k; j0 += DOT_U) {
        T v[DOT_U][NC];
#pragma unroll
        for (int u = 0; u < DOT_U; ++u) {
#pragma unroll
            for (int r = 0; r < NC; ++r) v[u][r] = T(0);
            if (j0 + u < k) row_load<T, RT>(vbase + (size_t)(j0 + u) * 4 * n_rows, p, c, v[u]);
        }
#pragma unroll
        for (int u = 0; u < DOT_U; ++u)
#pragma unroll
            for (int r = 0; r < NC; ++r) s[r] -= hs[j0 + u] * v[u][r];
    }
#pragma unroll
    for (int r = 0; r < NC; ++r) s[r] *= sc;
    row_store<T, RT>(vbase + (size_t)k * 4 * n_rows, p, c, s);
    if (p >= n0) return;
    dinv_row<T, RT>(d, s, xr);
    if (held(e.case_row, case_done, p)) {
#pragma unroll
        for (int r = 0; r < NC; ++r) xr[r] = T(0);
    }
    row_store<T, RT>(x, p, c, xr);
}

// Classical Gram-Schmidt twice against the Krylov basis v_0..v_{nv-1}
// (v_j = V + j*n), in three passes over it and two reductions:
//   k_imp_spmv_dots   w = M x, h1 = V^T w
//   k_imp_cgs         w -= V h1, h2 = V^T w and w.w
//   k_imp_next_vec    w -= V h2, scaled to v_{k+1}, by the next step
// The norm after the second update comes from Pythagoras, w.w - h2.h2 (the
// basis is orthonormal and h2 a rounding correction), so the second update
// needs no reduction of its own.  Where h2.h2 is more than half of w.w -- near
// a breakdown, the first update left mostly rounding -- the difference would
// lose digits, down to a zero that ends the solve as converged: there the last
// block forms the updated vector and its norm.  Up to a half the difference is
// good to five units of the vectors' rounding.
// The per-thread sums of all outputs are reduced across a warp together: a
// butterfly that halves the outputs a lane holds at every step takes 31 (16
// for up to 16 outputs) additions of a warp instead of 5 per output -- in
// FP64 each of them holds the FP64 pipe for 18.6 cycles, and this reduction
// was most of the kernel.  FP32 sums are added as unevaluated triples (error-free
// two-sums, 72 bits) on the FP32 lanes; double takes over after it.  Each block
// writes its partial sums; the last block to finish adds them in a fixed
// pattern (a warp per group of blocks, then over the warps), so the result is
// deterministic, and re-arms the counter.
// 16-byte chunks of a vector in T, their dot product and w -= h v
template <class T> struct Vec16;
template <> struct Vec16<float> { using type = float4; static constexpr int W = 4; };
template <> struct Vec16<double> { using type = double2; static constexpr int W = 2; };
__device__ __forceinline__ float vdot(const float4 a, const float4 b) {
    return ((a.x * b.x + a.y * b.y) + a.z * b.z) + a.w * b.w;
}
__device__ __forceinline__ double vdot(const double2 a, const double2 b) { return a.x * b.x + a.y * b.y; }
__device__ __forceinline__ void vsub(float4& w, const float h, const float4 v) {
    w.x -= h * v.x; w.y -= h * v.y; w.z -= h * v.z; w.w -= h * v.w;
}
__device__ __forceinline__ void vsub(double2& w, const double h, const double2 v) {
    w.x -= h * v.x; w.y -= h * v.y;
}

// Sums of acc[0..W-1] over the warp; lane j (mod W) gets output j
template <int W>
__device__ __forceinline__ double warp_sums(const double* acc, const int lane) {
    double a[W];
#pragma unroll
    for (int j = 0; j < W; ++j) a[j] = acc[j];
#pragma unroll
    for (int m = W / 2; m > 0; m >>= 1) {
        const bool up = lane & m;
#pragma unroll
        for (int j = 0; j < m; ++j) {
            const double give = up ? a[j] : a[j + m];
            a[j] = (up ? a[j + m] : a[j]) + __shfl_xor_sync(0xffffffffu, give, m);
        }
    }
#pragma unroll
    for (int m = W; m < 32; m <<= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], m);
    return a[0];
}
// Unevaluated sum h + m + l of FP32 numbers, level by level of the butterfly:
// two numbers give an exact pair, two pairs an exact triple but for 2^-72, and so
// on, so the sum of the warp has all the bits a double holds.
struct Triple {
    float h, m, l;
    __device__ __forceinline__ Triple from(const int lane_mask, const int level) const {
        Triple o;
        o.h = __shfl_xor_sync(0xffffffffu, h, lane_mask);
        o.m = level > 0 ? __shfl_xor_sync(0xffffffffu, m, lane_mask) : 0.f;
        o.l = level > 1 ? __shfl_xor_sync(0xffffffffu, l, lane_mask) : 0.f;
        return o;
    }
    __device__ __forceinline__ void add(const Triple& o, const int level) {
        float e, e1, e2;
        h = two_sum(h, o.h, e);
        if (level == 0) {
            m = e;
            return;
        }
        m = two_sum(m, o.m, e1);
        m = two_sum(m, e, e2);
        l = level > 1 ? (l + o.l) + (e1 + e2) : e1 + e2;
    }
};
template <int W>
__device__ __forceinline__ double warp_sums(const float* acc, const int lane) {
    // a double would hold any sum of these, so they are brought to the middle of
    // FP32's range if one could overflow, or if all are so small that the last
    // parts could underflow
    float mx = 0.f;
#pragma unroll
    for (int j = 0; j < W; ++j) mx = fmaxf(mx, fabsf(acc[j]));
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
    const float sc = mx > 0x1p122f ? 0x1p-6f : (mx < 0x1p-40f && mx > 0.f ? 0x1p100f : 1.f);
    Triple a[W];
#pragma unroll
    for (int j = 0; j < W; ++j) a[j] = Triple{acc[j], 0.f, 0.f};
    if (sc != 1.f) {
#pragma unroll
        for (int j = 0; j < W; ++j) a[j].h *= sc;
    }
    int level = 0;
#pragma unroll
    for (int m = W / 2; m > 0; m >>= 1, ++level) {
        const bool up = lane & m;
#pragma unroll
        for (int j = 0; j < m; ++j) {
            const Triple give = up ? a[j] : a[j + m];
            a[j] = up ? a[j + m] : a[j];
            a[j].add(give.from(m, level), level);
        }
    }
#pragma unroll
    for (int m = W; m < 32; m <<= 1, ++level) a[0].add(a[0].from(m, level), level);
    // (an infinity or a NaN among the summands: h alone is their sum)
    const double t = fabsf(a[0].h) <= 3.402823466e38f ? ((double)a[0].l + (double)a[0].m) + (double)a[0].h : (double)a[0].h;
    return sc == 1.f ? t : t * (sc < 1.f ? 0x1p6 : 0x1p-100);
}

// Arnoldi step j = c->k, classical Gram-Schmidt twice: h1 (first pass) and
// h2 (second pass) sum to column j, ww is the squared norm after the second.
// One warp, the earlier rotations staged in shared memory ahead of time
// (givens_stage), so the chain runs on shared memory, not on dependent global
// loads; then the new subdiagonal entry, its rotation and the residual
// estimate.
struct GivensCol {
    double col[GM_M + 2], cs[GM_M], sn[GM_M];
};
__device__ __forceinline__ void givens_stage(const GmresCtl* c, const double* h1, const int j, GivensCol& g) {
    const int t = threadIdx.x;
    if (t <= j) g.col[t] = ldw(&h1[t]);
    if (t < j) {
        g.cs[t] = ldw(&c->cs[t]);
        g.sn[t] = ldw(&c->sn[t]);
    }
}
__device__ __forceinline__ void givens(GmresCtl* c, const double h2, const double ww, GivensCol& g, double* scale) {
    using namespace fp64;
    const int lane = threadIdx.x, j = c->k;
    // ww: the squared norm after the second update; h2 in lanes 0..j
    if (lane <= j) g.col[lane] += h2;
    __syncwarp();
    if (lane == 0) {
        const double gj = c->g[j], tol = c->tol;
        const int iters = c->iters + 1, max_iters = c->max_iters;
        double a = g.col[0];
        for (int i = 0; i < j; ++i) {
            const double b = g.col[i + 1];
            g.col[i] = g.cs[i] * a + g.sn[i] * b;
            a = -g.sn[i] * a + g.cs[i] * b;
        }
        const double hn = root(fmax(ww, 0.0));
        c->hnext = hn;
        scale[0] = hn > 0 ? div(1.0, hn) : 0.0;
        const double b = hn, r = root(a * a + b * b);
        const Den ir = den(r);
        const double cj = r > 0 ? quot(a, ir) : 1.0, sj = r > 0 ? quot(b, ir) : 0.0;
        c->cs[j] = cj;
        c->sn[j] = sj;
        g.col[j] = r;
        g.col[j + 1] = 0;
        const double res = fabs(sj * gj);
        c->g[j + 1] = -sj * gj;
        c->g[j] = cj * gj;
        c->res = res;
        c->k = j + 1;
        c->iters = iters;
        const int st = (res <= tol || j + 1 == GM_M || hn == 0 || iters >= max_iters) ? 1 : 0;
        c->stop = st;
        if (c->graph) cudaGraphSetConditional(c->hin, st ? 0 : 1);
    }
    __syncwarp();
    for (int t = lane; t <= j + 1; t += 32) c->H[t + (GM_M + 1) * j] = g.col[t];
}

// The block's and, in the last block to finish, the whole sum of the threads'
// acc[0..nout-1] over the grid's blocks of NT threads; true in the last block's
// first nout threads, with the sums in `total`.
template <class T, int NT, bool ONE>
__device__ __forceinline__ bool grid_sums(const T* acc, const int nout, double* part, unsigned* counter,
                                          double& total) {
    const int blk = (int)blockIdx.x, nblk = (int)gridDim.x;
    constexpr int NW = NT / 32;
    __shared__ double sh[NW][32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    if (ONE) {
        const double v = warp_sums<1>(acc, lane);
        if (lane == 0) sh[wp][0] = v;
    } else if (nout > 16) {
        const double v = warp_sums<32>(acc, lane);
        if (lane < nout) sh[wp][lane] = v;
    } else {
        const double v = warp_sums<16>(acc, lane);
        if (lane < nout) sh[wp][lane] = v;
    }
    __syncthreads();
    if ((int)threadIdx.x < nout) {
        double t = 0;
#pragma unroll
        for (int k = 0; k < NW; ++k) t += sh[k][threadIdx.x];
        part[(size_t)blk * nout + threadIdx.x] = t;
        __threadfence();  // the partials are visible before the block is counted
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == (unsigned)nblk - 1;
    __syncthreads();
    if (!last) return false;
    __threadfence();
    // a warp reads the outputs of one block side by side; warp g takes blocks
    // g, g + NW, ... with eight loads in flight (one output: a block per thread)
    constexpr int U = 8;
    const int j = ONE ? 0 : lane, g = ONE ? (int)threadIdx.x : wp, st = ONE ? NT : NW;
    double t[U];
#pragma unroll
    for (int u = 0; u < U; ++u) t[u] = 0;
    if (j < nout)
        for (int b = g; b < nblk; b += U * st)
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (b + u * st < nblk) t[u] += __ldcg(&part[(size_t)(b + u * st) * nout + j]);
    double v = ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
    if (ONE) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) sh[wp][0] = v;
    } else {
        sh[wp][lane] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) *counter = 0;
    if ((int)threadIdx.x >= nout) return false;
    double sum = 0;
#pragma unroll
    for (int k = 0; k < NW; ++k) sum += sh[k][threadIdx.x];
    total = sum;
    return true;
}

// Squared norm of w - sum_j h2_j v_j by one block (thread j holds h2_j, hs is
// overwritten with them); for the threads of the first warp.  w as the whole
// grid has left it.  Rare: out of line.
template <class T>
__device__ __noinline__ double updated_norm(const int nc, const int nv, const typename Vec16<T>::type* V,
                                            const typename Vec16<T>::type* w, const double h2, T* hs) {
    __shared__ double sh[DOT_THREADS / 32];
    if ((int)threadIdx.x < nv) hs[threadIdx.x] = (T)h2;
    __syncthreads();
    T acc[1] = {0};
    for (int i = threadIdx.x; i < nc; i += blockDim.x) {
        typename Vec16<T>::type wi = __ldcg(&w[i]);
        for (int j = 0; j < nv; ++j) vsub(wi, hs[j], __ldcg(&V[(size_t)j * nc + i]));
        acc[0] += vdot(wi, wi);
    }
    const double v = warp_sums<1>(acc, threadIdx.x & 31);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0;
#pragma unroll
    for (int k = 0; k < DOT_THREADS / 32; ++k) t += sh[k];
    return t;
}

// w -= sum_j h1_j v_j, then h2_j = v_j . w and w.w, and in the last block the
// step's column.  A chunk of every vector stays in registers for the second
// product (one block per SM); the first chunk's are read ahead of the wait (the
// basis is complete before this kernel's predecessor started, as is *vk).
template <class T>
__global__ void __launch_bounds__(DOT_THREADS, 1) k_imp_cgs(const int n, const T* V, T* w, const double* h1,
                                                            double* part, unsigned* counter, double* h2, GmresCtl* c,
                                                            double* scale) {
    __shared__ T hs[GM_M + 2];
    __shared__ GivensCol gc;
    using VT = typename Vec16<T>::type;
    const int nc = n / Vec16<T>::W, nv = ldw(&c->k) + 1;
    const VT* Vv = reinterpret_cast<const VT*>(V);
    VT* wv = reinterpret_cast<VT*>(w);
    VT vv[GM_M + 1];
    auto basis = [&](const int i) {
#pragma unroll
        for (int j0 = 0; j0 <= GM_M; j0 += DOT_U)
            if (j0 < nv)
#pragma unroll
                for (int j = j0; j < j0 + DOT_U && j <= GM_M; ++j)
                    vv[j] = j < nv ? ldw(&Vv[(size_t)j * nc + i]) : VT();
    };
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 < nc) basis(i0);
    pdl_wait();
    if (ldw(&c->stop)) {  // a step launched after the cycle's end
        if (c->graph && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(c->hin, 0);
        return;
    }
    if (threadIdx.x < GM_M + 2) hs[threadIdx.x] = (int)threadIdx.x < nv ? (T)ldw(&h1[threadIdx.x]) : T(0);
    if (threadIdx.x < 32) givens_stage(c, h1, nv - 1, gc);
    __syncthreads();
    // per-thread partial sums in T over 16-byte chunks of the vectors (a few
    // chunks each; n is 4 * cells, so whole chunks)
    T acc[GM_M + 2], sq = 0;
#pragma unroll
    for (int j = 0; j < GM_M + 2; ++j) acc[j] = 0;
    for (int i = i0; i < nc; i += gridDim.x * blockDim.x) {
        VT wi = ldw(&wv[i]);
        if (i != i0) basis(i);
#pragma unroll
        for (int j0 = 0; j0 <= GM_M; j0 += DOT_U)
            if (j0 < nv)
#pragma unroll
                for (int j = j0; j < j0 + DOT_U && j <= GM_M; ++j) vsub(wi, hs[j], vv[j]);
        wv[i] = wi;
        sq += vdot(wi, wi);
#pragma unroll
        for (int j0 = 0; j0 <= GM_M; j0 += DOT_U)
            if (j0 < nv)
#pragma unroll
                for (int j = j0; j < j0 + DOT_U && j <= GM_M; ++j) acc[j] += vdot(vv[j], wi);
    }
    // output nv (at most GM_M) is w.w
#pragma unroll
    for (int j = 1; j < GM_M + 2; ++j)
        if (j == nv) acc[j] = sq;
    double t = 0;
    const bool mine = grid_sums<T, DOT_THREADS, false>(acc, nv + 1, part, counter, t);
    if (!__syncthreads_or(mine)) return;
    __shared__ bool direct;
    double hh = 0, ww = 0;
    if (threadIdx.x < 32) {
        hh = (int)threadIdx.x < nv ? t * t : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) hh += __shfl_xor_sync(0xffffffffu, hh, o);
        ww = __shfl_sync(0xffffffffu, t, nv);
        if ((int)threadIdx.x < nv) h2[threadIdx.x] = t;
        if (threadIdx.x == 0) direct = !(2.0 * hh <= ww);
    }
    __syncthreads();
    if (direct) ww = updated_norm<T>(nc, nv, Vv, wv, t, hs);
    else ww -= hh;
    if (threadIdx.x < 32) givens(c, t, ww, gc, scale);
}

// out = w.w
template <class T>
__global__ void __launch_bounds__(DOT_THREADS) k_imp_sq(const int n, const T* w, double* part, unsigned* counter,
                                                        double* out, const int* stop) {
    pdl_wait();
    if (stop && ldw(stop)) return;
    using VT = typename Vec16<T>::type;
    const VT* wv = reinterpret_cast<const VT*>(w);
    T acc[1] = {0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n / Vec16<T>::W; i += gridDim.x * blockDim.x) {
        const VT wi = ldw(&wv[i]);
        acc[0] += vdot(wi, wi);
    }
    double t;
    if (grid_sums<T, DOT_THREADS, true>(acc, 1, part, counter, t)) out[0] = t;
}

// w = M x and out_j = v_j . w, j <= *vk, in one pass over the rows: the
// product's row is in registers when the basis is read, and one launch and one
// pass over w less per Arnoldi step.
template <class T, int RT>
__global__ void __launch_bounds__(DOT_THREADS, 2)
    k_imp_spmv_dots(const int n_rows, const Ell e, const T* __restrict__ dblk, const T* __restrict__ off, const T* x,
                    T* w, const int* vk, const T* V, double* part, unsigned* counter, double* out, const int* stop,
                    const int* __restrict__ case_done) {
    constexpr int NC = 4 / RT;
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    int4 col = make_int4(-1, -1, -1, -1);
    Row<T> d[NC];
    if (t0 < RT * (long long)n_rows) {
        const int p = (int)(t0 / RT), c = NC * (int)(t0 % RT);
        col = __ldg(&e.col[p]);
        diag_rows<T, RT>(dblk, p, c, d);
    }
    pdl_wait();
    if (ldw(stop)) return;
    const int nv = ldw(vk) + 1;
    T acc[GM_M + 2];
#pragma unroll
    for (int j = 0; j < GM_M + 2; ++j) acc[j] = 0;
    for (long long t = t0; t < RT * (long long)n_rows; t += (long long)gridDim.x * blockDim.x) {
        const int p = (int)(t / RT), c = NC * (int)(t % RT);
        if (t != t0) {
            col = __ldg(&e.col[p]);
            diag_rows<T, RT>(dblk, p, c, d);
        }
        T y[NC];
#pragma unroll
        for (int r = 0; r < NC; ++r) y[r] = T(0);
        if (!held(e.case_row, case_done, p)) spmv_row<T, RT>(n_rows, col, d, off, x, p, c, y);
        row_store<T, RT>(w, p, c, y);
#pragma unroll
        for (int j0 = 0; j0 <= GM_M; j0 += DOT_U)
            if (j0 < nv) {
                T v[DOT_U][NC];
#pragma unroll
                for (int u = 0; u < DOT_U; ++u) {
#pragma unroll
                    for (int r = 0; r < NC; ++r) v[u][r] = T(0);
                    if (j0 + u < nv) row_load<T, RT>(V + (size_t)(j0 + u) * 4 * n_rows, p, c, v[u]);
                }
#pragma unroll
                for (int u = 0; u < DOT_U; ++u) {
                    if constexpr (NC == 1) acc[j0 + u] += v[u][0] * y[0];
                    else acc[j0 + u] += ((v[u][0] * y[0] + v[u][1] * y[1]) + v[u][2] * y[2]) + v[u][3] * y[3];
                }
            }
    }
    double s;
    if (grid_sums<T, DOT_THREADS, false>(acc, nv, part, counter, s)) out[threadIdx.x] = s;
}

// Back substitution R y = g over the k steps of the cycle: one warp, a lane
// per unknown, each solved unknown's column taken off the lanes that still
// wait (the triangle is staged in shared memory).
__global__ void __launch_bounds__(32) k_imp_solve_y(GmresCtl* c) {
    __shared__ double R[GM_M * GM_M];
    const int k = c->k, i = threadIdx.x;
    for (int t = i; t < k * k; t += 32) {
        const int r = t % k, l = t / k;
        R[r + GM_M * l] = c->H[r + (GM_M + 1) * l];
    }
    double g = i < k ? c->g[i] : 0.0;
    __syncwarp();
    const double d = i < k ? R[i + GM_M * i] : 0.0;
    const double inv = d != 0 ? 1.0 / d : 0.0;
    for (int l = k - 1; l >= 0; --l) {
        if (i == l) {  // g / d: the product with 1/d and one correction
            const double y = g * inv;
            g = fma(fma(-y, d, g), inv, y);
        }
        const double yl = __shfl_sync(0xffffffffu, g, l);
        if (i < l) g -= R[i + GM_M * l] * yl;
    }
    if (i < k) c->y[i] = g;
}

// t = sum_j y_j v_j over the k steps
template <class T>
__global__ void __launch_bounds__(256) k_imp_lincomb(const int n, const T* __restrict__ V, const GmresCtl* __restrict__ c,
                                                     T* __restrict__ t) {
    __shared__ T ys[GM_M];
    const int k = c->k;
    if ((int)threadIdx.x < k) ys[threadIdx.x] = (T)c->y[threadIdx.x];
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    T s = 0;
    for (int j = 0; j < k; ++j) s += ys[j] * V[(size_t)j * n + i];
    t[i] = s;
}

// x (double) += z;  r = b - y  (b double), both 4N long
template <class T>
__global__ void __launch_bounds__(256) k_imp_addx(const int n, const T* __restrict__ z, double* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] += (double)z[i];
}
// r = b - y, b in device cell order, r and y in row order (4N long)
template <class T>
__global__ void __launch_bounds__(256) k_imp_resid(const int n, const double* __restrict__ b,
                                                   const int* __restrict__ perm, const T* __restrict__ y,
                                                   T* __restrict__ r, const int* __restrict__ stop) {
    if (stop && *stop) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) r[i] = (T)(b[4 * (size_t)__ldg(&perm[i >> 2]) + (i & 3)] - (double)y[i]);
}
// t = b in row order (b in device cell order)
template <class T>
__global__ void __launch_bounds__(256) k_imp_gather_b(const int n, const double* __restrict__ b,
                                                      const int* __restrict__ perm, T* __restrict__ t) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) t[i] = (T)b[4 * (size_t)__ldg(&perm[i >> 2]) + (i & 3)];
}
template <class T>
__global__ void __launch_bounds__(256) k_imp_cast(const int n, const double* __restrict__ x, T* __restrict__ t,
                                                  const int* __restrict__ stop) {
    if (stop && *stop) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) t[i] = (T)x[i];
}

// q += relax * dq over the real cells; dq also becomes qW (the reference's
// qW holds the last linear solution, read by get_uniform_residual)
// (dq in row order, q and qW in device cell order)
__global__ void __launch_bounds__(256) k_imp_update(const int n, const double* __restrict__ dq,
                                                    const int* __restrict__ perm, const double relax,
                                                    double* __restrict__ q, double* __restrict__ qW) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t j = 4 * (size_t)__ldg(&perm[i >> 2]) + (i & 3);
    q[j] += dq[i] * relax;
    qW[j] = dq[i];
}

// case of each row (batch)
__global__ void k_imp_case_rows(const int n, const int* __restrict__ perm, const int* __restrict__ case_of,
                                int* __restrict__ case_row) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) case_row[p] = case_of[perm[p]];
}

// GMRES initialisation of a cycle: g = (beta, 0, ...), stop = beta <= tol
__global__ void k_imp_cycle_init(GmresCtl* c, const double* __restrict__ rr, double* __restrict__ scale, const int first,
                                 const double rel_tol, const int max_iters) {
    if (!first && c->halt) return;
    const double beta = sqrt(fmax(rr[0], 0.0));
    if (first) {
        c->tol = rel_tol * beta;
        c->iters = 0;
        c->max_iters = max_iters;
    }
    for (int i = 0; i <= GM_M; ++i) c->g[i] = 0;
    c->g[0] = beta;
    c->res = beta;
    c->k = 0;
    c->stop = (beta <= c->tol) ? 1 : 0;
    c->halt = c->stop;
    scale[0] = beta > 0 ? 1.0 / beta : 0.0;
    if (first && c->graph) cudaGraphSetConditional(c->hout, c->stop ? 0 : 1);
}

// Start of a restart cycle (inside the restart loop's body): enter the
// Arnoldi loop unless the cycle is already converged
__global__ void k_imp_enter(GmresCtl* c) {
    if (c->graph) cudaGraphSetConditional(c->hin, c->stop ? 0 : 1);
}

// End of a restart cycle: another one if not converged and under the limit
__global__ void k_imp_outer_check(GmresCtl* c) {
    const int cont = (c->res > c->tol) && (c->iters < c->max_iters) && (c->k > 0);
    c->halt = cont ? 0 : 1;
    if (c->graph) cudaGraphSetConditional(c->hout, cont ? 1 : 0);
}

// ------------------------------------------------------------ adjoint
// M -> M^T in place: row p, slot s takes (O_qp)^T from the copy `src` of the
// off-diagonal blocks; the diagonal block and its ILU(0) inverse are
// transposed in their row.  The transposed inverses are exactly the ILU(0)
// factors of M^T in the same colour order (D~' = D~^T by induction over
// the colours), so the Gauss-Seidel sweep then applies P^T.
template <class T>
__global__ void __launch_bounds__(128) k_imp_transpose(const int N, const Ell e, const T* __restrict__ src,
                                                       T* __restrict__ off, T* __restrict__ dblk,
                                                       T* __restrict__ dinv) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= N) return;
    const int4 col = __ldg(&e.col[p]);
    const int4 tr = __ldg(&e.tr[p]);
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
        if (pick(col, s) < 0) continue;
        const int t2 = pick(tr, s);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) off[ell_at<T>(N, p, s, 4 * r + c)] = src[ell_at<T>(N, t2 >> 2, t2 & 3, 4 * c + r)];
    }
    T* D = dblk + 16 * (size_t)p;
    T* I = dinv + 16 * (size_t)p;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = r + 1; c < 4; ++c) {
            T t = D[4 * r + c];
            D[4 * r + c] = D[4 * c + r];
            D[4 * c + r] = t;
            t = I[4 * r + c];
            I[4 * r + c] = I[4 * c + r];
            I[4 * c + r] = t;
        }
}

}  // namespace dev

// ----------------------------------------------------------------- host
namespace {

inline int nb_(long long n, int b) { return (int)((n + b - 1) / b); }

}  // namespace

struct ImplicitEngine {
    bool f32 = false;
    bool graph = true;  // GMRES as one graph with device-side loops, else a host loop
    int N = 0, F = 0, n4 = 0;
    int n_colors = 0;
    std::vector<int> color_ptr;
    void* jf = nullptr;    // face Jacobians J, K (16 T each)
    void* dblk = nullptr;  // diagonal block of each row
    void* dinv = nullptr;  // its ILU(0) inverse
    void* off = nullptr;   // off-diagonal blocks, 4 slots per row
    int* perm = nullptr;   // device cell of each row (rows grouped by colour)
    int4* ell_col = nullptr;
    int4* ell_face = nullptr;
    int4* ell_tr = nullptr;
    int* case_row = nullptr;          // batch: case of each row
    const int* case_row_src = nullptr;  // the case_of it was formed from
    int* singular = nullptr;
    void* V = nullptr;     // (GM_M+1) x 4N
    void* w = nullptr;     // 4N
    void* z = nullptr;     // 4N
    void* t = nullptr;     // 4N
    double* x = nullptr;   // 4N, the solution dQ
    double* part = nullptr;
    unsigned* counter = nullptr;  // last-block counter of the dot kernel
    double* small = nullptr;  // h1[GM_M+1], h2[GM_M+1], ww, scale
    cudaGraphExec_t cyc[2] = {nullptr, nullptr};  // cyc[0]: the GMRES solve graph
    cudaStream_t s2 = nullptr, s3 = nullptr;      // capture streams of the loop bodies
    const void* cyc_b = nullptr;                  // right-hand side the graphs were captured with
    int nbd = 0, nbd1 = 0;  // blocks of the dot passes (two / one per SM)
    // the top of the sweep as one launch (k_imp_gs_tail): up from colour tail0,
    // down to colour tail_down; rows of a backward stage in blist
    int tail0 = 0, tail_down = 0;
    dev::TailStages tail{};
    int* blist = nullptr;
    dev::GmresCtl* ctl = nullptr;
    dev::GmresCtl* h_ctl = nullptr;
    int last_iters = 0;

    size_t ts() const { return f32 ? 4 : 8; }
    dev::Ell ell() const { return dev::Ell{perm, ell_col, ell_face, ell_tr, case_row}; }
};

void implicit_destroy(ImplicitEngine* e);

// cslot, cnbr: the host copies of the cell slots (4 per cell, device order)
ImplicitEngine* implicit_create(const StepArgs& a, bool f32, bool graph, const std::vector<int>& colors,
                                const int* cslot, const int* cnbr, cudaStream_t s) {
    // freed again if any step below throws
    std::unique_ptr<ImplicitEngine, void (*)(ImplicitEngine*)> guard(new ImplicitEngine(), implicit_destroy);
    ImplicitEngine* e = guard.get();
    e->f32 = f32;
    e->graph = graph;
    e->N = a.n_cells;
    e->F = a.n_faces;
    e->n4 = 4 * a.n_cells;
    const int N = e->N;
    int nc = 0;
    for (int c : colors) nc = std::max(nc, c + 1);
    e->n_colors = nc;
    e->color_ptr.assign(nc + 1, 0);
    for (int c : colors) e->color_ptr[c + 1]++;
    for (int c = 0; c < nc; ++c) e->color_ptr[c + 1] += e->color_ptr[c];
    // rows: the cells of colour 0, then colour 1, ..., each in device order
    std::vector<int> perm(N), rowof(N), fill(e->color_ptr.begin(), e->color_ptr.end() - 1);
    for (int i = 0; i < N; ++i) perm[fill[colors[i]]++] = i;
    for (int p = 0; p < N; ++p) rowof[perm[p]] = p;
    std::vector<int> ecol(4 * (size_t)N, -1), eface(4 * (size_t)N, 0), etr(4 * (size_t)N, -1);
    for (int p = 0; p < N; ++p) {
        const int i = perm[p];
        for (int k = 0; k < 4; ++k) {
            const int fs = cslot[4 * (size_t)i + k], o = cnbr[4 * (size_t)i + k];
            eface[4 * (size_t)p + k] = fs;
            if (fs != 0 && o >= 0) ecol[4 * (size_t)p + k] = rowof[o];
        }
    }
    for (int p = 0; p < N; ++p)
        for (int k = 0; k < 4; ++k) {
            const int q = ecol[4 * (size_t)p + k];
            if (q < 0) continue;
            const int f = std::abs(eface[4 * (size_t)p + k]);
            for (int k2 = 0; k2 < 4; ++k2)
                if (std::abs(eface[4 * (size_t)q + k2]) == f) etr[4 * (size_t)p + k] = 4 * q + k2;
            if (etr[4 * (size_t)p + k] < 0) throw Error(7, "implicit solver: face slots are not symmetric");
        }
    // the sweep's top: forward stages of the last colours, then backward ones
    // over the rows with a neighbour of a higher colour, as long as one block
    // does them faster than the launches they save.  In FP64 one SM's two lanes
    // need 1.5 us for 64 rows (with 600 rows in the tail a step at 16k rows
    // took 12 us longer); in FP32 a tail of 640 rows in dependent stages is
    // slower than its launches too (six iterations at 16k rows 106.6 ms, 97.7
    // with 64 and with 200; 201k rows, Spalart-Allmaras, 12.5 against 12.2 ms)
    const int TAIL_ROWS = 64;
    std::vector<int> blist;
    auto higher = [&](int c) {
        std::vector<int> rows;
        for (int p = e->color_ptr[c]; p < e->color_ptr[c + 1]; ++p)
            for (int k = 0; k < 4; ++k)
                if (ecol[4 * (size_t)p + k] >= e->color_ptr[c + 1]) {
                    rows.push_back(p);
                    break;
                }
        return rows;
    };
    int budget = TAIL_ROWS, t0 = nc;
    while (t0 > 1 && nc - t0 < dev::GS_TAIL / 2 && e->color_ptr[t0] - e->color_ptr[t0 - 1] <= budget) {
        --t0;
        budget -= e->color_ptr[t0 + 1] - e->color_ptr[t0];
    }
    e->tail0 = t0;
    e->tail_down = nc - 1;
    if (t0 < nc) {
        for (int c = t0; c < nc; ++c) {
            const int k = e->tail.m++;
            e->tail.c0[k] = e->color_ptr[c];
            e->tail.n[k] = e->color_ptr[c + 1] - e->color_ptr[c];
            e->tail.fwd[k] = 1;
        }
        for (int c = nc - 2; c >= std::max(t0 - 1, 0) && e->tail.m < dev::GS_TAIL; --c) {
            const std::vector<int> rows = higher(c);
            if ((int)rows.size() > budget) break;
            budget -= (int)rows.size();
            const int k = e->tail.m++;
            e->tail.c0[k] = (int)blist.size();
            e->tail.n[k] = (int)rows.size();
            e->tail.fwd[k] = 0;
            blist.insert(blist.end(), rows.begin(), rows.end());
            e->tail_down = c;
        }
        if (e->tail.m < 2) {  // nothing saved
            e->tail.m = 0;
            e->tail0 = nc;
            e->tail_down = nc - 1;
        }
    }
    const size_t T = e->ts();
    auto chk = [](cudaError_t r) {
        if (r != cudaSuccess) throw Error(7, std::string("implicit solver: ") + cudaGetErrorString(r));
    };
    const size_t N1 = std::max(N, 1);
    chk(cudaMalloc(&e->jf, (size_t)e->F * 32 * T));
    chk(cudaMalloc(&e->dblk, N1 * 16 * T));
    chk(cudaMalloc(&e->dinv, N1 * 16 * T));
    chk(cudaMalloc(&e->off, N1 * 64 * T));
    chk(cudaMalloc((void**)&e->perm, N1 * sizeof(int)));
    chk(cudaMalloc((void**)&e->ell_col, N1 * sizeof(int4)));
    chk(cudaMalloc((void**)&e->ell_face, N1 * sizeof(int4)));
    chk(cudaMalloc((void**)&e->ell_tr, N1 * sizeof(int4)));
    chk(cudaMalloc((void**)&e->blist, std::max<size_t>(blist.size(), 1) * sizeof(int)));
    chk(cudaMemcpyAsync(e->blist, blist.data(), blist.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    chk(cudaMalloc((void**)&e->singular, sizeof(int)));
    chk(cudaMalloc(&e->V, (size_t)(dev::GM_M + 1) * e->n4 * T));
    chk(cudaMalloc(&e->w, (size_t)e->n4 * T));
    chk(cudaMalloc(&e->z, (size_t)e->n4 * T));
    chk(cudaMalloc(&e->t, (size_t)e->n4 * T));
    chk(cudaMalloc((void**)&e->x, (size_t)e->n4 * 8));
    int dev_id = 0, sms = 0;
    cudaGetDevice(&dev_id);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev_id);
    // one 16-byte chunk per thread until every SM holds two blocks (more would
    // leave the last block too many partial sums); a system of 16k rows in
    // FP64 ran on 64 blocks with two chunks per thread before
    const int chunks = (int)(((size_t)e->n4 * e->ts()) / 16);
    e->nbd = std::max(1, std::min(2 * std::max(sms, 1), nb_(chunks, dev::DOT_THREADS)));
    e->nbd1 = std::max(1, std::min(std::max(sms, 1), e->nbd));
    chk(cudaMalloc((void**)&e->part, (size_t)e->nbd * (dev::GM_M + 1) * 8));
    chk(cudaMalloc((void**)&e->small, (2 * (dev::GM_M + 1) + 2) * 8));
    chk(cudaMalloc((void**)&e->counter, sizeof(unsigned)));
    chk(cudaMemsetAsync(e->counter, 0, sizeof(unsigned), s));
    chk(cudaMalloc((void**)&e->ctl, sizeof(dev::GmresCtl)));
    chk(cudaHostAlloc((void**)&e->h_ctl, sizeof(dev::GmresCtl), cudaHostAllocDefault));
    chk(cudaMemcpyAsync(e->perm, perm.data(), (size_t)N * sizeof(int), cudaMemcpyHostToDevice, s));
    chk(cudaMemcpyAsync(e->ell_col, ecol.data(), (size_t)N * sizeof(int4), cudaMemcpyHostToDevice, s));
    chk(cudaMemcpyAsync(e->ell_face, eface.data(), (size_t)N * sizeof(int4), cudaMemcpyHostToDevice, s));
    chk(cudaMemcpyAsync(e->ell_tr, etr.data(), (size_t)N * sizeof(int4), cudaMemcpyHostToDevice, s));
    chk(cudaMemsetAsync(e->jf, 0, (size_t)e->F * 32 * T, s));
    chk(cudaMemsetAsync(e->off, 0, N1 * 64 * T, s));
    e->h_ctl->graph = graph ? 1 : 0;
    chk(cudaMemcpyAsync(&e->ctl->graph, &e->h_ctl->graph, sizeof(int), cudaMemcpyHostToDevice, s));
    chk(cudaStreamSynchronize(s));
    return guard.release();
}

void implicit_destroy(ImplicitEngine* e) {
    if (!e) return;
    for (int k = 0; k < 2; ++k)
        if (e->cyc[k]) cudaGraphExecDestroy(e->cyc[k]);
    if (e->s2) cudaStreamDestroy(e->s2);
    if (e->s3) cudaStreamDestroy(e->s3);
    for (void* p : {e->jf, e->dblk, e->dinv, e->off, (void*)e->perm, (void*)e->ell_col, (void*)e->ell_face,
                    (void*)e->ell_tr, (void*)e->blist, (void*)e->case_row, (void*)e->singular, e->V, e->w, e->z, e->t, (void*)e->x,
                    (void*)e->part, (void*)e->small, (void*)e->ctl, (void*)e->counter})
        if (p) cudaFree(p);
    if (e->h_ctl) cudaFreeHost(e->h_ctl);
    delete e;
}

// fillRhoLHS (solver.h:1016-1090): dt from the state of parity p at the CFL
// in a.cfl, face Jacobians, diagonal blocks and their inverses.
namespace {
template <class T>
void fill_t(ImplicitEngine* e, const StepArgs& a, const dev::KM<double>& m, const dev::d4* q, cudaStream_t s) {
    using namespace dev;
    const int nf = nb_(a.n_faces, 128), nc = nb_(a.n_cells, 128);
    if (a.visc == 1)
        k_imp_jac<T, 1><<<nf, 128, 0, s>>>(m, a.n_faces, q, (const d4*)a.gx, (const d4*)a.gy, (T*)e->jf, a.ctrl);
    else if (a.visc == 2)
        k_imp_jac<T, 2><<<nf, 128, 0, s>>>(m, a.n_faces, q, (const d4*)a.gx, (const d4*)a.gy, (T*)e->jf, a.ctrl);
    else
        k_imp_jac<T, 0><<<nf, 128, 0, s>>>(m, a.n_faces, q, (const d4*)a.gx, (const d4*)a.gy, (T*)e->jf, a.ctrl);
    const Ell el = e->ell();
    k_imp_assemble<T><<<nc, 128, 0, s>>>(m, el, (const double*)a.dt, (const T*)e->jf, (T*)e->dblk, (T*)e->dinv,
                                         (T*)e->off, e->singular, a.ctrl, a.case_done, a.cctrl);
    for (int c = 1; c < e->n_colors; ++c) {
        const int c0 = e->color_ptr[c], cn = e->color_ptr[c + 1] - c0;
        if (cn > 0)
            k_imp_ilu<T><<<nb_(cn, 128), 128, 0, s>>>(el, e->N, (const T*)e->dblk, (const T*)e->off, c0, cn,
                                                      (T*)e->dinv, e->singular, a.case_done, a.cctrl, a.ctrl);
    }
}
}  // namespace

void implicit_fill(ImplicitEngine* e, const StepArgs& a0, int p, cudaStream_t s) {
    using namespace dev;
    StepArgs a = a0;
    a.variant = 0;  // the prep that also forms dt
    a.second = 0;   // gradients only when viscous (solver.h:1023-1026)
    a.need_grad = a.visc >= 1 ? 1 : 0;
    if (a.case_of && e->case_row_src != a.case_of) {
        // a batch: the case of each row, formed once
        if (!e->case_row && cudaMalloc((void**)&e->case_row, (size_t)std::max(e->N, 1) * sizeof(int)) != cudaSuccess)
            throw Error(7, "implicit solver: out of device memory");
        k_imp_case_rows<<<nb_(e->N, 256), 256, 0, s>>>(e->N, e->perm, a.case_of, e->case_row);
        e->case_row_src = a.case_of;
    }
    const KM<double> m = make_km<double>(a);
    launch_prep<double, double>(a, m, (const d4*)a.qm[p], s);
    cudaMemsetAsync(e->singular, 0, sizeof(int), s);
    const d4* q = (const d4*)a.qm[p];
    if (e->f32) fill_t<float>(e, a, m, q, s);
    else fill_t<double>(e, a, m, q, s);
}

namespace {

template <class T>
struct Ops {
    ImplicitEngine* e;
    const StepArgs& a;
    cudaStream_t s;
    dev::KM<double> m;
    Ops(ImplicitEngine* e_, const StepArgs& a_, cudaStream_t s_) : e(e_), a(a_), s(s_), m(dev::make_km<double>(a_)) {}
    T* vec(int j) const { return (T*)e->V + (size_t)j * e->n4; }
    int* stop() const { return &e->ctl->stop; }
    void spmv(const T* x, T* y, const int* st) const {
        launch_pdl(dev::k_imp_spmv<T>, nb_(e->N, 256), 256, 0, s, e->N, e->ell(), (const T*)e->dblk, (const T*)e->off, x,
                   y, st, a.case_done);
    }
    // t = b in row order
    void gather_b(const double* b, T* t) const {
        dev::k_imp_gather_b<T><<<nb_(e->n4, 256), 256, 0, s>>>(e->n4, b, e->perm, t);
    }
    // four threads per row for a launch over n rows?
    // (measured, whole implicit iteration: FP64 16k rows 60.3 ms with one thread
    // per row always, 44.9 ms with four; FP32 131k rows 17.6 ms with one always,
    // 19.4 ms with four always, 16.9 ms with four below 40,000 rows)
    static bool four(long long n) { return n < 40000; }
    // one symmetric multicolour block Gauss-Seidel sweep from x = 0 (the
    // ILU(0) factors in the colour ordering); the input is r, or the current
    // Krylov vector V + k*n when rk is given.  The forward sweep forms every
    // cell (reading lower colours only) from colour `first` on; the backward
    // sweep skips the top colour, whose value it would form again unchanged.
    // The sweep's top, from colour e->tail0 up and down again, is one launch.
    void precond(const T* r, const int* rk, T* x, const int* st, int first = 0) const {
        auto colour = [&](int c, bool fwd) {
            const int c0 = e->color_ptr[c], cn = e->color_ptr[c + 1] - c0;
            if (cn == 0) return;
            if (four(cn))
                launch_pdl(dev::k_imp_gs<T, 4>, nb_(4LL * cn, 128), 128, 0, s, e->ell(), e->N, (const T*)e->dinv,
                           (const T*)e->off, c0, cn, r, rk, (long long)e->n4, x, st, a.case_done, fwd);
            else
                launch_pdl(dev::k_imp_gs<T, 1>, nb_(cn, 128), 128, 0, s, e->ell(), e->N, (const T*)e->dinv,
                           (const T*)e->off, c0, cn, r, rk, (long long)e->n4, x, st, a.case_done, fwd);
        };
        const int C = e->n_colors, t0 = std::max(e->tail0, first);
        const bool tail = e->tail.m > 0 && t0 == e->tail0;
        for (int c = first; c < (tail ? t0 : C); ++c) colour(c, true);
        if (tail)
            launch_pdl(dev::k_imp_gs_tail<T>, 1, 1024, 0, s, e->ell(), e->N, (const T*)e->dinv, (const T*)e->off,
                       e->tail, e->blist, r, rk, (long long)e->n4, x, st, a.case_done);
        for (int c = (tail ? e->tail_down : C - 1) - 1; c >= 0; --c) colour(c, false);
    }
    // out = w.w
    void norm2(const T* w, double* out, const int* st) const {
        launch_pdl(dev::k_imp_sq<T>, e->nbd, dev::DOT_THREADS, 0, s, e->n4, w, e->part, e->counter, out, st);
    }
    // Arnoldi step k: v_k from the vector the last step left, z = P^-1 v_k,
    // w = M z, CGS2 against v_0..v_k, column k of the Hessenberg matrix
    void arnoldi_step(T* V, T* w, T* z, double* h1, double* h2, double* sc, const int* k, const int* st) const {
        if (four(e->N)) {
            launch_pdl(dev::k_imp_next_vec<T, 4>, nb_(e->n4, 128), 128, 0, s, e->ell(), e->N, (const T*)e->dinv,
                       e->color_ptr[1], w, h2, sc, V, k, z, st, a.case_done);
            precond(V, k, z, st, 1);
            launch_pdl(dev::k_imp_spmv_dots<T, 4>, e->nbd, dev::DOT_THREADS, 0, s, e->N, e->ell(), (const T*)e->dblk,
                       (const T*)e->off, z, w, k, V, e->part, e->counter, h1, st, a.case_done);
        } else {
            launch_pdl(dev::k_imp_next_vec<T, 1>, nb_(e->N, 128), 128, 0, s, e->ell(), e->N, (const T*)e->dinv,
                       e->color_ptr[1], w, h2, sc, V, k, z, st, a.case_done);
            precond(V, k, z, st, 1);
            launch_pdl(dev::k_imp_spmv_dots<T, 1>, e->nbd, dev::DOT_THREADS, 0, s, e->N, e->ell(), (const T*)e->dblk,
                       (const T*)e->off, z, w, k, V, e->part, e->counter, h1, st, a.case_done);
        }
        launch_pdl(dev::k_imp_cgs<T>, e->nbd1, dev::DOT_THREADS, 0, s, e->n4, V, w, h1, e->part, e->counter, h2,
                   e->ctl, sc);
    }
};

// Adds a WHILE node at the capture position of stream st (the work captured
// next on st follows the loop) and returns its body graph.
cudaGraph_t add_while(cudaStream_t st, cudaGraphConditionalHandle* h) {
    cudaStreamCaptureStatus cs;
    cudaGraph_t g;
    const cudaGraphNode_t* deps = nullptr;
    const cudaGraphEdgeData* ed = nullptr;
    size_t nd = 0;
    auto chk = [](cudaError_t r) {
        if (r != cudaSuccess) throw Error(7, std::string("implicit solver graph: ") + cudaGetErrorString(r));
    };
    chk(cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, &ed, &nd));
    chk(cudaGraphConditionalHandleCreate(h, g, 0, cudaGraphCondAssignDefault));
    cudaGraphNodeParams p{};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = *h;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    chk(cudaGraphAddNode(&node, g, deps, ed, nd, &p));
    chk(cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
    return p.conditional.phGraph_out[0];
}

// The whole GMRES solve of M dQ = b as one graph: restart cycles and Arnoldi
// steps are WHILE loops whose conditions the kernels set on the device, so
// a solve runs without host round trips and without idle launches.
template <class T>
cudaGraphExec_t build_gmres_graph(ImplicitEngine* e, const Ops<T>& o0, const double* b, cudaStream_t s,
                                  cudaStream_t s2, cudaStream_t s3, int max_iters) {
    using namespace dev;
    const int n = e->n4;
    double* h1 = e->small;
    double* h2 = e->small + (GM_M + 1);
    double* ww = e->small + 2 * (GM_M + 1);
    double* scale = ww + 1;
    int* kptr = &e->ctl->k;
    int* stop = &e->ctl->stop;
    int* halt = &e->ctl->halt;
    auto chk = [](cudaError_t r) {
        if (r != cudaSuccess) throw Error(7, std::string("implicit solver graph: ") + cudaGetErrorString(r));
    };
    cudaGraphConditionalHandle hout, hin;
    // main graph: first cycle set-up, the restart loop, the control block back to the host
    chk(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    Ops<T> o(e, o0.a, s);
    T* w = (T*)e->w;  // the vector that becomes v_0 (scaled by the first Arnoldi step)
    cudaMemsetAsync(e->x, 0, (size_t)n * 8, s);
    o.gather_b(b, w);
    o.norm2(w, ww, nullptr);
    k_imp_cycle_init<<<1, 1, 0, s>>>(e->ctl, ww, scale, 1, 1e-2, max_iters);
    cudaGraph_t body_out = add_while(s, &hout);
    cudaMemcpyAsync(e->h_ctl, e->ctl, sizeof(GmresCtl), cudaMemcpyDeviceToHost, s);
    cudaGraph_t G;
    chk(cudaStreamEndCapture(s, &G));
    // restart-cycle body: the Arnoldi loop, the update of x, the next residual
    chk(cudaStreamBeginCaptureToGraph(s2, body_out, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    {
        Ops<T> q(e, o0.a, s2);
        k_imp_enter<<<1, 1, 0, s2>>>(e->ctl);
        cudaGraph_t body_in = add_while(s2, &hin);
        k_imp_solve_y<<<1, 32, 0, s2>>>(e->ctl);
        k_imp_lincomb<T><<<nb_(n, 256), 256, 0, s2>>>(n, q.vec(0), e->ctl, (T*)e->t);
        q.precond((const T*)e->t, nullptr, (T*)e->z, nullptr);
        k_imp_addx<T><<<nb_(n, 256), 256, 0, s2>>>(n, (const T*)e->z, e->x);
        k_imp_outer_check<<<1, 1, 0, s2>>>(e->ctl);
        k_imp_cast<T><<<nb_(n, 256), 256, 0, s2>>>(n, e->x, (T*)e->t, halt);
        q.spmv((const T*)e->t, (T*)e->z, halt);
        k_imp_resid<T><<<nb_(n, 256), 256, 0, s2>>>(n, b, e->perm, (const T*)e->z, w, halt);
        q.norm2(w, ww, halt);
        k_imp_cycle_init<<<1, 1, 0, s2>>>(e->ctl, ww, scale, 0, 1e-2, max_iters);
        chk(cudaStreamEndCapture(s2, &body_out));
        chk(cudaStreamBeginCaptureToGraph(s3, body_in, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        Ops<T> r(e, o0.a, s3);
        r.arnoldi_step(r.vec(0), w, (T*)e->z, h1, h2, scale, kptr, stop);
        chk(cudaStreamEndCapture(s3, &body_in));
    }
    cudaGraphExec_t ex;
    const cudaError_t ri = cudaGraphInstantiate(&ex, G, 0);
    cudaGraphDestroy(G);
    chk(ri);
    e->h_ctl->hin = hin;
    e->h_ctl->hout = hout;
    chk(cudaMemcpyAsync(&e->ctl->hin, &e->h_ctl->hin, 2 * sizeof(cudaGraphConditionalHandle), cudaMemcpyHostToDevice,
                        s));
    chk(cudaStreamSynchronize(s));
    return ex;
}

// The same solve as build_gmres_graph with the two loops on the host: the
// control block is read back after every Arnoldi step, so each kernel is a
// plain launch (for profilers; slower by one host round trip per step).
template <class T>
int gmres_host_loop(ImplicitEngine* e, const StepArgs& a, const double* b, cudaStream_t s, int max_iters) {
    using namespace dev;
    const int n = e->n4;
    double* h1 = e->small;
    double* h2 = e->small + (GM_M + 1);
    double* ww = e->small + 2 * (GM_M + 1);
    double* scale = ww + 1;
    int* kptr = &e->ctl->k;
    int* stop = &e->ctl->stop;
    int* halt = &e->ctl->halt;
    Ops<T> o(e, a, s);
    auto read_ctl = [&]() {
        // stop, k, iters, halt: the loop conditions
        if (cudaMemcpyAsync(e->h_ctl, e->ctl, 4 * sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            throw Error(7, "implicit solver: GMRES failed");
    };
    T* w = (T*)e->w;
    cudaMemsetAsync(e->x, 0, (size_t)n * 8, s);
    o.gather_b(b, w);
    o.norm2(w, ww, nullptr);
    k_imp_cycle_init<<<1, 1, 0, s>>>(e->ctl, ww, scale, 1, 1e-2, max_iters);
    read_ctl();
    if (!e->h_ctl->stop) {
        for (;;) {
            for (;;) {  // Arnoldi steps of the cycle
                read_ctl();
                if (e->h_ctl->stop) break;
                o.arnoldi_step(o.vec(0), w, (T*)e->z, h1, h2, scale, kptr, stop);
            }
            k_imp_solve_y<<<1, 32, 0, s>>>(e->ctl);
            k_imp_lincomb<T><<<nb_(n, 256), 256, 0, s>>>(n, o.vec(0), e->ctl, (T*)e->t);
            o.precond((const T*)e->t, nullptr, (T*)e->z, nullptr);
            k_imp_addx<T><<<nb_(n, 256), 256, 0, s>>>(n, (const T*)e->z, e->x);
            k_imp_outer_check<<<1, 1, 0, s>>>(e->ctl);
            k_imp_cast<T><<<nb_(n, 256), 256, 0, s>>>(n, e->x, (T*)e->t, halt);
            o.spmv((const T*)e->t, (T*)e->z, halt);
            k_imp_resid<T><<<nb_(n, 256), 256, 0, s>>>(n, b, e->perm, (const T*)e->z, w, halt);
            o.norm2(w, ww, halt);
            k_imp_cycle_init<<<1, 1, 0, s>>>(e->ctl, ww, scale, 0, 1e-2, max_iters);
            read_ctl();
            if (e->h_ctl->halt) break;
        }
    }
    read_ctl();
    return e->h_ctl->iters;
}

template <class T>
int gmres(ImplicitEngine* e, const StepArgs& a, const double* b, cudaStream_t s, int max_iters) {
    if (!e->graph) return gmres_host_loop<T>(e, a, b, s, max_iters);
    Ops<T> o(e, a, s);
    if (e->cyc_b != b || !e->cyc[0]) {
        if (e->cyc[0]) cudaGraphExecDestroy(e->cyc[0]);
        e->cyc[0] = nullptr;
        if (!e->s2) {
            cudaStreamCreateWithFlags(&e->s2, cudaStreamNonBlocking);
            cudaStreamCreateWithFlags(&e->s3, cudaStreamNonBlocking);
        }
        e->cyc[0] = build_gmres_graph<T>(e, o, b, s, e->s2, e->s3, max_iters);
        e->cyc_b = b;
    }
    if (cudaGraphLaunch(e->cyc[0], s) != cudaSuccess) throw Error(7, "implicit solver: graph launch failed");
    if (cudaStreamSynchronize(s) != cudaSuccess) throw Error(7, "implicit solver: GMRES failed");
    return e->h_ctl->iters;
}

}  // namespace

// Solves M dQ = b (b: FP64 right-hand side over the real cells, AoS) and
// applies q += relax dQ to the FP64 state; dQ is also copied to qW.
// Returns the Krylov iterations, or -1 if a diagonal block was singular.
int implicit_solve_update(ImplicitEngine* e, const StepArgs& a, int p, const double* b, double relax,
                          cudaStream_t s) {
    int sing = 0;
    cudaMemcpyAsync(&sing, e->singular, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    if (sing) return -1;
    const int it = e->f32 ? gmres<float>(e, a, b, s, 500) : gmres<double>(e, a, b, s, 500);
    dev::k_imp_update<<<nb_(e->n4, 256), 256, 0, s>>>(e->n4, e->x, e->perm, relax, (double*)a.qm[p],
                                                      (double*)a.Rq);
    e->last_iters = it;
    return it;
}

// out = scale * (area .* x) (area null: 1) in device order, x the engine's
// last GMRES solution (row order)
namespace dev {
template <class T>
__global__ void __launch_bounds__(256) k_imp_scatter(const int n, const T* __restrict__ x,
                                                     const int* __restrict__ perm, const double* __restrict__ area,
                                                     const double scale, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = __ldg(&perm[i >> 2]);
    out[4 * (size_t)c + (i & 3)] = scale * (area ? area[c] : 1.0) * (double)x[i];
}
}  // namespace dev

// The engine's linear solve as an operator: M x = b (M^T after
// implicit_transpose) by the same GMRES the implicit iteration uses, then
// out = scale * (area .* x) in device order.  b must stay at one address
// between calls (the solve graph is captured for it).  Returns the Krylov
// iterations, -1 if a diagonal block was singular.
int implicit_apply_inverse(ImplicitEngine* e, const StepArgs& a, const double* b, const double* area, double scale,
                           double* out, cudaStream_t s) {
    int sing = 0;
    cudaMemcpyAsync(&sing, e->singular, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    if (sing) return -1;
    const int it = e->f32 ? gmres<float>(e, a, b, s, 500) : gmres<double>(e, a, b, s, 500);
    dev::k_imp_scatter<double><<<nb_(e->n4, 256), 256, 0, s>>>(e->n4, e->x, e->perm, area, scale, out);
    e->last_iters = it;
    return it;
}

namespace {
template <class T>
void sweep_t(ImplicitEngine* e, const StepArgs& a, const double* b, const double* area, double scale, double* out,
             cudaStream_t s) {
    Ops<T> o(e, a, s);
    o.gather_b(b, (T*)e->t);
    o.precond((const T*)e->t, nullptr, (T*)e->z, nullptr);
    dev::k_imp_scatter<T><<<nb_(e->n4, 256), 256, 0, s>>>(e->n4, (const T*)e->z, e->perm, area, scale, out);
}
}  // namespace

// The engine's preconditioner alone as an operator: one symmetric
// multicolour block Gauss-Seidel sweep with the ILU(0) factors (of M, or of
// M^T after implicit_transpose), out = scale * (area .* x) in device order.
// Returns -1 if a diagonal block was singular, else 0.
int implicit_apply_sweep(ImplicitEngine* e, const StepArgs& a, const double* b, const double* area, double scale,
                         double* out, cudaStream_t s) {
    int sing = 0;
    cudaMemcpyAsync(&sing, e->singular, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    if (sing) return -1;
    if (e->f32) sweep_t<float>(e, a, b, area, scale, out, s);
    else sweep_t<double>(e, a, b, area, scale, out, s);
    return 0;
}

// The filled system transposed in place (M -> M^T, the ILU(0) factors ->
// those of M^T) for the adjoint's linear solves.  The next implicit_fill
// forms M again.  FP64 engines.
void implicit_transpose(ImplicitEngine* e, cudaStream_t s) {
    using namespace dev;
    if (e->f32) throw Error(7, "implicit solver: the adjoint needs an FP64 engine");
    // the Krylov basis (124 T per row) holds the copy of the blocks (64 T per row)
    cudaMemcpyAsync(e->V, e->off, (size_t)e->N * 64 * sizeof(double), cudaMemcpyDeviceToDevice, s);
    k_imp_transpose<double><<<nb_(e->N, 128), 128, 0, s>>>(e->N, e->ell(), (const double*)e->V, (double*)e->off,
                                                           (double*)e->dblk, (double*)e->dinv);
}

}  // namespace afx
