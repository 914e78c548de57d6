// Adjoint of the FP64 residual: u = (dR/dq)^T v and b = (dR/dbq)^T v for the
// residual R(q) of the explicit solver's first stage (solver.h:745-799 with
// the gradient of solver.h:428-469 and the limiter of solver.h:517-593, all
// formed from q), where bq are the stored boundary (farfield) states.
//
// Reverse sweep in three gather kernels, deterministic and atomic-free:
//   k_adj_face   per face: the flux functional sum_m w_m F_m of the face weight
//                w = L*(v_c1/A_c1 - v_c0/A_c0) differentiated by a reverse
//                sweep through the flux written out by hand (roe_reverse,
//                laminar_reverse): all 8 (laminar: 16) derivatives for about
//                one and a half times the flux's own work.
//   k_adj_cell   per cell: gathers its faces' numbers into the state,
//                limiter and gradient adjoints of the reconstruction
//                q + phi .* (grad q . d), then reverses its limiter (active
//                face of the min, neighbour of the max/min) -- the
//                neighbour terms are left as (target, weight) pairs.
//   k_adj_final  per cell: adds the limiter pairs that target it and the
//                Green-Gauss gradient's reverse over its faces, and writes
//                the boundary-state adjoint of its boundary faces.
// Face Jacobians are never formed.  Roe flux with the entropy fix and every
// boundary type, and the laminar term (then the face gradient's inputs too,
// reversed through average_gradients); first or second order; both limiters.
#include "afx_dual.cuh"
#include "afx_kernels_impl.cuh"

namespace afx {
namespace dev {

constexpr int ADJ_NONE = (int)0x80000000;  // limiter target: none / the cell itself

__device__ __forceinline__ int pick4(const int4 v, const int k) { return pick(v, k); }

// One eigenvalue a = entropy_corr(sqrt(x^2 + 1e-4), 0.05 c): its value and its
// derivatives in x and c, of the branch the value takes.
__device__ __forceinline__ double eig_reverse(const double x, const double d, const fp64::Den& id, double& dx,
                                              double& dc) {
    using namespace fp64;
    const double s2 = x * x + 1e-4, s = root(s2);
    if (less(d, s)) {
        dx = div(x, s);
        dc = 0.0;
        return s;
    }
    dx = quot(x, id);
    const double r = quot(s2, id);  // s^2 / d
    dc = 0.05 * __fma_rn(-0.5, quot(r, id), 0.5);
    return 0.5 * (r + d);
}

// bL[k] = sum_m w_m dF_m/dqL_k and bR likewise for the Roe flux F
// (physics.h:168-228): the flux's values forward (roe_flux2), then every
// statement's adjoint in reverse order.  x_ below is the derivative of the
// functional in x; fused multiply-adds throughout (the FP64 pipe bounds the
// kernel: about 330 of its instructions per face; eight directions of forward
// dual numbers took about 1,900 and 24 quotients each).  394k faces: 3.87 ->
// 0.33 ms; the whole vJP of 262k cells 6.46 -> 1.27 ms.
__device__ __forceinline__ void roe_reverse(const double gamma, const double nx, const double ny, const double* qL,
                                            const double* qR, const double* w, double* bL, double* bR) {
    using namespace fp64;
    const auto mad = [](const double a, const double b, const double c) { return __fma_rn(a, b, c); };
    const double g1 = gamma - 1.0;
    const double iL = div(1.0, qL[0]), iR = div(1.0, qR[0]);
    const double uL = qL[1] * iL, vL = qL[2] * iL, uR = qR[1] * iR, vR = qR[2] * iR;
    const double kL = 0.5 * mad(uL, uL, vL * vL), kR = 0.5 * mad(uR, uR, vR * vR);
    const double pL = g1 * mad(-qL[0], kL, qL[3]), pR = g1 * mad(-qR[0], kR, qR[3]);
    const double VL = mad(uL, nx, vL * ny), VR = mad(uR, nx, vR * ny);
    const double eL = qL[3] + pL, eR = qR[3] + pR, hL = eL * iL, hR = eR * iR;
    const double sL = root(qL[0]), sR = root(qR[0]), rho = sL * sR;
    const double is = div(1.0, sL + sR);
    const double u = mad(uL, sL, uR * sR) * is, v = mad(vL, sL, vR * sR) * is, h = mad(hL, sL, hR * sR) * is;
    const double q2 = mad(u, u, v * v);
    const double c2 = g1 * mad(-0.5, q2, h), c = root(c2), ic2 = div(1.0, c2);
    const double V = mad(u, nx, v * ny);
    const double d = 0.05 * c;
    const Den id = den(d);
    double x1, x2, x3, y1, y2, y3;
    const double a1 = eig_reverse(V - c, d, id, x1, y1);
    const double a2 = eig_reverse(V, d, id, x2, y2);
    const double a3 = eig_reverse(V + c, d, id, x3, y3);
    const double dp = pR - pL, dV = VR - VL, du = uR - uL, dv = vR - vL, rc = rho * c, t = rc * dV;
    const double hi = 0.5 * ic2;
    const double b1 = (dp - t) * hi, b5 = (dp + t) * hi, b2 = mad(-dp, ic2, qR[0] - qL[0]);
    const double k1 = a1 * b1, k2 = a2 * b2, k3 = a2 * rho, k5 = a3 * b5;
    // F = (A - S) / 2: z for A, -z for the dissipation S
    const double z0 = 0.5 * w[0], z1 = 0.5 * w[1], z2 = 0.5 * w[2], z3 = 0.5 * w[3];
    const double zn = mad(z1, nx, z2 * ny);
    const double zu = mad(z1, u, mad(z2, v, z0));       // z0 + z1 u + z2 v
    const double zc = c * mad(z3, V, zn);               // c (z1 nx + z2 ny + z3 V)
    const double k1_ = -(mad(z3, h, zu) - zc), k5_ = -(mad(z3, h, zu) + zc), k2_ = -mad(0.5 * z3, q2, zu);
    const double k3_ = -(mad(z1, du, z2 * dv) - dV * zn + z3 * (mad(u, du, v * dv) - V * dV));
    const double ks = k1 + k2 + k5, kd = k5 - k1, zk = z3 * k3;
    double u_ = -mad(z1, ks, zk * du), v_ = -mad(z2, ks, zk * dv), h_ = -z3 * (k1 + k5);
    double c_ = -kd * mad(z3, V, zn), V_ = -mad(z3 * c, kd, -zk * dV), q2_ = -0.5 * z3 * k2;
    const double du_ = -k3 * mad(z3, u, z1), dv_ = -k3 * mad(z3, v, z2);
    double dV_ = k3 * mad(z3, V, zn);
    // k1 = a1 b1, k2 = a2 b2, k3 = a2 rho, k5 = a3 b5
    const double a1_ = k1_ * b1, a3_ = k5_ * b5, a2_ = mad(k2_, b2, k3_ * rho);
    const double b1_ = k1_ * a1, b5_ = k5_ * a3, b2_ = k2_ * a2;
    const double t_ = (b5_ - b1_) * hi, tdV = t_ * dV;
    double rho_ = mad(k3_, a2, tdV * c);
    const double dp_ = mad(b1_ + b5_, hi, -b2_ * ic2);
    dV_ = mad(t_, rc, dV_);
    c_ = mad(tdV, rho, c_);
    double c2_ = ic2 * (mad(b2_ * dp, ic2, 0.0) - mad(b1_, b1, b5_ * b5));
    // eigenvalues
    const double e1 = a1_ * x1, e3 = a3_ * x3;
    V_ += mad(a2_, x2, e1 + e3);
    c_ += (e3 - e1) + mad(a1_, y1, mad(a2_, y2, a3_ * y3));
    // c, V, Roe averages
    c2_ = mad(c_ * c, 0.5 * ic2, c2_);
    h_ = mad(g1, c2_, h_);
    q2_ = mad(-0.5 * g1, c2_, q2_);
    u_ = mad(2.0 * u, q2_, mad(V_, nx, u_)) * is;
    v_ = mad(2.0 * v, q2_, mad(V_, ny, v_)) * is;
    h_ *= is;
    const double sL_ = mad(rho_, sR, mad(u_, uL - u, mad(v_, vL - v, h_ * (hL - h))));
    const double sR_ = mad(rho_, sL, mad(u_, uR - u, mad(v_, vR - v, h_ * (hR - h))));
    // each side: V, p, u, v, H, sqrt(rho) and the fluxes A
    const auto side = [&](const double* q, const double ir, const double uu, const double vv, const double kk,
                          const double VV, const double ee, const double hh, const double ss, const double s_,
                          const double sg, double* b) {
        const double Vs_ = mad(sg, dV_, mad(z0, q[0], mad(z1, q[1], mad(z2, q[2], z3 * ee))));
        const double H_ = h_ * ss * ir;                                  // of e + p over rho
        const double p_ = mad(sg, dp_, mad(z3, VV, zn)) + H_;
        const double us_ = mad(u_, ss, mad(sg, du_, Vs_ * nx)) * ir;      // of rho u at fixed rho
        const double vs_ = mad(v_, ss, mad(sg, dv_, Vs_ * ny)) * ir;
        const double gp = g1 * p_;
        b[3] = mad(z3, VV, H_) + gp;
        b[1] = mad(z1, VV, us_) - gp * uu;
        b[2] = mad(z2, VV, vs_) - gp * vv;
        b[0] = mad(sg, b2_, mad(z0, VV, mad(gp, kk, -mad(H_, hh, mad(us_, uu, vs_ * vv))))) +
               0.5 * s_ * (ss * ir);                                     // 1/sqrt(rho) = sqrt(rho)/rho
    };
    side(qL, iL, uL, vL, kL, VL, eL, hL, sL, sL_, -1.0, bL);
    side(qR, iR, uR, vR, kR, VR, eR, hR, sR, sR_, 1.0, bR);
}

// Adds sum_m w_m d(laminar term)_m to bL, bR (both states) and sets gxb, gyb
// (the face gradient's x and y parts); the term is subtracted from the flux
// (physics.h:230-258).
__device__ __forceinline__ void laminar_reverse(const KM<double>& m, const double nx, const double ny,
                                                const double* qL, const double* qR, const double* gx,
                                                const double* gy, const double* w, double* bL, double* bR,
                                                double* gxb, double* gyb) {
    using namespace fp64;
    const auto mad = [](const double a, const double b, const double c) { return __fma_rn(a, b, c); };
    const double g1 = m.gamma - 1.0, mu = m.mu, kh = m.kheat;
    double q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) q[k] = 0.5 * (qL[k] + qR[k]);
    const double ir = div(1.0, q[0]), U = q[1] * ir, V = q[2] * ir, ke = 0.5 * mad(U, U, V * V);
    const double pr = g1 * mad(q[3], ir, -ke);   // p / rho
    const double irR = ir * div(1.0, m.R);
    // velocity and temperature gradients (calc_grad_u/v/temp, physics.h:33-82)
    const auto parts = [&](const double* g, double& gu, double& gv, double& gT) {
        gu = mad(-U, g[0], g[1]) * ir;
        gv = mad(-V, g[0], g[2]) * ir;
        const double gp = g1 * mad(ke, g[0], mad(-V, g[2], mad(-U, g[1], g[3])));
        gT = mad(-pr, g[0], gp) * irR;
    };
    double ux, vx, Tx, uy, vy, Ty;
    parts(gx, ux, vx, Tx);
    parts(gy, uy, vy, Ty);
    const double div3 = (ux + vy) * (1.0 / 3.0);
    const double xx = 2.0 * mu * (ux - div3), yy = 2.0 * mu * (vy - div3), xy = mu * (uy + vx);
    const double a1 = -w[1], a2 = -w[2], a3 = -w[3];
    const double xx_ = nx * mad(a3, U, a1), yy_ = ny * mad(a3, V, a2);
    const double xy_ = mad(a1, ny, a2 * nx) + a3 * mad(nx, V, ny * U);
    double U_ = a3 * mad(nx, xx, ny * xy), V_ = a3 * mad(nx, xy, ny * yy), r_ = 0.0, pr_ = 0.0;
    const double s3 = (xx_ + yy_) * (1.0 / 3.0);
    const double ux_ = 2.0 * mu * (xx_ - s3), vy_ = 2.0 * mu * (yy_ - s3), xym = mu * xy_;
    const auto back = [&](const double* g, const double gu, const double gv, const double gT, const double gu_,
                          const double gv_, const double gT_, double* gb) {
        const double T_ = gT_ * irR, p_ = g1 * T_, gur = gu_ * ir, gvr = gv_ * ir;
        gb[0] = mad(p_, ke, -mad(T_, pr, mad(gur, U, gvr * V)));
        gb[1] = mad(-p_, U, gur);
        gb[2] = mad(-p_, V, gvr);
        gb[3] = p_;
        pr_ = mad(-T_, g[0], pr_);
        U_ += mad(p_, mad(U, g[0], -g[1]), -gur * g[0]);
        V_ += mad(p_, mad(V, g[0], -g[2]), -gvr * g[0]);
        r_ -= ir * mad(gT_, gT, mad(gu_, gu, gv_ * gv));
    };
    back(gx, ux, vx, Tx, ux_, xym, a3 * nx * kh, gxb);
    back(gy, uy, vy, Ty, xym, vy_, a3 * ny * kh, gyb);
    // p / rho = (gamma - 1)(e/rho - (U^2 + V^2)/2)
    const double gp = g1 * pr_;
    U_ = mad(-gp, U, U_) * ir;
    V_ = mad(-gp, V, V_) * ir;
    const double e_ = gp * ir;
    double b[4];
    b[0] = r_ - mad(e_, q[3] * ir, mad(U_, U, V_ * V));
    b[1] = U_;
    b[2] = V_;
    b[3] = e_;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        bL[k] = mad(0.5, b[k], bL[k]);
        bR[k] = mad(0.5, b[k], bR[k]);
    }
}

// Derivatives of limiter_value in (dqg, delta_max, delta_min) for its active
// branch; lim: its value
__device__ __forceinline__ void limiter_reverse(const int kind, const double g, const double dmx, const double dmn,
                                                const double K3a, const double lim, double* o) {
    using namespace fp64;
    o[0] = o[1] = o[2] = 0.0;
    if (kind == 0) {
        // lim = (d^2 + K + 2 g d) / (d^2 + 2 g^2 + d g + K)
        if (!(fabs(g) > 1e-16)) return;
        const double d = g > 0.0 ? dmx : dmn;
        const Den iq = den(d * d + 2.0 * g * g + d * g + K3a);
        o[0] = quot(2.0 * d - lim * (4.0 * g + d), iq);
        o[g > 0.0 ? 1 : 2] = quot(2.0 * (d + g) - lim * (2.0 * d + g), iq);
        return;
    }
    const double dd = dmx - dmn, s2 = dd * dd;
    if (s2 <= K3a) return;
    double sig = 0.0, ds = 0.0;  // ds: d sig / d delta_max (delta_min: the negative)
    if (s2 <= 2.0 * K3a) {
        const Den ik = den(K3a);
        const double y = quot(s2, ik) - 1.0;
        sig = 2.0 * y * y * y - 3.0 * y * y + 1.0;
        ds = quot(6.0 * y * (y - 1.0), ik) * 2.0 * dd;
    }
    // the polynomial (Michalak) limiter of y = delta / g is y - y^2/4 up to y = 2
    double l = 1.0, dg = 0.0, dy = 0.0;
    if (fabs(g) > 1e-14) {
        const Den ig = den(g);
        const double y = quot(g > 0.0 ? dmx : dmn, ig);
        if (y < 2.0) {
            l = y - 0.25 * y * y;
            dy = quot(1.0 - 0.5 * y, ig);
            dg = -dy * y;
        }
    }
    o[0] = (1.0 - sig) * dg;
    o[1] = ds * (1.0 - l) + (g > 0.0 ? (1.0 - sig) * dy : 0.0);
    o[2] = -ds * (1.0 - l) + (g > 0.0 ? 0.0 : (1.0 - sig) * dy);
}

// sum_m d ghost_m/d(dir) * w_m (dir 0-3: interior state, 4-7: boundary
// state); out of line, by value: boundary faces are few, and inlined it takes
// the registers of every face and cell
static __device__ __noinline__ double ghost_dir(const int bt, const double gamma, const double nx, const double ny,
                                                const d4 qi, const d4 qb, const int dir, const d4 w) {
    const double x[4] = {qi.x, qi.y, qi.z, qi.w}, y[4] = {qb.x, qb.y, qb.z, qb.w};
    Dual a[4], b[4], g[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        a[k] = Dual(x[k], dir == k ? 1.0 : 0.0);
        b[k] = Dual(y[k], dir == k + 4 ? 1.0 : 0.0);
    }
    ghost_state<Dual>(bt, Dual(gamma), Dual(nx), Dual(ny), a, b, g);
    return g[0].d * w.x + g[1].d * w.y + g[2].d * w.z + g[3].d * w.w;
}
__device__ __forceinline__ d4 vec4(const double* v) {
    d4 r;
    r.x = v[0]; r.y = v[1]; r.z = v[2]; r.w = v[3];
    return r;
}

// Per face, FB = 2 (inviscid) or 8 (laminar) 4-vectors of fbar:
// [qL_bar, qR_bar (or the boundary state's), and with the laminar term
//  gxa_bar, gya_bar, qa_bar, gxb_bar, gyb_bar, qb_bar] -- a/b: the face's
// cells as the face gradient sees them (solver.h:359-398)
template <bool SECOND, int VISC>
__global__ void __launch_bounds__(128) k_adj_face(const KM<double> m, const int n_faces, const d4* __restrict__ q,
                                                  const d4* __restrict__ gx, const d4* __restrict__ gy,
                                                  const d4* __restrict__ phi, const d4* __restrict__ v,
                                                  d4* __restrict__ fbar) {
    constexpr int FB = VISC == 1 ? 8 : 2;
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_faces) return;
    const int2 cc = __ldg(&m.fcell[f]);
    const double2 n = __ldg(&m.fn[f]);
    const double L = __ldg(&m.fLg[f]).x;
    double q0[4], q1[4], qL[4], qR[4], w[4], v0[4];
    double g0x[4] = {0, 0, 0, 0}, g0y[4] = {0, 0, 0, 0}, g1x[4] = {0, 0, 0, 0}, g1y[4] = {0, 0, 0, 0};
    ld4(&q[cc.x], q0);
    if (SECOND || VISC == 1) {
        ld4(&gx[cc.x], g0x);
        ld4(&gy[cc.x], g0y);
    }
    if (SECOND) {
        double p0[4];
        ld4(&phi[cc.x], p0);
        const double2 d0 = __ldg(&m.fd0[f]);
        reconstruct(q0, g0x, g0y, p0, d0.x, d0.y, qL);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) qL[k] = q0[k];
    }
    ld4(&v[cc.x], v0);
    const Div<double> iA0(__ldg(&m.area[cc.x]));
    int bt = BT_INTERNAL;
    if (cc.y >= 0) {
        double v1[4];
        ld4(&q[cc.y], q1);
        if (SECOND || VISC == 1) {
            ld4(&gx[cc.y], g1x);
            ld4(&gy[cc.y], g1y);
        }
        if (SECOND) {
            double p1[4];
            ld4(&phi[cc.y], p1);
            const double2 d1 = __ldg(&m.fd1[f]);
            reconstruct(q1, g1x, g1y, p1, d1.x, d1.y, qR);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) qR[k] = q1[k];
        }
        ld4(&v[cc.y], v1);
        const Div<double> iA1(__ldg(&m.area[cc.y]));
        // R_c0 -= F*L/A_c0, R_c1 += F*L/A_c1
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = L * (iA1(v1[k]) - iA0(v0[k]));
    } else {
        bt = __ldg(&m.btype[-cc.y - 1]);
        ld4(&m.bq[-cc.y - 1], q1);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            qR[k] = q1[k];
            w[k] = -L * iA0(v0[k]);
        }
    }
    // the face gradient of the laminar term (member states, cell gradients;
    // a boundary side has zero gradient)
    const bool lam = VISC == 1 && two_sided(bt);
    double fgx[4] = {0, 0, 0, 0}, fgy[4] = {0, 0, 0, 0};
    double4 t = make_double4(0, 0, 1, 0);  // (t0, t1, lij): zero adjoint on a face without the term
    if (lam) {
        const d4 tt = ldv4d(&m.ft[f]);
        t = make_double4(tt.x, tt.y, tt.z, tt.w);
        face_gradient(q0, q1, g0x, g0y, g1x, g1y, tt, fgx, fgy);
    }
    double out[VISC == 1 ? 16 : 8];
    if (two_sided(bt)) {
        roe_reverse(m.gamma, n.x, n.y, qL, qR, w, out, out + 4);
    } else {
        // the ghost state's derivatives by dual numbers (boundary faces alone)
        double qg[4], bi[4], bg[4];
        ghost_state(bt, m.gamma, n.x, n.y, qL, qR, qg);
        roe_reverse(m.gamma, n.x, n.y, qL, qg, w, bi, bg);
#pragma unroll 1
        for (int dir = 0; dir < 8; ++dir)
            out[dir] = (dir < 4 ? bi[dir & 3] : 0.0) + ghost_dir(bt, m.gamma, n.x, n.y, vec4(qL), vec4(qR), dir, vec4(bg));
    }
    if constexpr (VISC == 1) {
#pragma unroll
        for (int k = 8; k < 16; ++k) out[k] = 0.0;
        if (lam) laminar_reverse(m, n.x, n.y, qL, qR, fgx, fgy, w, out, out + 4, out + 8, out + 12);
    }
    d4* fb = fbar + (size_t)FB * f;
    st4(&fb[0], out);
    st4(&fb[1], out + 4);
    if (VISC == 1) {
        // reverse of face_gradient (solver.h:359-398), component by component:
        // fg = gbar - ((gbar . t) - (qa - qb)/lij) t, gbar the mean gradient
        double ga_x[4], ga_y[4], qa_b[4], gb_x[4], gb_y[4], qb_b[4];
        const Div<double> it(t.z);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const double fx = out[8 + k], fy = out[12 + k];
            const double e = -(t.x * fx + t.y * fy);  // adjoint of grad_dot - grad_dir
            const double mx = fx + e * t.x, my = fy + e * t.y;
            ga_x[k] = gb_x[k] = 0.5 * mx;
            ga_y[k] = gb_y[k] = 0.5 * my;
            qa_b[k] = it(-e);
            qb_b[k] = it(e);
        }
        st4(&fb[2], ga_x);
        st4(&fb[3], ga_y);
        st4(&fb[4], qa_b);
        st4(&fb[5], gb_x);
        st4(&fb[6], gb_y);
        st4(&fb[7], qb_b);
    }
}

template <bool SECOND, int VISC>
__global__ void __launch_bounds__(128) k_adj_cell(const KM<double> m, const d4* __restrict__ q,
                                                  const d4* __restrict__ gx, const d4* __restrict__ gy,
                                                  const d4* __restrict__ phi, const d4* __restrict__ fbar,
                                                  d4* __restrict__ qbar, d4* __restrict__ gbx, d4* __restrict__ gby,
                                                  d4* __restrict__ lw, int4* __restrict__ lt) {
    constexpr int FB = VISC == 1 ? 8 : 2;
    constexpr bool GRAD = SECOND || VISC == 1;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.n_cells) return;
    const int4 sl = __ldg(&m.cslot[i]);
    const int4 nb = __ldg(&m.cnbr[i]);
    double qb[4] = {0, 0, 0, 0}, pb[4] = {0, 0, 0, 0}, bx[4] = {0, 0, 0, 0}, by[4] = {0, 0, 0, 0};
    double qi[4], gxi[4], gyi[4], ph[4];
    if (SECOND) {
        ld4(&q[i], qi);
        ld4(&gx[i], gxi);
        ld4(&gy[i], gyi);
        ld4(&phi[i], ph);
    }
    double dxs[4] = {0, 0, 0, 0}, dys[4] = {0, 0, 0, 0};
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int fs = pick(sl, s);
        if (fs == 0) continue;
        const bool own0 = fs > 0;
        const int f = (own0 ? fs : -fs) - 1;
        double side[4];
        const d4* fb = fbar + (size_t)FB * f;
        ld4(&fb[own0 ? 0 : 1], side);
#pragma unroll
        for (int k = 0; k < 4; ++k) qb[k] += side[k];
        if (VISC == 1) {
            // the face gradient's use of this cell's member state and gradient
            double sgx[4], sgy[4], sq[4];
            ld4(&fb[own0 ? 2 : 5], sgx);
            ld4(&fb[own0 ? 3 : 6], sgy);
            ld4(&fb[own0 ? 4 : 7], sq);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                qb[k] += sq[k];
                bx[k] += sgx[k];
                by[k] += sgy[k];
            }
        }
        if (SECOND) {
            const double2 d = own0 ? __ldg(&m.fd0[f]) : __ldg(&m.fd1[f]);
            dxs[s] = d.x;
            dys[s] = d.y;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                pb[k] += side[k] * (gxi[k] * d.x + gyi[k] * d.y);
                bx[k] += side[k] * ph[k] * d.x;
                by[k] += side[k] * ph[k] * d.y;
            }
        }
    }
    if (SECOND) {
        // neighbour max/min with the cell that attains them (smax/smin order)
        double qmx[4], qmn[4];
        int tmx[4], tmn[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            qmx[k] = qmn[k] = qi[k];
            tmx[k] = tmn[k] = ADJ_NONE;
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (pick(sl, s) == 0) continue;
            const int o = pick(nb, s);
            double qo[4];
            bool use = true;
            if (o >= 0) {
                ld4(&q[o], qo);
            } else {
                const int bt = __ldg(&m.btype[-o - 1]);
                use = bt != BT_SLIP && bt != BT_WALL;
                ld4(&m.bq[-o - 1], qo);
            }
            if (!use) continue;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (fp64::less(qmx[k], qo[k])) {
                    qmx[k] = qo[k];
                    tmx[k] = o;
                }
                if (fp64::less(qo[k], qmn[k])) {
                    qmn[k] = qo[k];
                    tmn[k] = o;
                }
            }
        }
        const double A = __ldg(&m.area[i]);
        const double Ka = m.limk * dsqrt(A);
        const double K3a = Ka * Ka * Ka;
        double wmx[4] = {0, 0, 0, 0}, wmn[4] = {0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            double lim = 1.0;
            int sa = -1;
            for (int s = 0; s < 4; ++s) {
                if (pick(sl, s) == 0) continue;
                const double dqg = gxi[k] * dxs[s] + gyi[k] * dys[s];
                const double lv = limiter_value(m.limiter, dqg, qmx[k] - qi[k], qmn[k] - qi[k], K3a);
                if (fp64::less(lv, lim)) {
                    lim = lv;
                    sa = s;
                }
            }
            if (sa < 0 || pb[k] == 0.0) continue;
            const double dx = sa == 0 ? dxs[0] : sa == 1 ? dxs[1] : sa == 2 ? dxs[2] : dxs[3];
            const double dy = sa == 0 ? dys[0] : sa == 1 ? dys[1] : sa == 2 ? dys[2] : dys[3];
            const double dqg = gxi[k] * dx + gyi[k] * dy;
            double dl[3];
            limiter_reverse(m.limiter, dqg, qmx[k] - qi[k], qmn[k] - qi[k], K3a, lim, dl);
            bx[k] += pb[k] * dl[0] * dx;
            by[k] += pb[k] * dl[0] * dy;
            // delta_max = qmax - q_i, delta_min = qmin - q_i
            if (tmx[k] != ADJ_NONE) {
                wmx[k] = pb[k] * dl[1];
                qb[k] -= wmx[k];
            }
            if (tmn[k] != ADJ_NONE) {
                wmn[k] = pb[k] * dl[2];
                qb[k] -= wmn[k];
            }
        }
        st4(&lw[2 * (size_t)i], wmx);
        st4(&lw[2 * (size_t)i + 1], wmn);
        lt[2 * (size_t)i] = make_int4(tmx[0], tmx[1], tmx[2], tmx[3]);
        lt[2 * (size_t)i + 1] = make_int4(tmn[0], tmn[1], tmn[2], tmn[3]);
    }
    if (GRAD) {
        st4(&gbx[i], bx);
        st4(&gby[i], by);
    }
    st4(&qbar[i], qb);
}

template <bool SECOND, int VISC>
__global__ void __launch_bounds__(128) k_adj_final(const KM<double> m, const d4* __restrict__ q,
                                                   const d4* __restrict__ fbar, const d4* __restrict__ qbar,
                                                   const d4* __restrict__ gbx, const d4* __restrict__ gby,
                                                   const d4* __restrict__ lw, const int4* __restrict__ lt,
                                                   d4* __restrict__ u, d4* __restrict__ bqbar) {
    constexpr int FB = VISC == 1 ? 8 : 2;
    constexpr bool GRAD = SECOND || VISC == 1;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m.n_cells) return;
    const int4 sl = __ldg(&m.cslot[j]);
    const int4 nb = __ldg(&m.cnbr[j]);
    double uj[4];
    ld4(&qbar[j], uj);
    double bxj[4], byj[4], qj[4], gjx[4], gjy[4];  // gj: over the area
    const Div<double> iAj(__ldg(&m.area[j]));
    if (GRAD) {
        ld4(&gbx[j], bxj);
        ld4(&gby[j], byj);
        ld4(&q[j], qj);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            gjx[k] = iAj(bxj[k]);
            gjy[k] = iAj(byj[k]);
        }
    }
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
        const int fs = pick(sl, s);
        if (fs == 0) continue;
        const bool own0 = fs > 0;
        const int f = (own0 ? fs : -fs) - 1;
        const int o = pick(nb, s);
        const double2 n = __ldg(&m.fn[f]);
        const double2 Lg = __ldg(&m.fLg[f]);
        if (o >= 0) {
            if (!GRAD) continue;
            if (SECOND) {
                // limiter terms of the neighbour that point at this cell
                double wx[4], wn[4];
                ld4(&lw[2 * (size_t)o], wx);
                ld4(&lw[2 * (size_t)o + 1], wn);
                const int4 tx = __ldg(&lt[2 * (size_t)o]);
                const int4 tn = __ldg(&lt[2 * (size_t)o + 1]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (pick4(tx, k) == j) uj[k] += wx[k];
                    if (pick4(tn, k) == j) uj[k] += wn[k];
                }
            }
            // Green-Gauss face value (q_c0 (1-g) + (q_c0 + q_c1)/2 g) L, added
            // to cell 0's sum and subtracted from cell 1's
            double bxo[4], byo[4];
            ld4(&gbx[o], bxo);
            ld4(&gby[o], byo);
            const Div<double> iAo(__ldg(&m.area[o]));
            const double g = Lg.y;
            const double wself = own0 ? ((1.0 - g) + 0.5 * g) : 0.5 * g;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double gox = iAo(bxo[k]), goy = iAo(byo[k]);
                const double s0x = own0 ? gjx[k] : gox, s1x = own0 ? gox : gjx[k];
                const double s0y = own0 ? gjy[k] : goy, s1y = own0 ? goy : gjy[k];
                const double fb = n.x * (s0x - s1x) + n.y * (s0y - s1y);
                uj[k] += fb * wself * Lg.x;
            }
        } else {
            // boundary face b of this cell (always its cell 0)
            const int b = -o - 1;
            double bb[4];
            ld4(&fbar[(size_t)FB * f + 1], bb);
            if (VISC == 1) {
                // a two-sided boundary's face gradient reads the boundary state
                double qbb[4];
                ld4(&fbar[(size_t)FB * f + 7], qbb);
#pragma unroll
                for (int k = 0; k < 4; ++k) bb[k] += qbb[k];
            }
            if (SECOND) {
                double wx[4], wn[4];
                ld4(&lw[2 * (size_t)j], wx);
                ld4(&lw[2 * (size_t)j + 1], wn);
                const int4 tx = __ldg(&lt[2 * (size_t)j]);
                const int4 tn = __ldg(&lt[2 * (size_t)j + 1]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (pick4(tx, k) == o) bb[k] += wx[k];
                    if (pick4(tn, k) == o) bb[k] += wn[k];
                }
            }
            if (GRAD) {
                // face value (q_j (1-g) + ghost(q_j, bq) g) L
                const int bt = __ldg(&m.btype[b]);
                double qbc[4], fb[4];
                ld4(&m.bq[b], qbc);
                const double g = Lg.y;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    fb[k] = iAj(n.x * bxj[k] + n.y * byj[k]) * Lg.x;
                    uj[k] += fb[k] * (1.0 - g);
                }
#pragma unroll 1
                for (int dir = 0; dir < 8; ++dir) {
                    const double t = g * ghost_dir(bt, m.gamma, n.x, n.y, vec4(qj), vec4(qbc), dir, vec4(fb));
                    if (dir < 4) uj[dir] += t;
                    else bb[dir - 4] += t;
                }
            }
            st4(&bqbar[b], bb);
        }
    }
    st4(&u[j], uj);
}

// One adjoint pseudo-time stage: lam_k = lam_0 + alpha*relax*dt*(u + g), with
// ||u + g||^2 block partials on the last stage.
__global__ void __launch_bounds__(256) k_adj_update(const int n, const d4* __restrict__ lam0,
                                                    const d4* __restrict__ u, const d4* __restrict__ g,
                                                    const double* __restrict__ dt, const double alpha,
                                                    const double relax, d4* __restrict__ lam_out,
                                                    double* __restrict__ partials) {
    __shared__ double sh[32];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double sq = 0;
    if (i < n) {
        double l0[4], ui[4], gi[4], out[4];
        ld4(&lam0[i], l0);
        ld4(&u[i], ui);
        ld4(&g[i], gi);
        const double d = __ldg(&dt[i]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const double r = ui[k] + gi[k];
            out[k] = l0[k] + r * d * alpha * relax;
            sq += r * r;
        }
        st4(&lam_out[i], out);
    }
    if (partials) {
        const double t = block_sum(sq, sh);
        if (threadIdx.x == 0) partials[blockIdx.x] = t;
    }
}

// dJ/dq of a force coefficient J = cx*fx + cy*fy over the patch edges
// (post.h:341-384): cp = 2/(gamma M^2) (p/p_inf - 1) of each edge's cell.
// One thread walks the edges in order, so a cell with two patch edges sums
// them in a fixed order.
__global__ void k_objective_grad(const ForceArgs f, const double cx, const double cy, d4* __restrict__ g) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    const d4* q = (const d4*)f.q;
    const double dx = f.xmax - f.xmin;
    const double c = 2. / (f.gamma * f.mach_inf * f.mach_inf) / f.p_inf;
    for (int e = 0; e < f.n; ++e) {
        double qc[4];
        ld4(&q[f.cell[e]], qc);
        const double* ge = f.geo + 5 * e;
        const double u = qc[1] / qc[0], v = qc[2] / qc[0];
        const double s = c * (cx * ge[2] + cy * ge[3]) * ge[4] / dx * (f.gamma - 1);
        d4& o = g[f.cell[e]];
        o.x += s * 0.5 * (u * u + v * v);
        o.y -= s * u;
        o.z -= s * v;
        o.w += s;
    }
}

}  // namespace dev

void enqueue_adjoint_prep(const StepArgs& a0, int p, bool with_dt, cudaStream_t s) {
    StepArgs a = a0;
    a.variant = with_dt ? 0 : 1;  // variant 0's prep also forms the local time step
    const dev::KM<double> m = dev::make_km<double>(a);
    dev::launch_prep<double, double>(a, m, (const dev::d4*)a.qm[p], s);
}

namespace {
template <bool SECOND, int VISC>
void vjp_launch(const StepArgs& a, int p, const AdjArgs& j, cudaStream_t s) {
    using namespace dev;
    const KM<double> m = make_km<double>(a);
    const d4* q = (const d4*)a.qm[p];
    const d4* gx = (const d4*)a.gx;
    const d4* gy = (const d4*)a.gy;
    const d4* ph = (const d4*)a.phi;
    const int B = 128;
    const int nf = nblocks(a.n_faces, B), nc = nblocks(a.n_cells, B);
    k_adj_face<SECOND, VISC><<<nf, B, 0, s>>>(m, a.n_faces, q, gx, gy, ph, (const d4*)j.v, (d4*)j.fbar);
    k_adj_cell<SECOND, VISC><<<nc, B, 0, s>>>(m, q, gx, gy, ph, (const d4*)j.fbar, (d4*)j.qbar, (d4*)j.gbx,
                                              (d4*)j.gby, (d4*)j.lw, (int4*)j.lt);
    k_adj_final<SECOND, VISC><<<nc, B, 0, s>>>(m, q, (const d4*)j.fbar, (const d4*)j.qbar, (const d4*)j.gbx,
                                               (const d4*)j.gby, (const d4*)j.lw, (const int4*)j.lt, (d4*)j.u,
                                               (d4*)j.bqbar);
}
}  // namespace

void enqueue_vjp(const StepArgs& a, int p, const AdjArgs& j, cudaStream_t s) {
    if (a.visc == 1) {
        if (a.second) vjp_launch<true, 1>(a, p, j, s);
        else vjp_launch<false, 1>(a, p, j, s);
    } else {
        if (a.second) vjp_launch<true, 0>(a, p, j, s);
        else vjp_launch<false, 0>(a, p, j, s);
    }
}

void enqueue_adjoint_update(int n, const void* lam0, const void* u, const void* g, const void* dt, double alpha,
                            double relax, void* lam_out, double* partials, cudaStream_t s) {
    dev::k_adj_update<<<(n + 255) / 256, 256, 0, s>>>(n, (const dev::d4*)lam0, (const dev::d4*)u,
                                                        (const dev::d4*)g, (const double*)dt, alpha, relax,
                                                        (dev::d4*)lam_out, partials);
}

void enqueue_objective_grad(const ForceArgs& f, double cx, double cy, void* g, cudaStream_t s) {
    dev::k_objective_grad<<<1, 1, 0, s>>>(f, cx, cy, (dev::d4*)g);
}

}  // namespace afx
