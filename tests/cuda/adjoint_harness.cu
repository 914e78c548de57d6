// The integer FP64 operations and the hand-reversed face fluxes on the GPU, on
// host arrays: the adjoint's unit as it is shipped, and C entries around parts of it.
#include "../../aeroflex_gb300/csrc/afx_adjoint.cu"

using namespace afx;
using namespace afx::dev;

namespace ha {

struct Buf {
    void* d = nullptr;
    void* h;
    size_t n;
    Buf(void* host, size_t bytes) : h(host), n(bytes) {
        cudaMalloc(&d, n);
        cudaMemcpy(d, h, n, cudaMemcpyHostToDevice);
    }
    ~Buf() {
        cudaMemcpy(h, d, n, cudaMemcpyDeviceToHost);
        cudaFree(d);
    }
    template <class U> U* p() const { return (U*)d; }
};

// op 0 x / y, 1 x / (2 y) by twice(), 2 sqrt(|x|), 3 sqrt(x), 4 x y, 5 x < y,
// 6 x <= y, 7 (float)x and whether it is taken, 8 (double)(float)x
__global__ void k_ops(const int op, const int n, const double* x, const double* y, double* mine, double* theirs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = x[i], b = y[i];
    double m = 0, t = 0;
    if (op == 0) m = fp64::div(a, b), t = __ddiv_rn(a, b);
    if (op == 1) m = fp64::quot(a, fp64::twice(fp64::den(b))), t = __ddiv_rn(a, __dmul_rn(2.0, b));
    if (op == 2) m = fp64::root(fabs(a)), t = __dsqrt_rn(fabs(a));
    if (op == 3) m = fp64::root(a), t = __dsqrt_rn(a);
    if (op == 4) m = fp64::mul(a, b), t = __dmul_rn(a, b);
    if (op == 5) m = fp64::less(a, b), t = a < b;
    if (op == 6) m = fp64::less_equal(a, b), t = a <= b;
    if (op == 7) {
        uint32_t r;
        const bool ok = fp64::narrow(a, r);
        const float f = __double2float_rn(a);
        m = ok ? (double)r : -1.0;
        t = a == 0.0 || (fabs(a) >= 1.1754943508222875e-38 && fabs(a) < 0x1p128) ? (double)__float_as_uint(f) : -1.0;
    }
    if (op == 8) {
        const float f = __double2float_rn(a);
        m = fp64::widen(__float_as_uint(f));
        t = fabsf(f) < 1.17549435e-38f ? copysign(0.0, a) : (double)f;
    }
    mine[i] = m;
    theirs[i] = t;
}

// The seeds over all arguments the operations give them (24 bits of [1, 2), for
// the root [1, 4)): largest errors below and above the exact value, in units of
// the last place of [0.5, 1), 2^-24, in 1/256 of it
__global__ void k_seeds(const int root, int* worst) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;  // 2^23 (root: 2^24) threads
    const uint32_t u = (root && i >> 23 ? 0x40000001u : 0x3f800001u) + (i & 0x7fffffu);
    const double f = __uint_as_float(u);
    const double e = root ? 1.0 / sqrt(f) : 1.0 / f;
    const double s = __uint_as_float(root ? fp64::seed_rsqrt(u) : fp64::seed_rcp(u));
    const int d = (int)floor((s - e) * 0x1p32 + 0.5);
    if (d < 0) atomicMax(&worst[0], -d);
    else atomicMax(&worst[1], d);
}

// reverse (mine) and eight (laminar: sixteen) forward directions (theirs) of
// sum_m w_m F_m; per face: nx, ny, qL, qR, w, gx, gy (22 numbers)
__global__ void k_face(const int visc, const KM<double> m, const int n, const double* in, double* mine, double* theirs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double a[22], b[16], fwd[16];
    for (int k = 0; k < 22; ++k) a[k] = in[22 * i + k];
    for (int k = 0; k < 16; ++k) b[k] = fwd[k] = 0.0;
    const double *qL = a + 2, *qR = a + 6, *w = a + 10, *gx = a + 14, *gy = a + 18;
    roe_reverse(m.gamma, a[0], a[1], qL, qR, w, b, b + 4);
    if (visc) laminar_reverse(m, a[0], a[1], qL, qR, gx, gy, w, b, b + 4, b + 8, b + 12);
#pragma unroll 1
    for (int dir = 0; dir < (visc ? 16 : 8); ++dir) {
        Dual x[16], F[4];
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = Dual(k < 8 ? a[2 + k] : a[6 + k], k == dir ? 1.0 : 0.0);
        roe_flux<Dual>(Dual(m.gamma), Dual(a[0]), Dual(a[1]), x, x + 4, F);
        if (visc)
            laminar_flux<Dual>(Dual(m.gamma), Dual(m.R), Dual(m.mu), Dual(m.kheat), Dual(a[0]), Dual(a[1]), x, x + 4,
                               x + 8, x + 12, F);
        double t = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) t += w[k] * F[k].d;
        fwd[dir] = t;
    }
    for (int k = 0; k < 16; ++k) {
        mine[16 * i + k] = b[k];
        theirs[16 * i + k] = fwd[k];
    }
}

}  // namespace ha
using namespace ha;

extern "C" {

int ha_ops(int op, int n, double* x, double* y, double* mine, double* theirs) {
    Buf a(x, n * 8), b(y, n * 8), c(mine, n * 8), d(theirs, n * 8);
    k_ops<<<(n + 255) / 256, 256>>>(op, n, a.p<double>(), b.p<double>(), c.p<double>(), d.p<double>());
    return cudaDeviceSynchronize() != cudaSuccess;
}

int ha_seeds(int root, int* worst) {
    Buf a(worst, 2 * sizeof(int));
    k_seeds<<<(root ? 1 << 24 : 1 << 23) / 256, 256>>>(root, a.p<int>());
    return cudaDeviceSynchronize() != cudaSuccess;
}

int ha_face(int visc, int n, double gamma, double R, double mu, double kheat, double* in, double* mine, double* theirs) {
    KM<double> m{};
    m.gamma = gamma;
    m.R = R;
    m.mu = mu;
    m.kheat = kheat;
    Buf a(in, n * 22 * 8), c(mine, n * 16 * 8), d(theirs, n * 16 * 8);
    k_face<<<(n + 63) / 64, 64>>>(visc, m, n, a.p<double>(), c.p<double>(), d.p<double>());
    return cudaDeviceSynchronize() != cudaSuccess;
}

}  // extern "C"
