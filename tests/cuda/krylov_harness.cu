// The linear solver's kernels one at a time, on host arrays: the unit as it is
// shipped, and C entries around it (built by the tests that use it).
#include "../../aeroflex_gb300/csrc/afx_implicit.cu"

using namespace afx;
using namespace afx::dev;

namespace {

struct Buf {  // a device copy of a host array, copied back at the end if asked
    void* d = nullptr;
    void* h;
    size_t n;
    bool back;
    Buf(const void* host, size_t bytes, bool b = false) : h(const_cast<void*>(host)), n(bytes), back(b) {
        cudaMalloc(&d, n ? n : 16);
        if (h) cudaMemcpy(d, h, n, cudaMemcpyHostToDevice);
        else cudaMemset(d, 0, n);
    }
    ~Buf() {
        if (back) cudaMemcpy(h, d, n, cudaMemcpyDeviceToHost);
        cudaFree(d);
    }
    template <class U> U* p() const { return (U*)d; }
};

template <class T>
int sq(int n, int blocks, const T* w, double* out) {
    {
        Buf dw(w, n * sizeof(T)), part(nullptr, blocks * 8), cnt(nullptr, 4), o(out, 8, true);
        launch_pdl(k_imp_sq<T>, blocks, DOT_THREADS, 0, nullptr, n, dw.p<T>(), part.p<double>(), cnt.p<unsigned>(),
                   o.p<double>(), nullptr);
        if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    }
    return 0;
}

// Gram-Schmidt of w against the k + 1 vectors in V (given h1), and the step's
// column after rotations by zero angles: h2 and {hnext, res, stop, k} come back
template <class T>
int cgs(int n, int k, int blocks, const T* V, T* w, const double* h1, double g, double tol, double* h2, double* st) {
    GmresCtl c{};
    c.k = k;
    c.max_iters = 500;
    c.tol = tol;
    c.g[k] = g;
    for (int i = 0; i < GM_M; ++i) c.cs[i] = 1.0;
    {
        Buf dV(V, (size_t)(k + 1) * n * sizeof(T)), dw(w, n * sizeof(T), true), dh1(h1, (k + 1) * 8);
        Buf part(nullptr, blocks * (GM_M + 1) * 8), cnt(nullptr, 4), dh2(h2, (k + 1) * 8, true), sc(nullptr, 8);
        Buf dc(&c, sizeof(c), true);
        launch_pdl(k_imp_cgs<T>, blocks, DOT_THREADS, 0, nullptr, n, dV.p<T>(), dw.p<T>(), dh1.p<double>(),
                   part.p<double>(), cnt.p<unsigned>(), dh2.p<double>(), dc.p<GmresCtl>(), sc.p<double>());
        if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    }
    st[0] = c.hnext;
    st[1] = c.res;
    st[2] = c.stop;
    st[3] = c.k;
    return 0;
}

// One colour (rows c0 .. c0 + n - 1) of the sweep over x, with rt threads per row
template <class T>
int gs(int rt, int N, int c0, int n, int fwd, const int* col, const T* dinv, const T* off, const T* r, T* x) {
    {
        Buf dc(col, N * sizeof(int4)), di(dinv, 16 * (size_t)N * sizeof(T)), dof(off, 64 * (size_t)N * sizeof(T));
        Buf dr(r, 4 * (size_t)N * sizeof(T)), dx(x, 4 * (size_t)N * sizeof(T), true);
        const Ell e{nullptr, dc.p<int4>(), nullptr, nullptr, nullptr};
        if (rt == 4)
            launch_pdl(k_imp_gs<T, 4>, nb_(4LL * n, 128), 128, 0, nullptr, e, N, di.p<T>(), dof.p<T>(), c0, n, dr.p<T>(),
                       nullptr, 0LL, dx.p<T>(), nullptr, nullptr, fwd != 0);
        else
            launch_pdl(k_imp_gs<T, 1>, nb_(n, 128), 128, 0, nullptr, e, N, di.p<T>(), dof.p<T>(), c0, n, dr.p<T>(),
                       nullptr, 0LL, dx.p<T>(), nullptr, nullptr, fwd != 0);
        if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    }
    return 0;
}

}  // namespace

extern "C" {

int hk_gs_f32(int rt, int N, int c0, int n, int fwd, const int* col, const float* dinv, const float* off, const float* r,
              float* x) {
    return gs<float>(rt, N, c0, n, fwd, col, dinv, off, r, x);
}
int hk_gs_f64(int rt, int N, int c0, int n, int fwd, const int* col, const double* dinv, const double* off,
              const double* r, double* x) {
    return gs<double>(rt, N, c0, n, fwd, col, dinv, off, r, x);
}

int hk_sq_f32(int n, int blocks, const float* w, double* out) { return sq<float>(n, blocks, w, out); }
int hk_sq_f64(int n, int blocks, const double* w, double* out) { return sq<double>(n, blocks, w, out); }
int hk_cgs_f32(int n, int k, int blocks, const float* V, float* w, const double* h1, double g, double tol, double* h2,
               double* st) {
    return cgs<float>(n, k, blocks, V, w, h1, g, tol, h2, st);
}
int hk_cgs_f64(int n, int k, int blocks, const double* V, double* w, const double* h1, double g, double tol,
               double* h2, double* st) {
    return cgs<double>(n, k, blocks, V, w, h1, g, tol, h2, st);
}

}  // extern "C"
