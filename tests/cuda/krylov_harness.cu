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

}  // namespace

extern "C" {

int hk_sq_f32(int n, int blocks, const float* w, double* out) { return sq<float>(n, blocks, w, out); }
int hk_sq_f64(int n, int blocks, const double* w, double* out) { return sq<double>(n, blocks, w, out); }

}  // extern "C"
