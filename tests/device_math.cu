// Entries to the functions of the kernels' headers, so that tests run the code that
// the kernels run: host entries to the __host__ __device__ ones, and a kernel per
// device function that takes one array element per thread (host arrays in and out).
#include <vector>
#include "pic_adjoint.cuh"
#include "pic_plain_math.cuh"

namespace {
__global__ void k_div(int n, const double *a, const double *h, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = pic::div_by(a[i], h[i], 1.0 / h[i]);
}
__global__ void k_trunc(int n, const double *t, int *floor_i, double *floor_v, int *trunc_i, int *exact) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    floor_v[i] = pic::floor_pos(t[i], floor_i[i]);
    bool e = true;
    trunc_i[i] = pic::trunc_checked(t[i], e);
    exact[i] = e;
}
// the two contributions s and r of a node in quanta: its sums, with the 64-bit and
// with the int32 remainder word of scale 2^bits
__global__ void k_split(int n, const double *s, const double *r, int bits, long long *wide, long long *narrow) {
    __shared__ unsigned w[4 * 64];  // a node per thread, its words 64 apart
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned *m = w + threadIdx.x;
    if (i >= n) return;
    m[0] = m[64] = m[128] = m[192] = 0u;
    pic::fx_put2(m, 64, s[i]);
    pic::fx_put2(m, 64, r[i]);
    pic::fx_get<false>(m, 64, wide[2 * i], wide[2 * i + 1]);
    const double scale = ldexp(1.0, bits);
    m[0] = m[64] = m[128] = m[192] = 0u;
    pic::fx_put_lo32(m, 64, s[i], scale);
    pic::fx_put_lo32(m, 64, r[i], scale);
    pic::fx_get<true>(m, 64, narrow[2 * i], narrow[2 * i + 1]);
}
// device copies of host arrays, freed together
struct Arrays {
    std::vector<void *> p;
    bool ok = true;
    template <class T>
    T *get(const T *host, size_t n) {
        void *d = nullptr;
        ok = ok && cudaMalloc(&d, n * sizeof(T)) == cudaSuccess;
        if (ok) p.push_back(d);
        if (ok && host) ok = cudaMemcpy(d, host, n * sizeof(T), cudaMemcpyHostToDevice) == cudaSuccess;
        return (T *)d;
    }
    template <class T>
    void put(T *host, const T *d, size_t n) {
        ok = ok && cudaMemcpy(host, d, n * sizeof(T), cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    ~Arrays() {
        for (void *d : p) cudaFree(d);
    }
};
}  // namespace

extern "C" {
int dm_out_mixed_align() { return (int)alignof(pic::OutMixed); }
int dm_out_mixed_size() { return (int)sizeof(pic::OutMixed); }
int dm_max_slots() { return pic::kMaxSlots; }
int dm_max_slot(int it) { return pic::max_slot(it); }
int dm_max_cleared(int it) { return pic::max_cleared(it); }
int dm_no_quantum() { return pic::kNoQuantum; }
int dm_quantum_plain(int E, unsigned hi) {
    return pic::quantum_for(E, pic::exponent_hi(hi), pic::kKeepPlain, pic::kLeastPlain);
}
int dm_quantum_mixed(int E, unsigned bits) {
    return pic::quantum_for(E, pic::exponent_f(bits), pic::kKeepMix, pic::kLeastMix);
}
// 0: done
int dm_gpu_div(int n, const double *a, const double *h, double *out) {
    Arrays A;
    const double *da = A.get(a, n), *dh = A.get(h, n);
    double *o = A.get<double>(nullptr, n);
    if (!A.ok) return 1;
    k_div<<<(n + 255) / 256, 256>>>(n, da, dh, o);
    A.put(out, o, n);
    return !A.ok;
}
int dm_gpu_trunc(int n, const double *t, int *floor_i, double *floor_v, int *trunc_i, int *exact) {
    Arrays A;
    const double *dt = A.get(t, n);
    int *fi = A.get<int>(nullptr, n), *ti = A.get<int>(nullptr, n), *ex = A.get<int>(nullptr, n);
    double *fv = A.get<double>(nullptr, n);
    if (!A.ok) return 1;
    k_trunc<<<(n + 255) / 256, 256>>>(n, dt, fi, fv, ti, ex);
    A.put(floor_i, fi, n);
    A.put(floor_v, fv, n);
    A.put(trunc_i, ti, n);
    A.put(exact, ex, n);
    return !A.ok;
}
int dm_gpu_split(int n, const double *s, const double *r, int bits, long long *wide, long long *narrow) {
    Arrays A;
    const double *ds = A.get(s, n), *dr = A.get(r, n);
    long long *w = A.get<long long>(nullptr, 2 * (size_t)n), *v = A.get<long long>(nullptr, 2 * (size_t)n);
    if (!A.ok) return 1;
    k_split<<<(n + 63) / 64, 64>>>(n, ds, dr, bits, w, v);
    A.put(wide, w, 2 * (size_t)n);
    A.put(narrow, v, 2 * (size_t)n);
    return !A.ok;
}
}
