// Differentiable run of the FP32 mixed form: the fixed-order push and the
// adjoint particle kernels.  Same arithmetic as k_push_mixed (cell units,
// FP32 offsets and momenta, rsqrtf).  A CTA's current is summed in its window in
// 64-bit fixed point and added to the FP64 global J; the adjoint runs in FP32 per
// particle, and its field adjoints are summed likewise.  Field transposes and the
// host sequence: pic_adjoint.cu.
#include <cuda_runtime.h>
#include <math.h>
#include "pic0buf.h"
#include "pic_internal.cuh"
#include "pic_handle.cuh"
#include <type_traits>
#include "pic_adjoint.cuh"

namespace pic {

namespace {

constexpr int kT = 256;
constexpr float kOneBelow = 0.99999994f;  // largest float < 1

// GetField in cell units (k_push_mixed): the node-staggered tap is 2 with
// weight 1 - o, the centre-staggered tap 2 + (o >= 1/2) with weight
// (1/2 or 3/2) - o; component c is node-staggered along d when
// (E_c and d == c) or (H_c and d != c)
struct MTaps {
    int tc[3];
    float wn[3], wc[3];
};
__device__ __forceinline__ void taps_mixed(const float x[3], MTaps &T) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
        T.tc[d] = 2 + (x[d] >= 0.5f);
        T.wn[d] = 1.f - x[d];
        T.wc[d] = (T.tc[d] == 2 ? 0.5f : 1.5f) - x[d];
    }
}
__device__ __forceinline__ void comp_taps_m(const MTaps &T, int c, int t[3], float w[3]) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
        bool nd = c < 3 ? d == c : d != c - 3;
        t[d] = nd ? 2 : T.tc[d];
        w[d] = nd ? T.wn[d] : T.wc[d];
    }
}
// trilinear interpolation of the eight taps at A, A + dx, ...
__device__ __forceinline__ float interp_gm(const float *__restrict__ A, int dx, int dy, const float w[3]) {
    const int dz = 1;
    float sx = w[0], sy = w[1], sz = w[2];
    float sx1 = 1.f - sx, sy1 = 1.f - sy, sz1 = 1.f - sz;
    float t1 = sx * (sy * (sz * A[0] + sz1 * A[dz]) + sy1 * (sz * A[dy] + sz1 * A[dy + dz]));
    float t2 = sx1 * (sy * (sz * A[dx] + sz1 * A[dx + dz]) + sy1 * (sz * A[dx + dy] + sz1 * A[dx + dy + dz]));
    return t1 + t2;
}
// A particle's view of the fields: the CTA's window in shared memory (WIN) or
// the arrays in global memory; base[c] points at the node of its cell
template <bool WIN>
struct FieldViewM {
    const float *base[6];
    int dx, dy;
};
template <class V>
__device__ __forceinline__ void gather_fields_m(const V &A, const float x[3], float F[6]) {
    MTaps T;
    taps_mixed(x, T);
#pragma unroll
    for (int c = 0; c < 6; c++) {
        int t[3];
        float w[3];
        comp_taps_m(T, c, t, w);
        F[c] = interp_gm(A.base[c] + (t[0] - 2) * A.dx + (t[1] - 2) * A.dy + (t[2] - 2), A.dx, A.dy, w);
    }
}

// Particle::Move in FP32 as in k_push_mixed, with the adjoint's intermediates
struct BorisM {
    float t, u[3], g1, ps, b[3], s[3], rs, up[3], pp[3], ig, ct[3], xe[3];
};
__device__ __forceinline__ void boris_mixed(float tau1, const float ct[3], const float p[3], const float F[6],
                                            const float xs[3], BorisM &B) {
    B.t = tau1;
    float pu = p[0], pv = p[1], pw = p[2];
    pu += tau1 * F[0];
    pv += tau1 * F[1];
    pw += tau1 * F[2];
    B.u[0] = pu; B.u[1] = pv; B.u[2] = pw;
    B.g1 = rsqrtf(pu * pu + pv * pv + pw * pw + 1.f);
    float ps = tau1 * B.g1;
    B.ps = ps;
    float bx = ps * F[3], by = ps * F[4], bz = ps * F[5];
    B.b[0] = bx; B.b[1] = by; B.b[2] = bz;
    float su = pu + pv * bz - pw * by;
    float sv = pv + pw * bx - pu * bz;
    float sw = pw + pu * by - pv * bx;
    B.s[0] = su; B.s[1] = sv; B.s[2] = sw;
    float q1 = bx * bx, q2 = by * by, q3 = bz * bz, q4 = bx * by, q5 = by * bz, q6 = bz * bx;
    float rs = 1.f / (q1 + 1.f + q2 + q3);
    B.rs = rs;
    float pu1 = ((q1 + 1.f) * su + (q4 + bz) * sv + (q6 - by) * sw) * rs;
    float pv1 = ((q4 - bz) * su + (q2 + 1.f) * sv + (q5 + bx) * sw) * rs;
    float pw1 = ((q6 + by) * su + (q5 - bx) * sv + (q3 + 1.f) * sw) * rs;
    B.up[0] = pu1; B.up[1] = pv1; B.up[2] = pw1;
    pu = pu1 + F[0] * tau1;
    pv = pv1 + F[1] * tau1;
    pw = pw1 + F[2] * tau1;
    B.pp[0] = pu; B.pp[1] = pv; B.pp[2] = pw;
    B.ig = rsqrtf(pu * pu + pv * pv + pw * pw + 1.f);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        B.ct[d] = ct[d];
        B.xe[d] = xs[d] + ct[d] * (B.ig * B.pp[d]);
    }
}

// cell-centre crossings and the split point (split_point in pic_mixed.cu)
struct SplitM {
    int m, i1[3], i2[3];
    float x2[3], sr;
};
__device__ __forceinline__ void split_mixed(const float xs[3], const float xe[3], SplitM &S) {
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        S.i1[d] = 2 + (xs[d] >= 0.5f);
        S.i2[d] = 2 + (xe[d] >= 0.5f) + (xe[d] >= 1.5f) - (xe[d] < -0.5f);
        float dl = xe[d] - xs[d];
        bool c = S.i1[d] != S.i2[d];
        num += c ? (0.5f - xs[d]) * dl : 0.f;
        den += c ? dl * dl : 0.f;
    }
    S.m = 4 * (S.i1[0] != S.i2[0]) + 2 * (S.i1[1] != S.i2[1]) + (S.i1[2] != S.i2[2]);
    const bool any = den > 0.f;
    const float sr = any ? __fdividef(num, den) : 1.f;
    S.sr = sr;
#pragma unroll
    for (int d = 0; d < 3; d++) S.x2[d] = (S.i1[d] != S.i2[d]) ? 0.5f : xs[d] + (xe[d] - xs[d]) * sr;
}
__device__ __forceinline__ bool stencil_ok(const int iv[3]) {
    return iv[0] >= 2 && iv[0] <= 3 && iv[1] >= 2 && iv[1] <= 3 && iv[2] >= 2 && iv[2] <= 3;
}

// pqr_mixed (pic_mixed.cu): add(component, x, y, z node offset from the
// particle's cell, FP32 contribution); nothing where the segment has no length
template <class Add>
__device__ __forceinline__ void seg_mixed(const int iv[3], const float xs[3], const float xe[3], float wx, float wy,
                                          float wz, Add add) {
    float dx = 0.5f * (xs[0] + xe[0]) - ((float)iv[0] - 2.5f);
    float dy = 0.5f * (xs[1] + xe[1]) - ((float)iv[1] - 2.5f);
    float dz = 0.5f * (xs[2] + xe[2]) - ((float)iv[2] - 2.5f);
    float dx1 = 1.f - dx, dy1 = 1.f - dy, dz1 = 1.f - dz;
    float su = xe[0] - xs[0], sv = xe[1] - xs[1], sw = xe[2] - xs[2];
    const float r12 = 1.f / 12.f;
    float s1 = sv * sw * r12, s2 = su * sw * r12, s3 = su * sv * r12;
    su *= wx;
    sv *= wy;
    sw *= wz;
    if (su == 0.f && sv == 0.f && sw == 0.f) return;
    const int a = iv[0] - 2, b = iv[1] - 2, c = iv[2] - 2;
    add(0, a, b, c, su * (dy1 * dz1 + s1));
    add(0, a, b, c + 1, su * (dy1 * dz - s1));
    add(0, a, b + 1, c, su * (dy * dz1 - s1));
    add(0, a, b + 1, c + 1, su * (dy * dz + s1));
    add(1, a, b, c, sv * (dx1 * dz1 + s2));
    add(1, a, b, c + 1, sv * (dx1 * dz - s2));
    add(1, a + 1, b, c, sv * (dx * dz1 - s2));
    add(1, a + 1, b, c + 1, sv * (dx * dz + s2));
    add(2, a, b, c, sw * (dx1 * dy1 + s3));
    add(2, a, b + 1, c, sw * (dx1 * dy - s3));
    add(2, a + 1, b, c, sw * (dx * dy1 - s3));
    add(2, a + 1, b + 1, c, sw * (dx * dy + s3));
}

// transpose of seg_mixed (cell units: h = 1, weights wx, wy, wz); L: lambda_J
// at the particle's cell (float in the window, double in global memory)
template <class T>
__device__ __forceinline__ void seg_mixed_rev(const T *L0, const T *L1, const T *L2, int ex, int ey, const int iv[3],
                                              const float xs[3], const float xe[3], float cu, float cv, float cw,
                                              float gs[3], float ge[3]) {
    float dx = 0.5f * (xs[0] + xe[0]) - ((float)iv[0] - 2.5f);
    float dy = 0.5f * (xs[1] + xe[1]) - ((float)iv[1] - 2.5f);
    float dz = 0.5f * (xs[2] + xe[2]) - ((float)iv[2] - 2.5f);
    float dx1 = 1.f - dx, dy1 = 1.f - dy, dz1 = 1.f - dz;
    float Dx = xe[0] - xs[0], Dy = xe[1] - xs[1], Dz = xe[2] - xs[2];
    const float r12 = 1.f / 12.f;
    float s1 = Dy * Dz * r12, s2 = Dx * Dz * r12, s3 = Dx * Dy * r12;
    float Ax = cu * Dx, Ay = cv * Dy, Az = cw * Dz;
    const int n = (iv[0] - 2) * ex + (iv[1] - 2) * ey + (iv[2] - 2);
    const int ez = 1;
    float Lx0 = (float)L0[n], Lx1 = (float)L0[n + ez], Lx2 = (float)L0[n + ey], Lx3 = (float)L0[n + ey + ez];
    float Ly0 = (float)L1[n], Ly1 = (float)L1[n + ez], Ly2 = (float)L1[n + ex], Ly3 = (float)L1[n + ex + ez];
    float Lz0 = (float)L2[n], Lz1 = (float)L2[n + ey], Lz2 = (float)L2[n + ex], Lz3 = (float)L2[n + ex + ey];
    float Fx = Lx0 * (dy1 * dz1 + s1) + Lx1 * (dy1 * dz - s1) + Lx2 * (dy * dz1 - s1) + Lx3 * (dy * dz + s1);
    float Fy = Ly0 * (dx1 * dz1 + s2) + Ly1 * (dx1 * dz - s2) + Ly2 * (dx * dz1 - s2) + Ly3 * (dx * dz + s2);
    float Fz = Lz0 * (dx1 * dy1 + s3) + Lz1 * (dx1 * dy - s3) + Lz2 * (dx * dy1 - s3) + Lz3 * (dx * dy + s3);
    float Kx = Lx0 - Lx1 - Lx2 + Lx3, Ky = Ly0 - Ly1 - Ly2 + Ly3, Kz = Lz0 - Lz1 - Lz2 + Lz3;
    float gDx = cu * Fx + (Ay * Ky * Dz + Az * Kz * Dy) * r12;
    float gDy = cv * Fy + (Ax * Kx * Dz + Az * Kz * Dx) * r12;
    float gDz = cw * Fz + (Ax * Kx * Dy + Ay * Ky * Dx) * r12;
    float gdx = Ay * (-Ly0 * dz1 - Ly1 * dz + Ly2 * dz1 + Ly3 * dz) + Az * (-Lz0 * dy1 - Lz1 * dy + Lz2 * dy1 + Lz3 * dy);
    float gdy = Ax * (-Lx0 * dz1 - Lx1 * dz + Lx2 * dz1 + Lx3 * dz) + Az * (-Lz0 * dx1 + Lz1 * dx1 - Lz2 * dx + Lz3 * dx);
    float gdz = Ax * (-Lx0 * dy1 + Lx1 * dy1 - Lx2 * dy + Lx3 * dy) + Ay * (-Ly0 * dx1 + Ly1 * dx1 - Ly2 * dx + Ly3 * dx);
    gs[0] += 0.5f * gdx - gDx; ge[0] += 0.5f * gdx + gDx;
    gs[1] += 0.5f * gdy - gDy; ge[1] += 0.5f * gdy + gDy;
    gs[2] += 0.5f * gdz - gDz; ge[2] += 0.5f * gdz + gDz;
}

// transpose of the split point (crossing planes at 1/2; axes as template arguments)
template <int O>
__device__ __forceinline__ float rbx_rev_m(float sr, const float xo[3], const float xn[3], const float g2[3],
                                           float gx[3], float gn[3]) {
    gx[O] += g2[O] * (1.f - sr);
    gn[O] += g2[O] * sr;
    return g2[O] * (xn[O] - xo[O]);
}
template <int A, int O0, int O1>
__device__ __forceinline__ void split_rev1_m(const SplitM &S, const float xo[3], const float xn[3],
                                             const float g2[3], float gx[3], float gn[3]) {
    const float sr = S.sr;
    float lsr = rbx_rev_m<O0>(sr, xo, xn, g2, gx, gn) + rbx_rev_m<O1>(sr, xo, xn, g2, gx, gn);
    float D = xn[A] - xo[A];
    gx[A] += lsr * (0.5f - xn[A]) / (D * D);
    gn[A] -= lsr * sr / D;
}
template <int A, int B, int O>
__device__ __forceinline__ void split_rev2_m(const SplitM &S, const float xo[3], const float xn[3],
                                             const float g2[3], float gx[3], float gn[3]) {
    const float sr = S.sr;
    float lsr = rbx_rev_m<O>(sr, xo, xn, g2, gx, gn);
    float Da = xn[A] - xo[A], Db = xn[B] - xo[B];
    float f = lsr / (Da * Da + Db * Db);
    float ca = 0.5f - xo[A], cb = 0.5f - xo[B];
    gx[A] += f * (-Da - ca + 2.f * sr * Da);
    gn[A] += f * (ca - 2.f * sr * Da);
    gx[B] += f * (-Db - cb + 2.f * sr * Db);
    gn[B] += f * (cb - 2.f * sr * Db);
}
__device__ __forceinline__ void split_rev_m(const SplitM &S, const float xo[3], const float xn[3], const float g2[3],
                                            float gx[3], float gn[3]) {
    switch (S.m) {
        case 1: split_rev1_m<2, 0, 1>(S, xo, xn, g2, gx, gn); break;
        case 2: split_rev1_m<1, 0, 2>(S, xo, xn, g2, gx, gn); break;
        case 4: split_rev1_m<0, 1, 2>(S, xo, xn, g2, gx, gn); break;
        case 3: split_rev2_m<1, 2, 0>(S, xo, xn, g2, gx, gn); break;
        case 5: split_rev2_m<0, 2, 1>(S, xo, xn, g2, gx, gn); break;
        case 6: split_rev2_m<0, 1, 2>(S, xo, xn, g2, gx, gn); break;
        default: break;  // 7: the centre of the cell
    }
}

// per-species constants of the particle kernels (formed once per CTA: the FP64
// divisions behind them cost more than a particle's FP32 work)
struct MixConst {
    float tau1, ct[3], w[3];
};
__device__ __forceinline__ MixConst mix_const(const Grid &g, const MixSp &S) {
    MixConst K;
    K.tau1 = (float)(S.q_m * g.tau * 0.5);
    K.ct[0] = (float)(g.tau / g.hx); K.ct[1] = (float)(g.tau / g.hy); K.ct[2] = (float)(g.tau / g.hz);
    K.w[0] = (float)(S.m * g.hx / g.tau); K.w[1] = (float)(S.m * g.hy / g.tau); K.w[2] = (float)(S.m * g.hz / g.tau);
    return K;
}

constexpr int kW = kT / 32;          // warps per CTA
constexpr int kDirectBlocks = 4, kDirectAdjBlocks = 3;  // CTAs per SM of the kernels without a window
constexpr int kQueueMix = 48;        // queued second segments per warp: drained at 16, at most 15 + 32
constexpr int kFlatWindowMix = 800;  // nodes of the forward's window: 56 KB of shared memory, three CTAs per SM (80 registers)
constexpr int kAdjWindowMix = 672;   // nodes of the adjoint's: 73 KB, three

// shared memory of a thread's next particle (cp.async, as in k_push_plain): N values, then the cell
template <int N>
struct NextMix {
    float *v;
    __device__ __forceinline__ NextMix(void *base) {
        v = (float *)base + (threadIdx.x >> 5) * ((N + 1) * 32) + (threadIdx.x & 31);
    }
    static constexpr size_t bytes = (size_t)kW * (N + 1) * 32 * sizeof(float);
    __device__ __forceinline__ void start(const MixSp &S, float *const *lam, int64_t j) const {
#pragma unroll
        for (int a = 0; a < 6; a++) cp_async<4>(v + 32 * a, S.v[a] + j);
        if (N > 6)
#pragma unroll
            for (int a = 0; a < 6; a++) cp_async<4>(v + 32 * (6 + a), lam[a] + j);
        cp_async<4>(v + 32 * N, S.cell + j);
    }
    __device__ __forceinline__ int cell() const { return __float_as_int(v[32 * N]); }
    __device__ __forceinline__ void take3(int from, float x[3]) const {
#pragma unroll
        for (int d = 0; d < 3; d++) x[d] = v[32 * (from + d)];
    }
};

// stages the window's nodes of N arrays src[c] into dst (cn floats apart)
template <int N, class T, bool WRAP>
__device__ __forceinline__ void stage_window_m(const Grid &g, const AdjWindow<WRAP> &w, int cn, const T *const *src, float *dst) {
    for (int e = threadIdx.x; e < w.nn; e += blockDim.x) {
        size_t n;
        if (!w.grid_node(g, e, n)) continue;
#pragma unroll
        for (int q = 0; q < N; q++) dst[q * cn + e] = (float)src[q][n];
    }
}

// ---- fixed-order push of the FP32 form.  One CTA per chunk of consecutive
// particles with the chunk's window staged in shared memory, as
// k_flat_push_plain; the FP32 contributions are summed in 64-bit fixed point
// (quantum 2^-62 of the light-speed bound of the chunk, but at least 2^-51 of one
// particle's: 2^-52 |m| of rounding beside the 2^-25 |m| h / tau that an offset's own
// FP32 rounding makes) and added to the FP64 global J once.  DIRECT: no window (see
// AdjState::direct_from).
// Bound: instruction issue (1059 instructions per 32 particles, issue slots 65 %
// busy).  128x32x32 cells, 12.6M particles: 0.916 -> 0.635 ms per step, with the
// window's strides at compile time and chained launches 0.587 (before:
// taps gathered from and currents added to global memory; four CTAs per SM at
// 64 registers: 0.688; lanes spread over 4 or 8 places: 0.625, 0.660, and slower
// at 3M particles).
template <bool DIRECT>
__global__ void __launch_bounds__(kT, DIRECT ? kDirectBlocks : 3) k_flat_push_mixed(const __grid_constant__ MixParams P) {
    chain_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ AdjWindow<false> sWin;
    __shared__ int sRed[15 * kW], sQn[kW], sFar;
    __shared__ double sQ, sInvQ;
    __shared__ MixConst sK;
    const Grid &g = P.g;
    const AdjChunk ch = P.chunks[blockIdx.x];
    const int s = ch.species, count = ch.count;
    const MixSp &S = P.sp[s];
    unsigned char *sTail = smem_raw + (size_t)kFlatWindowMix * 48;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *qd = (float *)sTail + warp * 7 * kQueueMix;  // x2, xe, then the cell and class code
    const NextMix<6> next(sTail + (size_t)kW * 7 * kQueueMix * sizeof(float));
    AdjWindow<false> w{};
    if (!DIRECT) {
        if ((int)threadIdx.x < count) next.start(S, nullptr, ch.first + threadIdx.x);
        w = chunk_window(g, S.cell + ch.first, count, kFlatWindowMix, sRed, &sWin);
    }
    // (see AdjWindow: the strides at compile time where the window has them)
    auto body = [&](auto fixed) {
    constexpr bool FIX = decltype(fixed)::value;
    const int SZ = FIX ? kFixSZ : w.SZ, dX = FIX ? kFixSX : w.SX, dY = SZ, nn = w.nn;
    const int cn = FIX ? kFlatWindowMix : nn;  // between the components
    unsigned *sLo = (unsigned *)smem_raw, *sHi = sLo + 3 * cn;
    float *sF = (float *)(sHi + 3 * cn);
    if (threadIdx.x == 0) {
        int e2, e1;
        frexp(2.5 * fabs(S.m) * (double)count, &e2);
        frexp(1.0834 * fabs(S.m), &e1);
        const int eq = max(e2 - 62, e1 - 51);
        sQ = ldexp(1.0, eq);
        sInvQ = ldexp(1.0, -eq);
        sK = mix_const(g, S);
        sFar = 0;
    }
    const float *src[6] = {P.E[0], P.E[1], P.E[2], P.H[0], P.H[1], P.H[2]};
    if (!DIRECT) {
        stage_window_m<6>(g, w, cn, src, sF);
        for (int e = threadIdx.x; e < 6 * cn; e += blockDim.x) sLo[e] = 0u;
        if (lane == 0) sQn[warp] = 0;
    }
    __syncthreads();
    const MixConst &K = sK;
    const double inv_q = sInvQ;
    const int nc[3] = {g.nx, g.ny, g.nz};
    unsigned bad = 0;
    int qn = 0;
    auto put = [&](int n0) {
        return [=](int c, int a, int b, int k, float v) {
            const int n = c * cn + n0 + a * dX + b * dY + k;
            const long long iv = __double_as_longlong(fma((double)v, inv_q, kRound)) - 0x4338000000000000ll;
            if (iv) shared_add64(sLo + n, sHi + n, iv);
        };
    };
    for (int jw = threadIdx.x - lane;; jw += blockDim.x) {
        const bool tail = jw >= count;
        if (tail && qn == 0) break;
        const int jc = jw + lane;
        const int64_t j = ch.first + jc;
        int cell = -1;
        float xs[3], p[3];
        if (DIRECT) {
            if (jc < count) {
                cell = S.cell[j];
#pragma unroll
                for (int d = 0; d < 3; d++) { xs[d] = S.v[d][j]; p[d] = S.v[3 + d][j]; }
            }
        } else {
            cp_async_wait_all();
            if (jc < count) {
                cell = next.cell();
                next.take3(0, xs);
                next.take3(3, p);
            }
            __syncwarp();  // the reads come before the next copies into the same place
            if (jc + (int)blockDim.x < count) next.start(S, nullptr, j + blockDim.x);
        }
        if (cell >= 0) {
            int c3[3];
            g.cell_ijk(cell, c3[0], c3[1], c3[2]);
            int u3[3], n0 = 0;
            const bool in = !DIRECT && w.place(c3, dX, dY, u3, n0);
            if (!DIRECT && !in) atomicAdd(&sFar, 1);
            float F[6];
            if (in) {
                FieldViewM<true> V;
#pragma unroll
                for (int c = 0; c < 6; c++) V.base[c] = sF + c * cn + n0;
                V.dx = dX; V.dy = dY;
                gather_fields_m(V, xs, F);
            } else {
                FieldViewM<false> V;
#pragma unroll
                for (int c = 0; c < 6; c++) V.base[c] = src[c] + g.node(c3[0], c3[1], c3[2]);
                V.dx = g.NY * g.pz; V.dy = g.pz;
                gather_fields_m(V, xs, F);
            }
            BorisM B;
            boris_mixed(K.tau1, K.ct, p, F, xs, B);
            if (!(isfinite(B.pp[0]) && isfinite(B.pp[1]) && isfinite(B.pp[2]))) bad |= ST_NAN;
            float xe[3] = {B.xe[0], B.xe[1], B.xe[2]};
            SplitM SP;
            split_mixed(xs, xe, SP);
            if (!stencil_ok(SP.i2) || !(isfinite(xe[0]) && isfinite(xe[1]) && isfinite(xe[2]))) {
                bad |= ST_STENCIL;
            } else if (in) {
                seg_mixed(SP.i1, xs, SP.x2, K.w[0], K.w[1], K.w[2], put(n0));
                // the second segment: from a cell-centre plane, or the rounding of
                // x2 = xs + (xe - xs) where none is crossed
                if (SP.x2[0] != xe[0] || SP.x2[1] != xe[1] || SP.x2[2] != xe[2]) {
                    const int e = atomicAdd(&sQn[warp], 1);
#pragma unroll
                    for (int d = 0; d < 3; d++) {
                        qd[d * kQueueMix + e] = SP.x2[d];
                        qd[(3 + d) * kQueueMix + e] = xe[d];
                    }
                    qd[6 * kQueueMix + e] =
                        __int_as_float((n0 << 3) | (SP.i2[0] - 2) | ((SP.i2[1] - 2) << 1) | ((SP.i2[2] - 2) << 2));
                }
            } else {
                auto far = [&](int c, int a, int b, int k, float v) {
                    atomicAdd(&P.J[c][g.node(c3[0] + a, c3[1] + b, c3[2] + k)], (double)v);
                };
                seg_mixed(SP.i1, xs, SP.x2, K.w[0], K.w[1], K.w[2], far);
                seg_mixed(SP.i2, SP.x2, xe, K.w[0], K.w[1], K.w[2], far);
            }
            // new cell (Reflect and migration in cell units, as k_push_mixed)
#pragma unroll
            for (int d = 0; d < 3; d++) {
                if (xe[d] >= 1.f) {
                    xe[d] -= 1.f;
                    c3[d] = c3[d] + 1 == nc[d] ? 0 : c3[d] + 1;
                } else if (xe[d] < 0.f) {
                    xe[d] += 1.f;
                    c3[d] = c3[d] == 0 ? nc[d] - 1 : c3[d] - 1;
                }
                xe[d] = fminf(fmaxf(xe[d], 0.f), kOneBelow);
            }
            const MixOut &O = P.out[s];
            O.cell[j] = g.cell_of(c3[0], c3[1], c3[2]);
            O.v[0][j] = xe[0]; O.v[1][j] = xe[1]; O.v[2][j] = xe[2];
            O.v[3][j] = B.pp[0]; O.v[4][j] = B.pp[1]; O.v[5][j] = B.pp[2];
        }
        if (DIRECT) continue;
        // ---- the warp's queued second segments, one per lane
        __syncwarp();
        qn = sQn[warp];
        if (qn >= (tail ? 1 : 16)) {
            const int d = qn < 32 ? qn : 32;
            if (lane < d) {
                const int e = qn - d + lane, code = __float_as_int(qd[6 * kQueueMix + e]);
                const int iv[3] = {2 + (code & 1), 2 + ((code >> 1) & 1), 2 + ((code >> 2) & 1)};
                float sa[3], sb[3];
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    sa[q] = qd[q * kQueueMix + e];
                    sb[q] = qd[(3 + q) * kQueueMix + e];
                }
                seg_mixed(iv, sa, sb, K.w[0], K.w[1], K.w[2], put(code >> 3));
            }
            qn -= d;
            __syncwarp();
            if (lane == 0) sQn[warp] = qn;
        }
        __syncwarp();
    }
    if (!DIRECT) {
        __syncthreads();
        if (threadIdx.x == 0 && P.far && sFar) atomicAdd(P.far, sFar);
        for (int e = threadIdx.x; e < 3 * nn; e += blockDim.x) {
            const int comp = e / nn, r = e - comp * nn, a = comp * cn + r;
            const long long v = (long long)(((unsigned long long)sHi[a] << 32) | sLo[a]);
            size_t n;
            if (v == 0 || !w.grid_node(g, r, n)) continue;
            atomicAdd(&P.J[comp][n], (double)v * sQ);
        }
    }
    if (bad) atomicOr(&P.st->flags, bad);
    };
    if (!DIRECT && w.fixed()) body(std::true_type{});
    else body(std::false_type{});
}

// The reverse of one particle's step up to the adjoint of its interpolated
// fields (reverse_particle in pic_adjoint.cu): in gn, lP the incoming lambda_x
// and lambda_p, out gx, lu and lF
template <class V, class T>
__device__ __forceinline__ void reverse_particle_m(const MixConst &K, const V &A, const T *L0, const T *L1, const T *L2,
                                                   int lx, int ly, const float xs[3], const float p[3], float gn[3],
                                                   float lP[3], float gx[3], float lu[3], float lF[6]) {
    float F[6];
    gather_fields_m(A, xs, F);
    BorisM B;
    boris_mixed(K.tau1, K.ct, p, F, xs, B);
    SplitM SP;
    split_mixed(xs, B.xe, SP);
#pragma unroll
    for (int d = 0; d < 3; d++) gx[d] = 0.f;
    if (stencil_ok(SP.i2)) {
        float g2[3] = {0.f, 0.f, 0.f}, sb[3];
        // without a crossing the first segment is the whole step
#pragma unroll
        for (int d = 0; d < 3; d++) sb[d] = SP.m != 0 ? SP.x2[d] : B.xe[d];
        seg_mixed_rev(L0, L1, L2, lx, ly, SP.i1, xs, sb, K.w[0], K.w[1], K.w[2], gx, g2);
        if (SP.m != 0) {
            seg_mixed_rev(L0, L1, L2, lx, ly, SP.i2, SP.x2, B.xe, K.w[0], K.w[1], K.w[2], g2, gn);
            split_rev_m(SP, xs, B.xe, g2, gx, gn);
        } else {
#pragma unroll
            for (int d = 0; d < 3; d++) gn[d] += g2[d];
        }
    }
    // xe = xs + ct * ig * p'
    float dot = 0.f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        gx[d] += gn[d];
        dot += gn[d] * B.ct[d] * B.pp[d];
    }
    const float ig3 = B.ig * B.ig * B.ig;
#pragma unroll
    for (int d = 0; d < 3; d++) lP[d] = lP[d] + B.ig * B.ct[d] * gn[d] - ig3 * dot * B.pp[d];
#pragma unroll
    for (int d = 0; d < 3; d++) lF[d] = B.t * lP[d];
    const float *b = B.b, *sv = B.s, *up = B.up, *u = B.u;
    float bl = b[0] * lP[0] + b[1] * lP[1] + b[2] * lP[2];
    float bs = b[0] * sv[0] + b[1] * sv[1] + b[2] * sv[2];
    float lu_ = lP[0] * up[0] + lP[1] * up[1] + lP[2] * up[2];
    const float inv = B.rs;
    float bxl[3] = {b[1] * lP[2] - b[2] * lP[1], b[2] * lP[0] - b[0] * lP[2], b[0] * lP[1] - b[1] * lP[0]};
    float lxs[3] = {lP[1] * sv[2] - lP[2] * sv[1], lP[2] * sv[0] - lP[0] * sv[2], lP[0] * sv[1] - lP[1] * sv[0]};
    float ls[3], lb[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        ls[d] = (lP[d] + b[d] * bl + bxl[d]) * inv;
        lb[d] = (bs * lP[d] + bl * sv[d] + lxs[d] - 2.f * lu_ * b[d]) * inv;
    }
    lu[0] = ls[0] + (b[1] * ls[2] - b[2] * ls[1]);
    lu[1] = ls[1] + (b[2] * ls[0] - b[0] * ls[2]);
    lu[2] = ls[2] + (b[0] * ls[1] - b[1] * ls[0]);
    lb[0] += ls[1] * u[2] - ls[2] * u[1];
    lb[1] += ls[2] * u[0] - ls[0] * u[2];
    lb[2] += ls[0] * u[1] - ls[1] * u[0];
    float lps = 0.f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        lF[3 + d] = B.ps * lb[d];
        lps += lb[d] * F[3 + d];
    }
    const float cps = -B.t * B.g1 * B.g1 * B.g1 * lps;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        lu[d] += cps * u[d];
        lF[d] += B.t * lu[d];
    }
}

// One component of the interpolation's transpose: gi += lam * dF/dx (V: the
// particle's cell in the component's array, strides dX, dY), add(x, y, z, lam
// times the x and y weights, lower and upper z weight)
template <int C, class Add>
__device__ __forceinline__ void reverse_component_m(const float *V, int dX, int dY, const float xs[3], float lam,
                                                    float gi[3], Add add) {
    MTaps T;
    taps_mixed(xs, T);
    int t[3];
    float w[3];
    comp_taps_m(T, C, t, w);
    const int tx = t[0] - 2, ty = t[1] - 2, tz = t[2] - 2;
    const float wx = w[0], wy = w[1], wz = w[2], vx = 1.f - wx, vy = 1.f - wy, vz = 1.f - wz;
    V += tx * dX + ty * dY + tz;
    float yl[2], yd[2], yz[2];
#pragma unroll
    for (int a = 0; a < 2; a++) {
        const float v0 = V[a * dX], v1 = V[a * dX + 1], v2 = V[a * dX + dY], v3 = V[a * dX + dY + 1];
        const float z0 = wz * v0 + vz * v1, z1 = wz * v2 + vz * v3;
        yl[a] = wy * z0 + vy * z1;
        yd[a] = z1 - z0;
        yz[a] = wy * (v1 - v0) + vy * (v3 - v2);
    }
    gi[0] += lam * (yl[1] - yl[0]);
    gi[1] += lam * (wx * yd[0] + vx * yd[1]);
    gi[2] += lam * (wx * yz[0] + vx * yz[1]);
#pragma unroll
    for (int q = 0; q < 4; q++) add(tx + (q >> 1), ty + (q & 1), tz, lam * ((q >> 1 ? vx : wx) * (q & 1 ? vy : wy)), wz, vz);
}

// a particle outside its chunk's window: everything through global memory
__device__ __forceinline__ void reverse_global_m(const MixParams &P, int s, int64_t j) {
    const Grid &g = P.g;
    const MixSp &S = P.sp[s];
    float *const *Lm = P.lam[s];
    const MixConst K = mix_const(g, S);
    float xs[3] = {S.v[0][j], S.v[1][j], S.v[2][j]}, p[3] = {S.v[3][j], S.v[4][j], S.v[5][j]};
    float gn[3] = {Lm[0][j], Lm[1][j], Lm[2][j]}, lP[3] = {Lm[3][j], Lm[4][j], Lm[5][j]};
    int c3[3];
    g.cell_ijk(S.cell[j], c3[0], c3[1], c3[2]);
    const size_t n = g.node(c3[0], c3[1], c3[2]);
    FieldViewM<false> V;
#pragma unroll
    for (int c = 0; c < 3; c++) { V.base[c] = P.E[c] + n; V.base[3 + c] = P.H[c] + n; }
    V.dx = g.NY * g.pz; V.dy = g.pz;
    float gx[3], lu[3], lF[6], gi[3] = {0.f, 0.f, 0.f};
    reverse_particle_m(K, V, P.LJ[0] + n, P.LJ[1] + n, P.LJ[2] + n, V.dx, V.dy, xs, p, gn, lP, gx, lu, lF);
    auto put = [&](double *L) {
        return [=](int a, int b, int c, float v, float wz, float vz) {
            double *r = L + a * V.dx + b * V.dy + c;
            atomicAdd(r, (double)(v * wz));
            atomicAdd(r + 1, (double)(v * vz));
        };
    };
    reverse_component_m<0>(V.base[0], V.dx, V.dy, xs, lF[0], gi, put(P.LE[0] + n));
    reverse_component_m<1>(V.base[1], V.dx, V.dy, xs, lF[1], gi, put(P.LE[1] + n));
    reverse_component_m<2>(V.base[2], V.dx, V.dy, xs, lF[2], gi, put(P.LE[2] + n));
    reverse_component_m<3>(V.base[3], V.dx, V.dy, xs, lF[3], gi, put(P.LH[0] + n));
    reverse_component_m<4>(V.base[4], V.dx, V.dy, xs, lF[4], gi, put(P.LH[1] + n));
    reverse_component_m<5>(V.base[5], V.dx, V.dy, xs, lF[5], gi, put(P.LH[2] + n));
#pragma unroll
    for (int d = 0; d < 3; d++) {
        Lm[d][j] = gx[d] + gi[d];
        Lm[3 + d][j] = lu[d];
    }
}

__device__ __noinline__ void reverse_far_m(const MixParams &P, int s, int64_t j) { reverse_global_m(P, s, j); }
// all particles of a step that way
__global__ void __launch_bounds__(kT, kDirectAdjBlocks) k_adj_direct_mixed(const __grid_constant__ MixParams P) {
    chain_enter();
    const AdjChunk ch = P.chunks[blockIdx.x];
    const int lane = threadIdx.x & 31, mine = (lane >> 3) * 64 + (threadIdx.x >> 5) * 8 + (lane & 7);
    for (int e = mine; e < ch.count; e += blockDim.x) reverse_global_m(P, ch.species, ch.first + e);
}

// ---- adjoint of the particle part of one step (k_adj_particles_plain in FP32):
// one CTA per chunk with its window of E, H and lambda_J staged; lambda_E and
// lambda_H are summed there in 64-bit words in units of 2^-30 of the largest
// |lambda of a field value| of a batch of 256 particles (quantum_for) and added
// to the FP64 global arrays at the end.  A contribution fits an int32, so its add touches the high
// word only when the low one carries or borrows.
// Bound: instruction issue and the shared-memory pipe.  128x32x32 cells: 1.90 ->
// 1.37 ms per reverse step, with windows past the grid's ends 1.32 (two CTAs per
// SM at 128 registers: 1.46; before: two
// kernels that gathered from global memory).
__global__ void __launch_bounds__(kT, 3) k_adj_particles_mixed(const __grid_constant__ MixParams P) {
    chain_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ AdjWindow<true> sWin;
    __shared__ int sRed[15 * kW], sFar;
    __shared__ unsigned sMax[kMaxSlots];
    __shared__ MixConst sK;
    const Grid &g = P.g;
    const AdjChunk ch = P.chunks[blockIdx.x];
    const int s = ch.species, count = ch.count;
    const MixSp &S = P.sp[s];
    float *const *Lm = P.lam[s];
    const NextMix<12> next(smem_raw + (size_t)kAdjWindowMix * 84);
    unsigned short *sList = (unsigned short *)(smem_raw + (size_t)kAdjWindowMix * 84 + NextMix<12>::bytes);
    // lanes as in k_adj_particles_plain
    const int lane = threadIdx.x & 31, mine = (lane >> 3) * 64 + (threadIdx.x >> 5) * 8 + (lane & 7);
    if (mine < count) next.start(S, Lm, ch.first + mine);
    const AdjWindow<true> w = chunk_window(g, S.cell + ch.first, count, kAdjWindowMix, sRed, &sWin);
    const int nn = w.nn, dX = w.SY * w.SZ, dY = w.SZ;
    float *sF = (float *)smem_raw, *sL = sF + 6 * nn;
    unsigned *sLo = (unsigned *)(sL + 3 * nn), *sHi = sLo + 6 * nn;
    const float *src[6] = {P.E[0], P.E[1], P.E[2], P.H[0], P.H[1], P.H[2]};
    stage_window_m<6>(g, w, nn, src, sF);
    stage_window_m<3>(g, w, nn, P.LJ, sL);
    for (int e = threadIdx.x; e < 12 * nn; e += blockDim.x) sLo[e] = 0u;
    if (threadIdx.x == 0) { sFar = 0; sMax[0] = sMax[1] = sMax[2] = 0u; sK = mix_const(g, S); }
    __syncthreads();
    const MixConst &K = sK;
    int E = kNoQuantum;  // contributions below 2^E = 2^30 quanta
    float inv_q = 0.f;
    auto flush = [&](bool again) {
        if (E == kNoQuantum) return;
        const double q = pow2_d(E - kBitsMix);
        double *const dst[6] = {P.LE[0], P.LE[1], P.LE[2], P.LH[0], P.LH[1], P.LH[2]};
        for (int e = threadIdx.x; e < 6 * nn; e += blockDim.x) {
            const long long v = (long long)(((unsigned long long)sHi[e] << 32) | sLo[e]);
            if (v == 0) continue;
            if (again) sHi[e] = sLo[e] = 0u;
            const int comp = e / nn, r = e - comp * nn;
                size_t n;
                if (w.grid_node(g, r, n)) atomicAdd(&dst[comp][n], (double)v * q);
        }
    };
    for (int base = 0, it = 0; base < count; base += blockDim.x, it++) {
        const int jc = base + mine;
        const int64_t j = ch.first + jc;
        int cell = -1;
        float xs[3], p[3], gn[3], lP[3];
        cp_async_wait_all();
        if (jc < count) {
            cell = next.cell();
            next.take3(0, xs);
            next.take3(3, p);
            next.take3(6, gn);
            next.take3(9, lP);
        }
        __syncwarp();
        if (jc + (int)blockDim.x < count) next.start(S, Lm, j + blockDim.x);
        int c3[3] = {0, 0, 0}, n0 = 0;
        bool near = cell >= 0;
        if (near) {
            int u[3];
            g.cell_ijk(cell, c3[0], c3[1], c3[2]);
            if (!w.place(c3, dX, dY, u, n0)) {
                near = false;
                sList[atomicAdd(&sFar, 1)] = (unsigned short)jc;
            }
        }
        float gx[3], lu[3], lF[6], gi[3] = {0.f, 0.f, 0.f};
        unsigned amax = 0u;  // bits of the largest |lambda_F|
        if (near) {
            FieldViewM<true> V;
#pragma unroll
            for (int c = 0; c < 6; c++) V.base[c] = sF + c * nn + n0;
            V.dx = dX; V.dy = dY;
            reverse_particle_m(K, V, sL + n0, sL + nn + n0, sL + 2 * nn + n0, dX, dY, xs, p, gn, lP, gx, lu, lF);
#pragma unroll
            for (int c = 0; c < 6; c++) amax = max(amax, __float_as_uint(lF[c]) & 0x7fffffffu);
            if (amax >= 0x7f800000u) {  // no fixed point for an infinity or a NaN
                near = false;
                amax = 0u;
                sList[atomicAdd(&sFar, 1)] = (unsigned short)jc;
            }
        }
        // the block's largest |lambda_F| against the quantum in use
        const unsigned wm = __reduce_max_sync(0xffffffffu, amax);
        if (lane == 0 && wm) atomicMax(&sMax[max_slot(it)], wm);
        __syncthreads();
        const unsigned bm = sMax[max_slot(it)];
        if (threadIdx.x == 0) sMax[max_cleared(it)] = 0u;
        const int En = bm ? quantum_for(E, exponent_f(bm), kKeepMix, kLeastMix) : E;
        if (En != E) {  // block-uniform
            flush(true);
            E = En;
            inv_q = __uint_as_float((unsigned)(kBitsMix - E + 127) << 23);
            __syncthreads();
        }
        if (near && amax) {
            auto put = [&](int c) {
                unsigned *lo = sLo + c * nn + n0;
                return [=](int a, int b, int k, float v, float wz, float vz) {
                    unsigned *r = lo + a * dX + b * dY + k;
                    const float vq = v * inv_q;
                    shared_add64_small(r, r + 6 * nn, __float2int_rn(vq * wz));
                    shared_add64_small(r + 1, r + 1 + 6 * nn, __float2int_rn(vq * vz));
                };
            };
            const float *V = sF + n0;
            reverse_component_m<0>(V, dX, dY, xs, lF[0], gi, put(0));
            reverse_component_m<1>(V + nn, dX, dY, xs, lF[1], gi, put(1));
            reverse_component_m<2>(V + 2 * nn, dX, dY, xs, lF[2], gi, put(2));
            reverse_component_m<3>(V + 3 * nn, dX, dY, xs, lF[3], gi, put(3));
            reverse_component_m<4>(V + 4 * nn, dX, dY, xs, lF[4], gi, put(4));
            reverse_component_m<5>(V + 5 * nn, dX, dY, xs, lF[5], gi, put(5));
        }
        if (near) {
#pragma unroll
            for (int d = 0; d < 3; d++) {
                Lm[d][j] = gx[d] + gi[d];
                Lm[3 + d][j] = lu[d];
            }
        }
    }
    __syncthreads();
    flush(false);
    for (int e = threadIdx.x; e < sFar; e += blockDim.x) reverse_far_m(P, s, ch.first + sList[e]);
}

__global__ void k_gather_native(SpeciesView S, const int64_t *__restrict__ d0, int *cell, float *ox, float *oy,
                                float *oz, float *px, float *py, float *pz) {
    int t = blockIdx.x;
    int start = S.tile_start[t], n = S.tile_count[t];
    int64_t base = d0[t];
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        int slot = start + j;
        int64_t d = base + j;
        cell[d] = S.cell[slot];
        ox[d] = S.ox[slot]; oy[d] = S.oy[slot]; oz[d] = S.oz[slot];
        px[d] = S.fx[slot]; py[d] = S.fy[slot]; pz[d] = S.fz[slot];
    }
}
__global__ void k_widen(const float *__restrict__ lp, const float *__restrict__ a, const float *__restrict__ b,
                        const float *__restrict__ c, int64_t n, double *out) {
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    out[j] = lp[j];
    out[n + j] = lp[n + j];
    out[2 * n + j] = lp[2 * n + j];
    out[3 * n + j] = a[j];
    out[4 * n + j] = b[j];
    out[5 * n + j] = c[j];
}

}  // namespace

cudaError_t launch_flat_push_mixed(const MixParams &P, int nchunks, bool direct, cudaStream_t s) {
    if (nchunks <= 0) return cudaSuccess;
    if (direct) return launch_chained(k_flat_push_mixed<true>, dim3(nchunks), dim3(kT), s, P);
    const size_t smem = (size_t)kFlatWindowMix * 48 + (size_t)kW * 7 * kQueueMix * sizeof(float) + NextMix<6>::bytes;
    cudaError_t e = cudaFuncSetAttribute(k_flat_push_mixed<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_chained_smem(k_flat_push_mixed<false>, dim3(nchunks), dim3(kT), smem, s, P);
}

cudaError_t launch_adj_particles_mixed(const MixParams &P, int nchunks, bool direct, cudaStream_t s) {
    if (nchunks <= 0) return cudaSuccess;
    if (direct) return launch_chained(k_adj_direct_mixed, dim3(nchunks), dim3(kT), s, P);
    const size_t smem = (size_t)kAdjWindowMix * 84 + NextMix<12>::bytes + kAdjChunk * sizeof(unsigned short);
    cudaError_t e = cudaFuncSetAttribute(k_adj_particles_mixed, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_chained_smem(k_adj_particles_mixed, dim3(nchunks), dim3(kT), smem, s, P);
}

void adj_gather_mixed(const Grid &g, const SpeciesView &S, const int64_t *d0, int *cell, void *const v[6],
                      cudaStream_t s) {
    k_gather_native<<<g.ntiles, 256, 0, s>>>(S, d0, cell, (float *)v[0], (float *)v[1], (float *)v[2],
                                             (float *)v[3], (float *)v[4], (float *)v[5]);
}

void adj_widen_mixed(const float *lp, const float *const p0[3], int64_t n, double *out6, cudaStream_t s) {
    if (n <= 0) return;
    k_widen<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(lp, p0[0], p0[1], p0[2], n, out6);
}

}  // namespace pic
