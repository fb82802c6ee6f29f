// Differentiable run of the PIC step (pic_forward / pic_backward): a forward
// pass that keeps every particle in a fixed order and checkpoints the state,
// and hand-written reverse-mode (adjoint) kernels.  Plain form: FP64, same
// arithmetic as k_push_plain (compiled with -fmad=false like it); the FP32
// form lives in pic_adjoint_mixed.cu.
//
// Forward map of one step (Plasma::Step, gpu_plasma.h:605-620), per piece:
//   Q = A E, H_a = H + Q                 (emh1, kernels.cu:1052-1073)
//   particles: F = W(x) [E, H_a]; (p', x') = Boris(p, F, x)   (particle.h:65-202)
//   J = sum_p D(x, x')                    (CurrentToMesh/pqr, cell.h:1306-1693)
//   J <- P J                              (periodicCurrentElement, kernels.cu:1124-1146)
//   H' = H_a + Q                          (emh2, kernels.cu:1024-1049)
//   E' = G (E + tau C H' - tau J)         (emeElement + periodicElement, kernels.cu:1091-1110)
// The reverse step applies the transposes in the opposite order.  Particles
// never change order in this pass (their cell index is rewritten in place),
// so a particle's adjoint (lambda_x, lambda_p) follows it from step to step;
// the deposit's transpose is a gather of lambda_J at the particle's 12 nodes
// per segment and the interpolation's transpose a scatter of lambda_F.
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <string.h>
#include <vector>
#include <algorithm>
#include "pic0buf.h"
#include "pic_internal.cuh"
#include "pic_kernels.cuh"
#include "pic_handle.cuh"
#include <type_traits>
#include "pic_adjoint.cuh"
#include "pic_plain_math.cuh"
#include "pic_fold.cuh"

namespace pic {

namespace {

constexpr int kT = 256;

// ================================================================ plain ==
// one species in flat order: packed cell, global FP64 positions, momenta
struct FlatSp {
    int64_t n;
    double q_m, m;
    int *cell;
    double *v[6];  // x y z px py pz
};
// where the push writes the state after the step (may alias the input)
struct FlatOut {
    int *cell;
    double *v[6];
};
struct FlatParams {
    Grid g;
    int nsp;
    const AdjChunk *chunks;  // one per CTA
    int64_t off[kMaxSpecies + 1];
    FlatSp sp[kMaxSpecies];
    FlatOut out[kMaxSpecies];
    const double *E[3];
    const double *H[3];
    double *J[3];
    AdjStatus *st;
    // discrete choices of this step, one 48-bit code per particle (flat index):
    // bmode 1 records them, 2 replays them (see branch_code)
    unsigned long long *branch;
    int bmode;
    int *far;  // counts the particles outside their chunk's window (null: not)
};
// adjoint of one species: lambda_x (3) and lambda_p (3), same order
struct LamSp {
    double *v[6];
};
struct AdjParams {
    FlatParams f;  // state at the start of the step; E = E_n, H = H_a (after the B half step)
    LamSp lam[kMaxSpecies];
    const double *LJ[3];  // lambda_J (after the fold's transpose)
    double *LE[3];        // lambda_E_n (scatter target)
    double *LH[3];        // lambda_H_a (scatter target)
};

constexpr int kW = kT / 32;        // warps per CTA
constexpr int kDirectBlocks = 3, kDirectAdjBlocks = 2;  // CTAs per SM of the kernels without a window
constexpr int kQueuePlain = 48;    // queued second segments per warp, as in k_push_plain
constexpr int kFlatWindow = 900;   // nodes of the forward's window: 109 KB of shared memory, two CTAs per SM
constexpr int kAdjWindow = 704;    // nodes of the adjoint's: 112 KB

// shared memory of a thread's next particle (cp.async, as in k_push_plain)
constexpr size_t kNextBytes = (size_t)kW * (6 * 32 + 16) * sizeof(double);
struct NextParticle {
    double *v;
    int *c;
    __device__ __forceinline__ NextParticle(void *base) {
        const int lane = threadIdx.x & 31;
        double *b = (double *)base + (threadIdx.x >> 5) * (6 * 32 + 16);
        v = b + lane;
        c = (int *)(b + 6 * 32) + lane;
    }
    __device__ __forceinline__ void start(const FlatSp &S, int64_t j) const {
        cp_async<4>(c, S.cell + j);
#pragma unroll
        for (int a = 0; a < 6; a++) cp_async<8>(v + 32 * a, S.v[a] + j);
    }
    __device__ __forceinline__ int take(double x[3], double p[3]) const {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            x[d] = v[32 * d];
            p[d] = v[32 * (3 + d)];
        }
        return *c;
    }
};

// the same for its six adjoints
constexpr size_t kNextLamBytes = (size_t)kW * 6 * 32 * sizeof(double);
struct NextLam {
    double *v;
    __device__ __forceinline__ NextLam(void *base) {
        v = (double *)base + (threadIdx.x >> 5) * (6 * 32) + (threadIdx.x & 31);
    }
    __device__ __forceinline__ void start(const LamSp &L, int64_t j) const {
#pragma unroll
        for (int a = 0; a < 6; a++) cp_async<8>(v + 32 * a, L.v[a] + j);
    }
    __device__ __forceinline__ void take(double lx[3], double lp[3]) const {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            lx[d] = v[32 * d];
            lp[d] = v[32 * (3 + d)];
        }
    }
};

// A particle's view of the fields: the CTA's window in shared memory (WIN) or
// the arrays in global memory.  n0 is the node of the particle's cell.
template <bool WIN>
struct FieldView {
    const double *base[6];
    int n0, dx, dy;
    __device__ __forceinline__ int at(int tx, int ty, int tz) const {
        return n0 + (tx - 2) * dx + (ty - 2) * dy + (tz - 2);
    }
};
// component c (0..2 E, 3..5 H) is node-staggered along axis d when
// (E_c and d == c) or (H_c and d != c)
__device__ __forceinline__ constexpr bool node_axis(int c, int d) { return c < 3 ? d == c : d != c - 3; }

// GetField (cell.h:1257-1290) at the particle; false if a tap left the stencil
// (that component is then 0, as in k_push_plain)
template <class V>
__device__ __forceinline__ bool gather_fields(const V &A, const AxisTaps T[3], double F[6]) {
    // every tap in 2..3; each of the six indices is some component's
    if ((((T[0].tn ^ 2) | (T[0].tc ^ 2) | (T[1].tn ^ 2) | (T[1].tc ^ 2) | (T[2].tn ^ 2) | (T[2].tc ^ 2)) & ~1) != 0) {
#pragma unroll
        for (int c = 0; c < 6; c++) F[c] = 0.0;
        return false;
    }
#pragma unroll
    for (int c = 0; c < 6; c++) {
        const bool nx = node_axis(c, 0), ny = node_axis(c, 1), nz = node_axis(c, 2);
        const int n = A.at(nx ? T[0].tn : T[0].tc, ny ? T[1].tn : T[1].tc, nz ? T[2].tn : T[2].tc);
        const double wx = nx ? T[0].wn : T[0].wc, wy = ny ? T[1].wn : T[1].wc, wz = nz ? T[2].wn : T[2].wc;
        F[c] = trilinear(A.base[c] + n, A.dx, A.dy, wx, 1. - wx, wy, 1. - wy, wz, 1. - wz);
    }
    return true;
}

// zigzag split of CurrentToMesh, cell.h:1306-1422
struct Split {
    int m, i1[3], i2[3];
    double x2[3], sr;
};

// one pqr segment (cell.h:1511-1693) into the global J, FP64 atomics (particles
// outside their CTA's window); rc[d] = m / (tau * h_e * h_f)
__device__ __forceinline__ void seg_global(double *const J[3], const Grid &g, int ci, int cl, int ck, const int iv[3],
                                           const double x[3], const double x1[3], const double rc[3],
                                           const double o3[3], unsigned &bad) {
    const double hx = g.hx, hy = g.hy, hz = g.hz;
    const double dx = (0.50 * (x[0] + x1[0]) - hx * ((double)iv[0] - 2.50) - o3[0]);
    const double dy = (0.50 * (x[1] + x1[1]) - hy * ((double)iv[1] - 2.50) - o3[1]);
    const double dz = (0.50 * (x[2] + x1[2]) - hz * ((double)iv[2] - 2.50) - o3[2]);
    const double dx1 = hx - dx, dy1 = hy - dy, dz1 = hz - dz;
    double su = x1[0] - x[0], sv = x1[1] - x[1], sw = x1[2] - x[2];
    constexpr double kTwelfth = 1.0 / 12.0;
    const double s1 = sv * sw * kTwelfth, s2 = su * sw * kTwelfth, s3 = su * sv * kTwelfth;
    su = su * rc[0];
    sv = sv * rc[1];
    sw = sw * rc[2];
    if (iv[0] < 2 || iv[0] > 3 || iv[1] < 2 || iv[1] > 3 || iv[2] < 2 || iv[2] > 3) { bad |= ST_STENCIL; return; }
    const size_t n = g.node(ci + iv[0] - 2, cl + iv[1] - 2, ck + iv[2] - 2);
    const size_t ez = 1, ey = g.pz, ex = (size_t)g.NY * g.pz;
    double *Jx = J[0], *Jy = J[1], *Jz = J[2];
    atomicAdd(&Jx[n], su * fma(dy1, dz1, s1));
    atomicAdd(&Jx[n + ez], su * fma(dy1, dz, -s1));
    atomicAdd(&Jx[n + ey], su * fma(dy, dz1, -s1));
    atomicAdd(&Jx[n + ey + ez], su * fma(dy, dz, s1));
    atomicAdd(&Jy[n], sv * fma(dx1, dz1, s2));
    atomicAdd(&Jy[n + ez], sv * fma(dx1, dz, -s2));
    atomicAdd(&Jy[n + ex], sv * fma(dx, dz1, -s2));
    atomicAdd(&Jy[n + ex + ez], sv * fma(dx, dz, s2));
    atomicAdd(&Jz[n], sw * fma(dx1, dy1, s3));
    atomicAdd(&Jz[n + ey], sw * fma(dx1, dy, -s3));
    atomicAdd(&Jz[n + ex], sw * fma(dx, dy1, -s3));
    atomicAdd(&Jz[n + ex + ey], sw * fma(dx, dy, s3));
}

// transpose of a pqr segment: lambda_J (L: three components, n the segment's
// base node, ex, ey the node strides) gathered at its 12 nodes gives the
// gradient with respect to the segment's end points (added to gs, ge)
__device__ __forceinline__ void seg_rev(const double *L0, const double *L1, const double *L2, int n, int ex, int ey,
                                        const Grid &g, const int iv[3], const double xs[3], const double xe[3],
                                        const double rc[3], const double o3[3], double gs[3], double ge[3]) {
    constexpr double kTwelfth = 1.0 / 12.0;
    const double hx = g.hx, hy = g.hy, hz = g.hz;
    const double dx = 0.5 * (xs[0] + xe[0]) - hx * ((double)iv[0] - 2.5) - o3[0];
    const double dy = 0.5 * (xs[1] + xe[1]) - hy * ((double)iv[1] - 2.5) - o3[1];
    const double dz = 0.5 * (xs[2] + xe[2]) - hz * ((double)iv[2] - 2.5) - o3[2];
    const double dx1 = hx - dx, dy1 = hy - dy, dz1 = hz - dz;
    const double Dx = xe[0] - xs[0], Dy = xe[1] - xs[1], Dz = xe[2] - xs[2];
    const double s1 = Dy * Dz * kTwelfth, s2 = Dx * Dz * kTwelfth, s3 = Dx * Dy * kTwelfth;
    const double Ax = rc[0] * Dx, Ay = rc[1] * Dy, Az = rc[2] * Dz;
    // per component the four nodes as sums over its two transverse axes:
    // F = sum L (weight + or - s), K = L00 - L01 - L10 + L11, and the weights'
    // derivatives along the two axes
    double a, b, c, d;
    a = L0[n]; b = L0[n + 1]; c = L0[n + ey]; d = L0[n + ey + 1];
    const double Kx = (a - b) + (d - c);
    const double xz0 = fma(a, dz1, b * dz), xz1 = fma(c, dz1, d * dz);   // z sums of the lower and the upper y row
    const double Fx = fma(dy1, xz0, fma(dy, xz1, s1 * Kx));
    const double x_dy = xz1 - xz0, x_dz = fma(dy1, b - a, dy * (d - c));
    a = L1[n]; b = L1[n + 1]; c = L1[n + ex]; d = L1[n + ex + 1];
    const double Ky = (a - b) + (d - c);
    const double yz0 = fma(a, dz1, b * dz), yz1 = fma(c, dz1, d * dz);
    const double Fy = fma(dx1, yz0, fma(dx, yz1, s2 * Ky));
    const double y_dx = yz1 - yz0, y_dz = fma(dx1, b - a, dx * (d - c));
    a = L2[n]; b = L2[n + ey]; c = L2[n + ex]; d = L2[n + ex + ey];
    const double Kz = (a - b) + (d - c);
    const double zy0 = fma(a, dy1, b * dy), zy1 = fma(c, dy1, d * dy);
    const double Fz = fma(dx1, zy0, fma(dx, zy1, s3 * Kz));
    const double z_dx = zy1 - zy0, z_dy = fma(dx1, b - a, dx * (d - c));
    // d/d(D): direct factor and the D-products in s1, s2, s3
    const double kx = Ax * Kx * kTwelfth, ky = Ay * Ky * kTwelfth, kz = Az * Kz * kTwelfth;
    const double gDx = fma(rc[0], Fx, fma(ky, Dz, kz * Dy));
    const double gDy = fma(rc[1], Fy, fma(kx, Dz, kz * Dx));
    const double gDz = fma(rc[2], Fz, fma(kx, Dy, ky * Dx));
    // d/d(dx, dy, dz): the bilinear node weights
    const double gdx = fma(Ay, y_dx, Az * z_dx), gdy = fma(Ax, x_dy, Az * z_dy), gdz = fma(Ax, x_dz, Ay * y_dz);
    gs[0] += fma(0.5, gdx, -gDx); ge[0] += fma(0.5, gdx, gDx);
    gs[1] += fma(0.5, gdy, -gDy); ge[1] += fma(0.5, gdy, gDy);
    gs[2] += fma(0.5, gdz, -gDz); ge[2] += fma(0.5, gdz, gDz);
}

// transpose of the split point x2(xo, xn): adds g2 . dx2/dxo to gx, . dx2/dxn
// to gn.  Axis indices are template arguments so the 3-vectors stay in registers.
template <int O>
__device__ __forceinline__ double rbx_rev(double sr, const double xo[3], const double xn[3], const double g2[3],
                                          double gx[3], double gn[3]) {
    // x2[O] = xo[O] + (xn[O] - xo[O]) sr
    gx[O] += g2[O] * (1.0 - sr);
    gn[O] += g2[O] * sr;
    return g2[O] * (xn[O] - xo[O]);
}
template <int A, int O0, int O1>  // one plane crossed on axis A: sr = (c - xo)/(xn - xo)
__device__ __forceinline__ void split_rev1(const Split &S, const double xo[3], const double xn[3],
                                           const double g2[3], double gx[3], double gn[3]) {
    const double sr = S.sr;
    double lsr = rbx_rev<O0>(sr, xo, xn, g2, gx, gn) + rbx_rev<O1>(sr, xo, xn, g2, gx, gn);
    double D = xn[A] - xo[A];
    gx[A] += lsr * (S.x2[A] - xn[A]) / (D * D);
    gn[A] -= lsr * sr / D;
}
template <int A, int B, int O>  // two planes: sr = sum_d (c_d - xo_d)(xn_d - xo_d) / sum_d (xn_d - xo_d)^2
__device__ __forceinline__ void split_rev2(const Split &S, const double xo[3], const double xn[3],
                                           const double g2[3], double gx[3], double gn[3]) {
    const double sr = S.sr;
    double lsr = rbx_rev<O>(sr, xo, xn, g2, gx, gn);
    double Da = xn[A] - xo[A], Db = xn[B] - xo[B];
    double f = lsr / (Da * Da + Db * Db);
    double ca = S.x2[A] - xo[A], cb = S.x2[B] - xo[B];
    gx[A] += f * (-Da - ca + 2.0 * sr * Da);
    gn[A] += f * (ca - 2.0 * sr * Da);
    gx[B] += f * (-Db - cb + 2.0 * sr * Db);
    gn[B] += f * (cb - 2.0 * sr * Db);
}
__device__ __forceinline__ void split_rev(const Split &S, const double xo[3], const double xn[3], const double g2[3],
                                          double gx[3], double gn[3]) {
    switch (S.m) {
        case 1: split_rev1<2, 0, 1>(S, xo, xn, g2, gx, gn); break;
        case 2: split_rev1<1, 0, 2>(S, xo, xn, g2, gx, gn); break;
        case 4: split_rev1<0, 1, 2>(S, xo, xn, g2, gx, gn); break;
        case 3: split_rev2<1, 2, 0>(S, xo, xn, g2, gx, gn); break;
        case 5: split_rev2<0, 2, 1>(S, xo, xn, g2, gx, gn); break;
        case 6: split_rev2<0, 1, 2>(S, xo, xn, g2, gx, gn); break;
        default: break;  // 7: the split point is a fixed corner; 0 / >7: no split
    }
}

// the wrap of Reflect (cell.h:1427-1478) as a choice (0 keep, 1 subtract xm, 2
// add xm, 3 the x == xm case: 0); apply_wrap(x, xm, wrap_choice(x, xm)) ==
// reflect_plain(x, xm)
__device__ __forceinline__ int wrap_choice(double x, double xm) {
    return x > xm ? 1 : (x < 0.0 ? 2 : (x == xm ? 3 : 0));
}
__device__ __forceinline__ double apply_wrap(double x, double xm, int w) {
    return w == 1 ? x - xm : (w == 2 ? xm + x : (w == 3 ? 0.0 : x));
}

// Frozen branches.  Per particle and step, the discrete choices of the flat
// FP64 push, 16 bits per axis d at bit 16 d: tap indices tn-1, tc-1, the
// integer parts nI - c_d and cI - c_d of the interpolation weights (c the
// cell index), the zigzag cell-centre indices i1-1 and i2-1, the periodic
// wrap and the cell move + 1, 2 bits each.  A forward that replays them is a
// smooth function of the initial state near the recorded run, and it is the
// map the adjoint differentiates, so its finite differences check the
// adjoint without the kinks and jumps of the deposit.
constexpr unsigned ST_BRANCH_RANGE = 64u;  // a choice outside its 2-bit field (recording)
__device__ __forceinline__ bool pack2(unsigned long long &code, int v, int shift) {
    code |= (unsigned long long)(v & 3) << shift;
    return v >= 0 && v <= 3;
}
__device__ __forceinline__ int unpack2(unsigned long long code, int shift) { return (int)((code >> shift) & 3ull); }
// receivers of a departing particle along one axis (GPU_ArrangeFlights, kernels.cu:316-370)
// (count of receiving cells along one axis; `first` = the first of them)
__device__ __forceinline__ int receivers_g(double x, int c, int N, double h, int &first) {
    int n = 0;
    first = c;
#pragma unroll
    for (int d = -1; d <= 1; d++) {
        int j = c + d;
        if (j >= N) j -= N;
        else if (j < 0) j += N;
        double x0 = (double)j * h;
        if ((x0 <= x) && (x < x0 + h)) {
            if (n == 0) first = j;
            n++;
        }
    }
    return n;
}

// flyDirection (cell.h:694-701) + receivers: the particle's new cell.  In the
// fixed-order pass a particle has exactly one successor; the reference's
// rare boundary cases with zero or several receiving cells are counted
// (AdjStatus::ambiguous) and resolved to the first receiver / the old cell.
__device__ __forceinline__ int new_cell_plain(const Grid &g, int cell, int i, int l, int k, const double x[3],
                                              unsigned long long &amb) {
    const double hx = g.hx, hy = g.hy, hz = g.hz;
    const double x0 = (double)i * hx, y0 = (double)l * hy, z0 = (double)k * hz;
    double px = x[0], py = x[1], pz = x[2];
    int dxd = (((px > x0 + hx) && (px < x0 + 2 * hx)) || ((px < hx) && (i == g.nx - 1)))
                  ? 2 : (((px < x0) || ((px > g.lx - hx) && (i == 0))) ? 0 : 1);
    int dyd = (((py > y0 + hy) && (py < y0 + 2 * hy)) || ((py < hy) && (l == g.ny - 1)))
                  ? 2 : (((py < y0) || ((py > g.ly - hy) && (l == 0))) ? 0 : 1);
    int dzd = (((pz > z0 + hz) && (pz < z0 + 2 * hz)) || ((pz < hz) && (k == g.nz - 1)))
                  ? 2 : (((pz < z0) || ((pz > g.lz - hz) && (k == 0))) ? 0 : 1);
    if (dxd * 9 + dyd * 3 + dzd == 13) return cell;
    int rx, ry, rz;
    int nrx = receivers_g(px, i, g.nx, hx, rx);
    int nry = receivers_g(py, l, g.ny, hy, ry);
    int nrz = receivers_g(pz, k, g.nz, hz, rz);
    if (nrx * nry * nrz != 1) amb++;
    if (nrx == 0 || nry == 0 || nrz == 0) return cell;
    return g.cell_of(rx, ry, rz);
}

// stages the window's nodes of N arrays src[c] into dst (cn doubles apart)
template <int N, bool WRAP>
__device__ __forceinline__ void stage_window(const Grid &g, const AdjWindow<WRAP> &w, int cn, const double *const *src,
                                             double *dst) {
    for (int e = threadIdx.x; e < w.nn; e += blockDim.x) {
        size_t n;
        if (!w.grid_node(g, e, n)) continue;
#pragma unroll
        for (int q = 0; q < N; q++) dst[q * cn + e] = src[q][n];
    }
}

// ---- flat forward step of all particles (push + deposit + cell update).
//
// One CTA per chunk of consecutive particles (they share a neighbourhood: the
// fixed order is tile by tile at the start of the run).  The chunk's window --
// the nodes around its cells -- is staged into shared memory, and its current
// is summed there in the exact fixed point of k_push_plain and added to the
// global J once; a particle outside the window gathers from and adds to
// global memory.  DIRECT: no window, all particles as those outside it (see
// AdjState::direct_from).  Bound: dependent FP64 operations, as k_push_plain.  128x32x32
// cells, 12.6M particles: 1.58 -> 1.12 ms per step (before: taps gathered from
// and currents added to global memory, one particle per thread); with the
// deposit's tests gone and the window's strides at compile time 0.98.
template <int BMODE, bool DIRECT>
__global__ void __launch_bounds__(kT, DIRECT ? kDirectBlocks : 2) k_flat_push_plain(FlatParams P) {
    chain_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ AdjWindow<false> sWin;
    __shared__ int sRed[15 * kW], sQn[kW], sFar;
    __shared__ double sQ, sInvQ;
    double *sF = (double *)smem_raw;
    unsigned long long *sJ = (unsigned long long *)(sF + 6 * kFlatWindow);  // 9 words per node (pqr_plain)
    unsigned char *sTail = smem_raw + (size_t)kFlatWindow * (6 * sizeof(double) + 3 * 12);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *qd = (double *)sTail + warp * 6 * kQueuePlain;
    int *qc = (int *)((double *)sTail + kW * 6 * kQueuePlain) + warp * kQueuePlain;
    const NextParticle next(sTail + (size_t)kW * kQueuePlain * 52);
    const Grid &g = P.g;
    const AdjChunk ch = P.chunks[blockIdx.x];
    const int s = ch.species, count = ch.count;
    const FlatSp &S = P.sp[s];
    AdjWindow<false> w{};
    if (!DIRECT) {
        if ((int)threadIdx.x < count) next.start(S, ch.first + threadIdx.x);
        w = chunk_window(g, S.cell + ch.first, count, kFlatWindow, sRed, &sWin);
    }
    // (see AdjWindow: the strides at compile time where the window has them)
    auto body = [&](auto fixed) {
    constexpr bool FIX = decltype(fixed)::value;
    const int SZ = FIX ? kFixSZ : w.SZ, dX = FIX ? kFixSX : w.SX, dY = SZ, nn = w.nn;
    const int cn = FIX ? kFlatWindow : nn;  // between the components
    const double *src[6] = {P.E[0], P.E[1], P.E[2], P.H[0], P.H[1], P.H[2]};
    if (!DIRECT) {
        if (threadIdx.x == 0) {
            sFar = 0;
            // the quantum of k_push_plain's tile current, for this chunk
            int e2, e1;
            frexp(2.5 * fabs(S.m) * (double)count, &e2);
            frexp(1.0834 * fabs(S.m), &e1);
            const int eq = max(e2 - 62, e1 - 51);
            sQ = ldexp(1.0, eq);
            sInvQ = ldexp(1.0, -eq);
        }
        stage_window<6>(g, w, cn, src, sF);
        for (int e = threadIdx.x; e < 9 * cn; e += blockDim.x) ((unsigned *)sJ)[e] = 0u;
        if (lane == 0) sQn[warp] = 0;
        __syncthreads();
    }
    const double h3[3] = {g.hx, g.hy, g.hz}, r3[3] = {1.0 / g.hx, 1.0 / g.hy, 1.0 / g.hz};
    const double tau = g.tau, tau1 = S.q_m * tau * 0.5;
    const double lo_scale = ldexp(1.0, fx_lo32_bits(count));
    // the charge weight over pqr's tau*h*h divisors, and in quanta
    const double rg[3] = {S.m / (tau * g.hy * g.hz), S.m / (tau * g.hx * g.hz), S.m / (tau * g.hx * g.hy)};
    const double inv_q = DIRECT ? 1.0 : sInvQ, rc[3] = {rg[0] * inv_q, rg[1] * inv_q, rg[2] * inv_q};
    const double L3[3] = {g.lx, g.ly, g.lz};
    const int n3[3] = {g.nx, g.ny, g.nz};
    unsigned bad = 0;
    unsigned long long amb = 0;
    int qn = 0;  // entries in this warp's queue of second segments (warp-uniform)
    for (int jw = threadIdx.x - lane;; jw += blockDim.x) {
        const bool tail = jw >= count;
        if (tail && qn == 0) break;
        const int jc = jw + lane;
        const int64_t j = ch.first + jc;
        int cell = -1;
        double x[3] = {0.0, 0.0, 0.0}, p[3] = {0.0, 0.0, 0.0};
        if (DIRECT) {
            if (jc < count) {
                cell = S.cell[j];
#pragma unroll
                for (int d = 0; d < 3; d++) { x[d] = S.v[d][j]; p[d] = S.v[3 + d][j]; }
            }
        } else {
            cp_async_wait_all();
            if (jc < count) cell = next.take(x, p);
            __syncwarp();  // the reads come before the next copies into the same place
            if (jc + (int)blockDim.x < count) next.start(S, j + blockDim.x);
        }
        if (cell >= 0) {
            int c3[3];
            g.cell_ijk(cell, c3[0], c3[1], c3[2]);
            int u3[3] = {0, 0, 0}, n0 = 0;
            const bool in = !DIRECT && w.place(c3, dX, dY, u3, n0);
            if (!DIRECT && !in) atomicAdd(&sFar, 1);
            const double o3[3] = {(double)c3[0] * h3[0], (double)c3[1] * h3[1], (double)c3[2] * h3[2]};
            const unsigned long long rcode = BMODE == 2 ? P.branch[P.off[s] + j] : 0ull;
            AxisTaps T[3];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                if (BMODE == 2) {
                    T[d].tn = unpack2(rcode, 16 * d) + 1;
                    T[d].tc = unpack2(rcode, 16 * d + 2) + 1;
                    T[d].nI = unpack2(rcode, 16 * d + 4) + c3[d];
                    T[d].cI = unpack2(rcode, 16 * d + 6) + c3[d];
                    T[d].i1 = unpack2(rcode, 16 * d + 8) + 1;
                    const double q = div_by(x[d], h3[d], r3[d]);
                    T[d].wn = (double)T[d].nI - q;
                    T[d].wc = (double)T[d].cI - 0.5 - q;
                } else {
                    axis_taps(x[d], o3[d], h3[d], r3[d], T[d]);
                }
            }
            double F[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            // the reference's GetField gives no field at a negative coordinate;
            // positions are wrapped into [0, L) so a run never meets it, and a
            // replay of frozen branches, whose wraps are fixed, leaves it out
            if (BMODE == 2 || !(x[0] < 0 || x[1] < 0 || x[2] < 0)) {
                bool ok;
                if (in) {
                    FieldView<true> A;
#pragma unroll
                    for (int c = 0; c < 6; c++) A.base[c] = sF + c * cn;
                    A.n0 = n0; A.dx = dX; A.dy = dY;
                    ok = gather_fields(A, T, F);
                } else {
                    FieldView<false> A;
#pragma unroll
                    for (int c = 0; c < 6; c++) A.base[c] = src[c] + g.node(c3[0], c3[1], c3[2]);
                    A.n0 = 0; A.dx = g.NY * g.pz; A.dy = g.pz;
                    ok = gather_fields(A, T, F);
                }
                if (!ok) bad |= ST_STENCIL;
            }
            double p2;
            const double ig = boris_move(tau1, F, p, p2);
            if (!isfinite(p2) && !(isfinite(p[0]) && isfinite(p[1]) && isfinite(p[2]))) bad |= ST_NAN;
            Split SP;
            double x1[3];
            bool exact = true;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                x1[d] = x[d] + tau * (ig * p[d]);
                SP.i1[d] = T[d].i1;
                SP.i2[d] = BMODE == 2 ? unpack2(rcode, 16 * d + 10) + 1
                                      : trunc_checked((div_by(x1[d] - o3[d], h3[d], r3[d]) + 1.5) + 1, exact);
            }
            if (!exact) { bad |= ST_STENCIL; SP.i2[0] = 0; }
            SP.m = relay_point(x, x1, o3, h3, SP.i1, SP.i2, SP.x2, SP.sr);
            const bool cross = SP.m >= 1 && SP.m <= 7;
            double sb[3];
#pragma unroll
            for (int d = 0; d < 3; d++) sb[d] = cross ? SP.x2[d] : x1[d];
            if (in) {
                pqr_plain<true>((unsigned *)sJ, lo_scale, cn, dX, dY, u3[0] - 2, u3[1] - 2, u3[2] - 2, SP.i1,
                                x, sb, g.hx, g.hy, g.hz, rc, o3[0], o3[1], o3[2], bad);
                if (cross) {
                    if (SP.i2[0] >= 2 && SP.i2[0] <= 3 && SP.i2[1] >= 2 && SP.i2[1] <= 3 && SP.i2[2] >= 2 &&
                        SP.i2[2] <= 3) {
                        const int e = atomicAdd(&sQn[warp], 1);  // < 15 + 32: drained at 16
#pragma unroll
                        for (int d = 0; d < 3; d++) {
                            qd[d * kQueuePlain + e] = SP.x2[d];
                            qd[(3 + d) * kQueuePlain + e] = x1[d];
                        }
                        // window-local node of the cell, 9 bits each (a window has at most kFlatWindow nodes), and class bits
                        qc[e] = (u3[0] << 21) | (u3[1] << 12) | (u3[2] << 3) | (SP.i2[0] - 2) |
                                ((SP.i2[1] - 2) << 1) | ((SP.i2[2] - 2) << 2);
                    } else {
                        bad |= ST_STENCIL;
                    }
                }
            } else {
                seg_global(P.J, g, c3[0], c3[1], c3[2], SP.i1, x, sb, rg, o3, bad);
                if (cross) seg_global(P.J, g, c3[0], c3[1], c3[2], SP.i2, SP.x2, x1, rg, o3, bad);
            }
            int wr[3];
            double xr[3];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                wr[d] = BMODE == 2 ? unpack2(rcode, 16 * d + 12) : wrap_choice(x1[d], L3[d]);
                xr[d] = apply_wrap(x1[d], L3[d], wr[d]);
            }
            int ncell;
            if (BMODE == 2) {
                int r[3];
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    r[d] = c3[d] + unpack2(rcode, 16 * d + 14) - 1;
                    r[d] = r[d] < 0 ? r[d] + n3[d] : (r[d] >= n3[d] ? r[d] - n3[d] : r[d]);
                }
                ncell = g.cell_of(r[0], r[1], r[2]);
            } else {
                // within [x0, x0 + h] on every axis: stays (see k_push_plain)
                const bool inside = xr[0] >= o3[0] && xr[0] <= o3[0] + h3[0] && xr[1] >= o3[1] &&
                                    xr[1] <= o3[1] + h3[1] && xr[2] >= o3[2] && xr[2] <= o3[2] + h3[2];
                ncell = inside ? cell : new_cell_plain(g, cell, c3[0], c3[1], c3[2], xr, amb);
            }
            if (BMODE == 1) {
                unsigned long long code = 0ull;
                bool inrange = true;
                int r[3];
                g.cell_ijk(ncell, r[0], r[1], r[2]);
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    int mv = r[d] - c3[d];
                    mv = mv > 1 ? mv - n3[d] : (mv < -1 ? mv + n3[d] : mv);
                    inrange &= pack2(code, T[d].tn - 1, 16 * d);
                    inrange &= pack2(code, T[d].tc - 1, 16 * d + 2);
                    inrange &= pack2(code, T[d].nI - c3[d], 16 * d + 4);
                    inrange &= pack2(code, T[d].cI - c3[d], 16 * d + 6);
                    inrange &= pack2(code, SP.i1[d] - 1, 16 * d + 8);
                    inrange &= pack2(code, SP.i2[d] - 1, 16 * d + 10);
                    inrange &= pack2(code, wr[d], 16 * d + 12);
                    inrange &= pack2(code, mv + 1, 16 * d + 14);
                }
                P.branch[P.off[s] + j] = code;
                if (!inrange) bad |= ST_BRANCH_RANGE;
            }
            const FlatOut &O = P.out[s];
            O.cell[j] = ncell;
            O.v[0][j] = xr[0]; O.v[1][j] = xr[1]; O.v[2][j] = xr[2];
            O.v[3][j] = p[0]; O.v[4][j] = p[1]; O.v[5][j] = p[2];
        }
        if (DIRECT) continue;
        // ---- the warp's queued second segments, one per lane
        __syncwarp();
        qn = sQn[warp];
        if (qn >= (tail ? 1 : 16)) {
            const int d = qn < 32 ? qn : 32;
            if (lane < d) {
                const int e = qn - d + lane;
                const int code = qc[e], a = code >> 21, b = (code >> 12) & 511, c = (code >> 3) & 511;
                const int iv[3] = {2 + (code & 1), 2 + ((code >> 1) & 1), 2 + ((code >> 2) & 1)};
                double sa[3], se[3];
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    sa[q] = qd[q * kQueuePlain + e];
                    se[q] = qd[(3 + q) * kQueuePlain + e];
                }
                pqr_plain<true>((unsigned *)sJ, lo_scale, cn, dX, dY, a - 2, b - 2, c - 2, iv, sa, se, g.hx, g.hy, g.hz, rc,
                                (double)w.at(0, a) * g.hx, (double)w.at(1, b) * g.hy, (double)w.at(2, c) * g.hz, bad);
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
            long long ih, il;
            fx_get<true>((const unsigned *)sJ + a, 3 * cn, ih, il);
            size_t n;
            if ((ih == 0 && il == 0) || !w.grid_node(g, r, n)) continue;
            atomicAdd(&P.J[comp][n], ((double)ih + (double)il / lo_scale) * sQ);
        }
    }
    if (bad) atomicOr(&P.st->flags, bad);
    if (amb) atomicAdd(&P.st->ambiguous, amb);
    };
    if (!DIRECT && w.fixed()) body(std::true_type{});
    else body(std::false_type{});
}

// The taps in few registers: bit d tn - 2, bit 3 + d tc - 2, bit 6 + d cI - nI
// (wc = wn -+ 1/2), bit 9: a tap left the stencil (the forward has reported it)
struct PackedTaps {
    unsigned bits;
    double wn[3];
    __device__ __forceinline__ int tap(bool node, int d) const { return (int)(bits >> (node ? d : 3 + d)) & 1; }
    __device__ __forceinline__ double weight(bool node, int d) const {
        return node ? wn[d] : wn[d] + (bits >> (6 + d) & 1u ? 0.5 : -0.5);
    }
};
__device__ __forceinline__ PackedTaps pack_taps(const AxisTaps T[3]) {
    PackedTaps P;
    P.bits = 0u;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        P.bits |= ((unsigned)(T[d].tn - 2) & 1u) << d;
        P.bits |= ((unsigned)(T[d].tc - 2) & 1u) << (3 + d);
        P.bits |= ((unsigned)(T[d].cI - T[d].nI) & 1u) << (6 + d);
        if ((unsigned)(T[d].tn - 2) > 1u || (unsigned)(T[d].tc - 2) > 1u) P.bits |= 512u;
        P.wn[d] = T[d].wn;
    }
    return P;
}

// The reverse of one particle's step up to the adjoint of its interpolated
// fields: recomputes the push (cell indices c3, o3 the cell's corner, fields and
// lambda_J from V and LJ, L0 the cell's node in LJ with strides lx, ly), and
// transposes the deposit and the push.  In: gn, lP the incoming lambda_x and
// lambda_p (Reflect: identity).  Out: gx = lambda_x without the interpolation's
// part, lu = lambda_p, lF, the taps.  false: the push saw no field here.
struct ReverseConst {
    double h3[3], r3[3], rg[3], tau, tau1;
};
__device__ __forceinline__ ReverseConst reverse_const(const Grid &g, const FlatSp &S) {
    ReverseConst K;
    K.h3[0] = g.hx; K.h3[1] = g.hy; K.h3[2] = g.hz;
#pragma unroll
    for (int d = 0; d < 3; d++) K.r3[d] = 1.0 / K.h3[d];
    K.tau = g.tau;
    K.tau1 = S.q_m * g.tau * 0.5;
    K.rg[0] = S.m / (g.tau * g.hy * g.hz);
    K.rg[1] = S.m / (g.tau * g.hx * g.hz);
    K.rg[2] = S.m / (g.tau * g.hx * g.hy);
    return K;
}
template <class V>
__device__ __forceinline__ bool reverse_particle(const Grid &g, const ReverseConst &K, const V &A, const double *L0,
                                                 const double *L1, const double *L2, int ln, int lx, int ly,
                                                 const int c3[3], const double x[3], const double p[3], double gn[3],
                                                 double lP[3], PackedTaps &PT, double gx[3], double lu[3],
                                                 double lF[6]) {
    const double *h3 = K.h3, *r3 = K.r3;
    AxisTaps T[3];
    const double o3[3] = {(double)c3[0] * h3[0], (double)c3[1] * h3[1], (double)c3[2] * h3[2]};
    const bool seen = !(x[0] < 0 || x[1] < 0 || x[2] < 0);  // else the push saw zero fields
#pragma unroll
    for (int d = 0; d < 3; d++) axis_taps(x[d], o3[d], h3[d], r3[d], T[d]);
    double F[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (seen) gather_fields(A, T, F);
    BorisPlain B;
    boris_plain(K.tau1, F, p, B);
    Split SP;
    double x1[3];
    bool exact = true;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        x1[d] = x[d] + K.tau * (B.g2 * B.pp[d]);
        SP.i1[d] = T[d].i1;
        SP.i2[d] = trunc_checked((div_by(x1[d] - o3[d], h3[d], r3[d]) + 1.5) + 1, exact);
        gx[d] = 0.0;
    }
    PT = pack_taps(T);
    if (!exact) SP.i2[0] = 0;
    SP.m = relay_point(x, x1, o3, h3, SP.i1, SP.i2, SP.x2, SP.sr);
    // deposit transpose
    {
        auto rev = [&](const int iv[3], const double a[3], const double b[3], double ga[3], double gb[3]) {
            if (iv[0] < 2 || iv[0] > 3 || iv[1] < 2 || iv[1] > 3 || iv[2] < 2 || iv[2] > 3) return;
            seg_rev(L0, L1, L2, ln + (iv[0] - 2) * lx + (iv[1] - 2) * ly + (iv[2] - 2), lx, ly, g, iv, a, b, K.rg, o3, ga,
                    gb);
        };
        const bool cross = SP.m >= 1 && SP.m <= 7;
        double sb[3], g2[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int d = 0; d < 3; d++) sb[d] = cross ? SP.x2[d] : x1[d];
        rev(SP.i1, x, sb, gx, g2);
        if (cross) {
            rev(SP.i2, SP.x2, x1, g2, gn);
            split_rev(SP, x, x1, g2, gx, gn);
        } else {
#pragma unroll
            for (int d = 0; d < 3; d++) gn[d] += g2[d];
        }
    }
    // x1 = x + tau g2 p'
#pragma unroll
    for (int d = 0; d < 3; d++) gx[d] += gn[d];
    const double tg = K.tau * B.g2;
    const double dot = tg * B.g2 * B.g2 * fma(gn[0], B.pp[0], fma(gn[1], B.pp[1], gn[2] * B.pp[2]));
#pragma unroll
    for (int d = 0; d < 3; d++) lP[d] = fma(tg, gn[d], fma(-dot, B.pp[d], lP[d]));
    // p' = u' + t E, u' = (s + b (b.s) + s x b) / sd
    const double *b = B.b, *sv = B.s, *up = B.up, *u = B.u;
    const double inv = B.isd;
    const double bl = fma(b[0], lP[0], fma(b[1], lP[1], b[2] * lP[2]));
    const double bs = fma(b[0], sv[0], fma(b[1], sv[1], b[2] * sv[2]));
    const double lu_ = -2.0 * fma(lP[0], up[0], fma(lP[1], up[1], lP[2] * up[2]));
    double ls[3], lb[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int e = (d + 1) % 3, f = (d + 2) % 3;
        ls[d] = fma(b[d], bl, fma(b[e], lP[f], fma(-b[f], lP[e], lP[d]))) * inv;
        lb[d] = fma(bs, lP[d], fma(bl, sv[d], fma(lP[e], sv[f], fma(-lP[f], sv[e], lu_ * b[d])))) * inv;
    }
    // s = u + u x b
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int e = (d + 1) % 3, f = (d + 2) % 3;
        lu[d] = fma(b[e], ls[f], fma(-b[f], ls[e], ls[d]));
        lb[d] = fma(ls[e], u[f], fma(-ls[f], u[e], lb[d]));
    }
    // b = ps H, ps = t (1 + u^2)^-1/2; u = p + t E
    const double lps = fma(lb[0], F[3], fma(lb[1], F[4], lb[2] * F[5]));
    const double cps = -K.tau1 * B.g1 * B.g1 * B.g1 * lps;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        lu[d] = fma(cps, u[d], lu[d]);
        lF[d] = K.tau1 * (lP[d] + lu[d]);
        lF[3 + d] = B.ps * lb[d];
    }
    return seen && !(PT.bits & 512u);
}

// One component of the interpolation's transpose: gi += lam * dF/dx (V: the
// cell's node in the component's array, strides dX, dY), add(o, w): weight w
// belongs to the node o = (x, y, z) bits away from the tap base.
template <int C, class Add>
__device__ __forceinline__ void reverse_component(const double *V, int dX, int dY, const PackedTaps &T, double lam,
                                                  double gi[3], Add add) {
    constexpr bool nx = node_axis(C, 0), ny = node_axis(C, 1), nz = node_axis(C, 2);
    const int tx = T.tap(nx, 0), ty = T.tap(ny, 1), tz = T.tap(nz, 2);
    const double wx = T.weight(nx, 0), wy = T.weight(ny, 1), wz = T.weight(nz, 2);
    const double vx = 1. - wx, vy = 1. - wy, vz = 1. - wz;
    V += tx * dX + ty * dY + tz;
    // z, then y, then x: sums and differences
    double yl[2], yd[2], yz[2];
#pragma unroll
    for (int a = 0; a < 2; a++) {
        const double v0 = V[a * dX], v1 = V[a * dX + 1], v2 = V[a * dX + dY], v3 = V[a * dX + dY + 1];
        const double z0 = fma(vz, v1, wz * v0), z1 = fma(vz, v3, wz * v2);
        yl[a] = fma(vy, z1, wy * z0);
        yd[a] = z1 - z0;
        yz[a] = fma(vy, v3 - v2, wy * (v1 - v0));
    }
    gi[0] = fma(lam, yl[1] - yl[0], gi[0]);
    gi[1] = fma(lam, fma(vx, yd[1], wx * yd[0]), gi[1]);
    gi[2] = fma(lam, fma(vx, yz[1], wx * yz[0]), gi[2]);
#pragma unroll
    for (int t = 0; t < 4; t++) add(tx + (t >> 1), ty + (t & 1), tz, (t >> 1 ? vx : wx) * (t & 1 ? vy : wy), wz, vz);
}

// a particle outside its chunk's window: everything through global memory
__device__ __forceinline__ void reverse_global(const AdjParams &A, int s, int64_t j) {
    const FlatParams &P = A.f;
    const Grid &g = P.g;
    const FlatSp &S = P.sp[s];
    const LamSp &Lm = A.lam[s];
    const ReverseConst K = reverse_const(g, S);
    double x[3] = {S.v[0][j], S.v[1][j], S.v[2][j]}, p[3] = {S.v[3][j], S.v[4][j], S.v[5][j]};
    double gn[3] = {Lm.v[0][j], Lm.v[1][j], Lm.v[2][j]}, lP[3] = {Lm.v[3][j], Lm.v[4][j], Lm.v[5][j]};
    int c3[3];
    g.cell_ijk(S.cell[j], c3[0], c3[1], c3[2]);
    const size_t n = g.node(c3[0], c3[1], c3[2]);
    FieldView<false> V;
#pragma unroll
    for (int c = 0; c < 3; c++) { V.base[c] = P.E[c] + n; V.base[3 + c] = P.H[c] + n; }
    V.n0 = 0; V.dx = g.NY * g.pz; V.dy = g.pz;
    PackedTaps T;
    double gx[3], lu[3], lF[6], gi[3] = {0.0, 0.0, 0.0};
    if (reverse_particle(g, K, V, A.LJ[0] + n, A.LJ[1] + n, A.LJ[2] + n, 0, V.dx, V.dy, c3, x, p, gn, lP, T, gx, lu, lF)) {
        auto put = [&](double *L, double lam) {
            return [=](int tx, int ty, int tz, double xy, double wz, double vz) {
                double *r = L + tx * V.dx + ty * V.dy + tz;
                atomicAdd(r, lam * xy * wz);
                atomicAdd(r + 1, lam * xy * vz);
            };
        };
        reverse_component<0>(V.base[0], V.dx, V.dy, T, lF[0], gi, put(A.LE[0] + n, lF[0]));
        reverse_component<1>(V.base[1], V.dx, V.dy, T, lF[1], gi, put(A.LE[1] + n, lF[1]));
        reverse_component<2>(V.base[2], V.dx, V.dy, T, lF[2], gi, put(A.LE[2] + n, lF[2]));
        reverse_component<3>(V.base[3], V.dx, V.dy, T, lF[3], gi, put(A.LH[0] + n, lF[3]));
        reverse_component<4>(V.base[4], V.dx, V.dy, T, lF[4], gi, put(A.LH[1] + n, lF[4]));
        reverse_component<5>(V.base[5], V.dx, V.dy, T, lF[5], gi, put(A.LH[2] + n, lF[5]));
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
        Lm.v[d][j] = fma(gi[d], K.r3[d], gx[d]);
        Lm.v[3 + d][j] = lu[d];
    }
}

__device__ __noinline__ void reverse_far(const AdjParams &A, int s, int64_t j) { reverse_global(A, s, j); }
// all particles of a step that way
__global__ void __launch_bounds__(kT, kDirectAdjBlocks) k_adj_direct_plain(const __grid_constant__ AdjParams A) {
    chain_enter();
    const AdjChunk ch = A.f.chunks[blockIdx.x];
    const int lane = threadIdx.x & 31, mine = (lane >> 3) * 64 + (threadIdx.x >> 5) * 8 + (lane & 7);
    for (int e = mine; e < ch.count; e += blockDim.x) reverse_global(A, ch.species, ch.first + e);
}

// ---- adjoint of the particle part of one step: recompute the push, transpose
// the deposit and the push, transpose the interpolation.
//
// One CTA per chunk, with the chunk's window of E, H and lambda_J staged and
// lambda_E, lambda_H summed in shared memory (64-bit fixed point, added to the
// global arrays once); particles outside the window are done at the end through
// global memory.  The interpolated fields are formed again from the staged
// window instead of being kept by the forward (48 B written and read per
// particle and step).  The quantum follows the largest |lambda of a field
// value| of the 256 particles at hand: where that outgrows the quantum in use,
// the sums so far are added to the global arrays and start again at one that
// leaves 2^-48 of it.  A particle whose adjoints are not finite goes the same way
// as those outside: the FP64 sums in global memory then show it.
// Bound: latency at 16 warps per SM (128 registers, some spills) and the shared
// memory pipe (64 %: 91 shared atomics and 110 loads per particle).  128x32x32
// cells: 3.3 -> 2.3 ms per reverse step (before: two kernels, lambda of the
// field values and the fields themselves passed through global memory).
__global__ void __launch_bounds__(kT, 2) k_adj_particles_plain(const __grid_constant__ AdjParams A) {
    chain_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ AdjWindow<true> sWin;
    __shared__ int sRed[15 * kW], sFar;
    __shared__ unsigned sMax[kMaxSlots];
    const FlatParams &P = A.f;
    const Grid &g = P.g;
    const AdjChunk ch = P.chunks[blockIdx.x];
    const int s = ch.species, count = ch.count;
    const FlatSp &S = P.sp[s];
    const LamSp &Lm = A.lam[s];
    const NextParticle next(smem_raw + (size_t)kAdjWindow * 120);
    const NextLam lnext(smem_raw + (size_t)kAdjWindow * 120 + kNextBytes);
    unsigned short *sList =
        (unsigned short *)(smem_raw + (size_t)kAdjWindow * 120 + kNextBytes + kNextLamBytes);  // kAdjChunk entries
    __shared__ ReverseConst sK;  // in shared memory: registers are short
    // a warp takes 4 runs of 8 particles out of 4 places of the block's 256:
    // consecutive particles mostly share a cell, and adds to one address queue
    // up (one run of 32: 254 ps per particle and reverse step, 8 of 4: 189, 16 of
    // 2: 208, 4 of 8: 185; c3's 12.6M particles)
    const int lane = threadIdx.x & 31, mine = (lane >> 3) * 64 + (threadIdx.x >> 5) * 8 + (lane & 7);
    if (mine < count) {
        next.start(S, ch.first + mine);
        lnext.start(Lm, ch.first + mine);
    }
    const AdjWindow<true> w = chunk_window(g, S.cell + ch.first, count, kAdjWindow, sRed, &sWin);
    const int nn = w.nn, dX = w.SY * w.SZ, dY = w.SZ;
    double *sF = (double *)smem_raw, *sL = sF + 6 * nn;
    unsigned *sLo = (unsigned *)(sL + 3 * nn), *sHi = sLo + 6 * nn;
    const double *src[6] = {P.E[0], P.E[1], P.E[2], P.H[0], P.H[1], P.H[2]};
    stage_window<6>(g, w, nn, src, sF);
    stage_window<3>(g, w, nn, A.LJ, sL);
    for (int e = threadIdx.x; e < 12 * nn; e += blockDim.x) sLo[e] = 0u;
    if (threadIdx.x == 0) { sFar = 0; sMax[0] = sMax[1] = sMax[2] = 0u; sK = reverse_const(g, S); }
    __syncthreads();
    const ReverseConst &K = sK;
    // contributions below 2^50 quanta, at most kAdjChunk per node and component: sums below 2^61
    int E = kNoQuantum;
    double inv_q = 0.0;
    auto flush = [&](bool again) {
        if (E != kNoQuantum) {
            const double q = pow2_d(E - kBitsPlain);
            double *const dst[6] = {A.LE[0], A.LE[1], A.LE[2], A.LH[0], A.LH[1], A.LH[2]};
            for (int e = threadIdx.x; e < 6 * nn; e += blockDim.x) {
                const long long v = (long long)(((unsigned long long)sHi[e] << 32) | sLo[e]);
                if (v == 0) continue;
                if (again) sHi[e] = sLo[e] = 0u;
                const int comp = e / nn, r = e - comp * nn;
                        size_t n;
                        if (w.grid_node(g, r, n)) atomicAdd(&dst[comp][n], (double)v * q);
            }
        }
    };
    for (int base = 0, it = 0; base < count; base += blockDim.x, it++) {
        const int jc = base + mine;
        const int64_t j = ch.first + jc;
        int cell = -1;
        double x[3], p[3], gn[3], lP[3];
        cp_async_wait_all();
        if (jc < count) {
            cell = next.take(x, p);
            lnext.take(gn, lP);
        }
        __syncwarp();
        if (jc + (int)blockDim.x < count) {
            next.start(S, j + blockDim.x);
            lnext.start(Lm, j + blockDim.x);
        }
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
        PackedTaps T;
        double gx[3], lu[3], lF[6], gi[3] = {0.0, 0.0, 0.0};
        bool seen = false;
        unsigned amax = 0u;  // high word of the largest |lambda_F|
        if (near) {
            FieldView<true> V;
#pragma unroll
            for (int c = 0; c < 6; c++) V.base[c] = sF + c * nn;
            V.n0 = n0; V.dx = dX; V.dy = dY;
            seen = reverse_particle(g, K, V, sL, sL + nn, sL + 2 * nn, n0, dX, dY, c3, x, p, gn, lP, T, gx, lu, lF);
            if (seen) {
#pragma unroll
                for (int c = 0; c < 6; c++) amax = max(amax, (unsigned)__double2hiint(lF[c]) & 0x7fffffffu);
                if (amax >= 0x7ff00000u) {  // no fixed point for an infinity or a NaN
                    near = false;
                    amax = 0u;
                    sList[atomicAdd(&sFar, 1)] = (unsigned short)jc;
                }
            }
        }
        // the block's largest |lambda_F| against the quantum in use
        const unsigned wm = __reduce_max_sync(0xffffffffu, amax);
        if (lane == 0 && wm) atomicMax(&sMax[max_slot(it)], wm);
        __syncthreads();
        const unsigned bm = sMax[max_slot(it)];
        if (threadIdx.x == 0) sMax[max_cleared(it)] = 0u;
        const int En = bm ? quantum_for(E, exponent_hi(bm), kKeepPlain, kLeastPlain) : E;
        if (En != E) {  // block-uniform
            flush(true);
            E = En;
            inv_q = pow2_d(kBitsPlain - E);
            __syncthreads();
        }
        if (near && amax) {
            auto put = [&](int c) {
                const double lam = lF[c] * inv_q;
                unsigned *lo = sLo + c * nn + n0;
                return [=](int tx, int ty, int tz, double xy, double wz, double vz) {
                    unsigned *r = lo + tx * dX + ty * dY + tz;
                    const double v = lam * xy;
                    shared_add64(r, r + 6 * nn, __double_as_longlong(fma(v, wz, kRound)) - 0x4338000000000000ll);
                    shared_add64(r + 1, r + 1 + 6 * nn, __double_as_longlong(fma(v, vz, kRound)) - 0x4338000000000000ll);
                };
            };
            const double *V = sF + n0;
            reverse_component<0>(V, dX, dY, T, lF[0], gi, put(0));
            reverse_component<1>(V + nn, dX, dY, T, lF[1], gi, put(1));
            reverse_component<2>(V + 2 * nn, dX, dY, T, lF[2], gi, put(2));
            reverse_component<3>(V + 3 * nn, dX, dY, T, lF[3], gi, put(3));
            reverse_component<4>(V + 4 * nn, dX, dY, T, lF[4], gi, put(4));
            reverse_component<5>(V + 5 * nn, dX, dY, T, lF[5], gi, put(5));
        }
        if (near) {
#pragma unroll
            for (int d = 0; d < 3; d++) {
                Lm.v[d][j] = fma(gi[d], K.r3[d], gx[d]);
                Lm.v[3 + d][j] = lu[d];
            }
        }
    }
    __syncthreads();
    flush(false);
    for (int e = threadIdx.x; e < sFar; e += blockDim.x) reverse_far(A, s, ch.first + sList[e]);
}

// ------------------------------------------------------------- fields --
// Yee update ranges (MagneticFieldTrace, gpu_plasma.h:524-551; GetElectricFieldStartsDirs, gpu_plasma.h:286-304)
__device__ __forceinline__ bool in_H(const Grid &g, int c, int i, int l, int k) {
    if (i < 0 || l < 0 || k < 0) return false;
    if (c == 0) return i <= g.nx + 1 && l <= g.ny && k <= g.nz;
    if (c == 1) return i <= g.nx && l <= g.ny + 1 && k <= g.nz;
    return i <= g.nx && l <= g.ny && k <= g.nz + 1;
}
__device__ __forceinline__ bool in_E(const Grid &g, int c, int i, int l, int k) {
    if (i < 0 || l < 0 || k < 0 || i > g.nx || l > g.ny || k > g.nz) return false;
    if (c == 0) return l >= 1 && k >= 1;
    if (c == 1) return i >= 1 && k >= 1;
    return i >= 1 && l >= 1;
}

struct FieldAdj {
    Grid g;
    double cx, cy, cz, tau;
    double *LE[3], *LH[3], *LJ[3], *LQ[3];
};

// E update transpose (5) and the start of B completion's transpose (4):
//   lambda_J = -tau lambda_E on the E ranges, lambda_H += C^T lambda_E,
//   lambda_Q = lambda_H (new) on the H ranges
__global__ void k_adj_e_update(const __grid_constant__ FieldAdj A) {
    chain_enter();
    const Grid &g = A.g;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;  // node of an x plane
    if (q >= g.NY * g.NZ) return;
    const int l = q / g.NZ, k = q - l * g.NZ, i = blockIdx.y;
    size_t m = g.node(i, l, k);
    auto LEv = [&](int c, int di, int dl, int dk) -> double {
        return in_E(g, c, i + di, l + dl, k + dk) ? A.LE[c][g.node(i + di, l + dl, k + dk)] : 0.0;
    };
    double ex0 = LEv(0, 0, 0, 0), ey0 = LEv(1, 0, 0, 0), ez0 = LEv(2, 0, 0, 0);
    A.LJ[0][m] = -A.tau * ex0;
    A.LJ[1][m] = -A.tau * ey0;
    A.LJ[2][m] = -A.tau * ez0;
    double hx = A.LH[0][m] + A.cz * (ey0 - LEv(1, 0, 0, 1)) - A.cy * (ez0 - LEv(2, 0, 1, 0));
    double hy = A.LH[1][m] - A.cz * (ex0 - LEv(0, 0, 0, 1)) + A.cx * (ez0 - LEv(2, 1, 0, 0));
    double hz = A.LH[2][m] + A.cy * (ex0 - LEv(0, 0, 1, 0)) - A.cx * (ey0 - LEv(1, 1, 0, 0));
    A.LH[0][m] = hx;
    A.LH[1][m] = hy;
    A.LH[2][m] = hz;
    A.LQ[0][m] = in_H(g, 0, i, l, k) ? hx : 0.0;
    A.LQ[1][m] = in_H(g, 1, i, l, k) ? hy : 0.0;
    A.LQ[2][m] = in_H(g, 2, i, l, k) ? hz : 0.0;
}

// transpose of the B half step (1): lambda_Q += lambda_H_a on the H ranges,
// lambda_E += A^T lambda_Q (gather form: each E node collects from the Q
// nodes whose difference reads it).  Then the loss injection of the step before
// (inject: its E after the step, of component comp; null: none):
// lambda_E_comp += w2 E on nodes 1..N
template <typename T>
__global__ void k_adj_b_half(const __grid_constant__ FieldAdj A, const T *__restrict__ inject, int comp, double w2) {
    chain_enter();
    const Grid &g = A.g;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;  // node of an x plane
    if (q >= g.NY * g.NZ) return;
    const int l = q / g.NZ, k = q - l * g.NZ, i = blockIdx.y;
    size_t m = g.node(i, l, k);
    auto LQt = [&](int c, int di, int dl, int dk) -> double {
        int a = i + di, b = l + dl, cc = k + dk;
        if (!in_H(g, c, a, b, cc)) return 0.0;
        size_t q = g.node(a, b, cc);
        return A.LQ[c][q] + A.LH[c][q];
    };
    double qx = LQt(0, 0, 0, 0), qy = LQt(1, 0, 0, 0), qz = LQt(2, 0, 0, 0);
    // Qx = 0.5 (cz (Ey[+z] - Ey) - cy (Ez[+y] - Ez))
    // Qy = 0.5 (cx (Ez[+x] - Ez) - cz (Ex[+z] - Ex))
    // Qz = 0.5 (cy (Ex[+y] - Ex) - cx (Ey[+x] - Ey))
    double lex = -0.5 * A.cz * (LQt(1, 0, 0, -1) - qy) + 0.5 * A.cy * (LQt(2, 0, -1, 0) - qz);
    double ley = 0.5 * A.cz * (LQt(0, 0, 0, -1) - qx) - 0.5 * A.cx * (LQt(2, -1, 0, 0) - qz);
    double lez = -0.5 * A.cy * (LQt(0, 0, -1, 0) - qx) + 0.5 * A.cx * (LQt(1, -1, 0, 0) - qy);
    A.LE[0][m] += lex;
    A.LE[1][m] += ley;
    A.LE[2][m] += lez;
    if (inject && k >= 1 && k <= g.nz && l >= 1 && l <= g.ny && i >= 1 && i <= g.nx) A.LE[comp][m] += w2 * (double)inject[m];
}

// lines of one axis (getGlobalBoundaryCellNumber, cell.h:885-889)
__device__ __forceinline__ void line_g(const Grid &g, int dir, int a, int b, size_t &base, size_t &stride) {
    if (dir == 0) { base = (size_t)a * g.pz + b; stride = (size_t)g.NY * g.pz; }
    else if (dir == 1) { base = (size_t)a * g.NY * g.pz + b; stride = g.pz; }
    else { base = ((size_t)a * g.NY + b) * g.pz; stride = 1; }
}

// transpose of the J fold (pic_fold.cuh)
__global__ void k_adj_j_fold(Grid g, double *Lx, double *Ly, double *Lz) {
    chain_enter();
    double *const L[3] = {Lx, Ly, Lz};
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < fold_orbits(g)) fold_adjoint(g, L, idx);
}

// transpose of the E ghost copies E[0] = E[N], E[N+1] = E[1] (periodicElement, kernels.cu:1104-1110)
struct GPass {
    double *L;
    int dir, s1, e1, s2, e2, N;
};
struct GPasses {
    GPass p[3];
    int n;
};
__global__ void k_adj_ghosts(Grid g, GPasses P) {
    chain_enter();
    if ((int)blockIdx.y >= P.n) return;
    GPass q = P.p[blockIdx.y];
    int A = q.e1 - q.s1 + 1, B = q.e2 - q.s2 + 1;
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= A * B) return;
    size_t base, st;
    line_g(g, q.dir, q.s1 + idx / B, q.s2 + idx % B, base, st);
    double *L = q.L + base;
    size_t n1 = st, nN = (size_t)q.N * st, nN1 = (size_t)(q.N + 1) * st;
    L[n1] += L[nN1];
    L[nN1] = 0.0;
    L[nN] += L[0];
    L[0] = 0.0;
}

// loss injection of the last step: lambda_E_c += 2 w E_c on nodes 1..N
template <typename T>
__global__ void k_inject(Grid g, const T *__restrict__ E, double *LE, double w2) {
    int k = blockIdx.x * blockDim.x + threadIdx.x, l = blockIdx.y, i = blockIdx.z;
    if (k < 1 || k > g.nz || l < 1 || l > g.ny || i < 1 || i > g.nx) return;
    size_t n = g.node(i, l, k);
    LE[n] += w2 * (double)E[n];
}

// bins -> flat order (tile by tile, slot order): packed cell and FP64 values
__global__ void k_flat_gather_plain(SpeciesView S, const int64_t *__restrict__ d0, int *cell, double *x, double *y,
                                    double *z, double *px, double *py, double *pz) {
    int t = blockIdx.x;
    int start = S.tile_start[t], n = S.tile_count[t];
    int64_t base = d0[t];
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        int slot = start + j;
        int64_t d = base + j;
        cell[d] = S.cell[slot];
        x[d] = S.x[slot]; y[d] = S.y[slot]; z[d] = S.z[slot];
        px[d] = S.px[slot]; py[d] = S.py[slot]; pz[d] = S.pz[slot];
    }
}

// p += eps * dp for one species, dp interleaved (px, py, pz) in the order of
// pic_get_particles (tiles in order, slots in order)
__global__ void k_perturb_momenta(SpeciesView S, int mixed, const int64_t *__restrict__ d0,
                                  const double *__restrict__ dp, double eps) {
    const int t = blockIdx.x;
    const int start = S.tile_start[t], n = S.tile_count[t];
    const int64_t base = d0[t];
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const int slot = start + j;
        const double *q = dp + 3 * (base + j);
        if (mixed) {
            S.fx[slot] = (float)((double)S.fx[slot] + eps * q[0]);
            S.fy[slot] = (float)((double)S.fy[slot] + eps * q[1]);
            S.fz[slot] = (float)((double)S.fz[slot] + eps * q[2]);
        } else {
            S.px[slot] += eps * q[0];
            S.py[slot] += eps * q[1];
            S.pz[slot] += eps * q[2];
        }
    }
}

// d_drift and d_vth partial sums: out[0..2] += lambda_p, out[3] += lambda_p . (p - drift)
__global__ void k_param_grads(int64_t n, const double *__restrict__ lpx, const double *__restrict__ lpy,
                              const double *__restrict__ lpz, const double *__restrict__ px,
                              const double *__restrict__ py, const double *__restrict__ pz, double dx, double dy,
                              double dz, double *out4) {
    __shared__ double red[4][kT / 32];
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
        a[0] += lpx[j];
        a[1] += lpy[j];
        a[2] += lpz[j];
        a[3] += lpx[j] * (px[j] - dx) + lpy[j] * (py[j] - dy) + lpz[j] * (pz[j] - dz);
    }
    for (int q = 0; q < 4; q++)
        for (int o = 16; o > 0; o >>= 1) a[q] += __shfl_down_sync(0xffffffffu, a[q], o);
    int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int q = 0; q < 4; q++) red[q][w] = a[q];
    __syncthreads();
    if (threadIdx.x < 4) {
        double s = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) s += red[threadIdx.x][q];
        atomicAdd(&out4[threadIdx.x], s);
    }
}

// interleave (px, py, pz) of one species into n x 3
__global__ void k_interleave(int64_t n, const double *__restrict__ a, const double *__restrict__ b,
                             const double *__restrict__ c, double *out) {
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    out[3 * j] = a[j];
    out[3 * j + 1] = b[j];
    out[3 * j + 2] = c[j];
}

inline dim3 node_grid(const Grid &g) { return dim3((g.NZ + 31) / 32, g.NY, g.NX); }
inline dim3 plane_blocks(const Grid &g) { return dim3((g.NY * g.NZ + kT - 1) / kT, g.NX); }
inline unsigned blocks_of(int64_t n) { return (unsigned)((n + kT - 1) / kT); }

}  // namespace

// ======================================================== host: buffers ==
// One particle state of the whole population, carved from one allocation:
// per species the packed cells, then 6 value arrays, each 256-byte aligned.
size_t adj_state_bytes(const AdjState &A) {
    size_t b = 0;
    for (int s = 0; s < A.nsp; s++) {
        b += align256((size_t)A.n[s] * sizeof(int));
        b += 6 * align256((size_t)A.n[s] * A.elem);
    }
    return b;
}
void adj_state_view(const AdjState &A, char *base, int *cell[kMaxSpecies], void *v[kMaxSpecies][6]) {
    size_t o = 0;
    for (int s = 0; s < A.nsp; s++) {
        cell[s] = (int *)(base + o);
        o += align256((size_t)A.n[s] * sizeof(int));
        for (int a = 0; a < 6; a++) {
            v[s][a] = base + o;
            o += align256((size_t)A.n[s] * A.elem);
        }
    }
}

}  // namespace pic

using namespace pic;
using namespace pic_host;

namespace {

// ---- plain-form launch helpers
FlatParams flat_params(pic_handle *h, AdjState &A, char *state, void *const F[PIC_FIELD_COUNT],
                       char *out = nullptr) {
    FlatParams P;
    memset(&P, 0, sizeof(P));
    P.g = h->g;
    P.nsp = A.nsp;
    int *cell[kMaxSpecies];
    void *v[kMaxSpecies][6];
    adj_state_view(A, state, cell, v);
    P.off[0] = 0;
    for (int s = 0; s < A.nsp; s++) {
        P.sp[s].n = A.n[s];
        P.sp[s].q_m = h->sp[s].v.q_m;
        P.sp[s].m = h->sp[s].v.m;
        P.sp[s].cell = cell[s];
        for (int a = 0; a < 6; a++) P.sp[s].v[a] = (double *)v[s][a];
        P.off[s + 1] = P.off[s] + A.n[s];
    }
    for (int c = 0; c < 3; c++) {
        P.E[c] = (const double *)F[PIC_EX + c];
        P.H[c] = (const double *)F[PIC_HX + c];
        P.J[c] = (double *)F[PIC_JX + c];
    }
    adj_state_view(A, out ? out : state, cell, v);
    for (int s = 0; s < A.nsp; s++) {
        P.out[s].cell = cell[s];
        for (int a = 0; a < 6; a++) P.out[s].v[a] = (double *)v[s][a];
    }
    P.chunks = A.chunks;
    P.st = A.st;
    P.branch = A.step_branch;
    P.bmode = A.step_branch ? A.step_bmode : 0;
    return P;
}

int64_t total_particles(const AdjState &A) {
    int64_t t = 0;
    for (int s = 0; s < A.nsp; s++) t += A.n[s];
    return t;
}

// (see far_passed) two words in turn: the host has read one before the step that
// writes there again is enqueued
constexpr int kFarPoll = 8;
unsigned long long *far_slot(pic_handle *h, int n) { return (unsigned long long *)(h->hred + 6 + (n / kFarPoll & 1)); }
FarPost far_post(pic_handle *h, const AdjState &A, const double *hist, int n) {
    FarPost p;
    if (hist && n % kFarPoll == kFarPoll - 1 && n < A.direct_from) {
        p.far = A.far + n;
        p.host = far_slot(h, n);
        p.step = n;
    }
    return p;
}

// one forward step of the flat state on the field set F (plain): particles read
// from `state`, written to `out` (the same buffer when out is null).  keep: E and
// the half-step H of the step go there (six arrays; null: the half-step H to A.ha).
// hist: receives the sums of E_c^2 after the step (null: none, a recompute); n: the step.
// Five chained launches (before: eight operations, one after the other, and a
// copy of the fields in a recompute); the reverse of a step is six (before:
// eight).  Small runs wait on them: 16x8x8 cells, 24.6k particles, FP64 forward
// 33.0 -> 26.1 us per step, backward 93.8 -> 70.7; 64x32x32 cells, 3.1M FP32
// 201 -> 187 and 662 -> 630.
int flat_step_plain(pic_handle *h, AdjState &A, char *state, void *const F[PIC_FIELD_COUNT], char *out, char *keep,
                    double *hist, int n) {
    const Grid &g = h->g;
    cudaStream_t s = h->stream;
    const size_t N = g.nodes_pitched();
    double *Ha = keep ? (double *)keep + 3 * N : (double *)A.ha;
    flat_begin_plain(g, (const double *const *)&F[PIC_EX], (const double *const *)&F[PIC_HX], Ha, (double *)F[PIC_JX],
                     (double *)keep, s);  // J: the three arrays lie one after another
    FlatParams P = flat_params(h, A, state, F, out);
    for (int c = 0; c < 3; c++) P.H[c] = Ha + c * N;
    P.far = hist ? A.far + n : nullptr;
    if (A.nchunks > 0 && n >= A.direct_from) {
        auto *kern = P.bmode == 0 ? k_flat_push_plain<0, true>
                                  : (P.bmode == 1 ? k_flat_push_plain<1, true> : k_flat_push_plain<2, true>);
        CK(launch_chained(kern, dim3(A.nchunks), dim3(kT), s, P), "flat push");
    } else if (A.nchunks > 0) {
        auto *kern = P.bmode == 0 ? k_flat_push_plain<0, false>
                                  : (P.bmode == 1 ? k_flat_push_plain<1, false> : k_flat_push_plain<2, false>);
        const size_t smem = (size_t)kFlatWindow * (6 * sizeof(double) + 3 * 12) + (size_t)kW * kQueuePlain * 52 + kNextBytes;
        CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "flat push");
        CK(launch_chained_smem(kern, dim3(A.nchunks), dim3(kT), smem, s, P), "flat push");
    }
    fold_b_twice_plain(g, (double *const *)F, s);
    yee_e_update_plain(g, (double *const *)F, s);
    e_ghosts_plain(g, (double *)F[PIC_EX], (double *)F[PIC_EY], (double *)F[PIC_EZ],
                   h->cfg.ghosts == PIC_GHOSTS_PERIODIC, s, nullptr, nullptr, hist, nullptr, far_post(h, A, hist, n));
    CK(cudaGetLastError(), "flat step fields");
    return PIC_OK;
}

// ghost passes of e_ghosts_t (PeriodicBoundaries arguments, gpu_plasma.h:486-505), as two launches
void ghost_passes(const Grid &g, double *const L[3], int periodic, GPasses &A, GPasses &B, int &maxn) {
    A = GPasses{};
    B = GPasses{};
    maxn = 0;
    int Nx = g.nx, Ny = g.ny, Nz = g.nz;
    auto add = [&](GPasses &P, double *E, int dir, int s1, int e1, int s2, int e2, int N) {
        P.p[P.n++] = GPass{E, dir, s1, e1, s2, e2, N};
        int n = (e1 - s1 + 1) * (e2 - s2 + 1);
        if (n > maxn) maxn = n;
    };
    if (periodic) add(A, L[0], 1, 0, Nx, 1, Nz, Ny);
    add(A, L[1], 0, 0, Ny, 1, Nz, Nx);
    add(A, L[2], 0, 1, Ny, 0, Nz, Nx);
    add(B, L[0], 2, 0, Nx, 0, Ny + 1, Nz);
    add(B, L[1], 2, 0, Nx + 1, 0, Ny, Nz);
    if (periodic) add(B, L[2], 1, 0, Nx + 1, 0, Nz, Ny);
}

int check_adj_status(pic_handle *h, AdjState &A, const char *where) {
    AdjStatus st;
    CK(cudaMemcpyAsync(&st, A.st, sizeof(st), cudaMemcpyDeviceToHost, h->stream), "status");
    CK(cudaStreamSynchronize(h->stream), "sync");
    A.ambiguous = st.ambiguous;
    if (st.flags & ST_NAN) return set_err(h, PIC_ERR_NAN, "non-finite momentum in the differentiable run");
    if (st.flags & ST_BRANCH_RANGE)
        return set_err(h, PIC_ERR_STATE, "branch recording: a discrete choice outside its recorded range");
    if (st.flags & ST_STENCIL) {
        char msg[160];
        snprintf(msg, sizeof(msg), "%s: a particle moved more than half a cell in one step", where);
        return set_err(h, PIC_ERR_STENCIL, msg);
    }
    return PIC_OK;
}

// a buffer of the run: the one kept for this use when its size suits, else a new one
int adj_alloc(pic_handle *h, AdjSlot slot, void **p, size_t bytes, const char *what) {
    AdjState::Buf &b = h->adj->pool[slot];
    if (bytes == 0) bytes = 256;
    if (b.p && !kept_serves(b.cap, bytes)) {
        cudaFree(b.p);
        b.p = nullptr;
    }
    if (!b.p) {
        cudaError_t e = dev_alloc(h, &b.p, bytes);
        if (e != cudaSuccess) {
            b.p = nullptr;
            char msg[200];
            snprintf(msg, sizeof(msg), "differentiable run: cannot allocate %s (%.2f GB); use a larger ckpt_every or "
                     "fewer particles", what, bytes / 1e9);
            cudaGetLastError();
            return set_err(h, PIC_ERR_NOMEM, msg);
        }
        b.cap = bytes;
    }
    b.used = 1;
    *p = b.p;
    return PIC_OK;
}

}  // namespace

namespace pic_host {

void adj_free(pic_handle *h) {
    if (!h || !h->adj) return;
    AdjState *A = h->adj;
    for (AdjState::Buf &b : A->pool)
        if (b.p) cudaFree(b.p);
    if (A->e0) cudaEventDestroy(A->e0);
    if (A->e1) cudaEventDestroy(A->e1);
    delete A;
    h->adj = nullptr;
}

bool adj_reclaim(pic_handle *h) {
    if (!h || !h->adj) return false;
    bool any = false;
    for (AdjState::Buf &b : h->adj->pool)
        if (b.p && !b.used) {
            cudaFree(b.p);
            b.p = nullptr;
            any = true;
        }
    return any;
}

}  // namespace pic_host

// ====================================================== host: forward ==
namespace {

// field arrays of one state in the form's type: E, H (6 arrays)
inline size_t field_bytes(const pic_handle *h) {
    return h->g.nodes_pitched() * (h->mixed ? sizeof(float) : sizeof(double));
}
// recompute field set: E, H in the form's type, then J (and Q) in FP64
void rf_view(pic_handle *h, AdjState &A, void *RF[PIC_FIELD_COUNT]) {
    const size_t fb = field_bytes(h), db = h->g.nodes_pitched() * sizeof(double);
    for (int a = 0; a < PIC_FIELD_COUNT; a++)
        RF[a] = a < 6 ? A.rf + a * fb : A.rf + 6 * fb + (a - 6) * db;
    if (h->mixed) RF[PIC_QX] = RF[PIC_QY] = RF[PIC_QZ] = nullptr;
}

MixParams mix_params(pic_handle *h, AdjState &A, char *state, void *const F[PIC_FIELD_COUNT], char *out) {
    MixParams P;
    memset(&P, 0, sizeof(P));
    P.g = h->g;
    P.nsp = A.nsp;
    int *cell[kMaxSpecies];
    void *v[kMaxSpecies][6];
    adj_state_view(A, state, cell, v);
    P.off[0] = 0;
    for (int s = 0; s < A.nsp; s++) {
        P.sp[s].n = A.n[s];
        P.sp[s].q_m = h->sp[s].v.q_m;
        P.sp[s].m = h->sp[s].v.m;
        P.sp[s].cell = cell[s];
        for (int a = 0; a < 6; a++) P.sp[s].v[a] = (float *)v[s][a];
        P.off[s + 1] = P.off[s] + A.n[s];
    }
    adj_state_view(A, out ? out : state, cell, v);
    for (int s = 0; s < A.nsp; s++) {
        P.out[s].cell = cell[s];
        for (int a = 0; a < 6; a++) P.out[s].v[a] = (float *)v[s][a];
    }
    for (int c = 0; c < 3; c++) {
        P.E[c] = (const float *)F[PIC_EX + c];
        P.H[c] = (const float *)F[PIC_HX + c];
        P.J[c] = (double *)F[PIC_JX + c];
    }
    P.chunks = A.chunks;
    P.st = A.st;
    return P;
}

// one forward step of the fixed-order state on the field set F (see flat_step_plain)
int flat_step(pic_handle *h, AdjState &A, char *state, void *const F[PIC_FIELD_COUNT], char *out, char *keep,
              double *hist, int n) {
    if (!h->mixed) return flat_step_plain(h, A, state, F, out, keep, hist, n);
    const Grid &g = h->g;
    cudaStream_t s = h->stream;
    float *const *E = (float *const *)&F[PIC_EX];
    float *const *H = (float *const *)&F[PIC_HX];
    const size_t N = g.nodes_pitched();
    float *Ha = keep ? (float *)keep + 3 * N : (float *)A.ha;
    flat_begin_mixed(g, (const float *const *)E, (const float *const *)H, Ha, (double *)F[PIC_JX], (float *)keep, s);
    MixParams P = mix_params(h, A, state, F, out);
    for (int c = 0; c < 3; c++) P.H[c] = Ha + c * N;
    P.far = hist ? A.far + n : nullptr;
    CK(launch_flat_push_mixed(P, A.nchunks, n >= A.direct_from, s), "flat push");
    fold_b_mixed(g, E, H, (double *const *)&F[PIC_JX], s);
    yee_e_update_mixed(g, E, H, (double *const *)&F[PIC_JX], s);
    e_ghosts_mixed(g, E[0], E[1], E[2], h->cfg.ghosts == PIC_GHOSTS_PERIODIC, s, nullptr, nullptr, hist, nullptr,
                   far_post(h, A, hist, n));
    CK(cudaGetLastError(), "flat step fields");
    return PIC_OK;
}

// Steps without windows.  A chunk's particles share a window while they stay near
// each other; in a hot or long run they spread, and those outside the window go
// through global memory in kernels whose shared memory leaves no L1: with half of
// them outside the reverse step took 3 times as long as kernels without windows.  A
// run whose fraction outside passes far_limit therefore goes on without.  far[n] is
// that fraction's numerator of step n.  limit: where the two were equally fast
// (64x32x32 cells, vth .2, steps of half a cell at light speed; particles per cell and
// species p, fraction: FP64 forward 16 0, 64 .02, 250 .06, reverse 16 .02, 64 .03,
// 250 .13; FP32 forward 16 .02, 64 .5, 250 .65, reverse 16 .09, 64 .12, 250 .27).
// With vth .3 for 100 steps: FP64 960 and 5140 us per step forward and backward ->
// 610 and 2040, FP32 618 and 4250 -> 485 and 1720.
double far_limit(bool mixed, bool reverse, double p) {
    if (!mixed) return reverse ? .005 + p / 2000 : p / 4000;
    return reverse ? .08 + p / 1300 : std::min(.65, std::max(0.0, (p - 12) / 110));
}
// the first reverse step without windows: from the forward's counts, which end where
// it went on without windows itself; from there they grow as in the last 8 steps
int reverse_direct_from(const std::vector<int> &far, int known, double particles, double limit) {
    const int steps = (int)far.size();
    for (int n = 0; n < known; n++)
        if (far[n] > limit * particles) return n;
    if (known >= steps || known < 9) return known < steps ? known : steps;
    const double last = far[known - 1], slope = std::max(0.0, (last - far[known - 9]) / 8);
    for (int n = known; n < steps; n++)
        if (last + slope * (n - known + 1) > limit * particles) return n;
    return steps;
}

// The forward learns of far[n] from the kernels themselves: every kFarPoll steps the
// last kernel of a step writes the count and the step to pinned memory, and the host,
// which enqueues ahead, waits there for the count of kFarPoll + 1 steps ago.  The
// device still has kFarPoll steps to do then.
bool far_passed(pic_handle *h, int n, double limit) {
    const volatile unsigned long long *slot = far_slot(h, n);
    for (long long spin = 1;; spin++) {
        const unsigned long long v = *slot;
        if ((int)(v >> 32) >= n + 1) return (double)(unsigned)v > limit;
        // finished, or failed: the run's end reports it
        if (spin % 4096 == 0) {
            if (cudaStreamQuery(h->stream) != cudaErrorNotReady) return false;
            cudaGetLastError();  // not the next launch's
        }
    }
}

int forward_run(pic_handle *h, AdjState &A) {
    const Grid &g = h->g;
    cudaStream_t st = h->stream;
    const size_t fbytes = field_bytes(h);
    const double particles = (double)total_particles(A);
    const double limit = particles * far_limit(h->mixed, false, particles / ((double)A.nsp * g.ncells()));
    for (int q = 0; q < 2; q++) *(volatile unsigned long long *)far_slot(h, q * kFarPoll) = 0ull;
    CK(cudaEventRecord(A.e0, st), "event");
    for (int n = 0; n < A.steps; n++) {
        if (n >= 2 * kFarPoll && n % kFarPoll == 0 && A.direct_from == A.steps && far_passed(h, n - kFarPoll - 1, limit))
            A.direct_from = n;
        if (n % A.K == 0) {
            int c = n / A.K;
            CK(cudaMemcpyAsync(A.ckp + (size_t)c * A.pbytes, A.cur, A.pbytes, cudaMemcpyDeviceToDevice, st), "ckpt");
            for (int a = 0; a < 6; a++)
                CK(cudaMemcpyAsync(A.ckf + ((size_t)c * 6 + a) * fbytes, h->f[PIC_EX + a], fbytes,
                                   cudaMemcpyDeviceToDevice, st), "ckpt fields");
        }
        const size_t np_all = (size_t)total_particles(A);
        if (A.branch_mode == 1) {
            A.step_branch = A.branch + (size_t)n * np_all;
            A.step_bmode = 1;
        } else if (A.branch_mode == 2) {
            A.step_branch = const_cast<unsigned long long *>(A.branch_src) + (size_t)n * np_all;
            A.step_bmode = 2;
        }
        int rc = flat_step(h, A, A.cur, h->f, nullptr, nullptr, A.hist + 3 * n, n);
        A.step_branch = nullptr;
        A.step_bmode = 0;
        if (rc) return rc;
    }
    CK(cudaEventRecord(A.e1, st), "event");
    return PIC_OK;
}

// reverse of step n: EH = E before the step and H after its half step (form's
// type, 6 arrays); last: E after the step, for the last step of the run (else null).
// The loss of the other steps is injected at the end of the reverse of the step
// after them, whose E before the step is their E after it.
int reverse_step(pic_handle *h, AdjState &A, const pic_loss &L, int n, char *state, const char *EH, const char *last) {
    const Grid &g = h->g;
    cudaStream_t st = h->stream;
    const size_t N = g.nodes_pitched();
    const size_t fb = field_bytes(h);
    double *LE[3], *LH[3], *LJ[3], *LQ[3];
    for (int c = 0; c < 3; c++) {
        LE[c] = A.lamf + (0 + c) * N;
        LH[c] = A.lamf + (3 + c) * N;
        LJ[c] = A.lamf + (6 + c) * N;
        LQ[c] = A.lamf + (9 + c) * N;
    }
    const double w2 = 2.0 * g.hx * g.hy * g.hz;
    if (last && L.window >= 1) {
        const char *Ec = last + (size_t)L.field * fb;
        if (h->mixed) k_inject<float><<<node_grid(g), 32, 0, st>>>(g, (const float *)Ec, LE[L.field], w2);
        else k_inject<double><<<node_grid(g), 32, 0, st>>>(g, (const double *)Ec, LE[L.field], w2);
    }
    // ghost copies (second launch first)
    GPasses GA, GB;
    int maxn;
    ghost_passes(g, LE, h->cfg.ghosts == PIC_GHOSTS_PERIODIC, GA, GB, maxn);
    dim3 gg((maxn + 127) / 128, 3);
    launch_chained(k_adj_ghosts, gg, dim3(128), st, g, GB);
    launch_chained(k_adj_ghosts, gg, dim3(128), st, g, GA);
    FieldAdj FA;
    FA.g = g;
    FA.cx = g.tau / g.hx;
    FA.cy = g.tau / g.hy;
    FA.cz = g.tau / g.hz;
    FA.tau = g.tau;
    for (int c = 0; c < 3; c++) { FA.LE[c] = LE[c]; FA.LH[c] = LH[c]; FA.LJ[c] = LJ[c]; FA.LQ[c] = LQ[c]; }
    launch_chained(k_adj_e_update, plane_blocks(g), dim3(kT), st, FA);
    launch_chained(k_adj_j_fold, dim3((fold_orbits(g) + 127) / 128), dim3(128), st, g, LJ[0], LJ[1], LJ[2]);
    void *F[PIC_FIELD_COUNT] = {};
    for (int c = 0; c < 6; c++) F[PIC_EX + c] = (void *)(EH + c * fb);
    // E before this step, where the step before it has a loss term
    const char *inject = n >= 1 && n - 1 >= A.steps - L.window ? EH + (size_t)L.field * fb : nullptr;
    size_t o = 0;
    if (!h->mixed) {
        AdjParams P;
        memset(&P, 0, sizeof(P));
        P.f = flat_params(h, A, state, F);
        for (int s = 0; s < A.nsp; s++) {
            for (int a = 0; a < 6; a++) P.lam[s].v[a] = (double *)A.lamp + o + (size_t)a * A.n[s];
            o += 6 * (size_t)A.n[s];
        }
        for (int c = 0; c < 3; c++) { P.LJ[c] = LJ[c]; P.LE[c] = LE[c]; P.LH[c] = LH[c]; }
        if (A.nchunks > 0 && n >= A.direct_adj_from) {
            CK(launch_chained(k_adj_direct_plain, dim3(A.nchunks), dim3(kT), st, P), "adjoint particles");
        } else if (A.nchunks > 0) {
            const size_t smem = (size_t)kAdjWindow * 120 + kNextBytes + kNextLamBytes + kAdjChunk * sizeof(unsigned short);
            CK(cudaFuncSetAttribute(k_adj_particles_plain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
               "adjoint particles");
            CK(launch_chained_smem(k_adj_particles_plain, dim3(A.nchunks), dim3(kT), smem, st, P), "adjoint particles");
        }
        launch_chained(k_adj_b_half<double>, plane_blocks(g), dim3(kT), st, FA, (const double *)inject, L.field, w2);
    } else {
        MixParams P = mix_params(h, A, state, F, nullptr);
        for (int s = 0; s < A.nsp; s++) {
            for (int a = 0; a < 6; a++) P.lam[s][a] = (float *)A.lamp + o + (size_t)a * A.n[s];
            o += 6 * (size_t)A.n[s];
        }
        for (int c = 0; c < 3; c++) { P.LJ[c] = LJ[c]; P.LE[c] = LE[c]; P.LH[c] = LH[c]; }
        CK(launch_adj_particles_mixed(P, A.nchunks, n >= A.direct_adj_from, st), "adjoint particles");
        launch_chained(k_adj_b_half<float>, plane_blocks(g), dim3(kT), st, FA, (const float *)inject, L.field, w2);
    }
    CK(cudaGetLastError(), "reverse step");
    return PIC_OK;
}

int backward_run(pic_handle *h, AdjState &A, const pic_loss &L) {
    const Grid &g = h->g;
    cudaStream_t st = h->stream;
    const size_t N = g.nodes_pitched();
    const size_t fbytes = field_bytes(h);
    CK(cudaMemsetAsync(A.lamp, 0, A.lamp_bytes, st), "zero lambda");
    CK(cudaMemsetAsync(A.lamf, 0, 12 * N * sizeof(double), st), "zero lambda fields");
    void *RF[PIC_FIELD_COUNT];
    rf_view(h, A, RF);
    CK(cudaEventRecord(A.e0, st), "event");
    const size_t ehb = 6 * fbytes;  // E and H of one state (the first arrays of rf)
    for (int seg = A.nseg - 1; seg >= 0; seg--) {
        const int start = seg * A.K, end = std::min(start + A.K, A.steps), len = end - start;
        const int K2 = A.K2, nsub = (len + K2 - 1) / K2;
        if (nsub > 1) {
            // second level: recompute the segment once, keeping the state and E/H at
            // the start of every sub-segment (the running state lives in segp[0])
            CK(cudaMemcpyAsync(A.segp, A.ckp + (size_t)seg * A.pbytes, A.pbytes, cudaMemcpyDeviceToDevice, st),
               "restore");
            CK(cudaMemcpyAsync(A.rf, A.ckf + (size_t)seg * ehb, ehb, cudaMemcpyDeviceToDevice, st), "restore fields");
            for (int j = 0; j < len; j++) {
                if (j % K2 == 0) {
                    const int q = j / K2;
                    CK(cudaMemcpyAsync(A.subp + (size_t)q * A.pbytes, A.segp, A.pbytes, cudaMemcpyDeviceToDevice, st),
                       "sub-checkpoint");
                    CK(cudaMemcpyAsync(A.subf + (size_t)q * ehb, A.rf, ehb, cudaMemcpyDeviceToDevice, st),
                       "sub-checkpoint fields");
                    if (q == nsub - 1) break;  // the last sub-segment starts here
                }
                int rc = flat_step(h, A, A.segp, RF, nullptr, nullptr, nullptr, start + j);
                if (rc) return rc;
            }
        }
        for (int q = nsub - 1; q >= 0; q--) {
            const int s0 = start + q * K2, s1 = std::min(s0 + K2, end), slen = s1 - s0;
            const char *sp = nsub > 1 ? A.subp + (size_t)q * A.pbytes : A.ckp + (size_t)seg * A.pbytes;
            const char *sf = nsub > 1 ? A.subf + (size_t)q * ehb : A.ckf + (size_t)seg * ehb;
            CK(cudaMemcpyAsync(A.segp, sp, A.pbytes, cudaMemcpyDeviceToDevice, st), "restore");
            CK(cudaMemcpyAsync(A.rf, sf, ehb, cudaMemcpyDeviceToDevice, st), "restore fields");
            for (int j = 0; j < slen; j++) {
                int rc = flat_step(h, A, A.segp + (size_t)j * A.pbytes, RF, A.segp + (size_t)(j + 1) * A.pbytes,
                                   A.segf + (size_t)j * ehb, nullptr, s0 + j);
                if (rc) return rc;
            }
            for (int j = slen - 1; j >= 0; j--) {
                int rc = reverse_step(h, A, L, s0 + j, A.segp + (size_t)j * A.pbytes, A.segf + (size_t)j * ehb,
                                      s0 + j == A.steps - 1 ? A.rf : nullptr);
                if (rc) return rc;
            }
        }
    }
    CK(cudaEventRecord(A.e1, st), "event");
    return PIC_OK;
}

}  // namespace

// ============================================================ C ABI ==
extern "C" {

int pic_forward(pic_handle *h, int steps, int ckpt_every) { return pic_forward2(h, steps, ckpt_every, ckpt_every); }

// pic_forward2, or (src != null) a forward that replays the discrete choices
// recorded by src's last forward
static int forward_impl(pic_handle *h, int steps, int ckpt_every, int sub_every, const pic_handle *src) {
    if (!h) return PIC_ERR_ARG;
    if (steps < 1 || ckpt_every < 1) return set_err(h, PIC_ERR_ARG, "pic_forward: steps and ckpt_every must be >= 1");
    if (sub_every < 1 || sub_every > ckpt_every)
        return set_err(h, PIC_ERR_ARG, "pic_forward2: sub_every must be in 1..ckpt_every");
    int rc = set_device(h);
    if (rc) return rc;
    if ((rc = need_particles(h))) return rc;
    // the last run's buffers stay for this one
    AdjState *Ap = new AdjState();
    if (h->adj) {
        for (int q = 0; q < kAdjSlots; q++) {
            Ap->pool[q] = h->adj->pool[q];
            Ap->pool[q].used = 0;
            h->adj->pool[q].p = nullptr;
        }
        adj_free(h);
    }
    h->adj = Ap;
    AdjState &A = *Ap;
    A.mixed = h->mixed;
    A.elem = h->mixed ? sizeof(float) : sizeof(double);
    A.nsp = h->cfg.nspecies;
    A.steps = steps;
    A.K = ckpt_every;
    A.K2 = sub_every;
    A.nseg = (steps + ckpt_every - 1) / ckpt_every;
    const Grid &g = h->g;
    std::vector<std::vector<int>> counts(A.nsp);
    for (int s = 0; s < A.nsp; s++) {
        if ((rc = tile_counts(h, s, counts[s]))) return rc;
        int64_t t = 0;
        for (int c : counts[s]) t += c;
        A.n[s] = t;
    }
    A.pbytes = adj_state_bytes(A);
    std::vector<AdjChunk> chunks;
    {
        // each tile's particles of a species in equal chunks: large enough to
        // pay for a chunk's window, small enough to fill the GPU a few times
        const int64_t per = total_particles(A) / (8 * h->sms);
        const int most = (int)std::min<int64_t>(kAdjChunk, std::max<int64_t>(kT, (per + kT - 1) / kT * kT));
        for (int s = 0; s < A.nsp; s++) {
            int64_t at = 0;
            for (int c : counts[s]) {
                const int pieces = (c + most - 1) / most;
                for (int q = 0; q < pieces; q++) {
                    const int64_t a = (int64_t)c * q / pieces, b = (int64_t)c * (q + 1) / pieces;
                    chunks.push_back(AdjChunk{at + a, (int)(b - a), s});
                }
                at += c;
            }
        }
        A.nchunks = (int)chunks.size();
    }
    const size_t fbytes = g.nodes_pitched() * (h->mixed ? sizeof(float) : sizeof(double));
    if (src) {
        const AdjState *S = src->adj;
        bool same = S && S->branch && !h->mixed && S->nsp == A.nsp && S->steps >= steps;
        for (int s = 0; same && s < A.nsp; s++) same = S->n[s] == A.n[s];
        if (!same)
            return set_err(h, PIC_ERR_ARG,
                           "pic_forward_replay: the source needs a recorded FP64 forward of at least as many steps "
                           "and the same particle counts");
        A.branch_mode = 2;
        A.branch_src = S->branch;
    } else if (h->branch_record && !h->mixed) {
        if ((rc = adj_alloc(h, kAdjBranch, (void **)&A.branch,
                            (size_t)steps * (size_t)total_particles(A) * sizeof(unsigned long long),
                            "the branch record")))
            return rc;
        A.branch_mode = 1;
    }
    CK(cudaEventCreate(&A.e0), "event");
    CK(cudaEventCreate(&A.e1), "event");
    if ((rc = adj_alloc(h, kAdjCur, (void **)&A.cur, A.pbytes, "the particle state"))) return rc;
    if ((rc = adj_alloc(h, kAdjCkp, (void **)&A.ckp, A.pbytes * A.nseg, "the particle checkpoints"))) return rc;
    if ((rc = adj_alloc(h, kAdjCkf, (void **)&A.ckf, fbytes * 6 * A.nseg, "the field checkpoints"))) return rc;
    if ((rc = adj_alloc(h, kAdjHist, (void **)&A.hist, sizeof(double) * 4 * steps, "the history"))) return rc;
    if ((rc = adj_alloc(h, kAdjSt, (void **)&A.st, sizeof(AdjStatus), "the status"))) return rc;
    if ((rc = adj_alloc(h, kAdjRed, (void **)&A.red, sizeof(double) * 8, "the reduction scratch"))) return rc;
    if ((rc = adj_alloc(h, kAdjHa, (void **)&A.ha, fbytes * 3, "the half-step B"))) return rc;
    if ((rc = adj_alloc(h, kAdjChunks, (void **)&A.chunks, sizeof(AdjChunk) * chunks.size(), "the chunk table"))) return rc;
    CK(cudaMemcpyAsync(A.chunks, chunks.data(), sizeof(AdjChunk) * chunks.size(), cudaMemcpyHostToDevice, h->stream),
       "chunk table");
    CK(cudaStreamSynchronize(h->stream), "sync");
    // kept buffers that this run has no use for
    if (!A.branch && A.pool[kAdjBranch].p) { cudaFree(A.pool[kAdjBranch].p); A.pool[kAdjBranch].p = nullptr; }
    if (A.K2 == A.K)
        for (int q : {kAdjSubp, kAdjSubf})
            if (A.pool[q].p) { cudaFree(A.pool[q].p); A.pool[q].p = nullptr; }
    CK(cudaMemsetAsync(A.hist, 0, sizeof(double) * 4 * steps, h->stream), "zero history");
    A.far = (int *)(A.hist + 3 * steps);
    A.direct_from = A.direct_adj_from = steps;
    CK(cudaMemsetAsync(A.st, 0, sizeof(AdjStatus), h->stream), "zero status");
    // bins -> flat order
    int *cell[kMaxSpecies];
    void *v[kMaxSpecies][6];
    adj_state_view(A, A.cur, cell, v);
    int64_t *d0 = (int64_t *)h->dense;  // I/O staging, free between calls: a double per node, more than one per tile
    for (int s = 0; s < A.nsp; s++) {
        std::vector<int64_t> start(g.ntiles + 1);
        int64_t acc = 0;
        for (int t = 0; t < g.ntiles; t++) { start[t] = acc; acc += counts[s][t]; }
        start[g.ntiles] = acc;
        CK(cudaMemcpyAsync(d0, start.data(), (g.ntiles + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, h->stream),
           "H2D");
        if (!h->mixed)
            k_flat_gather_plain<<<g.ntiles, 256, 0, h->stream>>>(h->sp[s].v, d0, cell[s], (double *)v[s][0],
                                                                 (double *)v[s][1], (double *)v[s][2],
                                                                 (double *)v[s][3], (double *)v[s][4],
                                                                 (double *)v[s][5]);
        else
            adj_gather_mixed(g, h->sp[s].v, d0, cell[s], v[s], h->stream);
        CK(cudaGetLastError(), "flat gather");
        CK(cudaStreamSynchronize(h->stream), "sync");
    }
    rc = forward_run(h, A);
    if (rc) return rc;
    if ((rc = check_adj_status(h, A, "pic_forward"))) return rc;
    CK(cudaEventElapsedTime(&A.t_fwd, A.e0, A.e1), "timing");
    A.hhist.resize(3 * (size_t)steps);
    CK(cudaMemcpy(A.hhist.data(), A.hist, sizeof(double) * 3 * steps, cudaMemcpyDeviceToHost), "history");
    const double w = g.hx * g.hy * g.hz;
    for (double &x : A.hhist) x *= w;
    std::vector<int> far(steps);
    CK(cudaMemcpy(far.data(), A.far, sizeof(int) * steps, cudaMemcpyDeviceToHost), "particles outside the windows");
    A.direct_adj_from = reverse_direct_from(far, A.direct_from, (double)total_particles(A),
                                            far_limit(h->mixed, true, (double)total_particles(A) / ((double)A.nsp * g.ncells())));
    // the handle continues from the final state: flat order -> bins
    for (int s = 0; s < A.nsp; s++) {
        if (!h->mixed)
            rc = build_bins(h, s, A.n[s], cell[s], (const double *)v[s][0], (const double *)v[s][1],
                            (const double *)v[s][2], (const double *)v[s][3], (const double *)v[s][4],
                            (const double *)v[s][5], nullptr);
        else
            rc = build_bins_f(h, s, A.n[s], cell[s], (const float *)v[s][0], (const float *)v[s][1],
                              (const float *)v[s][2], (const float *)v[s][3], (const float *)v[s][4],
                              (const float *)v[s][5]);
        if (rc) return rc;
    }
    h->kin_valid = 0;
    A.have_forward = 1;
    return PIC_OK;
}

int pic_forward2(pic_handle *h, int steps, int ckpt_every, int sub_every) {
    return forward_impl(h, steps, ckpt_every, sub_every, nullptr);
}

int pic_branch_record(pic_handle *h, int on) {
    if (!h) return PIC_ERR_ARG;
    if (on && h->mixed) return set_err(h, PIC_ERR_ARG, "pic_branch_record: the FP64 plain form only");
    h->branch_record = on ? 1 : 0;
    return PIC_OK;
}

int pic_perturb_momenta(pic_handle *h, int species, int64_t n, const double *dp, double eps) {
    if (!h || species < 0 || species >= h->cfg.nspecies || n < 0 || (n > 0 && !dp))
        return set_err(h, PIC_ERR_ARG, "bad argument");
    int rc = set_device(h);
    if (rc) return rc;
    if ((rc = need_particles(h))) return rc;
    const Grid &g = h->g;
    std::vector<int> counts;
    if ((rc = tile_counts(h, species, counts))) return rc;
    std::vector<int64_t> d0(g.ntiles + 1);
    int64_t acc = 0;
    for (int t = 0; t < g.ntiles; t++) { d0[t] = acc; acc += counts[t]; }
    d0[g.ntiles] = acc;
    if (acc != n) return set_err(h, PIC_ERR_ARG, "pic_perturb_momenta: n is not the species' particle count");
    if (n == 0) return PIC_OK;
    ScratchGuard guard(h);
    int64_t *dd = nullptr;
    double *dv = nullptr;
    CK(guard.alloc(&dd, g.ntiles + 1), "alloc");
    CK(guard.alloc(&dv, (size_t)n * 3), "alloc");
    CK(cudaMemcpyAsync(dd, d0.data(), (g.ntiles + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, h->stream), "H2D");
    CK(cudaMemcpyAsync(dv, dp, (size_t)n * 3 * sizeof(double), cudaMemcpyHostToDevice, h->stream), "H2D");
    k_perturb_momenta<<<g.ntiles, 256, 0, h->stream>>>(h->sp[species].v, h->mixed, dd, dv, eps);
    CK(cudaGetLastError(), "perturb momenta");
    CK(cudaStreamSynchronize(h->stream), "perturb momenta");
    h->kin_valid = 0;
    return PIC_OK;
}

int pic_forward_replay(pic_handle *h, int steps, const pic_handle *recorded) {
    if (!h || !recorded) return PIC_ERR_ARG;
    if (h->mixed) return set_err(h, PIC_ERR_ARG, "pic_forward_replay: the FP64 plain form only");
    return forward_impl(h, steps, steps, steps, recorded);
}

int pic_forward_history(pic_handle *h, double *out) {
    if (!h || !out) return PIC_ERR_ARG;
    if (!h->adj || !h->adj->have_forward) return set_err(h, PIC_ERR_STATE, "no pic_forward run");
    memcpy(out, h->adj->hhist.data(), h->adj->hhist.size() * sizeof(double));
    return PIC_OK;
}

int pic_loss_value(pic_handle *h, const pic_loss *loss, double *value) {
    if (!h || !loss || !value) return PIC_ERR_ARG;
    if (!h->adj || !h->adj->have_forward) return set_err(h, PIC_ERR_STATE, "no pic_forward run");
    const AdjState &A = *h->adj;
    if (loss->field < 0 || loss->field > 2 || loss->window < 1 || loss->window > A.steps)
        return set_err(h, PIC_ERR_ARG, "pic_loss: field must be PIC_EX..PIC_EZ and window in 1..steps");
    double s = 0.0;
    for (int n = A.steps - loss->window; n < A.steps; n++) s += A.hhist[3 * (size_t)n + loss->field];
    *value = s;
    return PIC_OK;
}

int pic_backward(pic_handle *h, const pic_loss *loss, pic_grads *grads) {
    if (!h || !loss || !grads) return PIC_ERR_ARG;
    int rc = set_device(h);
    if (rc) return rc;
    if (!h->adj || !h->adj->have_forward) return set_err(h, PIC_ERR_STATE, "pic_backward needs a pic_forward run");
    AdjState &A = *h->adj;
    if ((rc = pic_loss_value(h, loss, &grads->loss))) return rc;
    if (loss->species < 0 || loss->species >= A.nsp) return set_err(h, PIC_ERR_ARG, "pic_loss: bad species");
    const Grid &g = h->g;
    const size_t N = g.nodes_pitched();
    const size_t fbytes = N * (h->mixed ? sizeof(float) : sizeof(double));
    int64_t np = total_particles(A);
    if (!A.rf) {  // the last of them: after a failure the next call gets the rest
        if ((rc = adj_alloc(h, kAdjSegp, (void **)&A.segp, A.pbytes * (size_t)(A.K2 + 1), "the segment states"))) return rc;
        if ((rc = adj_alloc(h, kAdjSegf, (void **)&A.segf, fbytes * 6 * (size_t)A.K2, "the segment fields"))) return rc;
        if (A.K2 < A.K) {
            const size_t nsub = (size_t)(A.K + A.K2 - 1) / A.K2;
            if ((rc = adj_alloc(h, kAdjSubp, (void **)&A.subp, A.pbytes * nsub, "the sub-checkpoint states"))) return rc;
            if ((rc = adj_alloc(h, kAdjSubf, (void **)&A.subf, fbytes * 6 * nsub, "the sub-checkpoint fields"))) return rc;
        }
        A.lamp_bytes = (size_t)np * 6 * A.elem;
        if ((rc = adj_alloc(h, kAdjLamp, (void **)&A.lamp, A.lamp_bytes, "the particle adjoints"))) return rc;
        if ((rc = adj_alloc(h, kAdjLamf, (void **)&A.lamf, N * sizeof(double) * 12, "the field adjoints"))) return rc;
        if ((rc = adj_alloc(h, kAdjRf, (void **)&A.rf, N * sizeof(double) * PIC_FIELD_COUNT, "the recompute fields")))
            return rc;
    }
    CK(cudaMemsetAsync(A.st, 0, sizeof(AdjStatus), h->stream), "zero status");
    rc = backward_run(h, A, *loss);
    if (rc) return rc;
    if ((rc = check_adj_status(h, A, "pic_backward"))) return rc;
    CK(cudaEventElapsedTime(&A.t_bwd, A.e0, A.e1), "timing");
    // gradients of the species' initial momenta (adjoint after the sweep) and
    // of its drift / spread; initial momenta from checkpoint 0
    const int s = loss->species;
    const int64_t n = A.n[s];
    size_t o = 0;
    for (int q = 0; q < s; q++) o += 6 * (size_t)A.n[q];
    int *cell0[kMaxSpecies];
    void *v0[kMaxSpecies][6];
    adj_state_view(A, A.ckp, cell0, v0);
    double out4[4] = {0.0, 0.0, 0.0, 0.0};
    double *lp = nullptr;  // FP64 copies of lambda_p (and p0) for the mixed form
    if (n > 0) {
        // their place, and the interleaved gradient's: the segment's states,
        // which the sweep is done with, where they are large enough
        ScratchGuard guard(h);
        const size_t lp_bytes = h->mixed ? align256((size_t)n * 6 * sizeof(double)) : 0;
        const size_t need = lp_bytes + (size_t)n * 3 * sizeof(double);
        char *stage = A.segp;
        if (A.pool[kAdjSegp].cap < need) CK(guard.alloc(&stage, need), "alloc");
        CK(cudaMemsetAsync(A.red, 0, 4 * sizeof(double), h->stream), "zero");
        const double *l3[3], *p3[3];
        if (!h->mixed) {
            for (int a = 0; a < 3; a++) {
                l3[a] = (const double *)A.lamp + o + (size_t)(3 + a) * n;
                p3[a] = (const double *)v0[s][3 + a];
            }
        } else {
            lp = (double *)stage;
            adj_widen_mixed((const float *)A.lamp + o + 3 * (size_t)n, (const float *const *)&v0[s][3], n, lp,
                            h->stream);
            for (int a = 0; a < 3; a++) {
                l3[a] = lp + (size_t)a * n;
                p3[a] = lp + (size_t)(3 + a) * n;
            }
        }
        k_param_grads<<<592, kT, 0, h->stream>>>(n, l3[0], l3[1], l3[2], p3[0], p3[1], p3[2], loss->drift[0],
                                                 loss->drift[1], loss->drift[2], A.red);
        CK(cudaMemcpyAsync(out4, A.red, 4 * sizeof(double), cudaMemcpyDeviceToHost, h->stream), "D2H");
        if (grads->d_p0 && grads->n >= n) {
            double *tmp = (double *)(stage + lp_bytes);
            k_interleave<<<blocks_of(n), kT, 0, h->stream>>>(n, l3[0], l3[1], l3[2], tmp);
            CK(cudaMemcpyAsync(grads->d_p0, tmp, (size_t)n * 3 * sizeof(double), cudaMemcpyDeviceToHost, h->stream),
               "D2H");
        }
        CK(cudaStreamSynchronize(h->stream), "sync");
    }
    bool fits = grads->n >= n;
    grads->n = n;
    for (int a = 0; a < 3; a++) grads->d_drift[a] = out4[a];
    grads->d_vth = loss->vth > 0 ? out4[3] / loss->vth : 0.0;
    if (grads->d_p0 && !fits) return set_err(h, PIC_ERR_ARG, "pic_grads: d_p0 capacity too small");
    return PIC_OK;
}

int pic_adjoint_timings(pic_handle *h, float *out2) {
    if (!h || !out2) return PIC_ERR_ARG;
    if (!h->adj) return set_err(h, PIC_ERR_STATE, "no differentiable run");
    out2[0] = h->adj->t_fwd;
    out2[1] = h->adj->t_bwd;
    return PIC_OK;
}

int pic_adjoint_free(pic_handle *h) {
    if (!h) return PIC_ERR_ARG;
    if (set_device(h)) return h->status;
    adj_free(h);
    return PIC_OK;
}

}  // extern "C"
