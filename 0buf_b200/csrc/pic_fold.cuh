// The periodic fold of the current and its transpose, all three axes and
// components in one pass.
//
// periodicCurrentElement (kernels.cu:1124-1146) on every line of the x, then the
// y, then the z axis (SetPeriodicCurrents, gpu_plasma.h:926-993) couples, per
// axis of N nodes, only the nodes of {0, N-2} and of {1, N-1}; the others stand
// alone.  Nodes therefore fall into orbits of 1, 2, 4 or 8 (one such pair per
// axis at most), no orbit touches another, and a thread that loads its orbit,
// applies the three axes in order in registers and stores it gives the bits of
// the three passes over memory without their launches.
#pragma once
#include "pic_internal.cuh"

namespace pic {

// orbits that hold a pair on some axis
__host__ __device__ inline int fold_orbits(const Grid &g) {
    return 2 * g.ny * g.nz + (g.nx - 2) * 2 * g.nz + (g.nx - 2) * (g.ny - 2) * 2;
}
// classes per axis of orbit idx: 0 the pair {0, N-2}, 1 the pair {1, N-1}, c >= 2 the node c
__device__ __forceinline__ void fold_classes(const Grid &g, int idx, int c[3]) {
    const int a = 2 * g.ny * g.nz, b = (g.nx - 2) * 2 * g.nz;
    if (idx < a) {
        c[2] = idx % g.nz;
        c[1] = (idx / g.nz) % g.ny;
        c[0] = idx / (g.nz * g.ny);
    } else if (idx < a + b) {
        idx -= a;
        c[2] = idx % g.nz;
        c[1] = (idx / g.nz) % 2;
        c[0] = 2 + idx / (2 * g.nz);
    } else {
        idx -= a + b;
        c[2] = idx % 2;
        c[1] = 2 + (idx / 2) % (g.ny - 2);
        c[0] = 2 + idx / (2 * (g.ny - 2));
    }
}

// loads orbit idx of A (component comp), applies op(axis, class, lower, upper)
// to its pairs, axis by axis in the order first, first + step, ..., and stores it
template <class Op>
__device__ __forceinline__ void fold_orbit(const Grid &g, double *A, int idx, bool reverse, Op op) {
    int c[3];
    fold_classes(g, idx, c);
    const int N[3] = {g.NX, g.NY, g.NZ};
    const size_t st[3] = {(size_t)g.NY * g.pz, (size_t)g.pz, 1};
    size_t base = 0, up[3];
    bool pair[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        pair[d] = c[d] < 2;
        base += (size_t)c[d] * st[d];
        up[d] = pair[d] ? (size_t)(N[d] - 2) * st[d] : 0;  // 0 -> N-2, 1 -> N-1
    }
    double v[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const bool have = (!(q & 4) || pair[0]) && (!(q & 2) || pair[1]) && (!(q & 1) || pair[2]);
        v[q] = have ? A[base + (q & 4 ? up[0] : 0) + (q & 2 ? up[1] : 0) + (q & 1 ? up[2] : 0)] : 0.0;
    }
#pragma unroll
    for (int e = 0; e < 3; e++) {
        const int d = reverse ? 2 - e : e, bit = 4 >> d;
        if (!pair[d]) continue;
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (!(q & bit)) op(d, c[d], v[q], v[q | bit]);
    }
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const bool have = (!(q & 4) || pair[0]) && (!(q & 2) || pair[1]) && (!(q & 1) || pair[2]);
        if (have) A[base + (q & 4 ? up[0] : 0) + (q & 2 ? up[1] : 0) + (q & 1 ? up[2] : 0)] = v[q];
    }
}

// the fold: J1 += J[N-1] (not along the component's own axis), J[N-1] = J1 (not
// y of Jy); J0 += J[N-2], J[N-2] = J0
__device__ __forceinline__ void fold_current(const Grid &g, double *const J[3], int idx) {
#pragma unroll
    for (int comp = 0; comp < 3; comp++)
        fold_orbit(g, J[comp], idx, false, [&](int d, int cls, double &a, double &b) {
            if (cls == 1) {
                if (d != comp) a += b;
                if (d != 1 || comp != 1) b = a;
            } else {
                a += b;
                b = a;
            }
        });
}
// its transpose
__device__ __forceinline__ void fold_adjoint(const Grid &g, double *const L[3], int idx) {
#pragma unroll
    for (int comp = 0; comp < 3; comp++)
        fold_orbit(g, L[comp], idx, true, [&](int d, int cls, double &a, double &b) {
            if (cls == 1) {
                if (d != 1 || comp != 1) {
                    a += b;
                    b = 0.0;
                }
                if (d != comp) b += a;
            } else {
                a += b;
                b = 0.0;
                b += a;
            }
        });
}

}  // namespace pic
