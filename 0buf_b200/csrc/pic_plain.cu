// Plain form (FP64, reference arithmetic) kernels of the B200 PIC step.
//
// Compiled with -fmad=false.  The field kernels evaluate the reference's FP64
// expressions in the reference's order (citations per function) as separate IEEE
// multiplies and adds like its host build: given the same current, the fields match
// the CPU oracle bit for bit.  The push takes every index, crossing and wrap from its
// positions as the reference does, bit for bit; its continuous values
// (interpolation, rotation, weights) are fused and rounded once where the reference
// rounds twice (pic_plain_math.cuh), and the current is summed in fixed point.
#include <cuda_runtime.h>
#include <math.h>
#include <algorithm>
#include "pic_internal.cuh"
#include "pic_kernels.cuh"
#include "pic_plain_math.cuh"
#include "pic_fold.cuh"

namespace pic {
namespace {

// ------------------------------------------------------------------ Yee --
// emh1_Element (kernels.cu:1052-1073) for the three components over the
// MagneticFieldTrace ranges of MagneticStageOne (gpu_plasma.h:524-538):
//   Hx: i<=Nx+1, l<=Ny, k<=Nz   Q = 0.5*(tau/hz*(Ey[+z]-Ey) - tau/hy*(Ez[+y]-Ez))
//   Hy: i<=Nx, l<=Ny+1, k<=Nz   Q = 0.5*(tau/hx*(Ez[+x]-Ez) - tau/hz*(Ex[+z]-Ex))
//   Hz: i<=Nx, l<=Ny, k<=Nz+1   Q = 0.5*(tau/hy*(Ex[+y]-Ex) - tau/hx*(Ey[+x]-Ey))
__global__ void k_b_half_plain(Grid g, const double *__restrict__ Ex, const double *__restrict__ Ey,
                               const double *__restrict__ Ez, double *Hx, double *Hy, double *Hz, double *Qx,
                               double *Qy, double *Qz, double cx, double cy, double cz,
                               unsigned long long *stamps) {
    chain_enter();
    stamp_entry(stamps, 0);
    // one thread per node of an x plane (l, k flattened: no idle z tail)
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= g.NY * g.NZ) return;
    const int l = q / g.NZ, k = q - l * g.NZ, i = blockIdx.y;
    size_t n = g.node(i, l, k);
    size_t sx = (size_t)g.NY * g.pz, sy = g.pz;
    if (i <= g.nx + 1 && l <= g.ny && k <= g.nz) {
        double e1_n1 = Ey[n + 1], e1_n = Ey[n], e2_n2 = Ez[n + sy], e2_n = Ez[n];
        double t = 0.5 * (cz * (e1_n1 - e1_n) - cy * (e2_n2 - e2_n));
        Qx[n] = t;
        Hx[n] += t;
    }
    if (i <= g.nx && l <= g.ny + 1 && k <= g.nz) {
        double e1_n1 = Ez[n + sx], e1_n = Ez[n], e2_n2 = Ex[n + 1], e2_n = Ex[n];
        double t = 0.5 * (cx * (e1_n1 - e1_n) - cz * (e2_n2 - e2_n));
        Qy[n] = t;
        Hy[n] += t;
    }
    if (i <= g.nx && l <= g.ny && k <= g.nz + 1) {
        double e1_n1 = Ex[n + sy], e1_n = Ex[n], e2_n2 = Ey[n + sx], e2_n = Ey[n];
        double t = 0.5 * (cy * (e1_n1 - e1_n) - cx * (e2_n2 - e2_n));
        Qz[n] = t;
        Hz[n] += t;
    }
}

// emh2_Element (kernels.cu:1024-1049) over the same ranges; q: node of x plane i
// (l, k flattened: no idle z tail)
__device__ __forceinline__ void b_complete_node(const Grid &g, int i, int q, double *Hx, double *Hy, double *Hz,
                                                const double *__restrict__ Qx, const double *__restrict__ Qy,
                                                const double *__restrict__ Qz) {
    if (q >= g.NY * g.NZ) return;
    const int l = q / g.NZ, k = q - l * g.NZ;
    size_t n = g.node(i, l, k);
    if (i <= g.nx + 1 && l <= g.ny && k <= g.nz) Hx[n] += Qx[n];
    if (i <= g.nx && l <= g.ny + 1 && k <= g.nz) Hy[n] += Qy[n];
    if (i <= g.nx && l <= g.ny && k <= g.nz + 1) Hz[n] += Qz[n];
}
__global__ void k_b_complete_plain(Grid g, double *Hx, double *Hy, double *Hz, const double *__restrict__ Qx,
                                   const double *__restrict__ Qy, const double *__restrict__ Qz) {
    chain_enter();
    b_complete_node(g, blockIdx.y, blockIdx.x * blockDim.x + threadIdx.x, Hx, Hy, Hz, Qx, Qy, Qz);
}
// the J fold and the B completion, which touch different arrays, in one launch:
// the first `folds` blocks fold, the others complete
__global__ void k_fold_b_plain(Grid g, int folds, int per_plane, double *Jx, double *Jy, double *Jz, double *Hx,
                               double *Hy, double *Hz, const double *__restrict__ Qx, const double *__restrict__ Qy,
                               const double *__restrict__ Qz, unsigned long long *stamps) {
    chain_enter();
    stamp_entry(stamps, 4);
    if ((int)blockIdx.x < folds) {
        double *const J[3] = {Jx, Jy, Jz};
        const int idx = blockIdx.x * blockDim.x + threadIdx.x;
        if (idx < fold_orbits(g)) fold_current(g, J, idx);
        return;
    }
    const int b = blockIdx.x - folds, i = b / per_plane;
    b_complete_node(g, i, (b - i * per_plane) * blockDim.x + threadIdx.x, Hx, Hy, Hz, Qx, Qy, Qz);
}


// Q of emh1_Element at a node of the given component's range (k_b_half_plain's expressions)
template <int C>
__device__ __forceinline__ double q_plain(const double *__restrict__ Ex, const double *__restrict__ Ey,
                                          const double *__restrict__ Ez, size_t n, size_t sx, size_t sy, double cx,
                                          double cy, double cz) {
    if (C == 0) return 0.5 * (cz * (Ey[n + 1] - Ey[n]) - cy * (Ez[n + sy] - Ez[n]));
    if (C == 1) return 0.5 * (cx * (Ez[n + sx] - Ez[n]) - cz * (Ex[n + 1] - Ex[n]));
    return 0.5 * (cy * (Ex[n + sy] - Ex[n]) - cx * (Ey[n + sx] - Ey[n]));
}
// (see flat_begin_plain) one thread per node of an x plane, z pads included
__global__ void k_flat_begin_plain(Grid g, const double *__restrict__ Ex, const double *__restrict__ Ey,
                                   const double *__restrict__ Ez, const double *__restrict__ Hx,
                                   const double *__restrict__ Hy, const double *__restrict__ Hz, double *Ha, double *J,
                                   double *keepE, double cx, double cy, double cz) {
    chain_enter();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= g.NY * g.pz) return;
    const int l = q / g.pz, k = q - l * g.pz, i = blockIdx.y;
    const size_t n = g.node(i, l, k), N = g.nodes_pitched();
    J[n] = 0.0;
    J[N + n] = 0.0;
    J[2 * N + n] = 0.0;
    if (k >= g.NZ) return;
    const size_t sx = (size_t)g.NY * g.pz, sy = g.pz;
    double hx = Hx[n], hy = Hy[n], hz = Hz[n];
    if (i <= g.nx + 1 && l <= g.ny && k <= g.nz) hx += q_plain<0>(Ex, Ey, Ez, n, sx, sy, cx, cy, cz);
    if (i <= g.nx && l <= g.ny + 1 && k <= g.nz) hy += q_plain<1>(Ex, Ey, Ez, n, sx, sy, cx, cy, cz);
    if (i <= g.nx && l <= g.ny && k <= g.nz + 1) hz += q_plain<2>(Ex, Ey, Ez, n, sx, sy, cx, cy, cz);
    Ha[n] = hx;
    Ha[N + n] = hy;
    Ha[2 * N + n] = hz;
    if (keepE) {
        keepE[n] = Ex[n];
        keepE[N + n] = Ey[n];
        keepE[2 * N + n] = Ez[n];
    }
}
// (see fold_b_twice_plain) the first `folds` blocks fold, the others step B
__global__ void k_fold_b_twice_plain(Grid g, int folds, int per_plane, double *Jx, double *Jy, double *Jz,
                                     const double *__restrict__ Ex, const double *__restrict__ Ey,
                                     const double *__restrict__ Ez, double *Hx, double *Hy, double *Hz, double *Qx,
                                     double *Qy, double *Qz, double cx, double cy, double cz) {
    chain_enter();
    if ((int)blockIdx.x < folds) {
        double *const J[3] = {Jx, Jy, Jz};
        const int idx = blockIdx.x * blockDim.x + threadIdx.x;
        if (idx < fold_orbits(g)) fold_current(g, J, idx);
        return;
    }
    const int b = blockIdx.x - folds, i = b / per_plane;
    const int q = (b - i * per_plane) * blockDim.x + threadIdx.x;
    if (q >= g.NY * g.NZ) return;
    const int l = q / g.NZ, k = q - l * g.NZ;
    const size_t n = g.node(i, l, k), sx = (size_t)g.NY * g.pz, sy = g.pz;
    if (i <= g.nx + 1 && l <= g.ny && k <= g.nz) {
        const double t = q_plain<0>(Ex, Ey, Ez, n, sx, sy, cx, cy, cz);
        if (Qx) Qx[n] = t;
        Hx[n] = (Hx[n] + t) + t;
    }
    if (i <= g.nx && l <= g.ny + 1 && k <= g.nz) {
        const double t = q_plain<1>(Ex, Ey, Ez, n, sx, sy, cx, cy, cz);
        if (Qy) Qy[n] = t;
        Hy[n] = (Hy[n] + t) + t;
    }
    if (i <= g.nx && l <= g.ny && k <= g.nz + 1) {
        const double t = q_plain<2>(Ex, Ey, Ez, n, sx, sy, cx, cy, cz);
        if (Qz) Qz[n] = t;
        Hz[n] = (Hz[n] + t) + t;
    }
}

// emeElement (kernels.cu:1091-1102) over GetElectricFieldStartsDirs ranges
// (gpu_plasma.h:286-304) as called by ElectricFieldEvaluate (gpu_plasma.h:455-483):
//   Ex: i in [0,Nx], l in [1,Ny], k in [1,Nz]: += tau/hy*(Hz-Hz[-y]) - tau/hz*(Hy-Hy[-z]) - tau*Jx
//   Ey: i in [1,Nx], l in [0,Ny], k in [1,Nz]: += tau/hz*(Hx-Hx[-z]) - tau/hx*(Hz-Hz[-x]) - tau*Jy
//   Ez: i in [1,Nx], l in [1,Ny], k in [0,Nz]: += tau/hx*(Hy-Hy[-x]) - tau/hy*(Hx-Hx[-y]) - tau*Jz
__global__ void k_e_update_plain(Grid g, double *Ex, double *Ey, double *Ez, const double *__restrict__ Hx,
                                 const double *__restrict__ Hy, const double *__restrict__ Hz,
                                 const double *__restrict__ Jx, const double *__restrict__ Jy,
                                 const double *__restrict__ Jz, double cx, double cy, double cz, double tau) {
    chain_enter();
    // one thread per node of an x plane (l, k flattened: no idle z tail)
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= g.NY * g.NZ) return;
    const int l = q / g.NZ, k = q - l * g.NZ, i = blockIdx.y;
    size_t n = g.node(i, l, k);
    size_t sx = (size_t)g.NY * g.pz, sy = g.pz;
    if (i <= g.nx && l >= 1 && l <= g.ny && k >= 1 && k <= g.nz)
        Ex[n] += cy * (Hz[n] - Hz[n - sy]) - cz * (Hy[n] - Hy[n - 1]) - tau * Jx[n];
    if (i >= 1 && i <= g.nx && l <= g.ny && k >= 1 && k <= g.nz)
        Ey[n] += cz * (Hx[n] - Hx[n - 1]) - cx * (Hz[n] - Hz[n - sx]) - tau * Jy[n];
    if (i >= 1 && i <= g.nx && l >= 1 && l <= g.ny && k <= g.nz)
        Ez[n] += cx * (Hy[n] - Hy[n - sx]) - cy * (Hx[n] - Hx[n - sy]) - tau * Jz[n];
}


// --------------------------------------------------------- boundaries --
// A "line" is the set of nodes along one axis at fixed other two indices.
struct Line {
    size_t base, stride;
};
__device__ __forceinline__ Line line_of(const Grid &g, int dir, int a, int b) {
    // getGlobalBoundaryCellNumber, cell.h:885-889: dir 0 -> (N, a, b), 1 -> (a, N, b), 2 -> (a, b, N)
    Line L;
    if (dir == 0) { L.base = (size_t)a * g.pz + b; L.stride = (size_t)g.NY * g.pz; }
    else if (dir == 1) { L.base = (size_t)a * g.NY * g.pz + b; L.stride = g.pz; }
    else { L.base = ((size_t)a * g.NY + b) * g.pz; L.stride = 1; }
    return L;
}

// periodicCurrentElement (kernels.cu:1124-1146) on all axes (pic_fold.cuh).  One
// launch instead of one per axis (with the other launches saved, the field kernels
// of a 32x4x4 step 21.4 -> 13.3 us).
__global__ void k_j_fold(Grid g, double *Jx, double *Jy, double *Jz) {
    chain_enter();
    double *const J[3] = {Jx, Jy, Jz};
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < fold_orbits(g)) fold_current(g, J, idx);
}

// PeriodicBoundaries (gpu_plasma.h:802-870) = periodicElement (kernels.cu:1104-1110)
// E[0] = E[N] then E[N+1] = E[1] on each line of [s1,e1] x [s2,e2]
struct GhostPass {
    void *E;
    int dir, s1, e1, s2, e2, N;
};
// The reference runs the passes in two rounds, A then B.  No node is written
// by both rounds, and no A pass reads a node that B writes; the only order
// between them is B reading ghosts that A wrote.  All passes are copies, so B
// reading A's source node instead gives the same bits, and both rounds run
// in one launch: passes p[0 .. nA) are A, p[nA .. n) are B.
struct GhostPasses {
    GhostPass p[6];
    int nA, n;
};
// node (c[0], c[1], c[2]) of array E, moved to the node an A pass copies into
// it when an A pass writes it
__device__ __forceinline__ size_t ghost_source(const Grid &g, const GhostPasses &P, const void *E, int c[3]) {
    for (int a = 0; a < P.nA; a++) {
        const GhostPass &q = P.p[a];
        if (q.E != E) continue;
        const int d = q.dir;
        const int ca = d == 0 ? c[1] : c[0], cb = d == 2 ? c[1] : c[2];  // the line's (a, b), as in line_of
        if (ca < q.s1 || ca > q.e1 || cb < q.s2 || cb > q.e2) continue;
        if (c[d] == 0) c[d] = q.N;
        else if (c[d] == q.N + 1) c[d] = 1;
    }
    return g.node(c[0], c[1], c[2]);
}
// out (pinned host memory, may be null): the step's status goes there with this
// last kernel of a step instead of by a copy after it.  hist (may be null):
// the sums over nodes 1..N of E_c^2, which no pass writes, are added to it by
// the rows of blocks after the passes'
constexpr int kHistRows = 4;
template <typename T>
__global__ void k_e_ghosts(Grid g, GhostPasses P, const DevStatus *st, DevStatus *out, const T *__restrict__ Ex,
                           const T *__restrict__ Ey, const T *__restrict__ Ez, double *hist,
                           unsigned long long *stamps, FarPost post) {
    chain_enter();
    if (post.host && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
        *(volatile unsigned long long *)post.host = (unsigned long long)(post.step + 1) << 32 | (unsigned)*post.far;
    if (out && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < sizeof(DevStatus) / sizeof(unsigned))
        ((volatile unsigned *)out)[threadIdx.x] = ((const unsigned *)st)[threadIdx.x];
    if ((int)blockIdx.y >= P.n) {
        __shared__ double red[3][4];
        double a[3] = {0.0, 0.0, 0.0};
        const int inner = g.nx * g.ny * g.nz, rows = gridDim.y - P.n;
        for (int q = ((blockIdx.y - P.n) * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; q < inner;
             q += rows * gridDim.x * blockDim.x) {
            const int k = q % g.nz, il = q / g.nz, l = il % g.ny, i = il / g.ny;
            const size_t n = g.node(i + 1, l + 1, k + 1);
            const double ex = (double)Ex[n], ey = (double)Ey[n], ez = (double)Ez[n];
            a[0] += ex * ex;
            a[1] += ey * ey;
            a[2] += ez * ez;
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            for (int o = 16; o > 0; o >>= 1) a[c] += __shfl_down_sync(0xffffffffu, a[c], o);
            if ((threadIdx.x & 31) == 0) red[c][threadIdx.x >> 5] = a[c];
        }
        __syncthreads();
        if (threadIdx.x < 3) {
            double sum = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) sum += red[threadIdx.x][w];
            atomicAdd(&hist[threadIdx.x], sum);
        }
        return;
    }
    const GhostPass q = P.p[blockIdx.y];
    const int A = q.e1 - q.s1 + 1, B = q.e2 - q.s2 + 1;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= A * B) return;
    const int la = q.s1 + idx / B, lb = q.s2 + idx % B;
    const Line L = line_of(g, q.dir, la, lb);
    T *E = (T *)q.E;
    size_t srcN = L.base + (size_t)q.N * L.stride, src1 = L.base + L.stride;
    if ((int)blockIdx.y >= P.nA) {
        // line coordinates (x along dir) as in line_of
        int cN[3], c1[3];
        const int d = q.dir, o1 = d == 0 ? 1 : 0, o2 = d == 2 ? 1 : 2;
        cN[o1] = c1[o1] = la;
        cN[o2] = c1[o2] = lb;
        cN[d] = q.N;
        c1[d] = 1;
        srcN = ghost_source(g, P, q.E, cN);
        src1 = ghost_source(g, P, q.E, c1);
    }
    E[L.base] = E[srcN];
    E[L.base + (size_t)(q.N + 1) * L.stride] = E[src1];
    // the step's end: the latest of the blocks (larger than any earlier step's)
    if (stamps && threadIdx.x == 0) atomicMax(&stamps[5], global_ns());
}


// ------------------------------------------------------- particle push --
// Interpolate3D, cell.h:1054-1153, on the staged field tile.  (bi,bl,bk) is
// the tile-local node of reference tile index (0,0,0) of the particle's cell,
// i.e. cell_local - 2; the reference tile index (i,l,k) must stay in 2..3 so
// that all 8 taps lie in the staged nodes [cell, cell+2].
__device__ __forceinline__ double interp_plain(const double *__restrict__ T, int SY, int SZ, int bi, int bl,
                                               int bk, int i, int l, int k, double sx, double sx1, double sy,
                                               double sy1, double sz, double sz1) {
    return trilinear(T + ((bi + i) * SY + (bl + l)) * SZ + (bk + k), SY * SZ, SZ, sx, sx1, sy, sy1, sz, sz1);
}

// flyDirection (cell.h:694-701): whether the particle leaves its cell
__device__ __forceinline__ bool moved_cell(const Grid &g, int i, int l, int k, double x, double y, double z, double x0,
                                           double y0, double z0) {
    const double hx = g.hx, hy = g.hy, hz = g.hz;
    int dxd = (((x > x0 + hx) && (x < x0 + 2 * hx)) || ((x < hx) && (i == g.nx - 1)))
                  ? 2 : (((x < x0) || ((x > g.lx - hx) && (i == 0))) ? 0 : 1);
    int dyd = (((y > y0 + hy) && (y < y0 + 2 * hy)) || ((y < hy) && (l == g.ny - 1)))
                  ? 2 : (((y < y0) || ((y > g.ly - hy) && (l == 0))) ? 0 : 1);
    int dzd = (((z > z0 + hz) && (z < z0 + 2 * hz)) || ((z < hz) && (k == g.nz - 1)))
                  ? 2 : (((z < z0) || ((z > g.lz - hz) && (k == 0))) ? 0 : 1);
    return dxd * 9 + dyd * 3 + dzd != 13;
}

// per-axis receivers of a departing particle: the cells of {c-1, c, c+1}
// (wrapped, getWrapCellNumber cell.h:806-853) whose isPointInCell (cell.h:717)
// holds -- the receivers of GPU_ArrangeFlights (kernels.cu:316-370)
__device__ __forceinline__ int receivers(double x, int c, int N, double h, int out[3]) {
    int n = 0;
    for (int d = -1; d <= 1; d++) {
        int j = c + d;
        if (j >= N) j -= N;
        else if (j < 0) j += N;
        double x0 = (double)j * h;
        if ((x0 <= x) && (x < x0 + h)) out[n++] = j;
    }
    return n;
}

// One bin's arrays: CTA-uniform pointers to its first slot, indexed by 32-bit
// offsets within the bin
struct BinP {
    int *cell;
    double *x, *y, *z, *px, *py, *pz;
    __device__ __forceinline__ BinP(const SpeciesView &S, int start)
        : cell(S.cell + start), x(S.x + start), y(S.y + start), z(S.z + start), px(S.px + start), py(S.py + start),
          pz(S.pz + start) {}
};

// 256 threads, two CTAs per SM: 16 warps per SM at up to 126 registers, no
// spills.  While 64-bit shared atomics were compare-and-swap loops, 512-thread
// CTAs at 64 registers (32 warps, ~240 B of spills) hid their round trips
// better (c2 push 208.7 ms against 246.5 at 256 threads); with the split
// 64-bit add (shared_add64) 256 threads win: 71.1 ms against 72.7 (384: 75.0,
// 448: 76.0).
//
// Bound: dependent FP64 operations (4 warps per scheduler at 128 registers;
// `wait` is the top stall, FP64 pipe 47 %, shared-memory pipe 65 %, DRAM 24 %).
// What shortened the chains, 256x64x64 cells, 201M particles: 17.1 ms; exact
// cheaper quotients, truncations and roundings and fused multiply-adds
// (pic_plain_math.cuh; 1648 -> 1367 instructions per 32 particles) 14.0 ms; the
// next particle by cp.async instead of a load at its use 12.4 ms (then 320
// threads 14.6, 384 15.4, 512 15.6).  A third of the instructions were integer
// ones; with the tile's dimensions fixed at compile time, one check of all taps,
// deposits without tests for zero and uniform bin pointers 1394 -> 1137
// instructions, and 128x64x64 cells, 50.3M particles, 3.22 -> 2.74 ms.
// Then the shared-memory pipe was 76 % busy, half of it adds to one address taking
// turns: a second tile current for the odd lanes and separate low and high words
// 2.74 -> 2.63 ms (2.75 -> 2.65 with bins no longer in cell order).
#ifndef PIC_PLAIN_THREADS
#define PIC_PLAIN_THREADS 256
#endif
#ifndef PIC_PLAIN_MIN_BLOCKS
#define PIC_PLAIN_MIN_BLOCKS 2
#endif
constexpr int kPlainThreads = PIC_PLAIN_THREADS;  // threads per CTA of k_push_plain
// per-warp queue of second zigzag segments: drained when it holds 16 or more
// (at most 32 per drain), so it never holds more than 15 + 32 entries
constexpr int kQPlain = 48;
static_assert(kPlainThreads % 32 == 0, "whole warps");
static_assert(kPlainThreads == kPushThreads, "the slices of a tile are cut in blocks of kPushThreads particles");
#ifdef PIC_PLAIN_MIN_BLOCKS
#define PIC_PLAIN_BOUNDS __launch_bounds__(kPlainThreads, PIC_PLAIN_MIN_BLOCKS)
#else
#define PIC_PLAIN_BOUNDS __launch_bounds__(kPlainThreads)
#endif
// SPLIT: P.slices CTAs share a tile (see StepParams::slices)
// TX, TY, TZ: the tile's cells per axis when fixed at compile time (the offsets of
// taps and deposits become immediates), 0 to take them from the grid
template <bool LO32, bool SPLIT, int TX, int TY, int TZ>
__global__ void PIC_PLAIN_BOUNDS k_push_plain(const __grid_constant__ StepParams P) {
    chain_enter();
    stamp_entry(P.stamps, 2);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int sNHoles, sNFront, sNMove;
    __shared__ double sRed[kPlainThreads / 32];
    __shared__ double sQ, sInvQ, sLoScale;
    __shared__ int sQn[kPlainThreads / 32];  // entries in each warp's segment queue
    const Grid &g = P.g;
    const int t = SPLIT ? blockIdx.x / P.slices : blockIdx.x;
    SliceRange slice = {0, 0};
    if (SPLIT) slice = slice_blocks(P, t, blockIdx.x - t * P.slices, kPlainThreads);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tk = t % g.ntz, tl = (t / g.ntz) % g.nty, ti = t / (g.ntz * g.nty);
    const int tx = TX ? TX : g.tx, ty = TY ? TY : g.ty, tz = TZ ? TZ : g.tz;
    const int i0 = ti * tx, l0 = tl * ty, k0 = tk * tz;
    const int SX = tx + 2, SY = ty + 2, SZ = tz + 2;
    const int nn = SX * SY * SZ;
    double *sF = (double *)smem_raw;  // Ex Ey Ez Hx Hy Hz
    // fixed-point tile J (pqr_plain): 3 nn low and 3 nn high words, then the
    // remainder's (3 nn low, 3 nn high words, or 3 nn int32)
    unsigned long long *sJ = (unsigned long long *)(sF + 6 * nn);
    // (lo32 with room for it: two currents, even lanes in one, odd lanes in the other)
    const int jstride = (9 * nn + 1) / 2, jcopies = LO32 ? P.jcopies : 1;
    const int jwords = jcopies == 2 ? 2 * jstride : 6 * nn;
    unsigned *myJ = (unsigned *)(sJ + (LO32 ? (lane & (jcopies - 1)) * jstride : 0));
    int *sHoles = (int *)(sJ + jwords);
    int *sFront = sHoles + kHoleMax;
    // this warp's segment queue: x2 and xn (6 x kQPlain doubles), and the
    // start cell (tile-local) with the segment's centre-cell bits
    double *qd = (double *)(sHoles + 2 * kHoleMax) + warp * 6 * kQPlain;
    int *qc = (int *)((double *)(sHoles + 2 * kHoleMax) + (kPlainThreads / 32) * 6 * kQPlain) + warp * kQPlain;
    // this thread's next particle (P.prefetch): 6 values 32 lanes apart, then the cell
    double *sNext = (double *)(sHoles + 2 * kHoleMax + (kPlainThreads / 32) * 13 * kQPlain) + warp * (6 * 32 + 16) + lane;
    int *sNextCell = (int *)(sNext - lane + 6 * 32) + lane;
    const bool pre = P.prefetch != 0;
    if (threadIdx.x == 0) {
        double bound = 0.0, one = 0.0;
        long long ntile = 0;
        for (int s = 0, first = 0; s < P.nsp; s++) {
            const int count = P.sp[s].tile_count[t];
            int jbeg = 0, jend = count;
            if (SPLIT) slice_range(slice, first, count, kPlainThreads, jbeg, jend);
            first += (count + kPlainThreads - 1) / kPlainThreads;
            bound += 2.5 * fabs(P.sp[s].m) * (double)(jend - jbeg);
            if (jend > jbeg) one = fmax(one, 1.0834 * fabs(P.sp[s].m));
            ntile += jend - jbeg;
        }
        // a quantum that holds every sum of the tile below 2^62 and every single
        // contribution below 2^51 (fx_put2).  The second alone decides in tiles of
        // fewer than about 800 particles: with the remainder word a contribution is
        // rounded at 2^-71 |m| or below, where the rounding of its end point x1
        // (2^-54 x1 / tau, and x1 > tau 2^-17 but for a few particles at a box face)
        // is 2^-71 |m| at least and mostly 2^-54 |m|
        int e2, e1;
        frexp(bound, &e2);  // bound < 2^e2
        frexp(one, &e1);
        const int eq = max(e2 - 62, e1 - 51);
        sQ = ldexp(1.0, eq);
        sInvQ = ldexp(1.0, -eq);
        sLoScale = LO32 ? ldexp(1.0, fx_lo32_bits(ntile)) : 1099511627776.0;  // 2^L or 2^40
    }

    // stage E^n and H^{n+1/2} of nodes [i0, i0+tx+2) x [l0, ..) x [k0, ..)
    // (GPU_SetFieldsToCells, kernels.cu:32-49, for all cells of the tile at once)
    const double *const *E = (const double *const *)P.E;
    const double *const *H = (const double *const *)P.H;
    for (int idx = threadIdx.x; idx < nn; idx += blockDim.x) {
        int c = idx % SZ, b = (idx / SZ) % SY, a = idx / (SZ * SY);
        int gi = i0 + a, gl = l0 + b, gk = k0 + c;
        bool in = gi < g.NX && gl < g.NY && gk < g.NZ;
        size_t n = in ? g.node(gi, gl, gk) : 0;
        sF[idx] = in ? E[0][n] : 0.0;
        sF[nn + idx] = in ? E[1][n] : 0.0;
        sF[2 * nn + idx] = in ? E[2][n] : 0.0;
        sF[3 * nn + idx] = in ? H[0][n] : 0.0;
        sF[4 * nn + idx] = in ? H[1][n] : 0.0;
        sF[5 * nn + idx] = in ? H[2][n] : 0.0;
    }
    for (int idx = threadIdx.x; idx < jwords; idx += blockDim.x) sJ[idx] = 0ull;
    __syncthreads();

    const double hx = g.hx, hy = g.hy, hz = g.hz, tau = g.tau;
    const double rhx = 1.0 / hx, rhy = 1.0 / hy, rhz = 1.0 / hz;
    const double lo_scale = sLoScale;
    unsigned bad = 0;
    double kin = 0.0;
    unsigned long long moved = 0, dropped = 0, dup = 0;
    OutPlain *outbox = (OutPlain *)P.outbox;

    for (int s = 0, first = 0; s < P.nsp; s++) {
        const SpeciesView &S = P.sp[s];
        const int start = S.tile_start[t];
        // the particles [jbeg, count) of the bin are this CTA's
        int count = S.tile_count[t], jbeg = 0;
        if (SPLIT) {
            const int all = count;
            slice_range(slice, first, all, kPlainThreads, jbeg, count);
            first += (all + kPlainThreads - 1) / kPlainThreads;
            if (jbeg == count) continue;
        }
        const BinP bin(S, start);
        const double M = S.m / S.q_m, tau1 = S.q_m * tau * 0.5;
        // the charge weight over pqr's tau*h*h divisors, in quanta (a power of two)
        const double mq = S.m * sInvQ;
        const double rc[3] = {mq / (tau * hy * hz), mq / (tau * hx * hz), mq / (tau * hx * hy)};
        if (!SPLIT) {
            if (threadIdx.x == 0) { sNHoles = 0; sNFront = 0; sNMove = 0; }
            __syncthreads();
        }
        int qn = 0;  // entries in this warp's segment queue (warp-uniform)
        if (lane == 0) sQn[warp] = 0;
        // the particle of the next iteration comes asynchronously (cp.async) into
        // shared memory while the current one is processed: registers are full,
        // and the loads were a fifth of the kernel's stalls
        auto prefetch = [&](int jn) {
            if (jn < count) {
                const unsigned q = (unsigned)jn;
                cp_async<4>(sNextCell, bin.cell + q);
                cp_async<8>(sNext, bin.x + q);
                cp_async<8>(sNext + 32, bin.y + q);
                cp_async<8>(sNext + 64, bin.z + q);
                cp_async<8>(sNext + 96, bin.px + q);
                cp_async<8>(sNext + 128, bin.py + q);
                cp_async<8>(sNext + 160, bin.pz + q);
            }
        };
        if (pre) prefetch(jbeg + threadIdx.x);
        __syncwarp();
        // Whole warps iterate together (the queue is drained by whole warps),
        // and past the last particle until the queue is empty.
        for (int jw = jbeg + threadIdx.x - lane;; jw += blockDim.x) {
            const bool tail = jw >= count;
            if (tail && qn == 0) break;
            const int j = jw + lane;
            const unsigned slot = (unsigned)j;  // within the bin
            // cell < 0: past the bin's end, or a dead slot left by an overflowed compaction
            int cell = -1;
            double x = 0.0, y = 0.0, z = 0.0, p[3] = {0.0, 0.0, 0.0};
            if (pre) {
                cp_async_wait_all();
                if (j < count) {
                    cell = *sNextCell;
                    x = sNext[0]; y = sNext[32]; z = sNext[64];
                    p[0] = sNext[96]; p[1] = sNext[128]; p[2] = sNext[160];
                }
                __syncwarp();  // the reads come before the next copies into the same place
                prefetch(j + (int)blockDim.x);
            } else if (j < count) {
                cell = bin.cell[slot];
                x = bin.x[slot]; y = bin.y[slot]; z = bin.z[slot];
                p[0] = bin.px[slot]; p[1] = bin.py[slot]; p[2] = bin.pz[slot];
            }
            int i = 0, l = 0, k = 0;
            if (cell >= 0) g.cell_ijk(cell, i, l, k);
            const int bi = i - i0 - 2, bl = l - l0 - 2, bk = k - k0 - 2;
            const bool in_tile = (unsigned)(bi + 2) < (unsigned)tx && (unsigned)(bl + 2) < (unsigned)ty && (unsigned)(bk + 2) < (unsigned)tz;
            if (cell >= 0 && !in_tile) bad |= ST_BADCELL;  // a bin entry outside its tile: never index the tile with it
            if (cell >= 0 && in_tile) {
                // Cell ctor, cell.h:731-737
                const double x0 = (double)i * hx, y0 = (double)l * hy, z0 = (double)k * hz;
                AxisTaps X, Y, Z;
                axis_taps(x, x0, hx, rhx, X);
                axis_taps(y, y0, hy, rhy, Y);
                axis_taps(z, z0, hz, rhz, Z);

                // ---- Cell::GetField, cell.h:1257-1290
                double F[6];
                // every tap in 2..3; each of the six indices is some component's
                const bool taps = (((X.tn ^ 2) | (X.tc ^ 2) | (Y.tn ^ 2) | (Y.tc ^ 2) | (Z.tn ^ 2) | (Z.tc ^ 2)) & ~1) == 0;
                const bool negative = x < 0 || y < 0 || z < 0;
                if (!taps && !negative) bad |= ST_STENCIL;
                if (!taps || negative) {
#pragma unroll
                    for (int c = 0; c < 6; c++) F[c] = 0.0;
                } else {
                    const double s1 = X.wn, s2 = X.wc, s3 = Y.wn, s4 = Y.wc, s5 = Z.wn, s6 = Z.wc;
                    const double s11 = 1. - s1, s21 = 1. - s2, s31 = 1. - s3, s41 = 1. - s4, s51 = 1. - s5, s61 = 1. - s6;
                    F[0] = interp_plain(sF, SY, SZ, bi, bl, bk, X.tn, Y.tc, Z.tc, s1, s11, s4, s41, s6, s61);
                    F[1] = interp_plain(sF + nn, SY, SZ, bi, bl, bk, X.tc, Y.tn, Z.tc, s2, s21, s3, s31, s6, s61);
                    F[2] = interp_plain(sF + 2 * nn, SY, SZ, bi, bl, bk, X.tc, Y.tc, Z.tn, s2, s21, s4, s41, s5, s51);
                    F[3] = interp_plain(sF + 3 * nn, SY, SZ, bi, bl, bk, X.tc, Y.tn, Z.tn, s2, s21, s3, s31, s5, s51);
                    F[4] = interp_plain(sF + 4 * nn, SY, SZ, bi, bl, bk, X.tn, Y.tc, Z.tn, s1, s11, s4, s41, s5, s51);
                    F[5] = interp_plain(sF + 5 * nn, SY, SZ, bi, bl, bk, X.tn, Y.tn, Z.tc, s1, s11, s3, s31, s6, s61);
                }
                // ---- Particle::Move, particle.h:65-202
                double p2;
                const double ig = boris_move(tau1, F, p, p2);
                const double pu = p[0], pv = p[1], pw = p[2];
                double xn[3] = {x + tau * (ig * pu), y + tau * (ig * pv), z + tau * (ig * pw)};
                if (!isfinite(p2) && !(isfinite(pu) && isfinite(pv) && isfinite(pw))) bad |= ST_NAN;
                // gamma - 1 = p^2 / (gamma + 1) without cancellation
                kin += M * (p2 * ig / (1.0 + ig));

                // ---- Cell::CurrentToMesh, cell.h:1306-1422
                {
                    double xo[3] = {x, y, z}, x2[3], sr;
                    const double h3[3] = {hx, hy, hz}, r3[3] = {rhx, rhy, rhz}, o3[3] = {x0, y0, z0};
                    const int i1[3] = {X.i1, Y.i1, Z.i1};
                    int i2[3];
                    bool exact = true;
#pragma unroll
                    for (int d = 0; d < 3; d++)  // getCellNumberCenterCurrent, cell.h:577-578
                        i2[d] = trunc_checked((div_by(xn[d] - o3[d], h3[d], r3[d]) + 1.5) + 1, exact);
                    if (!exact) { bad |= ST_STENCIL; i2[0] = 0; }
                    const int m = relay_point(xo, xn, o3, h3, i1, i2, x2, sr);
                    // the first segment here: xo -> xn, or xo -> x2 when the step
                    // crosses a cell-centre plane.  The second, x2 -> xn, goes to
                    // the warp's queue and is deposited with the warp's other
                    // crossings, 16 to 32 at a time, so that a few crossing lanes do
                    // not make the whole warp run the deposit twice.
                    const bool cross = m >= 1 && m <= 7;
                    double sb[3];
#pragma unroll
                    for (int d = 0; d < 3; d++) sb[d] = cross ? x2[d] : xn[d];
                    pqr_plain<LO32>(myJ, lo_scale, nn, SY * SZ, SZ, bi, bl, bk, i1, xo, sb, hx, hy, hz, rc, x0, y0, z0, bad);
                    if (cross) {
                        if (i2[0] >= 2 && i2[0] <= 3 && i2[1] >= 2 && i2[1] <= 3 && i2[2] >= 2 && i2[2] <= 3) {
                            const int e = atomicAdd(&sQn[warp], 1);  // < 15 + 32: drained at 16
#pragma unroll
                            for (int d = 0; d < 3; d++) {
                                qd[d * kQPlain + e] = x2[d];
                                qd[(3 + d) * kQPlain + e] = xn[d];
                            }
                            qc[e] = ((((bi + 2) * ty + (bl + 2)) * tz + (bk + 2)) << 3) | (i2[0] - 2) |
                                    ((i2[1] - 2) << 1) | ((i2[2] - 2) << 2);
                        } else {
                            bad |= ST_STENCIL;  // pqr's own stencil check
                        }
                    }
                }
                x = reflect_plain(xn[0], g.lx);
                y = reflect_plain(xn[1], g.ly);
                z = reflect_plain(xn[2], g.lz);

                // ---- flyDirection (cell.h:694-701) and the receivers of K8.  A
                // particle within [x0, x0 + h] on every axis stays: the wrap
                // cases (x < h in the last cell, x > L - h in the first) lie at
                // least a cell away from that interval.
                const bool inside = x >= x0 && x <= x0 + hx && y >= y0 && y <= y0 + hy && z >= z0 && z <= z0 + hz;
                int newcell = cell;
                bool leave = false;
                int rx[3], ry[3], rz[3], nrx = 1, nry = 1, nrz = 1;
                if (!inside && moved_cell(g, i, l, k, x, y, z, x0, y0, z0)) {
                    nrx = receivers(x, i, g.nx, hx, rx);
                    nry = receivers(y, l, g.ny, hy, ry);
                    nrz = receivers(z, k, g.nz, hz, rz);
                    int ncopy = nrx * nry * nrz;
                    if (ncopy == 1 && g.tile_of_cell(rx[0], ry[0], rz[0]) == t) {
                        newcell = g.cell_of(rx[0], ry[0], rz[0]);
                    } else {
                        leave = true;
                        if (ncopy == 0) dropped++;
                        if (ncopy > 1) dup++;
                        if (ncopy > 0) {
                            unsigned e = atomicAdd(&P.st->out_count, (unsigned)ncopy);
                            if (e + ncopy > P.out_cap) {
                                bad |= ST_OUTBOX;
                            } else {
                                for (int a = 0; a < nrx; a++)
                                    for (int b = 0; b < nry; b++)
                                        for (int c = 0; c < nrz; c++) {
                                            OutPlain o;
                                            o.x = x; o.y = y; o.z = z; o.px = pu; o.py = pv; o.pz = pw;
                                            o.cell = g.cell_of(rx[a], ry[b], rz[c]);
                                            o.species = s;
                                            outbox[e++] = o;
                                        }
                                moved++;
                            }
                        }
                    }
                }
                if (leave) {
                    bin.cell[slot] = -1;
                    const size_t e = (size_t)s * g.ntiles + t;
                    const unsigned hpos = SPLIT ? atomicAdd(&P.hole_count[e], 1u) : (unsigned)atomicAdd(&sNHoles, 1);
                    if (!list_hole(S, t, SPLIT ? P.holes + e * kHoleMax : sHoles, hpos, j)) bad |= ST_HOLES;
                } else {
                    bin.cell[slot] = newcell;
                    bin.x[slot] = x; bin.y[slot] = y; bin.z[slot] = z;
                    bin.px[slot] = pu; bin.py[slot] = pv; bin.pz[slot] = pw;
                }
            }  // particle
            // ---- the warp's queued second segments, one per lane
            __syncwarp();
            qn = sQn[warp];
            if (qn >= (tail ? 1 : 16)) {
                const int d = qn < 32 ? qn : 32;
                if (lane < d) {
                    const int e = qn - d + lane;
                    const int code = qc[e], lc = code >> 3;
                    const int a = lc / (ty * tz), b = (lc / tz) % ty, c = lc % tz;
                    const int qi = i0 + a, ql = l0 + b, qk = k0 + c;
                    const int iv[3] = {2 + (code & 1), 2 + ((code >> 1) & 1), 2 + ((code >> 2) & 1)};
                    double sa[3], sb[3];
#pragma unroll
                    for (int dd = 0; dd < 3; dd++) {
                        sa[dd] = qd[dd * kQPlain + e];
                        sb[dd] = qd[(3 + dd) * kQPlain + e];
                    }
                    pqr_plain<LO32>(myJ, lo_scale, nn, SY * SZ, SZ, a - 2, b - 2, c - 2, iv, sa, sb, hx, hy, hz, rc,
                                    (double)qi * hx, (double)ql * hy, (double)qk * hz, bad);
                }
                qn -= d;
                __syncwarp();
                if (lane == 0) sQn[warp] = qn;
            }
            __syncwarp();
        }
        if (SPLIT) continue;  // the tile's last CTA compacts its bins
        __syncthreads();
        // ---- compaction of the tile bin (replaces GPU_MakeDepartureLists_rm, kernels.cu:219-242)
        const int L = sNHoles;
        const HoleList holes = hole_list(S, t, sHoles, false), fronts = hole_list(S, t, sFront, true);
        if (L > 0 && L <= holes.limit()) {
            const int newcount = count - L;
            for (int r = threadIdx.x; r < L; r += blockDim.x) {
                int h = *holes.at(r);
                if (h < newcount) *fronts.at(atomicAdd(&sNFront, 1)) = h;
            }
            __syncthreads();
            for (int r = threadIdx.x; r < L; r += blockDim.x) {
                int src = start + newcount + r;
                if (S.cell[src] >= 0) {
                    int m = atomicAdd(&sNMove, 1);
                    if (m >= sNFront) { bad |= ST_BADCELL; continue; }
                    int dst = start + *fronts.at(m);
                    S.cell[dst] = S.cell[src];
                    S.x[dst] = S.x[src]; S.y[dst] = S.y[src]; S.z[dst] = S.z[src];
                    S.px[dst] = S.px[src]; S.py[dst] = S.py[src]; S.pz[dst] = S.pz[src];
                }
            }
            if (threadIdx.x == 0) S.tile_count[t] = newcount;
        }
        __syncthreads();
    }

    if (SPLIT) __syncthreads();
    // ---- tile J -> global J (GPU_WriteAllCurrents, kernels.cu:83-112)
    for (int idx = threadIdx.x; idx < 3 * nn; idx += blockDim.x) {
        long long ih, il;
        fx_get<LO32>((const unsigned *)sJ + idx, 3 * nn, ih, il);
        if (jcopies == 2) {
            long long ih2, il2;
            fx_get<LO32>((const unsigned *)(sJ + jstride) + idx, 3 * nn, ih2, il2);
            ih += ih2;
            il += il2;
        }
        if (ih != 0 || il != 0) {
            int comp = idx / nn, r = idx % nn;
            int c = r % SZ, b = (r / SZ) % SY, a = r / (SZ * SY);
            if (i0 + a < g.NX && l0 + b < g.NY && k0 + c < g.NZ)
                atomicAdd(&P.J[comp][g.node(i0 + a, l0 + b, k0 + c)],
                          ((double)ih + (double)il / lo_scale) * sQ);  // exact scale: a power of two
        }
    }
    // ---- kinetic energy and counters
    for (int o = 16; o > 0; o >>= 1) kin += __shfl_down_sync(0xffffffffu, kin, o);
    if ((threadIdx.x & 31) == 0) sRed[threadIdx.x >> 5] = kin;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) tot += sRed[w];
        atomicAdd(&P.st->kinetic, tot);
    }
    if (SPLIT && last_of_tile(P, t, &sNHoles)) {
        compact_tile(P, t, sHoles, bad, [](const SpeciesView &S, int dst, int src) {
            S.cell[dst] = __ldcg(&S.cell[src]);
            S.x[dst] = __ldcg(&S.x[src]); S.y[dst] = __ldcg(&S.y[src]); S.z[dst] = __ldcg(&S.z[src]);
            S.px[dst] = __ldcg(&S.px[src]); S.py[dst] = __ldcg(&S.py[src]); S.pz[dst] = __ldcg(&S.pz[src]);
        });
    }
    if (bad) atomicOr(&P.st->flags, bad);
    if (moved) atomicAdd(&P.st->moved, moved);
    if (dropped) atomicAdd(&P.st->dropped, dropped);
    if (dup) atomicAdd(&P.st->duplicated, dup);
}

}  // namespace

// ------------------------------------------------------------ launchers --
constexpr int kPlaneThreads = 256;
static inline dim3 plane_grid(const Grid &g) {
    return dim3((g.NY * g.NZ + kPlaneThreads - 1) / kPlaneThreads, g.NX);
}

void yee_b_half_plain(const Grid &g, double *const F[12], cudaStream_t s, unsigned long long *stamps) {
    // getMagneticFieldTimeMeshFactors, gpu_plasma.h:512-522
    double cx = g.tau / (g.hx), cy = g.tau / (g.hy), cz = g.tau / g.hz;
    launch_chained(k_b_half_plain, plane_grid(g), dim3(kPlaneThreads), s, g, F[PIC_EX], F[PIC_EY], F[PIC_EZ], F[PIC_HX],
                   F[PIC_HY], F[PIC_HZ], F[PIC_QX], F[PIC_QY], F[PIC_QZ], cx, cy, cz, stamps);
}

void yee_b_complete_plain(const Grid &g, double *const F[12], cudaStream_t s) {
    launch_chained(k_b_complete_plain, plane_grid(g), dim3(kPlaneThreads), s, g, F[PIC_HX], F[PIC_HY], F[PIC_HZ],
                   F[PIC_QX], F[PIC_QY], F[PIC_QZ]);
}

void yee_e_update_plain(const Grid &g, double *const F[12], cudaStream_t s) {
    double cx = g.tau / (g.hx), cy = g.tau / (g.hy), cz = g.tau / g.hz;
    launch_chained(k_e_update_plain, plane_grid(g), dim3(kPlaneThreads), s, g, F[PIC_EX], F[PIC_EY], F[PIC_EZ],
                   F[PIC_HX], F[PIC_HY], F[PIC_HZ], F[PIC_JX], F[PIC_JY], F[PIC_JZ], cx, cy, cz, g.tau);
}


void j_fold(const Grid &g, double *Jx, double *Jy, double *Jz, cudaStream_t s) {
    launch_chained(k_j_fold, dim3((fold_orbits(g) + 127) / 128), dim3(128), s, g, Jx, Jy, Jz);
}

void fold_b_plain(const Grid &g, double *const F[12], cudaStream_t s, unsigned long long *stamps) {
    const int folds = (fold_orbits(g) + kPlaneThreads - 1) / kPlaneThreads;
    const dim3 plane = plane_grid(g);
    launch_chained(k_fold_b_plain, dim3(folds + plane.x * plane.y), dim3(kPlaneThreads), s, g, folds, (int)plane.x,
                   F[PIC_JX], F[PIC_JY], F[PIC_JZ], F[PIC_HX], F[PIC_HY], F[PIC_HZ], F[PIC_QX], F[PIC_QY], F[PIC_QZ], stamps);
}

void flat_begin_plain(const Grid &g, const double *const E[3], const double *const H[3], double *Ha, double *J,
                      double *keepE, cudaStream_t s) {
    const double cx = g.tau / g.hx, cy = g.tau / g.hy, cz = g.tau / g.hz;
    launch_chained(k_flat_begin_plain, dim3((g.NY * g.pz + kPlaneThreads - 1) / kPlaneThreads, g.NX), dim3(kPlaneThreads),
                   s, g, E[0], E[1], E[2], H[0], H[1], H[2], Ha, J, keepE, cx, cy, cz);
}

void fold_b_twice_plain(const Grid &g, double *const F[12], cudaStream_t s) {
    const double cx = g.tau / g.hx, cy = g.tau / g.hy, cz = g.tau / g.hz;
    const int folds = (fold_orbits(g) + kPlaneThreads - 1) / kPlaneThreads;
    const dim3 plane = plane_grid(g);
    launch_chained(k_fold_b_twice_plain, dim3(folds + plane.x * plane.y), dim3(kPlaneThreads), s, g, folds, (int)plane.x,
                   F[PIC_JX], F[PIC_JY], F[PIC_JZ], F[PIC_EX], F[PIC_EY], F[PIC_EZ], F[PIC_HX], F[PIC_HY], F[PIC_HZ],
                   F[PIC_QX], F[PIC_QY], F[PIC_QZ], cx, cy, cz);
}

// ElectricFieldComponentEvaluatePeriodic for Ex, Ey, Ez (gpu_plasma.h:432-452,
// arguments gpu_plasma.h:486-505).  Reference mode skips the y pass of Ex and
// Ez; periodic mode performs it.  Round A holds the first pass of each
// component, round B the second; both run in one launch (GhostPasses).
template <typename T>
static void e_ghosts_t(const Grid &g, T *Ex, T *Ey, T *Ez, int periodic, cudaStream_t s, const DevStatus *st,
                       DevStatus *out, double *hist, unsigned long long *stamps, FarPost post) {
    int Nx = g.nx, Ny = g.ny, Nz = g.nz;
    GhostPasses P{};
    int maxn = 0;
    auto add = [&](T *E, int dir, int s1, int e1, int s2, int e2, int N) {
        P.p[P.n++] = GhostPass{(void *)E, dir, s1, e1, s2, e2, N};
        int n = (e1 - s1 + 1) * (e2 - s2 + 1);
        if (n > maxn) maxn = n;
    };
    // round A: the first pass of each component
    if (periodic) add(Ex, 1, 0, Nx, 1, Nz, Ny);
    add(Ey, 0, 0, Ny, 1, Nz, Nx);
    add(Ez, 0, 1, Ny, 0, Nz, Nx);
    P.nA = P.n;
    // round B: the second (Ey's z pass reads the x ghosts of round A)
    add(Ex, 2, 0, Nx, 0, Ny + 1, Nz);
    add(Ey, 2, 0, Nx + 1, 0, Ny, Nz);
    if (periodic) add(Ez, 1, 0, Nx + 1, 0, Nz, Ny);
    launch_chained(k_e_ghosts<T>, dim3((maxn + 127) / 128, P.n + (hist ? kHistRows : 0)), dim3(128), s, g, P, st, out, Ex, Ey,
                   Ez, hist, stamps, post);
}
void e_ghosts_plain(const Grid &g, double *Ex, double *Ey, double *Ez, int periodic, cudaStream_t s,
                    const DevStatus *st, DevStatus *out, double *hist, unsigned long long *stamps, FarPost post) {
    e_ghosts_t<double>(g, Ex, Ey, Ez, periodic, s, st, out, hist, stamps, post);
}
void e_ghosts_mixed(const Grid &g, float *Ex, float *Ey, float *Ez, int periodic, cudaStream_t s, const DevStatus *st,
                    DevStatus *out, double *hist, unsigned long long *stamps, FarPost post) {
    e_ghosts_t<float>(g, Ex, Ey, Ez, periodic, s, st, out, hist, stamps, post);
}

// shared memory of the next particle of every thread
constexpr size_t kPlainPrefetch = (size_t)(kPlainThreads / 32) * (6 * 32 + 16) * sizeof(double);

size_t push_smem_plain(const Grid &g) {
    size_t nn = (size_t)(g.tx + 2) * (g.ty + 2) * (g.tz + 2);
    return 6 * nn * sizeof(double) + 6 * nn * sizeof(unsigned long long) + 2 * kHoleMax * sizeof(int) +
           (size_t)(kPlainThreads / 32) * kQPlain * (6 * sizeof(double) + sizeof(int));
}

using PushPlainFn = void (*)(StepParams);
template <bool LO32, bool SPLIT>
static PushPlainFn push_plain_fn(const Grid &g) {
    if (g.tx == 8 && g.ty == 4 && g.tz == 8) return k_push_plain<LO32, SPLIT, 8, 4, 8>;
    if (g.tx == 8 && g.ty == 4 && g.tz == 4) return k_push_plain<LO32, SPLIT, 8, 4, 4>;
    return k_push_plain<LO32, SPLIT, 0, 0, 0>;
}
// the instantiation for a grid's tile: fixed dimensions for the automatic tiles, else runtime
static PushPlainFn push_plain_fn(const Grid &g, bool lo32, bool split) {
    if (lo32) return split ? push_plain_fn<true, true>(g) : push_plain_fn<true, false>(g);
    return split ? push_plain_fn<false, true>(g) : push_plain_fn<false, false>(g);
}

cudaError_t launch_push_plain(const StepParams &in, bool lo32, cudaStream_t s) {
    StepParams p = in;
    size_t smem = push_smem_plain(p.g);
    // prefetch through shared memory where it leaves as many CTAs on an SM
    int dev = 0, per_sm = 0, per_block = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&per_block, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    auto fit = [&](size_t b) { return std::min<size_t>(PIC_PLAIN_MIN_BLOCKS, (size_t)per_sm / (b + 2048)); };
    p.prefetch = smem + kPlainPrefetch <= (size_t)per_block && fit(smem + kPlainPrefetch) >= fit(smem);
    if (p.prefetch) smem += kPlainPrefetch;
    // a second tile current likewise
    const size_t nn = (size_t)(p.g.tx + 2) * (p.g.ty + 2) * (p.g.tz + 2);
    const size_t second = (2 * ((9 * nn + 1) / 2) - 6 * nn) * sizeof(unsigned long long);
    p.jcopies = lo32 && smem + second <= (size_t)per_block && fit(smem + second) >= fit(smem) ? 2 : 1;
    if (p.jcopies == 2) smem += second;
    const bool split = p.slices > 1;
    const PushPlainFn kern = push_plain_fn(p.g, lo32, split);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_chained_smem(kern, dim3(p.g.ntiles * (split ? p.slices : 1)), dim3(kPlainThreads), smem, s, p);
}

}  // namespace pic
