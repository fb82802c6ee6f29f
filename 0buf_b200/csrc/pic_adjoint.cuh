// State of the differentiable run (pic_forward / pic_backward), shared by the
// plain-form (pic_adjoint.cu) and FP32-form (pic_adjoint_mixed.cu) units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <vector>
#include "pic0buf.h"
#include "pic_internal.cuh"

struct pic_handle;

namespace pic {

struct AdjStatus {
    unsigned flags;                // ST_STENCIL / ST_NAN seen in the run
    unsigned pad;
    unsigned long long ambiguous;  // cell changes with zero or several receiving cells (resolved, counted)
};

// a run of consecutive particles of one species in the fixed order, all from
// one tile at the start: the work of one CTA of the particle kernels
constexpr int kAdjChunk = 2048;  // particles at most
struct AdjChunk {
    int64_t first;  // index within the species
    int count, species;
};

// the device buffers of the run, by use
enum AdjSlot {
    kAdjBranch, kAdjCur, kAdjCkp, kAdjCkf, kAdjHist, kAdjSt, kAdjRed, kAdjChunks, kAdjSegp, kAdjSegf, kAdjSubp, kAdjSubf,
    kAdjLamp, kAdjLamf, kAdjRf, kAdjHa, kAdjSlots
};

// Buffers live until pic_adjoint_free / pic_destroy; the next pic_forward takes
// over those of about its own size (an optimiser's evaluations then allocate
// nothing) and frees the others.  Buffers that no run uses at the moment are
// given back when a device allocation of the handle fails (adj_reclaim).
// A "particle state" is the whole population in the fixed order of the run:
// per species the packed cells then 6 value arrays (plain: FP64 global
// positions and momenta; mixed: FP32 in-cell offsets and momenta).
struct AdjState {
    struct Buf {
        void *p;
        size_t cap;
        int used;  // by the current run
    } pool[kAdjSlots];
    int mixed;
    size_t elem;       // bytes per particle value (8 plain, 4 mixed)
    int nsp;
    int64_t n[kMaxSpecies];
    int steps, K, nseg;
    int K2;            // sub-checkpoint interval inside a segment (== K: one level)
    size_t pbytes;     // one particle state
    char *cur;         // the forward's running state
    char *ckp;         // nseg particle checkpoints
    char *ckf;         // nseg x (E, H): 6 field arrays each, in the form's field type
    char *segp;        // K2+1 particle states of the (sub-)segment being reversed
    char *segf;        // K2 x (E, H after the half step) of that (sub-)segment's steps
    char *subp;        // two levels: ceil(K/K2) sub-checkpoint states of the segment being reversed
    char *subf;        // two levels: their (E, H)
    char *lamp;        // per species lambda_x (3) and lambda_p (3), form's element type
    size_t lamp_bytes;
    double *lamf;      // FP64 lambda_E, lambda_H, lambda_J, lambda_Q (12 arrays)
    char *rf;          // field set of the recompute (form's layout: 12 arrays)
    char *ha;          // B after the half step of a step whose fields are not kept (3 arrays)
    AdjChunk *chunks;  // nchunks of them, device
    int nchunks;
    double *hist;      // steps x 3: sum over nodes 1..N of E_c^2 after each step
    // frozen branches (plain form): mode 1 records every step's discrete
    // choices into branch (steps x particles codes), mode 2 replays those of
    // branch_src; step_branch / step_bmode are what the next flat push uses
    unsigned long long *branch;
    const unsigned long long *branch_src;
    int branch_mode;
    unsigned long long *step_branch;
    int step_bmode;
    double *red;       // reduction scratch
    AdjStatus *st;
    std::vector<double> hhist;  // host copy of hist x cell volume
    cudaEvent_t e0, e1;
    float t_fwd, t_bwd;
    unsigned long long ambiguous;
    int have_forward;
};

inline size_t align256(size_t b) { return (b + 255) / 256 * 256; }

// ---- a chunk's window: the box of cells whose nodes a CTA keeps in shared memory
struct AdjWindow {
    int i0, l0, k0, cx, cy, cz;  // first cell and cells per axis
    int SY, SZ, nn;              // node strides and nodes: (cx+2)(cy+2)(cz+2)
    __device__ __forceinline__ bool holds(int i, int l, int k) const {
        return (unsigned)(i - i0) < (unsigned)cx && (unsigned)(l - l0) < (unsigned)cy && (unsigned)(k - k0) < (unsigned)cz;
    }
    // window-local node of a cell (its lower corner)
    __device__ __forceinline__ int node(int i, int l, int k) const { return ((i - i0) * SY + (l - l0)) * SZ + (k - k0); }
};
// The window of `count` particles' cells with at most `cap` nodes: their
// bounding box where that fits.  Otherwise (particles that wandered off, or a
// chunk that lies on both sides of a periodic boundary) a box around their mean
// position, taken periodically, cut at the grid's edge and shrunk on its longest
// axis until it fits; the particles outside it use global memory.  Every thread
// of the CTA calls it; red holds 15 ints per warp.
__device__ __forceinline__ AdjWindow chunk_window(const Grid &g, const int *__restrict__ cell, int count, int cap,
                                                  int *red, AdjWindow *out) {
    const unsigned FULL = 0xffffffffu;
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n3[3] = {g.nx, g.ny, g.nz};
    int at[3];  // the middle particle's cell: the others' periodic distances are taken from it
    g.cell_ijk(cell[count / 2], at[0], at[1], at[2]);
    int lo[3], hi[3], dlo[3], dhi[3], sum[3];
#pragma unroll
    for (int d = 0; d < 3; d++) { lo[d] = dlo[d] = 0x7fffffff; hi[d] = dhi[d] = -0x7fffffff; sum[d] = 0; }
    for (int j = threadIdx.x; j < count; j += blockDim.x) {
        int c[3];
        g.cell_ijk(cell[j], c[0], c[1], c[2]);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            int e = c[d] - at[d];
            if (2 * e > n3[d]) e -= n3[d];
            else if (2 * e < -n3[d]) e += n3[d];
            lo[d] = min(lo[d], c[d]); hi[d] = max(hi[d], c[d]);
            dlo[d] = min(dlo[d], e); dhi[d] = max(dhi[d], e);
            sum[d] += e;
        }
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int r[5] = {__reduce_min_sync(FULL, lo[d]), __reduce_max_sync(FULL, hi[d]), __reduce_min_sync(FULL, dlo[d]),
                          __reduce_max_sync(FULL, dhi[d]), __reduce_add_sync(FULL, sum[d])};
        if ((threadIdx.x & 31) == 0)
            for (int q = 0; q < 5; q++) red[(5 * d + q) * nw + warp] = r[q];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int a[3], b[3];
        int64_t nodes = 1;
        for (int d = 0; d < 3; d++) {
            const int *r = red + 5 * d * nw;
            a[d] = r[0];
            b[d] = r[nw];
            for (int w = 1; w < nw; w++) { a[d] = min(a[d], r[w]); b[d] = max(b[d], r[nw + w]); }
            nodes *= b[d] - a[d] + 3;
        }
        if (nodes > cap) {
            int mid[3];
            for (int d = 0; d < 3; d++) {
                const int *r = red + 5 * d * nw;
                int mn = r[2 * nw], mx = r[3 * nw], sm = r[4 * nw];
                for (int w = 1; w < nw; w++) {
                    mn = min(mn, r[2 * nw + w]); mx = max(mx, r[3 * nw + w]); sm += r[4 * nw + w];
                }
                const int m = at[d] + (int)rintf((float)sm / (float)count);
                mid[d] = m < 0 ? m + n3[d] : (m >= n3[d] ? m - n3[d] : m);
                a[d] = max(max(at[d] + mn + mid[d] - m, 0), mid[d] - 15);
                b[d] = min(min(at[d] + mx + mid[d] - m, n3[d] - 1), mid[d] + 15);
                a[d] = min(a[d], mid[d]);
                b[d] = max(b[d], mid[d]);
            }
            while ((b[0] - a[0] + 3) * (b[1] - a[1] + 3) * (b[2] - a[2] + 3) > cap) {
                int d = 0;
                for (int e = 1; e < 3; e++)
                    if (b[e] - a[e] > b[d] - a[d]) d = e;
                if (b[d] - mid[d] >= mid[d] - a[d]) b[d]--;
                else a[d]++;
            }
        }
        AdjWindow w;
        w.i0 = a[0]; w.l0 = a[1]; w.k0 = a[2];
        w.cx = b[0] - a[0] + 1; w.cy = b[1] - a[1] + 1; w.cz = b[2] - a[2] + 1;
        w.SY = w.cy + 2; w.SZ = w.cz + 2;
        w.nn = (w.cx + 2) * w.SY * w.SZ;
        *out = w;
    }
    __syncthreads();
    return *out;
}
// e with 2^(e-1) <= x < 2^e for a positive normal float, at least -120
__device__ __forceinline__ int adj_exponent(float x) {
    const int e = x > 0.f ? (int)((__float_as_uint(x) >> 23) & 0xff) - 126 : -120;
    return max(e, -120);
}

// 2^e as a double from its exponent bits (|e| < 1000)
__device__ __forceinline__ double pow2_d(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
size_t adj_state_bytes(const AdjState &A);
void adj_state_view(const AdjState &A, char *base, int *cell[kMaxSpecies], void *v[kMaxSpecies][6]);

// ---- FP32 form (pic_adjoint_mixed.cu): particle kernels of the fixed-order pass
struct MixSp {
    int64_t n;
    double q_m, m;
    int *cell;     // packed cell
    float *v[6];   // in-cell offsets (cell units) and momenta
};
struct MixOut {
    int *cell;
    float *v[6];
};
struct MixParams {
    Grid g;
    int nsp;
    const AdjChunk *chunks;     // one per CTA
    int64_t off[kMaxSpecies + 1];
    MixSp sp[kMaxSpecies];      // state at the start of the step
    MixOut out[kMaxSpecies];    // push: state after the step (may alias sp)
    const float *E[3];
    const float *H[3];          // push: H after the half step
    double *J[3];
    AdjStatus *st;
    // adjoint
    float *lam[kMaxSpecies][6]; // lambda_x (cell units), lambda_p
    const double *LJ[3];
    double *LE[3], *LH[3];
};
cudaError_t launch_flat_push_mixed(const MixParams &P, int nchunks, cudaStream_t s);
cudaError_t launch_adj_particles_mixed(const MixParams &P, int nchunks, cudaStream_t s);
void adj_gather_mixed(const Grid &g, const SpeciesView &S, const int64_t *d0, int *cell, void *const v[6],
                      cudaStream_t s);
// lambda_p (3 FP32 arrays of n) and p0 (3 FP32 arrays) -> 6 FP64 arrays of n
void adj_widen_mixed(const float *lp, const float *const p0[3], int64_t n, double *out6, cudaStream_t s);

}  // namespace pic
