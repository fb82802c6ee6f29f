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
    int *far;          // steps: particles outside their chunk's window, as far as windows were used
    // the first steps, forward and in reverse, whose particle kernels use no windows
    int direct_from, direct_adj_from;
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

// ---- a chunk's window: the periodic box of cells whose nodes a CTA keeps in shared memory
// The forward's strides are those of 8 x 12 nodes in y and z, x planes two nodes
// further apart against bank conflicts, where that is enough (a tile of 4 x 8
// cells and a cell of drift on either side), fits, and the chunk is not small:
// offsets of taps and sums are then immediates.  128x32x32 cells: FP64 1.047 ->
// .978 ms per step, FP32 .617 -> .587 (planes 96 nodes apart: 1.152 and .641).
// The adjoint kernels, short of registers, lose by it (FP64 2.27 -> 2.31 ms).
// WRAP: an axis whose cells run past the grid's end and go on at 0 has the nodes of
// its cells up to the end (two more than cells), then those of its cells from 0 on.
constexpr int kFixSX = 98, kFixSY = 8, kFixSZ = 12;  // nodes per x plane, y plane, z line
constexpr int kFixCount = 1024;  // particles that pay for the padding
template <bool WRAP>
struct AdjWindow {
    int lo[3], cells[3], n[3];  // per axis: first cell, cells, the grid's cells
    int N1, N2;                 // nodes along y and z
    int SX, SY, SZ, nn;         // node strides, and nodes of the window with the strides' padding
    // the strides are kFixSY and kFixSZ: kernels then have them at compile time
    __device__ __forceinline__ bool fixed() const { return SX == kFixSX && SY == kFixSY && SZ == kFixSZ; }
    // window-local node of a cell (its lower corner); false: outside
    // (sx, sy: its strides)
    __device__ __forceinline__ bool place(const int c[3], int sx, int sy, int u[3], int &node) const {
        bool in = true;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const int v = c[d] - lo[d], on = WRAP && v < 0 ? n[d] : 0;  // on: past the end
            in = in && (unsigned)(v + on) < (unsigned)cells[d];
            u[d] = v + on + (on ? 2 : 0);
        }
        node = u[0] * sx + u[1] * sy + u[2];
        return in;
    }
    // the grid's node at position u of axis d; for the lower corner of a cell, its cell
    __device__ __forceinline__ int at(int d, int u) const {
        const int end = n[d] - lo[d] + 2;
        return !WRAP || u < end ? lo[d] + u : u - end;
    }
    // the grid's node of window node e; false: padding
    __device__ __forceinline__ bool grid_node(const Grid &g, int e, size_t &n) const {
        const int sx = WRAP ? SY * SZ : SX, a = e / sx, bc = e - a * sx, b = bc / SZ, c = bc - b * SZ;
        n = g.node(at(0, a), at(1, b), at(2, c));
        return WRAP || (b < N1 && c < N2);
    }
};
// nodes of an axis whose window starts at cell lo
__device__ __forceinline__ int window_nodes(int lo, int cells, int n) { return cells + 2 + (lo + cells > n ? 2 : 0); }

// The window of `count` particles' cells with at most `cap` nodes: per axis the
// smaller of their bounding box and the periodic one, where that fits; else the
// periodic box around their mean, cut at the grid's ends and then shrunk on its
// longest axis until it fits, and the particles outside it use global memory.  Every thread of the CTA calls it;
// red holds 15 ints per warp.
// Particles that crossed the grid's end would else go through global memory, one
// at a time, while their CTA waits: with WRAP in the adjoint kernels (and 704
// instead of 640 nodes in FP64, 672 in FP32) 16x8x8 cells 45.2 -> 30.4 us per
// reverse step (FP64), 128x32x32 2.298 -> 2.273 ms (FP64), 1.350 -> 1.314
// (FP32).  The forward pushes don't gain: particles outside take little longer
// there (FP32 64x32x32 cells 187 us without, 191 with).
template <bool WRAP>
__device__ __forceinline__ AdjWindow<WRAP> chunk_window(const Grid &g, const int *__restrict__ cell, int count, int cap,
                                                        int *red, AdjWindow<WRAP> *out) {
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
    if (threadIdx.x < 15) {  // the warps' results, one of the 15 per lane
        int *r = red + threadIdx.x * nw, v = r[0];
        const int kind = threadIdx.x % 5;
        for (int q = 1; q < nw; q++) v = kind == 4 ? v + r[q] : (kind & 1 ? max(v, r[q]) : min(v, r[q]));
        r[0] = v;
    }
    if (threadIdx.x < 32) __syncwarp();
    if (threadIdx.x == 0) {
        AdjWindow<WRAP> w;
        int a[3], b[3], m[3];  // periodic box and mean, as distances from at
        int64_t nodes = 1;
        for (int d = 0; d < 3; d++) {
            const int *r = red + 5 * d * nw;
            const int l0 = r[0], h0 = r[nw], sm = r[4 * nw];
            a[d] = r[2 * nw];
            b[d] = r[3 * nw];
            m[d] = (int)rintf((float)sm / (float)count);
            w.n[d] = n3[d];
            w.lo[d] = at[d] + a[d];
            if (w.lo[d] < 0) w.lo[d] += n3[d];
            w.cells[d] = b[d] - a[d] + 1;
            if ((!WRAP && w.lo[d] + w.cells[d] > n3[d]) || window_nodes(w.lo[d], w.cells[d], n3[d]) >= h0 - l0 + 3) {
                w.lo[d] = l0;
                w.cells[d] = h0 - l0 + 1;
            }
            nodes *= window_nodes(w.lo[d], w.cells[d], n3[d]);
        }
        if (nodes > cap) {
            int s[3];
            for (int d = 0; d < 3; d++) {
                m[d] = min(max(m[d], a[d]), b[d]);
                a[d] = max(a[d], m[d] - 15);
                b[d] = min(b[d], m[d] + 15);
                if (b[d] - a[d] + 1 > n3[d]) {  // both ends half the axis away: the same cell
                    if (b[d] > m[d]) b[d]--;
                    else a[d]++;
                }
            }
            for (;;) {
                nodes = 1;
                for (int d = 0; d < 3; d++) {
                    s[d] = at[d] + a[d];
                    s[d] = s[d] < 0 ? s[d] + n3[d] : (s[d] >= n3[d] ? s[d] - n3[d] : s[d]);
                    nodes *= window_nodes(s[d], b[d] - a[d] + 1, n3[d]);
                }
                if (WRAP && nodes <= cap) break;
                // first what lies past the grid's end, few particles for three nodes or more
                int cut = -1, lost = WRAP ? 4 : 0x7fffffff;
                for (int d = 0; d < 3; d++) {
                    const int len = b[d] - a[d] + 1, before = n3[d] - s[d];
                    const int l = m[d] - a[d] < before ? len - before : before;
                    if (before < len && l < lost) { cut = d; lost = l; }
                }
                if (cut >= 0) {
                    if (m[cut] - a[cut] < n3[cut] - s[cut]) b[cut] -= lost;
                    else a[cut] += lost;
                    continue;
                }
                if (nodes <= cap) break;
                int d = 0;
                for (int e = 1; e < 3; e++)
                    if (b[e] - a[e] > b[d] - a[d]) d = e;
                if (b[d] - m[d] >= m[d] - a[d]) b[d]--;
                else a[d]++;
            }
            for (int d = 0; d < 3; d++) {
                w.lo[d] = s[d];
                w.cells[d] = b[d] - a[d] + 1;
            }
        }
        const int N0 = window_nodes(w.lo[0], w.cells[0], n3[0]);
        w.N1 = window_nodes(w.lo[1], w.cells[1], n3[1]);
        w.N2 = window_nodes(w.lo[2], w.cells[2], n3[2]);
        const bool fix = !WRAP && count >= kFixCount && w.N1 <= kFixSY && w.N2 <= kFixSZ && N0 * kFixSX <= cap;
        w.SY = fix ? kFixSY : w.N1;
        w.SZ = fix ? kFixSZ : w.N2;
        w.SX = fix ? kFixSX : w.SY * w.SZ;
        w.nn = N0 * w.SX;
        *out = w;
    }
    __syncthreads();
    return *out;
}
// The block-wide maximum that the adjoint kernels take of every batch of 256
// particles lies in one of three slots of shared memory: batch `it` collects into
// max_slot(it), one barrier follows, every thread reads the slot, and thread 0
// clears max_cleared(it), where batch it + 2 will collect.  Between two barriers
// the threads then read slot it, clear slot it + 2 and collect into slot it + 1,
// in any order: with two slots a late clear wiped out the next batch's maximum.
constexpr int kMaxSlots = 3;
__host__ __device__ __forceinline__ int max_slot(int it) { return it % kMaxSlots; }
__host__ __device__ __forceinline__ int max_cleared(int it) { return (it + 2) % kMaxSlots; }
// The quantum of the sums in a window: contributions up to 2^E, E from the largest
// |lambda of a field value| of the batch at hand (its bits, which order as the
// values do), two powers of two above it at first.  Where a batch's largest is
// past 2^E, or more than `keep` powers of two below it, the sums so far go to the
// global arrays and the window starts again at the batch's own quantum: a chunk's
// particles are not rounded in the units of a strongly amplified one among them.
// keep: no contribution is rounded more coarsely than by 2^-45 (FP64) or 2^-23
// (FP32) of its batch's largest.
constexpr int kNoQuantum = -2000;  // none yet
// e with 2^(e-1) <= x < 2^e, from the high word of a non-negative normal double
__host__ __device__ __forceinline__ int exponent_hi(unsigned hi) { return (int)(hi >> 20) - 1022; }
// the same from the bits of a non-negative normal float
__host__ __device__ __forceinline__ int exponent_f(unsigned bits) { return (int)(bits >> 23) - 126; }
// E for a batch of exponent e when E0 is in use, at least `least`; E0 if that does
__host__ __device__ __forceinline__ int quantum_for(int E0, int e, int keep, int least) {
    const int own = e + 2 < least ? least : e + 2;
    return e > E0 || (e + keep < E0 && own < E0) ? own : E0;
}
// quanta below 2^E, as powers of two; least E: 2^(E - 50) and its inverse are
// normal doubles, 2^(30 - E) a normal float
constexpr int kBitsPlain = 50, kBitsMix = 30;
constexpr int kKeepPlain = kBitsPlain - 44, kKeepMix = kBitsMix - 22;
constexpr int kLeastPlain = -900, kLeastMix = -93;

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
    int *far;                   // push: counts the particles outside their chunk's window (null: not)
    // adjoint
    float *lam[kMaxSpecies][6]; // lambda_x (cell units), lambda_p
    const double *LJ[3];
    double *LE[3], *LH[3];
};
cudaError_t launch_flat_push_mixed(const MixParams &P, int nchunks, bool direct, cudaStream_t s);
cudaError_t launch_adj_particles_mixed(const MixParams &P, int nchunks, bool direct, cudaStream_t s);
void adj_gather_mixed(const Grid &g, const SpeciesView &S, const int64_t *d0, int *cell, void *const v[6],
                      cudaStream_t s);
// lambda_p (3 FP32 arrays of n) and p0 (3 FP32 arrays) -> 6 FP64 arrays of n
void adj_widen_mixed(const float *lp, const float *const p0[3], int64_t n, double *out6, cudaStream_t s);

}  // namespace pic
