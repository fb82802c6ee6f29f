// Internal definitions of the B200 PIC step: geometry, device views of the
// state, the status word and the sizes of the tile layout.
//
// Data layout in HBM
//   fields   one array per component (E, H, J, Q), (Nx+2) x (Ny+2) x Pz with
//            Pz = round_up(Nz+2, 4) so every z row starts on a 32-byte
//            boundary (TMA rows, float4/double2 access).  The caller sees the
//            reference layout (Pz = Nz+2) through pic_get_field/pic_set_field.
//   particles one SoA set per species, binned by TILE: a tile is a block of
//            tx*ty*tz interior cells; tile t owns slots
//            [tile_start[t], tile_start[t+1]) of which the first tile_count[t]
//            are live.  Each particle carries its int32 interior cell index
//            ((i*Ny + l)*Nz + k); the plain form stores global FP64 positions,
//            the mixed form FP32 in-cell offsets in [0,1).  A particle that
//            crosses a cell boundary inside its tile only rewrites its cell
//            index; only tile leavers move (outbox -> insert).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include <utility>
#include "pic0buf.h"

namespace pic {

constexpr int kMaxSpecies = PIC_MAX_SPECIES;
constexpr int kSMs = 148;               // of a B200: the grids of walks over nodes, particles and tiles
constexpr int kHoleMax = 1024;          // departures per tile per species listed before the spill list
constexpr int kHoleSpill = 16;          // one spill entry per this many slots of the bin
constexpr int kPushThreads = 256;       // threads of a push CTA: particles per block of a slice
constexpr unsigned kOutboxChunk = 16;   // outbox slots a warp of the FP32 push takes at once

// status flag bits (DevStatus::flags)
enum : unsigned {
    ST_STENCIL = 1u,     // stencil index outside the staged tile (CFL)
    ST_OUTBOX = 2u,      // outbox overflow
    ST_HOLES = 4u,       // hole list overflow
    ST_NAN = 8u,         // non-finite momentum
    ST_TILE_FULL = 16u,  // arrivals did not fit their tile (kept in the outbox, rebin needed)
    ST_BADCELL = 32u,    // a bin held a cell outside its tile, or the compaction did not pair up
    ST_TMA = 64u,        // the field tile's TMA load did not complete within the wait limit
};

struct DevStatus {
    unsigned flags;
    unsigned out_count;        // outbox entries this step
    unsigned overflow_count;   // outbox entries that did not fit their tile
    unsigned full_species;     // bit s: species s has such entries
    unsigned long long moved;  // particles written to the outbox
    unsigned long long dropped;
    unsigned long long duplicated;
    double kinetic;            // sum (m/q_m)(gamma-1) accumulated by the push
    double pad1[3];
};

struct Grid {
    int nx, ny, nz;     // interior cells
    int NX, NY, NZ;     // nx+2, ny+2, nz+2
    int pz;             // z pitch of device field arrays
    int tx, ty, tz;     // cells per tile
    int ntx, nty, ntz;  // tiles per axis
    int ntiles;
    int bz, by;         // bits of the packed cell index used by k and by l
    double lx, ly, lz, hx, hy, hz, tau;
    __host__ __device__ size_t nodes_pitched() const { return (size_t)NX * NY * pz; }
    __host__ __device__ size_t nodes_ref() const { return (size_t)NX * NY * NZ; }
    __host__ __device__ size_t node(int i, int l, int k) const { return ((size_t)i * NY + l) * pz + k; }
    __host__ __device__ int ncells() const { return nx * ny * nz; }
    // a particle's int32 cell index packs (i, l, k) as bit fields, so the hot
    // loops decode it with shifts and masks instead of integer division
    __host__ __device__ int cell_of(int i, int l, int k) const { return (i << (by + bz)) | (l << bz) | k; }
    __host__ __device__ void cell_ijk(int c, int &i, int &l, int &k) const {
        k = c & ((1 << bz) - 1);
        l = (c >> bz) & ((1 << by) - 1);
        i = c >> (by + bz);
    }
    __host__ __device__ int dense_of(int i, int l, int k) const { return (i * ny + l) * nz + k; }
    __host__ __device__ int tile_of_cell(int i, int l, int k) const {
        return ((i / tx) * nty + (l / ty)) * ntz + (k / tz);
    }
};

// The field kernels after the push (J fold, B, E, E ghosts) run as a chain
// of programmatically dependent launches: each is launched with
// cudaLaunchAttributeProgrammaticStreamSerialization, and every CTA first
// waits in hardware for the previous grid to complete and flush
// (griddepcontrol.wait), then lets the next grid be scheduled
// (griddepcontrol.launch_dependents).  The next grid's CTAs thus take SM
// slots as this grid's retire and start the moment it is done, instead of
// after a full launch gap; every CTA of a grid has started before the next
// grid's are scheduled, so waiting CTAs never hold slots the running grid
// needs.  For a kernel launched without the attribute both are no-ops.
__device__ __forceinline__ void chain_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// Time stamps of a step's kernels (nanoseconds of the GPU's global timer), one
// per phase boundary, in place of events between the launches: an event is work
// of its own on the stream and keeps the next kernel from being launched ahead
// (32x4x4 cells, FP64 72 -> 53 us per step, FP32 62 -> 46 without its six).
constexpr int kStamps = 6;
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void stamp_entry(unsigned long long *stamps, int k) {
    if (stamps && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) stamps[k] = global_ns();
}
template <typename... P, typename... A>
inline cudaError_t launch_chained_smem(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                       A &&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A &&... args) {
    return launch_chained_smem(kernel, grid, block, 0, s, std::forward<A>(args)...);
}

// Tile current accumulation in 64-bit fixed point.  Each contribution is
// rounded to the tile's quantum q = 2^(E-62), where 2^E exceeds
// bound = 2.5 * sum_s |m_s| * count_s(tile): one particle segment adds at most
// 1.03 |m| to a node (pqr, cell.h:1578-1616, with |dx| < tau and the stencil
// in range), two segments per particle, so no tile sum can overflow.  The
// sums are exact integer sums, so the tile current does not depend on the
// order in which the threads add.  Rounding: |error| <= q/2 per contribution.
//
// Every 64-bit add into shared memory goes through shared_add64: two native
// 32-bit atomics.  The add of the low halves returns the old low word, so the
// carry of each add is known exactly and goes into the high word with the
// high half.  Integer adds modulo 2^32 commute, so the pair, read as one
// little-endian 64-bit word after a barrier, is the exact sum modulo 2^64 --
// what a 64-bit atomicAdd gives -- whatever the interleaving.  Measured: a
// 64-bit shared-memory atomicAdd costs about 8 atomic instructions per add
// in the FP64 push (lanes of a warp often share a node), and the split took
// the c2 FP64 push from 106.4 to 72.4 ms.
__device__ __forceinline__ void shared_add64(unsigned *plo, unsigned *phi, long long v) {
    const unsigned lo = (unsigned)v;
    const unsigned old = atomicAdd(plo, lo);
    const unsigned hi = (unsigned)((unsigned long long)v >> 32) + (old + lo < old ? 1u : 0u);
    if (hi) atomicAdd(phi, hi);
}
__device__ __forceinline__ void shared_add64(unsigned long long *w, long long v) {
    unsigned *p = (unsigned *)w;  // p[0] low word, p[1] high word
    shared_add64(p, p + 1, v);
}
// a 32-bit addend: the high word changes only when the low one carries (or, for
// a negative addend, does not)
__device__ __forceinline__ void shared_add64_small(unsigned *plo, unsigned *phi, int v) {
    const unsigned lo = (unsigned)v;
    const unsigned old = atomicAdd(plo, lo);
    const unsigned hi = (unsigned)(v >> 31) + (old + lo < old ? 1u : 0u);
    if (hi) atomicAdd(phi, hi);
}
__device__ __forceinline__ void fx_addf(unsigned long long *a, float v, float inv_q) {
    long long iv = __float2ll_rn(v * inv_q);
    if (iv) shared_add64(a, iv);
}
// Two-word form for the FP64 plain form.  The bound above assumes every
// particle moves at c; a dense slow plasma (thousands of particles per cell at
// v ~ 1e-3, whose beam and return currents cancel) adds contributions ~1e-9 of
// the bound, which a single word rounds at ~1e-10 of their size.  The second
// word takes each contribution's remainder in units of q * 2^-40:
//   s = v / q (exact: q is a power of two), r = rint(s), s - r exact
//   (Sterbenz: |s - r| <= 1/2 and r, s within a factor 2 when r != 0),
// so the error is <= q * 2^-41 per contribution, and both adds are exact
// integer adds (order-independent).  |lo| grows by <= 2^39 per add: 2^24
// adds into one node before it could overflow, i.e. 8M particles in a tile
// (kFxMaxTileSlots guards it).
constexpr int kFxLoBits = 40;
constexpr long long kFxMaxTileSlots = 1ll << 23;
// s is in quanta with |s| < 2^51 and is rounded by adding 1.5 * 2^52 (to
// nearest even, as rint): conversions between FP64 and integers run at a
// quarter of the FP64 add rate.
constexpr double kRound = 0x1.8p52;
// a contribution rounded by u = s + kRound, into a node's low and high word
__device__ __forceinline__ void shared_add_rounded(unsigned *plo, unsigned *phi, double u) {
    const unsigned lo = (unsigned)__double2loint(u);
    const unsigned old = atomicAdd(plo, lo);
    const unsigned hi = (unsigned)__double2hiint(u) - 0x43380000u + (old + lo < old ? 1u : 0u);
    if (hi) atomicAdd(phi, hi);
}
// (w: the node's low word; its high word and the remainder's low and high word
// follow at distances of d: arrays of low and of high words use all banks, where
// pairs of them put every low word on an even one)
__device__ __forceinline__ void fx_put2(unsigned *w, int d, double s) {
    const double u = s + kRound, r = s - (u - kRound);  // the exact remainder
    shared_add_rounded(w, w + d, u);
    shared_add_rounded(w + 2 * d, w + 3 * d, fma(r, 1099511627776.0, kRound));  // 2^40
}
// The same split with an int32 second word (native 32-bit shared atomics: a
// c2 FP64 push takes 22 ms less than with the 64-bit word).  The remainder
// s - r (|s - r| <= 1/2) is counted in units of q * 2^-L, so one add is at
// most 2^(L-1) in magnitude.  A tile of N particles adds at most 2N times to
// one word (two zigzag segments per particle, one add per node of a segment),
// so L = 31 - bits(N), N < 2^bits(N), keeps every sum below N 2^L < 2^31:
// exact and order-independent like the 64-bit word, with |error| <=
// q * 2^-(L+1) per contribution.  The push uses it when every tile's
// capacity gives L >= kFxLo32MinBits (tiles below 2^17 particles; the
// reference's default run, 2.6e5 particles per tile, keeps the 64-bit word).
constexpr int kFxLo32MinBits = 14;
__device__ __forceinline__ int fx_lo32_bits(long long n) {
    int b = 0;
    while ((1ll << b) <= n) b++;
    return 31 - b;
}
__device__ __forceinline__ void fx_put_lo32(unsigned *w, int d, double s, double lo_scale) {
    const double u = s + kRound, r = s - (u - kRound);
    shared_add_rounded(w, w + d, u);
    atomicAdd((int *)w + 2 * d, __double2loint(fma(r, lo_scale, kRound)));  // lo_scale = 2^L: exact
}
// the sums in the words of a node (LO32: with the int32 remainder)
template <bool LO32>
__device__ __forceinline__ void fx_get(const unsigned *w, int d, long long &ih, long long &il) {
    ih = (long long)(((unsigned long long)w[d] << 32) | w[0]);
    il = LO32 ? (long long)(int)w[2 * d] : (long long)(((unsigned long long)w[3 * d] << 32) | w[2 * d]);
}

struct SpeciesView {
    // plain form
    double *x, *y, *z, *px, *py, *pz;
    // mixed form
    float *ox, *oy, *oz, *fx, *fy, *fz;
    int *cell;
    int *tile_start;  // ntiles + 1
    int *tile_count;  // ntiles
    // holes of a push past the first kHoleMax of a bin, and the compaction's
    // front holes past theirs: slots / 8 ints (see HoleList)
    int *spill;
    double q_m, m;
};

// The holes that a push leaves in one bin: the first kHoleMax entries in
// `base` (shared memory, or global memory when several CTAs share the tile),
// the rest in the bin's part of the spill list, one entry per kHoleSpill slots.
// A second list of the same shape takes the compaction's front holes.  Dense
// hot tiles need the spill: at 700 particles per cell and vth 0.1 about 2000
// leave a tile per step, and a list of 1024 alone had the host rebin every
// species after nearly every step.
struct HoleList {
    int *base, *spill;
    int cap;  // spill entries
    __device__ __forceinline__ int limit() const { return kHoleMax + cap; }
    __device__ __forceinline__ int *at(int r) const { return r < kHoleMax ? base + r : spill + (r - kHoleMax); }
};
__device__ __forceinline__ HoleList hole_list(const SpeciesView &S, int t, int *base, bool front) {
    HoleList h;
    const int a = S.tile_start[t];
    h.base = base;
    h.cap = (S.tile_start[t + 1] - a) / kHoleSpill;
    h.spill = S.spill + a / (kHoleSpill / 2) + (front ? h.cap : 0);
    return h;
}

// one migrating particle (plain form): 56 bytes
struct OutPlain {
    double x, y, z, px, py, pz;
    int cell, species;
};
// one migrating particle (mixed form): 32 bytes, read and written in halves of 16
struct __align__(16) OutMixed {
    float ox, oy, oz, px, py, pz;
    int cell, species;
};
static_assert(sizeof(OutMixed) == 32 && alignof(OutMixed) == 16, "two 128-bit accesses");

// Momenta of the live particles among slots start + {j, j + B, j + 2B, j + 3B}
// (B = blockDim.x) below start + jend, zeros for the others.  All loads are
// issued before any is looked at: a reduction that loads one particle at a time
// waits for it.
__device__ __forceinline__ void load_momenta4(int mixed, const SpeciesView &S, int start, int j, int jend,
                                              double p[4][3]) {
    bool live[4];
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const int q = j + v * (int)blockDim.x, slot = start + q;
        live[v] = q < jend && S.cell[slot] >= 0;
        p[v][0] = p[v][1] = p[v][2] = 0.0;
        if (q < jend) {
            if (mixed) { p[v][0] = S.fx[slot]; p[v][1] = S.fy[slot]; p[v][2] = S.fz[slot]; }
            else { p[v][0] = S.px[slot]; p[v][1] = S.py[slot]; p[v][2] = S.pz[slot]; }
        }
    }
#pragma unroll
    for (int v = 0; v < 4; v++)
        if (!live[v]) p[v][0] = p[v][1] = p[v][2] = 0.0;
}

struct StepParams {
    Grid g;
    int nsp;
    int mixed;
    SpeciesView sp[kMaxSpecies];
    long long slots;  // of the species with the most
    // plain: double fields; mixed: float E/H, double J
    const void *E[3];
    const void *H[3];
    double *J[3];
    void *outbox;
    unsigned out_cap;
    DevStatus *st;
    // mixed push: per species, the largest contribution bound of the last
    // push (float, 0 = none yet) and the one this push records (float bits,
    // atomicMax); sizes the int32 tile current's quantum
    const float *lb_prev;
    unsigned *lb_cur;
    // mixed push: nonzero when H in memory is the full-step field and the
    // push forms the B half step of its staged tile itself (pic_step); zero
    // when the sub-step call pic_b_half has already advanced H
    int b_half;
    // a tile's bins are shared out to `slices` CTAs (1: one CTA per tile; the
    // pointers below are then unused).  The CTAs of a tile list their leavers'
    // slots in holes ([species][tile][kHoleMax], filled to hole_count
    // [species][tile]) and count themselves off in ticket[tile]; the last one
    // compacts the tile's bins.  hole_count and ticket start a push at zero.
    int slices;
    int *holes;
    unsigned *hole_count, *ticket;
    int prefetch;  // plain push: the next particle comes through shared memory (set by its launcher)
    int jcopies;   // plain push: tile currents per CTA, 1 or 2 (set by its launcher)
    unsigned long long *stamps;  // kStamps of the step (null: a sub-step call)
};

// one 4- or 8-byte asynchronous copy from global to shared memory
template <int B>
__device__ __forceinline__ void cp_async(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(B)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Shares that a reduction over the bins deals a tile out in, by `rows` rows of blocks
// (one per species, or one for all): enough blocks for eight per SM where the tiles
// alone are too few, but none of fewer than kShareLeast particles.  A momentum call on
// 8x8x8 cells of 4 particles took 37 us with 3552 blocks of one or two particles each,
// takes 25; 64x32x32 cells, eight species of 8, 62 and 47.
constexpr int kShareLeast = 1024;
inline int tile_shares(const StepParams &p, int rows) {
    const int most = 8 * kSMs, tiles = p.g.ntiles * rows;
    return (int)std::min<long long>((most + tiles - 1) / tiles, 1 + p.nsp / rows * p.slots / kShareLeast);
}
// those of them that a tile of n particles fills, one at least; blocks without a
// share add nothing
__device__ __forceinline__ int shares_filled(long long n, int shares) {
    const long long s = (n + kShareLeast - 1) / kShareLeast;
    return s < 1 ? 1 : (s < shares ? (int)s : shares);
}

// The particles of one species that slice q of P.slices of tile t handles:
// [jbeg, jend) of the bin.  The bins of all species, cut into blocks of
// `threads` particles and laid end to end, are dealt out evenly, so the slices
// of a tile cover every particle once and each is a few whole iterations.
struct SliceRange {
    int lo, hi;  // blocks of this slice
};
__device__ __forceinline__ SliceRange slice_blocks(const StepParams &P, int t, int q, int threads) {
    long long w = 0;
    for (int s = 0; s < P.nsp; s++) w += (P.sp[s].tile_count[t] + threads - 1) / threads;
    SliceRange r;
    r.lo = (int)(w * q / P.slices);
    r.hi = (int)(w * (q + 1) / P.slices);
    return r;
}
// this slice's particles of a species whose first block is block `first`
__device__ __forceinline__ void slice_range(const SliceRange &r, int first, int count, int threads, int &jbeg, int &jend) {
    const long long a = (long long)(r.lo - first) * threads, b = (long long)(r.hi - first) * threads;
    jbeg = (int)(a < 0 ? 0 : (a > count ? count : a));
    jend = (int)(b < jbeg ? jbeg : (b > count ? count : b));
}

// lists hole j as entry r of a bin's holes; false when the list is full
__device__ __forceinline__ bool list_hole(const SpeciesView &S, int t, int *base, unsigned r, int j) {
    if (r < (unsigned)kHoleMax) {
        base[r] = j;
        return true;
    }
    const HoleList h = hole_list(S, t, base, false);
    if (r >= (unsigned)h.limit()) return false;
    *h.at((int)r) = j;
    return true;
}

// True in the last CTA of tile t to get here, whose threads then see what the
// tile's other CTAs wrote (fence, ticket, fence).  No CTA waits for another.
// Every thread calls it; flag is shared memory.
__device__ __forceinline__ bool last_of_tile(const StepParams &P, int t, int *flag) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        *flag = atomicAdd(&P.ticket[t], 1u) == (unsigned)P.slices - 1u;
        __threadfence();
    }
    __syncthreads();
    return *flag != 0;
}

// Compaction of tile t's bin of species s by one CTA, from the holes that all
// the tile's CTAs listed: the last live particles move into the holes in front
// of the new count.  front: kHoleMax ints and ctr: 2 ints of shared memory;
// move(dst, src) copies one particle.  The data comes from other SMs, so it is
// read past L1 (__ldcg).
template <class Move>
__device__ __forceinline__ void compact_listed(const StepParams &P, int t, int s, int *front, int *ctr, unsigned &bad,
                                               Move move) {
    const SpeciesView &S = P.sp[s];
    const size_t e = (size_t)s * P.g.ntiles + t;
    const unsigned listed = __ldcg(&P.hole_count[e]);
    const HoleList holes = hole_list(S, t, P.holes + e * kHoleMax, false), fronts = hole_list(S, t, front, true);
    if (listed == 0u || listed > (unsigned)holes.limit()) return;
    const int nh = (int)listed, start = S.tile_start[t], newcount = S.tile_count[t] - nh;
    if (threadIdx.x == 0) ctr[0] = ctr[1] = 0;
    __syncthreads();
    for (int r = threadIdx.x; r < nh; r += blockDim.x) {
        const int h = __ldcg(holes.at(r));
        if (h < newcount) *fronts.at(atomicAdd(&ctr[0], 1)) = h;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < nh; r += blockDim.x) {
        const int src = start + newcount + r;
        if (__ldcg(&S.cell[src]) >= 0) {
            const int m = atomicAdd(&ctr[1], 1);
            if (m >= ctr[0]) { bad |= ST_BADCELL; continue; }
            move(start + *fronts.at(m), src);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) S.tile_count[t] = newcount;
    __syncthreads();
}

// Compaction of all of tile t's bins by the last CTA of the tile, from the holes
// that the tile's CTAs listed.  work: 2 kHoleMax ints of shared memory.  The
// species go through compact_listed's two phases side by side where the list of
// fronts of all of them fits there (a wait for memory per phase instead of per
// phase and species: 32x4x4 cells, push FP64 24.0 -> 22.1 us, FP32 with the
// field loads beside the quantum 21.4 -> 18.4), else one after the other.
template <class Move>
__device__ __forceinline__ void compact_tile(const StepParams &P, int t, int *work, unsigned &bad, Move move) {
    int *nh = work, *start = nh + kMaxSpecies, *keep = start + kMaxSpecies, *nfront = keep + kMaxSpecies,
        *nmove = nfront + kMaxSpecies, *fronts = nmove + kMaxSpecies;
    constexpr int kRoom = 2 * kHoleMax - 5 * kMaxSpecies;
    if ((int)threadIdx.x < P.nsp) {
        const int s = threadIdx.x;
        const SpeciesView &S = P.sp[s];
        const size_t e = (size_t)s * P.g.ntiles + t;
        const unsigned listed = __ldcg(&P.hole_count[e]);
        const int a = S.tile_start[t], b = S.tile_start[t + 1], count = S.tile_count[t];
        const int n = listed <= (unsigned)(kHoleMax + (b - a) / kHoleSpill) ? (int)listed : 0;
        nh[s] = n;
        start[s] = a;
        keep[s] = count - n;
        nfront[s] = nmove[s] = 0;
    }
    __syncthreads();
    int total = 0;
    for (int s = 0; s < P.nsp; s++) total += nh[s];
    if (total > kRoom) {
        __syncthreads();  // before work is used otherwise
        for (int s = 0; s < P.nsp; s++) compact_listed(P, t, s, work + kHoleMax, work, bad, [&](int dst, int src) { move(P.sp[s], dst, src); });
        return;
    }
    // entry r of the species' lists one after another: species s, its entry, its first
    auto find = [&](int r, int &s, int &first) {
        s = first = 0;
        while (r - first >= nh[s]) first += nh[s++];
    };
    for (int r = threadIdx.x; r < total; r += blockDim.x) {
        int s, first;
        find(r, s, first);
        const HoleList holes = hole_list(P.sp[s], t, P.holes + ((size_t)s * P.g.ntiles + t) * kHoleMax, false);
        const int h = __ldcg(holes.at(r - first));
        if (h < keep[s]) fronts[first + atomicAdd(&nfront[s], 1)] = h;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < total; r += blockDim.x) {
        int s, first;
        find(r, s, first);
        const SpeciesView &S = P.sp[s];
        const int src = start[s] + keep[s] + r - first;
        if (__ldcg(&S.cell[src]) >= 0) {
            const int m = atomicAdd(&nmove[s], 1);
            if (m >= nfront[s]) { bad |= ST_BADCELL; continue; }
            move(S, start[s] + fronts[first + m], src);
        }
    }
    __syncthreads();
    if ((int)threadIdx.x < P.nsp && nh[threadIdx.x]) P.sp[threadIdx.x].tile_count[t] = keep[threadIdx.x];
}

// FP32 form: TMA descriptors of the six E/H field arrays (3D {Nz+2, Ny+2,
// Nx+2} FP32 with the pitched z row, box = one tile + halo); a kernel
// parameter (__grid_constant__), so the descriptors live in parameter space
struct MixedMaps {
    CUtensorMap m[6];
};


}  // namespace pic
