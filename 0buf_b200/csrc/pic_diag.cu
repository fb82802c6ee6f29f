// Charge-conservation diagnostic of the B200 PIC step, in FP64 on the GPU.
//
// The reference has no charge density.  Its zigzag deposit (CurrentToMesh,
// cell.h:1306-1422, with pqr's linear weights, cell.h:1511-1693) and its E
// update (emeElement, kernels.cu:1091-1102) conserve a discrete Gauss law
// exactly when the charge is assigned as follows (derived from the deposit's
// stencil, pinned by the oracle tests):
//   rho[N]  = sum_p m_p W_x W_y W_z,  W = the linear (cloud-in-cell) weight of
//             the particle on the node at position (N - 1/2) h per axis, i.e.
//             the nodes sit at cell centres; a particle in cell i with in-cell
//             offset f (cell units) has the nodes i + (f >= 1/2) and one up,
//             the upper one with weight f + 1/2 - (f >= 1/2);
//   fold    per axis x, y, z: rho[n] += rho[0], rho[1] += rho[n+1], then the
//             ghosts rho[0] = rho[n], rho[n+1] = rho[1] -- the transverse-line
//             form of the current fold (periodicCurrentElement,
//             kernels.cu:1124-1146);
//   div E   (div E)[N] = sum_a (E_a[N] - E_a[N - e_a]) / h_a on interior nodes.
// Then G = div E - rho on the interior nodes does not change from step to
// step: E changes by -tau J and rho by -tau div J, the curl terms cancel.
// pic_gauss_check reports how far G has moved from a stored baseline.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>
#include <algorithm>
#include <type_traits>
#include "pic0buf.h"
#include "pic_internal.cuh"
#include "pic_kernels.cuh"
#include "pic_plain_math.cuh"
#include "pic_handle.cuh"

namespace pic {
namespace {

// The particles of every species in a share of a tile (blockIdx.y of
// shares_filled) add their eight weights into shared (tx+2)(ty+2)(tz+2) node boxes
// in 64-bit fixed point (exact and order-independent: q = 2^(E-62) with 2^E >
// sum |m| over the tile's particles, each node receives at most that much), and
// the boxes are added into the global rho.  A contribution below 2^51 quanta
// (every tile of 2048 equal charges or more) is rounded by adding 1.5 * 2^52
// instead of by a conversion.
//
// Bound: the 16 shared atomics per particle, before them same-address conflicts
// and the loads.  Consecutive particles mostly share a cell, so lanes add into
// `copies` boxes in turn, whose nodes lie 4 banks apart, and the next particle is
// loaded before the current one is processed.  50.3M particles, 6x4x8 and 8x4x8
// tiles: FP32 696 -> 399 us, FP64 752 -> 447 us (one box 714 and 712, two 637,
// four 483 and 491; 16 boxes, which leave three CTAs per SM, 427 and 546); with
// the tile's dimensions at compile time 386 and 408.  805M FP32 9.95 -> 5.26 ms.
// With few tiles each is dealt out to several CTAs: the reference's default run
// (13 tiles of 500k particles) 3546 -> 100 us FP64, 2118 -> 87 us FP32.
// The copies: as many as five CTAs per SM leave room for.
constexpr int kRhoCopies = 8, kRhoBytes = 40 * 1024;
// words of a copy: nn low, nn high, and a pad
__host__ __device__ inline int rho_stride(int nn) { return (2 * nn + 31) / 32 * 32 + 4; }
// TX, TY, TZ: the tile's cells per axis when fixed at compile time, 0 to take them
// from the grid
template <bool MIXED, int TX, int TY, int TZ>
__global__ void __launch_bounds__(256) k_charge_tile(StepParams P, int copies, double *rho) {
    using T = typename std::conditional<MIXED, float, double>::type;
    const Grid &g = P.g;
    const int nsp = P.nsp;
    const SpeciesView *sp = P.sp;
    extern __shared__ unsigned sR[];
    __shared__ double sQ, sInvQ;
    __shared__ int sMagic;
    const int t = blockIdx.x;
    const int tk = t % g.ntz, tl = (t / g.ntz) % g.nty, ti = t / (g.ntz * g.nty);
    const int tx = TX ? TX : g.tx, ty = TY ? TY : g.ty, tz = TZ ? TZ : g.tz;
    const int i0 = ti * tx, l0 = tl * ty, k0 = tk * tz;
    const int SX = tx + 2, SY = ty + 2, SZ = tz + 2;
    const int nn = SX * SY * SZ, stride = rho_stride(nn);
    long long inside = 0;
    for (int s = 0; s < nsp; s++) inside += sp[s].tile_count[t];
    const int filled = shares_filled(inside, gridDim.y);
    if ((int)blockIdx.y >= filled) return;  // the whole block
    if (threadIdx.x == 0) {
        double bound = 0.0, one = 0.0;
        for (int s = 0; s < nsp; s++) {
            bound += fabs(sp[s].m) * (double)sp[s].tile_count[t];
            if (sp[s].tile_count[t] > 0) one = fmax(one, fabs(sp[s].m));
        }
        int e2;
        frexp(bound > 0.0 ? bound : 1.0, &e2);
        sQ = ldexp(1.0, e2 - 62);
        sInvQ = ldexp(1.0, 62 - e2);
        sMagic = one * sInvQ < 0x1p51;
    }
    for (int idx = threadIdx.x; idx < copies * stride; idx += blockDim.x) sR[idx] = 0u;
    __syncthreads();
    const double inv_q = sInvQ;
    const bool magic = sMagic;
    const double rhx = 1.0 / g.hx, rhy = 1.0 / g.hy, rhz = 1.0 / g.hz;
    unsigned *mine = sR + (threadIdx.x & (copies - 1)) * stride;
    for (int s = 0; s < nsp; s++) {
        const SpeciesView &S = sp[s];
        const int start = S.tile_start[t];
        const long long all = S.tile_count[t];
        const unsigned jbeg = (unsigned)(all * blockIdx.y / filled), jend = (unsigned)(all * (blockIdx.y + 1) / filled);
        const double mq = S.m * inv_q;  // exact: inv_q is a power of two
        const int *cell = S.cell + start;
        const T *px = MIXED ? (const T *)(S.ox + start) : (const T *)(S.x + start);
        const T *py = MIXED ? (const T *)(S.oy + start) : (const T *)(S.y + start);
        const T *pz = MIXED ? (const T *)(S.oz + start) : (const T *)(S.z + start);
        int nc = -1;
        T nx = 0, ny = 0, nz = 0;
        auto load = [&](unsigned j) {
            nc = -1;
            if (j < jend) { nc = cell[j]; nx = px[j]; ny = py[j]; nz = pz[j]; }
        };
        load(jbeg + threadIdx.x);
        for (unsigned j = jbeg + threadIdx.x; j < jend; j += blockDim.x) {
            const int c = nc;
            const T x = nx, y = ny, z = nz;
            load(j + blockDim.x);
            int i, l, k;
            g.cell_ijk(c, i, l, k);
            double fx, fy, fz;
            if (MIXED) {
                fx = (double)x; fy = (double)y; fz = (double)z;
            } else {
                fx = div_by(x, g.hx, rhx) - (double)i;
                fy = div_by(y, g.hy, rhy) - (double)l;
                fz = div_by(z, g.hz, rhz) - (double)k;
            }
            const bool ux = fx >= 0.5, uy = fy >= 0.5, uz = fz >= 0.5;
            // weights of the upper node
            const double ax = fx + (ux ? -0.5 : 0.5), ay = fy + (uy ? -0.5 : 0.5), az = fz + (uz ? -0.5 : 0.5);
            // tile-local lower node
            i += (int)ux - i0; l += (int)uy - l0; k += (int)uz - k0;
            // a dead slot, or a bin entry outside its tile (never expected)
            if (c < 0 || (unsigned)i >= (unsigned)SX - 1u || (unsigned)l >= (unsigned)SY - 1u || (unsigned)k >= (unsigned)SZ - 1u)
                continue;
            unsigned *R = mine + (i * SY + l) * SZ + k;
            const double wx[2] = {mq * (1.0 - ax), mq * ax}, wy[2] = {1.0 - ay, ay}, wz[2] = {1.0 - az, az};
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const double wxy = wx[b >> 1] * wy[b & 1];
                unsigned *r = R + ((b >> 1) * SY + (b & 1)) * SZ;
                if (magic) {
                    shared_add_rounded(r, r + nn, fma(wxy, wz[0], kRound));
                    shared_add_rounded(r + 1, r + 1 + nn, fma(wxy, wz[1], kRound));
                } else {
                    shared_add64(r, r + nn, __double2ll_rn(wxy * wz[0]));
                    shared_add64(r + 1, r + 1 + nn, __double2ll_rn(wxy * wz[1]));
                }
            }
        }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nn; idx += blockDim.x) {
        long long v = 0;
        for (int q = 0; q < copies; q++)
            v += (long long)(((unsigned long long)sR[q * stride + nn + idx] << 32) | sR[q * stride + idx]);
        if (v == 0) continue;
        const int c = idx % SZ, b = (idx / SZ) % SY, a = idx / (SZ * SY);
        if (i0 + a < g.NX && l0 + b < g.NY && k0 + c < g.NZ) atomicAdd(&rho[g.node(i0 + a, l0 + b, k0 + c)], (double)v * sQ);
    }
}

// periodic fold of rho along one axis, on every line of that axis
__global__ void k_rho_fold(Grid g, double *rho, int dir) {
    const int A = dir == 0 ? g.NY : g.NX;
    const int B = dir == 2 ? g.NY : g.NZ;
    const int n = dir == 0 ? g.nx : (dir == 1 ? g.ny : g.nz);
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= A * B) return;
    const int a = idx / B, b = idx % B;
    size_t base, stride;
    if (dir == 0) { base = (size_t)a * g.pz + b; stride = (size_t)g.NY * g.pz; }
    else if (dir == 1) { base = (size_t)a * g.NY * g.pz + b; stride = g.pz; }
    else { base = ((size_t)a * g.NY + b) * g.pz; stride = 1; }
    double *r = rho + base;
    r[(size_t)n * stride] += r[0];
    r[stride] += r[(size_t)(n + 1) * stride];
    r[0] = r[(size_t)n * stride];
    r[(size_t)(n + 1) * stride] = r[stride];
}

// G = div E - rho on the interior nodes (0 on the ghosts); optional baseline
// copy; reductions into red[0] max |G - G0|, red[1] max |rho|, red[2] sum (G - G0)^2,
// red[3] max |G0| (non-negative doubles compared through their bit patterns)
// (a block walks over many nodes and reduces once: one atomic per warp on the
// same four addresses took 1.65 ms of a 512x128x128 call, this takes 0.27).  The
// maxima are taken of the bit patterns: a NaN is above every number and stays.
__device__ __forceinline__ unsigned long long max_bits(unsigned long long m, unsigned long long v) { return v > m ? v : m; }
__device__ __forceinline__ unsigned long long abs_bits(double v) {
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}
template <typename T>
__global__ void k_gauss(Grid g, const T *__restrict__ Ex, const T *__restrict__ Ey, const T *__restrict__ Ez,
                        const double *__restrict__ rho, double *G, double *G0, int set_baseline, double *red) {
    __shared__ unsigned long long part[3][8];
    __shared__ double part2[8];
    unsigned long long m[3] = {0ull, 0ull, 0ull};  // |G - G0|, |rho|, |G0|
    double d2 = 0.0;
    const size_t sx = (size_t)g.NY * g.pz, sy = g.pz;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rows = g.NX * g.NY, stride = gridDim.x * (blockDim.x >> 5);
    for (int row = blockIdx.x * (blockDim.x >> 5) + warp; row < rows; row += stride) {
        const int i = row / g.NY, l = row - i * g.NY;
        const bool inner = i >= 1 && i <= g.nx && l >= 1 && l <= g.ny;
        for (int k = lane; k < g.NZ; k += 32) {
            const size_t n = g.node(i, l, k);
            double v = 0.0;
            if (inner && k >= 1 && k <= g.nz) {
                v = ((double)Ex[n] - (double)Ex[n - sx]) / g.hx + ((double)Ey[n] - (double)Ey[n - sy]) / g.hy +
                    ((double)Ez[n] - (double)Ez[n - 1]) / g.hz - rho[n];
                m[1] = max_bits(m[1], abs_bits(rho[n]));
            }
            if (G) G[n] = v;
            if (set_baseline) G0[n] = v;
            const double base = set_baseline ? v : G0[n];
            m[0] = max_bits(m[0], abs_bits(v - base));
            d2 += (v - base) * (v - base);
            m[2] = max_bits(m[2], abs_bits(base));
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int q = 0; q < 3; q++) m[q] = max_bits(m[q], __shfl_down_sync(0xffffffffu, m[q], o));
        d2 += __shfl_down_sync(0xffffffffu, d2, o);
    }
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 3; q++) part[q][warp] = m[q];
        part2[warp] = d2;
    }
    __syncthreads();
    const int nw = blockDim.x >> 5;
    if (threadIdx.x < 3) {
        unsigned long long v = 0ull;
        for (int w = 0; w < nw; w++) v = max_bits(v, part[threadIdx.x][w]);
        atomicMax((unsigned long long *)&red[threadIdx.x == 2 ? 3 : threadIdx.x], v);
    } else if (threadIdx.x == 3) {
        double v = 0.0;
        for (int w = 0; w < nw; w++) v += part2[w];
        atomicAdd(&red[2], v);
    }
}

// total mechanical momentum per species, sum over particles of (m/q_m) p, in
// FP64: a block walks over shares of tiles of one species, out[3 s + a] (one
// atomic per block: a block per tile and species spent a c2 call, 3.1 ms, on
// 400k atomics to nine addresses and single loads in flight; now 2.2 ms)
__global__ void k_momentum(StepParams P, int shares, double *out) {
    __shared__ double red[3][32];
    const SpeciesView &S = P.sp[blockIdx.y];
    const double M = S.m / S.q_m;
    double acc[3] = {0.0, 0.0, 0.0};
    bool any = false;
    for (int u = blockIdx.x; u < P.g.ntiles * shares; u += gridDim.x) {
        const int t = u / shares, q = u - t * shares;
        const long long n = S.tile_count[t];
        const int filled = shares_filled(n, shares);
        if (q >= filled) continue;
        any = true;
        const int start = S.tile_start[t], jend = (int)(n * (q + 1) / filled);
        for (int j = (int)(n * q / filled) + threadIdx.x; j < jend; j += 4 * blockDim.x) {
            double p[4][3];
            load_momenta4(P.mixed, S, start, j, jend, p);
#pragma unroll
            for (int v = 0; v < 4; v++) {
                acc[0] += M * p[v][0]; acc[1] += M * p[v][1]; acc[2] += M * p[v][2];
            }
        }
    }
    if (!any) return;  // the whole block
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int a = 0; a < 3; a++) {
        double v = acc[a];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[a][w] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double tot = 0.0;
        for (int i = 0; i < nw; i++) tot += red[threadIdx.x][i];
        atomicAdd(&out[3 * blockIdx.y + threadIdx.x], tot);
    }
}

}  // namespace

cudaError_t momentum(const StepParams &p, double *out, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(out, 0, 3 * p.nsp * sizeof(double), s);
    if (e != cudaSuccess) return e;
    const int shares = tile_shares(p, p.nsp);
    k_momentum<<<dim3(std::min(p.g.ntiles * shares, 8 * kSMs), p.nsp), 256, 0, s>>>(p, shares, out);
    return cudaGetLastError();
}

cudaError_t charge_density(const StepParams &p, double *rho, cudaStream_t s) {
    const Grid &g = p.g;
    cudaError_t e = cudaMemsetAsync(rho, 0, g.nodes_pitched() * sizeof(double), s);
    if (e != cudaSuccess) return e;
    const size_t box = rho_stride((g.tx + 2) * (g.ty + 2) * (g.tz + 2)) * sizeof(unsigned);
    int copies = kRhoCopies;
    while (copies > 1 && copies * box > (size_t)kRhoBytes) copies /= 2;
    const size_t smem = copies * box;
    // fixed dimensions for the automatic tiles of most grids, else runtime
    auto *k = p.mixed ? (g.tx == 6 && g.ty == 4 && g.tz == 8 ? k_charge_tile<true, 6, 4, 8> : k_charge_tile<true, 0, 0, 0>)
                      : (g.tx == 8 && g.ty == 4 && g.tz == 8 ? k_charge_tile<false, 8, 4, 8> : k_charge_tile<false, 0, 0, 0>);
    if (smem > 48 * 1024) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    k<<<dim3(g.ntiles, tile_shares(p, 1)), 256, smem, s>>>(p, copies, rho);
    for (int dir = 0; dir < 3; dir++) {
        const int A = dir == 0 ? g.NY : g.NX;
        const int B = dir == 2 ? g.NY : g.NZ;
        k_rho_fold<<<(A * B + 127) / 128, 128, 0, s>>>(g, rho, dir);
    }
    return cudaGetLastError();
}

cudaError_t gauss_residual(const Grid &g, int mixed, const void *const E[3], const double *rho, double *G, double *G0,
                           int set_baseline, double *red, cudaStream_t s) {
    const int bx = 256, grid = std::min((g.NX * g.NY + 7) / 8, 8 * kSMs);
    if (mixed)
        k_gauss<float><<<grid, bx, 0, s>>>(g, (const float *)E[0], (const float *)E[1], (const float *)E[2], rho, G,
                                           G0, set_baseline, red);
    else
        k_gauss<double><<<grid, bx, 0, s>>>(g, (const double *)E[0], (const double *)E[1], (const double *)E[2], rho,
                                            G, G0, set_baseline, red);
    return cudaGetLastError();
}

}  // namespace pic

// ------------------------------------------------------------------ C ABI --
using namespace pic;
using namespace pic_host;

namespace {
int ensure_diag(pic_handle *h) {
    const size_t bytes = h->g.nodes_pitched() * sizeof(double);
    if (!h->rho) {  // all three or none
        double *d[3] = {nullptr, nullptr, nullptr};
        cudaError_t e = cudaSuccess;
        for (int a = 0; a < 3 && e == cudaSuccess; a++) e = dev_alloc(h, (void **)&d[a], bytes);
        if (e == cudaSuccess) e = cudaMemsetAsync(d[2], 0, bytes, h->stream);
        if (e != cudaSuccess) {
            for (double *p : d)
                if (p) dev_free(h, p);
            return cuda_err(h, e, "alloc the charge diagnostic");
        }
        h->rho = d[0]; h->gauss = d[1]; h->gauss0 = d[2];
        h->gauss_has_base = 0;
    }
    return PIC_OK;
}

int compute_rho(pic_handle *h) {
    int rc = need_particles(h);
    if (rc) return rc;
    if ((rc = ensure_diag(h))) return rc;
    StepParams p = make_params(h);
    CK(charge_density(p, h->rho, h->stream), "charge density");
    return PIC_OK;
}

int run_gauss(pic_handle *h, int set_baseline, double *red4) {
    int rc = compute_rho(h);
    if (rc) return rc;
    const void *E[3] = {h->f[PIC_EX], h->f[PIC_EY], h->f[PIC_EZ]};
    double *red = h->dred + 4;  // the first word counts the blocks of field_energy
    CK(cudaMemsetAsync(red, 0, 4 * sizeof(double), h->stream), "memset");
    CK(gauss_residual(h->g, h->mixed, E, h->rho, h->gauss, h->gauss0, set_baseline, red, h->stream), "gauss");
    if (set_baseline) h->gauss_has_base = 1;
    if (red4) {
        CK(cudaMemcpyAsync(h->hred, red, 4 * sizeof(double), cudaMemcpyDeviceToHost, h->stream), "D2H");
        CK(cudaStreamSynchronize(h->stream), "sync");
        for (int i = 0; i < 4; i++) red4[i] = h->hred[i];
    }
    return PIC_OK;
}
}  // namespace

extern "C" {

int pic_charge_density(pic_handle *h, double *rho_host) {
    if (!h) return PIC_ERR_ARG;
    int rc = set_device(h);
    if (rc) return rc;
    if ((rc = compute_rho(h))) return rc;
    if (rho_host) {
        CK(pitched_to_dense(h->g, h->rho, 0, h->dense, h->stream), "field layout");
        CK(cudaMemcpyAsync(rho_host, h->dense, h->g.nodes_ref() * sizeof(double), cudaMemcpyDeviceToHost, h->stream),
           "D2H rho");
    }
    CK(cudaStreamSynchronize(h->stream), "sync");
    return PIC_OK;
}

int pic_gauss_residual(pic_handle *h, double *g_host) {
    if (!h) return PIC_ERR_ARG;
    int rc = set_device(h);
    if (rc) return rc;
    if ((rc = run_gauss(h, 0, nullptr))) return rc;
    if (g_host) {
        CK(pitched_to_dense(h->g, h->gauss, 0, h->dense, h->stream), "field layout");
        CK(cudaMemcpyAsync(g_host, h->dense, h->g.nodes_ref() * sizeof(double), cudaMemcpyDeviceToHost, h->stream),
           "D2H residual");
    }
    CK(cudaStreamSynchronize(h->stream), "sync");
    return PIC_OK;
}

int pic_momentum(pic_handle *h, double *out) {
    if (!h || !out) return PIC_ERR_ARG;
    int rc = set_device(h);
    if (rc) return rc;
    if ((rc = need_particles(h))) return rc;
    if ((rc = ensure_diag(h))) return rc;
    StepParams p = make_params(h);
    // the rho array is free scratch between diagnostic calls
    CK(momentum(p, h->rho, h->stream), "momentum");
    CK(cudaMemcpyAsync(out, h->rho, 3 * p.nsp * sizeof(double), cudaMemcpyDeviceToHost, h->stream), "D2H momentum");
    CK(cudaStreamSynchronize(h->stream), "sync");
    return PIC_OK;
}

int pic_gauss_check(pic_handle *h, int set_baseline, double *out4) {
    if (!h || !out4) return PIC_ERR_ARG;
    int rc = set_device(h);
    if (rc) return rc;
    if (!set_baseline && !(h->rho && h->gauss_has_base))
        return set_err(h, PIC_ERR_ARG, "pic_gauss_check: no baseline yet (call it with set_baseline = 1 first)");
    double red[4];
    if ((rc = run_gauss(h, set_baseline, red))) return rc;
    int64_t nodes = (int64_t)h->g.nx * h->g.ny * h->g.nz;
    out4[0] = red[0];
    out4[1] = red[1];
    out4[2] = sqrt(red[2] / (double)nodes);
    out4[3] = red[3];
    return PIC_OK;
}

}  // extern "C"
