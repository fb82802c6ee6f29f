// FP64 arithmetic shared by the plain form's push (pic_plain.cu) and the
// fixed-order push of its differentiable run (pic_adjoint.cu).
//
// Which operations keep the reference's bits and which do not:
//   - every quotient that an index comes from ((x - x0) / h, x / h) and every
//     truncation is the reference's, bit for bit, by cheaper operations;
//   - sums of products whose value is continuous (the interpolation, the Boris
//     rotation, the deposit's weights) use fused multiply-adds, one rounding
//     where the reference has two;
//   - 1 / sqrt(v) is rsqrt(v): measured on a B200 within 0.51 ulp for v in [1, 1e12],
//     where the two operations are within 1.5.
// Both translation units are compiled with -fmad=false: a product and a sum
// are fused only where fma() is written.
#pragma once
#include <cuda_runtime.h>
#include "pic_internal.cuh"

namespace pic {

// a / h correctly rounded, rh = 1 / h correctly rounded (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", 1990: with a
// correctly rounded reciprocal and a faithful quotient, one exact remainder
// step gives the correctly rounded quotient; the first step here makes the
// quotient faithful).  Five operations and no branch; a division by a variable
// costs about fifteen and a range check.
__device__ __forceinline__ double div_by(double a, double h, double rh) {
    double q = a * rh;
    q = fma(fma(-q, h, a), rh, q);
    return fma(fma(-q, h, a), rh, q);
}

// (int)t and t rounded down for 0 <= t < 2^32: adding 2^52 rounded down leaves
// the integer part in the low word.  Conversions between FP64 and integers run
// at a quarter of the FP64 add rate.  For t < 0, t >= 2^32 or NaN trunc_checked's
// exact is false and i no index.  floor_pos does not tell: the taps it serves come
// from a particle that lies in its box, u + 1 below 2^32, and a negative t gives a
// negative index, which the callers' range checks report.
__device__ __forceinline__ double floor_pos(double t, int &i) {
    const double m = __dadd_rd(t, 0x1p52);
    i = __double2loint(m);
    return m - 0x1p52;
}
__device__ __forceinline__ int trunc_checked(double t, bool &exact) {
    const double m = __dadd_rd(t, 0x1p52);
    exact = exact && __double2hiint(m) == 0x43300000;
    return __double2loint(m);
}

// One axis of Cell::GetField (cell.h:1257-1290, InverseKernel 1010-1047) and of
// CurrentToMesh's start class (getCellNumberCenterCurrent, cell.h:577-578):
// tap indices of the node- and the centre-staggered components, the integer
// parts of their lower weights, the weights, and the cell-centre index
struct AxisTaps {
    int tn, tc, nI, cI, i1;
    double wn, wc;
};
__device__ __forceinline__ void axis_taps(double x, double x0, double h, double rh, AxisTaps &T) {
    const double u = div_by(x - x0, h, rh), g = div_by(x, h, rh);
    floor_pos(u + 1.0, T.tn);
    T.tn += 1;
    floor_pos((u + 1.0) + 1.5, T.tc);
    floor_pos((u + 1.5) + 1, T.i1);
    T.wn = floor_pos(g + 1.0, T.nI) - g;
    T.wc = floor_pos(g + 1.5, T.cI) - 0.5 - g;
}

// Interpolate3D (cell.h:1054-1153) of the eight taps at A, A + dx, ...; w =
// lower weights, v = upper
__device__ __forceinline__ double trilinear(const double *__restrict__ A, int dx, int dy, double wx, double vx,
                                            double wy, double vy, double wz, double vz) {
    const double a00 = fma(vz, A[1], wz * A[0]), a01 = fma(vz, A[dy + 1], wz * A[dy]);
    const double a10 = fma(vz, A[dx + 1], wz * A[dx]), a11 = fma(vz, A[dx + dy + 1], wz * A[dx + dy]);
    return fma(vx, fma(vy, a11, wy * a10), wx * fma(vy, a01, wy * a00));
}

// Reflect, cell.h:1427-1478 (the reference sums three products with 0 or 1)
__device__ __forceinline__ double reflect_plain(double x, double xm) {
    return x > xm ? x - xm : (x < 0.0 ? xm + x : (x == xm ? 0.0 : x));
}

// Particle::Move, particle.h:65-202, with the intermediates its transpose needs:
// u after the first half kick, b, s = u + u x b, up the rotated momentum, pp the
// new one, g1 and g2 the two 1 / gamma, p2 = pp^2
struct BorisPlain {
    double u[3], g1, ps, b[3], s[3], isd, up[3], pp[3], p2, g2;
};
__device__ __forceinline__ void boris_plain(double tau1, const double F[6], const double p[3], BorisPlain &B) {
    const double pu = fma(tau1, F[0], p[0]), pv = fma(tau1, F[1], p[1]), pw = fma(tau1, F[2], p[2]);
    B.u[0] = pu; B.u[1] = pv; B.u[2] = pw;
    B.g1 = rsqrt(fma(pu, pu, fma(pv, pv, fma(pw, pw, 1.0))));
    B.ps = tau1 * B.g1;
    const double bx = B.ps * F[3], by = B.ps * F[4], bz = B.ps * F[5];
    B.b[0] = bx; B.b[1] = by; B.b[2] = bz;
    const double su = fma(pv, bz, fma(-pw, by, pu)), sv = fma(pw, bx, fma(-pu, bz, pv)),
                 sw = fma(pu, by, fma(-pv, bx, pw));
    B.s[0] = su; B.s[1] = sv; B.s[2] = sw;
    // the rotation (I + b b^T + [b]x) s / (1 + b^2)
    B.isd = 1.0 / fma(bx, bx, fma(by, by, fma(bz, bz, 1.0)));
    const double bs = fma(bx, su, fma(by, sv, bz * sw));
    B.up[0] = fma(bx, bs, fma(bz, sv, fma(-by, sw, su)));
    B.up[1] = fma(by, bs, fma(bx, sw, fma(-bz, su, sv)));
    B.up[2] = fma(bz, bs, fma(by, su, fma(-bx, sv, sw)));
#pragma unroll
    for (int d = 0; d < 3; d++) {
        B.pp[d] = fma(B.up[d], B.isd, tau1 * F[d]);
        B.up[d] *= B.isd;
    }
    B.p2 = fma(B.pp[0], B.pp[0], fma(B.pp[1], B.pp[1], B.pp[2] * B.pp[2]));
    B.g2 = rsqrt(B.p2 + 1.0);
}
// p and the new momentum; returns 1 / gamma of the new momentum, p2 its square
__device__ __forceinline__ double boris_move(double tau1, const double F[6], double p[3], double &p2) {
    BorisPlain B;
    boris_plain(tau1, F, p, B);
#pragma unroll
    for (int d = 0; d < 3; d++) p[d] = B.pp[d];
    p2 = B.p2;
    return B.g2;
}

// CurrentToMesh's relay point x2 (cell.h:1338-1403) of a step xo -> xn whose
// cell-centre indices are i1 and i2; returns the crossing code m = 4|di| + 2|dl|
// + |dk| (1..7: two segments) and the ratio sr of the straight path
__device__ __forceinline__ int relay_point(const double xo[3], const double xn[3], const double o3[3],
                                           const double h3[3], const int i1[3], const int i2[3], double x2[3],
                                           double &sr) {
    x2[0] = x2[1] = x2[2] = 0.0;
    sr = 0.0;
    const int m = 4 * abs(i2[0] - i1[0]) + 2 * abs(i2[1] - i1[1]) + abs(i2[2] - i1[2]);
#define AVG(d) (h3[d] * (((double)i1[d] + (double)i2[d]) * 0.5 - 2.0) + o3[d])
#define RATIO(d) ((x2[d] - xo[d]) / (xn[d] - xo[d]))
#define PROD(d) ((x2[d] - xo[d]) * (xn[d] - xo[d]))
#define RBX(d) (xo[d] + (xn[d] - xo[d]) * sr)
#define SQ(v) ((v) * (v))
    switch (m) {
        case 1: x2[2] = AVG(2); sr = RATIO(2); x2[0] = RBX(0); x2[1] = RBX(1); break;
        case 2: x2[1] = AVG(1); sr = RATIO(1); x2[0] = RBX(0); x2[2] = RBX(2); break;
        case 3:
            x2[1] = AVG(1); x2[2] = AVG(2);
            sr = (PROD(2) + PROD(1)) / (SQ(xn[2] - xo[2]) + SQ(xn[1] - xo[1]));
            x2[0] = RBX(0);
            break;
        case 4: x2[0] = AVG(0); sr = RATIO(0); x2[1] = RBX(1); x2[2] = RBX(2); break;
        case 5:
            x2[0] = AVG(0); x2[2] = AVG(2);
            sr = (PROD(2) + PROD(0)) / (SQ(xn[2] - xo[2]) + SQ(xn[0] - xo[0]));
            x2[1] = RBX(1);
            break;
        case 6:
            x2[0] = AVG(0); x2[1] = AVG(1);
            sr = (PROD(1) + PROD(0)) / (SQ(xn[1] - xo[1]) + SQ(xn[0] - xo[0]));
            x2[2] = RBX(2);
            break;
        case 7: x2[0] = AVG(0); x2[1] = AVG(1); x2[2] = AVG(2); break;
        default: break;
    }
#undef AVG
#undef RATIO
#undef PROD
#undef RBX
#undef SQ
    return m;
}

// pqr, cell.h:1511-1693, accumulating into the tile J (shared memory).  The
// reference's divisions by 12 and by tau*h*h are multiplications by their
// reciprocals (rc[d] = 1 / (tau * h_e * h_f) times the charge weight and the
// inverse quantum, precomputed): the products feed only the current's
// magnitude, never an index, and differ from the quotients by an ulp.  sJ: 3 nn
// low words, 3 nn high words, then the remainders (LO32: 3 nn int32, fx_put_lo32;
// else 3 nn low and 3 nn high words, fx_put2).  ex, ey: node strides.
template <bool LO32>
__device__ __forceinline__ void pqr_plain(unsigned *__restrict__ sJ, double lo_scale, int nn, int ex, int ey,
                                          int bi, int bl, int bk, const int iv[3], const double x[3],
                                          const double x1[3], double hx, double hy, double hz, const double rc[3],
                                          double x0, double y0, double z0, unsigned &bad) {
    const double dx = (0.50 * (x[0] + x1[0]) - hx * ((double)iv[0] - 2.50) - x0);
    const double dy = (0.50 * (x[1] + x1[1]) - hy * ((double)iv[1] - 2.50) - y0);
    const double dz = (0.50 * (x[2] + x1[2]) - hz * ((double)iv[2] - 2.50) - z0);
    const double dx1 = hx - dx, dy1 = hy - dy, dz1 = hz - dz;
    double su = x1[0] - x[0], sv = x1[1] - x[1], sw = x1[2] - x[2];
    constexpr double kTwelfth = 1.0 / 12.0;
    const double s1 = sv * sw * kTwelfth, s2 = su * sw * kTwelfth, s3 = su * sv * kTwelfth;
    su = su * rc[0];
    sv = sv * rc[1];
    sw = sw * rc[2];
    if (iv[0] < 2 || iv[0] > 3 || iv[1] < 2 || iv[1] > 3 || iv[2] < 2 || iv[2] > 3) { bad |= ST_STENCIL; return; }
    const int n = (bi + iv[0]) * ex + (bl + iv[1]) * ey + (bk + iv[2]), ez = 1;
    // component c, node offset o from n, contribution v in quanta
    auto add = [&](int c, int o, double v) {
        unsigned *w = sJ + c * nn + n + o;
        if (LO32) fx_put_lo32(w, 3 * nn, v, lo_scale);
        else fx_put2(w, 3 * nn, v);
    };
    add(0, 0, su * fma(dy1, dz1, s1));
    add(0, ez, su * fma(dy1, dz, -s1));
    add(0, ey, su * fma(dy, dz1, -s1));
    add(0, ey + ez, su * fma(dy, dz, s1));
    add(1, 0, sv * fma(dx1, dz1, s2));
    add(1, ez, sv * fma(dx1, dz, -s2));
    add(1, ex, sv * fma(dx, dz1, -s2));
    add(1, ex + ez, sv * fma(dx, dz, s2));
    add(2, 0, sw * fma(dx1, dy1, s3));
    add(2, ey, sw * fma(dx1, dy, -s3));
    add(2, ex, sw * fma(dx, dy1, -s3));
    add(2, ex + ey, sw * fma(dx, dy, s3));
}

}  // namespace pic
