// FP64 arithmetic shared by the plain form's push (pic_plain.cu) and the
// fixed-order push of its differentiable run (pic_adjoint.cu).
//
// Which operations keep the reference's bits and which do not:
//   - every quotient that an index comes from ((x - x0) / h, x / h) and every
//     truncation is the reference's, bit for bit, by cheaper operations;
//   - sums of products whose value is continuous (the interpolation, the Boris
//     rotation, the deposit's weights) use fused multiply-adds, one rounding
//     where the reference has two;
//   - 1 / sqrt(v) is rsqrt(v), within an ulp like the two operations.
// Both translation units are compiled with -fmad=false: a product and a sum
// are fused only where fma() is written.
#pragma once
#include <cuda_runtime.h>

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
// at a quarter of the FP64 add rate.  For t < 0 (or t >= 2^32, or NaN) exact
// is false and i is not in any index range that its caller then uses.
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
// tap indices of the node- and the centre-staggered components, their lower
// weights, and the cell-centre index
struct AxisTaps {
    int tn, tc, i1;
    double wn, wc;
};
__device__ __forceinline__ void axis_taps(double x, double x0, double h, double rh, AxisTaps &T) {
    const double u = div_by(x - x0, h, rh), g = div_by(x, h, rh);
    floor_pos(u + 1.0, T.tn);
    T.tn += 1;
    floor_pos((u + 1.0) + 1.5, T.tc);
    floor_pos((u + 1.5) + 1, T.i1);
    int n;
    T.wn = floor_pos(g + 1.0, n) - g;
    T.wc = floor_pos(g + 1.5, n) - 0.5 - g;
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

// Particle::Move, particle.h:65-202: p and the new momentum; returns 1 / gamma
// of the new momentum, p2 its square
__device__ __forceinline__ double boris_move(double tau1, const double F[6], double p[3], double &p2) {
    double pu = fma(tau1, F[0], p[0]), pv = fma(tau1, F[1], p[1]), pw = fma(tau1, F[2], p[2]);
    const double ps = tau1 * rsqrt(fma(pu, pu, fma(pv, pv, fma(pw, pw, 1.0))));
    const double bx = ps * F[3], by = ps * F[4], bz = ps * F[5];
    const double su = fma(pv, bz, fma(-pw, by, pu)), sv = fma(pw, bx, fma(-pu, bz, pv)),
                 sw = fma(pu, by, fma(-pv, bx, pw));
    // the rotation (I + b b^T + [b]x) s / (1 + b^2)
    const double isd = 1.0 / fma(bx, bx, fma(by, by, fma(bz, bz, 1.0)));
    const double bs = fma(bx, su, fma(by, sv, bz * sw));
    pu = fma(fma(bx, bs, fma(bz, sv, fma(-by, sw, su))), isd, tau1 * F[0]);
    pv = fma(fma(by, bs, fma(bx, sw, fma(-bz, su, sv))), isd, tau1 * F[1]);
    pw = fma(fma(bz, bs, fma(by, su, fma(-bx, sv, sw))), isd, tau1 * F[2]);
    p[0] = pu; p[1] = pv; p[2] = pw;
    p2 = fma(pu, pu, fma(pv, pv, pw * pw));
    return rsqrt(p2 + 1.0);
}

}  // namespace pic
