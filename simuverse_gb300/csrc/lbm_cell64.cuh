// lbm_cell64.cuh -- BGK of one fluid cell in FP64.  GB300 runs 0.53 T FP64 operations a second
// (measured), so a step is bound by how many a cell takes: the general collision's 80 made a step of a
// 2048^2 channel take 0.636 ms, of which its memory traffic needs 0.09 ms.  Here there are 60, and the
// step takes 0.499 ms, 95 % of that rate:
//   * rho u u is taken as the momentum times the velocity, so that no product with rho is left;
//   * omega is folded into the weights and the products of constants come with the launch;
//   * opposite populations share the even part of their equilibrium, and each takes the odd part, with its sign,
//     and its own relaxation by one fused multiply-add;
//   * the reciprocal is the hardware's approximation r (20 bits) and one step of the third-order
//     Newton-Schulz iteration, r (1 + e + e^2) with e = 1 - rho r: what is left, e^3, is below 2^-58.
// Precision.  The rest population closes the sum of what leaves, as in the general collision, so that the rounding of
// the weights moves no mass; 2 w3 lies within a factor of two of omega, which makes omega - 2 w3 exact and the
// momentum close.  Against arithmetic of more than 64 bits of significand, over relaxation times of 0.505 to 2.7 and
// densities that vary by 0.3 to 30 %, the error of a collision is 0.80 to 0.99 times the general one's (RMS), that of a
// cell's mass 0.99 to 1.01 times.  (59 operations, with weights rounded to omega's last place so that they close by
// themselves and a rest population of its own, took 0.492 ms a step, and up to 7 times the general error.)
#pragma once

#include "lbm_common.cuh"

namespace lbm {

struct Bgk64 {
    double omega;
    double om1;      // 1 - omega
    double w, wd;    // omega times the weights of the axes and the diagonals
    double c, cd;    // what u.u adds to the even part beside (e.u)^2: -1.5 w, and on the diagonals 4.5 wd - 1.5 wd
    double q, qd;    // 4.5 omega times the axes' weight; twice that of the diagonals for the mixed term
    double w3, w3d;  // 3 omega times the weights
    explicit Bgk64(double relax) : omega(relax), om1(1.0 - relax) {
        w = omega / 9.0;
        wd = 0.25 * w;
        c = -omega / 6.0;
        cd = -0.5 * c;
        q = 0.5 * omega;
        qd = 0.25 * omega;
        w3 = omega / 3.0;
        w3d = 0.25 * (omega - 2.0 * w3);
    }
};

__device__ __forceinline__ double recip64(double a) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a));
    const double e = __fma_rn(-a, r, 1.0);
    return __fma_rn(r, __fma_rn(e, e, e), r);
}

__device__ __forceinline__ void bgk64(const double (&d)[9], const Bgk64& k, double (&o)[9], double& rho, double& ux,
                                      double& uy) {
    const double d57 = d[5] - d[7], d86 = d[8] - d[6];
    const double drho = d[0] + (((d[1] + d[3]) + (d[2] + d[4])) + ((d[5] + d[7]) + (d[6] + d[8])));
    const double jx = (d[1] - d[3]) + (d57 + d86), jy = (d[4] - d[2]) + (d86 - d57);
    rho = 1.0 + drho;
    const double inv = recip64(rho);
    ux = jx * inv;
    uy = jy * inv;
    const double xx = jx * ux, yy = jy * uy, xy = jx * uy, uu = xx + yy;
    const double a = __fma_rn(k.w, drho, k.c * uu), b = __fma_rn(k.wd, drho, k.cd * uu);
    const auto pair = [&](int j, int i, double even, double w, double e) {
        o[j] = __fma_rn(k.om1, d[j], __fma_rn(w, e, even));
        o[i] = __fma_rn(k.om1, d[i], __fma_rn(-w, e, even));
    };
    pair(1, 3, __fma_rn(k.q, xx, a), k.w3, jx);
    pair(4, 2, __fma_rn(k.q, yy, a), k.w3, jy);
    pair(8, 6, __fma_rn(k.qd, xy, b), k.w3d, jx + jy);
    pair(5, 7, __fma_rn(-k.qd, xy, b), k.w3d, jx - jy);
    o[0] = drho - (((o[1] + o[3]) + (o[2] + o[4])) + ((o[5] + o[7]) + (o[6] + o[8])));
}

}  // namespace lbm
