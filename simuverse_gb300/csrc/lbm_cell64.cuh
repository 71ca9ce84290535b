// lbm_cell64.cuh -- BGK of one fluid cell in FP64.  GB300 runs 0.53 T FP64 operations a second
// (measured), so a step is bound by how many a cell takes: the general collision's 80 made a step of a
// 2048^2 channel take 0.636 ms, of which its memory traffic needs 0.09 ms.  Here there are 59, and the
// step takes 0.492 ms, 95 % of that rate:
//   * rho u u is taken as the momentum times the velocity, so that no product with rho is left;
//   * omega is folded into the weights and the products of constants come with the launch;
//   * opposite populations are relaxed as half their sum and half their difference;
//   * the reciprocal is the hardware's approximation r (20 bits) and one step of the third-order
//     Newton-Schulz iteration, r (1 + e + e^2) with e = 1 - rho r: what is left, e^3, is below 2^-58.
#pragma once

#include "lbm_common.cuh"

namespace lbm {

// The constants close without a rounding, so that no step gains or loses mass or momentum by them:
// w is a multiple of omega's last place, which makes 5 w and w0 = omega - 5 w exact; 2 w3 lies within a
// factor of two of omega, which makes omega - 2 w3 exact.
struct Bgk64 {
    double omega;
    double om1, half1;     // 1 - omega and half of it
    double w0, w, wd;      // omega times the weights: at rest, on the axes, on the diagonals
    double q, qd;          // 4.5 omega times the weights of the axes and the diagonals
    double w3, w3d;        // 3 omega times them
    explicit Bgk64(double relax) : omega(relax), om1(1.0 - relax), half1(0.5 * om1) {
        w = (omega / 9.0 + omega) - omega;
        wd = 0.25 * w;
        w0 = omega - 5.0 * w;
        q = 0.5 * omega;
        qd = 0.125 * omega;
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
    const double s13 = d[1] + d[3], s24 = d[2] + d[4], s57 = d[5] + d[7], s68 = d[6] + d[8];
    const double d13 = d[1] - d[3], d42 = d[4] - d[2], d57 = d[5] - d[7], d86 = d[8] - d[6];
    const double drho = d[0] + ((s13 + s24) + (s57 + s68));
    const double jx = d13 + (d57 + d86), jy = d42 + (d86 - d57);
    rho = 1.0 + drho;
    const double inv = recip64(rho);
    ux = jx * inv;
    uy = jy * inv;
    const double xx = jx * ux, yy = jy * uy, xy = jx * uy, uu = xx + yy;
    const double t0 = __fma_rn(-1.5, uu, drho);  // what all equilibrium deviations share, over their weight
    const double a = k.w * t0, ad = k.wd * t0;
    const auto pair = [&](int j, int i, double even, double odd) {
        o[j] = even + odd;
        o[i] = even - odd;
    };
    pair(1, 3, __fma_rn(k.half1, s13, __fma_rn(k.q, xx, a)), __fma_rn(k.half1, d13, k.w3 * jx));
    pair(4, 2, __fma_rn(k.half1, s24, __fma_rn(k.q, yy, a)), __fma_rn(k.half1, d42, k.w3 * jy));
    pair(8, 6, __fma_rn(k.half1, s68, __fma_rn(k.qd, __fma_rn(2.0, xy, uu), ad)),
         __fma_rn(k.half1, d86, k.w3d * (jx + jy)));
    pair(5, 7, __fma_rn(k.half1, s57, __fma_rn(k.qd, __fma_rn(-2.0, xy, uu), ad)),
         __fma_rn(k.half1, d57, k.w3d * (jx - jy)));
    o[0] = __fma_rn(k.om1, d[0], k.w0 * t0);
}

}  // namespace lbm
