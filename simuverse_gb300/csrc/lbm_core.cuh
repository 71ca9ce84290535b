// lbm_core.cuh -- the FP32 collision of physics mode written operation by operation, for one cell
// (V = float) or for two cells at once (V = float2).
//
// Every product, sum and fused multiply-add is an explicit round-to-nearest operation, so the
// compiler neither contracts nor reorders anything: all step kernels that use the core (one cell
// per thread, the fused multi-step kernel, the batched forms) give the same bits, and a call of
// n steps gives the same state however the steps are grouped into launches.  The FP32 sequence is the
// one that the compiler had chosen for the plain expressions of phys_collide (which products it fuses
// with which sums was found by comparing candidate sequences with that kernel's results), so states
// and fields are bit for bit those of earlier versions.
//
// float2 maps to the packed FP32x2 instructions.  They run the FP32 pipe at the same lane rate
// as scalar ones (measured on GB300: 39.7 T multiply-adds a second packed, 38.7 T scalar) but
// take half the issue slots, which the fused kernel needs for its loads and stores.  A packed
// instruction reads registers only and negates nothing: signs are kept in constants and in the
// negative reciprocal and velocity.  The assembler of CUDA 13.0 fuses a packed product with a packed sum
// or difference where nothing else uses the product, although both ask for round-to-nearest (seen
// in results; the scalar forms are left alone): no such pair appears below unless the product is exact.
#pragma once

#include "lbm_common.cuh"

namespace lbm {

__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 a, b, r;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "sub.rn.f32x2 r, a, b;\n\tmov.b64 {%0, %1}, r;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

template <class V>
struct VecOf {
    using S = V;
    __host__ __device__ __forceinline__ static V all(S s) { return s; }
};
template <>
struct VecOf<float2> {
    using S = float;
    __host__ __device__ __forceinline__ static float2 all(float s) { return make_float2(s, s); }
};

// The collision's constants as values of V: the relaxation rate, the axis and diagonal weights (times
// 3 as well), literals.
template <class V>
struct BgkConst {
    using S = typename VecOf<V>::S;
    S omega;
    V om, omn, om1, w1, w5, w31, w35, c45, one, mone, m15;
    __host__ __device__ explicit BgkConst(S o)
        : omega(o), om(VecOf<V>::all(o)), omn(VecOf<V>::all(-o)), om1(VecOf<V>::all(S(1) - o)),
          w1(VecOf<V>::all(PW<S>(1))), w5(VecOf<V>::all(PW<S>(5))), w31(VecOf<V>::all(S(3) * PW<S>(1))),
          w35(VecOf<V>::all(S(3) * PW<S>(5))), c45(VecOf<V>::all(S(4.5))), one(VecOf<V>::all(S(1))),
          mone(VecOf<V>::all(S(-1))), m15(VecOf<V>::all(S(-1.5))) {}
};

__device__ __forceinline__ float rcp_approx(float a) {  // within 1 ulp (PTX ISA, rcp.approx)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
// Negative reciprocal -1 / a.  FP32: the hardware approximation and one Newton-Raphson step on its
// residual (the textbook iteration), for densities and equilibria, which are far from the ends of
// the range; on all 2^23 significands it equals the correctly rounded reciprocal.
__device__ __forceinline__ float vrcpn(float a, const BgkConst<float>&) {
    const float r = rcp_approx(-a);
    return __fmaf_rn(r, __fmaf_rn(a, r, 1.0f), r);
}
__device__ __forceinline__ float2 vrcpn(float2 a, const BgkConst<float2>& k) {
    const float2 r = make_float2(rcp_approx(-a.x), rcp_approx(-a.y));
    return __ffma2_rn(r, __ffma2_rn(a, r, k.one), r);
}

// density deviation and momentum of the pulled deviations
template <class V>
__device__ __forceinline__ void core_moments(const V (&d)[9], V& drho, V& jx, V& jy) {
    const V d57 = vsub(d[5], d[7]), d86 = vsub(d[8], d[6]);
    drho = vadd(d[0], vadd(vadd(vadd(d[1], d[3]), vadd(d[2], d[4])), vadd(vadd(d[5], d[7]), vadd(d[6], d[8]))));
    jx = vadd(vsub(d[1], d[3]), vadd(d57, d86));
    jy = vadd(vsub(d[4], d[2]), vsub(d86, d57));
}
// the rest population that closes the mass balance: the outgoing deviations sum to drho up to rounding
template <class V>
__device__ __forceinline__ V core_rest(const V (&o)[9], V drho) {
    return vsub(drho, vadd(vadd(vadd(o[1], o[3]), vadd(o[2], o[4])), vadd(vadd(o[5], o[7]), vadd(o[6], o[8]))));
}

// What BGK and KBC share: density, negative velocity, and per opposite pair (j, inv j) the negative
// velocity component ne and the even part y = drho + rho (4.5 (e.u)^2 - 1.5 u.u) of the equilibrium
// deviation over w.  Pairs in the order 1 / 3, 4 / 2, 8 / 6, 5 / 7.
template <class V>
__device__ __forceinline__ void core_even(const BgkConst<V>& k, V drho, V jx, V jy, V& rho, V& nux, V& nuy, V& nusq,
                                          V (&ne)[4], V (&y)[4]) {
    rho = vadd(drho, k.one);
    const V ninv = vrcpn(rho, k);
    nux = vmul(jx, ninv);
    nuy = vmul(jy, ninv);
    nusq = vmul(vfma(nux, nux, vmul(nuy, nuy)), k.m15);
    ne[0] = nux;
    ne[1] = nuy;
    ne[2] = vadd(nux, nuy);
    ne[3] = vfma(nuy, k.mone, nux);
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = vfma(rho, vfma(vmul(ne[i], k.c45), ne[i], nusq), drho);
}

// BGK of the deviations d on opposite pairs: even part w y, odd part 3 w rho e.u.  Moments come from
// core_moments (plus half the force where one acts); rho and the negative velocity come back.
template <class V>
__device__ __forceinline__ void core_bgk(const V (&d)[9], const BgkConst<V>& k, V drho, V jx, V jy, V (&o)[9], V& rho,
                                         V& nux, V& nuy) {
    constexpr int J[4] = {1, 4, 8, 5};
    V nusq, ne[4], y[4];
    core_even<V>(k, drho, jx, jy, rho, nux, nuy, nusq, ne, y);
    const V r1 = vmul(rho, k.w31), r5 = vmul(rho, k.w35);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const V sym = vmul(vmul(y[i], i < 2 ? k.w1 : k.w5), k.om), nz = vmul(i < 2 ? r1 : r5, ne[i]);
        o[J[i]] = vfma(k.om1, d[J[i]], vfma(k.omn, nz, sym));
        o[INV(J[i])] = vfma(k.om1, d[INV(J[i])], vfma(k.om, nz, sym));
    }
    o[0] = core_rest<V>(o, drho);
}
// Guo's forcing terms (1 - omega / 2) w_j (3 (e - u) + 9 (e.u) e) . F of a cell that a force acts on
template <class S>
__device__ __forceinline__ void core_guo(const BgkConst<S>& k, S ux, S uy, S Fx, S Fy, S drho, S (&o)[9]) {
    const S gf = vfma(S(-0.5), k.omega, S(1));
    const S uF = vfma(ux, Fx, vmul(uy, Fy));
#pragma unroll
    for (int j = 1; j < 9; ++j) {
        const S eF = EX(j) == 0 ? S(EY(j)) * Fy : (EY(j) == 0 ? S(EX(j)) * Fx : vadd(S(EX(j)) * Fx, S(EY(j)) * Fy));
        const S eu = EX(j) == 0 ? S(EY(j)) * uy : (EY(j) == 0 ? S(EX(j)) * ux : vadd(S(EX(j)) * ux, S(EY(j)) * uy));
        o[j] = vfma(vmul(gf, PW<S>(j)), vfma(S(3), vsub(eF, uF), vmul(vmul(S(9), eu), eF)), o[j]);
    }
    o[0] = core_rest<S>(o, drho);
}

// Zou-He velocity inlet on a west face: the unknown populations 1, 5, 8 from the known ones
template <class S>
__device__ __forceinline__ void core_inlet(S (&d)[9], S ux, S uy) {
    const S known = vadd(vadd(vadd(d[0], d[2]), d[4]), vmul(S(2), vadd(vadd(d[3], d[6]), d[7])));
    const S rho = vadd(S(1), known) / vsub(S(1), ux);
    const S rux = vmul(rho, ux), half = vmul(S(0.5), vmul(rho, uy)), sixth = rux / S(6);
    const S d42 = vmul(S(0.5), vsub(d[4], d[2]));
    d[1] = vfma(S(2) / S(3), rux, d[3]);
    d[5] = vsub(vadd(vadd(d[7], d42), sixth), half);
    d[8] = vadd(vadd(vsub(d[6], d42), sixth), half);
}

// zero-gradient outflow anchored at rho = 1: f_j <- f_j / rho
template <class S>
__device__ __forceinline__ void core_outlet(S (&d)[9], const BgkConst<S>& k) {
    S dr = d[0];
#pragma unroll
    for (int j = 1; j < 9; ++j) dr = vadd(dr, d[j]);
    const S inv = -vrcpn(vadd(S(1), dr), k);
#pragma unroll
    for (int j = 0; j < 9; ++j) d[j] = vmul(vfma(-PW<S>(j), dr, d[j]), inv);
}

// entropic KBC (Karlin, Bosch & Chikatamarla 2014) on the natural moments: f = k + s + h with the
// shear part s from N = Pxx - Pyy and Pxy (s = N/4 on the x axis, -N/4 on the y axis, sigma lambda
// Pxy / 4 on the diagonals); f' = f - beta (2 ds + gamma dh), beta = omega / 2 (BGK's shear viscosity),
// gamma = 1/beta - (2 - 1/beta) <ds|dh> / <dh|dh> with <x|y> = sum x_i y_i / feq_i, the stabiliser
// that keeps the entropy production right; gamma = 2 is BGK.
//
// gamma from the negative products nsh = -<ds|dh>, nhh = -<dh|dh> and ib = 1 / beta
__device__ __forceinline__ float kbc_gamma(float nsh, float nhh, float ib) {
    return nhh < -1e-30f ? __fmaf_rn(-(2.0f - ib), nsh / nhh, ib) : 2.0f;
}
__device__ __forceinline__ float2 kbc_gamma(float2 nsh, float2 nhh, float ib) {
    return make_float2(kbc_gamma(nsh.x, nhh.x, ib), kbc_gamma(nsh.y, nhh.y, ib));
}
template <class V>
__device__ __forceinline__ void core_kbc(const V (&d)[9], const BgkConst<V>& k, V drho, V jx, V jy, V (&o)[9], V& rho,
                                         V& nux, V& nuy) {
    using S = typename VecOf<V>::S;
    const auto C = [](S s) { return VecOf<V>::all(s); };
    constexpr int J[4] = {1, 4, 8, 5};
    V nusq, ne[4], y[4], q[9], n[9];
    core_even<V>(k, drho, jx, jy, rho, nux, nuy, nusq, ne, y);
    const V r1 = vmul(rho, k.w31), r5 = vmul(rho, k.w35), r1n = vmul(r1, k.mone), r5n = vmul(r5, k.mone);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const V s = vmul(y[i], i < 2 ? k.w1 : k.w5);
        q[J[i]] = vfma(i < 2 ? r1n : r5n, ne[i], s);
        q[INV(J[i])] = vfma(i < 2 ? r1 : r5, ne[i], s);
    }
    const V t0 = vfma(rho, nusq, drho);
    n[0] = vfma(t0, C(-PW<S>(0)), d[0]);
#pragma unroll
    for (int j = 1; j < 9; ++j) n[j] = vsub(d[j], q[j]);
    // the shear part: +-ds on the axes, +-dp on the diagonals (quarters are exact)
    const V dn = vmul(vsub(vadd(n[1], n[3]), vadd(n[2], n[4])), C(S(0.25)));
    const V dp = vmul(vsub(vadd(n[8], n[6]), vadd(n[5], n[7])), C(S(0.25)));
    const V dnn = vmul(dn, k.mone), dpn = vmul(dp, k.mone);
    V nsh = C(S(0)), nhh = nsh;
#pragma unroll
    for (int j = 0; j < 9; ++j) {  // n becomes the higher-moment part dh = n - ds
        const bool plus = j == 1 || j == 3 || j == 8 || j == 6;
        if (j) n[j] = plus ? vsub(n[j], j <= 4 ? dn : dp) : vadd(n[j], j <= 4 ? dn : dp);
        const V ng = vrcpn(j ? vadd(q[j], C(PW<S>(j))) : vfma(t0, C(PW<S>(0)), C(PW<S>(0))), k);  // -1 / feq
        if (j) nsh = vfma(vmul(plus ? (j <= 4 ? dn : dp) : (j <= 4 ? dnn : dpn), n[j]), ng, nsh);
        nhh = vfma(vmul(n[j], n[j]), ng, nhh);
    }
    const S beta = S(0.5) * k.omega;
    const V gamma = kbc_gamma(nsh, nhh, S(1) / beta), nb = C(-beta), two = C(S(2)), twon = C(S(-2));
#pragma unroll
    for (int j = 1; j < 9; ++j) {
        const bool plus = j == 1 || j == 3 || j == 8 || j == 6;
        o[j] = vfma(nb, vfma(plus ? two : twon, j <= 4 ? dn : dp, vmul(gamma, n[j])), d[j]);
    }
    o[0] = core_rest<V>(o, drho);
}

// the collisions the core implements
__host__ __device__ constexpr bool core_has(int coll) { return coll == LBM_COLLISION_BGK || coll == LBM_COLLISION_KBC; }

template <int COLL, class V>
__device__ __forceinline__ void core_collide(const V (&d)[9], const BgkConst<V>& k, V drho, V jx, V jy, V (&o)[9],
                                             V& rho, V& nux, V& nuy) {
    if constexpr (COLL == LBM_COLLISION_KBC) core_kbc<V>(d, k, drho, jx, jy, o, rho, nux, nuy);
    else core_bgk(d, k, drho, jx, jy, o, rho, nux, nuy);
}

// One cell's boundary rules on the pulled deviations, collision and forcing: the scalar form.
template <class S, int COLL>
__device__ __forceinline__ void core_cell(S (&d)[9], int m, unsigned fl, size_t c, uint16_t* __restrict__ flags,
                                          lbm_lattice_info* __restrict__ info, S omega, S (&o)[9], S& rho, S& ux,
                                          S& uy) {
    const BgkConst<S> k(omega);
    if (m == LBM_INLET) {
        const lbm_lattice_info in = info[c];
        core_inlet<S>(d, S(in.vx), S(in.vy));
    }
    if (m == LBM_OUTLET) core_outlet<S>(d, k);
    S drho, jx, jy, nux, nuy;
    core_moments<S>(d, drho, jx, jy);
    if (m == LBM_EXTERNAL_FORCE) {  // Guo forcing with the reference's block_iter countdown
        lbm_lattice_info in = info[c];
        if (in.block_iter > 0) {
            in.block_iter = in.block_iter - 1;
            if (in.block_iter == 0) {
                in.material = LBM_BULK;
                const unsigned nf = (fl & ~FL_MAT_MASK) | LBM_BULK;
                flags[c] = (uint16_t)(nf | plain_bit(nf));
            }
            info[c] = in;
        }
        const S Fx = S(in.vx), Fy = S(in.vy);
        core_collide<COLL, S>(d, k, drho, vfma(S(0.5), Fx, jx), vfma(S(0.5), Fy, jy), o, rho, nux, nuy);
        core_guo<S>(k, -nux, -nuy, Fx, Fy, drho, o);
    } else {
        core_collide<COLL, S>(d, k, drho, jx, jy, o, rho, nux, nuy);
    }
    ux = -nux;
    uy = -nuy;
}

}  // namespace lbm
