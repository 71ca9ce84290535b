// lbm_march_ref.cuh -- T fused time steps under the reference's rules (contracted arithmetic,
// LBM_ARITH_FAST): the march of lbm_march.cuh with the collision of collide_stream.wgsl:40-87 and the
// walls of boundary.wgsl.
//
// A step hands the population of a fluid cell strictly inside the outer ring that faces a solid
// neighbour to that wall's slot, where the same cell, and no other, finds it in the next step: between
// fused steps it is taken from the cell itself, and the last step stores it in the wall.  Fluid cells
// on the outer ring hand nothing over; what they pull from a wall are slots that no step writes, read
// from the buffer that a single step would read.
//
// The rounding sequence is the one-step kernel's (found like the collision's in lbm_core.cuh), so
// states and fields are those of single steps bit for bit.  The exact arithmetic is not fused: its
// separate products and sums, which the packed instructions do not keep apart, bound it by issue slots.
// Measured on the Poiseuille scene at 8192^2: a frame of two steps 1.58 ms before, 1.07 ms now (126 GLUPS,
// 5.4 TB/s = 80 % of the measured copy rate; three steps per pass 189 GLUPS).  What bounds a frame of two steps:
// memory, with a quarter of the reads done twice at the edges of windows and segments; three steps per pass issue in
// 57 % of the slots at 2.8 warps per scheduler, with DRAM at 4.9 TB/s.
#pragma once

#include "lbm_march.cuh"

namespace lbm {

template <class V>
struct RefConst {
    using S = float;
    float omega;
    V om, om1, w0, w1, w5, one, mone, m15, c45, c3, c3n;
    __host__ __device__ explicit RefConst(float o)
        : omega(o), om(VecOf<V>::all(o)), om1(VecOf<V>::all(1.0f - o)), w0(VecOf<V>::all(REF_W(0))),
          w1(VecOf<V>::all(REF_W(1))), w5(VecOf<V>::all(REF_W(5))), one(VecOf<V>::all(1.0f)),
          mone(VecOf<V>::all(-1.0f)), m15(VecOf<V>::all(-1.5f)), c45(VecOf<V>::all(4.5f)), c3(VecOf<V>::all(3.0f)),
          c3n(VecOf<V>::all(-3.0f)) {}
};

// v limited to [0, top], NaN kept (collide_stream.wgsl:79-83 compares)
__device__ __forceinline__ float ref_limit(float v, float top) {
    float r;
    asm("{\n\t.reg .f32 t;\n\tmax.NaN.f32 t, %1, 0f00000000;\n\tmin.NaN.f32 %0, t, %2;\n\t}" : "=f"(r) : "f"(v), "f"(top));
    return r;
}

enum { ROW_FORCE = 2, ROW_RING = 4 };  // row classes of this mode beside ROW_MIXED
__device__ __forceinline__ bool ref_forced(unsigned f) {
    const int m = (int)(f & FL_MAT_MASK);
    return m == LBM_INLET || m == LBM_EXTERNAL_FORCE;
}
// class of a row, with the directions in which some fluid cell hands its population to a wall
__device__ __forceinline__ int ref_row_class(unsigned fq) {
    if (__all_sync(0xffffffffu, (fq & (FL_PLAIN | FL_PLAIN << 16)) == (FL_PLAIN | FL_PLAIN << 16))) return ROW_PLAIN;
    const unsigned lo = is_solid((int)(fq & FL_MAT_MASK)) ? 0u : fq & 0xffffu;
    const unsigned hi = is_solid((int)((fq >> 16) & FL_MAT_MASK)) ? 0u : fq >> 16;
    const int all = (int)__reduce_or_sync(0xffffffffu, lo | hi);
    const bool force = __any_sync(0xffffffffu, ref_forced(fq & 0xffffu) || ref_forced(fq >> 16));
    return (all & (int)(0x1FEu << FL_DIR_SHIFT)) | ROW_MIXED | (force ? ROW_FORCE : 0) | (all & (int)FL_RING ? ROW_RING : 0);
}

// a forcing cell's velocity (collide_stream.wgsl:55-71; permanent ones: nothing counts down here)
__device__ __forceinline__ InletVel ref_force(unsigned fq, int xa, int xb, int y, const FusedLattice& L) {
    InletVel v = {0.0f, 0.0f, 0.0f, 0.0f};
    if (ref_forced(fq & 0xffffu)) {
        const lbm_lattice_info in = fused_info(L.info, xa, y, L.pitch, L.ny);
        v.ax = in.vx;
        v.ay = in.vy;
    }
    if (ref_forced(fq >> 16)) {
        const lbm_lattice_info in = fused_info(L.info, xb, y, L.pitch, L.ny);
        v.bx = in.vx;
        v.by = in.vy;
    }
    return v;
}

// what a fluid cell (x, y) on the outer ring pulls from solid neighbours: slots that no step writes
__device__ __noinline__ void ref_ring_cell(float* d, int x, int y, const float* buf, const uint16_t* flags, int nx, int ny,
                                           uint32_t N) {
    for (int j = 1; j < 9; ++j) {
        const uint32_t i = (uint32_t)wrap_to(y - EY(j), ny) * (uint32_t)nx + (uint32_t)wrap_to(x - EX(j), nx);
        if (in_bounds((unsigned long long)i, N, BS_FUSED_PULL) && is_solid((int)(flags[i] & FL_MAT_MASK)))
            d[j] = __ldcg(buf + (size_t)j * N + i);
    }
}

// One row of one step.  kept: shared address of the row's own outgoing population 1 of the step
// before (0 in the first step, whose pulls from walls are in memory); buf: the buffer a single step
// would read; field: the step stores its macro field (the one-step kernel fuses the rest population the
// other way round in that case).
template <bool MIXED>
__device__ __forceinline__ void ref_row(float2 (&d)[9], uint32_t kept, int cls, unsigned fq, const InletVel& force, int xa,
                                        int xb, int y, const float* buf, bool field, const FusedLattice& L, const RefConst<float2>& k,
                                        float2 (&o)[9], float2& rho, float2& nux, float2& nuy) {
    if (MIXED && kept && cls != ROW_PLAIN) {
        const unsigned la = is_solid((int)(fq & FL_MAT_MASK)) ? 0u : fq, lb = is_solid((int)((fq >> 16) & FL_MAT_MASK)) ? 0u : fq >> 16;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            if (!(cls & dir_group(g))) continue;  // warp-uniform
#pragma unroll
            for (int i = 1; i < 9; ++i) {  // population i was handed over and comes back as inv i
                if (!(dir_group(g) >> (FL_DIR_SHIFT + i) & 1)) continue;
                lds_where(d[INV(i)].x, kept + 256 * (i - 1), la & (1u << (FL_DIR_SHIFT + i)));
                lds_where(d[INV(i)].y, kept + 256 * (i - 1) + 128, lb & (1u << (FL_DIR_SHIFT + i)));
            }
        }
        if (cls & ROW_RING) {
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const unsigned f = h ? fq >> 16 : fq & 0xffffu;
                if ((f & FL_RING) && !is_solid((int)(f & FL_MAT_MASK))) {
                    float e[9];
#pragma unroll
                    for (int j = 0; j < 9; ++j) e[j] = h ? d[j].y : d[j].x;
                    ref_ring_cell(e, h ? xb : xa, y, buf, L.flags, L.nx, L.ny, L.N);
#pragma unroll
                    for (int j = 0; j < 9; ++j) {
                        if (h) d[j].y = e[j];
                        else d[j].x = e[j];
                    }
                }
            }
            __syncwarp();
        }
    }
    float2 jx, jy;
    core_moments<float2>(d, rho, jx, jy);
    rho = make_float2(fminf(fmaxf(rho.x, 0.8f), 1.2f), fminf(fmaxf(rho.y, 0.8f), 1.2f));
    const float2 r0 = make_float2(rcp_approx(-rho.x), rcp_approx(-rho.y));
    const float2 ninv = vfma(r0, vfma(rho, r0, k.one), r0);  // -1 / rho, as vrcpn
    nux = vmul(jx, ninv);
    nuy = vmul(jy, ninv);
    const bool fa = MIXED && (cls & ROW_FORCE) && ref_forced(fq & 0xffffu), fb = MIXED && (cls & ROW_FORCE) && ref_forced(fq >> 16);
    if (MIXED && (cls & ROW_FORCE)) {
        if (fa) {
            nux.x = __fmul_rn(__fmul_rn(0.5f, force.ax), ninv.x);
            nuy.x = __fmul_rn(__fmul_rn(0.5f, force.ay), ninv.x);
        }
        if (fb) {
            nux.y = __fmul_rn(__fmul_rn(0.5f, force.bx), ninv.y);
            nuy.y = __fmul_rn(__fmul_rn(0.5f, force.by), ninv.y);
        }
    }
    const float2 base = vfma(vfma(nux, nux, vmul(nuy, nuy)), k.m15, k.one);
    const float2 ow0 = vmul(vmul(rho, k.w0), k.om), ow1 = vmul(vmul(rho, k.w1), k.om), ow5 = vmul(vmul(rho, k.w5), k.om);
    if (field) o[0] = vfma(ow0, base, vmul(k.om1, d[0]));
    else o[0] = vfma(k.om1, d[0], vmul(ow0, base));
    const float2 ne[4] = {nux, nuy, vadd(nux, nuy), vfma(nuy, k.mone, nux)};
    const float2 p1 = vmul(ow1, k.c3n), m1 = vmul(ow1, k.c3), p5 = vmul(ow5, k.c3n), m5 = vmul(ow5, k.c3);
    constexpr int J[4] = {1, 4, 8, 5};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 sym = vmul(i < 2 ? ow1 : ow5, vfma(vmul(ne[i], k.c45), ne[i], base));
        o[J[i]] = vfma(k.om1, d[J[i]], vfma(i < 2 ? p1 : p5, ne[i], sym));
        o[INV(J[i])] = vfma(k.om1, d[INV(J[i])], vfma(i < 2 ? m1 : m5, ne[i], sym));
    }
    if (MIXED && (cls & ROW_FORCE)) {
#pragma unroll
        for (int j = 1; j < 9; ++j) {
            const float w = 3.0f * REF_W(j);
            const auto along = [&](float fx, float fy) {
                return EX(j) == 0 ? (float)EY(j) * fy : (EY(j) == 0 ? (float)EX(j) * fx : __fadd_rn((float)EX(j) * fx, (float)EY(j) * fy));
            };
            if (fa) o[j].x = __fmaf_rn(w, along(force.ax, force.ay), o[j].x);
            if (fb) o[j].y = __fmaf_rn(w, along(force.bx, force.by), o[j].y);
        }
    }
#pragma unroll
    for (int j = 0; j < 9; ++j) o[j] = make_float2(ref_limit(o[j].x, REF_MAX(j)), ref_limit(o[j].y, REF_MAX(j)));
}

// leaves the populations that a row of class cls hands to walls for its own next step
__device__ __forceinline__ void keep_handed(uint32_t at, int cls, const float2 (&C)[9]) {
#pragma unroll
    for (int g = 0; g < 3; ++g) {
        if (!(cls & dir_group(g))) continue;  // warp-uniform
#pragma unroll
        for (int i = 1; i < 9; ++i)
            if (dir_group(g) >> (FL_DIR_SHIFT + i) & 1) sts_pair(at + 256 * (i - 1), C[i]);
    }
}

// the last step's store of one cell of a mixed row: wall slots, own slots, zeros between walls
__device__ __forceinline__ void ref_store_cell(const FusedLattice& L, bool mine, unsigned f, uint32_t i, const float (&v)[9]) {
    if (!mine || !in_bounds((unsigned long long)i, L.N, BS_FUSED_STORE)) return;
    if (is_solid((int)(f & FL_MAT_MASK))) {
#pragma unroll
        for (int j = 0; j < 9; ++j)
            if (f & (1u << (FL_DIR_SHIFT + j))) (L.B + (size_t)j * L.N)[i] = 0.0f;
        return;
    }
#pragma unroll
    for (int j = 0; j < 9; ++j) {
        if (f & (1u << (FL_DIR_SHIFT + j))) {
            const uint32_t w = (uint32_t)((int)i + EY(j) * L.nx + EX(j));
            if (in_bounds((unsigned long long)w, L.N, BS_FUSED_STORE)) (L.B + (size_t)INV(j) * L.N)[w] = v[j];
            (L.B + (size_t)j * L.N)[i] = 0.0f;
        } else {
            (L.B + (size_t)j * L.N)[i] = v[j];
        }
    }
}

// One warp: T steps of the window whose first stored column is x0 (a multiple of 4 when VEC), rows
// [y0, y1); see march_window.
template <int T, bool VEC>
__device__ __forceinline__ void march_ref_window(const FusedLattice& L, const RefConst<float2>& kin, int x0, int y0, int y1,
                                                 bool macro, uint32_t smem) {
    static_assert(T == 2 || T == 3, "fused steps");
    constexpr int HALO = T - 1;
    constexpr int IN = 4 - HALO;
    int lane = threadIdx.x & 31;
    hold(lane);
    RefConst<float2> k = kin;
    hold(k.om); hold(k.om1); hold(k.w0); hold(k.w1); hold(k.w5); hold(k.one); hold(k.mone); hold(k.m15); hold(k.c45);
    hold(k.c3); hold(k.c3n);
    const int xa = wrap_to(x0 - HALO + lane, L.nx), xb = wrap_to(x0 - HALO + 32 + lane, L.nx);
    uint32_t kept = smem + KEPT_OFF + 4 * lane;
    hold(kept);

    MarchLoader<VEC> ld;
    ld.init(L, x0 - 4, lane);
    MarchRing R1, R2;
    const float2 z = make_float2(0.0f, 0.0f);
    R1.o0 = R1.o1 = R1.o3 = R1.o4 = R1.o7 = R1.o8 = R1.p4 = R1.p7 = R1.p8 = z;
    R2 = R1;
    constexpr unsigned PLAIN2 = FL_PLAIN | FL_PLAIN << 16;
    unsigned f0, f1 = PLAIN2, f2 = PLAIN2;
    int c0, c1 = ROW_PLAIN, c2 = ROW_PLAIN;

    int yr = wrap_row(y0 - HALO, L.ny);
    int ym = yr == 0 ? L.ny - 1 : yr - 1, yl = yr + 1 == L.ny ? 0 : yr + 1;
    const uint32_t off = 4 * (IN + lane);
    uint32_t sm = smem + off;
    uint32_t s0 = sm + SLOT_BYTES, sp = s0 + SLOT_BYTES, sn = sp + SLOT_BYTES, sf = sn + SLOT_BYTES;
    int yn = yl + 1 == L.ny ? 0 : yl + 1;
    ld.issue(L, (uint32_t)ym * (uint32_t)L.pitch, sm - off);
    ld.issue(L, (uint32_t)yr * (uint32_t)L.pitch, s0 - off);
    ld.issue(L, (uint32_t)yl * (uint32_t)L.pitch, sp - off);
    ld.issue(L, (uint32_t)yn * (uint32_t)L.pitch, sn - off);
    const auto flags_of = [&](uint32_t slot, int y) { return march_flags<VEC>(L, slot, IN + lane, xa, xb, y); };
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    __syncwarp();
    unsigned fn = flags_of(s0, yr);
    InletVel vn = ref_force(fn, xa, xb, yr, L);

    const int end = y1 + HALO;
#pragma unroll 1
    for (int r = y0 - HALO; r < end; ++r) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const int yf = yn + 1 == L.ny ? 0 : yn + 1;
        if (r + 2 < end) ld.issue(L, (uint32_t)yf * (uint32_t)L.pitch, sf - off);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        f0 = fn;
        c0 = ref_row_class(f0);
        const InletVel v0 = vn;
        fn = flags_of(sp, yl);
        vn = ref_force(fn, xa, xb, yl, L);
        const int ys = T == 2 ? ym : (ym == 0 ? L.ny - 1 : ym - 1);

        const auto rows = [&](auto mixed) {
            constexpr bool MIXED = decltype(mixed)::value;
            const auto force_of = [&](int cls, unsigned fq, int y) {
                return MIXED && (cls & ROW_FORCE) ? ref_force(fq, xa, xb, y, L) : InletVel{0.0f, 0.0f, 0.0f, 0.0f};
            };
            float2 d1[9], d2[9], d3[9], C1[9], C2[9], o[9], rho, nux, nuy;
            ring_pulls<false>(R1, lane, 0, 0, 0, 0, d2);
            if (T > 2) ring_pulls<false>(R2, lane, 0, 0, 0, 0, d3);
#pragma unroll
            for (int j = 0; j < 9; ++j)
                d1[j] = lds_pair((EY(j) == 1 ? sm : (EY(j) == -1 ? sp : s0)) + 4 * (MARCH_RAW * j - EX(j)));
            ref_row<MIXED>(d1, 0, c0, f0, v0, xa, xb, yr, L.A, false, L, k, C1, rho, nux, nuy);
            ring_push<false>(R1, C1, lane, 0, 0, d2);
            ref_row<MIXED>(d2, kept, c1, f1, force_of(c1, f1, ym), xa, xb, ym, L.B, T == 2 && macro, L, k, T == 2 ? o : C2, rho, nux, nuy);
            if (MIXED && c0 != ROW_PLAIN) keep_handed(kept, c0, C1);
            if constexpr (T > 2) {
                ring_push<false>(R2, C2, lane, 0, 0, d3);
                ref_row<MIXED>(d3, kept + 2048, c2, f2, force_of(c2, f2, ys), xa, xb, ys, L.A, macro, L, k, o, rho, nux, nuy);
                if (MIXED && c1 != ROW_PLAIN) keep_handed(kept + 2048, c1, C2);
            }
            if (r >= y0 + HALO) {
                RowOut t;
                t.row = (uint32_t)ys * (uint32_t)L.pitch;
                t.ca = x0 - HALO + lane;
                const int xe = min(x0 + MARCH_OUT, L.nx);
                t.sa = t.ca >= x0 && t.ca < xe;
                t.sb = t.ca + 32 >= x0 && t.ca + 32 < xe;
                if (!MIXED) {
                    store_row(L, t, true, true, macro, o, rho, nux, nuy);
                } else {
                    const unsigned fs = T == 2 ? f1 : f2;
                    const bool wa = is_solid((int)(fs & FL_MAT_MASK)), wb = is_solid((int)((fs >> 16) & FL_MAT_MASK));
                    float e[9];
#pragma unroll
                    for (int j = 0; j < 9; ++j) e[j] = o[j].x;
                    ref_store_cell(L, t.sa, fs & 0xffffu, t.row + (uint32_t)xa, e);
#pragma unroll
                    for (int j = 0; j < 9; ++j) e[j] = o[j].y;
                    ref_store_cell(L, t.sb, fs >> 16, t.row + (uint32_t)xb, e);
                    if (macro) store_macro(L, t, !wa, !wb, rho, nux, nuy);
                }
            }
        };
        if ((c0 | c1 | (T > 2 ? c2 : 0)) == ROW_PLAIN) rows(std::false_type{});
        else rows(std::true_type{});

        f2 = f1;
        c2 = c1;
        f1 = f0;
        c1 = c0;
        ym = yr;
        yr = yl;
        yl = yn;
        yn = yf;
        const uint32_t t = sm;
        sm = s0;
        s0 = sp;
        sp = sn;
        sn = sf;
        sf = t;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

}  // namespace lbm
