// lbm_march.cuh -- T fused time steps of an FP32 physics-mode lattice in one pass over memory, for
// large lattices.
//
// One warp owns a window of 64 columns and walks down the rows of a segment.  Rows of the current
// buffer come through a ring in shared memory; the outgoing populations of steps 1 .. T - 1 never
// leave registers: step s + 1 of row r - 1 needs step s of rows r - 2, r - 1 and r, which the warp has
// just computed, and the neighbour columns come by warp shuffle.  Only step T is stored.  A window
// loses one column on each side per fused step, and a segment of H rows computes T - 1 more rows above
// and below for its first step.
//
// Why: one step per pass moves 74 bytes per cell and ran at 94 % of the measured copy bandwidth;
// T = 3 moves about 26 bytes per cell and step.  The march needs no barrier, and loads are in flight
// during two rows' arithmetic; tiles in shared memory (K = 4 steps, one copy of the region) were
// measured slower, their load phases are exposed (4096^2 without solids: 152 against 211 GLUPS with the same arithmetic).
// Measured, BGK, GLUPS before (one step per launch) and now: channel with disks 4096^2 91 and 174,
// 8192^2 86 and 186; KBC 2048^2 63 and 106.  Rows with bounce-backs cost 1.5 times a plain row, rows with an
// inlet or outflow cell twice.  What bounds it now: 55 % of the issue slots at three warps per
// scheduler (registers), waits for fixed latencies; DRAM at 60 to 75 % of the measured copy rate.
//
// Cells next to a solid bounce their own outgoing population back (a select); inlet, outflow,
// moving-wall and forcing cells take the rules of lbm_fused.cuh.  All arithmetic is the core's, so the
// state is that of T single steps bit for bit.  Not for lattices whose forcing cells count down
// (the host keeps those on the one-step kernel): rows are computed by several warps.
#pragma once

#include "lbm_fused.cuh"

namespace lbm {

constexpr int MARCH_W = 64;    // columns of a window
constexpr int MARCH_OUT = 60;  // columns it stores: 64 - 2 (T - 1) for T = 3, and a multiple of 4 (T = 2 as well)

// the value of the column to the right for both halves of a row; column 63 gets one of no meaning
__device__ __forceinline__ float2 from_right(float2 v, int lane) {
    const int src = (lane + 1) & 31;
    const float a = __shfl_sync(0xffffffffu, v.x, src), b = __shfl_sync(0xffffffffu, v.y, src);
    return make_float2(lane == 31 ? b : a, b);
}
__device__ __forceinline__ float lds_f32(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float2 lds_pair(uint32_t a) { return make_float2(lds_f32(a), lds_f32(a + 128)); }
__device__ __forceinline__ void sts_pair(uint32_t a, float2 v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v.x) : "memory");
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a + 128), "f"(v.y) : "memory");
}
// v = the word at a where m is not zero: one predicated load, no select
__device__ __forceinline__ void lds_where(float& v, uint32_t a, unsigned m) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.shared.f32 %0, [%1];\n\t}"
                 : "+f"(v)
                 : "r"(a), "r"(m)
                 : "memory");
}
__device__ __forceinline__ unsigned lds_u16(uint32_t a) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
    return v;
}

// Slot of one lattice row: the nine planes of MARCH_RAW columns (the window and two more on each
// side) and their flag words.  A warp keeps five slots: rows r - 1, r, r + 1 feed step 1 of row r while
// rows r + 2 and r + 3 are on their way, so a load has two iterations to arrive, without a register
// waiting for it (with four slots and one iteration 4096^2 without solids ran 5 % slower).
constexpr int MARCH_RAW = 68;
constexpr int SLOT_FLAGS = 9 * MARCH_RAW * 4;  // byte offset of the flag words
constexpr int SLOT_BYTES = SLOT_FLAGS + ((MARCH_RAW * 2 + 15) / 16) * 16;
constexpr int KEPT_OFF = 5 * SLOT_BYTES;            // own outgoing populations 1 .. 8 of steps 1 and 2
// bytes per warp that fuses t steps
__host__ __device__ constexpr int march_smem(int t) { return KEPT_OFF + (t - 1) * 8 * 256; }

// The copies of a warp.  VEC (rows a multiple of 4 cells long): 16-byte copies of four cells, two
// planes at a time by the two halves of the warp, then the seventeenth chunk of all nine planes;
// else 4-byte copies of single cells.
template <bool VEC>
struct MarchLoader {
    uint32_t src0, src1, src2;  // cell offsets in a row (VEC: the first with its plane's, 0 or 1)
    int lane;
    // raw0: the slot's first column (a multiple of 4 when VEC), from -4 to nx
    __device__ __forceinline__ void init(const FusedLattice& L, int raw0, int ln) {
        lane = ln;
        if constexpr (VEC) {  // a chunk lies in one row: the pitch is a multiple of 4 cells, and so is raw0
            src0 = (uint32_t)(lane >> 4) * L.N + (uint32_t)wrap_to(raw0 + 4 * (lane & 15), L.pitch);
            src1 = (uint32_t)wrap_to(raw0 + 64, L.pitch);
            src2 = (uint32_t)wrap_to(raw0 + 4 * min(lane, 16), L.pitch);
        } else {
            src0 = (uint32_t)wrap_to(raw0 + lane, L.nx);
            src1 = (uint32_t)wrap_to(raw0 + 32 + lane, L.nx);
            src2 = (uint32_t)wrap_to(raw0 + 64 + (lane & 3), L.nx);
        }
    }
    // row offset o (cells) into the slot at dst (shared address)
    __device__ __forceinline__ void issue(const FusedLattice& L, uint32_t o, uint32_t dst) const {
        if constexpr (VEC) {
            const uint32_t d = dst + (lane >> 4) * (4 * MARCH_RAW) + 16 * (lane & 15);
#pragma unroll
            for (int j = 0; j < 9; j += 2)
                if ((j < 8 || lane < 16) && in_bounds((unsigned long long)src0 + o + (unsigned long long)j * L.N + 3, 9ull * L.N, BS_FUSED_PULL))
                    cp_async_to<16>(d + 4 * MARCH_RAW * j, L.A + (size_t)j * L.N + (src0 + o));
            // (eight planes of 2^29 cells or more are past 32 bits)
            if (lane < 9 && in_bounds((unsigned long long)src1 + o + 3, L.N, BS_FUSED_PULL))
                cp_async_to<16>(dst + 4 * MARCH_RAW * lane + 256, L.A + (size_t)lane * L.N + (src1 + o));
            if (lane < 17 && in_bounds((unsigned long long)src2 + o + 3, L.N, BS_FUSED_FLAGS))
                cp_async_to<8>(dst + SLOT_FLAGS + 8 * lane, L.flags + (src2 + o));
        } else {
#pragma unroll
            for (int j = 0; j < 9; ++j) {
                const float* P = L.A + (size_t)j * L.N + o;
                const uint32_t d = dst + 4 * (MARCH_RAW * j + lane);
                if (in_bounds((unsigned long long)src0 + o, L.N, BS_FUSED_PULL)) cp_async_to<4>(d, P + src0);
                if (in_bounds((unsigned long long)src1 + o, L.N, BS_FUSED_PULL)) cp_async_to<4>(d + 128, P + src1);
            }
            // the last four columns of eight planes, then of the ninth
            if (in_bounds((unsigned long long)src2 + o, L.N, BS_FUSED_PULL)) {
                cp_async_to<4>(dst + 4 * (MARCH_RAW * (lane >> 2) + 64 + (lane & 3)),
                               L.A + (size_t)(lane >> 2) * L.N + o + src2);
                if (lane < 4) cp_async_to<4>(dst + 4 * (MARCH_RAW * 8 + 64 + lane), L.A + (size_t)8 * L.N + o + src2);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
};

// flag words of a lane's two cells in row y, whose slot address (at the lane's first cell, column `col`
// of the slot) is `slot`
template <bool VEC>
__device__ __forceinline__ unsigned march_flags(const FusedLattice& L, uint32_t slot, int col, int xa, int xb, int y) {
    if constexpr (VEC) {
        const uint32_t fa = slot + SLOT_FLAGS - 2 * col;
        return lds_u16(fa) | lds_u16(fa + 64) << 16;
    } else {
        const uint32_t o = (uint32_t)y * (uint32_t)L.pitch;
        const bool in = in_bounds((unsigned long long)o + xa, L.N, BS_FUSED_FLAGS) &&
                        in_bounds((unsigned long long)o + xb, L.N, BS_FUSED_FLAGS);
        return in ? (unsigned)__ldg(L.flags + (o + (uint32_t)xa)) | (unsigned)__ldg(L.flags + (o + (uint32_t)xb)) << 16
                  : FL_PLAIN | FL_PLAIN << 16;
    }
}

// what a step hands to the next one between rows: outgoing populations of its last row (o0 .. o8: those
// that the row itself or the row below pulls), and the pulls that its last row takes from above
struct MarchRing {
    float2 o0, o1, o3, o4, o7, o8;
    float2 p4, p7, p8;
};

// the part of a row's pulls that the ring holds, and the ring's own pulls moved on by one row.  The
// row's class is cls, the next row's cn (flag words fq, fn): an outflow cell pulls from its own column.
template <bool MIXED>
__device__ __forceinline__ void ring_pulls(MarchRing& R, int lane, int cls, unsigned fq, int cn, unsigned fn,
                                           float2 (&d)[9]) {
    d[0] = R.o0;
    d[1] = from_left(R.o1, lane);
    d[3] = from_right(R.o3, lane);
    d[4] = R.p4;
    d[7] = R.p7;
    d[8] = R.p8;
    R.p4 = R.o4;
    R.p7 = from_right(R.o7, lane);
    R.p8 = from_left(R.o8, lane);
    if (MIXED && (cls & (ROW_FACE | ROW_RARE))) {
        if ((fq & FL_MAT_MASK) == LBM_OUTLET) d[3].x = R.o3.x;
        if (((fq >> 16) & FL_MAT_MASK) == LBM_OUTLET) d[3].y = R.o3.y;
    }
    if (MIXED && (cn & (ROW_FACE | ROW_RARE))) {
        if ((fn & FL_MAT_MASK) == LBM_OUTLET) R.p7.x = R.o7.x;
        if (((fn >> 16) & FL_MAT_MASK) == LBM_OUTLET) R.p7.y = R.o7.y;
    }
}
// the pulls from the row below, whose outgoing populations are C; C goes into the ring
template <bool MIXED>
__device__ __forceinline__ void ring_push(MarchRing& R, const float2 (&C)[9], int lane, int cls, unsigned fq,
                                          float2 (&d)[9]) {
    d[2] = C[2];
    d[5] = from_left(C[5], lane);
    d[6] = from_right(C[6], lane);
    if (MIXED && (cls & (ROW_FACE | ROW_RARE))) {
        if ((fq & FL_MAT_MASK) == LBM_OUTLET) d[6].x = C[6].x;
        if (((fq >> 16) & FL_MAT_MASK) == LBM_OUTLET) d[6].y = C[6].y;
    }
    R.o0 = C[0];
    R.o1 = C[1];
    R.o3 = C[3];
    R.o4 = C[4];
    R.o7 = C[7];
    R.o8 = C[8];
}

// directions (flag bits) with e_x = 1, -1 and 0
__host__ __device__ constexpr int dir_group(int g) {
    return g == 0 ? (1 << 1 | 1 << 5 | 1 << 8) << FL_DIR_SHIFT
                  : (g == 1 ? (1 << 3 | 1 << 6 | 1 << 7) << FL_DIR_SHIFT : (1 << 2 | 1 << 4) << FL_DIR_SHIFT);
}
// leaves what the bounce-backs of a row of class cls read in the next step: its own populations
__device__ __forceinline__ void keep_own(uint32_t at, int cls, const float2 (&C)[9]) {
#pragma unroll
    for (int g = 0; g < 3; ++g) {
        if (!(cls & dir_group(g))) continue;  // warp-uniform
#pragma unroll
        for (int j = 1; j < 9; ++j)
            if (dir_group(g) >> (FL_DIR_SHIFT + INV(j)) & 1) sts_pair(at + 256 * (j - 1), C[j]);
    }
}

// One row of one step: bounce-back (own: shared address of the cell's own outgoing population 1 of
// the step before, `stride` bytes from one population to the next), inlet, outflow, collision, rare cells.
template <int COLL, bool MIXED>
__device__ __forceinline__ void march_row(float2 (&d)[9], uint32_t own, int stride, int cls, unsigned fq, const InletVel& vel, int xa, int xb,
                                          int y, const FusedLattice& L, const BgkConst<float2>& k, float2 (&o)[9],
                                          float2& rho, float2& nux, float2& nuy) {
    if (MIXED && cls != ROW_PLAIN) {
        // by groups of directions, as walls ask for them: from the west, from the east, straight
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            if (!(cls & dir_group(g))) continue;  // warp-uniform
#pragma unroll
            for (int j = 1; j < 9; ++j) {
                if (!(dir_group(g) >> (FL_DIR_SHIFT + j) & 1)) continue;
                const uint32_t a = own + (uint32_t)((INV(j) - 1) * stride);
                lds_where(d[j].x, a, fq & (1u << (FL_DIR_SHIFT + j)));
                lds_where(d[j].y, a + 128, fq & (1u << (16 + FL_DIR_SHIFT + j)));
            }
        }
        if (cls & ROW_FACE) face_cells(d, fq, vel, k.omega);
    }
    float2 drho, jx, jy;
    core_moments<float2>(d, drho, jx, jy);
    core_collide<COLL, float2>(d, k, drho, jx, jy, o, rho, nux, nuy);
    if (MIXED && (cls & ROW_RARE)) rare_cells<COLL>(d, fq, xa, xb, y, L, k.omega, o, rho, nux, nuy);
}

// One warp: T steps of the window whose first stored column is x0 (a multiple of 4 when VEC), rows
// [y0, y1).  smem: the warp's march_smem(T) bytes (shared address, 16-byte aligned).
template <int T, int COLL, bool VEC>
__device__ __forceinline__ void march_window(const FusedLattice& L, const BgkConst<float2>& kin, int x0, int y0, int y1,
                                             bool macro, uint32_t smem) {
    static_assert(T == 2 || T == 3, "steps of one pass");
    constexpr int HALO = T - 1;
    constexpr int IN = 4 - HALO;  // the window's first column in a slot
    int lane = threadIdx.x & 31;
    hold(lane);
    BgkConst<float2> k = kin;  // in registers: packed instructions take no other operands
    hold(k.om); hold(k.omn); hold(k.om1); hold(k.w1); hold(k.w5); hold(k.w31); hold(k.w35); hold(k.c45);
    hold(k.one); hold(k.mone); hold(k.m15);
    const int WN = VEC ? L.pitch : L.nx;  // where columns wrap (a padded row never reaches round)
    const int xa = wrap_to(x0 - HALO + lane, WN), xb = wrap_to(x0 - HALO + 32 + lane, WN);
    uint32_t kept = smem + KEPT_OFF + 4 * lane;
    hold(kept);

    MarchLoader<VEC> ld;
    ld.init(L, x0 - 4, lane);
    MarchRing R1, R2;
    const float2 z = make_float2(0.0f, 0.0f);
    R1.o0 = R1.o1 = R1.o3 = R1.o4 = R1.o7 = R1.o8 = R1.p4 = R1.p7 = R1.p8 = z;
    R2 = R1;
    constexpr unsigned PLAIN2 = FL_PLAIN | FL_PLAIN << 16;
    unsigned f0, f1 = PLAIN2, f2 = PLAIN2;  // flag words of rows r, r - 1, r - 2
    int c0, c1 = ROW_PLAIN, c2 = ROW_PLAIN;  // and their classes

    int yr = wrap_row(y0 - HALO, L.ny);  // wrapped row of step 1
    int ym = yr == 0 ? L.ny - 1 : yr - 1, yl = yr + 1 == L.ny ? 0 : yr + 1;
    // slots of rows r - 1 .. r + 3, at the lane's first cell: every access below is a constant offset away
    uint32_t sm = smem + 4 * (IN + lane);
    uint32_t s0 = sm + SLOT_BYTES, sp = s0 + SLOT_BYTES, sn = sp + SLOT_BYTES, sf = sn + SLOT_BYTES;
    const uint32_t off = 4 * (IN + lane);
    int yn = yl + 1 == L.ny ? 0 : yl + 1;
    ld.issue(L, (uint32_t)ym * (uint32_t)L.pitch, sm - off);
    ld.issue(L, (uint32_t)yr * (uint32_t)L.pitch, s0 - off);
    ld.issue(L, (uint32_t)yl * (uint32_t)L.pitch, sp - off);
    ld.issue(L, (uint32_t)yn * (uint32_t)L.pitch, sn - off);
    const auto flags_of = [&](uint32_t slot, int y) { return march_flags<VEC>(L, slot, IN + lane, xa, xb, y); };

    asm volatile("cp.async.wait_group 2;" ::: "memory");  // the first two rows
    __syncwarp();
    unsigned fn = flags_of(s0, yr);  // the next row's flag words and inlet velocities, one row ahead
    InletVel vn = inlet_vel(fn, xa, xb, yr, L);

    const int end = y1 + HALO;
#pragma unroll 1
    for (int r = y0 - HALO; r < end; ++r) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");  // all but the row after the next one
        __syncwarp();  // the row below has arrived for every lane, and nobody reads row r - 2 any more
        const int yf = yn + 1 == L.ny ? 0 : yn + 1;
        if (r + 2 < end) ld.issue(L, (uint32_t)yf * (uint32_t)L.pitch, sf - off);
        else asm volatile("cp.async.commit_group;" ::: "memory");  // an empty group keeps the count
        f0 = fn;
        c0 = row_class(f0);
        const InletVel v0 = vn;
        fn = flags_of(sp, yl);
        vn = inlet_vel(fn, xa, xb, yl, L);
        const int ys = T == 2 ? ym : (ym == 0 ? L.ny - 1 : ym - 1);  // row of step T

        const auto rows = [&](auto mixed) {
            constexpr bool MIXED = decltype(mixed)::value;
            // later steps' inlet velocities are in the first-level cache by now
            const auto vel_of = [&](int cls, unsigned fq, int y) {
                return MIXED && (cls & ROW_FACE) ? inlet_vel(fq, xa, xb, y, L) : InletVel{0.0f, 0.0f, 0.0f, 0.0f};
            };
            float2 d1[9], d2[9], d3[9], C1[9], C2[9], o[9], rho, nux, nuy;
            // pulls from the rings first: their registers take the new rows
            ring_pulls<MIXED>(R1, lane, c1, f1, c0, f0, d2);
            if (T > 2) ring_pulls<MIXED>(R2, lane, c2, f2, c1, f1, d3);
#pragma unroll
            for (int j = 0; j < 9; ++j)
                d1[j] = lds_pair((EY(j) == 1 ? sm : (EY(j) == -1 ? sp : s0)) + 4 * (MARCH_RAW * j - EX(j)));
            if (MIXED && (c0 & (ROW_FACE | ROW_RARE))) {  // outflow cells pull from their own column
                const float2 e3 = lds_pair(s0 + 4 * MARCH_RAW * 3), e6 = lds_pair(sp + 4 * MARCH_RAW * 6),
                             e7 = lds_pair(sm + 4 * MARCH_RAW * 7);
                if ((f0 & FL_MAT_MASK) == LBM_OUTLET) { d1[3].x = e3.x; d1[6].x = e6.x; d1[7].x = e7.x; }
                if (((f0 >> 16) & FL_MAT_MASK) == LBM_OUTLET) { d1[3].y = e3.y; d1[6].y = e6.y; d1[7].y = e7.y; }
            }
            march_row<COLL, MIXED>(d1, s0 + 4 * MARCH_RAW, 4 * MARCH_RAW, c0, f0, v0, xa, xb, yr, L, k, C1, rho, nux, nuy);
            ring_push<MIXED>(R1, C1, lane, c1, f1, d2);
            march_row<COLL, MIXED>(d2, kept, 256, c1, f1, vel_of(c1, f1, ym), xa, xb, ym, L, k, T == 2 ? o : C2, rho, nux,
                                   nuy);
            if (MIXED && c0 != ROW_PLAIN) keep_own(kept, c0, C1);
            if constexpr (T > 2) {
                ring_push<MIXED>(R2, C2, lane, c2, f2, d3);
                march_row<COLL, MIXED>(d3, kept + 2048, 256, c2, f2, vel_of(c2, f2, ys), xa, xb, ys, L, k, o, rho, nux, nuy);
                if (MIXED && c1 != ROW_PLAIN) keep_own(kept + 2048, c1, C2);
            }
            if (r >= y0 + HALO) {
                RowOut t;
                t.row = (uint32_t)ys * (uint32_t)L.pitch;
                t.ca = x0 - HALO + lane;
                const int xe = min(x0 + MARCH_OUT, L.nx);
                t.sa = t.ca >= x0 && t.ca < xe;
                t.sb = t.ca + 32 >= x0 && t.ca + 32 < xe;
                const unsigned fs = T == 2 ? f1 : f2;
                store_row(L, t, !MIXED || !is_solid((int)(fs & FL_MAT_MASK)),
                          !MIXED || !is_solid((int)((fs >> 16) & FL_MAT_MASK)), macro, o, rho, nux, nuy);
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
