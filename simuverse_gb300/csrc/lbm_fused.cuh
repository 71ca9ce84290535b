// lbm_fused.cuh -- what the kernels of fused time steps share: the lattice, row classes, the rules
// of cells at inlets, outflows, moving walls and under a force, and the store of a finished row.
// A row is 64 columns wide: lane l holds columns l and l + 32 as the halves of packed FP32x2 values.
#pragma once

#include <type_traits>

#include "lbm_core.cuh"

namespace lbm {

// the lattice a launch works on; planes are N elements apart
struct FusedLattice {
    const float* __restrict__ A;
    float* __restrict__ B;
    const uint16_t* __restrict__ flags;
    const lbm_lattice_info* __restrict__ info;
    float* __restrict__ macro;
    int nx, pitch, ny;
    uint32_t N;  // pitch * ny
};

__device__ __forceinline__ int wrap_to(int v, int n) {  // v in [-n, 2 n)
    return v < 0 ? v + n : (v >= n ? v - n : v);
}
__device__ __forceinline__ int wrap_row(int v, int n) {  // any v above -n: a region may be taller than the lattice
    return v < 0 ? v + n : (v >= n ? v % n : v);
}
template <int BYTES>
__device__ __forceinline__ void cp_async_to(uint32_t dst, const void* src) {
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}

// the value of the column to the left for both halves of a row; column 0 gets one of no meaning
__device__ __forceinline__ float2 from_left(float2 v, int lane) {
    const int src = (lane + 31) & 31;
    const float a = __shfl_sync(0xffffffffu, v.x, src), b = __shfl_sync(0xffffffffu, v.y, src);
    return make_float2(a, lane == 0 ? a : b);
}

// a row's class: 0 where every cell is plain; else the bits below, and bit FL_DIR_SHIFT + j for every
// direction j that some cell bounces back
enum { ROW_PLAIN = 0, ROW_MIXED = 1, ROW_FACE = 2, ROW_RARE = 4 };
// cells whose rule needs more than a bounce-back, inlet or outflow: a moving wall beside it, or a force
__device__ __forceinline__ bool rare_cell(unsigned f) {
    return (int)(f & FL_MAT_MASK) == LBM_EXTERNAL_FORCE || (f & FL_MOVING);
}
__device__ __forceinline__ bool face_cell(unsigned f) {  // inlet and outflow without such a rule
    const int m = (int)(f & FL_MAT_MASK);
    return (m == LBM_INLET || m == LBM_OUTLET) && !(f & FL_MOVING);
}
// warp-uniform class of a row whose flag words are fq (two cells per lane)
__device__ __forceinline__ int row_class(unsigned fq) {
    if (__all_sync(0xffffffffu, (fq & (FL_PLAIN | FL_PLAIN << 16)) == (FL_PLAIN | FL_PLAIN << 16))) return ROW_PLAIN;
    // a row that is not plain: the directions that some cell bounces back come with the class
    const int dirs = (int)(__reduce_or_sync(0xffffffffu, fq | fq >> 16) & (0x1FEu << FL_DIR_SHIFT));
    const bool face = __any_sync(0xffffffffu, face_cell(fq & 0xffffu) || face_cell(fq >> 16));
    const bool rare = __any_sync(0xffffffffu, rare_cell(fq & 0xffffu) || rare_cell(fq >> 16));
    return dirs | ROW_MIXED | (face ? ROW_FACE : 0) | (rare ? ROW_RARE : 0);
}
__device__ __forceinline__ lbm_lattice_info fused_info(const lbm_lattice_info* info, int x, int y, int pitch, int ny) {
    const uint32_t i = (uint32_t)y * (uint32_t)pitch + (uint32_t)x;
    const lbm_lattice_info none = {0, 0, 0.0f, 0.0f};
    return in_bounds((unsigned long long)i, (unsigned long long)pitch * ny, BS_FUSED_INFO) ? info[i] : none;
}

// A rare cell is handed over in memory: its pulled populations with the bounce-back done, and back
// the outgoing populations, then density and negative velocity.  A function of its own, so that the step
// loop's code stays small.
template <int COLL>
__device__ __noinline__ void rare_cell_step(float* io, unsigned f, int x, int y, const lbm_lattice_info* info, int nx,
                                            int pitch, int ny, float omega) {
    const BgkConst<float> k(omega);
    const int m = (int)(f & FL_MAT_MASK);
    float d[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) d[j] = io[j];
    if (f & FL_MOVING) {
#pragma unroll
        for (int j = 1; j < 9; ++j) {
            if (!(f & (1u << (FL_DIR_SHIFT + j)))) continue;
            const int sx = (m == LBM_OUTLET && EX(j) == -1) ? x : wrap_to(x - EX(j), nx);
            const lbm_lattice_info si = fused_info(info, sx, wrap_to(y - EY(j), ny), pitch, ny);
            const float uw = (EX(j) == 0 ? 0.0f : (float)EX(j) * si.vx) + (EY(j) == 0 ? 0.0f : (float)EY(j) * si.vy);
            if (uw != 0.0f) d[j] = add_rn(d[j], mul_rn(6.0f * PW<float>(j), uw));
        }
    }
    const bool forced = m == LBM_EXTERNAL_FORCE;  // a permanent force: nothing counts down here
    const lbm_lattice_info in =
        forced || m == LBM_INLET ? fused_info(info, x, y, pitch, ny) : lbm_lattice_info{0, 0, 0.0f, 0.0f};
    if (m == LBM_INLET) core_inlet<float>(d, in.vx, in.vy);
    if (m == LBM_OUTLET) core_outlet<float>(d, k);
    float drho, jx, jy, o[9], rho, nux, nuy;
    core_moments<float>(d, drho, jx, jy);
    if (forced) {
        jx = vfma(0.5f, in.vx, jx);
        jy = vfma(0.5f, in.vy, jy);
    }
    core_collide<COLL, float>(d, k, drho, jx, jy, o, rho, nux, nuy);
    if (forced) core_guo<float>(k, -nux, -nuy, in.vx, in.vy, drho, o);
#pragma unroll
    for (int j = 0; j < 9; ++j) io[j] = o[j];
    io[9] = rho;
    io[10] = nux;
    io[11] = nuy;
}

// velocities of a lane's inlet cells (zero elsewhere)
struct InletVel {
    float ax, ay, bx, by;
};
__device__ __forceinline__ InletVel inlet_vel(unsigned fq, int xa, int xb, int y, const FusedLattice& L) {
    InletVel v = {0.0f, 0.0f, 0.0f, 0.0f};
    if ((fq & FL_MAT_MASK) == LBM_INLET) {
        const lbm_lattice_info in = fused_info(L.info, xa, y, L.pitch, L.ny);
        v.ax = in.vx;
        v.ay = in.vy;
    }
    if (((fq >> 16) & FL_MAT_MASK) == LBM_INLET) {
        const lbm_lattice_info in = fused_info(L.info, xb, y, L.pitch, L.ny);
        v.bx = in.vx;
        v.by = in.vy;
    }
    return v;
}

// Inlet and outflow rules on the pulled populations (bounce-back done, outflow populations in place)
__device__ __forceinline__ void face_cells(float2 (&d)[9], unsigned fq, const InletVel& v, float omega) {
    if (__any_sync(0xffffffffu, face_cell(fq & 0xffffu))) {
        if (face_cell(fq & 0xffffu)) {
            float e[9];
#pragma unroll
            for (int j = 0; j < 9; ++j) e[j] = d[j].x;
            if ((fq & FL_MAT_MASK) == LBM_INLET) core_inlet<float>(e, v.ax, v.ay);
            else core_outlet<float>(e, BgkConst<float>(omega));
#pragma unroll
            for (int j = 0; j < 9; ++j) d[j].x = e[j];
        }
        __syncwarp();
    }
    if (__any_sync(0xffffffffu, face_cell(fq >> 16))) {
        if (face_cell(fq >> 16)) {
            float e[9];
#pragma unroll
            for (int j = 0; j < 9; ++j) e[j] = d[j].y;
            if (((fq >> 16) & FL_MAT_MASK) == LBM_INLET) core_inlet<float>(e, v.bx, v.by);
            else core_outlet<float>(e, BgkConst<float>(omega));
#pragma unroll
            for (int j = 0; j < 9; ++j) d[j].y = e[j];
        }
        __syncwarp();
    }
}

// The rare cells of a row, after its packed collision
template <int COLL>
__device__ __forceinline__ void rare_cells(const float2 (&d)[9], unsigned fq, int xa, int xb, int y, const FusedLattice& L,
                                          float omega, float2 (&o)[9], float2& rho, float2& nux, float2& nuy) {
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        const unsigned f = h ? fq >> 16 : fq & 0xffffu;
        if (rare_cell(f)) {
            float io[12];
#pragma unroll
            for (int j = 0; j < 9; ++j) io[j] = h ? d[j].y : d[j].x;
            rare_cell_step<COLL>(io, f, h ? xb : xa, y, L.info, L.nx, L.pitch, L.ny, omega);
#pragma unroll
            for (int j = 0; j < 9; ++j) {
                if (h) o[j].y = io[j];
                else o[j].x = io[j];
            }
            if (h) { rho.y = io[9]; nux.y = io[10]; nuy.y = io[11]; }
            else { rho.x = io[9]; nux.x = io[10]; nuy.x = io[11]; }
        }
    }
}

// keeps a value in registers: the compiler may not load it again where it is used
__device__ __forceinline__ void hold(float2& v) { asm volatile("" : "+f"(v.x), "+f"(v.y)); }
__device__ __forceinline__ void hold(int& v) { asm volatile("" : "+r"(v)); }
__device__ __forceinline__ void hold(uint32_t& v) { asm volatile("" : "+r"(v)); }

// the stored part of a row in global memory
struct RowOut {
    uint32_t row;  // offset of the row's first cell
    int ca;        // the lane's first column
    bool sa, sb;   // whether its two cells are stored
};
// macro field of a row's two cells; ga, gb: fluid (a solid cell's is zero)
__device__ __forceinline__ void store_macro(const FusedLattice& L, const RowOut& t, bool ga, bool gb, float2 rho,
                                            float2 nux, float2 nuy) {
    const long long i = (long long)t.row + t.ca;
    float* m = L.macro + i;
    if (t.sa && in_bounds((unsigned long long)i, L.N, BS_FUSED_MACRO)) {
        m[0] = ga ? rho.x : 0.0f;
        m[(size_t)L.N] = ga ? -nux.x : 0.0f;
        m[(size_t)2 * L.N] = ga ? -nuy.x : 0.0f;
    }
    if (t.sb && in_bounds((unsigned long long)(i + 32), L.N, BS_FUSED_MACRO)) {
        m[32] = gb ? rho.y : 0.0f;
        m[(size_t)L.N + 32] = gb ? -nux.y : 0.0f;
        m[(size_t)2 * L.N + 32] = gb ? -nuy.y : 0.0f;
    }
}
__device__ __forceinline__ void store_row(const FusedLattice& L, const RowOut& t, bool ga, bool gb, bool macro,
                                          const float2 (&o)[9], float2 rho, float2 nux, float2 nuy) {
    // signed: the first column may lie left of the lattice where the second lies in it
    const long long i = (long long)t.row + t.ca;
    float* q = L.B + i;
    if (t.sa && ga && in_bounds((unsigned long long)i, L.N, BS_FUSED_STORE)) {
#pragma unroll
        for (int j = 0; j < 9; ++j) q[(size_t)j * L.N] = o[j].x;
    }
    if (t.sb && gb && in_bounds((unsigned long long)(i + 32), L.N, BS_FUSED_STORE)) {
#pragma unroll
        for (int j = 0; j < 9; ++j) q[(size_t)j * L.N + 32] = o[j].y;
    }
    if (macro) store_macro(L, t, ga, gb, rho, nux, nuy);
}

}  // namespace lbm
