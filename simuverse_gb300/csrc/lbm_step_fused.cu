// lbm_step_fused.cu -- fused time steps of a single lattice: how many steps one launch takes, and the
// kernel over march_window (lbm_march.cuh).
#include <algorithm>

#include "lbm_internal.h"
#include "lbm_march.cuh"
#include "lbm_march_ref.cuh"

namespace lbm {

// One-warp blocks per SM the kernels are compiled for: 168 registers, no spills.  (A spill costs far more
// than extra warps give, as the shared memory leaves little first-level cache; 13 or 14 blocks ran 10 to
// 60 % slower, 8 to 11 the same to 10 % slower.)
constexpr int MARCH_BLOCKS = 12;

// One warp per block: a finished warp's place is taken at once.  The windows at the lattice's left
// and right edge, which hold the inlet and outflow columns and take longer, come first.
struct MarchTask {
    int x0, y0, y1;
};
__device__ __forceinline__ MarchTask march_task(int rows, int windows, int segments, int ny) {
    const int t = (int)blockIdx.x;
    int w, seg;
    if (windows < 3 || t < 2 * segments) {
        const int e = windows < 3 ? windows : 2;
        seg = t / e;
        w = t % e == 0 ? 0 : windows - 1;
    } else {
        seg = (t - 2 * segments) / (windows - 2);
        w = 1 + (t - 2 * segments) % (windows - 2);
    }
    return {w * MARCH_OUT, seg * rows, min(seg * rows + rows, ny)};
}

template <int T, int COLL, bool VEC>
__global__ void __launch_bounds__(32, MARCH_BLOCKS)
    k_phys_march(const __grid_constant__ FusedLattice L, const __grid_constant__ BgkConst<float2> k, int rows,
                 int windows, int segments, bool macro) {
    extern __shared__ __align__(16) unsigned char march_mem[];
    const MarchTask t = march_task(rows, windows, segments, L.ny);
    march_window<T, COLL, VEC>(L, k, t.x0, t.y0, t.y1, macro, (uint32_t)__cvta_generic_to_shared(march_mem));
}

template <int T, bool VEC>
__global__ void __launch_bounds__(32, MARCH_BLOCKS)
    k_ref_march(const __grid_constant__ FusedLattice L, const __grid_constant__ RefConst<float2> k, int rows, int windows,
                int segments, bool macro) {
    extern __shared__ __align__(16) unsigned char march_mem[];
    const MarchTask t = march_task(rows, windows, segments, L.ny);
    march_ref_window<T, VEC>(L, k, t.x0, t.y0, t.y1, macro, (uint32_t)__cvta_generic_to_shared(march_mem));
}

__global__ void __launch_bounds__(256) k_count_rows(const uint16_t* __restrict__ flags, int nx, int ny, bool reference,
                                                    unsigned long long* __restrict__ out) {
    const int windows = (nx + MARCH_OUT - 1) / MARCH_OUT, lane = (int)threadIdx.x & 31;
    const size_t total = (size_t)windows * ny, warps = (size_t)gridDim.x * (blockDim.x / 32);
    RowCounts n;
    for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; i < total; i += warps) {
        const int y = (int)(i / windows), x0 = (int)(i % windows) * MARCH_OUT - 2 + lane;
        bool forced = false, rare = false, face = false, mixed = false, inner = false;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int x = ((x0 + 32 * h) % nx + nx) % nx;
            const unsigned f = flags[(size_t)y * nx + x];
            const bool wall = is_solid((int)(f & FL_MAT_MASK));
            inner |= wall && x >= 2 && x < nx - 2 && y >= 2 && y < ny - 2;
            mixed |= !(f & FL_PLAIN);
            if (reference) {
                face |= !wall && (ref_forced(f) || (f & FL_RING));
            } else {
                forced |= (int)(f & FL_MAT_MASK) == LBM_EXTERNAL_FORCE;
                rare |= rare_cell(f);
                face |= face_cell(f);
            }
        }
        n.forced += __any_sync(0xffffffffu, forced);
        n.rare += __any_sync(0xffffffffu, rare);
        n.face += __any_sync(0xffffffffu, face);
        n.mixed += __any_sync(0xffffffffu, mixed);
        n.inner += __any_sync(0xffffffffu, inner);
    }
    if (lane == 0 && n.mixed) {
        atomicAdd(out, n.forced);
        atomicAdd(out + 1, n.rare);
        atomicAdd(out + 2, n.face);
        atomicAdd(out + 3, n.mixed);
        atomicAdd(out + 4, n.inner);
    }
}
cudaError_t launch_count_rows(lbm_handle* h, cudaStream_t s) {
    static_assert(sizeof(RowCounts) == 5 * sizeof(unsigned long long), "as k_count_rows writes them");
    const cudaError_t e = cudaMemsetAsync(h->d_count + 1, 0, sizeof(RowCounts), s);
    if (e != cudaSuccess) return e;
    k_count_rows<<<RED_BLOCKS, 256, 0, s>>>(h->d_flags, h->nx, h->ny, h->p.mode == LBM_MODE_REFERENCE, h->d_count + 1);
    return cudaGetLastError();
}
RowCounts scene_rows(const lbm_handle* h) {
    const unsigned long long windows = (unsigned long long)(h->nx + MARCH_OUT - 1) / MARCH_OUT, ny = (unsigned long long)h->ny;
    RowCounts n;
    if (h->p.scene == LBM_SCENE_PERIODIC) return n;
    n.mixed = 2 * (windows + ny);  // at the border (disks are not counted)
    if (h->p.scene == LBM_SCENE_CAVITY) n.rare = windows;  // under the lid
    if (h->p.scene == LBM_SCENE_CHANNEL) n.face = 2 * ny;
    return n;
}

bool has_fused_form(const lbm_handle* h) {
    return h->p.dtype == LBM_DTYPE_F32 && h->p.kernel == LBM_KERNEL_AUTO &&
           (h->p.mode == LBM_MODE_PHYSICS ? core_has(h->p.collision) : h->p.arith == LBM_ARITH_FAST);
}

// Lattices from this size on may take fused steps.  Below it a launch has too few windows and segments to hide the
// latency of a row: 1000 x 700 ran 10.4 us a step in single steps and 11.1 fused (600 x 375 6.3 and 7.0).
constexpr size_t FUSED_CELLS = 800000, FUSED_WALLS = 850000;

// Whether T fused steps are faster than T single ones.  Time of single steps over that of fused ones, measured over
// widths of 64 to 60,000 columns and 0.8 to 8 million cells, two steps a launch / three:
//   * BGK in a periodic box 1.15 to 1.55 / 1.3 to 2.1 from 0.8 million cells on.  Walls and faces sit in the first and the
//     last window, which then hold up a short pass: cavities 0.87 to 1.1 / 0.87 to 1.1 at 0.82 million, 1.07 to 1.2 at 1.25;
//     channels 0.87 to 1.0 at 0.82, 0.97 to 1.1 / 1.0 to 1.1 at 1.25 million.  KBC, whose rows take longer, the same
//     0.3 million cells later (cavities 0.83 to 1.0 at 0.82 million, 1.0 to 1.25 at 1.6).
//   * The reference's rules, whose walls are stored through memory: boxes 0.72 to 0.92 / 0.84 to 1.06 at 0.82 million, 0.97
//     to 1.1 / 1.14 to 1.3 at 1.6, with a forcing column 0.66 to 0.76 / 0.74 to 0.85, 0.8 to 1.0 / 0.9 to 1.1 at 1.6 and
//     1.0 to 1.2 / 1.1 to 1.35 at 2.8 million.
//   * Columns: a window stores 60.  64 wide: 0.73 / 0.68 (channel), 121: 0.66, 181: 0.75; with three quarters of the lanes
//     filled, faces counted as 1.3 windows more, no case above these sizes is slower than 0.97 (0.8 for two steps of the
//     reference's rules: 240 wide, with a forcing column, 0.87).
//   * Rows of less than 24 cells of height: 0.7 to 0.8 at 1.25 million cells.
//   * Forcing cells, and cells beside moving walls, run a function of their own for the whole row: 1 % of such cells
//     0.9 / 0.57, one in each window 0.75 / 0.62, all 0.54 / 0.46.  A lid is one row of them.  A column of them in 50
//     windows costs nothing at 9 million cells (1.4 / 1.8), but 0.83 / 0.92 at 2.3 million.
//   * Walls inside the lattice cost single steps more than fused ones: with 10 % of the cells solid, at random, a million
//     cells gain 1.48 (BGK) and 1.35 (KBC).  In six of ten rows of the windows they lift the lines above for physics
//     mode, and in one of five they decide below FUSED_WALLS.  (Not all gain so close to the line: single obstacles in
//     0.7 % of the cells 0.9 to 1.2 / 0.8 to 1.15, narrow lattices and the reference's boxes 0.6 to 0.9.
//     tests/test_gpu_fused.py counts launches of those.)
static bool march_pays(const lbm_handle* h, int T) {
    const size_t windows = (size_t)(h->nx + MARCH_OUT - 1) / MARCH_OUT, rows = windows * (size_t)h->ny;
    const RowCounts& n = h->rows;
    if (n.rare > 2 * windows + 16 && !(h->N >= 8000000 && n.rare <= rows / 32)) return false;
    if (h->N < FUSED_WALLS) return 5 * n.inner >= rows;
    const bool faces = n.face >= (size_t)h->ny / 2, walls = n.mixed > 0;
    const bool reference = h->p.mode == LBM_MODE_REFERENCE;
    const double filled = (double)h->nx / (MARCH_OUT * ((double)windows + (faces ? 1.3 : 0.0)));
    if (filled < (reference && T == 2 ? 0.8 : 0.75) || (h->ny < 24 && walls)) return false;
    if (reference) return h->N >= (T == 3 ? (faces ? 1950000u : 1550000u) : (faces ? 2750000u : 1950000u));
    if ((!walls && !faces) || 10 * n.inner >= 6 * rows) return true;
    return h->N >= (h->p.collision == LBM_COLLISION_KBC ? 1550000u : (faces ? 1300000u : 1200000u));
}

int fused_steps(const lbm_handle* h, int left) {
    if (!has_fused_form(h) || h->p.macro_every_step || h->countdown > 0 || h->nx < MARCH_W || h->ny < 8 || h->N < FUSED_CELLS)
        return 1;
    const bool two = even_steps(h) && march_pays(h, 2);
    if (left >= 3 && !(left == 4 && two) && march_pays(h, 3)) return 3;
    return left >= 2 && two ? 2 : 1;
}

static FusedLattice fused_lattice(const lbm_handle* h) {
    return {(const float*)h->buf[h->cur], (float*)h->buf[h->cur ^ 1], h->d_flags, h->d_info, h->d_macro,
            h->nx, h->nx, h->ny, (uint32_t)h->N};
}
// launches a march kernel: its shared memory is allowed once per device, its tasks cut here
template <int T, class K, class C>
static cudaError_t march_launch(PerDevice<int>& setup, K* kernel, const C& k, lbm_handle* h, bool macro, cudaStream_t s) {
    int sms = 0;
    const cudaError_t e = setup.get(
        h->device,
        [=](int& n) {
            const cudaError_t r = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, h->device);
            return r != cudaSuccess ? r : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, march_smem(T));
        },
        &sms);
    if (e != cudaSuccess) return e;
    // Rows of a segment: 24 or more, so that the T - 1 rows it computes twice above and below stay few;
    // more where eight waves of warps are left anyway (the rows around solids take longer, and late
    // warps are short then).  With less than four waves the last one is filled: whole waves of
    // shorter segments.  4096^2 with disks ran 1.3 times faster in six to eight waves than in one;
    // without solids 4 % slower in eight than in two to four.
    const int windows = (h->nx + MARCH_OUT - 1) / MARCH_OUT;
    const long slots = (long)sms * MARCH_BLOCKS;
    int rows = std::max(24, (int)((long)h->ny * windows / (slots * 8)));
    const long waves = ((long)windows * ((h->ny + rows - 1) / rows) + slots - 1) / slots;
    if (waves < 4) {
        const long most = std::max(1L, waves * slots / windows);
        rows = std::max(8, (int)((h->ny + most - 1) / most));
    }
    const int segments = (h->ny + rows - 1) / rows;
    kernel<<<(unsigned)(windows * segments), 32, march_smem(T), s>>>(fused_lattice(h), k, rows, windows, segments, macro);
    return cudaGetLastError();
}
template <int T, int COLL, bool VEC>
static cudaError_t march_v(lbm_handle* h, bool macro, cudaStream_t s) {
    static PerDevice<int> setup;
    return march_launch<T>(setup, k_phys_march<T, COLL, VEC>, BgkConst<float2>(h->omega), h, macro, s);
}
template <int T, bool VEC>
static cudaError_t ref_v(lbm_handle* h, bool macro, cudaStream_t s) {
    static PerDevice<int> setup;
    return march_launch<T>(setup, k_ref_march<T, VEC>, RefConst<float2>(h->omega), h, macro, s);
}

template <int COLL, bool VEC>
static cudaError_t fused_c(lbm_handle* h, int K, bool macro, cudaStream_t s) {
    return K == 3 ? march_v<3, COLL, VEC>(h, macro, s) : march_v<2, COLL, VEC>(h, macro, s);
}
cudaError_t launch_fused(lbm_handle* h, int steps, bool write_macro, cudaStream_t s) {
    const bool vec = h->nx % 4 == 0;
    if (h->p.mode == LBM_MODE_REFERENCE) {
        if (steps == 3) return vec ? ref_v<3, true>(h, write_macro, s) : ref_v<3, false>(h, write_macro, s);
        return vec ? ref_v<2, true>(h, write_macro, s) : ref_v<2, false>(h, write_macro, s);
    }
    if (h->p.collision == LBM_COLLISION_KBC)
        return vec ? fused_c<LBM_COLLISION_KBC, true>(h, steps, write_macro, s) : fused_c<LBM_COLLISION_KBC, false>(h, steps, write_macro, s);
    return vec ? fused_c<LBM_COLLISION_BGK, true>(h, steps, write_macro, s) : fused_c<LBM_COLLISION_BGK, false>(h, steps, write_macro, s);
}

#ifdef LBM_BOUNDS_CHECK
cudaError_t bounds_take_fused(BoundsRecord* out) { return bounds_take_local(out); }
#endif

}  // namespace lbm
