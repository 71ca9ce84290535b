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

// Whether fused steps are faster than single ones.  Time of single steps over that of fused ones, two steps a launch /
// three, with three lattices on three streams and with one alone:
//   * 420 to 5000 columns, 0.82 million cells.  Periodic BGK 1.5 / 1.7, alone 1.15 / 1.3; cavity 1.45 / 1.6, alone
//     1.0 / 1.0; channel 1.4 / 1.5, alone 0.95 / 0.95.  KBC 1.35 / 1.3, 1.25 / 1.2 and 1.2 / 1.1, alone 1.1, 0.95 and 0.9.  The
//     reference's box 1.35 / 1.4, alone 0.8 / 0.9, with a forcing column 1.27 / 1.33, alone 0.7 / 0.8.  At 2 million 1.5 / 2.0,
//     1.5 / 2.0, 1.5 / 1.9, KBC 1.5 to 1.55, reference 1.5 / 1.75; alone all gain.  (A lattice alone near the line is held
//     up by its first and last windows, with walls and faces, in a pass too short to hide them.)
//   * Columns.  A window stores 60, windows with faces cost 1.5 to 2 more, walls up to 0.6; a width off a multiple of four
//     copies cell by cell (0.75 of the speed, KBC 0.9).  Channels of 64, 100, 121, 150 and 181 columns 0.65 / 0.58,
//     1.0 / 0.95, 0.63 / 0.62, 0.9 / 0.87 and 0.75 / 0.72, of 240 and 300 1.25 / 1.3 and 1.4 / 1.45.  What is left of a
//     window, times the gain of a wide lattice, has to reach 1: of 398 lattices above the lines (64 to 5000 columns, 0.8
//     to 2.8 million cells, three at a time) two are slower than 0.95, at 0.9; of 178 below, seven gain more than 1.2.
//   * Less than 24 rows with walls: 0.7 to 0.8.
//   * Forcing cells, and cells beside moving walls, run a function of their own for the whole row: 1 % of such cells
//     1.0 / 0.5, one in each window 0.8 / 0.6, all 0.55 / 0.45.  A lid is one row of them; a column of them in 25 windows 1.4 /
//     1.6 (alone 0.83 / 0.92), twice in 17 windows 1.3 / 1.2 (0.8 / 0.7).
//   * Walls inside the lattice cost single steps more than fused ones: with 10 % of the cells solid, at random, a million
//     cells gain 1.85 / 2.1 (alone 1.5).  So in one of five rows of the windows they decide below FUSED_WALLS.  (Narrow
//     lattices lose there all the same, 0.6 to 0.9: tests/test_gpu_fused.py counts launches of those.)
static bool march_pays(const lbm_handle* h) {
    const size_t windows = (size_t)(h->nx + MARCH_OUT - 1) / MARCH_OUT, rows = windows * (size_t)h->ny;
    const RowCounts& n = h->rows;
    if (n.rare > std::max(2 * windows + 16, rows / 16)) return false;
    if (h->N < FUSED_WALLS && 5 * n.inner >= rows) return true;
    const bool kbc = h->p.collision == LBM_COLLISION_KBC, reference = h->p.mode == LBM_MODE_REFERENCE;
    const bool faces = n.face >= (size_t)h->ny / 2, walls = n.mixed > 0;
    if (h->ny < 24 && walls) return false;
    const double more = faces ? (kbc ? 2.0 : 1.5) : (walls ? (kbc || reference ? 0.6 : 0.3) : 0.0);
    const double copies = h->nx % 4 == 0 ? 1.0 : (kbc ? 0.9 : 0.75);
    const double left = copies * h->nx / (MARCH_OUT * ((double)windows + more));
    return left >= (kbc ? (faces && h->N < 1200000 ? 0.72 : 0.63) : (reference ? 0.6 : 0.53));
}

int fused_steps(const lbm_handle* h, int left) {
    if (left < 2 || !has_fused_form(h) || h->p.macro_every_step || h->countdown > 0 || h->nx < MARCH_W || h->ny < 8 ||
        h->N < FUSED_CELLS || !march_pays(h))
        return 1;
    const bool even = even_steps(h);
    if (left >= 3 && !(left == 4 && even)) return 3;
    return even ? 2 : 1;
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
