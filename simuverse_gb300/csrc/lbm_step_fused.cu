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

// Lattices from this size on take fused steps.  Below it a launch has too few windows and segments
// to hide the latency of a row: 1000 x 700 runs 10.4 us a step in single steps and 11.1 fused when it
// has the GPU to itself, 1000 x 1000 12.5 and 8.2 (and 600 x 375 6.3 and 7.0).
constexpr size_t FUSED_CELLS = 800000;

int fused_steps(const lbm_handle* h, int left) {
    if (h->p.dtype != LBM_DTYPE_F32 || h->p.kernel != LBM_KERNEL_AUTO || h->p.macro_every_step || h->countdown > 0 ||
        h->nx < MARCH_W || h->ny < 8 || h->N < FUSED_CELLS)
        return 1;
    if (h->p.mode == LBM_MODE_PHYSICS ? !core_has(h->p.collision) : h->p.arith != LBM_ARITH_FAST) return 1;
    const bool even = even_steps(h);
    if (left >= 3 && !(left == 4 && even)) return 3;
    return left >= 2 && even ? 2 : 1;
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
