// lbm_step_cluster.cu -- many FP32 physics-mode steps of a small lattice in one launch, the lattice kept in
// the shared memory of one cluster.
//
// Why: a 256 x 256 step is 65536 cells, a few microseconds of launch and memory latency around little
// work: chained launches took 6.1 us a step alone on the GPU, 2.05 us with three lattices on three streams.
// Sixteen blocks of a cluster hold 97 thousand cells between them, so the populations are loaded
// and stored once per launch, neighbouring bands are read through distributed shared memory, and a step
// ends with the cluster's hardware barrier instead of a launch.
//
// One copy of the lattice is enough with the AA pattern (Bailey, Myre, Walsh, Lilja & Saar, ICPP 2009):
// an even step reads population j of a cell at its neighbour c - e_j and leaves the outgoing
// population of the opposite direction there, so that the next, odd step finds all it needs in the cell's
// own slots, and writes its results there as well.  A direction that bounces back uses the cell's
// own slot instead of the solid neighbour's.  Only the outflow cells of the last column read what is
// another cell's to write: their own column's populations 3, 6 and 7, or their own 8 and 5 where that column
// is solid.  The last column's five are kept beside the lattice, one set per step parity.
//
// A warp computes rows of one window of up to 64 columns, two cells a lane, with the core's packed
// arithmetic: the state is that of single steps bit for bit.
//
// Measured, a step of a long call before and now: cavity 256^2 2.06 and 1.38 us with three lattices on three
// streams, 5.7 and 4.1 us alone; periodic 256^2 1.95 and 0.98, 4.2 and 3.0; cavity 64^2 2.06 and 0.52, 5.7
// and 1.7.  What bounds it: sixteen warps a block (126 registers a lane; 20 or 24 warps spill) that
// compute their rows one after the other at 46 % of the issue slots (fixed latencies of the arithmetic,
// the FP32 pipe), and the step's critical path: the warps at walls, whose rows take 1.5 times a plain one,
// and the barrier.  (A barrier that orders shared memory only gave 4 %; selecting a bounce-back's address
// instead of branching made the cavity 2.2 times as fast.)
#include <algorithm>

#include "lbm_fused.cuh"
#include "lbm_internal.h"

namespace lbm {

constexpr int CL_BLOCKS = 16;     // blocks of the cluster: bands of rows
constexpr int CL_THREADS = 512;
constexpr int CL_WARPS = CL_THREADS / 32;
constexpr int CL_CELLS = 5984;    // cells of a block's band
constexpr int CL_COLUMNS = 64 * CL_WARPS;  // widest lattice: a warp stays in one window
constexpr int CL_PLANE = 4 * CL_CELLS;
constexpr int CL_FLAGS = 9 * CL_PLANE;              // byte offsets in shared memory
constexpr int CL_EDGE = CL_FLAGS + 2 * CL_CELLS;    // last column's outgoing populations, for two steps
constexpr int CL_KEPT = 5;                          // 3, 6, 7, 8, 5
constexpr int CL_ROW_BYTES = 8 * CL_KEPT + 8;       // those, and the first column's inlet velocity
constexpr int CL_ROWS = (227 * 1024 - CL_EDGE) / CL_ROW_BYTES;  // most rows of a band: the rest of a block's 227 KB
constexpr int cluster_smem(int rows) { return CL_EDGE + CL_ROW_BYTES * rows; }

__host__ __device__ constexpr int cluster_kept(int i) { return i == 0 ? 3 : (i < 3 ? 5 + i : (i == 3 ? 8 : 5)); }

struct ClusterShape {
    int windows, width;  // windows of a row, and the columns of all but the last one
    int sets;            // warps that share a window
    int rows;            // rows of the largest band
};

__device__ __forceinline__ float lds(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ float ldc(uint32_t a) {  // a: an address in the cluster's shared memory
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void stc(uint32_t a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ uint32_t where(unsigned m, uint32_t a, uint32_t b) {  // m ? a : b, never a branch
    uint32_t r;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tselp.b32 %0, %2, %3, p;\n\t}" : "=r"(r) : "r"(m), "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ bool solid_cell(unsigned f) {  // (a bit test: comparisons become a jump table)
    return ((1u << LBM_BOUNDARY | 1u << LBM_OBSTACLE) >> (f & FL_MAT_MASK)) & 1u;
}
__device__ __forceinline__ uint32_t of_block(uint32_t a, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// a lane's place: its two cells are 32 columns apart; byte offsets in a row of the first cell and of the
// columns beside the cells (the second cell's left one lies in the same window)
struct ClusterColumns {
    int x;               // column of the first cell
    bool va, vb;         // cells of the window
    uint32_t c, ma, pa, pb;
    __device__ __forceinline__ uint32_t first(int ex) const { return ex == 1 ? ma : (ex == -1 ? pa : c); }
    __device__ __forceinline__ uint32_t second(int ex) const { return ex == 1 ? c + 124 : (ex == -1 ? pb : c + 128); }
};
// A row of the band and its neighbours; far: from an address of this block to the same in the cluster's memory
struct ClusterRow {
    uint32_t row, up, down, far;
    uint32_t kept_out;                    // where the last column's populations go
    uint32_t kept, kept_up, kept_down;    // and those of the step before
    uint32_t inlet;                       // velocity of the first column's inlet
    int kept_stride;
    int y, cls;
    unsigned fq;
    bool last_column;
};

// what moving walls add to the populations that a row's cells bounce back; a solid cell's own slots 0 and 1
// hold its velocity
template <int J, bool FAR>
__device__ __forceinline__ void moving_wall(float2& d, const ClusterRow& t, const ClusterColumns& c) {
    if (!(t.cls & (1 << (FL_DIR_SHIFT + J)))) return;  // warp-uniform
    const auto term = [&](unsigned f, bool second) {
        const bool moves = (f & FL_MOVING) && (f & (1u << (FL_DIR_SHIFT + J)));
        const int ex = (f & FL_MAT_MASK) == LBM_OUTLET && EX(J) == -1 ? 0 : EX(J);
        const uint32_t at = (EY(J) == 1 ? t.up : (EY(J) == -1 ? t.down : t.row)) + (second ? c.second(moves ? ex : 0) : c.first(moves ? ex : 0));
        constexpr bool other = FAR && EY(J) != 0;
        const float vx = other ? ldc(at) : lds(at), vy = other ? ldc(at + CL_PLANE) : lds(at + CL_PLANE);
        const float uw = (EX(J) == 0 ? 0.0f : (float)EX(J) * vx) + (EY(J) == 0 ? 0.0f : (float)EY(J) * vy);
        return moves && uw != 0.0f ? uw : 0.0f;
    };
    const float ua = term(t.fq & 0xffffu, false), ub = term(t.fq >> 16, true);
    if (ua != 0.0f) d.x = add_rn(d.x, mul_rn(6.0f * PW<float>(J), ua));
    if (ub != 0.0f) d.y = add_rn(d.y, mul_rn(6.0f * PW<float>(J), ub));
}
// inlet velocities: the first column's are in shared memory
__device__ __forceinline__ InletVel cluster_inlet(unsigned fq, const ClusterRow& t, const ClusterColumns& c, const FusedLattice& L) {
    const bool here = (fq & FL_MAT_MASK) == LBM_INLET && c.x == 0;
    InletVel v = inlet_vel(here ? fq & ~FL_MAT_MASK : fq, c.x, c.x + 32, t.y, L);
    if (here) {
        v.ax = lds(t.inlet);
        v.ay = lds(t.inlet + 4);
    }
    return v;
}

// One row.  PULL: an even step.  MIXED: not a plain row.  FAR: a neighbour row is another block's (up and
// down are addresses in the cluster's memory).  LAST: the results go to global memory.
template <int COLL, bool PULL, bool MIXED, bool FAR, bool LAST>
__device__ __forceinline__ void cluster_row(const FusedLattice& L, const BgkConst<float2>& k, const ClusterColumns& c,
                                            const ClusterRow& t, bool macro) {
    float2 d[9], o[9], rho, nux, nuy;
    const unsigned fa = t.fq & 0xffffu, fb = t.fq >> 16;
    // directions whose bounce-back uses the cell's own slot (an outflow cell's 6 and 7 are beside the lattice)
    constexpr unsigned OWN67 = 1u << (FL_DIR_SHIFT + 6) | 1u << (FL_DIR_SHIFT + 7);
    const unsigned ba = MIXED && PULL ? fa & ~((fa & FL_MAT_MASK) == LBM_OUTLET ? OWN67 : 0u) : 0u;
    const unsigned bb = MIXED && PULL ? fb & ~((fb & FL_MAT_MASK) == LBM_OUTLET ? OWN67 : 0u) : 0u;
    uint32_t pa[9], pb[9];  // where population j of the two cells comes from, and INV(j) goes to
#pragma unroll
    for (int j = 0; j < 9; ++j) {
        const bool other = PULL && FAR && EY(j) != 0;  // an address in the cluster's memory
        const uint32_t self = t.row + c.c + CL_PLANE * INV(j) + (other ? t.far : 0u);
        if (PULL) {
            const uint32_t r = (EY(j) == 1 ? t.up : (EY(j) == -1 ? t.down : t.row)) + CL_PLANE * j;
            pa[j] = r + c.first(EX(j));
            pb[j] = r + c.second(EX(j));
            if (MIXED && j) {
                pa[j] = where(ba & (1u << (FL_DIR_SHIFT + j)), self, pa[j]);
                pb[j] = where(bb & (1u << (FL_DIR_SHIFT + j)), self + 128, pb[j]);
            }
        } else {
            pa[j] = self;
            pb[j] = self + 128;
        }
        d[j] = other ? make_float2(ldc(pa[j]), ldc(pb[j])) : make_float2(lds(pa[j]), lds(pb[j]));
    }
    if (MIXED) {
        if (t.cls & (ROW_FACE | ROW_RARE)) {
            // an outflow cell (in the last column) pulls 3, 6 and 7 from its own column
            const auto outflow = [&](unsigned f, bool first) {
                if ((f & FL_MAT_MASK) != LBM_OUTLET) return;
                const int n = t.kept_stride;
                const float e3 = lds(t.kept);
                const auto beside = [](uint32_t at) { return FAR ? ldc(at) : lds(at); };
                const float e6 = f & (1u << (FL_DIR_SHIFT + 6)) ? lds(t.kept + 3 * n) : beside(t.kept_down + n);
                const float e7 = f & (1u << (FL_DIR_SHIFT + 7)) ? lds(t.kept + 4 * n) : beside(t.kept_up + 2 * n);
                (first ? d[3].x : d[3].y) = e3;
                (first ? d[6].x : d[6].y) = e6;
                (first ? d[7].x : d[7].y) = e7;
            };
            outflow(fa, true);
            outflow(fb, false);
            __syncwarp();
        }
        if (t.cls & ROW_RARE) {
            moving_wall<1, FAR>(d[1], t, c);
            moving_wall<2, FAR>(d[2], t, c);
            moving_wall<3, FAR>(d[3], t, c);
            moving_wall<4, FAR>(d[4], t, c);
            moving_wall<5, FAR>(d[5], t, c);
            moving_wall<6, FAR>(d[6], t, c);
            moving_wall<7, FAR>(d[7], t, c);
            moving_wall<8, FAR>(d[8], t, c);
        }
        const unsigned still = t.fq & ~(FL_MOVING | FL_MOVING << 16);  // walls are done: an inlet beside one is an inlet
        if (t.cls & (ROW_FACE | ROW_RARE)) face_cells(d, still, cluster_inlet(still, t, c, L), k.omega);
    }
    float2 drho, jx, jy;
    core_moments<float2>(d, drho, jx, jy);
    core_collide<COLL, float2>(d, k, drho, jx, jy, o, rho, nux, nuy);
    if (MIXED && (t.cls & ROW_RARE))
        rare_cells<COLL>(d, t.fq & ~(FL_MOVING | FL_MOVING << 16), c.x, c.x + 32, t.y, L, k.omega, o, rho, nux, nuy);
    const bool ga = !MIXED || !solid_cell(fa), gb = !MIXED || !solid_cell(fb);
    if (LAST) {
        RowOut out;
        out.row = (uint32_t)t.y * (uint32_t)L.pitch;
        out.ca = c.x;
        out.sa = c.va;
        out.sb = c.vb;
        store_row(L, out, ga, gb, macro, o, rho, nux, nuy);
        return;
    }
    const bool wa = c.va && ga, wb = c.vb && gb;
#pragma unroll
    for (int j = 0; j < 9; ++j) {  // (after an odd step every population is in its own plane again)
        if (PULL && FAR && EY(j) != 0) {
            if (wa) stc(pa[j], o[INV(j)].x);
            if (wb) stc(pb[j], o[INV(j)].y);
        } else {
            if (wa) sts(pa[j], o[INV(j)].x);
            if (wb) sts(pb[j], o[INV(j)].y);
        }
    }
    if (t.last_column) {
        const bool la = c.va && c.x == L.nx - 1, lb = c.vb && c.x + 32 == L.nx - 1;
#pragma unroll
        for (int i = 0; i < CL_KEPT; ++i) {
            if (la) sts(t.kept_out + i * t.kept_stride, o[cluster_kept(i)].x);
            if (lb) sts(t.kept_out + i * t.kept_stride, o[cluster_kept(i)].y);
        }
    }
}

template <int COLL>
__global__ void __launch_bounds__(CL_THREADS, 1)
    k_phys_cluster(const __grid_constant__ FusedLattice Lin, const __grid_constant__ BgkConst<float2> kin, ClusterShape shape,
                   int steps, bool macro) {
    extern __shared__ __align__(16) unsigned char cluster_mem[];
    const FusedLattice& L = Lin;
    const uint32_t f = (uint32_t)__cvta_generic_to_shared(cluster_mem);
    uint16_t* flags = reinterpret_cast<uint16_t*>(cluster_mem + CL_FLAGS);
    const int rank = (int)blockIdx.x, before = (rank + CL_BLOCKS - 1) % CL_BLOCKS, after = (rank + 1) % CL_BLOCKS;
    const int base = L.ny / CL_BLOCKS, extra = L.ny % CL_BLOCKS;
    const int rows = base + (rank < extra), rows_before = base + (before < extra);
    const int y0 = rank * base + min(rank, extra);
    const int kept_stride = 4 * shape.rows;
    const uint32_t inlets = f + CL_EDGE + 2 * CL_KEPT * kept_stride;

    // the band, population by population: consecutive cells of a plane
    const uint32_t first = (uint32_t)y0 * (uint32_t)L.nx;
    const auto load = [&](auto cells) {
        constexpr int CELLS = decltype(cells)::value;
        for (int c = CELLS * (int)threadIdx.x; c < rows * L.nx; c += CELLS * CL_THREADS) {
            if (!in_bounds((unsigned long long)first + c + (CELLS - 1), L.N, BS_FUSED_PULL)) continue;
#pragma unroll
            for (int j = 0; j < 9; ++j) cp_async_to<4 * CELLS>(f + CL_PLANE * j + 4 * c, L.A + (size_t)j * L.N + first + c);
            if constexpr (CELLS == 4) cp_async_to<8>(f + CL_FLAGS + 2 * c, L.flags + first + c);
            else flags[c] = L.flags[first + c];
        }
    };
    if (L.nx % 4 == 0) load(std::integral_constant<int, 4>{});  // every band starts at a multiple of four cells
    else load(std::integral_constant<int, 1>{});
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int c = (int)threadIdx.x; c < rows * L.nx; c += CL_THREADS) {
        if (!is_solid((int)(flags[c] & FL_MAT_MASK)) || !in_bounds((unsigned long long)first + c, L.N, BS_FUSED_INFO)) continue;
        const lbm_lattice_info wall = L.info[first + c];
        sts(f + 4 * c, wall.vx);
        sts(f + CL_PLANE + 4 * c, wall.vy);
    }
    for (int r = (int)threadIdx.x; r < rows; r += CL_THREADS) {
        const uint32_t e = f + 4 * (r * L.nx + L.nx - 1), to = f + CL_EDGE + CL_KEPT * kept_stride + 4 * r;  // as of an odd step
#pragma unroll
        for (int i = 0; i < CL_KEPT; ++i) sts(to + i * kept_stride, lds(e + CL_PLANE * cluster_kept(i)));
        const lbm_lattice_info in = fused_info(L.info, 0, y0 + r, L.pitch, L.ny);
        sts(inlets + 8 * r, in.vx);
        sts(inlets + 8 * r + 4, in.vy);
    }
    cluster_barrier();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w = warp / shape.sets, sub = warp % shape.sets, x0 = w * shape.width, end = min(shape.width, L.nx - x0);
    const int count = w < shape.windows && sub < rows ? (rows - sub + shape.sets - 1) / shape.sets : 0;  // the warp's rows
    ClusterColumns c;
    c.x = x0 + lane;  // (columns past the window's end are read, as whatever follows in the plane, and not stored)
    c.va = lane < end;
    c.vb = lane + 32 < end;
    c.c = 4 * c.x;
    c.ma = 4 * wrap_to(c.x - 1, L.nx);
    c.pa = 4 * wrap_to(c.x + 1, L.nx);
    c.pb = 4 * wrap_to(c.x + 33, L.nx);
    hold(c.c); hold(c.ma); hold(c.pa); hold(c.pb);
    const uint32_t prev = of_block(f, before), next = of_block(f, after), far = of_block(f, rank) - f;
    const int pitch = 4 * L.nx;
    const auto flags_of = [&](int r) {
        const uint16_t* q = flags + r * L.nx;
        return (c.va ? (unsigned)q[c.x] : FL_PLAIN) | (c.vb ? (unsigned)q[c.x + 32] : FL_PLAIN) << 16;
    };
    unsigned plain = 0, solid = 0;  // rows of the warp, by number: plain ones, and those without a cell to compute
    for (int i = 0; i < count; ++i) {
        const unsigned fq = flags_of(sub + i * shape.sets);
        if (row_class(fq) == ROW_PLAIN) plain |= 1u << i;
        if (__all_sync(0xffffffffu, (!c.va || solid_cell(fq)) && (!c.vb || solid_cell(fq >> 16))))
            solid |= 1u << i;
    }
    BgkConst<float2> k = kin;  // in registers: packed instructions take no other operands
    hold(k.om); hold(k.omn); hold(k.om1); hold(k.w1); hold(k.w5); hold(k.w31); hold(k.w35); hold(k.c45);
    hold(k.one); hold(k.mone); hold(k.m15);

    const auto step = [&](auto pull, auto last, int odd) {
        constexpr bool PULL = decltype(pull)::value, LAST = decltype(last)::value;
        const int set = odd ? CL_KEPT * kept_stride : 0;  // of the last column's populations: written in this step
#pragma unroll 1
        for (int i = 0; i < count; ++i) {
            if (!LAST && (solid >> i & 1)) continue;
            const int r = sub + i * shape.sets;
            const bool edge = r == 0 || r + 1 == rows;
            ClusterRow t;
            t.row = f + pitch * r;
            t.far = far;
            t.last_column = x0 + end == L.nx;
            t.kept_stride = kept_stride;
            t.kept_out = f + CL_EDGE + set + 4 * r;
            if (!LAST && (plain >> i & 1) && !(PULL && edge)) {
                t.up = t.row - pitch;
                t.down = t.row + pitch;
                t.fq = FL_PLAIN | FL_PLAIN << 16;
                cluster_row<COLL, PULL, false, false, false>(L, k, c, t, macro);
                continue;
            }
            t.y = y0 + r;
            t.fq = flags_of(r);
            t.cls = row_class(t.fq);
            t.inlet = inlets + 8 * r;
            const uint32_t kept = CL_EDGE + CL_KEPT * kept_stride - set;
            t.kept = f + kept + 4 * r;
            if (!LAST && !edge) {
                t.up = t.row - pitch;
                t.down = t.row + pitch;
                t.kept_up = t.kept - 4;
                t.kept_down = t.kept + 4;
                cluster_row<COLL, PULL, true, false, false>(L, k, c, t, macro);
            } else {
                t.up = r > 0 ? t.row - pitch + far : prev + pitch * (rows_before - 1);
                t.down = r + 1 < rows ? t.row + pitch + far : next;
                t.kept_up = r > 0 ? t.kept - 4 + far : prev + kept + 4 * (rows_before - 1);
                t.kept_down = r + 1 < rows ? t.kept + 4 + far : next + kept;
                cluster_row<COLL, PULL, true, true, LAST>(L, k, c, t, macro);
            }
        }
        __syncwarp();
        cluster_barrier();  // (after the last step too: no block leaves while another may read its rows)
    };
#pragma unroll 1
    for (int s = 0; s + 1 < steps; ++s) {
        if (s & 1) step(std::false_type{}, std::false_type{}, 1);
        else step(std::true_type{}, std::false_type{}, 0);
    }
    if (steps & 1) step(std::true_type{}, std::true_type{}, 0);
    else step(std::false_type{}, std::true_type{}, 1);
}

constexpr int CL_MOST_STEPS = 1024;  // of a launch, which ends within a few milliseconds

static void cluster_config(cudaLaunchConfig_t& c, cudaLaunchAttribute& a, int smem, cudaStream_t s) {
    c.gridDim = dim3(CL_BLOCKS);
    c.blockDim = dim3(CL_THREADS);
    c.dynamicSmemBytes = (size_t)smem;
    c.stream = s;
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim = {CL_BLOCKS, 1, 1};
    c.attrs = &a;
    c.numAttrs = 1;
}
static int cluster_rows(const lbm_handle* h) { return (h->ny + CL_BLOCKS - 1) / CL_BLOCKS; }
static int cluster_windows(int nx) { return (nx + 63) / 64; }
static int cluster_sets(int nx) { return CL_WARPS / cluster_windows(nx); }

// the kernel's set-up on a device; 0: no such cluster fits it
template <int COLL>
static cudaError_t cluster_ready(int device, int* ready) {
    static PerDevice<int> setup;
    return setup.get(
        device,
        [](int& n) {
            const void* kernel = (const void*)k_phys_cluster<COLL>;
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, cluster_smem(CL_ROWS));
            cudaLaunchConfig_t c = {};
            cudaLaunchAttribute a;
            cluster_config(c, a, cluster_smem(CL_ROWS), nullptr);
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, kernel, &c);
            return e;
        },
        ready);
}

int cluster_steps(const lbm_handle* h, int left) {
    if (left < 4 || h->p.mode != LBM_MODE_PHYSICS || !has_fused_form(h) || h->p.macro_every_step || h->countdown > 0 ||
        !h->outlets_last || h->ny < CL_BLOCKS || h->nx > CL_COLUMNS || cluster_rows(h) > CL_ROWS ||
        cluster_rows(h) * h->nx > CL_CELLS)
        return 1;
    // Rows that a warp computes one after the other, and the calls that are long enough for them.  Steps of
    // 64^2 cells (one row) ran 4.3 times faster with a lattice to themselves and 6.1 times with three on as
    // many streams (calls of 64 steps; of 4 steps 1.4 and 2.3), of 192^2 (three) 1.9 and 2.8, of 256^2
    // (four) 1.4 and 2.0 in a periodic box and 1.4 and 1.5 in a cavity; calls of 4 steps lose there (0.8 and
    // 1.0), and 300^2 (seven rows) lost up to a third alone.  Inlets and outflows, and KBC, take longer a row:
    // 192^2 gains 1.0 to 1.2 alone and 1.4 to 1.8 in calls of 16 and 64 steps, 256^2 ran 0.8 alone.
    const int windows = cluster_windows(h->nx), sets = cluster_sets(h->nx), warp_rows = (cluster_rows(h) + sets - 1) / sets;
    const bool kbc = h->p.collision == LBM_COLLISION_KBC, costly = h->faces || kbc;
    if (warp_rows > (costly ? 3 : 4) || left < (costly ? (warp_rows < 3 ? 6 : 16) : 2 * warp_rows + 2)) return 1;
    // A step ends with its slowest warp.  Forcing cells run a function of their own, in memory, for the whole row: with
    // 1 % of them BGK ran 1.2 to 1.7 times as fast as single steps at 128^2 (alone 0.87 to 1.4), 0.8 to 0.9 at 192^2, 0.65 to
    // 0.75 at 256^2, KBC 1.2 to 1.5 at 64^2 (alone 0.85 to 1.45), 1.0 to 1.3 at 128^2 (0.7 to 1.2), 0.6 at 192^2.  Moving walls through the
    // lattice: 1.3 and more, but 0.9 to 1.05 at 256^2 (alone 0.7) and, with KBC, 1.04 to 1.15 at 192^2 (0.8).
    const RowCounts& n = h->rows;
    if (n.forced > 16 && (warp_rows > 1 || (kbc && cluster_rows(h) * windows > 4))) return 1;
    if (n.rare > 2ull * windows + 48 && (warp_rows >= 4 || (kbc && warp_rows >= 3))) return 1;
    int ready = 0;
    const cudaError_t e = h->p.collision == LBM_COLLISION_KBC ? cluster_ready<LBM_COLLISION_KBC>(h->device, &ready)
                                                              : cluster_ready<LBM_COLLISION_BGK>(h->device, &ready);
    if (e != cudaSuccess) cudaGetLastError();  // not for the next launch's check
    if (e != cudaSuccess || ready < 1) return 1;
    const int steps = std::min(left, CL_MOST_STEPS);
    return steps % 2 == 1 || even_steps(h) ? steps : steps - 1;
}

template <int COLL>
static cudaError_t cluster_c(lbm_handle* h, int steps, bool macro, cudaStream_t s) {
    // (solid cells' slots are not written)
    const FusedLattice L = {(const float*)h->buf[h->cur], (float*)h->buf[h->cur ^ 1], h->d_flags, h->d_info,
                            h->d_macro, h->nx, h->nx, h->ny, (uint32_t)h->N};
    ClusterShape shape;
    shape.windows = cluster_windows(h->nx);
    shape.width = (h->nx + shape.windows - 1) / shape.windows;
    shape.sets = cluster_sets(h->nx);
    shape.rows = cluster_rows(h);
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute a;
    cluster_config(c, a, cluster_smem(shape.rows), s);
    return cudaLaunchKernelEx(&c, k_phys_cluster<COLL>, L, BgkConst<float2>(h->omega), shape, steps, macro);
}
cudaError_t launch_cluster(lbm_handle* h, int steps, bool write_macro, cudaStream_t s) {
    return h->p.collision == LBM_COLLISION_KBC ? cluster_c<LBM_COLLISION_KBC>(h, steps, write_macro, s)
                                               : cluster_c<LBM_COLLISION_BGK>(h, steps, write_macro, s);
}

void cluster_cells(lbm_handle* h, const lbm_lattice_info* info, bool also) {
    const bool fits = h->N <= (size_t)CL_BLOCKS * CL_CELLS;  // else nobody asks
    bool last = fits, faces = false;
    for (size_t c = 0; fits && c < h->N; ++c) {
        faces |= info[c].material == LBM_INLET || info[c].material == LBM_OUTLET;
        last &= info[c].material != LBM_OUTLET || (int)(c % (size_t)h->nx) == h->nx - 1;
    }
    h->outlets_last = last && (!also || h->outlets_last);
    h->faces = faces || (also && h->faces);
}

#ifdef LBM_BOUNDS_CHECK
cudaError_t bounds_take_cluster(BoundsRecord* out) { return bounds_take_local(out); }
#endif

}  // namespace lbm
