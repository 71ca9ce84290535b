// lbm_closure_tc.cuh -- the closure network's inference as one fused kernel on the 5th-generation
// tensor cores (tcgen05.mma, accumulators in tensor memory).  Included by lbm_closure.cu inside
// namespace lbm::closure, after the per-cell helpers (load_dev, non_equilibrium, pack_bf16x2).
//
// y = conv3(relu(conv2(relu(conv1(x0))))) of the whole periodic field, with x0 = the features of
// the lattice's populations computed on the fly: the activations never leave shared memory and
// tensor memory.
//
// Tiling.  A CTA owns a strip of OUT_W = 124 output columns and TC_ROWS = 32 output rows and walks
// down its rows.  A row of every activation -- input features (16 channels), layer-1 and layer-2
// outputs (32 channels, BF16) -- holds POS = 130 positions, position p being column x0 - 3 + p
// (wrapped): one MMA row block of 128 positions plus the two positions a 3-wide stencil reads
// beyond them.  Output position p of a layer is MMA row p - 1; each layer loses one position per
// side, so layer 3 is valid at positions 3..126 = the strip's 124 columns.
//
// Rows stacked along N.  A layer reads each of its input rows r once: for each column shift dx
// (and 16-channel chunk) one MMA multiplies the 128 positions starting at dx by the weights of
// all three row taps dy side by side (N = 3 x cout), contributing to output rows r + 1 - dy.
// Output row o accumulates in tensor-memory slot o % 3 (cout columns each); the weights are
// stored in the row-tap order [2, 1, 0, 2, 1], so the order a row r needs -- slot k receives
// tap (r + 1 - k) mod 3 -- is three consecutive blocks starting at (1 - r) mod 3.  A row is
// complete after its last contributing input row; the epilogue reads it, zeroes the slot with
// tcgen05.st for row o + 3, and writes the BF16 activations (bias, ReLU) to the next layer's
// input, double-buffered in shared memory.  Per input row: layer 1 3 MMAs of M128 N96 K16,
// layer 2 6 of M128 N96 K16, layer 3 6 of M128 N48 K16.
//
// Operands.  Shared-memory matrices in the canonical K-major layout without swizzle: core
// matrices of 8 rows x 16 bytes (8 BF16 channels); an activation row stores its channel groups as
// planes of POS x 16 bytes, so the descriptor's leading (K-direction) byte offset is POS * 16 and
// its stride (8-row) offset 128; weights [dx][channel group][row-tap block 5][cout][8] with leading
// offset 5 * cout * 16.  The descriptor encoding and the accumulator lane layout (warp w reads
// TMEM lanes 32 (w % 4) .. + 31 = MMA rows with tcgen05.ld 32x32b) were checked against a host
// product before use.  The CTA's two warpgroups split every epilogue by accumulator columns.
//
// Schedule.  Step a issues one batch: layer 1 on input row a, layer 2 on layer-1 row a - 2,
// layer 3 on layer-2 row a - 4 (rows finished in earlier steps), committed to one mbarrier.
// While the batch runs the block loads the populations of input row a + 1; after it, the
// epilogues finish layer-1 row a - 1, layer-2 row a - 3 and layer-3 row a - 5 (the output row,
// to global memory) and store the features of row a + 1.  Generic shared-memory writes are fenced
// to the async proxy before the next batch.  Thread 0 waits on the mbarrier with a 1 s limit
// and the block follows its outcome; a timed-out wait records LBM_ERR_TIMEOUT, waits (bounded)
// for the MMAs in flight, frees the tensor memory and leaves.
#pragma once

namespace tc {

constexpr int POS = 130;           // ring-row positions: columns x0 - 3 .. x0 + 126
constexpr int OUT_W = 124;         // output columns per strip (positions 3 .. 126)
constexpr int TC_ROWS = 32;        // output rows per CTA
constexpr int TC_THREADS = 256;  // two warpgroups: each epilogue is split between them by columns
constexpr int PLANE = POS * 16;    // bytes of one 8-channel group of a ring row
constexpr int IN_ROW = 2 * PLANE;  // 16 input channels
constexpr int H_ROW = 4 * PLANE;   // 32 hidden channels
constexpr int OFF_IN = 0;                        // input rows, double-buffered
constexpr int OFF_L1 = OFF_IN + 2 * IN_ROW;      // layer-1 rows, double-buffered
constexpr int OFF_L2 = OFF_L1 + 2 * H_ROW;       // layer-2 rows, double-buffered
constexpr int OFF_W1 = OFF_L2 + 2 * H_ROW;       // [dx 3][group 2][block 5][cout 32] x 16 B
constexpr int OFF_W2 = OFF_W1 + 3 * 2 * 5 * 32 * 16;  // [3][4][5][32]
constexpr int OFF_W3 = OFF_W2 + 3 * 4 * 5 * 32 * 16;  // [3][4][5][16]
constexpr int OFF_BIAS = OFF_W3 + 3 * 4 * 5 * 16 * 16;
constexpr int OFF_BAR = OFF_BIAS + 80 * 4;
constexpr int OFF_TSLOT = OFF_BAR + 8;
constexpr int SMEM_BYTES = ((OFF_TSLOT + 4 + 127) / 128) * 128;
// accumulators: layer 1 columns 0-95 (3 row slots of 32), layer 2 96-191, layer 3 192-239
constexpr int TM_L1 = 0, TM_L2 = 96, TM_L3 = 192;
constexpr int TMEM_COLS = 256;
constexpr unsigned long long WAIT_NS = 1000000000ull;

static_assert(OFF_L1 % 16 == 0 && OFF_L2 % 16 == 0 && OFF_W1 % 16 == 0 && OFF_W2 % 16 == 0 && OFF_W3 % 16 == 0,
              "operands must start on 16-byte boundaries");
static_assert(OFF_BAR % 8 == 0, "mbarriers are 8-byte aligned");
static_assert(2 * SMEM_BYTES <= 227 * 1024, "two CTAs per SM");

__device__ __forceinline__ unsigned su32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: start address, leading (K) and stride (8-row) byte offsets,
// descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t sdesc(unsigned addr, unsigned lbo, unsigned sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}
// instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M x N
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma(unsigned dtmem, uint64_t a, uint64_t b, uint32_t id, unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
        "l"(a), "l"(b), "r"(id), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ bool elect_one() {  // one thread of a converged warp
    unsigned p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0u;
}
__device__ __forceinline__ bool bar_try(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool bar_wait_bounded(unsigned bar, unsigned parity) {
    if (bar_try(bar, parity)) return true;
    const unsigned long long t0 = now_ns();
    while (!bar_try(bar, parity))
        if (now_ns() - t0 > WAIT_NS) return false;
    return true;
}

// 16 / 8 consecutive accumulator columns of this thread's lane
__device__ __forceinline__ void tmem_ld16(unsigned taddr, float (&v)[16]) {
    unsigned r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

// two such rows with one wait
__device__ __forceinline__ void tmem_ld16x2(unsigned ta, unsigned tb, float (&a)[16], float (&b)[16]) {
    unsigned r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
          "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]),
          "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(ta), "r"(tb)
        : "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        a[j] = __uint_as_float(r[j]);
        b[j] = __uint_as_float(r[16 + j]);
    }
}

// zeros into 16 / 8 consecutive accumulator columns of this thread's lane
__device__ __forceinline__ void tmem_zero16(unsigned taddr) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(
                     taddr),
                 "r"(0u)
                 : "memory");
}
__device__ __forceinline__ void tmem_zero8(unsigned taddr) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr), "r"(0u)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld8(unsigned taddr, float (&v)[8]) {
    unsigned r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[j]);
}

// 16 hidden activations, channels 16 h .. 16 h + 15 (bias + ReLU, BF16), into ring row `row` at
// position p: channel groups 2 h and 2 h + 1
__device__ __forceinline__ void store_hidden16(unsigned char* row, int p, int h, const float (&v16)[16],
                                               const float* bias) {
#pragma unroll
    for (int gg = 0; gg < 2; ++gg) {
        const int g = 2 * h + gg;
        const float* vv = v16 + 8 * gg;
        const float* bb = bias + 8 * g;
        uint4 q;
        q.x = pack_bf16x2(fmaxf(vv[0] + bb[0], 0.0f), fmaxf(vv[1] + bb[1], 0.0f));
        q.y = pack_bf16x2(fmaxf(vv[2] + bb[2], 0.0f), fmaxf(vv[3] + bb[3], 0.0f));
        q.z = pack_bf16x2(fmaxf(vv[4] + bb[4], 0.0f), fmaxf(vv[5] + bb[5], 0.0f));
        q.w = pack_bf16x2(fmaxf(vv[6] + bb[6], 0.0f), fmaxf(vv[7] + bb[7], 0.0f));
        *reinterpret_cast<uint4*>(row + g * PLANE + p * 16) = q;
    }
}

// the MMAs of one input row r of a layer: per column shift dx and 16-channel chunk kc, the 128
// positions starting at dx times the three row taps' weights side by side (N = 3 x COUT), into
// the three accumulator slots; the weight blocks start at (1 - r) mod 3 of the stored order
template <int KC, int COUT>
__device__ __forceinline__ void issue_row(unsigned dtmem, unsigned in_row, int r, unsigned wts) {
    constexpr uint32_t ID = idesc_bf16(128, 3 * COUT);
    constexpr unsigned LBO_W = 5 * COUT * 16;
    const int s0 = ((1 - r) % 3 + 3) % 3;
#pragma unroll
    for (int dx = 0; dx < 3; ++dx)
#pragma unroll
        for (int kc = 0; kc < KC; ++kc) {
            const uint64_t a = sdesc(in_row + (unsigned)(dx * 16 + 2 * kc * PLANE), PLANE, 128);
            const uint64_t b = sdesc(wts + (unsigned)(((dx * 2 * KC + 2 * kc) * 5 + s0) * COUT * 16), LBO_W, 128);
            mma(dtmem, a, b, ID, 1u);
        }
}

// Inference of the whole network on an nx x ny periodic lattice.  d: the lattice's populations
// (FP32 deviations, 9 planes); w1 [9][32][16], w2 [9][32][32], w3 [9][16][32] BF16 (tap, cout,
// cin); b1 [32], b2 [32], b3 [16] FP32.  With d_next == nullptr the outputs go to y ([nx * ny][16]
// FP32, 9 used); otherwise the correction is applied here: d_next = d + inv_s_out * P(y) cell by
// cell (P removes a cell's density and momentum), d_next being a buffer other than d (the CTAs
// read each other's halo rows of d).  With zp != nullptr (and d_next == nullptr) the outputs go
// projected, P(y), to 9 planes of nx * ny floats instead of y.
// Grid (ceil(nx / OUT_W), ceil(ny / TC_ROWS)), TC_THREADS threads, SMEM_BYTES dynamic shared memory.
__global__ void __launch_bounds__(TC_THREADS, 2)
    k_closure_fused(const float* __restrict__ d, int nx, int ny, float s_in, int inputs,
                    const __nv_bfloat16* __restrict__ w1, const __nv_bfloat16* __restrict__ w2,
                    const __nv_bfloat16* __restrict__ w3, const float* __restrict__ b1, const float* __restrict__ b2,
                    const float* __restrict__ b3, float* __restrict__ y, float* __restrict__ d_next, float inv_s_out,
                    float* __restrict__ zp, int* __restrict__ status) {
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ int s_ok;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int x0 = blockIdx.x * OUT_W, ys = blockIdx.y * TC_ROWS;
    const size_t N = (size_t)nx * ny;
    unsigned char* ring_in = sm + OFF_IN;
    unsigned char* ring_l1 = sm + OFF_L1;
    unsigned char* ring_l2 = sm + OFF_L2;
    float* bias = reinterpret_cast<float*>(sm + OFF_BIAS);  // b1 [0, 32), b2 [32, 64), b3 [64, 80)
    const unsigned bar = su32(sm + OFF_BAR);
    unsigned* tslot = reinterpret_cast<unsigned*>(sm + OFF_TSLOT);

    // activation rows to zero (positions no layer writes stay finite); weights to the operand
    // layout, row-tap block i holding tap dy = (2 - i) mod 3
    for (int i = tid; i < OFF_W1 / 16; i += TC_THREADS) reinterpret_cast<uint4*>(sm)[i] = make_uint4(0, 0, 0, 0);
    for (int i = tid; i < 3 * 2 * 5 * 32; i += TC_THREADS) {  // (dx, group, block, cout)
        const int n = i % 32, blk = (i / 32) % 5, g = (i / 160) % 2, dx = i / 320;
        const int t = 3 * ((2 - blk + 3) % 3) + dx;
        *reinterpret_cast<uint4*>(sm + OFF_W1 + i * 16) = *reinterpret_cast<const uint4*>(w1 + (t * 32 + n) * 16 + g * 8);
    }
    for (int i = tid; i < 3 * 4 * 5 * 32; i += TC_THREADS) {
        const int n = i % 32, blk = (i / 32) % 5, g = (i / 160) % 4, dx = i / 640;
        const int t = 3 * ((2 - blk + 3) % 3) + dx;
        *reinterpret_cast<uint4*>(sm + OFF_W2 + i * 16) = *reinterpret_cast<const uint4*>(w2 + (t * 32 + n) * 32 + g * 8);
    }
    for (int i = tid; i < 3 * 4 * 5 * 16; i += TC_THREADS) {
        const int n = i % 16, blk = (i / 16) % 5, g = (i / 80) % 4, dx = i / 320;
        const int t = 3 * ((2 - blk + 3) % 3) + dx;
        *reinterpret_cast<uint4*>(sm + OFF_W3 + i * 16) = *reinterpret_cast<const uint4*>(w3 + (t * 16 + n) * 32 + g * 8);
    }
    if (tid < 32) {
        bias[tid] = b1[tid];
        bias[32 + tid] = b2[tid];
        if (tid < 16) bias[64 + tid] = b3[tid];
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tslot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    const unsigned tmem = *tslot;
    // warp w reads TMEM lanes 32 (w % 4) .. + 31 (MMA rows = positions - 1); warpgroup h = w / 4
    // takes half of every accumulator row's columns
    const int lane_q = warp & 3, half = warp >> 2;
    const int mrow = lane_q * 32 + (tid & 31);  // this thread's MMA row
    const unsigned lane_off = (unsigned)(lane_q * 32) << 16;
    // every accumulator slot starts at zero (each warpgroup its half of the columns)
#pragma unroll
    for (int k = 0; k < 6; ++k) tmem_zero16(tmem + lane_off + 32 * k + 16 * half);  // layers 1 and 2
#pragma unroll
    for (int k = 0; k < 3; ++k) tmem_zero8(tmem + lane_off + TM_L3 + 16 * k + 8 * half);
    tmem_wait_st();
    unsigned parity = 0u;
    bool alive = true;

    // the populations of input row a (lattice row ys - 3 + a, wrapped) at this thread's position
    // (< POS), loaded ahead of their use: the second warpgroup has the first 128 positions, as the first
    // one writes the projected outputs (with both on the first, and a wait for each layer's accumulators, a
    // call on 1024^2 took 89.7 us; now 88.2.  What bounds it: a step's MMAs and its epilogues take turns,
    // the tensor pipe is busy for 41 % (sm__pipe_tc_cycles_active) with two blocks on the SM)
    static_assert(POS <= TC_THREADS, "one position a thread");
    const int fp = (tid + TC_THREADS / 2) % TC_THREADS;
    float pre[9];
    auto load_row = [&](int a) {
        const int gy = ((ys - 3 + a) % ny + ny) % ny;
        if (fp < POS) load_dev(d, N, (size_t)gy * nx + ((x0 - 3 + fp) % nx + nx) % nx, pre);
    };
    // features of the prefetched row into input buffer a % 2
    auto store_features = [&](int a) {
        if (fp >= POS) return;
        unsigned char* row = ring_in + (a % 2) * IN_ROW;
        float v[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) v[i] = pre[i];
        if (inputs == LBM_CLOSURE_INPUT_EQ) {
            float n[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) n[i] = v[i];
            non_equilibrium(n);
#pragma unroll
            for (int i = 0; i < 9; ++i) v[i] -= n[i];
        } else {
            non_equilibrium(v);
        }
        *reinterpret_cast<uint4*>(row + fp * 16) =
            make_uint4(pack_bf16x2(s_in * v[0], s_in * v[1]), pack_bf16x2(s_in * v[2], s_in * v[3]),
                       pack_bf16x2(s_in * v[4], s_in * v[5]), pack_bf16x2(s_in * v[6], s_in * v[7]));
        *reinterpret_cast<uint4*>(row + PLANE + fp * 16) = make_uint4(pack_bf16x2(s_in * v[8], 0.0f), 0u, 0u, 0u);
    };
    const auto slot = [](int row) { return ((row % 3) + 3) % 3; };

    // Local rows: input a = lattice row ys - 3 + a (0 .. TC_ROWS + 5); layer-1 rows 1 .. TC_ROWS + 4,
    // layer-2 rows 2 .. TC_ROWS + 3 and layer-3 rows 3 .. TC_ROWS + 2 (= output row ys + e - 3) are
    // the complete ones that the next layer uses; the partial rows at the ends are discarded.
    // Step a: layer-1 MMAs on input row a, layer-2 MMAs on layer-1 row a - 2, layer-3 MMAs on
    // layer-2 row a - 4; then layer-1 row a - 1, layer-2 row a - 3 and layer-3 row a - 5 are
    // complete, read out and their slots zeroed.  A buffer written in step a (layer-1 row a - 1,
    // layer-2 row a - 3, input row a + 1) was last read by the batch of step a - 1.
    load_row(0);
    store_features(0);
    fence_async_smem();
    __syncthreads();
    constexpr int STEPS = TC_ROWS + 8;
    for (int a = 0; a < STEPS; ++a) {
        const bool m1 = a <= TC_ROWS + 5;               // layer-1 MMAs on input row a
        const bool m2 = a >= 3 && a <= TC_ROWS + 6;     // layer-2 MMAs on layer-1 row a - 2
        const bool m3 = a >= 6;                         // layer-3 MMAs on layer-2 row a - 4
        if (tid == 0) {
            fence_after();
            if (m1) issue_row<1, 32>(tmem + TM_L1, su32(ring_in + (a % 2) * IN_ROW), a, su32(sm + OFF_W1));
            if (m2) issue_row<2, 32>(tmem + TM_L2, su32(ring_l1 + ((a - 2) % 2) * H_ROW), a - 2, su32(sm + OFF_W2));
            if (m3) issue_row<2, 16>(tmem + TM_L3, su32(ring_l2 + ((a - 4) % 2) * H_ROW), a - 4, su32(sm + OFF_W3));
            commit(bar);
        }
        const bool next = a + 1 <= TC_ROWS + 5;
        if (next) load_row(a + 1);
        if (tid == 0) s_ok = bar_wait_bounded(bar, parity) ? 1 : 0;
        __syncthreads();
        if (!s_ok) {
            alive = false;
            break;
        }
        bar_try(bar, parity);  // complete: acquire the phase in every thread
        parity ^= 1u;
        fence_after();
        if (m1 || m2) {
            // layer-1 row a - 1 (rows 1 .. TC_ROWS + 4 are used) and layer-2 row a - 3 (2 .. TC_ROWS + 3) are complete
            const unsigned t1 = tmem + lane_off + TM_L1 + 32 * slot(a - 1) + 16 * half;
            const unsigned t2 = tmem + lane_off + TM_L2 + 32 * slot(a - 3) + 16 * half;
            float v1[16], v2[16];
            tmem_ld16x2(t1, t2, v1, v2);
            if (m1) {
                if (a - 1 >= 1) store_hidden16(ring_l1 + ((a - 1) % 2) * H_ROW, mrow + 1, half, v1, bias);
                tmem_zero16(t1);
            }
            if (m2) {
                if (a - 3 >= 2) store_hidden16(ring_l2 + ((a - 3) % 2) * H_ROW, mrow + 1, half, v2, bias + 32);
                tmem_zero16(t2);
            }
        }
        if (m3) {  // layer-3 row a - 5 complete: output row ys + a - 8 (rows 3 .. TC_ROWS + 2)
            const int p = mrow + 1, oy = ys + a - 8, ox = x0 - 3 + p;
            const bool valid = a - 5 >= 3 && p >= 3 && p < 3 + OUT_W && ox < nx && oy < ny;
            const unsigned t0 = tmem + lane_off + TM_L3 + 16 * slot(a - 5);
            if (d_next == nullptr && zp == nullptr) {  // the outputs, split between the warpgroups
                const unsigned t = t0 + 8 * half;
                if (a - 5 >= 3) {
                    float v[8];
                    tmem_ld8(t, v);
                    if (valid) {
                        const float* bb = bias + 64 + 8 * half;
                        float4* o = reinterpret_cast<float4*>(y + ((size_t)oy * nx + ox) * 16 + 8 * half);
                        o[0] = make_float4(v[0] + bb[0], v[1] + bb[1], v[2] + bb[2], v[3] + bb[3]);
                        o[1] = make_float4(v[4] + bb[4], v[5] + bb[5], v[6] + bb[6], v[7] + bb[7]);
                    }
                }
                tmem_zero8(t);
            } else if (half == 0) {  // the projected outputs: added to the populations, or as planes
                if (a - 5 >= 3) {
                    float v[16];
                    tmem_ld16(t0, v);
                    if (valid) {
                        float q[9];
#pragma unroll
                        for (int i = 0; i < 9; ++i) q[i] = v[i] + bias[64 + i];
                        project9(q);
                        const size_t c = (size_t)oy * nx + ox;
                        if (d_next != nullptr) {
#pragma unroll
                            for (int i = 0; i < 9; ++i)
                                d_next[c + (size_t)i * N] = d[c + (size_t)i * N] + inv_s_out * q[i];
                        } else {
#pragma unroll
                            for (int i = 0; i < 9; ++i) zp[c + (size_t)i * N] = q[i];
                        }
                    }
                }
                tmem_zero16(t0);
            }
        }
        tmem_wait_st();
        if (next) store_features(a + 1);
        fence_before();
        fence_async_smem();
        __syncthreads();
    }
    if (!alive) {  // a wait ran out: record it and let the MMAs in flight finish before freeing
        if (tid == 0) {
            atomicExch(status, LBM_ERR_TIMEOUT);
            bar_wait_bounded(bar, parity);
        }
        fence_before();
        __syncthreads();
    }
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// ------------------------------------------------------------------------------------------
// Weight gradients of one layer on the tensor cores (training):
//   dW[tap][ci][co] = sum_cells x[cell + off(tap)][ci] g[cell][co],   db[co] = sum_cells g[cell][co]
// over every cell of nimg images of H x W (W % 64 == 0; inputs outside an image read as zero),
// as GEMMs with the cells as the K dimension.  A tile is 64 columns of one gradient row y and of the three
// input rows y - 1 .. y + 1 that it meets.  Per column tap dx one MMA chain multiplies A = the input
// rows' channels stacked along M (row dy * CIN + ci, then eight rows of ones, whose product is db; what
// follows up to 128 rows is whatever the stage holds there and is ignored), its cells starting at dx, by
// B = the gradient row's channels (N = COUT), into the tensor-memory columns dx * COUT, accumulated over
// all the CTA's tiles.
// A CTA takes a contiguous range of tiles, numbered down the rows of each 64-column strip of each image.
//
// Staging.  With channels contiguous (NHWC) a cell's channels are the M (N) direction of the operands, so
// the MN-major canonical layout -- 8 cells x 8 channels, 16 bytes a cell -- needs no transposition:
// cp.async writes each 16-byte chunk to its place, plane by plane of 8 channels (66 cells of 16 bytes, which
// spreads a warp's chunks over the banks), and a column tap is an offset of 16 bytes in the
// descriptor.  Eight warps copy into a ring of four stages; a ninth one issues the MMAs
// and commits each tile's to the stage's "empty" barrier.  Waits are bounded (1 s).
// Each CTA writes its partial sums in the CUDA-core kernel's layout, so k_dweight_final reduces them the
// same way.
//
// What bounds it: the 16-byte copies, about one a cycle and SM (each input row is read by three tiles, from L2
// after the first).  Transposing every tile with ldmatrix between two block barriers took 95, 84 and 79 us for
// 8 images of 256^2 (32 x 32, 32 x 16 and 16 x 32 channels), 3300 cycles of mostly waiting a tile; this takes
// 40, 33 and 29 us.
// (Two gradient rows a tile, N = 2 COUT, need half the input copies, but their sums are rounded in another
// order, which ten training steps amplify.)
constexpr int DW_TILE = 64;
constexpr int DW_COPIERS = 256;
constexpr int DW_THREADS = DW_COPIERS + 32;

template <int CIN, int COUT>
struct DwLayout {
    static constexpr int XC = CIN / 8, GC = COUT / 8;   // 8-channel groups
    static constexpr int COLS = DW_TILE + 2;
    static constexpr int PLANE_B = COLS * 16;           // [cell][16 B] of one group of one row
    static constexpr int OFF_ONES = 3 * XC * PLANE_B;   // a plane of ones, after the input's [row][group]
    static constexpr int OFF_G = OFF_ONES + PLANE_B;    // gradient planes
    static constexpr int STAGE = (3 * XC + 1 + GC > 16 ? 3 * XC + 1 + GC : 16) * PLANE_B;  // (M = 128 reads sixteen)
    static constexpr int NSTAGE = 4;                    // (six or eight measured 1 to 4 % slower)
    static constexpr int OFF_BAR = NSTAGE * STAGE;      // full[NSTAGE], empty[NSTAGE], done
    static constexpr int OFF_TSLOT = OFF_BAR + 8 * (2 * NSTAGE + 1);
    static constexpr int SMEM = OFF_TSLOT + 8;
    static constexpr int TMEM = 4 * COUT;               // three column taps are used; it comes in powers of two
    static_assert(3 * CIN + 8 <= 128, "three input rows and the ones fit M");
    static_assert(STAGE % 16 == 0 && OFF_BAR % 8 == 0, "alignment");
    static_assert(TMEM == 64 || TMEM == 128, "tensor memory comes in powers of two");
    static_assert(SMEM <= 227 * 1024, "one CTA per SM");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(DW_THREADS, 1)
    k_dweight_tc(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ g, int nimg, int H, int W,
                 float* __restrict__ partials, int* __restrict__ status) {
    using L = DwLayout<CIN, COUT>;
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ int s_fail, s_ok;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned full0 = su32(sm + L::OFF_BAR), empty0 = full0 + 8 * L::NSTAGE, done = empty0 + 8 * L::NSTAGE;
    unsigned* tslot = reinterpret_cast<unsigned*>(sm + L::OFF_TSLOT);
    const int tiles_x = W / DW_TILE, ntiles = nimg * tiles_x * H;
    // this CTA's tiles: a contiguous range of t = (img * tiles_x + strip) * H + y, one at least
    const int G = (int)gridDim.x;
    const int t_begin = (int)(((long long)ntiles * blockIdx.x) / G), t_end = (int)(((long long)ntiles * (blockIdx.x + 1)) / G);
    const int count = t_end - t_begin;

    for (int i = tid; i < L::NSTAGE * L::COLS; i += DW_THREADS)  // BF16 1.0
        *reinterpret_cast<uint4*>(sm + i / L::COLS * L::STAGE + L::OFF_ONES + i % L::COLS * 16) =
            make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);
    if (tid == 0) {
        s_fail = 0;
        for (int k = 0; k < L::NSTAGE; ++k) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(full0 + 8 * k), "r"(DW_COPIERS) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty0 + 8 * k) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(done) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tslot)), "r"(L::TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    const unsigned tmem = *tslot;

    if (warp < DW_COPIERS / 32) {
        // A thread copies the same chunks of every tile: their offsets from the tile's first cell, and to
        // the stage, with the image borders that put a chunk outside in the low bits.
        constexpr int NX = 3 * L::COLS * L::XC, NG = DW_TILE * L::GC, KX = (NX + DW_COPIERS - 1) / DW_COPIERS;
        static_assert(NG <= DW_COPIERS && NX > (KX - 1) * DW_COPIERS, "one gradient chunk a thread");
        enum { LEFT = 1, RIGHT = 2, ABOVE = 4, BELOW = 8 };
        int from[KX];
        unsigned to[KX];
#pragma unroll
        for (int k = 0; k < KX; ++k) {
            const int q = tid + k * DW_COPIERS, cg = q % L::XC, cell = q / L::XC % L::COLS, r = q / (L::XC * L::COLS);
            from[k] = ((r - 1) * W + cell - 1) * CIN + cg * 8;
            to[k] = (unsigned)((r * L::XC + cg) * L::PLANE_B + cell * 16) | (cell == 0 ? LEFT : 0) |
                    (cell == L::COLS - 1 ? RIGHT : 0) | (r == 0 ? ABOVE : 0) | (r == 2 ? BELOW : 0);
        }
        const int gcell = tid / L::GC, gcg = tid % L::GC;
        const unsigned sm0 = su32(sm), gto = (unsigned)(L::OFF_G + gcg * L::PLANE_B + gcell * 16);
        int y = t_begin % H, x0 = t_begin / H % tiles_x * DW_TILE;
        size_t row0 = (size_t)(t_begin / H / tiles_x) * H * W;  // the image's first cell
        for (int i = 0; i < count; ++i) {
            const int b = i % L::NSTAGE;
            if (i >= L::NSTAGE && !__all_sync(0xffffffffu, bar_wait_bounded(empty0 + 8 * b, (i / L::NSTAGE - 1) & 1))) {
                s_fail = 1;
                break;
            }
            const size_t cell0 = row0 + (size_t)y * W + x0;
            const __nv_bfloat16 *xt = x + cell0 * CIN, *gt = g + (cell0 + gcell) * COUT + gcg * 8;
            const unsigned border = (x0 == 0 ? LEFT : 0u) | (x0 + DW_TILE == W ? RIGHT : 0u) | (y == 0 ? ABOVE : 0u) | (y == H - 1 ? BELOW : 0u);
            const unsigned stage = sm0 + b * L::STAGE;
#pragma unroll
            for (int k = 0; k < KX; ++k) {
                if (k == KX - 1 && tid + k * DW_COPIERS >= NX) break;
                const bool in = !(to[k] & border);
                cp_async16_at(stage + (to[k] & ~15u), in ? xt + from[k] : x, in);
            }
            if (NG == DW_COPIERS || tid < NG) cp_async16_at(stage + gto, gt, true);
            if (++y == H) {
                y = 0;
                if ((x0 += DW_TILE) == W) {
                    x0 = 0;
                    row0 += (size_t)H * W;
                }
            }
            // arrives when this thread's copies so far are in shared memory
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full0 + 8 * b) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        constexpr uint32_t ID = idesc_bf16(128, COUT) | 1u << 15 | 1u << 16;  // both operands MN-major
        // MN-major: the leading offset is from 8 cells to the next, the stride from 8 channels to the next
        const uint64_t a0 = sdesc(su32(sm), 128, L::PLANE_B), b0 = sdesc(su32(sm + L::OFF_G), 128, L::PLANE_B);
        // the warp walks the tiles together, so that descriptors are warp-uniform values, and one
        // elected thread issues (issuing from a lane of a divergent warp was the bottleneck)
        int b = 0;
        unsigned phase = 0u;
        for (int i = 0; i < count; ++i) {
            if (!__all_sync(0xffffffffu, bar_wait_bounded(full0 + 8 * b, phase))) {
                s_fail = 1;
                break;
            }
            fence_async_smem();  // the copies went through the generic proxy (a fence by the copiers would drain their queue)
            fence_after();
            const uint64_t as = a0 + (uint64_t)(b * (L::STAGE >> 4)), bs = b0 + (uint64_t)(b * (L::STAGE >> 4));
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < DW_TILE / 16; ++ks)
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx)
                        mma(tmem + (unsigned)(dx * COUT), as + (uint64_t)(16 * ks + dx), bs + (uint64_t)(16 * ks), ID, i > 0 || ks > 0);
                commit(empty0 + 8 * b);
            }
            __syncwarp();
            if (++b == L::NSTAGE) {
                b = 0;
                phase ^= 1u;
            }
        }
        if (elect_one()) commit(done);  // covers every MMA of the CTA
        __syncwarp();
    }
    __syncthreads();
    if (tid == 0) s_ok = bar_wait_bounded(done, 0) && !s_fail;
    __syncthreads();
    if (s_ok) {
        fence_after();
        if (warp < 8) {
            const int quarter = warp & 3, m = quarter * 32 + lane, dy = m / CIN, ci = m % CIN;
            float* p = partials + (size_t)blockIdx.x * (9 * CIN * COUT + COUT);
            for (int q = warp >> 2; q < 3 * COUT / 16; q += 2) {
                float v[16];
                tmem_ld16(tmem + ((unsigned)(quarter * 32) << 16) + (unsigned)(16 * q), v);
                const int dx = 16 * q / COUT, co = 16 * q % COUT;
                float* o = dy < 3 ? p + (size_t)((dy * 3 + dx) * CIN + ci) * COUT + co
                                  : (m == 3 * CIN && dx == 1 ? p + 9 * CIN * COUT + co : nullptr);
                if (o != nullptr)
#pragma unroll
                    for (int k = 0; k < 16; k += 4) *reinterpret_cast<float4*>(o + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
            }
        }
    } else if (tid == 0) {
        atomicExch(status, LBM_ERR_TIMEOUT);  // (the MMAs in flight had their second above)
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM) : "memory");
    }
}

// ------------------------------------------------------------------------------------------
// One 3x3 convolution of the training path on the tcgen05 tensor cores, the same operation as
// k_conv3x3 (non-periodic: cells outside an image read as zero): in [nimg][H][W][CIN] BF16,
// wk [9][COUT][CIN] BF16 (tap = 3 (dy + 1) + (dx + 1)), bias [COUT] FP32; out [nimg][H][W][COUT]
// BF16 with bias and ReLU (EPI_BIAS_RELU), FP32 with bias (EPI_BIAS_F32), or BF16 where the mask
// activation is positive (EPI_MASK, the input gradient of a ReLU layer).
//
// The inference kernel's schedule for one layer: a CTA owns 128 output columns (positions
// x0 .. x0 + 127 = MMA rows) and CONV_TC_ROWS output rows and walks its input rows y0 - 1 ..
// y0 + CONV_TC_ROWS.  Each input row (130 positions, x0 - 1 .. x0 + 128) is read once: per column
// shift dx and 16-channel chunk one MMA multiplies the 128 positions starting at dx by the three
// row taps' weights side by side (N = 3 COUT), the row-tap blocks stored in the order [2, 1, 0, 2,
// 1] so that output row o always lands in accumulator slot o mod 3.  After input row r the output
// row r - 1 is complete: its slot is read, the epilogue written to global memory and the slot
// zeroed.  Input rows are copied two ahead with cp.async, by warps 1 to 7: thread 0 fences them to
// the async proxy when they have landed and issues the MMAs, as a fence would drain a copier's queue.  The mask
// of the output row is loaded while the MMAs run.  Thread 0 waits (1 s limit) for each row's commit, and a
// wait that runs out records LBM_ERR_TIMEOUT, waits (bounded) for the MMAs in flight and frees the
// tensor memory.  (The five calls of a training step on 8 x 256^2 took 148 us with every thread copying and
// fencing one row ahead, now 145; the turns of MMAs and epilogue bound them.)
constexpr int CONV_TC_ROWS = 8;
constexpr int CONV_TC_THREADS = 256;
constexpr int CONV_TC_TMEM = 128;

template <int CIN, int COUT>
struct ConvTcLayout {
    static constexpr int GIN = CIN / 8;                       // 8-channel groups of an input row
    static constexpr int IN_ROW = GIN * PLANE;                // [group][130 positions][16 B]
    static constexpr int NROW = 3;                            // input rows: one read, two on their way
    static constexpr int OFF_W = NROW * IN_ROW;               // [dx 3][group][block 5][cout][16 B]
    static constexpr int W_BYTES = 3 * GIN * 5 * COUT * 16;
    static constexpr int OFF_BIAS = OFF_W + W_BYTES;
    static constexpr int OFF_BAR = OFF_BIAS + COUT * 4;
    static constexpr int OFF_TSLOT = OFF_BAR + 8;
    static constexpr int SMEM = ((OFF_TSLOT + 4 + 127) / 128) * 128;
    static_assert(CIN % 16 == 0 && (COUT == 16 || COUT == 32), "channel counts of the closure layers");
    static_assert(3 * COUT <= CONV_TC_TMEM, "accumulator slots fit the allocation");
    static_assert(OFF_W % 16 == 0 && OFF_BAR % 8 == 0, "alignment");
};

template <int CIN, int COUT, int EPI>
__global__ void __launch_bounds__(CONV_TC_THREADS, 4)
    k_conv_tc(const __nv_bfloat16* __restrict__ in, void* __restrict__ out, const __nv_bfloat16* __restrict__ wk,
              const float* __restrict__ bias, const __nv_bfloat16* __restrict__ mask, int H, int W,
              int* __restrict__ status) {
    using L = ConvTcLayout<CIN, COUT>;
    constexpr int KC = CIN / 16;
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ int s_ok;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int img = blockIdx.z, y0 = blockIdx.y * CONV_TC_ROWS, x0 = blockIdx.x * 128;
    const size_t img_off = (size_t)img * H * W;
    unsigned char* ring = sm;
    float* sbias = reinterpret_cast<float*>(sm + L::OFF_BIAS);
    const unsigned bar = su32(sm + L::OFF_BAR);
    unsigned* tslot = reinterpret_cast<unsigned*>(sm + L::OFF_TSLOT);

    // weights to the operand layout, row-tap block i holding tap dy = (2 - i) mod 3
    for (int i = tid; i < 3 * L::GIN * 5 * COUT; i += CONV_TC_THREADS) {  // (dx, group, block, cout)
        const int n = i % COUT, blk = (i / COUT) % 5, g = (i / (5 * COUT)) % L::GIN, dx = i / (5 * COUT * L::GIN);
        const int t = 3 * ((2 - blk + 3) % 3) + dx;
        *reinterpret_cast<uint4*>(sm + L::OFF_W + i * 16) =
            *reinterpret_cast<const uint4*>(wk + ((size_t)t * COUT + n) * CIN + g * 8);
    }
    if (EPI != EPI_MASK && tid < COUT) sbias[tid] = bias[tid];
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tslot)),
                     "r"(CONV_TC_TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // input row gy (zero outside the image) into ring buffer b: group g, position p = column x0 - 1 + p
    auto stage = [&](int gy, int b) {
        unsigned char* row = ring + b * L::IN_ROW;
        for (int i = tid - 32; i < L::GIN * POS && warp > 0; i += CONV_TC_THREADS - 32) {
            const int p = i % POS, g = i / POS, gx = x0 - 1 + p;
            const bool ok = gy >= 0 && gy < H && gx >= 0 && gx < W;
            const __nv_bfloat16* src = ok ? in + (img_off + (size_t)gy * W + gx) * CIN + g * 8 : in;
            cp_async16(reinterpret_cast<unsigned*>(row + g * PLANE + p * 16), src, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(y0 - 1, 0);
    stage(y0, 1);
    fence_before();
    __syncthreads();
    fence_after();
    const unsigned tmem = *tslot;
    const int lane_q = warp & 3, half = warp >> 2;
    const unsigned lane_off = (unsigned)(lane_q * 32) << 16;
    constexpr int HC = COUT / 2;  // accumulator columns per warpgroup
    // every slot starts at zero (each warpgroup its half of the columns)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if constexpr (HC == 16) tmem_zero16(tmem + lane_off + k * COUT + half * HC);
        else tmem_zero8(tmem + lane_off + k * COUT + half * HC);
    }
    tmem_wait_st();
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    fence_async_smem();  // the weights
    fence_before();
    __syncthreads();
    unsigned parity = 0u;
    bool alive = true;
    const int nrows = min(CONV_TC_ROWS, H - y0);  // output rows of this CTA
    for (int a = 0; a < nrows + 2; ++a) {  // input row y0 - 1 + a
        const int gy = y0 - 1 + a;
        if (tid == 0) {
            fence_async_smem();  // the row's copies went through the generic proxy (the copiers' own fence would drain their queue)
            fence_after();
            issue_row<KC, COUT>(tmem, su32(ring + a % L::NROW * L::IN_ROW), gy, su32(sm + L::OFF_W));
            commit(bar);
        }
        // two rows ahead, into the buffer that row a - 1's MMAs read (an empty group keeps the count)
        if (a + 2 < nrows + 2) stage(gy + 2, (a + 2) % L::NROW);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        // the mask of the output row that this input row completes, while the MMAs run
        const int go = gy - 1, p = lane_q * 32 + lane, gx = x0 + p, c0 = half * HC;
        const size_t cell = img_off + (size_t)go * W + gx;
        const bool stored = go >= y0 && gx < W;
        uint4 mk[HC / 8];
        if (EPI == EPI_MASK && stored)
#pragma unroll
            for (int q = 0; q < HC / 8; ++q) mk[q] = reinterpret_cast<const uint4*>(mask + cell * COUT + c0)[q];
        if (tid == 0) s_ok = bar_wait_bounded(bar, parity) ? 1 : 0;
        __syncthreads();
        if (!s_ok) {
            alive = false;
            break;
        }
        bar_try(bar, parity);  // complete: acquire the phase in every thread
        parity ^= 1u;
        fence_after();
        // output row gy - 1 is complete; rows before y0 only had to be cleared
        const int slot = ((go % 3) + 3) % 3;
        const unsigned t = tmem + lane_off + slot * COUT + half * HC;
        if (go >= y0) {
            float v[HC];
            if constexpr (HC == 16) tmem_ld16(t, v);
            else tmem_ld8(t, v);
            if (stored) {
                if (EPI == EPI_BIAS_F32) {
                    float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + cell * COUT + c0);
#pragma unroll
                    for (int q = 0; q < HC / 4; ++q)
                        o[q] = make_float4(v[4 * q] + sbias[c0 + 4 * q], v[4 * q + 1] + sbias[c0 + 4 * q + 1],
                                           v[4 * q + 2] + sbias[c0 + 4 * q + 2], v[4 * q + 3] + sbias[c0 + 4 * q + 3]);
                } else {
                    unsigned w[HC / 2];
                    if (EPI == EPI_BIAS_RELU) {
#pragma unroll
                        for (int q = 0; q < HC / 2; ++q)
                            w[q] = pack_bf16x2(fmaxf(v[2 * q] + sbias[c0 + 2 * q], 0.0f),
                                               fmaxf(v[2 * q + 1] + sbias[c0 + 2 * q + 1], 0.0f));
                    } else {  // EPI_MASK
#pragma unroll
                        for (int q4 = 0; q4 < HC / 8; ++q4) {
                            const uint4 mm = mk[q4];
                            const unsigned mw[4] = {mm.x, mm.y, mm.z, mm.w};
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                const __nv_bfloat162 m2 = *reinterpret_cast<const __nv_bfloat162*>(&mw[q]);
                                const int k = 8 * q4 + 2 * q;
                                w[4 * q4 + q] = pack_bf16x2(__bfloat162float(m2.x) > 0.0f ? v[k] : 0.0f,
                                                            __bfloat162float(m2.y) > 0.0f ? v[k + 1] : 0.0f);
                            }
                        }
                    }
                    uint4* o = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(out) + cell * COUT + c0);
#pragma unroll
                    for (int q = 0; q < HC / 8; ++q) o[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
                }
            }
        }
        if constexpr (HC == 16) tmem_zero16(t);
        else tmem_zero8(t);
        tmem_wait_st();
        asm volatile("cp.async.wait_group 1;" ::: "memory");  // input row a + 1 landed
        fence_before();
        __syncthreads();
    }
    if (!alive) {  // a wait ran out: record it and let the MMAs in flight finish before freeing
        if (tid == 0) {
            atomicExch(status, LBM_ERR_TIMEOUT);
            bar_wait_bounded(bar, parity);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(CONV_TC_TMEM)
                     : "memory");
    }
}

}  // namespace tc
