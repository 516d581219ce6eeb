// Emulator MLP: forward, backward and AdamW for an ensemble of small multilayer perceptrons that map
// library parameters to per-frequency strain statistics.  No reference counterpart (the reference's
// emulators are Gaussian processes, holodeck/gps/); the training data are libraries the GPU SAM
// itself writes.
//
// Network: E members, each K_0 (inputs, padded to 16) -> N_0 -> ... -> N_{L-1} (outputs), SiLU after
// every layer but the last.  Weights bf16, row-major [N_l][K_l]; biases and master weights fp32.
// Activations between layers are bf16, pre-activations and outputs fp32, and every product is
// accumulated in fp32.
//
// All three contractions (forward Y = X W^T, input gradient dX = dZ W, weight gradient
// dW = dZ^T X) run on the tensor cores the same way: a CTA of 256 threads owns a 128-row output tile
// of NT columns in tensor memory (tcgen05.alloc, fp32 accumulators), stages the operands in shared
// memory in the canonical no-swizzle K-major layout (8 x 16-byte core matrices), one elected thread
// issues tcgen05.mma (kind::f16, bf16 x bf16 -> fp32, M = 128, K = 16 per instruction) and commits
// them to an mbarrier, and the epilogue reads the accumulator back with tcgen05.ld (one TMEM lane per
// output row) and fuses bias, activation or the activation's derivative.
//   * Forward (k_mlp_fwd_tma): both operands are row-major tiles, staged by the tensor memory
//     accelerator (cp.async.bulk.tensor, one box of 8 columns per K-group) against an mbarrier;
//     the whole reduction axis (<= 256) at once, output columns split 64 per CTA, so a layer is one
//     copy / MMA / read-back round trip on (row tiles x column tiles x members) CTAs.
//   * Input and weight gradients (k_mlp_bwd, one launch per layer for both): operands that lie
//     transposed in memory are staged through registers by 8 x 8 blocks; the input gradient stages the
//     whole reduction axis with columns split 64 per CTA, the weight gradient reduces one 128-row batch
//     split per CTA, also 64 columns wide.
// Every wait is bounded: on expiry the kernel flags HGB_STATUS_ITERATION_LIMIT, frees its tensor
// memory and returns.
//
// Dynamic shared memory per CTA is 100 KB, so at most two CTAs share an SM and their allocations
// (at most 256 columns each) always fit the SM's 512 TMEM columns (an allocation never waits).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <cooperative_groups.h>

#include <atomic>
#include <mutex>

#include "hgb_common.cuh"

namespace cg = cooperative_groups;

namespace {

typedef __nv_bfloat16 bf16;

constexpr int TM = 128;            // output rows per CTA (tcgen05 M)
constexpr int NMAX = 256;          // widest layer (tcgen05 N limit for M = 128)
constexpr int LAYER_THREADS = 256;         // eight warps stage a layer's tile and share its epilogue
constexpr int SMEM_DYN = 100 * 1024;       // holds both staged slices; caps residency at two CTAs per SM
constexpr uint64_t WAIT_NS = 1000000000ull;   // a wait for the tensor core gives up after 1 s
constexpr int WIDTH = 256;                 // row stride (elements) of the hidden activation buffers

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// byte offset of element (r, k) of a staged slice (k < KC) in the canonical layout
template <int KC>
__device__ __forceinline__ int slice_off(int r, int k) {
    return (((r >> 3) * (KC / 8) + (k >> 3)) << 7) + ((r & 7) << 4) + ((k & 7) << 1);
}

// shared-memory matrix descriptor: start address, leading byte offset `lbo` (next core matrix along
// K), stride byte offset `sbo` (next 8-row group), descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// instruction descriptor of kind::f16: fp32 accumulator, bf16 A and B, both K-major, M x N
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// non-blocking test of the phase with the given parity
__device__ __forceinline__ bool mbar_test(uint32_t mbar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// wait for the phase with the given parity to complete, for at most WAIT_NS
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    if (mbar_test(mbar, parity)) return true;
    const uint64_t t0 = global_ns();
    while (!mbar_test(mbar, parity))
        if (global_ns() - t0 > WAIT_NS) return false;
    return true;
}

// 16 consecutive fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ float sigmoidf_(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigmoidf_(z); }
__device__ __forceinline__ float silu_grad(float z) {
    const float s = sigmoidf_(z);
    return s * (1.0f + z * (1.0f - s));
}

union Pack8 {
    uint4 u;
    bf16 h[8];
};

// eight consecutive values, in one access where the buffer allows it
__device__ __forceinline__ uint4 load8(const bf16 *p, bool aligned) {
    if (aligned) return *(const uint4 *)p;
    Pack8 v;
#pragma unroll
    for (int i = 0; i < 8; i++) v.h[i] = p[i];
    return v.u;
}

// ---- epilogues of the three contractions and the gradients' operand loaders -------------------------
// A loader: 8 consecutive reduction entries of output row r; B loader: the same for output column n.
// Both return zeros outside the operands.

struct FwdOp {   // epilogue of the forward: Y[b][n] = act(acc + bias[n]) (operands staged by TMA)
    const bf16 *x;
    long x_es;
    int ldx;
    const bf16 *w;
    long w_es;
    const float *bias;
    long b_es;
    int K, N, batch, act;
    float *pre;        // fp32 pre-activations [b][ldp] (hidden layers; may be null)
    long pre_es;
    bf16 *y;           // bf16 activations [b][ldy] (hidden layers)
    long y_es;
    float *out;        // fp32 outputs [b][N] (last layer)
    long out_es;
    int ldp, ldy;

    __device__ void store(int e, int row, int n0, const float (&v)[16]) const {
        if (row >= batch || n0 >= N) return;
        const float *bb = bias + e * b_es + n0;
        if (act) {
            Pack8 p0, p1;
            float z[16];
#pragma unroll
            for (int i = 0; i < 16; i++) z[i] = v[i] + bb[i];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                p0.h[i] = __float2bfloat16_rn(silu(z[i]));
                p1.h[i] = __float2bfloat16_rn(silu(z[i + 8]));
            }
            uint4 *yd = (uint4 *)(y + e * y_es + (long)row * ldy + n0);
            yd[0] = p0.u;
            yd[1] = p1.u;
            if (pre) {
                float4 *pd = (float4 *)(pre + e * pre_es + (long)row * ldp + n0);
#pragma unroll
                for (int i = 0; i < 4; i++) pd[i] = make_float4(z[4 * i], z[4 * i + 1], z[4 * i + 2], z[4 * i + 3]);
            }
        } else {
            float4 *od = (float4 *)(out + e * out_es + (long)row * N + n0);
#pragma unroll
            for (int i = 0; i < 4; i++)
                od[i] = make_float4(v[4 * i] + bb[4 * i], v[4 * i + 1] + bb[4 * i + 1], v[4 * i + 2] + bb[4 * i + 2],
                                    v[4 * i + 3] + bb[4 * i + 3]);
        }
    }
};

struct DxOp {   // dZprev[b][k] = (sum_n dZ[b][n] W[n][k]) * silu'(Zprev[b][k])
    static constexpr int KC = 256, NT = 64;
    const bf16 *dz;    // [b][WIDTH], reduction over its first N columns
    long dz_es;
    const bf16 *w;     // [N][K]
    long w_es;
    bool w_aligned;    // every member's weights start on 16 bytes
    const float *pre;  // Zprev [b][WIDTH]
    long pre_es;
    bf16 *dzp;         // dZprev [b][WIDTH]
    long dzp_es;
    int K, N, batch;

    __device__ uint4 load_a(int e, int row, int n) const {
        if (row >= batch || n >= N) return make_uint4(0, 0, 0, 0);
        return *(const uint4 *)(dz + e * dz_es + (long)row * WIDTH + n);
    }
    // row n + j of W, columns k .. k + 7: block (k, n) of the transposed operand
    __device__ uint4 row_b(int e, int k, int n, int j) const {
        if (k >= K || n + j >= N) return make_uint4(0, 0, 0, 0);
        return load8(w + e * w_es + (long)(n + j) * K + k, w_aligned);
    }
    __device__ void store(int e, int row, int k0, const float (&v)[16]) const {
        if (row >= batch || k0 >= K) return;
        const float4 *zp = (const float4 *)(pre + e * pre_es + (long)row * WIDTH + k0);
        float z[16];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 q = zp[i];
            z[4 * i] = q.x;
            z[4 * i + 1] = q.y;
            z[4 * i + 2] = q.z;
            z[4 * i + 3] = q.w;
        }
        Pack8 p0, p1;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            p0.h[i] = __float2bfloat16_rn(v[i] * silu_grad(z[i]));
            p1.h[i] = __float2bfloat16_rn(v[i + 8] * silu_grad(z[i + 8]));
        }
        uint4 *d = (uint4 *)(dzp + e * dzp_es + (long)row * WIDTH + k0);
        d[0] = p0.u;
        d[1] = p1.u;
    }
};

struct DwOp {   // part[s][n][k] = sum over this split's rows b of dZ[b][n] X[b][k]
    static constexpr int KC = HGB_MLP_SPLIT_ROWS, NT = 64;
    const bf16 *dz;    // [b][WIDTH]
    long dz_es;
    const bf16 *x;     // layer input [b][ldx]
    long x_es;
    int ldx;
    bool x_aligned;    // every row starts on 16 bytes (widths are multiples of 16)
    float *part;       // [E][S][N][K]
    int K, N, batch, nsplit;

    __device__ uint4 row_a(int e, int split, int n, int r, int j) const {   // r: row offset inside the split
        const int b = split * HGB_MLP_SPLIT_ROWS + r + j;
        if (n >= N || b >= batch) return make_uint4(0, 0, 0, 0);
        return *(const uint4 *)(dz + e * dz_es + (long)b * WIDTH + n);
    }
    __device__ uint4 row_b(int e, int split, int k, int r, int j) const {
        const int b = split * HGB_MLP_SPLIT_ROWS + r + j;
        if (k >= K || b >= batch) return make_uint4(0, 0, 0, 0);
        return load8(x + e * x_es + (long)b * ldx + k, x_aligned);
    }
    __device__ void store(int e, int split, int n, int k0, const float (&v)[16]) const {
        if (n >= N || k0 >= K) return;
        float4 *d = (float4 *)(part + (((long)e * nsplit + split) * N + n) * K + k0);
#pragma unroll
        for (int i = 0; i < 4; i++) d[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
};

template <int N>
__host__ __device__ constexpr int tmem_cols() { return N <= 32 ? 32 : N <= 64 ? 64 : N <= 128 ? 128 : 256; }

// Transposes an 8 x 8 block of bf16, rows in r[0..7], in registers: the pairs and quads move by naming,
// the halves by byte permutes.
__device__ __forceinline__ void transpose8(const uint4 (&r)[8], uint4 (&t)[8]) {
    uint32_t o[8][4];
#pragma unroll
    for (int c = 0; c < 4; c++) {   // columns 2 c and 2 c + 1
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t lo = (&r[2 * j].x)[c], hi = (&r[2 * j + 1].x)[c];
            o[2 * c][j] = __byte_perm(lo, hi, 0x5410);
            o[2 * c + 1][j] = __byte_perm(lo, hi, 0x7632);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) t[i] = make_uint4(o[i][0], o[i][1], o[i][2], o[i][3]);
}

// the core matrices of rows x .. x + 7, reduction entries r .. r + 7, from eight rows of the row-major
// buffer that has x fastest: row(j) holds reduction entry r + j
template <int KC, class Row>
__device__ __forceinline__ void stage_transposed(uint8_t *s, int x, int r, const Row &row) {
    uint4 in[8], t[8];
#pragma unroll
    for (int j = 0; j < 8; j++) in[j] = row(j);
    transpose8(in, t);
#pragma unroll
    for (int i = 0; i < 8; i++) *(uint4 *)(s + slice_off<KC>(x + i, r)) = t[i];
}

// One layer of the backward pass in one launch: the blocks of the input gradient (128 batch rows x 64
// columns each, first: the next layer waits for them) and those of the weight gradient (128 outputs x
// 64 inputs of one 128-row batch split).  Both read dZ of the layer and depend on nothing else of each
// other's.  Operands that lie transposed in memory are staged by 8 x 8 blocks, eight 16-byte loads a
// thread and a register transpose (gathering them two bytes at a time took most of the time): at batch
// 512 and 4 members of 256 x 256, 24 + 23 us a layer for the two gradients in launches of their own and
// with four warps a block,
// 13 us for both.
struct BwdLayer {
    DxOp dx;
    DwOp dw;
    int dx_rows, dx_cols;              // tiles of the input gradient (0 for the first layer)
    int dw_rows, dw_cols, nsplit;      // tiles and batch splits of the weight gradient
};

__global__ void __launch_bounds__(LAYER_THREADS) k_mlp_bwd(const __grid_constant__ BwdLayer L, int *status) {
    constexpr int NT = 64, COLS = tmem_cols<NT>();
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = blockIdx.y, n_dx = L.dx_rows * L.dx_cols;
    const bool is_dx = (int)blockIdx.x < n_dx;
    const uint32_t mb = smem_u32(&mbar);

    if (warp == 0) tmem_alloc(smem_u32(&tmem_slot), COLS);
    if (threadIdx.x == 0) mbar_init(mb, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    int row0, col0, split = 0, npad, red;
    uint8_t *sa = smem, *sb;
    if (is_dx) {
        row0 = ((int)blockIdx.x / L.dx_cols) * TM;
        col0 = ((int)blockIdx.x % L.dx_cols) * NT;
        npad = min(NT, L.dx.K - col0);      // widths are multiples of 16
        red = L.dx.N;
        sb = smem + TM * DxOp::KC * 2;
        const int kg = red / 8;
#pragma unroll 8
        for (int v = threadIdx.x; v < TM * kg; v += LAYER_THREADS) {
            const int r = v % TM, g = v / TM;
            *(uint4 *)(sa + slice_off<DxOp::KC>(r, g * 8)) = L.dx.load_a(e, row0 + r, g * 8);
        }
        for (int v = threadIdx.x; v < (npad / 8) * kg; v += LAYER_THREADS) {
            const int x = (v % (npad / 8)) * 8, n = (v / (npad / 8)) * 8;
            stage_transposed<DxOp::KC>(sb, x, n, [&](int j) { return L.dx.row_b(e, col0 + x, n, j); });
        }
    } else {
        int i = (int)blockIdx.x - n_dx;
        split = i % L.nsplit;
        i /= L.nsplit;
        row0 = (i / L.dw_cols) * TM;
        col0 = (i % L.dw_cols) * NT;
        npad = min(NT, L.dw.K - col0);
        red = HGB_MLP_SPLIT_ROWS;           // rows beyond the batch are zeros
        sb = smem + TM * DwOp::KC * 2;
        constexpr int KG = HGB_MLP_SPLIT_ROWS / 8;
        for (int v = threadIdx.x; v < (TM / 8) * KG; v += LAYER_THREADS) {
            const int x = (v % (TM / 8)) * 8, r = (v / (TM / 8)) * 8;
            stage_transposed<DwOp::KC>(sa, x, r, [&](int j) { return L.dw.row_a(e, split, row0 + x, r, j); });
        }
        for (int v = threadIdx.x; v < (npad / 8) * KG; v += LAYER_THREADS) {
            const int x = (v % (npad / 8)) * 8, r = (v / (npad / 8)) * 8;
            stage_transposed<DwOp::KC>(sb, x, r, [&](int j) { return L.dw.row_b(e, split, col0 + x, r, j); });
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
        tc_fence_after();
        const uint32_t idesc = idesc_bf16(TM, npad);
        const uint32_t sbo = 16 * (is_dx ? DxOp::KC : DwOp::KC);
        for (int s = 0; s < red / 16; s++)
            mma_bf16(tmem, smem_desc(smem_u32(sa) + 256 * s, 128, sbo), smem_desc(smem_u32(sb) + 256 * s, 128, sbo),
                     idesc, s > 0 ? 1u : 0u);
        mma_commit(mb);
    }
    const bool ok = __syncthreads_and(mbar_wait(mb, 0));
    tc_fence_after();
    if (ok) {
        const int m = (warp & 3) * 32 + lane;   // a warp reads the TMEM lanes of its place among four
        const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        for (int n0 = (warp >> 2) * 16; n0 < npad; n0 += 32) {
            float v[16];
            tmem_ld16(lane_addr + (uint32_t)n0, v);
            if (is_dx) L.dx.store(e, row0 + m, col0 + n0, v);
            else L.dw.store(e, split, row0 + m, col0 + n0, v);
        }
    } else {
        if (threadIdx.x == 0) hgb::flag(status, HGB_STATUS_ITERATION_LIMIT);
        mbar_wait(mb, 0);   // give the tensor core a last bounded chance to finish
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, COLS);
}

// ---- forward with TMA operand staging ----------------------------------------------------------------
// The forward's operands are plain row-major tiles (activations [b][k], weights [n][k]), so the tensor
// memory accelerator stages them: a box of 8 columns x R rows lands in shared memory as R rows of
// 16 bytes, which is one K-group of core matrices for all R rows (8-row groups 128 B apart).  Stacking
// the K-groups gives the canonical K-major layout with leading byte offset 16 R and stride byte
// offset 128.  One thread issues every copy against one mbarrier (expect_tx of the boxes' bytes;
// out-of-range rows and columns arrive as zeros), then the MMAs against the same barrier's next phase.

constexpr int FWD_NT = 64;   // output columns per CTA
constexpr int FWD_KMAX = 256;

__device__ __forceinline__ void mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(dst),
        "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(mbar)
        : "memory");
}

// blockIdx.x: 128-row tile, blockIdx.y: 64-column tile, blockIdx.z: member.  xmap: [members or 1][rows][K]
// activations (x_member != 0 when each member has its own), wmap: [members][N][K] weights.
__global__ void __launch_bounds__(LAYER_THREADS) k_mlp_fwd_tma(const __grid_constant__ CUtensorMap xmap,
                                                         const __grid_constant__ CUtensorMap wmap, FwdOp op,
                                                         int x_member, int *status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    constexpr int COLS = tmem_cols<FWD_NT>();
    uint8_t *sa = smem;                          // K/8 groups of 128 rows x 16 B
    uint8_t *sb = smem + TM * FWD_KMAX * 2;      // K/8 groups of 64 rows x 16 B
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = blockIdx.z, row0 = blockIdx.x * TM, col0 = blockIdx.y * FWD_NT;
    const int ncols = min(FWD_NT, op.N - col0);
    const int groups = op.K / 8;
    const uint32_t mb = smem_u32(&mbar);

    if (warp == 0) tmem_alloc(smem_u32(&tmem_slot), COLS);
    if (threadIdx.x == 0) mbar_init(mb, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    if (warp == 0) {   // a lane per K-group: one thread's 64 boxes, one after another, set the pace before
        if (lane == 0) mbar_expect_tx(mb, (uint32_t)groups * (TM + FWD_NT) * 16);
        __syncwarp();
        for (int g = lane; g < groups; g += 32) {
            tma_load_3d(smem_u32(sa + g * TM * 16), &xmap, g * 8, row0, x_member ? e : 0, mb);
            tma_load_3d(smem_u32(sb + g * FWD_NT * 16), &wmap, g * 8, col0, e, mb);
        }
    }
    bool ok = __syncthreads_and(mbar_wait(mb, 0));
    uint32_t pending = 0;   // parity of a phase still to complete when a wait gives up
    if (ok) {
        if (threadIdx.x == 0) {
            tc_fence_after();
            const uint32_t idesc = idesc_bf16(TM, ncols);
            for (int s = 0; s < op.K / 16; s++)
                mma_bf16(tmem, smem_desc(smem_u32(sa) + 2 * TM * 16 * s, TM * 16, 128),
                         smem_desc(smem_u32(sb) + 2 * FWD_NT * 16 * s, FWD_NT * 16, 128), idesc, s > 0 ? 1u : 0u);
            mma_commit(mb);
        }
        ok = __syncthreads_and(mbar_wait(mb, 1));
        pending = 1;
    }
    tc_fence_after();
    if (ok) {
        const int m = (warp & 3) * 32 + lane;   // a warp reads the TMEM lanes of its place among four
        const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        for (int n0 = (warp >> 2) * 16; n0 < ncols; n0 += 32) {
            float v[16];
            tmem_ld16(lane_addr + (uint32_t)n0, v);
            op.store(e, row0 + m, col0 + n0, v);
        }
    } else {
        if (threadIdx.x == 0) hgb::flag(status, HGB_STATUS_ITERATION_LIMIT);
        mbar_wait(mb, pending);   // a last bounded wait for the copies or MMAs in flight
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, COLS);
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    });
    return fn;
}

// bf16 tensor [d2][d1][d0] (d0 contiguous), strides in bytes, boxes of b0 x b1 x 1, zero fill outside
int encode_bf16_3d(CUtensorMap *map, const void *base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1,
                   uint64_t s2, uint32_t b0, uint32_t b1) {
    PFN_cuTensorMapEncodeTiled_v12000 fn = tensor_map_encoder();
    if (!fn) {
        hgb::set_cuda_error(cudaErrorNotSupported);
        return HGB_ERR_CUDA;
    }
    cuuint64_t dims[3] = {d0, d1, d2};
    cuuint64_t strides[2] = {s1, s2};
    cuuint32_t box[3] = {b0, b1, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        hgb::set_cuda_error(cudaErrorInvalidValue);
        return HGB_ERR_INVALID_ARGUMENT;
    }
    return HGB_OK;
}

int launch_fwd_tma(const FwdOp &op, long x_member_stride_elems, int members, int *status, cudaStream_t st) {
    static std::atomic<bool> attr_set{false};
    if (!attr_set.load(std::memory_order_acquire)) {
        cudaError_t err = cudaFuncSetAttribute(k_mlp_fwd_tma, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_DYN);
        if (err != cudaSuccess) {
            hgb::set_cuda_error(err);
            return HGB_ERR_CUDA;
        }
        attr_set.store(true, std::memory_order_release);
    }
    CUtensorMap xmap, wmap;
    const uint64_t xrow = (uint64_t)op.ldx * 2;
    const int x_member = x_member_stride_elems != 0;
    int rc = encode_bf16_3d(&xmap, op.x, (uint64_t)op.K, (uint64_t)op.batch, x_member ? (uint64_t)members : 1, xrow,
                            x_member ? (uint64_t)x_member_stride_elems * 2 : xrow * (uint64_t)op.batch, 8, TM);
    if (rc) return rc;
    rc = encode_bf16_3d(&wmap, op.w, (uint64_t)op.K, (uint64_t)op.N, (uint64_t)members, (uint64_t)op.K * 2,
                        (uint64_t)op.w_es * 2, 8, FWD_NT);
    if (rc) return rc;
    dim3 grid((unsigned)hgb::ceil_div(op.batch, TM), (unsigned)hgb::ceil_div(op.N, FWD_NT), (unsigned)members);
    k_mlp_fwd_tma<<<grid, LAYER_THREADS, SMEM_DYN, st>>>(xmap, wmap, op, x_member, status);
    return hgb::check_launch();
}

// ---- loss, gradient reduction, optimiser ----------------------------------------------------------

struct NetView {
    int L, E;
    int K[HGB_MLP_MAX_LAYERS], N[HGB_MLP_MAX_LAYERS];
    long w_off[HGB_MLP_MAX_LAYERS], p_off[HGB_MLP_MAX_LAYERS], b_off[HGB_MLP_MAX_LAYERS];
    long n_w, n_p;   // bf16 weights and fp32 parameters per member
};

NetView view_of(const hgb_mlp *net) {
    NetView v{};
    v.L = net->n_layers;
    v.E = net->n_members;
    long ow = 0, op = 0;
    for (int l = 0; l < v.L; l++) {
        v.K[l] = net->dims[l];
        v.N[l] = net->dims[l + 1];
        v.w_off[l] = ow;
        v.p_off[l] = op;
        v.b_off[l] = op + (long)v.N[l] * v.K[l];
        ow += (long)v.N[l] * v.K[l];
        op += (long)v.N[l] * v.K[l] + v.N[l];
    }
    v.n_w = ow;
    v.n_p = op;
    return v;
}

// dZ of the last layer = d loss / d out (bf16) of loss[e] = mean (out - target)^2, and this block's part
// of the loss's sum (added up in block order by k_grad_reduce).  One block per member took 162 us of a
// 512-row step; over MSE_BLOCKS blocks a member it is 7 us.
constexpr int MSE_BLOCKS = 32;

__global__ void __launch_bounds__(256) k_mse(int batch, int nout, const float *__restrict__ out, const float *__restrict__ target,
                      long t_es, bf16 *__restrict__ dz, long dz_es, float *__restrict__ part) {
    const int e = blockIdx.y;
    const float scale = 2.0f / ((float)batch * (float)nout);
    const long total = (long)batch * nout;
    float acc = 0.0f;
    for (long i = (long)blockIdx.x * 256 + threadIdx.x; i < total; i += 256L * MSE_BLOCKS) {
        const long b = i / nout, n = i % nout;
        const float d = out[e * total + i] - target[e * t_es + i];
        acc += d * d;
        dz[e * dz_es + b * WIDTH + n] = __float2bfloat16_rn(scale * d);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    __shared__ float red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float v = red[0];
        for (int w = 1; w < 8; w++) v += red[w];
        part[e * MSE_BLOCKS + blockIdx.x] = v;
    }
}

struct GradArgs {
    NetView v;
    int batch, nsplit;
    const float *part[HGB_MLP_MAX_LAYERS];   // [E][S][N][K]
    const bf16 *dz[HGB_MLP_MAX_LAYERS];      // [E][B][WIDTH]
    long dz_es;
    float *grad;                             // [E][n_p]
    const float *loss_part;                  // [E][MSE_BLOCKS]
    float *loss;                             // [E] or null
    int w_blocks, bias_tiles;                // blocks of the weights; 32-output tiles of one member's biases
};

// weight gradients: the split partials summed in split order, one thread each (blocks of the first
// `w_blocks`, the rest of the grid being: one block per member, layer and 32 outputs, whose eight warps
// sum dZ over an eighth of the batch each for the bias gradients; then one block for the losses).  A
// single thread per bias walked the whole batch: 23 us, 12 us now.
__global__ void __launch_bounds__(256) k_grad_reduce(GradArgs a) {
    const int t = threadIdx.x;
    if ((int)blockIdx.x < a.w_blocks) {
        const long idx = (long)blockIdx.x * 256 + t;
        if (idx >= (long)a.v.E * a.v.n_p) return;
        const int e = (int)(idx / a.v.n_p);
        const long p = idx % a.v.n_p;
        int l = 0;
        while (l + 1 < a.v.L && p >= a.v.p_off[l + 1]) l++;
        if (p >= a.v.b_off[l]) return;
        const long nk = (long)a.v.K[l] * a.v.N[l];
        const float *pp = a.part[l] + (long)e * a.nsplit * nk + (p - a.v.p_off[l]);
        float g = 0.0f;
        for (int s = 0; s < a.nsplit; s++) g += pp[(long)s * nk];
        a.grad[idx] = g;
        return;
    }
    __shared__ float red[8][32];
    int i = (int)blockIdx.x - a.w_blocks;
    if (i == a.v.E * a.bias_tiles) {
        for (int e = t; a.loss && e < a.v.E; e += 256) {
            float v = 0.0f;
            for (int k = 0; k < MSE_BLOCKS; k++) v += a.loss_part[e * MSE_BLOCKS + k];
            a.loss[e] = v / ((float)a.batch * (float)a.v.N[a.v.L - 1]);
        }
        return;
    }
    const int e = i / a.bias_tiles;
    i %= a.bias_tiles;
    int l = 0;
    while (i >= (a.v.N[l] + 31) / 32) i -= (a.v.N[l++] + 31) / 32;
    const int n = 32 * i + (t & 31), warp = t >> 5;
    float g = 0.0f;
    if (n < a.v.N[l]) {
        const bf16 *d = a.dz[l] + e * a.dz_es + n;
        for (int b = warp; b < a.batch; b += 8) g += __bfloat162float(d[(long)b * WIDTH]);
    }
    red[warp][t & 31] = g;
    __syncthreads();
    if (warp == 0 && n < a.v.N[l]) {
        for (int w = 1; w < 8; w++) g += red[w][t];
        a.grad[(long)e * a.v.n_p + a.v.b_off[l] + n] = g;
    }
}

// decoupled AdamW on the fp32 master parameters; weights (not biases) decay; bf16 weight copies written
__global__ void k_adamw(NetView v, float *__restrict__ params, const float *__restrict__ grad, float *__restrict__ m1,
                        float *__restrict__ m2, bf16 *__restrict__ w, float lr, float b1, float b2, float eps, float wd,
                        float bc1, float bc2) {
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long)v.E * v.n_p) return;
    const int e = (int)(idx / v.n_p);
    const long p = idx % v.n_p;
    int l = 0;
    while (l + 1 < v.L && p >= v.p_off[l + 1]) l++;
    const bool is_w = p < v.b_off[l];
    const float g = grad[idx];
    const float a = b1 * m1[idx] + (1.0f - b1) * g;
    const float b = b2 * m2[idx] + (1.0f - b2) * g * g;
    m1[idx] = a;
    m2[idx] = b;
    float x = params[idx];
    if (is_w) x -= lr * wd * x;
    x -= lr * (a / bc1) / (sqrtf(b / bc2) + eps);
    params[idx] = x;
    if (is_w) w[(long)e * v.n_w + v.w_off[l] + (p - v.p_off[l])] = __float2bfloat16_rn(x);
}

__global__ void k_pack_weights(NetView v, const float *__restrict__ params, bf16 *__restrict__ w) {
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long)v.E * v.n_p) return;
    const int e = (int)(idx / v.n_p);
    const long p = idx % v.n_p;
    int l = 0;
    while (l + 1 < v.L && p >= v.p_off[l + 1]) l++;
    if (p < v.b_off[l]) w[(long)e * v.n_w + v.w_off[l] + (p - v.p_off[l])] = __float2bfloat16_rn(params[idx]);
}

int check_net(const hgb_mlp *net) {
    if (!net || net->n_layers < 1 || net->n_layers > HGB_MLP_MAX_LAYERS || net->n_members < 1) return 0;
    if (net->n_members > 65535) return 0;
    for (int l = 0; l <= net->n_layers; l++) {
        const int d = net->dims[l];
        if (d < 16 || d > NMAX || (d & 15)) return 0;
    }
    return 1;
}

int launch_bwd(const BwdLayer &L, int members, int *status, cudaStream_t st) {
    static std::atomic<bool> attr_set{false};   // idempotent; set before the first launch
    if (!attr_set.load(std::memory_order_acquire)) {
        cudaError_t err = cudaFuncSetAttribute(k_mlp_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_DYN);
        if (err != cudaSuccess) {
            hgb::set_cuda_error(err);
            return HGB_ERR_CUDA;
        }
        attr_set.store(true, std::memory_order_release);
    }
    const unsigned blocks = (unsigned)((long)L.dx_rows * L.dx_cols + (long)L.dw_rows * L.dw_cols * L.nsplit);
    k_mlp_bwd<<<dim3(blocks, (unsigned)members), LAYER_THREADS, SMEM_DYN, st>>>(L, status);
    return hgb::check_launch();
}

const float *param_bias(const hgb_mlp *net, const NetView &v, int l) { return net->params + v.b_off[l]; }

// ---- fused forward for small query batches --------------------------------------------------------
// One cluster of FUSED_CL CTAs per member; CTA r of the cluster owns output columns
// [r N_l / FUSED_CL, (r + 1) N_l / FUSED_CL) of every layer l.  At the start it bulk-copies its
// column slice of every layer's weights (cp.async.bulk, one mbarrier per layer, so the later layers'
// copies overlap the first layers' arithmetic) into shared memory.  A layer is a matrix-vector
// product per query on the CUDA cores (a batch of at most FUSED_QMAX rows would leave a 128-row
// tensor-core tile almost empty): each warp takes every fourth column, its lanes split the
// reduction axis in runs of 8, fp32 products, and the warp's columns are summed together by one
// transposing shuffle reduction.  The hidden activations
// (bias, SiLU, rounded to bf16 as in the layered forward) are stored into the next activation
// buffer of every CTA of the cluster (distributed shared memory), and one cluster barrier per layer
// publishes them; the buffers alternate, so a CTA writing layer l + 1's inputs never meets a peer
// still reading layer l's.  The last layer writes fp32 outputs.  The copies' waits are bounded: on
// expiry the CTA flags HGB_STATUS_ITERATION_LIMIT and keeps taking part in every cluster barrier
// (its outputs are not valid), and waits once more, bounded, for its copies before it returns.
// The biases of all of the CTA's columns are loaded into shared memory at the start (one round trip
// instead of one per column).  Inputs, outputs and the status word are read and written with plain
// accesses, so they may be pinned host memory (device-accessible under unified addressing): a
// graphed query then needs no copy nodes.  The status bit is set with a plain read-modify-write.
constexpr int FUSED_CL = 8;
constexpr int FUSED_QMAX = HGB_MLP_FUSED_MAX_BATCH;
constexpr int FUSED_THREADS = 128;
constexpr int FUSED_ACT_BYTES = FUSED_QMAX * WIDTH * 2;   // one bf16 activation buffer
constexpr int FUSED_NCMAX = NMAX / FUSED_CL;              // columns per CTA and layer, at most

struct FusedArgs {
    int L, batch;
    int K[HGB_MLP_MAX_LAYERS], N[HGB_MLP_MAX_LAYERS];
    int w_smem[HGB_MLP_MAX_LAYERS];     // byte offset of layer l's weight slice in shared memory
    long w_off[HGB_MLP_MAX_LAYERS], b_off[HGB_MLP_MAX_LAYERS];
    long n_w, n_p;
    const bf16 *weights;
    const float *params;
    const bf16 *x;
    long x_es;
    float *out;
    int *status;
};

// global -> this CTA's shared memory, completion counted on mbar (16-byte aligned, size % 16 == 0)
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(mbar)
                 : "memory");
}

__device__ __forceinline__ float dot8_bf16(uint4 a, uint4 b, float acc) {
    const __nv_bfloat162 *pa = reinterpret_cast<const __nv_bfloat162 *>(&a);
    const __nv_bfloat162 *pb = reinterpret_cast<const __nv_bfloat162 *>(&b);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 fa = __bfloat1622float2(pa[i]), fb = __bfloat1622float2(pb[i]);
        acc = fmaf(fa.x, fb.x, acc);
        acc = fmaf(fa.y, fb.y, acc);
    }
    return acc;
}

__global__ void __cluster_dims__(FUSED_CL, 1, 1) __launch_bounds__(FUSED_THREADS)
    k_mlp_fwd_fused(const __grid_constant__ FusedArgs a) {
    extern __shared__ __align__(128) unsigned char fsm[];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int e = blockIdx.y;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    bf16 *act0 = (bf16 *)fsm;
    bf16 *act1 = (bf16 *)(fsm + FUSED_ACT_BYTES);
    uint64_t *mbar = (uint64_t *)(fsm + 2 * FUSED_ACT_BYTES);
    float *sbias = (float *)(fsm + 2 * FUSED_ACT_BYTES + 128);   // [layer][FUSED_NCMAX]
    if (t == 0) {
        for (int l = 0; l < a.L; l++) mbar_init(smem_u32(&mbar[l]), 1);
    }
    for (int i = t; i < a.L * FUSED_NCMAX; i += FUSED_THREADS) {
        const int l = i / FUSED_NCMAX, n = i % FUSED_NCMAX, nc = a.N[l] / FUSED_CL;
        if (n < nc) sbias[i] = __ldg(a.params + e * a.n_p + a.b_off[l] + rank * nc + n);
    }
    __syncthreads();
    if (t == 0) {
        for (int l = 0; l < a.L; l++) {
            const int nc = a.N[l] / FUSED_CL;
            const uint32_t bytes = (uint32_t)nc * (uint32_t)a.K[l] * 2u;
            mbar_expect_tx(smem_u32(&mbar[l]), bytes);
            bulk_g2s(smem_u32(fsm + a.w_smem[l]), a.weights + e * a.n_w + a.w_off[l] + (long)rank * nc * a.K[l], bytes,
                     smem_u32(&mbar[l]));
        }
    }
    const int Q = a.batch;
    for (int i = t; i < Q * a.K[0]; i += FUSED_THREADS) {
        const int q = i / a.K[0], k = i % a.K[0];
        act0[q * WIDTH + k] = a.x[e * a.x_es + (long)q * a.K[0] + k];
    }
    cluster.sync();   // every CTA of the cluster runs before any stores into its shared memory
    bool ok = true;
    for (int l = 0; l < a.L; l++) {
        const int K = a.K[l], N = a.N[l], nc = N / FUSED_CL, c0 = rank * nc;
        if (ok && !mbar_wait(smem_u32(&mbar[l]), 0)) ok = false;
        const bf16 *W = (const bf16 *)(fsm + a.w_smem[l]);   // [nc][K]
        const bf16 *X = (l & 1) ? act1 : act0;
        bf16 *Y = (l & 1) ? act0 : act1;
        const float *bias = sbias + l * FUSED_NCMAX;
        const bool last = l == a.L - 1;
        // warp w: columns n = w + 4 j, j < ncw (at most 8); lane k: reduction entries 8k .. 8k + 7
        // (K <= 256, so one run per lane).  The eight column sums are reduced together: three
        // exchange levels halve the set a lane carries (4 + 2 + 1 shuffles), two more finish the
        // sum, and lane 4 j ends with column j's total, so the eight epilogues run side by side.
        const int ncw = (nc - warp + 3) / 4;
        const bool has_run = lane < K / 8;
        const int jl = 4 * ((lane >> 4) & 1) + 2 * ((lane >> 3) & 1) + ((lane >> 2) & 1);
        for (int q = 0; q < Q; q++) {
            float v[8];
            const uint4 xv = has_run ? *(const uint4 *)(X + q * WIDTH + lane * 8) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int j = 0; j < 8; j++)
                v[j] = (has_run && j < ncw) ? dot8_bf16(*(const uint4 *)(W + (long)(warp + 4 * j) * K + lane * 8), xv, 0.0f)
                                            : 0.0f;
            const bool h1 = (lane >> 4) & 1, h2 = (lane >> 3) & 1, h3 = (lane >> 2) & 1;
            float w4[4], w2[2];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float keep = h1 ? v[i + 4] : v[i], give = h1 ? v[i] : v[i + 4];
                w4[i] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float keep = h2 ? w4[i + 2] : w4[i], give = h2 ? w4[i] : w4[i + 2];
                w2[i] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
            }
            float acc = (h3 ? w2[1] : w2[0]) + __shfl_xor_sync(0xffffffffu, h3 ? w2[0] : w2[1], 4);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            if ((lane & 3) == 0 && jl < ncw) {
                const int n = warp + 4 * jl;
                const float z = acc + bias[n];
                if (last) {
                    a.out[((long)e * Q + q) * N + c0 + n] = z;
                } else {
                    const bf16 y = __float2bfloat16_rn(silu(z));
#pragma unroll
                    for (int r = 0; r < FUSED_CL; r++) cluster.map_shared_rank(Y, r)[q * WIDTH + c0 + n] = y;
                }
            }
        }
        cluster.sync();   // layer l + 1's inputs are in every CTA; layer l's are no longer read
    }
    if (!ok) {
        if (t == 0) {
            if (a.status) *(volatile int *)a.status |= HGB_STATUS_ITERATION_LIMIT;
            for (int l = 0; l < a.L; l++) mbar_wait(smem_u32(&mbar[l]), 0);   // bounded: copies in flight
        }
        __syncthreads();
    }
}

size_t fused_smem_bytes(const NetView &v, FusedArgs *fa) {
    // two activation buffers, the mbarriers, the biases, then the weight slices
    size_t off = 2 * (size_t)FUSED_ACT_BYTES + 128 + (((size_t)v.L * FUSED_NCMAX * 4 + 127) & ~(size_t)127);
    for (int l = 0; l < v.L; l++) {
        if (fa) fa->w_smem[l] = (int)off;
        off += ((size_t)(v.N[l] / FUSED_CL) * v.K[l] * 2 + 127) & ~(size_t)127;
    }
    return off;
}

}  // namespace

extern "C" {

long hgb_mlp_param_count(const hgb_mlp *net) { return check_net(net) ? view_of(net).n_p : -1; }

long hgb_mlp_weight_count(const hgb_mlp *net) { return check_net(net) ? view_of(net).n_w : -1; }

int hgb_mlp_forward(const hgb_mlp *net, const uint16_t *x, long x_member_stride, int batch, uint16_t *act,
                    float *pre, float *out, int *d_status, void *stream) {
    HGB_CHECK_ARG(check_net(net) && net->params && net->weights && x && act && out && batch >= 0);
    HGB_CHECK_ARG(x_member_stride >= 0);
    if (batch == 0) return HGB_OK;
    const NetView v = view_of(net);
    cudaStream_t st = (cudaStream_t)stream;
    const long hid_es = (long)batch * WIDTH;            // member stride of one layer's hidden buffer
    const long hid_ls = (long)v.E * hid_es;             // layer stride
    for (int l = 0; l < v.L; l++) {
        FwdOp op{};
        const bool first = l == 0, last = l == v.L - 1;
        op.x = first ? (const bf16 *)x : (const bf16 *)act + (l - 1) * hid_ls;
        op.x_es = first ? x_member_stride : hid_es;
        op.ldx = first ? v.K[0] : WIDTH;
        op.w = (const bf16 *)net->weights + v.w_off[l];
        op.w_es = v.n_w;
        op.bias = param_bias(net, v, l);
        op.b_es = v.n_p;
        op.K = v.K[l];
        op.N = v.N[l];
        op.batch = batch;
        op.act = last ? 0 : 1;
        op.pre = (last || !pre) ? nullptr : pre + l * hid_ls;
        op.pre_es = hid_es;
        op.ldp = WIDTH;
        op.y = last ? nullptr : (bf16 *)act + l * hid_ls;
        op.y_es = hid_es;
        op.ldy = WIDTH;
        op.out = last ? out : nullptr;
        op.out_es = (long)batch * v.N[l];
        int rc = launch_fwd_tma(op, op.x_es, v.E, d_status, st);
        if (rc) return rc;
    }
    return HGB_OK;
}

int hgb_mlp_forward_fused(const hgb_mlp *net, const uint16_t *x, long x_member_stride, int batch, float *out,
                          int *d_status, void *stream) {
    HGB_CHECK_ARG(check_net(net) && net->params && net->weights && x && out && batch >= 0);
    HGB_CHECK_ARG(x_member_stride >= 0 && batch <= HGB_MLP_FUSED_MAX_BATCH && net->n_members <= 65535);
    HGB_CHECK_ARG(((uintptr_t)net->weights & 15) == 0);   // bulk-copy source alignment
    if (batch == 0) return HGB_OK;
    const NetView v = view_of(net);
    FusedArgs fa{};
    fa.L = v.L;
    fa.batch = batch;
    for (int l = 0; l < v.L; l++) {
        fa.K[l] = v.K[l];
        fa.N[l] = v.N[l];
        fa.w_off[l] = v.w_off[l];
        fa.b_off[l] = v.b_off[l];
    }
    fa.n_w = v.n_w;
    fa.n_p = v.n_p;
    fa.weights = (const bf16 *)net->weights;
    fa.params = net->params;
    fa.x = (const bf16 *)x;
    fa.x_es = x_member_stride;
    fa.out = out;
    fa.status = d_status;
    const size_t smem = fused_smem_bytes(v, &fa);
    int rc = hgb::ensure_dyn_smem((const void *)k_mlp_fwd_fused, smem);
    if (rc) return rc;
    dim3 grid(FUSED_CL, (unsigned)v.E);
    k_mlp_fwd_fused<<<grid, FUSED_THREADS, smem, (cudaStream_t)stream>>>(fa);
    return hgb::check_launch();
}

int hgb_emulator_query(const hgb_mlp *net, const double *params, int n_queries, int n_params, const double *lo,
                       const double *hi, const double *mu, const double *sd, int n_out, uint16_t *x_host,
                       float *out_host, int *status_host, double *result, void *stream) {
    HGB_CHECK_ARG(check_net(net) && params && lo && hi && mu && sd && x_host && out_host && status_host && result);
    HGB_CHECK_ARG(n_queries >= 1 && n_queries <= HGB_MLP_FUSED_MAX_BATCH && n_params >= 1);
    HGB_CHECK_ARG(n_params <= net->dims[0] && n_out >= 1 && n_out <= net->dims[net->n_layers]);
    const int K0 = net->dims[0], NL = net->dims[net->n_layers], E = net->n_members;
    // inputs: 2 (p - lo) / (hi - lo) - 1 rounded to float, then to bf16 (nearest, ties to even)
    for (int q = 0; q < n_queries; q++)
        for (int k = 0; k < K0; k++) {
            uint16_t bits = 0;
            if (k < n_params) {
                const double u = (params[(long)q * n_params + k] - lo[k]) / (hi[k] - lo[k]);
                const float f = (float)(2.0 * u - 1.0);
                uint32_t w;
                memcpy(&w, &f, sizeof(w));
                bits = (uint16_t)((w + 0x7FFFu + ((w >> 16) & 1u)) >> 16);
            }
            x_host[(long)q * K0 + k] = bits;
        }
    *(volatile int *)status_host = 0;
    int rc = hgb_mlp_forward_fused(net, x_host, 0, n_queries, out_host, status_host, stream);
    if (rc) return rc;
    cudaError_t err = cudaStreamSynchronize((cudaStream_t)stream);
    if (err != cudaSuccess) {
        hgb::set_cuda_error(err);
        return HGB_ERR_CUDA;
    }
    if (*(volatile int *)status_host) return HGB_ERR_DEVICE_LIMIT;
    // the ensemble mean in the statistics' units: mean over members, then * sd + mu
    for (int q = 0; q < n_queries; q++)
        for (int k = 0; k < n_out; k++) {
            double acc = 0.0;
            for (int e = 0; e < E; e++) acc += (double)out_host[((long)e * n_queries + q) * NL + k];
            result[(long)q * n_out + k] = acc / E * sd[k] + mu[k];
        }
    return HGB_OK;
}

size_t hgb_mlp_backward_workspace_bytes(const hgb_mlp *net, int batch) {
    if (!check_net(net) || batch <= 0) return 0;
    const NetView v = view_of(net);
    const int nsplit = (int)hgb::ceil_div(batch, HGB_MLP_SPLIT_ROWS);
    size_t bytes = sizeof(uint16_t) * (size_t)v.L * v.E * batch * WIDTH;   // dZ per layer
    for (int l = 0; l < v.L; l++) bytes += sizeof(float) * (size_t)v.E * nsplit * v.N[l] * v.K[l];
    return bytes + sizeof(float) * (size_t)v.E * MSE_BLOCKS;
}

int hgb_mlp_backward(const hgb_mlp *net, const uint16_t *x, long x_member_stride, int batch, const uint16_t *act,
                     const float *pre, const float *out, const float *target, long target_member_stride, float *grad,
                     float *loss, void *workspace, size_t workspace_bytes, int *d_status, void *stream) {
    HGB_CHECK_ARG(check_net(net) && net->params && net->weights && x && act && pre && out && target && grad);
    HGB_CHECK_ARG(batch >= 1 && x_member_stride >= 0 && target_member_stride >= 0);
    HGB_CHECK_ARG(workspace && workspace_bytes >= hgb_mlp_backward_workspace_bytes(net, batch));
    const NetView v = view_of(net);
    cudaStream_t st = (cudaStream_t)stream;
    const long hid_es = (long)batch * WIDTH, hid_ls = (long)v.E * hid_es;
    const int nsplit = (int)hgb::ceil_div(batch, HGB_MLP_SPLIT_ROWS);
    bf16 *dz = (bf16 *)workspace;
    float *part = (float *)((char *)workspace + sizeof(uint16_t) * (size_t)v.L * hid_ls);
    GradArgs ga{};
    ga.v = v;
    ga.batch = batch;
    ga.nsplit = nsplit;
    ga.dz_es = hid_es;
    ga.grad = grad;
    {
        float *pp = part;
        for (int l = 0; l < v.L; l++) {
            ga.part[l] = pp;
            ga.dz[l] = dz + l * hid_ls;
            pp += (size_t)v.E * nsplit * v.N[l] * v.K[l];
        }
    }
    const int last = v.L - 1;
    float *loss_part = part;
    for (int l = 0; l < v.L; l++) loss_part += (size_t)v.E * nsplit * v.N[l] * v.K[l];
    k_mse<<<dim3(MSE_BLOCKS, (unsigned)v.E), 256, 0, st>>>(batch, v.N[last], out, target, target_member_stride,
                                                           dz + last * hid_ls, hid_es, loss_part);
    int rc = hgb::check_launch();
    if (rc) return rc;
    for (int l = last; l >= 0; l--) {
        BwdLayer L{};
        L.dw.dz = dz + l * hid_ls;
        L.dw.dz_es = hid_es;
        L.dw.x = l == 0 ? (const bf16 *)x : (const bf16 *)act + (l - 1) * hid_ls;
        L.dw.x_es = l == 0 ? x_member_stride : hid_es;
        L.dw.ldx = l == 0 ? v.K[0] : WIDTH;
        L.dw.x_aligned = l > 0 || (((uintptr_t)x | (uintptr_t)(2 * x_member_stride)) & 15) == 0;
        L.dw.part = const_cast<float *>(ga.part[l]);
        L.dw.K = v.K[l];
        L.dw.N = v.N[l];
        L.dw.batch = batch;
        L.dw.nsplit = nsplit;
        L.dw_rows = (int)hgb::ceil_div(v.N[l], TM);
        L.dw_cols = (int)hgb::ceil_div(v.K[l], DwOp::NT);
        L.nsplit = nsplit;
        if (l > 0) {
            L.dx.dz = dz + l * hid_ls;
            L.dx.dz_es = hid_es;
            L.dx.w = (const bf16 *)net->weights + v.w_off[l];
            L.dx.w_es = v.n_w;
            L.dx.w_aligned = ((uintptr_t)net->weights & 15) == 0;   // layers and members: multiples of 256 values
            L.dx.pre = pre + (l - 1) * hid_ls;
            L.dx.pre_es = hid_es;
            L.dx.dzp = dz + (l - 1) * hid_ls;
            L.dx.dzp_es = hid_es;
            L.dx.K = v.K[l];
            L.dx.N = v.N[l];
            L.dx.batch = batch;
            L.dx_rows = (int)hgb::ceil_div(batch, TM);
            L.dx_cols = (int)hgb::ceil_div(v.K[l], DxOp::NT);
        }
        if ((rc = launch_bwd(L, v.E, d_status, st))) return rc;
    }
    ga.loss_part = loss_part;
    ga.loss = loss;
    ga.w_blocks = (int)hgb::ceil_div((long)v.E * v.n_p, 256);
    ga.bias_tiles = 0;
    for (int l = 0; l < v.L; l++) ga.bias_tiles += (v.N[l] + 31) / 32;
    k_grad_reduce<<<(unsigned)(ga.w_blocks + v.E * ga.bias_tiles + 1), 256, 0, st>>>(ga);
    return hgb::check_launch();
}

int hgb_mlp_adamw(const hgb_mlp *net, float *params, const float *grad, float *m1, float *m2, uint16_t *weights,
                  int step, float lr, float beta1, float beta2, float eps, float weight_decay, void *stream) {
    HGB_CHECK_ARG(check_net(net) && params && grad && m1 && m2 && weights && step >= 1);
    const NetView v = view_of(net);
    const long np = (long)v.E * v.n_p;
    const float bc1 = 1.0f - powf(beta1, (float)step), bc2 = 1.0f - powf(beta2, (float)step);
    k_adamw<<<(unsigned)hgb::ceil_div(np, 256), 256, 0, (cudaStream_t)stream>>>(
        v, params, grad, m1, m2, (bf16 *)weights, lr, beta1, beta2, eps, weight_decay, bc1, bc2);
    return hgb::check_launch();
}

int hgb_mlp_pack_weights(const hgb_mlp *net, const float *params, uint16_t *weights, void *stream) {
    HGB_CHECK_ARG(check_net(net) && params && weights);
    const NetView v = view_of(net);
    const long np = (long)v.E * v.n_p;
    k_pack_weights<<<(unsigned)hgb::ceil_div(np, 256), 256, 0, (cudaStream_t)stream>>>(v, params, (bf16 *)weights);
    return hgb::check_launch();
}

}  // extern "C"
