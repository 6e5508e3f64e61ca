// W8A8 integer GEMM: C (s32) = A (u8 activations) x W (s8 weights), exact, on tcgen05 (kind::i8) with the
// accumulator in tensor memory; plus the dequantize epilogue of the reference as a separate element-wise pass.
//
//   C[t, r] = sum_k A[t, k] * W[r, k]          t < M tokens, r < N weight rows        (all integers, no rounding)
//
// Counterpart: avx512_int8::gemm_int8 / dequantize_i32_to_f32 (src/macros/matmul_x86_int8.rs:307-440), whose B
// operand is [K, N] row-major s8 (and a packed copy of it).  Here the weight is repacked once into 16 KB tile
// images (128 rows x 128 k, 128-byte swizzle, order [row tile][k-step]) and the u8 activations are turned into
// the same kind of images per call, so every operand stage is a plain bulk copy; one thread issues four
// tcgen05.mma of K = 32 per stage into a 128 x N s32 accumulator; eight warps store it (transposed through
// shared memory, 16 bytes per lane).  Weights on the M side as in the other prefill kernels.
#include "common.cuh"
#include "tc05.cuh"

#include <cfloat>
#include <type_traits>

namespace gllmk {

constexpr int I8_BM = 128, I8_BN = 256, I8_TILE = 16384;
constexpr int I8_MAX_STAGES = 4;
// a stage = MT weight tiles + up to two activation tiles; MT = 2 (two accumulators share one activation stage)
// needs a third fewer bytes from L2 per MAC, which is what bounds this kernel
template <int MT>
__host__ __device__ constexpr int i8_stage_bytes() { return MT * I8_TILE + 2 * I8_TILE; }
template <int MT>
__host__ __device__ constexpr int i8_stages() { return MT == 2 ? 3 : 4; }
constexpr int I8_EPI_WARPS = 8;
constexpr int I8_THREADS = 64 + 32 * I8_EPI_WARPS;     // warp 0: copies, warp 1: MMA + TMEM, then the epilogue warps
template <int MT>
__host__ __device__ constexpr size_t i8_smem() { return (size_t)i8_stages<MT>() * i8_stage_bytes<MT>() + 1024; }

struct I8Params {
    const uint8_t *w;   // weight tile images
    const uint8_t *xt;  // activation tile images [token tile of 128][k-step][16384]
    int64_t n;
    int row_tiles;
    int nks;            // k-steps of 128
    int m;
    void *c;            // [m, n] row-major, leading dimension ldc: s32 products, or (EPI) the finished f32 outputs
    int64_t ldc;
    int vec;
    int *status;
    // EPI (a whole W8A8 linear layer): the epilogue of dequant_i32_kernel on the accumulator while it is in registers
    const float *scale_a;   // device memory: written by the activation quantizer of the same stream
    const int32_t *colsum;  // sum_k W[j, k]: the activations are stored as q + 128
    const float *bias;      // nullptr: none
    float scale_b;
    int act;
};

// v / (1 + exp(-z)): SiLU with z = v; the tanh form of GELU, 0.5 v (1 + tanh(u)) = v / (1 + exp(-2u)), with z = 2u (and no
// cancellation for negative u).  The quotient is Markstein's (q = v y, q += (v - q d) y, y an approximate 1 / d): no branch,
// so the chains of a thread's 32 elements overlap; the compiler's IEEE division has one per element, and the fused
// epilogue of gemm_i8_pair_kernel then took 134 us on W[11008, 4096] x 2048 (82 now; the product without it 72).
// y comes from d / 8, because 1 / d itself would be 0 from d = 2^126 on (SiLU(-88) = -0 instead of -5e-37).
// v and q infinite (v = inf, d = 1) or exp overflown (d = inf, y = 0): the residual is the NaN of inf - inf or 0 * inf.  fmax takes
// the other operand then, and q is the answer (inf, or 0).
__device__ __forceinline__ float sigmoid_times(float v, float z) {
    const float d = 1.0f + expf(-z);
    float y;  // 1 / 8 <= d / 8 <= 2^125: neither side of the reciprocal is subnormal
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d * 0.125f));
    y *= 0.125f;
    const float q = v * y;
    return fmaf(fmaxf(fmaf(-q, d, v), -FLT_MAX), y, q);
}
// dequantize_i32_to_f32 (src/macros/matmul_x86_int8.rs:414-456, scalar tail semantics): (c as f32) * scale_a * scale_b
// (+ bias[j]), then the activation of src/macros/gemm_epilogue.rs:131-152
template <int ACT>
__device__ __forceinline__ float i8_dequant(int32_t c, float scale_a, float scale_b, bool has_bias, float bias) {
    float v = __fmul_rn(__fmul_rn((float)c, scale_a), scale_b);
    if (has_bias) v = __fadd_rn(v, bias);
    if (ACT == 1) v = v < 0.0f ? 0.0f : v;
    else if (ACT == 2) v = sigmoid_times(v, v);
    else if (ACT == 3) v = sigmoid_times(v, 2.0f * (0.7978845608f * (v + 0.044715f * v * v * v)));
    return v;
}
// the activation as a compile-time constant (GELU and GEGLU share a formula)
template <typename F>
__device__ __forceinline__ void with_act(int act, F &&f) {
    if (act == 0) f(std::integral_constant<int, 0>{});
    else if (act == 1) f(std::integral_constant<int, 1>{});
    else if (act == 2) f(std::integral_constant<int, 2>{});
    else f(std::integral_constant<int, 3>{});
}

// One 32-row x 32-token block of accumulators (lane = weight row) made ready for the 32-bit store helper: the s32 bit
// patterns as they are, or (EPI) the layer's f32 outputs.  In the linear layer the accumulator never goes to memory: as a
// pass of its own over the s32 products this epilogue moved 8 bytes per output (W[11008, 4096] x 2048 tokens: 95 of 230 us).
struct I8Lane {  // what a lane's weight row contributes (EPI)
    float scale_a, bias;
    int32_t off;  // 128 * colsum of the row: exact, the s32 range holds both terms for k < 66000
};
template <bool EPI>
__device__ __forceinline__ I8Lane i8_lane(const I8Params &p, int64_t row) {
    I8Lane l{0.0f, 0.0f, 0};
    if constexpr (EPI) {
        l.scale_a = *p.scale_a;
        if (row < p.n) {
            l.off = 128 * p.colsum[row];
            if (p.bias) l.bias = p.bias[row];
        }
    }
    return l;
}
template <bool EPI>
__device__ __forceinline__ void i8_finish(const I8Params &p, const I8Lane &l, const uint32_t (&v)[32], float (&o)[32]) {
    if constexpr (EPI) {
        with_act(p.act, [&](auto act) {
#pragma unroll
            for (int j = 0; j < 32; j++) o[j] = i8_dequant<act.value>((int32_t)v[j] - l.off, l.scale_a, p.scale_b, p.bias != nullptr, l.bias);
        });
    } else {
#pragma unroll
        for (int j = 0; j < 32; j++) o[j] = __uint_as_float(v[j]);
    }
}

__device__ __forceinline__ void i8_bulk(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}

// ---- repack: s8 weights [K, N] (layout 0, the reference's B) or [N, K] (layout 1) -> tile images; thread = 16 k of a row
__global__ void __launch_bounds__(256) repack_i8_kernel(const int8_t *__restrict__ b, uint8_t *__restrict__ out, int64_t n, int64_t k,
                                                        int64_t k_pad, int layout, size_t total) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;  // (k chunk, padded row): rows fastest for layout 0
    if (idx >= total) return;
    const int64_t n_pad = (n + 127) / 128 * 128;
    const int64_t row = (int64_t)(idx % (size_t)n_pad), kc = (int64_t)(idx / (size_t)n_pad);
    uint32_t v[4] = {0, 0, 0, 0};
    if (row < n) {
        for (int i = 0; i < 16; i++) {
            const int64_t kk = kc * 16 + i;
            if (kk < k) {
                const uint8_t by = (uint8_t)(layout == 0 ? b[kk * n + row] : b[row * k + kk]);
                v[i >> 2] |= (uint32_t)by << (8 * (i & 3));
            }
        }
    }
    const size_t tile = (size_t)(row >> 7) * (size_t)(k_pad >> 7) + (size_t)(kc >> 3);
    *reinterpret_cast<uint4 *>(out + tile * I8_TILE + tc::sw128_offset((int)(row & 127), (int)(kc & 7))) = make_uint4(v[0], v[1], v[2], v[3]);
}

// ---- u8 activations [m, k] (leading dimension lda, any alignment) -> tile images; grid (k-steps, token tiles of 128)
__global__ void __launch_bounds__(256) stage_act_u8_kernel(const uint8_t *__restrict__ a, int64_t lda, int m, int64_t k,
                                                           uint8_t *__restrict__ xt) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const int ks = blockIdx.x, tile = blockIdx.y;
    uint8_t *dst = xt + ((size_t)tile * gridDim.x + ks) * I8_TILE;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int item = threadIdx.x + 256 * i, row = item >> 3, chunk = item & 7;
        const int64_t tok = (int64_t)tile * 128 + row, k0 = (int64_t)ks * 128 + chunk * 16;
        uint32_t v[4] = {0, 0, 0, 0};
        if (tok < m) {
            const uint8_t *src = a + tok * lda + k0;
            for (int j = 0; j < 16; j++)
                if (k0 + j < k) v[j >> 2] |= (uint32_t)src[j] << (8 * (j & 3));
        }
        *reinterpret_cast<uint4 *>(dst + tc::sw128_offset(row, chunk)) = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

// grid (groups of MT weight-row tiles, token tiles of 256); ntok = MMA N (multiple of 32, <= 256)
template <int MT, bool EPI>
__global__ void __launch_bounds__(I8_THREADS, 1) gemm_i8_kernel(const __grid_constant__ I8Params p, const int ntok) {
    constexpr int I8_STAGES = i8_stages<MT>(), I8_STAGE_BYTES = i8_stage_bytes<MT>();
    constexpr uint32_t TMEM_COLS = MT == 2 ? 512 : 256;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * I8_MAX_STAGES + 1];
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_s;
    const uint32_t smem_s = (tc::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t full = tc::smem_u32(&bars[0]), empty = tc::smem_u32(&bars[I8_MAX_STAGES]), accum = tc::smem_u32(&bars[2 * I8_MAX_STAGES]);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile0 = (int)blockIdx.x * MT;
    const int mt = min(MT, p.row_tiles - tile0);  // row tiles this CTA really has
    const int64_t tok0 = (int64_t)blockIdx.y * I8_BN;
    volatile int *abort_flag = &abort_s;

    if (threadIdx.x == 0) {
        abort_s = 0;
        for (int s = 0; s < I8_STAGES; s++) {
            tc::mbar_init(full + 8 * s, 1);
            tc::mbar_init(empty + 8 * s, 1);
        }
        tc::mbar_init(accum, 1);
        tc::mbar_init_fence();
    }
    if (warp == 1) tc::tmem_alloc(tc::smem_u32(&tmem_base_s), TMEM_COLS);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base_s;

    if (warp == 0 && lane == 0) {
        // ---------------- copies: one weight tile and one or two activation tiles per k-step ----------------
        const int halves = (ntok + 127) / 128;
        const uint32_t bbytes = (uint32_t)ntok * 128u;
        const uint32_t hb[2] = {ntok > 128 ? (uint32_t)I8_TILE : bbytes, bbytes - (uint32_t)I8_TILE};
        asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the activation images are complete from here on
        for (int ks = 0; ks < p.nks; ks++) {
            const int s = ks % I8_STAGES;
            if (ks >= I8_STAGES && !tc::mbar_wait(empty + 8 * s, (uint32_t)((ks / I8_STAGES - 1) & 1), abort_flag)) {
                abort_s = 1;
                atomicExch(p.status, 41);
                break;
            }
            const uint32_t st = smem_s + s * I8_STAGE_BYTES;
            tc::mbar_expect_tx(full + 8 * s, (uint32_t)(mt * I8_TILE) + bbytes);
            for (int i = 0; i < mt; i++)
                i8_bulk(st + i * I8_TILE, p.w + ((size_t)(tile0 + i) * p.nks + ks) * I8_TILE, I8_TILE, full + 8 * s);
            for (int h = 0; h < halves; h++)
                i8_bulk(st + MT * I8_TILE + h * I8_TILE, p.xt + ((size_t)((tok0 >> 7) + h) * p.nks + ks) * I8_TILE, hb[h], full + 8 * s);
        }
    } else if (warp == 1) {
        // ---------------- MMA issue: weights signed (operand A), activations unsigned (operand B) ----------------
        // (the whole warp walks the k-steps, one elected lane issues: addresses and descriptors are uniform values)
        const uint32_t idesc = tc::idesc_i8(I8_BM, ntok, 1, 0), tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
        asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the bound of the waits starts when the images exist
        for (int ks = 0; ks < p.nks; ks++) {
            const int s = ks % I8_STAGES;
            if (!tc::mbar_spin_warp(full + 8 * s, (uint32_t)((ks / I8_STAGES) & 1), abort_flag)) {
                if (lane == 0) {
                    abort_s = 1;
                    atomicExch(p.status, 42);
                }
                break;
            }
            tc::fence_after_sync();
            const uint32_t st = smem_s + s * I8_STAGE_BYTES;
            const uint64_t bd = tc::smem_desc_sw128(st + MT * I8_TILE);
            if (tc::elect_one()) {
                for (int i = 0; i < mt; i++) {
                    const uint64_t ad = tc::smem_desc_sw128(st + i * I8_TILE);
#pragma unroll
                    for (int j = 0; j < 4; j++) tc::mma_i8(tmem_u + 256u * (uint32_t)i, ad + 2 * j, bd + 2 * j, idesc, (uint32_t)((ks | j) != 0));
                }
                tc::mma_commit(empty + 8 * s);
                if (ks == p.nks - 1) tc::mma_commit(accum);
            }
            __syncwarp();
        }
    }
    __syncwarp();

    if (warp >= 2) {
        // ---------------- epilogue: warp w reads TMEM lane quadrant w % 4 = weight rows ----------------
        const int quad = warp & 3;
        asm volatile("griddepcontrol.wait;\n" ::: "memory");  // as the MMA warp; and this thread reads the activation scale
        bool ok = !abort_s && tc::mbar_wait(accum, 0u, abort_flag);
        if (!ok && !abort_s) {
            abort_s = 1;
            atomicExch(p.status, 43);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            tc::fence_after_sync();
            // all MMAs have completed, so the stages are free: each warp stages its blocks in 4 KB of stage 0
            uint8_t *stage = smem_raw + (smem_s - tc::smem_u32(smem_raw)) + (warp - 2) * 4096;
            for (int i = 0; i < mt; i++) {
                const int64_t row0 = (int64_t)(tile0 + i) * I8_BM;
                const I8Lane l = i8_lane<EPI>(p, row0 + 32 * quad + lane);
                for (int c = 32 * ((warp - 2) >> 2); c < ntok; c += 32 * (I8_EPI_WARPS / 4)) {
                    uint32_t v[32];
                    tc::tmem_ld32(tmem + ((uint32_t)(32 * quad) << 16) + 256u * (uint32_t)i + (uint32_t)c, v);
                    tc::tmem_ld_wait();
                    float o[32];
                    i8_finish<EPI>(p, l, v, o);
                    tc::store_block_32x32<false>(p.c, p.ldc, row0 + 32 * quad, tok0 + c, p.n, p.m, o, stage, lane, p.vec);
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) tc::tmem_dealloc(tmem, TMEM_COLS);
}

// ---------------------------------------------------------------------------------------------
// m > 128: CTA pairs (tcgen05 cta_group::2, MMA M = 256), persistent, two accumulators.
//
// The kernel above runs at what an SM can take in from L2: 64 KB per k-step for two 128 x 256 tiles.  As a pair, each
// CTA brings in its own 128 weight rows and HALF of the 256-token activation tile (the tensor core reads the other half
// from the partner's shared memory): 32 KB per k-step and tile.  One 256-column accumulator per tile leaves room for a
// second one, so the eight epilogue warps store tile i while the MMA thread fills the accumulator of tile i + 1, and the
// grid is the resident pairs with tiles dealt round robin.  Structure and hand-shakes are those of gemm_fp4_pair_kernel
// (gemm_fp4.cu) without the scale-factor path: the partner's copy thread cannot signal the leader's barrier with a plain
// bulk copy, so a relay thread forwards "my stage has landed"; stages go back to both CTAs with one commit per barrier.
// ---------------------------------------------------------------------------------------------
constexpr int I8P_STAGES = 6, I8P_STAGE_BYTES = 2 * I8_TILE, I8P_EPI_WARPS = 8;
constexpr int I8P_THREADS = 64 + 32 * I8P_EPI_WARPS;
constexpr size_t I8P_SMEM = (size_t)I8P_STAGES * I8P_STAGE_BYTES + (size_t)I8P_EPI_WARPS * 4096 + 1024;

template <bool EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(I8P_THREADS, 1)
gemm_i8_pair_kernel(const __grid_constant__ I8Params p, const int tok_tiles, const int x_tiles) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[3 * I8P_STAGES + 4];
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_s;
    const uint32_t smem_s = (tc::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t full = tc::smem_u32(&bars[0]), empty = tc::smem_u32(&bars[I8P_STAGES]), full2 = tc::smem_u32(&bars[2 * I8P_STAGES]);
    const uint32_t accum_full = tc::smem_u32(&bars[3 * I8P_STAGES]), accum_empty = accum_full + 16;  // two each
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = tc::cluster_ctarank();
    const int pair = (int)(blockIdx.x >> 1), npairs = (int)(gridDim.x >> 1);
    const int row_pairs = (p.row_tiles + 1) >> 1;
    const int ntiles = row_pairs * tok_tiles;
    volatile int *abort_flag = &abort_s;

    if (threadIdx.x == 0) {
        abort_s = 0;
        for (int s = 0; s < I8P_STAGES; s++) {
            tc::mbar_init(full + 8 * s, 1);
            tc::mbar_init(empty + 8 * s, 1);
            tc::mbar_init(full2 + 8 * s, 1);
        }
        for (int a = 0; a < 2; a++) {
            tc::mbar_init(accum_full + 8 * a, 1);
            tc::mbar_init(accum_empty + 8 * a, 2 * I8P_EPI_WARPS);  // the epilogue warps of both CTAs (used in the leader only)
        }
        tc::mbar_init_fence();
    }
    if (warp == 1) tc::tmem_alloc_pair(tc::smem_u32(&tmem_base_s), 512);
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_arrive();  // both CTAs' barriers exist before either CTA arrives on the other's
    tc::cluster_wait();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base_s;

    if (warp == 0 && lane == 0) {
        // ---------------- copies: own weight rows, own half of the activation tile ----------------
        uint32_t g = 0;
        asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the activation images are complete from here on
        for (int t = pair; t < ntiles && !*abort_flag; t += npairs) {
            const int rp = t / tok_tiles, tt = t % tok_tiles;
            const int my_row_tile = 2 * rp + (int)rank, my_x_tile = 2 * tt + (int)rank;
            const bool a_ok = my_row_tile < p.row_tiles, b_ok = my_x_tile < x_tiles;
            // rows / tokens that do not exist are not copied: what the stage holds there only reaches accumulator rows /
            // columns that are never stored
            const uint32_t tx = (a_ok ? (uint32_t)I8_TILE : 0u) + (b_ok ? (uint32_t)I8_TILE : 0u);
            for (int ks = 0; ks < p.nks; ks++, g++) {
                const uint32_t s = g % I8P_STAGES;
                if (g >= (uint32_t)I8P_STAGES && !tc::mbar_wait_cluster(empty + 8 * s, (g / I8P_STAGES - 1) & 1u, abort_flag)) {
                    abort_s = 1;
                    atomicExch(p.status, 44);
                    break;
                }
                const uint32_t st = smem_s + s * I8P_STAGE_BYTES;
                tc::mbar_expect_tx(full + 8 * s, tx);
                if (a_ok) i8_bulk(st, p.w + ((size_t)my_row_tile * p.nks + ks) * I8_TILE, I8_TILE, full + 8 * s);
                if (b_ok) i8_bulk(st + I8_TILE, p.xt + ((size_t)my_x_tile * p.nks + ks) * I8_TILE, I8_TILE, full + 8 * s);
            }
        }
    } else if (warp == 1 && lane == 0 && rank != 0) {
        // ---------------- partner CTA: tell the leader when this CTA's stage has landed ----------------
        uint32_t g = 0;
        bool ok = true;
        asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the bound of the waits starts when the images exist
        for (int t = pair; t < ntiles && ok && !*abort_flag; t += npairs)
            for (int ks = 0; ks < p.nks; ks++, g++) {
                const uint32_t s = g % I8P_STAGES;
                if (!tc::mbar_wait(full + 8 * s, (g / I8P_STAGES) & 1u, abort_flag)) {
                    abort_s = 1;
                    atomicExch(p.status, 45);
                    ok = false;
                    break;
                }
                // the stage's bytes are in place before this arrive is issued (the barrier phase was observed)
                tc::mbar_arrive_cluster_relaxed(tc::map_to_cta(full2 + 8 * s, 0));
            }
    } else if (warp == 1 && rank == 0) {
        // ---------------- leader CTA: MMA issue for the pair, accumulator (tile & 1) ----------------
        // (the whole warp walks the k-steps, one elected lane issues: addresses and descriptors are uniform values)
        const uint32_t idesc = tc::idesc_i8(256, I8_BN, 1, 0);  // weights signed (operand A), activations unsigned (operand B)
        const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
        asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the bound of the waits starts when the images exist
        uint32_t g = 0, it = 0;
        bool ok = true;
        for (int t = pair; t < ntiles && ok; t += npairs, it++) {
            const uint32_t acc = it & 1u;
            // the tile before last used this accumulator: all sixteen epilogue warps of the pair have read it out
            if (it >= 2 && !tc::mbar_spin_warp_cluster(accum_empty + 8 * acc, ((it >> 1) - 1) & 1u, abort_flag)) {
                if (lane == 0) {
                    abort_s = 1;
                    atomicExch(p.status, 46);
                }
                break;
            }
            tc::fence_after_sync();
            const uint32_t td = tmem_u + 256u * acc;
            for (int ks = 0; ks < p.nks; ks++, g++) {
                const uint32_t s = g % I8P_STAGES, ph = (g / I8P_STAGES) & 1u;
                if (!tc::mbar_spin_warp(full + 8 * s, ph, abort_flag) || !tc::mbar_spin_warp_cluster(full2 + 8 * s, ph, abort_flag)) {
                    if (lane == 0) {
                        abort_s = 1;
                        atomicExch(p.status, 42);
                    }
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                const uint32_t st = smem_s + s * I8P_STAGE_BYTES;
                const uint64_t ad = tc::smem_desc_sw128(st), bd = tc::smem_desc_sw128(st + I8_TILE);
                const uint32_t empty1 = tc::map_to_cta(empty + 8 * s, 1), full1 = tc::map_to_cta(accum_full + 8 * acc, 1);
                if (tc::elect_one()) {
#pragma unroll
                    for (int j = 0; j < 4; j++) tc::mma_i8_pair(td, ad + 2 * j, bd + 2 * j, idesc, (uint32_t)((ks | j) != 0));
                    // once these MMAs have completed, stage s is free in BOTH CTAs
                    tc::mma_commit_pair(empty + 8 * s);
                    tc::mma_commit_pair(empty1);
                    if (ks == p.nks - 1) {
                        tc::mma_commit_pair(accum_full + 8 * acc);
                        tc::mma_commit_pair(full1);
                    }
                }
                __syncwarp();
            }
        }
    }
    __syncwarp();

    if (warp >= 2) {
        // ---------------- epilogue: this CTA's 128 rows x 256 tokens of accumulator (tile & 1) ----------------
        // warp w reads TMEM lane quadrant w % 4; the two warps of a quadrant take 128 token columns each
        const int quad = warp & 3, half = (warp - 2) >> 2;
        uint8_t *stage = smem_raw + (smem_s - tc::smem_u32(smem_raw)) + (size_t)I8P_STAGES * I8P_STAGE_BYTES + (size_t)(warp - 2) * 4096;
        const uint32_t accum_empty_leader = tc::map_to_cta(accum_empty, 0);
        uint32_t it = 0;
        asm volatile("griddepcontrol.wait;\n" ::: "memory");  // this thread reads the activation scale
        for (int t = pair; t < ntiles; t += npairs, it++) {
            const uint32_t acc = it & 1u;
            bool ok = !abort_s && tc::mbar_wait_cluster(accum_full + 8 * acc, (it >> 1) & 1u, abort_flag);
            if (!ok && !abort_s) {
                abort_s = 1;
                atomicExch(p.status, 43);
            }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc::fence_after_sync();
            const int rp = t / tok_tiles, tt = t % tok_tiles;
            const int64_t row0 = (int64_t)(2 * rp + (int)rank) * I8_BM + 32 * quad, tok0 = (int64_t)tt * I8_BN + 128 * half;
            const uint32_t tbase = tmem + ((uint32_t)(32 * quad) << 16) + 256u * acc + (uint32_t)(128 * half);
            const I8Lane l = i8_lane<EPI>(p, row0 + lane);
#pragma unroll 1
            for (int c = 0; c < 128; c += 32) {
                uint32_t v[32];
                tc::tmem_ld32(tbase + (uint32_t)c, v);
                tc::tmem_ld_wait();
                if (row0 < p.n && tok0 + c < p.m) {
                    float o[32];
                    i8_finish<EPI>(p, l, v, o);
                    tc::store_block_32x32<false>(p.c, p.ldc, row0, tok0 + c, p.n, p.m, o, stage, lane, p.vec);
                }
            }
            // this warp's reads of the accumulator are complete (wait::ld): the leader may reuse it for the tile after next
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive_cluster_relaxed(accum_empty_leader + 8 * acc);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    // neither CTA may leave (or give TMEM back) while the pair's MMAs can still read its shared memory
    tc::cluster_arrive();
    tc::cluster_wait();
    if (warp == 1) tc::tmem_dealloc_pair(tmem, 512);
}

// the epilogue as a pass of its own (gllmk_dequantize_i32_f32)
__global__ void __launch_bounds__(256) dequant_i32_kernel(const int32_t *__restrict__ c, float *__restrict__ out, int64_t n, float scale_a,
                                                          float scale_b, const float *__restrict__ bias, int act, size_t total) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const float b = bias ? bias[idx % (size_t)n] : 0.0f;
    with_act(act, [&](auto a) { out[idx] = i8_dequant<a.value>(c[idx], scale_a, scale_b, bias != nullptr, b); });
}

// ---------------------------------------------------------------------------------------------
// one warp per weight row j: colsum[j] = sum_k B[k, j]
__global__ void __launch_bounds__(256) i8_colsum_kernel(const int8_t *__restrict__ b, int64_t n, int64_t k, int layout, int32_t *__restrict__ colsum) {
    const int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (j >= n) return;
    int32_t acc = 0;
    for (int64_t kk = lane; kk < k; kk += 32) acc += layout == 0 ? (int32_t)b[kk * n + j] : (int32_t)b[j * k + kk];
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) colsum[j] = acc;
}

int32_t i8_weight_fill(Ctx *c, Weight *w, const int8_t *b_dev, int layout, cudaStream_t s) {
    const size_t total = (size_t)w->n_pad * (size_t)(w->k_pad / 16);
    repack_i8_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(b_dev, static_cast<uint8_t *>(w->qs), w->n, w->k, w->k_pad, layout, total);
    GK_CUDA(c, cudaGetLastError());
    if (w->aux) {  // per-column sums of B: the zero-point correction of the f32 -> u8 activation path
        i8_colsum_kernel<<<(unsigned)((w->n * 32 + 255) / 256), 256, 0, s>>>(b_dev, w->n, w->k, layout, static_cast<int32_t *>(w->aux));
        GK_CUDA(c, cudaGetLastError());
    }
    return GLLMK_STATUS_OK;
}

// quantize_from_fp32 / QuantFormat::Int8PerTensor (src/compiler/quant_convert.rs:17-20,165-177): scale = max|x| / 127,
// q = (x / scale).round().clamp(-128, 127) as i8 (round half away from zero; NaN, i.e. 0 / 0 for an all-zero tensor, -> 0).
//
// Two passes, both bound by reading x (the second finds it in L2 up to ~100 MB): the maximum (quantize.cu), then this kernel,
// whose loads of x run before it waits for the first.  x [2048, 4096] from a cold cache: 8 + 16 us (4-byte loads, an atomic
// maximum and a byte image that a third pass turned into tile images: 24 + 41 + 9 us).
constexpr int AQ_ROWS = 8;  // rows (16-byte loads in flight) per thread

// IMG: the quantized activations (as q + 128) go straight into the tile images the integer GEMM copies (128 tokens x 128 k,
// swizzled); otherwise to q [rows, ldq].  A warp takes 128 k of a row (16 bytes in, 4 bytes out per lane: whole lines both
// ways, an image row is one 128-byte line), a thread AQ_ROWS rows, all loaded first.  grid (k / 128, rows / (8 AQ_ROWS)).  Tokens past the last one are
// not written: what an image holds there only reaches accumulator columns that are never stored.
template <bool IMG>
__global__ void __launch_bounds__(256) act_quant_i8_kernel(const float *__restrict__ x, int64_t rows, int64_t k, int64_t ld, int vec,
                                                           uint8_t *__restrict__ q, int64_t ldq, int qvec, int offset,
                                                           const AmaxOut *amax, float *scale_out) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t k0 = (int64_t)blockIdx.x * 128 + 4 * lane;
    float4 v[AQ_ROWS];
#pragma unroll
    for (int i = 0; i < AQ_ROWS; i++) {
        const int64_t r = (int64_t)blockIdx.y * (8 * AQ_ROWS) + 8 * i + warp;
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) {
            const float *src = x + r * ld + k0;
            if (vec && k0 < k) v[i] = __ldg(reinterpret_cast<const float4 *>(src));
            else if (!vec) {
                if (k0 < k) v[i].x = src[0];
                if (k0 + 1 < k) v[i].y = src[1];
                if (k0 + 2 < k) v[i].z = src[2];
                if (k0 + 3 < k) v[i].w = src[3];
            }
        }
    }
    asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the maximum is complete from here on
    const float a = __ldcg(&amax->amax), scale = __fdiv_rn(a, 127.0f);
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        scale_out[0] = scale;
        if (!IMG) scale_out[1] = a;
    }
    // f / scale, correctly rounded: one reciprocal for all elements and two of Markstein's corrections (the first makes the
    // quotient faithful, the second exact); scales so small or large that a step could leave the normal range divide
    const bool fast = scale > 1e-30f && scale < 1e30f;
    const float y = fast ? __frcp_rn(scale) : 0.0f;
    const auto quant = [&](float f) -> uint32_t {
        if (fast) {
            float d = f * y;
            d = fmaf(fmaf(-d, scale, f), y, d);
            f = fmaf(fmaf(-d, scale, f), y, d);
        } else {
            f = __fdiv_rn(f, scale);
        }
        f = roundf(f);
        if (f != f) f = 0.0f;
        f = fminf(fmaxf(f, -128.0f), 127.0f);
        return (uint32_t)((int)f + offset) & 0xFFu;
    };
#pragma unroll
    for (int i = 0; i < AQ_ROWS; i++) {
        const int64_t r = (int64_t)blockIdx.y * (8 * AQ_ROWS) + 8 * i + warp;
        if (r >= rows) continue;
        const uint32_t w = quant(v[i].x) | (quant(v[i].y) << 8) | (quant(v[i].z) << 16) | (quant(v[i].w) << 24);
        if (IMG) {
            uint8_t *dst = q + ((size_t)(r >> 7) * gridDim.x + blockIdx.x) * I8_TILE;
            *reinterpret_cast<uint32_t *>(dst + tc::sw128_offset((int)(r & 127), lane >> 2) + 4 * (lane & 3)) = w;
        } else if (qvec && k0 + 3 < k) {
            *reinterpret_cast<uint32_t *>(q + r * ldq + k0) = w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (k0 + j < k) q[r * ldq + k0 + j] = (uint8_t)(w >> (8 * j));
        }
    }
}

// img: q is the tile images of the integer GEMM (ldq unused), otherwise [rows, ldq] bytes
static int32_t act_quant(Ctx *c, const float *x, int64_t rows, int64_t k, int64_t ld, uint8_t *q, int64_t ldq, int offset, bool img,
                         float *scale_dev, cudaStream_t s) {
    const int vec = (((uintptr_t)x & 15) == 0 && ld % 4 == 0 && k % 4 == 0) ? 1 : 0;
    const int qvec = (((uintptr_t)q & 3) == 0 && ldq % 4 == 0) ? 1 : 0;
    const int32_t rc = amax_launch(c, x, rows, k, ld, nullptr, s);
    if (rc) return rc;
    const AmaxOut *amax = amax_out(c);
    // row groups beyond the grid's y limit: launches of their own (each writes the same scale)
    const int64_t step = (int64_t)65534 * 8 * AQ_ROWS;  // a multiple of the 128 rows of an image
    for (int64_t r0 = 0; r0 < rows; r0 += step) {
        const int64_t nr = rows - r0 < step ? rows - r0 : step;
        const dim3 grid((unsigned)((k + 127) / 128), (unsigned)((nr + 8 * AQ_ROWS - 1) / (8 * AQ_ROWS)));
        uint8_t *dst = img ? q + (size_t)(r0 >> 7) * ((size_t)(k + 127) / 128) * I8_TILE : q + r0 * ldq;
        GK_CUDA(c, img ? launch_after(act_quant_i8_kernel<true>, true, grid, 256, 0, s, x + r0 * ld, nr, k, ld, vec, dst, ldq, qvec, offset, amax, scale_dev)
                       : launch_after(act_quant_i8_kernel<false>, true, grid, 256, 0, s, x + r0 * ld, nr, k, ld, vec, dst, ldq, qvec, offset, amax, scale_dev));
    }
    return GLLMK_STATUS_OK;
}
int32_t act_quant_i8_launch(Ctx *c, const float *x, int64_t rows, int64_t k, int64_t ld, uint8_t *q, int64_t ldq, int offset,
                            float *scale_dev, cudaStream_t s) {
    return act_quant(c, x, rows, k, ld, q, ldq, offset, false, scale_dev, s);
}

template <int MT, bool EPI>
static int32_t i8_launch_mt(Ctx *c, const I8Params &p, dim3 grid, int ntok, cudaStream_t s) {
    static bool attr_set[64] = {};  // function attributes are per device
    const int dev_slot = c->device & 63;
    if (!attr_set[dev_slot]) {
        GK_CUDA(c, cudaFuncSetAttribute(gemm_i8_kernel<MT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)i8_smem<MT>()));
        attr_set[dev_slot] = true;
    }
    GK_CUDA(c, launch_after(gemm_i8_kernel<MT, EPI>, true, grid, I8_THREADS, i8_smem<MT>(), s, p, ntok));
    return GLLMK_STATUS_OK;
}

// Activation images a launch over m tokens reads: 128 tokens each, pairs of them when the token tile is 256 wide
static int i8_act_tiles(int m) { return m > 128 ? 2 * ((m + I8_BN - 1) / I8_BN) : 1; }

// The product from the activation images in the context's scratch (written by the kernel just launched on `s`); p holds the
// output and, with EPI, the epilogue's operands.
template <bool EPI>
static int32_t i8_product(Ctx *c, const Weight *w, I8Params p, int m, cudaStream_t s) {
    const int ntok = m > 128 ? I8_BN : (m + 31) / 32 * 32;
    const int mtiles = (m + I8_BN - 1) / I8_BN;
    p.w = static_cast<const uint8_t *>(w->qs);
    p.xt = static_cast<const uint8_t *>(c->act);
    p.n = w->n;
    p.row_tiles = (int)(w->n_pad / I8_BM);
    p.nks = (int)(w->k_pad / 128);
    p.m = m;
    p.vec = (((uintptr_t)p.c & 15) == 0 && (p.ldc * 4) % 16 == 0) ? 1 : 0;
    p.status = c->status_dev;
    // estimated times in k-steps of a 128 x 256 tile (waves x (k-steps per CTA x relative step cost + a fixed prologue /
    // epilogue worth ~8 steps)): one row tile per CTA, two row tiles per CTA (a third fewer bytes per MAC), CTA pairs
    // (half the bytes per MAC of one tile per CTA; measured 0.82 of the two-tile form on W[11008, 4096] x 2048, 1.06 x 512)
    const auto waves = [&](int ctas) { return (double)((ctas + c->sm_count - 1) / c->sm_count); };
    const int pairs = (p.row_tiles + 1) / 2;
    const double t1 = waves(mtiles * p.row_tiles) * (p.nks + 8.0), t2 = waves(mtiles * pairs) * (2.0 * p.nks * 0.75 + 8.0);
    const int half_sms = c->sm_count / 2 > 0 ? c->sm_count / 2 : 1;
    const double tp = (double)((mtiles * pairs + half_sms - 1) / half_sms) * (p.nks * 0.6 + 8.0);
    if (m > 128 && (c->gemm_i8_pair == 2 || (c->gemm_i8_pair == 1 && tp < 0.9 * (t1 < t2 ? t1 : t2)))) {
        const void *fn = (const void *)gemm_i8_pair_kernel<EPI>;
        static int pairs_resident[64] = {};  // per device: CTA pairs resident at once (0 = not yet asked)
        const int dev_slot = c->device & 63;
        if (!pairs_resident[dev_slot]) {
            GK_CUDA(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)I8P_SMEM));
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)c->sm_count & ~1u);
            cfg.blockDim = dim3((unsigned)I8P_THREADS);
            cfg.dynamicSmemBytes = I8P_SMEM;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = 2;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int nclusters = 0;
            if (cudaOccupancyMaxActiveClusters(&nclusters, fn, &cfg) != cudaSuccess || nclusters < 1) {
                (void)cudaGetLastError();
                nclusters = c->sm_count / 2;
            }
            pairs_resident[dev_slot] = nclusters < c->sm_count / 2 ? nclusters : c->sm_count / 2;
        }
        const int ntiles = pairs * mtiles;
        const int npairs = ntiles < pairs_resident[dev_slot] ? ntiles : pairs_resident[dev_slot];
        GK_CUDA(c, launch_after(gemm_i8_pair_kernel<EPI>, true, dim3(2u * (unsigned)npairs), I8P_THREADS, I8P_SMEM, s, p, mtiles, i8_act_tiles(m)));
        return GLLMK_STATUS_OK;
    }
    if (ntok > 128 && t2 < t1) return i8_launch_mt<2, EPI>(c, p, dim3((unsigned)pairs, (unsigned)mtiles), ntok, s);
    return i8_launch_mt<1, EPI>(c, p, dim3((unsigned)p.row_tiles, (unsigned)mtiles), ntok, s);
}

int32_t gemm_i8_launch(Ctx *c, const Weight *w, const uint8_t *a, int64_t lda, int m, int32_t *out, int64_t ldc, cudaStream_t s) {
    const int nks = (int)(w->k_pad / 128), atiles = i8_act_tiles(m);
    int32_t rc = ensure_act(c, (size_t)atiles * nks * I8_TILE);
    if (rc) return rc;
    stage_act_u8_kernel<<<dim3((unsigned)nks, (unsigned)atiles), 256, 0, s>>>(a, lda, m, w->k, static_cast<uint8_t *>(c->act));
    GK_CUDA(c, cudaGetLastError());
    I8Params p{};
    p.c = out;
    p.ldc = ldc;
    return i8_product<false>(c, w, p, m, s);
}

// A whole linear layer: per-tensor quantization of x into the GEMM's tile images, the product, the f32 epilogue on the
// accumulator.  Three launches, x read twice, y written once.
int32_t w8a8_linear_launch(Ctx *c, const Weight *w, const float *x, int64_t ldx, int m, float *y, int64_t ldy, float scale_b, const float *bias,
                           int act, cudaStream_t s) {
    int32_t rc = ensure_act(c, (size_t)i8_act_tiles(m) * (size_t)(w->k_pad / 128) * I8_TILE);
    if (rc) return rc;
    float *scale = &amax_out(c)->scale;
    rc = act_quant(c, x, m, w->k, ldx, static_cast<uint8_t *>(c->act), 0, 128, true, scale, s);
    if (rc) return rc;
    I8Params p{};
    p.c = y;
    p.ldc = ldy;
    p.scale_a = scale;
    p.colsum = static_cast<const int32_t *>(w->aux);
    p.bias = bias;
    p.scale_b = scale_b;
    p.act = act;
    return i8_product<true>(c, w, p, m, s);
}

int32_t dequant_i32_launch(Ctx *c, const int32_t *ci, float *out, int64_t m, int64_t n, float scale_a, float scale_b, const float *bias,
                           int act, cudaStream_t s) {
    const size_t total = (size_t)m * (size_t)n;
    if (total == 0) return GLLMK_STATUS_OK;
    dequant_i32_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(ci, out, n, scale_a, scale_b, bias, act, total);
    GK_CUDA(c, cudaGetLastError());
    return GLLMK_STATUS_OK;
}

}  // namespace gllmk
