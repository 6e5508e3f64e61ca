// Mixture-of-experts plumbing around the grouped expert GEMM, with the reference's data conventions
// (scalar-ops/src/moe.rs:59-157): the top-k selection writes expert indices as u32 bit patterns stored in f32
// slots followed by the renormalised weights; the recombination adds weight * expert row in k order.
// Between the two, the (token, k) slots are grouped per expert (what gllmk_gemm_grouped takes) and the
// activation rows gathered in that order.
#include <cuda_bf16.h>

#include "common.cuh"

namespace gllmk {

constexpr int MOE_MAX_TOPK = 16;
constexpr int MOE_MAX_EXPERTS = 1024;

// scalar_topk, one thread per token: insertion of each expert's probability into a descending list with a
// strict '>' (the earlier expert wins a tie, NaN never enters), then weights = value * (1 / sum) (0 if sum <= 0).
// Bound by latency (a few thousand probabilities in all): the list lives in registers (K slots, unrolled; the compiler kept a
// list of run-time length in local memory) and eight probabilities are loaded before they are looked at.
template <int K>
__global__ void __launch_bounds__(32) moe_topk_kernel(const float *__restrict__ probs, float *__restrict__ out, int64_t seq, int ne, int top_k) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= seq) return;
    uint32_t ti[K];
    float tv[K];
#pragma unroll
    for (int i = 0; i < K; i++) { ti[i] = 0u; tv[i] = __int_as_float(0xFF800000); }
    const float *row = probs + s * ne;
    for (int e0 = 0; e0 < ne; e0 += 8) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = e0 + j < ne ? __ldg(row + e0 + j) : __int_as_float(0x7FC00000);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            float cv = v[j];
            uint32_t ci = (uint32_t)(e0 + j);
            bool in = false;  // from the first slot it beats on, every slot moves down by one
#pragma unroll
            for (int i = 0; i < K; i++) {
                in = in || cv > tv[i];
                if (in) {
                    const float pv = tv[i];
                    const uint32_t pi = ti[i];
                    tv[i] = cv; ti[i] = ci;
                    cv = pv; ci = pi;
                }
            }
        }
    }
    float sum = 0.0f;
#pragma unroll
    for (int ki = 0; ki < K; ki++)
        if (ki < top_k) sum = __fadd_rn(sum, tv[ki]);
    const float inv = sum > 0.0f ? __fdiv_rn(1.0f, sum) : 0.0f;
#pragma unroll
    for (int ki = 0; ki < K; ki++)
        if (ki < top_k) {
            out[s * top_k + ki] = __uint_as_float(ti[ki]);
            out[seq * top_k + s * top_k + ki] = __fmul_rn(tv[ki], inv);
        }
}

// Grouping of the slots per expert, stable: the g-th slot of expert e (in slot order) becomes row offs[e] + g:
// perm[row] = slot, inv[slot] = row.  Slots whose index is >= ne belong to no expert (the reference skips them,
// scalar-ops/src/moe_dispatch_packed.rs:113-116): inv[slot] = -1.
// One block: each of its 32 warps counts a contiguous run of slots per expert (match_any: 32 slots per step), the counts are
// scanned over warps and experts in shared memory, and the warps walk their runs again and place them.  The offsets go to
// page-locked host memory.  A serial chain of slots / 1024 steps, twice, in one launch: 1024 slots 7 us (a warp per expert
// that walked all slots, a launch for the counts, a copy to the host and back and a launch to place: 22 us and two waits).
constexpr int MOE_ROUTE_THREADS = 1024;
__global__ void __launch_bounds__(MOE_ROUTE_THREADS) moe_route_kernel(const float *__restrict__ idx, int64_t slots, int ne, int *host_offs,
                                                                      int *__restrict__ perm, int *__restrict__ inv) {
    extern __shared__ int cnt[];  // [32 warps][ne]
    __shared__ int wsum[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < 32 * ne; i += MOE_ROUTE_THREADS) cnt[i] = 0;
    __syncthreads();
    const int64_t run = ((slots + 31) / 32 + 31) / 32 * 32, lo = warp * run, hi = lo + run < slots ? lo + run : slots;
    int *mine = cnt + warp * ne;
    const auto walk = [&](auto &&f) {  // f(slot, expert or 0xFFFFFFFF, lanes with the same expert)
        for (int64_t s0 = lo; s0 < hi; s0 += 128) {
            uint32_t id[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int64_t s = s0 + 32 * j + lane;
                id[j] = s < hi ? __float_as_uint(__ldg(idx + s)) : 0xFFFFFFFFu;
                if (id[j] >= (uint32_t)ne) id[j] = 0xFFFFFFFFu;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                f(s0 + 32 * j + lane, id[j], __match_any_sync(0xffffffffu, id[j]));
                __syncwarp();
            }
        }
    };
    walk([&](int64_t, uint32_t id, uint32_t same) {
        if (id != 0xFFFFFFFFu && lane == __ffs((int)same) - 1) mine[id] += __popc(same);
    });
    __syncthreads();
    // thread = expert: exclusive scan over the warps' runs, then over the experts
    const int e = threadIdx.x;
    int total = 0;
    if (e < ne)
        for (int w = 0; w < 32; w++) {
            const int c = cnt[w * ne + e];
            cnt[w * ne + e] = total;
            total += c;
        }
    int scan = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, scan, o);
        if (lane >= o) scan += v;
    }
    if (lane == 31) wsum[warp] = scan;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; w++) before += wsum[w];
    const int first = before + scan - total;
    if (e < ne) {
        for (int w = 0; w < 32; w++) cnt[w * ne + e] += first;
        reinterpret_cast<volatile int *>(host_offs)[e] = first;
        if (e == ne - 1) reinterpret_cast<volatile int *>(host_offs)[ne] = first + total;
    }
    __syncthreads();
    walk([&](int64_t s, uint32_t id, uint32_t same) {
        if (id != 0xFFFFFFFFu) {
            const int row = mine[id] + __popc(same & ((1u << lane) - 1u));
            perm[row] = (int)s;
            inv[s] = row;
        } else if (s < hi) {
            inv[s] = -1;
        }
        __syncwarp();
        if (id != 0xFFFFFFFFu && lane == __ffs((int)same) - 1) mine[id] += __popc(same);
    });
}

// Rows in grouped order, V = the widest unit (16, 4 or 2 bytes) that the addresses and the row length allow; n units per row.
// Bound by memory; 1024 rows of 8 KB with 2-byte units 8.6 us, with 16-byte units 4.5 us.
template <typename V>
__global__ void __launch_bounds__(256) moe_gather_kernel(const V *__restrict__ x, int64_t ldx, const int *__restrict__ perm, int top_k, int64_t n,
                                                         V *__restrict__ out, int64_t ldo) {
    const int64_t g = blockIdx.x;
    const V *src = x + (int64_t)(perm[g] / top_k) * ldx;
    V *dst = out + g * ldo;
#pragma unroll 4
    for (int64_t c = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.y * blockDim.x) dst[c] = __ldg(src + c);
}

// scalar_weighted_sum: out[s, d] = ((0 + w_0 * r_0[d]) + w_1 * r_1[d]) + ... with a separate multiply and add per
// term.  inv == nullptr: expert_outputs is the reference's [expert][seq][hidden] buffer; else it holds the grouped
// rows and inv[s * top_k + ki] names the row (negative: the slot has no expert and adds nothing).
// Bound by reading the rows: thread = two pieces of VEC elements (16-byte loads where everything is aligned), the rows of four
// terms loaded before the first is added.  512 tokens x 2 rows of 14336 (88 MB, 13 us at 6.65 TB/s): 35 us with 4-byte loads, one
// row at a time; 18 us with one piece per thread; 14.2 us.
template <int VEC>
__global__ void __launch_bounds__(256) moe_wsum_kernel(const float *__restrict__ eo, const float *__restrict__ idx, const float *__restrict__ wts,
                                                       const int *__restrict__ inv, float *__restrict__ out, int64_t seq, int64_t hidden,
                                                       int64_t ld, int top_k, int ne) {
    const int64_t s = blockIdx.x;
    constexpr int U = VEC == 4 ? 2 : 1;  // pieces of VEC elements per thread, 256 threads apart
    constexpr int64_t SPAN = 256 * VEC;
    for (int64_t d0 = (int64_t)blockIdx.y * (U * SPAN) + threadIdx.x * VEC; d0 < hidden; d0 += (int64_t)gridDim.y * (U * SPAN)) {
        float acc[U][VEC];
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int i = 0; i < VEC; i++) acc[u][i] = 0.0f;
        for (int k0 = 0; k0 < top_k; k0 += 4) {
            float v[4][U][VEC], w[4];
            bool has[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                has[j] = false;
                const float *row = eo;
                if (k0 + j < top_k) {
                    const int64_t slot = s * top_k + k0 + j;
                    w[j] = __ldg(wts + slot);
                    if (inv) {
                        const int r = __ldg(inv + slot);
                        has[j] = r >= 0;
                        row = eo + (int64_t)r * ld;
                    } else {
                        const uint32_t e = __float_as_uint(__ldg(idx + slot));
                        has[j] = e < (uint32_t)ne;
                        row = eo + ((int64_t)e * seq + s) * ld;
                    }
                }
                if (has[j]) {
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int64_t d = d0 + u * SPAN;
                        if constexpr (VEC == 4) {
                            const float4 t = d < hidden ? __ldg(reinterpret_cast<const float4 *>(row + d)) : make_float4(0.f, 0.f, 0.f, 0.f);
                            v[j][u][0] = t.x; v[j][u][1] = t.y; v[j][u][2] = t.z; v[j][u][3] = t.w;
                        } else {
                            v[j][u][0] = __ldg(row + d);
                        }
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (has[j])
#pragma unroll
                    for (int u = 0; u < U; u++)
#pragma unroll
                        for (int i = 0; i < VEC; i++) acc[u][i] = __fadd_rn(acc[u][i], __fmul_rn(w[j], v[j][u][i]));
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int64_t d = d0 + u * SPAN;
            if (d < hidden) {
                if constexpr (VEC == 4) *reinterpret_cast<float4 *>(out + s * hidden + d) = make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
                else out[s * hidden + d] = acc[u][0];
            }
        }
    }
}

template <typename V>
static void gather_launch(const void *x, int64_t ldx_bytes, const int *perm, int64_t rows, int top_k, int64_t row_bytes, void *out, int64_t ldo_bytes,
                          cudaStream_t s) {
    const int64_t n = row_bytes / (int64_t)sizeof(V);
    // four units per thread, at least two warps
    const int64_t want = (n / 4 + 31) / 32 * 32;
    const int threads = (int)(want < 64 ? 64 : (want > 256 ? 256 : want));
    const int64_t y = (n + 4 * threads - 1) / (4 * threads);
    moe_gather_kernel<V><<<dim3((unsigned)rows, (unsigned)(y > 64 ? 64 : y)), threads, 0, s>>>(static_cast<const V *>(x), ldx_bytes / (int64_t)sizeof(V), perm,
                                                                                             top_k, n, static_cast<V *>(out), ldo_bytes / (int64_t)sizeof(V));
}

}  // namespace gllmk

using namespace gllmk;

extern "C" int32_t gllmk_moe_topk(gllmk_ctx ctx, const float *gate_probs_dev, float *out_dev, int64_t seq_len, int32_t num_experts,
                                  int32_t top_k, void *stream) {
    if (!ctx || !gate_probs_dev || !out_dev) return GLLMK_STATUS_INVALID_ARG;
    Ctx *c = static_cast<Ctx *>(ctx);
    if (seq_len < 0 || num_experts < 1) return fail(c, GLLMK_STATUS_INVALID_ARG, "moe_topk: bad shape");
    if (top_k < 1 || top_k > MOE_MAX_TOPK) return fail(c, GLLMK_STATUS_UNSUPPORTED, "moe_topk: top_k=%d outside 1..%d", top_k, MOE_MAX_TOPK);
    if (seq_len == 0) return GLLMK_STATUS_OK;
    DeviceGuard g(c->device);
    const unsigned grid = (unsigned)((seq_len + 31) / 32);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (top_k <= 2) moe_topk_kernel<2><<<grid, 32, 0, s>>>(gate_probs_dev, out_dev, seq_len, num_experts, top_k);
    else if (top_k <= 4) moe_topk_kernel<4><<<grid, 32, 0, s>>>(gate_probs_dev, out_dev, seq_len, num_experts, top_k);
    else if (top_k <= 8) moe_topk_kernel<8><<<grid, 32, 0, s>>>(gate_probs_dev, out_dev, seq_len, num_experts, top_k);
    else moe_topk_kernel<MOE_MAX_TOPK><<<grid, 32, 0, s>>>(gate_probs_dev, out_dev, seq_len, num_experts, top_k);
    GK_CUDA(c, cudaGetLastError());
    return GLLMK_STATUS_OK;
}

extern "C" int32_t gllmk_moe_route(gllmk_ctx ctx, const float *indices_dev, int64_t seq_len, int32_t num_experts, int32_t top_k,
                                   int64_t *row_offsets_host, int32_t *perm_dev, int32_t *inv_dev, void *stream) {
    if (!ctx || !indices_dev || !row_offsets_host || !perm_dev || !inv_dev) return GLLMK_STATUS_INVALID_ARG;
    Ctx *c = static_cast<Ctx *>(ctx);
    if (num_experts < 1 || num_experts > MOE_MAX_EXPERTS)
        return fail(c, GLLMK_STATUS_UNSUPPORTED, "moe_route: num_experts=%d outside 1..%d", num_experts, MOE_MAX_EXPERTS);
    const int64_t slots = seq_len * (int64_t)top_k;
    if (seq_len < 0 || top_k < 1 || slots > 0x7fffffff) return fail(c, GLLMK_STATUS_INVALID_ARG, "moe_route: bad shape");
    DeviceGuard g(c->device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int32_t rc = ensure_host_word(c);
    if (rc) return rc;
    static bool attr_set[64] = {};  // function attributes are per device
    if (!attr_set[c->device & 63]) {
        GK_CUDA(c, cudaFuncSetAttribute(moe_route_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * MOE_MAX_EXPERTS * (int)sizeof(int)));
        attr_set[c->device & 63] = true;
    }
    int *offs = static_cast<int *>(c->host_word);
    moe_route_kernel<<<1, MOE_ROUTE_THREADS, 32 * (size_t)num_experts * sizeof(int), s>>>(indices_dev, slots, num_experts, offs, perm_dev, inv_dev);
    GK_CUDA(c, cudaGetLastError());
    GK_CUDA(c, cudaStreamSynchronize(s));
    for (int e = 0; e <= num_experts; e++) row_offsets_host[e] = reinterpret_cast<volatile int *>(offs)[e];
    return GLLMK_STATUS_OK;
}

extern "C" int32_t gllmk_moe_gather(gllmk_ctx ctx, const void *x_dev, int32_t dtype, int64_t ldx, const int32_t *perm_dev, int64_t rows,
                                    int32_t top_k, int64_t k, void *out_dev, int64_t ldo, void *stream) {
    if (!ctx || !x_dev || !perm_dev || !out_dev) return GLLMK_STATUS_INVALID_ARG;
    Ctx *c = static_cast<Ctx *>(ctx);
    if (dtype != GLLMK_DTYPE_F32 && dtype != GLLMK_DTYPE_BF16) return fail(c, GLLMK_STATUS_UNSUPPORTED, "moe_gather: dtype");
    if (rows < 0 || rows > 0x7fffffff || top_k < 1 || k < 1 || ldx < k || ldo < k) return fail(c, GLLMK_STATUS_INVALID_ARG, "moe_gather: bad shape");
    if (rows == 0) return GLLMK_STATUS_OK;
    DeviceGuard g(c->device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int64_t es = dtype == GLLMK_DTYPE_F32 ? 4 : 2, lx = ldx * es, lo = ldo * es, nb = k * es;
    const uint64_t all = (uint64_t)(uintptr_t)x_dev | (uint64_t)(uintptr_t)out_dev | (uint64_t)lx | (uint64_t)lo | (uint64_t)nb;
    if (all % 16 == 0) gather_launch<uint4>(x_dev, lx, perm_dev, rows, top_k, nb, out_dev, lo, s);
    else if (all % 4 == 0) gather_launch<uint32_t>(x_dev, lx, perm_dev, rows, top_k, nb, out_dev, lo, s);
    else gather_launch<unsigned short>(x_dev, lx, perm_dev, rows, top_k, nb, out_dev, lo, s);
    GK_CUDA(c, cudaGetLastError());
    return GLLMK_STATUS_OK;
}

extern "C" int32_t gllmk_moe_weighted_sum(gllmk_ctx ctx, const float *expert_outputs_dev, int64_t ld, const float *indices_dev,
                                          const float *weights_dev, const int32_t *inv_dev, float *out_dev, int64_t seq_len,
                                          int64_t hidden, int32_t top_k, int32_t num_experts, void *stream) {
    if (!ctx || !expert_outputs_dev || !indices_dev || !weights_dev || !out_dev) return GLLMK_STATUS_INVALID_ARG;
    Ctx *c = static_cast<Ctx *>(ctx);
    if (seq_len < 0 || seq_len > 0x7fffffff || hidden < 1 || ld < hidden || top_k < 1 || num_experts < 1)
        return fail(c, GLLMK_STATUS_INVALID_ARG, "moe_weighted_sum: bad shape");
    if (seq_len == 0) return GLLMK_STATUS_OK;
    DeviceGuard g(c->device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool vec = hidden % 4 == 0 && ld % 4 == 0 && ((uintptr_t)expert_outputs_dev & 15) == 0 && ((uintptr_t)out_dev & 15) == 0;
    const int64_t per_block = vec ? 2048 : 256, y = (hidden + per_block - 1) / per_block;
    const dim3 grid((unsigned)seq_len, (unsigned)(y > 64 ? 64 : y));
    if (vec) moe_wsum_kernel<4><<<grid, 256, 0, s>>>(expert_outputs_dev, indices_dev, weights_dev, inv_dev, out_dev, seq_len, hidden, ld, top_k, num_experts);
    else moe_wsum_kernel<1><<<grid, 256, 0, s>>>(expert_outputs_dev, indices_dev, weights_dev, inv_dev, out_dev, seq_len, hidden, ld, top_k, num_experts);
    GK_CUDA(c, cudaGetLastError());
    return GLLMK_STATUS_OK;
}
