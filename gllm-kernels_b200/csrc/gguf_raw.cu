// The other GGUF block formats of the reference's CPU quant path — Q6_K, Q5_K, Q8_K (256 elements per block) and
// Q4_0, Q5_0 (32 elements per block) — kept on the device as the reference stores them, row after row of blocks
// (Q6_K blocks, 210 bytes, sit in 224-byte slots so that every block starts on a 16-byte boundary).
//
// Decode: one rule per format (an "item" = the elements one data byte, or byte group, yields) with the reference's
// operation order (separately rounded products, no fused multiply-add): matrix decode, embedding gather and the
// host drop-ins are bit-exact.
//
// GEMV: gemv_raw.cu, except Q4_0 / Q5_0 rows that are not whole groups of 256 elements.  Those rows start on any even address
// and take the kernel below: a warp owns two weight rows, streams them through two shared-memory stages with cp.async and
// accumulates integer dot products (dp2a) against s16 fixed-point activations (16 bits per 32-element group, error ~1.5e-5
// of the group maximum).
//
// Reference: src/macros/quant_primitive/k_quant.rs:92-101 (Q8_K), :381-436 (Q5_K), :441-472 (Q6_K);
//            src/macros/quant_primitive/classic.rs:15-29 (Q4_0), :484-504 (Q5_0); block structs src/quant.rs:132-157, 254-275.
#include "common.cuh"

namespace gllmk {

namespace {

__device__ __forceinline__ float f16_at(const uint8_t *p) {
    return __half2float(__ushort_as_half((unsigned short)(p[0] | (p[1] << 8))));
}

// get_scale_min_k4 of the K-quants (k_quant.rs:388-397): sub-block j's 6-bit scale and min
__device__ __forceinline__ void scale_min_k4(int j, const uint8_t *s, float &sc, float &m) {
    if (j < 4) {
        sc = (float)(s[j] & 63);
        m = (float)(s[j + 4] & 63);
    } else {
        sc = (float)((s[j + 4] & 0xF) | ((s[j - 4] >> 6) << 4));
        m = (float)((s[j + 4] >> 4) | ((s[j] >> 6) << 4));
    }
}

// Per format: BS elements and BB bytes per block, ITEMS work items per block, EPI elements per item.
// item(b, it, v, e): decodes item `it` of the block at b into values v[] of elements e[] (indices in the block).
template <int QT>
struct Fmt;

template <>
struct Fmt<GLLMK_QUANT_Q6_K> {  // ql[128] @0, qh[64] @128, scales[16] i8 @192, d f16 @208
    static constexpr int BS = FD_Q6K.block_size, BB = FD_Q6K.block_bytes, DB = 224, ITEMS = 64, EPI = 4;  // DB: bytes per block slot on the device
    static __device__ __forceinline__ void item(const uint8_t *b, int it, float *v, int *e) {
        const int g = it >> 5, l = it & 31, is = l >> 4;
        const uint8_t la = b[FD_Q6K.data_offset + g * 64 + l], lb = b[FD_Q6K.data_offset + g * 64 + l + 32], h = b[FD_Q6K.data_high_offset + g * 32 + l];
        const int8_t *sc = reinterpret_cast<const int8_t *>(b + FD_Q6K.sub_scales_offset + g * 8);
        const float d = f16_at(b + FD_Q6K.scale_offset);
        const int q1 = (int)((la & 0xF) | (((h >> 0) & 3) << 4)) - FD_Q6K.static_bias;
        const int q2 = (int)((lb & 0xF) | (((h >> 2) & 3) << 4)) - FD_Q6K.static_bias;
        const int q3 = (int)((la >> 4) | (((h >> 4) & 3) << 4)) - FD_Q6K.static_bias;
        const int q4 = (int)((lb >> 4) | (((h >> 6) & 3) << 4)) - FD_Q6K.static_bias;
        v[0] = __fmul_rn(__fmul_rn(d, (float)sc[is]), (float)q1);
        v[1] = __fmul_rn(__fmul_rn(d, (float)sc[is + 2]), (float)q2);
        v[2] = __fmul_rn(__fmul_rn(d, (float)sc[is + 4]), (float)q3);
        v[3] = __fmul_rn(__fmul_rn(d, (float)sc[is + 6]), (float)q4);
        e[0] = g * 128 + l;
        e[1] = e[0] + 32;
        e[2] = e[0] + 64;
        e[3] = e[0] + 96;
    }
};

template <>
struct Fmt<GLLMK_QUANT_Q5_K> {  // d @0, dmin @2, scales[12] @4, qh[32] @16, qs[128] @48
    static constexpr int BS = FD_Q5K.block_size, BB = FD_Q5K.block_bytes, DB = 176, ITEMS = 128, EPI = 2;
    static __device__ __forceinline__ void item(const uint8_t *b, int it, float *v, int *e) {
        const int g = it >> 5, l = it & 31;
        const float d = f16_at(b + FD_Q5K.scale_offset), mn = f16_at(b + FD_Q5K.scale_min_offset);
        float sc1, m1, sc2, m2;
        scale_min_k4(2 * g, b + FD_Q5K.sub_scales_offset, sc1, m1);
        scale_min_k4(2 * g + 1, b + FD_Q5K.sub_scales_offset, sc2, m2);
        const uint8_t q = b[FD_Q5K.data_offset + g * 32 + l], h = b[FD_Q5K.data_high_offset + l];
        const int v1 = (q & 0xF) + (((h >> (2 * g)) & 1) ? 16 : 0);
        const int v2 = (q >> 4) + (((h >> (2 * g + 1)) & 1) ? 16 : 0);
        v[0] = __fsub_rn(__fmul_rn(__fmul_rn(d, sc1), (float)v1), __fmul_rn(mn, m1));
        v[1] = __fsub_rn(__fmul_rn(__fmul_rn(d, sc2), (float)v2), __fmul_rn(mn, m2));
        e[0] = g * 64 + l;
        e[1] = e[0] + 32;
    }
};

template <>
struct Fmt<GLLMK_QUANT_Q8_K> {  // d f32 @0, qs[256] i8 @4, bsums[16] i16 @260 (not used by decode)
    static constexpr int BS = FD_Q8K.block_size, BB = FD_Q8K.block_bytes, DB = 292, ITEMS = 64, EPI = 4;
    static __device__ __forceinline__ void item(const uint8_t *b, int it, float *v, int *e) {
        const float d = __uint_as_float((uint32_t)b[0] | ((uint32_t)b[1] << 8) | ((uint32_t)b[2] << 16) | ((uint32_t)b[3] << 24));
#pragma unroll
        for (int j = 0; j < 4; j++) {
            // lanes take neighbouring bytes: element it + 64 j
            e[j] = it + 64 * j;
            v[j] = __fmul_rn(d, (float)(int8_t)b[FD_Q8K.data_offset + e[j]]);
        }
    }
};

template <>
struct Fmt<GLLMK_QUANT_Q4_0> {  // d @0, qs[16] @2: byte j -> elements j (low nibble) and j + 16 (high nibble)
    static constexpr int BS = FD_Q4_0.block_size, BB = FD_Q4_0.block_bytes, DB = 18, ITEMS = 16, EPI = 2;
    static __device__ __forceinline__ void item(const uint8_t *b, int it, float *v, int *e) {
        const float d = f16_at(b);
        const uint8_t q = b[FD_Q4_0.data_offset + it];
        v[0] = __fmul_rn(d, __fsub_rn((float)(q & 0xF), (float)FD_Q4_0.static_bias));
        v[1] = __fmul_rn(d, __fsub_rn((float)(q >> 4), (float)FD_Q4_0.static_bias));
        e[0] = it;
        e[1] = it + 16;
    }
};

template <>
struct Fmt<GLLMK_QUANT_Q5_0> {  // d @0, qh[4] @2 (bit j = fifth bit of element j), qs[16] @6
    static constexpr int BS = FD_Q5_0.block_size, BB = FD_Q5_0.block_bytes, DB = 22, ITEMS = 16, EPI = 2;
    static __device__ __forceinline__ void item(const uint8_t *b, int it, float *v, int *e) {
        const float d = f16_at(b);
        const uint32_t qh = (uint32_t)b[2] | ((uint32_t)b[3] << 8) | ((uint32_t)b[4] << 16) | ((uint32_t)b[5] << 24);
        const uint8_t q = b[FD_Q5_0.data_offset + it];
        const uint32_t lo = (q & 0xF) | (((qh >> it) & 1u) << 4), hi = (q >> 4) | (((qh >> (it + 16)) & 1u) << 4);
        v[0] = __fmul_rn(d, __fsub_rn((float)lo, (float)FD_Q5_0.static_bias));
        v[1] = __fmul_rn(d, __fsub_rn((float)hi, (float)FD_Q5_0.static_bias));
        e[0] = it;
        e[1] = it + 16;
    }
};

// ---- matrix decode / embedding gather: out[r, :] = decode(row ids ? ids[r] : r); rows outside [0, n) -> zeros ----
template <int QT>
__global__ void __launch_bounds__(256) raw_dequant_kernel(const uint8_t *__restrict__ w, int64_t n, int64_t nb,
                                                          const int32_t *__restrict__ ids, float *__restrict__ out,
                                                          size_t total, int stride) {
    using F = Fmt<QT>;
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;  // (out row, block, item)
    if (idx >= total) return;
    const int it = (int)(idx % F::ITEMS);
    const size_t rb = idx / F::ITEMS;
    const int64_t blk = (int64_t)(rb % (size_t)nb), orow = (int64_t)(rb / (size_t)nb);
    float *o = out + ((size_t)orow * nb + blk) * F::BS;
    float v[F::EPI];
    int e[F::EPI];
    int64_t row = orow;
    if (ids) row = ids[orow];
    if (row < 0 || row >= n) {
        F::item(w, it, v, e);  // element indices only (block 0 of the matrix always exists)
#pragma unroll
        for (int j = 0; j < F::EPI; j++) o[e[j]] = 0.0f;
        return;
    }
    F::item(w + ((size_t)row * nb + blk) * (size_t)stride, it, v, e);
#pragma unroll
    for (int j = 0; j < F::EPI; j++) o[e[j]] = v[j];
}

// ---- streaming GEMV on integer dot products ------------------------------------------------------
// The activations are quantized once per call to s16 with one f32 scale per 32 elements (act_quant_kernel); a weight
// "unit" is a few 32-bit words of four s8 weight values each, assembled from the block's bit fields with word-wide
// logic, with the block's f32 factor.  Two dp2a (s16 x s8) per word and token, then acc += x_scale * w_scale * dot.
constexpr int RG_WARPS = 8;
constexpr int RG_CHUNK = 2048;  // block bytes staged per warp and pass (two stages of this size per warp)

// x [m tokens, k] (any strides) -> xq s16 [m, k] and xs f32 [m, k / 32] with x ~= xs * xq: 16-bit fixed point per
// 32-element group (relative error ~1.5e-5 of the group's largest value).  One warp per 32 elements.
__global__ void __launch_bounds__(256) act_quant_kernel(const float *__restrict__ x, int64_t xst, int64_t xsk, int m, int64_t k,
                                                        int16_t *__restrict__ xq, float *__restrict__ xs) {
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int64_t per_tok = k >> 5;
    if (warp >= per_tok * m) return;
    const int64_t t = warp / per_tok, b = warp % per_tok;
    const float v = x[(size_t)t * xst + (size_t)(b * 32 + lane) * xsk];
    float a = fabsf(v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
    const float sc = a * (1.0f / 32767.0f);
    const float q = a > 0.0f ? fminf(fmaxf(rintf(v / sc), -32767.0f), 32767.0f) : 0.0f;
    xq[(size_t)t * k + b * 32 + lane] = (int16_t)(int)q;
    if (lane == 0) xs[(size_t)t * per_tok + b] = sc;
}

// f16 field at a 2-byte aligned address
__device__ __forceinline__ float f16_even(const uint8_t *p) {
    return __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(p)));
}
// 16 bytes global -> shared without passing registers (both addresses 16-byte aligned)
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
// 32-bit word at a 2-byte aligned shared-memory address (block sizes and field offsets are all even)
__device__ __forceinline__ uint32_t ld32(const uint8_t *p) {
    const unsigned short *h = reinterpret_cast<const unsigned short *>(p);
    return (uint32_t)h[0] | ((uint32_t)h[1] << 16);
}
// bits 0..3 of v -> bit 0 of bytes 0..3
__device__ __forceinline__ uint32_t spread4(uint32_t v) { return ((v & 0xFu) * 0x00204081u) & 0x01010101u; }

// Per format: UNITS per block, NW words per unit (NW / 2 pairs).
// unit(b, u, q, ko, ws): words q[] (four values each, as s8); words 2i and 2i + 1 are neighbours in k: pair i starts at
// element ko[i] of the block (a multiple of 8) and has the weight factor ws[i].
template <int QT>
struct Dp;

template <>
struct Dp<GLLMK_QUANT_Q4_0> {
    static constexpr int UNITS = 2, NW = 4;
    static __device__ __forceinline__ void unit(const uint8_t *b, int u, uint32_t *q, int *ko, float *ws) {
        const uint32_t W0 = ld32(b + FD_Q4_0.data_offset + 8 * u), W1 = ld32(b + FD_Q4_0.data_offset + 4 + 8 * u);
        // a nibble with bit 3 flipped is q - 8 in 4-bit two's complement; in the high half of a byte it is the s8 16 (q - 8)
        q[0] = ((W0 ^ 0x08080808u) << 4) & 0xF0F0F0F0u;
        q[1] = ((W1 ^ 0x08080808u) << 4) & 0xF0F0F0F0u;
        q[2] = (W0 ^ 0x80808080u) & 0xF0F0F0F0u;
        q[3] = (W1 ^ 0x80808080u) & 0xF0F0F0F0u;
        ko[0] = 8 * u;
        ko[1] = 16 + 8 * u;
        ws[0] = ws[1] = 0.0625f * f16_even(b + FD_Q4_0.scale_offset);
    }
};

template <>
struct Dp<GLLMK_QUANT_Q5_0> {
    static constexpr int UNITS = 2, NW = 4;
    static __device__ __forceinline__ void unit(const uint8_t *b, int u, uint32_t *q, int *ko, float *ws) {
        const uint32_t W0 = ld32(b + FD_Q5_0.data_offset + 8 * u), W1 = ld32(b + FD_Q5_0.data_offset + 4 + 8 * u),
                       qh = ld32(b + FD_Q5_0.data_high_offset);
        // a 5-bit value with bit 4 flipped is q - 16 in 5-bit two's complement; three places up it is the s8 8 (q - 16)
        q[0] = ((((W0 & 0x0F0F0F0Fu) | (spread4(qh >> (8 * u)) << 4)) ^ 0x10101010u) << 3) & 0xF8F8F8F8u;
        q[1] = ((((W1 & 0x0F0F0F0Fu) | (spread4(qh >> (8 * u + 4)) << 4)) ^ 0x10101010u) << 3) & 0xF8F8F8F8u;
        q[2] = (((((W0 >> 4) & 0x0F0F0F0Fu) | (spread4(qh >> (16 + 8 * u)) << 4)) ^ 0x10101010u) << 3) & 0xF8F8F8F8u;
        q[3] = (((((W1 >> 4) & 0x0F0F0F0Fu) | (spread4(qh >> (20 + 8 * u)) << 4)) ^ 0x10101010u) << 3) & 0xF8F8F8F8u;
        ko[0] = 8 * u;
        ko[1] = 16 + 8 * u;
        ws[0] = ws[1] = 0.125f * f16_even(b);
    }
};

struct RawGemvParams {
    const uint8_t *w;
    const int16_t *xq;  // [m, k]
    const float *xs;    // [m, k / 32]
    float *y;
    const float *row_scales;
    int64_t n, nb, k, yst, ysr, n_row_scales;
    int m;
};

constexpr int RG_ROWS = 2;  // rows per warp: their words meet the same activations, loaded once

template <int QT, int MT>
__global__ void __launch_bounds__(RG_WARPS * 32) raw_gemv_kernel(const RawGemvParams p) {
    using F = Fmt<QT>;
    using D = Dp<QT>;
    constexpr int R = RG_ROWS, CH = RG_CHUNK / R;
    constexpr int LPB = D::UNITS < 32 ? 32 / D::UNITS : 1;   // blocks one warp pass over the units covers
    constexpr int CB = (CH / F::DB) / LPB * LPB;             // whole blocks per row and pass, no idle lanes inside a pass
    __shared__ __align__(16) uint8_t buf[RG_WARPS][2][R][CH + 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k32 = (int)(p.k >> 5);
    const int64_t groups = (p.n + R - 1) / R;
    for (int64_t grp = (int64_t)blockIdx.x * RG_WARPS + warp; grp < groups; grp += (int64_t)gridDim.x * RG_WARPS) {
        const uint8_t *rowp[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int64_t row = grp * R + r < p.n ? grp * R + r : p.n - 1;  // a surplus row repeats the last one; not stored
            rowp[r] = p.w + (size_t)row * p.nb * F::DB;
        }
        for (int t0 = 0; t0 < p.m; t0 += MT) {
            float acc[R][MT];
            const int16_t *xq[MT];
            const float *xs[MT];
#pragma unroll
            for (int t = 0; t < MT; t++) {
                const int tok = t0 + t < p.m ? t0 + t : p.m - 1;  // surplus slots repeat the last token; not stored
                xq[t] = p.xq + (size_t)tok * p.k;
                xs[t] = p.xs + (size_t)tok * k32;
#pragma unroll
                for (int r = 0; r < R; r++) acc[r][t] = 0.0f;
            }
            // two shared-memory stages per warp: the copies of pass i + 1 (cp.async, 16 bytes each) run while pass i
            // is computed.  Copies start at the aligned address below the pass: up to 15 bytes before it and after the
            // row are copied and ignored (the weight buffer starts 256-byte aligned and ends with 16 spare bytes).
            const auto issue = [&](int b0, int st) {
                const int nblk = (int)p.nb - b0 < CB ? (int)p.nb - b0 : CB;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const uint8_t *src = rowp[r] + (size_t)b0 * F::DB;
                    const uintptr_t a0 = reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)15;
                    const int n16 = ((int)(reinterpret_cast<uintptr_t>(src) - a0) + nblk * F::DB + 15) >> 4;
                    for (int i = lane; i < n16; i += 32) cp_async16(buf[warp][st][r] + 16 * i, reinterpret_cast<const uint8_t *>(a0) + 16 * i);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            __syncwarp();
            issue(0, 0);
            int st = 0;
            for (int b0 = 0; b0 < (int)p.nb; b0 += CB, st ^= 1) {
                const int nblk = (int)p.nb - b0 < CB ? (int)p.nb - b0 : CB;
                if (b0 + CB < (int)p.nb) {
                    issue(b0 + CB, st ^ 1);
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                } else {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                }
                __syncwarp();
                const uint8_t *sb[R];
#pragma unroll
                for (int r = 0; r < R; r++)
                    sb[r] = buf[warp][st][r] + (int)(reinterpret_cast<uintptr_t>(rowp[r] + (size_t)b0 * F::DB) & 15);
                for (int u = lane; u < nblk * D::UNITS; u += 32) {
                    const int blk = u / D::UNITS;
                    uint32_t q[R][D::NW];
                    int ko[D::NW / 2];
                    float ws[R][D::NW / 2];
#pragma unroll
                    for (int r = 0; r < R; r++) D::unit(sb[r] + blk * F::DB, u % D::UNITS, q[r], ko, ws[r]);
                    const int kb = (b0 + blk) * F::BS;
#pragma unroll
                    for (int j = 0; j < D::NW / 2; j++) {
                        const int kk = kb + ko[j];
#pragma unroll
                        for (int t = 0; t < MT; t++) {
                            const int4 xw = __ldg(reinterpret_cast<const int4 *>(xq[t] + kk));  // eight s16 activations
                            const float s = __ldg(xs[t] + (kk >> 5));
#pragma unroll
                            for (int r = 0; r < R; r++) {
                                // s16 x s8 products: a word's elements 0, 1 against one register, 2, 3 against the next
                                const int q0 = (int)q[r][2 * j], q1 = (int)q[r][2 * j + 1];
                                const float dot =
                                    (float)__dp2a_hi(xw.w, q1, __dp2a_lo(xw.z, q1, __dp2a_hi(xw.y, q0, __dp2a_lo(xw.x, q0, 0))));
                                acc[r][t] = fmaf(s * ws[r][j], dot, acc[r][t]);
                            }
                        }
                    }
                }
                __syncwarp();  // every lane is done with this stage before the next pass's copies overwrite it
            }
#pragma unroll
            for (int r = 0; r < R; r++)
#pragma unroll
                for (int t = 0; t < MT; t++) {
                    float a = acc[r][t];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                    const int64_t row = grp * R + r;
                    if (lane == 0 && t0 + t < p.m && row < p.n) {
                        if (p.n_row_scales == 1) a *= p.row_scales[0];
                        else if (p.n_row_scales > 1) a *= p.row_scales[row];
                        p.y[(size_t)(t0 + t) * p.yst + (size_t)row * p.ysr] = a;
                    }
                }
        }
    }
}

// Q6_K: reference blocks (210 bytes) <-> device slots (224 bytes); one thread per 2 bytes
__global__ void q6k_pad_kernel(const unsigned short *__restrict__ src, unsigned short *__restrict__ dst, size_t total, int to_device) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const size_t blk = idx / 105, o = idx % 105;
    if (to_device) dst[blk * 112 + o] = src[blk * 105 + o];
    else dst[blk * 105 + o] = src[blk * 112 + o];
}

inline unsigned grid_1d(size_t total, int block) { return (unsigned)((total + block - 1) / block); }

template <int QT>
int32_t dequant_t(Ctx *c, const uint8_t *w, int64_t n, int64_t nb, const int32_t *ids, size_t rows, float *out, cudaStream_t s,
                  bool dev_layout) {
    const size_t total = rows * (size_t)nb * Fmt<QT>::ITEMS;
    if (total == 0) return GLLMK_STATUS_OK;
    if (total > (size_t)0x7fffffff * 256) return fail(c, GLLMK_STATUS_INVALID_ARG, "decode: matrix too large for one launch");
    raw_dequant_kernel<QT><<<grid_1d(total, 256), 256, 0, s>>>(w, n, nb, ids, out, total, dev_layout ? Fmt<QT>::DB : Fmt<QT>::BB);
    GK_CUDA(c, cudaGetLastError());
    return GLLMK_STATUS_OK;
}

template <int QT>
int32_t gemv_t(Ctx *c, const RawGemvParams &p, cudaStream_t s) {
    // 16 rows per CTA and pass; enough CTAs to fill every SM several times over, never more than the rows need
    int64_t ctas = (p.n + RG_WARPS * RG_ROWS - 1) / (RG_WARPS * RG_ROWS);
    const int64_t cap = (int64_t)c->sm_count * 6;
    if (ctas > cap) ctas = cap;
    if (p.m == 1) raw_gemv_kernel<QT, 1><<<(unsigned)ctas, RG_WARPS * 32, 0, s>>>(p);
    else if (p.m <= 4) raw_gemv_kernel<QT, 4><<<(unsigned)ctas, RG_WARPS * 32, 0, s>>>(p);
    else raw_gemv_kernel<QT, 8><<<(unsigned)ctas, RG_WARPS * 32, 0, s>>>(p);
    GK_CUDA(c, cudaGetLastError());
    return GLLMK_STATUS_OK;
}

}  // namespace

bool raw_format(int32_t qt) {
    return qt == GLLMK_QUANT_Q6_K || qt == GLLMK_QUANT_Q5_K || qt == GLLMK_QUANT_Q8_K || qt == GLLMK_QUANT_Q4_0 ||
           qt == GLLMK_QUANT_Q5_0;
}

int raw_dev_block_bytes(int32_t qt) {
    switch (qt) {
        case GLLMK_QUANT_Q6_K: return Fmt<GLLMK_QUANT_Q6_K>::DB;
        case GLLMK_QUANT_Q5_K: return Fmt<GLLMK_QUANT_Q5_K>::DB;
        case GLLMK_QUANT_Q8_K: return Fmt<GLLMK_QUANT_Q8_K>::DB;
        case GLLMK_QUANT_Q4_0: return Fmt<GLLMK_QUANT_Q4_0>::DB;
        case GLLMK_QUANT_Q5_0: return Fmt<GLLMK_QUANT_Q5_0>::DB;
    }
    return 0;
}

// reference-layout blocks (device memory) -> the weight's device buffer, and back
int32_t raw_fill(Ctx *c, const Weight *w, const void *blocks, cudaStream_t s) {
    GK_CUDA(c, cudaMemsetAsync(w->qs, 0, w->qs_bytes, s));
    if (w->qt == GLLMK_QUANT_Q6_K) {
        const size_t total = (size_t)w->n * w->nb * 105;
        q6k_pad_kernel<<<grid_1d(total, 256), 256, 0, s>>>(static_cast<const unsigned short *>(blocks),
                                                           static_cast<unsigned short *>(w->qs), total, 1);
        GK_CUDA(c, cudaGetLastError());
    } else {
        GK_CUDA(c, cudaMemcpyAsync(w->qs, blocks, w->ref_bytes, cudaMemcpyDeviceToDevice, s));
    }
    return GLLMK_STATUS_OK;
}
int32_t raw_unfill(Ctx *c, const Weight *w, void *blocks, cudaStream_t s) {
    if (w->qt == GLLMK_QUANT_Q6_K) {
        const size_t total = (size_t)w->n * w->nb * 105;
        q6k_pad_kernel<<<grid_1d(total, 256), 256, 0, s>>>(static_cast<const unsigned short *>(w->qs),
                                                           static_cast<unsigned short *>(blocks), total, 0);
        GK_CUDA(c, cudaGetLastError());
    } else {
        GK_CUDA(c, cudaMemcpyAsync(blocks, w->qs, w->ref_bytes, cudaMemcpyDeviceToDevice, s));
    }
    return GLLMK_STATUS_OK;
}

// dev_layout: blocks at the device stride (a weight's buffer); otherwise consecutive reference blocks
int32_t raw_dequant(Ctx *c, int32_t qt, const uint8_t *w, int64_t n, int64_t nb, const int32_t *ids, size_t rows, float *out,
                    cudaStream_t s, bool dev_layout) {
    switch (qt) {
        case GLLMK_QUANT_Q6_K: return dequant_t<GLLMK_QUANT_Q6_K>(c, w, n, nb, ids, rows, out, s, dev_layout);
        case GLLMK_QUANT_Q5_K: return dequant_t<GLLMK_QUANT_Q5_K>(c, w, n, nb, ids, rows, out, s, dev_layout);
        case GLLMK_QUANT_Q8_K: return dequant_t<GLLMK_QUANT_Q8_K>(c, w, n, nb, ids, rows, out, s, dev_layout);
        case GLLMK_QUANT_Q4_0: return dequant_t<GLLMK_QUANT_Q4_0>(c, w, n, nb, ids, rows, out, s, dev_layout);
        case GLLMK_QUANT_Q5_0: return dequant_t<GLLMK_QUANT_Q5_0>(c, w, n, nb, ids, rows, out, s, dev_layout);
    }
    return fail(c, GLLMK_STATUS_UNSUPPORTED, "decode: quant type %d", qt);
}

int32_t raw_gemv_launch(Ctx *c, const Weight *w, const float *x, int64_t xst, int64_t xsk, int m, float *y, int64_t yst,
                        int64_t ysr, const float *row_scales, int64_t n_row_scales, cudaStream_t s) {
    if (raw_mma_takes(c, w)) return raw_mma_launch(c, w, x, xst, xsk, m, y, yst, ysr, row_scales, n_row_scales, s);
    // activations -> s16 + one f32 scale per 32 elements, in the context's activation scratch
    const size_t qb = (2 * (size_t)m * w->k + 255) & ~(size_t)255;
    int32_t rc = ensure_act(c, qb + (size_t)m * (w->k / 32) * sizeof(float));
    if (rc) return rc;
    int16_t *xq = static_cast<int16_t *>(c->act);
    float *xs = reinterpret_cast<float *>(static_cast<char *>(c->act) + qb);
    const size_t qthreads = (size_t)m * (w->k / 32) * 32;
    act_quant_kernel<<<grid_1d(qthreads, 256), 256, 0, s>>>(x, xst, xsk, m, w->k, xq, xs);
    GK_CUDA(c, cudaGetLastError());
    RawGemvParams p{};
    p.w = static_cast<const uint8_t *>(w->qs);
    p.xq = xq;
    p.xs = xs;
    p.k = w->k;
    p.y = y;
    p.row_scales = row_scales;
    p.n_row_scales = row_scales ? n_row_scales : 0;
    p.n = w->n;
    p.nb = w->nb;
    p.yst = yst;
    p.ysr = ysr;
    p.m = m;
    if (w->qt == GLLMK_QUANT_Q4_0) return gemv_t<GLLMK_QUANT_Q4_0>(c, p, s);
    if (w->qt == GLLMK_QUANT_Q5_0) return gemv_t<GLLMK_QUANT_Q5_0>(c, p, s);
    return fail(c, GLLMK_STATUS_UNSUPPORTED, "gemv: quant type %d", w->qt);
}

}  // namespace gllmk
