// Decode path over the row-major GGUF formats (Q6_K, Q5_K, Q8_K; Q4_0 and Q5_0 when a row is whole groups of 256 elements):
// fused dequantize + GEMV on the integer tensor core (mma.sync m16n8, s8 / u8), any number of tokens in passes of 16.
//
// What bounds it: the weight stream, next to an instruction budget of about 60 issue slots per 16 rows x 32 weights at the full
// HBM rate.  So, as in the tiled Q4_K / Q8_0 kernel (gemv.cu), the packed integers become operand A with two to four logic
// operations per word, and everything per 32 or 16 weights stays in integers:
//   * activations are three s8 digits per value and 256-element block, x = amax / 8355711 * (65536 d1 + 256 d2 + d3): 24 bits,
//     rounding error 6e-8 of the block's maximum, and the three digits of a token are three COLUMNS of the product, each an
//     activation vector of its own whose scale carries the digit's weight.  (s16 per 32 elements, the previous scheme, needs a
//     conversion and a float scale per 32 weights, row and token.)  A block with a 32-element run whose maximum lies more than 255
//     times below the block's — there s16 per run would be the finer form — carries what the three digits leave as a second
//     slice of three more, and is walked twice: the error is nowhere larger than 16 bits per run gave.
//   * Q5_K's 6-bit and Q6_K's 8-bit sub-scales multiply the s32 sums (one IMAD each), Q8_K chains the accumulator over the whole
//     block, and only Q4_0 / Q5_0, whose scale is an f16 per 32 weights, go through f32 per MMA (the accumulator starts at
//     1.5 * 2^23 so that its bits ARE a float: no conversion instruction).
// A CTA owns 128 rows (a warp 16) and walks 256-element blocks; rows come in with cp.async (a row's block is 144 .. 304
// contiguous bytes) through a ring of stages, together with the block's activation slice, which the eight warps share.  The
// (row group, block) sequence is cut evenly over the resident CTAs and partial sums meet in gemv.cu's fashion, in slot order.
//
// Time per product in microseconds, staging included, back to back in a CUDA graph (rate of the reference bytes at one token), and
// in brackets the kernels before: dp2a on CUDA cores, and for Q6_K of two tokens and more an MMA kernel of 16 rows per CTA whose
// warps staged the activations each for themselves:
//   W[8192, 28672]   1 token            8 tokens     16 tokens         W[11008, 4096], 5 tokens
//   Q6_K             50 (62)  3.9 TB/s   74 (100)    120 (135)         20
//   Q5_K             45 (73)  3.6 TB/s   63          89 (590)          19 (61)
//   Q8_K             54 (69)  4.9 TB/s   63          87                19
//   Q4_0             39 (53)  3.3 TB/s   59          83 (590)          18
//   Q5_0             54 (67)  3.0 TB/s   72          98 (590)          21
// With a wide block in every CTA 1.7 times that (geometric mean); the flags and scales of the second slices cost the others 3 %.
#include "common.cuh"
#include "share_plan.cuh"

namespace gllmk {

namespace {

constexpr int RM_WARPS = 8, RM_ROWS = 16 * RM_WARPS;
constexpr int RM_PITCH = 288;  // digits of a column: 256 bytes, padded so that four columns' 8-byte fragments fall on different banks
constexpr int RM_PASS = 16;    // tokens per pass

__host__ __device__ constexpr int rm_groups(int m) { return (3 * m + 7) / 8; }  // MMA column groups
// slice of one block: [3m][288] digits, [3m][16] digit sums of the eight 32-element runs (S = 64 hi + lo: 8 hi, 8 lo), [8 groups] f32
__host__ __device__ constexpr uint32_t rm_slice_bytes(int m) { return (uint32_t)(3 * m) * (RM_PITCH + 16) + 32u * (uint32_t)rm_groups(m); }
// image: a slice per block, then as many for the rests of wide blocks.  Token t's block is wide: the word behind its first column's digits
__host__ __device__ constexpr size_t rm_image_bytes(int m, int64_t nb) { return 2 * (size_t)nb * rm_slice_bytes(m); }
__host__ __device__ constexpr uint32_t rm_flag_at(int tok) { return (uint32_t)(3 * tok) * RM_PITCH + 256u; }
constexpr float RM_WIDE = 255.0f;             // 8355711 / 32767: block maximum over a run's, from which on s16 per run is the finer form
constexpr float RM_REST = 2.0f * 8355711.0f;  // the rest is at most half a step: digits of rest * RM_REST

struct RmStage {
    const float *x;
    int64_t xst, xsk, k;
    int m, sums;
    uint8_t *img, *rest;
};

// q (24 bits, |q| <= 8355711) -> digit i of the three words, added to the digit sums
__device__ __forceinline__ void rm_digits(int q, int i, uint32_t (&w)[3], int (&s)[3]) {
    const int d3 = ((q + 128) & 255) - 128, q2 = (q - d3) >> 8;
    const int d2 = ((q2 + 128) & 255) - 128, d1 = (q2 - d2) >> 8;
    w[0] |= (uint32_t)(d1 & 255) << (8 * i);
    w[1] |= (uint32_t)(d2 & 255) << (8 * i);
    w[2] |= (uint32_t)(d3 & 255) << (8 * i);
    s[0] += d1;
    s[1] += d2;
    s[2] += d3;
}
// The words of elements kk .. kk + 3 of a block, and (sums) the digit sums of the run's eight lanes
__device__ __forceinline__ void rm_store(uint8_t *slice, int m, int tok, int kk, const uint32_t (&w)[3], int (&s)[3], int sums) {
    const int ncol = 3 * m, run = kk >> 5, j = (kk >> 2) & 7;
#pragma unroll
    for (int d = 0; d < 3; d++)
        *reinterpret_cast<uint32_t *>(slice + (3 * tok + d) * RM_PITCH + 32 * run + 8 * (j & 3) + 4 * (j >> 2)) = w[d];
    if (sums) {
#pragma unroll
        for (int d = 0; d < 3; d++) {
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) s[d] += __shfl_xor_sync(0xffffffffu, s[d], o);
            if (j == 0) {
                uint8_t *sp = slice + ncol * RM_PITCH + (3 * tok + d) * 16;
                sp[run] = (uint8_t)(int8_t)(s[d] >> 6);
                sp[8 + run] = (uint8_t)(s[d] & 63);
            }
        }
    }
}

// Thread = four elements; a CTA's 64 threads = one 256-element block.  In a run, elements 4t .. 4t + 3 and 16 + 4t .. + 3 are lane t's two
// operand-B words (byte 8t of the run).
__global__ void __launch_bounds__(64) raw_mma_stage_kernel(const RmStage p) {
    __shared__ float wmax[2], wmin[2];
    __shared__ int wbad[2];
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const int tok = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t k0 = ((int64_t)blockIdx.x * 64 + threadIdx.x) * 4;  // k is a multiple of 256: a block is inside or outside as a whole
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (k0 < p.k) {
        const float *xr = p.x + (int64_t)tok * p.xst + k0 * p.xsk;
        if (p.xsk == 1 && (reinterpret_cast<uintptr_t>(xr) & 15) == 0) {
            const float4 q = *reinterpret_cast<const float4 *>(xr);
            v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = xr[i * p.xsk];
        }
    }
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
    const float inf = __int_as_float(0x7F800000);
    int bad = !(fabsf(v[0]) < inf) || !(fabsf(v[1]) < inf) || !(fabsf(v[2]) < inf) || !(fabsf(v[3]) < inf);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    float low = amax > 0.0f ? amax : inf;  // smallest maximum of a run that is not all zero
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        low = fminf(low, __shfl_xor_sync(0xffffffffu, low, o));
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) { wmax[warp] = amax; wmin[warp] = low; wbad[warp] = bad; }
    __syncthreads();
    if (k0 >= p.k) return;
    amax = fmaxf(wmax[0], wmax[1]);
    bad = wbad[0] | wbad[1];
    const bool wide = !bad && amax > RM_WIDE * fminf(wmin[0], wmin[1]);
    // tiny blocks are pre-scaled by 2^64 so that 8355711 / amax stays finite
    const float pre = amax < 1e-20f ? 18446744073709551616.0f : 1.0f;
    const float inv = (amax > 0.0f && !bad) ? 8355711.0f / (amax * pre) : 0.0f;
    uint32_t w[3] = {0, 0, 0};
    int s[3] = {0, 0, 0};
    float rest[4];  // what the digits leave, in steps: exact, |rest| <= 1/2
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float f = (v[i] * pre) * inv, r = fminf(fmaxf(rintf(f), -8355711.0f), 8355711.0f);
        rest[i] = f - r;
        rm_digits(bad ? 0 : (int)r, i, w, s);
    }
    const int ncol = 3 * p.m, kk = (int)(k0 & 255);
    const int64_t at = (k0 >> 8) * (int64_t)rm_slice_bytes(p.m);
    uint8_t *slice = p.img + at, *slice2 = p.rest + at;
    rm_store(slice, p.m, tok, kk, w, s, p.sums);
    const uint32_t scales = (uint32_t)ncol * (RM_PITCH + 16);
    if (kk < 12) {  // three threads: one digit's column each
        const float unit = kk == 0 ? 65536.0f / 8355711.0f : (kk == 4 ? 256.0f / 8355711.0f : 1.0f / 8355711.0f);
        const uint32_t at_col = scales + 4 * (3 * tok + (kk >> 2));
        // an all-zero block: digits 0, times 1, so that an infinite weight scale still gives NaN
        *reinterpret_cast<float *>(slice + at_col) = bad ? __int_as_float(0x7FC00000) : (amax > 0.0f ? amax * unit : 1.0f);
        // 0: when another token's block is wide, this token's second slice is read too, and not written
        *reinterpret_cast<float *>(slice2 + at_col) = wide ? amax * (unit * (1.0f / RM_REST)) : 0.0f;
    }
    if (kk == 16) *reinterpret_cast<uint32_t *>(slice + rm_flag_at(tok)) = wide ? 1u : 0u;
    if (tok == 0 && kk >= 32 && kk < 64) {  // columns that only fill up the last group: at most seven
        const int col = ncol + ((kk - 32) >> 2);
        if (col < 8 * rm_groups(p.m)) {
            *reinterpret_cast<float *>(slice + scales + 4 * col) = 0.0f;
            *reinterpret_cast<float *>(slice2 + scales + 4 * col) = 0.0f;
        }
    }
    if (wide) {  // the CTA as a whole
        w[0] = w[1] = w[2] = 0;
        s[0] = s[1] = s[2] = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) rm_digits((int)fminf(fmaxf(rintf(rest[i] * RM_REST), -8355711.0f), 8355711.0f), i, w, s);
        rm_store(slice2, p.m, tok, kk, w, s, p.sums);
    }
}

// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t sm_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void cp16(uint32_t smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ float half_bits(uint32_t h) { return __half2float(__ushort_as_half((unsigned short)h)); }

// c = a x b + init (init in all four)
template <bool A_SIGNED>
__device__ __forceinline__ void mma32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b, int init) {
    if (A_SIGNED)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
                     : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y), "r"(init));
    else
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
                     : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y), "r"(init));
}
// c += a x b
__device__ __forceinline__ void mma32_acc(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y));
}
template <bool A_SIGNED>
__device__ __forceinline__ void mma16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    if (A_SIGNED)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};\n"
                     : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                     : "r"(a0), "r"(a1), "r"(b), "r"(0));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};\n"
                     : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                     : "r"(a0), "r"(a1), "r"(b), "r"(0));
}

// byte i of w, zero- or sign-extended
__device__ __forceinline__ int byte_u(uint32_t w, int i) { return (int)__byte_perm(w, 0u, 0x4440u + (uint32_t)i); }
__device__ __forceinline__ int byte_s(uint32_t w, int i) { return (int)(int8_t)(w >> (8 * i)); }

// Operand B of one lane: fragments of column group ng, run r at col(ng) + 32 r.  Lanes of columns past the last token read a zero
// region; only the last group has such columns.
struct RmCols {
    uint32_t first, last, sum_first, sum_last, scales;
};
template <int NG>
__device__ __forceinline__ uint32_t col_addr(const RmCols &x, int ng) { return ng == NG - 1 ? x.last : x.first + (uint32_t)(ng * 8 * RM_PITCH); }
template <int NG>
__device__ __forceinline__ uint32_t sum_addr(const RmCols &x, int ng) { return ng == NG - 1 ? x.sum_last : x.sum_first + (uint32_t)(ng * 8 * 16); }

// tot[ng][0, 1]: row g, columns 8 ng + 2t, + 1; [2, 3]: row g + 8.  REST (x may be a second slice): a column of scale 0 has no rest
// and adds nothing, whatever the slice holds there and the weight's scale is (0 * inf).
template <int NG, bool REST>
__device__ __forceinline__ void add_scaled(const RmCols &x, int t, int ng, const float (&f)[4], float (&tot)[NG][4]) {
    const uint2 s = lds64(x.scales + 32 * ng + 8 * t);
    const float sa = __uint_as_float(s.x), sb = __uint_as_float(s.y);
    if (!REST || sa != 0.0f) {
        tot[ng][0] = fmaf(sa, f[0], tot[ng][0]);
        tot[ng][2] = fmaf(sa, f[2], tot[ng][2]);
    }
    if (!REST || sb != 0.0f) {
        tot[ng][1] = fmaf(sb, f[1], tot[ng][1]);
        tot[ng][3] = fmaf(sb, f[3], tot[ng][3]);
    }
}

// Per format: BYTES of a row per 256 elements, CH 16-byte copies per row and block, PITCH of a row in shared memory (the 16 bytes
// four lanes read of eight rows fall on different banks), ALIGNED: every row's block starts on a 16-byte boundary.
// block(): one block of rows g (at r0) and g + 8 (at r8).
template <int QT>
struct Rm;

template <>
struct Rm<GLLMK_QUANT_Q5_K> {
    static constexpr int BYTES = 176, CH = 11, PITCH = 176;
    static constexpr bool ALIGNED = true;
    template <int NG, bool REST>
    static __device__ __forceinline__ void block(uint32_t r0, uint32_t r8, int t, const RmCols &x, float (&tot)[NG][4]) {
        static_assert(FD_Q5K.scale_offset == 0 && FD_Q5K.scale_min_offset == 2 && FD_Q5K.sub_scales_offset == 4 && FD_Q5K.data_high_offset == 16,
                      "Q5_K header is the block's first 16 bytes");
        // get_scale_min_k4 (k_quant.rs:388-397) for four sub-blocks at a time
        const uint4 h0 = lds128(r0), h8 = lds128(r8);
        const uint32_t sc0[2] = {h0.y & 0x3F3F3F3Fu, (h0.w & 0x0F0F0F0Fu) | ((h0.y >> 2) & 0x30303030u)};
        const uint32_t sc8[2] = {h8.y & 0x3F3F3F3Fu, (h8.w & 0x0F0F0F0Fu) | ((h8.y >> 2) & 0x30303030u)};
        const uint32_t ra = r0 + 4 * t, rb = r8 + 4 * t;
        const uint32_t H[4] = {lds32(ra + FD_Q5K.data_high_offset), lds32(rb + FD_Q5K.data_high_offset), lds32(ra + FD_Q5K.data_high_offset + 16),
                               lds32(rb + FD_Q5K.data_high_offset + 16)};
        int acc[NG][4];
#pragma unroll
        for (int ng = 0; ng < NG; ng++) acc[ng][0] = acc[ng][1] = acc[ng][2] = acc[ng][3] = 0;
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const uint32_t o = FD_Q5K.data_offset + 32 * p;
            const uint32_t Q[4] = {lds32(ra + o), lds32(rb + o), lds32(ra + o + 16), lds32(rb + o + 16)};
#pragma unroll
            for (int hs = 0; hs < 2; hs++) {
                const int sub = 2 * p + hs;
                uint32_t a[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint32_t hb = sub <= 4 ? H[i] << (4 - sub) : H[i] >> (sub - 4);  // bit `sub` of every byte -> bit 4
                    a[i] = ((hs ? Q[i] >> 4 : Q[i]) & 0x0F0F0F0Fu) | (hb & 0x10101010u);
                }
                const int s0 = byte_u(sc0[sub >> 2], sub & 3), s8 = byte_u(sc8[sub >> 2], sub & 3);
#pragma unroll
                for (int ng = 0; ng < NG; ng++) {
                    int c[4];
                    mma32<false>(c, a[0], a[1], a[2], a[3], lds64(col_addr<NG>(x, ng) + 32 * sub), 0);
                    acc[ng][0] += s0 * c[0];  // at most 8 * 63 * 32 * 31 * 128
                    acc[ng][1] += s0 * c[1];
                    acc[ng][2] += s8 * c[2];
                    acc[ng][3] += s8 * c[3];
                }
            }
        }
        // mins: A = the eight m of a row in k-slots 0 .. 7, B = the runs' digit sums split as 64 hi + lo
        const uint32_t m0 = t == 0 ? h0.z & 0x3F3F3F3Fu : (t == 1 ? ((h0.w >> 4) & 0x0F0F0F0Fu) | ((h0.z >> 2) & 0x30303030u) : 0u);
        const uint32_t m8 = t == 0 ? h8.z & 0x3F3F3F3Fu : (t == 1 ? ((h8.w >> 4) & 0x0F0F0F0Fu) | ((h8.z >> 2) & 0x30303030u) : 0u);
        const float d0 = half_bits(h0.x & 0xFFFF), mn0 = half_bits(h0.x >> 16), d8 = half_bits(h8.x & 0xFFFF), mn8 = half_bits(h8.x >> 16);
#pragma unroll
        for (int ng = 0; ng < NG; ng++) {
            const uint32_t sa = sum_addr<NG>(x, ng) + 4 * (t & 1);
            int hi[4], lo[4];
            mma16<false>(hi, m0, m8, lds32(sa));
            mma16<false>(lo, m0, m8, lds32(sa + 8));
            const float f[4] = {fmaf(d0, (float)acc[ng][0], -(mn0 * (float)(64 * hi[0] + lo[0]))),
                                fmaf(d0, (float)acc[ng][1], -(mn0 * (float)(64 * hi[1] + lo[1]))),
                                fmaf(d8, (float)acc[ng][2], -(mn8 * (float)(64 * hi[2] + lo[2]))),
                                fmaf(d8, (float)acc[ng][3], -(mn8 * (float)(64 * hi[3] + lo[3])))};
            add_scaled<NG, REST>(x, t, ng, f, tot);
        }
    }
};

template <>
struct Rm<GLLMK_QUANT_Q6_K> {
    static constexpr int BYTES = 224, CH = 14, PITCH = 240;
    static constexpr bool ALIGNED = true;
    // lo: a word whose bits 2 .. 5 of every byte are the low nibble; hi: bits 6 and 7 the high pair -> s8 4 (q - 32) (top bit flipped)
    static __device__ __forceinline__ uint32_t word(uint32_t lo, uint32_t hi) {
        return ((lo & 0x3C3C3C3Cu) | 0x80808080u) ^ (hi & 0xC0C0C0C0u);
    }
    template <int NG, bool REST>
    static __device__ __forceinline__ void block(uint32_t r0, uint32_t r8, int t, const RmCols &x, float (&tot)[NG][4]) {
        const uint4 S0 = lds128(r0 + FD_Q6K.sub_scales_offset), S8 = lds128(r8 + FD_Q6K.sub_scales_offset);
        const uint32_t s0w[4] = {S0.x, S0.y, S0.z, S0.w}, s8w[4] = {S8.x, S8.y, S8.z, S8.w};
        int acc[NG][4];
#pragma unroll
        for (int ng = 0; ng < NG; ng++) acc[ng][0] = acc[ng][1] = acc[ng][2] = acc[ng][3] = 0;
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
            // [16-element half of a run][row g, row g + 8]
            uint32_t A[2][2], B[2][2], H[2][2];
#pragma unroll
            for (int is = 0; is < 2; is++)
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const uint32_t rr = (r ? r8 : r0) + 4 * t + 16 * is;
                    A[is][r] = lds32(rr + FD_Q6K.data_offset + 64 * hh);
                    B[is][r] = lds32(rr + FD_Q6K.data_offset + 64 * hh + 32);
                    H[is][r] = lds32(rr + FD_Q6K.data_high_offset + 32 * hh);
                }
#pragma unroll
            for (int j = 0; j < 4; j++) {  // run 4 hh + j
                uint32_t q[2][2];
#pragma unroll
                for (int is = 0; is < 2; is++)
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        const uint32_t w = (j & 1) ? B[is][r] : A[is][r];
                        q[is][r] = word(j < 2 ? w << 2 : w >> 2, j == 3 ? H[is][r] : H[is][r] << (6 - 2 * j));
                    }
#pragma unroll
                for (int ng = 0; ng < NG; ng++) {
                    const uint2 b = lds64(col_addr<NG>(x, ng) + 32 * (4 * hh + j));
#pragma unroll
                    for (int is = 0; is < 2; is++) {
                        const int sb = 8 * hh + is + 2 * j;
                        const int s0 = byte_s(s0w[sb >> 2], sb & 3), s8 = byte_s(s8w[sb >> 2], sb & 3);
                        int c[4];
                        mma16<true>(c, q[is][0], q[is][1], is ? b.y : b.x);
                        acc[ng][0] += s0 * c[0];  // at most 16 * 128 * 16 * 128 * 128 = 2^29
                        acc[ng][1] += s0 * c[1];
                        acc[ng][2] += s8 * c[2];
                        acc[ng][3] += s8 * c[3];
                    }
                }
            }
        }
        const float d0 = 0.25f * half_bits(lds16(r0 + FD_Q6K.scale_offset)), d8 = 0.25f * half_bits(lds16(r8 + FD_Q6K.scale_offset));
#pragma unroll
        for (int ng = 0; ng < NG; ng++) {
            const float f[4] = {d0 * (float)acc[ng][0], d0 * (float)acc[ng][1], d8 * (float)acc[ng][2], d8 * (float)acc[ng][3]};
            add_scaled<NG, REST>(x, t, ng, f, tot);
        }
    }
};

template <>
struct Rm<GLLMK_QUANT_Q8_K> {
    // 292-byte blocks: a copy starts at the 16-byte boundary below the block
    static constexpr int BYTES = 292, CH = 19, PITCH = 304;
    static constexpr bool ALIGNED = false;
    template <int NG, bool REST>
    static __device__ __forceinline__ void block(uint32_t r0, uint32_t r8, int t, const RmCols &x, float (&tot)[NG][4]) {
        const uint32_t ra = r0 + FD_Q8K.data_offset + 4 * t, rb = r8 + FD_Q8K.data_offset + 4 * t;
        int acc[NG][4];
#pragma unroll
        for (int ng = 0; ng < NG; ng++) acc[ng][0] = acc[ng][1] = acc[ng][2] = acc[ng][3] = 0;
#pragma unroll
        for (int run = 0; run < 8; run++) {
            const uint32_t a0 = lds32(ra + 32 * run), a1 = lds32(rb + 32 * run), a2 = lds32(ra + 32 * run + 16), a3 = lds32(rb + 32 * run + 16);
#pragma unroll
            for (int ng = 0; ng < NG; ng++) mma32_acc(acc[ng], a0, a1, a2, a3, lds64(col_addr<NG>(x, ng) + 32 * run));
        }
        const float d0 = __uint_as_float(lds32(r0 + FD_Q8K.scale_offset)), d8 = __uint_as_float(lds32(r8 + FD_Q8K.scale_offset));
#pragma unroll
        for (int ng = 0; ng < NG; ng++) {
            const float f[4] = {d0 * (float)acc[ng][0], d0 * (float)acc[ng][1], d8 * (float)acc[ng][2], d8 * (float)acc[ng][3]};
            add_scaled<NG, REST>(x, t, ng, f, tot);
        }
    }
};

// Q4_0 / Q5_0: eight 32-element blocks (18 / 22 bytes) in a row's group of 256; odd blocks' payloads are 4-byte aligned, even ones' not
constexpr int RM_MAGIC = 0x4B400000;          // bits of 1.5 * 2^23: + c (|c| < 2^22) is the float 12582912 + c
constexpr float RM_MAGIC_F = 12582912.0f;
__device__ __forceinline__ uint32_t lds32_at(uint32_t a, bool aligned) { return aligned ? lds32(a) : lds16(a) | (lds16(a + 2) << 16); }

template <int QT>
struct RmClassic {
    static constexpr bool Q5 = QT == GLLMK_QUANT_Q5_0;
    static constexpr int BB = Q5 ? FD_Q5_0.block_bytes : FD_Q4_0.block_bytes, DATA = Q5 ? FD_Q5_0.data_offset : FD_Q4_0.data_offset;
    static constexpr int BYTES = 8 * BB, CH = BYTES / 16, PITCH = BYTES;
    static constexpr bool ALIGNED = true;
    template <int NG, bool REST>
    static __device__ __forceinline__ void block(uint32_t r0, uint32_t r8, int t, const RmCols &x, float (&tot)[NG][4]) {
        float cs[NG][4];
#pragma unroll
        for (int ng = 0; ng < NG; ng++) cs[ng][0] = cs[ng][1] = cs[ng][2] = cs[ng][3] = 0.0f;
#pragma unroll
        for (int b = 0; b < 8; b++) {
            uint32_t a[4];  // row g: elements 4t .. , row g + 8, row g: 16 + 4t .., row g + 8
            float d[2];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const uint32_t rr = (r ? r8 : r0) + BB * b;
                const uint32_t W = lds32_at(rr + DATA + 4 * t, (BB * b + DATA) % 4 == 0);
                if constexpr (Q5) {
                    // a 5-bit value with bit 4 flipped is q - 16 in 5-bit two's complement; three places up it is the s8 8 (q - 16)
                    const uint32_t qh = lds32_at(rr + FD_Q5_0.data_high_offset, (BB * b + FD_Q5_0.data_high_offset) % 4 == 0) >> (4 * t);
                    const uint32_t lo5 = ((qh & 0xFu) * 0x00204081u) & 0x01010101u, hi5 = (((qh >> 16) & 0xFu) * 0x00204081u) & 0x01010101u;
                    a[r] = ((W << 3) & 0x78787878u) | ((lo5 << 7) ^ 0x80808080u);
                    a[2 + r] = ((W >> 1) & 0x78787878u) | ((hi5 << 7) ^ 0x80808080u);
                    d[r] = 0.125f * half_bits(lds16(rr + FD_Q5_0.scale_offset));
                } else {
                    // a nibble with bit 3 flipped is q - 8 in 4-bit two's complement; in the high half of a byte it is the s8 16 (q - 8)
                    a[r] = ((W << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
                    a[2 + r] = (W & 0xF0F0F0F0u) ^ 0x80808080u;
                    d[r] = 0.0625f * half_bits(lds16(rr + FD_Q4_0.scale_offset));
                }
            }
#pragma unroll
            for (int ng = 0; ng < NG; ng++) {
                int c[4];
                mma32<true>(c, a[0], a[1], a[2], a[3], lds64(col_addr<NG>(x, ng) + 32 * b), RM_MAGIC);  // |c| <= 32 * 128 * 128 = 2^19
                cs[ng][0] = fmaf(d[0], __int_as_float(c[0]) - RM_MAGIC_F, cs[ng][0]);
                cs[ng][1] = fmaf(d[0], __int_as_float(c[1]) - RM_MAGIC_F, cs[ng][1]);
                cs[ng][2] = fmaf(d[1], __int_as_float(c[2]) - RM_MAGIC_F, cs[ng][2]);
                cs[ng][3] = fmaf(d[1], __int_as_float(c[3]) - RM_MAGIC_F, cs[ng][3]);
            }
        }
#pragma unroll
        for (int ng = 0; ng < NG; ng++) add_scaled<NG, REST>(x, t, ng, cs[ng], tot);
    }
};
template <>
struct Rm<GLLMK_QUANT_Q4_0> : RmClassic<GLLMK_QUANT_Q4_0> {};
template <>
struct Rm<GLLMK_QUANT_Q5_0> : RmClassic<GLLMK_QUANT_Q5_0> {};

struct RmParams {
    const uint8_t *w;
    const uint8_t *img, *rest;
    float *y;
    const float *row_scales;
    int64_t n_row_scales;
    int64_t n, yst, ysr;
    uint32_t pitch;   // bytes of a row
    int nb;           // 256-element blocks per row
    int m;
    int stages;
    int per_cta, rem; // (row group, block) units per CTA: the first `rem` CTAs own one more
    int maxslot;
    float *partial;   // [tiles of 16 rows][maxslot][16 tokens][16 rows]
    int *counters;    // [tiles] arrivals, zero between launches
};

__device__ __forceinline__ int rm_cta_of(const RmParams &p, int64_t u) {
    const int64_t big = (int64_t)p.rem * (p.per_cta + 1);
    return u < big ? (int)(u / (p.per_cta + 1)) : p.rem + (int)((u - big) / p.per_cta);
}

// Adds the shares of TL tokens (t0, t0 + 2, ...) in slot order, SU slots' loads in flight at a time.
template <int TL, int SU>
__device__ __forceinline__ void rm_sum(const RmParams &p, const float *part, int t0, int nsl, float sc, float *y) {
    float v[TL];
#pragma unroll
    for (int i = 0; i < TL; i++) v[i] = 0.0f;
    for (int s = 0; s < nsl; s += SU) {
        float q[SU][TL];
#pragma unroll
        for (int u = 0; u < SU; u++)
#pragma unroll
            for (int i = 0; i < TL; i++) q[u][i] = s + u < nsl && t0 + 2 * i < p.m ? __ldcg(part + (size_t)(s + u) * 256 + (t0 + 2 * i) * 16) : 0.0f;
#pragma unroll
        for (int u = 0; u < SU; u++)
#pragma unroll
            for (int i = 0; i < TL; i++) v[i] += q[u][i];
    }
#pragma unroll
    for (int i = 0; i < TL; i++)
        if (t0 + 2 * i < p.m) y[(size_t)(t0 + 2 * i) * p.yst] = p.n_row_scales > 0 ? v[i] * sc : v[i];
}

// This warp's share of a row tile is complete: red[16][rp] holds its column sums.  The last contributing CTA adds the shares in
// slot order and writes y.  FEW (one or two tokens): a plain loop over the shares; the batches' registers, live across this call,
// cost the one-group kernels 10 % of their whole time (Q4_0 W[8192, 28672] 38.7 against 42.4 us).
template <bool FEW>
__device__ __noinline__ void rm_flush(const RmParams &p, const float *red, int rp, int64_t tile, int slot, int nsl) {
    const int lane = threadIdx.x & 31, r = lane & 15, t0 = lane >> 4;
    float *base = p.partial + (size_t)tile * p.maxslot * 256;
    if (nsl > 1) {
        float *mine = base + (size_t)slot * 256;
        for (int tok = t0; tok < p.m; tok += 2) {
            const float *c = red + r * rp + 3 * tok;
            __stcg(mine + tok * 16 + r, (c[2] + c[1]) + c[0]);
        }
        __threadfence();
        __syncwarp();
        int arrived = 0;
        if (lane == 0) arrived = atomicAdd(p.counters + tile, 1);
        arrived = __shfl_sync(0xffffffffu, arrived, 0);
        if (arrived != nsl - 1) return;
        __threadfence();
        if (lane == 0) p.counters[tile] = 0;  // ready for the next launch
    }
    const int64_t row = tile * 16 + r;
    if (row >= p.n) return;
    float sc = 1.0f;
    if (p.n_row_scales == 1) sc = p.row_scales[0];
    else if (p.n_row_scales > 1) sc = p.row_scales[row];
    float *y = p.y + (size_t)row * p.ysr;
    if (nsl > 1) {
        // one L2 round trip per batch, not per share (W[4096, 4096], 16 tokens, 15 shares per tile: 21 -> 18 us)
        if (FEW) {
            for (int tok = t0; tok < p.m; tok += 2) {
                float v = 0.0f;
                for (int s = 0; s < nsl; s++) v += __ldcg(base + (size_t)s * 256 + tok * 16 + r);
                y[(size_t)tok * p.yst] = p.n_row_scales > 0 ? v * sc : v;
            }
        } else if (p.m <= 8) rm_sum<4, 4>(p, base + r, t0, nsl, sc, y);
        else rm_sum<8, 4>(p, base + r, t0, nsl, sc, y);
        return;
    }
    for (int tok = t0; tok < p.m; tok += 2) {
        const float *c = red + r * rp + 3 * tok;
        const float v = (c[2] + c[1]) + c[0];
        y[(size_t)tok * p.yst] = p.n_row_scales > 0 ? v * sc : v;
    }
}

template <int QT>
__host__ __device__ constexpr uint32_t rm_stage_bytes(int m) { return RM_ROWS * Rm<QT>::PITCH + rm_slice_bytes(m); }
__host__ __device__ constexpr uint32_t rm_red_bytes(int ng) { return RM_WARPS * 16 * (8 * ng + 1) * 4; }
// shared memory: stages | zero columns (256 bytes) | column sums of the eight warps
template <int QT>
__host__ __device__ constexpr size_t rm_smem_bytes(int m, int stages) {
    return (size_t)stages * rm_stage_bytes<QT>(m) + 256 + rm_red_bytes(rm_groups(m));
}
__host__ __device__ constexpr int rm_min_ctas(int ng) { return ng <= 2 ? 3 : 2; }

template <int QT, int NG>
__device__ __noinline__ void rm_wide(const RmParams &p, int i0);

// The CTA's units from number i0 on.  WIDE: i0 is a wide block whose first walk is done, with the sums so far in `red`; wide blocks are
// walked twice.
template <int QT, int NG, bool WIDE>
__device__ __forceinline__ void rm_body(const RmParams &p, const int i0) {
    using F = Rm<QT>;
    constexpr int CH = F::CH;
    extern __shared__ __align__(128) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int ncol = 3 * p.m, S = p.stages, nb = p.nb;
    const uint32_t slice = rm_slice_bytes(p.m), stage = RM_ROWS * F::PITCH + slice;
    const uint32_t base = sm_addr(smem), zero = base + S * stage;
    float *red = reinterpret_cast<float *>(smem + (size_t)S * stage + 256) + warp * 16 * (8 * NG + 1);
    const int64_t u0 = (int64_t)blockIdx.x * p.per_cta + min((int)blockIdx.x, p.rem) + i0;
    const int n = p.per_cta + ((int)blockIdx.x < p.rem ? 1 : 0) - i0;

    // ---- copies: the producer's position runs S - 1 steps ahead of the consumer's ----
    // Half a warp per row piece (a whole one for Q8_K's nineteen 16-byte chunks): lane = chunk, so a copy is one instruction and one
    // addition (with chunk i = lane + 32 j of all sixteen pieces instead, the index arithmetic took a third of the kernel's
    // instructions: Q6_K W[8192, 28672], one token 52 us)
    int64_t ptg = u0 / nb;
    int pb = (int)(u0 - ptg * nb);
    constexpr int LPR = CH > 16 ? 32 : 16, RPI = 32 / LPR;  // lanes per row piece, row pieces per instruction
    const int hrow = lane / LPR, ch = lane % LPR;
    const uint32_t wdst = base + (16 * warp + hrow) * F::PITCH + 16 * ch;
    const uint8_t *wsrc = nullptr;  // this lane's chunk of the first row piece it copies
    int rows = 0;                   // rows of the warp's tile inside the matrix
    const auto set_tile = [&]() {
        const int64_t row0 = ptg * RM_ROWS + 16 * warp;
        rows = row0 + 16 <= p.n ? 16 : (row0 < p.n ? (int)(p.n - row0) : 0);
        wsrc = p.w + (size_t)(row0 + (hrow < rows ? hrow : 0)) * p.pitch + (size_t)pb * F::BYTES + 16 * ch;
    };
    const auto copy_rows = [&](int st) {
        if (ch < CH) {
            uint32_t dst = wdst + st * stage;
            if (rows == 16) {
                const uint8_t *src = wsrc;
#pragma unroll
                for (int j = 0; j < 16 / RPI; j++, src += (size_t)RPI * p.pitch, dst += RPI * F::PITCH)
                    cp16(dst, F::ALIGNED ? src : reinterpret_cast<const uint8_t *>(reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)15));
            } else {
                // the matrix ends inside the tile: rows past the last one are not copied (what they yield is not stored)
                for (int r = hrow; r < rows; r += RPI, dst += RPI * F::PITCH) {
                    const uintptr_t src = reinterpret_cast<uintptr_t>(wsrc) + (size_t)(r - hrow) * p.pitch;
                    cp16(dst, reinterpret_cast<const uint8_t *>(F::ALIGNED ? src : src & ~(uintptr_t)15));
                }
            }
        }
    };
    const auto copy_slice = [&](int b, int st) {
        const uint8_t *src = p.img + (size_t)b * slice;
        const uint32_t dst = base + st * stage + RM_ROWS * F::PITCH;
        for (uint32_t o = threadIdx.x * 16; o < slice; o += RM_WARPS * 32 * 16) cp16(dst + o, src + o);
    };
    const auto advance = [&]() {
        wsrc += F::BYTES;
        if (++pb == nb) {
            pb = 0;
            ptg++;
            set_tile();
        }
    };
    if (threadIdx.x < 64) asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(zero + 4 * threadIdx.x), "r"(0) : "memory");
    set_tile();
    {
        // weights of the first stages do not depend on the staging kernel; the activation slices do
        int bs[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            bs[i] = pb;
            if (i < S - 1 && i < n) {
                copy_rows(i);
                advance();
            }
        }
        asm volatile("griddepcontrol.wait;\n" ::: "memory");  // everything before this grid in the stream is complete from here on
#pragma unroll
        for (int i = 0; i < 3; i++)
            if (i < S - 1) {
                if (i < n) copy_slice(bs[i], i);
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
    }

    const bool last_on = (NG - 1) * 8 + g < ncol;
    // row g (+ 8), column 8 ng + 2t (+ 1) of the warp's sums
    const auto red_at = [&](int ng, int j) -> float & { return red[(g + 8 * (j >> 1)) * (8 * NG + 1) + 8 * ng + 2 * t + (j & 1)]; };
    float tot[NG][4];
#pragma unroll
    for (int ng = 0; ng < NG; ng++)
#pragma unroll
        for (int j = 0; j < 4; j++) tot[ng][j] = WIDE ? red_at(ng, j) : 0.0f;
    int64_t tg = u0 / nb;
    int b = (int)(u0 - tg * nb), st = 0;
    for (int i = 0; i < n; i++) {
        // stage i has landed for this thread, and behind the barrier for all; nobody reads stage i - 1 any more
        if (S == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
        else if (S == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 2;" ::: "memory");
        __syncthreads();
        if (i + S - 1 < n) {
            const int ps = st == 0 ? S - 1 : st - 1;
            copy_rows(ps);
            copy_slice(pb, ps);
            advance();
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const int64_t row0 = tg * RM_ROWS + 16 * warp;
        const uint32_t xs = base + st * stage + RM_ROWS * F::PITCH;
        const uint32_t flag = lds32(lane < p.m ? xs + rm_flag_at(lane) : zero);
#pragma unroll 1
        for (int pass = WIDE && i == 0 ? 1 : 0;; pass++) {
            if (WIDE && pass > 0) {
                // the rests take the slice's place in the stage
                __syncthreads();
                const uint8_t *src = p.rest + (size_t)b * slice;
                for (uint32_t o = threadIdx.x * 16; o < slice; o += RM_WARPS * 32 * 16) {
                    const uint4 q = __ldcg(reinterpret_cast<const uint4 *>(src + o));
                    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(xs + o), "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w) : "memory");
                }
                __syncthreads();
            }
            if (row0 < p.n) {
                uint32_t r0 = base + st * stage + (16 * warp + g) * F::PITCH, r8 = r0 + 8 * F::PITCH;
                if (!F::ALIGNED) {
                    // where the block starts in its first 16 bytes
                    const uint32_t ra = (uint32_t)reinterpret_cast<uintptr_t>(p.w) + (uint32_t)b * F::BYTES + (uint32_t)(row0 + g) * p.pitch;
                    r0 += ra & 15u;
                    r8 += (ra + 8 * p.pitch) & 15u;
                }
                RmCols x;
                x.first = xs + g * RM_PITCH + 8 * t;
                x.last = last_on ? x.first + (NG - 1) * 8 * RM_PITCH : zero;
                x.sum_first = xs + ncol * RM_PITCH + g * 16;
                x.sum_last = last_on ? x.sum_first + (NG - 1) * 8 * 16 : zero;
                x.scales = xs + ncol * (RM_PITCH + 16);
                F::template block<NG, WIDE>(r0, r8, t, x, tot);
            }
            if (!WIDE || pass > 0 || !__any_sync(0xffffffffu, flag != 0)) break;
        }
        if (!WIDE && __any_sync(0xffffffffu, flag != 0)) {
            // A wide block (all warps see the same): the rest of the way out of line, for the plain loop's registers (second walk inside
            // it: Q8_K W[8192, 28672] x 16 tokens 90 us, now 87; 83 without the second slice).
#pragma unroll
            for (int ng = 0; ng < NG; ng++)
#pragma unroll
                for (int j = 0; j < 4; j++) red_at(ng, j) = tot[ng][j];
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            rm_wide<QT, NG>(p, i);
            return;
        }
        st = st + 1 == S ? 0 : st + 1;
        if (++b == nb || i + 1 == n) {
            if (row0 < p.n) {
                const int64_t first = tg * nb;
                const int slot0 = rm_cta_of(p, first), nsl = rm_cta_of(p, first + nb - 1) - slot0 + 1;
#pragma unroll
                for (int ng = 0; ng < NG; ng++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        red_at(ng, j) = tot[ng][j];
                        tot[ng][j] = 0.0f;
                    }
                __syncwarp();
                rm_flush<NG == 1>(p, red, 8 * NG + 1, tg * RM_WARPS + warp, (int)blockIdx.x - slot0, nsl);
                __syncwarp();
            }
            b = 0;
            tg++;
        }
    }
}
template <int QT, int NG>
__device__ __noinline__ void rm_wide(const RmParams &p, int i0) { rm_body<QT, NG, true>(p, i0); }

template <int QT, int NG>
__global__ void __launch_bounds__(RM_WARPS * 32, rm_min_ctas(NG)) raw_mma_gemv_kernel(const __grid_constant__ RmParams p) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    rm_body<QT, NG, false>(p, 0);
}

// Resident CTAs per SM and stages for (format, groups, tokens): as many CTAs as the registers allow with two stages, then as many
// stages (at most four) as still fit them.  Asked once per device.
template <int QT, int NG>
cudaError_t rm_plan(int device, int m, int *ctas, int *stages) {
    static int cache[16][RM_PASS + 1];  // ctas * 8 + stages, 0 = not yet asked
    if (device >= 0 && device < 16 && cache[device][m]) {
        *ctas = cache[device][m] >> 3;
        *stages = cache[device][m] & 7;
        return cudaSuccess;
    }
    cudaError_t e = cudaFuncSetAttribute(raw_mma_gemv_kernel<QT, NG>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    int n = 0, s = 2;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, raw_mma_gemv_kernel<QT, NG>, RM_WARPS * 32, rm_smem_bytes<QT>(m, 2));
    if (e != cudaSuccess) return e;
    if (n < 1) return cudaErrorInvalidConfiguration;
    for (; s < 4; s++) {
        if (rm_smem_bytes<QT>(m, s + 1) > 227 * 1024) break;
        int more = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&more, raw_mma_gemv_kernel<QT, NG>, RM_WARPS * 32, rm_smem_bytes<QT>(m, s + 1));
        if (e != cudaSuccess) return e;
        if (more < n) break;
    }
    if (device >= 0 && device < 16) cache[device][m] = n * 8 + s;
    *ctas = n;
    *stages = s;
    return cudaSuccess;
}

template <int QT, int NG>
int32_t rm_pass(Ctx *c, RmParams &p, cudaStream_t s) {
    int per_sm = 1;
    GK_CUDA(c, (rm_plan<QT, NG>(c->device, p.m, &per_sm, &p.stages)));
    if (c->gemv_ctas_per_sm > 0 && c->gemv_ctas_per_sm < per_sm) per_sm = (int)c->gemv_ctas_per_sm;
    const int64_t groups = (p.n + RM_ROWS - 1) / RM_ROWS, units = groups * p.nb;
    const int64_t ctas = decode_ctas(units, (int64_t)c->sm_count * per_sm, per_sm, p.nb, NG > 1, false);
    if (units / ctas > 0x3fffffff) return fail(c, GLLMK_STATUS_INVALID_ARG, "gemv: matrix too large");
    p.per_cta = (int)(units / ctas);
    p.rem = (int)(units % ctas);
    p.maxslot = (p.nb - 1) / p.per_cta + 2;
    const size_t tiles = (size_t)groups * RM_WARPS;
    int32_t rc = ensure_red(c, tiles * p.maxslot * 256 * sizeof(float));
    if (!rc) rc = ensure_cnt(c, tiles * sizeof(int));
    if (rc) return rc;
    p.partial = static_cast<float *>(c->red);
    p.counters = static_cast<int *>(c->cnt);
    GK_CUDA(c, launch_after(raw_mma_gemv_kernel<QT, NG>, c->gemv_pdl != 0, dim3((unsigned)ctas), RM_WARPS * 32, rm_smem_bytes<QT>(p.m, p.stages), s, p));
    return GLLMK_STATUS_OK;
}

template <int QT>
int32_t rm_format(Ctx *c, RmParams &p, cudaStream_t s) {
    switch (rm_groups(p.m)) {
        case 1: return rm_pass<QT, 1>(c, p, s);
        case 2: return rm_pass<QT, 2>(c, p, s);
        case 3: return rm_pass<QT, 3>(c, p, s);
        case 4: return rm_pass<QT, 4>(c, p, s);
        case 5: return rm_pass<QT, 5>(c, p, s);
        default: return rm_pass<QT, 6>(c, p, s);
    }
}

}  // namespace

// Q4_0 / Q5_0 rows of whole 256-element groups start on 16-byte boundaries; the others stay on the dp2a kernel (gguf_raw.cu), and
// so does everything it can take when the context says so
bool raw_mma_takes(const Ctx *c, const Weight *w) {
    const bool classic = w->qt == GLLMK_QUANT_Q4_0 || w->qt == GLLMK_QUANT_Q5_0;
    return !classic || (w->k % 256 == 0 && c->raw_gemv_mma != 0);
}

int32_t raw_mma_launch(Ctx *c, const Weight *w, const float *x, int64_t xst, int64_t xsk, int m, float *y, int64_t yst, int64_t ysr,
                       const float *row_scales, int64_t n_row_scales, cudaStream_t s) {
    const int64_t nb = w->k / 256;
    const int most = m < RM_PASS ? m : RM_PASS;
    int32_t rc = ensure_act(c, rm_image_bytes(most, nb));
    if (rc) return rc;
    RmParams p{};
    p.w = static_cast<const uint8_t *>(w->qs);
    p.row_scales = row_scales;
    p.n_row_scales = row_scales ? n_row_scales : 0;
    p.n = w->n;
    p.yst = yst;
    p.ysr = ysr;
    p.nb = (int)nb;
    p.pitch = (uint32_t)((w->qs_bytes - 16) / (size_t)w->n);
    for (int t0 = 0; t0 < m; t0 += RM_PASS) {
        p.m = m - t0 < RM_PASS ? m - t0 : RM_PASS;
        p.y = y + (int64_t)t0 * yst;
        uint8_t *img = static_cast<uint8_t *>(c->act), *rest = img + (size_t)nb * rm_slice_bytes(p.m);
        p.img = img;
        p.rest = rest;
        RmStage sp{x + (int64_t)t0 * xst, xst, xsk, w->k, p.m, w->qt == GLLMK_QUANT_Q5_K, img, rest};
        GK_CUDA(c, launch_after(raw_mma_stage_kernel, c->gemv_pdl != 0 && !c->peer_waits, dim3((unsigned)nb, (unsigned)p.m), 64, 0, s, sp));
        switch (w->qt) {
            case GLLMK_QUANT_Q6_K: rc = rm_format<GLLMK_QUANT_Q6_K>(c, p, s); break;
            case GLLMK_QUANT_Q5_K: rc = rm_format<GLLMK_QUANT_Q5_K>(c, p, s); break;
            case GLLMK_QUANT_Q8_K: rc = rm_format<GLLMK_QUANT_Q8_K>(c, p, s); break;
            case GLLMK_QUANT_Q4_0: rc = rm_format<GLLMK_QUANT_Q4_0>(c, p, s); break;
            case GLLMK_QUANT_Q5_0: rc = rm_format<GLLMK_QUANT_Q5_0>(c, p, s); break;
            default: return fail(c, GLLMK_STATUS_UNSUPPORTED, "gemv: quant type %d", w->qt);
        }
        if (rc) return rc;
    }
    return GLLMK_STATUS_OK;
}

}  // namespace gllmk
