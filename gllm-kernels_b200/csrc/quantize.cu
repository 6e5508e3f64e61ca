// On-device quantizers f32 -> Q4_K / Q8_0 / MXFP4 / NVFP4 blocks in the reference's byte formats.
// The reference ships no encoder for these formats; the rules below are this library's own and
// are the exact inverse conventions of the decoders (k_quant.rs:7-56, classic.rs:860-868,
// quant_mxfp4.rs:72-109, quant.rs:77-86).  All arithmetic is plain IEEE f32 (the library is
// compiled with -fmad=false) so a CPU implementation of the same rules produces identical bytes.
#include "common.cuh"

namespace gllmk {

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// nearest E2M1 code; ties go to the code with an even low bit; zero keeps code 0 (+0)
__device__ __forceinline__ uint32_t nearest_e2m1(float v) {
    const float mags[8] = {0.0f, 0.5f, 1.0f, 1.5f, 2.0f, 3.0f, 4.0f, 6.0f};
    const float a = fabsf(v);
    int best = 0;
    float bd = a;
#pragma unroll
    for (int c = 1; c < 8; c++) {
        const float dist = fabsf(a - mags[c]);
        if (dist < bd || (dist == bd && (c & 1) == 0)) { bd = dist; best = c; }
    }
    if (best == 0) return 0u;
    return (uint32_t)best | ((v < 0.0f) ? 8u : 0u);
}

// Eight values -> one word of E2M1 codes (nearest_e2m1 of each; element 0 in the low nibble) by the hardware conversion, which
// rounds to nearest with ties to the even code as well.  It keeps the sign of a zero, which is taken off again.
__device__ __forceinline__ uint32_t e2m1x8(const float (&v)[8]) {
    uint32_t w;
    asm("{\n.reg .b8 a, b, c, d;\n"
        "cvt.rn.satfinite.e2m1x2.f32 a, %2, %1;\ncvt.rn.satfinite.e2m1x2.f32 b, %4, %3;\n"
        "cvt.rn.satfinite.e2m1x2.f32 c, %6, %5;\ncvt.rn.satfinite.e2m1x2.f32 d, %8, %7;\n"
        "mov.b32 %0, {a, b, c, d};\n}\n"
        : "=r"(w)
        : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
    const uint32_t nonzero = ((w & 0x77777777u) + 0x77777777u) & 0x88888888u;  // bit 3 of every nibble whose magnitude is not 0
    return w & (0x77777777u | nonzero);
}
// largest magnitude the conversion above is used for (beyond it, and for NaN, nearest_e2m1 decides value by value: the scale
// was clamped, or the input is not finite)
constexpr float E2M1_FAST = 1024.0f;
__device__ __forceinline__ bool all_below(const float (&v)[8], float lim) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 8; i++) ok = ok && fabsf(v[i]) < lim;  // false for NaN
    return ok;
}
__device__ __noinline__ uint32_t e2m1x8_slow(const float (&v)[8]) {
    uint32_t w = 0;
    for (int i = 0; i < 8; i++) w |= nearest_e2m1(v[i]) << (4 * i);
    return w;
}
// eight consecutive floats; vec = the address is 16-byte aligned
__device__ __forceinline__ void load8(const float *x, int vec, float (&v)[8]) {
    if (vec) {
        const float4 a = __ldg(reinterpret_cast<const float4 *>(x)), b = __ldg(reinterpret_cast<const float4 *>(x) + 1);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __ldg(x + i);
    }
}
__device__ __forceinline__ float max_abs8(const float (&v)[8]) {
    float a = fabsf(v[0]);
#pragma unroll
    for (int i = 1; i < 8; i++) a = fmaxf(a, fabsf(v[i]));
    return a;
}

// f32_to_e4m3, src/compiler/codegen/vm/numerical_sim.rs:2751-2808, for v >= 0
__device__ __forceinline__ uint32_t f32_to_ue4m3(float v) {
    if (v != v) return 0x7Fu;
    float a = fabsf(v);
    if (a > 448.0f) a = 448.0f;
    if (a == 0.0f) return 0u;
    const uint32_t ab = (uint32_t)__float_as_int(a);
    int e4 = (int)(ab >> 23) - 127 + 7;
    const uint32_t m23 = ab & 0x7FFFFFu;
    int m3;
    if (e4 <= 0) {
        e4 = 0;
        m3 = (int)roundf(a * 512.0f);
    } else {
        const int top3 = (int)(m23 >> 20);
        const uint32_t rem = m23 & 0xFFFFFu, half = 0x80000u;
        int m = top3;
        if (rem > half || (rem == half && (top3 & 1) == 1)) {
            m += 1;
            if (m > 7) { m = 0; e4 += 1; }
        }
        if (e4 > 15) { e4 = 15; m3 = 7; }
        else m3 = m;
    }
    e4 = clampi(e4, 0, 15);
    m3 = clampi(m3, 0, 7);
    return ((uint32_t)e4 << 3) | (uint32_t)m3;
}

// ---- Q4_K: one warp per 256-block, lane l handles elements l, 32+l, ... (one per sub-block) ----
__global__ void __launch_bounds__(256) quantize_q4k_kernel(const float *__restrict__ x, uint8_t *__restrict__ out,
                                                            size_t nblocks) {
    const size_t blk = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (blk >= nblocks) return;
    const float *xb = x + blk * 256;
    uint8_t *b = out + blk * 144;
    float v[8], s[8], o[8];
    float smax = 0.0f, omax = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        v[j] = xb[j * 32 + lane];
        float lo = fminf(v[j], 0.0f), hi = fmaxf(v[j], 0.0f);
#pragma unroll
        for (int d = 16; d; d >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, d));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d));
        }
        s[j] = (hi - lo) / 15.0f;
        o[j] = -lo;
        smax = fmaxf(smax, s[j]);
        omax = fmaxf(omax, o[j]);
    }
    const __half dh = __float2half_rn(smax / 63.0f), mh = __float2half_rn(omax / 63.0f);
    const float d = __half2float(dh), dmin = __half2float(mh);
    int sc[8], mn[8];
    uint32_t q[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        sc[j] = (d > 0.0f) ? clampi((int)rintf(s[j] / d), 0, 63) : 0;
        mn[j] = (dmin > 0.0f) ? clampi((int)rintf(o[j] / dmin), 0, 63) : 0;
        const float ds = d * (float)sc[j], off = dmin * (float)mn[j];
        q[j] = (ds > 0.0f) ? (uint32_t)clampi((int)rintf((v[j] + off) / ds), 0, 15) : 0u;
    }
    if (lane == 0) {
        *reinterpret_cast<unsigned short *>(b) = __half_as_ushort(dh);
        *reinterpret_cast<unsigned short *>(b + 2) = __half_as_ushort(mh);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            b[4 + j] = (uint8_t)(sc[j] | ((sc[j + 4] >> 4) << 6));
            b[8 + j] = (uint8_t)(mn[j] | ((mn[j + 4] >> 4) << 6));
            b[12 + j] = (uint8_t)((sc[j + 4] & 15) | ((mn[j + 4] & 15) << 4));
        }
    }
#pragma unroll
    for (int g = 0; g < 4; g++) b[16 + 32 * g + lane] = (uint8_t)(q[2 * g] | (q[2 * g + 1] << 4));
}

// ---- Q8_0: one warp per 32-block ----
__global__ void __launch_bounds__(256) quantize_q80_kernel(const float *__restrict__ x, uint8_t *__restrict__ out,
                                                            size_t nblocks) {
    const size_t blk = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (blk >= nblocks) return;
    const float v = x[blk * 32 + lane];
    float amax = fabsf(v);
#pragma unroll
    for (int d = 16; d; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
    const __half dh = __float2half_rn(amax / 127.0f);
    const float d = __half2float(dh);
    const int q = (d > 0.0f) ? clampi((int)roundf(v / d), -127, 127) : 0;
    uint8_t *b = out + blk * 34;
    if (lane == 0) *reinterpret_cast<unsigned short *>(b) = __half_as_ushort(dh);
    b[2 + lane] = (uint8_t)(int8_t)q;
}

// The two FP4 encoders are bound by reading x once.  A lane takes eight consecutive elements (two 16-byte loads, one 4-byte
// store of codes), two such units in flight per thread; the block's maximum is a few shuffles.  x [2048, 4096], NVFP4, from a
// cold cache: 12 us (34 with 8-byte loads, 1-byte stores, a search of the eight magnitudes and an IEEE division per element).
constexpr int QF_UNITS = 2;

// ---- MXFP4 (block 32 = 4 lanes), split output (16 nibble bytes + 1 E8M0 byte) ----
__global__ void __launch_bounds__(256) quantize_mxfp4_kernel(const float *__restrict__ x, int vec, uint32_t *__restrict__ blocks,
                                                              uint8_t *__restrict__ scales, size_t units) {
    const size_t u0 = (size_t)blockIdx.x * (256 * QF_UNITS) + threadIdx.x;
    float v[QF_UNITS][8];
#pragma unroll
    for (int j = 0; j < QF_UNITS; j++) {
        const size_t u = u0 + 256 * j;
        if (u < units) load8(x + 8 * u, vec, v[j]);
        else
#pragma unroll
            for (int i = 0; i < 8; i++) v[j][i] = 0.0f;
    }
#pragma unroll
    for (int j = 0; j < QF_UNITS; j++) {
        const size_t u = u0 + 256 * j;
        float amax = max_abs8(v[j]);
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        int byte = 127;
        if (amax > 0.0f) {
            int p;
            const float f = frexpf(amax, &p);  // smallest e with 6 * 2^e >= amax
            const int e = (f <= 0.75f) ? p - 3 : p - 2;
            byte = clampi(e + 127, 1, 254);
        }
        // 2^(127 - byte), exactly (byte 254: 2^-127, a subnormal)
        const float inv = __int_as_float(byte == 254 ? 0x00400000 : (254 - byte) << 23);
        float q[8];
#pragma unroll
        for (int i = 0; i < 8; i++) q[i] = v[j][i] * inv;
        const uint32_t w = all_below(q, E2M1_FAST) ? e2m1x8(q) : e2m1x8_slow(q);
        if (u < units) {
            blocks[u] = w;
            if ((u & 3) == 0) scales[u >> 2] = (uint8_t)byte;
        }
    }
}

// ---- NVFP4 (block 64 = 4 x 16 elements, 8 lanes): 4 UE4M3 bytes, 32 code bytes; global from device memory or by value ----
__global__ void __launch_bounds__(256) quantize_nvfp4_kernel(const float *__restrict__ x, int vec, uint8_t *__restrict__ out,
                                                              const float *__restrict__ global_ptr, float global, size_t units) {
    const size_t u0 = (size_t)blockIdx.x * (256 * QF_UNITS) + threadIdx.x;
    float v[QF_UNITS][8];
#pragma unroll
    for (int j = 0; j < QF_UNITS; j++) {
        const size_t u = u0 + 256 * j;
        if (u < units) load8(x + 8 * u, vec, v[j]);
        else
#pragma unroll
            for (int i = 0; i < 8; i++) v[j][i] = 0.0f;
    }
    asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the global scale is complete from here on
    if (global_ptr) global = __ldcg(global_ptr);
#pragma unroll
    for (int j = 0; j < QF_UNITS; j++) {
        const size_t u = u0 + 256 * j;
        float amax = max_abs8(v[j]);
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));  // 2 lanes = 16 elements
        const uint32_t sb = f32_to_ue4m3(amax / (6.0f * global)) & 0x7Fu;
        const float s = global * e4m3_to_f32(sb);
        uint32_t w = 0;
        if (s > 0.0f) {
            // v / s, correctly rounded: one reciprocal per lane and two of Markstein's corrections per element (the first makes
            // the quotient faithful, the second exact) where no step can leave the normal range
            float q[8];
            const bool fast = s > 1e-30f && s < 1e30f;
            const float y = fast ? __frcp_rn(s) : 0.0f;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float d = v[j][i] * y;
                d = fmaf(fmaf(-d, s, v[j][i]), y, d);
                q[i] = fmaf(fmaf(-d, s, v[j][i]), y, d);
            }
            if (fast && all_below(q, E2M1_FAST)) {
                w = e2m1x8(q);
            } else {
#pragma unroll
                for (int i = 0; i < 8; i++) q[i] = v[j][i] / s;
                w = e2m1x8_slow(q);
            }
        }
        if (u < units) {
            uint8_t *b = out + (u >> 3) * 36;
            *reinterpret_cast<uint32_t *>(b + 4 + 4 * (u & 7)) = w;
            if ((u & 1) == 0) b[(u & 7) >> 1] = (uint8_t)sb;
        }
    }
}

// ---- largest magnitude of a tensor (f32::max semantics: NaN is ignored) ---------------------------------------------
// Bound by reading x: 16-byte loads, eight in flight per thread; block maxima in the context's small device scratch, and the
// block that finishes last reduces them and writes what the next kernel needs, so no other launch lies in between.
// x [2048, 4096] from a cold cache: 11 us (25 us with 4-byte loads and an atomic maximum, 32 us with 4-byte loads and a
// second launch; without the last block's reduction 8 us, but then every block of the next kernel has to do it).
constexpr int AMAX_SEG = 8192;  // elements a block takes at a time
__global__ void __launch_bounds__(256) amax_kernel(const float *__restrict__ x, int64_t rows, int64_t k, int64_t ld, int vec, AmaxOut *out,
                                                   float *host_global) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    __shared__ float red[8];
    __shared__ int last_s;
    const int64_t segs = (k + AMAX_SEG - 1) / AMAX_SEG, units = rows * segs;
    float a = 0.0f;
    for (int64_t u = blockIdx.x; u < units; u += gridDim.x) {
        const int64_t r = u / segs, c0 = (u - r * segs) * AMAX_SEG;
        const float *src = x + r * ld + c0;
        const int n = (int)(k - c0 < AMAX_SEG ? k - c0 : AMAX_SEG);
        if (vec) {
            float4 v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int c = 4 * ((int)threadIdx.x + 256 * i);
                v[i] = c < n ? __ldg(reinterpret_cast<const float4 *>(src + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) a = fmaxf(fmaxf(a, fmaxf(fabsf(v[i].x), fabsf(v[i].y))), fmaxf(fabsf(v[i].z), fabsf(v[i].w)));
        } else {
#pragma unroll 8
            for (int c = threadIdx.x; c < n; c += 256) a = fmaxf(a, fabsf(src[c]));
        }
    }
    const auto block_max = [&]() {  // valid in thread 0
#pragma unroll
        for (int o = 16; o; o >>= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = a;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; i++) a = fmaxf(a, red[i]);
    };
    block_max();
    if (threadIdx.x == 0) {
        __stcg(out->part + blockIdx.x, a);
        __threadfence();
        last_s = atomicAdd(&out->arrived, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last_s) return;
    __threadfence();
    a = 0.0f;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += 256) a = fmaxf(a, __ldcg(out->part + i));
    __syncthreads();
    block_max();
    if (threadIdx.x == 0) {
        const float g = (a > 0.0f) ? a / (6.0f * 448.0f) : 1.0f;  // NVFP4's global scale, 1 when all zero
        out->arrived = 0;  // ready for the next launch
        out->amax = a;
        out->global = g;
        if (host_global) *reinterpret_cast<volatile float *>(host_global) = g;  // page-locked host memory
    }
}

int32_t amax_launch(Ctx *c, const float *x, int64_t rows, int64_t k, int64_t ld, float *host_global, cudaStream_t s) {
    const int vec = (((uintptr_t)x & 15) == 0 && ld % 4 == 0 && k % 4 == 0) ? 1 : 0;
    if (ld == k) k *= rows, rows = 1;  // contiguous rows are one long row
    const int64_t units = rows * ((k + AMAX_SEG - 1) / AMAX_SEG);
    amax_kernel<<<(unsigned)(units < AMAX_PARTS ? units : AMAX_PARTS), 256, 0, s>>>(x, rows, k, ld, vec, amax_out(c), host_global);
    GK_CUDA(c, cudaGetLastError());
    return GLLMK_STATUS_OK;
}

int32_t quantize_launch(Ctx *c, int32_t qt, const float *x, int64_t rows, int64_t k, int mx_block, void *blocks,
                        void *scales, float *global_scale, cudaStream_t s) {
    const size_t count = (size_t)rows * (size_t)k;
    if (qt == GLLMK_QUANT_Q4K) {
        const size_t nb = count / 256;
        quantize_q4k_kernel<<<(unsigned)((nb + 7) / 8), 256, 0, s>>>(x, (uint8_t *)blocks, nb);
    } else if (qt == GLLMK_QUANT_Q8_0) {
        const size_t nb = count / 32;
        quantize_q80_kernel<<<(unsigned)((nb + 7) / 8), 256, 0, s>>>(x, (uint8_t *)blocks, nb);
    } else if (qt == GLLMK_QUANT_MXFP4) {
        if (mx_block != 32) return fail(c, GLLMK_STATUS_UNSUPPORTED, "quantize: MXFP4 block_size %d (only 32)", mx_block);
        const size_t units = count / 8;
        quantize_mxfp4_kernel<<<(unsigned)((units + 256 * QF_UNITS - 1) / (256 * QF_UNITS)), 256, 0, s>>>(
            x, ((uintptr_t)x & 15) == 0, (uint32_t *)blocks, (uint8_t *)scales, units);
    } else if (qt == GLLMK_QUANT_NVFP4) {
        const bool given = *global_scale > 0.0f;
        if (!given) {
            int32_t rc = ensure_host_word(c);
            if (!rc) rc = amax_launch(c, x, 1, (int64_t)count, (int64_t)count, static_cast<float *>(c->host_word), s);
            if (rc) return rc;
        }
        const size_t units = count / 8;
        const unsigned grid = (unsigned)((units + 256 * QF_UNITS - 1) / (256 * QF_UNITS));
        const int vec = ((uintptr_t)x & 15) == 0;
        uint8_t *out = static_cast<uint8_t *>(blocks);
        if (given) quantize_nvfp4_kernel<<<grid, 256, 0, s>>>(x, vec, out, nullptr, *global_scale, units);
        else GK_CUDA(c, launch_after(quantize_nvfp4_kernel, true, dim3(grid), 256, 0, s, x, vec, out, &amax_out(c)->global, 0.0f, units));
        GK_CUDA(c, cudaGetLastError());
        if (!given) {
            // the call returns the scale, so it waits; and it waits for the blocks, not for the first pass alone: whoever holds the
            // scale may read them on any stream, and the encoder reads the context's small scratch, which the next call rewrites
            GK_CUDA(c, cudaEventRecord(c->host_word_ready, s));
            GK_CUDA(c, cudaEventSynchronize(c->host_word_ready));
            *global_scale = *static_cast<volatile float *>(c->host_word);
        }
    } else {
        return fail(c, GLLMK_STATUS_UNSUPPORTED, "quantize: unknown quant type %d", qt);
    }
    GK_CUDA(c, cudaGetLastError());
    return GLLMK_STATUS_OK;
}

}  // namespace gllmk
