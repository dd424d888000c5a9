// NVFP4 quantisation arithmetic shared by the stand-alone quantiser (act_quant.cu) and the fused linear's own
// activation prologue (slab_kernel.cuh). Every step is one IEEE fp32 operation, so a CPU restatement matches bit for bit:
//     t    = bmax / gs                      per 16-element block
//     sfD  = e4m3_rn_sat(t / D)             D = 6 or 4
//     d    = f32(sfD) * gs
//     code = e2m1_rn(x / d)                 round-to-nearest-even on {0,.5,1,1.5,2,3,4,6}, saturating; 0 if d == 0, sign only if x is NaN
//     mse rule: err_D = sum_{j=0..15} (x_j - value(code_j) * d)^2 in index order (separate multiply and add);
//               the block takes D = 4 iff err_4 < err_6.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

namespace biloco {
namespace qm {

__device__ __forceinline__ uint32_t e2m1_rn(float q) {
    const float a = fabsf(q);
    uint32_t c = (a > 0.25f) + (a >= 0.75f) + (a > 1.25f) + (a >= 1.75f) + (a > 2.5f) + (a >= 3.5f) + (a > 5.0f);
    return c | ((__float_as_uint(q) >> 31) << 3);
}
__device__ __forceinline__ float e2m1_value(uint32_t code) {
    const uint32_t m = code & 7u;
    // 0, .5, 1, 1.5, 2, 3, 4, 6
    const float mag = m < 4u ? 0.5f * (float)m : (m == 4u ? 2.0f : (m == 5u ? 3.0f : (m == 6u ? 4.0f : 6.0f)));
    return (code & 8u) ? -mag : mag;
}
__device__ __forceinline__ float e4m3_to_float(uint8_t b) {
    const __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)b, __NV_E4M3);
    return __half2float(__half(h));
}
__device__ __forceinline__ uint8_t float_to_e4m3_sat(float v) {
    return (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
}

// bf16 pair -> two floats, optionally divided by the smoothing pair and rounded back to bf16
__device__ __forceinline__ void unpack_smoothed(uint32_t w, uint32_t sm, bool smooth, float& lo, float& hi) {
    lo = __uint_as_float(w << 16);
    hi = __uint_as_float(w & 0xFFFF0000u);
    if (smooth) {
        lo = __bfloat162float(__float2bfloat16_rn(__fdiv_rn(lo, __uint_as_float(sm << 16))));
        hi = __bfloat162float(__float2bfloat16_rn(__fdiv_rn(hi, __uint_as_float(sm & 0xFFFF0000u))));
    }
}

// One element per lane, sixteen lanes per block (lanes 0-15 and 16-31 of a warp hold one block each, all 32 lanes must
// call): the block-wide steps -- maximum, the squared errors summed in index order, packing -- go through shuffles.
// Returns in the block's first lane (lane % 16 == 0) the eight bytes of codes (element 2i in bits 0-3 of byte i) and the
// block's E4M3 scale. rule: 0 static_6, 1 static_4, 2 mse.
__device__ __forceinline__ void quant_lane16(float x, int lane, float gs, int rule, uint2& codes, uint8_t& sf) {
    const int base = lane & 16;
    float bmax = fabsf(x);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, o));
    const float t = __fdiv_rn(bmax, gs);
    uint32_t c6 = 0, c4 = 0;
    uint8_t s6 = 0, s4 = 0;
    float e6 = 0.f, e4 = 0.f;
#pragma unroll
    for (int cand = 0; cand < 2; ++cand) {
        if (cand == 0 && rule == 1) continue;
        if (cand == 1 && rule == 0) continue;
        const uint8_t sfv = float_to_e4m3_sat(__fdiv_rn(t, cand == 0 ? 6.0f : 4.0f));
        const float d = __fmul_rn(e4m3_to_float(sfv), gs);
        const uint32_t c = d > 0.f ? e2m1_rn(__fdiv_rn(x, d)) : 0u;
        float err = 0.f;
        if (rule == 2) {
            const float diff = __fsub_rn(x, __fmul_rn(e2m1_value(c), d));
            const float sq = __fmul_rn(diff, diff);
#pragma unroll
            for (int i = 0; i < 16; ++i) err = __fadd_rn(err, __shfl_sync(0xffffffffu, sq, base + i));   // index order
        }
        if (cand == 0) { c6 = c; s6 = sfv; e6 = err; } else { c4 = c; s4 = sfv; e4 = err; }
    }
    uint32_t code;
    if (rule == 0 || (rule == 2 && !(e4 < e6))) { code = c6; sf = s6; } else { code = c4; sf = s4; }
    // pack: two codes per byte, four bytes per word; the words of elements 0-7 and 8-15 end up in lanes base and base + 8
    uint32_t w = code | (__shfl_down_sync(0xffffffffu, code, 1) << 4);
    w |= (__shfl_down_sync(0xffffffffu, w, 2) << 8) | (__shfl_down_sync(0xffffffffu, w, 4) << 16) |
         (__shfl_down_sync(0xffffffffu, w, 6) << 24);
    codes = make_uint2(w, __shfl_down_sync(0xffffffffu, w, 8));
}

// Eight floats -> eight E2M1 codes (element i in bits 4i .. 4i+3), round to nearest even, saturating: the hardware conversion.
__device__ __forceinline__ uint32_t e2m1_pack8(const float* q) {
    uint32_t w;
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\tcvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\tcvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
        "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
        : "=r"(w) : "f"(q[0]), "f"(q[1]), "f"(q[2]), "f"(q[3]), "f"(q[4]), "f"(q[5]), "f"(q[6]), "f"(q[7]));
    return w;
}
__device__ __forceinline__ void e2m1_unpack8(uint32_t w, float* v) {
    uint32_t h[4];
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\tmov.b32 {b0, b1, b2, b3}, %4;\n\t"
        "cvt.rn.f16x2.e2m1x2 %0, b0;\n\tcvt.rn.f16x2.e2m1x2 %1, b1;\n\tcvt.rn.f16x2.e2m1x2 %2, b2;\n\tcvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
        : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3]) : "r"(w));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h[i]));
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}

// The larger of two values; NaN if either is (fmaxf drops it).
__device__ __forceinline__ float max_nan(float a, float b) {
    float m;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
    return m;
}

// Half a block (eight bf16 values) that holds a NaN: the largest of the other elements, and what the conversion instructions would
// make 6 -- the code of a NaN element is its sign bit over zero. `keep` has the other elements' nibbles, `sign` the NaN elements' sign
// bits. Out of line: inlined, this rare path cost the prompt's quantiser 1.5 us at 96 rows of 5120.
struct NanHalf { float bmax; uint32_t keep, sign; };
static __device__ __noinline__ NanHalf nan_half(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
    NanHalf n = {0.f, 0xffffffffu, 0u};
    const uint32_t w[4] = {w0, w1, w2, w3};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float x = __uint_as_float((j & 1) ? w[j >> 1] & 0xFFFF0000u : w[j >> 1] << 16);
        n.bmax = fmaxf(n.bmax, fabsf(x));
        if (x != x) { n.keep &= ~(15u << (4 * j)); n.sign |= (__float_as_uint(x) >> 31) << (4 * j + 3); }
    }
    return n;
}
__device__ __forceinline__ NanHalf nan_half(const float* x) {      // (bf16 values)
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = (__float_as_uint(x[2 * e]) >> 16) | (__float_as_uint(x[2 * e + 1]) & 0xFFFF0000u);
    return nan_half(w[0], w[1], w[2], w[3]);
}

// Codes e2m1_rn(x_j / d) of half a block. The quotients are not formed: x_j times the reciprocal, made 2^-20 smaller and 2^-20
// larger (more than the few 2^-24 the product can be off by), gives the same code both ways unless the quotient lies at a
// rounding boundary; only then (about one half block in 12000 on random data) are the IEEE quotients taken.
__device__ __forceinline__ uint32_t codes8(const float* x, float d, uint32_t keep, uint32_t sign) {
    if (!(d > 0.f)) return 0u;
    float q[8];
    if (d > 1e-30f && d < 1e30f) {
        const float r = __frcp_rn(d), rl = r * (1.0f - 9.5367431640625e-7f), rh = r * (1.0f + 9.5367431640625e-7f);
#pragma unroll
        for (int j = 0; j < 8; ++j) q[j] = x[j] * rl;
        const uint32_t lo = e2m1_pack8(q);
#pragma unroll
        for (int j = 0; j < 8; ++j) q[j] = x[j] * rh;
        if (lo == e2m1_pack8(q)) return (lo & keep) | sign;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) q[j] = __fdiv_rn(x[j], d);
    return (e2m1_pack8(q) & keep) | sign;
}

// One thread, one block of sixteen values (the throughput form: thousands of blocks): the arithmetic of the file header.
// KEEP_NAN (weights): a NaN makes the block's maximum and with it its scale NaN (0x7f, codes 0), and a tensor scale that is not
// positive gives a scale of zero, as torch's maximum and clamp have it. Otherwise (activations) the block's maximum and the codes leave NaN elements out.
template <bool KEEP_NAN>
__device__ __forceinline__ void quant_block16(const float (&x)[16], float gs, int rule, uint2& codes, uint8_t& sf) {
    float bmax = 0.f;
    uint32_t keep[2] = {0xffffffffu, 0xffffffffu}, sign[2] = {0u, 0u};
#pragma unroll
    for (int j = 0; j < 16; ++j) bmax = max_nan(bmax, fabsf(x[j]));
    if (!KEEP_NAN && bmax != bmax) {
        const NanHalf l = nan_half(x), h = nan_half(x + 8);
        bmax = fmaxf(l.bmax, h.bmax);
        keep[0] = l.keep; keep[1] = h.keep; sign[0] = l.sign; sign[1] = h.sign;
    }
    float t = __fdiv_rn(bmax, gs);
    if (KEEP_NAN && t <= 0.f) t = 0.f;
    uint2 c[2];
    uint8_t s[2] = {0, 0};
    float e[2] = {0.f, 0.f};
#pragma unroll
    for (int cand = 0; cand < 2; ++cand) {
        if (cand == 0 && rule == 1) continue;
        if (cand == 1 && rule == 0) continue;
        s[cand] = float_to_e4m3_sat(__fdiv_rn(t, cand == 0 ? 6.0f : 4.0f));
        const float d = __fmul_rn(e4m3_to_float(s[cand]), gs);
        c[cand] = make_uint2(codes8(x, d, keep[0], sign[0]), codes8(x + 8, d, keep[1], sign[1]));
        if (rule == 2) {
            float v[16];
            e2m1_unpack8(c[cand].x, v);
            e2m1_unpack8(c[cand].y, v + 8);
            float err = 0.f;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float diff = __fsub_rn(x[j], __fmul_rn(v[j], d));
                err = __fadd_rn(err, __fmul_rn(diff, diff));
            }
            e[cand] = err;
        }
    }
    const bool four = rule == 1 || (rule == 2 && e[1] < e[0]);
    codes = four ? c[1] : c[0];
    sf = four ? s[1] : s[0];
}

}  // namespace qm
}  // namespace biloco
