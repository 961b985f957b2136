// One cache row (one token of one kv head) through the append arithmetic, with the row spread over a warp:
// lane L holds elements L, L+32, L+64, ...  Shared by the append kernel and by the decode kernel's fused
// single-token append, so both write bit-identical rows.  Arithmetic follows MIInfer's store kernel
// (gfx906/kernels/qwen3_primitives.hip:7257-7300): K RMSNorm -> RoPE -> amax/127 scale -> round-half-even
// int8, every step with explicit IEEE operations (no fused contraction) so a host restatement reproduces the bits.
#pragma once

#include "kv_common.cuh"

namespace b200kv {

// The rotation of every pair a lane holds (NeoX: registers j and j + NJ/2; sectioned: registers 0 and 1).  It depends on the
// position alone, so a caller that knows the position ahead of the row computes it while it waits for the row.
template <int D>
struct Rotation { float sn[D / 64], cs[D / 64]; };
template <int D>
__device__ __forceinline__ void row_rotation(Rotation<D>& r, int lane, uint32_t position, int rope_mode, const float* inv_freq, float sectioned_step) {
    if (rope_mode == B200KV_ROPE_NEOX_FULL) {
#pragma unroll
        for (int j = 0; j < D / 64; ++j) sincos_pinned(__fmul_rn(static_cast<float>(position), inv_freq[lane + 32 * j]), &r.sn[j], &r.cs[j]);
    } else if (rope_mode == B200KV_ROPE_SECTIONED64) {
        float angle = static_cast<float>(position);
#pragma unroll 8
        for (int i = 0; i < 32; ++i) angle = i < lane ? __fmul_rn(angle, sectioned_step) : angle;   // as many products as the lane's number, no branch per product
        sincos_pinned(angle, &r.sn[0], &r.cs[0]);
    }
}

// A lane's norm weights, fetched ahead of the row's arithmetic (in the middle of it they were a trip to L2 of their own).
template <int D>
__device__ __forceinline__ void load_norm_weight(const float* k_norm_weight, int lane, float (&w)[D / 32]) {
#pragma unroll
    for (int j = 0; j < D / 32; ++j) w[j] = k_norm_weight != nullptr ? k_norm_weight[lane + 32 * j] : 1.0f;
}

// K side before quantization: optional RMSNorm * weight, then RoPE.
template <int D>
__device__ __forceinline__ void transform_k_row(float (&k)[D / 32], int lane, bool norm, const float (&w)[D / 32], float epsilon, int rope_mode,
                                                const Rotation<D>& r) {
    constexpr int NJ = D / 32;
    if (norm) {
        // the reference's shared-memory tree (stride D/2 .. 1) as register adds + a shuffle-down tree over the same pairs
        float sq[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) sq[j] = __fmul_rn(k[j], k[j]);
#pragma unroll
        for (int half = NJ / 2; half >= 1; half >>= 1)
#pragma unroll
            for (int j = 0; j < half; ++j) sq[j] = __fadd_rn(sq[j], sq[j + half]);
        float ss = sq[0];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss = __fadd_rn(ss, __shfl_down_sync(0xffffffffu, ss, o));
        ss = __shfl_sync(0xffffffffu, ss, 0);
        const float rms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, static_cast<float>(D)), epsilon)));
#pragma unroll
        for (int j = 0; j < NJ; ++j) k[j] = __fmul_rn(__fmul_rn(k[j], rms), w[j]);
    }
    if (rope_mode == B200KV_ROPE_NEOX_FULL) {
#pragma unroll
        for (int j = 0; j < NJ / 2; ++j) {
            const float x0 = k[j], x1 = k[j + NJ / 2];
            k[j] = __fsub_rn(__fmul_rn(x0, r.cs[j]), __fmul_rn(x1, r.sn[j]));
            k[j + NJ / 2] = __fadd_rn(__fmul_rn(x0, r.sn[j]), __fmul_rn(x1, r.cs[j]));
        }
    } else if (rope_mode == B200KV_ROPE_SECTIONED64) {
        const float x0 = k[0], x1 = k[1];
        k[0] = __fsub_rn(__fmul_rn(x0, r.cs[0]), __fmul_rn(x1, r.sn[0]));
        k[1] = __fadd_rn(__fmul_rn(x0, r.sn[0]), __fmul_rn(x1, r.cs[0]));
    }
}

__device__ __forceinline__ int quantize_s8(float v) {
    // round to nearest even and saturate to [-128, 127] (NaN -> 0): __float2int_rn followed by the clamp, in one step
    int q;
    asm("cvt.rni.sat.s8.f32 %0, %1;" : "=r"(q) : "f"(v));
    return q;
}
// max over the warp of non-negative floats (NaN counts as 0, as with fmaxf): one redux on the bit patterns
__device__ __forceinline__ float warp_amax(float a) {
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(a, 0.0f))));
}

// Quantizer: q[j] is this lane's int8 of block j (or of the row); returns the fp32 scale of block `lane` (lanes below NJ;
// row_scale: of the row, every lane).  The cache stores __float2half_rn of it.  Each IEEE division is taken by one lane.
template <int NJ>
__device__ __forceinline__ float quantize_row(const float (&x)[NJ], bool row_scale, int lane, int (&q)[NJ]) {
    float amax_mine = 0.0f;
    if (row_scale) {
        float amax = 0.0f;
#pragma unroll
        for (int j = 0; j < NJ; ++j) amax = fmaxf(amax, fabsf(x[j]));
        amax_mine = warp_amax(amax);
    } else {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const float amax = warp_amax(fabsf(x[j]));
            if (lane == j) amax_mine = amax;
        }
    }
    const float scale = (amax_mine > 0.0f) ? __fdiv_rn(amax_mine, 127.0f) : 1.0f;
    const float inv_mine = (scale > 0.0f) ? __fdiv_rn(1.0f, scale) : 1.0f;
#pragma unroll
    for (int j = 0; j < NJ; ++j) q[j] = quantize_s8(__fmul_rn(x[j], row_scale ? inv_mine : __shfl_sync(0xffffffffu, inv_mine, j)));
    return scale;
}

}  // namespace b200kv
