// Fused KV append: (optional K RMSNorm) -> RoPE on K -> int8 quantization with
// fp16 block scales (or fp16 passthrough) -> cache write, for K and V of every
// (token, kv_head) row in one launch.
//
// Behaviour follows MIInfer's store kernel
// (gfx906/kernels/qwen3_primitives.hip:7213-7326): same operation order, same
// quantizer, positions optionally read from device-resident state.  The mapping
// is new: the unit of work is 1024 elements of K or of V of one token -- eight kv heads at head_dim 128, four at 256, 32
// q8_0 blocks -- and every warp of a grid sized to the device takes one contiguous run of units.
//   - The next unit's input is fetched into registers as it lies (16 of them for fp16) before the arithmetic of the current one.
//   - D/8 lanes hold a row, lane l of them elements 4l .. 4l+3 and D/2 + 4l .. D/2 + 4l+3: NeoX pairs (i, i + d/2) lie in
//     one lane, sectioned pairs (i, i + 32) eight lanes apart, and every store is four bytes of int8 per lane.
//   - The reference's shared-memory binary tree for the sum of squares (stride d/2 .. 1) becomes one register add and a
//     butterfly that adds exactly the same pairs (addition commutes: identical bits); each exchange halves the values a
//     lane carries.
//   - The 32 block maxima are reduced the same way, eight values over eight lanes in seven shuffles, and come out one
//     block per lane -- so each IEEE division (scale, reciprocal, 1/rms) is taken once, by one lane.
//   - The sines and cosines depend on the token only; they are computed while the unit's data is in flight.
//   - Products run two to an instruction (f32x2), four int8 are packed by two cvt.pack.
// Bound by instruction issue (half of all issue slots at 8192 tokens; the writes stay in L2): 8192 tokens x 8 heads of 128
// dims, fp16 to q8_0, take 17.1 us.  A layout with lanes 32 elements apart, element-wise K accesses and one redux per block
// took 21.8 us; this layout with its input in a cp.async ring 20.0 us alone, and its shared memory kept the next
// layer's launch off SMs that still held attention CTAs (4 us a layer).
// The row arithmetic is the same, operation for operation, as append_row.cuh's (used by the decode kernel's fused
// single-token append and the query-side kernel): all three write identical bits.
#include "append_row.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace b200kv {

struct AppendParams {
    b200kv_view view;
    const void* key;
    const void* value;
    const float* k_norm_weight;
    const b200kv_prefill_state* prefill_state;
    const b200kv_decode_state* decode_state;
    uint32_t token_count;
    uint32_t base_position;
    int rope_mode;
    float epsilon;
    float sectioned_step;    // powf(theta, -2/64)
    float inv_freq[128];     // NeoX: powf(theta, -2i/d), i < d/2
    // Dependents come in behind this kernel's wait (kv_common.cuh), or at once where its CTAs take every slot of the device: no CTA of
    // a decode kernel, several times the size of one of these, can then start before one of these has gone, and none goes
    // before the wait.  (12 launches of 8192 tokens: 205 us so, 216 behind the wait.)
    int fills_device;
};

constexpr int kAppendWarps = 2;
constexpr int kUnitElems = 1024;       // 32 q8_0 blocks: one scale per lane
template <bool IN_F16>
constexpr int kAppendCtasPerSm = IN_F16 ? 10 : 8;   // 20 warps of 96 registers: a unit, the next one's raw input and the rotation (fp32 input: 16 of 128);
                                                    // head_dim 256 with fp16 input spills 8 bytes of them

// Two fp32 products in one instruction (.ftz as the scalar intrinsics under this build).
__device__ __forceinline__ Pair mul2(Pair a, Pair b) { Pair r; asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
// Sums of products are taken one at a time: an f32x2 add behind an f32x2 multiply came out contracted (measured: single
// fp16 results one unit off the oracle's), the scalar intrinsics never are.
__device__ __forceinline__ Pair add_products(Pair t, Pair u) {
    const float2 a = unpack_pair(t), b = unpack_pair(u);
    return pack_pair(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}
__device__ __forceinline__ Pair sub_products(Pair t, Pair u) {
    const float2 a = unpack_pair(t), b = unpack_pair(u);
    return pack_pair(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y));
}

// Four consecutive input elements as they lie in memory, and as two pairs of floats.
template <bool IN_F16> struct Raw4 { uint2 v; };
template <> struct Raw4<false> { float4 v; };
template <bool IN_F16>
__device__ __forceinline__ Raw4<IN_F16> load4(const void* src, size_t element, bool vec) {
    Raw4<IN_F16> r;
    if constexpr (IN_F16) {
        const __half* s = static_cast<const __half*>(src) + element;
        if (vec) {
            r.v = *reinterpret_cast<const uint2*>(s);
        } else {
            const uint16_t* u = reinterpret_cast<const uint16_t*>(s);
            r.v = make_uint2(u[0] | (static_cast<uint32_t>(u[1]) << 16), u[2] | (static_cast<uint32_t>(u[3]) << 16));
        }
    } else {
        const float* s = static_cast<const float*>(src) + element;
        r.v = vec ? *reinterpret_cast<const float4*>(s) : make_float4(s[0], s[1], s[2], s[3]);
    }
    return r;
}
template <bool IN_F16>
__device__ __forceinline__ void widen(const Raw4<IN_F16>& r, Pair (&x)[2]) {
    if constexpr (IN_F16) {
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.v.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&r.v.y));
        x[0] = pack_pair(a.x, a.y); x[1] = pack_pair(b.x, b.y);
    } else {
        x[0] = pack_pair(r.v.x, r.v.y); x[1] = pack_pair(r.v.z, r.v.w);
    }
}
__device__ __forceinline__ float amax4(const Pair (&x)[2]) {
    const float2 a = unpack_pair(x[0]), b = unpack_pair(x[1]);
    return fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y))), 0.0f);   // a NaN counts as 0, as in warp_amax
}
// round to nearest even, saturate to [-128, 127], NaN -> 0: quantize_s8 on four values, packed
__device__ __forceinline__ uint32_t quantize4(const Pair (&x)[2], float inv) {
    const Pair inv2 = pack_pair(inv, inv);
    const float2 a = unpack_pair(mul2(x[0], inv2)), b = unpack_pair(mul2(x[1], inv2));
    uint32_t w;
    asm("{ .reg .b32 t; cvt.pack.sat.s8.s32.b32 t, %4, %3, 0; cvt.pack.sat.s8.s32.b32 %0, %2, %1, t; }"
        : "=r"(w) : "r"(__float2int_rn(a.x)), "r"(__float2int_rn(a.y)), "r"(__float2int_rn(b.x)), "r"(__float2int_rn(b.y)));
    return w;
}
__device__ __forceinline__ uint2 half4(const Pair (&x)[2]) {
    const float2 a = unpack_pair(x[0]), b = unpack_pair(x[1]);
    const __half2 lo = __floats2half2_rn(a.x, a.y), hi = __floats2half2_rn(b.x, b.y);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

template <int D, bool IN_F16>
__global__ void __launch_bounds__(kAppendWarps * 32, kAppendCtasPerSm<IN_F16>)
append_kernel(const __grid_constant__ AppendParams p, const bool vec) {
    constexpr int LPR = D / 8;                  // lanes per row
    constexpr int RPS = 32 / LPR;               // rows per step
    constexpr int HB = kUnitElems / D;          // kv heads per unit, four steps
    constexpr int NB = D / 32;                  // q8_0 blocks per row
    static_assert(HB == 4 * RPS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int l = lane & (LPR - 1), sub = lane / LPR;          // lane of the row, row of the step
    const int rope_mode = p.rope_mode;
    // NeoX: the lane rotates pairs 4l .. 4l+3; the two rows of a step at head_dim 128 share them, so each of their lanes
    // evaluates two and fetches the other two
    constexpr int SC = 4 / RPS;
    float freq[SC];
    if (rope_mode == B200KV_ROPE_NEOX_FULL)
#pragma unroll
        for (int i = 0; i < SC; ++i) freq[i] = p.inv_freq[4 * l + SC * sub + i];
    if (p.fills_device) pdl_launch_dependents();   // the next kernel may become resident; it orders itself against this one
    pdl_wait();                // K/V inputs and the device-side position come from preceding kernels

    uint32_t base_position = p.base_position;
    uint32_t token_count = p.token_count;
    uint64_t capacity = p.view.capacity;
    if (p.prefill_state != nullptr) {
        base_position = p.prefill_state->base_position;
        token_count = min(token_count, p.prefill_state->token_count);
        if (p.prefill_state->kv_capacity > 0) capacity = p.prefill_state->kv_capacity;
    } else if (p.decode_state != nullptr) {
        base_position = p.decode_state->position;
        token_count = min(token_count, 1u);
    }
    const uint32_t H = p.view.kv_heads;
    const uint32_t mode = p.view.quant_mode;
    const bool k_q8 = (mode == B200KV_Q8_F16 || mode == B200KV_Q8_Q8);
    const bool v_q8 = (mode == B200KV_F16_Q8 || mode == B200KV_Q8_Q8);
    const bool row_scale = p.view.qblock == D;
    const bool have_norm = p.k_norm_weight != nullptr;

    // Units in the order token, pass (HB heads), side (K, V).  (32-bit arithmetic: the host keeps units below 2^32.)
    const uint32_t passes = (H + HB - 1) / HB;
    const uint32_t total_units = token_count * passes * 2;
    const uint32_t warps = gridDim.x * kAppendWarps;
    const uint32_t per_warp = (total_units + warps - 1) / warps;
    const uint32_t unit0 = min(total_units, (blockIdx.x * kAppendWarps + warp) * per_warp);
    const uint32_t unit1 = min(total_units, unit0 + per_warp);

    struct Cursor { uint32_t token, pass, side; };
    auto advance = [&](Cursor& c) {
        if (++c.side == 2) {
            c.side = 0;
            if (++c.pass == passes) { c.pass = 0; ++c.token; }
        }
    };
    auto inside = [&](const Cursor& c) { return static_cast<uint64_t>(base_position) + c.token < capacity; };   // never write outside the cache
    auto heads = [&](const Cursor& c) { return static_cast<int>(min(static_cast<uint32_t>(HB), H - c.pass * HB)); };
    Raw4<IN_F16> raw[4][2];   // per step: elements 4l .. and D/2 + 4l .. of the unit that comes next
    auto fetch = [&](const Cursor& c) {
        const void* src = c.side == 0 ? p.key : p.value;
        const size_t e0 = (static_cast<size_t>(c.token) * H + c.pass * HB + sub) * D + 4 * l;
        const int hn = heads(c);
#pragma unroll
        for (int s = 0; s < 4; ++s)
            if (s * RPS + sub < hn) {
                raw[s][0] = load4<IN_F16>(src, e0 + s * RPS * D, vec);
                raw[s][1] = load4<IN_F16>(src, e0 + s * RPS * D + D / 2, vec);
            } else {
                raw[s][0] = raw[s][1] = Raw4<IN_F16>{};
            }
    };

    Pair sn[2], cs[2];   // NeoX: pairs 4l + i; sectioned: pairs 4 (l % 8) + i
    auto rotation = [&](uint32_t position) {
        if (rope_mode == B200KV_ROPE_NEOX_FULL) {
            float s[SC], c[SC];
#pragma unroll
            for (int i = 0; i < SC; ++i) sincos_pinned(__fmul_rn(static_cast<float>(position), freq[i]), &s[i], &c[i]);
            if constexpr (RPS == 1) {
                sn[0] = pack_pair(s[0], s[1]); sn[1] = pack_pair(s[2], s[3]);
                cs[0] = pack_pair(c[0], c[1]); cs[1] = pack_pair(c[2], c[3]);
            } else {
                const Pair sm = pack_pair(s[0], s[1]), cm = pack_pair(c[0], c[1]);
                const Pair so = __shfl_xor_sync(0xffffffffu, sm, 16), co = __shfl_xor_sync(0xffffffffu, cm, 16);
                sn[0] = sub ? so : sm; sn[1] = sub ? sm : so;
                cs[0] = sub ? co : cm; cs[1] = sub ? cm : co;
            }
        } else if (rope_mode == B200KV_ROPE_SECTIONED64) {
            float angle = static_cast<float>(position), s, c;
            for (int i = 0; i < lane; ++i) angle = __fmul_rn(angle, p.sectioned_step);
            sincos_pinned(angle, &s, &c);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int src = 4 * (lane & 7) + 2 * i;
                sn[i] = pack_pair(__shfl_sync(0xffffffffu, s, src), __shfl_sync(0xffffffffu, s, src + 1));
                cs[i] = pack_pair(__shfl_sync(0xffffffffu, c, src), __shfl_sync(0xffffffffu, c, src + 1));
            }
        }
    };

    // FAST: a full unit (hn == HB) of a q8_0 side -- every check is decided at compile time.  Rows of a ragged unit that do
    // not exist came in as zeros and are only not stored.
    auto process = [&](auto fast_c, const Cursor& cur, Pair (&a)[4][2], Pair (&b)[4][2], uint64_t position, int hn) {
        constexpr bool FAST = decltype(fast_c)::value;
        if constexpr (FAST) hn = HB;
        const bool is_k = cur.side == 0;
        const bool quantised = FAST || (is_k ? k_q8 : v_q8), rows = !FAST && row_scale;
        if (is_k) {
            if (have_norm) {
                float ss_mine = 0.0f;
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const bool up2 = lane & (LPR / 2), up1 = lane & (LPR / 4);
                    const Pair q01 = add_products(mul2(a[s][0], a[s][0]), mul2(b[s][0], b[s][0])), q23 = add_products(mul2(a[s][1], a[s][1]), mul2(b[s][1], b[s][1]));   // stride D/2
                    const float2 t = unpack_pair(add_products(up2 ? q23 : q01, __shfl_xor_sync(0xffffffffu, up2 ? q01 : q23, LPR / 2)));                                // stride D/4
                    float ss = __fadd_rn(up1 ? t.y : t.x, __shfl_xor_sync(0xffffffffu, up1 ? t.x : t.y, LPR / 4));                                        // stride D/8
#pragma unroll
                    for (int o = LPR / 8; o > 0; o >>= 1) ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, o));                                        // down to stride 4
                    ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, LPR / 2));                                                                        // stride 2
                    ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, LPR / 4));                                                                        // stride 1
                    if ((lane & 3) == s) ss_mine = ss;
                }
                const float r_mine = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss_mine, static_cast<float>(D)), p.epsilon)));
                Pair w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float* src = p.k_norm_weight + (i >> 1) * (D / 2) + 4 * l + 2 * (i & 1);
                    w[i] = pack_pair(src[0], src[1]);
                }
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const float r = __shfl_sync(0xffffffffu, r_mine, (lane & ~3) | s);
                    const Pair r2 = pack_pair(r, r);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        a[s][i] = mul2(mul2(a[s][i], r2), w[i]);
                        b[s][i] = mul2(mul2(b[s][i], r2), w[2 + i]);
                    }
                }
            }
            if (rope_mode == B200KV_ROPE_NEOX_FULL) {
#pragma unroll
                for (int s = 0; s < 4; ++s)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const Pair x0 = a[s][i], x1 = b[s][i];
                        a[s][i] = sub_products(mul2(x0, cs[i]), mul2(x1, sn[i]));
                        b[s][i] = add_products(mul2(x0, sn[i]), mul2(x1, cs[i]));
                    }
            } else if (rope_mode == B200KV_ROPE_SECTIONED64) {
                // elements 0-31 lie in lanes 0-7 of the row (x0 cos - x1 sin), 32-63 in lanes 8-15 (x0 sin + x1 cos)
                const bool second = lane & 8;
#pragma unroll
                for (int s = 0; s < 4; ++s)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const Pair other = __shfl_xor_sync(0xffffffffu, a[s][i], 8);
                        const Pair t = mul2(a[s][i], cs[i]), u = mul2(other, sn[i]);
                        if (l < 16) a[s][i] = second ? add_products(u, t) : sub_products(t, u);
                    }
            }
        }
        const uint64_t row0 = (static_cast<uint64_t>(cur.pass) * HB + sub) * capacity + position;   // this lane's cache row of step 0; the next step's is RPS * capacity on
        if (!quantised) {
            __half* dst = static_cast<__half*>(is_k ? p.view.key_f16 : p.view.value_f16) + row0 * D + 4 * l;
#pragma unroll
            for (int s = 0; s < 4; ++s, dst += RPS * capacity * D) {
                if (s * RPS + sub >= hn) break;
                *reinterpret_cast<uint2*>(dst) = half4(a[s]);
                *reinterpret_cast<uint2*>(dst + D / 2) = half4(b[s]);
            }
            return;
        }
        // ---- block maxima: values 2s (elements below D/2) and 2s + 1, over the eight lanes of a block; lane keeps value lane % 8.
        float m[8];
#pragma unroll
        for (int s = 0; s < 4; ++s) { m[2 * s] = amax4(a[s]); m[2 * s + 1] = amax4(b[s]); }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < o; ++i) m[i] = fmaxf(up ? m[i + o] : m[i], __shfl_xor_sync(0xffffffffu, up ? m[i] : m[i + o], o));
        }
        float amax = m[0];
        if (rows) {
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
#pragma unroll
            for (int o = 8; o < LPR; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        }
        // ---- scales: amax / 127, its reciprocal, the fp16 scale to the cache -- one block per lane
        const float scale = (amax > 0.0f) ? __fdiv_rn(amax, 127.0f) : 1.0f;
        const float inv_mine = (scale > 0.0f) ? __fdiv_rn(1.0f, scale) : 1.0f;
        {
            const int s = (lane & 7) >> 1, block = (lane & 1) * (NB / 2) + (l >> 3);
            __half* plane = static_cast<__half*>(is_k ? p.view.key_scales : p.view.value_scales);
            const uint64_t r = row0 + s * RPS * capacity;
            if (s * RPS + sub < hn && (!rows || block == 0)) plane[rows ? r : r * NB + block] = __float2half_rn(scale);
        }
        int8_t* dst = (is_k ? p.view.key_q8 : p.view.value_q8) + row0 * D + 4 * l;
#pragma unroll
        for (int s = 0; s < 4; ++s, dst += RPS * capacity * D) {
            const float inv_a = __shfl_sync(0xffffffffu, inv_mine, (lane & 24) | (2 * s)), inv_b = __shfl_sync(0xffffffffu, inv_mine, (lane & 24) | (2 * s + 1));
            const uint32_t wa = quantize4(a[s], inv_a), wb = quantize4(b[s], inv_b);
            if (FAST || s * RPS + sub < hn) {
                *reinterpret_cast<uint32_t*>(dst) = wa;
                *reinterpret_cast<uint32_t*>(dst + D / 2) = wb;
            }
        }
    };

    Cursor cur{unit0 / (2 * passes), (unit0 / 2) % passes, unit0 & 1};
    if (unit0 < unit1 && inside(cur)) fetch(cur);
    if (!p.fills_device) pdl_launch_dependents();
    uint32_t rotated_token = 0xffffffffu;
    for (uint32_t unit = unit0; unit < unit1; ++unit) {
        const uint64_t position = static_cast<uint64_t>(base_position) + cur.token;
        if (cur.side == 0 && cur.token != rotated_token) {
            rotated_token = cur.token;
            rotation(static_cast<uint32_t>(position));
        }
        Pair a[4][2], b[4][2];
#pragma unroll
        for (int s = 0; s < 4; ++s) { widen<IN_F16>(raw[s][0], a[s]); widen<IN_F16>(raw[s][1], b[s]); }
        Cursor next = cur;
        advance(next);
        if (unit + 1 < unit1 && inside(next)) fetch(next);   // under this unit's arithmetic
        if (inside(cur)) {
            const int hn = heads(cur);
            if (!row_scale && hn == HB && (cur.side == 0 ? k_q8 : v_q8)) process(std::true_type{}, cur, a, b, position, hn);
            else process(std::false_type{}, cur, a, b, position, hn);
        }
        cur = next;
    }
}

}  // namespace b200kv

using namespace b200kv;

extern "C" int b200kv_append(const b200kv_view* view, const void* key, const void* value, int dtype,
                             const float* k_norm_weight, int rope_mode, float theta, float epsilon,
                             uint32_t token_count, uint32_t base_position,
                             const b200kv_prefill_state* prefill_state, const b200kv_decode_state* decode_state,
                             void* stream) {
    int rc = validate_view(view);
    if (rc != B200KV_OK) return rc;
    if (key == nullptr || value == nullptr || (dtype != B200KV_F16 && dtype != B200KV_F32)) return B200KV_ERR_INVALID;
    if (rope_mode < B200KV_ROPE_NONE || rope_mode > B200KV_ROPE_SECTIONED64) return B200KV_ERR_INVALID;
    if (!std::isfinite(theta) || !std::isfinite(epsilon)) return B200KV_ERR_INVALID;
    if (rope_mode != B200KV_ROPE_NONE && !(theta > 0.0f)) return B200KV_ERR_INVALID;
    if (token_count == 0) return B200KV_OK;
    if (prefill_state == nullptr && decode_state == nullptr &&
        static_cast<uint64_t>(base_position) + token_count > view->capacity)
        return B200KV_ERR_RANGE;
    rc = ensure_device();
    if (rc != B200KV_OK) return rc;

    AppendParams p{};
    p.view = *view;
    p.key = key;
    p.value = value;
    p.k_norm_weight = k_norm_weight;
    p.prefill_state = prefill_state;
    p.decode_state = decode_state;
    // A bound above any cache's capacity, where the count is on the device: as many tokens as the kernel's 32-bit unit numbers hold (with
    // more than eight heads of 128 dims that is 2^30, a cache of terabytes).
    const uint64_t passes = (static_cast<uint64_t>(view->kv_heads) + kUnitElems / view->head_dim - 1) / (kUnitElems / view->head_dim);
    if (prefill_state != nullptr || decode_state != nullptr) token_count = static_cast<uint32_t>(std::min<uint64_t>(token_count, 0xffffffffu / (2 * passes)));
    p.token_count = token_count;
    p.base_position = base_position;
    p.rope_mode = rope_mode;
    p.epsilon = epsilon;
    rope_constants(rope_mode, theta, view->head_dim, p.inv_freq, &p.sectioned_step);

    const uint32_t d = view->head_dim;
    const uint64_t units = 2 * token_count * passes;
    if (units >= (1ull << 32)) return B200KV_ERR_RANGE;
    int device = 0, sms = 0;
    B200KV_CUDA_TRY(cudaGetDevice(&device));
    B200KV_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const bool f16 = (dtype == B200KV_F16);
    const uint64_t resident = static_cast<uint64_t>(sms) * (f16 ? kAppendCtasPerSm<true> : kAppendCtasPerSm<false>);
    const unsigned grid = static_cast<unsigned>(std::min<uint64_t>((units + kAppendWarps - 1) / kAppendWarps, resident));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // vector loads need aligned inputs (a lane's four elements start at a multiple of four of them)
    const bool vec = ((reinterpret_cast<uintptr_t>(key) | reinterpret_cast<uintptr_t>(value)) & 15u) == 0;
    const dim3 block(kAppendWarps * 32);
    cudaError_t err;
    auto launch = [&](auto kernel, std::atomic<int>& slots) {   // slots: CTAs of the kernel that fit on an SM
        int n = slots.load(std::memory_order_relaxed);
        if (n == 0) {
            const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kAppendWarps * 32, 0);
            if (e != cudaSuccess) return e;
            slots.store(n, std::memory_order_relaxed);
        }
        p.fills_device = grid >= static_cast<uint64_t>(sms) * n;
        return launch_kernel(kernel, grid, block, 0, s, true, p, vec);
    };
    static std::atomic<int> slots[4] = {};
    if (d == 128) err = f16 ? launch(append_kernel<128, true>, slots[0]) : launch(append_kernel<128, false>, slots[1]);
    else err = f16 ? launch(append_kernel<256, true>, slots[2]) : launch(append_kernel<256, false>, slots[3]);
    B200KV_CUDA_TRY(err);
    return B200KV_OK;
}
