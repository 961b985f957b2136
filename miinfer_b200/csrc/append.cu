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
//   - D/16 lanes hold a row, lane l of them elements 8l .. 8l+7 and D/2 + 8l .. D/2 + 8l+7: NeoX pairs (i, i + d/2) lie in
//     one lane, sectioned pairs (i, i + 32) four lanes apart, and every access is 16 bytes of fp16 or eight of int8 per lane, in whole lines.
//   - The reference's shared-memory binary tree for the sum of squares (stride d/2 .. 1) becomes one register add and a
//     butterfly that adds exactly the same pairs (addition commutes: identical bits); each exchange halves the values a
//     lane carries.
//   - The 32 block maxima are reduced the same way, four values over four lanes in three shuffles, and come out one
//     block per lane -- so each IEEE division (scale, reciprocal, 1/rms) is taken once, by one lane.
//   - The sines and cosines depend on the token only; the first token's are computed ahead of the dependency wait where the host knows the position.
//   - Products run two to an instruction (f32x2), four int8 are packed by two cvt.pack.
// Bound by instruction issue and the latencies of 16 to 20 warps an SM (60 % of issue slots while it runs at 8192 tokens; the writes stay in L2): 8192 tokens x 8 heads of 128
// dims, fp16 to q8_0, take 15.95 us, 37 tokens 2.4 (16.9 and 2.6 with four consecutive elements a lane, runs of equal length and every rotation behind the wait; 4 heads of
// 256: 17.5 -> 16.5, 512 tokens 3.8 -> 3.1).  Runs of 16 elements a lane have fewer instructions (600 a unit, 630 here, 690 before) and accesses of half sectors: 15.8 us, but fp32
// input 21.3 (18.1 here).  Input of the first unit or the norm weights prefetched: slower at every size.  A layout with lanes 32 elements apart, element-wise K accesses and one redux per block
// took 21.8 us, one with its input in a cp.async ring 20.0 us alone, and its shared memory kept the next
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
constexpr int kRun = 8;                // consecutive elements of each half of a row in a lane: 16 bytes of fp16, so that a warp's accesses are whole lines
// CTAs per SM.  fp32 input (two registers for every one of fp16 that is under way): 8, 16 warps of 128 registers.  fp16 input has both: 8, or 10 of 96 registers, of which 16 to 28
// bytes spill (pick_ctas).
constexpr int kFewCtas = 8, kManyCtas = 10;
// A warp's work comes in whole units.  Up to four a warp, fewer and faster warps are the better choice, but for the sizes that end in two units of the many warps and three of
// the few; beyond that the many are level or better.  us a launch, 8 / 10 CTAs, q8_0, 8 heads of 128 and 4 of 256: 256 tokens 2.84 / 3.06 and 3.11 / 3.37, 2048 6.2 / 7.0
// and 6.1 / 6.7, 2960 8.5 / 7.7 and 8.7 / 7.5, 3500 9.0 / 9.8 and 9.3 / 10.1, 5000 11.4 / 11.6 and 12.4 / 11.8, 8192 16.4 / 15.95 and 17.4 / 16.5.
static int pick_ctas(uint64_t units, uint32_t sms) {
    const uint64_t few = static_cast<uint64_t>(sms) * kFewCtas * kAppendWarps, many = static_cast<uint64_t>(sms) * kManyCtas * kAppendWarps;
    return units > 4 * few || (units > 2 * few && units <= 2 * many) ? kManyCtas : kFewCtas;
}

// What the pointers of a launch are aligned to 16 bytes for.
enum AppendAlign : uint32_t { kInputAligned = 1, kWeightAligned = 2 };   // (the planes always are: validate_view)

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

// A lane's eight consecutive input elements as they lie in memory, and as four pairs of floats.
template <bool IN_F16> struct RawRun { uint4 v[IN_F16 ? 1 : 2]; };
template <bool IN_F16>
__device__ __forceinline__ void load_run(RawRun<IN_F16>& r, const void* src, size_t element, bool aligned) {
    constexpr int N = IN_F16 ? 1 : 2;
    if (aligned) {
        const uint4* s = reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(src) + element * (IN_F16 ? 2 : 4));
#pragma unroll
        for (int i = 0; i < N; ++i) r.v[i] = s[i];
    } else if constexpr (IN_F16) {
        const uint16_t* s = static_cast<const uint16_t*>(src) + element;
        auto two = [&](int i) { return s[i] | (static_cast<uint32_t>(s[i + 1]) << 16); };
#pragma unroll
        for (int i = 0; i < N; ++i) r.v[i] = make_uint4(two(8 * i), two(8 * i + 2), two(8 * i + 4), two(8 * i + 6));
    } else {
        const uint32_t* s = static_cast<const uint32_t*>(src) + element;
#pragma unroll
        for (int i = 0; i < N; ++i) r.v[i] = make_uint4(s[4 * i], s[4 * i + 1], s[4 * i + 2], s[4 * i + 3]);
    }
}
template <bool IN_F16>
__device__ __forceinline__ void widen(const RawRun<IN_F16>& r, Pair (&x)[kRun / 2]) {
    if constexpr (IN_F16) {
        auto two = [](uint32_t w) { const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w)); return pack_pair(f.x, f.y); };
        x[0] = two(r.v[0].x); x[1] = two(r.v[0].y); x[2] = two(r.v[0].z); x[3] = two(r.v[0].w);
    } else {
        auto two = [](uint32_t a, uint32_t b) { return pack_pair(__uint_as_float(a), __uint_as_float(b)); };
#pragma unroll
        for (int i = 0; i < 2; ++i) { x[2 * i] = two(r.v[i].x, r.v[i].y); x[2 * i + 1] = two(r.v[i].z, r.v[i].w); }
    }
}
// Largest magnitude of eight values, two more a step; a NaN counts as 0, as in warp_amax.
__device__ __forceinline__ float amax_run(const Pair (&x)[kRun / 2]) {
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < kRun / 2; ++i) {
        const float2 v = unpack_pair(x[i]);
        asm("max.ftz.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(fabsf(v.x)), "f"(fabsf(v.y)));
    }
    return m;
}
// round to nearest even, saturate to [-128, 127], NaN -> 0: quantize_s8 on four values, packed
__device__ __forceinline__ uint32_t quantize4(Pair x0, Pair x1, Pair inv2) {
    const float2 a = unpack_pair(mul2(x0, inv2)), b = unpack_pair(mul2(x1, inv2));
    uint32_t w;
    asm("{ .reg .b32 t; cvt.pack.sat.s8.s32.b32 t, %4, %3, 0; cvt.pack.sat.s8.s32.b32 %0, %2, %1, t; }"
        : "=r"(w) : "r"(__float2int_rn(a.x)), "r"(__float2int_rn(a.y)), "r"(__float2int_rn(b.x)), "r"(__float2int_rn(b.y)));
    return w;
}
__device__ __forceinline__ uint2 quantize_run(const Pair (&x)[kRun / 2], float inv) {
    const Pair inv2 = pack_pair(inv, inv);
    return make_uint2(quantize4(x[0], x[1], inv2), quantize4(x[2], x[3], inv2));
}
__device__ __forceinline__ uint32_t half_pair(Pair x) {
    const float2 f = unpack_pair(x);
    const __half2 h = __floats2half2_rn(f.x, f.y);
    return *reinterpret_cast<const uint32_t*>(&h);
}
template <int D, bool IN_F16, int CTAS>
__global__ void __launch_bounds__(kAppendWarps * 32, CTAS)
append_kernel(const __grid_constant__ AppendParams p, const uint32_t align) {
    constexpr int LPR = D / (2 * kRun);         // lanes per row
    constexpr int HB = kUnitElems / D;          // kv heads per unit: its rows
    constexpr int NB = D / 32;                  // q8_0 blocks per row
    constexpr int RPS = 32 / LPR;               // rows per step
    constexpr int SC = kRun / RPS;              // NeoX pairs a lane evaluates; the eight it rotates by come from the lanes of its number in the step's rows
    constexpr int LPB = 32 / kRun;              // lanes per q8_0 block
    static_assert(HB == 2 * RPS && LPB == 4);   // two steps
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int l = lane & (LPR - 1), sub = lane / LPR;          // lane of the row, row of the step
    const int rope_mode = p.rope_mode;
    float freq[SC];
    if (rope_mode == B200KV_ROPE_NEOX_FULL)
#pragma unroll
        for (int i = 0; i < SC; ++i) freq[i] = p.inv_freq[kRun * l + SC * sub + i];
    if (p.fills_device) pdl_launch_dependents();   // the next kernel may become resident; it orders itself against this one
    // K/V inputs and the device-side position come from preceding kernels.  Where the position is known on the host, the first token's rotation is taken ahead of the
    // wait.
    bool waited = p.prefill_state != nullptr || p.decode_state != nullptr;
    if (waited) pdl_wait();

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

    // Units in the order token, pass (HB heads), side (K, V); the warps' runs differ by one unit at most.  (32-bit arithmetic: the host keeps units
    // below 2^32.)
    const uint32_t passes = (H + HB - 1) / HB;
    const uint32_t total_units = token_count * passes * 2;
    const uint32_t warps = gridDim.x * kAppendWarps, me = blockIdx.x * kAppendWarps + warp;
    const uint32_t per_warp = total_units / warps, longer = total_units % warps;
    const uint32_t unit0 = me * per_warp + min(me, longer);
    const uint32_t unit1 = unit0 + per_warp + (me < longer ? 1 : 0);

    struct Cursor { uint32_t token, pass, side; };
    auto advance = [&](Cursor& c) {
        if (++c.side == 2) {
            c.side = 0;
            if (++c.pass == passes) { c.pass = 0; ++c.token; }
        }
    };
    auto inside = [&](const Cursor& c) { return static_cast<uint64_t>(base_position) + c.token < capacity; };   // never write outside the cache
    auto heads = [&](const Cursor& c) { return static_cast<int>(min(static_cast<uint32_t>(HB), H - c.pass * HB)); };
    RawRun<IN_F16> raw[2][2];   // per step: elements 8l .. and D/2 + 8l .. of the unit that comes next; a row that does not exist comes as zeros and is only not stored
    auto fetch = [&](const Cursor& c) {
        const void* src = c.side == 0 ? p.key : p.value;
        const size_t e0 = (static_cast<size_t>(c.token) * H + c.pass * HB + sub) * D + kRun * l;
        const int hn = heads(c);
#pragma unroll
        for (int s = 0; s < 2; ++s)
            if (s * RPS + sub < hn) {
                load_run<IN_F16>(raw[s][0], src, e0 + s * RPS * D, align & kInputAligned);
                load_run<IN_F16>(raw[s][1], src, e0 + s * RPS * D + D / 2, align & kInputAligned);
            } else {
                raw[s][0] = raw[s][1] = RawRun<IN_F16>{};
            }
    };

    Pair sn[kRun / 2], cs[kRun / 2];   // NeoX: pairs 8l + i; sectioned: pairs 8 (l % 4) + i
    auto rotation = [&](uint32_t position) {
        if (rope_mode == B200KV_ROPE_NEOX_FULL) {
            float s[SC], c[SC];
#pragma unroll
            for (int i = 0; i < SC; ++i) sincos_pinned(__fmul_rn(static_cast<float>(position), freq[i]), &s[i], &c[i]);
            auto of = [&](const float (&t)[SC], int k) { return __shfl_sync(0xffffffffu, t[k % SC], (k / SC) * LPR + l); };
#pragma unroll
            for (int i = 0; i < kRun / 2; ++i) {
                sn[i] = pack_pair(of(s, 2 * i), of(s, 2 * i + 1));
                cs[i] = pack_pair(of(c, 2 * i), of(c, 2 * i + 1));
            }
        } else if (rope_mode == B200KV_ROPE_SECTIONED64) {
            float angle = static_cast<float>(position), s, c;
            for (int i = 0; i < lane; ++i) angle = __fmul_rn(angle, p.sectioned_step);
            sincos_pinned(angle, &s, &c);
            auto of = [&](float t, int k) { return __shfl_sync(0xffffffffu, t, kRun * (l & 3) + k); };
#pragma unroll
            for (int i = 0; i < kRun / 2; ++i) {
                sn[i] = pack_pair(of(s, 2 * i), of(s, 2 * i + 1));
                cs[i] = pack_pair(of(c, 2 * i), of(c, 2 * i + 1));
            }
        }
    };

    using Rows = Pair[2][kRun / 2];   // a lane's run of each step's row
    auto transform_k = [&](Rows& a, Rows& b) {
        if (have_norm) {
            float ss_mine = 0.0f;
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                // stride D/2 in the lane; strides D/4 .. 8 between lanes, each exchange halving the values a lane carries (the odd ones leave) as long as
                // there are several, then the strides below 8, each between the lanes that an exchange has parted
                float v[kRun];
#pragma unroll
                for (int i = 0; i < kRun / 2; ++i) {
                    const float2 q = unpack_pair(add_products(mul2(a[s][i], a[s][i]), mul2(b[s][i], b[s][i])));
                    v[2 * i] = q.x; v[2 * i + 1] = q.y;
                }
#pragma unroll
                for (int m = LPR / 2, n = kRun / 2; n > 0; m >>= 1, n >>= 1) {
                    const bool up = lane & m;
#pragma unroll
                    for (int i = 0; i < n; ++i) v[i] = __fadd_rn(up ? v[2 * i + 1] : v[2 * i], __shfl_xor_sync(0xffffffffu, up ? v[2 * i] : v[2 * i + 1], m));
                }
                float ss = v[0];
#pragma unroll
                for (int m = LPR / kRun / 2; m > 0; m >>= 1) ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, m));   // D = 256: stride 8
#pragma unroll
                for (int m = LPR / kRun; m < LPR; m <<= 1) ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, m));     // strides 4, 2, 1
                if ((lane & 1) == s) ss_mine = ss;
            }
            const float r_mine = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss_mine, static_cast<float>(D)), p.epsilon)));
            Pair r2[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const float r = __shfl_sync(0xffffffffu, r_mine, (lane & ~1) | s);
                r2[s] = pack_pair(r, r);
            }
            auto weigh = [&](Rows& x, const float* w) {
#pragma unroll
                for (int i = 0; i < kRun / 4; ++i) {
                    float4 f;
                    if (align & kWeightAligned) f = *reinterpret_cast<const float4*>(w + 4 * i);
                    else f = make_float4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        x[s][2 * i] = mul2(mul2(x[s][2 * i], r2[s]), pack_pair(f.x, f.y));
                        x[s][2 * i + 1] = mul2(mul2(x[s][2 * i + 1], r2[s]), pack_pair(f.z, f.w));
                    }
                }
            };
            weigh(a, p.k_norm_weight + kRun * l);
            weigh(b, p.k_norm_weight + D / 2 + kRun * l);
        }
        if (rope_mode == B200KV_ROPE_NEOX_FULL) {
#pragma unroll
            for (int s = 0; s < 2; ++s)
#pragma unroll
                for (int i = 0; i < kRun / 2; ++i) {
                    const Pair x0 = a[s][i], x1 = b[s][i];
                    a[s][i] = sub_products(mul2(x0, cs[i]), mul2(x1, sn[i]));
                    b[s][i] = add_products(mul2(x0, sn[i]), mul2(x1, cs[i]));
                }
        } else if (rope_mode == B200KV_ROPE_SECTIONED64) {
            // elements 0-31 lie in lanes 0-3 of the row (x0 cos - x1 sin), 32-63 in lanes 4-7 (x0 sin + x1 cos)
#pragma unroll
            for (int s = 0; s < 2; ++s)
#pragma unroll
                for (int i = 0; i < kRun / 2; ++i) {
                    const Pair other = __shfl_xor_sync(0xffffffffu, a[s][i], 4);
                    const Pair t = mul2(a[s][i], cs[i]), u = mul2(other, sn[i]);
                    if (l < 8) a[s][i] = l & 4 ? add_products(u, t) : sub_products(t, u);
                }
        }
    };

    // BLOCKS: a q8_0 side, decided at compile time.
    auto store = [&](auto blocks_c, const Cursor& cur, const Rows& a, const Rows& b, uint64_t position) {
        constexpr bool BLOCKS = decltype(blocks_c)::value;
        const bool is_k = cur.side == 0;
        const int hn = heads(cur);
        const uint64_t row0 = (static_cast<uint64_t>(cur.pass) * HB + sub) * capacity + position;   // this lane's cache row of step 0; the next step's is RPS * capacity on
        if (!BLOCKS && !(is_k ? k_q8 : v_q8)) {
            __half* dst = static_cast<__half*>(is_k ? p.view.key_f16 : p.view.value_f16) + row0 * D + kRun * l;
            auto run = [](const Pair (&x)[kRun / 2]) { return make_uint4(half_pair(x[0]), half_pair(x[1]), half_pair(x[2]), half_pair(x[3])); };
#pragma unroll
            for (int s = 0; s < 2; ++s, dst += RPS * capacity * D) {
                if (s * RPS + sub >= hn) break;
                *reinterpret_cast<uint4*>(dst) = run(a[s]);
                *reinterpret_cast<uint4*>(dst + D / 2) = run(b[s]);
            }
            return;
        }
        // ---- block maxima: values 2s (elements below D/2) and 2s + 1, over the four lanes of a block; lane keeps value lane % 4.
        float m[4] = {amax_run(a[0]), amax_run(b[0]), amax_run(a[1]), amax_run(b[1])};
#pragma unroll
        for (int o = 2; o > 0; o >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < o; ++i) m[i] = fmaxf(up ? m[i + o] : m[i], __shfl_xor_sync(0xffffffffu, up ? m[i] : m[i + o], o));
        }
        const bool rows = !BLOCKS && row_scale;
        float amax = m[0];
        if (rows) {
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
#pragma unroll
            for (int o = LPB; o < LPR; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        }
        // ---- scales: amax / 127, its reciprocal, the fp16 scale to the cache -- one block per lane
        const float scale = (amax > 0.0f) ? __fdiv_rn(amax, 127.0f) : 1.0f;
        const float inv_mine = (scale > 0.0f) ? __fdiv_rn(1.0f, scale) : 1.0f;
        {
            const int s = (lane & 3) >> 1, block = (lane & 1) * (NB / 2) + l / LPB;
            __half* plane = static_cast<__half*>(is_k ? p.view.key_scales : p.view.value_scales);
            const uint64_t r = row0 + s * RPS * capacity;
            if (s * RPS + sub < hn && (!rows || block == 0)) plane[rows ? r : r * NB + block] = __float2half_rn(scale);
        }
        int8_t* dst = (is_k ? p.view.key_q8 : p.view.value_q8) + row0 * D + kRun * l;
#pragma unroll
        for (int s = 0; s < 2; ++s, dst += RPS * capacity * D) {
            const uint2 qa = quantize_run(a[s], __shfl_sync(0xffffffffu, inv_mine, (lane & 28) | (2 * s)));
            const uint2 qb = quantize_run(b[s], __shfl_sync(0xffffffffu, inv_mine, (lane & 28) | (2 * s + 1)));
            if (s * RPS + sub < hn) {
                *reinterpret_cast<uint2*>(dst) = qa;
                *reinterpret_cast<uint2*>(dst + D / 2) = qb;
            }
        }
    };

    Cursor cur{unit0 / (2 * passes), (unit0 / 2) % passes, unit0 & 1};
    if (waited) {
        if (unit0 < unit1 && inside(cur)) fetch(cur);
        if (!p.fills_device) pdl_launch_dependents();
    }
    uint32_t rotated_token = 0xffffffffu;
    for (uint32_t unit = unit0; unit < unit1; ++unit) {
        const uint64_t position = static_cast<uint64_t>(base_position) + cur.token;
        if (cur.side == 0 && cur.token != rotated_token) {
            rotated_token = cur.token;
            rotation(static_cast<uint32_t>(position));
        }
        if (!waited) {
            waited = true;
            pdl_wait();
            if (inside(cur)) fetch(cur);
            if (!p.fills_device) pdl_launch_dependents();
        }
        Rows a, b;
#pragma unroll
        for (int s = 0; s < 2; ++s) { widen<IN_F16>(raw[s][0], a[s]); widen<IN_F16>(raw[s][1], b[s]); }
        Cursor next = cur;
        advance(next);
        if (unit + 1 < unit1 && inside(next)) fetch(next);   // under this unit's arithmetic
        if (inside(cur)) {
            if (cur.side == 0) transform_k(a, b);
            if (!row_scale && (cur.side == 0 ? k_q8 : v_q8)) store(std::true_type{}, cur, a, b, position);
            else store(std::false_type{}, cur, a, b, position);
        }
        cur = next;
    }
    if (!waited) pdl_wait();
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
    const int ctas = f16 ? pick_ctas(units, static_cast<uint32_t>(sms)) : kFewCtas;
    const unsigned grid = static_cast<unsigned>(std::min<uint64_t>((units + kAppendWarps - 1) / kAppendWarps, static_cast<uint64_t>(sms) * ctas));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // 16-byte loads need aligned pointers (a lane's runs start at multiples of eight elements)
    const auto aligned = [](auto... ptr) { return ((reinterpret_cast<uintptr_t>(ptr) | ...) & 15u) == 0; };
    const uint32_t align = (aligned(key, value) ? kInputAligned : 0u) | (aligned(k_norm_weight) ? kWeightAligned : 0u);
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
        return launch_kernel(kernel, grid, block, 0, s, true, p, align);
    };
    static std::atomic<int> slots[6] = {};
    if (d == 128) err = !f16 ? launch(append_kernel<128, false, kFewCtas>, slots[0]) : ctas == kFewCtas ? launch(append_kernel<128, true, kFewCtas>, slots[1]) : launch(append_kernel<128, true, kManyCtas>, slots[2]);
    else err = !f16 ? launch(append_kernel<256, false, kFewCtas>, slots[3]) : ctas == kFewCtas ? launch(append_kernel<256, true, kFewCtas>, slots[4]) : launch(append_kernel<256, true, kManyCtas>, slots[5]);
    B200KV_CUDA_TRY(err);
    return B200KV_OK;
}
