// Streaming split-K GQA decode attention for every cache mode: fp16 or int8 K and V in any combination, int8 with one scale
// per block of 32 or per row, head_dim 128 or 256, up to 8 query heads per kv head, any capacity, one session or many.
// (int8 K and V at head_dim 128 with 1, 2 or 4 heads per kv head go to decode_tc5.cu / decode_q8.cu where the capacity allows.)
//
// The arithmetic is MIInfer's decode stage 1 (gfx906/kernels/qwen3_primitives.hip:7371-7485) with block scales, its stage 2
// follows in the same launch (decode_tail.cuh), and so does the single-token append of a decode step.
//
// Bound by HBM; the kernel's job is to keep enough bytes in flight and to spend few enough instructions per byte.
//  * One CTA = one (kv head, split, session); all query heads of the kv head share every byte that is read.  (The kernel this
//    one replaced gave each query head its own warp, read K and V once per head with one dependent round trip per position,
//    and ran at 0.06 of the HBM rate.)
//  * Each warp walks its own tiles of 16 positions (warp w of W takes tiles w, w + W, ...): no barrier between warps until the
//    end.  A tile is two UNITS, its K rows and its V rows, which the warp copies with cp.async into a private ring (about 24 KB;
//    8 warps on an SM keep 130 KB or more in flight), 16-byte chunks XORed with the row number so that ldmatrix
//    reads without bank conflicts (242 to 255 registers a thread at head_dim 256, no spills).  Rows of any alignment above 16 bytes work, rows past the end are zero-filled.
//  * S = Q K^T and O = P V run on mma.sync m16n8k16 with fp32 accumulation.  M = 16 is 8 heads x 2 terms: rows 0-7 hold the
//    high and rows 8-15 the low fp16 half of every query element (and of every weight), 22 bits in all, so the products are
//    those of an fp32 kernel and the two halves of a score sit in one thread.  K and V are exact in fp16: fp16 planes as they
//    are, int8 converted as integers (their scales multiply the fp32 block sums of S, and the weights of P).  Tensor
//    throughput is no limit here: 64 instructions of 16 x 8 x 16 per 16 positions at head_dim 256.
//  * The score fragments are the A operand of P V as they lie.  The dims of an int8 k step, and the columns of an int8 V
//    tile, are taken in the order in which ldmatrix delivers bytes; Q's fragments and the final store permute accordingly.
//  * Online softmax per warp in base 2 with a lazy reference: the accumulators are rescaled only when a head's maximum has
//    grown by more than 2^4 since the last rescale.  P V runs on weights scaled by a power of two that keeps weight x value scale
//    within fp16's normal range (chosen from the value scales seen; re-chosen, with a rescale, when larger ones appear).
// Measured, decode steps of 4 kv heads of 256 and 24 query heads back to back in a graph, append and merge inside, us a layer: fp16 cache 7.0 at
// 1500 positions, 10.9 at 6001 (the kernel this one replaced and its merge kernel: 64), 26.1 at 32768 (5.1 TB/s), 90 at 131072 (6.0 TB/s); q8_0
// 7.7 at 1500, 9.1 at 4000, 23.5 at 32768 (254), 77 at 131072 -- there the conversions of int8 show, and the tcgen05 kernels are faster.
// 24 sessions of 200 to 6000 positions in one launch, q8_0: 44 us (657).
// At a few thousand positions a launch is a chain of latencies.  Of the 7.0 cycles a warp spends on an instruction at 7777 positions, one scale per
// row, 1.3 wait for the instruction itself, 1.2 for memory and 1.1 for the one before; hence partials emitted two dims at a time, the copies' code
// once for both sides, 32-bit split bounds, and the merge's gate fetched early.  Together: q8_0 4000 positions 9.9 -> 9.0 us, one scale per row 7777
// 11.3 -> 10.6, fp16 6001 11.4 -> 10.75.
#include "decode_tail.cuh"

#include <climits>

namespace b200kv {

namespace {

constexpr int kTile = 16;                     // positions per tile
// The tensor core truncates (towards zero) where an fp32 instruction rounds, so a chain of MMAs into one accumulator leaves a bias of
// half a unit per link.  Scores are therefore chains of kChain MMAs added up by fp32 instructions, and where a warp may have more than
// kLongTiles tiles the O accumulators are emptied into fp32 sums every kHold of them (HOLD; those launches are bound by HBM, in the
// others the extra code costs 2 to 7 %).  Relative error against float64, fp16 cache: 24 / 4 heads of 256, 6001 positions 2.1e-7 (one
// chain of 16 per score: 5.5e-7; fp32 dot products lane by lane: 2.3e-7); 32 / 8 heads of 128, 131072 positions, 57 tiles a warp: 4e-7
// (never emptied: 1.1e-6; lane by lane: 7.9e-7).
template <int KF> constexpr int kChain = KF == 1 ? 4 : 2;
constexpr int kLongTiles = 24, kHold = 16;
enum Fmt { F16 = 0, ROW = 1, BLOCK = 2 };     // a side's storage: fp16, int8 with one scale per row, int8 with a scale per 32 dims

template <int D, int FMT>
struct Unit {   // one tile of one side in shared memory: rows, then scales
    static constexpr int kRow = FMT == F16 ? 2 * D : D;                                 // bytes per row
    static constexpr int kScale = FMT == F16 ? 0 : FMT == BLOCK ? kTile * (D / 32) * 2 : 64;   // row scales: 32 bytes, up to 2 bytes of alignment
    static constexpr int kBytes = kTile * kRow + kScale;
};

template <int D, int KF, int VF, int WARPS>
struct Plan {
    static constexpr int kThreads = WARPS * 32;
    static constexpr int kQBytes = D / 16 * 32 * 16;                                    // A fragments of Q: [k step][lane][16 bytes]
    static constexpr int kSlot = Unit<D, KF>::kBytes > Unit<D, VF>::kBytes ? Unit<D, KF>::kBytes : Unit<D, VF>::kBytes;
    using Scratch = tail::RowScratch<2 * D>;                                            // an appended row, one side
    static constexpr int kMisc = WARPS * 8 * 8 + 8 * 4 + 2 * static_cast<int>(sizeof(Scratch));   // per-warp (m, l), qmul, row
    static constexpr int kRing = 26 * 1024;                                             // per warp
    static constexpr int kUnits = kRing / kSlot < 12 ? kRing / kSlot : 12;
    static constexpr int kOffRing = kQBytes;
    static constexpr int kOffMisc = kOffRing + WARPS * kUnits * kSlot;
    static constexpr int kAlloc = kOffMisc + kMisc;
    static constexpr int kOutStride = D + 16;                                           // floats between heads of a warp's accumulators in shared memory
    static_assert(kUnits >= 3, "a unit in use and two in flight");
    static_assert(kUnits * kSlot >= 8 * kOutStride * 4, "the accumulators fit where the ring was");
    static_assert(kQBytes >= (8 + 3 * 64 * 2) * 4, "the merger's scratch fits where Q was");
    static_assert(kAlloc * (8 / WARPS) <= 232448 - 1024 * (8 / WARPS), "8 warps per SM");
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, bool live) {   // zero-fills when not live
    const int n = live ? BYTES : 0;
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two int8 (selected by `sel` out of w ^ 0x80..) as exact fp16
template <uint32_t SEL>
__device__ __forceinline__ uint32_t i8x2(uint32_t biased) {
    const uint32_t h = __byte_perm(biased, 0x64646464u, SEL);          // halves 0x64b: 1024 + b
    const __half2 v = __hadd2(*reinterpret_cast<const __half2*>(&h), __float2half2_rn(-1152.0f));
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack2(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2*>(&v)); }
// A fragment of P for 16 positions: rows 0-7 the fp16 value of each weight, rows 8-15 what rounding left
__device__ __forceinline__ void split_p(const float (&p)[4], uint32_t (&a)[4]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        a[2 * i] = pack2(p[2 * i], p[2 * i + 1]);
        const float2 h = unpack2(a[2 * i]);
        a[2 * i + 1] = pack2(p[2 * i] - h.x, p[2 * i + 1] - h.y);
    }
}
// The sum of a value's two terms.  Where the first is infinite or NaN it is the result: the second is 0 x infinity, or what was left of infinity.
__device__ __forceinline__ float terms(float hi, float lo) { return fabsf(hi) < INFINITY ? hi + lo : hi; }
__device__ __forceinline__ float exp2i(int e) { return __int_as_float((e + 127) << 23); }   // 2^e for normal results
__device__ __forceinline__ float quad_max(float v) {
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
    return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}

template <int D, int KF, int VF, int WARPS, bool HOLD>
__global__ void __launch_bounds__(WARPS * 32, 8 / WARPS) decode_stream_kernel(const __grid_constant__ DecodeParams p) {
    using P = Plan<D, KF, VF, WARPS>;
    using KU = Unit<D, KF>;
    using VU = Unit<D, VF>;
    constexpr int SEG = D / 128;
    constexpr float kLazy = 4.0f;                     // log2 of how far the weights may outgrow the reference
    extern __shared__ __align__(128) uint8_t smem[];
    if (p.new_key == nullptr) pdl_launch_dependents();   // the next kernel of the stream may become resident as SMs free up; it orders itself

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // kv head fastest for one session, splits fastest for many (as in decode_tc5.cu)
    const uint32_t kv_head = p.head_fastest ? blockIdx.x : blockIdx.y, split = p.head_fastest ? blockIdx.y : blockIdx.x, session = blockIdx.z;
    const b200kv_view& view = session_view(p, session);
    uint32_t begin, end;
    resolve_range(p, session, view, &begin, &end);
    const int G = static_cast<int>(p.query_heads / view.kv_heads);
    uint32_t num_splits = p.num_splits;
    if (p.lengths != nullptr) {   // as many splits as this session's own length warrants; the surplus CTAs leave at once
        const uint32_t want = (end - begin + p.split_positions - 1) / p.split_positions;
        num_splits = min(num_splits, max(want, 1u));
        if (split >= num_splits) {
            if (p.ws_tagged == nullptr) {   // the separate merge kernel reads every split of the launch: an empty partial
                pdl_wait();
                for (int idx = tid; idx < G * D; idx += P::kThreads)
                    tail::emit_partial<SEG>(p, session, split, num_splits, kv_head * G + idx / D, idx % D, 0.0f, -INFINITY, 0.0f);
            }
            return;
        }
    }
    // this CTA's positions: whole tiles counted from `begin`
    const uint32_t tiles = (end - begin) / kTile + ((end - begin) % kTile != 0);
    const TileRange range = split_tiles<WARPS>(tiles, split, num_splits, p.late_splits);
    const uint32_t t0 = range.begin, t1 = range.end;
    const uint32_t pos0 = begin + t0 * kTile;
    const int my_tiles = static_cast<int>((t1 - t0 + WARPS - 1 - warp) / WARPS);   // tiles of this warp

    // A fused append: the row is left out of the copies, produced by the two warps behind the last tile's (they hold the fewest
    // tiles), and patched into the tile by its warp.
    const bool appends = tail::appends_row(p, begin, end);
    const uint32_t needed_end = appends ? end - 1 : end;
    const uint32_t early_end = needed_end > p.overlap_tail ? needed_end - p.overlap_tail : 0;   // rows from here on wait for the preceding kernel
    const bool fuse = appends && split + 1 == num_splits;   // the last split holds the last position
    const int last_warp = fuse ? static_cast<int>((t1 - t0 - 1) % WARPS) : -1;
    const bool makes_key = fuse && warp == (last_warp + 1) % WARPS, makes_value = fuse && warp == (last_warp + 2) % WARPS;
    const uint32_t copy_end = fuse ? end - 1 : end;

    const uint64_t head_row0 = static_cast<uint64_t>(kv_head) * view.capacity;
    const uint8_t* k_rows = (KF == F16 ? static_cast<const uint8_t*>(view.key_f16) : reinterpret_cast<const uint8_t*>(view.key_q8)) + head_row0 * KU::kRow;
    const uint8_t* v_rows = (VF == F16 ? static_cast<const uint8_t*>(view.value_f16) : reinterpret_cast<const uint8_t*>(view.value_q8)) + head_row0 * VU::kRow;
    const uint8_t* k_scales = static_cast<const uint8_t*>(view.key_scales) + head_row0 * (KF == BLOCK ? D / 16 : 2);
    const uint8_t* v_scales = static_cast<const uint8_t*>(view.value_scales) + head_row0 * (VF == BLOCK ? D / 16 : 2);

    const uint32_t ring = smem_u32(smem) + P::kOffRing + warp * (P::kUnits * P::kSlot);
    float* ml_s = reinterpret_cast<float*>(smem + P::kOffMisc);     // [WARPS][8] {m, l}
    float* qmul_s = ml_s + WARPS * 16;                              // [8]
    typename P::Scratch* new_row = reinterpret_cast<typename P::Scratch*>(qmul_s + 8);   // K, V

    // ---- one unit (K or V rows of the warp's tile t) into ring slot `slot` -----------------------------------
    auto copy_side = [&](auto fmt_c, const uint8_t* rows, const uint8_t* scales, uint32_t pos, uint32_t dst) {
        constexpr int FMT = decltype(fmt_c)::value;
        using U = Unit<D, FMT>;
        constexpr int CPR = U::kRow / 16;          // 16-byte chunks per row: 8, 16 or 32
        const bool full = pos + kTile <= copy_end;
        const uint8_t* src = rows + static_cast<uint64_t>(pos) * U::kRow + lane * 16;   // rows of a kv head are contiguous
#pragma unroll
        for (int it = 0; it < CPR / 2; ++it) {
            const int id = it * 32 + lane, row = id / CPR, c = id % CPR;
            const bool live = full || pos + row < copy_end;
            cp_async<16>(dst + row * U::kRow + ((c ^ (row & 7)) << 4), live ? src + it * 512 : rows, live);
        }
        if constexpr (FMT == BLOCK) {
            constexpr int SB = D / 16;             // scale bytes per row
            const bool live = full || pos + lane < copy_end;
            if (lane < kTile) cp_async<SB>(dst + kTile * U::kRow + lane * SB, live ? scales + (static_cast<uint64_t>(pos) + lane) * SB : scales, live);
        } else if constexpr (FMT == ROW) {
            // 2-byte scales start on any even address: the aligned words around them, nine at most
            const uintptr_t a = reinterpret_cast<uintptr_t>(scales + static_cast<uint64_t>(pos) * 2), word = (a & ~static_cast<uintptr_t>(3)) + lane * 4;
            const bool live = word < reinterpret_cast<uintptr_t>(scales + static_cast<uint64_t>(copy_end) * 2);
            if (lane < 9) cp_async<4>(dst + kTile * U::kRow + lane * 4, reinterpret_cast<const void*>(live ? word : a & ~static_cast<uintptr_t>(3)), live);
        }
    };
    auto tile_pos = [&](int t) { return pos0 + static_cast<uint32_t>(t * WARPS + warp) * kTile; };
    int next_unit = 0, next_slot = 0;             // units issued so far; slot of the next one
    auto issue = [&]() {
        const int t = next_unit >> 1;
        if (t < my_tiles) {
            const uint32_t dst = ring + next_slot * P::kSlot;
            const bool v = next_unit & 1;
            if constexpr (KF == VF) copy_side(std::integral_constant<int, KF>{}, v ? v_rows : k_rows, v ? v_scales : k_scales, tile_pos(t), dst);   // half the code
            else if (v) copy_side(std::integral_constant<int, VF>{}, v_rows, v_scales, tile_pos(t), dst);
            else copy_side(std::integral_constant<int, KF>{}, k_rows, k_scales, tile_pos(t), dst);
        }
        cp_commit();                              // an empty group keeps the count
        ++next_unit;
        next_slot = next_slot + 1 == P::kUnits ? 0 : next_slot + 1;
    };

    // old rows do not depend on the preceding kernels: their copies start before the wait for those
    while (next_unit < P::kUnits - 1 && (next_unit >> 1) < my_tiles && min(tile_pos(next_unit >> 1) + kTile, copy_end) <= early_end) issue();
    // The queries on their way to L2.  Not for one session over an int8 cache, whose launch is the shortest chain up to the wait.  Without -> with, us: fp16, one session, 32 / 8 heads
    // of 128, 36 layers at 1081 positions 187.5 -> 184.5, 24 / 4 of 256, 16 at 2500 140.5 -> 139.2; many, int8, 24 / 4 of 256, 8 layers, 4 sessions of 2000 152.1 -> 149.3, 17 of 1389
    // 146.0 -> 143.1; one session, q8_0, 32 / 8 of 128, 36 layers at 640 203.8 -> 206.7, 782 208.1 -> 209.6.
    if constexpr (WARPS == 4 || (KF == F16 && VF == F16)) {
        const uint32_t row = D * (p.q_is_f16 ? 2 : 4);
        if (split == 0 && warp == WARPS - 1) prefetch_lines(static_cast<const uint8_t*>(p.q) + (static_cast<size_t>(session) * p.query_heads + kv_head * G) * row, G * row, lane);
    }
    Rotation<D> rot{};
    if (makes_key) row_rotation<D>(rot, lane, end - 1, p.rope_mode, p.inv_freq, p.sectioned_step);   // needs the position only
    pdl_wait();
    float new_x[D / 32], norm[D / 32];
    if (makes_key || makes_value) {
        tail::load_new_row<D>(makes_key ? p.new_key : p.new_value, p.new_is_f16, kv_head, lane, new_x);
        load_norm_weight<D>(p.k_norm_weight, lane, norm);
    }
    while (next_unit < P::kUnits - 1) issue();
    if (p.new_key != nullptr) pdl_launch_dependents();   // an appending launch: see pdl_launch_dependents

    // ---- Q: scaled by a power of two per head (largest element to [2^13, 2^14)), split into two fp16 terms, as A fragments ----
    for (int h = warp; h < 8; h += WARPS) {
        constexpr int NP = D / 64;                // pairs of dims per lane
        float q[2 * NP];
        float amax = 0.0f;
        if (h < G) {
            const size_t base = (static_cast<size_t>(session) * p.query_heads + kv_head * G + h) * D;
            if (p.q_pairs && p.q_is_f16) {        // all loads of a head in flight together
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    const float2 v = __half22float2(*reinterpret_cast<const __half2*>(static_cast<const __half*>(p.q) + base + (i * 32 + lane) * 2));
                    q[2 * i] = v.x; q[2 * i + 1] = v.y;
                }
            } else if (p.q_pairs) {
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    const float2 v = *reinterpret_cast<const float2*>(static_cast<const float*>(p.q) + base + (i * 32 + lane) * 2);
                    q[2 * i] = v.x; q[2 * i + 1] = v.y;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 2 * NP; ++i) {
                    const size_t at = base + ((i >> 1) * 32 + lane) * 2 + (i & 1);
                    q[i] = p.q_is_f16 ? __half2float(static_cast<const __half*>(p.q)[at]) : static_cast<const float*>(p.q)[at];
                }
            }
#pragma unroll
            for (int i = 0; i < 2 * NP; ++i) amax = fmaxf(amax, fabsf(q[i]));
            amax = warp_max(amax);
        } else {
#pragma unroll
            for (int i = 0; i < 2 * NP; ++i) q[i] = 0.0f;
        }
        const int exponent = static_cast<int>(__float_as_uint(amax) >> 23) - 127;             // floor(log2 amax); amax >= 0
        const int up = amax > 0.0f ? max(-100, min(100, 13 - exponent)) : 0;
        const float mult = exp2i(up);
        if (lane == 0) qmul_s[h] = p.scale * 1.4426950408889634f * exp2i(-up);                // scores in base-2 units
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            const int pair = i * 32 + lane, ks = pair >> 3, w = pair & 7;                     // dims 16 ks + 2 w, + 1
            const int c = KF == F16 ? w & 3 : w >> 1, half = KF == F16 ? w >> 2 : w & 1;
            const float x = q[2 * i] * mult, y = q[2 * i + 1] * mult;
            const uint32_t hi = pack2(x, y);
            const float2 hf = unpack2(hi);
            *reinterpret_cast<uint2*>(smem + ((ks * 32 + h * 4 + c) * 4 + half * 2) * 4) = make_uint2(hi, pack2(x - hf.x, y - hf.y));
        }
    }
    __syncthreads();
    const float qmul = qmul_s[lane >> 2];
    if (makes_key || makes_value) {
        if (makes_key) tail::store_new_key<D>(p, view, new_x, norm, rot, head_row0 + end - 1, lane, new_row);
        else tail::store_new_value<D>(view, new_x, head_row0 + end - 1, lane, new_row + 1);
        __threadfence_block();
        asm volatile("bar.arrive 3, 96;" ::: "memory");
    }

    // ---- the tile loop: lane / 4 = query head, lane % 4 = positions 2c, 2c + 1, 2c + 8, 2c + 9 of the tile -------
    constexpr int NT = D / 8;
    float o[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[i][j] = 0.0f;
    float m_ref = -INFINITY, l_run = 0.0f;        // this head's reference (base-2 units); sum over this thread's positions
    float vs_cap = 0.0f;                          // largest value scale the weights' multiplier allows for, a power of two
    int p_exp = VF == F16 ? 10 : 0;               // log2 of that multiplier; weights <= 2^kLazy: x 2^10 keeps them below 2^14
    const int c4 = lane & 3;
    // ldmatrix addresses: lane l names row (l & 7) + 8 * ((l >> 3) & 1) of the tile, 16-byte chunk (l >> 4) of the pair read
    const int lrow = (lane & 7) + ((lane >> 3) & 1) * 8, lchunk = lane >> 4;
    int slot = 0;
    auto acquire = [&]() -> uint32_t {            // the next unit in order; returns its address
        cp_wait<P::kUnits - 2>();
        __syncwarp();
        issue();                                  // into the slot whose unit was consumed before this one
        const uint32_t a = ring + slot * P::kSlot;
        slot = slot + 1 == P::kUnits ? 0 : slot + 1;
        return a;
    };
    const int patch_tile = warp == last_warp ? my_tiles - 1 : -1;
    auto patch = [&](auto fmt_c, uint32_t unit, const typename P::Scratch& row) {   // the appended row into its unit
        constexpr int FMT = decltype(fmt_c)::value;
        using U = Unit<D, FMT>;
        const uint32_t r = (end - 1 - begin) % kTile;
        uint8_t* at = smem + (unit - smem_u32(smem));
        if (lane < U::kRow / 16)
            *reinterpret_cast<uint4*>(at + r * U::kRow + ((lane ^ (r & 7)) << 4)) = *reinterpret_cast<const uint4*>(row.data + lane * 16);
        if constexpr (FMT == BLOCK) {
            if (lane < D / 32) reinterpret_cast<__half*>(at + kTile * U::kRow)[r * (D / 32) + lane] = row.scales[lane];
        } else if constexpr (FMT == ROW) {
            const uint8_t* plane = &row == new_row ? k_scales : v_scales;
            const uintptr_t skew = reinterpret_cast<uintptr_t>(plane + static_cast<uint64_t>(end - 1 - r) * 2) & 2u;
            if (lane == 0) *reinterpret_cast<__half*>(at + kTile * U::kRow + skew + r * 2) = row.scales[0];
        }
    };
    // Sums of earlier tiles and how far they have been rescaled since.  `local` is 0, but not to the compiler: the array stays out
    // of the registers.
    float held[HOLD ? 2 * NT : 1], held_by = 1.0f;
    uint32_t local = 0;
    if constexpr (HOLD) asm volatile("mov.u32 %0, 0;" : "=r"(local));
    auto unhold = [&]() {
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                o[i][j] = fmaf(held[local + 2 * i + j], held_by, terms(o[i][j], o[i][j + 2]));
                o[i][j + 2] = 0.0f;
            }
    };
    auto hold = [&](bool first) {
        if (!first) unhold();
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                held[local + 2 * i + j] = terms(o[i][j], o[i][j + 2]);
                o[i][j] = o[i][j + 2] = 0.0f;
            }
        held_by = 1.0f;
    };
    auto rescale = [&](float f) {
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) o[i][j] *= f;
        if constexpr (HOLD) held_by *= f;
    };

    for (int t = 0; t < my_tiles; ++t) {
        const uint32_t pos = tile_pos(t);
        if constexpr (HOLD) {
            if (t % kHold == 0 && t != 0) hold(t == kHold);
        }
        if (t == patch_tile) {                    // the appended row's tile: both units have to be there
            cp_wait<0>();
            asm volatile("bar.sync 3, 96;" ::: "memory");   // ... and both sides of the row
            patch(std::integral_constant<int, KF>{}, ring + slot * P::kSlot, new_row[0]);
            patch(std::integral_constant<int, VF>{}, ring + (slot + 1 == P::kUnits ? 0 : slot + 1) * P::kSlot, new_row[1]);
            __syncwarp();
        }
        // ---------------- S = Q K^T ----------------
        float s[4];
        {
            const uint32_t unit = acquire();
            const uint8_t* scale_at = smem + (unit - smem_u32(smem)) + kTile * KU::kRow;
            const uint32_t row_at = unit + lrow * KU::kRow;
            const int flip = lrow & 7;
            if constexpr (KF == BLOCK) {
                constexpr int NB = D / 32;
                uint32_t ks[4][NB / 2];           // this thread's positions' scales, two blocks per word
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint8_t* src = scale_at + (2 * c4 + (i & 1) + (i >> 1) * 8) * (NB * 2);
                    if constexpr (NB == 8) *reinterpret_cast<uint4*>(ks[i]) = *reinterpret_cast<const uint4*>(src);
                    else *reinterpret_cast<uint2*>(ks[i]) = *reinterpret_cast<const uint2*>(src);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) s[i] = 0.0f;
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    uint32_t r[4];
                    ldsm4(row_at + (((2 * b + lchunk) ^ flip) << 4), r);
                    float acc[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const uint4 qa = *reinterpret_cast<const uint4*>(smem + ((2 * b + k) * 32 + lane) * 16);
                        const uint32_t a[4] = {qa.x, qa.y, qa.z, qa.w};
                        const uint32_t w0 = r[2 * k] ^ 0x80808080u, w1 = r[2 * k + 1] ^ 0x80808080u;
                        mma(acc[0], a, i8x2<0x4140>(w0), i8x2<0x4342>(w0));
                        mma(acc[1], a, i8x2<0x4140>(w1), i8x2<0x4342>(w1));
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 sc = unpack2(ks[i][b >> 1]);
                        s[i] = fmaf(acc[i >> 1][i & 1] + acc[i >> 1][(i & 1) + 2], (b & 1) ? sc.y : sc.x, s[i]);
                    }
                }
            } else {
                // Launches of few tiles a warp run through most code once or twice and wait for instructions more than for anything else: one
                // session's score loop is rolled up.
                constexpr int kRolled = HOLD || WARPS == 4 ? D / 16 : 2;
                float hi[4] = {0.0f, 0.0f, 0.0f, 0.0f}, lo[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll kRolled
                for (int k0 = 0; k0 < D / 16; k0 += kChain<KF>) {
                    float acc[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
#pragma unroll
                    for (int ks = k0; ks < k0 + kChain<KF>; ++ks) {
                        const uint4 qa = *reinterpret_cast<const uint4*>(smem + (ks * 32 + lane) * 16);
                        const uint32_t a[4] = {qa.x, qa.y, qa.z, qa.w};
                        uint32_t r[4];
                        if constexpr (KF == F16) {
                            ldsm4(row_at + (((2 * ks + lchunk) ^ flip) << 4), r);
                            mma(acc[0], a, r[0], r[2]);
                            mma(acc[1], a, r[1], r[3]);
                        } else if ((ks & 1) == 0) {   // one ldmatrix serves two k steps of int8
                            const uint4 qb = *reinterpret_cast<const uint4*>(smem + ((ks + 1) * 32 + lane) * 16);
                            const uint32_t a2[4] = {qb.x, qb.y, qb.z, qb.w};
                            ldsm4(row_at + (((ks + lchunk) ^ flip) << 4), r);
#pragma unroll
                            for (int i = 0; i < 4; ++i) r[i] ^= 0x80808080u;
                            mma(acc[0], a, i8x2<0x4140>(r[0]), i8x2<0x4342>(r[0]));
                            mma(acc[1], a, i8x2<0x4140>(r[1]), i8x2<0x4342>(r[1]));
                            mma(acc[0], a2, i8x2<0x4140>(r[2]), i8x2<0x4342>(r[2]));
                            mma(acc[1], a2, i8x2<0x4140>(r[3]), i8x2<0x4342>(r[3]));
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) { hi[i] += acc[i >> 1][i & 1]; lo[i] += acc[i >> 1][(i & 1) + 2]; }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) s[i] = terms(hi[i], lo[i]);
                if constexpr (KF == ROW) {
                    const uint8_t* src = scale_at + (reinterpret_cast<uintptr_t>(k_scales + static_cast<uint64_t>(pos) * 2) & 2u);
#pragma unroll
                    for (int i = 0; i < 4; ++i) s[i] *= __half2float(*reinterpret_cast<const __half*>(src + (2 * c4 + (i & 1) + (i >> 1) * 8) * 2));
                }
            }
        }
        // ---------------- online softmax ----------------
        float pw[4];
        {
            float mt = -INFINITY;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s[i] = pos + 2 * c4 + (i & 1) + (i >> 1) * 8 < end ? s[i] * qmul : -INFINITY;
                mt = fmaxf(mt, s[i]);
            }
            mt = quad_max(mt);
            const bool grown = mt > m_ref + kLazy || (m_ref == -INFINITY && mt > -INFINITY);
            if (__any_sync(0xffffffffu, grown)) {
                const float m_new = grown ? mt : m_ref;
                const float f = m_ref == -INFINITY ? 0.0f : exp2f(m_ref - m_new);   // 1 for the heads that keep theirs
                const float keep = grown ? f : 1.0f;
                rescale(keep);
                l_run *= keep;
                m_ref = m_new;
            }
            const float ref = m_ref == -INFINITY ? 0.0f : m_ref;
#pragma unroll
            for (int i = 0; i < 4; ++i) pw[i] = exp2f(s[i] - ref);
            l_run += (pw[0] + pw[1]) + (pw[2] + pw[3]);
        }
        // ---------------- O += P V ----------------
        {
            const uint32_t unit = acquire();
            const uint8_t* scale_at = smem + (unit - smem_u32(smem)) + kTile * VU::kRow;
            const uint32_t row_at = unit + lrow * VU::kRow;
            const int flip = lrow & 7;
            auto fit_multiplier = [&](float largest) {   // `largest` finite |value scale| of the tile, the same in every lane
                if (largest > vs_cap) {
                    // room for 2^kLazy x a cap one binade above what was seen: product x multiplier <= 2^15
                    const int e = max(-100, min(100, static_cast<int>(__float_as_uint(largest) >> 23) - 127 + 2));
                    const int fit = 15 - static_cast<int>(kLazy) - e;
                    if (vs_cap > 0.0f) rescale(exp2i(max(-126, fit - p_exp)));
                    vs_cap = exp2i(e);
                    p_exp = fit;
                }
            };
            if constexpr (VF == BLOCK) {
                constexpr int NB = D / 32;
                uint32_t vs[4][NB / 2];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint8_t* src = scale_at + (2 * c4 + (i & 1) + (i >> 1) * 8) * (NB * 2);
                    if constexpr (NB == 8) *reinterpret_cast<uint4*>(vs[i]) = *reinterpret_cast<const uint4*>(src);
                    else *reinterpret_cast<uint2*>(vs[i]) = *reinterpret_cast<const uint2*>(src);
                }
                __half2 big = __float2half2_rn(0.0f);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int w = 0; w < NB / 2; ++w) big = __hmax2(big, __habs2(*reinterpret_cast<const __half2*>(&vs[i][w])));
                float largest = quad_max(fmaxf(__low2float(big), __high2float(big)));
                if (__any_sync(0xffffffffu, largest == INFINITY)) {   // an infinite scale is its own block's affair
                    float finite = 0.0f;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int w = 0; w < NB / 2; ++w) {
                            const float2 sc = unpack2(vs[i][w]);
                            if (fabsf(sc.x) < INFINITY) finite = fmaxf(finite, fabsf(sc.x));
                            if (fabsf(sc.y) < INFINITY) finite = fmaxf(finite, fabsf(sc.y));
                        }
                    largest = quad_max(finite);
                }
                fit_multiplier(largest);
#pragma unroll
                for (int i = 0; i < 4; ++i) pw[i] *= exp2i(p_exp);
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    float pb[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 sc = unpack2(vs[i][b >> 1]);
                        pb[i] = pw[i] * ((b & 1) ? sc.y : sc.x);
                    }
                    uint32_t a[4], r[4];
                    split_p(pb, a);
                    ldsm4_t(row_at + (((2 * b + lchunk) ^ flip) << 4), r);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {   // chunk 2b + k: even dims, odd dims
                        const uint32_t w0 = r[2 * k] ^ 0x80808080u, w1 = r[2 * k + 1] ^ 0x80808080u;
                        mma(o[4 * b + 2 * k], a, i8x2<0x4240>(w0), i8x2<0x4240>(w1));
                        mma(o[4 * b + 2 * k + 1], a, i8x2<0x4341>(w0), i8x2<0x4341>(w1));
                    }
                }
            } else {
                if constexpr (VF == ROW) {
                    const uint8_t* src = scale_at + (reinterpret_cast<uintptr_t>(v_scales + static_cast<uint64_t>(pos) * 2) & 2u);
                    float vs[4], big = 0.0f;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        vs[i] = __half2float(*reinterpret_cast<const __half*>(src + (2 * c4 + (i & 1) + (i >> 1) * 8) * 2));
                        if (pos + 2 * c4 + (i & 1) + (i >> 1) * 8 >= end) vs[i] = 0.0f;   // a word may carry a scale past the end
                        if (fabsf(vs[i]) < INFINITY) big = fmaxf(big, fabsf(vs[i]));
                    }
                    fit_multiplier(quad_max(big));
#pragma unroll
                    for (int i = 0; i < 4; ++i) pw[i] *= exp2i(p_exp) * vs[i];
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) pw[i] *= exp2i(p_exp);
                }
                uint32_t a[4];
                split_p(pw, a);
#pragma unroll
                for (int j = 0; j < VU::kRow / 32; ++j) {   // two 16-byte chunks of every row per ldmatrix
                    uint32_t r[4];
                    ldsm4_t(row_at + (((2 * j + lchunk) ^ flip) << 4), r);
                    if constexpr (VF == F16) {
                        mma(o[2 * j], a, r[0], r[1]);
                        mma(o[2 * j + 1], a, r[2], r[3]);
                    } else {
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const uint32_t w0 = r[2 * k] ^ 0x80808080u, w1 = r[2 * k + 1] ^ 0x80808080u;
                            mma(o[4 * j + 2 * k], a, i8x2<0x4240>(w0), i8x2<0x4240>(w1));
                            mma(o[4 * j + 2 * k + 1], a, i8x2<0x4341>(w0), i8x2<0x4341>(w1));
                        }
                    }
                }
            }
        }
    }

    // ---- the warps' states, through the ring's memory, into one partial of the CTA --------------------------------
    cp_wait<0>();
    if constexpr (HOLD) {
        if (my_tiles > kHold) unhold();
    }
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
    if (c4 == 0) *reinterpret_cast<float2*>(ml_s + (warp * 8 + (lane >> 2)) * 2) = make_float2(m_ref, l_run);
    {
        float* mine = reinterpret_cast<float*>(smem + P::kOffRing + warp * (P::kUnits * P::kSlot)) + (lane >> 2) * P::kOutStride;
        const float inv = exp2i(-p_exp);
        __syncwarp();                             // every lane is past its last ldmatrix
#pragma unroll
        for (int i = 0; i < NT; i += 2) {
            const float e0 = terms(o[i][0], o[i][2]) * inv, e1 = terms(o[i][1], o[i][3]) * inv;
            const float f0 = terms(o[i + 1][0], o[i + 1][2]) * inv, f1 = terms(o[i + 1][1], o[i + 1][3]) * inv;
            if constexpr (VF == F16) {            // n tile i: dims 8i + 2c, + 1
                *reinterpret_cast<float2*>(mine + 8 * i + 2 * c4) = make_float2(e0, e1);
                *reinterpret_cast<float2*>(mine + 8 * (i + 1) + 2 * c4) = make_float2(f0, f1);
            } else {                              // n tiles i, i + 1: the even and the odd dims of one 16-byte chunk
                *reinterpret_cast<float4*>(mine + 8 * i + 4 * c4) = make_float4(e0, f0, e1, f1);
            }
        }
    }
    __syncthreads();
    for (int idx = 2 * tid; idx < G * D; idx += 2 * P::kThreads) {
        const int h = idx / D, dim = idx % D;
        // The head's maximum and sum over the warps, by every thread for itself: one barrier and eight threads' chain less (us a layer: 32 / 8 heads of 128,
        // q8_0 2000 positions 7.10 -> 6.97, fp16 5000 7.86 -> 7.70; 24 / 4 of 256, q8_0 4000 9.92 -> 9.79, one scale per row 7777 12.21 -> 12.09).
        float2 ml[WARPS];
        float M = -INFINITY, L = 0.0f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            ml[w] = *reinterpret_cast<const float2*>(ml_s + (w * 8 + h) * 2);
            M = fmaxf(M, ml[w].x);
        }
        float2 a = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float2 x = *reinterpret_cast<const float2*>(smem + P::kOffRing + w * (P::kUnits * P::kSlot) + (h * P::kOutStride + dim) * 4);
            const float f = ml[w].x == -INFINITY ? 0.0f : exp2f(ml[w].x - M);
            L = fmaf(ml[w].y, f, L);
            a.x = fmaf(x.x, f, a.x); a.y = fmaf(x.y, f, a.y);
        }
        tail::emit_partial2<SEG>(p, session, split, num_splits, kv_head * G + h, dim, a, M * 0.6931471805599453f, L);
    }
    if (p.ws_tagged == nullptr) return;           // a separate merge kernel follows
    __syncthreads();
    tail::fused_merge<SEG, WARPS * 32>(p, session, kv_head, split, num_splits, G, reinterpret_cast<float*>(smem));
}

template <int D, int KF, int VF, int WARPS, bool HOLD>
int launch_kernel_of(const DecodeParams& p, dim3 grid, cudaStream_t stream) {
    using P = Plan<D, KF, VF, WARPS>;
    static std::atomic<uint64_t> done{0};   // one per kernel instantiation: devices that have opted in
    const cudaError_t attr_err = opt_in_dynamic_smem(reinterpret_cast<const void*>(decode_stream_kernel<D, KF, VF, WARPS, HOLD>), P::kAlloc, done);
    if (attr_err != cudaSuccess) { set_last_cuda_error(attr_err, "cudaFuncSetAttribute(decode_stream)"); return B200KV_ERR_CUDA; }
    B200KV_CUDA_TRY(launch_kernel(decode_stream_kernel<D, KF, VF, WARPS, HOLD>, grid, dim3(P::kThreads), P::kAlloc, stream, true, p));
    return B200KV_OK;
}

template <int D, int KF, int VF, int WARPS>
int launch_one(const DecodeParams& p, bool hold, dim3 grid, cudaStream_t s) {
    return hold ? launch_kernel_of<D, KF, VF, WARPS, true>(p, grid, s) : launch_kernel_of<D, KF, VF, WARPS, false>(p, grid, s);
}

template <int D, int WARPS>
int launch_mode(const DecodeParams& p, const b200kv_view& g, dim3 grid, cudaStream_t s) {
    const bool blocks = g.qblock == 32;
    const bool hold = p.split_positions / kTile > static_cast<uint32_t>(kLongTiles * WARPS);   // positions a split may have, over its warps (shorter last splits give no warp more tiles)
    switch (g.quant_mode) {
        case B200KV_F16_F16: return launch_one<D, F16, F16, WARPS>(p, hold, grid, s);
        case B200KV_Q8_F16: return blocks ? launch_one<D, BLOCK, F16, WARPS>(p, hold, grid, s) : launch_one<D, ROW, F16, WARPS>(p, hold, grid, s);
        case B200KV_F16_Q8: return blocks ? launch_one<D, F16, BLOCK, WARPS>(p, hold, grid, s) : launch_one<D, F16, ROW, WARPS>(p, hold, grid, s);
        default: return blocks ? launch_one<D, BLOCK, BLOCK, WARPS>(p, hold, grid, s) : launch_one<D, ROW, ROW, WARPS>(p, hold, grid, s);
    }
}

// One session: CTAs of 8 warps, one per SM, because fewer and larger splits leave fewer partials to merge.  Many sessions: CTAs
// of 4 warps, two per SM, so that one CTA's start and end overlap another's loop.
bool many_sessions(const DecodeParams& p) { return p.sessions > 1 || p.lengths != nullptr; }

}  // namespace

// Splits of the longest session.
uint32_t pick_splits_stream(uint32_t kv_heads, uint32_t query_heads, uint32_t head_dim, uint32_t sessions, uint32_t max_length) {
    const bool many = sessions > 1;
    const uint32_t slots = many ? 296u : 148u, units = kv_heads * sessions;
    uint32_t s = slots / units;                        // at most one wave of CTAs
    if (s == 0) s = 1;
    if (many) {   // mixed lengths: the longest session in pieces of at most 2048 positions, as the int8 kernels' default
        const uint32_t by_length = (max_length + 2047) / 2048;
        if (by_length > s) s = by_length;
    }
    // one tile per warp in every split -- or, of a short context, fewer, as long as every merge unit has a CTA of its own
    const uint32_t merge_units = query_heads / kv_heads * (head_dim / 128u);
    const uint32_t tiles = (max_length + kTile - 1) / kTile;
    uint32_t most = (tiles + 7) / 8;
    if (most < merge_units) most = merge_units < tiles ? merge_units : tiles;
    if (s > most) s = most;
    const uint32_t cap = max_splits_per_session(sessions);
    if (s > cap) s = cap;
    return s ? s : 1;
}

// Whether the merge may run inside the launch: the CTAs of a session wait for one another, so all of a session's CTAs have to
// fit on the device together (CTAs are dispatched in block order, a session's side by side).
bool stream_merge_fits(uint32_t kv_heads, uint32_t num_splits, bool many, uint32_t sms) {
    return static_cast<uint64_t>(kv_heads) * num_splits <= (many ? 2u : 1u) * sms;
}

int launch_decode_stream(const DecodeParams& p_in, const b200kv_view& geometry, uint32_t max_length, cudaStream_t stream) {
    DecodeParams p = p_in;
    p.overlap_tail = launch_overlap_tail();
    // many sessions: the split count is that of the longest; a session gets one split per `split_positions` of its own length
    const uint32_t per_split = (max_length + p.num_splits - 1) / (p.num_splits ? p.num_splits : 1);
    p.split_positions = (per_split + 127u) / 128u * 128u;
    if (p.split_positions < 128u) p.split_positions = 128u;
    const bool many = many_sessions(p);
    p.head_fastest = many ? 0u : 1u;
    // One session under launch overlap: as many CTAs as the launch before has mergers find an SM only when those leave, 1 to 2 us behind the others, and
    // the merge waits for the slowest; their splits hold a round of tiles less where that costs the others none (split_bounds.h).  Step, fp16 cache, us a
    // layer, even -> shorter last splits, launches back to back: 32 / 8 heads of 128, 5000 positions 9.1 -> 8.15, 10000 11.6 -> 10.7, 30000 22.4 ->
    // 22.05; 24 / 4 heads of 256, 10000 13.05 -> 11.6, 20000 18.25 -> 17.1, 30000 24.15 -> 23.25.  Nobody is late behind a kernel that does not let its
    // dependents in early, which a launch cannot know: there the longer splits cost 0 to 1.8 % (10000: 15.55 -> 15.8 and 16.75 -> 16.95).  Without the
    // rule's rounds (13000 positions of the second, 6600 of the first) they cost 3 to 5 % there and without overlap.
    const uint32_t mergers = p.query_heads / geometry.kv_heads * (geometry.head_dim / 128u);
    p.late_splits = many ? 0u : late_splits(p.overlap_tail > 0, p.ws_tagged != nullptr, geometry.kv_heads, p.num_splits, mergers, device_sms());
    const dim3 grid = many ? dim3(p.num_splits, geometry.kv_heads, p.sessions) : dim3(geometry.kv_heads, p.num_splits, 1);
    if (geometry.head_dim == 128) return many ? launch_mode<128, 4>(p, geometry, grid, stream) : launch_mode<128, 8>(p, geometry, grid, stream);
    return many ? launch_mode<256, 4>(p, geometry, grid, stream) : launch_mode<256, 8>(p, geometry, grid, stream);
}

}  // namespace b200kv
