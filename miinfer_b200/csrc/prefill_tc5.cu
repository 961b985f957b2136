// Suffix / prefill attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA).
//
// Same function as prefill_mma.cu (MIInfer's suffix kernels,
// gfx906/kernels/qwen3_primitives.hip:6788-7119 and 6637-6725), built for sm_100a:
//
//  1. A streaming pre-pass dequantises the positions the chunk can see, [0, kv_end), once per launch into an
//     fp16 scratch in the caller's workspace (K and V planes, [kv_head][row][d]); with int8 -> fp16 exact up to
//     the one rounding of q * scale.  The scratch (35.6 MB at 8704 x 4 x 256) stays in the 126 MB L2.  fp16 sides of the cache
//     are read where they lie.
//  2. The attention kernel gives each CTA 128 query ROWS of one kv head (a row is a (token, head-of-group)
//     pair, so the G heads of a group share every K/V tile) and walks the causal range in tiles of 64 positions,
//     two tiles at a time:
//       - the K ring (two stages of a PAIR of tiles each) and the V ring are fed with TMA
//         tensor copies (64x64 boxes, 128-byte swizzle: exactly the canonical shared-memory layout of the MMA
//         operands; the two tiles of a pair lie in rows 0-63 and 64-127 of every slab, one B operand);
//       - one lane of a warp that stays together issues S = Q.K^T (tcgen05.mma M128, K = d, Q read from TMEM), another O += P.V per tile
//         (M128 x N = d, K = 64; V consumed MN-major, as stored) into the O accumulator in TMEM; completion is tracked by
//         tcgen05.commit on mbarriers;
//       - groups of 128 softmax threads, one thread per row in each, take the tiles in turn: tcgen05.ld the S row, scale/mask (causal
//         length per row, .hip:6829), online softmax in base 2 with LAZY rescaling (O and the running sums are only rescaled when a row's
//         maximum grows by more than 2^8; P <= 256 fits fp16; the row's reference maximum is handed from tile to tile through shared
//         memory), hand P over as fp16, and at the end scale O by 1/sum, apply the sigmoid gate (.hip:6714-6723) and store.
//     head_dim 256: two groups; S for a pair of tiles at once (N = 128: issuing an MMA takes 50 clocks and more, the tensor pipe 32 at N = 64 and 64 at
//     N = 128), P in shared memory.  TMEM: S (pair) | Q | O.
//     head_dim 128: S tile by tile into four buffers of TMEM columns, P written over its own scores (the A operand of P.V comes from there), two warps that
//     issue S.  One row tile a CTA has four groups and four tiles under way (a tile takes 790 clocks, 512 of them MMAs; the softmax threads' chain through
//     it 3000).  A CTA takes TWO row tiles, two groups and buffers each, where there are enough of them: they share every K and V tile, and set-up, Q and output
//     come once for both; their S and O fill TMEM, so Q is an A operand in shared memory.
// Every mbarrier wait is bounded; a wait that runs out poisons the output rows with NaN, and the CTA still frees
// its TMEM and exits.
#include "decode_common.cuh"
#include "dequant.cuh"
#include "mbarrier_wait.cuh"
#include "reference_word.h"

#include <algorithm>
#include <cstring>
#include <mutex>

namespace b200kv {

namespace {

constexpr int kBM = 128;          // query rows per row tile; a CTA takes one or two (RT)
constexpr int kBN = 64;           // positions per KV tile
constexpr int kKPairs = 2;                         // K ring: stages of two tiles each (one S MMA covers a pair)
constexpr float kRescaleThreshold = 8.0f;        // log2 units
constexpr uint32_t kMaxKvSplits = 16;

struct Tc5Params {
    CUtensorMap kmap, vmap;      // fp16 [kv_heads][rows][d], box 1 x 64 x 64, 128-byte swizzle; zeros past the rows
    const void* q;               // [token][query_heads][D]
    int q_is_f16;
    const float* gate;
    float* out;
    uint32_t token_count, base_position;
    const b200kv_prefill_state* prefill_state;
    uint32_t query_heads, kv_heads;
    uint64_t capacity;           // cache capacity (causal ranges past it give zero rows)
    uint32_t scratch_rows;       // rows per kv head in the fp16 scratch
    float scale_log2;
    // KV split: split z walks tiles [ntiles*z/S, ntiles*(z+1)/S) of its rows and leaves an unnormalised partial
    // (O, reference maximum, sum) for prefill_merge_kernel.  kv_splits == 1: the kernel writes the output itself.
    uint32_t kv_splits;
    uint32_t sms;                // of the device: CTAs of a wave
    uint32_t rows_padded;        // query rows per kv head, rounded up to the row tile
    float* part_o;               // [split][kv_head][rows_padded][D]
    float2* part_ml;             // [split][kv_head][rows_padded] {maximum in log2 units, sum}
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}

// Shared-memory matrix descriptor (sm_100 format): start address, leading/stride byte offsets (all >> 4),
// descriptor version 1, 128-byte swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}
// Instruction descriptor for kind::f16: fp32 accumulate, fp16 A and B, M x N, operand majors (0 = K-major, 1 = MN-major).
__host__ __device__ constexpr uint32_t umma_idesc(uint32_t m, uint32_t n, uint32_t a_mn_major, uint32_t b_mn_major) {
    return (1u << 4) | (a_mn_major << 15) | (b_mn_major << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
        "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
        "%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
          "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
          "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
          "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15])),
          "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])), "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])),
          "r"(__float_as_uint(v[20])), "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
          "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])), "r"(__float_as_uint(v[27])),
          "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])), "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
        : "memory");
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
        "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st32_bits(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
        "%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
          "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]),
          "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]),
          "r"(v[30]), "r"(v[31])
        : "memory");
}
// P.V with the A operand (P, fp16, K-major: one query row per TMEM lane, two elements per 32-bit column) read from TMEM
__device__ __forceinline__ void umma_f16_a_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// Brings [src, src + bytes) on its way to L2; both multiples of 16.
__device__ __forceinline__ void prefetch_l2(const void* src, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
// Two fp32 values in one instruction, and the largest of three.
__device__ __forceinline__ Pair fma_pair(Pair a, Pair b, Pair c) { Pair r; asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ Pair add_pair(Pair a, Pair b) { Pair r; asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ float max3(float a, float b, float c) { float r; asm("max.ftz.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
// A wait of a whole warp, which stays together: all lanes go on or none.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)); }
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <int D, int RT>
struct Layout {
    // warps: the softmax groups of every row tile (one thread per query row in each, which take the tiles in turn), then the warps of the other roles
    static constexpr int kGroups = D == 128 ? 4 / RT : 2;  // softmax groups of a row tile; tile j is group j % kGroups's
    static constexpr int kSoftmaxThreads = RT * kGroups * 128;
    static constexpr int kTmaWarp = kSoftmaxThreads / 32;  // TMA producer of the K tiles
    static constexpr int kSWarp = kTmaWarp + 1;            // S = Q.K^T issuer / TMEM owner
    static constexpr int kIssuers = D == 128 ? 2 : 1;      // warps that issue S (two row tiles: one each; one: even and odd tiles)
    static constexpr int kPvWarp = kSWarp + kIssuers;      // O += P.V issuer
    static constexpr int kTmaVWarp = kPvWarp + 1;         // D == 256: TMA producer of the V tiles (a K load never waits for a V stage)
    static constexpr int kThreads = (kPvWarp + (D == 256 ? 2 : 1)) * 32;
    static constexpr int kRows = RT * kBM;
    static constexpr bool kQInTmem = RT == 1;              // two row tiles' S, P and O fill TMEM: their Q stays in shared memory
    static constexpr int kSlabs = D / 64;                  // 128-byte (64 x fp16) slabs along d
    static constexpr int kTileBytes = kSlabs * kBN * 128;  // one K or V tile: [slab][row][128 B]
    static constexpr int kPairBytes = 2 * kTileBytes;      // two K tiles as one B operand: [slab][128 rows][128 B]
    static constexpr int kOffK = 0;
    static constexpr int kOffV = kOffK + kKPairs * kPairBytes;
    static constexpr int kVTiles = D == 128 ? 5 : 2;       // V ring: with one producer for K and V, K must not wait for a V stage
    static constexpr int kOffP = kOffV + kVTiles * kTileBytes;   // D == 256: [group][row][128 B] fp16 P tiles; 4 KB a warp in which Q (kQInTmem) and O are turned (two row tiles: over their Q)
    static constexpr int kPBytes = kBM * 128;
    static constexpr int kOffQ = kOffP + (kQInTmem ? RT * kGroups * kPBytes : 0); // [row tile][slab][row][128 B]
    static constexpr int kQBytes = kSlabs * kBM * 128;
    static constexpr int kOffBar = kOffQ + (kQInTmem ? 0 : RT * kQBytes);
    // head_dim 128: P as an A operand in TMEM, in the first 32 columns of its own scores, which takes its writes and reads out of shared memory, and S tile
    // by tile in as many buffers as there are groups.  32 / 8 heads, us a layer, against two groups (one row tile) and pairs of S tiles with P in shared
    // memory (two): 461 over 8919 109 -> 97, 1024 over 8192 180 -> 169, 2048 fresh 58.7 -> 57.1.
    // At 256 S, Q and O leave no columns for P beside a pair of S tiles; with single ones in their place a layer of 512 tokens over 8192 took
    // 134 us, not 125.
    static constexpr bool kPInTmem = D == 128;
    // mbarriers; the ones after V_EMPTY are per row tile, S_EMPTY and the P pairs (kPInTmem: S_FULL too) per row tile and softmax group
    static constexpr int kBufs = RT * kGroups;
    static constexpr int K_FULL = 0, K_EMPTY = 2, V_FULL = 4, V_EMPTY = V_FULL + kVTiles, S_FULL = V_EMPTY + kVTiles, S_EMPTY = S_FULL + (kPInTmem ? kBufs : RT),
                         P_FULL = S_EMPTY + (kPInTmem ? 0 : kBufs), P_EMPTY = P_FULL + kBufs, O_DONE = P_EMPTY + kBufs, Q_FULL = O_DONE + RT, V_TAIL = Q_FULL + 1, kNumBars = V_TAIL + 1;
    static constexpr int kOffSlot = kOffBar + (kNumBars * 8 + 15) / 16 * 16;
    static constexpr int kOffRef = kOffSlot + 16;                 // [rows] {reference maximum, sequence}: handed from tile to tile
    // [group][128 rows] partial row sums of a row tile in its epilogue, where its own score MMAs are through: over the K
    // ring, or over the row tile's Q where the other row tile may still need K
    static constexpr int kSumStride = kGroups * kBM * 4;
    static constexpr int kOffSum = kQInTmem ? kOffK : kOffRef + kRows * 8;
    static constexpr int kTotal = kOffRef + kRows * 8 + (kQInTmem ? 0 : RT * kSumStride);
    static constexpr int kAlloc = kTotal;   // the dynamic shared memory is declared 1024-byte aligned; the kernel checks it
    static_assert(kAlloc <= 232448, "227 KB per CTA");
    static constexpr uint32_t kTmemCols = 512;
    // S: RT x kGroups x 64, P (kPInTmem, fp16 pairs) in the first 32 of its S; Q (RT == 1): D/2 (fp16 pairs), O: RT x D
    static constexpr uint32_t kColS = 0, kColQ = kPInTmem ? 384 : 128, kColO = 256;
    static_assert(kColO + RT * D <= 512 && (RT == 2 || (kPInTmem ? kColO + D <= kColQ && kColQ + D / 2 <= 512 : kColQ + D / 2 <= kColO)), "TMEM columns");
};

// The eight rows a lane takes of a warp's 32 (every fourth from `row`; rows are tokens' heads of one kv head) in [token][query_heads][D]: elements from
// the row of the warp's first token, which lie close enough for 32 bits.  One division, then additions.  (Two divisions for each row were 1.3 us
// of a CTA's start and as much of its end, 64-bit offsets worked out along with the loads and stores 0.3 us of each 32 columns of output.)
template <int D>
struct RowOffsets {
    uint32_t rel[8];
    int valid;   // rows that exist: the first `valid` of the eight
    __device__ __forceinline__ RowOffsets(uint32_t warp_row0, uint32_t turn_row, uint32_t G, uint32_t query_heads, uint32_t total_rows) {
        const uint32_t tokens = 4 / G, step_in_group = 4 - tokens * G;
        uint32_t in_group = warp_row0 % G + turn_row, token = in_group / G;
        in_group -= token * G;
        uint32_t off = (token * query_heads + in_group) * D;
        const uint32_t step = (tokens * query_heads + step_in_group) * D, wrap = (query_heads - G) * D;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            rel[i] = off;
            off += step;
            in_group += step_in_group;
            if (in_group >= G) { in_group -= G; off += wrap; }
        }
        valid = warp_row0 + turn_row < total_rows ? static_cast<int>(min((total_rows - warp_row0 - turn_row + 3) / 4, 8u)) : 0;
    }
};

// STATE: the position comes from a device-side state (one row tile a CTA).
template <int D, int RT, bool STATE>
__global__ void __launch_bounds__(Layout<D, RT>::kThreads, 1) prefill_tc5_kernel(const __grid_constant__ Tc5Params p) {
    using L = Layout<D, RT>;
    constexpr int kThreads = L::kThreads;
    constexpr int kTmaWarp = L::kTmaWarp, kSWarp = L::kSWarp, kPvWarp = L::kPvWarp, kTmaVWarp = L::kTmaVWarp;
    constexpr int K_FULL = L::K_FULL, K_EMPTY = L::K_EMPTY, V_FULL = L::V_FULL, V_EMPTY = L::V_EMPTY, S_FULL = L::S_FULL, S_EMPTY = L::S_EMPTY,
                  P_FULL = L::P_FULL, P_EMPTY = L::P_EMPTY, O_DONE = L::O_DONE, Q_FULL = L::Q_FULL, V_TAIL = L::V_TAIL;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw;
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar0 = sbase + L::kOffBar;
    auto bar = [&](int i) { return bar0 + i * 8; };
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kOffSlot);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // Row tiles from the last (the longest causal range) to the first, kv heads and KV splits of a row tile next to each
    // other: the CTAs dispatched last are the short ones, and a fresh chunk's last wave is nearly even.
    const uint32_t split_u = blockIdx.x % p.kv_splits, tile_head = blockIdx.x / p.kv_splits;
    const uint32_t kv_head = tile_head % p.kv_heads;
    const uint32_t G = p.query_heads / p.kv_heads;
    uint32_t base = p.base_position, count = p.token_count;
    if constexpr (STATE) {
        pdl_wait();   // the state may be the preceding kernel's output
        base = p.prefill_state->base_position;
        count = min(count, p.prefill_state->token_count);
    }
    const uint32_t total_rows = p.token_count * G;
    const uint32_t row0 = ((total_rows + L::kRows - 1) / L::kRows - 1 - tile_head / p.kv_heads) * L::kRows;
    // The next kernel of the stream (the merge of the KV splits) may become resident once every CTA has got here; it
    // orders itself against this one.  This kernel's own dependency wait comes after its set-up.
    pdl_launch_dependents();

    // longest causal range among this CTA's rows (rows are token-major; see prefill_mma.cu)
    uint32_t kv_end = 0;
    if (count > 0 && p.capacity > base) {
        const uint32_t t_first = row0 / G, t_last = (min(row0 + L::kRows, total_rows) - 1) / G;
        const uint64_t t_cap = p.capacity - base - 1;
        uint64_t t_max = t_last;
        if (t_max > count - 1) t_max = count - 1;
        if (t_max > t_cap) t_max = t_cap;
        if (t_max >= t_first) kv_end = base + static_cast<uint32_t>(t_max) + 1u;
    }
    if (kv_end > p.scratch_rows) kv_end = p.scratch_rows;   // never read past what the pre-pass wrote
    const int ntiles_all = static_cast<int>((kv_end + kBN - 1) / kBN);
    const int split = static_cast<int>(split_u), nsplit = static_cast<int>(p.kv_splits);
    const int tile0 = static_cast<int>(static_cast<long long>(ntiles_all) * split / nsplit);
    const int ntiles = static_cast<int>(static_cast<long long>(ntiles_all) * (split + 1) / nsplit) - tile0;   // tiles of this CTA

    // The layout (swizzled TMA tiles, MMA descriptors) needs the 1024-byte alignment the declaration above asks for; the
    // allocation has no slack for rounding up, so that a CTA of the neighbouring kernels fits beside this one on an SM.
    // Should a driver ever hand out another base, nothing of the layout is touched: the CTA's rows come out as NaN.
    if ((sbase & 1023u) != 0) {
        pdl_wait();
        const float nan = __int_as_float(0x7fc00000);
        for (uint32_t r = tid; r < static_cast<uint32_t>(L::kRows); r += kThreads)
            if (nsplit > 1 && row0 + r < total_rows)
                p.part_ml[(static_cast<size_t>(split) * p.kv_heads + kv_head) * p.rows_padded + row0 + r] = make_float2(0.0f, nan);
        if (nsplit == 1)
            for (uint32_t i = tid; i < static_cast<uint32_t>(L::kRows) * (D / 4); i += kThreads) {
                const uint32_t gr = row0 + i / (D / 4);
                if (gr >= total_rows) continue;
                const size_t off = (static_cast<size_t>(gr / G) * p.query_heads + kv_head * G + gr % G) * D + (i % (D / 4)) * 4;
                *reinterpret_cast<float4*>(p.out + off) = make_float4(nan, nan, nan, nan);
            }
        return;
    }

    const int live_tiles = min(RT, static_cast<int>((total_rows - row0 + kBM - 1) / kBM));   // row tiles that hold rows
    // ---- set-up: barriers, TMEM, Q ---------------------------------------------------------------------------
    // At head_dim 128 nothing of this waits for the rest: a CTA that takes another's place has its Q on its way into registers and its first K tiles into their
    // ring before its barriers are everybody's, and the CTA before has called its Q to L2.  (Set-up, then the loads: 1.5 us of every CTA but the first
    // wave's, which set up ahead of the dependency wait.  32 / 8 heads, us a layer: 1024 over 8192 175.5 -> 171, 37 over 3000 20.35 -> 19.7, 225 fresh 13.5 -> 13.0.  At 256 the same text
    // comes out of the compiler with a slower tile loop, 512 over 8192 125.7 -> 130.7.)
    constexpr bool kEarlyQ = D == 128;
    const int turn_row = lane >> 3, turn_chunk = lane & 7;
    const int rt = RT == 1 ? 0 : warp >> 3;                // row tile
    const uint32_t tile_row0 = row0 + rt * kBM, warp_row0 = tile_row0 + (warp & 3) * 32;
    // A pair of K tiles into its ring stage, tile 2i in rows 0-63 and tile 2i+1 in rows 64-127 of every slab (D == 256: one MMA instruction of N = 128 covers
    // both).
    auto issue_k = [&](int i) {
        const int ps = i % kKPairs, n = min(2, ntiles - 2 * i);
        mbar_expect_tx(bar(K_FULL + ps), n * L::kTileBytes);
        for (int t = 0; t < n; ++t)
            for (int s = 0; s < L::kSlabs; ++s)
                tma_load_3d(sbase + L::kOffK + ps * L::kPairBytes + s * (2 * kBN * 128) + t * (kBN * 128), &p.kmap, s * 64,
                            (tile0 + 2 * i + t) * kBN, kv_head, bar(K_FULL + ps));
    };
    // The query rows from r0 on of kv head `head` on their way to L2 (a prefetch reads nothing yet: whatever still writes them, the loads behind the wait
    // see).  A warp.
    auto prefetch_q = [&](uint32_t r0, uint32_t head) {
        const uint32_t elem = p.q_is_f16 ? 2 : 4, t_last = (min(r0 + L::kRows, total_rows) - 1) / G;
        for (uint32_t t = r0 / G + lane; t <= t_last; t += 32)
            prefetch_l2(static_cast<const uint8_t*>(p.q) + (static_cast<size_t>(t) * p.query_heads + head * G) * D * elem, G * D * elem);
    };
    constexpr int kTurns = D / 128;            // 32 columns = 64 dims per store; all loads are in flight together
    constexpr int kQWarps = RT * 8;            // two threads of a row each take half of it
    auto fetch_q = [&](const RowOffsets<D>& rows, uint4 (&q)[kTurns][8]) {
        auto fetch = [&](auto f16) {
            const size_t base0 = (static_cast<size_t>(warp_row0 / G) * p.query_heads + kv_head * G) * D + ((warp >> 2) & 1) * (D / 2) + turn_chunk * 8;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int k = 0; k < kTurns; ++k) {
                    q[k][i] = make_uint4(0, 0, 0, 0);
                    if (i >= rows.valid) continue;
                    if (f16()) {
                        q[k][i] = *reinterpret_cast<const uint4*>(static_cast<const __half*>(p.q) + base0 + rows.rel[i] + k * 64);
                    } else {
                        const float* src = static_cast<const float*>(p.q) + base0 + rows.rel[i] + k * 64;
                        const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
                        q[k][i] = make_uint4(pack_half2(a.x, a.y), pack_half2(a.z, a.w), pack_half2(b.x, b.y), pack_half2(b.z, b.w));
                    }
                }
        };
        if constexpr (RT == 2) fetch([&] { return p.q_is_f16 != 0; });   // (a branch around both: 1 % slower with two row tiles, 2 to 6 % faster with one)
        else if (p.q_is_f16) fetch([] { return true; });
        else fetch([] { return false; });
    };
    if (kEarlyQ ? warp == kTmaWarp && lane == 0 : tid == 0) {
        for (int i = 0; i < (STATE ? L::kNumBars : L::V_TAIL); ++i) {
            uint32_t count = 1;
            if (i >= S_EMPTY && i < P_EMPTY) count = kBM;   // S_EMPTY and P_FULL: a group's threads
            else if (i == Q_FULL) count = RT * 256;
            else if (i >= K_EMPTY && i < V_FULL) count = RT == 2 ? live_tiles : L::kIssuers;   // K: the warps that read it
            mbar_init(bar(i), count);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < L::kRows * 2; i += kThreads) reinterpret_cast<uint32_t*>(smem + L::kOffRef)[i] = 0;
    if (warp == kSWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(L::kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    [[maybe_unused]] uint4 early_q[kTurns][8];
    // one wave of CTAs: Q ahead of the wait (24 / 4 heads, 37 fp32 tokens over 3001: 24.3 -> 24.1 us a layer)
    if (kEarlyQ && warp == kTmaWarp && split_u == 0 && gridDim.x <= p.sms) prefetch_q(row0, kv_head);
    if constexpr (kEarlyQ) {
        if (warp < kQWarps) {
            const RowOffsets<D> rows(warp_row0, turn_row, G, p.query_heads, total_rows);
            pdl_wait();   // Q, the fp16 scratch and the device-side state come from preceding kernels
            fetch_q(rows, early_q);
        } else {
            pdl_wait();
            if (warp == kTmaWarp && lane == 0 && ntiles > 0) issue_k(0);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (!kEarlyQ && warp == kTmaWarp && split_u == 0 && gridDim.x <= p.sms) prefetch_q(row0, kv_head);
    [[maybe_unused]] const RowOffsets<D> late_rows(warp_row0, turn_row, G, p.query_heads, total_rows);
    if constexpr (!kEarlyQ) pdl_wait();
    bool failed = false;
    // The query rows of the CTA that takes this one's place, as far as the order of dispatch tells.  A warp.
    auto next_q = [&] {
        const uint32_t next = blockIdx.x + p.sms;
        if (next < gridDim.x && next % p.kv_splits == 0)
            prefetch_q(((total_rows + L::kRows - 1) / L::kRows - 1 - next / p.kv_splits / p.kv_heads) * L::kRows, next / p.kv_splits % p.kv_heads);
    };

    auto copy_v = [&](int j, int full) {
        mbar_expect_tx(bar(full), L::kTileBytes);
        for (int s = 0; s < L::kSlabs; ++s)
            tma_load_3d(sbase + L::kOffV + j % L::kVTiles * L::kTileBytes + s * (kBN * 128), &p.vmap, s * 64, (tile0 + j) * kBN, kv_head, bar(full));
    };
    auto load_v = [&](int j) -> bool {
        if (!mbar_wait(bar(V_EMPTY + j % L::kVTiles), static_cast<uint32_t>((j / L::kVTiles) & 1) ^ 1)) return false;
        copy_v(j, V_FULL + j % L::kVTiles);
        return true;
    };
    // With a device-side state the maps end at the capacity and not at the visible rows: the last tile's rows from kv_end on bring whatever lies in the cache, and a weight of zero times NaN
    // is NaN.  The warp that feeds the V ring clears them before it hands the tile over (the swizzle stays within a row).  A kernel of its own has it: the text alone
    // cost the others 0.6 % (37 over 3000, 32 / 8 heads of 128).
    [[maybe_unused]] const int whole_tiles = STATE && kv_end % kBN != 0 ? ntiles - 1 : ntiles;   // tiles handed over as they land
    [[maybe_unused]] auto load_last_v = [&](bool ok) {   // a warp; `ok`: lane 0 has handed over the others
        const int j = ntiles - 1, st = j % L::kVTiles;
        if (lane == 0 && ok && mbar_wait(bar(V_EMPTY + st), static_cast<uint32_t>((j / L::kVTiles) & 1) ^ 1)) copy_v(j, V_TAIL);
        __syncwarp();
        if (!mbar_wait_warp(bar(V_TAIL), 0)) return;
        for (int s = 0; s < L::kSlabs; ++s)
            for (uint32_t at = kv_end % kBN * 128 + lane * 16; at < kBN * 128; at += 32 * 16)
                *reinterpret_cast<uint4*>(smem + L::kOffV + st * L::kTileBytes + s * (kBN * 128) + at) = make_uint4(0, 0, 0, 0);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(V_FULL + st));
    };

    if (D == 128 && warp == kTmaWarp) {
        // =============================== TMA producer, K and V tiles ===============================
        auto load_k = [&](int i) -> bool {
            if (!mbar_wait(bar(K_EMPTY + i % kKPairs), static_cast<uint32_t>((i / kKPairs) & 1) ^ 1)) return false;
            issue_k(i);
            return true;
        };
        bool ok = mbar_wait(bar(Q_FULL), 0);
        next_q();
        if (p.gate != nullptr && split_u == 0) {
            const uint32_t t_last = (min(row0 + L::kRows, total_rows) - 1) / G;
            for (uint32_t t = row0 / G + lane; t <= t_last; t += 32)
                prefetch_l2(p.gate + (static_cast<size_t>(t) * p.query_heads + kv_head * G) * D, G * D * 4);
        }
        if (lane == 0) {
            for (int j = 0; ok && j < whole_tiles; ++j) {
                if ((j & 1) == 0 && j + 2 < ntiles) ok = load_k((j >> 1) + 1);
                ok = ok && load_v(j);
            }
        }
        if constexpr (STATE)
            if (whole_tiles < ntiles) load_last_v(ok);
    } else if (warp == kTmaWarp) {
        // =============================== TMA producer, K tiles ===============================
        // Q first: nothing can start without it, and 148 CTAs that fill their rings at once keep L2 busy for over 3 us.  The first pair of K
        // tiles goes along with it, the other stages are asked for when it is in.
        if (lane == 0)
            for (int i = 0; 2 * i < ntiles; ++i) {
                if (i == 1 && !mbar_wait(bar(Q_FULL), 0)) break;
                if (!mbar_wait(bar(K_EMPTY + i % kKPairs), static_cast<uint32_t>((i / kKPairs) & 1) ^ 1)) break;
                issue_k(i);
            }
    } else if (D == 256 && warp == kTmaVWarp) {
        // =============================== TMA producer, V tiles ===============================
        const bool have_q = mbar_wait(bar(Q_FULL), 0);
        // The gate on its way to L2 for the epilogue or the merge: the kv head's G rows of a token are contiguous, a lane takes a token.
        if (p.gate != nullptr && split_u == 0) {
            const uint32_t t_last = (min(row0 + L::kRows, total_rows) - 1) / G;
            for (uint32_t t = row0 / G + lane; t <= t_last; t += 32)
                prefetch_l2(p.gate + (static_cast<size_t>(t) * p.query_heads + kv_head * G) * D, G * D * 4);
        }
        bool ok = have_q;
        if (lane == 0)
            for (int j = 0; ok && j < whole_tiles; ++j) ok = load_v(j);
        if constexpr (STATE)
            if (whole_tiles < ntiles) load_last_v(ok);
    } else if (warp >= kSWarp && warp < kPvWarp) {
        // =============================== S = Q.K^T issuer ===============================
        // The warp stays together and one lane issues (D == 128): loop counters and descriptors live in uniform registers, which an MMA takes them from
        // (from a branch on the lane number an MMA cost 50 to 105 clocks to issue, against the 32 to 64 these run).
        if constexpr (L::kPInTmem) {
            constexpr uint32_t idesc = umma_idesc(kBM, kBN, 0, 0);
            const int rt = RT == 2 ? warp - kSWarp : 0, first = RT == 2 ? 0 : warp - kSWarp;
            constexpr int kStep = RT == 2 ? 1 : L::kIssuers;
            const uint64_t k_desc = umma_desc(sbase + L::kOffK, 16, 1024);
            [[maybe_unused]] const uint64_t q_desc = umma_desc(sbase + L::kOffQ + rt * L::kQBytes, 16, 1024);
            bool ok = rt < live_tiles && mbar_wait_warp(bar(Q_FULL), 0);
            for (int j = first; ok && j < ntiles; j += kStep) {
                const int i = j >> 1, ps = i % kKPairs, buf = rt * L::kGroups + j % L::kGroups;
                // the K pair is there, and the weights that lie in the buffer have been used
                ok = mbar_wait_both(bar(K_FULL + ps), static_cast<uint32_t>((i / kKPairs) & 1), bar(P_EMPTY + buf), static_cast<uint32_t>((j / L::kGroups) & 1) ^ 1);
                if (!ok) break;
                tc_fence_after();
                const uint64_t b = k_desc + ((ps * L::kPairBytes + (j & 1) * (kBN * 128)) >> 4);
                const uint32_t d = tmem_base + L::kColS + buf * kBN;
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        const uint64_t bk = b + (((kk >> 2) * (2 * kBN * 128) + (kk & 3) * 32) >> 4);
                        if constexpr (L::kQInTmem) umma_f16_a_tmem(d, tmem_base + L::kColQ + kk * 8, bk, idesc, kk > 0);
                        else umma_f16(d, q_desc + (((kk >> 2) * (kBM * 128) + (kk & 3) * 32) >> 4), bk, idesc, kk > 0);
                    }
                    umma_commit(bar(S_FULL + buf));
                    if (RT == 1 || (j & 1) == 1 || j + 1 == ntiles) umma_commit(bar(K_EMPTY + ps));   // this warp is through with the pair
                }
                __syncwarp();
            }
        } else {
            // One chain of D/16 MMAs per PAIR of tiles (N = 128: the first tile's scores land in S columns 0-63, the second
            // one's in 64-127): half as many instructions to issue as tile by tile.
            constexpr uint32_t idesc_pair = umma_idesc(kBM, 2 * kBN, 0, 0), idesc_one = umma_idesc(kBM, kBN, 0, 0);
            const uint64_t k_desc = umma_desc(sbase + L::kOffK, 16, 1024);
            bool ok = mbar_wait_warp(bar(Q_FULL), 0);
            for (int i = 0; ok && 2 * i < ntiles; ++i) {
                const int ps = i % kKPairs, n = min(2, ntiles - 2 * i);
                const uint32_t ph = static_cast<uint32_t>(i & 1) ^ 1, idesc = n == 2 ? idesc_pair : idesc_one;
                // both groups have read the previous pair's scores (only the last pair can be a single tile)
                ok = mbar_wait_both(bar(K_FULL + ps), static_cast<uint32_t>((i / kKPairs) & 1), bar(S_EMPTY), ph) && mbar_wait_warp(bar(S_EMPTY + 1), ph);
                if (!ok) break;
                tc_fence_after();
                const uint64_t b = k_desc + ((ps * L::kPairBytes) >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk)
                        umma_f16_a_tmem(tmem_base + L::kColS, tmem_base + L::kColQ + kk * 8, b + (((kk >> 2) * (2 * kBN * 128) + (kk & 3) * 32) >> 4), idesc, kk > 0);
                    umma_commit(bar(S_FULL));         // scores ready for both softmax groups
                    umma_commit(bar(K_EMPTY + ps));   // K stage may be refilled
                }
                __syncwarp();
            }
        }
    } else if (warp == kPvWarp) {
        // =============================== O += P.V issuer ===============================
        if constexpr (D == 128) {
            constexpr uint32_t idesc_o = umma_idesc(kBM, D, 0, 1);
            const uint64_t v_desc = umma_desc(sbase + L::kOffV, kBN * 128, 1024);
            bool ok = true;
            for (int j = 0; ok && j < ntiles; ++j) {
                const int vs = j % L::kVTiles, st = j % L::kGroups;
                const uint32_t ph = static_cast<uint32_t>((j / L::kGroups) & 1);
                const uint64_t b = v_desc + ((vs * L::kTileBytes) >> 4);
#pragma unroll
                for (int rt = 0; rt < RT; ++rt) {
                    if (RT > 1 && rt >= live_tiles) break;
                    const int buf = rt * L::kGroups + st;
                    ok = rt == 0 ? mbar_wait_both(bar(V_FULL + vs), static_cast<uint32_t>((j / L::kVTiles) & 1), bar(P_FULL + buf), ph) : mbar_wait_warp(bar(P_FULL + buf), ph);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < kBN / 16; ++kk)   // V: MN-major, 16 positions per step
                            umma_f16_a_tmem(tmem_base + L::kColO + rt * D, tmem_base + L::kColS + buf * kBN + kk * 8, b + ((kk * (16 * 128)) >> 4), idesc_o, (j > 0 || kk > 0));
                        umma_commit(bar(P_EMPTY + buf));   // the buffer is free for scores, O holds tiles 0..j
                        if (j == ntiles - 1) umma_commit(bar(O_DONE + rt));   // O complete: the epilogue's signal for all groups
                        if (rt + 1 == live_tiles) umma_commit(bar(V_EMPTY + vs));
                    }
                    __syncwarp();
                }
            }
        } else {
            constexpr uint32_t idesc_o = umma_idesc(kBM, D, 0, 1);
            const uint64_t v_desc = umma_desc(sbase + L::kOffV, kBN * 128, 1024), p_desc = umma_desc(sbase + L::kOffP, 16, 1024);
            bool ok = true;
            for (int j = 0; ok && j < ntiles; ++j) {
                const int st = j & 1;
                const uint32_t ph = static_cast<uint32_t>((j >> 1) & 1);
                ok = mbar_wait_both(bar(V_FULL + st), ph, bar(P_FULL + st), ph);
                if (!ok) break;
                tc_fence_after();
                const uint64_t a = p_desc + ((st * L::kPBytes) >> 4), b = v_desc + ((st * L::kTileBytes) >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < kBN / 16; ++kk)
                        umma_f16(tmem_base + L::kColO, a + ((kk * 32) >> 4), b + ((kk * (16 * 128)) >> 4), idesc_o, (j > 0 || kk > 0));
                    umma_commit(bar(P_EMPTY + st));   // P buffer free, O holds tiles 0..j
                    if (j == ntiles - 1) umma_commit(bar(O_DONE));   // O complete: the epilogue's signal for both groups
                    umma_commit(bar(V_EMPTY + st));
                }
                __syncwarp();
            }
        }
    } else {
        // =============================== Q rows ===============================
        // Q: the CTA's rows as fp16 pairs in TMEM (row = lane, dims 2c and 2c+1 in column c), the A operand of every S MMA:
        // read from there it costs no shared-memory bandwidth.  Two of a row's threads store half of the
        // row.  A warp reads its 32 rows four at a time, 128 (fp32: 256) contiguous bytes each, and turns them through
        // its own 4 KB of the P tiles (a load per thread and row touched 32 lines an instruction); the first pair of K
        // tiles is on its way meanwhile.  From the dependency wait to the last row: 0.8 us (two row tiles of 128 dims; 3.8 behind full rings and with
        // a division a row), 3.3 us (one of 256 from HBM; 4.5).
        uint8_t* const turn = smem + L::kOffP + warp * 4096;   // [32 rows][8 chunks of 16 B], chunk c of row r at c ^ (r & 7)
        if (warp < kQWarps) {
            uint4 q[kTurns][8];
            if constexpr (kEarlyQ) {
#pragma unroll
                for (int k = 0; k < kTurns; ++k)
#pragma unroll
                    for (int i = 0; i < 8; ++i) q[k][i] = early_q[k][i];
            } else {
                fetch_q(late_rows, q);
            }
            const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
            const int half = (warp >> 2) & 1;
#pragma unroll
            for (int k = 0; k < kTurns; ++k) {
                const int c0 = 32 * k;
                uint4 (&v)[8] = q[k];
                if constexpr (!L::kQInTmem) {   // the swizzled A operand itself: slab `half * D/128 + c0/32` of the row tile
                    uint8_t* slab = smem + L::kOffQ + rt * L::kQBytes + (half * (D / 128) + c0 / 32) * (kBM * 128) + (warp & 3) * (32 * 128);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int row = 4 * i + turn_row;
                        *reinterpret_cast<uint4*>(slab + row * 128 + ((turn_chunk ^ (row & 7)) << 4)) = v[i];
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int row = 4 * i + turn_row;
                        *reinterpret_cast<uint4*>(turn + row * 128 + ((turn_chunk ^ (row & 7)) << 4)) = v[i];
                    }
                    __syncwarp();
                    uint32_t w[32];
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const uint4 q4 = *reinterpret_cast<const uint4*>(turn + lane * 128 + ((c ^ (lane & 7)) << 4));
                        w[4 * c] = q4.x; w[4 * c + 1] = q4.y; w[4 * c + 2] = q4.z; w[4 * c + 3] = q4.w;
                    }
                    __syncwarp();
                    tmem_st32_bits(tmem_base + lane_base + L::kColQ + half * (D / 4) + c0, w);
                }
            }
            if constexpr (L::kQInTmem) {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
            } else {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            mbar_arrive(bar(Q_FULL));
            // no barrier: what a warp turns its rows in are its own rows of its group's P tile
        }
        // =============================== softmax rows ===============================
        // Groups of 128 threads, one thread per query row in each, take the tiles in turn (a warp reaches the 32 TMEM lanes of its number modulo
        // 4), so as many tiles are in flight: while one group works through its exponentials the others' S arrive and their P.V run.  A row's reference maximum is handed
        // from tile to tile through an 8-byte {value, sequence} word in shared memory; each thread keeps the partial row
        // sum of its own tiles, relative to the reference it last saw.
        const int r = tid & (kBM - 1), grp = (tid >> 7) % L::kGroups;   // row of this thread in its row tile == its TMEM lane; its tiles
        const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t gr = tile_row0 + r;
        const int walked = RT == 1 || rt < live_tiles ? ntiles : 0;
        uint32_t len = 0;
        if (gr < total_rows) {
            const uint32_t token = gr / G;
            const uint64_t l64 = static_cast<uint64_t>(base) + token + 1u;
            len = (token < count && l64 <= p.capacity) ? static_cast<uint32_t>(l64) : 0u;
        }
        volatile unsigned long long* ref = reinterpret_cast<volatile unsigned long long*>(smem + L::kOffRef) + rt * kBM + r;
        auto ref_after = [&](uint32_t seq, float* value) -> bool {   // the reference as tile seq-1 left it
            // Rolled up at 256: less code in the longer of the tile loops, whose warps wait for instructions (0.7 stalls an issue; 0.3 at 128, where it makes no
            // difference).  24 / 4 heads, us a layer back to back: 512 over 8192 125.0 -> 123.7, 300 over 8192 83.1 -> 82.2, 37 over 3001 25.2 -> 24.9.
#pragma unroll (D == 256 ? 1 : 4)
            for (uint32_t spin = 0; spin < kSpin; ++spin) {
                const unsigned long long w = *ref;
                if (static_cast<uint32_t>(w >> 32) == seq) { *value = __uint_as_float(static_cast<uint32_t>(w)); return true; }
            }
            return false;
        };
        float m_known = -INFINITY, l_sum = 0.0f;   // l_sum is relative to m_known
        auto rebase = [&](float m_new) {
            if (m_new != m_known) {
                l_sum *= (m_known == -INFINITY) ? 0.0f : ex2_approx(m_known - m_new);
                m_known = m_new;
            }
        };
        const int buf = rt * L::kGroups + grp;
        const uint32_t s_col = L::kColS + buf * kBN, o_col = L::kColO + rt * D;
        const int nt = L::kGroups == 4 ? (walked + grp + 1) / 2 : walked;
        for (int j = grp; j < nt; j += 2) {
            const int t = L::kGroups == 4 ? 2 * j - grp : j;   // the tile: every second, or with four groups every fourth from the group's first
            const uint32_t ph = static_cast<uint32_t>((t / L::kGroups) & 1);   // parity of the group's tile
            // The loop holds warp-wide loads, stores and votes, so a warp leaves it as a whole: a lane whose wait runs out goes on, with values nobody
            // will see, up to the one vote below.
            bool lost = !mbar_wait(bar(S_FULL + (L::kPInTmem ? buf : rt)), ph);
            tc_fence_after();
            float s[kBN];
            {
                uint32_t lo[32], hi[32];
                tmem_ld32_nowait(tmem_base + lane_addr + s_col, lo);
                tmem_ld32_nowait(tmem_base + lane_addr + s_col + 32, hi);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) { s[i] = __uint_as_float(lo[i]); s[32 + i] = __uint_as_float(hi[i]); }
            }
            if constexpr (!L::kPInTmem) {
                tc_fence_before();
                mbar_arrive(bar(S_EMPTY + buf));   // this row of S is in registers
            }
            const uint32_t pos0 = static_cast<uint32_t>(tile0 + t) * kBN;
            // Raw scores stay unscaled; the softmax scale is folded into the exponent: p = 2^(s*c - m*c).  The loop's instructions count: products and
            // sums go in pairs, maxima three values at a time.  32 / 8 heads of 128, 1024 tokens over 8192: 168.0 -> 163.7 us; 24 / 4 of 256, 512 over
            // 8192: 111.6 -> 110.3.
            // Only the tiles that straddle this row's causal length need the mask.
            if (pos0 + kBN > len) {
#pragma unroll
                for (int i = 0; i < kBN; ++i) s[i] = (pos0 + i < len) ? s[i] : -INFINITY;
            }
            float m4[4] = {s[0], s[1], s[2], s[3]};   // four chains of two values a step
#pragma unroll
            for (int i = 4; i + 8 <= kBN; i += 8)
#pragma unroll
                for (int c = 0; c < 4; ++c) m4[c] = max3(m4[c], s[i + c], s[i + 4 + c]);
#pragma unroll
            for (int c = 0; c < 4; ++c) m4[c] = fmaxf(m4[c], s[kBN - 4 + c]);
            const float mt = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * p.scale_log2;   // scale > 0: the maximum commutes with it
            // the reference as the previous tile (another group's) left it; lazy rescale: keep it unless this tile's
            // maximum outgrew it by more than the threshold
            float m_prev = -INFINITY;
            if (t > 0 && !ref_after(static_cast<uint32_t>(t), &m_prev)) lost = true;
            float alpha = 1.0f, m_new = m_prev;
            if (mt > m_prev + kRescaleThreshold || (m_prev == -INFINITY && mt > -INFINITY)) {
                alpha = (m_prev == -INFINITY) ? 0.0f : ex2_approx(m_prev - mt);
                m_new = mt;
            }
            // published at once (the thread of the row's next tile waits for it): no later work may be scheduled before it
            asm volatile("st.volatile.shared.u64 [%0], %1;" ::"r"(smem_u32(const_cast<unsigned long long*>(ref))),
                         "l"(reference_word(__float_as_uint(m_new), static_cast<uint32_t>(t) + 1u)) : "memory");
            // With four groups it is read back as well: what follows depends on the number found beside it, so no exponential can be scheduled ahead of the store.  (Without
            // that the store came behind all of them, by the compiler's choice and by small changes around it: a tile took 1050 clocks, not 820.)  The value stays the thread's own
            // whatever is found.  Two groups wait less for each other.  Two row tiles of 128, us: 2048 fresh x 8 layers 464.8 with it, 460.5 as it is, 1200 over 4000 1130 and
            // 1117, 4096 over 8192 x 2 1500 and 1469.  At 256 it costs up to 5 % (300 over 8192, 24 / 4 heads), and a shuffle behind the store, which did better in one text of
            // this kernel, 2 % in this one: 512 over 8192 125.8 us a layer back to back as it is, 129.5 with it.
            if constexpr (L::kGroups == 4) {
                uint32_t seq_found;
                asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(seq_found) : "r"(smem_u32(const_cast<unsigned long long*>(ref)) + 4) : "memory");
                m_new = __uint_as_float(own_reference(seq_found, __float_as_uint(m_new)));
            }
            rebase(m_new);
            const float neg_ref = (m_new == -INFINITY) ? 0.0f : -m_new;
            Pair sum = 0;
            uint32_t pk[kBN / 2];
            const Pair scale2 = pack_pair(p.scale_log2, p.scale_log2), ref2 = pack_pair(neg_ref, neg_ref);
#pragma unroll
            for (int i = 0; i < kBN; i += 2) {
                const float2 e = unpack_pair(fma_pair(pack_pair(s[i], s[i + 1]), scale2, ref2));
                const __half2 h = __floats2half2_rn(ex2_approx(e.x), ex2_approx(e.y));
                pk[i >> 1] = *reinterpret_cast<const uint32_t*>(&h);
                // the sum uses the rounded values the MMA will multiply, so numerator and denominator stay consistent
                const float2 hf = __half22float2(h);
                sum = add_pair(sum, pack_pair(hf.x, hf.y));
            }
            {
                const float2 halves = unpack_pair(sum);
                l_sum += halves.x + halves.y;
            }
            // this group's P buffer is free once the P.V of its previous tile has completed
            if constexpr (!L::kPInTmem) {
                if (!mbar_wait(bar(P_EMPTY + buf), ph ^ 1)) lost = true;
                tc_fence_after();
            }
            if (__any_sync(0xffffffffu, alpha != 1.0f || lost) && (t > 0 || __any_sync(0xffffffffu, lost))) {
                // rare: the reference moved.  O holds tiles 0..t-1 once the previous tile's P.V (another group's) has
                // completed; then this warp rescales its 32 rows of O in TMEM before its own P is released.
                if (t > 0 && !mbar_wait(bar(P_EMPTY + rt * L::kGroups + (t - 1) % L::kGroups), static_cast<uint32_t>(((t - 1) / L::kGroups) & 1))) lost = true;
                if (__any_sync(0xffffffffu, lost)) { failed = true; break; }
                tc_fence_after();
#pragma unroll 1
                for (int c0 = 0; c0 < D; c0 += 32) {
                    float o[32];
                    tmem_ld32(tmem_base + lane_addr + o_col + c0, o);
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] *= alpha;
                    tmem_st32(tmem_base + lane_addr + o_col + c0, o);
                }
            }
            if constexpr (L::kPInTmem) {
                tmem_st32_bits(tmem_base + lane_addr + s_col, pk);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");   // and the rescale's stores, if any
            } else {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");   // the rescale's stores, if any
                uint8_t* prow = smem + L::kOffP + buf * L::kPBytes + r * 128;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<uint4*>(prow + ((c ^ (r & 7)) << 4)) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            tc_fence_before();
            mbar_arrive(bar(P_FULL + buf));
        }
        // ---- epilogue: O / sum, gate, store; the columns are divided among a row's threads ----
        const bool partial = nsplit > 1, gated = !partial && p.gate != nullptr;
        const size_t part_row0 = (static_cast<size_t>(split) * p.kv_heads + kv_head) * p.rows_padded + row0;
        constexpr int kCols = D / L::kGroups;
        const int col0 = grp * kCols;
        const RowOffsets<D> rows(warp_row0, turn_row, G, p.query_heads, total_rows);   // worked out anew: no registers for it in between
        const size_t out0 = (static_cast<size_t>(warp_row0 / G) * p.query_heads + kv_head * G) * D + col0 + 4 * turn_chunk;
        float4 g[8];
        auto fetch_gate = [&](int i, int c0) {
            if (i < rows.valid) g[i] = *reinterpret_cast<const float4*>(p.gate + out0 + rows.rel[i] + c0);
        };
        // D == 256: ahead of the last P.V, the next columns' behind the use of these (at 128 there are no registers for that)
        if (D == 256 && gated) {
#pragma unroll
            for (int i = 0; i < 8; ++i) fetch_gate(i, 0);
        }
        if (!failed && walked > 0 && !mbar_wait(bar(O_DONE + rt), 0)) failed = true;
        tc_fence_after();
        {
            float m_final = -INFINITY;
            if (!failed && walked > 0 && !ref_after(static_cast<uint32_t>(walked), &m_final)) failed = true;
            rebase(m_final);
            float* sums = reinterpret_cast<float*>(smem + L::kOffSum + rt * L::kSumStride);
            sums[grp * kBM + r] = failed ? __int_as_float(0x7fc00000) : l_sum;
            // the row tile's threads (a branch over two constant barriers duplicates what follows: 4 % slower with two row tiles)
            if constexpr (RT == 1) asm volatile("bar.sync 2, %0;" ::"n"(L::kSoftmaxThreads) : "memory");
            else asm volatile("bar.sync %0, 256;" ::"r"(2 + rt) : "memory");
            l_sum = sums[r] + sums[kBM + r];
            if constexpr (L::kGroups == 4) l_sum += sums[2 * kBM + r] + sums[3 * kBM + r];
            // The warp's O may be read.  A sum that is NaN, because another of the row's threads gave up or because of the data, is its own row's affair.
            const bool have_o = walked > 0 && !__any_sync(0xffffffffu, failed);
            if (l_sum != l_sum) failed = true;
            const float m_ref = m_final;
            const float inv = l_sum > 0.0f ? 1.0f / l_sum : 0.0f;
            if (partial && gr < total_rows && grp == 0)   // a poisoned or empty partial is recognised by its sum
                p.part_ml[part_row0 + rt * kBM + r] = make_float2(m_ref, failed ? __int_as_float(0x7fc00000) : (len == 0 ? 0.0f : l_sum));
            // Rows leave 32 columns at a time through the same 4 KB per warp: read back four rows an instruction, 128
            // contiguous bytes each, so that the gate is fetched and the result stored in whole lines.
            float* const dst = partial ? p.part_o + (part_row0 + (warp_row0 - row0) + turn_row) * D + col0 + 4 * turn_chunk : p.out + out0;
            const bool zero = len == 0 && !partial;
            const float factor = failed ? __int_as_float(0x7fc00000) : partial ? 1.0f : inv;
#pragma unroll 1
            for (int c0 = 0; c0 < kCols; c0 += 32) {
                [[maybe_unused]] float4 gs[8];
                if (gated) {
                    if constexpr (D == 256) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            gs[i].x = 1.0f / (1.0f + __expf(-g[i].x)); gs[i].y = 1.0f / (1.0f + __expf(-g[i].y));
                            gs[i].z = 1.0f / (1.0f + __expf(-g[i].z)); gs[i].w = 1.0f / (1.0f + __expf(-g[i].w));
                        }
                    }
                    if (D == 128 || c0 + 32 < kCols) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) fetch_gate(i, D == 128 ? c0 : c0 + 32);
                    }
                }
                float o[32];
                // tcgen05.ld is warp-collective: every lane takes part, rows past the launch only skip the store
                if (have_o) {
                    tmem_ld32(tmem_base + lane_addr + o_col + col0 + c0, o);
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = 0.0f;
                }
                if (zero && !failed) {   // no position visible: zeros whatever lies there
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = 0.0f;
                }
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<float4*>(turn + lane * 128 + ((c ^ (lane & 7)) << 4)) =
                        make_float4(o[4 * c] * factor, o[4 * c + 1] * factor, o[4 * c + 2] * factor, o[4 * c + 3] * factor);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int row = 4 * i + turn_row;
                    float4 v = *reinterpret_cast<const float4*>(turn + row * 128 + ((turn_chunk ^ (row & 7)) << 4));
                    if (gated) {
                        if constexpr (D == 256) {
                            v.x *= gs[i].x; v.y *= gs[i].y; v.z *= gs[i].z; v.w *= gs[i].w;
                        } else {
                            v.x *= 1.0f / (1.0f + __expf(-g[i].x)); v.y *= 1.0f / (1.0f + __expf(-g[i].y));
                            v.z *= 1.0f / (1.0f + __expf(-g[i].z)); v.w *= 1.0f / (1.0f + __expf(-g[i].w));
                        }
                    }
                    if (i < rows.valid) *reinterpret_cast<float4*>(dst + (partial ? static_cast<uint32_t>(4 * i * D) : rows.rel[i]) + c0) = v;
                }
                __syncwarp();
            }
        }
    }

    // ---- teardown: every role arrives here, with or without a timeout; TMEM is always released ----
    tc_fence_before();
    __syncthreads();
    if (warp == kSWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(L::kTmemCols) : "memory");
    }
}

// ---- merge of the KV splits: out = sum_s O_s 2^(m_s - M) / sum_s l_s 2^(m_s - M), gate -------------------------------
struct PrefillMergeParams {
    const float* part_o;
    const float2* part_ml;
    const float* gate;
    float* out;
    uint32_t kv_splits, kv_heads, query_heads, rows_padded, total_rows;   // total_rows = token_count * G per kv head
};

template <int D, uint32_t MAX_SPLITS>   // kv_splits <= MAX_SPLITS
__global__ void __launch_bounds__(256) prefill_merge_kernel(const __grid_constant__ PrefillMergeParams p) {
    constexpr int VPR = D / 4;   // float4 per row
    pdl_launch_dependents();
    pdl_wait();   // the partials are the attention kernel's output
    const uint32_t kv_head = blockIdx.y, G = p.query_heads / p.kv_heads;
    const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= static_cast<size_t>(p.total_rows) * VPR) return;
    const uint32_t gr = static_cast<uint32_t>(idx / VPR), c = static_cast<uint32_t>(idx % VPR) * 4;
    const uint32_t token = gr / G, head = kv_head * G + gr % G;
    const size_t off = (static_cast<size_t>(token) * p.query_heads + head) * D + c;
    float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (p.gate != nullptr) g = *reinterpret_cast<const float4*>(p.gate + off);
    // every load of the row's splits, and the gate's, is issued before the first is used; an empty split's O is zeros and counts for nothing
    float2 ml[MAX_SPLITS];
    float4 o[MAX_SPLITS];
#pragma unroll
    for (uint32_t s = 0; s < MAX_SPLITS; ++s) {
        ml[s] = make_float2(-INFINITY, 0.0f);
        o[s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (s < p.kv_splits) {
            const size_t row = (static_cast<size_t>(s) * p.kv_heads + kv_head) * p.rows_padded + gr;
            ml[s] = p.part_ml[row];
            o[s] = *reinterpret_cast<const float4*>(p.part_o + row * D + c);
        }
    }
    float M = -INFINITY;
#pragma unroll
    for (uint32_t s = 0; s < MAX_SPLITS; ++s)
        if (!(ml[s].y <= 0.0f) && ml[s].x != -INFINITY) M = fmaxf(M, ml[s].x);   // keeps NaN partials in play
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float lsum = 0.0f;
#pragma unroll
    for (uint32_t s = 0; s < MAX_SPLITS; ++s) {
        if (ml[s].y <= 0.0f || (ml[s].x == -INFINITY && ml[s].y == ml[s].y)) continue;   // a sum that is NaN poisons its row
        const float w = exp2f(ml[s].x - M);
        acc.x = fmaf(o[s].x, w, acc.x); acc.y = fmaf(o[s].y, w, acc.y); acc.z = fmaf(o[s].z, w, acc.z); acc.w = fmaf(o[s].w, w, acc.w);
        lsum = fmaf(ml[s].y, w, lsum);
    }
    const float inv = lsum > 0.0f ? 1.0f / lsum : (lsum == lsum ? 0.0f : lsum);
    float4 v = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
    if (p.gate != nullptr) {
        v.x *= 1.0f / (1.0f + __expf(-g.x)); v.y *= 1.0f / (1.0f + __expf(-g.y));
        v.z *= 1.0f / (1.0f + __expf(-g.z)); v.w *= 1.0f / (1.0f + __expf(-g.w));
    }
    *reinterpret_cast<float4*>(p.out + off) = v;
}

// ---- pre-pass: dequantise [0, rows) of every kv head to fp16 ---------------------------------------------------------
struct DequantParams {
    b200kv_view view;
    __half* k_out;       // [kv_heads][scratch_rows][D]
    __half* v_out;
    uint32_t rows;       // positions that hold data; rows from here up to row_end are zero-filled
    uint32_t scratch_rows;
    uint32_t row_begin;  // this launch converts positions [row_begin, row_end): the rows below were converted ahead of
    uint32_t row_end;    // the chunk (b200kv_prefill_prepare), possibly beside the previous layer's attention
    uint32_t side0;      // first side the launch converts
};

// A thread converts kDequantUnits pieces of 8 elements, a block's threads side by side and all of a thread's loads in flight together: a warp
// reads 256 contiguous bytes and writes 512.  Bound by the bytes to and from L2 (19 MB in, 36 MB out for 8704 positions of 4 kv heads of 256);
// with one piece of 16 elements a thread, in four waves of blocks, a layer of 512 tokens over 8192 took 118.2 us in place of 114.8, one of 128
// tokens (8 kv heads of 128) 43.0 in place of 41.0.
constexpr int kDequantUnits = 8;
template <int D>
__global__ void __launch_bounds__(256, 4) dequant_prefix_kernel(const __grid_constant__ DequantParams p) {
    constexpr uint32_t CPR = D / 8;
    pdl_launch_dependents();
    pdl_wait();   // the cache rows of this chunk come from the append kernel just before
    const uint32_t head = blockIdx.y, side = p.side0 + blockIdx.z;   // side 0 = K, 1 = V
    const uint32_t mode = p.view.quant_mode;
    const bool q8 = side == 0 ? (mode == B200KV_Q8_F16 || mode == B200KV_Q8_Q8) : (mode == B200KV_F16_Q8 || mode == B200KV_Q8_Q8);
    const uint32_t nblk = D / p.view.qblock;
    const uint64_t head_row0 = static_cast<uint64_t>(head) * p.view.capacity;
    const int8_t* q = (side == 0 ? p.view.key_q8 : p.view.value_q8) + head_row0 * D;
    const __half* sc = static_cast<const __half*>(side == 0 ? p.view.key_scales : p.view.value_scales) + head_row0 * nblk;
    const __half* f16 = static_cast<const __half*>(side == 0 ? p.view.key_f16 : p.view.value_f16) + head_row0 * D;
    __half* out = (side == 0 ? p.k_out : p.v_out) + static_cast<size_t>(head) * p.scratch_rows * D;
    const uint32_t row0 = p.row_begin + blockIdx.x * (256 * kDequantUnits / CPR) + threadIdx.x / CPR, c = threadIdx.x % CPR;
    uint4 v[kDequantUnits];   // int8: the first two words
    __half scale[kDequantUnits];
#pragma unroll
    for (int i = 0; i < kDequantUnits; ++i) {
        const uint32_t pos = row0 + i * (256 / CPR);
        // padding rows of the last tile are zeroed: P is 0 there, but 0 * (stale NaN) would still poison O
        v[i] = make_uint4(0, 0, 0, 0);
        scale[i] = __ushort_as_half(0);
        if (pos >= p.rows) continue;
        const size_t at = static_cast<size_t>(pos) * D + c * 8;
        if (q8) {
            const uint2 raw = *reinterpret_cast<const uint2*>(q + at);
            v[i].x = raw.x; v[i].y = raw.y;
            scale[i] = sc[static_cast<size_t>(pos) * nblk + (nblk == 1 ? 0 : c / 4)];
        } else {
            v[i] = *reinterpret_cast<const uint4*>(f16 + at);
        }
    }
#pragma unroll
    for (int i = 0; i < kDequantUnits; ++i) {
        const uint32_t pos = row0 + i * (256 / CPR);
        if (pos >= p.row_end) break;
        *reinterpret_cast<uint4*>(out + static_cast<size_t>(pos) * D + c * 8) = q8 ? dequant8(make_uint2(v[i].x, v[i].y), scale[i]) : v[i];
    }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn tc5_encoder() {
    static EncodeFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeFn>(sym);
        else
            (void)cudaGetLastError();
    });
    return fn;
}

// Planes [kv_heads][plane_rows][d] of which `rows` rows a head are read.
bool encode_f16_plane(CUtensorMap* map, const void* base, uint32_t d, uint64_t rows, uint64_t plane_rows, uint32_t kv_heads) {
    EncodeFn fn = tc5_encoder();
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {d, rows, kv_heads};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(d) * 2, plane_rows * d * 2};
    const cuuint32_t box[3] = {64, kBN, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// An fp16 side of the cache is read where it lies; only int8 sides go through the scratch.  (The map ends at the rows the launch may see, so the last tile's
// other rows come as zeros, as in the scratch; with a device-side state that is the capacity, and the kernel clears what lies past the visible rows.)  24 / 4 heads of
// 256, us a layer: 67 over 4826 30.8 -> 24.0.  Where the caller has converted rows ahead
// (b200kv_prefill_prepare) the copy is completed and used.  A chunk that sees no more than one tile goes through the scratch as well, which is no gain (fp16 caches, 16 layers, us, so -> in
// place: 16 tokens of 32 / 8 heads of 128 219 -> 181, 20 fp32 tokens of 24 / 4 of 256 263 -> 235): tests/test_prefill_prepass_gpu.py looks for the copy behind such a call.
struct Sides { bool k, v; };   // sides that go through the scratch
Sides scratch_sides(const b200kv_view& view, uint64_t rows, uint32_t prepared_rows) {
    const auto direct = [&](bool q8, const void* plane) {
        return !q8 && prepared_rows == 0 && rows > kBN && (reinterpret_cast<uintptr_t>(plane) & 15) == 0 && view.capacity * view.head_dim * 2 < (1ull << 40);
    };
    return {!direct(is_k_q8(view.quant_mode), view.key_f16), !direct(is_v_q8(view.quant_mode), view.value_f16)};
}

// The pre-pass over positions [row_begin, row_end) of every kv head, of one or both sides.
template <int D>
int launch_dequant(const b200kv_view& view, __half* k_scratch, __half* v_scratch, uint32_t rows, uint32_t scratch_rows,
                   uint32_t row_begin, uint32_t row_end, Sides sides, cudaStream_t stream) {
    if (row_begin >= row_end || (!sides.k && !sides.v)) return B200KV_OK;
    DequantParams dp{};
    dp.side0 = sides.k ? 0 : 1;
    dp.view = view;
    dp.k_out = k_scratch;
    dp.v_out = v_scratch;
    dp.rows = rows;
    dp.scratch_rows = scratch_rows;
    dp.row_begin = row_begin;
    dp.row_end = row_end;
    constexpr uint32_t rows_per_block = 256 * kDequantUnits / (D / 8);
    const unsigned blocks = (row_end - row_begin + rows_per_block - 1) / rows_per_block;
    B200KV_CUDA_TRY(launch_kernel(dequant_prefix_kernel<D>, dim3(blocks, view.kv_heads, sides.k && sides.v ? 2 : 1), dim3(256), 0, stream, true, dp));
    return B200KV_OK;
}

template <int D, int RT, bool STATE>
int launch_tc5(const b200kv_view& view, Tc5Params& p, __half* k_scratch, __half* v_scratch, uint32_t rows, uint32_t prepared_rows,
               cudaStream_t stream) {
    using L = Layout<D, RT>;
    static std::atomic<uint64_t> done{0};   // one per kernel instantiation: devices that have opted in
    const cudaError_t attr_err = opt_in_dynamic_smem(reinterpret_cast<const void*>(prefill_tc5_kernel<D, RT, STATE>), L::kAlloc, done);
    if (attr_err != cudaSuccess) { set_last_cuda_error(attr_err, "cudaFuncSetAttribute(prefill_tc5)"); return B200KV_ERR_CUDA; }
    if (rows > 0) {
        const int rc = launch_dequant<D>(view, k_scratch, v_scratch, rows, p.scratch_rows, prepared_rows < rows ? prepared_rows : rows,
                                         p.scratch_rows, scratch_sides(view, rows, prepared_rows), stream);
        if (rc != B200KV_OK) return rc;
    }
    const uint32_t G = p.query_heads / p.kv_heads;
    const uint32_t row_tiles = (p.token_count * G + L::kRows - 1) / L::kRows;
    B200KV_CUDA_TRY(launch_kernel(prefill_tc5_kernel<D, RT, STATE>, dim3(row_tiles * p.kv_heads * p.kv_splits), dim3(L::kThreads), L::kAlloc, stream, true, p));
    if (p.kv_splits > 1) {
        PrefillMergeParams mp{};
        mp.part_o = p.part_o;
        mp.part_ml = p.part_ml;
        mp.gate = p.gate;
        mp.out = p.out;
        mp.kv_splits = p.kv_splits;
        mp.kv_heads = p.kv_heads;
        mp.query_heads = p.query_heads;
        mp.rows_padded = p.rows_padded;
        mp.total_rows = p.token_count * G;
        const size_t work = static_cast<size_t>(mp.total_rows) * (D / 4);
        // A thread's loads are laid out for the most splits of its kernel: 38, 64, 93 and 114 registers, i.e. six, four, two and two blocks an SM.  24 / 4 heads
        // of 256, us a layer, for 4 and 16 alone -> these: 128 over 8192 (6 splits) 47.5 -> 44.7, 37 over 3001 (11) 26.5 -> 25.8.
        const auto merge = p.kv_splits <= 4   ? prefill_merge_kernel<D, 4>
                           : p.kv_splits <= 8  ? prefill_merge_kernel<D, 8>
                           : p.kv_splits <= 12 ? prefill_merge_kernel<D, 12>
                                               : prefill_merge_kernel<D, kMaxKvSplits>;
        B200KV_CUDA_TRY(launch_kernel(merge, dim3(static_cast<unsigned>((work + 255) / 256), p.kv_heads), dim3(256), 0, stream, true, mp));
    }
    return B200KV_OK;
}

}  // namespace

size_t prefill_tc5_workspace_bytes(uint32_t rows, uint32_t kv_heads, uint32_t head_dim) {
    const size_t r = (static_cast<size_t>(rows) + kBN - 1) / kBN * kBN;
    return 2 * r * kv_heads * head_dim * sizeof(__half) + 1024;   // K and V planes, 1 KB to align the base
}

// Extra workspace that lets a launch split the KV range of every row tile over several CTAs (partials of `splits` splits).
size_t prefill_tc5_split_bytes(uint32_t token_count, uint32_t query_heads, uint32_t kv_heads, uint32_t head_dim, uint32_t splits) {
    if (kv_heads == 0 || query_heads % kv_heads != 0) return 0;
    const size_t rows_padded = (static_cast<size_t>(token_count) * (query_heads / kv_heads) + kBM - 1) / kBM * kBM;
    return static_cast<size_t>(splits) * kv_heads * rows_padded * (head_dim + 2) * sizeof(float);
}

// How many KV splits: the number with the least estimated time, for `units` CTAs of one or two row tiles, up to `tiles` KV tiles and `average` of them.  A wave
// of a CTA an SM (148 where the costs were fitted) costs its tiles and a few us; CTAs take the place of one another as they end, so a last wave that is not full may cost less than a whole
// one, and from the second wave on the length that counts may lie between the longest causal range and the average; a split costs its partials' way out
// and back, and the merge.  The constants of single row tiles are fitted to 66 (head_dim 128) and 93 (256) chunks of 16 to 2048 tokens over 0 to 32000 at 32 / 8 and 24 / 4
// heads, every number of splits timed: the choice is 0.4 and 0.3 % above the best on average, 6.5 and 5 % at most (1.5 and 0.6, 12 and 15 % with the constants before).  us a layer, graphs of
// 16 layers (4 from 1000 tokens on) with the store kernel, q8_0, in a short burst, the choice marked *:
//   32 heads of 128:  37 over 3000 (16 units):  1: 34.3, 4: 19.2, 6: 19.2, *9: 17.9, 10: 24.2       128 over 8192 (32):  1: 69, 2: 46.2, *4: 33.8, 5: 48
//                     300 over 300 (80):  *1: 15.0, 2: 22.7       300 over 8192:  1: 80, 2: 82, *3: 64.6, 4: 76       461 over 8192 (120):  *1: 83, 2: 87, 3: 94
//   24 of 256:        20 over 16000 (4):  8: 53, 12: 43, *16: 40                     37 over 3000 (8):  1: 46, 4: 23.1, 8: 21.3, 11: 20.3, *12: 19.9, 14: 20.5, 16: 20.3
//                     128 over 8192 (24):  1: 100, 4: 43.9, *6: 39.9, 7: 58          300 over 8192 (60):  1: 104, *2: 70, 3: 96
//                     300 over 300 (60):  1: 21.4, *2: 21.7, 3: 29.2           1024 over 16000 (192):  1: 395, *2: 376, 3: 405
//                     461 over 8192 (88):  1: 122, 2: 126, *3: 103, 4: 116           512 over 8192 (96):  1: 108, 2: 125, *3: 106, 4: 125 (in a long run, at the power limit, 125 and 125 for 1 and 3)
// Two row tiles a CTA have costs of their own.  They were fitted when the weights still went through shared memory; as the loop is now:
//                     1200 over 4000 (152):  1: 145.5, *2: 144.3, 3: 144.9        1200 over 8192:  1: 262, 2: 236, *3: 226, 4: 228
//                     1600 over 4000 (200):  *1: 155, 2: 159             1500 over 20000 (192):  1: 615, 2: 529, *3: 530, 4: 624
//                     3000 over 8192 (376):  *1: 493, 2: 537             4096 over 8192 (512):  *1: 673, 2: 707
// (Another number of splits is another reference for the same row, and its fp16 weights round otherwise: 37 over 3001 at 24 / 4 heads, 12 splits for 11, moved by 2.4e-4 of its
// norm; 4.12e-4 off float64 with 12, 4.13e-4 with 11.)
static uint32_t pick_kv_splits(uint32_t units, uint32_t tiles, double average, uint32_t most, uint32_t head_dim, uint32_t tiles_per_cta, uint32_t sms) {
    struct Costs { double tile_us, wave_us, last_wave, longest, merge_us, partial_us; };
    const Costs c = tiles_per_cta == 2 ? Costs{1.0, 3.0, 0.6, 1.0, 0.0, 0.07} : head_dim == 256 ? Costs{0.62, 12.4, 0.5, 0.42, 0.0, 0.024} : Costs{0.43, 1.95, 1.0, 0.07, 1.3, 0.017};
    uint32_t best = 1;
    double best_us = 0.0;
    for (uint32_t s = 1; s <= kMaxKvSplits && s <= (most > 1 ? most : 1); ++s) {
        const uint64_t ctas = static_cast<uint64_t>(units) * s, full = ctas / sms, rest = ctas % sms;
        const double waves = static_cast<double>(full) + (rest == 0 ? 0.0 : full == 0 ? 1.0 : c.last_wave + (1.0 - c.last_wave) * static_cast<double>(rest) / sms);
        const double walked = ctas <= sms ? tiles : c.longest * tiles + (1.0 - c.longest) * average;
        const double us = waves * (walked * c.tile_us / s + c.wave_us) + (s > 1 ? c.merge_us + c.partial_us * static_cast<double>(ctas) : 0.0);
        if (s == 1 || us < best_us) { best = s; best_us = us; }
    }
    return best;
}

// Returns B200KV_ERR_UNSUPPORTED when this path cannot run (no workspace, no TMA encoder); the caller then uses the
// register-resident mma.sync kernel.
int launch_prefill_tc5(const b200kv_view& view, const void* q, int q_is_f16, const float* gate, float* out,
                       uint32_t token_count, uint32_t base_position, const b200kv_prefill_state* prefill_state,
                       uint32_t query_heads, float scale, void* workspace, size_t workspace_bytes, uint32_t prepared_rows,
                       cudaStream_t stream) {
    // rows the chunk can see: known on the host unless a device-side state overrides it (then: the whole cache)
    uint64_t rows = prefill_state ? view.capacity : static_cast<uint64_t>(base_position) + token_count;
    if (rows > view.capacity) rows = view.capacity;
    const uint32_t scratch_rows = static_cast<uint32_t>((rows + kBN - 1) / kBN * kBN);
    if (workspace == nullptr || workspace_bytes < prefill_tc5_workspace_bytes(static_cast<uint32_t>(rows), view.kv_heads, view.head_dim))
        return B200KV_ERR_UNSUPPORTED;
    if (static_cast<uint64_t>(view.kv_heads) * scratch_rows > 0x7fffffffull) return B200KV_ERR_UNSUPPORTED;
    uint8_t* ws = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(workspace) + 1023) & ~static_cast<uintptr_t>(1023));
    __half* k_scratch = reinterpret_cast<__half*>(ws);
    __half* v_scratch = k_scratch + static_cast<size_t>(view.kv_heads) * scratch_rows * view.head_dim;
    Tc5Params p{};
    const Sides sides = scratch_sides(view, rows, prepared_rows);
    const auto encode = [&](CUtensorMap* map, bool scratch, const __half* copy, const void* plane) {
        return scratch ? encode_f16_plane(map, copy, view.head_dim, scratch_rows, scratch_rows, view.kv_heads)
                       : encode_f16_plane(map, plane, view.head_dim, rows, view.capacity, view.kv_heads);
    };
    if (!encode(&p.kmap, sides.k, k_scratch, view.key_f16) || !encode(&p.vmap, sides.v, v_scratch, view.value_f16)) return B200KV_ERR_UNSUPPORTED;
    p.q = q;
    p.q_is_f16 = q_is_f16;
    p.gate = gate;
    p.out = out;
    p.token_count = token_count;
    p.base_position = base_position;
    p.prefill_state = prefill_state;
    p.query_heads = query_heads;
    p.kv_heads = view.kv_heads;
    p.capacity = view.capacity;
    p.scratch_rows = scratch_rows;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.sms = device_sms();
    // head_dim 128: two row tiles per CTA where that still leaves every SM a CTA.  Both take the same K and V tiles, and set-up, Q and output come once for both.
    // Fewer rows spread better as single tiles.  (With a device-side state single tiles always: their kernel is the one that clears stale rows.)
    const uint32_t row_tiles_128 = static_cast<uint32_t>((static_cast<uint64_t>(token_count) * (query_heads / view.kv_heads) + kBM - 1) / kBM);
    const uint32_t tiles_per_cta = view.head_dim == 128 && prefill_state == nullptr && (row_tiles_128 + 1) / 2 * static_cast<uint64_t>(view.kv_heads) >= p.sms ? 2u : 1u;
    // KV split when the row tiles alone leave SMs idle and the caller's workspace has room for the partials
    p.kv_splits = 1;
    {
        const uint32_t row_tiles = (row_tiles_128 + tiles_per_cta - 1) / tiles_per_cta;
        // A device-side state leaves the range unknown here (no split).  Every split walks a few tiles: three of the longest range, or,
        // where the chunk's own triangle is longer than its prefix, eight of the prefix, which is all that its first rows see.
        const uint32_t tiles = static_cast<uint32_t>((rows + kBN - 1) / kBN), prefix_tiles = (base_position + kBN - 1) / kBN;
        const uint32_t most = prefill_state != nullptr ? 1 : base_position >= token_count ? tiles / 3 : prefix_tiles / 8;
        const double average = std::min<double>(tiles, (base_position + 0.5 * token_count) / kBN);
        uint32_t want = pick_kv_splits(row_tiles * view.kv_heads, tiles, average, most, view.head_dim, tiles_per_cta, p.sms);
        const size_t scratch = prefill_tc5_workspace_bytes(static_cast<uint32_t>(rows), view.kv_heads, view.head_dim);
        while (want > 1 && workspace_bytes < scratch + 1024 + prefill_tc5_split_bytes(token_count, query_heads, view.kv_heads, view.head_dim, want)) --want;
        if (want > 1) {
            p.kv_splits = want;
            p.rows_padded = row_tiles_128 * kBM;   // what the workspace is sized for; rows past the chunk's are never stored
            uint8_t* part = reinterpret_cast<uint8_t*>(v_scratch + static_cast<size_t>(view.kv_heads) * scratch_rows * view.head_dim);
            part = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(part) + 1023) & ~static_cast<uintptr_t>(1023));
            p.part_o = reinterpret_cast<float*>(part);
            p.part_ml = reinterpret_cast<float2*>(p.part_o + static_cast<size_t>(want) * view.kv_heads * p.rows_padded * view.head_dim);
        }
    }
    const auto launch = prefill_state != nullptr ? (view.head_dim == 256 ? launch_tc5<256, 1, true> : launch_tc5<128, 1, true>)
                        : view.head_dim == 256   ? launch_tc5<256, 1, false>
                        : tiles_per_cta == 2     ? launch_tc5<128, 2, false>
                                                 : launch_tc5<128, 1, false>;
    return launch(view, p, k_scratch, v_scratch, static_cast<uint32_t>(rows), prepared_rows, stream);
}

// The pre-pass alone, for positions [0, prepared_rows), into the scratch laid out for a chunk that sees `rows` positions
// (the same `rows` the attention call derives: base_position + token_count, or the capacity with a device-side state).
int launch_prefill_tc5_prepare(const b200kv_view& view, uint32_t prepared_rows, uint64_t rows, void* workspace, size_t workspace_bytes,
                               cudaStream_t stream) {
    if (rows > view.capacity) rows = view.capacity;
    if (prepared_rows > rows) return B200KV_ERR_RANGE;
    const uint32_t scratch_rows = static_cast<uint32_t>((rows + kBN - 1) / kBN * kBN);
    if (workspace == nullptr || workspace_bytes < prefill_tc5_workspace_bytes(static_cast<uint32_t>(rows), view.kv_heads, view.head_dim))
        return B200KV_ERR_WORKSPACE;
    if (static_cast<uint64_t>(view.kv_heads) * scratch_rows > 0x7fffffffull) return B200KV_ERR_UNSUPPORTED;
    uint8_t* ws = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(workspace) + 1023) & ~static_cast<uintptr_t>(1023));
    __half* k_scratch = reinterpret_cast<__half*>(ws);
    __half* v_scratch = k_scratch + static_cast<size_t>(view.kv_heads) * scratch_rows * view.head_dim;
    return view.head_dim == 128 ? launch_dequant<128>(view, k_scratch, v_scratch, prepared_rows, scratch_rows, 0, prepared_rows, Sides{true, true}, stream)
                                : launch_dequant<256>(view, k_scratch, v_scratch, prepared_rows, scratch_rows, 0, prepared_rows, Sides{true, true}, stream);
}

}  // namespace b200kv
