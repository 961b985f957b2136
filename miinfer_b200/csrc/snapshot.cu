// Prefix snapshot / restore of one layer's KV cache.
//
// The blob layout is the raw compact layout of MIInfer's
// AttentionLayerKvCacheStorage::download_raw / upload_raw
// (src/prefill_v2/kv_cache.cpp:214-369): K first, per kv head the int8 slice of
// `tokens` rows followed by that head's scale slice (or one fp16 slice), then V
// the same way.  The reference issues 2-4 memcpys per kv head; here a snapshot in
// device memory is one kernel launch over all planes (and, for the snapshot pool, over
// all layers), as is the clone from cache to cache; to and from host memory every plane
// is ONE strided 2D copy (row = one head's `tokens` positions, source pitch =
// capacity, destination pitch = the per-head record).
#include "kv_common.cuh"

#include <cuda.h>   // types and enums only; the entry point is fetched at run time

namespace b200kv {

// ---- device-to-device copies of strided spans -----------------------------------------------------------------
// A snapshot is a set of spans (one kv head's `tokens` rows of one plane), each contiguous on both sides.  One launch
// takes the spans of up to kCopyLayers layers.  Bound by HBM: every byte is read once and written once.  The spans are cut
// into chunks of kCopyChunk bytes that the CTAs of a grid sized to the device take in turn, so a launch has no tail of long
// spans however many layers, heads and rows it covers; a thread keeps kCopyUnroll 16-byte loads in flight.
//   Alignment: cache planes start on 16 bytes but a blob's slices start wherever the ones before them end (two bytes
// per row and scale), so the store side is aligned first and a load that is then misaligned is put together from the two
// aligned 16-byte words it straddles (the second one is the neighbour thread's first: an L1 hit).
// Measured, 16 layers x 4 kv heads x 4096 rows x d = 256 q8_0 (142.6 MB, read and written both times): capture + restore 1138 us as 128
// 2D copies (4 us of host time each), 99 us as two launches of this kernel.
constexpr int kCopyLayers = 48;
constexpr uint32_t kCopyChunk = 16384;
constexpr int kCopyUnroll = 4;
constexpr int kCopyThreads = 256;

struct CopyLayer {
    const uint8_t* src[4];
    uint8_t* dst[4];
    uint64_t src_rows, dst_rows;   // rows between consecutive heads on a cache side (its capacity); unused on a blob side
};
struct CopyParams {
    CopyLayer layer[kCopyLayers];
    uint32_t layers, planes, heads;
    uint32_t row_bytes[4];         // bytes of one row of each plane
    uint64_t tokens;
    uint64_t src_record[4];        // != 0: bytes between consecutive heads of that plane (a blob) instead of rows x row_bytes
    uint64_t dst_record[4];
    uint32_t chunks[4];            // chunks of one span of each plane
    uint32_t span_chunks;          // their sum: chunks of one head of one layer
    uint32_t total_chunks;
};

__device__ __forceinline__ uint4 load16_unaligned(const uint8_t* src, uint32_t shift) {   // shift = src & 15, even
    const uint4* a = reinterpret_cast<const uint4*>(src - shift);
    const uint4 x = __ldg(a);
    if (shift == 0) return x;
    const uint4 y = __ldg(a + 1);
    const uint32_t w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    const uint32_t first = shift >> 2, bits = (shift & 3u) * 8u;
    uint32_t v[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) v[i] = first == 0 ? w[i] : first == 1 ? w[i + 1] : first == 2 ? w[i + 2] : w[min(i + 3, 7)];
    return make_uint4(__funnelshift_r(v[0], v[1], bits), __funnelshift_r(v[1], v[2], bits), __funnelshift_r(v[2], v[3], bits),
                      __funnelshift_r(v[3], v[4], bits));
}

__global__ void __launch_bounds__(kCopyThreads) copy_spans_kernel(const __grid_constant__ CopyParams p) {
    for (uint32_t c = blockIdx.x; c < p.total_chunks; c += gridDim.x) {
        const uint32_t span = c / p.span_chunks;
        uint32_t k = c - span * p.span_chunks;
        const uint32_t l = span / p.heads, head = span - l * p.heads;
        int plane = 0;
        while (k >= p.chunks[plane]) k -= p.chunks[plane++];
        const CopyLayer& y = p.layer[l];
        const uint64_t row = p.row_bytes[plane], bytes = p.tokens * row;
        const uint8_t* src = y.src[plane] + head * (p.src_record[plane] ? p.src_record[plane] : y.src_rows * row);
        uint8_t* dst = y.dst[plane] + head * (p.dst_record[plane] ? p.dst_record[plane] : y.dst_rows * row);
        // the chunk [b0, b1) of the span; inner boundaries lie on 16-byte boundaries of the store side
        const uint64_t skew = (16u - (reinterpret_cast<uintptr_t>(dst) & 15u)) & 15u;
        const uint64_t b0 = k == 0 ? 0 : min(bytes, skew + static_cast<uint64_t>(k) * kCopyChunk);
        const uint64_t b1 = k + 1 == p.chunks[plane] ? bytes : min(bytes, skew + static_cast<uint64_t>(k + 1) * kCopyChunk);
        const uint64_t v0 = min(b1, b0 == 0 ? skew : b0), n16 = (b1 - v0) / 16;
        const uint32_t shift = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src + v0) & 15u);
        for (uint64_t i = threadIdx.x; i < n16; i += kCopyThreads * kCopyUnroll) {
            uint4 r[kCopyUnroll];
#pragma unroll
            for (int u = 0; u < kCopyUnroll; ++u)
                if (i + u * kCopyThreads < n16) r[u] = load16_unaligned(src + v0 + (i + u * kCopyThreads) * 16, shift);
#pragma unroll
            for (int u = 0; u < kCopyUnroll; ++u)
                if (i + u * kCopyThreads < n16) *reinterpret_cast<uint4*>(dst + v0 + (i + u * kCopyThreads) * 16) = r[u];
        }
        // the unaligned ends, in 2-byte units (every plane holds 2-byte or wider units)
        for (uint64_t b = b0 + threadIdx.x * 2u; b < v0; b += kCopyThreads * 2u)
            *reinterpret_cast<uint16_t*>(dst + b) = *reinterpret_cast<const uint16_t*>(src + b);
        for (uint64_t b = v0 + n16 * 16 + threadIdx.x * 2u; b < b1; b += kCopyThreads * 2u)
            *reinterpret_cast<uint16_t*>(dst + b) = *reinterpret_cast<const uint16_t*>(src + b);
    }
}

struct SidePlanes {
    bool q8;
    uint8_t* data;    // int8 plane or fp16 plane
    uint8_t* scales;  // fp16 scale plane (q8 only)
};

static SidePlanes k_side(const b200kv_view& v) {
    return is_k_q8(v.quant_mode) ? SidePlanes{true, reinterpret_cast<uint8_t*>(v.key_q8), static_cast<uint8_t*>(v.key_scales)}
                                 : SidePlanes{false, static_cast<uint8_t*>(v.key_f16), nullptr};
}
static SidePlanes v_side(const b200kv_view& v) {
    return is_v_q8(v.quant_mode) ? SidePlanes{true, reinterpret_cast<uint8_t*>(v.value_q8), static_cast<uint8_t*>(v.value_scales)}
                                 : SidePlanes{false, static_cast<uint8_t*>(v.value_f16), nullptr};
}

static size_t side_record_bytes(const b200kv_view& v, bool q8, uint64_t tokens) {
    const size_t d = v.head_dim, nblk = d / v.qblock;
    return q8 ? tokens * (d + 2 * nblk) : tokens * d * 2;
}

// The planes of a view in blob order (K data, K scales, V data, V scales) with their row sizes.
struct PlaneList {
    uint8_t* base[4];
    uint32_t row_bytes[4];
    uint32_t count;
};
static PlaneList planes_of(const b200kv_view& v) {
    PlaneList out{};
    const uint32_t d = v.head_dim, scale_bytes = d / v.qblock * 2u;
    auto side = [&](const SidePlanes& s) {
        out.base[out.count] = s.data;
        out.row_bytes[out.count++] = s.q8 ? d : d * 2u;
        if (s.q8) { out.base[out.count] = s.scales; out.row_bytes[out.count++] = scale_bytes; }
    };
    side(k_side(v));
    side(v_side(v));
    return out;
}

static int launch_copy(CopyParams& p, cudaStream_t stream) {
    uint64_t per_head = 0;
    for (uint32_t i = 0; i < p.planes; ++i) {
        // 16 bytes more than the span: the first inner boundary may lie up to 15 bytes behind a multiple of the chunk
        p.chunks[i] = static_cast<uint32_t>((p.tokens * p.row_bytes[i] + 15 + kCopyChunk - 1) / kCopyChunk);
        per_head += p.chunks[i];
    }
    const uint64_t total = per_head * p.heads * p.layers;
    if (per_head > 0xffffffffull || total > 0xffffffffull) return B200KV_ERR_UNSUPPORTED;
    p.span_chunks = static_cast<uint32_t>(per_head);
    p.total_chunks = static_cast<uint32_t>(total);
    const unsigned grid = static_cast<unsigned>(total < 148u * 8u ? total : 148u * 8u);   // eight CTAs of 256 threads fill an SM
    copy_spans_kernel<<<grid, kCopyThreads, 0, stream>>>(p);
    B200KV_CUDA_TRY(cudaGetLastError());
    return B200KV_OK;
}

static bool same_shape(const b200kv_view& a, const b200kv_view& b) {
    return a.kv_heads == b.kv_heads && a.head_dim == b.head_dim && a.qblock == b.qblock && a.quant_mode == b.quant_mode;
}

// One launch per run of up to kCopyLayers layers of one geometry (capacities may differ); everything in this device's memory.
static int copy_layers_here(const b200kv_view* views, uint32_t layers, uint64_t tokens, uint8_t* blob, const uint64_t* layer_bytes, bool to_blob,
                            cudaStream_t stream) {
    for (uint32_t l0 = 0; l0 < layers;) {
        CopyParams p{};
        while (l0 + p.layers < layers && p.layers < static_cast<uint32_t>(kCopyLayers) && same_shape(views[l0 + p.layers], views[l0])) ++p.layers;
        p.heads = views[l0].kv_heads;
        p.tokens = tokens;
        const PlaneList shape = planes_of(views[l0]);
        p.planes = shape.count;
        // where a plane's first head starts in a snapshot, and the distance between its heads (one side's record)
        uint64_t start[4], side_start = 0;
        const uint32_t k_planes = is_k_q8(views[l0].quant_mode) ? 2u : 1u;
        for (uint32_t side = 0, i = 0; side < 2; ++side) {
            const uint32_t end = side == 0 ? k_planes : shape.count;
            uint64_t record = 0;
            for (uint32_t j = i; j < end; ++j) record += tokens * shape.row_bytes[j];
            uint64_t at = side_start;
            for (; i < end; ++i) {
                start[i] = at;
                at += tokens * shape.row_bytes[i];
                p.row_bytes[i] = shape.row_bytes[i];
                (to_blob ? p.dst_record : p.src_record)[i] = record;
            }
            side_start += record * p.heads;
        }
        for (uint32_t l = 0; l < p.layers; ++l) {
            const PlaneList cache = planes_of(views[l0 + l]);
            CopyLayer& y = p.layer[l];
            y.src_rows = y.dst_rows = views[l0 + l].capacity;
            for (uint32_t i = 0; i < p.planes; ++i) {
                uint8_t* in_blob = blob + start[i];
                y.src[i] = to_blob ? cache.base[i] : in_blob;
                y.dst[i] = to_blob ? in_blob : cache.base[i];
            }
            blob += layer_bytes[l0 + l];
        }
        const int rc = launch_copy(p, stream);
        if (rc != B200KV_OK) return rc;
        l0 += p.layers;
    }
    return B200KV_OK;
}

static int copy_cache_to_cache(const b200kv_view& dst, const b200kv_view& src, uint64_t tokens, cudaStream_t stream) {
    CopyParams p{};
    p.layers = 1;
    p.heads = src.kv_heads;
    p.tokens = tokens;
    const PlaneList from = planes_of(src), to = planes_of(dst);
    p.planes = from.count;
    p.layer[0].src_rows = src.capacity;
    p.layer[0].dst_rows = dst.capacity;
    for (uint32_t i = 0; i < p.planes; ++i) {
        p.row_bytes[i] = from.row_bytes[i];
        p.layer[0].src[i] = from.base[i];
        p.layer[0].dst[i] = to.base[i];
    }
    return launch_copy(p, stream);
}

// Whether the copy kernel may touch all of it: ordinary memory of the current device (anything else takes the copy engine, which
// also reaches host memory and other devices).  The driver is asked once per mapping, which is one physical allocation and so
// lies on one device: a caching allocator's planes share a few (16 layers x 4 planes of a short prefix: asking for every plane took
// 12 us a capture and restore, more than the copies).
namespace {
using PointerQuery = CUresult (*)(unsigned int, CUpointer_attribute*, void**, CUdeviceptr);
PointerQuery pointer_query() {
    static PointerQuery fn = [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &sym, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
            return reinterpret_cast<PointerQuery>(sym);
        (void)cudaGetLastError();
        return static_cast<PointerQuery>(nullptr);
    }();
    return fn;
}

class DeviceMemory {
public:
    explicit DeviceMemory(int device) : device_(device), query_(pointer_query()) {}
    bool holds(const void* p) {
        const uint64_t at = reinterpret_cast<uintptr_t>(p);
        for (uint32_t i = 0; i < kept_; ++i)
            if (at - base_[i] < size_[i]) return true;
        if (query_ == nullptr) return false;
        uint32_t type = 0, managed = 0;
        int device = -1;
        uint64_t base = 0, size = 0;
        CUpointer_attribute names[5] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED, CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL,
                                        CU_POINTER_ATTRIBUTE_MAPPING_BASE_ADDR, CU_POINTER_ATTRIBUTE_MAPPING_SIZE};
        void* values[5] = {&type, &managed, &device, &base, &size};
        if (query_(5, names, values, at) != CUDA_SUCCESS || type != CU_MEMORYTYPE_DEVICE || managed != 0 || device != device_) return false;
        if (at - base < size) {
            const uint32_t slot = kept_ < kRanges ? kept_++ : next_++ % kRanges;
            base_[slot] = base;
            size_[slot] = size;
        }
        return true;
    }

private:
    static constexpr uint32_t kRanges = 16;
    uint64_t base_[kRanges], size_[kRanges];
    uint32_t kept_ = 0, next_ = 0;
    int device_;
    PointerQuery query_;
};
}  // namespace

static bool all_on_this_device(const b200kv_view* views, uint32_t layers, const void* blob) {
    int device = -1;
    if (cudaGetDevice(&device) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    DeviceMemory here(device);
    if ((reinterpret_cast<uintptr_t>(blob) & 1u) != 0 || !here.holds(blob)) return false;
    for (uint32_t l = 0; l < layers; ++l) {
        const PlaneList planes = planes_of(views[l]);
        for (uint32_t i = 0; i < planes.count; ++i)
            if (!here.holds(planes.base[i])) return false;
    }
    return true;
}

// One side (K or V) between the cache and the blob; to_blob selects direction.
static int copy_side(const b200kv_view& v, const SidePlanes& side, uint64_t tokens, uint8_t* blob, bool to_blob,
                     cudaStream_t s) {
    const size_t d = v.head_dim, nblk = d / v.qblock;
    const size_t record = side_record_bytes(v, side.q8, tokens);
    auto copy2d = [&](uint8_t* cache_plane, size_t bytes_per_pos, size_t blob_offset) -> cudaError_t {
        const size_t width = tokens * bytes_per_pos, cache_pitch = static_cast<size_t>(v.capacity) * bytes_per_pos;
        return to_blob ? cudaMemcpy2DAsync(blob + blob_offset, record, cache_plane, cache_pitch, width, v.kv_heads, cudaMemcpyDefault, s)
                       : cudaMemcpy2DAsync(cache_plane, cache_pitch, blob + blob_offset, record, width, v.kv_heads, cudaMemcpyDefault, s);
    };
    if (side.q8) {
        B200KV_CUDA_TRY(copy2d(side.data, d, 0));
        B200KV_CUDA_TRY(copy2d(side.scales, nblk * 2, tokens * d));
    } else {
        B200KV_CUDA_TRY(copy2d(side.data, d * 2, 0));
    }
    return B200KV_OK;
}

int snapshot_copy_layers(const b200kv_view* views, uint32_t layers, uint64_t tokens, uint8_t* blob, const uint64_t* layer_bytes, bool to_blob,
                         cudaStream_t stream) {
    if (tokens == 0) return B200KV_OK;
    if (all_on_this_device(views, layers, blob)) return copy_layers_here(views, layers, tokens, blob, layer_bytes, to_blob, stream);
    for (uint32_t l = 0; l < layers; blob += layer_bytes[l++]) {
        const SidePlanes ks = k_side(views[l]), vs = v_side(views[l]);
        int rc = copy_side(views[l], ks, tokens, blob, to_blob, stream);
        if (rc != B200KV_OK) return rc;
        rc = copy_side(views[l], vs, tokens, blob + side_record_bytes(views[l], ks.q8, tokens) * views[l].kv_heads, to_blob, stream);
        if (rc != B200KV_OK) return rc;
    }
    return B200KV_OK;
}

static int snapshot_copy(const b200kv_view* view, uint64_t tokens, void* blob, bool to_blob, void* stream) {
    int rc = validate_view(view);
    if (rc != B200KV_OK) return rc;
    if (tokens > view->capacity) return B200KV_ERR_RANGE;  // the reference throws here (kv_cache.cpp:228-230)
    if (tokens == 0 || blob == nullptr) return B200KV_OK;  // the reference returns silently (kv_cache.cpp:231)
    if ((rc = ensure_device()) != B200KV_OK) return rc;
    const uint64_t bytes = 0;   // of no use with one layer
    return snapshot_copy_layers(view, 1, tokens, static_cast<uint8_t*>(blob), &bytes, to_blob, static_cast<cudaStream_t>(stream));
}

}  // namespace b200kv

using namespace b200kv;

extern "C" {

size_t b200kv_snapshot_bytes(const b200kv_view* view, uint64_t tokens) {
    if (view == nullptr || view->qblock == 0) return 0;
    return (side_record_bytes(*view, is_k_q8(view->quant_mode), tokens) +
            side_record_bytes(*view, is_v_q8(view->quant_mode), tokens)) * view->kv_heads;
}

int b200kv_snapshot_save(const b200kv_view* view, uint64_t tokens, void* dst, void* stream) {
    return snapshot_copy(view, tokens, dst, true, stream);
}

int b200kv_snapshot_restore(const b200kv_view* view, uint64_t tokens, const void* src, void* stream) {
    return snapshot_copy(view, tokens, const_cast<void*>(src), false, stream);
}

int b200kv_snapshot_clone(const b200kv_view* dst, const b200kv_view* src, uint64_t tokens, void* stream) {
    int rc;
    if ((rc = validate_view(dst)) != B200KV_OK || (rc = validate_view(src)) != B200KV_OK) return rc;
    if (dst->head_dim != src->head_dim || dst->kv_heads != src->kv_heads || dst->qblock != src->qblock ||
        dst->quant_mode != src->quant_mode)
        return B200KV_ERR_INVALID;
    if (tokens > dst->capacity || tokens > src->capacity) return B200KV_ERR_RANGE;
    if (tokens == 0) return B200KV_OK;
    if ((rc = ensure_device()) != B200KV_OK) return rc;
    return copy_cache_to_cache(*dst, *src, tokens, static_cast<cudaStream_t>(stream));
}

}  // extern "C"

// ---- dequantising download (inspection and tests) ----------------------------------------------------------------
// AttentionLayerKvCacheStorage::download_key / download_value, src/prefill_v2/kv_cache.cpp:132-212: the first `tokens`
// positions of one side as fp32 [kv_head][tokens][head_dim] in HOST memory, int8 values multiplied by their fp16
// scale (here: the scale of their block), fp16 values widened.  Like the reference's it is a blocking host routine
// (it stages the raw planes in host memory and converts there); it is not part of the per-token path.
#include <vector>

namespace {
int download_side(const b200kv_view* view, uint64_t tokens, float* host_dst, bool key, cudaStream_t stream) {
    using namespace b200kv;
    int rc = validate_view(view);
    if (rc != B200KV_OK) return rc;
    if (host_dst == nullptr && tokens > 0) return B200KV_ERR_INVALID;
    if (tokens > view->capacity) return B200KV_ERR_RANGE;   // the reference throws (kv_cache.cpp:133-135)
    if (tokens == 0) return B200KV_OK;
    if ((rc = ensure_device()) != B200KV_OK) return rc;
    const uint32_t H = view->kv_heads, d = view->head_dim, nblk = d / view->qblock;
    const bool q8 = key ? is_k_q8(view->quant_mode) : is_v_q8(view->quant_mode);
    try {
        if (q8) {
            std::vector<int8_t> q(static_cast<size_t>(H) * tokens * d);
            std::vector<uint16_t> sc(static_cast<size_t>(H) * tokens * nblk);
            const int8_t* src_q = key ? view->key_q8 : view->value_q8;
            const uint8_t* src_s = static_cast<const uint8_t*>(key ? view->key_scales : view->value_scales);
            B200KV_CUDA_TRY(cudaMemcpy2DAsync(q.data(), tokens * d, src_q, view->capacity * d, tokens * d, H, cudaMemcpyDeviceToHost, stream));
            B200KV_CUDA_TRY(cudaMemcpy2DAsync(sc.data(), tokens * nblk * 2, src_s, view->capacity * nblk * 2, tokens * nblk * 2, H,
                                              cudaMemcpyDeviceToHost, stream));
            B200KV_CUDA_TRY(cudaStreamSynchronize(stream));
            for (size_t row = 0; row < static_cast<size_t>(H) * tokens; ++row)
                for (uint32_t b = 0; b < nblk; ++b) {
                    const float scale = __half2float(__ushort_as_half(sc[row * nblk + b]));
                    for (uint32_t i = 0; i < view->qblock; ++i) {
                        const size_t idx = row * d + b * view->qblock + i;
                        host_dst[idx] = static_cast<float>(q[idx]) * scale;
                    }
                }
        } else {
            std::vector<uint16_t> h(static_cast<size_t>(H) * tokens * d);
            const void* src = key ? view->key_f16 : view->value_f16;
            B200KV_CUDA_TRY(cudaMemcpy2DAsync(h.data(), tokens * d * 2, src, view->capacity * d * 2, tokens * d * 2, H, cudaMemcpyDeviceToHost, stream));
            B200KV_CUDA_TRY(cudaStreamSynchronize(stream));
            for (size_t i = 0; i < h.size(); ++i) host_dst[i] = __half2float(__ushort_as_half(h[i]));
        }
    } catch (const std::exception&) {
        return B200KV_ERR_CUDA;
    }
    return B200KV_OK;
}
}  // namespace

extern "C" int b200kv_download_key(const b200kv_view* view, uint64_t tokens, float* host_dst, void* stream) {
    return download_side(view, tokens, host_dst, true, static_cast<cudaStream_t>(stream));
}
extern "C" int b200kv_download_value(const b200kv_view* view, uint64_t tokens, float* host_dst, void* stream) {
    return download_side(view, tokens, host_dst, false, static_cast<cudaStream_t>(stream));
}
