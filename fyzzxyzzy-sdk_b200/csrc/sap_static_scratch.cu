// Sweep-and-prune overlap pairs of one scene's finite shapes, computed
// without allocating memory.
//
// The world's broadphase (broadphase.cu) keeps its sort keys, sweep records
// and per-owner pair buckets in buffers the world allocates when a scene is
// uploaded or when the pair budget grows.  Some callers cannot allocate at
// the point where they need a pair set: a frame loop that shares the GPU with
// other work and must not take the device-wide synchronisation that
// cudaMalloc / cudaFree imply, or a process that runs under a fixed device
// memory budget reserved up front.  This entry point serves them: the pair
// set and canonical order of the world's broadphase, with its working set in
// a fixed file-scope device array instead of allocated buffers.
//
// Pair semantics follow the reference's full sweep (src/native/scene.cpp,
// Scene::update_pairs 2635-2704): two finite shapes pair when their encoded
// bounds overlap on all three axes, they belong to different bodies and at
// least one body is dynamic.  Output is (a, b) with a < b, ascending.
//
// Limits and sharing:
//  * at most kStaticSapMaxShapes shapes per call (larger inputs are rejected
//    before anything is launched);
//  * every call on a device uses the same scratch array, so calls whose
//    kernels may overlap in time (different streams, different host threads
//    without ordering) race and corrupt each other's results; order them on
//    one stream;
//  * the first call on a device resolves the scratch array's address with
//    cudaGetSymbolAddress (which loads this module on that device) and
//    raises the kernels' dynamic shared-memory limits; make that first call
//    before any stream capture on the device.  The resolved address is kept
//    per CUDA context, so a context made after cudaDeviceReset resolves it
//    again on its first call;
//  * when the pair total exceeds the caller's capacity, only whole owner
//    buckets that end within the capacity are written: the list is then a
//    prefix of the full canonical list (deterministic), and the total tells
//    the caller how much room a complete list needs.
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include <initializer_list>
#include <mutex>
#include "fyzz_b200.h"

namespace fyzz::b200 {
namespace {

constexpr uint32_t kStaticSapMaxShapes = FYZZ_B200_STATIC_SAP_MAX_SHAPES;
static_assert(kStaticSapMaxShapes == 8192u, "the rejection message states the limit");
// Scratch layout, 32 bytes a shape (256 KiB at the maximum):
//   cnt      u32            pairs owned by each shape (the lower shape id)
//   partner  u16 x kKept    its first partners, ascending
constexpr uint32_t kKept = 14;
constexpr size_t kPartnerOff = size_t(kStaticSapMaxShapes) * 4;
constexpr size_t kScratchBytes = kPartnerOff + size_t(kStaticSapMaxShapes) * kKept * 2;
static_assert(kScratchBytes == 256u * 1024u && kStaticSapMaxShapes <= 65536u, "documented size; partners fit 16 bits");

static __device__ __align__(256) unsigned char g_sap_scratch[kScratchBytes];

// The whole device tests every shape against all shapes of larger id:
// lanes hold 32 consecutive candidates, so an owner's pairs come out in
// partner order by ballots and nothing is sorted.  At 8,192 shapes that is
// 1.05 million 32-wide tests in x and z, four comparisons and a vote each; a
// candidate's y and body are read only where some lane passes them.  Every
// block holds all shapes in shared memory (28 bytes each, 224 KiB at the
// maximum): with only x there, two thirds of the x tests went on to a round
// trip to L2 (317 us).  The sort + sweep in one CTA that this replaces waited
// for one SM's barriers and scattered L2 reads: 1,453 us on 8,192 shapes
// with 23,200 pairs; this takes 78.
struct Owner {
    uint32_t id, mnx, mxx, mny, mxy, mnz, mxz, body;
};
__device__ __forceinline__ Owner load_owner(const uint32_t* __restrict__ bounds, const uint32_t* __restrict__ body,
                                            uint32_t i) {
    const uint32_t* b = bounds + 6 * size_t(i);
    return {i, b[0], b[3], b[1], b[4], b[2], b[5], body[i]};
}
// x and z.  In x the shape that starts first (lower id on ties) must reach
// the other's start, as in a sweep over the sorted minima; while no bounds
// are inverted (kInverted false) that is the plain interval test.
template <bool kInverted> __device__ __forceinline__ bool overlap_xz(const Owner& a, const uint4& c) {
    const bool x = kInverted ? (c.x >= a.mnx ? c.x <= a.mxx : a.mnx <= c.y) : c.x <= a.mxx && a.mnx <= c.y;
    return x && c.z <= a.mxz && a.mnz <= c.w;
}
// The rest of the test: y, different bodies, one of them dynamic.
__device__ __forceinline__ bool overlap_rest(const Owner& a, uint2 y, uint32_t body) {
    return (body & 0x7fffffffu) != (a.body & 0x7fffffffu) && ((body | a.body) >> 31) && y.x <= a.mxy && a.mny <= y.y;
}

// Every shape in shared memory: {min x, max x, min z, max z}, {min y, max y}
// and body, padded to whole chunks of 32.
constexpr size_t kShapeSmem = sizeof(uint4) + sizeof(uint2) + sizeof(uint32_t);
constexpr size_t kMaxShapeSmem = size_t(kStaticSapMaxShapes) * kShapeSmem;
static_assert(kMaxShapeSmem <= 224u * 1024u, "every shape fits one block's shared memory");
struct Shapes {
    uint4* xz;
    uint2* y;
    uint32_t* body;
    __device__ Shapes(uint4* smem, uint32_t padded) : xz(smem) {
        y = reinterpret_cast<uint2*>(xz + padded);
        body = reinterpret_cast<uint32_t*>(y + padded);
    }
    // Loads all shapes; returns whether some bounds are inverted in x.
    __device__ __forceinline__ bool load(const uint32_t* __restrict__ bounds, const uint32_t* __restrict__ bodies,
                                         uint32_t n, uint32_t padded) const {
        bool inverted = false;
        // four shapes' loads in flight a thread: one at a time, their round
        // trips took 50 us of either kernel
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < padded; i += blockDim.x) {
            const bool in = i < n;
            const uint32_t* b = bounds + 6 * size_t(in ? i : 0u);
            const uint32_t v0 = b[0], v1 = b[1], v2 = b[2], v3 = b[3], v4 = b[4], v5 = b[5], v6 = bodies[in ? i : 0u];
            xz[i] = in ? make_uint4(v0, v3, v2, v5) : make_uint4(~0u, 0u, ~0u, 0u);
            y[i] = make_uint2(v1, v4);
            body[i] = v6;
            inverted |= in && v0 > v3;
        }
        return __syncthreads_or(inverted);
    }
};

// N owners' pairs among the chunks [base, end): counts them and keeps each
// owner's first kKept partners.
template <bool kInverted, int N>
__device__ __forceinline__ void scan_chunks(const Shapes& S, const Owner (&o)[4], uint32_t (&found)[4], uint32_t base,
                                            uint32_t end, uint32_t n, uint16_t* kept) {
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    for (; base < end; base += 32) {
        const uint32_t j = base + lane;
        const uint4 c = S.xz[j];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            bool hit = overlap_xz<kInverted>(o[k], c);
            if (!__any_sync(0xffffffffu, hit)) continue;
            hit = hit && j > o[k].id && j < n && overlap_rest(o[k], S.y[j], S.body[j]);
            const uint32_t bits = __ballot_sync(0xffffffffu, hit);
            const uint32_t at = found[k] + __popc(bits & lt);
            if (hit && at < kKept) kept[o[k].id * kKept + at] = uint16_t(j);
            found[k] += __popc(bits);
        }
    }
}

// Four owners a warp, two from either end of the shapes, so that every warp
// tests the same number of candidates; the two at the back join when their
// candidates begin.
constexpr int kCountThreads = 512;
__global__ void __launch_bounds__(kCountThreads) k_sap_count(const uint32_t* __restrict__ bounds,
                                                             const uint32_t* __restrict__ body, uint32_t n,
                                                             unsigned char* scratch) {
    extern __shared__ uint4 smem[];
    const uint32_t padded = (n + 31u) & ~31u;
    const Shapes S(smem, padded);
    const bool inverted = S.load(bounds, body, n, padded);
    uint32_t* cnt = reinterpret_cast<uint32_t*>(scratch);
    uint16_t* kept = reinterpret_cast<uint16_t*>(scratch + kPartnerOff);
    const uint32_t lane = threadIdx.x & 31u, w = (blockIdx.x * kCountThreads + threadIdx.x) >> 5;
    const uint32_t half = (n + 1) / 2;   // owners below half from the front, the others from the back
    if (2 * w >= half) return;
    Owner o[4];
    uint32_t found[4] = {0, 0, 0, 0};
    bool on[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t at = 2 * w + (k & 1u);
        on[k] = k < 2 ? at < half : at < n - half;
        o[k] = load_owner(bounds, body, !on[k] ? 0u : k < 2 ? at : n - 1u - at);
        if (!on[k]) o[k].id = n;         // no candidate lies after it
    }
    const uint32_t front = (2 * w + 1) & ~31u, back = (n - 2 * w - 1u) & ~31u;   // from owner n - 2 - 2w on
    if (inverted) {
        scan_chunks<true, 2>(S, o, found, front, back, n, kept);
        scan_chunks<true, 4>(S, o, found, max(front, back), n, n, kept);
    } else {
        scan_chunks<false, 2>(S, o, found, front, back, n, kept);
        scan_chunks<false, 4>(S, o, found, max(front, back), n, n, kept);
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
        if (on[k] && lane == 0) cnt[o[k].id] = found[k];
}

// Sum of v over the block (valid on every thread); `warp_sum` has a slot a
// warp.
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* warp_sum) {
    v = __reduce_add_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31u) == 0) warp_sum[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t sum = 0;
    for (uint32_t w = 0; w < blockDim.x / 32u; ++w) sum += warp_sum[w];
    return sum;
}

// A block sums the counts before its kFillOwners owners and all of them for
// itself (cheaper than a launch of its own), then its warps write their
// owners' buckets: the kept partners, or, for an owner with more, the
// candidates tested again, from shared memory like the counting (only
// blocks with such an owner load the shapes; from global memory those owners
// alone took 96 us).  A bucket is written only when all of it fits, so a
// truncated list is a canonical prefix.
constexpr int kFillThreads = 512;
constexpr uint32_t kFillOwners = 64;   // owners a block
__global__ void __launch_bounds__(kFillThreads) k_sap_fill(const uint32_t* __restrict__ bounds,
                                                           const uint32_t* __restrict__ body, uint32_t n,
                                                           uint32_t* __restrict__ pairs, uint32_t cap,
                                                           uint32_t* __restrict__ count, const unsigned char* scratch) {
    extern __shared__ uint4 smem[];
    __shared__ uint32_t warp_sum[kFillThreads / 32], off[kFillOwners + 1];
    const uint32_t* cnt = reinterpret_cast<const uint32_t*>(scratch);
    const uint16_t* kept = reinterpret_cast<const uint16_t*>(scratch + kPartnerOff);
    const uint32_t first = blockIdx.x * kFillOwners;
    uint32_t before = 0, all = 0;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < n; i += kFillThreads) {
        const uint32_t c = cnt[i];
        all += c;
        before += i < first ? c : 0u;
    }
    before = block_sum(before, warp_sum);
    if (blockIdx.x == 0) {
        all = block_sum(all, warp_sum);
        if (threadIdx.x == 0) *count = all;
    }
    const uint32_t own = threadIdx.x < kFillOwners && first + threadIdx.x < n ? cnt[first + threadIdx.x] : 0u;
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    uint32_t incl = own;
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= uint32_t(d)) incl += x;
    }
    __syncthreads();
    if (lane == 31) warp_sum[threadIdx.x >> 5] = incl;
    __syncthreads();
    if (threadIdx.x < kFillOwners) off[threadIdx.x] = before + incl - own + (threadIdx.x >= 32 ? warp_sum[0] : 0u);
    if (threadIdx.x == 0) off[kFillOwners] = before + warp_sum[0] + warp_sum[1];
    const uint32_t padded = (n + 31u) & ~31u;
    const Shapes S(smem, padded);
    bool inverted = false;
    if (__syncthreads_or(own > kKept)) inverted = S.load(bounds, body, n, padded);
    for (uint32_t q = threadIdx.x >> 5; q < kFillOwners && first + q < n; q += kFillThreads / 32) {
        const uint32_t i = first + q, begin = off[q], end = off[q + 1];
        if (begin == end || end > cap) continue;
        uint32_t* p = pairs + 2 * size_t(begin);
        if (end - begin <= kKept) {
            if (lane < end - begin) {
                p[2 * lane] = i;
                p[2 * lane + 1] = kept[i * kKept + lane];
            }
            continue;
        }
        const Owner o = load_owner(bounds, body, i);
        uint32_t found = 0;
        for (uint32_t base = (i + 1) & ~31u; base < n && found < end - begin; base += 32) {
            const uint32_t j = base + lane;
            const uint4 c = S.xz[j];
            bool hit = inverted ? overlap_xz<true>(o, c) : overlap_xz<false>(o, c);
            if (!__any_sync(0xffffffffu, hit)) continue;
            hit = hit && j > i && j < n && overlap_rest(o, S.y[j], S.body[j]);
            const uint32_t bits = __ballot_sync(0xffffffffu, hit);
            const size_t at = found + __popc(bits & lt);
            if (hit) {
                p[2 * at] = i;
                p[2 * at + 1] = j;
            }
            found += __popc(bits);
        }
    }
}
static_assert(kFillOwners == 64, "two warps scan a block's owners");

constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
unsigned char* g_scratch[kMaxDevices] = {};
void* g_scratch_ctx[kMaxDevices] = {};       // the CUDA context g_scratch[dev] was resolved in
using CtxGetCurrent = int (*)(void**);       // the driver's cuCtxGetCurrent
CtxGetCurrent g_ctx_get = nullptr;

// Copies a message into the caller's buffer (no formatting, no allocation).
void put_message(char* out, size_t len, const char* a, const char* b = "") {
    if (!out || len == 0) return;
    size_t k = 0;
    for (const char* s : {a, b})
        for (; *s && k + 1 < len; ++s) out[k++] = *s;
    out[k] = '\0';
}

// Once per device (per CUDA context of the device: a context made after
// cudaDeviceReset loads this module again), with that device current:
// resolve the scratch array's address and allow the kernels the shared
// memory their largest input needs.
int setup_device(int dev, unsigned char** out, char* msg, size_t msg_len) {
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    if (!g_ctx_get) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q{};
        const cudaError_t e = cudaGetDriverEntryPoint("cuCtxGetCurrent", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) {
            put_message(msg, msg_len, "cuCtxGetCurrent unavailable: ", cudaGetErrorString(e));
            return FYZZ_B200_RUNTIME_ERROR;
        }
        g_ctx_get = reinterpret_cast<CtxGetCurrent>(fn);
    }
    void* ctx = nullptr;
    if (g_ctx_get(&ctx) != 0 || !ctx) {
        put_message(msg, msg_len, "no current CUDA context");
        return FYZZ_B200_RUNTIME_ERROR;
    }
    if (!g_scratch[dev] || g_scratch_ctx[dev] != ctx) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_sap_scratch);
        if (e != cudaSuccess || !p) {
            put_message(msg, msg_len, "cudaGetSymbolAddress failed: ", cudaGetErrorString(e));
            return FYZZ_B200_RUNTIME_ERROR;
        }
        e = cudaFuncSetAttribute(k_sap_count, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kMaxShapeSmem));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_sap_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kMaxShapeSmem));
        if (e != cudaSuccess) {
            put_message(msg, msg_len, "cudaFuncSetAttribute failed: ", cudaGetErrorString(e));
            return FYZZ_B200_RUNTIME_ERROR;
        }
        g_scratch[dev] = static_cast<unsigned char*>(p);
        g_scratch_ctx[dev] = ctx;
    }
    *out = g_scratch[dev];
    return FYZZ_B200_OK;
}

}  // namespace
}  // namespace fyzz::b200

extern "C" int fyzz_b200_sap_pairs_static_scratch(const uint32_t* bounds_dev, const uint32_t* body_dev,
                                                  uint32_t n_shapes, uint32_t* pairs_dev,
                                                  uint32_t pair_cap, uint32_t* count_dev, void* stream,
                                                  char* message, size_t message_len) {
    using namespace fyzz::b200;
    put_message(message, message_len, "");
    if (n_shapes > kStaticSapMaxShapes) {
        put_message(message, message_len,
                    "n_shapes exceeds FYZZ_B200_STATIC_SAP_MAX_SHAPES (the fixed scratch array "
                    "holds 8192 shapes); split the scene or use the world's broadphase");
        return FYZZ_B200_INVALID_ARGUMENT;
    }
    if (!count_dev || (n_shapes && (!bounds_dev || !body_dev)) || (pair_cap && !pairs_dev)) {
        put_message(message, message_len, "null device pointer");
        return FYZZ_B200_INVALID_ARGUMENT;
    }
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        put_message(message, message_len, "no usable current CUDA device: ", cudaGetErrorString(e));
        return FYZZ_B200_RUNTIME_ERROR;
    }
    unsigned char* scratch = nullptr;
    if (const int rc = setup_device(dev, &scratch, message, message_len)) return rc;
    const auto st = static_cast<cudaStream_t>(stream);
    const uint32_t warps = ((n_shapes + 1) / 2 + 1) / 2;
    const size_t smem = size_t((n_shapes + 31u) & ~31u) * kShapeSmem;
    if (n_shapes > 1)
        k_sap_count<<<(warps * 32 + kCountThreads - 1) / kCountThreads, kCountThreads, smem, st>>>(
            bounds_dev, body_dev, n_shapes, scratch);
    // a single shape has no pairs: its bucket is not counted
    const uint32_t owners = n_shapes > 1 ? n_shapes : 0u;
    k_sap_fill<<<owners ? (owners + kFillOwners - 1) / kFillOwners : 1u, kFillThreads, smem, st>>>(
        bounds_dev, body_dev, owners, pairs_dev, pair_cap, count_dev, scratch);
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        put_message(message, message_len, "launch failed: ", cudaGetErrorString(e));
        return FYZZ_B200_RUNTIME_ERROR;
    }
    return FYZZ_B200_OK;
}
