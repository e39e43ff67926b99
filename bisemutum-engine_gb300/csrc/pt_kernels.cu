// pt_kernels.cu — the sm_103a kernels of the wavefront path-tracing pass.
//
// One render is a sequence of chunks; each chunk runs
//   k_camera -> k_trace(extend 0) -> k_shade(0) -> k_trace(extend 1, shadow 0) -> k_shade(1) -> ...
//            -> k_trace(shadow of the last segment)
// over device-resident queues whose sizes live in device counters, so no
// stage waits for the host and a whole render can be captured as one CUDA
// graph.  Stage <-> reference shader:
//   k_camera   generate_camera_ray_cs   (direction_sample/generate_camera_ray.hlsl:4-16)
//   k_trace    extension rays: rt_gbuffer_rgen/rchit/rmiss (rt_gbuffer.hlsl:7-36, hits/rt_gbuffer_hit.hlsl:6-18);
//              shadow rays: the visibility term of the direct light (there: shadow maps,
//              lights.hlsl:27-104; here: any-hit rays)
//   k_shade    deferred_lighting_secondary_cs + sample_secondary_ray_cs
//              (deferred_lighting_secondary.hlsl:11-111, sample_secondary_ray.hlsl:11-69)
//   k_resolve  additive blit + pt_accumulate_cs (path_tracing.cpp:436-478, pt_accumulate.hlsl:3-11)
// Compiled with --fmad=false: every float operation outside the explicit
// __fmaf_rn of the box test rounds once, as on the CPU oracle.
#include <cuda_runtime.h>

#include "bsm_pt.h"
#include "pt_device.h"
#include "pt_sky.cuh"
#include "pt_trace.cuh"
#include "pt_scene.cuh"
#include "pt_lights.cuh"
#include "pt_gbuffer.cuh"
#include "bvh_quant_lanes.cuh"
#include "mlp.cuh"

namespace bsm {

// Warp-aggregated queue allocation: one atomic per warp, slots in lane order.
// Must be reached by all 32 lanes (pred may be false).
__device__ __forceinline__ uint32_t warp_alloc(bool pred, uint32_t* counter) {
    uint32_t b = __ballot_sync(0xffffffffu, pred);
    uint32_t base = 0;
    int lane = threadIdx.x & 31;
    if (b != 0u && lane == __ffs(b) - 1) base = atomicAdd(counter, (uint32_t)__popc(b));
    base = __shfl_sync(0xffffffffu, base, b != 0u ? __ffs(b) - 1 : 0);
    return base + (uint32_t)__popc(b & lanemask_lt());
}

// Queue slots for the threads of a block with `pred`, grouped by the direction
// of `dir`: its octant and its dominant axis, 24 bins (one atomic on `counter`
// per block).  Consecutive slots then hold rays heading the same way from
// neighbouring paths, which keeps the warps of the next traversal and shading
// launches coherent.  The lanes of a warp that share a bin take their ranks
// from one shared-memory atomic; warp 0 scans the bins.  Every
// thread of the block must call it with the same `parity`, alternating 0 / 1
// from call to call, after s_dir_cnt[0] was cleared: each call clears the
// other parity's counters for the next one, so it needs two block barriers
// instead of three.  Returns 0 for threads without pred.
constexpr uint32_t kDirBins = 24;   // octant x dominant axis
static_assert(kDirBins <= 32, "one warp scans the bins");
__shared__ uint32_t s_dir_cnt[2][kDirBins + 1];
__device__ __forceinline__ uint32_t block_alloc_by_direction(bool pred, V3 dir, uint32_t* counter, int parity) {
    __shared__ uint32_t s_off[2][kDirBins], s_base[2];
    const float ax = fabsf(dir.x), ay = fabsf(dir.y), az = fabsf(dir.z);
    const uint32_t dom = (ax >= ay && ax >= az) ? 0u : (ay >= az ? 1u : 2u);
    uint32_t key = pred ? ((dir.x < 0.0f ? 1u : 0u) | (dir.y < 0.0f ? 2u : 0u) | (dir.z < 0.0f ? 4u : 0u)) * 3u + dom
                        : kDirBins;
    // one shared atomic per bin present in the warp (the lanes of a bin share it)
    const uint32_t peers = __match_any_sync(0xffffffffu, key);
    const uint32_t leader = (uint32_t)__ffs(peers) - 1u;
    uint32_t rank = 0;
    if ((threadIdx.x & 31u) == leader && pred) rank = atomicAdd(&s_dir_cnt[parity][key], (uint32_t)__popc(peers));
    rank = __shfl_sync(0xffffffffu, rank, (int)leader) + (uint32_t)__popc(peers & lanemask_lt());
    __syncthreads();
    if (threadIdx.x < 32) {   // exclusive prefix over the bins by warp 0, one bin per lane
        const uint32_t lane = threadIdx.x;
        const uint32_t c = lane < kDirBins ? s_dir_cnt[parity][lane] : 0u;
        uint32_t x = c;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane < kDirBins) s_off[parity][lane] = x - c;
        const uint32_t total = __shfl_sync(0xffffffffu, x, 31);
        if (lane == 0) s_base[parity] = total ? atomicAdd(counter, total) : 0u;
    }
    if (threadIdx.x <= kDirBins) s_dir_cnt[parity ^ 1][threadIdx.x] = 0u;
    __syncthreads();
    return pred ? s_base[parity] + s_off[parity][key] + rank : 0u;
}

// A path's contribution to its pixel: FP32 atomics, or the call's fixed-point sums when `fx` is set
// (BSM_PT_DETERMINISTIC).
__device__ __forceinline__ void accum_add(float4* accum, unsigned long long* fx, uint32_t idx, V3 c) {
    if (fx) accum_fixed_add(fx, idx, c.x, c.y, c.z);
    else atomicAdd(accum + idx, make_float4(c.x, c.y, c.z, 0.0f));
}

// ---------------------------------------------------------------- camera ----
// generate_camera_ray.hlsl:9-11 restated without the matrices: the inverse
// reverse-Z projection of (ndc, 1, 1) is (ndc.x * aspect * tan, ndc.y * tan, -1),
// rotated by the camera basis.  (jx, jy) is the position inside the pixel.
__device__ __forceinline__ V3 camera_dir(const DevView& v, uint32_t px, uint32_t py, float jx, float jy) {
    float uvx = ((float)px + jx) / (float)v.width;
    float uvy = ((float)py + jy) / (float)v.height;
    float ndx = uvx * 2.0f - 1.0f;
    float ndy = 1.0f - uvy * 2.0f;
    V3 dl = normalize(v3(ndx * v.aspect * v.tan_half, ndy * v.tan_half, -1.0f));
    V3 s = v3(v.s[0], v.s[1], v.s[2]), u = v3(v.u[0], v.u[1], v.u[2]), f = v3(v.f[0], v.f[1], v.f[2]);
    return normalize(s * dl.x + u * dl.y + (-f) * dl.z);
}

// Pixel of rank k in the order in which a view's pixels are traced: bands of four rows, each in tiles of eight by
// four pixels (narrower at the right and bottom edges), so that a warp's rays spread as little as they can.
__device__ __forceinline__ void tile_pixel(uint32_t k, uint32_t width, uint32_t height, uint32_t& x, uint32_t& y) {
    const uint32_t band = (uint32_t)((uint64_t)k / (4ull * width)), r = k - band * 4u * width;
    const uint32_t rows = min(4u, height - 4u * band);
    const uint32_t tile = r / (8u * rows), p = r - tile * 8u * rows;
    const uint32_t cols = min(8u, width - 8u * tile);
    const uint32_t dy = p / cols;
    x = 8u * tile + p - dy * cols;
    y = 4u * band + dy;
}
// Views of fewer samples per pixel than this are traced in tiles; with more a warp holds one pixel's samples or fewer, and
// rows need no divisions by the tile. Frames, ms, tiles / rows: 1 spp, 1080p terrain 3.738 / 3.772; 8 spp, 640x360 room
// 1.484 / 1.493; 16 spp, 1080p terrain 41.52 / 41.66; 24 to 48 spp within 0.3 % either way; 64 spp, 1080p room
// 70.14 / 69.86, terrain 160.5 / 160.3.
constexpr uint32_t kTileSpp = 32;

__global__ void k_camera(const DevView* __restrict__ views, uint32_t n_views, uint64_t path_begin,
                         uint32_t path_count, Wavefront wf, uint32_t max_segments_cap) {
    uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid == 0) wf.counters[kCntQueue + 0] = path_count;
    if (gid >= path_count) return;
    uint64_t p = path_begin + gid;
    // view lookup (views sorted by path_base)
    uint32_t lo = 0, hi = n_views - 1;
    while (lo < hi) {
        uint32_t mid = (lo + hi + 1) >> 1;
        if (views[mid].path_base <= p) lo = mid; else hi = mid - 1;
    }
    const DevView& v = views[lo];
    uint64_t local = p - v.path_base + v.first_path;
    // pixel-major order: the samples of a pixel are neighbours in the queue, so a warp traces the (near-)
    // identical camera rays of one or a few pixels together, and their later rays start from the same
    // points.  Every path's random stream depends only on its pixel and sample, so the order changes no
    // result (measured on the 1920x1080x64 terrain frame: 1274 -> 1515 Mrays/s against sample-major).
    const uint32_t rank = (uint32_t)(local / v.spp);
    const uint32_t sample = (uint32_t)(local - (uint64_t)rank * v.spp);
    uint32_t px, py;
    if (v.spp < kTileSpp) {
        tile_pixel(rank, v.width, v.height, px, py);
    } else {
        py = rank / v.width;
        px = rank - py * v.width;
    }
    const uint32_t pixel = py * v.width + px;
    Pcg g = pcg_seed(path_initstate(v.seed, v.sample_offset + sample, pixel), (uint64_t)pixel);
    float jx = 0.5f, jy = 0.5f;
    if (v.flags & BSM_PT_JITTER) { jx = pcg_uniform(g); jy = pcg_uniform(g); }
    V3 dw = camera_dir(v, px, py, jx, jy);
    uint32_t maxseg = v.max_segments < max_segments_cap ? v.max_segments : max_segments_cap;
    wf.ray_o[0][gid] = make_float4(v.pos[0], v.pos[1], v.pos[2], v.t_min);
    wf.ray_d[0][gid] = make_float4(dw.x, dw.y, dw.z, v.ray_length);
    wf.path[0][gid] = make_uint4(v.accum_base + pixel, (maxseg << 8) | (lo << 16), (uint32_t)g.state,
                                 (uint32_t)(g.state >> 32));
    wf.thr[0][gid] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
}

// ---------------------------------------------------------------- extend ----
// Counting variant of the closest-hit stage (BSM_PT_COUNT_TRAVERSAL).
struct CountRays {
    const float4 *ray_o, *ray_d;
    const uint4* path;
    float4* hits;
    __device__ __forceinline__ bool any(uint32_t) const { return false; }
    __device__ __forceinline__ void load(uint32_t i, float4& o, float4& d) const { o = ray_o[i]; d = ray_d[i]; }
    __device__ __forceinline__ void hit(uint32_t i, uint32_t leaf, float t, float u, float v, uint32_t) const {
        hits[i] = make_float4(t, __uint_as_float(leaf), u, v);
    }
    __device__ __forceinline__ void miss(uint32_t i, float tmax) const { hit(i, kMissPrim, tmax, 0.0f, 0.0f, kMissPrim); }
    __device__ __forceinline__ uint32_t seed(uint32_t i) const { return path[i].z; }   // the path's PCG32 word
};
template <bool kOpacity>
__global__ void __launch_bounds__(256) k_extend_count(DevScene sc, CountRays rays, uint32_t* counters,
                                                      unsigned long long* stats, uint32_t seg, int postpone_sp,
                                                      int refill_min) {
    const uint32_t n = counters[kCntQueue + seg];
    if (blockIdx.x == 0 && threadIdx.x == 0) stats[kStatExtend + seg] += n;
    TraceCounters c{0, 0};
    trace_queue<true, kOpacity>(sc.nodes, sc.tris, n, counters + kCntWork + 2 * seg, rays, &c, postpone_sp, refill_min);
    uint32_t cn = c.nodes, ct = c.tris;
    for (int off = 16; off > 0; off >>= 1) {
        cn += __shfl_xor_sync(0xffffffffu, cn, off);
        ct += __shfl_xor_sync(0xffffffffu, ct, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(stats + kStatNodes, (unsigned long long)cn);
        atomicAdd(stats + kStatTris, (unsigned long long)ct);
    }
}

// ------------------------------------------------------- extend + shadow ----
// The extension rays of segment `ext` (closest hit) and the shadow rays of
// segment `shd` (any hit) as one queue: index i < n_ext is extension ray i,
// then the sun rays from the front of the shadow queue, then the sky rays from
// its back.  A launch is bound by instruction issue while its queue lasts and
// by the latency of its last rays after that (60-100 us on the terrain: a
// grazing ray visits over 100 nodes, each a round trip to L2).  Both kinds are
// queued by the same shading launch and neither reads what the other writes,
// so tracing them together leaves one such tail per segment instead of two.
// Against a launch per kind: 128x128 preview of the room 534 -> 381 us,
// 1920x1080 1-spp frame of the 1.48 M-triangle terrain 5.01 -> 4.21 ms, its
// 64-spp frame 180.6 -> 179.1 ms.
struct TraceArgs {
    const float4 *ray_o, *ray_d;
    const uint4* path;
    float4* hit;
    const float4 *sh_o, *sh_d, *sh_c;
    const uint32_t* sh_seed;
    float4* accum;
    unsigned long long* accum_fx;
    uint32_t* counters;
    unsigned long long* stats;
    uint32_t ext, shd, sh_last;   // segments (kNoSegment: none); the shadow queue's last slot
    uint32_t ext_cnt, sun_cnt, sky_cnt;   // the queues' sizes in `counters` (kCntZero: left out)
    uint32_t min_rays, max_rays;  // the kernel leaves queues of other lengths alone
    int postpone_sp, refill_min;
};
struct TraceRays {
    const TraceArgs& a;
    uint32_t n_ext, n_front, n;   // extension rays; with the sun rays; all
    __device__ __forceinline__ uint32_t* work() const {
        return a.counters + kCntWork + (a.ext < kNoSegment ? 2u * a.ext : 2u * a.shd + 1u);
    }
    __device__ __forceinline__ uint32_t slot(uint32_t i) const { return i < n_front ? i - n_ext : a.sh_last - (i - n_front); }
    __device__ __forceinline__ bool any(uint32_t i) const { return i >= n_ext; }
    __device__ __forceinline__ void load(uint32_t i, float4& o, float4& d) const {
        if (i < n_ext) { o = __ldg(a.ray_o + i); d = __ldg(a.ray_d + i); }
        else { const uint32_t k = slot(i); o = __ldg(a.sh_o + k); d = __ldg(a.sh_d + k); }
    }
    // the hit record of a two-level scene carries the instance in place of u
    __device__ __forceinline__ void hit(uint32_t i, uint32_t leaf, float t, float u, float v, uint32_t inst) const {
        if (i < n_ext) a.hit[i] = make_float4(t, __uint_as_float(leaf), inst != kMissPrim ? __uint_as_float(inst) : u, v);
    }
    __device__ __forceinline__ void miss(uint32_t i, float tmax) const {
        if (i < n_ext) {
            a.hit[i] = make_float4(tmax, __uint_as_float(kMissPrim), 0.0f, 0.0f);
        } else {
            const float4 c = __ldg(a.sh_c + slot(i));
            accum_add(a.accum, a.accum_fx, __float_as_uint(c.w), v3(c.x, c.y, c.z));
        }
    }
    // opacity seed: the path's PCG32 word, or the shadow ray's own
    __device__ __forceinline__ uint32_t seed(uint32_t i) const {
        return i < n_ext ? __ldg(&a.path[i].z) : (a.sh_seed ? __ldg(a.sh_seed + slot(i)) : 0u);
    }
};
// The launch's queue sizes from the device counters; the first thread adds them to the statistics.
__device__ __forceinline__ TraceRays trace_rays(const TraceArgs& a) {
    const uint32_t n_ext = a.counters[a.ext_cnt], n_sun = a.counters[a.sun_cnt], n_sky = a.counters[a.sky_cnt];
    const uint32_t n = n_ext + n_sun + n_sky;
    if (n < a.min_rays || n > a.max_rays) return TraceRays{a, 0u, 0u, 0u};
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (n_ext) a.stats[kStatExtend + a.ext] += n_ext;
        if (n_sun + n_sky) a.stats[kStatShadow + a.shd] += n_sun + n_sky;
    }
    return TraceRays{a, n_ext, n_ext + n_sun, n};
}

template <int kMinBlocks, bool kOpacity>
__global__ void __launch_bounds__(256, kMinBlocks) k_trace(const CwNode* __restrict__ nodes,
                                                           const CwTri* __restrict__ tris,
                                                           const __grid_constant__ TraceArgs a) {
    const TraceRays rays = trace_rays(a);
    trace_queue<false, kOpacity>(nodes, tris, rays.n, rays.work(), rays, nullptr, a.postpone_sp, a.refill_min);
}

// The camera rays of chunks over the group kernel's limit: a ray per thread,
// in queue order and without the persistent loop.  The rays of a warp are an
// 8x4 tile of pixels or the samples of one pixel and walk the same nodes, so
// handing finished lanes rays of another tile gains nothing, and the loop's
// votes, queue reads and postponed leaves are instructions in a launch that is
// bound by their issue.  Against k_trace for these rays: 1920x1080 frame of
// the 1.48 M-triangle terrain with 64 spp 161.4 -> 158.5 ms, with one
// 3744 -> 3620 us, 256x256x16 room 1119 -> 1088 us.  64 registers (8 blocks of
// 128 an SM): without the bound 159.6 ms.  In two levels the same change loses
// (1287 -> 1395 us): rays of one tile enter different instances.
template <bool kOpacity>
__global__ void __launch_bounds__(128, 8) k_trace_first(const CwNode* __restrict__ nodes, const CwTri* __restrict__ tris,
                                                        const __grid_constant__ TraceArgs a) {
    const TraceRays rays = trace_rays(a);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rays.n) return;
    float4 o, d;
    rays.load(i, o, d);
    float t, u, v;
    const uint32_t leaf =
        trace_ray<false, false>(make_ray(o, d), d.w, nodes, tris, t, u, v, nullptr, kOpacity ? rays.seed(i) : 0u);
    rays.hit(i, leaf, t, u, v, kMissPrim);
}

// The shadow rays of the camera rays' hits towards the lights, in the same way:
// those of one pixel's samples or of a tile start next to one another and head
// the same way.  In k_trace's queue behind the extension rays the warps reach
// them with rays at every stage of their walks and never hold a pixel's 32 rays
// together; a launch of its own keeps them so (k_trace alone for them already
// gains from 16 spp on).
template <bool kOpacity>
__global__ void __launch_bounds__(128, 8) k_trace_sun(const CwNode* __restrict__ nodes, const CwTri* __restrict__ tris,
                                                      const __grid_constant__ TraceArgs a) {
    const TraceRays rays = trace_rays(a);
    for (uint64_t k = blockIdx.x * blockDim.x + threadIdx.x; k < rays.n; k += gridDim.x * blockDim.x) {
        const uint32_t i = (uint32_t)k;
        float4 o, d;
        rays.load(i, o, d);
        float t, u, v;
        if (trace_ray<true, false>(make_ray(o, d), d.w, nodes, tris, t, u, v, nullptr,
                                   kOpacity ? rays.seed(i) : 0u) == kMissPrim)
            rays.miss(i, d.w);
    }
}

// k_trace for small chunks and short queues: eight lanes per ray.  A
// kernel of its own, because its loop in k_trace costs that one registers
// (1080p 64-spp frame 160.8 -> 168.7 ms with both), and 80 registers are worth
// more here than occupancy (64 of them spill: 443 against 377 us for a 128x128
// 8-segment frame of the room; 96: 369, but slower from 256x256 on).
template <bool kOpacity>
__global__ void __launch_bounds__(kGroupBlock, 6) k_trace_group(const CwNode* __restrict__ nodes,
                                                                const CwTri* __restrict__ tris,
                                                                const __grid_constant__ TraceArgs a) {
    __shared__ GroupStacks stacks;
    const TraceRays rays = trace_rays(a);
    trace_queue_group<kOpacity>(nodes, tris, rays.n, rays.work(), rays, stacks);
}

// The same for two-level scenes: trace_queue2 (TLAS leaves enter instances).
// 80 registers: at 64 the loop spills (1,000 instances, 1-spp 4-segment frame:
// 1241 -> 1116 us at 641x359, 2437 -> 2313 us at 1280x720).
template <bool kOpacity>
__global__ void __launch_bounds__(256, 3) k_trace2(const CwNode* __restrict__ tlas, const InstDev* __restrict__ insts,
                                                   const float* __restrict__ mat_tr,
                                                   const __grid_constant__ TraceArgs a) {
    const TraceRays rays = trace_rays(a);
    trace_queue2<kOpacity>(tlas, insts, mat_tr, rays.n, rays.work(), rays, a.postpone_sp, a.refill_min);
}

// The same in two levels.
template <bool kOpacity>
__global__ void __launch_bounds__(kGroupBlock, kGroup2Blocks) k_trace2_group(const CwNode* __restrict__ tlas,
                                                                 const InstDev* __restrict__ insts,
                                                                 const float* __restrict__ mat_tr,
                                                                 const __grid_constant__ TraceArgs a) {
    __shared__ GroupStacks2 stacks;
    const TraceRays rays = trace_rays(a);
    trace_queue2_group<kOpacity>(tlas, insts, mat_tr, rays.n, rays.work(), rays, stacks);
}

// ----------------------------------------------------------------- shade ----
// kGeneral: point, spot or rect lights, or radiance-cache queries; the slim
// variant (directional lights only, no cache) leaves that code out.
template <bool kGeneral>
__global__ void __launch_bounds__(512, 2) k_shade(DevScene sc, const DevView* __restrict__ views, Wavefront wf,
                                               int q, uint32_t seg, float4* accum) {
    const uint32_t n = wf.counters[kCntQueue + seg];
    const uint32_t cap = wf.capacity;
    const uint32_t sh_cap = cap * (sc.num_lights + 1u);
    const float4* __restrict__ in_o = wf.ray_o[q];
    const float4* __restrict__ in_d = wf.ray_d[q];
    const uint4* __restrict__ in_p = wf.path[q];
    const float4* __restrict__ in_t = wf.thr[q];
    float4* out_o = wf.ray_o[q ^ 1];
    float4* out_d = wf.ray_d[q ^ 1];
    uint4* out_p = wf.path[q ^ 1];
    float4* out_t = wf.thr[q ^ 1];
    const uint32_t stride = gridDim.x * blockDim.x;
    if (threadIdx.x <= kDirBins) s_dir_cnt[0][threadIdx.x] = 0u;
    __syncthreads();
    int parity = 0;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride, parity ^= 1) {
        uint32_t i = base + threadIdx.x;
        bool active = i < n;
        float4 o4 = make_float4(0, 0, 0, 0), d4 = make_float4(0, 0, 1, 0), h4 = make_float4(0, 0, 0, 0);
        float4 t4 = make_float4(0, 0, 0, 0);
        uint4 m4 = make_uint4(0, 0, 0, 0);
        if (active) { o4 = in_o[i]; d4 = in_d[i]; h4 = wf.hit[i]; t4 = in_t[i]; m4 = in_p[i]; }
        uint32_t leaf = active ? __float_as_uint(h4.y) : kMissPrim;
        bool is_hit = active && leaf != kMissPrim;
        uint32_t segi = m4.y & 0xffu, maxseg = (m4.y >> 8) & 0xffu, view_id = m4.y >> 16;
        V3 thr = v3(t4.x, t4.y, t4.z);
        V3 d = v3(d4.x, d4.y, d4.z);
        bool sky_nee = sc.num_lights + 1u > 0u;  // placeholder, refined below per view
        uint32_t vflags = 0;
        uint32_t stream = 0;
        uint32_t cache_seg = 0;
        float cache_rough = 0.0f;
        if (active) {
            const DevView& v = views[view_id];
            vflags = v.flags;
            stream = m4.x - v.accum_base;
            cache_seg = v.cache_segment;
            cache_rough = v.cache_min_rough;
        }
        sky_nee = (vflags & BSM_PT_NO_SKY_NEE) == 0u;
        if (active && !is_hit) {
            // deferred_lighting_secondary.hlsl:23-29: skybox x weight on a miss,
            // here with the MIS weight against sky next-event estimation.
            V3 le = sky_eval(sc.sky, d);
            float w = 1.0f;
            if (segi > 0u && sky_nee) {
                float pb = t4.w;
                float pl = sky_pdf(sc.sky, d);
                float pb2 = pb * pb, pl2 = pl * pl;
                w = pb2 + pl2 > 0.0f ? pb2 / (pb2 + pl2) : 1.0f;
            }
            V3 c = thr * le * w;
            if (max_comp(c) > 0.0f) accum_add(accum, wf.accum_fx, m4.x, c);
        }
        // surface at the hit: N shades (the interpolated vertex normal where the scene has them), Ng offsets
        V3 N = v3(0.0f, 0.0f, 1.0f), Ng = N, P = v3(0.0f, 0.0f, 0.0f);
        Surface surf;
        surf.base_color = v3s(0.5f); surf.f0 = v3s(0.04f); surf.f90 = v3s(1.0f); surf.roughness = 0.5f; surf.ior = 1.5f;
        if (is_hit) {
            V3 ng, edge;
            uint32_t mi;
            hit_geometry(sc, leaf, sc.insts ? __float_as_uint(h4.z) : kMissPrim, ng, edge, mi);
            if (dot(ng, d) > 0.0f) ng = -ng;
            Ng = ng;
            N = ng;
            if (sc.tri_normals) {
                N = shading_normal(sc, leaf, h4.z, h4.w, ng);
                if (dot(N, d) > 0.0f) N = -N;
            }
            P = v3(o4.x, o4.y, o4.z) + d * h4.x;
            float4 m0 = sc.materials[2 * mi], m1 = sc.materials[2 * mi + 1];
            surf.base_color = v3(m0.x, m0.y, m0.z);
            surf.roughness = m0.w;
            surf.f0 = v3(m1.x, m1.y, m1.z);
        }
        Frame fr = create_frame(N);
        V3 V = -d;
        Pcg g;
        g.state = ((uint64_t)m4.w << 32) | m4.z;
        g.inc = ((uint64_t)stream << 1) | 1u;
        float u_sky0 = 0.0f, u_sky1 = 0.0f, u_sky2 = 0.0f, u_lobe = 0.0f, u_b0 = 0.0f, u_b1 = 0.0f;
        if (is_hit) {
            u_sky0 = pcg_uniform(g); u_sky1 = pcg_uniform(g); u_sky2 = pcg_uniform(g); u_lobe = pcg_uniform(g);
            u_b0 = pcg_uniform(g); u_b1 = pcg_uniform(g);
        }
        // radiance cache: a hit of the cache segment (or a later one, when the earlier hits were too smooth)
        // becomes a query (NRC-style termination) — the cache's prediction includes the direct light there
        bool cache_q = kGeneral && is_hit && cache_seg != 0u && segi >= cache_seg &&
                       (surf.roughness >= cache_rough || segi + 1u >= maxseg);
        {
            uint32_t slot = warp_alloc(cache_q, wf.counters + kCntCache);
            if (cache_q) {
                if (slot < cap && wf.cache_q) {
                    float raw[kMlpRaw];
                    mlp_raw_inputs(P, v3(sc.box_lo[0], sc.box_lo[1], sc.box_lo[2]),
                                   v3(sc.box_inv[0], sc.box_inv[1], sc.box_inv[2]), -d, N, surf.roughness,
                                   surf.base_color, (float)segi * 0.125f, raw);
                    float4* qd = wf.cache_q + 4 * (size_t)slot;
                    qd[0] = make_float4(raw[0], raw[1], raw[2], raw[3]);
                    qd[1] = make_float4(raw[4], raw[5], raw[6], raw[7]);
                    qd[2] = make_float4(raw[8], raw[9], raw[10], raw[11]);
                    qd[3] = make_float4(thr.x, thr.y, thr.z, __uint_as_float(m4.x));
                } else {
                    atomicOr(wf.counters + kCntError, 1u);
                }
            }
        }
        if (cache_q) is_hit = false;  // no NEE, no continuation at a cache vertex
        V3 org = P + Ng * sc.ray_offset;
        const DevView* vp = views + view_id;
        float ray_len = is_hit ? vp->ray_length : 0.0f;
        float tmin = is_hit ? vp->t_min : 0.0f;
        float rx = 0.001f, ry = 0.001f;
        aniso_roughness(surf.roughness, &rx, &ry);
        V3 lv = to_local(fr, V);
        float p_spec = spec_probability(surf, lv.z);
        // next-event estimation towards the lights (lights.hlsl:10-25; rect lights sampled by area),
        // deferred_lighting_secondary.hlsl:51-96.  Rect lights draw their two uniforms here, after
        // the vertex's six, in light order.
        for (uint32_t l = 0; l < (uint32_t)kMaxLights; ++l) {
            if (l >= sc.num_lights) break;
            const DevLight& lt = sc.lights[l];
            V3 c = v3s(0.0f), L = v3s(0.0f);
            float smax = ray_len;
            float ur0 = 0.0f, ur1 = 0.0f;
            if (kGeneral && is_hit && __float_as_uint(lt.a.w) == kLightRect) {
                ur0 = pcg_uniform(g);
                ur1 = pcg_uniform(g);
            }
            bool emit = false;
            if (is_hit && (vflags & BSM_PT_NO_SUN_NEE) == 0u) {
                V3 e;
                bool lit;
                if (kGeneral) {
                    lit = light_sample(lt, P, ur0, ur1, ray_len, L, smax, e);
                } else {  // directional: light_sample's first case
                    L = v3(lt.a.x, lt.a.y, lt.a.z);
                    e = v3(lt.b.x, lt.b.y, lt.b.z);
                    smax = ray_len;
                    lit = true;
                }
                if (lit) {
                    V3 f = surface_eval_lit(N, fr.x, fr.y, V, L, surf);
                    c = thr * e * f;
                    emit = max_comp(c) > 0.0f;
                }
            }
            uint32_t slot = warp_alloc(emit, wf.counters + kCntShadow + seg);
            if (emit) {
                if (slot < cap * sc.num_lights) {
                    wf.sh_o[slot] = make_float4(org.x, org.y, org.z, tmin);
                    wf.sh_d[slot] = make_float4(L.x, L.y, L.z, smax);
                    wf.sh_c[slot] = make_float4(c.x, c.y, c.z, __uint_as_float(m4.x));
                    if (sc.has_non_opaque && wf.sh_seed) wf.sh_seed[slot] = (uint32_t)g.state;
                } else {
                    atomicOr(wf.counters + kCntError, 1u);
                }
            }
        }
        // next-event estimation: sky, MIS (power heuristic) against BSDF sampling
        {
            V3 c = v3s(0.0f), L = v3s(0.0f);
            bool emit = false;
            if (is_hit && sky_nee) {
                float pl;
                V3 le;
                L = sky_sample(sc.sky, u_sky0, u_sky1, u_sky2, pl, le);
                if (pl > 0.0f) {
                    V3 f = surface_eval_lit(N, fr.x, fr.y, V, L, surf);
                    if (max_comp(f) > 0.0f) {
                        V3 ll = to_local(fr, L);
                        float pb = mixture_pdf(lv, ll, rx, ry, p_spec);
                        float pl2 = pl * pl, pb2 = pb * pb;
                        float w = pl2 / (pl2 + pb2);
                        c = thr * le * f * (w / pl);
                        emit = max_comp(c) > 0.0f;
                    }
                }
            }
            uint32_t slot = warp_alloc(emit, wf.counters + kCntSky + seg);
            if (emit) {
                if (slot < cap) {
                    uint32_t k = sh_cap - 1u - slot;   // sky rays fill the queue from the back
                    wf.sh_o[k] = make_float4(org.x, org.y, org.z, tmin);
                    wf.sh_d[k] = make_float4(L.x, L.y, L.z, ray_len);
                    wf.sh_c[k] = make_float4(c.x, c.y, c.z, __uint_as_float(m4.x));
                    if (sc.has_non_opaque && wf.sh_seed) wf.sh_seed[k] = (uint32_t)g.state;
                } else {
                    atomicOr(wf.counters + kCntError, 1u);
                }
            }
        }
        // next direction: lobe mixture (sample_secondary_ray.hlsl:16-28 termination, :51-64 weight)
        bool cont = false;
        V3 nthr = v3s(0.0f), L = v3s(0.0f);
        float pdf = 0.0f;
        if (is_hit && segi + 1u < maxseg && max_comp(thr) >= 0.001f) {
            V3 ll;
            if (u_lobe < p_spec) {
                V3 h = ggx_vndf_sample(lv, rx, ry, u_b0, u_b1);
                ll = reflect(-lv, h);
            } else {
                ll = cos_hemisphere_sample(u_b0, u_b1);
            }
            if (ll.z > 0.0f) {
                L = to_world(fr, ll);
                pdf = mixture_pdf(lv, ll, rx, ry, p_spec);
                V3 f = surface_eval_lit(N, fr.x, fr.y, V, L, surf);
                V3 w = pdf > 0.0f ? f / pdf : v3s(0.0f);
                if (!isfinite(w.x) || !isfinite(w.y) || !isfinite(w.z)) w = v3s(0.0f);
                nthr = thr * w;
                cont = max_comp(nthr) > 0.0f;
            }
        }
        // the next rays, grouped by direction per block (sorting the sky shadow rays by octant measured no gain)
        uint32_t slot = block_alloc_by_direction(cont, L, wf.counters + kCntQueue + seg + 1, parity);
        if (cont) {
            if (slot < cap) {
                out_o[slot] = make_float4(org.x, org.y, org.z, tmin);
                out_d[slot] = make_float4(L.x, L.y, L.z, ray_len);
                out_p[slot] = make_uint4(m4.x, (m4.y & 0xffffff00u) | (segi + 1u), (uint32_t)g.state,
                                         (uint32_t)(g.state >> 32));
                out_t[slot] = make_float4(nthr.x, nthr.y, nthr.z, pdf);
            } else {
                atomicOr(wf.counters + kCntError, 1u);
            }
        }
    }
}

// --------------------------------------------------------------- resolve ----
// The call's fixed-point sums added to the FP32 accumulator, one add per pixel and channel.
__global__ void k_fold_fixed(const unsigned long long* __restrict__ fx, float4* __restrict__ accum, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long* p = fx + 3 * (size_t)i;
    float4 a = accum[i];
    a.x += (float)((double)p[0] * 0x1p-32);
    a.y += (float)((double)p[1] * 0x1p-32);
    a.z += (float)((double)p[2] * 0x1p-32);
    accum[i] = a;
}

__global__ void k_resolve_fixed(const unsigned long long* __restrict__ fx, uint32_t width, uint32_t height,
                                float inv_spp, float4* __restrict__ out, uint32_t pitch) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= width || y >= height) return;
    const unsigned long long* p = fx + 3 * ((size_t)y * width + x);
    out[(size_t)y * pitch + x] = make_float4((float)((double)p[0] * 0x1p-32) * inv_spp,
                                             (float)((double)p[1] * 0x1p-32) * inv_spp,
                                             (float)((double)p[2] * 0x1p-32) * inv_spp, 1.0f);
}

__global__ void k_resolve(const float4* __restrict__ accum, uint32_t width, uint32_t height, float inv_spp,
                          float4* __restrict__ out, uint32_t pitch) {
    uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t y = blockIdx.y;
    if (x >= width || y >= height) return;
    float4 a = accum[(size_t)y * width + x];
    out[(size_t)y * pitch + x] = make_float4(a.x * inv_spp, a.y * inv_spp, a.z * inv_spp, 1.0f);
}

// ------------------------------------------------------- vertex normals ----
// The three vertex normals of every leaf triangle, in leaf order, from the
// scene's per-vertex normals (indexed like the positions).
__global__ void k_gather_normals(const CwTri* __restrict__ tris, uint32_t n, const float* __restrict__ vn,
                                 const uint32_t* __restrict__ idx, float4* __restrict__ out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t prim = tris[i].prim;
    for (int k = 0; k < 3; ++k) {
        const size_t v = idx ? idx[3 * (size_t)prim + k] : 3 * (size_t)prim + k;
        out[3 * (size_t)i + k] = make_float4(vn[3 * v], vn[3 * v + 1], vn[3 * v + 2], 0.0f);
    }
}

// ------------------------------------------------------ stage entry points ----
// Rays of the stage entry points (a caller's array) and of small views' primary
// outputs (a pixel-centre camera ray per pixel), on the wavefront's loops.
struct StageArgs {
    const float4* rays;       // a caller's rays (origin/tmin, direction/tmax)
    uint4* hits;              // t, primitive id, u, v of each ray
    uint8_t* occluded;        // or whether it hit anything
    float4* rec;              // or, of the camera rays of `view`, hit records (t, leaf, u, v) for k_primary_rec
    const CwTri* tris;        // for the primitive ids
    const InstDev* insts;
    uint32_t n;
    uint32_t* work;           // [2], zero between launches; null: the launch takes its rays without a counter
    float near;               // k_stage: how far apart the origins of rays that are traced side by side may be
    int postpone_sp, refill_min;
    DevView view;
};
// A kernel is made for one kind of rays and output: asking which at every ray and hit cost the loops 2 to 4 % and
// registers (non-opaque materials, 1,000,003 closest hits in the room: 376 -> 323 us). kStageEither, which asks, is for
// two kernels that come out slower when they know (stage2_out).
enum : int { kStageHits, kStageOccluded, kStageRec, kStageEither };
template <int kOut>
struct StageRays {
    const StageArgs& a;
    __device__ __forceinline__ bool to_hits() const { return kOut == kStageEither ? a.hits != nullptr : kOut == kStageHits; }
    __device__ __forceinline__ bool any(uint32_t) const { return kOut == kStageEither ? a.occluded != nullptr : kOut == kStageOccluded; }
    __device__ __forceinline__ void load(uint32_t i, float4& o, float4& d) const {
        if (kOut == kStageEither ? a.rays != nullptr : kOut != kStageRec) {
            o = __ldg(a.rays + 2 * (size_t)i);
            d = __ldg(a.rays + 2 * (size_t)i + 1);
            return;
        }
        o = make_float4(a.view.pos[0], a.view.pos[1], a.view.pos[2], a.view.t_min);
        const uint32_t py = i / a.view.width;
        const V3 dw = camera_dir(a.view, i - py * a.view.width, py, 0.5f, 0.5f);
        d = make_float4(dw.x, dw.y, dw.z, a.view.ray_length);
    }
    __device__ __forceinline__ void hit(uint32_t i, uint32_t leaf, float t, float u, float v, uint32_t inst) const {
        if (to_hits()) {
            const uint32_t prim = inst != kMissPrim ? a.insts[inst].prim_base + a.insts[inst].tris[leaf].prim
                                                    : a.tris[leaf].prim;
            a.hits[i] = make_uint4(__float_as_uint(t), prim, __float_as_uint(u), __float_as_uint(v));
        } else if (kOut == kStageEither ? a.occluded != nullptr : kOut != kStageRec) {
            a.occluded[i] = 1;
        } else {
            a.rec[i] = make_float4(t, __uint_as_float(leaf), u, v);
        }
    }
    __device__ __forceinline__ void miss(uint32_t i, float tmax) const {
        if (to_hits()) a.hits[i] = make_uint4(__float_as_uint(tmax), kMissPrim, 0u, 0u);
        else if (kOut == kStageEither ? a.occluded != nullptr : kOut != kStageRec) a.occluded[i] = 0;
        else a.rec[i] = make_float4(tmax, __uint_as_float(kMissPrim), 0.0f, 0.0f);
    }
    // opacity decisions: a caller's rays draw with seed 0, a pixel's with the camera-ray PCG word of sample 0 of
    // an unjittered render
    __device__ __forceinline__ uint32_t seed(uint32_t i) const {
        if (kOut == kStageEither ? a.rays != nullptr : kOut != kStageRec) return 0u;
        return (uint32_t)pcg_seed(path_initstate(a.view.seed, a.view.sample_offset, i), (uint64_t)i).state;
    }
};

// The work counter goes back to zero when the launch's last block is done with it.
__device__ __forceinline__ void stage_done(uint32_t* work) {
    if (!work) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(work + 1, 1u) == gridDim.x - 1u) { work[0] = 0u; work[1] = 0u; }
    }
}
// Eight lanes per ray: the first rays of every warp come without a counter, so a grid that holds all of them needs
// none (the one in shared memory only says that the rays are out).
__device__ __forceinline__ uint32_t* group_work(const StageArgs& a, uint32_t* s_work) {
    if (a.work) return a.work;
    if (threadIdx.x == 0) *s_work = 0u;
    __syncthreads();
    return s_work;
}

// A ray per thread: no queue and no counter.
template <int kOut, bool kTwoLevel>
__global__ void __launch_bounds__(128, kTwoLevel ? 5 : 8) k_stage_ray(const CwNode* __restrict__ nodes,
                                                                      const CwTri* __restrict__ tris,
                                                                      const InstDev* __restrict__ insts,
                                                                      const float* __restrict__ mat_tr,
                                                                      const __grid_constant__ StageArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    constexpr bool kAny = kOut == kStageOccluded;
    const StageRays<kOut> rays{a};
    float4 o, d;
    rays.load(i, o, d);
    float t, u, v;
    uint32_t inst = kMissPrim, leaf;
    if (kTwoLevel) leaf = trace_ray2<kAny>(make_ray(o, d), d.w, nodes, insts, mat_tr, t, u, v, inst, rays.seed(i));
    else leaf = trace_ray<kAny, false>(make_ray(o, d), d.w, nodes, tris, t, u, v, nullptr, rays.seed(i));
    if (leaf == kMissPrim) rays.miss(i, d.w);
    else rays.hit(i, leaf, t, u, v, inst);
}

// More rays than fit at once, whose lanes take new ones when theirs are done:
// with a ray per thread every warp waits for its longest ray.  But rays that
// start side by side and head the same way are done together, and the loop's
// votes, queue reads and postponed leaves then cost more than the waiting (a
// quarter of the time where materials are not opaque), so a warp whose 32 rays
// are alike traces them a ray per lane and looks at the next 32.  A ray per
// thread / the loop alone / this kernel, us, closest hits of 1,000,003 rays:
// incoherent ones in 1.48 M triangles 653 / 416 / 408, in the room 384 / 266 / 261;
// a camera's 246 / 301 / 261 and 219 / 299 / 247, with non-opaque materials 310 / 484 / 358.
template <bool kOpacity, int kOut>
__global__ void __launch_bounds__(128, 8) k_stage(const CwNode* __restrict__ nodes, const CwTri* __restrict__ tris,
                                                  const __grid_constant__ StageArgs a) {
    constexpr uint32_t kFull = 0xffffffffu;
    constexpr bool kAny = kOut == kStageOccluded;
    const StageRays<kOut> rays{a};
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t head = 0u;
    while (true) {
        if (lane == 0) head = atomicAdd(a.work, 32u);
        head = __shfl_sync(kFull, head, 0);
        if (head >= a.n) break;
        const uint32_t i = min(head + lane, a.n - 1u);
        float4 o, d;
        rays.load(i, o, d);
        const uint32_t oct = (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
        const uint32_t oct0 = __shfl_sync(kFull, oct, 0);
        const float x0 = __shfl_sync(kFull, o.x, 0), y0 = __shfl_sync(kFull, o.y, 0), z0 = __shfl_sync(kFull, o.z, 0);
        const bool alike = oct == oct0 && fabsf(o.x - x0) <= a.near && fabsf(o.y - y0) <= a.near && fabsf(o.z - z0) <= a.near;
        if (!__all_sync(kFull, alike)) break;
        if (head + lane < a.n) {
            float t, u, v;
            const uint32_t leaf =
                trace_ray<kAny, false>(make_ray(o, d), d.w, nodes, tris, t, u, v, nullptr, kOpacity ? rays.seed(i) : 0u);
            if (leaf == kMissPrim) rays.miss(i, d.w);
            else rays.hit(i, leaf, t, u, v, kMissPrim);
        }
        __syncwarp();
    }
    if (head < a.n)
        trace_queue<false, kOpacity, true>(nodes, tris, a.n, a.work, rays, nullptr, a.postpone_sp, a.refill_min, head);
    stage_done(a.work);
}
template <bool kOpacity, int kOut>
__global__ void __launch_bounds__(kGroupBlock, 6) k_stage_group(const CwNode* __restrict__ nodes,
                                                                const CwTri* __restrict__ tris,
                                                                const __grid_constant__ StageArgs a) {
    __shared__ GroupStacks stacks;
    __shared__ uint32_t s_work;
    trace_queue_group<kOpacity>(nodes, tris, a.n, group_work(a, &s_work), StageRays<kOut>{a}, stacks);
    stage_done(a.work);
}
template <bool kOpacity, int kOut>
__global__ void __launch_bounds__(kGroupBlock, kGroup2Blocks) k_stage2_group(const CwNode* __restrict__ tlas,
                                                                 const InstDev* __restrict__ insts,
                                                                 const float* __restrict__ mat_tr,
                                                                 const __grid_constant__ StageArgs a) {
    __shared__ GroupStacks2 stacks;
    __shared__ uint32_t s_work;
    trace_queue2_group<kOpacity>(tlas, insts, mat_tr, a.n, group_work(a, &s_work), StageRays<kOut>{a}, stacks);
    stage_done(a.work);
}
// Closest hits of opaque and any hits of non-opaque scenes come out slower when their kernel knows its output, the other
// two faster (1,500,003 incoherent rays, 300 instances, knowing / asking: closest 705 / 576 and non-opaque 628 / 697 us,
// any 261 / 290 and 454 / 403).
constexpr int stage2_out(bool opacity, int out) {
    return opacity == (out == kStageOccluded) ? (int)kStageEither : out;
}
template <bool kOpacity, int kOut>
__global__ void __launch_bounds__(128, 8) k_stage2(const CwNode* __restrict__ tlas, const InstDev* __restrict__ insts,
                                                   const float* __restrict__ mat_tr,
                                                   const __grid_constant__ StageArgs a) {
    trace_queue2<kOpacity>(tlas, insts, mat_tr, a.n, a.work, StageRays<kOut>{a}, a.postpone_sp, a.refill_min);
    stage_done(a.work);
}

// ------------------------------------------------------ primary outputs ----
// The primary-hit outputs of the pass: one pixel-centre camera ray per pixel and
// its closest hit, as the reference's first trace of a frame
// (generate_camera_ray.hlsl:9-15, rt_gbuffer.hlsl:7-36), written as reverse-Z
// depth (pt_depth.hlsl:7-16), the packed G-buffer (gbuffer.hlsl:18-31) and hit
// positions.  The normal is the geometric one faced towards the ray (as
// k_shade), the tangent the triangle's first edge.  A miss writes depth 0, hit
// position (direction, -1) and a zero G-buffer.  Outputs are tightly packed
// width*height arrays; any may be null.
struct PrimaryOut {
    float* depth;
    float4* gb[4];
    float4* hitpos;
    float near_z, far_z;
};
// Writes pixel i's outputs for its hit (leaf, t, u, v, instance).
__device__ __forceinline__ void write_primary(const DevScene& sc, const DevView& v, const PrimaryOut& out, uint32_t i,
                                              V3 dw, uint32_t leaf, float t, float hu, float hv, uint32_t inst) {
    const V3 eye = v3(v.pos[0], v.pos[1], v.pos[2]);
    float g[16];
    float z = 0.0f;
    float4 hp;
    if (leaf == kMissPrim) {
#pragma unroll
        for (int k = 0; k < 16; ++k) g[k] = 0.0f;
        hp = make_float4(dw.x, dw.y, dw.z, -1.0f);
    } else {
        V3 ng, edge;
        uint32_t mi;
        hit_geometry(sc, leaf, inst, ng, edge, mi);
        if (dot(ng, dw) > 0.0f) ng = -ng;
        if (sc.tri_normals) {
            ng = shading_normal(sc, leaf, hu, hv, ng);
            if (dot(ng, dw) > 0.0f) ng = -ng;
        }
        V3 T = normalize(edge);
        float4 m0 = sc.materials[2 * mi], m1 = sc.materials[2 * mi + 1];
        pack_gbuffer(ng, T, v3(m0.x, m0.y, m0.z), v3(m1.x, m1.y, m1.z), m0.w, g);
        V3 P = eye + dw * t;
        z = reverse_z_depth(eye, v3(v.f[0], v.f[1], v.f[2]), P, out.near_z, out.far_z);
        hp = make_float4(P.x, P.y, P.z, t);
    }
    if (out.depth) out.depth[i] = z;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (out.gb[k]) out.gb[k][i] = make_float4(g[4 * k], g[4 * k + 1], g[4 * k + 2], g[4 * k + 3]);
    if (out.hitpos) out.hitpos[i] = hp;
}
// Seed of a pixel's opacity decisions: sample 0 of an unjittered render (its camera-ray PCG word).
__device__ __forceinline__ uint32_t primary_seed(const DevView& v, uint32_t i) {
    return (uint32_t)pcg_seed(path_initstate(v.seed, v.sample_offset, i), (uint64_t)i).state;
}

// One pixel per lane, eight by four pixels per warp, sixteen by eight per block.
// The camera rays of such a tile visit nearly the same nodes, so a lane's own
// loop with neither queue nor refills is the fastest here, at 64 registers, and
// the outputs leave in whole sectors.  1920x1080 of the 1.48 M-triangle terrain:
// 831 us with a row of pixels per warp, 637 in tiles, 608 in tiles at 64
// registers (691 with the queue loop's postponed triangles, 748 as hit records
// from the persistent loop and a second kernel).
template <bool kTwoLevel>
__global__ void __launch_bounds__(128, kTwoLevel ? 5 : 8) k_primary(DevScene sc, const __grid_constant__ DevView v,
                                                                    PrimaryOut out) {
    const uint32_t across = (v.width + 15u) / 16u, ty = blockIdx.x / across, tx = blockIdx.x - ty * across;
    const uint32_t w = threadIdx.x >> 5, l = threadIdx.x & 31u;
    const uint32_t px = tx * 16u + (w & 1u) * 8u + (l & 7u), py = ty * 8u + (w >> 1) * 4u + (l >> 3);
    if (px >= v.width || py >= v.height) return;
    const uint32_t i = py * v.width + px;
    const V3 dw = camera_dir(v, px, py, 0.5f, 0.5f);
    RayPre r = make_ray(make_float4(v.pos[0], v.pos[1], v.pos[2], v.t_min), make_float4(dw.x, dw.y, dw.z, v.ray_length));
    float t, hu, hv;
    uint32_t inst = kMissPrim, leaf;
    const uint32_t seed = sc.has_non_opaque ? primary_seed(v, i) : 0u;
    if (kTwoLevel) leaf = trace_ray2<false>(r, v.ray_length, sc.nodes, sc.insts, sc.mat_tr, t, hu, hv, inst, seed);
    else leaf = trace_ray<false, false>(r, v.ray_length, sc.nodes, sc.tris, t, hu, hv, nullptr, seed);
    write_primary(sc, v, out, i, dw, leaf, t, hu, hv, inst);
}
// Small views, from the hit records that k_stage_group left in one of the outputs.
__global__ void __launch_bounds__(128) k_primary_rec(DevScene sc, const __grid_constant__ DevView v, PrimaryOut out,
                                                     const float4* rec) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.width * v.height) return;
    const float4 h = rec[i];
    const uint32_t py = i / v.width;
    write_primary(sc, v, out, i, camera_dir(v, i - py * v.width, py, 0.5f, 0.5f), __float_as_uint(h.y), h.x, h.z, h.w,
                  kMissPrim);
}

__global__ void __launch_bounds__(256) k_trace_count(DevScene sc, const float4* __restrict__ rays, uint32_t n,
                                                     uint2* __restrict__ counts) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 o = rays[2 * (size_t)i], d = rays[2 * (size_t)i + 1];
    RayPre r = make_ray(o, d);
    float t, u, v;
    TraceCounters c{0, 0};
    trace_ray<false, true>(r, d.w, sc.nodes, sc.tris, t, u, v, &c);
    counts[i] = make_uint2(c.nodes, c.tris);
}

// ------------------------------------------------------ moved instances ----
// New records and world boxes of moved instances, a thread per instance, in the
// operation order of the host's invert_affine and instance_world_box (double
// precision, each operation rounded once), so the values are the same bits.  `sum`
// (zero before): [0] the complement of the first transform that is not finite or
// invertible, [1..3] complements of the box minima's order keys, [4..6] the
// maxima's.  On the host one core took 190 us for 1,000 instances.
__device__ __forceinline__ uint32_t order_key(float f) {   // unsigned order = float order
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__global__ void __launch_bounds__(128) k_inst_move(const float* __restrict__ transforms,
                                                   const InstSrc* __restrict__ src, uint32_t n,
                                                   InstMoved* __restrict__ out, uint32_t* sum) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float m[12];
    bool ok = true;
    for (int k = 0; k < 12; ++k) {
        m[k] = transforms[12 * (size_t)i + k];
        ok = ok && isfinite(m[k]);
    }
    const double L00 = m[0], L01 = m[1], L02 = m[2], t0 = m[3];
    const double L10 = m[4], L11 = m[5], L12 = m[6], t1 = m[7];
    const double L20 = m[8], L21 = m[9], L22 = m[10], t2 = m[11];
    const double c00 = L11 * L22 - L12 * L21, c01 = L02 * L21 - L01 * L22, c02 = L01 * L12 - L02 * L11;
    const double c10 = L12 * L20 - L10 * L22, c11 = L00 * L22 - L02 * L20, c12 = L02 * L10 - L00 * L12;
    const double c20 = L10 * L21 - L11 * L20, c21 = L01 * L20 - L00 * L21, c22 = L00 * L11 - L01 * L10;
    const double det = L00 * c00 + L01 * c10 + L02 * c20;
    ok = ok && isfinite(det) && fabs(det) > 1e-30;
    if (!ok) {
        atomicMax(sum, ~i);
        return;
    }
    const InstSrc g = src[i];
    InstMoved& o = out[g.leaf];
    const double r[9] = {c00 / det, c01 / det, c02 / det, c10 / det, c11 / det, c12 / det, c20 / det, c21 / det, c22 / det};
    for (int k = 0; k < 3; ++k) {
        o.w2o[4 * k] = (float)r[3 * k];
        o.w2o[4 * k + 1] = (float)r[3 * k + 1];
        o.w2o[4 * k + 2] = (float)r[3 * k + 2];
        o.w2o[4 * k + 3] = (float)(-(r[3 * k] * t0 + r[3 * k + 1] * t1 + r[3 * k + 2] * t2));
    }
    for (int k = 0; k < 12; ++k) o.o2w[k] = m[k];
    double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int c = 0; c < 8; ++c) {
        const double p[3] = {(c & 1) ? g.hi[0] : g.lo[0], (c & 2) ? g.hi[1] : g.lo[1], (c & 4) ? g.hi[2] : g.lo[2]};
        for (int k = 0; k < 3; ++k) {
            const double w = (double)m[4 * k] * p[0] + (double)m[4 * k + 1] * p[1] + (double)m[4 * k + 2] * p[2] +
                             (double)m[4 * k + 3];
            mn[k] = w < mn[k] ? w : mn[k];
            mx[k] = mx[k] < w ? w : mx[k];
        }
    }
    double mag = 0.0;
    for (int k = 0; k < 3; ++k) {
        const double a = fabs(mn[k]) < fabs(mx[k]) ? fabs(mx[k]) : fabs(mn[k]);
        mag = mag < a ? a : mag;
    }
    const double pad = 1e-5 * mag + 1e-30;
    for (int k = 0; k < 3; ++k) {
        float l = (float)(mn[k] - pad), h = (float)(mx[k] + pad);
        while ((double)l > mn[k] - pad) l = nextafterf(l, -INFINITY);
        while ((double)h < mx[k] + pad) h = nextafterf(h, INFINITY);
        o.box[k] = l;
        o.box[3 + k] = h;
        atomicMax(sum + 1 + k, ~order_key(l));
        atomicMax(sum + 4 + k, order_key(h));
    }
}
__global__ void __launch_bounds__(128) k_inst_apply(const InstMoved* __restrict__ moved, uint32_t n,
                                                    InstDev* __restrict__ insts, float* __restrict__ inst_box) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const InstMoved& o = moved[i];
    for (int k = 0; k < 12; ++k) { insts[i].w2o[k] = o.w2o[k]; insts[i].o2w[k] = o.o2w[k]; }
    for (int k = 0; k < 6; ++k) inst_box[6 * (size_t)i + k] = o.box[k];
}

// ------------------------------------------------------------- TLAS refit ----
// Refits the TLAS for new instance boxes, a breadth-first level at a time from
// the deepest up (nodes of a level are contiguous in the builder's order).  A
// node's eight child boxes come from the instance boxes of its leaf slots (TLAS
// leaves hold one instance) and from the boxes its internal children wrote a
// level earlier; the node's frame and bytes are then quantised outward exactly as
// the host builder does (tlas_quantise), a slot per lane.  A launch per level
// with a thread per node took 42 us for each of the five levels of 1,000
// instances; 20 us for all of them now.
__device__ __forceinline__ void refit_node(CwNode* nodes, float* node_box, const float* inst_box, uint32_t ni, bool in) {
    const uint32_t s = threadIdx.x % kWideLanes;
    uint32_t imask = 0, tmask = 0, child = 0, tri = 0;
    if (in) {
        const CwNode* n = nodes + ni;
        imask = n->imask;
        tmask = n->tri_mask;
        child = n->child_base;
        tri = n->tri_base;
    }
    const bool inner = (imask >> s) & 1u, leaf = !inner && ((tmask >> (2u * s)) & 3u) != 0u;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    if (inner || leaf) {
        const float* b = inner ? node_box + 6 * (size_t)(child + (uint32_t)__popc(imask & ((1u << s) - 1u)))
                               : inst_box + 6 * (size_t)(tri + (uint32_t)__popc(tmask & ((1u << (2u * s)) - 1u)));
        for (int k = 0; k < 3; ++k) { lo[k] = b[k]; hi[k] = b[3 + k]; }
    }
    float nlo[3], nhi[3];
    for (int k = 0; k < 3; ++k) { nlo[k] = wide_min(lo[k]); nhi[k] = wide_max(hi[k]); }
    quantise_lanes(reinterpret_cast<uint8_t*>(nodes + ni), inner || leaf, s, in, lo, hi, nlo, nhi);
    if (in && s < 6u) node_box[6 * (size_t)ni + s] = s == 0 ? nlo[0] : s == 1 ? nlo[1] : s == 2 ? nlo[2]
                                                   : s == 3 ? nhi[0] : s == 4 ? nhi[1] : nhi[2];
}
constexpr uint32_t kRefitThreads = 1024, kRefitNodes = kRefitThreads / kWideLanes;
struct RefitLevels { uint32_t begin[kMaxTlasDepth + 2]; };

// Levels [0, n) by one block, with barriers between them.
__global__ void __launch_bounds__(kRefitThreads) k_tlas_refit(CwNode* nodes, float* node_box, const float* inst_box,
                                                              RefitLevels lv, uint32_t n) {
    for (uint32_t l = n; l-- > 0u;) {
        for (uint32_t base = lv.begin[l]; base < lv.begin[l + 1]; base += kRefitNodes) {
            const uint32_t ni = base + threadIdx.x / kWideLanes;
            refit_node(nodes, node_box, inst_box, ni, ni < lv.begin[l + 1]);
        }
        __syncthreads();
    }
}
// One level by as many blocks as it needs.
__global__ void __launch_bounds__(256) k_tlas_level(CwNode* nodes, float* node_box, const float* inst_box,
                                                    uint32_t begin, uint32_t end) {
    const uint32_t ni = begin + (blockIdx.x * blockDim.x + threadIdx.x) / kWideLanes;
    refit_node(nodes, node_box, inst_box, ni, ni < end);
}

// ------------------------------------------------------------ launchers ----
void launch_inst_move(cudaStream_t st, const float* transforms, const InstSrc* src, uint32_t n, InstMoved* out,
                      uint32_t* sum) {
    k_inst_move<<<(n + 127) / 128, 128, 0, st>>>(transforms, src, n, out, sum);
}
void launch_inst_apply(cudaStream_t st, const InstMoved* moved, uint32_t n, InstDev* insts, float* inst_box) {
    k_inst_apply<<<(n + 127) / 128, 128, 0, st>>>(moved, n, insts, inst_box);
}
void launch_tlas_refit(cudaStream_t st, CwNode* nodes, float* node_box, const float* inst_box,
                       const uint32_t* level_begin, uint32_t levels) {
    // one block takes the levels below the first one that is too wide for a few rounds of it
    uint32_t narrow = 0;
    while (narrow < levels && narrow <= (uint32_t)kMaxTlasDepth &&
           level_begin[narrow + 1] - level_begin[narrow] <= 8u * kRefitNodes)
        ++narrow;
    for (uint32_t l = levels; l-- > narrow;) {
        const uint32_t n = level_begin[l + 1] - level_begin[l];
        k_tlas_level<<<(n * kWideLanes + 255u) / 256u, 256, 0, st>>>(nodes, node_box, inst_box, level_begin[l],
                                                                   level_begin[l + 1]);
    }
    if (narrow == 0) return;
    RefitLevels lv{};
    for (uint32_t l = 0; l <= narrow; ++l) lv.begin[l] = level_begin[l];
    k_tlas_refit<<<1, kRefitThreads, 0, st>>>(nodes, node_box, inst_box, lv, narrow);
}
// Small chunks are generated and shaded in blocks of 128 threads, so that 16,384 paths reach 128 SMs and not 32; larger
// ones in blocks of 512, over which the direction grouping of the next rays spans. 8-segment 1-spp frames, us, 512 / 128
// threads for shading: room 128^2 376 / 362, 256^2 528 / 511, 512^2 896 / 875, 1.48 M triangles 512^2 1232 / 1213, 275,400
// paths 1258 / 1235, from 724^2 on level; for camera rays the two differ by 0.2 % from 200,000 paths on. 64 spp at 1080p
// take 161.3 ms with 512 for shading.
constexpr uint32_t kSmallBlockPaths = 300000;

void launch_camera(const LaunchCfg& lc, cudaStream_t st, const DevView* views, uint32_t n_views,
                   uint64_t path_begin, uint32_t path_count, const Wavefront& wf, uint32_t max_segments) {
    const uint32_t block = path_count <= kSmallBlockPaths ? 128u : (uint32_t)lc.block_shade;
    uint32_t blocks = (path_count + block - 1) / block;
    if (blocks == 0) blocks = 1;
    k_camera<<<blocks, block, 0, st>>>(views, n_views, path_begin, path_count, wf, max_segments);
}
void launch_gather_normals(cudaStream_t st, const CwTri* tris, uint32_t n, const float* vn, const uint32_t* idx,
                           float4* out) {
    if (n) k_gather_normals<<<(n + 255) / 256, 256, 0, st>>>(tris, n, vn, idx, out);
}

// Which kernel traces a segment's queue. Eight lanes per ray win while a launch is as long as its longest ray, a
// lane per ray where throughput counts. The queues' lengths are known only to the device, so:
//  * chunks of up to kGroupPaths paths (two levels: kGroupPaths2) take the group kernel for every segment;
//  * chunks of up to kMixedPaths launch both after the first segment, and each leaves the queues of the other's
//    length alone (2 us for the one that does; the first segment's queue is the chunk itself);
//  * larger chunks, whose later queues are long too, take the lane-per-ray kernel.
// 8-segment 1-spp frames, us, lane / group / both: room 181^2 629 / 433 / 455, 256^2 680 / 549 / 524, 362^2
// 772 / 839 / 670, 512^2 922 / - / 889, 724^2 1180 / - / 1181; 1.48 M triangles 181^2 983 / 643 / 700, 256^2
// 1050 / 825 / 766, 362^2 1173 / 1222 / 934, 512^2 1395 / - / 1240, 724^2 1828 / - / 1775; at 1024^2 (and over)
// both change nothing. Two levels (4 segments, 1,000 instances): 128x72 873 / 443, 320x180 1021 / 661 / 740,
// 641x359 1255 / 2012 / 1238.
constexpr uint32_t kGroupPaths = 40960, kGroupPaths2 = 98304, kMixedPaths = 1000000;
// Longest queue for the group kernel. One level: of 45,000, 70,000 and 100,000 the first is the best in the room
// (512^2 889 / 900 / 927 us) and the second in the terrain (512^2 1251 / 1228 / 1241 us); two levels: 60,000 and
// 90,000 are level, 120,000 is slower (641x359 1240 / 1238 / 1311 us).
constexpr uint32_t kGroupQueue = 56000, kGroupQueue2 = 90000;

// Chunks of more paths than this trace the first hits' rays to the lights in a launch of their own. Frames of 8
// segments, us, in one queue / on their own: 1920x1080 of 1.48 M triangles 64 spp 158500 / 155000, 4 spp 11502 /
// 11361, 1 spp 3616 / 3634; 1280x720x4 5553 / 5520 (250 k triangles 4005 / 3952), 1024^2 2636 / 2685. (First in the
// common queue instead of a launch: 64 spp 155700, but 1 spp 3641, with the longer extension rays as its tail.)
constexpr uint32_t kFirstShadowPaths = 3000000;

void launch_trace(const LaunchCfg& lc, cudaStream_t st, const DevScene& sc, const Wavefront& wf, int q, uint32_t ext,
                  uint32_t shd, float4* accum, uint32_t paths, bool first) {
    if (ext < kNoSegment && shd < kNoSegment && !one_trace_launch(paths, sc.num_lights)) {
        launch_trace(lc, st, sc, wf, q, kNoSegment, shd, accum, paths, first);
        launch_trace(lc, st, sc, wf, q, ext, kNoSegment, accum, paths, first);
        return;
    }
    TraceArgs a{wf.ray_o[q], wf.ray_d[q], wf.path[q], wf.hit, wf.sh_o, wf.sh_d, wf.sh_c, wf.sh_seed, accum,
                wf.accum_fx, wf.counters, wf.stats, ext, shd, wf.capacity * (sc.num_lights + 1u) - 1u,
                ext < kNoSegment ? kCntQueue + ext : kCntZero, shd < kNoSegment ? kCntShadow + shd : kCntZero,
                shd < kNoSegment ? kCntSky + shd : kCntZero, 0u, 0xffffffffu, lc.postpone_sp, lc.refill_min};
    const bool op = sc.has_non_opaque != 0, two = sc.insts != nullptr;
    const bool only = paths <= (two ? kGroupPaths2 : kGroupPaths), mix = !only && paths <= kMixedPaths && ext != 0u;
    if (!only && !two && ext == 0u && shd == kNoSegment) {
        const uint32_t grid = (uint32_t)(((uint64_t)paths + 127u) / 128u);
        if (op) k_trace_first<true><<<grid, 128, 0, st>>>(sc.nodes, sc.tris, a);
        else k_trace_first<false><<<grid, 128, 0, st>>>(sc.nodes, sc.tris, a);
        return;
    }
    if (first && shd == 0u && !two && paths > kFirstShadowPaths && sc.num_lights != 0u) {
        TraceArgs b = a;
        b.ext_cnt = b.sky_cnt = kCntZero;
        const uint32_t grid = (uint32_t)(((uint64_t)paths + 127u) / 128u);   // one light's rays; the loop takes others'
        if (op) k_trace_sun<true><<<grid, 128, 0, st>>>(sc.nodes, sc.tris, b);
        else k_trace_sun<false><<<grid, 128, 0, st>>>(sc.nodes, sc.tris, b);
        a.sun_cnt = kCntZero;
    }
    const uint32_t limit = two ? kGroupQueue2 : kGroupQueue;
    if (only || mix) {
        if (mix) a.max_rays = limit;
        if (two && op) k_trace2_group<true><<<lc.grid_group2, kGroupBlock, 0, st>>>(sc.nodes, sc.insts, sc.mat_tr, a);
        else if (two) k_trace2_group<false><<<lc.grid_group2, kGroupBlock, 0, st>>>(sc.nodes, sc.insts, sc.mat_tr, a);
        else if (op) k_trace_group<true><<<lc.grid_group, kGroupBlock, 0, st>>>(sc.nodes, sc.tris, a);
        else k_trace_group<false><<<lc.grid_group, kGroupBlock, 0, st>>>(sc.nodes, sc.tris, a);
        if (only) return;
        a.min_rays = limit + 1u;
        a.max_rays = 0xffffffffu;
    }
    if (two) {
        if (op) k_trace2<true><<<lc.grid_persistent2, lc.block_trace, 0, st>>>(sc.nodes, sc.insts, sc.mat_tr, a);
        else k_trace2<false><<<lc.grid_persistent2, lc.block_trace, 0, st>>>(sc.nodes, sc.insts, sc.mat_tr, a);
        return;
    }
#define BSM_TRACE(B, O) k_trace<B, O><<<lc.grid_persistent, lc.block_trace, 0, st>>>(sc.nodes, sc.tris, a)
    if (lc.regcap) { if (op) BSM_TRACE(4, true); else BSM_TRACE(4, false); }
    else { if (op) BSM_TRACE(1, true); else BSM_TRACE(1, false); }
#undef BSM_TRACE
}
void launch_extend_count(const LaunchCfg& lc, cudaStream_t st, const DevScene& sc, const Wavefront& wf, int q,
                         uint32_t seg) {
    if (sc.insts) { launch_trace(lc, st, sc, wf, q, seg, kNoSegment, nullptr, 0xffffffffu); return; }   // counters: single-level only
    const CountRays rays{wf.ray_o[q], wf.ray_d[q], wf.path[q], wf.hit};
    if (sc.has_non_opaque)
        k_extend_count<true><<<lc.grid_persistent, lc.block_trace, 0, st>>>(sc, rays, wf.counters, wf.stats, seg,
                                                                            lc.postpone_sp, lc.refill_min);
    else
        k_extend_count<false><<<lc.grid_persistent, lc.block_trace, 0, st>>>(sc, rays, wf.counters, wf.stats, seg,
                                                                             lc.postpone_sp, lc.refill_min);
}
void launch_shade(const LaunchCfg& lc, cudaStream_t st, const DevScene& sc, const DevView* views,
                  const Wavefront& wf, int q, uint32_t seg, float4* accum, uint32_t paths, bool cache) {
    const uint32_t block = paths <= kSmallBlockPaths ? 128u : (uint32_t)lc.block_shade;
    const uint32_t grid = min((uint32_t)lc.grid_shade, (uint32_t)(((uint64_t)paths + block - 1) / block));
    if (cache || !sc.dir_lights_only) k_shade<true><<<grid, block, 0, st>>>(sc, views, wf, q, seg, accum);
    else k_shade<false><<<grid, block, 0, st>>>(sc, views, wf, q, seg, accum);
}
void launch_resolve(cudaStream_t st, const float4* accum, uint32_t width, uint32_t height, float inv_spp,
                    float4* out, uint32_t pitch_px) {
    dim3 grid((width + 255) / 256, height);
    k_resolve<<<grid, 256, 0, st>>>(accum, width, height, inv_spp, out, pitch_px);
}
void launch_resolve_fixed(cudaStream_t st, const unsigned long long* fx, uint32_t width, uint32_t height,
                          float inv_spp, float4* out, uint32_t pitch_px) {
    dim3 grid((width + 255) / 256, height);
    k_resolve_fixed<<<grid, 256, 0, st>>>(fx, width, height, inv_spp, out, pitch_px);
}
void launch_fold_fixed(cudaStream_t st, const unsigned long long* fx, float4* accum, uint32_t n) {
    if (n == 0) return;
    k_fold_fixed<<<(unsigned)(((uint64_t)n + 255) / 256), 256, 0, st>>>(fx, accum, n);
}
// Which kernel traces a call's rays: eight lanes per ray up to `group` rays, then a ray per thread up to `thread`, then
// lanes that take new rays.  Closest (c) and any (a) hits of incoherent rays and of a camera's, us, in the three ways:
//  * one level: c in 1.48 M triangles 71 / 78 / 87 at 30,000 rays, 86 / 83 / 90 at 40,000, camera 68 / 74 / 80; a in the
//    room 45 / 35 / 40 at 40,000.  A ray per thread while the GPU holds all of them (155,648: c - / 138 / 149, a - / 60 /
//    66), and twice as many where materials are not opaque and the third loop is longest (300,007: - / 186 / 184, camera
//    160 / 230);
//  * two levels: c in 1,000 instances 188 / 195 / 170 at 60,000, camera 196 / 289 / 233.  Rays of few instances are short:
//    a in eight 21 / 23 / 25 at 20,000, 33 / 19 / 23 at 40,000; 52 / 59 and camera 32 / 39 at 300,007 (second and third),
//    140 / 118 and 74 / 82 at 1,000,003; c in eight 32 / 27 / 29 at 30,000, in 32 75 / 46 / 44 at 80,000.  Any hits are
//    between: in 300 instances 61 / 52 / 60 and camera 39 / 67 / 60 at 40,000, 73 / 52 / 51 and 47 / 66 / 57 at 60,000; in
//    1,000 93 / 76 / 78 and 76 / 122 / 110.
struct StageLimits { uint32_t group, thread; };
static StageLimits stage_limits(const LaunchCfg& lc, bool two, bool op, bool any, uint32_t instances) {
    if (!two) return {40000u, (uint32_t)lc.grid_stage * 128u * (op ? 2u : 1u)};
    if (instances < 64u) return any ? StageLimits{25000u, 400000u} : StageLimits{32000u, 100000u};
    if (instances < 500u && any) return {40000u, 100000u};
    return {60000u, 0u};
}
// Views of at most this many pixels take that way too, their hit records waiting in one of the outputs for
// k_primary_rec: 35 / 58 us against 37 / 113 us in k_primary at 128x128 (room / 1.48 M triangles); at 230x170
// 48 / 86 against 41 / 111. Not for a pixel or two (a pick), where the second launch shows: 14.6 us against 12.5.
constexpr uint32_t kGroupPixels = 24576, kMinGroupPixels = 4;

template <bool kOpacity, int kOut>
static void launch_stage_kernel(const LaunchCfg& lc, cudaStream_t st, const DevScene& sc, StageArgs& a) {
    const bool two = sc.insts != nullptr;
    const StageLimits lim = stage_limits(lc, two, kOpacity, kOut == kStageOccluded, sc.num_instances);
    if (kOut == kStageRec || a.n <= lim.group) {
        const uint32_t all = (a.n + 128u / kGroupLanes - 1u) / (128u / kGroupLanes), full = two ? lc.grid_group2 : lc.grid_group;
        if (all <= full) a.work = nullptr;
        const uint32_t grid = a.work ? full : all;
        if constexpr (kOut != kStageRec) {
            if (two) {
                k_stage2_group<kOpacity, kOut><<<grid, kGroupBlock, 0, st>>>(sc.nodes, sc.insts, sc.mat_tr, a);
                return;
            }
        }
        k_stage_group<kOpacity, kOut><<<grid, kGroupBlock, 0, st>>>(sc.nodes, sc.tris, a);
        return;
    }
    if constexpr (kOut != kStageRec) {
        const uint32_t all = (uint32_t)(((uint64_t)a.n + 127u) / 128u);
        if (a.n <= lim.thread || !a.work || a.n > kMaxTraceRays) {   // (a counter is for as many rays as it can count)
            if (two) k_stage_ray<kOut, true><<<all, 128, 0, st>>>(sc.nodes, sc.tris, sc.insts, sc.mat_tr, a);
            else k_stage_ray<kOut, false><<<all, 128, 0, st>>>(sc.nodes, sc.tris, sc.insts, sc.mat_tr, a);
            return;
        }
        const uint32_t grid = min((uint32_t)(two ? lc.grid_stage2 : lc.grid_stage), all);
        if (two) k_stage2<kOpacity, stage2_out(kOpacity, kOut)><<<grid, 128, 0, st>>>(sc.nodes, sc.insts, sc.mat_tr, a);
        else k_stage<kOpacity, kOut><<<grid, 128, 0, st>>>(sc.nodes, sc.tris, a);
    }
}
template <int kOut>
static void launch_stage(const LaunchCfg& lc, cudaStream_t st, const DevScene& sc, StageArgs& a) {
    a.tris = sc.tris;
    a.insts = sc.insts;
    a.near = sc.ray_offset * 1562.5f;   // a 32nd of the scene's extent
    a.postpone_sp = 16;
    a.refill_min = 8;
    if (sc.has_non_opaque) launch_stage_kernel<true, kOut>(lc, st, sc, a);
    else launch_stage_kernel<false, kOut>(lc, st, sc, a);
}
void launch_trace_closest(const LaunchCfg& lc, cudaStream_t st, const DevScene& sc, const float4* rays, uint32_t n,
                          uint4* hits, uint32_t* work) {
    if (n == 0) return;
    StageArgs a{};
    a.rays = rays;
    a.hits = hits;
    a.n = n;
    a.work = work;
    launch_stage<kStageHits>(lc, st, sc, a);
}
void launch_trace_any(const LaunchCfg& lc, cudaStream_t st, const DevScene& sc, const float4* rays, uint32_t n,
                      uint8_t* occluded, uint32_t* work) {
    if (n == 0) return;
    StageArgs a{};
    a.rays = rays;
    a.occluded = occluded;
    a.n = n;
    a.work = work;
    launch_stage<kStageOccluded>(lc, st, sc, a);
}
void launch_primary(const LaunchCfg& lc, cudaStream_t st, const DevScene& sc, const DevView& v, float near_z,
                    float far_z, float* depth, float4* const gb[4], float4* hitpos, uint32_t* work) {
    const uint32_t n = v.width * v.height;
    if (n == 0) return;
    const PrimaryOut out{depth, {gb[0], gb[1], gb[2], gb[3]}, hitpos, near_z, far_z};
    float4* rec = hitpos ? hitpos : gb[0] ? gb[0] : gb[1] ? gb[1] : gb[2] ? gb[2] : gb[3];
    if (rec && !sc.insts && n >= kMinGroupPixels && n <= kGroupPixels) {
        StageArgs a{};
        a.rec = rec;
        a.n = n;
        a.work = work;
        a.view = v;
        launch_stage<kStageRec>(lc, st, sc, a);
        k_primary_rec<<<(n + 127) / 128, 128, 0, st>>>(sc, v, out, rec);
        return;
    }
    const uint32_t blocks = ((v.width + 15u) / 16u) * ((v.height + 7u) / 8u);
    if (sc.insts) k_primary<true><<<blocks, 128, 0, st>>>(sc, v, out);
    else k_primary<false><<<blocks, 128, 0, st>>>(sc, v, out);
}
void launch_trace_count(cudaStream_t st, const DevScene& sc, const float4* rays, uint32_t n, uint2* counts) {
    if (n == 0) return;
    k_trace_count<<<(n + 127) / 128, 128, 0, st>>>(sc, rays, n, counts);
}

// Occupancy-derived grid of the persistent kernels: every SM filled.
void query_launch_cfg(int device, int block_trace, LaunchCfg* lc) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    int per_sm = 0, per_sm_shade = 0;
    if (lc->regcap)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace<4, true>, block_trace, 0);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace<1, true>, block_trace, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_shade, k_shade<true>, 512, 0);
    int per_sm2 = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm2, k_trace2<true>, block_trace, 0);
    if (per_sm2 < 1) per_sm2 = 1;
    lc->grid_persistent2 = sms * per_sm2;
    if (per_sm < 1) per_sm = 1;
    if (per_sm_shade < 1) per_sm_shade = 1;
    lc->block_trace = block_trace;
    int per_sm_stage = 0, per_sm_stage2 = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_stage, k_stage<true, kStageHits>, 128, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_stage2, k_stage2<true, kStageEither>, 128, 0);
    lc->grid_stage = sms * (per_sm_stage < 1 ? 1 : per_sm_stage);
    lc->grid_stage2 = sms * (per_sm_stage2 < 1 ? 1 : per_sm_stage2);
    int per_sm_group = 0, per_sm_group2 = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_group2, k_trace2_group<true>, kGroupBlock, 0);
    lc->grid_group2 = sms * (per_sm_group2 < 1 ? 1 : per_sm_group2);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_group, k_trace_group<true>, kGroupBlock, 0);
    lc->grid_group = sms * (per_sm_group < 1 ? 1 : per_sm_group);
    lc->grid_persistent = sms * per_sm;
    lc->block_shade = 512;   // the direction grouping of the next rays spans a block
    lc->grid_shade = sms * per_sm_shade * 4;
}

}  // namespace bsm
