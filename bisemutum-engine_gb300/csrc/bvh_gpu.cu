// bvh_gpu.cu — device build of the compressed 8-wide BVH (sm_103a).
//
// Replaces the driver-side BLAS build the reference requests through
// AccelerationStructure and runs on the GPU (bisemutum/src/graphics/accel.cpp:77-87,
// recorded by GraphicsManager::execute_immediately, graphics_manager.cpp:475-478).
// The tree is defined as in the host builder (bvh_build.cpp): a binary BVH by
// binned SAH over triangle centroids (Wald 2007), collapsed into 8-wide nodes by
// the SAH-optimal dynamic programme of Ylitie, Karras and Laine (HPG 2017) or by
// opening the largest child, children placed in octant slots, child boxes
// quantised outward to 8 bits per plane (bvh_quant.h).  Four phases:
//   1. triangle boxes and the scene's box and centroid bounds, one thread per
//      triangle;
//   2. the binary BVH top-down, one breadth-first level per round while a node
//      holds more than kSmall triangles. Per level every CTA bins chunks of a
//      node's triangle references into 3 x 32 centroid bins in shared memory and
//      merges them into the node's bins with one atomic per bin value; one warp
//      per node picks the split of least SAH cost; a stable partition writes the
//      children's references (warp ballots, chunk offsets from the chunks' own
//      bin counts); the children become leaves, small nodes or next-level nodes.
//      The host queues the levels in batches and looks only then. Nodes of at
//      most kSmall triangles are finished by one warp each in shared memory, from
//      32 triangles on with a triangle per lane;
//   3. the collapse's dynamic programme bottom-up: a thread per binary leaf
//      climbs towards the root and stops at every node whose other child is not
//      done yet (the second thread to arrive computes the node; Karras 2012);
//   4. the 8-wide nodes top-down, one level per round, eight lanes per node: each
//      node gathers its up to eight children, assigns octant slots and quantises
//      their boxes; a scan over the level gives each node its first child and
//      first triangle, and a second pass writes the leaf triangles and the next
//      level's queue, so nodes and triangles come out in breadth-first order as
//      on the host.
// Split decisions use exact bin counts and boxes (order-independent atomics on
// ordered float keys), and every partition is stable, so the tree does not
// depend on the order in which CTAs run.
#include "bvh_gpu.h"

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "bvh_quant_lanes.cuh"

namespace bsm {
namespace {

constexpr uint32_t kNone = 0xffffffffu;
constexpr int kBins = 32;                  // lanes of a warp: one bin per lane
constexpr uint32_t kChunk = 4096;          // references per CTA in a level pass, at most
// Chunks of a build of T triangles: large ones cost fewer merges, small ones fill the GPU in the top levels, where a
// level has few nodes (builds of 20,504 / 250,050 / 1,482,242 / 4,973,058 triangles take 1.23 / 2.24 / 4.95 / 14.1 ms
// with 4,096 per chunk, 1.14 / 2.10 / 4.90 / 14.3 with 2,048 and 1.10 / 1.97 / 4.98 / 14.7 with 1,024).
uint32_t chunk_size(uint32_t T) { return T < 600000u ? 1024u : T < 3000000u ? 2048u : kChunk; }
constexpr uint32_t kSmall = 128;           // nodes of at most this many triangles are finished by one warp
constexpr int kSmallWarps = 4;             // warps per CTA of the small-node kernel
constexpr uint32_t kLevelThreads = 256;
constexpr uint8_t kDecLeaf = 0xff, kDecInner = 0xfe, kDecSame = 0xfd;
constexpr uint32_t kKeyLo = 0xffffffffu;   // initial key of a minimum
constexpr uint32_t kKeyHi = 0u;            // initial key of a maximum

// error bits of Counters::error
enum : uint32_t {
    kErrIndex = 1, kErrFinite = 2, kErrNodes = 4, kErrGather = 8, kErrLeaf = 16, kErrStack = 32, kErrClimb = 64,
    kErrWide = 128, kErrPartition = 256
};

struct BNode {                 // binary node
    float lo[3];
    uint32_t left;             // kNone: a leaf
    float hi[3];
    uint32_t right;
    uint32_t first, count;     // reference range (all nodes)
    uint32_t parent, pad;
};
static_assert(sizeof(BNode) == 48, "BNode must be 48 bytes");

struct Task {                  // a node still to split: its reference range and centroid bounds
    uint32_t node, begin, end;
    uint32_t aux;              // in a level: its first chunk; in the small list: the reference buffer (0 or 1)
    float clo[3], chi[3];
};
struct Bin { uint32_t cnt, lo[3], hi[3]; };      // box as ordered float keys
struct Split { int axis; int bin; uint32_t leaf; uint32_t nl; };
struct ChunkBins { uint16_t below[3][kBins]; };   // a chunk's references in the bins below each, per axis
struct ChildAcc { uint32_t box[2][6]; uint32_t cen[2][6]; };   // per side: lo xyz, hi xyz (keys)
struct WideLevel { uint32_t nodes, node_base, tri_base, pad; };   // a level's 8-wide nodes, its first node and triangle
struct Counters { uint32_t nodes, tasks[2], chunks[2], small_tasks, error, depth; WideLevel wide[2]; uint32_t wide_blocks, pad[3]; };
struct WideRec { uint32_t child[8]; };     // binary node per slot (kNone: empty slot)

// Order-preserving map of floats to unsigned keys (-0 below +0), so that
// unsigned atomicMin/atomicMax compute float minima and maxima exactly.
__device__ __forceinline__ uint32_t fkey(float f) {
    uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float funkey(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

__device__ __forceinline__ float area6(const float* lo, const float* hi) {
    float dx = fmaxf(0.0f, hi[0] - lo[0]), dy = fmaxf(0.0f, hi[1] - lo[1]), dz = fmaxf(0.0f, hi[2] - lo[2]);
    return 2.0f * (dx * dy + dy * dz + dz * dx);
}

__device__ __forceinline__ int bin_of(float c, float lo, float scale, int B) {
    int b = (int)((c - lo) * scale);
    return min(max(b, 0), B - 1);
}

__device__ __forceinline__ float axis_scale(const Task& t, int a, int B) {
    float ext = t.chi[a] - t.clo[a];
    return ext > 0.0f ? (float)B / ext : 0.0f;
}

__device__ __forceinline__ float centroid(const float4& l, const float4& h, int a) {
    return a == 0 ? 0.5f * (l.x + h.x) : (a == 1 ? 0.5f * (l.y + h.y) : 0.5f * (l.z + h.z));
}

__device__ __forceinline__ float warp_min(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// ------------------------------------------------------------ phase 1 ----
__global__ void __launch_bounds__(256) k_tri_boxes(const float* __restrict__ pos, uint32_t nv,
                                                   const uint32_t* __restrict__ idx, uint32_t nt,
                                                   float4* __restrict__ box, uint32_t* __restrict__ refs,
                                                   uint32_t* __restrict__ gkeys, Counters* cnt) {
    __shared__ float s_red[8][12];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    float v[12];   // box lo, box hi, centroid lo, centroid hi
    for (int k = 0; k < 3; ++k) { v[k] = v[6 + k] = INFINITY; v[3 + k] = v[9 + k] = -INFINITY; }
    if (t < nt) {
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (int c = 0; c < 3; ++c) {
            uint32_t vi = idx ? idx[3 * (size_t)t + c] : 3 * t + c;
            if (vi >= nv) { atomicOr(&cnt->error, kErrIndex); vi = 0; }
            for (int k = 0; k < 3; ++k) {
                float p = pos[3 * (size_t)vi + k];
                if (!isfinite(p)) atomicOr(&cnt->error, kErrFinite);
                lo[k] = fminf(lo[k], p);
                hi[k] = fmaxf(hi[k], p);
            }
        }
        box[2 * (size_t)t] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        box[2 * (size_t)t + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
        refs[t] = t;
        for (int k = 0; k < 3; ++k) {
            float c = 0.5f * (lo[k] + hi[k]);
            v[k] = lo[k]; v[3 + k] = hi[k]; v[6 + k] = c; v[9 + k] = c;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < 12; ++k) {
        bool mx = (k % 6) >= 3;
        v[k] = mx ? warp_max(v[k]) : warp_min(v[k]);
        if (lane == 0) s_red[warp][k] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        const int k = threadIdx.x;
        bool mx = (k % 6) >= 3;
        float r = s_red[0][k];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) r = mx ? fmaxf(r, s_red[w][k]) : fminf(r, s_red[w][k]);
        if (mx) atomicMax(&gkeys[k], fkey(r)); else atomicMin(&gkeys[k], fkey(r));
    }
}

// ------------------------------------------------------------ phase 2 ----
// The passes of a level run on what the level before left on the device (its
// tasks and their number), so the host queues the levels without waiting.  A
// block takes chunks of at most kChunk references of one task in turn.
__global__ void k_bins_init(Bin* bins, uint32_t n, ChildAcc* acc, uint32_t nacc) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        Bin b;
        b.cnt = 0;
        for (int k = 0; k < 3; ++k) { b.lo[k] = kKeyLo; b.hi[k] = kKeyHi; }
        bins[i] = b;
    }
    if (i < nacc) {
        ChildAcc a;
        for (int s = 0; s < 2; ++s)
            for (int k = 0; k < 3; ++k) {
                a.box[s][k] = kKeyLo; a.box[s][3 + k] = kKeyHi;
                a.cen[s][k] = kKeyLo; a.cen[s][3 + k] = kKeyHi;
            }
        acc[i] = a;
    }
}

// Adds a warp's references to one axis' shared bins.  Neighbouring references
// mostly share a bin (they are in input order within a node), and 32 atomics on
// one address take turns, so up to three groups of eight or more lanes with a
// common bin are reduced in registers first (builds of 1.48 M / 4.97 M triangles:
// one group 4.78 / 13.56 ms, two 4.69 / 13.26, three 4.70 / 13.36, six 4.73 / 13.46;
// three groups of at least 2 / 4 / 8 lanes 4.73 / 13.57, 4.70 / 13.36, 4.68 / 13.21).
__device__ __forceinline__ void bin_axis(Bin* sb, bool act, uint32_t bin, const uint32_t* kl, const uint32_t* kh) {
    uint32_t rest = __ballot_sync(0xffffffffu, act);
    for (int round = 0; round < 3 && rest != 0u; ++round) {
        const int leader = __ffs(rest) - 1;
        const uint32_t lb = __shfl_sync(0xffffffffu, bin, leader);
        const uint32_t m = __ballot_sync(0xffffffffu, bin == lb) & rest;
        if (__popc(m) < 8) break;
        if ((m >> (threadIdx.x & 31u)) & 1u) {
            uint32_t lo[3], hi[3];
            for (int k = 0; k < 3; ++k) { lo[k] = __reduce_min_sync(m, kl[k]); hi[k] = __reduce_max_sync(m, kh[k]); }
            if ((int)(threadIdx.x & 31u) == leader) {
                Bin& b = sb[lb];
                atomicAdd(&b.cnt, (uint32_t)__popc(m));
                for (int k = 0; k < 3; ++k) { atomicMin(&b.lo[k], lo[k]); atomicMax(&b.hi[k], hi[k]); }
            }
        }
        rest &= ~m;
    }
    if ((rest >> (threadIdx.x & 31u)) & 1u) {
        Bin& b = sb[bin];
        atomicAdd(&b.cnt, 1u);
        for (int k = 0; k < 3; ++k) { atomicMin(&b.lo[k], kl[k]); atomicMax(&b.hi[k], kh[k]); }
    }
}

// Bins a chunk's references by centroid, per axis, into shared bins, merges the
// non-empty bins into the task's and leaves the chunk's running counts for the
// partition.
__global__ void __launch_bounds__(kLevelThreads) k_bin(const uint32_t* __restrict__ chunk_task,
                                                       const Task* __restrict__ tasks,
                                                       const uint32_t* __restrict__ refs,
                                                       const float4* __restrict__ box, Bin* __restrict__ gbins,
                                                       ChunkBins* __restrict__ cbins, const Counters* cnt, int cur, uint32_t chunk, int B) {
    __shared__ Bin sb[3 * kBins];
    const uint32_t nch = cnt->error ? 0u : cnt->chunks[cur];
    for (uint32_t c = blockIdx.x; c < nch; c += gridDim.x) {
        for (int i = threadIdx.x; i < 3 * kBins; i += blockDim.x) {
            sb[i].cnt = 0;
            for (int k = 0; k < 3; ++k) { sb[i].lo[k] = kKeyLo; sb[i].hi[k] = kKeyHi; }
        }
        __syncthreads();
        const uint32_t ti = chunk_task[c];
        const Task tk = tasks[ti];
        const uint32_t begin = tk.begin + (c - tk.aux) * chunk, end = min(tk.end, begin + chunk);
        float sc[3];
        for (int a = 0; a < 3; ++a) sc[a] = axis_scale(tk, a, B);
        uint32_t i = begin + threadIdx.x;
        float4 nl = make_float4(0, 0, 0, 0), nh = nl;
        auto fetch = [&]() {
            if (i >= end) return;
            const uint32_t r = refs[i];
            nl = box[2 * (size_t)r];
            nh = box[2 * (size_t)r + 1];
        };
        fetch();
        for (uint32_t base = begin; base < end; base += kLevelThreads) {
            const bool act = i < end;
            const float4 l = nl, h = nh;
            i += kLevelThreads;
            fetch();   // the next references' boxes, while these are binned (42 -> 39 us a level)
            const uint32_t kl[3] = {fkey(l.x), fkey(l.y), fkey(l.z)}, kh[3] = {fkey(h.x), fkey(h.y), fkey(h.z)};
            for (int a = 0; a < 3; ++a) {
                if (!(sc[a] > 0.0f)) continue;   // the same for the whole block
                bin_axis(sb + a * kBins, act, act ? (uint32_t)bin_of(centroid(l, h, a), tk.clo[a], sc[a], B) : 255u, kl, kh);
            }
        }
        __syncthreads();
        Bin* g = gbins + (size_t)ti * 3 * kBins;
        for (int i = threadIdx.x; i < 3 * kBins; i += blockDim.x) {
            const uint32_t n = sb[i].cnt;
            uint32_t x = n;   // a warp holds one axis' bins
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if ((threadIdx.x & 31u) >= o) x += y;
            }
            cbins[c].below[i / kBins][i % kBins] = (uint16_t)(x - n);
            if (n == 0) continue;
            atomicAdd(&g[i].cnt, n);
            for (int k = 0; k < 3; ++k) { atomicMin(&g[i].lo[k], sb[i].lo[k]); atomicMax(&g[i].hi[k], sb[i].hi[k]); }
        }
        __syncthreads();
    }
}
static_assert(kBins == 32 && kChunk < 65536, "a warp scans an axis' bins; a chunk's counts fit 16 bits");

// The least-cost split over three axes of binned SAH (bvh_build.cpp Builder::build):
// cost(split before bin b) = area(left) * n_left + area(right) * n_right, axes
// in order and bins ascending, the first minimum kept.  One warp; lane = bin.
// `bins(a)` returns this lane's bin of axis a.  Returns the axis (-1: none); the
// boxes of the two sides are left in lane *best_bin.
template <class GetBin>
__device__ int warp_best_split(const Task& tk, int B, GetBin bins, int* best_bin, uint32_t* best_nl, float* best_cost,
                               float side[2][6]) {
    const int lane = threadIdx.x & 31;
    float best = INFINITY;
    int bax = -1, bbin = 0;
    uint32_t bnl = 0;
    for (int a = 0; a < 3; ++a) {
        if (!(tk.chi[a] - tk.clo[a] > 0.0f)) continue;
        Bin b = bins(a);
        uint32_t n = lane < B ? b.cnt : 0u;
        float lo[3], hi[3];
        for (int k = 0; k < 3; ++k) {
            lo[k] = n ? funkey(b.lo[k]) : INFINITY;
            hi[k] = n ? funkey(b.hi[k]) : -INFINITY;
        }
        // inclusive prefix (bins 0..lane) and suffix (bins lane..31)
        uint32_t ln = n, rn = n;
        float llo[3], lhi[3], rlo[3], rhi[3];
        for (int k = 0; k < 3; ++k) { llo[k] = rlo[k] = lo[k]; lhi[k] = rhi[k] = hi[k]; }
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t un = __shfl_up_sync(0xffffffffu, ln, off), dn = __shfl_down_sync(0xffffffffu, rn, off);
            float ul[3], uh[3], dl[3], dh[3];
            for (int k = 0; k < 3; ++k) {
                ul[k] = __shfl_up_sync(0xffffffffu, llo[k], off);
                uh[k] = __shfl_up_sync(0xffffffffu, lhi[k], off);
                dl[k] = __shfl_down_sync(0xffffffffu, rlo[k], off);
                dh[k] = __shfl_down_sync(0xffffffffu, rhi[k], off);
            }
            if (lane >= off) {
                ln += un;
                for (int k = 0; k < 3; ++k) { llo[k] = fminf(llo[k], ul[k]); lhi[k] = fmaxf(lhi[k], uh[k]); }
            }
            if (lane + off < 32) {
                rn += dn;
                for (int k = 0; k < 3; ++k) { rlo[k] = fminf(rlo[k], dl[k]); rhi[k] = fmaxf(rhi[k], dh[k]); }
            }
        }
        // split before bin `lane`: left = prefix of lane - 1, right = suffix of lane
        uint32_t pn = __shfl_up_sync(0xffffffffu, ln, 1);
        float pl[3], ph[3];
        for (int k = 0; k < 3; ++k) {
            pl[k] = __shfl_up_sync(0xffffffffu, llo[k], 1);
            ph[k] = __shfl_up_sync(0xffffffffu, lhi[k], 1);
        }
        float cost = INFINITY;
        if (lane >= 1 && lane < B && pn > 0 && rn > 0) cost = area6(pl, ph) * (float)pn + area6(rlo, rhi) * (float)rn;
        float m = cost;
        int ml = lane;
        for (int o = 16; o > 0; o >>= 1) {
            float om = __shfl_xor_sync(0xffffffffu, m, o);
            int ol = __shfl_xor_sync(0xffffffffu, ml, o);
            if (om < m || (om == m && ol < ml)) { m = om; ml = ol; }
        }
        uint32_t nl_at = __shfl_sync(0xffffffffu, pn, ml);
        if (m < best) {
            best = m; bax = a; bbin = ml; bnl = nl_at;
            for (int k = 0; k < 3; ++k) { side[0][k] = pl[k]; side[0][3 + k] = ph[k]; side[1][k] = rlo[k]; side[1][3 + k] = rhi[k]; }
        }
    }
    *best_bin = bbin;
    *best_nl = bnl;
    *best_cost = best;
    return bax;
}

// Split or leaf of a node of `cnt` triangles and box area `parent_area`, as bvh_build.cpp decides.
__device__ __forceinline__ Split decide(int bax, int bbin, uint32_t bnl, float best, uint32_t cnt, float parent_area,
                                        uint32_t max_leaf) {
    Split s;
    s.leaf = 0;
    s.axis = bax;
    s.bin = bbin;
    s.nl = bnl;
    float split_cost = parent_area > 0.0f ? 1.0f + best / parent_area : INFINITY;
    if (bax < 0) {
        if (cnt <= max_leaf) s.leaf = 1;
        else s.nl = cnt / 2;   // every centroid in one place: split by index
    } else if (cnt <= max_leaf && (float)cnt <= split_cost) {
        s.leaf = 1;
    }
    if (s.leaf) s.nl = cnt;
    return s;
}

// The split of every task (a warp each, its bins cleared for the next level) and
// where its chunks' left references go.
__global__ void k_split(const Task* __restrict__ tasks, Bin* __restrict__ gbins, const ChunkBins* __restrict__ cbins,
                        const BNode* __restrict__ nodes, Split* __restrict__ splits, uint32_t* __restrict__ left_base,
                        ChildAcc* __restrict__ acc, Counters* cnt, int cur, uint32_t chunk, int B, uint32_t max_leaf) {
    const int lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt->tasks[cur ^ 1] = cnt->chunks[cur ^ 1] = 0u;   // the last level's
    // other warps may set the error word while this one starts: its lanes have to agree on what they read
    const uint32_t nt = __shfl_sync(0xffffffffu, cnt->error ? 0u : cnt->tasks[cur], 0), warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nt; w += warps) {
        const Task tk = tasks[w];
        int bbin;
        uint32_t bnl;
        float best, side[2][6];
        int bax = warp_best_split(tk, B, [&](int a) {
            Bin e;
            e.cnt = 0;
            return lane < B ? gbins[((size_t)w * 3 + a) * kBins + lane] : e;
        }, &bbin, &bnl, &best, side);
        if (bax >= 0 && lane == bbin)
            for (int c = 0; c < 2; ++c)
                for (int k = 0; k < 6; ++k) acc[w].box[c][k] = fkey(side[c][k]);
        Bin z;
        z.cnt = 0;
        for (int k = 0; k < 3; ++k) { z.lo[k] = kKeyLo; z.hi[k] = kKeyHi; }
        for (int a = 0; a < 3; ++a) gbins[((size_t)w * 3 + a) * kBins + lane] = z;
        const BNode nd = nodes[tk.node];
        const Split s = decide(bax, bbin, bnl, best, tk.end - tk.begin, area6(nd.lo, nd.hi), max_leaf);
        if (lane == 0) splits[w] = s;
        const uint32_t n = (tk.end - tk.begin + chunk - 1u) / chunk;
        uint32_t carry = 0;
        for (uint32_t base = 0; base < n; base += 32) {
            const uint32_t c = base + lane;
            uint32_t left = 0;
            if (c < n) {
                const uint32_t size = min(chunk, tk.end - tk.begin - c * chunk);
                if (s.leaf) left = size;
                else if (s.axis < 0) left = s.nl > c * chunk ? min(size, s.nl - c * chunk) : 0u;
                else left = cbins[tk.aux + c].below[s.axis][s.bin];
            }
            uint32_t x = left;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (c < n) left_base[tk.aux + c] = tk.begin + carry + x - left;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0 && carry != s.nl) atomicOr(&cnt->error, kErrPartition);
    }
}

__device__ __forceinline__ bool goes_left(const Task& tk, const Split& sp, uint32_t i, const float4& l,
                                          const float4& h, int B) {
    if (sp.leaf) return true;
    if (sp.axis < 0) return i - tk.begin < sp.nl;
    const int a = sp.axis;
    return bin_of(centroid(l, h, a), tk.clo[a], axis_scale(tk, a, B), B) < sp.bin;
}

// Adds the boxes of the lanes `m` (`in`: this lane is one of them) to a shared box of keys, for splits by index. With six
// atomics per reference on the task's own box, 1,500,000 triangles through one point took 26.6 ms to build; 4.4 ms so.
__device__ __forceinline__ void add_boxes(uint32_t* s_box, bool in, uint32_t m, const float4& l, const float4& h) {
    if (!in) return;
    const bool first = (threadIdx.x & 31u) == (uint32_t)__ffs(m) - 1u;
    for (int k = 0; k < 3; ++k) {
        const uint32_t lo = __reduce_min_sync(m, fkey(k == 0 ? l.x : k == 1 ? l.y : l.z));
        const uint32_t hi = __reduce_max_sync(m, fkey(k == 0 ? h.x : k == 1 ? h.y : h.z));
        if (first) { atomicMin(s_box + k, lo); atomicMax(s_box + 3 + k, hi); }
    }
}

// Stable partition of a chunk: its left references from left_base on, its right
// ones behind the task's left part (both in chunk order); the children's
// centroid bounds are reduced over the block and merged into the task's.  Their
// boxes are already there, from the split's bins, unless the task was split by
// index.  Bound by the latency of reference, box and barrier in turn: the next
// box is fetched over the one barrier of a round, and without the boxes'
// minima the kernel fits five blocks an SM (51 registers; 70 before, 1.6 waves
// of the 724 chunks of 1.48 M triangles).  37 -> 17 us a level there, 0.53 ->
// 0.31 ms over the build; with four blocks an SM the build takes 4.75 ms
// against 4.70.
__global__ void __launch_bounds__(kLevelThreads, 5) k_partition(const uint32_t* __restrict__ chunk_task,
                                                             const Task* __restrict__ tasks,
                                                             const Split* __restrict__ splits,
                                                             const uint32_t* __restrict__ left_base,
                                                             const uint32_t* __restrict__ in,
                                                             uint32_t* __restrict__ out,
                                                             const float4* __restrict__ box,
                                                             ChildAcc* __restrict__ acc, const Counters* cnt, int cur, uint32_t chunk, int B) {
    constexpr int kWarps = kLevelThreads / 32;
    __shared__ uint32_t s_wl[2][kWarps], s_wr[2][kWarps];
    __shared__ float s_red[kWarps][12];
    __shared__ uint32_t s_box[12];   // split by index: the boxes of the two sides as keys
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t nch = cnt->error ? 0u : cnt->chunks[cur];   // after an error the offsets may be wrong
    for (uint32_t c = blockIdx.x; c < nch; c += gridDim.x) {
        const uint32_t ti = chunk_task[c];
        const Task tk = tasks[ti];
        const Split sp = splits[ti];
        const uint32_t begin = tk.begin + (c - tk.aux) * chunk, end = min(tk.end, begin + chunk);
        float v[12];   // centroid lo(3) hi(3) of the left side, then of the right
        for (int k = 0; k < 12; ++k) v[k] = (k % 6) < 3 ? INFINITY : -INFINITY;
        uint32_t lb = left_base[c], rb = tk.begin + sp.nl + (begin - lb);
        uint32_t r = 0, i = begin + threadIdx.x;
        float4 l = make_float4(0, 0, 0, 0), h = l;
        if (i < end) { r = in[i]; l = box[2 * (size_t)r]; h = box[2 * (size_t)r + 1]; }
        const bool by_index = sp.axis < 0;   // no bins (the same for the whole block)
        if (by_index) {
            if (threadIdx.x < 12) s_box[threadIdx.x] = threadIdx.x % 6 < 3 ? kKeyLo : kKeyHi;
            __syncthreads();
        }
        int par = 0;
        for (uint32_t base = begin; base < end; base += kLevelThreads, i += kLevelThreads, par ^= 1) {
            const bool act = i < end;
            const bool left = act && goes_left(tk, sp, i, l, h, B), right = act && !left;
            const uint32_t wl = __ballot_sync(0xffffffffu, left), wr = __ballot_sync(0xffffffffu, right);
            if (lane == 0) { s_wl[par][warp] = __popc(wl); s_wr[par][warp] = __popc(wr); }
            // the next references' boxes are on their way over the barrier (which also keeps this half of the
            // counts until every warp is past the reads below)
            const uint32_t r_now = r;
            const float4 l_now = l, h_now = h;
            if (i + kLevelThreads < end) { r = in[i + kLevelThreads]; l = box[2 * (size_t)r]; h = box[2 * (size_t)r + 1]; }
            if (by_index) {
                add_boxes(s_box, left, wl, l_now, h_now);
                add_boxes(s_box + 6, right, wr, l_now, h_now);
            }
            if (act) {
                for (int k = 0; k < 3; ++k) {
                    const float cc = centroid(l_now, h_now, k);
                    if (left) { v[k] = fminf(v[k], cc); v[3 + k] = fmaxf(v[3 + k], cc); }
                    else { v[6 + k] = fminf(v[6 + k], cc); v[9 + k] = fmaxf(v[9 + k], cc); }
                }
            }
            __syncthreads();
            uint32_t pl = 0, pr = 0, tl = 0, tr = 0;
            for (int w = 0; w < kWarps; ++w) {
                if (w < warp) { pl += s_wl[par][w]; pr += s_wr[par][w]; }
                tl += s_wl[par][w];
                tr += s_wr[par][w];
            }
            if (left) out[lb + pl + __popc(wl & lt)] = r_now;
            if (right) out[rb + pr + __popc(wr & lt)] = r_now;
            lb += tl;
            rb += tr;
        }
        for (int k = 0; k < 12; ++k) {
            const uint32_t key = fkey(v[k]);
            const uint32_t m = (k % 6) >= 3 ? __reduce_max_sync(0xffffffffu, key) : __reduce_min_sync(0xffffffffu, key);
            if (lane == 0) s_red[warp][k] = funkey(m);
        }
        __syncthreads();
        if (by_index && threadIdx.x < 12) {   // (an empty side's keys change nothing)
            uint32_t* dst = &acc[ti].box[threadIdx.x / 6][threadIdx.x % 6];
            if (threadIdx.x % 6 < 3) atomicMin(dst, s_box[threadIdx.x]); else atomicMax(dst, s_box[threadIdx.x]);
        }
        if (threadIdx.x < 12) {
            const int k = threadIdx.x;
            const bool mx = (k % 6) >= 3;
            float x = s_red[0][k];
            for (int w = 1; w < kWarps; ++w) x = mx ? fmaxf(x, s_red[w][k]) : fminf(x, s_red[w][k]);
            if (x != INFINITY && x != -INFINITY) {   // else that side is empty in this chunk
                uint32_t* dst = &acc[ti].cen[k / 6][k % 6];
                if (mx) atomicMax(dst, fkey(x)); else atomicMin(dst, fkey(x));
            }
        }
        __syncthreads();
    }
}

// Children of every split task: two binary nodes each; a child of one triangle
// is a leaf, a child of at most kSmall goes to the small list with the buffer
// that holds its references, any other to the next level, with its chunks.
// Chunks are handed out by a counter, in any order of tasks: nothing depends on
// it, and a scan over the tasks was a launch of its own (builds of 20 k / 1.48 M
// triangles 1.06 / 4.52 -> 1.035 / 4.46 ms without it).
__global__ void k_make_children(const Task* __restrict__ tasks, const Split* __restrict__ splits,
                                ChildAcc* __restrict__ acc, const uint32_t* __restrict__ refs,
                                BNode* __restrict__ nodes, uint32_t* __restrict__ final_refs, Task* __restrict__ next,
                                uint32_t next_cap, Task* __restrict__ small, uint32_t small_cap,
                                uint32_t* __restrict__ chunk_task, uint32_t chunk_cap, uint32_t chunk, Counters* cnt,
                                int cur, uint32_t max_nodes) {
    const uint32_t nt = cnt->error ? 0u : cnt->tasks[cur];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nt; i += gridDim.x * blockDim.x) {
        const Task tk = tasks[i];
        const Split sp = splits[i];
        if (sp.leaf) {   // cannot be: a task holds more than kSmall references
            atomicOr(&cnt->error, kErrLeaf);
            continue;
        }
        const uint32_t id = atomicAdd(&cnt->nodes, 2u);
        if (id + 2u > max_nodes) { atomicOr(&cnt->error, kErrNodes); continue; }
        nodes[tk.node].left = id;
        nodes[tk.node].right = id + 1u;
        const ChildAcc a = acc[i];
        ChildAcc z;
        for (int s = 0; s < 2; ++s) {
            for (int k = 0; k < 3; ++k) {
                z.box[s][k] = kKeyLo; z.box[s][3 + k] = kKeyHi;
                z.cen[s][k] = kKeyLo; z.cen[s][3 + k] = kKeyHi;
            }
            const uint32_t cb = s ? tk.begin + sp.nl : tk.begin, ce = s ? tk.end : tk.begin + sp.nl;
            BNode n;
            for (int k = 0; k < 3; ++k) { n.lo[k] = funkey(a.box[s][k]); n.hi[k] = funkey(a.box[s][3 + k]); }
            n.left = n.right = kNone;
            n.first = cb;
            n.count = ce - cb;
            n.parent = tk.node;
            n.pad = 0;
            nodes[id + s] = n;
            if (n.count <= 1u) {
                if (n.count == 1u) final_refs[cb] = refs[cb];
                continue;
            }
            Task c;
            c.node = id + s;
            c.begin = cb;
            c.end = ce;
            c.aux = (uint32_t)(cur ^ 1);
            for (int k = 0; k < 3; ++k) { c.clo[k] = funkey(a.cen[s][k]); c.chi[k] = funkey(a.cen[s][3 + k]); }
            if (n.count <= kSmall) {
                const uint32_t slot = atomicAdd(&cnt->small_tasks, 1u);
                if (slot < small_cap) small[slot] = c; else atomicOr(&cnt->error, kErrNodes);
            } else {
                const uint32_t slot = atomicAdd(&cnt->tasks[cur ^ 1], 1u);
                const uint32_t nc = (n.count + chunk - 1u) / chunk;
                c.aux = atomicAdd(&cnt->chunks[cur ^ 1], nc);
                if (slot < next_cap && c.aux + nc <= chunk_cap) {
                    next[slot] = c;
                    for (uint32_t k = 0; k < nc; ++k) chunk_task[c.aux + k] = slot;
                } else {
                    atomicOr(&cnt->error, kErrNodes);
                }
            }
        }
        acc[i] = z;   // for the next level's task
    }
}

// A new pair of binary nodes: the children of `node`, left then right.
__device__ __forceinline__ void write_child(BNode* nodes, uint32_t id, uint32_t parent, const float* lo, const float* hi,
                                            uint32_t first, uint32_t count) {
    uint4* p = reinterpret_cast<uint4*>(nodes + id);
    p[0] = make_uint4(__float_as_uint(lo[0]), __float_as_uint(lo[1]), __float_as_uint(lo[2]), kNone);
    p[1] = make_uint4(__float_as_uint(hi[0]), __float_as_uint(hi[1]), __float_as_uint(hi[2]), kNone);
    p[2] = make_uint4(first, count, parent, 0u);
}

// A small node's working set in shared memory: its references and their boxes.
struct SmallSet {
    uint32_t ref[kSmall];
    float lo[3][kSmall], hi[3][kSmall];
};

// Finishes a range of at most 32 references, one per lane, all of its nodes of
// a level together.  The split of least cost of every node is found without
// bins: a split between two bins is named by the first reference behind it, so
// every lane sums up the boxes left and right of its own bin over its node's
// references (broadcast by shuffles), for the three axes at once.  The counts,
// boxes and costs are those of the bins, and the least cost of the first axis
// and then the lowest bin is taken as k_split takes it.  Bound by the issue of
// minima and maxima (half rate), not by warps in flight: centroid bounds and
// the least cost come from scans over a node's lanes (log2 of its size in steps)
// instead of loops over its references: 1.48 M / 4.97 M triangles in 4.51 / 12.7
// ms, with the loops 4.61 / 13.06.  Scans over lanes sorted by bin in place of
// the remaining loop gain 1 % more for twice the code and were left out.
__device__ __forceinline__ void finish_lanes(SmallSet& S, uint32_t base, uint32_t n, uint32_t root_first, uint32_t node,
                                             float area, BNode* __restrict__ nodes, Counters* cnt, int B,
                                             uint32_t max_leaf, uint32_t max_nodes) {
    constexpr uint32_t kFull = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    const bool in = lane < n;
    uint32_t ref = 0;
    float lo[3] = {0.0f, 0.0f, 0.0f}, hi[3] = {0.0f, 0.0f, 0.0f};
    if (in) {
        ref = S.ref[base + lane];
        for (int k = 0; k < 3; ++k) { lo[k] = S.lo[k][base + lane]; hi[k] = S.hi[k][base + lane]; }
    }
    // this lane's node: references [s0, s0 + sc) of the range
    uint32_t s0 = in ? 0u : lane, sc = in ? n : 1u;
    bool open = sc >= 2u;
    while (true) {
        const uint32_t most = __reduce_max_sync(kFull, open ? sc : 0u);
        if (most == 0u) break;
        float cen[3], cl[3], ch[3];
        for (int k = 0; k < 3; ++k) { cen[k] = 0.5f * (lo[k] + hi[k]); cl[k] = ch[k] = cen[k]; }
        const int last = (int)(s0 + sc - 1u);   // of this lane's node
        for (uint32_t o = 1; o < most; o <<= 1)
            for (int k = 0; k < 3; ++k) {
                const float l = __shfl_up_sync(kFull, cl[k], o), h = __shfl_up_sync(kFull, ch[k], o);
                if (lane >= s0 + o) { cl[k] = fminf(cl[k], l); ch[k] = fmaxf(ch[k], h); }
            }
        for (int k = 0; k < 3; ++k) { cl[k] = __shfl_sync(kFull, cl[k], last); ch[k] = __shfl_sync(kFull, ch[k], last); }
        uint32_t bins = 0;       // this lane's bin per axis, 8 bits each
        bool use[3];
        for (int k = 0; k < 3; ++k) {
            const float ext = ch[k] - cl[k];
            const float scale = ext > 0.0f ? (float)B / ext : 0.0f;
            use[k] = ext > 0.0f && scale > 0.0f;
            if (use[k]) bins |= (uint32_t)bin_of(cen[k], cl[k], scale, B) << (8 * k);
        }
        // boxes and count left of each axis' own bin, box from it on
        float L[3][6], R[3][6];
        uint32_t nl[3] = {0u, 0u, 0u};
        for (int a = 0; a < 3; ++a)
            for (int k = 0; k < 3; ++k) { L[a][k] = R[a][k] = INFINITY; L[a][3 + k] = R[a][3 + k] = -INFINITY; }
        for (uint32_t j = 0; j < most; ++j) {
            const uint32_t src = open && j < sc ? s0 + j : lane;   // a lane's own box once more changes nothing
            const uint32_t ob = __shfl_sync(kFull, bins, (int)src);
            float o[6];
            for (int k = 0; k < 3; ++k) {
                o[k] = __shfl_sync(kFull, lo[k], (int)src);
                o[3 + k] = __shfl_sync(kFull, hi[k], (int)src);
            }
            for (int a = 0; a < 3; ++a) {
                if (((ob >> (8 * a)) & 255u) < ((bins >> (8 * a)) & 255u)) {
                    nl[a]++;
                    for (int k = 0; k < 3; ++k) { L[a][k] = fminf(L[a][k], o[k]); L[a][3 + k] = fmaxf(L[a][3 + k], o[3 + k]); }
                } else {
                    for (int k = 0; k < 3; ++k) { R[a][k] = fminf(R[a][k], o[k]); R[a][3 + k] = fmaxf(R[a][3 + k], o[3 + k]); }
                }
            }
        }
        float best = INFINITY;
        uint32_t key = kNone;    // axis, then bin; and the lane it came from
        for (int a = 0; a < 3; ++a) {
            if (!use[a] || nl[a] == 0u) continue;
            const float c = area6(L[a], L[a] + 3) * (float)nl[a] + area6(R[a], R[a] + 3) * (float)(sc - nl[a]);
            if (c < best) { best = c; key = ((uint32_t)a << 16) | (((bins >> (8 * a)) & 255u) << 8) | lane; }
        }
        for (uint32_t o = 1; o < most; o <<= 1) {
            const float ob = __shfl_up_sync(kFull, best, o);
            const uint32_t ok = __shfl_up_sync(kFull, key, o);
            if (lane >= s0 + o && (ob < best || (ob == best && ok < key))) { best = ob; key = ok; }
        }
        best = __shfl_sync(kFull, best, last);
        key = __shfl_sync(kFull, key, last);
        const bool split_axis = key != kNone;
        const int axis = split_axis ? (int)(key >> 16) : -1;
        const Split sp = decide(axis, 0, 0u, best, sc, area, max_leaf);
        if (open && sp.leaf) open = false;
        // stable partition
        const bool left = open && (split_axis ? ((bins >> (8 * axis)) & 255u) < ((key >> 8) & 255u) : lane - s0 < sc / 2u);
        const uint32_t lmask = __ballot_sync(kFull, left);
        const uint32_t seg = sc >= 32u ? kFull : ((1u << sc) - 1u) << s0, below = seg & ((1u << lane) - 1u);
        const uint32_t nleft = (uint32_t)__popc(lmask & seg);
        // the children's boxes: the winning lane has both, unless the node was split by index
        const int win = split_axis ? (int)(key & 255u) : (int)lane;
        float bl[6], br[6];
        for (int k = 0; k < 6; ++k) {
            const float l = axis == 0 ? L[0][k] : axis == 1 ? L[1][k] : L[2][k];   // this lane's view of the axis
            const float r = axis == 0 ? R[0][k] : axis == 1 ? R[1][k] : R[2][k];
            bl[k] = __shfl_sync(kFull, l, win);   // the whole node agrees on the axis
            br[k] = __shfl_sync(kFull, r, win);
        }
        const bool by_index = open && !split_axis;
        if (__ballot_sync(kFull, by_index) != 0u) {
            if (by_index)
                for (int k = 0; k < 3; ++k) { bl[k] = br[k] = INFINITY; bl[3 + k] = br[3 + k] = -INFINITY; }
            for (uint32_t j = 0; j < most; ++j) {
                const uint32_t src = open && j < sc ? s0 + j : lane;
                const bool ol = (lmask >> src) & 1u;
                for (int k = 0; k < 3; ++k) {
                    const float l = __shfl_sync(kFull, lo[k], (int)src), h = __shfl_sync(kFull, hi[k], (int)src);
                    if (by_index && j < sc) {
                        if (ol) { bl[k] = fminf(bl[k], l); bl[3 + k] = fmaxf(bl[3 + k], h); }
                        else { br[k] = fminf(br[k], l); br[3 + k] = fmaxf(br[3 + k], h); }
                    }
                }
            }
        }
        const bool lead = open && lane == s0;
        const uint32_t leads = __ballot_sync(kFull, lead);
        uint32_t id = 0;
        if (leads != 0u) {
            if (lane == 0) id = atomicAdd(&cnt->nodes, 2u * (uint32_t)__popc(leads));
            id = __shfl_sync(kFull, id, 0);
            if (id + 2u * (uint32_t)__popc(leads) > max_nodes) {
                if (lane == 0) atomicOr(&cnt->error, kErrNodes);
                return;
            }
        }
        id += 2u * (uint32_t)__popc(leads & ((1u << s0) - 1u));
        if (lead) {
            nodes[node].left = id;
            nodes[node].right = id + 1u;
            write_child(nodes, id, node, bl, bl + 3, root_first + base + s0, nleft);
            write_child(nodes, id + 1u, node, br, br + 3, root_first + base + s0 + nleft, sc - nleft);
        }
        __syncwarp();
        if (open) {
            const uint32_t at = base + (left ? s0 + (uint32_t)__popc(lmask & below) : s0 + nleft + (uint32_t)__popc(~lmask & below));
            S.ref[at] = ref;
            for (int k = 0; k < 3; ++k) { S.lo[k][at] = lo[k]; S.hi[k][at] = hi[k]; }
        }
        __syncwarp();
        if (open) {
            ref = S.ref[base + lane];
            for (int k = 0; k < 3; ++k) { lo[k] = S.lo[k][base + lane]; hi[k] = S.hi[k][base + lane]; }
            const bool in_left = lane - s0 < nleft;
            node = in_left ? id : id + 1u;
            area = in_left ? area6(bl, bl + 3) : area6(br, br + 3);
            if (in_left) { sc = nleft; } else { s0 += nleft; sc -= nleft; }
            open = sc >= 2u;
        }
        __syncwarp();
    }
}

// Finishes the subtree of one small node per warp with its references and boxes
// in shared memory: the same binned SAH splits and stable partitions down to 32
// references, which finish_lanes takes from there.  Children wait on a per-warp
// stack (every entry holds two or more references of a disjoint range, so at
// most kSmall / 2 entries are live).  Splitting every node on its own, with
// bins and three scans for two references as for a hundred, took 3.38 ms of the
// 1.48 M-triangle terrain's build; 1.09 ms now (predicated instead of branching sums: 1.39;
// nodes of up to 64 / 96 references here and larger ones in the level passes: builds 4.64 / 4.60 ms against 4.51).
__global__ void __launch_bounds__(kSmallWarps * 32, 5) k_small(const Task* __restrict__ small, uint32_t nsmall,
                                                            const uint32_t* __restrict__ refs0,
                                                            const uint32_t* __restrict__ refs1,
                                                            uint32_t* __restrict__ final_refs,
                                                            const float4* __restrict__ box, BNode* __restrict__ nodes,
                                                            Counters* cnt, int B, uint32_t max_leaf,
                                                            uint32_t max_nodes) {
    __shared__ SmallSet s_set[kSmallWarps];
    __shared__ union { Bin bins[3 * kBins]; SmallSet tmp; } s_work[kSmallWarps];
    __shared__ uint32_t s_stack[kSmallWarps][kSmall / 2][3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t task = blockIdx.x * kSmallWarps + warp;
    if (task >= nsmall) return;   // whole warps; no block-wide barrier below
    const uint32_t lt = (1u << lane) - 1u;
    const Task root = small[task];
    const uint32_t n0 = root.end - root.begin;
    if (n0 > kSmall) { if (lane == 0) atomicOr(&cnt->error, kErrStack); return; }
    SmallSet& S = s_set[warp];
    SmallSet& T = s_work[warp].tmp;
    Bin* SB = s_work[warp].bins;
    for (uint32_t i = lane; i < n0; i += 32) {
        const uint32_t r = (root.aux ? refs1 : refs0)[root.begin + i];
        const float4 l = box[2 * (size_t)r], h = box[2 * (size_t)r + 1];
        S.ref[i] = r;
        S.lo[0][i] = l.x; S.lo[1][i] = l.y; S.lo[2][i] = l.z;
        S.hi[0][i] = h.x; S.hi[1][i] = h.y; S.hi[2][i] = h.z;
    }
    int sp = 0;
    if (lane == 0) { s_stack[warp][0][0] = root.node; s_stack[warp][0][1] = 0; s_stack[warp][0][2] = n0; }
    sp = 1;
    __syncwarp();
    while (sp > 0) {
        --sp;
        const uint32_t node = s_stack[warp][sp][0], b = s_stack[warp][sp][1], e = s_stack[warp][sp][2];
        __syncwarp();
        const uint32_t n = e - b;
        const float area = area6(nodes[node].lo, nodes[node].hi);
        if (n <= 32u) {
            finish_lanes(S, b, n, root.begin, node, area, nodes, cnt, B, max_leaf, max_nodes);
            __syncwarp();
            continue;
        }
        // centroid bounds
        Task tk;
        tk.node = node;
        tk.begin = b;
        tk.end = e;
        float cl[3] = {INFINITY, INFINITY, INFINITY}, chv[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (uint32_t i = b + lane; i < e; i += 32)
            for (int a = 0; a < 3; ++a) {
                const float c = 0.5f * (S.lo[a][i] + S.hi[a][i]);
                cl[a] = fminf(cl[a], c);
                chv[a] = fmaxf(chv[a], c);
            }
        for (int a = 0; a < 3; ++a) { tk.clo[a] = warp_min(cl[a]); tk.chi[a] = warp_max(chv[a]); }
        // bins
        for (int i = lane; i < 3 * kBins; i += 32) {
            SB[i].cnt = 0;
            for (int k = 0; k < 3; ++k) { SB[i].lo[k] = kKeyLo; SB[i].hi[k] = kKeyHi; }
        }
        __syncwarp();
        float sc[3];
        for (int a = 0; a < 3; ++a) sc[a] = axis_scale(tk, a, B);
        for (uint32_t i = b + lane; i < e; i += 32) {
            uint32_t kl[3], kh[3];
            for (int k = 0; k < 3; ++k) { kl[k] = fkey(S.lo[k][i]); kh[k] = fkey(S.hi[k][i]); }
            for (int a = 0; a < 3; ++a) {
                if (!(sc[a] > 0.0f)) continue;
                Bin& bb = SB[a * kBins + bin_of(0.5f * (S.lo[a][i] + S.hi[a][i]), tk.clo[a], sc[a], B)];
                atomicAdd(&bb.cnt, 1u);
                for (int k = 0; k < 3; ++k) { atomicMin(&bb.lo[k], kl[k]); atomicMax(&bb.hi[k], kh[k]); }
            }
        }
        __syncwarp();
        int bbin;
        uint32_t bnl;
        float best, bx[2][6];
        int bax = warp_best_split(tk, B, [&](int a) {
            Bin z;
            z.cnt = 0;
            return lane < B ? SB[a * kBins + lane] : z;
        }, &bbin, &bnl, &best, bx);
        const Split s = decide(bax, bbin, bnl, best, n, area, max_leaf);   // never a leaf: leaves hold at most two
        __syncwarp();
        // stable partition through T
        uint32_t lc = 0, rc = 0;
        for (uint32_t base = b; base < e; base += 32) {
            const uint32_t i = base + lane;
            const bool act = i < e;
            float lo[3] = {0.0f, 0.0f, 0.0f}, hi[3] = {0.0f, 0.0f, 0.0f};
            bool left = false;
            if (act) {
                for (int k = 0; k < 3; ++k) { lo[k] = S.lo[k][i]; hi[k] = S.hi[k][i]; }
                if (s.axis < 0) {
                    left = i - b < s.nl;
                } else {
                    const int a = s.axis;
                    const float c = a == 0 ? 0.5f * (lo[0] + hi[0]) : a == 1 ? 0.5f * (lo[1] + hi[1]) : 0.5f * (lo[2] + hi[2]);
                    left = bin_of(c, tk.clo[a], sc[a], B) < s.bin;
                }
            }
            const bool right = act && !left;
            const uint32_t wl = __ballot_sync(0xffffffffu, left), wr = __ballot_sync(0xffffffffu, right);
            if (act) {
                const uint32_t at = left ? lc + __popc(wl & lt) : s.nl + rc + __popc(wr & lt);
                T.ref[at] = S.ref[i];
                for (int k = 0; k < 3; ++k) { T.lo[k][at] = lo[k]; T.hi[k][at] = hi[k]; }
            }
            lc += __popc(wl);
            rc += __popc(wr);
        }
        __syncwarp();
        for (uint32_t i = lane; i < n; i += 32) {
            S.ref[b + i] = T.ref[i];
            for (int k = 0; k < 3; ++k) { S.lo[k][b + i] = T.lo[k][i]; S.hi[k][b + i] = T.hi[k][i]; }
        }
        const uint32_t mid = b + s.nl;
        int writer = bbin;   // the children's boxes are in the lane of the split's bin
        if (s.axis < 0) {    // split by index: no bins
            writer = 0;
            for (int c = 0; c < 2; ++c)
                for (int k = 0; k < 3; ++k) {
                    float lo = INFINITY, hi = -INFINITY;
                    for (uint32_t i = (c ? mid : b) + lane; i < (c ? e : mid); i += 32) {
                        lo = fminf(lo, T.lo[k][i - b]);
                        hi = fmaxf(hi, T.hi[k][i - b]);
                    }
                    bx[c][k] = warp_min(lo);
                    bx[c][3 + k] = warp_max(hi);
                }
        }
        uint32_t id = 0;
        if (lane == 0) id = atomicAdd(&cnt->nodes, 2u);
        id = __shfl_sync(0xffffffffu, id, 0);
        if (id + 2u > max_nodes) {
            if (lane == 0) atomicOr(&cnt->error, kErrNodes);
            return;
        }
        if (lane == writer) {
            nodes[node].left = id;
            nodes[node].right = id + 1u;
            write_child(nodes, id, node, bx[0], bx[0] + 3, root.begin + b, s.nl);
            write_child(nodes, id + 1u, node, bx[1], bx[1] + 3, root.begin + mid, e - mid);
        }
        // push right then left (left is finished first); single-reference children are leaves
        for (int c = 0; c < 2; ++c) {
            const uint32_t cb = c == 0 ? mid : b, ce = c == 0 ? e : mid;
            if (ce - cb <= 1u) continue;
            if (sp >= (int)(kSmall / 2)) {
                if (lane == 0) atomicOr(&cnt->error, kErrStack);
                return;
            }
            if (lane == 0) {
                s_stack[warp][sp][0] = id + (c == 0 ? 1u : 0u);
                s_stack[warp][sp][1] = cb;
                s_stack[warp][sp][2] = ce;
            }
            ++sp;
        }
        __syncwarp();
    }
    __syncwarp();
    for (uint32_t i = lane; i < n0; i += 32) final_refs[root.begin + i] = S.ref[i];
}

// ------------------------------------------------------------ phase 3 ----
// Adds to one of kSahSums partial sums, a warp at a time: no barrier, since a block's last climbers are far behind
// its first, and no address that every warp adds to.
constexpr uint32_t kSahSums = 256;
__device__ __forceinline__ void add_sah(double v, double* sums) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31u) == 0u) atomicAdd(sums + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) % kSahSums, v);
}

// cost(n, i) for i = 1..8 and the decisions, as the host's Collapse::run; the
// nodes' areas and leaf counts go to the tree's SAH cost on the way.
// A climb is one round trip to L2 after another: the parent's node is loaded
// while its counter is on the way, the node's own costs stay in registers, and
// the counter's atomic releases and acquires by itself, which costs less than a
// full fence on both sides of it (builds of 1.48 M / 4.97 M triangles 4.67 /
// 13.2 -> 4.63 / 13.05 ms; with the fences kept 4.69 / 13.3).
__device__ __forceinline__ double climb(const BNode* __restrict__ nodes, uint32_t n, uint32_t i,
                                        uint32_t* __restrict__ visits, float4* __restrict__ cost,
                                        uint2* __restrict__ dec, uint8_t* __restrict__ isplit, uint32_t max_leaf,
                                        float tri_cost, Counters* cnt) {
    if (i >= n) return 0.0;
    const BNode L = nodes[i];
    if (L.left != kNone) return 0.0;   // climbs start at leaves
    double sah;
    float c[8];   // the costs of the node just finished
    {
        const float a = area6(L.lo, L.hi);
        sah = (double)a * (double)L.count;
        const float leaf = L.count <= max_leaf ? a * (float)L.count * tri_cost : INFINITY;
        for (int k = 0; k < 8; ++k) c[k] = leaf;
        cost[2 * (size_t)i] = make_float4(leaf, leaf, leaf, leaf);
        cost[2 * (size_t)i + 1] = make_float4(leaf, leaf, leaf, leaf);
        constexpr uint32_t same = kDecSame * 0x01010101u;
        dec[i] = make_uint2((same & 0xffffff00u) | kDecLeaf, same);
    }
    uint32_t x = L.parent, from = i;
    for (uint32_t guard = 0; x != kNone; ++guard) {
        if (guard > n) { atomicOr(&cnt->error, kErrClimb); return sah; }
        // the parent's node (earlier kernels') comes with the answer whether the other child is done
        const BNode X = nodes[x];
        uint32_t before;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(visits + x) : "memory");
        if (before == 0u) return sah;
        const bool right = X.right == from;
        const uint32_t other = right ? X.left : X.right;
        const float4 oa = __ldcg(&cost[2 * (size_t)other]), ob = __ldcg(&cost[2 * (size_t)other + 1]);
        const float o[8] = {oa.x, oa.y, oa.z, oa.w, ob.x, ob.y, ob.z, ob.w};
        float cl[8], cr[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) { cl[k] = right ? o[k] : c[k]; cr[k] = right ? c[k] : o[k]; }
        float dist[9];
        uint32_t arg[9];
#pragma unroll
        for (int j = 2; j <= 8; ++j) {
            dist[j] = INFINITY;
            arg[j] = 1;
#pragma unroll
            for (int k = 1; k < j; ++k) {
                float v = cl[k - 1] + cr[j - k - 1];
                if (v < dist[j]) { dist[j] = v; arg[j] = (uint32_t)k; }
            }
        }
        const float a = area6(X.lo, X.hi);
        sah += (double)a;
        const float leaf = X.count <= max_leaf ? a * (float)X.count * tri_cost : INFINITY;
        const float inner = a + dist[8];   // node cost 1
        uint32_t d[2] = {0u, 0u};
        if (leaf <= inner) { c[0] = leaf; d[0] = kDecLeaf; } else { c[0] = inner; d[0] = kDecInner; }
#pragma unroll
        for (int k = 2; k <= 8; ++k) {
            uint32_t e;
            if (c[k - 2] <= dist[k]) { c[k - 1] = c[k - 2]; e = kDecSame; }
            else { c[k - 1] = dist[k]; e = arg[k]; }
            d[(k - 1) >> 2] |= e << (8 * ((k - 1) & 3));
        }
        cost[2 * (size_t)x] = make_float4(c[0], c[1], c[2], c[3]);
        cost[2 * (size_t)x + 1] = make_float4(c[4], c[5], c[6], c[7]);
        dec[x] = make_uint2(d[0], d[1]);
        isplit[x] = (uint8_t)arg[8];
        from = x;
        x = X.parent;
    }
    return sah;
}

__global__ void __launch_bounds__(256, 6) k_collapse(const BNode* __restrict__ nodes, uint32_t n,
                                                  uint32_t* __restrict__ visits, float4* __restrict__ cost,
                                                  uint2* __restrict__ dec, uint8_t* __restrict__ isplit,
                                                  uint32_t max_leaf, float tri_cost, double* sah, Counters* cnt) {
    add_sah(climb(nodes, n, blockIdx.x * blockDim.x + threadIdx.x, visits, cost, dec, isplit, max_leaf, tri_cost, cnt), sah);
}

__global__ void __launch_bounds__(256) k_sah_cost(const BNode* __restrict__ nodes, uint32_t n, double* out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    double v = 0.0;
    if (i < n) {
        const BNode b = nodes[i];
        v = (double)area6(b.lo, b.hi) * (b.left == kNone ? (double)b.count : 1.0);
    }
    add_sah(v, out);
}

// ------------------------------------------------------------ phase 4 ----
struct WideCfg {
    const BNode* nodes;
    const uint8_t* dec;
    const uint8_t* isplit;
    bool optimal;
    uint32_t max_leaf;
};

__device__ __forceinline__ bool wide_leaf(const WideCfg& w, uint32_t x) {
    if (w.optimal) return w.dec[8 * (size_t)x] == kDecLeaf;
    const BNode& b = w.nodes[x];
    return b.left == kNone || b.count <= w.max_leaf;
}

// ---- 8 lanes per 8-wide node ----
constexpr uint32_t kWideThreads = 256;
constexpr uint32_t kWideTile = kWideThreads / kWideLanes;   // nodes per block and round
static_assert(kWideTile == 32, "one warp scans a tile's nodes");

// First child and triangle of every tile within the level, and the next level, by the last block of k_wide_nodes
// (a launch of its own per level cost builds of 20 k / 1.48 M triangles 0.02 ms).
__device__ __forceinline__ void wide_scan(uint2* sums, const WideLevel& lv, uint32_t wnode_cap, uint32_t num_tris,
                                          Counters* cnt, int cur) {
    __shared__ uint2 s_w[kWideThreads / 32];
    const uint32_t n = __syncthreads_or(__ldcg(&cnt->error) != 0u) ? 0u : (lv.nodes + kWideTile - 1u) / kWideTile;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint2 carry = make_uint2(0u, 0u);
    for (uint32_t base = 0; base < n; base += kWideThreads) {
        const uint32_t i = base + threadIdx.x;
        const uint2 v = i < n ? __ldcg(sums + i) : make_uint2(0u, 0u);
        uint2 x = v;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t yx = __shfl_up_sync(0xffffffffu, x.x, o), yy = __shfl_up_sync(0xffffffffu, x.y, o);
            if (lane >= o) { x.x += yx; x.y += yy; }
        }
        if (lane == 31u) s_w[warp] = x;
        __syncthreads();
        uint2 before = make_uint2(0u, 0u), all = before;
        for (uint32_t k = 0; k < kWideThreads / 32; ++k) {
            const uint2 t = s_w[k];
            if (k < warp) { before.x += t.x; before.y += t.y; }
            all.x += t.x;
            all.y += t.y;
        }
        __syncthreads();
        if (i < n) sums[i] = make_uint2(carry.x + before.x + x.x - v.x, carry.y + before.y + x.y - v.y);
        carry.x += all.x;
        carry.y += all.y;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        WideLevel next{carry.x, lv.node_base + lv.nodes, lv.tri_base + carry.y, 0u};
        if (n == 0u) next = WideLevel{0u, lv.node_base, lv.tri_base, 0u};
        else cnt->depth += 1u;
        if ((uint64_t)next.node_base + next.nodes > wnode_cap || next.tri_base > num_tris) {
            atomicOr(&cnt->error, kErrWide);
            next.nodes = 0u;
        }
        cnt->wide[cur ^ 1] = next;
    }
}

// The nodes of a level: each gathers its up to eight children, assigns octant
// slots and quantises their boxes, a child per lane, with its first child and
// triangle counted from the start of its tile.  (A thread per node took 0.50 ms
// for the gathering and 1.04 ms for quantising and writing of the 1.48 M-
// triangle terrain, most of it one node's serial chain per level; 0.42 and
// 0.09 ms now.)
__global__ void __launch_bounds__(kWideThreads) k_wide_nodes(const uint32_t* __restrict__ queue, WideCfg w,
                                                             WideRec* __restrict__ rec, uint2* __restrict__ tile_sums,
                                                             CwNode* __restrict__ wnodes, uint32_t wnode_cap,
                                                             uint32_t num_tris, Counters* cnt, int cur) {
    __shared__ uint2 s_entry[kWideTile][kWideLanes];
    __shared__ uint32_t s_child[kWideTile][kWideLanes];
    __shared__ uint4 s_image[kWideTile][sizeof(CwNode) / 16];
    __shared__ uint32_t s_ni[kWideTile], s_nt[kWideTile];
    constexpr uint32_t kFull = 0xffffffffu;
    const WideLevel lv = cnt->wide[cur];
    // other blocks may set the error word while this one starts: its threads have to agree on what they read
    const uint32_t nq = __syncthreads_or(cnt->error != 0u) ? 0u : lv.nodes;
    const uint32_t g = threadIdx.x / kWideLanes, sub = threadIdx.x % kWideLanes;
    const uint32_t shift = (threadIdx.x & 31u) & ~(kWideLanes - 1u);   // the group's first lane in its warp
    for (uint32_t tile = blockIdx.x; tile * kWideTile < nq; tile += gridDim.x) {
        const uint32_t q = tile * kWideTile + g;
        const bool node_ok = q < nq;
        const uint32_t bi = node_ok ? queue[q] : 0u;
        uint32_t x = kNone;      // this lane's child; lanes are in the order of the children
        bool bad = false;
        const bool root_leaf = node_ok && wide_leaf(w, bi);
        s_entry[g][sub] = make_uint2(0u, 0u);
        s_child[g][sub] = kNone;
        if (sub < sizeof(CwNode) / 16) s_image[g][sub] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        if (root_leaf && sub == 0) x = bi;   // a root that is a single leaf
        if (w.optimal) {
            // an entry of budget i at lane p stands for the children at lanes p .. p + i - 1
            uint32_t i = 0;
            if (node_ok && !root_leaf) {
                const uint32_t k = w.isplit[bi];
                if (sub == 0) { x = w.nodes[bi].left; i = k; }
                if (sub == k) { x = w.nodes[bi].right; i = 8u - k; }
                if (k == 0u || k > 7u) { bad = true; x = kNone; i = 0u; }
            }
            __syncwarp();
            for (int round = 0; round < 8; ++round) {
                const bool open = x != kNone && i > 1u;
                if (__ballot_sync(kFull, open) == 0u) break;
                if (open) {
                    const uint2 d = *reinterpret_cast<const uint2*>(w.dec + 8 * (size_t)x);
                    auto dec = [&](uint32_t j) { return (uint32_t)((j < 4u ? d.x >> (8u * j) : d.y >> (8u * (j - 4u))) & 255u); };
                    while (i > 1u && dec(i - 1u) == kDecSame) --i;
                    if (i > 1u) {
                        const uint32_t k2 = dec(i - 1u), l = w.nodes[x].left, r = w.nodes[x].right;
                        if (k2 == 0u || k2 >= i || l == kNone) {
                            bad = true;
                            i = 0u;
                        } else {
                            s_entry[g][sub + k2] = make_uint2(r, i - k2);
                            x = l;
                            i = k2;
                        }
                    }
                }
                __syncwarp();
                const uint2 e = s_entry[g][sub];
                if (e.y != 0u) { x = e.x; i = e.y; s_entry[g][sub] = make_uint2(0u, 0u); }
                __syncwarp();
            }
        } else {
            if (node_ok && !root_leaf) {
                if (sub == 0) x = w.nodes[bi].left;
                if (sub == 1) x = w.nodes[bi].right;
            }
            bool more = node_ok && !root_leaf;
            for (uint32_t nc = 2; nc < kWideLanes; ++nc) {   // open the largest child, the first of equal ones
                float area = -1.0f;
                if (more && x != kNone && !wide_leaf(w, x)) area = area6(w.nodes[x].lo, w.nodes[x].hi);
                const float most = wide_max(area);
                const uint32_t at = (__ballot_sync(kFull, area == most) >> shift) & 0xffu;
                if (most < 0.0f) more = false;
                const uint32_t src = (uint32_t)__ffs(at) - 1u;
                const uint32_t opened = __shfl_sync(kFull, x, (int)(shift + src));
                if (more) {
                    if (sub == nc) x = w.nodes[opened].right;
                    if (sub == src) x = w.nodes[opened].left;
                }
            }
        }
        if (wide_or(bad ? 1u : 0u) != 0u) {
            if (sub == 0) atomicOr(&cnt->error, kErrGather);
            x = kNone;
        }
        const bool valid = x != kNone;
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        uint32_t count = 0;
        bool leaf = false;
        if (valid) {
            const uint4* p = reinterpret_cast<const uint4*>(w.nodes + x);
            const uint4 n0 = p[0], n1 = p[1], n2 = p[2];
            lo[0] = __uint_as_float(n0.x); lo[1] = __uint_as_float(n0.y); lo[2] = __uint_as_float(n0.z);
            hi[0] = __uint_as_float(n1.x); hi[1] = __uint_as_float(n1.y); hi[2] = __uint_as_float(n1.z);
            count = n2.y;
            leaf = wide_leaf(w, x);
        }
        float nlo[3], nhi[3], d[3];
        for (int k = 0; k < 3; ++k) {
            nlo[k] = wide_min(lo[k]);
            nhi[k] = wide_max(hi[k]);
            d[k] = 0.5f * (lo[k] + hi[k]) - 0.5f * (nlo[k] + nhi[k]);
        }
        // greedy octant slots: in every round the child and free slot whose direction agrees best, the first child
        // and then the first slot of equal ones
        uint32_t used = 0, slot = kNone;
        const uint32_t nc = (uint32_t)__popc((__ballot_sync(kFull, valid) >> shift) & 0xffu);
        for (uint32_t round = 0; round < kWideLanes; ++round) {
            float best = -INFINITY;
            uint32_t key = kNone;
            if (valid && slot == kNone)
                for (uint32_t s = 0; s < 8u; ++s) {
                    if ((used >> s) & 1u) continue;
                    const float cost = ((s & 1u) ? d[0] : -d[0]) + ((s & 2u) ? d[1] : -d[1]) + ((s & 4u) ? d[2] : -d[2]);
                    if (cost > best || key == kNone) { best = cost; key = (sub << 3) | s; }
                }
            for (int o = 1; o < (int)kWideLanes; o <<= 1) {
                const float ob = __shfl_xor_sync(kFull, best, o);
                const uint32_t ok = __shfl_xor_sync(kFull, key, o);
                if (ok != kNone && (key == kNone || ob > best || (ob == best && ok < key))) { best = ob; key = ok; }
            }
            if (round < nc) {
                used |= 1u << (key & 7u);
                if ((key >> 3) == sub) slot = key & 7u;
            }
        }
        // Where centres or distances overflow, costs are infinite or NaN and the lanes may not have agreed: the children
        // take the slots in their order (as comparing the pairs one after the other gives if all costs are NaN).
        const bool far = valid && !(fabsf(d[0]) + fabsf(d[1]) + fabsf(d[2]) < INFINITY);
        if (((__ballot_sync(kFull, far) >> shift) & 0xffu) != 0u) slot = sub;
        if (leaf && (count == 0u || count > kMaxLeafTris)) {
            atomicOr(&cnt->error, kErrLeaf);
            leaf = false;
            count = 0u;
        }
        const uint32_t imask = wide_or(valid && !leaf && count != 0u ? 1u << slot : 0u);
        const uint32_t tmask = wide_or(leaf ? ((1u << count) - 1u) << (2u * slot) : 0u);
        uint8_t* image = reinterpret_cast<uint8_t*>(s_image[g]);
        quantise_lanes(image, valid, slot, nc != 0u, lo, hi, nlo, nhi);
        if (valid) s_child[g][slot] = x;
        if (sub == 0) {
            image[15] = (uint8_t)imask;
            reinterpret_cast<uint32_t*>(image)[6] = tmask;   // tri_mask, padding
            s_ni[g] = (uint32_t)__popc(imask);
            s_nt[g] = (uint32_t)__popc(tmask);
        }
        __syncthreads();
        if (threadIdx.x < 32) {   // first child and triangle of every node within the tile
            const uint32_t vi = s_ni[threadIdx.x], vt = s_nt[threadIdx.x];
            uint32_t xi = vi, xt = vt;
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t yi = __shfl_up_sync(kFull, xi, o), yt = __shfl_up_sync(kFull, xt, o);
                if (threadIdx.x >= o) { xi += yi; xt += yt; }
            }
            s_ni[threadIdx.x] = xi - vi;
            s_nt[threadIdx.x] = xt - vt;
            if (threadIdx.x == 31) tile_sums[tile] = make_uint2(xi, xt);
        }
        __syncthreads();
        if (node_ok) {
            rec[q].child[sub] = s_child[g][sub];
            if (lv.node_base + q >= wnode_cap) {
                if (sub == 0) atomicOr(&cnt->error, kErrWide);
            } else if (sub < sizeof(CwNode) / 16) {
                uint4 v = s_image[g][sub];
                if (sub == 1) { v.x = s_ni[g]; v.y = s_nt[g]; }
                reinterpret_cast<uint4*>(wnodes + lv.node_base + q)[sub] = v;
            }
        }
        __syncthreads();
    }
    // the block that ends last scans the tiles
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd(&cnt->wide_blocks, 1u) == gridDim.x - 1u;
        if (s_last) cnt->wide_blocks = 0u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    wide_scan(tile_sums, lv, wnode_cap, num_tris, cnt, cur);
}

struct TriSrc {
    const float* pos;
    const uint32_t* idx;
    const uint32_t* mat;
    const float* transp;
    uint32_t num_materials;
    const uint32_t* final_refs;
};

__device__ void emit_tri(const TriSrc& s, uint32_t t, CwTri* out) {
    CwTri c;
    float v[3][3];
    for (int k = 0; k < 3; ++k) {
        const size_t vi = s.idx ? s.idx[3 * (size_t)t + k] : 3 * (size_t)t + k;
        v[k][0] = s.pos[3 * vi];
        v[k][1] = s.pos[3 * vi + 1];
        v[k][2] = s.pos[3 * vi + 2];
    }
    c.v0x = v[0][0]; c.v0y = v[0][1]; c.v0z = v[0][2];
    c.v1x = v[1][0]; c.v1y = v[1][1]; c.v1z = v[1][2];
    c.v2x = v[2][0]; c.v2y = v[2][1]; c.v2z = v[2][2];
    c.prim = t;
    c.material = s.mat ? s.mat[t] : 0u;
    const float tr = (s.transp && c.material < s.num_materials) ? s.transp[c.material] : 0.0f;
    c.pad = __float_as_uint(tr);
    *out = c;
}

// The level's nodes get their places, their leaf triangles are written and their
// internal children queued; a slot per lane.
__global__ void __launch_bounds__(kWideThreads) k_wide_emit(const WideRec* __restrict__ rec,
                                                            const uint2* __restrict__ sums, WideCfg w, TriSrc src,
                                                            CwNode* __restrict__ wnodes, CwTri* __restrict__ wtris,
                                                            uint32_t num_tris, uint32_t* __restrict__ next_queue,
                                                            uint32_t queue_cap, Counters* cnt, int cur) {
    const WideLevel lv = cnt->wide[cur];
    const uint32_t nq = __syncthreads_or(cnt->error != 0u) ? 0u : lv.nodes;   // read once, as in k_wide_nodes
    const uint32_t g = threadIdx.x / kWideLanes, s = threadIdx.x % kWideLanes;
    const uint32_t node_lanes = 0xffu << (threadIdx.x & 31u & ~(kWideLanes - 1u));   // they agree on q
    for (uint32_t tile = blockIdx.x; tile * kWideTile < nq; tile += gridDim.x) {
        const uint32_t q = tile * kWideTile + g;
        if (q >= nq) continue;   // no barrier below
        const uint2 sum = sums[tile];
        uint4* p = reinterpret_cast<uint4*>(wnodes + lv.node_base + q);
        const uint32_t imask = p[0].w >> 24;
        uint4 h = p[1];
        const uint32_t child = rec[q].child[s], tm = h.z & 0xffffu;
        const uint32_t first = sum.x + h.x, tri = lv.tri_base + sum.y + h.y;
        __syncwarp(node_lanes);   // every lane of the node has read the header before it is rewritten
        if (s == 0) {
            h.x = lv.node_base + lv.nodes + first;
            h.y = tri;
            p[1] = h;
        }
        if ((imask >> s) & 1u) {
            const uint32_t at = first + (uint32_t)__popc(imask & ((1u << s) - 1u));
            if (at < queue_cap) next_queue[at] = child;
            else atomicOr(&cnt->error, kErrWide);
        }
        const uint32_t c = (uint32_t)__popc((tm >> (2u * s)) & 3u);
        if (c != 0u) {   // a leaf's references are consecutive, also those of a collapsed pair
            const uint32_t at = tri + (uint32_t)__popc(tm & ((1u << (2u * s)) - 1u)), ref = w.nodes[child].first;
            for (uint32_t j = 0; j < c; ++j) {
                if (at + j >= num_tris) { atomicOr(&cnt->error, kErrLeaf); break; }
                emit_tri(src, src.final_refs[ref + j], &wtris[at + j]);
            }
        }
    }
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Scratch layout for num_tris triangles (all offsets 256-byte aligned).
struct Layout {
    size_t box, refs0, refs1, final_refs, bnodes, visits, cost, dec, isplit, tasks0, tasks1, small, bins,
        splits, acc, chunk_task, chunk_bins, left_base, queue0, queue1, rec, tile_sums, wnodes, counters, gkeys, sah, total;
    uint32_t max_nodes, task_cap, small_cap, chunk_cap, wnode_cap;
};

Layout make_layout(uint32_t T) {
    Layout L{};
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off += align256(std::max<size_t>(bytes, 16)); return o; };
    L.max_nodes = 2 * T;
    L.task_cap = T / kSmall + 2;
    L.small_cap = T / 2 + 2;
    L.chunk_cap = T / chunk_size(T) + L.task_cap + 2;
    L.wnode_cap = T + 1;
    L.box = take((size_t)T * 32);
    L.refs0 = take((size_t)T * 4);
    L.refs1 = take((size_t)T * 4);
    L.final_refs = take((size_t)T * 4);
    L.bnodes = take((size_t)L.max_nodes * sizeof(BNode));
    L.visits = take((size_t)L.max_nodes * 4);
    L.cost = take((size_t)L.max_nodes * 32);
    L.dec = take((size_t)L.max_nodes * 8);
    L.isplit = take((size_t)L.max_nodes);
    L.tasks0 = take((size_t)L.task_cap * sizeof(Task));
    L.tasks1 = take((size_t)L.task_cap * sizeof(Task));
    L.small = take((size_t)L.small_cap * sizeof(Task));
    L.bins = take((size_t)L.task_cap * 3 * kBins * sizeof(Bin));
    L.splits = take((size_t)L.task_cap * sizeof(Split));
    L.acc = take((size_t)L.task_cap * sizeof(ChildAcc));
    L.chunk_task = take((size_t)L.chunk_cap * 4);
    L.chunk_bins = take((size_t)L.chunk_cap * sizeof(ChunkBins));
    L.left_base = take((size_t)L.chunk_cap * 4);
    L.queue0 = take((size_t)L.wnode_cap * 4);
    L.queue1 = take((size_t)L.wnode_cap * 4);
    L.rec = take((size_t)L.wnode_cap * sizeof(WideRec));
    L.tile_sums = take((size_t)(L.wnode_cap / kWideTile + 1) * 8);
    L.wnodes = take((size_t)L.wnode_cap * sizeof(CwNode));
    L.counters = take(sizeof(Counters));
    L.gkeys = take(12 * 4);
    L.sah = take(kSahSums * 8);
    L.total = off;
    return L;
}

uint32_t blocks_for(uint64_t n, uint32_t threads) { return (uint32_t)std::max<uint64_t>(1, (n + threads - 1) / threads); }

std::string error_text(uint32_t e) {
    std::string m;
    if (e & kErrIndex) m += " vertex index out of range;";
    if (e & kErrFinite) m += " non-finite vertex position;";
    if (e & kErrNodes) m += " node or task capacity exceeded;";
    if (e & kErrGather) m += " wide-node gather failed;";
    if (e & kErrLeaf) m += " leaf size out of range;";
    if (e & kErrStack) m += " small-node stack overflow;";
    if (e & kErrClimb) m += " collapse climb did not end;";
    if (e & kErrWide) m += " wide-node capacity exceeded;";
    if (e & kErrPartition) m += " partition count mismatch;";
    return m;
}

}  // namespace

uint64_t device_build_scratch_bytes(uint32_t num_tris) { return make_layout(num_tris).total; }
uint64_t device_build_output_bytes(uint32_t num_tris) {
    return (uint64_t)(num_tris + 1) * sizeof(CwNode) + (uint64_t)num_tris * sizeof(CwTri);
}

bool build_cwbvh_device(cudaStream_t st, const float* pos, uint32_t nv, const uint32_t* idx, uint32_t T,
                        const uint32_t* mat, const float* transparency, uint32_t num_materials,
                        const bsm_bvh_opts* opts_in, DeviceBvhResult& out, std::string& err) {
    auto t0 = std::chrono::steady_clock::now();
    out = DeviceBvhResult{};
    if (T == 0) { err = "scene has no triangles"; return false; }
    if (T >= kTriGroupFlag) { err = "more than 2^31 - 1 triangles in one BVH"; return false; }
    bsm_bvh_opts opts{};
    if (opts_in) opts = *opts_in;
    if (opts.sah_bins > (uint32_t)kBins) { err = "the device builder takes at most 32 SAH bins"; return false; }
    const int B = opts.sah_bins ? (int)std::max(opts.sah_bins, 4u) : kBins;
    const uint32_t max_leaf = opts.max_leaf_tris ? std::min(opts.max_leaf_tris, kMaxLeafTris) : kMaxLeafTris;
    const bool optimal = opts.collapse == BSM_COLLAPSE_SAH_OPTIMAL;
    const uint32_t bin_leaf = optimal ? 1u : max_leaf;   // the collapse chooses the leaves itself
    const float tri_cost = opts.tri_cost > 0.0f ? opts.tri_cost : 1.0f;

    const Layout L = make_layout(T);
    char* base = nullptr;
    cudaError_t e = cudaMalloc(&base, L.total);
    if (e != cudaSuccess) {
        cudaGetLastError();
        err = std::string("device BVH scratch: ") + cudaGetErrorString(e);
        return false;
    }
    CwTri* wtris = nullptr;
    e = cudaMalloc(&wtris, (size_t)T * sizeof(CwTri));
    if (e != cudaSuccess) {
        cudaGetLastError();
        cudaFree(base);
        err = std::string("device BVH triangles: ") + cudaGetErrorString(e);
        return false;
    }
    auto P = [&](size_t o) { return (void*)(base + o); };
    float4* box = (float4*)P(L.box);
    uint32_t* refs[2] = {(uint32_t*)P(L.refs0), (uint32_t*)P(L.refs1)};
    uint32_t* final_refs = (uint32_t*)P(L.final_refs);
    BNode* bnodes = (BNode*)P(L.bnodes);
    Task* tasks[2] = {(Task*)P(L.tasks0), (Task*)P(L.tasks1)};
    Task* small = (Task*)P(L.small);
    Bin* bins = (Bin*)P(L.bins);
    Split* splits = (Split*)P(L.splits);
    ChildAcc* acc = (ChildAcc*)P(L.acc);
    uint32_t* chunk_task = (uint32_t*)P(L.chunk_task);
    ChunkBins* chunk_bins = (ChunkBins*)P(L.chunk_bins);
    uint32_t* left_base = (uint32_t*)P(L.left_base);
    Counters* cnt = (Counters*)P(L.counters);
    uint32_t* gkeys = (uint32_t*)P(L.gkeys);
    double* sah = (double*)P(L.sah);

    bool ok = false;
    std::string why;
#define DB_CK(call)                                                          \
    do {                                                                     \
        cudaError_t e_ = (call);                                             \
        if (e_ != cudaSuccess) { why = std::string(#call) + ": " + cudaGetErrorString(e_); goto done; } \
    } while (0)
    {
        int dev = 0, sms = 0;
        DB_CK(cudaGetDevice(&dev));
        DB_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        // ---- phase 1 ----
        uint32_t keys0[12];
        for (int k = 0; k < 12; ++k) keys0[k] = (k % 6) >= 3 ? kKeyHi : kKeyLo;
        DB_CK(cudaMemsetAsync(cnt, 0, sizeof(Counters), st));
        DB_CK(cudaMemsetAsync(sah, 0, kSahSums * 8, st));
        DB_CK(cudaMemcpyAsync(gkeys, keys0, sizeof(keys0), cudaMemcpyHostToDevice, st));
        DB_CK(cudaMemsetAsync(P(L.visits), 0, (size_t)L.max_nodes * 4, st));
        k_tri_boxes<<<blocks_for(T, 256), 256, 0, st>>>(pos, nv, idx, T, box, refs[0], gkeys, cnt);
        DB_CK(cudaGetLastError());
        uint32_t keys[12];
        Counters hc;
        DB_CK(cudaMemcpyAsync(keys, gkeys, sizeof(keys), cudaMemcpyDeviceToHost, st));
        DB_CK(cudaMemcpyAsync(&hc, cnt, sizeof(hc), cudaMemcpyDeviceToHost, st));
        DB_CK(cudaStreamSynchronize(st));
        if (hc.error) { why = "device BVH build:" + error_text(hc.error); goto done; }
        auto unkey = [](uint32_t k) {
            uint32_t b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
            float f;
            std::memcpy(&f, &b, 4);
            return f;
        };
        // root node 0
        BNode root;
        for (int k = 0; k < 3; ++k) { root.lo[k] = unkey(keys[k]); root.hi[k] = unkey(keys[3 + k]); }
        root.left = root.right = kNone;
        root.first = 0;
        root.count = T;
        root.parent = kNone;
        root.pad = 0;
        DB_CK(cudaMemcpyAsync(bnodes, &root, sizeof(root), cudaMemcpyHostToDevice, st));
        uint32_t one = 1;
        DB_CK(cudaMemcpyAsync(&cnt->nodes, &one, 4, cudaMemcpyHostToDevice, st));
        Task rt;
        rt.node = 0;
        rt.begin = 0;
        rt.end = T;
        rt.aux = 0;
        for (int k = 0; k < 3; ++k) { rt.clo[k] = unkey(keys[6 + k]); rt.chi[k] = unkey(keys[9 + k]); }
        uint32_t nsmall = 0;
        if (T == 1) {
            DB_CK(cudaMemcpyAsync(final_refs, refs[0], 4, cudaMemcpyDeviceToDevice, st));
        } else if (T <= kSmall) {
            DB_CK(cudaMemcpyAsync(small, &rt, sizeof(rt), cudaMemcpyHostToDevice, st));
            nsmall = 1;
        } else {
            // ---- phase 2: levels of large nodes ----
            // A level has at most 2^level tasks and T / chunk chunks and one per task. The first batch of levels
            // is as many as an even tree has plus four; after it the host looks whether tasks are left.
            DB_CK(cudaMemcpyAsync(tasks[0], &rt, sizeof(rt), cudaMemcpyHostToDevice, st));
            DB_CK(cudaMemcpyAsync(&cnt->tasks[0], &one, 4, cudaMemcpyHostToDevice, st));
            k_bins_init<<<blocks_for((uint64_t)L.task_cap * 3 * kBins, 256), 256, 0, st>>>(bins, L.task_cap * 3 * kBins, acc,
                                                                                          L.task_cap);
            const uint32_t chunk = chunk_size(T), root_chunks = (T + chunk - 1u) / chunk;
            DB_CK(cudaMemcpyAsync(&cnt->chunks[0], &root_chunks, 4, cudaMemcpyHostToDevice, st));
            DB_CK(cudaMemsetAsync(chunk_task, 0, (size_t)root_chunks * 4, st));
            uint32_t batch = 4;
            while ((uint64_t)kSmall << (batch - 4) < T) ++batch;
            uint32_t ntasks = 1;
            for (uint32_t level = 0; ntasks > 0;) {
                if (level > T) { why = "device BVH build: levels do not end"; goto done; }
                for (uint32_t k = 0; k < batch; ++k, ++level) {
                    const int cur = (int)(level & 1u);   // tasks[cur] and refs[cur] are the level's
                    const uint32_t max_tasks = level < 31u ? std::min(1u << level, L.task_cap) : L.task_cap;
                    const uint32_t max_chunks = std::min(T / chunk + max_tasks + 1u, L.chunk_cap);
                    const uint32_t grid = std::min(max_chunks, (uint32_t)sms * 8u);
                    k_bin<<<grid, kLevelThreads, 0, st>>>(chunk_task, tasks[cur], refs[cur], box, bins, chunk_bins, cnt, cur, chunk,
                                                          B);
                    k_split<<<std::min(blocks_for((uint64_t)max_tasks * 32, 128), (uint32_t)sms * 8u), 128, 0, st>>>(
                        tasks[cur], bins, chunk_bins, bnodes, splits, left_base, acc, cnt, cur, chunk, B, bin_leaf);
                    k_partition<<<grid, kLevelThreads, 0, st>>>(chunk_task, tasks[cur], splits, left_base, refs[cur],
                                                                refs[cur ^ 1], box, acc, cnt, cur, chunk, B);
                    k_make_children<<<std::min(blocks_for(max_tasks, 64), (uint32_t)sms * 4u), 64, 0, st>>>(
                        tasks[cur], splits, acc, refs[cur ^ 1], bnodes, final_refs, tasks[cur ^ 1], L.task_cap, small,
                        L.small_cap, chunk_task, L.chunk_cap, chunk, cnt, cur, L.max_nodes);
                }
                DB_CK(cudaGetLastError());
                DB_CK(cudaMemcpyAsync(&hc, cnt, sizeof(hc), cudaMemcpyDeviceToHost, st));
                DB_CK(cudaStreamSynchronize(st));
                if (hc.error) { why = "device BVH build:" + error_text(hc.error); goto done; }
                ntasks = hc.tasks[level & 1u];
                nsmall = hc.small_tasks;
                batch = 4;
            }
        }
        if (nsmall > 0)
            k_small<<<blocks_for(nsmall, kSmallWarps), kSmallWarps * 32, 0, st>>>(small, nsmall, refs[0], refs[1],
                                                                                 final_refs, box, bnodes, cnt, B,
                                                                                 bin_leaf, L.max_nodes);
        DB_CK(cudaGetLastError());
        DB_CK(cudaMemcpyAsync(&hc, cnt, sizeof(hc), cudaMemcpyDeviceToHost, st));
        DB_CK(cudaStreamSynchronize(st));
        if (hc.error) { why = "device BVH build:" + error_text(hc.error); goto done; }
        const uint32_t nb = hc.nodes;
        // ---- phase 3 ----
        if (optimal)
            k_collapse<<<blocks_for(nb, 256), 256, 0, st>>>(bnodes, nb, (uint32_t*)P(L.visits), (float4*)P(L.cost),
                                                            (uint2*)P(L.dec), (uint8_t*)P(L.isplit), max_leaf,
                                                            tri_cost, sah, cnt);
        else
            k_sah_cost<<<blocks_for(nb, 256), 256, 0, st>>>(bnodes, nb, sah);
        DB_CK(cudaGetLastError());
        // ---- phase 4 ----
        WideCfg wc;
        wc.nodes = bnodes;
        wc.dec = (const uint8_t*)P(L.dec);
        wc.isplit = (const uint8_t*)P(L.isplit);
        wc.optimal = optimal;
        wc.max_leaf = max_leaf;
        TriSrc ts;
        ts.pos = pos;
        ts.idx = idx;
        ts.mat = mat;
        ts.transp = transparency;
        ts.num_materials = num_materials;
        ts.final_refs = final_refs;
        uint32_t* queue[2] = {(uint32_t*)P(L.queue0), (uint32_t*)P(L.queue1)};
        uint32_t zero = 0;
        DB_CK(cudaMemcpyAsync(queue[0], &zero, 4, cudaMemcpyHostToDevice, st));   // the binary root
        const WideLevel top{1u, 0u, 0u, 0u};
        DB_CK(cudaMemcpyAsync(&cnt->wide[0], &top, sizeof(top), cudaMemcpyHostToDevice, st));
        // levels in batches, as above; a level has at most 8^level nodes. A level's two launches that find nothing left
        // cost 5 us, which the smallest builds would notice (2 / 9 triangles 0.16 / 0.19 ms, with twelve levels 0.22 / 0.23).
        uint32_t wide_level = 0, wide_left = 1;
        for (uint32_t batch = T <= 8u ? 1u : T <= 32u ? 4u : 12u; wide_left > 0; batch = 4) {
            if (wide_level > T) { why = "device BVH build: wide levels do not end"; goto done; }
            for (uint32_t k = 0; k < batch; ++k, ++wide_level) {
                const int cur = (int)(wide_level & 1u);
                const uint32_t max_nodes = wide_level < 10u ? std::min(1u << (3 * wide_level), L.wnode_cap) : L.wnode_cap;
                const uint32_t grid = std::min(blocks_for(max_nodes, kWideTile), (uint32_t)sms * 8u);
                k_wide_nodes<<<grid, kWideThreads, 0, st>>>(queue[cur], wc, (WideRec*)P(L.rec), (uint2*)P(L.tile_sums),
                                                            (CwNode*)P(L.wnodes), L.wnode_cap, T, cnt, cur);
                k_wide_emit<<<grid, kWideThreads, 0, st>>>((const WideRec*)P(L.rec), (const uint2*)P(L.tile_sums), wc, ts,
                                                           (CwNode*)P(L.wnodes), wtris, T, queue[cur ^ 1], L.wnode_cap, cnt,
                                                           cur);
            }
            DB_CK(cudaGetLastError());
            DB_CK(cudaMemcpyAsync(&hc, cnt, sizeof(hc), cudaMemcpyDeviceToHost, st));
            DB_CK(cudaStreamSynchronize(st));
            if (hc.error) { why = "device BVH build:" + error_text(hc.error); goto done; }
            wide_left = hc.wide[wide_level & 1u].nodes;
        }
        const uint32_t level_base = hc.wide[wide_level & 1u].node_base, tri_cursor = hc.wide[wide_level & 1u].tri_base,
                       depth = hc.depth;
        double hsah = 0.0, part[kSahSums];
        DB_CK(cudaMemcpyAsync(part, sah, sizeof(part), cudaMemcpyDeviceToHost, st));
        DB_CK(cudaStreamSynchronize(st));
        for (double v : part) hsah += v;
        if (tri_cursor != T) { why = "device BVH build: triangle count mismatch"; goto done; }
        CwNode* nodes_out = nullptr;
        DB_CK(cudaMalloc(&nodes_out, (size_t)level_base * sizeof(CwNode)));
        e = cudaMemcpyAsync(nodes_out, P(L.wnodes), (size_t)level_base * sizeof(CwNode), cudaMemcpyDeviceToDevice, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            cudaFree(nodes_out);
            why = std::string("device BVH nodes: ") + cudaGetErrorString(e);
            goto done;
        }
        const double ra = (double)((root.hi[0] - root.lo[0]) * (root.hi[1] - root.lo[1]) +
                                   (root.hi[1] - root.lo[1]) * (root.hi[2] - root.lo[2]) +
                                   (root.hi[2] - root.lo[2]) * (root.hi[0] - root.lo[0])) * 2.0;
        out.nodes = nodes_out;
        out.tris = wtris;
        out.num_nodes = level_base;
        out.num_tris = T;
        out.max_depth = depth;
        out.sah_cost = ra > 0.0 ? hsah / ra : 0.0;
        ok = true;
    }
done:
#undef DB_CK
    cudaStreamSynchronize(st);
    cudaFree(base);
    if (!ok) {
        cudaFree(wtris);
        cudaGetLastError();
        err = why.empty() ? "device BVH build failed" : why;
        return false;
    }
    out.build_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return true;
}

}  // namespace bsm
