// mgbvh_device.cuh — device-side types and the warp subtree builder.
//
// A subtree whose root holds at most 32 objects is built by one warp, all nodes
// of one depth at a time (warp_build_subtree below): each node is a range of
// lanes, and object sets are 32-bit masks over the subtree's sorted orders.
#pragma once

#include <cstdint>

#include "mgbvh_exact.cuh"
#include "../../include/mgbvh.h"

namespace mgbvh {

constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr uint32_t kSmallMax = 32;  // warp subtree size
constexpr uint32_t kMaxBins = 32;
constexpr uint32_t kNoKey = 0xFFFFFFFFu;

// Split parameters, the const generics and BvhSettings of the crate.
struct Params {
    uint32_t min_leaf;        // MIN_LEAF_OBJECTS
    uint32_t max_leaf;        // MAX_LEAF_OBJECTS
    uint32_t max_depth;       // BvhSettings::max_depth
    uint32_t bins;            // 0: len.clamp(16,32)
    uint32_t adaptive_max_n;  // adaptive sweep for len <= this (<= 32)
    uint32_t adaptive_steps;  // 0: len.clamp(8,32)
    uint32_t medium_max;      // nodes above this go through the level passes (<= 1024)
};

// Streamed output: the node slots split into kStreamChunks ranges; a subtree
// of <= 32 objects whose children pair starts in range c is built by the
// c-th launch of the small kernel.
constexpr uint32_t kStreamChunks = 8;

__host__ __device__ __forceinline__ uint32_t stream_chunk(uint32_t pair, uint32_t slots) {
    const uint32_t c = static_cast<uint32_t>((static_cast<uint64_t>(pair) * kStreamChunks) / slots);
    return c < kStreamChunks ? c : kStreamChunks - 1u;
}

// First slot of chunk c (c = kStreamChunks: the slot count).
__host__ __device__ __forceinline__ uint32_t stream_chunk_begin(uint32_t c, uint32_t slots) {
    return static_cast<uint32_t>((static_cast<uint64_t>(c) * slots + kStreamChunks - 1u) / kStreamChunks);
}

// Device counters and flags of one build.
struct Counters {
    uint32_t error;         // first mgbvh_status error code, 0 if none
    uint32_t error_site;    // which check failed (for messages)
    uint32_t height;        // max depth of a split node (bvh/src/lib.rs:656)
    uint32_t median_splits;
    uint32_t depth_capped;  // leaves cut by max_depth holding > 1 object
    uint32_t holes;         // leaves holding > 1 object (node slots to compact)
    uint32_t lvl[3][2];     // [level % 3] {large tasks, tiles} of a level pass
    uint32_t n_medium;
    uint32_t n_small;
    uint32_t root_keys[12];  // object bounds lo/hi keys, centroid lo/hi keys
    uint32_t learned;        // nodes where a proposal of the split network replaced the binned split
    uint32_t n_med;          // level-pass nodes waiting for a forced median split (the median passes)
    uint32_t medium_take;    // next subtree CTA task to take (subtree CTAs take tasks in turn)
    uint32_t small_take;     // next small-subtree task to take (warps take tasks in turn)
    uint32_t mtake[8];       // streamed output: the same, per slot chunk (subtree CTA tasks)
    uint32_t stake[8];       // streamed output: the same, per slot chunk (small-subtree tasks)
    // streamed output (slot chunks): subtrees of 33..medium_max objects per
    // chunk, their placement cursors and sorted ranges; subtrees of <= 32
    // objects selected so far, the sorted range of each chunk's, and the CTAs
    // of each chunk's selection pass that finished
    uint32_t mbk[8];
    uint32_t mbcur[8];
    uint32_t mrange[9];
    uint32_t s2n;
    uint32_t srange[9];
    uint32_t sdone[8];
};

enum ErrorSite : uint32_t {
    kSiteNone = 0,
    kSiteIndex = 1,        // a triangle index past the vertex count
    kSiteCount = 2,        // partition count differs from the split's count
    kSiteContain = 3,      // a centroid outside its child's bounds
    kSiteMedian = 4,       // forced median of a level-pass node: counts of its halves differ
    kSiteCapacity = 5,
    kSiteMeshIndex = 6,  // an instance names a mesh past the mesh count
};

__device__ __forceinline__ void set_error(Counters* c, int status, uint32_t site) {
    if (atomicCAS(&c->error, 0u, static_cast<uint32_t>(status)) == 0u) c->error_site = site;
}

// Where a finished node goes. Node slots follow the reference's numbering
// (pre-order over child pairs, gt child first, bvh/src/lib.rs:650-663),
// computed in closed form under the assumption that every leaf holds one
// object: the gt child of a node whose children sit at P has its children at
// P + 2, the lt child at P + 2 * len_gt. Leaves with more objects leave
// unused slots ("holes") that a compaction pass removes afterwards.
struct Out {
    mgbvh_node* nodes;
    uint32_t* lens;
    uint8_t* used;
    uint32_t* perm;
    Counters* ctr;
    uint32_t node_cap;  // slots in nodes/lens/used
};

// The 8 words of a node are written by lanes 0..7 (one 32-byte store), the
// length by lane 8 and the used flag by lane 9. All arguments warp-uniform.
__device__ __forceinline__ void warp_store_node(const Out& o, uint32_t slot, const float* b,
                                                uint32_t start, uint32_t len, uint32_t child,
                                                uint32_t lane) {
    if (slot >= o.node_cap) {  // cannot happen with the closed-form slots; never write past
        if (lane == 0) set_error(o.ctr, MGBVH_ERR_CAPACITY, kSiteCapacity);
        return;
    }
    uint32_t w = 0;
    switch (lane) {
        case 0: w = __float_as_uint(b[0]); break;
        case 1: w = __float_as_uint(b[1]); break;
        case 2: w = __float_as_uint(b[2]); break;
        case 3: w = start; break;
        case 4: w = __float_as_uint(b[3]); break;
        case 5: w = __float_as_uint(b[4]); break;
        case 6: w = __float_as_uint(b[5]); break;
        case 7: w = child; break;
        default: break;
    }
    if (lane < 8) reinterpret_cast<uint32_t*>(o.nodes + slot)[lane] = w;
    if (lane == 8) o.lens[slot] = len;
    if (lane == 9) o.used[slot] = 1;
}

__device__ __forceinline__ void box_empty(float* b) {
    b[0] = b[1] = b[2] = __int_as_float(0x7F800000);
    b[3] = b[4] = b[5] = __int_as_float(0xFF800000);
}

__device__ __forceinline__ void box_grow(float* b, float lx, float ly, float lz, float hx, float hy,
                                         float hz) {
    b[0] = fminf(b[0], lx);
    b[1] = fminf(b[1], ly);
    b[2] = fminf(b[2], lz);
    b[3] = fmaxf(b[3], hx);
    b[4] = fmaxf(b[4], hy);
    b[5] = fmaxf(b[5], hz);
}

__device__ __forceinline__ bool box_contains(const float* b, float x, float y, float z) {
    const bool empty = b[3] < b[0] || b[4] < b[1] || b[5] < b[2];
    return !empty && x >= b[0] && y >= b[1] && z >= b[2] && x <= b[3] && y <= b[4] && z <= b[5];
}

// v[i] for i < 3 with selects: a run-time index into a local array would
// put the array in local memory.
__device__ __forceinline__ float sel3(const float* v, uint32_t i) {
    return i == 0 ? v[0] : (i == 1 ? v[1] : v[2]);
}

// box_contains on box a (first) or box b, chosen with selects on constant
// indexes (a pointer chosen at run time would put both boxes in local memory).
__device__ __forceinline__ bool box_contains2(const float* a, const float* b, bool first, float x, float y,
                                              float z) {
    float bb[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) bb[i] = first ? a[i] : b[i];
    return box_contains(bb, x, y, z);
}

// box_grow on box a (first) or box b, with selects on constant indexes.
__device__ __forceinline__ void box_grow2(float* a, float* b, bool first, float lx, float ly, float lz,
                                          float hx, float hy, float hz) {
    const float l[3] = {lx, ly, lz}, h[3] = {hx, hy, hz};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        a[i] = first ? fminf(a[i], l[i]) : a[i];
        a[3 + i] = first ? fmaxf(a[3 + i], h[i]) : a[3 + i];
        b[i] = first ? b[i] : fminf(b[i], l[i]);
        b[3 + i] = first ? b[3 + i] : fmaxf(b[3 + i], h[i]);
    }
}

// 64-bit candidate key: total_cmp(cost), then axis, then candidate index —
// the first minimum of min_by over axes of min_by over candidates.
__device__ __forceinline__ uint64_t cand_key(float cost, uint32_t axis, uint32_t idx) {
    return (static_cast<uint64_t>(fkey(cost)) << 32) | (axis << 8) | idx;
}

__device__ __forceinline__ bool leaf_rule(uint32_t n, uint32_t depth, const Params& P) {
    return n <= 1u || depth == P.max_depth || (n <= P.max_leaf && n < 2u * P.min_leaf);  // bvh/src/lib.rs:548, 556
}

// Minimum and maximum over the warp (one instruction on sm_100a).
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Warp-wide minimum of 64-bit keys via two 32-bit reductions.
__device__ __forceinline__ uint64_t warp_min_key(uint64_t k) {
    const uint32_t hi = static_cast<uint32_t>(k >> 32), lo = static_cast<uint32_t>(k);
    const uint32_t mh = __reduce_min_sync(kFull, hi);
    const uint32_t ml = __reduce_min_sync(kFull, hi == mh ? lo : kNoKey);
    return (static_cast<uint64_t>(mh) << 32) | ml;
}

// Prefix (inclusive) and suffix (inclusive) unions across lanes of one
// axis's bins: count and box. Lanes at or past `bins` carry empty bins.
struct BinScan {
    uint32_t pre_cnt, suf_cnt;
    float pre[6], suf[6];
};

__device__ __forceinline__ void bin_scan(uint32_t cnt, const float* box, uint32_t lane,
                                         BinScan& s) {
    s.pre_cnt = cnt;
    s.suf_cnt = cnt;
    for (int i = 0; i < 6; ++i) s.pre[i] = s.suf[i] = box[i];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t pc = __shfl_up_sync(kFull, s.pre_cnt, off);
        const uint32_t sc = __shfl_down_sync(kFull, s.suf_cnt, off);
        float pv[6], sv[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            pv[i] = __shfl_up_sync(kFull, s.pre[i], off);
            sv[i] = __shfl_down_sync(kFull, s.suf[i], off);
        }
        if (lane >= static_cast<uint32_t>(off)) {
            s.pre_cnt += pc;
            s.pre[0] = fminf(s.pre[0], pv[0]);
            s.pre[1] = fminf(s.pre[1], pv[1]);
            s.pre[2] = fminf(s.pre[2], pv[2]);
            s.pre[3] = fmaxf(s.pre[3], pv[3]);
            s.pre[4] = fmaxf(s.pre[4], pv[4]);
            s.pre[5] = fmaxf(s.pre[5], pv[5]);
        }
        if (lane + off < 32u) {
            s.suf_cnt += sc;
            s.suf[0] = fminf(s.suf[0], sv[0]);
            s.suf[1] = fminf(s.suf[1], sv[1]);
            s.suf[2] = fminf(s.suf[2], sv[2]);
            s.suf[3] = fmaxf(s.suf[3], sv[3]);
            s.suf[4] = fmaxf(s.suf[4], sv[4]);
            s.suf[5] = fmaxf(s.suf[5], sv[5]);
        }
    }
}

// Best binned candidate held by this lane over the three axes
// (evaluate_binned_split for split index i = lane, bvh/src/lib.rs:255-290,
// 373-388). cnt/box: this lane's bin (lane = bin index) per axis.
struct Cand {
    uint64_t key;
    uint32_t n_lt;
    float lt[6], gt[6];
    float thr;  // adaptive threshold (unused for binned)
};

// load(a, cnt, box6): this lane's bin on axis a.
template <class Load>
__device__ __forceinline__ void binned_candidates_f(Load load, const bool* axis_ok, uint32_t bins,
                                                    uint32_t n, float sa_p, const Params& P,
                                                    uint32_t lane, Cand& best) {
    best.key = ~0ull;
#pragma unroll 1
    for (uint32_t a = 0; a < 3; ++a) {
        // selects, not a run-time index: axis_ok stays in registers
        const bool ok = a == 0 ? axis_ok[0] : (a == 1 ? axis_ok[1] : axis_ok[2]);
        if (!ok) continue;  // warp-uniform
        uint32_t ca;
        float ba[6];
        load(a, ca, ba);
        BinScan s;
        bin_scan(ca, ba, lane, s);
        // lt of candidate i = prefix through bin i-1
        uint32_t lt_cnt = __shfl_up_sync(kFull, s.pre_cnt, 1);
        float lt[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) lt[i] = __shfl_up_sync(kFull, s.pre[i], 1);
        if (lane >= 1 && lane < bins) {
            const uint32_t gt_cnt = s.suf_cnt;
            const float cost =
                split_cost(surface_area6(lt), surface_area6(s.suf), sa_p, lt_cnt, gt_cnt);
            (void)n;
            if (lt_cnt >= P.min_leaf && gt_cnt >= P.min_leaf) {
                const uint64_t k = cand_key(cost, a, lane);
                if (k < best.key) {
                    best.key = k;
                    best.n_lt = lt_cnt;
                    for (int i = 0; i < 6; ++i) {
                        best.lt[i] = lt[i];
                        best.gt[i] = s.suf[i];
                    }
                    best.thr = 0.0f;
                }
            }
        }
    }
}

// The bins held in registers per axis (read by selects: run-time indexes
// into cnt and box would put them in local memory).
__device__ __forceinline__ void binned_candidates(const uint32_t* cnt, const float (*box)[6],
                                                  const bool* axis_ok, uint32_t bins, uint32_t n,
                                                  float sa_p, const Params& P, uint32_t lane,
                                                  Cand& best) {
    binned_candidates_f(
        [&](uint32_t a, uint32_t& ca, float* ba) {
            ca = a == 0 ? cnt[0] : (a == 1 ? cnt[1] : cnt[2]);
#pragma unroll
            for (int i = 0; i < 6; ++i) ba[i] = a == 0 ? box[0][i] : (a == 1 ? box[1][i] : box[2][i]);
        },
        axis_ok, bins, n, sa_p, P, lane, best);
}

// Pull a candidate's payload from lane `src` to all lanes.
__device__ __forceinline__ void shfl_cand(Cand& c, uint32_t src) {
    c.n_lt = __shfl_sync(kFull, c.n_lt, src);
    c.thr = __shfl_sync(kFull, c.thr, src);
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        c.lt[i] = __shfl_sync(kFull, c.lt[i], src);
        c.gt[i] = __shfl_sync(kFull, c.gt[i], src);
    }
}

// Centroid bounds of the lt and gt objects a lane has placed, and whether one
// of them was NaN (which no bounds contain).
struct SideBounds {
    float lt[6], gt[6];  // min xyz, max xyz
    bool nan;

    __device__ __forceinline__ SideBounds() : nan(false) {
        box_empty(lt);
        box_empty(gt);
    }
    __device__ __forceinline__ void add(bool first, const float* c) {
        nan |= c[0] != c[0] || c[1] != c[1] || c[2] != c[2];
        if (first)
            box_grow(lt, c[0], c[1], c[2], c[0], c[1], c[2]);
        else
            box_grow(gt, c[0], c[1], c[2], c[0], c[1], c[2]);
    }
};

// Bin index of a centroid on one axis of a node, as bin_of gives it. Instead of
// the divide, the centroid is scaled by bins / ext; the exact form runs only
// where the scaled value lies within 2^-14 of an integer (the two differ by
// less than 2^-16: a few roundings of a value below 32), or on axes whose
// extent or position is extreme.
struct BinMap {
    float cmin, ext, cmin2, scale, top;
    uint32_t bins;
    bool fast, ok;  // ok: the axis has an extent (bvh/src/lib.rs:339)

    __device__ __forceinline__ BinMap() {}
    __device__ __forceinline__ BinMap(float cmn, float cmx, uint32_t n_bins) {
        cmin = cmn;
        ext = __fsub_rn(cmx, cmn);
        bins = n_bins;
        ok = !(ext == 0.0f);
        fast = ext >= 7.888609052210118e-31f && ext <= 1.2676506002282294e30f && fabsf(cmn) <= 8.507059173023462e37f;
        cmin2 = __fadd_rn(cmn, cmn);
        const float b = __uint2float_rn(n_bins);
        scale = __fdividef(__fmul_rn(b, 0.5f), ext);
        top = __fsub_rn(b, 0.6f);
    }
    __device__ __forceinline__ uint32_t operator()(float lo, float hi) const {
        // t = scaled value - 0.5 rounds to the integer below the scaled value;
        // both ends of the range are clamped to a value inside their bin
        float t = __fmaf_rn(__fsub_rn(__fadd_rn(lo, hi), cmin2), scale, -0.5f);
        t = fminf(fmaxf(t, -0.4f), top);
        const float u = __fadd_rn(t, 12582912.0f);  // 1.5 * 2^23: the integer in the low bits
        const float off = __fsub_rn(t, __fsub_rn(u, 12582912.0f));
        uint32_t b = __float_as_uint(u) & 31u;
        if (!fast || fabsf(off) > 0.49993896484375f) b = bin_of(center_of(lo, hi), cmin, ext, bins);
        return b;
    }
};

// Box coordinates as keys for which a larger key is the union: zero is below
// every key, so cleared bins are empty. Lower bounds: ~fkey; both are two
// operations each way.
__device__ __forceinline__ uint32_t key_lo(float f) {
    const int u = __float_as_int(f);
    return static_cast<uint32_t>(u ^ (~(u >> 31) & 0x7FFFFFFF));
}
__device__ __forceinline__ uint32_t key_hi(float f) {
    const int u = __float_as_int(f);
    return static_cast<uint32_t>(u) ^ (static_cast<uint32_t>(u >> 31) | 0x80000000u);
}
__device__ __forceinline__ float unkey_lo(uint32_t k) {
    const int u = static_cast<int>(k);
    return __int_as_float(u ^ (~(u >> 31) & 0x7FFFFFFF));
}
__device__ __forceinline__ float unkey_hi(uint32_t k) {
    const int u = static_cast<int>(k);
    return __uint_as_float(k ^ (static_cast<uint32_t>(~(u >> 31)) | 0x80000000u));
}

// A node's bins in shared memory: [axis][bin]{count, key_lo xyz, key_hi xyz},
// cleared to zero; 7 more words after each axis put the 18 sequences of one
// bin in different banks.
constexpr uint32_t kSweepAxis = 32u * 7u + 7u;
constexpr uint32_t kSweepWords = 3u * kSweepAxis;

__device__ __forceinline__ void clear_bins(uint32_t* wb, uint32_t tid, uint32_t nthreads) {
    for (uint32_t w = tid; w < kSweepWords; w += nthreads) wb[w] = 0u;
}

// Adds an object to its bins; returns the bins (5 bits per axis). On the axes in
// `dense` a box key goes to its bin only where it extends the bin as read
// before: lanes that share a bin read it at once, while their atomics on one
// word take turns.
__device__ __forceinline__ uint32_t add_to_bins(uint32_t* wb, const BinMap* map, const float4& lo, const float4& hi,
                                                uint32_t dense = 0) {
    const uint32_t k[6] = {key_lo(lo.x), key_lo(lo.y), key_lo(lo.z), key_hi(hi.x), key_hi(hi.y), key_hi(hi.z)};
    const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
    uint32_t code = 0;
#pragma unroll
    for (uint32_t a = 0; a < 3; ++a) {
        if (!map[a].ok) continue;  // the same for every object of the node
        const uint32_t b = map[a](l[a], h[a]);
        code |= b << (5u * a);
        uint32_t* w = wb + a * kSweepAxis + b * 7u;
        atomicAdd(w, 1u);
        if ((dense >> a) & 1u) {
            bool more[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) more[i] = k[i] > *reinterpret_cast<volatile uint32_t*>(w + 1 + i);
#pragma unroll
            for (int i = 0; i < 6; ++i)
                if (more[i]) atomicMax(w + 1 + i, k[i]);
        } else {
#pragma unroll
            for (int i = 0; i < 6; ++i) atomicMax(w + 1 + i, k[i]);
        }
    }
    return code;
}

// The axes (bits 0..2) on which at least kDenseLanes lanes' objects fall in
// lane 0's bin. All lanes take part; lane 0 has an object.
constexpr uint32_t kDenseLanes = 8;
__device__ __forceinline__ uint32_t shared_bins(const BinMap* map, const float4& lo, const float4& hi, bool valid) {
    const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
    uint32_t dense = 0;
#pragma unroll
    for (uint32_t a = 0; a < 3; ++a) {
        const uint32_t b = valid ? map[a](l[a], h[a]) : kMaxBins;
        const uint32_t same = __ballot_sync(kFull, b == __shfl_sync(kFull, b, 0));
        dense |= __popc(same) >= kDenseLanes ? 1u << a : 0u;
    }
    return dense;
}

struct SweepResult {
    bool found;
    uint32_t axis, bin, n_lt, cost;  // cost: its bits
    float lt[6], gt[6];
    uint32_t cnt[3];  // objects of bin `lane` on each axis
};

// One warp: the best binned split of a node of n objects whose bins are wb
// (evaluate_binned_split over every split index and axis, bvh/src/lib.rs:
// 255-290, 331-389; first minimum of cost, axis, index). Destroys the boxes
// in wb, not the counts.
//
// The prefix and suffix unions of the 3 x 6 coordinate sequences run
// sequentially, one lane per sequence with its 32 bins in registers, and pass
// through wb to the lanes that hold the candidates (lane = split index): 3 x 32
// shared-memory accesses and 62 maxima, where shuffle scans of every lane's
// bins take 5 steps of 2 x 7 shuffles per axis.
__device__ __forceinline__ SweepResult sweep_bins(uint32_t* wb, const BinMap* map, uint32_t n, const NodeArea& area,
                                                  const Params& P, uint32_t lane) {
    SweepResult r;
    uint32_t* const seq = wb + (lane < 18u ? (lane / 6u) * kSweepAxis + 1u + lane % 6u : 0u);
    uint32_t v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = seq[7 * j];
#pragma unroll
    for (int a = 0; a < 3; ++a) r.cnt[a] = wb[a * kSweepAxis + 7u * lane];
    __syncwarp();
    // objects in the bins below the lane's, per axis
    uint32_t below01 = r.cnt[0] | (r.cnt[1] << 16), below2 = r.cnt[2];
#pragma unroll
    for (uint32_t d = 1; d < 32u; d <<= 1) {
        const uint32_t u = __shfl_up_sync(kFull, below01, d), w = __shfl_up_sync(kFull, below2, d);
        if (lane >= d) {
            below01 += u;
            below2 += w;
        }
    }
    below01 -= r.cnt[0] | (r.cnt[1] << 16);
    below2 -= r.cnt[2];
    if (lane < 18u) {
        uint32_t run = v[0];
#pragma unroll
        for (int j = 1; j < 32; ++j) {
            seq[7 * j] = run;
            run = max(run, v[j]);
        }
    }
    __syncwarp();
    float sa_lt[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const uint32_t* w = wb + a * kSweepAxis + 7u * lane + 1u;
        sa_lt[a] = surface_area(unkey_lo(w[0]), unkey_lo(w[1]), unkey_lo(w[2]), unkey_hi(w[3]), unkey_hi(w[4]),
                                unkey_hi(w[5]));
    }
    __syncwarp();
    if (lane < 18u) {
        uint32_t run = v[31];
#pragma unroll
        for (int j = 31; j > 0; --j) {
            seq[7 * j] = run;
            run = max(run, v[j - 1]);
        }
    }
    __syncwarp();
    uint32_t best = kNoKey, axis = 3;
#pragma unroll
    for (uint32_t a = 0; a < 3; ++a) {
        const uint32_t nl = a == 0 ? below01 & 0xFFFFu : (a == 1 ? below01 >> 16 : below2), ng = n - nl;
        const uint32_t* w = wb + a * kSweepAxis + 7u * lane + 1u;
        const float sa_gt = surface_area(unkey_lo(w[0]), unkey_lo(w[1]), unkey_lo(w[2]), unkey_hi(w[3]),
                                         unkey_hi(w[4]), unkey_hi(w[5]));
        if (map[a].ok && lane >= 1u && lane < map[a].bins && nl >= P.min_leaf && ng >= P.min_leaf) {
            // (never negative: the bits order as the costs do)
            const uint32_t ck = __float_as_uint(area.split_cost(sa_lt[a], sa_gt, nl, ng));
            if (ck < best) {
                best = ck;
                axis = a;
            }
        }
    }
    r.cost = __reduce_min_sync(kFull, best);
    r.found = r.cost != kNoKey;
    const uint32_t w0 = __ballot_sync(kFull, best == r.cost && axis == 0u),
                   w1 = __ballot_sync(kFull, best == r.cost && axis == 1u),
                   w2 = __ballot_sync(kFull, best == r.cost && axis == 2u);
    r.axis = w0 ? 0u : (w1 ? 1u : 2u);
    r.bin = r.found ? __ffs(w0 ? w0 : (w1 ? w1 : w2)) - 1u : 1u;
    const uint32_t nl = r.axis == 0 ? below01 & 0xFFFFu : (r.axis == 1 ? below01 >> 16 : below2);
    r.n_lt = __shfl_sync(kFull, nl, r.bin);
    const uint32_t* w = wb + r.axis * kSweepAxis + 7u * r.bin + 1u;
    uint32_t run = v[0];
#pragma unroll
    for (uint32_t j = 1; j < 32u; ++j) run = j < r.bin ? max(run, v[j]) : run;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const uint32_t l = __shfl_sync(kFull, run, r.axis * 6u + i);
        r.lt[i] = i < 3 ? unkey_lo(l) : unkey_hi(l);
        r.gt[i] = i < 3 ? unkey_lo(w[i]) : unkey_hi(w[i]);
    }
    __syncwarp();
    return r;
}

// Segmented reductions over contiguous lane ranges [s, end): shuffle-down
// tree bounded by the segment end, then a broadcast from the segment's first
// lane; maxn (warp-uniform) is the longest segment, past which no step adds
// anything. Every lane takes part with full masks (per-segment masks in one
// warp serialize: one pass per distinct mask).
__device__ __forceinline__ uint32_t seg_min(uint32_t v, uint32_t lane, uint32_t s, uint32_t end, uint32_t maxn) {
    for (uint32_t d = 1; d < maxn; d <<= 1) {
        const uint32_t u = __shfl_down_sync(kFull, v, d);
        if (lane + d < end) v = min(v, u);
    }
    return __shfl_sync(kFull, v, s);
}

__device__ __forceinline__ uint32_t seg_max(uint32_t v, uint32_t lane, uint32_t s, uint32_t end, uint32_t maxn) {
    for (uint32_t d = 1; d < maxn; d <<= 1) {
        const uint32_t u = __shfl_down_sync(kFull, v, d);
        if (lane + d < end) v = max(v, u);
    }
    return __shfl_sync(kFull, v, s);
}

// Lexicographic (hi, lo) minimum over the segment.
__device__ __forceinline__ void seg_min2(uint32_t& hi, uint32_t& lo, uint32_t lane, uint32_t s, uint32_t end,
                                         uint32_t maxn) {
    for (uint32_t d = 1; d < maxn; d <<= 1) {
        const uint32_t uh = __shfl_down_sync(kFull, hi, d);
        const uint32_t ul = __shfl_down_sync(kFull, lo, d);
        if (lane + d < end && (uh < hi || (uh == hi && ul < lo))) {
            hi = uh;
            lo = ul;
        }
    }
    hi = __shfl_sync(kFull, hi, s);
    lo = __shfl_sync(kFull, lo, s);
}

// Programmatic dependent launch: a kernel launched with programmatic stream
// serialization may be scheduled while its predecessor in the stream is
// still finishing. griddepcontrol.wait blocks until the predecessor grid has
// completed and its memory operations are visible (a no-op for an ordinary
// launch); the kernel then lets its own dependent grid be scheduled. Called
// first in every kernel of the build pipeline, before any read of a
// predecessor's output.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Lanes [s, s+n) as a mask.
__device__ __forceinline__ uint32_t seg_mask(uint32_t s, uint32_t n) {
    return n >= 32u ? kFull : (((1u << n) - 1u) << s);
}

// Writes one node from a single lane (two 16-byte stores).
__device__ __forceinline__ void lane_store_node(const Out& o, uint32_t slot, const float* b,
                                                uint32_t start, uint32_t len, uint32_t child) {
    if (slot >= o.node_cap) {
        set_error(o.ctr, MGBVH_ERR_CAPACITY, kSiteCapacity);
        return;
    }
    float4* p = reinterpret_cast<float4*>(o.nodes + slot);
    p[0] = make_float4(b[0], b[1], b[2], __uint_as_float(start));
    p[1] = make_float4(b[3], b[4], b[5], __uint_as_float(child));
    o.lens[slot] = len;
    o.used[slot] = 1;
}

// A warp's tables of one subtree of n0 <= 32 objects.
//
// Every object set the builder looks at is a set of the subtree's n0 objects,
// kept as masks over nine orders: for each of the six box coordinates, bit b
// stands for the object at place b of that coordinate's order (its lower
// bounds descending, its upper bounds ascending), so the union box's
// coordinate is the value at the mask's highest bit, which lane b holds: one
// find-leading-one and one shuffle instead of a min/max over the set. Orders
// 6..8 are the centroids' on each axis, ascending. The objects left of a
// threshold on axis a are the first m of its order, for whatever node of the
// subtree: pm[a][q][m - 1] holds them as bits of order q, made once, and a
// node's left side is that mask and the node's own.
constexpr uint32_t kOrders = 9;

struct alignas(16) SubtreeSmem {
    uint32_t head[32];  // (reads for m = 0, whose value is not used, fall here)
    uint32_t pm[3][kOrders][32];  // 32 words a plane: lanes with different m read different banks
    uint32_t rt[32];   // by place on axis 0: the object's bit in each coordinate's order (5 bits each)
    uint32_t ids[32];  // by place on axis 0: the object's id
    uint32_t x[32];    // exchange space
};

// What a lane holds of the tables: coordinate q's value at bit `lane`, and the
// centroid on axis a at place `lane` of its order (NaN past the last).
struct SubtreeRegs {
    float val[6], cen[3];
};

// Highest set bit of a mask; -1 for an empty one (a shuffle reads lane 31
// then, and the value is not used).
__device__ __forceinline__ int top_bit(uint32_t m) {
    int r;
    asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(m));
    return r;
}

// Split profiles other than the reference's own (every node of <= 32 objects
// adaptive, with one threshold per object: steps = len.clamp(8,32) = len for
// 8 <= len <= 32, one centroid per object below 8; bvh/src/lib.rs:417-437).
__host__ __device__ __forceinline__ bool subtree_general(const Params& P) {
    return P.adaptive_steps != 0u || P.adaptive_max_n != kSmallMax;
}

// Fills T for the objects of lanes 0 .. n0-1 (lo, hi, id; 2 <= n0 <= 32) and
// returns this lane's object word: its place on axis a at bits 5a, and the
// number of objects with a lower centroid on a at bits 15 + 5a.
__device__ __forceinline__ uint32_t subtree_tables(const float* lo, const float* hi, uint32_t id, uint32_t n0,
                                                   uint32_t lane, SubtreeSmem& T, SubtreeRegs& R) {
    static_assert(sizeof(T.pm) >= 32 * 48 + 9 * 128, "the sort space fits in the prefix masks' space");
    const uint32_t below = (1u << lane) - 1u;
    // sort keys: NaN coordinates rank where fminf / fmaxf ignore them, NaN
    // centroids last
    float v[9], c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        c[a] = center_of(lo[a], hi[a]);
        v[a] = fminf(lo[a], __int_as_float(0x7F800000));
        v[3 + a] = fmaxf(hi[a], __int_as_float(0xFF800000));
        v[6 + a] = fminf(c[a], __int_as_float(0x7F800000));
    }
    float4* keys = reinterpret_cast<float4*>(&T.pm[0][0][0]);
    uint32_t* sp = &T.pm[0][0][0] + 32 * 12;  // 9 x 32 words
    keys[3 * lane] = make_float4(v[0], v[1], v[2], v[3]);
    keys[3 * lane + 1] = make_float4(v[4], v[5], v[6], v[7]);
    keys[3 * lane + 2] = make_float4(v[8], 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (uint32_t q = 0; q < 9; ++q) sp[32u * q + lane] = 0u;
    __syncwarp();
    uint32_t r[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) r[q] = 0;
#pragma unroll 4
    for (uint32_t j = 0; j < n0; ++j) {  // one address per step: broadcast loads
        const float4 k0 = keys[3 * j], k1 = keys[3 * j + 1];
        const float k2 = keys[3 * j + 2].x;
        r[0] += k0.x < v[0] ? 1u : 0u;
        r[1] += k0.y < v[1] ? 1u : 0u;
        r[2] += k0.z < v[2] ? 1u : 0u;
        r[3] += k0.w < v[3] ? 1u : 0u;
        r[4] += k1.x < v[4] ? 1u : 0u;
        r[5] += k1.y < v[5] ? 1u : 0u;
        r[6] += k1.z < v[6] ? 1u : 0u;
        r[7] += k1.w < v[7] ? 1u : 0u;
        r[8] += k2 < v[8] ? 1u : 0u;
    }
    // equal keys take consecutive places in lane order
    const bool mine = lane < n0;
    if (mine) {
#pragma unroll
        for (uint32_t q = 0; q < 9; ++q) atomicOr(&sp[32u * q + r[q]], 1u << lane);
    }
    __syncwarp();
    uint32_t word = 0, bits = 0, place[9];
#pragma unroll
    for (uint32_t q = 0; q < 9; ++q) place[q] = r[q] + (mine ? __popc(sp[32u * q + r[q]] & below) : 0u);
    __syncwarp();
    float* rows = reinterpret_cast<float*>(sp);
    if (mine) {
#pragma unroll
        for (uint32_t q = 0; q < 6; ++q) {
            const uint32_t b = q < 3 ? 31u - place[q] : place[q];
            rows[32u * q + b] = v[q];
            bits |= b << (5u * q);
        }
#pragma unroll
        for (uint32_t a = 0; a < 3; ++a) {
            rows[32u * (6u + a) + place[6 + a]] = c[a];
            // (a NaN centroid is below no threshold and no threshold itself)
            word |= place[6 + a] << (5u * a) | (c[a] == c[a] ? r[6 + a] : 0u) << (15u + 5u * a);
        }
        T.rt[place[6]] = bits;
        T.ids[place[6]] = id;
    } else {
#pragma unroll
        for (uint32_t a = 0; a < 3; ++a) rows[32u * (6u + a) + lane] = __int_as_float(0x7FFFFFFF);
    }
    __syncwarp();
#pragma unroll
    for (uint32_t q = 0; q < 6; ++q) R.val[q] = rows[32u * q + lane];
#pragma unroll
    for (uint32_t a = 0; a < 3; ++a) R.cen[a] = rows[32u * (6u + a) + lane];
    // prefix masks: lane p takes the object at place p of the axis's order
    uint32_t* xw = &T.pm[0][0][0];  // the keys' space: bits and words by place
#pragma unroll
    for (uint32_t a = 0; a < 3; ++a) {
        if (mine) {
            xw[64u * a + place[6 + a]] = bits;
            xw[64u * a + 32u + place[6 + a]] = word;
        }
    }
    __syncwarp();
    uint32_t pb[3], pw[3];
#pragma unroll
    for (uint32_t a = 0; a < 3; ++a) {
        pb[a] = xw[64u * a + lane];
        pw[a] = xw[64u * a + 32u + lane];
    }
    __syncwarp();
#pragma unroll
    for (uint32_t a = 0; a < 3; ++a) {
        uint32_t w[kOrders];
#pragma unroll
        for (uint32_t q = 0; q < kOrders; ++q) {
            const uint32_t b = q < 6 ? pb[a] >> (5u * q) : pw[a] >> (5u * (q - 6u));
            w[q] = mine ? 1u << (b & 31u) : 0u;
        }
#pragma unroll
        for (uint32_t d = 1; d < 32u; d <<= 1) {
#pragma unroll
            for (uint32_t q = 0; q < kOrders; ++q) {
                if (q == 6u + a) continue;
                const uint32_t u = __shfl_up_sync(kFull, w[q], d);
                if (lane >= d) w[q] |= u;
            }
        }
        w[6 + a] = mine ? below | (1u << lane) : (1u << n0) - 1u;  // the axis's own order
#pragma unroll
        for (uint32_t q = 0; q < kOrders; ++q) {
            T.pm[a][q][lane] = w[q];
        }
    }
    __syncwarp();
    return word;
}

// The candidate of an object (place `place`, centroid c, predecessor's
// centroid prev) on an axis of a node that takes evenly spaced thresholds
// (n >= 8 adaptive) or bins: the split whose gt side starts at this object in
// the node's centroid order, with the lowest threshold or bin index that makes
// this split. False when no threshold falls between the object and its
// predecessor. The sets {c < threshold i} and {bin < i} are prefixes of the
// centroid order (threshold and bin are monotone), so these are all the
// different splits of the sweep, each with its first index.
__device__ __forceinline__ bool ordered_candidate(float c, float prev, float cmin, float cmax, uint32_t n,
                                                  bool adaptive, const Params& P, uint32_t& idx) {
    const float ext = __fsub_rn(cmax, cmin);
    if (adaptive) {  // bvh/src/lib.rs:428-441: the first threshold above prev, if not above c
        const uint32_t steps = P.adaptive_steps ? P.adaptive_steps : n;
        const float step = __fdiv_rn(ext, __uint2float_rn(steps));
        uint32_t lo = 0, hi = steps;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (prev < adaptive_threshold(cmin, step, mid))
                hi = mid;
            else
                lo = mid + 1u;
        }
        idx = lo;
        return lo < steps && !(c < adaptive_threshold(cmin, step, lo));
    }
    if (ext == 0.0f) return false;  // bvh/src/lib.rs:339
    const uint32_t bins = P.bins ? P.bins : min(max(n, 16u), 32u);
    const uint32_t b = bin_of(prev, cmin, ext, bins);
    idx = b + 1u;
    return b < bin_of(c, cmin, ext, bins);
}

struct MedianIo {
    SubtreeRegs regs;
    float nb[6];             // in: the node's box; out: the lane's half's
    uint32_t node[kOrders];  // out: the lane's half as masks
    uint32_t word;           // in and out: the lane's object
};

// median_split (bvh/src/lib.rs:444-491, 528-530) of the segments whose lanes
// have `odd`: on axes 0, 1, 2 in turn over the same list, stable; the halves
// are those of the final (axis-2) order, their boxes the cheapest axis's. All
// lanes take part. Rare: nodes that no threshold or bin tells apart.
__device__ __forceinline__ void median_segments(bool odd, uint32_t s, uint32_t n, uint32_t m, uint32_t ss, uint32_t se,
                                             uint32_t maxn, SubtreeSmem& T, MedianIo& io) {
    const SubtreeRegs R = io.regs;
    const NodeArea area(io.nb);
    uint32_t word = io.word;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t half = n / 2u;
    float wb[6];
    uint32_t best_ck = 0;
#pragma unroll 1
    for (uint32_t a = 0; a < 3; ++a) {
        const float cen = a == 0 ? R.cen[0] : (a == 1 ? R.cen[1] : R.cen[2]);
        const uint32_t key = fkey(__shfl_sync(kFull, cen, (word >> (5u * a)) & 31u));
        uint32_t rank = 0;
        for (uint32_t r = 0; r < maxn; ++r) {
            const bool use = odd && r < n;
            const uint32_t kj = __shfl_sync(kFull, key, use ? s + r : lane);
            if (use) rank += (kj < key || (kj == key && s + r < lane)) ? 1u : 0u;
        }
        const uint32_t lm = __ballot_sync(kFull, odd && rank < half) & m;
        T.x[odd ? (rank < half ? s + __popc(lm & below) : s + half + __popc(m & ~lm & below)) : lane] = word;
        __syncwarp();
        word = T.x[lane];
        __syncwarp();
        const uint32_t bits = T.rt[word & 31u];
        const bool in_lt = odd && lane < s + half, in_gt = odd && lane >= s + half;
        float l6[6], g6[6];
#pragma unroll
        for (uint32_t i = 0; i < 6; ++i) {
            const uint32_t k = fkey(__shfl_sync(kFull, R.val[i], (bits >> (5u * i)) & 31u));
            if (i < 3) {
                l6[i] = funkey(seg_min(in_lt ? k : kKeyPosInf, lane, ss, se, maxn));
                g6[i] = funkey(seg_min(in_gt ? k : kKeyPosInf, lane, ss, se, maxn));
            } else {
                l6[i] = funkey(seg_max(in_lt ? k : kKeyNegInf, lane, ss, se, maxn));
                g6[i] = funkey(seg_max(in_gt ? k : kKeyNegInf, lane, ss, se, maxn));
            }
        }
        const uint32_t ck = fkey(area.split_cost(surface_area6(l6), surface_area6(g6), half, n - half));
        if (a == 0u || ck < best_ck) {
            best_ck = ck;
#pragma unroll
            for (int i = 0; i < 6; ++i) wb[i] = in_lt ? l6[i] : g6[i];
        }
    }
    const uint32_t bits = T.rt[word & 31u];
    uint32_t hm[kOrders];
#pragma unroll
    for (uint32_t q = 0; q < kOrders; ++q) hm[q] = 0;
    for (uint32_t r = 0; r < maxn; ++r) {
        const uint32_t src = odd && r < n ? s + r : lane;
        const uint32_t bj = __shfl_sync(kFull, bits, src), wj = __shfl_sync(kFull, word, src);
        if (odd && r < n && (r < half) == (lane < s + half)) {
#pragma unroll
            for (uint32_t q = 0; q < kOrders; ++q)
                hm[q] |= 1u << ((q < 6u ? bj >> (5u * q) : wj >> (5u * (q - 6u))) & 31u);
        }
    }
    io.word = word;
#pragma unroll
    for (uint32_t q = 0; q < kOrders; ++q) io.node[q] = hm[q];
#pragma unroll
    for (int i = 0; i < 6; ++i) io.nb[i] = wb[i];
}

// Builds the subtree rooted at a node of n0 <= 32 objects. Lane i < n0 holds
// object i of the node's range (starting at global position `base`). Writes
// every node of the subtree and the permutation entries of its range.
// kGeneral: any split profile (subtree_general).
//
// Every node of one depth is evaluated at the same time, each on its own lane
// range (segment): a lane holds the candidate of its object or threshold on
// each axis, with both sides' boxes read from the tables (SubtreeSmem).
// What bounds it: issued instructions (75-80% of the issue slots). A merge of
// every object into every candidate, O(n^2) per node, took 465M warp
// instructions on the level-8 icosphere's 59,272 subtrees (22 objects, 5.1
// depths each): 0.544 ms. With the orders sorted once per subtree (about 1,500
// instructions) and 36 mask-and-shuffle reads per lane and depth (700-900
// instructions a depth) it is 321M: 0.386 ms. The general profiles use the same
// tables in place of a depth-first form with one node at a time: 65,536 random
// triangles at 16 bins, 0.325 -> 0.047 ms; 16.8M mixed triangles, 8.3 -> 5.3 ms.
template <bool kGeneral>
__device__ void warp_build_subtree(const float* lo, const float* hi, uint32_t id, uint32_t n0, uint32_t base,
                                   uint32_t slot0, uint32_t pair0, uint32_t depth0, uint32_t nbase, uint32_t tbase,
                                   const float* bounds0, const Params& P, const Out& O, SubtreeSmem& T) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t below = (1u << lane) - 1u;
    if (leaf_rule(n0, depth0, P)) {  // warp-uniform; the queued roots split
        if (lane == 0) {
            lane_store_node(O, nbase + slot0, bounds0, base - tbase, n0, 0u);
            if (n0 > 1u) {
                atomicAdd(&O.ctr->holes, 1u);
                if (depth0 == P.max_depth) atomicAdd(&O.ctr->depth_capped, 1u);
            }
        }
        if (lane < n0) O.perm[base + lane] = id;
        return;
    }
    __syncwarp();  // the previous subtree's table reads are done
    SubtreeRegs R;
    uint32_t word = subtree_tables(lo, hi, id, n0, lane, T, R);
    uint32_t s = 0, n = n0, slot = slot0, pair = pair0, depth = depth0;
    bool live = lane < n0;
    uint32_t node[kOrders];  // the segment's objects as a mask of each order
#pragma unroll
    for (uint32_t q = 0; q < kOrders; ++q) node[q] = live ? T.pm[0][q][31] : 0u;
    float nb[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) nb[i] = bounds0[i];
    uint32_t hmax = 0, n_median = 0, n_holes = 0, n_capped = 0;
    if (lane == 0) lane_store_node(O, nbase + slot, nb, base - tbase, n, pair);

    while (__any_sync(kFull, live)) {
        const uint32_t m = live ? seg_mask(s, n) : (1u << lane);
        const uint32_t ss = live ? s : lane, se = live ? s + n : lane + 1u;  // reduction range
        const uint32_t maxn = __reduce_max_sync(kFull, live ? n : 0u);
        const NodeArea area(nb);
        // this lane's candidate per axis: the lt side's size in the axis's
        // order. Below 8 objects every object's own centroid is a threshold
        uint32_t cut[3], idx[3] = {lane, lane, lane};
        bool ok[3] = {live, live, live};
#pragma unroll
        for (int a = 0; a < 3; ++a) cut[a] = (word >> (15 + 5 * a)) & 31u;
        if constexpr (kGeneral) {
            const bool adaptive = n <= P.adaptive_max_n;
            const bool ordered = live && !(adaptive && n < 8u);
            if (__any_sync(kFull, ordered)) {
#pragma unroll
                for (uint32_t a = 0; a < 3; ++a) {
                    const uint32_t place = (word >> (5u * a)) & 31u;
                    const uint32_t before = node[6 + a] & ((1u << place) - 1u);
                    const float c = __shfl_sync(kFull, R.cen[a], place);
                    const float prev = __shfl_sync(kFull, R.cen[a], top_bit(before));
                    const float cmin = __shfl_sync(kFull, R.cen[a], __ffs(node[6 + a]) - 1);
                    const float cmax = __shfl_sync(kFull, R.cen[a], top_bit(node[6 + a]));
                    if (ordered) {
                        cut[a] = place;
                        ok[a] = before != 0u && ordered_candidate(c, prev, cmin, cmax, n, adaptive, P, idx[a]);
                    }
                }
            }
        } else if (maxn >= 8u) {
            // adaptive steps over the segment's centroid bounds
            // (bvh/src/lib.rs:428-441, 499-509), one threshold per lane; the
            // lt side's size by binary search in the axis's order
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float cmin = __shfl_sync(kFull, R.cen[a], __ffs(node[6 + a]) - 1);
                const float cmax = __shfl_sync(kFull, R.cen[a], top_bit(node[6 + a]));
                // (1: lanes of other nodes, whose step is not used)
                const float ext = live && n >= 8u ? __fsub_rn(cmax, cmin) : 1.0f;
                const float step = __fdiv_rn(ext, __uint2float_rn(n));
                const float thr = adaptive_threshold(cmin, step, lane - s);
                uint32_t p = 0;
#pragma unroll
                for (uint32_t h = 16; h > 0; h >>= 1)
                    if (__shfl_sync(kFull, R.cen[a], p + h - 1u) < thr) p += h;
                if (__shfl_sync(kFull, R.cen[a], p) < thr) ++p;
                if (n >= 8u) cut[a] = p;
            }
        }
        // costs are never negative (ordered_cost): their bits order as they do,
        // all below "none"
        uint32_t best = kNoKey, win = 0;
#pragma unroll
        for (uint32_t a = 0; a < 3; ++a) {
            float lb[6], gb[6];
            uint32_t nl = 0;
#pragma unroll
            for (uint32_t q = 0; q < 6; ++q) {
                const uint32_t pre = (&T.pm[a][q][0])[static_cast<int>(cut[a]) - 1];
                if (q == 0) nl = __popc(pre & node[0]);
                lb[q] = __shfl_sync(kFull, R.val[q], top_bit(pre & node[q]));
                gb[q] = __shfl_sync(kFull, R.val[q], top_bit(~pre & node[q]));
            }
            const uint32_t ng = n - nl;
            if (ok[a] && cut[a] && nl >= P.min_leaf && ng >= P.min_leaf) {  // :407
                const uint32_t ck = __float_as_uint(area.split_cost(surface_area6(lb), surface_area6(gb), nl, ng));
                if (ck < best) {
                    best = ck;
                    win = (a << 8) | idx[a];
                }
            }
        }
        // first minimum of (cost, axis, index) in the segment: axis, and the
        // lane that holds it
        uint32_t axis, src;
        if constexpr (kGeneral) {
            win = (win << 8) | lane;  // one object per index: the lane breaks no tie
            seg_min2(best, win, lane, ss, se, maxn);
            axis = win >> 16;
            src = win & 31u;
        } else {
            // indexes follow the lanes: the first lane of the lowest axis
            const uint32_t own = best;
            if (maxn == n0) {  // one segment
                best = __reduce_min_sync(kFull, best);
            } else {
                for (uint32_t d = 1; d < maxn; d <<= 1) {
                    const uint32_t u = __shfl_down_sync(kFull, best, d);
                    if (lane + d < se) best = min(best, u);
                }
                best = __shfl_sync(kFull, best, ss);
            }
            const uint32_t w0 = __ballot_sync(kFull, own == best && win < 256u) & m,
                           w1 = __ballot_sync(kFull, own == best && win < 512u) & m,
                           w2 = __ballot_sync(kFull, own == best) & m;
            axis = w0 ? 0u : (w1 ? 1u : 2u);
            src = __ffs(w0 ? w0 : (w1 ? w1 : w2)) - 1;
        }
        const bool found = live && best != kNoKey;
        const uint32_t wcut =
            (__shfl_sync(kFull, cut[0] | (cut[1] << 8) | (cut[2] << 16), src) >> (8u * axis)) & 63u;
        const bool median = live && !found && n > P.max_leaf;  // bvh/src/lib.rs:527-531
        const bool leaf = live && n <= P.max_leaf &&
                          (!found || __uint_as_float(best) >= leaf_cost(n));  // :576-583
        const bool split = found && !leaf;
        // partition (bvh/src/lib.rs:597-612), stable
        const bool pred = split && ((word >> (5u * axis)) & 31u) < wcut;
        const uint32_t ltm = __ballot_sync(kFull, pred) & m;
        uint32_t n_lt = __popc(ltm);
        T.x[split ? (pred ? s + __popc(ltm & below) : s + n_lt + __popc(m & ~ltm & below)) : lane] = word;
        __syncwarp();
        word = T.x[lane];
        __syncwarp();
        if (split) {
            const uint32_t side = lane < s + n_lt ? 0u : 0xFFFFFFFFu;
#pragma unroll
            for (uint32_t q = 0; q < kOrders; ++q) node[q] &= (&T.pm[axis][q][0])[static_cast<int>(wcut) - 1] ^ side;
            if (n_lt == 0u || n_lt == n) {  // cannot happen: the winner has objects on both sides
                set_error(O.ctr, MGBVH_ERR_ASSERT, kSiteCount);
                live = false;
            }
        }
        bool odd = false;  // a median of other than two objects with equal centroids
        if (__any_sync(kFull, median)) {
            // median_split on axes 0, 1, 2 over the same list (:444-491, :528-530)
            const uint32_t half = n / 2u;
            bool same = true;  // two objects with equal centroids: the first is lt on every axis
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const uint32_t c = __float_as_uint(__shfl_sync(kFull, R.cen[a], (word >> (5 * a)) & 31u));
                same &= c == __shfl_sync(kFull, c, lane == s ? s + 1u : s);
            }
            odd = median && !(n == 2u && same);
            if (median) {
                n_lt = half;
                if (lane == s) n_median++;
            }
            if (__any_sync(kFull, odd)) {
                MedianIo io;
                io.word = word;
                io.regs = R;
#pragma unroll
                for (int i = 0; i < 6; ++i) io.nb[i] = nb[i];
                median_segments(odd, s, n, m, ss, se, maxn, T, io);
                word = io.word;
                if (odd) {
#pragma unroll
                    for (uint32_t q = 0; q < kOrders; ++q) node[q] = io.node[q];
#pragma unroll
                    for (int i = 0; i < 6; ++i) nb[i] = io.nb[i];
                }
            }
            if (median && !odd) {
                const uint32_t bits = T.rt[word & 31u];
#pragma unroll
                for (uint32_t q = 0; q < kOrders; ++q)
                    node[q] = 1u << ((q < 6u ? bits >> (5u * q) : word >> (5u * (q - 6u))) & 31u);
            }
        }
        const bool parted = split || median;
        float c[3];
#pragma unroll
        for (uint32_t a = 0; a < 3; ++a) c[a] = __shfl_sync(kFull, R.cen[a], (word >> (5u * a)) & 31u);
#pragma unroll
        for (uint32_t q = 0; q < 6; ++q) {
            const float v = __shfl_sync(kFull, R.val[q], top_bit(node[q]));
            if (parted && !odd) nb[q] = v;
        }
        if (parted) {
            // containment of the centroids in their side's bounds (:637-646)
            if (!box_contains(nb, c[0], c[1], c[2])) set_error(O.ctr, MGBVH_ERR_ASSERT, kSiteContain);
            if (lane == s) hmax = max(hmax, depth + 1u);
            const uint32_t n_gt = n - n_lt;
            if (lane < s + n_lt) {
                n = n_lt;
                slot = pair + 1u;
                pair = pair + 2u * n_gt;
            } else {
                s = s + n_lt;
                n = n_gt;
                slot = pair;
                pair = pair + 2u;
            }
            depth++;
            // each child is written as it comes to be: a leaf where the leaf
            // rule stops it (:556), else with its children's slots
            const bool cleaf = leaf_rule(n, depth, P);
            if (lane == s) {
                lane_store_node(O, nbase + slot, nb, base + s - tbase, n, cleaf ? 0u : pair);
                if (cleaf && n > 1u) {
                    n_holes++;
                    if (depth == P.max_depth) n_capped++;
                }
            }
            if (cleaf) {
                O.perm[base + lane] = T.ids[word & 31u];
                live = false;
            }
        }
        if (leaf) {  // no split is worth it: the node was written as an inner one
            if (lane == s) {
                if (nbase + slot < O.node_cap) O.nodes[nbase + slot].child_node = 0u;
                if (n > 1u) n_holes++;
            }
            O.perm[base + lane] = T.ids[word & 31u];
            live = false;
        }
    }
    // counters: one atomic per warp
    const uint32_t hm = __reduce_max_sync(kFull, hmax);
    const uint32_t med = __reduce_add_sync(kFull, n_median);
    const uint32_t hol = __reduce_add_sync(kFull, n_holes);
    const uint32_t cap = __reduce_add_sync(kFull, n_capped);
    if (lane == 0) {
        if (hm) atomicMax(&O.ctr->height, hm - 1u);
        if (med) atomicAdd(&O.ctr->median_splits, med);
        if (hol) atomicAdd(&O.ctr->holes, hol);
        if (cap) atomicAdd(&O.ctr->depth_capped, cap);
    }
}

}  // namespace mgbvh
