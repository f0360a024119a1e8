// st_sah.cu — device binned-SAH BVH build (TLAS "binned SAH" mode, and BLAS on request).
//
// The same specification as the CPU oracle's orc_binned_sah:
//   centroid (min+max)*0.5; a node's box and centroid box are unions under the IEEE total order;
//   per axis with centroid extent e > 0, bin = clamp((c - lo) * (32 / e)) in [0, 31];
//   a split after bin k costs halfArea(L)*nL + halfArea(R)*nR (AABB.h:39), empty sides skipped,
//   the lowest cost wins with ties to the lower axis then the lower k; with no candidate the range
//   is split at its middle; the partition is stable; the split nodes of a level get child pairs in
//   level order (pair p -> slots 1+2p, 2+2p); depth = level; height = deepest leaf.
// Every count is an integer and every box a min/max of ordered bits, so nothing depends on the order
// in which threads meet.
//
// A range is split by as many threads as it is worth: above kCap items by many blocks (two launches a
// level), above kSub by one block in shared memory, and from there a block of its own builds it to its
// leaves, a warp for each range of a level, the smallest ranges (most of a tree) without bins.  The
// numbering comes last: a level's split nodes are counted from left to right (the nodes of a level lie
// in the order of their ranges), and the nodes are written to the slots this gives.  Nothing waits for
// the host but the splitting of ranges above kCap.
// Bound by latency (a split is a chain of reductions, a few microseconds whatever its size), so what
// counts is how many ranges are split at once and how few launches there are.  One launch per step
// and level with a block for each range, and the level's totals read back by the host, took 1.42 ms of
// a 4096-box TLAS update and 8 ms for 327,680 triangles; one block for everything up to 4096 items
// 0.5 ms.
#include <cstdio>
#include "st_kernels.h"

namespace st {

constexpr int kBins = 32;
constexpr u32t kCap = 4096;            // items one block splits in shared memory
constexpr u32t kSub = 256;             // items a block builds to the leaves
constexpr u32t kTiny = 10;             // items up to which a range is split without bins (3 axes x 10 lanes)
constexpr int kMidThreads = 1024, kMidWarps = kMidThreads / 32, kMidGroups = 8;
constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr u32t kPer = (kSub + kThreads - 1) / kThreads;
constexpr u32t kChunk = 2048;          // items per block when binning / partitioning a large range
constexpr int kBinWords = 13;          // large ranges: count + box(6) + centroid box(6)
constexpr int kSweepWords = 7;         // in shared memory: count + box(6), [axis][word][bin]
constexpr int kWarpBins = 3 * kSweepWords * kBins;

// The move is opaque on purpose: written as __float_as_uint the bits of a NaN were not kept.
__device__ __forceinline__ unsigned ob(float f) {
    unsigned u;
    asm("mov.b32 %0, %1;" : "=r"(u) : "f"(f));
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fo(unsigned k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k); }
__device__ __forceinline__ u32t bin_of(float c, float lo, float scale) {
    float t = (c - lo) * scale;
    if (!(t > 0.0f)) return 0;
    if (t >= (float)(kBins - 1)) return kBins - 1;
    return (u32t)t;
}
__device__ __forceinline__ float half_area_bits(const unsigned *b) {
    float ex = fo(b[3]) - fo(b[0]), ey = fo(b[4]) - fo(b[1]), ez = fo(b[5]) - fo(b[2]);
    return ex * ey + ey * ez + ez * ex;
}
__device__ __forceinline__ void empty6(unsigned *b) {
    b[0] = b[1] = b[2] = 0xFFFFFFFFu;
    b[3] = b[4] = b[5] = 0u;
}
__device__ __forceinline__ void grow6(unsigned *b, const unsigned *c) {
    for (int q = 0; q < 3; q++) { b[q] = min(b[q], c[q]); b[3 + q] = max(b[3 + q], c[3 + q]); }
}
__device__ __forceinline__ void atomic_grow6(unsigned *b, const unsigned *c) {
    for (int q = 0; q < 3; q++) { atomicMin(b + q, c[q]); atomicMax(b + 3 + q, c[3 + q]); }
}
__device__ __forceinline__ void warp_grow6(unsigned *b) {
    for (int q = 0; q < 3; q++) {
        b[q] = __reduce_min_sync(0xFFFFFFFFu, b[q]);
        b[3 + q] = __reduce_max_sync(0xFFFFFFFFu, b[3 + q]);
    }
}
// The axes of a range with centroid box `c`: where its bins start and how wide they are.
struct Axes { float lo[3], scale[3]; bool valid[3]; };
__device__ __forceinline__ Axes axes_of(const unsigned *c) {
    Axes A;
    for (int a = 0; a < 3; a++) {
        const float l = fo(c[a]), e = fo(c[3 + a]) - l;
        A.valid[a] = e > 0.0f;
        A.lo[a] = l;
        A.scale[a] = A.valid[a] ? (float)kBins / e : 0.0f;
    }
    return A;
}
__device__ __forceinline__ void write_node(BVHNode &o, const unsigned *b, u32t first, u32t count, u32t level) {
    o.aabb.min.x = fo(b[0]); o.aabb.min.y = fo(b[1]); o.aabb.min.z = fo(b[2]);
    o.aabb.max.x = fo(b[3]); o.aabb.max.y = fo(b[4]); o.aabb.max.z = fo(b[5]);
    o.first_child_id = first;
    o.child_count = (uint16_t)count;
    o.depth = (uint16_t)level;
}

// A split: after which bin of which axis (key = axis * 32 + bin, kNoSplit: at the middle), and how
// many items go left.
constexpr u32t kNoSplit = 0xFFFFFFFFu;
struct Split { float cost; u32t key, nleft; };
__device__ __forceinline__ Split better(Split a, Split b) {
    return b.cost < a.cost || (b.cost == a.cost && b.key < a.key) ? b : a;
}
__device__ __forceinline__ Split warp_best(Split s) {
    for (int off = 16; off; off >>= 1) {
        Split o;
        o.cost = __shfl_xor_sync(0xFFFFFFFFu, s.cost, off);
        o.key = __shfl_xor_sync(0xFFFFFFFFu, s.key, off);
        o.nleft = __shfl_xor_sync(0xFFFFFFFFu, s.nleft, off);
        s = better(s, o);
    }
    return s;
}
// One axis' bins, a lane each: its box and count; the best split of the axis (all lanes agree).
__device__ __forceinline__ Split sweep_axis(const unsigned *mine, u32t n, int axis, int lane) {
    unsigned L[6], R[6];
    u32t nl = n;
    for (int q = 0; q < 6; q++) L[q] = R[q] = mine[q];
    for (int off = 1; off < 32; off <<= 1) {
        unsigned u[6], d[6];
        const u32t c = __shfl_up_sync(0xFFFFFFFFu, nl, off);
        for (int q = 0; q < 6; q++) {
            u[q] = __shfl_up_sync(0xFFFFFFFFu, L[q], off);
            d[q] = __shfl_down_sync(0xFFFFFFFFu, R[q], off);
        }
        if (lane >= off) { nl += c; grow6(L, u); }
        if (lane + off < 32) grow6(R, d);
    }
    const u32t total = __shfl_sync(0xFFFFFFFFu, nl, 31), nr = total - nl;
    for (int q = 0; q < 6; q++) R[q] = __shfl_down_sync(0xFFFFFFFFu, R[q], 1);
    Split s{INFINITY, kNoSplit, 0};
    if (lane < 31 && nl && nr) {
        const float cost = half_area_bits(L) * (float)nl + half_area_bits(R) * (float)nr;
        if (cost < INFINITY) s = Split{cost, (u32t)(axis * kBins + lane), nl};
    }
    return warp_best(s);
}

// ---- a range built to its leaves by one block ---------------------------------------------------
// A range of the ids, what made it, and its first level; `source`: which of the two id buffers holds it.
struct SahTask {
    u32t begin, end, level, source;
    u32t parent, side;                 // the large node it is a child of (kNoSplit: the root), and which child
};
// A node as a block leaves it when the numbering is not known yet.
struct SahRecord {
    unsigned box[6];
    u32t first, count;                 // leaf: first item and count; inner (count 0): its split's rank in the level
    u32t level, index;                 // level of the tree, index in the range's level
};
// A split range above kSub items, as the numbering needs it.
struct LargeNode {
    unsigned box[6];
    u32t begin, level, parent, side;
};
// Counters of a build, in device memory.
struct SahCounts {
    u32t large[2], chunks[2];          // ranges above kCap and their chunks: this level's, the next level's
    u32t mids, nodes, subtrees;        // ranges above kSub left to a block, large nodes so far, ranges up to kSub
    u32t info[4];                      // -, height, pairs
    unsigned root[6];                  // the root's centroid box
};
struct SubtreeShared {
    unsigned box[6][kSub];             // the items' boxes as ordered bits, by place in the range at its start
    unsigned bins[kWarps][kWarpBins];
    uint16_t order[2][kSub];           // the items in their present order (two buffers, a level apart)
    uint16_t task[2][kSub][2];         // this level's and the next level's ranges: begin, end
    unsigned red[6];
    u32t warp_sum[kWarps];
};
constexpr u32t kMidTasks = kCap / kSub;    // ranges above kSub items of one block: fewer than this
struct MidShared {
    unsigned box[6][kCap];
    uint16_t order[2][kCap];
    SahTask task[2][kMidTasks];        // begin and end within the block's range
    u32t tasks[2];
    unsigned bins[kMidGroups][kWarpBins], red[kMidGroups][12];
    Split axis_split[kMidGroups][3];
    u32t child[kMidGroups][2], warp_sum[kMidWarps];
};

template <class Shared>
__device__ __forceinline__ void item_bits(const Shared &S, u32t it, unsigned *b) {
    for (int q = 0; q < 6; q++) b[q] = S.box[q][it];
}
template <class Shared>
__device__ __forceinline__ float item_centroid(const Shared &S, u32t it, int a) {
    return (fo(S.box[a][it]) + fo(S.box[3 + a][it])) * 0.5f;
}
__device__ __forceinline__ void clear_bins(unsigned *bins, u32t at, u32t step) {
    for (u32t k = at; k < (u32t)kWarpBins; k += step) {
        const u32t w = (k / kBins) % kSweepWords;
        bins[k] = w >= 1 && w <= 3 ? 0xFFFFFFFFu : 0u;
    }
}
template <class Shared>
__device__ __forceinline__ void bin_item(unsigned *bins, const Axes &A, const Shared &S, u32t it) {
    unsigned b[6];
    item_bits(S, it, b);
    for (int a = 0; a < 3; a++) {
        if (!A.valid[a]) continue;
        unsigned *d = bins + a * kSweepWords * kBins + bin_of((fo(b[a]) + fo(b[3 + a])) * 0.5f, A.lo[a], A.scale[a]);
        atomicAdd(d, 1u);
        for (int q = 0; q < 3; q++) { atomicMin(d + (1 + q) * kBins, b[q]); atomicMax(d + (4 + q) * kBins, b[3 + q]); }
    }
}
__device__ __forceinline__ Split sweep_bins(const unsigned *bins, const Axes &A, int a, int lane) {
    if (!A.valid[a]) return Split{INFINITY, kNoSplit, 0};
    const unsigned *d = bins + a * kSweepWords * kBins + lane;
    unsigned b[6];
    for (int q = 0; q < 6; q++) b[q] = d[(1 + q) * kBins];
    return sweep_axis(b, d[0], a, lane);
}
template <class Shared>
__device__ __forceinline__ bool goes_left(const Shared &S, const Axes &A, const Split &s, u32t it, u32t place) {
    if (s.key == kNoSplit) return place < s.nleft;
    const int a = s.key / kBins;
    return bin_of(item_centroid(S, it, a), A.lo[a], A.scale[a]) <= s.key % kBins;
}
// Every candidate split of a tiny range, a lane each: after the bin of item i on axis a (a split after
// a bin that holds no item parts the items as the next lower bin that holds some, and ties go to it).
__device__ __forceinline__ Split tiny_split(const SubtreeShared &S, const Axes &A, const uint16_t *ord, u32t cnt, int lane) {
    const int a = lane / (int)kTiny;
    const u32t i = lane % kTiny;
    const bool on = a < 3 && i < cnt && A.valid[a];
    u32t bin = kBins;
    if (on) bin = bin_of(item_centroid(S, ord[i], a), A.lo[a], A.scale[a]);
    unsigned L[6], R[6];
    empty6(L);
    empty6(R);
    u32t nl = 0;
    for (u32t j = 0; j < cnt; j++) {
        const u32t other = __shfl_sync(0xFFFFFFFFu, bin, (a < 3 ? a : 2) * (int)kTiny + (int)j);
        unsigned b[6];
        item_bits(S, ord[j], b);
        if (other <= bin) { grow6(L, b); nl++; }
        else grow6(R, b);
    }
    Split s{INFINITY, kNoSplit, 0};
    if (on && nl < cnt) {
        const float cost = half_area_bits(L) * (float)nl + half_area_bits(R) * (float)(cnt - nl);
        if (cost < INFINITY) s = Split{cost, a * kBins + bin, nl};
    }
    return warp_best(s);
}

// A range's items into shared memory.
template <class Shared>
__device__ __forceinline__ void load_items(Shared &S, const float *aabbs, const u32t *ids, u32t base, u32t cnt) {
    for (u32t k = threadIdx.x; k < cnt; k += blockDim.x) {
        const u32t it = ids ? ids[base + k] : base + k;
        const float2 *f = reinterpret_cast<const float2 *>(aabbs + 6 * (size_t)it);
        const float2 p = f[0], q = f[1], r = f[2];
        S.box[0][k] = ob(p.x); S.box[1][k] = ob(p.y); S.box[2][k] = ob(q.x);
        S.box[3][k] = ob(q.y); S.box[4][k] = ob(r.x); S.box[5][k] = ob(r.y);
        S.order[0][k] = (uint16_t)k;
    }
}
// The left items before each thread's, over a block of WARPS warps (all threads call; `sums` is
// reused: the caller syncs before the next use).
template <int WARPS>
__device__ __forceinline__ u32t block_exclusive(u32t v, u32t *sums, u32t &total) {
    const u32t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u32t x = v;
    for (int off = 1; off < 32; off <<= 1) {
        const u32t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
        if (lane >= (u32t)off) x += y;
    }
    if (lane == 31) sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        u32t w = lane < WARPS ? sums[lane] : 0;
        for (int off = 1; off < 32; off <<= 1) {
            const u32t y = __shfl_up_sync(0xFFFFFFFFu, w, off);
            if (lane >= (u32t)off) w += y;
        }
        if (lane < WARPS) sums[lane] = w;
    }
    __syncthreads();
    total = sums[WARPS - 1];
    return (warp ? sums[warp - 1] : 0) + x - v;
}

// A barrier of one group of warps (1 <= id <= kMidGroups).
__device__ __forceinline__ void group_sync(u32t id, u32t threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Ranges of kSub to kCap items, a block each: split level after level, a level's ranges side by side,
// each by its share of the block's warps (a split is a chain of steps, some 10 us with 32 warps or with
// four: one after another, and down to 512 items only, they took 80 us of a 4096-box build, side by side
// down to 256 60 to 75, and the subtrees 75 instead of 140); children of at most kSub items (or a leaf's) are left to sah_subtree_kernel.  The ranges are mids[0, C->mids), or with
// mids == null the whole build, [0, n), of items in their own order.
__global__ void __launch_bounds__(kMidThreads, 1) sah_mid_kernel(const float *aabbs, SahCounts *C, const SahTask *mids, u32t n,
                                                                 u32t max_leaf, u32t *ids0, u32t *ids1, LargeNode *nodes,
                                                                 SahTask *subtrees) {
    extern __shared__ __align__(16) unsigned char raw[];
    MidShared &S = *reinterpret_cast<MidShared *>(raw);
    const u32t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u32t ranges = mids ? C->mids : 1;
    for (u32t range = blockIdx.x; range < ranges; range += gridDim.x) {
        SahTask T{0, n, 0, 0, kNoSplit, 0};
        if (mids) T = mids[range];
        const u32t *ids = !mids ? nullptr : T.source ? ids1 : ids0;      // null: the identity
        u32t *parted = T.source ? ids0 : ids1;                // the children's items go to the other buffer
        const u32t base = T.begin;
        __syncthreads();
        load_items(S, aabbs, ids, base, T.end - T.begin);
        if (tid == 0) {
            S.task[0][0] = SahTask{0, T.end - T.begin, T.level, 0, T.parent, T.side};
            S.tasks[0] = 1;
            S.tasks[1] = 0;
        }
        __syncthreads();
        for (int cur = 0; S.tasks[cur]; cur ^= 1) {
            const uint16_t *ord = S.order[cur];
            uint16_t *ord_next = S.order[cur ^ 1];
            const u32t nt = S.tasks[cur];
            u32t groups = 1;
            while (groups < nt && groups < (u32t)kMidGroups) groups *= 2;
            const u32t warps = kMidWarps / groups, threads = 32 * warps;
            const u32t g = warp / warps, gw = warp % warps, gt = tid % threads;
            unsigned *bins = S.bins[g], *red = S.red[g];
            for (u32t t = g; t < nt; t += groups) {
                const SahTask K = S.task[cur][t];
                const u32t b = K.begin, e = K.end, c = e - b;
                unsigned bx[6], cb[6];
                empty6(bx);
                empty6(cb);
                if (gt < 12) red[gt] = gt % 6 < 3 ? 0xFFFFFFFFu : 0u;
                clear_bins(bins, gt, threads);
                group_sync(1 + g, threads);
                for (u32t k = b + gt; k < e; k += threads) {
                    unsigned it[6], ct[6];
                    item_bits(S, ord[k], it);
                    for (int q = 0; q < 3; q++) ct[q] = ct[3 + q] = ob((fo(it[q]) + fo(it[3 + q])) * 0.5f);
                    grow6(bx, it);
                    grow6(cb, ct);
                }
                __syncwarp();
                warp_grow6(bx);
                warp_grow6(cb);
                if (lane == 0) { atomic_grow6(red, bx); atomic_grow6(red + 6, cb); }
                group_sync(1 + g, threads);
                const Axes A = axes_of(red + 6);
                for (u32t k = b + gt; k < e; k += threads) bin_item(bins, A, S, ord[k]);
                group_sync(1 + g, threads);
                if (gw < 3) {
                    const Split s = sweep_bins(bins, A, (int)gw, (int)lane);
                    if (lane == 0) S.axis_split[g][gw] = s;
                }
                group_sync(1 + g, threads);
                Split s = better(better(S.axis_split[g][0], S.axis_split[g][1]), S.axis_split[g][2]);
                if (s.key == kNoSplit) s.nleft = c / 2;
                // stable partition: a thread takes consecutive places, its warp's and then the group's
                // prefix sums give the left items before them
                const u32t per = (c + threads - 1) / threads;
                const u32t k0 = b + min(gt * per, c), k1 = b + min((gt + 1) * per, c);
                u32t left = 0;
                for (u32t k = k0; k < k1; k++) left += goes_left(S, A, s, ord[k], k - b);
                __syncwarp();
                u32t x = left;
                for (int off = 1; off < 32; off <<= 1) {
                    const u32t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
                    if (lane >= (u32t)off) x += y;
                }
                if (lane == 31) S.warp_sum[warp] = x;
                group_sync(1 + g, threads);
                u32t before = x - left;
                for (u32t w = 0; w < gw; w++) before += S.warp_sum[warp - gw + w];
                for (u32t k = k0; k < k1; k++) {
                    const uint16_t it = ord[k];
                    const bool l = goes_left(S, A, s, it, k - b);
                    ord_next[l ? b + before : b + s.nleft + (k - b - before)] = it;
                    before += l;
                }
                if (gt == 0) {
                    const u32t self = atomicAdd(&C->nodes, 1u);
                    LargeNode &o = nodes[self];
                    for (int q = 0; q < 6; q++) o.box[q] = red[q];
                    o.begin = base + b; o.level = K.level; o.parent = K.parent; o.side = K.side;
                    for (u32t side = 0; side < 2; side++) {
                        SahTask N{side ? b + s.nleft : b, side ? e : b + s.nleft, K.level + 1, T.source ? 0u : 1u, self, side};
                        const u32t nc = N.end - N.begin;
                        S.child[g][side] = nc <= kSub || nc <= max_leaf;
                        if (S.child[g][side]) {
                            N.begin += base;
                            N.end += base;
                            subtrees[atomicAdd(&C->subtrees, 1u)] = N;
                        } else {
                            S.task[cur ^ 1][atomicAdd(&S.tasks[cur ^ 1], 1u)] = N;
                        }
                    }
                }
                group_sync(1 + g, threads);
                // a child that leaves takes its items, in their order, with it
                for (u32t k = b + gt; k < e; k += threads) {
                    if (!S.child[g][k - b < s.nleft ? 0 : 1]) continue;
                    const u32t it = base + ord_next[k];
                    parted[base + k] = ids ? ids[it] : it;
                }
                group_sync(1 + g, threads);
            }
            __syncthreads();
            if (tid == 0) S.tasks[cur] = 0;
            __syncthreads();
        }
    }
}

// Ranges of at most kSub items, and leaves of any size, a block each, to the leaves: records at
// 2 * begin, the splits of the range's level l counted in splits[begin + l], the number of its levels
// in levels[range].  With subtrees == null the range is the whole build, [0, n), and the nodes are
// written to their slots as they come, info = {-, height, pairs}.
__global__ void __launch_bounds__(kThreads) sah_subtree_kernel(const float *aabbs, SahCounts *C, const SahTask *subtrees, u32t n,
                                                               u32t max_leaf, const u32t *ids0, const u32t *ids1,
                                                               u32t *out_order, BVHNode *nodes, u32t *info,
                                                               SahRecord *records, u32t *splits, u32t *levels) {
    __shared__ SubtreeShared S;
    const u32t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u32t ranges = subtrees ? C->subtrees : 1;
    for (u32t range = blockIdx.x; range < ranges; range += gridDim.x) {
        SahTask T{0, n, 0, 0, kNoSplit, 0};
        if (subtrees) T = subtrees[range];
        const u32t *ids = T.source ? ids1 : ids0;             // null: the identity
        const u32t cnt = T.end - T.begin, base = T.begin;
        SahRecord *rec = subtrees ? records + 2 * (size_t)base : nullptr;
        __syncthreads();
        if (cnt <= max_leaf) {                                // one leaf, of any size
            unsigned b[6];
            empty6(b);
            if (tid < 6) S.red[tid] = tid < 3 ? 0xFFFFFFFFu : 0u;
            __syncthreads();
            for (u32t k = tid; k < cnt; k += kThreads) {
                const u32t it = ids ? ids[base + k] : base + k;
                out_order[base + k] = it;
                for (int q = 0; q < 6; q++) {
                    const unsigned w = ob(aabbs[6 * (size_t)it + q]);
                    b[q] = q < 3 ? min(b[q], w) : max(b[q], w);
                }
            }
            warp_grow6(b);
            if (lane == 0) atomic_grow6(S.red, b);
            __syncthreads();
            if (tid == 0) {
                if (!rec) {
                    write_node(nodes[0], S.red, 0, cnt, 0);
                    info[0] = 0; info[1] = 1; info[2] = 0;
                } else {
                    for (int q = 0; q < 6; q++) rec[0].box[q] = S.red[q];
                    rec[0].first = base; rec[0].count = cnt; rec[0].level = T.level; rec[0].index = 0;
                    splits[base] = 0;
                    levels[range] = 1;
                    atomicMax(info + 1, T.level);
                }
            }
            continue;
        }
        load_items(S, aabbs, ids, base, cnt);
        if (tid == 0) { S.task[0][0][0] = 0; S.task[0][0][1] = (uint16_t)cnt; }
        __syncthreads();
        u32t nt = 1, pairs = 0, written = 0, level = 0, height = 0;
        for (int cur = 0; nt; cur ^= 1, level++) {
            const uint16_t *ord = S.order[cur];
            uint16_t *ord_next = S.order[cur ^ 1];
            // the ranks of the level's splits, left to right
            u32t mine = 0, level_splits;
            for (u32t k = kPer * tid; k < min(kPer * tid + kPer, nt); k++)
                mine += (u32t)(S.task[cur][k][1] - S.task[cur][k][0]) > max_leaf;
            u32t rank = block_exclusive<kWarps>(mine, S.warp_sum, level_splits);
            for (u32t k = kPer * tid; k < min(kPer * tid + kPer, nt); k++) {
                const u32t b = S.task[cur][k][0], e = S.task[cur][k][1];
                if (e - b > max_leaf) {
                    S.task[cur ^ 1][2 * rank][0] = (uint16_t)b;      // (the middle is filled in by the split)
                    S.task[cur ^ 1][2 * rank + 1][1] = (uint16_t)e;
                    // the split finds its rank in its range's first place of the next order, which is
                    // free until the range is parted into it
                    ord_next[b] = (uint16_t)rank;
                    rank++;
                }
            }
            __syncthreads();
            for (u32t t = warp; t < nt; t += kWarps) {
                const u32t b = S.task[cur][t][0], e = S.task[cur][t][1], c = e - b;
                const bool leaf = c <= max_leaf;
                unsigned bx[6], cb[6];
                empty6(bx);
                empty6(cb);
                for (u32t k = b + lane; k < e; k += 32) {
                    unsigned it[6], ct[6];
                    item_bits(S, ord[k], it);
                    for (int q = 0; q < 3; q++) ct[q] = ct[3 + q] = ob((fo(it[q]) + fo(it[3 + q])) * 0.5f);
                    grow6(bx, it);
                    grow6(cb, ct);
                }
                warp_grow6(bx);
                u32t first = base + b;
                if (leaf) {
                    for (u32t k = b + lane; k < e; k += 32) {
                        const u32t it = base + ord[k];
                        out_order[base + k] = ids ? ids[it] : it;
                    }
                } else {
                    warp_grow6(cb);
                    const Axes A = axes_of(cb);
                    const u32t r = ord_next[b];
                    __syncwarp();
                    Split s;
                    if (c <= kTiny) {
                        s = tiny_split(S, A, ord + b, c, (int)lane);
                    } else {
                        unsigned *bins = S.bins[warp];
                        clear_bins(bins, lane, 32);
                        __syncwarp();
                        for (u32t k = b + lane; k < e; k += 32) bin_item(bins, A, S, ord[k]);
                        __syncwarp();
                        s = sweep_bins(bins, A, 0, (int)lane);
                        s = better(s, sweep_bins(bins, A, 1, (int)lane));
                        s = better(s, sweep_bins(bins, A, 2, (int)lane));
                        __syncwarp();
                    }
                    if (s.key == kNoSplit) s.nleft = c / 2;
                    u32t before = 0;
                    for (u32t k0 = b; k0 < e; k0 += 32) {
                        const u32t k = k0 + lane;
                        const uint16_t it = k < e ? ord[k] : 0;
                        const bool l = k < e && goes_left(S, A, s, it, k - b);
                        const unsigned m = __ballot_sync(0xFFFFFFFFu, l);
                        const u32t lb = before + __popc(m & ((1u << lane) - 1u));
                        if (k < e) ord_next[l ? b + lb : b + s.nleft + (k - b - lb)] = it;
                        before += __popc(m);
                    }
                    if (lane == 0) S.task[cur ^ 1][2 * r][1] = S.task[cur ^ 1][2 * r + 1][0] = (uint16_t)(b + s.nleft);
                    first = rec ? r : 1 + 2 * (pairs + r);
                }
                if (lane == 0) {
                    if (!rec) {
                        write_node(nodes[written + t], bx, first, leaf ? c : 0, level);
                    } else {
                        SahRecord &o = rec[written + t];
                        for (int q = 0; q < 6; q++) o.box[q] = bx[q];
                        o.first = first; o.count = leaf ? c : 0; o.level = T.level + level; o.index = t;
                    }
                }
            }
            if (rec && tid == 0) splits[base + level] = level_splits;
            if (level_splits < nt) height = level;             // some range of the level is a leaf
            written += nt;
            pairs += level_splits;
            nt = 2 * level_splits;
            __syncthreads();
        }
        if (tid == 0) {
            if (!rec) {
                info[0] = 0;
                info[1] = height < 1 ? 1 : height;
                info[2] = pairs;
            } else {
                levels[range] = level;
                atomicMax(info + 1, T.level + height);
            }
        }
    }
}

// ---- ranges above kCap items: many blocks each, a level at a time ------------------------------------
struct LargeTask {
    SahTask t;
    u32t chunk0;                       // its first chunk of this level
    unsigned cbox[6];
};
__global__ void sah_init_kernel(SahCounts *C) {
    if (threadIdx.x < 6) C->root[threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;
    if (threadIdx.x == 0) {
        C->large[0] = C->large[1] = C->chunks[0] = C->chunks[1] = C->mids = C->nodes = C->subtrees = 0;
        C->info[1] = 1;
        C->info[2] = 0;
    }
}
__global__ void sah_root_kernel(const float *aabbs, u32t n, SahCounts *C) {
    unsigned c[6];
    empty6(c);
    for (u32t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float *a = aabbs + 6 * (size_t)i;
        unsigned ct[6];
        for (int q = 0; q < 3; q++) ct[q] = ct[3 + q] = ob((a[q] + a[3 + q]) * 0.5f);
        grow6(c, ct);
    }
    warp_grow6(c);
    if ((threadIdx.x & 31) == 0) atomic_grow6(C->root, c);
}
__device__ __forceinline__ u32t chunks_of(const SahTask &t) { return (t.end - t.begin + kChunk - 1) / kChunk; }
__device__ void clear_large_bins(unsigned *g, u32t at, u32t step) {
    for (u32t k = at; k < 3u * kBins; k += step) {
        g[k * kBinWords] = 0;
        empty6(g + k * kBinWords + 1);
        empty6(g + k * kBinWords + 7);
    }
}
__global__ void sah_first_kernel(u32t n, SahCounts *C, LargeTask *tasks, u32t *chunk_task, unsigned *bins) {
    const SahTask t{0, n, 0, 2, kNoSplit, 0};
    if (threadIdx.x == 0) {
        LargeTask L;
        L.t = t;
        L.chunk0 = 0;
        for (int q = 0; q < 6; q++) L.cbox[q] = C->root[q];
        tasks[0] = L;
        C->large[0] = 1;
        C->chunks[0] = chunks_of(t);
    }
    for (u32t k = threadIdx.x; k < chunks_of(t); k += blockDim.x) chunk_task[k] = 0;
    clear_large_bins(bins, threadIdx.x, blockDim.x);
}
// source 2: the identity (the root's level)
__device__ __forceinline__ u32t item_at(const u32t *ids0, const u32t *ids1, u32t source, u32t k) {
    return source == 2 ? k : source ? ids1[k] : ids0[k];
}
// One chunk of a large range: its items binned in shared memory, then added to the range's bins; the
// chunk's own counts are kept for the partition.
__global__ void sah_bin_kernel(const float *aabbs, const SahCounts *C, int now, const LargeTask *tasks, const u32t *chunk_task,
                               const u32t *ids0, const u32t *ids1, unsigned *bins, uint16_t *chunk_counts) {
    __shared__ unsigned sb[3 * kBins * kBinWords];
    if (blockIdx.x >= C->chunks[now]) return;
    const u32t r = chunk_task[blockIdx.x];
    const LargeTask L = tasks[r];
    clear_large_bins(sb, threadIdx.x, blockDim.x);
    __syncthreads();
    const Axes A = axes_of(L.cbox);
    const bool none = !(A.valid[0] | A.valid[1] | A.valid[2]);      // the box is still wanted: bin 0 of axis 0
    const u32t first = L.t.begin + (blockIdx.x - L.chunk0) * kChunk, last = min(L.t.end, first + kChunk);
    for (u32t k = first + threadIdx.x; k < last; k += blockDim.x) {
        const u32t i = item_at(ids0, ids1, L.t.source, k);
        float f[6];
        unsigned it[6], ct[6];
        for (int q = 0; q < 6; q++) { f[q] = aabbs[6 * (size_t)i + q]; it[q] = ob(f[q]); }
        float c[3];
        for (int q = 0; q < 3; q++) { c[q] = (f[q] + f[3 + q]) * 0.5f; ct[q] = ct[3 + q] = ob(c[q]); }
        for (int a = 0; a < 3; a++) {
            if (!A.valid[a] && !(none && a == 0)) continue;
            unsigned *b = sb + (a * kBins + (none ? 0 : bin_of(c[a], A.lo[a], A.scale[a]))) * kBinWords;
            atomicAdd(b, 1u);
            atomic_grow6(b + 1, it);
            atomic_grow6(b + 7, ct);
        }
    }
    __syncthreads();
    unsigned *g = bins + (size_t)r * 3 * kBins * kBinWords;
    for (int k = threadIdx.x; k < 3 * kBins; k += blockDim.x) {
        const unsigned *b = sb + k * kBinWords;
        chunk_counts[(size_t)blockIdx.x * 3 * kBins + k] = (uint16_t)b[0];
        if (!b[0]) continue;
        unsigned *d = g + k * kBinWords;
        atomicAdd(d, b[0]);
        atomic_grow6(d + 1, b + 1);
        atomic_grow6(d + 7, b + 7);
    }
}
// One large range: its split is found (every block finds it, a warp for each axis), its items are
// parted into the other id buffer, and the first chunk's block writes its node and its children.
__global__ void sah_part_kernel(const float *aabbs, SahCounts *C, int now, u32t max_leaf, const LargeTask *tasks,
                                const u32t *chunk_task, u32t *ids0, u32t *ids1, const unsigned *bins,
                                const uint16_t *chunk_counts, LargeTask *next, u32t *next_chunk_task, unsigned *next_bins,
                                LargeNode *nodes, SahTask *mids, SahTask *subtrees) {
    __shared__ Split axis_split[3];
    __shared__ u32t warp_sums[8], left_before, child[2], place[2];
    __shared__ unsigned cb[2][6];
    if (blockIdx.x >= C->chunks[now]) return;
    const u32t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u32t r = chunk_task[blockIdx.x];
    const LargeTask L = tasks[r];
    const u32t chunk = blockIdx.x - L.chunk0, cnt = L.t.end - L.t.begin;
    const Axes A = axes_of(L.cbox);
    const unsigned *g = bins + (size_t)r * 3 * kBins * kBinWords;
    if (tid == 0) left_before = 0;
    if (warp < 3) {
        Split s{INFINITY, kNoSplit, 0};
        if (A.valid[warp]) {
            const unsigned *b = g + (warp * kBins + lane) * kBinWords;
            s = sweep_axis(b + 1, b[0], (int)warp, (int)lane);
        }
        if (lane == 0) axis_split[warp] = s;
    }
    __syncthreads();
    Split s = better(better(axis_split[0], axis_split[1]), axis_split[2]);
    const bool middle = s.key == kNoSplit;
    if (middle) s.nleft = cnt / 2;
    const int axis = middle ? 0 : (int)(s.key / kBins);
    const u32t kbin = s.key % kBins;
    // the left items in the chunks before this one
    if (!middle) {
        u32t c = 0;
        for (u32t k = tid; k < chunk * kBins; k += blockDim.x)
            if (k % kBins <= kbin) c += chunk_counts[((size_t)(L.chunk0 + k / kBins) * 3 + axis) * kBins + k % kBins];
        c = __reduce_add_sync(0xFFFFFFFFu, c);
        if (lane == 0) atomicAdd(&left_before, c);
    }
    __syncthreads();
    const u32t first = L.t.begin + chunk * kChunk, last = min(L.t.end, first + kChunk);
    const u32t target = L.t.source == 0 ? 1u : 0u;
    u32t *out = target ? ids1 : ids0;
    u32t carry = middle ? min(chunk * kChunk, s.nleft) : left_before;
    for (u32t b0 = first; b0 < last; b0 += blockDim.x) {
        const u32t k = b0 + tid;
        const bool in = k < last;
        const u32t i = in ? item_at(ids0, ids1, L.t.source, k) : 0;
        bool l = false;
        if (in) {
            if (middle) l = k - L.t.begin < s.nleft;
            else l = bin_of((aabbs[6 * (size_t)i + axis] + aabbs[6 * (size_t)i + 3 + axis]) * 0.5f, A.lo[axis], A.scale[axis]) <= kbin;
        }
        const unsigned ball = __ballot_sync(0xFFFFFFFFu, l);
        if (lane == 0) warp_sums[warp] = __popc(ball);
        __syncthreads();
        u32t before = carry, sum = 0;
        for (u32t w = 0; w < blockDim.x / 32; w++) {
            if (w < warp) before += warp_sums[w];
            sum += warp_sums[w];
        }
        before += __popc(ball & ((1u << lane) - 1u));
        if (in) out[l ? L.t.begin + before : L.t.begin + s.nleft + (k - L.t.begin - before)] = i;
        carry += sum;
        __syncthreads();
    }
    if (chunk) return;
    // the range's node and its children, by the block of its first chunk
    if (tid < 2) child[tid] = kNoSplit;
    if (tid < 12) cb[tid / 6][tid % 6] = tid % 6 < 3 ? 0xFFFFFFFFu : 0u;
    __shared__ u32t self;
    if (tid == 0) self = atomicAdd(&C->nodes, 1u);
    __syncthreads();
    if (middle)       // the children's centroid boxes from the items (rare: all centroids equal)
        for (u32t k = L.t.begin + tid; k < L.t.end; k += blockDim.x) {
            const u32t i = item_at(ids0, ids1, L.t.source, k);
            unsigned ct[6];
            for (int q = 0; q < 3; q++) ct[q] = ct[3 + q] = ob((aabbs[6 * (size_t)i + q] + aabbs[6 * (size_t)i + 3 + q]) * 0.5f);
            atomic_grow6(cb[k - L.t.begin < s.nleft ? 0 : 1], ct);
        }
    if (warp == 0) {
        const int va = A.valid[0] ? 0 : A.valid[1] ? 1 : A.valid[2] ? 2 : 0;
        unsigned b[6];
        for (int q = 0; q < 6; q++) b[q] = g[(va * kBins + lane) * kBinWords + 1 + q];
        warp_grow6(b);
        if (lane == 0) {
            LargeNode &o = nodes[self];
            for (int q = 0; q < 6; q++) o.box[q] = b[q];
            o.begin = L.t.begin; o.level = L.t.level; o.parent = L.t.parent; o.side = L.t.side;
        }
        if (!middle) {
            for (int side = 0; side < 2; side++) {
                empty6(b);
                if ((lane <= kbin) == (side == 0))
                    for (int q = 0; q < 6; q++) b[q] = g[(axis * kBins + lane) * kBinWords + 7 + q];
                warp_grow6(b);
                if (lane == 0) for (int q = 0; q < 6; q++) cb[side][q] = b[q];
            }
        }
    }
    __syncthreads();
    if (tid < 2) {
        SahTask t{tid ? L.t.begin + s.nleft : L.t.begin, tid ? L.t.end : L.t.begin + s.nleft, L.t.level + 1, target, self, tid};
        const u32t c = t.end - t.begin;
        if (c > kCap && c > max_leaf) {
            LargeTask N;
            N.t = t;
            for (int q = 0; q < 6; q++) N.cbox[q] = cb[tid][q];
            child[tid] = atomicAdd(&C->large[now ^ 1], 1u);
            N.chunk0 = place[tid] = atomicAdd(&C->chunks[now ^ 1], chunks_of(t));
            next[child[tid]] = N;
        } else if (c > kSub && c > max_leaf) {
            mids[atomicAdd(&C->mids, 1u)] = t;
        } else {
            subtrees[atomicAdd(&C->subtrees, 1u)] = t;
        }
    }
    __syncthreads();
    for (int side = 0; side < 2; side++) {
        if (child[side] == kNoSplit) continue;
        const u32t c = side ? cnt - s.nleft : s.nleft;
        for (u32t k = tid; k < (c + kChunk - 1) / kChunk; k += blockDim.x) next_chunk_task[place[side] + k] = child[side];
        clear_large_bins(next_bins + (size_t)child[side] * 3 * kBins * kBinWords, tid, blockDim.x);
    }
}
__global__ void sah_next_level_kernel(SahCounts *C, int now) { C->large[now] = C->chunks[now] = 0; }

// ---- numbering --------------------------------------------------------------------------------------
// The parts of the tree are its large nodes, one split each, and its subtrees, splits[begin + l] at
// their level l, in order.  Sorted by where they begin, the parts of a level lie from left to right.
__device__ __forceinline__ u32t part_begin(const LargeNode *nodes, const SahTask *subtrees, u32t nl, u32t j) {
    return j < nl ? nodes[j].begin : subtrees[j - nl].begin;
}
__global__ void sah_sort_kernel(const SahCounts *C, const LargeNode *nodes, const SahTask *subtrees, u32t *sorted) {
    __shared__ u32t begins[256];
    const u32t nl = C->nodes, n = nl + C->subtrees;
    for (u32t j0 = blockIdx.x * blockDim.x; j0 < n; j0 += gridDim.x * blockDim.x) {
        const u32t j = j0 + threadIdx.x, mine = j < n ? part_begin(nodes, subtrees, nl, j) : 0;
        u32t before = 0;
        for (u32t i0 = 0; i0 < n; i0 += blockDim.x) {
            __syncthreads();
            if (i0 + threadIdx.x < n) begins[threadIdx.x] = part_begin(nodes, subtrees, nl, i0 + threadIdx.x);
            __syncthreads();
            for (u32t k = 0; k < min(blockDim.x, n - i0); k++) before += begins[k] < mine || (begins[k] == mine && i0 + k < j);
        }
        if (j < n) sorted[before] = j;
    }
}
// A block per level: rank[begin + l] (subtrees) and large_rank (large nodes) = how many of the level's
// split nodes lie left of the part's; totals[level] = all of the level.
__global__ void sah_rank_kernel(const SahCounts *C, const LargeNode *nodes, const SahTask *subtrees, const u32t *levels,
                                const u32t *splits, const u32t *sorted, u32t *rank, u32t *large_rank, u32t *totals) {
    __shared__ u32t sums[kWarps];
    const u32t nl = C->nodes, n = nl + C->subtrees, height = C->info[1];
    for (u32t level = blockIdx.x; level <= height; level += gridDim.x) {
        u32t carry = 0;
        for (u32t p0 = 0; p0 < n; p0 += kThreads) {
            const u32t p = p0 + threadIdx.x;
            u32t count = 0, total;
            u32t *out = nullptr;
            if (p < n) {
                const u32t j = sorted[p];
                if (j < nl) {
                    if (nodes[j].level == level) { count = 1; out = large_rank + j; }
                } else {
                    const SahTask t = subtrees[j - nl];
                    if (level >= t.level && level - t.level < levels[j - nl]) {
                        const u32t at = t.begin + level - t.level;
                        count = splits[at];
                        out = rank + at;
                    }
                }
            }
            const u32t before = block_exclusive<kWarps>(count, sums, total);
            if (out) *out = carry + before;
            carry += total;
            __syncthreads();
        }
        if (threadIdx.x == 0) totals[level] = carry;
    }
}
// totals -> the pairs of the levels before; one warp
__global__ void sah_base_kernel(SahCounts *C, u32t *totals) {
    u32t run = 0;
    for (u32t l0 = 0; l0 <= C->info[1]; l0 += 32) {
        const u32t l = l0 + threadIdx.x, v = l <= C->info[1] ? totals[l] : 0;
        u32t x = v;
        for (int off = 1; off < 32; off <<= 1) {
            const u32t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
            if (threadIdx.x >= (u32t)off) x += y;
        }
        if (l <= C->info[1]) totals[l] = run + x - v;
        run += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
    if (threadIdx.x == 0) C->info[2] = run;
}
__global__ void sah_emit_kernel(const SahCounts *C, const LargeNode *nodes, const SahTask *subtrees, const u32t *levels,
                                const u32t *rank, const u32t *large_rank, const u32t *base, const SahRecord *records,
                                const u32t *splits, BVHNode *out) {
    const u32t nl = C->nodes, ns = C->subtrees;
    auto child_slot = [&](u32t parent, u32t side) {
        return parent == kNoSplit ? 0u : 1 + 2 * (base[nodes[parent].level] + large_rank[parent]) + side;
    };
    for (u32t s = blockIdx.x; s < ns; s += gridDim.x) {
        const SahTask t = subtrees[s];
        u32t count = 1;                                            // its nodes: the root and two per split
        for (u32t l = 0; l < levels[s]; l++) count += 2 * splits[t.begin + l];
        for (u32t k = threadIdx.x; k < count; k += blockDim.x) {
            const SahRecord R = records[2 * (size_t)t.begin + k];
            const u32t l = R.level - t.level;
            const u32t slot = l ? 1 + 2 * (base[R.level - 1] + rank[t.begin + l - 1]) + R.index : child_slot(t.parent, t.side);
            write_node(out[slot], R.box, R.count ? R.first : 1 + 2 * (base[R.level] + rank[t.begin + l] + R.first), R.count, R.level);
        }
    }
    for (u32t j = blockIdx.x * blockDim.x + threadIdx.x; j < nl; j += gridDim.x * blockDim.x) {
        const LargeNode N = nodes[j];
        write_node(out[child_slot(N.parent, N.side)], N.box, 1 + 2 * (base[N.level] + large_rank[j]), 0, N.level);
    }
}

// ---- host driver ------------------------------------------------------------------------------
namespace {
struct SahLayout {
    size_t ids0, ids1, records, splits, rank, large_rank, totals, sorted, subtrees, levels, mids, task_a, task_b, chunk_a,
        chunk_b, bins_a, bins_b, counts, nodes, chunk_counts;
    u32t max_large, max_chunks;
    size_t bytes = 0;
};
// Ranges above kCap items at one level: fewer than n / kCap.  Large nodes and subtrees: a split may part
// as little as one item from the rest, so fewer than n of either.
SahLayout sah_layout(u32t n) {
    SahLayout L;
    L.max_large = n / kCap + 2;
    L.max_chunks = n / kChunk + L.max_large + 2;
    auto add = [&](size_t b) { size_t off = L.bytes; L.bytes += (b + 255) & ~(size_t)255; return off; };
    L.counts = add(sizeof(SahCounts));
    L.ids0 = add(sizeof(u32t) * (size_t)n);
    L.ids1 = add(sizeof(u32t) * (size_t)n);
    L.records = add(sizeof(SahRecord) * 2 * (size_t)n);
    L.splits = add(sizeof(u32t) * (size_t)n);
    L.rank = add(sizeof(u32t) * (size_t)n);
    L.large_rank = add(sizeof(u32t) * (size_t)n);
    L.totals = add(sizeof(u32t) * ((size_t)n + 2));
    L.sorted = add(sizeof(u32t) * 2 * (size_t)n);
    L.subtrees = add(sizeof(SahTask) * (size_t)n);
    L.levels = add(sizeof(u32t) * (size_t)n);
    L.nodes = add(sizeof(LargeNode) * (size_t)n);
    L.mids = add(sizeof(SahTask) * (size_t)(n / kSub + 1));
    L.task_a = add(sizeof(LargeTask) * L.max_large);
    L.task_b = add(sizeof(LargeTask) * L.max_large);
    L.chunk_a = add(sizeof(u32t) * L.max_chunks);
    L.chunk_b = add(sizeof(u32t) * L.max_chunks);
    L.bins_a = add(sizeof(unsigned) * (size_t)L.max_large * 3 * kBins * kBinWords);
    L.bins_b = add(sizeof(unsigned) * (size_t)L.max_large * 3 * kBins * kBinWords);
    L.chunk_counts = add(sizeof(uint16_t) * (size_t)L.max_chunks * 3 * kBins);
    return L;
}
}  // namespace

size_t sah_scratch_bytes(u32t n) { return sah_layout(n).bytes; }

bool sah_without_wait(u32t n, u32t max_leaf) { return n <= kCap || n <= max_leaf; }

cudaError_t sah_enqueue(const float *aabbs, u32t n, u32t max_leaf, BVHNode *out_nodes, u32t *out_order, void *scratch,
                        u32t **info, cudaStream_t st) {
    char *base = static_cast<char *>(scratch);
    const SahLayout Lo = sah_layout(n);
    SahCounts *C = (SahCounts *)(base + Lo.counts);
    *info = C->info;
    cudaError_t e = cudaFuncSetAttribute(sah_mid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MidShared));
    if (e != cudaSuccess) return e;
    if (n <= kSub || n <= max_leaf) {
        sah_subtree_kernel<<<1, kThreads, 0, st>>>(aabbs, nullptr, nullptr, n, max_leaf, nullptr, nullptr, out_order, out_nodes,
                                                   C->info, nullptr, nullptr, nullptr);
        return cudaGetLastError();
    }
    u32t *ids0 = (u32t *)(base + Lo.ids0), *ids1 = (u32t *)(base + Lo.ids1);
    SahRecord *records = (SahRecord *)(base + Lo.records);
    u32t *splits = (u32t *)(base + Lo.splits), *rank = (u32t *)(base + Lo.rank), *totals = (u32t *)(base + Lo.totals);
    u32t *large_rank = (u32t *)(base + Lo.large_rank), *levels = (u32t *)(base + Lo.levels), *sorted = (u32t *)(base + Lo.sorted);
    SahTask *subtrees = (SahTask *)(base + Lo.subtrees), *mids = (SahTask *)(base + Lo.mids);
    LargeNode *nodes = (LargeNode *)(base + Lo.nodes);
    sah_init_kernel<<<1, 32, 0, st>>>(C);
    if (n <= kCap) {
        sah_mid_kernel<<<1, kMidThreads, sizeof(MidShared), st>>>(aabbs, C, nullptr, n, max_leaf, ids0, ids1, nodes,
                                                                  subtrees);
    } else {
        LargeTask *task[2] = {(LargeTask *)(base + Lo.task_a), (LargeTask *)(base + Lo.task_b)};
        u32t *chunk[2] = {(u32t *)(base + Lo.chunk_a), (u32t *)(base + Lo.chunk_b)};
        unsigned *bins[2] = {(unsigned *)(base + Lo.bins_a), (unsigned *)(base + Lo.bins_b)};
        uint16_t *chunk_counts = (uint16_t *)(base + Lo.chunk_counts);
        sah_root_kernel<<<min((n + 255) / 256, 1184u), 256, 0, st>>>(aabbs, n, C);
        sah_first_kernel<<<1, 256, 0, st>>>(n, C, task[0], chunk[0], bins[0]);
        // the levels of the ranges above kCap: a few are enqueued between looks at how many are left
        // (launches for a level that is not there end at once)
        SahCounts now;
        now.large[0] = 1;
        for (u32t level = 0; now.large[level & 1];) {
            for (int k = 0; k < 4; k++, level++) {
                const int c = level & 1;
                sah_bin_kernel<<<Lo.max_chunks, 256, 0, st>>>(aabbs, C, c, task[c], chunk[c], ids0, ids1, bins[c], chunk_counts);
                sah_part_kernel<<<Lo.max_chunks, 256, 0, st>>>(aabbs, C, c, max_leaf, task[c], chunk[c], ids0, ids1, bins[c],
                                                               chunk_counts, task[c ^ 1], chunk[c ^ 1], bins[c ^ 1], nodes,
                                                               mids, subtrees);
                sah_next_level_kernel<<<1, 1, 0, st>>>(C, c);
            }
            e = cudaMemcpyAsync(&now, C, sizeof(now), cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) return e;
        }
        if (now.mids)
            sah_mid_kernel<<<min(now.mids, 1184u), kMidThreads, sizeof(MidShared), st>>>(aabbs, C, mids, n, max_leaf, ids0, ids1,
                                                                                      nodes, subtrees);
    }
    // few subtrees for every block of these grids to have one, or more than one for each: both are loops
    const u32t grid = min(max(n / 128, 1u), 1184u);
    sah_subtree_kernel<<<grid, kThreads, 0, st>>>(aabbs, C, subtrees, n, max_leaf, ids0, ids1, out_order, nullptr, C->info,
                                                  records, splits, levels);
    sah_sort_kernel<<<min(max(n / 4096, 1u), 148u), 256, 0, st>>>(C, nodes, subtrees, sorted);
    sah_rank_kernel<<<64, kThreads, 0, st>>>(C, nodes, subtrees, levels, splits, sorted, rank, large_rank, totals);
    sah_base_kernel<<<1, 32, 0, st>>>(C, totals);
    sah_emit_kernel<<<grid, 128, 0, st>>>(C, nodes, subtrees, levels, rank, large_rank, totals, records, splits, out_nodes);
    return cudaGetLastError();
}

cudaError_t sah_build(const float *aabbs, u32t n, u32t max_leaf, BVHNode *out_nodes, u32t *out_order, u32t info[2],
                      cudaStream_t st, void *scratch) {
    if (n == 0) { info[0] = info[1] = 0; return cudaSuccess; }
    u32t got[3] = {0, 0, 0}, *dev_info = nullptr;
    cudaError_t e = sah_enqueue(aabbs, n, max_leaf, out_nodes, out_order, scratch, &dev_info, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(got, dev_info, sizeof(got), cudaMemcpyDeviceToHost, st);
    const cudaError_t e2 = cudaStreamSynchronize(st);
    info[0] = 1 + 2 * got[2];
    info[1] = got[1] < 1 ? 1 : got[1];
    return e != cudaSuccess ? e : e2;
}

}  // namespace st
