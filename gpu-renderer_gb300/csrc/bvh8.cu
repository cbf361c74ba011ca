// 8-wide BVH with 8-bit quantised child boxes (Node8Q), collapsed from the
// binary LBVH level by level.
//
// Each 8-wide node starts from one binary node's two children and repeatedly
// opens the inner child with the largest surface area, until it has 8
// children or only leaves (the greedy collapse of wide-BVH builders). Its
// children are then assigned to slots by position: slot bit a means "on the
// high side along axis a", chosen greedily by the score
// sum_a (+/-)(child centre - node centre)_a, so that a ray visiting inner
// children in order of (slot ^ octant) goes roughly near to far. Boxes are
// quantised outward against the exact planes q * 2^e + lo (lo the node's
// lower corner), whose ray distances the traversal measures with one FMA per
// plane.
//
// Nodes are numbered breadth first, level by level: a level's nodes are
// collapsed (eight lanes each), their inner-child and leaf counts are prefix-
// summed, and the children become the next level at consecutive indices, so
// a node's inner children are contiguous from child_base and its leaf
// triangles contiguous from tri_base (copied into the layout's own triangle
// array). The numbering is deterministic. All levels run in one cooperative
// launch; the host reads the sizes once, at its end.
#include <algorithm>

#include "gr_internal.h"
#include "grid_sync.cuh"
#include "quant.cuh"

namespace gr {
namespace {

using namespace q8;

constexpr int kThreads8 = 256;
constexpr int kWarps8 = kThreads8 / 32;
constexpr int kLanesPerNode = 8;                  // lanes collapsing one 8-wide node
constexpr int kNodesPerWarp = 32 / kLanesPerNode;
constexpr int32_t kEmptySlot = INT32_MIN;
constexpr uint32_t kMaxLevels8 = 72;
constexpr uint32_t kAloneNodes = kWarps8 * kNodesPerWarp;  // levels that one block takes in one step

// 8-wide planes: plane(q) = q * 2^e + lo, taken EXACTLY (the traversal
// measures it as fma(q, 2^e / d, (lo - o) / d) with error margins, never
// rounding the plane itself); e grows until plane(255) >= hi. q * 2^e is a
// float, so each comparison of a plane with a coordinate is decided exactly
// from the rounded sum and its two-sum error.
constexpr int kMaxExp8 = 119;  // 255 * 2^e stays finite

__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }

// Sign of (a + b) - v, exactly: -1, 0 or +1.
__device__ __forceinline__ int cmp_sum(float a, float b, float v) {
    const float s = __fadd_rn(a, b);
    if (s != v) return s < v ? -1 : 1;
    const float bp = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
    return e < 0.0f ? -1 : (e > 0.0f ? 1 : 0);
}

__device__ __forceinline__ int cmp_plane(int q, float scale, float lo, float v) {
    return cmp_sum(__fmul_rn((float)q, scale), lo, v);
}

__device__ __forceinline__ int pick_exponent8(float lo, float hi, uint32_t* err) {
    const float extent = __fsub_rn(hi, lo);
    int e = -126;
    if (extent > 0.0f) {
        const float q = __fdiv_rn(extent, 255.0f);
        int ex = (int)(__float_as_uint(q) >> 23) - 126;  // q = m * 2^ex with m in [1/2, 1)
        if (ex <= -126 || ex >= 129) frexpf(q, &ex);     // subnormal or infinite
        e = max(-126, min(kMaxExp8, ex - 1));
    }
    while (cmp_plane(255, pow2f(e), lo, hi) < 0) {
        if (e >= kMaxExp8) {
            atomicOr(err, ERR_RANGE);  // extent beyond about 2^127: not representable
            break;
        }
        ++e;
    }
    return e;
}

__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }

// Largest q with plane(q) <= v and smallest q with plane(q) >= v, by search (any input).
__device__ __noinline__ uint32_t quant_search8(float v, float scale, float lo, bool upper) {
    int q = upper ? 255 : 0;
    for (int step = 128; step > 0; step >>= 1) {
        if (!upper && q + step <= 255 && cmp_plane(q + step, scale, lo, v) <= 0) q += step;
        if (upper && q - step >= 0 && cmp_plane(q - step, scale, lo, v) >= 0) q -= step;
    }
    return (uint32_t)q;
}

// The same for lo <= v <= plane(255) (v may be NaN, as the search takes it) and
// lo, plane(255) finite: x = (v - lo) / scale is rounded once, by the
// subtraction (inv = 1 / scale is a power of two), and rounding keeps order, so
// its floor or ceiling can be off only when x is a whole number, and then the
// sign of the subtraction's error (two-sum) decides. A nonzero difference whose
// quotient underflows to 0 lies above plane(0).
__device__ __forceinline__ uint32_t quant_lo8(float v, float inv, float lo) {
    const float d = __fsub_rn(v, lo), x = __fmul_rn(d, inv);
    const float f = __fadd_rd(x, 8388608.0f);  // 2^23 + floor(x)
    const float b = __fsub_rn(d, v);           // two-sum of v and -lo
    const float err = __fsub_rn(__fsub_rn(v, __fsub_rn(d, b)), __fadd_rn(lo, b));
    const bool exact = __fsub_rn(f, 8388608.0f) == x;
    const uint32_t q = __float_as_uint(f) & 0xFFu;
    return exact && err < 0.0f ? q - 1u : (isnan(x) ? 0u : q);
}

__device__ __forceinline__ uint32_t quant_hi8(float v, float inv, float lo) {
    const float d = __fsub_rn(v, lo), x = __fmul_rn(d, inv);
    const float f = __fadd_ru(x, 8388608.0f);  // 2^23 + ceil(x)
    const float b = __fsub_rn(d, v);
    const float err = __fsub_rn(__fsub_rn(v, __fsub_rn(d, b)), __fadd_rn(lo, b));
    const bool exact = __fsub_rn(f, 8388608.0f) == x;
    const uint32_t q = __float_as_uint(f) & 0xFFu;
    return exact && (err > 0.0f || (q == 0u && d > 0.0f)) ? q + 1u : (isnan(x) ? 0u : q);
}

__device__ __forceinline__ float half_area(const CBox& b) {
    const float dx = __fsub_rn(b.hi[0], b.lo[0]);
    const float dy = __fsub_rn(b.hi[1], b.lo[1]);
    const float dz = __fsub_rn(b.hi[2], b.lo[2]);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dy), __fmul_rn(dy, dz)), __fmul_rn(dz, dx));
}

// What the host reads back: nodes and leaf triangles written, whether a
// capacity was exceeded (the build then stopped with no more writes), and the
// error bits with which the nodes cannot be traversed: a barrier gave up, here or
// in the binary build, or a reference was out of range (`failed` starts at zero).
struct Size8 {
    uint32_t nodes, tris, overflow, failed;
};

// Where the build stands between two levels.
struct Level8 {
    uint32_t n, out_base, tri_cursor, level;
};

struct Build8 {
    const Node* nodes;
    const Tri* tris;
    const BvhMeta* meta;
    uint32_t* frontier[2];     // binary ids of a level's nodes, levels alternate
    int32_t* slots;            // 8 child references per node of the level, by slot
    unsigned long long* bsum;  // per block: inner children | leaves << 32 of its nodes
    Node8Q* out;               // nodes [0, cap) go here (the layout's own array, kept from an earlier build)
    uint32_t cap;
    Node8Q* rest;              // nodes [cap, ..) here (scratch, same indices)
    Tri* tris8;
    uint32_t max_nodes, max_tris, num_tris;
    Size8* size;
    Level8* handed;            // what block 0 hands to the others after levels of its own
    uint32_t* sync;
    uint32_t* err;
};

// A reference that cannot be in a sound binary tree was seen and skipped.
__device__ __noinline__ void out_of_range(const Build8& B) {
    atomicOr(B.err, ERR_RANGE);
    atomicOr(&B.size->failed, (uint32_t)ERR_RANGE);
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ uint32_t group_max(uint32_t x) {
#pragma unroll
    for (int d = 1; d < kLanesPerNode; d <<= 1) x = max(x, __shfl_xor_sync(0xFFFFFFFFu, x, d));
    return x;
}

// Eight lanes per 8-wide node, four nodes per warp: lane k of a group holds
// candidate child k. Every choice is made exactly as one thread scanning the
// candidates in order would make it (first largest on ties), so the node does
// not depend on the lanes' arithmetic order. Loops run the same number of
// times in every group, so each shuffle has the whole warp. Writes the node
// (without its bases) through the warp's shared records `rec` and its 8 slot
// references when `have`; adds the warp's inner children and leaves to the counts.
__device__ __forceinline__ void collapse_group(const Build8& B, bool have, uint32_t root_id, Node8Q* __restrict__ out,
                                               int32_t* __restrict__ sref_out, uint32_t (*rec)[24], int32_t (*sref)[8],
                                               uint32_t& inner, uint32_t& leaves) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    constexpr int W = kLanesPerNode;
    const int lane = threadIdx.x & 31, k = lane & (W - 1), g = lane / W;
    int32_t ref = kEmptySlot;
    CBox box = {{0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f}};
    float lo[3] = {0.0f, 0.0f, 0.0f}, hi[3] = {0.0f, 0.0f, 0.0f};
    int cnt8 = 0;
    if (have) {
        const Node root = B.nodes[root_id];
        box = child_box(root, k & 1);
        if (k < 2) ref = k ? root.q3.y : root.q3.x;
        cnt8 = 2;
        // the node's box: its binary children's boxes are the exact minima and
        // maxima of everything below, whatever is opened
        const CBox b0 = child_box(root, 0), b1 = child_box(root, 1);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(b0.lo[a], b1.lo[a]);
            hi[a] = fmaxf(b0.hi[a], b1.hi[a]);
        }
    }
    // an inner candidate's node is fetched towards L2 as soon as it becomes a
    // candidate, so opening it later waits on L2 rather than DRAM
    if (ref >= 0) prefetch_l2(B.nodes + ref);
    // open the inner candidate with the largest surface area (at most 6 times);
    // scanned in order a NaN area is kept only when it comes first
    for (int step = 0; step < 6; ++step) {
        const bool cand = ref >= 0;  // lanes past cnt8 hold no reference
        const uint32_t cands = (__ballot_sync(kAll, cand) >> (g * W)) & 0xFFu;
        const bool open = cands != 0 && cnt8 < 8;
        if (!__any_sync(kAll, open)) break;
        // areas are +0 .. inf or NaN, whose bits are in order as integers
        const float area = half_area(box);
        uint32_t key = cand ? __float_as_uint(area) : 0u;
        if (isnan(area)) key = cand && k == __ffs(cands) - 1 ? 0xFFFFFFFFu : 0u;
        const uint32_t top = group_max(key);
        const uint32_t at = (__ballot_sync(kAll, cand && key == top) >> (g * W)) & 0xFFu;
        const int best = __ffs(at) - 1;
        const int32_t rb = __shfl_sync(kAll, ref, max(best, 0), W);
        if (open && (k == best || k == cnt8)) {
            // the opened lane takes the first child, the next free one the second
            const float4* nd = reinterpret_cast<const float4*>(B.nodes + rb);
            const int c = k == best ? 0 : 1;
            const float4 xy = __ldg(nd + c);
            const float2 z = __ldg(reinterpret_cast<const float2*>(nd + 2) + c);
            ref = __ldg(reinterpret_cast<const int32_t*>(nd + 3) + c);
            box.lo[0] = xy.x; box.hi[0] = xy.y; box.lo[1] = xy.z; box.hi[1] = xy.w; box.lo[2] = z.x; box.hi[2] = z.y;
            if (ref >= 0) prefetch_l2(B.nodes + ref);
        }
        if (open) ++cnt8;
    }
    // this lane's child scored against every slot
    const float dx = __fsub_rn(__fadd_rn(box.lo[0], box.hi[0]), __fadd_rn(lo[0], hi[0]));
    const float dy = __fsub_rn(__fadd_rn(box.lo[1], box.hi[1]), __fadd_rn(lo[1], hi[1]));
    const float dz = __fsub_rn(__fadd_rn(box.lo[2], box.hi[2]), __fadd_rn(lo[2], hi[2]));
    float sc[8];
    bool odd_score = false;  // infinite or NaN
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        sc[s] = __fadd_rn(__fadd_rn((s & 1) ? dx : -dx, (s & 2) ? dy : -dy), (s & 4) ? dz : -dz);
        odd_score |= !finite(sc[s]);
    }
    // greedy assignment: the best (score, then lowest child, then lowest slot)
    // first. That order is strict, so a pair that is the best left of its child
    // and the best left of its slot is one the greedy rule takes: a round takes
    // all such pairs of the node at once (two or three rounds instead of eight).
    // Lane s also holds column s of the scores (an 8 x 8 transpose). Taken rows
    // and columns score -inf, below every finite score.
    uint32_t used = 0;
    int my_slot = -1;
    if (!__any_sync(kAll, k < cnt8 && odd_score)) {
        if (k >= cnt8) {
#pragma unroll
            for (int s = 0; s < 8; ++s) sc[s] = -INFINITY;
        }
        float col[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) col[s] = sc[s];
#pragma unroll
        for (int d = 1; d < W; d <<= 1) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (i & d) continue;
                const float got = __shfl_xor_sync(kAll, (k & d) ? col[i] : col[i ^ d], d);
                if (k & d) col[i] = got;
                else col[i ^ d] = got;
            }
        }
        uint32_t left = (1u << cnt8) - 1u;  // children without a slot
        for (int round = 0; round < 8; ++round) {  // each round takes at least the best pair left of every node
            if (!__any_sync(kAll, left != 0)) break;
            const float rm = fmaxf(fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3])),
                                   fmaxf(fmaxf(sc[4], sc[5]), fmaxf(sc[6], sc[7])));
            const float cm = fmaxf(fmaxf(fmaxf(col[0], col[1]), fmaxf(col[2], col[3])),
                                   fmaxf(fmaxf(col[4], col[5]), fmaxf(col[6], col[7])));
            int rs = 7, cs = 7;  // the first slot of this child's best, the first child of this slot's
#pragma unroll
            for (int s = 6; s >= 0; --s) {
                rs = sc[s] == rm ? s : rs;
                cs = col[s] == cm ? s : cs;
            }
            const int mate = __shfl_sync(kAll, cs, rs, W);  // the best child of this child's best slot
            const int back = __shfl_sync(kAll, rs, cs, W);  // the best slot of this slot's best child
            const bool row = (left >> k & 1u) && mate == k;
            const bool column = !(used >> k & 1u) && (left >> cs & 1u) && back == k;
            const uint32_t rows = (__ballot_sync(kAll, row) >> (g * W)) & 0xFFu;
            const uint32_t columns = (__ballot_sync(kAll, column) >> (g * W)) & 0xFFu;
            if (row) my_slot = rs;
            left &= ~rows;
            used |= columns;
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                if (columns >> s & 1u) sc[s] = -INFINITY;
                if (rows >> s & 1u) col[s] = -INFINITY;
            }
        }
        if (left != 0 && k == 0) out_of_range(B);  // cannot happen
    } else {
        // an infinite or NaN score in the warp: fold the group's pairs in order, as one thread would
        for (int it = 0; it < 8; ++it) {
            int win = -1;
            float wsc = 0.0f;
            for (int j = 0; j < W; ++j) {
                const bool tj = __shfl_sync(kAll, my_slot, j, W) >= 0;
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const float x = __shfl_sync(kAll, sc[s], j, W);
                    if (j < cnt8 && !tj && !(used >> s & 1u) && (win < 0 || x > wsc)) {
                        win = 8 * j + s;
                        wsc = x;
                    }
                }
            }
            if (it < cnt8 && win >= 0) {
                used |= 1u << (win & 7);
                if (k == (win >> 3)) my_slot = win & 7;
            }
        }
    }
    // quantise: per-axis exponents (lanes 0-2), then this lane's child's six planes
    uint32_t my_be = 0;
    if (have && k < 3) my_be = (uint32_t)(pick_exponent8(k == 0 ? lo[0] : (k == 1 ? lo[1] : lo[2]),
                                                         k == 0 ? hi[0] : (k == 1 ? hi[1] : hi[2]), B.err) + 127);
    uint32_t be[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) be[a] = __shfl_sync(kAll, my_be, a, W);
    const bool child = k < cnt8 && my_slot >= 0;
    uint32_t imask = child && ref >= 0 ? 1u << my_slot : 0u;
#pragma unroll
    for (int d = 1; d < W; d <<= 1) imask |= __shfl_xor_sync(kAll, imask, d, W);
    // the node's 24 words through shared memory: each child drops its bytes
    uint32_t* r = rec[g];
    int32_t* sr = sref[g];
    __syncwarp();  // the records of the warp's last nodes have been read
#pragma unroll
    for (int j = 0; j < 3; ++j) r[k + 8 * j] = 0u;
    sr[k] = kEmptySlot;
    __syncwarp();
    if (child) {
        unsigned char* q = reinterpret_cast<unsigned char*>(r + 8);
        bool plain = true;  // finite planes that reach the node's corner
#pragma unroll
        for (int a = 0; a < 3; ++a) plain &= finite(lo[a]) && finite(hi[a]) && be[a] < (uint32_t)(kMaxExp8 + 127);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float scale = __uint_as_float(be[a] << 23), inv = __uint_as_float((254u - be[a]) << 23);
            q[16 * a + my_slot] = (unsigned char)(plain ? quant_lo8(box.lo[a], inv, lo[a])
                                                        : quant_search8(box.lo[a], scale, lo[a], false));
            q[16 * a + 8 + my_slot] = (unsigned char)(plain ? quant_hi8(box.hi[a], inv, lo[a])
                                                            : quant_search8(box.hi[a], scale, lo[a], true));
        }
        sr[my_slot] = ref;
    }
    if (k < 3) r[k] = __float_as_uint(k == 0 ? lo[0] : (k == 1 ? lo[1] : lo[2]));
    if (k == 3) r[3] = be[0] | (be[1] << 8) | (be[2] << 16) | (imask << 24);
    if (k == 6) r[6] = used;
    __syncwarp();
    if (have) {
        uint32_t* o = reinterpret_cast<uint32_t*>(out);
#pragma unroll
        for (int j = 0; j < 3; ++j) o[k + 8 * j] = r[k + 8 * j];
        sref_out[k] = sr[k];
    }
    inner += __popc(__ballot_sync(kAll, child && ref >= 0));
    leaves += __popc(__ballot_sync(kAll, child && ref < 0));
}

// The whole build. Per level: each warp collapses a run of consecutive nodes
// (four at a time) and counts their children; a grid barrier; every block sums
// the blocks before it, and each warp gives its nodes' children their places
// (a ballot over a step's 32 slots ranks them: inner children become the next
// level, leaf triangles are copied); a second barrier. Small levels go to as
// few warps a block as they need, on all blocks, so their few nodes run on many
// SMs. A level of at most 32 nodes, one step of a block's warps, is block 0's
// alone: no grid barrier, until a level is larger (it then hands the state over)
// or none is left. One launch replaces three a level and a host read-back every
// four: the 1M-triangle soup (8 levels, 284 Ki nodes) takes 0.21 ms instead of
// 0.49. A small level of all blocks costs 11 us (collapsing one node 5 us of
// dependent loads, two barriers 4.5, the places 1.8), so with such levels left to
// one block a rebuild and 1,024 rays take 103 us instead of 110 at 300 triangles,
// 178 instead of 184 at 10,000, 568 instead of 572 at 1M. The 242 Ki-node level
// takes 60 to 90 us a block, issue bound (1,240 warp instructions for four nodes;
// 1,510 before the slots were assigned in rounds and the planes quantised without
// a search). 4 blocks an SM (64 registers, 8 bytes of spills) against 3 was 877
// against 886 us for a rebuilt 1M-triangle BVH and 262,144 rays; prefetching the
// next nodes' neighbourhoods to L1 or L2 changed nothing.
__global__ void __launch_bounds__(kThreads8, 4) k8_build(Build8 B) {
    __shared__ uint32_t s_rec[kWarps8][kNodesPerWarp][24];
    __shared__ int32_t s_ref[kWarps8][kNodesPerWarp][8];
    __shared__ unsigned long long s_warp[kWarps8], s_before[kWarps8], s_total[kWarps8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t g = lane / kLanesPerNode, k = lane & (kLanesPerNode - 1);
    uint32_t n = 1, out_base = 0, tri_cursor = 0, level = 0, arrived = 0, overflow = 0;
    // A block whose barrier gave up leaves; it does not arrive again, so the others'
    // next barrier gives up too.
    bool met = true;
    while (n != 0) {
        const bool alone = n <= kAloneNodes;
        if (alone && blockIdx.x != 0) {
            met = grid_sync(B.sync, ++arrived * gridDim.x, B.err);
            if (!met) break;
            const uint4 h = __ldcg(reinterpret_cast<const uint4*>(B.handed));
            n = h.x;
            out_base = h.y;
            tri_cursor = h.z;
            level = h.w;
            continue;
        }
        const uint32_t grid = alone ? 1u : gridDim.x;  // blocks that share the level
        const uint32_t* frontier = (level & 1) ? B.frontier[1] : B.frontier[0];
        const uint64_t per_block = (uint64_t)grid * kNodesPerWarp;
        const uint32_t active = (uint32_t)min((uint64_t)kWarps8, (n + per_block - 1) / per_block);  // warps a block
        const uint64_t steps = ((uint64_t)n + per_block * active - 1) / (per_block * active);
        const uint64_t first = ((uint64_t)blockIdx.x * active + warp) * steps * kNodesPerWarp;
        const uint32_t begin = (uint32_t)warp < active ? (uint32_t)min((uint64_t)n, first) : n;
        const uint32_t end = (uint32_t)warp < active ? (uint32_t)min((uint64_t)n, first + steps * kNodesPerWarp) : n;
        uint32_t inner = 0, leaves = 0;
        for (uint32_t base = begin; base < end; base += kNodesPerWarp) {  // the same trip count for the whole warp
            const uint32_t i = base + g;
            bool have = i < end;
            const uint32_t id = !have ? 0u : (level == 0 ? B.meta->root : __ldcg(frontier + i));
            if (have && id >= B.max_nodes) {
                out_of_range(B);
                have = false;
            }
            const uint32_t at = out_base + i;
            collapse_group(B, have, id, (at < B.cap ? B.out : B.rest) + at, B.slots + 8ull * i, s_rec[warp],
                           s_ref[warp], inner, leaves);
        }
        if (lane == 0) s_warp[warp] = (unsigned long long)inner | ((unsigned long long)leaves << 32);
        __syncthreads();
        unsigned long long before = 0, total = 0;
        if (!alone) {
            if (threadIdx.x == 0) {
                unsigned long long sum = 0;
                for (int w = 0; w < kWarps8; ++w) sum += s_warp[w];
                B.bsum[blockIdx.x] = sum;
            }
            met = grid_sync(B.sync, ++arrived * grid, B.err);
            if (!met) break;
            for (uint32_t j = threadIdx.x; j < grid; j += kThreads8) {
                const unsigned long long v = __ldcg(B.bsum + j);
                total += v;
                if (j < blockIdx.x) before += v;
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                before += __shfl_xor_sync(0xFFFFFFFFu, before, d);
                total += __shfl_xor_sync(0xFFFFFFFFu, total, d);
            }
            if (lane == 0) {
                s_before[warp] = before;
                s_total[warp] = total;
            }
            __syncthreads();
            before = 0;
            total = 0;
        }
        for (int w = 0; w < kWarps8; ++w) {
            before += alone ? 0ull : s_before[w];
            total += alone ? s_warp[w] : s_total[w];
            if (w < warp) before += s_warp[w];
        }
        const uint32_t next_base = out_base + n;
        const uint64_t next_n = (uint32_t)total, next_tri = tri_cursor + (total >> 32);
        if (next_base + next_n > B.max_nodes || next_tri > B.max_tris || level >= kMaxLevels8) {
            overflow = 1;  // the same for every block that shares the level
            if (alone && threadIdx.x == 0) *B.handed = Level8{0u, out_base, tri_cursor, level};
            if (alone) met = grid_sync(B.sync, ++arrived * gridDim.x, B.err);
            break;
        }
        uint32_t in_run = (uint32_t)before, leaf_run = (uint32_t)(before >> 32);
        uint32_t* next = (level & 1) ? B.frontier[0] : B.frontier[1];
        for (uint32_t base = begin; base < end; base += kNodesPerWarp) {
            const uint32_t i = base + g;
            const bool have = i < end;
            const int32_t r = have ? B.slots[8ull * i + k] : kEmptySlot;
            const uint32_t mi = __ballot_sync(0xFFFFFFFFu, r >= 0);
            const uint32_t ml = __ballot_sync(0xFFFFFFFFu, r < 0 && r != kEmptySlot);
            const uint32_t lt = (1u << lane) - 1u, gt = (1u << (g * kLanesPerNode)) - 1u;  // lanes before, groups before
            if (have && k == 0) {
                const uint32_t at = out_base + i;
                Node8Q* nd = (at < B.cap ? B.out : B.rest) + at;
                *reinterpret_cast<uint2*>(&nd->child_base) =
                    make_uint2(next_base + in_run + __popc(mi & gt), tri_cursor + leaf_run + __popc(ml & gt));
            }
            if (r >= 0) {
                const uint32_t to = in_run + __popc(mi & lt);
                if (to < B.max_nodes) next[to] = (uint32_t)r;
            } else if (r != kEmptySlot) {
                const uint32_t to = tri_cursor + leaf_run + __popc(ml & lt), from = (uint32_t)(~r);
                if (to < B.max_tris && from < B.num_tris) B.tris8[to] = B.tris[from];
                else out_of_range(B);
            }
            in_run += __popc(mi);
            leaf_run += __popc(ml);
        }
        out_base = next_base;
        tri_cursor = (uint32_t)next_tri;
        n = (uint32_t)next_n;
        ++level;
        if (alone && n <= kAloneNodes && n != 0) {
            __syncthreads();
        } else {
            if (alone && threadIdx.x == 0) *B.handed = Level8{n, out_base, tri_cursor, level};
            met = grid_sync(B.sync, ++arrived * gridDim.x, B.err);
            if (!met) break;
        }
    }
    if (threadIdx.x != 0) return;
    uint32_t failed = met ? 0u : (uint32_t)ERR_TIMEOUT;
    if (blockIdx.x == 0) {
        B.size->nodes = out_base;
        B.size->tris = tri_cursor;
        B.size->overflow = overflow;
        failed |= __ldcg(B.err) & ERR_TIMEOUT;  // the binary nodes are incomplete
    }
    if (failed) atomicOr(&B.size->failed, failed);
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace

cudaError_t bvh8_build(BvhBuffers& b, uint32_t n, DevBuf& scratch, int num_sms, cudaStream_t s) {
    b.count8 = 0;
    b.tris8_count = 0;
    if (n == 0) return cudaSuccess;
    const size_t maxnodes = n > 1 ? n - 1 : 1;
    const size_t maxtris = std::max<size_t>(n, 2);  // a lone triangle fills both children of its node
    // resident blocks: the launch's barriers need every block on the GPU at once
    int dev = 0, coop = 0, per_sm = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k8_build, kThreads8, 0)) != cudaSuccess) return e;
    // a level has at most n - 1 nodes, four to a warp and step
    uint32_t grid = (uint32_t)std::min<size_t>(std::max(1, num_sms) * (size_t)std::max(1, per_sm),
                                               (maxnodes + kNodesPerWarp - 1) / kNodesPerWarp);
    if (!coop) grid = 1;
    // scratch: two frontiers, slot refs, block sums, sizes and barrier counter, the nodes
    size_t off = 0;
    const size_t o_f0 = off; off += align256(4 * maxnodes);
    const size_t o_f1 = off; off += align256(4 * maxnodes);
    const size_t o_sl = off; off += align256(32 * maxnodes);
    const size_t o_bs = off; off += align256(8 * (size_t)grid);
    const size_t o_sz = off; off += 256;  // Size8, then the barrier counter at 64 and Level8 at 128
    const size_t o_nd = off; off += align256(sizeof(Node8Q) * maxnodes);
    if ((e = scratch.ensure(off)) != cudaSuccess) return e;
    if ((e = b.tris8.ensure(sizeof(Tri) * maxtris)) != cudaSuccess) return e;
    char* base = (char*)scratch.p;
    Build8 B;
    B.nodes = (const Node*)b.nodes.p;
    B.tris = (const Tri*)b.tris.p;
    B.meta = (const BvhMeta*)b.meta.p;
    B.frontier[0] = (uint32_t*)(base + o_f0);
    B.frontier[1] = (uint32_t*)(base + o_f1);
    B.slots = (int32_t*)(base + o_sl);
    B.bsum = (unsigned long long*)(base + o_bs);
    B.out = (Node8Q*)b.nodes8.p;
    B.cap = b.nodes8.p ? (uint32_t)std::min<size_t>(b.nodes8.bytes / sizeof(Node8Q), maxnodes) : 0u;
    B.rest = (Node8Q*)(base + o_nd);
    B.tris8 = (Tri*)b.tris8.p;
    B.max_nodes = (uint32_t)maxnodes;
    B.max_tris = (uint32_t)maxtris;
    B.num_tris = n;
    B.size = (Size8*)(base + o_sz);
    B.sync = (uint32_t*)(base + o_sz + 64);
    B.handed = (Level8*)(base + o_sz + 128);
    B.err = &((BvhMeta*)b.meta.p)->err;
    if ((e = cudaMemsetAsync(base + o_sz, 0, 256, s)) != cudaSuccess) return e;
    for (;;) {
        if (grid == 1) {  // a lone block meets nobody at its barriers
            k8_build<<<1, kThreads8, 0, s>>>(B);
            e = cudaGetLastError();
        } else {
            void* args[] = {&B};
            e = cudaLaunchCooperativeKernel((const void*)k8_build, dim3(grid), dim3(kThreads8), args, 0, s);
        }
        if (e != cudaErrorCooperativeLaunchTooLarge) break;
        (void)cudaGetLastError();  // e.g. a client held to part of the SMs
        grid = (grid + 1) / 2;
    }
    if (e != cudaSuccess) return e;
    Size8 h{};
    if ((e = cudaMemcpyAsync(&h, B.size, sizeof(h), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    if (h.failed & ERR_TIMEOUT) return cudaErrorLaunchTimeout;
    if (h.overflow || h.failed) return cudaErrorInvalidValue;
    if (h.nodes > B.cap) {  // the layout's array grows: what it held stays in place
        const auto copy = [&](Node8Q* to, const void* from, uint32_t count) {
            return count ? cudaMemcpyAsync(to, from, sizeof(Node8Q) * count, cudaMemcpyDeviceToDevice, s) : cudaSuccess;
        };
        const size_t bytes = sizeof(Node8Q) * h.nodes;
        DevBuf grown;
        e = grown.ensure(bytes);
        if (e == cudaSuccess) {
            if ((e = copy((Node8Q*)grown.p, b.nodes8.p, B.cap)) != cudaSuccess) return e;
            if ((e = copy((Node8Q*)grown.p + B.cap, B.rest + B.cap, h.nodes - B.cap)) != cudaSuccess) return e;
            if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
            std::swap(grown.p, b.nodes8.p);
            std::swap(grown.bytes, b.nodes8.bytes);
        } else if (e == cudaErrorMemoryAllocation && B.cap) {
            // no room for both arrays: the old one's nodes wait in the scratch, whose first nodes are unused
            (void)cudaGetLastError();
            if ((e = copy(B.rest, b.nodes8.p, B.cap)) != cudaSuccess) return e;
            if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
            if ((e = b.nodes8.ensure(bytes)) != cudaSuccess) return e;  // frees the old array first
            if ((e = copy((Node8Q*)b.nodes8.p, B.rest, h.nodes)) != cudaSuccess) return e;
            if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
        } else {
            return e;
        }
    }
    b.count8 = h.nodes;
    b.tris8_count = h.tris;
    return cudaSuccess;
}

}  // namespace gr
