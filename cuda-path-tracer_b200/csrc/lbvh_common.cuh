// Pieces of the LBVH build shared by the reference-format build (lbvh.cu) and
// the split traversal BVH (split.cu): key traits and Morton helpers, box helpers, the 40-B
// traversal child slot, and the radix tree with its boxes and records.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "cpt.h"
#include "cpt_device.cuh"

namespace cpt {

template <typename K> struct KeyTraits;
template <> struct KeyTraits<uint32_t> { static constexpr int passes = 4, order = 10, total_bits = 32; };
template <> struct KeyTraits<uint64_t> { static constexpr int passes = 8, order = 21, total_bits = 64; };

// Bit spreading for the 3-D interleave (x -> bit 3i, y -> 3i+1, z -> 3i+2, the
// layout of morton.h:63-102): the standard shift-and-mask "part 1 by 2" sequence
// on 64 bits, valid for inputs of up to 21 bits.
__device__ __forceinline__ uint64_t spread3(uint32_t v)
{
    uint64_t x = v & 0x1FFFFFull;
    x = (x | (x << 32)) & 0x001F00000000FFFFull;
    x = (x | (x << 16)) & 0x001F0000FF0000FFull;
    x = (x | (x << 8)) & 0x100F00F00F00F00Full;
    x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

// quantize (math_util.h:10-13): clamp(int(x * n), 0, n - 1); cvt.rzi saturates and maps NaN to 0.
__device__ __forceinline__ uint32_t quantize(float x, uint32_t n)
{
    int32_t q = __float2int_rz(__fmul_rn(x, (float)n));
    int32_t hi = (int32_t)(n - 1);
    q = q < hi ? q : hi;
    return (uint32_t)(q > 0 ? q : 0);
}

struct Box { float mn[3], mx[3]; };

// True when a sort pass of this build gave up a look-back wait (CPT_STATUS_TIMEOUT):
// the kernels after the sort then return at once, leaving their outputs unwritten,
// and the build reports CPT_ERR_DEVICE_TIMEOUT. The status word is only read here,
// in kernels launched after the sort, so the kernel boundary orders it.
__device__ __forceinline__ bool sort_timed_out(const uint32_t* status)
{
    return (__ldcg(status) & CPT_STATUS_TIMEOUT) != 0u;
}

// Common-prefix length of keys i and j (-1 past the ends); equal keys go on with their
// positions (BVHBuilder.cu:107-201).
template <typename K>
__device__ __forceinline__ int key_delta(const K* __restrict__ keys, K ki, int n, int i, int j)
{
    if (j < 0 || j >= n) return -1;
    K kj = __ldg(keys + j);
    if (ki == kj) return __clz(i ^ j) + KeyTraits<K>::total_bits;
    if (sizeof(K) == 8) return __clzll((long long)(ki ^ kj));
    return __clz((int)(ki ^ kj));
}

__device__ __forceinline__ Box leaf_box(const float v[9])
{
    Box b;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        float mn = FLT_MAX, mx = -FLT_MAX;
#pragma unroll
        for (int vv = 0; vv < 3; ++vv) { mn = gmin(mn, v[3 * vv + ax]); mx = gmax(mx, v[3 * vv + ax]); }
        b.mn[ax] = mn;
        b.mx[ax] = mx;
    }
    return b;
}


// Arrival counter of a bottom-up walk: one atomic increment that releases this thread's
// earlier stores and acquires those of the thread that came before it at the same
// parent, device-wide.
__device__ __forceinline__ int arrive_acq_rel(int* counter)
{
    int r;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(r) : "l"(counter) : "memory");
    return r;
}

// ---------------------------------------------------------------------------
// Topology, boxes and traversal records in two launches (the radix tree of
// BVHBuilder.cu:107-201 and the bottom-up boxes of :39-98).
//
// A node of the radix tree splits two neighbouring leaves g and g + 1 and covers the leaves
// around them whose neighbours are all closer than those two (a longer common prefix): from
// the last split before g with a shorter prefix to the next one after it. Splits and nodes
// correspond one to one, and a node's reference index is the right end of its range if it is
// a left child, the left end if it is a right child — which of the two it is, the prefixes at
// its ends tell (the longer one is the nearer split, its parent's). So everything about a
// node follows from the prefix lengths of neighbours.
//
// tree_block: kTreeBlock consecutive leaves per block. In shared memory: both ends of every
// node by descent in a table of minima, its box from a table of the boxes of 2^k leaves in
// a row (a range is the union of two of them, which overlap), its children's boxes, and the
// records, copied out in rows. No key searches in memory, no counters, no divergent walk.
// What is left are the few nodes whose range leaves the block (about one in twelve); the
// finished subtrees below them go on a list.
//
// tree_climb: a thread per finished subtree goes up. The first child to arrive at a split
// leaves its range's far end there and goes; the second takes it with an acquire-release
// exchange (which also publishes and acquires the boxes) and makes the node.
//
// A node's box is the union of its leaves in order, each bound the last of equal ones (glm's
// min and max select their second argument), so the grouping does not show in the bytes — unless
// a bound is NaN: then min(a, min(NaN, c)) is not min(min(a, NaN), c), and a block that holds one
// unites its boxes child by child instead (Leaf::kAnyGrouping: a union that ignores NaN).
//
// 5.24 M triangles (1.22 GB of DRAM traffic): 724 us as a launch of key searches per node and
// a walk per leaf through the records in memory (a third of the lanes left at every level, 25 %
// of issue slots used); now 482 + 122. What bounds tree_block is shared memory (65 % of the L1
// pipe's time) and the barriers and loads that three blocks an SM cannot hide (five: 428); blocks
// of 128 leaves took 40 us less there and 43 more above. tree_climb is a chain of about 20 steps
// of 2 us, a release, an exchange and the sibling's box each, so small trees gain least (65,538
// triangles: 61 us as the former launches, 58 as these).
// ---------------------------------------------------------------------------
constexpr int kTreeBlock = 256;
constexpr int kTreeLevels = 9;  // tables of 1, 2, ... 256 in a row
constexpr int kNoEnd = -1;      // ends[g]: no child of split g has arrived
// The tree kernels run three blocks an SM, in the 132 KB split of the shared memory that the
// renderer's traversal has too: an SM that traces on another stream then need not fall idle to
// change it. Frames of C2 with the next scene's builds beside them take 122.8 ms a step with
// three blocks, 136 to 139 with four (196 KB) and 136 with five (228 KB); 5.24 M triangles alone
// 1,275, 1,223 and 1,213 us.
constexpr int kTreeBlocks = 3;
constexpr int kTreeSplitKb = 132;
constexpr int kTreeCarveout = 100 * kTreeSplitKb / 228;  // percent of the most (228 KB), as the driver is asked for it
constexpr int kTreeListWord = 16;  // the list's count among the 32 zeroed tile counters (a sort uses 9 at most)

// Blocks of 128 threads for tree_climb over the subtrees of `blocks` blocks (a grid-stride
// loop: about 40 subtrees come from a block).
inline int tree_top_blocks(uint64_t blocks, int sms)
{
    const uint64_t want = (blocks * 40 + 127) / 128;
    return (int)(want < 1 ? 1 : want > (uint64_t)sms * 16 ? (uint64_t)sms * 16 : want);
}

// Node word of a traversal record past the tree's last internal node (a tree over fewer
// leaves than its arrays hold, the split tree): no valid node word has both type bits and
// an all-ones left index.
constexpr uint32_t kUnusedNode = 0xFFFFFFFFu;

// One tree's arrays. ends: one word per split.
template <typename K>
struct TreeArrays {
    const K* keys;
    uint32_t n;
    uint32_t* children;
    uint32_t* parents_leaf;
    uint32_t* parents_internal;
    float* nodes;  // 96-B records
    cpt_bbox* node_boxes;
    int* ends;
    uint32_t* status;
};

// The subtrees that tree_block finished: their first and last leaves, in any order.
struct TreeList {
    uint32_t* first;
    uint32_t* last;
    uint32_t* count;  // zeroed before
};

struct TreeSmem {
    union {
        float4 row[2][2][kTreeBlock];  // boxes of 2^k leaves in a row, two levels: (lo, -), (hi, -)
        float4 record[6 * kTreeBlock];
    };
    float slot[kTreeBlock][10];        // the leaves' child slots
    float box[kTreeBlock][6];          // node boxes by node index
    uint8_t least[kTreeLevels][kTreeBlock + 8];  // minima of 2^k prefix lengths in a row (+ 1, 0 past the ends)
    uint8_t whole[kTreeBlock];         // by split: the node's range lies in the block
    uint8_t made[kTreeBlock];          // by node index: its record is here
};

// A record's meta words: Node word, right child's index, the other end of the leaf range.
__device__ __forceinline__ float4 record_meta(uint32_t g, bool left_internal, bool right_internal, uint32_t far_end)
{
    const uint32_t word = (g << 2) | (right_internal ? 2u : 0u) | (left_internal ? 1u : 0u);
    return make_float4(__uint_as_float(word), __uint_as_float(g + 1u), __uint_as_float(far_end), 0.0f);
}

// (1 KB of each block is the system's)
static_assert(kTreeBlocks * (sizeof(TreeSmem) + 1024) <= kTreeSplitKb * 1024, "the blocks fit the split");

// The leaves [base, base + count) of tree T (count <= kTreeBlock threads' worth; all of the
// block's threads call). leaf.load(i, slot, box) gives leaf i's child slot and box and writes
// what the leaf's own arrays hold; Leaf::lo / hi unite bounds. off: added to the listed leaves.
template <typename K, typename Leaf>
__device__ __forceinline__ void tree_block(TreeSmem& sm, const TreeArrays<K>& T, uint32_t base, uint32_t count,
                                           const Leaf& leaf, const TreeList& list, uint32_t off)
{
    const int t = threadIdx.x, nb = (int)count, n = (int)T.n;
    // prefix lengths + 1: entry h is that of leaves base + h - 1 and base + h
    for (int h = t; h <= kTreeBlock; h += kTreeBlock) {
        int d = 255;
        if (h <= nb) {
            const int i = (int)base + h - 1;
            d = i < 0 || i + 1 >= n ? 0 : 1 + key_delta(T.keys, __ldg(T.keys + i), n, i, i + 1);
        }
        sm.least[0][h] = (uint8_t)d;
    }
    float bx[6];
    bool unordered = false;
    if (t < nb) {
        float slot[10];
        leaf.load(base + (uint32_t)t, slot, bx);
#pragma unroll
        for (int k = 0; k < 10; ++k) sm.slot[t][k] = slot[k];
        sm.row[0][0][t] = make_float4(bx[0], bx[1], bx[2], 0.f);
        sm.row[0][1][t] = make_float4(bx[3], bx[4], bx[5], 0.f);
        if (!Leaf::kAnyGrouping)
#pragma unroll
            for (int c = 0; c < 6; ++c) unordered = unordered || bx[c] != bx[c];
    }
    sm.made[t] = 0;
    unordered = __syncthreads_or(unordered);
#pragma unroll
    for (int k = 1; k < kTreeLevels; ++k) {
        const int o = 1 << (k - 1);
        for (int h = t; h <= kTreeBlock; h += kTreeBlock)
            sm.least[k][h] = h + o <= kTreeBlock ? min(sm.least[k - 1][h], sm.least[k - 1][h + o]) : (uint8_t)0;
        __syncthreads();
    }
    // the node that splits leaves t and t + 1: [lo, hi], when both ends are in the block
    int lo = 0, hi = 0;
    bool node = false;
    if (t + 1 < nb) {
        const uint32_t d = sm.least[0][t + 1];
        int r = t + 2, l = t;
#pragma unroll
        for (int k = kTreeLevels - 1; k >= 0; --k) {
            const int w = 1 << k;
            if (r + w <= nb + 1 && sm.least[k][r] > d) r += w;
            if (l - w >= -1 && sm.least[k][l - w + 1] > d) l -= w;
        }
        node = r <= nb && l >= 0;
        lo = l;
        hi = r - 1;
    }
    sm.whole[t] = node;
    if (t < nb && !node && (int)base + t + 1 < n) T.ends[base + (uint32_t)t] = kNoEnd;
    const int at = node ? (sm.least[0][hi + 1] > sm.least[0][lo] ? hi : lo) : 0;
    float nbx[6];
    if (unordered) {  // child by child, a node when both its children are there (node t's: t and t + 1)
        bool todo = node;
        while (__syncthreads_or(todo)) {
            const bool ready = todo && (lo == t || sm.made[t]) && (hi == t + 1 || sm.made[t + 1]);
            __syncthreads();
            if (ready) {
                const float4 a = sm.row[0][0][t], b = sm.row[0][1][t], c = sm.row[0][0][t + 1], d = sm.row[0][1][t + 1];
                const float lf[6] = {a.x, a.y, a.z, b.x, b.y, b.z}, rf[6] = {c.x, c.y, c.z, d.x, d.y, d.z};
#pragma unroll
                for (int c6 = 0; c6 < 6; ++c6) {
                    const float l6 = lo == t ? lf[c6] : sm.box[t][c6], r6 = hi == t + 1 ? rf[c6] : sm.box[t + 1][c6];
                    nbx[c6] = c6 < 3 ? Leaf::lo(l6, r6) : Leaf::hi(l6, r6);
                    sm.box[at][c6] = nbx[c6];
                }
                sm.made[at] = 1;
                todo = false;
            }
        }
    }
    // boxes: a range of len leaves is the union of its first and its last 2^k, 2^k <= len < 2^(k + 1)
    const int mine = node ? 31 - __clz(hi - lo + 1) : -1;
#pragma unroll 1
    for (int k = 0; k < kTreeLevels && !unordered; ++k) {
        const float4(*row)[kTreeBlock] = sm.row[k & 1];
        float4(*next)[kTreeBlock] = sm.row[(k + 1) & 1];
        const int w = 1 << k;
        if (mine == k) {
            const float4 a = row[0][lo], b = row[0][hi - w + 1], c = row[1][lo], d = row[1][hi - w + 1];
            nbx[0] = Leaf::lo(a.x, b.x); nbx[1] = Leaf::lo(a.y, b.y); nbx[2] = Leaf::lo(a.z, b.z);
            nbx[3] = Leaf::hi(c.x, d.x); nbx[4] = Leaf::hi(c.y, d.y); nbx[5] = Leaf::hi(c.z, d.z);
        }
        if (k + 1 < kTreeLevels && t + 2 * w <= nb) {
            const float4 a = row[0][t + w], b = row[1][t + w];
            bx[0] = Leaf::lo(bx[0], a.x); bx[1] = Leaf::lo(bx[1], a.y); bx[2] = Leaf::lo(bx[2], a.z);
            bx[3] = Leaf::hi(bx[3], b.x); bx[4] = Leaf::hi(bx[4], b.y); bx[5] = Leaf::hi(bx[5], b.z);
            next[0][t] = make_float4(bx[0], bx[1], bx[2], 0.f);
            next[1][t] = make_float4(bx[3], bx[4], bx[5], 0.f);
        }
        if (!__syncthreads_or(mine > k)) break;
    }
    __syncthreads();  // the rows give way to the records
    if (node) {
        sm.made[at] = 1;
#pragma unroll
        for (int c = 0; c < 6; ++c) sm.box[at][c] = nbx[c];
    }
    __syncthreads();
    if (node) {
        const uint32_t g = base + (uint32_t)t, idx = base + (uint32_t)at;
        const bool li = lo < t, ri = hi > t + 1;
        float2* rec = reinterpret_cast<float2*>(sm.record + 6 * at);
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const int c = t + side;
            const bool internal = side ? ri : li;
            const float2* s2 = reinterpret_cast<const float2*>(internal ? sm.box[c] : sm.slot[c]);
#pragma unroll
            for (int k = 0; k < 5; ++k) rec[5 * side + k] = internal && k > 2 ? make_float2(0.f, 0.f) : s2[k];
            (internal ? T.parents_internal : T.parents_leaf)[g + (uint32_t)side] = idx;
        }
        const float4 meta = record_meta(g, li, ri, base + (uint32_t)(at == lo ? hi : lo));
        sm.record[6 * at + 5] = meta;
        T.children[idx] = __float_as_uint(meta.x);
        if (idx == 0u && lo == 0 && hi == n - 1) T.parents_internal[0] = CPT_INVALID_INDEX;
    }
    // subtrees whose parent's range leaves the block: leaf t, and the node of split t
#pragma unroll
    for (int what = 0; what < 2; ++what) {
        const int l = what ? lo : t, h = what ? hi : t;
        bool top = what ? node : t < nb;
        if (top) {
            const int up = sm.least[0][h + 1] > sm.least[0][l] ? h : l - 1;  // its parent's split
            top = up < 0 || up >= nb - 1 || !sm.whole[up];
            if (base == 0 && l == 0 && h == n - 1) top = false;  // the root
        }
        const unsigned m = __ballot_sync(0xFFFFFFFFu, top);
        if (m) {
            const int leader = __ffs(m) - 1, lane = t & 31;
            uint32_t p = 0;
            if (lane == leader) p = atomicAdd(list.count, (uint32_t)__popc(m));
            p = __shfl_sync(0xFFFFFFFFu, p, leader) + (uint32_t)__popc(m & ((1u << lane) - 1u));
            if (top) {
                list.first[p] = off + base + (uint32_t)l;
                list.last[p] = off + base + (uint32_t)h;
            }
        }
    }
    __syncthreads();
    float4* out = reinterpret_cast<float4*>(T.nodes) + 6 * (size_t)base;
    for (int q = t; q < 6 * nb; q += kTreeBlock)
        if (sm.made[q / 6]) out[q] = sm.record[q];
    float2* boxes = reinterpret_cast<float2*>(T.node_boxes + base);
    const float2* sbox = reinterpret_cast<const float2*>(sm.box);
    for (int q = t; q < 3 * nb; q += kTreeBlock)
        if (sm.made[q / 3]) boxes[q] = sbox[q];
}

// From the subtree over leaves [l, r] of tree T up. leaf.reload(i, slot, box): a leaf that
// tree_block loaded.
template <typename K, typename Leaf>
__device__ __forceinline__ void tree_climb(const TreeArrays<K>& T, uint32_t l, uint32_t r, const Leaf& leaf)
{
    const int n = (int)T.n;
    float box[6], slot[10];
    bool internal = l != r;
    auto load_box = [&](uint32_t node, float b[6]) {
        const float2* q = reinterpret_cast<const float2*>(T.node_boxes + node);
        const float2 x0 = __ldcg(q), x1 = __ldcg(q + 1), x2 = __ldcg(q + 2);
        b[0] = x0.x; b[1] = x0.y; b[2] = x1.x; b[3] = x1.y; b[4] = x2.x; b[5] = x2.y;
    };
    auto prefix = [&](uint32_t i, int j) { return key_delta(T.keys, __ldg(T.keys + i), n, (int)i, j); };
    int dl = prefix(l, (int)l - 1), dr = prefix(r, (int)r + 1);
    if (internal) load_box(dr > dl ? r : l, box);
    else leaf.reload(l, slot, box);
    if (l == 0u && r == T.n - 1u) return;  // (the root; tree_block does not list it)
    bool left = dr > dl;
    uint32_t g = left ? r : l - 1u;  // the parent's split
    auto arrive = [&](uint32_t end) {
        int other;
        asm volatile("atom.acq_rel.gpu.global.exch.b32 %0, [%1], %2;"
                     : "=r"(other)
                     : "l"(T.ends + g), "r"((int)end)
                     : "memory");
        return other;
    };
    // (every step widens the range, so the walk ends)
    for (int other = arrive(left ? l : r); other != kNoEnd;) {  // (else the sibling goes on from here)
        const uint32_t far_end = (uint32_t)other, sib = left ? g + 1u : g;
        if (left ? far_end <= g || far_end >= T.n : far_end > g) {  // not a tree (unsorted keys)
            atomicOr(T.status, CPT_STATUS_BAD_INDEX);
            return;
        }
        const bool sib_internal = far_end != sib;
        float sbox[6], sslot[10];
        if (sib_internal) load_box(sib, sbox);
        else leaf.reload(sib, sslot, sbox);
        if (left) {
            r = far_end;
            dr = prefix(r, (int)r + 1);
        } else {
            l = far_end;
            dl = prefix(l, (int)l - 1);
        }
        const uint32_t idx = dr > dl ? r : l, split = g;
        const bool was_left = left, own_internal = internal;
        float own[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) own[c] = box[c];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            box[c] = left ? Leaf::lo(box[c], sbox[c]) : Leaf::lo(sbox[c], box[c]);
            box[3 + c] = left ? Leaf::hi(box[3 + c], sbox[3 + c]) : Leaf::hi(sbox[3 + c], box[3 + c]);
        }
        float2* ob = reinterpret_cast<float2*>(T.node_boxes + idx);
        ob[0] = make_float2(box[0], box[1]);
        ob[1] = make_float2(box[2], box[3]);
        ob[2] = make_float2(box[4], box[5]);
        internal = true;
        // on to the parent at once (its release waits for the box alone); the record, which no
        // climb reads, is written while the exchange is under way
        const bool root = l == 0u && r == T.n - 1u;
        left = dr > dl;
        g = left ? r : l - 1u;
        other = root ? kNoEnd : arrive(left ? l : r);
        float2* rec = reinterpret_cast<float2*>(T.nodes + 24 * (size_t)idx);
        float2* mine = rec + (was_left ? 0 : 5);
        float2* its = rec + (was_left ? 5 : 0);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const float2 zero = make_float2(0.f, 0.f);
            mine[k] = !own_internal ? make_float2(slot[2 * k], slot[2 * k + 1])
                      : k < 3       ? make_float2(own[2 * k], own[2 * k + 1])
                                    : zero;
            its[k] = !sib_internal ? make_float2(sslot[2 * k], sslot[2 * k + 1])
                     : k < 3       ? make_float2(sbox[2 * k], sbox[2 * k + 1])
                                   : zero;
        }
        const bool li = was_left ? own_internal : sib_internal, ri = was_left ? sib_internal : own_internal;
        const float4 meta = record_meta(split, li, ri, idx == l ? r : l);
        reinterpret_cast<float4*>(rec)[5] = meta;
        T.children[idx] = __float_as_uint(meta.x);
        (li ? T.parents_internal : T.parents_leaf)[split] = idx;
        (ri ? T.parents_internal : T.parents_leaf)[split + 1u] = idx;
        if (root) T.parents_internal[0] = CPT_INVALID_INDEX;
    }
}

// Leaves that are triangles: sorted position i holds triangle order[i] of tris_in, copied to
// tris_out (the reference's permuted soup).
struct TriangleLeaves {
    const float* tris_in;
    const uint32_t* order;
    uint32_t order_base;  // (a batch: the scene's first input index)
    uint32_t n;
    float* tris_out;
    uint32_t* status;

    static constexpr bool kAnyGrouping = false;
    static __device__ __forceinline__ float lo(float a, float b) { return gmin(a, b); }
    static __device__ __forceinline__ float hi(float a, float b) { return gmax(a, b); }
    static __device__ __forceinline__ void make(uint32_t i, const float2 v2[5], float slot[10], float box[6])
    {
        const float v[9] = {v2[0].x, v2[0].y, v2[1].x, v2[1].y, v2[2].x, v2[2].y, v2[3].x, v2[3].y, v2[4].x};
        // v0, the leaf's index (the triangle a hit reports), v1 - v0, v2 - v0
        slot[0] = v[0]; slot[1] = v[1]; slot[2] = v[2];
        slot[3] = __uint_as_float(i);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            slot[4 + a] = __fsub_rn(v[3 + a], v[a]);
            slot[7 + a] = __fsub_rn(v[6 + a], v[a]);
        }
        const Box b = leaf_box(v);  // BVHBuilder.cu:73-74, BBox.cpp:26-30
#pragma unroll
        for (int a = 0; a < 3; ++a) { box[a] = b.mn[a]; box[3 + a] = b.mx[a]; }
    }
    __device__ __forceinline__ void load(uint32_t i, float slot[10], float box[6]) const
    {
        const uint32_t v = order[i];
        uint32_t src = v >= order_base ? v - order_base : n;
        if (src >= n) {  // only after a failed sort pass (its status is already set): stay in bounds
            atomicOr(status, CPT_STATUS_BAD_INDEX);
            src = n - 1;
        }
        const float2* s2 = reinterpret_cast<const float2*>(tris_in + 10ull * src);
        float2* o2 = reinterpret_cast<float2*>(tris_out + 10ull * i);
        float2 x[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) x[k] = __ldg(s2 + k);
#pragma unroll
        for (int k = 0; k < 5; ++k) o2[k] = x[k];
        make(i, x, slot, box);
    }
    __device__ __forceinline__ void reload(uint32_t i, float slot[10], float box[6]) const
    {
        const float2* s2 = reinterpret_cast<const float2*>(tris_out + 10ull * i);
        float2 x[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) x[k] = __ldcg(s2 + k);
        make(i, x, slot, box);
    }
};

}  // namespace cpt
