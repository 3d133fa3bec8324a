// Split traversal BVH (cpt_lbvh_split): a second, traversal-only LBVH over pieces
// of the triangles, for scenes whose long thin triangles (the hairball) have
// boxes far larger than the triangles: every ray crossing such a box must test
// the triangle. Cutting a long triangle into pieces along its longest axis and
// giving each piece the box of the triangle clipped to its slab shrinks the boxes
// a ray crosses roughly by the piece count.
//
// The reference-format BVH (cpt_lbvh_build) is untouched and stays bit-exact;
// this one is built from its Morton-sorted triangles and only changes which
// nodes a ray visits. Its leaves hold the whole triangle (v0, the triangle's
// sorted index, v1 - v0, v2 - v0), so a ray tests the same triangle with the same
// arithmetic and reports the same index; the closest hit is the same triangle
// unless two triangles are hit at exactly the same distance, where the visiting
// order decides. Piece boxes contain the exact clipped triangle: along the split
// axis they are the slab bounds, across it the clipped polygon's extent widened
// by 2^-20 of the coordinates' magnitude (and kept inside the triangle's box), so
// rounding in the clipping cannot drop a hit.
//
// Steps (all on the device, one stream, the piece count never leaves the GPU):
//   k_split_weight/total  w_i = sqrt(max(0, area(box_i) - 2 area(tri_i))), sum in fixed order
//   k_split_count         pieces s_i = 1 + min(63, floor(extra * w_i / sum w)) -> sum s_i <= n + extra
//   k_split_scan_tiles    piece offsets of each 1024-triangle tile, total piece count
//   k_split_first         each triangle's first piece (exclusive offsets, in place of the counts),
//                         every fourth piece's triangle
//   k_split_emit          pieces, 4 per thread (balanced however the triangles are cut):
//                         clipped boxes, Morton keys of their centres in the root box,
//                         digit histograms, zeroed look-back state
//   k_scan_offsets, k_onesweep x P   as the main build, on the device count
//   k_split_tree_blocks, k_split_tree_top   topology, boxes and 96-B traversal nodes, as the main
//                         build's over leaves that are pieces
//   k_treelet             (CPT_SPLIT_TREELET) treelet restructuring of the Karras topology
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <algorithm>
#include "cpt.h"
#include "cpt_device.cuh"
#include "cpt_internal.h"
#include "lbvh_common.cuh"
#include "onesweep.cuh"

namespace cpt {
namespace {

constexpr int kSplitBlock = 256;
constexpr int kMaxPieces = 64;
constexpr int kScanItems = 4;
constexpr int kScanTile = kSplitBlock * kScanItems;  // triangles per count tile
constexpr int kWeightBlocks = 1024;

__device__ __forceinline__ void tri_box(const cpt_triangle& t, float lo[3], float hi[3])
{
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = fminf(fminf(t.v0[a], t.v1[a]), t.v2[a]);
        hi[a] = fmaxf(fmaxf(t.v0[a], t.v1[a]), t.v2[a]);
    }
}

__device__ __forceinline__ float split_weight(const cpt_triangle& t)
{
    float lo[3], hi[3];
    tri_box(t, lo, hi);
    const float ex = hi[0] - lo[0], ey = hi[1] - lo[1], ez = hi[2] - lo[2];
    const float box_area = 2.0f * (ex * ey + ey * ez + ez * ex);
    float e1[3], e2[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) { e1[a] = t.v1[a] - t.v0[a]; e2[a] = t.v2[a] - t.v0[a]; }
    const float cx = e1[1] * e2[2] - e1[2] * e2[1], cy = e1[2] * e2[0] - e1[0] * e2[2];
    const float cz = e1[0] * e2[1] - e1[1] * e2[0];
    const float tri_area = 0.5f * sqrtf(cx * cx + cy * cy + cz * cz);
    const float w = sqrtf(fmaxf(box_area - 2.0f * tri_area, 0.0f));
    return isfinite(w) ? w : 0.0f;
}

__device__ __forceinline__ double block_sum(double v)
{
    __shared__ double s_warp[kSplitBlock / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < kSplitBlock / 32; ++k) t += s_warp[k];
    return t;  // valid on thread 0
}

__global__ void __launch_bounds__(kSplitBlock) k_split_weight(const cpt_triangle* __restrict__ tris, uint32_t n,
                                                              double* __restrict__ partial)
{
    double acc = 0.0;
    for (uint32_t i = blockIdx.x * kSplitBlock + threadIdx.x; i < n; i += gridDim.x * kSplitBlock)
        acc += (double)split_weight(tris[i]);
    const double t = block_sum(acc);
    if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

// The partial sums in block order: one thread adds them (the order is part of the result),
// from shared memory, where every thread has put one (1024 dependent loads from device
// memory took 40 us, 4 now).
__global__ void __launch_bounds__(kWeightBlocks) k_split_total(const double* __restrict__ partial,
                                                               double* __restrict__ total)
{
    __shared__ double s_part[kWeightBlocks];
    s_part[threadIdx.x] = partial[threadIdx.x];
    __syncthreads();
    if (threadIdx.x != 0) return;
    double t = 0.0;
#pragma unroll 16
    for (int b = 0; b < kWeightBlocks; ++b) t += s_part[b];
    *total = t;
}

// Exclusive scan of one value per thread over the block; returns the block total
// through *total (all threads).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total)
{
    __shared__ uint32_t s_warp[kSplitBlock / 32 + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (int k = 0; k < kSplitBlock / 32; ++k) {
            const uint32_t t = s_warp[k];
            s_warp[k] = run;
            run += t;
        }
        s_warp[kSplitBlock / 32] = run;
    }
    __syncthreads();
    const uint32_t r = s_warp[warp] + x - v;
    *total = s_warp[kSplitBlock / 32];
    __syncthreads();
    return r;
}

__device__ __forceinline__ uint32_t piece_count(const cpt_triangle& t, double total, double extra)
{
    if (!(total > 0.0)) return 1u;
    const double share = extra * (double)split_weight(t) / total;
    const double extra_i = floor(share);
    return 1u + (uint32_t)fmin(extra_i, (double)(kMaxPieces - 1));
}

__global__ void __launch_bounds__(kSplitBlock) k_split_count(const cpt_triangle* __restrict__ tris, uint32_t n,
                                                             const double* __restrict__ total, double extra,
                                                             uint32_t* __restrict__ counts,
                                                             uint32_t* __restrict__ tile_sums)
{
    const double tot = *total;
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const uint32_t i = blockIdx.x * kScanTile + k * kSplitBlock + threadIdx.x;
        if (i >= n) break;
        const uint32_t c = piece_count(tris[i], tot, extra);
        counts[i] = c;
        sum += c;
    }
    uint32_t block_total;
    block_exclusive_scan(sum, &block_total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = block_total;
}

// Tile sums -> exclusive tile offsets (in place) and the piece count; one block.
__global__ void __launch_bounds__(1024) k_split_scan_tiles(uint32_t* __restrict__ tile_sums, uint32_t tiles,
                                                           uint32_t capacity, uint32_t* __restrict__ n_pieces,
                                                           uint32_t* __restrict__ status)
{
    __shared__ uint32_t s_warp[32];
    const int per = (int)((tiles + 1023) / 1024), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t loc = 0;
    for (int k = 0; k < per; ++k) {
        const uint32_t t = threadIdx.x * per + k;
        if (t < tiles) loc += tile_sums[t];
    }
    auto warp_scan = [&](uint32_t x) {  // inclusive
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        return x;
    };
    const uint32_t x = warp_scan(loc);
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) s_warp[lane] = warp_scan(s_warp[lane]);
    __syncthreads();
    uint32_t run = (warp ? s_warp[warp - 1] : 0u) + x - loc;
    if (threadIdx.x == 0) {
        uint32_t all = s_warp[31];
        if (all > capacity) {  // cannot happen (the shares sum to at most `extra`); stay in bounds
            atomicOr(status, CPT_STATUS_BAD_INDEX);
            all = capacity;
        }
        *n_pieces = all;
    }
    for (int k = 0; k < per; ++k) {
        const uint32_t t = threadIdx.x * per + k;
        if (t < tiles) {
            const uint32_t v = tile_sums[t];
            tile_sums[t] = run;
            run += v;
        }
    }
}

// Box of triangle t clipped to lo_s <= x_axis <= hi_s (conservative, see the file comment):
// Sutherland-Hodgman against x >= lo_s, then x <= hi_s. The first clip leaves up to four of
// six possible points (each corner, and after it the cut of the edge that leaves it); the
// second only needs each point's successor and the extent of what remains, so it runs over
// the six from the last to the first with the successor carried along, all in registers
// (an array of points in local memory, indexed at run time, took 3 x as long).
__device__ __forceinline__ void clip_box(const cpt_triangle& t, int axis, float lo_s, float hi_s, const float tlo[3],
                                         const float thi[3], float bmn[3], float bmx[3])
{
    const float v[3][3] = {{t.v0[0], t.v0[1], t.v0[2]}, {t.v1[0], t.v1[1], t.v1[2]}, {t.v2[0], t.v2[1], t.v2[2]}};
    auto along = [&](const float (&p)[3]) { return axis == 0 ? p[0] : axis == 1 ? p[1] : p[2]; };
    float pt[6][3];
    bool have[6];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float(&a)[3] = v[k];
        const float(&b)[3] = v[(k + 1) % 3];
        const float da = along(a) - lo_s, db = along(b) - lo_s;
        const bool ina = da >= 0.f, inb = db >= 0.f;
        const float s = da / (da - db);
        have[2 * k] = ina;
        have[2 * k + 1] = ina != inb;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            pt[2 * k][c] = a[c];
            pt[2 * k + 1][c] = a[c] + s * (b[c] - a[c]);
        }
    }
    float nx[3] = {0.f, 0.f, 0.f};  // the successor of the last point: the first one there is
#pragma unroll
    for (int k = 5; k >= 0; --k)
#pragma unroll
        for (int c = 0; c < 3; ++c) nx[c] = have[k] ? pt[k][c] : nx[c];
    float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    bool any = false;
#pragma unroll
    for (int k = 5; k >= 0; --k) {
        if (!have[k]) continue;
        const float(&a)[3] = pt[k];
        const float da = hi_s - along(a), db = hi_s - along(nx);
        const bool ina = da >= 0.f, inb = db >= 0.f;
        any = any || ina || inb;
        if (ina)
#pragma unroll
            for (int c = 0; c < 3; ++c) { mn[c] = fminf(mn[c], a[c]); mx[c] = fmaxf(mx[c], a[c]); }
        if (ina != inb) {
            const float s = da / (da - db);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float x = a[c] + s * (nx[c] - a[c]);
                mn[c] = fminf(mn[c], x);
                mx[c] = fmaxf(mx[c], x);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) nx[c] = a[c];
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) { bmn[a] = tlo[a]; bmx[a] = thi[a]; }
    if (any) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float eps = (fabsf(mn[a]) + fabsf(mx[a]) + (thi[a] - tlo[a])) * 9.5367431640625e-07f;  // 2^-20
            bmn[a] = fmaxf(mn[a] - eps, tlo[a]);
            bmx[a] = fminf(mx[a] + eps, thi[a]);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (a == axis) {
            bmn[a] = fmaxf(lo_s, tlo[a]);
            bmx[a] = fminf(hi_s, thi[a]);
        }
}

// Pieces per thread of k_split_emit.
constexpr int kEmitPieces = 4;

// Piece counts -> exclusive per-triangle piece offsets, in place (tile offsets from
// k_split_scan_tiles, a block scan inside the tile). owner[j / kEmitPieces]: the triangle of
// piece j, for every multiple j of kEmitPieces (where the emitting threads start).
__global__ void __launch_bounds__(kSplitBlock) k_split_first(uint32_t n, uint32_t* __restrict__ counts,
                                                             const uint32_t* __restrict__ tile_offsets,
                                                             uint32_t* __restrict__ owner, uint32_t capacity)
{
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t c[kScanItems];
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const uint32_t i = base + k;
        c[k] = i < n ? counts[i] : 0u;
        sum += c[k];
    }
    uint32_t block_total;
    uint32_t off = tile_offsets[blockIdx.x] + block_exclusive_scan(sum, &block_total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const uint32_t i = base + k;
        if (i < n) counts[i] = off;
        for (uint32_t j = (off + kEmitPieces - 1) / kEmitPieces; j * kEmitPieces < off + c[k]; ++j)
            if (j * kEmitPieces < capacity) owner[j] = i;
        off += c[k];
    }
}

// Pieces of the triangles, kEmitPieces consecutive pieces per thread whatever the
// triangles they come from (a long hairball triangle is cut into up to 64 pieces); the
// first one's triangle comes from owner. Writes the piece box, its Morton key and all the
// digit histograms of the sort, and zeroes the sort's look-back state. 11.8 M pieces:
// 64 pieces per thread after a binary search, clipping in local memory, 1,475 us (15 % of
// the warps resident; 355 us for the 100,000 of a small scene); now 348 us
// and 15 (4, 8 and 16 pieces per thread are within 2 %).
template <typename K>
__global__ void __launch_bounds__(kSplitBlock, 4) k_split_emit(const cpt_triangle* __restrict__ tris, uint32_t n,
                                                            const uint32_t* __restrict__ first,
                                                            const uint32_t* __restrict__ owner,
                                                            const uint32_t* __restrict__ n_pieces,
                                                            const cpt_bbox* __restrict__ root,
                                                            float4* __restrict__ pieces, K* __restrict__ keys,
                                                            uint32_t* __restrict__ hist, uint32_t* __restrict__ zero,
                                                            size_t zero_words)
{
    constexpr int P = KeyTraits<K>::passes;
    constexpr int order = KeyTraits<K>::order;
    __shared__ uint32_t s_hist[P * kRadix];
    for (int i = threadIdx.x; i < P * kRadix; i += kSplitBlock) s_hist[i] = 0;
    {
        const size_t gtid = (size_t)blockIdx.x * kSplitBlock + threadIdx.x, gsize = (size_t)gridDim.x * kSplitBlock;
        for (size_t i = gtid; i < zero_words; i += gsize) zero[i] = 0;
    }
    __syncthreads();
    float rmn[3], rinv[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        rmn[a] = root->min[a];
        rinv[a] = __frcp_rn(__fsub_rn(root->max[a], root->min[a]));
    }
    const uint32_t cells = 1u << order;
    const uint32_t np = *n_pieces;
    const uint64_t j0 = ((uint64_t)blockIdx.x * kSplitBlock + threadIdx.x) * kEmitPieces;
    if (j0 < np) {
        uint32_t i = min(owner[j0 / kEmitPieces], n - 1);
        uint32_t fi = first[i];
        uint32_t ei = i + 1 < n ? first[i + 1] : np;
        cpt_triangle t = tris[i];
        float tlo[3], thi[3];
        int axis = 0;
        float ext = 0.f;
        auto setup = [&]() {
            tri_box(t, tlo, thi);
            axis = 0;
            ext = thi[0] - tlo[0];
            if (thi[1] - tlo[1] > ext) { axis = 1; ext = thi[1] - tlo[1]; }
            if (thi[2] - tlo[2] > ext) { axis = 2; ext = thi[2] - tlo[2]; }
        };
        setup();
        const uint32_t jend = j0 + kEmitPieces < (uint64_t)np ? (uint32_t)(j0 + kEmitPieces) : np;
        for (uint32_t j = (uint32_t)j0; j < jend; ++j) {
            while (j >= ei && i + 1 < n) {  // the next triangle with pieces
                ++i;
                fi = ei;
                ei = i + 1 < n ? first[i + 1] : np;
                t = tris[i];
                setup();
            }
            const uint32_t s = ei - fi, p = j - fi;
            float bmn[3], bmx[3];
            if (s == 1) {
#pragma unroll
                for (int a = 0; a < 3; ++a) { bmn[a] = tlo[a]; bmx[a] = thi[a]; }
            } else {
                const float la = axis == 0 ? tlo[0] : axis == 1 ? tlo[1] : tlo[2];
                const float ha = axis == 0 ? thi[0] : axis == 1 ? thi[1] : thi[2];
                const float lo_s = p == 0 ? la : la + ext * ((float)p / (float)s);
                const float hi_s = p + 1 == s ? ha : la + ext * ((float)(p + 1) / (float)s);
                clip_box(t, axis, lo_s, hi_s, tlo, thi, bmn, bmx);
            }
            pieces[2 * (size_t)j] = make_float4(bmn[0], bmn[1], bmn[2], __uint_as_float(i));
            pieces[2 * (size_t)j + 1] = make_float4(bmx[0], bmx[1], bmx[2], 0.f);
            uint32_t q[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float c = 0.5f * (bmn[a] + bmx[a]);
                q[a] = quantize(__fmul_rn(__fsub_rn(c, rmn[a]), rinv[a]), cells);
            }
            const uint64_t key = spread3(q[0]) | (spread3(q[1]) << 1) | (spread3(q[2]) << 2);
            keys[j] = (K)key;
#pragma unroll
            for (int pp = 0; pp < P; ++pp) atomicAdd(&s_hist[pp * kRadix + (uint32_t)((key >> (8 * pp)) & 0xFF)], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < P * kRadix; i += kSplitBlock)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// Leaves that are pieces: sorted position i holds piece order[i], whose box goes to
// leaf_boxes; the slot is the whole triangle and its sorted index.
struct PieceLeaves {
    const cpt_triangle* tris;
    const float4* pieces;
    const uint32_t* order;
    float4* leaf_boxes;
    uint32_t n, n_tris;
    uint32_t* status;

    static constexpr bool kAnyGrouping = true;
    static __device__ __forceinline__ float lo(float a, float b) { return fminf(a, b); }
    static __device__ __forceinline__ float hi(float a, float b) { return fmaxf(a, b); }
    __device__ __forceinline__ void get(uint32_t i, float slot[10], float4& a, float4& b) const
    {
        uint32_t src = order[i];
        if (src >= n) {
            atomicOr(status, CPT_STATUS_BAD_INDEX);
            src = n - 1;
        }
        a = pieces[2 * (size_t)src];
        b = pieces[2 * (size_t)src + 1];
        uint32_t tri = __float_as_uint(a.w);
        if (tri >= n_tris) {
            atomicOr(status, CPT_STATUS_BAD_INDEX);
            tri = n_tris - 1;
        }
        const cpt_triangle t = tris[tri];
        slot[0] = t.v0[0]; slot[1] = t.v0[1]; slot[2] = t.v0[2];
        slot[3] = __uint_as_float(tri);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            slot[4 + k] = __fsub_rn(t.v1[k], t.v0[k]);
            slot[7 + k] = __fsub_rn(t.v2[k], t.v0[k]);
        }
    }
    __device__ __forceinline__ void load(uint32_t i, float slot[10], float box[6]) const
    {
        float4 a, b;
        get(i, slot, a, b);
        box[0] = a.x; box[1] = a.y; box[2] = a.z; box[3] = b.x; box[4] = b.y; box[5] = b.z;
        leaf_boxes[2 * (size_t)i] = make_float4(a.x, a.y, a.z, 0.f);
        leaf_boxes[2 * (size_t)i + 1] = make_float4(b.x, b.y, b.z, 0.f);
    }
    __device__ __forceinline__ void reload(uint32_t i, float slot[10], float box[6]) const
    {
        float4 a, b;
        get(i, slot, a, b);
        box[0] = a.x; box[1] = a.y; box[2] = a.z; box[3] = b.x; box[4] = b.y; box[5] = b.z;
    }
};

// The split tree over *n_pieces sorted pieces (lbvh_common.cuh); node_cap: the records of
// `nodes`, those past the tree marked unused.
template <typename K>
__global__ void __launch_bounds__(kTreeBlock, kTreeBlocks) k_split_tree_blocks(TreeArrays<K> T, PieceLeaves leaf, TreeList list,
                                                                  const uint32_t* __restrict__ n_pieces,
                                                                  uint32_t node_cap)
{
    __shared__ TreeSmem sm;
    wait_for_previous();
    let_next_start();
    T.n = leaf.n = *n_pieces;
    const uint32_t base = blockIdx.x * kTreeBlock, i = base + threadIdx.x;
    if (i + 1u >= T.n && i < node_cap)
        reinterpret_cast<float4*>(T.nodes)[6 * (size_t)i + 5] = make_float4(__uint_as_float(kUnusedNode), 0.f, 0.f, 0.f);
    if (sort_timed_out(T.status) || base >= T.n) return;  // no sorted pieces, or none here (uniform)
    tree_block(sm, T, base, min((uint32_t)kTreeBlock, T.n - base), leaf, list, 0u);
}

template <typename K>
__global__ void __launch_bounds__(128) k_split_tree_top(TreeArrays<K> T, PieceLeaves leaf, TreeList list,
                                                        const uint32_t* __restrict__ n_pieces)
{
    wait_for_previous();
    let_next_start();
    if (sort_timed_out(T.status)) return;
    T.n = leaf.n = *n_pieces;
    const uint32_t m = *list.count;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < m; p += gridDim.x * blockDim.x)
        tree_climb(T, list.first[p], list.last[p], leaf);
}

// ---------------------------------------------------------------------------
// Treelet restructuring (CPT_SPLIT_TREELET; Karras and Aila, "Fast Parallel
// Construction of High-Quality Bounding Volume Hierarchies", HPG 2013), applied to
// the split tree after its boxes. The cost of a tree is the sum of the surface
// areas of its internal nodes (the surface-area heuristic with the leaves fixed:
// every piece stays one leaf). A bottom-up walk with arrival counters
// reaches a node once both its subtrees are final; where the node has at least
// gamma leaves, its warp forms a treelet — the node's two children, then, up to 7
// leaves, the internal treelet leaf of largest area replaced by its two children —
// and finds the least-cost topology over those leaves by dynamic programming over
// their subsets, c(S) = area(S) + min over splits S = P + (S \ P) of c(P) + c(S \ P)
// (one leaf: 0), the lanes sharing out the 966 (subset, split) pairs of 7 leaves.
// A cheaper topology that is no taller than the old one replaces it in the same
// nodes (the treelet root keeps its index, box and parent). The result does not
// depend on timing: a treelet sees only its finished subtree, areas and sums are
// rounded without contraction, and equal costs go to the smallest split mask.
// One round with gamma = 4 (treelets of 4 to 6 leaves where a subtree has fewer
// than 7): on the C2 scene more rounds (gamma doubling) lower the binary tree's cost
// a little further but raise the node visits of the 8-wide tree collapsed from it.
// Since no treelet grows taller, the tree is never taller than the Karras tree it
// starts from.
// ---------------------------------------------------------------------------
constexpr int kTreeletBlock = 128;
constexpr int kTreeletWarps = kTreeletBlock / 32;
constexpr int kTreeletLeaves = 7;
constexpr int kTreeletSubsets = 1 << kTreeletLeaves;
#ifndef CPT_TREELET_ROUNDS
#define CPT_TREELET_ROUNDS 1
#endif
#ifndef CPT_TREELET_GAMMA
#define CPT_TREELET_GAMMA 4
#endif
#ifndef CPT_TREELET_GAMMA_SHIFT
#define CPT_TREELET_GAMMA_SHIFT 1  // gamma doubles every round
#endif
constexpr int kTreeletRounds = CPT_TREELET_ROUNDS;
constexpr int kTreeletGamma = CPT_TREELET_GAMMA;
constexpr int kTreeletMaxLevels = 1024;

// Half the surface area of a box (lo xyz, hi xyz), rounded alike on every run.
__device__ __forceinline__ float half_area(const float* b)
{
    const float dx = __fsub_rn(b[3], b[0]), dy = __fsub_rn(b[4], b[1]), dz = __fsub_rn(b[5], b[2]);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dy), __fmul_rn(dy, dz)), __fmul_rn(dz, dx));
}

// A warp's treelet. Lane k stands for treelet leaf k while it is formed. c comes first, at a
// multiple of its 512 B in shared memory: a subset's byte offset is then or-ed into its address.
struct alignas(512) TreeletWarp {
    float c[kTreeletSubsets];            // least cost over a subset (its area until its size class is done)
    float box[kTreeletLeaves][6];
    float slot[kTreeletLeaves][10];      // the leaves' 40-B child slots, read before any rewrite
    uint32_t id[kTreeletLeaves];         // internal node index, or piece position for a leaf
    uint32_t height[kTreeletLeaves];
    uint32_t size[kTreeletLeaves];
    uint32_t inode[kTreeletLeaves - 1];  // the treelet's internal nodes, [0] = its root
    uint8_t split[kTreeletSubsets];      // and the part of it with its lowest leaf
    // the new topology: node j covers subset sub[j], its children are treelet leaf k (< 8) or node 8 + j
    uint8_t sub[kTreeletLeaves - 1], child[kTreeletLeaves - 1][2], node_depth[kTreeletLeaves - 1];
    uint8_t leaf_depth[kTreeletLeaves];
};

// The subsets of 7 leaves by size: 21 of 2 (from 0), 35 of 3 (21), 35 of 4 (56), 21 of 5 (91),
// 7 of 6 (112) and the whole (119).
__constant__ uint8_t kTreeletOrder[120] = {
    3, 5, 6, 9, 10, 12, 17, 18, 20, 24, 33, 34, 36, 40, 48, 65, 66, 68, 72, 80, 96,
    7, 11, 13, 14, 19, 21, 22, 25, 26, 28, 35, 37, 38, 41, 42, 44, 49, 50, 52, 56, 67, 69, 70, 73, 74, 76, 81, 82, 84, 88,
    97, 98, 100, 104, 112,
    15, 23, 27, 29, 30, 39, 43, 45, 46, 51, 53, 54, 57, 58, 60, 71, 75, 77, 78, 83, 85, 86, 89, 90, 92, 99, 101, 102, 105,
    106, 108, 113, 114, 116, 120,
    31, 47, 55, 59, 61, 62, 79, 87, 91, 93, 94, 103, 107, 109, 110, 115, 117, 118, 121, 122, 124,
    63, 95, 111, 119, 123, 125, 126, 127};

// What treelet_form leaves in registers, the same in every lane.
struct TreeletForm {
    uint32_t m;              // treelet leaves (0: bad index met)
    uint32_t internal_mask;  // bit k: treelet leaf k is an internal node
    float old_cost;          // summed area of the treelet's internal nodes
};

// Forms the treelet rooted at internal node r (the whole warp): one coalesced load per opened
// node brings both child slots; the lanes of the two new treelet leaves fetch what hangs on
// them (boxes of pieces, sizes and heights of nodes).
__device__ __forceinline__ TreeletForm treelet_form(const float* __restrict__ nodes,
                                                    const float4* __restrict__ leaf_boxes,
                                                    const uint2* __restrict__ info, uint32_t n, uint32_t r,
                                                    TreeletWarp& w, uint32_t* __restrict__ status)
{
    const uint32_t lane = threadIdx.x & 31u;
    TreeletForm f;
    f.old_cost = 0.f;
    uint32_t m = 0, q = r, k0 = 0, id = 0, size = 0, height = 0;
    uint32_t cand = 0;  // an internal leaf's area as bits + 1
    bool internal = false, ok = true;
    __syncwarp();  // the last treelet's readers are done
    for (uint32_t ni = 0;; ++ni) {
        const uint32_t k1 = m ? m : 1u;
        if (lane == 0) w.inode[ni] = q;
        // words 0-9 the left slot, 10-19 the right, 20 the Node word, 21 the right child
        const float wd = lane < 22u ? __ldcg(nodes + 24 * (size_t)q + lane) : 0.f;
        const uint32_t word = __shfl_sync(0xFFFFFFFFu, __float_as_uint(wd), 20);
        const uint32_t right = __shfl_sync(0xFFFFFFFFu, __float_as_uint(wd), 21);
        const uint32_t side = lane >= 10u ? 1u : 0u, at = lane - 10u * side;
        const bool side_internal = (word >> side) & 1u;
        const uint32_t side_id = side ? right : word >> 2;
        ok = ok && !__any_sync(0xFFFFFFFFu, side_internal ? side_id >= n - 1 : side_id >= n);
        if (!ok) break;
        if (lane < 20u) {
            const uint32_t k = side ? k1 : k0;
            w.slot[k][at] = wd;
            if (at < 6u)  // an internal child's slot starts with its box
                w.box[k][at] = side_internal
                                   ? wd
                                   : reinterpret_cast<const float*>(leaf_boxes)[8 * (size_t)side_id + at + (at >= 3u)];
        }
        if (lane == k0 || lane == k1) {
            const bool rhs = lane == k1;
            internal = (word >> (rhs ? 1 : 0)) & 1u;
            id = rhs ? right : word >> 2;
            const uint2 g = internal ? __ldcg(info + id) : make_uint2(1u, 0u);
            size = g.x;
            height = g.y;
        }
        __syncwarp();
        if (lane == k0 || lane == k1) {
            const float a = half_area(w.box[lane]);
            cand = internal && a >= 0.f ? __float_as_uint(a) + 1u : 0u;
        }
        if (m == 0) {
            float rb[6];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                rb[a] = fminf(w.box[0][a], w.box[1][a]);
                rb[3 + a] = fmaxf(w.box[0][3 + a], w.box[1][3 + a]);
            }
            f.old_cost = half_area(rb);
        }
        m = k1 + 1u;
        if (m == (uint32_t)kTreeletLeaves) break;
        const uint32_t mx = __reduce_max_sync(0xFFFFFFFFu, lane < m ? cand : 0u);
        if (mx == 0u) break;
        k0 = (uint32_t)__ffs(__ballot_sync(0xFFFFFFFFu, lane < m && cand == mx)) - 1u;  // the first of largest area
        q = __shfl_sync(0xFFFFFFFFu, id, k0);
        f.old_cost = __fadd_rn(f.old_cost, __uint_as_float(mx - 1u));
    }
    if (!ok && lane == 0) atomicOr(status, CPT_STATUS_BAD_INDEX);
    f.m = ok ? m : 0u;
    f.internal_mask = __ballot_sync(0xFFFFFFFFu, lane < m && internal);
    if (lane < m) {
        w.id[lane] = id;
        w.size[lane] = size;
        w.height[lane] = height;
    }
    __syncwarp();
    return f;
}

__device__ __forceinline__ float treelet_cost(uint32_t address)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(address));
    return v;
}

// Subsets of kK leaves listed at subs, each shared by kG lanes (at most 32 lanes in all): the
// least c(P) + c(S \ P) over the splits P (with S's lowest leaf, P != S), the smallest P on
// equal sums. A lane goes through its splits in ascending order (sub - rest & rest steps
// through the subsets of rest); of kG lanes each fixes rest's highest log2(kG) leaves. Masks
// are byte offsets into c (4 x the subset), or-ed onto its address.
template <int kK, int kG>
__device__ __forceinline__ void treelet_class(const uint8_t* subs, int count, uint32_t full, uint32_t c_at,
                                              TreeletWarp& w)
{
    const int lane = threadIdx.x & 31;
    const int rho = lane / kG;
    const uint32_t S = rho < count ? subs[rho] : 0u;
    const bool valid = S != 0u && !(S & ~full);
    float best = INFINITY;
    uint32_t bp = 0xFFFFFFFFu;
    if (valid) {
        const uint32_t low = S & (0u - S), S4 = 4u * S;
        uint32_t rest = S ^ low, fixed = low;
        if (kG > 1) {
#pragma unroll
            for (int g = kG / 2; g >= 1; g /= 2) {
                const uint32_t top = 1u << (31 - __clz(rest));
                rest ^= top;
                if (lane & g) fixed |= top;
            }
        }
        rest *= 4u;
        fixed = c_at | 4u * fixed;
        // kG == 1: every split but P == S, the last; else that one is the last lane's last, and
        // (its lanes' first splits being real ones) is passed over by its sum
        constexpr int kSteps = (1 << (kK - 1)) / kG - (kG == 1 ? 1 : 0);
        uint32_t sub = 0;
        if (kG == 1 || kSteps > 1 || fixed != (c_at | S4)) {
            best = __fadd_rn(treelet_cost(fixed), treelet_cost(fixed ^ S4));
            bp = fixed;
        }
#pragma unroll
        for (int j = 1; j < kSteps; ++j) {
            sub = (sub - rest) & rest;
            const uint32_t P = fixed | sub;
            float v = __fadd_rn(treelet_cost(P), treelet_cost(P ^ S4));
            if (kG > 1 && j == kSteps - 1 && P == (c_at | S4)) v = INFINITY;
            if (v < best) { best = v; bp = P; }
        }
    }
#pragma unroll
    for (int o = 1; o < kG; o <<= 1) {
        const float ov = __shfl_xor_sync(0xFFFFFFFFu, best, o);
        const uint32_t op = __shfl_xor_sync(0xFFFFFFFFu, bp, o);
        if (ov < best || (ov == best && op < bp)) { best = ov; bp = op; }
    }
    if (valid && (lane % kG) == 0) {
        w.c[S] = __fadd_rn(w.c[S], best);
        w.split[S] = (uint8_t)((bp >> 2) & 127u);
    }
}

// Solves the warp's formed treelet (rooted at a node whose subtree is h_before tall)
// and rewrites it if cheaper and no taller; called by the whole warp.
__device__ __forceinline__ void treelet_solve(float* __restrict__ nodes, uint32_t* __restrict__ parents_leaf,
                                              uint32_t* __restrict__ parents_internal, uint2* __restrict__ info,
                                              uint32_t h_before, const TreeletForm& f, const uint8_t* order,
                                              TreeletWarp& w)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t m = f.m;
    if (m < 3) return;
    const uint32_t full = (1u << m) - 1u;
    // areas: the lane's bits pick among leaves 0-4, leaves 5 and 6 are added in turn
    {
        float b[6] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
        auto add = [&](float (&x)[6], int k) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                x[a] = fminf(x[a], w.box[k][a]);
                x[3 + a] = fmaxf(x[3 + a], w.box[k][3 + a]);
            }
        };
#pragma unroll
        for (int k = 0; k < 5; ++k)
            if ((lane >> k) & 1u)
                if (k < 3 || (uint32_t)k < m) add(b, k);
        auto put = [&](const float (&x)[6], uint32_t S) {
            if (S && !(S & ~full)) w.c[S] = __popc(S) == 1 ? 0.f : half_area(x);
        };
        put(b, lane);
        if (m > 6) {
            float c[6];
#pragma unroll
            for (int a = 0; a < 6; ++a) c[a] = b[a];
            add(c, 6);
            put(c, lane | 64u);
            add(c, 5);
            put(c, lane | 96u);
        }
        if (m > 5) {
            add(b, 5);
            put(b, lane | 32u);
        }
    }
    __syncwarp();
    // (the 33rd to 35th subsets of 3 and 4 leaves share lanes: 1 step instead of 3 and 7)
    const uint32_t c_at = (uint32_t)__cvta_generic_to_shared(w.c);
    treelet_class<2, 1>(order, 21, full, c_at, w);
    __syncwarp();
    treelet_class<3, 1>(order + 21, 32, full, c_at, w);
    if (m > 6) treelet_class<3, 4>(order + 53, 3, full, c_at, w);
    __syncwarp();
    if (m > 3) {
        treelet_class<4, 1>(order + 56, 32, full, c_at, w);
        if (m > 6) treelet_class<4, 8>(order + 88, 3, full, c_at, w);
        __syncwarp();
    }
    if (m > 4) {
        treelet_class<5, 1>(order + 91, 21, full, c_at, w);
        __syncwarp();
    }
    if (m > 5) {
        treelet_class<6, 4>(order + 112, 7, full, c_at, w);
        __syncwarp();
    }
    if (m > 6) {
        treelet_class<7, 32>(order + 119, 1, full, c_at, w);
        __syncwarp();
    }
    if (!(w.c[full] < __fmul_rn(f.old_cost, 0.999999f))) return;
    // the new topology, top-down
    if (lane == 0) {
        uint32_t cnt = 1;
        w.sub[0] = (uint8_t)full;
        w.node_depth[0] = 0;
        for (uint32_t j = 0; j < cnt; ++j) {
            const uint32_t S = w.sub[j], P = w.split[S], depth = w.node_depth[j] + 1u;
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const uint32_t X = side ? S ^ P : P;
                if (__popc(X) == 1) {
                    const uint32_t k = (uint32_t)__ffs(X) - 1u;
                    w.child[j][side] = (uint8_t)k;
                    w.leaf_depth[k] = (uint8_t)depth;
                } else {
                    w.child[j][side] = (uint8_t)(8u + cnt);
                    w.sub[cnt] = (uint8_t)X;
                    w.node_depth[cnt] = (uint8_t)depth;
                    ++cnt;  // (a binary tree over m leaves has m - 1 nodes)
                }
            }
        }
    }
    __syncwarp();
    // lanes 2 j and 2 j + 1: the two children of node j
    const uint32_t j = lane >> 1, side = lane & 1u;
    const bool mine = j < m - 1u;
    uint32_t h = 0, sz = 0;
    if (mine) {
        const uint32_t S = w.sub[j], d = w.node_depth[j];
        for (uint32_t k = 0; k < m; ++k)
            if ((S >> k) & 1u) {
                h = max(h, w.height[k] + w.leaf_depth[k] - d);
                sz += w.size[k];
            }
    }
    if (__shfl_sync(0xFFFFFFFFu, h, 0) > h_before) return;
    const uint32_t nd = mine ? w.inode[j] : 0u;
    uint32_t id = 0, bit = 0;
    if (mine) {
        const uint32_t c = w.child[j][side];
        float2* out = reinterpret_cast<float2*>(nodes + 24 * (size_t)nd + 10 * side);
        if (c < 8u) {
            id = w.id[c];
            const float2* s2 = reinterpret_cast<const float2*>(w.slot[c]);
#pragma unroll
            for (int a = 0; a < 5; ++a) out[a] = s2[a];
            bit = (f.internal_mask >> c) & 1u;
            (bit ? parents_internal : parents_leaf)[id] = nd;
        } else {
            const uint32_t X = w.sub[c - 8u];
            id = w.inode[c - 8u];
            bit = 1u;
            float b[6] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
            for (uint32_t k = 0; k < m; ++k)
                if ((X >> k) & 1u)
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        b[a] = fminf(b[a], w.box[k][a]);
                        b[3 + a] = fmaxf(b[3 + a], w.box[k][3 + a]);
                    }
            out[0] = make_float2(b[0], b[1]);
            out[1] = make_float2(b[2], b[3]);
            out[2] = make_float2(b[4], b[5]);
            out[3] = out[4] = make_float2(0.f, 0.f);
            parents_internal[id] = nd;
        }
    }
    const uint32_t rid = __shfl_xor_sync(0xFFFFFFFFu, id, 1), rbit = __shfl_xor_sync(0xFFFFFFFFu, bit, 1);
    if (mine && side == 0u) {
        const uint32_t word = (id << 2) | (rbit << 1) | bit;
        reinterpret_cast<float4*>(nodes + 24 * (size_t)nd)[5] =
            make_float4(__uint_as_float(word), __uint_as_float(rid), 0.f, 0.f);
        info[nd] = make_uint2(sz, h);
    }
    __threadfence();
    __syncwarp();  // the climbing lane's arrival at the next node releases every lane's stores
}

// A round of treelet restructuring over the split tree: every piece's walker goes
// up; the second arrival at a node records its size and height and, at gamma or
// more leaves, has its warp form and solve the node's treelet.
//
// Issue-bound (67 % of cycles) and behind it the chain of a treelet's dependent fetches. The
// whole warp forms, solves and rewrites a treelet: 11.8 M pieces (1.3 M-triangle hairball
// scene, ratio 8.0) in 12.0 ms against 23.8 when lane 0 gathered the leaves and wrote the
// new topology alone and the splits came from a table; the trees are the same bytes. 10
// blocks per SM (48 registers): with 9 the scene's whole build took 24.8 ms, with 10 24.6,
// with 12 25.1, with 16 (32 registers, spills) 26.4.
__global__ void __launch_bounds__(kTreeletBlock, 10) k_treelet(const uint32_t* __restrict__ n_pieces,
                                                          float* __restrict__ nodes,
                                                          const float4* __restrict__ leaf_boxes,
                                                          uint32_t* __restrict__ parents_leaf,
                                                          uint32_t* __restrict__ parents_internal,
                                                          int* __restrict__ counters, uint2* __restrict__ info,
                                                          uint32_t gamma, uint32_t* __restrict__ status)
{
    __shared__ uint8_t s_order[120];
    __shared__ TreeletWarp s_warp[kTreeletWarps];
    if (threadIdx.x < 120) s_order[threadIdx.x] = kTreeletOrder[threadIdx.x];
    __syncthreads();
    const uint32_t n = *n_pieces;
    if (n < 3) return;
    if (sort_timed_out(status)) return;  // (uniform over the launch: set before it started)
    TreeletWarp& w = s_warp[threadIdx.x >> 5];
    const uint32_t i = blockIdx.x * kTreeletBlock + threadIdx.x;
    bool active = i < n;
    uint32_t node = active ? parents_leaf[i] : CPT_INVALID_INDEX;
    uint32_t height = 0;
    for (int level = 0; __any_sync(0xFFFFFFFFu, active); ++level) {
        bool process = false;
        if (active) {
            if (node == CPT_INVALID_INDEX) {
                active = false;  // passed the root
            } else if (node >= n - 1 || level >= kTreeletMaxLevels) {
                atomicOr(status, CPT_STATUS_BAD_INDEX);
                active = false;
            } else {
                const int arrived = arrive_acq_rel(&counters[node]);
                if (arrived != 1) {
                    if (arrived != 0) atomicOr(status, CPT_STATUS_BAD_INDEX);
                    active = false;
                } else {
                    const float4 meta = __ldcg(reinterpret_cast<const float4*>(nodes + 24 * (size_t)node + 20));
                    const uint32_t word = __float_as_uint(meta.x);
                    const uint32_t ids[2] = {word >> 2, __float_as_uint(meta.y)};
                    uint32_t size = 0;
                    bool ok = true;
                    height = 0;
                    for (int side = 0; side < 2; ++side) {
                        if ((word >> side) & 1u) {
                            if (ids[side] >= n - 1) { ok = false; continue; }
                            const uint2 g = __ldcg(info + ids[side]);
                            size += g.x;
                            height = max(height, g.y);
                        } else {
                            if (ids[side] >= n) ok = false;
                            size += 1u;
                        }
                    }
                    if (!ok) {
                        atomicOr(status, CPT_STATUS_BAD_INDEX);
                        active = false;
                    } else {
                        height += 1u;
                        info[node] = make_uint2(size, height);
                        process = size >= gamma;
                    }
                }
            }
        }
        uint32_t todo = __ballot_sync(0xFFFFFFFFu, process);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1u;
            const uint32_t r = __shfl_sync(0xFFFFFFFFu, node, src);
            const uint32_t hr = __shfl_sync(0xFFFFFFFFu, height, src);
            const TreeletForm f = treelet_form(nodes, leaf_boxes, info, n, r, w, status);
            treelet_solve(nodes, parents_leaf, parents_internal, info, hr, f, s_order, w);
        }
        if (active) node = __ldcg(parents_internal + node);
    }
}

template <typename K>
struct SplitScratch {
    double* partial;
    double* total;
    uint32_t* counts;
    uint32_t* tile_sums;
    uint32_t* n_pieces;
    float4* pieces;
    K* keys[2];
    uint32_t* vals[2];
    uint32_t* hist;
    uint32_t* offsets;
    uint32_t* zero;
    size_t zero_words;
    uint32_t* children;
    uint32_t* parents_leaf;
    uint32_t* parents_internal;
    int* counters;
    cpt_bbox* node_boxes;
    float4* leaf_boxes;
    uint2* info;  // treelet restructuring: per internal node (leaves, height)
};

template <typename K>
size_t split_layout(uint32_t n, uint32_t cap, bool treelet, void* base, SplitScratch<K>* out)
{
    constexpr int P = KeyTraits<K>::passes;
    Carver c(base);
    SplitScratch<K> s;
    const uint32_t ctiles = (n + kScanTile - 1) / kScanTile;
    s.partial = c.take<double>(kWeightBlocks);
    s.total = c.take<double>(1);
    s.counts = c.take<uint32_t>(n);
    s.tile_sums = c.take<uint32_t>(ctiles);
    s.n_pieces = c.take<uint32_t>(1);
    s.pieces = c.take<float4>(2ull * cap);
    s.keys[0] = c.take<K>(cap);
    s.keys[1] = c.take<K>(cap);
    s.vals[0] = c.take<uint32_t>(cap);
    s.vals[1] = c.take<uint32_t>(cap);
    s.hist = c.take<uint32_t>((size_t)P * kRadix);
    s.offsets = c.take<uint32_t>((size_t)P * kRadix);
    s.zero_words = sort_zero_words(cap, P);
    s.zero = c.take<uint32_t>(sort_zero_reserve(cap, P));
    s.children = c.take<uint32_t>(cap);
    s.parents_leaf = c.take<uint32_t>(cap);
    s.parents_internal = c.take<uint32_t>(cap);
    s.counters = c.take<int>(cap);
    s.node_boxes = c.take<cpt_bbox>(cap);
    s.leaf_boxes = c.take<float4>(2ull * cap);
    s.info = treelet ? c.take<uint2>(cap) : nullptr;
    if (out) *out = s;
    return c.used();
}

inline uint64_t split_capacity(uint32_t n, float extra_ratio)
{
    const double r = extra_ratio > 0.f ? (double)extra_ratio : 0.0;
    return (uint64_t)n + (uint64_t)floor(r * (double)n);
}

template <typename K>
int split_impl(cpt_bvh* bvh, uint32_t cap, bool treelet, void* nodes, void* scratch,
               cudaStream_t stream)
{
    constexpr int P = KeyTraits<K>::passes;
    const uint32_t n = bvh->n;
    SplitScratch<K> s;
    split_layout<K>(n, cap, treelet, scratch, &s);
    const uint32_t ctiles = (n + kScanTile - 1) / kScanTile;
    const double extra = (double)(cap - n);
    CPT_CUDA_TRY(cudaMemsetAsync(s.hist, 0, sizeof(uint32_t) * P * kRadix, stream));
    k_split_weight<<<kWeightBlocks, kSplitBlock, 0, stream>>>(bvh->tris, n, s.partial);
    CPT_LAUNCH_CHECK();
    k_split_total<<<1, kWeightBlocks, 0, stream>>>(s.partial, s.total);
    CPT_LAUNCH_CHECK();
    k_split_count<<<ctiles, kSplitBlock, 0, stream>>>(bvh->tris, n, s.total, extra, s.counts, s.tile_sums);
    CPT_LAUNCH_CHECK();
    k_split_scan_tiles<<<1, 1024, 0, stream>>>(s.tile_sums, ctiles, cap, s.n_pieces, bvh->status);
    CPT_LAUNCH_CHECK();
    uint32_t* owner = s.children;  // (free until the topology is built)
    k_split_first<<<ctiles, kSplitBlock, 0, stream>>>(n, s.counts, s.tile_sums, owner, cap);
    CPT_LAUNCH_CHECK();
    const uint32_t eblocks = (uint32_t)(((uint64_t)cap + (uint64_t)kSplitBlock * kEmitPieces - 1) /
                                        ((uint64_t)kSplitBlock * kEmitPieces));
    k_split_emit<K><<<eblocks, kSplitBlock, 0, stream>>>(bvh->tris, n, s.counts, owner, s.n_pieces, bvh->node_boxes,
                                                         s.pieces, s.keys[0], s.hist, s.zero, s.zero_words);
    CPT_LAUNCH_CHECK();
    launch_early(start_early(cap), k_scan_offsets, P, kRadix, 0, stream, s.hist, s.offsets);
    CPT_LAUNCH_CHECK();
    const uint32_t tiles = sort_tiles(cap);
    uint32_t* lookback = s.zero + 32;
    const K* keys;
    if constexpr (sizeof(K) == 8) {  // as 32-bit halves: the sorted keys end in keys[1]
        if (const int rc = onesweep_sort64_halves(reinterpret_cast<const uint64_t*>(s.keys[0]),
                                                  reinterpret_cast<uint64_t*>(s.keys[1]), cap, 0, s.n_pieces, s.vals,
                                                  s.offsets, lookback, s.zero, bvh->status, SortWait(), true, false,
                                                  stream))
            return rc;
        keys = s.keys[1];
    } else {
        for (int p = 0; p < P; ++p) {
            const K* kin = s.keys[p & 1];
            K* kout = s.keys[(p + 1) & 1];
            const uint32_t* vin = p == 0 ? nullptr : s.vals[(p + 1) & 1];
            uint32_t* vout = s.vals[p & 1];
            uint32_t* lb = lookback + (size_t)p * tiles * kRadix;
            const int rc = p == 0 ? onesweep_launch<K, true>(kin, vin, kout, vout, cap, 0, s.n_pieces, 0, s.offsets, lb,
                                                             s.zero, bvh->status, SortWait(), stream)
                                  : onesweep_launch<K, false>(kin, vin, kout, vout, cap, 0, s.n_pieces, 8 * p,
                                                              s.offsets + p * kRadix, lb, s.zero + p, bvh->status,
                                                              SortWait(), stream);
            if (rc) return rc;
        }
        keys = s.keys[P & 1];
    }
    const uint32_t* order = s.vals[(P - 1) & 1];
    // the list of finished subtrees: the other value and key buffers, free after the sort,
    // counted in a word that k_split_emit zeroed
    const TreeArrays<K> T{keys,        0u, s.children, s.parents_leaf, s.parents_internal, static_cast<float*>(nodes),
                          s.node_boxes, s.counters, bvh->status};
    const PieceLeaves leaf{bvh->tris, s.pieces, order, s.leaf_boxes, 0u, n, bvh->status};
    const TreeList list{s.vals[P & 1], reinterpret_cast<uint32_t*>(keys == s.keys[0] ? s.keys[1] : s.keys[0]),
                        s.zero + kTreeListWord};
    const uint32_t blocks = (cap + kTreeBlock - 1) / kTreeBlock;
    CPT_CUDA_TRY(cudaFuncSetAttribute(k_split_tree_blocks<K>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      kTreeCarveout));
    launch_early(start_early(cap), k_split_tree_blocks<K>, blocks, kTreeBlock, 0, stream, T, leaf, list, s.n_pieces,
                 cap - 1);
    CPT_LAUNCH_CHECK();
    launch_early(start_early(cap), k_split_tree_top<K>, tree_top_blocks(blocks, sm_count()), 128, 0, stream, T, leaf, list,
                 s.n_pieces);
    CPT_LAUNCH_CHECK();
    if (treelet) {
        for (int round = 0; round < kTreeletRounds; ++round) {
            CPT_CUDA_TRY(cudaMemsetAsync(s.counters, 0, sizeof(int) * (size_t)cap, stream));
            k_treelet<<<(cap + kTreeletBlock - 1) / kTreeletBlock, kTreeletBlock, 0, stream>>>(
                s.n_pieces, static_cast<float*>(nodes), s.leaf_boxes, s.parents_leaf, s.parents_internal, s.counters,
                s.info, (uint32_t)kTreeletGamma << (CPT_TREELET_GAMMA_SHIFT * round), bvh->status);
            CPT_LAUNCH_CHECK();
        }
    }
    return CPT_OK;
}

}  // namespace
}  // namespace cpt

using namespace cpt;

extern "C" size_t cpt_lbvh_split_bytes(uint32_t n, int morton_bits, float extra_ratio, uint32_t flags,
                                       size_t* node_bytes)
{
    if (n < 2 || n > kMaxTriangles || (morton_bits != 30 && morton_bits != 63)) return 0;
    if (!(extra_ratio >= 0.f) || !(extra_ratio <= 64.f)) return 0;  // the range cpt_lbvh_split accepts
    const bool treelet = flags & CPT_SPLIT_TREELET;
    if (flags & ~CPT_SPLIT_TREELET) return 0;
    const uint64_t cap = split_capacity(n, extra_ratio);
    if (cap >= (1ull << 31)) return 0;
    if (node_bytes) *node_bytes = align_up((size_t)(cap - 1) * 96, 256);
    return morton_bits == 30 ? split_layout<uint32_t>(n, (uint32_t)cap, treelet, nullptr, nullptr)
                             : split_layout<uint64_t>(n, (uint32_t)cap, treelet, nullptr, nullptr);
}

extern "C" int cpt_lbvh_split(cpt_bvh* bvh, float extra_ratio, uint32_t flags, void* nodes, size_t node_bytes,
                              void* scratch, size_t scratch_bytes, cudaStream_t stream)
{
    CPT_RANGE("cpt_lbvh_split");
    if (!bvh || !bvh->tris || !bvh->node_boxes || !bvh->status || !nodes || !scratch) return CPT_ERR_INVALID_ARGUMENT;
    if (!(extra_ratio >= 0.f) || !(extra_ratio <= 64.f)) return CPT_ERR_INVALID_ARGUMENT;
    size_t nb = 0;
    const size_t need = cpt_lbvh_split_bytes(bvh->n, bvh->morton_bits, extra_ratio, flags, &nb);
    if (!need) return CPT_ERR_INVALID_ARGUMENT;
    if (scratch_bytes < need || node_bytes < nb) return CPT_ERR_SCRATCH_TOO_SMALL;
    if ((reinterpret_cast<uintptr_t>(nodes) & 15) || (reinterpret_cast<uintptr_t>(scratch) & 255))
        return CPT_ERR_INVALID_ARGUMENT;
    const uint32_t cap = (uint32_t)split_capacity(bvh->n, extra_ratio);
    const bool treelet = flags & CPT_SPLIT_TREELET;
    const int rc = bvh->morton_bits == 30 ? split_impl<uint32_t>(bvh, cap, treelet, nodes, scratch, stream)
                                          : split_impl<uint64_t>(bvh, cap, treelet, nodes, scratch, stream);
    if (rc) return rc;
    bvh->split_nodes = nodes;
    bvh->split_capacity = cap;
    bvh->wide_nodes = nullptr;  // a wide tree of the previous binary tree is stale
    bvh->wide_tris = nullptr;
    bvh->wide_capacity = 0;
    return CPT_OK;
}
