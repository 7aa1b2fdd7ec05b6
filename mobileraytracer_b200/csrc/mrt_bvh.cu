// mrt_bvh.cu - BVH construction.
//
// REFERENCE tree: BVH<T>::BVH + build + getSplitIndex_SAH (BVH.hpp:64-155, 273-311) restated on the
// host with the same float operations and node numbering, then uploaded.  The reference never
// reorders primitives, so leaf offsets index the input arrays.
//
// FAST tree: built on the device.  Triangle boxes padded outward -> 30-bit Morton codes of the
// centroids, cells halved along their longest side -> stable LSD radix sort (own kernels) -> Karras'
// parallel hierarchy ("Maximizing parallelism in the construction of BVHs, octrees and k-d trees", HPG
// 2012) -> bottom-up box fit, which also works out for every binary node the cheapest way to turn its subtree into wide
// nodes -> the binary tree collapsed along those choices into 8-wide nodes with 16-bit quantised
// child boxes (128 bytes: one cache line per traversal step), children placed in slots by octant,
// internal children numbered consecutively, the leaf children's triangles copied to consecutive
// 48-byte records.  A traversal step of the 8-wide tree replaces about three of the binary tree's,
// shortening the chain of dependent node fetches per ray.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "mrt_internal.h"

using namespace mrt;
using namespace mrt_host;

namespace {

// ============================== reference tree (host) =======================================
struct HBox {
    V3 mn, mx;
};

HBox hunion(const HBox &b1, const HBox &b2) { return HBox{vmin(b1.mn, b2.mn), vmax(b1.mx, b2.mx)}; }   // AABB.cpp:52-60
float harea(const HBox &b) {   // AABB.cpp:37-49
    const float lx = b.mx.x - b.mn.x, ly = b.mx.y - b.mn.y, lz = b.mx.z - b.mn.z;
    const float bt = 2 * lx * lz, xy = 2 * lx * ly, zy = 2 * lz * ly;
    return bt + xy + zy;
}

uint32_t sah_split(const HBox *boxes, uint32_t N, std::vector<float> &la, std::vector<float> &ra) {
    const uint32_t L = 2;
    la.assign(N - L, 0.0f);
    ra.assign(N - L, 0.0f);
    HBox lb = boxes[0];
    la[0] = harea(lb);
    for (uint32_t i = 1; i < N - L; ++i) { lb = hunion(lb, boxes[i]); la[i] = harea(lb); }
    HBox rb = boxes[N - 1];
    ra[N - L - 1] = harea(rb);
    for (uint32_t i = N - 2; i > L; --i) { rb = hunion(rb, boxes[i]); ra[i - L] = harea(rb); }
    uint32_t split = L;
    float min_sah = (float)L * la[L - 1] + (float)(N - L) * ra[L - 1];
    for (uint32_t i = L; i < N - L; ++i) {
        const float sl = (float)(i + 1) * la[i];
        const float sr = (float)(N - (i + 1)) * ra[i];
        const float sah = sl + sr;
        if (sah < min_sah) { split = i + 1; min_sah = sah; }
    }
    return split;
}

std::vector<RefNode> ref_build(const std::vector<HBox> &pboxes) {
    const uint32_t N = (uint32_t)pboxes.size();
    if (N == 0) return std::vector<RefNode>(1, RefNode{{0, 0, 0}, {0, 0, 0}, 0, 0});
    std::vector<RefNode> nodes(2 * (size_t)N - 1, RefNode{{0, 0, 0}, {0, 0, 0}, 0, 0});
    std::vector<HBox> boxes(N);
    std::vector<float> la, ra;
    uint32_t st_id[512] = {0}, st_b[512] = {0}, st_e[512] = {0};
    uint32_t sp = 1, id = 0, begin = 0, end = N, max_id = 0;
    do {
        HBox nb = pboxes[begin];
        boxes[0] = nb;
        const uint32_t size = end - begin;
        for (uint32_t i = begin + 1; i < end; ++i) {
            nb = hunion(pboxes[i], nb);
            boxes[i - begin] = pboxes[i];
        }
        RefNode &nd = nodes[id];
        nd.mn[0] = nb.mn.x; nd.mn[1] = nb.mn.y; nd.mn[2] = nb.mn.z;
        nd.mx[0] = nb.mx.x; nd.mx[1] = nb.mx.y; nd.mx[2] = nb.mx.z;
        if (size <= 2) {
            nd.offset = begin;
            nd.count = size;
            --sp; id = st_id[sp]; begin = st_b[sp]; end = st_e[sp];
        } else {
            const uint32_t left = max_id + 1, right = left + 1;
            nd.offset = left;
            max_id = std::max(right, max_id);
            const uint32_t split = size <= 4 ? 2 : sah_split(boxes.data(), size, la, ra);
            if (sp >= 512) break;   // the reference's fixed 512-entry stack (BVH.hpp:93-95)
            st_id[sp] = right; st_b[sp] = begin + split; st_e[sp] = end; ++sp;
            id = left;
            end = begin + split;
        }
    } while (sp > 0);
    nodes.resize(max_id + 1);
    return nodes;
}

// ============================== FAST tree (device) ===========================================
constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;

// padded triangle boxes (min.xyz, max.xyz as two float4) and the centroid bounds
__global__ void k_tri_boxes(uint32_t n, const float4 *__restrict__ a4, const float4 *__restrict__ ab4,
                            const float4 *__restrict__ ac4, float4 *bmin, float4 *bmax, uint32_t *cbounds) {
    __shared__ uint32_t smin[3][32], smax[3][32];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float c[3] = {0, 0, 0};
    bool valid = i < n;
    if (valid) {
        const V3 A = v3(a4[i]), ab = v3(ab4[i]), ac = v3(ac4[i]);
        const V3 B = A + ab, C = A + ac;
        V3 mn = vmin(A, vmin(B, C)), mx = vmax(A, vmax(B, C));
        const float m = fmaxf(fmaxf(fmaxf(fabsf(mn.x), fabsf(mx.x)), fmaxf(fabsf(mn.y), fabsf(mx.y))),
                              fmaxf(fabsf(mn.z), fabsf(mx.z)));
        const float e = fmaxf(fmaxf(mx.x - mn.x, mx.y - mn.y), mx.z - mn.z);
        const float pad = 4e-6f * m + 2e-5f * e + 1e-30f;
        mn = subs(mn, pad);
        mx = adds(mx, pad);
        bmin[i] = make_float4(mn.x, mn.y, mn.z, 0.0f);
        bmax[i] = make_float4(mx.x, mx.y, mx.z, 0.0f);
        c[0] = 0.5f * (mn.x + mx.x); c[1] = 0.5f * (mn.y + mx.y); c[2] = 0.5f * (mn.z + mx.z);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < 3; ++k) {
        uint32_t lo = valid ? float_order(c[k]) : 0xFFFFFFFFu, hi = valid ? float_order(c[k]) : 0u;
        for (int o = 16; o > 0; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
        }
        if (lane == 0) { smin[k][warp] = lo; smax[k][warp] = hi; }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int k = threadIdx.x;
        uint32_t lo = 0xFFFFFFFFu, hi = 0u;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { lo = min(lo, smin[k][w]); hi = max(hi, smax[k][w]); }
        atomicMin(&cbounds[k], lo);
        atomicMax(&cbounds[3 + k], hi);
    }
}

// 30 bits along the three axes of the centroid bounds: each halves the cells along their longest side, an axis at
// most 13 times.  Sides are compared by their octave (equal ones: x, y, z in turn): by their lengths, a soup whose
// bounds are a thousandth off a cube gets another order of the axes, and its 1080p frame took 1,135 us, not 1,112.
// Ten bits an axis in turn, whatever the sides, cut flat scenes across their thin axis as often as along the
// others; cubes of a 1024th of the longest side leave a model with one far triangle beside it a handful of cells.
// Surface-area cost of the binary tree of 300,000 triangles against ten bits an axis in turn: sides 1 : 0.2 : 1
// 0.78 (cubes 0.78), 100 : 1 : 1 0.30 (0.31), a cube of side 2 and one triangle 30, 200, 1,000 and 10^6 away 0.63,
// 0.33, 0.21 and 1.00 (0.65, 1.61, 19.9, 84.6).  At most 10, 12 or 14 bits an axis: 0.58, 0.26 and 0.20 at 1,000,
// 1.00, 1.00 and 1.01 at 10^6.  Nodes that a random ray visits in a soup of 1,000,000 alone 49, with a triangle
// 200, 1,000 and 10^4 away 53, 58 and 177 (472, 16,163 and 100,530 with cubes, 149, 291 and 315 with ten bits in
// turn); in the 524,288-triangle heightfield 6.2 (6.3, 7.2).
constexpr int kCodeBits = 30, kAxisBits = 13;
__global__ void __launch_bounds__(256) k_morton(uint32_t n, const float4 *__restrict__ bmin, const float4 *__restrict__ bmax,
                                                const uint32_t *__restrict__ cbounds, uint32_t *keys, uint32_t *vals) {
    __shared__ uint8_t axis_of[3 * kAxisBits];   // by place from the top bit
    float mn[3], ext[3];
    for (int k = 0; k < 3; ++k) {
        mn[k] = order_float(cbounds[k]);
        ext[k] = order_float(cbounds[3 + k]) - mn[k];
        if (!(ext[k] > 0.0f && ext[k] <= 3.0e38f)) ext[k] = 0.0f;   // finite sides only
    }
    if (threadIdx.x < 3 * kAxisBits) {   // halving h of axis a goes behind those of longer cells
        const float side = fmaxf(ext[0], fmaxf(ext[1], ext[2]));
        int octave[3];
        for (int k = 0; k < 3; ++k) octave[k] = ext[k] > 0.0f ? (int)rintf(log2f(side / ext[k])) : 1024;
        const int a = threadIdx.x / kAxisBits, h = threadIdx.x % kAxisBits, own = octave[a] + h;
        int place = 0;
        for (int k = 0; k < 3; ++k)   // halvings j of axis k with octave[k] + j below own, or equal and k below a
            place += min(max(own - octave[k] + (k < a ? 1 : 0), 0), kAxisBits);
        axis_of[place] = (uint8_t)a;
    }
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 lo = bmin[i], hi = bmax[i];
    const float c[3] = {0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z)};
    uint32_t q[3];   // the place along an axis, top bit first
    for (int k = 0; k < 3; ++k) {
        float u = ext[k] > 0.0f ? (c[k] - mn[k]) / ext[k] : 0.5f;
        u = fminf(fmaxf(u, 0.0f), 1.0f);
        q[k] = min((uint32_t)(u * (float)(1 << kAxisBits)), (1u << kAxisBits) - 1u) << (32 - kAxisBits);
    }
    uint32_t code = 0;
    for (int b = 0; b < kCodeBits; ++b) {
        const int a = axis_of[b];
        const uint32_t v = a == 0 ? q[0] : a == 1 ? q[1] : q[2];
        code = code << 1 | v >> 31;
        if (a == 0) q[0] <<= 1;
        else if (a == 1) q[1] <<= 1;
        else q[2] <<= 1;
    }
    keys[i] = code;
    vals[i] = i;
}

// --- stable LSD radix sort, 8-bit digits --------------------------------------------------------
__global__ void k_rs_hist(const uint32_t *__restrict__ keys, uint32_t n, int shift, uint32_t *hist, uint32_t nblocks) {
    __shared__ uint32_t cnt[256];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * kSortTile;
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t e = base + r * kSortThreads + threadIdx.x;
        if (e < n) atomicAdd(&cnt[(keys[e] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * nblocks + blockIdx.x] = cnt[threadIdx.x];
}

// exclusive scan of each digit's row of per-block counts in place (one block of 256 threads per
// digit), the row sums to total[digit]; k_rs_scatter adds the digits before a row.  (One block over
// all 256 rows took 105 us a pass at 1,000,000 keys, 12 % of the build's kernels; the rows take 3 us.)
__global__ void __launch_bounds__(256) k_rs_scan_rows(uint32_t *hist, uint32_t nblocks, uint32_t *total) {
    __shared__ uint32_t wsum[8];
    uint32_t *row = hist + (size_t)blockIdx.x * nblocks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint32_t b = 0; b < nblocks; b += 256) {
        const uint32_t i = b + threadIdx.x;
        const uint32_t v = i < nblocks ? row[i] : 0u;
        uint32_t incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t w = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += w;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        uint32_t before = 0, all = 0;
        for (int w = 0; w < 8; ++w) {
            if (w < warp) before += wsum[w];
            all += wsum[w];
        }
        if (i < nblocks) row[i] = carry + before + incl - v;
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

__global__ void k_rs_scatter(const uint32_t *__restrict__ kin, const uint32_t *__restrict__ vin, uint32_t *kout,
                             uint32_t *vout, uint32_t n, int shift, const uint32_t *__restrict__ hist, uint32_t nblocks,
                             const uint32_t *__restrict__ digit_total) {
    __shared__ uint32_t base[256], running[256], total[256];
    __shared__ uint32_t wcnt[kSortThreads / 32][256];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    {   // the keys of smaller digits, then this block's place in its digit's row
        const uint32_t v = digit_total[tid];
        uint32_t incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t w = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += w;
        }
        if (lane == 31) total[warp] = incl;
        __syncthreads();
        uint32_t before = 0;
        for (int w = 0; w < warp; ++w) before += total[w];
        base[tid] = before + incl - v + hist[tid * nblocks + blockIdx.x];
        __syncthreads();
    }
    running[tid] = 0;
    const uint32_t lt_mask = (1u << lane) - 1u;
    for (int r = 0; r < kSortItems; ++r) {
        for (int w = 0; w < kSortThreads / 32; ++w) wcnt[w][tid] = 0;
        __syncthreads();
        const uint32_t e = blockIdx.x * kSortTile + r * kSortThreads + tid;
        const bool valid = e < n;
        uint32_t key = 0, val = 0, d = 256;
        if (valid) { key = kin[e]; val = vin[e]; d = (key >> shift) & 255u; }
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
        const uint32_t rank = __popc(peers & lt_mask);
        if (valid && rank == 0) wcnt[warp][d] = __popc(peers);
        __syncthreads();
        {
            uint32_t acc = 0;
            for (int w = 0; w < kSortThreads / 32; ++w) { const uint32_t c = wcnt[w][tid]; wcnt[w][tid] = acc; acc += c; }
            total[tid] = acc;
        }
        __syncthreads();
        if (valid) {
            const uint32_t pos = base[d] + running[d] + wcnt[warp][d] + rank;
            kout[pos] = key;
            vout[pos] = val;
        }
        __syncthreads();
        running[tid] += total[tid];
    }
}

// --- Karras hierarchy --------------------------------------------------------------------------
__device__ __forceinline__ int kdelta(const uint32_t *keys, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const uint32_t a = keys[i], b = keys[j];
    if (a == b) return 32 + __clz((uint32_t)(i ^ j));
    return __clz(a ^ b);
}

constexpr uint32_t kLeafBit = 0x80000000u;

__global__ void k_karras(int n, const uint32_t *__restrict__ keys, uint32_t *left, uint32_t *right, uint32_t *first,
                         uint32_t *last, uint32_t *parent_int, uint32_t *parent_leaf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = (kdelta(keys, n, i, i + 1) - kdelta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = kdelta(keys, n, i, i - d);
    int lmax = 2;
    while (kdelta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (kdelta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = kdelta(keys, n, i, j);
    int s = 0;
    for (int t = (l + 1) >> 1;; t = (t + 1) >> 1) {
        if (kdelta(keys, n, i, i + (s + t) * d) > dnode) s += t;
        if (t == 1) break;
    }
    const int gamma = i + s * d + min(d, 0);
    const int f = min(i, j), la = max(i, j);
    const uint32_t lc = (f == gamma) ? (kLeafBit | (uint32_t)gamma) : (uint32_t)gamma;
    const uint32_t rc = (la == gamma + 1) ? (kLeafBit | (uint32_t)(gamma + 1)) : (uint32_t)(gamma + 1);
    left[i] = lc;
    right[i] = rc;
    first[i] = (uint32_t)f;
    last[i] = (uint32_t)la;
    if (lc & kLeafBit) parent_leaf[lc & ~kLeafBit] = (uint32_t)i; else parent_int[lc] = (uint32_t)i;
    if (rc & kLeafBit) parent_leaf[rc & ~kLeafBit] = (uint32_t)i; else parent_int[rc] = (uint32_t)i;
}

__device__ __forceinline__ void child_box(uint32_t c, const uint32_t *__restrict__ vals, const float4 *bmin,
                                          const float4 *bmax, const float4 *imin, const float4 *imax, float4 &lo,
                                          float4 &hi) {
    if (c & kLeafBit) {
        const uint32_t t = vals[c & ~kLeafBit];
        lo = bmin[t];
        hi = bmax[t];
    } else {
        lo = __ldcg(&imin[c]);
        hi = __ldcg(&imax[c]);
    }
}

__device__ __forceinline__ float half_area(float4 lo, float4 hi) {
    const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return dx * dy + dy * dz + dz * dx;
}

// --- the cheapest wide nodes of every subtree --------------------------------------------------------
// Ylitie, Karras and Laine, "Efficient Incoherent Ray Traversal on GPUs Through Compressed Wide BVHs"
// (HPG 2017), section 3.1: C(n, j) = the least surface-area cost of a binary subtree n held in at most j
// child slots of a wide node, j = 1..7.  One slot holds a leaf of up to leaf_max triangles (kTriCost x
// triangles x box area) or a wide node of its own (box area x kNodeCost + the best split of 8 slots over
// n's two children); more slots hold the best split of j over the two children, or fewer of them.  The
// costs of a node and the choices behind them (one word) are worked out bottom-up in the pass that fits
// the boxes: 28 additions and comparisons a node.  Against opening the largest child until a node is
// full, the nodes visited per camera ray go from 24.8 to 23.6 on the 1,000,000-triangle soup (tree
// 36.4 -> 30 MB) and from 9.1 to 8.8 on the heightfield (14.4 -> 13.8 after a bounce; 12.2 -> 7.9 MB).
#ifndef MRT_BVH_TRI_COST
#define MRT_BVH_TRI_COST 0.9f
#endif
constexpr float kTriCost = MRT_BVH_TRI_COST, kNodeCost = 1.0f;

struct SlotCosts {      // 32 bytes per binary internal node
    float c[7];         // C(n, 1..7)
    uint32_t choice;    // bit 0: one slot holds a leaf; bits 1-3: slots of the left child when n is a wide
                        // node (of 8); bits 4 + 3 (j - 2)..: slots of the left child out of j (0: as j - 1)
};
__device__ __forceinline__ uint32_t choice_node_split(uint32_t choice) { return (choice >> 1) & 7u; }
__device__ __forceinline__ uint32_t choice_split(uint32_t choice, uint32_t j) { return (choice >> (4u + 3u * (j - 2u))) & 7u; }

__device__ __forceinline__ void child_costs(uint32_t c, float4 lo, float4 hi, const SlotCosts *costs, float (&out)[7]) {
    if (c & kLeafBit) {
        const float a = kTriCost * half_area(lo, hi);
        for (int j = 0; j < 7; ++j) out[j] = a;
        return;
    }
    const float4 a = __ldcg(reinterpret_cast<const float4 *>(&costs[c])), b = __ldcg(reinterpret_cast<const float4 *>(&costs[c]) + 1);
    out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w; out[4] = b.x; out[5] = b.y; out[6] = b.z;
}

// least L(k) + R(j - k) over k = 1..j-1 (at most 7 slots a side)
template <int J>
__device__ __forceinline__ float best_split(const float (&l)[7], const float (&r)[7], uint32_t &k_best) {
    float best = l[0] + r[J - 2 < 6 ? J - 2 : 6];
    k_best = 1;
#pragma unroll
    for (int k = 2; k < J; ++k) {
        const float v = l[k - 1] + r[J - k - 1];
        if (v < best) { best = v; k_best = (uint32_t)k; }
    }
    return best;
}

template <int J>
__device__ __forceinline__ void cost_of_slots(const float (&l)[7], const float (&r)[7], SlotCosts &s) {
    uint32_t k;
    const float v = best_split<J>(l, r, k);
    // (on a tie the split: subtrees without area still fill their nodes)
    if (v <= s.c[J - 2]) { s.c[J - 1] = v; s.choice |= k << (4 + 3 * (J - 2)); }
    else s.c[J - 1] = s.c[J - 2];
}

__global__ void k_fit(int n, int leaf_max, const uint32_t *__restrict__ vals, const float4 *__restrict__ bmin,
                      const float4 *__restrict__ bmax, const uint32_t *__restrict__ left, const uint32_t *__restrict__ right,
                      const uint32_t *__restrict__ first, const uint32_t *__restrict__ last,
                      const uint32_t *__restrict__ parent_int, const uint32_t *__restrict__ parent_leaf, uint32_t *counter,
                      float4 *imin, float4 *imax, SlotCosts *costs) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    uint32_t node = parent_leaf[j];
    for (int guard = 0; guard < 4096 && node < (uint32_t)(n - 1); ++guard) {
        __threadfence();
        if (atomicAdd(&counter[node], 1u) == 0u) return;   // the other child is not ready yet
        const uint32_t lc = left[node], rc = right[node];
        float4 l0, l1, r0, r1;
        child_box(lc, vals, bmin, bmax, imin, imax, l0, l1);
        child_box(rc, vals, bmin, bmax, imin, imax, r0, r1);
        const float4 lo = make_float4(fminf(l0.x, r0.x), fminf(l0.y, r0.y), fminf(l0.z, r0.z), 0.0f);
        const float4 hi = make_float4(fmaxf(l1.x, r1.x), fmaxf(l1.y, r1.y), fmaxf(l1.z, r1.z), 0.0f);
        __stcg(&imin[node], lo);
        __stcg(&imax[node], hi);
        float l[7], r[7];
        child_costs(lc, l0, l1, costs, l);
        child_costs(rc, r0, r1, costs, r);
        SlotCosts s;
        const float area = half_area(lo, hi);
        uint32_t k8;
        const float as_node = kNodeCost * area + best_split<8>(l, r, k8);
        const uint32_t tris = last[node] - first[node] + 1u;
        const float as_leaf = kTriCost * (float)tris * area;
        const bool leaf = tris <= (uint32_t)leaf_max && as_leaf <= as_node;
        s.c[0] = leaf ? as_leaf : as_node;
        s.choice = (leaf ? 1u : 0u) | (k8 << 1);
        cost_of_slots<2>(l, r, s);
        cost_of_slots<3>(l, r, s);
        cost_of_slots<4>(l, r, s);
        cost_of_slots<5>(l, r, s);
        cost_of_slots<6>(l, r, s);
        cost_of_slots<7>(l, r, s);
        __stcg(reinterpret_cast<float4 *>(&costs[node]), make_float4(s.c[0], s.c[1], s.c[2], s.c[3]));
        __stcg(reinterpret_cast<float4 *>(&costs[node]) + 1, make_float4(s.c[4], s.c[5], s.c[6], __uint_as_float(s.choice)));
        if (node == 0) return;
        node = parent_int[node];
    }
}

// ------------------------------ binary -> 8-wide compressed nodes ------------------------------
// A wide node holds its binary node's two children in 8 slots by the choices above.  Its box is the
// union of the children's boxes; per axis the children's planes are quantised on a grid p + 2^E q
// (16-bit q, lo rounded down and hi up, so every quantised box contains the exact one), the children
// are placed in slots by the octant of their centre within the node, internal children get consecutive
// node indices (one allocation per node), and the triangles of the leaf children are copied to
// consecutive records (one allocation per node).  One launch per level of the wide tree; a level's size
// stays on the device (ctrs), so levels follow each other without a host round trip.
struct CollapseItem {
    uint32_t bin;     // binary node (kLeafBit: a single triangle, the whole scene)
    uint32_t node;    // the wide node it becomes
};

struct BinTree {
    const uint32_t *vals;             // triangle of each place in Morton order
    const float4 *bmin, *bmax;        // triangle boxes
    const uint32_t *left, *right, *first, *last;
    const float4 *imin, *imax;        // inner boxes
    const SlotCosts *costs;
    uint32_t n;
    __device__ bool is_leaf(uint32_t c) const { return (c & kLeafBit) || (costs[c].choice & 1u); }
};

// ctrs: [0] nodes allocated, [1] error, [2] triangles placed, [kLevelCtr + l] items of level l
constexpr int kLevelCtr = 4, kMaxLevels = 68;   // the binary tree is at most 62 levels deep

// grid step exponent E of one axis (2^E >= extent / 65534)
__device__ __forceinline__ int grid_exponent(float lo, float hi) {
    const double want = ((double)hi - (double)lo) / 65534.0;
    if (!(want > 0x1p-126)) return -126;
    int ex = 0;
    const double m = frexp(want, &ex);   // want = m 2^ex, m in [0.5, 1)
    return m == 0.5 ? ex - 1 : ex;
}
// a child's planes on the grid of step 1 / inv_step (a power of two), lo rounded down and hi up (with a
// 2^-20 step guard against the rounding of the double-precision subtraction), as lo | hi << 16
__device__ __forceinline__ uint32_t quantise(float p, double inv_step, float lo, float hi) {
    double ql = floor(((double)lo - (double)p) * inv_step - 0x1p-20);
    double qh = ceil(((double)hi - (double)p) * inv_step + 0x1p-20);
    ql = fmin(fmax(ql, 0.0), 65535.0);
    qh = fmin(fmax(qh, 0.0), 65535.0);
    return (uint32_t)ql | ((uint32_t)qh << 16);
}

// Eight lanes make one wide node, a lane per child.  (One thread per node, its 512 slot
// comparisons and 48 double-precision divisions in a row, took 20 to 30 us a level however few its nodes; a
// 200,003-triangle scene opened and rendered once took 2.58 ms, 2.32 now.)
constexpr int kCollapseThreads = 128, kGroups = kCollapseThreads / kWide;
__global__ void __launch_bounds__(kCollapseThreads) k_collapse(BinTree t, const CollapseItem *__restrict__ in, int level,
                                                               CollapseItem *out, uint32_t cap, uint32_t *nodes,
                                                               const float4 *__restrict__ a4, const float4 *__restrict__ ab4,
                                                               const float4 *__restrict__ ac4, float4 *tris, uint32_t *ctrs) {
    if (ctrs[1]) return;   // after an error the level's items may be unwritten
    const uint32_t n_in = min(ctrs[kLevelCtr + level], cap);
    const int lane = threadIdx.x & (kWide - 1), group = threadIdx.x / kWide;
    const int lane0 = threadIdx.x & 31 & ~(kWide - 1);       // the group's first lane in its warp
    const uint32_t mask = 0xFFu << lane0;
    auto from = [&](auto v, int k) { return __shfl_sync(mask, v, lane0 + k); };
    for (uint32_t i = blockIdx.x * kGroups + group; i < n_in; i += gridDim.x * kGroups) {
        const CollapseItem it = in[i];
        // 1. the children: the binary node's two children in 8 slots, split on along the choices, all lanes'
        // subtrees a step at a time (the chain of loads is as long as the deepest split, not as their number)
        if (it.node >= cap) { if (lane == 0) atomicMax(&ctrs[1], 1u); continue; }
        uint32_t c = it.bin, slots = 0, m = 1;
        bool split = false;                       // the lane's subtree may have to be split further
        if (!t.is_leaf(it.bin)) {                 // (else the root of a scene of at most kMaxLeafTris triangles)
            const uint32_t k8 = choice_node_split(t.costs[it.bin].choice);
            c = lane == 0 ? t.left[it.bin] : t.right[it.bin];
            slots = lane == 0 ? k8 : 8u - k8;
            m = 2;
            split = lane < 2;
        }
        while (__any_sync(mask, split)) {
            uint32_t k = 0, right = 0, right_slots = 0;
            if (split && !(c & kLeafBit)) {
                const uint32_t choice = t.costs[c].choice;
                uint32_t j = min(slots, 7u);
                while (j > 1u && (k = choice_split(choice, j)) == 0u) --j;
                if (k) {
                    right = t.right[c];
                    right_slots = j - k;
                    c = t.left[c];
                    slots = k;
                }
            }
            // the right halves go to the next free lanes (the slots add up to at most 8, so there are enough)
            const uint32_t splitting = (__ballot_sync(mask, k != 0u) >> lane0) & 0xFFu;
            const int mine = lane - (int)m;        // a free lane takes the half of the mine-th splitting lane
            const int n_split = __popc(splitting);
            uint32_t rest = splitting;
            for (int q = 0; q < mine; ++q) rest &= rest - 1u;
            const bool take = mine >= 0 && mine < n_split;
            const int src = take ? __ffs(rest) - 1 : lane;
            const uint32_t c_in = __shfl_sync(mask, right, lane0 + src), s_in = __shfl_sync(mask, right_slots, lane0 + src);
            split = k != 0u;
            if (take) { c = c_in; slots = s_in; split = true; }
            m += (uint32_t)n_split;
        }
        if (m > (uint32_t)kWide) { if (lane == 0) atomicMax(&ctrs[1], 1u); continue; }
        // 2. a lane's child: its box, and the node's
        const bool have = lane < (int)m;
        float4 lo = make_float4(3.0e38f, 3.0e38f, 3.0e38f, 0.0f), hi = make_float4(-3.0e38f, -3.0e38f, -3.0e38f, 0.0f);
        bool internal = false;
        uint32_t first = 0, count = 0;
        if (have) {
            if (c & kLeafBit) {
                first = c & ~kLeafBit;
                count = 1;
                const uint32_t tri = t.vals[first];
                lo = t.bmin[tri];
                hi = t.bmax[tri];
            } else {
                lo = t.imin[c];
                hi = t.imax[c];
                internal = !t.is_leaf(c);
                if (!internal) {
                    first = t.first[c];
                    count = t.last[c] - first + 1u;
                }
            }
        }
        float nlx = lo.x, nly = lo.y, nlz = lo.z, nhx = hi.x, nhy = hi.y, nhz = hi.z;
        for (int o = 1; o < kWide; o <<= 1) {
            nlx = fminf(nlx, __shfl_xor_sync(mask, nlx, o)); nly = fminf(nly, __shfl_xor_sync(mask, nly, o));
            nlz = fminf(nlz, __shfl_xor_sync(mask, nlz, o)); nhx = fmaxf(nhx, __shfl_xor_sync(mask, nhx, o));
            nhy = fmaxf(nhy, __shfl_xor_sync(mask, nhy, o)); nhz = fmaxf(nhz, __shfl_xor_sync(mask, nhz, o));
        }
        // 3. slots by octant: the child whose centre lies on the high side of axis a prefers slots with bit a
        // set; the best (child, slot) of those left is placed, m times
        const float dx = 0.5f * (lo.x + hi.x) - 0.5f * (nlx + nhx), dy = 0.5f * (lo.y + hi.y) - 0.5f * (nly + nhy),
                    dz = 0.5f * (lo.z + hi.z) - 0.5f * (nlz + nhz);
        uint32_t used = 0;
        int slot = -1;
        for (uint32_t round = 0; round < m; ++round) {
            float best = 3.0e38f;
            int bs = -1, bk = kWide;
            if (have && slot < 0)
                for (int sl = 0; sl < kWide; ++sl) {
                    if ((used >> sl) & 1u) continue;
                    const float v = ((sl & 1) ? -dx : dx) + ((sl & 2) ? -dy : dy) + ((sl & 4) ? -dz : dz);
                    if (v < best || bs < 0) { best = v < best ? v : best; bs = sl; bk = lane; }   // (a free slot whatever v)
                }
            for (int o = 1; o < kWide; o <<= 1) {
                const float v = __shfl_xor_sync(mask, best, o);
                const int k = __shfl_xor_sync(mask, bk, o), sl = __shfl_xor_sync(mask, bs, o);
                if (k < kWide && (bk == kWide || v < best || (v == best && k < bk))) { best = v; bk = k; bs = sl; }
            }
            if (lane == bk) slot = bs;
            used |= 1u << bs;
        }
        // the lanes without a child take the free slots (their planes are an inverted box, their meta byte 0)
        {
            uint32_t rest = ~used & 0xFFu;
            for (int k = (int)m; k < lane; ++k) rest &= rest - 1u;
            if (!have) slot = __ffs(rest) - 1;
        }
        // 4. places: internal children in slot order, the leaf children's triangles in slot order
        const uint32_t imask = __reduce_or_sync(mask, internal ? 1u << slot : 0u);
        const uint32_t n_int = (uint32_t)__popc(imask), n_lt = __reduce_add_sync(mask, count);
        uint32_t offset = 0;
        for (int k = 0; k < kWide; ++k) {
            const uint32_t ck = from(count, k);
            if (from(slot, k) < slot) offset += ck;
        }
        uint32_t child_base = 0, qpos = 0, tri_base = 0;
        if (lane == 0) {
            if (n_int) child_base = atomicAdd(&ctrs[0], n_int);
            if (n_int) qpos = atomicAdd(&ctrs[kLevelCtr + level + 1], n_int);
            if (n_lt) tri_base = atomicAdd(&ctrs[2], n_lt);
        }
        child_base = from(child_base, 0);
        qpos = from(qpos, 0);
        tri_base = from(tri_base, 0);
        const bool leaf_ok = !have || internal || (count > 0 && count <= kMaxLeafTris && (uint64_t)first + count <= t.n);
        const int ex = grid_exponent(nlx, nhx), ey = grid_exponent(nly, nhy), ez = grid_exponent(nlz, nhz);
        const uint32_t error = ((uint64_t)child_base + n_int > cap || (uint64_t)qpos + n_int > cap || (uint64_t)tri_base + n_lt > t.n ||
                                !__all_sync(mask, leaf_ok)) ? 1u : ex > 127 || ey > 127 || ez > 127 ? 2u : 0u;
        if (error) { if (lane == 0) atomicMax(&ctrs[1], error); continue; }
        // 5. the node's words, the next level's items, the triangle records
        uint32_t *w = nodes + (size_t)it.node * kNodeWords;
        if (lane == 0) {
            *reinterpret_cast<uint4 *>(w) = make_uint4(__float_as_uint(nlx), __float_as_uint(nly), __float_as_uint(nlz),
                                                       (uint32_t)(ex + 127) | ((uint32_t)(ey + 127) << 8) |
                                                           ((uint32_t)(ez + 127) << 16) | (imask << 24));
            w[kNodeChildBase] = child_base;
            w[kNodeTriBase] = tri_base;
        }
        w[node_plane_word(0, slot)] = have ? quantise(nlx, ldexp(1.0, -ex), lo.x, hi.x) : 0xFFFFu;
        w[node_plane_word(1, slot)] = have ? quantise(nly, ldexp(1.0, -ey), lo.y, hi.y) : 0xFFFFu;
        w[node_plane_word(2, slot)] = have ? quantise(nlz, ldexp(1.0, -ez), lo.z, hi.z) : 0xFFFFu;
        reinterpret_cast<uint8_t *>(w + kNodeMeta)[slot] = count ? (uint8_t)((((1u << count) - 1u) << 5) | offset) : (uint8_t)0;
        if (internal) {
            const uint32_t rank = (uint32_t)__popc(imask & ((1u << slot) - 1u));
            out[qpos + rank] = CollapseItem{c, child_base + rank};
        }
        for (uint32_t j = 0; j < count; ++j) {
            const uint32_t tri = t.vals[first + j];
            const float4 a = a4[tri];
            float4 *rec = tris + 3 * (size_t)(tri_base + offset + j);
            rec[0] = make_float4(a.x, a.y, a.z, __uint_as_float(tri));
            rec[1] = ab4[tri];
            rec[2] = ac4[tri];
        }
    }
}

}  // namespace

namespace mrt_host {

int leaf_max_setting() {
    static int v = [] {
        const char *e = getenv("MRT_BVH_LEAF_MAX");
        const int x = e ? atoi(e) : (int)kMaxLeafTris;   // the largest subtree the surface-area leaf choice may keep as one leaf
        return x < 1 ? 1 : (x > (int)kMaxLeafTris ? (int)kMaxLeafTris : x);
    }();
    return v;
}

int build_fast_bvh(MrtScene *s) {
    MrtContext *ctx = s->ctx;
    cudaStream_t q = ctx->stream;
    const uint32_t n = s->n_tri;
    // planes and spheres are walked in order in FAST mode; only triangles get the tree
    if (n == 0) {
        s->fnode_count = 0;
        s->dev.n_fnodes = 0;
        s->dev.fnodes = nullptr;
        s->dev.ftris = nullptr;
        return MRT_OK;
    }
    if (n >= kMaxFastTris) {
        set_error(ctx, "fast bvh: at most %u triangles", kMaxFastTris - 1u);
        return MRT_ERR_ARG;
    }
    int st = MRT_OK;
    st = dev_alloc(ctx, s->ftris, 48ull * n);
    if (st != MRT_OK) return st;
    DevBuf bmin, bmax, cb, keys[2], vals[2], hist, total, lft, rgt, fst, lst, pint, pleaf, ctr, imin, imax, costs;
    const uint32_t nblocks = (n + kSortTile - 1) / kSortTile;
    auto A = [&](DevBuf &b, size_t bytes) { if (st == MRT_OK) st = dev_alloc(ctx, b, bytes); };
    A(bmin, 16ull * n); A(bmax, 16ull * n); A(cb, 64);
    A(keys[0], 4ull * n); A(keys[1], 4ull * n); A(vals[0], 4ull * n); A(vals[1], 4ull * n);
    A(hist, 4ull * 256 * nblocks); A(total, 4ull * 256);
    A(lft, 4ull * n); A(rgt, 4ull * n); A(fst, 4ull * n); A(lst, 4ull * n);
    A(pint, 4ull * n); A(pleaf, 4ull * n); A(ctr, 4ull * n); A(imin, 16ull * n); A(imax, 16ull * n);
    A(costs, sizeof(SlotCosts) * (size_t)n);
    if (st == MRT_OK) {
        const uint32_t init[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
        st = cuda_status(ctx, cudaMemcpyAsync(cb.ptr, init, sizeof(init), cudaMemcpyHostToDevice, q), "bvh init");
    }
    int cur = 0;
    if (st == MRT_OK) {
        const uint32_t g = (n + 255) / 256;
        k_tri_boxes<<<g, 256, 0, q>>>(n, s->dev.tri_a, s->dev.tri_ab, s->dev.tri_ac, (float4 *)bmin.ptr,
                                      (float4 *)bmax.ptr, (uint32_t *)cb.ptr);
        k_morton<<<g, 256, 0, q>>>(n, (const float4 *)bmin.ptr, (const float4 *)bmax.ptr, (const uint32_t *)cb.ptr,
                                   (uint32_t *)keys[0].ptr, (uint32_t *)vals[0].ptr);
        for (int shift = 0; shift < kCodeBits; shift += 8) {
            k_rs_hist<<<nblocks, kSortThreads, 0, q>>>((const uint32_t *)keys[cur].ptr, n, shift, (uint32_t *)hist.ptr, nblocks);
            k_rs_scan_rows<<<256, 256, 0, q>>>((uint32_t *)hist.ptr, nblocks, (uint32_t *)total.ptr);
            k_rs_scatter<<<nblocks, kSortThreads, 0, q>>>((const uint32_t *)keys[cur].ptr, (const uint32_t *)vals[cur].ptr,
                                                          (uint32_t *)keys[1 - cur].ptr, (uint32_t *)vals[1 - cur].ptr, n,
                                                          shift, (const uint32_t *)hist.ptr, nblocks, (const uint32_t *)total.ptr);
            cur = 1 - cur;
        }
        if (n > 1) {
            const uint32_t *svals = (const uint32_t *)vals[cur].ptr;
            cudaMemsetAsync(ctr.ptr, 0, 4ull * n, q);
            k_karras<<<(n - 1 + 255) / 256, 256, 0, q>>>((int)n, (const uint32_t *)keys[cur].ptr, (uint32_t *)lft.ptr,
                                                          (uint32_t *)rgt.ptr, (uint32_t *)fst.ptr, (uint32_t *)lst.ptr,
                                                          (uint32_t *)pint.ptr, (uint32_t *)pleaf.ptr);
            k_fit<<<(n + 255) / 256, 256, 0, q>>>((int)n, leaf_max_setting(), svals, (const float4 *)bmin.ptr,
                                                  (const float4 *)bmax.ptr, (const uint32_t *)lft.ptr,
                                                  (const uint32_t *)rgt.ptr, (const uint32_t *)fst.ptr,
                                                  (const uint32_t *)lst.ptr, (const uint32_t *)pint.ptr,
                                                  (const uint32_t *)pleaf.ptr, (uint32_t *)ctr.ptr, (float4 *)imin.ptr,
                                                  (float4 *)imax.ptr, (SlotCosts *)costs.ptr);
        }
        st = cuda_status(ctx, cudaGetLastError(), "fast bvh kernels");
        if (st == MRT_OK) st = cuda_status(ctx, cudaStreamSynchronize(q), "fast bvh build");
    }
    if (st != MRT_OK) drain(ctx);
    DevBuf *tmp[] = {&cb, &keys[0], &keys[1], &vals[1 - cur], &hist, &total, &pint, &pleaf, &ctr};
    for (DevBuf *b : tmp) dev_free(*b);
    // collapse into 8-wide compressed nodes, level by level, from the root
    DevBuf wide, queue[2], wctr;
    const uint32_t cap = n;   // every wide node but the root of a single-triangle scene is a binary internal node
    A(wide, 4ull * kNodeWords * cap);
    A(queue[0], sizeof(CollapseItem) * cap);
    A(queue[1], sizeof(CollapseItem) * cap);
    uint32_t h[kLevelCtr + kMaxLevels + 1] = {0};
    A(wctr, sizeof(h));
    h[0] = 1;              // the root node
    h[kLevelCtr] = 1;      // the root item
    if (st == MRT_OK) {
        const CollapseItem root{n > 1 ? 0u : kLeafBit, 0u};
        st = cuda_status(ctx, cudaMemcpyAsync(queue[0].ptr, &root, sizeof(root), cudaMemcpyHostToDevice, q), "collapse");
        if (st == MRT_OK) st = cuda_status(ctx, cudaMemcpyAsync(wctr.ptr, h, sizeof(h), cudaMemcpyHostToDevice, q), "collapse");
    }
    const BinTree bt{(const uint32_t *)vals[cur].ptr, (const float4 *)bmin.ptr, (const float4 *)bmax.ptr,
                     (const uint32_t *)lft.ptr, (const uint32_t *)rgt.ptr, (const uint32_t *)fst.ptr,
                     (const uint32_t *)lst.ptr, (const float4 *)imin.ptr, (const float4 *)imax.ptr,
                     (const SlotCosts *)costs.ptr, n};
    // the first ten levels at once (a million triangles take eight to ten), then four more at a time
    for (int level = 0; st == MRT_OK && h[1] == 0 && h[kLevelCtr + level] > 0;) {
        for (const int stop = level + (level == 0 ? 10 : 4); level < stop; ++level) {
            if (level + 1 > kMaxLevels) { st = MRT_ERR_LIMIT; break; }
            const uint64_t most = level < 9 ? std::min<uint64_t>(1ull << (3 * level), cap) : cap;   // items of a level
            const uint32_t blocks = (uint32_t)std::min<uint64_t>((most + kGroups - 1) / kGroups, (uint64_t)ctx->sm_count * 16);
            k_collapse<<<blocks, kCollapseThreads, 0, q>>>(bt, (const CollapseItem *)queue[level & 1].ptr, level,
                                              (CollapseItem *)queue[1 - (level & 1)].ptr, cap, (uint32_t *)wide.ptr,
                                              s->dev.tri_a, s->dev.tri_ab, s->dev.tri_ac, (float4 *)s->ftris.ptr,
                                              (uint32_t *)wctr.ptr);
        }
        if (st == MRT_OK) st = cuda_status(ctx, cudaGetLastError(), "collapse");
        if (st == MRT_OK) st = cuda_status(ctx, cudaMemcpyAsync(h, wctr.ptr, sizeof(h), cudaMemcpyDeviceToHost, q), "collapse");
        if (st == MRT_OK) st = cuda_status(ctx, cudaStreamSynchronize(q), "collapse");
    }
    if (st == MRT_OK && (h[1] != 0 || h[2] != n)) {
        set_error(ctx, h[1] == 2 ? "fast bvh: scene extent beyond the 2^127 grid step"
                                 : "fast bvh: inconsistent binary tree while collapsing");
        st = MRT_ERR_LIMIT;
    }
    const uint64_t n_wide = h[0];
    if (st == MRT_OK) {   // exact-size copy; the scratch goes
        st = dev_alloc(ctx, s->fnodes, 4ull * kNodeWords * n_wide);
        if (st == MRT_OK)
            st = cuda_status(ctx, cudaMemcpyAsync(s->fnodes.ptr, wide.ptr, 4ull * kNodeWords * n_wide,
                                                  cudaMemcpyDeviceToDevice, q), "collapse copy");
        if (st == MRT_OK) st = cuda_status(ctx, cudaStreamSynchronize(q), "collapse copy");
    }
    if (st != MRT_OK) drain(ctx);
    DevBuf *tmp2[] = {&wide, &queue[0], &queue[1], &wctr, &bmin, &bmax, &vals[cur], &lft, &rgt, &fst, &lst, &imin, &imax, &costs};
    for (DevBuf *b : tmp2) dev_free(*b);
    if (st != MRT_OK) return st;
    s->fnode_count = n_wide;
    s->dev.n_fnodes = (uint32_t)n_wide;
    s->dev.fnodes = (const float4 *)s->fnodes.ptr;
    s->dev.ftris = (const float4 *)s->ftris.ptr;
    return MRT_OK;
}

int build_reference_bvh(MrtScene *s) {
    MrtContext *ctx = s->ctx;
    const int got = host_triangles(s);
    if (got != MRT_OK) return got;
    for (int k = 0; k < 3; ++k) {
        std::vector<HBox> boxes;
        if (k == kTriangle) {
            boxes.resize(s->n_tri);
            for (uint32_t i = 0; i < s->n_tri; ++i) {   // Triangle::getAABB, Triangle.cpp:145-152
                const float *p = &s->h_tri[9ull * i];
                const V3 A{p[0], p[1], p[2]}, ab{p[3], p[4], p[5]}, ac{p[6], p[7], p[8]};
                const V3 B = A + ab, C = A + ac;
                boxes[i] = HBox{vmin(A, vmin(B, C)), vmax(A, vmax(B, C))};
            }
        } else if (k == kSphere) {
            boxes.resize(s->n_sph);
            for (uint32_t i = 0; i < s->n_sph; ++i) {   // Sphere::getAABB, Sphere.cpp:94-100
                const float *c = &s->h_sph[4ull * i];
                const float r = sqrtf(c[3]);
                const V3 ctr{c[0], c[1], c[2]};
                boxes[i] = HBox{subs(ctr, r), adds(ctr, r)};
            }
        } else {
            boxes.resize(s->n_pln);
            for (uint32_t i = 0; i < s->n_pln; ++i) {   // Plane::getAABB / getRightVector, Plane.cpp:80-105
                const float *p = &s->h_pln[6ull * i];
                const V3 n{p[3], p[4], p[5]}, pt{p[0], p[1], p[2]};
                V3 right{0, 0, 0};
                if (n.x >= 1) right = V3{0, 1, 1};
                else if (n.y >= 1) right = V3{1, 0, 1};
                else if (n.z >= 1) right = V3{1, 1, 0};
                else if (n.x <= -1) right = V3{0, 1, 1};
                else if (n.y <= -1) right = V3{1, 0, 1};
                else if (n.z <= -1) right = V3{1, 1, 0};
                right = normalize(right);
                boxes[i] = HBox{pt + right * -100.0f, pt + right * 100.0f};
            }
        }
        const std::vector<RefNode> nodes = ref_build(boxes);
        int st = dev_alloc(ctx, s->rnodes[k], sizeof(RefNode) * nodes.size());
        if (st == MRT_OK)
            st = cuda_status(ctx, cudaMemcpyAsync(s->rnodes[k].ptr, nodes.data(), sizeof(RefNode) * nodes.size(),
                                                  cudaMemcpyHostToDevice, ctx->stream), "upload bvh");
        if (st == MRT_OK) st = cuda_status(ctx, cudaStreamSynchronize(ctx->stream), "upload bvh");
        if (st != MRT_OK) return st;
        s->rnode_count[k] = nodes.size();
        s->dev.rnodes[k] = (const RefNode *)s->rnodes[k].ptr;
        s->dev.rnode_count[k] = (uint32_t)nodes.size();
    }
    return MRT_OK;
}

}  // namespace mrt_host
