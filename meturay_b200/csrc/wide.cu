// 8-wide BVH with quantised child boxes, collapsed on the GPU from the LBVH,
// and its closest-hit traversal.
//
// Why: the binary traversal is bound by the L1/LSU data path (64 bytes per
// two child boxes).  A wide node carries eight child boxes quantised to 8
// bits per plane relative to the node's own box: 80 bytes for up to eight
// children.  Per box test that is 10 bytes instead of 32, and one node fetch
// replaces about three binary levels.
//
// Collapse (top-down, one launch per level of the wide tree): a wide node is
// formed from a binary node by choosing which binary descendants become its
// (at most eight) children.  Default: the surface-area dynamic program of
// Ylitie, Karras and Laine ("Efficient Incoherent Ray Traversal on GPUs
// Through Compressed Wide BVHs", HPG 2017), with one-triangle leaves: a
// bottom-up pass gives every binary node g the least sum of wide-node
// surface areas that represents its subtree as at most i children,
// cost(g, i) for i = 1..8, and the collapse follows its choices.  Without
// it, the internal child with the largest surface area is opened until the
// node has eight children or only leaves.
// Internal children get consecutive wide-node slots and leaf children
// consecutive triangle slots; slots are handed out by atomic counters per
// level, so the first 1 + 8 + 64 slots are the top three levels.  The
// binary LBVH (reference numbering) is unchanged: this is a traversal layout
// derived from it.
//
// Node (80 B = five 16-byte loads):
//   n0 = (box.lo.xyz, exps): exps = ex | ey << 8 | ez << 16 | imask << 24
//   n1 = (childBase, triBase, leafMask, 0)
//   n2 = (qlo.x[0..7], qlo.y[0..7]), n3 = (qlo.z[0..7], qhi.x[0..7]),
//   n4 = (qhi.y[0..7], qhi.z[0..7])
// Slot k holds an internal child (imask bit k: node childBase + the number
// of internal children in lower slots), a leaf (leafMask bit k: triangle
// triBase + the number of leaves in lower slots) or nothing.
// A child plane decodes as lo + q * 2^(e-127); quantisation rounds outward,
// so decoded boxes contain the exact child boxes.
#include <type_traits>

#include "../../include/mrb200.h"
#include "common.cuh"
#include "wide.cuh"
#include "pool.cuh"

namespace mrb {

namespace {

struct WorkItem {
    uint32_t bnode;  // binary node (global index, >= n inner)
    uint32_t slot;   // wide node slot
};

__device__ __forceinline__ void child_box(uint32_t g, uint32_t n, const float* __restrict__ inner,
                                          const float* __restrict__ triAabb,
                                          const uint32_t* __restrict__ sortedIdx, float lo[3],
                                          float hi[3]) {
    const float* b = (g < n) ? triAabb + 6 * size_t(sortedIdx[g]) : inner + 6 * size_t(g - n);
    for (int c = 0; c < 3; c++) {
        lo[c] = b[c];
        hi[c] = b[3 + c];
    }
}

__device__ __forceinline__ float half_area(const float lo[3], const float hi[3]) {
    float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
    return dx * dy + dy * dz + dz * dx;
}

// Exponent byte e (scale 2^(e-127)) so that extent / scale <= 255.
__device__ __forceinline__ uint32_t quant_exponent(float extent) {
    if (!(extent > 0.0f)) return 1u;  // degenerate axis: planes decode to lo exactly
    float x = extent / 255.0f;
    uint32_t bits = __float_as_uint(x);
    uint32_t e = (bits >> 23) & 0xFFu;
    if (bits & 0x7FFFFFu) e += 1u;  // round up to a power of two
    // make sure the rounded division cannot exceed 255
    while (e < 254u && extent / __uint_as_float(e << 23) > 255.0f) e++;
    return e < 1u ? 1u : e;
}

// ---------------------------------------------------------------------------
// Surface-area collapse plan
//   cost(leaf, i) = 0 (every triangle is a leaf child exactly once)
//   D(g, i)       = min over k in 1..i-1 of cost(left, k) + cost(right, i - k)
//   E(g, 2) = D(g, 2), E(g, i) = min(E(g, i - 1), D(g, i))
//   cost(g, 1)    = area(g) + E(g, 8)          (g becomes a wide node)
//   cost(g, i)    = min(cost(g, 1), E(g, i))   (i >= 2)
// Plan per inner node (8 bytes): byte 0 bit i - 1 set where cost(g, i) takes
// cost(g, 1) (g stays one child), byte i - 1 (i = 2..8) the k of D(g, i), 0
// where E(g, i) = E(g, i - 1).  D(g, 2) always has k = 1.
// ---------------------------------------------------------------------------
__global__ void k_plan_parents(const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                               uint32_t n, uint32_t* parent, uint32_t* flags) {
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j + 1 < n;
         j += gridDim.x * blockDim.x) {
        parent[left[j]] = n + j;
        parent[right[j]] = n + j;
        flags[j] = 0u;
    }
}

// One thread per leaf walks up; the second arrival at a node evaluates it
// (the pattern of the LBVH's bottom-up box pass).  The walk ends at the root.
__global__ void k_plan_up(const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                          const float* __restrict__ inner, const uint32_t* __restrict__ parent,
                          const uint32_t* __restrict__ root, uint32_t n, uint32_t* flags,
                          float* cost, uint2* plan) {
    const uint32_t top = *root;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t g = parent[i];
        while (true) {
            __threadfence();
            if (atomicAdd(flags + (g - n), 1u) == 0u) break;  // the sibling is not done yet
            __threadfence();
            const uint32_t j = g - n;
            const uint32_t l = left[j], r = right[j];
            float cl[9], cr[9];
            auto load = [&](uint32_t child, float* c) {
                float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
                if (child >= n) {
                    const float4* p = reinterpret_cast<const float4*>(cost + 8 * size_t(child - n));
                    a = __ldcg(p);
                    b = __ldcg(p + 1);
                }
                c[1] = a.x; c[2] = a.y; c[3] = a.z; c[4] = a.w;
                c[5] = b.x; c[6] = b.y; c[7] = b.z; c[8] = b.w;
            };
            load(l, cl);
            load(r, cr);
            float E[9];
            uint32_t ks[9];
#pragma unroll
            for (int c = 2; c <= 8; c++) {
                float best = 0.0f;
                uint32_t bk = 0;
#pragma unroll
                for (int k = 1; k < c; k++) {
                    const float v = cl[k] + cr[c - k];
                    if (bk == 0 || v < best) {
                        best = v;
                        bk = uint32_t(k);
                    }
                }
                if (c > 2 && E[c - 1] <= best) {
                    best = E[c - 1];
                    bk = 0;
                }
                E[c] = best;
                ks[c] = bk;
            }
            const float* b = inner + 6 * size_t(j);
            const float dx = b[3] - b[0], dy = b[4] - b[1], dz = b[5] - b[2];
            const float c1 = (dx * dy + dy * dz + dz * dx) + E[8];
            uint32_t single = 0;
            for (int c = 2; c <= 8; c++) {
                if (c1 <= E[c]) single |= 1u << (c - 1);
                E[c] = fminf(c1, E[c]);
            }
            float4* cj = reinterpret_cast<float4*>(cost + 8 * size_t(j));
            cj[0] = make_float4(c1, E[2], E[3], E[4]);
            cj[1] = make_float4(E[5], E[6], E[7], E[8]);
            plan[j] = make_uint2(single | (ks[2] << 8) | (ks[3] << 16) | (ks[4] << 24),
                                 ks[5] | (ks[6] << 8) | (ks[7] << 16) | (ks[8] << 24));
            if (g == top) break;
            g = parent[g];
        }
    }
}

__device__ __forceinline__ uint32_t plan_byte(uint2 p, int b) {
    return ((b < 4 ? p.x : p.y) >> (8 * (b & 3))) & 0xFFu;
}

// One level of the collapse: a team of eight lanes makes each wide node of the
// level's queue, one lane per child slot (four nodes per warp; every lane takes
// part in the warp's votes and shuffles).  One thread per node spent 68 us on a
// level however few its nodes (1M triangles, 16 levels): the dependent reads
// of the plan, the 8 x 8 greedy matching and the eight children's boxes, one
// after the other.
constexpr int kCollapseBlock = 128;
__global__ void __launch_bounds__(kCollapseBlock) k_collapse(
    const WorkItem* __restrict__ qin, const uint32_t* __restrict__ qinCount, WorkItem* qout,
    uint32_t* qoutCount, uint32_t* nodeCounter, uint32_t* triCounter, uint32_t n,
    const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
    const float* __restrict__ inner, const float* __restrict__ triAabb,
    const uint32_t* __restrict__ sortedIdx, const float* __restrict__ pos,
    const uint32_t* __restrict__ idx, const uint32_t* __restrict__ key,
    const uint8_t* __restrict__ cull, const uint2* __restrict__ plan, WideNode* nodes, float4* tv0,
    float4* te0, float4* te1) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    __shared__ uint32_t shNode[kCollapseBlock], shSlots[kCollapseBlock];
    const uint32_t lane = threadIdx.x & 7u, shift = threadIdx.x & 24u;
    const uint32_t team0 = threadIdx.x & ~7u;  // the team's first thread
    const uint32_t count = *qinCount;
    const uint32_t warps = (gridDim.x * kCollapseBlock) >> 5;
    for (uint32_t w0 = 4u * ((blockIdx.x * kCollapseBlock + threadIdx.x) >> 5); w0 < count;
         w0 += 4u * warps) {
        const uint32_t w = w0 + (shift >> 3);
        const bool valid = w < count;
        const WorkItem it = valid ? qin[w] : WorkItem{0u, 0u};
        // ---- children: one per lane, left to right
        uint32_t x = kInvalid;  // this lane's child
        if (plan) {
            // lane p with i slots holds p .. p + i - 1; a split keeps the left
            // child's and hands the right child's to lane p + k
            uint32_t slots = 0;
            bool open = false, own = false;
            if (valid && lane == 0) {
                x = it.bnode;
                slots = 8;
                open = own = true;
            }
            while (__any_sync(kAll, open)) {
                shSlots[threadIdx.x] = 0;
                __syncwarp();
                if (open) {
                    if (!own && (x < n || slots == 1)) {
                        open = false;
                    } else {
                        const uint2 pl = plan[x - n];
                        if (!own && ((pl.x >> (slots - 1)) & 1u)) {
                            open = false;
                        } else {
                            uint32_t k;
                            while ((k = plan_byte(pl, int(slots) - 1)) == 0u) slots--;
                            // left takes k slots, right the rest (each >= 1)
                            shNode[threadIdx.x + k] = right[x - n];
                            shSlots[threadIdx.x + k] = slots - k;
                            x = left[x - n];
                            slots = k;
                            own = false;
                        }
                    }
                }
                __syncwarp();
                if (shSlots[threadIdx.x]) {
                    x = shNode[threadIdx.x];
                    slots = shSlots[threadIdx.x];
                    open = true;
                }
                __syncwarp();
            }
        } else {
            // open the largest internal child until eight children
            float area = -1.0f;  // internal children only
            auto set = [&](uint32_t g) {
                x = g;
                area = -1.0f;
                if (g >= n) {
                    float lo[3], hi[3];
                    child_box(g, n, inner, triAabb, sortedIdx, lo, hi);
                    area = half_area(lo, hi);
                    if (!(area == area)) area = 0.0f;  // NaN boxes: any order will do
                }
            };
            if (valid && lane < 2) set(lane == 0 ? left[it.bnode - n] : right[it.bnode - n]);
            uint32_t nc = 2;
            while (true) {
                float best = (x != kInvalid && x >= n) ? area : -1.0f;
                uint32_t at = lane;
                bool has = x != kInvalid && x >= n;
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) {
                    const float ob = __shfl_xor_sync(kAll, best, o);
                    const uint32_t oa = __shfl_xor_sync(kAll, at, o);
                    const bool oh = __shfl_xor_sync(kAll, has, o);
                    if (oh && (!has || ob > best || (ob == best && oa < at))) {
                        best = ob;
                        at = oa;
                        has = true;
                    }
                }
                const bool go = valid && has && nc < 8u;
                if (!__any_sync(kAll, go)) break;
                const uint32_t b = __shfl_sync(kAll, x, int(at), 8);
                if (go) {
                    if (lane == at) set(left[b - n]);
                    if (lane == nc) set(right[b - n]);
                    nc++;
                }
            }
        }
        // ---- slot of each child: the octant of its centroid around the
        // node's centre, matched greedily by the largest projection on the
        // octant's diagonal, so that slot ^ (ray octant) orders the children
        // roughly front to back for any ray direction
        float blo[3] = {0.0f, 0.0f, 0.0f}, bhi[3] = {0.0f, 0.0f, 0.0f};  // the node's box
        if (valid) child_box(it.bnode, n, inner, triAabb, sortedIdx, blo, bhi);
        {
            float dc[3] = {0.0f, 0.0f, 0.0f};
            if (x != kInvalid) {
                float lo[3], hi[3];
                child_box(x, n, inner, triAabb, sortedIdx, lo, hi);
                for (int c = 0; c < 3; c++) dc[c] = (lo[c] + hi[c]) - (blo[c] + bhi[c]);
            }
            shNode[threadIdx.x] = kInvalid;
            __syncwarp();
            uint32_t usedSlot = 0;
            bool wait = x != kInvalid;  // not placed yet
            while (__any_sync(kAll, wait)) {
                float bc = 0.0f;
                uint32_t bs = 8u, bk = lane;
#pragma unroll
                for (uint32_t sl = 0; sl < 8; sl++) {
                    float cost = -(((sl & 1) ? dc[0] : -dc[0]) + ((sl & 2) ? dc[1] : -dc[1]) +
                                   ((sl & 4) ? dc[2] : -dc[2]));
                    if (!(cost == cost)) cost = kFltMax;  // NaN or infinite boxes
                    if (wait && !((usedSlot >> sl) & 1u) && (bs == 8u || cost < bc)) {
                        bc = cost;
                        bs = sl;
                    }
                }
                // least cost, then lowest child, of the team
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) {
                    const float oc = __shfl_xor_sync(kAll, bc, o);
                    const uint32_t os = __shfl_xor_sync(kAll, bs, o);
                    const uint32_t ok = __shfl_xor_sync(kAll, bk, o);
                    if (os != 8u && (bs == 8u || oc < bc || (oc == bc && ok < bk))) {
                        bc = oc;
                        bs = os;
                        bk = ok;
                    }
                }
                if (bs != 8u) {
                    usedSlot |= 1u << bs;
                    if (lane == bk) {
                        shNode[team0 + bs] = x;
                        wait = false;
                    }
                }
            }
            __syncwarp();
            x = shNode[threadIdx.x];  // from here the child in this lane's slot
            __syncwarp();
        }
        const bool isInner = x != kInvalid && x >= n, isLeaf = x != kInvalid && x < n;
        const uint32_t imask = (__ballot_sync(kAll, isInner) >> shift) & 0xFFu;
        const uint32_t leafMask = (__ballot_sync(kAll, isLeaf) >> shift) & 0xFFu;
        uint32_t childBase = 0, triBase = 0, qbase = 0;
        if (valid && lane == 0) {
            if (imask) {
                childBase = atomicAdd(nodeCounter, uint32_t(__popc(imask)));
                qbase = atomicAdd(qoutCount, uint32_t(__popc(imask)));
            }
            if (leafMask) triBase = atomicAdd(triCounter, uint32_t(__popc(leafMask)));
        }
        childBase = __shfl_sync(kAll, childBase, 0, 8);
        triBase = __shfl_sync(kAll, triBase, 0, 8);
        qbase = __shfl_sync(kAll, qbase, 0, 8);
        if (!valid) continue;

        uint8_t* bytes = reinterpret_cast<uint8_t*>(nodes + it.slot);
        uint32_t e[3];
        for (int c = 0; c < 3; c++) e[c] = quant_exponent(bhi[c] - blo[c]);
        if (lane == 0)
            *reinterpret_cast<float4*>(bytes) = make_float4(
                blo[0], blo[1], blo[2],
                __uint_as_float(e[0] | (e[1] << 8) | (e[2] << 16) | (imask << 24)));
        if (lane == 1)
            *reinterpret_cast<uint4*>(bytes + 16) = make_uint4(childBase, triBase, leafMask, 0u);
        float lo[3], hi[3];
        if (x != kInvalid) child_box(x, n, inner, triAabb, sortedIdx, lo, hi);
        for (int c = 0; c < 3; c++) {
            uint32_t q0 = 255u, q1 = 0u;  // an empty slot never hits
            if (x != kInvalid) {
                // outward rounding in double: exact for float inputs and
                // power-of-two scales (the product with 2^(127 - e) is the
                // quotient)
                const double inv = __longlong_as_double(int64_t(1150 - int(e[c])) << 52);
                double ql = floor((double(lo[c]) - double(blo[c])) * inv);
                double qh = ceil((double(hi[c]) - double(blo[c])) * inv);
                ql = ql < 0.0 ? 0.0 : (ql > 255.0 ? 255.0 : ql);
                qh = qh < 0.0 ? 0.0 : (qh > 255.0 ? 255.0 : qh);
                q0 = static_cast<uint32_t>(ql);
                q1 = static_cast<uint32_t>(qh);
            }
            bytes[32 + 8 * c + lane] = static_cast<uint8_t>(q0);
            bytes[56 + 8 * c + lane] = static_cast<uint8_t>(q1);
        }
        const uint32_t below = (1u << lane) - 1u;
        if (isInner) {
            const uint32_t r = uint32_t(__popc(imask & below));
            qout[qbase + r] = WorkItem{x, childBase + r};
        } else if (isLeaf) {
            // leaf: the triangle, reordered into this node's leaf block
            const uint32_t t = sortedIdx[x];
            const uint32_t s = triBase + uint32_t(__popc(leafMask & below));
            const uint32_t i0 = idx[3 * size_t(t)], i1 = idx[3 * size_t(t) + 1],
                           i2 = idx[3 * size_t(t) + 2];
            const V3 p0 = ld3(pos + 3 * size_t(i0)), p1 = ld3(pos + 3 * size_t(i1)),
                     p2 = ld3(pos + 3 * size_t(i2));
            const V3 e0 = p1 - p0, e1 = p2 - p0;
            tv0[s] = make_float4(p0.x, p0.y, p0.z, __uint_as_float(t));
            te0[s] = make_float4(e0.x, e0.y, e0.z, __uint_as_float(key[t]));
            te1[s] = make_float4(e1.x, e1.y, e1.z, __uint_as_float(cull ? uint32_t(cull[t]) : 0u));
        }
    }
}

// Counters of a collapse, zeroed before: wide nodes, triangles, then the queue
// length of each level.
constexpr int kMaxLevels = 4 * 96;
constexpr int kCounters = 2 + kMaxLevels + 1;
__global__ void k_collapse_init(WorkItem* q0, uint32_t* counters, const uint32_t* root) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        q0[0] = WorkItem{*root, 0u};
        counters[0] = 1;  // slot 0 = root
        counters[2] = 1;  // level 0
    }
}

// ---------------------------------------------------------------------------
// Traversal
// ---------------------------------------------------------------------------
// The top two levels (1 + 8 nodes) are read from shared memory.  Three
// levels (73 nodes, 5.8 KB per block) measured 2 % slower on both
// clusters-1M and Cornell: the smaller carve-out leaves more of the SM's
// on-chip memory to L1, which serves the lower levels.  None at all was
// faster on clusters-1M but 13 % slower on Cornell.
constexpr int kCachedNodes = 9;
constexpr int kWideStack = 128;  // sorted order: one entry per pushed child
constexpr int kWideGroups = 48;  // octant order: at most one group per level

__device__ __forceinline__ float safe_dir(float d) {
    return (fabsf(d) > 1e-20f) ? d : copysignf(1e-20f, d);
}

__device__ __forceinline__ uint32_t byte_of(uint32_t w, int k) { return (w >> (8 * k)) & 0xFFu; }

__device__ __forceinline__ void cas(uint32_t& a, uint32_t& b) {
    const uint32_t lo = min(a, b), hi = max(a, b);
    a = lo;
    b = hi;
}
// Optimal 19-comparator network for eight keys (ascending).
__device__ __forceinline__ void sort8(uint32_t k[8]) {
    cas(k[0], k[2]); cas(k[1], k[3]); cas(k[4], k[6]); cas(k[5], k[7]);
    cas(k[0], k[4]); cas(k[1], k[5]); cas(k[2], k[6]); cas(k[3], k[7]);
    cas(k[0], k[1]); cas(k[2], k[3]); cas(k[4], k[5]); cas(k[6], k[7]);
    cas(k[2], k[4]); cas(k[3], k[5]);
    cas(k[1], k[4]); cas(k[3], k[6]);
    cas(k[1], k[2]); cas(k[3], k[4]); cas(k[5], k[6]);
}

__device__ __forceinline__ void tri_test(const WideAccelDev& acc, uint32_t s, V3 o, V3 d,
                                         float tmin, float& closest, int& hitTri, float& hb0,
                                         float& hb1) {
    float4 a = __ldg(acc.tv0 + s), b = __ldg(acc.te0 + s), c = __ldg(acc.te1 + s);
    V3 v0 = {a.x, a.y, a.z}, e0 = {b.x, b.y, b.z}, e1 = {c.x, c.y, c.z};
    bool cull = __float_as_uint(c.w) != 0u;
    V3 p = cross(d, e1);
    float det = dot(e0, p);
    if ((cull && (det < 1.0e-7f)) || (fabsf(det) < 1.0e-7f)) return;
    float invDet = 1.0f / det;
    V3 tv = o - v0;
    float u = dot(tv, p) * invDet;
    if (u < 0.0f || u > 1.0f) return;
    V3 q = cross(tv, e0);
    float v = dot(d, q) * invDet;
    if ((v < 0.0f) || (v + u) > 1.0f) return;
    float t = dot(e1, q) * invDet;
    if (t <= 1.0e-7f) return;
    if (t >= tmin && t < closest) {
        closest = t;
        hitTri = static_cast<int>(s);
        hb0 = 1.0f - u - v;
        hb1 = u;
    }
}

template <int k>
using IntC = std::integral_constant<int, k>;

// Per-ray state of a traversal: the ray, its closest hit so far and the
// node to visit next (-1: done).  The stack lives beside it.
struct WideRay {
    V3 o, d, inv;
    float tmin, closest, hb0, hb1;
    int hitTri, node, sp;
    uint32_t oct;  // sign bits of the direction: x | y << 1 | z << 2
};

__device__ __forceinline__ void wide_ray_begin(WideRay& r, float4 ro, float4 rd) {
    r.o = V3{ro.x, ro.y, ro.z};
    r.d = V3{rd.x, rd.y, rd.z};
    r.tmin = ro.w;
    r.closest = rd.w;
    r.hb0 = r.hb1 = 0.0f;
    r.hitTri = -1;
    r.inv = V3{1.0f / safe_dir(rd.x), 1.0f / safe_dir(rd.y), 1.0f / safe_dir(rd.z)};
    r.oct = (r.inv.x < 0.0f ? 1u : 0u) | (r.inv.y < 0.0f ? 2u : 0u) | (r.inv.z < 0.0f ? 4u : 0u);
    r.node = 0;
    r.sp = 0;
}

// A node's words and its child slabs in the ray's frame: child plane q
// lies at t = q * a + b per axis; the near and far plane words are chosen
// per axis from the direction's sign.  The top `cached` nodes are read from
// shared memory (sNodes), the rest through the read-only cache.
struct NodeSlabs {
    uint32_t childBase, triBase, leafMask, imask;
    float ax, ay, az, bx, by, bz;
    uint32_t qn[6], qf[6];  // x0 x1 y0 y1 z0 z1: bytes of slots 0-3 and 4-7
};

// Two floats in one 64-bit register pair, and their fused multiply-add in one
// instruction (each half rounds as __fmaf_rn).
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// The slabs of the octant kernels, two slots per packed instruction.  The bytes
// of the near planes become floats by a permute under the exponent of 2^23 and
// one addition that takes 2^23 off again, those of the far planes on the XU pipe,
// and one multiply-add gives two planes, bit for bit the values of child_span.
// The node loop is bound by instructions issued.  Clusters 1M, camera rays: 1.75
// ms with one slot per instruction, 1.60 ms so, 1.63 ms with the far planes by
// permutes too; a million incoherent rays (refill) 1.00, 0.94 and 0.97 ms.  The
// sorted kernels keep the plain form, which is no slower there.
struct PackedSlabs {
    uint64_t ax, ay, az, bx, by, bz;  // each twice
};
__device__ __forceinline__ PackedSlabs packed_slabs(const NodeSlabs& s) {
    return {pack2(s.ax, s.ax), pack2(s.ay, s.ay), pack2(s.az, s.az),
            pack2(s.bx, s.bx), pack2(s.by, s.by), pack2(s.bz, s.bz)};
}
template <int kk, bool kXu>
__device__ __forceinline__ uint64_t plane_pair(uint32_t w) {
    if constexpr (kXu) return pack2(float(byte_of(w, kk)), float(byte_of(w, kk + 1)));
    return add2(pack2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7550u | kk)),
                      __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7550u | (kk + 1)))),
                pack2(-8388608.0f, -8388608.0f));
}
// Entry and exit distances of child slots k and k + 1 (compile-time, k even).
template <int k>
__device__ __forceinline__ void child_spans(const NodeSlabs& s, const PackedSlabs& p, float tmin,
                                            float closest, float tn[2], float tf[2]) {
    constexpr int h = k < 4 ? 0 : 1, kk = k & 3;
    float nx[2], ny[2], nz[2], fx[2], fy[2], fz[2];
    unpack2(fma2(plane_pair<kk, false>(s.qn[0 + h]), p.ax, p.bx), nx[0], nx[1]);
    unpack2(fma2(plane_pair<kk, false>(s.qn[2 + h]), p.ay, p.by), ny[0], ny[1]);
    unpack2(fma2(plane_pair<kk, false>(s.qn[4 + h]), p.az, p.bz), nz[0], nz[1]);
    unpack2(fma2(plane_pair<kk, true>(s.qf[0 + h]), p.ax, p.bx), fx[0], fx[1]);
    unpack2(fma2(plane_pair<kk, true>(s.qf[2 + h]), p.ay, p.by), fy[0], fy[1]);
    unpack2(fma2(plane_pair<kk, true>(s.qf[4 + h]), p.az, p.bz), fz[0], fz[1]);
#pragma unroll
    for (int j = 0; j < 2; j++) {
        tn[j] = fmaxf(fmaxf(nx[j], ny[j]), fmaxf(nz[j], tmin));
        tf[j] = fminf(fminf(fx[j], fy[j]), fminf(fz[j], closest));
    }
}

__device__ __forceinline__ void node_slabs(const WideAccelDev& acc, const WideNode* sNodes,
                                           int cached, int node, const WideRay& r,
                                           NodeSlabs& s) {
    uint4 w0, w1, w2, w3, w4;
    if (node < cached) {
        const uint4* sm = reinterpret_cast<const uint4*>(sNodes + node);
        w0 = sm[0]; w1 = sm[1]; w2 = sm[2]; w3 = sm[3]; w4 = sm[4];
    } else {
        const uint4* g = reinterpret_cast<const uint4*>(acc.nodes + node);
        w0 = __ldg(g); w1 = __ldg(g + 1); w2 = __ldg(g + 2); w3 = __ldg(g + 3);
        w4 = __ldg(g + 4);
    }
    const float sx = __uint_as_float((w0.w & 0xFFu) << 23);
    const float sy = __uint_as_float(((w0.w >> 8) & 0xFFu) << 23);
    const float sz = __uint_as_float(((w0.w >> 16) & 0xFFu) << 23);
    s.imask = w0.w >> 24;
    // t = (lo + q*s - o) * inv = q * (s*inv) + (lo - o) * inv
    s.ax = sx * r.inv.x;
    s.ay = sy * r.inv.y;
    s.az = sz * r.inv.z;
    s.bx = (__uint_as_float(w0.x) - r.o.x) * r.inv.x;
    s.by = (__uint_as_float(w0.y) - r.o.y) * r.inv.y;
    s.bz = (__uint_as_float(w0.z) - r.o.z) * r.inv.z;
    s.childBase = w1.x;
    s.triBase = w1.y;
    s.leafMask = w1.z;
    const bool px = r.inv.x >= 0.0f, py = r.inv.y >= 0.0f, pz = r.inv.z >= 0.0f;
    s.qn[0] = px ? w2.x : w3.z; s.qn[1] = px ? w2.y : w3.w;
    s.qf[0] = px ? w3.z : w2.x; s.qf[1] = px ? w3.w : w2.y;
    s.qn[2] = py ? w2.z : w4.x; s.qn[3] = py ? w2.w : w4.y;
    s.qf[2] = py ? w4.x : w2.z; s.qf[3] = py ? w4.y : w2.w;
    s.qn[4] = pz ? w3.x : w4.z; s.qn[5] = pz ? w3.y : w4.w;
    s.qf[4] = pz ? w4.z : w3.x; s.qf[5] = pz ? w4.w : w3.y;
}

// Entry and exit distance of child slot k (compile-time k).
template <int k>
__device__ __forceinline__ void child_span(const NodeSlabs& s, float tmin, float closest,
                                           float& tn, float& tf) {
    constexpr int h = k < 4 ? 0 : 1, kk = k & 3;
    const float tnx = __fmaf_rn(float(byte_of(s.qn[0 + h], kk)), s.ax, s.bx);
    const float tfx = __fmaf_rn(float(byte_of(s.qf[0 + h], kk)), s.ax, s.bx);
    const float tny = __fmaf_rn(float(byte_of(s.qn[2 + h], kk)), s.ay, s.by);
    const float tfy = __fmaf_rn(float(byte_of(s.qf[2 + h], kk)), s.ay, s.by);
    const float tnz = __fmaf_rn(float(byte_of(s.qn[4 + h], kk)), s.az, s.bz);
    const float tfz = __fmaf_rn(float(byte_of(s.qf[4 + h], kk)), s.az, s.bz);
    tn = fmaxf(fmaxf(tnx, tny), fmaxf(tnz, tmin));
    tf = fminf(fminf(tfx, tfy), fminf(tfz, closest));
}


// One node of the traversal in exact front-to-back order: the hit internal
// children are sorted by entry distance, the nearest entered and the others
// pushed one by one with their distance (entries beyond the closest hit are
// dropped when pushed or popped).  The triangles of hit leaf children are
// tested after the eight box tests, before the push, so the box tests carry
// no triangle test between them (measured on Cornell at 1080p: 12.5 ->
// 11.1 ms of traversal per frame).  False when the ray is done.
template <bool kCount, int kStack>
__device__ __forceinline__ bool visit_sorted(const WideAccelDev& acc, const WideNode* sNodes,
                                             int cached, WideRay& r, uint2* stack,
                                             uint32_t& nodeVisits, uint32_t& triTests,
                                             uint32_t* errorFlag) {
    if (kCount) nodeVisits++;
    NodeSlabs s;
    node_slabs(acc, sNodes, cached, r.node, r, s);
    // internal children that are hit, keyed by entry distance:
    // (distance bits with the low three cleared) | slot
    uint32_t key[8];
    uint32_t m = 0;  // bit slot for each hit slot
    auto child = [&](auto kc) {
        constexpr int k = decltype(kc)::value;
        float tn, tf;
        child_span<k>(s, r.tmin, r.closest, tn, tf);
        const bool hit = tn <= tf;
        key[k] = (hit && ((s.imask >> k) & 1u)) ? ((__float_as_uint(tn) & 0x7FFFFFF8u) | uint32_t(k))
                                                : 0xFFFFFFFFu;
        if (hit) m |= 1u << k;
    };
    child(IntC<0>{}); child(IntC<1>{}); child(IntC<2>{}); child(IntC<3>{});
    child(IntC<4>{}); child(IntC<5>{}); child(IntC<6>{}); child(IntC<7>{});
    uint32_t leafHits = m & s.leafMask;
    while (leafHits) {
        const uint32_t k = uint32_t(__ffs(int(leafHits)) - 1);
        leafHits &= leafHits - 1u;
        if (kCount) triTests++;
        tri_test(acc, s.triBase + uint32_t(__popc(s.leafMask & ((1u << k) - 1u))), r.o, r.d,
                 r.tmin, r.closest, r.hitTri, r.hb0, r.hb1);
    }
    sort8(key);
    // push the farther hits (farthest first), enter the nearest
    int next = -1;
#pragma unroll
    for (int j = 7; j >= 0; j--) {
        if (key[j] == 0xFFFFFFFFu) continue;
        const float tn = __uint_as_float(key[j] & ~7u);
        if (tn > r.closest) continue;
        const uint32_t slot = key[j] & 7u;
        const uint32_t c = s.childBase + uint32_t(__popc(s.imask & ((1u << slot) - 1u)));
        if (j == 0) {
            next = int(c);
        } else if (r.sp < kStack) {
            stack[r.sp++] = make_uint2(c, key[j] & ~7u);
        } else {
            atomicExch(errorFlag, 3u);
        }
    }
    // the nearest hit may lie beyond the closest triangle: fall through to
    // the stack
    while (next < 0 && r.sp > 0) {
        const uint2 e = stack[--r.sp];
        if (__uint_as_float(e.y) <= r.closest) next = int(e.x);
    }
    r.node = next;
    return next >= 0;
}

// One node of the traversal in octant order: the collapse put every child
// in the slot of its centroid's octant around the node's centre, so the
// order slot ^ oct runs roughly front to back without sorting.  The stack
// holds node groups: the child base of a visited node, its internal-child
// mask and the bits of its hit internal children still to visit, one entry
// per node however many children were hit.  A child's node index is the
// child base plus the number of internal children in lower slots.  The
// triangles of hit leaf children are tested after the eight box tests, so
// the box tests carry no triangle test between them.  False when the ray
// is done.
template <bool kCount, int kStack>
__device__ __forceinline__ bool visit_octant(const WideAccelDev& acc, const WideNode* sNodes,
                                             int cached, WideRay& r, uint2* stack,
                                             uint32_t& nodeVisits, uint32_t& triTests,
                                             uint32_t* errorFlag) {
    if (kCount) nodeVisits++;
    NodeSlabs s;
    node_slabs(acc, sNodes, cached, r.node, r, s);
    const PackedSlabs p = packed_slabs(s);
    uint32_t m = 0;  // bit slot for each hit slot
    auto child = [&](auto kc) {
        constexpr int k = decltype(kc)::value;
        float tn[2], tf[2];
        child_spans<k>(s, p, r.tmin, r.closest, tn, tf);
        if (tn[0] <= tf[0]) m |= 1u << k;
        if (tn[1] <= tf[1]) m |= 1u << (k + 1);
    };
    child(IntC<0>{}); child(IntC<2>{}); child(IntC<4>{}); child(IntC<6>{});
    uint32_t leafHits = m & s.leafMask;
    while (leafHits) {
        const uint32_t k = uint32_t(__ffs(int(leafHits)) - 1);
        leafHits &= leafHits - 1u;
        if (kCount) triTests++;
        tri_test(acc, s.triBase + uint32_t(__popc(s.leafMask & ((1u << k) - 1u))), r.o, r.d,
                 r.tmin, r.closest, r.hitTri, r.hb0, r.hb1);
    }
    // hit internal children, bit k moved to k ^ oct (swapping bit pairs,
    // then pairs of pairs, then nibbles, as the octant's bits say)
    uint32_t hits = m & s.imask;
    hits = (r.oct & 1u) ? (((hits & 0x55u) << 1) | ((hits >> 1) & 0x55u)) : hits;
    hits = (r.oct & 2u) ? (((hits & 0x33u) << 2) | ((hits >> 2) & 0x33u)) : hits;
    hits = (r.oct & 4u) ? (((hits & 0x0Fu) << 4) | ((hits >> 4) & 0x0Fu)) : hits;
    uint32_t base = s.childBase, im = s.imask;
    if (hits == 0) {  // resume the most recent group with pending children
        if (r.sp == 0) {
            r.node = -1;
            return false;
        }
        const uint2 e = stack[--r.sp];
        base = e.x;
        im = e.y >> 8;
        hits = e.y & 0xFFu;
    }
    const uint32_t b = uint32_t(__ffs(int(hits)) - 1);
    const uint32_t slot = b ^ r.oct;
    hits &= hits - 1u;
    if (hits) {
        if (r.sp < kStack) stack[r.sp++] = make_uint2(base, (im << 8) | hits);
        else atomicExch(errorFlag, 3u);
    }
    r.node = int(base + uint32_t(__popc(im & ((1u << slot) - 1u))));
    return true;
}

template <bool kCount, bool kOctant, int kStack>
__device__ __forceinline__ bool wide_visit(const WideAccelDev& acc, const WideNode* sNodes,
                                           int cached, WideRay& r, uint2* stack,
                                           uint32_t& nodeVisits, uint32_t& triTests,
                                           uint32_t* errorFlag) {
    if (kOctant)
        return visit_octant<kCount, kStack>(acc, sNodes, cached, r, stack, nodeVisits, triTests,
                                            errorFlag);
    return visit_sorted<kCount, kStack>(acc, sNodes, cached, r, stack, nodeVisits, triTests,
                                        errorFlag);
}

// Stack entries per ray: the sorted order pushes one entry per child, the
// octant order one per node group (at most one per level).
template <bool kOctant>
struct WideStack {
    static constexpr int value = kOctant ? kWideGroups : kWideStack;
};

// Closest hit of one ray in one 8-wide tree, in either child order.
template <bool kCount, bool kOctant, int kStack>
__device__ __forceinline__ void trace_wide_ray(const WideAccelDev& acc, const WideNode* sNodes,
                                               int cached, float4 ro, float4 rd, WideRay& r,
                                               uint32_t& nodeVisits, uint32_t& triTests,
                                               uint32_t* errorFlag) {
    wide_ray_begin(r, ro, rd);
    if (acc.triCount == 1) {
        if (kCount) triTests++;
        tri_test(acc, 0, r.o, r.d, r.tmin, r.closest, r.hitTri, r.hb0, r.hb1);
    } else if (acc.triCount > 1) {
        uint2 stack[kStack];
        while (wide_visit<kCount, kOctant, kStack>(acc, sNodes, cached, r, stack, nodeVisits,
                                                   triTests, errorFlag)) {
        }
    }
}

// A next-event ray of a plain tracer that something stops brings no radiance, so
// it is reported as a miss and shading skips it: half of closed Cornell's hits
// (1080p, four samples per pixel, five depths: shading 3.99 -> 3.15 ms per frame).
// The WFPG tracer counts what stopped its rays and marks none.  Stopping
// the traversal at the first triangle nearer than the light was tried: the test
// in the node loops cost more (11.4 -> 11.6 ms; open scenes 3 %) than it saved.
__device__ __forceinline__ void write_hit(const WideAccelDev& acc, const HitOut& out, uint32_t i,
                                          float tmin, int hitTri, float closest, float hb0,
                                          float hb1) {
    uint32_t key = kBatchNull;
    if (hitTri >= 0) {
        key = __float_as_uint(__ldg(&acc.te0[hitTri].w));
        const uint32_t mark = __float_as_uint(tmin);
        if (out.shadowRays && is_shadow_tmin(mark) &&
            key != ((kBatchLight << kIdBits) | (mark & 0x7FFFFFu)))
            key = kBatchNull;
    }
    if (key != kBatchNull) {
        out.key[i] = key;
        out.prim[i] = __float_as_uint(__ldg(&acc.tv0[hitTri].w));
        out.t[i] = closest;
        out.bary[i] = make_float2(hb0, hb1);
    } else {
        out.key[i] = kBatchNull;
        out.prim[i] = kInvalid;
        out.t[i] = closest;
        out.bary[i] = make_float2(0.0f, 0.0f);
    }
}

__device__ __forceinline__ void load_top_nodes(const WideAccelDev& acc, WideNode* sNodes,
                                               int cached) {
    for (int i = threadIdx.x; i < cached * 5; i += blockDim.x)
        reinterpret_cast<uint4*>(sNodes)[i] = __ldg(reinterpret_cast<const uint4*>(acc.nodes) + i);
    __syncthreads();
}

__device__ __forceinline__ void add_work(unsigned long long* counters, uint32_t nodeVisits,
                                         uint32_t triTests) {
    unsigned long long a = nodeVisits, b = triTests;
    for (int s = 16; s > 0; s >>= 1) {
        a += __shfl_xor_sync(0xFFFFFFFFu, a, s);
        b += __shfl_xor_sync(0xFFFFFFFFu, b, s);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(counters + 0, a);
        atomicAdd(counters + 1, b);
    }
}

// Eight 128-thread blocks per SM (64 registers, no spill): the traversal's
// dependent loads and ALU chains want resident warps more than registers,
// but not at the price of spills.  Octant order on clusters-1M: 2.66 ms of
// traversal per frame at eight blocks, 2.70 at nine (56 registers), 2.84 at
// ten (48, spilling); sorted order on the closed Cornell frame: 34.5 ms at
// eight, 34.9 at nine.
template <bool kCount, bool kOctant>
__global__ void __launch_bounds__(128, 8) k_trace_wide(WideAccelDev acc,
                                                    const float4* __restrict__ rayO,
                                                    const float4* __restrict__ rayD,
                                                    const uint32_t* __restrict__ dCount,
                                                    uint32_t hCount, HitOut out,
                                                    uint32_t* errorFlag,
                                                    unsigned long long* counters) {
    __shared__ WideNode sNodes[kCachedNodes];
    const int cached = acc.nodeCount < uint32_t(kCachedNodes) ? int(acc.nodeCount) : kCachedNodes;
    load_top_nodes(acc, sNodes, cached);
    const uint32_t n = dCount ? *dCount : hCount;
    uint32_t nodeVisits = 0, triTests = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        WideRay r;
        trace_wide_ray<kCount, kOctant, WideStack<kOctant>::value>(
            acc, sNodes, cached, rayO[i], rayD[i], r, nodeVisits, triTests, errorFlag);
        write_hit(acc, out, i, r.tmin, r.hitTri, r.closest, r.hb0, r.hb1);
    }
    if (kCount) add_work(counters, nodeVisits, triTests);
}

// Lanes refilled: a lane whose ray is done takes its warp's next ray once
// kRefillLanes lanes (or all) are idle, so a warp of rays with uneven path
// lengths keeps its lanes busy until its rays run out.  Warp w owns the
// 32-ray chunks w, w + W, w + 2W, ... (W warps in the grid) and hands their
// rays out in order; the set of rays a warp traces is the same as without
// refilling, only the lanes they run on differ.  Refilling mixes rays of
// neighbouring chunks in one warp: a gain for the scattered rays of later
// bounces, a loss for coherent camera rays (measured per depth by the
// tracer's order tuning).
constexpr int kRefillLanes = 8;

template <bool kCount, bool kOctant>
__global__ void __launch_bounds__(128, 8) k_trace_wide_refill(WideAccelDev acc,
                                                           const float4* __restrict__ rayO,
                                                           const float4* __restrict__ rayD,
                                                           const uint32_t* __restrict__ dCount,
                                                           uint32_t hCount, HitOut out,
                                                           uint32_t* errorFlag,
                                                           unsigned long long* counters) {
    constexpr int kStack = WideStack<kOctant>::value;
    __shared__ WideNode sNodes[kCachedNodes];
    const int cached = acc.nodeCount < uint32_t(kCachedNodes) ? int(acc.nodeCount) : kCachedNodes;
    load_top_nodes(acc, sNodes, cached);
    const uint32_t n = dCount ? *dCount : hCount;
    uint32_t nodeVisits = 0, triTests = 0;
    if (acc.triCount < 2) {
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
             i += gridDim.x * blockDim.x) {
            WideRay r;
            trace_wide_ray<kCount, kOctant, kStack>(acc, sNodes, cached, rayO[i], rayD[i], r,
                                                    nodeVisits, triTests, errorFlag);
            write_hit(acc, out, i, r.tmin, r.hitTri, r.closest, r.hb0, r.hb1);
        }
    } else {
        const uint32_t lane = threadIdx.x & 31u;
        const uint64_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        const uint64_t nWarps = (gridDim.x * blockDim.x) >> 5;
        uint32_t next = 0;  // rays of the warp's sequence handed out (warp-uniform)
        bool more = warp * 32u < n, active = false;
        uint32_t ri = 0;
        WideRay r;
        r.node = -1;
        uint2 stack[kStack];
        while (true) {
            if (more) {
                const uint32_t need = __ballot_sync(0xFFFFFFFFu, !active);
                if (__popc(need) >= kRefillLanes || need == 0xFFFFFFFFu) {
                    if (!active) {
                        const uint32_t j = next + uint32_t(__popc(need & ((1u << lane) - 1u)));
                        const uint64_t idx = (warp + uint64_t(j >> 5) * nWarps) * 32u + (j & 31u);
                        if (idx < n) {
                            ri = uint32_t(idx);
                            wide_ray_begin(r, rayO[ri], rayD[ri]);
                            active = true;
                        }
                    }
                    next += uint32_t(__popc(need));
                    more = (warp + uint64_t(next >> 5) * nWarps) * 32u + (next & 31u) < n;
                }
            }
            if (!__any_sync(0xFFFFFFFFu, active)) break;
            if (!active) continue;
            if (!wide_visit<kCount, kOctant, kStack>(acc, sNodes, cached, r, stack, nodeVisits,
                                                     triTests, errorFlag)) {
                write_hit(acc, out, ri, r.tmin, r.hitTri, r.closest, r.hb0, r.hb1);
                active = false;
            }
        }
    }
    if (kCount) add_work(counters, nodeVisits, triTests);
}

// ---------------------------------------------------------------------------
// One warp per ray, for a few thousand rays
// ---------------------------------------------------------------------------
// With one lane per ray so few rays leave most schedulers a warp or none, and
// the launch lasts as long as its longest ray's chain of node visits, each a
// dependent read and eight box tests (2,000 rays over 1M triangles: 96 us).
// Here a warp takes a ray: up to four pending nodes at a time, one per team of
// eight lanes, one child slot per lane; the triangles of all hit leaves at once,
// one per lane.  Lane k of a team has slot k ^ (ray octant), so that lower lanes
// are nearer and the hits are pushed to be taken in that order, the top node's
// first.  Entries keep their distance and are dropped once a nearer hit is
// known.  The nodes taken beside the top one are speculative; what they cost
// is idle hardware here, which is why larger launches trace with one lane per
// ray (wide_warp_rays).  The fastest of those kernels and this one, random rays over
// clusters 1M and Cornell: 2,000 rays 97 and 24 us, 41 and 13; 16,000 rays 103 and
// 60, 58 and 27; 32,000 rays 110 and 102, 60 and 46; the same at 64,000.
constexpr int kWarpStack = 256;       // entries per warp
constexpr int kWarpBlock = 128;

__global__ void __launch_bounds__(kWarpBlock) k_trace_wide_warp(
    WideAccelDev acc, const float4* __restrict__ rayO, const float4* __restrict__ rayD, uint32_t n,
    HitOut out, uint32_t* errorFlag) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    __shared__ uint2 stacks[kWarpBlock / 32][kWarpStack];
    const uint32_t lane = threadIdx.x & 31u, team = lane >> 3;
    uint2* stack = stacks[threadIdx.x >> 5];
    const uint32_t warps = (gridDim.x * kWarpBlock) >> 5;
    uint32_t nodeVisits = 0, triTests = 0;  // not asked for
    for (uint32_t i = (blockIdx.x * kWarpBlock + threadIdx.x) >> 5; i < n; i += warps) {
        WideRay r;
        uint32_t owner = 0;
        wide_ray_begin(r, rayO[i], rayD[i]);
        const uint32_t slot = (lane & 7u) ^ r.oct;
        int sp = 1;
        __syncwarp();
        if (lane == 0) stack[0] = make_uint2(0u, 0u);
        __syncwarp();
        while (sp > 0) {
            // deep in the stack one node at a time, as a plain depth-first
            // traversal, which adds at most seven entries per level
            const int take = sp > kWarpStack / 2 ? 1 : min(sp, 4);
            uint2 e = make_uint2(0u, 0u);
            bool active = int(team) < take;
            if (active) {
                e = stack[sp - 1 - int(team)];
                active = __uint_as_float(e.y) <= r.closest;
            }
            sp -= take;
            bool inner = false, leaf = false;
            uint32_t child = 0;
            float tn = 0.0f;
            if (active) {
                const uint4* g = reinterpret_cast<const uint4*>(acc.nodes + e.x);
                const uint8_t* q = reinterpret_cast<const uint8_t*>(g + 2) + slot;
                const uint4 w0 = __ldg(g), w1 = __ldg(g + 1);
                const float lx = float(__ldg(q)), ly = float(__ldg(q + 8)),
                            lz = float(__ldg(q + 16)), hx = float(__ldg(q + 24)),
                            hy = float(__ldg(q + 32)), hz = float(__ldg(q + 40));
                const float ax = __uint_as_float((w0.w & 0xFFu) << 23) * r.inv.x;
                const float ay = __uint_as_float(((w0.w >> 8) & 0xFFu) << 23) * r.inv.y;
                const float az = __uint_as_float(((w0.w >> 16) & 0xFFu) << 23) * r.inv.z;
                const float bx = (__uint_as_float(w0.x) - r.o.x) * r.inv.x;
                const float by = (__uint_as_float(w0.y) - r.o.y) * r.inv.y;
                const float bz = (__uint_as_float(w0.z) - r.o.z) * r.inv.z;
                const bool px = !(r.oct & 1u), py = !(r.oct & 2u), pz = !(r.oct & 4u);
                tn = fmaxf(fmaxf(__fmaf_rn(px ? lx : hx, ax, bx), __fmaf_rn(py ? ly : hy, ay, by)),
                           fmaxf(__fmaf_rn(pz ? lz : hz, az, bz), r.tmin));
                const float tf =
                    fminf(fminf(__fmaf_rn(px ? hx : lx, ax, bx), __fmaf_rn(py ? hy : ly, ay, by)),
                          fminf(__fmaf_rn(pz ? hz : lz, az, bz), r.closest));
                if (tn <= tf) {
                    const uint32_t imask = w0.w >> 24, below = (1u << slot) - 1u;
                    inner = (imask >> slot) & 1u;
                    leaf = (w1.z >> slot) & 1u;
                    child = inner ? w1.x + uint32_t(__popc(imask & below))
                                  : w1.y + uint32_t(__popc(w1.z & below));
                }
            }
            if (__any_sync(kAll, leaf)) {
                float t = r.closest, b0 = 0.0f, b1 = 0.0f;
                int tri = -1;
                if (leaf) tri_test(acc, child, r.o, r.d, r.tmin, t, tri, b0, b1);
                // distances are positive: their bits order as they do
                const uint32_t key = tri >= 0 ? __float_as_uint(t) : kAll;
                const uint32_t best = __reduce_min_sync(kAll, key);
                if (best != kAll) {
                    owner = uint32_t(__ffs(int(__ballot_sync(kAll, key == best))) - 1);
                    r.closest = __uint_as_float(best);
                    if (lane == owner) {
                        r.hitTri = tri;
                        r.hb0 = b0;
                        r.hb1 = b1;
                    }
                }
            }
            const uint32_t push = __ballot_sync(kAll, inner);
            if (sp + __popc(push) > kWarpStack) {
                // a tree deeper than any the builds make: this ray again, by
                // one lane with the octant kernel's stack
                if (lane == 0)
                    trace_wide_ray<false, true, kWideGroups>(acc, nullptr, 0, rayO[i], rayD[i], r,
                                                             nodeVisits, triTests, errorFlag);
                owner = 0;
                break;
            }
            // the first lane's child on top
            if (inner)
                stack[sp + __popc(push & ~((2u << lane) - 1u))] =
                    make_uint2(child, __float_as_uint(tn));
            sp += __popc(push);
            __syncwarp();
        }
        if (lane == owner)
            write_hit(acc, out, i, r.tmin, r.hitTri, r.closest, r.hb0, r.hb1);
    }
}

// Rays of many scenes: each ray's tree is its job's (RayAux::pad is the job
// slot).  No shared-memory top levels: neighbouring rays may use different
// trees.  kRefill: as k_trace_wide_refill, a warp's idle lanes take its next
// rays (the scattered rays after the first depth; camera rays are coherent).
// 64 registers, as many warps as the single-scene kernels.  24 jobs on 6 Cornell
// scenes of 64,000 triangles and fewer, 4 frames: 15.5 ms without, 13.7 ms so.
template <int kBlock, int kStack, bool kOctant, bool kRefill>
__global__ void __launch_bounds__(kBlock, 1024 / kBlock) k_trace_wide_jobs(
    const JobDev* __restrict__ jobs, const RayAux* __restrict__ aux,
    const float4* __restrict__ rayO, const float4* __restrict__ rayD,
    const uint32_t* __restrict__ dCount, uint32_t hCount, HitOut out, uint32_t* errorFlag) {
    constexpr int kEntries = kOctant ? kWideGroups : kStack;
    const uint32_t n = dCount ? *dCount : hCount;
    uint32_t nodeVisits = 0, triTests = 0;
    if constexpr (!kRefill) {
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
             i += gridDim.x * blockDim.x) {
            const WideAccelDev acc = jobs[aux[i].pad].wide;
            WideRay r;
            trace_wide_ray<false, kOctant, kEntries>(acc, nullptr, 0, rayO[i], rayD[i], r,
                                                     nodeVisits, triTests, errorFlag);
            write_hit(acc, out, i, r.tmin, r.hitTri, r.closest, r.hb0, r.hb1);
        }
    } else {
        const uint32_t lane = threadIdx.x & 31u;
        const uint64_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        const uint64_t nWarps = (gridDim.x * blockDim.x) >> 5;
        uint32_t next = 0;  // rays of the warp's sequence handed out (warp-uniform)
        bool more = warp * 32u < n, active = false;
        uint32_t ri = 0;
        WideAccelDev acc{};
        WideRay r;
        r.node = -1;
        uint2 stack[kEntries];
        while (true) {
            if (more) {
                const uint32_t need = __ballot_sync(0xFFFFFFFFu, !active);
                if (__popc(need) >= kRefillLanes || need == 0xFFFFFFFFu) {
                    if (!active) {
                        const uint32_t j = next + uint32_t(__popc(need & ((1u << lane) - 1u)));
                        const uint64_t idx = (warp + uint64_t(j >> 5) * nWarps) * 32u + (j & 31u);
                        if (idx < n) {
                            ri = uint32_t(idx);
                            acc = jobs[aux[ri].pad].wide;
                            wide_ray_begin(r, rayO[ri], rayD[ri]);
                            active = true;
                        }
                    }
                    next += uint32_t(__popc(need));
                    more = (warp + uint64_t(next >> 5) * nWarps) * 32u + (next & 31u) < n;
                }
            }
            if (!__any_sync(0xFFFFFFFFu, active)) break;
            if (!active) continue;
            bool going = false;
            if (acc.triCount > 1)
                going = wide_visit<false, kOctant, kEntries>(acc, nullptr, 0, r, stack, nodeVisits,
                                                             triTests, errorFlag);
            else if (acc.triCount == 1)
                tri_test(acc, 0, r.o, r.d, r.tmin, r.closest, r.hitTri, r.hb0, r.hb1);
            if (!going) {
                write_hit(acc, out, ri, r.tmin, r.hitTri, r.closest, r.hb0, r.hb1);
                active = false;
            }
        }
    }
}

}  // namespace

namespace {
size_t align256(size_t b) { return (b + 255) & ~size_t(255); }
size_t queue_bytes(uint32_t n) {
    return align256(size_t(n + 1) * sizeof(WorkItem) * 2 + size_t(kCounters) * 4);
}
}  // namespace

size_t wide_scratch_bytes(uint32_t n) {
    // two work queues of n items and the counters; the collapse plan: parents
    // (2n), arrival flags (n), costs (8n) and plans (n)
    return queue_bytes(n) + align256(size_t(2) * n * 4) + align256(size_t(n) * 4) +
           align256(size_t(8) * n * 4) + align256(size_t(n) * 8);
}

int wide_build(const WideBuildIn& in, WideNode* nodes, float4* tv0, float4* te0, float4* te1,
               void* scratch, uint32_t* nodeCountOut, cudaStream_t stream) {
    const uint32_t n = in.n;
    if (n < 2) {
        set_error("wide BVH: needs at least two triangles");
        return MRB_E_ARG;
    }
    WorkItem* q[2];
    q[0] = static_cast<WorkItem*>(scratch);
    q[1] = q[0] + (n + 1);
    uint32_t* counters = reinterpret_cast<uint32_t*>(q[1] + (n + 1));
    const uint2* plan = nullptr;
    if (in.collapse == kWideCollapseSah) {
        char* b = static_cast<char*>(scratch) + queue_bytes(n);
        uint32_t* parent = reinterpret_cast<uint32_t*>(b);
        b += align256(size_t(2) * n * 4);
        uint32_t* flags = reinterpret_cast<uint32_t*>(b);
        b += align256(size_t(n) * 4);
        float* cost = reinterpret_cast<float*>(b);
        b += align256(size_t(8) * n * 4);
        uint2* pl = reinterpret_cast<uint2*>(b);
        const uint32_t g = std::min<uint32_t>((n + 255) / 256, 148u * 8u);
        k_plan_parents<<<g, 256, 0, stream>>>(in.left, in.right, n, parent, flags);
        k_plan_up<<<g, 256, 0, stream>>>(in.left, in.right, in.inner, parent, in.root, n, flags,
                                         cost, pl);
        MRB_CUDA(cudaGetLastError());
        plan = pl;
    }
    MRB_CUDA(cudaMemsetAsync(counters, 0, size_t(kCounters) * 4, stream));
    k_collapse_init<<<1, 32, 0, stream>>>(q[0], counters, in.root);
    MRB_CUDA(cudaGetLastError());
    // one launch per level; the host checks for an empty queue every 8 levels
    const uint32_t grid = std::min<uint32_t>(n / (kCollapseBlock / 8) + 1, 148u * 16u);
    for (int level = 0; level < kMaxLevels; level++) {
        uint32_t* qc = counters + 2 + level;
        k_collapse<<<grid, kCollapseBlock, 0, stream>>>(
            q[level & 1], qc, q[(level & 1) ^ 1], qc + 1, counters, counters + 1, n, in.left,
            in.right, in.inner, in.triAabb, in.sortedIdx, in.pos, in.idx, in.key, in.cull, plan,
            nodes, tv0, te0, te1);
        MRB_CUDA(cudaGetLastError());
        if ((level & 7) == 7) {
            uint32_t h[2], left = 0;
            MRB_CUDA(cudaMemcpyAsync(h, counters, 8, cudaMemcpyDeviceToHost, stream));
            MRB_CUDA(cudaMemcpyAsync(&left, qc + 1, 4, cudaMemcpyDeviceToHost, stream));
            MRB_CUDA(cudaStreamSynchronize(stream));
            if (left == 0) {
                if (h[1] != n) {
                    set_error("wide BVH: %u of %u triangles placed", h[1], n);
                    return MRB_E_DEVICE;
                }
                *nodeCountOut = h[0];
                return 0;
            }
        }
    }
    set_error("wide BVH: collapse did not finish");
    return MRB_E_DEVICE;
}

int trace_closest_wide_few(const WideAccelDev& acc, const float4* rayO, const float4* rayD,
                           uint32_t n, const HitOut& out, uint32_t* errorFlag,
                           cudaStream_t stream) {
    k_trace_wide_warp<<<std::min((n + 3u) / 4u, 148u * 16u), kWarpBlock, 0, stream>>>(
        acc, rayO, rayD, n, out, errorFlag);
    MRB_CUDA(cudaGetLastError());
    return 0;
}

int trace_closest_wide(const WideAccelDev& acc, const float4* rayO, const float4* rayD,
                       const uint32_t* dCount, uint32_t maxCount, const HitOut& out,
                       uint32_t* errorFlag, cudaStream_t stream, unsigned long long* counters,
                       int order) {
    if (maxCount == 0) return 0;
    uint32_t blocks = (maxCount + 127) / 128;
    blocks = blocks < 148u * 16u ? blocks : 148u * 16u;
    auto go = [&](auto kernel) {
        kernel<<<blocks, 128, 0, stream>>>(acc, rayO, rayD, dCount, maxCount, out, errorFlag,
                                           counters);
    };
    const bool c = counters != nullptr;
    switch (order) {
        case kWideSorted: c ? go(k_trace_wide<true, false>) : go(k_trace_wide<false, false>); break;
        case kWideOctant: c ? go(k_trace_wide<true, true>) : go(k_trace_wide<false, true>); break;
        case kWideSortedRefill:
            c ? go(k_trace_wide_refill<true, false>) : go(k_trace_wide_refill<false, false>);
            break;
        case kWideOctantRefill:
            c ? go(k_trace_wide_refill<true, true>) : go(k_trace_wide_refill<false, true>);
            break;
        default:
            set_error("wide traversal: order %d unknown", order);
            return MRB_E_ARG;
    }
    MRB_CUDA(cudaGetLastError());
    return 0;
}

namespace {
// Seeded probe rays over the scene's box: origins uniform in it, directions
// uniform on the sphere (Philox counter (i, 0, 0x60000, 0)).
__global__ void k_probe_rays(const float* __restrict__ ext, uint32_t n, float4* rayO,
                             float4* rayD) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const Rand4 r = philox_uniform4(i, 0u, 0x60000u, 0u, 0x5eedu, 0u);
        const Rand4 q = philox_uniform4(i, 1u, 0x60000u, 0u, 0x5eedu, 0u);
        float o[3];
        for (int c = 0; c < 3; c++) o[c] = ext[c] + r.u[c] * (ext[3 + c] - ext[c]);
        const float z = 1.0f - 2.0f * q.u[0];
        const float rr = sqrtf(fmaxf(0.0f, 1.0f - z * z));
        float sn, cs;
        pm_sincos(6.2831853f * q.u[1], sn, cs);
        rayO[i] = make_float4(o[0], o[1], o[2], 0.0f);
        rayD[i] = make_float4(rr * cs, rr * sn, z, 3.0e38f);
    }
}
}  // namespace

namespace {
constexpr uint32_t kProbe = 1u << 16;
struct ProbeBuffers {
    float4 *ro, *rd;
    HitOut ho;
    unsigned long long* work;  // two pairs of counters
    uint32_t* err;
};
ProbeBuffers probe_buffers(void* scratch) {
    ProbeBuffers b{};
    b.ro = static_cast<float4*>(scratch);
    b.rd = b.ro + kProbe;
    b.work = reinterpret_cast<unsigned long long*>(b.rd + kProbe);
    b.ho.bary = reinterpret_cast<float2*>(b.work + 4);
    b.ho.key = reinterpret_cast<uint32_t*>(b.ho.bary + kProbe);
    b.ho.prim = b.ho.key + kProbe;
    b.ho.t = reinterpret_cast<float*>(b.ho.prim + kProbe);
    b.err = reinterpret_cast<uint32_t*>(b.ho.t + kProbe);
    return b;
}
}  // namespace

size_t wide_probe_bytes() { return size_t(kProbe) * (16 + 16 + 4 + 4 + 4 + 8) + 64; }

int wide_order_autotune(const WideAccelDev& acc, const float* dExtent, void* scratch,
                        cudaStream_t st, int* orderOut, float* msOut) {
    const ProbeBuffers b = probe_buffers(scratch);
    // pass 0, on a few rays, loads the kernels; of the two timed passes the
    // faster counts.  Everything is enqueued, then waited for once.
    constexpr int kPasses = 3;
    cudaEvent_t e[kPasses][kWideOrders + 1] = {};
    int rc = 0;
    k_probe_rays<<<(kProbe + 255) / 256, 256, 0, st>>>(dExtent, kProbe, b.ro, b.rd);
    for (int pass = 0; pass < kPasses && rc == 0; pass++)
        for (int order = 0; order <= kWideOrders && rc == 0; order++) {
            if (cudaEventCreate(&e[pass][order]) != cudaSuccess) rc = MRB_E_CUDA;
            cudaEventRecord(e[pass][order], st);
            if (rc == 0 && order < kWideOrders)
                rc = trace_closest_wide(acc, b.ro, b.rd, nullptr, pass ? kProbe : kProbe / 16, b.ho,
                                        b.err, st, nullptr, order);
        }
    const cudaError_t waited = cudaStreamSynchronize(st);
    float best[kWideOrders];
    for (int o = 0; o < kWideOrders; o++) {
        best[o] = 1e30f;
        for (int pass = 1; pass < kPasses && rc == 0; pass++) {
            float ms = 0.0f;
            if (cudaEventElapsedTime(&ms, e[pass][o], e[pass][o + 1]) == cudaSuccess)
                best[o] = std::min(best[o], ms);
        }
    }
    for (auto& pass : e)
        for (cudaEvent_t ev : pass)
            if (ev) cudaEventDestroy(ev);
    if (rc) return rc;
    MRB_CUDA(waited);
    MRB_CUDA(cudaGetLastError());
    int pick = 0;
    for (int o = 1; o < kWideOrders; o++)
        if (best[o] < best[pick]) pick = o;
    *orderOut = pick;
    if (msOut)
        for (int o = 0; o < kWideOrders; o++) msOut[o] = best[o];
    return 0;
}

int wide_probe_compare(const WideAccelDev& a, const WideAccelDev& b, const float* dExtent,
                       void* scratch, cudaStream_t st, double bytesOut[2]) {
    const ProbeBuffers p = probe_buffers(scratch);
    MRB_CUDA(cudaMemsetAsync(p.work, 0, 32, st));
    MRB_CUDA(cudaMemsetAsync(p.err, 0, 4, st));
    k_probe_rays<<<(kProbe + 255) / 256, 256, 0, st>>>(dExtent, kProbe, p.ro, p.rd);
    for (int which = 0; which < 2; which++)
        if (int rc = trace_closest_wide(which ? b : a, p.ro, p.rd, nullptr, kProbe, p.ho, p.err, st,
                                        p.work + 2 * which, kWideOctant))
            return rc;
    unsigned long long h[4] = {0ull, 0ull, 0ull, 0ull};
    MRB_CUDA(cudaMemcpyAsync(h, p.work, 32, cudaMemcpyDeviceToHost, st));
    MRB_CUDA(cudaStreamSynchronize(st));
    for (int which = 0; which < 2; which++)
        bytesOut[which] = double(h[2 * which]) * double(sizeof(WideNode)) +
                          double(h[2 * which + 1]) * 48.0;
    return 0;
}

template <int kBlock, int kStack, bool kOctant>
static int launch_jobs(const JobDev* jobs, const RayAux* aux, const float4* rayO,
                       const float4* rayD, const uint32_t* dCount, uint32_t maxCount,
                       const HitOut& out, uint32_t* errorFlag, bool refill, cudaStream_t stream) {
    uint32_t blocks = (maxCount + kBlock - 1) / kBlock;
    const uint32_t cap = 148u * (2048u / kBlock);
    blocks = blocks < cap ? blocks : cap;
    if (refill)
        k_trace_wide_jobs<kBlock, kStack, kOctant, true><<<blocks, kBlock, 0, stream>>>(
            jobs, aux, rayO, rayD, dCount, maxCount, out, errorFlag);
    else
        k_trace_wide_jobs<kBlock, kStack, kOctant, false><<<blocks, kBlock, 0, stream>>>(
            jobs, aux, rayO, rayD, dCount, maxCount, out, errorFlag);
    MRB_CUDA(cudaGetLastError());
    return 0;
}

template <int kBlock>
static int launch_jobs_stack(const JobDev* jobs, const RayAux* aux, const float4* rayO,
                             const float4* rayD, const uint32_t* dCount, uint32_t maxCount,
                             const HitOut& out, uint32_t* errorFlag, int stack, bool refill,
                             cudaStream_t stream) {
    if (stack == 0)
        return launch_jobs<kBlock, kWideStack, true>(jobs, aux, rayO, rayD, dCount, maxCount, out,
                                                     errorFlag, refill, stream);
    if (stack > 64)
        return launch_jobs<kBlock, 128, false>(jobs, aux, rayO, rayD, dCount, maxCount, out,
                                               errorFlag, refill, stream);
    return launch_jobs<kBlock, 64, false>(jobs, aux, rayO, rayD, dCount, maxCount, out, errorFlag,
                                          refill, stream);
}

int trace_closest_wide_jobs(const JobDev* jobs, const RayAux* aux, const float4* rayO,
                            const float4* rayD, const uint32_t* dCount, uint32_t maxCount,
                            const HitOut& out, uint32_t* errorFlag, int block, int stack,
                            bool refill, cudaStream_t stream) {
    if (maxCount == 0) return 0;
    switch (block) {
        case 64:
            return launch_jobs_stack<64>(jobs, aux, rayO, rayD, dCount, maxCount, out, errorFlag,
                                         stack, refill, stream);
        case 256:
            return launch_jobs_stack<256>(jobs, aux, rayO, rayD, dCount, maxCount, out, errorFlag,
                                          stack, refill, stream);
        default:
            return launch_jobs_stack<128>(jobs, aux, rayO, rayD, dCount, maxCount, out, errorFlag,
                                          stack, refill, stream);
    }
}

}  // namespace mrb
