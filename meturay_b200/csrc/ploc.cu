// Traversal tree by parallel locally-ordered clustering (PLOC; Meister and
// Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume
// Hierarchy Construction", IEEE TVCG 2018), from the LBVH's Morton-sorted
// leaves.
//
// The LBVH splits where the Morton codes split, so over a sparse scene its
// upper nodes are loose boxes around far-apart geometry and rays open many
// of them to find nothing.  PLOC builds bottom-up instead: every cluster
// (first the leaves, in Morton order) looks for the neighbour within a
// window of kRadius clusters on either side whose merged box has the least
// surface area; mutually nearest pairs merge into a new inner node; the
// survivors are compacted, keeping their Morton order, and the step repeats
// until one cluster is left.  Every step is deterministic: ties go to the
// lower index and new nodes are numbered by a prefix sum over the merging
// pairs.
//
// The result uses the LBVH's numbering (leaf g < n is sorted slot g, inner
// node j is global n + j), so the 8-wide collapse (wide.cu) takes it as it
// takes the LBVH.  The LBVH itself, in the reference's numbering, is kept
// unchanged for its parity checks and the binary traversal.
#include <algorithm>

#include "../../include/mrb200.h"
#include "common.cuh"
#include "ploc.cuh"

namespace mrb {
namespace {

constexpr int kRadius = 16;
constexpr int kTile = 256;                      // clusters per block of a step
constexpr int kStepBlock = kTile + 2 * kRadius; // one thread per nearest neighbour needed
constexpr int kFinal = 1024;                    // clusters one block finishes by itself
constexpr int kBatch = 8;                       // steps enqueued between looks at the count
constexpr uint32_t kSpinLimit = 1u << 24;

// Where the clustering stands: clusters left, inner nodes made, steps taken.
struct PlocState {
    uint32_t m, base, steps;
};
// What the host reads after a batch: the last state, and the give-up word that
// lies behind it (1 once a look-back has given up).
struct PlocProgress {
    PlocState state;
    uint32_t gaveUp;
};

__device__ __forceinline__ void node_box(uint32_t g, const PlocIn& in, const float* inner,
                                         float b[6]) {
    const float* s = (g < in.n) ? in.triAabb + 6 * size_t(in.sortedIdx[g])
                                : inner + 6 * size_t(g - in.n);
    for (int c = 0; c < 6; c++) b[c] = s[c];
}

__device__ __forceinline__ float merged_area(const float* a, const float* b) {
    const float dx = fmaxf(a[3], b[3]) - fminf(a[0], b[0]);
    const float dy = fmaxf(a[4], b[4]) - fminf(a[1], b[1]);
    const float dz = fmaxf(a[5], b[5]) - fminf(a[2], b[2]);
    return dx * dy + dy * dz + dz * dx;
}

// Nearest neighbour of cluster i (of m) in [i - kRadius, i + kRadius]; boxes
// points at cluster i's box, its neighbours' boxes lie beside it.
__device__ __forceinline__ int nearest(const float* boxes, int i, int m) {
    float best = INFINITY;
    int bj = (i == 0) ? 1 : i - 1;
    for (int d = -kRadius; d <= kRadius; d++) {
        const int j = i + d;
        if (d == 0 || j < 0 || j >= m) continue;
        const float a = merged_area(boxes, boxes + 6 * d);
        if (a < best) {  // ascending j: equal areas keep the lower index
            best = a;
            bj = j;
        }
    }
    return bj;
}

// Exclusive block sum of packed counts (merges << 16 | keeps) over the first
// 32 * kWarps threads; total for all threads.  Every thread calls it.
template <int kWarps>
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* warpSum, uint32_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warpSum[warp] = x;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (int w = 0; w < kWarps; w++) {
        if (w == warp) before = all;
        all += warpSum[w];
    }
    total = all;
    return before + x - v;
}

// The merge of clusters a and b into inner node `node`.
__device__ __forceinline__ void make_node(const PlocOut& out, uint32_t node, uint32_t a, uint32_t b,
                                          const float* ba, const float* bb, float* box) {
    for (int c = 0; c < 3; c++) {
        box[c] = fminf(ba[c], bb[c]);
        box[3 + c] = fmaxf(ba[3 + c], bb[3 + c]);
    }
    float* o = out.inner + 6 * size_t(node);
    for (int c = 0; c < 6; c++) o[c] = box[c];
    out.left[node] = a;
    out.right[node] = b;
}

// One clustering step in one kernel: every cluster's nearest neighbour (the
// tile's and kRadius more on either side, from boxes staged in shared memory),
// the mutually nearest pairs, the prefix sums over merging pairs and surviving
// clusters (decoupled look-back over the tiles, taken by ticket), the new
// nodes and the compacted survivors.  It was seven launches and two copies to
// the host per step, which the launch and copy latencies bounded (1M
// triangles: 74 steps of 50 us; here 48 launches of 18 us on average, then
// 131 us in k_ploc_finish for the last kFinal clusters).
// Counts and node numbers travel on the device: step k reads state k and
// leaves state k + 1.  With kFinal clusters or fewer, or after a look-back that
// gave up, a step does nothing.  The give-up word may be set while a block
// starts, so one thread reads it for the block: the others' share of the boxes
// is either there or not looked at.
__global__ void __launch_bounds__(kStepBlock) k_ploc_step(const uint32_t* __restrict__ C,
                                                          uint32_t* __restrict__ Cout, PlocIn in,
                                                          PlocOut out, const PlocState* cur,
                                                          PlocState* next, uint32_t* ticket,
                                                          uint32_t* error,
                                                          unsigned long long* status) {
    __shared__ float sb[(kTile + 4 * kRadius) * 6];
    __shared__ uint32_t ids[kTile + 4 * kRadius];
    __shared__ int nn[kStepBlock];
    __shared__ uint32_t warpSum[kStepBlock / 32];
    __shared__ uint32_t tileId;
    __shared__ unsigned long long prefix;
    const int tid = int(threadIdx.x);
    const PlocState st = *cur;
    const int m = int(st.m);
    if (st.m <= uint32_t(kFinal)) {
        if (blockIdx.x == 0 && tid == 0) *next = st;
        return;
    }
    if (tid == 0) tileId = *error ? kInvalid : atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = tileId;
    if (tile == kInvalid) return;
    const int b0 = int(tile) * kTile;
    if (b0 >= m) return;
    for (int k = tid; k < kTile + 4 * kRadius; k += kStepBlock) {
        const int j = b0 - 2 * kRadius + k;
        if (j >= 0 && j < m) {
            ids[k] = C[j];
            node_box(ids[k], in, out.inner, sb + 6 * k);
        }
    }
    __syncthreads();
    {
        const int i = b0 - kRadius + tid;
        nn[tid] = (i >= 0 && i < m) ? nearest(sb + 6 * (tid + kRadius), i, m) : -1;
    }
    __syncthreads();
    const int i = b0 + tid;  // threads below kTile: the tile's clusters
    const bool mine = tid < kTile && i < m;
    uint32_t flags = 0;
    int j = 0;
    if (mine) {
        j = nn[tid + kRadius];
        const bool mutual = nn[j - b0 + kRadius] == i;
        flags = ((mutual && i < j) ? 0x10000u : 0u) | ((mutual && i > j) ? 0u : 1u);
    }
    uint32_t total;
    const uint32_t before = block_scan<kStepBlock / 32>(flags, warpSum, total);
    if (tid < 32) {
        // status: 2 flag bits (1 the tile's counts, 2 those up to it),
        // 31 bits of merges, 31 of survivors; 32 tiles per look back
        constexpr unsigned long long kCounts = (1ull << 62) - 1ull;
        const unsigned long long own =
            (static_cast<unsigned long long>(total >> 16) << 31) | (total & 0xFFFFu);
        volatile unsigned long long* s = status;
        unsigned long long sum = 0;
        if (tile > 0) {
            if (tid == 0) s[tile] = (1ull << 62) | own;
            uint32_t spins = 0;
            for (int64_t k = int64_t(tile) - 1;;) {
                const int64_t at = k - tid;
                const unsigned long long w = at >= 0 ? s[at] : 2ull << 62;
                const uint32_t missing = __ballot_sync(0xFFFFFFFFu, (w >> 62) == 0ull);
                const uint32_t prefixes = __ballot_sync(0xFFFFFFFFu, (w >> 62) == 2ull);
                // tiles up to the nearest prefix, before the first missing one
                const int upTo = prefixes ? __ffs(int(prefixes)) : 32;
                const int usable = missing ? min(upTo, __ffs(int(missing)) - 1) : upTo;
                unsigned long long v = tid < usable ? w & kCounts : 0ull;
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
                sum += v;
                if (prefixes && usable == upTo) break;
                k -= usable;
                if (usable == 0 && ++spins > kSpinLimit) {
                    if (tid == 0) atomicExch(error, 1u);
                    break;
                }
            }
        }
        if (tid == 0) {
            s[tile] = (2ull << 62) | (sum + own);
            prefix = sum;
            if (b0 + kTile >= m) {
                const unsigned long long all = sum + own;
                next->m = uint32_t(all & 0x7FFFFFFFull);
                next->base = st.base + uint32_t(all >> 31);
                next->steps = st.steps + 1u;
            }
        }
    }
    __syncthreads();
    if (!mine || !(flags & 1u)) return;
    const uint32_t at = uint32_t(prefix & 0x7FFFFFFFull) + (before & 0xFFFFu);
    uint32_t c = ids[tid + 2 * kRadius];
    if (flags >> 16) {
        const uint32_t node = st.base + uint32_t(prefix >> 31) + (before >> 16);
        const int kj = j - b0 + 2 * kRadius;
        float box[6];
        make_node(out, node, c, ids[kj], sb + 6 * (tid + 2 * kRadius), sb + 6 * kj, box);
        c = in.n + node;
    }
    Cout[at] = c;
}

// The last steps in one block: at most kFinal clusters, their boxes in shared
// memory, until one is left.
__global__ void __launch_bounds__(kFinal) k_ploc_finish(const uint32_t* __restrict__ C0,
                                                        const uint32_t* __restrict__ C1, PlocIn in,
                                                        PlocOut out, PlocState* state) {
    __shared__ float sb[kFinal * 6];
    __shared__ uint32_t ids[kFinal];
    __shared__ int nn[kFinal];
    __shared__ uint32_t warpSum[kFinal / 32];
    const int i = int(threadIdx.x);
    int m = int(state->m);
    uint32_t base = state->base, steps = state->steps;
    const uint32_t* C = (steps & 1u) ? C1 : C0;
    if (i < m) {
        ids[i] = C[i];
        node_box(ids[i], in, out.inner, sb + 6 * i);
    }
    __syncthreads();
    // every step merges at least the pair with the least merged area
    for (int step = 0; step < kFinal && m > 1; step++) {
        if (i < m) nn[i] = nearest(sb + 6 * i, i, m);
        __syncthreads();
        uint32_t flags = 0, c = 0;
        int j = 0;
        float box[6];
        if (i < m) {
            j = nn[i];
            const bool mutual = nn[j] == i;
            flags = ((mutual && i < j) ? 0x10000u : 0u) | ((mutual && i > j) ? 0u : 1u);
            c = ids[i];
            for (int k = 0; k < 6; k++) box[k] = sb[6 * i + k];
        }
        uint32_t total;
        const uint32_t before = block_scan<kFinal / 32>(flags, warpSum, total);
        if (flags >> 16) {
            const uint32_t node = base + (before >> 16);
            float own[6];
            for (int k = 0; k < 6; k++) own[k] = box[k];
            make_node(out, node, c, ids[j], own, sb + 6 * j, box);
            c = in.n + node;
        }
        __syncthreads();
        if (flags & 1u) {
            const uint32_t at = before & 0xFFFFu;
            ids[at] = c;
            for (int k = 0; k < 6; k++) sb[6 * at + k] = box[k];
        }
        m = int(total & 0xFFFFu);
        base += total >> 16;
        steps++;
        __syncthreads();
    }
    if (i == 0) {
        *out.root = ids[0];
        state->m = uint32_t(m);
        state->base = base;
        state->steps = steps;
    }
}

__global__ void k_ploc_iota(uint32_t* C, uint32_t n, PlocState* state, uint32_t* error) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        C[i] = i;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *state = PlocState{n, 0u, 0u};
        *error = 0u;
    }
}

// Sum of the inner boxes' half surface areas (the SAH's node term) in
// double; blocks reduce in shared memory and add their sums atomically.
__global__ void __launch_bounds__(256) k_area_sum(const float* __restrict__ inner, uint32_t count,
                                                  double* out) {
    __shared__ double red[256];
    double a = 0.0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count;
         i += gridDim.x * blockDim.x) {
        const float* b = inner + 6 * size_t(i);
        const double dx = double(b[3]) - b[0], dy = double(b[4]) - b[1], dz = double(b[5]) - b[2];
        a += dx * dy + dy * dz + dz * dx;
    }
    red[threadIdx.x] = a;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (int(threadIdx.x) < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(out, red[0]);
}

inline uint32_t grid_of(uint32_t n, uint32_t block) {
    const uint32_t b = (n + block - 1) / block;
    return std::max(1u, std::min(b, 148u * 16u));
}

}  // namespace

int inner_area_sum(const float* inner, uint32_t count, double* scratch8, double* out,
                   cudaStream_t st) {
    MRB_CUDA(cudaMemsetAsync(scratch8, 0, 8, st));
    if (count) k_area_sum<<<grid_of(count, 256), 256, 0, st>>>(inner, count, scratch8);
    MRB_CUDA(cudaGetLastError());
    MRB_CUDA(cudaMemcpyAsync(out, scratch8, 8, cudaMemcpyDeviceToHost, st));
    MRB_CUDA(cudaStreamSynchronize(st));
    return 0;
}

namespace {
size_t align256(size_t v) { return (v + 255) & ~size_t(255); }
size_t step_tiles(uint32_t m) { return (size_t(m) + kTile - 1) / kTile; }
constexpr size_t kStateBytes = kBatch * sizeof(PlocState) + sizeof(PlocProgress);
}  // namespace

PlocArrays ploc_arrays(uint32_t n) {
    // in size_t throughout: the boxes alone pass 4 GB from 178,956,972 leaves on
    const size_t inner = size_t(n) - 1;
    PlocArrays a{};
    auto take = [&](size_t bytes) {
        const size_t at = a.bytes;
        a.bytes += align256(bytes);
        return at;
    };
    a.left = take(inner * 4);
    a.right = take(inner * 4);
    a.inner = take(inner * 24);
    a.root = take(4);
    // C x2; the states; the tickets and the tile status of a batch
    a.scratch = take(2 * align256(size_t(n) * 4) + align256(kStateBytes) + align256(kBatch * 4) +
                     kBatch * step_tiles(n) * 8);
    return a;
}

int ploc_build(const PlocIn& in, const PlocOut& out, void* scratch, uint32_t* iterations,
               cudaStream_t st) {
    const uint32_t n = in.n;
    if (n < 2) {
        set_error("PLOC: needs at least two leaves");
        return MRB_E_ARG;
    }
    char* p = static_cast<char*>(scratch);
    uint32_t* C[2];
    for (auto& c : C) {
        c = reinterpret_cast<uint32_t*>(p);
        p += align256(size_t(n) * 4);
    }
    PlocState* state = reinterpret_cast<PlocState*>(p);
    PlocProgress* progress = reinterpret_cast<PlocProgress*>(state + kBatch);
    p += align256(kStateBytes);
    uint32_t* tickets = reinterpret_cast<uint32_t*>(p);
    p += align256(kBatch * 4);
    unsigned long long* status = reinterpret_cast<unsigned long long*>(p);
    k_ploc_iota<<<grid_of(n, 256), 256, 0, st>>>(C[0], n, state, &progress->gaveUp);
    MRB_CUDA(cudaGetLastError());
    PlocState h{n, 0u, 0u};
    // every step merges at least the pair with the globally least merged
    // area, so n - 1 steps bound the loop
    while (h.m > uint32_t(kFinal)) {
        const size_t tiles = step_tiles(h.m);
        MRB_CUDA(cudaMemsetAsync(tickets, 0, align256(kBatch * 4) + kBatch * tiles * 8, st));
        // an even number of steps: each batch starts from C[0]
        for (int k = 0; k < kBatch; k++)
            k_ploc_step<<<static_cast<uint32_t>(tiles), kStepBlock, 0, st>>>(
                C[k & 1], C[(k & 1) ^ 1], in, out, state + k, state + k + 1, tickets + k,
                &progress->gaveUp, status + k * tiles);
        MRB_CUDA(cudaGetLastError());
        const uint32_t before = h.m;
        PlocProgress now;
        MRB_CUDA(cudaMemcpyAsync(&now, progress, sizeof(now), cudaMemcpyDeviceToHost, st));
        MRB_CUDA(cudaMemcpyAsync(state, &progress->state, sizeof(PlocState),
                                 cudaMemcpyDeviceToDevice, st));
        MRB_CUDA(cudaStreamSynchronize(st));
        if (now.gaveUp) {
            set_error("PLOC: a look-back gave up");
            return MRB_E_DEVICE;
        }
        h = now.state;
        if (h.m >= before || h.m + h.base != n) {
            set_error("PLOC: %u clusters and %u inner nodes of %u leaves after %u steps", h.m,
                      h.base, n, h.steps);
            return MRB_E_DEVICE;
        }
    }
    k_ploc_finish<<<1, kFinal, 0, st>>>(C[0], C[1], in, out, state);
    MRB_CUDA(cudaGetLastError());
    MRB_CUDA(cudaMemcpyAsync(&h, state, sizeof(h), cudaMemcpyDeviceToHost, st));
    MRB_CUDA(cudaStreamSynchronize(st));
    if (h.m != 1 || h.base != n - 1) {
        set_error("PLOC: %u clusters and %u inner nodes left after %u steps", h.m, h.base, h.steps);
        return MRB_E_DEVICE;
    }
    if (iterations) *iterations = h.steps;
    return 0;
}

}  // namespace mrb
