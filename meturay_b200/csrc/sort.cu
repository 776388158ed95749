// Onesweep LSD radix sort of (key, value) pairs, 8-bit digits.
//
// Semantics follow cub::DeviceRadixSort::SortPairs / SortPairsDescending as
// the reference calls them (ParallelRadixSort.cuh:60-100, RayMemory.cu:187-228,
// LinearBVH.hpp:489-492): stable, on bits [beginBit, endBit), ascending or
// descending.  Structure (Adinets & Merrill, "Onesweep", 2022):
//   1. one read of the keys builds the digit histograms of every pass;
//   2. per pass, one kernel: each CTA takes tiles by atomic ticket, ranks
//      their keys with warp-level match multisplit, resolves its global digit
//      offsets (the scanned histogram and a decoupled look-back), reorders the
//      tile through shared memory and writes coalesced runs.
// A wavefront's partition by material is the same two kernels reading HitKeys:
// the dense keys are formed on the way in, the portion table comes from the
// histogram, an odd number of passes lands without a copy, and the sorted keys
// are not written where only the order is wanted.  Per depth that is a memset
// and one launch plus one per pass; it was three memsets and six launches plus
// one per pass (Cornell 128x128, 5 depths: 0.10 -> 0.06 ms a frame; closed
// Cornell 1920x1080 with 4 samples: 0.96 -> 0.53 ms).
// The element count may live on the device (rays whose count a previous
// kernel produced); tiles past the count exit at once, so the sort needs no
// host synchronisation and can be captured in a CUDA graph.
#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "sort.cuh"

namespace mrb {

namespace {

// What a partition by material key adds to a sort.
struct PartitionJob {
    uint32_t idBits;
    uint32_t* batchCount;            // 8, zero before the histogram kernel
    PortionTable table;
    unsigned long long* rayTotal;    // may be null
    uint32_t* nextCount;             // may be null
};

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 16;
constexpr int kTile = kThreads * kItems;  // 4096
// Up to kSmallCount elements the tiles are of 1,024, up to kMidCount of 2,048:
// the block's serial part (the ranking, item by item) is shorter and more SMs
// work, while the look-back has more tiles to walk.  Three passes of 32-bit pairs,
// then eight of 64-bit Morton codes, with these tiles and with kTile (us): 65,536
// pairs 43 and 65; 300,000 58 and 65, 117 and 133; 400,000 67 and 63, 134 and 134;
// 450,000 72 and 65, 134 and 134; 600,000 73 and 72, 150 and 149.
constexpr int kSmallItems = 4, kMidItems = 8;
constexpr uint32_t kSmallCount = 200u * kThreads * kSmallItems;
constexpr uint32_t kMidCount = 200u * kThreads * kMidItems;
__host__ __device__ __forceinline__ uint32_t tile_size(uint32_t n) {
    return uint32_t(kThreads) * (n <= kSmallCount ? kSmallItems : n <= kMidCount ? kMidItems : kItems);
}
__host__ __device__ __forceinline__ uint32_t tile_count(uint32_t n) {
    const uint32_t t = tile_size(n);
    return n / t + (n % t ? 1u : 0u);
}
// Most tiles of any count up to maxCount.
inline uint32_t max_tiles(uint32_t maxCount) {
    return std::max({tile_count(maxCount), tile_count(std::min(maxCount, kMidCount)),
                     tile_count(std::min(maxCount, kSmallCount))});
}
constexpr uint32_t kSpinLimit = 1u << 24;
constexpr int kLook = 8;  // predecessors read at once by the look-back

// Tile status word: a flag (count of the tile known / prefix known) over a
// value.  Up to kEpochLimit elements the flags are numbered through the
// passes (2 * pass + 1, 2 * pass + 2 in five bits), so that the words one
// pass leaves behind read as "not there yet" in the next and only the first
// pass needs them cleared, which the histogram kernel does for the tiles in
// use.  Above it the values need 30 bits, and a memset clears every pass.
constexpr uint32_t kEpochLimit = 1u << 27;
struct StatusFlags {
    uint32_t aggregate, prefix, valueMask;
};
inline StatusFlags status_flags(uint32_t maxCount, int pass) {
    if (maxCount <= kEpochLimit)
        return {(2u * uint32_t(pass) + 1u) << 27, (2u * uint32_t(pass) + 2u) << 27,
                (1u << 27) - 1u};
    return {1u << 30, 2u << 30, (1u << 30) - 1u};
}

template <class K>
__device__ __forceinline__ uint32_t digit_of(K k, int bit, uint32_t mask, bool desc) {
    uint32_t d = static_cast<uint32_t>(k >> bit) & mask;
    return desc ? (mask - d) : d;
}

// A key as it is read: itself, or (kDense) a HitKey as its dense partition
// key, batch over the material index in idBits.
template <bool kDense, class K>
__device__ __forceinline__ K read_key(K k, uint32_t idBits) {
    if constexpr (kDense) return ((k >> kIdBits) << idBits) | (k & ((1u << idBits) - 1u));
    return k;
}

// Whether the three batch bits of a dense key fall into two digits.
__device__ __forceinline__ bool batch_straddles(uint32_t idBits) { return (idBits & 7u) > 5u; }

// Histograms of every pass (hist[p * 256 + d], digit bits beginBit + 8p) and,
// in use for the first pass, the status words cleared (clearStatus).  With
// kDense block 0 starts the portion table, adds the ray count to rayTotal and
// clears nextCount, and batches whose bits fall into two digits are counted
// apart.
template <class K, bool kDense>
__global__ void __launch_bounds__(kThreads) k_histogram(const K* __restrict__ keys,
                                                        const uint32_t* __restrict__ dCount,
                                                        uint32_t hCount, int beginBit, int endBit,
                                                        int desc, uint32_t* __restrict__ hist,
                                                        uint32_t* __restrict__ status,
                                                        int clearStatus, PartitionJob P) {
    __shared__ uint32_t sh[8][256];
    __shared__ uint32_t shBatch[8];
    const int passes = (endBit - beginBit + 7) / 8;
    for (int i = threadIdx.x; i < passes * 256; i += kThreads) (&sh[0][0])[i] = 0;
    if (kDense && threadIdx.x < 8) shBatch[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t n = dCount ? *dCount : hCount;
    const uint32_t first = blockIdx.x * kThreads + threadIdx.x, stride = gridDim.x * kThreads;
    if (clearStatus) {
        const uint32_t words = tile_count(n) * 256u;
        for (uint32_t i = first; i < words; i += stride) status[i] = 0u;
    }
    if (kDense && blockIdx.x == 0 && threadIdx.x < 8) {
        P.table.offset[threadIdx.x] = 0;
        P.table.end[threadIdx.x] = 0;
        if (threadIdx.x == 0) {
            *P.table.nonNull = n;
            if (P.rayTotal) *P.rayTotal += n;
            if (P.nextCount) *P.nextCount = 0u;
        }
    }
    for (uint32_t i = first; i < n; i += stride) {
        const K raw = keys[i];
        const K k = read_key<kDense>(raw, P.idBits);
        for (int p = 0; p < passes; p++) {
            int bit = beginBit + 8 * p;
            int nb = min(8, endBit - bit);
            uint32_t mask = (1u << nb) - 1u;
            atomicAdd(&sh[p][digit_of(k, bit, mask, desc != 0)], 1u);
        }
        if (kDense && batch_straddles(P.idBits)) atomicAdd(&shBatch[(raw >> kIdBits) & 7u], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += kThreads) {
        uint32_t v = (&sh[0][0])[i];
        if (v) atomicAdd(hist + i, v);
    }
    if (kDense && threadIdx.x < 8 && shBatch[threadIdx.x])
        atomicAdd(P.batchCount + threadIdx.x, shBatch[threadIdx.x]);
}

template <class K>
struct SortSmem {
    K keys[kTile];
    uint32_t vals[kTile];
    uint32_t warpHist[kWarps][256];
    uint32_t digitStart[256];
    uint32_t globalBase[256];
    uint32_t warpSum[2][kWarps];
    uint32_t batch[8];
    uint32_t tile;
    uint32_t validCount;
};

// Exclusive sums over the block's 256 threads of two values at once.
__device__ __forceinline__ void block_exclusive2(uint32_t a, uint32_t b, uint32_t (*warpSum)[kWarps],
                                                 uint32_t& ea, uint32_t& eb) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t xa = a, xb = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t ya = __shfl_up_sync(0xFFFFFFFFu, xa, o);
        const uint32_t yb = __shfl_up_sync(0xFFFFFFFFu, xb, o);
        if (lane >= o) {
            xa += ya;
            xb += yb;
        }
    }
    if (lane == 31) {
        warpSum[0][warp] = xa;
        warpSum[1][warp] = xb;
    }
    __syncthreads();
    uint32_t ba = 0, bb = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++)
        if (w < warp) {
            ba += warpSum[0][w];
            bb += warpSum[1][w];
        }
    ea = ba + xa - a;
    eb = bb + xb - b;
}

// One pass.  Blocks take tiles by ticket until none is left; hist holds the
// pass's digit counts, scanned here.  kDense: keysIn are HitKeys.  keysOut
// may be null (the last pass of a caller that only wants the order).
// Two blocks per SM (128 registers), with the values of a tile in flight while
// the digits are looked up.  Four blocks of 64 registers (three with 8-byte keys) that
// read the values when they need them took longer above a million pairs, and above 4M
// longer than tiles without a ticket loop; three of 85 gain 3 to 8 % from 8M on and lose
// 6 to 15 % between.  Three passes of 32-bit pairs by two, three and four blocks
// (us): 1M 93, 93 and 112; 2M 145, 165 and 158; 4M 231, 237 and 266; 16M 796, 749 and 878;
// eight of 64-bit Morton codes: 1M 184 and (three) 217; 4M 485 and 603; 16M 1,656
// and 1,948.
constexpr int kSweepBlocks = 2;
// Lanes of vmask with this lane's digit.  A match takes a turn per distinct
// digit, a vote per bit eight turns always.  The 64-bit keys are Morton codes,
// whose low digits are random: 1M pairs, eight passes, 206 us with matches and 184
// with votes, 4M 572 and 488.  The 32-bit keys are mostly a wavefront's materials, few
// distinct ones: 4M pairs of 2 to 12 different keys, two passes, 98 to 102 us with
// matches and 110 with votes; of 40 113 and 111, of random ones 153 and 129.  Large
// sorts of 64-bit keys look for a single digit first, as the high ones of equal or
// neighbouring codes are (at three blocks per SM, 4M pairs of 40 different keys 594 us
// without, 490 so, of random ones 601 and 610); small ones lose 6 % by it.
template <class K, int kN>
__device__ __forceinline__ uint32_t same_digit(uint32_t vmask, uint32_t dig) {
    if constexpr (sizeof(K) == 4) return __match_any_sync(vmask, dig);
    if constexpr (kN == kItems) {
        int all;
        __match_all_sync(vmask, dig, &all);
        if (all) return vmask;
    }
    uint32_t peers = vmask;
#pragma unroll
    for (int b = 0; b < 8; b++) {
        const bool on = (dig >> b) & 1u;
        const uint32_t v = __ballot_sync(vmask, on);
        peers &= on ? v : ~v;
    }
    return peers;
}

template <class K, bool kDense, int kN>
__device__ __forceinline__ void sweep_tiles(
    SortSmem<K>& sm, const K* __restrict__ keysIn, K* __restrict__ keysOut,
    const uint32_t* __restrict__ valsIn, uint32_t* __restrict__ valsOut, uint32_t n,
    const uint32_t* __restrict__ hist, uint32_t* tileStatus, uint32_t* tileTicket, int bit,
    int nbits, int desc, const StatusFlags& flags, const PartitionJob& P, uint32_t* errorFlag) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t mask = (1u << nbits) - 1u;
    const uint32_t ltMask = (1u << lane) - 1u;
    const uint32_t tiles = tile_count(n);
    // more blocks than tiles would crowd the tiles on the SMs that start first
    // (at four blocks per SM, 480 blocks for 245 tiles of a million pairs: 128 us,
    // 99 us so)
    if (blockIdx.x >= tiles) return;
    for (;;) {
        if (tid == 0) sm.tile = atomicAdd(tileTicket, 1u);
        __syncthreads();
        const uint32_t tile = sm.tile;
        if (tile >= tiles) return;
        for (int i = tid; i < kWarps * 256; i += kThreads) (&sm.warpHist[0][0])[i] = 0;
        const uint32_t base = tile * uint32_t(kThreads * kN);
        if (kDense && tile == 0) {
            // portions of the descending order: a batch follows all higher ones
            if (tid < 8) sm.batch[tid] = batch_straddles(P.idBits) ? P.batchCount[tid] : 0u;
            __syncthreads();
            if (!batch_straddles(P.idBits)) {
                const int p = int(P.idBits >> 3), bits = min(8, int(P.idBits) + 3 - 8 * p);
                const uint32_t c = tid < (1 << bits) ? hist[p * 256 + tid] : 0u;
                const uint32_t digit = uint32_t((1 << bits) - 1 - tid);  // descending
                if (c) atomicAdd(&sm.batch[(digit >> (P.idBits & 7u)) & 7u], c);
                __syncthreads();
            }
            if (tid < 8) {
                uint32_t before = 0;
                for (int b = tid + 1; b < 8; b++) before += sm.batch[b];
                const uint32_t c = sm.batch[tid];
                if (c) {
                    P.table.offset[tid] = before;
                    P.table.end[tid] = before + c;
                }
                if (tid == int(kBatchNull)) *P.table.nonNull = n - c;
            }
        }
        __syncthreads();

        // ---- load: warp w owns 32 * kN elements, item-major ----
        K key[kN];
        uint32_t place[kN];  // digit << 16 | rank
        const uint32_t wbase = base + warp * (32 * kN);
#pragma unroll
        for (int i = 0; i < kN; i++) {
            uint32_t idx = wbase + i * 32 + lane;
            bool ok = idx < n;
            key[i] = ok ? read_key<kDense>(keysIn[idx], P.idBits) : K(0);
        }
        // ---- warp-level multisplit ranking (stable: item-major, lane order) ----
        uint32_t* wh = sm.warpHist[warp];
#pragma unroll
        for (int i = 0; i < kN; i++) {
            uint32_t idx = wbase + i * 32 + lane;
            bool ok = idx < n;
            uint32_t vmask = __ballot_sync(0xFFFFFFFFu, ok);
            if (ok) {
                const uint32_t dig = digit_of(key[i], bit, mask, desc != 0);
                const uint32_t peers = same_digit<K, kN>(vmask, dig);
                uint32_t prior = wh[dig];
                __syncwarp(vmask);
                if (lane == (__ffs(peers) - 1)) wh[dig] = prior + __popc(peers);
                place[i] = (dig << 16) | (prior + __popc(peers & ltMask));
            }
            __syncwarp();
        }
        __syncthreads();

        // the values: in flight during the look-back
        uint32_t val[kN];
#pragma unroll
        for (int i = 0; i < kN; i++) {
            const uint32_t idx = wbase + i * 32 + lane;
            val[i] = valsIn ? (idx < n ? valsIn[idx] : 0u) : idx;
        }
        // ---- per digit: warp prefix, tile count, look-back ----
        {
            const uint32_t d = tid;  // kThreads == 256 digits
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < kWarps; w++) {
                uint32_t c = sm.warpHist[w][d];
                sm.warpHist[w][d] = run;
                run += c;
            }
            const uint32_t total = run;
            volatile uint32_t* st = tileStatus;
            st[tile * 256 + d] = (tile == 0 ? flags.prefix : flags.aggregate) | total;
            // this tile's and the whole pass's exclusive digit counts
            uint32_t start, passBase;
            block_exclusive2(total, hist[d], sm.warpSum, start, passBase);
            sm.digitStart[d] = start;
            if (d == 255) sm.validCount = start + total;

            // decoupled look-back over earlier tiles for digit d, kLook words
            // per round trip: one at a time, the walk over the tiles that are
            // in flight together (all of a sort of a million pairs) took most
            // of a pass
            uint32_t excl = 0;
            if (tile > 0) {
                int32_t k = static_cast<int32_t>(tile) - 1;
                uint32_t spins = 0;
                bool done = false;
                while (!done) {
                    uint32_t w[kLook];
#pragma unroll
                    for (int j = 0; j < kLook; j++)
                        w[j] = k - j >= 0 ? st[(k - j) * 256 + int32_t(d)] : flags.prefix;
#pragma unroll
                    for (int j = 0; j < kLook; j++) {
                        const uint32_t flag = w[j] & ~flags.valueMask;
                        if (done || (flag != flags.aggregate && flag != flags.prefix)) break;
                        excl += w[j] & flags.valueMask;
                        done = flag == flags.prefix;
                        k--;
                    }
                    if (!done && ++spins > kSpinLimit) {
                        atomicExch(errorFlag, 1u);
                        break;
                    }
                }
                __threadfence();
                st[tile * 256 + d] = flags.prefix | (excl + total);
            }
            sm.globalBase[d] = passBase + excl;
        }
        __syncthreads();

        // ---- reorder the tile through shared memory ----
#pragma unroll
        for (int i = 0; i < kN; i++) {
            uint32_t idx = wbase + i * 32 + lane;
            if (idx < n) {
                const uint32_t dig = place[i] >> 16;
                uint32_t p = sm.digitStart[dig] + sm.warpHist[warp][dig] + (place[i] & 0xFFFFu);
                sm.keys[p] = key[i];
                sm.vals[p] = val[i];
            }
        }
        __syncthreads();
        const uint32_t cnt = sm.validCount;
        for (uint32_t j = tid; j < cnt; j += kThreads) {
            K k = sm.keys[j];
            uint32_t d = digit_of(k, bit, mask, desc != 0);
            uint32_t g = sm.globalBase[d] + (j - sm.digitStart[d]);
            if (keysOut) keysOut[g] = k;
            valsOut[g] = sm.vals[j];
        }
        __syncthreads();
    }
}

template <class K, bool kDense>
__global__ void __launch_bounds__(kThreads, kSweepBlocks) k_onesweep(
    const K* __restrict__ keysIn, K* __restrict__ keysOut, const uint32_t* __restrict__ valsIn,
    uint32_t* __restrict__ valsOut, const uint32_t* __restrict__ dCount, uint32_t hCount,
    const uint32_t* __restrict__ hist, uint32_t* tileStatus, uint32_t* tileTicket, int bit,
    int nbits, int desc, StatusFlags flags, PartitionJob P, uint32_t* errorFlag) {
    extern __shared__ __align__(16) unsigned char smemRaw[];
    SortSmem<K>& sm = *reinterpret_cast<SortSmem<K>*>(smemRaw);
    const uint32_t n = dCount ? *dCount : hCount;
    if (n <= kSmallCount)
        sweep_tiles<K, kDense, kSmallItems>(sm, keysIn, keysOut, valsIn, valsOut, n, hist,
                                            tileStatus, tileTicket, bit, nbits, desc, flags, P,
                                            errorFlag);
    else if (n <= kMidCount)
        sweep_tiles<K, kDense, kMidItems>(sm, keysIn, keysOut, valsIn, valsOut, n, hist,
                                          tileStatus, tileTicket, bit, nbits, desc, flags, P,
                                          errorFlag);
    else
        sweep_tiles<K, kDense, kItems>(sm, keysIn, keysOut, valsIn, valsOut, n, hist, tileStatus,
                                       tileTicket, bit, nbits, desc, flags, P, errorFlag);
}

template <class K>
__global__ void k_copy_back(const K* __restrict__ ks, K* __restrict__ kd,
                            const uint32_t* __restrict__ vs, uint32_t* __restrict__ vd,
                            const uint32_t* __restrict__ dCount, uint32_t hCount) {
    const uint32_t n = dCount ? *dCount : hCount;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        kd[i] = ks[i];
        vd[i] = vs[i];
    }
}

inline size_t align_up(size_t v) { return (v + 255) & ~size_t(255); }

// Head of the scratch, cleared by one memset per sort: eight 256-bin
// histograms, eight pass tickets, the give-up flag, eight batch counts.
constexpr size_t kHistBytes = size_t(8) * 256 * 4;
constexpr size_t kHeadBytes = kHistBytes + size_t(8 + 1 + 8) * 4;

// The attribute is set once per device, before any stream capture; the lock
// keeps two host threads' first sorts on a device from racing.
template <class K, bool kDense>
int configure() {
    constexpr int kMaxDevices = 64;
    static bool configured[kMaxDevices] = {};
    static std::mutex configuredMutex;
    int dev = 0;
    MRB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) {
        set_error("radix sort: device %d out of the supported range [0, %d)", dev, kMaxDevices);
        return -1;
    }
    std::lock_guard<std::mutex> lock(configuredMutex);
    if (!configured[dev]) {
        MRB_CUDA(cudaFuncSetAttribute(k_onesweep<K, kDense>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(sizeof(SortSmem<K>))));
        configured[dev] = true;
    }
    return 0;
}

// Sorts srcKeys (HitKeys with kDense; srcVals null: 0..n-1) into dstKeys (may
// be srcKeys) and dstVals (may be srcVals).  Without keysWanted the sorted
// keys are left unwritten; dstKeys is scratch then.
template <class K, bool kDense>
int sort_impl(const K* srcKeys, const uint32_t* srcVals, K* dstKeys, uint32_t* dstVals,
              const uint32_t* dCount, uint32_t maxCount, int beginBit, int endBit, bool desc,
              void* temp, size_t tempBytes, cudaStream_t stream, PartitionJob P, bool keysWanted) {
    if (tempBytes < radix_sort_temp_bytes(maxCount, sizeof(K), beginBit, endBit)) {
        set_error("radix sort: scratch of %zu bytes is below the %zu required", tempBytes,
                  radix_sort_temp_bytes(maxCount, sizeof(K), beginBit, endBit));
        return -1;
    }
    const int passes = (endBit - beginBit + 7) / 8;
    const uint32_t tiles = max_tiles(maxCount);
    unsigned char* p = static_cast<unsigned char*>(temp);
    uint32_t* hist = reinterpret_cast<uint32_t*>(p);
    uint32_t* tickets = hist + 8 * 256;
    uint32_t* err = tickets + 8;
    P.batchCount = err + 1;
    p += align_up(kHeadBytes);
    uint32_t* status = reinterpret_cast<uint32_t*>(p);
    p += align_up((size_t(tiles) + 1) * 256 * 4);
    K* keysAlt = reinterpret_cast<K*>(p);
    p += align_up(size_t(maxCount) * sizeof(K));
    uint32_t* valsAlt = reinterpret_cast<uint32_t*>(p);
    if (int r = configure<K, kDense>()) return r;
    const bool epochs = maxCount <= kEpochLimit;
    // An in-place sort with an odd number of passes ends in the scratch and
    // is copied back; every other one lands where it is wanted.
    const bool back = srcKeys == dstKeys && (passes & 1);
    MRB_CUDA(cudaMemsetAsync(hist, 0, kHeadBytes, stream));
    const uint32_t histGrid = std::min(148u * 4u, maxCount / kThreads + 1u);
    k_histogram<K, kDense><<<histGrid, kThreads, 0, stream>>>(
        srcKeys, dCount, maxCount, beginBit, endBit, desc ? 1 : 0, hist, status, epochs ? 1 : 0, P);
    // as many blocks as run at once; each takes tiles until they are used up,
    // so a small count on the device costs no blocks that only look for work
    const uint32_t grid = std::min(tiles, 148u * uint32_t(kSweepBlocks));
    const K* kin = srcKeys;
    const uint32_t* vin = srcVals;
    for (int pass = 0; pass < passes && maxCount > 0; pass++) {
        const int bit = beginBit + 8 * pass;
        const int nb = (endBit - bit) < 8 ? (endBit - bit) : 8;
        const bool alt = ((passes - 1 - pass) & 1) != (back ? 1 : 0);
        K* kout = alt ? keysAlt : dstKeys;
        K* kwrite = (pass + 1 < passes || keysWanted) ? kout : nullptr;
        uint32_t* vout = alt ? valsAlt : dstVals;
        if (!epochs) MRB_CUDA(cudaMemsetAsync(status, 0, size_t(tiles) * 256 * 4, stream));
        const StatusFlags flags = status_flags(maxCount, pass);
        if (kDense && pass == 0)
            k_onesweep<K, kDense><<<grid, kThreads, sizeof(SortSmem<K>), stream>>>(
                kin, kwrite, vin, vout, dCount, maxCount, hist, status, tickets, bit, nb,
                desc ? 1 : 0, flags, P, err);
        else
            k_onesweep<K, false><<<grid, kThreads, sizeof(SortSmem<K>), stream>>>(
                kin, kwrite, vin, vout, dCount, maxCount, hist + pass * 256, status, tickets + pass,
                bit, nb, desc ? 1 : 0, flags, P, err);
        kin = kout;
        vin = vout;
    }
    if (back)
        k_copy_back<K><<<148 * 4, 256, 0, stream>>>(keysAlt, dstKeys, valsAlt, dstVals, dCount,
                                                   maxCount);
    MRB_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace

size_t radix_sort_temp_bytes(uint32_t maxCount, int keyBytes, int beginBit, int endBit) {
    const int passes = (endBit - beginBit + 7) / 8;
    const size_t tiles = max_tiles(maxCount);
    size_t bytes = 0;
    bytes += align_up(kHeadBytes);                          // histograms, tickets, error flag
    bytes += align_up((tiles + 1) * 256 * 4);               // tile status
    bytes += align_up(size_t(maxCount) * keyBytes);         // key ping-pong
    bytes += align_up(size_t(maxCount) * 4);                // value ping-pong
    (void)passes;
    return bytes;
}

template <class K>
int radix_sort_pairs(K* keys, uint32_t* vals, const uint32_t* dCount, uint32_t maxCount,
                     int beginBit, int endBit, bool desc, void* temp, size_t tempBytes,
                     cudaStream_t stream, bool valsAreIota) {
    if (endBit <= beginBit || maxCount == 0) return 0;
    return sort_impl<K, false>(keys, valsAreIota ? nullptr : vals, keys, vals, dCount, maxCount,
                               beginBit, endBit, desc, temp, tempBytes, stream, PartitionJob{}, true);
}

int partition_rays(const uint32_t* hitKey, const uint32_t* dCount, uint32_t maxCount,
                   uint32_t idBits, uint32_t* sortedIds, uint32_t* sortedDense, bool keysWanted,
                   const PortionTable& table, void* temp, size_t tempBytes, cudaStream_t stream,
                   unsigned long long* rayTotal, uint32_t* nextCount) {
    PartitionJob P{};
    P.idBits = idBits;
    P.table = table;
    P.rayTotal = rayTotal;
    P.nextCount = nextCount;
    // one read of the HitKeys for the histograms and one in the first pass:
    // the dense keys are formed on the way in
    if (int r = configure<uint32_t, false>()) return r;
    return sort_impl<uint32_t, true>(hitKey, nullptr, sortedDense, sortedIds, dCount, maxCount, 0,
                                     3 + int(idBits), true, temp, tempBytes, stream, P, keysWanted);
}

uint32_t* radix_sort_error_flag(void* temp, uint32_t) {
    return reinterpret_cast<uint32_t*>(static_cast<unsigned char*>(temp) + kHistBytes) + 8;
}

template int radix_sort_pairs<uint64_t>(uint64_t*, uint32_t*, const uint32_t*, uint32_t, int, int,
                                        bool, void*, size_t, cudaStream_t, bool);
template int radix_sort_pairs<uint32_t>(uint32_t*, uint32_t*, const uint32_t*, uint32_t, int, int,
                                        bool, void*, size_t, cudaStream_t, bool);

}  // namespace mrb
