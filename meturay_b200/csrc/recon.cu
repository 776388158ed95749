// Reconstruction filters: splat camera samples onto the image.
//
// The reference (GPUReconFilter.h:59-260, GPUReconFilterKC.cuh:34-377)
// expands every sample to the pixels its filter reaches (one (pixel,
// sample) pair per pixel), radix-sorts the pairs by pixel and reduces each
// pixel's run with a block or warp reduction.  Here:
//   - the general entry point (any image coordinates) sorts a list with the
//     onesweep sort, its length staying on the device (no host round trip, so
//     the splat can sit inside a captured graph), and every pixel sums its
//     samples in ascending sample order.  With a radius below 0.75 the list
//     holds the pairs of pixel and sample (count, scan, write in sample order)
//     and a thread sums a pixel's run; with larger ones it holds a sample once
//     per tile of 8 x 8 pixels that its window touches, and a warp walks a
//     tile's samples for half of its pixels, or a block those of a tile on
//     which samples crowd;
//   - the tracer's own samples lie on the camera's stratified grid, so each
//     pixel finds its candidates by index arithmetic in a small
//     neighbourhood and sums them in the same ascending sample order: the
//     same bits as the general path, with no pairs, no sort and no atomics.
// Per pixel, ascending sample order is also the order of the reference's
// own CPU expectation (Test_TracerCUDA/T_ReconFilter.cu:96-140).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "../../include/mrb200.h"
#include "recon.cuh"
#include "scan.cuh"
#include "sort.cuh"

namespace mrb {

namespace {

inline size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

// Where a sample lands: modf of its image coordinates and the window of
// pixel offsets KCExpandSamplesToPixels walks (GPUReconFilterKC.cuh:44-91).
struct SamplePix {
    float fx, fy;        // integer parts (as floats)
    int32_t ix, iy;      // integer parts (as ints)
    int32_t x0, x1, y0, y1;  // offset window [x0, x1) x [y0, y1)
    bool ok;
};

__host__ __device__ inline SamplePix sample_pix(float cx, float cy, uint32_t wh) {
    SamplePix s{};
    // coordinates beyond +-1e9 (or NaN) reach no pixel of any image this
    // library accepts; they are dropped instead of overflowing the ints
    s.ok = fabsf(cx) < 1.0e9f && fabsf(cy) < 1.0e9f;
    if (!s.ok) return s;
    s.fx = truncf(cx);
    s.fy = truncf(cy);
    const float relX = cx - s.fx, relY = cy - s.fy;
    s.ix = static_cast<int32_t>(s.fx);
    s.iy = static_cast<int32_t>(s.fy);
    const int32_t range = static_cast<int32_t>(wh);
    const int32_t lo = -(range - 1) / 2, hi = (range + 2) / 2;
    s.x0 = lo; s.x1 = hi; s.y0 = lo; s.y1 = hi;
    // even windows lean towards the half of the pixel the sample is in
    if (range % 2 == 0) {
        if (relX < 0.5f) { s.x0 -= 1; s.x1 -= 1; }
        if (relY < 0.5f) { s.y0 -= 1; s.y1 -= 1; }
    }
    return s;
}

// The distance test for offset (x, y) (radius 0: the sample's own pixel).
__host__ __device__ inline bool sample_reaches(const SamplePix& s, float cx, float cy, int32_t x,
                                               int32_t y, uint32_t wh, float r2) {
    if (wh == 1u) return true;
    const float pcx = (s.fx + static_cast<float>(x)) + 0.5f;
    const float pcy = (s.fy + static_cast<float>(y)) + 0.5f;
    const float dx = cx - pcx, dy = cy - pcy;
    return (dx * dx + dy * dy) <= r2;
}

__host__ __device__ inline bool in_segment(const ImageSeg& g, int32_t px, int32_t py) {
    return px >= 0 && px < g.resW && py >= 0 && py < g.resH && px >= g.offX &&
           px < g.offX + g.w && py >= g.offY && py < g.offY + g.h;
}

// ---------------------------------------------------------------------------
// Small radii: pairs of pixel and sample
// ---------------------------------------------------------------------------
// Pass 1: number of (pixel, sample) pairs per sample.
__global__ void __launch_bounds__(256) k_expand_count(const float2* __restrict__ coords, uint32_t n,
                                                      ReconFilterDev f, ImageSeg g,
                                                      uint32_t* __restrict__ count) {
    const float r2 = f.radius * f.radius;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float2 c = coords[i];
        const SamplePix s = sample_pix(c.x, c.y, f.wh);
        uint32_t k = 0;
        if (s.ok) {
            for (int32_t y = s.y0; y < s.y1; y++)
                for (int32_t x = s.x0; x < s.x1; x++)
                    if (sample_reaches(s, c.x, c.y, x, y, f.wh, r2) &&
                        in_segment(g, s.ix + x, s.iy + y))
                        k++;
        }
        count[i] = k;
    }
}

// Pass 2: the pairs themselves, at the sample's scanned offset, in the
// reference's (y, x) window order.  Keys are segment-local pixel indices.
__global__ void __launch_bounds__(256) k_expand_write(const float2* __restrict__ coords, uint32_t n,
                                                      ReconFilterDev f, ImageSeg g,
                                                      const uint32_t* __restrict__ offset,
                                                      uint32_t* __restrict__ keys,
                                                      uint32_t* __restrict__ vals) {
    const float r2 = f.radius * f.radius;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float2 c = coords[i];
        const SamplePix s = sample_pix(c.x, c.y, f.wh);
        if (!s.ok) continue;
        uint32_t o = offset[i];
        for (int32_t y = s.y0; y < s.y1; y++)
            for (int32_t x = s.x0; x < s.x1; x++) {
                const int32_t px = s.ix + x, py = s.iy + y;
                if (!sample_reaches(s, c.x, c.y, x, y, f.wh, r2) || !in_segment(g, px, py))
                    continue;
                keys[o] = static_cast<uint32_t>((py - g.offY) * g.w + (px - g.offX));
                vals[o] = i;
                o++;
            }
    }
}

// Run boundaries of the sorted keys: [begin[p], end[p]) for every pixel
// that received a pair (both stay 0 for the others).
__global__ void __launch_bounds__(256) k_pixel_bounds(const uint32_t* __restrict__ keys,
                                                      const uint32_t* __restrict__ dCount,
                                                      uint32_t* __restrict__ begin,
                                                      uint32_t* __restrict__ end) {
    const uint32_t n = *dCount;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t k = keys[i];
        if (i == 0 || keys[i - 1] != k) begin[k] = i;
        if (i + 1 == n || keys[i + 1] != k) end[k] = i + 1;
    }
}

// KCFilterToImgBlock / KCFilterToImgWarp (GPUReconFilterKC.cuh:146-377):
// one thread per segment pixel sums its run in sample order, then adds the
// sums into the image and the weight into the sample counts.
template <int C>
__global__ void __launch_bounds__(256) k_filter_pixels(
    const uint32_t* __restrict__ begin, const uint32_t* __restrict__ end,
    const uint32_t* __restrict__ vals, const float* __restrict__ values,
    const float2* __restrict__ coords, ReconFilterDev f, ImageSeg g, float multiplier,
    float* __restrict__ pixels, float* __restrict__ counts) {
    const uint32_t total = static_cast<uint32_t>(g.w) * static_cast<uint32_t>(g.h);
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < total;
         q += gridDim.x * blockDim.x) {
        const uint32_t b = begin[q], e = end[q];
        if (b == e) continue;
        const int32_t gx = static_cast<int32_t>(q % static_cast<uint32_t>(g.w)) + g.offX;
        const int32_t gy = static_cast<int32_t>(q / static_cast<uint32_t>(g.w)) + g.offY;
        const float pcx = static_cast<float>(gx) + 0.5f, pcy = static_cast<float>(gy) + 0.5f;
        float acc[C];
        for (int k = 0; k < C; k++) acc[k] = 0.0f;
        float wsum = 0.0f;
        for (uint32_t i = b; i < e; i++) {
            const uint32_t sid = vals[i];
            const float2 c = coords[sid];
            const float w = recon_weight(f, pcx, pcy, c.x, c.y) * multiplier;
            wsum += w;
            if constexpr (C == 4) {
                const float4 v = reinterpret_cast<const float4*>(values)[sid];
                acc[0] += w * v.x;
                acc[1] += w * v.y;
                acc[2] += w * v.z;
                acc[3] += w * v.w;
            } else {
                acc[0] += w * values[sid];
            }
        }
        if constexpr (C == 4) {
            float4* p4 = reinterpret_cast<float4*>(pixels) + q;
            float4 p = *p4;
            p.x += acc[0];
            p.y += acc[1];
            p.z += acc[2];
            p.w += acc[3];
            *p4 = p;
        } else {
            pixels[q] += acc[0];
        }
        counts[q] += wsum;
    }
}

// ---------------------------------------------------------------------------
// Larger radii: tiles of pixels
// ---------------------------------------------------------------------------
// Tiles of the segment that a sample's window touches.
constexpr int32_t kTileSide = 8;
struct TileSpan {
    int32_t x0, x1, y0, y1;  // [x0, x1) x [y0, y1)
};
__device__ __forceinline__ TileSpan tile_span(const SamplePix& s, const ImageSeg& g) {
    if (!s.ok) return {0, 0, 0, 0};
    // the window, relative to the segment and clipped to its pixels in the image
    const int64_t x = int64_t(s.ix) - g.offX, y = int64_t(s.iy) - g.offY;
    const int64_t ax = max(x + s.x0, int64_t(max(0, -g.offX)));
    const int64_t bx = min(x + s.x1, int64_t(min(g.w, g.resW - g.offX)));
    const int64_t ay = max(y + s.y0, int64_t(max(0, -g.offY)));
    const int64_t by = min(y + s.y1, int64_t(min(g.h, g.resH - g.offY)));
    if (ax >= bx || ay >= by) return {0, 0, 0, 0};
    return {int32_t(ax) / kTileSide, int32_t(bx - 1) / kTileSide + 1,
            int32_t(ay) / kTileSide, int32_t(by - 1) / kTileSide + 1};
}

// Pass 1: number of tiles per sample.  Also clears the tiles' runs and the
// lengths of the lists behind them.
__global__ void __launch_bounds__(256) k_tile_count(const float2* __restrict__ coords, uint32_t n,
                                                    uint32_t wh, ImageSeg g,
                                                    uint32_t* __restrict__ count,
                                                    uint32_t* __restrict__ clear, uint32_t words) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x)
        clear[i] = 0u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float2 c = coords[i];
        const TileSpan t = tile_span(sample_pix(c.x, c.y, wh), g);
        count[i] = uint32_t(t.x1 - t.x0) * uint32_t(t.y1 - t.y0);
    }
}

// Pass 2: the (tile, sample) entries, at the sample's scanned offset.
__global__ void __launch_bounds__(256) k_tile_write(const float2* __restrict__ coords, uint32_t n,
                                                    uint32_t wh, ImageSeg g, int32_t tilesX,
                                                    const uint32_t* __restrict__ offset,
                                                    uint32_t* __restrict__ keys,
                                                    uint32_t* __restrict__ vals) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float2 c = coords[i];
        const TileSpan t = tile_span(sample_pix(c.x, c.y, wh), g);
        uint32_t o = offset[i];
        for (int32_t y = t.y0; y < t.y1; y++)
            for (int32_t x = t.x0; x < t.x1; x++) {
                keys[o] = static_cast<uint32_t>(y * tilesX + x);
                vals[o++] = i;
            }
    }
}

// A tile with more samples than this is taken by a block (crowded_tile) instead
// of two warps.  Up to kFew tiles with over kCrowd samples lie on the SMs all at
// once, and the longest walk of a warp is what the splat waits for; with more of
// them the warps keep the SMs busy and a block gains only on long runs.  Radius 1,
// whole splat, warps alone and blocks from 128 and 1,024 samples on (us): 20,000
// samples in 10 x 10 pixels 651 and 164, in 100 x 100 (200 a tile) 68 and 60; but
// 1080p (32,400 tiles) with 150 a tile 522 and 585 with blocks from 128 on.  640 x 360
// (3,600 tiles) with 800 a tile 355 and 332 with blocks from 512 on, 1080p with 800
// 2,450 and 2,600; 640 x 360 with 1,600 622 and 544.
constexpr uint32_t kCrowd = 128, kDense = 1024, kFew = 1024;
__device__ __forceinline__ uint32_t crowd_limit(uint32_t crowded) {
    return crowded <= kFew ? kCrowd : kDense;
}

// Run boundaries of the sorted keys: [begin, end) for every tile that has
// samples (both stay 0 for the others), and the lists of the tiles with long
// runs: the sample kCrowd (kDense) places into a run enters its tile.  Past kFew
// entries the first list is not used, so it need not be complete, and its
// counter, which all of them would wait for, is left alone.
__global__ void __launch_bounds__(256) k_tile_bounds(const uint32_t* __restrict__ keys,
                                                     const uint32_t* __restrict__ dCount,
                                                     uint2* __restrict__ tiles, CrowdLists lists) {
    const uint32_t n = *dCount;
    auto enters = [&](uint32_t i, uint32_t k, uint32_t limit) {
        return i >= limit && keys[i - limit] == k && (i == limit || keys[i - limit - 1] != k);
    };
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t k = keys[i];
        if (i == 0 || keys[i - 1] != k) tiles[k].x = i;
        if (i + 1 == n || keys[i + 1] != k) tiles[k].y = i + 1;
        if (enters(i, k, kCrowd) && __ldcg(lists.counts) <= kFew)
            lists.crowd[atomicAdd(lists.counts, 1u)] = k;
        if (enters(i, k, kDense)) lists.dense[atomicAdd(lists.counts + 1, 1u)] = k;
    }
}

// A pixel's sums into the image.
template <int C>
__device__ __forceinline__ void add_to_pixel(const ImageSeg& g, int32_t qx, int32_t qy,
                                             const float* acc, float wsum,
                                             float* __restrict__ pixels,
                                             float* __restrict__ counts) {
    const size_t q = size_t(qy) * size_t(g.w) + size_t(qx);
    if constexpr (C == 4) {
        float4* p4 = reinterpret_cast<float4*>(pixels) + q;
        float4 p = *p4;
        p.x += acc[0];
        p.y += acc[1];
        p.z += acc[2];
        p.w += acc[3];
        *p4 = p;
    } else {
        pixels[q] += acc[0];
    }
    counts[q] += wsum;
}

constexpr int kSplatBlock = 256;
constexpr int kSplatWarps = kSplatBlock / 32;
constexpr int kTilePixels = kTileSide * kTileSide;

// A block's shared memory: samples (coordinates with the window's first pixel,
// values) of each warp's round, or of a crowded tile's round with the votes.
template <int C>
struct SplatSmem {
    typename std::conditional<C == 4, float4, float>::type value[kSplatBlock];
    union {
        float4 place[kSplatBlock];
        struct {
            float2 at[kSplatBlock];
            uint32_t reach[kTilePixels][kSplatWarps + 1];       // a bit per sample of each warp
            uint8_t list[kTilePixels][kSplatBlock + 4];         // a pixel's samples, ascending
        } crowd;
    };
};

// A tile with a long run, by a block: 256 samples a round, one per thread.  Each
// warp votes, pixel by pixel, which of its 32 samples reach the pixel; four threads
// per pixel make the votes a list and sum its samples in order, one channel each.
// A warp of k_filter_tiles goes through a run 32 samples at a time and takes a step
// for every sample that touches any of its 32 pixels; here eight warps share the
// reads and tests, and a pixel's threads step over what does not reach it.  Bound
// by the rounds' chain: some 1,200 cycles of votes, 900 of lists and 600 of sums.
// Radius 1, whole splat, by pairs, by warps and so (us): 20,000 samples in one pixel
// 2,505, 1,112 and 1,024; in 10 x 10 222, 651 and 164; in 30 x 30 100, 153 and 74;
// 200,000 in 30 x 30 322, 1,024 and 239; 65,536 on 32 x 32 132, 324 and 99.  In 10 x 10 a
// thread per pixel for all four channels took 192 and not 148 (both in a launch of
// their own), the votes bit by bit instead of from a list 184 and not 163.
template <int C>
__device__ __forceinline__ void crowded_tile(SplatSmem<C>& S, uint2 range, int32_t ox, int32_t oy,
                                             const uint32_t* __restrict__ vals,
                                             const float* __restrict__ values,
                                             const float2* __restrict__ coords,
                                             const ReconFilterDev& f, const ImageSeg& g,
                                             float multiplier, float* __restrict__ pixels,
                                             float* __restrict__ counts) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    // four threads per pixel, one channel each
    const uint32_t p = tid >> 2, part = tid & 3u;
    const float r2 = f.radius * f.radius;
    const int32_t qx = ox + int32_t(p & 7u), qy = oy + int32_t(p >> 3);
    const float pcx = static_cast<float>(qx + g.offX) + 0.5f;
    const float pcy = static_cast<float>(qy + g.offY) + 0.5f;
    float acc = 0.0f, wsum = 0.0f;
    bool hit = false;
    // ids are read two rounds ahead, coordinates and values one
    auto id_at = [&](uint32_t i) { return i < range.y ? __ldg(vals + i) : 0u; };
    float2 c = make_float2(0.0f, 0.0f);
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto sample_at = [&](uint32_t i, uint32_t id) {
        if (i >= range.y) return;
        c = __ldg(coords + id);
        if constexpr (C == 4) v = __ldg(reinterpret_cast<const float4*>(values) + id);
        else v.x = __ldg(values + id);
    };
    sample_at(range.x + tid, id_at(range.x + tid));
    uint32_t id1 = id_at(range.x + kSplatBlock + tid);
    for (uint32_t base = range.x; base < range.y; base += kSplatBlock) {
        // squared distances to the tile's columns, infinite beyond the window
        float dx2[kTileSide];
        int32_t y0 = 0, y1 = 0;
#pragma unroll
        for (int k = 0; k < kTileSide; k++) dx2[k] = INFINITY;
        if (base + tid < range.y) {
            const SamplePix s = sample_pix(c.x, c.y, f.wh);
            const int32_t x0 = s.ix + s.x0 - (ox + g.offX), x1 = x0 + (s.x1 - s.x0);
            y0 = s.iy + s.y0 - (oy + g.offY);
            y1 = y0 + (s.y1 - s.y0);
#pragma unroll
            for (int k = 0; k < kTileSide; k++) {
                const float dx = c.x - (static_cast<float>(ox + g.offX + k) + 0.5f);
                if (k >= x0 && k < x1) dx2[k] = dx * dx;
            }
        }
#pragma unroll
        for (int y = 0; y < kTileSide; y++) {
            const float dy = c.y - (static_cast<float>(oy + g.offY + y) + 0.5f);
            const float dy2 = (y >= y0 && y < y1) ? dy * dy : INFINITY;
#pragma unroll
            for (int x = 0; x < kTileSide; x++) {
                const uint32_t reach = __ballot_sync(kAll, dx2[x] + dy2 <= r2);
                if (lane == 0) S.crowd.reach[y * kTileSide + x][warp] = reach;
            }
        }
        S.crowd.at[tid] = c;
        if constexpr (C == 4) S.value[tid] = v;
        else S.value[tid] = v.x;
        const uint32_t i1 = base + kSplatBlock + tid;
        sample_at(i1, id1);
        id1 = id_at(i1 + kSplatBlock);
        __syncthreads();
        // the pixel's votes as a list, two words by each of its threads
        uint32_t w0 = S.crowd.reach[p][2u * part], w1 = S.crowd.reach[p][2u * part + 1u];
        const uint32_t own = uint32_t(__popc(w0) + __popc(w1));
        uint32_t upTo = own;
#pragma unroll
        for (uint32_t o = 1; o < 4u; o <<= 1) {
            const uint32_t below = __shfl_up_sync(kAll, upTo, o, 4);
            if (part >= o) upTo += below;
        }
        const uint32_t count = __shfl_sync(kAll, upTo, 3, 4);
        hit |= count > 0u;
        uint8_t* out = S.crowd.list[p] + (upTo - own);
        for (; w0; w0 &= w0 - 1u) *out++ = uint8_t(64u * part + uint32_t(__ffs(int(w0)) - 1));
        for (; w1; w1 &= w1 - 1u)
            *out++ = uint8_t(64u * part + 32u + uint32_t(__ffs(int(w1)) - 1));
        __syncwarp();
        // its samples in order, four at a time but for the sums
        for (uint32_t k = 0; k < count; k += 4u) {
            const uint32_t four = *reinterpret_cast<const uint32_t*>(&S.crowd.list[p][k]);
            float weight[4], val[4];
#pragma unroll
            for (uint32_t j = 0; j < 4u; j++) {
                const uint32_t h = (four >> (8u * j)) & 0xFFu;
                const float2 at = S.crowd.at[h];
                weight[j] = recon_weight(f, pcx, pcy, at.x, at.y) * multiplier;
                if constexpr (C == 4)
                    val[j] = reinterpret_cast<const float*>(&S.value[h])[part];
                else
                    val[j] = S.value[h];
            }
#pragma unroll
            for (uint32_t j = 0; j < 4u; j++)
                if (k + j < count) {
                    wsum += weight[j];
                    acc += weight[j] * val[j];
                }
        }
        __syncthreads();
    }
    if (hit && qx < g.w && qy < g.h && in_segment(g, qx + g.offX, qy + g.offY)) {
        const size_t q = size_t(qy) * size_t(g.w) + size_t(qx);
        if (C == 4 || part == 0u) pixels[q * C + (C == 4 ? part : 0u)] += acc;
        if (part == 0u) counts[q] += wsum;
    }
}

// KCFilterToImgBlock / KCFilterToImgWarp (GPUReconFilterKC.cuh:146-377): a warp
// per 8 x 4 pixels.  It reads its tile's samples 32 at a time, one per lane, and
// keeps those whose window touches its pixels; then it takes these in order from
// shared memory, every lane holding the sample against its own pixel.  So a pixel
// sums its samples in ascending order, whatever their number.  Bound by the reads
// of ids and coordinates, hence the two rounds ahead.  1M samples, 1080p, tent of
// radius 1, whole splat: 340 us by pairs, 228 us so.  Tiles of 16 x 16 (1.3 entries
// per sample instead of 1.6) were 4 % slower.
// The last crowdBlocks blocks take the crowded tiles.  In a launch of their own
// these cost 4 us a call and start only after the others; six blocks per SM (40
// registers) because at five the reads of sparse images are slower (100,000 samples
// on 1080p 90 and 94 us), although crowds gain 8 %.
template <int C, int kType>
__global__ void __launch_bounds__(kSplatBlock, 6) k_filter_tiles(
    const uint2* __restrict__ tiles, CrowdLists lists, uint32_t crowdBlocks, int32_t tilesX,
    const uint32_t* __restrict__ vals, const float* __restrict__ values,
    const float2* __restrict__ coords, ReconFilterDev f, ImageSeg g, float multiplier,
    float* __restrict__ pixels, float* __restrict__ counts) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    __shared__ __align__(16) SplatSmem<C> S;
    f.type = kType;
    if (blockIdx.x >= gridDim.x - crowdBlocks) {
        const bool few = lists.counts[0] <= kFew;
        const uint32_t count = lists.counts[few ? 0 : 1];
        for (uint32_t i = blockIdx.x - (gridDim.x - crowdBlocks); i < count; i += crowdBlocks) {
            const int32_t t = int32_t((few ? lists.crowd : lists.dense)[i]);
            crowded_tile<C>(S, tiles[t], (t % tilesX) * kTileSide, (t / tilesX) * kTileSide, vals,
                            values, coords, f, g, multiplier, pixels, counts);
        }
        return;
    }
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // the warp's and the lane's pixel, in the segment
    const int32_t blocksX = (tilesX + 1) / 2, block = int32_t(blockIdx.x);
    const int32_t wx = (block % blocksX) * 16 + int32_t(warp & 1u) * 8;
    const int32_t wy = (block / blocksX) * 16 + int32_t(warp >> 1) * 4;
    if (wx >= g.w || wy >= g.h) return;
    const uint2 range = tiles[(wy / kTileSide) * tilesX + wx / kTileSide];
    if (range.x == range.y || range.y - range.x > crowd_limit(lists.counts[0])) return;
    const uint32_t mine = 32u * warp;  // this warp's place in S
    const int32_t qx = wx + int32_t(lane & 7u), qy = wy + int32_t(lane >> 3);
    const int32_t gx = qx + g.offX, gy = qy + g.offY;
    const float pcx = static_cast<float>(gx) + 0.5f, pcy = static_cast<float>(gy) + 0.5f;
    const float r2 = f.radius * f.radius;
    const SamplePix any = sample_pix(0.5f, 0.5f, f.wh);
    const int32_t extent = any.x1 - any.x0;  // of a window, per axis
    float acc[C];
    for (int k = 0; k < C; k++) acc[k] = 0.0f;
    float wsum = 0.0f;
    bool hit = false;
    // ids are read two rounds ahead and coordinates one
    auto id_at = [&](uint32_t i) { return i < range.y ? __ldg(vals + i) : 0u; };
    auto coord_at = [&](uint32_t i, uint32_t id) {
        return i < range.y ? __ldg(coords + id) : make_float2(0.0f, 0.0f);
    };
    uint32_t id = id_at(range.x + lane), id1 = id_at(range.x + 32u + lane);
    float2 c = coord_at(range.x + lane, id);
    for (uint32_t base = range.x; base < range.y; base += 32u) {
        const uint32_t i = base + lane;
        const uint32_t id2 = id_at(i + 64u);
        const float2 c1 = coord_at(i + 32u, id1);
        int32_t lowX = 0, lowY = 0;
        bool touches = false;
        if (i < range.y) {
            const SamplePix s = sample_pix(c.x, c.y, f.wh);
            lowX = s.ix + s.x0;
            lowY = s.iy + s.y0;
            const int32_t dx = wx + g.offX - lowX, dy = wy + g.offY - lowY;
            touches = dx > -8 && dx < extent && dy > -4 && dy < extent;
        }
        const uint32_t some = __ballot_sync(kAll, touches);
        if (touches) {
            const uint32_t at = uint32_t(__popc(some & ((1u << lane) - 1u)));
            S.place[mine + at] = make_float4(c.x, c.y, __int_as_float(lowX), __int_as_float(lowY));
            if constexpr (C == 4)
                S.value[mine + at] = reinterpret_cast<const float4*>(values)[id];
            else
                S.value[mine + at] = values[id];
        }
        __syncwarp();
        const int count = __popc(some);
#pragma unroll 4
        for (int h = 0; h < count; h++) {
            const float4 s = S.place[mine + uint32_t(h)];
            const float* v = reinterpret_cast<const float*>(&S.value[mine + uint32_t(h)]);
            const float dx = s.x - pcx, dy = s.y - pcy;
            const bool reaches =
                (uint32_t(gx - __float_as_int(s.z)) < uint32_t(extent)) &
                (uint32_t(gy - __float_as_int(s.w)) < uint32_t(extent)) &
                ((dx * dx + dy * dy) <= r2);
            float w = 0.0f;
            if (kType <= kReconTent || reaches) w = recon_weight(f, pcx, pcy, s.x, s.y) * multiplier;
            wsum = reaches ? wsum + w : wsum;
            for (int k = 0; k < C; k++)
                acc[k] = reaches ? acc[k] + w * v[k] : acc[k];
            hit |= reaches;
        }
        __syncwarp();
        id = id1;
        id1 = id2;
        c = c1;
    }
    // a tile may stick out of the segment and a segment out of the image
    if (hit && qx < g.w && qy < g.h && in_segment(g, gx, gy))
        add_to_pixel<C>(g, qx, qy, acc, wsum, pixels, counts);
}

// Tracer splat over the camera's sample grid.  Sample sid = sy * (W*sp) + sx
// belongs to pixel (sx / sp, sy / sp) and its image coordinates lie within
// one pixel of it, so pixel p can only receive samples of the pixels q with
// q in [p - hi, p - loMin + 1] per axis (the window offsets being
// [loMin, hi)).  Rows then columns ascending = ascending sample order.
__global__ void __launch_bounds__(256) k_filter_grid(const float4* __restrict__ samples,
                                                     const float2* __restrict__ coords,
                                                     uint32_t width, uint32_t height, uint32_t sp,
                                                     ReconFilterDev f, float multiplier,
                                                     float4* __restrict__ image) {
    const int32_t range = static_cast<int32_t>(f.wh);
    const int32_t hi = (range + 2) / 2;
    const int32_t loMin = -(range - 1) / 2 - ((range % 2 == 0) ? 1 : 0);
    const float r2 = f.radius * f.radius;
    const int32_t S = static_cast<int32_t>(sp);
    const int32_t SW = static_cast<int32_t>(width) * S, SH = static_cast<int32_t>(height) * S;
    const uint32_t total = width * height;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < total;
         p += gridDim.x * blockDim.x) {
        const int32_t px = static_cast<int32_t>(p % width), py = static_cast<int32_t>(p / width);
        const float pcx = static_cast<float>(px) + 0.5f, pcy = static_cast<float>(py) + 0.5f;
        const int32_t sy0 = max(0, (py - hi) * S), sy1 = min(SH, (py - loMin + 2) * S);
        const int32_t sx0 = max(0, (px - hi) * S), sx1 = min(SW, (px - loMin + 2) * S);
        float ax = 0.0f, ay = 0.0f, az = 0.0f, wsum = 0.0f;
        for (int32_t sy = sy0; sy < sy1; sy++)
            for (int32_t sx = sx0; sx < sx1; sx++) {
                const uint32_t sid = static_cast<uint32_t>(sy) * static_cast<uint32_t>(SW) +
                                     static_cast<uint32_t>(sx);
                const float2 c = coords[sid];
                const SamplePix s = sample_pix(c.x, c.y, f.wh);
                if (!s.ok) continue;
                const int32_t x = px - s.ix, y = py - s.iy;
                if (x < s.x0 || x >= s.x1 || y < s.y0 || y >= s.y1) continue;
                if (!sample_reaches(s, c.x, c.y, x, y, f.wh, r2)) continue;
                const float w = recon_weight(f, pcx, pcy, c.x, c.y) * multiplier;
                const float4 v = samples[sid];
                wsum += w;
                ax += w * v.x;
                ay += w * v.y;
                az += w * v.z;
            }
        float4 acc = image[p];
        image[p] = make_float4(acc.x + ax, acc.y + ay, acc.z + az, acc.w + wsum);
    }
}

// The same splat for a 16x16 pixel tile per block: the tile's samples with
// their halo (coordinates and values) are staged once in shared memory by
// coalesced row loads, then each thread sums its pixel's window from there in
// the order of k_filter_grid (rows, then columns, ascending), so the image is
// the same bit for bit; only the reads change (each sample was read by up to
// win^2 pixels through L1/L2).
constexpr int32_t kFilterTile = 16;
__global__ void __launch_bounds__(256) k_filter_grid_tiled(const float4* __restrict__ samples,
                                                           const float2* __restrict__ coords,
                                                           uint32_t width, uint32_t height,
                                                           uint32_t sp, ReconFilterDev f,
                                                           float multiplier,
                                                           float4* __restrict__ image) {
    extern __shared__ float4 smem[];
    const int32_t range = static_cast<int32_t>(f.wh);
    const int32_t hi = (range + 2) / 2;
    const int32_t loMin = -(range - 1) / 2 - ((range % 2 == 0) ? 1 : 0);
    const float r2 = f.radius * f.radius;
    const int32_t S = static_cast<int32_t>(sp);
    const int32_t SW = static_cast<int32_t>(width) * S, SH = static_cast<int32_t>(height) * S;
    // staged sample rectangle: pixels [t0 - hi, t0 + tile - 1 - loMin + 1], times S
    const int32_t span = (kFilterTile + hi - loMin + 1) * S;
    float4* sv = smem;                                           // span * span values
    float2* sc = reinterpret_cast<float2*>(smem + span * span);  // span * span coordinates
    const int32_t tilesX = (static_cast<int32_t>(width) + kFilterTile - 1) / kFilterTile;
    const int32_t tx0 = (static_cast<int32_t>(blockIdx.x) % tilesX) * kFilterTile;
    const int32_t ty0 = (static_cast<int32_t>(blockIdx.x) / tilesX) * kFilterTile;
    const int32_t ox = (tx0 - hi) * S, oy = (ty0 - hi) * S;      // staged origin (samples)
    // A sample's coordinates may round into the pixel beside its own.  Where
    // no staged sample's did (nearly every tile), the windows need not be
    // widened by that pixel: with one sample per pixel and a 3-pixel window, 9
    // candidates per pixel instead of 25 (1080p, the same window: 107 -> 75 us with
    // one sample per pixel, 355 -> 238 us with four).
    bool own = true;
    for (int32_t i = threadIdx.x; i < span * span; i += blockDim.x) {
        const int32_t ly = i / span, lx = i - ly * span;
        const int32_t sy = oy + ly, sx = ox + lx;
        if (sy >= 0 && sy < SH && sx >= 0 && sx < SW) {
            const size_t sid = size_t(sy) * size_t(SW) + size_t(sx);
            const float2 c = coords[sid];
            sc[i] = c;
            sv[i] = samples[sid];
            const SamplePix s = sample_pix(c.x, c.y, f.wh);
            own = own && s.ok && s.ix == sx / S && s.iy == sy / S;
        }
    }
    const int32_t slack = __syncthreads_and(own) ? 0 : 1;
    const int32_t px = tx0 + static_cast<int32_t>(threadIdx.x) % kFilterTile;
    const int32_t py = ty0 + static_cast<int32_t>(threadIdx.x) / kFilterTile;
    if (px >= static_cast<int32_t>(width) || py >= static_cast<int32_t>(height)) return;
    const float pcx = static_cast<float>(px) + 0.5f, pcy = static_cast<float>(py) + 0.5f;
    const int32_t sy0 = max(0, (py - hi + 1 - slack) * S),
                  sy1 = min(SH, (py - loMin + 1 + slack) * S);
    const int32_t sx0 = max(0, (px - hi + 1 - slack) * S),
                  sx1 = min(SW, (px - loMin + 1 + slack) * S);
    float ax = 0.0f, ay = 0.0f, az = 0.0f, wsum = 0.0f;
    for (int32_t sy = sy0; sy < sy1; sy++)
        for (int32_t sx = sx0; sx < sx1; sx++) {
            const int32_t li = (sy - oy) * span + (sx - ox);
            const float2 c = sc[li];
            const SamplePix s = sample_pix(c.x, c.y, f.wh);
            if (!s.ok) continue;
            const int32_t x = px - s.ix, y = py - s.iy;
            if (x < s.x0 || x >= s.x1 || y < s.y0 || y >= s.y1) continue;
            if (!sample_reaches(s, c.x, c.y, x, y, f.wh, r2)) continue;
            const float w = recon_weight(f, pcx, pcy, c.x, c.y) * multiplier;
            const float4 v = sv[li];
            wsum += w;
            ax += w * v.x;
            ay += w * v.y;
            az += w * v.z;
        }
    const size_t p = size_t(py) * width + size_t(px);
    float4 acc = image[p];
    image[p] = make_float4(acc.x + ax, acc.y + ay, acc.z + az, acc.w + wsum);
}

// KCCheckPixels (ImageMemory.cu:34-60)
__global__ void __launch_bounds__(256) k_check_pixels(float* __restrict__ pixels, uint32_t channels,
                                                      size_t count) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < count;
         i += size_t(gridDim.x) * blockDim.x) {
        if (channels == 4) {
            float4* p4 = reinterpret_cast<float4*>(pixels) + i;
            const float4 v = *p4;
            if (isnan(v.x) || isnan(v.y) || isnan(v.z) || isnan(v.w))
                *p4 = make_float4(1.0e30f, 0.0f, 1.0e30f, 1.0f);
        } else if (isnan(pixels[i])) {
            pixels[i] = 1.0e30f;
        }
    }
}

inline uint32_t grid_of(size_t n, uint32_t cap) {
    size_t g = (n + 255) / 256;
    if (g == 0) g = 1;
    return static_cast<uint32_t>(g < cap ? g : cap);
}

inline int key_bits(uint32_t pixels) {
    int b = 1;
    while (b < 32 && (uint64_t(1) << b) < pixels) b++;
    return b;
}

}  // namespace

int recon_filter_make(const char* type, float radius, uint32_t optCount, const char* const* names,
                      const float* values, ReconFilterDev* out) {
    if (!type || !out || (optCount && (!names || !values))) {
        set_error("recon filter: null argument");
        return MRB_E_ARG;
    }
    // the window grows with the radius (wh^2 pairs per sample); 64 pixels
    // is far beyond any filter the tracer configurations use
    if (!(radius >= 0.0f) || !(radius <= 64.0f)) {
        set_error("recon filter: radius %g outside [0, 64]", double(radius));
        return MRB_E_ARG;
    }
    auto option = [&](const char* key, float* v) {
        for (uint32_t i = 0; i < optCount; i++)
            if (names[i] && std::strcmp(names[i], key) == 0) {
                *v = values[i];
                return true;
            }
        return false;
    };
    ReconFilterDev f{};
    f.radius = radius;
    f.wh = filter_pixel_wh(radius);
    if (std::strcmp(type, "Box") == 0) {
        f.type = kReconBox;
    } else {
        if (radius == 0.0f) {
            set_error("recon filter: radius 0 is only defined for the Box filter");
            return MRB_E_ARG;
        }
        if (std::strcmp(type, "Tent") == 0) {
            f.type = kReconTent;
            f.recipRadius = 1.0f / radius;
        } else if (std::strcmp(type, "Gaussian") == 0) {
            float alpha;
            if (!option("alpha", &alpha)) {
                set_error("Gauss Filter parameter \"alpha\" not found");
                return MRB_E_ARG;
            }
            f.type = kReconGaussian;
            f.negAlpha = -alpha;
            f.gaussEdge = recon_gauss(f, radius);
        } else if (std::strcmp(type, "Mitchell") == 0) {
            float b, c;
            if (!option("b", &b)) {
                set_error("Mitchell Filter parameter \"b\" not found");
                return MRB_E_ARG;
            }
            if (!option("c", &c)) {
                set_error("Mitchell Filter parameter \"c\" not found");
                return MRB_E_ARG;
            }
            // GPUMitchellFilterFunctor (GPUReconFilterMitchell.h:78-95)
            const float t = 1.0f / 6.0f;
            f.type = kReconMitchell;
            f.recipRadius = 1.0f / radius;
            f.c01[0] = t * (12 - 9 * b - 6 * c);
            f.c01[1] = t * (-18 + 12 * b + 6 * c);
            f.c01[2] = 0.0f;
            f.c01[3] = t * (6 + 2 * b + 0 * c);
            f.c12[0] = t * (-1 * b - 6 * c);
            f.c12[1] = t * (6 * b + 30 * c);
            f.c12[2] = t * (-12 * b - 48 * c);
            f.c12[3] = t * (8 * b + 24 * c);
        } else {
            set_error("recon filter: unknown type \"%s\" (Box, Tent, Gaussian, Mitchell)", type);
            return MRB_E_ARG;
        }
    }
    *out = f;
    return 0;
}

// Most tiles that a sample's window touches.
static uint32_t tiles_per_sample(const ReconFilterDev& f) {
    const uint32_t axis = (f.wh + uint32_t(kTileSide) - 2u) / uint32_t(kTileSide) + 1u;
    return axis * axis;
}
static uint32_t tile_columns(const ImageSeg& seg) {
    return uint32_t(seg.w - 1) / uint32_t(kTileSide) + 1u;
}
static uint32_t tile_total(const ImageSeg& seg) {
    return tile_columns(seg) * (uint32_t(seg.h - 1) / uint32_t(kTileSide) + 1u);
}

// Whether a splat lists samples by tile or by pixel.  A sample reaches pi r^2
// pixels and touches (1 + (wh - 1) / 8)^2 tiles on average: 1.8 and 1.6 with a radius
// of 0.75, 1.1 and 1.6 with 0.6.  Pairs and tiles, whole splat (us), 104,000 and 4.1M
// samples on 1080p, then 16,000 on 128 x 128 and 262,000 on 256 x 256: radius 0.6 94 and 90,
// 515 and 681, 58 and 55, 81 and 101; 0.75 98 and 90, 677 and 689, 58 and 54, 89 and 90;
// 0.8 102 and 90, 753 and 691, 59 and 54, 92 and 91.
static bool use_tiles(const ReconFilterDev& f) { return f.radius >= 0.75f; }

// Carves the scratch of a splat out of base (null: only adds up its bytes).
static size_t carve(unsigned char* base, const ReconFilterDev& f, uint32_t n, const ImageSeg& seg,
                    ReconScratch& s) {
    size_t at = 0;
    auto take = [&](size_t bytes) {
        unsigned char* p = base ? base + at : nullptr;
        at += align256(bytes);
        return p;
    };
    const bool tiles = use_tiles(f);
    const size_t entries = size_t(n) * (tiles ? tiles_per_sample(f) : f.wh * f.wh);
    const size_t lists = tiles ? tile_total(seg) : size_t(seg.w) * size_t(seg.h);
    s.count = reinterpret_cast<uint32_t*>(take((size_t(n) + 1) * 4));
    s.offset = reinterpret_cast<uint32_t*>(take((size_t(n) + 1) * 4));
    s.scanTemp = take(exclusive_scan_temp_bytes(n));
    s.keys = reinterpret_cast<uint32_t*>(take(entries * 4));
    s.vals = reinterpret_cast<uint32_t*>(take(entries * 4));
    s.entries = static_cast<uint32_t>(entries);
    s.bits = key_bits(static_cast<uint32_t>(lists));
    s.sortTempBytes = radix_sort_temp_bytes(s.entries, 4, 0, s.bits);
    s.sortTemp = take(s.sortTempBytes);
    if (tiles) {
        // runs, the number of crowded tiles (cleared with them) and their list
        // the runs, the lengths of the two lists (cleared with them), the lists: a
        // tile in one has more than kCrowd (kDense) entries
        const size_t crowd = std::min(lists, entries / kCrowd);
        s.tiles = reinterpret_cast<uint2*>(
            take(lists * 8 + 8 + (crowd + std::min(lists, entries / kDense)) * 4));
        s.crowds.counts = reinterpret_cast<uint32_t*>(s.tiles + lists);
        s.crowds.crowd = s.crowds.counts + 2;
        s.crowds.dense = s.crowds.crowd + crowd;
    } else {
        s.begin = reinterpret_cast<uint32_t*>(take(lists * 4));
        s.end = reinterpret_cast<uint32_t*>(take(lists * 4));
    }
    return at;
}

size_t recon_scratch_bytes(const ReconFilterDev& f, uint32_t n, const ImageSeg& seg) {
    ReconScratch s{};
    return carve(nullptr, f, n, seg, s);
}

ReconScratch recon_scratch_carve(void* base, const ReconFilterDev& f, uint32_t n,
                                 const ImageSeg& seg) {
    ReconScratch s{};
    carve(static_cast<unsigned char*>(base), f, n, seg, s);
    return s;
}

static int splat_pairs(const ReconFilterDev& f, const ImageSeg& seg, const float* values,
                       uint32_t channels, const float2* coords, uint32_t n, float multiplier,
                       float* pixels, float* counts, const ReconScratch& s, cudaStream_t stream) {
    const size_t pix = size_t(seg.w) * size_t(seg.h);
    const uint32_t g = grid_of(n, 148 * 8);
    k_expand_count<<<g, 256, 0, stream>>>(coords, n, f, seg, s.count);
    if (exclusive_scan_u32(s.count, s.offset, n, s.scanTemp, stream)) return MRB_E_CUDA;
    k_expand_write<<<g, 256, 0, stream>>>(coords, n, f, seg, s.offset, s.keys, s.vals);
    const uint32_t* dTotal = s.offset + n;
    if (radix_sort_pairs<uint32_t>(s.keys, s.vals, dTotal, s.entries, 0, s.bits, false, s.sortTemp,
                                   s.sortTempBytes, stream, false))
        return MRB_E_CUDA;
    MRB_CUDA(cudaMemsetAsync(s.begin, 0, pix * 4, stream));
    MRB_CUDA(cudaMemsetAsync(s.end, 0, pix * 4, stream));
    k_pixel_bounds<<<grid_of(s.entries, 148 * 8), 256, 0, stream>>>(s.keys, dTotal, s.begin, s.end);
    const uint32_t gp = grid_of(pix, 148 * 16);
    if (channels == 4)
        k_filter_pixels<4><<<gp, 256, 0, stream>>>(s.begin, s.end, s.vals, values, coords, f, seg,
                                                   multiplier, pixels, counts);
    else
        k_filter_pixels<1><<<gp, 256, 0, stream>>>(s.begin, s.end, s.vals, values, coords, f, seg,
                                                   multiplier, pixels, counts);
    MRB_CUDA(cudaGetLastError());
    return 0;
}

static int splat_tiles(const ReconFilterDev& f, const ImageSeg& seg, const float* values,
                       uint32_t channels, const float2* coords, uint32_t n, float multiplier,
                       float* pixels, float* counts, const ReconScratch& s, cudaStream_t stream) {
    const int32_t columns = static_cast<int32_t>(tile_columns(seg));
    const uint32_t g = grid_of(n, 148 * 8);
    const uint32_t words = 2u * tile_total(seg) + 2u;
    k_tile_count<<<grid_of(std::max(n, words), 148 * 8), 256, 0, stream>>>(
        coords, n, f.wh, seg, s.count, reinterpret_cast<uint32_t*>(s.tiles), words);
    if (exclusive_scan_u32(s.count, s.offset, n, s.scanTemp, stream)) return MRB_E_CUDA;
    k_tile_write<<<g, 256, 0, stream>>>(coords, n, f.wh, seg, columns, s.offset, s.keys, s.vals);
    const uint32_t* dTotal = s.offset + n;
    if (radix_sort_pairs<uint32_t>(s.keys, s.vals, dTotal, s.entries, 0, s.bits, false, s.sortTemp,
                                   s.sortTempBytes, stream, false))
        return MRB_E_CUDA;
    k_tile_bounds<<<grid_of(s.entries, 148 * 8), 256, 0, stream>>>(s.keys, dTotal, s.tiles,
                                                                   s.crowds);
    // a tile lists a sample once, so few samples crowd no tile
    const uint32_t crowdBlocks =
        n > kCrowd ? std::min({148u * 6u, tile_total(seg), s.entries / kCrowd}) : 0u;
    const uint32_t blocks =
        crowdBlocks + (uint32_t(seg.w - 1) / 16u + 1u) * (uint32_t(seg.h - 1) / 16u + 1u);
    auto launch = [&](auto ch, auto type) {
        k_filter_tiles<decltype(ch)::value, decltype(type)::value>
            <<<blocks, kSplatBlock, 0, stream>>>(s.tiles, s.crowds, crowdBlocks, columns, s.vals,
                                                 values, coords, f, seg, multiplier, pixels, counts);
    };
    auto of_type = [&](auto ch) {
        switch (f.type) {
            case kReconBox: launch(ch, std::integral_constant<int, kReconBox>{}); break;
            case kReconTent: launch(ch, std::integral_constant<int, kReconTent>{}); break;
            case kReconGaussian: launch(ch, std::integral_constant<int, kReconGaussian>{}); break;
            default: launch(ch, std::integral_constant<int, kReconMitchell>{}); break;
        }
    };
    if (channels == 4) of_type(std::integral_constant<int, 4>{});
    else of_type(std::integral_constant<int, 1>{});
    MRB_CUDA(cudaGetLastError());
    return 0;
}

int recon_filter_to_img(const ReconFilterDev& f, const ImageSeg& seg, const float* values,
                        uint32_t channels, const float2* coords, uint32_t n, float multiplier,
                        float* pixels, float* counts, const ReconScratch& s, cudaStream_t stream) {
    if (n == 0 || seg.w <= 0 || seg.h <= 0) return 0;
    const auto splat = use_tiles(f) ? splat_tiles : splat_pairs;
    return splat(f, seg, values, channels, coords, n, multiplier, pixels, counts, s, stream);
}

int recon_filter_grid(const ReconFilterDev& f, const float4* samples, const float2* coords,
                      uint32_t width, uint32_t height, uint32_t sp, float multiplier,
                      float4* image, cudaStream_t stream) {
    const size_t pix = size_t(width) * height;
    // the tiled form where its staged rectangle fits the default 48 KB of
    // shared memory (1 and 2 samples per pixel axis with small filters)
    const int32_t range = static_cast<int32_t>(f.wh);
    const int32_t hi = (range + 2) / 2;
    const int32_t loMin = -(range - 1) / 2 - ((range % 2 == 0) ? 1 : 0);
    const size_t span = size_t(kFilterTile + hi - loMin + 1) * sp;
    const size_t smemBytes = span * span * (sizeof(float4) + sizeof(float2));
    if (smemBytes <= 48 * 1024) {
        const size_t tiles = size_t((width + kFilterTile - 1) / kFilterTile) *
                             ((height + kFilterTile - 1) / kFilterTile);
        k_filter_grid_tiled<<<static_cast<uint32_t>(tiles), 256, smemBytes, stream>>>(
            samples, coords, width, height, sp, f, multiplier, image);
    } else {
        k_filter_grid<<<grid_of(pix, 148 * 16), 256, 0, stream>>>(samples, coords, width, height,
                                                                 sp, f, multiplier, image);
    }
    MRB_CUDA(cudaGetLastError());
    return 0;
}

int image_check_pixels(float* pixels, uint32_t channels, size_t count, cudaStream_t stream) {
    if (count == 0) return 0;
    k_check_pixels<<<grid_of(count, 148 * 8), 256, 0, stream>>>(pixels, channels, count);
    MRB_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace mrb

// ---------------------------------------------------------------------------
// C ABI: GPUReconFilterI (GPUReconFilterI.h:6-33) and ImageMemory
// (ImageMemory.h:14-78)
// ---------------------------------------------------------------------------
struct mrb_recon_filter {
    mrb::ReconFilterDev f{};
    char type[16] = {};
    void* scratch = nullptr;
    size_t scratchBytes = 0;
    ~mrb_recon_filter() {
        if (scratch) cudaFree(scratch);
    }
};

struct mrb_image {
    int32_t resW = 0, resH = 0, offX = 0, offY = 0, w = 0, h = 0;
    uint32_t channels = 4;
    float* pixels = nullptr;
    float* counts = nullptr;
    void* mem = nullptr;
    ~mrb_image() {
        if (mem) cudaFree(mem);
    }
    size_t pixel_count() const { return size_t(w) * size_t(h); }
    mrb::ImageSeg seg() const { return mrb::ImageSeg{offX, offY, w, h, resW, resH}; }
};

namespace mrb {
const ReconFilterDev* recon_filter_dev(const mrb_recon_filter* f) { return f ? &f->f : nullptr; }
}  // namespace mrb

namespace {
int image_alloc(mrb_image* im) {
    if (im->mem) cudaFree(im->mem);
    im->mem = nullptr;
    im->pixels = im->counts = nullptr;
    const size_t pix = im->pixel_count();
    if (pix == 0) return 0;
    const size_t pbytes = (pix * im->channels * 4 + 255) & ~size_t(255);
    cudaError_t e = cudaMalloc(&im->mem, pbytes + pix * 4);
    if (e != cudaSuccess) {
        cudaGetLastError();
        im->mem = nullptr;
        mrb::set_error("image: cudaMalloc of %zu bytes failed: %s", pbytes + pix * 4,
                       cudaGetErrorString(e));
        return MRB_E_OOM;
    }
    im->pixels = static_cast<float*>(im->mem);
    im->counts = reinterpret_cast<float*>(static_cast<unsigned char*>(im->mem) + pbytes);
    MRB_CUDA(cudaMemset(im->mem, 0, pbytes + pix * 4));
    return 0;
}
}  // namespace

extern "C" {

int mrb_recon_filter_create(const char* type, float radius, uint32_t option_count,
                            const char* const* option_names, const float* option_values,
                            mrb_recon_filter** out) {
    if (!out) {
        mrb::set_error("recon filter: null output");
        return MRB_E_ARG;
    }
    *out = nullptr;
    mrb::ReconFilterDev f;
    int r = mrb::recon_filter_make(type, radius, option_count, option_names, option_values, &f);
    if (r) return r;
    mrb_recon_filter* h = new mrb_recon_filter();
    h->f = f;
    std::strncpy(h->type, type, sizeof(h->type) - 1);
    *out = h;
    return 0;
}

void mrb_recon_filter_destroy(mrb_recon_filter* f) { delete f; }

const char* mrb_recon_filter_type(const mrb_recon_filter* f) { return f ? f->type : nullptr; }

size_t mrb_recon_filter_used_bytes(const mrb_recon_filter* f) { return f ? f->scratchBytes : 0; }

uint32_t mrb_recon_filter_pixel_wh(float radius) { return mrb::filter_pixel_wh(radius); }

float mrb_recon_filter_weight(const mrb_recon_filter* f, float pixel_x, float pixel_y,
                              float sample_x, float sample_y) {
    if (!f) return 0.0f;
    return mrb::recon_weight(f->f, pixel_x, pixel_y, sample_x, sample_y);
}

int mrb_recon_filter_to_img(mrb_recon_filter* f, mrb_image* img, const float* d_values,
                            uint32_t channels, const float* d_img_coords, uint32_t sample_count,
                            float scalar_multiplier, void* stream) {
    if (!f || !img || (sample_count && (!d_values || !d_img_coords))) {
        mrb::set_error("recon filter: null argument");
        return MRB_E_ARG;
    }
    if (channels != img->channels) {
        mrb::set_error("recon filter: %u-channel values into a %u-channel image", channels,
                       img->channels);
        return MRB_E_ARG;
    }
    if ((channels == 4 && (reinterpret_cast<uintptr_t>(d_values) & 15)) ||
        (reinterpret_cast<uintptr_t>(d_img_coords) & 7)) {
        mrb::set_error("recon filter: values need 16-byte (RGBA) and coordinates 8-byte alignment");
        return MRB_E_ARG;
    }
    if (sample_count == 0 || img->pixel_count() == 0) return 0;
    if (size_t(sample_count) * f->f.wh * f->f.wh >= (size_t(1) << 32)) {
        mrb::set_error("recon filter: %u samples x %u pixels each exceed 2^32 pairs", sample_count,
                       f->f.wh * f->f.wh);
        return MRB_E_ARG;
    }
    const mrb::ImageSeg seg = img->seg();
    const size_t need = mrb::recon_scratch_bytes(f->f, sample_count, seg);
    if (need > f->scratchBytes) {
        if (f->scratch) {
            cudaFree(f->scratch);
            f->scratch = nullptr;
            f->scratchBytes = 0;
        }
        cudaError_t e = cudaMalloc(&f->scratch, need);
        if (e != cudaSuccess) {
            cudaGetLastError();
            f->scratch = nullptr;
            mrb::set_error("recon filter: cudaMalloc of %zu bytes failed: %s", need,
                           cudaGetErrorString(e));
            return MRB_E_OOM;
        }
        f->scratchBytes = need;
    }
    const mrb::ReconScratch s = mrb::recon_scratch_carve(f->scratch, f->f, sample_count, seg);
    return mrb::recon_filter_to_img(f->f, seg, d_values, channels,
                                    reinterpret_cast<const float2*>(d_img_coords), sample_count,
                                    scalar_multiplier, img->pixels, img->counts, s,
                                    static_cast<cudaStream_t>(stream));
}

int mrb_image_create(int32_t width, int32_t height, uint32_t channels, mrb_image** out) {
    if (!out || width <= 0 || height <= 0 || (channels != 1 && channels != 4) ||
        int64_t(width) * height > (int64_t(1) << 31)) {
        mrb::set_error("image: bad size %dx%d or channel count %u (1 or 4)", width, height,
                       channels);
        return MRB_E_ARG;
    }
    mrb_image* im = new mrb_image();
    im->resW = im->w = width;
    im->resH = im->h = height;
    im->channels = channels;
    int r = image_alloc(im);
    if (r) {
        delete im;
        return r;
    }
    *out = im;
    return 0;
}

void mrb_image_destroy(mrb_image* img) { delete img; }

int mrb_image_reportion(mrb_image* img, int32_t start_x, int32_t start_y, int32_t end_x,
                        int32_t end_y) {
    if (!img) return MRB_E_ARG;
    // ImageMemory::Reportion (ImageMemory.cu:111-137): end clamped to the resolution
    end_x = end_x < img->resW ? end_x : img->resW;
    end_y = end_y < img->resH ? end_y : img->resH;
    if (start_x < 0 || start_y < 0 || end_x < start_x || end_y < start_y) {
        mrb::set_error("image: portion [%d,%d)-[%d,%d) outside the image", start_x, start_y,
                       end_x, end_y);
        return MRB_E_ARG;
    }
    img->offX = start_x;
    img->offY = start_y;
    img->w = end_x - start_x;
    img->h = end_y - start_y;
    return image_alloc(img);
}

int mrb_image_resize(mrb_image* img, int32_t width, int32_t height) {
    if (!img) return MRB_E_ARG;
    // ImageMemory::Resize: the segment must still fit
    if (width <= 0 || height <= 0 || img->offX + img->w > width || img->offY + img->h > height) {
        mrb::set_error("image: resolution %dx%d does not hold the current portion", width, height);
        return MRB_E_ARG;
    }
    img->resW = width;
    img->resH = height;
    return 0;
}

int mrb_image_reset(mrb_image* img, void* stream) {
    if (!img) return MRB_E_ARG;
    if (!img->mem) return 0;
    const size_t pix = img->pixel_count();
    const size_t pbytes = (pix * img->channels * 4 + 255) & ~size_t(255);
    MRB_CUDA(cudaMemsetAsync(img->mem, 0, pbytes + pix * 4, static_cast<cudaStream_t>(stream)));
    return 0;
}

int mrb_image_info(const mrb_image* img, int32_t* info7) {
    if (!img || !info7) return MRB_E_ARG;
    const int32_t v[7] = {img->offX, img->offY, img->w, img->h, img->resW, img->resH,
                          static_cast<int32_t>(img->channels)};
    std::memcpy(info7, v, sizeof(v));
    return 0;
}

int mrb_image_device(const mrb_image* img, float** d_pixels, float** d_sample_counts) {
    if (!img) return MRB_E_ARG;
    if (d_pixels) *d_pixels = img->pixels;
    if (d_sample_counts) *d_sample_counts = img->counts;
    return 0;
}

int mrb_image_get(mrb_image* img, float* host_pixels, float* host_counts, void* stream) {
    if (!img || !host_pixels || !host_counts) return MRB_E_ARG;
    const size_t pix = img->pixel_count();
    if (pix == 0) return 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // ImageMemory::GetImageToCPU (ImageMemory.cu:150-190): NaN check, copy, reset
    if (mrb::image_check_pixels(img->pixels, img->channels, pix, st)) return MRB_E_CUDA;
    MRB_CUDA(cudaMemcpyAsync(host_pixels, img->pixels, pix * img->channels * 4,
                             cudaMemcpyDeviceToHost, st));
    MRB_CUDA(cudaMemcpyAsync(host_counts, img->counts, pix * 4, cudaMemcpyDeviceToHost, st));
    if (mrb_image_reset(img, stream)) return MRB_E_CUDA;
    MRB_CUDA(cudaStreamSynchronize(st));
    return 0;
}

}  // extern "C"

#include "io.cuh"

extern "C" int mrb_image_write(mrb_image* img, const char* path) {
    if (!img || !path) return MRB_E_ARG;
    const size_t pix = img->pixel_count();
    if (pix == 0) return MRB_E_ARG;
    std::vector<float> px(pix * img->channels), cnt(pix);
    MRB_CUDA(cudaMemcpy(px.data(), img->pixels, px.size() * 4, cudaMemcpyDeviceToHost));
    MRB_CUDA(cudaMemcpy(cnt.data(), img->counts, cnt.size() * 4, cudaMemcpyDeviceToHost));
    return mrb::write_averaged(path, px.data(), cnt.data(), 1, static_cast<uint32_t>(img->w),
                               static_cast<uint32_t>(img->h), img->channels, img->channels);
}
