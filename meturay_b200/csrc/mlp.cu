// Learned guiding MLP on the tcgen05 tensor cores.
//
// Shared-memory operand layout (no swizzle, "interleaved" core matrices):
// a core matrix is 8 rows x 16 bytes (8 bf16), its rows 16 bytes apart.
//   activations  X / H / G  (128 samples x F features): core matrix
//                (sample group sg, feature group fg) at sg*(F/8)*128 + fg*128
//   weights      W (in x 64 out): core matrix (input group ig, output group
//                og) at ig*1024 + og*128, each of its rows one input's 8
//                outputs
// One copy of each serves every product it enters:
//   forward      D[s][o] = sum_i X[s][i] W[i][o]      A = X  K-major,
//                                                     B = W  MN-major
//   input grad   dX[s][i] = sum_o G[s][o] W[i][o]     A = G  K-major,
//                                                     B = W  K-major
//   weight grad  dW^T[o][i] = sum_s G[s][o] X[s][i]   A = G  MN-major,
//                                                     B = X  MN-major
// Forward and input gradients use M = 128 (one sample per TMEM lane);
// weight gradients use M = 64 (output features; TMEM lanes 0-15, 32-47,
// 64-79, 96-111) and accumulate in TMEM over all tiles a CTA processes.
// One elected thread issues the MMAs; completion is signalled through an
// mbarrier whose waits are bounded (on expiry the kernel flags an error,
// frees its tensor memory and returns).
#include "../../include/mrb200.h"
#include "mlp_tile.cuh"

namespace mrb {

namespace {

// ---- shared by inference and training -------------------------------------
// 128-bit loads of feature rows into the bf16 activation buffer (rows past n
// zero): per load instruction a warp takes 16 features of 8 rows, so that its
// eight 64-byte pieces fill whole sectors and its 8-byte stores the 256 bytes
// of two core matrices.  kRows rows per warp, a multiple of 8.
template <int kRows>
__device__ __forceinline__ void load_rows(unsigned char* x, const float* __restrict__ in,
                                          uint32_t n, uint32_t tileRow, uint32_t firstRow) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int g = 0; g < kRows / 8; g++) {
        const uint32_t row = firstRow + 8u * g + (lane >> 2);
        const bool ok = tileRow + row < n;
        const float4* p = reinterpret_cast<const float4*>(in + size_t(tileRow + row) * kMlpIn) +
                          (lane & 3u);
        float4 q[kMlpIn / 16];
#pragma unroll
        for (int c = 0; c < kMlpIn / 16; c++)
            q[c] = ok ? __ldg(p + 4 * c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int c = 0; c < kMlpIn / 16; c++) {
            uint2 w;
            w.x = uint32_t(bf16_bits(q[c].x)) | (uint32_t(bf16_bits(q[c].y)) << 16);
            w.y = uint32_t(bf16_bits(q[c].z)) | (uint32_t(bf16_bits(q[c].w)) << 16);
            *reinterpret_cast<uint2*>(x + act_offset(row, 16u * c + 4u * (lane & 3u), kMlpIn)) = w;
        }
    }
}

// kCols columns from col0 of this thread's row, bias added (and ReLU) and
// rounded to bf16, into an activation buffer of 64 features.
template <int kCols>
__device__ __forceinline__ void store_hidden(unsigned char* h, uint32_t row, uint32_t col0,
                                             const float* v, const float* bias) {
#pragma unroll
    for (int c = 0; c < kCols / 8; c++) {
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float a = fmaxf(v[8 * c + 2 * k] + bias[8 * c + 2 * k], 0.0f);
            const float b = fmaxf(v[8 * c + 2 * k + 1] + bias[8 * c + 2 * k + 1], 0.0f);
            w[k] = uint32_t(bf16_bits(a)) | (uint32_t(bf16_bits(b)) << 16);
        }
        *reinterpret_cast<uint4*>(h + act_offset(row, col0 + 8u * c, 64)) =
            make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// The forward product of layer l, issued by one thread (A: 128 rows of the
// layer's inputs, K-major; B: its weights, MN-major).
template <class SM>
__device__ __forceinline__ void issue_forward(SM& S, uint32_t tmem, const unsigned char* A, int l) {
    const uint32_t K = (l == 0) ? kMlpIn : 64;
    const uint32_t a0 = smem_u32(A), b0 = smem_u32(S.w + image_layer_offset(l));
    for (uint32_t k0 = 0; k0 < K; k0 += 16) {
        const uint64_t ad = smem_desc(a0 + (k0 / 8) * 128u, 128u, (K / 8) * 128u);
        const uint64_t bd = smem_desc(b0 + (k0 / 8) * 1024u, 1024u, 128u);
        mma_bf16(tmem + kColD, ad, bd, idesc_bf16(128, 64, false, true), k0 > 0 ? 1u : 0u);
    }
}

// Weights by one bulk copy into shared memory, biases, barriers and TMEM.
// The copy completes on S.wbar (weights_wait), so that a block's first input
// rows are read meanwhile.
template <class SM>
__device__ __forceinline__ void prologue_async(SM& S, const MlpDev& m, uint32_t cols) {
    if (threadIdx.x == 0) {
        mbar_init(&S.mbar, 1);
        mbar_init(&S.wbar, 1);
        S.fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                         smem_u32(&S.wbar)),
                     "r"(uint32_t(kMlpImageBytes))
                     : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
            "[%3];" ::"r"(smem_u32(S.w)),
            "l"(__cvta_generic_to_global(m.wImage)), "r"(uint32_t(kMlpImageBytes)),
            "r"(smem_u32(&S.wbar))
            : "memory");
    }
    for (uint32_t i = threadIdx.x; i < kMlpLayers * 64; i += blockDim.x) {
        const int l = int(i / 64), o = int(i % 64);
        S.bias[l][o] = m.params[mlp_layer_offset(l) + (l == 0 ? kMlpIn : 64) * 64 + o];
    }
    if (threadIdx.x < 32) {
        tmem_alloc(&S.tmem, cols);
        tmem_relinquish();
    }
}
// Every thread of the block; false (for all of them) when the bounded wait
// for the weights gave up.
template <class SM>
__device__ __forceinline__ bool weights_wait(SM& S, uint32_t* errorFlag) {
    // the thread that set the barrier up and issues the products waits; the
    // others learn the outcome at the block's barrier
    bool ok = threadIdx.x != 0 || mbar_wait(&S.wbar, 0);
    tc_fence_before();
    ok = __syncthreads_and(ok) != 0;
    tc_fence_after();
    if (!ok && threadIdx.x == 0) set_flag(errorFlag);
    return ok;
}

// ---- inference ----------------------------------------------------------------
// Two warpgroups per tile of 128 rows: warp w reads the accumulator's lanes of
// its quarter (w % 4) and 32 of its 64 columns, which halves the serial part
// of every layer (TMEM to registers, bias, ReLU, rounding, shared memory), the
// chain that bounds the kernel; four blocks per SM fill the waits.  The output
// tile is staged over the input buffer and leaves by one bulk copy.  65,536
// rows: 23.4 us with one thread per row, its own row's reads and writes and the
// weights copied before the input; 13.6 us so (31 MB, 4.9 us at the memory's
// rate).
constexpr int kInferThreads = 256;
struct alignas(1024) MlpInferSmem {
    unsigned char w[kMlpImageBytes];
    unsigned char x[kMlpTile * kMlpIn * 2];  // the input tile, each hidden layer, the outputs
    float bias[kMlpLayers][64];
    uint64_t mbar, wbar;
    uint32_t tmem;
    uint32_t fail;
};
static_assert(kMlpTile * kMlpIn * 2 == kMlpTile * kMlpOut * 4, "x holds an output tile");

__global__ void __launch_bounds__(kInferThreads, 4) k_mlp_infer(MlpDev m,
                                                                const float* __restrict__ in,
                                                                float* __restrict__ out,
                                                                uint32_t maxN,
                                                                const uint32_t* __restrict__ dCount) {
    extern __shared__ __align__(1024) unsigned char smemRaw[];
    MlpInferSmem& S = *reinterpret_cast<MlpInferSmem*>(smemRaw);
    const uint32_t n = dCount ? min(*dCount, maxN) : maxN;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t quarter = (warp & 3u) * 32u, row = quarter + lane, col = (warp >> 2) * 32u;
    const uint32_t tiles = (n + kMlpTile - 1) / kMlpTile;
    prologue_async(S, m, 64);
    uint32_t phase = 0;
    bool first = true, ok = true;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        load_rows<kMlpTile / 8>(S.x, in, n, t * kMlpTile, warp * (kMlpTile / 8));
        fence_async_smem();
        if (first) {
            if (!(ok = weights_wait(S, m.errorFlag))) break;
            first = false;
        } else {
            __syncthreads();
        }
        const uint32_t tmem = S.tmem;
#pragma unroll 1
        for (int l = 0; l < kMlpLayers && ok; l++) {
            if (threadIdx.x == 0) {
                issue_forward(S, tmem, S.x, l);
                mma_commit(&S.mbar);
            }
            if (!(ok = mlp_wait(S, phase, m.errorFlag))) break;
            float v[32];
            tmem_ld16(tmem + (quarter << 16) + kColD + col, v);
            tmem_ld16(tmem + (quarter << 16) + kColD + col + 16u, v + 16);
            tmem_wait_ld();
            const float* bias = S.bias[l] + col;
            if (l < kMlpLayers - 1) {
                store_hidden<32>(S.x, row, col, v, bias);
            } else {
                float4* o = reinterpret_cast<float4*>(S.x + row * (kMlpOut * 4) + col * 4);
#pragma unroll
                for (int c = 0; c < 8; c++)
                    if (col + 4u * c < uint32_t(kMlpOut))
                        o[c] = make_float4(v[4 * c] + bias[4 * c], v[4 * c + 1] + bias[4 * c + 1],
                                           v[4 * c + 2] + bias[4 * c + 2],
                                           v[4 * c + 3] + bias[4 * c + 3]);
            }
            fence_async_smem();
            tc_fence_before();
            __syncthreads();
            tc_fence_after();
        }
        if (!ok) break;
        if (threadIdx.x == 0) {
            const uint32_t rows = min(n - t * kMlpTile, uint32_t(kMlpTile));
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                             __cvta_generic_to_global(out + size_t(t) * kMlpTile * kMlpOut)),
                         "r"(smem_u32(S.x)), "r"(rows * uint32_t(kMlpOut * 4))
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
        __syncthreads();
    }
    // a block without a tile still owns its copy
    if (first && ok) weights_wait(S, m.errorFlag);
    mlp_epilogue(S, S.tmem, 64);
}

// ---- training -----------------------------------------------------------------
// Sixteen warps per tile of 128 samples: warp w has the accumulator lanes of
// quarter w % 4 and 16 of its 64 columns, so a thread handles a quarter of a
// sample's row in every step of the chain, and two of its eight lobes in the
// loss.  Bias gradients are column sums of the output gradients: one more
// product, with a matrix whose first column is ones, instead of shuffles over
// every column.  The input gradient of a layer is issued before its weight
// gradient, which then runs under the epilogue.  Bound by that chain's latency:
// 16,384 samples (one tile per block) took 53.0 us with one thread per sample,
// 18.3 us so.
constexpr int kTrainThreads = 512;
constexpr uint32_t kRawStride = 41;  // words per row of raw outputs: odd, no bank conflicts
struct alignas(1024) MlpSmem {
    unsigned char w[kMlpImageBytes];       // weight images, all layers
    unsigned char x[kMlpTile * kMlpIn * 2];
    unsigned char h[3][kMlpTile * 64 * 2];  // post-ReLU activations of the hidden layers
    unsigned char g[2][kMlpTile * 64 * 2];  // output gradients (ping-pong)
    unsigned char ones[256];                // two core matrices: bf16 (1, 0, ..., 0) rows
    float raw[kMlpTile * kRawStride];       // raw outputs; then, per lobe, the loss terms
    float bias[kMlpLayers][64];
    uint64_t mbar, wbar;
    uint32_t tmem;
    uint32_t fail;
};
// TMEM columns: the 128 x 64 accumulator (kColD), then dW^T of each layer
// (64 rows x the layer's inputs) and the bias gradients (8 columns each, the
// first in use).
__host__ __device__ constexpr uint32_t col_dw(int l) {
    return l == 0 ? 64u : 64u + 80u + 64u * uint32_t(l - 1);
}
__host__ __device__ constexpr uint32_t col_db(int l) { return 336u + 8u * uint32_t(l); }

// d(-w log q(dir))/d raw of one sample's lobes 2 cg and 2 cg + 1 into
// g[0..9], by the four threads of the sample (cg = 0..3): each puts its lobes'
// logit, log normaliser and kappa (mu . dir - 1) into terms (3 floats per
// lobe, 24 per sample); after the block's barrier each reads all eight.
struct LobePair {
    float mu[2][3], kappa[2], len[2], r3[2], c[2];
};
__device__ __forceinline__ LobePair lobe_terms(const float* r, float wx, float wy, float wz,
                                               float* terms) {
    LobePair p;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float x = r[5 * k], y = r[5 * k + 1], z = r[5 * k + 2];
        p.len[k] = sqrtf(x * x + y * y + z * z + 1e-12f);
        p.mu[k][0] = x / p.len[k];
        p.mu[k][1] = y / p.len[k];
        p.mu[k][2] = z / p.len[k];
        p.r3[k] = r[5 * k + 3];
        const float lk = fminf(fmaxf(p.r3[k], -10.0f), kMlpLogKappaMax);
        p.kappa[k] = expf(lk);
        p.c[k] = p.mu[k][0] * wx + p.mu[k][1] * wy + p.mu[k][2] * wz;
        terms[3 * k] = r[5 * k + 4];
        terms[3 * k + 1] = lk - logf(2.0f * kPiF) - logf(-expm1f(-2.0f * p.kappa[k]));
        terms[3 * k + 2] = p.kappa[k] * (p.c[k] - 1.0f);
    }
    return p;
}
__device__ __forceinline__ float lobe_grads(const LobePair& p, const float* terms, uint32_t cg,
                                            float wx, float wy, float wz, float weight, float* g) {
    float lse = -INFINITY;
#pragma unroll
    for (int k = 0; k < kMlpLobes; k++) lse = fmaxf(lse, terms[3 * k]);
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < kMlpLobes; k++) s += expf(terms[3 * k] - lse);
    lse += logf(s);
    float lobeLog[kMlpLobes], m = -INFINITY;
#pragma unroll
    for (int k = 0; k < kMlpLobes; k++) {
        lobeLog[k] = (terms[3 * k] - lse) + terms[3 * k + 1] + terms[3 * k + 2];
        m = fmaxf(m, lobeLog[k]);
    }
    s = 0.0f;
#pragma unroll
    for (int k = 0; k < kMlpLobes; k++) s += expf(lobeLog[k] - m);
    const float lq = m + logf(s);
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const float* t = terms + 3 * (2 * cg + j);
        const float logPi = t[0] - lse;
        const float gamma = expf((logPi + t[1] + t[2]) - lq);
        const float pi = expf(logPi);
        const float kap = p.kappa[j], c = p.c[j];
        // direction: (I - mu mu^T) (w kappa) / |r|
        const float sd = -weight * gamma * kap / p.len[j];
        g[5 * j + 0] = sd * (wx - c * p.mu[j][0]);
        g[5 * j + 1] = sd * (wy - c * p.mu[j][1]);
        g[5 * j + 2] = sd * (wz - c * p.mu[j][2]);
        // concentration through kappa = exp(r3) inside the clamp
        const float dlog = 1.0f / kap - 2.0f / expm1f(2.0f * kap) + (c - 1.0f);
        g[5 * j + 3] = (p.r3[j] > -10.0f && p.r3[j] < kMlpLogKappaMax)
                           ? -weight * gamma * dlog * kap
                           : 0.0f;
        // weight logit (softmax)
        g[5 * j + 4] = -weight * (gamma - pi);
    }
    return -lq;
}

__global__ void __launch_bounds__(kTrainThreads, 1) k_mlp_train(
    MlpDev m, const float* __restrict__ in, const float* __restrict__ targets, uint32_t maxN,
    const uint32_t* __restrict__ dCount, float* __restrict__ grad, float* __restrict__ loss) {
    extern __shared__ __align__(1024) unsigned char smemRaw[];
    MlpSmem& S = *reinterpret_cast<MlpSmem*>(smemRaw);
    const uint32_t n = dCount ? min(*dCount, maxN) : maxN;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t q = warp & 3u, cg = warp >> 2;
    const uint32_t row = 32u * q + lane, col = 16u * cg;
    const uint32_t tiles = (n + kMlpTile - 1) / kMlpTile;
    prologue_async(S, m, 512);
    if (threadIdx.x < 128) {  // 16 rows of 8 bf16: (1, 0, ..., 0)
        reinterpret_cast<uint16_t*>(S.ones)[threadIdx.x] = (threadIdx.x & 7u) == 0u ? 0x3F80u : 0u;
    }
    uint32_t phase = 0;
    bool first = true, ok = true;
    float lossSum = 0.0f, weightSum = 0.0f;
    uint32_t tmem = 0;
    const uint32_t acc = (32u * q) << 16;
    auto sync_smem = [&]() {
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    };
    for (uint32_t t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
        const uint32_t s = t * kMlpTile + row;
        load_rows<kMlpTile / 16>(S.x, in, n, t * kMlpTile, warp * (kMlpTile / 16));
        float4 tg = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (s < n) tg = __ldg(reinterpret_cast<const float4*>(targets) + s);
        fence_async_smem();
        if (first) {
            if (!(ok = weights_wait(S, m.errorFlag))) break;
            tmem = S.tmem;
        } else {
            __syncthreads();
        }
#pragma unroll 1
        for (int l = 0; l < kMlpLayers; l++) {
            if (threadIdx.x == 0) {
                issue_forward(S, tmem, l == 0 ? S.x : S.h[l - 1], l);
                mma_commit(&S.mbar);
            }
            if (!(ok = mlp_wait(S, phase, m.errorFlag))) break;
            float v[16];
            tmem_ld16(tmem + acc + kColD + col, v);
            tmem_wait_ld();
            if (l < kMlpLayers - 1) {
                store_hidden<16>(S.h[l], row, col, v, S.bias[l] + col);
            } else {
#pragma unroll
                for (int k = 0; k < 16; k++)
                    if (col + k < uint32_t(kMlpOut))
                        S.raw[row * kRawStride + col + k] = v[k] + S.bias[l][col + k];
            }
            sync_smem();
        }
        if (!ok) break;
        // output gradient of -w log q(dir), zero for a sample without weight
        {
            float r[10], g[10];
            float* raw = S.raw + row * kRawStride;
#pragma unroll
            for (int k = 0; k < 10; k++) {
                r[k] = raw[10u * cg + k];
                g[k] = 0.0f;
            }
            __syncthreads();  // the loss terms take the raw outputs' place
            const LobePair p = lobe_terms(r, tg.x, tg.y, tg.z, raw + 6u * cg);
            __syncthreads();
            if (tg.w > 0.0f) {
                const float nll = lobe_grads(p, raw, cg, tg.x, tg.y, tg.z, tg.w, g);
                if (cg == 0) {
                    lossSum += tg.w * nll;
                    weightSum += tg.w;
                }
            }
            // columns 10 cg .. 10 cg + 9, and 6 of the zero columns 40 .. 63
#pragma unroll
            for (int k = 0; k < 5; k++)
                *reinterpret_cast<uint32_t*>(S.g[0] + act_offset(row, 10u * cg + 2u * k, 64)) =
                    uint32_t(bf16_bits(g[2 * k])) | (uint32_t(bf16_bits(g[2 * k + 1])) << 16);
#pragma unroll
            for (int k = 0; k < 3; k++)
                *reinterpret_cast<uint32_t*>(S.g[0] + act_offset(row, 40u + 6u * cg + 2u * k, 64)) = 0u;
        }
        sync_smem();
        // backward, output layer first
        int cur = 0;
#pragma unroll 1
        for (int l = kMlpLayers - 1; l >= 0; l--) {
            const unsigned char* X = (l == 0) ? S.x : S.h[l - 1];
            const uint32_t F = (l == 0) ? kMlpIn : 64;
            if (threadIdx.x == 0) {
                const uint32_t gA = smem_u32(S.g[cur]), xB = smem_u32(X), o1 = smem_u32(S.ones);
                if (l > 0) {
                    // dX[s][i] = sum_o G[s][o] W[i][o]: A = G K-major, B = W K-major
                    const uint32_t w0 = smem_u32(S.w + image_layer_offset(l));
                    for (uint32_t k0 = 0; k0 < 64; k0 += 16) {
                        const uint64_t ad = smem_desc(gA + (k0 / 8) * 128u, 128u, 1024u);
                        const uint64_t bd = smem_desc(w0 + (k0 / 8) * 128u, 128u, 1024u);
                        mma_bf16(tmem + kColD, ad, bd, idesc_bf16(128, 64, false, false),
                                 k0 > 0 ? 1u : 0u);
                    }
                    mma_commit(&S.mbar);
                }
                // dW^T[o][i] += sum_s G[s][o] X[s][i]: M = 64 outputs, N = F inputs,
                // K = 128 samples; both operands MN-major (sample groups are the K
                // chunks, 8 * row stride apart).  db[o] += sum_s G[s][o] the same way.
                for (uint32_t k0 = 0; k0 < kMlpTile; k0 += 16) {
                    const uint64_t ad = smem_desc(gA + (k0 / 8) * 1024u, 1024u, 128u);
                    const uint64_t bd = smem_desc(xB + (k0 / 8) * (F / 8) * 128u, (F / 8) * 128u, 128u);
                    const uint64_t od = smem_desc(o1, 128u, 128u);
                    const uint32_t more = (first && k0 == 0) ? 0u : 1u;
                    mma_bf16(tmem + col_dw(l), ad, bd, idesc_bf16(64, int(F), true, true), more);
                    mma_bf16(tmem + col_db(l), ad, od, idesc_bf16(64, 8, true, true), more);
                }
                if (l == 0) mma_commit(&S.mbar);
            }
            if (!(ok = mlp_wait(S, phase, m.errorFlag))) break;
            if (l > 0) {
                float dx[16];
                tmem_ld16(tmem + acc + kColD + col, dx);
                const uint4 h0 = *reinterpret_cast<const uint4*>(S.h[l - 1] + act_offset(row, col, 64));
                const uint4 h1 =
                    *reinterpret_cast<const uint4*>(S.h[l - 1] + act_offset(row, col + 8u, 64));
                const uint32_t hw[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
                tmem_wait_ld();
                uint32_t w[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    // activations are rounded ReLU outputs: positive or zero
                    const float a = (hw[k] & 0x7FFFu) ? dx[2 * k] : 0.0f;
                    const float b = (hw[k] & 0x7FFF0000u) ? dx[2 * k + 1] : 0.0f;
                    w[k] = uint32_t(bf16_bits(a)) | (uint32_t(bf16_bits(b)) << 16);
                }
                *reinterpret_cast<uint4*>(S.g[cur ^ 1] + act_offset(row, col, 64)) =
                    make_uint4(w[0], w[1], w[2], w[3]);
                *reinterpret_cast<uint4*>(S.g[cur ^ 1] + act_offset(row, col + 8u, 64)) =
                    make_uint4(w[4], w[5], w[6], w[7]);
                cur ^= 1;
            }
            sync_smem();
        }
        first = false;
    }
    // gradients out of TMEM: the lanes 0..15 of quarter q hold rows (outputs)
    // 16 q .. 16 q + 15 of every dW^T; the 17 chunks of 16 inputs are spread
    // over the four column groups
    if (ok && !first) {
        const uint32_t o = 16u * q + lane;
#pragma unroll 1
        for (uint32_t c = cg; c < 17u; c += 4u) {
            const int l = c < 5u ? 0 : int((c - 5u) / 4u) + 1;
            const uint32_t i0 = l == 0 ? 16u * c : 16u * ((c - 5u) & 3u);
            float* gw = grad + mlp_layer_offset(l);
            float v[16];
            tmem_ld16(tmem + acc + col_dw(l) + i0, v);
            tmem_wait_ld();
            if (lane < 16u) {
#pragma unroll
                for (int k = 0; k < 16; k++) atomicAdd(gw + (i0 + k) * 64 + o, v[k]);
            }
        }
        const int l = int(cg);
        const float b = tmem_ld1(tmem + acc + col_db(l));
        if (lane < 16u) atomicAdd(grad + mlp_layer_offset(l) + (l == 0 ? kMlpIn : 64) * 64 + o, b);
        if (cg == 0) {
            for (int sh = 16; sh > 0; sh >>= 1) {
                lossSum += __shfl_xor_sync(0xFFFFFFFFu, lossSum, sh);
                weightSum += __shfl_xor_sync(0xFFFFFFFFu, weightSum, sh);
            }
            if (lane == 0) {
                atomicAdd(loss + 0, lossSum);
                atomicAdd(loss + 1, weightSum);
            }
        }
    } else if (first && ok) {
        ok = weights_wait(S, m.errorFlag);  // a block without a tile still owns its copy
    }
    mlp_epilogue(S, S.tmem, 512);
}

// Parameter i: its layer, and for weights (i, o) and the image offset.
__device__ __forceinline__ bool param_weight(uint32_t i, int& l, uint32_t& in, uint32_t& out) {
    l = 0;
    while (l + 1 < kMlpLayers && i >= uint32_t(mlp_layer_offset(l + 1))) l++;
    const uint32_t local = i - uint32_t(mlp_layer_offset(l));
    const uint32_t K = (l == 0) ? kMlpIn : 64;
    if (local >= K * 64) return false;  // a bias
    in = local / 64;
    out = local % 64;
    return true;
}

// The output layer's columns past the 40 outputs (weights and biases) and
// the input rows past the 78 features stay zero.
__device__ __forceinline__ bool param_frozen(uint32_t i) {
    int l;
    uint32_t in, out;
    if (param_weight(i, l, in, out))
        return (l == kMlpLayers - 1 && out >= kMlpOut) || (l == 0 && in >= kMlpFeatures);
    const uint32_t o = (i - uint32_t(mlp_layer_offset(l))) % 64;
    return l == kMlpLayers - 1 && o >= kMlpOut;
}

__global__ void __launch_bounds__(256) k_mlp_adam(float* __restrict__ params, float* __restrict__ m1,
                                                  float* __restrict__ m2, const uint32_t* step,
                                                  float* __restrict__ grad,
                                                  const float* __restrict__ loss, float lr,
                                                  uint16_t* __restrict__ image) {
    const bool empty = !(loss[1] > 0.0f);  // a batch without weight: no step
    const uint32_t t = *step + 1u;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - powf(b1, float(t)), c2 = 1.0f - powf(b2, float(t));
    const float inv = 1.0f / fmaxf(loss[1], 1e-20f);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < uint32_t(kMlpParams);
         i += gridDim.x * blockDim.x) {
        float p = params[i];
        if (!empty && !param_frozen(i)) {
            const float g = grad[i] * inv;
            const float a = b1 * m1[i] + (1.0f - b1) * g;
            const float b = b2 * m2[i] + (1.0f - b2) * g * g;
            m1[i] = a;
            m2[i] = b;
            p -= lr * (a / c1) / (sqrtf(b / c2) + 1e-8f);
            params[i] = p;
        }
        grad[i] = 0.0f;
        int l;
        uint32_t in, out;
        if (param_weight(i, l, in, out))
            image[(image_layer_offset(l) + w_offset(in, out)) / 2] = bf16_bits(p);
    }
}

__global__ void k_mlp_step(uint32_t* step, const float* loss) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && loss[1] > 0.0f) *step += 1u;
}

__global__ void __launch_bounds__(256) k_mlp_image(const float* __restrict__ params,
                                                   uint16_t* __restrict__ image) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < uint32_t(kMlpParams);
         i += gridDim.x * blockDim.x) {
        int l;
        uint32_t in, out;
        if (param_weight(i, l, in, out))
            image[(image_layer_offset(l) + w_offset(in, out)) / 2] = bf16_bits(params[i]);
    }
}

__global__ void __launch_bounds__(256) k_mlp_encode(const float* __restrict__ pos,
                                                    const float* __restrict__ nrm,
                                                    const float* __restrict__ wo, uint32_t n,
                                                    float* __restrict__ out) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        float f[kMlpIn];
        encode_vertex(pos[3 * s], pos[3 * s + 1], pos[3 * s + 2], nrm[3 * s], nrm[3 * s + 1],
                      nrm[3 * s + 2], wo[3 * s], wo[3 * s + 1], wo[3 * s + 2], f);
        float4* d = reinterpret_cast<float4*>(out + size_t(s) * kMlpIn);
#pragma unroll
        for (int c = 0; c < kMlpIn / 4; c++)
            d[c] = make_float4(f[4 * c], f[4 * c + 1], f[4 * c + 2], f[4 * c + 3]);
    }
}

int mlp_smem_setup() {
    static bool done[64] = {};
    int dev = 0;
    MRB_CUDA(cudaGetDevice(&dev));
    if (!done[dev & 63]) {
        MRB_CUDA(cudaFuncSetAttribute(k_mlp_infer,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      int(sizeof(MlpInferSmem))));
        MRB_CUDA(cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      int(sizeof(MlpSmem))));
        done[dev & 63] = true;
    }
    return 0;
}

uint32_t mlp_grid(uint32_t n, uint32_t perSm = 1) {
    const uint32_t tiles = (n + kMlpTile - 1) / kMlpTile;
    const uint32_t cap = 148u * perSm;
    return tiles < cap ? (tiles ? tiles : 1u) : cap;
}

}  // namespace

int mlp_forward(const MlpDev& m, const float* in, uint32_t n, float* out, cudaStream_t st,
                const uint32_t* dCount) {
    if (n == 0) return 0;
    if (mlp_smem_setup()) return MRB_E_CUDA;
    k_mlp_infer<<<mlp_grid(n, 4), kInferThreads, sizeof(MlpInferSmem), st>>>(m, in, out, n, dCount);
    MRB_CUDA(cudaGetLastError());
    return 0;
}

int mlp_gradients(const MlpDev& m, const float* in, const float* targets, uint32_t n, float* grad,
                  float* loss, cudaStream_t st, const uint32_t* dCount, uint32_t maxCtas) {
    if (n == 0) return 0;
    if (mlp_smem_setup()) return MRB_E_CUDA;
    uint32_t grid = mlp_grid(n);
    if (maxCtas && grid > maxCtas) grid = maxCtas;
    k_mlp_train<<<grid, kTrainThreads, sizeof(MlpSmem), st>>>(m, in, targets, n, dCount, grad, loss);
    MRB_CUDA(cudaGetLastError());
    return 0;
}

int mlp_adam(float* params, float* m1, float* m2, uint32_t* step, float* grad, const float* loss,
             float lr, uint16_t* wImage, cudaStream_t st) {
    k_mlp_adam<<<(kMlpParams + 255) / 256, 256, 0, st>>>(params, m1, m2, step, grad, loss, lr,
                                                        wImage);
    k_mlp_step<<<1, 32, 0, st>>>(step, loss);
    MRB_CUDA(cudaGetLastError());
    return 0;
}

int mlp_build_image(const float* params, uint16_t* wImage, cudaStream_t st) {
    k_mlp_image<<<(kMlpParams + 255) / 256, 256, 0, st>>>(params, wImage);
    MRB_CUDA(cudaGetLastError());
    return 0;
}

int mlp_encode(const float* pos, const float* nrm, const float* wo, uint32_t n, float* out,
               cudaStream_t st) {
    if (n == 0) return 0;
    k_mlp_encode<<<(n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8, 256, 0, st>>>(pos, nrm,
                                                                                     wo, n, out);
    MRB_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace mrb

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
#include "objects.cuh"

struct mrb_mlp {
    mrb_system* sys = nullptr;
    DBuf params, m1, m2, grad, loss, step, image, err;
    mrb::MlpDev dev() const {
        return mrb::MlpDev{params.as<float>(), image.as<uint16_t>(), err.as<uint32_t>()};
    }
};

namespace {
int mlp_check(mrb_mlp* m, cudaStream_t st) {
    uint32_t e = 0;
    MRB_CUDA(cudaMemcpyAsync(&e, m->err.p, 4, cudaMemcpyDeviceToHost, st));
    MRB_CUDA(cudaStreamSynchronize(st));
    if (e) {
        mrb::set_error("MLP: a tensor-core wait gave up");
        return MRB_E_DEVICE;
    }
    return 0;
}
}  // namespace

namespace mrb {
MlpDev mlp_dev(const mrb_mlp* m) { return m->dev(); }
float* mlp_params(mrb_mlp* m) { return m->params.as<float>(); }
int mlp_train_step_dev(mrb_mlp* m, const float* in, const float* targets, uint32_t maxN,
                       const uint32_t* dCount, float lr, cudaStream_t st, uint32_t maxCtas) {
    MRB_CUDA(cudaMemsetAsync(m->loss.p, 0, 8, st));
    int r = mlp_gradients(m->dev(), in, targets, maxN, m->grad.as<float>(), m->loss.as<float>(),
                          st, dCount, maxCtas);
    if (r) return r;
    return mlp_adam(m->params.as<float>(), m->m1.as<float>(), m->m2.as<float>(),
                    m->step.as<uint32_t>(), m->grad.as<float>(), m->loss.as<float>(), lr,
                    m->image.as<uint16_t>(), st);
}
uint32_t* mlp_error_flag(mrb_mlp* m) { return m->err.as<uint32_t>(); }
float* mlp_loss(mrb_mlp* m) { return m->loss.as<float>(); }
size_t mlp_state_bytes() { return size_t(kMlpParams) * 4 * 3 + 16 + kMlpImageBytes; }
// Parameters, optimiser state and weight image to / from a device buffer.
int mlp_state_copy(mrb_mlp* m, void* buf, bool save, cudaStream_t st) {
    const size_t P = size_t(kMlpParams) * 4;
    unsigned char* b = static_cast<unsigned char*>(buf);
    DBuf* parts[5] = {&m->params, &m->m1, &m->m2, &m->step, &m->image};
    const size_t sizes[5] = {P, P, P, 16, kMlpImageBytes};
    for (int i = 0; i < 5; i++) {
        if (save) MRB_CUDA(cudaMemcpyAsync(b, parts[i]->p, sizes[i], cudaMemcpyDeviceToDevice, st));
        else MRB_CUDA(cudaMemcpyAsync(parts[i]->p, b, sizes[i], cudaMemcpyDeviceToDevice, st));
        b += sizes[i];
    }
    return 0;
}
}  // namespace mrb

extern "C" {

uint32_t mrb_mlp_param_count(void) { return uint32_t(mrb::kMlpParams); }

int mrb_mlp_create(mrb_system* sys, mrb_mlp** out) {
    if (!sys || !out) return MRB_E_ARG;
    *out = nullptr;
    MRB_CUDA(cudaSetDevice(sys->device));
    mrb_mlp* m = new mrb_mlp();
    m->sys = sys;
    const size_t P = size_t(mrb::kMlpParams) * 4;
    int r;
    if ((r = m->params.alloc(P)) || (r = m->m1.alloc(P)) || (r = m->m2.alloc(P)) ||
        (r = m->grad.alloc(P)) || (r = m->loss.alloc(16)) || (r = m->step.alloc(16)) ||
        (r = m->image.alloc(mrb::kMlpImageBytes)) || (r = m->err.alloc(16))) {
        delete m;
        return r;
    }
    cudaError_t e = cudaSuccess;
    for (DBuf* b : {&m->params, &m->m1, &m->m2, &m->grad, &m->loss, &m->step, &m->image, &m->err})
        if (e == cudaSuccess) e = cudaMemset(b->p, 0, b->bytes);
    if (e != cudaSuccess) {
        delete m;
        MRB_CUDA(e);
    }
    *out = m;
    return 0;
}

void mrb_mlp_destroy(mrb_mlp* m) { delete m; }

int mrb_mlp_set_params(mrb_mlp* m, const float* host) {
    if (!m || !host) return MRB_E_ARG;
    const size_t P = size_t(mrb::kMlpParams) * 4;
    MRB_CUDA(cudaMemcpy(m->params.p, host, P, cudaMemcpyHostToDevice));
    MRB_CUDA(cudaMemset(m->m1.p, 0, P));
    MRB_CUDA(cudaMemset(m->m2.p, 0, P));
    MRB_CUDA(cudaMemset(m->grad.p, 0, P));
    MRB_CUDA(cudaMemset(m->step.p, 0, 16));
    if (mrb::mlp_build_image(m->params.as<float>(), m->image.as<uint16_t>(), nullptr))
        return MRB_E_CUDA;
    MRB_CUDA(cudaDeviceSynchronize());
    return 0;
}

int mrb_mlp_get_params(const mrb_mlp* m, float* host) {
    if (!m || !host) return MRB_E_ARG;
    MRB_CUDA(cudaMemcpy(host, m->params.p, size_t(mrb::kMlpParams) * 4, cudaMemcpyDeviceToHost));
    return 0;
}

int mrb_mlp_encode(const float* d_pos, const float* d_nrm, const float* d_wo, uint32_t n,
                   float* d_features, void* stream) {
    if (n && (!d_pos || !d_nrm || !d_wo || !d_features)) return MRB_E_ARG;
    return mrb::mlp_encode(d_pos, d_nrm, d_wo, n, d_features, static_cast<cudaStream_t>(stream));
}

int mrb_mlp_forward(mrb_mlp* m, const float* d_features, uint32_t n, float* d_out, void* stream) {
    if (!m || (n && (!d_features || !d_out))) return MRB_E_ARG;
    if ((reinterpret_cast<uintptr_t>(d_features) | reinterpret_cast<uintptr_t>(d_out)) & 15) {
        mrb::set_error("MLP: features and outputs need 16-byte alignment");
        return MRB_E_ARG;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int r = mrb::mlp_forward(m->dev(), d_features, n, d_out, st);
    return r ? r : mlp_check(m, st);
}

int mrb_mlp_gradients(mrb_mlp* m, const float* d_features, const float* d_targets, uint32_t n,
                      float* d_grad, float* d_loss, void* stream) {
    if (!m || !d_grad || !d_loss || (n && (!d_features || !d_targets))) return MRB_E_ARG;
    if ((reinterpret_cast<uintptr_t>(d_features) | reinterpret_cast<uintptr_t>(d_targets)) & 15) {
        mrb::set_error("MLP: features and targets need 16-byte alignment");
        return MRB_E_ARG;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int r = mrb::mlp_gradients(m->dev(), d_features, d_targets, n, d_grad, d_loss, st);
    return r ? r : mlp_check(m, st);
}

int mrb_mlp_train_step(mrb_mlp* m, const float* d_features, const float* d_targets, uint32_t n,
                       float lr, float* host_loss2, void* stream) {
    if (!m || (n && (!d_features || !d_targets))) return MRB_E_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    MRB_CUDA(cudaMemsetAsync(m->loss.p, 0, 8, st));
    int r = mrb::mlp_gradients(m->dev(), d_features, d_targets, n, m->grad.as<float>(),
                               m->loss.as<float>(), st);
    if (r) return r;
    if (host_loss2)
        MRB_CUDA(cudaMemcpyAsync(host_loss2, m->loss.p, 8, cudaMemcpyDeviceToHost, st));
    r = mrb::mlp_adam(m->params.as<float>(), m->m1.as<float>(), m->m2.as<float>(),
                      m->step.as<uint32_t>(), m->grad.as<float>(), m->loss.as<float>(), lr,
                      m->image.as<uint16_t>(), st);
    if (r) return r;
    return mlp_check(m, st);
}

}  // extern "C"
