// Training and inference of the learned path-guiding proposal (guide.cuh)
// on the fifth-generation tensor cores, and the dl_guide C ABI.
//
// One training step on a batch of n records {position, normal, sampled
// direction w, its sampling pdf p, radiance estimate L along w}:
//   loss = -(1/n) sum_i min((L_i / p_i) / mean(L / p), 20) * log q(w_i)
// (an estimate of the KL divergence from the normalised incident radiance to
// the mixture q, up to a constant), then one Adam update.  Kernels:
//   k_guide_weight_sum   mean(L / p) over the batch (once for the steps of a
//                        call, which take the same records)
//   k_guide_train        forward, loss gradient, backward and the weight
//                        and bias gradients per 128-record tile (tcgen05.mma),
//                        activations kept in shared memory, gradient sums in
//                        tensor memory; one partial gradient per block
//   k_guide_grad_reduce  the blocks' partial gradients summed; in a training
//                        step also Adam on the fp32 master weights, which
//                        refreshes the tensor cores' fp16 weight image
// Inference (k_guide_infer, and the guided material kernels in render.cu)
// runs on tcgen05 too (guide_tc.cuh).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "guide.cuh"
#include "guide_tc.cuh"
#include "internal.h"
#include "scene.h"

namespace dl {

// ------------------------------------------------------------- inference
static_assert(kGImgTrainBytes == kGuideImageBytes, "image size");

// Raw network outputs (40 per row) of n input rows, 128 rows per tile on
// the tensor cores; each of a block's five warpgroups walks its own tiles
// (one block per SM: five tiles' chains of dependent layers overlap, one
// weight copy in shared memory).
constexpr int kInferGroups = 5;
using InferSmem = GuideTcSmemT<kInferGroups>;
constexpr int kInferThreads = kTcRows * kInferGroups;
static_assert(sizeof(InferSmem) + 1024 <= 227 * 1024, "one inference block per SM");

__global__ void __launch_bounds__(kInferThreads, 1) k_guide_infer(const void* image, const float* in, float* out,
                                                                   int n, unsigned* err) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    InferSmem& S = *reinterpret_cast<InferSmem*>(dyn_smem);
    const int ntiles = (n + kTcRows - 1) / kTcRows;
    if ((int)blockIdx.x * kInferGroups >= ntiles) return;
    const int g = tc_group(), row = tc_row();
    uint32_t phase = 0;
    bool ok = guide_tc_begin(S, image, err);
    for (int tile = blockIdx.x * kInferGroups + g; ok && tile < ntiles; tile += gridDim.x * kInferGroups) {
        const int r = tile * kTcRows + row;
        float x[kGIn] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (r < n)
            for (int i = 0; i < kGIn; i++) x[i] = in[(size_t)kGIn * r + i];
        wg_sync(g);  // the previous tile's outputs have been read
        encode_row_tc(x, S.act[g], row);
        ok = guide_tc_forward(S, g, phase, err);
        if (ok) {
            // the tile's rows are contiguous in `out`: copy them out as
            // consecutive 16-byte chunks (coalesced stores), 10 per row
            wg_sync(g);
            const int rows = min(kTcRows, n - tile * kTcRows);
            float4* dst = reinterpret_cast<float4*>(out + (size_t)tile * kTcRows * kGOut);
            const float* src = tc_out_row(S, g, 0);
            for (int c = row; c < rows * (kGOut / 4); c += kTcRows) {
                const float* q = src + (c / (kGOut / 4)) * kTcOutStride + 4 * (c % (kGOut / 4));
                dst[c] = make_float4(q[0], q[1], q[2], q[3]);
            }
        }
    }
    guide_tc_end(S, phase);
}

// -------------------------------------------------------------- training
// Record weights L/p are normalised by their batch mean and clamped at this
// multiple of it: a few records near the sun would otherwise carry the
// whole gradient of a batch.
constexpr float kGTargetClamp = 20.f;

// Per block of 256 threads, the sum of L / p over its records into
// part[blockIdx.x] (the training kernel adds the blocks' sums); block 0
// also clears the batch's loss accumulator.
constexpr int kWsumThreads = 256, kWsumMaxBlocks = 1024;
__global__ void __launch_bounds__(kWsumThreads) k_guide_weight_sum(const GuideRecord* s, int n, int stride,
                                                                    float* part, float* loss) {
    tc::pdl_launch_dependents();
    __shared__ float s_w[kWsumThreads / 32];
    float acc = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const GuideRecord& r = s[(size_t)i * stride];
        acc += r.pdf > 0.f ? r.L / r.pdf : 0.f;
    }
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int k = 0; k < kWsumThreads / 32; k++) t += s_w[k];
        part[blockIdx.x] = t;
        if (blockIdx.x == 0) *loss = 0.f;
    }
}

// Half of the loss gradient of one record, computed by two threads: this
// one takes lobes 4h .. 4h + 3, from their 20 outputs o[0..19] (bias
// added).  The lobes are decoded as decode_lobes does and the mixture's pdf
// taken as vmf_pdf (guide.cuh), here with the hardware's fast exponential,
// logarithm and division -- this runs once per record and training step,
// latency-bound, and the gradients stay within the oracle's 1e-2 -- where
// the renderer's sampling keeps the accurate forms.  The mixture's
// normalisation needs both halves: each thread publishes, in `mine`, its
// largest logit, its sum of exp(logit - that) and the same sum weighted by
// the lobes' pdfs, and reads the other half's from `other` after `exchange`,
// which waits for it and returns the record's loss weight (both halves then
// hold the same sums, added in the same order).  Writes the 20 gradients,
// times that weight, to d; returns the record's loss, -weight log q.
template <typename F>
__device__ __forceinline__ float record_grad_half(const float* o, float3 w, float4* mine, const float4* other,
                                                  F exchange, float* d) {
    constexpr int kH = kGLobes / 2;
    float mx = -1e30f;
#pragma unroll
    for (int j = 0; j < kH; j++) mx = fmaxf(mx, o[5 * j + 4]);
    float3 mu[kH];
    float kap[kH], e[kH], inv_len[kH], pdf[kH], dt[kH], e2[kH], ia[kH];
    bool clamped[kH];
    float se = 0.f, sq = 0.f;
#pragma unroll
    for (int j = 0; j < kH; j++) {
        const float3 m = f3(o[5 * j], o[5 * j + 1], o[5 * j + 2]);
        const float len2 = m.x * m.x + m.y * m.y + m.z * m.z;
        if (len2 > 1e-12f) {
            inv_len[j] = rsqrtf(len2);
            mu[j] = f3(m.x * inv_len[j], m.y * inv_len[j], m.z * inv_len[j]);
        } else {
            inv_len[j] = 0.f;
            mu[j] = f3(0.f, 0.f, 1.f);
        }
        const float lk = o[5 * j + 3];
        clamped[j] = lk < kGLogKappaMin || lk > kGLogKappaMax;
        const float k = __expf(fminf(fmaxf(lk, kGLogKappaMin), kGLogKappaMax));
        kap[j] = k;
        e[j] = __expf(o[5 * j + 4] - mx);
        dt[j] = mu[j].x * w.x + mu[j].y * w.y + mu[j].z * w.z;
        // e^{-2k} and 1 / (1 - e^{-2k}), shared by the pdf and its kappa derivative
        e2[j] = __expf(-2.f * k);
        ia[j] = __fdividef(1.f, 1.f - e2[j]);
        pdf[j] = k < 1e-4f ? 0.25f * kInvPiF : k * ia[j] * (0.5f * kInvPiF) * __expf(k * (dt[j] - 1.f));
        se += e[j];
        sq += e[j] * pdf[j];
    }
    *mine = make_float4(mx, se, sq, 0.f);
    const float scale = exchange();
    const float4 x = *other;
    const float M = fmaxf(mx, x.x);
    const float am = __expf(mx - M), ao = __expf(x.x - M);
    const float lsum = se * am + x.y * ao;   // sum of exp(logit - M) over the 8 lobes
    const float inv_sum = __fdividef(1.f, lsum);
    const float q = (sq * am + x.z * ao) * inv_sum;
#pragma unroll
    for (int j = 0; j < 5 * kH; j++) d[j] = 0.f;
    if (!(q > 1e-30f) || !(scale > 0.f) || !isfinite(scale)) return 0.f;
    const float inv_q = __fdividef(1.f, q);
#pragma unroll
    for (int j = 0; j < kH; j++) {
        const float lam = e[j] * am * inv_sum, k = kap[j];
        const float r = lam * pdf[j] * inv_q;
        // d(-log q)/d(logit_j) = -(r_j - lambda_j)
        d[5 * j + 4] = -scale * (r - lam);
        // d(-log q)/d(log kappa_j) = -r_j (1 - 2k / (e^{2k} - 1) + k (mu.w - 1)),
        // 2k / (e^{2k} - 1) = 2k e^{-2k} / (1 - e^{-2k})
        if (!clamped[j]) {
            const float t = k < 1e-4f ? 0.f : 1.f - 2.f * k * e2[j] * ia[j] + k * (dt[j] - 1.f);
            d[5 * j + 3] = -scale * r * t;
        }
        // d(-log q)/dm_j = -r_j kappa_j (w - (mu.w) mu) / |m_j|
        const float f = -scale * r * k * inv_len[j];
        d[5 * j + 0] = f * (w.x - dt[j] * mu[j].x);
        d[5 * j + 1] = f * (w.y - dt[j] * mu[j].y);
        d[5 * j + 2] = f * (w.z - dt[j] * mu[j].z);
    }
    return -scale * __logf(q);
}

// One training batch on the tensor cores, in three kernels:
//
//   k_guide_weight_sum  per-block sums of the records' L / pdf (the loss's
//                    target normalisation).
//   k_guide_train    one block per SM over a range of 128-record tiles, two
//                    tiles at a time: two groups of 256 threads walk one tile
//                    each and one thread of a seventeenth warp issues every
//                    tcgen05.mma of both, both operands in shared memory and
//                    the fp32 accumulator in tensor memory.  Per tile:
//                      forward  x -> h1 -> h2 -> outputs (3 products);
//                      the loss and dLoss/dOutput of each record (d0, fp16);
//                      backward d2 = (d0 W3) * [h2 > 0], d1 = (d2 W2) *
//                               [h1 > 0] (B operands W3^T, W2^T from the
//                               weight image);
//                      the tile's share of the weight and bias gradients,
//                               accumulated in tensor memory over the
//                               block's tiles (K = the tile's records):
//                               d0^T [1 | h2] (b3, dW3), d2^T [h1 | 1] (dW2,
//                               b2) and d1^T [x | 1] (dW1, b1).
//                    A tile's activations are one matrix of 128 records in the
//                    canonical layout, which the forward and backward products
//                    read as a K-major operand and the gradient products as
//                    an MN-major one (M or N = features, K = records); d2
//                    takes h2's place and d1 takes h1's, each when the
//                    gradient product that reads the activation is done.
//                    A group splits each epilogue's 64 accumulator columns
//                    over its two warpgroups, and each record's loss (four
//                    lobes each).  At the end each block writes its gradient
//                    sums from tensor memory to global memory, feature-major
//                    (coalesced stores; layout below).
//   k_guide_grad_reduce  sums the blocks' partials in a fixed order (no
//                    atomics) into the gradient, in the parameter layout,
//                    applying the loss's 1/n.
//
// Loss scaling: the fp16 activation gradients leave out the loss's 1/n
// (with n ~ 1e5 records most of them would be fp16 subnormals); they
// saturate at the fp16 range, and the 1/n is applied, in fp32, in the
// reduction.
//
// What bounds it: a tile is a chain of six dependent steps -- products, their
// completion, an epilogue over 128 rows, a barrier -- of 10600 cycles when a
// block works on one tile, the tensor cores busy for 2600 of them (48
// products of 128 rows, 48 to 82 cycles each: at these widths the operands'
// way from shared memory sets the time).  The second tile in the first one's
// waits makes it 13400 cycles for two.  The issuing warp keeps its control
// flow converged and predicates the instructions on one lane: descriptors
// then stay in uniform registers (issued from one lane's branch, a product
// took 100 cycles).  131072 records: 51.8 us for the batch's kernels with one
// tile at a time and its two warpgroups, 41.5 with two; 64 records 15 us
// either way.  Shared memory holds two tiles, not three (88 KB each, beside
// 47 KB of weights).
// The two chains' products are issued in a fixed order (step by step, the
// first group's before the second's), so that the gradient sums are added
// tile by tile in the same order whatever the groups' timing.
constexpr int kTrGroup = 2 * kTcRows;                  // threads of a group: two warpgroups
constexpr int kTrGroups = 2;
constexpr int kTrThreads = kTrGroups * kTrGroup + 32;  // and the issuing warp
// a tile's operand matrix [x | 1 | h1, then d1 | 1 | h2, then d2 | d0]
// (halves per record, feature offsets)
constexpr int kR1x = kGEnc, kRh1 = kR1x + 16, kR1h = kRh1 + kGHid, kRh2 = kR1h + 16, kRd0 = kRh2 + kGHid;
constexpr int kRK = kRd0 + kGOutPad;
// tensor memory: the gradient sums -- [dW1 | b1], [dW2 | b2], [b3 | dW3] --
// and each group's forward / backward accumulator (64 columns, reused by
// every product)
constexpr int kTrCols = 512;
constexpr int kAcc1 = 0, kAcc2 = kAcc1 + kGEnc + 16, kAcc3 = kAcc2 + kGHid + 16, kAccF = kAcc3 + kGHid + 16;
static_assert(kAccF + kTrGroups * kGHid <= kTrCols, "tensor-memory columns");
constexpr float kHalfMax = 65504.f;
// A block's gradient sums in global memory, feature-major so that a warp's
// 32 units (accumulator lanes) of one feature are 32 consecutive floats:
// dW1 as [feature][unit], b1, dW2 as [feature][unit], b2, dW3 as
// [feature][output] (40 outputs), b3.
constexpr int kPW1 = 0, kPB1 = kPW1 + kGEnc * kGHid, kPW2 = kPB1 + kGHid, kPB2 = kPW2 + kGHid * kGHid;
constexpr int kPW3 = kPB2 + kGHid, kPB3 = kPW3 + kGHid * kGOut, kPSums = kPB3 + kGOut;   // 16040 floats

// The parameter (guide.cuh layout) that slot t of a block's sums holds.
__host__ __device__ constexpr int guide_sum_param(int t) {
    return t < kPB1   ? kGW1 + (t - kPW1) % kGHid * kGEnc + (t - kPW1) / kGHid
           : t < kPW2 ? kGB1 + t - kPB1
           : t < kPB2 ? kGW2 + (t - kPW2) % kGHid * kGHid + (t - kPW2) / kGHid
           : t < kPW3 ? kGB2 + t - kPB2
           : t < kPB3 ? kGW3 + (t - kPW3) % kGOut * kGHid + (t - kPW3) / kGOut
                      : kGB3 + t - kPB3;
}
static_assert(guide_sum_param(kPSums - 1) == kGB3 + kGOut - 1 && guide_sum_param(kPB3 - 1) == kGW3 + (kGOut - 1) * kGHid + kGHid - 1,
              "sum layout");

struct GuideTrSmem {
    // (a gradient product's 128 rows of A may start at a tile's last features
    // and reach up to 1.3 KB past it -- the other tile or the weights -- in
    // rows of the accumulator that nobody reads)
    alignas(128) __half rec[kTrGroups][kTcRows * kRK];
    alignas(128) __half w[kGImgHalves];       // the weight image: weights, biases,
    float bias[kGImgBiases];                  // W2^T and W3^T
    __half w2t[kGHid * kGHid];
    __half w3t[kGHid * kGOutPad];
    uint64_t bar_w;                           // the weight image has landed
    uint64_t bar_ready[kTrGroups];            // the group's step is written (8 warps)
    uint64_t bar_done[kTrGroups];             // its product is in the accumulator
    uint64_t bar_grad[kTrGroups];             // its gradient products have read their operands
    uint64_t bar_ex[kTrGroups];               // the mixture sums are written (8 warps)
    uint64_t bar_end;                         // every product of the block is complete
    uint32_t tmem;
    float mean[kTrGroups];
    int fail;
};
static_assert(offsetof(GuideTrSmem, w2t) - offsetof(GuideTrSmem, w) == kGImgW2T &&
                  offsetof(GuideTrSmem, w3t) - offsetof(GuideTrSmem, w) == kGImgW3T, "image layout");
static_assert(sizeof(GuideTrSmem) + 1024 <= 227 * 1024, "one training block per SM");
// no other tensor-memory user of this library (the guided material blocks,
// 107 KB; the inference block, 218 KB) fits beside a block: its 512 columns
// are free
static_assert(sizeof(GuideTrSmem) + 1024 + 107 * 1024 > 228 * 1024, "one tensor-memory user per SM");

__device__ __forceinline__ uint32_t as_u32(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 as_h2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }
// Two values as fp16, saturated at the fp16 range (NaN: the lower end).
__device__ __forceinline__ __half2 pack_h2_sat(float a, float b) {
    const __half2 lim = __float2half2_rn(kHalfMax);
    return __hmin2(__hmax2(__floats2half2_rn(a, b), __hneg2(lim)), lim);
}

// An encoded input into features 24 i .. 24 i + 23 of row r.
__device__ __forceinline__ void tr_store_input(const __half2* h, __half* rec, int r, int i) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
        uint4 q;
        q.x = *reinterpret_cast<const uint32_t*>(&h[4 * c]);
        q.y = *reinterpret_cast<const uint32_t*>(&h[4 * c + 1]);
        q.z = *reinterpret_cast<const uint32_t*>(&h[4 * c + 2]);
        q.w = *reinterpret_cast<const uint32_t*>(&h[4 * c + 3]);
        *reinterpret_cast<uint4*>(rec + canon_index(r, i * 2 * kGFreq + 8 * c, kRK)) = q;
    }
}

// Bias + ReLU of the 32 accumulator columns c0 .. c0 + 31 (at t, the warp's
// lanes) into the record's features hf + c0.
__device__ __forceinline__ void tr_hidden_epilogue(uint32_t t, int c0, const float* bias, __half* rec, int r, int hf) {
    float v[32];
    tc::ld_32x32b_x32(t + c0, v);
    const __half2 zero = __float2half2_rn(0.f);
    auto act = [&](int j) {
        return as_u32(__hmax2(__floats2half2_rn(v[j] + bias[c0 + j], v[j + 1] + bias[c0 + j + 1]), zero));
    };
#pragma unroll
    for (int q = 0; q < 32; q += 8)
        *reinterpret_cast<uint4*>(rec + canon_index(r, hf + c0 + q, kRK)) =
            make_uint4(act(q), act(q + 2), act(q + 4), act(q + 6));
}

// The gradients in the 32 accumulator columns c0 .. c0 + 31, as fp16
// (saturated), where the activation they belong to (the record's features hf
// + c0, which they will replace) is positive.
__device__ __forceinline__ void tr_masked(uint32_t t, int c0, const __half* rec, int r, int hf, uint4* p) {
    float v[32];
    tc::ld_32x32b_x32(t + c0, v);
    const __half2 zero = __float2half2_rn(0.f);
    auto grad = [&](int j, uint32_t h) { return as_u32(pack_h2_sat(v[j], v[j + 1])) & __hgt2_mask(as_h2(h), zero); };
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint4 h = *reinterpret_cast<const uint4*>(rec + canon_index(r, hf + c0 + 8 * q, kRK));
        p[q] = make_uint4(grad(8 * q, h.x), grad(8 * q + 2, h.y), grad(8 * q + 4, h.z), grad(8 * q + 6, h.w));
    }
}
__device__ __forceinline__ void tr_store_features(const uint4* p, __half* rec, int r, int f) {
#pragma unroll
    for (int q = 0; q < 4; q++) *reinterpret_cast<uint4*>(rec + canon_index(r, f + 8 * q, kRK)) = p[q];
}

// acc (128 x N) = A x W^T: A = K features from af of the tile at rec
// (K-major); W [N][K] at w (rows of K halves).  A descriptor's address field
// counts 16 bytes and the tiles end below 2^18, so that steps along K add to it.
template <int K, int N>
__device__ __forceinline__ void tr_issue(bool leader, uint32_t acc, uint32_t rec, int af, uint32_t w) {
    constexpr uint32_t idesc = tc::idesc_f16_f32(kTcRows, N);
    const uint64_t a = tc::smem_desc(rec + (af / 8) * 128, 128, kRK * 16), b = tc::smem_desc(w, 128, K * 16);
#pragma unroll
    for (int ks = 0; ks < K / 16; ks++)
        tc::mma_f16_by(leader, acc, a + ks * (256 / 16), b + ks * (256 / 16), idesc, ks > 0 ? 1u : 0u);
}

// Gradient sums (acc, N columns) += A^T B over the tile's 128 records, 16
// per instruction (the block's first tile initialises them): A = 128
// features of the tile from af (those past the wanted ones fill accumulator
// lanes that are never read), B = N features from bf, both MN-major.
template <int N>
__device__ __forceinline__ void tr_issue_grad(bool leader, uint32_t acc, uint32_t rec, int af, int bf, bool first) {
    constexpr uint32_t idesc = tc::idesc_f16_f32(kTcRows, N, true, true);
    const uint64_t a = tc::smem_desc(rec + (af / 8) * 128, kRK * 16, 128);
    const uint64_t b = tc::smem_desc(rec + (bf / 8) * 128, kRK * 16, 128);
#pragma unroll
    for (int ks = 0; ks < kTcRows / 16; ks++)
        tc::mma_f16_by(leader, acc, a + ks * 2 * kRK, b + ks * 2 * kRK, idesc, first && ks == 0 ? 0u : 1u);
}

// The block's products, step by step of each pair of tiles, the first
// group's before the second's: one converged warp, one lane of which issues
// them.  Returns false when a wait ran out.
__device__ __forceinline__ bool tr_issue_all(GuideTrSmem& S, const void* image, int ntiles) {
    constexpr int kSteps = 6;
    const bool leader = tc::elect_one();
    // the weights, once the kernel before (an Adam step, perhaps) has written
    // them: they land while the first tiles' records load and encode
    tc::pdl_wait();
    tc::fence_global_to_async();
    if (leader) tc::bulk_load(S.w, image, kGImgTrainBytes, &S.bar_w);
    __syncwarp();
    const uint32_t T = S.tmem, wa = tc::smem_addr(S.w);
    auto wait = [](uint64_t* bar, uint32_t ph) {
        return __any_sync(0xffffffffu, !tc::mbar_wait(bar, ph, kTcWaitNs)) == 0;
    };
    bool ok = wait(&S.bar_w, 0);
    uint32_t ph = 0;
    for (int tile = blockIdx.x, pair = 0; ok && tile < ntiles; tile += kTrGroups * gridDim.x, pair++) {
        for (int step = 0; ok && step < kSteps; step++, ph ^= 1u) {
            for (int g = 0; g < kTrGroups && tile + g * (int)gridDim.x < ntiles; g++) {
                ok = wait(&S.bar_ready[g], ph);
                if (!ok) break;
                tc::fence_after_sync();
                const uint32_t F = T + kAccF + g * kGHid, rec = tc::smem_addr(S.rec[g]);
                const bool first = pair == 0 && g == 0;
                if (step == 0) {          // x -> h1
                    tr_issue<kGEnc, kGHid>(leader, F, rec, 0, wa + 2 * kGImgW1);
                } else if (step == 1) {   // h1 -> h2
                    tr_issue<kGHid, kGHid>(leader, F, rec, kRh1, wa + 2 * kGImgW2);
                } else if (step == 2) {   // h2 -> outputs
                    tr_issue<kGHid, kGOutPad>(leader, F, rec, kRh2, wa + 2 * kGImgW3);
                } else if (step == 3) {   // d0 W3 -> d2; d0^T [1 | h2]
                    tr_issue<kGOutPad, kGHid>(leader, F, rec, kRd0, wa + kGImgW3T);
                    tc::commit_by(leader, &S.bar_done[g]);
                    tr_issue_grad<kGHid + 16>(leader, T + kAcc3, rec, kRd0, kR1h, first);
                } else if (step == 4) {   // d2 W2 -> d1; d2^T [h1 | 1]
                    tr_issue<kGHid, kGHid>(leader, F, rec, kRh2, wa + kGImgW2T);
                    tc::commit_by(leader, &S.bar_done[g]);
                    tr_issue_grad<kGHid + 16>(leader, T + kAcc2, rec, kRh2, kRh1, first);
                } else {                  // d1^T [x | 1]
                    tr_issue_grad<kGEnc + 16>(leader, T + kAcc1, rec, kRh1, 0, first);
                }
                tc::commit_by(leader, step < 3 ? &S.bar_done[g] : &S.bar_grad[g]);
            }
        }
    }
    tc::commit_by(leader, &S.bar_end);
    return ok;
}

__global__ void __launch_bounds__(kTrThreads, 1) k_guide_train(const void* image, const GuideRecord* s, int n,
                                                                int stride, const float* wsum, int nwsum,
                                                                float* partial, float* loss, unsigned* err) {
    extern __shared__ __align__(128) unsigned char dyn_smem[];
    GuideTrSmem& S = *reinterpret_cast<GuideTrSmem*>(dyn_smem);
    const int tid = threadIdx.x, lane = tid & 31;
    const bool issuer = tid >= kTrGroups * kTrGroup;                // the issuing warp
    const int grp = (tid / kTrGroup) % kTrGroups, gt = tid % kTrGroup;
    const int g = gt >> 7, r = gt & (kTcRows - 1);                  // half of the group, record of the tile
    const int ntiles = (n + kTcRows - 1) / kTcRows;
    if (tid == kTrGroups * kTrGroup) {
        tc::mbar_init(&S.bar_w, 1);
        tc::mbar_init(&S.bar_end, 1);
        for (int i = 0; i < kTrGroups; i++) {
            tc::mbar_init(&S.bar_ready[i], kTrGroup / 32);
            tc::mbar_init(&S.bar_done[i], 1);
            tc::mbar_init(&S.bar_grad[i], 1);
            tc::mbar_init(&S.bar_ex[i], kTrGroup / 32);
        }
        S.fail = 0;
    }
    if (issuer) tc::tmem_alloc(&S.tmem, kTrCols);
    tc::pdl_launch_dependents();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t T = S.tmem;
    const uint32_t lanes = (uint32_t)(tid & 96) << 16;              // this warp's accumulator lanes
    float lacc = 0.f;
    bool failed = false;
    // bounded wait of the whole warp; a warp whose wait ran out leaves its
    // loop, and the waits of the others then run out in turn
    auto wait = [&](uint64_t* bar, uint32_t& ph) {
        const bool ok = tc::mbar_wait(bar, ph, kTcWaitNs);
        ph ^= 1u;
        failed = __any_sync(0xffffffffu, !ok) != 0;
        tc::fence_after_sync();
        return !failed;
    };
    if (issuer) {
        failed = !tr_issue_all(S, image, ntiles);
    } else {
        __half* rec = S.rec[grp];
        const uint32_t tf = T + kAccF + grp * kGHid + lanes;        // the group's accumulator, this warp's lanes
        const int ch = 32 * g;                                      // this warpgroup's epilogue columns
        uint32_t ph_w = 0, ph_done = 0, ph_grad = 0, ph_ex = 0;
        // this warp's part of a step is written and its accumulator reads are done
        auto ready = [&]() {
            tc::fence_smem_to_async();
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&S.bar_ready[grp]);
        };
        // inputs 3g .. 3g + 2 of a record (zeros past the last one); each is
        // loaded a product or two before it is used
        auto load_inputs = [&](int row, float* in) {
            const float* q = reinterpret_cast<const float*>(s + (size_t)row * stride);
#pragma unroll
            for (int i = 0; i < 3; i++) in[i] = row < n ? q[3 * g + i] : 0.f;
        };
        const int step = kTrGroups * gridDim.x;
        int tile = blockIdx.x + grp * (int)gridDim.x;
        if (tile < ntiles) {
            // what every tile shares -- the columns of ones, the zeros after
            // d0's 40 outputs -- and the first tile's encoding
            const uint32_t one2 = as_u32(__float2half2_rn(1.f));
            const uint4 ones = make_uint4(one2, one2, one2, one2);
            *reinterpret_cast<uint4*>(rec + canon_index(r, kR1x + 8 * g, kRK)) = ones;
            *reinterpret_cast<uint4*>(rec + canon_index(r, kR1h + 8 * g, kRK)) = ones;
            if (g == 0) *reinterpret_cast<uint4*>(rec + canon_index(r, kRd0 + kGOut, kRK)) = make_uint4(0u, 0u, 0u, 0u);
            float in[3];
            load_inputs(tile * kTcRows + r, in);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                __half2 h[kGFreq];
                encode_scalar_h2(in[i], h);
                tr_store_input(h, rec, r, 3 * g + i);
            }
            ready();
        }
        tc::pdl_wait();   // the kernels before have finished: the weights are summed, `partial` is free
        if (tile < ntiles) {
            if (gt < 32) {   // the batch's mean weight, summed the same way in every block
                float sum = 0.f;
#pragma unroll 8
                for (int j = lane; j < nwsum; j += 32) sum += wsum[j];
                for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (lane == 0) S.mean[grp] = sum / (float)n;
            }
            (void)wait(&S.bar_w, ph_w);   // the biases
        }
        for (; tile < ntiles && !failed; tile += step) {
            const int row = tile * kTcRows + r;
            const bool more = tile + step < ntiles;
            if (!wait(&S.bar_done[grp], ph_done)) break;
            tr_hidden_epilogue(tf, ch, S.bias + kGImgB1, rec, r, kRh1);
            ready();
            if (!wait(&S.bar_done[grp], ph_done)) break;
            tr_hidden_epilogue(tf, ch, S.bias + kGImgB2, rec, r, kRh2);
            ready();
            // the record's direction, pdf and radiance: in[6] | w[3], pdf, L
            float2 q0 = make_float2(0.f, 0.f), q1 = q0, q2 = q0;
            if (row < n) {
                const float2* q = reinterpret_cast<const float2*>(s + (size_t)row * stride) + 3;
                q0 = q[0];
                q1 = q[1];
                q2 = q[2];
            }
            if (!wait(&S.bar_done[grp], ph_done)) break;
            {   // loss and dLoss/dOutput (times n) of the record, lobes 4g .. 4g + 3, into d0 (features 20g ..)
                float o[20];
                float v[32];
                tc::ld_32x32b_x32(tf + 16 * g, v);   // columns 16g .. 16g + 31 hold outputs 20g .. 20g + 19
#pragma unroll
                for (int j = 0; j < 20; j++) o[j] = (g ? v[4 + j] : v[j]) + S.bias[kGImgB3 + 20 * g + j];
                float dd[20];
                // the halves' sums change hands in d0's place: each half's lie
                // where the other half, having read them, writes its gradients
                float4* ex_mine = reinterpret_cast<float4*>(rec + canon_index(r, kRd0 + (g ? 0 : 24), kRK));
                const float4* ex_other = reinterpret_cast<float4*>(rec + canon_index(r, kRd0 + (g ? 24 : 0), kRK));
                const float lr = record_grad_half(
                    o, f3(q0.x, q0.y, q1.x), ex_mine, ex_other,
                    [&]() {
                        __syncwarp();
                        if (lane == 0) tc::mbar_arrive(&S.bar_ex[grp]);
                        (void)wait(&S.bar_ex[grp], ph_ex);
                        // the record's loss weight times n (the mean was written before the exchange)
                        const float mean = S.mean[grp], pdf = q1.y, Lr = q2.x;
                        return row < n && pdf > 0.f && mean > 0.f ? fminf(Lr / pdf / mean, kGTargetClamp) : 0.f;
                    },
                    dd);
                if (failed) break;
                if (g == 0) lacc += lr;
#pragma unroll
                for (int c = 0; c < 20; c += 4)
                    *reinterpret_cast<uint2*>(rec + canon_index(r, kRd0 + 20 * g + c, kRK)) =
                        make_uint2(as_u32(pack_h2_sat(dd[c], dd[c + 1])), as_u32(pack_h2_sat(dd[c + 2], dd[c + 3])));
            }
            ready();
            float in[3] = {0.f, 0.f, 0.f};   // of the next tile
            if (more) load_inputs(row + step * kTcRows, in);
            uint4 p[4];
            if (!wait(&S.bar_done[grp], ph_done)) break;
            tr_masked(tf, ch, rec, r, kRh2, p);
            if (!wait(&S.bar_grad[grp], ph_grad)) break;   // dW3's product has read h2
            tr_store_features(p, rec, r, kRh2 + ch);
            ready();
            if (!wait(&S.bar_done[grp], ph_done)) break;
            tr_masked(tf, ch, rec, r, kRh1, p);
            if (!wait(&S.bar_grad[grp], ph_grad)) break;   // dW2's product has read h1
            tr_store_features(p, rec, r, kRh1 + ch);
            ready();
            if (!wait(&S.bar_grad[grp], ph_grad)) break;
            if (more) {
#pragma unroll
                for (int i = 0; i < 3; i++) { __half2 h[kGFreq]; encode_scalar_h2(in[i], h); tr_store_input(h, rec, r, 3 * g + i); }
                ready();
            }
        }
    }
    if (failed && lane == 0) {
        S.fail = 1;
        atomicOr(err, kErrTensorWait);
    }
    // every product of the block complete
    __syncthreads();
    uint32_t ph_end = 0;
    if (!wait(&S.bar_end, ph_end) && lane == 0) {
        S.fail = 1;
        atomicOr(err, kErrTensorWait);
    }
    __syncthreads();
    const bool live = S.fail == 0 && (int)blockIdx.x < ntiles;
    for (int o = 16; o; o >>= 1) lacc += __shfl_xor_sync(0xffffffffu, lacc, o);
    if (!issuer && g == 0 && lane == 0) atomicAdd(loss, lacc / (float)n);
    // the block's gradient sums (feature-major: each store of a warp writes
    // one feature of its 32 units, 128 contiguous bytes): accumulator lanes
    // 0..63 hold unit r of layer 1, unit r of layer 2 and output r (< 40);
    // the four warpgroups split the columns
    float* out = partial + (size_t)blockIdx.x * kPSums;
    // ncols (16 or 32) columns from col: column j to out[dst + j * stride];
    // stride 0: a bias (its 16 columns of ones hold the same sum), column 0 only
    auto run = [&](uint32_t col, int ncols, int dst, int stride, bool keep) {
        float v[32];
        if (!live) {
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = 0.f;
        } else if (ncols == 32) {
            tc::ld_32x32b_x32(T + lanes + col, v);
        } else {
            tc::ld_32x32b_x16(T + lanes + col, v);
        }
        if (keep && stride == 0) out[dst] = v[0];
        if (keep && stride > 0)
            for (int j = 0; j < ncols; j++) out[dst + j * stride] = v[j];
    };
    if (!issuer && r < kGHid) {
        const int wg = 2 * grp + g;
        const int o = min(r, kGOut - 1);
        const bool keep = r < kGOut;
        run(kAcc1 + 32 * wg, 32, kPW1 + 32 * wg * kGHid + r, kGHid, true);
        if (wg == 0) {
            run(kAcc1 + 128, 16, kPW1 + 128 * kGHid + r, kGHid, true);
            run(kAcc2, 32, kPW2 + r, kGHid, true);
        } else if (wg == 1) {
            run(kAcc1 + kGEnc, 16, kPB1 + r, 0, true);
            run(kAcc2 + 32, 32, kPW2 + 32 * kGHid + r, kGHid, true);
        } else if (wg == 2) {
            run(kAcc2 + kGHid, 16, kPB2 + r, 0, true);
            run(kAcc3 + 16, 32, kPW3 + o, kGOut, keep);
        } else {
            run(kAcc3, 16, kPB3 + o, 0, keep);
            run(kAcc3 + 48, 32, kPW3 + 32 * kGOut + o, kGOut, keep);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (issuer) {
        if (S.fail) (void)tc::mbar_wait(&S.bar_w, 0, kTcWaitNs);   // the weight copy, after a failed wait
        __syncwarp();
        tc::fence_after_sync();
        tc::tmem_dealloc(T, kTrCols);
    }
}

// Adam's state and this step's constants.
struct AdamStep {
    float* w32;              // fp32 master weights
    unsigned char* image;    // the tensor cores' weight image
    float *m, *v;
    float lr, b1, b2, c1, c2, eps;
};

// The padding of layer 3 (rows 40..47 and their biases): parameters without
// a slot in the blocks' sums, kept zero.
constexpr int kPPads = kGParams - kPSums;
__host__ __device__ constexpr int guide_pad_param(int t) {
    return t < (kGOutPad - kGOut) * kGHid ? kGW3 + kGOut * kGHid + t : kGB3 + kGOut + t - (kGOutPad - kGOut) * kGHid;
}
static_assert(guide_pad_param(0) == kGW3 + kGOut * kGHid && guide_pad_param(kPPads - 1) == kGParams - 1, "padding");

// The gradient of parameter p = guide_sum_param(t): (1/n) times the sum over
// the training blocks of their sums' slot t.  A block takes 32 consecutive
// slots; its 8 warps split the blocks' sums and add theirs in shared memory.
// kAdam: the warp that has the gradients updates their parameters (fp32
// master, weight image) and clears the batch's loss if `loss` is
// given (for the next batch of a call).  Otherwise grad[p] is written.  The
// padding parameters have no slots: Adam clears them.
//
// The sums (9.7 MB over 152 blocks, in the L2 cache) wait on latency, not on
// bandwidth: a warp has all of its loads in flight (four at a time made a
// training step of 131072 records 42.5 us long, twenty 39).  With the update
// as a kernel of its own, and the records' weights summed anew for each step
// of a call, a step took 43.4 us (18.6 instead of 12.4 with 1000 records).
constexpr int kRedWarps = 8;
constexpr int kRedLoads = 20;   // of a warp in flight: its share of 152 blocks' sums
template <bool kAdam>
__global__ void __launch_bounds__(32 * kRedWarps) k_guide_grad_reduce(const float* partial, int nblocks, float inv_n,
                                                                      float* grad, AdamStep A, float* loss) {
    __shared__ float s_sum[kRedWarps][32];
    if (kAdam) tc::pdl_launch_dependents();
    tc::pdl_wait();   // k_guide_train has written every block's partials
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int t = blockIdx.x * 32 + lane;
    const int p = t < kPSums ? guide_sum_param(t) : t < kPSums + kPPads ? guide_pad_param(t - kPSums) : -1;
    float m = 0.f, v = 0.f, x = 0.f;   // Adam's state of the parameter, on its way meanwhile
    if (kAdam && w == 0 && t < kPSums) {
        m = A.m[p];
        v = A.v[p];
        x = A.w32[p];
    }
    float acc = 0.f;
    if (t < kPSums) {
        for (int b0 = w; b0 < nblocks; b0 += kRedWarps * kRedLoads) {
            float q[kRedLoads];
#pragma unroll
            for (int k = 0; k < kRedLoads; k++) {
                const int b = b0 + k * kRedWarps;
                q[k] = b < nblocks ? partial[(size_t)b * kPSums + t] : 0.f;
            }
#pragma unroll
            for (int k = 0; k < kRedLoads; k++) acc += q[k];
        }
    }
    s_sum[w][lane] = acc;
    __syncthreads();
    if (w != 0) return;
    if (kAdam && loss && t == 0) *loss = 0.f;
    if (t < kPSums) {
        float sum = 0.f;
#pragma unroll
        for (int k = 0; k < kRedWarps; k++) sum += s_sum[k][lane];
        const float g = sum * inv_n;
        if (kAdam) {
            // (the roundings are spelt out: Adam's quotient magnifies them)
            m = fmaf(1.f - A.b1, g, __fmul_rn(A.b1, m));
            v = fmaf(__fmul_rn(1.f - A.b2, g), g, __fmul_rn(A.b2, v));
            x = __fsub_rn(x, __fmul_rn(A.lr, m / A.c1) / __fadd_rn(sqrtf(v / A.c2), A.eps));
            A.m[p] = m;
            A.v[p] = v;
        } else {
            grad[p] = g;
        }
    }
    if (kAdam && p >= 0) {
        A.w32[p] = x;   // (the padding: 0)
        write_image(A.image, p, x);
    }
}

__global__ void k_guide_image(const float* w32, unsigned char* image) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kGParams; i += gridDim.x * blockDim.x)
        write_image(image, i, w32[i]);
}

// ------------------------------------------------------------------ host
namespace {

// Deterministic initial weights: uniform(-b, b) with b = sqrt(6 / fan_in)
// for the ReLU layers (He), 0.1 * sqrt(3 / fan_in) for the output layer;
// biases 0 except log kappa = 1 (broad lobes at first).
void init_params(uint64_t seed, std::vector<float>& w) {
    w.assign(kGParams, 0.f);
    uint64_t st = splitmix64(seed ^ 0x6a09e667f3bcc909ULL);
    auto uni = [&]() {
        st = splitmix64(st);
        return (float)((st >> 40) * (1.0 / 16777216.0)) * 2.f - 1.f;
    };
    const float b1 = std::sqrt(6.f / kGEnc), b2 = std::sqrt(6.f / kGHid), b3 = 0.1f * std::sqrt(3.f / kGHid);
    for (int i = 0; i < kGHid * kGEnc; i++) w[kGW1 + i] = b1 * uni();
    for (int i = 0; i < kGHid * kGHid; i++) w[kGW2 + i] = b2 * uni();
    for (int r = 0; r < kGOut; r++)
        for (int c = 0; c < kGHid; c++) w[kGW3 + r * kGHid + c] = b3 * uni();
    for (int j = 0; j < kGLobes; j++) {
        // spread the initial mean directions over the sphere
        float z = 1.f - 2.f * (j + 0.5f) / kGLobes, r = std::sqrt(std::max(0.f, 1.f - z * z));
        float ph = 2.399963f * j;
        w[kGB3 + 5 * j] = r * std::cos(ph);
        w[kGB3 + 5 * j + 1] = r * std::sin(ph);
        w[kGB3 + 5 * j + 2] = z;
        w[kGB3 + 5 * j + 3] = 1.f;
    }
}

}  // namespace

void guide_init_params(uint64_t seed, std::vector<float>& w) { init_params(seed, w); }

void guide_upload_params(dl_guide* G, const float* host) {
    cudaStream_t st = G->ctx->stream;
    DL_CUDA(cudaMemcpyAsync(G->w32.ptr, host, kGParams * 4, cudaMemcpyHostToDevice, st));
    k_guide_image<<<64, 256, 0, st>>>(G->w32.as<float>(), G->image.as<unsigned char>());
    DL_CUDA(cudaGetLastError());
}

// A launch on `st` that may begin while the previous kernel of the stream is
// still running (programmatic stream serialization); the kernel waits for
// that kernel (griddepcontrol.wait) before it reads what it wrote.
template <typename... KArgs, typename... Args>
static cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                    Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Training blocks for a batch of n records: one per SM, at most one per tile.
static int64_t train_blocks(const dl_guide* G, int64_t n) {
    const int64_t ntiles = (n + kTcRows - 1) / kTcRows;
    return std::max<int64_t>(1, std::min<int64_t>(ntiles, std::max(1, G->ctx->num_sms)));
}

// Device buffers of a training batch of up to n records: the blocks' partial
// gradients and the weight sums.  Called before any training launch,
// outside graph captures and render loops.
void guide_reserve(dl_guide* G, int64_t n) {
    G->partial.ensure((size_t)train_blocks(G, n) * kPSums * 4);
    G->wsum.ensure(kWsumMaxBlocks * sizeof(float));
}

// The training kernels of one batch: `n` device records, every `stride`-th.
// The loss sum lands in scratch[1].  `weigh`: sum the records' weights first
// (a batch that repeats the last one on this stream skips it; its loss has
// been cleared).  With `adam` the parameters are updated, else the gradient
// goes to G->grad (entries outside the network's parameters untouched).
// guide_reserve(G, n) must have run.
static void launch_batch(dl_guide* G, const void* d_recs, int64_t n, int stride, cudaStream_t st, bool weigh,
                         const AdamStep* adam, bool clear_loss) {
    if (!G->ctx->train_ready) {
        DL_CUDA(cudaFuncSetAttribute(k_guide_train, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(GuideTrSmem)));
        DL_CUDA(cudaFuncSetAttribute(k_guide_train, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        G->ctx->train_ready = true;
    }
    const int nb = (int)train_blocks(G, n);
    if (n < 1 || G->partial.bytes < (size_t)nb * kPSums * 4 || G->wsum.bytes < kWsumMaxBlocks * sizeof(float))
        throw Error(DL_ERR_INVALID_ARG, "guide training buffers not reserved for this batch");
    float* sc = G->scratch.as<float>();   // [1]: the loss
    unsigned* err = reinterpret_cast<unsigned*>(G->scratch.as<char>() + kGuideErrOffset);
    const GuideRecord* R = static_cast<const GuideRecord*>(d_recs);
    const int nws = (int)std::min<int64_t>(kWsumMaxBlocks, (n + kWsumThreads - 1) / kWsumThreads);
    float* wsum = G->wsum.as<float>();
    if (weigh) k_guide_weight_sum<<<nws, kWsumThreads, 0, st>>>(R, (int)n, stride, wsum, sc + 1);
    // each kernel starts its prologue while its predecessor runs
    // (programmatic dependent launch) and waits for it before using what it
    // wrote; the predecessors have waited for theirs
    float* part = G->partial.as<float>();
    float* grad = G->grad.as<float>();
    const void* img = G->image.ptr;
    const int ni = (int)n;
    const float inv_n = 1.f / (float)n;
    DL_CUDA(launch_dependent(k_guide_train, dim3(nb), dim3(kTrThreads), sizeof(GuideTrSmem), st, img, R, ni, stride,
                             (const float*)wsum, nws, part, sc + 1, err));
    if (adam)
        DL_CUDA(launch_dependent(k_guide_grad_reduce<true>, dim3((kPSums + kPPads + 31) / 32), dim3(32 * kRedWarps), 0,
                                 st, (const float*)part, nb, inv_n, (float*)nullptr, *adam,
                                 clear_loss ? sc + 1 : (float*)nullptr));
    else
        DL_CUDA(launch_dependent(k_guide_grad_reduce<false>, dim3((kPSums + 31) / 32), dim3(32 * kRedWarps), 0, st,
                                 (const float*)part, nb, inv_n, grad, AdamStep{}, (float*)nullptr));
    DL_CUDA(cudaGetLastError());
}

void guide_gradient(dl_guide* G, const void* d_recs, int64_t n, int stride, cudaStream_t st) {
    launch_batch(G, d_recs, n, stride, st, true, nullptr, false);
}

static void guide_steps(dl_guide* G, const void* d_recs, int64_t n, int stride, int steps, cudaStream_t st) {
    for (int k = 0; k < steps; k++) {
        G->step += 1;
        AdamStep A;
        A.w32 = G->w32.as<float>();
        A.image = G->image.as<unsigned char>();
        A.m = G->m.as<float>();
        A.v = G->v.as<float>();
        A.lr = G->cfg.learning_rate;
        A.b1 = 0.9f;
        A.b2 = 0.999f;
        A.c1 = 1.f - std::pow(A.b1, (float)G->step);
        A.c2 = 1.f - std::pow(A.b2, (float)G->step);
        A.eps = 1e-8f;
        launch_batch(G, d_recs, n, stride, st, k == 0, &A, k + 1 < steps);
    }
}

void guide_step(dl_guide* G, const void* d_recs, int64_t n, int stride, cudaStream_t st) {
    guide_steps(G, d_recs, n, stride, 1, st);
}

// Train on `n` device records: `steps` Adam steps over the same batch.
float guide_train(dl_guide* G, const void* d_recs, int64_t n, int steps) {
    cudaStream_t st = G->ctx->stream;
    float loss = 0.f;
    guide_reserve(G, n);
    guide_steps(G, d_recs, n, 1, steps, st);
    if (steps > 0) {
        DL_CUDA(cudaMemcpyAsync(&loss, G->scratch.as<float>() + 1, 4, cudaMemcpyDeviceToHost, st));
        DL_CUDA(cudaStreamSynchronize(st));
    }
    return loss;
}

// Blocks of k_guide_infer resident at once on one SM, from its registers and
// shared memory; a context's first call raises the kernel's shared-memory limit.
static int infer_blocks_per_sm() {
    DL_CUDA(cudaFuncSetAttribute(k_guide_infer, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(InferSmem)));
    DL_CUDA(cudaFuncSetAttribute(k_guide_infer, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    int dev = 0;
    DL_CUDA(cudaGetDevice(&dev));
    cudaDeviceProp prop;
    DL_CUDA(cudaGetDeviceProperties(&prop, dev));
    cudaFuncAttributes fa;
    DL_CUDA(cudaFuncGetAttributes(&fa, k_guide_infer));
    const int regs_per_warp = ((fa.numRegs + 7) / 8) * 8 * 32;
    const int by_regs = prop.regsPerMultiprocessor / std::max(1, regs_per_warp * (kInferThreads / 32));
    const size_t smem = sizeof(InferSmem) + fa.sharedSizeBytes + prop.reservedSharedMemPerBlock;
    return std::max(1, std::min(by_regs, (int)(prop.sharedMemPerMultiprocessor / smem)));
}

void guide_forward(dl_guide* G, const float* d_in, float* d_out, int64_t n) {
    int& per_sm = G->ctx->infer_per_sm;
    if (per_sm == 0) per_sm = infer_blocks_per_sm();
    cudaStream_t st = G->ctx->stream;
    unsigned* err = reinterpret_cast<unsigned*>(G->scratch.as<char>() + kGuideErrOffset);
    DL_CUDA(cudaMemsetAsync(err, 0, sizeof(unsigned), st));
    const int64_t ntiles = (n + kTcRows - 1) / kTcRows;
    const int blocks =
        (int)std::min<int64_t>((ntiles + kInferGroups - 1) / kInferGroups, (int64_t)G->ctx->num_sms * per_sm);
    k_guide_infer<<<blocks, kInferThreads, sizeof(InferSmem), st>>>(G->image.ptr, d_in, d_out, (int)n, err);
    DL_CUDA(cudaGetLastError());
}

}  // namespace dl
