// nrc.cu -- neural radiance cache: host object, FP32 training on the CUDA cores, loss, Adam / EMA,
// sampling.
//
// The object mirrors `struct NRC` of crates/akari_cpp_ext/cpp_ext/akari_tcnn.cu:84-248: it owns the
// weights, the optimiser state and its scratch; the caller owns the input / output / target
// matrices. Unlike the reference, no call synchronises the device unless documented.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "nrc.cuh"

namespace sty {
namespace {

constexpr int W = kNrcWidth;

// ---- FP32 training forward, register-tiled --------------------------------------------------
// One persistent CTA per SM: every hidden layer's weights transposed into shared memory once
// (wt[l][k][j] = W_l[j][k]), the output layer as stored. Two groups of 256 threads each walk their
// own tiles of FT samples (named barrier per group), each with two activation buffers [64 k][FT + 4]
// (k-major; the padding puts consecutive rows 16 bytes apart in bank order). Thread (ty, tx) =
// (t / 16, t % 16) of a group computes FT / 16 samples x outputs 4 tx .. 4 tx + 3, two samples to a
// packed FMA: at FT = 128 two 16-byte activation loads and one 16-byte weight load feed 32 FMAs per k.
// FT: 64 where 128-sample tiles would leave SMs or groups idle (f32_gradient).
// Every output is summed over k = 0 .. 63 in order with fmaf, so both tile sizes agree bit for bit.
template <int FT>
constexpr int tile_pitch() { return FT + 4; }
template <int FT>
__host__ __device__ inline size_t fwd_tiled_floats(const NrcNet &n) {
    return (size_t)n.layers * W * W + (size_t)((n.out_dims * W + 3) & ~3) + 4 * (size_t)W * tile_pitch<FT>();
}
// acc[i][j] += w[j] * v[2 i .. 2 i + 1] over FT / 16 samples, v at `p`
template <int FT>
__device__ __forceinline__ void fma_rows(float2 (&acc)[FT / 32][4], const float *p, const float4 &w4) {
    float2 v[FT / 32];
#pragma unroll
    for (int i = 0; i < FT / 32; i += 2) {
        const float4 q = *reinterpret_cast<const float4 *>(p + 2 * i);
        v[i] = make_float2(q.x, q.y);
        v[i + 1] = make_float2(q.z, q.w);
    }
    const float wv[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
    for (int i = 0; i < FT / 32; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = make_float2(fmaf(wv[j], v[i].x, acc[i][j].x), fmaf(wv[j], v[i].y, acc[i][j].y));
}
// thread (ty, tx)'s sums as rows 4 tx + j of a k-major buffer
template <int FT>
__device__ __forceinline__ void store_cols(float *buf, int ty, int tx, const float2 (&acc)[FT / 32][4]) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        float *dst = buf + (4 * tx + j) * tile_pitch<FT>() + FT / 16 * ty;
#pragma unroll
        for (int i = 0; i < FT / 32; i += 2)
            *reinterpret_cast<float4 *>(dst + 2 * i) = make_float4(acc[i][j].x, acc[i][j].y, acc[i + 1][j].x, acc[i + 1][j].y);
    }
}
template <int FT>
__global__ void __launch_bounds__(512, 1) k_fwd_f32_tiled(NrcNet n, int c4, const float *__restrict__ wg, uint32_t count,
                                                          const NrcRows rows, float *__restrict__ output,
                                                          float *__restrict__ acts) {
    extern __shared__ __align__(16) float sm[];
    constexpr int FP = tile_pitch<FT>(), NS = FT / 16;
    const int L = n.layers, O = n.out_dims;
    float *wt = sm;
    float *wo = wt + (size_t)L * W * W;
    const int grp = threadIdx.x >> 8, tid = threadIdx.x & 255;
    float *buf0 = wo + ((O * W + 3) & ~3) + (size_t)grp * 2 * W * FP;
    float *buf1 = buf0 + W * FP;
    for (int e = threadIdx.x; e < L * W * W / 4; e += 512) {  // neighbouring threads take neighbouring rows j: no bank conflicts
        const int l = e / (W * W / 4), j = e % W, k = e / W % (W / 4) * 4;
        const float4 v = *reinterpret_cast<const float4 *>(wg + nrc_w_offset(l) + (size_t)j * W + k);
        float *dst = wt + (size_t)l * W * W + k * W + j;
        dst[0] = v.x;
        dst[W] = v.y;
        dst[2 * W] = v.z;
        dst[3 * W] = v.w;
    }
    for (int e = threadIdx.x; e < O * W; e += 512) wo[e] = wg[nrc_w_offset(L) + e];
    __syncthreads();
    auto group_sync = [&]() { asm volatile("bar.sync %0, 256;" ::"r"(1 + grp) : "memory"); };
    const int ty = tid >> 4, tx = tid & 15;
    const uint64_t ntiles = (count + FT - 1) / FT;
    for (uint64_t tile = blockIdx.x + (uint64_t)gridDim.x * grp; tile < ntiles; tile += 2 * (uint64_t)gridDim.x) {
        const uint64_t s0 = tile * FT;
        if (c4) {  // encode into buf0[k][sample]: two threads per sample, 32 columns each
            if (tid < 2 * FT) {
                const int r = tid % FT, half = tid / FT;
                const uint64_t i = s0 + r;
                const float *src = rows.input + (i < count ? rows.index((uint32_t)i) : 0) * kNrcC4Dims + 4 * half;
                float x[kNrcC4Half], enc[32];
#pragma unroll
                for (int d = 0; d < kNrcC4Half; d++) x[d] = i < count && (half == 1 || d < 5) ? src[d] : 0.0f;
                if (half == 0)
                    nrc_encode_c4<0>(x, enc);
                else
                    nrc_encode_c4<1>(x, enc);
#pragma unroll
                for (int k = 0; k < 32; k++) buf0[(32 * half + k) * FP + r] = i < count ? enc[k] : 0.0f;
                if (i < count)
#pragma unroll
                    for (int k = 0; k < 32; k += 4)
                        *reinterpret_cast<float4 *>(acts + i * W + 32 * half + k) =
                            make_float4(enc[k], enc[k + 1], enc[k + 2], enc[k + 3]);
            }
        } else if (tid < FT) {
            const uint64_t i = s0 + tid;
            float enc[W];
            if (i < count) {
                nrc_encode(n, rows.input + rows.index((uint32_t)i) * n.in_dims, enc);
            } else {
#pragma unroll
                for (int k = 0; k < W; k++) enc[k] = 0.0f;
            }
#pragma unroll
            for (int k = 0; k < W; k++) buf0[k * FP + tid] = enc[k];
            if (i < count)
#pragma unroll
                for (int k = 0; k < W; k += 4)
                    *reinterpret_cast<float4 *>(acts + i * W + k) = make_float4(enc[k], enc[k + 1], enc[k + 2], enc[k + 3]);
        }
        group_sync();
        float *cur = buf0, *nxt = buf1;
        for (int l = 0; l < L; l++) {
            const float *w = wt + (size_t)l * W * W + 4 * tx;
            const float *av = cur + NS * ty;
            float2 acc[FT / 32][4];
#pragma unroll
            for (int i = 0; i < FT / 32; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll 8
            for (int k = 0; k < W; k++) fma_rows<FT>(acc, av + k * FP, *reinterpret_cast<const float4 *>(w + k * W));
#pragma unroll
            for (int i = 0; i < FT / 32; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = make_float2(fmaxf(acc[i][j].x, 0.0f), fmaxf(acc[i][j].y, 0.0f));
            store_cols<FT>(nxt, ty, tx, acc);
#pragma unroll
            for (int i = 0; i < FT / 32; i++) {
                const uint64_t s = s0 + NS * ty + 2 * i;
                float *dst = acts + ((size_t)(l + 1) * count + s) * W + 4 * tx;
                if (s < count) *reinterpret_cast<float4 *>(dst) = make_float4(acc[i][0].x, acc[i][1].x, acc[i][2].x, acc[i][3].x);
                if (s + 1 < count)
                    *reinterpret_cast<float4 *>(dst + W) = make_float4(acc[i][0].y, acc[i][1].y, acc[i][2].y, acc[i][3].y);
            }
            group_sync();
            float *t = cur;
            cur = nxt;
            nxt = t;
        }
        if (tid < FT && s0 + tid < count) {
            for (int c = 0; c < O; c++) {
                float a = 0.0f;
#pragma unroll
                for (int k = 0; k < W; k++) a = fmaf(wo[c * W + k], cur[k * FP + tid], a);
                output[(s0 + tid) * O + c] = a;
            }
        }
        group_sync();  // the next tile's encoding overwrites buf0
    }
}

// dpre: [layers+1][B][64]: row l < layers = dL/d(pre-activation of hidden layer l),
// row `layers` = dL/d(output) (first out_dims entries).
// ---- loss gradient + FP32 backward, register-tiled ------------------------------------------
// The same persistent layout as k_fwd_f32_tiled: the weights as stored ([j][k]: for a summed row j
// the outputs k are contiguous), two groups of 256 threads on their own tiles of FT samples, thread
// (ty, tx) holding FT / 16 samples x units 4 tx .. 4 tx + 3. Per tile: the relative-L2 gradient g of
// each sample, dH = W_out^T g, then per hidden layer l (last first) dP_l = dH where act_{l+1} > 0 (to
// dpre and to a k-major buffer) and dH = W_l^T dP_l. Every sum runs over its index in order with fmaf, so
// dpre is bit-identical at both tile sizes.
template <int FT>
__host__ __device__ inline size_t bwd_tiled_floats(const NrcNet &n) {
    return (size_t)n.layers * W * W + (size_t)((n.out_dims * W + 3) & ~3) +
           2 * ((size_t)W * tile_pitch<FT>() + kNrcOutPad * FT);
}
template <int FT>
__global__ void __launch_bounds__(512, 1) k_bwd_f32_tiled(NrcNet n, const float *__restrict__ wg, uint32_t B,
                                                          const float *__restrict__ pred, const NrcRows rows,
                                                          const float *__restrict__ acts, float *__restrict__ dpre,
                                                          float *__restrict__ loss_acc) {
    extern __shared__ __align__(16) float sm[];
    constexpr int FP = tile_pitch<FT>(), NS = FT / 16;
    const int L = n.layers, O = n.out_dims;
    float *ws = sm;                              // [L][64 j][64 k] as stored
    float *wo = ws + (size_t)L * W * W;          // [O][64]
    const int grp = threadIdx.x >> 8, tid = threadIdx.x & 255;
    float *dpb = wo + ((O * W + 3) & ~3) + (size_t)grp * ((size_t)W * FP + kNrcOutPad * FT);  // [64 j][FP]
    float *gb = dpb + W * FP;                    // [O][FT]: the loss gradient, k-major
    for (size_t e = threadIdx.x * 4; e < nrc_param_count(n); e += 512 * 4)
        *reinterpret_cast<float4 *>(ws + e) = *reinterpret_cast<const float4 *>(wg + e);
    __syncthreads();
    auto group_sync = [&]() { asm volatile("bar.sync %0, 256;" ::"r"(1 + grp) : "memory"); };
    const int ty = tid >> 4, tx = tid & 15;
    const float norm = 1.0f / ((float)B * (float)O);
    float lsum = 0.0f;
    const uint32_t ntiles = (B + FT - 1) / FT;
    for (uint32_t tile = blockIdx.x + gridDim.x * grp; tile < ntiles; tile += 2 * gridDim.x) {
        const uint32_t s0 = tile * FT;
        if (tid < FT) {
            const uint32_t i = s0 + tid;
            const float *target = rows.target + (i < B ? rows.index(i) : 0) * O;
            for (int c = 0; c < O; c++) {
                float g = 0.0f;
                if (i < B) {
                    const float p = pred[(size_t)i * O + c], t = target[c];
                    const float den = p * p + 0.01f;  // relative L2, prediction treated as constant below
                    lsum += (p - t) * (p - t) / den;
                    g = 2.0f * (p - t) / den * norm;
                    dpre[((size_t)L * B + i) * W + c] = g;
                }
                gb[c * FT + tid] = g;
            }
        }
        group_sync();
        // dH = W_out^T g
        float2 acc[FT / 32][4];
#pragma unroll
        for (int i = 0; i < FT / 32; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = make_float2(0.0f, 0.0f);
        for (int c = 0; c < O; c++)
            fma_rows<FT>(acc, gb + c * FT + NS * ty, *reinterpret_cast<const float4 *>(wo + c * W + 4 * tx));
        for (int l = L - 1; l >= 0; l--) {
            // dP_l = dH where act_{l+1} > 0 -> dpre and dpb[j][sample]
#pragma unroll
            for (int i = 0; i < FT / 32; i++) {
                const uint32_t s = s0 + NS * ty + 2 * i;
                float4 h0 = make_float4(0.f, 0.f, 0.f, 0.f), h1 = h0;
                const float *src = acts + ((size_t)(l + 1) * B + s) * W + 4 * tx;
                if (s < B) h0 = *reinterpret_cast<const float4 *>(src);
                if (s + 1 < B) h1 = *reinterpret_cast<const float4 *>(src + W);
                acc[i][0] = make_float2(h0.x > 0.0f ? acc[i][0].x : 0.0f, h1.x > 0.0f ? acc[i][0].y : 0.0f);
                acc[i][1] = make_float2(h0.y > 0.0f ? acc[i][1].x : 0.0f, h1.y > 0.0f ? acc[i][1].y : 0.0f);
                acc[i][2] = make_float2(h0.z > 0.0f ? acc[i][2].x : 0.0f, h1.z > 0.0f ? acc[i][2].y : 0.0f);
                acc[i][3] = make_float2(h0.w > 0.0f ? acc[i][3].x : 0.0f, h1.w > 0.0f ? acc[i][3].y : 0.0f);
                float *dst = dpre + ((size_t)l * B + s) * W + 4 * tx;
                if (s < B) *reinterpret_cast<float4 *>(dst) = make_float4(acc[i][0].x, acc[i][1].x, acc[i][2].x, acc[i][3].x);
                if (s + 1 < B)
                    *reinterpret_cast<float4 *>(dst + W) = make_float4(acc[i][0].y, acc[i][1].y, acc[i][2].y, acc[i][3].y);
            }
            if (l == 0) break;
            group_sync();  // the previous layer's dpb reads are done
            store_cols<FT>(dpb, ty, tx, acc);
            group_sync();
            // dH = W_l^T dP_l: dH[k] = sum_j W_l[j][k] dP_l[j]
            const float *w = ws + nrc_w_offset(l) + 4 * tx;
            const float *dv = dpb + NS * ty;
#pragma unroll
            for (int i = 0; i < FT / 32; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll 8
            for (int j = 0; j < W; j++) fma_rows<FT>(acc, dv + j * FP, *reinterpret_cast<const float4 *>(w + j * W));
        }
        group_sync();  // the next tile overwrites gb and dpb
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if ((threadIdx.x & 31) == 0 && loss_acc && lsum != 0.0f) atomicAdd(loss_acc, lsum / ((float)B * (float)O));
}

// ---- weight gradient: grad_l[j][k] = sum_i dpre_l[i][j] * acts_l[i][k] ----------------------
// Grid (chunks of kWgChunk samples, layers + 1, 4 quadrants of 32 x 32 outputs), 64 threads, thread
// (ty, tx) = (t / 8, t % 8) owning 4 x 4 outputs as packed pairs over k: per sample two 16-byte
// shared-memory loads feed 16 FMAs. The samples' rows arrive 32 at a time by cp.async, five groups
// ahead (two ahead left the block waiting for them: 34 us). Each chunk stores its partial sums at part + chunk * np; k_sum_chunks adds the chunks in
// order, so the gradient does not depend on scheduling. Every output is summed over the chunk's
// samples in order with fmaf(dpre, act, acc) (samples past the batch add fmaf(0, 0, acc)): the
// quadrants give the partials of one block per chunk and layer bit for bit, but a 2^14 batch of a
// 5-layer network is 336 blocks instead of 96 on 152 SMs (32 us, 43 before).
constexpr int kWgChunk = 1024;
constexpr int kWgRows = 32, kWgStages = 6;
__global__ void __launch_bounds__(64) k_wgrad_f32(NrcNet n, uint32_t B, const float *__restrict__ acts,
                                                  const float *__restrict__ dpre, size_t np,
                                                  float *__restrict__ part) {
    __shared__ __align__(16) float st[kWgStages][2][kWgRows][32];  // dpre and activation columns of 32 samples
    const int l = blockIdx.y, j0 = (blockIdx.z >> 1) * 32, k0 = (blockIdx.z & 1) * 32;
    const int rows = l < n.layers ? W : n.out_dims;
    if (j0 >= rows) return;
    const uint32_t i0 = blockIdx.x * kWgChunk, i1 = min(B, i0 + kWgChunk);
    const int ty = threadIdx.x >> 3, tx = threadIdx.x & 7;
    const float *src[2] = {dpre + (size_t)l * B * W + j0, acts + (size_t)l * B * W + k0};
    const uint32_t groups = (i1 - i0 + kWgRows - 1) / kWgRows;
    auto fetch = [&](uint32_t g) {
        if (g < groups) {
#pragma unroll
            for (int u = 0; u < 2 * kWgRows * 8 / 64; u++) {
                const int e = threadIdx.x + u * 64, arr = e / (kWgRows * 8), r = e / 8 % kWgRows, c4 = e % 8;
                const uint32_t s = i0 + g * kWgRows + (uint32_t)r;
                const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(&st[g % kWgStages][arr][r][4 * c4]));
                const uint32_t bytes = s < i1 ? 16u : 0u;  // 0: the destination is zero-filled
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst),
                             "l"(src[arr] + (size_t)(s < i1 ? s : i0) * W + 4 * c4), "r"(bytes)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float2 acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i][0] = acc[i][1] = make_float2(0.0f, 0.0f);
    for (uint32_t g = 0; g + 1 < kWgStages; g++) fetch(g);
    for (uint32_t g = 0; g < groups; g++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kWgStages - 2) : "memory");
        __syncthreads();  // group g is in shared memory, and group g - 1 has been read by both warps
        fetch(g + kWgStages - 1);
        const float(*sd)[32] = st[g % kWgStages][0], (*sh)[32] = st[g % kWgStages][1];
#pragma unroll 8
        for (int r = 0; r < kWgRows; r++) {
            const float4 a4 = *reinterpret_cast<const float4 *>(&sd[r][4 * ty]);
            const float4 b4 = *reinterpret_cast<const float4 *>(&sh[r][4 * tx]);
            const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                acc[i][0] = make_float2(fmaf(av[i], b4.x, acc[i][0].x), fmaf(av[i], b4.y, acc[i][0].y));
                acc[i][1] = make_float2(fmaf(av[i], b4.z, acc[i][1].x), fmaf(av[i], b4.w, acc[i][1].y));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int j = j0 + 4 * ty + i;
        if (j < rows)
            *reinterpret_cast<float4 *>(part + blockIdx.x * np + nrc_w_offset(l) + (size_t)j * W + k0 + 4 * tx) =
                make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y);
    }
}

// grad[p] = part[0][p] + part[1][p] + ... in chunk order (one sequential FP32 sum per parameter;
// np is a multiple of 64: layers x 64 x 64 + outputs x 64). A block owns kSumP parameters: its 256
// threads stage a slab of up to kSumC chunk rows into shared memory with 16-byte loads, every load of
// the slab issued before the first store (16 in flight per thread), then kSumP threads continue their
// sums over the slab in order. The 152 per-CTA partials of a tensor-core training step are one slab.
constexpr int kSumP = 64, kSumC = 256, kSumLd = kSumC / (256 / (kSumP / 4));

// ---- Adam + EMA (akari_tcnn.cu:42-83 for the EMA) --------------------------------------------
// img / img_ema: the BF16 operand images of w and ema (BF16 networks), img3 / img3_ema: the piece images of
// the hidden weights (FP32 networks), kept current here; null where the network has none.
struct AdamArgs {
    float *w, *m, *v, *ema;
    float lr, b1, b2, eps, bc1, bc2, ema_decay, ema_old, ema_new;
    size_t n_hidden;
    uint16_t *img, *img_ema, *img3, *img3_ema;
    float wide_bound;  // FP32 networks: the counts of weights past it, wide[0] of w and wide[1] of ema
    uint32_t *wide;
};
__device__ __forceinline__ void adam_step(const AdamArgs &o, size_t p, float gr) {
    const float mm = o.b1 * o.m[p] + (1.0f - o.b1) * gr;
    const float vv = o.b2 * o.v[p] + (1.0f - o.b2) * gr * gr;
    o.m[p] = mm;
    o.v[p] = vv;
    const float w0 = o.w[p], e0 = o.ema[p];
    const float wn = w0 - o.lr * (mm / o.bc1) / (sqrtf(vv / o.bc2) + o.eps);
    o.w[p] = wn;
    const float en = (e0 * o.ema_decay * o.ema_old + wn * (1.0f - o.ema_decay)) * o.ema_new;
    o.ema[p] = en;
    if (o.img) {
        nrc_store_bf16(o.img, p, wn);
        nrc_store_bf16(o.img_ema, p, en);
    }
    if (o.img3 && p < o.n_hidden) {
        nrc_store_pieces(o.img3, p, wn);
        nrc_store_pieces(o.img3_ema, p, en);
    }
    if (o.img3) {
        const int dw = (int)nrc_is_wide(wn, o.wide_bound) - (int)nrc_is_wide(w0, o.wide_bound);
        const int de = (int)nrc_is_wide(en, o.wide_bound) - (int)nrc_is_wide(e0, o.wide_bound);
        if (dw) atomicAdd(o.wide, (uint32_t)dw);
        if (de) atomicAdd(o.wide + 1, (uint32_t)de);
    }
}

// OPT: the summed gradient goes straight into the optimiser step and not to memory
template <bool OPT>
__global__ void __launch_bounds__(256) k_sum_chunks(size_t np, uint32_t chunks, uint32_t slab_rows,
                                                    const float *__restrict__ part, float *__restrict__ grad,
                                                    const AdamArgs opt) {
    extern __shared__ float4 slab4[];  // [slab_rows][kSumP / 4]
    const float *slab = reinterpret_cast<const float *>(slab4);
    const int t = threadIdx.x, c4 = t % (kSumP / 4), r0 = t / (kSumP / 4);
    const size_t p0 = (size_t)blockIdx.x * kSumP;
    const float4 *src = reinterpret_cast<const float4 *>(part + p0) + c4;
    const size_t row4 = np / 4;
    float s = 0.0f;
    for (uint32_t c0 = 0; c0 < chunks; c0 += slab_rows) {
        const uint32_t nc = min(slab_rows, chunks - c0);
        float4 v[kSumLd];
#pragma unroll
        for (int j = 0; j < kSumLd; j++) {
            const uint32_t r = (uint32_t)r0 + (uint32_t)j * (256 / (kSumP / 4));
            if (r < nc) v[j] = src[(size_t)(c0 + r) * row4];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kSumLd; j++) {
            const uint32_t r = (uint32_t)r0 + (uint32_t)j * (256 / (kSumP / 4));
            if (r < nc) slab4[r * (kSumP / 4) + c4] = v[j];
        }
        __syncthreads();
        if (t < kSumP)
            for (uint32_t r = 0; r < nc; r++) s += slab[r * kSumP + t];
    }
    if (t < kSumP && p0 + (size_t)t < np) {
        if (OPT)
            adam_step(opt, p0 + t, s);
        else
            grad[p0 + t] = s;
    }
}
template <bool OPT>
sty_status sum_chunks(size_t np, uint32_t chunks, const float *part, float *grad, const AdamArgs &opt, cudaStream_t st) {
    const uint32_t rows = chunks < (uint32_t)kSumC ? (chunks > 0 ? chunks : 1u) : (uint32_t)kSumC;
    const size_t smem = rows * kSumP * sizeof(float);
    if (smem > 48 * 1024)  // beyond the default dynamic shared-memory limit
        STY_TRY(check_cuda(cudaFuncSetAttribute(k_sum_chunks<OPT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)(kSumC * kSumP * 4)),
                           "attr k_sum_chunks"));
    k_sum_chunks<OPT><<<(unsigned)((np + kSumP - 1) / kSumP), 256, smem, st>>>(np, chunks, rows, part, grad, opt);
    return check_launch("k_sum_chunks");
}

// ---- batch sampling into the batch buffers (grid networks; the others gather in their kernels) ----
__global__ void k_collect(uint32_t B, const NrcRows rows, int in_dims, int out_dims, float *__restrict__ bin,
                          float *__restrict__ btg) {
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B) return;
    const uint64_t idx = rows.index(b);
    // the row's loads in batches of 8 before their stores, so the random-row latency is paid once
    // per batch, not once per value
    const float *src = rows.input + idx * in_dims;
    float *dst = bin + (size_t)b * in_dims;
    for (int d0 = 0; d0 < in_dims; d0 += 8) {
        float v[8];
#pragma unroll
        for (int d = 0; d < 8; d++) v[d] = d0 + d < in_dims ? src[d0 + d] : 0.0f;
#pragma unroll
        for (int d = 0; d < 8; d++)
            if (d0 + d < in_dims) dst[d0 + d] = v[d];
    }
    float u[kNrcOutPad];
#pragma unroll
    for (int c = 0; c < kNrcOutPad; c++) u[c] = c < out_dims ? rows.target[idx * out_dims + c] : 0.0f;
#pragma unroll
    for (int c = 0; c < kNrcOutPad; c++)
        if (c < out_dims) btg[(size_t)b * out_dims + c] = u[c];
}

__global__ void k_init_weights(size_t np, NrcNet n, uint64_t seed, float *w) {
    const size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (p >= np) return;
    uint64_t st = 0, inc = ((uint64_t)p << 1) | 1ull;
    nrc_pcg_step(st, inc);
    st += seed;
    nrc_pcg_step(st, inc);
    const float u = (float)nrc_pcg_step(st, inc) * (1.0f / 4294967296.0f);
    const size_t hid = (size_t)n.layers * W * W;
    const float fan_out = p < hid ? (float)W : (float)n.out_dims;
    const float s = sqrtf(6.0f / ((float)W + fan_out));  // uniform Xavier
    w[p] = (2.0f * u - 1.0f) * s;
}

}  // namespace
}  // namespace sty

using namespace sty;

struct sty_nrc {
    sty_nrc_config cfg;
    NrcNet net;
    size_t np = 0;
    float *w = nullptr, *m = nullptr, *v = nullptr, *g = nullptr, *ema = nullptr;
    // Operand images of w and ema for the tensor cores: BF16 networks img, FP32 networks (inference) img3,
    // the three-piece images. They are written where w and ema are (creation, load, optimiser step), in
    // the same stream, so a call that only reads the network writes nothing.
    uint16_t *img = nullptr, *img_ema = nullptr;
    uint16_t *img3 = nullptr, *img3_ema = nullptr;
    uint32_t *wide = nullptr;  // how many of w's and of ema's parameters are too wide for the pieces (FP32 networks)
    float *bin = nullptr, *btg = nullptr, *bpred = nullptr, *acts = nullptr, *dpre = nullptr, *loss = nullptr;
    float *gpart = nullptr;  // per-chunk weight-gradient partials
    GridModel *grid = nullptr;  // the composite-encoding network (sty_nrc_create_grid), else null
    bool layered = false;       // grid network: STY_NRC_GRID_LAYERED (no tensor-core inference)
    uint32_t bcap = 0;
    uint64_t step = 0;  // optimiser steps taken (Adam t, EMA iteration)
    float lr = 0.0f;
    bool img_dirty = true;  // the grid network's packed operands are older than w / ema
};

namespace sty {
uint32_t nrc_batch_size(const sty_nrc *nr) { return nr->cfg.batch_size; }
uint32_t nrc_input_dims(const sty_nrc *nr) { return nr->cfg.input_dims; }
}  // namespace sty

namespace {

bool tc_training(const sty_nrc *nr) {
    return !nr->grid && nr->cfg.precision == STY_NRC_BF16 && nr->net.layers <= kNrcTcTrainMaxLayers;
}

sty_status ensure_batch(sty_nrc *nr, uint32_t B) {
    if (B <= nr->bcap) return STY_OK;
    void *ptrs[] = {nr->bin, nr->btg, nr->bpred, nr->acts, nr->dpre, nr->gpart};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    nr->bin = nr->btg = nr->bpred = nr->acts = nr->dpre = nr->gpart = nullptr;
    const NrcNet &n = nr->net;
    if (nr->grid) {  // the composite-encoding network: a gathered batch, no partials
        STY_TRY(check_cuda(device_malloc(&nr->bin, (size_t)B * n.in_dims * 4), "alloc batch input"));
        STY_TRY(check_cuda(device_malloc(&nr->btg, (size_t)B * n.out_dims * 4), "alloc batch target"));
    } else {
        if (!tc_training(nr)) {
            STY_TRY(check_cuda(device_malloc(&nr->bpred, (size_t)B * n.out_dims * 4), "alloc batch pred"));
            STY_TRY(check_cuda(device_malloc(&nr->acts, (size_t)(n.layers + 1) * B * kNrcWidth * 4), "alloc activations"));
            STY_TRY(check_cuda(device_malloc(&nr->dpre, (size_t)(n.layers + 1) * B * kNrcWidth * 4), "alloc gradients"));
        }
        size_t chunks = (B + kWgChunk - 1) / kWgChunk;
        if (nr->cfg.precision == STY_NRC_BF16) chunks = std::max<size_t>(chunks, nrc_tc_train_ctas(B));
        STY_TRY(check_cuda(device_malloc(&nr->gpart, chunks * nr->np * 4), "alloc gradient partials"));
    }
    nr->bcap = B;
    return STY_OK;
}

template <int FT>
sty_status f32_tiled(sty_nrc *nr, uint32_t B, const NrcRows &rows, int sms, cudaStream_t st) {
    const NrcNet &n = nr->net;
    const uint32_t ntiles = (B + FT - 1) / FT;
    const unsigned grid = std::min<uint32_t>(ntiles, (uint32_t)sms);  // one group's tile per SM before a second group's
    const size_t fsmem = fwd_tiled_floats<FT>(n) * sizeof(float), bsmem = bwd_tiled_floats<FT>(n) * sizeof(float);
    STY_TRY(check_cuda(cudaFuncSetAttribute(k_fwd_f32_tiled<FT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fsmem),
                       "attr k_fwd_f32_tiled"));
    k_fwd_f32_tiled<FT><<<grid, 512, fsmem, st>>>(n, nrc_is_c4(n) ? 1 : 0, nr->w, B, rows, nr->bpred, nr->acts);
    STY_TRY(check_launch("k_fwd_f32_tiled"));
    STY_TRY(check_cuda(cudaFuncSetAttribute(k_bwd_f32_tiled<FT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsmem),
                       "attr k_bwd_f32_tiled"));
    k_bwd_f32_tiled<FT><<<grid, 512, bsmem, st>>>(n, nr->w, B, nr->bpred, rows, nr->acts, nr->dpre, nr->loss);
    return check_launch("k_bwd_f32_tiled");
}

// Forward, loss gradient, backward and weight gradient of a batch on the CUDA cores: *chunks partials
// in nr->gpart.
sty_status f32_gradient(sty_nrc *nr, uint32_t B, const NrcRows &rows, uint32_t *chunks, cudaStream_t st) {
    const NrcNet &n = nr->net;
    int dev = 0, optin = 0, sms = 0;
    STY_TRY(check_cuda(cudaGetDevice(&dev), "cudaGetDevice"));
    STY_TRY(check_cuda(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev), "attr smem"));
    STY_TRY(check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr SMs"));
    // 128-sample tiles load a weight for twice the FMAs; below a tile per group (2 per SM) 64-sample tiles
    // use twice the SMs: forward + backward of a 2^14 batch 54 us instead of 109 (128 tiles, two to an
    // SM, on 64 SMs). Networks of 6 to 8 layers leave room for 64-sample tiles only.
    const bool fits = std::max(fwd_tiled_floats<128>(n), bwd_tiled_floats<128>(n)) * sizeof(float) <= (size_t)optin;
    if (fits && B > 128u * 2u * (uint32_t)sms)
        STY_TRY(f32_tiled<128>(nr, B, rows, sms, st));
    else
        STY_TRY(f32_tiled<64>(nr, B, rows, sms, st));
    *chunks = (B + kWgChunk - 1) / kWgChunk;
    k_wgrad_f32<<<dim3(*chunks, n.layers + 1, 4), 64, 0, st>>>(n, B, nr->acts, nr->dpre, nr->np, nr->gpart);
    return check_launch("k_wgrad_f32");
}

// Gradient partials of one batch in nr->gpart, *chunks of them to be added in order (loss added to
// nr->loss): the fused BF16 tensor-core step for BF16 caches of at most kNrcTcTrainMaxLayers layers, else
// the FP32 kernels. (Not the grid network's, which has no partials.)
sty_status batch_partials(sty_nrc *nr, uint32_t B, const NrcRows &rows, uint32_t *chunks, cudaStream_t st) {
    if (!tc_training(nr)) return f32_gradient(nr, B, rows, chunks, st);
    *chunks = nrc_tc_train_ctas(B);
    return nrc_tc_train(nr->net, nr->img, B, rows, nr->gpart, nr->np, nr->loss, *chunks, st);
}
sty_status grid_batch_gradient(sty_nrc *nr, uint32_t B, const float *in, const float *target, float *grad, cudaStream_t st) {
    STY_TRY(grid_pack(nr->grid, nr->w, nullptr, st));
    nr->img_dirty = true;
    return grid_gradient(nr->grid, B, in, target, grad, nr->loss, st);
}

// the operand images after w and ema were written outside the optimiser step
sty_status pack_images(sty_nrc *nr, cudaStream_t st) {
    if (nr->img) {
        STY_TRY(nrc_tc_pack(nr->net, nr->w, nr->img, st));
        STY_TRY(nrc_tc_pack(nr->net, nr->ema, nr->img_ema, st));
    }
    if (nr->img3) {
        STY_TRY(nrc_f32tc_pack(nr->net, nr->w, nr->img3, nr->wide, st));
        STY_TRY(nrc_f32tc_pack(nr->net, nr->ema, nr->img3_ema, nr->wide + 1, st));
    }
    return STY_OK;
}

sty_status infer(sty_nrc *nr, bool ema, uint64_t count, const float *in, float *out, cudaStream_t st) {
    if (count == 0) return STY_OK;
    if (nr->grid) {
        if (nr->img_dirty) STY_TRY(grid_pack(nr->grid, nr->w, nr->ema, st));
        nr->img_dirty = false;
        return grid_infer(nr->grid, ema, !nr->layered, count, in, out, st);
    }
    if (nr->cfg.precision == STY_NRC_BF16)
        return nrc_tc_forward(nr->net, ema ? nr->img_ema : nr->img, count, in, out, st);
    return nrc_f32tc_forward(nr->net, ema ? nr->ema : nr->w, ema ? nr->img3_ema : nr->img3, nr->wide + (ema ? 1 : 0), count, in, out,
                             st);
}

void free_nrc(sty_nrc *nr) {
    grid_destroy(nr->grid);
    void *ptrs[] = {nr->w, nr->m, nr->v, nr->g, nr->ema, nr->img, nr->img_ema, nr->bin,
                    nr->btg, nr->bpred, nr->acts, nr->dpre, nr->loss, nr->gpart, nr->img3, nr->img3_ema, nr->wide};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    delete nr;
}

}  // namespace

extern "C" {

sty_status sty_nrc_create(const sty_nrc_config *cfg, sty_nrc **out) {
    clear_error();
    STY_ARG_CHECK(cfg && out, "sty_nrc_create: null argument");
    STY_ARG_CHECK(cfg->input_dims >= 1 && cfg->input_dims <= STY_NRC_MAX_INPUTS, "input_dims must be in [1, 16]");
    STY_ARG_CHECK(cfg->output_dims >= 1 && cfg->output_dims <= (uint32_t)kNrcOutPad, "output_dims must be in [1, 16]");
    STY_ARG_CHECK(cfg->hidden_layers >= 1 && cfg->hidden_layers <= (uint32_t)kNrcMaxLayers,
                  "hidden_layers must be in [1, 8]");
    STY_ARG_CHECK(cfg->batch_size >= 128 && cfg->batch_size % 128 == 0, "batch_size must be a multiple of 128");
    STY_ARG_CHECK(cfg->precision == STY_NRC_FP32 || cfg->precision == STY_NRC_BF16, "unknown precision");
    uint32_t enc = 0;
    for (uint32_t d = 0; d < cfg->input_dims; d++) enc += 2 * cfg->freqs[d];
    STY_ARG_CHECK(enc <= (uint32_t)kNrcWidth, "encoded width %u exceeds 64", enc);
    STY_ARG_CHECK(cfg->decay_interval > 0 && cfg->learning_rate > 0.0f, "decay_interval and learning_rate must be > 0");
    sty_nrc *nr = new sty_nrc();
    nr->cfg = *cfg;
    nr->net.in_dims = (int)cfg->input_dims;
    nr->net.out_dims = (int)cfg->output_dims;
    nr->net.layers = (int)cfg->hidden_layers;
    for (int d = 0; d < STY_NRC_MAX_INPUTS; d++) nr->net.freqs[d] = cfg->freqs[d];
    nr->np = nrc_param_count(nr->net);
    nr->lr = cfg->learning_rate;
    sty_status s = STY_OK;
    auto alloc = [&](void **p, size_t bytes, const char *what) {
        if (s == STY_OK) s = check_cuda(device_malloc(p, bytes), what);
    };
    alloc((void **)&nr->w, nr->np * 4, "alloc weights");
    alloc((void **)&nr->m, nr->np * 4, "alloc adam m");
    alloc((void **)&nr->v, nr->np * 4, "alloc adam v");
    alloc((void **)&nr->ema, nr->np * 4, "alloc ema");
    alloc((void **)&nr->loss, 4, "alloc loss");
    if (cfg->precision == STY_NRC_BF16) {
        alloc((void **)&nr->img, nrc_tc_image_elems(nr->net) * 2, "alloc bf16 image");
        alloc((void **)&nr->img_ema, nrc_tc_image_elems(nr->net) * 2, "alloc bf16 ema image");
    }
    if (cfg->precision == STY_NRC_FP32) {
        alloc((void **)&nr->img3, nrc_f32tc_image_elems(nr->net) * 2, "alloc piece images");
        alloc((void **)&nr->img3_ema, nrc_f32tc_image_elems(nr->net) * 2, "alloc ema piece images");
        alloc((void **)&nr->wide, 8, "alloc wide weights");
    }
    if (s == STY_OK) s = ensure_batch(nr, cfg->batch_size);
    if (s == STY_OK) {
        k_init_weights<<<(unsigned)((nr->np + 255) / 256), 256>>>(nr->np, nr->net, cfg->seed, nr->w);
        s = check_launch("k_init_weights");
    }
    if (s == STY_OK) s = check_cuda(cudaMemcpy(nr->ema, nr->w, nr->np * 4, cudaMemcpyDeviceToDevice), "init ema");
    if (s == STY_OK) s = check_cuda(cudaMemset(nr->m, 0, nr->np * 4), "zero m");
    if (s == STY_OK) s = check_cuda(cudaMemset(nr->v, 0, nr->np * 4), "zero v");
    if (s == STY_OK) s = pack_images(nr, nullptr);
    if (s == STY_OK) s = check_cuda(cudaDeviceSynchronize(), "sty_nrc_create");
    if (s != STY_OK) {
        free_nrc(nr);
        return s;
    }
    *out = nr;
    return STY_OK;
}

sty_status sty_nrc_create_grid(const sty_nrc_grid_config *gc, sty_nrc **out) {
    clear_error();
    STY_ARG_CHECK(gc && out, "sty_nrc_create_grid: null argument");
    STY_ARG_CHECK(gc->batch_size >= 128 && gc->batch_size % 128 == 0, "batch_size must be a multiple of 128");
    STY_ARG_CHECK(gc->decay_interval > 0 && gc->learning_rate > 0.0f, "decay_interval and learning_rate must be > 0");
    STY_ARG_CHECK((gc->flags & ~(STY_NRC_GRID_LAYERED | STY_NRC_GRID_FP16)) == 0, "unknown flags 0x%x", gc->flags);
    sty_nrc *nr = new sty_nrc();
    nr->layered = (gc->flags & STY_NRC_GRID_LAYERED) != 0;
    size_t np = 0, n_mlp = 0;
    sty_status s = grid_create(gc, &nr->grid, &np, &n_mlp);
    if (s != STY_OK) {
        delete nr;
        return s;
    }
    // the fields the shared training loop reads (batch sampling, Adam, decay, EMA)
    sty_nrc_config &c = nr->cfg;
    std::memset(&c, 0, sizeof(c));
    c.input_dims = gc->input_dims;
    c.output_dims = gc->output_dims;
    c.batch_size = gc->batch_size;
    c.hidden_layers = gc->hidden_layers;
    c.precision = STY_NRC_BF16;
    c.learning_rate = gc->learning_rate;
    c.beta1 = gc->beta1;
    c.beta2 = gc->beta2;
    c.epsilon = gc->epsilon;
    c.ema_decay = gc->ema_decay;
    c.decay_base = gc->decay_base;
    c.decay_interval = gc->decay_interval;
    c.seed = gc->seed;
    nr->net.in_dims = (int)gc->input_dims;
    nr->net.out_dims = (int)gc->output_dims;
    nr->net.layers = 1;
    nr->np = np;
    nr->lr = gc->learning_rate;
    auto alloc = [&](void **p, size_t bytes, const char *what) {
        if (s == STY_OK) s = check_cuda(device_malloc(p, bytes), what);
    };
    alloc((void **)&nr->w, np * 4, "alloc parameters");
    alloc((void **)&nr->m, np * 4, "alloc adam m");
    alloc((void **)&nr->v, np * 4, "alloc adam v");
    alloc((void **)&nr->g, np * 4, "alloc grad");
    alloc((void **)&nr->ema, np * 4, "alloc ema");
    alloc((void **)&nr->loss, 4, "alloc loss");
    if (s == STY_OK) s = ensure_batch(nr, gc->batch_size);
    if (s == STY_OK) s = grid_init_params(nr->grid, gc->seed, nr->w, nullptr);
    if (s == STY_OK) s = check_cuda(cudaMemcpy(nr->ema, nr->w, np * 4, cudaMemcpyDeviceToDevice), "init ema");
    if (s == STY_OK) s = check_cuda(cudaMemset(nr->m, 0, np * 4), "zero m");
    if (s == STY_OK) s = check_cuda(cudaMemset(nr->v, 0, np * 4), "zero v");
    if (s == STY_OK) s = check_cuda(cudaDeviceSynchronize(), "sty_nrc_create_grid");
    if (s != STY_OK) {
        free_nrc(nr);
        return s;
    }
    *out = nr;
    return STY_OK;
}

sty_status sty_nrc_destroy(sty_nrc *nr) {
    clear_error();
    if (!nr) return STY_OK;
    cudaDeviceSynchronize();
    free_nrc(nr);
    return STY_OK;
}

sty_status sty_nrc_param_count(sty_nrc *nr, uint64_t *count) {
    clear_error();
    STY_ARG_CHECK(nr && count, "sty_nrc_param_count: null argument");
    *count = nr->np;
    return STY_OK;
}

sty_status sty_nrc_save_params(sty_nrc *nr, float *host) {
    clear_error();
    STY_ARG_CHECK(nr && host, "sty_nrc_save_params: null argument");
    STY_TRY(check_cuda(cudaDeviceSynchronize(), "sync before save"));
    return check_cuda(cudaMemcpy(host, nr->w, nr->np * 4, cudaMemcpyDeviceToHost), "save params");
}

sty_status sty_nrc_load_params(sty_nrc *nr, const float *host) {
    clear_error();
    STY_ARG_CHECK(nr && host, "sty_nrc_load_params: null argument");
    STY_TRY(check_cuda(cudaDeviceSynchronize(), "sync before load"));
    STY_TRY(check_cuda(cudaMemcpy(nr->w, host, nr->np * 4, cudaMemcpyHostToDevice), "load params"));
    STY_TRY(check_cuda(cudaMemcpy(nr->ema, host, nr->np * 4, cudaMemcpyHostToDevice), "load ema"));
    nr->img_dirty = true;
    if (nr->grid) grid_params_changed(nr->grid);
    STY_TRY(pack_images(nr, nullptr));
    return check_cuda(cudaDeviceSynchronize(), "sync after load");
}

sty_status sty_nrc_set_learning_rate(sty_nrc *nr, float lr) {
    clear_error();
    STY_ARG_CHECK(nr && lr > 0.0f, "sty_nrc_set_learning_rate: bad argument");
    nr->lr = lr;
    return STY_OK;
}

sty_status sty_nrc_get_learning_rate(sty_nrc *nr, float *lr) {
    clear_error();
    STY_ARG_CHECK(nr && lr, "sty_nrc_get_learning_rate: null argument");
    *lr = nr->lr;
    return STY_OK;
}

sty_status sty_nrc_reset_optimizer(sty_nrc *nr) {
    clear_error();
    STY_ARG_CHECK(nr, "sty_nrc_reset_optimizer: null nrc");
    STY_TRY(check_cuda(cudaMemset(nr->m, 0, nr->np * 4), "zero m"));
    STY_TRY(check_cuda(cudaMemset(nr->v, 0, nr->np * 4), "zero v"));
    if (nr->grid) STY_TRY(grid_reset_steps(nr->grid));
    nr->step = 0;
    return STY_OK;
}

sty_status sty_nrc_inference(sty_nrc *nr, uint64_t count, const float *in, float *out, void *stream) {
    clear_error();
    STY_ARG_CHECK(nr && (count == 0 || (in && out)), "sty_nrc_inference: null argument");
    return infer(nr, true, count, in, out, as_stream(stream));
}

sty_status sty_nrc_train_inference(sty_nrc *nr, uint64_t count, const float *in, float *out, void *stream) {
    clear_error();
    STY_ARG_CHECK(nr && (count == 0 || (in && out)), "sty_nrc_train_inference: null argument");
    return infer(nr, false, count, in, out, as_stream(stream));
}

sty_status sty_nrc_gradient(sty_nrc *nr, uint32_t B, const float *in, const float *target, float *grad,
                            float *loss_out, void *stream) {
    clear_error();
    STY_ARG_CHECK(nr && in && target && grad && B > 0, "sty_nrc_gradient: bad argument");
    cudaStream_t st = as_stream(stream);
    STY_TRY(ensure_batch(nr, B));
    STY_TRY(check_cuda(cudaMemsetAsync(nr->loss, 0, 4, st), "zero loss"));
    if (nr->grid) {
        // straight into the caller's buffer where its alignment allows the tables' 16-byte atomics
        float *dst = (reinterpret_cast<uintptr_t>(grad) & 15) == 0 ? grad : nr->g;
        STY_TRY(grid_batch_gradient(nr, B, in, target, dst, st));
        if (dst != grad)
            STY_TRY(check_cuda(cudaMemcpyAsync(grad, dst, nr->np * 4, cudaMemcpyDeviceToDevice, st), "copy grad"));
    } else {
        uint32_t chunks = 0;
        STY_TRY(batch_partials(nr, B, NrcRows{in, target, false, 0, 0, 0, 0}, &chunks, st));
        STY_TRY(sum_chunks<false>(nr->np, chunks, nr->gpart, grad, AdamArgs{}, st));
    }
    if (loss_out) {
        STY_TRY(check_cuda(cudaMemcpyAsync(loss_out, nr->loss, 4, cudaMemcpyDeviceToHost, st), "read loss"));
        STY_TRY(check_cuda(cudaStreamSynchronize(st), "sync loss"));
    }
    return STY_OK;
}

sty_status sty_nrc_train(sty_nrc *nr, uint64_t count, uint64_t n_iters, const float *in, const float *target,
                         float *loss_out, void *stream) {
    clear_error();
    STY_ARG_CHECK(nr && in && target && count > 0, "sty_nrc_train: bad argument");
    cudaStream_t st = as_stream(stream);
    const sty_nrc_config &c = nr->cfg;
    const uint32_t B = c.batch_size;
    STY_TRY(check_cuda(cudaMemsetAsync(nr->loss, 0, 4, st), "zero loss"));
    for (uint64_t it = 0; it < n_iters; it++) {
        const NrcRows rows = {in, target, true, c.seed, nr->step * B, count, fastmod_magic(count)};
        uint32_t chunks = 0;
        if (nr->grid) {
            k_collect<<<(B + 255) / 256, 256, 0, st>>>(B, rows, nr->net.in_dims, nr->net.out_dims, nr->bin, nr->btg);
            STY_TRY(check_launch("k_collect"));
            STY_TRY(grid_batch_gradient(nr, B, nr->bin, nr->btg, nr->g, st));
        } else {
            STY_TRY(batch_partials(nr, B, rows, &chunks, st));
        }
        nr->step++;
        const double t = (double)nr->step;
        const float lr_t = nr->lr * (float)std::pow((double)c.decay_base, std::floor((t - 1.0) / c.decay_interval));
        const float bc1 = (float)(1.0 - std::pow((double)c.beta1, t));
        const float bc2 = (float)(1.0 - std::pow((double)c.beta2, t));
        const float ema_old = (float)(1.0 - std::pow((double)c.ema_decay, t - 1.0));
        const float ema_new = (float)(1.0 / (1.0 - std::pow((double)c.ema_decay, t)));
        if (nr->grid) {
            STY_TRY(grid_adam(nr->grid, nr->w, nr->m, nr->v, nr->g, nr->ema, lr_t, c.beta1, c.beta2, c.epsilon, bc1,
                              bc2, c.ema_decay, ema_old, ema_new, st));
            nr->img_dirty = true;
        } else {
            const AdamArgs o = {nr->w, nr->m, nr->v, nr->ema, lr_t, c.beta1, c.beta2, c.epsilon, bc1, bc2, c.ema_decay,
                                ema_old, ema_new, nrc_w_offset(nr->net.layers), nr->img, nr->img_ema, nr->img3, nr->img3_ema,
                                nrc_wide_bound(nr->net), nr->wide};
            STY_TRY(sum_chunks<true>(nr->np, chunks, nr->gpart, nullptr, o, st));
        }
    }
    if (loss_out) {
        float l = 0.0f;
        STY_TRY(check_cuda(cudaMemcpyAsync(&l, nr->loss, 4, cudaMemcpyDeviceToHost, st), "read loss"));
        STY_TRY(check_cuda(cudaStreamSynchronize(st), "sync loss"));
        *loss_out = n_iters ? l / (float)n_iters : 0.0f;
    }
    return STY_OK;
}

}  // extern "C"
