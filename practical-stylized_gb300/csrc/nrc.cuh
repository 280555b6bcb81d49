// nrc.cuh -- neural radiance cache: shared definitions of the FP32 and BF16 (tcgen05) paths.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"
#include "fastmod.h"

namespace sty {

constexpr int kNrcWidth = 64;      // hidden width and encoded input width
constexpr int kNrcMaxLayers = 8;   // hidden layers supported
constexpr int kNrcOutPad = 16;     // output rows padded to one MMA N tile

struct NrcNet {
    int in_dims, out_dims, layers;     // layers = hidden layers; weight matrices = layers + 1
    uint32_t freqs[STY_NRC_MAX_INPUTS];
};

// offsets (floats) of the weight matrices in the flat FP32 parameter vector:
// layer l < layers: [64 out][64 in]; output layer: [out_dims][64]
__host__ __device__ inline size_t nrc_w_offset(int l) { return (size_t)l * kNrcWidth * kNrcWidth; }
__host__ __device__ inline size_t nrc_param_count(const NrcNet &n) {
    return (size_t)n.layers * kNrcWidth * kNrcWidth + (size_t)n.out_dims * kNrcWidth;
}

// Frequency encoding of one sample: dim d contributes sin(2^k pi x), cos(2^k pi x), k < freqs[d],
// in order (d, k, sin, cos); the tail up to 64 is zero. One sincosf per dim, higher octaves by the
// double-angle identities sin 2a = 2 sin a cos a, cos 2a = 1 - 2 sin^2 a.
__device__ __forceinline__ void nrc_encode(const NrcNet &n, const float *x, float enc[kNrcWidth]) {
    int o = 0;
#pragma unroll 1
    for (int d = 0; d < n.in_dims; d++) {
        float s, c;
        sincospif(x[d], &s, &c);
        for (uint32_t k = 0; k < n.freqs[d]; k++) {
            enc[o] = s;
            enc[o + 1] = c;
            o += 2;
            const float s2 = 2.0f * s * c;
            c = fmaf(-2.0f * s, s, 1.0f);
            s = s2;
        }
    }
    for (; o < kNrcWidth; o++) enc[o] = 0.0f;
}

// The frequency table of the neural-cache workload network (11 inputs, octaves 4,4,4,3,3,3,3,2,2,2,2 -> 64
// columns) fixed at compile time: columns 32 HALF .. 32 HALF + 31 of nrc_encode, every column in a static
// register, no per-pair branch or table lookup. x holds the inputs the half needs: 0 .. 4, or 4 .. 10 (input
// 4's octaves lie in both halves).
constexpr int kNrcC4Half = 7;
constexpr int kNrcC4Dims = 11;
__device__ constexpr int kNrcC4Freqs[kNrcC4Dims] = {4, 4, 4, 3, 3, 3, 3, 2, 2, 2, 2};
inline bool nrc_is_c4(const NrcNet &n) {
    const int f[kNrcC4Dims] = {4, 4, 4, 3, 3, 3, 3, 2, 2, 2, 2};
    if (n.in_dims != kNrcC4Dims) return false;
    for (int d = 0; d < kNrcC4Dims; d++)
        if ((int)n.freqs[d] != f[d]) return false;
    return true;
}
template <int HALF>
__device__ __forceinline__ void nrc_encode_c4(const float (&x)[kNrcC4Half], float (&enc)[32]) {
    int o = 0;  // pairs before dim d
#pragma unroll
    for (int d = 0; d < kNrcC4Dims; d++) {
        if (o < 16 * HALF + 16 && o + kNrcC4Freqs[d] > 16 * HALF) {
            float s, c;
            sincospif(x[d - 4 * HALF], &s, &c);
#pragma unroll
            for (int k = 0; k < kNrcC4Freqs[d]; k++) {
                const int p = o + k - 16 * HALF;
                if (p >= 0 && p < 16) {
                    enc[2 * p] = s;
                    enc[2 * p + 1] = c;
                }
                const float s2 = 2.0f * s * c;
                c = fmaf(-2.0f * s, s, 1.0f);
                s = s2;
            }
        }
        o += kNrcC4Freqs[d];
    }
}

// The rows of a training batch: sample b is row `index(b)` of input / target. A sampled batch draws its rows
// uniformly from `count` (collect_batch, akari_tcnn.cu:15-38: one Pcg32 stream per sample of the run, number
// base + b); an explicit one takes them in order. The training kernels gather by it themselves: the copy of
// the batch it replaces was a launch and 5 to 8 us.
__device__ __forceinline__ uint32_t nrc_pcg_step(uint64_t &state, uint64_t inc) {
    const uint64_t old = state;
    state = old * 0x5851f42d4c957f2dULL + inc;
    const uint32_t xs = (uint32_t)(((old >> 18) ^ old) >> 27);
    const uint32_t rot = (uint32_t)(old >> 59);
    return (xs >> rot) | (xs << ((~rot + 1u) & 31u));
}
struct NrcRows {
    const float *input, *target;
    bool sampled;
    uint64_t seed, base, count, magic;  // magic = fastmod_magic(count): r % count without a 64-bit division
    __device__ __forceinline__ uint64_t index(uint32_t b) const {
        if (!sampled) return b;
        uint64_t st = 0;
        const uint64_t inc = ((base + b) << 1) | 1ull;
        nrc_pcg_step(st, inc);
        st += seed;
        nrc_pcg_step(st, inc);
        const uint64_t hi = nrc_pcg_step(st, inc);
        return fastmod((hi << 32) | nrc_pcg_step(st, inc), count, magic);
    }
};

// BF16 tensor-core path (nrc_tc.cu)
struct NrcTcWeights;  // device buffers in the UMMA shared-memory image layout
sty_status nrc_tc_pack(const NrcNet &n, const float *w_fp32, uint16_t *w_img, cudaStream_t st);
size_t nrc_tc_image_elems(const NrcNet &n);
sty_status nrc_tc_forward(const NrcNet &n, const uint16_t *w_img, uint64_t count, const float *input, float *output,
                          cudaStream_t st);
// Fused BF16 training step (forward, relative-L2 gradient, backward, weight gradient) over a batch
// of B samples on `ctas` CTAs (nrc_tc_train_ctas); per-CTA gradient sums go to part[ctas][np].
constexpr int kNrcTcTrainMaxLayers = 6;
uint32_t nrc_tc_train_ctas(uint32_t B);
sty_status nrc_tc_train(const NrcNet &n, const uint16_t *w_img, uint32_t B, const NrcRows &rows, float *part, size_t np, float *loss, uint32_t ctas, cudaStream_t st);

// BF16 operand image (nrc_tc_pack) of parameter i for the value v: per layer a K-major image, the output
// layer's behind the hidden ones
__device__ __forceinline__ void nrc_store_bf16(uint16_t *img, size_t i, float v) {
    const uint32_t e = (uint32_t)(i & (kNrcWidth * kNrcWidth - 1)), row = e / kNrcWidth, k = e % kNrcWidth;
    img[(i - e) + ((row >> 3) * 8u + (k >> 3)) * 64u + (row & 7u) * 8u + (k & 7u)] =
        __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// FP32 inference on the tensor cores (nrc_f32tc.cu): the hidden layers' weights as three BF16 pieces,
// per layer three K-major operand images of 64 x 64. The pieces sum to w (1 + kNrcUnbias): tcgen05
// truncates its accumulations, which takes ~0.7 x 2^-24 off a layer's outputs on average, and the
// third piece, whose last place is 2^-25 of w, gives it back:
// without it the outputs of a 5 x 64 network were 2.0e-7 too small on average, with it 1e-8 too large,
// and |mean| <= 3e-8 over 1 to 8 layers (a property of this chip's accumulators, not of the network: tests hold it to
// 1e-7 at other weights).
constexpr float kNrcUnbias = 4.2e-8f;
size_t nrc_f32tc_image_elems(const NrcNet &n);
// piece images of hidden weight i (flat parameter index, < layers * 64 * 64) for the value v
__device__ __forceinline__ void nrc_store_pieces(uint16_t *img, size_t i, float v) {
    const uint32_t e = (uint32_t)(i & (kNrcWidth * kNrcWidth - 1)), row = e / kNrcWidth, k = e % kNrcWidth;
    uint16_t *dst = img + (i - e) * 3 + ((row >> 3) * 8u + (k >> 3)) * 64u + (row & 7u) * 8u + (k & 7u);
    float r = v;
#pragma unroll
    for (int p = 0; p < 3; p++) {
        const __nv_bfloat16 b = __float2bfloat16_rn(r);
        dst[p * kNrcWidth * kNrcWidth] = __bfloat16_as_ushort(b);
        r -= __bfloat162float(b);
        if (p == 1) r = fmaf(v, kNrcUnbias, r);
    }
}
// Where a piece or a sum could leave FP32's range the pieces do not add up (the first one of an infinity leaves a NaN behind
// it), so a network that holds a weight past this bound, or a NaN, is run row by row on the CUDA cores: with every weight
// of L + 1 matrices within it, each matrix multiplies the range of |activations| <= 1 by at most 64 times it, 2^120 in all.
// `wide` counts such weights; whoever writes a parameter keeps the count.
inline float nrc_wide_bound(const NrcNet &n) { return exp2f(120.0f / (float)(n.layers + 1) - 6.0f); }
__device__ __forceinline__ bool nrc_is_wide(float v, float bound) { return !(fabsf(v) <= bound); }
sty_status nrc_f32tc_pack(const NrcNet &n, const float *w, uint16_t *img, uint32_t *wide, cudaStream_t st);
sty_status nrc_f32tc_forward(const NrcNet &n, const float *w, const uint16_t *img, const uint32_t *wide, uint64_t count,
                             const float *input, float *output, cudaStream_t st);
// The reference's composite-encoding network (nrc_grid.cu)
struct GridModel;
sty_status grid_create(const sty_nrc_grid_config *c, GridModel **out, size_t *n_params, size_t *n_mlp);
void grid_destroy(GridModel *g);
sty_status grid_init_params(GridModel *g, uint64_t seed, float *w, cudaStream_t st);
sty_status grid_pack(GridModel *g, const float *w, const float *ema, cudaStream_t st);
// inference with the EMA or the current parameters (packed by grid_pack with both sets); the
// tensor-core path (tile encoder + MMA kernel) when the network fits it and allow_tc, else the
// layer-by-layer path on the tcgen05 row GEMMs (gemm_tc.cu)
sty_status grid_infer(GridModel *g, bool ema, bool allow_tc, uint64_t count, const float *in, float *out,
                      cudaStream_t st);
// the optimiser step (tiny-cuda-nn's Adam: sparse over the tables, per-entry step counts) and the EMA;
// keeps the FP16 table copy current
sty_status grid_adam(GridModel *g, float *w, float *m, float *v, const float *grad, float *ema, float lr, float b1,
                     float b2, float eps, float bc1, float bc2, float ema_decay, float ema_old, float ema_new,
                     cudaStream_t st);
// the parameters were overwritten outside the optimiser (load): the FP16 table copy is stale
void grid_params_changed(GridModel *g);
// zero the tables' per-entry Adam step counts (optimiser reset)
sty_status grid_reset_steps(GridModel *g);
// loss and full parameter gradient of B rows with the current parameters (packed by grid_pack)
sty_status grid_gradient(GridModel *g, uint32_t B, const float *x, const float *target, float *grad, float *loss,
                         cudaStream_t st);

}  // namespace sty
