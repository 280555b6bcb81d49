// nrc_f32tc.cu -- the FP32 network of the radiance cache with its layer products on the tensor cores.
//
// Every FP32 operand is split into three BF16 pieces, x = x1 + x2 + x3 (round to nearest, each piece the
// rounding of what the ones before leave: 3 x 8 bits are FP32's 24, so the split is exact), and a
// product a.w is the six piece products down to 2^-24 of it: a1w1, a1w2, a2w1, a2w2, a1w3, a3w1, each
// exact, summed by tcgen05.mma into FP32 accumulators in TMEM. An accumulation truncates, so what
// counts is how often a sum is cut at the result's magnitude: the small products go first, and
// the four K steps of a1w1 are shared between the two accumulators, two cuts each (error of the outputs in the
// 2-norm, relative, against FP64 for one 5 x 64 network: 3.5e-7 with all four in one accumulator, 3.1e-7 so, 2.4e-7
// with the bias of the cuts given back, nrc.cuh; 4.1e-7 with FMA chains on the CUDA cores. Other weights and
// inputs give other figures at about the same ratio: half to two thirds).
//
// Bound: the chain of MMAs and epilogues (load, ReLU, split, store of every activation) of the two tiles an SM has room
// for: the tensor pipe is busy 65 % of the time, issue slots 54 %; with 4 of the 18 MMAs of a layer the kernel takes 95 %
// of its time. 2 073 600 queries 0.34 ms, 129 601 queries 30 us (the register-tiled CUDA-core kernel this replaces:
// 1.99 ms, 164 us).
//
// Inference only: the training step stays on the CUDA cores (nrc.cu). Adam divides by the root of the
// squared gradient, so weights whose gradient is all rounding follow that rounding; a training run
// with other sums agrees with the earlier one only until such a weight matters.
// Two tiles of 128 samples per CTA, one CTA per SM, so one tile's epilogue runs under the other's
// MMAs. A tile has 8 warps: a sample is a TMEM lane and two threads, 32 of the 64 units each (with one
// thread per sample the SM held 8 warps, and the encoder and the splits waited on their own latency:
// 2 073 600 queries of the 5 x 64 network 0.60 ms,
// 0.54 with two threads). TMEM per tile: two 64-column accumulators (D1, D2: a layer's output is their sum),
// the next layer's A operand, 3 pieces of 32 columns, and 32 columns for the output layer's exchange.
// Weights: per layer three K-major images of 64 x 64 in shared memory, w1 and w2 adjacent, so one
// N = 128 MMA takes a piece of the activations to both.
// The 64 -> <= 16 output layer stays on the CUDA cores: an MMA round trip costs more than its 192 FMAs a
// sample.
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "nrc.cuh"
#include "tc.cuh"

namespace sty {
namespace {
using namespace tc;

constexpr int W = kNrcWidth;
constexpr int TM = 128;
constexpr int kTiles = 2;                     // tiles in flight per CTA
constexpr int kGT = 256;                      // threads per tile
constexpr uint32_t kCols = 256;               // TMEM columns per tile: D1 64, D2 64, A 3 x 32, exchange 2 x 16
constexpr uint32_t kImg = W * W * 2;          // bytes of one piece of a layer
constexpr uint32_t kLayer = 3 * kImg;         // w1, w2, w3


__global__ void k_pack3(int layers, uint32_t np, float bound, const float *__restrict__ w, uint16_t *__restrict__ img,
                        uint32_t *__restrict__ wide) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    const float v = w[i];
    if (i < (uint32_t)layers * W * W) nrc_store_pieces(img, i, v);
    if (nrc_is_wide(v, bound)) atomicAdd(wide, 1u);
}

struct Args {
    NrcNet n;
    int c4;
    const uint16_t *img;
    const float *w;        // FP32 parameters
    const uint32_t *wide;  // nrc_is_wide weights among them
    uint64_t count;
    const float *input;
    float *output;
    uint32_t *status;
};

__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&q)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3]), "r"(q[4]), "r"(q[5]), "r"(q[6]), "r"(q[7]), "r"(q[8]), "r"(q[9]),
        "r"(q[10]), "r"(q[11]), "r"(q[12]), "r"(q[13]), "r"(q[14]), "r"(q[15])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float lo16(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi16(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// this thread's 32 columns as the three pieces of the A operand
__device__ __forceinline__ void store_a(uint32_t areg, const float (&h)[32]) {
    uint32_t q[3][16];
#pragma unroll
    for (int j = 0; j < 16; j++) {
        const float2 m1 = make_float2(-1.0f, -1.0f);
        float2 v = make_float2(h[2 * j], h[2 * j + 1]);
        q[0][j] = pack2_bf16(v.x, v.y);
        v = ffma2(make_float2(lo16(q[0][j]), hi16(q[0][j])), m1, v);
        q[1][j] = pack2_bf16(v.x, v.y);
        v = ffma2(make_float2(lo16(q[1][j]), hi16(q[1][j])), m1, v);
        q[2][j] = pack2_bf16(v.x, v.y);
    }
#pragma unroll
    for (int p = 0; p < 3; p++) tmem_st16(areg + 32u * p, q[p]);
}
// The six piece products of a layer, 4 K steps each, small ones first.
__device__ __forceinline__ void issue_forward(uint32_t d, uint32_t a, uint32_t w) {
    const uint32_t wide = idesc_bf16(TM, 2 * W), one = idesc_bf16(TM, W);
#pragma unroll
    for (int kk = 0; kk < 4; kk++) mma_ts(d, a + 32u + 8u * kk, make_desc(w + 256u * kk), wide, kk > 0);
#pragma unroll
    for (int kk = 0; kk < 4; kk++) mma_ts(d, a + 64u + 8u * kk, make_desc(w + 256u * kk), one, 1u);
#pragma unroll
    for (int kk = 0; kk < 4; kk++) mma_ts(d + 64u, a + 8u * kk, make_desc(w + 2u * kImg + 256u * kk), one, 1u);
#pragma unroll
    for (int kk = 2; kk < 4; kk++) mma_ts(d, a + 8u * kk, make_desc(w + kImg + 256u * kk), one, 1u);
#pragma unroll
    for (int kk = 0; kk < 2; kk++) mma_ts(d, a + 8u * kk, make_desc(w + 256u * kk), wide, 1u);
#pragma unroll
    for (int kk = 2; kk < 4; kk++) mma_ts(d + 64u, a + 8u * kk, make_desc(w + 256u * kk), one, 1u);
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const float (&v)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "r"(taddr));
}

// A network with wide weights: every row by one thread, each sum over k = 0 .. 63 in order with fmaf, so that what overflows
// does as it does in FP32 (the bits of the CUDA-core kernel that this one replaced).
__device__ __noinline__ void rows_f32(const Args &a) {
    float buf[2][W];
    for (uint64_t row = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; row < a.count; row += (uint64_t)gridDim.x * blockDim.x) {
        nrc_encode(a.n, a.input + row * a.n.in_dims, buf[0]);
        for (int l = 0; l <= a.n.layers; l++) {
            const bool out = l == a.n.layers;
            const float *h = buf[l & 1], *w = a.w + nrc_w_offset(l);
            for (int j = 0; j < (out ? a.n.out_dims : W); j++, w += W) {
                float s = 0.0f;
                for (int k = 0; k < W; k++) s = fmaf(w[k], h[k], s);
                if (out)
                    a.output[row * a.n.out_dims + j] = s;
                else
                    buf[(l + 1) & 1][j] = fmaxf(s, 0.0f);
            }
        }
    }
}

// OM: output columns kept in registers (4, or 16 for wider outputs)
template <int OM>
__global__ void __launch_bounds__(kGT * kTiles, 1) k_nrc_f32tc(const Args a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar[kTiles], wbar;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) float wo[kNrcOutPad * W];
    const int tid = threadIdx.x, warp = (int)uniform(threadIdx.x >> 5), grp = warp / (kGT / 32), half = (warp / 4) & 1, t = tid & 127;
    const bool issuer = warp % (kGT / 32) == 0;  // the tile's issuing warp
    const uint32_t bar_id = 1u + (uint32_t)grp;
    const int L = a.n.layers, O = a.n.out_dims;
    const uint32_t wide = *reinterpret_cast<const volatile uint32_t *>(a.wide);
    for (int e = tid; e < O * W; e += kGT * kTiles) wo[e] = a.w[nrc_w_offset(L) + e];
    if (tid == 0) {
        for (int g = 0; g < kTiles; g++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[g])) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&wbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // the weight images, copied while the first tiles are encoded
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&wbar)), "r"((uint32_t)L * kLayer)
                     : "memory");
        for (int l = 0; l < L; l++)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             smem_u32(smem) + (uint32_t)l * kLayer),
                         "l"(reinterpret_cast<const uint8_t *>(a.img) + (size_t)l * kLayer), "r"(kLayer), "r"(smem_u32(&wbar))
                         : "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = uniform(tmem_slot) + kCols * (uint32_t)grp;
    const uint32_t areg = tmem + 128u;
    const uint32_t lane_off = ((uint32_t)(warp & 3) * 32u) << 16;
    const uint32_t mine = tmem + lane_off + 32u * half;                 // this thread's columns of D1 (D2: + 64)
    const uint32_t amine = areg + lane_off + 16u * half;                // of the A pieces
    const uint32_t exch = tmem + lane_off + 224u;                       // the upper half's share of the output layer, columns 16 .. 31
    const float *wo_mine = wo + 32 * half;
    const uint32_t wbase = smem_u32(smem);
    uint64_t *bar = &mbar[grp];
    uint32_t phase = 0;
    bool failed = false;  // uniform over the tile's threads

    bool ok = true;  // this thread's waits came through; the tile's threads agree on it in publish()
    auto wait_mma = [&]() {
        ok = mbar_wait(bar, phase, a.status) && ok;
        phase ^= 1u;
        fence_after();
    };
    // the tile's TMEM accesses so far come before those issued next; false if any wait ran out
    auto publish = [&]() -> bool {
        tmem_wait_st();
        fence_before();
        const bool all = bar_and_n(bar_id, kGT, ok);
        fence_after();
        return all;
    };
    auto load_sum = [&](float (&h)[32]) {
        float u[32];
        tmem_ld32(mine, h);
        tmem_ld32(mine + 64u, u);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 32; k += 2) {
            const float2 r = ffma2(make_float2(u[k], u[k + 1]), make_float2(1.0f, 1.0f), make_float2(h[k], h[k + 1]));
            h[k] = r.x;
            h[k + 1] = r.y;
        }
    };

    bool loaded = false;  // the weight images have arrived
    const uint64_t ntiles = wide ? 0 : (a.count + TM - 1) / TM;
    if (wide) rows_f32(a);
    // the workload encoder's inputs of this thread's half, loaded a tile ahead (asm volatile: not sunk to
    // their use)
    float xr[kNrcC4Half];
    auto load_x = [&](uint64_t tl) {
        const uint64_t r = tl * TM + t;
        const bool v = a.c4 && tl < ntiles && r < a.count;
        const float *p = a.input + r * kNrcC4Dims + 4 * half;
#pragma unroll
        for (int i = 0; i < kNrcC4Half; i++) {
            xr[i] = 0.0f;
            if (v && (half == 1 || i < 5)) asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(xr[i]) : "l"(p + i));
        }
    };
    load_x(blockIdx.x + (uint64_t)gridDim.x * grp);
    // one tile per SM before any SM gets a second
    for (uint64_t tile = blockIdx.x + (uint64_t)gridDim.x * grp; tile < ntiles && !failed;
         tile += (uint64_t)gridDim.x * kTiles) {
        const uint64_t row = tile * TM + t;
        const bool valid = row < a.count;
        float h[32];
        if (!valid) {
#pragma unroll
            for (int k = 0; k < 32; k++) h[k] = 0.0f;
        } else if (a.c4) {
            if (half == 0)
                nrc_encode_c4<0>(xr, h);
            else
                nrc_encode_c4<1>(xr, h);
        } else {
            float enc[W];
            nrc_encode(a.n, a.input + row * a.n.in_dims, enc);
#pragma unroll
            for (int k = 0; k < 32; k++) h[k] = half == 0 ? enc[k] : enc[32 + k];
        }
        load_x(tile + (uint64_t)gridDim.x * kTiles);
        store_a(amine, h);
        if (!loaded) {
            ok = mbar_wait(&wbar, 0, a.status);
            loaded = true;
        }
        if (!publish()) {
            failed = true;
            break;
        }
        float pred[OM];
#pragma unroll
        for (int c = 0; c < OM; c++) pred[c] = 0.0f;
        for (int l = 0; l < L; l++) {
            if (issuer && elect_one()) {
                issue_forward(tmem, areg, wbase + (uint32_t)l * kLayer);
                mma_commit(bar);
            }
            wait_mma();
            load_sum(h);
#pragma unroll
            for (int k = 0; k < 32; k++) h[k] = fmaxf(h[k], 0.0f);
            if (l + 1 < L) {
                store_a(amine, h);
            } else {  // output layer: this thread's 32 units, then the two halves' sums
#pragma unroll
                for (int c = 0; c < OM; c++)
                    if (c < O) {
#pragma unroll
                        for (int k = 0; k < 32; k += 4) {
                            const float4 w4 = *reinterpret_cast<const float4 *>(wo_mine + c * W + k);
                            pred[c] = fmaf(w4.x, h[k], pred[c]);
                            pred[c] = fmaf(w4.y, h[k + 1], pred[c]);
                            pred[c] = fmaf(w4.z, h[k + 2], pred[c]);
                            pred[c] = fmaf(w4.w, h[k + 3], pred[c]);
                        }
                    }
#pragma unroll
                for (int c = 0; c < OM; c += 4) {
                    const float v[4] = {pred[c], pred[c + 1], pred[c + 2], pred[c + 3]};
                    if (half == 1) tmem_st4(exch + 16u + c, v);
                }
            }
            if (!publish()) {
                failed = true;
                break;
            }
        }
        if (failed) break;
        // (the next tile's first publish orders these reads before the exchange is written again)
        if (half == 0) {
#pragma unroll
            for (int c = 0; c < OM; c += 4) {
                float v[4];
                tmem_ld4(exch + 16u + c, v);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (valid && c + e < O) a.output[row * O + c + e] = pred[c + e] + v[e];
            }
        }
    }
    if (failed) mbar_wait(bar, phase, a.status);  // one more bounded wait before the columns are released
    if (!loaded) mbar_wait(&wbar, 0, a.status);   // no copy in flight when the block ends
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_slot) : "memory");
}

template <int OM>
sty_status launch(Args a, cudaStream_t st) {
    a.c4 = nrc_is_c4(a.n) ? 1 : 0;
    a.status = device_status_ptr();
    if (!a.status) {
        set_error("device status word unavailable");
        return STY_ERR_CUDA;
    }
    int dev = 0, sms = 0;
    STY_TRY(check_cuda(cudaGetDevice(&dev), "cudaGetDevice"));
    STY_TRY(check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr SMs"));
    // at least 120 KB so that one CTA (and its 512 TMEM columns) owns the SM
    const size_t smem = std::max<size_t>((size_t)a.n.layers * kLayer, 122880);
    STY_TRY(check_cuda(cudaFuncSetAttribute(k_nrc_f32tc<OM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                       "attr k_nrc_f32tc"));
    const uint64_t ntiles = (a.count + TM - 1) / TM;
    k_nrc_f32tc<OM><<<(unsigned)std::min<uint64_t>(ntiles, (uint64_t)sms), kGT * kTiles, smem, st>>>(a);
    return check_launch("k_nrc_f32tc");
}

}  // namespace

size_t nrc_f32tc_image_elems(const NrcNet &n) { return (size_t)n.layers * 3 * W * W; }
sty_status nrc_f32tc_pack(const NrcNet &n, const float *w, uint16_t *img, uint32_t *wide, cudaStream_t st) {
    const uint32_t np = (uint32_t)nrc_param_count(n);
    STY_TRY(check_cuda(cudaMemsetAsync(wide, 0, 4, st), "zero wide weights"));
    k_pack3<<<(np + 255) / 256, 256, 0, st>>>(n.layers, np, nrc_wide_bound(n), w, img, wide);
    return check_launch("k_pack3");
}
sty_status nrc_f32tc_forward(const NrcNet &n, const float *w, const uint16_t *img, const uint32_t *wide, uint64_t count,
                             const float *input, float *output, cudaStream_t st) {
    Args a{};
    a.n = n;
    a.img = img;
    a.w = w;
    a.wide = wide;
    a.count = count;
    a.input = input;
    a.output = output;
    return n.out_dims <= 4 ? launch<4>(a, st) : launch<kNrcOutPad>(a, st);
}

}  // namespace sty
