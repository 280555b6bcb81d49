// pf_adjoint.cu -- adjoint of the screen-space NL-PF filter + smoothed ramp style node.
//
// Forward (see include/sty_gb300.h): f_i = N_i / D_i with D_i = sum_j w_ij, N_i = sum_j w_ij in_j,
//   w_ij = exp(a_ij), a_ij = -rho_ij / (2 sx^2) - |p_i - p_j|^2 / (2 sp^2) - (1 - n_i.n_j) / sn^2,
//   out_i = sum_k sigmoid(s (lum(f_i) - t_k)) (c_k - c_{k-1}); image = spp mean; L = |image - T|^2.
// Backward, per valid record i with g_i = dL/dout_i = 2 (image - T) / spp:
//   style:  dL/dc_k += g_i (sig_k - sig_{k+1}),  dL/dt_k += -s sig'_k (g_i . dc_k),
//           dL/ds += sum_k sig'_k (lum_i - t_k) (g_i . dc_k),  h_i = dL/df_i = (sum_k s sig'_k g_i.dc_k) * Y
//           with Y the Rec.709 luminance weights;
//   filter: df_i/dtheta = sum_j dw_ij/dtheta (in_j - f_i) / D_i with dw/dsx = w rho / sx^3,
//           dw/dsp = w |dp|^2 / sp^3, dw/dsn = 2 w (1 - n.n) / sn^3.
// The image and its loss are the forward filter's. The sweep over the staged candidate rows sums D_i and the three bandwidth
// terms with f_i and h_i; where sweep_gives_f() a sweep of the same kernel before it has formed f_i by the same
// operations. Per-thread results are reduced per block into a partial vector; one block per entry sums the partials in a
// fixed order (deterministic).
#include <mutex>

#include "common.cuh"
#include "pf_screen.cuh"
#include "style.cuh"

namespace sty {
namespace {

constexpr int TW = 32, TH = 4, NT = TW * TH, CH = 4, NF = 10;  // staged: p(3) n(3) bias in(3)
constexpr int NG = 36;
constexpr float kL2E = 1.4426950408889634f;

struct AdjArgs {
    const float *pos[3], *nrm[3], *rad[3], *thr[3];
    const int32_t *valid;
    const float *in_next;
    const float *dimg;  // dL/dimage per pixel, interleaved rgb
    float *f;           // filtered radiance, planes of W H S
    int W, H, R;
    uint32_t depth;
    float sx, sp, sn;
    float s, t[8], c[8][3];
    int nsteps;
    float *partials;  // [gridDim.x][NG]
};

__device__ __forceinline__ float sigm(float x) { return 1.0f / (1.0f + expf(-x)); }

// What a query holds during the sweep. The exponent is formed negated, -a log2(e) = isn' om + isp' d2 + isx' rho with
// om = 1 - n_i.n_j summed from the candidate's bias, 1 where the record is valid and kNone where it is not: its weight is
// then exactly 0, for which isn' is kept from falling below kLeast (where om has no weight left any more).
constexpr float kNone = 1e30f, kLeast = 1e-20f;
struct Query {
    float p[3], n[3];   // position; normal, negated
    float h[3], nhf;    // dL/df; -h.f
};
struct Sums {
    float d, e[3];  // sum w; first sweep: sums of w in; second: sums of t = w h.(in_j - f_i) times rho, d2, om
};

// One candidate row for 4 spp on packed FP32: a candidate pixel's 4 samples come in as one 16-byte load per
// field and are paired (0, 1) and (2, 3) against a query duplicated in both lanes, so no value has to be
// moved into a pair. 15 (first sweep) or 19 FFMA2 and 2 MUFU per query and pair.
template <bool FIRST>
__device__ __forceinline__ void row4(const float *__restrict__ rowp, int plane, int lx, int R, int dy, float isx2, float isp2,
                                     float isn, const Query (&q)[4], Sums (&out)[4]) {
    const float2 zero2 = make_float2(0.0f, 0.0f), one2 = make_float2(1.0f, 1.0f), m1 = make_float2(-1.0f, -1.0f);
    const float2 isp = make_float2(isp2, isp2), isn2 = make_float2(isn, isn);
    float2 acc[4][4];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[k][j] = zero2;
#pragma unroll 1
    for (int dx = -R; dx <= R; dx++) {
        const float rho = (float)(dx * dx + dy * dy);
        const float2 arho = make_float2(rho * isx2, rho * isx2), rho2 = make_float2(rho, rho);
        const float *cp = rowp + (lx + R + dx) * 4;
        float4 v[NF];
#pragma unroll
        for (int k = 0; k < NF; k++) v[k] = *reinterpret_cast<const float4 *>(cp + k * plane);
#pragma unroll
        for (int t = 0; t < 2; t++) {
            float2 c[NF];
#pragma unroll
            for (int k = 0; k < NF; k++) c[k] = t == 0 ? make_float2(v[k].x, v[k].y) : make_float2(v[k].z, v[k].w);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                auto two = [](float x) { return make_float2(x, x); };
                const float2 ex = ffma2(c[0], m1, two(q[k].p[0])), ey = ffma2(c[1], m1, two(q[k].p[1])),
                             ez = ffma2(c[2], m1, two(q[k].p[2]));
                const float2 d2 = ffma2(ez, ez, ffma2(ey, ey, ffma2(ex, ex, zero2)));
                const float2 om = ffma2(two(q[k].n[2]), c[5], ffma2(two(q[k].n[1]), c[4], ffma2(two(q[k].n[0]), c[3], c[6])));
                const float2 na = ffma2(om, isn2, ffma2(d2, isp, arho));
                const float2 w = make_float2(ex2_approx(-na.x), ex2_approx(-na.y));
                acc[k][0] = ffma2(w, one2, acc[k][0]);
                if constexpr (FIRST) {
#pragma unroll
                    for (int j = 0; j < 3; j++) acc[k][1 + j] = ffma2(w, c[7 + j], acc[k][1 + j]);
                } else {
                    const float2 u = ffma2(two(q[k].h[2]), c[9], ffma2(two(q[k].h[1]), c[8], ffma2(two(q[k].h[0]), c[7], two(q[k].nhf))));
                    const float2 tt = ffma2(w, u, zero2);
                    acc[k][1] = ffma2(tt, rho2, acc[k][1]);
                    acc[k][2] = ffma2(tt, d2, acc[k][2]);
                    acc[k][3] = ffma2(tt, om, acc[k][3]);
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        out[k].d = acc[k][0].x + acc[k][0].y;
#pragma unroll
        for (int j = 0; j < 3; j++) out[k].e[j] = acc[k][j + 1].x + acc[k][j + 1].y;
    }
}
template <int S, bool FIRST>
__device__ __forceinline__ void row_any(const float *__restrict__ rowp, int plane, int lx, int R, int dy, float isx2, float isp2,
                                        float isn, const Query (&q)[S], Sums (&out)[S]) {
#pragma unroll
    for (int k = 0; k < S; k++) out[k] = {0.0f, {0.0f, 0.0f, 0.0f}};
    for (int dx = -R; dx <= R; dx++) {
        const float rho = (float)(dx * dx + dy * dy), arho = __fmul_rn(rho, isx2);
        const int cb = (lx + R + dx) * S;
#pragma unroll
        for (int t = 0; t < S; t++) {
            float c[NF];
#pragma unroll
            for (int k = 0; k < NF; k++) c[k] = rowp[k * plane + cb + t];
#pragma unroll
            for (int k = 0; k < S; k++) {
                const float ex = q[k].p[0] - c[0], ey = q[k].p[1] - c[1], ez = q[k].p[2] - c[2];
                const float d2 = fmaf(ez, ez, fmaf(ey, ey, __fmul_rn(ex, ex)));
                const float om = fmaf(q[k].n[2], c[5], fmaf(q[k].n[1], c[4], fmaf(q[k].n[0], c[3], c[6])));
                const float w = ex2_approx(-fmaf(om, isn, fmaf(d2, isp2, arho)));
                out[k].d += w;
                if constexpr (FIRST) {
#pragma unroll
                    for (int j = 0; j < 3; j++) out[k].e[j] = fmaf(w, c[7 + j], out[k].e[j]);
                } else {
                    const float tt = w * fmaf(q[k].h[2], c[9], fmaf(q[k].h[1], c[8], fmaf(q[k].h[0], c[7], q[k].nhf)));
                    out[k].e[0] = fmaf(tt, rho, out[k].e[0]);
                    out[k].e[1] = fmaf(tt, d2, out[k].e[1]);
                    out[k].e[2] = fmaf(tt, om, out[k].e[2]);
                }
            }
        }
    }
}

// Bound by the FMA pipe (60 % busy; the data pipe of L1 and shared memory 32 %) with 12 warps per SM, which do not cover
// the staging of the rows and its barriers. 512 x 512, 4 spp, radius 8: the whole adjoint 3.06 ms with two sweeps (the
// first for f and D), a candidate duplicated into each pair, 220 registers and one block of 8 warps per SM; 1.88 with one
// sweep on the forward filter's f, 1.65 with blocks of 32 x 4 pixels, three to an SM (32 x 12, one to an SM: 1.81).
template <int S, bool FIRST>
__global__ void __launch_bounds__(NT, S == 4 ? 3 : 1) k_pf_adjoint(const AdjArgs a) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float red[NT / 32][NG];
    const int R = a.R, CW = TW + 2 * R, plane = CH * CW * S;
    const uint32_t gx = (uint32_t)(a.W + TW - 1) / TW;
    const int tx0 = (int)(blockIdx.x % gx) * TW, ty0 = (int)(blockIdx.x / gx) * TH;
    const int lx = threadIdx.x % TW, ly = threadIdx.x / TW;
    const int x = tx0 + lx, y = ty0 + ly;
    const bool inside = x < a.W && y < a.H;
    const size_t N = (size_t)a.W * a.H * S, dbase = (size_t)a.depth * N;
    const float isx2 = kL2E / (2.0f * a.sx * a.sx), isp2 = kL2E / (2.0f * a.sp * a.sp),
                isn = fmaxf(kL2E / (a.sn * a.sn), kLeast);

    // a warp's sums of gradient entries k0 .. k0 + n - 1
    auto reduce = [&](const float *v0, int k0, int n) {
#pragma unroll
        for (int k = 0; k < n; k++) {
            float v = v0[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][k0 + k] = v;
        }
    };
    Query q[S];
    bool qv[S];
    // queries; in the second sweep the style's backward from f
    {
    float gsum[NG - 3];
#pragma unroll
    for (int k = 0; k < NG - 3; k++) gsum[k] = 0.0f;
#pragma unroll
    for (int s = 0; s < S; s++) {
        const size_t j = inside ? ((size_t)y * a.W + x) * S + s : 0, g = dbase + j;
        qv[s] = inside && a.valid[g] != 0;
        q[s].nhf = 0.0f;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            q[s].p[k] = inside ? a.pos[k][g] : 0.0f;
            q[s].n[k] = inside ? -a.nrm[k][g] : 0.0f;
            q[s].h[k] = 0.0f;
        }
        if (FIRST || !qv[s]) continue;
        const float f[3] = {a.f[j], a.f[N + j], a.f[2 * N + j]};
        const float *gp = a.dimg + 3 * ((size_t)y * a.W + x);
        const float gr[3] = {gp[0] / S, gp[1] / S, gp[2] / S};
        const float cl[3] = {fminf(fmaxf(f[0], 0.0f), 1e5f), fminf(fmaxf(f[1], 0.0f), 1e5f), fminf(fmaxf(f[2], 0.0f), 1e5f)};
        const float lum = cl[0] * 0.2126f + cl[1] * 0.7152f + cl[2] * 0.0722f;
        float dlum = 0.0f, prev[3] = {0.0f, 0.0f, 0.0f}, sg_prev = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (k >= a.nsteps) break;
            const float sg = sigm(a.s * (lum - a.t[k]));
            const float dsg = sg * (1.0f - sg);
            const float gdc = gr[0] * (a.c[k][0] - prev[0]) + gr[1] * (a.c[k][1] - prev[1]) + gr[2] * (a.c[k][2] - prev[2]);
            dlum += a.s * dsg * gdc;
            gsum[0] += dsg * (lum - a.t[k]) * gdc;  // d/ds
            gsum[1 + k] += -a.s * dsg * gdc;        // d/dt_k
            // d out / d c_k = sig_k - sig_{k+1}: accumulate sig_k here, subtract at k+1
#pragma unroll
            for (int ch = 0; ch < 3; ch++) {
                if (k > 0) gsum[9 + 3 * (k > 0 ? k - 1 : 0) + ch] += gr[ch] * (sg_prev - sg);
                if (k + 1 == a.nsteps) gsum[9 + 3 * k + ch] += gr[ch] * sg;
                prev[ch] = a.c[k][ch];
            }
            sg_prev = sg;
        }
        const float Y[3] = {0.2126f, 0.7152f, 0.0722f};
#pragma unroll
        for (int ch = 0; ch < 3; ch++) q[s].h[ch] = f[ch] > 0.0f && f[ch] < 1e5f ? dlum * Y[ch] : 0.0f;
        q[s].nhf = -(q[s].h[0] * f[0] + q[s].h[1] * f[1] + q[s].h[2] * f[2]);
    }
    if (!FIRST) reduce(gsum, 0, NG - 3);
    }

    KahanF acc[S][4];
#pragma unroll
    for (int s = 0; s < S; s++)
#pragma unroll
        for (int k = 0; k < 4; k++) acc[s][k] = {0.0f, 0.0f};
    const int row_lo = ty0 - R, row_hi = ty0 + TH - 1 + R;
    for (int cy = row_lo; cy <= row_hi; cy += CH) {
        __syncthreads();
        for (int idx = threadIdx.x; idx < plane; idx += NT) {
            const int r = idx / (CW * S), rem = idx - r * (CW * S), col = rem / S, s = rem - col * S;
            const int gy = cy + r, gx = tx0 - R + col;
            bool ok = gy >= 0 && gy < a.H && gx >= 0 && gx < a.W && gy <= row_hi;
            size_t j = 0;
            if (ok) {
                j = ((size_t)gy * a.W + gx) * S + s;
                ok = a.valid[dbase + j] != 0;
            }
            const size_t g = dbase + j;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                sm[k * plane + idx] = ok ? a.pos[k][g] : 0.0f;
                sm[(3 + k) * plane + idx] = ok ? a.nrm[k][g] : 0.0f;
                float in = 0.0f;
                if (ok) {
                    in = a.rad[k][g];
                    if (a.in_next) in = fmaf(a.thr[k][g], a.in_next[k * N + j], in);
                }
                sm[(7 + k) * plane + idx] = in;
            }
            sm[6 * plane + idx] = ok ? 1.0f : kNone;
        }
        __syncthreads();
        for (int r = 0; r < CH; r++) {
            const int dy = cy + r - y;
            if (dy < -R || dy > R) continue;
            Sums part[S];
            const float *rowp = sm + r * CW * S;
            if constexpr (S == 4) row4<FIRST>(rowp, plane, lx, R, dy, isx2, isp2, isn, q, part);
            else row_any<S, FIRST>(rowp, plane, lx, R, dy, isx2, isp2, isn, q, part);
#pragma unroll
            for (int s = 0; s < S; s++) {
                acc[s][0].add(part[s].d);
#pragma unroll
                for (int k = 0; k < 3; k++) acc[s][k + 1].add(part[s].e[k]);
            }
        }
    }
    if constexpr (FIRST) {
#pragma unroll
        for (int s = 0; s < S; s++) {
            if (!inside) break;
            const size_t j = ((size_t)y * a.W + x) * S + s;
#pragma unroll
            for (int k = 0; k < 3; k++) a.f[k * N + j] = qv[s] ? acc[s][k + 1].s / acc[s][0].s : 0.0f;
        }
        return;
    }
    float bw[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int s = 0; s < S; s++) {
        if (!qv[s]) continue;
        const float inv = 1.0f / acc[s][0].s;
        bw[0] += acc[s][1].s * inv / (a.sx * a.sx * a.sx);
        bw[1] += acc[s][2].s * inv / (a.sp * a.sp * a.sp);
        bw[2] += 2.0f * acc[s][3].s * inv / (a.sn * a.sn * a.sn);
    }
    reduce(bw, NG - 3, 3);
    __syncthreads();
    if (threadIdx.x < NG) {
        float v = 0.0f;
        for (int w = 0; w < NT / 32; w++) v += red[w][threadIdx.x];
        a.partials[(size_t)blockIdx.x * NG + threadIdx.x] = v;
    }
}

// image = spp mean of the styled filtered radiance (0 where a record is invalid); dimg = 2 (image - target); loss
// partials per block
__global__ void k_img_loss(const float *f, const int32_t *valid, const sty_style_program style, uint32_t depth, int W, int H, int S,
                           const float *target, float *dimg, float *lpart) {
    __shared__ float red[8];
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t N = (size_t)W * H * S;
    float l = 0.0f;
    if (p < W * H) {
        float m[3] = {0.0f, 0.0f, 0.0f};
        for (int s = 0; s < S; s++) {
            const size_t j = (size_t)p * S + s;
            if (!valid[j]) continue;
            const f3 o = style_apply(style, depth, f3{f[j], f[N + j], f[2 * N + j]});
            m[0] += o.x;
            m[1] += o.y;
            m[2] += o.z;
        }
        for (int c = 0; c < 3; c++) {
            const float d = m[c] / S - target[3 * (size_t)p + c];
            dimg[3 * (size_t)p + c] = 2.0f * d;
            l += d * d;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
        lpart[blockIdx.x] = t;
    }
}

// Sum of per-block partial vectors, one block per entry: thread t adds partials t, t + 256, ... compensated, the
// threads' sums are added pairwise. The order is fixed. (One thread per entry, all partials in a row:
// 35 us at 1024 blocks, bound by the chain of loads; now 3.)
__global__ void __launch_bounds__(256) k_reduce_partials(const float *partials, int nblocks, int width, float *outv) {
    __shared__ float sum[256], comp[256];
    const int k = blockIdx.x, t = threadIdx.x;
    KahanF s = {0.0f, 0.0f};
    for (int b = t; b < nblocks; b += 256) s.add(partials[(size_t)b * width + k]);
    sum[t] = s.s;
    comp[t] = s.c;
    for (int o = 128; o > 0; o >>= 1) {
        __syncthreads();
        if (t < o) {
            KahanF r = {sum[t], comp[t] + comp[t + o]};
            r.add(sum[t + o]);
            sum[t] = r.s;
            comp[t] = r.c;
        }
    }
    if (t == 0) outv[k] = sum[0];
}

template <int S, bool FIRST>
sty_status launch_sweep(const AdjArgs &a, cudaStream_t st) {
    const int CW = TW + 2 * a.R;
    const size_t smem = (size_t)NF * CH * CW * S * sizeof(float);
    STY_TRY(check_cuda(cudaFuncSetAttribute(k_pf_adjoint<S, FIRST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                       "attr k_pf_adjoint"));
    const unsigned grid = (unsigned)((a.W + TW - 1) / TW) * (unsigned)((a.H + TH - 1) / TH);
    k_pf_adjoint<S, FIRST><<<grid, NT, smem, st>>>(a);
    return check_launch("k_pf_adjoint");
}
template <bool FIRST>
sty_status sweep(const AdjArgs &a, int S, cudaStream_t st) {
    switch (S) {
        case 1: return launch_sweep<1, FIRST>(a, st);
        case 2: return launch_sweep<2, FIRST>(a, st);
        case 4: return launch_sweep<4, FIRST>(a, st);
        default: return launch_sweep<8, FIRST>(a, st);
    }
}

// Whether f_i is formed by the sweep's own operations, so that the sums of w (in_j - f_i) cancel with the weights they are
// made of, or taken from the forward filter, whose weights are rounded otherwise. Error of the gradient's norm against 64
// bits with the filter's f, over 39 sets of records and bandwidths, as a multiple of that with the sweep's (geometric mean,
// largest): 1 sample 1.0, 2.8; 2 samples 1.6, 38 (2.8e-6 for 7e-8); 4 samples (whose filter subtracts a tile's
// centre from the positions before it scales them) 0.9, 2.1; 8 samples 1.4, 12. The 2.1 and the like are surfaces with
// sigma_nrm <= 0.05: the filter rounds the normal term's factor into the normals. The first sweep takes
// 0.8 ms at 512 x 512, 4 spp, radius 8, where the whole is 1.65 without it (2 spp 0.91 and 0.65; before, with f always so, 1.08).
bool sweep_gives_f(int spp, float sigma_nrm) { return spp == 2 || spp == 8 || sigma_nrm < 0.1f; }

// everything both entry points launch, with their scratch: f 3 N floats, dimg 3 per pixel, parts NG per block, lparts one per
// 256 pixels, lsum 1
sty_status run_adjoint(const sty_pf_records *rec, uint32_t depth, int32_t radius, const float prm[36], uint32_t n_steps,
                       const float *in_next, const float *target, float *f, float *dimg, float *parts, float *lparts, float *lsum,
                       float *grad, cudaStream_t st) {
    const int Wd = rec->width, Hd = rec->height, S = rec->spp;
    const size_t N = (size_t)Wd * Hd * S;
    const int nb = ((Wd + TW - 1) / TW) * ((Hd + TH - 1) / TH), lb = (Wd * Hd + 255) / 256;
    // the ramp node (at this depth only), applied to the forward filter's result
    sty_style_program prog;
    memset(&prog, 0, sizeof(prog));
    prog.n_nodes = 1;
    sty_style_node &nd = prog.nodes[0];
    nd.kind = STY_STYLE_RAMP_SMOOTH;
    nd.depth_mask = 1u << (depth > 31 ? 31 : depth);
    nd.n = (int32_t)n_steps;
    nd.p[0] = prm[0];
    for (uint32_t k = 0; k < n_steps; k++) {
        nd.p[1 + k] = prm[1 + k];
        for (int c = 0; c < 3; c++) nd.p[9 + 3 * k + c] = prm[9 + 3 * k + c];
    }
    AdjArgs a;
    for (int k = 0; k < 3; k++) {
        a.pos[k] = rec->pos[k];
        a.nrm[k] = rec->nrm[k];
        a.rad[k] = rec->rad[k];
        a.thr[k] = rec->thr[k];
    }
    a.valid = rec->valid;
    a.in_next = in_next;
    a.dimg = dimg;
    a.f = f;
    a.W = Wd;
    a.H = Hd;
    a.R = radius;
    a.depth = depth;
    a.sx = prm[33];
    a.sp = prm[34];
    a.sn = prm[35];
    a.s = prm[0];
    for (int k = 0; k < 8; k++) {
        a.t[k] = prm[1 + k];
        for (int c = 0; c < 3; c++) a.c[k][c] = prm[9 + 3 * k + c];
    }
    a.nsteps = (int)n_steps;
    a.partials = parts;
    const sty_pf_screen_params sp = {radius, prm[33], prm[34], prm[35]};
    STY_TRY(screen_filter_depth(rec, depth, &sp, nullptr, in_next, f, nullptr, false, st));
    k_img_loss<<<lb, 256, 0, st>>>(f, rec->valid + (size_t)depth * N, prog, depth, Wd, Hd, S, target, dimg, lparts);
    STY_TRY(check_launch("k_img_loss"));
    if (sweep_gives_f(S, prm[35])) STY_TRY(sweep<true>(a, S, st));
    STY_TRY(sweep<false>(a, S, st));
    k_reduce_partials<<<NG, 256, 0, st>>>(parts, nb, NG, grad);
    STY_TRY(check_launch("k_reduce_partials"));
    k_reduce_partials<<<1, 256, 0, st>>>(lparts, lb, 1, lsum);
    return check_launch("k_reduce_partials(loss)");
}

}  // namespace
}  // namespace sty

using namespace sty;

extern "C" sty_status sty_pf_adjoint(const sty_pf_records *rec, uint32_t depth, int32_t radius, const float prm[36],
                                     uint32_t n_steps, const float *in_next, const float *target, float *grad,
                                     float *loss_out, void *stream) {
    clear_error();
    STY_ARG_CHECK(rec && prm && target && grad, "sty_pf_adjoint: null argument");
    STY_ARG_CHECK(n_steps >= 1 && n_steps <= 8, "n_steps must be in [1, 8]");
    STY_ARG_CHECK(radius >= 0 && radius <= 32, "radius must be in [0, 32]");
    STY_ARG_CHECK(prm[33] > 0.0f && prm[34] > 0.0f && prm[35] > 0.0f, "bandwidths must be > 0");
    STY_ARG_CHECK(depth < (uint32_t)rec->depths, "depth out of range");
    STY_ARG_CHECK(rec->spp == 1 || rec->spp == 2 || rec->spp == 4 || rec->spp == 8, "spp must be 1, 2, 4 or 8");
    cudaStream_t st = as_stream(stream);
    const int Wd = rec->width, Hd = rec->height, S = rec->spp;
    const size_t N = (size_t)Wd * Hd * S;
    const int gx = (Wd + TW - 1) / TW, gy = (Hd + TH - 1) / TH, nb = gx * gy;
    const int npix = Wd * Hd, lb = (npix + 255) / 256;
    float *out = nullptr, *dimg = nullptr, *parts = nullptr, *lparts = nullptr, *lsum = nullptr;
    sty_status s = check_cuda(device_malloc_async((void **)&out, 3 * N * 4, st), "alloc adjoint out");
    if (s == STY_OK) s = check_cuda(device_malloc_async((void **)&dimg, (size_t)npix * 3 * 4, st), "alloc dimg");
    if (s == STY_OK) s = check_cuda(device_malloc_async((void **)&parts, (size_t)nb * NG * 4, st), "alloc partials");
    if (s == STY_OK) s = check_cuda(device_malloc_async((void **)&lparts, (size_t)lb * 4, st), "alloc loss partials");
    if (s == STY_OK) s = check_cuda(device_malloc_async((void **)&lsum, 4, st), "alloc loss");
    if (s == STY_OK)
        s = run_adjoint(rec, depth, radius, prm, n_steps, in_next, target, out, dimg, parts, lparts, lsum, grad, st);
    if (s == STY_OK && loss_out) {
        s = check_cuda(cudaMemcpyAsync(loss_out, lsum, 4, cudaMemcpyDeviceToHost, st), "read loss");
        if (s == STY_OK) s = check_cuda(cudaStreamSynchronize(st), "sync loss");
    }
    void *ptrs[] = {out, dimg, parts, lparts, lsum};
    for (void *p : ptrs)
        if (p) cudaFreeAsync(p, st);
    return s;
}

// ---- allocation-free variant ---------------------------------------------------------------
// For callers that cannot allocate device memory: a host integrator whose device memory is owned
// and budgeted by another runtime (the reference sizes its NL-PF scratch from the `vram` config key
// and allocates every buffer through its own device layer), or a render loop that must not fail on
// an allocation half-way through a frame. Their scratch lives in one fixed device array, reserved
// when the library is loaded on a device and held until the process exits.
namespace sty {
namespace {
constexpr size_t kNaMaxRecords = size_t(1) << 18;           // width * height * spp of the depth
constexpr size_t kNaMaxPixels = size_t(1) << 16;            // width * height
constexpr size_t kNaMaxBlocks = 4096;                       // 32 x 8 pixels each, two blocks of the kernel
constexpr size_t kNaMaxLossBlocks = kNaMaxPixels / 256;
constexpr size_t kNaOut = 0;                                // 3 * kNaMaxRecords floats
constexpr size_t kNaDimg = kNaOut + 3 * kNaMaxRecords;      // 3 * kNaMaxPixels
constexpr size_t kNaParts = kNaDimg + 3 * kNaMaxPixels;     // 2 * kNaMaxBlocks * 36
constexpr size_t kNaLParts = kNaParts + 2 * kNaMaxBlocks * NG;  // kNaMaxLossBlocks
constexpr size_t kNaLoss = kNaLParts + kNaMaxLossBlocks;    // 1 (padded)
constexpr size_t kNaFloats = kNaLoss + 64;                  // 1,278,272 floats = 4.88 MiB

// The scratch itself. Host code must not pass this name to a kernel: on the host it is only a
// stand-in for the symbol; the device address comes from cudaGetSymbolAddress below.
static __device__ __align__(256) float g_adjoint_scratch[kNaFloats];

// Device address of g_adjoint_scratch on the current device, looked up with that device current on
// the first call there (and again if the device's context was replaced: a device reset reloads the
// module, possibly at another address).
sty_status noalloc_scratch(float **out) {
    struct Entry {
        float *ptr = nullptr;
        uint64_t ctx = 0;
    };
    static Entry cache[64];
    static std::mutex mu;
    int dev = -1;
    STY_TRY(check_cuda(cudaGetDevice(&dev), "cudaGetDevice"));
    if (dev < 0 || dev >= 64) {
        set_error("device ordinal %d out of range", dev);
        return STY_ERR_UNSUPPORTED;
    }
    std::lock_guard<std::mutex> lock(mu);
    const uint64_t ctx = current_context_id();
    if (!cache[dev].ptr || ctx == 0 || cache[dev].ctx != ctx) {
        void *addr = nullptr;
        STY_TRY(check_cuda(cudaGetSymbolAddress(&addr, g_adjoint_scratch), "cudaGetSymbolAddress(adjoint scratch)"));
        cache[dev].ptr = static_cast<float *>(addr);
        cache[dev].ctx = current_context_id();
    }
    *out = cache[dev].ptr;
    return STY_OK;
}
}  // namespace
}  // namespace sty

extern "C" sty_status sty_pf_adjoint_noalloc(const sty_pf_records *rec, uint32_t depth, int32_t radius,
                                             const float prm[36], uint32_t n_steps, const float *in_next,
                                             const float *target, float *grad, float *loss_out, void *stream) {
    clear_error();
    STY_ARG_CHECK(rec && prm && target && grad, "sty_pf_adjoint_noalloc: null argument");
    STY_ARG_CHECK(n_steps >= 1 && n_steps <= 8, "n_steps must be in [1, 8]");
    STY_ARG_CHECK(radius >= 0 && radius <= 32, "radius must be in [0, 32]");
    STY_ARG_CHECK(prm[33] > 0.0f && prm[34] > 0.0f && prm[35] > 0.0f, "bandwidths must be > 0");
    STY_ARG_CHECK(depth < (uint32_t)rec->depths, "depth out of range");
    STY_ARG_CHECK(rec->spp == 1 || rec->spp == 2 || rec->spp == 4 || rec->spp == 8, "spp must be 1, 2, 4 or 8");
    STY_ARG_CHECK(rec->width > 0 && rec->height > 0, "empty image");
    const int Wd = rec->width, Hd = rec->height, S = rec->spp;
    const size_t N = (size_t)Wd * Hd * S, npix = (size_t)Wd * Hd;
    STY_ARG_CHECK(N <= kNaMaxRecords,
                  "sty_pf_adjoint_noalloc: %zu records per depth exceed the fixed scratch limit of %zu "
                  "(width * height * spp); use sty_pf_adjoint", N, kNaMaxRecords);
    STY_ARG_CHECK(npix <= kNaMaxPixels,
                  "sty_pf_adjoint_noalloc: %zu pixels exceed the fixed scratch limit of %zu; use sty_pf_adjoint",
                  npix, kNaMaxPixels);
    const size_t tiles = (size_t)((Wd + 31) / 32) * ((Hd + 7) / 8);
    static_assert(TH == 4 && TW == 32, "at most two blocks per tile of 32 x 8 pixels");
    STY_ARG_CHECK(tiles <= kNaMaxBlocks, "sty_pf_adjoint_noalloc: %zu tiles exceed the fixed scratch limit of %zu",
                  tiles, kNaMaxBlocks);
    float *scratch = nullptr;
    STY_TRY(noalloc_scratch(&scratch));
    float *out = scratch + kNaOut, *dimg = scratch + kNaDimg, *parts = scratch + kNaParts;
    float *lparts = scratch + kNaLParts, *lsum = scratch + kNaLoss;
    cudaStream_t st = as_stream(stream);
    // Every scratch region is fully overwritten before it is read (no accumulation into scratch), so
    // nothing has to be cleared between calls.
    STY_TRY(run_adjoint(rec, depth, radius, prm, n_steps, in_next, target, out, dimg, parts, lparts, lsum, grad, st));
    if (loss_out) {
        STY_TRY(check_cuda(cudaMemcpyAsync(loss_out, lsum, 4, cudaMemcpyDeviceToHost, st), "read loss"));
        STY_TRY(check_cuda(cudaStreamSynchronize(st), "sync loss"));
    }
    return STY_OK;
}
