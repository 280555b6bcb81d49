// brpt.cu -- the branching path tracer (crates/akari_integrator/src/branching_pt.rs): the paper's
// BrPT baseline and, with inner_samples = [1], the plain stylized path tracer of
// configs/teaser/pt.json.
//
// Per pixel a tree of vertices. A vertex whose surface is rough (average roughness > 0.01) and is
// the k-th rough vertex of its path takes inner_samples[k] branches (1 beyond the list, 1 at smooth
// vertices, none at max_depth); each branch is one light sample (NEE, the light's style at depth + 1
// with the vertex's updated flags) and one BSDF sample whose continuation ray makes the child vertex
// (kernel_advance :543-726). Bottom-up, a vertex's radiance is
//   style_depth(Le + (1/n) sum_branches (direct_s + throughput_s * L_child_s * mis_child_s))
// with the style picked by the flags the vertex inherited (kernel_propagate :240-500, the
// non-debiased estimator; mis_child is the child's emission weight, :568-575); the depth-0 vertex's
// radiance is the pixel sample.
//
// GB300 layout: one breadth-first wavefront per depth over SoA slot planes. A vertex's children are
// one contiguous block (exclusive scan of the branch counts), so the tree needs no linked lists or
// atomics, a child finds its parent by binary search over the scan, and the bottom-up sums run in a
// fixed order (deterministic). Pixels go through in passes sized so the worst-case tree fits the
// `vram_mb` budget (the reference's pixels_per_pass rule, :806-846).
// Sampling: hierarchical 64-bit keys -- the camera slot of pixel px in repeat r keys on
// (seed, r, px), a child on (its parent's key, branch index) -- each seeding one PCG32 stream
// (2 draws for the camera; per branch 3 for the light, then 3 for the BSDF), so an image does not
// depend on how pixels are grouped into passes. The reference draws from a per-slot PCG32 buffer
// whose slots are handed out by atomics; that assignment is not reproducible, so no stream of it is
// matched here.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "scene.cuh"
#include "style.cuh"
#include "tracer.cuh"

namespace sty {
const sty_camera &scene_camera(const sty_scene *s);
bool style_program_valid(const sty_style_program *p);
}  // namespace sty

namespace sty {
namespace {

constexpr uint32_t kBrSlotBytes = 100;  // 22 four-byte planes + one 8-byte key per slot

struct BrSlots {
    float *p[3], *ng[3], *wo[3], *rad[3], *thr[3], *dir[3], *mis;
    uint32_t *prim, *flags, *ab, *nchild, *cbase;
    uint64_t *key;
};
struct BrInner {
    uint32_t n;
    uint32_t v[STY_BRPT_MAX_LEVELS];
};

__device__ __forceinline__ sty_pcg32 key_stream(uint64_t key) {
    sty_pcg32 g;
    g.state = 0;
    g.inc = (key << 1) | 1ull;
    pcg_next(g);
    g.state += splitmix64(key);
    pcg_next(g);
    return g;
}
__device__ __forceinline__ uint64_t child_key(uint64_t parent, uint32_t s) {
    return splitmix64(parent ^ (0x9e3779b97f4a7c15ull * (uint64_t)(s + 1u)));
}
__device__ __forceinline__ F3 hit_point(const SceneView &sc, const Hit &h) {
    const float *tp = sc.tri_pos + 9 * (size_t)h.prim;
    const float b0 = 1.0f - h.b1 - h.b2;
    return f3m(b0 * tp[0] + h.b1 * tp[3] + h.b2 * tp[6], b0 * tp[1] + h.b1 * tp[4] + h.b2 * tp[7],
               b0 * tp[2] + h.b1 * tp[5] + h.b2 * tp[8]);
}
__device__ __forceinline__ F3 tri_ng(const SceneView &sc, uint32_t prim) {
    return f3m(sc.tri_normal[3 * prim], sc.tri_normal[3 * prim + 1], sc.tri_normal[3 * prim + 2]);
}
__device__ __forceinline__ void put3(float *const (&pl)[3], size_t i, F3 v) {
    pl[0][i] = v.x;
    pl[1][i] = v.y;
    pl[2][i] = v.z;
}
__device__ __forceinline__ F3 get3(float *const (&pl)[3], size_t i) { return f3m(pl[0][i], pl[1][i], pl[2][i]); }

// key of repeat r: every pixel sample of that repeat keys on it
__host__ __device__ __forceinline__ uint64_t repeat_key(uint64_t seed, uint64_t r) {
    return splitmix64(splitmix64(seed ^ 0x4252505400000000ull) + r);
}
// branch count of a vertex at `depth` (kernel_advance :598-620)
template <bool PRINC>
__device__ __forceinline__ uint32_t branch_count(const SceneView &sc, const sty_scene_material &m, F3 ng, F3 wo, uint32_t ab,
                                                 uint32_t depth, uint32_t max_depth, const BrInner &inner) {
    if (depth + 1 > max_depth) return 0u;
    return lobe_roughness<PRINC>(m, sc.ggx_tab, ng, wo) > 0.01f ? (ab < inner.n ? inner.v[ab] : 1u) : 1u;
}
// depth 0: the camera slots of samples q0 .. q0 + n, sample q = repeat * npx + pixel (kernel_init
// :501-541)
// with their branch counts, and a 0 behind the last one: the scan over n + 1 counts ends in their total
template <bool PRINC>
__global__ void k_br_camera(SceneView sc, CamArgs cam, uint32_t n, uint64_t q0, uint32_t npx, uint64_t seed,
                            uint64_t first_repeat, uint32_t max_depth, BrInner inner, BrSlots s, unsigned long long *hits) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) s.nchild[n] = 0u;
    if (i >= n) return;
    const uint64_t q = q0 + i;
    const uint32_t px = (uint32_t)(q % npx);
    const uint64_t key = splitmix64(repeat_key(seed, first_repeat + q / npx) + px);
    sty_pcg32 st = key_stream(key);
    F3 ro, rd;
    camera_ray(cam, px, st, &ro, &rd);
    s.key[i] = key;
    s.flags[i] = 0;
    s.ab[i] = 0;
    s.mis[i] = 1.0f;
    put3(s.thr, i, f3m(1.0f, 1.0f, 1.0f));
    const float o3[3] = {ro.x, ro.y, ro.z}, d3[3] = {rd.x, rd.y, rd.z};
    const Hit h = trace_closest(sc, o3, d3, 0.0f, 1e20f, NONE);
    s.prim[i] = h.prim;
    if (h.prim == NONE) {
        s.nchild[i] = 0u;
        put3(s.rad, i, f3m(0.0f, 0.0f, 0.0f));
        return;
    }
    atomicAdd(hits, 1ull);
    const F3 p = hit_point(sc, h), ng = tri_ng(sc, h.prim);
    const sty_scene_material m = sc.materials[sc.tri_material[h.prim]];
    F3 le;
    float mis;
    emitter_le(sc, m, h.prim, p, ng, rd, 0, ro, 0.0f, &le, &mis);
    put3(s.p, i, p);
    put3(s.ng, i, ng);
    put3(s.wo, i, -rd);
    s.nchild[i] = branch_count<PRINC>(sc, m, ng, -rd, 0u, 0u, max_depth, inner);
    put3(s.rad, i, le);
}

// The children of one depth in three kernels (kernel_advance :622-712): the samples of every branch, the
// walks of all their rays, the children's vertices. A walk's length differs from ray to ray, so in one
// kernel 7 of a warp's 32 lanes were at work on average. Between the kernels a child's planes carry its
// two rays:
//   shadow   rad = origin, ng = direction, mis = length, nchild = the light's triangle (NONE: no ray),
//            dir = what the sample adds if nothing is in the way
//   next     p = origin, wo = -direction, thr = throughput, cbase = pdf (0: no ray); after the walk p = the
//            hit's barycentrics and triangle
//   both     prim = the triangle they leave
__device__ __forceinline__ uint32_t parent_of(const BrSlots &s, uint32_t pbase, uint32_t n_par, uint32_t j) {
    uint32_t lo = 0, hi = n_par - 1;  // the last parent whose block starts at or before j
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1u) >> 1;
        if (s.cbase[pbase + mid] <= j) lo = mid;
        else hi = mid - 1u;
    }
    return pbase + lo;
}
// (Closures, two blocks per SM: 1 % faster than without the bound, and their lobes round as in the one kernel that
// did samples and walks before: principled room at 64 x 36 the same film, without the bound 1e-8 off, glass room 4e-6.)
template <bool PRINC>
__global__ void __launch_bounds__(256, PRINC ? 2 : 3) k_br_sample(SceneView sc, uint32_t n_child, uint32_t pbase, uint32_t n_par, uint32_t cbase0,
                            uint32_t depth, const sty_style_program *progs, uint32_t n_progs, BrSlots s,
                            unsigned long long *next_ray) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j == 0) *next_ray = 0;
    if (j >= n_child) return;
    const uint32_t pg = parent_of(s, pbase, n_par, j), sidx = j - s.cbase[pg], cg = cbase0 + j;
    const uint32_t prim = s.prim[pg];
    const F3 p = get3(s.p, pg), ng = get3(s.ng, pg), wo = get3(s.wo, pg);
    const sty_scene_material m = sc.materials[sc.tri_material[prim]];
    const uint32_t new_flags = update_flags(m, s.flags[pg]);
    const uint32_t ab = s.ab[pg] + (lobe_roughness<PRINC>(m, sc.ggx_tab, ng, wo) > 0.01f ? 1u : 0u);
    const uint64_t key = child_key(s.key[pg], sidx);
    sty_pcg32 st = key_stream(key);
    // NEE (sample_light :727-783, shaded with balance MIS in sample_surface_and_shade_direct :170-197)
    F3 direct = f3m(0.0f, 0.0f, 0.0f);
    uint32_t lt = NONE;
    {
        NeeSample n;
        if (nee_candidate(sc, p, ng, new_flags, depth, progs, n_progs, st, &n)) {
            F3 f;
            const float bp = bsdf_eval<PRINC>(m, ng, ng, wo, n.wi, &f, sc.ggx_tab);
            const float w = n.pdf / (n.pdf + bp) / n.pdf;
            direct = f3m(n.li.x * f.x, n.li.y * f.y, n.li.z * f.z) * w;
            lt = n.lt;
            put3(s.rad, cg, n.so);
            put3(s.ng, cg, n.wi);
            s.mis[cg] = n.tmax;
        }
    }
    put3(s.dir, cg, direct);
    s.nchild[cg] = lt;
    s.key[cg] = key;
    s.flags[cg] = new_flags;
    s.ab[cg] = ab;
    s.prim[cg] = prim;
    const float usel = next_1d(st), u0 = next_1d(st), u1 = next_1d(st);
    float pdf = 0.0f;
    const F3 wi = bsdf_sample<PRINC>(m, ng, ng, wo, usel, u0, u1, &pdf, sc.ggx_tab);
    if (!(pdf > 0.0f)) {
        s.cbase[cg] = 0u;
        return;
    }
    F3 f;
    bsdf_eval<PRINC>(m, ng, ng, wo, wi, &f, sc.ggx_tab);
    put3(s.p, cg, offset_ray_origin(p, face_forward(ng, wi)));
    put3(s.wo, cg, -wi);
    put3(s.thr, cg, f * (1.0f / pdf));
    s.cbase[cg] = __float_as_uint(pdf);
}

// Rays 0 .. n - 1 are the children's shadow rays, n .. 2 n - 1 their next ones. Bound by instruction issue
// (3.0 to 3.2 of 4 per cycle), so what counts is how many lanes an instruction serves:
// - persistent, a lane whose ray is done gets the next one, once kRefill of them wait (a ray's set-up is
//   some 100 instructions of the whole warp); looked at every kWalkSteps steps;
// - a step is either a node or one triangle, whichever more lanes are at; the others wait.
// Room of 49.6 k triangles, 160 x 90, 16 x 8 x 4 branches, depth 8: 66.8 ms for a render with one kernel on a
// binary tree, 56.7 on the 4-wide one, 48.1 with the walk as its own kernel taking nodes and leaves in
// turn, 37.0 with the vote; 32.0 with the planes kept by the scene. Cornell box: 9.9 ms, now 6.7. 8, 10, 12 blocks
// per SM are within 1 %; refilling at 8 lanes 2 % slower, at 32 (no refill) 12 %.
constexpr int kWalkThreads = 128, kWalkSteps = 8, kRefill = 16;
__global__ void __launch_bounds__(kWalkThreads, 10) k_br_walk(SceneView sc, uint32_t n, uint32_t cbase0, BrSlots s,
                                                             unsigned long long *next) {
    uint2 stack[kStack];
    Walk w;
    const uint64_t total = 2 * (uint64_t)n;
    const uint32_t lane = threadIdx.x & 31;
    bool active = false, shadow = false, drained = false;
    uint32_t cg = 0;
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, !active);
        if (!drained && (idle == 0xffffffffu || __popc(idle) >= kRefill)) {
            unsigned long long first = 0;
            if (lane == 0) first = atomicAdd(next, (unsigned long long)__popc(idle));
            first = __shfl_sync(0xffffffffu, first, 0);
            drained = first + __popc(idle) >= total;
            const uint64_t r = first + __popc(idle & ((1u << lane) - 1u));
            if (!active && r < total) {
                shadow = r < n;
                cg = cbase0 + (uint32_t)(shadow ? r : r - n);
                const uint32_t prim = s.prim[cg];
                if (shadow) {
                    const uint32_t lt = s.nchild[cg];
                    if (lt != NONE) {
                        const F3 o = get3(s.rad, cg), d = get3(s.ng, cg);
                        const float o3[3] = {o.x, o.y, o.z}, d3[3] = {d.x, d.y, d.z};
                        w.start(o3, d3, 0.0f, s.mis[cg], prim, lt);
                        active = true;
                    }
                } else if (s.cbase[cg] != 0u) {
                    const F3 o = get3(s.p, cg), d = -get3(s.wo, cg);
                    const float o3[3] = {o.x, o.y, o.z}, d3[3] = {d.x, d.y, d.z};
                    w.start(o3, d3, 0.0f, 1e20f, prim, prim);
                    active = true;
                }
            }
        }
        if (drained && __ballot_sync(0xffffffffu, active) == 0) return;
#pragma unroll 1
        for (int k = 0; k < kWalkSteps; k++) {
            const bool at_node = active && w.at_node(), at_leaf = active && !w.at_node();
            const int nodes = __popc(__ballot_sync(0xffffffffu, at_node)), leaves = __popc(__ballot_sync(0xffffffffu, at_leaf));
            bool more = true;
            if (nodes >= leaves) {
                if (at_node) more = w.node(sc, stack);
            } else if (at_leaf) {
                const bool hit = w.triangle(sc);
                if (hit && shadow) more = false;
                else if (w.at_node()) more = w.pop(stack);
            }
            if (active && !more) {
                active = false;
                if (!shadow) {
                    s.p[0][cg] = w.h.b1;
                    s.p[1][cg] = w.h.b2;
                    s.p[2][cg] = __uint_as_float(w.h.prim);
                } else if (w.h.prim != NONE) {
                    put3(s.dir, cg, f3m(0.0f, 0.0f, 0.0f));
                }
            }
        }
    }
}

// a 0 goes behind the last branch count, as in k_br_camera
template <bool PRINC>
__global__ void __launch_bounds__(256) k_br_vertex(SceneView sc, uint32_t n_child, uint32_t pbase, uint32_t n_par, uint32_t cbase0,
                                                   uint32_t depth, uint32_t max_depth, BrInner inner, BrSlots s,
                                                   unsigned long long *hits) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t cg = cbase0 + j;
    Hit h;
    h.prim = NONE;
    float pdf = 0.0f;
    if (j < n_child) {
        pdf = __uint_as_float(s.cbase[cg]);
        if (pdf > 0.0f) {
            h.b1 = s.p[0][cg];
            h.b2 = s.p[1][cg];
            h.prim = __float_as_uint(s.p[2][cg]);
        }
    }
    const uint32_t got = __ballot_sync(0xffffffffu, h.prim != NONE);
    if ((threadIdx.x & 31) == 0 && got) atomicAdd(hits, (unsigned long long)__popc(got));
    if (j == 0) s.nchild[cbase0 + n_child] = 0u;
    if (j >= n_child) return;
    s.prim[cg] = h.prim;
    if (h.prim == NONE) {
        s.nchild[cg] = 0u;
        s.mis[cg] = 1.0f;
        put3(s.rad, cg, f3m(0.0f, 0.0f, 0.0f));
        put3(s.thr, cg, f3m(0.0f, 0.0f, 0.0f));
        return;
    }
    const F3 q = hit_point(sc, h), qn = tri_ng(sc, h.prim);
    const sty_scene_material mq = sc.materials[sc.tri_material[h.prim]];
    F3 p = f3m(0.0f, 0.0f, 0.0f);  // the parent's point: read for emitters only
    if (mq.emission[0] > 0.0f || mq.emission[1] > 0.0f || mq.emission[2] > 0.0f)
        p = get3(s.p, parent_of(s, pbase, n_par, j));
    F3 le;
    float mis;
    emitter_le(sc, mq, h.prim, q, qn, -get3(s.wo, cg), depth + 1, p, pdf, &le, &mis);
    put3(s.p, cg, q);
    put3(s.ng, cg, qn);
    put3(s.rad, cg, le);
    s.mis[cg] = mis;
    s.nchild[cg] = branch_count<PRINC>(sc, mq, qn, get3(s.wo, cg), s.ab[cg], depth + 1, max_depth, inner);
}

// bottom-up radiance of one depth (kernel_propagate); depth 0 leaves the pixel samples in `rad`
__global__ void __launch_bounds__(256, 5) k_br_propagate(SceneView sc, uint32_t n, uint32_t base, uint32_t cbase0, uint32_t depth,
                               const sty_style_program *progs, uint32_t n_progs, BrSlots s) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t g = base + i;
    f3 out = {0.0f, 0.0f, 0.0f};
    const uint32_t prim = s.prim[g];
    if (prim != NONE) {
        F3 li = get3(s.rad, g);
        const uint32_t nc = s.nchild[g];
        if (nc) {
            F3 dsum = f3m(0.0f, 0.0f, 0.0f), isum = f3m(0.0f, 0.0f, 0.0f);
            const uint32_t c0 = cbase0 + s.cbase[g];
            for (uint32_t k = 0; k < nc; k++) {
                const uint32_t c = c0 + k;
                dsum = dsum + get3(s.dir, c);
                if (s.prim[c] != NONE) {
                    const F3 t = get3(s.thr, c), r = get3(s.rad, c);
                    isum = isum + f3m(t.x * r.x, t.y * r.y, t.z * r.z) * s.mis[c];
                }
            }
            li = li + (dsum + isum) * (1.0f / (float)nc);
        }
        out = {li.x, li.y, li.z};
        const uint32_t fl = s.flags[g];
        if (!(fl & 1u)) {
            const int32_t pi = sc.materials[sc.tri_material[prim]].style[style_index(fl)];
            if (pi >= 0 && (uint32_t)pi < n_progs) {
                const F3 p = get3(s.p, g);
                out = style_apply(progs[pi], depth, out, f3{p.x, p.y, p.z});
            }
        }
        put3(s.rad, g, f3m(out.x, out.y, out.z));
    } else if (depth == 0) {
        put3(s.rad, g, f3m(0.0f, 0.0f, 0.0f));
    }
}
// film += weight * sample for every sample of the pass, per pixel in repeat order (film.add_sample):
// the sequence of FP64 additions does not depend on how samples are grouped into passes
__global__ void k_br_film(uint32_t npx, uint64_t q0, uint32_t n, BrSlots s, double weight, double *film) {
    const uint32_t px = blockIdx.x * blockDim.x + threadIdx.x;
    if (px >= npx) return;
    uint64_t q = q0 + (px + npx - (uint32_t)(q0 % npx)) % npx;  // the pass's first sample of px
    double *fp = film + 3 * (size_t)px;
    for (; q < q0 + n; q += npx) {
        const size_t i = (size_t)(q - q0);
        fp[0] += weight * s.rad[0][i];
        fp[1] += weight * s.rad[1][i];
        fp[2] += weight * s.rad[2][i];
    }
}

}  // namespace
}  // namespace sty

using namespace sty;

sty_status sty_brpt_render(sty_scene *scene, const sty_brpt_config *cfg, const sty_style_program *programs,
                           uint32_t n_programs, double *film, sty_brpt_stats *stats, void *stream) {
    clear_error();
    STY_ARG_CHECK(scene && cfg && film, "sty_brpt_render: null argument");
    STY_ARG_CHECK(cfg->max_depth <= 64, "max_depth must be <= 64");
    STY_ARG_CHECK(cfg->n_levels >= 1 && cfg->n_levels <= STY_BRPT_MAX_LEVELS, "n_levels must be in [1, %d]",
                  STY_BRPT_MAX_LEVELS);
    for (uint32_t k = 0; k < cfg->n_levels; k++)
        STY_ARG_CHECK(cfg->inner_samples[k] >= 1 && cfg->inner_samples[k] <= 65536, "inner_samples[%u] must be in [1, 65536]",
                      k);
    STY_ARG_CHECK(cfg->repeats >= 1 && cfg->vram_mb >= 1, "repeats and vram_mb must be >= 1");
    STY_ARG_CHECK((uint64_t)cfg->first_repeat + cfg->repeats <= 0xFFFFFFFFull, "first_repeat + repeats overflows");
    STY_ARG_CHECK(n_programs <= 64 && (n_programs == 0 || programs), "bad style programs");
    for (uint32_t k = 0; k < n_programs; k++)
        STY_ARG_CHECK(style_program_valid(&programs[k]), "style program %u is invalid", k);
    const cudaStream_t st = as_stream(stream);
    const sty_camera &cam = scene_camera(scene);
    const uint32_t npx = cam.width * cam.height;
    // worst-case tree per pixel: every vertex rough and every ray hitting
    double worst = 0.0, level = 1.0;
    for (uint32_t d = 0; d <= cfg->max_depth; d++) {
        worst += level;
        level *= d < cfg->n_levels ? cfg->inner_samples[d] : 1.0;
    }
    const double budget = (double)cfg->vram_mb * 1048576.0 / kBrSlotBytes;
    uint64_t ppp = (uint64_t)(budget / worst);
    if (ppp == 0) {
        set_error("vram_mb (%u) is below one pixel's worst-case vertex tree (%.0f vertices)", cfg->vram_mb, worst);
        return STY_ERR_ARG;
    }
    ppp = std::min<uint64_t>(ppp, (uint64_t)npx * cfg->repeats);
    ppp = std::min<uint64_t>(ppp, (uint64_t)(2147483647.0 / worst));
    STY_ARG_CHECK(ppp >= 1, "vertex tree of one pixel exceeds 2^31 slots");
    const uint64_t cap = (uint64_t)((double)ppp * worst) + 2;  // (one slot behind the last for the scan's total)

    // slot planes, keys first (8-byte), in one workspace
    size_t scan_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (const uint32_t *)nullptr, (uint32_t *)nullptr, (uint32_t)cap);
    size_t at = 0;
    auto place = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 255) & ~(size_t)255;
        return o;
    };
    const size_t o_key = place(cap * 8), o_f = place(cap * 4 * 19), o_u = place(cap * 4 * 5),
                 o_prog = place(std::max<uint32_t>(n_programs, 1) * sizeof(sty_style_program)), o_count = place(16),
                 o_scan = place(scan_bytes);
    void *ws = nullptr;
    size_t ws_bytes = 0;
    STY_TRY(scene_take_workspace(scene, at, (size_t)cfg->vram_mb << 20, &ws, &ws_bytes));
    auto cleanup = [&]() { scene_give_workspace(scene, ws, ws_bytes); };
    char *const wp = static_cast<char *>(ws);
    BrSlots sl;
    sl.key = (uint64_t *)(wp + o_key);
    float *fpl = (float *)(wp + o_f);
    uint32_t *upl = (uint32_t *)(wp + o_u);
    sty_style_program *dprog = (sty_style_program *)(wp + o_prog);
    unsigned long long *dhits = (unsigned long long *)(wp + o_count), *dnext = dhits + 1;
    void *dscan = wp + o_scan;
    sty_status s = STY_OK;
    {
        int k = 0;
        auto fp = [&]() { return fpl + (size_t)(k++) * cap; };
        for (int a = 0; a < 3; a++) sl.p[a] = fp();
        for (int a = 0; a < 3; a++) sl.ng[a] = fp();
        for (int a = 0; a < 3; a++) sl.wo[a] = fp();
        for (int a = 0; a < 3; a++) sl.rad[a] = fp();
        for (int a = 0; a < 3; a++) sl.thr[a] = fp();
        for (int a = 0; a < 3; a++) sl.dir[a] = fp();
        sl.mis = fp();
        sl.prim = upl;
        sl.flags = upl + cap;
        sl.ab = upl + 2 * cap;
        sl.nchild = upl + 3 * cap;
        sl.cbase = upl + 4 * cap;
    }
    BrInner inner;
    inner.n = cfg->n_levels;
    for (uint32_t k = 0; k < STY_BRPT_MAX_LEVELS; k++) inner.v[k] = k < cfg->n_levels ? cfg->inner_samples[k] : 1u;
    const SceneView sv = scene_view(scene);
    const CamArgs ca = make_camera(cam);
    int dev = 0, sms = 0, per_sm = 0;
    if (s == STY_OK) s = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (s == STY_OK) s = check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr SMs");
    if (s == STY_OK)
        s = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_br_walk, kWalkThreads, 0), "k_br_walk occupancy");
    if (s != STY_OK) {
        cleanup();
        return s;
    }
    const uint64_t walk_blocks = (uint64_t)std::max(per_sm, 1) * sms;
    auto run = [&]() -> sty_status {
        if (n_programs)
            STY_TRY(check_cuda(cudaMemcpyAsync(dprog, programs, n_programs * sizeof(sty_style_program),
                                               cudaMemcpyHostToDevice, st), "upload programs"));
        STY_TRY(check_cuda(cudaMemsetAsync(dhits, 0, 8, st), "zero counter"));
        uint64_t slots = 0, passes = 0, max_pass = 0;
        const double weight = 1.0 / cfg->repeats;
        std::vector<uint32_t> cnt, off;
        const uint64_t total = (uint64_t)npx * cfg->repeats;
        {
            for (uint64_t q0 = 0; q0 < total; q0 += ppp) {
                const uint32_t P = (uint32_t)std::min<uint64_t>(ppp, total - q0);
                cnt.assign(1, P);
                off.assign(1, 0);
                (sv.any_closure ? k_br_camera<true> : k_br_camera<false>)<<<(P + 255) / 256, 256, 0, st>>>(
                    sv, ca, P, q0, npx, cfg->seed, cfg->first_repeat, cfg->max_depth, inner, sl, dhits);
                STY_TRY(check_launch("k_br_camera"));
                for (uint32_t d = 0; d <= cfg->max_depth; d++) {
                    const uint32_t n = cnt[d], base = off[d];
                    size_t tb = scan_bytes;
                    STY_TRY(check_cuda(cub::DeviceScan::ExclusiveSum(dscan, tb, sl.nchild + base, sl.cbase + base,
                                                                     n + 1, st),
                                       "scan branch counts"));
                    count_launch();
                    uint32_t next = 0;  // (below 2^31: the branch counts of a worst-case tree are)
                    STY_TRY(check_cuda(cudaMemcpyAsync(&next, sl.cbase + base + n, 4, cudaMemcpyDeviceToHost, st),
                                       "read total"));
                    STY_TRY(check_cuda(cudaStreamSynchronize(st), "sync"));
                    if (next == 0) break;
                    if ((uint64_t)base + n + next + 1 > cap) {
                        set_error("vertex tree overflow (%llu slots, capacity %llu)",
                                  (unsigned long long)(base + n + next), (unsigned long long)cap);
                        return STY_ERR_ITER_LIMIT;
                    }
                    off.push_back(base + n);
                    cnt.push_back(next);
                    const unsigned blocks = (next + 255) / 256;
                    (sv.any_closure ? k_br_sample<true> : k_br_sample<false>)<<<blocks, 256, 0, st>>>(
                        sv, next, base, n, base + n, d, dprog, n_programs, sl, dnext);
                    STY_TRY(check_launch("k_br_sample"));
                    const uint64_t need = (2 * (uint64_t)next + kWalkThreads - 1) / kWalkThreads;
                    k_br_walk<<<(unsigned)std::min<uint64_t>(need, walk_blocks), kWalkThreads, 0, st>>>(
                        sv, next, base + n, sl, dnext);
                    STY_TRY(check_launch("k_br_walk"));
                    (sv.any_closure ? k_br_vertex<true> : k_br_vertex<false>)<<<blocks, 256, 0, st>>>(
                        sv, next, base, n, base + n, d, cfg->max_depth, inner, sl, dhits);
                    STY_TRY(check_launch("k_br_vertex"));
                }
                for (int d = (int)cnt.size() - 1; d >= 0; d--) {
                    const uint32_t cb = (size_t)d + 1 < off.size() ? off[d + 1] : 0u;
                    k_br_propagate<<<(cnt[d] + 255) / 256, 256, 0, st>>>(sv, cnt[d], off[d], cb, (uint32_t)d, dprog,
                                                                         n_programs, sl);
                    STY_TRY(check_launch("k_br_propagate"));
                }
                k_br_film<<<(npx + 255) / 256, 256, 0, st>>>(npx, q0, P, sl, weight, film);
                STY_TRY(check_launch("k_br_film"));
                uint64_t pass_slots = 0;
                for (uint32_t c : cnt) pass_slots += c;
                slots += pass_slots;
                max_pass = std::max(max_pass, pass_slots);
                passes++;
            }
        }
        if (stats) {
            unsigned long long h = 0;
            STY_TRY(check_cuda(cudaMemcpyAsync(&h, dhits, 8, cudaMemcpyDeviceToHost, st), "read counter"));
            STY_TRY(check_cuda(cudaStreamSynchronize(st), "sync"));
            stats->vertices = h;
            stats->slots = slots;
            stats->passes = passes;
            stats->pixels_per_pass = ppp;
            stats->max_pass_slots = max_pass;
        }
        return check_cuda(cudaStreamSynchronize(st), "sty_brpt_render");
    };
    s = run();
    cudaStreamSynchronize(st);
    cleanup();
    return s;
}
