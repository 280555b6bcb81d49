// scene.cuh -- device view of a scene: 4-wide BVH nodes, triangles, materials; watertight intersection.
#pragma once

#include "bvh.cuh"
#include "common.cuh"

namespace sty {

struct TriGeom {        // 48 bytes, triangle slot order (BVH leaf order)
    float4 v0;          // w = original triangle id (as bits)
    float4 v1;
    float4 v2;
};

struct SceneView {
    const BvhNode *nodes;
    const TriGeom *tris;            // slot order
    const uint32_t *tri_material;   // by original id
    const float *tri_normal;        // by original id, 3 per triangle (unit geometric normal)
    const float *tri_area;          // by original id
    const sty_scene_material *materials;
    uint32_t n_tris, n_materials;
    // emitters: triangles with non-zero emission, sampled by area x luminance (CDF)
    const uint32_t *light_tris;     // original ids
    const float *light_cdf;         // n_lights + 1 entries, cdf[0] = 0, cdf[n] = 1
    uint32_t n_lights;
    const float *tri_pos;           // by original id, 9 per triangle
    const float *ggx_tab;           // the principled BSDF's albedo table (bsdf.cuh)
    uint32_t any_closure;           // some material is STY_MAT_PRINCIPLED / STY_MAT_GLASS
};

struct Hit {
    float t, b1, b2;
    uint32_t prim;  // original id, 0xffffffff = miss
};

// Watertight ray/triangle intersection (Woop, Benthin, Wald 2013) in explicitly rounded f32 with the
// double-precision fallback when an edge function is exactly zero. Returns true and updates *hit
// when the triangle is hit in (tmin, hit->t) or at hit->t with a lower id.
// The test's axis permutation is the rotation that brings the largest direction component last. (Swapping
// the first two axes for a negative one, as published, negates U, V, W, det and T exactly and changes
// nothing that is derived from them.)
struct RayPre {
    float o[3];  // rotated
    int kz;
    float Sx, Sy, Sz;
    float tmin;
};
template <typename T>
__host__ __device__ __forceinline__ void rotate3(int kz, T x, T y, T z, T &rx, T &ry, T &rz) {
    rx = kz == 0 ? y : kz == 1 ? z : x;
    ry = kz == 0 ? z : kz == 1 ? x : y;
    rz = kz == 0 ? x : kz == 1 ? y : z;
}
__host__ __device__ inline RayPre ray_pre(const float o[3], const float d[3], float tmin) {
    RayPre r;
    const float ax = fabsf(d[0]), ay = fabsf(d[1]), az = fabsf(d[2]);
    int kz = 0;
    if (ay > ax) kz = 1;
    if (az > (kz == 0 ? ax : ay)) kz = 2;
    r.kz = kz;
    rotate3(kz, o[0], o[1], o[2], r.o[0], r.o[1], r.o[2]);
    float dx, dy, dz;
    rotate3(kz, d[0], d[1], d[2], dx, dy, dz);
#ifdef __CUDA_ARCH__
    r.Sx = __fdiv_rn(dx, dz);
    r.Sy = __fdiv_rn(dy, dz);
    r.Sz = __fdiv_rn(1.0f, dz);
#else
    r.Sx = dx / dz;
    r.Sy = dy / dz;
    r.Sz = 1.0f / dz;
#endif
    r.tmin = tmin;
    return r;
}

#ifdef __CUDA_ARCH__
#define STY_FM(a, b) __fmul_rn(a, b)
#define STY_FS(a, b) __fsub_rn(a, b)
#define STY_FA(a, b) __fadd_rn(a, b)
#define STY_FD(a, b) __fdiv_rn(a, b)
#define STY_DFMS(a, b, c, d) __dsub_rn(__dmul_rn(a, b), __dmul_rn(c, d))
#else
#define STY_DFMS(a, b, c, d) ((a) * (b) - (c) * (d))
#define STY_FM(a, b) ((a) * (b))
#define STY_FS(a, b) ((a) - (b))
#define STY_FA(a, b) ((a) + (b))
#define STY_FD(a, b) ((a) / (b))
#endif

__host__ __device__ inline bool intersect_tri(const RayPre &r, const float v0[3], const float v1[3], const float v2[3],
                                              uint32_t prim, Hit *hit) {
    float p[3], q[3], w[3];
    rotate3(r.kz, v0[0], v0[1], v0[2], p[0], p[1], p[2]);
    rotate3(r.kz, v1[0], v1[1], v1[2], q[0], q[1], q[2]);
    rotate3(r.kz, v2[0], v2[1], v2[2], w[0], w[1], w[2]);
    const float Ak = STY_FS(p[2], r.o[2]), Bk = STY_FS(q[2], r.o[2]), Ck = STY_FS(w[2], r.o[2]);
    const float Ax = STY_FS(STY_FS(p[0], r.o[0]), STY_FM(r.Sx, Ak)), Ay = STY_FS(STY_FS(p[1], r.o[1]), STY_FM(r.Sy, Ak));
    const float Bx = STY_FS(STY_FS(q[0], r.o[0]), STY_FM(r.Sx, Bk)), By = STY_FS(STY_FS(q[1], r.o[1]), STY_FM(r.Sy, Bk));
    const float Cx = STY_FS(STY_FS(w[0], r.o[0]), STY_FM(r.Sx, Ck)), Cy = STY_FS(STY_FS(w[1], r.o[1]), STY_FM(r.Sy, Ck));
    float U = STY_FS(STY_FM(Cx, By), STY_FM(Cy, Bx));
    float V = STY_FS(STY_FM(Ax, Cy), STY_FM(Ay, Cx));
    float W = STY_FS(STY_FM(Bx, Ay), STY_FM(By, Ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {  // fall back to double on exact zeros
        U = (float)STY_DFMS((double)Cx, (double)By, (double)Cy, (double)Bx);
        V = (float)STY_DFMS((double)Ax, (double)Cy, (double)Ay, (double)Cx);
        W = (float)STY_DFMS((double)Bx, (double)Ay, (double)By, (double)Ax);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    const float det = STY_FA(STY_FA(U, V), W);
    if (det == 0.0f) return false;
    const float Az = STY_FM(r.Sz, Ak), Bz = STY_FM(r.Sz, Bk), Cz = STY_FM(r.Sz, Ck);
    const float T = STY_FA(STY_FA(STY_FM(U, Az), STY_FM(V, Bz)), STY_FM(W, Cz));
    const float t = STY_FD(T, det);
    if (!(t > r.tmin)) return false;
    if (t > hit->t || (t == hit->t && prim >= hit->prim)) return false;
    hit->t = t;
    hit->b1 = STY_FD(V, det);
    hit->b2 = STY_FD(W, det);
    hit->prim = prim;
    return true;
}

// Slab tests of a node's children. Per axis and child the two planes' distances are fma(f, k, b) with
// f = 1 + q 2^-15 made from the byte q by one permute; near and far planes are picked by the
// direction's sign, so a NaN (a box or an origin without finite coordinates) drops the axis from fmaxf /
// fminf, and the child is kept. Entry and exit are widened by 2^-20 of themselves, which covers the
// rounding of k and b where the origin is far from the box along the axis; where it is not, their
// rounding is below a grid step, the boxes' own margin.
struct RayBox {
    float o[3], inv[3];
};
__device__ __forceinline__ RayBox ray_box(const float o[3], const float d[3]) {
    RayBox r;
    // A direction component of (nearly) 0 beside the others as 1e-24 of the largest: finite, so that the axis still excludes
    // the boxes the ray passes; the boxes' margin keeps those it lies in or touches. Where that underflows (directions
    // below 1e-14) the inverse is infinite, every plane's distance a NaN, and the axis excludes nothing.
    const float least = 1e-24f * fmaxf(fmaxf(fabsf(d[0]), fabsf(d[1])), fabsf(d[2]));
#pragma unroll
    for (int a = 0; a < 3; a++) {
        r.o[a] = o[a];
        const float v = copysignf(fmaxf(fabsf(d[a]), least), d[a]);
        // the approximate reciprocal of the whole range, subnormal results among it (__fdividef gives 0 past 2^126); its
        // error scales both planes alike, far below the widening
        asm("rcp.approx.f32 %0, %1;" : "=f"(r.inv[a]) : "f"(v));
    }
    return r;
}
struct NodeData {
    uint4 a, b, c, d;
};
__device__ __forceinline__ NodeData node_load(const BvhNode *n) {
    const uint4 *p = reinterpret_cast<const uint4 *>(n);
    return {__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3)};
}
// entry distances of the children whose box meets [tmin, tmax]; returns their mask
__device__ __forceinline__ uint32_t node_hits(const NodeData &n, const RayBox &r, float tmin, float tmax, float (&tn)[4]) {
    const float org[3] = {__uint_as_float(n.a.x), __uint_as_float(n.a.y), __uint_as_float(n.a.z)};
    const uint32_t lo[3] = {n.b.x, n.b.y, n.b.z}, hi[3] = {n.b.w, n.c.x, n.c.y};
    float k[3], b[3];
    uint32_t nw[3], fw[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        k[a] = r.inv[a] * __uint_as_float(((n.a.w >> (8 * a)) & 0xffu) << 23) * 32768.0f;
        b[a] = (org[a] - r.o[a]) * r.inv[a] - k[a];
        const bool neg = r.inv[a] < 0.0f;
        nw[a] = neg ? hi[a] : lo[a];
        fw[a] = neg ? lo[a] : hi[a];
    }
    const uint32_t nc = n.a.w >> 24;
    uint32_t mask = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        float t0 = tmin, t1 = tmax;
        float e0 = -3.0e38f, e1 = 3.0e38f;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const uint32_t sel = 0x7604u | ((uint32_t)c << 4);
            e0 = fmaxf(e0, fmaf(__uint_as_float(__byte_perm(nw[a], 0x3f800000u, sel)), k[a], b[a]));
            e1 = fminf(e1, fmaf(__uint_as_float(__byte_perm(fw[a], 0x3f800000u, sel)), k[a], b[a]));
        }
        t0 = fmaxf(t0, fmaf(fabsf(e0), -9.5367432e-07f, e0));
        t1 = fminf(t1, fmaf(fabsf(e1), 9.5367432e-07f, e1));
        tn[c] = t0;
        if ((uint32_t)c < nc && t0 <= t1) mask |= 1u << c;
    }
    return mask;
}
__device__ __forceinline__ uint32_t node_child(const NodeData &n, int c) {
    return c == 0 ? n.c.z : c == 1 ? n.c.w : c == 2 ? n.d.x : n.d.y;
}
// One ray's walk through the tree. Stack entries: node index or first triangle slot, and the entry distance
// with the triangle count (0: a node) in its last 3 bits (rounded down, so nothing is culled that would
// not have been). `ex0`, `ex1`: original ids skipped.
struct Walk {
    RayPre rp;
    RayBox rb;
    Hit h;
    uint32_t ex0, ex1;
    uint2 cur;
    int sp;
    __device__ __forceinline__ void start(const float o[3], const float d[3], float tmin, float tmax, uint32_t e0, uint32_t e1) {
        h.t = tmax;
        h.prim = 0xffffffffu;
        h.b1 = h.b2 = 0.0f;
        rp = ray_pre(o, d, tmin);
        rb = ray_box(o, d);
        ex0 = e0;
        ex1 = e1;
        cur = make_uint2(0u, 0u);  // the root: node 0 (count 0: internal)
        sp = 0;
    }
    __device__ __forceinline__ bool at_node() const { return (cur.y & 7u) == 0; }
    // the next entry that can hold a hit; false if there is none
    __device__ __forceinline__ bool pop(const uint2 *stack) {
        float te;  // (an entry distance of 0 may stand for one below 0: never culled)
        do {
            if (sp == 0) return false;
            cur = stack[--sp];
            te = __uint_as_float(cur.y & ~7u);
        } while (te > 0.0f && te > h.t * (1.0f + 1e-6f));
        return true;
    }
    // to the nearest child of the node the ray meets, the others on the stack, far ones first; false when done
    __device__ __forceinline__ bool node(const SceneView &s, uint2 *stack) {
        const NodeData n = node_load(s.nodes + cur.x);
        float tn[4];
        // cull against a slightly inflated best distance: a flat leaf box's entry can round one ulp
        // past a triangle hit at exactly the best distance (a tie on a shared edge), and the lower id
        // must still be found
        const uint32_t mask = node_hits(n, rb, rp.tmin, h.t * (1.0f + 1e-6f), tn);
        // keys: entry distance (positive, or 0 after clamping) with the child number in the last 2 bits
        uint32_t key[4];
#pragma unroll
        for (int c = 0; c < 4; c++)
            key[c] = (mask >> c) & 1u ? ((__float_as_uint(fmaxf(tn[c], 0.0f)) & ~3u) | (uint32_t)c) : 0xffffffffu;
        auto order = [&](int i, int j) {
            const uint32_t a = min(key[i], key[j]), b = max(key[i], key[j]);
            key[i] = a;
            key[j] = b;
        };
        order(0, 1);
        order(2, 3);
        order(0, 2);
        order(1, 3);
        order(1, 2);
        if (key[0] == 0xffffffffu) return pop(stack);
        auto entry = [&](uint32_t kk) {
            const int c = (int)(kk & 3u);
            return make_uint2(node_child(n, c), (kk & ~7u) | ((n.d.z >> (8 * c)) & 7u));
        };
#pragma unroll
        for (int i = 3; i > 0; i--)
            if (key[i] != 0xffffffffu && sp < kStack) stack[sp++] = entry(key[i]);
        cur = entry(key[0]);
        return true;
    }
    // the leaf's next triangle, which leaves the leaf; true if it became the hit
    __device__ __forceinline__ bool triangle(const SceneView &s) {
        const float4 *tg = reinterpret_cast<const float4 *>(s.tris + cur.x);
        const float4 v0 = __ldg(tg), v1 = __ldg(tg + 1), v2 = __ldg(tg + 2);
        cur.x++;
        cur.y--;
        const uint32_t id = __float_as_uint(v0.w);
        if (id == ex0 || id == ex1) return false;
        const float a0[3] = {v0.x, v0.y, v0.z}, a1[3] = {v1.x, v1.y, v1.z}, a2[3] = {v2.x, v2.y, v2.z};
        return intersect_tri(rp, a0, a1, a2, id, &h);
    }
    // the leaf's triangles; true if one of them became the hit
    __device__ __forceinline__ bool leaf(const SceneView &s) {
        bool any = false;
        while (!at_node()) any = triangle(s) || any;
        return any;
    }
};

// Closest hit in (tmin, tmax]; `exclude` = original id skipped (the triangle the ray leaves). The hit is the
// least (t, id) of all triangles the ray meets, whatever order the walk takes.
__device__ inline Hit trace_closest(const SceneView &s, const float o[3], const float d[3], float tmin, float tmax,
                                    uint32_t exclude) {
    uint2 stack[kStack];
    Walk w;
    w.start(o, d, tmin, tmax, exclude, exclude);
    for (;;) {
        while (w.at_node())
            if (!w.node(s, stack)) return w.h;
        w.leaf(s);
        if (!w.pop(stack)) return w.h;
    }
}

// Any hit in (tmin, tmax] skipping two triangles (shadow rays).
__device__ inline bool trace_any(const SceneView &s, const float o[3], const float d[3], float tmin, float tmax,
                                 uint32_t ex0, uint32_t ex1) {
    uint2 stack[kStack];
    Walk w;
    w.start(o, d, tmin, tmax, ex0, ex1);
    for (;;) {
        while (w.at_node())
            if (!w.node(s, stack)) return false;
        if (w.leaf(s)) return true;
        if (!w.pop(stack)) return false;
    }
}

SceneView scene_view(const sty_scene *s);
// A device workspace of at least `bytes`: the one the scene has parked, unless that is larger than `most` (and than
// `bytes`), or a new one. It belongs to the call until it gives it back, which it does when no work on it is in flight. A scene
// keeps one of at most 8 GB until it is trimmed or destroyed, or until an allocation of this library finds memory short
// (release_workspaces); others are freed. Safe from several threads.
sty_status scene_take_workspace(sty_scene *s, size_t bytes, size_t most, void **ptr, size_t *got);
void scene_give_workspace(sty_scene *s, void *ptr, size_t bytes);
// device buffers kept by a scene between renders (defined in trace.cu)
void render_cache_free(void *cache);

}  // namespace sty
