// Device side of the bake: the resident scene, the ray queries and per-texel visibility.
//
// Ray queries restate the reference's Occluders (src/bake/occluder.rs:171-251): two-sided
// Möller–Trumbore with hits for 0 <= t <= max, any-hit for shadow rays, closest-hit with ties
// going to the lowest occluder index, optional alpha test. The BVH only prunes: node boxes are
// padded and the slab test keeps a relative slack, so no triangle the exact test would report is
// ever culled and results equal a scan over every occluder.
#pragma once

#include <cuda_runtime.h>

#include "dl_host.hpp"
#include "dl_math.cuh"
#include "dl_slab.hpp"

namespace dl {

// Everything the kernels read, as device pointers (one struct passed by value).
struct DevScene {
    // BVH and triangles in leaf order
    const TravNode *nodes;
    // triangles as 3 float4 each, one 48-byte record per triangle (a leaf's triangles are
    // contiguous): v0 (w: occluder index bits), e1 = v1 - v0, e2 = v2 - v0
    const float4 *tris;
    uint32_t occluders;
    // occluder index -> mesh, triangle in mesh, position in leaf order
    const uint32_t *occ_mesh, *occ_tri, *occ_leaf;
    // meshes (sorted order)
    uint32_t mesh_count;
    const uint32_t *mesh_vertex_base, *mesh_index_base, *mesh_tri_base, *mesh_res;
    const uint32_t *mesh_flags;  // kMesh* bits
    const uint64_t *mesh_id;
    const float *mesh_albedo;     // 3 per mesh
    const uint32_t *mesh_alpha;   // 4 per mesh: byte offset, width, height, cutoff bits
    const uint8_t *alpha_pool;
    // vertex data (global vertex index = base + local)
    const float *positions, *normals, *uv1, *uv0;  // 3, 3, 2, 2 per vertex
    const uint32_t *indices;                       // local vertex indices
    // triangles
    uint32_t triangles;
    const uint32_t *tri_mesh;
    // lights in slot order
    uint32_t light_count, local_lights;
    const DevLight *lights;
    // options
    uint64_t seed;
    uint32_t area_samples, area_min_samples, sky_samples;
    uint32_t colored_bounce;
    // refined form: the epsilon of the binary64 re-test and its square
    float refine_eps, refine_eps2;
    // the coherent order (sky_sample_order) of a sky count beyond kMaxOrdered, or null
    const uint16_t *sky_order;
    // sample_cells (dl_host.hpp) for n = 16, 32, ..., kMaxOrdered back to back (n's start at n - 16)
    const uint16_t *order_cells, *cell_samples;
};
constexpr uint32_t kMaxOrdered = 4096;
// The net that n samples are traced in the coherent order of: n itself when it is a power of two, else
// the next one, as long as n fills five eighths of it (a lane idles where the order's sample is n or
// more); 0: no such net. The first n points of the sequence are the first n of any larger net. Where the line
// lies, on a 77 k triangle terrain: sky samples 144, 160, 176, 192 in the net of 256 20.3, 20.7, 21.1, 21.6 ms, in
// index order 19.3, 21.3, 23.3, 25.3 ms; sun bounces of 72, 80, 88, 96 in the net of 128 14.4, 14.9, 15.4, 15.9 ms, in
// index order 14.3, 15.9, 17.5, 19.1 ms.
__host__ __device__ __forceinline__ uint32_t ordered_net(uint32_t n, uint32_t least, uint32_t most) {
    uint32_t net = least;
    while (net < n && net < most) net *= 2;
    return n <= net && 8ull * n >= 5ull * net ? net : 0;
}
// The shift of a net of n samples (n a power of two from 16 to kMaxOrdered) by `off` in whole
// cells, packed as x | y << 8 | xbits << 16 | ybits << 24.
__device__ __forceinline__ uint32_t net_shift(uint32_t n, f2 off) {
    uint32_t m = 31 - __clz(n), xb = (m + 1) / 2, yb = m / 2;
    uint32_t sx = min((1u << xb) - 1, (uint32_t)(off.x * (float)(1u << xb)));
    uint32_t sy = min((1u << yb) - 1, (uint32_t)(off.y * (float)(1u << yb)));
    return sx | sy << 8 | xb << 16 | yb << 24;
}
// Sample of rank k of a net of n samples shifted by `shift` (net_shift): the point of the cell of
// rank k moved back by the shift, so that texels with different shifts send their rank-k rays in
// about the same direction. A permutation of 0 .. n-1 over k.
__device__ __forceinline__ uint32_t shifted_sample(const DevScene &sc, uint32_t n, uint32_t shift, uint32_t k) {
    const uint32_t c = sc.order_cells[n - 16 + k];
    const uint32_t xb = (shift >> 16) & 0xFFu, yb = shift >> 24;
    const uint32_t cx = ((c & 0xFFu) - (shift & 0xFFu)) & ((1u << xb) - 1u);
    const uint32_t cy = ((c >> 8) - ((shift >> 8) & 0xFFu)) & ((1u << yb) - 1u);
    return sc.cell_samples[n - 16 + (cy << xb | cx)];
}
enum : uint32_t { kMeshNormals = 1, kMeshOccludes = 2, kMeshAlpha = 4 };

__device__ __forceinline__ float4 ldg4(const float4 *p) { return __ldg(p); }

// AlphaTexture::is_opaque (src/bake/input.rs:79-97) at the hit's interpolated UV0.
__device__ __forceinline__ uint32_t wrap_texel(float coordinate, uint32_t size) {
    float r = fmodf(coordinate, 1.0f);
    if (r < 0.0f) r = r + 1.0f;
    float t = floorf(r * (float)size);
    if (isfinite(t)) {
        uint32_t u = f2u(t);
        return u < size - 1 ? u : size - 1;
    }
    return 0;
}
__device__ __noinline__ bool alpha_blocks(const DevScene &sc, uint32_t occ, float u, float v) {
    uint32_t m = sc.occ_mesh[occ];
    if (!(sc.mesh_flags[m] & kMeshAlpha)) return true;
    const uint32_t *tex = sc.mesh_alpha + m * 4;
    uint32_t width = tex[1], height = tex[2];
    if (width == 0 || height == 0) return true;
    const uint32_t *c = sc.indices + sc.mesh_index_base[m] + (size_t)sc.occ_tri[occ] * 3;
    uint32_t vb = sc.mesh_vertex_base[m];
    float wx = 1.0f - u - v;
    const float *a = sc.uv0 + (size_t)(vb + c[0]) * 2, *b = sc.uv0 + (size_t)(vb + c[1]) * 2,
                *d = sc.uv0 + (size_t)(vb + c[2]) * 2;
    float uvx = a[0] * wx + b[0] * u + d[0] * v;
    float uvy = a[1] * wx + b[1] * u + d[1] * v;
    uint32_t x = wrap_texel(uvx, width), y = wrap_texel(uvy, height);
    uint8_t alpha = sc.alpha_pool[tex[0] + (size_t)y * width + x];
    return (float)alpha / 255.0f >= __uint_as_float(tex[3]);
}

// intersect (occluder.rs:225-251) on a triangle stored as v0, e1 = v1 - v0, e2 = v2 - v0.
__device__ __forceinline__ bool tri_test(float4 v0, float4 e1v, float4 e2v, f3 o, f3 d, float max, float &t,
                                         float &u, float &v) {
    f3 e1{e1v.x, e1v.y, e1v.z}, e2{e2v.x, e2v.y, e2v.z};
    f3 p = cross(d, e2);
    float det = dot(e1, p);
    if (det == 0.0f || !isfinite(det)) return false;
    float inv = 1.0f / det;
    f3 s{o.x - v0.x, o.y - v0.y, o.z - v0.z};
    u = dot(s, p) * inv;
    if (!(u >= 0.0f && u <= 1.0f)) return false;
    f3 q = cross(s, e1);
    v = dot(d, q) * inv;
    if (v < 0.0f || u + v > 1.0f) return false;
    t = dot(e2, q) * inv;
    return t >= 0.0f && t <= max;
}

struct Hit {
    float t, u, v;
    uint32_t occluder;
};

// Node visits and triangle tests of traversals, counted only in the instrumented kernel variant
// the benchmark uses for its roofline bytes; `retests` counts the refined form's binary64
// re-tests.
struct Visits {
    unsigned long long nodes, tris, retests;
};

// The ray/triangle test of occluder `occ` in binary64 on its original vertices (the stored
// e1/e2 are rounded binary32 differences). The operation order is intersect's; u, v and t are
// rounded to binary32 once at the end.
__device__ __noinline__ bool tri_test_fp64(const DevScene &sc, uint32_t occ, f3 o, f3 d, float max, float &t,
                                           float &u, float &v) {
    uint32_t m = sc.occ_mesh[occ];
    const uint32_t *c = sc.indices + sc.mesh_index_base[m] + (size_t)sc.occ_tri[occ] * 3;
    uint32_t vb = sc.mesh_vertex_base[m];
    const float *pa = sc.positions + (size_t)(vb + c[0]) * 3, *pb = sc.positions + (size_t)(vb + c[1]) * 3,
                *pc = sc.positions + (size_t)(vb + c[2]) * 3;
    d3 a{pa[0], pa[1], pa[2]};
    d3 e1 = sub(d3{pb[0], pb[1], pb[2]}, a), e2 = sub(d3{pc[0], pc[1], pc[2]}, a);
    d3 dd = widen(d);
    d3 p = cross(dd, e2);
    double det = dot(e1, p);
    if (det == 0.0 || !isfinite(det)) return false;
    double inv = 1.0 / det;
    d3 s = sub(widen(o), a);
    double ud = dot(s, p) * inv;
    if (!(ud >= 0.0 && ud <= 1.0)) return false;
    d3 q = cross(s, e1);
    double vd = dot(dd, q) * inv;
    if (vd < 0.0 || ud + vd > 1.0) return false;
    double td = dot(e2, q) * inv;
    if (!(td >= 0.0 && td <= (double)max)) return false;
    t = (float)td;
    u = (float)ud;
    v = (float)vd;
    return true;
}

// The refined form's test: the binary32 test decides unless the ray is nearly parallel to the
// plane (|det| <= eps |e1| |d x e2|) or u, v, u + v or t lie within eps of their bounds (t's
// margin is eps * max(1, max) for a finite max, eps otherwise); those rays are re-tested in
// binary64. Outside the margins the binary32 verdict and hit equal tri_test's. `err` bounds how far a
// binary32 t may be from the binary64 test's (0 for a re-tested one; infinite where it has no bound).
__device__ __forceinline__ bool tri_test_refined(const DevScene &sc, float4 v0, float4 e1v, float4 e2v, f3 o, f3 d,
                                                 float max, float &t, float &u, float &v, Visits *vis, float &err) {
    const float eps = sc.refine_eps;
    f3 e1{e1v.x, e1v.y, e1v.z}, e2{e2v.x, e2v.y, e2v.z};
    f3 p = cross(d, e2);
    float det = dot(e1, p);
    err = 0.0f;
    if (det * det > sc.refine_eps2 * (dot(e1, e1) * dot(p, p))) {
        float inv = 1.0f / det;
        f3 s{o.x - v0.x, o.y - v0.y, o.z - v0.z};
        u = dot(s, p) * inv;
        if (!(u >= -eps && u <= 1.0f + eps)) return false;
        f3 q = cross(s, e1);
        v = dot(d, q) * inv;
        if (!(v >= -eps) || u + v > 1.0f + eps) return false;
        t = dot(e2, q) * inv;
        float margin = eps * (isfinite(max) ? fmaxf(max, 1.0f) : 1.0f);
        if (!(t >= -margin && t <= max + margin)) return false;
        bool near = u < eps || u > 1.0f - eps || v < eps || u + v > 1.0f - eps || t < margin || t > max - margin;
        if (!near) {
            // numerator and determinant are sums of products rounded a few times each, within 8 * 2^-24 of
            // |s||e1||e2| and |d||e1||e2| (the edges' own rounding included); 2^-20 leaves a factor of 2
            const float size1 = fabsf(e1.x) + fabsf(e1.y) + fabsf(e1.z), size2 = fabsf(e2.x) + fabsf(e2.y) + fabsf(e2.z);
            const float sizes = fabsf(s.x) + fabsf(s.y) + fabsf(s.z);
            const float unit = size1 * size2 * fabsf(inv) * 9.5367431640625e-07f;  // 2^-20
            err = unit < 0.005f ? unit * (sizes + 1.75f * fabsf(t)) + fabsf(t) * 2.384185791015625e-07f : INFINITY;
            return true;
        }
    }
    ++vis->retests;
    return tri_test_fp64(sc, __float_as_uint(v0.w), o, d, max, t, u, v);
}

// Entries of a traversal stack (>= BVH depth; the host refuses deeper trees). A thread's stack is local
// memory: a ray holds a few entries of the 8 to 28 that its tree could need, and only the lines in use take
// room in L1, where shared stacks took their worst case from it for every resident thread (14 KB a block
// of the outdoor level, 140 KB of the SM's 256). Shared -> local: a 77 k triangle terrain's visibility 24.6 ->
// 23.5 ms at 10 blocks, the rooms' local gather 24.9 -> 23.7 ms at 8, rooms under panels and tubes 6.4 -> 6.2 ms.
constexpr int kStack = 64;

// A node's 64 bytes in two 32-byte loads.
struct NodeData {
    Pair c0, c1, h0, h1, cz, hz;
    int ref0, ref1;
};
__device__ __forceinline__ NodeData load_node(const TravNode *n) {
    NodeData d;
    Pair refs, zero;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
        : "=l"(d.c0), "=l"(d.c1), "=l"(d.h0), "=l"(d.h1)
        : "l"(n));
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
        : "=l"(d.cz), "=l"(d.hz), "=l"(refs), "=l"(zero)
        : "l"(reinterpret_cast<const char *>(n) + 32));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(d.ref0), "=r"(d.ref1) : "l"(refs));
    return d;
}

// Takes a closest-hit candidate of the refined form against the nearest so far: true when it is the
// nearer one. The form orders candidates by the binary64 test's distance (rounded to binary32, ties to
// the lowest occluder) and takes the winner's barycentrics from it. Binary64 runs at a small fraction
// of binary32's rate here, and inside the traversal for a few lanes at a time, so a candidate keeps its
// binary32 distance while that and its error bound leave the order beyond doubt, and only the winner
// is tested in binary64, after the loops, with the warp's other winners. Where the order is open both are
// tested at once, and alpha-tested candidates always are. `lost`: a nearest candidate that
// binary64 then rejected may have hidden others; the caller traverses again, testing EACH candidate in
// binary64. Testing every candidate where it was met took 58.5 ms for the bounce-refined terrain's
// gather, this takes 29.9 ms; the refined decals' gather 29.4 ms and 16.2 ms, their burial 2.3 ms and 1.0 ms.
template <bool EACH>
__device__ __forceinline__ bool refined_candidate(const DevScene &sc, f3 o, f3 d, float max, bool alpha, Visits *vis,
                                                  uint32_t occ, float &t, float &u, float &v, float &terr, bool &found,
                                                  Hit &hit, float &err, bool &lost) {
    auto exact = [&]() {
        if (terr == 0.0f) return true;
        ++vis->retests;
        terr = 0.0f;
        return tri_test_fp64(sc, occ, o, d, max, t, u, v);
    };
    if ((EACH || alpha || !isfinite(t) || !isfinite(terr)) && !exact()) return false;
    if (alpha && !alpha_blocks(sc, occ, u, v)) return false;
    if (!found) return true;
    if (t + terr < hit.t - err) return true;
    if (t - terr > hit.t + err) return false;
    if (!exact()) return false;
    if (err > 0.0f) {
        ++vis->retests;
        err = 0.0f;
        if (!tri_test_fp64(sc, hit.occluder, o, d, max, hit.t, hit.u, hit.v) || !isfinite(hit.t)) {
            lost = true;
            found = false;
            hit.t = INFINITY;
            return true;
        }
    }
    return t < hit.t || (t == hit.t && occ < hit.occluder);
}

// How a warp's lanes leave the traversal's two loops. Most of its idle lanes wait at their border (14 of 32
// threads active). kFew: the last lanes still among inner nodes, when fewer than 8, wait for the others'
// leaves, which shorten those rays' ranges and bring their lanes back: a 77 k triangle terrain's sun gather 19.6 ms
// plain, 18.5, 18.2, 18.3 ms at 4, 8, 12; other closest hits gain nothing (burial in rooms 0.38 -> 0.42 ms,
// photons 3.32 -> 3.39 ms), any-hit rays lose 6 %. kOneLeaf: back to inner nodes after one leaf: the sun gather's shadow
// rays (its 18.2 -> 17.7 ms), rays towards local lights and the local gather's, whose directions differ from lane to
// lane (36 rooms' 48.8 -> 41.7 ms; holding a first leaf back until every lane has one, with votes among lanes named
// beforehand, 48.1 ms); the sky's and the sun's lose 2 to 10 %.
enum class NodeLoop { kPlain, kFew, kOneLeaf };

template <bool COUNT>
__device__ bool traverse_each(const DevScene &sc, f3 o, f3 dir, float max, bool alpha, int *stack, Hit &hit,
                              Visits *vis);

// Any-hit (ANY) or closest-hit traversal of the BVH2. Child references: >= 0 an inner node,
// < 0 a leaf ~(first << 3 | count). `stack` is this thread's kStack entries in local
// memory. For closest-hit, `hit` gets the nearest t (ties to the lowest
// occluder index, as occluder.rs:205-210) and that test's barycentrics, which equal the ones
// the reference recomputes with max = infinity.
template <bool ANY, bool COUNT = false, bool REFINE = false, bool EACH = false, NodeLoop LOOP = NodeLoop::kPlain>
__device__ bool traverse(const DevScene &sc, f3 o, f3 dir, float max, bool alpha, int *stack, Hit &hit,
                         Visits *vis = nullptr) {
    hit.t = INFINITY;
    hit.u = hit.v = 0.0f;
    hit.occluder = 0xFFFFFFFFu;
    if (sc.occluders == 0) return false;
    f3 d{dir.x + 0.0f, dir.y + 0.0f, dir.z + 0.0f};  // -0 -> +0 (occluder.rs:171-178)
    const RaySlabs slabs = ray_slabs(o, d);
    float tmax = fmaxf(max, 0.0f);
    float err = 0.0f;  // refined closest hits: the bound on hit.t's error, 0 once it is the binary64 one
    bool found = false, lost = false;
    int sp = 0;
    int ref = 0;
    // while-while traversal (Aila & Laine 2009): descend inner nodes until a leaf is reached,
    // then test leaves until an inner node comes off the stack, so a warp's lanes run the same
    // loop body together instead of alternating node and leaf work per lane (NodeLoop varies it).
    for (;;) {
        while (ref >= 0) {
            const NodeData nd = load_node(sc.nodes + ref);
            if (COUNT) ++vis->nodes;
            bool h0, h1;
            float n0, n1;
            slab_pair(nd.c0, nd.c1, nd.h0, nd.h1, nd.cz, nd.hz, slabs, ANY ? tmax : fminf(tmax, REFINE ? hit.t + err : hit.t), h0, h1, n0,
                      n1);
            // an empty child (~0, only beside a root leaf) reads as a leaf of no triangles
            const int r0 = nd.ref0, r1 = nd.ref1;
            if (h0 && h1) {
                bool swap = n1 < n0;
                stack[sp] = swap ? r0 : r1;
                ++sp;
                ref = swap ? r1 : r0;
            } else if (h0 || h1) {
                ref = h0 ? r0 : r1;
            } else {
                if (sp == 0) goto done;
                ref = stack[--sp];
            }
            if (LOOP == NodeLoop::kFew && __popc(__activemask()) < 8) break;
        }
        if (ref < 0) do {
            uint32_t packed = (uint32_t)(~ref);
            uint32_t first = packed >> 3, count = packed & 7u;
            for (uint32_t k = 0; k < count; ++k) {
                uint32_t i = first + k;
                const float4 *tp = sc.tris + (size_t)i * 3;
                float4 v0 = ldg4(tp);
                if (COUNT) ++vis->tris;
                float t, u, v;
                float terr = 0.0f;
                bool ok = REFINE ? tri_test_refined(sc, v0, ldg4(tp + 1), ldg4(tp + 2), o, d, max, t, u, v, vis, terr)
                                 : tri_test(v0, ldg4(tp + 1), ldg4(tp + 2), o, d, max, t, u, v);
                if (!ok) continue;
                uint32_t occ = __float_as_uint(v0.w);
                if (!ANY && REFINE) {
                    if (!refined_candidate<EACH>(sc, o, d, max, alpha, vis, occ, t, u, v, terr, found, hit, err, lost))
                        continue;
                } else if (alpha && !alpha_blocks(sc, occ, u, v)) {
                    continue;
                }
                if (ANY) return true;
                if (isfinite(t) && (REFINE || t < hit.t || (t == hit.t && occ < hit.occluder))) {
                    found = true;
                    err = terr;
                    hit.t = t;
                    hit.u = u;
                    hit.v = v;
                    hit.occluder = occ;
                }
            }
            if (sp == 0) goto done;
            ref = stack[--sp];
        } while (LOOP != NodeLoop::kOneLeaf && ref < 0);
    }
done:
    if (!ANY && REFINE) {
        // the winner's binary64 distance and barycentrics, the warp's lanes together
        if (found && err > 0.0f) {
            ++vis->retests;
            if (!tri_test_fp64(sc, hit.occluder, o, d, max, hit.t, hit.u, hit.v) || !isfinite(hit.t)) lost = true;
        }
        if (!EACH && lost) return traverse_each<COUNT>(sc, o, dir, max, alpha, stack, hit, vis);
    }
    return found;
}

template <bool COUNT>
__device__ __noinline__ bool traverse_each(const DevScene &sc, f3 o, f3 dir, float max, bool alpha, int *stack,
                                           Hit &hit, Visits *vis) {
    return traverse<false, COUNT, true, true>(sc, o, dir, max, alpha, stack, hit, vis);
}

template <bool COUNT = false, bool REFINE = false, NodeLoop LOOP = NodeLoop::kPlain>
__device__ __forceinline__ bool occluded(const DevScene &sc, f3 o, f3 d, float max, bool alpha, int *stack,
                                         Visits *vis = nullptr) {
    Hit h;
    return traverse<true, COUNT, REFINE, false, LOOP>(sc, o, d, max, alpha, stack, h, vis);
}

}  // namespace dl
