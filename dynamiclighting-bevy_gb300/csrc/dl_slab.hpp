// The occluder BVH's nodes as the traversal reads them, and the slab test of a node's two boxes.
//
// A box is stored as centre and half extent per axis. On one axis the ray meets the slab around
// t_c = (c - o) / d at t_c -+ h / |d|, so near and far come out of two multiply-adds with no
// minimum and maximum of the two planes' distances: a node's test is 9 packed (two at a time)
// multiply-adds, 4 three-input and 4 two-input minima and maxima, where the plane form needs 12 multiply-adds
// and 24 minima and maxima. The traversal is bound by instruction issue and, within that, by the
// integer/comparison pipe, which runs minima and maxima at half the multiply-adds' rate (ncu on the
// quarter-size outdoor case with the plane form: issue slots 83 % busy, that pipe 55 %, the
// multiply-add pipe 31 %; with this one 68 % and 38 %, at 64 registers). On the full outdoor bake
// (546k triangles) the visibility stage went from 131.8 ms to 123.7 ms and the sun gather from
// 94.5 ms to 87.2 ms; the room grid's local gather from 71.7 ms to 67.3 ms.
#pragma once

#include <cstdint>

#include "dl_math.cuh"

namespace dl {

// 64 bytes: x and y of both children side by side (one packed operation each), then z of both.
struct alignas(32) TravNode {
    float cxy[4];    // centres c0x, c0y, c1x, c1y
    float hxy[4];    // half extents h0x, h0y, h1x, h1y
    float z[4];      // c0z, c1z, h0z, h1z
    int32_t ref[2];  // >= 0 an inner node, < 0 a leaf ~(first << 3 | count), ~0 an empty child
    uint32_t zero[2];
};

// Centre and half extent of [lo, hi] such that [c - h, c + h] covers it: the relative growth of h
// (2^-22) is above the rounding of its subtraction. An inverted box (lo > hi, an empty child)
// keeps a negative h, which no ray enters.
DL_HD void trav_box(float lo, float hi, float &c, float &h) {
    c = lo * 0.5f + hi * 0.5f;
    const float up = hi - c, down = c - lo;
    h = up > down ? up : down;
    if (h > 0.0f) h = h * 1.0000002384185791f;
}
// A node from its children's (padded) boxes, given per child as lo xyz and hi xyz.
DL_HD TravNode trav_node(const float lo0[3], const float hi0[3], const float lo1[3], const float hi1[3], int32_t ref0,
                         int32_t ref1) {
    TravNode n;
    trav_box(lo0[0], hi0[0], n.cxy[0], n.hxy[0]);
    trav_box(lo0[1], hi0[1], n.cxy[1], n.hxy[1]);
    trav_box(lo1[0], hi1[0], n.cxy[2], n.hxy[2]);
    trav_box(lo1[1], hi1[1], n.cxy[3], n.hxy[3]);
    trav_box(lo0[2], hi0[2], n.z[0], n.z[2]);
    trav_box(lo1[2], hi1[2], n.z[1], n.z[3]);
    n.ref[0] = ref0;
    n.ref[1] = ref1;
    n.zero[0] = n.zero[1] = 0;
    return n;
}

// Two binary32 values in one 64-bit register and the packed multiply-add on them (each half rounds
// as fmaf does).
#if defined(__CUDA_ARCH__)
typedef unsigned long long Pair;
DL_HD Pair pair_of(float x, float y) {
    Pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
DL_HD void halves(Pair p, float &x, float &y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(p));
}
DL_HD Pair fma2(Pair a, Pair b, Pair c) {
    Pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
DL_HD float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
DL_HD float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
#else
struct Pair {
    float x, y;
};
DL_HD Pair pair_of(float x, float y) { return Pair{x, y}; }
DL_HD void halves(Pair p, float &x, float &y) {
    x = p.x;
    y = p.y;
}
DL_HD Pair fma2(Pair a, Pair b, Pair c) { return Pair{fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)}; }
DL_HD float max3(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }
DL_HD float min3(float a, float b, float c) { return fminf(fminf(a, b), c); }
#endif

// A ray's constants for the slab tests: reciprocal direction i, its magnitude a, -a, and -o * i.
struct RaySlabs {
    Pair ixy, iz, axy, az, nxy, nz, oxy, oz;
};
// The reciprocal of a direction component for the slab tests. A component below 1e-20 counts as
// 1e-20 with its sign: the ray then drifts by 1e-20 of its length, far below the boxes' padding, and
// centre and half extent times the reciprocal stay finite for coordinates up to 1e18.
DL_HD float slab_inverse(float d) {
    if (!(fabsf(d) >= 1.0e-20f)) d = copysignf(1.0e-20f, d);
#if defined(__CUDA_ARCH__)
    return __fdividef(1.0f, d);  // within 2 ulp: it only prunes, and slab_pair's exit slack covers it
#else
    return 1.0f / d;
#endif
}
DL_HD RaySlabs ray_slabs(f3 o, f3 d) {
    const f3 i{slab_inverse(d.x), slab_inverse(d.y), slab_inverse(d.z)};
    RaySlabs r;
    r.ixy = pair_of(i.x, i.y);
    r.iz = pair_of(i.z, i.z);
    r.axy = pair_of(fabsf(i.x), fabsf(i.y));
    r.az = pair_of(fabsf(i.z), fabsf(i.z));
    r.nxy = pair_of(-fabsf(i.x), -fabsf(i.y));
    r.nz = pair_of(-fabsf(i.z), -fabsf(i.z));
    const float oz = -(o.z * i.z);
    r.oxy = pair_of(-(o.x * i.x), -(o.y * i.y));
    r.oz = pair_of(oz, oz);
    return r;
}

// Slab test of both children of a node against the ray's [0, tmax]: whether each may be hit, and
// where the ray enters it. It only prunes, so it may err towards visiting and never the other
// way: boxes are padded by 1e-5 of their coordinates when they are built, each axis' distances
// scale by one factor within 2^-22 of 1 (the reciprocal) and round a few times at 2^-24 of the
// distance from the ray's origin, and the exit distance gets a relative slack of 2e-6 for it.
DL_HD void slab_pair(Pair c0, Pair c1, Pair h0, Pair h1, Pair cz, Pair hz, const RaySlabs &r, float tmax, bool &hit0,
                     bool &hit1, float &near0, float &near1) {
    const Pair t0 = fma2(c0, r.ixy, r.oxy), t1 = fma2(c1, r.ixy, r.oxy), tz = fma2(cz, r.iz, r.oz);
    const Pair n0 = fma2(h0, r.nxy, t0), n1 = fma2(h1, r.nxy, t1), nz = fma2(hz, r.nz, tz);
    const Pair f0 = fma2(h0, r.axy, t0), f1 = fma2(h1, r.axy, t1), fz = fma2(hz, r.az, tz);
    float ax, ay, bx, by, az, bz;
    halves(n0, ax, ay);
    halves(n1, bx, by);
    halves(nz, az, bz);
    const float en0 = fmaxf(max3(ax, ay, az), 0.0f), en1 = fmaxf(max3(bx, by, bz), 0.0f);
    halves(f0, ax, ay);
    halves(f1, bx, by);
    halves(fz, az, bz);
    const float ex0 = fminf(min3(ax, ay, az), tmax), ex1 = fminf(min3(bx, by, bz), tmax);
    const float slack = 1.0f + 2.0e-6f;
    hit0 = en0 <= ex0 * slack;
    hit1 = en1 <= ex1 * slack;
    near0 = en0;
    near1 = en1;
}

}  // namespace dl
