// The bake pipeline on one GPU and the C ABI (include/dynlight.h).
//
// Stages, on one stream (the queue's two kernels on two), each a kernel over the whole scene (every mesh at once):
//   setup      per triangle: face normal, crop rect, light association (mesh_bake.rs:141-173)
//   regions    per (mesh, light): union of crop rects -> one shadow grid (mesh_bake.rs:175-192)
//   texels     per triangle: owned grid, centered + touched texels (texels.rs, mesh_texels.rs)
//   burial     per texel: <= 8 closest-hit rays (mesh_texels.rs:57-88,111-135)
//   visibility per (pair, texel): point/area/sun/sky shadow rays (mesh_bake.rs:203-267)
//              batched: persistent kernels over a device work queue;
//              plain: one launch per mesh, a warp per triangle, lanes over texels
//   optimize   per triangle: drop lights with no lit texel nearby (shadows.rs:54-73)
//   seams      per region: pad unvisited texels (seams.rs:15-39)
//   serialize  per triangle/entry: header words, light data, cropped and dilated shadow words
//              (shadows.rs:87-159, seams.rs:43-71, triangle_words.rs:47-89)
// Sizes that decide later allocations are read back between stages (a handful of 8-byte copies).
#include <cub/cub.cuh>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <tuple>
#include <vector>

#include "dl_bvh.hpp"
#include "dl_bvh_rules.hpp"
#include "dl_kernels.cuh"

namespace dl {

constexpr int kBlock = 128;
constexpr uint32_t kNoRect = 0xFFFFFFFFu;
constexpr uint64_t kBurialStream = 0x627572696564ull;  // mesh_texels.rs:26

struct Counters {
    unsigned long long rays, burial_rays, lights_removed, bounce_rays, photon_rays, cancelled;
    unsigned long long node_visits, tri_tests;  // instrumented visibility kernel only
    unsigned long long retests;                 // refined form: binary64 re-tests
    unsigned long long gather_node_visits, gather_tri_tests;  // instrumented gather kernel only
};

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
    return v;
}
// Adds a whole warp's re-test counts to the counters (every lane calls it).
__device__ __forceinline__ void add_retests(Counters *ctr, unsigned long long n) {
    unsigned long long w = warp_sum(n);
    if (lane_id() == 0 && w) atomicAdd(&ctr->retests, w);
}

// ================================ sample order tables ====================================

// The tables of shifted_sample (DevScene's `order_cells`, `cell_samples`) for n = 16, 32, ..., kMaxOrdered, a
// thread per sample: what sample_cells (dl_host.hpp) finds by sorting. On the host that took 0.7 ms of every
// session, a fifth of the smallest bake.
__global__ void k_sample_tables(uint16_t *cells, uint16_t *samples) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x + 16;
    if (i >= 2 * kMaxOrdered) return;
    const uint32_t m = 31 - __clz(i), n = 1u << m, j = i - n, base = n - 16;
    const NetCell c = net_cell(j, m);
    cells[base + c.rank] = (uint16_t)(c.x | c.y << 8);
    samples[base + (c.y << ((m + 1) / 2) | c.x)] = (uint16_t)j;
}

// ================================ setup and association ==================================

__global__ void k_setup(DevScene sc, float4 *tri_face, uint4 *tri_crop, uint32_t *tri_count) {
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= sc.triangles) return;
    TriData d;
    load_tri(sc, t, d);
    f3 face = normalize_or_zero(cross(sub(d.v[1], d.v[0]), sub(d.v[2], d.v[0])));
    uint32_t count = 0;
    associate(sc, d, face, [&](uint32_t) { ++count; });
    Rect c = crop_rect(d.uv, d.res);
    tri_face[t] = make_float4(face.x, face.y, face.z, is_zero(face) ? 0.0f : 1.0f);
    tri_crop[t] = make_uint4(c.min_x, c.min_y, c.max_x, c.max_y);
    tri_count[t] = count;
}

__global__ void k_assoc_fill(DevScene sc, const float4 *tri_face, const uint4 *tri_crop, const uint32_t *tri_off,
                             uint32_t *pair_light, uint32_t *pair_tri, uint32_t *region_rect) {
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= sc.triangles) return;
    TriData d;
    load_tri(sc, t, d);
    float4 f = tri_face[t];
    uint4 c = tri_crop[t];
    uint32_t p = tri_off[t];
    associate(sc, d, f3{f.x, f.y, f.z}, [&](uint32_t s) {
        pair_light[p] = s;
        pair_tri[p] = t;
        ++p;
        uint32_t *r = region_rect + ((size_t)d.mesh * sc.light_count + s) * 4;
        atomicMin(r, c.x);
        atomicMin(r + 1, c.y);
        atomicMax(r + 2, c.z);
        atomicMax(r + 3, c.w);
    });
}

__global__ void k_fill_u32(uint32_t *p, size_t n, uint32_t a, uint32_t b) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = (i & 2) ? b : a;  // 4-word records (a, a, b, b)
}

// Words of each (mesh, light) region grid: bits for 1-bit lights, one byte per texel else.
__global__ void k_region_words(const uint32_t *region_rect, const DevLight *lights, uint32_t entries, uint32_t L,
                               uint32_t *words) {
    uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e > entries) return;
    if (e == entries) {
        words[e] = 0;
        return;
    }
    const uint32_t *r = region_rect + (size_t)e * 4;
    if (r[0] == kNoRect) {
        words[e] = 0;
        return;
    }
    uint64_t n = (uint64_t)(r[2] - r[0] + 1) * (r[3] - r[1] + 1);
    words[e] = lights[e % L].shadow_bits == 1 ? (uint32_t)((n + 31) / 32) : (uint32_t)((n + 3) / 4);
}

// Index i of a row-major grid of width w as column and row; grids beyond 2^32 texels are rare, so
// the division is a 32-bit one where it can be (the 64-bit one takes several times the instructions).
__device__ __forceinline__ void grid_xy(uint64_t i, uint32_t w, uint32_t &x, uint32_t &y) {
    if (i <= 0xFFFFFFFFull) {
        y = (uint32_t)i / w;
        x = (uint32_t)i - y * w;
    } else {
        y = (uint32_t)(i / w);
        x = (uint32_t)(i % w);
    }
}

// The kernels below take a warp (or a block) per triangle, pair, entry or region. With few of them
// (a room of large walls) most of the chip would wait for a few warps that walk thousands of texels
// each, so the launch adds a second grid dimension: part y of gridDim.y takes every gridDim.y-th
// run of the job's texels (grid_parts). On the small room (72 triangles, 8 texels/m) k_crop took 367 us
// with one part and 19 us so, k_pad_seams 152 us and 8 us, the three k_texels passes 208 us and 26 us,
// the two k_unburied passes 80 us and 9 us (also from 32-bit index divisions).

// ================================ texels ===============================================

// Slots for a warp's `n` texels of triangle t: parts of a triangle share a cursor. The order of a
// triangle's texels does not matter to any result (a texel's streams are keyed by its coordinates).
__device__ __forceinline__ uint32_t take_slots(uint32_t *cursor, uint32_t t, uint32_t n, uint32_t &local) {
    if (gridDim.y == 1) {
        const uint32_t at = local;
        local += n;
        return at;
    }
    uint32_t at = 0;
    if (lane_id() == 0 && n) at = atomicAdd(cursor + t, n);
    return __shfl_sync(0xFFFFFFFFu, at, 0);
}

// MODE 0: count centered texels and set the owned grid; MODE 1: count touched texels;
// MODE 2: write centered and touched texels from tex_off[t]. A warp per triangle and part; counts are
// added to `count`, which starts at 0, as do the cursors.
template <int MODE>
__global__ void k_texels(DevScene sc, const float4 *tri_face, uint32_t *owned, const uint64_t *grid_off,
                         uint32_t *count, uint32_t *cursor, const uint32_t *tex_off, uint32_t *tex_xy, float4 *tex_pos,
                         float4 *tex_nrm, uint32_t *tex_tri) {
    uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    unsigned lane = lane_id();
    if (t >= sc.triangles) return;
    float4 f = tri_face[t];
    if (f.w == 0.0f) return;
    f3 face{f.x, f.y, f.z};
    TriData d;
    load_tri(sc, t, d);
    uint32_t res = d.res;
    uint32_t *own = owned + grid_off[d.mesh];
    const uint64_t first = (uint64_t)blockIdx.y * 32, stride = (uint64_t)gridDim.y * 32;
    uint32_t counted = 0, local = 0;
    const uint32_t out = MODE == 2 ? tex_off[t] : 0;
    auto write = [&](bool take, unsigned ballot, uint32_t x, uint32_t y, f3 wts) {
        const uint32_t at = take_slots(cursor, t, __popc(ballot), local);
        if (!take) return;
        const uint32_t o = out + at + __popc(ballot & ((1u << lane) - 1u));
        f3 pos, nrm;
        surface_at(d, face, wts, pos, nrm);
        tex_xy[o] = x | (y << 16);
        tex_pos[o] = make_float4(pos.x, pos.y, pos.z, 0.0f);
        tex_nrm[o] = make_float4(nrm.x, nrm.y, nrm.z, 0.0f);
        tex_tri[o] = t;
    };
    if (MODE == 0 || MODE == 2) {
        Rect r = center_rect(d.uv, res, 0.0f);
        uint32_t w = r.max_x - r.min_x + 1;
        uint64_t n = (uint64_t)w * (r.max_y - r.min_y + 1);
        for (uint64_t base = first; base < n; base += stride) {
            uint64_t i = base + lane;
            bool inside = false;
            uint32_t x = 0, y = 0;
            f3 wts;
            if (i < n) {
                grid_xy(i, w, x, y);
                x += r.min_x;
                y += r.min_y;
                inside = uv_barycentrics(d.uv, texel_center(x, y, res), wts);
            }
            unsigned ballot = __ballot_sync(0xFFFFFFFFu, inside);
            if (MODE == 0) {
                if (inside) {
                    uint64_t bit = (uint64_t)x + (uint64_t)y * res;
                    atomicOr(own + bit / 32, 1u << (bit % 32));
                }
                counted += __popc(ballot);
            } else {
                write(inside, ballot, x, y, wts);
            }
        }
    }
    // touched texels (texels.rs:78-121)
    if (MODE != 0) {
        float s = (float)res;
        f2 mn, mx;
        uv_bounds(d.uv, mn, mx);
        uint32_t x0 = f2u(fmaxf(floorf(mn.x * s), 0.0f)), y0 = f2u(fmaxf(floorf(mn.y * s), 0.0f));
        uint32_t x1 = f2u(fminf(floorf(mx.x * s), s - 1.0f)), y1 = f2u(fminf(floorf(mx.y * s), s - 1.0f));
        float half = 0.5f / s;
        if (x1 >= x0 && y1 >= y0) {
            uint32_t w = x1 - x0 + 1;
            uint64_t n = (uint64_t)w * (y1 - y0 + 1);
            for (uint64_t base = first; base < n; base += stride) {
                uint64_t i = base + lane;
                bool take = false;
                uint32_t x = 0, y = 0;
                f3 wts;
                if (i < n) {
                    grid_xy(i, w, x, y);
                    x += x0;
                    y += y0;
                    uint64_t bit = (uint64_t)x + (uint64_t)y * res;
                    bool is_owned = (own[bit / 32] >> (bit % 32)) & 1u;
                    if (!is_owned) {
                        f2 center = texel_center(x, y, res);
                        if (nearest_weights(d.uv, center, wts)) {
                            float nx = d.uv[0].x * wts.x + d.uv[1].x * wts.y + d.uv[2].x * wts.z;
                            float ny = d.uv[0].y * wts.x + d.uv[1].y * wts.y + d.uv[2].y * wts.z;
                            take = fmaxf(fabsf(nx - center.x), fabsf(ny - center.y)) <= half;
                        }
                    }
                }
                unsigned ballot = __ballot_sync(0xFFFFFFFFu, take);
                if (MODE == 1) counted += __popc(ballot);
                else write(take, ballot, x, y, wts);
            }
        }
    }
    if (MODE != 2 && lane == 0 && counted) atomicAdd(count + t, counted);
}

// Burial test per texel (mesh_texels.rs:57-88). Buried texels are dropped from tracing.
template <bool REFINE>
__global__ void __launch_bounds__(kBlock) k_burial(DevScene sc, uint32_t texels, const uint32_t *tex_xy,
                                                   const float4 *tex_pos, const uint32_t *tex_tri,
                                                   const float4 *tri_face, uint8_t *buried, Counters *ctr) {
    int stack[kStack];
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t rays = 0;
    Visits vis{0, 0, 0};
    if (i < texels) {
        uint32_t t = tex_tri[i];
        uint32_t m = sc.tri_mesh[t];
        float4 f = tri_face[t], p = tex_pos[i];
        f3 normal{f.x, f.y, f.z};
        uint32_t xy = tex_xy[i];
        f3 origin = add(f3{p.x, p.y, p.z}, scale(normal, kRayOffset));
        Pcg rng = stream6(sc.seed, sc.mesh_id[m], kBurialStream, t - sc.mesh_tri_base[m], xy & 0xFFFFu, xy >> 16);
        float turn = rng.next_f32();
        buried[i] = is_buried<REFINE>(sc, normal, origin, turn, stack, rays, &vis) ? 1 : 0;
    }
    unsigned r = __reduce_add_sync(0xFFFFFFFFu, rays);
    if (lane_id() == 0 && r) atomicAdd(&ctr->burial_rays, (unsigned long long)r);
    if (REFINE) add_retests(ctr, vis.retests);
}

// Per triangle: how many of its texels are not buried, then those texels (a warp per triangle and part).
template <bool WRITE>
__global__ void k_unburied(uint32_t triangles, const uint32_t *tex_off, const uint8_t *buried, uint32_t *count,
                           uint32_t *cursor, const uint32_t *ctex_off, const uint32_t *tex_xy, const float4 *tex_pos,
                           const float4 *tex_nrm, uint32_t *c_xy, float4 *c_pos, float4 *c_nrm) {
    uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    unsigned lane = lane_id();
    if (t >= triangles) return;
    uint32_t b = tex_off[t], e = tex_off[t + 1];
    uint32_t kept = 0, local = 0;
    uint32_t out = WRITE ? ctex_off[t] : 0;
    for (uint64_t base = b + (uint64_t)blockIdx.y * 32; base < e; base += (uint64_t)gridDim.y * 32) {
        const uint64_t i = base + lane;
        bool keep = i < e && !buried[i];
        unsigned ballot = __ballot_sync(0xFFFFFFFFu, keep);
        if (WRITE) {
            const uint32_t at = take_slots(cursor, t, __popc(ballot), local);
            if (keep) {
                uint32_t o = out + at + __popc(ballot & ((1u << lane) - 1u));
                c_xy[o] = tex_xy[i];
                c_pos[o] = tex_pos[i];
                c_nrm[o] = tex_nrm[i];
            }
        }
        kept += __popc(ballot);
    }
    if (!WRITE && lane == 0 && kept) atomicAdd(count + t, kept);
}

// ================================ visibility ===========================================

struct TraceArgs {
    const uint32_t *pair_tri, *pair_light;
    const uint32_t *ctex_off, *ctex_xy;
    const float4 *ctex_pos, *ctex_nrm, *tri_face;
    const uint64_t *grid_off;  // visited grid word offset per mesh
    uint32_t *visited;
    const uint32_t *region_rect, *region_off;
    uint32_t *region_pool;
    Counters *ctr;
    // batched queue: items of sky pairs first, then soft, then hard
    const uint32_t *order, *item_off;
    uint32_t pairs;
    unsigned long long items;
    unsigned long long *head;      // chunks claimed in the per-lane phase
    unsigned long long *head_sky;  // chunks claimed in the grouped sky phase
    const volatile uint32_t *cancel;
    uint32_t grab;         // warp-steps per claimed chunk
    uint32_t sky_items;    // items of the sky pairs at the front of the queue
    uint32_t sky_lanes;    // lanes sharing one sky texel's samples (1: no grouped phase)
    uint32_t sample_every; // tuning trials: claim one chunk in `sample_every` (1: all)
};

// The visibility result of (pair p, texel x, y of mesh m) into the visited grid and the light's
// region grid (mesh_bake.rs:231-248): a bit for 1-bit lights, an atomic max of the level otherwise.
__device__ __forceinline__ void store_texel(const DevScene &sc, const TraceArgs &a, uint32_t m, uint32_t s,
                                            uint32_t x, uint32_t y, uint32_t level, uint32_t bits) {
    uint32_t res = sc.mesh_res[m];
    uint64_t bit = (uint64_t)x + (uint64_t)y * res;
    atomicOr(a.visited + a.grid_off[m] + bit / 32, 1u << (bit % 32));
    size_t e = (size_t)m * sc.light_count + s;
    const uint32_t *r = a.region_rect + e * 4;
    uint32_t w = r[2] - r[0] + 1;
    uint64_t idx = (uint64_t)(x - r[0]) + (uint64_t)(y - r[1]) * w;
    uint32_t *g = a.region_pool + a.region_off[e];
    if (bits == 1) {
        if (level) atomicOr(g + idx / 32, 1u << (idx % 32));
    } else if (level) {
        uint32_t *word = g + idx / 4;
        uint32_t shift = (uint32_t)(idx % 4) * 8;
        uint32_t cur = *word;
        for (;;) {
            if (((cur >> shift) & 0xFFu) >= level) break;
            uint32_t want = (cur & ~(0xFFu << shift)) | (level << shift);
            uint32_t prev = atomicCAS(word, cur, want);
            if (prev == cur) break;
            cur = prev;
        }
    }
}

// One (pair, texel) of the visibility loop (mesh_bake.rs:231-248); returns the rays traced.
template <bool COUNT = false, bool REFINE = false, bool QUEUED = false>
__device__ __forceinline__ uint32_t trace_texel(const DevScene &sc, const TraceArgs &a, uint32_t p, uint32_t k,
                                                int *stack, Visits *vis = nullptr) {
    uint32_t t = a.pair_tri[p], s = a.pair_light[p];
    uint32_t m = sc.tri_mesh[t];
    uint32_t ci = a.ctex_off[t] + k;
    uint32_t xy = a.ctex_xy[ci];
    uint32_t x = xy & 0xFFFFu, y = xy >> 16;
    float4 pp = a.ctex_pos[ci], nn = a.ctex_nrm[ci], f = a.tri_face[t];
    f3 pos{pp.x, pp.y, pp.z}, nrm{nn.x, nn.y, nn.z};
    f3 origin = add(pos, scale(f3{f.x, f.y, f.z}, kRayOffset));
    const DevLight &l = sc.lights[s];
    Tracer<COUNT, REFINE, QUEUED> tr{sc, origin, (l.flags & kLightAlpha) != 0, stack, vis};
    Vis v = texel_shadow(sc, s, sc.mesh_id[m], x, y, pos, nrm, tr);
    if (!v.some) return 0;
    store_texel(sc, a, m, s, x, y, v.level, l.shadow_bits);
    return v.rays;
}

// The pair holding queue item `item`: item_off[lo] <= item < item_off[lo + 1].
__device__ __forceinline__ uint32_t pair_of(const TraceArgs &a, unsigned long long item) {
    uint32_t lo = 0, hi = a.pairs;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if ((unsigned long long)a.item_off[mid] <= item) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Whether a warp's lane 0 should stop claiming work: the cancel flag is read every 16th claim;
// once it is seen, the warp counts itself in `ctr->cancelled` and every later claim stops too.
constexpr uint32_t kStopped = 0x80000000u;
__device__ __forceinline__ bool cancel_seen(const volatile uint32_t *cancel, Counters *ctr, uint32_t &grabs) {
    if (grabs & kStopped) return true;
    if ((++grabs & 15u) == 0 && *cancel) {
        grabs |= kStopped;
        atomicAdd(&ctr->cancelled, 1ull);
        return true;
    }
    return false;
}

// Claims the next chunk of a queue phase for the warp: the first item of chunk c is
// first + c * size * sample_every. Returns `end` when the phase is drained or cancelled.
__device__ __forceinline__ unsigned long long claim(const TraceArgs &a, unsigned long long *head,
                                                    unsigned long long first, unsigned long long size,
                                                    unsigned long long end, uint32_t &grabs) {
    unsigned long long base = 0;
    if (lane_id() == 0) {
        if (cancel_seen(a.cancel, a.ctr, grabs)) {
            base = end;
        } else {
            unsigned long long c = atomicAdd(head, 1ull);
            base = first + c * size * a.sample_every;
            if (base > end) base = end;
        }
    }
    return __shfl_sync(0xFFFFFFFFu, base, 0);
}

// Batched form: persistent warps pull chunks of (pair, texel) items from one queue. Items are
// ordered sky pairs first, then soft, then hard, so the longest work starts first. The sky items are
// a kernel's of their own: W = sky_lanes lanes share one texel, each tracing every W-th rank
// of its samples in the shift-aligned coherent order, and the open counts are summed across the
// group (an integer sum, so the level is the same as one lane tracing them all in index order).
// MINB is the launch bound's blocks per SM (the register budget). Apart from the other lights' code the sky's
// loop needs 40 registers at 12 blocks with a quarter of the spills (a 77 k triangle terrain's visibility 23.5 ms in one
// kernel at 10, 23.1 ms in two).
template <bool COUNT, bool REFINE, int MINB>
__global__ void __launch_bounds__(kBlock, MINB) k_trace_sky(DevScene sc, TraceArgs a) {
    int stack[kStack];
    unsigned lane = lane_id();
    unsigned long long rays = 0;
    Visits vis{0, 0, 0};
    uint32_t grabs = 0;
    const uint32_t W = a.sky_lanes;
    const uint32_t per_step = 32 / W, sub = lane % W;
    const unsigned long long end = a.sky_items;
    for (;;) {
        unsigned long long base = claim(a, a.head_sky, 0, (unsigned long long)per_step * a.grab, end, grabs);
        if (base >= end) break;
        uint32_t cur = pair_of(a, base);
        for (uint32_t g = 0; g < a.grab; ++g) {
            unsigned long long item = base + (unsigned long long)g * per_step + lane / W;
            bool valid = item < end;
            uint32_t open = 0, t = 0, s = 0, m = 0, x = 0, y = 0;
            if (valid) {
                while ((unsigned long long)a.item_off[cur + 1] <= item) ++cur;
                uint32_t p = a.order[cur];
                t = a.pair_tri[p];
                s = a.pair_light[p];
                m = sc.tri_mesh[t];
                uint32_t ci = a.ctex_off[t] + (uint32_t)(item - a.item_off[cur]);
                uint32_t xy = a.ctex_xy[ci];
                x = xy & 0xFFFFu;
                y = xy >> 16;
                float4 pp = a.ctex_pos[ci], nn = a.ctex_nrm[ci], f = a.tri_face[t];
                f3 nrm{nn.x, nn.y, nn.z};
                f3 origin = add(f3{pp.x, pp.y, pp.z}, scale(f3{f.x, f.y, f.z}, kRayOffset));
                const DevLight &l = sc.lights[s];
                Tracer<COUNT, REFINE> tr{sc, origin, (l.flags & kLightAlpha) != 0, stack, &vis};
                // sky_visibility (sky.rs:30-44), samples sub, sub + W, ...
                Pcg rng = stream5(sc.seed, sc.mesh_id[m], l.id, x, y);
                f2 off;
                off.x = rng.next_f32();
                off.y = rng.next_f32();
                f3 side, across;
                ortho_pair(nrm, side, across);
                // in the shift-aligned coherent order when the sample count allows it: the
                // warp's texels (neighbours) then trace their rank-k rays in about one direction
                // (terrain with 200 samples in the net of 256: 22.7 ms, in index order 27.8 ms)
                const uint32_t n = sc.sky_samples, net = ordered_net(n, 16, kMaxOrdered);
                const uint32_t shift = net ? net_shift(net, off) : 0u, ranks = net ? net : n;
                for (uint32_t k = sub; k < ranks; k += W) {
                    const uint32_t j = net ? shifted_sample(sc, net, shift, k) : sc.sky_order ? sc.sky_order[k] : k;
                    if (j < n && !tr(cosine_direction_basis(nrm, side, across, spread(j, off, true)), INFINITY))
                        ++open;
                }
            }
            for (uint32_t o = 1; o < W; o <<= 1) open += __shfl_xor_sync(0xFFFFFFFFu, open, o);
            if (valid && sub == 0) {
                uint32_t samples = sc.sky_samples;
                float fraction = (float)open / (float)(samples > 1 ? samples : 1);
                const DevLight &l = sc.lights[s];
                store_texel(sc, a, m, s, x, y, level_of(fraction, l.shadow_bits), l.shadow_bits);
                rays += samples;
            }
        }
    }
    unsigned long long r = warp_sum(rays);
    if (lane == 0 && r) atomicAdd(&a.ctr->rays, r);
    if (COUNT) {
        unsigned long long n = warp_sum(vis.nodes), t = warp_sum(vis.tris);
        if (lane == 0) {
            atomicAdd(&a.ctr->node_visits, n);
            atomicAdd(&a.ctr->tri_tests, t);
        }
    }
    if (REFINE) add_retests(a.ctr, vis.retests);
}

// The items behind the sky's, one lane an item. Rays towards local lights leave the leaf loop after each leaf
// (rooms under panels and tubes 6.2 -> 5.5 ms).
template <bool COUNT, bool REFINE, int MINB>
__global__ void __launch_bounds__(kBlock, MINB) k_trace_batched(DevScene sc, TraceArgs a) {
    int stack[kStack];
    unsigned lane = lane_id();
    unsigned long long rays = 0;
    Visits vis{0, 0, 0};
    uint32_t grabs = 0;
    for (;;) {
        unsigned long long base = claim(a, a.head, a.sky_items, 32ull * a.grab, a.items, grabs);
        if (base >= a.items) break;
        uint32_t cur = pair_of(a, base);  // per lane, advances monotonically over the chunk
        for (uint32_t g = 0; g < a.grab; ++g) {
            unsigned long long item = base + (unsigned long long)g * 32 + lane;
            if (item < a.items) {
                while ((unsigned long long)a.item_off[cur + 1] <= item) ++cur;
                rays += trace_texel<COUNT, REFINE, true>(
                    sc, a, a.order[cur], (uint32_t)(item - a.item_off[cur]), stack, &vis);
            }
        }
    }
    unsigned long long r = warp_sum(rays);
    if (lane == 0 && r) atomicAdd(&a.ctr->rays, r);
    if (COUNT) {
        unsigned long long n = warp_sum(vis.nodes), t = warp_sum(vis.tris);
        if (lane == 0) {
            atomicAdd(&a.ctr->node_visits, n);
            atomicAdd(&a.ctr->tri_tests, t);
        }
    }
    if (REFINE) add_retests(a.ctr, vis.retests);
}

// Plain form: one launch per mesh; a warp per triangle, its lights in order, lanes over texels.
__global__ void __launch_bounds__(kBlock) k_trace_plain(DevScene sc, TraceArgs a, uint32_t first_tri,
                                                         uint32_t tri_count, const uint32_t *tri_pair_off) {
    int stack[kStack];
    unsigned lane = lane_id();
    unsigned long long rays = 0;
    uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < tri_count; w += warps) {
        uint32_t t = first_tri + w;
        uint32_t n = a.ctex_off[t + 1] - a.ctex_off[t];
        for (uint32_t p = tri_pair_off[t]; p < tri_pair_off[t + 1]; ++p)
            for (uint32_t k = lane; k < n; k += 32) rays += trace_texel(sc, a, p, k, stack);
    }
    unsigned long long r = warp_sum(rays);
    if (lane == 0 && r) atomicAdd(&a.ctr->rays, r);
}

// Queue construction: pairs in class order (sky, soft, hard) and their item prefix sums. One scan of
// packed counts (sky pairs in the low word, soft ones in the high word) places all three classes.
__global__ void k_pair_class(DevScene sc, const uint32_t *pair_light, uint32_t pairs, unsigned long long *flag) {
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > pairs) return;
    unsigned long long f = 0;
    if (p < pairs) {
        const DevLight &l = sc.lights[pair_light[p]];
        f = l.shape == DL_SHAPE_SKY ? 1ull : l.shadow_bits > 1 ? 1ull << 32 : 0ull;
    }
    flag[p] = f;
}
__global__ void k_pair_scatter(const unsigned long long *flag, const unsigned long long *pos, uint32_t pairs,
                               uint32_t *order, uint32_t *sky_pairs) {
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned long long total = pos[pairs];
    const uint32_t skies = (uint32_t)total, softs = (uint32_t)(total >> 32);
    if (p == 0) *sky_pairs = skies;
    if (p >= pairs) return;
    const unsigned long long f = flag[p], at = pos[p];
    const uint32_t sky = (uint32_t)at, soft = (uint32_t)(at >> 32);
    order[f == 1 ? sky : f ? skies + soft : skies + softs + (p - sky - soft)] = p;
}
// The queue's items and, of them, the sky's (sizes[2], sizes[3]) from the sky pairs' count in sizes[0].
__global__ void k_queue_sizes(const uint32_t *item_off, uint32_t pairs, uint32_t *sizes) {
    const uint32_t items = item_off[pairs], sky_items = item_off[sizes[0]];
    sizes[2] = items;
    sizes[3] = sky_items;
}
__global__ void k_item_counts(const uint32_t *order, const uint32_t *pair_tri, const uint32_t *ctex_off,
                              uint32_t pairs, uint32_t *cnt) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > pairs) return;
    if (i == pairs) {
        cnt[i] = 0;
        return;
    }
    uint32_t t = pair_tri[order[i]];
    cnt[i] = ctex_off[t + 1] - ctex_off[t];
}


// ================================ one bounce ===========================================

// PhotonCube::build (bounce.rs:48-70): every cube texel of every local bounce light.
template <bool REFINE>
__global__ void __launch_bounds__(kBlock) k_photons(DevScene sc, const uint32_t *cube_lights, uint32_t cubes,
                                                    uint32_t res, Photon *photons, Counters *ctr) {
    int stack[kStack];
    uint64_t per = 6ull * res * res;
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    Visits vis{0, 0, 0};
    if (i < per * cubes) {
        uint32_t cube = (uint32_t)(i / per);
        uint32_t rem = (uint32_t)(i % per);
        uint32_t face = rem / (res * res), y = (rem % (res * res)) / res, x = rem % res;
        const DevLight &l = sc.lights[cube_lights[cube]];
        photons[i] = make_photon<REFINE>(sc, l, cube_texel_direction(face, x, y, res), stack,
                                         &vis);
    }
    if (REFINE) add_retests(ctr, vis.retests);
}

// Pairs whose light bakes bounce, in pair order.
__global__ void k_pair_compact(const uint32_t *flag, const uint32_t *pos, uint32_t pairs, uint32_t *out) {
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < pairs && flag[p]) out[pos[p]] = p;
}
__global__ void k_bounce_flag(DevScene sc, const uint32_t *pair_light, uint32_t pairs, uint32_t *flag) {
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > pairs) return;
    flag[p] = p < pairs && (sc.lights[pair_light[p]].flags & kLightBounce) ? 1u : 0u;
}

struct BounceArgs {
    const uint32_t *pair_tri, *pair_light;
    const uint32_t *ctex_off, *ctex_xy;
    const float4 *ctex_pos, *tri_face;
    const uint32_t *bpairs, *bitem_off;
    uint32_t bpair_count;
    unsigned long long items;
    const Photon *photons;
    uint32_t res;
    float4 *value;  // xyz: gathered value, w: 1 when gathered
    Counters *ctr;
    uint32_t lanes;         // lanes sharing one texel's samples (1, 2, 4, 8, 16 or 32)
    uint32_t sample_every;  // tuning trials: one claimed step in `sample_every` (1: all)
    uint32_t buffered;      // sun samples a lane group can hold for the aligned order (0: none)
    float4 *scratch;        // per lane group (blockIdx * groups + group): 2 * buffered float4
    unsigned long long *head;  // steps claimed so far (32 / lanes items per step)
    const volatile uint32_t *cancel;  // the bake's cancel flag, read every 16th claim
};

// gather_triangle / gather_sun (bounce.rs:235-292, sun_bounce.rs:24-80): a group of `lanes`
// lanes per (bounce pair, texel) item. Each round, lane k of a group evaluates sample
// round * lanes + k; the group leader then adds the round's contributions in sample order, so
// the sum is the reference's sequential one for any group size.
// Sun gathers with a sample count that fills a net up to `buffered` (ordered_net) take their samples in
// the shift-aligned coherent order instead (shifted_sample): round r of every group in the warp
// traces ranks r * lanes + k, so the warp's texels (neighbours along a triangle) send their rays
// in about the same directions. A sample whose closest hit faces the sun and is lit by it
// stores its value, its index and its shadow ray's origin in the next free slot of the group's
// scratch (global memory; slots are taken in arrival order, so a group touches only as many as
// it holds, a few lines that stay in L2) and sets its bit in the group's mask (shared memory).
// After the closest-hit rounds the group traces the held shadow rays together, W at a time
// (parallel rays towards the sun), marking blocked ones in a second mask; each open sample's
// value then moves to its rank among the open samples (popcounts of the masks), and the group
// loads those values W at a time while the leader adds them, in sample order, as the reference
// does (sun_bounce.rs:70). Dynamic shared memory holds only the groups' masks
// (the per-round contributions go to the leader by shuffles), so that the rest of each SM's
// unified L1/shared memory stays L1 cache for the BVH. MINB is the launch bound's blocks per SM
// (the register budget: 6, 8, 9 and 10 give 80, 64, 56 and 48 registers a thread). Without SUNS the sun's half is
// left out (no sun in the scene gathers): 136 bytes of spill stores at 9 blocks instead of 296, nine rooms' gather
// 22.0 -> 21.5 ms (with an earlier traversal loop; 12.5 ms now). A form without the local half measured the same as this one.
template <bool COUNT, bool REFINE, int MINB, bool SUNS = true>
__global__ void __launch_bounds__(kBlock, MINB) k_gather(DevScene sc, BounceArgs a) {
    extern __shared__ uint32_t masks[];
    int stack[kStack];
    const uint32_t lane = lane_id(), W = a.lanes, sub = lane % W, per_step = 32 / W;
    // this lane group's masks (shared memory: samples whose hit is lit, then those whose shadow
    // ray is blocked) and scratch (global memory) for aligned sun gathers
    const uint32_t group = (threadIdx.x >> 5) * per_step + lane / W, words = a.buffered / 32;
    const unsigned group_lanes = W == 32 ? 0xFFFFFFFFu : ((1u << W) - 1u) << (lane / W * W);
    uint32_t *lit = masks + (size_t)group * 2 * words;
    uint32_t *blocked = lit + words;
    float4 *scratch = a.scratch + ((size_t)blockIdx.x * (kBlock / W) + group) * 2 * a.buffered;
    for (uint32_t w = sub; w < 2 * words; w += W) lit[w] = 0u;
    __syncwarp();
    unsigned long long rays = 0;
    Visits vis{0, 0, 0};
    uint32_t grabs = 0;
    for (;;) {
        unsigned long long step = ~0ull;
        if (lane == 0 && !cancel_seen(a.cancel, a.ctr, grabs)) step = atomicAdd(a.head, 1ull);
        step = __shfl_sync(0xFFFFFFFFu, step, 0);
        if (step == ~0ull) break;  // cancelled (uniform across the warp)
        unsigned long long base = step * per_step * a.sample_every;
        if (base >= a.items) break;  // uniform across the warp
        unsigned long long item = base + lane / W;
        bool valid = item < a.items, active = false, sun = false;
        uint32_t samples = 0, s = 0;
        f3 pos{0, 0, 0}, normal{0, 0, 0}, origin{0, 0, 0};
        LocalGather lg;
        SunGather sg;
        if (valid) {
            uint32_t lo = 0, hi = a.bpair_count;
            while (hi - lo > 1) {
                uint32_t mid = (lo + hi) >> 1;
                if ((unsigned long long)a.bitem_off[mid] <= item) lo = mid;
                else hi = mid;
            }
            uint32_t p = a.bpairs[lo];
            uint32_t t = a.pair_tri[p];
            s = a.pair_light[p];
            uint32_t m = sc.tri_mesh[t];
            uint32_t ci = a.ctex_off[t] + (uint32_t)(item - a.bitem_off[lo]);
            uint32_t xy = a.ctex_xy[ci];
            float4 pp = a.ctex_pos[ci], f = a.tri_face[t];
            pos = f3{pp.x, pp.y, pp.z};
            normal = f3{f.x, f.y, f.z};
            origin = add(pos, scale(normal, kRayOffset));
            const DevLight &l = sc.lights[s];
            samples = l.bounce_samples;
            sun = SUNS && l.shape == DL_SHAPE_SUN;
            if (sun) {
                sun_setup(sc, l, sc.mesh_id[m], xy & 0xFFFFu, xy >> 16, normal, sg);
                active = true;
            } else {
                active = local_setup(sc, l, sc.mesh_id[m], xy & 0xFFFFu, xy >> 16, pos, sub, lg);
            }
        }
        if (!active) samples = 0;
        const uint32_t net = sun && active && a.buffered ? ordered_net(samples, 32, a.buffered) : 0u;
        const bool aligned = SUNS && net != 0;
        const uint32_t shift = aligned ? net_shift(net, sg.off) : 0u, ranks = aligned ? net : samples;
        FSum3<REFINE> sum;
        uint32_t filled = 0;  // aligned sun gathers: scratch slots filled so far (the same in the group)
        const uint32_t rounds = __reduce_max_sync(0xFFFFFFFFu, (ranks + W - 1) / W);
        for (uint32_t r = 0; r < rounds; ++r) {
            const uint32_t k = r * W + sub;
            if (aligned) {
                SunHit h{f3{0.0f, 0.0f, 0.0f}, f3{0.0f, 0.0f, 0.0f}, false};
                uint32_t i = samples;
                if (k < net) i = shifted_sample(sc, net, shift, k);
                if (i < samples) {
                    h = sun_hit<COUNT, REFINE>(sc, sc.lights[s], origin, normal, sg, i, stack,  &vis);
                    rays += h.pending ? 2 : 1;
                }
                // the group's pending samples of this round take the next slots, in lane order
                const unsigned mine = __ballot_sync(group_lanes, h.pending);
                if (h.pending) {
                    const uint32_t slot = filled + __popc(mine & ((1u << lane) - 1u));
                    scratch[2 * slot] = make_float4(h.value.x, h.value.y, h.value.z, __uint_as_float(i));
                    scratch[2 * slot + 1] = make_float4(h.point.x, h.point.y, h.point.z, 0.0f);
                    atomicOr(&lit[i >> 5], 1u << (i & 31u));
                }
                filled += __popc(mine);
                continue;  // no per-round sum: the phases below add the values in sample order
            }
            Contribution c{f3{0.0f, 0.0f, 0.0f}, false, 0};
            if (k < samples) {
                const DevLight &l = sc.lights[s];
                if (SUNS && sun) {
                    c = sun_sample<COUNT, REFINE>(sc, l, origin, normal, sg, k, stack,  &vis);
                } else {
                    Tracer<COUNT, REFINE> tr{sc, origin, (l.flags & kLightAlpha) != 0, stack, &vis};
                    c = local_sample(sc, l, a.photons + (size_t)l.cube * 6 * a.res * a.res, a.res, normal, lg, k, tr);
                    lg.rng.advance(2ull * (W - 1));  // to the lane's next sample, k + W
                }
                rays += c.rays;
            }
            // the leader adds the round's contributions in sample order, from the group's lanes
            const uint32_t lane0 = lane - sub, n = samples > r * W ? min(W, samples - r * W) : 0u;
            for (uint32_t j = 0; j < n; ++j) {
                const float x = __shfl_sync(group_lanes, c.value.x, lane0 + j);
                const float y = __shfl_sync(group_lanes, c.value.y, lane0 + j);
                const float z = __shfl_sync(group_lanes, c.value.z, lane0 + j);
                const int add = __shfl_sync(group_lanes, (int)c.add, lane0 + j);
                if (sub == 0 && add) sum.add(f3{x, y, z});
            }
        }
        __syncwarp();
        if (aligned) {
            // the shadow rays of the held samples, slot by slot across the group's lanes
            for (uint32_t j = sub; j < filled; j += W) {
                const float4 q = scratch[2 * j + 1];
                const uint32_t i = __float_as_uint(scratch[2 * j].w);
                if (!sun_open<COUNT, REFINE>(sc, sc.lights[s], f3{q.x, q.y, q.z}, stack,  &vis))
                    atomicOr(&blocked[i >> 5], 1u << (i & 31u));
            }
        }
        __syncwarp();
        uint32_t open_count = 0;
        if (aligned) {
            // each open sample's value moves to its rank among the open samples in sample order
            // (into the shadow-ray origins' half of the slots, which is no longer read)
            for (uint32_t j = sub; j < filled; j += W) {
                const float4 v = scratch[2 * j];
                const uint32_t i = __float_as_uint(v.w), w = i >> 5, b = i & 31u;
                const uint32_t open = lit[w] & ~blocked[w];
                if ((open >> b) & 1u) {
                    uint32_t rank = __popc(open & ((1u << b) - 1u));
                    for (uint32_t u = 0; u < w; ++u) rank += __popc(lit[u] & ~blocked[u]);
                    scratch[2 * rank + 1] = v;
                }
            }
            for (uint32_t u = 0; u < net / 32; ++u) open_count += __popc(lit[u] & ~blocked[u]);
        }
        __syncwarp();
        if (aligned) {
            // the group loads the ordered values W at a time; the leader adds them in order
            const uint32_t lane0 = lane - sub;
            for (uint32_t base = 0; base < open_count; base += W) {
                float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (base + sub < open_count) q = scratch[2 * (base + sub) + 1];
                const uint32_t n = min(W, open_count - base);
                for (uint32_t t = 0; t < n; ++t) {
                    const float x = __shfl_sync(group_lanes, q.x, lane0 + t);
                    const float y = __shfl_sync(group_lanes, q.y, lane0 + t);
                    const float z = __shfl_sync(group_lanes, q.z, lane0 + t);
                    if (sub == 0) sum.add(f3{x, y, z});
                }
            }
            for (uint32_t w = sub; w < 2 * words; w += W) lit[w] = 0u;  // lit, then blocked
        }
        __syncwarp();
        if (valid && sub == 0) {
            f3 v{0.0f, 0.0f, 0.0f};
            if (active) v = divs(scale(sum.value(), sc.lights[s].bounce_intensity), (float)samples);
            a.value[item] = make_float4(v.x, v.y, v.z, active ? 1.0f : 0.0f);
        }
    }
    unsigned long long total = warp_sum(rays);
    if (lane_id() == 0 && total) atomicAdd(&a.ctr->bounce_rays, total);
    if (COUNT) {
        unsigned long long n = warp_sum(vis.nodes), t = warp_sum(vis.tris);
        if (lane_id() == 0) {
            atomicAdd(&a.ctr->gather_node_visits, n);
            atomicAdd(&a.ctr->gather_tri_tests, t);
        }
    }
    if (REFINE) add_retests(a.ctr, vis.retests);
}

// ================================ maps for moving meshes =================================
// Baked when dynamic_geometry is not LightingOnly (src/bake/baker.rs:114-152).

constexpr uint32_t kCubeRes = 64;                     // DISTANCE_CUBE_RESOLUTION (distance_cubes.rs:22)
constexpr uint64_t kProbeStream = 0x736b7970726f6265ull;  // PROBE_STREAM (sky_probes.rs:22)

// bake_distance_cubes (distance_cubes.rs:29-75): one thread per word, texels 2w (low half) and
// 2w + 1 of face f of light l; a ray from the light's centre through the texel centre, its
// closest hit within the radius, else the radius, as f16.
template <bool REFINE>
__global__ void __launch_bounds__(kBlock) k_distance_cubes(DevScene sc, uint32_t lights, uint32_t *out,
                                                           Counters *ctr) {
    int stack[kStack];
    const uint32_t per_face = kCubeRes * kCubeRes / 2;
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    Visits vis{0, 0, 0};
    if (i < (uint64_t)lights * 6 * per_face) {
        uint32_t l = (uint32_t)(i / (6 * per_face)), face = (uint32_t)(i / per_face % 6), w = (uint32_t)(i % per_face);
        const DevLight &L = sc.lights[l];
        float d[2];
        for (uint32_t k = 0; k < 2; ++k) {
            uint32_t texel = 2 * w + k;
            f3 dir = cube_texel_direction(face, texel % kCubeRes, texel / kCubeRes, kCubeRes);
            Hit h;
            d[k] = traverse<false, false, REFINE>(sc, L.position, dir, L.radius, (L.flags & kLightAlpha) != 0,
                                                  stack, h, &vis)
                       ? h.t
                       : L.radius;
        }
        out[i] = f16_bits(d[1]) << 16 | f16_bits(d[0]);
    }
    if (REFINE) add_retests(ctr, vis.retests);
}

// bake_sun_map (sun_map.rs:25-74): one thread per word (texels 2w and 2w + 1, rows of
// increasing y), a closest-hit ray along the sun's rays from the near plane, depth over the
// map's depth as unorm16; a miss (or the odd texel past the end) stores 1.
struct SunMapArgs {
    f3 side, up, along, bmin;
    float texel, depth;
    uint32_t res, words, alpha;
    uint32_t *out;
};
__device__ __forceinline__ uint32_t unorm16(float d) { return f2u(roundf(clampf(d, 0.0f, 1.0f) * 65535.0f)); }
template <bool REFINE>
__global__ void __launch_bounds__(kBlock) k_sun_map(DevScene sc, SunMapArgs a, Counters *ctr) {
    int stack[kStack];
    uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    Visits vis{0, 0, 0};
    if (w < a.words) {
        float d[2];
        for (uint32_t k = 0; k < 2; ++k) {
            uint32_t i = 2 * w + k;
            d[k] = 1.0f;
            if (i < a.res * a.res) {
                float across = a.bmin.x + ((float)(i % a.res) + 0.5f) * a.texel;
                float down = a.bmin.y + ((float)(i / a.res) + 0.5f) * a.texel;
                f3 origin = add(add(scale(a.side, across), scale(a.up, down)), scale(a.along, a.bmin.z));
                Hit h;
                if (traverse<false, false, REFINE>(sc, origin, a.along, a.depth, a.alpha != 0, stack, h, &vis))
                    d[k] = h.t / a.depth;
            }
        }
        a.out[w] = unorm16(d[1]) << 16 | unorm16(d[0]);
    }
    if (REFINE) add_retests(ctr, vis.retests);
}

// trace_probe (sky_probes.rs:83-109), kProbeLanes lanes per (probe, axis): the sky samples around
// the axis, each a closest hit (a hit at distance 0 counts as none); the open share and the rays
// that reached a triangle's back, both counts, so the lanes' samples add up in any order. One lane a
// job left the chip a few thousand threads of 64 to 256 rays each: a room's 3087 probes took 394 us,
// with 8 lanes 117 us (all maps of that room with 4, 8, 16 lanes: 193, 163, 157 us).
struct ProbeArgs {
    f3 origin;
    float spacing;
    uint32_t cx, cy, alpha;
    unsigned long long jobs;  // probes * 6
    float *open;
    uint32_t *back;
};
constexpr uint32_t kProbeLanes = 8;
template <bool REFINE>
__global__ void __launch_bounds__(kBlock) k_sky_probes(DevScene sc, ProbeArgs a, Counters *ctr) {
    int stack[kStack];
    const unsigned long long thread = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x, i = thread / kProbeLanes;
    const uint32_t sub = (uint32_t)(thread % kProbeLanes);
    Visits vis{0, 0, 0};
    uint32_t open = 0, back = 0;
    const uint32_t samples = sc.sky_samples;
    if (i < a.jobs) {
        uint64_t probe = i / 6;
        uint32_t axis = (uint32_t)(i % 6);
        uint32_t x = (uint32_t)(probe % a.cx), y = (uint32_t)(probe % ((uint64_t)a.cx * a.cy) / a.cx),
                 z = (uint32_t)(probe / ((uint64_t)a.cx * a.cy));
        f3 position = add(a.origin, f3{(float)x * a.spacing, (float)y * a.spacing, (float)z * a.spacing});
        f3 normal{0.0f, 0.0f, 0.0f};
        float sign = (axis & 1) ? -1.0f : 1.0f;
        if (axis < 2) normal.x = sign;
        else if (axis < 4) normal.y = sign;
        else normal.z = sign;
        Pcg rng = stream6(sc.seed, kProbeStream, x, y, z, axis);
        f2 off;
        off.x = rng.next_f32();
        off.y = rng.next_f32();
        f3 side, across;
        ortho_pair(normal, side, across);
        for (uint32_t taken = sub; taken < samples; taken += kProbeLanes) {
            f3 dir = cosine_direction_basis(normal, side, across, spread(taken, off, true));
            Hit h;
            bool found = traverse<false, false, REFINE>(sc, position, dir, INFINITY, a.alpha != 0, stack, h, &vis) &&
                         h.t > 0.0f;
            if (found && dot(hit_face_normal(sc, h), dir) > 0.0f) ++back;
            if (!found) ++open;
        }
    }
    for (uint32_t o = 1; o < kProbeLanes; o <<= 1) {
        open += __shfl_xor_sync(0xFFFFFFFFu, open, o);
        back += __shfl_xor_sync(0xFFFFFFFFu, back, o);
    }
    if (i < a.jobs && sub == 0) {
        a.open[i] = (float)open / (float)(samples > 1 ? samples : 1);
        a.back[i] = back;
    }
    if (REFINE) add_retests(ctr, vis.retests);
}

// The bounce window of a (mesh, light) entry: its crops' union grown by 4 (bounce_map.rs:30-43).
__host__ __device__ __forceinline__ Rect bounce_window(const uint32_t *r, uint32_t res) {
    uint32_t last = res - 1;
    return Rect{r[0] >= 4 ? r[0] - 4 : 0, r[1] >= 4 ? r[1] - 4 : 0, min(r[2] + 4, last), min(r[3] + 4, last)};
}

__global__ void k_window_sizes(DevScene sc, const uint32_t *region_rect, uint32_t entries, uint32_t *size) {
    uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e > entries) return;
    size[e] = 0;
    if (e == entries) return;
    const uint32_t *r = region_rect + (size_t)e * 4;
    uint32_t s = e % sc.light_count, m = e / sc.light_count;
    if (r[0] == kNoRect || !(sc.lights[s].flags & kLightBounce)) return;
    Rect w = bounce_window(r, sc.mesh_res[m]);
    size[e] = (w.max_x - w.min_x + 1) * (w.max_y - w.min_y + 1);
}

// Later triangles overwrite shared texels (bounce.rs:202-209): the highest triangle index that
// gathered a texel owns it; a second pass writes the owner's value.
template <bool WRITE>
__global__ void k_bounce_scatter(DevScene sc, BounceArgs a, const uint32_t *region_rect, const uint32_t *woff,
                                 uint32_t *owner, float4 *map) {
    unsigned long long item = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= a.items) return;
    float4 v = a.value[item];
    if (v.w == 0.0f) return;
    uint32_t lo = 0, hi = a.bpair_count;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if ((unsigned long long)a.bitem_off[mid] <= item) lo = mid;
        else hi = mid;
    }
    uint32_t p = a.bpairs[lo];
    uint32_t t = a.pair_tri[p], s = a.pair_light[p];
    uint32_t m = sc.tri_mesh[t];
    size_t e = (size_t)m * sc.light_count + s;
    Rect w = bounce_window(region_rect + e * 4, sc.mesh_res[m]);
    uint32_t xy = a.ctex_xy[a.ctex_off[t] + (uint32_t)(item - a.bitem_off[lo])];
    uint32_t x = xy & 0xFFFFu, y = xy >> 16;
    size_t idx = woff[e] + (size_t)(y - w.min_y) * (w.max_x - w.min_x + 1) + (x - w.min_x);
    uint32_t key = t - sc.mesh_tri_base[m] + 1;
    if (!WRITE)
        atomicMax(owner + idx, key);
    else if (owner[idx] == key)
        map[idx] = make_float4(v.x, v.y, v.z, 0.0f);
}

struct BlurWeights {
    float w[7];
    float sum;
};

// The bounce map's filter (bounce_map.rs:67-112) on a tile of kTileW x kTileH texels of a window of
// w x h: the tile and a halo of 4 (3 of the blur, 1 of the dilation) into shared memory, the dilation
// (:67-87: the first positive texel among itself and its 8 neighbours in a fixed order; outside the window
// reads 0), then one blur pass across and one down (:92-112: sample coordinates clamped to the map,
// reads outside the window are 0, sum in tap order, divided by the weights' sum). `clamp` holds the map's
// first and last column (x, y) and row (z, w) in window coordinates. A window is read once, so
// small ones are bound by launch latency and large ones by the passes' shared-memory reads: which
// texels are positive is worked out once, as a bit mask per row, so that the dilation reads one
// texel instead of nine, and a thread blurs kRun outputs in a row from one set of taps in registers.
// For callers of the filter alone (k_noalloc_filter), three launches with their intermediates in global
// memory took 12.3 us a call for 61 x 45 texels and 18.4 us for 512 x 512; one launch of tiles takes
// 6.1 us and 12.3 us (3.9 us and 10.2 us on the device). Tiles of 16 rows took 5.7 us and 10.3 us on
// the device: a small window then has too few blocks. In the bake (k_bounce_filter) a block per window,
// its passes in global memory, took 397 us on a room of large walls and 643 us on a terrain tile;
// tiles take 23 us and 40 us.
constexpr int kTileW = 32, kTileH = 8, kTileThreads = 256, kRun = 4;
constexpr int kRawW = kTileW + 8, kRawH = kTileH + 8, kWideW = kTileW + 6, kWideH = kTileH + 6;
struct FilterTile {
    float raw[kRawH][kRawW * 3], wide[kWideH][kWideW * 3], across[kWideH][kTileW * 3];
    unsigned long long lit[kRawH];  // bit c: texel c of the row has a positive channel
};
template <class Load, class Store>
__device__ __forceinline__ void filter_tile(FilterTile &s, int tx, int ty, int w, int h, int4 clamp,
                                            const BlurWeights &bw, Load load, Store store) {
    const int tid = threadIdx.x;
#pragma unroll 3
    for (int i = tid; i < kRawH * kRawW; i += kTileThreads) {
        const int row = i / kRawW, c = i % kRawW, x = tx - 4 + c, y = ty - 4 + row;
        float v[3] = {0.0f, 0.0f, 0.0f};
        if (x >= 0 && x < w && y >= 0 && y < h) load(x, y, v);
        for (int j = 0; j < 3; ++j) s.raw[row][c * 3 + j] = v[j];
    }
    __syncthreads();
    for (int row = tid >> 5; row < kRawH; row += kTileThreads / 32) {
        const int lane = tid & 31;
        const float *v = &s.raw[row][lane * 3], *u = &s.raw[row][(32 + (lane & 7)) * 3];
        const unsigned low = __ballot_sync(0xFFFFFFFFu, fmaxf(fmaxf(v[0], v[1]), v[2]) > 0.0f);
        const unsigned high = __ballot_sync(0xFFFFFFFFu, fmaxf(fmaxf(u[0], u[1]), u[2]) > 0.0f);
        if (lane == 0) s.lit[row] = low | (unsigned long long)(high & 0xFFu) << 32;
    }
    __syncthreads();
    for (int i = tid; i < kWideH * kWideW; i += kTileThreads) {
        const int row = i / kWideW, c = i % kWideW;
        const unsigned top = (unsigned)(s.lit[row] >> c) & 7u, mid = (unsigned)(s.lit[row + 1] >> c) & 7u,
                       low = (unsigned)(s.lit[row + 2] >> c) & 7u;
        // itself, the row above, left and right, the row below: the lowest bit is the first in order
        const unsigned order = (mid >> 1 & 1u) | top << 1 | (mid & 1u) << 4 | (mid >> 2) << 5 | low << 6;
        const int k = __ffs(order) - 1;  // -1: none
        const int dy = k <= 0 ? 1 : k < 4 ? 0 : k < 6 ? 1 : 2;
        const int dx = k <= 0 ? 1 : k < 4 ? k - 1 : k == 4 ? 0 : k == 5 ? 2 : k - 6;
        const float *v = &s.raw[row + dy][(c + dx) * 3];
        // zero outside the window too, so that the blur only clamps its taps to the map
        const int x = tx - 3 + c, y = ty - 3 + row;
        const bool none = k < 0 || x < 0 || x >= w || y < 0 || y >= h;
        for (int j = 0; j < 3; ++j) s.wide[row][c * 3 + j] = none ? 0.0f : v[j];
    }
    __syncthreads();
    // across: a thread takes kRun texels of one channel of a row, down: kRun rows of one column's channel
    for (int i = tid; i < kWideH * 3 * (kTileW / kRun); i += kTileThreads) {
        const int run = i % (kTileW / kRun), j = i / (kTileW / kRun) % 3, row = i / (kTileW / kRun * 3), c0 = run * kRun;
        float tap[kRun + 6];
#pragma unroll
        for (int k = 0; k < kRun + 6; ++k)
            tap[k] = s.wide[row][(min(max(tx + c0 + k - 3, clamp.x), clamp.y) - tx + 3) * 3 + j];
#pragma unroll
        for (int o = 0; o < kRun; ++o) {
            float sum = 0.0f;
#pragma unroll
            for (int k = 0; k < 7; ++k) sum = sum + tap[o + k] * bw.w[k];
            s.across[row][(c0 + o) * 3 + j] = sum / bw.sum;
        }
    }
    __syncthreads();
    for (int i = tid; i < kTileW * 3 * (kTileH / kRun); i += kTileThreads) {
        const int c = i % (kTileW * 3), r0 = i / (kTileW * 3) * kRun;
        if (tx + c / 3 >= w) continue;
        float tap[kRun + 6];
#pragma unroll
        for (int k = 0; k < kRun + 6; ++k) tap[k] = s.across[min(max(ty + r0 + k - 3, clamp.z), clamp.w) - ty + 3][c];
#pragma unroll
        for (int o = 0; o < kRun; ++o) {
            float sum = 0.0f;
#pragma unroll
            for (int k = 0; k < 7; ++k) sum = sum + tap[o + k] * bw.w[k];
            if (ty + r0 + o < h) store(tx + c / 3, ty + r0 + o, c % 3, sum / bw.sum);
        }
    }
}

// The filter of every (mesh, light) window: the scattered map A into the filtered map B, a block per
// window and part, tile by tile.
__global__ void __launch_bounds__(kTileThreads) k_bounce_filter(DevScene sc, const uint32_t *region_rect,
                                                                const uint32_t *woff, const uint32_t *wsize,
                                                                const float4 *A, float4 *B, BlurWeights bw) {
    __shared__ FilterTile tile;
    const size_t e = blockIdx.x;
    if (!wsize[e]) return;
    const uint32_t res = sc.mesh_res[e / sc.light_count];
    const Rect r = bounce_window(region_rect + e * 4, res);
    const int w = (int)(r.max_x - r.min_x + 1), h = (int)(r.max_y - r.min_y + 1);
    const int4 clamp = make_int4(-(int)r.min_x, (int)(res - 1 - r.min_x), -(int)r.min_y, (int)(res - 1 - r.min_y));
    const float4 *a = A + woff[e];
    float4 *b = B + woff[e];
    const uint32_t across = (w + kTileW - 1) / kTileW, tiles = across * ((h + kTileH - 1) / kTileH);
    for (uint32_t k = blockIdx.y; k < tiles; k += gridDim.y) {
        filter_tile(tile, (int)(k % across) * kTileW, (int)(k / across) * kTileH, w, h, clamp, bw,
                    [&](int x, int y, float v[3]) {
                        const float4 q = a[(size_t)y * w + x];
                        v[0] = q.x;
                        v[1] = q.y;
                        v[2] = q.z;
                    },
                    [&](int x, int y, int j, float v) { reinterpret_cast<float *>(b + (size_t)y * w + x)[j] = v; });
        __syncthreads();
    }
}

// BounceMap::crop's "lit" test (bounce_map.rs:124-136) per bounce pair: a warp per part scans the
// triangle's crop in the filtered window; `pair_bounce` starts at 0.
__global__ void k_bounce_lit(DevScene sc, BounceArgs a, const uint4 *tri_crop, const uint32_t *region_rect,
                             const uint32_t *woff, const float4 *map, uint8_t *pair_bounce) {
    uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    unsigned lane = lane_id();
    if (b >= a.bpair_count) return;
    uint32_t p = a.bpairs[b];
    uint32_t t = a.pair_tri[p], s = a.pair_light[p];
    uint32_t m = sc.tri_mesh[t];
    size_t e = (size_t)m * sc.light_count + s;
    Rect w = bounce_window(region_rect + e * 4, sc.mesh_res[m]);
    uint32_t ww = w.max_x - w.min_x + 1;
    uint4 c = tri_crop[t];
    uint32_t cw = c.z - c.x + 1;
    uint64_t n = (uint64_t)cw * (c.w - c.y + 1);
    bool lit = false;
    for (uint64_t base = (uint64_t)blockIdx.y * 32; base < n && !lit; base += (uint64_t)gridDim.y * 32) {
        uint64_t i = base + lane;
        bool l = false;
        if (i < n) {
            uint32_t x, y;
            grid_xy(i, cw, x, y);
            float4 v = map[woff[e] + (size_t)(c.y + y - w.min_y) * ww + (c.x + x - w.min_x)];
            l = fmaxf(fmaxf(v.x, v.y), v.z) > 0.0f;
        }
        lit = __any_sync(0xFFFFFFFFu, l);
    }
    if (lane == 0 && lit) pair_bounce[p] = 1;
}

__device__ __forceinline__ uint64_t bounce_words(uint4 crop, uint32_t bits, bool colored) {
    uint64_t n = (uint64_t)(crop.z - crop.x + 5) * (crop.w - crop.y + 5);
    if (colored) return (n * 3 * bits + 31) / 32;
    uint32_t per = 32 / bits;
    return (n + per - 1) / per;
}

// pack_bounce / pack_bounce_rgb (bounce_pack.rs:28-71) of one kept entry: the padded crop grid
// of the filtered map, dithered from the stream [seed, mesh, light, triangle] in texel order. A value
// takes a draw only when it is lit, so how far the stream has come depends on every value before: a warp
// takes a round of pixels at once (32, or as many as fill whole words), counts the lit values before
// each lane's with ballots, and each lane jumps the stream there. A round's pixels fill whole words: a
// lane per word picks them from their lanes. A thread per entry, drawing one after another, took 749 us
// for nine rooms (17 lights, colored, 5 bits) and this takes 347 us.
__global__ void k_pack_bounce(DevScene sc, uint32_t entries, const uint32_t *entry_pair,
                              const unsigned long long *entry_bdst, const uint32_t *pair_tri,
                              const uint32_t *pair_light, const uint4 *tri_crop, const uint32_t *region_rect,
                              const uint32_t *woff, const float4 *map, uint32_t *words) {
    constexpr unsigned all = 0xFFFFFFFFu;
    const uint32_t e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = lane_id();
    if (e >= entries) return;  // uniform across the warp
    const unsigned long long dst = entry_bdst[e];
    if (dst == ~0ull) return;
    const uint32_t p = entry_pair[e], t = pair_tri[p], s = pair_light[p], m = sc.tri_mesh[t];
    const DevLight &l = sc.lights[s];
    if (l.bounce_bits == 8) return;  // undithered: k_pack_bounce8
    const size_t re = (size_t)m * sc.light_count + s;
    const Rect w = bounce_window(region_rect + re * 4, sc.mesh_res[m]);
    const uint32_t ww = w.max_x - w.min_x + 1, base = woff[re];
    const uint4 c = tri_crop[t];
    const uint32_t gw = c.z - c.x + 5, gh = c.w - c.y + 5, bits = l.bounce_bits;
    Pcg rng = stream4(sc.seed, sc.mesh_id[m], l.id, t - sc.mesh_tri_base[m]);
    const bool colored = sc.colored_bounce != 0;
    // colored: one bit stream of pixels 3 * bits wide; else floor(32 / bits) pixels a word, the
    // rest of each word zero
    const uint32_t pixel_bits = colored ? 3 * bits : bits, per = 32 / bits;
    const uint32_t pixels = colored ? 32 : 32 / per * per, round_words = colored ? 3 * bits : pixels / per;
    const uint64_t n = (uint64_t)gw * gh;
    uint64_t out = dst;
    for (uint64_t at = 0; at < n; at += pixels, out += round_words) {
        const uint64_t i = at + lane;
        const bool mine = lane < pixels && i < n;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (mine) {
            uint32_t gx, gy;
            grid_xy(i, gw, gx, gy);
            if (gx >= 2 && gy >= 2 && gx < gw - 2 && gy < gh - 2)
                v = map[base + (size_t)(c.y + gy - 2 - w.min_y) * ww + (c.x + gx - 2 - w.min_x)];
        }
        const unsigned r = __ballot_sync(all, mine && bounce_draws(v.x, bits));
        const unsigned g = __ballot_sync(all, mine && colored && bounce_draws(v.y, bits));
        const unsigned b = __ballot_sync(all, mine && colored && bounce_draws(v.z, bits));
        const unsigned below = (1u << lane) - 1u;
        uint32_t pixel = 0;
        if (mine) {
            Pcg own = rng;
            own.advance(__popc(r & below) + __popc(g & below) + __popc(b & below));
            pixel = quantize_bounce(v.x, bits, own);
            if (colored) {
                pixel |= quantize_bounce(v.y, bits, own) << bits;
                pixel |= quantize_bounce(v.z, bits, own) << (2 * bits);
            }
        }
        rng.advance(__popc(r) + __popc(g) + __popc(b));
        // lane j < round_words assembles word j
        const uint64_t left = n - at;
        const uint32_t have = left < pixels ? (uint32_t)left : pixels;  // pixels of this round
        const uint32_t used = colored ? (have * pixel_bits + 31) / 32 : (have + per - 1) / per;
        const uint32_t first = colored ? lane * 32 / pixel_bits : lane * per;
        const uint32_t most = colored ? 32 / pixel_bits + 2 : per;  // pixels that may touch a word
        uint32_t word = 0;
        for (uint32_t k = 0; k < most; ++k) {
            const uint32_t from = first + k, value = __shfl_sync(all, pixel, from & 31u);
            if (from >= have) continue;
            const int shift = colored ? (int)(from * pixel_bits) - (int)(lane * 32) : (int)(k * bits);
            if (shift >= 32) continue;
            word |= shift >= 0 ? value << shift : value >> -shift;
        }
        if (lane < used) words[out + lane] = word;
    }
}

// pack_bounce(_rgb) for 8-bit bounce (bounce_pack.rs:28-86), which has no dither (its amplitude
// is 0, so no random draw is taken): every pixel quantizes on its own, so a warp packs an entry's
// part, each lane four consecutive pixels — one word of four 8-bit pixels, or three words of four
// 24-bit RGB pixels — in the padded crop grid's row-major order, as the sequential packer does.
__global__ void k_pack_bounce8(DevScene sc, uint32_t entries, const uint32_t *entry_pair,
                               const unsigned long long *entry_bdst, const uint32_t *pair_tri,
                               const uint32_t *pair_light, const uint4 *tri_crop, const uint32_t *region_rect,
                               const uint32_t *woff, const float4 *map, uint32_t *words) {
    const uint32_t e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = lane_id();
    if (e >= entries) return;  // uniform across the warp
    const unsigned long long dst = entry_bdst[e];
    if (dst == ~0ull) return;
    const uint32_t p = entry_pair[e], t = pair_tri[p], s = pair_light[p], m = sc.tri_mesh[t];
    const DevLight &l = sc.lights[s];
    if (l.bounce_bits != 8) return;  // dithered: k_pack_bounce
    const size_t re = (size_t)m * sc.light_count + s;
    const Rect w = bounce_window(region_rect + re * 4, sc.mesh_res[m]);
    const uint32_t ww = w.max_x - w.min_x + 1, base = woff[re];
    const uint4 c = tri_crop[t];
    const int gw = (int)(c.z - c.x + 5), gh = (int)(c.w - c.y + 5);
    const uint64_t n = (uint64_t)gw * gh;
    const bool colored = sc.colored_bounce != 0;
    const uint64_t nwords = colored ? (n * 24 + 31) / 32 : (n + 3) / 4;
    Pcg none{0, 0};  // never drawn from at 8 bits
    for (uint64_t g = lane + (uint64_t)blockIdx.y * 32; g * 4 < n; g += (uint64_t)gridDim.y * 32) {
        uint32_t px[4];
        for (int k = 0; k < 4; ++k) {
            const uint64_t i = g * 4 + k;
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            uint32_t ux, uy;
            grid_xy(i, (uint32_t)gw, ux, uy);
            const int gx = (int)ux, gy = (int)uy;
            if (i < n && gx >= 2 && gy >= 2 && gx < gw - 2 && gy < gh - 2) {
                const uint32_t x = c.x + gx - 2, y = c.y + gy - 2;
                v = map[base + (size_t)(y - w.min_y) * ww + (x - w.min_x)];
            }
            px[k] = 0;
            if (i < n) {
                px[k] = quantize_bounce(v.x, 8, none);
                if (colored) px[k] |= quantize_bounce(v.y, 8, none) << 8 | quantize_bounce(v.z, 8, none) << 16;
            }
        }
        if (colored) {
            const uint32_t out[3] = {px[0] | px[1] << 24, px[1] >> 8 | px[2] << 16, px[2] >> 16 | px[3] << 8};
            for (int k = 0; k < 3; ++k)
                if (g * 3 + k < nwords) words[dst + g * 3 + k] = out[k];
        } else {
            words[dst + g] = px[0] | px[1] << 8 | px[2] << 16 | px[3] << 24;
        }
    }
}

// ================================ optimize, seams, serialize ===========================

__device__ __forceinline__ uint32_t region_get(const uint32_t *pool, uint32_t off, const uint32_t *r, uint32_t bits,
                                               int64_t x, int64_t y) {
    if (x < (int64_t)r[0] || y < (int64_t)r[1] || x > (int64_t)r[2] || y > (int64_t)r[3]) return 0;
    uint64_t w = r[2] - r[0] + 1;
    uint64_t idx = (uint64_t)(x - r[0]) + (uint64_t)(y - r[1]) * w;
    if (bits == 1) return (pool[off + idx / 32] >> (idx % 32)) & 1u;
    return (pool[off + idx / 4] >> ((idx % 4) * 8)) & 0xFFu;
}

// LightEntries::optimize (shadows.rs:54-73) + any_light (:136-144): a warp per pair and part scans the
// triangle's optimize rect within the light's region for any lit texel; `keep` starts at 0.
__global__ void k_optimize(DevScene sc, uint32_t pairs, const uint32_t *pair_tri, const uint32_t *pair_light,
                           const uint32_t *region_rect, const uint32_t *region_off, const uint32_t *region_pool,
                           const uint8_t *pair_bounce, uint8_t *keep) {
    uint32_t p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    unsigned lane = lane_id();
    if (p >= pairs) return;
    uint32_t t = pair_tri[p], s = pair_light[p];
    bool k = pair_bounce && pair_bounce[p];
    if (!k) {
        TriData d;
        load_tri(sc, t, d);
        size_t e = (size_t)d.mesh * sc.light_count + s;
        Rect o = center_rect(d.uv, d.res, 1.0f);
        const uint32_t *r = region_rect + e * 4;
        uint32_t min_x = max(o.min_x, r[0]), max_x = min(o.max_x, r[2]);
        uint32_t min_y = max(o.min_y, r[1]), max_y = min(o.max_y, r[3]);
        if (min_x <= max_x && min_y <= max_y) {
            uint32_t w = max_x - min_x + 1;
            uint64_t n = (uint64_t)w * (max_y - min_y + 1);
            uint32_t bits = sc.lights[s].shadow_bits, roff = region_off[e];
            for (uint64_t base = (uint64_t)blockIdx.y * 32; base < n && !k; base += (uint64_t)gridDim.y * 32) {
                uint64_t i = base + lane;
                uint32_t x = 0, y = 0;
                if (i < n) grid_xy(i, w, x, y);
                bool lit = i < n && region_get(region_pool, roff, r, bits, min_x + x, min_y + y) != 0;
                k = __any_sync(0xFFFFFFFFu, lit);
            }
        }
    }
    if (lane == 0 && k) keep[p] = 1;
}
// Marks the kept pairs' regions as used and counts the kept entries per triangle.
__global__ void k_kept(DevScene sc, uint32_t pairs, const uint32_t *pair_tri, const uint32_t *pair_light,
                       const uint8_t *keep, uint32_t *kept_count, uint8_t *used, Counters *ctr) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = p < pairs, kept = in && keep[p];
    if (kept) {
        const uint32_t t = pair_tri[p];
        used[(size_t)sc.tri_mesh[t] * sc.light_count + pair_light[p]] = 1;
        atomicAdd(kept_count + t, 1u);
    }
    const unsigned removed = __ballot_sync(0xFFFFFFFFu, in && !kept);
    if (lane_id() == 0 && removed) atomicAdd(&ctr->lights_removed, (unsigned long long)__popc(removed));
}

// pad_seams (seams.rs:15-39) on every used region; a block per (mesh, light) entry and part. It reads
// visited texels and writes the others, so parts do not meet.
__global__ void k_pad_seams(DevScene sc, const uint8_t *used, const uint32_t *region_rect, const uint32_t *region_off,
                            uint32_t *region_pool, const uint32_t *visited, const uint64_t *grid_off) {
    size_t e = blockIdx.x;
    if (!used[e]) return;
    const uint32_t *r = region_rect + e * 4;
    uint32_t m = (uint32_t)(e / sc.light_count), s = (uint32_t)(e % sc.light_count);
    uint32_t res = sc.mesh_res[m];
    const uint32_t *vis = visited + grid_off[m];
    uint32_t bits = sc.lights[s].shadow_bits;
    uint32_t off = region_off[e];
    uint32_t w = r[2] - r[0] + 1, h = r[3] - r[1] + 1;
    auto visited_at = [&](int64_t x, int64_t y) -> bool {
        if (x < 0 || y < 0 || x >= (int64_t)res || y >= (int64_t)res) return false;
        uint64_t bit = (uint64_t)x + (uint64_t)y * res;
        return (vis[bit / 32] >> (bit % 32)) & 1u;
    };
    const int dxs[4] = {-1, 1, 0, 0}, dys[4] = {0, 0, -1, 1};
    const uint64_t n = (uint64_t)w * h, stride = (uint64_t)gridDim.y * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.y * blockDim.x + threadIdx.x; i < n; i += stride) {
        uint32_t ux, uy;
        grid_xy(i, w, ux, uy);
        int64_t x = (int64_t)r[0] + ux, y = (int64_t)r[1] + uy;
        if (visited_at(x, y)) continue;
        uint32_t level = 0;
        for (int k = 0; k < 4; ++k) {
            int64_t nx = x + dxs[k], ny = y + dys[k];
            if (visited_at(nx, ny))
                level = max(level, region_get(region_pool, off, r, bits, nx, ny));
            else if (visited_at(x + 2 * dxs[k], y + 2 * dys[k]))
                level = max(level, region_get(region_pool, off, r, bits, x + 2 * dxs[k], y + 2 * dys[k]));
        }
        if (!level) continue;  // unvisited texels hold 0 already
        if (bits == 1)
            atomicOr(region_pool + off + i / 32, 1u << (i % 32));
        else
            reinterpret_cast<uint8_t *>(region_pool + off)[i] = (uint8_t)level;
    }
}

__device__ __forceinline__ uint64_t shadow_words(uint4 crop, uint32_t bits) {
    uint64_t n = (uint64_t)(crop.z - crop.x + 5) * (crop.w - crop.y + 5);
    uint32_t per = 32 / bits;
    return (n + per - 1) / per;
}

// Words per triangle: light data (1 + stride per kept light) and payload.
__global__ void k_tri_words(DevScene sc, const uint32_t *tri_off, const uint32_t *pair_light, const uint8_t *keep,
                            const uint8_t *pair_bounce, const uint4 *tri_crop, uint32_t stride,
                            unsigned long long *ld_words, unsigned long long *pl_words) {
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t > sc.triangles) return;
    if (t == sc.triangles) {
        ld_words[t] = pl_words[t] = 0;
        return;
    }
    uint4 c = tri_crop[t];
    unsigned long long ld = 1, pl = 0;
    for (uint32_t p = tri_off[t]; p < tri_off[t + 1]; ++p)
        if (keep[p]) {
            const DevLight &l = sc.lights[pair_light[p]];
            ld += stride;
            pl += shadow_words(c, l.shadow_bits);
            if (stride == 3 && pair_bounce[p]) pl += bounce_words(c, l.bounce_bits, sc.colored_bounce != 0);
        }
    ld_words[t] = ld;
    pl_words[t] = pl;
}

__global__ void k_mesh_words(DevScene sc, const unsigned long long *ld_scan, const unsigned long long *pl_scan,
                             unsigned long long *mesh_words) {
    uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m > sc.mesh_count) return;
    if (m == sc.mesh_count) {
        mesh_words[m] = 0;
        return;
    }
    uint32_t a = sc.mesh_tri_base[m], b = sc.mesh_tri_base[m + 1];
    mesh_words[m] = 4ull * (b - a) + (ld_scan[b] - ld_scan[a]) + (pl_scan[b] - pl_scan[a]);
}

// serialize_triangles (triangle_words.rs:47-89): headers, light data, and where each kept
// entry's shadow words go.
__global__ void k_serialize(DevScene sc, const uint32_t *tri_off, const uint32_t *pair_light, const uint8_t *keep,
                            const uint8_t *pair_bounce, const uint4 *tri_crop, uint32_t stride,
                            const unsigned long long *ld_scan, const unsigned long long *pl_scan,
                            const unsigned long long *mesh_base, const uint32_t *entry_off, uint32_t *words,
                            uint32_t *entry_pair, unsigned long long *entry_dst, unsigned long long *entry_bdst) {
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= sc.triangles) return;
    uint32_t m = sc.tri_mesh[t];
    uint32_t first = sc.mesh_tri_base[m], tris = sc.mesh_tri_base[m + 1] - first;
    unsigned long long base = mesh_base[m];
    uint32_t ld_total = (uint32_t)(ld_scan[first + tris] - ld_scan[first]);
    uint32_t ld = 4 * tris + (uint32_t)(ld_scan[t] - ld_scan[first]);
    uint32_t pl = 4 * tris + ld_total + (uint32_t)(pl_scan[t] - pl_scan[first]);
    uint4 c = tri_crop[t];
    uint32_t lt = t - first;
    words[base + 4 * lt] = ld;
    words[base + 4 * lt + 1] = c.x - 2u;
    words[base + 4 * lt + 2] = c.y - 2u;
    words[base + 4 * lt + 3] = c.z - c.x + 5;
    uint32_t count = 0;
    uint32_t e = entry_off[t];
    for (uint32_t p = tri_off[t]; p < tri_off[t + 1]; ++p) {
        if (!keep[p]) continue;
        uint32_t s = pair_light[p];
        const DevLight &l = sc.lights[s];
        uint32_t at = ld + 1 + count * stride;
        words[base + at] = s;
        words[base + at + 1] = pl;
        entry_pair[e] = p;
        entry_dst[e] = base + pl;
        pl += (uint32_t)shadow_words(c, l.shadow_bits);
        entry_bdst[e] = ~0ull;
        if (stride == 3) {
            words[base + at + 2] = 0;
            if (pair_bounce[p]) {
                words[base + at + 2] = pl;
                entry_bdst[e] = base + pl;
                pl += (uint32_t)bounce_words(c, l.bounce_bits, sc.colored_bounce != 0);
            }
        }
        ++count;
        ++e;
    }
    words[base + ld] = count;
}

// crop_shadows (shadows.rs:148-159) with dilate_shadows (seams.rs:43-71), packed as
// ShadowGrid::into_words (shadow_grid.rs:91-106). A warp per kept entry, a lane per word; every
// texel of the padded grid is computed from the region directly:
//   interior: the region's level; inner ring: 3x3 max of the interior; outer ring: 3x3 max of
//   interior and inner ring.
__device__ __forceinline__ uint32_t crop_level(const uint32_t *pool, uint32_t off, const uint32_t *r, uint32_t bits,
                                               uint4 c, int gw, int gh, int gx, int gy) {
    auto interior = [&](int x, int y) -> uint32_t {
        if (x < 2 || y < 2 || x >= gw - 2 || y >= gh - 2) return 0;
        return region_get(pool, off, r, bits, (int64_t)c.x + x - 2, (int64_t)c.y + y - 2);
    };
    auto inner = [&](int x, int y) -> uint32_t {
        uint32_t v = 0;
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) v = max(v, interior(x + dx, y + dy));
        return v;
    };
    bool outer = gx == 0 || gy == 0 || gx == gw - 1 || gy == gh - 1;
    if (outer) {
        uint32_t v = 0;
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) {
                int x = gx + dx, y = gy + dy;
                if (x < 0 || y < 0 || x >= gw || y >= gh) continue;
                bool ring = x == 0 || y == 0 || x == gw - 1 || y == gh - 1;
                if (ring) continue;  // outer ring cells are 0 after the first pass
                bool in_ring = x == 1 || y == 1 || x == gw - 2 || y == gh - 2;
                v = max(v, in_ring ? inner(x, y) : interior(x, y));
            }
        return v;
    }
    bool in_ring = gx == 1 || gy == 1 || gx == gw - 2 || gy == gh - 2;
    return in_ring ? inner(gx, gy) : interior(gx, gy);
}

constexpr int kCropBytes = 2048;  // per-warp staging grid in shared memory (texels)

// 1-bit words LSB first (bits.rs:40-46): word w holds texels 32w .. 32w + 31, so lane j's texel of
// word w is bit j of a warp ballot. A warp alone ends each round of 32 words with one coalesced store
// per lane; parts take single words, every parts-th one.
template <class Texel>
__device__ __forceinline__ void ballot_words(uint64_t n, uint64_t nw, uint32_t *out, unsigned lane, uint32_t part,
                                             uint32_t parts, Texel texel) {
    if (parts > 1) {
        for (uint64_t w = part; w < nw; w += parts) {
            const uint64_t i = w * 32 + lane;
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, i < n && texel(i) != 0);
            if (lane == 0) out[w] = b;
        }
        return;
    }
    for (uint64_t base = 0; base < nw; base += 32) {
        uint32_t mine = 0;
        for (uint32_t k = 0; k < 32 && base + k < nw; ++k) {
            uint64_t i = (base + k) * 32 + lane;
            uint32_t b = __ballot_sync(0xFFFFFFFFu, i < n && texel(i) != 0);
            if (lane == k) mine = b;
        }
        if (base + lane < nw) out[base + lane] = mine;
    }
}

__global__ void __launch_bounds__(kBlock) k_crop(DevScene sc, uint32_t entries, const uint32_t *entry_pair,
                                                const unsigned long long *entry_dst, const uint32_t *pair_tri,
                                                const uint32_t *pair_light, const uint4 *tri_crop,
                                                const uint32_t *region_rect, const uint32_t *region_off,
                                                const uint32_t *region_pool, uint32_t *words) {
    __shared__ uint8_t stage[kBlock / 32][kCropBytes];
    uint32_t e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    unsigned lane = lane_id();
    if (e >= entries) return;
    uint8_t *g = stage[threadIdx.x >> 5];
    uint32_t p = entry_pair[e];
    uint32_t t = pair_tri[p], s = pair_light[p];
    uint32_t m = sc.tri_mesh[t];
    uint4 c = tri_crop[t];
    size_t re = (size_t)m * sc.light_count + s;
    const uint32_t *r = region_rect + re * 4;
    uint32_t off = region_off[re];
    uint32_t bits = sc.lights[s].shadow_bits;
    int gw = (int)(c.z - c.x + 5), gh = (int)(c.w - c.y + 5);
    uint64_t n = (uint64_t)gw * gh;
    uint32_t per = 32 / bits;
    uint64_t nw = (n + per - 1) / per;
    unsigned long long dst = entry_dst[e];
    if (n > (uint64_t)kCropBytes) {
        // large crops: every texel straight from the region, the words shared by the parts
        if (bits == 1) {
            ballot_words(n, nw, words + dst, lane, blockIdx.y, gridDim.y, [&](uint64_t i) {
                uint32_t x, y;
                grid_xy(i, (uint32_t)gw, x, y);
                return crop_level(region_pool, off, r, bits, c, gw, gh, (int)x, (int)y);
            });
            return;
        }
        for (uint64_t wi = (uint64_t)blockIdx.y * 32 + lane; wi < nw; wi += (uint64_t)gridDim.y * 32) {
            uint32_t word = 0, x, y;
            grid_xy(wi * per, (uint32_t)gw, x, y);
            for (uint32_t j = 0; j < per && wi * per + j < n; ++j) {
                word |= crop_level(region_pool, off, r, bits, c, gw, gh, (int)x, (int)y) << (j * bits);
                if (++x == (uint32_t)gw) {
                    x = 0;
                    ++y;
                }
            }
            words[dst + wi] = word;
        }
        return;
    }
    if (blockIdx.y) return;  // one part takes a small crop whole
    auto interior = [&](int x, int y) { return x >= 2 && y >= 2 && x < gw - 2 && y < gh - 2; };
    auto outer = [&](int x, int y) { return x == 0 || y == 0 || x == gw - 1 || y == gh - 1; };
    // the crop: interior texels from the region, padding rings zero
    for (int i = lane; i < (int)n; i += 32) {
        int x = i % gw, y = i / gw;
        g[i] = interior(x, y) ? (uint8_t)region_get(region_pool, off, r, bits, (int64_t)c.x + x - 2,
                                                     (int64_t)c.y + y - 2)
                              : 0;
    }
    __syncwarp();
    // first ring pass: inner ring = 3x3 max of the crop (only interior texels are non-zero there)
    for (int i = lane; i < (int)n; i += 32) {
        int x = i % gw, y = i / gw;
        if (interior(x, y) || outer(x, y)) continue;
        uint32_t v = 0;
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx)
                if (interior(x + dx, y + dy)) v = max(v, (uint32_t)g[(y + dy) * gw + x + dx]);
        g[i] = (uint8_t)v;
    }
    __syncwarp();
    // second ring pass: outer ring = 3x3 max of interior and inner ring (outer cells are 0 then)
    for (int i = lane; i < (int)n; i += 32) {
        int x = i % gw, y = i / gw;
        if (!outer(x, y)) continue;
        uint32_t v = 0;
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) {
                int xx = x + dx, yy = y + dy;
                if (xx < 0 || yy < 0 || xx >= gw || yy >= gh || outer(xx, yy)) continue;
                v = max(v, (uint32_t)g[yy * gw + xx]);
            }
        g[i] = (uint8_t)v;
    }
    __syncwarp();
    if (bits == 1) {
        ballot_words(n, nw, words + dst, lane, 0, 1, [&](uint64_t i) { return (uint32_t)g[i]; });
        return;
    }
    for (uint64_t wi = lane; wi < nw; wi += 32) {
        uint32_t word = 0;
        for (uint32_t j = 0; j < per; ++j) {
            uint64_t i = wi * per + j;
            if (i >= n) break;
            word |= (uint32_t)g[i] << (j * bits);
        }
        words[dst + wi] = word;
    }
}

// ================================ payload on the device ====================================
// The .dynlight payload assembled next to the resident words and its CRC-32 computed there, so
// the host receives finished bytes (src/bake/format/mod.rs:101-119,170-213).

// One piece of the payload: `len` words from `src` (device memory) to payload word `dst`.
struct PayloadSegment {
    unsigned long long dst;
    const uint32_t *src;
    unsigned long long len;
};
// A block per segment and part. Bound by memory (8 bytes a word); a few hundred segments of a quarter
// megabyte leave the chip idle at a block each: 26 MB in 235 segments took 1432 us, in parts 40 us.
__global__ void k_payload_gather(const PayloadSegment *seg, uint32_t *out) {
    PayloadSegment g = seg[blockIdx.x];
    const unsigned long long stride = (unsigned long long)gridDim.y * blockDim.x;
    for (unsigned long long i = (unsigned long long)blockIdx.y * blockDim.x + threadIdx.x; i < g.len; i += stride)
        out[g.dst + i] = g.src[i];
}

constexpr uint32_t kCrcChunkWords = 16384;  // 64 KiB chunks, 128 threads x 512 bytes
struct CrcShifts {
    uint32_t m[7][32];  // shift of the CRC register by 512 * 2^l bytes, l = 0 .. 6, as GF(2) columns
};
__device__ __forceinline__ uint32_t gf2_times(const uint32_t *m, uint32_t v) {
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i)
        if ((v >> i) & 1u) r ^= m[i];
    return r;
}
// The raw CRC-32 register (from zero, no inversion) of every full 64 KiB chunk: each of 128
// threads runs 512 bytes by slicing by 4 over little-endian words (Kounavis & Berry 2008), then
// the block combines the parts pairwise, raw(A B) = shift(raw(A), |B|) ^ raw(B).
__global__ void __launch_bounds__(128) k_crc_chunks(const uint32_t *data, unsigned long long chunks,
                                                    const uint32_t *tables, CrcShifts sh, uint32_t *out) {
    __shared__ uint32_t t[4][256];
    __shared__ uint32_t part[128];
    __shared__ uint32_t m[7][32];
    for (int i = threadIdx.x; i < 1024; i += 128) t[i / 256][i % 256] = tables[i];
    for (int i = threadIdx.x; i < 224; i += 128) m[i / 32][i % 32] = sh.m[i / 32][i % 32];
    __syncthreads();
    for (unsigned long long chunk = blockIdx.x; chunk < chunks; chunk += gridDim.x) {
        const uint32_t *p = data + chunk * kCrcChunkWords + threadIdx.x * 128;
        uint32_t c = 0;
        for (int i = 0; i < 128; ++i) {
            c ^= p[i];
            c = t[3][c & 0xFF] ^ t[2][(c >> 8) & 0xFF] ^ t[1][(c >> 16) & 0xFF] ^ t[0][c >> 24];
        }
        part[threadIdx.x] = c;
        __syncthreads();
        for (int l = 0; l < 7; ++l) {
            unsigned stride = 1u << l;
            if ((threadIdx.x & (2 * stride - 1)) == 0)
                part[threadIdx.x] = gf2_times(m[l], part[threadIdx.x]) ^ part[threadIdx.x + stride];
            __syncthreads();
        }
        if (threadIdx.x == 0) out[chunk] = part[0];
        __syncthreads();
    }
}

// ================================ host side =================================================

namespace {

thread_local std::string g_error;
std::mutex g_busy;

struct CudaError {
    cudaError_t code;
    const char *what;
};

#define CK(x)                                                      \
    do {                                                           \
        cudaError_t e__ = (x);                                     \
        if (e__ != cudaSuccess) throw CudaError{e__, #x};          \
    } while (0)

// Launch errors surface here, named by the kernel that caused them.
#define LAUNCHED(name)                                       \
    do {                                                     \
        cudaError_t e__ = cudaGetLastError();                \
        if (e__ != cudaSuccess) throw CudaError{e__, name};  \
    } while (0)

// Device memory comes from the device's default stream-ordered pool, allocated and freed on the
// session's stream. The pool keeps what sessions free (its release threshold is raised once per
// device), so the next bake's allocations reuse it without new cudaMalloc/cudaFree calls;
// dl_release_memory hands it back to the driver.
std::mutex g_pool_lock;
std::vector<int> g_pooled_devices;  // devices whose default pool keeps freed memory
void keep_freed_device_memory(int device) {
    std::lock_guard<std::mutex> guard(g_pool_lock);
    if (std::find(g_pooled_devices.begin(), g_pooled_devices.end(), device) != g_pooled_devices.end()) return;
    cudaMemPool_t pool;
    CK(cudaDeviceGetDefaultMemPool(&pool, device));
    uint64_t keep = ~0ull;
    CK(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    g_pooled_devices.push_back(device);
}
// Returns the pooled memory of every device the library has baked on (no other device is touched).
void release_pooled_device_memory() {
    std::lock_guard<std::mutex> guard(g_pool_lock);
    for (int d : g_pooled_devices) {
        cudaMemPool_t pool;
        if (cudaDeviceGetDefaultMemPool(&pool, d) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
    }
}
// The device memory a session holds (scene, BVH, its build scratch, every stage's buffers)
// against the caller's cap (dl_bake_config.max_device_mib; 0: none). An allocation past the cap
// fails like a failed cudaMallocAsync, so the bake reports DL_OUT_OF_MEMORY.
struct DeviceBudget {
    uint64_t cap = 0, held = 0;
    void reserve(size_t b) {
        if (cap && held + b > cap)
            throw CudaError{cudaErrorMemoryAllocation, "device memory cap (dl_bake_config.max_device_mib)"};
        held += b;
    }
    void release(size_t b) { held -= std::min<uint64_t>(held, b); }
};

void *dev_malloc(size_t bytes, cudaStream_t st, DeviceBudget *budget) {
    void *p = nullptr;
    const size_t b = std::max<size_t>(bytes, 16);
    if (budget) budget->reserve(b);
    cudaError_t e = cudaMallocAsync(&p, b, st);
    if (e != cudaSuccess) {
        if (budget) budget->release(b);
        throw CudaError{e, "cudaMallocAsync"};
    }
    return p;
}

template <class T>
T *dev_alloc(std::vector<void *> &owned, cudaStream_t st, size_t count, uint64_t &bytes, DeviceBudget *budget) {
    size_t b = std::max<size_t>(count * sizeof(T), 16);
    void *p = dev_malloc(b, st, budget);
    owned.push_back(p);
    bytes += b;
    return static_cast<T *>(p);
}

double ms_since(std::chrono::steady_clock::time_point t0) {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

}  // namespace

// A named pool of device buffers, grown on demand and reused across runs of one session;
// allocated and freed on the session's stream.
struct Pool {
    std::map<std::string, std::pair<void *, size_t>> bufs;
    cudaStream_t stream = nullptr;
    DeviceBudget *budget = nullptr;
    uint64_t bytes = 0;
    template <class T>
    T *get(const std::string &name, size_t count) {
        size_t b = std::max<size_t>(count * sizeof(T), 16);
        auto it = bufs.find(name);
        if (it != bufs.end() && it->second.second >= b) return static_cast<T *>(it->second.first);
        if (it != bufs.end()) {
            cudaFreeAsync(it->second.first, stream);
            bytes -= it->second.second;
            if (budget) budget->release(it->second.second);
            bufs.erase(it);
        }
        void *p = dev_malloc(b, stream, budget);
        bufs[name] = {p, b};
        bytes += b;
        return static_cast<T *>(p);
    }
    // Frees every buffer on the stream; the session calls it before destroying its stream.
    void release() {
        for (auto &kv : bufs) {
            cudaFreeAsync(kv.second.first, stream);
            if (budget) budget->release(kv.second.second);
        }
        bufs.clear();
        bytes = 0;
    }
};

}  // namespace dl

using namespace dl;

struct dl_session {
    HostScene host;
    dl_bake_options options{};
    dl_bake_config config{};
    int device = 0;
    int sms = 0;
    cudaStream_t stream = nullptr, side = nullptr;
    std::vector<void *> owned;
    uint64_t scene_bytes = 0;
    DevScene sc{};
    std::vector<uint64_t> grid_off;  // visited/owned word offset per mesh
    uint64_t grid_words = 0;
    std::vector<uint32_t> mesh_tri_base;
    Pool pool;
    DeviceBudget budget;  // device memory held against config.max_device_mib
    Counters *ctr = nullptr;
    uint32_t *cancel_dev = nullptr;
    dl_bake_report report{};
    uint64_t launches = 0;
    // last run's results (device)
    bool have_result = false;
    uint64_t out_words = 0;
    std::vector<unsigned long long> mesh_words;
    uint32_t *words_dev = nullptr;
    Counters counters{};
    uint64_t texels = 0;
    // last run's filtered bounce maps: window offsets per (mesh, light) entry, RGB texels, and the
    // entries' region rectangles (null when the run baked no bounce)
    const uint32_t *bounce_woff = nullptr;
    const float4 *bounce_map = nullptr;
    const uint32_t *region_rect = nullptr;
    // last run's maps for moving meshes (device buffers in the pool)
    const uint32_t *cube_words = nullptr;
    uint64_t cube_word_count = 0;
    std::vector<SunMapSetup> sun_setups;
    std::vector<const uint32_t *> sun_texels;
    ProbeGridSetup probe_grid;
    const float *probe_open = nullptr;
    const uint32_t *probe_back = nullptr;
    cudaEvent_t marks[9] = {};  // stage boundaries of the last run
    // the visibility stage's second kernel runs beside the first (made by the first run that has both)
    cudaStream_t branch = nullptr;
    cudaEvent_t forks[2] = {};
    // the payload of the last payload_build (device, in the pool) and the readers' streams
    const uint32_t *payload_dev = nullptr;
    uint64_t payload_words = 0;
    std::vector<cudaStream_t> readers;
    ~dl_session() {
        for (cudaStream_t r : readers) cudaStreamDestroy(r);
        for (auto &e : marks)
            if (e) cudaEventDestroy(e);
        for (auto &e : forks)
            if (e) cudaEventDestroy(e);
        if (branch) cudaStreamDestroy(branch);
        if (stream) {
            // back to the stream-ordered pool (kept for the next session), in stream order
            pool.release();
            for (void *p : owned) cudaFreeAsync(p, stream);
            cudaStreamSynchronize(stream);
            cudaStreamDestroy(stream);
        }
        if (side) cudaStreamDestroy(side);
    }
};

namespace dl {
namespace {

// Stack entries per thread that the scene's tree needs, rounded up to 4 (what the report names; the
// stacks themselves are kStack entries of local memory).
uint32_t stack_depth(const dl_session &s) { return std::max<uint32_t>(8, (s.host.bvh_depth + 3) & ~3u); }

void scan_u32(dl_session &s, const uint32_t *in, uint32_t *out, size_t n) {
    size_t temp = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, temp, in, out, n, s.stream));
    void *tmp = s.pool.get<uint8_t>("scan_tmp", temp);
    CK(cub::DeviceScan::ExclusiveSum(tmp, temp, in, out, n, s.stream));
    s.launches += 2;
}
void scan_u64(dl_session &s, const unsigned long long *in, unsigned long long *out, size_t n) {
    size_t temp = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, temp, in, out, n, s.stream));
    void *tmp = s.pool.get<uint8_t>("scan_tmp", temp);
    CK(cub::DeviceScan::ExclusiveSum(tmp, temp, in, out, n, s.stream));
    s.launches += 2;
}
template <class T>
T read_back(dl_session &s, const T *p) {
    T v;
    CK(cudaMemcpyAsync(&v, p, sizeof(T), cudaMemcpyDeviceToHost, s.stream));
    CK(cudaStreamSynchronize(s.stream));
    return v;
}
unsigned grid_for(size_t n, unsigned block = kBlock) { return (unsigned)std::max<size_t>(1, (n + block - 1) / block); }
// Grid of `jobs` jobs of `threads` threads each, with parts (second dimension) while the jobs alone
// leave the chip short of warps: up to kParts, aiming at kPartThreads threads (a few times what
// the SMs hold: parts of jobs that turn out small end at once). The stages that use it, at 2^18, 2^20, 2^22: a
// room under every light 0.41, 0.38, 0.38 ms, a terrain tile 0.86, 0.88, 0.98 ms, foliage 0.50, 0.53, 0.67 ms.
// Most (mesh, light) entries have no region: for them the parts are counted as if a warp took an entry.
constexpr size_t kParts = 64, kPartThreads = 1u << 20;
dim3 grid_parts(size_t jobs, unsigned threads = 32, unsigned block = kBlock) {
    const size_t want = kPartThreads / std::max<size_t>(1, jobs * threads);
    return dim3(grid_for(jobs * threads, block), (unsigned)std::min(kParts, std::max<size_t>(1, want)));
}

// Blocks the caller until the stream drains, forwarding a cancel request to the device flag. A
// forwarded request's copy (on the side stream) is waited for too, so that it cannot land after
// the next run has cleared the flag.
void wait(dl_session &s, dl_progress *progress) {
    bool forwarded = false;
    for (;;) {
        cudaError_t q = cudaStreamQuery(s.stream);
        if (q == cudaSuccess) {
            if (forwarded) CK(cudaStreamSynchronize(s.side));
            return;
        }
        if (q != cudaErrorNotReady) throw CudaError{q, "stream"};
        if (progress && progress->cancel && !forwarded) {
            static const uint32_t one = 1;
            CK(cudaMemcpyAsync(s.cancel_dev, &one, 4, cudaMemcpyHostToDevice, s.side));
            forwarded = true;
        }
        std::this_thread::yield();
    }
}

// A run that stops on the cancel flag: its report records how many warps of the device work
// queues saw the flag and stopped claiming work (0 when the request came between stages).
dl_status cancelled_run(dl_session &s) {
    Counters c{};
    CK(cudaMemcpyAsync(&c, s.ctr, sizeof(Counters), cudaMemcpyDeviceToHost, s.stream));
    CK(cudaStreamSynchronize(s.stream));
    s.report.cancel_stops = (uint32_t)c.cancelled;
    return DL_CANCELLED;
}

// Host buffers of freed results' words, handed to the next result. They are pinned (page-locked)
// when the driver allows it, so that the download runs as a DMA copy at the link's rate instead
// of through the driver's staging buffers, and a reused buffer needs no first-touch page faults
// either. At most kCacheBytes are held.
struct WordCache {
    static constexpr size_t kCacheBytes = size_t(2) << 30;
    struct Buffer {
        size_t cap;  // words
        uint32_t *p;
        bool pinned;
    };
    std::mutex lock;
    std::vector<Buffer> free;
    size_t held = 0;
    static void release(const Buffer &b) {
        if (b.pinned) cudaFreeHost(b.p);  // fails harmlessly once the runtime has shut down at exit
        else delete[] b.p;
    }
    Buffer take(size_t n) {
        {
            std::lock_guard<std::mutex> guard(lock);
            size_t best = free.size();
            for (size_t i = 0; i < free.size(); ++i)
                if (free[i].cap >= n && (best == free.size() || free[i].cap < free[best].cap)) best = i;
            if (best < free.size()) {
                Buffer b = free[best];
                free.erase(free.begin() + best);
                held -= b.cap * 4;
                return b;
            }
        }
        size_t cap = n ? n : 1;
        void *p = nullptr;
        if (cudaHostAlloc(&p, cap * 4, cudaHostAllocPortable) == cudaSuccess) return Buffer{cap, (uint32_t *)p, true};
        cudaGetLastError();  // no pinned memory to be had: a pageable buffer (a slower copy)
        return Buffer{cap, new uint32_t[cap], false};
    }
    void clear() {
        std::lock_guard<std::mutex> guard(lock);
        for (const Buffer &b : free) release(b);
        free.clear();
        held = 0;
    }
    void give(const Buffer &b) {
        std::lock_guard<std::mutex> guard(lock);
        while (held + b.cap * 4 > kCacheBytes && !free.empty()) {  // drop the oldest
            held -= free.front().cap * 4;
            release(free.front());
            free.erase(free.begin());
        }
        if (b.cap * 4 > kCacheBytes) {
            release(b);
            return;
        }
        free.push_back(b);
        held += b.cap * 4;
    }
};
WordCache &word_cache() {
    static WordCache *c = new WordCache;  // never destroyed: results may be freed during exit
    return *c;
}

// `progress`, when given, is checked for cancellation once validation has passed and before the
// first CUDA call: as in the reference (baker.rs:32-55), invalid input reports its own error even
// when the bake was already cancelled.
dl_status create(const dl_bake_input *in, const dl_bake_options *o, const dl_bake_config *cfg, dl_session *&out,
                 const dl_progress *progress = nullptr) {
    auto s = std::make_unique<dl_session>();
    s->options = *o;
    if (cfg) s->config = *cfg;
    if (s->config.form > DL_FORM_BOUNCE_REFINED) {
        g_error = "unknown bake form " + std::to_string(s->config.form);
        return DL_INVALID_ARGUMENT;
    }
    uint32_t lanes = s->config.sample_lanes;
    if (lanes > 32 || (lanes & (lanes - 1))) {
        g_error = "sample_lanes must be 0 or a power of two up to 32";
        return DL_INVALID_ARGUMENT;
    }
    const uint32_t mb = s->config.min_blocks, gmb = s->config.gather_min_blocks;
    if (!(mb == 0 || (mb >= 7 && mb <= 10) || mb == 12)) {
        g_error = "min_blocks must be 0, 7, 8, 9, 10 or 12";
        return DL_INVALID_ARGUMENT;
    }
    if (!(gmb == 0 || gmb == 6 || (gmb >= 8 && gmb <= 10))) {
        g_error = "gather_min_blocks must be 0, 6, 8, 9 or 10";
        return DL_INVALID_ARGUMENT;
    }
    float eps = s->config.refine_epsilon;
    if (!(eps >= 0.0f && eps <= 0.01f)) {
        g_error = "refine_epsilon must lie in [0, 0.01]";
        return DL_INVALID_ARGUMENT;
    }
    if (eps == 0.0f) s->config.refine_epsilon = 1.0e-4f;
    std::string err;
    auto t_prep = std::chrono::steady_clock::now();
    dl_status st = prepare_scene(*in, *o, s->host, err);
    if (st != DL_OK) {
        g_error = err;
        return st;
    }
    HostScene &h = s->host;
    for (uint32_t r : h.resolution)
        if (r > 65535) {
            g_error = "shadow maps larger than 65535 texels per side are not supported";
            return DL_UNSUPPORTED;
        }
    if (progress && progress->cancel) {
        g_error = "the bake was cancelled";
        return DL_CANCELLED;
    }
    s->report.ms_host[0] = ms_since(t_prep);
    // the occluder BVH: on the host's cores when asked, else on the device once the triangles
    // are uploaded (the same tree)
    const bool host_bvh = s->config.host_bvh != 0;
    if (host_bvh) {
        auto t_bvh = std::chrono::steady_clock::now();
        build_bvh(h);
        s->report.ms_host[1] = ms_since(t_bvh);
        // the traversal stack holds one entry per level below the root
        if (h.bvh_depth >= (uint32_t)kStack) {
            g_error = "occluder BVH deeper than the traversal stack";
            return DL_UNSUPPORTED;
        }
    }
    auto t_up = std::chrono::steady_clock::now();
    s->device = (int)s->config.device;
    CK(cudaSetDevice(s->device));
    CK(cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, s->device));
    CK(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
    CK(cudaStreamCreateWithFlags(&s->side, cudaStreamNonBlocking));
    keep_freed_device_memory(s->device);
    s->pool.stream = s->stream;
    s->budget.cap = (uint64_t)s->config.max_device_mib << 20;
    s->pool.budget = &s->budget;

    // flatten meshes
    uint32_t M = (uint32_t)h.meshes.size();
    std::vector<uint32_t> vbase(M + 1, 0), ibase(M + 1, 0), tbase(M + 1, 0), flags(M), alpha(M * 4, 0);
    std::vector<uint64_t> ids(M);
    std::vector<float> albedo(M * 3);
    std::vector<uint8_t> alpha_pool;
    for (uint32_t m = 0; m < M; ++m) {
        const dl_mesh &mm = *h.meshes[m];
        vbase[m + 1] = vbase[m] + mm.vertex_count;
        ibase[m + 1] = ibase[m] + (uint32_t)mm.index_count;
        tbase[m + 1] = tbase[m] + (uint32_t)(mm.index_count / 3);
        ids[m] = mm.id;
        for (int k = 0; k < 3; ++k) albedo[m * 3 + k] = mm.albedo[k];
        flags[m] = (mm.normals ? kMeshNormals : 0) | (mm.occludes ? kMeshOccludes : 0) |
                   (mm.alpha && mm.uv0 ? kMeshAlpha : 0);
        if (mm.alpha && mm.uv0) {
            alpha[m * 4] = (uint32_t)alpha_pool.size();
            alpha[m * 4 + 1] = mm.alpha->width;
            alpha[m * 4 + 2] = mm.alpha->height;
            std::memcpy(&alpha[m * 4 + 3], &mm.alpha->cutoff, 4);
            size_t n = (size_t)mm.alpha->width * mm.alpha->height;
            for (size_t i = 0; i < n; ++i) alpha_pool.push_back(mm.alpha->rgba8[i * 4 + 3]);
        }
    }
    uint32_t V = vbase[M], I = ibase[M], T = tbase[M];
    uint32_t N = (uint32_t)h.occ_mesh.size();
    // Every array of the scene goes into one pinned staging buffer (reused across sessions through the
    // result-word cache; it goes back once the stream has drained), the per-vertex and per-index arrays
    // flattened into it by the host's cores, and from there in one DMA copy into one device allocation.
    struct Packed {
        size_t bytes = 0;
        size_t add(size_t n) {
            const size_t at = bytes;
            bytes += (std::max<size_t>(n, 16) + 255) & ~size_t(255);
            return at;
        }
    } pack;
    const size_t at_occ_mesh = pack.add(N * 4ull), at_occ_tri = pack.add(N * 4ull), at_vbase = pack.add((M + 1) * 4ull),
                 at_ibase = pack.add((M + 1) * 4ull), at_tbase = pack.add((M + 1) * 4ull), at_res = pack.add(M * 4ull),
                 at_flags = pack.add(M * 4ull), at_ids = pack.add(M * 8ull), at_albedo = pack.add(M * 12ull),
                 at_alpha = pack.add(M * 16ull), at_alpha_pool = pack.add(alpha_pool.size()),
                 at_lights = pack.add(h.lights.size() * sizeof(DevLight)), at_pos = pack.add(V * 12ull),
                 at_nrm = pack.add(V * 12ull), at_uv1 = pack.add(V * 8ull), at_uv0 = pack.add(V * 8ull),
                 at_idx = pack.add(I * 4ull), at_tri_mesh = pack.add(T * 4ull);
    struct Staging {
        WordCache::Buffer b;
        cudaStream_t stream;
        ~Staging() {
            if (stream) cudaStreamSynchronize(stream);
            word_cache().give(b);
        }
    } staging{word_cache().take(pack.bytes / 4), s->stream};
    char *const host_at = reinterpret_cast<char *>(staging.b.p);
    float *pos = reinterpret_cast<float *>(host_at + at_pos), *nrm = reinterpret_cast<float *>(host_at + at_nrm),
          *uv1 = reinterpret_cast<float *>(host_at + at_uv1), *uv0 = reinterpret_cast<float *>(host_at + at_uv0);
    uint32_t *idx = reinterpret_cast<uint32_t *>(host_at + at_idx),
             *tri_mesh = reinterpret_cast<uint32_t *>(host_at + at_tri_mesh);
    auto flatten = [&](uint32_t m) {
        const dl_mesh &mm = *h.meshes[m];
        std::memcpy(&pos[(size_t)vbase[m] * 3], mm.positions, mm.vertex_count * 12ull);
        if (mm.normals) std::memcpy(&nrm[(size_t)vbase[m] * 3], mm.normals, mm.vertex_count * 12ull);
        else std::memset(&nrm[(size_t)vbase[m] * 3], 0, mm.vertex_count * 12ull);
        for (uint32_t v = 0; v < mm.vertex_count; ++v) {
            float a = mm.uv1[v * 2], b = mm.uv1[v * 2 + 1];
            bool ok = std::isfinite(a) && std::isfinite(b);  // mesh_builder.rs:30-40
            uv1[((size_t)vbase[m] + v) * 2] = ok ? a : 0.0f;
            uv1[((size_t)vbase[m] + v) * 2 + 1] = ok ? b : 0.0f;
        }
        if (mm.uv0) std::memcpy(&uv0[(size_t)vbase[m] * 2], mm.uv0, mm.vertex_count * 8ull);
        else std::memset(&uv0[(size_t)vbase[m] * 2], 0, mm.vertex_count * 8ull);
        std::memcpy(&idx[ibase[m]], mm.indices, mm.index_count * 4ull);
        for (uint32_t t = tbase[m]; t < tbase[m + 1]; ++t) tri_mesh[t] = m;
    };
    {
        // meshes split into contiguous runs of about equal vertex and index counts, one per thread
        // (starting threads costs more than flattening a small scene: upload with one thread and with 16, at 356 K
        // vertices and indices 0.28 and 0.44 ms, at 722 K 0.50 and 0.50 ms, at 1.04 M 0.69 and 0.54 ms)
        const unsigned cores = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
        const unsigned hw = (uint64_t)V + I < (3u << 18) ? 1u : cores;
        const uint64_t per = ((uint64_t)V + I) / hw + 1;
        std::vector<uint32_t> cut{0};
        uint64_t acc = 0;
        for (uint32_t m = 0; m < M; ++m) {
            acc += (uint64_t)h.meshes[m]->vertex_count + h.meshes[m]->index_count;
            if (acc >= per && m + 1 < M) {
                cut.push_back(m + 1);
                acc = 0;
            }
        }
        cut.push_back(M);
        std::vector<std::thread> pool;
        for (size_t r = 0; r + 2 < cut.size(); ++r)
            pool.emplace_back([&, r] {
                for (uint32_t m = cut[r]; m < cut[r + 1]; ++m) flatten(m);
            });
        for (uint32_t m = cut[cut.size() - 2]; m < cut.back(); ++m) flatten(m);
        for (auto &t : pool) t.join();
    }
    s->grid_off.resize(M + 1);
    s->grid_words = 0;
    for (uint32_t m = 0; m < M; ++m) {
        s->grid_off[m] = s->grid_words;
        s->grid_words += ((uint64_t)h.resolution[m] * h.resolution[m] + 31) / 32;
    }
    s->grid_off[M] = s->grid_words;
    s->mesh_tri_base = tbase;

    uint64_t &bytes = s->scene_bytes;
    auto up = [&](const void *src, size_t n, auto *&dst) {
        using T = std::remove_const_t<std::remove_pointer_t<std::remove_reference_t<decltype(dst)>>>;
        T *p = dev_alloc<T>(s->owned, s->stream, n / sizeof(T) + 1, bytes, &s->budget);
        if (n) CK(cudaMemcpyAsync(p, src, n, cudaMemcpyHostToDevice, s->stream));
        dst = p;
        s->report.h2d_bytes += n;
    };
    DevScene &sc = s->sc;
    sc.occluders = N;
    char *const dev_at = reinterpret_cast<char *>(dev_alloc<uint8_t>(s->owned, s->stream, pack.bytes, bytes, &s->budget));
    auto put = [&](size_t at, const void *src, size_t n) {
        if (src && n) std::memcpy(host_at + at, src, n);
        s->report.h2d_bytes += n;
    };
    auto placed = [&](size_t at, auto *&dst) { dst = reinterpret_cast<std::remove_reference_t<decltype(dst)>>(dev_at + at); };
    put(at_occ_mesh, h.occ_mesh.data(), N * 4ull);
    put(at_occ_tri, h.occ_tri.data(), N * 4ull);
    put(at_vbase, vbase.data(), vbase.size() * 4);
    put(at_ibase, ibase.data(), ibase.size() * 4);
    put(at_tbase, tbase.data(), tbase.size() * 4);
    put(at_res, h.resolution.data(), M * 4ull);
    put(at_flags, flags.data(), M * 4ull);
    put(at_ids, ids.data(), M * 8ull);
    put(at_albedo, albedo.data(), M * 12ull);
    put(at_alpha, alpha.data(), M * 16ull);
    put(at_alpha_pool, alpha_pool.data(), alpha_pool.size());
    put(at_lights, h.lights.data(), h.lights.size() * sizeof(DevLight));
    s->report.h2d_bytes += (uint64_t)V * 40 + I * 4ull + T * 4ull;  // flattened in place
    CK(cudaMemcpyAsync(dev_at, host_at, pack.bytes, cudaMemcpyHostToDevice, s->stream));
    sc.mesh_count = M;
    placed(at_occ_mesh, sc.occ_mesh);
    placed(at_occ_tri, sc.occ_tri);
    placed(at_vbase, sc.mesh_vertex_base);
    placed(at_ibase, sc.mesh_index_base);
    placed(at_tbase, sc.mesh_tri_base);
    placed(at_res, sc.mesh_res);
    placed(at_flags, sc.mesh_flags);
    placed(at_ids, sc.mesh_id);
    placed(at_albedo, sc.mesh_albedo);
    placed(at_alpha, sc.mesh_alpha);
    placed(at_alpha_pool, sc.alpha_pool);
    placed(at_lights, sc.lights);
    placed(at_pos, sc.positions);
    placed(at_nrm, sc.normals);
    placed(at_uv1, sc.uv1);
    placed(at_uv0, sc.uv0);
    placed(at_idx, sc.indices);
    placed(at_tri_mesh, sc.tri_mesh);
    double ms_bvh_device = 0.0;
    if (host_bvh) {
        std::vector<uint32_t> occ_leaf(N);
        for (uint32_t k = 0; k < N; ++k) {
            uint32_t occ;
            std::memcpy(&occ, &h.tris[k * 12 + 3], 4);
            occ_leaf[occ] = k;
        }
        std::vector<TravNode> nodes(h.nodes.size());
        for (size_t i = 0; i < nodes.size(); ++i) nodes[i] = traversal_node(h.nodes[i]);
        up(nodes.data(), nodes.size() * sizeof(TravNode), sc.nodes);
        up(h.tris.data(), h.tris.size() * 4, sc.tris);
        up(occ_leaf.data(), N * 4ull, sc.occ_leaf);
    } else {
        auto t_bvh = std::chrono::steady_clock::now();
        DeviceBvhInput bi{sc.positions, sc.indices, sc.mesh_vertex_base, sc.mesh_index_base, sc.occ_mesh,
                          sc.occ_tri, N, &s->budget.held, s->budget.cap};
        DeviceBvh db;
        try {
            build_bvh_device(bi, [&](size_t b) { return (void *)dev_alloc<uint8_t>(s->owned, s->stream, b, bytes, &s->budget); }, s->stream,
                             db);
        } catch (const DeviceBvhError &e) {
            throw CudaError{e.code, e.what};
        }
        ms_bvh_device = ms_since(t_bvh);
        s->report.ms_host[1] = ms_bvh_device;
        // the traversal stack holds one entry per level below the root
        if (db.depth >= (uint32_t)kStack) {
            g_error = "occluder BVH deeper than the traversal stack";
            return DL_UNSUPPORTED;
        }
        h.bvh_depth = db.depth;
        h.bvh_node_count = db.node_count;
        sc.nodes = db.nodes;
        sc.tris = db.tris;
        sc.occ_leaf = db.occ_leaf;
        if (N == 0) {  // no occluders: small placeholders, which traversal never reads
            sc.nodes = dev_alloc<TravNode>(s->owned, s->stream, 1, bytes, &s->budget);
            sc.tris = dev_alloc<float4>(s->owned, s->stream, 3, bytes, &s->budget);
            sc.occ_leaf = dev_alloc<uint32_t>(s->owned, s->stream, 1, bytes, &s->budget);
        }
    }
    sc.triangles = T;
    sc.light_count = (uint32_t)h.lights.size();
    sc.local_lights = h.local_lights;
    sc.seed = o->seed;
    sc.area_samples = o->area_light_samples;
    sc.area_min_samples = o->area_light_min_samples;
    sc.sky_samples = o->sky_samples;
    constexpr uint32_t kTable = 2 * kMaxOrdered - 16;
    uint16_t *tables = dev_alloc<uint16_t>(s->owned, s->stream, 2 * kTable, bytes, &s->budget);
    k_sample_tables<<<grid_for(kTable), kBlock, 0, s->stream>>>(tables, tables + kTable);
    LAUNCHED("k_sample_tables");
    sc.order_cells = tables;
    sc.cell_samples = tables + kTable;
    sc.sky_order = nullptr;
    std::vector<uint16_t> sky_order;  // for counts beyond the tables; its upload ends before this returns
    if (o->sky_samples > kMaxOrdered) {
        sky_order = sky_sample_order(o->sky_samples);
        if (!sky_order.empty()) up(sky_order.data(), sky_order.size() * 2, sc.sky_order);
    }
    sc.colored_bounce = o->colored_bounce;
    sc.refine_eps = s->config.refine_epsilon;
    sc.refine_eps2 = sc.refine_eps * sc.refine_eps;
    s->ctr = dev_alloc<Counters>(s->owned, s->stream, 1, bytes, &s->budget);
    s->cancel_dev = dev_alloc<uint32_t>(s->owned, s->stream, 1, bytes, &s->budget);
    CK(cudaStreamSynchronize(s->stream));  // allocations and uploads done (the side stream and
                                           // synchronous copies use them from here on)
    for (auto &e : s->marks) CK(cudaEventCreate(&e));
    s->report.ms_host[2] = ms_since(t_up) - ms_bvh_device;
    s->report.bvh_nodes = h.bvh_node_count;
    s->report.occluders = N;
    out = s.release();
    return DL_OK;
}


// The device pipeline of one bake. Reads back the sizes it needs between stages; everything
// else stays on the device until dl_session_result.
// ---- launch shapes of the batched visibility and gather kernels ---------------------------------
// Knobs: chunk size (warp-steps per claimed chunk), lanes sharing one sky texel's or gathered texel's
// samples, the launch bound's blocks per SM (the register budget: 7, 8, 9, 10 or 12 blocks of 128
// threads give 72, 64, 56, 48 or 40 registers per thread; the gather's 6 gives 80). A rule picks the shape:
// - sky lanes grow with the sample count, 8 from 256 samples, 4 from 128, 2 from 64, but at most 4 from
//   1 M items. Lanes that share a texel's aligned samples trace neighbouring directions, and few texels
//   with long sample loops leave the last warps alone. Visibility of a terrain tile (0.5 M items, 256
//   samples) at 1, 2, 4, 8, 16 lanes: 11.8, 9.7, 8.6, 8.4, 8.6 ms; of the outdoor quarter (2.6 M) 42.1, 38.1,
//   37.0, 38.4, 40.0 ms; of terrain with 200 samples (1.6 M) 25.2, 22.4, 21.3, 21.9, 22.6 ms; of foliage (128
//   samples) 4.5, 2.8, 1.9, 2.0, 2.1 ms; of a room (64 samples) 0.38, 0.35, 0.35, 0.36, 0.36 ms.
// - 12 blocks per SM for the sky (a 77 k triangle terrain at 9, 10, 12, 14: 23.5, 23.4, 23.1, 26.9 ms; sky rays
//   wait on the tree's far nodes, more warps hide it), 8 for the rest (rooms under panels and tubes at 8, 9,
//   10: 5.5, 5.6, 5.7 ms), 8 and 7 in the refined form (decals at 7, 8, 9, 10 for the sky: 18.4, 18.1, 19.0,
//   19.7 ms). Chunks of 32 items (the level: 64 take 1 % longer).
// - gathers with a sun take 10 blocks (a terrain of 77 k triangles 17.5 ms, at 9 17.7 ms) and 8 lanes, from 1 M
//   items 4 (tile, 1 to 16 lanes: 10.2, 8.0, 7.2, 6.8, 7.0 ms; the quarter 30.3, 27.0, 26.8, 27.1, 29.5 ms),
//   local ones alone 9 (nine rooms with 2 lanes at 6, 8, 9, 10: 14.0, 12.6, 12.5, 12.3 ms) and 2 lanes (at 9
//   blocks 1, 2, 4, 8: 13.0, 12.5, 12.3, 12.8 ms), refined ones 8 and 4 lanes (terrain 26.1, 23.1, 22.6, 23.3, 25.7 ms, decals 16.1, 14.6,
//   14.4, 15.4, 16.9 ms).
// From 1 M visibility items (256 K gather items) neighbouring register budgets are tried too, each on a
// small share of the real queue's chunks with scratch counters; their results are the same levels and
// values that the real pass writes (OR and max, and values that it overwrites), so the trials change no
// output. Lanes and chunks are left to the rule: on a small share the finer shapes look better than they
// are. The wide search that this replaces took up to 0.6 s of a first bake and ended within 2 % of
// the rule. The register budget that the trials picked, and nothing else, is kept per process, keyed by the device,
// the queue's shape and the lanes, chunk and buffer that they ran with: the rest follows from each bake's
// own samples, lights and memory cap.
using TraceKernel = void (*)(DevScene, TraceArgs);
struct TraceTune {
    uint32_t grab = 1, sky_lanes = 1, minb = 7, rest_minb = 7, stack_depth = kStack, trials = 0;
    TraceKernel sky = nullptr, rest = nullptr;  // null: no such items
    uint32_t sky_blocks = 0, rest_blocks = 0;
    double ms = 0.0;
};

// The queue's two kernels: the grouped sky phase, and the items behind it.
TraceKernel sky_kernel(bool count, bool refine, uint32_t minb) {
    if (count) return refine ? k_trace_sky<true, true, 7> : k_trace_sky<true, false, 7>;
    if (refine) return k_trace_sky<false, true, 8>;
    switch (minb) {
        case 8: return k_trace_sky<false, false, 8>;
        case 9: return k_trace_sky<false, false, 9>;
        case 10: return k_trace_sky<false, false, 10>;
        case 12: return k_trace_sky<false, false, 12>;
        default: return k_trace_sky<false, false, 7>;
    }
}
TraceKernel trace_kernel(bool count, bool refine, uint32_t minb) {
    if (count) return refine ? k_trace_batched<true, true, 7> : k_trace_batched<true, false, 7>;
    if (refine) return k_trace_batched<false, true, 7>;
    switch (minb) {
        case 8: return k_trace_batched<false, false, 8>;
        case 9: return k_trace_batched<false, false, 9>;
        case 10: return k_trace_batched<false, false, 10>;
        case 12: return k_trace_batched<false, false, 12>;
        default: return k_trace_batched<false, false, 7>;
    }
}

struct TuneKey {
    int device;
    uint64_t items, sky_items, pairs, occluders, nodes;
    uint32_t flags, blocks_per_sm, lanes, grab, buffered;
    bool operator<(const TuneKey &o) const {
        return std::tie(device, items, sky_items, pairs, occluders, nodes, flags, blocks_per_sm, lanes, grab, buffered) <
               std::tie(o.device, o.items, o.sky_items, o.pairs, o.occluders, o.nodes, o.flags, o.blocks_per_sm, o.lanes,
                        o.grab, o.buffered);
    }
};
std::mutex g_tune_lock;
std::map<TuneKey, uint32_t> g_tune_cache, g_gather_cache;  // the register budget (launch bound)
// The budget kept for a key, 0 when there is none.
uint32_t cached_budget(const std::map<TuneKey, uint32_t> &cache, const TuneKey &key) {
    std::lock_guard<std::mutex> guard(g_tune_lock);
    const auto it = cache.find(key);
    return it == cache.end() ? 0u : it->second;
}

TraceTune trace_tune(dl_session &s, TraceArgs ta, bool refine, bool count, dl_progress *progress) {
    const dl_bake_config &c = s.config;
    TraceTune best;
    best.stack_depth = stack_depth(s);
    auto blocks_of = [&](TraceKernel k) {
        int per_sm = 0;
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kBlock, 0));
        if (c.blocks_per_sm) per_sm = std::min(per_sm, (int)c.blocks_per_sm);
        return (uint32_t)std::max(1, per_sm) * (uint32_t)s.sms;
    };
    // the sky's kernel has the rule's budget and the items behind it theirs
    auto shape_for = [&](uint32_t minb) {
        best.minb = minb;
        best.sky = ta.sky_items ? sky_kernel(count, refine, minb) : nullptr;
        best.rest_minb = ta.sky_items && !c.min_blocks ? 8 : minb;
        best.rest = ta.items > ta.sky_items ? trace_kernel(count, refine, best.rest_minb) : nullptr;
        best.sky_blocks = best.sky ? blocks_of(best.sky) : 0;
        best.rest_blocks = best.rest ? blocks_of(best.rest) : 0;
    };
    const uint32_t n = s.options.sky_samples;
    const uint32_t sky_lanes = n >= 256 && ta.items < (1u << 20) ? 8 : n >= 128 ? 4 : n >= 64 ? 2 : 1;
    best.grab = c.chunk_texels ? std::max(1u, c.chunk_texels / 32) : 1u;
    best.sky_lanes = c.sample_lanes ? c.sample_lanes : ta.sky_items ? sky_lanes : 1u;
    std::vector<uint32_t> minbs = count             ? std::vector<uint32_t>{7}
                                  : refine          ? std::vector<uint32_t>{ta.sky_items ? 8u : 7u}
                                  : c.min_blocks    ? std::vector<uint32_t>{c.min_blocks}
                                  : ta.sky_items    ? std::vector<uint32_t>{12, 10}
                                                    : std::vector<uint32_t>{8, 9, 10};
    const uint32_t every = ta.items >= (4u << 20) ? 32 : ta.items >= (1u << 20) ? 16 : 0;
    const bool tune = !c.no_autotune && every && minbs.size() > 1 && !(progress && progress->cancel);
    shape_for(minbs[0]);
    if (!tune) return best;
    const TuneKey key{s.device, ta.items, ta.sky_items, ta.pairs, s.host.occ_mesh.size(), s.host.bvh_node_count,
                      0, c.blocks_per_sm, best.sky_lanes, best.grab, 0};
    if (const uint32_t kept = cached_budget(g_tune_cache, key)) {
        shape_for(kept);
        return best;
    }
    cudaStream_t st = s.stream;
    Counters *scratch = s.pool.get<Counters>("tune_counters", 1);
    ta.ctr = scratch;
    ta.sample_every = every;
    cudaEvent_t a, b;
    CK(cudaEventCreate(&a));
    CK(cudaEventCreate(&b));
    float best_ms = INFINITY;
    auto t0 = std::chrono::steady_clock::now();
    ta.grab = best.grab;
    ta.sky_lanes = best.sky_lanes;
    uint32_t fastest = minbs[0];
    for (uint32_t minb : minbs) {
        shape_for(minb);
        CK(cudaMemsetAsync(ta.head, 0, 2 * sizeof(unsigned long long), st));
        CK(cudaEventRecord(a, st));
        // only the kernel whose budget is open: the items behind a sky keep theirs
        if (best.sky) best.sky<<<best.sky_blocks, kBlock, 0, st>>>(s.sc, ta);
        else best.rest<<<best.rest_blocks, kBlock, 0, st>>>(s.sc, ta);
        CK(cudaGetLastError());
        CK(cudaEventRecord(b, st));
        CK(cudaEventSynchronize(b));
        float ms = 0.0f;
        CK(cudaEventElapsedTime(&ms, a, b));
        ++best.trials;
        if (ms < best_ms) {
            best_ms = ms;
            fastest = minb;
        }
    }
    shape_for(fastest);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    best.ms = ms_since(t0);
    std::lock_guard<std::mutex> guard(g_tune_lock);
    g_tune_cache[key] = fastest;
    return best;
}

// The gather's shape, the same way.
struct GatherTune {
    uint32_t lanes = 1, minb = 6, blocks = 1, trials = 0, buffered = 0;
    double ms = 0.0;
};
using GatherKernel = void (*)(DevScene, BounceArgs);
// `suns`: whether the scene gathers a sun's bounce.
GatherKernel gather_kernel(bool refine, uint32_t minb, bool suns, bool count = false) {
    if (count) return k_gather<true, false, 6>;
    if (refine) return k_gather<false, true, 8>;
    if (!suns && minb == 8) return k_gather<false, false, 8, false>;
    if (!suns && minb == 9) return k_gather<false, false, 9, false>;
    if (!suns && minb == 10) return k_gather<false, false, 10, false>;
    return minb == 8    ? k_gather<false, false, 8>
           : minb == 9  ? k_gather<false, false, 9>
           : minb == 10 ? k_gather<false, false, 10>
                        : k_gather<false, false, 6>;
}
bool gathers_suns(const dl_session &s) {
    for (const DevLight &l : s.host.lights)
        if (l.shape == DL_SHAPE_SUN && (l.flags & kLightBounce)) return true;
    return false;
}
// Shared memory of a gather launch: for aligned sun gathers two masks of `buffered` bits per lane
// group (at most 8 KB).
size_t gather_smem(uint32_t lanes, uint32_t buffered) {
    return (size_t)(kBlock / lanes) * 2 * (buffered / 32) * sizeof(uint32_t);
}
// The samples a lane group holds for aligned sun gathers: the largest net of a sun's bounce samples,
// from 32 to 256 (0 when there is none). Under a device-memory cap only counts that are powers of two
// themselves take the scratch that this needs; others gather without it.
uint32_t gather_buffer(const dl_session &s) {
    uint32_t most = 0;
    for (const DevLight &l : s.host.lights)
        if (l.shape == DL_SHAPE_SUN && (l.flags & kLightBounce)) {
            const uint32_t n = l.bounce_samples, net = ordered_net(n, 32, 256);
            if (net == n || !s.budget.cap) most = std::max(most, net);
        }
    return most;
}
// The lane groups' scratch of a gather launch (2 float4 per held sample per group), from the session's pool.
float4 *gather_scratch(dl_session &s, uint32_t blocks, uint32_t lanes, uint32_t buffered) {
    return s.pool.get<float4>("gather_scratch", (size_t)blocks * (kBlock / lanes) * 2 * buffered);
}

GatherTune gather_tune(dl_session &s, BounceArgs ba, uint32_t bpairs, bool refine, dl_progress *progress) {
    const dl_bake_config &c = s.config;
    const bool sun = gathers_suns(s);
    GatherTune best;
    auto blocks_for = [&](uint32_t minb, uint32_t w) {
        int per_sm = 0;
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gather_kernel(refine, minb, sun), kBlock,
                                                         gather_smem(w, gather_buffer(s))));
        if (c.blocks_per_sm) per_sm = std::min(per_sm, (int)c.blocks_per_sm);
        return (uint32_t)std::max(1, per_sm) * (uint32_t)s.sms;
    };
    best.lanes = c.sample_lanes ? c.sample_lanes : refine || (sun && ba.items >= (1u << 20)) ? 4u : sun ? 8u : 2u;
    std::vector<uint32_t> minbs = refine                ? std::vector<uint32_t>{8}
                                  : c.gather_min_blocks ? std::vector<uint32_t>{c.gather_min_blocks}
                                  : sun                 ? std::vector<uint32_t>{10, 9}
                                                        : std::vector<uint32_t>{9, 10};
    const uint32_t every = ba.items >= (1u << 20) ? 32 : ba.items >= (1u << 18) ? 16 : 0;
    // the refined gather always takes 8 (64 registers: 173 ms on the outdoor scene against 178 ms at
    // 80 registers and 173 ms at 48, its binary64 re-tests spill)
    best.minb = minbs[0];
    best.buffered = gather_buffer(s);
    best.blocks = blocks_for(best.minb, best.lanes);
    if (c.no_autotune || !every || minbs.size() == 1 || (progress && progress->cancel))
        return best;
    const TuneKey key{s.device, ba.items, 0, bpairs, s.host.occ_mesh.size(), s.host.bvh_node_count,
                      sun ? 1u : 0u, c.blocks_per_sm, best.lanes, 0, best.buffered};
    if (const uint32_t kept = cached_budget(g_gather_cache, key)) {
        best.minb = kept;
        best.blocks = blocks_for(kept, best.lanes);
        return best;
    }
    cudaStream_t st = s.stream;
    ba.ctr = s.pool.get<Counters>("tune_counters", 1);
    ba.sample_every = every;
    cudaEvent_t a, b;
    CK(cudaEventCreate(&a));
    CK(cudaEventCreate(&b));
    auto t0 = std::chrono::steady_clock::now();
    float best_ms = INFINITY;
    ba.lanes = best.lanes;
    ba.buffered = best.buffered;
    for (uint32_t minb : minbs) {
        const uint32_t blocks = blocks_for(minb, best.lanes);
        ba.scratch = gather_scratch(s, blocks, best.lanes, ba.buffered);
        CK(cudaMemsetAsync(ba.head, 0, sizeof(unsigned long long), st));
        CK(cudaEventRecord(a, st));
        gather_kernel(refine, minb, sun)<<<blocks, kBlock, gather_smem(best.lanes, ba.buffered), st>>>(
            s.sc, ba);
        CK(cudaGetLastError());
        CK(cudaEventRecord(b, st));
        CK(cudaEventSynchronize(b));
        float ms = 0.0f;
        CK(cudaEventElapsedTime(&ms, a, b));
        ++best.trials;
        if (ms < best_ms) {
            best_ms = ms;
            best.minb = minb;
            best.blocks = blocks;
        }
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    best.ms = ms_since(t0);
    std::lock_guard<std::mutex> guard(g_tune_lock);
    g_gather_cache[key] = best.minb;
    return best;
}

// Distance cubes, sun maps and sky probes of the run (src/bake/baker.rs:114-152), queued on the
// session's stream; nothing for LightingOnly.
void bake_maps(dl_session &s, bool refine) {
    const HostScene &h = s.host;
    cudaStream_t st = s.stream;
    Pool &P = s.pool;
    s.cube_words = nullptr;
    s.cube_word_count = 0;
    s.sun_setups.clear();
    s.sun_texels.clear();
    s.probe_grid = ProbeGridSetup{};
    s.probe_open = nullptr;
    s.probe_back = nullptr;
    if (s.options.dynamic_geometry == DL_GEOMETRY_LIGHTING_ONLY) return;
    if (h.local_lights) {
        s.cube_word_count = (uint64_t)h.local_lights * 6 * kCubeRes * kCubeRes / 2;
        uint32_t *cubes = P.get<uint32_t>("cube_words", s.cube_word_count);
        (refine ? k_distance_cubes<true>
                : k_distance_cubes<false>)<<<grid_for(s.cube_word_count), kBlock, 0, st>>>(
            s.sc, h.local_lights, cubes, s.ctr);
        LAUNCHED("k_distance_cubes");
        ++s.launches;
        s.cube_words = cubes;
    }
    bool any_sky = false, sky_alpha = false;
    for (uint32_t slot = h.local_lights; slot < h.lights.size(); ++slot) {
        const DevLight &l = h.lights[slot];
        if (l.shape == DL_SHAPE_SKY) {
            any_sky = true;
            sky_alpha |= (l.flags & kLightAlpha) != 0;
        }
        if (l.shape != DL_SHAPE_SUN) continue;
        SunMapSetup m = sun_map_setup(h, slot, s.options.sun_map_resolution);
        const uint32_t *texels = nullptr;
        if (!m.empty) {
            SunMapArgs a{};
            a.side = m.side;
            a.up = m.up;
            a.along = m.along;
            a.bmin = m.bmin;
            a.texel = m.texel;
            a.depth = m.depth;
            a.res = m.resolution;
            a.words = (uint32_t)(((uint64_t)m.resolution * m.resolution + 1) / 2);
            a.alpha = (l.flags & kLightAlpha) != 0;
            a.out = P.get<uint32_t>("sun_map_" + std::to_string(s.sun_setups.size()), a.words);
            (refine ? k_sun_map<true> : k_sun_map<false>)<<<grid_for(a.words), kBlock, 0, st>>>(s.sc, a, s.ctr);
            LAUNCHED("k_sun_map");
            ++s.launches;
            texels = a.out;
        }
        s.sun_setups.push_back(m);
        s.sun_texels.push_back(texels);
    }
    if (any_sky) {
        s.probe_grid = sky_probe_grid(h, s.options.sky_probe_spacing);
        if (s.probe_grid.present) {
            ProbeArgs a{};
            a.origin = s.probe_grid.origin;
            a.spacing = s.probe_grid.spacing;
            a.cx = s.probe_grid.counts[0];
            a.cy = s.probe_grid.counts[1];
            a.alpha = sky_alpha;
            a.jobs = s.probe_grid.count() * 6;
            a.open = P.get<float>("probe_open", a.jobs);
            a.back = P.get<uint32_t>("probe_back", a.jobs);
            (refine ? k_sky_probes<true>
                    : k_sky_probes<false>)<<<grid_for(a.jobs * kProbeLanes), kBlock, 0, st>>>(s.sc, a, s.ctr);
            LAUNCHED("k_sky_probes");
            ++s.launches;
            s.probe_open = a.open;
            s.probe_back = a.back;
        }
    }
}

dl_status run(dl_session &s, dl_progress *progress) {
    DevScene &sc = s.sc;
    const uint32_t T = sc.triangles, M = sc.mesh_count, L = sc.light_count;
    Pool &P = s.pool;
    cudaStream_t st = s.stream;
    const bool refine = s.config.form == DL_FORM_REFINED;
    // the refined predicates and compensated sums for the bounce stages only (photon cubes and
    // gathers): masks stay the bit-exact forms', bounce follows the refined form
    const bool refine_bounce = refine || s.config.form == DL_FORM_BOUNCE_REFINED;
    s.launches = 0;
    s.have_result = false;
    s.payload_dev = nullptr;
    s.bounce_woff = nullptr;
    s.bounce_map = nullptr;
    s.region_rect = nullptr;
    if (progress && progress->cancel) return DL_CANCELLED;
    if (progress) {
        progress->stage = 2;  // BakeStage::Meshes (src/bake/progress.rs:8-16)
        progress->total = M;
        progress->done = 0;
    }
    auto check_cancel = [&]() { return progress && progress->cancel; };
    cudaEvent_t e0, e1, v0, v1, g0, g1;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    CK(cudaEventCreate(&v0));
    CK(cudaEventCreate(&v1));
    CK(cudaEventCreate(&g0));
    CK(cudaEventCreate(&g1));
    struct EventGuard {
        cudaEvent_t *e[6];
        ~EventGuard() {
            for (auto *x : e) cudaEventDestroy(*x);
        }
    } guard{{&e0, &e1, &v0, &v1, &g0, &g1}};
    bool gathered = false;
    CK(cudaEventRecord(e0, st));
    CK(cudaMemsetAsync(s.ctr, 0, sizeof(Counters), st));
    CK(cudaMemsetAsync(s.cancel_dev, 0, 4, st));
    s.report.photon_rays = 0;
    s.report.tuned_chunk_texels = s.report.tuned_sample_lanes = s.report.tuned_blocks_per_sm = 0;
    s.report.tuned_stack_depth = s.report.tuned_min_blocks = s.report.tune_trials = 0;
    s.report.ms_tune = 0.0;
    s.report.tuned_gather_lanes = s.report.tuned_gather_min_blocks = s.report.tuned_gather_blocks_per_sm = 0;
    s.report.cancel_stops = 0;
    s.report.bounce_items = 0;
    if (T == 0) {
        // no triangles: every mesh serializes to no words (triangle_words.rs:47-56)
        CK(cudaEventRecord(v0, st));
        CK(cudaEventRecord(v1, st));
        s.launches = 0;
        bake_maps(s, refine);
        CK(cudaEventRecord(e1, st));
        CK(cudaStreamSynchronize(st));
        s.mesh_words.assign(M + 1, 0);
        s.counters = Counters{};
        s.out_words = 0;
        s.words_dev = nullptr;
        s.texels = 0;
        s.report.ms_device = s.report.ms_visibility = s.report.ms_gather = 0.0;
        s.report.pairs = 0;
        s.report.kernel_launches = s.launches;
        s.have_result = true;
        return DL_OK;
    }

    CK(cudaEventRecord(s.marks[0], st));
    // ---- setup + association
    float4 *tri_face = P.get<float4>("tri_face", T);
    uint4 *tri_crop = P.get<uint4>("tri_crop", T);
    uint32_t *tri_cnt = P.get<uint32_t>("tri_cnt", T + 1);
    uint32_t *tri_off = P.get<uint32_t>("tri_off", T + 1);
    CK(cudaMemsetAsync(tri_cnt + T, 0, 4, st));
    if (T) {
        k_setup<<<grid_for(T), kBlock, 0, st>>>(sc, tri_face, tri_crop, tri_cnt);
        LAUNCHED("k_setup");
        ++s.launches;
    }
    scan_u32(s, tri_cnt, tri_off, T + 1);
    const uint32_t pairs = read_back(s, tri_off + T);
    const size_t entries = (size_t)M * L;
    uint32_t *pair_light = P.get<uint32_t>("pair_light", pairs);
    uint32_t *pair_tri = P.get<uint32_t>("pair_tri", pairs);
    uint32_t *region_rect = P.get<uint32_t>("region_rect", entries * 4);
    if (entries) {
        k_fill_u32<<<grid_for(entries * 4), kBlock, 0, st>>>(region_rect, entries * 4, kNoRect, 0u);
        LAUNCHED("k_fill_u32");
        ++s.launches;
    }
    if (T) {
        k_assoc_fill<<<grid_for(T), kBlock, 0, st>>>(sc, tri_face, tri_crop, tri_off, pair_light, pair_tri,
                                                     region_rect);
        LAUNCHED("k_assoc_fill");
        ++s.launches;
    }
    uint32_t *region_words = P.get<uint32_t>("region_words", entries + 1);
    uint32_t *region_off = P.get<uint32_t>("region_off", entries + 1);
    k_region_words<<<grid_for(entries + 1), kBlock, 0, st>>>(region_rect, sc.lights, (uint32_t)entries, L ? L : 1,
                                                             region_words);
    LAUNCHED("k_region_words");
    ++s.launches;
    scan_u32(s, region_words, region_off, entries + 1);
    const uint32_t region_total = read_back(s, region_off + entries);
    uint32_t *region_pool = P.get<uint32_t>("region_pool", region_total);
    CK(cudaMemsetAsync(region_pool, 0, region_total * 4ull, st));

    CK(cudaEventRecord(s.marks[1], st));
    // ---- texels
    uint64_t *grid_off = P.get<uint64_t>("grid_off", M + 1);
    CK(cudaMemcpyAsync(grid_off, s.grid_off.data(), (M + 1) * 8ull, cudaMemcpyHostToDevice, st));
    uint32_t *owned = P.get<uint32_t>("owned", s.grid_words);
    uint32_t *visited = P.get<uint32_t>("visited", s.grid_words);
    CK(cudaMemsetAsync(owned, 0, s.grid_words * 4, st));
    CK(cudaMemsetAsync(visited, 0, s.grid_words * 4, st));
    uint32_t *cursor = P.get<uint32_t>("cursor", T + 1);
    uint32_t *tex_cnt = P.get<uint32_t>("tex_cnt", T + 1);
    uint32_t *tex_off = P.get<uint32_t>("tex_off", T + 1);
    const dim3 warp_grid = grid_parts(T);
    CK(cudaMemsetAsync(tex_cnt, 0, (T + 1) * 4ull, st));
    CK(cudaMemsetAsync(cursor, 0, (T + 1) * 4ull, st));
    k_texels<0><<<warp_grid, kBlock, 0, st>>>(sc, tri_face, owned, grid_off, tex_cnt, nullptr, nullptr, nullptr, nullptr,
                                              nullptr, nullptr);
    LAUNCHED("k_texels");
    k_texels<1><<<warp_grid, kBlock, 0, st>>>(sc, tri_face, owned, grid_off, tex_cnt, nullptr, nullptr, nullptr, nullptr,
                                              nullptr, nullptr);
    LAUNCHED("k_texels");
    s.launches += 2;
    scan_u32(s, tex_cnt, tex_off, T + 1);
    const uint32_t texels_all = read_back(s, tex_off + T);
    uint32_t *tex_xy = P.get<uint32_t>("tex_xy", texels_all);
    float4 *tex_pos = P.get<float4>("tex_pos", texels_all);
    float4 *tex_nrm = P.get<float4>("tex_nrm", texels_all);
    uint32_t *tex_tri = P.get<uint32_t>("tex_tri", texels_all);
    uint8_t *buried = P.get<uint8_t>("buried", texels_all);
    if (T) {
        k_texels<2><<<warp_grid, kBlock, 0, st>>>(sc, tri_face, owned, grid_off, nullptr, cursor, tex_off, tex_xy,
                                                  tex_pos, tex_nrm, tex_tri);
        LAUNCHED("k_texels");
        ++s.launches;
    }
    CK(cudaEventRecord(s.marks[2], st));
    if (texels_all) {
        auto burial = refine ? k_burial<true> : k_burial<false>;
        burial<<<grid_for(texels_all), kBlock, 0, st>>>(sc, texels_all, tex_xy, tex_pos, tex_tri, tri_face, buried,
                                                        s.ctr);
        LAUNCHED("k_burial");
        ++s.launches;
    }
    uint32_t *ctex_cnt = P.get<uint32_t>("ctex_cnt", T + 1);
    uint32_t *ctex_off = P.get<uint32_t>("ctex_off", T + 1);
    CK(cudaMemsetAsync(ctex_cnt, 0, (T + 1) * 4ull, st));
    CK(cudaMemsetAsync(cursor, 0, (T + 1) * 4ull, st));
    if (T) {
        k_unburied<false><<<warp_grid, kBlock, 0, st>>>(T, tex_off, buried, ctex_cnt, nullptr, nullptr, nullptr, nullptr,
                                                        nullptr, nullptr, nullptr, nullptr);
        LAUNCHED("k_unburied");
        ++s.launches;
    }
    scan_u32(s, ctex_cnt, ctex_off, T + 1);
    const uint32_t texels = read_back(s, ctex_off + T);
    uint32_t *ctex_xy = P.get<uint32_t>("ctex_xy", texels);
    float4 *ctex_pos = P.get<float4>("ctex_pos", texels);
    float4 *ctex_nrm = P.get<float4>("ctex_nrm", texels);
    if (T) {
        k_unburied<true><<<warp_grid, kBlock, 0, st>>>(T, tex_off, buried, nullptr, cursor, ctex_off, tex_xy, tex_pos,
                                                       tex_nrm, ctex_xy, ctex_pos, ctex_nrm);
        LAUNCHED("k_unburied");
        ++s.launches;
    }
    s.texels = texels;
    if (check_cancel()) return DL_CANCELLED;

    CK(cudaEventRecord(s.marks[3], st));
    // ---- visibility
    TraceArgs ta{};
    ta.pair_tri = pair_tri;
    ta.pair_light = pair_light;
    ta.ctex_off = ctex_off;
    ta.ctex_xy = ctex_xy;
    ta.ctex_pos = ctex_pos;
    ta.ctex_nrm = ctex_nrm;
    ta.tri_face = tri_face;
    ta.grid_off = grid_off;
    ta.visited = visited;
    ta.region_rect = region_rect;
    ta.region_off = region_off;
    ta.region_pool = region_pool;
    ta.ctr = s.ctr;
    ta.cancel = s.cancel_dev;
    if (s.config.form == DL_FORM_PLAIN) {
        CK(cudaEventRecord(v0, st));
        for (uint32_t m = 0; m < M; ++m) {
            uint32_t first = s.mesh_tri_base[m], count = s.mesh_tri_base[m + 1] - first;
            if (!count) continue;
            unsigned blocks = (unsigned)std::min<size_t>(grid_for((size_t)count * 32), (size_t)s.sms * 16);
            k_trace_plain<<<blocks, kBlock, 0, st>>>(sc, ta, first, count, tri_off);
            LAUNCHED("k_trace_plain");
            ++s.launches;
            if (progress) progress->done = m + 1;
        }
        CK(cudaEventRecord(v1, st));
    } else {
        // queue: pairs ordered sky, soft, hard; item prefix sums over their texel counts
        uint32_t *order = P.get<uint32_t>("order", pairs + 1);
        // packed class flags and their scan, then (in the same room) item counts and their prefix sums
        unsigned long long *flag = P.get<unsigned long long>("queue", 2 * ((size_t)pairs + 1));
        unsigned long long *fpos = flag + pairs + 1;
        uint32_t *icnt = reinterpret_cast<uint32_t *>(flag), *item_off = reinterpret_cast<uint32_t *>(fpos);
        unsigned long long *heads = P.get<unsigned long long>("heads", 2);
        uint32_t *sizes = reinterpret_cast<uint32_t *>(heads);  // until the queue is drained
        k_pair_class<<<grid_for(pairs + 1), kBlock, 0, st>>>(sc, pair_light, pairs, flag);
        LAUNCHED("k_pair_class");
        scan_u64(s, flag, fpos, pairs + 1);
        k_pair_scatter<<<grid_for(pairs), kBlock, 0, st>>>(flag, fpos, pairs, order, sizes);
        LAUNCHED("k_pair_scatter");
        k_item_counts<<<grid_for(pairs + 1), kBlock, 0, st>>>(order, pair_tri, ctex_off, pairs, icnt);
        LAUNCHED("k_item_counts");
        scan_u32(s, icnt, item_off, pairs + 1);
        k_queue_sizes<<<1, 1, 0, st>>>(item_off, pairs, sizes);
        LAUNCHED("k_queue_sizes");
        s.launches += 4;
        const unsigned long long queued = read_back(s, heads + 1);
        const uint32_t items = (uint32_t)queued, sky_items = (uint32_t)(queued >> 32);
        s.report.work_items = items;
        ta.order = order;
        ta.item_off = item_off;
        ta.pairs = pairs;
        ta.items = items;
        ta.head = heads;
        ta.head_sky = heads + 1;
        ta.sky_items = sky_items;
        ta.sample_every = 1;
        const bool count = s.config.count_visits != 0;  // instrumented variant: counts node visits
        TraceTune tune = trace_tune(s, ta, refine, count, progress);
        s.report.tuned_chunk_texels = tune.grab * 32;
        s.report.tuned_sample_lanes = tune.sky_lanes;
        s.report.tuned_blocks_per_sm = std::max(tune.sky_blocks ? tune.sky_blocks : tune.rest_blocks, (uint32_t)s.sms) / s.sms;
        s.report.tuned_stack_depth = tune.stack_depth;
        s.report.tuned_min_blocks = tune.minb;
        s.report.tune_trials = tune.trials;
        s.report.ms_tune = tune.ms;
        ta.grab = tune.grab;
        ta.sky_lanes = tune.sky_lanes;
        CK(cudaEventRecord(v0, st));
        CK(cudaMemsetAsync(heads, 0, 2 * sizeof(unsigned long long), st));
        // The two kernels claim from heads of their own, so they run side by side: blocks of one take the
        // SMs that the other's last blocks leave (a 77 k triangle terrain 24.1 -> 23.4 ms, foliage 2.58 -> 1.95 ms).
        // Launched directly: a graph of these nodes saves nothing and cost a one-off bake its instantiation.
        // One after the other where a caller bounds the persistent blocks per SM: the bound holds for both together.
        const bool fork = tune.sky && tune.rest && !s.config.blocks_per_sm;
        if (fork) {
            if (!s.branch) {
                CK(cudaStreamCreateWithFlags(&s.branch, cudaStreamNonBlocking));
                for (auto &e : s.forks) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
            }
            CK(cudaEventRecord(s.forks[0], st));
            CK(cudaStreamWaitEvent(s.branch, s.forks[0], 0));
        }
        if (tune.sky) tune.sky<<<tune.sky_blocks, kBlock, 0, st>>>(sc, ta);
        if (tune.rest) tune.rest<<<tune.rest_blocks, kBlock, 0, fork ? s.branch : st>>>(sc, ta);
        const cudaError_t launched = cudaGetLastError();
        if (fork) {
            CK(cudaEventRecord(s.forks[1], s.branch));
            CK(cudaStreamWaitEvent(st, s.forks[1], 0));
        }
        CK(launched);
        s.launches += (tune.sky != nullptr) + (tune.rest != nullptr);
        CK(cudaEventRecord(v1, st));
    }
    wait(s, progress);
    if (check_cancel()) return cancelled_run(s);

    CK(cudaEventRecord(s.marks[4], st));
    // ---- one bounce: photon cubes, gathers, bounce maps (bounce.rs:48-217)
    const HostScene &hs = s.host;
    uint8_t *pair_bounce = P.get<uint8_t>("pair_bounce", pairs);
    CK(cudaMemsetAsync(pair_bounce, 0, pairs, st));
    uint32_t *woff = nullptr;
    float4 *bmap = nullptr;
    if (hs.bounce_in_scene && pairs) {
        const uint32_t res = s.options.photon_cube_resolution;
        const uint32_t cubes = (uint32_t)hs.cube_lights.size();
        const uint64_t photons_n = 6ull * res * res * cubes;
        Photon *photons = P.get<Photon>("photons", photons_n);
        if (cubes) {
            uint32_t *cube_lights = P.get<uint32_t>("cube_lights", cubes);
            CK(cudaMemcpyAsync(cube_lights, hs.cube_lights.data(), cubes * 4ull, cudaMemcpyHostToDevice, st));
            auto photon = refine_bounce ? k_photons<true> : k_photons<false>;
            photon<<<grid_for(photons_n), kBlock, 0, st>>>(sc, cube_lights, cubes, res, photons, s.ctr);
            LAUNCHED("k_photons");
            ++s.launches;
        }
        s.report.photon_rays = photons_n;
        uint32_t *bflag = P.get<uint32_t>("bflag", pairs + 1);
        uint32_t *bpos = P.get<uint32_t>("bpos", pairs + 1);
        k_bounce_flag<<<grid_for(pairs + 1), kBlock, 0, st>>>(sc, pair_light, pairs, bflag);
        LAUNCHED("k_bounce_flag");
        scan_u32(s, bflag, bpos, pairs + 1);
        const uint32_t bcount = read_back(s, bpos + pairs);
        uint32_t *bpairs = P.get<uint32_t>("bpairs", bcount + 1);
        k_pair_compact<<<grid_for(pairs), kBlock, 0, st>>>(bflag, bpos, pairs, bpairs);
        LAUNCHED("k_pair_compact");
        uint32_t *bcnt = P.get<uint32_t>("bcnt", bcount + 1);
        uint32_t *bitem_off = P.get<uint32_t>("bitem_off", bcount + 1);
        k_item_counts<<<grid_for(bcount + 1), kBlock, 0, st>>>(bpairs, pair_tri, ctex_off, bcount, bcnt);
        LAUNCHED("k_item_counts");
        scan_u32(s, bcnt, bitem_off, bcount + 1);
        const uint32_t bitems = read_back(s, bitem_off + bcount);
        s.report.bounce_items = bitems;
        s.launches += 3;
        float4 *bval = P.get<float4>("bval", bitems);
        BounceArgs ba{};
        ba.pair_tri = pair_tri;
        ba.pair_light = pair_light;
        ba.ctex_off = ctex_off;
        ba.ctex_xy = ctex_xy;
        ba.ctex_pos = ctex_pos;
        ba.tri_face = tri_face;
        ba.bpairs = bpairs;
        ba.bitem_off = bitem_off;
        ba.bpair_count = bcount;
        ba.items = bitems;
        ba.photons = photons;
        ba.res = res;
        ba.value = bval;
        ba.ctr = s.ctr;
        ba.cancel = s.cancel_dev;
        if (bitems) {
            ba.head = P.get<unsigned long long>("gather_head", 1);
            ba.sample_every = 1;
            GatherTune g = gather_tune(s, ba, bcount, refine_bounce, progress);
            ba.lanes = g.lanes;
            ba.buffered = g.buffered;
            ba.scratch = gather_scratch(s, g.blocks, g.lanes, g.buffered);
            s.report.tuned_gather_lanes = g.lanes;
            s.report.tuned_gather_min_blocks = g.minb;
            s.report.tuned_gather_blocks_per_sm = g.blocks / (uint32_t)s.sms;
            s.report.tune_trials += g.trials;
            s.report.ms_tune += g.ms;
            CK(cudaMemsetAsync(ba.head, 0, sizeof(unsigned long long), st));
            // the instrumented variant (counting node visits and triangle tests) when asked
            CK(cudaEventRecord(g0, st));
            gather_kernel(refine_bounce, g.minb, gathers_suns(s), s.config.count_visits != 0 && !refine_bounce)<<<
                g.blocks, kBlock, gather_smem(g.lanes, g.buffered), st>>>(sc, ba);
            LAUNCHED("k_gather");
            CK(cudaEventRecord(g1, st));
            gathered = true;
            ++s.launches;
        }
        // windows per (mesh, bounce light)
        uint32_t *wsize = P.get<uint32_t>("wsize", entries + 1);
        woff = P.get<uint32_t>("woff", entries + 1);
        k_window_sizes<<<grid_for(entries + 1), kBlock, 0, st>>>(sc, region_rect, (uint32_t)entries, wsize);
        LAUNCHED("k_window_sizes");
        scan_u32(s, wsize, woff, entries + 1);
        const uint32_t wtotal = read_back(s, woff + entries);
        uint32_t *owner = P.get<uint32_t>("owner", wtotal);
        float4 *mapA = P.get<float4>("mapA", wtotal);
        bmap = P.get<float4>("mapB", wtotal);
        CK(cudaMemsetAsync(owner, 0, wtotal * 4ull, st));
        CK(cudaMemsetAsync(mapA, 0, wtotal * 16ull, st));
        if (bitems) {
            k_bounce_scatter<false><<<grid_for(bitems), kBlock, 0, st>>>(sc, ba, region_rect, woff, owner, mapA);
            LAUNCHED("k_bounce_scatter");
            k_bounce_scatter<true><<<grid_for(bitems), kBlock, 0, st>>>(sc, ba, region_rect, woff, owner, mapA);
            LAUNCHED("k_bounce_scatter");
            s.launches += 2;
        }
        BlurWeights bw;
        std::copy(hs.blur_weights, hs.blur_weights + 7, bw.w);
        bw.sum = hs.blur_weight_sum;
        k_bounce_filter<<<dim3((unsigned)entries, grid_parts(entries).y), kTileThreads, 0, st>>>(
            sc, region_rect, woff, wsize, mapA, bmap, bw);
        LAUNCHED("k_bounce_filter");
        if (bcount) {
            k_bounce_lit<<<grid_parts(bcount), kBlock, 0, st>>>(sc, ba, tri_crop, region_rect, woff, bmap,
                                                                           pair_bounce);
            LAUNCHED("k_bounce_lit");
            ++s.launches;
        }
        s.launches += 3;
    }

    CK(cudaEventRecord(s.marks[5], st));
    // ---- optimize, seams
    uint8_t *keep = P.get<uint8_t>("keep", pairs);
    uint32_t *kept_cnt = P.get<uint32_t>("kept_cnt", T + 1);
    uint32_t *entry_off = P.get<uint32_t>("entry_off", T + 1);
    uint8_t *used = P.get<uint8_t>("used", entries);
    CK(cudaMemsetAsync(used, 0, entries, st));
    CK(cudaMemsetAsync(kept_cnt, 0, (T + 1) * 4ull, st));
    if (pairs) {
        CK(cudaMemsetAsync(keep, 0, pairs, st));
        k_optimize<<<grid_parts(pairs), kBlock, 0, st>>>(sc, pairs, pair_tri, pair_light, region_rect, region_off,
                                                         region_pool, pair_bounce, keep);
        LAUNCHED("k_optimize");
        k_kept<<<grid_for(pairs), kBlock, 0, st>>>(sc, pairs, pair_tri, pair_light, keep, kept_cnt, used, s.ctr);
        LAUNCHED("k_kept");
        s.launches += 2;
    }
    if (entries) {
        k_pad_seams<<<dim3((unsigned)entries, grid_parts(entries).y), kBlock, 0, st>>>(sc, used, region_rect, region_off, region_pool, visited,
                                                          grid_off);
        LAUNCHED("k_pad_seams");
        ++s.launches;
    }
    scan_u32(s, kept_cnt, entry_off, T + 1);
    const uint32_t kept = read_back(s, entry_off + T);

    CK(cudaEventRecord(s.marks[6], st));
    // ---- serialize
    const uint32_t stride = s.host.bounce_in_scene ? 3 : 2;
    unsigned long long *ld_words = P.get<unsigned long long>("ld_words", T + 1);
    unsigned long long *pl_words = P.get<unsigned long long>("pl_words", T + 1);
    unsigned long long *ld_scan = P.get<unsigned long long>("ld_scan", T + 1);
    unsigned long long *pl_scan = P.get<unsigned long long>("pl_scan", T + 1);
    k_tri_words<<<grid_for(T + 1), kBlock, 0, st>>>(sc, tri_off, pair_light, keep, pair_bounce, tri_crop, stride,
                                                    ld_words, pl_words);
    LAUNCHED("k_tri_words");
    ++s.launches;
    scan_u64(s, ld_words, ld_scan, T + 1);
    scan_u64(s, pl_words, pl_scan, T + 1);
    unsigned long long *mesh_words = P.get<unsigned long long>("mesh_words", M + 1);
    unsigned long long *mesh_base = P.get<unsigned long long>("mesh_base", M + 1);
    k_mesh_words<<<grid_for(M + 1), kBlock, 0, st>>>(sc, ld_scan, pl_scan, mesh_words);
    LAUNCHED("k_mesh_words");
    ++s.launches;
    scan_u64(s, mesh_words, mesh_base, M + 1);
    const unsigned long long total_words = read_back(s, mesh_base + M);
    uint32_t *words = P.get<uint32_t>("words", total_words);
    uint32_t *entry_pair = P.get<uint32_t>("entry_pair", kept);
    unsigned long long *entry_dst = P.get<unsigned long long>("entry_dst", kept);
    unsigned long long *entry_bdst = P.get<unsigned long long>("entry_bdst", kept);
    if (T) {
        k_serialize<<<grid_for(T), kBlock, 0, st>>>(sc, tri_off, pair_light, keep, pair_bounce, tri_crop, stride, ld_scan,
                                                    pl_scan, mesh_base, entry_off, words, entry_pair, entry_dst,
                                                    entry_bdst);
        LAUNCHED("k_serialize");
        ++s.launches;
    }
    if (kept) {
        k_crop<<<grid_parts(kept), kBlock, 0, st>>>(sc, kept, entry_pair, entry_dst, pair_tri, pair_light,
                                                               tri_crop, region_rect, region_off, region_pool, words);
        LAUNCHED("k_crop");
        ++s.launches;
        if (bmap) {
            k_pack_bounce<<<grid_for((size_t)kept * 32), kBlock, 0, st>>>(sc, kept, entry_pair, entry_bdst, pair_tri, pair_light,
                                                             tri_crop, region_rect, woff, bmap, words);
            LAUNCHED("k_pack_bounce");
            k_pack_bounce8<<<grid_parts(kept), kBlock, 0, st>>>(
                sc, kept, entry_pair, entry_bdst, pair_tri, pair_light, tri_crop, region_rect, woff, bmap, words);
            LAUNCHED("k_pack_bounce8");
            s.launches += 2;
        }
    }
    CK(cudaEventRecord(s.marks[7], st));
    // ---- maps for moving meshes
    bake_maps(s, refine);
    CK(cudaEventRecord(s.marks[8], st));
    CK(cudaEventRecord(e1, st));
    s.mesh_words.resize(M + 1);
    CK(cudaMemcpyAsync(s.mesh_words.data(), mesh_words, (M + 1) * 8ull, cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&s.counters, s.ctr, sizeof(Counters), cudaMemcpyDeviceToHost, st));
    wait(s, progress);
    if (check_cancel()) return cancelled_run(s);
    float ms = 0.0f, vms = 0.0f;
    CK(cudaEventElapsedTime(&ms, e0, e1));
    CK(cudaEventElapsedTime(&vms, v0, v1));
    s.report.ms_device = ms;
    s.report.ms_visibility = vms;
    float gms = 0.0f;
    if (gathered) CK(cudaEventElapsedTime(&gms, g0, g1));
    s.report.ms_gather = gms;
    for (int k = 0; k < 8; ++k) {
        float ms_k = 0.0f;
        CK(cudaEventElapsedTime(&ms_k, s.marks[k], s.marks[k + 1]));
        s.report.ms_stages[k] = ms_k;
    }
    s.report.pairs = pairs;
    s.report.shadow_rays = s.counters.rays;
    s.report.burial_rays = s.counters.burial_rays;
    s.report.bounce_rays = s.counters.bounce_rays;
    s.report.node_visits = s.counters.node_visits;
    s.report.tri_tests = s.counters.tri_tests;
    s.report.gather_node_visits = s.counters.gather_node_visits;
    s.report.gather_tri_tests = s.counters.gather_tri_tests;
    s.report.retests = s.counters.retests;
    s.report.kernel_launches = s.launches;
    s.report.device_bytes = s.scene_bytes + P.bytes;
    s.out_words = total_words;
    s.words_dev = words;
    s.bounce_woff = woff;
    s.bounce_map = bmap;
    s.region_rect = region_rect;
    s.have_result = true;
    if (progress) {  // BakeStage::Done with its counters cleared, as progress.begin(Done, 0) leaves them
        progress->done = 0;
        progress->total = 0;
        progress->stage = 4;
    }
    return DL_OK;
}

// The result in one host allocation: the scene struct, its arrays, then the words.
struct HostResult {
    dl_baked_scene scene;
    std::vector<dl_baked_light> lights;
    std::vector<dl_light_bvh_node> bvh;
    std::vector<dl_baked_mesh> meshes;
    uint32_t *words = nullptr;  // buffer.p
    WordCache::Buffer buffer{0, nullptr, false};  // from word_cache()
    ~HostResult() {
        if (buffer.p) word_cache().give(buffer);
    }
    std::vector<uint32_t> cubes;
    std::vector<std::vector<uint32_t>> sun_words;
    std::vector<dl_sun_map> sun_maps;
    std::vector<uint32_t> probe_words;
    dl_sky_probes probes{};
};

// Copies n words into host memory mapped for the device (pinned, written over the CPU-GPU link
// by the SMs): 16-byte stores to the 16-byte aligned `dst`, 16-byte loads where `src` is aligned too, the tail
// word by word.
__global__ void k_copy_words(const uint32_t *src, uint32_t *dst, uint64_t n) {
    const uint64_t n4 = n / 4, stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint4 *d4 = reinterpret_cast<uint4 *>(dst);
    if (reinterpret_cast<uintptr_t>(src) % 16 == 0) {
        const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
        for (uint64_t i = first; i < n4; i += stride) d4[i] = s4[i];
    } else {
        for (uint64_t i = first; i < n4; i += stride)
            d4[i] = make_uint4(src[4 * i], src[4 * i + 1], src[4 * i + 2], src[4 * i + 3]);
    }
    for (uint64_t i = n4 * 4 + first; i < n; i += stride) dst[i] = src[i];
}

// The last run's scene. With `download` false the triangle words, distance cubes and sun map
// texels stay on the device and the scene's pointers to them are device pointers (for the
// device-side payload encode); everything else is on the host either way.
dl_status assemble(dl_session &s, std::unique_ptr<HostResult> &r, bool download) {
    if (!s.have_result) {
        g_error = "no finished run in this session";
        return DL_INVALID_ARGUMENT;
    }
    r = std::make_unique<HostResult>();
    const HostScene &h = s.host;
    const uint32_t *words = s.words_dev;
    if (download) {
        r->buffer = word_cache().take(s.out_words);
        r->words = r->buffer.p;
        uint32_t *mapped = nullptr;
        if (s.out_words && r->buffer.pinned &&
            cudaHostGetDevicePointer((void **)&mapped, r->words, 0) == cudaSuccess) {
            // the SMs write the words into the pinned buffer: as fast as the copy engine here,
            // and steadier (the copy engine's rate varied 10x between sessions on some machines)
            k_copy_words<<<s.sms * 8, 256, 0, s.stream>>>(s.words_dev, mapped, s.out_words);
            LAUNCHED("k_copy_words");
            CK(cudaStreamSynchronize(s.stream));
        } else if (s.out_words) {
            cudaGetLastError();  // a buffer the device cannot map: the copy engine
            CK(cudaMemcpy(r->words, s.words_dev, s.out_words * 4, cudaMemcpyDeviceToHost));
        }
        words = r->words;
        s.report.d2h_bytes = s.out_words * 4 + (s.mesh_words.size() * 8) + sizeof(Counters);
    }
    uint64_t at = 0;
    for (uint32_t m = 0; m < h.meshes.size(); ++m) {
        const dl_mesh &mm = *h.meshes[m];
        dl_baked_mesh b{};
        b.id = mm.id;
        b.content_hash = mm.content_hash;
        b.resolution = h.resolution[m];
        b.occludes = mm.occludes ? 1 : 0;
        b.triangles = words + at;
        b.word_count = s.mesh_words[m];
        at += s.mesh_words[m];
        r->meshes.push_back(b);
    }
    const dl_bake_options &o = s.options;
    for (size_t i = 0; i < h.light_ptrs.size(); ++i) {
        const dl_light &l = *h.light_ptrs[i];
        const DevLight &d = h.lights[i];
        dl_baked_light b{};
        b.id = l.id;
        for (int k = 0; k < 3; ++k) b.origin[k] = l.position[k];
        b.radius = l.radius;
        b.shape = l.shape;
        // the file's shape record (format/lights.rs:27-52): rotation and size only for area/sun
        bool shaped = l.shape != DL_SHAPE_POINT && l.shape != DL_SHAPE_SKY;
        b.rotation[0] = shaped ? l.rotation[0] : 0.0f;
        b.rotation[1] = shaped ? l.rotation[1] : 0.0f;
        b.rotation[2] = shaped ? l.rotation[2] : 0.0f;
        b.rotation[3] = shaped ? l.rotation[3] : 1.0f;
        b.size[0] = shaped ? l.size[0] : 0.0f;
        b.size[1] = (l.shape == DL_SHAPE_RECTANGLE || l.shape == DL_SHAPE_TUBE) ? l.size[1] : 0.0f;
        b.bounce_bits = d.bounce_bits;
        b.shadow_bits_per_texel = d.shadow_bits;
        r->lights.push_back(b);
    }
    r->bvh = h.light_bvh;
    dl_baked_scene &sc = r->scene;
    sc = dl_baked_scene{};
    sc.settings.bounce = h.bounce_in_scene;
    sc.settings.colored_bounce = h.bounce_in_scene && o.colored_bounce;
    sc.settings.dynamic_geometry = o.dynamic_geometry;
    sc.settings.pixel_density = o.pixel_density;
    sc.settings.max_lightmap_size = o.max_lightmap_size;
    sc.settings.distance_cube_resolution = 64;
    sc.light_count = r->lights.size();
    sc.lights = r->lights.data();
    sc.light_bvh_count = r->bvh.size();
    sc.light_bvh = r->bvh.data();
    sc.mesh_count = r->meshes.size();
    sc.meshes = r->meshes.data();
    // maps for moving meshes
    if (s.cube_word_count && download) {
        r->cubes.resize(s.cube_word_count);
        CK(cudaMemcpy(r->cubes.data(), s.cube_words, s.cube_word_count * 4, cudaMemcpyDeviceToHost));
    }
    std::vector<const uint32_t *> sun_dev;
    for (size_t i = 0; i < s.sun_setups.size(); ++i) {
        const SunMapSetup &m = s.sun_setups[i];
        dl_sun_map d{};
        std::vector<uint32_t> texels;
        const uint32_t *dev = nullptr;
        if (m.empty) {
            texels.assign(1, 0xFFFFFFFFu);  // pack_sun_depth(1, 1)
            d.resolution = 1;
        } else {
            d.resolution = m.resolution;
            for (int k = 0; k < 12; ++k) d.rows[k] = m.rows[k];
            d.word_count = ((uint64_t)m.resolution * m.resolution + 1) / 2;
            if (download) {
                texels.resize(d.word_count);
                CK(cudaMemcpy(texels.data(), s.sun_texels[i], texels.size() * 4, cudaMemcpyDeviceToHost));
            } else {
                dev = s.sun_texels[i];
            }
        }
        r->sun_words.push_back(std::move(texels));
        r->sun_maps.push_back(d);
        sun_dev.push_back(dev);
    }
    for (size_t i = 0; i < r->sun_maps.size(); ++i) {
        if (sun_dev[i]) {
            r->sun_maps[i].texels = sun_dev[i];
        } else {
            r->sun_maps[i].word_count = r->sun_words[i].size();
            r->sun_maps[i].texels = r->sun_words[i].data();
        }
    }
    if (s.probe_grid.present) {
        const ProbeGridSetup &g = s.probe_grid;
        std::vector<float> open(g.count() * 6);
        std::vector<uint32_t> back(g.count() * 6);
        CK(cudaMemcpy(open.data(), s.probe_open, open.size() * 4, cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(back.data(), s.probe_back, back.size() * 4, cudaMemcpyDeviceToHost));
        r->probe_words = sky_probe_words(g, open.data(), back.data(), o.sky_samples);
        dl_sky_probes &p = r->probes;
        p.origin[0] = g.origin.x;
        p.origin[1] = g.origin.y;
        p.origin[2] = g.origin.z;
        p.spacing = g.spacing;
        for (int k = 0; k < 3; ++k) p.counts[k] = g.counts[k];
        p.word_count = r->probe_words.size();
        p.words = r->probe_words.data();
    }
    if (download) {
        for (const auto &w : r->sun_words) s.report.d2h_bytes += w.size() * 4;
        s.report.d2h_bytes += r->cubes.size() * 4 + (s.probe_grid.present ? s.probe_grid.count() * 6 * 8 : 0);
        sc.distance_cube_words = r->cubes.size();
        sc.distance_cubes = r->cubes.empty() ? nullptr : r->cubes.data();
    } else {
        sc.distance_cube_words = s.cube_word_count;
        sc.distance_cubes = s.cube_words;
    }
    sc.sun_map_count = r->sun_maps.size();
    sc.sun_maps = r->sun_maps.empty() ? nullptr : r->sun_maps.data();
    sc.sky_probes = s.probe_grid.present ? &r->probes : nullptr;
    sc.stats.meshes = (uint32_t)h.meshes.size();
    sc.stats.triangles = h.triangles;
    sc.stats.texels = s.texels;
    sc.stats.rays = s.counters.rays;
    sc.stats.lights_removed = s.counters.lights_removed;
    sc.stats.bounce_rays = s.counters.bounce_rays;
    sc.stats.triangle_words = s.out_words;
    return DL_OK;
}

// Collects the payload as host-written runs and device word arrays (payload order, word units).
struct DeviceSink {
    std::vector<uint32_t> host;         // host-written words, in order
    std::vector<PayloadSegment> segs;   // src of a host run: offset into `host` until uploaded
    std::vector<bool> from_host;
    unsigned long long at = 0;          // payload words so far
    const dl_session *session;          // whose device arrays `words` takes as they are
    void run(uint32_t v) {
        if (segs.empty() || !from_host.back() || segs.back().dst + segs.back().len != at) {
            segs.push_back(PayloadSegment{at, reinterpret_cast<const uint32_t *>(host.size()), 0});
            from_host.push_back(true);
        }
        host.push_back(v);
        ++segs.back().len;
        ++at;
    }
    void u32(uint32_t v) { run(v); }
    void u64(uint64_t v) {
        run((uint32_t)v);
        run((uint32_t)(v >> 32));
    }
    void f32(float f) {
        uint32_t v;
        std::memcpy(&v, &f, 4);
        run(v);
    }
    void words(const uint32_t *w, uint64_t n) {
        u64(n);
        if (!n) return;
        const dl_session &s = *session;
        bool device = w == s.cube_words || std::find(s.sun_texels.begin(), s.sun_texels.end(), w) != s.sun_texels.end();
        device |= s.words_dev && w >= s.words_dev && w < s.words_dev + s.out_words;
        if (!device) {
            for (uint64_t i = 0; i < n; ++i) run(w[i]);
            return;
        }
        segs.push_back(PayloadSegment{at, w, n});
        from_host.push_back(false);
        at += n;
    }
};

// The payload of the last run built on the device, its CRC-32 from per-chunk CRCs combined on the
// host; payload_read copies it out.
void payload_build(dl_session &s, HostResult &r, uint64_t &length, uint32_t &crc) {
    s.payload_dev = nullptr;
    DeviceSink sink;
    sink.session = &s;
    emit_payload(r.scene, sink);
    const unsigned long long words = sink.at;
    Pool &P = s.pool;
    cudaStream_t strm = s.stream;
    uint32_t *payload = P.get<uint32_t>("payload", words);
    uint32_t *host_dev = P.get<uint32_t>("payload_host", sink.host.size());
    CK(cudaMemcpyAsync(host_dev, sink.host.data(), sink.host.size() * 4, cudaMemcpyHostToDevice, strm));
    for (size_t i = 0; i < sink.segs.size(); ++i)
        if (sink.from_host[i]) sink.segs[i].src = host_dev + reinterpret_cast<uintptr_t>(sink.segs[i].src);
    PayloadSegment *segs = P.get<PayloadSegment>("payload_segs", sink.segs.size());
    CK(cudaMemcpyAsync(segs, sink.segs.data(), sink.segs.size() * sizeof(PayloadSegment), cudaMemcpyHostToDevice,
                       strm));
    k_payload_gather<<<dim3((unsigned)sink.segs.size(), grid_parts(sink.segs.size(), 256).y), 256, 0, strm>>>(segs,
                                                                                                            payload);
    LAUNCHED("k_payload_gather");
    // CRC of the full chunks on the device, of the rest on the host
    const unsigned long long chunks = words / kCrcChunkWords, done = chunks * kCrcChunkWords;
    std::vector<uint32_t> chunk_crc(chunks), rest(words - done);
    // shifts of the CRC register by 512 * 2^l bytes, and by a chunk
    struct Shifts {
        CrcShifts part;
        uint32_t chunk[32];
        Shifts() {
            for (int i = 0; i < 32; ++i) {
                for (int l = 0; l < 7; ++l) part.m[l][i] = crc32_shift(1u << i, 512ull << l);
                chunk[i] = crc32_shift(1u << i, (uint64_t)kCrcChunkWords * 4);
            }
        }
    };
    static const Shifts shifts;
    if (chunks) {
        uint32_t *tables = P.get<uint32_t>("crc_tables", 1024);
        CK(cudaMemcpyAsync(tables, crc32_tables(), 1024 * 4, cudaMemcpyHostToDevice, strm));
        uint32_t *out = P.get<uint32_t>("chunk_crc", chunks);
        unsigned blocks = (unsigned)std::min<unsigned long long>(chunks, (unsigned long long)s.sms * 16);
        k_crc_chunks<<<blocks, 128, 0, strm>>>(payload, chunks, tables, shifts.part, out);
        LAUNCHED("k_crc_chunks");
        CK(cudaMemcpyAsync(chunk_crc.data(), out, chunks * 4, cudaMemcpyDeviceToHost, strm));
    }
    if (!rest.empty())
        CK(cudaMemcpyAsync(rest.data(), payload + done, rest.size() * 4, cudaMemcpyDeviceToHost, strm));
    CK(cudaStreamSynchronize(strm));
    uint32_t c = 0xFFFFFFFFu;
    for (unsigned long long k = 0; k < chunks; ++k) {
        uint32_t shifted = 0;
        for (int i = 0; i < 32; ++i)
            if ((c >> i) & 1u) shifted ^= shifts.chunk[i];
        c = shifted ^ chunk_crc[k];
    }
    c = crc32_update(c, reinterpret_cast<const uint8_t *>(rest.data()), rest.size() * 4);
    crc = c ^ 0xFFFFFFFFu;
    length = words * 4;
    s.payload_dev = payload;
    s.payload_words = words;
}

// Copies the built payload into `dst` (pageable host memory, in general not touched before). The
// host's cores share it, each in pieces through its own pinned buffer: the SMs write a piece over
// the CPU-GPU link while the core copies the previous one on. Bound by the cores' page faults and
// copies (the link alone moves the level's 505 MB in 2.6 ms); one core behind the driver's staging copy, and a
// second copy into the caller's object, took 71 ms for them, this takes 12 to 14 ms, 2.5 ms for the rooms' 68 MB
// (was 12 ms), 0.7 ms for 20 MB. kPiece also sets how many cores take part; at 128 K, 512 K, 2 M words: 505 MB
// 12.0, 11.7, 12.0 ms, 68 MB 2.4, 2.4, 2.6 ms, 20 MB 1.2, 0.7, 1.1 ms.
void payload_read(dl_session &s, uint8_t *dst) {
    constexpr uint64_t kPiece = 512 * 1024;  // words
    const uint64_t words = s.payload_words;
    const uint64_t want = (words + 2 * kPiece - 1) / (2 * kPiece);
    const unsigned hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    const unsigned n = (unsigned)std::min<uint64_t>(hw, std::max<uint64_t>(1, want));
    while (s.readers.size() < n) {
        cudaStream_t r;
        CK(cudaStreamCreateWithFlags(&r, cudaStreamNonBlocking));
        s.readers.push_back(r);
    }
    std::vector<cudaError_t> failed(n, cudaSuccess);
    auto part = [&](unsigned t) noexcept {
        const uint64_t piece = std::min(kPiece, std::max<uint64_t>(words, 1));
        cudaError_t e = cudaSetDevice(s.device);
        WordCache::Buffer b{0, nullptr, false};
        try {
            b = word_cache().take(2 * piece);
        } catch (...) {
            failed[t] = cudaErrorMemoryAllocation;
            return;
        }
        uint32_t *mapped = nullptr;
        if (e == cudaSuccess && b.pinned && cudaHostGetDevicePointer((void **)&mapped, b.p, 0) != cudaSuccess) {
            cudaGetLastError();
            mapped = nullptr;
        }
        const uint64_t first = words * t / n, last = words * (t + 1) / n;
        uint64_t pending = 0, pending_at = 0;
        unsigned half = 0;
        for (uint64_t at = first; e == cudaSuccess && at < last; at += piece, half ^= 1) {
            const uint64_t len = std::min(piece, last - at);
            uint32_t *to = b.p + half * piece;
            if (mapped) {
                k_copy_words<<<16, 256, 0, s.readers[t]>>>(s.payload_dev + at, mapped + half * piece, len);
                e = cudaGetLastError();
            } else {
                e = cudaMemcpyAsync(to, s.payload_dev + at, len * 4, cudaMemcpyDeviceToHost, s.readers[t]);
            }
            if (pending) std::memcpy(dst + pending_at * 4, b.p + (half ^ 1) * piece, pending * 4);
            const cudaError_t w = cudaStreamSynchronize(s.readers[t]);
            if (e == cudaSuccess) e = w;
            pending = len;
            pending_at = at;
        }
        if (e == cudaSuccess && pending) std::memcpy(dst + pending_at * 4, b.p + (half ^ 1) * piece, pending * 4);
        try {
            word_cache().give(b);
        } catch (...) {
            WordCache::release(b);
        }
        failed[t] = e;
    };
    std::vector<std::thread> threads;
    unsigned started = 1;
    try {
        for (; started < n; ++started) threads.emplace_back(part, started);
    } catch (...) {  // no thread to be had: this one takes the parts left
    }
    part(0);
    for (unsigned t = started; t < n; ++t) part(t);
    for (auto &t : threads) t.join();
    for (cudaError_t e : failed)
        if (e != cudaSuccess) throw CudaError{e, "payload read"};
}

// The occluder BVH's nodes with their boxes as planes, for dl_session_occluder_bvh. The device
// holds centres and half extents, from which the planes do not follow exactly; they are minima and
// maxima over the triangles below (padded), so they are taken again from the resident triangles,
// children before parents (a node's index is below its children's). `dev`: the device's nodes.
std::vector<BvhNode> plane_nodes(dl_session &s, const std::vector<TravNode> &dev) {
    const DevScene &sc = s.sc;
    const HostScene &h = s.host;
    const uint32_t count = h.bvh_node_count, M = sc.mesh_count;
    std::vector<float> tris((size_t)sc.occluders * 12);
    std::vector<uint32_t> vbase(M + 1), ibase(M + 1);
    CK(cudaMemcpy(tris.data(), sc.tris, tris.size() * 4, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(vbase.data(), sc.mesh_vertex_base, (M + 1) * 4ull, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(ibase.data(), sc.mesh_index_base, (M + 1) * 4ull, cudaMemcpyDeviceToHost));
    std::vector<float> pos((size_t)vbase[M] * 3);
    std::vector<uint32_t> idx(ibase[M]);
    CK(cudaMemcpy(pos.data(), sc.positions, pos.size() * 4, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(idx.data(), sc.indices, idx.size() * 4, cudaMemcpyDeviceToHost));
    struct Box {
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        void add(const float *l, const float *u) {
            for (int a = 0; a < 3; ++a) {
                lo[a] = bvh_min(lo[a], l[a]);
                hi[a] = bvh_max(hi[a], u[a]);
            }
        }
    };
    std::vector<Box> all(count);  // each node's children together
    std::vector<BvhNode> out(count);
    for (uint32_t i = count; i-- > 0;) {
        Box b[2];
        for (int c = 0; c < 2; ++c) {
            const int32_t ref = dev[i].ref[c];
            if (ref >= 0) {
                b[c] = all[ref];
            } else {
                const uint32_t packed = (uint32_t)~ref;
                for (uint32_t k = packed >> 3; k < (packed >> 3) + (packed & 7u); ++k) {
                    uint32_t occ;
                    std::memcpy(&occ, &tris[(size_t)k * 12 + 3], 4);
                    const uint32_t m = h.occ_mesh[occ], *v = &idx[ibase[m] + (size_t)h.occ_tri[occ] * 3];
                    for (int j = 0; j < 3; ++j) {
                        const float *p = &pos[(size_t)(vbase[m] + v[j]) * 3];
                        b[c].add(p, p);
                    }
                }
            }
            all[i].add(b[c].lo, b[c].hi);
            if (ref == ~0) {
                for (int a = 0; a < 3; ++a) {
                    b[c].lo[a] = 1e30f;
                    b[c].hi[a] = -1e30f;
                }
            } else {
                bvh_pad_box(b[c].lo, b[c].hi);
            }
        }
        BvhNode &n = out[i];
        n = BvhNode{};
        for (int a = 0; a < 2; ++a) {
            n.c0[2 * a] = b[0].lo[a];
            n.c0[2 * a + 1] = b[0].hi[a];
            n.c1[2 * a] = b[1].lo[a];
            n.c1[2 * a + 1] = b[1].hi[a];
            n.c2[2 * a] = b[a].lo[2];
            n.c2[2 * a + 1] = b[a].hi[2];
            n.ref[a] = dev[i].ref[a];
        }
    }
    return out;
}

dl_status result(dl_session &s, dl_baked_scene *&out) {
    std::unique_ptr<HostResult> r;
    dl_status st = assemble(s, r, true);
    if (st != DL_OK) return st;
    out = &r.release()->scene;
    return DL_OK;
}

}  // namespace
}  // namespace dl

// ================================ C ABI ====================================================

#define DL_GUARD(body)                                                                \
    try {                                                                             \
        body                                                                          \
    } catch (const CudaError &e) {                                                    \
        g_error = std::string(e.what) + ": " + cudaGetErrorString(e.code);            \
        return e.code == cudaErrorMemoryAllocation ? DL_OUT_OF_MEMORY : DL_CUDA_ERROR; \
    } catch (const std::bad_alloc &) {                                                \
        g_error = "host allocation failed";                                           \
        return DL_OUT_OF_MEMORY;                                                      \
    } catch (...) {                                                                   \
        g_error = "unexpected failure";                                               \
        return DL_CUDA_ERROR;                                                         \
    }

// dl_session_create with an optional progress whose cancel flag create() checks.
static dl_status session_create(const dl_bake_input *input, const dl_bake_options *options,
                                const dl_bake_config *config, const dl_progress *progress, dl_session **out) {
    if (!input || !options || !out) {
        g_error = "null argument";
        return DL_INVALID_ARGUMENT;
    }
    *out = nullptr;
    DL_GUARD({
        dl_session *s = nullptr;
        auto t0 = std::chrono::steady_clock::now();
        dl_status st = create(input, options, config, s, progress);
        if (st != DL_OK) return st;
        s->report.ms_upload = ms_since(t0);
        *out = s;
        return DL_OK;
    })
}

extern "C" {

uint32_t dl_abi_version(void) { return DL_ABI_VERSION; }

const char *dl_status_string(dl_status status) {
    switch (status) {
        case DL_OK: return "ok";
        case DL_CANCELLED: return "cancelled";
        case DL_DUPLICATE_ID: return "duplicate id";
        case DL_INVALID_MESH: return "invalid mesh";
        case DL_INVALID_LIGHT: return "invalid light";
        case DL_INVALID_OPTIONS: return "invalid options";
        case DL_CUDA_ERROR: return "cuda error";
        case DL_OUT_OF_MEMORY: return "out of memory";
        case DL_QUEUE_TIMEOUT: return "queue timeout";
        case DL_BUSY: return "busy";
        case DL_UNSUPPORTED: return "unsupported";
        case DL_INVALID_ARGUMENT: return "invalid argument";
    }
    return "unknown";
}

const char *dl_last_error(void) { return g_error.c_str(); }

void dl_default_options(dl_bake_options *o) {
    if (!o) return;
    *o = dl_bake_options{};
    o->pixel_density = 128.0f;
    o->max_lightmap_size = 2048;
    o->bounce_compression = 8;
    o->dynamic_geometry = DL_GEOMETRY_ANGULAR;
    o->skip_bounce = 0;
    o->photon_cube_resolution = 512;
    o->area_light_samples = 64;
    o->area_light_min_samples = 16;
    o->sun_map_resolution = 2048;
    o->sky_samples = 64;
    o->sky_probe_spacing = 1.0f;
    o->colored_bounce = 0;
    o->seed = 0;
}

dl_status dl_session_create(const dl_bake_input *input, const dl_bake_options *options,
                            const dl_bake_config *config, dl_session **out) {
    return session_create(input, options, config, nullptr, out);
}

dl_status dl_session_run(dl_session *s, dl_progress *progress) {
    if (!s) {
        g_error = "null session";
        return DL_INVALID_ARGUMENT;
    }
    DL_GUARD({
        CK(cudaSetDevice(s->device));
        return run(*s, progress);
    })
}

dl_status dl_session_result(dl_session *s, dl_baked_scene **out) {
    if (!s || !out) {
        g_error = "null argument";
        return DL_INVALID_ARGUMENT;
    }
    *out = nullptr;
    DL_GUARD({
        CK(cudaSetDevice(s->device));
        auto t0 = std::chrono::steady_clock::now();
        dl_status st = result(*s, *out);
        s->report.ms_download = ms_since(t0);
        return st;
    })
}

dl_status dl_session_bounce_map(dl_session *s, uint64_t mesh_id, uint32_t slot, uint32_t rect[4], float *rgb,
                                uint32_t cap, uint32_t *texels) {
    if (!s || !rect || !texels || (cap && !rgb)) {
        g_error = "null argument";
        return DL_INVALID_ARGUMENT;
    }
    *texels = 0;
    if (!s->have_result) {
        g_error = "no finished run in this session";
        return DL_INVALID_ARGUMENT;
    }
    const HostScene &h = s->host;
    uint32_t m = 0;
    while (m < h.meshes.size() && h.meshes[m]->id != mesh_id) ++m;
    if (m == h.meshes.size() || slot >= h.lights.size()) {
        g_error = "no such mesh id or light slot";
        return DL_INVALID_ARGUMENT;
    }
    if (!s->bounce_map || !(h.lights[slot].flags & kLightBounce)) return DL_OK;
    DL_GUARD({
        CK(cudaSetDevice(s->device));
        size_t e = (size_t)m * h.lights.size() + slot;
        uint32_t r[4];
        uint32_t off[2];
        CK(cudaMemcpy(r, s->region_rect + e * 4, sizeof r, cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(off, s->bounce_woff + e, sizeof off, cudaMemcpyDeviceToHost));
        if (r[0] == kNoRect) return DL_OK;
        Rect w = bounce_window(r, h.resolution[m]);
        rect[0] = w.min_x;
        rect[1] = w.min_y;
        rect[2] = w.max_x;
        rect[3] = w.max_y;
        uint32_t n = off[1] - off[0];
        *texels = n;
        if (cap) {
            std::vector<float4> v(std::min(n, cap));
            CK(cudaMemcpy(v.data(), s->bounce_map + off[0], v.size() * sizeof(float4), cudaMemcpyDeviceToHost));
            for (size_t k = 0; k < v.size(); ++k) {
                rgb[k * 3] = v[k].x;
                rgb[k * 3 + 1] = v[k].y;
                rgb[k * 3 + 2] = v[k].z;
            }
        }
        return DL_OK;
    })
}

dl_status dl_session_occluder_bvh(dl_session *s, void *nodes, uint64_t node_cap, float *triangles,
                                  uint64_t tri_cap, uint32_t *node_count, uint32_t *depth) {
    if (!s || !node_count || !depth || (node_cap && !nodes) || (tri_cap && !triangles)) {
        g_error = "null argument";
        return DL_INVALID_ARGUMENT;
    }
    const HostScene &h = s->host;
    *node_count = h.bvh_node_count;
    *depth = h.bvh_depth;
    DL_GUARD({
        CK(cudaSetDevice(s->device));
        uint64_t n = std::min<uint64_t>(node_cap, h.bvh_node_count);
        if (n) {
            // the boxes come from the host; the device's nodes have to be the ones that they make
            std::vector<TravNode> dev(h.bvh_node_count);
            CK(cudaMemcpy(dev.data(), s->sc.nodes, dev.size() * sizeof(TravNode), cudaMemcpyDeviceToHost));
            const std::vector<BvhNode> boxes = h.nodes.empty() ? plane_nodes(*s, dev) : h.nodes;
            const size_t bad = first_unlike(boxes.data(), dev.data(), dev.size());
            if (bad < dev.size()) {
                g_error = "occluder BVH node " + std::to_string(bad) + " of the device does not hold its triangles' boxes";
                return DL_CUDA_ERROR;
            }
            std::memcpy(nodes, boxes.data(), n * sizeof(BvhNode));
        }
        uint64_t t = std::min<uint64_t>(tri_cap, s->sc.occluders);
        if (t) CK(cudaMemcpy(triangles, s->sc.tris, t * 3 * sizeof(float4), cudaMemcpyDeviceToHost));
        return DL_OK;
    })
}

dl_status dl_session_payload_build(dl_session *s, uint64_t *length, uint32_t *crc) {
    if (!s || !length) {
        g_error = "null argument";
        return DL_INVALID_ARGUMENT;
    }
    *length = 0;
    DL_GUARD({
        CK(cudaSetDevice(s->device));
        std::unique_ptr<HostResult> r;
        dl_status st = assemble(*s, r, false);
        if (st != DL_OK) return st;
        uint32_t c = 0;
        payload_build(*s, *r, *length, c);
        if (crc) *crc = c;
        return DL_OK;
    })
}

dl_status dl_session_payload_read(dl_session *s, uint8_t *bytes, uint64_t length) {
    if (!s || !bytes) {
        g_error = "null argument";
        return DL_INVALID_ARGUMENT;
    }
    if (!s->payload_dev || length != s->payload_words * 4) {
        g_error = "no built payload of this length in this session";
        return DL_INVALID_ARGUMENT;
    }
    DL_GUARD({
        CK(cudaSetDevice(s->device));
        payload_read(*s, bytes);
        return DL_OK;
    })
}

dl_status dl_session_encode_payload(dl_session *s, uint8_t **bytes, uint64_t *length, uint32_t *crc) {
    if (!s || !bytes || !length) {
        g_error = "null argument";
        return DL_INVALID_ARGUMENT;
    }
    *bytes = nullptr;
    *length = 0;
    uint64_t n = 0;
    uint32_t c = 0;
    dl_status st = dl_session_payload_build(s, &n, &c);
    if (st != DL_OK) return st;
    uint8_t *b = static_cast<uint8_t *>(std::malloc(n ? n : 1));
    if (!b) {
        g_error = "host allocation failed";
        return DL_OUT_OF_MEMORY;
    }
    st = dl_session_payload_read(s, b, n);
    if (st != DL_OK) {
        std::free(b);
        return st;
    }
    *bytes = b;
    *length = n;
    if (crc) *crc = c;
    return DL_OK;
}

dl_status dl_session_report(const dl_session *s, dl_bake_report *report) {
    if (!s || !report) {
        g_error = "null argument";
        return DL_INVALID_ARGUMENT;
    }
    *report = s->report;
    return DL_OK;
}

void dl_session_destroy(dl_session *s) { delete s; }

void dl_release_memory(void) {
    word_cache().clear();
    release_pooled_device_memory();
}

void dl_baked_scene_free(dl_baked_scene *scene) { delete reinterpret_cast<HostResult *>(scene); }

dl_status dl_bake_ex(const dl_bake_input *input, const dl_bake_options *options, const dl_bake_config *config,
                     dl_progress *progress, dl_baked_scene **out, dl_bake_report *report) {
    if (!input || !options || !out) {
        g_error = "null argument";
        return DL_INVALID_ARGUMENT;
    }
    *out = nullptr;
    std::unique_lock<std::mutex> lock(g_busy, std::try_to_lock);
    if (!lock.owns_lock()) {
        g_error = "another bake is running in this process";
        return DL_BUSY;
    }
    auto t0 = std::chrono::steady_clock::now();
    if (progress) progress->stage = 0;
    dl_session *s = nullptr;
    dl_status st = session_create(input, options, config, progress, &s);
    if (st != DL_OK) return st;
    std::unique_ptr<dl_session> owner(s);
    st = dl_session_run(s, progress);
    if (st == DL_CANCELLED) {
        g_error = "the bake was cancelled";
        if (report) {
            *report = s->report;
            report->ms_total = ms_since(t0);
        }
    }
    if (st != DL_OK) return st;
    st = dl_session_result(s, out);
    if (report) {
        *report = s->report;
        report->ms_total = ms_since(t0);
    }
    return st;
}

dl_status dl_bake(const dl_bake_input *input, const dl_bake_options *options, dl_progress *progress,
                  dl_baked_scene **out) {
    dl_bake_config cfg{};
    return dl_bake_ex(input, options, &cfg, progress, out, nullptr);
}

dl_status dl_encode_payload(const dl_baked_scene *scene, uint8_t **bytes, uint64_t *length, uint32_t *crc) {
    if (!scene || !bytes || !length) {
        g_error = "null argument";
        return DL_INVALID_ARGUMENT;
    }
    try {
        std::vector<uint8_t> p = encode_payload(*scene);
        uint8_t *b = static_cast<uint8_t *>(std::malloc(p.size() ? p.size() : 1));
        if (!b) {
            g_error = "host allocation failed";
            return DL_OUT_OF_MEMORY;
        }
        if (!p.empty()) std::memcpy(b, p.data(), p.size());
        *bytes = b;
        *length = p.size();
        if (crc) *crc = crc32_ieee(p.data(), p.size());
        return DL_OK;
    } catch (...) {
        g_error = "host allocation failed";
        return DL_OUT_OF_MEMORY;
    }
}

void dl_free(void *p) { std::free(p); }

}  // extern "C"

// ================================ non-allocating bounce filter ============================
//
// dl_filter_bounce_window_noalloc: the bounce map filter of the bake (dilate, then the 7-tap
// separable blur; the body of k_bounce_filter) on one window held in caller-owned device
// buffers, for callers that cannot allocate device memory — an engine applying the filter from
// inside its own fixed memory budget, or from code that must not call cudaMalloc (while a
// stream is being captured, or on a frame thread). One launch, intermediates in shared memory.

namespace dl {

constexpr uint32_t kNoallocMaxTexels = DL_NOALLOC_MAX_TEXELS;

namespace {

constexpr int kNoallocDevices = 64;  // devices beyond are refused, as they always were

// A block filters a tile of the window (filter_tile).
__global__ void __launch_bounds__(kTileThreads) k_noalloc_filter(const float *in, float *out, int w, int h, int4 clamp,
                                                                 BlurWeights bw) {
    __shared__ FilterTile tile;
    filter_tile(tile, blockIdx.x * kTileW, blockIdx.y * kTileH, w, h, clamp, bw,
                [&](int x, int y, float v[3]) {
                    const float *q = in + ((size_t)y * w + x) * 3;
                    for (int j = 0; j < 3; ++j) v[j] = q[j];
                },
                [&](int x, int y, int j, float v) { out[((size_t)y * w + x) * 3 + j] = v; });
}

// gaussian_weights(7, 5.0) (bounce_map.rs:140-151) in f32, exp rounded once from binary64.
BlurWeights blur_weights() {
    BlurWeights bw{};
    const float sigma2 = 5.0f * 5.0f;
    float sum = 0.0f;
    for (int i = -3; i <= 3; ++i) {
        float w = (1.0f / sqrtf(2.0f * kPiF * sigma2)) * (float)std::exp((double)(-(float)(i * i) / (2.0f * sigma2)));
        bw.w[i + 3] = w;
        sum += w;
    }
    for (int k = 0; k < 7; ++k) {
        bw.w[k] = bw.w[k] / sum;
        bw.sum += bw.w[k];
    }
    return bw;
}

}  // namespace
}  // namespace dl

extern "C" dl_status dl_filter_bounce_window_noalloc(const float *in_rgb, float *out_rgb, uint32_t width,
                                                     uint32_t height, uint32_t x0, uint32_t y0, uint32_t map_size,
                                                     void *stream) {
    using namespace dl;
    if (!in_rgb || !out_rgb) {
        g_error = "the input and output windows must be device buffers";
        return DL_INVALID_ARGUMENT;
    }
    uint64_t n = (uint64_t)width * height;
    if (width == 0 || height == 0 || n > kNoallocMaxTexels) {
        g_error = "window of " + std::to_string(width) + " x " + std::to_string(height) +
                  " texels: the non-allocating filter takes 1 to " + std::to_string(kNoallocMaxTexels) + " texels";
        return DL_INVALID_ARGUMENT;
    }
    {
        // the output is written while the input is still read: the two byte ranges must not meet
        const uintptr_t a = reinterpret_cast<uintptr_t>(in_rgb), b = reinterpret_cast<uintptr_t>(out_rgb);
        const uintptr_t bytes = (uintptr_t)(n * 3 * sizeof(float));
        if (a < b + bytes && b < a + bytes) {
            g_error = "the input and output windows overlap; they must be distinct device buffers";
            return DL_INVALID_ARGUMENT;
        }
    }
    if ((uint64_t)x0 + width > map_size || (uint64_t)y0 + height > map_size) {
        g_error = "the window does not lie inside the map";
        return DL_INVALID_ARGUMENT;
    }
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) {
        g_error = std::string("cudaGetDevice: ") + cudaGetErrorString(e);
        return DL_CUDA_ERROR;
    }
    if (device < 0 || device >= kNoallocDevices) {
        g_error = "the non-allocating filter runs on devices 0 to " + std::to_string(kNoallocDevices - 1) +
                  ", the current device is " + std::to_string(device);
        return DL_UNSUPPORTED;
    }
    static const BlurWeights bw = blur_weights();
    // the map's first and last column and row in window coordinates, as far as a tap can reach
    const int far = (int)kNoallocMaxTexels + 64;
    const int4 clamp = make_int4(-(int)std::min<uint32_t>(x0, 64), (int)std::min<uint32_t>(map_size - 1 - x0, far),
                                 -(int)std::min<uint32_t>(y0, 64), (int)std::min<uint32_t>(map_size - 1 - y0, far));
    const dim3 tiles((width + kTileW - 1) / kTileW, (height + kTileH - 1) / kTileH);
    k_noalloc_filter<<<tiles, kTileThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        in_rgb, out_rgb, (int)width, (int)height, clamp, bw);
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        g_error = std::string("bounce filter launch: ") + cudaGetErrorString(e);
        return DL_CUDA_ERROR;
    }
    return DL_OK;
}

// ================================ cache read bandwidth =================================
// No counterpart in the reference. The roofline of the traversal kernels: their node and
// triangle reads come from the L1 and L2 caches (the scene's BVH fits in L2), so their bound is
// the read bandwidth of those caches, which this measures with a plain streaming read.

namespace dl {
namespace {

// Each thread reads four float4 per iteration (independent loads in flight). Level 2: the
// blocks stream the whole buffer with L1-bypassing loads (ld.global.cg), `passes` times, so
// every byte comes from L2 (for a buffer that fits in it). Level 1: each block re-reads its own `slice` float4s with cached
// loads (ld.global.nc), so after the first pass every byte comes from its SM's L1.
__global__ void __launch_bounds__(256) k_probe_read(const float4 *__restrict__ buf, uint64_t n4, uint32_t passes,
                                                    uint32_t level, uint64_t slice, float *sink) {
    float acc = 0.0f;
    const float4 *base = buf;
    uint64_t count = n4, first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride =
        (uint64_t)gridDim.x * blockDim.x;
    if (level == 1) {
        base = buf + ((uint64_t)blockIdx.x * slice) % (n4 - slice + 1);
        count = slice;
        first = threadIdx.x;
        stride = blockDim.x;
    }
    for (uint32_t p = 0; p < passes; ++p) {
        uint64_t i = first;
        for (; i + 3 * stride < count; i += 4 * stride) {
            float4 a, b, c, d;
            if (level == 1) {
                a = __ldg(base + i);
                b = __ldg(base + i + stride);
                c = __ldg(base + i + 2 * stride);
                d = __ldg(base + i + 3 * stride);
            } else {
                a = __ldcg(base + i);
                b = __ldcg(base + i + stride);
                c = __ldcg(base + i + 2 * stride);
                d = __ldcg(base + i + 3 * stride);
            }
            acc += (a.x + b.y) + (c.z + d.w);
        }
        for (; i < count; i += stride) {
            float4 a = level == 1 ? __ldg(base + i) : __ldcg(base + i);
            acc += a.x;
        }
    }
    if (acc == -1.0f) sink[0] = acc;  // never true for the zero buffer; keeps the loads
}

}  // namespace
}  // namespace dl

extern "C" dl_status dl_probe_read_bandwidth(int device, uint32_t level, uint64_t bytes, uint32_t passes,
                                             double *gbs) {
    using namespace dl;
    if (!gbs || (level != 1 && level != 2) || passes == 0 || bytes < (1u << 20) || bytes > (1ull << 32)) {
        g_error = "dl_probe_read_bandwidth: level 1 or 2, 1 MiB to 4 GiB and at least one pass";
        return DL_INVALID_ARGUMENT;
    }
    *gbs = 0.0;
    int previous = 0;
    cudaError_t e = cudaGetDevice(&previous);
    if (e == cudaSuccess) e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        g_error = std::string("dl_probe_read_bandwidth: cudaSetDevice: ") + cudaGetErrorString(e);
        return DL_CUDA_ERROR;
    }
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    float4 *buf = nullptr;
    float *sink = nullptr;
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    dl_status st = DL_OK;
    const uint64_t n4 = bytes / sizeof(float4);
    const uint64_t slice = 32 * 1024 / sizeof(float4);  // level 1: 32 KiB per block, 4 blocks per SM
    const unsigned blocks = (unsigned)std::max(1, sms) * 4;
    double best = 0.0;
    e = cudaMalloc(&buf, n4 * sizeof(float4));
    if (e == cudaSuccess) e = cudaMalloc(&sink, sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(buf, 0, n4 * sizeof(float4));
    if (e == cudaSuccess) e = cudaEventCreate(&t0);
    if (e == cudaSuccess) e = cudaEventCreate(&t1);
    for (int rep = 0; e == cudaSuccess && rep < 6; ++rep) {
        // the first run is a warm-up: it brings the buffer into L2 (and the slices into L1)
        cudaEventRecord(t0, 0);
        k_probe_read<<<blocks, 256>>>(buf, n4, passes, level, slice, sink);
        cudaEventRecord(t1, 0);
        e = cudaEventSynchronize(t1);
        if (e != cudaSuccess) break;
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, t0, t1);
        const double read = level == 1 ? (double)blocks * slice * sizeof(float4) * passes
                                       : (double)n4 * sizeof(float4) * passes;
        if (rep > 0 && ms > 0.0f) best = std::max(best, read / (ms * 1e-3) / 1e9);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) {
        g_error = std::string("dl_probe_read_bandwidth: ") + cudaGetErrorString(e);
        st = e == cudaErrorMemoryAllocation ? DL_OUT_OF_MEMORY : DL_CUDA_ERROR;
    }
    if (t0) cudaEventDestroy(t0);
    if (t1) cudaEventDestroy(t1);
    if (buf) cudaFree(buf);
    if (sink) cudaFree(sink);
    cudaSetDevice(previous);
    *gbs = best;
    return st;
}
