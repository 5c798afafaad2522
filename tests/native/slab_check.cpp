// The slab test of dl_slab.hpp against exact geometry: a ray aimed (in binary32) at a point of a box
// must be reported as entering the padded box built for it, for boxes and origins of every scale the
// bake takes, axis-parallel rays and rays with vanishing components, finite and infinite ranges; a
// box well behind the ray or beyond its range must not. Built and run by tests/test_slab.py.
#include <cmath>
#include <cstdio>

#include "dl_bvh_rules.hpp"
#include "dl_slab.hpp"

using namespace dl;

static uint64_t state = 11;
static double rnd() {
    state = splitmix64(state);
    return (double)(state >> 11) / 9007199254740992.0;
}
static double span(double lo, double hi) { return lo + (hi - lo) * rnd(); }

int main() {
    long missed = 0, entered = 0, far_hits = 0, far_cases = 0, uncovered = 0;
    const double scales[] = {1e-3, 1.0, 40.0, 600.0, 3e4, 1e7, 5e8};
    for (int it = 0; it < 2000000; ++it) {
        const double scale = scales[(int)(rnd() * 7)];
        float lo[2][3], hi[2][3], o[3], target[3];
        const double size = scale * std::pow(10.0, span(-5.0, 0.0));
        for (int c = 0; c < 2; ++c)
            for (int a = 0; a < 3; ++a) {
                const double at = span(-scale, scale), w = rnd() < 0.2 ? 0.0 : size * rnd();
                lo[c][a] = (float)at;
                hi[c][a] = (float)(at + w);
                if (hi[c][a] < lo[c][a]) hi[c][a] = lo[c][a];
            }
        const int c = it & 1;
        for (int a = 0; a < 3; ++a) {
            target[a] = (float)(lo[c][a] + ((double)hi[c][a] - lo[c][a]) * rnd());
            if (target[a] < lo[c][a]) target[a] = lo[c][a];
            if (target[a] > hi[c][a]) target[a] = hi[c][a];
            // origins beside the box, elsewhere in the scene, or level with the target on an axis
            const double u = rnd();
            o[a] = u < 0.25 ? target[a] : u < 0.5 ? (float)(target[a] + span(-size, size)) : (float)span(-scale, scale);
        }
        const double dx = (double)target[0] - o[0], dy = (double)target[1] - o[1], dz = (double)target[2] - o[2];
        const double len = std::sqrt(dx * dx + dy * dy + dz * dz);
        if (!(len > 0.0)) continue;
        f3 d{(float)(dx / len), (float)(dy / len), (float)(dz / len)};
        if (rnd() < 0.05) d.x = d.x == 0.0f ? (float)std::pow(10.0, span(-44.0, -21.0)) : d.x;
        for (int k = 0; k < 2; ++k) bvh_pad_box(lo[k], hi[k]);
        const TravNode n = trav_node(lo[0], hi[0], lo[1], hi[1], 1, 2);
        for (int k = 0; k < 2; ++k)
            for (int a = 0; a < 3; ++a) {
                const double ce = a < 2 ? n.cxy[2 * k + a] : n.z[k], h = a < 2 ? n.hxy[2 * k + a] : n.z[2 + k];
                if (ce - h > lo[k][a] || ce + h < hi[k][a]) ++uncovered;
            }
        const float range = rnd() < 0.5 ? INFINITY : (float)(len * 1.000001);
        auto slabs = [&](f3 dir, float tmax, bool hit[2]) {
            float near[2];
            slab_pair(Pair{n.cxy[0], n.cxy[1]}, Pair{n.cxy[2], n.cxy[3]}, Pair{n.hxy[0], n.hxy[1]},
                      Pair{n.hxy[2], n.hxy[3]}, Pair{n.z[0], n.z[1]}, Pair{n.z[2], n.z[3]},
                      ray_slabs(f3{o[0], o[1], o[2]}, dir), tmax, hit[0], hit[1], near[0], near[1]);
        };
        bool hit[2];
        slabs(d, range, hit);
        ++entered;
        if (!hit[c]) {
            if (missed++ < 5)
                std::printf("missed: o %.9g %.9g %.9g d %.9g %.9g %.9g len %.9g\n", o[0], o[1], o[2], d.x, d.y, d.z, len);
        }
        // pruning: the opposite ray and a range ending well before the box
        const double margin = 4.0 * size + 4e-5 * std::fmax(1.0, scale);
        if (len > 4.0 * margin) {
            ++far_cases;
            slabs(f3{-d.x, -d.y, -d.z}, INFINITY, hit);
            far_hits += hit[c];
            slabs(d, (float)(len - 2.0 * margin), hit);
            far_hits += hit[c];
        }
    }
    // an empty child (inverted box) is never entered
    const float lo[3] = {-1, -1, -1}, hi[3] = {1, 1, 1}, elo[3] = {1e30f, 1e30f, 1e30f}, ehi[3] = {-1e30f, -1e30f, -1e30f};
    const TravNode e = trav_node(lo, hi, elo, ehi, 1, ~0);
    long empty = 0;
    for (int it = 0; it < 1000; ++it) {
        const f3 d = normalize(f3{(float)span(-1, 1), (float)span(-1, 1), (float)span(-1, 1)});
        bool h0, h1;
        float n0, n1;
        slab_pair(Pair{e.cxy[0], e.cxy[1]}, Pair{e.cxy[2], e.cxy[3]}, Pair{e.hxy[0], e.hxy[1]},
                  Pair{e.hxy[2], e.hxy[3]}, Pair{e.z[0], e.z[1]}, Pair{e.z[2], e.z[3]},
                  ray_slabs(f3{0.1f, 0.2f, 0.3f}, d), INFINITY, h0, h1, n0, n1);
        empty += h1 || !h0;
    }
    std::printf("entered %ld missed %ld uncovered %ld far cases %ld far hits %ld empty %ld\n", entered, missed,
                uncovered, far_cases, far_hits, empty);
    return missed || uncovered || far_hits || empty ? 1 : 0;
}
