// The slab test of dl_slab.hpp where its rounding matters most: rays aimed (in binary32) at points of a box's
// faces, edges and corners, also ones that graze it along a face or leave from a point of it, must be reported
// as entering the padded box, for boxes and origins of every scale the bake takes and finite and infinite
// ranges. Built and run by tests/test_slab_edges.py.
#include <cmath>
#include <cstdio>

#include "dl_bvh_rules.hpp"
#include "dl_slab.hpp"

using namespace dl;

static uint64_t state = 23;
static double rnd() {
    state = splitmix64(state);
    return (double)(state >> 11) / 9007199254740992.0;
}
static double span(double lo, double hi) { return lo + (hi - lo) * rnd(); }

int main() {
    const double scales[] = {1e-3, 1.0, 40.0, 600.0, 3e4, 1e7, 5e8};
    long aimed[4] = {0, 0, 0, 0}, missed = 0, grazing = 0, starting = 0;
    for (int it = 0; it < 3000000; ++it) {
        const double scale = scales[(int)(rnd() * 7)], size = scale * std::pow(10.0, span(-5.0, 0.0));
        float lo[3], hi[3], o[3], target[3];
        int bounds = 0;  // axes on which the target lies on one of the box's planes: 1 a face, 2 an edge, 3 a corner
        for (int a = 0; a < 3; ++a) {
            const double at = span(-scale, scale), w = rnd() < 0.2 ? 0.0 : size * rnd();
            lo[a] = (float)at;
            hi[a] = (float)(at + w);
            if (hi[a] < lo[a]) hi[a] = lo[a];
            const double u = rnd();
            target[a] = u < 0.35 ? lo[a] : u < 0.7 ? hi[a] : (float)(lo[a] + ((double)hi[a] - lo[a]) * rnd());
            if (target[a] < lo[a]) target[a] = lo[a];
            if (target[a] > hi[a]) target[a] = hi[a];
            bounds += target[a] == lo[a] || target[a] == hi[a];
        }
        for (int a = 0; a < 3; ++a) {
            const double u = rnd();
            o[a] = u < 0.25 ? target[a] : u < 0.4 ? (rnd() < 0.5 ? lo[a] : hi[a])
                   : u < 0.7 ? (float)(target[a] + span(-size, size)) : (float)span(-scale, scale);
        }
        const double dx = (double)target[0] - o[0], dy = (double)target[1] - o[1], dz = (double)target[2] - o[2];
        const double len = std::sqrt(dx * dx + dy * dy + dz * dz);
        f3 d{(float)(dx / len), (float)(dy / len), (float)(dz / len)};
        if (!(len > 0.0)) {  // from the point itself, in any direction
            d = normalize(f3{(float)span(-1, 1), (float)span(-1, 1), (float)span(-1, 1)});
            ++starting;
        }
        grazing += len > 0.0 && bounds && (d.x == 0.0f || d.y == 0.0f || d.z == 0.0f);
        bvh_pad_box(lo, hi);
        const TravNode n = trav_node(lo, hi, lo, hi, 1, 2);
        const float ranges[] = {INFINITY, (float)(len * 1.000001)};
        bool hit[2];
        float near[2];
        slab_pair(Pair{n.cxy[0], n.cxy[1]}, Pair{n.cxy[2], n.cxy[3]}, Pair{n.hxy[0], n.hxy[1]}, Pair{n.hxy[2], n.hxy[3]},
                  Pair{n.z[0], n.z[1]}, Pair{n.z[2], n.z[3]}, ray_slabs(f3{o[0], o[1], o[2]}, d), ranges[it & 1], hit[0],
                  hit[1], near[0], near[1]);
        ++aimed[bounds];
        if ((!hit[0] || !hit[1]) && missed++ < 5)
            std::printf("missed: o %.9g %.9g %.9g d %.9g %.9g %.9g len %.9g\n", o[0], o[1], o[2], d.x, d.y, d.z, len);
    }
    std::printf("inside %ld faces %ld edges %ld corners %ld grazing %ld starting %ld missed %ld\n", aimed[0], aimed[1], aimed[2],
                aimed[3], grazing, starting, missed);
    return missed != 0;
}
