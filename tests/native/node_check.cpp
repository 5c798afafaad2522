// The comparison of dl_session_occluder_bvh (first_unlike, dl_host.hpp): nodes that trav_node makes of the
// boxes pass, and a node with a box too large or too small by one step, swapped boxes, swapped axes or another
// reference is named. Built and run by tests/test_nodes.py.
#include <cmath>
#include <cstdio>
#include <vector>

#include "dl_host.hpp"

using namespace dl;

int main() {
    std::vector<BvhNode> boxes(5);
    for (size_t i = 0; i < boxes.size(); ++i) {
        BvhNode &b = boxes[i];
        b = BvhNode{};
        for (int k = 0; k < 4; ++k) {  // lo, hi pairs, no two alike
            b.c0[k] = (float)(i * 7 + k * k) * 0.37f + (k % 2 ? 1.5f : -2.0f);
            b.c1[k] = (float)(i * 5 + k * k) * 1.91f + (k % 2 ? 40.0f : 8.0f);
            b.c2[k] = (float)(i * 3 + k) * -0.11f + (k % 2 ? 600.0f : -3.0f);
        }
        b.ref[0] = (int32_t)i + 1;
        b.ref[1] = ~(int32_t)(i << 3 | 2);
    }
    boxes[4].c1[0] = boxes[4].c1[2] = boxes[4].c2[2] = 1e30f;  // an empty child
    boxes[4].c1[1] = boxes[4].c1[3] = boxes[4].c2[3] = -1e30f;
    boxes[4].ref[1] = ~0;
    std::vector<TravNode> held;
    for (const BvhNode &b : boxes) held.push_back(traversal_node(b));
    const size_t n = boxes.size();
    int wrong = first_unlike(boxes.data(), held.data(), n) != n;
    auto planted = [&](size_t at, auto change) {
        std::vector<TravNode> h = held;
        change(h[at]);
        if (first_unlike(boxes.data(), h.data(), n) != at) {
            ++wrong;
            std::printf("a change of node %zu passed\n", at);
        }
    };
    for (size_t at = 0; at < n; ++at) {
        for (int k = 0; k < 4; ++k) {
            planted(at, [&](TravNode &t) { t.hxy[k] = std::nextafter(t.hxy[k], INFINITY); });
            planted(at, [&](TravNode &t) { t.hxy[k] *= 2.0f; });
            planted(at, [&](TravNode &t) { t.cxy[k] = std::nextafter(t.cxy[k], -INFINITY); });
            planted(at, [&](TravNode &t) { t.z[k] = std::nextafter(t.z[k], INFINITY); });
        }
        planted(at, [&](TravNode &t) { std::swap(t.cxy[0], t.cxy[2]), std::swap(t.hxy[0], t.hxy[2]), std::swap(t.cxy[1], t.cxy[3]),
                                       std::swap(t.hxy[1], t.hxy[3]), std::swap(t.z[0], t.z[1]), std::swap(t.z[2], t.z[3]); });
        planted(at, [&](TravNode &t) { std::swap(t.hxy[0], t.hxy[1]); });
        planted(at, [&](TravNode &t) { std::swap(t.ref[0], t.ref[1]); });
        planted(at, [&](TravNode &t) { t.ref[1] ^= 1; });
    }
    // NaN for NaN, whatever its bits
    boxes[2].c2[1] = INFINITY;
    boxes[2].c2[0] = -INFINITY;
    held[2] = traversal_node(boxes[2]);
    wrong += !(held[2].z[0] != held[2].z[0]);
    held[2].z[0] = -held[2].z[0];
    wrong += first_unlike(boxes.data(), held.data(), n) != n;
    std::printf("wrong %d\n", wrong);
    return wrong != 0;
}
