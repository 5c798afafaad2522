// The table-driven sine and cosine that the baker runs (sincos_reduce, sincos_sum, pair_rounds_to): values equal
// to the binary64 path's, the share of arguments left to that path, and the worst relative error of the sums before
// rounding, which has to stay below the 2^-36 that the rounding test allows for. Arguments: random ones up to 16
// in four distributions; around every table step, half step and multiple of pi/2 up to 16; with a second
// argument, every binary32 of both signs from 2^-27 up to 16 instead (eight threads, a few minutes).
// Built and run by tests/test_sincos_table.py.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

#include "dl_math.cuh"

using namespace dl;

struct Totals {
    unsigned long long checked = 0, mismatches = 0, fallbacks = 0;
    double worst = 0.0;
    void add(float x, bool count_fallback) {
        ++checked;
        float s, c;
        sincos_f(x, s, c);
        double sd, cd;
        sincos_d((double)x, sd, cd);
        const float s64 = (float)sd, c64 = (float)cd, only = sin_f(x);
        if (std::memcmp(&s, &s64, 4) || std::memcmp(&c, &c64, 4) || std::memcmp(&only, &s64, 4)) ++mismatches;
        SinCosArg a;
        float t;
        if (!sincos_reduce(x, a)) {
            fallbacks += count_fallback;
            return;
        }
        const FF fs = sincos_sum(a.e.sh, a.e.sl, a.e.ch, a.e.cl, a), fc = sincos_sum(a.e.ch, a.e.cl, -a.e.sh, -a.e.sl, a);
        const bool taken = pair_rounds_to(fs, t) && pair_rounds_to(fc, t);
        fallbacks += count_fallback && !taken;
        for (int k = 0; k < 2; ++k) {
            const FF f = k ? fc : fs;
            const double want = k ? cd : sd, err = std::fabs(((double)f.h + (double)f.l - want) / want);
            if (want != 0.0 && err > worst) worst = err;
        }
    }
    void merge(const Totals &o) {
        checked += o.checked;
        mismatches += o.mismatches;
        fallbacks += o.fallbacks;
        worst = o.worst > worst ? o.worst : worst;
    }
};
static float from_bits(uint32_t b) {
    float f;
    std::memcpy(&f, &b, 4);
    return f;
}

int main(int argc, char **argv) {
    const unsigned long long n = argc > 1 ? strtoull(argv[1], nullptr, 10) : 1000000ull;
    Totals all, near;
    if (argc > 2) {
        const uint32_t lo = 100u << 23, hi = 131u << 23;  // 2^-27 .. 16
        std::vector<Totals> part(8);
        std::vector<std::thread> threads;
        for (uint32_t t = 0; t < 8; ++t)
            threads.emplace_back([&, t] {
                for (uint32_t b = lo + t; b < hi; b += 8) {
                    part[t].add(from_bits(b), true);
                    part[t].add(from_bits(b | 0x80000000u), true);
                }
            });
        for (auto &t : threads) t.join();
        for (const Totals &p : part) all.merge(p);
    } else {
        uint64_t state = 4242;
        for (unsigned long long i = 0; i < n; ++i) {
            state = splitmix64(state);
            const float u = (float)((state >> 40) * (1.0 / 16777216.0));
            switch (i % 4) {
                case 0: all.add(u * 6.2831855f, true); break;
                case 1: all.add(u * 3.1415927f - 0.78539819f, true); break;
                case 2: all.add(u * 31.999f - 15.9995f, true); break;
                default: all.add(from_bits((107u + (uint32_t)((state >> 20) % 24u)) << 23 |
                                           ((uint32_t)(state >> 41) & 0x7FFFFFu) | (uint32_t)(state & 1u) << 31), true);
            }
        }
        for (int half = -1303; half <= 1303; ++half) {  // half steps of pi/256 up to 16, 64 values on both sides
            if (!half) continue;
            uint32_t b;
            const float at = (float)(half * (3.14159265358979323846 / 256.0));
            std::memcpy(&b, &at, 4);
            for (int d = -64; d <= 64; ++d) near.add(from_bits(b + d), false);
        }
    }
    std::printf("checked %llu mismatches %llu fallbacks %llu worst 2^%.3f\n", all.checked + near.checked,
                all.mismatches + near.mismatches, all.fallbacks, std::log2(std::fmax(all.worst, near.worst)));
    return 0;
}
