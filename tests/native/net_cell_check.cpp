// The cell formula of the device's sample tables (net_cell, dl_math.cuh) against the host's sorted orders
// (sky_sample_order, sample_cells) for every net of the tables, 16 to 4096 samples. Built and run by tests/test_net_cells.py.
#include <cstdio>

#include "dl_host.hpp"

int main() {
    int failures = 0, nets = 0;
    for (uint32_t m = 4; m <= 12; ++m, ++nets) {
        const uint32_t n = 1u << m, xb = (m + 1) / 2;
        const std::vector<uint16_t> order = dl::sky_sample_order(n);
        const dl::SampleCells cells = dl::sample_cells(n);
        for (uint32_t j = 0; j < n; ++j) {
            const dl::NetCell c = dl::net_cell(j, m);
            failures += c.rank >= n || (c.y << xb | c.x) >= n;
            if (failures) break;
            failures += order[c.rank] != j || cells.cells[c.rank] != (c.x | c.y << 8) || cells.samples[c.y << xb | c.x] != j;
        }
    }
    std::printf("nets %d failures %d\n", nets, failures);
    return failures != 0;
}
