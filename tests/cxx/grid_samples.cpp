// Prints, for body counts and world layouts around the sample's limits, what a
// grid's cells are sized from: count, first and last sample, largest gap
// (checked by tests/test_grid_samples.py).
#include <cstdio>

#include "gridsample.h"

int main() {
    for (int n : {1, 2, 4095, 4096, 4097, 5121, 8191, 8192, 8193, 10241, 12287, 15361, 16383, 65535, 65536}) {
        const int step = cpgpu::grid_sample_step(n), m = cpgpu::grid_sample_count(n);
        std::printf("%d %d %d %d\n", n, m, (m - 1) * step, step);
    }
    // 130 worlds of 40, one of 2,100, 3 of 40, one of 3,000: only the large ones count
    std::vector<int> start{0};
    for (int k = 0; k < 130; k++) start.push_back(start.back() + 40);
    start.push_back(start.back() + 2100);
    for (int k = 0; k < 3; k++) start.push_back(start.back() + 40);
    start.push_back(start.back() + 3000);
    for (int i : cpgpu::grid_samples(start, 2048)) std::printf("%d\n", i);
    return 0;
}
