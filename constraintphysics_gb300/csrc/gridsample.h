// gridsample.h — which boxes size the pair grid's cells (pairs.cuh): at most
// kGridSamples of the boxes that go into it, evenly spaced from the first on.
// (A sample that misses them gives no cells, and every box is then tested against
// all later ones: a world of 2,300 bodies behind 130 worlds of 40, pair stage 195
// us from the batch's first 5,120 bodies, 71 from the large world's own.)
#pragma once
#include <vector>

namespace cpgpu {

constexpr int kGridSamples = 4096;
constexpr int grid_sample_step(int n) { return n > kGridSamples ? (n + kGridSamples - 1) / kGridSamples : 1; }
// samples of n boxes: box k * step for every k below this
constexpr int grid_sample_count(int n) { return (n + grid_sample_step(n) - 1) / grid_sample_step(n); }

// The sampled bodies of a batch whose world w holds the bodies start[w] to
// start[w + 1]: worlds above `large` bodies go into the grid, their bodies count
inline std::vector<int> grid_samples(const std::vector<int>& start, int large) {
    long long total = 0;
    for (size_t w = 0; w + 1 < start.size(); w++)
        if (start[w + 1] - start[w] > large) total += start[w + 1] - start[w];
    const int step = grid_sample_step((int)total);
    std::vector<int> out;
    long long at = 0, next = 0;   // grid bodies before this world; the next one to sample
    for (size_t w = 0; w + 1 < start.size(); w++) {
        const int n = start[w + 1] - start[w];
        if (n <= large) continue;
        for (; next < at + n; next += step) out.push_back(start[w] + (int)(next - at));
        at += n;
    }
    return out;
}

}  // namespace cpgpu
