// Shape of a batched multigrid launch (host).
#pragma once

#include <algorithm>
#include <functional>
#include <queue>
#include <vector>

namespace cicy {

constexpr int kMgBatchShapes = 3;
constexpr int kMgBatchCtas[kMgBatchShapes] = {16, 8, 4};  // CTAs per cluster

// Which of kMgBatchCtas the batch's clusters take; rows: of each system, resident: clusters of each shape
// that fit at once (7, 15 and 33 on a B200).  -1 when none fits.
//
// Large clusters solve a system sooner, small ones solve more systems at once, so the number of systems
// decides: 16 CTAs while they fit in one round, 8 up to two rounds of those, else 4 (ms with 16 / 8 / 4
// CTAs, sides 2 - 3.5 um, 1.5 %: 6 systems 2.5 / 3.1 / 4.4, 16 4.0 / 3.3 / 4.8; sides 2 - 3 um: 24 systems
// 4.8 / 3.2 / 4.1, 48 9.5 / 5.5 / 4.2).  But a system much larger than the others ends the batch, and a small
// cluster takes up to 2.5 times as long over it (58,149 rows 7.3 / 10.5 / 17.4): a larger shape is taken when
// the launch, replayed with estimated solves (systems largest first, each to the next free cluster; about
// n / (n + 8,000) iterations of 2,000 + n / CTAs), ends 1.3 times sooner, which is what the estimate can
// tell apart.  So 20 systems of 2,344 rows with one of 58,149 take 16 CTAs (7.2 / 10.6 / 17.4), and so do
// the first 32 realisations of the Monte-Carlo sweep (up to 155,980 rows: 16.4 / 22.1 / 38.6; by their
// number alone 4).
inline int mg_batch_shape(std::vector<int> rows, const int (&resident)[kMgBatchShapes]) {
    const int count = (int)rows.size();
    int shape = count <= resident[0] ? 0 : count <= 2 * resident[1] ? 1 : 2;
    while (shape > 0 && resident[shape] < 1) shape--;
    while (shape + 1 < kMgBatchShapes && resident[shape] < 1) shape++;
    if (resident[shape] < 1) return -1;
    std::sort(rows.begin(), rows.end(), std::greater<int>());
    auto end_of = [&](int s) {
        std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
        for (int c = 0; c < std::min(resident[s], count); c++) free_at.push(0.0);
        double end = 0;
        for (double n : rows) {
            const double t = free_at.top() + n / (n + 8000.0) * (2000.0 + n / kMgBatchCtas[s]);
            free_at.pop();
            free_at.push(t);
            end = std::max(end, t);
        }
        return end;
    };
    double limit = end_of(shape) / 1.3;
    for (int s = shape - 1; s >= 0; s--) {
        if (resident[s] < 1) continue;
        const double end = end_of(s);
        if (end < limit) {
            shape = s;
            limit = end;
        }
    }
    return shape;
}

}  // namespace cicy
