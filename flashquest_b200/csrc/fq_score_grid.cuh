// Grid of the streaming page-score kernel (fq_scores.cu).  Plain C++: tests/test_score_grid.py runs it on the host.
#pragma once
#include <stdint.h>

namespace fq {

// CTAs per SM that the kernel's launch bound guarantees for NR query heads a pass and CH 8-channel chunks a lane, and that the
// grid is laid out in.  Four heads of 128 channels keep 64 values of q per lane and take 168 registers: three CTAs of 128
// threads fit an SM.  All others fit four and more, and 64 KiB of loads in flight are enough.
// Measured with 32 / 8 heads of 128 channels, laid out in four CTAs -> in three: 4 x 8 rows of 2048 pages 11.7 -> 8.6 us, of 8192
// 31.5 -> 25.5; 8 x 8 rows 17.5 -> 15.3 and 59.1 -> 48.9; 16 x 8 rows 27.8 -> 27.3 and 93.0 -> 92.4.
constexpr int score_stream_ctas_per_sm(int NR, int CH) { return NR > 3 && CH > 1 ? 3 : 4; }

// CTAs per (batch, kv head) row: whole waves of `resident` CTAs, at least 64 pages each; 0: fewer than 64 pages per resident
// CTA, where the ring never fills and the short CTAs of the other kernel start sooner.
inline int score_stream_ctas(int rows, int P, int resident) {
    if ((int64_t)rows * P < (int64_t)resident * 64) return 0;
    int best = 1;
    double best_t = 1e30;
    for (int c = 1; c <= 64 && c * 64 <= P; ++c) {
        const double t = (double)((rows * (int64_t)c + resident - 1) / resident) / c * (1.0 + 0.004 * c);
        if (t < best_t) { best_t = t; best = c; }
    }
    return best;
}

}  // namespace fq
