// Experts' rows laid out as runs of whole 128-row tiles, in steps of more than 128 rows: room and slices of K (host code).
#pragma once
#include <algorithm>
#include <cstddef>

namespace fl {

// rows of the experts' runs: whole 128-row tiles per expert that any row picked
inline size_t run_capacity(size_t picks, size_t experts) { return 128 * (picks / 128 + std::min(picks, experts)); }

// Slices of K for the runs' plain GEMM: few experts of few rows leave most of the chip idle (340 rows, 8 experts, 2048 columns: 64 tiles of 128 x 256).
// An expert's rows are not known here; with its share of the picks and a tenth more, the slices whose waves are shortest, up to four of at least eight
// k blocks; a slice costs its way to memory and back, about a twentieth of a tile's time for 64 tiles.  Whole prompt, one slice -> this, us: experts of
// 2816, width 1024, 130 / 286 / 400 / 583 tokens 503 -> 477, 528 -> 499, 548 -> 528, 610 -> 589; of 5632, width 2048, 130 / 200 / 1000 tokens 734 -> 694,
// 753 -> 711, 1417 -> 1377 (four slices of 256 tiles, at 1531 tokens: 1973 -> 1995).
inline int runs_tiles_each(int picks, int groups) { return ((int)(1.1 * picks / groups) + 1 + 127) / 128; }
inline int runs_ksplit(int picks, int groups, int N, int K, int sms) {
    const int tiles = std::min(groups, picks) * runs_tiles_each(picks, groups) * ((N + 255) / 256), nk = (K + 63) / 64;
    int best = 1;
    double cost = 1e30;
    for (int ks = 1; ks <= 4 && (ks == 1 || nk / ks >= 8); ++ks) {
        const double t = (double)((tiles * ks + sms - 1) / sms) / ks + 0.05 / 64 * tiles * ks;
        if (t < cost) { cost = t; best = ks; }
    }
    while (best > 1 && (nk + best - 1) / best * (best - 1) >= nk) --best;         // none of them is empty
    return best;
}

// The most rows, slices included, of any step of 129 to R rows (one of fewer rows may be cut along K more often).  Steps whose picks fill the same
// whole tiles have the same room; where an expert's share ends at the same tile too, the same slices.  (Every step by itself, for every layer: 17 ms of host time in front of
// the first step of 16384 rows of 60 layers.)
inline size_t runs_most_rows(int top, int experts, int N, int K, int sms, size_t R) {
    size_t most = 0;
    for (size_t T = 129; T <= R;) {
        const int picks = (int)T * top;
        const size_t last = picks < experts ? T : std::min<size_t>(R, ((size_t)(picks / 128 + 1) * 128 - 1) / top);
        int ks = runs_ksplit(picks, experts, N, K, sms);
        if (runs_tiles_each(picks, experts) != runs_tiles_each((int)last * top, experts))
            for (size_t t = T + 1; t <= last; ++t) ks = std::max(ks, runs_ksplit((int)t * top, experts, N, K, sms));
        most = std::max(most, ks * run_capacity(picks, experts));
        T = last + 1;
    }
    return most;
}

}  // namespace fl
