// park_rows.cuh -- where the warp sums of cg_dia.cu's rows go (plain C++, also
// for a host compiler).
//
// A thread's Q rows are summed in groups of up to 8: row q of all threads is
// kDiaCgTilesPerRow tiles, and warp w's sums of a group end in the lanes that
// multi_warp_sum leaves them in, a row each.
#pragma once

namespace nm {

constexpr int kDiaCgGroup = 8;  // rows of a group
constexpr int kDiaCgMaxQ = 14;  // most rows of a thread
constexpr int kDiaCgTilesPerRow = 2;  // 512 threads in 256-row tiles
constexpr int kDiaCgMaxOwnTiles = kDiaCgMaxQ * kDiaCgTilesPerRow;  // of a CTA

// Sums formed together (multi_warp_sum's P) for rows in groups of N.
constexpr int park_width(int N) { return N <= 1 ? 1 : (N <= 2 ? 2 : (N <= 4 ? 4 : 8)); }

// The row (0..Q-1) whose sum `lane` holds after the group that starts at row
// q0, -1 when it holds none: lanes without a row of their own, and the places
// of rows that the last group does not have (11 rows: 8 and 3).
constexpr int park_row(int lane, int q0, int Q) {
    const int N = Q < kDiaCgGroup ? Q : kDiaCgGroup, P = park_width(N), lanes = 32 / P;
    const int q = lane / lanes;
    return lane % lanes == 0 && q < N && q0 + q < Q ? q0 + q : -1;
}

}  // namespace nm
