// batch_shape.cuh -- how the multi-RHS kernels of the diagonal form (dia.cu)
// cut their work (plain C++, also for a host compiler).
#pragma once

#include <algorithm>
#include <cstdint>

namespace nm {

constexpr int kDiaBatchThreads = 128;
constexpr int kDiaBatchCols = 16;  // columns of a chunk, at most
constexpr int kDiaBatchRun = 192;  // rows of a run, at most

struct DiaBatchShape {
    int lg = 0;          // a row's columns of a chunk lie on 2^lg lanes
    int nchunk = 0;
    int chunk_cols = 0;
    int run = 0;         // rows of a CTA
    int64_t grid = 0;    // CTAs; the launch takes at most INT32_MAX
};

// k columns (vec of them to a lane) of nrows rows on `sms` SMs.
inline DiaBatchShape dia_batch_shape(int64_t nrows, int64_t k, int vec, int sms) {
    DiaBatchShape b;
    // lanes per row: 16 columns to a chunk, or 8 where that saves 8 % of the
    // lanes (k = 100: 52 against 56 lanes, but 1.2 times the time)
    const int64_t groups = (k + vec - 1) / vec;
    while ((int64_t(1) << b.lg) < groups && (vec << b.lg) < kDiaBatchCols) ++b.lg;
    auto slots = [&](int l) { return ((groups + (int64_t(1) << l) - 1) >> l) << l; };
    if ((int64_t(1) << b.lg) < groups && b.lg > 0 && 25 * slots(b.lg - 1) < 23 * slots(b.lg))
        --b.lg;
    const int64_t nchunk = slots(b.lg) >> b.lg;
    b.nchunk = static_cast<int>(nchunk);
    b.chunk_cols = static_cast<int>(vec * ((groups + nchunk - 1) / nchunk));
    const int64_t step = kDiaBatchThreads >> b.lg;
    // Shorter runs where there are too few rows to fill the GPU with them.
    const int64_t run = std::max<int64_t>(step, nrows * nchunk / (int64_t(sms) * 16));
    b.run = static_cast<int>((std::min<int64_t>(run, kDiaBatchRun) + step - 1) / step * step);
    b.grid = (nrows + b.run - 1) / b.run * nchunk;
    return b;
}

// The CSR kernels' cut of the same work (spmv.cu): lanes per row, column chunks
// per lane in one pass, and the lane-columns of all passes together.
struct CsrBatchShape {
    int tpr_log2 = 0;
    int ch = 1;
    int64_t slots = 0;
};

constexpr int kBatchChunks = 4;  // most column chunks per lane in one pass

inline CsrBatchShape csr_batch_shape(int64_t k, int vec) {
    CsrBatchShape c;
    const int64_t groups = (k + vec - 1) / vec;  // lane-columns needed for one pass
    while ((int64_t(1) << c.tpr_log2) < groups && c.tpr_log2 < 5) ++c.tpr_log2;
    const int64_t need = (groups + (int64_t(1) << c.tpr_log2) - 1) >> c.tpr_log2;
    // as many chunks as k needs, in the widths the kernels have (1, 2, 4)
    c.ch = need >= kBatchChunks ? 4 : (need >= 2 ? 2 : 1);
    const int64_t pass = int64_t(c.ch) << c.tpr_log2;
    c.slots = (groups + pass - 1) / pass * pass;
    return c;
}

// Whether the kernels of the diagonal form take a product of k columns.  They
// read a row's masks and values once for each 16 columns, the CSR kernels once
// for all columns of a pass; so where a pass of those is two or four chunks
// wide and leaves few of its lanes idle, they are the faster ones, unless
// nearly every row has an entry on each of a few diagonals (`full`), which
// leaves the masks nothing to ask, or there are no values to read
// (`constant`), or X and Y are twice L2 and more, where walking the rows in
// order saves the most.  Time of the CSR kernels over that of these at 30,000 and
// 300,000 rows: 9 diagonals, 5 of them in a row, k = 64 1.5 and 1.3, k = 100
// 0.99 and 1.2, k = 128 0.86 and 1.05, k = 127 0.56 and 0.72; 7 varying full
// diagonals, k = 100 1.1 and 1.3, k = 128 0.92 and 1.13, k = 127 0.81 and 0.96;
// 7 constant full diagonals, k = 127 0.98 and 1.2; 16 diagonals, 10 of them in
// a row, k = 100 0.75 and 0.83.
inline bool dia_batch_takes(int64_t nrows, int ndiag, bool full, bool constant, int64_t k, int vec,
                            const DiaBatchShape& b) {
    constexpr double kLarge = 2 * 126e6;  // bytes of X and Y
    const CsrBatchShape c = csr_batch_shape(k, vec);
    if (c.ch < 2 || 6 * (int64_t(b.nchunk) << b.lg) < 5 * c.slots) return true;
    if (full) return constant || (c.ch == 2 && ndiag <= 12);
    if (c.ch > 2) return false;
    return ndiag <= 3 || (ndiag <= 9 && vec == 2 && 16.0 * double(nrows) * double(k) > kLarge);
}

}  // namespace nm
