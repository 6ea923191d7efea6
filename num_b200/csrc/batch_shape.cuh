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
    // lanes per row: 16 columns to a chunk, or 8 where that leaves fewer
    // lanes idle in the last one
    const int64_t groups = (k + vec - 1) / vec;
    while ((int64_t(1) << b.lg) < groups && (vec << b.lg) < kDiaBatchCols) ++b.lg;
    auto slots = [&](int l) { return ((groups + (int64_t(1) << l) - 1) >> l) << l; };
    if ((int64_t(1) << b.lg) < groups && b.lg > 0 && slots(b.lg - 1) < slots(b.lg)) --b.lg;
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

}  // namespace nm
