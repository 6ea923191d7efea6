// cg_dia.cu -- plain CG of a matrix in diagonal form, on chip over all SMs.
//
// Same algorithm, stopping rule and iterates as cg_solve_local
// (src/cg_solver.hpp:133-196).  One cooperative launch runs the whole solve:
//
//  * CTA c owns B consecutive 256-row tiles; thread t of its 512 owns rows t,
//    t + 512, ...: x, r and Ap of a row stay in one thread's registers.  The
//    matrix is its masks (registers) and its diagonals' values: constants, or
//    read through L1 and L2.
//  * The direction p sits in shared memory: the CTA's own rows and every row
//    its diagonals reach (up to one piece per diagonal, merged where they
//    meet), so a product is one shared-memory read.  Every CTA forms the new
//    direction of all of them itself, fma(beta, p, r), the owner's operation
//    on the owner's doubles; what travels is r.
//  * What travels carries its own arrival: a 16-byte word {value, number of
//    the iteration}, written and read as one 128-bit access.  A reader polls
//    the word until its number is the one it waits for, so no fence, flag or
//    counter is needed, and a word is not written again before every reader
//    has used it: r of the next iteration is formed from sums that contain
//    each reader's products with this one.
//  * The two dot products go the same way: a CTA publishes its sums as such
//    words in a 128-byte line of its own, and every CTA reads all lines (two
//    sets of lines in turn, since a CTA may publish the next sums before a
//    slower one has read these).  These two exchanges are all the
//    synchronisation of an iteration; r travels under the second one.
//  * Beyond kDiaCgTileSums tiles r travels as plain doubles instead, read two
//    to a load behind a flag per CTA: the words' bytes and the instructions
//    for them were what an iteration took there.  A CTA raises its flag (after
//    a fence) and waits for those of the CTAs that hold its reach while the
//    second sums travel.  Per iteration, with words -> with flags: 100^3
//    19.5 -> 15.1 us, 90^3 17.6 -> 12.6, 80^3 11.5 -> 9.6, 1000^2 12.7 -> 10.7.
//  * A line has one writer and is polled at one word: with the words of
//    several CTAs in a line, or all of them polled, the polls held up the
//    stores and each other (22,500 rows: 17,000 cycles for the two exchanges
//    of an iteration against 5,800).  The scalars are formed by one warp: a
//    division in all 512 threads costs 300 cycles of the FP64 pipe.
//  * Up to kDiaCgTileSums tiles the sums are per tile, in the order every
//    other CG path uses (reduce256 over the tiles), so the bits are theirs;
//    beyond, per CTA (its tile sums by a warp's shuffle tree), so that they
//    also depend on the number of SMs.
//
// Every wait is bounded (kWaitLimitNs); a CTA that gives up sets the error
// word and the state to kCgDeviceError and leaves, and the others give up in
// turn.
#include <algorithm>

#include "cg.cuh"
#include "dia.cuh"
#include "park_rows.cuh"

namespace nm {
namespace {

constexpr int kDiaCgThreads = 512;
constexpr int kDiaCgTileSums = 1024;  // 262,144 rows
constexpr int kDiaCgMaxDiag = 8;
constexpr int64_t kDiaCgMinRows = 32768;
constexpr size_t kDiaCgMaxSmem = 208 * 1024;
constexpr int kDiaCgMaxGrid = 160;
constexpr int kDiaCgSets = 3;  // sets of lines: two of sums in turn, one of flags
constexpr int kDiaCgLine = 8;  // words of a CTA's line: its tiles, at most 8
static_assert(kDiaCgTilesPerRow == kDiaCgThreads / kThreads, "tiles of a row of all threads");

struct DiaCgArgs {
    DiaView<double> D;
    int32_t ndiag;
    CgState* st;
    const double* P0;  // p_0 = r_0 (the initial kernel)
    const double* R0;
    ulonglong2* rword;  // per row: {r, iteration}; without tile sums r alone, in 8 bytes
    ulonglong2* lines;  // 2 x grid lines of {sum, exchange}, grid lines of {0, iteration}
    unsigned int* err;
    int32_t ntile, tiles_per_cta;
    int32_t early_r;  // shared memory has room for the r of other CTAs' rows
};

// The rows a CTA keeps the direction of: the union of its own rows and of
// [row0 + off, row1 + off) for each diagonal, clipped to the matrix, in merged
// ascending segments, one behind the other in shared memory.
struct DiaReach {
    int32_t nseg, total, own;  // own: slot of row row0
    int32_t row[kDiaCgMaxDiag + 1], len[kDiaCgMaxDiag + 1], base[kDiaCgMaxDiag + 1];
    int32_t delta[kDiaCgMaxDiag];  // slot of (row row0 + i, diagonal k): i + delta[k]
};

__host__ __device__ inline void dia_reach(const int32_t* off, int nd, int32_t n, int32_t row0,
                                          int32_t row1, DiaReach* out) {
    out->nseg = 0;
    int32_t total = 0;
    bool own_done = false;
    // ascending starts: the diagonals in order, the own rows (offset 0) among them
    for (int k = 0; k <= nd; ++k) {
        int32_t o;
        if (!own_done && (k == nd || off[k] >= 0)) {
            own_done = true;
            o = 0;
            --k;  // diagonal k comes next
        } else if (k < nd) {
            o = off[k];
        } else {
            break;
        }
        const int64_t a64 = int64_t(row0) + o, b64 = int64_t(row1) + o;
        const int32_t a = static_cast<int32_t>(a64 < 0 ? 0 : (a64 > n ? n : a64));
        const int32_t b = static_cast<int32_t>(b64 < 0 ? 0 : (b64 > n ? n : b64));
        if (b <= a) continue;
        int s = out->nseg - 1;
        if (s >= 0 && a <= out->row[s] + out->len[s]) {
            const int32_t e = out->row[s] + out->len[s];
            if (b > e) {
                out->len[s] += b - e;
                total += b - e;
            }
        } else {
            ++s;
            out->nseg = s + 1;
            out->row[s] = a;
            out->len[s] = b - a;
            total += (total ^ a) & 1;  // even rows at even slots
            out->base[s] = total;
            total += b - a;
        }
    }
    out->total = total;
    for (int k = -1; k < nd; ++k) {
        const int32_t o = k < 0 ? 0 : off[k];
        const int64_t a64 = int64_t(row0) + o, b64 = int64_t(row1) + o;
        int32_t d = 0;
        if (b64 > 0 && a64 < n) {
            const int64_t a = a64 < 0 ? 0 : a64;
            int s = 0;
            while (s + 1 < out->nseg && a >= int64_t(out->row[s]) + out->len[s]) ++s;
            d = static_cast<int32_t>(out->base[s] + a64 - out->row[s]);
        }
        if (k < 0) out->own = d;
        else out->delta[k] = d;
    }
}

__device__ __forceinline__ void st_word(ulonglong2* p, double v, uint64_t seq) {
    asm volatile(
        "{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\t"
        "st.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
        "l"(__double_as_longlong(v)), "l"(seq)
        : "memory");
}

__device__ __forceinline__ ulonglong2 ld_word(const ulonglong2* p) {
    ulonglong2 r;
    asm volatile(
        "{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\t"
        "mov.b128 {%0, %1}, w;\n\t}"
        : "=l"(r.x), "=l"(r.y)
        : "l"(p)
        : "memory");
    return r;
}

// The value of *p once it carries `seq` (`w`: a first look at it); *ok turns
// false when the wait gave up.
__device__ __forceinline__ double wait_word(const ulonglong2* p, ulonglong2 w, uint64_t seq,
                                            unsigned int* err, bool* ok) {
    if (w.y != seq && *ok) {
        const uint64_t t0 = global_timer_ns();
        for (uint32_t it = 1;; ++it) {
            w = ld_word(p);
            if (w.y == seq) break;
            if ((it & 255u) == 0 && (global_timer_ns() - t0 > kWaitLimitNs || it > (1u << 30))) {
                atomicOr(err, kErrWaitTimeout);
                *ok = false;
                break;
            }
        }
    }
    return __longlong_as_double(static_cast<long long>(w.x));
}

// Shared memory of the exchanges.
struct DiaExchange {
    double scr[kDiaCgMaxOwnTiles][kWarps];  // this CTA's tiles: a sum per warp
    double sv[kDiaCgTileSums];  // everyone's sums
    double red[kWarps];
    double sc[4];               // what `scalars` leaves
    double rel;                 // the residual the stopping test looks at
};

// The warp sums of the values of the thread's rows q0, q0 + 1, ... (a group of
// its Q), parked per tile and warp.
template <int Q>
__device__ __forceinline__ void park_sums(const double (&d)[kDiaCgGroup], int q0,
                                          double (*scr)[kWarps]) {
    static_assert(Q <= kDiaCgMaxQ, "room in scr");
    constexpr int N = Q < kDiaCgGroup ? Q : kDiaCgGroup, P = park_width(N);
    double v[P];
#pragma unroll
    for (int q = 0; q < P; ++q) v[q] = q < N ? d[q] : 0.0;
    multi_warp_sum<P>(v);
    const int warp = threadIdx.x >> 5, row = park_row(threadIdx.x & 31, q0, Q);
    if (row >= 0) scr[row * kDiaCgTilesPerRow + warp / kWarps][warp % kWarps] = v[0];
}

// Publishes this CTA's sums (parked in X.scr; the caller has synchronised).
template <bool TILES>
__device__ __forceinline__ void publish(const DiaCgArgs& a, uint64_t phase, int ntile_own,
                                        DiaExchange& X) {
    const int t = threadIdx.x;
    ulonglong2* line =
        a.lines + (size_t(phase & 1u) * gridDim.x + blockIdx.x) * kDiaCgLine;
    if constexpr (TILES) {
        if (t < ntile_own) {
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) s += X.scr[t][w];
            st_word(line + t, s, phase);
        }
    } else if (t < 32) {
        double s = 0.0;
        if (t < ntile_own) {
#pragma unroll
            for (int w = 0; w < kWarps; ++w) s += X.scr[t][w];
        }
        s = warp_sum(s);
        if (t == 0) st_word(line, s, phase);
    }
}

// Everyone's sums of this exchange and their total in the fixed order: the
// first 256 threads read the lines while the others run meanwhile(); one warp
// then calls scalars(total, sc), and all threads find sc filled.  False in
// every thread when a wait gave up (meanwhile() clears its ok).
template <bool TILES, class M, class F>
__device__ __forceinline__ bool gather(const DiaCgArgs& a, uint64_t phase, DiaExchange& X,
                                       const M& meanwhile, const F& scalars) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int G = gridDim.x;
    const ulonglong2* lines = a.lines + size_t(phase & 1u) * G * kDiaCgLine;
    bool ok = true;
    if (t >= kThreads) {
        meanwhile(ok);
    } else {
        // thread t waits for CTA t's line: its first words (one sector)
        if (t < G) {
            const ulonglong2* line = lines + t * kDiaCgLine;
            const int first = TILES ? t * a.tiles_per_cta : t;
            const bool two = TILES && a.tiles_per_cta > 1 && first + 1 < a.ntile;
            const ulonglong2 w0 = ld_word(line);
            const ulonglong2 w1 = two ? ld_word(line + 1) : w0;
            X.sv[first] = wait_word(line, w0, phase, a.err, &ok);
            if (two) X.sv[first + 1] = wait_word(line + 1, w1, phase, a.err, &ok);
        }
        if (TILES && a.tiles_per_cta > 2) {
            // then its other words, written with the first: eight threads to a
            // line, so that a load covers whole lines
            asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
            constexpr int kPass = kDiaCgMaxGrid * kDiaCgLine / kThreads;
            const int w = t & (kDiaCgLine - 1);
            ulonglong2 v[kPass];
            bool in[kPass];
#pragma unroll
            for (int i = 0; i < kPass; ++i) {
                const int c = (t >> 3) + (kThreads / kDiaCgLine) * i;
                in[i] = w >= 2 && c < G && w < a.tiles_per_cta && c * a.tiles_per_cta + w < a.ntile;
                if (in[i]) v[i] = ld_word(lines + c * kDiaCgLine + w);
            }
#pragma unroll
            for (int i = 0; i < kPass; ++i) {
                const int c = (t >> 3) + (kThreads / kDiaCgLine) * i;
                if (in[i])
                    X.sv[c * a.tiles_per_cta + w] =
                        wait_word(lines + c * kDiaCgLine + w, v[i], phase, a.err, &ok);
            }
        }
    }
    ok = __syncthreads_and(ok);
    if constexpr (TILES) {
        if (warp < kWarps) {  // reduce256
            double s = 0.0;
            for (int i = t; i < a.ntile; i += kThreads) s += X.sv[i];
            s = warp_sum(s);
            if (lane == 0) X.red[warp] = s;
            asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
        }
        if (warp == 0) {
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) s += X.red[w];
            scalars(s, X.sc);
        }
    } else if (warp == 0) {
        double s = 0.0;
        for (int i = lane; i < G; i += 32) s += X.sv[i];
        s = warp_sum(s);
        scalars(__shfl_sync(0xffffffffu, s, 0), X.sc);
    }
    __syncthreads();
    return ok;
}

template <int Q, int KC, bool CONST, bool TILES>
__global__ void __launch_bounds__(kDiaCgThreads, 1) cg_dia_kernel(const DiaCgArgs a) {
    constexpr int NT = kDiaCgThreads;
    extern __shared__ __align__(16) double pe[];  // the direction on DiaReach's rows
    __shared__ DiaExchange X;
    __shared__ DiaReach reach;
    __shared__ int32_t near[2 * kDiaCgMaxDiag];
    // the reach without the own rows: {first row, end row, slot - row, 0}
    __shared__ int4 pieces[kDiaCgMaxDiag + 2];
    __shared__ int32_t npiece, split;
    const int t = threadIdx.x;
    CgState* st = a.st;
    if (__ldcg(&st->done)) return;  // the initial kernel decided already
    const int32_t n = a.D.n;
    const int tile0 = blockIdx.x * a.tiles_per_cta;
    const int ntile_own = min(a.tiles_per_cta, a.ntile - tile0);
    const int32_t row0 = tile0 * kThreads;
    const int32_t row1 = min(n, (tile0 + ntile_own) * kThreads);
    double* xg = st->x;
    const double bnorm = __ldcg(&st->bnorm), tol = __ldcg(&st->tol);
    const int32_t max_iter = __ldcg(&st->max_iter), guard = __ldcg(&st->guard);
    double rr = __ldcg(&st->rr);
    int32_t iter = __ldcg(&st->iter);
    if (t == 0) {
        dia_reach(a.D.off, a.ndiag, n, row0, row1, &reach);
        int np = 0;
        for (int s = 0; s < reach.nseg; ++s) {
            const int32_t first = reach.row[s], end = first + reach.len[s];
            const int32_t shift = reach.base[s] - first;
            const int32_t lo = min(end, row0), hi = max(first, row1);
            if (first < lo) pieces[np++] = make_int4(first, lo, shift, 0);
            if (hi < end) pieces[np++] = make_int4(hi, end, shift, 0);
        }
        npiece = np;
        // the split nearest to half of the rows; none where one piece holds
        // three quarters of them
        int total = 0, best = 0, most = 0;
        for (int s = 0; s < np; ++s) total += pieces[s].y - pieces[s].x;
        most = total - total / 4;
        for (int s = 1, before = 0; s < np; ++s) {
            before += pieces[s - 1].y - pieces[s - 1].x;
            const int larger = max(before, total - before);
            if (larger < most) {
                most = larger;
                best = s;
            }
        }
        split = best;
    }
    __syncthreads();
    const int32_t own = reach.own;

    double cv[KC];
    int32_t at[KC];  // slot of (this thread's first row, diagonal k)
#pragma unroll
    for (int k = 0; k < KC; ++k) {
        cv[k] = a.D.cval[k];
        at[k] = t + (k < a.ndiag ? reach.delta[k] : 0);
    }
    const uint8_t* mask = static_cast<const uint8_t*>(a.D.mask);
    double r[Q], ap[Q], x[Q];
    uint32_t m[(Q + 3) / 4] = {};  // masks, four to a word
    uint32_t shown = 0;            // bit q: another CTA keeps row q's direction too
    uint32_t have = 0;             // bit q: the thread has a row q
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int32_t row = row0 + q * NT + t;
        r[q] = ap[q] = x[q] = 0.0;
        if (row < row1) {
            have |= 1u << q;
            m[q / 4] |= uint32_t(mask[row]) << (8 * (q % 4));
            r[q] = __ldcg(a.R0 + row);
            x[q] = xg[row];
            for (int k = 0; k < a.ndiag; ++k) {
                const int64_t i = int64_t(row) - a.D.off[k];  // the row that reads this one
                if (i >= 0 && i < n && (i < row0 || i >= row1)) shown |= 1u << q;
            }
        }
    }
    for (int s = 0; s < reach.nseg; ++s)
        for (int e = t; e < reach.len[s]; e += NT)
            pe[reach.base[s] + e] = __ldcg(a.P0 + reach.row[s] + e);
    __syncthreads();

    double* rplain = reinterpret_cast<double*>(a.rword);
    ulonglong2* flags = a.lines + size_t(2) * gridDim.x * kDiaCgLine;
    if (!TILES && t < 2 * kDiaCgMaxDiag) {  // the CTAs of each diagonal's first and last row
        const int d = t >> 1;
        int c = -1;
        if (d < a.ndiag) {
            const int64_t f = int64_t(row0) + a.D.off[d], l = int64_t(row1) - 1 + a.D.off[d];
            if (l >= 0 && f < n) {
                const int64_t row = t & 1 ? (l < n ? l : n - 1) : (f > 0 ? f : 0);
                c = static_cast<int>(row / (int64_t(a.tiles_per_cta) * kThreads));
            }
        }
        near[t] = c == int(blockIdx.x) ? -1 : c;
    }
    uint64_t phase = 0;
    double beta = 0.0;
    bool failed = false;
    int status = kCgOk;
    for (uint64_t k = 1;; ++k) {
        // (kept from being unpacked ahead of the loop into a register a bit)
#pragma unroll
        for (int j = 0; j < (Q + 3) / 4; ++j) asm volatile("" : "+r"(m[j]));
        asm volatile("" : "+r"(have), "+r"(shown));
        // ---- Ap = A p (serial CSR-order row sums), p.Ap ----
#pragma unroll
        for (int q0 = 0; q0 < Q; q0 += kDiaCgGroup) {
            constexpr int N = kDiaCgGroup;
            double d[N];
#pragma unroll
            for (int j = 0; j < N; ++j) {
                d[j] = 0.0;
                const int q = q0 + j;
                if (q >= Q) continue;
                const uint32_t mq = (m[q / 4] >> (8 * (q % 4))) & 0xffu;
                double xs[KC], vs[KC];
#pragma unroll
                for (int e = 0; e < KC; ++e) {
                    xs[e] = 0.0;
                    vs[e] = cv[e];
                    if (mq >> e & 1u) {
                        xs[e] = pe[at[e] + q * NT];
                        if constexpr (!CONST)
                            vs[e] = __ldg(static_cast<const double*>(a.D.val) + e * a.D.ld +
                                          (row0 + q * NT + t));
                    }
                }
                double acc = 0.0;
#pragma unroll
                for (int e = 0; e < KC; ++e)
                    if (mq >> e & 1u) acc = add_rn(acc, mul_rn(vs[e], xs[e]));
                ap[q] = acc;
                if (have >> q & 1u) d[j] = fma(pe[own + q * NT + t], acc, 0.0);
                if (j % 2 == 1) asm volatile("" ::: "memory");  // two rows' loads in flight
            }
            park_sums<Q>(d, q0, X.scr);
        }
        __syncthreads();
        publish<TILES>(a, ++phase, ntile_own, X);
        // the stopping test of the last iteration, while the sums travel
        auto test = [&](bool&) {
            if (k > 1 && t == NT - 1) X.rel = sqrt(rr) / bnorm;
        };
        if (!gather<TILES>(a, phase, X, test, [&](double pAp, double* sc) {
                const double alpha = rr / pAp;
                if (t == 0) {
                    sc[0] = pAp;
                    sc[1] = alpha;
                }
            })) {
            failed = true;
            break;
        }
        if (k > 1) {
            const double rel = X.rel;
            if (rel < tol) {
                if (blockIdx.x == 0 && t == 0) {
                    st->iter = iter; st->converged = 1; st->iters = iter; st->final_res = rel;
                    st->rr = rr;
                }
                break;
            }
            if (iter >= max_iter) {
                if (blockIdx.x == 0 && t == 0) {
                    st->iter = iter; st->converged = 0; st->iters = max_iter; st->final_res = rel;
                    st->beta = beta; st->rr = rr;
                }
                break;
            }
        }
        const double pAp = X.sc[0], alpha = X.sc[1];
        if (guard && fabs(pAp) < 1e-300) {
            status = kCgBreakdown;
            if (blockIdx.x == 0 && t == 0) {
                st->pAp = pAp;
                st->converged = 0;
                st->iters = iter;
                st->final_res = sqrt(rr) / bnorm;
            }
            break;
        }
        // ---- x += alpha p, r -= alpha Ap, r.r; r to the CTAs that keep the row ----
#pragma unroll
        for (int q0 = 0; q0 < Q; q0 += kDiaCgGroup) {
            double d[kDiaCgGroup];
#pragma unroll
            for (int j = 0; j < kDiaCgGroup; ++j) {
                d[j] = 0.0;
                const int q = q0 + j;
                if (q >= Q) continue;
                if (have >> q & 1u) {
                    r[q] = fma(-alpha, ap[q], r[q]);  // r = -alpha*Ap + r
                    if (shown >> q & 1u) {
                        if constexpr (TILES) st_word(a.rword + (row0 + q * NT + t), r[q], k);
                        else __stcg(rplain + (row0 + q * NT + t), r[q]);
                    }
                    x[q] = fma(alpha, pe[own + q * NT + t], x[q]);  // x = alpha*p + x
                    d[j] = fma(r[q], r[q], 0.0);
                }
            }
            park_sums<Q>(d, q0, X.scr);
        }
        __syncthreads();
        publish<TILES>(a, ++phase, ntile_own, X);
        // The other CTAs' rows of r, by the threads of this CTA from `first_t`
        // on; where shared memory has room for them, while the sums travel.
        auto others = [&](int first_t, auto flight, bool& ok, auto&& use) {
            constexpr int N = decltype(flight)::value;  // words in flight per thread
            const int nt = NT - first_t;
            for (int s = 0; s < reach.nseg; ++s) {
                const int32_t len = reach.len[s], first = reach.row[s], base = reach.base[s];
                for (int e0 = t - first_t; e0 < len; e0 += nt * N) {
                    ulonglong2 w[N];
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        const int e = e0 + j * nt;
                        const bool mine = first + e >= row0 && first + e < row1;
                        if (e < len && !mine) w[j] = ld_word(a.rword + first + e);
                    }
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        const int e = e0 + j * nt;
                        const bool mine = first + e >= row0 && first + e < row1;
                        if (e < len && !mine)
                            use(base + e, wait_word(a.rword + first + e, w[j], k, a.err, &ok));
                    }
                }
            }
        };
        double* hr = pe + reach.total;
        // Without TILES: two rows to a load, from an even row on, eight loads
        // in flight per thread; half of the threads take the pieces before
        // `split`, the others the rest, so that two pieces are under way.
        auto plain = [&] {
            const bool both = split == 0, upper = !both && t >= NT / 2;
            const int nt = both ? NT : NT / 2, tt = upper ? t - NT / 2 : t;
            const int s1 = both || upper ? npiece : split;
            for (int s = upper ? split : 0; s < s1; ++s) {
                constexpr int N = 8;
                const int4 pc = pieces[s];
                const int32_t e1 = (pc.x & ~1) + 2 * tt;
                double* const p2 = pe + pc.z;
                for (int32_t e0 = e1; e0 < pc.y; e0 += 2 * nt * N) {
                    double2 w[N];
#pragma unroll
                    for (int j = 0; j < N; ++j)
                        if (e0 + 2 * nt * j < pc.y)
                            w[j] = __ldcg(reinterpret_cast<const double2*>(rplain + e0 + 2 * nt * j));
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        const int32_t e = e0 + 2 * nt * j;
                        if (e >= pc.x && e + 1 < pc.y) {
                            double2 v = *reinterpret_cast<double2*>(p2 + e);
                            v.x = fma(beta, v.x, w[j].x);
                            v.y = fma(beta, v.y, w[j].y);
                            *reinterpret_cast<double2*>(p2 + e) = v;
                        } else if (e >= pc.x && e < pc.y) {
                            p2[e] = fma(beta, p2[e], w[j].x);
                        } else if (e < pc.x && e + 1 < pc.y) {
                            p2[e + 1] = fma(beta, p2[e + 1], w[j].y);
                        }
                    }
                }
            }
        };
        auto early = [&](bool& ok) {
            if constexpr (!TILES) {
                // this CTA's flag, and those of the CTAs that hold its reach
                if (t == kThreads) {
                    __threadfence();
                    st_word(flags + blockIdx.x * kDiaCgLine, 0.0, k);
                } else if (t >= kThreads + 32 && t < kThreads + 32 + 2 * kDiaCgMaxDiag) {
                    const int c = near[t - kThreads - 32];
                    if (c >= 0) {
                        const ulonglong2* f = flags + c * kDiaCgLine;
                        wait_word(f, ld_word(f), k, a.err, &ok);
                        __threadfence();
                    }
                }
            } else if (a.early_r) {
                others(kThreads, std::integral_constant<int, 4>(), ok,
                       [&](int i, double rj) { hr[i] = rj; });
            }
        };
        if (!gather<TILES>(a, phase, X, early, [&](double rr_new, double* sc) {
                const double b = rr_new / rr;
                if (t == 0) {
                    sc[0] = rr_new;
                    sc[1] = b;
                }
            })) {
            failed = true;
            break;
        }
        rr = X.sc[0];
        beta = X.sc[1];
        ++iter;  // the stopping test: in the next exchange, before anything else is changed
        // ---- p = r + beta p: own rows, then the rows of other CTAs ----
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (have >> q & 1u)
                pe[own + q * NT + t] = fma(beta, pe[own + q * NT + t], r[q]);
        if constexpr (!TILES) {
            plain();
            __syncthreads();
        } else if (a.early_r) {
            for (int s = 0; s < reach.nseg; ++s)
                for (int e = t; e < reach.len[s]; e += NT) {
                    const int32_t row = reach.row[s] + e, i = reach.base[s] + e;
                    if (row < row0 || row >= row1) pe[i] = fma(beta, pe[i], hr[i]);
                }
            __syncthreads();
        } else {
            bool ok = true;
            others(0, std::integral_constant<int, 8>(), ok, [&](int i, double rj) { pe[i] = fma(beta, pe[i], rj); });
            if (!__syncthreads_and(ok)) {
                failed = true;
                break;
            }
        }
    }
    if (failed) {
        if (t == 0) {
            atomicExch(&st->status, kCgDeviceError);
            atomicExch(&st->done, 1);
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int32_t row = row0 + q * NT + t;
        if (row < row1) xg[row] = x[q];
    }
    if (blockIdx.x == 0 && t == 0) {
        if (status != kCgOk) st->status = status;
        st->done = 1;
    }
}

template <int Q, int KC>
const void* dia_cg_fn(bool constant) {
    return constant ? reinterpret_cast<const void*>(cg_dia_kernel<Q, KC, true, true>)
                    : reinterpret_cast<const void*>(cg_dia_kernel<Q, KC, false, true>);
}

template <int KC>
const void* dia_cg_k(bool tiles, int Q, bool constant) {
    if (tiles) {
        if (Q == 1) return dia_cg_fn<1, KC>(constant);
        if (Q == 2) return dia_cg_fn<2, KC>(constant);
        return dia_cg_fn<4, KC>(constant);
    }
    if (Q == 4) return reinterpret_cast<const void*>(cg_dia_kernel<4, KC, true, false>);
    if (Q == 8) return reinterpret_cast<const void*>(cg_dia_kernel<8, KC, true, false>);
    if (Q == 11) return reinterpret_cast<const void*>(cg_dia_kernel<11, KC, true, false>);
    return reinterpret_cast<const void*>(cg_dia_kernel<14, KC, true, false>);
}

// Rows per thread of the kernel that takes `Q` (0: none does).  11: 90^3, of
// 10 rows per thread, takes 12.6 us per iteration, with the kernel for 14 15.9.
int q_class(bool tiles, int Q) {
    if (tiles) return Q <= 1 ? 1 : (Q <= 2 ? 2 : (Q <= 4 ? 4 : 0));
    return Q <= 4 ? 4 : (Q <= 8 ? 8 : (Q <= 11 ? 11 : (Q <= 14 ? 14 : 0)));
}

const void* dia_cg_kernel_for(const nm_csr* A, const CgWorkspace* ws) {
    const int nd = A->dia.ndiag;
    const bool c = A->dia.constant;
    if (nd <= 3) return dia_cg_k<3>(ws->dia_tiles, ws->dia_q, c);
    if (nd <= 5) return dia_cg_k<5>(ws->dia_tiles, ws->dia_q, c);
    if (nd <= 7) return dia_cg_k<7>(ws->dia_tiles, ws->dia_q, c);
    return dia_cg_k<8>(ws->dia_tiles, ws->dia_q, c);
}

size_t dia_cg_bytes(const CgWorkspace* ws) {
    return sizeof(ulonglong2) *
           (size_t(kDiaCgSets * kDiaCgLine) * size_t(ws->dia_grid) + size_t(ws->n));
}

}  // namespace

int plan_dia(const nm_csr* A, CgWorkspace* ws) {
    ws->dia = false;
    const int64_t n = A->nrows;
    // rows of at most 8 nonzeros in blocks of whole 256-row tiles, so that
    // the row-block sums of the other paths are tile sums
    if (A->dia.ndiag < 1 || A->dia.ndiag > kDiaCgMaxDiag || !A->use_dia()) return NM_OK;
    if (A->tune.max_rows != kThreads) return NM_OK;
    const int64_t ntile = (n + kThreads - 1) / kThreads;
    if (A->nblk != ntile) return NM_OK;
    // Small systems stay on one cluster, whose barriers are shorter (100^2: 3.5
    // against 4.0 us per iteration; 32^3: the same; 200^2: 5.4 against 4.5).
    if (n <= kDiaCgMinRows) return NM_OK;
    // Beyond the tile sums' range values that vary are streamed from L2 for
    // every product by too few threads (100^3: 46 us per iteration, 43 on the
    // CUDA-graph path; 64^3: 12.7 against 19).
    if (ntile > kDiaCgTileSums && !A->dia.constant) return NM_OK;
    const int sms = sm_count();
    const int B = static_cast<int>((ntile + sms - 1) / sms);
    ws->dia_tiles = ntile <= kDiaCgTileSums;
    ws->dia_q = q_class(ws->dia_tiles, (B * kThreads + kDiaCgThreads - 1) / kDiaCgThreads);
    if (ws->dia_q == 0) return NM_OK;
    ws->dia_b = B;
    ws->dia_grid = static_cast<int>((ntile + B - 1) / B);
    int32_t total = 0;
    for (int c = 0; c < ws->dia_grid; ++c) {
        DiaReach reach;
        const int32_t row0 = c * B * kThreads;
        dia_reach(A->dia.off, A->dia.ndiag, A->nrows, row0,
                  static_cast<int32_t>(std::min<int64_t>(n, int64_t(row0) + B * kThreads)), &reach);
        total = std::max(total, reach.total);
    }
    ws->dia_smem = sizeof(double) * size_t(total);
    if (ws->dia_smem > kDiaCgMaxSmem || ws->dia_grid > kDiaCgMaxGrid) return NM_OK;
    // Other CTAs' words of r under the second exchange, by half the threads,
    // where shared memory has room (500^2: 7.9 against 8.4 us per iteration
    // after it).
    ws->dia_early = ws->dia_tiles && 2 * ws->dia_smem <= kDiaCgMaxSmem;
    if (ws->dia_early) ws->dia_smem *= 2;
    const void* fn = dia_cg_kernel_for(A, ws);
    NM_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(kDiaCgMaxSmem)));
    int occ = 0;
    NM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kDiaCgThreads, ws->dia_smem));
    if (int64_t(occ) * sms < ws->dia_grid) return NM_OK;
    // the sums' lines and the words of r, allocated for this solve only
    if (cudaMalloc(&ws->dia_mem, dia_cg_bytes(ws)) !=
        cudaSuccess) {
        cudaGetLastError();  // no room: the other paths run
        ws->dia_mem = nullptr;
        return NM_OK;
    }
    ws->dia = true;
    return NM_OK;
}

int launch_dia_cg(const nm_csr* A, CgWorkspace* ws, cudaStream_t s) {
    // every word unnumbered (iterations and exchanges count from 1)
    NM_CUDA_TRY(cudaMemsetAsync(ws->dia_mem, 0, dia_cg_bytes(ws), s));
    DiaCgArgs a;
    a.D = dia_view<double>(A->dia, A->nrows);
    a.ndiag = A->dia.ndiag;
    a.st = ws->st;
    a.P0 = ws->p;
    a.R0 = ws->r;
    a.lines = static_cast<ulonglong2*>(ws->dia_mem);
    a.rword = a.lines + size_t(kDiaCgSets * kDiaCgLine) * ws->dia_grid;
    a.err = ws->err;
    a.ntile = A->nblk;
    a.tiles_per_cta = ws->dia_b;
    a.early_r = ws->dia_early;
    void* args[] = {&a};
    NM_CUDA_TRY(cudaLaunchCooperativeKernel(dia_cg_kernel_for(A, ws), dim3(ws->dia_grid),
                                            dim3(kDiaCgThreads), args, ws->dia_smem, s));
    return NM_OK;
}

}  // namespace nm
