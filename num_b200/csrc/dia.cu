// dia.cu -- finding a matrix's diagonal form (dia.cuh), and its SpMV.
#include <algorithm>
#include <cstring>

#include "batch_shape.cuh"
#include "dia.cuh"

namespace nm {

namespace {

// What the search kernel finds, in device memory (nm_csr::d_dia_room).
constexpr int kDiaSlots = kDiaMax + 1;         // one more than allowed: overflow
constexpr int32_t kDiaNoOff = INT32_MIN;       // col - row is never this
constexpr uint64_t kDiaNoVal = 0x7FF0D1A0D1A0D1A0ull;  // a signalling NaN
struct DiaTable {
    int32_t off[kDiaSlots];
    uint32_t overflow;  // more than kDiaMax diagonals
    uint32_t disorder;  // a row's columns do not ascend
    uint32_t varying;   // some diagonal holds different numbers
    unsigned long long pairs;  // (warp of 32 rows, diagonal) pairs with an entry
    uint64_t val[kDiaSlots];
};
static_assert(sizeof(DiaTable) <= kDiaTableBytes, "table room");

template <typename V>
__device__ __forceinline__ uint64_t value_bits(V v) {
    if constexpr (std::is_same_v<V, double>)
        return static_cast<uint64_t>(__double_as_longlong(v));
    else if constexpr (std::is_same_v<V, float>)
        return __float_as_uint(v);
    else
        return __bfloat16_as_ushort(v);
}

// The offsets a look at some rows on the host found, each with the position of
// one entry on it: the table's first contents.  (From an empty table every
// thread of the search goes for the same slots at once: 1.3 ms of atomics on
// 250,000 rows.)
struct DiaSeed {
    int32_t count;
    int32_t off[kDiaMax];
    int32_t at[kDiaMax];
};

template <typename V>
__global__ void dia_seed_kernel(DiaSeed seed, const V* __restrict__ vals, DiaTable* T) {
    const int s = threadIdx.x;
    if (s < kDiaSlots) {
        T->off[s] = s < seed.count ? seed.off[s] : kDiaNoOff;
        T->val[s] = s < seed.count ? value_bits(vals[seed.at[s]]) : kDiaNoVal;
    }
    if (s == 0) {
        T->overflow = T->disorder = T->varying = 0u;
        T->pairs = 0ull;
    }
}

// Every offset col - row of the matrix into the table (new ones in the order
// found), whether the columns of each row ascend, and whether the entries of
// each diagonal are all the same number.  A CTA keeps a copy of the table in
// shared memory, so global atomics happen once per offset and CTA.
template <typename V>
__global__ void __launch_bounds__(kThreads)
    dia_find_kernel(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                    const V* __restrict__ vals, int32_t nrows, DiaTable* T) {
    __shared__ volatile int32_t off[kDiaSlots];
    __shared__ volatile uint64_t val[kDiaSlots];
    if (threadIdx.x < kDiaSlots) {
        off[threadIdx.x] = __ldcg(&T->off[threadIdx.x]);
        val[threadIdx.x] = __ldcg(reinterpret_cast<unsigned long long*>(&T->val[threadIdx.x]));
    }
    __syncthreads();
    bool varying = false;
    for (int64_t r = int64_t(blockIdx.x) * kThreads + threadIdx.x; r < nrows;
         r += int64_t(gridDim.x) * kThreads) {
        if (__ldcg(&T->overflow) | __ldcg(&T->disorder)) return;
        const int32_t z1 = __ldg(rp + r + 1);
        int32_t prev = -1;
        for (int32_t z = __ldg(rp + r); z < z1; ++z) {
            const int32_t c = __ldg(ci + z);
            if (c <= prev) {
                T->disorder = 1u;
                return;
            }
            prev = c;
            const int32_t d = c - static_cast<int32_t>(r);
            // its slot: the first that holds it; an empty slot of the copy is
            // taken (or found taken) in the table, one read of a slot a turn
            int s = 0;
            while (s < kDiaSlots) {
                int32_t have = off[s];
                if (have == kDiaNoOff) {
                    const int32_t old = atomicCAS(&T->off[s], kDiaNoOff, d);
                    have = old == kDiaNoOff ? d : old;
                    off[s] = have;
                }
                if (have == d) break;
                ++s;
            }
            if (s >= kDiaMax) {
                T->overflow = 1u;
                return;
            }
            if (!varying) {
                const uint64_t b = value_bits(__ldg(vals + z));
                uint64_t have = val[s];
                if (have == kDiaNoVal) {
                    const unsigned long long old =
                        atomicCAS(reinterpret_cast<unsigned long long*>(&T->val[s]),
                                  static_cast<unsigned long long>(kDiaNoVal), b);
                    have = old == kDiaNoVal ? b : old;
                    val[s] = have;
                }
                varying = have != b || b == kDiaNoVal;
                if (varying) T->varying = 1u;
            }
        }
    }
}

struct DiaOffsets {
    int32_t off[kDiaMax];
};

// Masks (and, where val is set, values by diagonal) from the CSR arrays; per
// warp of 32 rows the diagonals it touches are counted into T->pairs.
template <typename V, typename M>
__global__ void __launch_bounds__(kThreads)
    dia_fill_kernel(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                    const V* __restrict__ vals, int32_t nrows, DiaOffsets o, M* __restrict__ mask,
                    V* __restrict__ val, int64_t ld, DiaTable* T) {
    const int64_t r = int64_t(blockIdx.x) * kThreads + threadIdx.x;
    uint32_t m = 0;
    if (r < nrows) {
        const int32_t z1 = __ldg(rp + r + 1);
        int k = 0;  // columns ascend, so do their diagonals
        for (int32_t z = __ldg(rp + r); z < z1; ++z) {
            const int32_t d = __ldg(ci + z) - static_cast<int32_t>(r);
            while (k < kDiaMax - 1 && o.off[k] != d) ++k;
            m |= 1u << k;
            if (val) val[int64_t(k) * ld + r] = __ldg(vals + z);
        }
        mask[r] = static_cast<M>(m);
    }
    const uint32_t any = __reduce_or_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && any) atomicAdd(&T->pairs, static_cast<unsigned long long>(__popc(any)));
}

int64_t row_ctas(const nm_csr* A) { return (int64_t(A->nrows) + kThreads - 1) / kThreads; }

template <typename V>
int launch_search(const nm_csr* A, const DiaSeed& seed) {
    DiaTable* T = reinterpret_cast<DiaTable*>(A->d_dia_room);
    const V* vals = static_cast<const V*>(A->d_values);
    dia_seed_kernel<V><<<1, 32>>>(seed, vals, T);
    dia_find_kernel<V><<<static_cast<int>(std::min<int64_t>(row_ctas(A), int64_t(sm_count()) * 8)),
                         kThreads>>>(A->d_row_ptr, A->d_col_idx, vals, A->nrows, T);
    NM_CHECK_LAUNCH();
    return NM_OK;
}

template <typename V>
int take_form(nm_csr* A) {
    DiaTable* T = reinterpret_cast<DiaTable*>(A->d_dia_room);
    const V* vals = static_cast<const V*>(A->d_values);
    const int32_t n = A->nrows;
    const int64_t want = row_ctas(A);
    DiaTable h;
    NM_CUDA_TRY(cudaMemcpy(&h, T, sizeof h, cudaMemcpyDeviceToHost));
    if (h.overflow || h.disorder) return NM_OK;
    int order[kDiaSlots], nd = 0;
    for (int s = 0; s < kDiaMax; ++s)
        if (h.off[s] != kDiaNoOff) order[nd++] = s;
    if (nd == 0) return NM_OK;
    std::sort(order, order + nd, [&](int a, int b) { return h.off[a] < h.off[b]; });
    const bool constant = h.varying == 0;
    if (!constant && 2 * int64_t(A->nnz) < int64_t(nd) * n) return NM_OK;  // mostly padding
    DiaForm f;
    f.constant = constant;
    f.ld = dia_ld(n);
    DiaOffsets o{};
    for (int k = 0; k < kDiaMax; ++k) {
        f.off[k] = o.off[k] = k < nd ? h.off[order[k]] : 0;
        if (k >= nd || !constant) continue;
        const uint64_t b = h.val[order[k]];
        if (sizeof(V) == 8) {
            std::memcpy(&f.cval[k], &b, 8);
        } else {
            const uint32_t u = sizeof(V) == 4 ? uint32_t(b) : uint32_t(b) << 16;
            float x;
            std::memcpy(&x, &u, 4);
            f.cval[k] = x;
        }
    }
    f.d_mask = A->d_dia_room + kDiaTableBytes;
    if (!constant) {
        const size_t need = sizeof(V) * size_t(nd) * size_t(f.ld);
        f.own_val = need > A->dia_copy_room;
        if (!f.own_val)
            f.d_val = A->d_dia_room + kDiaTableBytes + dia_mask_room(n);
        else if (!alloc_copy(&f.d_val, need))
            return NM_OK;  // no room beside the CSR arrays: they serve alone
    }
    if (nd <= 8)
        dia_fill_kernel<V, uint8_t><<<static_cast<int>(want), kThreads>>>(
            A->d_row_ptr, A->d_col_idx, vals, n, o, static_cast<uint8_t*>(f.d_mask),
            static_cast<V*>(f.d_val), f.ld, T);
    else
        dia_fill_kernel<V, uint16_t><<<static_cast<int>(want), kThreads>>>(
            A->d_row_ptr, A->d_col_idx, vals, n, o, static_cast<uint16_t*>(f.d_mask),
            static_cast<V*>(f.d_val), f.ld, T);
    cudaError_t e = cudaGetLastError();
    bool ragged = false;
    if (constant) {
        if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);  // complete for every stream
    } else {
        // A warp reads a whole 32-row piece of every diagonal one of its rows
        // has: rows that share their diagonals read little they do not use.
        if (e == cudaSuccess) e = cudaMemcpy(&h, T, sizeof h, cudaMemcpyDeviceToHost);
        ragged = 32 * h.pairs > (unsigned long long)A->nnz * 5 / 4 + 32 * kDiaMax;
    }
    if (e != cudaSuccess || ragged) {
        if (f.own_val) cudaFree(f.d_val);
        NM_CUDA_TRY(e);
        return NM_OK;
    }
    f.ndiag = nd;
    A->dia = f;
    return NM_OK;
}

// ---------------------------------------------------------------------------
// y = A x.  kDiaR rows per thread and step, a persistent grid; the masks of
// the next step are loaded under this step's products.  A warp whose rows all
// have every diagonal takes a path without predicates.  Offsets and constant
// values sit in registers: as kernel-parameter operands they cost a load per
// use (118 against 50 instructions per warp of rows).
// ---------------------------------------------------------------------------
constexpr int kDiaThreads = 128;

// A BF16 value, read only if `in`: as an `if` around the load of 16 bits it
// becomes a branch, and a row's loads then wait for one another.
__device__ __forceinline__ __nv_bfloat16 ld_bf16_cs_if(const __nv_bfloat16* p, bool in) {
    unsigned short v;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.b16 %0, 0;\n\t"
        "@q ld.global.cs.u16 %0, [%1];\n\t}"
        : "=h"(v)
        : "l"(p), "r"(unsigned(in)));
    return __ushort_as_bfloat16(v);
}

template <typename V, typename X, typename A, int KC, bool CONST, int R>
__global__ void __launch_bounds__(kDiaThreads)
    spmv_dia_kernel(const DiaView<A> D, int ndiag, const X* __restrict__ x, X* __restrict__ y) {
    using M = DiaMask<KC>;
    const M* __restrict__ mask = static_cast<const M*>(D.mask);
    const V* __restrict__ val = static_cast<const V*>(D.val);
    const uint32_t full_mask = (1u << ndiag) - 1u;
    const int64_t n = D.n, step = int64_t(gridDim.x) * (kDiaThreads * R);
    int32_t off[KC];
    A cv[KC];
#pragma unroll
    for (int k = 0; k < KC; ++k) {
        off[k] = D.off[k];
        asm volatile("" : "+r"(off[k]));
        cv[k] = D.cval[k];
        if constexpr (CONST && sizeof(A) == 8) asm volatile("" : "+d"(cv[k]));
        if constexpr (CONST && sizeof(A) == 4) asm volatile("" : "+f"(cv[k]));
    }
    int64_t b = int64_t(blockIdx.x) * (kDiaThreads * R) + threadIdx.x;
    uint32_t m[R];
#pragma unroll
    for (int r = 0; r < R; ++r) m[r] = b + r * kDiaThreads < n ? mask[b + r * kDiaThreads] : 0u;
    for (; b - int(threadIdx.x) < n; b += step) {
        const X* xp[KC];
#pragma unroll
        for (int k = 0; k < KC; ++k) xp[k] = x + (b + off[k]);
        A xs[R][KC], vs[R][KC];
        bool full[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            full[r] = KC == ndiag && __all_sync(0xffffffffu, m[r] == full_mask);
            const V* vp = val + (b + r * kDiaThreads);
            if (full[r]) {
#pragma unroll
                for (int k = 0; k < KC; ++k) {
                    xs[r][k] = static_cast<A>(__ldg(xp[k] + r * kDiaThreads));
                    vs[r][k] = CONST ? cv[k] : widen<V, A>(ld_value_cs(vp + k * D.ld));
                }
            } else {
#pragma unroll
                for (int k = 0; k < KC; ++k) {
                    xs[r][k] = A(0);
                    vs[r][k] = cv[k];
                    const bool in = m[r] >> k & 1u;
                    if (in) xs[r][k] = static_cast<A>(__ldg(xp[k] + r * kDiaThreads));
                    if constexpr (!CONST && sizeof(V) == 2)
                        vs[r][k] = __bfloat162float(ld_bf16_cs_if(vp + k * D.ld, in));
                    else if constexpr (!CONST)
                        if (in) vs[r][k] = widen<V, A>(ld_value_cs(vp + k * D.ld));
                }
            }
        }
        uint32_t mn[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int64_t nx = b + step + r * kDiaThreads;
            mn[r] = nx < n ? mask[nx] : 0u;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            A acc = A(0);
            const int64_t row = b + r * kDiaThreads;
            if (full[r]) {
#pragma unroll
                for (int k = 0; k < KC; ++k) acc = add_rn(acc, mul_rn(vs[r][k], xs[r][k]));
                y[row] = static_cast<X>(acc);
            } else {
#pragma unroll
                for (int k = 0; k < KC; ++k)
                    if (m[r] >> k & 1u) acc = add_rn(acc, mul_rn(vs[r][k], xs[r][k]));
                if (row < n) y[row] = static_cast<X>(acc);
            }
            m[r] = mn[r];
        }
    }
}

template <typename V, typename X, typename A, int KC, bool CONST, int R>
int launch_dia_r(const nm_csr* M, const X* x, X* y, cudaStream_t s) {
    int occ = 0;
    const auto fn = spmv_dia_kernel<V, X, A, KC, CONST, R>;
    const int st = kernel_occupancy(reinterpret_cast<const void*>(fn), kDiaThreads, &occ);
    if (st != NM_OK) return st;
    const int64_t need = (int64_t(M->nrows) + kDiaThreads * R - 1) / (kDiaThreads * R);
    const int grid = static_cast<int>(std::min<int64_t>(need, int64_t(sm_count()) * occ));
    fn<<<grid, kDiaThreads, 0, s>>>(dia_view<A>(M->dia, M->nrows), M->dia.ndiag, x, y);
    NM_CHECK_LAUNCH();
    return NM_OK;
}

// One row per thread while the rows fit the resident threads at one each (no
// thread then waits for a second row's loads), else two.
template <typename V, typename X, typename A, int KC>
int launch_dia_k(const nm_csr* M, const X* x, X* y, cudaStream_t s) {
    const bool one = int64_t(M->nrows) <= int64_t(sm_count()) * 1024;
    if (M->dia.constant)
        return one ? launch_dia_r<V, X, A, KC, true, 1>(M, x, y, s)
                   : launch_dia_r<V, X, A, KC, true, 2>(M, x, y, s);
    return one ? launch_dia_r<V, X, A, KC, false, 1>(M, x, y, s)
               : launch_dia_r<V, X, A, KC, false, 2>(M, x, y, s);
}

template <typename V, typename X, typename A>
int launch_dia_t(const nm_csr* M, const void* x, void* y, cudaStream_t s) {
    const X* xx = static_cast<const X*>(x);
    X* yy = static_cast<X*>(y);
    const int nd = M->dia.ndiag;
    if (nd <= 3) return launch_dia_k<V, X, A, 3>(M, xx, yy, s);
    if (nd <= 5) return launch_dia_k<V, X, A, 5>(M, xx, yy, s);
    if (nd <= 7) return launch_dia_k<V, X, A, 7>(M, xx, yy, s);
    if (nd <= 8) return launch_dia_k<V, X, A, 8>(M, xx, yy, s);
    if (nd <= 9) return launch_dia_k<V, X, A, 9>(M, xx, yy, s);  // 16-bit masks from here on
    if (nd <= 12) return launch_dia_k<V, X, A, 12>(M, xx, yy, s);
    return launch_dia_k<V, X, A, kDiaMax>(M, xx, yy, s);
}

// ---------------------------------------------------------------------------
// Y = A X for k right-hand sides (row-major).  A CTA walks a run of
// consecutive rows, for a chunk of at most 16 columns; a row's columns of the
// chunk lie on 2^lg consecutive lanes, VEC to a lane.  Walking in row order,
// the CTA finds the rows of X that its near diagonals share in L1: 128 bytes a
// row, and at each step only the outermost diagonals bring new ones.  (One
// warp per row over all columns, rows strided over the GPU, reads 5.5 rows of
// X from L2 per row on a 7-point stencil; this reads 3.2.)  The chunks of a
// run are neighbouring CTAs, so that whole rows of X come from HBM once.
// ---------------------------------------------------------------------------
//
// 100^3, k = 128 (2.14 GB): 431 us against 650 us; k = 33: 191 against 454;
// 500^2, k = 17: 29 against 109.  32-column chunks 537 us, 8-column 555;
// CTAs of 256 threads on 512-row runs 455 us, of 512 threads 484; 96- and
// 320-row runs 442 and 473 us.  What is left waits on X
// from L2: registers allow 28 of 64 warps per SM, and L1 holds 36 % of the
// loads.
template <int KC, bool CONST, int VEC>
__global__ void __launch_bounds__(kDiaBatchThreads)
    batch_dia_kernel(const DiaView<double> D, int ndiag, int32_t k, int lg, int chunk_cols, int nchunk,
                     int32_t run, const double* __restrict__ X, double* __restrict__ Y) {
    using M = DiaMask<KC>;
    const M* __restrict__ mask = static_cast<const M*>(D.mask);
    const double* __restrict__ val = static_cast<const double*>(D.val);
    const int chunk = blockIdx.x % nchunk;
    const int64_t r_begin = int64_t(blockIdx.x / nchunk) * run;
    const int64_t r_end = min(int64_t(D.n), r_begin + run);
    const int c = chunk * chunk_cols + (threadIdx.x & ((1 << lg) - 1)) * VEC;
    const bool in = c < min(k, (chunk + 1) * chunk_cols);
    const int step = kDiaBatchThreads >> lg;
    // Distances to the diagonals' rows of X and their values in registers.
    int64_t dist[KC];
    double cv[KC];
#pragma unroll
    for (int e = 0; e < KC; ++e) {
        dist[e] = int64_t(D.off[e]) * k;
        cv[e] = D.cval[e];
        asm volatile("" : "+l"(dist[e]));
        if constexpr (CONST) asm volatile("" : "+d"(cv[e]));
    }
    const uint32_t full_mask = (1u << ndiag) - 1u;
    int64_t row = r_begin + (threadIdx.x >> lg);
    const double* xp = X + row * k + c;
    double* yp = Y + row * k + c;
    const int64_t adv = int64_t(step) * k;
    uint32_t m = row < r_end && in ? mask[row] : 0u;
    for (; row - (threadIdx.x >> lg) < r_end; row += step, xp += adv, yp += adv) {
        double x[KC][VEC], v[KC];
        const uint32_t mc = m;
        const bool full = KC == ndiag && __all_sync(0xffffffffu, mc == full_mask);
        auto load = [&](int e) {
            if constexpr (VEC == 2) {
                const double2 t = __ldg(reinterpret_cast<const double2*>(xp + dist[e]));
                x[e][0] = t.x;
                x[e][1] = t.y;
            } else {
                x[e][0] = __ldg(xp + dist[e]);
            }
            v[e] = CONST ? cv[e] : __ldg(val + e * D.ld + row);
        };
        if (full) {
#pragma unroll
            for (int e = 0; e < KC; ++e) load(e);
        } else {
#pragma unroll
            for (int e = 0; e < KC; ++e)
                if (mc >> e & 1u) load(e);
        }
        m = row + step < r_end && in ? mask[row + step] : 0u;
        double acc[VEC];
#pragma unroll
        for (int q = 0; q < VEC; ++q) acc[q] = 0.0;
        if (full) {
#pragma unroll
            for (int e = 0; e < KC; ++e)
#pragma unroll
                for (int q = 0; q < VEC; ++q) acc[q] = add_rn(acc[q], mul_rn(v[e], x[e][q]));
        } else {
#pragma unroll
            for (int e = 0; e < KC; ++e)
                if (mc >> e & 1u) {
#pragma unroll
                    for (int q = 0; q < VEC; ++q) acc[q] = add_rn(acc[q], mul_rn(v[e], x[e][q]));
                }
        }
        if (in && row < r_end) {
            if constexpr (VEC == 2) *reinterpret_cast<double2*>(yp) = make_double2(acc[0], acc[1]);
            else yp[0] = acc[0];
        }
    }
}

// The same for more than 8 diagonals of which a row uses few (a periodic grid's
// wrap-around diagonals): a row's diagonals are taken from its mask, kDiaBits
// at a time, instead of asking each in turn.  Where rows have nearly all of
// them (mostly_full) the unrolled kernel takes those matrices too: 16
// varying diagonals, 300,000 rows, k = 9 1.4 times as fast, k = 63 1.7 times;
// with 0.6 of them there it is 0.9 times as fast.
constexpr int kDiaBits = 6;

template <bool CONST, int VEC>
__global__ void __launch_bounds__(kDiaBatchThreads)
    batch_dia_bits_kernel(const DiaView<double> D, int32_t k, int lg, int chunk_cols, int nchunk,
                          int32_t run, const double* __restrict__ X, double* __restrict__ Y) {
    __shared__ int64_t dist[kDiaMax];  // to the diagonal's row of X
    __shared__ double cv[kDiaMax];
    if (threadIdx.x < kDiaMax) {
        dist[threadIdx.x] = int64_t(D.off[threadIdx.x]) * k;
        cv[threadIdx.x] = D.cval[threadIdx.x];
    }
    __syncthreads();
    const uint16_t* __restrict__ mask = static_cast<const uint16_t*>(D.mask);
    const double* __restrict__ val = static_cast<const double*>(D.val);
    const int chunk = blockIdx.x % nchunk;
    const int64_t r_begin = int64_t(blockIdx.x / nchunk) * run;
    const int64_t r_end = min(int64_t(D.n), r_begin + run);
    const int c = chunk * chunk_cols + (threadIdx.x & ((1 << lg) - 1)) * VEC;
    if (c >= min(k, (chunk + 1) * chunk_cols)) return;
    const int step = kDiaBatchThreads >> lg;
    int64_t row = r_begin + (threadIdx.x >> lg);
    uint32_t m = row < r_end ? mask[row] : 0u;
    for (; row < r_end; row += step) {
        uint32_t left = m;
        m = row + step < r_end ? mask[row + step] : 0u;
        const double* xp = X + row * k + c;
        double acc[VEC];
#pragma unroll
        for (int q = 0; q < VEC; ++q) acc[q] = 0.0;
        while (left) {
            double x[kDiaBits][VEC], v[kDiaBits];
            const int cnt = __popc(left);
#pragma unroll
            for (int j = 0; j < kDiaBits; ++j)
                if (j < cnt) {
                    const int e = __ffs(left) - 1;
                    left &= left - 1u;
                    if constexpr (VEC == 2) {
                        const double2 t = __ldg(reinterpret_cast<const double2*>(xp + dist[e]));
                        x[j][0] = t.x;
                        x[j][1] = t.y;
                    } else {
                        x[j][0] = __ldg(xp + dist[e]);
                    }
                    v[j] = CONST ? cv[e] : __ldg(val + e * D.ld + row);
                }
#pragma unroll
            for (int j = 0; j < kDiaBits; ++j)
                if (j < cnt) {
#pragma unroll
                    for (int q = 0; q < VEC; ++q) acc[q] = add_rn(acc[q], mul_rn(v[j], x[j][q]));
                }
        }
        double* yp = Y + row * k + c;
        if constexpr (VEC == 2) *reinterpret_cast<double2*>(yp) = make_double2(acc[0], acc[1]);
        else yp[0] = acc[0];
    }
}

// Nearly every row has an entry on every diagonal (7 in 8).
bool mostly_full(const nm_csr* A) {
    return 8 * int64_t(A->nnz) >= 7 * int64_t(A->dia.ndiag) * A->nrows;
}

template <int KC, bool CONST, int VEC>
void launch_batch_dia_t(const nm_csr* A, const DiaBatchShape& b, const double* X, double* Y,
                        int32_t k, cudaStream_t s) {
    const auto D = dia_view<double>(A->dia, A->nrows);
    const unsigned g = static_cast<unsigned>(b.grid);
    if (KC > 8 && !mostly_full(A))
        batch_dia_bits_kernel<CONST, VEC><<<g, kDiaBatchThreads, 0, s>>>(
            D, k, b.lg, b.chunk_cols, b.nchunk, b.run, X, Y);
    else
        batch_dia_kernel<KC, CONST, VEC><<<g, kDiaBatchThreads, 0, s>>>(
            D, A->dia.ndiag, k, b.lg, b.chunk_cols, b.nchunk, b.run, X, Y);
}

template <int KC>
void launch_batch_dia_k(const nm_csr* A, const DiaBatchShape& b, const double* X, double* Y,
                        int32_t k, bool vec2, cudaStream_t s) {
    if (A->dia.constant) {
        if (vec2) launch_batch_dia_t<KC, true, 2>(A, b, X, Y, k, s);
        else launch_batch_dia_t<KC, true, 1>(A, b, X, Y, k, s);
    } else {
        if (vec2) launch_batch_dia_t<KC, false, 2>(A, b, X, Y, k, s);
        else launch_batch_dia_t<KC, false, 1>(A, b, X, Y, k, s);
    }
}

// The diagonals of some rows, on the host: a matrix of scattered columns shows
// more than kDiaMax there (false) and costs nothing more.  *varying: the looked
// at entries of a diagonal differ (where the values, of es bytes, are given).
bool look_at_rows(const int32_t* rp, const int32_t* ci, int32_t nrows, DiaSeed* seed,
                  const void* vals = nullptr, size_t es = 0, bool* varying = nullptr) {
    const char* v = static_cast<const char*>(vals);
    if (nrows == 0 || rp[nrows] == 0) return false;
    constexpr int kLook = 64;
    for (int q = 0; q < kLook; ++q) {
        const int32_t r = static_cast<int32_t>(int64_t(nrows - 1) * q / (kLook - 1));
        if (rp[r + 1] - rp[r] > kDiaMax) return false;
        for (int32_t z = rp[r]; z < rp[r + 1]; ++z) {
            const int32_t d = ci[z] - r;
            const int s = int(std::find(seed->off, seed->off + seed->count, d) - seed->off);
            if (s < seed->count) {
                if (v) *varying |= std::memcmp(v + es * z, v + es * seed->at[s], es) != 0;
                continue;
            }
            if (seed->count == kDiaMax) return false;
            seed->off[seed->count] = d;
            seed->at[seed->count++] = z;
        }
    }
    return true;
}

}  // namespace

bool may_be_diagonal(const int32_t* row_ptr, const int32_t* col_idx, const void* values,
                     size_t value_bytes, int32_t nrows, size_t* copy_bytes) {
    DiaSeed seed{};
    bool varying = false;
    const bool may =
        look_at_rows(row_ptr, col_idx, nrows, &seed, values, value_bytes, &varying);
    const int64_t nnz = nrows > 0 ? row_ptr[nrows] : 0;
    *copy_bytes = may && varying && 2 * nnz >= int64_t(seed.count) * nrows
                      ? value_bytes * size_t(seed.count) * size_t(dia_ld(nrows))
                      : 0;
    return may;
}

int search_dia_form(const nm_csr* A) {
    if (!A->d_dia_room) return NM_OK;
    DiaSeed seed{};
    look_at_rows(A->h_row_ptr.data(), A->h_col_idx.data(), A->nrows, &seed);
    switch (A->dtype) {
        case NM_F64: return launch_search<double>(A, seed);
        case NM_F32: return launch_search<float>(A, seed);
        default: return launch_search<__nv_bfloat16>(A, seed);
    }
}

int take_dia_form(nm_csr* A) {
    if (!A->d_dia_room) return NM_OK;
    switch (A->dtype) {
        case NM_F64: return take_form<double>(A);
        case NM_F32: return take_form<float>(A);
        default: return take_form<__nv_bfloat16>(A);
    }
}

int launch_spmv_dia(const nm_csr* A, const void* x, void* y, cudaStream_t s) {
    switch (A->dtype) {
        case NM_F64: return launch_dia_t<double, double, double>(A, x, y, s);
        case NM_F32: return launch_dia_t<float, float, float>(A, x, y, s);
        default: return launch_dia_t<__nv_bfloat16, float, float>(A, x, y, s);
    }
}

bool batch_on_diagonals(const nm_csr* A, int32_t k, bool vec2) {
    if (A->dia.ndiag == 0) return false;
    const int vec = vec2 ? 2 : 1;
    if (csr_batch_shape(k, vec).ch < 2) return true;
    return dia_batch_takes(A->nrows, A->dia.ndiag, mostly_full(A), A->dia.constant, k, vec,
                           dia_batch_shape(A->nrows, k, vec, sm_count()));
}

int launch_batch_dia(const nm_csr* A, const double* X, double* Y, int32_t k, bool vec2,
                     cudaStream_t s) {
    const int nd = A->dia.ndiag;
    const DiaBatchShape b = dia_batch_shape(A->nrows, k, vec2 ? 2 : 1, sm_count());
    if (b.grid > INT32_MAX) return fail(NM_ERR_INVALID, "batch_spmv: problem too large");
    if (nd <= 3) launch_batch_dia_k<3>(A, b, X, Y, k, vec2, s);
    else if (nd <= 5) launch_batch_dia_k<5>(A, b, X, Y, k, vec2, s);
    else if (nd <= 7) launch_batch_dia_k<7>(A, b, X, Y, k, vec2, s);
    else if (nd <= 8) launch_batch_dia_k<8>(A, b, X, Y, k, vec2, s);
    else if (nd <= 9) launch_batch_dia_k<9>(A, b, X, Y, k, vec2, s);
    else if (nd <= 12) launch_batch_dia_k<12>(A, b, X, Y, k, vec2, s);
    else launch_batch_dia_k<kDiaMax>(A, b, X, Y, k, vec2, s);
    NM_CHECK_LAUNCH();
    return NM_OK;
}

}  // namespace nm
