// dia.cuh -- matrices whose nonzeros lie on few diagonals, in diagonal form.
//
// A stencil's nonzeros sit on a handful of diagonals col - row = off[k].  When
// every row's columns ascend (so that a row's CSR order is the order of its
// diagonals) and the whole matrix has at most kDiaMax of them, a row is its
// bits in a mask (bit k: the row has an entry on diagonal k) and its values:
// no column index and no row offset is read.  The values are stored diagonal
// by diagonal, val[k * ld + row], so that a warp's 32 rows read them with one
// coalesced load per diagonal and nothing is staged; absent entries take room
// there but are never read.  Where all entries of each diagonal are the same
// number (the constant-coefficient Laplacians) there is no value array at all.
//
// A row's sum is formed entry by entry in ascending diagonal order with
// unfused multiply and add, over the present entries only: the operations of
// the row-block kernel's thread rows (and of the reference's serial row loop,
// src/spmv_kernel.hpp:90-97), so the same bits.
#pragma once

#include "csr.cuh"

namespace nm {

// Kernel-side view: offsets and constant values by value.
template <typename A>
struct DiaView {
    int32_t n;  // rows
    int64_t ld;
    int32_t off[kDiaMax];
    A cval[kDiaMax];   // the diagonals' values (constant form)
    const void* mask;  // uint8_t up to 8 diagonals, else uint16_t
    const void* val;   // V[ndiag][ld] (unused in the constant form)
};

// The mask type of a kernel compiled for up to KC diagonals.
template <int KC>
using DiaMask = std::conditional_t<(KC <= 8), uint8_t, uint16_t>;

template <typename A>
DiaView<A> dia_view(const DiaForm& f, int32_t nrows) {
    DiaView<A> D{};
    D.n = nrows;
    D.ld = f.ld;
    for (int k = 0; k < kDiaMax; ++k) {
        D.off[k] = f.off[k];
        D.cval[k] = static_cast<A>(f.cval[k]);
    }
    D.mask = f.d_mask;
    D.val = f.d_val;
    return D;
}

}  // namespace nm
