// Columns of a hybrid block's entries as k_gs_block (gs.cu) uses them.  Its loads
// run past an item's end, where the stage holds other items' columns or values,
// so a column may be any 32-bit word until it is clamped.  Plain C++, so that the
// rule can be checked on the host.
#pragma once

#ifdef __CUDACC__
#define XK_HD __host__ __device__ __forceinline__
#else
#define XK_HD inline
#endif

namespace xk {

// rows of block b (the last one may be short)
XK_HD int gs_block_rows(int n, int brows, int b) {
    const int left = n - b * brows;
    return left < brows ? left : brows;
}
// column word -> row of the block, or lim for everything else (a row of zeros:
// padding entries, whose column is one past a full block, read it too)
XK_HD int gs_block_column(int word, int lim) {
    return (unsigned)word < (unsigned)lim ? word : lim;
}

}  // namespace xk
