// Chunks of the inner products (sm_100a).  The order of the sums: lane sum l of
// a chunk of 256 rows is the fma chain over its rows l, l + 32, ..., l + 224,
// and the 32 lane sums fold pairwise, s[l] += s[l + off], off = 16 .. 1.
//
// A warp reads whole lines of the block vectors: TPR lanes per row with V
// columns each, RPI = 32 / TPR rows at a time.  The lane sums of a thread's rows
// (l = q + RPI j) fold by 16 .. RPI in the thread itself; taken in bit-reversed
// order of j they merge as they come, so log2(TPR) + 1 partial sums of V columns
// are held instead of NV.  What is left folds over the lanes of the rows.
//
// Bound: HBM.  One lane to a row read NV columns of a row by itself, 32 lines for
// a load (FP64, NV 16, 3 pairs of 6 vectors of 884736 rows: 177 us; now 106, 104 at
// the copy bandwidth), and on few rows a warp to a chunk was a chain of its loads
// (32768 rows, NV 16, the pairs of two vectors: 58 us; now 3.1 with a chunk split
// over 8 warps, NV 4 5.9 -> 2.4, NV 1 3.3 -> 2.0).
#pragma once
#include <algorithm>
#include <cstring>
#include "kernels.cuh"

namespace xk {

// V columns a lane: 16 bytes, 8 of FP32 vectors where the sums of several pairs
// would take too many registers (one pair, NV 8, 1500000 rows: 15.6 us, 18.5 with 8
// bytes a lane).  SPLIT: see DotSplit.
template <class TI, int NV, int ND> struct DotShape {
    static constexpr int V = NV == 1 ? 1 : NV >= 4 && ND == 1 && sizeof(TI) == 4 ? 4 : 2, TPR = NV / V, RPI = 32 / TPR;
    static constexpr bool SPLIT = TPR >= (ND == 1 ? 2 : 4);
    static constexpr int LOG = TPR == 1 ? 0 : TPR == 2 ? 1 : TPR == 4 ? 2 : TPR == 8 ? 3 : 4;
};

// Sums in a tree as they come: the i-th completes the pairs that its low bits close.
template <int LOG, int C> struct DotStack {
    double st[LOG > 0 ? LOG : 1][C];
    __device__ __forceinline__ void push(int i, double (&v)[C]) {
#pragma unroll
        for (int k = 0; k < LOG; ++k) {
            if (!((i >> k) & 1)) {
#pragma unroll
                for (int c = 0; c < C; ++c) st[k][c] = v[c];
                return;
            }
#pragma unroll
            for (int c = 0; c < C; ++c) v[c] = __dadd_rn(st[k][c], v[c]);
        }
    }
};

template <int LOG> __device__ __forceinline__ int dot_bitrev(int i) { return LOG == 0 ? 0 : (int)(__brev((unsigned)i) >> (32 - (LOG > 0 ? LOG : 1))); }

// folds over the lanes of the rows; the lanes of row 0 hold the chunk's sums
template <class S, int C> __device__ __forceinline__ void dot_fold_lanes(double (&v)[C]) {
    constexpr int TPR = S::TPR;
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
        for (int off = 16; off >= TPR; off >>= 1) v[c] = __dadd_rn(v[c], __shfl_xor_sync(0xffffffffu, v[c], off));
}

// The warps of a chunk (W of them, this one the sub-th; neighbours in the block)
// put their subtrees together in warp 0: false for the others.
template <class S, int C>
__device__ __forceinline__ bool dot_join(int W, int sub, double *sm, double (&v)[C]) {
    if (W == 1) return true;
    constexpr int LOG = S::LOG < 3 ? S::LOG : 3;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < C; ++c) sm[(warp * C + c) * 32 + lane] = v[c];
    __syncthreads();
    if (sub != 0) return false;
    DotStack<LOG, C> tree;
    for (int w = 0; w < W; ++w) {
#pragma unroll
        for (int c = 0; c < C; ++c) v[c] = sm[((warp + w) * C + c) * 32 + lane];
        tree.push(w, v);
    }
    return true;
}

// AL: p lies on a boundary of the loads, min(16, V * sizeof(TI)) bytes
template <class TI, int V, bool AL> __device__ __forceinline__ void dot_ld(const TI *p, TI (&r)[V]) {
    if constexpr (V == 1 || !AL) {
#pragma unroll
        for (int e = 0; e < V; ++e) r[e] = __ldg(p + e);
    } else if constexpr (sizeof(TI) == 8) {
#pragma unroll
        for (int e = 0; e < V; e += 2) {
            const double2 w = __ldg(reinterpret_cast<const double2 *>(p + e));
            r[e] = w.x, r[e + 1] = w.y;
        }
    } else if constexpr (V == 4) {
        const float4 w = __ldg(reinterpret_cast<const float4 *>(p));
        r[0] = w.x, r[1] = w.y, r[2] = w.z, r[3] = w.w;
    } else {
        const float2 w = __ldg(reinterpret_cast<const float2 *>(p));
        r[0] = w.x, r[1] = w.y;
    }
}

// This thread's part of ND pairs over the cnt <= 256 rows from row0, the subtree
// `sub` of W.  SH: the pairs are (a, b), (a, a), (b, b) of two vectors.
template <class TI, int NV, int ND, bool SH, bool AL = true>
__device__ __forceinline__ void dot_chunk(const TI *const (&A)[ND], const TI *const (&B)[ND], i64 row0, int cnt, int W,
                                          int sub, double (&out)[ND * DotShape<TI, NV, ND>::V]) {
    typedef DotShape<TI, NV, ND> S;
    constexpr int V = S::V, C = ND * V, B8 = sizeof(TI) * V <= 8 ? 2 : 1;
    constexpr int U = S::TPR == 1 ? (V == 4 || (NV == 1 && ND >= 3) ? 4 : 8) : (SH || ND == 1 ? 4 : 2) * B8;  // rows of a sum in flight
    const int lane = threadIdx.x & 31, q = lane / S::TPR, k0 = lane % S::TPR * V, JW = S::TPR / W;
    DotStack<S::LOG, C> tree;
#pragma unroll 1
    for (int i = 0; i < JW; ++i) {
        const int r = dot_bitrev<S::LOG>(sub * JW + i) * S::RPI + q;
        const i64 o = (row0 + r) * NV + k0;
#pragma unroll
        for (int c = 0; c < C; ++c) out[c] = 0.0;
        if (cnt == 256) {
#pragma unroll
            for (int m = 0; m < 8; m += U) {
                TI a[U][SH ? 1 : ND][V], b[U][SH ? 1 : ND][V];
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int d = 0; d < (SH ? 1 : ND); ++d) {
                        dot_ld<TI, V, AL>(A[d] + o + (m + u) * 32 * NV, a[u][d]);
                        dot_ld<TI, V, AL>(B[d] + o + (m + u) * 32 * NV, b[u][d]);
                    }
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int d = 0; d < ND; ++d)
#pragma unroll
                        for (int e = 0; e < V; ++e) {
                            const TI x = SH ? (d == 2 ? b[u][0][e] : a[u][0][e]) : a[u][SH ? 0 : d][e];
                            const TI y = SH ? (d == 1 ? a[u][0][e] : b[u][0][e]) : b[u][SH ? 0 : d][e];
                            out[d * V + e] = fma((double)x, (double)y, out[d * V + e]);
                        }
            }
        } else {
            for (int m = 0; m < 8 && r + 32 * m < cnt; ++m)
#pragma unroll
                for (int d = 0; d < ND; ++d) {
                    TI a[V], b[V];
                    dot_ld<TI, V, AL>(A[d] + o + m * 32 * NV, a);
                    dot_ld<TI, V, AL>(B[d] + o + m * 32 * NV, b);
#pragma unroll
                    for (int e = 0; e < V; ++e) out[d * V + e] = fma((double)a[e], (double)b[e], out[d * V + e]);
                }
        }
        tree.push(i, out);
    }
}

// Warps per chunk (W) and per block.  Below 16 warps per SM chunks are split, as
// far as a warp has several sums, and spread over the SMs (unsplit, 4096 rows of NV
// 16 are 16 warps with 64 loads in turn each).  Operands beyond L2 are split too
// where a row has four lanes or more, or two for one pair: the warps of a chunk then
// read lines next to each other at the same time (us, split and not: one pair, FP64
// NV 16 1000000 rows 43.6 and 46.5, NV 8 3000000 rows 64 and 73, NV 4 35.8 and 37.8,
// FP32 NV 32 600000 rows 31 and 42; two pairs, FP64 NV 4 1000000 rows 24.9 and 24.3;
// in L2, FP32 NV 16 600000 rows, 12.2 and 12.0).  Blocks of four warps start and end more
// evenly than of eight (FP64 NV 1 600000 rows 5.67 and 5.92, FP32 NV 1, three pairs,
// 3000000 rows 15.2 and 16.4).
struct DotSplit {
    int W, warps;
    unsigned blocks;
};
template <class S> inline DotSplit dot_split(i64 nch, int sms, i64 bytes, int block) {
    DotSplit s;
    s.W = 1;
    while (s.W < 8 && s.W < S::TPR && (nch * s.W < 16 * (i64)sms || (S::SPLIT && bytes > 110000000))) s.W *= 2;
    s.warps = nch * s.W >= 4 * (i64)sms ? std::max(s.W, block) : s.W;
    s.blocks = (unsigned)((nch * s.W + s.warps - 1) / s.warps);
    return s;
}

}  // namespace xk
