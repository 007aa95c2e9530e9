// Gauss-Seidel sweeps over a level-ordered copy of the matrix (sm_100a).
//
// The rows are stored level by level (block by block for hybrid plans), a
// level's rows cut into items of at most one warp (see GsDir).  Warps take the
// items in order, round robin, so while one warp computes a level the others
// already hold the entries, t and old x of the next levels.
//
//   k_gs_block : one CTA per hybrid block (or one CTA for a whole narrow
//                schedule), forward and backward sweep in one launch.  The
//                block's x tile is held in shared memory when it fits (XS),
//                else x is read through the L1; a ring of mbarriers says
//                which levels are complete.
//   k_gs_flow  : one single-process sweep on the whole device (cooperative
//                launch).  New values go to a second vector that the
//                launcher has filled with a sentinel; a row that needs one
//                reads it until it is there, so there is no flag, fence or
//                barrier between two levels.
//
// What bounds them is the chain from level to level: the arrival of the
// previous level's values, the rest of the row's FMA chain, the store (k_gs_block
// on 80^3 in 444 blocks: DRAM at 12 % of its rate, L1 39 %, issue 31 %).  Measured
// (B200, both sweeps of one call, 27-point operators; before: one CTA barrier,
// TMA wait and gather per level):
//   k_gs_block FP32 NV=16, 444 blocks   64^3 227 -> 113 us, 80^3 367 -> 244 us
//              FP32 NV=16, 148 blocks   64^3 336 -> 111 us
//              FP64 NV=4, one CTA       12^3 483 -> 128 us
//   k_gs_flow  FP64 NV=8                48^3 2320 -> 1204 us
//              FP64 NV=1, 7-point       40^3 793 -> 237 us
// Found on the way: a predicate or branch per entry (row ends, padding) costs
// more than the entry; selecting between two shared pointers makes generic
// loads of them; lanes of 8 bytes (half the FMAs a lane, twice the items) lose
// 40 % because a warp's own instruction stream is what a level waits for; a
// nanosleep or a single polling lane changes nothing.
//
// Every wait is bounded by a wall-clock limit; on expiry the error word is set
// and the CTA leaves after its own copies in flight have landed.
#include "gs_columns.h"
#include "kernels.cuh"
#include <algorithm>
#include <climits>
#include <cstdio>

namespace xk {

namespace {

constexpr unsigned long long kLimitNs = kGsWaitNs;

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned smem_u32(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

// 16-byte global -> shared copy, tracked per thread
__device__ __forceinline__ void cp_async16_cg(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait_group() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }

template <class T, int V> struct VW;
template <> struct VW<double, 1> { typedef double t; };
template <> struct VW<double, 2> { typedef double2 t; };
template <> struct VW<float, 1> { typedef float t; };
template <> struct VW<float, 2> { typedef float2 t; };
template <> struct VW<float, 4> { typedef float4 t; };

// A lane owns 16 bytes of a row (V columns), TPR lanes a row.
template <class T, int NV> struct Sh {
    static constexpr int V = (NV * (int)sizeof(T) >= 16) ? 16 / (int)sizeof(T) : NV;
    static constexpr int TPR = NV / V;
};

template <class T, int V>
__device__ __forceinline__ void vld(const T *p, T (&r)[V]) {
    typedef typename VW<T, V>::t W;
    W w = *reinterpret_cast<const W *>(p);
    memcpy(r, &w, sizeof(W));
}
template <class T, int V>
__device__ __forceinline__ void vldg(const T *p, T (&r)[V]) {
    typedef typename VW<T, V>::t W;
    W w = __ldg(reinterpret_cast<const W *>(p));
    memcpy(r, &w, sizeof(W));
}
template <class T, int V>
__device__ __forceinline__ void vst(T *p, const T (&r)[V]) {
    typedef typename VW<T, V>::t W;
    W w;
    memcpy(&w, r, sizeof(W));
    *reinterpret_cast<W *>(p) = w;
}

// loads and stores of values that other CTAs write or read during the launch
__device__ __forceinline__ void rld(const float *p, float (&r)[1]) {
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(r[0]) : "l"(p) : "memory");
}
// r = new value (read past the L1) where fresh, else the old one (read-only path)
__device__ __forceinline__ void ld2(bool fresh, const double *pn, const double *po, double (&r)[1]) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q ld.relaxed.gpu.global.f64 %0, [%1];\n"
                 " @!q ld.global.nc.f64 %0, [%2];\n}" : "=d"(r[0]) : "l"(pn), "l"(po), "r"((int)fresh) : "memory");
}
__device__ __forceinline__ void ld2(bool fresh, const float *pn, const float *po, float (&r)[1]) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q ld.relaxed.gpu.global.f32 %0, [%1];\n"
                 " @!q ld.global.nc.f32 %0, [%2];\n}" : "=f"(r[0]) : "l"(pn), "l"(po), "r"((int)fresh) : "memory");
}
__device__ __forceinline__ void ld2(bool fresh, const float *pn, const float *po, float (&r)[2]) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %4, 0;\n @q ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];\n"
                 " @!q ld.global.nc.v2.f32 {%0, %1}, [%3];\n}"
                 : "=f"(r[0]), "=f"(r[1]) : "l"(pn), "l"(po), "r"((int)fresh) : "memory");
}
__device__ __forceinline__ void ld2(bool fresh, const double *pn, const double *po, double (&r)[2]) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %4, 0;\n @q ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];\n"
                 " @!q ld.global.nc.v2.f64 {%0, %1}, [%3];\n}"
                 : "=d"(r[0]), "=d"(r[1]) : "l"(pn), "l"(po), "r"((int)fresh) : "memory");
}
__device__ __forceinline__ void ld2(bool fresh, const float *pn, const float *po, float (&r)[4]) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %6, 0;\n @q ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                 " @!q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%5];\n}"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]) : "l"(pn), "l"(po), "r"((int)fresh) : "memory");
}
// the new value once more where on, without a branch
__device__ __forceinline__ void rld_on(bool on, const double *p, double (&r)[2]) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];\n}"
                 : "+d"(r[0]), "+d"(r[1]) : "l"(p), "r"((int)on) : "memory");
}
__device__ __forceinline__ void rld_on(bool on, const float *p, float (&r)[4]) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %5, 0;\n @q ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];\n}"
                 : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]) : "l"(p), "r"((int)on) : "memory");
}
__device__ __forceinline__ void rld_on(bool on, const double *p, double (&r)[1]) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q ld.relaxed.gpu.global.f64 %0, [%1];\n}"
                 : "+d"(r[0]) : "l"(p), "r"((int)on) : "memory");
}
__device__ __forceinline__ void rld_on(bool on, const float *p, float (&r)[1]) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q ld.relaxed.gpu.global.f32 %0, [%1];\n}"
                 : "+f"(r[0]) : "l"(p), "r"((int)on) : "memory");
}
__device__ __forceinline__ void rld_on(bool on, const float *p, float (&r)[2]) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];\n}"
                 : "+f"(r[0]), "+f"(r[1]) : "l"(p), "r"((int)on) : "memory");
}
__device__ __forceinline__ void rst(double *p, const double (&r)[1]) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(r[0]) : "memory");
}
__device__ __forceinline__ void rst(double *p, const double (&r)[2]) {
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(r[0]), "d"(r[1]) : "memory");
}
__device__ __forceinline__ void rst(float *p, const float (&r)[4]) {
    asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(r[0]), "f"(r[1]), "f"(r[2]),
                 "f"(r[3])
                 : "memory");
}
__device__ __forceinline__ void rst(float *p, const float (&r)[1]) {
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(r[0]) : "memory");
}
__device__ __forceinline__ void rst(float *p, const float (&r)[2]) {
    asm volatile("st.relaxed.gpu.global.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(r[0]), "f"(r[1]) : "memory");
}

// the value that marks an element of the output vector as not yet written: the
// bit pattern the launcher's memset leaves (a NaN); a result that happens to
// have it is stored as another NaN
__device__ __forceinline__ bool unwritten(double v) { return __double_as_longlong(v) == -1ll; }
__device__ __forceinline__ bool unwritten(float v) { return __float_as_int(v) == -1; }
__device__ __forceinline__ double written(double v) { return unwritten(v) ? __longlong_as_double(0x7ff8000000000000ll) : v; }
__device__ __forceinline__ float written(float v) { return unwritten(v) ? __int_as_float(0x7fc00000) : v; }

// shared-memory loads by 32-bit address
__device__ __forceinline__ void xls(unsigned a, float (&r)[4]) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]) : "r"(a));
}
__device__ __forceinline__ void xls(unsigned a, double (&r)[2]) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(r[0]), "=d"(r[1]) : "r"(a));
}
__device__ __forceinline__ void xls(unsigned a, float (&r)[1]) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r[0]) : "r"(a));
}
__device__ __forceinline__ void xls(unsigned a, float (&r)[2]) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(r[0]), "=f"(r[1]) : "r"(a));
}
__device__ __forceinline__ void xls(unsigned a, double (&r)[1]) {
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(r[0]) : "r"(a));
}
// the same through the L1 (stores of this CTA update it)
__device__ __forceinline__ void xlg(const void *a, float (&r)[4]) {
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]) : "l"(a));
}
__device__ __forceinline__ void xlg(const void *a, double (&r)[2]) {
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(r[0]), "=d"(r[1]) : "l"(a));
}
__device__ __forceinline__ void xlg(const void *a, float (&r)[1]) {
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(r[0]) : "l"(a));
}
__device__ __forceinline__ void xlg(const void *a, float (&r)[2]) {
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(r[0]), "=f"(r[1]) : "l"(a));
}
__device__ __forceinline__ void xlg(const void *a, double (&r)[1]) {
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(r[0]) : "l"(a));
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned cnt) {
    asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(cnt) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar, unsigned cnt) {
    asm volatile("mbarrier.arrive.release.cta.shared.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(cnt) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned long long *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cta.shared.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait on an mbarrier phase; false on expiry (then, or when another
// warp's wait has expired, *fail is set)
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity, volatile int *fail,
                                          unsigned long long limit) {
    if (mbar_try(bar, parity)) return true;
    const unsigned long long t0 = now_ns();
    unsigned spins = 0;
    while (!mbar_try(bar, parity)) {
        if ((++spins & 15) == 0) {
            if (*fail) return false;
            if (now_ns() - t0 > limit) {
                *fail = 1;
                return false;
            }
        }
    }
    return true;
}

// One item: `rows` rows of one level (level-ordered rows r0 ..), all padded to
// `groups` groups of four entries; k0: the groups before the first one in which a
// row reads the previous level; extra: arrivals on the level's barrier beyond the
// item's own.
struct Item {
    int r0, level, extra, packed;
    __device__ __forceinline__ int rows() const { return packed & 63; }
    __device__ __forceinline__ int k0() const { return packed >> 8 & 255; }
    __device__ __forceinline__ int groups() const { return (int)((unsigned)packed >> 16); }
    __device__ __forceinline__ int entries() const { return 4 * groups() * rows(); }
};
__device__ __forceinline__ Item item_get(const int4 *items, int it, int end) {
    if (it >= end) return Item{0, 0, 0, 0};
    const int4 a = __ldg(items + it);
    return Item{a.x, a.y, a.z, a.w};
}

// This lane's row of an item, q counted in the item (lanes past its rows repeat
// the last one; they read but never write).  Only loads: nothing here waits.
template <class T> struct LaneRow {
    int row, e0;  // row id, the item's first entry
    T di;
};
template <class T>
__device__ __forceinline__ LaneRow<T> lane_row(const Item &a, const GsDir &d, int q) {
    const int p = a.r0 + max(min(q, a.rows() - 1), 0);
    const int4 w = __ldg(d.meta + p);
    if constexpr (sizeof(T) == 4) return LaneRow<T>{w.x, w.y, __int_as_float(w.w)};
    else return LaneRow<T>{w.x, w.y, __ldg(reinterpret_cast<const T *>(d.linvd) + p)};
}

// the warp's copy of entries [e0, e0 + ne) into its stage (eb entries: columns,
// then values); one cp.async group whether or not they fit
template <class T>
__device__ __forceinline__ void stage_entries(int e0, int ne, int eb, unsigned char *buf, const int *lci, const T *lva,
                                              int lane) {
    if (ne <= eb) {
        int *sc = reinterpret_cast<int *>(buf);
        T *sv = reinterpret_cast<T *>(buf + (size_t)eb * 4);
        for (int k = lane * 4; k < ne; k += 128) cp_async16_cg(sc + k, lci + e0 + k);
        constexpr int PER = 16 / (int)sizeof(T);
        for (int k = lane * PER; k < ne; k += 32 * PER) cp_async16_cg(sv + k, lva + e0 + k);
    }
    cp_async_commit();
}

// One group of row q of a staged item of R rows: columns or values in pieces of
// 16 bytes, [group][piece][row], so that the rows of a warp read neighbouring
// banks; a: the address of the group's piece 0 of row q, r16 = 16 R.
__device__ __forceinline__ void lds4(unsigned a, unsigned, int (&c)[4]) {
    asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a));
}
__device__ __forceinline__ void lds4(unsigned a, unsigned, float (&v)[4]) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(a));
}
__device__ __forceinline__ void lds4(unsigned a, unsigned r16, double (&v)[4]) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[2 * h]), "=d"(v[2 * h + 1]) : "r"(a + h * r16));
}

// the row of zeros that padding entries (value +0) read where x is
// in global memory: fma(-0, +0, s) == s for every s
__device__ __align__(16) double g_zero_row[32];

}  // namespace

// ---------------------------------------------------------------- one CTA per block
// Levels are published through a ring of mbarriers: level L completes phase
// L / kRing of barrier L % kRing once its items have arrived (once each, the last
// one also for the items that the block's widest level has more).  A warp
// holds one item at a time and the items in flight are consecutive, so no
// warp waits on a level more than NT / 32 ahead of the completed ones and the
// ring's parities are unambiguous.
constexpr int kRing = 32;
// reads past the last stage: three groups of 32 rows of FP64 values
constexpr int kStageSlack = 3 * 32 * 32;

template <class T, int NV, bool XS, int NT>
__global__ void __launch_bounds__(NT, 512 / NT) k_gs_block(const __grid_constant__ GsDir fw,
                                                                   const __grid_constant__ GsDir bw,
                                                                   const T *__restrict__ t, T *x,
                                                                   const T *__restrict__ relax, int brows, int n,
                                                                   int eb, int split, unsigned long long limit,
                                                                   int *err) {
    constexpr int V = Sh<T, NV>::V, TPR = Sh<T, NV>::TPR, RPW = 32 / TPR, W = NT / 32;
    static_assert(W + 2 <= kRing, "ring parities");
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ __align__(8) unsigned long long s_bar[2][kRing];
    __shared__ volatile int s_fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q = lane / TPR, l = lane % TPR;
    const int b = blockIdx.x;
    const int xb = b * brows;  // first row of the block
    // what a column may be at most: with the x tile one past a full block (its row
    // of zeros), else one past the rows that this block has
    const int lim = XS ? brows : gs_block_rows(n, brows, b);
    const int stage_bytes = eb * (4 + (int)sizeof(T));
    unsigned char *sbuf = dyn + (size_t)warp * 2 * stage_bytes;
    const unsigned sba = smem_u32(sbuf);
    T *xs = reinterpret_cast<T *>(dyn + (size_t)W * 2 * stage_bytes + kStageSlack);
    if (XS) {
        const int cnt = min(brows, n - xb) * NV;
        const T *xg = x + (size_t)xb * NV;
        for (int k = tid * V; k < cnt; k += NT * V) {
            T w[V];
            vld<T, V>(xg + k, w);
            vst<T, V>(xs + k, w);
        }
        for (int k = tid; k < NV; k += NT) xs[(size_t)brows * NV + k] = T(0);  // the row of zeros
    }
    if (tid < 2 * kRing) mbar_init(&s_bar[0][0] + tid, (unsigned)__ldg((tid < kRing ? fw : bw).imax + b) << split);
    if (tid == 0) {
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    T rl[V];
#pragma unroll
    for (int e = 0; e < V; ++e) rl[e] = relax[l * V + e];
    __syncthreads();
    // x of column c of the block (lim: a row of zeros), this lane's columns: a
    // column becomes a shared-memory address (XS), or stays a column
    constexpr int RB = NV * (int)sizeof(T);
    const unsigned xsa = smem_u32(xs) + l * V * (int)sizeof(T);
    const char *xga = reinterpret_cast<const char *>(x + (size_t)xb * NV + l * V);
    const char *zga = reinterpret_cast<const char *>(g_zero_row) + l * V * sizeof(T);
    auto where = [&](int c) -> int { return XS ? (int)(xsa + (unsigned)c * RB) : c; };
    auto xld = [&](int w, T(&r)[V]) {
        if constexpr (XS) xls((unsigned)w, r);
        else xlg(w < lim ? xga + (size_t)w * RB : zga, r);
    };
    for (int pass = 0; pass < 2; ++pass) {
        const GsDir &d = pass ? bw : fw;
        const T *lva = reinterpret_cast<const T *>(d.lva);
        unsigned long long *bar = s_bar[pass];
        if (pass) __syncthreads();
        // an item is taken by 1 << split warps, each with RPW of its rows
        const int end = __ldg(d.bitem + b + 1) << split;
        int it = (__ldg(d.bitem + b) << split) + warp;
        auto get = [&](int k) { return item_get(d.items, k < end ? k >> split : 0, k < end ? INT_MAX : 0); };
        auto rowq = [&](int k) { return (k & ((1 << split) - 1)) * RPW + q; };
        // three items ahead: the descriptor; two: the lane's row; one: its t
        // and its entries
        Item a = get(it), a1 = get(it + W), a2 = get(it + 2 * W);
        LaneRow<T> r = lane_row<T>(a, d, rowq(it)), r1 = lane_row<T>(a1, d, rowq(it + W));
        stage_entries<T>(r.e0, a.entries(), eb, sbuf, d.lci, lva, lane);
        T tv[V];
        vldg<T, V>(t + (size_t)r.row * NV + l * V, tv);
        int cur = 0;
        for (; it < end; it += W) {
            stage_entries<T>(r1.e0, a1.entries(), eb, sbuf + (size_t)(cur ^ 1) * stage_bytes, d.lci, lva, lane);
            T t1[V];
            vldg<T, V>(t + (size_t)r1.row * NV + l * V, t1);
            const LaneRow<T> r2 = lane_row<T>(a2, d, rowq(it + 2 * W));
            const Item a3 = get(it + 3 * W);
            T sum[V], xo[V];
#pragma unroll
            for (int e = 0; e < V; ++e) sum[e] = tv[e];
            cp_async_wait_group<1>();
            __syncwarp();
            // shared-memory addresses of this row's columns and values
            const int rows = a.rows(), qi = rowq(it), ne = a.entries();
            const bool mine = qi < rows;
            const unsigned sa = sba + (unsigned)(cur * stage_bytes), r16 = 16u * rows;
            const unsigned ca = sa + 16u * min(qi, rows - 1), va = ca + 4u * eb;
            auto ldc = [&](int g, int (&c)[4]) {
                lds4(ca + r16 * g, r16, c);
#pragma unroll
                for (int u = 0; u < 4; ++u) c[u] = where(gs_block_column(c[u], lim));
            };
            auto ldv = [&](int g, T(&v)[4]) { lds4(va + (unsigned)(sizeof(T) / 4) * r16 * g, r16, v); };
            auto ldx = [&](const int (&c)[4], T(&xv)[4][V]) {
#pragma unroll
                for (int u = 0; u < 4; ++u) xld(c[u], xv[u]);
            };
            auto chain = [&](const T(&v)[4], const T(&xv)[4][V]) {
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int e = 0; e < V; ++e) sum[e] = fma(-v[u], xv[u][e], sum[e]);
            };
            T v0[4], v1[4], x0[4][V], x1[4][V];
            int c0[4], c1[4];
            const unsigned lev = (unsigned)a.level;
            bool ok = true;
            // Segments of the rows, one copy of the code for all of them: the
            // groups before the item's first fresh one (in which a row reads the
            // previous level), which need only the levels before that, and the
            // rest; or, of a row longer than the stage, eb entries at a time.
            const bool longrow = ne > eb;
            const int k0 = longrow ? 0 : a.k0();
            int done = 0;  // long row: entries summed
            if (lev > 1 && !longrow) ok = mbar_wait(bar + (lev - 2) % kRing, (lev - 2) / kRing & 1, &s_fail, limit);
            xld(where(r.row - xb), xo);  // only this row's own item writes it
            int g = 0, g1 = k0 > 0 ? k0 : a.groups();
            bool last = k0 == 0;
            for (;;) {
                if (longrow) {
                    const int cnt = min(eb, ne - done);
                    __syncwarp();
                    stage_entries<T>(r.e0 + done, cnt, eb, sbuf + (size_t)cur * stage_bytes, d.lci, lva, lane);
                    cp_async_wait_all();
                    __syncwarp();
                    done += cnt;
                    last = done == ne;
                    g = 0;
                    g1 = cnt >> 2;
                }
                // before the wait: the first two groups' addresses.  Loads run up
                // to three groups past the segment's end (their columns are whatever
                // the stage holds there, clamped to the block's own rows, and nothing
                // uses them), so that the loop has one branch a group.
                ldc(g, c0);
                ldc(g + 1, c1);
                if (last || longrow)
                    if (lev > 0) ok = ok && mbar_wait(bar + (lev - 1) % kRing, (lev - 1) / kRing & 1, &s_fail, limit);
                // one verdict for the warp: its lanes leave together or not at all
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                ldx(c0, x0);
                ldx(c1, x1);
                ldv(g, v0);
                while (g < g1) {
                    ldv(g + 1, v1);
                    ldc(g + 2, c0);
                    chain(v0, x0);
                    if (++g >= g1) break;
                    ldx(c0, x0);
                    ldv(g + 1, v0);
                    ldc(g + 2, c1);
                    chain(v1, x1);
                    ldx(c1, x1);
                    ++g;
                }
                if (last) break;
                if (!longrow) {
                    g = k0;
                    g1 = a.groups();
                    last = true;
                }
            }
            if (!ok) break;
            if (mine) {
#pragma unroll
                for (int e = 0; e < V; ++e) xo[e] = fma(rmul(rl[e], r.di), sum[e], xo[e]);
                if (XS) vst<T, V>(xs + (r.row - xb) * NV + l * V, xo);
                else vst<T, V>(x + (size_t)r.row * NV + l * V, xo);
            }
            __syncwarp();
            if (lane == 0) {
                const bool lastsub = ((it + 1) & ((1 << split) - 1)) == 0;
                mbar_arrive(bar + lev % kRing, 1u + (lastsub ? (unsigned)a.extra << split : 0u));
            }
            if (XS && pass && mine) vst<T, V>(x + (size_t)r.row * NV + l * V, xo);
            a = a1;
            a1 = a2;
            a2 = a3;
            r = r1;
            r1 = r2;
#pragma unroll
            for (int e = 0; e < V; ++e) tv[e] = t1[e];
            cur ^= 1;
        }
        cp_async_wait_all();
    }
    __syncthreads();
    if (tid == 0 && s_fail) atomicExch(err, 1);
}

// ---------------------------------------------------------------- one sweep, whole device
// xin: the values before the sweep; xout: the sentinel everywhere, each row
// written once.  Row i reads xout for the columns the sweep has passed
// (c < i forward, c > i backward) and xin for the others.
template <class T, int NV>
__global__ void __launch_bounds__(256, 1) k_gs_flow(const __grid_constant__ GsDir d, int nitems, int forward,
                                                    const T *__restrict__ t, const T *__restrict__ xin, T *xout,
                                                    const T *__restrict__ relax, int n, int eb, int split, int *err) {
    constexpr int V = Sh<T, NV>::V, TPR = Sh<T, NV>::TPR, RPW = 32 / TPR, W = 8;
    extern __shared__ __align__(128) unsigned char dyn[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q = lane / TPR, l = lane % TPR;
    const int step = W * gridDim.x;
    const int stage_bytes = eb * (4 + (int)sizeof(T));
    unsigned char *sbuf = dyn + (size_t)warp * 2 * stage_bytes;
    const unsigned sba = smem_u32(sbuf);
    const T *lva = reinterpret_cast<const T *>(d.lva);
    T rl[V];
#pragma unroll
    for (int e = 0; e < V; ++e) rl[e] = relax[l * V + e];
    const int end = nitems << split;
    int it = warp * gridDim.x + blockIdx.x;
    auto get = [&](int k) { return item_get(d.items, k < end ? k >> split : 0, k < end ? INT_MAX : 0); };
    auto rowq = [&](int k) { return (k & ((1 << split) - 1)) * RPW + q; };
    Item a = get(it), a1 = get(it + step), a2 = get(it + 2 * step);
    LaneRow<T> r = lane_row<T>(a, d, rowq(it)), r1 = lane_row<T>(a1, d, rowq(it + step));
    stage_entries<T>(r.e0, a.entries(), eb, sbuf, d.lci, lva, lane);
    int cur = 0;
    for (; it < end; it += step) {
        stage_entries<T>(r1.e0, a1.entries(), eb, sbuf + (size_t)(cur ^ 1) * stage_bytes, d.lci, lva, lane);
        const LaneRow<T> r2 = lane_row<T>(a2, d, rowq(it + 2 * step));
        const Item a3 = get(it + 3 * step);
        T sum[V], xo[V];
        vldg<T, V>(t + (size_t)r.row * NV + l * V, sum);
        vldg<T, V>(xin + (size_t)r.row * NV + l * V, xo);
        cp_async_wait_group<1>();
        __syncwarp();
        const int rows = a.rows(), qi = rowq(it), ne = a.entries();
        const bool mine = qi < rows;
        const unsigned sa = sba + (unsigned)(cur * stage_bytes), r16 = 16u * rows;
        const unsigned ca = sa + 16u * min(qi, rows - 1), va = ca + 4u * eb;
        // a window of eight groups in registers: all their loads are under way
        // before the first wait, and a group is replaced by the one eight
        // further on as soon as it is summed
        T x[8][4][V];
        unsigned pend = 0;  // bit 4 k + u: entry u of window group k was not there when last read
        unsigned cw = ca, vw = va;
        auto issue = [&](int k, int g) {
            int c[4];
            lds4(cw + r16 * g, r16, c);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool fresh = c[u] < n && (forward ? c[u] < r.row : c[u] > r.row);
                const size_t o = (size_t)c[u] * NV + l * V;
                ld2(fresh, xout + o, c[u] < n ? xin + o : reinterpret_cast<const T *>(g_zero_row) + l * V, x[k][u]);
                pend |= (unsigned)fresh << (4 * k + u);
            }
        };
        // window group k (group g of the rows) once more where it was not there
        auto look = [&](int k, int g) {
            int c[4];
            lds4(cw + r16 * g, r16, c);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const unsigned bit = 1u << (4 * k + u);
                bool miss = false;
#pragma unroll
                for (int e = 0; e < V; ++e) miss |= unwritten(x[k][u][e]);
                miss = miss && (pend & bit);
                if (!miss) pend &= ~bit;
                rld_on(miss, xout + (size_t)c[u] * NV + l * V, x[k][u]);
            }
        };
        bool ok = true;
        for (int done = 0; ok && done < ne;) {
            // a row longer than the stage: eb entries at a time
            const int cnt = min(eb, ne - done), ng = cnt / (4 * rows);
            if (ne > eb) {
                __syncwarp();
                stage_entries<T>(r.e0 + done, cnt, eb, sbuf + (size_t)cur * stage_bytes, d.lci, lva, lane);
                cp_async_wait_all();
                __syncwarp();
                cw = sa;
                vw = sa + 4u * eb;
            }
            done += cnt;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k < ng) issue(k, k);
            for (int g = 0; ok && g < ng; g += 8) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (!ok || g + k >= ng) break;
                    unsigned spins = 0;
                    unsigned long long t0 = 0;
                    while (__any_sync(0xffffffffu, pend & (15u << (4 * k)))) {
                        look(k, g + k);
                        if (g + k + 1 < ng) look((k + 1) & 7, g + k + 1);
                        if ((++spins & 63) == 0) {
                            // one verdict for the warp
                            bool give = *(volatile int *)err != 0;
                            if (t0 == 0) t0 = now_ns();
                            else if (now_ns() - t0 > kLimitNs) {
                                atomicExch(err, 1);
                                give = true;
                            }
                            if (__any_sync(0xffffffffu, give)) {
                                ok = false;
                                break;
                            }
                        }
                    }
                    if (!ok) break;
                    T v[4];
                    lds4(vw + (unsigned)(sizeof(T) / 4) * r16 * (g + k), r16, v);
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int e = 0; e < V; ++e) sum[e] = fma(-v[u], x[k][u][e], sum[e]);
                    if (g + k + 8 < ng) issue(k, g + k + 8);
                }
            }
        }
        if (!ok) break;
        if (mine) {
#pragma unroll
            for (int e = 0; e < V; ++e) xo[e] = written(fma(rmul(rl[e], r.di), sum[e], xo[e]));
            rst(xout + (size_t)r.row * NV + l * V, xo);
        }
        __syncwarp();
        a = a1;
        a1 = a2;
        a2 = a3;
        r = r1;
        r1 = r2;
        cur ^= 1;
    }
    cp_async_wait_all();
}

static int device_sms() {
    thread_local int dev = -1, sms = 0;
    int d = 0;
    cudaGetDevice(&d);
    if (d != dev) {
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d);
        dev = d;
    }
    return sms > 0 ? sms : 1;
}

constexpr int kSmemMax = 227 * 1024;
constexpr int kStageMax = 256;  // entries of one stage (except where a step of one item has more)

int gs_rows_per_item(Prec p, int nv) {
    const int row = nv * (p == Prec::F64 ? 8 : 4);
    return row <= 16 ? 32 : 32 / (row / 16);
}
int gs_item_entries() { return kStageMax; }
// warps per item, as a shift: an item may have more rows than a warp
static int item_split(int rows, int rpw) {
    int s = 0;
    while ((rpw << s) < rows) ++s;
    return s;
}

int gs_item_warps(Prec p, int nv, int rows) { return 1 << item_split(rows, gs_rows_per_item(p, nv)); }

template <class T, int NV, bool XS, int NT>
static cudaError_t gs_block_l(int nblocks, const GsDir &f, const GsDir &b, const T *t, T *x, const T *relax, int brows,
                              int n, int eb, int split, size_t smem, unsigned long long limit, int *err, cudaStream_t s) {
    auto k = k_gs_block<T, NV, XS, NT>;
    // the limit belongs to the kernel: set for every launch (sizes differ)
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<nblocks, NT, smem, s>>>(f, b, t, x, relax, brows, n, eb, split, limit, err);
    return cudaGetLastError();
}

template <class T, int NV>
static cudaError_t gs_block_t(int nblocks, const GsDir &f, const GsDir &b, const void *t, void *x, const void *relax,
                              i64 brows, i64 n, int emax, int *err, bool *tile, cudaStream_t s,
                              unsigned long long limit) {
    const int eb = std::min(std::max(emax, 8), kStageMax), split = item_split(f.rows, 32 / Sh<T, NV>::TPR);
    // blocks per SM that must be resident for one wave, and the threads of a
    // CTA so that their registers fit
    const int per = std::min(4, (nblocks + device_sms() - 1) / device_sms());
    const int nt = per == 1 ? 512 : per == 2 ? 256 : 128;
    const size_t stage = (size_t)(nt / 32) * 2 * eb * (4 + sizeof(T)) + kStageSlack;
    const size_t tl = (size_t)(brows + 1) * NV * sizeof(T);  // + the row of zeros
    *tile = stage + tl + 1280 <= (size_t)kSmemMax / per;
    note_launch();
#define GO(XS, NT) gs_block_l<T, NV, XS, NT>(nblocks, f, b, (const T *)t, (T *)x, (const T *)relax, (int)brows, (int)n, \
                                             eb, split, stage + (XS ? tl : 0), limit, err, s)
    if (nt == 512) return *tile ? GO(true, 512) : GO(false, 512);
    if (nt == 256) return *tile ? GO(true, 256) : GO(false, 256);
    return *tile ? GO(true, 128) : GO(false, 128);
#undef GO
}

template <class T, int NV>
static cudaError_t gs_flow_t(const GsDir &d, int nitems, int nlev, int forward, const void *t, const void *xin,
                             void *xout, const void *relax, i64 n, int emax, int *err, cudaStream_t s) {
    int eb = std::min(std::max(emax, 8), kStageMax), split = item_split(d.rows, 32 / Sh<T, NV>::TPR);
    const size_t smem = (size_t)8 * 2 * eb * (4 + sizeof(T));
    auto k = k_gs_flow<T, NV>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(xout, 0xff, (size_t)n * NV * sizeof(T), s);
    if (e != cudaSuccess) return e;
    int g = (int)std::min<i64>(device_sms(), std::max<i64>(1, (((i64)nitems << split) * 8 / std::max(nlev, 1) + 7) / 8));
    GsDir dd = d;
    const T *tt = (const T *)t, *xi = (const T *)xin, *rl = (const T *)relax;
    T *xo = (T *)xout;
    int ni = (int)n;
    void *args[] = {&dd, &nitems, &forward, &tt, &xi, &xo, &rl, &ni, &eb, &split, &err};
    note_launch();
    return cudaLaunchCooperativeKernel((const void *)k, dim3(g), dim3(256), args, smem, s);
}

#define NV_SWITCH(nv, FN)                                                                         \
    switch (nv) {                                                                                  \
    case 1: return FN(1);                                                                          \
    case 2: return FN(2);                                                                          \
    case 4: return FN(4);                                                                          \
    case 8: return FN(8);                                                                          \
    case 16: return FN(16);                                                                        \
    case 32: return FN(32);                                                                        \
    default: return cudaErrorInvalidValue;                                                         \
    }

cudaError_t gs_sweep_block(Prec p, int nv, int nblocks, const GsDir &f, const GsDir &b, const void *t, void *x,
                           const void *relax, i64 brows, i64 n, int emax, int *err, bool *tile, cudaStream_t s,
                           unsigned long long limit_ns) {
    if (p == Prec::F64) {
#define F(NV) gs_block_t<double, NV>(nblocks, f, b, t, x, relax, brows, n, emax, err, tile, s, limit_ns)
        NV_SWITCH(nv, F)
#undef F
    } else {
#define F(NV) gs_block_t<float, NV>(nblocks, f, b, t, x, relax, brows, n, emax, err, tile, s, limit_ns)
        NV_SWITCH(nv, F)
#undef F
    }
}

cudaError_t gs_sweep_flow(Prec p, int nv, const GsDir &d, int nitems, int nlev, int forward, const void *t,
                          const void *xin, void *xout, const void *relax, i64 n, int emax, int *err, cudaStream_t s) {
    if (p == Prec::F64) {
#define F(NV) gs_flow_t<double, NV>(d, nitems, nlev, forward, t, xin, xout, relax, n, emax, err, s)
        NV_SWITCH(nv, F)
#undef F
    } else {
#define F(NV) gs_flow_t<float, NV>(d, nitems, nlev, forward, t, xin, xout, relax, n, emax, err, s)
        NV_SWITCH(nv, F)
#undef F
    }
}

// ---------------------------------------------------------------- wait self-test
// The bounded waits above, made to run out on purpose with a short limit:
// which = 0: every CTA but the first reads an element of a vector that CTA 0
// never writes, as k_gs_flow does; which = 1: an mbarrier phase that nothing
// completes, as k_gs_block's levels.  Every thread returns; nothing is left in
// flight.  Used by the tests to check that an expired wait surfaces as an
// error status instead of a hang.
__global__ void k_wait_selftest(int which, unsigned long long limit, float *words, int *err) {
    if (which == 0) {
        if (blockIdx.x == 0 || threadIdx.x != 0) return;  // the missing store
        const unsigned long long t0 = now_ns();
        float v[1];
        for (rld(words, v); unwritten(v[0]); rld(words, v))
            if (now_ns() - t0 > limit) {
                atomicExch(err, 1);
                return;
            }
        return;
    }
    __shared__ __align__(8) unsigned long long bar;
    __shared__ volatile int fail;
    if (threadIdx.x == 0) {
        fail = 0;
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0 && !mbar_wait(&bar, 0u, &fail, limit)) atomicExch(err, 2);
    __syncthreads();
}

cudaError_t wait_selftest(int which, int ncta, unsigned long long limit_ns, unsigned *words, int *err,
                          cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(words, 0xff, 256, s);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(err, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
    note_launch();
    k_wait_selftest<<<which == 0 ? ncta : 1, 128, 0, s>>>(which, limit_ns, reinterpret_cast<float *>(words), err);
    return cudaGetLastError();
}

}  // namespace xk
