// Kernels of the learned initial guess: a 3-D convolutional encoder-decoder
// trained and evaluated on the GPU (sm_100a).
//
// Tensors are channels-last BF16 volumes [nb][d][h][w][cs] addressed through a
// channel window (c0, c) of a buffer with cs channels per voxel, so that the
// decoder's concatenations are plain channel offsets.  Channel counts and
// offsets are multiples of 16.  Weights are [cout][27][cin] BF16 (tap t =
// (dz+1)*9 + (dy+1)*3 + (dx+1)), biases FP32; every product is accumulated in
// FP32 on the tensor cores (mma.sync m16n8k16 BF16).
//
//   conv3d   : implicit GEMM, M = voxels (tiles of 128), N = cout (tiles of 16,
//              32 or 64), K = 27 taps x cin in chunks of 16 channels; A and B
//              chunks are staged in shared memory by cp.async (4-stage ring,
//              zero fill outside the volume), fragments by ldmatrix.  The
//              epilogue adds the bias, applies ReLU and stores BF16 (or adds
//              to the stored value, for gradients that meet at a skip).
//   wgrad    : dW[co][t][ci] += sum_p g[p][co] * in[p + off(t)][ci], one CTA
//              per (set of boxes, 16-channel chunk of ci, up to 64 channels of
//              co) with all 27 taps, operands loaded transposed by
//              ldmatrix.trans, FP32 atomics into dW.
//   backward data = conv3d of the gradient with the flipped, transposed
//              weights (weight_flip).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include "kernels.cuh"
#include <algorithm>
#include <cstdint>
#include <cstdio>

typedef __nv_bfloat16 bf16;

namespace {

__device__ __forceinline__ unsigned smem_u32(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

// 16-byte async copy global -> shared; src_bytes = 0 fills zeros
__device__ __forceinline__ void cp16(void *dst, const void *src, unsigned src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src),
                 "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void ldm_x4(unsigned (&r)[4], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldm_x2(unsigned (&r)[2], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1])
                 : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldm_x4_a(unsigned (&r)[4], unsigned a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}
__device__ __forceinline__ void ldm_x4_ta(unsigned (&r)[4], unsigned a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}

// D = A (16x16, row) * B (16x8, col) + D, BF16 inputs, FP32 accumulate
__device__ __forceinline__ void mma16816(float (&d)[4], const unsigned (&a)[4], unsigned b0,
                                         unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Shared-memory rows of 16 channels (32 bytes): the two 16-byte halves of
// row r are swapped when bit 2 of r is set, so that 8 consecutive rows read by
// one ldmatrix hit 8 distinct bank groups.
__device__ __forceinline__ int sw32(int r, int h) { return r * 32 + ((h ^ ((r >> 2) & 1)) << 4); }

struct Vol {
    int nb, d, h, w;
    __host__ __device__ __forceinline__ i64 count() const { return (i64)nb * d * h * w; }
};

constexpr int BM = 128;  // voxels per CTA tile
constexpr int NS = 4;    // pipeline stages

// conv3d: out[v][oc0 + n] (+)= act(bias[n] + sum_t sum_c in[v+off(t)][ic0 + c] w[n][t][c]);
// flags: 1 ReLU, 2 accumulate, 4 FP32 output (out is then a float buffer)
template <int BN>
__global__ void __launch_bounds__(128) k_conv3d(const bf16 *__restrict__ in, int ics, int ic0,
                                                int cin, const bf16 *__restrict__ w,
                                                const float *__restrict__ bias, bf16 *out, int ocs,
                                                int oc0, int cout, Vol g, int flags) {
    __shared__ __align__(128) unsigned char sa[NS][BM * 32];
    __shared__ __align__(128) unsigned char sb[NS][BN * 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const i64 nvox = g.count();
    const i64 v0 = (i64)blockIdx.x * BM;
    const int n0 = blockIdx.y * BN;
    const int kc = cin / 16;          // channel chunks per tap
    const int nk = 27 * kc;           // K chunks
    const i64 myv = v0 + tid;         // the voxel whose A row this thread stages
    const bool vin = myv < nvox;
    int vx = 0, vy = 0, vz = 0;
    if (vin) {
        vx = (int)(myv % g.w);
        vy = (int)((myv / g.w) % g.h);
        vz = (int)((myv / ((i64)g.w * g.h)) % g.d);
    }

    auto stage = [&](int k, int s) {
        const int t = k / kc, cb = (k % kc) * 16;
        // A: 128 rows of 16 channels, two 16-byte halves each
        const int dz = t / 9 - 1, dy = (t / 3) % 3 - 1, dx = t % 3 - 1;
        const bool inside = vin && (unsigned)(vz + dz) < (unsigned)g.d &&
                            (unsigned)(vy + dy) < (unsigned)g.h && (unsigned)(vx + dx) < (unsigned)g.w;
        const i64 src = inside ? myv + ((i64)dz * g.h + dy) * g.w + dx : -1;
        const bf16 *pa = in + (src < 0 ? 0 : src) * ics + ic0 + cb;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
            cp16(&sa[s][sw32(tid, hh)], pa + hh * 8, src < 0 ? 0u : 16u);
        // B: BN rows (output channels) of 16 k values
        for (int q = tid; q < BN * 2; q += 128) {
            const int r = q >> 1, hh = q & 1;
            const bf16 *pb = w + ((i64)(n0 + r) * 27 + t) * cin + cb + hh * 8;
            cp16(&sb[s][sw32(r, hh)], pb, 16u);
        }
    };

    float acc[2][BN / 8][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < BN / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;

#pragma unroll
    for (int s = 0; s < NS - 1; ++s) {
        if (s < nk) stage(s, s);
        cp_commit();
    }
    for (int k = 0; k < nk; ++k) {
        cp_wait<NS - 2>();
        __syncthreads();
        if (k + NS - 1 < nk) stage(k + NS - 1, (k + NS - 1) % NS);
        cp_commit();
        const int s = k % NS;
        unsigned a[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = warp * 32 + i * 16 + (lane & 15);
            ldm_x4(a[i], &sa[s][sw32(r, lane >> 4)]);
        }
#pragma unroll
        for (int j = 0; j < BN / 16; ++j) {
            // two n8 tiles: lanes 0-7 rows n 0-7 k0, 8-15 n 0-7 k8, 16-23 n 8-15 k0, 24-31 n 8-15 k8
            const int r = j * 16 + (lane & 7) + ((lane >> 4) << 3);
            unsigned bq[4];
            ldm_x4(bq, &sb[s][sw32(r, (lane >> 3) & 1)]);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                mma16816(acc[i][2 * j], a[i], bq[0], bq[1]);
                mma16816(acc[i][2 * j + 1], a[i], bq[2], bq[3]);
            }
        }
        if (BN % 16) {
            const int j = BN / 16;
            const int r = j * 16 + (lane & 7);
            unsigned bq[2];
            ldm_x2(bq, &sb[s][sw32(r, (lane >> 3) & 1)]);
#pragma unroll
            for (int i = 0; i < 2; ++i) mma16816(acc[i][2 * j], a[i], bq[0], bq[1]);
        }
    }
    cp_wait<0>();
    // epilogue: rows g = lane/4 (+8), columns 2*(lane%4) (+1)
    const bool relu = flags & 1, accum = flags & 2, f32out = flags & 4;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < BN / 8; ++j)
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                const i64 v = v0 + warp * 32 + i * 16 + (lane >> 2) + hr * 8;
                if (v >= nvox) continue;
                const int n = n0 + j * 8 + 2 * (lane & 3);
                float y0 = acc[i][j][2 * hr], y1 = acc[i][j][2 * hr + 1];
                if (bias) {
                    y0 += bias[n];
                    y1 += bias[n + 1];
                }
                if (relu) {
                    y0 = fmaxf(y0, 0.f);
                    y1 = fmaxf(y1, 0.f);
                }
                if (f32out) {
                    float2 *pf = reinterpret_cast<float2 *>(reinterpret_cast<float *>(out) + v * ocs + oc0 + n);
                    if (accum) {
                        const float2 o = *pf;
                        y0 += o.x;
                        y1 += o.y;
                    }
                    *pf = make_float2(y0, y1);
                    continue;
                }
                __nv_bfloat162 *po = reinterpret_cast<__nv_bfloat162 *>(out + v * ocs + oc0 + n);
                if (accum) {
                    const float2 o = __bfloat1622float2(*po);
                    y0 += o.x;
                    y1 += o.y;
                }
                *po = __floats2bfloat162_rn(y0, y1);
            }
}

// conv3d on boxes of BZ x 8 x 8 voxels: warp z owns one plane of the box (64
// voxels, four MMA row tiles) and BN output channels.  For every 16-channel chunk
// the box's halo is staged once, in planes of 8 channels (16-byte rows: eight
// consecutive voxels fill the 32 banks at any tap's shift), and the A operand of
// a tap is read from it by ldmatrix at a constant offset.  CTAs are persistent:
// the next chunk (or box) is copied while this one computes, and the weights stay
// in shared memory for all boxes when they fit (WRES), else each chunk brings its
// own.  Voxels outside the volume are zeros; outputs outside it are not stored.
// Same sums as k_conv3d, chunk by chunk (the order of the kernel before).
// Bound: the fragments' reads from shared memory (66 % of its wavefronts), four A
// and BN / 16 B fragments for BN / 2 mma, and the tensor pipe behind them (60 % of its
// cycles).  48 -> 16 channels, 8 x 64^3: 274 us, 318 TFLOP/s; 602 us by the kernel
// before, which staged halo and weights for 128 voxels at a time with nothing under
// way meanwhile.
template <int BN, int BZ> struct BoxShape {
    static constexpr int NT = 32 * BZ, ROWS = (BZ + 2) * 100, HBYTES = 2 * ROWS * 16, WBYTES = 27 * BN * 32;
};
template <int BN, int BZ, bool WRES>
__global__ void __launch_bounds__(32 * BZ, BN == 16 ? 16 / BZ : BZ == 8 || BN == 64 ? 1 : 2) k_conv3d_box(const bf16 *__restrict__ in, int ics, int ic0, int cin,
                                                        const bf16 *__restrict__ w, const float *__restrict__ bias,
                                                        bf16 *out, int ocs, int oc0, Vol g, int nbx, int nby, int nbz,
                                                        int nboxes, int flags) {
    typedef BoxShape<BN, BZ> S;
    constexpr int NT = S::NT, LT = NT / 20, NL = ((BZ + 2) * 10 + LT - 1) / LT;
    constexpr int STAGE = S::HBYTES + (WRES ? 0 : S::WBYTES);
    extern __shared__ __align__(128) unsigned char dyn[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kc = cin / 16, n0 = blockIdx.y * BN;
    unsigned char *stg = dyn + (WRES ? kc * S::WBYTES : 0);
    // weights of chunk c, [tap][half][n] rows of 16 bytes
    auto weights = [&](int c, unsigned char *dst) {
        for (int p = tid; p < 27 * BN * 2; p += NT) {
            const int hh = p & 1, n = (p >> 1) % BN, t = (p >> 1) / BN;
            cp16(dst + ((t * 2 + hh) * BN + n) * 16, w + ((i64)(n0 + n) * 27 + t) * cin + c * 16 + hh * 8, 16u);
        }
    };
    if (WRES)
        for (int c = 0; c < kc; ++c) weights(c, dyn + c * S::WBYTES);
    // halo pieces of this thread: half and x fixed, lines (y, z) LT apart.  A line's
    // offset and the faces of the box's halo it lies on are tabled once; a box
    // whose halo crosses the volume's boundary leaves those faces out.
    const int hh = tid & 1, hx = (tid >> 1) % 10, hl = tid / 20;
    const bool loader = tid < LT * 20;
    __shared__ int2 s_line[NL * LT];
    for (int k = tid; k < NL * LT; k += NT) {
        const int z = k / 10, y = k % 10;
        s_line[k] = k < (BZ + 2) * 10 ? make_int2((z * g.h + y) * g.w * ics, (y == 0) | (y == 9) << 1 | (z == 0) << 2 | (z == BZ + 1) << 3)
                                      : make_int2(0, 64);
    }
    const int fx = (hx == 0) << 4 | (hx == 9) << 5;
    const bool whole = g.w % 8 == 0 && g.h % 8 == 0 && g.d % BZ == 0;  // no box reaches past the volume by more than its halo
    __syncthreads();
    int sx = 0, sy = 0, sz = 0;  // origin of the staged box's halo
    i64 sb = 0;                  // first plane of its volume
    auto stage = [&](int box, int c, int s) {
        if (c == 0) {
            int q = box;
            sx = (q % nbx) * 8 - 1;
            q /= nbx;
            sy = (q % nby) * 8 - 1;
            q /= nby;
            sz = (q % nbz) * BZ - 1;
            sb = (i64)(q / nbz) * g.d;
        }
        unsigned char *sh = stg + s * STAGE;
        if (!WRES) weights(c, sh + S::HBYTES);
        if (loader) {
            const bf16 *src = in + (((sb + sz) * g.h + sy) * g.w + sx + hx) * ics + ic0 + c * 16 + hh * 8;
            unsigned char *dst = sh + hh * (S::ROWS * 16) + hx * 16 + hl * 160;
            if (whole) {
                const int out_ = ((sy < 0) | (sy + 10 > g.h) << 1 | (sz < 0) << 2 | (sz + BZ + 2 > g.d) << 3 | (sx < 0) << 4 |
                                  (sx + 10 > g.w) << 5);
#pragma unroll
                for (int k = 0; k < NL; ++k) {
                    const int2 ln = s_line[hl + k * LT];
                    const bool ok = ((ln.y | fx) & out_) == 0;
                    if (ln.y < 64) cp16(dst + k * LT * 160, ok ? src + ln.x : in, ok ? 16u : 0u);
                }
            } else {
                const bool okx = (unsigned)(sx + hx) < (unsigned)g.w;
#pragma unroll
                for (int k = 0; k < NL; ++k) {
                    const int ln = hl + k * LT, z = ln / 10, y = ln - 10 * z;
                    if (ln < (BZ + 2) * 10) {
                        const bool ok = okx && (unsigned)(sy + y) < (unsigned)g.h && (unsigned)(sz + z) < (unsigned)g.d;
                        cp16(dst + k * LT * 160, ok ? src + ((i64)z * g.h + y) * g.w * ics : in, ok ? 16u : 0u);
                    }
                }
            }
        }
        cp_commit();
    };
    const unsigned base0 = smem_u32(stg), wbase = WRES ? smem_u32(dyn) : base0 + S::HBYTES;
    // this lane's rows: A (voxel lane & 15 of a tile, half lane >> 4), B (output
    // channel, half)
    const unsigned aa = (unsigned)((lane >> 4) * (S::ROWS * 16) + (warp * 100 + ((lane >> 3) & 1) * 10 + (lane & 7)) * 16);
    const unsigned ba = (unsigned)(((lane >> 3) & 1) * (BN * 16) + ((lane & 7) + ((lane >> 4) << 3)) * 16);
    const bool relu = flags & 1, accum = flags & 2, f32out = flags & 4;
    int box = blockIdx.x, s = 0;
    if (box < nboxes) stage(box, 0, 0);
    for (; box < nboxes; box += gridDim.x) {
        float acc[4][BN / 8][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < BN / 8; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
        for (int c = 0; c < kc; ++c, s ^= 1) {
            if (c + 1 < kc) stage(box, c + 1, s ^ 1);
            else if (box + (int)gridDim.x < nboxes) stage(box + gridDim.x, 0, s ^ 1);
            else cp_commit();
            cp_wait<1>();
            __syncthreads();
            const unsigned ab = base0 + (unsigned)(s * STAGE) + aa;
            const unsigned bb = wbase + (unsigned)(WRES ? c * S::WBYTES : s * STAGE) + ba;
            // a tap's fragments are read while the one before multiplies (at 64
            // output channels the accumulators leave no registers for that, and
            // 32 mma a tap hide the reads)
            constexpr int NB = BN == 64 ? 1 : 2;
            unsigned a[NB][4][4], bq[NB][BN / 16][4];
            auto frag = [&](int t, unsigned(&af)[4][4], unsigned(&bf)[BN / 16][4]) {
                const unsigned at = ab + (unsigned)(((t / 9) * 100 + (t / 3) % 3 * 10 + t % 3) * 16);
#pragma unroll
                for (int i = 0; i < 4; ++i) ldm_x4_a(af[i], at + (unsigned)(i * 20 * 16));
#pragma unroll
                for (int j = 0; j < BN / 16; ++j) ldm_x4_a(bf[j], bb + (unsigned)(t * BN * 32 + j * 256));
            };
            if (NB == 2) frag(0, a[0], bq[0]);
#pragma unroll
            for (int t = 0; t < 27; ++t) {
                const int u = t & (NB - 1);
                if (NB == 1) frag(t, a[0], bq[0]);
                else if (t + 1 < 27) frag(t + 1, a[u ^ 1], bq[u ^ 1]);
#pragma unroll
                for (int j = 0; j < BN / 16; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        mma16816(acc[i][2 * j], a[u][i], bq[u][j][0], bq[u][j][1]);
                        mma16816(acc[i][2 * j + 1], a[u][i], bq[u][j][2], bq[u][j][3]);
                    }
            }
            __syncthreads();
        }
        int q = box;
        const int x0 = (q % nbx) * 8;
        q /= nbx;
        const int y0 = (q % nby) * 8;
        q /= nby;
        const int z = (q % nbz) * BZ + warp;
        const i64 vb = (i64)(q / nbz) * g.d;
        const int x = x0 + (lane >> 2);
        const i64 o0 = (((vb + z) * g.h + y0) * g.w + x) * ocs + oc0 + n0 + 2 * (lane & 3);
        const int rows = x < g.w && z < g.d ? min(8, g.h - y0) : 0, ystep = g.w * ocs;
        if (!accum && !f32out) {
#pragma unroll
            for (int j = 0; j < BN / 8; ++j) {
                const float b0 = bias ? __ldg(bias + n0 + j * 8 + 2 * (lane & 3)) : 0.f;
                const float b1 = bias ? __ldg(bias + n0 + j * 8 + 2 * (lane & 3) + 1) : 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float u = acc[i / 2][j][2 * (i & 1)], v = acc[i / 2][j][2 * (i & 1) + 1];
                    if (bias) {
                        u += b0;
                        v += b1;
                    }
                    if (relu) {
                        u = fmaxf(u, 0.f);
                        v = fmaxf(v, 0.f);
                    }
                    if (i < rows)
                        *reinterpret_cast<__nv_bfloat162 *>(out + o0 + (i64)i * ystep + j * 8) = __floats2bfloat162_rn(u, v);
                }
            }
            continue;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                if (2 * i + hr >= rows) continue;
                const i64 o = o0 + (i64)(2 * i + hr) * ystep;
#pragma unroll
                for (int j = 0; j < BN / 8; ++j) {
                    const int n = n0 + j * 8 + 2 * (lane & 3);
                    float y0v = acc[i][j][2 * hr], y1v = acc[i][j][2 * hr + 1];
                    if (bias) {
                        y0v += __ldg(bias + n);
                        y1v += __ldg(bias + n + 1);
                    }
                    if (relu) {
                        y0v = fmaxf(y0v, 0.f);
                        y1v = fmaxf(y1v, 0.f);
                    }
                    if (f32out) {
                        float2 *pf = reinterpret_cast<float2 *>(reinterpret_cast<float *>(out) + o + j * 8);
                        if (accum) {
                            const float2 ov = *pf;
                            y0v += ov.x;
                            y1v += ov.y;
                        }
                        *pf = make_float2(y0v, y1v);
                        continue;
                    }
                    __nv_bfloat162 *po = reinterpret_cast<__nv_bfloat162 *>(out + o + j * 8);
                    if (accum) {
                        const float2 ov = __bfloat1622float2(*po);
                        y0v += ov.x;
                        y1v += ov.y;
                    }
                    *po = __floats2bfloat162_rn(y0v, y1v);
                }
            }
    }
    cp_wait<0>();
}

// wgrad: dw[co][t][ci] += sum over the CTA's boxes of g[p][co] * in[p + off(t)][ci]
// for one 16-channel chunk of ci and CO output channels, all 27 taps at once.  A
// box is 2 x 8 x 8 voxels; its gradients and the chunk's halo (4 x 10 x 10 voxels)
// are staged once, in planes of 8 channels (16-byte rows: eight consecutive
// voxels fill the 32 banks, at any tap's shift, without a swizzle), while the
// box before computes.  The eight warps share the taps (warp w: w, w + 8, ..), so
// a fragment of the gradient serves 3 or 4 taps, and every partial sum stays in
// registers until the CTA's boxes are done (FP32 atomics, one per CTA and
// weight).  Voxels outside the volume are zeros on both sides.
// Bound: the tensor pipe by mma.sync (53 % of its cycles) and the fragments' latency.  cin 96, cout
// 32, 4 x 32^3: 90 us, 240 TFLOP/s; 569 us by the kernel before, which staged the
// gradient and a shifted input once per tap and chunk.
constexpr int WG_HALO = 4 * 10 * 10, WG_VOX = 128;
template <int CO> struct WgradShape {
    static constexpr int GBYTES = (CO / 8) * WG_VOX * 16, HBYTES = 2 * WG_HALO * 16, STAGE = GBYTES + HBYTES;
};
// I: type of box numbers and of offsets inside a box (int, or i64 for planes or
// counts beyond it)
template <int CO, class I>
__global__ void __launch_bounds__(256, CO == 64 ? 1 : 2) k_wgrad(const bf16 *__restrict__ in, int ics, int ic0, int cin,
                                                                 const bf16 *__restrict__ gr, int gcs, int gc0,
                                                                 float *dw, Vol g, int nbx, int nby, int nbz,
                                                                 I nboxes) {
    typedef WgradShape<CO> S;
    extern __shared__ __align__(128) unsigned char dyn[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cb = blockIdx.y * 16, o0 = blockIdx.z * CO;
    // 16-byte pieces of this thread, the same of every box: halo piece p is half
    // p & 1 of halo voxel p >> 1, gradient piece p channels 8 (p % (CO / 8)) .. of
    // box voxel p / (CO / 8); offsets from the box's origin and, for the halo, the
    // faces it lies on
    constexpr int NH = (2 * WG_HALO + 255) / 256, NG = CO / 8 * WG_VOX / 256;
    int hf[NH];
    I ho[NH], go[NG];
    auto halo_at = [&](int k, int &x, int &y, int &z) {
        const int v = (tid + 256 * k) >> 1;
        x = v % 10 - 1;
        y = v / 10 % 10 - 1;
        z = v / 100 - 1;
        return v < WG_HALO;
    };
    auto grad_at = [&](int k, int &x, int &y, int &z) {
        const int v = (tid + 256 * k) / (CO / 8);
        x = v & 7;
        y = v >> 3 & 7;
        z = v >> 6;
    };
#pragma unroll
    for (int k = 0; k < NH; ++k) {
        int x, y, z;
        const bool on = halo_at(k, x, y, z);
        ho[k] = (((I)z * g.h + y) * g.w + x) * ics + (tid & 1) * 8;
        hf[k] = on ? (x < 0) | (x == 8) << 1 | (y < 0) << 2 | (y == 8) << 3 | (z < 0) << 4 | (z == 2) << 5 : 64;
    }
#pragma unroll
    for (int k = 0; k < NG; ++k) {
        int x, y, z;
        grad_at(k, x, y, z);
        go[k] = (((I)z * g.h + y) * g.w + x) * gcs + (tid + 256 * k) % (CO / 8) * 8;
    }
    const bool whole = g.w % 8 == 0 && g.h % 8 == 0 && g.d % 2 == 0;
    auto stage = [&](I box, int s) {
        I q = box;
        const int x0 = (int)(q % nbx) * 8;
        q /= nbx;
        const int y0 = (int)(q % nby) * 8;
        q /= nby;
        const int z0 = (int)(q % nbz) * 2;
        const i64 v0 = (((i64)(q / nbz) * g.d + z0) * g.h + y0) * g.w + x0;
        unsigned char *sg = dyn + s * S::STAGE, *sh = sg + S::GBYTES + (tid & 1) * (WG_HALO * 16) + (tid >> 1) * 16;
        const bf16 *pi = in + v0 * ics + ic0 + cb, *pg = gr + v0 * gcs + gc0 + o0;
        unsigned char *dg = sg + tid % (CO / 8) * (WG_VOX * 16) + tid / (CO / 8) * 16;  // 256 is a multiple of CO / 8
        if (whole) {
            const int out_ = (x0 == 0) | (x0 + 8 == g.w) << 1 | (y0 == 0) << 2 | (y0 + 8 == g.h) << 3 | (z0 == 0) << 4 |
                             (z0 + 2 == g.d) << 5;
#pragma unroll
            for (int k = 0; k < NH; ++k) {
                const bool ok = (hf[k] & out_) == 0;
                if (hf[k] < 64) cp16(sh + k * 128 * 16, ok ? pi + ho[k] : in, ok ? 16u : 0u);
            }
#pragma unroll
            for (int k = 0; k < NG; ++k) cp16(dg + k * (256 / (CO / 8)) * 16, pg + go[k], 16u);
        } else {
#pragma unroll
            for (int k = 0; k < NH; ++k) {
                int x, y, z;
                halo_at(k, x, y, z);
                const bool ok = (unsigned)(x0 + x) < (unsigned)g.w && (unsigned)(y0 + y) < (unsigned)g.h &&
                                (unsigned)(z0 + z) < (unsigned)g.d;
                if (hf[k] < 64) cp16(sh + k * 128 * 16, ok ? pi + ho[k] : in, ok ? 16u : 0u);
            }
#pragma unroll
            for (int k = 0; k < NG; ++k) {
                int x, y, z;
                grad_at(k, x, y, z);
                const bool ok = x0 + x < g.w && y0 + y < g.h && z0 + z < g.d;
                cp16(dg + k * (256 / (CO / 8)) * 16, ok ? pg + go[k] : gr, ok ? 16u : 0u);
            }
        }
        cp_commit();
    };
    float acc[4][CO / 16][2][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int m = 0; m < CO / 16; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[j][m][h][e] = 0.f;
    // this lane's addresses inside a stage: gradient rows and, per tap, halo rows
    const unsigned ga = (unsigned)((((lane >> 3) & 1) * WG_VOX + (lane & 7) + ((lane >> 4) << 3)) * 16);
    unsigned ha[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int t = min(warp + 8 * j, 26);
        // voxel of this lane in a group of 16: x = lane & 7, y = lane >> 3 & 1
        const int row = ((t / 9) * 10 + (t / 3) % 3 + ((lane >> 3) & 1)) * 10 + t % 3 + (lane & 7);
        ha[j] = (unsigned)(S::GBYTES + (lane >> 4) * (WG_HALO * 16) + row * 16);
    }
    const int taps = warp < 3 ? 4 : 3;
    I box = blockIdx.x;
    int s = 0;
    if (box < nboxes) stage(box, 0);
    for (; box < nboxes; box += gridDim.x, s ^= 1) {
        if (box + (int)gridDim.x < nboxes) stage(box + gridDim.x, s ^ 1);
        else cp_commit();
        cp_wait<1>();
        __syncthreads();
        const unsigned base = smem_u32(dyn) + (unsigned)(s * S::STAGE);
        // 16 voxels a step: two rows of 8 in plane z = k / 4; the next tap's
        // fragment is read while this one multiplies
        unsigned a[CO / 16][4], bq[2][4];
        ldm_x4_ta(bq[0], base + ha[0]);
        const bool low = (int)(box / nbx % nby) * 8 + 4 >= g.h;  // the box's rows y >= 4 lie outside: zeros
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if ((k & 3) >= 2 && low) continue;
#pragma unroll
            for (int m = 0; m < CO / 16; ++m) ldm_x4_ta(a[m], base + ga + (unsigned)((2 * m * WG_VOX + 16 * k) * 16));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int kn = j == 3 ? k + 1 : k, jn = (j + 1) & 3;  // what follows (tap 3 repeats tap 26 on five warps)
                if (j == 3 && (k & 3) == 1 && low) ldm_x4_ta(bq[0], base + ha[0] + (unsigned)((k / 4 + 1) % 2 * 1600));
                else if (kn < 8) ldm_x4_ta(bq[(j + 1) & 1], base + ha[jn] + (unsigned)(((kn / 4) * 100 + (kn % 4) * 20) * 16));
                if (j == 3 && taps == 3) continue;
#pragma unroll
                for (int m = 0; m < CO / 16; ++m) {
                    mma16816(acc[j][m][0], a[m], bq[j & 1][0], bq[j & 1][1]);
                    mma16816(acc[j][m][1], a[m], bq[j & 1][2], bq[j & 1][3]);
                }
            }
        }
        __syncthreads();
    }
    cp_wait<0>();
    const bool pairs = reinterpret_cast<uintptr_t>(dw) % 8 == 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j == 3 && taps == 3) break;
        float *dwt = dw + (i64)(warp + 8 * j) * cin + cb;  // dw[co][t][ci] = dwt[co * 27 * cin + ci]
#pragma unroll
        for (int m = 0; m < CO / 16; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const int co = o0 + m * 16 + (lane >> 2) + (e >> 1) * 8, ci = h * 8 + 2 * (lane & 3);
                    float *p = dwt + (i64)co * 27 * cin + ci;
                    if (pairs) {
                        asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(acc[j][m][h][e]), "f"(acc[j][m][h][e + 1]) : "memory");
                    } else {
                        atomicAdd(p, acc[j][m][h][e]);
                        atomicAdd(p + 1, acc[j][m][h][e + 1]);
                    }
                }
    }
}

// w [cout][27][cin] -> wt [cin][27][cout] with taps reversed (backward data)
__global__ void k_weight_flip(const bf16 *__restrict__ w, bf16 *__restrict__ wt, int cout, int cin) {
    const i64 total = (i64)cout * 27 * cin;
    for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (i64)gridDim.x * blockDim.x) {
        const int ci = (int)(q % cin);
        const i64 r = q / cin;
        const int t = (int)(r % 27), co = (int)(r / 27);
        wt[((i64)ci * 27 + (26 - t)) * cout + co] = w[q];
    }
}

// Elementwise volume kernels work on groups of 8 channels (16 bytes), which
// every channel count and offset here allows (multiples of 16).
struct Oct {
    float v[8];
};
__device__ __forceinline__ Oct ld8(const bf16 *p) {
    const uint4 u = *reinterpret_cast<const uint4 *>(p);
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u);
    Oct o;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 f = __bfloat1622float2(h[k]);
        o.v[2 * k] = f.x;
        o.v[2 * k + 1] = f.y;
    }
    return o;
}
__device__ __forceinline__ void st8(bf16 *p, const Oct &o) {
    uint4 u;
    __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&u);
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(o.v[2 * k], o.v[2 * k + 1]);
    *reinterpret_cast<uint4 *>(p) = u;
}

// g[p][gc0 + c] *= (act[p][ac0 + c] > 0), 8 channels a thread
__global__ void k_relu_bwd(bf16 *g, int gcs, int gc0, const bf16 *__restrict__ act, int acs, int ac0,
                           int c8, i64 nvox) {
    const i64 total = nvox * c8;
    for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (i64)gridDim.x * blockDim.x) {
        const i64 p = q / c8;
        const int k = (int)(q - p * c8) * 8;
        bf16 *pg = g + p * gcs + gc0 + k;
        uint4 w = *reinterpret_cast<const uint4 *>(pg);
        const uint4 av = *reinterpret_cast<const uint4 *>(act + p * acs + ac0 + k);
        const __nv_bfloat16 *ah = reinterpret_cast<const __nv_bfloat16 *>(&av);
        __nv_bfloat16 *gh = reinterpret_cast<__nv_bfloat16 *>(&w);
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (!(__bfloat162float(ah[e]) > 0.f)) gh[e] = __float2bfloat16(0.f);
        *reinterpret_cast<uint4 *>(pg) = w;
    }
}
// the same for channel counts, offsets or strides that are not multiples of 8
__global__ void k_relu_bwd1(bf16 *g, int gcs, int gc0, const bf16 *__restrict__ act, int acs, int ac0,
                            int c, i64 nvox) {
    const i64 total = nvox * c;
    for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (i64)gridDim.x * blockDim.x) {
        const i64 p = q / c;
        const int k = (int)(q % c);
        if (!(__bfloat162float(act[p * acs + ac0 + k]) > 0.f)) g[p * gcs + gc0 + k] = __float2bfloat16(0.f);
    }
}

// db[c] += sum_p g[p][gc0 + c]: a thread sums 8 channels over its voxels of the
// block's slice, the block's sums meet in shared memory, one atomic per channel
__global__ void __launch_bounds__(256) k_bias_grad(const bf16 *__restrict__ g, int gcs, int gc0, int c8, i64 nvox,
                                                   i64 slice, float *db) {
    __shared__ float red[256][9];
    const int tid = threadIdx.x, k = tid % c8, lanes = 256 / c8;
    const i64 p0 = (i64)blockIdx.x * slice, p1 = min(nvox, p0 + slice);
    float s[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) s[e] = 0.f;
#pragma unroll 4
    for (i64 p = p0 + tid / c8; p < p1; p += lanes) {
        const Oct o = ld8(g + p * gcs + gc0 + k * 8);
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e] += o.v[e];
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) red[tid][e] = s[e];
    __syncthreads();
    if (tid < c8 * 8) {
        float t = 0.f;
        for (int r = 0; r < lanes; ++r) t += red[r * c8 + tid / 8][tid % 8];
        atomicAdd(db + tid, t);
    }
}
// the same for channel counts, offsets or strides that are not multiples of 8
__global__ void k_bias_grad1(const bf16 *__restrict__ g, int gcs, int gc0, int c, i64 nvox,
                             i64 slice, float *db) {
    const int k = threadIdx.x % c;
    const int lanes = blockDim.x / c;
    const i64 p0 = (i64)blockIdx.x * slice, p1 = min(nvox, p0 + slice);
    float s = 0.f;
    for (i64 p = p0 + threadIdx.x / c; p < p1; p += lanes) s += __bfloat162float(g[p * gcs + gc0 + k]);
    atomicAdd(db + k, s);
}

// 2x2x2 average pooling of volume g (even sides): one thread per coarse voxel
// and 8 channels
__global__ void k_pool2(const bf16 *__restrict__ in, int ics, int ic0, bf16 *out, int ocs, int oc0,
                        int c, Vol g) {
    const int D = g.d / 2, H = g.h / 2, W = g.w / 2, c8 = c / 8;
    const i64 total = (i64)g.nb * D * H * W * c8;
    for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (i64)gridDim.x * blockDim.x) {
        const int k = (int)(q % c8) * 8;
        const i64 cv = q / c8;
        i64 r = cv;
        const int x = (int)(r % W); r /= W;
        const int y = (int)(r % H); r /= H;
        const int z = (int)(r % D);
        const i64 b = r / D;
        Oct s;
#pragma unroll
        for (int e = 0; e < 8; ++e) s.v[e] = 0.f;
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            const i64 v = ((b * g.d + 2 * z + (o >> 2)) * g.h + 2 * y + ((o >> 1) & 1)) * g.w + 2 * x + (o & 1);
            const Oct t = ld8(in + v * ics + ic0 + k);
#pragma unroll
            for (int e = 0; e < 8; ++e) s.v[e] += t.v[e];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) s.v[e] *= 0.125f;
        st8(out + cv * ocs + oc0 + k, s);
    }
}

// nearest upsampling of a (d/2, h/2, w/2) volume to g; mode 1 adds the
// pooled-gradient share (x 1/8) for the pooling backward, mode 0 copies.
// One thread per coarse voxel and 8 channels writes its 8 fine voxels.
__global__ void k_up2(const bf16 *__restrict__ in, int ics, int ic0, bf16 *out, int ocs, int oc0,
                      int c, Vol g, int mode) {
    const int D = g.d / 2, H = g.h / 2, W = g.w / 2, c8 = c / 8;
    const i64 total = (i64)g.nb * D * H * W * c8;
    for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (i64)gridDim.x * blockDim.x) {
        const int k = (int)(q % c8) * 8;
        const i64 cv = q / c8;
        i64 r = cv;
        const int x = (int)(r % W); r /= W;
        const int y = (int)(r % H); r /= H;
        const int z = (int)(r % D);
        const i64 b = r / D;
        const Oct src = ld8(in + cv * ics + ic0 + k);
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            const i64 v = ((b * g.d + 2 * z + (o >> 2)) * g.h + 2 * y + ((o >> 1) & 1)) * g.w + 2 * x + (o & 1);
            bf16 *po = out + v * ocs + oc0 + k;
            if (mode == 1) {
                Oct t = ld8(po);
#pragma unroll
                for (int e = 0; e < 8; ++e) t.v[e] += src.v[e] * 0.125f;
                st8(po, t);
            } else {
                st8(po, src);
            }
        }
    }
}

// backward of nearest upsampling: dIn[coarse] = sum of the 8 fine gradients
__global__ void k_up2_bwd(const bf16 *__restrict__ gfine, int gcs, int gc0, bf16 *gin, int ics,
                          int ic0, int c, Vol g) {
    const int D = g.d / 2, H = g.h / 2, W = g.w / 2, c8 = c / 8;
    const i64 total = (i64)g.nb * D * H * W * c8;
    for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (i64)gridDim.x * blockDim.x) {
        const int k = (int)(q % c8) * 8;
        const i64 cv = q / c8;
        i64 r = cv;
        const int x = (int)(r % W); r /= W;
        const int y = (int)(r % H); r /= H;
        const int z = (int)(r % D);
        const i64 b = r / D;
        Oct s;
#pragma unroll
        for (int e = 0; e < 8; ++e) s.v[e] = 0.f;
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            const i64 v = ((b * g.d + 2 * z + (o >> 2)) * g.h + 2 * y + ((o >> 1) & 1)) * g.w + 2 * x + (o & 1);
            const Oct t = ld8(gfine + v * gcs + gc0 + k);
#pragma unroll
            for (int e = 0; e < 8; ++e) s.v[e] += t.v[e];
        }
        st8(gin + cv * ics + ic0 + k, s);
    }
}

// loss = mean (pred - target)^2 over nvox voxels (pred = channel pc0 of an
// FP32 volume); grad[p][0] = 2 (pred - target) / nvox, other grad channels 0
__global__ void k_mse(const float *__restrict__ pred, int pcs, int pc0, const float *__restrict__ tgt,
                      bf16 *grad, int gcs, i64 nvox, float *loss) {
    float s = 0.f;
    for (i64 p = (i64)blockIdx.x * blockDim.x + threadIdx.x; p < nvox; p += (i64)gridDim.x * blockDim.x) {
        const float d = pred[p * pcs + pc0] - tgt[p];
        s += d * d;
        if (grad) {
            for (int k = 0; k < gcs; ++k) grad[p * gcs + k] = __float2bfloat16(0.f);
            grad[p * gcs] = __float2bfloat16(2.f * d / (float)nvox);
        }
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, s / (float)nvox);
}

// Adam on FP32 master weights; refreshes the BF16 copy
__global__ void k_adam(float *w, const float *__restrict__ gw, float *m, float *v, bf16 *wb, i64 n,
                       float lr, float b1, float b2, float eps, float c1, float c2) {
    for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (i64)gridDim.x * blockDim.x) {
        const float gq = gw[q];
        const float mq = b1 * m[q] + (1.f - b1) * gq;
        const float vq = b2 * v[q] + (1.f - b2) * gq * gq;
        m[q] = mq;
        v[q] = vq;
        const float wq = w[q] - lr * (mq / c1) / (sqrtf(vq / c2) + eps);
        w[q] = wq;
        if (wb) wb[q] = __float2bfloat16(wq);
    }
}

// network input: channel 0 = a[p], channel 1 = b[p], channels 2..15 = 0
__global__ void k_pack2(const float *__restrict__ a, const float *__restrict__ b, bf16 *out, i64 nvox) {
    for (i64 p = (i64)blockIdx.x * blockDim.x + threadIdx.x; p < nvox; p += (i64)gridDim.x * blockDim.x) {
        uint4 u0 = make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<__nv_bfloat162 *>(&u0.x) = __floats2bfloat162_rn(a[p], b[p]);
        uint4 *po = reinterpret_cast<uint4 *>(out + p * 16);
        po[0] = u0;
        po[1] = make_uint4(0u, 0u, 0u, 0u);
    }
}

// f32 out[p] = scale[p / per] * bf16 in[p][c0]
__global__ void k_unpack(const float *__restrict__ in, int cs, int c0, const float *__restrict__ scale,
                         i64 per, float *out, i64 nvox) {
    for (i64 p = (i64)blockIdx.x * blockDim.x + threadIdx.x; p < nvox; p += (i64)gridDim.x * blockDim.x)
        out[p] = in[p * cs + c0] * (scale ? scale[p / per] : 1.f);
}

// x0 in the solver's block-vector layout: x[v * nv + s] = scale[s] * in[s * per + v][c0]
__global__ void k_unpack_x0(const float *__restrict__ in, int cs, int c0, const float *__restrict__ scale,
                            int nv, i64 per, double *x) {
    const i64 total = per * nv;
    for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (i64)gridDim.x * blockDim.x) {
        const i64 v = q / nv;
        const int sidx = (int)(q % nv);
        x[q] = (double)in[(sidx * per + v) * cs + c0] * (double)scale[sidx];
    }
}

// ---------------------------------------------------------------- tcgen05 conv3d
// The same convolution on the 5th-generation tensor cores: implicit GEMM with
// M = 128 voxels, N = BN output channels, K = 16 channels of one tap per
// step.  The 128 threads stage A (the tap's shifted voxel rows) and B (the
// weights) by cp.async exactly as k_conv3d does: 32-byte rows with the
// 16-byte halves swapped on bit 2 of the row, which is the canonical K-major
// SWIZZLE_32B layout of the UMMA shared-memory descriptors (8-row groups 256
// bytes apart).  One thread issues tcgen05.mma (kind::f16, BF16 x BF16 ->
// FP32) into a TMEM accumulator of BN columns and commits each step to the
// stage's mbarrier, which tells the producers when the stage may be
// refilled.  The epilogue reads TMEM with tcgen05.ld (warp w: lanes 32w ..
// 32w+31 = its voxels).  Every mbarrier wait is bounded; on expiry the error
// word is set, the CTA stops issuing and frees its TMEM after the tensor
// pipe has drained (bounded as well).
__device__ int g_tc_err;

__device__ __forceinline__ unsigned long long tc_now() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void tc_mbar_init(unsigned long long *b) {
    asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool tc_mbar_try(unsigned long long *b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool tc_mbar_wait(unsigned long long *b, unsigned parity) {
    if (tc_mbar_try(b, parity)) return true;
    const unsigned long long t0 = tc_now();
    while (!tc_mbar_try(b, parity))
        if (tc_now() - t0 > 1000000000ull) return false;
    return true;
}
// K-major SWIZZLE_32B shared-memory matrix descriptor: start address, leading
// byte offset 1 (unused within one swizzle atom), stride between 8-row groups
// 256 bytes, descriptor version 1, layout type 6
__device__ __forceinline__ unsigned long long tc_desc(const void *p) {
    const unsigned long long a = (smem_u32(p) & 0x3FFFFu) >> 4;
    return a | (1ull << 16) | ((unsigned long long)(256 >> 4) << 32) | (1ull << 46) | (6ull << 61);
}

template <int BN>
__global__ void __launch_bounds__(128) k_conv3d_tc(const bf16 *__restrict__ in, int ics, int ic0, int cin,
                                                   const bf16 *__restrict__ w, const float *__restrict__ bias,
                                                   bf16 *out, int ocs, int oc0, int cout, Vol g, int flags) {
    constexpr int TCOLS = BN < 32 ? 32 : BN;  // TMEM columns (a power of two >= 32)
    __shared__ __align__(1024) unsigned char sa[NS][BM * 32];
    __shared__ __align__(1024) unsigned char sb[NS][BN * 32 < 1024 ? 1024 : BN * 32];
    __shared__ __align__(8) unsigned long long mbar[NS];
    __shared__ unsigned s_tmem;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const i64 nvox = g.count();
    const i64 v0 = (i64)blockIdx.x * BM;
    const int n0 = blockIdx.y * BN;
    const int kc = cin / 16;
    const int nk = 27 * kc;
    const i64 myv = v0 + tid;
    const bool vin = myv < nvox;
    int vx = 0, vy = 0, vz = 0;
    if (vin) {
        vx = (int)(myv % g.w);
        vy = (int)((myv / g.w) % g.h);
        vz = (int)((myv / ((i64)g.w * g.h)) % g.d);
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(TCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int q = 0; q < NS; ++q) tc_mbar_init(&mbar[q]);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_fail = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = s_tmem;
    // instruction descriptor: FP32 accumulator, BF16 A and B, both K-major,
    // N = BN, M = 128
    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(BN >> 3) << 17) | ((128u >> 4) << 24);

    auto stage = [&](int k, int st) {
        const int t = k / kc, cb = (k % kc) * 16;
        const int dz = t / 9 - 1, dy = (t / 3) % 3 - 1, dx = t % 3 - 1;
        const bool inside = vin && (unsigned)(vz + dz) < (unsigned)g.d && (unsigned)(vy + dy) < (unsigned)g.h &&
                            (unsigned)(vx + dx) < (unsigned)g.w;
        const i64 src = inside ? myv + ((i64)dz * g.h + dy) * g.w + dx : -1;
        const bf16 *pa = in + (src < 0 ? 0 : src) * ics + ic0 + cb;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) cp16(&sa[st][sw32(tid, hh)], pa + hh * 8, src < 0 ? 0u : 16u);
        for (int q = tid; q < BN * 2; q += 128) {
            const int r = q >> 1, hh = q & 1;
            const bf16 *pb = w + ((i64)(n0 + r) * 27 + t) * cin + cb + hh * 8;
            cp16(&sb[st][sw32(r, hh)], pb, 16u);
        }
    };
    unsigned uses[NS] = {0u, 0u, 0u, 0u};  // completed MMA phases awaited per stage
    bool ok = true;
#pragma unroll
    for (int q = 0; q < NS - 1; ++q) {
        if (q < nk) stage(q, q);
        cp_commit();
    }
    for (int k = 0; k < nk; ++k) {
        // refill the stage that step k-1 read once its MMA has completed
        const int kn = k + NS - 1;
        if (kn < nk) {
            const int st = kn % NS;
            if (k >= 1) {
                if (ok && !tc_mbar_wait(&mbar[st], uses[st] & 1u)) ok = false;
                uses[st]++;
            }
            stage(kn, st);
        }
        cp_commit();
        cp_wait<NS - 2>();
        // the copies of step k are complete: publish them to the tensor core
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        ok = __syncthreads_and(ok) != 0;
        if (!ok) break;
        if (tid == 0) {
            const int st = k % NS;
            const unsigned long long da = tc_desc(&sa[st][0]), db = tc_desc(&sb[st][0]);
            const unsigned acc = k > 0 ? 1u : 0u;
            asm volatile(
                "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
                "l"(da), "l"(db), "r"(idesc), "r"(acc)
                : "memory");
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&mbar[st]))
                         : "memory");
        }
    }
    cp_wait<0>();
    // the last step's commit completes after every earlier MMA
    if (ok && nk > 0) {
        const int st = (nk - 1) % NS;
        // phases of this stage awaited so far, plus the ones not awaited
        unsigned ph = uses[st];
        for (int k = st; k < nk; k += NS) {
            if ((unsigned)(k / NS) < ph) continue;
            if (!tc_mbar_wait(&mbar[st], (unsigned)(k / NS) & 1u)) { ok = false; break; }
        }
    }
    ok = __syncthreads_and(ok) != 0;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
        const bool relu = flags & 1, accum = flags & 2, f32out = flags & 4;
        const i64 v = v0 + warp * 32 + lane;
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 16) {
            unsigned r[16];
            const unsigned ta = tmem + ((unsigned)(warp * 32) << 16) + (unsigned)c0;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                "[%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                  "=r"(r[15])
                : "r"(ta));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (v >= nvox) continue;
#pragma unroll
            for (int e = 0; e < 16; e += 2) {
                const int n = n0 + c0 + e;
                float y0 = __uint_as_float(r[e]), y1 = __uint_as_float(r[e + 1]);
                if (bias) {
                    y0 += bias[n];
                    y1 += bias[n + 1];
                }
                if (relu) {
                    y0 = fmaxf(y0, 0.f);
                    y1 = fmaxf(y1, 0.f);
                }
                if (f32out) {
                    float2 *pf = reinterpret_cast<float2 *>(reinterpret_cast<float *>(out) + v * ocs + oc0 + n);
                    if (accum) {
                        const float2 o = *pf;
                        y0 += o.x;
                        y1 += o.y;
                    }
                    *pf = make_float2(y0, y1);
                } else {
                    __nv_bfloat162 *po = reinterpret_cast<__nv_bfloat162 *>(out + v * ocs + oc0 + n);
                    if (accum) {
                        const float2 o = __bfloat1622float2(*po);
                        y0 += o.x;
                        y1 += o.y;
                    }
                    *po = __floats2bfloat162_rn(y0, y1);
                }
            }
        }
    } else if (tid == 0) {
        atomicExch(&g_tc_err, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS) : "memory");
    }
}

// the tcgen05 kernel is used when switched on (xcnn_set_tc_conv(1))
int g_tc_conv = 0;

// the box kernel is the default; xcnn_set_box_conv(0) selects the
// voxel-tile kernel (both compute the same convolution)
int g_box_conv = 1;
bool box_conv_enabled() { return g_box_conv != 0; }

int grid_for(i64 n) {
    i64 g = (n + 255) / 256;
    const i64 most = xk::sm_count() * 16;
    return (int)(g < most ? (g < 1 ? 1 : g) : most);
}

int last_err() {
    xk::note_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        fprintf(stderr, "xcnn: %s\n", cudaGetErrorString(e));
        return 3;
    }
    return 0;
}

// all weights stay in shared memory while two CTAs still fit an SM
bool box_weights_resident(int bn, int kc) { return bn < 64 && kc * 27 * bn * 32 <= 56 * 1024; }

// Output channels and depth of the box kernel's CTAs: the pair with the least
// estimated time (SM cycles).  A round is a box of every CTA that fits; its chunk
// takes 27 taps, each no less than the latency of its reads and mma and no less
// than the resident warps' tensor and shared-memory cycles, and the issue of its
// copies: 48 cycles a 16-byte halo piece and 31 a weight piece of a thread, or 40
// and 91 divided among the warps of a scheduler.  All CTAs' copies share the L2 (70
// bytes a cycle and SM); resident weights are copied once.  The numbers minimise
// the loss of the choice over 804 layers (10 channel pairs, 3^3 to 40^3, 1 to 8
// volumes, all pairs timed): it is on average 1 % from the best pair.  The estimate
// before did not see that a small CTA has as many weights to copy as a large one:
// 3 x 24^3, 64 -> 64 took 63 us (bn 32, bz 2), now 49; 5 x 16^3, 128 -> 128 117 and 92;
// 6 x 24^3, 96 -> 32 86 and 60; 8 x 20^3, 16 -> 32 20.4 and 15.9.
struct BoxPlan {
    int bn, bz;
    double t;
};
BoxPlan box_plan(i64 plane, int d, int kc, int cout, int bn0) {
    BoxPlan best{bn0, 8, 1e300};
    const int sms = xk::sm_count();
    for (int bn = bn0; bn >= 16; bn /= 2)
        for (int bz = 8; bz >= 2; bz /= 2) {
            const i64 tasks = plane * ((d + bz - 1) / bz) * (cout / bn);
            const bool res = box_weights_resident(bn, kc);
            const int halo = (bz + 2) * 100 * 32, wb = 27 * bn * 32;
            const int sm = res ? 2 * halo + kc * wb : 2 * (halo + wb);
            const i64 fit = std::max(1, std::min(227 * 1024 / (sm + 2048), (bn == 16 ? 16 : 8) / bz));
            const i64 rounds = (tasks + sms * fit - 1) / (sms * fit);
            const double warps = (double)std::min<i64>(fit, (tasks + sms - 1) / sms) * bz;
            const double tap = std::max(14.0 + 2.0 * bn, 0.8 * warps * (0.79 * bn + 6.5));
            const double pieces = 1.0 / 16 / (32 * bz);  // of a thread, per byte
            const double copy = 260.0 + pieces * (halo * std::max(48.0, 40.0 / 4 * warps) +
                                                  (res ? 0.0 : wb * std::max(31.0, 91.0 / 4 * warps)));
            // a lone CTA on its SM has nobody to compute while it stages
            double t = (double)rounds * kc * (27 * tap + copy) * (fit == 1 ? 1.26 : 1.0) + 1100.0;
            t += 0.014 / sms * (double)tasks * kc * (halo + (res ? 0 : wb));
            if (res) t += 110.0 * pieces * kc * wb;
            if (t < best.t * 0.95) best = {bn, bz, t};
        }
    return best;
}

bool ch_ok(int c) { return c > 0 && c % 16 == 0; }

}  // namespace

extern "C" {

int xcnn_conv3d(const void *in, int ics, int ic0, int cin, const void *w, const float *bias, void *out,
                int ocs, int oc0, int cout, int nb, int d, int h, int wd, int flags, void *stream) {
    if (!ch_ok(cin) || !ch_ok(cout) || ic0 % 16 || oc0 % 16 || ics % 16 || ocs % 16 ||
        ic0 + cin > ics || oc0 + cout > ocs || nb <= 0 || d <= 0 || h <= 0 || wd <= 0)
        return 2;
    Vol g{nb, d, h, wd};
    const i64 nvox = (i64)nb * d * h * wd;
    cudaStream_t s = (cudaStream_t)stream;
    const int bn0 = cout % 64 == 0 ? 64 : (cout % 32 == 0 ? 32 : 16);
    const bf16 *pi = (const bf16 *)in;
    const bf16 *pw = (const bf16 *)w;
    bf16 *po = (bf16 *)out;
    if (g_tc_conv) {
        dim3 grid((unsigned)((nvox + BM - 1) / BM), (unsigned)(cout / bn0));
        if (bn0 == 64) k_conv3d_tc<64><<<grid, 128, 0, s>>>(pi, ics, ic0, cin, pw, bias, po, ocs, oc0, cout, g, flags);
        else if (bn0 == 32) k_conv3d_tc<32><<<grid, 128, 0, s>>>(pi, ics, ic0, cin, pw, bias, po, ocs, oc0, cout, g, flags);
        else k_conv3d_tc<16><<<grid, 128, 0, s>>>(pi, ics, ic0, cin, pw, bias, po, ocs, oc0, cout, g, flags);
        return last_err();
    }
    // box kernel unless padding the volume to boxes costs more than the
    // voxel-tile kernel's steps (one per tap and chunk, about 1300 cycles each
    // while its tiles fill an SM up to three times)
    auto up = [](int n, int m) { return (n + m - 1) / m; };
    const i64 plane = (i64)nb * up(h, 8) * up(wd, 8);
    const BoxPlan bp = box_plan(plane, d, cin / 16, cout, bn0);
    const int bn = bp.bn, bz = bp.bz;
    const i64 nboxes = plane * up(d, bz), tiles = (nvox + BM - 1) / BM * (cout / bn0);
    if (box_conv_enabled() && nboxes <= 0x3fffffff && bp.t < 27.0 * (cin / 16) * 1300.0 * (double)((tiles + 3 * xk::sm_count() - 1) / (3 * xk::sm_count())) &&
        (i64)10 * h * wd * ics <= 0x7fffffff && (i64)wd * ocs <= 0x7fffffff) {
#define LB(BN, BZ, WRES)                                                                                            \
    {                                                                                                               \
        typedef BoxShape<BN, BZ> S;                                                                                 \
        auto k = k_conv3d_box<BN, BZ, WRES>;                                                                        \
        const int sm = WRES ? 2 * S::HBYTES + cin / 16 * S::WBYTES : 2 * (S::HBYTES + S::WBYTES);                   \
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);                                   \
        int per = 0;                                                                                                \
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, S::NT, sm) != cudaSuccess || per < 1) per = 1;    \
        dim3 gb((unsigned)std::max<i64>(1, std::min<i64>(nboxes, (i64)xk::sm_count() * per / (cout / bn))), (unsigned)(cout / bn)); \
        k<<<gb, S::NT, sm, s>>>(pi, ics, ic0, cin, pw, bias, po, ocs, oc0, g, up(wd, 8), up(h, 8), up(d, bz), (int)nboxes, flags); \
    }
#define LBZ(BN, WRES)                                                                                               \
    if (bz == 8) LB(BN, 8, WRES) else if (bz == 4) LB(BN, 4, WRES) else LB(BN, 2, WRES)
        const bool res = box_weights_resident(bn, cin / 16);
        if (bn == 64) LBZ(64, false)
        else if (bn == 32) { if (res) LBZ(32, true) else LBZ(32, false) }
        else { if (res) LBZ(16, true) else LBZ(16, false) }
#undef LBZ
#undef LB
        return last_err();
    }
    dim3 grid((unsigned)((nvox + BM - 1) / BM), (unsigned)(cout / bn0));
    if (bn0 == 64) k_conv3d<64><<<grid, 128, 0, s>>>(pi, ics, ic0, cin, pw, bias, po, ocs, oc0, cout, g, flags);
    else if (bn0 == 32) k_conv3d<32><<<grid, 128, 0, s>>>(pi, ics, ic0, cin, pw, bias, po, ocs, oc0, cout, g, flags);
    else k_conv3d<16><<<grid, 128, 0, s>>>(pi, ics, ic0, cin, pw, bias, po, ocs, oc0, cout, g, flags);
    return last_err();
}

int xcnn_conv3d_wgrad(const void *in, int ics, int ic0, int cin, const void *grad, int gcs, int gc0,
                      int cout, float *dw, int nb, int d, int h, int wd, void *stream) {
    if (!ch_ok(cin) || ic0 % 16 || ics % 16 || gc0 % 16 || gcs % 16 || ic0 + cin > ics ||
        gc0 + cout > gcs || !(cout == 16 || cout == 32 || cout == 64 || cout == 128))
        return 2;
    Vol g{nb, d, h, wd};
    const int nbx = (wd + 7) / 8, nby = (h + 7) / 8, nbz = (d + 1) / 2;
    const i64 nboxes = (i64)nb * nbx * nby * nbz;
    const bool big = nboxes > 0x3fffffff || (i64)3 * h * wd * std::max(ics, gcs) > 0x7fffffff;
    const int co = cout > 64 ? 64 : cout, nci = cin / 16, nco = cout / co;
    // two CTAs per SM (one at 64 channels, whose partial sums fill the register
    // file), shared out over the channel chunks; every CTA has a box
    const i64 want = (i64)xk::sm_count() * (co == 64 ? 1 : 2) / (nci * nco);
    const unsigned slices = (unsigned)std::max<i64>(0, want < 1 ? std::min<i64>(1, nboxes) : std::min(want, nboxes));
    dim3 grid(slices, (unsigned)nci, (unsigned)nco);
    cudaStream_t s = (cudaStream_t)stream;
    const bf16 *pi = (const bf16 *)in;
    const bf16 *pg = (const bf16 *)grad;
#define LW(CO, I)                                                                                                 \
    {                                                                                                             \
        auto k = k_wgrad<CO, I>;                                                                                  \
        const int sm = 2 * WgradShape<CO>::STAGE;                                                                 \
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);                                 \
        k<<<grid, 256, sm, s>>>(pi, ics, ic0, cin, pg, gcs, gc0, dw, g, nbx, nby, nbz, (I)nboxes);                \
    }
#define LWI(I) { if (co == 16) LW(16, I) else if (co == 32) LW(32, I) else LW(64, I) }
    if (big) LWI(i64) else LWI(int)
#undef LWI
#undef LW
    return last_err();
}

int xcnn_weight_flip(const void *w, void *wt, int cout, int cin, void *stream) {
    const i64 n = (i64)cout * 27 * cin;
    k_weight_flip<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>((const bf16 *)w, (bf16 *)wt, cout, cin);
    return last_err();
}

int xcnn_relu_bwd(void *g, int gcs, int gc0, const void *act, int acs, int ac0, int c, int64_t nvox,
                  void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    const bool wide = c % 8 == 0 && gcs % 8 == 0 && gc0 % 8 == 0 && acs % 8 == 0 && ac0 % 8 == 0 &&
                      (uintptr_t)g % 16 == 0 && (uintptr_t)act % 16 == 0;
    if (wide) k_relu_bwd<<<grid_for(nvox * (c / 8)), 256, 0, s>>>((bf16 *)g, gcs, gc0, (const bf16 *)act, acs, ac0, c / 8, nvox);
    else k_relu_bwd1<<<grid_for(nvox * c), 256, 0, s>>>((bf16 *)g, gcs, gc0, (const bf16 *)act, acs, ac0, c, nvox);
    return last_err();
}

int xcnn_bias_grad(const void *g, int gcs, int gc0, int c, int64_t nvox, float *db, void *stream) {
    if (c <= 0 || c > 256 || 256 % c) return 2;
    cudaStream_t s = (cudaStream_t)stream;
    if (c % 8 == 0 && gcs % 8 == 0 && gc0 % 8 == 0 && (uintptr_t)g % 16 == 0 && nvox > 0) {
        // slices of about 64 voxels a thread row, at most four blocks per SM
        const i64 rows = 256 / (c / 8);
        const i64 blocks = std::min<i64>(xk::sm_count() * 4, (nvox + rows * 16 - 1) / (rows * 16));
        const i64 slice = (nvox + blocks - 1) / blocks;
        k_bias_grad<<<(unsigned)((nvox + slice - 1) / slice), 256, 0, s>>>((const bf16 *)g, gcs, gc0, c / 8, nvox, slice, db);
        return last_err();
    }
    const i64 slice = 4096;
    k_bias_grad1<<<(unsigned)((nvox + slice - 1) / slice), 256, 0, s>>>((const bf16 *)g, gcs, gc0, c, nvox, slice, db);
    return last_err();
}

int xcnn_pool2(const void *in, int ics, int ic0, void *out, int ocs, int oc0, int c, int nb, int d, int h,
               int w, void *stream) {
    if (d % 2 || h % 2 || w % 2 || c % 8 || ic0 % 8 || ics % 8 || oc0 % 8 || ocs % 8) return 2;
    Vol g{nb, d, h, w};
    k_pool2<<<grid_for(g.count() / 8 * (c / 8)), 256, 0, (cudaStream_t)stream>>>((const bf16 *)in, ics, ic0,
                                                                              (bf16 *)out, ocs, oc0, c, g);
    return last_err();
}

// fine volume (nb, d, h, w): mode 0 out = up(in); mode 1 out += up(in) / 8
int xcnn_up2(const void *in, int ics, int ic0, void *out, int ocs, int oc0, int c, int nb, int d, int h,
             int w, int mode, void *stream) {
    if (d % 2 || h % 2 || w % 2 || c % 8 || ic0 % 8 || ics % 8 || oc0 % 8 || ocs % 8) return 2;
    Vol g{nb, d, h, w};
    k_up2<<<grid_for(g.count() / 8 * (c / 8)), 256, 0, (cudaStream_t)stream>>>((const bf16 *)in, ics, ic0,
                                                                                 (bf16 *)out, ocs, oc0, c, g, mode);
    return last_err();
}

int xcnn_up2_bwd(const void *gfine, int gcs, int gc0, void *gin, int ics, int ic0, int c, int nb, int d,
                 int h, int w, void *stream) {
    if (d % 2 || h % 2 || w % 2 || c % 8 || gc0 % 8 || gcs % 8 || ic0 % 8 || ics % 8) return 2;
    Vol g{nb, d, h, w};
    k_up2_bwd<<<grid_for(g.count() / 8 * (c / 8)), 256, 0, (cudaStream_t)stream>>>(
        (const bf16 *)gfine, gcs, gc0, (bf16 *)gin, ics, ic0, c, g);
    return last_err();
}

int xcnn_mse(const void *pred, int pcs, int pc0, const float *tgt, void *grad, int gcs, int64_t nvox,
             float *loss, void *stream) {
    k_mse<<<grid_for(nvox), 256, 0, (cudaStream_t)stream>>>((const float *)pred, pcs, pc0, tgt, (bf16 *)grad,
                                                            gcs, nvox, loss);
    return last_err();
}

int xcnn_adam(float *w, const float *g, float *m, float *v, void *wb, int64_t n, float lr, float b1,
              float b2, float eps, int step, void *stream) {
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_adam<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(w, g, m, v, (bf16 *)wb, n, lr, b1, b2, eps, c1, c2);
    return last_err();
}

int xcnn_pack2(const float *a, const float *b, void *out, int64_t nvox, void *stream) {
    k_pack2<<<grid_for(nvox), 256, 0, (cudaStream_t)stream>>>(a, b, (bf16 *)out, nvox);
    return last_err();
}

int xcnn_unpack(const void *in, int cs, int c0, const float *scale, int64_t per, float *out, int64_t nvox,
                void *stream) {
    k_unpack<<<grid_for(nvox), 256, 0, (cudaStream_t)stream>>>((const float *)in, cs, c0, scale, per, out, nvox);
    return last_err();
}

int xcnn_unpack_x0(const void *in, int cs, int c0, const float *scale, int nv, int64_t per, double *x,
                   void *stream) {
    if (nv <= 0 || per <= 0 || !scale) return 2;
    k_unpack_x0<<<grid_for(per * nv), 256, 0, (cudaStream_t)stream>>>((const float *)in, cs, c0, scale, nv, per, x);
    return last_err();
}

int xcnn_set_tc_conv(int on) {
    const int old = g_tc_conv;
    g_tc_conv = on != 0;
    return old;
}
// 1 when a tcgen05 convolution gave up waiting on its tensor pipe since the
// last call (then cleared)
int xcnn_tc_error() {
    int h = 0;
    if (cudaMemcpyFromSymbol(&h, g_tc_err, sizeof(int)) != cudaSuccess) return -1;
    const int z = 0;
    if (h) cudaMemcpyToSymbol(g_tc_err, &z, sizeof(int));
    return h;
}
int xcnn_set_box_conv(int on) {
    const int old = g_box_conv;
    g_box_conv = on != 0;
    return old;
}

}  // extern "C"
