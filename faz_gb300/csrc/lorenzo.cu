// lorenzo.cu - the Lorenzo fast frontend for 3-D fields on the GPU
// (SZFastFrontend, include/QoZ/frontend/SZFastFrontend.hpp:170-437, with
// MetaLorenzoPredictor.hpp) and its stream section (save/load, lines 48-128).
//
// The reference walks blocks of bs^3 points in row-major order and predicts
// every point from reconstructed neighbours (one- or two-layer Lorenzo, chosen
// per block from the original data), keeping the reconstruction in a slab
// buffer padded with zeros.  That is the same as predicting from a full
// reconstructed field that reads as zero before the first plane, row and
// column, so a block depends only on its seven neighbours with smaller or equal
// block coordinates, and a block predicted by regression on none.  One launch of
// persistent warps takes the blocks diagonal by diagonal (bi + bj + bk), one warp
// per block.  Inside a Lorenzo block the warp walks the point diagonals
// i + j + k = s in a shared-memory tile that holds the block and its halo.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <functional>
#include <string>
#include <vector>

#include "common.cuh"
#include "host.h"
#include "internal.h"
#include "quant.cuh"

namespace faz {

namespace {

constexpr int kLorWarps = 8;     // blocks (warps) per CTA
constexpr int kLorMaxBs = 8;     // largest block edge on the GPU path
constexpr int kLorBatch = 8;     // tile loads in flight per lane
constexpr int kLorMaxRadius = 65536;  // quantbinCnt up to 131072 (32-bit codes above 65536 bins)

struct LorArgs {
    int64_t d1, d2, d3;   // field dims, slowest first
    int64_t nx, ny, nz;   // blocks per dim
    int bs;               // block edge
    int pd;               // prediction dimension (1, 2, 3)
    int lo, lo2;          // one- / two-layer Lorenzo allowed
    int reg;              // linear regression allowed
    const float *rp;      // per block: the 4 reconstructed regression coefficients
    LevelArgs q;          // quantiser (eb, 1/eb, radius, float split)
};

// MetaLorenzoPredictor.hpp:8-73 on a tile with strides (tx, ty, 1)
template <typename T>
__device__ __forceinline__ T lor_pred(const T *p, int tx, int ty, int pd, bool two) {
    if (two) {
        if (pd == 3)
            return (T)2 * p[-1] - p[-2] + (T)2 * p[-ty] - (T)4 * p[-ty - 1] + (T)2 * p[-ty - 2] - p[-2 * ty] +
                   (T)2 * p[-2 * ty - 1] - p[-2 * ty - 2] + (T)2 * p[-tx] - (T)4 * p[-tx - 1] + (T)2 * p[-tx - 2] -
                   (T)4 * p[-tx - ty] + (T)8 * p[-tx - ty - 1] - (T)4 * p[-tx - ty - 2] + (T)2 * p[-tx - 2 * ty] -
                   (T)4 * p[-tx - 2 * ty - 1] + (T)2 * p[-tx - 2 * ty - 2] - p[-2 * tx] + (T)2 * p[-2 * tx - 1] -
                   p[-2 * tx - 2] + (T)2 * p[-2 * tx - ty] - (T)4 * p[-2 * tx - ty - 1] + (T)2 * p[-2 * tx - ty - 2] -
                   p[-2 * tx - 2 * ty] + (T)2 * p[-2 * tx - 2 * ty - 1] - p[-2 * tx - 2 * ty - 2];
        if (pd == 2)
            return (T)2 * p[-tx] - p[-2 * tx] + (T)2 * p[-1] - (T)4 * p[-1 - tx] + (T)2 * p[-1 - 2 * tx] - p[-2] +
                   (T)2 * p[-2 - tx] - p[-2 - 2 * tx];
        return (T)2 * p[-1] - p[-2];
    }
    if (pd == 3) return p[-1] + p[-ty] + p[-tx] - p[-ty - 1] - p[-tx - 1] - p[-tx - ty] + p[-tx - ty - 1];
    if (pd == 2) return p[-1] + p[-tx] - p[-1 - tx];
    return p[-1];
}

// The same predictors on the original field (strides d0, d1, 1), returned in T
template <typename T>
__device__ __forceinline__ T lor_pred_g(const T *p, int64_t d0, int64_t d1, int pd, bool two) {
    if (two) {
        if (pd == 3)
            return (T)2 * p[-1] - p[-2] + (T)2 * p[-d1] - (T)4 * p[-d1 - 1] + (T)2 * p[-d1 - 2] - p[-2 * d1] +
                   (T)2 * p[-2 * d1 - 1] - p[-2 * d1 - 2] + (T)2 * p[-d0] - (T)4 * p[-d0 - 1] + (T)2 * p[-d0 - 2] -
                   (T)4 * p[-d0 - d1] + (T)8 * p[-d0 - d1 - 1] - (T)4 * p[-d0 - d1 - 2] + (T)2 * p[-d0 - 2 * d1] -
                   (T)4 * p[-d0 - 2 * d1 - 1] + (T)2 * p[-d0 - 2 * d1 - 2] - p[-2 * d0] + (T)2 * p[-2 * d0 - 1] -
                   p[-2 * d0 - 2] + (T)2 * p[-2 * d0 - d1] - (T)4 * p[-2 * d0 - d1 - 1] + (T)2 * p[-2 * d0 - d1 - 2] -
                   p[-2 * d0 - 2 * d1] + (T)2 * p[-2 * d0 - 2 * d1 - 1] - p[-2 * d0 - 2 * d1 - 2];
        if (pd == 2)
            return (T)2 * p[-d0] - p[-2 * d0] + (T)2 * p[-1] - (T)4 * p[-1 - d0] + (T)2 * p[-1 - 2 * d0] - p[-2] +
                   (T)2 * p[-2 - d0] - p[-2 - 2 * d0];
        return (T)2 * p[-1] - p[-2];
    }
    if (pd == 3) return p[-1] + p[-d1] + p[-d0] - p[-d1 - 1] - p[-d0 - 1] - p[-d0 - d1] + p[-d0 - d1 - 1];
    if (pd == 2) return p[-1] + p[-d0] - p[-1 - d0];
    return p[-1];
}

// meta_block_error_estimation_3d for one point (SZFastFrontend.hpp:440-495),
// regression off.  Noise constants from include/QoZ/utils/MetaDef.hpp:24-29.
template <typename T>
__device__ __forceinline__ void meta_est(const T *c, int64_t d0, int64_t d1, T prec, int pd, int lo, int lo2,
                                         double &el, double &el2) {
    const T cd = *c;
    double lp = 0, lp2 = 0;
    T noise = 0, noise2 = 0;
    const double n1 = pd == 3 ? 1.22 : (pd == 2 ? 0.81 : 0.5);
    const double n2 = pd == 3 ? 6.8 : (pd == 2 ? 2.76 : 1.08);
    if (lo2) {
        lp2 = (double)lor_pred_g(c, d0, d1, pd, true);
        noise2 = (T)(n2 * (double)prec);
    }
    if (lo) {
        lp = (double)lor_pred_g(c, d0, d1, pd, false);
        noise = (T)(n1 * (double)prec);
    }
    el += fabs((double)cd - lp) + (double)noise;
    el2 += fabs((double)cd - lp2) + (double)noise2;
}

// compute_regression_coeffcients_3d (MetaRegressionPredictor.hpp:104-139),
// float sums in the reference's loop order.
template <typename T>
__device__ void reg_coeffs(const T *d, int sx, int sy, int sz, int64_t d0, int64_t d1, float *rp) {
    const T *cur = d;
    float fx = 0.0f, fy = 0.0f, fz = 0.0f, f = 0;
    for (int i = 0; i < sx; i++) {
        float sum_x = 0;
        for (int j = 0; j < sy; j++) {
            float sum_y = 0;
            for (int k = 0; k < sz; k++) {
                const T cd = *cur;
                sum_y = (float)(sum_y + cd);
                fz = (float)(fz + (T)(cd * (T)k));
                cur++;
            }
            fy += sum_y * (float)j;
            sum_x += sum_y;
            cur += (d1 - sz);
        }
        fx += sum_x * (float)i;
        f += sum_x;
        cur += (d0 - sy * d1);
    }
    const float coeff = (float)(1.0 / (sx * sy * sz));
    rp[0] = (2 * fx / (float)(sx - 1) - f) * 6 * coeff / (float)(sx + 1);
    rp[1] = (2 * fy / (float)(sy - 1) - f) * 6 * coeff / (float)(sy + 1);
    rp[2] = (2 * fz / (float)(sz - 1) - f) * 6 * coeff / (float)(sz + 1);
    rp[3] = f * coeff - ((float)(sx - 1) * rp[0] / 2 + (float)(sy - 1) * rp[1] / 2 + (float)(sz - 1) * rp[2] / 2);
}

// meta_blockwise_selection_3d (SZFastFrontend.hpp:498-540), one thread per
// block: 0 Lorenzo, 1 regression, 2 two-layer Lorenzo.  The block's raw
// regression coefficients go to raw[4b..4b+3].
template <typename T>
__global__ void k_lor_select(LorArgs a, const T *__restrict__ X, uint16_t *__restrict__ ind, float *__restrict__ raw) {
    const int64_t nb = a.nx * a.ny * a.nz;
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const int64_t bk = b % a.nz, bj = (b / a.nz) % a.ny, bi = b / (a.nz * a.ny);
    const int bs = a.bs;
    const int sx = (bi + 1) * bs < a.d1 ? bs : (int)(a.d1 - bi * bs);
    const int sy = (bj + 1) * bs < a.d2 ? bs : (int)(a.d2 - bj * bs);
    const int sz = (bk + 1) * bs < a.d3 ? bs : (int)(a.d3 - bk * bs);
    int ms = sx < sy ? sx : sy;
    ms = ms < sz ? ms : sz;
    const int64_t d0 = a.d2 * a.d3, d1 = a.d3;
    const T *dp = X + bi * bs * d0 + bj * bs * d1 + bk * bs;
    const T prec = (T)a.q.eb;
    const bool ereg = a.reg && ms >= 2;
    float rp[4] = {0, 0, 0, 0};
    if (ereg) reg_coeffs(dp, sx, sy, sz, d0, d1, rp);
    double el = 0, el2 = 0, er = 0;
    auto est = [&](int x, int y, int z) {
        const T *c = dp + x * d0 + y * d1 + z;
        if (ereg) {
            // regression_predict_3d<T> (MetaRegressionPredictor.hpp:142-146)
            const T pr = (T)(rp[0] * (float)x + rp[1] * (float)y + rp[2] * (float)z + rp[3]);
            const T df = *c - pr;
            er += (double)(df < 0 ? -df : df);
        }
        meta_est(c, d0, d1, prec, a.pd, a.lo, a.lo2, el, el2);
    };
    for (int i = 2; i < ms - 1; i++) {
        const int m = ms - i;
        est(i, i, i);
        est(i, i, m);
        est(i, m, i);
        est(i, m, m);
    }
    if (ms > 3) est(ms - 1, ms - 1, ms - 1);
    int sel;
    if (ereg && (!a.lo || er <= el) && (!a.lo2 || er < el2)) sel = 1;
    else if (a.lo2 && (!a.lo || el2 <= el) && (!ereg || el2 <= er)) sel = 2;
    else sel = 0;
    ind[b] = (uint16_t)sel;
    if (raw) {
        for (int c = 0; c < 4; c++) raw[4 * b + c] = rp[c];
    }
}

// Loads with the L2 as the point of coherence: the wavefront reads blocks
// that other SMs wrote during the same launch, and L1 is not coherent.
template <typename T>
__device__ __forceinline__ T ld_coherent(const T *p) {
    return __ldcg(p);
}

__device__ __forceinline__ void lor_st_release(unsigned *p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ unsigned lor_ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Extents of block (bi, bj, bk) and its place in the field and the stream.
struct LorBlock {
    int sx, sy, sz;
    int64_t g0;     // element of its first point
    uint64_t pos0;  // stream position of its first code
    bool full;
};
__device__ __forceinline__ LorBlock lor_geom(const LorArgs &a, int64_t bi, int64_t bj, int64_t bk) {
    LorBlock b;
    const int bs = a.bs;
    b.sx = (bi + 1) * bs < a.d1 ? bs : (int)(a.d1 - bi * bs);
    b.sy = (bj + 1) * bs < a.d2 ? bs : (int)(a.d2 - bj * bs);
    b.sz = (bk + 1) * bs < a.d3 ? bs : (int)(a.d3 - bk * bs);
    const int64_t d0 = a.d2 * a.d3;
    b.g0 = bi * bs * d0 + bj * bs * a.d3 + bk * bs;
    b.pos0 = (uint64_t)(bi * bs) * (uint64_t)d0 + (uint64_t)(bj * bs) * (uint64_t)(b.sx * a.d3) +
             (uint64_t)(bk * bs) * (uint64_t)(b.sx * b.sy);
    b.full = b.sx == bs && b.sy == bs && b.sz == bs;
    return b;
}

// Tables of a full block, built once per CTA: lin[e] = i | j << 4 | k << 8 of
// linear point e; pts the same of the points by diagonal i + j + k (soff: first
// of each, then their number); halo[h] = i | j << 4 | k << 8 | tile index << 12 of the halo cells of
// the (bs + 2)^3 tile, the one-deep ones (coordinates >= 1) first.
struct LorTables {
    const uint16_t *lin, *pts, *soff;
    const uint32_t *halo;
    int n1, nh;  // one-deep halo cells, all of them
};
constexpr int kLorSteps = 3 * kLorMaxBs;
__host__ __device__ constexpr int lor_table_bytes(int bs) {
    return (4 * ((bs + 2) * (bs + 2) * (bs + 2) - bs * bs * bs) + 2 * (2 * bs * bs * bs + kLorSteps) + 3) / 4 * 4;
}

__device__ __forceinline__ LorTables lor_tables(int bs, unsigned char *mem) {
    __shared__ int cur[kLorSteps], hcur[2];
    const int n = bs * bs * bs, te = bs + 2, tn = te * te * te;
    LorTables t;
    t.n1 = (bs + 1) * (bs + 1) * (bs + 1) - n;
    t.nh = tn - n;
    uint32_t *halo = reinterpret_cast<uint32_t *>(mem);
    uint16_t *lin = reinterpret_cast<uint16_t *>(halo + t.nh), *pts = lin + n, *soff = pts + n;
    for (int i = threadIdx.x; i < kLorSteps; i += blockDim.x) cur[i] = 0;
    if (threadIdx.x < 2) hcur[threadIdx.x] = threadIdx.x ? t.n1 : 0;
    __syncthreads();
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const int i = e / (bs * bs), j = (e / bs) % bs, k = e % bs;
        lin[e] = (uint16_t)(i | (j << 4) | (k << 8));
        atomicAdd(&cur[i + j + k], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int sum = 0;
        for (int d = 0; d < kLorSteps; d++) {
            const int c = cur[d];
            soff[d] = (uint16_t)sum;
            cur[d] = sum;
            sum += c;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const int v = lin[e];
        pts[atomicAdd(&cur[(v & 15) + ((v >> 4) & 15) + (v >> 8)], 1)] = (uint16_t)v;
    }
    for (int e = threadIdx.x; e < tn; e += blockDim.x) {
        const int i = e / (te * te), j = (e / te) % te, k = e % te;
        if (i >= 2 && j >= 2 && k >= 2) continue;
        const int at = atomicAdd(&hcur[i >= 1 && j >= 1 && k >= 1 ? 0 : 1], 1);
        halo[at] = (uint32_t)i | ((uint32_t)j << 4) | ((uint32_t)k << 8) | ((uint32_t)e << 12);
    }
    __syncthreads();
    t.lin = lin;
    t.pts = pts;
    t.soff = soff;
    t.halo = halo;
    return t;
}

// the code kept in the slot of point e's value
template <typename T>
__device__ __forceinline__ unsigned *lor_code(T *xs, int e) {
    return reinterpret_cast<unsigned *>(xs + e);
}

// What a block needs of its own, before any neighbour is done: its original
// values (compression), or its codes (decompression; a load per point diagonal
// would put a memory round trip on each of the block's steps), in linear order or
// at slot[e].
template <typename T, bool DECOMP, typename C>
__device__ __forceinline__ void lor_load_own(const LorArgs &a, const LorBlock &b, const LorTables &tb,
                                             const uint16_t *slot, T *xs, const T *__restrict__ X,
                                             const C *__restrict__ codes) {
    const int lane = threadIdx.x & 31;
    const int64_t d0 = a.d2 * a.d3;
    const int nv = b.sx * b.sy * b.sz;
    for (int e0 = lane; e0 < nv; e0 += 32 * kLorBatch) {
        T v[kLorBatch];
        unsigned c[kLorBatch];
#pragma unroll
        for (int u = 0; u < kLorBatch; u++) {
            const int e = e0 + 32 * u;
            v[u] = 0;
            c[u] = 0;
            if (e >= nv) continue;
            if (DECOMP) {
                c[u] = codes[b.pos0 + e];
            } else if (b.full) {
                const int p = tb.lin[e];
                v[u] = X[b.g0 + (p & 15) * d0 + ((p >> 4) & 15) * a.d3 + (p >> 8)];
            } else {
                const int i = e / (b.sy * b.sz), r = e - i * b.sy * b.sz, j = r / b.sz, k = r - j * b.sz;
                v[u] = X[b.g0 + i * d0 + j * a.d3 + k];
            }
        }
#pragma unroll
        for (int u = 0; u < kLorBatch; u++) {
            if (e0 + 32 * u >= nv) continue;
            const int e = slot ? slot[e0 + 32 * u] : e0 + 32 * u;
            if (DECOMP) *lor_code<T>(xs, e) = c[u];
            else xs[e] = v[u];
        }
    }
}

// The halo of reconstructed values in the tile: one deep, two for the two-layer
// predictor; zero outside the field.
template <typename T>
__device__ __forceinline__ void lor_load_halo(const LorArgs &a, const LorBlock &b, const LorTables &tb, T *t,
                                              int64_t bi, int64_t bj, int64_t bk, bool two, const T *__restrict__ R) {
    const int lane = threadIdx.x & 31;
    const int64_t x0 = bi * a.bs, y0 = bj * a.bs, z0 = bk * a.bs, d0 = a.d2 * a.d3;
    // loads in batches of kLorBatch per lane, all issued before any is used
    if (b.full) {
        const int nh = two ? tb.nh : tb.n1;
        for (int h0 = lane; h0 < nh; h0 += 32 * kLorBatch) {
            T v[kLorBatch];
            uint32_t q[kLorBatch];
#pragma unroll
            for (int u = 0; u < kLorBatch; u++) {
                const int h = h0 + 32 * u;
                q[u] = h < nh ? tb.halo[h] : 0u;
                const int i = (int)(q[u] & 15u) - 2, j = (int)((q[u] >> 4) & 15u) - 2, k = (int)((q[u] >> 8) & 15u) - 2;
                v[u] = (h < nh && x0 + i >= 0 && y0 + j >= 0 && z0 + k >= 0)
                           ? ld_coherent(R + (b.g0 + i * d0 + j * a.d3 + k))
                           : (T)0;
            }
#pragma unroll
            for (int u = 0; u < kLorBatch; u++)
                if (h0 + 32 * u < nh) t[q[u] >> 12] = v[u];
        }
        return;
    }
    const int tz = b.sz + 2, tx = (b.sy + 2) * tz, tn = (b.sx + 2) * tx, lo = two ? 0 : 1;
    for (int e0 = lane; e0 < tn; e0 += 32 * kLorBatch) {
        T v[kLorBatch];
#pragma unroll
        for (int u = 0; u < kLorBatch; u++) {
            const int e = e0 + 32 * u;
            const int i = e / tx, r = e - i * tx, j = r / tz, k = r - j * tz;
            const bool cell = e < tn && (i < 2 || j < 2 || k < 2) && i >= lo && j >= lo && k >= lo;
            v[u] = (cell && x0 + i >= 2 && y0 + j >= 2 && z0 + k >= 2)
                       ? ld_coherent(R + (b.g0 + (i - 2) * d0 + (j - 2) * a.d3 + (k - 2)))
                       : (T)0;
        }
#pragma unroll
        for (int u = 0; u < kLorBatch; u++)
            if (e0 + 32 * u < tn) t[e0 + 32 * u] = v[u];
    }
}

// One block, one warp: a Lorenzo block's points diagonal by diagonal, each
// predicted from its reconstructed neighbours in the tile; a regression block's
// points all at once.
template <typename T, bool DECOMP, int QM, typename C>
__device__ __forceinline__ void lor_block(const LorArgs &a, const LorBlock &b, const LorTables &tb, T *t, T *xs,
                                          int sel, const float (&rp)[4], T *__restrict__ R, C *__restrict__ codes,
                                          T *__restrict__ scratch, const uint64_t *__restrict__ zpos, uint64_t nzp,
                                          const T *__restrict__ unpred) {
    const int lane = threadIdx.x & 31;
    const int64_t d0 = a.d2 * a.d3;
    // tile strides: (tx, ty, 1) over (sx + 2) x (sy + 2) x (sz + 2)
    const int ty = b.sz + 2, tx = (b.sy + 2) * ty;
    auto point = [&](int i, int j, int k, int e, T pred) -> T {
        const uint64_t pos = b.pos0 + (uint64_t)e;
        T v;
        if (!DECOMP) {
            v = xs[e];
            T uval;
            const int code = quant_point<T, QM>(v, pred, a.q, uval);
            codes[pos] = (C)code;
            if (code == 0) scratch[pos] = uval;
        } else {
            v = recover_point<T, QM>(pred, (int)*lor_code<T>(xs, e), pos, a.q, zpos, nzp, unpred);
        }
        R[b.g0 + i * d0 + j * a.d3 + k] = v;
        return v;
    };
    if (sel == 1) {
        const int nv = b.sx * b.sy * b.sz;
        for (int e = lane; e < nv; e += 32) {
            int i, j, k;
            if (b.full) {
                const int p = tb.lin[e];
                i = p & 15;
                j = (p >> 4) & 15;
                k = p >> 8;
            } else {
                i = e / (b.sy * b.sz);
                const int r = e - i * b.sy * b.sz;
                j = r / b.sz;
                k = r - j * b.sz;
            }
            // regression_predict_quantize_3d (MetaRegressionPredictor.hpp:148-189)
            point(i, j, k, e, (T)(rp[0] * (float)i + rp[1] * (float)j + rp[2] * (float)k + rp[3]));
        }
        return;
    }
    const bool two = sel == 2;
    const int nsteps = b.sx + b.sy + b.sz - 2;
    for (int s = 0; s < nsteps; s++) {
        for (int q = tb.soff[s] + lane; q < tb.soff[s + 1]; q += 32) {
            const int p = tb.pts[q], i = p & 15, j = (p >> 4) & 15, k = p >> 8;
            if (i >= b.sx || j >= b.sy || k >= b.sz) continue;
            T *c = t + (i + 2) * tx + (j + 2) * ty + (k + 2);
            *c = point(i, j, k, (i * b.sy + j) * b.sz + k, lor_pred(c, tx, ty, a.pd, two));
        }
        __syncwarp();
    }
}

// Tables of the fast path for full one-layer 3-D Lorenzo blocks of edge BS, whose
// diagonals have a lane per point; step s of lane l is at 32 * s + l: the point's
// tile index (at) and its element offset from the block's first point (off, < 0:
// no point); its value or code is at the same place in xs.
// slot[e]: the step of linear point e.  The halo cells of a lane, in registers:
// tile index and element offset, and which of the three neighbours behind they
// need (a cell outside the field reads zero).
template <int BS>
struct LorFast {
    static constexpr int kSteps = 3 * BS - 2;
    static constexpr int kSlots = 32 * kSteps;
    static constexpr int kHalo = ((BS + 1) * (BS + 1) * (BS + 1) - BS * BS * BS + 31) / 32;
    const int *at, *off;
    const uint16_t *slot;
    int hat[kHalo], hoff[kHalo];
    unsigned hneed[kHalo];
};
template <>
struct LorFast<0> {};
// bytes of the tables above, and of a warp's values in step order (0: no fast path)
constexpr bool lor_has_fast(int bs) { return bs == 5 || bs == 6; }
constexpr int lor_fast_bytes(int bs) {
    return lor_has_fast(bs) ? 8 * 32 * (3 * bs - 1) + 2 * ((bs * bs * bs + 1) / 2 * 2) : 0;
}
constexpr int lor_own(int bs) { return lor_has_fast(bs) ? 32 * (3 * bs - 2) : bs * bs * bs; }

template <int BS>
__device__ __forceinline__ void lor_fast_tables(const LorArgs &a, const LorTables &tb, unsigned char *mem,
                                                LorFast<BS> &f) {
    const int d0 = (int)(a.d2 * a.d3), d1 = (int)a.d3;
    int *at = reinterpret_cast<int *>(mem), *off = at + 32 * (f.kSteps + 1);
    uint16_t *slot = reinterpret_cast<uint16_t *>(off + 32 * (f.kSteps + 1));
    for (int i = threadIdx.x; i < 32 * (f.kSteps + 1); i += blockDim.x) {
        const int s = i >> 5, q = tb.soff[s] + (i & 31);
        at[i] = ((BS + 2) * (BS + 2) + BS + 2 + 1) * 2;  // any point of the block
        off[i] = -1;
        if (s < f.kSteps && q < tb.soff[s + 1]) {
            const int p = tb.pts[q], x = p & 15, y = (p >> 4) & 15, z = p >> 8;
            at[i] = ((x + 2) * (BS + 2) + y + 2) * (BS + 2) + z + 2;
            off[i] = x * d0 + y * d1 + z;
            slot[(x * BS + y) * BS + z] = (uint16_t)i;
        }
    }
#pragma unroll
    for (int u = 0; u < f.kHalo; u++) {
        const int h = (threadIdx.x & 31) + 32 * u;
        f.hat[u] = -1;
        f.hoff[u] = 0;
        f.hneed[u] = 0;
        if (h < tb.n1) {
            const uint32_t q = tb.halo[h];
            const int x = (int)(q & 15u) - 2, y = (int)((q >> 4) & 15u) - 2, z = (int)((q >> 8) & 15u) - 2;
            f.hat[u] = (int)(q >> 12);
            f.hoff[u] = x * d0 + y * d1 + z;
            f.hneed[u] = (x < 0 ? 1u : 0u) | (y < 0 ? 2u : 0u) | (z < 0 ? 4u : 0u);
        }
    }
    f.at = at;
    f.off = off;
    f.slot = slot;
    __syncthreads();
}

// One such block: a step is the seven neighbours, the prediction, the quantiser
// and two stores, everything else read a step ahead.  No lane branches away (a
// lane without a point computes on another's and stores nothing).  The loop is
// not unrolled: straight-line code for 16 steps misses the instruction cache
// (2.6 ms for the wavefront of a 100x500x500 field without regression, 1.8 ms this
// way).
template <typename T, bool DECOMP, int QM, int BS>
__device__ __forceinline__ void lor_full(const LorArgs &a, const LorBlock &b, const LorFast<BS> &f, T *t, T *xs,
                                         T *__restrict__ R, T *__restrict__ scratch,
                                         const uint64_t *__restrict__ zpos, uint64_t nzp,
                                         const T *__restrict__ unpred) {
    constexpr int ty = BS + 2, tx = ty * ty;
    const int lane = threadIdx.x & 31;
    const int *at = f.at + lane, *off = f.off + lane;
    T *x = xs + lane, *r0 = R + b.g0;
    int an = at[0], on = off[0];
    T xn = x[0];
#pragma unroll 1
    for (int s = 0; s < f.kSteps; s++) {
        T *c = t + an;
        const int o = on;
        T v = xn;
        T pred = c[-1] + c[-ty] + c[-tx] - c[-ty - 1] - c[-tx - 1] - c[-tx - ty] + c[-tx - ty - 1];
        an = at[32 * s + 32];
        on = off[32 * s + 32];
        if (s + 1 < f.kSteps) xn = x[32 * s + 32];
        if (!DECOMP) {
            if (o < 0) v = pred = (T)0;
            T uval;
            const int code = quant_point<T, QM>(v, pred, a.q, uval);
            *lor_code<T>(x, 32 * s) = (unsigned)code;
            // positions in the unpredictable values: the e-th of the block
            if (o >= 0 && code == 0) {
                const int d0 = (int)(a.d2 * a.d3), d1 = (int)a.d3, i = o / d0, j = (o - i * d0) / d1;
                scratch[b.pos0 + (i * BS + j) * BS + (o - i * d0 - j * d1)] = uval;
            }
        } else {
            unsigned code;
            std::memcpy(&code, &v, 4);
            if (o < 0) {
                code = (unsigned)a.q.radius;
                pred = (T)0;
            }
            uint64_t pos = b.pos0;
            if (code == 0) {
                const int d0 = (int)(a.d2 * a.d3), d1 = (int)a.d3, i = o / d0, j = (o - i * d0) / d1;
                pos += (i * BS + j) * BS + (o - i * d0 - j * d1);
            }
            v = recover_point<T, QM>(pred, (int)code, pos, a.q, zpos, nzp, unpred);
        }
        if (o >= 0) {
            *c = v;
            r0[o] = v;
        }
        __syncwarp();
    }
}

constexpr unsigned kLorWaitLimit = 1u << 22;  // polls (with back-off) of a block's neighbours before giving up

// The whole wavefront in one launch of persistent CTAs.  A warp takes a
// ticket, and with it the block order[ticket]: blocks come diagonal by diagonal
// (bi + bj + bk ascending).  A Lorenzo block waits for the seven neighbours it
// reads; they hold smaller tickets, taken by warps already running, so every
// wait ends.  A regression block reads none and waits for none.  Each wait is
// bounded all the same (error flag, then the block runs).  A finished block
// publishes done[b] = 1 with release semantics after its reconstruction is
// written.
//
// Bound by the latency of the longest chain of Lorenzo blocks (up to the 185
// diagonals of the 17 x 84 x 84 blocks of a 100x500x500 field), so what is on a
// block's path counts.  A diagonal of points is one step, a lane per point (27 at
// most for edge 6; a lane per (i, j) pair took two steps); the halo is one deep
// unless the two-layer predictor reads it; values and codes are on the SM before
// the wait; neighbours are polled with acquire loads and the flag is one release
// store after a warp barrier (a fence per lane on either side took 1,050 cycles
// each); codes are written after the flag.  The wavefront of that field with
// regression: 3.18 -> 1.45 ms, 3.49 -> 1.37 ms in decompression; a block on the
// path takes 8,000 cycles for its 16 steps, 1,750 for the halo, 1,150 to publish.
// BS: the block edge of lor_full's path, 0 for other edges.
template <typename T, bool DECOMP, int QM, typename C, int BS>
__global__ void __launch_bounds__(kLorWarps * 32, 2)
    k_lor_persist(LorArgs a, const uint32_t *__restrict__ order, uint32_t nblocks, unsigned *counter,
                  unsigned *done, int *err, const T *__restrict__ X, T *__restrict__ R,
                  C *__restrict__ codes, T *__restrict__ scratch, const uint16_t *__restrict__ ind,
                  const uint64_t *__restrict__ zpos, uint64_t nzp, const T *__restrict__ unpred) {
    extern __shared__ __align__(16) unsigned char lor_smem[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bs = BS ? BS : a.bs;
    const int tile = (bs + 2) * (bs + 2) * (bs + 2), tstride = tile + (BS ? lor_own(BS) : bs * bs * bs);
    T *t = reinterpret_cast<T *>(lor_smem) + (size_t)w * (size_t)tstride;
    T *xs = t + tile;
    const LorTables tb = lor_tables(bs, lor_smem + (size_t)kLorWarps * (size_t)tstride * sizeof(T));
    LorFast<BS> f;
    if constexpr (BS != 0)
        lor_fast_tables<BS>(a, tb,
                            lor_smem + (size_t)kLorWarps * (size_t)tstride * sizeof(T) + (size_t)lor_table_bytes(bs), f);
    const int64_t plane = a.ny * a.nz;
    // A warp takes its next ticket as it starts a block, so that the atomic's
    // round trip overlaps the block.  The smallest unfinished ticket is then
    // always some warp's current block (a warp's next ticket is larger than
    // its current one), whose neighbours hold smaller tickets: waits still end.
    unsigned nxt = 0;
    if (lane == 0) nxt = atomicAdd(counter, 1u);
    for (;;) {
        const unsigned tk = __shfl_sync(0xffffffffu, nxt, 0);
        if (tk >= nblocks) break;
        if (lane == 0) nxt = atomicAdd(counter, 1u);
        const int64_t b = order[tk];
        const int64_t bk = b % a.nz, bj = (b / a.nz) % a.ny, bi = b / plane;
        const LorBlock g = lor_geom(a, bi, bj, bk);
        // the block's own values or codes, its predictor selection and regression
        // coefficients need no neighbour: their loads overlap the wait
        int sel = ind[b];
        if (sel == 1 && a.rp == nullptr) sel = 0;  // a stream without coefficients
        const bool fast = BS != 0 && g.full && sel == 0 && a.pd == 3;
        const uint16_t *slot = nullptr;
        if constexpr (BS != 0) slot = fast ? f.slot : nullptr;
        lor_load_own<T, DECOMP, C>(a, g, tb, slot, xs, X, codes);
        float rp[4] = {0, 0, 0, 0};
        if (sel == 1)
            for (int c = 0; c < 4; c++) rp[c] = a.rp[4 * b + c];
        if (sel != 1) {
            // lanes 0..6 poll one neighbour each.  (Blocks of edge 1 read two
            // blocks back with two layers: those were done before the neighbour,
            // which waited for its own.)
            const int m = lane + 1;
            const int64_t di = m & 1, dj = (m >> 1) & 1, dk = (m >> 2) & 1;
            const unsigned *dep =
                lane < 7 && bi >= di && bj >= dj && bk >= dk ? done + (b - di * plane - dj * a.nz - dk) : nullptr;
            unsigned it = 0;
            while (!__all_sync(0xffffffffu, dep ? lor_ld_acquire(dep) != 0u : true)) {
                if (++it > kLorWaitLimit) {
                    if (lane == 0) atomicExch(err, 1);
                    break;
                }
                __nanosleep(20);
            }
            __syncwarp();
            if constexpr (BS != 0) {
                if (fast) {
                    const unsigned none = (bi > 0 ? 0u : 1u) | (bj > 0 ? 0u : 2u) | (bk > 0 ? 0u : 4u);
                    const T *r0 = R + g.g0;
                    T v[LorFast<BS>::kHalo];
#pragma unroll
                    for (int u = 0; u < LorFast<BS>::kHalo; u++)
                        v[u] = f.hat[u] >= 0 && !(f.hneed[u] & none) ? ld_coherent(r0 + f.hoff[u]) : (T)0;
#pragma unroll
                    for (int u = 0; u < LorFast<BS>::kHalo; u++)
                        if (f.hat[u] >= 0) t[f.hat[u]] = v[u];
                }
            }
            if (!fast) lor_load_halo<T>(a, g, tb, t, bi, bj, bk, sel == 2, R);
        }
        __syncwarp();
        if constexpr (BS != 0) {
            if (fast) lor_full<T, DECOMP, QM, BS>(a, g, f, t, xs, R, scratch, zpos, nzp, unpred);
        }
        if (!fast)
            lor_block<T, DECOMP, QM, C>(a, g, tb, t, xs, sel, rp, R, codes, scratch, zpos, nzp, unpred);
        // the barrier orders every lane's reconstruction writes before lane 0's
        // release store
        __syncwarp();
        if (lane == 0) lor_st_release(done + b, 1u);
        if constexpr (BS != 0 && !DECOMP) {
            if (fast)
                for (int e = lane; e < BS * BS * BS; e += 32)
                    codes[g.pos0 + e] = (C)*lor_code<T>(xs, f.slot[e]);
        }
        __syncwarp();
    }
}

// Blocks in diagonal order (any order inside a diagonal): base[d] the first place
// of diagonal d, cnt[d] (zeroed) its places taken.
__global__ void __launch_bounds__(256) k_lor_order(uint32_t nb, uint32_t ny, uint32_t nz,
                                                  const uint32_t *__restrict__ base, unsigned *cnt, uint32_t *order) {
    const uint32_t b = blockIdx.x * 256u + threadIdx.x;
    if (b >= nb) return;
    const uint32_t d = b % nz + (b / nz) % ny + b / nz / ny;
    order[base[d] + atomicAdd(cnt + d, 1u)] = b;
}

template <typename T>
LorArgs make_args(const uint64_t *dims, int bs, int pd, int lo, int lo2, double eb, int radius, int reg = 0) {
    LorArgs a;
    std::memset(&a, 0, sizeof(a));
    a.d1 = (int64_t)dims[0];
    a.d2 = (int64_t)dims[1];
    a.d3 = (int64_t)dims[2];
    a.bs = bs;
    a.nx = (a.d1 - 1) / bs + 1;
    a.ny = (a.d2 - 1) / bs + 1;
    a.nz = (a.d3 - 1) / bs + 1;
    a.pd = pd;
    a.lo = lo;
    a.lo2 = lo2;
    a.reg = reg;
    a.rp = nullptr;
    a.q.eb = eb;
    a.q.recip = 1.0 / eb;
    a.q.radius = radius;
    a.q.trim = 0;
    set_fast_path<T>(a.q);
    return a;
}

// Launches the wavefront on `st`; its error flag comes back to the returned
// pinned word, to be read (check_wavefront) once `st` is synchronised.
// C: uint16_t codes, or uint32_t for more than 65536 quantisation bins.
template <typename T, typename C>
const int *launch_wavefront(const LorArgs &a, bool decomp, const T *X, T *R, C *codes, T *scratch,
                            const uint16_t *ind, const uint64_t *zpos, uint64_t nz, const T *unpred, cudaStream_t st,
                            Counter &launches) {
    const bool straight = sizeof(T) == 4 && a.q.fast;
    // element offsets of the fast path are 32-bit
    const bool fast_bs = lor_has_fast(a.bs) && a.d1 * a.d2 * a.d3 < ((int64_t)1 << 31);
    // the warps' tiles and own values, then the CTA's tables
    const size_t smem = (size_t)kLorWarps *
                            (size_t)((a.bs + 2) * (a.bs + 2) * (a.bs + 2) + (fast_bs ? lor_own(a.bs) : a.bs * a.bs * a.bs)) * sizeof(T) +
                        (size_t)lor_table_bytes(a.bs) + (size_t)lor_fast_bytes(fast_bs ? a.bs : 0);
    void (*k)(LorArgs, const uint32_t *, uint32_t, unsigned *, unsigned *, int *, const T *, T *, C *, T *,
              const uint16_t *, const uint64_t *, uint64_t, const T *);
    // edges 6 (Config's 3-D default) and 5 (the tuner's trial) have lor_full's path
#define FAZ_LOR_PICK(BS)                                                                                \
    if (!decomp) k = straight ? k_lor_persist<T, false, 1, C, BS> : k_lor_persist<T, false, 0, C, BS>; \
    else k = straight ? k_lor_persist<T, true, 1, C, BS> : k_lor_persist<T, true, 0, C, BS>;
    if (fast_bs && a.bs == 6) {
        FAZ_LOR_PICK(6)
    } else if (fast_bs && a.bs == 5) {
        FAZ_LOR_PICK(5)
    } else {
        FAZ_LOR_PICK(0)
    }
#undef FAZ_LOR_PICK
    CK(allow_dynamic_smem((const void *)k));
    const uint64_t nb64 = (uint64_t)(a.nx * a.ny * a.nz);
    if (nb64 >= (1ull << 32)) throw Fail{FAZ_ERR_UNSUPPORTED, "too many Lorenzo blocks"};
    const uint32_t nb = (uint32_t)nb64;
    // blocks per diagonal bi + bj + bk = d: the pairs (bj, bk) of each sum, added
    // over a window of nx sums
    const int64_t nd = a.nx + a.ny + a.nz - 2, np = a.ny + a.nz - 1;
    auto pairs = [&](int64_t s) -> int64_t {
        return s < 0 || s >= np ? 0 : std::min(std::min(s + 1, np - s), std::min(a.ny, a.nz));
    };
    DevMem m(st);
    TableStage &ts = t_table_stage;
    uint32_t *hbase = (uint32_t *)ts.acquire((size_t)nd * 4);
    int64_t in_diag = 0, total = 0, widest = 0;
    for (int64_t d = 0; d < nd; d++) {
        in_diag += pairs(d) - pairs(d - a.nx);
        hbase[d] = (uint32_t)total;
        total += in_diag;
        widest = std::max(widest, in_diag);
    }
    if (total != (int64_t)nb) throw Fail{FAZ_ERR_DEVICE, "Lorenzo block order does not cover the blocks"};
    // zeroed: counter, done[nb], error flag, places taken per diagonal
    unsigned *sync = m.alloc<unsigned>((size_t)nb + 2 + (size_t)nd);
    int *derr = (int *)(sync + 1 + nb);
    unsigned *taken = sync + 2 + nb;
    uint32_t *dorder = m.alloc<uint32_t>((size_t)nb + (size_t)nd), *dbase = dorder + nb;
    CK(cudaMemcpyAsync(dbase, hbase, (size_t)nd * 4, cudaMemcpyHostToDevice, st));
    ts.release(st);
    CK(cudaMemsetAsync(sync, 0, ((size_t)nb + 2 + (size_t)nd) * 4, st));
    k_lor_order<<<(unsigned)((nb64 + 255) / 256), 256, 0, st>>>(nb, (uint32_t)a.ny, (uint32_t)a.nz, dbase, taken, dorder);
    launches(cudaGetLastError());
    int dev = 0, sms = 0, per_sm = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kLorWarps * 32, smem));
    if (per_sm < 1) throw Fail{FAZ_ERR_UNSUPPORTED, "Lorenzo block does not fit on an SM"};
    // never more CTAs than stay resident (waits rely on it), nor, when every block
    // waits for its neighbours, more warps than blocks on the widest diagonal: more
    // would only wait, and hold SMs that concurrent work (the tuner's other trials)
    // needs.  With regression blocks most tickets run at once.
    const uint64_t want = ((a.rp ? (uint64_t)nb : (uint64_t)widest) + kLorWarps - 1) / kLorWarps;
    const int grid = (int)std::min<uint64_t>((uint64_t)sms * (uint64_t)per_sm, want);
    k<<<grid, kLorWarps * 32, smem, st>>>(a, dorder, nb, sync, sync + 1, derr, X, R, codes, scratch, ind, zpos, nz,
                                          unpred);
    launches(cudaGetLastError());
    // the flag comes back through pinned memory: a copy to pageable memory
    // would hold the driver's pageable staging path while this kernel runs,
    // stalling concurrent pageable copies (the tuner's other trials)
    int *herr = (int *)t_pin_flag.get(64);
    CK(cudaMemcpyAsync(herr, derr, 4, cudaMemcpyDeviceToHost, st));
    return herr;
}

void check_wavefront(const int *herr) {
    if (*herr) throw Fail{FAZ_ERR_DEVICE, "Lorenzo wavefront: a block waited too long for its neighbours"};
}

template <typename T, typename C>
void run_wavefront(const LorArgs &a, bool decomp, const T *X, T *R, C *codes, T *scratch, const uint16_t *ind,
                   const uint64_t *zpos, uint64_t nz, const T *unpred, cudaStream_t st, Counter &launches) {
    const int *herr = launch_wavefront<T, C>(a, decomp, X, R, codes, scratch, ind, zpos, nz, unpred, st, launches);
    CK(cudaStreamSynchronize(st));
    check_wavefront(herr);
}

// meta_params as written by write(params, c) (include/QoZ/utils/MetaDef.hpp:33-60):
// 44 bytes, the reference's uninitialised padding written as zeros.
void put_meta_params(std::vector<uint8_t> &o, int bs, int pd, int lo, int lo2, int reg, double eb) {
    uint8_t m[44];
    std::memset(m, 0, sizeof m);
    const float prec = (float)eb;
    const float eb_lin = 1.0f * prec / 4 / (float)bs;
    const float eb_ind = (float)bs * eb_lin;
    int32_t v = bs;
    std::memcpy(m + 0, &v, 4);
    v = pd;
    std::memcpy(m + 4, &v, 4);
    m[8] = (uint8_t)(lo != 0);
    m[9] = (uint8_t)(lo2 != 0);
    m[10] = (uint8_t)(reg != 0);
    v = 2;  // lorenzo_padding_layer
    std::memcpy(m + 12, &v, 4);
    std::memcpy(m + 20, &eb_ind, 4);
    std::memcpy(m + 24, &eb_lin, 4);
    float f = 1.0f;  // reg_eb_base
    std::memcpy(m + 28, &f, 4);
    f = (float)bs;   // reg_eb_1
    std::memcpy(m + 32, &f, 4);
    f = 1.0f;        // sample_ratio
    std::memcpy(m + 36, &f, 4);
    m[40] = 1;       // lossless
    o.insert(o.end(), m, m + sizeof m);
}

// Regression coefficient precisions (MetaDef.hpp:54-59 and
// SZFastFrontend.hpp:229-235), in the element type T.
template <typename T>
void reg_precisions(int bs, double eb, T prec[4], T rprec[4]) {
    const float fprec = (float)eb;
    const float eb_lin = 1.0f * fprec / 4 / (float)bs;
    const float eb_ind = (float)bs * eb_lin;
    for (int i = 0; i < 3; i++) prec[i] = (T)eb_lin;
    prec[3] = (T)eb_ind;
    for (int i = 0; i < 4; i++) rprec[i] = (T)(1.0 / prec[i]);
}

// One coefficient x of the regression chain: quantised against the previous
// block's reconstructed one (prev), x and prev become its reconstruction; returns
// the code, 0 for an unpredictable coefficient.  rp2 = 1 / (2 prec): the halves
// ride in the factors (exact), the sign and the code are beside the chain, and the
// rare outcomes are branches, whose tests are not on it.
inline uint16_t reg_chain_step(float &prev, float &x, double prec, double rp2) {
    const float df = x - prev;
    const double diff = (double)df;
    const double h = std::fabs(diff) * rp2 + 0.5, p2 = std::copysign(2 * prec, diff);
    if (__builtin_expect(!(h < 32768), 0)) {
        prev = x;
        return 0;
    }
    const double k = std::trunc(h);
    const float dec = (float)((double)prev + k * p2);
    if (__builtin_expect(!(std::fabs((double)(float)(dec - x)) <= prec), 0)) {
        prev = x;
        return 0;
    }
    prev = dec;
    x = dec;
    return (uint16_t)((df < 0 ? -(int)k : (int)k) + 32768);
}

// compress_regression_coefficient_3d over the regression blocks in block
// order (MetaRegressionPredictor.hpp:10-40): each coefficient is predicted by
// the previous regression block's reconstructed one, a serial chain, four of
// them side by side, bound by the latency of a step's dependent arithmetic
// (75,000 blocks: 1.11 ms on a Grace core with integer conversions and selects on
// the chain, 0.93 ms without).  coef holds the blocks' coefficients and receives
// the reconstructed ones; types the codes, unp the unpredictable coefficients;
// returns the number of types.
template <typename T>
size_t reg_chain_compress(const uint16_t *ind, size_t nb, float *coef, int bs, double eb, uint16_t *types,
                          std::vector<float> &unp) {
    T prec[4], rprec[4];
    reg_precisions<T>(bs, eb, prec, rprec);
    const double p0 = (double)prec[0], p1 = (double)prec[1], p2 = (double)prec[2], p3 = (double)prec[3];
    const double r0 = (double)rprec[0] * 0.5, r1 = (double)rprec[1] * 0.5, r2 = (double)rprec[2] * 0.5,
                 r3 = (double)rprec[3] * 0.5;
    float c0 = 0, c1 = 0, c2 = 0, c3 = 0;
    size_t nt = 0;
    for (size_t b = 0; b < nb; b++) {
        if (ind[b] != 1) continue;
        float *x = coef + 4 * b;
        float x0 = x[0], x1 = x[1], x2 = x[2], x3 = x[3];
        const uint16_t k0 = reg_chain_step(c0, x0, p0, r0), k1 = reg_chain_step(c1, x1, p1, r1),
                       k2 = reg_chain_step(c2, x2, p2, r2), k3 = reg_chain_step(c3, x3, p3, r3);
        if (!k0) unp.push_back(x0);
        if (!k1) unp.push_back(x1);
        if (!k2) unp.push_back(x2);
        if (!k3) unp.push_back(x3);
        x[0] = x0;
        x[1] = x1;
        x[2] = x2;
        x[3] = x3;
        types[nt] = k0;
        types[nt + 1] = k1;
        types[nt + 2] = k2;
        types[nt + 3] = k3;
        nt += 4;
    }
    return nt;
}

// decode_regression_coefficients (MetaRegressionPredictor.hpp:42-80); rec
// receives the coefficients of the regression blocks
template <typename T>
void reg_chain_decompress(const uint16_t *ind, size_t nb, const uint16_t *types, size_t nt, const uint8_t *unp,
                          uint64_t nunp, float eb_lin, float eb_ind, float *rec) {
    T prec[4];
    for (int i = 0; i < 3; i++) prec[i] = (T)eb_lin;
    prec[3] = (T)eb_ind;
    float prev[4] = {0, 0, 0, 0};
    size_t ti = 0;
    uint64_t ui = 0;
    for (size_t b = 0; b < nb; b++) {
        if (ind[b] != 1) continue;
        if (nt - ti < 4) throw Fail{FAZ_ERR_FORMAT, "regression coefficient stream too short"};
        for (int c = 0; c < 4; c++) {
            const int tv = types[ti++];
            float v;
            if (tv == 0) {
                if (ui >= nunp) throw Fail{FAZ_ERR_FORMAT, "regression coefficient unpredictables exhausted"};
                std::memcpy(&v, unp + 4 * ui, 4);
                ui++;
            } else {
                v = (float)((double)prev[c] + (double)(2 * (tv - 32768)) * (double)prec[c]);
            }
            rec[4 * b + c] = v;
            prev[c] = v;
        }
    }
}

// pinned staging of the regression chain's selections, coefficients and types
inline thread_local Pinned t_pin_chain;

}  // namespace

void check_lorenzo3(const uint64_t *dims, int bs, int pd, int lo, int lo2, int reg, int radius) {
    if (!lo && !lo2 && !reg) throw Fail{FAZ_ERR_ARG, "all Lorenzo and regression predictors are disabled"};
    if (bs < 1 || bs > kLorMaxBs) throw Fail{FAZ_ERR_UNSUPPORTED, "Lorenzo block size must be 1..8 on the GPU path"};
    if (pd < 1 || pd > 3) throw Fail{FAZ_ERR_ARG, "pred_dim must be 1..3"};
    if (radius < 1 || radius > kLorMaxRadius)
        throw Fail{FAZ_ERR_UNSUPPORTED, "quantbinCnt above 131072 is not implemented on the GPU path"};
    for (int i = 0; i < 3; i++)
        if (dims[i] == 0) throw Fail{FAZ_ERR_ARG, "zero dimension"};
}

// SZ_compress_LorenzoReg for 3-D data (include/QoZ/api/impl/SZLorenzoReg.hpp:94-114):
// SZFastFrontend::compress_3d + save, then the general compressor's Huffman
// stage (SZGeneralCompressor.hpp:30-70).  Returns the pre-zstd payload in
// `out` (host).
template <typename T>
void lorenzo3_compress_payload(const uint64_t *dims, int bs, int pd, int lo, int lo2, int reg, double eb, int radius,
                               const T *dX, cudaStream_t st, Counter &launches, faz_timings &tm,
                               std::vector<uint8_t> &out) {
    check_lorenzo3(dims, bs, pd, lo, lo2, reg, radius);
    LorArgs a = make_args<T>(dims, bs, pd, lo, lo2, eb, radius, reg);
    const uint64_t n = dims[0] * dims[1] * dims[2];
    const uint64_t nb = (uint64_t)(a.nx * a.ny * a.nz);
    DevMem m(st);
    T *R = m.alloc<T>(n);
    T *scratch = m.alloc<T>(n);
    // 16-bit codes, or 32-bit ones for more than 65536 quantisation bins
    const bool wide = radius > 32768;
    uint16_t *codes16 = wide ? nullptr : m.alloc<uint16_t>(n);
    uint32_t *codes32 = wide ? m.alloc<uint32_t>(n) : nullptr;
    uint16_t *ind = m.alloc<uint16_t>(nb);
    unsigned long long *vcount = nullptr;
    if (verify_fast_path()) {
        vcount = m.alloc<unsigned long long>(1);
        CK(cudaMemsetAsync(vcount, 0, 8, st));
        a.q.verify = vcount;
    }
    Events ev_pred, ev_huff;
    CK(cudaEventRecord(ev_pred.a, st));
    float *raw = reg ? m.alloc<float>(4 * nb) : nullptr;
    k_lor_select<T><<<(unsigned)((nb + 255) / 256), 256, 0, st>>>(a, dX, ind, raw);
    launches(cudaGetLastError());
    // regression coefficients: the serial chain on the host, then the
    // reconstructed coefficients back to the device for the wavefront
    std::vector<float> runp;
    size_t ntypes = 0;
    uint64_t reg_count = 0;
    uint16_t *drtypes = nullptr;
    if (reg) {
        // coefficients, types and selections in pinned memory: no staging copies
        float *coef = (float *)t_pin_chain.get(nb * (16 + 8 + 2));
        uint16_t *types = (uint16_t *)(coef + 4 * nb), *hind = types + 4 * nb;
        CK(cudaMemcpyAsync(hind, ind, nb * 2, cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(coef, raw, nb * 16, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        auto th = clk::now();
        ntypes = reg_chain_compress<T>(hind, nb, coef, bs, eb, types, runp);
        reg_count = ntypes / 4;
        tm.host_ms += ms_since(th);
        CK(cudaMemcpyAsync(raw, coef, nb * 16, cudaMemcpyHostToDevice, st));
        a.rp = raw;
        if (reg_count) {
            drtypes = m.alloc<uint16_t>(ntypes);
            CK(cudaMemcpyAsync(drtypes, types, ntypes * 2, cudaMemcpyHostToDevice, st));
        }
    }
    // the predictor selections (and regression types) are final before the
    // wavefront: their Huffman stages run on a second stream meanwhile
    Events ev_sel, ev_side;
    CK(cudaEventRecord(ev_sel.a, st));
    StreamGuard side(nullptr, true);
    CK(cudaStreamWaitEvent(side.st, ev_sel.a, 0));
    DevMem m2(side.st);
    trace_step("lorenzo wavefront queued");
    const int *herr =
        wide ? launch_wavefront<T>(a, false, dX, R, codes32, scratch, ind, nullptr, 0, nullptr, st, launches)
             : launch_wavefront<T>(a, false, dX, R, codes16, scratch, ind, nullptr, 0, nullptr, st, launches);
    CK(cudaEventRecord(ev_pred.b, st));
    HuffEncoded hi, hc, hr;
    huffman_encode_device(ind, nb, 0, m2, side.st, launches, hi, tm);
    if (reg_count) huffman_encode_device(drtypes, ntypes, 32768, m2, side.st, launches, hr, tm);
    CK(cudaEventRecord(ev_side.a, side.st));
    CK(cudaStreamWaitEvent(st, ev_side.a, 0));
    CK(cudaStreamSynchronize(st));
    check_wavefront(herr);
    trace_step("lorenzo wavefront done");
    CK(cudaEventRecord(ev_huff.a, st));
    if (wide) huffman_encode_device(codes32, n, radius, m, st, launches, hc, tm);
    else huffman_encode_device(codes16, n, radius, m, st, launches, hc, tm);
    if (vcount) {
        unsigned long long vc = 0;
        CK(cudaMemcpy(&vc, vcount, 8, cudaMemcpyDeviceToHost));
        if (vc) throw Fail{FAZ_ERR_DEVICE, "float fast path disagreed with the double path at " + std::to_string(vc) + " points"};
    }
    const uint64_t nunpred = hc.nzero;
    T *unp = m.alloc<T>(nunpred ? nunpred : 1);
    if (nunpred && wide) launches(launch_compact_zeros<T>(codes32, n, hc.zc, hc.zoff, scratch, unp, st));
    if (nunpred && !wide) launches(launch_compact_zeros<T>(codes16, n, hc.zc, hc.zoff, scratch, unp, st));
    CK(cudaEventRecord(ev_huff.b, st));
    trace_step("lorenzo codebooks built");
    // SZFastFrontend::save: params, precision, meanInfo<T>{false, 0}, reg_count,
    // indicator tree + bits; LinearQuantizer::save; then the code tree + bits
    std::vector<uint8_t> h0;
    put_meta_params(h0, bs, pd, lo, lo2, reg, eb);
    put<double>(h0, eb);
    for (size_t i = 0; i < 2 * sizeof(T); i++) h0.push_back(0);
    put<uint64_t>(h0, reg_count);
    append_tree(h0, hi.cb, hi.nbytes);
    // encode_regression_coefficients (MetaRegressionPredictor.hpp:82-95)
    std::vector<uint8_t> hreg;
    if (reg_count) {
        put<uint64_t>(hreg, runp.size());
        const uint8_t *u = reinterpret_cast<const uint8_t *>(runp.data());
        hreg.insert(hreg.end(), u, u + runp.size() * 4);
        append_tree(hreg, hr.cb, hr.nbytes);
    }
    std::vector<uint8_t> h1;
    put<uint8_t>(h1, 2);
    put<double>(h1, eb);
    put<int32_t>(h1, radius);
    put<uint64_t>(h1, nunpred);
    std::vector<uint8_t> h2;
    append_tree(h2, hc.cb, hc.nbytes);
    const size_t rbits = reg_count ? hr.nbytes : 0;
    const size_t total =
        h0.size() + hi.nbytes + hreg.size() + rbits + h1.size() + nunpred * sizeof(T) + h2.size() + hc.nbytes;
    // device parts come back through the thread's pinned staging buffer
    // (copies to pageable memory serialise with other threads' copies)
    uint8_t *pin = payload_buffer(total);
    uint8_t *p = pin;
    std::memcpy(p, h0.data(), h0.size());
    p += h0.size();
    if (hi.nbytes) CK(cudaMemcpyAsync(p, hi.bits, hi.nbytes, cudaMemcpyDeviceToHost, st));
    p += hi.nbytes;
    if (!hreg.empty()) std::memcpy(p, hreg.data(), hreg.size());
    p += hreg.size();
    if (rbits) CK(cudaMemcpyAsync(p, hr.bits, rbits, cudaMemcpyDeviceToHost, st));
    p += rbits;
    std::memcpy(p, h1.data(), h1.size());
    p += h1.size();
    if (nunpred) CK(cudaMemcpyAsync(p, unp, nunpred * sizeof(T), cudaMemcpyDeviceToHost, st));
    p += nunpred * sizeof(T);
    std::memcpy(p, h2.data(), h2.size());
    p += h2.size();
    if (hc.nbytes) CK(cudaMemcpyAsync(p, hc.bits, hc.nbytes, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    emit_payload(out, pin, total);
    tm.unpred_count = nunpred;
    tm.payload_bytes = total;
    tm.predict_ms += ev_pred.ms();
    tm.huffman_ms += ev_huff.ms();
}

// SZ_decompress_LorenzoReg for 3-D data (SZLorenzoReg.hpp:117-135):
// SZFastFrontend::load + decompress_3d into dOut (device, dims[0]*dims[1]*dims[2] values).
template <typename T>
void lorenzo3_decompress(const uint8_t *pl, size_t psize, const uint64_t *dims, T *dOut, cudaStream_t st,
                         Counter &launches, faz_timings &tm) {
    WaitOnThrow wait(st);
    const uint8_t *p = pl, *end = pl + psize;
    auto need = [&](size_t k) {
        if ((size_t)(end - p) < k) throw Fail{FAZ_ERR_FORMAT, "truncated Lorenzo stream"};
    };
    need(44);
    int32_t bs, pd;
    std::memcpy(&bs, p, 4);
    std::memcpy(&pd, p + 4, 4);
    const int lo = p[8], lo2 = p[9], reg = p[10];
    float eb_ind, eb_lin;  // meta_params regression_param_eb_independent / _linear
    std::memcpy(&eb_ind, p + 20, 4);
    std::memcpy(&eb_lin, p + 24, 4);
    p += 44;
    need(8 + 2 * sizeof(T) + 8);
    p += 8;  // precision
    p += 2 * sizeof(T);  // meanInfo<T>
    uint64_t reg_count;
    std::memcpy(&reg_count, p, 8);
    p += 8;
    if (bs < 1 || bs > kLorMaxBs) throw Fail{FAZ_ERR_UNSUPPORTED, "Lorenzo block size must be 1..8 on the GPU path"};
    if (pd < 1 || pd > 3) throw Fail{FAZ_ERR_FORMAT, "bad pred_dim"};
    (void)lo;
    (void)lo2;
    (void)reg;
    const uint64_t n = dims[0] * dims[1] * dims[2];
    DevMem m(st);
    LorArgs a0 = make_args<T>(dims, bs, pd, 1, 1, 1.0, 1);
    const uint64_t nb = (uint64_t)(a0.nx * a0.ny * a0.nz);
    uint16_t *ind = m.alloc<uint16_t>(nb);
    Events ev_dec, ev_pred;
    CK(cudaEventRecord(ev_dec.a, st));
    huffman_decode_device(p, end, nb, ind, m, st, launches);
    if (reg_count > nb) throw Fail{FAZ_ERR_FORMAT, "bad regression block count"};
    float *drec = nullptr;
    // the coefficients' chain, on the host: runs while the GPU decodes the codes
    // (0.7 of the 1.3 ms before the wavefront of a 100x500x500 field when it came
    // first)
    std::function<void()> chain;
    if (reg_count) {
        // decode_regression_coefficients (MetaRegressionPredictor.hpp:42-80)
        need(8);
        uint64_t nrunp;
        std::memcpy(&nrunp, p, 8);
        p += 8;
        if ((size_t)(end - p) / 4 < nrunp) throw Fail{FAZ_ERR_FORMAT, "truncated regression coefficients"};
        const uint8_t *runp = p;
        p += nrunp * 4;
        uint16_t *dtypes = m.alloc<uint16_t>(4 * reg_count);
        huffman_decode_device(p, end, 4 * reg_count, dtypes, m, st, launches);
        float *rec = (float *)t_pin_chain.get(nb * (16 + 8 + 2));
        uint16_t *htypes = (uint16_t *)(rec + 4 * nb), *hind = htypes + 4 * nb;
        CK(cudaMemcpyAsync(hind, ind, nb * 2, cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(htypes, dtypes, 8 * reg_count, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        uint64_t nreg = 0;
        for (uint64_t b = 0; b < nb; b++) nreg += hind[b] == 1;
        if (nreg != reg_count) throw Fail{FAZ_ERR_FORMAT, "regression block count does not match the indicators"};
        drec = m.alloc<float>(4 * nb);
        chain = [=]() {
            reg_chain_decompress<T>(hind, nb, htypes, 4 * reg_count, runp, nrunp, eb_lin, eb_ind, rec);
            CK(cudaMemcpyAsync(drec, rec, nb * 16, cudaMemcpyHostToDevice, st));
        };
    }
    need(1 + 8 + 4 + 8);
    p += 1;
    double eb;
    std::memcpy(&eb, p, 8);
    p += 8;
    int32_t radius;
    std::memcpy(&radius, p, 4);
    p += 4;
    uint64_t nunpred;
    std::memcpy(&nunpred, p, 8);
    p += 8;
    if (!(eb > 0)) throw Fail{FAZ_ERR_FORMAT, "bad error bound"};
    if (radius < 1 || radius > kLorMaxRadius)
        throw Fail{FAZ_ERR_UNSUPPORTED, "quantbinCnt above 131072 is not implemented on the GPU path"};
    if ((size_t)(end - p) / sizeof(T) < nunpred) throw Fail{FAZ_ERR_FORMAT, "truncated unpredictable values"};
    T *dunp = m.alloc<T>(nunpred ? nunpred : 1);
    if (nunpred) CK(cudaMemcpyAsync(dunp, p, nunpred * sizeof(T), cudaMemcpyHostToDevice, st));
    p += nunpred * sizeof(T);
    const bool wide = radius > 32768;  // 32-bit codes for more than 65536 bins
    uint16_t *codes16 = wide ? nullptr : m.alloc<uint16_t>(n);
    uint32_t *codes32 = wide ? m.alloc<uint32_t>(n) : nullptr;
    uint64_t *zpos = nullptr;
    const uint64_t nz = nunpred;
    if (wide) decode_with_zeros(p, end, n, nz, codes32, m, st, launches, zpos, chain);
    else decode_with_zeros(p, end, n, nz, codes16, m, st, launches, zpos, chain);
    CK(cudaEventRecord(ev_dec.b, st));
    LorArgs a = make_args<T>(dims, bs, pd, 1, 1, eb, radius);
    a.rp = drec;
    unsigned long long *vcount = nullptr;
    if (verify_fast_path()) {
        vcount = m.alloc<unsigned long long>(1);
        CK(cudaMemsetAsync(vcount, 0, 8, st));
        a.q.verify = vcount;
    }
    CK(cudaEventRecord(ev_pred.a, st));
    if (wide) run_wavefront<T>(a, true, nullptr, dOut, codes32, nullptr, ind, zpos, nz, dunp, st, launches);
    else run_wavefront<T>(a, true, nullptr, dOut, codes16, nullptr, ind, zpos, nz, dunp, st, launches);
    CK(cudaEventRecord(ev_pred.b, st));
    CK(cudaStreamSynchronize(st));
    if (vcount) {
        unsigned long long vc = 0;
        CK(cudaMemcpy(&vc, vcount, 8, cudaMemcpyDeviceToHost));
        if (vc) throw Fail{FAZ_ERR_DEVICE, "float fast path disagreed with the double path at " + std::to_string(vc) + " points"};
    }
    tm.huffman_ms += ev_dec.ms();
    tm.predict_ms += ev_pred.ms();
}

template void lorenzo3_compress_payload<float>(const uint64_t *, int, int, int, int, int, double, int, const float *,
                                               cudaStream_t, Counter &, faz_timings &, std::vector<uint8_t> &);
template void lorenzo3_compress_payload<double>(const uint64_t *, int, int, int, int, int, double, int,
                                                const double *, cudaStream_t, Counter &, faz_timings &,
                                                std::vector<uint8_t> &);
template void lorenzo3_decompress<float>(const uint8_t *, size_t, const uint64_t *, float *, cudaStream_t, Counter &,
                                         faz_timings &);
template void lorenzo3_decompress<double>(const uint8_t *, size_t, const uint64_t *, double *, cudaStream_t,
                                          Counter &, faz_timings &);

}  // namespace faz
