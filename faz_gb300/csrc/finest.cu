// finest.cu - the finest interpolation level (lattice stride 1) of 3-D float
// fields, plane by plane.
//
// At stride 1 a block's lattice points split by the parity of their
// coordinates in sweep order (P0, P1, P2), SZInterpolationCompressor.hpp
// 3143-3360: all even = coarse (reconstructed by the previous level); odd
// along P0, even along P1 and P2 = sweep-1 targets, predicted along P0 from
// coarse points only; odd along P1, even along P2 = sweep-2 targets,
// predicted along P1 inside their P0-plane; odd along P2 = sweep-3 targets,
// predicted along P2 inside their row.  Once the block's coarse points are in
// shared memory every P0-plane is therefore independent of the others: one
// warp takes two planes, TMA tiled copies (cp.async.bulk.tensor) bring their
// original values into shared memory, and the warp runs the three sweeps there.
// The general level kernel (interp.cu) instead stages the block's whole even-P2
// lattice and walks lines with per-line bookkeeping.
//
// Lines of 32 or 33 points (all but those of a field's last, shorter blocks) go a
// line to a lane: the lane holds the line's values in registers, so a target costs
// no loads, the products 9x of the cubic stencil are shared between its
// neighbours, and the 16 targets of the line are independent of one another; its
// 16 codes are one run of 32 bytes in the stream, put together in registers and
// moved with 16-byte accesses.  Sweep 2 takes both planes' columns at once, a plane
// to a half-warp, sweep 3 a plane's rows.  Bound by instructions: with a target to a
// lane (five shared loads, stencil coefficients selected per lane and a 2-byte store
// each) it took 169 thread instructions a target, 0.60 ms for the 117 M targets of a
// 512^3 field; now 95 and 0.45 ms (decompression 0.48 ms, 0.77 ms in the block
// kernel).  58% of the issue slots are used: 16 warps an SM (registers, a line a
// lane, and shared memory, two planes a warp, both end there) wait for their own
// arithmetic first, then for instruction fetch; DRAM is at 21%.
//
// Stream positions are the ones of interp.cu (closed form from level, block,
// sweep, line and index; common.cuh): sweep-1 codes of a block interleave all
// planes, so they are staged in shared memory and moved once per block; sweep-2
// and sweep-3 codes of a plane are contiguous.
//
// Requirements (finest_possible): float data on the exact float quantiser
// path, P2 the contiguous axis, a 3-D field below 2^31 values, rows of 16-byte
// multiples in 16-byte aligned buffers (the tensor map's strides and x coordinates,
// decompression's 16-byte stores) and blocks of an edge up to 32 that is a multiple
// of 4.  It is used (finest_faster) for edge 32, where most lines have 32
// or 33 points.  Decompression moreover wants three quarters of the blocks to have
// both in-plane extents full: its single targets wait for their codes.  Measured
// against the block kernel of interp.cu, the line between them (finest level, ms,
// compression and decompression, plane kernel / block kernel):
//   512^3            0.45 / 0.83   0.48 / 0.77
//   300^3            0.13 / 0.19   0.16 / 0.17   (81 of 100 blocks full in the plane)
//   2464x60x60       0.08 / 0.09   0.11 / 0.08   (1 of 4)
//   500x510x509      0.78 / 0.78   0.78 / 0.73   (element copies and stores)
//   512^3, edge 16   1.80 / 1.74   (single targets throughout; edge 8: 7.6 / 4.5)
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <cstring>

#include "common.cuh"
#include "internal.h"
#include "quant.cuh"
#include "stencil.cuh"

namespace faz {

namespace {

constexpr int FW = 8;                  // warps per CTA
constexpr int FX = 36;                 // plane row pitch in floats (TMA box inner extent: 144 bytes)
constexpr int FROWS = 33;              // plane rows (block edge + 1)
constexpr int FC = 17;                 // coarse points per axis
constexpr uint32_t FPLANE_BYTES = FX * FROWS * 4;
constexpr int FXS_BYTES = (FPLANE_BYTES + 127) / 128 * 128;  // one plane; a warp has two
constexpr int FC_BYTES = (FC * FC * FC * 4 + 127) / 128 * 128;
constexpr int FSTAGE = FC * FC * 16 + 16;  // sweep-1 codes of a block + alignment shift
constexpr int FSTAGE_BYTES = (FSTAGE * 2 + 127) / 128 * 128;
constexpr int FSMEM = FC_BYTES + FSTAGE_BYTES + 2 * FW * FXS_BYTES + 128;
constexpr uint32_t FWAIT_LIMIT = 1u << 24;  // try_wait polls before a TMA wait gives up

__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// `planes` copies to come on the barrier
__device__ __forceinline__ void tma_expect(uint64_t *bar, int planes) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)),
                 "r"((uint32_t)planes * FPLANE_BYTES)
                 : "memory");
}
__device__ __forceinline__ void tma_plane(float *dst, const CUtensorMap *tm, int x, int y, int z, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(saddr(dst)),
        "l"(tm), "r"(x), "r"(y), "r"(z), "r"(saddr(bar))
        : "memory");
}

// Bounded wait for phase `phase` of the plane barrier; false when it gave up.
__device__ __forceinline__ bool tma_wait(uint64_t *bar, uint32_t phase) {
    uint32_t done = 0;
    for (uint32_t it = 0; it < FWAIT_LIMIT && !done; it++) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(saddr(bar)), "r"(phase)
            : "memory");
    }
    return __all_sync(0xffffffffu, done) != 0;
}

// One quantisation of the exact float path and its bookkeeping: the code goes
// to *dst, an unpredictable value to *udst.
__device__ __forceinline__ float finest_point(float v, float pred, const LevelArgs &a, bool emit, uint16_t *dst,
                                              float *udst) {
    float uv;
    const int code = quant_point<float, 1>(v, pred, a, uv);
    if (emit) {
        *dst = (uint16_t)code;
        if (code == 0) *udst = uv;
    }
    return v;
}

// ------------------------------------------------- a line to a lane
// Lines of n = 32 or 33 points: v[0..32] the line's values (v[32] unused for 32),
// 16 targets t at odd index 2t + 1.  Predictions in the reference's operation
// order, as make_stencil / eval_stencil give them.
template <int CUB>
__device__ __forceinline__ float line_pred(const float (&v)[33], int t, int n) {
    const int m = 2 * t + 1;
    if (!CUB) {
        if (t == 15 && n == 32) return linear1_any(v[28], v[30]);
        return (v[m - 1] + v[m + 1]) * 0.5f;
    }
    if (t == 0) return ((3.0f * v[0] + 6.0f * v[2]) - v[4]) * 0.125f;
    if (t == 14 && n == 32) return ((6.0f * v[28] - v[26]) + 3.0f * v[30]) * 0.125f;
    if (t == 15)
        return n == 32 ? ((3.0f * v[26] - 10.0f * v[28]) + 15.0f * v[30]) * 0.125f
                       : ((6.0f * v[30] - v[28]) + 3.0f * v[32]) * 0.125f;
    return (((9.0f * v[m - 1] - v[m - 3]) + 9.0f * v[m + 1]) - v[m + 3]) * 0.0625f;
}

// The 16 targets of a line: N the codes two to a word in target order (written, or
// in decompression read), v[odd] becomes the reconstruction.  Targets the float
// proofs leave undecided, and in decompression those of code 0, come back in the
// returned mask.
template <bool DECOMP, int CUB>
__device__ __forceinline__ unsigned line_targets(float (&v)[33], int n, const LevelArgs &a, uint32_t (&N)[8]) {
    unsigned bad = 0;
#pragma unroll
    for (int t = 0; t < 16; t++) {
        const float pred = line_pred<CUB>(v, t, n);
        bool und;
        float out;
        if (!DECOMP) {
            const int code = quantize_f32_straight(v[2 * t + 1], pred, a.rh, a.rl, a.eh, a.el, a.eblo, a.twor_f,
                                                   a.radius, out, und);
            N[t >> 1] = t & 1 ? N[t >> 1] | ((uint32_t)code << 16) : (uint32_t)code;
        } else {
            const int code = (int)((N[t >> 1] >> (16 * (t & 1))) & 0xffffu);
            und = dequant_f32_bracket(pred, int_to_float_small(code - a.radius), 2.0f * a.eh, 2.0f * a.el, out) ||
                  code == 0;
        }
        v[2 * t + 1] = out;
        bad |= und ? 1u << t : 0u;
    }
    return bad;
}

// The targets of `bad` again, by the double computation: `line` the line's values
// in shared memory (originals still), `st` its stride, `pos` the stream position of
// its first code.
template <bool DECOMP, int CUB>
__device__ __noinline__ void line_redo(const LevelArgs &a, unsigned bad, const float *line, int st, int n, uint64_t pos,
                                       const uint64_t *__restrict__ zpos, uint64_t nz, const float *__restrict__ unpred,
                                       const uint32_t *N, uint32_t *code_out, float *val_out) {
    // the results of one target at a time
    const int t = __ffs((int)bad) - 1, m = 2 * t + 1;
    const float pred = eval_stencil<CUB>(make_stencil<float>(m, n, a.cubic, st, 0), line);
    if (!DECOMP) {
        float v = line[m * st], uv;
        *code_out = (uint32_t)quantize_dp_f32(v, pred, a.eb, a.recip, a.radius, 0, uv);
        *val_out = v;
    } else {
        const int code = (int)((N[t >> 1] >> (16 * (t & 1))) & 0xffffu);
        *code_out = (uint32_t)code;
        *val_out = recover_dp_f32(pred, code, pos + line_rank(m, n, a.cubic), a.eb, a.radius, 0, zpos, nz, unpred);
    }
}

// Codes of a line from target order (N) to stream order (line_rank) and back.
template <int CUB>
__device__ __forceinline__ void to_stream(const uint32_t (&N)[8], int n, uint32_t (&R)[8]) {
    if (!CUB) {
#pragma unroll
        for (int i = 0; i < 8; i++) R[i] = N[i];
        return;
    }
#pragma unroll
    for (int i = 0; i < 6; i++) R[i] = __byte_perm(N[i], N[i + 1], 0x5432);
    R[6] = __byte_perm(N[6], n == 33 ? N[7] : N[0], 0x5432);
    R[7] = n == 33 ? __byte_perm(N[0], N[7], 0x7610) : N[7];
}
template <int CUB>
__device__ __forceinline__ void from_stream(const uint32_t (&R)[8], int n, uint32_t (&N)[8]) {
    if (!CUB) {
#pragma unroll
        for (int i = 0; i < 8; i++) N[i] = R[i];
        return;
    }
    N[0] = n == 33 ? __byte_perm(R[7], R[0], 0x5410) : __byte_perm(R[6], R[0], 0x5432);
#pragma unroll
    for (int i = 1; i < 7; i++) N[i] = __byte_perm(R[i - 1], R[i], 0x5432);
    N[7] = n == 33 ? __byte_perm(R[6], R[7], 0x7632) : R[7];
}

// Lanes of a run of lines write 16 codes (R) each at `dst`, one line after the
// other; A = dst's place in its 16 bytes, in codes, the same for every lane of the
// run.  Each lane writes the two aligned 16-byte pieces that begin in the last A
// codes of the lane before it (`prev`, that lane's R[4..7]); the run's first and
// last pieces, shared with other runs, code by code.
template <int A>
__device__ __forceinline__ void run_store(uint16_t *dst, const uint32_t (&R)[8], const uint32_t (&prev)[4], bool first,
                                          bool last) {
    constexpr int o = (8 - A) >> 1;
    auto word = [&](int j) { return j < 4 ? prev[j] : R[j - 4]; };
    uint32_t q[8];
#pragma unroll
    for (int i = 0; i < 8; i++) q[i] = (A & 1) ? __byte_perm(word(o + i), word(o + i + 1), 0x5432) : word(o + i);
    uint4 *d = reinterpret_cast<uint4 *>(dst - A);
    d[1] = make_uint4(q[4], q[5], q[6], q[7]);
    if constexpr (A == 0) {
        d[0] = make_uint4(q[0], q[1], q[2], q[3]);
    } else {
        if (!first) {
            d[0] = make_uint4(q[0], q[1], q[2], q[3]);
        } else {
#pragma unroll
            for (int j = A; j < 8; j++) dst[j - A] = (uint16_t)(q[j >> 1] >> (16 * (j & 1)));
        }
        if (last) {
#pragma unroll
            for (int j = 16 - A; j < 16; j++) dst[j] = (uint16_t)(R[j >> 1] >> (16 * (j & 1)));
        }
    }
}
// ... and read them: the three aligned pieces that hold them (the codes are
// allocated with 16 bytes to spare)
template <int A>
__device__ __forceinline__ void run_load(const uint16_t *src, uint32_t (&R)[8]) {
    const uint4 *d = reinterpret_cast<const uint4 *>(src - A);
    const uint4 x = d[0], y = d[1], z = A ? d[2] : make_uint4(0, 0, 0, 0);
    const uint32_t c[12] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w, z.x, z.y, z.z, z.w};
#pragma unroll
    for (int i = 0; i < 8; i++)
        R[i] = (A & 1) ? __byte_perm(c[A / 2 + i], c[A / 2 + i + 1], 0x5432) : c[A / 2 + i];
}
#define FAZ_RUN_CASES(F)                                                    \
    switch (((uintptr_t)at >> 1) & 7) {                                     \
    case 0: F(0); break;                                                    \
    case 1: F(1); break;                                                    \
    case 2: F(2); break;                                                    \
    case 3: F(3); break;                                                    \
    case 4: F(4); break;                                                    \
    case 5: F(5); break;                                                    \
    case 6: F(6); break;                                                    \
    default: F(7); break;                                                   \
    }

// One line per lane (`act`), `line` in shared memory with stride st, its codes at
// cb[off..off + 16) (stream position base + off).  `width` lanes make a run.
// Values: already in v; the odd ones become the reconstruction.  VERIFY: every target
// that the float proofs decided is computed again by the double computation, and the
// differences counted.
template <bool DECOMP, int CUB, bool VERIFY>
__device__ __forceinline__ void line_run(const LevelArgs &a, float (&v)[33], const float *line, int st, int n, bool act,
                                         int width, int in_run, int lanes, uint16_t *cb, float *ub, uint64_t base,
                                         int off, const uint64_t *__restrict__ zpos, uint64_t nz,
                                         const float *__restrict__ unpred) {
    uint32_t N[8], R[8];
    if (DECOMP) {
        const uint16_t *at = cb + off;
#pragma unroll
        for (int i = 0; i < 8; i++) R[i] = 0x80008000u;
        if (act) {
#define FAZ_RUN_LOAD(A) run_load<A>(at, R)
            FAZ_RUN_CASES(FAZ_RUN_LOAD)
#undef FAZ_RUN_LOAD
        }
        from_stream<CUB>(R, n, N);
    }
    unsigned bad = line_targets<DECOMP, CUB>(v, n, a, N);
    if constexpr (VERIFY) {
#pragma unroll 1
        for (unsigned todo = act ? ~bad & 0xffffu : 0u; todo; todo &= todo - 1) {
            const unsigned bit = todo & (0u - todo);
            uint32_t Nm[8], c;
            float val;
#pragma unroll
            for (int i = 0; i < 8; i++) Nm[i] = N[i];
            line_redo<DECOMP, CUB>(a, bit, line, st, n, base + (uint64_t)off, zpos, nz, unpred, Nm, &c, &val);
#pragma unroll
            for (int k = 0; k < 16; k++)
                if (bit == 1u << k && (c != ((N[k >> 1] >> (16 * (k & 1))) & 0xffffu) ||
                                       __float_as_uint(val) != __float_as_uint(v[2 * k + 1])))
                    atomicAdd(a.verify, 1ull);
        }
    }
    if (!act) bad = 0;
    while (bad) {
        uint32_t Nm[8], c;
        float val;
#pragma unroll
        for (int i = 0; i < 8; i++) Nm[i] = DECOMP ? N[i] : 0u;
        line_redo<DECOMP, CUB>(a, bad, line, st, n, base + (uint64_t)off, zpos, nz, unpred, Nm, &c, &val);
        const int t = __ffs((int)bad) - 1;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            if (k != t) continue;
            v[2 * k + 1] = val;
            if (!DECOMP) N[k >> 1] = k & 1 ? (N[k >> 1] & 0xffffu) | (c << 16) : (N[k >> 1] & 0xffff0000u) | c;
        }
        bad &= bad - 1;
    }
    if (!DECOMP) {
        // unpredictable targets (code 0): their values at their stream positions
        uint32_t zero = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) zero |= (N[i] - 0x00010001u) & ~N[i] & 0x80008000u;
        if (zero && act) {
#pragma unroll
            for (int k = 0; k < 16; k++)
                if (((N[k >> 1] >> (16 * (k & 1))) & 0xffffu) == 0) ub[off + line_rank(2 * k + 1, n, CUB)] = v[2 * k + 1];
        }
        to_stream<CUB>(N, n, R);
        uint32_t prev[4];
#pragma unroll
        for (int i = 0; i < 4; i++) prev[i] = __shfl_up_sync(0xffffffffu, R[4 + i], 1, width);
        if (act) {
            uint16_t *at = cb + off;
            const bool first = in_run == 0, last = in_run == lanes - 1;
#define FAZ_RUN_STORE(A) run_store<A>(at, R, prev, first, last)
            FAZ_RUN_CASES(FAZ_RUN_STORE)
#undef FAZ_RUN_STORE
        }
    }
}

// One target, any line: `line` with stride st in shared memory, code and value
// moved if `emit`.
template <bool DECOMP, int CUB>
__device__ __forceinline__ void one_target(const LevelArgs &a, float *line, int st, int m, int n, bool act, bool emit,
                                           uint16_t *cb, float *ub, uint64_t base, int off, uint64_t owner,
                                           const uint16_t *__restrict__ codes, const uint64_t *__restrict__ zpos,
                                           uint64_t nz, const float *__restrict__ unpred) {
    const float pred = eval_stencil<CUB>(make_stencil<float>(m, n, a.cubic, st, 0), (const float *)line);
    float v;
    if (!DECOMP) {
        v = finest_point(line[m * st], pred, a, act && emit, cb + off, ub + off);
    } else {
        const uint64_t pos = emit ? base + (uint64_t)off : owner;
        v = recover_point<float, 1>(pred, act ? (int)codes[pos] : a.radius, pos, a, zpos, nz, unpred);
    }
    if (act) line[m * st] = v;
}

// Compression (DECOMP = 0): originals in, codes and unpredictable values out.
// Decompression (DECOMP = 1): codes in, every reconstructed target of the block
// into W.  Either way the plane buffers end up holding the planes' reconstruction
// at even P2 indices (each value written where its original was read, once the
// original is no longer needed) and, in decompression, at odd ones too, to be
// written to W.  W holds the coarse points (earlier levels) in both directions.
template <bool DECOMP, int CUB, bool VERIFY>
__global__ void __launch_bounds__(FW * 32, 2)
    k_finest(LevelArgs a, const __grid_constant__ CUtensorMap tm, float *W, uint16_t *__restrict__ codes,
             float *__restrict__ scratch, const uint64_t *__restrict__ zpos, uint64_t nz,
             const float *__restrict__ unpred) {
    extern __shared__ __align__(128) unsigned char smem[];
    float *C = reinterpret_cast<float *>(smem);
    uint16_t *stage = reinterpret_cast<uint16_t *>(smem + FC_BYTES);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float *XA = reinterpret_cast<float *>(smem + FC_BYTES + FSTAGE_BYTES + 2 * warp * FXS_BYTES);
    float *XB = XA + FXS_BYTES / 4;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + FC_BYTES + FSTAGE_BYTES + 2 * FW * FXS_BYTES) + warp;

    int64_t bc[3];
    block_coords(a, blockIdx.x, bc);
    BlockGeom g;
    block_geom(a, bc, g);
    const int P0 = a.perm[0], P1 = a.perm[1];
    const int n0 = g.n0, n1 = g.n1, n2 = g.n2;
    const int k0 = g.k0, k1 = g.k1, k2 = g.k2;
    const int hh1 = (n1 + 1) / 2, h2 = g.h2;
    const int G0 = (int)pick3(P0, a.offs[0], a.offs[1], a.offs[2]);
    const int G1 = (int)pick3(P1, a.offs[0], a.offs[1], a.offs[2]);
    const int64_t origin = g.beg[0] * a.offs[0] + g.beg[1] * a.offs[1] + g.beg[2] * a.offs[2];
    float *wb = W + origin;
    const uint64_t base = a.block_off[blockIdx.x];
    uint16_t *cb = codes + base;                  // the block's codes
    float *ub = DECOMP ? nullptr : scratch + base;  // their unpredictable values
    const int cubic = a.cubic;
    const int sh1 = (int)(base & 7);

    if (!DECOMP && lane == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // coarse points of the block: C[c0][c1][c2] = W at (2c0, 2c1, 2c2)
    {
        const int rows = ((n0 + 1) / 2) * hh1;
        for (int r = warp; r < rows; r += FW) {
            const int c0 = r / hh1, c1 = r - c0 * hh1;
            const float *src = wb + 2 * c0 * G0 + 2 * c1 * G1;
            if (lane < h2) cp_async<4>(C + (c0 * FC + c1) * FC + lane, src + 2 * lane);
        }
        cp_async_wait_all();
    }
    int hold = 0;  // read here, with the loads above on their way
    if (DECOMP) {
        if (a.hold) hold = *a.hold;
        // the block's sweep-1 codes (they interleave all planes)
        const int cnt = (int)g.c1;
        const int a0 = (8 - sh1) & 7;
        const int nbody = cnt > a0 ? (cnt - a0) >> 3 : 0;
        const int tail0 = a0 + (nbody << 3);
        for (int i = tid; i < cnt; i += blockDim.x)
            if (i < a0 || i >= tail0) stage[sh1 + i] = cb[i];
        for (int j = tid; j < nbody; j += blockDim.x) {
            const int i = a0 + (j << 3);
            *reinterpret_cast<uint4 *>(stage + sh1 + i) = *reinterpret_cast<const uint4 *>(cb + i);
        }
    }
    __syncthreads();
    if (DECOMP && hold) return;

    const int t = lane & 15, half = lane >> 4;
    const int np = n0 - k0;   // planes with emitted codes
    const int w1 = n1 - k1;   // emitted rows (sweep 3)
    const int w2 = n2 - k2;   // emitted columns
    // lines of 32 or 33 points in both sweeps: a line to a lane
    const bool lines = n1 >= 32 && n2 >= 32;
    uint32_t phase = 0;
    // planes in pairs (an odd and an even P0 index) per warp, so that warps
    // get the same work
    for (int pp = warp; 2 * pp < np; pp += FW) {
        const int mA = k0 + 2 * pp;
        const int npl = mA + 1 < n0 ? 2 : 1;
        // the previous planes' reads and in-place writes come before the copies of
        // the next ones
        if (!DECOMP) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (!DECOMP) {
            if (lane == 0) {
                tma_expect(bar, npl);
                for (int s = 0; s < npl; s++) {
                    const int m0 = mA + s;
                    tma_plane(s ? XB : XA, &tm, (int)g.beg[2], (int)g.beg[1] + (P0 == 1 ? m0 : 0),
                              (int)g.beg[0] + (P0 == 0 ? m0 : 0), bar);
                }
            }
            if (!tma_wait(bar, phase)) {
                // the call fails; wait (bounded again) for the copies in flight
                // before the warp leaves, so that they do not land in shared
                // memory that another CTA may own by then
                if (lane == 0 && a.err) atomicExch(a.err, 1);
                (void)tma_wait(bar, phase);
                break;
            }
            phase ^= 1;
        }
        // sweep 1, or the coarse points of an even plane
#pragma unroll 1
        for (int s = 0; s < npl; s++) {
            const int m0 = mA + s;
            float *Xs = s ? XB : XA;
            if (!(m0 & 1)) {
                // even plane: its even-P1 / even-P2 points are coarse
                const float *cp = C + (m0 >> 1) * FC * FC;
                LineCursor lc;
                lc.init(lane, 32, h2);  // outer = e1, inner = e2
                for (int i = lane; i < hh1 * h2; i += 32, lc.next())
                    Xs[2 * lc.outer * FX + 2 * lc.inner] = cp[lc.outer * FC + lc.inner];
                continue;
            }
            // targets (m0, 2e1, 2e2) from the coarse planes; first the lines this
            // block emits (stream rank = flat index x t0 + rank in the line), then
            // those on its first planes, which the previous blocks emit (recomputed
            // in compression, decoded from their owners' streams in decompression)
            const Stencil<float> S1 = make_stencil<float>(m0, n0, cubic, FC * FC, 1);
            const int rk0 = line_rank(m0, n0, cubic);
            const int ne = g.ne1 * g.ne2;
            LineCursor lc;
            if (ne > 0) lc.init(lane, 32, g.ne2);
            for (int i0 = 0; i0 < ne; i0 += 32, lc.next()) {
                const int i = i0 + lane;
                const bool in = i < ne;
                const int e1 = k1 + (in ? lc.outer : 0), e2 = k2 + (in ? lc.inner : 0);
                const float pred = eval_stencil<CUB>(S1, C + e1 * FC + e2);
                const int rank = (in ? i : 0) * g.t0 + rk0;
                float *xp = Xs + 2 * e1 * FX + 2 * e2;
                float v;
                if (!DECOMP) v = finest_point(*xp, pred, a, in, stage + sh1 + rank, ub + rank);
                else v = recover_point<float, 1>(pred, (int)stage[sh1 + rank], base + rank, a, zpos, nz, unpred);
                if (in) *xp = v;
            }
            const int nfirst = k1 * h2 + k2 * (hh1 - k1);
            for (int j0 = 0; j0 < nfirst; j0 += 32) {
                const int j = j0 + lane;
                const bool in = j < nfirst;
                int e1 = 0, e2 = 0;
                if (in) {
                    if (j < k1 * h2) e2 = j;
                    else e1 = k1 + (j - k1 * h2);
                }
                const float pred = eval_stencil<CUB>(S1, C + e1 * FC + e2);
                float *xp = Xs + 2 * e1 * FX + 2 * e2;
                float v;
                if (!DECOMP) {
                    v = finest_point(*xp, pred, a, false, nullptr, nullptr);
                } else {
                    uint64_t pos = owner_pos_sweep1(a, g, bc, P1, a.perm[2], e1, e2, n2) + rk0;
                    if (pos >= a.ncodes) {
                        atomicExch(a.err, 1);
                        pos = 0;
                    }
                    v = recover_point<float, 1>(pred, (int)codes[pos], pos, a, zpos, nz, unpred);
                }
                if (in) *xp = v;
            }
        }
        __syncwarp();
        // sweep 2: targets (m0, 2t+1, 2e2), lines along P1, codes of column e2 at
        // c1 + ((m0 - k0) ne2 + e2 - k2) t1
        uint64_t own = 0;  // first-plane column: its owner's position (the previous block along P2)
        if (lines) {
            const int m0 = mA + half;
            float *Xs = half ? XB : XA;
            const bool pl = half < npl;
            const int pb = (int)g.c1 + (m0 - k0) * g.ne2 * 16;
            {
                // column 0, a target to a lane
                const int rk1 = line_rank(2 * t + 1, n1, cubic);
                if (DECOMP && k2) {
                    own = owner_pos_sweep2(a, g, bc, a.perm[2], (pl ? m0 : mA) - k0) + rk1;
                    if (own >= a.ncodes) {
                        atomicExch(a.err, 1);
                        own = 0;
                    }
                }
                one_target<DECOMP, CUB>(a, Xs, FX, 2 * t + 1, n1, pl, k2 == 0, cb, ub, base, pl ? pb + rk1 : 0, own,
                                        codes, zpos, nz, unpred);
            }
            // columns 1.., a column to a lane
            const bool act = pl && t + 1 < h2;
            const int e2 = act ? t + 1 : 1;
            float *col = Xs + 2 * e2;
            float v[33];
#pragma unroll
            for (int r = 0; r < 32; r++) v[r] = DECOMP && (r & 1) ? 0.0f : col[r * FX];
            v[32] = n1 == 33 ? col[32 * FX] : 0.0f;
            line_run<DECOMP, CUB, VERIFY>(a, v, col, FX, n1, act, 16, t, h2 - 1, cb, ub, base, act ? pb + (e2 - k2) * 16 : 0,
                                  zpos, nz, unpred);
            if (act) {
#pragma unroll
                for (int k = 0; k < 16; k++) col[(2 * k + 1) * FX] = v[2 * k + 1];
            }
        } else if (g.t1 > 0) {
            const bool act = t < g.t1;
            const int m1 = act ? 2 * t + 1 : 1;
            const int rk1 = line_rank(m1, n1, cubic);
#pragma unroll 1
            for (int s = 0; s < npl; s++) {
                const int m0 = mA + s;
                float *Xs = s ? XB : XA;
                const int pb = (int)g.c1 + (m0 - k0) * g.ne2 * g.t1 + rk1;
                if (DECOMP && k2) {
                    own = owner_pos_sweep2(a, g, bc, a.perm[2], m0 - k0) + rk1;
                    if (own >= a.ncodes) {
                        atomicExch(a.err, 1);
                        own = 0;
                    }
                }
                for (int e2b = 0; e2b < h2; e2b += 2) {
                    const int e2 = e2b + half;
                    const bool in = act && e2 < h2;
                    const int ec = e2 < h2 ? e2 : h2 - 1;
                    one_target<DECOMP, CUB>(a, Xs + 2 * ec, FX, m1, n1, in, ec >= k2, cb, ub, base,
                                            ec >= k2 ? pb + (ec - k2) * g.t1 : 0, own, codes, zpos, nz, unpred);
                }
            }
        }
        __syncwarp();
        // sweep 3: targets (m0, m1, 2t+1) of the emitted rows, lines along P2, codes
        // of row m1 at c1 + c2 + ((m0 - k0) w1 + m1 - k1) t2
        if (lines) {
            const int pb0 = (int)(g.c1 + g.c2) + 2 * pp * w1 * 16;
            if (k1 == 0) {
                // row 0, a target to a lane
                one_target<DECOMP, CUB>(a, half ? XB : XA, 1, 2 * t + 1, n2, half < npl, true, cb, ub, base,
                                        half < npl ? pb0 + half * w1 * 16 + line_rank(2 * t + 1, n2, cubic) : 0, 0, codes,
                                        zpos, nz, unpred);
            }
            // rows 1.., a row to a lane
            const bool act = lane + 1 < n1;
            const int m1 = act ? lane + 1 : 1;
#pragma unroll 1
            for (int s = 0; s < npl; s++) {
                float *row = (s ? XB : XA) + m1 * FX;
                float v[33];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const float4 q = *reinterpret_cast<const float4 *>(row + 4 * c);
                    v[4 * c] = q.x;
                    v[4 * c + 1] = q.y;
                    v[4 * c + 2] = q.z;
                    v[4 * c + 3] = q.w;
                }
                v[32] = n2 == 33 ? row[32] : 0.0f;
                line_run<DECOMP, CUB, VERIFY>(a, v, row, 1, n2, act, 32, lane, n1 - 1, cb, ub, base,
                                      act ? pb0 + (s * w1 + m1 - k1) * 16 : 0, zpos, nz, unpred);
                if (DECOMP && act) {
#pragma unroll
                    for (int c = 0; c < 8; c++)
                        *reinterpret_cast<float4 *>(row + 4 * c) =
                            make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
                }
            }
        } else if (g.t2 > 0) {
            const bool act = t < g.t2;
            const int m2 = act ? 2 * t + 1 : 1;
            const int rk2 = line_rank(m2, n2, cubic);
            const int hr = (w1 + 1) >> 1;  // rows per half-warp
#pragma unroll 1
            for (int s = 0; s < npl; s++) {
                float *Xs = s ? XB : XA;
                const int pb = (int)(g.c1 + g.c2) + (mA + s - k0) * w1 * g.t2 + rk2;
                for (int it = 0; it < hr; it++) {
                    const int rho = it + half * hr;
                    const bool in = act && rho < w1;
                    const int rc = rho < w1 ? rho : w1 - 1;
                    one_target<DECOMP, CUB>(a, Xs + (k1 + rc) * FX, 1, m2, n2, in, true, cb, ub, base, pb + rc * g.t2, 0,
                                            codes, zpos, nz, unpred);
                }
            }
        }
        if (DECOMP && w2 > 0) {
            // the planes' emitted rows and columns to W
            __syncwarp();
#pragma unroll 1
            for (int s = 0; s < npl; s++) {
                const int m0 = mA + s;
                const float *Xs = s ? XB : XA;
                float *dst = wb + m0 * G0;
                if (lines) {
                    // 32 columns of four rows at a time (column 0 and the coarse
                    // points are written again with the values they have), then
                    // column 32
                    for (int m1 = k1 + (lane >> 3); m1 < n1; m1 += 4)
                        *reinterpret_cast<float4 *>(dst + m1 * G1 + 4 * (lane & 7)) =
                            *reinterpret_cast<const float4 *>(Xs + m1 * FX + 4 * (lane & 7));
                    if (n2 == 33)
                        for (int m1 = k1 + lane; m1 < n1; m1 += 32) dst[m1 * G1 + 32] = Xs[m1 * FX + 32];
                    continue;
                }
                for (int m1 = k1; m1 < n1; m1++) {
                    float *drow = dst + m1 * G1;
                    const float *srow = Xs + m1 * FX;
                    const bool odd_row = (m0 | m1) & 1;  // no coarse point in the row
                    for (int m2 = k2 + lane; m2 < n2; m2 += 32)
                        if (odd_row || (m2 & 1)) drow[m2] = srow[m2];
                }
            }
        }
    }
    if (DECOMP) return;
    __syncthreads();
    // sweep-1 codes of the block, 16 bytes per store where aligned
    const int cnt = (int)g.c1;
    const int a0 = (8 - sh1) & 7;
    const int nbody = cnt > a0 ? (cnt - a0) >> 3 : 0;
    const int tail0 = a0 + (nbody << 3);
    for (int i = tid; i < cnt; i += blockDim.x)
        if (i < a0 || i >= tail0) cb[i] = stage[sh1 + i];
    for (int j = tid; j < nbody; j += blockDim.x) {
        const int i = a0 + (j << 3);
        *reinterpret_cast<uint4 *>(cb + i) = *reinterpret_cast<const uint4 *>(stage + sh1 + i);
    }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return (EncodeTiledFn) nullptr;
        return (EncodeTiledFn)p;
    }();
    return fn;
}

}  // namespace

bool finest_possible(const LevelArgs &a, bool decomp, const void *X, const void *W) {
    // block begins along the contiguous axis are TMA x coordinates: the edge is a
    // multiple of 4 values
    if (a.s != 1 || a.bs > 32 || (a.bs & 3) || a.write_back || !a.fast || a.trim != 0) return false;
    if (a.perm[2] != 2 || a.perm[0] > 1 || a.perm[1] > 1) return false;
    if (a.dims[0] < FROWS || a.dims[1] < FROWS || a.dims[2] < FX || (a.dims[2] & 3)) return false;
    if (a.dims[0] * a.dims[1] * a.dims[2] >= ((int64_t)1 << 31)) return false;
    if (decomp) return ((uintptr_t)W & 15) == 0;
    return ((uintptr_t)X & 15) == 0 && encode_tiled() != nullptr;
}

bool finest_faster(const LevelArgs &a, bool decomp) {
    if (a.bs != 32) return false;
    const int64_t d1 = a.dims[a.perm[1]], d2 = a.dims[2];
    return !decomp || 4 * (d1 / 32) * (d2 / 32) >= 3 * ((d1 + 31) / 32) * ((d2 + 31) / 32);
}

cudaError_t launch_finest(const LevelArgs &a, int64_t nblocks, bool decomp, const float *X, float *W,
                          uint16_t *codes, float *scratch, const uint64_t *zpos, uint64_t nz, const float *unpred,
                          cudaStream_t st) {
    CUtensorMap tm;
    std::memset(&tm, 0, sizeof(tm));
    if (!decomp) {
        const cuuint64_t gdim[3] = {(cuuint64_t)a.dims[2], (cuuint64_t)a.dims[1], (cuuint64_t)a.dims[0]};
        const cuuint64_t gstride[2] = {(cuuint64_t)a.dims[2] * 4, (cuuint64_t)(a.dims[1] * a.dims[2]) * 4};
        // the plane of P0 index m0: rows along P1, FX values along axis 2
        const cuuint32_t box[3] = {(cuuint32_t)FX, a.perm[0] == 0 ? (cuuint32_t)FROWS : 1u,
                                   a.perm[0] == 0 ? 1u : (cuuint32_t)FROWS};
        const cuuint32_t estride[3] = {1, 1, 1};
        CUresult r = encode_tiled()(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(X), gdim, gstride,
                                    box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    }
    void (*k)(LevelArgs, const CUtensorMap, float *, uint16_t *, float *, const uint64_t *, uint64_t, const float *);
    if (a.verify) {
        if (decomp) k = a.cubic ? k_finest<true, 1, true> : k_finest<true, 0, true>;
        else k = a.cubic ? k_finest<false, 1, true> : k_finest<false, 0, true>;
    } else {
        if (decomp) k = a.cubic ? k_finest<true, 1, false> : k_finest<true, 0, false>;
        else k = a.cubic ? k_finest<false, 1, false> : k_finest<false, 0, false>;
    }
    cudaError_t e = allow_dynamic_smem((const void *)k);
    if (e != cudaSuccess) return e;
    k<<<(unsigned)nblocks, FW * 32, FSMEM, st>>>(a, tm, W, codes, scratch, zpos, nz, unpred);
    return cudaGetLastError();
}

}  // namespace faz
