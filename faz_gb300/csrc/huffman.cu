// huffman.cu - Huffman histogram, encode and decode kernels.
//
// Stream format (include/QoZ/encoder/HuffmanEncoder.hpp:150-268): the codes
// of all symbols concatenated, most significant bit first, zero padded to a
// byte.  Encoding is a two-pass bit-offset scan; decoding of unmodified
// streams splits the bit string into fixed-size units, decodes each unit
// speculatively from its nominal start and repeats for units whose true start
// (the end of the previous unit's decode) differs, until every unit starts on
// a codeword boundary (Huffman codes self-synchronise within a few codewords).
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include "internal.h"

namespace faz {

// --------------------------------------------------------------- histogram
// Counts of every symbol, the stream position of its first occurrence, and the
// number of zero codes per sub-chunk of HSUB codes (for the compaction of the
// unpredictable values).  A CTA takes a run of consecutive sub-chunks, a warp one
// at a time, so that zero codes can later be compacted per warp with one running
// offset and no block barriers.
static constexpr uint64_t HSUB = 2048;
static constexpr int HWARPS = 32;
static constexpr uint64_t HCHUNK = HSUB * HWARPS;
static constexpr int HWIN = 4096;     // symbols around `center` counted in shared memory
static constexpr int HTHREADS = 512;  // four such CTAs an SM

// Symbols within the window are counted in shared memory (bin HWIN takes the
// others), with their first position in the CTA's run; a code touches that word
// only while its position beats the recorded one.  Symbols outside go to global
// counts, and to first[] (~position, 0: none) only while theirs beats the recorded
// one; zeros, often the most frequent of them, are counted per sub-chunk and added
// once.  The common code of eight in the window has no branch but the one that
// asks whether there is anything else to do: issue-bound (40 instructions a code
// with a test for each took 0.23 ms for the 134 M codes of a 512^3 field, 0.10 ms
// here; for the 37.7 M codes of a float64 field at rel 1e-6, 65,000 symbols, a
// global add and min for every code outside the window took 2.88 ms, 0.29 ms here).
// C: the code type, uint16_t, or uint32_t for quantisers of more than 65536 bins.
template <typename C>
__global__ void __launch_bounds__(HTHREADS) k_histogram(const C *__restrict__ codes, uint64_t n, uint64_t nsub,
                                                       uint64_t per_cta, int center, unsigned long long *hist,
                                                       unsigned long long *first, unsigned long long *zcount,
                                                       unsigned long long *nzero) {
    __shared__ unsigned scnt[HWIN + 1], sfirst[HWIN + 1];
    __shared__ unsigned long long ztotal;
    const int tid = threadIdx.x, lane = tid & 31;
    for (int i = tid; i <= HWIN; i += HTHREADS) {
        scnt[i] = 0;
        sfirst[i] = i < HWIN ? 0xffffffffu : 0u;  // the last bin's position is never beaten
    }
    if (tid == 0) ztotal = 0;
    __syncthreads();
    const int lo = center - HWIN / 2;
    const bool zero_inside = lo <= 0;
    const uint64_t c0 = blockIdx.x * per_cta;
    const uint64_t c1 = c0 + per_cta < nsub ? c0 + per_cta : nsub;
    const uint64_t base = c0 * HSUB;  // positions in the window are relative to it (below 2^32)
    auto outside = [&](int v, uint64_t i) {
        if (v != 0) {
            atomicAdd(&hist[v], 1ull);
            if (first[v] < ~(unsigned long long)i) atomicMax(&first[v], ~(unsigned long long)i);
        } else if (first[0] < ~(unsigned long long)i) {
            atomicMax(&first[0], ~(unsigned long long)i);
        }
    };
    for (uint64_t c = c0 + (tid >> 5); c < c1; c += HTHREADS / 32) {
        const uint64_t s0 = c * HSUB;
        unsigned zc = 0;
        if (sizeof(C) == 2 && s0 + HSUB <= n) {
            const uint4 *cv = reinterpret_cast<const uint4 *>(codes + s0) + lane;
            uint4 q = cv[0];
#pragma unroll 1
            for (int it = 0; it < (int)(HSUB / 256); it++) {
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
                if (it + 1 < (int)(HSUB / 256)) q = cv[32 * (it + 1)];
                const unsigned at = (unsigned)(s0 - base) + (unsigned)(256 * it + 8 * lane);
                unsigned todo = 0, out = 0;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const int v = (int)((w[k >> 1] >> (16 * (k & 1))) & 0xffffu);
                    const unsigned b = min((unsigned)(v - lo), (unsigned)HWIN);
                    atomicAdd(&scnt[b], 1u);
                    todo |= at + k < sfirst[b] ? 1u << k : 0u;
                    out |= b == HWIN ? 1u << k : 0u;
                    if (zero_inside) zc += v == 0;
                }
                if (todo | out) {
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const int v = (int)((w[k >> 1] >> (16 * (k & 1))) & 0xffffu);
                        if ((todo >> k) & 1) atomicMin(&sfirst[v - lo], at + k);
                        if ((out >> k) & 1) {
                            if (!zero_inside) zc += v == 0;
                            outside(v, s0 + (uint64_t)(256 * it + 8 * lane + k));
                        }
                    }
                }
            }
        } else {
            const uint64_t s1 = s0 + HSUB < n ? s0 + HSUB : n;
            for (uint64_t i = s0 + lane; i < s1; i += 32) {
                const int v = (int)codes[i];
                const unsigned b = (unsigned)(v - lo);
                zc += v == 0;
                if (b < HWIN) {
                    atomicAdd(&scnt[b], 1u);
                    if ((unsigned)(i - base) < sfirst[b]) atomicMin(&sfirst[b], (unsigned)(i - base));
                } else {
                    outside(v, i);
                }
            }
        }
        zc = __reduce_add_sync(0xffffffffu, zc);
        if (lane == 0) {
            zcount[c] = zc;
            if (zc) atomicAdd(&ztotal, (unsigned long long)zc);
        }
    }
    __syncthreads();
    for (int b = tid; b < HWIN; b += HTHREADS) {
        if (scnt[b]) {
            atomicAdd(&hist[lo + b], (unsigned long long)scnt[b]);
            const unsigned long long at = ~(unsigned long long)(base + sfirst[b]);
            if (first[lo + b] < at) atomicMax(&first[lo + b], at);
        }
    }
    if (tid == 0 && ztotal) {
        atomicAdd(nzero, ztotal);
        if (!zero_inside) atomicAdd(&hist[0], ztotal);
    }
}

// The symbols of non-zero count, compacted in no particular order:
// list[3k], list[3k+1], list[3k+2] = symbol, count, first position;
// *nlist = their number.
__global__ void __launch_bounds__(256) k_hist_compact(const unsigned long long *__restrict__ hist,
                                                     const unsigned long long *__restrict__ first, int nsym,
                                                     unsigned long long *list, unsigned int *nlist) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const bool nz = s < nsym && hist[s] != 0;
    const unsigned int m = __ballot_sync(0xffffffffu, nz);
    if (m == 0) return;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    unsigned int base = 0;
    if (lane == leader) base = atomicAdd(nlist, (unsigned int)__popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (nz) {
        const unsigned int k = base + (unsigned int)__popc(m & ((1u << lane) - 1u));
        list[3 * (size_t)k] = (unsigned long long)s;
        list[3 * (size_t)k + 1] = hist[s];
        list[3 * (size_t)k + 2] = ~first[s];
    }
}

// Zero-code count per warp sub-chunk, where no histogram of the same codes gives it.
__global__ void __launch_bounds__(1024) k_count_zeros(const uint16_t *__restrict__ codes, uint64_t n,
                                                      unsigned long long *zcount) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t s0 = (uint64_t)blockIdx.x * HCHUNK + (uint64_t)w * HSUB;
    uint64_t s1 = s0 + HSUB;
    if (s1 > n) s1 = n;
    unsigned int zc = 0;
    for (uint64_t i = s0 + lane; i < s1; i += 32) zc += codes[i] == 0;
    for (int o = 16; o > 0; o >>= 1) zc += __shfl_down_sync(0xffffffffu, zc, o);
    if (lane == 0) zcount[(uint64_t)blockIdx.x * HWARPS + w] = zc;
}

// Compaction of the zero codes of each warp sub-chunk, in stream order,
// starting at zoff[sub-chunk]: the values recorded at their positions (vals from
// scratch).
template <typename T, typename C>
__global__ void __launch_bounds__(1024) k_compact_zeros(const C *__restrict__ codes, uint64_t n,
                                                        const unsigned long long *zcount,
                                                        const unsigned long long *zoff, const T *scratch, T *vals) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t sub = (uint64_t)blockIdx.x * HWARPS + w;
    if (zcount[sub] == 0) return;
    const uint64_t s0 = sub * HSUB;
    uint64_t s1 = s0 + HSUB;
    if (s1 > n) s1 = n;
    unsigned long long run = zoff[sub];
    // 256 codes per warp step, four steps' loads in flight: lane L reads codes
    // [b + 8L, b + 8L + 8) with one 16-byte load (s0 is a multiple of HSUB and codes
    // is 256-byte aligned), so the zeros of a step come in stream order lane by lane
    uint64_t b = s0;
    for (; sizeof(C) == 2 && b + 1024 <= s1; b += 1024) {
        uint4 q[4];
#pragma unroll
        for (int r = 0; r < 4; r++) q[r] = *reinterpret_cast<const uint4 *>(codes + b + 256 * r + 8 * lane);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const uint32_t wd[4] = {q[r].x, q[r].y, q[r].z, q[r].w};
            unsigned int m = 0;  // bit k: code k of the lane's eight is zero
#pragma unroll
            for (int k = 0; k < 4; k++) {
                m |= (wd[k] & 0xffffu) == 0 ? 1u << (2 * k) : 0u;
                m |= (wd[k] >> 16) == 0 ? 1u << (2 * k + 1) : 0u;
            }
            if (!__any_sync(0xffffffffu, m != 0)) continue;
            const int c = __popc(m);
            int x = c;  // inclusive scan of the counts across lanes
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            const int total = __shfl_sync(0xffffffffu, x, 31);
            unsigned long long o = run + (unsigned long long)(x - c);
            while (m) {
                const int k = __ffs(m) - 1;
                m &= m - 1;
                vals[o] = scratch[b + 256 * r + 8 * lane + k];
                o++;
            }
            run += (unsigned long long)total;
        }
    }
    for (; b < s1; b += 32) {
        const uint64_t i = b + lane;
        const bool z = i < s1 && codes[i] == 0;
        const unsigned int bal = __ballot_sync(0xffffffffu, z);
        if (z) {
            const unsigned long long o = run + __popc(bal & ((1u << lane) - 1));
            vals[o] = scratch[i];
        }
        run += __popc(bal);
    }
}

// ------------------------------------------------------------------- scan
// Exclusive scan of n 64-bit values (out[n] = total): per-block totals,
// one-block scan of the totals, per-block scan with the block's offset.
static constexpr int SCAN_T = 512;
static constexpr int SCAN_E = 8;
static constexpr int SCAN_B = SCAN_T * SCAN_E;

__device__ __forceinline__ unsigned long long block_excl_scan(unsigned long long v, unsigned long long *sh,
                                                              unsigned long long &total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned long long x = v;
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        unsigned long long y = lane < nw ? sh[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long z = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) y += z;
        }
        sh[lane] = y;
    }
    __syncthreads();
    total = sh[nw - 1];
    unsigned long long wbase = w ? sh[w - 1] : 0;
    __syncthreads();
    return wbase + x - v;
}

__global__ void __launch_bounds__(SCAN_T) k_scan_reduce(const unsigned long long *in, uint64_t n,
                                                       unsigned long long *bsum) {
    __shared__ unsigned long long sh[32];
    uint64_t b0 = (uint64_t)blockIdx.x * SCAN_B;
    unsigned long long s = 0;
    for (int k = 0; k < SCAN_E; k++) {
        uint64_t i = b0 + (uint64_t)threadIdx.x * SCAN_E + k;
        if (i < n) s += in[i];
    }
    unsigned long long tot;
    block_excl_scan(s, sh, tot);
    if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

// one block: exclusive scan of nb block totals in place (nb <= any), total in bsum[nb]
__global__ void __launch_bounds__(1024) k_scan_top(unsigned long long *bsum, uint64_t nb) {
    __shared__ unsigned long long sh[32];
    unsigned long long carry = 0;
    for (uint64_t c = 0; c < nb; c += blockDim.x) {
        uint64_t i = c + threadIdx.x;
        unsigned long long v = i < nb ? bsum[i] : 0;
        unsigned long long tot;
        unsigned long long e = block_excl_scan(v, sh, tot);
        if (i < nb) bsum[i] = carry + e;
        carry += tot;
    }
    if (threadIdx.x == 0) bsum[nb] = carry;
}

__global__ void __launch_bounds__(SCAN_T) k_scan_down(const unsigned long long *in, uint64_t n,
                                                     const unsigned long long *bsum, unsigned long long *out,
                                                     uint64_t nb) {
    __shared__ unsigned long long sh[32];
    uint64_t b0 = (uint64_t)blockIdx.x * SCAN_B;
    unsigned long long v[SCAN_E];
    unsigned long long s = 0;
    for (int k = 0; k < SCAN_E; k++) {
        uint64_t i = b0 + (uint64_t)threadIdx.x * SCAN_E + k;
        v[k] = i < n ? in[i] : 0;
        s += v[k];
    }
    unsigned long long tot;
    unsigned long long e = block_excl_scan(s, sh, tot) + bsum[blockIdx.x];
    for (int k = 0; k < SCAN_E; k++) {
        uint64_t i = b0 + (uint64_t)threadIdx.x * SCAN_E + k;
        if (i < n) out[i] = e;
        e += v[k];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = bsum[nb];
}

// ------------------------------------------------------------------ encode
// Bits per chunk of ENC_CHUNK codes, their scan, then the packing.  (In one pass,
// the chunks' ends found by decoupled look-back, the 134 M codes of a 512^3 field
// took 670 us: 33,000 small chunks wait on one another.)  Long strings go through
// the three in slices, so that the first slice's copy to the host starts after an
// eighth of the bit counts, and the codes that the packing reads are still in L2:
// 1.83 -> 1.77 ms for the whole compression of that field.
// packed[state] = (length << 32) | code right-aligned (codes up to 32 bits);
// longer codes are read from code64 (MSB-aligned); len[state] = length.
static constexpr int ENC_PER_THREAD = 16;
static constexpr int ENC_THREADS = 256;
static constexpr int ENC_CHUNK = ENC_PER_THREAD * ENC_THREADS;

__device__ __forceinline__ uint32_t bswap32(uint32_t x) { return __byte_perm(x, 0, 0x0123); }

// the sixteen codes from t0 on, those past n - 1 zero
template <typename C>
__device__ __forceinline__ int enc_load(const C *__restrict__ codes, uint64_t n, uint64_t t0, C (&sym)[ENC_PER_THREAD]) {
    const int nvalid = t0 >= n ? 0 : (n - t0 >= ENC_PER_THREAD ? ENC_PER_THREAD : (int)(n - t0));
    if (sizeof(C) == 2 && nvalid == ENC_PER_THREAD) {
        // 16 codes = two 16-byte loads (codes is 256-byte aligned, t0 a multiple of 16)
        const uint4 *cv = reinterpret_cast<const uint4 *>(codes + t0);
        const uint4 qa = cv[0], qb = cv[1];
        const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
        for (int k = 0; k < ENC_PER_THREAD; k++) sym[k] = (C)((w[k >> 1] >> (16 * (k & 1))) & 0xffffu);
    } else {
#pragma unroll
        for (int k = 0; k < ENC_PER_THREAD; k++) sym[k] = k < nvalid ? codes[t0 + k] : (C)0;
    }
    return nvalid;
}

template <typename C>
__global__ void __launch_bounds__(ENC_THREADS) k_encode_bits(const C *__restrict__ codes, uint64_t n, int offset,
                                                            const uint8_t *__restrict__ len,
                                                            unsigned long long *chunkbits) {
    __shared__ unsigned ws[ENC_THREADS / 32];
    C sym[ENC_PER_THREAD];
    const int nvalid =
        enc_load(codes, n, (uint64_t)blockIdx.x * ENC_CHUNK + (uint64_t)threadIdx.x * ENC_PER_THREAD, sym);
    unsigned s = 0;
    if (nvalid == ENC_PER_THREAD) {
#pragma unroll
        for (int k = 0; k < ENC_PER_THREAD; k++) s += (unsigned)len[(int)sym[k] - offset];
    } else {
        for (int k = 0; k < nvalid; k++)
            s += (unsigned)len[(int)codes[(uint64_t)blockIdx.x * ENC_CHUNK + (uint64_t)threadIdx.x * ENC_PER_THREAD + k] -
                               offset];
    }
    s = __reduce_add_sync(0xffffffffu, s);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (int w = 0; w < ENC_THREADS / 32; w++) t += ws[w];
        chunkbits[blockIdx.x] = t;
    }
}

// Each thread packs ENC_PER_THREAD consecutive codes, four at a time while they
// fit in 32 bits together: about 30 thread instructions a code (pushed one by one
// 40, and 80% of the issue slots used; now 52%).  The 134 M codes of a 512^3 field: 26 us per eighth,
// behind the copy of the eighth before it (227 us in one piece before the copy).  Words in shared memory follow
// the 32-bit word grid of the output.
template <typename C>
__global__ void __launch_bounds__(ENC_THREADS) k_encode_pack(const C *__restrict__ codes, uint64_t n, int offset,
                                                            const unsigned long long *__restrict__ code64,
                                                            const unsigned long long *__restrict__ packed,
                                                            const unsigned long long *__restrict__ chunkoff,
                                                            uint64_t chunk0, uint32_t *out,
                                                            unsigned long long *host_end) {
    extern __shared__ uint32_t sw[];
    __shared__ unsigned wtot[ENC_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint64_t chunk = chunk0 + blockIdx.x;
    const unsigned long long gbit = chunkoff[chunk];
    const unsigned total = (unsigned)(chunkoff[chunk + 1] - gbit);
    // the end of a launch's codes, for the host that copies them
    if (host_end && tid == 0 && blockIdx.x == gridDim.x - 1) *(volatile unsigned long long *)host_end = gbit + total;
    if (total == 0) return;
    const uint64_t w0 = gbit >> 5;
    const int nwords = (int)(((gbit + total - 1) >> 5) - w0 + 1);
    for (int i = tid; i < nwords; i += ENC_THREADS) sw[i] = 0;
    // lengths and codes of this thread's symbols, zero bits for those past the end
    uint32_t code[ENC_PER_THREAD];
    unsigned len[ENC_PER_THREAD], mybits = 0;
    C sym[ENC_PER_THREAD];
    const int nvalid = enc_load(codes, n, chunk * ENC_CHUNK + (uint64_t)tid * ENC_PER_THREAD, sym);
    unsigned longest = 0;
    if (nvalid == ENC_PER_THREAD) {
        // no test per code: as branches they were most of the kernel's issue slots
#pragma unroll
        for (int k = 0; k < ENC_PER_THREAD; k++) {
            const unsigned long long e = packed[(int)sym[k] - offset];
            code[k] = (uint32_t)e;
            len[k] = (unsigned)(e >> 32);
        }
    } else {
#pragma unroll
        for (int k = 0; k < ENC_PER_THREAD; k++) {
            const unsigned long long e = k < nvalid ? packed[(int)sym[k] - offset] : 0ull;
            code[k] = (uint32_t)e;
            len[k] = (unsigned)(e >> 32);
        }
    }
#pragma unroll
    for (int k = 0; k < ENC_PER_THREAD; k++) {
        mybits += len[k];
        longest = max(longest, len[k]);
    }
    // exclusive scan of the threads' bit counts (warp shuffles + warp totals)
    unsigned x = mybits;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wtot[wid] = x;
    __syncthreads();
    unsigned before = x - mybits;
    for (int w = 0; w < wid; w++) before += wtot[w];
    // `word` is filled from the top, `fill` bits of it taken: the first bits of the
    // thread's first word are the thread's before it (ORed, as is its last word)
    const unsigned pos = (unsigned)(gbit & 31) + before;
    unsigned wi = pos >> 5, fill = pos & 31;
    const unsigned shared_word = wi;
    const bool shared_first = fill != 0;
    uint32_t word = 0;
    auto push = [&](uint32_t bits, unsigned l) {  // l <= 32, bits right-aligned
        const uint32_t top = __funnelshift_lc(0u, bits, 32 - l);  // bits << (32 - l), 0 for l = 0
        word |= top >> fill;
        const uint32_t next = __funnelshift_lc(0u, top, 32 - fill);
        fill += l;
        if (fill >= 32) {
            if (wi == shared_word && shared_first) atomicOr(&sw[wi], word);
            else sw[wi] = word;
            wi++;
            word = next;
            fill -= 32;
        }
    };
    if (longest <= 32) {
#pragma unroll
        for (int k = 0; k < ENC_PER_THREAD; k += 4) {
            const unsigned l01 = len[k] + len[k + 1], l23 = len[k + 2] + len[k + 3];
            if (l01 + l23 <= 32) {
                const uint32_t c01 = (code[k] << len[k + 1]) | code[k + 1];
                const uint32_t c23 = (code[k + 2] << len[k + 3]) | code[k + 3];
                push(__funnelshift_lc(0u, c01, l23) | c23, l01 + l23);
            } else {
#pragma unroll
                for (int j = k; j < k + 4; j++) push(code[j], len[j]);
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < ENC_PER_THREAD; k++) {
            if (len[k] <= 32) {
                push(code[k], len[k]);
            } else {
                // codes longer than 32 bits: right-align the MSB-aligned code
                const unsigned long long c = code64[(int)sym[k] - offset] >> (64 - len[k]);
                push((uint32_t)(c >> 32), len[k] - 32);
                push((uint32_t)c, 32);
            }
        }
    }
    if (fill > 0 && word) atomicOr(&sw[wi], word);
    __syncthreads();
    for (int i = tid; i < nwords; i += ENC_THREADS) {
        const uint32_t v = bswap32(sw[i]);
        if (i == 0 || i == nwords - 1) {
            if (v) atomicOr(&out[w0 + i], v);
        } else {
            out[w0 + i] = v;
        }
    }
}
// Where the chunks' bits begin: out[i] = out[0] + in[0] + .. + in[i - 1] for i <= n
// (`first`: out[0] = 0), by one CTA (a slice's 4096 chunks 8 us, a small string's
// 4; the general scan's three launches 13 and 9).  Also clears the words of the string in which a chunk
// begins or ends, which the packing ORs into (the words inside the chunks it
// stores); not the one a slice before this has begun.
__global__ void __launch_bounds__(1024) k_scan_chunks(const unsigned long long *__restrict__ in, uint64_t n,
                                                     unsigned long long *out, int first, uint32_t *words) {
    __shared__ unsigned long long sh[32];
    const unsigned long long begin = first ? 0 : out[0];
    unsigned long long carry = begin;
    // the word of a chunk's first bit, and that of the bit before it when it ends there
    auto clear = [&](unsigned long long bit) {
        if (first || (bit >> 5) > (begin >> 5)) words[bit >> 5] = 0;
        if ((bit & 31) == 0 && bit > 0 && (first || (bit >> 5) - 1 > (begin >> 5))) words[(bit >> 5) - 1] = 0;
    };
    for (uint64_t c = 0; c < n; c += 4096) {
        const uint64_t i0 = c + 4 * threadIdx.x;
        unsigned long long v[4], s = 0, tot;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = i0 + k < n ? in[i0 + k] : 0;
            s += v[k];
        }
        unsigned long long e = carry + block_excl_scan(s, sh, tot);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (i0 + k < n) {
                out[i0 + k] = e;
                clear(e);
            }
            e += v[k];
        }
        carry += tot;
    }
    if (threadIdx.x == 0) {
        out[n] = carry;
        clear(carry);
    }
}

// ------------------------------------------------------------------ decode
// The bit string is cut into units of DW 32-bit words, DEC_T units to a CTA.
//   k_decode_sync   every unit decodes from its nominal start (the codeword
//                   lengths alone), then the units of a CTA restart at their
//                   predecessor's end, in shared memory, until none moves;
//   k_decode_link   the first units of the CTAs restart at the previous CTA's
//                   end and the change runs on until it meets the recorded
//                   starts (one thread per CTA: nearly always within a unit);
//   k_decode_write  decodes the symbols and writes them.
// A table step takes every whole codeword of the next LUT_BITS bits, and four
// steps go through one 64-bit window in registers without a test for its end:
// the decode is bound by issue slots and shared-memory wavefronts, not by memory.
// For the 134 M codes (82 MB) of a 512^3 field the former per-symbol form (three
// segment words and a table word per symbol, two resynchronisation passes over
// every CTA) took 385 + 236 + 337 us, these passes 36 us per
// eighth of the string (hidden behind its copy but for the last) + 35 + 279 us.
// DW is odd so that the units of a warp start in different banks.
static constexpr int LUT_BITS = kLutBits;
static constexpr int LUT2_BITS = 8;                  // second table, below each prefix of a longer codeword
static constexpr uint32_t B_LONG = 1u << 12;         // lutB.y: longer codewords
static constexpr uint32_t DEC_NODE = 0x80000000u;    // second table: an inner node follows
static constexpr uint32_t DEC_LEAF = 0x80000000u;    // child: a leaf's state follows
static constexpr uint32_t DEC_BAD = 0x40000000u;     // child: a leaf with a negative state
static constexpr int DEC_T = 256;
static constexpr int DEC_HALO = 8;                   // words past the last unit
static constexpr int DEC_NB = 16;                    // boundaries recorded per unit
static constexpr int DEC_STEPS = 4;                  // table steps per 64-bit window
static_assert(DEC_STEPS * LUT_BITS <= 64, "a window holds its steps");
static constexpr int DEC_WT = 512;                   // units per CTA of the writing pass
static constexpr int DEC_ROWS = 3 + 2 * 4 + 1;       // words buffered per thread of it
// words per unit: long units for long bit strings (fewer restarts), short ones
// where there would be too few to fill the GPU (a 0.1 MB string has 1,450 units
// of 17 words, 6 CTAs)
static constexpr int DEC_LONG = 17, DEC_SHORT = 5;
static constexpr uint64_t DEC_SHORT_BITS = (uint64_t)1 << 25;

// lutA (per LUT_BITS prefix): length of the first codeword, bits and number of
// the whole codewords in the prefix, 4 bits each; a prefix of longer codewords
// has length 0 and its second-table slot << 4.
// lutB: up to three symbols (16 bits each, the third in y's high half; one of 32
// bits for wide codes), y's low half = their bits | first length << 4 | count << 8
// | zero symbols << 10; a prefix of longer codewords has y = B_LONG, x = slot.
// The second tables (per slot and next LUT2_BITS bits): lut2 as below, len2 the
// codeword's length alone (0: longer still, or damaged).  Longer codewords are
// a few per cent of the symbols, but with 32 lanes a warp meets one every few
// steps, so they cost one dependent load and no call.
__device__ __forceinline__ uint32_t dec_child(const uint32_t *child, uint32_t node, int bit) {
    return child[2 * (size_t)node + bit];
}

template <typename C>
__global__ void __launch_bounds__(256) k_decode_lut(const uint32_t *__restrict__ child, int offset, uint16_t *lutA,
                                                   uint2 *lutB, uint32_t *slot_node, unsigned *nslots) {
    const uint32_t v = blockIdx.x * 256 + threadIdx.x;
    uint32_t node = 0;
    int cnt = 0, bits_all = 0, bits_b = 0, len1 = 0, zeros = 0;
    uint32_t sx = 0, sy = 0;
    constexpr int maxsym = sizeof(C) == 2 ? 3 : 1;
    for (int b = 0; b < LUT_BITS; b++) {
        const uint32_t ch = dec_child(child, node, (v >> (LUT_BITS - 1 - b)) & 1);
        if (!(ch & DEC_LEAF)) {
            node = ch;
            continue;
        }
        const C sym = (C)((int)(ch & 0xffffffu) + offset);
        if (cnt < maxsym) {
            if (cnt < 2) sx |= (uint32_t)sym << (16 * cnt);
            else sy = (uint32_t)sym << 16;
            zeros += sym == 0;
            bits_b = b + 1;
        }
        if (cnt == 0) len1 = b + 1;
        cnt++;
        bits_all = b + 1;
        node = 0;
    }
    uint32_t slot = 0;
    if (cnt == 0) {
        slot = atomicAdd(nslots, 1u);
        slot_node[slot] = node;
    }
    lutA[v] = (uint16_t)(cnt == 0 ? slot << 4 : len1 | (bits_all << 4) | (cnt << 8));
    lutB[v] = cnt == 0 ? make_uint2(slot, B_LONG)
                       : make_uint2(sx, sy | (uint32_t)(bits_b | (len1 << 4) | ((cnt < maxsym ? cnt : maxsym) << 8) |
                                                        (zeros << 10)));
}

// Second table: CTA k fills the entries of slot k: (length << 24) | state, or
// DEC_NODE | node for codewords longer still, or 0 for a leaf without a state.
__global__ void __launch_bounds__(1 << LUT2_BITS) k_decode_lut2(const uint32_t *__restrict__ child,
                                                               const uint32_t *__restrict__ slot_node,
                                                               const unsigned *__restrict__ nslots, uint32_t *lut2,
                                                               uint8_t *len2) {
    if (blockIdx.x >= *nslots) return;
    uint32_t node = slot_node[blockIdx.x], e = 0;
    int b = 0;
    for (; b < LUT2_BITS; b++) {
        const uint32_t ch = dec_child(child, node, (threadIdx.x >> (LUT2_BITS - 1 - b)) & 1);
        if (ch & DEC_LEAF) {
            e = ch & DEC_BAD ? 0u : ((uint32_t)(LUT_BITS + b + 1) << 24) | (ch & 0xffffffu);
            break;
        }
        node = ch;
    }
    if (b == LUT2_BITS) e = DEC_NODE | node;
    lut2[((size_t)blockIdx.x << LUT2_BITS) + threadIdx.x] = e;
    len2[((size_t)blockIdx.x << LUT2_BITS) + threadIdx.x] = (uint8_t)(e & DEC_NODE ? 0u : e >> 24);
}

// A codeword longer than LUT_BITS + LUT2_BITS at the front of `win`, below
// second-table entry e: its length (0: damaged tree or longer than 64 bits) and
// state.
__device__ __noinline__ uint2 dec_long(const uint32_t *__restrict__ child, uint32_t e, uint64_t win) {
    if (!(e & DEC_NODE)) return make_uint2(0u, 0u);
    uint32_t node = e & 0xffffffu;
    for (int b = LUT_BITS + LUT2_BITS; b < 64; b++) {
        const uint32_t ch = dec_child(child, node, (int)((win >> (63 - b)) & 1));
        if (ch & DEC_LEAF) return make_uint2(ch & DEC_BAD ? 0u : (uint32_t)b + 1, ch & 0xffffffu);
        node = ch;
    }
    return make_uint2(0u, 0u);
}

__device__ __forceinline__ uint32_t bswap_w(uint32_t x) { return __byte_perm(x, 0, 0x0123); }

// word i of the bit string, staged in shared memory / read from global memory
struct WordsShared {
    const uint32_t *sw;
    __device__ __forceinline__ uint32_t operator()(uint32_t i) const { return sw[i]; }
};
struct WordsGlobal {
    const uint32_t *w32;
    uint64_t base, nwords;
    __device__ __forceinline__ uint32_t operator()(uint32_t i) const {
        return base + i < nwords ? bswap_w(w32[base + i]) : 0u;
    }
};

// 32 and 64 bits of the string from bit p
template <typename Words>
__device__ __forceinline__ uint32_t peek32(const Words &words, uint32_t p) {
    return __funnelshift_l(words((p >> 5) + 1), words(p >> 5), p & 31);
}
template <typename Words>
__device__ __forceinline__ uint64_t peek64(const Words &words, uint32_t p) {
    const uint32_t w = p >> 5, b = words(w + 1);
    return ((uint64_t)__funnelshift_l(b, words(w), p & 31) << 32) | __funnelshift_l(words(w + 2), b, p & 31);
}

// Entry of a slot's second table for the window `win`.
__device__ __forceinline__ size_t lut2_index(uint32_t slot, uint32_t win) {
    return ((size_t)slot << LUT2_BITS) + ((win >> (32 - LUT_BITS - LUT2_BITS)) & ((1u << LUT2_BITS) - 1));
}

// Length of the codeword at bit p (0: damaged).
template <typename Words>
__device__ __forceinline__ uint32_t dec_len(const DecodeTablesDev &t, const uint16_t *slut, const Words &words,
                                            uint32_t p) {
    const uint32_t win = peek32(words, p), e = slut[win >> (32 - LUT_BITS)];
    uint32_t n = e & 15;
    if (n == 0) {
        const size_t i = lut2_index(e >> 4, win);
        n = t.len2[i];
        if (n == 0) n = dec_long(t.child, t.lut2[i], peek64(words, p)).x;
    }
    return n;
}

// Pass codewords from bit p to the first boundary at or past `stop`: returns
// the boundary and adds the codewords to c.  On damage *err is set and `stop`
// returned, so that later passes stay within the unit.
template <typename Words>
__device__ __forceinline__ uint32_t dec_skip(const DecodeTablesDev &t, const uint16_t *slut, const Words &words,
                                             uint32_t p, uint32_t stop, unsigned &c, int *err) {
    // four whole prefixes at a time while they end within the unit
    while (p + DEC_STEPS * LUT_BITS <= stop) {
        const uint64_t win = peek64(words, p);
        uint32_t hi = (uint32_t)(win >> 32), lo = (uint32_t)win;
#pragma unroll
        for (int k = 0; k < DEC_STEPS; k++) {
            const uint32_t e = slut[hi >> (32 - LUT_BITS)];
            if ((e & 15) == 0) {
                const uint32_t n = dec_len(t, slut, words, p);
                if (n == 0) {
                    atomicExch(err, 1);
                    return stop;
                }
                p += n;
                c++;
                break;
            }
            const uint32_t b = (e >> 4) & 15;
            p += b;
            c += e >> 8;
            hi = __funnelshift_l(lo, hi, b);
            lo <<= b;
        }
    }
    while (p + LUT_BITS <= stop) {
        const uint32_t e = slut[peek32(words, p) >> (32 - LUT_BITS)];
        if ((e & 15) == 0) break;
        p += (e >> 4) & 15;
        c += e >> 8;
    }
    while (p < stop) {
        const uint32_t n = dec_len(t, slut, words, p);
        if (n == 0) {
            atomicExch(err, 1);
            return stop;
        }
        p += n;
        c++;
    }
    return p;
}

// The first run_bits of the string are expected to hold codewords of run_len
// bits (the anchor grid: the zero code over and over, which a decode that starts
// between two of them need never fall in step with; the units of such a run
// then settle one per restart, 0.5 ms for 1152 anchors): units there start at a
// multiple of run_len.  Like every start it is a guess that the restarts check.
// info[u]: start of unit u past its nominal start (< 64) | codewords << 8.
// cend[c]: end of CTA c's last unit past that unit's nominal end.
template <int DW>
__global__ void __launch_bounds__(DEC_T) k_decode_sync(DecodeTablesDev t, const uint32_t *__restrict__ w32,
                                                      uint64_t nwords, uint64_t nbits, uint64_t nunits, uint64_t cta0,
                                                      uint64_t run_bits, uint32_t run_len,
                                                      uint32_t *__restrict__ info, uint32_t *__restrict__ cend,
                                                      unsigned long long *__restrict__ ctot, int *flags) {
    constexpr uint32_t UNIT = DW * 32;
    constexpr int SEG = DEC_T * DW + DEC_HALO;
    __shared__ uint16_t slut[1 << LUT_BITS];
    __shared__ uint32_t sw[SEG];
    __shared__ uint16_t bnd[DEC_NB][DEC_T];
    __shared__ uint32_t send[DEC_T];
    __shared__ unsigned wsum[DEC_T / 32];
    const int tid = threadIdx.x;
    const uint64_t cta = cta0 + blockIdx.x;
    const uint64_t u0 = cta * DEC_T, g0 = u0 * UNIT;
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(t.lutA);
        for (int i = tid; i < (1 << LUT_BITS) / 8; i += DEC_T) reinterpret_cast<uint4 *>(slut)[i] = src[i];
        const uint64_t wb = u0 * DW;
        for (int i = tid; i < SEG; i += DEC_T) sw[i] = wb + i < nwords ? bswap_w(w32[wb + i]) : 0u;
    }
    __syncthreads();
    const uint64_t u = u0 + tid;
    const bool act = u < nunits;
    const uint32_t nominal = (uint32_t)tid * UNIT;
    uint32_t stop = nominal + UNIT;
    if (nbits - g0 < stop) stop = (uint32_t)(nbits - g0);
    const WordsShared words{sw};
    // speculative decode from the nominal start; its first boundaries are kept
    unsigned spec_cnt = 0;
    uint32_t spec_end = nominal, spec_start = nominal;
    if (act) {
        if (g0 + nominal < run_bits) {
            const uint32_t over = (uint32_t)((g0 + nominal) % run_len);
            if (over) spec_start += run_len - over;
        }
        int k = 0;
        uint32_t p = spec_start;
        for (; k < DEC_NB && p < stop; k++) {
            bnd[k][tid] = (uint16_t)(p - nominal);
            const uint32_t n = dec_len(t, slut, words, p);
            if (n == 0) break;  // reported by dec_skip
            p += n;
        }
        spec_cnt = k;
        for (; k < DEC_NB; k++) bnd[k][tid] = 0xffff;
        spec_end = dec_skip(t, slut, words, p, stop, spec_cnt, flags + 1);
    }
    // restart at the predecessor's end until no end moves; a decode that meets
    // a boundary of the speculative one coincides with it from there
    uint32_t start = spec_start, end = spec_end;
    unsigned cnt = spec_cnt;
    send[tid] = end;
    for (int it = 0; it < DEC_T; it++) {
        __syncthreads();
        const uint32_t s = tid ? send[tid - 1] : spec_start;
        const uint32_t was = end;
        if (act && s != start) {
            start = s;
            uint32_t p = s;
            unsigned c = 0;
            int j = 0;
            bool met = false;
            while (p < stop) {
                const uint32_t off = p - nominal;
                while (j < DEC_NB && bnd[j][tid] < off) j++;
                if (j == DEC_NB) break;
                if (bnd[j][tid] == off) {
                    met = true;
                    break;
                }
                const uint32_t n = dec_len(t, slut, words, p);
                if (n == 0) break;
                c++;
                p += n;
            }
            if (met) {
                c += spec_cnt - j;
                end = spec_end;
            } else {
                end = dec_skip(t, slut, words, p, stop, c, flags + 1);
            }
            cnt = c;
        }
        if (!__syncthreads_or(end != was)) break;
        send[tid] = end;
    }
    if (act) info[u] = (start - nominal) | (cnt << 8);
    if (tid == DEC_T - 1) cend[cta] = end - (nominal + UNIT);
    unsigned x = act ? cnt : 0;
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((tid & 31) == 0) wsum[tid >> 5] = x;
    __syncthreads();
    if (tid == 0) {
        unsigned s = 0;
        for (int i = 0; i < DEC_T / 32; i++) s += wsum[i];
        ctot[cta] = s;
    }
}

// Thread c: the units of CTA c from the end of CTA c - 1, until one starts
// where it was recorded to start.  cend_in / cend_out: ends before and after
// this pass; *flags = 1 when a CTA's end moved (another pass is needed).
template <int DW>
__global__ void __launch_bounds__(64) k_decode_link(DecodeTablesDev t, const uint32_t *__restrict__ w32,
                                                   uint64_t nwords, uint64_t nbits, uint64_t nunits, uint64_t ncta,
                                                   const uint32_t *__restrict__ cend_in, uint32_t *__restrict__ cend_out,
                                                   uint32_t *info, unsigned long long *ctot, int *flags) {
    constexpr uint32_t UNIT = DW * 32;
    constexpr int ROW = DW + 4;  // a unit's words and the three past it (odd: distinct banks)
    __shared__ uint16_t slut[1 << LUT_BITS];
    __shared__ uint32_t first[64 * ROW];
    for (int i = threadIdx.x; i < (1 << LUT_BITS) / 8; i += 64)
        reinterpret_cast<uint4 *>(slut)[i] = reinterpret_cast<const uint4 *>(t.lutA)[i];
    // the CTAs' first units, where the change nearly always ends: read word by
    // word from global memory they took 58 us of a 512^3 field's decode
    for (int i = threadIdx.x; i < 64 * ROW; i += 64) {
        const uint64_t w = ((uint64_t)blockIdx.x * 64 + i / ROW) * (DEC_T * DW) + i % ROW;
        first[i] = w < nwords ? bswap_w(w32[w]) : 0u;
    }
    __syncthreads();
    const uint64_t c = (uint64_t)blockIdx.x * 64 + threadIdx.x;
    if (c >= ncta) return;
    const uint32_t old_end = cend_in[c];
    uint32_t new_end = old_end;
    if (c > 0) {
        const uint64_t u0 = c * DEC_T, g0 = u0 * UNIT;
        uint32_t s = cend_in[c - 1];
        long long delta = 0;
        const WordsShared wf{first + threadIdx.x * ROW};
        const WordsGlobal wg{w32, u0 * DW, nwords};
        int k = 0;
        for (; k < DEC_T && u0 + k < nunits; k++) {
            const uint32_t rec = info[u0 + k];
            if ((rec & 255u) == s) break;
            uint32_t stop = (uint32_t)(k + 1) * UNIT;
            if (nbits - g0 < stop) stop = (uint32_t)(nbits - g0);
            unsigned n = 0;
            const uint32_t e = k == 0 ? dec_skip(t, slut, wf, s, stop, n, flags + 1)
                                      : dec_skip(t, slut, wg, (uint32_t)k * UNIT + s, stop, n, flags + 1);
            info[u0 + k] = s | (n << 8);
            delta += (long long)n - (long long)(rec >> 8);
            const uint32_t next = (uint32_t)(k + 1) * UNIT;
            s = e > next ? e - next : 0u;
        }
        if (k == DEC_T) new_end = s;
        if (delta) ctot[c] += (unsigned long long)delta;
    }
    cend_out[c] = new_end;
    if (new_end != old_end) atomicExch(flags, 1);
}

// Decode unit u from its start into out[offset of u...): 16-byte stores of
// eight 16-bit codes, the ends of a unit's range as single codes.  Warp w's codes
// begin at zstart[w] and hold zc[w] zeros (for the compaction of the
// unpredictable ones).  Issue-bound: a step takes up to three symbols; whole
// words of two codes go to the thread's column of a shared buffer (one bank, no
// conflicts), from which the threads store together.  Packing in registers with
// a store whenever a thread's 16 bytes were full took 216 M warp instructions for
// the 134 M codes of a 512^3 field, this 139 M (0.28 ms).
template <typename C, int DW>
__global__ void __launch_bounds__(DEC_WT) k_decode_write(DecodeTablesDev t, const uint32_t *__restrict__ w32,
                                                        uint64_t nwords, uint64_t nunits,
                                                        const uint32_t *__restrict__ info,
                                                        const unsigned long long *__restrict__ coff, uint64_t nout,
                                                        int offset, C *out, unsigned long long *zc,
                                                        unsigned long long *zstart) {
    extern __shared__ __align__(16) unsigned char dsm[];
    uint2 *slut = reinterpret_cast<uint2 *>(dsm);
    uint32_t *sw = reinterpret_cast<uint32_t *>(dsm + ((size_t)8 << LUT_BITS));
    __shared__ unsigned wsum[DEC_WT / 32];
    constexpr int SEG = DEC_WT * DW + DEC_HALO;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint32_t *col = sw + SEG + wid * (DEC_ROWS * 32) + lane;
    const uint64_t u0 = (uint64_t)blockIdx.x * DEC_WT;
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(t.lutB);
        for (int i = tid; i < (1 << LUT_BITS) / 2; i += DEC_WT) reinterpret_cast<uint4 *>(slut)[i] = src[i];
        const uint64_t wb = u0 * DW;
        for (int i = tid; i < SEG; i += DEC_WT) sw[i] = wb + i < nwords ? bswap_w(w32[wb + i]) : 0u;
    }
    const WordsShared words{sw};
    const uint64_t u = u0 + tid;
    const uint32_t rec = u < nunits ? info[u] : 0u;
    unsigned n = rec >> 8, x = n;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[wid] = x;
    __syncthreads();
    if (u0 + (uint64_t)wid * 32 >= nunits) return;  // no unit in this warp
    uint64_t o = coff[u0 / DEC_T] + (x - n);
    for (int w = 0; w < wid; w++) o += wsum[w];
    if (lane == 0) zstart[u >> 5] = o;
    if (o >= nout) n = 0;
    else if (nout - o < n) n = (unsigned)(nout - o);
    uint32_t p = (uint32_t)tid * (DW * 32) + (rec & 255u);
    unsigned left = n, nz = 0;
    // a codeword longer than the prefix in `win`, slot e.x, as an entry of one
    // symbol; returns its bits (0 on damage, reported by the passes before)
    auto long_entry = [&](uint2 &e, uint32_t win) -> uint32_t {
        const uint32_t e2 = t.lut2[lut2_index(e.x, win)];
        uint32_t state = e2 & 0xffffffu, bits = e2 >> 24;
        if ((int32_t)e2 <= 0) {
            const uint2 l = dec_long(t.child, e2, peek64(words, p));
            bits = l.x;
            state = l.y;
        }
        const C sym = (C)((int)state + offset);
        e = make_uint2(sym, (1u << 8) | (sym == 0 ? 1u << 10 : 0u));
        return bits;
    };
    if constexpr (sizeof(C) != 2) {  // wide codes: one store per symbol
        for (; left; left--) {
            const uint32_t win = peek32(words, p);
            uint2 e = slut[win >> (32 - LUT_BITS)];
            const uint32_t bits = e.y & B_LONG ? long_entry(e, win) : e.y & 15;
            if (bits == 0) break;
            p += bits;
            out[o + (n - left)] = (C)e.x;
            nz += e.x == 0;
        }
    } else {
        // the column holds whole words of two codes from ob on (k of them) and
        // `pend` the low half of the next one when half = 1; the first `lead`
        // codes at ob belong to the unit before
        uint16_t *ob = (uint16_t *)out + (o & ~(uint64_t)7);
        unsigned lead = (unsigned)(o & 7), k = lead >> 1, half = lead & 1;
        uint32_t pend = 0;
        // c codes of entry e, (pend,) s0, s1, s2 as two words; rows past the last
        // whole one are written again
        auto push = [&](uint2 e, unsigned c) {
            const uint32_t w0 = __byte_perm(pend, e.x, half ? 0x5410 : 0x7654);
            const uint32_t w1 = __byte_perm(e.x, e.y, half ? 0x7632 : 0x1076);
            col[32 * k] = w0;
            col[32 * k + 32] = w1;
            const unsigned tot = half + c;
            pend = tot < 2 ? w0 : w1;
            k += tot >> 1;
            half = tot & 1;
            left -= c;
        };
        auto store8 = [&](const uint32_t *cg) {
            const uint32_t q0 = cg[0], q1 = cg[32], q2 = cg[64], q3 = cg[96];
            if (lead == 0) {
                *reinterpret_cast<uint4 *>(ob) = make_uint4(q0, q1, q2, q3);
            } else {
                for (unsigned i = lead; i < 8; i++) {
                    const uint32_t w = i < 4 ? (i < 2 ? q0 : q1) : (i < 6 ? q2 : q3);
                    ob[i] = (uint16_t)(w >> (16 * (i & 1)));
                }
                lead = 0;
            }
            ob += 8;
        };
        auto flush = [&] {  // whole groups of eight codes; up to three words move down
            if (k >= 4) {
                store8(col);
                if (k >= 8) store8(col + 128);
                const uint32_t *cl = col + 32 * (k & ~3u);
                const uint32_t a = cl[0], b = cl[32], c = cl[64];
                col[0] = a;
                col[32] = b;
                col[64] = c;
                k &= 3;
            }
        };
        while (__any_sync(0xffffffffu, left >= 3 * DEC_STEPS)) {
            if (left >= 3 * DEC_STEPS) {
                const uint64_t win = peek64(words, p);
                uint32_t hi = (uint32_t)(win >> 32), lo = (uint32_t)win;
#pragma unroll
                for (int s = 0; s < DEC_STEPS; s++) {
                    uint2 e = slut[hi >> (32 - LUT_BITS)];
                    if (e.y & B_LONG) {
                        // its bits may reach past the window
                        const uint32_t b = long_entry(e, peek32(words, p));
                        if (b) {
                            p += b;
                            nz += (e.y >> 10) & 3;
                            push(e, 1);
                        } else {
                            left = 0;
                        }
                        break;
                    }
                    const uint32_t b = e.y & 15;
                    p += b;
                    hi = __funnelshift_l(lo, hi, b);
                    lo <<= b;
                    nz += (e.y >> 10) & 3;
                    push(e, (e.y >> 8) & 3);
                }
                flush();
            }
        }
        while (left) {
            const uint32_t win = peek32(words, p);
            uint2 e = slut[win >> (32 - LUT_BITS)];
            uint32_t b = e.y & 15;
            if (e.y & B_LONG) b = long_entry(e, win);
            if (b == 0) break;
            unsigned c = (e.y >> 8) & 3, z = (e.y >> 10) & 3;
            if (c > left) {  // the unit's last codes, one or two
                c = left;
                z = ((e.x & 0xffffu) == 0) + (c > 1 && (e.x >> 16) == 0);
            }
            p += b;
            nz += z;
            push(e, c);
            if (k >= 8) flush();
        }
        flush();
        for (unsigned i = lead; i < 2 * k; i++) ob[i] = (uint16_t)(col[32 * (i >> 1)] >> (16 * (i & 1)));
        if (half && 2 * k >= lead) ob[2 * k] = (uint16_t)pend;
    }
    __syncwarp();
    for (int d = 16; d > 0; d >>= 1) nz += __shfl_down_sync(0xffffffffu, nz, d);
    if (lane == 0) zc[u >> 5] = nz;
}

// The ranges of a stream of one symbol: RANGE codes each, all of them zero or
// none.
static constexpr uint64_t RANGE = 4096;
__global__ void __launch_bounds__(256) k_constant_ranges(uint64_t n, int zero, unsigned long long *zstart,
                                                        unsigned long long *zcount) {
    const uint64_t s = ((uint64_t)blockIdx.x * 256 + threadIdx.x) * RANGE;
    if (s >= n) return;
    zstart[s / RANGE] = s;
    zcount[s / RANGE] = zero ? (n - s < RANGE ? n - s : RANGE) : 0;
}

// Positions of the zero codes of the decoder's warps, in stream order: warp w's
// codes [zstart[w], zstart[w + 1]) hold zcount[w] zeros, the first of them the
// zoff[w]-th; the first `cap` positions are written.
template <typename C>
__global__ void __launch_bounds__(256) k_zero_positions(const C *__restrict__ codes, uint64_t n, uint64_t nranges,
                                                       const unsigned long long *__restrict__ zstart,
                                                       const unsigned long long *__restrict__ zcount,
                                                       const unsigned long long *__restrict__ zoff, uint64_t cap,
                                                       uint64_t *zpos) {
    const uint64_t w = (uint64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (w >= nranges || zcount[w] == 0) return;
    const int lane = threadIdx.x & 31;
    uint64_t s1 = w + 1 < nranges ? zstart[w + 1] : n;
    if (s1 > n) s1 = n;
    unsigned long long run = zoff[w];
    for (uint64_t b = zstart[w]; b < s1; b += 128) {
        // four rows of 32 codes in flight
        bool z[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint64_t i = b + 32 * k + lane;
            z[k] = i < s1 && codes[i] == 0;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const unsigned bal = __ballot_sync(0xffffffffu, z[k]);
            const unsigned long long o = run + __popc(bal & ((1u << lane) - 1));
            if (z[k] && o < cap) zpos[o] = b + 32 * k + lane;
            run += __popc(bal);
        }
    }
}

template <typename C>
__global__ void k_fill_u16(C *out, uint64_t n, C v) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = v;
}

// ------------------------------------------------------------ launchers

static inline unsigned grid_for(uint64_t n, uint64_t per) { return (unsigned)((n + per - 1) / per); }

uint64_t hist_subchunks(uint64_t n) { return ((n + HCHUNK - 1) / HCHUNK) * HWARPS; }

cudaError_t launch_hist_compact(const unsigned long long *hist, const unsigned long long *first, int nsym,
                                unsigned long long *list, unsigned int *nlist, cudaStream_t st) {
    k_hist_compact<<<(unsigned)((nsym + 255) / 256), 256, 0, st>>>(hist, first, nsym, list, nlist);
    return cudaGetLastError();
}

// hist, first and *nzero zeroed by the caller
template <typename C>
cudaError_t histogram_impl(const C *codes, uint64_t n, int center, unsigned long long *hist,
                           unsigned long long *first, unsigned long long *zcount, unsigned long long *nzero,
                           cudaStream_t st) {
    const uint64_t used = (n + HSUB - 1) / HSUB, nsub = hist_subchunks(n);
    // four CTAs per SM in one wave, at least a sub-chunk per warp each; a CTA's run
    // stays below 2^32 codes
    const uint64_t warps = HTHREADS / 32, wave = 4 * (uint64_t)sm_count();
    uint64_t per_cta = std::max<uint64_t>((used + wave - 1) / wave, std::min<uint64_t>(warps, 4));
    per_cta = std::min<uint64_t>(per_cta, (1ull << 31) / HSUB);
    // the sub-chunks past the last code
    cudaError_t e = cudaSuccess;
    if (nsub > used) e = cudaMemsetAsync(zcount + used, 0, (nsub - used) * 8, st);
    if (e != cudaSuccess) return e;
    k_histogram<C><<<grid_for(used, per_cta), HTHREADS, 0, st>>>(codes, n, used, per_cta, center, hist, first, zcount,
                                                                  nzero);
    return cudaGetLastError();
}
cudaError_t launch_histogram(const uint16_t *codes, uint64_t n, int center, unsigned long long *hist,
                             unsigned long long *first, unsigned long long *zcount, unsigned long long *nzero,
                             cudaStream_t st) {
    return histogram_impl(codes, n, center, hist, first, zcount, nzero, st);
}
cudaError_t launch_histogram(const uint32_t *codes, uint64_t n, int center, unsigned long long *hist,
                             unsigned long long *first, unsigned long long *zcount, unsigned long long *nzero,
                             cudaStream_t st) {
    return histogram_impl(codes, n, center, hist, first, zcount, nzero, st);
}

cudaError_t launch_count_zeros(const uint16_t *codes, uint64_t n, unsigned long long *zcount, cudaStream_t st) {
    k_count_zeros<<<grid_for(n, HCHUNK), 1024, 0, st>>>(codes, n, zcount);
    return cudaGetLastError();
}

template <typename T, typename C>
cudaError_t launch_compact_zeros(const C *codes, uint64_t n, const unsigned long long *zcount,
                                 const unsigned long long *zoff, const T *scratch, T *vals, cudaStream_t st) {
    k_compact_zeros<T, C><<<grid_for(n, HCHUNK), 1024, 0, st>>>(codes, n, zcount, zoff, scratch, vals);
    return cudaGetLastError();
}
#define FAZ_INST_COMPACT(T, C)                                                                               \
    template cudaError_t launch_compact_zeros<T, C>(const C *, uint64_t, const unsigned long long *,       \
                                                    const unsigned long long *, const T *, T *, cudaStream_t);
FAZ_INST_COMPACT(float, uint16_t)
FAZ_INST_COMPACT(double, uint16_t)
FAZ_INST_COMPACT(float, uint32_t)
FAZ_INST_COMPACT(double, uint32_t)
#undef FAZ_INST_COMPACT

uint64_t scan_temp_words(uint64_t n) { return (n + SCAN_B - 1) / SCAN_B + 1; }

cudaError_t launch_scan_u64(const unsigned long long *in, unsigned long long *out, uint64_t n,
                            unsigned long long *temp, cudaStream_t st) {
    uint64_t nb = (n + SCAN_B - 1) / SCAN_B;
    if (nb == 0) nb = 1;
    k_scan_reduce<<<(unsigned)nb, SCAN_T, 0, st>>>(in, n, temp);
    k_scan_top<<<1, 1024, 0, st>>>(temp, nb);
    k_scan_down<<<(unsigned)nb, SCAN_T, 0, st>>>(in, n, temp, out, nb);
    return cudaGetLastError();
}

uint64_t encode_chunks(uint64_t n) { return (n + ENC_CHUNK - 1) / ENC_CHUNK; }

template <typename C>
cudaError_t encode_pack_impl(const EncodeArgs &a, const C *codes, uint64_t n, uint64_t chunk0, uint64_t chunk1,
                             unsigned long long *host_end, cudaStream_t st) {
    if (chunk1 <= chunk0) return cudaSuccess;
    const int words = (int)(((uint64_t)ENC_CHUNK * (uint64_t)a.maxlen + 31) / 32 + 2);
    cudaError_t e = allow_dynamic_smem((const void *)k_encode_pack<C>);
    if (e != cudaSuccess) return e;
    const uint64_t n0 = chunk0 * ENC_CHUNK, n1 = std::min<uint64_t>(n, chunk1 * ENC_CHUNK);
    k_encode_bits<C><<<(unsigned)(chunk1 - chunk0), ENC_THREADS, 0, st>>>(codes + n0, n1 - n0, a.offset, a.len,
                                                                         a.chunkbits + chunk0);
    k_scan_chunks<<<1, 1024, 0, st>>>(a.chunkbits + chunk0, chunk1 - chunk0, a.chunkoff + chunk0, chunk0 == 0, a.out);
    k_encode_pack<C><<<(unsigned)(chunk1 - chunk0), ENC_THREADS, (size_t)words * 4, st>>>(
        codes, n, a.offset, a.code64, a.packed, a.chunkoff, chunk0, a.out, host_end);
    return cudaGetLastError();
}
cudaError_t launch_encode_pack(const EncodeArgs &a, const uint16_t *codes, uint64_t n, uint64_t chunk0,
                               uint64_t chunk1, unsigned long long *host_end, cudaStream_t st) {
    return encode_pack_impl(a, codes, n, chunk0, chunk1, host_end, st);
}
cudaError_t launch_encode_pack(const EncodeArgs &a, const uint32_t *codes, uint64_t n, uint64_t chunk0,
                               uint64_t chunk1, unsigned long long *host_end, cudaStream_t st) {
    return encode_pack_impl(a, codes, n, chunk0, chunk1, host_end, st);
}

int decode_unit_words(uint64_t nbits) { return nbits < DEC_SHORT_BITS ? DEC_SHORT : DEC_LONG; }
uint64_t decode_cta_units() { return DEC_T; }
size_t decode_lut2_entries(size_t slots) { return slots << LUT2_BITS; }

template <typename C>
cudaError_t launch_decode_tables(const DecodeTablesDev &t, int offset, uint32_t *slot_node, unsigned *nslots,
                                 size_t lut2_entries, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(nslots, 0, 4, st);
    if (e != cudaSuccess) return e;
    k_decode_lut<C><<<(1 << LUT_BITS) / 256, 256, 0, st>>>(t.child, offset, t.lutA, t.lutB, slot_node, nslots);
    k_decode_lut2<<<(unsigned)(lut2_entries >> LUT2_BITS), 1 << LUT2_BITS, 0, st>>>(t.child, slot_node, nslots, t.lut2,
                                                                                    t.len2);
    return cudaGetLastError();
}
template cudaError_t launch_decode_tables<uint16_t>(const DecodeTablesDev &, int, uint32_t *, unsigned *, size_t,
                                                    cudaStream_t);
template cudaError_t launch_decode_tables<uint32_t>(const DecodeTablesDev &, int, uint32_t *, unsigned *, size_t,
                                                    cudaStream_t);

cudaError_t launch_decode_sync(const DecodeTablesDev &t, const DecodeString &d, uint64_t cta0, uint64_t cta1,
                               uint32_t *info, uint32_t *cend, unsigned long long *ctot, int *flags, cudaStream_t st) {
    if (cta1 <= cta0) return cudaSuccess;
    auto k = d.unit_words == DEC_LONG ? k_decode_sync<DEC_LONG> : k_decode_sync<DEC_SHORT>;
    k<<<(unsigned)(cta1 - cta0), DEC_T, 0, st>>>(t, d.w32, d.nwords, d.nbits, d.nunits, cta0, d.run_bits, d.run_len, info,
                                                 cend, ctot, flags);
    return cudaGetLastError();
}

cudaError_t launch_decode_link(const DecodeTablesDev &t, const DecodeString &d, const uint32_t *cend_in,
                               uint32_t *cend_out, uint32_t *info, unsigned long long *ctot, int *flags,
                               cudaStream_t st) {
    const uint64_t ncta = (d.nunits + DEC_T - 1) / DEC_T;
    auto k = d.unit_words == DEC_LONG ? k_decode_link<DEC_LONG> : k_decode_link<DEC_SHORT>;
    k<<<grid_for(ncta, 64), 64, 0, st>>>(t, d.w32, d.nwords, d.nbits, d.nunits, ncta, cend_in, cend_out, info, ctot,
                                          flags);
    return cudaGetLastError();
}

template <typename C>
cudaError_t launch_decode_write(const DecodeTablesDev &t, const DecodeString &d, const uint32_t *info,
                                const unsigned long long *coff, uint64_t nout, int offset, C *out,
                                unsigned long long *zc, unsigned long long *zstart, cudaStream_t st) {
    auto k = d.unit_words == DEC_LONG ? k_decode_write<C, DEC_LONG> : k_decode_write<C, DEC_SHORT>;
    const size_t sm = ((size_t)8 << LUT_BITS) + (size_t)(DEC_WT * d.unit_words + DEC_HALO) * 4 +
                      (size_t)DEC_WT * DEC_ROWS * 4;
    cudaError_t e = allow_dynamic_smem((const void *)k);
    if (e != cudaSuccess) return e;
    k<<<grid_for(d.nunits, DEC_WT), DEC_WT, sm, st>>>(t, d.w32, d.nwords, d.nunits, info, coff, nout, offset, out, zc,
                                              zstart);
    return cudaGetLastError();
}
template cudaError_t launch_decode_write<uint16_t>(const DecodeTablesDev &, const DecodeString &, const uint32_t *,
                                                   const unsigned long long *, uint64_t, int, uint16_t *,
                                                   unsigned long long *, unsigned long long *, cudaStream_t);
template cudaError_t launch_decode_write<uint32_t>(const DecodeTablesDev &, const DecodeString &, const uint32_t *,
                                                   const unsigned long long *, uint64_t, int, uint32_t *,
                                                   unsigned long long *, unsigned long long *, cudaStream_t);

uint64_t decode_ranges(uint64_t nunits) { return (nunits + 31) / 32; }
uint64_t constant_ranges(uint64_t n) { return (n + RANGE - 1) / RANGE; }
cudaError_t launch_constant_ranges(uint64_t n, bool zero, unsigned long long *zstart, unsigned long long *zcount,
                                   cudaStream_t st) {
    k_constant_ranges<<<grid_for(constant_ranges(n), 256), 256, 0, st>>>(n, zero, zstart, zcount);
    return cudaGetLastError();
}

template <typename C>
cudaError_t launch_zero_positions(const C *codes, uint64_t n, uint64_t nranges, const unsigned long long *zstart,
                                  const unsigned long long *zcount, const unsigned long long *zoff, uint64_t cap,
                                  uint64_t *zpos, cudaStream_t st) {
    k_zero_positions<C><<<grid_for(nranges, 8), 256, 0, st>>>(codes, n, nranges, zstart, zcount, zoff, cap, zpos);
    return cudaGetLastError();
}
template cudaError_t launch_zero_positions<uint16_t>(const uint16_t *, uint64_t, uint64_t, const unsigned long long *,
                                                     const unsigned long long *, const unsigned long long *, uint64_t,
                                                     uint64_t *, cudaStream_t);
template cudaError_t launch_zero_positions<uint32_t>(const uint32_t *, uint64_t, uint64_t, const unsigned long long *,
                                                     const unsigned long long *, const unsigned long long *, uint64_t,
                                                     uint64_t *, cudaStream_t);

// one block: exclusive scan of n totals in place, their sum in v[n]
cudaError_t launch_scan_small(unsigned long long *v, uint64_t n, cudaStream_t st) {
    k_scan_top<<<1, 1024, 0, st>>>(v, n);
    return cudaGetLastError();
}

// one launch in the place of four copies of a word each
__global__ void k_decode_outcome(const int *flags, const unsigned long long *total, uint64_t need,
                                 const unsigned long long *zeros, uint64_t expect, int *hold, DecodeStatus *host) {
    DecodeStatus s;
    s.changed = flags ? flags[0] : 0;
    s.damaged = flags ? flags[1] : 0;
    s.total = total ? *total : need;
    s.zeros = zeros ? *zeros : 0;
    if (hold) *hold = s.changed || s.damaged || s.total < need || s.zeros != expect;
    *host = s;
}
cudaError_t launch_decode_outcome(const int *flags, const unsigned long long *total, uint64_t need,
                                  const unsigned long long *zeros, uint64_t expect, int *hold, DecodeStatus *host,
                                  cudaStream_t st) {
    k_decode_outcome<<<1, 1, 0, st>>>(flags, total, need, zeros, expect, hold, host);
    return cudaGetLastError();
}

cudaError_t launch_fill_u16(uint16_t *out, uint64_t n, uint16_t v, cudaStream_t st) {
    unsigned g = grid_for(n, 1024);
    if (g > 4096) g = 4096;
    if (g == 0) g = 1;
    k_fill_u16<uint16_t><<<g, 1024, 0, st>>>(out, n, v);
    return cudaGetLastError();
}
cudaError_t launch_fill_u16(uint32_t *out, uint64_t n, uint32_t v, cudaStream_t st) {
    unsigned g = grid_for(n, 1024);
    if (g > 4096) g = 4096;
    if (g == 0) g = 1;
    k_fill_u16<uint32_t><<<g, 1024, 0, st>>>(out, n, v);
    return cudaGetLastError();
}

}  // namespace faz
