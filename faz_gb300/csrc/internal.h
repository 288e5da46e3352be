// internal.h - host-side declarations shared by the library's translation units.
#pragma once
#include <cuda_runtime.h>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include "../../include/faz_gb300.h"
#include "common.cuh"

namespace faz {

// Let a kernel take up to the device's opt-in shared memory per block, once
// per (device, kernel).  Setting the limit to each launch's own need instead
// races: host threads launching the same kernel concurrently (the tuner's
// trials) can lower it between another thread's set and launch.
// largest l with 2^l <= d (d >= 1)
inline int floor_log2(uint64_t d) { return 63 - __builtin_clzll(d); }
// smallest l with 2^l >= d (ceil(log2(d)) for d >= 1)
inline int ceil_log2(uint64_t d) {
    int l = 0;
    while (((uint64_t)1 << l) < d) l++;
    return l;
}

// Level error bound (SZInterpolationCompressor.hpp:386-406, eb_ratio 0.5)
inline double level_eb(double eb, double alpha, double beta, int level) {
    if (alpha < 0) return level >= 3 ? eb * 0.5 : eb;
    if (alpha >= 1) {
        double cr = std::pow(alpha, level - 1);
        if (cr > beta) cr = beta;
        return eb / cr;
    }
    double cr = 1 - (level - 1) * alpha;
    if (cr < beta) cr = beta;
    return eb * cr;
}

inline cudaError_t allow_dynamic_smem(const void *func) {
    static std::mutex mu;
    static std::set<std::pair<int, const void *>> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> g(mu);
    if (done.count({dev, func})) return cudaSuccess;
    int optin = 0;
    e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, func);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
    if (e == cudaSuccess) done.insert({dev, func});
    return e;
}

// ---------------------------------------------------------------- kernels
template <typename T>
cudaError_t launch_minmax(const T *X, uint64_t n, T *pmin, T *pmax, int nblocks, cudaStream_t st);
int sm_count();  // SMs of the device current at the first call
template <typename T>
size_t level_smem_bytes(const LevelArgs &a);
// The levels of an interpolation plan, coarsest first (a batch of the kernels
// below takes up to kMaxPlanLevels).
constexpr int kMaxPlanLevels = 32;
struct LevelTable {
    LevelArgs a[kMaxPlanLevels];
    uint64_t first[kMaxPlanLevels];  // its first entry in the block-offset table
    uint64_t pos[kMaxPlanLevels];    // stream position of its first code
    int n;
};
// stream position of every block's first code into `off`
cudaError_t launch_block_offsets(const LevelTable &t, uint64_t nblocks, uint64_t *off, cudaStream_t st);
// How many of a plan's first levels are small enough for launch_small_levels, and
// the launch: the first point (unless anchors come instead) and those levels, in
// one CTA.
int small_levels(const LevelTable &t);
template <typename T>
cudaError_t launch_small_levels(const LevelTable &t, int n, bool decomp, bool first_point, double eb, const T *X, T *W,
                                uint16_t *codes, T *scratch, const uint64_t *zpos, uint64_t nz, const T *unpred,
                                cudaStream_t st);
// One interpolation level; *nlaunch grows by the kernel launches it made.
template <typename T>
cudaError_t launch_level(const LevelArgs &a, int64_t nblocks, bool decomp, const T *X, T *W, uint16_t *codes,
                         T *scratch, const uint64_t *zpos, uint64_t nz, const T *unpred, cudaStream_t st,
                         int *nlaunch);
// The finest level of a 3-D float field, plane by plane with TMA-staged
// planes (finest.cu): whether it can take a level, whether it is faster there than
// the block kernel, and its launch.
bool finest_possible(const LevelArgs &a, bool decomp, const void *X, const void *W);
bool finest_faster(const LevelArgs &a, bool decomp);
cudaError_t launch_finest(const LevelArgs &a, int64_t nblocks, bool decomp, const float *X, float *W,
                          uint16_t *codes, float *scratch, const uint64_t *zpos, uint64_t nz, const float *unpred,
                          cudaStream_t st);
template <typename T>
cudaError_t launch_first_point(bool decomp, const T *X, T *W, uint16_t *codes, T *scratch, double eb, int radius,
                               int trim, const uint64_t *zpos, uint64_t nz, const T *unpred, cudaStream_t st,
                               const int *hold = nullptr);
template <typename T>
cudaError_t launch_anchors(bool decomp, const T *X, T *W, uint16_t *codes, T *scratch, const T *unpred,
                           const int64_t *na, const int64_t *step, const int64_t *offs, cudaStream_t st,
                           const int *hold = nullptr);

// Batched compression: every field's first point / anchors and levels in one
// persistent launch from a device work queue (interp.cu).
struct BatchField {
    const void *X;
    void *W;
    uint16_t *codes;
    void *scratch;
    double eb, recip;  // base error bound (first point)
    int radius, trim;
    int anchor;        // 1: anchor grid (na, step, offs), 0: first point
    int64_t na[3], step[3], offs[3];
};
struct BatchGroup {
    int field;
    int kind;        // 0 first point, 1 anchors, 2 level
    int args;        // level: index into the LevelArgs table
    int dep;         // group whose items must all be done first (-1: none)
    int64_t nitems;  // work items (blocks; anchor chunks of `threads` anchors; 1)
    int64_t item0;   // first ticket of the group
};
template <typename T>
cudaError_t launch_interp_batch(const BatchGroup *groups, int ngroups, const BatchField *fields, const LevelArgs *largs,
                                uint64_t total, unsigned long long *counter, unsigned *done, int *err, bool wide,
                                int grid, int threads, size_t smem, cudaStream_t st);

template <typename T>
cudaError_t launch_minmax_batch(const T *const *X, const uint64_t *n, int nfields, T *pmin, T *pmax, int nblocks,
                                cudaStream_t st);
template <typename T, bool WIDE>
int batch_occupancy(int threads, size_t smem);

uint64_t hist_subchunks(uint64_t n);
// the symbols of non-zero count: list[3k..3k+2] = symbol, count, first
// position, in no particular order; *nlist (zeroed by the caller) their number
cudaError_t launch_hist_compact(const unsigned long long *hist, const unsigned long long *first, int nsym,
                                unsigned long long *list, unsigned int *nlist, cudaStream_t st);
// Huffman stage kernels; the uint32_t overloads serve quantisers of more than
// 65536 bins.  hist[nsym], first[nsym] (complemented positions) and *nzero zeroed
// by the caller; zcount: hist_subchunks(n) zero counts.
cudaError_t launch_histogram(const uint16_t *codes, uint64_t n, int center, unsigned long long *hist,
                             unsigned long long *first, unsigned long long *zcount, unsigned long long *nzero,
                             cudaStream_t st);
cudaError_t launch_histogram(const uint32_t *codes, uint64_t n, int center, unsigned long long *hist,
                             unsigned long long *first, unsigned long long *zcount, unsigned long long *nzero,
                             cudaStream_t st);
cudaError_t launch_count_zeros(const uint16_t *codes, uint64_t n, unsigned long long *zcount, cudaStream_t st);
template <typename T, typename C>
cudaError_t launch_compact_zeros(const C *codes, uint64_t n, const unsigned long long *zcount,
                                 const unsigned long long *zoff, const T *scratch, T *vals, cudaStream_t st);
uint64_t scan_temp_words(uint64_t n);
cudaError_t launch_scan_u64(const unsigned long long *in, unsigned long long *out, uint64_t n,
                            unsigned long long *temp, cudaStream_t st);
uint64_t encode_chunks(uint64_t n);
// Bit counts, offsets and packing of chunks [chunk0, chunk1) of n codes, after the
// chunks before them: code tables, bits and offsets per chunk, the output.  Three
// launches.  host_end (pinned, or null) receives the bits before chunk1.
struct EncodeArgs {
    int offset, maxlen;
    const unsigned long long *code64, *packed;
    const uint8_t *len;
    unsigned long long *chunkbits, *chunkoff;
    uint32_t *out;
};
cudaError_t launch_encode_pack(const EncodeArgs &a, const uint16_t *codes, uint64_t n, uint64_t chunk0,
                               uint64_t chunk1, unsigned long long *host_end, cudaStream_t st);
cudaError_t launch_encode_pack(const EncodeArgs &a, const uint32_t *codes, uint64_t n, uint64_t chunk0,
                               uint64_t chunk1, unsigned long long *host_end, cudaStream_t st);

// Huffman decoder (huffman.cu): the tree as child words (leaf flag | state, or
// node index), and the tables launch_decode_tables builds from it.
struct DecodeTablesDev {
    const uint32_t *child;     // 2 per node
    uint16_t *lutA;            // 2^kLutBits each
    uint2 *lutB;
    uint32_t *lut2;            // decode_lut2_entries(decode_slots) each
    uint8_t *len2;
};
struct DecodeString {
    const uint32_t *w32;
    uint64_t nwords, nbits, nunits;
    int unit_words;
    uint64_t run_bits;  // leading bits expected to repeat one codeword of run_len bits (0: none)
    uint32_t run_len;
};
int decode_unit_words(uint64_t nbits);  // words per unit of a string of nbits
uint64_t decode_cta_units();            // units per CTA of the synchronising pass
size_t decode_lut2_entries(size_t slots);
template <typename C>
cudaError_t launch_decode_tables(const DecodeTablesDev &t, int offset, uint32_t *slot_node, unsigned *nslots,
                                 size_t lut2_entries, cudaStream_t st);
// synchronising pass over CTAs [cta0, cta1); flags[0] = a CTA end moved (set by
// the link pass), flags[1] = damaged
cudaError_t launch_decode_sync(const DecodeTablesDev &t, const DecodeString &d, uint64_t cta0, uint64_t cta1,
                               uint32_t *info, uint32_t *cend, unsigned long long *ctot, int *flags, cudaStream_t st);
cudaError_t launch_decode_link(const DecodeTablesDev &t, const DecodeString &d, const uint32_t *cend_in,
                               uint32_t *cend_out, uint32_t *info, unsigned long long *ctot, int *flags,
                               cudaStream_t st);
template <typename C>
cudaError_t launch_decode_write(const DecodeTablesDev &t, const DecodeString &d, const uint32_t *info,
                                const unsigned long long *coff, uint64_t nout, int offset, C *out,
                                unsigned long long *zc, unsigned long long *zstart, cudaStream_t st);
// the zeros of the decoded codes: first code (zstart) and zero count (zcount) of
// each of decode_ranges(nunits) ranges, zoff the counts' exclusive scan; the
// first cap positions, sorted
uint64_t decode_ranges(uint64_t nunits);
// the ranges of n equal codes
uint64_t constant_ranges(uint64_t n);
cudaError_t launch_constant_ranges(uint64_t n, bool zero, unsigned long long *zstart, unsigned long long *zcount,
                                   cudaStream_t st);
template <typename C>
cudaError_t launch_zero_positions(const C *codes, uint64_t n, uint64_t nranges, const unsigned long long *zstart,
                                  const unsigned long long *zcount, const unsigned long long *zoff, uint64_t cap,
                                  uint64_t *zpos, cudaStream_t st);
cudaError_t launch_scan_small(unsigned long long *v, uint64_t n, cudaStream_t st);
// The outcome of a queued decode (flags and total null: a constant string; zeros null:
// not counted) into pinned memory, to be read once the stream is synchronised.
// *hold, when given: 0 where the codes are a field's, flags clear, at least `need` of
// them and `expect` zeros.
struct DecodeStatus {
    int changed, damaged;
    unsigned long long total, zeros;
};
cudaError_t launch_decode_outcome(const int *flags, const unsigned long long *total, uint64_t need,
                                  const unsigned long long *zeros, uint64_t expect, int *hold, DecodeStatus *host,
                                  cudaStream_t st);
cudaError_t launch_fill_u16(uint16_t *out, uint64_t n, uint16_t v, cudaStream_t st);
cudaError_t launch_fill_u16(uint32_t *out, uint64_t n, uint32_t v, cudaStream_t st);

// ------------------------------------------------------------ Huffman host
struct Codebook {
    int offset = 0;          // smallest symbol
    int stateNum = 0;        // max - min + 2
    int nodeCount = 0;       // 2 * distinct - 1
    int maxlen = 0;
    std::vector<uint64_t> code;  // per state, MSB-aligned
    std::vector<uint8_t> len;    // per state
    std::vector<uint8_t> tree;   // serialised tree (HuffmanEncoder::save body after the two ints)
};
// Build the reference codebook from symbol counts and first-occurrence
// positions (symbols with count 0 are absent).
int build_codebook(const std::vector<int> &syms, const std::vector<uint64_t> &counts,
                   const std::vector<uint64_t> &first, Codebook &cb, std::string &err);

struct DecodeTablesHost {
    int offset = 0;
    int nodeCount = 0;
    bool constant = false;       // single-symbol stream
    int constant_state = 0;
    bool shared = false;         // two parents name one inner node (a damaged stream)
    std::vector<uint32_t> child; // 2 per node: node index, or leaf flag | state (kChildLeaf, kChildBad)
};
constexpr uint32_t kChildLeaf = 0x80000000u;  // a leaf; its state in the low 24 bits
constexpr uint32_t kChildBad = 0x40000000u;   // with kChildLeaf: a negative state
// Parse HuffmanEncoder::save output at p (advances p) into the decode tree.
int parse_tree(const uint8_t *&p, const uint8_t *end, DecodeTablesHost &t, std::string &err);
// length of the codeword of `state` (0: none, or longer than 64 bits)
uint32_t leaf_depth(const DecodeTablesHost &t, int32_t state);
constexpr int kLutBits = 12;
// Bound on the kLutBits-bit prefixes that hold no whole codeword: each takes a
// slot of the decoder's second tables.
size_t decode_slots(const DecodeTablesHost &t);

// -------------------------------------------------------------- stream/io
void config_save(const faz_config &c, std::vector<uint8_t> &out);
// used (optional): bytes the Config occupies
int config_load(faz_config &c, const uint8_t *p, size_t n, size_t *used = nullptr);
int config_init(faz_config *c, int N, const uint64_t *dims);
int config_load_ini(faz_config *c, const char *path, std::string &err);

struct Zstd {
    bool ok = false;
    unsigned version = 0;
    size_t (*compress)(void *, size_t, const void *, size_t, int) = nullptr;
    size_t (*decompress)(void *, size_t, const void *, size_t) = nullptr;
    unsigned (*isError)(size_t) = nullptr;
    size_t (*bound)(size_t) = nullptr;
    unsigned long long (*frameContentSize)(const void *, size_t) = nullptr;
    size_t (*findFrameCompressedSize)(const void *, size_t) = nullptr;
    unsigned long long (*getFrameContentSize)(const void *, size_t) = nullptr;
    // advanced API (one frame compressed by worker threads); null if absent
    void *(*createCCtx)() = nullptr;
    size_t (*freeCCtx)(void *) = nullptr;
    size_t (*setParameter)(void *, int, int) = nullptr;
    size_t (*compress2)(void *, void *, size_t, const void *, size_t) = nullptr;
    // ZSTD_compress on a caller's context (the same frame); null if absent
    size_t (*compressCCtx)(void *, void *, size_t, const void *, size_t, int) = nullptr;
};
// ZSTD_compress at level 3 with this thread's reused context and output
// buffer (no allocation per call); returns the frame size
size_t zstd_level3_size(const Zstd &z, const void *src, size_t n);

// How the body of a Lossless_zstd stream (one level-3 frame in the reference,
// include/QoZ/lossless/Lossless_zstd.hpp:22-32) is written:
//   Single  - ZSTD_compress on the calling thread: the reference's own call,
//             byte for byte (FAZ_ZSTD_THREADS=0);
//   Workers - one level-3 frame compressed by zstd's worker threads in jobs of
//             a size fixed by the payload length, so the bytes do not depend
//             on the worker count (the default, FAZ_ZSTD_THREADS workers);
//   Frames  - independent level-3 frames of consecutive slices, compressed and
//             decompressed in parallel (FAZ_ZSTD_MULTIFRAME=1): a format
//             extension that ZSTD_decompress still reads.
enum class ZstdMode { Single, Workers, Frames };
struct ZstdPlan {
    ZstdMode mode = ZstdMode::Single;
    int threads = 0;   // workers (Workers) or host threads (Frames)
    int nframes = 1;   // Frames only
    int job = 0;       // Workers only: job size in bytes
};
ZstdPlan zstd_plan(size_t n);
size_t zstd_body_bound(const Zstd &z, size_t n, const ZstdPlan &p);
// `parallel` false compresses on the calling thread alone (one worker for
// Workers, frames one after another for Frames): the same bytes.
size_t zstd_compress_body(const Zstd &z, uint8_t *dst, size_t cap, const uint8_t *src, size_t n, const ZstdPlan &p,
                          bool parallel = true);
// Decodes one or more concatenated frames (independent frames in parallel).
size_t zstd_decompress_frames(const Zstd &z, uint8_t *dst, size_t raw, const uint8_t *src, size_t n, int threads);
int zstd_threads();  // FAZ_ZSTD_THREADS, default the host's cores up to 16
const Zstd &zstd_lib(std::string &err);

// ------------------------------------------------------------------ errors
void set_error(const std::string &msg);

}  // namespace faz
