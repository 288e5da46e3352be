// huffman_host.cpp - Huffman codebook construction and tree (de)serialisation.
//
// The GPU histogram gives every symbol's count and first stream position; the
// tree is then built on the host exactly as HuffmanEncoder::init does
// (include/QoZ/encoder/HuffmanEncoder.hpp:529-566): leaves enter a binary heap
// in the iteration order of the ska::unordered_map the reference fills with
// frequency[s[i]]++, pairs are merged until one root remains, and codes are
// read off the tree (left 0, right 1, build_code 493-521).  The serialised
// tree follows save/pad_tree (119-137, 569-633).
#include <algorithm>
#include <cstring>
#include <numeric>

#include "internal.h"

namespace faz {

namespace {

// Iteration order of ska::unordered_map<int, size_t> after inserting `keys`
// in order (include/QoZ/utils/ska_hash/unordered_map.hpp): separate chaining
// over a power-of-two bucket array (at least 4 buckets), bucket index = the
// top log2(B) bits of key * 0x9E3779B97F4A7C15 (fibonacci_hash_policy), new
// entries at the head of their chain, the array doubling when an insert
// would exceed one entry per bucket (entries move bucket by bucket, each
// chain front to back, to the head of their new chain), iteration from the
// last bucket down to bucket 0, each chain front to back.
std::vector<int> map_iteration_order(const std::vector<int> &keys) {
    const size_t n = keys.size();
    std::vector<int> next(n, -1);
    std::vector<int> head;
    size_t nb = 0;
    int shift = 63;
    auto bucket = [](int key, int sh) -> size_t {
        return (size_t)(((uint64_t)(int64_t)key * 0x9E3779B97F4A7C15ull) >> sh);
    };
    for (size_t k = 0; k < n; k++) {
        if (nb == 0 || k + 1 > nb) {
            size_t nnb = nb == 0 ? 4 : nb * 2;
            int lg = 0;
            while (((size_t)1 << lg) < nnb) lg++;
            int nsh = 64 - lg;
            std::vector<int> nh(nnb, -1);
            for (size_t b = 0; b < nb; b++) {
                for (int e = head[b]; e >= 0;) {
                    int nx = next[e];
                    size_t j = bucket(keys[e], nsh);
                    next[e] = nh[j];
                    nh[j] = e;
                    e = nx;
                }
            }
            head.swap(nh);
            nb = nnb;
            shift = nsh;
        }
        size_t j = bucket(keys[k], shift);
        next[k] = head[j];
        head[j] = (int)k;
    }
    std::vector<int> order;
    order.reserve(n);
    for (size_t b = nb; b-- > 0;)
        for (int e = head[b]; e >= 0; e = next[e]) order.push_back(e);
    return order;
}

// Binary min-heap on freq with the reference's sift rules (qinsert stops on
// parent <= new, qremove descends to the smaller child, the left one of equals,
// while parent > child), which decide between equal counts and so shape the tree.
// An entry is one word, freq << kNodeBits | node: siblings share a cache line, and
// a.freq < b.freq is a < (b with its node bits cleared).  The whole codebook of a
// 65,000-symbol alphabet (float64 at a tight bound) takes 6.9 ms on a Grace core,
// 5 ms of it here: 13.1 ms with 16-byte entries, an exit test on each level and a
// comparison sort of the first positions.
struct Heap {
    static constexpr int kNodeBits = 19;  // below 2^19 nodes (2^18 + 1 symbols), counts below 2^45
    static constexpr uint64_t kNode = ((uint64_t)1 << kNodeBits) - 1;
    std::vector<uint64_t> q;  // 1-based; room for a sibling past the last entry
    size_t n = 0;
    explicit Heap(size_t cap) : q(cap + 3) {}
    void insert(int nd, uint64_t fn) {
        const uint64_t x = fn << kNodeBits | (uint64_t)nd;
        size_t i = ++n, j;
        while ((j = i >> 1)) {
            if (!((fn << kNodeBits) < (q[j] & ~kNode))) break;
            q[i] = q[j];
            i = j;
        }
        q[i] = x;
    }
    int remove(uint64_t &freq) {
        const uint64_t top = q[1];
        freq = top >> kNodeBits;
        const uint64_t x = q[n--];
        if (n > 0) {
            // The last entry x sinks from the top along the path of smaller
            // children, past those smaller than itself.  Their counts do not
            // decrease down the path, so the whole path moves up first (a fixed
            // number of steps, the choice of child without a branch) and x climbs
            // back to its place, which is near the bottom.
            size_t i = 1, l;
            while ((l = i << 1) < n) {
                l += (size_t)(q[l + 1] < (q[l] & ~kNode));
                q[i] = q[l];
                i = l;
            }
            if (l == n) {
                q[i] = q[l];
                i = l;
            }
            const uint64_t xf = x & ~kNode;
            while ((l = i >> 1) && !(q[l] < xf)) {
                q[i] = q[l];
                i = l;
            }
            q[i] = x;
        }
        return (int)(top & kNode);
    }
};

// Indices 0 .. v.size() - 1 in ascending order of v (distinct values): a radix
// sort by 11-bit digits, or std::sort where that is shorter.
std::vector<int> order_of(const std::vector<uint64_t> &v) {
    const size_t n = v.size();
    struct E {
        uint64_t key;
        int index;
    };
    std::vector<E> a(n);
    uint64_t all = 0;
    for (size_t i = 0; i < n; i++) {
        a[i] = {v[i], (int)i};
        all |= v[i];
    }
    if (n < 512) {
        std::sort(a.begin(), a.end(), [](const E &x, const E &y) { return x.key < y.key; });
    } else {
        std::vector<E> b(n);
        for (int sh = 0; sh < 64 && (all >> sh) != 0; sh += 11) {
            uint32_t at[2048] = {0};
            for (const E &e : a) at[(e.key >> sh) & 2047]++;
            uint32_t sum = 0;
            for (uint32_t &c : at) {
                const uint32_t k = c;
                c = sum;
                sum += k;
            }
            for (const E &e : a) b[at[(e.key >> sh) & 2047]++] = e;
            a.swap(b);
        }
    }
    std::vector<int> o(n);
    for (size_t i = 0; i < n; i++) o[i] = a[i].index;
    return o;
}

template <typename W>
void put_le(std::vector<uint8_t> &o, W v) {
    uint8_t b[sizeof(W)];
    std::memcpy(b, &v, sizeof(W));
    o.insert(o.end(), b, b + sizeof(W));
}

}  // namespace

int build_codebook(const std::vector<int> &syms, const std::vector<uint64_t> &counts,
                   const std::vector<uint64_t> &first, Codebook &cb, std::string &err) {
    const size_t d = syms.size();
    if (d == 0) {
        err = "Huffman input is empty";
        return FAZ_ERR_ARG;
    }
    // distinct symbols in order of first occurrence = map insertion order
    // (first positions are distinct stream positions)
    if (d >= (size_t)1 << (Heap::kNodeBits - 1)) {
        err = "too many Huffman symbols";
        return FAZ_ERR_UNSUPPORTED;
    }
    const std::vector<int> byfirst = order_of(first);
    std::vector<int> keys(d);
    for (size_t i = 0; i < d; i++) keys[i] = syms[byfirst[i]];
    std::vector<int> ord = map_iteration_order(keys);
    int mn = *std::min_element(syms.begin(), syms.end());
    int mx = *std::max_element(syms.begin(), syms.end());
    cb.offset = mn;
    cb.stateNum = mx - mn + 2;
    // nodes: leaves 0 .. d-1 in heap insertion order, then the merged nodes;
    // a merged node's children always have smaller indices
    const size_t nn = 2 * d - 1;
    std::vector<int> left(nn, -1), right(nn, -1), state(d);
    Heap h(d);
    for (size_t k = 0; k < d; k++) {
        const int si = byfirst[ord[k]];
        state[k] = syms[si] - mn;
        h.insert((int)k, counts[si]);
    }
    size_t next = d;
    while (h.n > 1) {
        // the reference evaluates new_node(0, 0, qremove(), qremove()) right
        // to left: the first node removed is the right child
        uint64_t fa, fb;
        const int b = h.remove(fb);
        const int a = h.remove(fa);
        left[next] = a;
        right[next] = b;
        h.insert((int)next, fa + fb);
        next++;
    }
    const int root = (int)nn - 1;  // the last node merged
    // code lengths and bits (left 0, right 1), parents before children
    std::vector<uint8_t> len(nn, 0);
    std::vector<uint64_t> bits(nn, 0);
    for (size_t i = nn; i-- > d;) {
        if (len[i] >= 64) {
            err = "Huffman code longer than 64 bits";
            return FAZ_ERR_UNSUPPORTED;
        }
        len[left[i]] = len[right[i]] = (uint8_t)(len[i] + 1);
        bits[left[i]] = bits[i] << 1;
        bits[right[i]] = (bits[i] << 1) | 1;
    }
    cb.code.assign(cb.stateNum, 0);
    cb.len.assign(cb.stateNum, 0);
    cb.maxlen = 0;
    for (size_t k = 0; k < d; k++) {
        const int l = len[k];
        cb.code[state[k]] = l == 0 ? 0 : bits[k] << (64 - l);
        cb.len[state[k]] = (uint8_t)l;
        cb.maxlen = std::max(cb.maxlen, l);
    }
    // serialise (pad_tree): preorder numbering - a node, its left subtree,
    // its right subtree - from subtree sizes, then the L/R/C/t arrays
    const uint32_t nc = (uint32_t)nn;
    cb.nodeCount = (int)nc;
    std::vector<uint32_t> size(nn, 1), num(nn, 0);
    for (size_t i = d; i < nn; i++) size[i] = 1 + size[left[i]] + size[right[i]];
    num[root] = 0;
    std::vector<uint32_t> L(nc, 0), R(nc, 0);
    std::vector<int32_t> C(nc, 0);
    std::vector<uint8_t> t(nc, 0);
    for (size_t i = nn; i-- > 0;) {
        const uint32_t me = num[i];
        if (i < d) {
            C[me] = state[i];
            t[me] = 1;
            continue;
        }
        num[left[i]] = me + 1;
        num[right[i]] = me + 1 + size[left[i]];
        L[me] = num[left[i]];
        R[me] = num[right[i]];
    }
    const int w = nc <= 256 ? 1 : (nc <= 65536 ? 2 : 4);
    std::vector<uint8_t> &o = cb.tree;
    o.assign(1 + 2 * (size_t)nc * w + (size_t)nc * 4 + nc, 0);
    uint8_t *p = o.data();
    *p++ = 0;  // endian byte: little endian
    for (int pass = 0; pass < 2; pass++) {
        const std::vector<uint32_t> &A = pass ? R : L;
        for (uint32_t i = 0; i < nc; i++, p += w) {
            if (w == 1) {
                *p = (uint8_t)A[i];
            } else if (w == 2) {
                const uint16_t v = (uint16_t)A[i];
                std::memcpy(p, &v, 2);
            } else {
                std::memcpy(p, &A[i], 4);
            }
        }
    }
    std::memcpy(p, C.data(), (size_t)nc * 4);
    p += (size_t)nc * 4;
    std::memcpy(p, t.data(), nc);
    return FAZ_OK;
}

// HuffmanEncoder::load (include/QoZ/encoder/HuffmanEncoder.hpp:276-296): the
// tree as the child words that the GPU decoder's tables are built from.
int parse_tree(const uint8_t *&p, const uint8_t *end, DecodeTablesHost &t, std::string &err) {
    auto need = [&](size_t k) { return (size_t)(end - p) >= k; };
    if (!need(12)) {
        err = "truncated Huffman header";
        return FAZ_ERR_FORMAT;
    }
    int32_t offset;
    std::memcpy(&offset, p, 4);
    uint32_t nc = ((uint32_t)p[4] << 24) | ((uint32_t)p[5] << 16) | ((uint32_t)p[6] << 8) | p[7];
    p += 12;  // offset, nodeCount, stateNum/2
    if (nc == 0 || nc > (1u << 24)) {
        err = "bad Huffman node count";
        return FAZ_ERR_FORMAT;
    }
    int w = nc <= 256 ? 1 : (nc <= 65536 ? 2 : 4);
    size_t bytes = 1 + 2 * (size_t)nc * w + (size_t)nc * 4 + nc;
    if (!need(bytes)) {
        err = "truncated Huffman tree";
        return FAZ_ERR_FORMAT;
    }
    const uint8_t *q = p + 1;
    t.offset = offset;
    t.nodeCount = (int)nc;
    const uint8_t *ql = q, *qr = q + (size_t)nc * w, *qs = q + 2 * (size_t)nc * w, *qt = qs + (size_t)nc * 4;
    auto sym = [&](uint32_t i) {
        int32_t x;
        std::memcpy(&x, qs + 4 * (size_t)i, 4);
        return x;
    };
    auto index = [&](const uint8_t *a, uint32_t i) -> uint32_t {
        if (w == 1) return a[i];
        if (w == 2) {
            uint16_t x;
            std::memcpy(&x, a + 2 * (size_t)i, 2);
            return x;
        }
        uint32_t x;
        std::memcpy(&x, a + 4 * (size_t)i, 4);
        return x;
    };
    p += bytes;
    // a tree of more than 256 nodes is rebuilt with an internal root
    const bool root_leaf = nc <= 256 && qt[0];
    t.constant = root_leaf;
    t.constant_state = sym(0);
    if (root_leaf) return FAZ_OK;
    // children are numbered after their parent (preorder): reject anything
    // else so that every walk ends.  Two parents of one node are taken as they
    // always were (every walk still ends), but such a tree has more prefixes than
    // its nodes bound: see decode_slots.
    t.child.assign(2 * (size_t)nc, 0);
    std::vector<uint8_t> named(nc, 0);
    for (uint32_t i = 0; i < nc; i++) {
        if (i > 0 && qt[i]) continue;
        for (int k = 0; k < 2; k++) {
            const uint32_t c = index(k ? qr : ql, i);
            if (c <= i || c >= nc) {
                err = "malformed Huffman tree";
                return FAZ_ERR_FORMAT;
            }
            if (qt[c]) {
                const int32_t s = sym(c);
                t.child[2 * (size_t)i + k] = kChildLeaf | (s < 0 ? kChildBad : 0u) | ((uint32_t)s & 0xffffffu);
            } else {
                t.child[2 * (size_t)i + k] = c;
                t.shared |= named[c] != 0;
                named[c] = 1;
            }
        }
    }
    return FAZ_OK;
}

// A prefix without a leaf ends at an inner node.  Where every inner node has one parent,
// m such nodes of one depth are distinct and have at least m - 1 inner nodes above them;
// where one has two, every prefix may end at the same node.
size_t decode_slots(const DecodeTablesHost &t) {
    const size_t all = (size_t)1 << kLutBits;
    return t.shared ? all : std::min(all, (size_t)t.nodeCount / 2 + 1);
}

uint32_t leaf_depth(const DecodeTablesHost &t, int32_t state) {
    // children are numbered after their parents: one pass carries the depths down
    const size_t nc = t.child.size() / 2;
    std::vector<uint8_t> depth(nc, 0);
    for (size_t i = 0; i < nc; i++) {
        for (int k = 0; k < 2; k++) {
            const uint32_t c = t.child[2 * i + k];
            const uint8_t d = (uint8_t)std::min(255, depth[i] + 1);
            if (!(c & kChildLeaf)) {
                if (c < nc) depth[c] = d;
            } else if (!(c & kChildBad) && (int32_t)(c & 0xffffffu) == state) {
                return d <= 64 ? d : 0;
            }
        }
    }
    return 0;
}

}  // namespace faz
