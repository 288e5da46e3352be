// CPU check of the Huffman tree parser (faz_gb300/csrc/huffman_host.cpp): the
// second-table slots that decode_slots allows for against a walk of every prefix,
// for trees whose nodes have one parent and for damaged ones whose nodes have two.
// Usage: huffman_tree_check; prints each case, exit 1 on any mismatch.
#include <cstdio>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "../faz_gb300/csrc/internal.h"

using namespace faz;

struct Nodes {
    std::vector<uint32_t> left, right;
    std::vector<int32_t> sym;
    std::vector<uint8_t> leaf;
    uint32_t add(uint32_t l, uint32_t r, bool is_leaf, int32_t s) {
        left.push_back(l);
        right.push_back(r);
        sym.push_back(s);
        leaf.push_back(is_leaf);
        return (uint32_t)left.size() - 1;
    }
};

// HuffmanEncoder::save: offset, node and state counts, then the arrays
static std::vector<uint8_t> serialise(const Nodes &t) {
    const uint32_t nc = (uint32_t)t.left.size();
    const int w = nc <= 256 ? 1 : (nc <= 65536 ? 2 : 4);
    std::vector<uint8_t> o(4, 0);
    for (int k = 0; k < 2; k++)
        for (int s = 24; s >= 0; s -= 8) o.push_back((uint8_t)(nc >> s));
    o.push_back(0);
    auto put = [&](const void *p, size_t n) { o.insert(o.end(), (const uint8_t *)p, (const uint8_t *)p + n); };
    for (uint32_t x : t.left) put(&x, w);
    for (uint32_t x : t.right) put(&x, w);
    for (int32_t x : t.sym) put(&x, 4);
    put(t.leaf.data(), nc);
    return o;
}

// random tree in preorder
static uint32_t grow(Nodes &t, int leaves, std::mt19937 &rng) {
    const uint32_t i = t.add(0, 0, leaves == 1, (int32_t)(rng() & 0xffff));
    if (leaves == 1) return i;
    const int a = rng() % 4 ? 1 + (int)(rng() % (leaves - 1)) : 1;
    const uint32_t l = grow(t, a, rng), r = grow(t, leaves - a, rng);
    t.left[i] = l;
    t.right[i] = r;
    return i;
}

static int failures = 0;

static void check(const char *name, const Nodes &t, bool shared) {
    const std::vector<uint8_t> s = serialise(t);
    const uint8_t *p = s.data();
    DecodeTablesHost h;
    std::string err;
    const int rc = parse_tree(p, s.data() + s.size(), h, err);
    if (rc != FAZ_OK || p != s.data() + s.size()) {
        std::printf("%s: refused (%d %s)\n", name, rc, err.c_str());
        failures++;
        return;
    }
    size_t prefixes = 0;
    for (uint32_t v = 0; v < (1u << kLutBits); v++) {
        uint32_t node = 0;
        int b = 0;
        for (; b < kLutBits; b++) {
            const uint32_t c = h.child[2 * (size_t)node + ((v >> (kLutBits - 1 - b)) & 1)];
            if (c & kChildLeaf) break;
            node = c;
        }
        prefixes += b == kLutBits;
    }
    const bool ok = prefixes <= decode_slots(h) && decode_slots(h) <= (size_t)1 << kLutBits && h.shared == shared;
    std::printf("%s: %zu nodes, %zu prefixes, %zu slots%s\n", name, t.left.size(), prefixes, decode_slots(h),
                ok ? "" : " MISMATCH");
    failures += !ok;
}

int main() {
    std::mt19937 rng(7);
    // trees: few symbols, many, and one long chain of codewords
    for (int leaves : {2, 3, 40, 129, 5000, 40000}) {
        Nodes t;
        grow(t, leaves, rng);
        check("tree", t, false);
    }
    {
        Nodes t;
        for (uint32_t i = 0; i < 60; i++) t.add(2 * i + 1, 2 * i + 2, false, 0), t.add(0, 0, true, (int32_t)i);
        t.add(0, 0, true, 60);
        check("chain", t, false);
    }
    // a full tree whose deepest inner nodes all name one leaf: as many inner nodes
    // as a tree can have
    {
        Nodes t;
        const uint32_t inner = (1u << (kLutBits + 1)) - 1;
        for (uint32_t i = 0; i < inner; i++)
            t.add(std::min(2 * i + 1, inner), std::min(2 * i + 2, inner), false, 0);
        t.add(0, 0, true, 5);
        check("one leaf", t, false);
    }
    // node i names i + 1 twice: every prefix ends at node kLutBits
    for (int inner : {kLutBits, kLutBits + 1, kLutBits + 20}) {
        Nodes t;
        for (int i = 0; i < inner; i++) t.add(i + 1, i + 1, false, 0);
        t.add(0, 0, true, 3);
        check("repeated child", t, true);
    }
    // the same under a tree of 2-byte indices
    {
        Nodes t;
        grow(t, 400, rng);
        const uint32_t base = (uint32_t)t.left.size();
        for (int i = 0; i < 30; i++) t.add(base + i + 1, base + i + 1, false, 0);
        t.add(0, 0, true, 3);
        t.left[0] = base;
        check("repeated child below a tree", t, true);
    }
    // a tree in which one index repeats another's
    for (int k = 0; k < 20; k++) {
        Nodes t;
        grow(t, 300, rng);
        uint32_t i, j;
        do {
            i = rng() % t.left.size();
            j = rng() % t.left.size();
        } while (t.leaf[i] || t.leaf[j] || t.leaf[t.left[j]] || t.left[j] <= i || t.left[i] == t.left[j]);
        t.left[i] = t.left[j];
        check("repeated index", t, true);
    }
    return failures != 0;
}
