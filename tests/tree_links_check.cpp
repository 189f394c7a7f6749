// Host check of the child table's links (tree_links.cuh), run by
// test_tree_links.py: tree_links_check <bodies> <systems> <key bits> <seed>.
//
// Builds the radix tree over random sorted keys (by splitting ranges), the
// masks and prefix sums that the build kernels make, and links every record.
// Whole tree: each row holds exactly its cell's children. Prefix sums that lost
// a tile's prefix, and keys out of order: a row names only records behind its
// own, so that a walk down the rows ends.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "tree_links.cuh"

using namespace nbody;

namespace {

struct Build {
    std::vector<uint64_t> k;
    std::vector<int> seg, lo, hi, delta, iparent, lparent, top;
    std::vector<uint32_t> mask, P;
    int base = 0;
    BinaryTree t{};
    int64_t n = 0;

    int delta_of(int i, int j) const {
        if (base && seg[i] != seg[j]) return __builtin_clz(static_cast<unsigned>(seg[i] ^ seg[j]));
        if (k[i] != k[j]) return base + __builtin_clzll(k[i] ^ k[j]) - 1;
        return base + 63 + (i == j ? 32 : __builtin_clz(static_cast<unsigned>(i ^ j)));
    }
    // Node `id` covers [a, b]; its children carry the ids of the two places beside the split.
    void split(int id, int a, int b, int parent, int parent_level) {
        lo[id] = a;
        hi[id] = b;
        delta[id] = delta_of(a, b);
        iparent[id] = parent;
        const int L = level_c(delta[id], base);
        top[id] = parent < 0 ? L > -1 : L > parent_level;
        if (top[id]) mask[a] |= 1u << L;
        int g = a;
        while (g + 1 < b && delta_of(a, g + 1) > delta[id]) ++g;
        if (g == a) lparent[a] = id; else split(g, a, g, id, L);
        if (g + 1 == b) lparent[b] = id; else split(g + 1, g + 1, b, id, L);
    }
    bool lone(int i) const {
        const auto same = [&](int a, int b) { return k[a] == k[b] && seg[a] == seg[b]; };
        return !((i > 0 && same(i, i - 1)) || (i + 1 < n && same(i, i + 1)));
    }
    void scan(int lost_from) {  // lost_from >= 0: the tile that begins there takes no prefix before it
        uint32_t run = 0;
        for (int i = 0; i < n; ++i) {
            if (i == lost_from) run = 0;
            P[i] = run;
            run += bits_set(mask[i]) + (lone(i) ? 1 : 0);
        }
        P[n] = run;
    }
    // Links every record; returns the number refused. rows: 8 per record; parents as returned.
    int link(std::vector<int> &rows, std::vector<std::pair<int, int>> &links) {
        rows.assign(static_cast<size_t>(16 * n), -1);
        links.clear();
        int refused = 0;
        const auto one = [&](int p, uint64_t key, int idx) {
            const int par = link_child(t, mask.data(), P.data(), p, base, key, idx, rows.data());
            refused += par == kMisplaced;
            if (par >= 0) links.emplace_back(par, idx);
        };
        for (int i = 0; i < n; ++i) {
            if (i < n - 1 && top[i] && i > 0) one(iparent[i], k[lo[i]], record_of(t, mask.data(), P.data(), i, base));
            if (lone(i)) one(lparent[i], k[i], static_cast<int>(P[i]) + bits_set(mask[i]));
        }
        return refused;
    }
};

int fail(const char *what) {
    std::printf("FAILED: %s\n", what);
    return 1;
}

}  // namespace

int main(int argc, char **argv) {
    if (argc != 5) return fail("arguments");
    Build b;
    b.n = std::atoll(argv[1]);
    const int systems = std::atoi(argv[2]), bits = std::atoi(argv[3]);
    std::mt19937_64 rng(std::atoll(argv[4]));
    const int n = static_cast<int>(b.n);
    b.base = systems > 1 ? 32 : 0;
    std::vector<std::pair<int, uint64_t>> bodies(n);
    for (int i = 0; i < n; ++i) bodies[i] = {static_cast<int>(rng() % systems), (rng() >> (64 - bits)) << (63 - bits)};
    std::sort(bodies.begin(), bodies.end());
    for (auto &[s, key] : bodies) b.seg.push_back(s), b.k.push_back(key);
    for (auto *v : {&b.lo, &b.hi, &b.delta, &b.iparent, &b.lparent, &b.top}) v->assign(n, 0);
    b.mask.assign(n, 0);
    b.P.assign(n + 1, 0);
    b.split(0, 0, n - 1, -1, -1);
    b.t.lo = b.lo.data(), b.t.hi = b.hi.data(), b.t.delta = b.delta.data();
    b.t.iparent = b.iparent.data(), b.t.lparent = b.lparent.data(), b.t.top = b.top.data();

    for (int i = 0; i + 1 < n; ++i)
        if (out_of_order(b.k.data(), b.base ? b.seg.data() : nullptr, i)) return fail("sorted keys taken for unsorted");

    std::vector<int> rows;
    std::vector<std::pair<int, int>> links;
    b.scan(-1);
    if (b.link(rows, links) != 0) return fail("a whole tree's link was refused");
    // Pre-order: a record's children are the records linked to it, each once, by rising digit.
    std::vector<int> seen(static_cast<size_t>(b.P[n]), 0);
    for (auto &[par, idx] : links) ++seen[idx];
    int roots = 0;
    for (int s : seen) {
        if (s > 1) return fail("a record in two rows");
        roots += s == 0;
    }
    std::vector<int> present(systems, 0);
    for (int s : b.seg) present[s] = 1;
    if (roots != std::count(present.begin(), present.end(), 1)) return fail("records without a parent that are no roots");
    size_t in_rows = 0;
    for (size_t r = 0; 8 * r < rows.size(); ++r) {
        int before = static_cast<int>(r);
        for (int d = 0; d < 8; ++d)
            if (rows[8 * r + d] >= 0) {
                if (rows[8 * r + d] <= before) return fail("a row out of pre-order");
                before = rows[8 * r + d];
                ++in_rows;
            }
    }
    if (in_rows != links.size()) return fail("two children in one place");

    // A tile's prefix lost, at several places; then keys out of order under whole sums.
    int refused = 0;
    const auto rows_go_forward = [&] {
        for (size_t r = 0; 8 * r < rows.size(); ++r)
            for (int d = 0; d < 8; ++d)
                if (rows[8 * r + d] >= 0 && rows[8 * r + d] <= static_cast<int>(r)) return false;
        return true;
    };
    for (int q = 1; q < 8; ++q) {
        b.scan(static_cast<int>(static_cast<int64_t>(n) * q / 8));
        refused += b.link(rows, links);
        if (!rows_go_forward()) return fail("a row of overlapping records names an earlier one");
    }
    if (n >= 1000 && refused == 0) return fail("overlapping records went unnoticed");
    std::swap(b.k[n / 3], b.k[2 * n / 3]);
    bool noticed = b.k[n / 3] == b.k[2 * n / 3] || b.seg[n / 3] != b.seg[2 * n / 3];
    for (int i = 0; i + 1 < n; ++i) noticed = noticed || out_of_order(b.k.data(), b.base ? b.seg.data() : nullptr, i);
    if (!noticed) return fail("keys out of order went unnoticed");
    std::printf("ok: %zu links, %d refused\n", links.size(), refused);
    return 0;
}
