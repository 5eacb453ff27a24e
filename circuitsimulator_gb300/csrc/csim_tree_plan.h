// csim_tree_plan.h — host side of the tree sum (csim_tree.cuh): the chain of
// subcodes, the order of the coordinates, and the levels at which nodes are
// written out.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "csim_tree.cuh"

namespace csim {
namespace tree {

struct Plan {
    int t = 0, k = 0, r = 0;      // qubits, rows of L, its rank
    int slice = 0;                // a state's sum is that of 2^slice trees, one for each sum of the last `slice` generators
    int m[65] = {0};              // m[j]: vertices of a node of level j (m[r] = t)
    uint8_t perm[64] = {0};       // position -> coordinate; C_j lives on positions < m[j]
    uint64_t gen[64] = {0};       // gen[j]: generator of C_{j+1} over C_j, in positions
    uint64_t term[64] = {0};      // gen[j]'s part of the term index (bits of j in codeword(j) = sum of L's rows);
                                  // the index of a sum of generators is their sum's if r = k
    uint64_t x0 = 0;              // a root's X
    bool pairs = false;           // terms of |H^t>: products over vertex pairs (join_pairs) instead of codewords
    // levels of the written nodes, root (r - slice) first; the last one is the leaf kernel's
    // entry.  vert: their vertices
    std::vector<int> level, vert;
    int tj = 0, tv = 0;           // the table level, largest j with m[j] <= 8, and the table's vertices:
                                  // m[tj], or for tj = 0 the first (up to) 8 positions
};

// Chooses C_1 < C_2 < ...: each step adds the codeword with the fewest ones
// outside the support so far (all 2^d words of the remaining quotient code
// while d <= 16; beyond that the span of its first 16 rows).
inline void build_chain(const uint64_t* L, int k, int t, Plan& p) {
    p.t = t;
    p.k = k;
    struct Word {
        uint64_t v, term;
        void add(const Word& o) {
            v ^= o.v;
            term ^= o.term;
        }
    };
    std::vector<Word> rows((size_t)k);
    for (int r = 0; r < k; r++) rows[(size_t)r] = Word{L[r], 1ull << (k - 1 - r)};
    uint64_t supp = 0;
    uint64_t picked[64];
    p.r = 0;
    for (;;) {
        // a basis of the quotient code, reduced outside supp
        std::vector<Word> e;
        for (Word v : rows) {
            for (const Word& b : e) {
                const int c = __builtin_ctzll(b.v & ~supp);
                if ((v.v >> c) & 1) v.add(b);
            }
            if (!(v.v & ~supp)) continue;
            const int c = __builtin_ctzll(v.v & ~supp);
            for (Word& b : e)
                if ((b.v >> c) & 1) b.add(v);
            e.push_back(v);
        }
        if (e.empty()) break;
        const int d = std::min((int)e.size(), 16);
        Word x{0, 0};
        Word pick = e[0];
        int bw = 65;
        for (uint64_t i = 1; i < (1ull << d); i++) {
            x.add(e[(size_t)__builtin_ctzll(i)]);
            const int w = __builtin_popcountll(x.v & ~supp);
            if (w < bw) {
                bw = w;
                pick = x;
            }
        }
        const uint64_t best = pick.v;
        p.term[p.r] = pick.term;
        picked[p.r++] = best;
        const uint64_t add = best & ~supp;
        const int m0 = p.m[p.r - 1];
        int m = m0;
        for (uint64_t a = add; a; a &= a - 1) p.perm[m++] = (uint8_t)__builtin_ctzll(a);
        p.m[p.r] = m;
        supp |= best;
        rows = e;
    }
    // coordinates that are 0 in every codeword: contracted with the root's block
    int m = p.m[p.r];
    for (int c = 0; c < t; c++)
        if (!((supp >> c) & 1)) p.perm[m++] = (uint8_t)c;
    if (p.r > 0) p.m[p.r] = t;
    for (int j = 0; j < p.r; j++) {
        uint64_t g = 0;
        for (int i = 0; i < t; i++) g |= ((picked[j] >> p.perm[i]) & 1ull) << i;
        p.gen[j] = g;
    }
    p.tj = 0;
    // tables of up to 8 vertices: 6 at most is 34% slower at t = 40 (2^16 terms), where m[1] is often 7
    // or 8, 7 at most 27% slower at t = 24 (2^14).  With tj = 0, one leaf a table: 5, 6, 7 and 8 vertices
    // take 4.10, 3.97, 3.82 and 3.73 ms at t = 57 (256 states, 2^18), 3.46, 3.42, 3.40 and 3.41 at t = 64
    // (2048, 2^14), 0.37, 0.36, 0.35 and 0.35 at t = 40 (4096, 2^10)
    while (p.tj < p.r && p.m[p.tj + 1] <= 8) p.tj++;
    p.tv = p.tj > 0 ? p.m[p.tj] : std::min(t, 8);
}

// The terms of |H^t>: bit i of a term's index (LSB first) is the kind of the qubit
// pair ceil(t/2) - 1 - i; with odd t bit 0 is the last qubit alone, |+> for 0 and |0>
// for 1.  Pair i is at positions 2 i and 2 i + 1, the single qubit above them.
inline void build_pairs(int t, Plan& p) {
    p.t = t;
    p.pairs = true;
    const int n = t / 2, odd = t & 1;
    p.k = p.r = n + odd;
    for (int i = 0; i < n; i++) {
        const int q = 2 * (n - 1 - i);
        p.perm[2 * i] = (uint8_t)q;
        p.perm[2 * i + 1] = (uint8_t)(q + 1);
        p.gen[i] = 3ull << (2 * i);
        p.term[i] = 1ull << (i + odd);
        p.m[i] = 2 * i;
    }
    if (odd) {
        p.perm[t - 1] = (uint8_t)(t - 1);
        p.x0 = p.gen[n] = 1ull << (t - 1);  // codeword bit 1 is |+>, the term bit 0
        p.term[n] = 1;
        p.m[n] = 2 * n;
    }
    p.m[p.r] = t;
    p.tj = p.tv = 0;
}

// Levels of the written nodes by dynamic programming on the time for `count`
// states.  A stage from vp to vc vertices runs about 0.31 steps per vertex and
// node (pairs of siblings share a lane), each a pass over the rows still live, and
// every node pays for its loads and stores; a launch costs its latency, which
// decides when the states are few.
inline double stage_steps(int vp, int vc) { return 0.31 * (vp - vc) + 0.5; }
inline double stage_ops(int vp, int vc) {  // ALU operations per node
    const double w = vp > 32 ? (vc > 32 ? 2 : 1 + (vp - 32.0) / (vp - vc)) : 1;
    return stage_steps(vp, vc) * (80 + 2.6 * w * (vp + vc) / 2) + 2 * w * vp + 3 * vc + 50;
}
constexpr double kTreeOpsPerSecond = 1.6e13;  // 152 SMs, 64 lanes per cycle, 90% busy
inline double stage_seconds(int vp, int vc, double nodes) {
    const double latency = 4e-6 + 2 * stage_steps(vp, vc) * (0.35e-6 + 0.012e-6 * vp);
    return latency + nodes * stage_ops(vp, vc) / kTreeOpsPerSecond;
}
inline void choose_tree_levels(Plan& p, int64_t count) {
    const int r = p.r - p.slice;
    // candidates: index 0 the root (r, t), then (j, m[j]) for j = r - 1 .. tj, with the table's
    // vertices alone at level tj
    std::vector<int> lv{r}, vt{p.t};
    for (int j = r - 1; j > p.tj; j--) {
        lv.push_back(j);
        vt.push_back(p.m[j]);
    }
    if (p.t > p.tv && !p.pairs) {  // pairs: the leaf kernel takes the last ones
        lv.push_back(p.tj);
        vt.push_back(p.tv);
    }
    const int n = (int)lv.size();
    std::vector<double> cost((size_t)n, 1e300);
    std::vector<int> from((size_t)n, -1);
    cost[0] = 0;
    double best = 1e300;
    int end = 0;
    for (int i = 0; i < n; i++) {
        for (int h = 0; h < i; h++) {
            if (cost[(size_t)h] >= 1e300) continue;
            const double nodes = (double)count * (double)(1ull << (r - lv[(size_t)i]));
            const double c = cost[(size_t)h] + stage_seconds(vt[(size_t)h], vt[(size_t)i], nodes);
            if (c < cost[(size_t)i]) {
                cost[(size_t)i] = c;
                from[(size_t)i] = h;
            }
        }
        if (vt[(size_t)i] <= 16) {  // the leaf kernel may start here
            const double tables = (double)count * (double)(1ull << (r - p.tj));
            const double leaf = vt[(size_t)i] > p.tv ? stage_seconds(vt[(size_t)i], p.tv, tables) : 0;
            const double c = cost[(size_t)i] + leaf +
                             (double)count * (double)(1ull << (r - lv[(size_t)i])) * 60 / kTreeOpsPerSecond;
            if (c < best) {
                best = c;
                end = i;
            }
        }
    }
    p.level.clear();
    p.vert.clear();
    for (int i = end; i >= 0; i = from[(size_t)i]) {
        p.level.insert(p.level.begin(), lv[(size_t)i]);
        p.vert.insert(p.vert.begin(), vt[(size_t)i]);
    }
}

// Bytes of a tree's node planes in the two scratch halves (written levels alternate
// between them)
inline void tree_planes(const Plan& p, int64_t (&half)[2]) {
    half[0] = half[1] = 0;
    for (size_t i = 0; i < p.level.size(); i++) {
        const int64_t b = ((int64_t)node_words(p.vert[i]) * 4) << (p.level[0] - p.level[i]);
        half[i & 1] = std::max(half[i & 1], b);
    }
}

// The most that one tree's node planes may take.  They grow with the terms (64 qubits: 3.3 GB for
// 2^26, 49 GB for 2^30), so a larger state is several trees, each from a root of its own.  Random
// codes of up to 2^20 terms are one tree a state.
constexpr int64_t kTreePlanes = 64 << 20;

inline void choose_levels(Plan& p, int64_t count) {
    for (p.slice = 0;; p.slice++) {
        choose_tree_levels(p, count << p.slice);
        int64_t half[2];
        tree_planes(p, half);
        if (half[0] + half[1] <= kTreePlanes || p.r - p.slice <= p.tj) return;
    }
}

inline void make_plan(const uint64_t* L, int k, int t, int64_t count, Plan& p) {
    build_chain(L, k, t, p);
    choose_levels(p, count);
}

}  // namespace tree
}  // namespace csim
