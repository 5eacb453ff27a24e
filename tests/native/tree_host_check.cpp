// Host build of the tree sum (circuitsimulator_gb300/csrc/csim_tree.cuh and
// csim_tree_plan.h), for CPU tests only: the plan the host code makes and the
// node steps the kernels run, in the kernels' order, without a GPU.
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../circuitsimulator_gb300/csrc/csim_tree.cuh"
#include "../../circuitsimulator_gb300/csrc/csim_tree_plan.h"
#include "../../include/csim.h"

using namespace csim::tree;

namespace {

struct HostNode {
    uint64_t row[64];
    uint64_t d1, d2, h, x;
    int q, iso, dead;
};

template <class W>
Work<W> work_of(const HostNode& n, int mp, int mc) {
    const W pm = wlow<W>(mp), cm = wlow<W>(mc);
    Work<W> w{{(W)n.d1, (W)n.d2, (W)n.h, n.q, n.iso, 0}, 0, 0};
    w.sum = ((W)n.x ^ w.s.h) & pm & ~cm;
    w.live = cm | w.sum;
    return w;
}
template <class W, class R>
void take(HostNode& n, const Work<W>& w, const R& rows, int mc) {
    const W cm = wlow<W>(mc);
    n.d1 = (uint64_t)(w.s.d1 & cm);
    n.d2 = (uint64_t)(w.s.d2 & cm);
    n.h = (uint64_t)(w.s.h & cm);
    n.x &= (uint64_t)cm;
    n.q = w.s.q & 7;
    n.iso = w.s.iso;
    n.dead |= w.s.dead;
    for (int i = 0; i < mc; i++) n.row[i] = (uint64_t)((W)rows.get(i) & cm);
}

// terms of |H^t> (paired > 0): the pairs among the positions [mc, mp) joined
template <class W, class R>
void join(const R& rows, Work<W>& w, const HostNode& n, int mp, int mc, int paired) {
    const int hi = paired < mp ? paired : mp;
    if (hi <= mc) return;
    const W pm = wlow<W>(hi) & ~wlow<W>(mc);
    w.sum &= ~pm;
    w.live = wlow<W>(mc) | w.sum | pm;
    join_pairs<W>(rows, w, (W)n.x, mc, hi, true);
}
// row i of rows laid out as Rows<PL>
template <int PL>
void put_row(const Rows<PL>& rows, int i, uint64_t v) {
    const int u = i >> 2;
    for (int k = 0; k < PL; k++) {
        uint32_t* w = PL == 2 ? rows.p + 4 * (u >> 1) + 2 * (u & 1) + k : (k < 4 ? rows.p + 4 * u + k : rows.tails(u) + k - 4);
        reinterpret_cast<uint8_t*>(w)[i & 3] = (uint8_t)(v >> (8 * k));
    }
}

// contracts positions [mc, mp) of two siblings with the rows that the kernels
// use for mp vertices
template <int PL>
void stage_planes(HostNode& a, HostNode& b, int mp, int mc, int paired) {
    using W = typename RowWord<PL>::type;
    const size_t copy = (Rows<PL>::words(row_units(mp), 1) + 3) / 4 * 4;  // 16-byte chunks
    alignas(16) uint32_t w[2 * 16 * 8] = {0};
    const Rows<PL> r0 = Rows<PL>::at(w, 0, row_units(mp), 1), r1 = Rows<PL>::at(w + copy, 0, row_units(mp), 1);
    for (int i = 0; i < mp; i++) {
        put_row(r0, i, a.row[i]);
        put_row(r1, i, b.row[i]);
    }
    auto wa = work_of<W>(a, mp, mc), wb = work_of<W>(b, mp, mc);
    join(r0, wa, a, mp, mc, paired);
    join(r1, wb, b, mp, mc, paired);
    contract_pair<PL>(r0, copy, wa, wb, mc);
    take(a, wa, r0, mc);
    take(b, wb, r1, mc);
}
void stage(HostNode& a, HostNode& b, int mp, int mc, int paired) {
    switch (row_planes(mp)) {
    case 2: return stage_planes<2>(a, b, mp, mc, paired);
    case 3: return stage_planes<3>(a, b, mp, mc, paired);
    case 4: return stage_planes<4>(a, b, mp, mc, paired);
    case 5: return stage_planes<5>(a, b, mp, mc, paired);
    case 6: return stage_planes<6>(a, b, mp, mc, paired);
    case 7: return stage_planes<7>(a, b, mp, mc, paired);
    default: return stage_planes<8>(a, b, mp, mc, paired);
    }
}

HostNode root_of(const csim_state& th, const Plan& p) {
    csim::pc::Canon cs;
    uint64_t G[64], Jc[64], acol[64], h = 0;
    auto perm = [&](uint64_t v) {
        uint64_t r = 0;
        for (int i = 0; i < p.t; i++) r |= ((v >> p.perm[i]) & 1ull) << i;
        return r;
    };
    for (int a = 0; a < 64; a++) G[a] = a < th.k ? perm(th.G[a]) : 0;
    h = perm(th.h);
    csim::pc::canon_theta(th.n, th.k, th.Q, h, th.D1, th.D2, G, th.J, Jc, acol, cs);
    HostNode n{};
    const uint64_t nm = csim::pc::lowmask(th.n);
    for (int c = 0; c < th.n; c++) {
        n.row[c] |= Jc[c] | acol[c];
        for (int y = 0; y < th.n; y++)
            if ((acol[c] >> y) & 1) n.row[y] |= 1ull << c;
    }
    n.h = ~cs.P & nm;
    n.d1 = cs.D1;
    n.d2 = cs.D2 | (cs.bm & n.h);
    n.q = cs.Q;
    n.x = p.x0;
    return n;
}

}  // namespace

// Sums of all terms (2^k of code L; of |H^t> if L is null) for each theta, as the kernels' exact coordinates
// scaled by 2^t: out[8 a + 2 q] low and out[8 a + 2 q + 1] high word of
// coordinate q.  info (optional): r, table vertices, written levels.
extern "C" int tree_host_sums(const csim_state* theta, int ntheta, const uint64_t* L, int k, int t, int64_t count,
                              uint64_t* out, int* info) {
    Plan p;
    if (L) make_plan(L, k, t, count, p);  // the levels for `count` states
    else {
        build_pairs(t, p);
        choose_levels(p, count);
    }
    const int paired = p.pairs ? 2 * (t / 2) : 0;
    if (info) {
        info[0] = p.r;
        info[1] = p.tv;
        info[2] = (int)p.level.size();
        for (size_t i = 0; i < p.level.size(); i++) info[3 + i] = p.vert[i];
    }
    TableWords tables;
    for (int i = 0; i < 32; i++) tables.fill(i, p.tv);
    const int words = table_words(p.tv);
    for (int a = 0; a < ntheta; a++) {
        std::vector<HostNode> cur{root_of(theta[a], p)};
        for (size_t s = 1; s < p.level.size(); s++) {
            const int sb = p.level[s - 1] - p.level[s];
            std::vector<HostNode> next;
            for (const HostNode& par : cur)
                for (int c = 0; c < (1 << sb); c += 2) {
                    HostNode n = par;
                    for (int b = 1; b < sb; b++)
                        if ((c >> b) & 1) n.x ^= p.gen[p.level[s] + b];
                    HostNode o = n;
                    if (sb) o.x ^= p.gen[p.level[s]];
                    if (!par.dead) stage(n, o, p.vert[s - 1], p.vert[s], paired);
                    next.push_back(n);
                    if (sb) next.push_back(o);
                }
            cur.swap(next);
        }
        const int je = p.level.back(), m = p.vert.back();
        __int128 z[4] = {0, 0, 0, 0};
        for (const HostNode& entry : cur) {
            if (entry.dead) continue;
            uint64_t x = entry.x;
            for (int s = 0; s < (1 << (je - p.tj)); s++) {
                if (s) x ^= p.gen[p.tj + __builtin_ctz((unsigned)s)];
                HostNode n = entry;
                n.x = x;
                n.iso = 0;
                HostNode o = n;
                if (m > p.tv) stage(n, o, m, p.tv, paired);
                uint32_t r[2] = {0, 0};
                for (int i = 0; i < kTableVars && i < m; i++) r[i >> 2] |= (uint32_t)(n.row[i] & 0xFFu) << (8 * (i & 3));
                const uint32_t vm = wlow<uint32_t>(p.tv), d1 = (uint32_t)n.d1 & vm;
                int e0 = 0, e1 = 0, o0 = 0, o1 = 0;
                uint32_t S = ((uint32_t)(x ^ n.h)) & vm;
                auto leaves = [&](auto tb) {
                    build_table(r[0], r[1], d1, (uint32_t)n.d2 & vm, tables, tb);
                    for (int l = 0; l < (1 << p.tj); l++) {
                        if (l) S ^= (uint32_t)p.gen[__builtin_ctz((unsigned)l)] & vm;
                        table_leaf(tb, S, d1, tables, e0, e1, o0, o1);
                    }
                };
                if (words == 1) leaves(Table<1>());
                else if (words == 2) leaves(Table<2>());
                else if (words == 4) leaves(Table<4>());
                else leaves(Table<8>());
                if (n.dead) continue;
                int v[4] = {e0, o0 + o1, e1, o1 - o0};
                times_omega(v, n.q);
                if (n.iso & 1) times_sqrt2(v);
                __int128 y[4];
                for (int q = 0; q < 4; q++) y[q] = (__int128)v[q] << (n.iso >> 1);
                if (entry.iso & 1) times_sqrt2(y);
                for (int q = 0; q < 4; q++) z[q] += y[q] << (entry.iso >> 1);
            }
        }
        const int shift = t - p.tv;
        if (shift & 1) times_sqrt2(z);
        for (int q = 0; q < 4; q++) {
            const unsigned __int128 w = (unsigned __int128)z[q] << ((shift >> 1) + (p.k - p.r));
            out[8 * a + 2 * q] = (uint64_t)w;
            out[8 * a + 2 * q + 1] = (uint64_t)(w >> 64);
        }
    }
    return 0;
}
