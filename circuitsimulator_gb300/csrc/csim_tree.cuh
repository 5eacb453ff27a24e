// csim_tree.cuh — the sum of <theta|phi_x> over all codewords x of |L> as a
// walk over a binary tree of partial contractions, written once for the device
// (csim_tree.cu) and the host (a checker the CPU tests build).
//
// A term phi_x of |L> is a product of |0> (x_c = 0) and |+> (x_c = 1)
// (libcirc/stateprep.c:85-120), so <theta|phi_x> contracts theta's qubits one
// by one, and codewords that agree on some coordinates share those
// contractions.  The host chooses a chain of subcodes C_0 < C_1 < ... < C_r
// with small supports and orders the coordinates by it (csim_tree_plan.h): the
// node of a coset of C_j has contracted every coordinate outside supp(C_j), so
// it is a state of only m_j = |supp(C_j)| qubits.  A random 16-row code on 40
// qubits has m_1, m_2, ... around 7, 13, 17, 20, 23, 26: a term costs the
// contraction of seven qubits of a seven-qubit state, half of six more of a
// 13-qubit state, a quarter of four more, ...
//
// A node's state is prod_{c in H} Had_c  sum_z w^{q(z)} |z> over m bits z
// (w = e^{i pi/4}, Had a Hadamard), q(z) = Q + sum D_c z_c + 4 sum_{a<b} J_ab
// z_a z_b with D_c = 2 (2 D2_c + D1_c): a graph state with local Cliffords.
// Contracting qubit c:
//   x_c = 0 outside H, or x_c = 1 in H (<+|Had = <0|):  z_c = 0, the vertex goes;
//   otherwise 2^{-1/2} sum over z_c:
//     D_c odd: 1 + w^{D_c} w^{4 N.z} = sqrt2 w^{+-1} w^{-+2 (N.z mod 2)}, a local
//       complementation of c's neighbourhood N = J_c;
//     D_c even, N = 0: 2 or 0;
//     D_c even, N not 0: z_b = D2_c + (N \ b).z for a neighbour b; the qubit b
//       stays, as Had_b on a new bit with neighbourhood N \ b (a pivot along
//       the edge c b).  With b itself among the qubits to sum, the new bit is
//       contracted to 0 at once and both are gone.
// Every vertex not summed to a scalar contributes 2^{0/2}; only the isolated
// vertex adds 2^{1/2}, counted in `iso`.
#pragma once

#include <cstdint>

#include "csim_pair_core.cuh"

namespace csim {
namespace tree {

using pc::U32x4;
using pc::WordTraits;
using pc::uniform_any;
using pc::uniform_max;
using pc::wbit;
using pc::wlow;
using pc::wmask;

// The four bits of a nibble as the bytes 0 or 1 of a word (one multiply puts bit
// i at bit 8 i).  A row update is then v ^ P * bit ^ R * bit: the products run on
// the FMA pipe and one three-input XOR takes them in, where masking P and R takes
// two logic ops (the ALU pipe is the busy one: 90% in a stage).
CSIM_HD_INLINE uint32_t row_bits(uint32_t nib) { return (nib * 0x00204081u) & 0x01010101u; }
// all-ones masks of the four rows of a unit (one prmt per row replicates a sign)
CSIM_HD_INLINE void row_masks(uint32_t nib, uint32_t (&m)[4]) {
#ifdef __CUDA_ARCH__
    const uint32_t s = nib * 0x10204080u;
    asm("prmt.b32 %0, %1, 0, 0x8888;" : "=r"(m[0]) : "r"(s));
    asm("prmt.b32 %0, %1, 0, 0x9999;" : "=r"(m[1]) : "r"(s));
    asm("prmt.b32 %0, %1, 0, 0xAAAA;" : "=r"(m[2]) : "r"(s));
    asm("prmt.b32 %0, %1, 0, 0xBBBB;" : "=r"(m[3]) : "r"(s));
#else
    for (int i = 0; i < 4; i++) m[i] = (nib >> i) & 1u ? ~0u : 0u;
#endif
}
// the same for rows of 16 bits, two to a word (row 2i in the low half)
CSIM_HD_INLINE void half_masks(uint32_t nib, uint32_t& m01, uint32_t& m23) {
#ifdef __CUDA_ARCH__
    const uint32_t s = nib * 0x10204080u;
    asm("prmt.b32 %0, %1, 0, 0x9988;" : "=r"(m01) : "r"(s));
    asm("prmt.b32 %0, %1, 0, 0xBBAA;" : "=r"(m23) : "r"(s));
#else
    m01 = ((nib & 1u) ? 0xFFFFu : 0u) | ((nib & 2u) ? 0xFFFF0000u : 0u);
    m23 = ((nib & 4u) ? 0xFFFFu : 0u) | ((nib & 8u) ? 0xFFFF0000u : 0u);
#endif
}

// byte i of w, zero-extended
CSIM_HD_INLINE uint32_t pick_byte(uint32_t w, int i) {
#ifdef __CUDA_ARCH__
    return __byte_perm(w, 0u, 0x4440u | (unsigned)i);
#else
    return (w >> (8 * i)) & 0xFFu;
#endif
}

// One thread's J rows in memory laid out [unit][thread], 16-byte units `st`
// units apart.  rank2(n, U, P, V, R): row x ^= (x in U ? P : 0) ^ (x in V ? R : 0)
// for the rows x < n (whole units; rows past n hold nothing that is read).
struct Rows32 {  // four 32-bit rows to a unit
    uint32_t* p;
    int st;
    CSIM_HD_INLINE uint32_t get(int i) const { return p[(size_t)(i >> 2) * 4 * st + (i & 3)]; }
    CSIM_HD_INLINE U32x4* unit(int u) const { return reinterpret_cast<U32x4*>(p + (size_t)u * 4 * st); }
    CSIM_HD_INLINE void shift(size_t words) { p += words; }
    CSIM_HD_INLINE void rank2(int n, uint32_t U, uint32_t P, uint32_t V, uint32_t R) const {
        // nibble u of a mask: byte u/2 of its even or odd nibbles
        const uint32_t Ue = U & 0x0F0F0F0Fu, Uo = (U >> 4) & 0x0F0F0F0Fu, Ve = V & 0x0F0F0F0Fu, Vo = (V >> 4) & 0x0F0F0F0Fu;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (4 * u >= n) break;
            U32x4 v = *unit(u);
            const uint32_t a = row_bits(pick_byte((u & 1) ? Uo : Ue, u >> 1));
            const uint32_t b = row_bits(pick_byte((u & 1) ? Vo : Ve, u >> 1));
            v.a = v.a ^ (P * pick_byte(a, 0)) ^ (R * pick_byte(b, 0));
            v.b = v.b ^ (P * pick_byte(a, 1)) ^ (R * pick_byte(b, 1));
            v.c = v.c ^ (P * pick_byte(a, 2)) ^ (R * pick_byte(b, 2));
            v.d = v.d ^ (P * (a >> 24)) ^ (R * (b >> 24));
            *unit(u) = v;
        }
    }
};
struct Rows64 {  // low and high halves of four rows in a unit each
    uint32_t *lo, *hi;
    int st;
    CSIM_HD_INLINE uint64_t get(int i) const {
        const size_t o = (size_t)(i >> 2) * 4 * st + (i & 3);
        return (uint64_t)lo[o] | ((uint64_t)hi[o] << 32);
    }
    CSIM_HD_INLINE void shift(size_t words) {
        lo += words;
        hi += words;
    }
    CSIM_HD_INLINE U32x4* unit_lo(int u) const { return reinterpret_cast<U32x4*>(lo + (size_t)u * 4 * st); }
    CSIM_HD_INLINE U32x4* unit_hi(int u) const { return reinterpret_cast<U32x4*>(hi + (size_t)u * 4 * st); }
    CSIM_HD_INLINE void rank2(int n, uint64_t U, uint64_t P, uint64_t V, uint64_t R) const {
        const uint32_t Pl = (uint32_t)P, Ph = (uint32_t)(P >> 32), Rl = (uint32_t)R, Rh = (uint32_t)(R >> 32);
        for (int u = 0; 4 * u < n; u++) {
            U32x4 a = *unit_lo(u), b = *unit_hi(u);
            uint32_t mu[4], mv[4];
            row_masks((uint32_t)U & 15u, mu);
            row_masks((uint32_t)V & 15u, mv);
            a.a ^= (Pl & mu[0]) ^ (Rl & mv[0]);
            a.b ^= (Pl & mu[1]) ^ (Rl & mv[1]);
            a.c ^= (Pl & mu[2]) ^ (Rl & mv[2]);
            a.d ^= (Pl & mu[3]) ^ (Rl & mv[3]);
            b.a ^= (Ph & mu[0]) ^ (Rh & mv[0]);
            b.b ^= (Ph & mu[1]) ^ (Rh & mv[1]);
            b.c ^= (Ph & mu[2]) ^ (Rh & mv[2]);
            b.d ^= (Ph & mu[3]) ^ (Rh & mv[3]);
            *unit_lo(u) = a;
            *unit_hi(u) = b;
            U >>= 4;
            V >>= 4;
        }
    }
};
struct Rows16 {  // eight 16-bit rows to a unit
    uint32_t* p;
    int st;
    CSIM_HD_INLINE uint32_t get(int i) const {
        return reinterpret_cast<const uint16_t*>(p)[(size_t)(i >> 3) * 8 * st + (i & 7)];
    }
    CSIM_HD_INLINE U32x4* unit(int u) const { return reinterpret_cast<U32x4*>(p + (size_t)u * 4 * st); }
    CSIM_HD_INLINE void shift(size_t words) { p += words; }
    CSIM_HD_INLINE void rank2(int n, uint32_t U, uint32_t P, uint32_t V, uint32_t R) const {
        const uint32_t PP = P * 0x10001u, RR = R * 0x10001u;
        for (int u = 0; 8 * u < n; u++) {
            U32x4 v = *unit(u);
            uint32_t u0, u1, u2, u3, v0, v1, v2, v3;
            half_masks(U & 15u, u0, u1);
            half_masks((U >> 4) & 15u, u2, u3);
            half_masks(V & 15u, v0, v1);
            half_masks((V >> 4) & 15u, v2, v3);
            v.a ^= (PP & u0) ^ (RR & v0);
            v.b ^= (PP & u1) ^ (RR & v1);
            v.c ^= (PP & u2) ^ (RR & v2);
            v.d ^= (PP & u3) ^ (RR & v3);
            *unit(u) = v;
            U >>= 8;
            V >>= 8;
        }
    }
};

// The scalar part of a node: bit c of d1, d2, h belongs to vertex c
template <class W>
struct Node {
    W d1, d2, h;
    int q, iso, dead;  // w^q 2^{iso/2}; dead: the amplitude is 0
};

// A node being contracted: the vertices of `sum` are to be summed out (2^{-1/2}
// sum over z_c each) on the vertices `live` (sum within live; vertices outside
// live have been set to 0).
template <class W>
struct Work {
    Node<W> s;
    W sum, live;
};

// One step: c, the highest vertex of sum, and a second one where it can, as one
// rank-two update of the rows: after an odd c, a b that is odd once c is gone;
// with an even c, a neighbour b in `sum` (with no neighbour there, the pivot
// takes c alone).  The rows keep stale bits in the columns of vertices that are
// gone and on the diagonal: every row is masked by `live` when it is read.  All
// lanes of a warp call it together; a lane with nothing to sum changes nothing.
template <class W, class R>
CSIM_HD_INLINE void sum_step(const R& rows, Work<W>& w) {
    using T = WordTraits<W>;
    Node<W>& s = w.s;
    W sum = w.sum, live = w.live;
    const bool act = sum != (W)0;
    const int c = act ? T::bits - 1 - T::clz(sum) : 0;
    const W mc = act ? wbit<W>(c) : (W)0;
    sum ^= mc;
    live &= ~mc;
    const W N0 = act ? ((W)rows.get(c) & live) : (W)0;
    const bool odd = (s.d1 & mc) != (W)0, d = (s.d2 & mc) != (W)0;
    const W near = N0 & sum;
    const W pick = odd ? sum & (s.d1 ^ N0) : (near != (W)0 ? near : N0);
    const bool two = pick != (W)0;
    const int b = two ? T::bits - 1 - T::clz(pick) : 0;
    const W mb = two ? wbit<W>(b) : (W)0;
    const W gone = mb & sum;  // a pivot's b that is summed too: its new bit is contracted to 0
    const W N = N0 & ~mb;
    W M = two ? ((W)rows.get(b) & live & ~mb) : (W)0;
    const bool db1 = (s.d1 & mb) != (W)0;
    // D on N: odd adds 6 (d = 0) or 2 (d = 1); a pivot adds D_b's odd part times (1 - 2 d)
    const W plus = wmask<W>(odd != d);
    s.d2 ^= (odd ? N0 : (W)0) & mb & (s.d1 ^ plus);  // b's own D after an odd c
    const bool db2 = (s.d2 & mb) != (W)0;
    const W wn = (odd || db1) ? N : (W)0;
    s.d2 ^= wn & (s.d1 ^ plus);
    s.d1 ^= wn;
    if (odd) {
        M ^= (N0 & mb) ? N : (W)0;
        s.q += (d ? 7 : 1) + (two ? (db2 ? 7 : 1) : 0);
        s.d2 ^= M & (s.d1 ^ wmask<W>(!db2));
        s.d1 ^= M;
    } else {
        if (act && !two) {
            s.dead |= d ? 1 : 0;
            s.iso++;
        }
        s.q += d ? (db1 ? 2 : 0) + (db2 ? 4 : 0) : 0;
        s.d2 ^= (db2 ? N : (W)0) ^ (d ? M : (W)0) ^ (N & M);
    }
    // a pivot's new bit at b: D = 4 d, neighbourhood N, Hadamard toggled
    s.d1 &= ~mb;
    s.d2 = (s.d2 & ~mb) | (d ? mb : (W)0);
    s.h ^= mb;
    sum &= ~mb;
    live &= ~gone;
    // odd: rows of N get N, rows of M get M.  Pivot: rows of N get M (and N when D_b is odd),
    // rows of M get N, column b of both changes and row b becomes N
    const int n = uniform_max(T::bits - T::clz(live));
    rows.rank2(n, N | mb, odd ? N : M ^ wn ^ mb, M | (db1 ? (W)0 : mb), odd ? M : N ^ mb);
    w.sum = sum;
    w.live = live;
}

// Steps until no lane has a vertex of `until` left to sum
template <class W, class R>
CSIM_HD_INLINE void sum_out(const R& rows, Work<W>& w, W until) {
    while (uniform_any((w.sum & until) != (W)0)) sum_step<W>(rows, w);
}

// The same for two nodes of a lane, whose rows lie `words` apart: a lane goes on
// to its second node when it is done with its first, without waiting for the
// other lanes.  The number of steps varies between lanes (13 vertices, half of
// them to be summed: 3.9 on average, 5.9 in a warp's slowest lane), that of a
// pair of siblings much less: their x agree or are complements on most positions.
template <class W, class R>
CSIM_HD_INLINE void sum_out_pair(R rows, size_t words, Work<W>& a, Work<W>& b, W until) {
    Work<W> w = a;
    bool second = false;
    while (uniform_any(((w.sum & until) | (second ? (W)0 : b.sum & until)) != (W)0)) {
        if (!second && (w.sum & until) == (W)0) {
            a = w;
            w = b;
            rows.shift(words);
            second = true;
        }
        sum_step<W>(rows, w);
    }
    if (second) b = w;
    else a = w;
}

// Terms of |H^t> (libcirc/stateprep.c:36-81) are products of two-qubit states on the
// vertices 2 i, 2 i + 1: for a term bit 0 CZ|++>, for 1 (|00> + |11>) / sqrt2.  With
// an odd number of Hadamards on the two vertices they change places, with two each is
// its own image.  Contracting with the first is an edge between the vertices and a
// sum over both; with the second z_a = z_b: vertex a joins b and b is summed.
// Brings the pairs in positions [lo, hi) into that form (x: the term bits, one on
// each of a pair's positions); they are all in w.live before, in w.sum after.
template <class W, class R>
CSIM_HD_INLINE void join_pairs(const R& rows, Work<W>& w, W x, int lo, int hi, bool act) {
    using T = WordTraits<W>;
    Node<W>& s = w.s;
    for (int a = lo; a < hi; a += 2) {  // uniform
        const W ma = act ? wbit<W>(a) : (W)0, mb = act ? wbit<W>(a + 1) : (W)0;
        const bool bell = (((x >> a) ^ (s.h >> a) ^ (s.h >> (a + 1))) & (W)1) != (W)0;
        const W row = (W)rows.get(a) & w.live & ~ma;
        const W N = (bell && act) ? row & ~mb : ma;  // U; the other kind: the edge a b
        const bool jab = (row & mb) != (W)0;
        if (bell) {
            const bool a1 = (s.d1 & ma) != (W)0, a2 = (s.d2 & ma) != (W)0, b1 = (s.d1 & mb) != (W)0;
            s.d2 ^= (a2 != (a1 && b1)) != jab ? mb : (W)0;  // D_b += D_a + 4 J_ab
            s.d1 ^= a1 ? mb : (W)0;
            w.live &= ~ma;
        }
        w.sum |= bell ? mb : ma | mb;
        rows.rank2(uniform_max(T::bits - T::clz(w.live)), N, mb, mb, N);
    }
}

// Sums two sibling nodes down to their first mc vertices.  With rows of two words
// and mc <= 32 the second words are needed only until the vertices from 32 up are gone.
CSIM_HD_INLINE void contract_pair(const Rows32& rows, size_t words, Work<uint32_t>& a, Work<uint32_t>& b, int) {
    sum_out_pair<uint32_t>(rows, words, a, b, ~0u);
}
CSIM_HD_INLINE void contract_pair(const Rows64& rows, size_t words, Work<uint64_t>& a, Work<uint64_t>& b, int mc) {
    if (mc > 32) {
        sum_out_pair<uint64_t>(rows, words, a, b, ~0ull);
        return;
    }
    sum_out_pair<uint64_t>(rows, words, a, b, ~0xFFFFFFFFull);
    auto low = [](const Work<uint64_t>& w) {
        return Work<uint32_t>{{(uint32_t)w.s.d1, (uint32_t)w.s.d2, (uint32_t)w.s.h, w.s.q, w.s.iso, w.s.dead},
                              (uint32_t)w.sum, (uint32_t)w.live};
    };
    auto back = [](Work<uint64_t>& w, const Work<uint32_t>& n) {
        w.s = Node<uint64_t>{n.s.d1, n.s.d2, n.s.h, n.s.q, n.s.iso, n.s.dead};
        w.sum = n.sum;
        w.live = n.live;
    };
    Work<uint32_t> a32 = low(a), b32 = low(b);
    sum_out_pair<uint32_t>(Rows32{rows.lo, rows.st}, words, a32, b32, ~0u);
    back(a, a32);
    back(b, b32);
}

// ---------------------------------------------------------------- the last vertices
// A node of v <= 8 vertices as the truth table of q over its 2^v points, 32 to
// a word: with D_c = 2 (2 D2_c + D1_c), w^{q} = w^Q i^{p0 + 2 p1} where p0 = D1.z
// mod 2 and p1 = sum_i z_i (D2_i + sum_{j<i} (J_ij + D1_i D1_j) z_j) mod 2.  A
// leaf x sums the points z within S = x ^ h and costs two counts per word, and
// all leaves of the node share the table.
constexpr int kTableVars = 8;

// entry r < 32: the truth table over five bits z of parity(r & z); of z within r
CSIM_HD_INLINE uint32_t linear_word(uint32_t r) {
    uint32_t w = 0;
    for (uint32_t z = 0; z < 32; z++) w |= (uint32_t)(WordTraits<uint32_t>::popc(r & z) & 1) << z;
    return w;
}
CSIM_HD_INLINE uint32_t subset_word(uint32_t r) {
    uint32_t w = 0;
    for (uint32_t z = 0; z < 32; z++) w |= (uint32_t)((z & ~r) == 0u) << z;
    return w;
}

template <int WORDS>
struct Table {
    uint32_t a[WORDS], c[WORDS];  // points with p1 = 1 and p0 = 0; p0 = 1
};
// rows r[i]: J row i of vertex i (bits below i are used)
template <int WORDS>
CSIM_HD_INLINE void build_table(const uint32_t (&r)[kTableVars], uint32_t d1, uint32_t d2, const uint32_t* lin,
                                Table<WORDS>& t) {
    const uint32_t zw[5] = {0xAAAAAAAAu, 0xCCCCCCCCu, 0xF0F0F0F0u, 0xFF00FF00u, 0xFFFF0000u};
    uint32_t q1[WORDS], q0[WORDS];
    q1[0] = 0u;
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const uint32_t row = (r[i] ^ (((d1 >> i) & 1u) ? d1 : 0u)) & ((1u << i) - 1u);
        q1[0] ^= zw[i] & ((i ? lin[row] : 0u) ^ wmask<uint32_t>((d2 >> i) & 1u));
    }
    q0[0] = lin[d1 & 31u];
#pragma unroll
    for (int i = 5; (32 << (i - 5)) < 32 * WORDS; i++) {  // vertex i doubles the table: its linear form where z_i = 1
        const int half = 1 << (i - 5);
        const uint32_t row = r[i] ^ (((d1 >> i) & 1u) ? d1 : 0u);
        const uint32_t l = lin[row & 31u] ^ wmask<uint32_t>((d2 >> i) & 1u), o = wmask<uint32_t>((d1 >> i) & 1u);
        const uint32_t l5 = wmask<uint32_t>((row >> 5) & 1u), l6 = wmask<uint32_t>((row >> 6) & 1u);
#pragma unroll
        for (int w = 0; w < half; w++) {
            q1[half + w] = q1[w] ^ l ^ ((w & 1) ? l5 : 0u) ^ ((w & 2) ? l6 : 0u);
            q0[half + w] = q0[w] ^ o;
        }
    }
#pragma unroll
    for (int w = 0; w < WORDS; w++) {
        t.a[w] = q1[w] & ~q0[w];
        t.c[w] = q1[w] & q0[w];
    }
}
// 2^{-|S|/2} sum_{z in S} i^{p0 + 2 p1}, times 2^{v/2}, added to ev + sqrt2 od (re, im each)
template <int WORDS>
CSIM_HD_INLINE void table_leaf(const Table<WORDS>& t, uint32_t S, uint32_t d1, int v, const uint32_t* sub, int& evr,
                               int& evi, int& odr, int& odi) {
    using T = WordTraits<uint32_t>;
    uint32_t mk[WORDS];
    mk[0] = sub[S & 31u];
    int na = T::popc(mk[0] & t.a[0]), nc = T::popc(mk[0] & t.c[0]);
#pragma unroll
    for (int w = 1; w < WORDS; w++) {
        const int top = w >= 4 ? 4 : (w >= 2 ? 2 : 1);
        mk[w] = (S & (32u * top)) ? mk[w - top] : 0u;
        na += T::popc(mk[w] & t.a[w]);
        nc += T::popc(mk[w] & t.c[w]);
    }
    const int size = T::popc(S), n = 1 << size;
    const int n1 = (S & d1) ? n >> 1 : 0;  // points with p0 = 1
    const int re = n - n1 - 2 * na, im = n1 - 2 * nc;
    const int e = v - size, one = 1 << (e >> 1), mo = (e & 1) ? one : 0, me = one - mo;
    evr += re * me;
    evi += im * me;
    odr += re * mo;
    odi += im * mo;
}
CSIM_HD_INLINE int table_words(int v) { return v > 5 ? 1 << (v - 5) : 1; }

// y0 + y1 w + y2 w^2 + y3 w^3 times sqrt2 = w - w^3
template <class I>
CSIM_HD_INLINE void times_sqrt2(I (&y)[4]) {
    const I a = y[1] - y[3], b = y[0] + y[2], c = y[1] + y[3], d = y[2] - y[0];
    y[0] = a;
    y[1] = b;
    y[2] = c;
    y[3] = d;
}
// times w^q
template <class I>
CSIM_HD_INLINE void times_omega(I (&y)[4], int q) {
    if (q & 1) {
        const I t = -y[3];
        y[3] = y[2];
        y[2] = y[1];
        y[1] = y[0];
        y[0] = t;
    }
    if (q & 2) {
        const I a = -y[2], b = -y[3];
        y[2] = y[0];
        y[3] = y[1];
        y[0] = a;
        y[1] = b;
    }
    if (q & 4)
        for (int i = 0; i < 4; i++) y[i] = -y[i];
}

// ---------------------------------------------------------------- node records
// Nodes lie in planes of 32-bit words: word w of node i at base[w * count + i].
// m > 32 vertices: two words per row (low, high), then D1, D2, H, X (two words
// each), then the status; m > 16: one word per row, then D1, D2, H, X, status;
// else rows two to a word, then D1 | D2 << 16, H | X << 16, status.  X: the
// codeword bits of the node's message so far (positions < m are still to come).
CSIM_HD_INLINE int node_class(int m) { return m > 32 ? 64 : (m > 16 ? 32 : 16); }
CSIM_HD_INLINE int node_row_words(int m) { return m > 32 ? 2 * m : (m > 16 ? m : (m + 1) / 2); }
CSIM_HD_INLINE int node_words(int m) { return node_row_words(m) + (m > 32 ? 9 : (m > 16 ? 5 : 3)); }
CSIM_HD_INLINE uint32_t pack_status(int q, int iso, int dead) {
    return (uint32_t)(q & 7) | ((uint32_t)iso << 8) | (dead ? 0x80000000u : 0u);
}

}  // namespace tree
}  // namespace csim
