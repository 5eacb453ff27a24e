// csim_tree.cuh — the sum of <theta|phi_x> over all codewords x of |L> as a
// walk over a binary tree of partial contractions, written once for the device
// (csim_tree.cu) and the host (a program the CPU tests build).
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

// The bits of a nibble, one to a byte: times a byte, that byte where a bit is set
CSIM_HD_INLINE uint32_t spread_bits(uint32_t nib) { return (nib * 0x00204081u) & 0x01010101u; }
// byte i of w
CSIM_HD_INLINE uint32_t pick_byte(uint32_t w, int i) {
#ifdef __CUDA_ARCH__
    return __byte_perm(w, 0u, 0x4440u | (unsigned)i);
#else
    return (w >> (8 * i)) & 0xFFu;
#endif
}
// byte q of a, then byte q of b; the upper half is not 0
CSIM_HD_INLINE uint32_t pick_bytes(uint32_t a, uint32_t b, int q) {
#ifdef __CUDA_ARCH__
    return __byte_perm(a, b, 0x40u + 0x11u * (unsigned)q);
#else
    return ((a >> (8 * q)) & 0xFFu) | (((b >> (8 * q)) & 0xFFu) << 8);
#endif
}
// w with byte q of c as its third byte; the fourth is not 0
CSIM_HD_INLINE uint32_t set_third(uint32_t w, uint32_t c, int q) {
#ifdef __CUDA_ARCH__
    return __byte_perm(w, c, 0x0410u + 0x100u * (unsigned)q);
#else
    return (w & 0xFFFFu) | (((c >> (8 * q)) & 0xFFu) << 16);
#endif
}
// byte q of each of four words, as a word
CSIM_HD_INLINE uint32_t gather_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d, int q) {
#ifdef __CUDA_ARCH__
    const unsigned sel = 0x40u + 0x11u * (unsigned)q;
    return __byte_perm(__byte_perm(a, b, sel), __byte_perm(c, d, sel), 0x5410u);
#else
    return pick_byte(a, q) | (pick_byte(b, q) << 8) | (pick_byte(c, q) << 16) | (pick_byte(d, q) << 24);
#endif
}

// Byte planes of m-bit rows: 2 (at least) to 8
CSIM_HD_INLINE int row_planes(int m) { return m <= 16 ? 2 : (m + 7) / 8; }
CSIM_HD_INLINE int row_units(int m) { return (m + 3) / 4; }

// One thread's J rows, four to a unit, as byte planes: plane k of unit u is a word
// whose byte q is byte k of row 4 u + q.  A rank-two update of a unit is then two
// words of a bit per byte (the rows in U, those in V), their products with a byte of
// each pattern and one three-input XOR per plane, for as many planes as the rows have
// bytes.  The products run on the multiply-add pipe beside the logic ops: byte masks and
// two logic ops per plane are 2 to 3% slower, a word per row 3 to 10% (t = 32 to 57).
// Memory is laid out [16-byte chunk][thread]: a chunk holds planes 0..3 of a unit, or
// (two planes) those of two units.  Planes from 4 up follow as [unit][thread] tails of
// no more words than they need: shared memory limits the blocks per SM from 33
// vertices up.  Consecutive chunks (tails) of a lane are `st` chunks (tails) apart.
template <int PL>
struct Rows {
    static constexpr int tail = PL <= 4 ? 0 : PL - 4;  // words
    uint32_t *p, *tp;  // this lane's first chunk, first tail
    int st;
    CSIM_HD static int chunks(int units) { return PL == 2 ? (units + 1) / 2 : units; }
    // words a copy of `units` units takes in a block of `st` threads
    CSIM_HD static size_t words(int units, int st) { return (size_t)(4 * chunks(units) + tail * units) * st; }
    CSIM_HD static Rows at(uint32_t* base, int lane, int units, int st) {
        return Rows{base + 4 * lane, base + (size_t)4 * chunks(units) * st + tail * lane, st};
    }
    CSIM_HD_INLINE U32x4* chunk(int i) const { return reinterpret_cast<U32x4*>(p + (size_t)i * 4 * st); }
    CSIM_HD_INLINE uint32_t* tails(int u) const { return tp + (size_t)u * tail * st; }
    CSIM_HD_INLINE void shift(size_t words) {
        p += words;
        tp += words;
    }
    // planes 4 .. PL - 1 of unit u
    CSIM_HD_INLINE U32x4 get_tail(int u) const {
        if constexpr (tail == 1) return U32x4{*tails(u), 0u, 0u, 0u};
        else if constexpr (tail == 2) {
            const uint64_t v = *reinterpret_cast<const uint64_t*>(tails(u));
            return U32x4{(uint32_t)v, (uint32_t)(v >> 32), 0u, 0u};
        } else if constexpr (tail == 3) {
            const uint32_t* t = tails(u);
            return U32x4{t[0], t[1], t[2], 0u};
        } else
            return *reinterpret_cast<const U32x4*>(tails(u));
    }
    CSIM_HD_INLINE void set_tail(int u, const U32x4& v) const {
        if constexpr (tail == 1) *tails(u) = v.a;
        else if constexpr (tail == 2) *reinterpret_cast<uint64_t*>(tails(u)) = (uint64_t)v.a | ((uint64_t)v.b << 32);
        else if constexpr (tail == 3) {
            uint32_t* t = tails(u);
            t[0] = v.a;
            t[1] = v.b;
            t[2] = v.c;
        }
        else *reinterpret_cast<U32x4*>(tails(u)) = v;
    }
    // row i; bits from 8 PL up (PL = 2, 3) are not the row's
    CSIM_HD_INLINE uint64_t get(int i) const {
        const int u = i >> 2, q = i & 3;
        if constexpr (PL == 2) {
            const uint32_t* w = p + (size_t)(u >> 1) * 4 * st + 2 * (u & 1);
            return pick_bytes(w[0], w[1], q);
        } else {
            const U32x4 v = *chunk(u);
            if constexpr (PL == 3) return set_third(pick_bytes(v.a, v.b, q), v.c, q);
            const uint32_t lo = gather_bytes(v.a, v.b, v.c, v.d, q);
            if constexpr (PL <= 4) return lo;
            else if constexpr (tail == 1) return (uint64_t)lo | ((uint64_t)pick_byte(*tails(u), q) << 32);
            else {
                const U32x4 w = get_tail(u);
                return (uint64_t)lo | ((uint64_t)gather_bytes(w.a, w.b, w.c, w.d, q) << 32);
            }
        }
    }
    // row x ^= (x in U ? P : 0) ^ (x in V ? R : 0) for the rows x < n (whole units; rows past
    // n hold nothing that is read)
    CSIM_HD_INLINE void rank2(int n, uint64_t U, uint64_t P, uint64_t V, uint64_t R) const {
        uint32_t pk[PL], rk[PL];
#pragma unroll
        for (int k = 0; k < PL; k++) {
            pk[k] = pick_byte((uint32_t)(k < 4 ? P : P >> 32), k & 3);
            rk[k] = pick_byte((uint32_t)(k < 4 ? R : R >> 32), k & 3);
        }
        // nibble u of a mask: byte u / 2 of its even or odd nibbles
        constexpr uint64_t nibs = 0x0F0F0F0F0F0F0F0Full;
        const uint64_t ue = U & nibs, uo = (U >> 4) & nibs, ve = V & nibs, vo = (V >> 4) & nibs;
#pragma unroll
        for (int u = 0; u < 2 * PL; u += 2) {  // two units at a time
            if (4 * u >= n) break;
            const uint32_t me = spread_bits(pick_byte((uint32_t)(u < 8 ? ue : ue >> 32), (u >> 1) & 3)),
                           mo = spread_bits(pick_byte((uint32_t)(u < 8 ? uo : uo >> 32), (u >> 1) & 3)),
                           ne = spread_bits(pick_byte((uint32_t)(u < 8 ? ve : ve >> 32), (u >> 1) & 3)),
                           no = spread_bits(pick_byte((uint32_t)(u < 8 ? vo : vo >> 32), (u >> 1) & 3));
            if constexpr (PL == 2) {
                U32x4 v = *chunk(u >> 1);
                v.a ^= (me * pk[0]) ^ (ne * rk[0]);
                v.b ^= (me * pk[1]) ^ (ne * rk[1]);
                v.c ^= (mo * pk[0]) ^ (no * rk[0]);
                v.d ^= (mo * pk[1]) ^ (no * rk[1]);
                *chunk(u >> 1) = v;
            } else {
                update(u, me, ne, pk, rk);
                if (4 * (u + 1) < n) update(u + 1, mo, no, pk, rk);
            }
        }
    }

  private:
    CSIM_HD_INLINE void update(int u, uint32_t mu, uint32_t mv, const uint32_t (&pk)[PL], const uint32_t (&rk)[PL]) const {
        U32x4 v = *chunk(u);
        v.a ^= (mu * pk[0]) ^ (mv * rk[0]);
        v.b ^= (mu * pk[1]) ^ (mv * rk[1]);
        if constexpr (PL > 2) v.c ^= (mu * pk[2]) ^ (mv * rk[2]);
        if constexpr (PL > 3) v.d ^= (mu * pk[3]) ^ (mv * rk[3]);
        *chunk(u) = v;
        if constexpr (PL > 4) {
            U32x4 w = get_tail(u);
            w.a ^= (mu * pk[4]) ^ (mv * rk[4]);
            if constexpr (PL > 5) w.b ^= (mu * pk[5]) ^ (mv * rk[5]);
            if constexpr (PL > 6) w.c ^= (mu * pk[6]) ^ (mv * rk[6]);
            if constexpr (PL > 7) w.d ^= (mu * pk[7]) ^ (mv * rk[7]);
            set_tail(u, w);
        }
    }
};
// the word that holds a row of PL bytes
template <int PL>
struct RowWord {
    using type = uint32_t;
};
template <>
struct RowWord<5> {
    using type = uint64_t;
};
template <>
struct RowWord<6> {
    using type = uint64_t;
};
template <>
struct RowWord<7> {
    using type = uint64_t;
};
template <>
struct RowWord<8> {
    using type = uint64_t;
};

// The scalar part of a node: bit c of d1, d2, h belongs to vertex c
template <class W>
struct Node {
    W d1, d2, h;
    int q, iso, dead;  // w^q 2^{iso/2}; dead: the amplitude is 0
};

// all ones if x is not 0
template <class W>
CSIM_HD_INLINE W some(W x) {
    return wmask<W>(x != (W)0);
}
// the index of x's highest bit, -1 for x = 0; bit i as a word, 0 for i = -1
CSIM_HD_INLINE int top_index(uint32_t x) {
#ifdef __CUDA_ARCH__
    int i;
    asm("bfind.u32 %0, %1;" : "=r"(i) : "r"(x));
    return i;
#else
    return x ? 31 - __builtin_clz(x) : -1;
#endif
}
CSIM_HD_INLINE int top_index(uint64_t x) {
    const uint32_t hi = (uint32_t)(x >> 32);
    const int i = top_index(hi ? hi : (uint32_t)x);
    return hi ? i + 32 : i;
}
template <class W>
CSIM_HD_INLINE W bit_at(int i);
template <>
CSIM_HD_INLINE uint32_t bit_at<uint32_t>(int i) {
#ifdef __CUDA_ARCH__
    uint32_t m;
    asm("shl.b32 %0, 1, %1;" : "=r"(m) : "r"(i));  // 0 for a shift by 32 or more
    return m;
#else
    return (unsigned)i < 32u ? 1u << i : 0u;
#endif
}
template <>
CSIM_HD_INLINE uint64_t bit_at<uint64_t>(int i) {
    return (uint64_t)bit_at<uint32_t>(i) | ((uint64_t)bit_at<uint32_t>((int)((unsigned)i - 32u)) << 32);
}

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
// Written in masks (all ones or zero) and without branches: lanes differ in every
// condition, and a select by mask is one three-input logic op with what it selects for.
template <class W, class R>
CSIM_HD_INLINE void sum_step(const R& rows, Work<W>& w) {
    Node<W>& s = w.s;
    const int ic = top_index(w.sum), none = ic >> 31;  // nothing to sum: ic -1, none all ones
    const W mc = bit_at<W>(ic);
    const W sum1 = w.sum ^ mc, live1 = w.live & ~mc;
    const W N0 = (W)rows.get(ic < 0 ? 0 : ic) & live1 & ~(W)none;
    const W odd = some(s.d1 & mc), d = some(s.d2 & mc);
    const W near = N0 & sum1;
    const W even_pick = near != (W)0 ? near : N0;
    const W pick = (odd & sum1 & (s.d1 ^ N0)) | (~odd & even_pick);
    const int ib = top_index(pick), single = ib >> 31;
    const W mb = bit_at<W>(ib);
    const W M0 = (W)rows.get(ib < 0 ? 0 : ib) & live1 & ~(mb | (W)single);
    const W N = N0 & ~mb;
    const W db1 = some(s.d1 & mb);
    // D on N: odd adds 6 (d = 0) or 2 (d = 1); a pivot adds D_b's odd part times (1 - 2 d)
    const W plus = s.d1 ^ odd ^ d;
    const W joined = N0 & mb & odd;  // b's own D after an odd c
    const W d2 = s.d2 ^ (joined & plus);
    const W db2 = some(d2 & mb);
    const W wn = N & (odd | db1);
    const W M = M0 ^ (N & some(joined));
    const W d1 = s.d1 ^ wn;
    const W more = (odd & M & (d1 ^ ~db2)) | (~odd & ((N & (db2 ^ M)) ^ (M & d)));
    // a pivot's new bit at b: D = 4 d, neighbourhood N, Hadamard toggled
    s.d1 = (d1 ^ (M & odd)) & ~mb;
    s.d2 = ((d2 ^ (wn & plus) ^ more) & ~mb) | (d & mb);
    s.h ^= mb;
    // w^{1 - 2 d} and, with a second odd vertex, w^{1 - 2 d_b}; a pivot's w^{d D_b}.  Products of
    // the masks (0 or -1): multiply-adds run beside the logic ops
    const int o = (int)odd, di = (int)d, b1 = (int)db1, b2 = (int)db2;
    s.q -= o * (1 + 2 * di + ~single * -(1 + 2 * b2));
    s.q += (~o & di) * (2 * b1 + 4 * b2);
    const int lone = ~none & ~o & single;  // an even vertex without neighbours: 2 or 0, times 2^{-1/2}
    s.dead |= lone & di;
    s.iso -= lone;
    w.sum = sum1 & ~mb;
    w.live = live1 & ~(mb & sum1);  // a b that is summed too is gone: its new bit is contracted to 0
    // odd: rows of N get N, rows of M get M.  Pivot: rows of N get M (and N when D_b is odd),
    // rows of M get N, column b of both changes and row b becomes N
    const int n = uniform_max(top_index(w.live) + 1);
    rows.rank2(n, N | mb, wn ^ (~odd & (M ^ mb)), M | (mb & ~db1), (odd & M) | (~odd & (N ^ mb)));
}

// Steps for two nodes of a lane, whose rows lie `words` apart, until neither has a
// vertex of `until` left to sum: a lane goes on to its second node when it is done
// with its first, without waiting for the other lanes.  The number of steps varies between lanes (13 vertices, half of
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
        rows.rank2(uniform_max(top_index(w.live) + 1), N, mb, mb, N);
    }
}

// Sums two sibling nodes down to their first mc vertices.  With more than four
// planes and mc <= 32 the upper planes are needed only until the vertices from 32
// up are gone.
template <int PL, class W>
CSIM_HD_INLINE void contract_pair(const Rows<PL>& rows, size_t words, Work<W>& a, Work<W>& b, int mc) {
    if constexpr (PL <= 4) {
        sum_out_pair<W>(rows, words, a, b, ~(W)0);
    } else {
        if (mc > 32) {
            sum_out_pair<W>(rows, words, a, b, ~(W)0);
            return;
        }
        sum_out_pair<W>(rows, words, a, b, ~(W)0xFFFFFFFFu);
        auto low = [](const Work<W>& w) {
            return Work<uint32_t>{{(uint32_t)w.s.d1, (uint32_t)w.s.d2, (uint32_t)w.s.h, w.s.q, w.s.iso, w.s.dead},
                                  (uint32_t)w.sum, (uint32_t)w.live};
        };
        auto back = [](Work<W>& w, const Work<uint32_t>& n) {
            w.s = Node<W>{n.s.d1, n.s.d2, n.s.h, n.s.q, n.s.iso, n.s.dead};
            w.sum = n.sum;
            w.live = n.live;
        };
        Work<uint32_t> a32 = low(a), b32 = low(b);
        sum_out_pair<uint32_t>(Rows<4>{rows.p, rows.tp, rows.st}, words, a32, b32, ~0u);  // without the tails
        back(a, a32);
        back(b, b32);
    }
}

// ---------------------------------------------------------------- the last vertices
// A node of v <= 8 vertices as the truth table of q over its 2^v points, 32 to
// a word: with D_c = 2 (2 D2_c + D1_c), w^{q} = w^Q i^{p0 + 2 p1} where p0 = D1.z
// mod 2 and p1 = sum_i z_i (D2_i + sum_{j<i} (J_ij + D1_i D1_j) z_j) mod 2.  A
// leaf x sums the points z within S = x ^ h and costs two counts per word, and
// all leaves of the node share the table.
constexpr int kTableVars = 8;

// Lookup tables, by entry r < 32: the truth table over five bits z of parity(r & z); of
// z within r.  By r < 64, the edges among four of the bits (edge j i, j < i, in bit
// i (i - 1) / 2 + j): of sum of z_j z_i over the edges, mod 2.
CSIM_HD_INLINE uint32_t coordinate_word(int i) {  // of z_i
    return i == 0 ? 0xAAAAAAAAu : (i == 1 ? 0xCCCCCCCCu : (i == 2 ? 0xF0F0F0F0u : (i == 3 ? 0xFF00FF00u : 0xFFFF0000u)));
}
CSIM_HD_INLINE uint32_t linear_word(uint32_t r) {
    uint32_t w = 0;
#pragma unroll
    for (int i = 0; i < 5; i++) w ^= coordinate_word(i) & wmask<uint32_t>((r >> i) & 1u);
    return w;
}
CSIM_HD_INLINE uint32_t subset_word(uint32_t r) {
    uint32_t w = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < 5; i++) w &= ~coordinate_word(i) | wmask<uint32_t>((r >> i) & 1u);
    return w;
}
CSIM_HD_INLINE uint32_t edges_word(uint32_t r) {
    uint32_t w = 0;
#pragma unroll
    for (int i = 1; i < 4; i++)
#pragma unroll
        for (int j = 0; j < i; j++)
            w ^= coordinate_word(i) & coordinate_word(j) & wmask<uint32_t>((r >> (i * (i - 1) / 2 + j)) & 1u);
    return w;
}
struct TableWords {
    // by 2 |S| + (S meets D1): the points of S with p0 = 0 and p0 = 1, and 2^{(v - |S|) / 2} as
    // c + sqrt2 d
    U32x4 scale[2 * kTableVars + 2];
    uint32_t lin[32], sub[32], edges[64];
    CSIM_HD_INLINE void fill(int i, int v) {  // i = 0 .. 31; tables of v vertices
        lin[i] = linear_word((uint32_t)i);
        sub[i] = subset_word((uint32_t)i);
        edges[i] = edges_word((uint32_t)i);
        edges[32 + i] = edges_word((uint32_t)(32 + i));
        const int size = i >> 1;
        if (size <= v && size <= kTableVars) {
            const uint32_t n = 1u << size, n1 = (i & 1) ? n >> 1 : 0u;
            const int e = v - size;
            const uint32_t one = 1u << (e >> 1);
            scale[i] = U32x4{n - n1, n1, (e & 1) ? 0u : one, (e & 1) ? one : 0u};
        }
    }
};

template <int WORDS>
struct Table {
    uint32_t a[WORDS], c[WORDS];  // points with p1 = 1 and p0 = 0; p0 = 1
};
// r0, r4: the J rows of vertices 0..3 and 4..7, a byte each (bits below the vertex's are used)
template <int WORDS>
CSIM_HD_INLINE void build_table(uint32_t r0, uint32_t r4, uint32_t d1, uint32_t d2, const TableWords& tw, Table<WORDS>& t) {
    // D1_i D1_j joins the edges; vertices 0..3 are looked up at once
    r0 = (r0 ^ (spread_bits(d1 & 15u) * d1)) & 0x07030100u;
    r4 = (r4 ^ (spread_bits(d1 >> 4) * d1)) & 0x7F3F1F0Fu;
    uint32_t q1[WORDS], q0[WORDS];
    q1[0] = tw.edges[(r0 * ((1u << 18) | (1u << 11) | (1u << 5))) >> 26] ^ (tw.lin[pick_byte(r4, 0)] & 0xFFFF0000u) ^
            tw.lin[d2 & 31u];
    q0[0] = tw.lin[d1 & 31u];
#pragma unroll
    for (int i = 5; (32 << (i - 5)) < 32 * WORDS; i++) {  // vertex i doubles the table: its linear form where z_i = 1
        const int half = 1 << (i - 5);
        const uint32_t row = pick_byte(r4, i - 4);
        const uint32_t l = tw.lin[row & 31u] ^ wmask<uint32_t>((d2 >> i) & 1u), o = wmask<uint32_t>((d1 >> i) & 1u);
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
CSIM_HD_INLINE void table_leaf(const Table<WORDS>& t, uint32_t S, uint32_t d1, const TableWords& tw, int& evr, int& evi,
                               int& odr, int& odi) {
    using T = WordTraits<uint32_t>;
    uint32_t mk[WORDS];
    mk[0] = tw.sub[S & 31u];
    int na = T::popc(mk[0] & t.a[0]), nc = T::popc(mk[0] & t.c[0]);
#pragma unroll
    for (int w = 1; w < WORDS; w++) {
        const int top = w >= 4 ? 4 : (w >= 2 ? 2 : 1);
        mk[w] = (S & (32u * top)) ? mk[w - top] : 0u;
        na += T::popc(mk[w] & t.a[w]);
        nc += T::popc(mk[w] & t.c[w]);
    }
    const U32x4 sc = tw.scale[2 * T::popc(S) + ((S & d1) != 0u ? 1 : 0)];
    const int re = (int)sc.a - 2 * na, im = (int)sc.b - 2 * nc;
    evr += re * (int)sc.c;
    evi += im * (int)sc.c;
    odr += re * (int)sc.d;
    odi += im * (int)sc.d;
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
// `count` nodes of m vertices lie in planes: first planes of 16-byte vectors, vector v
// of node i at word 4 (v count + i), then the rows' tails (Rows<row_planes(m)>), tail u
// of node i at (u count + i) tail words, then (m > 16) a word with the status.  The
// vectors are the scalars D1, D2, H, X (m > 32: two, D1 D2 and H X, low word first;
// m <= 16: D1 | D2 << 16, H | X << 16, status, 0) and the rows' chunks.  X: the codeword
// bits of the node's message so far (positions < m are still to come).  Row and column
// bits from m up are not zero: whoever reads a row masks it.
CSIM_HD_INLINE int node_scalars(int m) { return m > 32 ? 2 : 1; }  // vectors
CSIM_HD_INLINE int node_vectors(int m) { return node_scalars(m) + (m > 16 ? row_units(m) : Rows<2>::chunks(row_units(m))); }
CSIM_HD_INLINE int row_tail(int m) { return m <= 32 ? 0 : row_planes(m) - 4; }
CSIM_HD_INLINE int node_words(int m) { return 4 * node_vectors(m) + row_tail(m) * row_units(m) + (m > 16 ? 1 : 0); }
CSIM_HD_INLINE uint32_t pack_status(int q, int iso, int dead) {
    return (uint32_t)(q & 7) | ((uint32_t)iso << 8) | (dead ? 0x80000000u : 0u);
}

}  // namespace tree
}  // namespace csim
