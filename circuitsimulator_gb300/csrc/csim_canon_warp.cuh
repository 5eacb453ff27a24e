// csim_canon_warp.cuh — a stabilizer state in pivot coordinates by one warp:
// pc::canon_theta's steps with lane l holding variables l (and l + 32): rows of G
// and J.  Shared by k_canon (csim_terms_tp.cu) and k_tree_draw (csim_tree.cu).
#pragma once

#include <cstdint>

#include "csim_pair_core.cuh"
#include "csim_warp.cuh"

namespace csim {

// coordinate-indexed mask of a variable-indexed one (variable a -> its pivot coordinate)
template <class W>
__device__ __forceinline__ W to_coords(W v, const unsigned char* piv) {
    W r = 0;
    while (v) {
        const int a = first_bit(v);
        v &= v - (W)1;
        r |= (W)1 << piv[a];
    }
    return r;
}

// The pivot form by variables: rows g (of G) and j (of J) of this lane's
// variables (NR each, as in WS), their pivot coordinates p, and the warp-uniform D,
// pivots P, shift wv (the variables whose pivot has h = 1) and dq (added to Q).
template <int NR>
struct CanonWarp {
    RW<NR> g[NR], j[NR];
    int p[NR];
    RW<NR> D1, D2, P, wv;
    int dq;
};

// In: g, j, D1, D2 as in the state (rows and bits below n and k only); h
template <int NR>
__device__ __forceinline__ void canon_warp(CanonWarp<NR>& s, int k, RW<NR> h) {
    using W = RW<NR>;
    const W km = low_mask<NR>(k);
    bool in[2] = {};
#pragma unroll
    for (int q = 0; q < NR; q++) s.p[q] = 0;
    // Gauss-Jordan on the rows of G: rows b of B += row a (u_a = u'_a + u'_b), J <- R J R^T with
    // rows in B getting J_a and rows in C getting B, D_b += D_a + 4 J_ab (pc::canon_theta)
    for (int a = 0; a < k; a++) {
        const W ga = row_get<NR>(s.g, a);
        const int pcol = ga ? first_bit(ga) : 0;
#pragma unroll
        for (int q = 0; q < NR; q++) {
            const int r = row_of<NR>(q);
            if (r == a) s.p[q] = pcol;
            in[q] = r < k && r != a && ((s.g[q] >> pcol) & (W)1);
        }
        const W B = ballot_i<NR>(in[0], in[NR - 1]);
        if (!B) continue;  // warp-uniform
        const W Ja = row_get<NR>(s.j, a);
        const W C = Ja ^ (((Ja >> a) & (W)1) ? B : (W)0);
#pragma unroll
        for (int q = 0; q < NR; q++) {
            const int r = row_of<NR>(q);
            if (in[q]) s.g[q] ^= ga;
            s.j[q] ^= (((B >> r) & (W)1) ? Ja : (W)0) ^ (((C >> r) & (W)1) ? B : (W)0);
        }
        const W c1 = ((s.D1 >> a) & (W)1) ? B : (W)0, c2 = ((s.D2 >> a) & (W)1) ? B : (W)0;  // D_b += D_a
        s.D2 ^= c2 ^ (s.D1 & c1) ^ (B & Ja);
        s.D1 ^= c1;
    }
    // shift v = u + w, w_a = h at a's pivot: in order of a, Q += D_a and D_a -> -D_a, D_b += 4 J_ab;
    // D_a as read at step a carries the earlier steps' flips J_{a'a}, a' < a in w
    bool w[2] = {};
#pragma unroll
    for (int q = 0; q < NR; q++) w[q] = row_of<NR>(q) < k && ((h >> s.p[q]) & (W)1);
    s.wv = ballot_i<NR>(w[0], w[NR - 1]);
    int dq = 0;
    W flips = 0, P = 0;
#pragma unroll
    for (int q = 0; q < NR; q++) {
        const int r = row_of<NR>(q);
        if (w[q]) {
            dq += 2 * (2 * (int)(((s.D2 >> r) ^ (W)popcount(s.j[q] & s.wv & low_mask<NR>(r))) & (W)1) +
                       (int)((s.D1 >> r) & (W)1));
            flips ^= s.j[q] & ~bit_of<NR>(r);
        }
        if (r < k) P |= bit_of<NR>(s.p[q]);
    }
    s.dq = warp_sum(dq);
    s.D2 ^= (s.D1 & s.wv) ^ (warp_xor(flips) & km);
    s.P = warp_or(P);
}

}  // namespace csim
