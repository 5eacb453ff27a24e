// csim_canon_warp.cuh — a stabilizer state in pivot coordinates by one warp:
// pc::canon_theta's steps with lane l holding variables l and l + 32 (rows of G
// and J).  Shared by k_canon (csim_terms_tp.cu) and k_tree_draw (csim_tree.cu).
#pragma once

#include <cstdint>

#include "csim_pair_core.cuh"
#include "csim_warp.cuh"

namespace csim {

__device__ __forceinline__ uint64_t ballot64(bool lo, bool hi) {
    return (uint64_t)__ballot_sync(kFull, lo) | ((uint64_t)__ballot_sync(kFull, hi) << 32);
}
// coordinate-indexed mask of a variable-indexed one (variable a -> its pivot coordinate)
__device__ __forceinline__ uint64_t to_coords(uint64_t v, const unsigned char* piv) {
    uint64_t r = 0ull;
    while (v) {
        const int a = __ffsll((long long)v) - 1;
        v &= v - 1ull;
        r |= 1ull << piv[a];
    }
    return r;
}

// The pivot form by variables: rows g (of G) and j (of J) of this lane's
// variables, their pivot coordinates p, and the warp-uniform D, pivots P, shift
// wv (the variables whose pivot has h = 1) and dq (added to Q).
struct CanonWarp {
    uint64_t g0, g1, j0, j1;
    int p0, p1;
    uint64_t D1, D2, P, wv;
    int dq;
};

// In: g0, g1, j0, j1, D1, D2 as in the state (rows and bits below n and k only); h
__device__ __forceinline__ void canon_warp(CanonWarp& s, int k, uint64_t h) {
    const int lane = threadIdx.x & 31, r0 = lane, r1 = lane + 32;  // this lane's variables
    const uint64_t km = pc::lowmask(k);
    s.p0 = s.p1 = 0;
    // Gauss-Jordan on the rows of G: rows b of B += row a (u_a = u'_a + u'_b), J <- R J R^T with
    // rows in B getting J_a and rows in C getting B, D_b += D_a + 4 J_ab (pc::canon_theta)
    for (int a = 0; a < k; a++) {
        const int src = a & 31;
        const bool up = a >= 32;
        const uint64_t ga = shfl64(up ? s.g1 : s.g0, src);
        const int pcol = ga ? __ffsll((long long)ga) - 1 : 0;
        if (lane == src) {
            if (up) s.p1 = pcol;
            else s.p0 = pcol;
        }
        const bool in0 = r0 < k && r0 != a && ((s.g0 >> pcol) & 1ull), in1 = r1 < k && r1 != a && ((s.g1 >> pcol) & 1ull);
        const uint64_t B = ballot64(in0, in1);
        if (!B) continue;  // warp-uniform
        if (in0) s.g0 ^= ga;
        if (in1) s.g1 ^= ga;
        const uint64_t Ja = shfl64(up ? s.j1 : s.j0, src);
        const uint64_t C = Ja ^ (((Ja >> a) & 1ull) ? B : 0ull);
        s.j0 ^= (((B >> r0) & 1ull) ? Ja : 0ull) ^ (((C >> r0) & 1ull) ? B : 0ull);
        s.j1 ^= (((B >> r1) & 1ull) ? Ja : 0ull) ^ (((C >> r1) & 1ull) ? B : 0ull);
        pc::add_D64(s.D1, s.D2, B, (int)((s.D1 >> a) & 1ull), (int)((s.D2 >> a) & 1ull));
        s.D2 ^= B & Ja;
    }
    // shift v = u + w, w_a = h at a's pivot: in order of a, Q += D_a and D_a -> -D_a, D_b += 4 J_ab;
    // D_a as read at step a carries the earlier steps' flips J_{a'a}, a' < a in w
    const bool w0 = r0 < k && ((h >> s.p0) & 1ull), w1 = r1 < k && ((h >> s.p1) & 1ull);
    s.wv = ballot64(w0, w1);
    int dq = 0;
    if (w0) dq += 2 * (2 * (int)(((s.D2 >> r0) ^ (uint64_t)__popcll(s.j0 & s.wv & pc::lowmask(r0))) & 1ull) +
                       (int)((s.D1 >> r0) & 1ull));
    if (w1) dq += 2 * (2 * (int)(((s.D2 >> r1) ^ (uint64_t)__popcll(s.j1 & s.wv & pc::lowmask(r1))) & 1ull) +
                       (int)((s.D1 >> r1) & 1ull));
    s.dq = (int)__reduce_add_sync(kFull, (unsigned)dq);
    const uint64_t flips = warp_xor64((w0 ? s.j0 & ~(1ull << r0) : 0ull) ^ (w1 ? s.j1 & ~(1ull << r1) : 0ull));
    s.D2 ^= (s.D1 & s.wv) ^ (flips & km);
    s.P = warp_or64((r0 < k ? 1ull << s.p0 : 0ull) | (r1 < k ? 1ull << s.p1 : 0ull));
}

}  // namespace csim
