// csim_rng.cuh — random words for randomStabilizerState on the device.
//
// The reference draws every random bit through the C library's rand()
// (libcirc/stabilizer/stabilizer.c:669-756, libcirc/utils/matrix.c:85-92).
// A state's draws are addressed here by their position c in that state's own
// sequence, from one of two sources:
//   * Philox-4x32-10 (Salmon et al., SC'11), counter (c/4, id, id_hi, c>>34),
//     key = seed: an independent stream per state, 31-bit outputs like rand();
//   * replay: words[base + c] >> shift, the exact values rand() returned to the
//     reference (shift 0), or its generator's raw words, whose upper 31 bits those
//     are (shift 1).
#pragma once

#include <cstdint>

#include "csim_warp.cuh"

namespace csim {

__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
        const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
        c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c;
}

struct DevRng {
    int mode;                // 0 = Philox, 1 = replay
    int shift;               // replay: 1 for raw words
    uint32_t k0, k1;         // Philox key
    uint32_t id0, id1;       // Philox stream (state index)
    const uint32_t* words;   // replay words
    int64_t base, end;       // replay segment [base, end)
    int64_t cur;             // next draw position

    __device__ __forceinline__ uint32_t at(int64_t c, int& err) const {
        if (mode == 1) {
            const int64_t q = base + c;
            if (q >= end) {
                err |= kErrReplay;
                return 0u;
            }
            return words[q] >> shift;
        }
        const uint4 r = philox4x32_10(make_uint4((uint32_t)(c >> 2), id0, id1, (uint32_t)(c >> 34)), k0, k1);
        const int j = (int)(c & 3);
        const uint32_t w = j == 0 ? r.x : (j == 1 ? r.y : (j == 2 ? r.z : r.w));
        return w >> 1;
    }

    __device__ __forceinline__ uint32_t next(int& err) { return at(cur++, err); }

    // ceil(n/8) bytes rand() % 256, bit j of byte b (MSB first) -> bit 8b+j.  Lane b
    // draws byte b, so the warp waits for one draw instead of eight.
    __device__ __forceinline__ uint64_t bits(int n, int& err) {
        const int bytes = (n + 7) / 8, b = threadIdx.x & 31;
        uint64_t w = 0ull;
        if (b < bytes) w = (uint64_t)(__brev(at(cur + b, err) & 255u) >> 24) << (8 * b);
        if (mode == 1 && __any_sync(kFull, (err & kErrReplay) != 0)) err |= kErrReplay;  // seen by every lane
        cur += bytes;
        return warp_or64(w) & lowmask(n);
    }
};

// The generator of one state: Philox stream (seed, id) (mode 0), or words
// [begin, end) as rand() values (mode 1) or raw words (mode 2)
__device__ __forceinline__ DevRng make_rng(int mode, uint64_t seed, uint64_t id, const uint32_t* words, int64_t begin,
                                           int64_t end) {
    DevRng r;
    r.mode = mode == 0 ? 0 : 1;
    r.shift = mode == 2 ? 1 : 0;
    r.k0 = (uint32_t)seed;
    r.k1 = (uint32_t)(seed >> 32);
    r.id0 = (uint32_t)id;
    r.id1 = (uint32_t)(id >> 32);
    r.words = words;
    r.base = begin;
    r.end = end;
    r.cur = 0;
    return r;
}

// randomStabilizerState (stabilizer.c:689-756).  cum[0..n] is the
// normalized cumulative distribution of eq. 79 computed on the host with the
// reference's own libm expressions (logeta, stabilizer.c:677-687).
template <int NR>
__device__ void random_state(WS<NR>& s, int n, DevRng& rng, const double* cum, int& err) {
    double sample = 0.0;
    for (int guard = 0; guard < 64; guard++) {  // rand() == 0 has probability 2^-31 per draw
        sample = 0.0 + (double)rng.next(err) / 2147483647.0;
        if (sample != 0.0 || (err & kErrReplay)) break;
    }
    int d = 0;
    for (; d <= n; d++)
        if (sample <= cum[d]) break;
    if (d > n) d = n;
    const int kt = n - d;
    init_identity<NR>(s, n);
    for (int guard = 0; s.k > kt; guard++) {
        if (guard > 4096 || (err & kErrReplay)) {
            err |= (err & kErrReplay) ? 0 : kErrArg;
            break;
        }
        const uint64_t xi = rng.bits(n, err);
        shrink<NR, true, true>(s, xi, 0);
    }
    s.h = rng.bits(n, err);
    s.D1 = rng.bits(n, err);
    s.D2 = rng.bits(n, err);
    // J: word base + x (x - 1) / 2 + c holds J[x][c], c < x, in its low bit, so the lower
    // triangle is a string of bits with row x at bit x (x - 1) / 2.  The warp draws it
    // into shared memory (each word once; a Philox block's four words by one lane),
    // lanes take their rows, and ballots give the columns (1024 states of 40 qubits: 34 us
    // when every lane drew the words of its own row, 11 us now; latency-bound).
    const int k = s.k;
    const int64_t base = rng.cur;
    const int nbits = k * (k - 1) / 2, lane = lane_id();
    __shared__ uint32_t tri_s[8][68];  // blocks have at most 8 warps; 2016 bits, up to 3 in front, a word beyond
    uint32_t* const tri = tri_s[threadIdx.x >> 5];
    const int lead = rng.mode == 1 ? 0 : (int)(base & 3);
    __syncwarp();
    if (rng.mode == 1) {
        for (int w = 0; 32 * w < nbits; w++) {
            const int i = 32 * w + lane;
            const uint32_t v = __ballot_sync(kFull, i < nbits && (rng.at(base + i, err) & 1u));
            if (lane == 0) tri[w] = v;
        }
    } else {
        for (int w = 0; 32 * w < nbits + lead; w += 4) {
            const int64_t q = (base >> 2) + 8 * w + lane;  // lane's block: words 4 q .. 4 q + 3
            const uint4 r = philox4x32_10(make_uint4((uint32_t)q, rng.id0, rng.id1, (uint32_t)(q >> 32)), rng.k0, rng.k1);
            uint32_t v = ((r.x >> 1) & 1u) | (r.y & 2u) | ((r.z & 2u) << 1) | ((r.w & 2u) << 2);
            v |= __shfl_down_sync(kFull, v, 1) << 4;
            v |= __shfl_down_sync(kFull, v, 2) << 8;
            v |= __shfl_down_sync(kFull, v, 4) << 16;
            if ((lane & 7) == 0) tri[w + (lane >> 3)] = v;
        }
    }
    __syncwarp();
    RW<NR> low[NR];  // J[x][c], c < x
#pragma unroll
    for (int sl = 0; sl < NR; sl++) {
        const int x = row_of<NR>(sl);
        low[sl] = 0ull;
        if (x >= 1 && x < k) {
            const int at = lead + x * (x - 1) / 2, w = at >> 5, sh = at & 31;
            const uint64_t v = (uint64_t)tri[w] | ((uint64_t)tri[w + 1] << 32);
            low[sl] = (RW<NR>)((v >> sh) | (sh ? (uint64_t)tri[w + 2] << (64 - sh) : 0ull)) & low_mask<NR>(x);
        }
    }
#pragma unroll
    for (int sl = 0; sl < NR; sl++) {
        const int x = row_of<NR>(sl);
        s.J[sl] = x < k ? low[sl] | ((RW<NR>)getbit(s.D1, x) << x) : (RW<NR>)0;  // J[x][x] = ((2 D[x]) mod 8) / 4
    }
    for (int x = 0; x < k; x++) {
        const RW<NR> col = ballot_bit<NR>(low, x);  // rows c > x with J[c][x] = 1
        if (lane == (x & 31)) {
            if (NR == 2 && x >= 32) s.J[NR - 1] |= col;
            else s.J[0] |= col;
        }
    }
    rng.cur = base + (int64_t)k * (k - 1) / 2;
    // every lane may have seen a different replay overrun
    if (__any_sync(kFull, (err & kErrReplay) != 0)) err |= kErrReplay;
}

}  // namespace csim
