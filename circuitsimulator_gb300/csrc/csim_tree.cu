// csim_tree.cu — kernels of the tree sum (csim_tree.cuh): all terms of a
// decomposition, |L> or |H^t>, for many states.
//   k_tree_draw   one warp per state: draws (or makes) it, projects it, and writes
//                 its graph form (csim_canon_warp.cuh) on coordinates in the plan's
//                 order as a root node
//   k_tree_stage  one thread per node of the next written level: contracts the
//                 coordinates between the two levels for its own message bits
//   k_tree_leaf   one thread per node of the last written level (or a part of
//                 one): the remaining levels, then the leaves' values from truth
//                 tables, summed exactly
//   k_tree_values one warp per state: its sum, as the sampler's value or as a row
//                 of exactProjector
#include <cuda_runtime.h>

#include <cstdint>

#include "csim_canon_warp.cuh"
#include "csim_rng.cuh"
#include "csim_tree.cuh"
#include "csim_tree.h"
#include "csim_values.cuh"
#include "csim_warp.cuh"

namespace csim {

using namespace tree;

namespace {

// the job of block b: the last one with block0 <= b
template <class J>
__device__ __forceinline__ const J& job_of(const J* jobs, int njobs, int64_t b) {
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (jobs[mid].block0 <= b) lo = mid;
        else hi = mid - 1;
    }
    return jobs[lo];
}

// bits of v in the plan's order (position -> coordinate)
__device__ __forceinline__ uint64_t permute_bits(uint64_t v, const unsigned char* perm, int t) {
    uint64_t r = 0ull;
    for (int i = 0; i < t; i++) r |= ((v >> perm[i]) & 1ull) << i;
    return r;
}

// stores row `pos` of node i among `count` nodes of m vertices
__device__ __forceinline__ void store_row(uint32_t* base, int64_t count, int64_t i, int m, int pos, uint64_t row) {
    if (m > 32) {
        base[(int64_t)(2 * pos) * count + i] = (uint32_t)row;
        base[(int64_t)(2 * pos + 1) * count + i] = (uint32_t)(row >> 32);
    } else if (m > 16) {
        base[(int64_t)pos * count + i] = (uint32_t)row;
    } else {
        reinterpret_cast<uint16_t*>(base + (int64_t)(pos >> 1) * count + i)[pos & 1] = (uint16_t)row;
    }
}
__device__ __forceinline__ void store_scalars(uint32_t* base, int64_t count, int64_t i, int m, uint64_t d1, uint64_t d2,
                                              uint64_t h, uint64_t x, uint32_t status) {
    uint32_t* p = base + (int64_t)node_row_words(m) * count + i;
    if (m > 32) {
        p[0] = (uint32_t)d1;
        p[count] = (uint32_t)(d1 >> 32);
        p[2 * count] = (uint32_t)d2;
        p[3 * count] = (uint32_t)(d2 >> 32);
        p[4 * count] = (uint32_t)h;
        p[5 * count] = (uint32_t)(h >> 32);
        p[6 * count] = (uint32_t)x;
        p[7 * count] = (uint32_t)(x >> 32);
        p[8 * count] = status;
    } else if (m > 16) {
        p[0] = (uint32_t)d1;
        p[count] = (uint32_t)d2;
        p[2 * count] = (uint32_t)h;
        p[3 * count] = (uint32_t)x;
        p[4 * count] = status;
    } else {
        p[0] = (uint32_t)d1 | ((uint32_t)d2 << 16);
        p[count] = (uint32_t)h | ((uint32_t)x << 16);
        p[2 * count] = status;
    }
}

}  // namespace

// ---------------------------------------------------------------- roots
namespace {

// the warp's scratch: the plan's order and the variables' pivots
struct RootShared {
    unsigned char perm[64];
    unsigned char piv[kTreeRootWarps][64];
};

// a state that the projector annihilates, or a bad one: its sum is 0
__device__ __forceinline__ void dead_root(const TreeRootJob& J, int64_t i) {
    if (lane_id() == 0) store_scalars(J.out, J.count, i, J.t, 0, 0, 0, 0, pack_status(0, 0, 1));
}

// Node i of the job from a state held by the warp
template <int NR>
__device__ void store_root(const TreeRootJob& J, int64_t i, const WS<NR>& st, RootShared& sh) {
    unsigned char* const piv = sh.piv[threadIdx.x >> 5];
    const int t = J.t, k = st.k;
    const uint64_t km = pc::lowmask(k), nm = pc::lowmask(t);
    const int r0 = lane_id(), r1 = r0 + 32;  // this lane's variables
    CanonWarp w;
    w.g0 = r0 < k ? permute_bits(st.G[0], sh.perm, t) : 0ull;
    w.g1 = NR == 2 && r1 < k ? permute_bits(st.G[NR - 1], sh.perm, t) : 0ull;
    w.j0 = r0 < k ? st.J[0] & km : 0ull;
    w.j1 = NR == 2 && r1 < k ? st.J[NR - 1] & km : 0ull;
    w.D1 = st.D1 & km;
    w.D2 = st.D2 & km;
    const uint64_t h = permute_bits(st.h, sh.perm, t);
    canon_warp(w, k, h);
    __syncwarp();
    piv[r0] = (unsigned char)(r0 < k ? w.p0 : 0);
    piv[r1] = (unsigned char)(r1 < k ? w.p1 : 0);
    __syncwarp();
    // pivots: vertices with J and D; a non-pivot coordinate y = b + a.v is Had on a vertex
    // joined to the variables in a, with D = 4 b
    uint64_t row0 = to_coords(w.j0, piv), row1 = to_coords(w.j1, piv), bm = 0ull;
    for (uint64_t np = ~w.P & nm; np;) {
        const int c = __ffsll((long long)np) - 1;
        np &= np - 1ull;
        const bool in0 = r0 < k && ((w.g0 >> c) & 1ull), in1 = r1 < k && ((w.g1 >> c) & 1ull);
        const uint64_t av = ballot64(in0, in1);
        if (in0) row0 |= 1ull << c;
        if (in1) row1 |= 1ull << c;
        if (r0 == (c & 31)) store_row(J.out, J.count, i, t, c, to_coords(av, piv));
        if ((((h >> c) & 1ull) ^ (uint64_t)(__popcll(w.wv & av) & 1)) != 0ull) bm |= 1ull << c;
    }
    if (r0 < k) store_row(J.out, J.count, i, t, w.p0, row0);
    if (r1 < k) store_row(J.out, J.count, i, t, w.p1, row1);
    if (r0 == 0)
        store_scalars(J.out, J.count, i, t, to_coords(w.D1, piv), to_coords(w.D2, piv) | bm, ~w.P & nm, J.x0,
                      pack_status(st.Q + w.dq, 0, 0));
}

}  // namespace

// Drawing, projecting and the graph form in one launch, the state never leaving the
// warp's registers.  Bound by the latency of a warp's serial steps: 1024 states of
// 40 qubits take 44 us; k_random_states, k_project and a kernel for the graph form
// took 11 + 29 + 26 us.  NR = 1: jobs of up to 32 qubits, 2: the others.
template <int NR>
__global__ void __launch_bounds__(32 * kTreeRootWarps) k_tree_draw(const TreeRootJob* jobs, int njobs, int* err) {
    __shared__ RootShared sh;
    const TreeRootJob& J = job_of(jobs, njobs, blockIdx.x);
    if ((int)threadIdx.x < J.t) sh.perm[threadIdx.x] = J.perm[threadIdx.x];
    __syncthreads();
    const int64_t i = ((int64_t)blockIdx.x - J.block0) * kTreeRootWarps + (threadIdx.x >> 5);
    if (i >= J.count) return;  // warp-uniform
    const TreeDraw& d = J.draw;
    const int64_t a = J.first + i;
    int e = 0;
    const bool replay = d.mode == 1 || d.mode == 2;
    DevRng rng = make_rng(replay ? d.mode : 0, d.seed, d.id + a, d.words, replay ? d.offsets[a] : 0,
                          replay ? d.offsets[a + 1] : 0);
    WS<NR> st;
    if (d.mode == 3) {  // uniform
        const int64_t j = (int64_t)d.id + a;
        if (d.k < 0) {
            prep_h<NR>(st, J.t, j);
        } else {
            uint64_t x = 0ull;
            for (int r = 0; r < d.k; r++)
                if ((j >> (d.k - 1 - r)) & 1) x ^= d.words64[r];
            prep_l<NR>(st, J.t, x);
        }
    } else {
        random_state<NR>(st, J.t, rng, d.cum, e);
    }
    int c = 0;  // the number of 2^{-1/2} factors, -1 once a measurement annihilates the state
    for (int r = 0; r < d.nstabs; r++) {
        const int res = measure_pauli<NR>(st, d.pm[r], d.pz[r], d.px[r]);
        if (res < 0) e |= kErrRange;
        if (res <= 0) {
            c = -1;
            break;
        }
        if (res == 2) c++;
    }
    if (lane_id() == 0) d.code[a] = c;
    if (c < 0) dead_root(J, i);
    else store_root<NR>(J, i, st, sh);
    e = (int)__reduce_or_sync(kFull, (unsigned)e);
    if (e && lane_id() == 0) atomicOr(err, e);
}

// ---------------------------------------------------------------- stages
template <class W>
struct StageRows;
template <>
struct StageRows<uint32_t> {
    using Rows = Rows32;
    static constexpr int words = 1;
    __device__ __forceinline__ static Rows at(uint32_t* smem, int, int tid) { return Rows{smem + 4 * tid, kTreeStageThreads}; }
};
template <>
struct StageRows<uint64_t> {
    using Rows = Rows64;
    static constexpr int words = 2;
    __device__ __forceinline__ static Rows at(uint32_t* smem, int units, int tid) {
        return Rows{smem + 4 * tid, smem + (size_t)units * 4 * kTreeStageThreads + 4 * tid, kTreeStageThreads};
    }
};

// two words of a plane, for two adjacent nodes (counts are even, so they are aligned)
__device__ __forceinline__ void store_two(uint32_t* plane, uint32_t at, uint32_t a, uint32_t b) {
    *reinterpret_cast<uint2*>(plane + at) = make_uint2(a, b);
}

// One thread per pair of siblings (nodes 2 i and 2 i + 1, whose messages differ in
// the lowest bit).  ALU-bound (90% of the pipe): a pair of 28 -> 15 vertices runs
// about 8 steps over some 20 rows.  The parent's rows are copied to shared memory
// twice, so a lane moves on from one sibling to the other without a load: a stage
// from 28 to 15 vertices took 985 us for 14.3e6 nodes with a node per thread, 576
// with a pair.
template <class W, bool PAIRS>
__global__ void __launch_bounds__(kTreeStageThreads) k_tree_stage(const TreeStageJob* jobs, int njobs) {
    extern __shared__ __align__(16) uint32_t smem[];
    const TreeStageJob& J = job_of(jobs, njobs, blockIdx.x);
    const int mp = J.mp, mc = J.mc, sub = J.sub;
    const int units = (mp + 3) / 4;
    const size_t copy = (size_t)units * 4 * kTreeStageThreads * StageRows<W>::words;  // words of a copy
    const auto rows = StageRows<W>::at(smem, units, threadIdx.x);
    const bool both = sub > 0;  // a stage of no message bits (a code without rows) has no siblings
    const uint32_t pairs = (uint32_t)(both ? J.count >> 1 : J.count);
    const uint32_t i = (uint32_t)((int64_t)blockIdx.x - J.block0) * kTreeStageThreads + threadIdx.x;
    const bool valid = i < pairs;
    const uint32_t pi = valid ? (both ? i >> (sub - 1) : i) : 0u;  // the parent
    const int64_t np = J.in_count;
    Work<W> a;
    W x;
    uint32_t status;
    {
        const uint32_t* p = J.in + (int64_t)node_row_words(mp) * np;  // uniform plane bases, 32-bit lane offset
        if constexpr (sizeof(W) == 8) {
            a.s.d1 = (W)p[pi] | ((W)(p + np)[pi] << 32);
            a.s.d2 = (W)(p + 2 * np)[pi] | ((W)(p + 3 * np)[pi] << 32);
            a.s.h = (W)(p + 4 * np)[pi] | ((W)(p + 5 * np)[pi] << 32);
            x = (W)(p + 6 * np)[pi] | ((W)(p + 7 * np)[pi] << 32);
            status = (p + 8 * np)[pi];
        } else if (mp > 16) {
            a.s.d1 = p[pi];
            a.s.d2 = (p + np)[pi];
            a.s.h = (p + 2 * np)[pi];
            x = (p + 3 * np)[pi];
            status = (p + 4 * np)[pi];
        } else {
            const uint32_t dd = p[pi], hx = (p + np)[pi];
            a.s.d1 = dd & 0xFFFFu;
            a.s.d2 = dd >> 16;
            a.s.h = hx & 0xFFFFu;
            x = hx >> 16;
            status = (p + 2 * np)[pi];
        }
    }
    const bool alive = valid && !(status & 0x80000000u);
    a.s.q = (int)(status & 7u);
    a.s.iso = (int)((status >> 8) & 0xFFu);
    a.s.dead = alive ? 0 : 1;
    for (int b = 1; b < sub; b++)
        if ((i >> (b - 1)) & 1u) x ^= (W)J.gen[b];
    // rows into shared memory, four to a unit (a dead parent's rows were never written)
    for (int u = 0; u < units; u++) {
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int r = 4 * u + q;
            lo[q] = hi[q] = 0u;
            if (r < mp && alive) {
                if constexpr (sizeof(W) == 8) {
                    lo[q] = (J.in + (int64_t)(2 * r) * np)[pi];
                    hi[q] = (J.in + (int64_t)(2 * r + 1) * np)[pi];
                } else if (mp > 16) {
                    lo[q] = (J.in + (int64_t)r * np)[pi];
                } else {
                    const uint32_t v = (J.in + (int64_t)(r >> 1) * np)[pi];
                    lo[q] = (r & 1) ? v >> 16 : v & 0xFFFFu;
                }
            }
        }
        auto second = rows;
        second.shift(copy);
        if constexpr (sizeof(W) == 8) {
            *rows.unit_lo(u) = *second.unit_lo(u) = U32x4{lo[0], lo[1], lo[2], lo[3]};
            *rows.unit_hi(u) = *second.unit_hi(u) = U32x4{hi[0], hi[1], hi[2], hi[3]};
        } else {
            *rows.unit(u) = *second.unit(u) = U32x4{lo[0], lo[1], lo[2], lo[3]};
        }
    }
    const W pm = wlow<W>(mp), cm = wlow<W>(mc), block = pm & ~cm;
    Work<W> c = a;
    const W xc = both ? x ^ (W)J.gen[0] : x;
    a.sum = alive ? (x ^ a.s.h) & block : (W)0;  // the others of the block are set to 0
    c.sum = (alive && both) ? (xc ^ c.s.h) & block : (W)0;
    auto two = rows;
    two.shift(copy);
    if constexpr (PAIRS) {
        const int hi = J.paired < mp ? J.paired : mp;
        const W pm2 = wlow<W>(hi) & block;  // the block's paired positions
        a.sum &= ~pm2;
        c.sum &= ~pm2;
        a.live = cm | a.sum | pm2;
        c.live = cm | c.sum | pm2;
        join_pairs<W>(rows, a, x, mc, hi, alive);
        join_pairs<W>(two, c, xc, mc, hi, alive && both);
    } else {
        a.live = cm | a.sum;
        c.live = cm | c.sum;
    }
    contract_pair(rows, copy, a, c, mc);
    if (!valid) return;
    const uint32_t sa = pack_status(a.s.q, a.s.iso, a.s.dead), sc = pack_status(c.s.q, c.s.iso, c.s.dead);
    uint32_t* const out = J.out;
    const int64_t nc = J.count;
    if (!both) {  // (a code without rows: one node per state)
        for (int r = 0; r < mc; r++) store_row(out, nc, i, mc, r, (uint64_t)(rows.get(r) & cm));
        store_scalars(out, nc, i, mc, (uint64_t)(a.s.d1 & cm), (uint64_t)(a.s.d2 & cm), (uint64_t)(a.s.h & cm),
                      (uint64_t)(x & cm), sa);
        return;
    }
    const uint32_t at = 2u * i;
    if (!(a.s.dead && c.s.dead)) {
        if (mc > 32) {
            for (int r = 0; r < mc; r++) {
                const uint64_t v = (uint64_t)(rows.get(r) & cm), w = (uint64_t)(two.get(r) & cm);
                store_two(out + (int64_t)(2 * r) * nc, at, (uint32_t)v, (uint32_t)w);
                store_two(out + (int64_t)(2 * r + 1) * nc, at, (uint32_t)(v >> 32), (uint32_t)(w >> 32));
            }
        } else if (mc > 16) {
            for (int r = 0; r < mc; r++)
                store_two(out + (int64_t)r * nc, at, (uint32_t)(rows.get(r) & cm), (uint32_t)(two.get(r) & cm));
        } else {
            for (int r = 0; r < mc; r += 2) {  // row mc, if mc is odd, lies within the parent's and is cleared by cm's bits
                const uint32_t hi = r + 1 < mc ? 0xFFFFFFFFu : 0xFFFFu;
                const uint32_t v = (uint32_t)(rows.get(r) & cm) | ((uint32_t)(rows.get(r + 1 < mc ? r + 1 : r) & cm) << 16);
                const uint32_t w = (uint32_t)(two.get(r) & cm) | ((uint32_t)(two.get(r + 1 < mc ? r + 1 : r) & cm) << 16);
                store_two(out + (int64_t)(r >> 1) * nc, at, v & hi, w & hi);
            }
        }
    }
    uint32_t* p = out + (int64_t)node_row_words(mc) * nc;
    const W xa = x & cm, xb = xc & cm;
    if (mc > 32) {
        const W va[4] = {a.s.d1 & cm, a.s.d2 & cm, a.s.h & cm, xa}, vc[4] = {c.s.d1 & cm, c.s.d2 & cm, c.s.h & cm, xb};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            store_two(p + (int64_t)(2 * q) * nc, at, (uint32_t)va[q], (uint32_t)vc[q]);
            store_two(p + (int64_t)(2 * q + 1) * nc, at, (uint32_t)((uint64_t)va[q] >> 32),
                      (uint32_t)((uint64_t)vc[q] >> 32));
        }
        store_two(p + 8 * nc, at, sa, sc);
    } else if (mc > 16) {
        store_two(p, at, (uint32_t)(a.s.d1 & cm), (uint32_t)(c.s.d1 & cm));
        store_two(p + nc, at, (uint32_t)(a.s.d2 & cm), (uint32_t)(c.s.d2 & cm));
        store_two(p + 2 * nc, at, (uint32_t)(a.s.h & cm), (uint32_t)(c.s.h & cm));
        store_two(p + 3 * nc, at, (uint32_t)xa, (uint32_t)xb);
        store_two(p + 4 * nc, at, sa, sc);
    } else {
        store_two(p, at, (uint32_t)(a.s.d1 & cm) | ((uint32_t)(a.s.d2 & cm) << 16),
                  (uint32_t)(c.s.d1 & cm) | ((uint32_t)(c.s.d2 & cm) << 16));
        store_two(p + nc, at, (uint32_t)(a.s.h & cm) | ((uint32_t)xa << 16), (uint32_t)(c.s.h & cm) | ((uint32_t)xb << 16));
        store_two(p + 2 * nc, at, sa, sc);
    }
}

// ---------------------------------------------------------------- leaves
__device__ __forceinline__ int64_t shfl_xor_i64(int64_t v, int m) { return (int64_t)shfl_xor64((uint64_t)v, m); }

// ALU-bound (80% of the pipe; the counts run on the XU pipe).  Six blocks per SM:
// 80 registers without spills; with 128 registers (four blocks) t = 40 is 1.5%
// slower and t = 48 3.5%, with 72 (seven) within 0.4%.
// ROWS: exactProjector rows, PAIRS: terms of |H^t> (TreeLeafJob).
template <int WORDS, bool ROWS, bool PAIRS>
__global__ void __launch_bounds__(kTreeLeafThreads, ROWS ? 4 : 6) k_tree_leaf(const TreeLeafJob* jobs, int njobs) {
    __shared__ uint32_t lin[32], sub[32];
    __shared__ __align__(16) uint32_t wrows[2 * 8 * kTreeLeafThreads];
    __shared__ int64_t red[kTreeLeafThreads / 32][4];
    const TreeLeafJob& J = job_of(jobs, njobs, blockIdx.x);
    const int tid = threadIdx.x;
    if (tid < 32) {
        lin[tid] = linear_word((uint32_t)tid);
        sub[tid] = subset_word((uint32_t)tid);
    }
    __syncthreads();
    const int m = J.m, tv = J.tv;
    const int64_t ti = ((int64_t)blockIdx.x - J.block0) * kTreeLeafThreads + tid;  // thread of the job
    const size_t copy = 8 * kTreeLeafThreads;
    const Rows16 rows{wrows + 4 * tid, kTreeLeafThreads}, rows2{wrows + copy + 4 * tid, kTreeLeafThreads};
    const uint32_t mm = wlow<uint32_t>(m), vm = wlow<uint32_t>(tv);
    const int64_t np = J.in_count;
    // a part's levels: table nodes, and leaves of a table (fewer than 2^tj if the part is smaller)
    const int below = J.je - J.split, tj = below < J.tj ? below : J.tj, nsub = 1 << (below - tj);
    int64_t z[4] = {0, 0, 0, 0};
    for (int rep = 0; rep < J.reps; rep++) {
        const int64_t part = ((int64_t)blockIdx.x - J.block0) * kTreeLeafThreads * J.reps + rep * kTreeLeafThreads + tid;
        const bool valid = ti < J.threads;
        const int64_t node = valid ? part >> J.split : 0;
        const uint32_t* const p = J.in + (int64_t)((m + 1) / 2) * np + node;
        const uint32_t status = p[2 * np];
        const bool alive = valid && !(status & 0x80000000u);
        if (!uniform_any(alive)) continue;
        uint32_t w[8];
#pragma unroll
        for (int q = 0; q < 8; q++) w[q] = (2 * q < m && alive) ? J.in[(int64_t)q * np + node] : 0u;
        const uint32_t dd = p[0], hx = p[np];
        const int iso0 = (int)((status >> 8) & 0xFFu);
        uint32_t x = hx >> 16;
        for (int b = 0; b < J.split; b++)
            if ((part >> b) & 1) x ^= J.gen[J.je - J.split + b];
        int64_t state = 0, row = 0, term = 0;  // ROWS: the state, its row, and the term index so far
        if constexpr (ROWS) {
            state = node >> J.nodes_log2;
            row = J.row0 + state;
            for (int b = 0; b < J.nodes_log2; b++)
                if ((node >> b) & 1) term ^= (int64_t)J.term[J.je + b];
            for (int b = 0; b < J.split; b++)
                if ((part >> b) & 1) term ^= (int64_t)J.term[J.je - J.split + b];
        }
        int y[4] = {0, 0, 0, 0};  // this part's sum, relative to 2^{iso0 / 2}
        // table nodes two at a time, in Gray code order
        for (int s = 0; s < nsub; s += 2) {
            if (s) x ^= J.gen[tj + __ffs(s) - 1];
            if constexpr (ROWS)
                if (s) term ^= (int64_t)J.term[tj + __ffs(s) - 1];
            const uint32_t x2 = nsub > 1 ? x ^ J.gen[tj] : x;
            Work<uint32_t> wa, wb;
            wa.s = Node<uint32_t>{dd & 0xFFFFu, dd >> 16, hx & 0xFFFFu, (int)(status & 7u), 0, 0};
            wb = wa;
            if (m > tv) {
                *rows.unit(0) = *rows2.unit(0) = U32x4{w[0], w[1], w[2], w[3]};
                if (m > 8) *rows.unit(1) = *rows2.unit(1) = U32x4{w[4], w[5], w[6], w[7]};
                if constexpr (PAIRS) {  // every position below paired is a pair's, a single qubit above them
                    const uint32_t pm = wlow<uint32_t>(m & ~1);
                    wa.sum = alive ? (x ^ wa.s.h) & mm & ~pm : 0u;
                    wb.sum = alive && nsub > 1 ? (x2 ^ wb.s.h) & mm & ~pm : 0u;
                    wa.live = pm | wa.sum;
                    wb.live = pm | wb.sum;
                    join_pairs<uint32_t>(rows, wa, x, 0, m & ~1, alive);
                    join_pairs<uint32_t>(rows2, wb, x2, 0, m & ~1, alive && nsub > 1);
                } else {
                    wa.sum = alive ? (x ^ wa.s.h) & mm & ~vm : 0u;
                    wb.sum = alive && nsub > 1 ? (x2 ^ wb.s.h) & mm & ~vm : 0u;
                    wa.live = vm | wa.sum;
                    wb.live = vm | wb.sum;
                }
                sum_out_pair<uint32_t>(rows, copy, wa, wb, ~0u);
            }
#pragma unroll 1
            for (int e = 0; e < 2; e++) {
                if (e && nsub == 1) break;  // uniform
                Node<uint32_t> nd;
                nd.d1 = e ? wb.s.d1 : wa.s.d1;
                nd.d2 = e ? wb.s.d2 : wa.s.d2;
                nd.h = e ? wb.s.h : wa.s.h;
                nd.q = e ? wb.s.q : wa.s.q;
                nd.iso = e ? wb.s.iso : wa.s.iso;
                nd.dead = e ? wb.s.dead : wa.s.dead;
                U32x4 u = U32x4{w[0], w[1], w[2], w[3]};
                if (m > tv) u = e ? *rows2.unit(0) : *rows.unit(0);
                const uint32_t r[kTableVars] = {u.a, u.a >> 16, u.b, u.b >> 16, u.c, u.c >> 16, u.d, u.d >> 16};
                const uint32_t d1 = nd.d1 & vm;
                Table<WORDS> tb;
                build_table<WORDS>(r, d1, nd.d2 & vm, lin, tb);
                int evr = 0, evi = 0, odr = 0, odi = 0;
                uint32_t S = ((e ? x2 : x) ^ nd.h) & vm;
                // (evr + i evi) + sqrt2 (odr + i odi), times w^q 2^{iso / 2}
                auto node_sum = [&](int (&v)[4]) {
                    v[0] = evr;
                    v[1] = odr + odi;
                    v[2] = evi;
                    v[3] = odi - odr;
                    times_omega(v, nd.q);
                    if (nd.iso & 1) times_sqrt2(v);
#pragma unroll
                    for (int q = 0; q < 4; q++) v[q] <<= nd.iso >> 1;
                };
                int v[4];
                if constexpr (ROWS) {
                    int64_t j = e ? term ^ (int64_t)J.term[tj] : term;
                    for (int l = 0; l < (1 << tj); l++) {
                        if (l) {
                            S ^= J.gen[__ffs(l) - 1] & vm;
                            j ^= (int64_t)J.term[__ffs(l) - 1];
                        }
                        if (j > row) table_leaf<WORDS>(tb, S, d1, tv, sub, evr, evi, odr, odi);
                        if (j == row && alive) {  // one leaf of a state
                            const int keep[4] = {evr, evi, odr, odi};
                            evr = evi = odr = odi = 0;
                            if (!nd.dead) table_leaf<WORDS>(tb, S, d1, tv, sub, evr, evi, odr, odi);
                            node_sum(v);
                            int64_t dz[4];
                            if (iso0 & 1) times_sqrt2(v);
                            for (int q = 0; q < 4; q++) dz[q] = (int64_t)v[q] << (iso0 >> 1);
                            if (J.shift & 1) times_sqrt2(dz);
                            for (int q = 0; q < 4; q++) J.diag[4 * state + q] = (__int128)dz[q] << (J.shift >> 1);
                            evr = keep[0];
                            evi = keep[1];
                            odr = keep[2];
                            odi = keep[3];
                        }
                    }
                } else {
                    for (int l = 0; l < (1 << tj); l++) {
                        if (l) S ^= J.gen[__ffs(l) - 1] & vm;
                        table_leaf<WORDS>(tb, S, d1, tv, sub, evr, evi, odr, odi);
                    }
                }
                if (alive && !nd.dead) {
                    node_sum(v);
#pragma unroll
                    for (int q = 0; q < 4; q++) y[q] += v[q];
                }
            }
            if (nsub > 1) {
                x = x2;
                if constexpr (ROWS) term ^= (int64_t)J.term[tj];
            }
        }
        if (iso0 & 1) times_sqrt2(y);
#pragma unroll
        for (int q = 0; q < 4; q++) z[q] += (int64_t)y[q] << (iso0 >> 1);
    }
    // sums of `group` consecutive threads (a power of two)
    const int group = J.group;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
        if (o < group) {  // uniform
#pragma unroll
            for (int q = 0; q < 4; q++) z[q] += shfl_xor_i64(z[q], o);
        }
    if (group > 32) {
        if ((tid & 31) == 0)
            for (int q = 0; q < 4; q++) red[tid >> 5][q] = z[q];
        __syncthreads();
        if (tid % group == 0)
            for (int w2 = 1; w2 < group / 32; w2++)
                for (int q = 0; q < 4; q++) z[q] += red[(tid >> 5) + w2][q];
    }
    if (tid % group == 0 && ti < J.threads) {
        if (J.shift & 1) times_sqrt2(z);
        __int128* o = J.part + 4 * (ti / group);
        for (int q = 0; q < 4; q++) o[q] = (__int128)((unsigned __int128)(__int128)z[q] << (J.shift >> 1));
    }
}

// ---------------------------------------------------------------- values
// One warp per state: the sum of its partial sums as a double.  factor[c]: the
// projection factor of c measurements that halved the norm.  *live counts the
// states that the projector left alive (0 for the others).  Without diag: out is
// singleProjectorSample's value 2^t |projfactor sum|^2 (innerprod.c:142); with it
// out and im are exactProjector's row, diag + 2 Re sum (innerprod.c:187-195), and
// live[2] counts the live rows' terms, row_terms - i for row i.
__global__ void __launch_bounds__(128) k_tree_values(const __int128* part, const __int128* diag, int64_t count,
                                                     int64_t parts, int t, const int* code, const double* factor,
                                                     double* out, double* im_out, unsigned long long* live,
                                                     int64_t row_terms) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= count) return;  // warp-uniform
    const int lane = lane_id(), q = lane & 3;
    const int c = code[i];
    __int128 z = 0;
    for (int64_t p = lane >> 2; p < parts; p += 8) z += part[4 * (i * parts + p) + q];
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) z += shfl_xor_i128(z, o);
    const __int128 d = diag && c >= 0 ? diag[4 * i + q] : 0;
    double a, b;
    warp_value(z, diag != nullptr, d, t, factor[c >= 0 ? c : 0], a, b);
    if (lane != 0) return;
    if (c >= 0) {
        atomicAdd(live, 1ull);
        if (diag) atomicAdd(live + 2, (unsigned long long)(row_terms - i));
    } else {
        a = b = 0;
    }
    if (im_out) {
        out[i] = a;
        im_out[i] = b;
    } else {
        out[i] = sample_value(a, b, t);
    }
}

// ---------------------------------------------------------------- launchers
int launch_tree_draw(const Launch& L, const TreeRootJob* jobs, int njobs, int64_t blocks, bool wide) {
    if (njobs <= 0 || blocks <= 0) return 0;
    if (blocks > 0x7fffffff) return -1;
    if (wide) k_tree_draw<2><<<(unsigned)blocks, 32 * kTreeRootWarps, 0, L.stream>>>(jobs, njobs, L.d_err);
    else k_tree_draw<1><<<(unsigned)blocks, 32 * kTreeRootWarps, 0, L.stream>>>(jobs, njobs, L.d_err);
    (*L.launches)++;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_tree_stage(const Launch& L, const TreeStageJob* jobs, int njobs, int64_t blocks, bool wide, int mmax,
                      bool pairs) {
    if (njobs <= 0 || blocks <= 0) return 0;
    if (blocks > 0x7fffffff || mmax < 1 || mmax > (wide ? 64 : 32)) return -1;
    // two copies of every lane's rows: at most 64 KB
    const size_t smem = 2 * (size_t)((mmax + 3) / 4) * 16 * kTreeStageThreads * (wide ? 2 : 1);
    const auto kernel = wide ? (pairs ? k_tree_stage<uint64_t, true> : k_tree_stage<uint64_t, false>)
                             : (pairs ? k_tree_stage<uint32_t, true> : k_tree_stage<uint32_t, false>);
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024) != cudaSuccess)
        return -1;
    kernel<<<(unsigned)blocks, kTreeStageThreads, smem, L.stream>>>(jobs, njobs);
    (*L.launches)++;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_tree_values(const Launch& L, const __int128* part, int64_t count, int64_t parts, int t, const int* code,
                       const double* factor, double* values, unsigned long long* live) {
    if (count <= 0) return 0;
    k_tree_values<<<(unsigned)((count + 3) / 4), 128, 0, L.stream>>>(part, nullptr, count, parts, t, code, factor, values,
                                                                     nullptr, live, 0);
    (*L.launches)++;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_tree_rows(const Launch& L, const __int128* part, const __int128* diag, int64_t count, int64_t parts, int t,
                     const int* code, const double* factor, double* re, double* im, unsigned long long* live,
                     int64_t row_terms) {
    if (count <= 0) return 0;
    k_tree_values<<<(unsigned)((count + 3) / 4), 128, 0, L.stream>>>(part, diag, count, parts, t, code, factor, re, im,
                                                                     live, row_terms);
    (*L.launches)++;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

namespace {
template <bool ROWS>
void (*leaf_kernel(int words, bool pairs))(const TreeLeafJob*, int) {
    if (pairs) return words == 1 ? k_tree_leaf<1, ROWS, true> : nullptr;
    return words == 1 ? k_tree_leaf<1, ROWS, false>
                      : (words == 2 ? k_tree_leaf<2, ROWS, false>
                                    : (words == 4 ? k_tree_leaf<4, ROWS, false>
                                                  : (words == 8 ? k_tree_leaf<8, ROWS, false> : nullptr)));
}
}  // namespace

int launch_tree_leaf(const Launch& L, const TreeLeafJob* jobs, int njobs, int64_t blocks, int words, bool rows,
                     bool pairs) {
    if (njobs <= 0 || blocks <= 0) return 0;
    const auto kernel = rows ? leaf_kernel<true>(words, pairs) : leaf_kernel<false>(words, pairs);
    if (blocks > 0x7fffffff || !kernel) return -1;
    kernel<<<(unsigned)blocks, kTreeLeafThreads, 0, L.stream>>>(jobs, njobs);
    (*L.launches)++;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace csim
