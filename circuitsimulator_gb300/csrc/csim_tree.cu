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
template <class W>
__device__ __forceinline__ W permute_bits(W v, const unsigned char* perm, int t) {
    W r = 0;
    for (int i = 0; i < t; i++) r |= ((v >> perm[i]) & (W)1) << i;
    return r;
}

// vector v of node i among `count` nodes, tail u, the status word of m > 16
__device__ __forceinline__ uint32_t* vector_at(uint32_t* base, int64_t count, int v, uint32_t i) {
    return base + 4 * ((int64_t)v * count + i);
}
__device__ __forceinline__ uint32_t* tail_at(uint32_t* base, int64_t count, int m, int u, uint32_t i) {
    return base + 4 * node_vectors(m) * count + ((int64_t)u * count + i) * row_tail(m);
}
__device__ __forceinline__ uint32_t* status_at(uint32_t* base, int64_t count, int m, uint32_t i) {
    return base + (int64_t)(node_words(m) - 1) * count + i;
}
__device__ __forceinline__ void store_vector(uint32_t* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    *reinterpret_cast<uint4*>(p) = make_uint4(a, b, c, d);
}

// stores row `pos` of node i among `count` nodes of m vertices
__device__ __forceinline__ void store_row(uint32_t* base, int64_t count, uint32_t i, int m, int pos, uint64_t row) {
    const int pl = row_planes(m), u = pos >> 2;
    for (int k = 0; k < pl; k++) {
        uint32_t* w = pl == 2 ? vector_at(base, count, node_scalars(m) + (u >> 1), i) + 2 * (u & 1) + k
                              : (k < 4 ? vector_at(base, count, node_scalars(m) + u, i) + k
                                       : tail_at(base, count, m, u, i) + (k - 4));
        reinterpret_cast<uint8_t*>(w)[pos & 3] = (uint8_t)(row >> (8 * k));
    }
}
__device__ __forceinline__ void store_scalars(uint32_t* base, int64_t count, uint32_t i, int m, uint64_t d1, uint64_t d2,
                                              uint64_t h, uint64_t x, uint32_t status) {
    uint32_t* p = vector_at(base, count, 0, i);
    if (m > 32) {
        store_vector(p, (uint32_t)d1, (uint32_t)(d1 >> 32), (uint32_t)d2, (uint32_t)(d2 >> 32));
        store_vector(p + 4 * count, (uint32_t)h, (uint32_t)(h >> 32), (uint32_t)x, (uint32_t)(x >> 32));
        *status_at(base, count, m, i) = status;
    } else if (m > 16) {
        store_vector(p, (uint32_t)d1, (uint32_t)d2, (uint32_t)h, (uint32_t)x);
        *status_at(base, count, m, i) = status;
    } else {
        store_vector(p, (uint32_t)d1 | ((uint32_t)d2 << 16), (uint32_t)h | ((uint32_t)x << 16), status, 0u);
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
__device__ __forceinline__ void dead_root(const TreeRootJob& J, uint32_t i) {
    if (lane_id() == 0) store_scalars(J.out, J.count, i, J.t, 0, 0, 0, 0, pack_status(0, 0, 1));
}

// Node i of the job from a state held by the warp
template <int NR>
__device__ void store_root(const TreeRootJob& J, uint32_t i, const WS<NR>& st, RootShared& sh) {
    using W = RW<NR>;
    unsigned char* const piv = sh.piv[threadIdx.x >> 5];
    const int t = J.t, k = st.k;
    const W km = low_mask<NR>(k), nm = low_mask<NR>(t);
    CanonWarp<NR> w;
#pragma unroll
    for (int q = 0; q < NR; q++) {  // this lane's variables
        const bool in = row_of<NR>(q) < k;
        w.g[q] = in ? permute_bits<W>(st.G[q], sh.perm, t) : (W)0;
        w.j[q] = in ? st.J[q] & km : (W)0;
    }
    w.D1 = st.D1 & km;
    w.D2 = st.D2 & km;
    const W h = permute_bits<W>(st.h, sh.perm, t);
    canon_warp<NR>(w, k, h);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NR; q++) piv[row_of<NR>(q)] = (unsigned char)w.p[q];
    __syncwarp();
    // pivots: vertices with J and D; a non-pivot coordinate y = b + a.v is Had on a vertex
    // joined to the variables in a, with D = 4 b
    W row[NR], had[NR] = {}, bm = 0;  // rows of this lane's variables, of its coordinates
#pragma unroll
    for (int q = 0; q < NR; q++) row[q] = to_coords<W>(w.j[q], piv);
    for (W np = ~w.P & nm; np;) {  // uniform
        const int c = first_bit(np);
        np &= np - (W)1;
        bool in[2] = {};
#pragma unroll
        for (int q = 0; q < NR; q++) {
            in[q] = row_of<NR>(q) < k && ((w.g[q] >> c) & (W)1);
            if (in[q]) row[q] |= bit_of<NR>(c);
        }
        const W av = ballot_i<NR>(in[0], in[NR - 1]);
#pragma unroll
        for (int q = 0; q < NR; q++)
            if (row_of<NR>(q) == c) had[q] = av;
        if ((getbit(h, c) ^ parity(w.wv & av)) != 0) bm |= bit_of<NR>(c);
    }
#pragma unroll
    for (int q = 0; q < NR; q++) {
        const int r = row_of<NR>(q);
        if (r < k) store_row(J.out, J.count, i, t, w.p[q], row[q]);
        had[q] = to_coords<W>(had[q], piv);
        if (r < t && !getbit(w.P, r)) store_row(J.out, J.count, i, t, r, had[q]);
    }
    if (lane_id() == 0) {
        uint64_t x = J.x0;
        for (int b = 0; b < J.slice; b++)
            if (((J.first + i) >> b) & 1) x ^= J.gen[b];
        store_scalars(J.out, J.count, i, t, to_coords<W>(w.D1, piv), to_coords<W>(w.D2, piv) | bm, ~w.P & nm, x,
                      pack_status(st.Q + w.dq, 0, 0));
    }
}

}  // namespace

// Drawing, projecting and the graph form in one launch, the state never leaving the
// warp's registers.  Bound by the latency of a warp's serial steps: 1024 states of
// 40 qubits take 44 us; k_random_states, k_project and a kernel for the graph form
// took 11 + 29 + 26 us.  NR = 1: jobs of up to 32 qubits, 2: the others.  Many states
// are bound by the instructions: 64,400 of up to 23 qubits 347 us (NR = 1).
template <int NR>
__global__ void __launch_bounds__(32 * kTreeRootWarps) k_tree_draw(const TreeRootJob* jobs, int njobs, int* err) {
    __shared__ RootShared sh;
    const TreeRootJob& J = job_of(jobs, njobs, blockIdx.x);
    if ((int)threadIdx.x < J.t) sh.perm[threadIdx.x] = J.perm[threadIdx.x];
    __syncthreads();
    const int64_t i = ((int64_t)blockIdx.x - J.block0) * kTreeRootWarps + (threadIdx.x >> 5);
    if (i >= J.count) return;  // warp-uniform
    const TreeDraw& d = J.draw;
    const int64_t a = (J.first + i) >> J.slice;
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
    if (c < 0) dead_root(J, (uint32_t)i);
    else store_root<NR>(J, (uint32_t)i, st, sh);
    e = (int)__reduce_or_sync(kFull, (unsigned)e);
    if (e && lane_id() == 0) atomicOr(err, e);
}

// ---------------------------------------------------------------- stages
// n vectors of V from the planes `from`, from + step, ... to two copies in shared memory
// (`copy` words apart), the vectors of one `stride` words apart: through registers, eight
// loads in flight
template <class V>
__device__ __forceinline__ void copy_twice(uint32_t* to, size_t copy, int stride, const uint32_t* from, int64_t step, int n) {
    for (int u = 0; u < n; u += 8) {
        V v[8];
#pragma unroll
        for (int b = 0; b < 8; b++)
            if (u + b < n) v[b] = *reinterpret_cast<const V*>(from + b * step);
#pragma unroll
        for (int b = 0; b < 8; b++)
            if (u + b < n) {
                *reinterpret_cast<V*>(to + b * stride) = v[b];
                *reinterpret_cast<V*>(to + copy + b * stride) = v[b];
            }
        from += 8 * step;
        to += 8 * stride;
    }
}
// The same past the registers, all in flight.  Rows from 33 vertices up: at t = 64 (2^14
// terms) their stages are 2 to 10% faster so, where few blocks fit an SM and a warp reads
// many parents; narrower rows are as fast or slower (a stage from 32 vertices whose warps
// read one parent each: 80 us, 60 through registers).
template <int BYTES>
__device__ __forceinline__ void copy_async_twice(uint32_t* to, size_t copy, int stride, const uint32_t* from, int64_t step,
                                                 int n) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(to);
    const uint32_t second = (uint32_t)(4 * copy);
    for (int u = 0; u < n; u++) {
        asm volatile("cp.async.ca.shared.global [%0], [%2], %3;\n\tcp.async.ca.shared.global [%1], [%2], %3;" ::"r"(a),
                     "r"(a + second), "l"(from), "n"(BYTES)
                     : "memory");
        from += step;
        a += 4 * (uint32_t)stride;
    }
}

// A node's rows (of `m` vertices, from rows of PL planes and `units` units) and scalars
template <int PL, class W>
__device__ __forceinline__ void store_node(uint32_t* out, int64_t count, uint32_t i, int m, const Rows<PL>& rows, int units,
                                           const Node<W>& s, W x) {
    const W cm = wlow<W>(m);
    const uint32_t status = pack_status(s.q, s.iso, s.dead);
    store_scalars(out, count, i, m, (uint64_t)(s.d1 & cm), (uint64_t)(s.d2 & cm), (uint64_t)(s.h & cm), (uint64_t)(x & cm),
                  status);
    if (s.dead) return;
    const int cu = row_units(m);
    uint32_t* p = vector_at(out, count, node_scalars(m), i);
    if (PL > 2 && m <= 16) {  // two units to a vector
        for (int u = 0; u < cu; u += 2) {
            const U32x4 a = *rows.chunk(u), b = *rows.chunk(u + 1 < units ? u + 1 : u);
            store_vector(p, a.a, a.b, b.a, b.b);
            p += 4 * count;
        }
        return;
    }
    const int n = PL == 2 ? Rows<2>::chunks(cu) : cu;
#pragma unroll 4
    for (int u = 0; u < n; u++) {
        const U32x4 v = *rows.chunk(u);
        store_vector(p, v.a, v.b, v.c, v.d);
        p += 4 * count;
    }
    if constexpr (PL > 4) {
        const int tw = row_tail(m);
        if (tw == 0) return;
        p = tail_at(out, count, m, 0, i);
        for (int u = 0; u < cu; u++) {
            const U32x4 v = rows.get_tail(u);
            if (tw == 1) *p = v.a;
            else if (tw == 2) *reinterpret_cast<uint2*>(p) = make_uint2(v.a, v.b);
            else if (tw == 4) store_vector(p, v.a, v.b, v.c, v.d);
            else {
                p[0] = v.a;
                p[1] = v.b;
                p[2] = v.c;
            }
            p += tw * count;
        }
    }
}

// One thread per pair of siblings (nodes 2 i and 2 i + 1, whose messages differ in
// the lowest bit).  The parent's rows are copied to shared memory twice, so a lane
// moves on from one sibling to the other without a load: a stage from 28 to 15
// vertices took 985 us for 14.3e6 nodes with a node per thread, 576 with a pair.
// Up to 32 vertices ALU-bound (75 to 86% of the pipe), above it by the latency of few
// resident warps: shared memory holds 6 to 18 (6 at 64 vertices, 12 at 48).
// Nodes move as 16-byte vectors and several loads at a time: with a load per word and
// no more than four in flight, rows of 64, 48 and 40 vertices took 39, 213 and 191 us
// (300 states of 64 qubits, 2^14 terms), now 24, 98 and 85.
template <int PL, bool PAIRS>
__global__ void __launch_bounds__(kTreeStageThreads) k_tree_stage(const TreeStageJob* jobs, int njobs) {
    using W = typename RowWord<PL>::type;
    extern __shared__ __align__(16) uint32_t smem[];
    const TreeStageJob& J = job_of(jobs, njobs, blockIdx.x);
    const int mp = J.mp, mc = J.mc, sub = J.sub;
    const int units = row_units(mp);
    const size_t copy = Rows<PL>::words(units, kTreeStageThreads);
    const Rows<PL> rows = Rows<PL>::at(smem, threadIdx.x, units, kTreeStageThreads);
    Rows<PL> two = rows;
    two.shift(copy);
    const bool both = sub > 0;  // a stage of no message bits (a code without rows) has no siblings
    const uint32_t pairs = (uint32_t)(both ? J.count >> 1 : J.count);
    const uint32_t i = (uint32_t)((int64_t)blockIdx.x - J.block0) * kTreeStageThreads + threadIdx.x;
    const bool valid = i < pairs;
    const uint32_t pi = valid ? (both ? i >> (sub - 1) : i) : 0u;  // the parent
    const int64_t np = J.in_count;
    // rows into shared memory, two copies (a dead parent's were never written: nothing uses them)
    const uint32_t* const vectors = J.in + 4 * ((int64_t)node_scalars(mp) * np + pi);
    if constexpr (PL <= 4) {
        copy_twice<uint4>(rows.p, copy, 4 * kTreeStageThreads, vectors, 4 * np, Rows<PL>::chunks(units));
    } else {
        constexpr int tw = Rows<PL>::tail;
        copy_async_twice<16>(rows.p, copy, 4 * kTreeStageThreads, vectors, 4 * np, units);
        const uint32_t* const tails = J.in + 4 * node_vectors(mp) * np + (int64_t)pi * tw;
        if constexpr (tw == 3) {
            for (int j = 0; j < 3; j++)
                copy_async_twice<4>(rows.tp + j, copy, tw * kTreeStageThreads, tails + j, tw * np, units);
        } else {
            copy_async_twice<4 * tw>(rows.tp, copy, tw * kTreeStageThreads, tails, tw * np, units);
        }
    }
    Work<W> a;
    W x;
    uint32_t status;
    {
        const uint4 s0 = *reinterpret_cast<const uint4*>(J.in + 4 * (int64_t)pi);
        if constexpr (sizeof(W) == 8) {
            const uint4 s1 = *reinterpret_cast<const uint4*>(J.in + 4 * (np + pi));
            a.s.d1 = (W)s0.x | ((W)s0.y << 32);
            a.s.d2 = (W)s0.z | ((W)s0.w << 32);
            a.s.h = (W)s1.x | ((W)s1.y << 32);
            x = (W)s1.z | ((W)s1.w << 32);
        } else if (PL > 2) {
            a.s.d1 = s0.x;
            a.s.d2 = s0.y;
            a.s.h = s0.z;
            x = s0.w;
        } else {
            a.s.d1 = s0.x & 0xFFFFu;
            a.s.d2 = s0.x >> 16;
            a.s.h = s0.y & 0xFFFFu;
            x = s0.y >> 16;
        }
        status = PL > 2 ? J.in[(int64_t)(node_words(mp) - 1) * np + pi] : s0.z;
    }
    const bool alive = valid && !(status & 0x80000000u);
    a.s.q = (int)(status & 7u);
    a.s.iso = (int)((status >> 8) & 0xFFu);
    a.s.dead = alive ? 0 : 1;
    for (int b = 1; b < sub; b++)
        if ((i >> (b - 1)) & 1u) x ^= (W)J.gen[b];
    if constexpr (PL > 4) asm volatile("cp.async.wait_all;" ::: "memory");  // a lane reads only what it copied itself
    const W pm = wlow<W>(mp), cm = wlow<W>(mc), block = pm & ~cm;
    Work<W> c = a;
    const W xc = both ? x ^ (W)J.gen[0] : x;
    a.sum = alive ? (x ^ a.s.h) & block : (W)0;  // the others of the block are set to 0
    c.sum = (alive && both) ? (xc ^ c.s.h) & block : (W)0;
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
    contract_pair<PL>(rows, copy, a, c, mc);
    if (!valid) return;
    store_node<PL, W>(J.out, J.count, both ? 2u * i : i, mc, rows, units, a.s, x);
    if (both) store_node<PL, W>(J.out, J.count, 2u * i + 1u, mc, two, units, c.s, xc);
}

// ---------------------------------------------------------------- leaves
__device__ __forceinline__ int64_t shfl_xor_i64(int64_t v, int m) { return (int64_t)shfl_xor64((uint64_t)v, m); }

// ALU-bound (87% of the pipe at t = 40; the counts run on the XU pipe).  Six blocks per SM:
// 80 registers; with 128 registers (four blocks) t = 40 is 1.5% slower and t = 48 3.5%, with
// 72 (seven) within 0.4%.  With ROWS 24 light queries take 2.98 ms with four, 2.93 with five
// and 2.90 with six, although tables of eight words then spill some registers.
// ROWS: exactProjector rows, PAIRS: terms of |H^t> (TreeLeafJob).
template <int WORDS, bool ROWS, bool PAIRS>
__global__ void __launch_bounds__(kTreeLeafThreads, 6) k_tree_leaf(const TreeLeafJob* jobs, int njobs) {
    __shared__ TableWords words;
    __shared__ uint32_t gen_s[16], term_s[ROWS ? 16 : 1];  // the levels' generators and their parts of the term index
    __shared__ __align__(16) uint32_t wrows[2 * 8 * kTreeLeafThreads];
    __shared__ int64_t red[kTreeLeafThreads / 32][4];
    const TreeLeafJob& J = job_of(jobs, njobs, blockIdx.x);
    const int tid = threadIdx.x;
    if (tid < 32) words.fill(tid, J.tv);
    else if (tid < 48) {
        const int b = tid - 32;
        gen_s[b] = b < J.je ? J.gen[b] : 0u;
        if constexpr (ROWS) term_s[b] = b < J.je ? (uint32_t)J.term[b] : 0u;
    }
    __syncthreads();
    const int m = J.m, tv = J.tv;
    const int64_t ti = ((int64_t)blockIdx.x - J.block0) * kTreeLeafThreads + tid;  // thread of the job
    const size_t copy = Rows<2>::words(4, kTreeLeafThreads);
    const Rows<2> rows = Rows<2>::at(wrows, tid, 4, kTreeLeafThreads), rows2 = Rows<2>::at(wrows + copy, tid, 4, kTreeLeafThreads);
    const uint32_t mm = wlow<uint32_t>(m), vm = wlow<uint32_t>(tv);
    const int64_t np = J.in_count;
    // a part's levels: table nodes, and leaves of a table (fewer than 2^tj if the part is smaller)
    const int below = J.je - J.split, tj = below < J.tj ? below : J.tj, nsub = 1 << (below - tj);
    int64_t z[4] = {0, 0, 0, 0};
    for (int rep = 0; rep < J.reps; rep++) {
        const int64_t part = ((int64_t)blockIdx.x - J.block0) * kTreeLeafThreads * J.reps + rep * kTreeLeafThreads + tid;
        const bool valid = ti < J.threads;
        const int64_t node = valid ? part >> J.split : 0;
        const uint4* const p = reinterpret_cast<const uint4*>(J.in) + node;
        const uint4 sc = *p;
        const uint32_t dd = sc.x, hx = sc.y, status = sc.z;
        const bool alive = valid && !(status & 0x80000000u);
        if (!uniform_any(alive)) continue;
        const uint4 none = make_uint4(0u, 0u, 0u, 0u);
        const uint4 w0 = alive && m > 0 ? p[np] : none, w1 = alive && m > 8 ? p[2 * np] : none;
        const int iso0 = (int)((status >> 8) & 0xFFu);
        uint32_t x = hx >> 16;
        const int split0 = J.je - J.split;  // levels from here up to je are split over threads
        for (int b = 0; b < J.split; b++)
            if ((part >> b) & 1) x ^= gen_s[split0 + b];
        int state = 0;  // ROWS: the state, its row, and the term index so far (below 2^30)
        uint32_t row = 0, term = 0;
        if constexpr (ROWS) {
            const int64_t number = J.node0 + node;
            state = (int)(number >> J.nodes_log2);
            row = (uint32_t)(J.row0 + state);
            for (int b = 0; b < J.nodes_log2; b++)
                if ((number >> b) & 1) term ^= (uint32_t)J.term[J.je + b];
            for (int b = 0; b < J.split; b++)
                if ((part >> b) & 1) term ^= term_s[split0 + b];
        }
        // this part's sum, relative to 2^{iso0 / 2}: at most 2^16 leaves of at most 2^12.  iso0 / 2 is at
        // most 24, a thread takes 8 parts and a sum 128 threads: z is at most 2^62
        int y[4] = {0, 0, 0, 0};
        // table nodes two at a time, in Gray code order
        for (int s = 0; s < nsub; s += 2) {
            if (s) x ^= gen_s[tj + __ffs(s) - 1];
            if constexpr (ROWS)
                if (s) term ^= term_s[tj + __ffs(s) - 1];
            const uint32_t x2 = nsub > 1 ? x ^ gen_s[tj] : x;
            Work<uint32_t> wa, wb;
            wa.s = Node<uint32_t>{dd & 0xFFFFu, dd >> 16, hx & 0xFFFFu, (int)(status & 7u), 0, 0};
            wb = wa;
            if (m > tv) {
                *rows.chunk(0) = *rows2.chunk(0) = U32x4{w0.x, w0.y, w0.z, w0.w};
                if (m > 8) *rows.chunk(1) = *rows2.chunk(1) = U32x4{w1.x, w1.y, w1.z, w1.w};
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
                uint32_t r0 = w0.x, r4 = w0.z;  // rows 0..3 and 4..7, a byte each
                if (m > tv) {
                    const U32x4 u = e ? *rows2.chunk(0) : *rows.chunk(0);
                    r0 = u.a;
                    r4 = u.c;
                }
                const uint32_t d1 = nd.d1 & vm;
                Table<WORDS> tb;
                build_table<WORDS>(r0, r4, d1, nd.d2 & vm, words, tb);
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
                    uint32_t j = e ? term ^ term_s[tj] : term;
                    for (int l = 0; l < (1 << tj); l++) {
                        if (l) {
                            S ^= gen_s[__ffs(l) - 1] & vm;
                            j ^= term_s[__ffs(l) - 1];
                        }
                        if (j > row) table_leaf<WORDS>(tb, S, d1, words, evr, evi, odr, odi);
                        if (j == row && alive) {  // one leaf of a state
                            const int keep[4] = {evr, evi, odr, odi};
                            evr = evi = odr = odi = 0;
                            if (!nd.dead) table_leaf<WORDS>(tb, S, d1, words, evr, evi, odr, odi);
                            node_sum(v);
                            int64_t dz[4];
                            if (iso0 & 1) times_sqrt2(v);
                            for (int q = 0; q < 4; q++) dz[q] = (int64_t)v[q] << (iso0 >> 1);
                            if (J.shift & 1) times_sqrt2(dz);
                            for (int q = 0; q < 4; q++) J.diag[4 * (int64_t)state + q] = (__int128)dz[q] << (J.shift >> 1);
                            evr = keep[0];
                            evi = keep[1];
                            odr = keep[2];
                            odi = keep[3];
                        }
                    }
                } else {
                    for (int l = 0; l < (1 << tj); l++) {
                        if (l) S ^= gen_s[__ffs(l) - 1] & vm;
                        table_leaf<WORDS>(tb, S, d1, words, evr, evi, odr, odi);
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
                if constexpr (ROWS) term ^= term_s[tj];
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
                                                     int64_t row_terms, const int* err) {
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
    if (i == 0) *(int*)(live + 1) = *err;  // of the kernels before
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

namespace {
template <bool PAIRS>
void (*stage_kernel(int planes))(const TreeStageJob*, int) {
    switch (planes) {
    case 2: return k_tree_stage<2, PAIRS>;
    case 3: return k_tree_stage<3, PAIRS>;
    case 4: return k_tree_stage<4, PAIRS>;
    case 5: return k_tree_stage<5, PAIRS>;
    case 6: return k_tree_stage<6, PAIRS>;
    case 7: return k_tree_stage<7, PAIRS>;
    case 8: return k_tree_stage<8, PAIRS>;
    default: return nullptr;
    }
}
}  // namespace

int launch_tree_stage(const Launch& L, const TreeStageJob* jobs, int njobs, int64_t blocks, int planes, int mmax,
                      bool pairs) {
    if (njobs <= 0 || blocks <= 0) return 0;
    const auto kernel = pairs ? stage_kernel<true>(planes) : stage_kernel<false>(planes);
    if (blocks > 0x7fffffff || !kernel || mmax < 1 || row_planes(mmax) != planes) return -1;
    // two copies of every lane's rows: 32 KB for rows of 64 vertices
    static_assert(2 * 4 * (4 + 4) * 16 * kTreeStageThreads <= 48 * 1024, "shared memory of a stage's block");
    const int units = row_units(mmax);
    const int chunks = planes == 2 ? Rows<2>::chunks(units) : units;
    const size_t smem = (size_t)2 * 4 * (4 * chunks + row_tail(mmax) * units) * kTreeStageThreads;
    kernel<<<(unsigned)blocks, kTreeStageThreads, smem, L.stream>>>(jobs, njobs);
    (*L.launches)++;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_tree_values(const Launch& L, const __int128* part, int64_t count, int64_t parts, int t, const int* code,
                       const double* factor, double* values, unsigned long long* live) {
    if (count <= 0) return 0;
    k_tree_values<<<(unsigned)((count + 3) / 4), 128, 0, L.stream>>>(part, nullptr, count, parts, t, code, factor, values,
                                                                     nullptr, live, 0, L.d_err);
    (*L.launches)++;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_tree_rows(const Launch& L, const __int128* part, const __int128* diag, int64_t count, int64_t parts, int t,
                     const int* code, const double* factor, double* re, double* im, unsigned long long* live,
                     int64_t row_terms) {
    if (count <= 0) return 0;
    k_tree_values<<<(unsigned)((count + 3) / 4), 128, 0, L.stream>>>(part, diag, count, parts, t, code, factor, re, im,
                                                                     live, row_terms, L.d_err);
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
