// csim_tree.h — jobs and launchers of the tree sum (csim_tree.cu), shared with
// the host code that builds them.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "csim_internal.h"

namespace csim {

// Every launch runs a table of jobs (one per group of states that share a
// decomposition); a job's blocks are [block0, the next job's block0).

// How k_tree_draw makes states (k_random_states, k_project): state a is state id + a
// of Philox stream `seed` (mode 0) or replays words [offsets[a], offsets[a + 1])
// (mode 1: rand() values, 2: raw words, csim_rng.cuh).  Mode 3: exactProjector's term states,
// state a is term id + a of the k-row code `words64` or (k < 0) of |H^t>.  code[a]
// as k_project writes it.
struct TreeDraw {
    int32_t mode, nstabs;
    uint64_t seed, id;
    const uint32_t* words;
    const int64_t* offsets;
    const double* cum;
    const int* pm;
    const uint64_t *pz, *px;
    int* code;
    const uint64_t* words64;
    int32_t k, pad;
};

// root nodes of `count` trees: tree i of the job is number first + i, 2^slice for each state of draw
struct TreeRootJob {
    TreeDraw draw;
    int64_t first;
    const uint8_t* perm;  // position -> coordinate (t of them)
    const uint64_t* gen;  // the `slice` generators whose sum a tree's number chooses
    uint32_t* out;        // node planes, one node per tree
    int64_t count, block0;
    uint64_t x0;          // the X of a state's first root
    int32_t t, slice;
};

// nodes of level jc from nodes of level jp = jc + sub (`count` of them, out, < 2^32)
struct TreeStageJob {
    const uint32_t* in;   // the first parent's node, planes in_count apart
    uint32_t* out;
    const uint64_t* gen;  // generators of the levels jc .. jp - 1, sub of them
    int64_t count, in_count, block0;
    int32_t mp, mc, sub;
    int32_t paired;       // terms of |H^t>: positions below this are pairs (join_pairs)
};

// sums below the nodes of level je (m <= 16 vertices).  A part is 2^-split of a
// node's leaves (split <= je); a block takes `reps` parts per thread, 128 consecutive parts
// at a time; a partial sum covers `group` threads.
struct TreeLeafJob {
    const uint32_t* in;   // the first node, planes in_count apart
    __int128* part;       // 4 int128 per partial sum
    int64_t in_count;
    int64_t threads, block0;
    int32_t m, je, tv, tj;
    int32_t split, reps, group, shift;  // sums are scaled by 2^{shift / 2}
    uint16_t gen[16];     // generators of the levels below je, positions < m
    // exactProjector rows: state a is row row0 + a; only its terms j > row are summed, term
    // j == row is written to diag + 4 a.  The job's first node is number node0, 2^nodes_log2 for
    // each state
    const uint64_t* term; // the generators' parts of the term index, all levels
    __int128* diag;
    int64_t row0, node0;
    int32_t nodes_log2, pad;
};

constexpr int kTreeRootWarps = 4;      // states per root block
// a warp: with rows above 32 vertices shared memory limits what an SM holds, and blocks of 64 threads are
// 1 to 1.6% slower (t = 57 and 64; up to t = 48 within 0.5%)
constexpr int kTreeStageThreads = 32;
constexpr int kTreeLeafThreads = 128;

// wide: the jobs' states have more than 32 qubits
int launch_tree_draw(const Launch& L, const TreeRootJob* jobs, int njobs, int64_t blocks, bool wide);
// planes: the jobs' parents' byte planes (tree::row_planes(mp)); mmax: the largest mp
int launch_tree_stage(const Launch& L, const TreeStageJob* jobs, int njobs, int64_t blocks, int planes, int mmax,
                      bool pairs);
// words: the jobs' table words (tree::table_words(tv)); rows: exactProjector rows; pairs: terms of |H^t> (one word)
int launch_tree_leaf(const Launch& L, const TreeLeafJob* jobs, int njobs, int64_t blocks, int words, bool rows,
                     bool pairs);

// values[i] of `count` states from `parts` partial sums each; factor: 65 doubles; *live is added to,
// the low word of live[1] becomes the device error word
int launch_tree_values(const Launch& L, const __int128* part, int64_t count, int64_t parts, int t, const int* code,
                       const double* factor, double* values, unsigned long long* live);
// the rows' values of exactProjector: re[i] + i im[i] = factor (diag + 2 Re sum of the parts);
// row_terms - i of each live row i is added to live[2]
int launch_tree_rows(const Launch& L, const __int128* part, const __int128* diag, int64_t count, int64_t parts, int t,
                     const int* code, const double* factor, double* re, double* im, unsigned long long* live,
                     int64_t row_terms);

}  // namespace csim
