// csim_tree.h — jobs and launchers of the tree sum (csim_tree.cu), shared with
// the host code that builds them.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "csim_internal.h"

namespace csim {

// Every launch runs a table of jobs (one per group of states that share a
// decomposition); a job's blocks are [block0, the next job's block0).

// root nodes of `count` states: state i of the job is states[index ? index[i] : first + i]
struct TreeRootJob {
    const int32_t* index;
    int64_t first;
    const uint8_t* perm;  // position -> coordinate (t of them)
    uint32_t* out;        // node planes, one node per state
    int64_t count, block0;
    int32_t t, pad;
};

// nodes of level jc from nodes of level jp = jc + sub (`count` of them, out, < 2^32)
struct TreeStageJob {
    const uint32_t* in;   // the first parent's node, planes in_count apart
    uint32_t* out;
    const uint64_t* gen;  // generators of the levels jc .. jp - 1, sub of them
    int64_t count, in_count, block0;
    int32_t mp, mc, sub, pad;
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
};

// How k_tree_draw makes its states (k_random_states, k_project): state a of the
// call is state id + a of Philox stream `seed` (mode 0) or replays words
// [offsets[a], offsets[a + 1]) (mode 1); code[a] as k_project writes it
struct TreeDraw {
    int32_t mode, nstabs;  // mode 2: the words are raw (csim_rng.cuh)
    uint64_t seed, id;
    const uint32_t* words;
    const int64_t* offsets;
    const double* cum;
    const int* pm;
    const uint64_t *pz, *px;
    int* code;
};

constexpr int kTreeRootWarps = 4;      // states per root block
constexpr int kTreeStageThreads = 64;
constexpr int kTreeLeafThreads = 128;

int launch_tree_root(const Launch& L, const TreeRootJob* jobs, int njobs, int64_t blocks, const GState* states,
                     const int* code);
int launch_tree_draw(const Launch& L, const TreeRootJob* jobs, int njobs, int64_t blocks, int t, const TreeDraw& d);
// wide: the jobs' parents have more than 32 vertices (two words per row); mmax: the largest mp
int launch_tree_stage(const Launch& L, const TreeStageJob* jobs, int njobs, int64_t blocks, bool wide, int mmax);
// words: the jobs' table words (tree::table_words(tv))
int launch_tree_leaf(const Launch& L, const TreeLeafJob* jobs, int njobs, int64_t blocks, int words);

// values[i] of `count` states from `parts` partial sums each; factor: 65 doubles; *live is added to
int launch_tree_values(const Launch& L, const __int128* part, int64_t count, int64_t parts, int t, const int* code,
                       const double* factor, double* values, unsigned long long* live);

}  // namespace csim
