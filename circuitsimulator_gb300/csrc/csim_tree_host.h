// csim_tree_host.h — the launches of a tree sum (csim_tree.cu) over groups of
// states, each group with its own decomposition: chunks that fit the scratch
// memory, the job tables and their order.  Used by the single-query sampler
// (csim_host.cpp) and the query engine (csim_engine.cpp).
#pragma once

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "csim_tree.cuh"
#include "csim_tree.h"
#include "csim_tree_plan.h"

namespace csim_host {

// A plan's arrays on the device: gen, term (64 words each), then perm (64 bytes)
constexpr size_t kTreePlanBytes = 2 * 64 * 8 + 64;

struct TreeGroup {
    const csim::tree::Plan* plan = nullptr;
    const unsigned char* dplan = nullptr;  // the plan's device arrays (kTreePlanBytes)
    csim::TreeDraw draw{};                 // its states are draw's states 0 .. count - 1
    int64_t count = 0;
    int64_t shape_count = 0;               // states that tree_leaf_shape is asked for (0: count)
    __int128* part = nullptr;              // device: parts_per_state partial sums for each state
    // exactProjector rows (TreeLeafJob) row0, row0 + 1, ..., and 4 int128 per state that are zero
    // before the launches
    bool rows = false;
    int64_t row0 = 0;
    __int128* diag = nullptr;
};
// whether the tree sums exactProjector rows of a plan: a term index for each leaf
inline bool tree_rows_ok(const csim::tree::Plan& p) { return p.r == p.k; }

// How the leaf kernel covers the states of a group.  Small groups split a
// node's leaves over several threads until the GPU has enough of them; large
// ones give each thread several nodes, so its reduction at the end is shared.
struct TreeLeafShape {
    int split = 0, reps = 1, group = 1;
    int64_t threads_per_tree = 1, parts_per_tree = 1, parts_per_state = 1;
};
inline TreeLeafShape tree_leaf_shape(const csim::tree::Plan& p, int64_t count) {
    TreeLeafShape s;
    const int je = p.level.back();
    const int64_t nodes = (int64_t)1 << (p.level[0] - je);
    count <<= p.slice;
    while (s.split < je && ((count * nodes) << s.split) < (1 << 17)) s.split++;
    const int64_t parts = nodes << s.split;
    while (s.reps < 8 && parts >= 2 * 128 * s.reps && count * parts / (2 * s.reps) >= (1 << 19)) s.reps *= 2;
    s.threads_per_tree = parts / s.reps;
    s.group = (int)std::min<int64_t>(s.threads_per_tree, csim::kTreeLeafThreads);
    s.parts_per_tree = std::max<int64_t>(1, s.threads_per_tree / csim::kTreeLeafThreads);
    s.parts_per_state = s.parts_per_tree << p.slice;
    return s;
}

// Bytes of node planes per state (each of its trees, one after another) in the two scratch halves
inline void tree_scratch_per_state(const csim::tree::Plan& p, int64_t (&half)[2]) { csim::tree::tree_planes(p, half); }

// Scratch of a run's node planes: every chunk pays the latency of its draws and first stages,
// about 0.2 ms at 40 to 64 qubits (256 states of 57 qubits, 2^18 terms: 5.36 ms with 1 GB, 5.05 with
// 2, 4.93 with 4; 4096 of 40, 2^16 terms: 7.96, 7.74, 7.62).  Where the memory is not to be had,
// a quarter of it will do, down to kTreeScratchMin.
constexpr size_t kTreeScratchMax = (size_t)4 << 30, kTreeScratchMin = (size_t)64 << 20;
// decompositions of more than 2^30 terms run on the pair kernels (node indices are 32 bits)
constexpr int kTreeMaxRows = 30;

class TreeRun {
  public:
    // Splits the groups into chunks whose node planes fit reserve()'s budget (one
    // tree at least).  Returns the scratch bytes needed.
    size_t layout(const std::vector<TreeGroup>& groups) {
        const size_t budget = budget_;
        chunks_.clear();
        scratch_ = 0;
        size_t used = 0;
        Chunk cur;
        for (const TreeGroup& g : groups) {
            int64_t half[2];
            tree_scratch_per_state(*g.plan, half);
            const int64_t per = half[0] + half[1];
            const int64_t trees = g.count << g.plan->slice;
            for (int64_t f = 0; f < trees;) {
                const int64_t room = (int64_t)((budget > used ? budget - used : 0)) / std::max<int64_t>(1, per);
                int64_t c = std::min(trees - f, room);
                if (c <= 0) {
                    if (!cur.pieces.empty()) {
                        chunks_.push_back(cur);
                        scratch_ = std::max(scratch_, used);
                        cur.pieces.clear();
                        used = 0;
                        continue;
                    }
                    c = 1;
                }
                // equal chunks of a large group
                if (cur.pieces.empty() && c < trees - f) {
                    const int64_t n = (trees - f + c - 1) / c;
                    c = (trees - f + n - 1) / n;
                }
                Piece pc{g, f, c, {used, 0}};
                used += align((size_t)(half[0] * c));
                pc.off[1] = used;
                used += align((size_t)(half[1] * c));
                cur.pieces.push_back(pc);
                f += c;
                if (f < trees) {  // the group's next trees start a chunk of their own
                    chunks_.push_back(cur);
                    scratch_ = std::max(scratch_, used);
                    cur.pieces.clear();
                    used = 0;
                }
            }
        }
        if (!cur.pieces.empty()) {
            chunks_.push_back(cur);
            scratch_ = std::max(scratch_, used);
        }
        return scratch_;
    }

    // layout() for the largest budget, `most` at most, whose scratch `alloc` (bytes -> 0 or an error) finds memory for
    template <class Alloc>
    int reserve(const std::vector<TreeGroup>& groups, Alloc alloc, size_t most = kTreeScratchMax) {
        for (budget_ = most;; budget_ = std::max(budget_ / 4, kTreeScratchMin)) {
            const int rc = alloc(layout(groups));
            if (rc == 0 || budget_ <= kTreeScratchMin) return rc;
        }
    }

    // The job tables, to be copied to the device (`scratch`: the device scratch)
    void build(unsigned char* scratch, std::vector<unsigned char>& blob) {
        blob.clear();
        steps_.clear();
        for (const Chunk& ch : chunks_) {
            std::vector<csim::TreeRootJob> roots[2];    // up to 32 qubits, more
            std::vector<csim::TreeLeafJob> leaves[16];  // by table words (1, 2, 4, 8), rows, pairs
            int64_t rb[2] = {}, lb[16] = {};
            size_t depth = 0;
            for (const Piece& p : ch.pieces) {
                const csim::tree::Plan& pl = *p.g.plan;
                csim::TreeRootJob r{};
                const int wide = pl.t > 32;
                r.draw = p.g.draw;
                r.first = p.first;
                r.perm = p.g.dplan + 2 * 64 * 8;
                r.gen = (const uint64_t*)p.g.dplan + pl.level[0];
                r.slice = pl.slice;
                r.x0 = pl.x0;
                r.out = (uint32_t*)(scratch + p.off[0]);
                r.count = p.count;
                r.block0 = rb[wide];
                r.t = pl.t;
                rb[wide] += (p.count + csim::kTreeRootWarps - 1) / csim::kTreeRootWarps;
                roots[wide].push_back(r);
                depth = std::max(depth, pl.level.size());
                const TreeLeafShape s = tree_leaf_shape(pl, p.g.shape_count ? p.g.shape_count : p.g.count);
                csim::TreeLeafJob l{};
                const int je = pl.level.back();
                l.in = (const uint32_t*)(scratch + p.off[(pl.level.size() - 1) & 1]);
                l.part = p.g.part + 4 * p.first * s.parts_per_tree;
                l.in_count = p.count << (pl.level[0] - je);
                l.threads = p.count * s.threads_per_tree;
                const int wc = std::max(0, pl.tv - 5) + (p.g.rows ? 4 : 0) + (pl.pairs ? 8 : 0);
                l.block0 = lb[wc];
                l.m = pl.vert.back();
                l.je = je;
                l.tv = pl.tv;
                l.tj = pl.tj;
                l.split = s.split;
                l.reps = s.reps;
                l.group = s.group;
                l.shift = pl.t - pl.tv + 2 * (pl.k - pl.r);  // each codeword 2^{k - r} times
                for (int j = 0; j < je; j++) l.gen[j] = (uint16_t)pl.gen[j];
                if (p.g.rows) {
                    l.node0 = p.first << (pl.level[0] - je);
                    l.row0 = p.g.row0;
                    l.term = (const uint64_t*)p.g.dplan + 64;
                    l.diag = p.g.diag;
                    l.nodes_log2 = pl.r - je;
                }
                lb[wc] += (l.threads + csim::kTreeLeafThreads - 1) / csim::kTreeLeafThreads;
                leaves[wc].push_back(l);
            }
            for (int wide = 0; wide < 2; wide++)
                if (!roots[wide].empty()) add(blob, Step{0, wide, 0, (int)roots[wide].size(), rb[wide], 0}, roots[wide]);
            for (size_t d = 1; d < depth; d++)
                for (int kind = 2 * 8 + 1; kind >= 2 * 2; kind--) {  // 2 * byte planes + pairs
                    std::vector<csim::TreeStageJob> st;
                    int64_t sb = 0;
                    int mmax = 0;
                    for (const Piece& p : ch.pieces) {
                        const csim::tree::Plan& pl = *p.g.plan;
                        if (pl.level.size() <= d || 2 * csim::tree::row_planes(pl.vert[d - 1]) + pl.pairs != kind)
                            continue;
                        csim::TreeStageJob j{};
                        j.in = (const uint32_t*)(scratch + p.off[(d - 1) & 1]);
                        j.out = (uint32_t*)(scratch + p.off[d & 1]);
                        j.gen = (const uint64_t*)p.g.dplan + pl.level[d];
                        j.in_count = p.count << (pl.level[0] - pl.level[d - 1]);
                        j.count = p.count << (pl.level[0] - pl.level[d]);
                        j.block0 = sb;
                        j.mp = pl.vert[d - 1];
                        j.mc = pl.vert[d];
                        j.sub = pl.level[d - 1] - pl.level[d];
                        j.paired = pl.pairs ? 2 * (pl.t / 2) : 0;
                        const int64_t threads = j.sub > 0 ? j.count / 2 : j.count;  // a pair of siblings each
                        sb += (threads + csim::kTreeStageThreads - 1) / csim::kTreeStageThreads;
                        mmax = std::max(mmax, j.mp);
                        st.push_back(j);
                    }
                    if (!st.empty()) add(blob, Step{1, kind, mmax, (int)st.size(), sb, 0}, st);
                }
            for (int wc = 0; wc < 16; wc++)
                if (!leaves[wc].empty()) add(blob, Step{2, wc >> 2, 1 << (wc & 3), (int)leaves[wc].size(), lb[wc], 0}, leaves[wc]);
        }
    }

    // Queues the launches; `djobs`: build()'s tables on the device.  after_first (optional)
    // is recorded behind the first launch.
    int launch(const csim::Launch& L, const unsigned char* djobs, cudaEvent_t after_first = nullptr) const {
        for (size_t i = 0; i < steps_.size(); i++) {
            const Step& s = steps_[i];
            const void* j = djobs + s.off;
            if (i == 1 && after_first && cudaEventRecord(after_first, L.stream) != cudaSuccess) return -1;
            const int rc =
                s.kind == 0   ? csim::launch_tree_draw(L, (const csim::TreeRootJob*)j, s.njobs, s.blocks, s.flags & 1)
                : s.kind == 1 ? csim::launch_tree_stage(L, (const csim::TreeStageJob*)j, s.njobs, s.blocks, s.flags >> 1, s.size,
                                                          s.flags & 1)
                              : csim::launch_tree_leaf(L, (const csim::TreeLeafJob*)j, s.njobs, s.blocks, s.size,
                                                         s.flags & 1, s.flags & 2);
            if (rc) return rc;
        }
        return 0;
    }

  private:
    struct Piece {
        TreeGroup g;
        int64_t first, count;  // trees
        size_t off[2];
    };
    struct Chunk {
        std::vector<Piece> pieces;
    };
    struct Step {
        int kind;  // 0 roots, 1 a stage, 2 leaves
        int flags;  // roots: 1 wide; stages: 2 * byte planes + pairs; leaves: bit 0 rows, bit 1 pairs
        int size;   // a stage's largest parent; the leaves' table words
        int njobs;
        int64_t blocks;
        size_t off;
    };
    static size_t align(size_t x) { return (x + 255) & ~(size_t)255; }
    template <class J>
    void add(std::vector<unsigned char>& blob, Step s, const std::vector<J>& jobs) {
        s.off = align(blob.size());
        blob.resize(s.off + jobs.size() * sizeof(J));
        memcpy(blob.data() + s.off, jobs.data(), jobs.size() * sizeof(J));
        steps_.push_back(s);
    }
    std::vector<Chunk> chunks_;
    std::vector<Step> steps_;
    size_t scratch_ = 0, budget_ = kTreeScratchMax;
};

// A plan's device image (kTreePlanBytes)
inline void tree_plan_image(const csim::tree::Plan& p, unsigned char* out) {
    memcpy(out, p.gen, 64 * 8);
    memcpy(out + 64 * 8, p.term, 64 * 8);
    memcpy(out + 2 * 64 * 8, p.perm, 64);
}

}  // namespace csim_host
