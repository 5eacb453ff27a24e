// Host build of the tree sum's job tables (circuitsimulator_gb300/csrc/csim_tree_host.h), for
// CPU tests only: launchers that check what the kernels would read and write.
#include <cstdint>
#include <set>
#include <vector>

#include "../../circuitsimulator_gb300/csrc/csim_tree_host.h"

extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
extern "C" cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }

namespace {

using csim::tree::node_words;

struct Range {
    int64_t begin, end;
};
int64_t scratch_bytes, bad, jobs;
std::vector<Range> live, made;  // node planes that the next stage may read, that this one has written
std::set<int64_t> trees, parts;
std::vector<int64_t> chunk_first;  // the first tree of the chunk's root jobs
const csim::tree::Plan* plan_of;

Range planes(const uint32_t* p, int64_t count, int m) {
    const int64_t b = (int64_t)(uintptr_t)p;
    return Range{b, b + 4 * count * node_words(m)};
}
void write(Range r) {
    if (r.begin < 0 || r.end > scratch_bytes) bad++;
    for (const Range& o : made) bad += r.begin < o.end && o.begin < r.end;
    for (const Range& o : live) bad += r.begin < o.end && o.begin < r.end;  // still to be read
    made.push_back(r);
    jobs++;
}
void read(Range r) {
    for (size_t i = 0; i < live.size(); i++)
        if (live[i].begin == r.begin && live[i].end == r.end) {
            live.erase(live.begin() + (int64_t)i);
            return;
        }
    bad++;
}

}  // namespace

namespace csim {
int launch_tree_draw(const Launch&, const TreeRootJob* j, int n, int64_t, bool) {
    if (!live.empty()) bad++;  // planes that nothing has read
    live.clear();
    chunk_first.clear();
    for (int i = 0; i < n; i++) {
        write(planes(j[i].out, j[i].count, j[i].t));
        chunk_first.push_back(j[i].first);
        bad += j[i].slice != plan_of->slice || (int64_t)(uintptr_t)j[i].gen != 8 * (plan_of->r - plan_of->slice);
        for (int64_t s = 0; s < j[i].count; s++) bad += !trees.insert(j[i].first + s).second;
    }
    live.swap(made);
    made.clear();
    return 0;
}
int launch_tree_stage(const Launch&, const TreeStageJob* j, int n, int64_t, int, int, bool) {
    for (int i = 0; i < n; i++) {
        if (j[i].in_count << j[i].sub != j[i].count) bad++;
        write(planes(j[i].out, j[i].count, j[i].mc));
        read(planes(j[i].in, j[i].in_count, j[i].mp));
    }
    live.insert(live.end(), made.begin(), made.end());
    made.clear();
    return 0;
}
int launch_tree_leaf(const Launch&, const TreeLeafJob* j, int n, int64_t, int, bool, bool) {
    for (int i = 0; i < n; i++) {
        read(planes(j[i].in, j[i].in_count, j[i].m));
        if ((j[i].threads * j[i].reps) >> j[i].split != j[i].in_count) bad++;
        if (j[i].term)  // rows: a node's number has the tree's, and the levels above je
            bad += j[i].nodes_log2 != plan_of->r - j[i].je ||
                   j[i].node0 != chunk_first[i] << (plan_of->r - plan_of->slice - j[i].je) || j[i].row0 || j[i].diag;
        for (int64_t p = 0; p < (j[i].threads + j[i].group - 1) / j[i].group; p++)
            if (!parts.insert((int64_t)(uintptr_t)j[i].part / 64 + p).second) bad++;
    }
    return 0;
}
}  // namespace csim

// out: reserve's status, its scratch bytes, job table entries of nodes, violations, trees per state, the partial sums
// that were written, those there are
extern "C" void tree_jobs(const uint64_t* L, int k, int t, int64_t count, int64_t room, int rows, int64_t* out) {
    csim::tree::Plan plan;
    if (L) csim::tree::make_plan(L, k, t, count, plan);
    else {
        csim::tree::build_pairs(t, plan);
        csim::tree::choose_levels(plan, count);
    }
    scratch_bytes = bad = jobs = 0;
    live.clear();
    made.clear();
    trees.clear();
    parts.clear();
    plan_of = &plan;
    csim_host::TreeGroup g;
    g.plan = &plan;
    g.count = count;
    g.rows = rows;
    csim_host::TreeRun run;
    out[0] = run.reserve({g}, [&](size_t b) {
        scratch_bytes = (int64_t)b;
        return (int64_t)b <= room ? 0 : -1;
    });
    out[1] = scratch_bytes;
    std::vector<unsigned char> blob;
    run.build(nullptr, blob);
    run.launch(csim::Launch{}, blob.data());
    out[2] = jobs;
    out[4] = 1 << plan.slice;
    out[3] = bad + ((int64_t)trees.size() != count * out[4]) + (!trees.empty() && *trees.rbegin() != count * out[4] - 1);
    out[5] = (int64_t)parts.size();
    out[6] = count * csim_host::tree_leaf_shape(plan, count).parts_per_state;
    for (int64_t p : parts) out[3] += p < 0 || p >= out[6];
}
