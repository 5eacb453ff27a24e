// Host build of the tree sum's chunking (circuitsimulator_gb300/csrc/csim_tree_host.h), for
// CPU tests only, with an allocator that has `room` bytes.
#include <cstdint>
#include <vector>

#include "../../circuitsimulator_gb300/csrc/csim_tree_host.h"

extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
namespace csim {  // launchers that are never called here
int launch_tree_draw(const Launch&, const TreeRootJob*, int, int64_t, bool) { return -1; }
int launch_tree_stage(const Launch&, const TreeStageJob*, int, int64_t, int, int, bool) { return -1; }
int launch_tree_leaf(const Launch&, const TreeLeafJob*, int, int64_t, int, bool, bool) { return -1; }
}  // namespace csim
extern "C" cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }

// out: reserve's status, its scratch bytes, allocations tried, the first chunk's states, bytes of
// node planes per state
extern "C" void tree_layout(const uint64_t* L, int k, int t, int64_t count, int64_t room, int64_t* out) {
    csim::tree::Plan plan;
    csim::tree::make_plan(L, k, t, count, plan);
    csim_host::TreeGroup g;
    g.plan = &plan;
    g.count = count;
    csim_host::TreeRun run;
    int64_t tried = 0, bytes = 0;
    out[0] = run.reserve({g}, [&](size_t b) {
        tried++;
        bytes = (int64_t)b;
        return (int64_t)b <= room ? 0 : -1;
    });
    out[1] = bytes;
    out[2] = tried;
    std::vector<unsigned char> blob;
    run.build(nullptr, blob);
    const csim::TreeRootJob& r = *(const csim::TreeRootJob*)blob.data();
    out[3] = r.count;
    int64_t half[2];
    csim_host::tree_scratch_per_state(plan, half);
    out[4] = half[0] + half[1];
}
