// csim_rand.cu — raw words of the C library's rand() and the states' places in them
// (csim_rand.h).
#include <cuda_runtime.h>

#include <cstdint>

#include "csim_rand.h"
#include "csim_warp.cuh"

namespace csim {

// ---------------------------------------------------------------- host tables
namespace {

// a b mod x^31 - x^28 - 1
void poly_mul(const uint32_t (&a)[31], const uint32_t (&b)[31], uint32_t (&out)[31]) {
    uint32_t p[61] = {};
    for (int i = 0; i < 31; i++)
        for (int j = 0; j < 31; j++) p[i + j] += a[i] * b[j];
    for (int i = 60; i >= 31; i--) {
        p[i - 3] += p[i];
        p[i - 31] += p[i];
    }
    for (int i = 0; i < 31; i++) out[i] = p[i];
}

// x^(kRawChunk 2^b), coefficient of x^m at m
struct RawJumps {
    uint32_t p[kRawJumps][31];
};
const RawJumps& raw_jumps() {
    struct Made : RawJumps {
        Made() {
            uint32_t r[31] = {1}, x[31] = {0, 1};
            for (int e = kRawChunk; e; e >>= 1) {
                if (e & 1) poly_mul(r, x, r);
                poly_mul(x, x, x);
            }
            for (int b = 0; b < kRawJumps; b++) {
                for (int m = 0; m < 31; m++) p[b][m] = r[m];
                poly_mul(r, r, r);
            }
        }
    };
    static const Made jumps;
    return jumps;
}

void draw_table(int n, const double* cum, DrawTable& t) {
    t.n = n;
    for (int d = 0; d <= n; d++) {  // the largest x whose sample is at most cum[d] (x = 0 always is)
        int64_t lo = 0, hi = 2147483647;
        while (lo < hi) {
            const int64_t x = (lo + hi + 1) / 2;
            const double sample = 0. + ((int32_t)x / (2147483647 / 1.0));
            if (sample <= cum[d]) lo = x;
            else hi = x - 1;
        }
        t.last[d] = (uint32_t)lo;
    }
}

// Words per segment of the chain of `states` states of up to `longest` words each: a power of two.
// Following a chain within a segment takes 30 ns a state, twice, the walk 300 ns a segment, so
// sqrt(5 states) states per segment are best.
int chain_segment(int64_t states, int longest) {
    int64_t s = 1 << 10;
    while (s < kMaxSegment && s * s < 5 * states * longest * longest / 2) s *= 2;
    return (int)s;
}

// The jobs of a launch, and the first block of each in the four kernels
template <int N>
struct DrawJobs {
    int n;
    int32_t raw0[N], len0[N], map0[N], place0[N];
    DrawJob job[N];
};
template <int N>
__device__ __forceinline__ int job_at(const int32_t (&first)[N], int n) {
    int j = 0;
    for (int i = 1; i < n; i++)
        if ((int)blockIdx.x >= first[i]) j = i;
    return j;
}

}  // namespace

void draw_job(int t, const double* cum, int64_t states, int percent, DrawJob& j) {
    draw_table(t, cum, j.table);
    j.entries = most_words(t);
    j.segment = chain_segment(states, j.entries);
    j.words = (j.entries * states + 4096) * percent / 100;
    j.states = states;
}

// ---------------------------------------------------------------- words
// The next 31 words from the last 31 (lane l < 31 holds word l): sums of every third
// word, from r[l - 3] on
__device__ __forceinline__ uint32_t next_words(uint32_t w, int lane) {
    const uint32_t from = __shfl_sync(kFull, w, 28 + lane % 3);
#pragma unroll
    for (int o = 3; o < 32; o *= 2) {
        const uint32_t v = __shfl_up_sync(kFull, w, o);
        if (lane >= o) w += v;
    }
    return w + from;
}

constexpr int kRawThreads = 256;

// A warp per kRawChunk words: jumps to its chunk (a jump: 31 products per word), then 31
// words at a time from the 31 before.  Bound by the latency of its serial steps: 361,000
// words in 10 us (the host makes one in 0.4 ns, 144 us).
template <int N>
__global__ void __launch_bounds__(kRawThreads) k_raw_words(const __grid_constant__ RawJumps jumps,
                                                           const __grid_constant__ DrawJobs<N> jobs) {
    __shared__ uint32_t win[kRawThreads / 32][64];
    const int lane = threadIdx.x & 31, ji = job_at<N>(jobs.raw0, jobs.n);
    const DrawJob& s = jobs.job[ji];
    const int64_t count = s.words;
    uint32_t* const buf = s.buf;
    uint32_t* const r = win[threadIdx.x >> 5];
    const int64_t chunk = ((int64_t)(blockIdx.x - jobs.raw0[ji]) * kRawThreads + threadIdx.x) >> 5;
    if (chunk == 0) {
        buf[lane] = s.history[lane];
        if (lane < kRawHistory - 32) buf[32 + lane] = s.history[32 + lane];
    }
    if (chunk * kRawChunk >= count) return;  // warp-uniform
    uint32_t w = lane < 31 ? s.history[kRawHistory - 31 + lane] : 0u;
    for (int b = 0; b < kRawJumps; b++) {
        if (!((chunk >> b) & 1)) continue;  // warp-uniform
        const uint32_t v = next_words(w, lane);
        __syncwarp();
        if (lane < 31) {
            r[lane] = w;
            r[31 + lane] = v;
        }
        __syncwarp();
        w = 0u;
#pragma unroll
        for (int m = 0; m < 31; m++) w += jumps.p[b][m] * r[m + lane];  // lane 31: unused
    }
    uint32_t* const out = buf + kRawHistory + chunk * kRawChunk;
    const int64_t left = count - chunk * kRawChunk;
    for (int i = 0; i < kRawChunk && i < left; i += 31) {
        w = next_words(w, lane);
        if (lane < 31 && i + lane < left) out[i + lane] = w;
    }
}

// ---------------------------------------------------------------- lengths
// The words of a state that starts at word i (randomStabilizerState,
// stabilizer.c:689-756): rand() until it is not 0, vectors of ceil(n / 8) words until
// d of them are independent, three vectors, the triangle of J.  A word per thread; the
// words' low bytes lie in shared memory, so a vector is two loads and a shift (loads of
// its words from L1: 52 us for 3.3e6 positions at n = 40, now 41).  Lanes differ in the
// dimension: ALU-bound with few of them busy.
constexpr int kLengthThreads = 256, kLengthReach = 256;  // words behind the block's that vectors are read from

template <int N>
__global__ void __launch_bounds__(kLengthThreads) k_draw_lengths(const __grid_constant__ DrawJobs<N> jobs) {
    __shared__ uint64_t bytes_s[(kLengthThreads + kLengthReach) / 8 + 1];
    const int ji = job_at<N>(jobs.len0, jobs.n);
    const DrawJob& s = jobs.job[ji];
    const DrawTable& t = s.table;
    const int64_t count = s.words;
    uint16_t* const len = s.len;
    const int64_t base = (int64_t)(blockIdx.x - jobs.len0[ji]) * kLengthThreads, i = base + threadIdx.x;
    const uint32_t* const w = s.buf + kRawHistory + base;
    const int there = (int)(count - base < (1 << 20) ? count - base : (1 << 20));  // words from the block's first on
    for (int q = threadIdx.x; q < kLengthThreads + kLengthReach; q += kLengthThreads)
        reinterpret_cast<uint8_t*>(bytes_s)[q] = q < there ? (uint8_t)(w[q] >> 1) : 0;
    if (threadIdx.x == 0) bytes_s[(kLengthThreads + kLengthReach) / 8] = 0;
    __syncthreads();
    const int n = t.n, bytes = (n + 7) / 8;
    // bits of a vector: of byte b the ones for qubits 8 b + j < n, most significant first
    const uint64_t keep = (bytes < 8 ? (1ull << (8 * bytes)) - 1 : ~0ull) & ~((uint64_t)((1u << (8 * bytes - n)) - 1) << (8 * (bytes - 1)));
    const auto vector = [&](int p) -> uint64_t {
        if (p + 8 <= kLengthThreads + kLengthReach) {
            const int q = p >> 3, sh = 8 * (p & 7);
            const uint64_t lo = bytes_s[q] >> sh;
            return (sh ? lo | (bytes_s[q + 1] << (64 - sh)) : lo) & keep;
        }
        uint64_t v = 0;
        for (int b = 0; b < bytes; b++) v |= (uint64_t)((w[p + b] >> 1) & 255u) << (8 * b);
        return v & keep;
    };
    const auto reduce = [](uint64_t v, uint64_t e) { return v & (e & (0 - e)) ? v ^ e : v; };  // e's lowest bit: its pivot
    int p = threadIdx.x;
    while (p < there && (w[p] >> 1) == 0u) p++;
    int d = 0, missing = 0;
    if (p < there) {
        const uint32_t x = w[p++] >> 1;
        while (d < n && x > t.last[d]) d++;
        // vectors until d are independent
        missing = d;
        if (d <= 2) {
            uint64_t e0 = 0;
            while (missing && p + bytes <= there) {
                const uint64_t v = reduce(vector(p), e0);
                p += bytes;
                if (v == 0) continue;
                e0 = e0 ? e0 : v;  // (the second is the last)
                missing--;
            }
        } else {
            uint64_t basis[64];
            int rank = 0;
            while (missing && p + bytes <= there) {
                uint64_t v = vector(p);
                p += bytes;
                for (int j = 0; j < rank; j++) v = reduce(v, basis[j]);
                if (v == 0) continue;
                basis[rank++] = v;
                missing--;
            }
        }
    } else {
        missing = 1;
    }
    const int k = n - d;
    p += 3 * bytes + k * (k - 1) / 2;
    const int words = p - (int)threadIdx.x;
    len[i] = (uint16_t)(missing == 0 && p <= there && words <= 0xFFFF ? words : 0);
}

// ---------------------------------------------------------------- the chain
constexpr int kChainThreads = 1024;
constexpr uint32_t kNoExit = 0xFFFFu;  // the words end in the segment

// the block's segment of lengths
__device__ __forceinline__ void load_segment(uint16_t* to, const uint16_t* from, int segment) {
    constexpr int kLoads = kMaxSegment / 8 / kChainThreads;
    uint4 v[kLoads];
#pragma unroll
    for (int j = 0; j < kLoads; j++) {
        const int at = (int)threadIdx.x + j * kChainThreads;
        if (at < segment / 8) v[j] = ((const uint4*)from)[at];
    }
#pragma unroll
    for (int j = 0; j < kLoads; j++) {
        const int at = (int)threadIdx.x + j * kChainThreads;
        if (at < segment / 8) ((uint4*)to)[at] = v[j];
    }
}

// map[e] of the block's segment: where the chain from its word e leaves it (words behind
// its end, kNoExit) and, in the upper half, how many states begin in it on the way
template <int N>
__global__ void __launch_bounds__(kChainThreads) k_chain_maps(const __grid_constant__ DrawJobs<N> jobs) {
    extern __shared__ __align__(16) uint16_t seg_s[];
    const int ji = job_at<N>(jobs.map0, jobs.n), b = blockIdx.x - jobs.map0[ji];
    const int segment = jobs.job[ji].segment, entries = jobs.job[ji].entries;
    uint32_t* const map = jobs.job[ji].map + (int64_t)b * entries;
    load_segment(seg_s, jobs.job[ji].len + (int64_t)b * segment, segment);
    __syncthreads();
    for (int e = threadIdx.x; e < entries; e += kChainThreads) {
        int p = e, states = 0;
        while (p < segment) {
            const int l = seg_s[p];
            if (l == 0) break;
            p += l;
            states++;
        }
        const int out = p - segment;  // (below 0: the words end)
        map[e] = (out < 0 || out >= (int)kNoExit ? kNoExit : (uint32_t)out) | ((uint32_t)states << 16);
    }
}

// The segments before the block's give the state that its first one is and the word it
// begins at; then its first thread places the segment's.  Bound by the latency of its
// serial loads: 2000 states of 12 qubits 15 us with k_chain_maps' 8, 4096 of 40 qubits
// 30 with 8; one thread over all segments, the next one loading meanwhile, took 72 and
// 203 us.
template <int N>
__global__ void __launch_bounds__(kChainThreads) k_chain_place(const __grid_constant__ DrawJobs<N> jobs) {
    extern __shared__ __align__(16) uint16_t seg_s[];
    __shared__ int64_t at_s;
    __shared__ int last_s;
    const int ji = job_at<N>(jobs.place0, jobs.n), b = blockIdx.x - jobs.place0[ji];
    const DrawJob& J = jobs.job[ji];
    const int segment = J.segment, entries = J.entries;
    const uint16_t* const len = J.len;
    const uint32_t* const map = J.map;
    const int64_t states = J.states;
    int64_t* const offs = J.offs;
    const bool last_segment = (int64_t)(b + 1) * segment >= J.words;
    load_segment(seg_s, len + (int64_t)b * segment, segment);
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t state = 0, at = 0;
        bool out_of_words = false;
        for (int s = 0; s < b && state < states && !out_of_words; s++) {
            const int64_t end = (int64_t)(s + 1) * segment;
            const int64_t e = at - (end - segment);
            if (e >= segment) continue;  // a state longer than a segment
            const uint32_t m = e < entries ? map[(int64_t)s * entries + e] : kNoExit;
            if ((m & 0xFFFFu) != kNoExit) {
                at = end + (m & 0xFFFFu);
                state += m >> 16;
                continue;
            }
            while (at < end && state < states && !out_of_words) {  // word by word
                const int l = len[at];
                out_of_words = l == 0;
                at += l;
                state += l != 0;
            }
        }
        // (state can have passed `states`: then a block before places the last one)
        const int64_t seg = (int64_t)b * segment;
        int last = 0;
        if (state < states && !out_of_words) {
            int64_t rel = at - seg;
            while (rel < segment && state < states) {
                const int l = seg_s[rel];
                out_of_words = l == 0;
                if (l == 0) break;
                offs[state++] = kRawHistory + seg + rel;
                rel += l;
            }
            at = seg + rel;
            last = state == states || out_of_words || last_segment;
            if (last) {
                J.chain->states = state;
                J.chain->words = at;
                for (; state <= states; state++) offs[state] = kRawHistory + at;  // the end, or no words
            }
        }
        at_s = at;
        last_s = last;
    }
    __syncthreads();
    if (last_s && threadIdx.x < kRawHistory) J.chain->history[threadIdx.x] = J.buf[at_s + threadIdx.x];
}

// ---------------------------------------------------------------- launchers
namespace {

template <int N>
int launch_jobs(const Launch& L, const DrawJob* jobs, int njobs) {
    DrawJobs<N> J;
    J.n = njobs;
    int64_t raw = 0, len = 0, maps = 0, place = 0;
    int segment = 0;
    for (int i = 0; i < njobs; i++) {
        const DrawJob& j = J.job[i] = jobs[i];
        if (j.states <= 0 || j.words <= 0 || j.words > kRawMax || j.table.n < 1 || j.table.n > 64 || j.entries < 1 ||
            j.segment < kLengthThreads || j.segment % kLengthThreads || j.segment > kMaxSegment)
            return -1;
        const int64_t chunks = (j.words + kRawChunk - 1) / kRawChunk, segments = j.padded() / j.segment;
        J.raw0[i] = (int32_t)raw;
        J.len0[i] = (int32_t)len;
        J.map0[i] = (int32_t)maps;
        J.place0[i] = (int32_t)place;
        raw += (chunks + kRawThreads / 32 - 1) / (kRawThreads / 32);
        len += j.padded() / kLengthThreads;
        maps += segments - 1;
        place += segments;
        segment = segment > j.segment ? segment : j.segment;
    }
    if (raw > 0x7fffffff || len > 0x7fffffff) return -1;
    const int smem = segment * (int)sizeof(uint16_t), most = kMaxSegment * (int)sizeof(uint16_t);
    if (cudaFuncSetAttribute(k_chain_maps<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess ||
        cudaFuncSetAttribute(k_chain_place<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess)
        return -1;
    k_raw_words<N><<<(unsigned)raw, kRawThreads, 0, L.stream>>>(raw_jumps(), J);
    k_draw_lengths<N><<<(unsigned)len, kLengthThreads, 0, L.stream>>>(J);
    if (maps > 0) k_chain_maps<N><<<(unsigned)maps, kChainThreads, smem, L.stream>>>(J);
    k_chain_place<N><<<(unsigned)place, kChainThreads, smem, L.stream>>>(J);
    *L.launches += maps > 0 ? 4 : 3;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace

int launch_draws(const Launch& L, const DrawJob* jobs, int njobs) {
    for (int i = 0; i < njobs; i += kDrawJobs) {
        const int n = njobs - i < kDrawJobs ? njobs - i : kDrawJobs;
        const int rc = n == 1 ? launch_jobs<1>(L, jobs + i, 1) : launch_jobs<kDrawJobs>(L, jobs + i, n);
        if (rc) return rc;
    }
    return 0;
}

}  // namespace csim
