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

}  // namespace

void raw_jumps(RawStart& s) {
    struct Jumps {
        uint32_t p[kRawJumps][31];
        Jumps() {
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
    static const Jumps jumps;
    for (int b = 0; b < kRawJumps; b++)
        for (int m = 0; m < 31; m++) s.jump[b][m] = jumps.p[b][m];
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
__global__ void __launch_bounds__(kRawThreads) k_raw_words(const __grid_constant__ RawStart s, int64_t count, uint32_t* buf) {
    __shared__ uint32_t win[kRawThreads / 32][64];
    const int lane = threadIdx.x & 31;
    uint32_t* const r = win[threadIdx.x >> 5];
    const int64_t chunk = ((int64_t)blockIdx.x * kRawThreads + threadIdx.x) >> 5;
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
        for (int m = 0; m < 31; m++) w += s.jump[b][m] * r[m + lane];  // lane 31: unused
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

__global__ void __launch_bounds__(kLengthThreads) k_draw_lengths(const __grid_constant__ DrawTable t, const uint32_t* buf,
                                                                 int64_t count, uint16_t* len) {
    __shared__ uint64_t bytes_s[(kLengthThreads + kLengthReach) / 8 + 1];
    const int64_t base = (int64_t)blockIdx.x * kLengthThreads, i = base + threadIdx.x;
    const uint32_t* const w = buf + kRawHistory + base;
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
__global__ void __launch_bounds__(kChainThreads) k_chain_maps(const uint16_t* len, int segment, int entries, uint32_t* map) {
    extern __shared__ __align__(16) uint16_t seg_s[];
    load_segment(seg_s, len + (int64_t)blockIdx.x * segment, segment);
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
        map[(int64_t)blockIdx.x * entries + e] = (out < 0 || out >= (int)kNoExit ? kNoExit : (uint32_t)out) | ((uint32_t)states << 16);
    }
}

// The segments before the block's give the state that its first one is and the word it
// begins at; then its first thread places the segment's.  Bound by the latency of its
// serial loads: 2000 states of 12 qubits 15 us with k_chain_maps' 8, 4096 of 40 qubits
// 30 with 8; one thread over all segments, the next one loading meanwhile, took 72 and
// 203 us.
__global__ void __launch_bounds__(kChainThreads) k_chain_place(const uint16_t* len, int segment, const uint32_t* buf, int entries,
                                                               const uint32_t* map, int64_t states, int64_t* offs,
                                                               DrawChain* chain) {
    extern __shared__ __align__(16) uint16_t seg_s[];
    __shared__ int64_t at_s;
    __shared__ int last_s;
    load_segment(seg_s, len + (int64_t)blockIdx.x * segment, segment);
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t state = 0, at = 0;
        bool out_of_words = false;
        for (int s = 0; s < (int)blockIdx.x && state < states && !out_of_words; s++) {
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
        const int64_t seg = (int64_t)blockIdx.x * segment;
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
            last = state == states || out_of_words || blockIdx.x + 1 == gridDim.x;
            if (last) {
                chain->states = state;
                chain->words = at;
                for (; state <= states; state++) offs[state] = kRawHistory + at;  // the end, or no words
            }
        }
        at_s = at;
        last_s = last;
    }
    __syncthreads();
    if (last_s && threadIdx.x < kRawHistory) chain->history[threadIdx.x] = buf[at_s + threadIdx.x];
}

// ---------------------------------------------------------------- launchers
int launch_raw_words(const Launch& L, const RawStart& s, int64_t count, uint32_t* buf) {
    if (count <= 0 || count > kRawMax) return -1;
    const int64_t chunks = (count + kRawChunk - 1) / kRawChunk, per = kRawThreads / 32;
    k_raw_words<<<(unsigned)((chunks + per - 1) / per), kRawThreads, 0, L.stream>>>(s, count, buf);
    (*L.launches)++;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_draw_lengths(const Launch& L, const DrawTable& t, const uint32_t* buf, int64_t count, int64_t padded,
                        uint16_t* len) {
    if (count <= 0 || padded <= 0 || padded > kRawMax || padded % kLengthThreads || t.n < 1 || t.n > 64) return -1;
    k_draw_lengths<<<(unsigned)(padded / kLengthThreads), kLengthThreads, 0, L.stream>>>(t, buf, count, len);
    (*L.launches)++;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_draw_chain(const Launch& L, const uint16_t* len, int64_t padded, int segment, const uint32_t* buf, int entries,
                      uint32_t* map, int64_t states, int64_t* offs, DrawChain* chain) {
    if (states <= 0 || segment < 8 || segment % 8 || segment > kMaxSegment || padded <= 0 || padded % segment ||
        padded > kRawMax || entries < 1)
        return -1;
    const unsigned segments = (unsigned)(padded / segment);
    const int smem = segment * (int)sizeof(uint16_t), most = kMaxSegment * (int)sizeof(uint16_t);
    if (cudaFuncSetAttribute(k_chain_maps, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess ||
        cudaFuncSetAttribute(k_chain_place, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess)
        return -1;
    if (segments > 1) {
        k_chain_maps<<<segments - 1, kChainThreads, smem, L.stream>>>(len, segment, entries, map);
        (*L.launches)++;
    }
    k_chain_place<<<segments, kChainThreads, smem, L.stream>>>(len, segment, buf, entries, map, states, offs, chain);
    (*L.launches)++;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace csim
