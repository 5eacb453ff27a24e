// csim_host.cpp — host side of libcsimgpu.so: the single-query C ABI of
// include/csim.h.
//
// Contexts, the batched primitives (innerProduct, exponentialSum, shrink,
// measurePauli, extend, randomStabilizerState, prepH/prepL), the estimator
// drivers (singleProjectorSample / sampledProjector / multiSampledProjector /
// exactProjector of libcirc/innerprod.c) and decompose (libcirc/probability.c:
// 307-415).  Shared helpers (the C library's rand() sequence, buffers, checks)
// are in csim_host_common.h; many queries at once go through csim_engine.cpp.
// All stabilizer algebra runs in the kernels; the host prepares inputs,
// converts the kernels' exact Z[w] sums to doubles and does the per-query
// reductions.
#include <mutex>

#include "csim_host_common.h"

using namespace csim_host;


// ---------------------------------------------------------------- context API
extern "C" void csim_ctx_destroy(csim_ctx* ctx);

extern "C" int csim_ctx_create(int device, csim_ctx** out) {
    if (!out) return CSIM_ERR_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= device || device < 0) return CSIM_ERR_NODEVICE;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return CSIM_ERR_NODEVICE;
    if (!(prop.major == 10 && prop.minor == 3)) {
        fprintf(stderr, "csim: device %d is sm_%d%d; libcsimgpu is built for sm_103a only\n", device, prop.major,
                prop.minor);
        return CSIM_ERR_NODEVICE;
    }
    csim_ctx* ctx = new csim_ctx();
    ctx->device = device;
    ctx->num_sms = prop.multiProcessorCount;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) !=
                                                    cudaSuccess ||
        cudaMalloc(&ctx->d_err, sizeof(int)) != cudaSuccess ||
        cudaMallocHost(&ctx->h_err, sizeof(int)) != cudaSuccess || cudaMemset(ctx->d_err, 0, sizeof(int)) != cudaSuccess) {
        delete ctx;
        return CSIM_ERR_CUDA;
    }
    for (int i = 0; i < 4; i++)
        if (cudaEventCreate(&ctx->ev[i]) != cudaSuccess) {
            csim_ctx_destroy(ctx);
            return CSIM_ERR_CUDA;
        }
    ctx->lr.seed(1);  // an unseeded rand() behaves as srand(1)
    *out = ctx;
    return CSIM_OK;
}

extern "C" void csim_ctx_destroy(csim_ctx* ctx) {
    if (!ctx) return;
    if (ctx->engine) {
        cudaSetDevice(ctx->device);
        engine_free(ctx->engine);
        ctx->engine = nullptr;
    }
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    for (int i = 0; i < kNumBufs + 32; i++)
        if (ctx->buf[i]) cudaFree(ctx->buf[i]);
    if (ctx->d_err) cudaFree(ctx->d_err);
    if (ctx->h_err) cudaFreeHost(ctx->h_err);
    for (int i = 0; i < 4; i++)
        if (ctx->ev[i]) cudaEventDestroy(ctx->ev[i]);
    for (int i = 0; i < kPinSlots; i++) {
        if (ctx->pin_ev[i]) cudaEventDestroy(ctx->pin_ev[i]);
        if (ctx->pin[i]) cudaFreeHost(ctx->pin[i]);
    }
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
}

extern "C" int csim_set_option(csim_ctx* ctx, int32_t option, int64_t value) {
    if (!ctx) return CSIM_ERR_ARG;
    switch (option) {
    case CSIM_OPT_PAIR_KERNEL:
        if (value < 0 || value > 5) return fail(ctx, CSIM_ERR_ARG, "pair kernel must be 0..5");
        ctx->pair_kernel = (int)value;
        return CSIM_OK;
    case CSIM_OPT_PER_THREAD:
        if (value < 0 || value > 64) return fail(ctx, CSIM_ERR_ARG, "per-thread pairs must be 0 (by t) or 1..64");
        ctx->per_thread = (int)value;
        return CSIM_OK;
    case CSIM_OPT_DIRECT_SLOTS:
        if (value < 0 || value > 64) return fail(ctx, CSIM_ERR_ARG, "direct slots must be 0 (by t) or 1..64");
        ctx->direct_slots = (int)value;
        return CSIM_OK;
    case CSIM_OPT_AUTOTUNE:
        if (value != 0 && value != 1) return fail(ctx, CSIM_ERR_ARG, "autotune must be 0 or 1");
        ctx->autotune = (int)value;
        return CSIM_OK;
    case CSIM_OPT_DRAW_WORDS:
        if (value < 1 || value > 100) return fail(ctx, CSIM_ERR_ARG, "draw words must be 1..100 percent");
        ctx->draw_percent = (int)value;
        return CSIM_OK;
    default:
        return fail(ctx, CSIM_ERR_ARG, "unknown option %d", option);
    }
}

extern "C" int csim_rng_position(csim_ctx* ctx, uint64_t seed, uint64_t first) {
    if (!ctx) return CSIM_ERR_ARG;
    ctx->philox_seed = seed;
    ctx->philox_next = first;
    return CSIM_OK;
}

extern "C" int csim_last_stats(const csim_ctx* ctx, csim_stats* out) {
    if (!ctx || !out) return CSIM_ERR_ARG;
    *out = ctx->stats;
    return CSIM_OK;
}

extern "C" const char* csim_last_error(const csim_ctx* ctx) { return ctx ? ctx->last_error.c_str() : ""; }
extern "C" int64_t csim_launch_count(const csim_ctx* ctx) { return ctx ? ctx->launches : 0; }

extern "C" int64_t csim_libc_rand_size(void) { return (int64_t)sizeof(LibcRand); }
extern "C" void csim_libc_rand_seed(void* state, uint32_t seed) { ((LibcRand*)state)->seed(seed); }
extern "C" int32_t csim_libc_rand_next(void* state) { return ((LibcRand*)state)->next(); }

// ---------------------------------------------------------------- primitives
extern "C" int csim_inner_product_exact(csim_ctx* ctx, int64_t count, const csim_state* a, const csim_state* b,
                                        int32_t* eps, int32_t* p, int32_t* m) {
    if (!ctx || count < 0 || (count && (!a || !b || !eps || !p || !m))) return fail(ctx, CSIM_ERR_ARG, "null argument");
    cudaSetDevice(ctx->device);
    int nra, nrb;
    CKR(check_states(ctx, a, count, &nra));
    CKR(check_states(ctx, b, count, &nrb));
    for (int64_t i = 0; i < count; i++)
        if (a[i].n != b[i].n) return fail(ctx, CSIM_ERR_ARG, "pair %lld: n differs", (long long)i);
    const int nr = std::max(nra, nrb);
    for (int64_t o = 0; o < count; o += kBatch) {
        const int64_t c = std::min(kBatch, count - o);
        csim_state *da, *db;
        void *d, *v;
        CKR(dput(ctx, kBufA, a + o, c, &da));
        CKR(dput(ctx, kBufB, b + o, c, &db));
        CKR(dbuf(ctx, kBufEps, 3 * c * 4, &d));  // eps, p, m
        if (csim::launch_inner_product(launch_of(ctx), nr, (const csim::GState*)da, (const csim::GState*)db, c, (int*)d,
                                       (int*)d + c, (int*)d + 2 * c))
            return fail(ctx, CSIM_ERR_CUDA, "inner product launch failed");
        CKR(finish_with(ctx, d, (size_t)(3 * c * 4), &v));
        memcpy(eps + o, v, (size_t)(c * 4));
        memcpy(p + o, (const int*)v + c, (size_t)(c * 4));
        memcpy(m + o, (const int*)v + 2 * c, (size_t)(c * 4));
    }
    return CSIM_OK;
}

extern "C" int csim_exponential_sum_exact(csim_ctx* ctx, int64_t count, csim_state* s, int32_t* eps, int32_t* p,
                                          int32_t* m) {
    if (!ctx || count < 0 || (count && (!s || !eps || !p || !m))) return fail(ctx, CSIM_ERR_ARG, "null argument");
    cudaSetDevice(ctx->device);
    int nr;
    CKR(check_states(ctx, s, count, &nr));
    for (int64_t o = 0; o < count; o += kBatch) {
        const int64_t c = std::min(kBatch, count - o);
        csim_state* ds;
        int *de, *dp, *dm;
        void* v;
        CKR(dput(ctx, kBufA, s + o, c, &ds));
        CKR(dbuf(ctx, kBufEps, c * 4, &v)); de = (int*)v;
        CKR(dbuf(ctx, kBufP, c * 4, &v)); dp = (int*)v;
        CKR(dbuf(ctx, kBufM, c * 4, &v)); dm = (int*)v;
        if (csim::launch_exp_sum(launch_of(ctx), nr, (csim::GState*)ds, c, de, dp, dm))
            return fail(ctx, CSIM_ERR_CUDA, "exponential sum launch failed");
        CKR(dget(ctx, s + o, ds, c));
        CKR(dget(ctx, eps + o, de, c));
        CKR(dget(ctx, p + o, dp, c));
        CKR(dget(ctx, m + o, dm, c));
        CKR(finish(ctx));
    }
    return CSIM_OK;
}

extern "C" int csim_shrink(csim_ctx* ctx, int64_t count, csim_state* s, const uint64_t* xi, const int32_t* alpha,
                           int32_t lazy, int32_t* status) {
    if (!ctx || count < 0 || (count && (!s || !xi || !alpha || !status))) return fail(ctx, CSIM_ERR_ARG, "null argument");
    cudaSetDevice(ctx->device);
    int nr;
    CKR(check_states(ctx, s, count, &nr));
    for (int64_t i = 0; i < count; i++)
        if (alpha[i] < 0) return fail(ctx, CSIM_ERR_ARG, "alpha must be >= 0");
    for (int64_t o = 0; o < count; o += kBatch) {
        const int64_t c = std::min(kBatch, count - o);
        csim_state* ds;
        uint64_t* dx;
        int32_t* dal;
        int* dst;
        void* v;
        CKR(dput(ctx, kBufA, s + o, c, &ds));
        CKR(dput(ctx, kBufXi, xi + o, c, &dx));
        CKR(dput(ctx, kBufAlpha, alpha + o, c, &dal));
        CKR(dbuf(ctx, kBufCode, c * 4, &v)); dst = (int*)v;
        if (csim::launch_shrink(launch_of(ctx), nr, (csim::GState*)ds, dx, dal, lazy, c, dst))
            return fail(ctx, CSIM_ERR_CUDA, "shrink launch failed");
        CKR(dget(ctx, s + o, ds, c));
        CKR(dget(ctx, status + o, dst, c));
        CKR(finish(ctx));
    }
    return CSIM_OK;
}

extern "C" int csim_measure_pauli(csim_ctx* ctx, int64_t count, csim_state* s, const int32_t* m, const uint64_t* zeta,
                                  const uint64_t* xi, double* norm) {
    if (!ctx || count < 0 || (count && (!s || !m || !zeta || !xi || !norm)))
        return fail(ctx, CSIM_ERR_ARG, "null argument");
    cudaSetDevice(ctx->device);
    int nr;
    CKR(check_states(ctx, s, count, &nr));
    for (int64_t o = 0; o < count; o += kBatch) {
        const int64_t c = std::min(kBatch, count - o);
        csim_state* ds;
        void *d, *v;
        const size_t bytes = (size_t)c * 8;
        CKR(staged_room(ctx, 1, 2 * bytes + bytes / 2, &v));  // xi, zeta, m
        memcpy(v, xi + o, bytes);
        memcpy((unsigned char*)v + bytes, zeta + o, bytes);
        memcpy((unsigned char*)v + 2 * bytes, m + o, bytes / 2);
        CKR(staged_send(ctx, 1, kBufXi, 2 * bytes + bytes / 2, &v));
        const uint64_t* const dx = (const uint64_t*)v;
        CKR(dput(ctx, kBufA, s + o, c, &ds));
        CKR(dbuf(ctx, kBufCode, c * 4, &d));
        if (csim::launch_measure(launch_of(ctx), nr, (csim::GState*)ds, (const int*)(dx + 2 * c), dx + c, dx, c, (int*)d))
            return fail(ctx, CSIM_ERR_CUDA, "measurePauli launch failed");
        CKR(dget(ctx, s + o, ds, c));
        CKR(finish_with(ctx, d, bytes / 2, &v));
        const int* const code = (const int*)v;
        for (int64_t i = 0; i < c; i++) norm[o + i] = code[i] == 0 ? 0.0 : (code[i] == 1 ? 1.0 : pow(2, -0.5));
    }
    return CSIM_OK;
}

extern "C" int csim_extend(csim_ctx* ctx, int64_t count, csim_state* s, const uint64_t* xi) {
    if (!ctx || count < 0 || (count && (!s || !xi))) return fail(ctx, CSIM_ERR_ARG, "null argument");
    cudaSetDevice(ctx->device);
    int nr;
    CKR(check_states(ctx, s, count, &nr));
    for (int64_t o = 0; o < count; o += kBatch) {
        const int64_t c = std::min(kBatch, count - o);
        csim_state* ds;
        uint64_t* dx;
        CKR(dput(ctx, kBufA, s + o, c, &ds));
        CKR(dput(ctx, kBufXi, xi + o, c, &dx));
        if (csim::launch_extend(launch_of(ctx), nr, (csim::GState*)ds, dx, c))
            return fail(ctx, CSIM_ERR_CUDA, "extend launch failed");
        CKR(dget(ctx, s + o, ds, c));
        CKR(finish(ctx));
    }
    return CSIM_OK;
}

namespace {

int upload_cum(csim_ctx* ctx, int n, double** dcum) {
    double cum[CSIM_MAX_QUBITS + 1];
    cum_table(n, cum);
    return dput(ctx, kBufCum, cum, (size_t)n + 1, dcum);
}

}  // namespace

extern "C" int csim_random_states(csim_ctx* ctx, int32_t n, int64_t count, uint64_t seed, uint64_t first,
                                  csim_state* out) {
    if (!ctx || count < 0 || (count && !out) || n < 1 || n > CSIM_MAX_QUBITS)
        return fail(ctx, CSIM_ERR_ARG, "bad argument");
    cudaSetDevice(ctx->device);
    for (int64_t o = 0; o < count; o += kBatch) {
        const int64_t c = std::min(kBatch, count - o);
        double* dcum;
        void* v;
        CKR(upload_cum(ctx, n, &dcum));
        CKR(dbuf(ctx, kBufA, c * sizeof(csim_state), &v));
        if (csim::launch_random_states(launch_of(ctx), n, c, 0, seed, first + o, nullptr, nullptr, dcum,
                                       (csim::GState*)v, nullptr))
            return fail(ctx, CSIM_ERR_CUDA, "random state launch failed");
        CKR(dget(ctx, out + o, (const csim_state*)v, c));
        CKR(finish(ctx));
    }
    return CSIM_OK;
}

extern "C" int csim_random_states_replay(csim_ctx* ctx, int32_t n, int64_t count, const uint32_t* words,
                                         const int64_t* offsets, csim_state* out) {
    if (!ctx || count < 0 || (count && (!out || !words || !offsets)) || n < 1 || n > CSIM_MAX_QUBITS)
        return fail(ctx, CSIM_ERR_ARG, "bad argument");
    cudaSetDevice(ctx->device);
    if (count == 0) return CSIM_OK;
    for (int64_t i = 0; i < count; i++)
        if (offsets[i + 1] < offsets[i] || offsets[i] < 0) return fail(ctx, CSIM_ERR_ARG, "offsets not increasing");
    const int64_t nw = offsets[count];
    std::vector<int64_t> rel(count + 1), consumed(count);
    for (int64_t i = 0; i <= count; i++) rel[i] = offsets[i] - offsets[0];
    double* dcum;
    uint32_t* dw;
    int64_t *doff, *dcon;
    void* v;
    CKR(upload_cum(ctx, n, &dcum));
    CKR(dput(ctx, kBufWords, words + offsets[0], (size_t)(nw - offsets[0]), &dw));
    CKR(dput(ctx, kBufOffsets, rel.data(), rel.size(), &doff));
    CKR(dbuf(ctx, kBufConsumed, count * 8, &v)); dcon = (int64_t*)v;
    CKR(dbuf(ctx, kBufA, count * sizeof(csim_state), &v));
    if (csim::launch_random_states(launch_of(ctx), n, count, 1, 0, 0, dw, doff, dcum, (csim::GState*)v, dcon))
        return fail(ctx, CSIM_ERR_CUDA, "random state launch failed");
    CKR(dget(ctx, out, (const csim_state*)v, count));
    CKR(dget(ctx, consumed.data(), dcon, count));
    CKR(finish(ctx));
    for (int64_t i = 0; i < count; i++)
        if (consumed[i] != rel[i + 1] - rel[i])
            return fail(ctx, CSIM_ERR_ARG, "state %lld consumed %lld words, segment holds %lld", (long long)i,
                        (long long)consumed[i], (long long)(rel[i + 1] - rel[i]));
    return CSIM_OK;
}

extern "C" int csim_prep_h(csim_ctx* ctx, int32_t t, int64_t count, const int64_t* idx, csim_state* out) {
    if (!ctx || count < 0 || (count && (!idx || !out)) || t < 1 || t > CSIM_MAX_QUBITS)
        return fail(ctx, CSIM_ERR_ARG, "bad argument");
    cudaSetDevice(ctx->device);
    const int64_t lim = (int64_t)1 << ((t + 1) / 2);
    for (int64_t i = 0; i < count; i++)
        if (idx[i] < 0 || idx[i] >= lim) return fail(ctx, CSIM_ERR_ARG, "term index out of range");
    for (int64_t o = 0; o < count; o += kBatch) {
        const int64_t c = std::min(kBatch, count - o);
        int64_t* di;
        void* v;
        CKR(dput(ctx, kBufIdx, idx + o, c, &di));
        CKR(dbuf(ctx, kBufA, c * sizeof(csim_state), &v));
        if (csim::launch_prep(launch_of(ctx), t, 1, nullptr, di, c, (csim::GState*)v))
            return fail(ctx, CSIM_ERR_CUDA, "prepH launch failed");
        CKR(dget(ctx, out + o, (const csim_state*)v, c));
        CKR(finish(ctx));
    }
    return CSIM_OK;
}

extern "C" int csim_prep_l(csim_ctx* ctx, int32_t t, const uint64_t* L, int32_t k, int64_t count, const int64_t* idx,
                           csim_state* out) {
    if (!ctx || count < 0 || (count && (!idx || !out || !L)) || t < 1 || t > CSIM_MAX_QUBITS || k < 0 || k > 62)
        return fail(ctx, CSIM_ERR_ARG, "bad argument");
    cudaSetDevice(ctx->device);
    for (int64_t o = 0; o < count; o += kBatch) {
        const int64_t c = std::min(kBatch, count - o);
        std::vector<uint64_t> cw(c);
        for (int64_t i = 0; i < c; i++) {
            if (idx[o + i] < 0 || idx[o + i] >= ((int64_t)1 << k)) return fail(ctx, CSIM_ERR_ARG, "term index out of range");
            cw[i] = codeword(idx[o + i], L, k) & (t >= 64 ? ~0ull : ((1ull << t) - 1));
        }
        uint64_t* dcw;
        void* v;
        CKR(dput(ctx, kBufCodewords, cw.data(), cw.size(), &dcw));
        CKR(dbuf(ctx, kBufA, c * sizeof(csim_state), &v));
        if (csim::launch_prep(launch_of(ctx), t, 0, dcw, nullptr, c, (csim::GState*)v))
            return fail(ctx, CSIM_ERR_CUDA, "prepL launch failed");
        CKR(dget(ctx, out + o, (const csim_state*)v, c));
        CKR(finish(ctx));
    }
    return CSIM_OK;
}

// ---------------------------------------------------------------- hot path
namespace {

// the terms |phi_j>, j in [j0, j0+nj): codewords (|L>) or prepared states (|H^t>).
// ordered: all 2^k codewords in ordered_codewords' order (sums over all terms only)
// G-slot bounds of the block-prefix kernel's occupancy classes for t, most
// zeros first: t, then each largest zero bound that lets one more block per SM
// be resident.  Classes that would hold under 3% of the 2^k codewords of L
// merge into the next heavier class (a launch's tail costs more than its
// occupancy gains).
int occupancy_bounds(csim_ctx* ctx, int t, const uint64_t* L, int k, std::vector<int>& bounds) {
    bounds.assign(1, t);
    int last = csim::terms_tp_occupancy(t, t);
    if (last < 1) return fail(ctx, CSIM_ERR_CUDA, "occupancy query failed");
    for (int g = t - 1; g >= 0; g--) {
        const int o = csim::terms_tp_occupancy(t, g);
        if (o < 1) return fail(ctx, CSIM_ERR_CUDA, "occupancy query failed");
        if (o > last) {
            bounds.push_back(g);
            last = o;
        }
    }
    // zero counts of the codewords (Gray code walk)
    std::vector<int64_t> hist(CSIM_MAX_QUBITS + 2, 0);
    uint64_t x = 0;
    hist[(size_t)t]++;
    for (int64_t i = 1; i < ((int64_t)1 << k); i++) {
        x ^= L[k - 1 - __builtin_ctzll((unsigned long long)i)];
        hist[(size_t)(t - __builtin_popcountll(x))]++;
    }
    const int64_t chi = (int64_t)1 << k;
    for (bool merged = true; merged && bounds.size() > 1;) {
        merged = false;
        for (size_t c = 1; c < bounds.size(); c++) {
            const int hi = bounds[c], lo = c + 1 < bounds.size() ? bounds[c + 1] : -1;
            int64_t n = 0;
            for (int z = lo + 1; z <= hi; z++) n += hist[(size_t)z];
            if (n * 100 < 3 * chi) {
                bounds.erase(bounds.begin() + (long)c);
                merged = true;
                break;
            }
        }
    }
    return 0;
}

// ordered with tn: the table of tn's kernel -- ordered_codewords with light
// bound tn->light (block-prefix kernel), or run_ordered_codewords with runs of
// tn->per_thread (run kernel); ctx->cw_split is then the light launch's first term.
int stage_terms(csim_ctx* ctx, int t, int exact, const uint64_t* L, int k, int64_t j0, int64_t nj,
                uint64_t** dcw, csim_state** dphis, bool ordered = false, const TpTune* tn = nullptr) {
    *dcw = nullptr;
    *dphis = nullptr;
    void* v;
    if (!exact && ordered && j0 == 0 && nj == ((int64_t)1 << k)) {
        const TpTune d0 = default_tune(t);
        if (!tn) tn = &d0;
        std::vector<uint64_t> key(L, L + k);
        key.push_back((uint64_t)k);
        key.push_back((uint64_t)t);
        key.push_back((uint64_t)tn->light);
        key.push_back((uint64_t)(tn->kernel == 3 ? 0 : tn->kernel));  // the direct kernel walks kernel 0's order
        key.push_back((uint64_t)(tn->kernel ? tn->per_thread : 0));
        if (key != ctx->cw_key || !ctx->buf[kBufCwOrdered]) {
            std::vector<uint64_t> cw;
            int64_t split;
            if (tn->kernel == 1) {
                split = run_ordered_codewords(L, k, t, tn->per_thread, tn->light, cw);
            } else if (tn->kernel == 2) {
                CKR(occupancy_bounds(ctx, t, L, k, ctx->cw_bounds));
                ordered_codewords_classes(L, k, t, ctx->cw_bounds, cw, ctx->cw_starts);
                split = 0;
            } else {
                ordered_codewords(L, k, t, tn->light, cw);
                split = light_split(cw, t, tn->light);
            }
            uint64_t* d;
            CKR(dput(ctx, kBufCwOrdered, cw.data(), cw.size(), &d));
            ctx->cw_key = key;
            ctx->cw_split = split;
        }
        *dcw = (uint64_t*)ctx->buf[kBufCwOrdered];
        return 0;
    }
    if (!exact) {
        uint64_t* dL;
        CKR(dput(ctx, kBufL, L, (size_t)k, &dL));
        CKR(dbuf(ctx, kBufCodewords, nj * 8, &v));
        if (csim::launch_codewords(launch_of(ctx), dL, k, j0, nj, (uint64_t*)v))
            return fail(ctx, CSIM_ERR_CUDA, "codeword launch failed");
        *dcw = (uint64_t*)v;
        return 0;
    }
    std::vector<int64_t> idx(nj);
    for (int64_t i = 0; i < nj; i++) idx[i] = j0 + i;
    int64_t* di;
    CKR(dput(ctx, kBufIdx, idx.data(), idx.size(), &di));
    CKR(dbuf(ctx, kBufPhis, nj * sizeof(csim_state), &v));
    if (csim::launch_prep(launch_of(ctx), t, 1, nullptr, di, nj, (csim::GState*)v))
        return fail(ctx, CSIM_ERR_CUDA, "prepH launch failed");
    *dphis = (csim_state*)v;
    return 0;
}


}  // namespace

extern "C" int csim_term_products(csim_ctx* ctx, int32_t t, int32_t exact, const uint64_t* L, int32_t k,
                                  int64_t ntheta, const csim_state* theta, int64_t j0, int64_t nj, int32_t* eps,
                                  int32_t* p, int32_t* m) {
    if (!ctx || ntheta < 0 || nj < 0 || j0 < 0 || (ntheta && nj && (!theta || !eps || !p || !m)))
        return fail(ctx, CSIM_ERR_ARG, "bad argument");
    cudaSetDevice(ctx->device);
    CKR(check_code(ctx, t, exact, L, k));
    const int64_t chi = exact ? ((int64_t)1 << ((t + 1) / 2)) : ((int64_t)1 << k);
    if (j0 + nj > chi) return fail(ctx, CSIM_ERR_ARG, "term range beyond chi");
    if (ntheta == 0 || nj == 0) return CSIM_OK;
    int nr;
    CKR(check_states(ctx, theta, ntheta, &nr, t));
    // the thread-per-pair kernel needs a symmetric J block (always true of drawn states)
    bool sym = true;
    for (int64_t a = 0; a < ntheta && sym; a++)
        for (int x = 0; x < theta[a].k && sym; x++)
            for (int y = 0; y < theta[a].k; y++)
                if (((theta[a].J[x] >> y) & 1) != ((theta[a].J[y] >> x) & 1)) {
                    sym = false;
                    break;
                }
    TpTune tn = default_tune(t);
    if (!exact && ctx->pair_kernel != 1 && sym) CKR(tune_for(ctx, t, &tn));
    uint64_t* dcw;
    csim_state* dphis;
    CKR(stage_terms(ctx, t, exact, L, k, j0, nj, &dcw, &dphis));
    const int64_t rows = std::max<int64_t>(1, std::min<int64_t>(ntheta, (1 << 22) / nj + 1));
    for (int64_t o = 0; o < ntheta; o += rows) {
        const int64_t c = std::min(rows, ntheta - o);
        csim_state* dth;
        void* v;
        CKR(dput(ctx, kBufA, theta + o, c, &dth));
        CKR(dbuf(ctx, kBufEps, c * nj * 4, &v));
        int* de = (int*)v;
        CKR(dbuf(ctx, kBufP, c * nj * 4, &v));
        int* dp = (int*)v;
        CKR(dbuf(ctx, kBufM, c * nj * 4, &v));
        int* dm = (int*)v;
        const int rc = (!exact && ctx->pair_kernel != 1 && sym)
                           ? csim::launch_terms_tp(launch_of(ctx), t, t, dcw, (const csim::GState*)dth, nullptr, c, j0,
                                                   nj, tn.per_thread, 2 * t, nullptr, 0, 0, de,
                                                   dp, dm)
                           : csim::launch_terms(launch_of(ctx), nr, exact ? 1 : 0, dcw, (const csim::GState*)dphis,
                                                (const csim::GState*)dth, nullptr, c, j0, nj, 64, 2 * t, nullptr,
                                                nullptr, de, dp, dm);
        if (rc) return fail(ctx, CSIM_ERR_CUDA, "term launch failed");
        CKR(dget(ctx, eps + o * nj, de, c * nj));
        CKR(dget(ctx, p + o * nj, dp, c * nj));
        CKR(dget(ctx, m + o * nj, dm, c * nj));
        CKR(finish(ctx));
    }
    return CSIM_OK;
}

namespace {


// The tree plan of a decomposition (|H^t> if exact, code L otherwise) for `count`
// states, kept from call to call while the decomposition is the same
void tree_plan_for(csim_ctx* ctx, int exact, const uint64_t* L, int k, int t, int64_t count) {
    std::vector<uint64_t> key;
    if (!exact) key.assign(L, L + k);
    key.push_back(exact ? ~0ull : (uint64_t)k);
    key.push_back((uint64_t)t);
    if (key != ctx->tree_key) {
        ctx->tree_key.clear();
        ctx->tree_plan = csim::tree::Plan();
        if (exact) csim::tree::build_pairs(t, ctx->tree_plan);
        else csim::tree::build_chain(L, k, t, ctx->tree_plan);
        ctx->tree_key = key;
    }
    csim::tree::choose_levels(ctx->tree_plan, count);
}

// A call's inputs on the device, one upload: the tree's job tables, the projector's rows,
// the d-distribution of randomStabilizerState, the projection factors, the tree plan, the
// code and the zero head of the results, which lie behind them
struct CallInputs {
    const int* pm;
    const uint64_t *pz, *px;
    const double *cum, *factor;
    const unsigned char* plan;
    const uint64_t* L;
    unsigned char* results;  // `head` bytes that are zero once the inputs are sent, then the rest
    unsigned char *host, *dev;
    size_t bytes;
};
constexpr size_t kCallJobs = 16 << 10;  // room for job tables in front

// Makes the inputs, with room for `results` bytes (head of them zero); send_inputs uploads them
int make_inputs(csim_ctx* ctx, const csim_projector* P, const csim::tree::Plan* plan, size_t head, size_t results,
                CallInputs* in, const uint64_t* L = nullptr, int k = 0) {
    const size_t n = (size_t)P->nstabs;
    const size_t o_pz = kCallJobs, o_px = o_pz + 8 * n, o_cum = o_px + 8 * n, o_factor = o_cum + 8 * (CSIM_MAX_QUBITS + 1),
                 o_plan = o_factor + 8 * (n + 1), o_L = o_plan + kTreePlanBytes, o_pm = o_L + 8 * (size_t)k,
                 o_res = (o_pm + 4 * n + 15) / 16 * 16;
    void* v;
    CKR(staged_room(ctx, 1, o_res + head, &v));
    unsigned char* const h = (unsigned char*)v;
    if (n) memcpy(h + o_pz, P->zs, 8 * n);
    if (n) memcpy(h + o_px, P->xs, 8 * n);
    cum_table(P->nqubits, (double*)(h + o_cum));
    for (size_t c = 0; c <= n; c++) ((double*)(h + o_factor))[c] = sqrt_half_power((int)c);
    if (plan) tree_plan_image(*plan, h + o_plan);
    else memset(h + o_plan, 0, kTreePlanBytes);
    if (k) memcpy(h + o_L, L, 8 * (size_t)k);
    for (size_t r = 0; r < n; r++) ((int32_t*)(h + o_pm))[r] = phase_m(P->phase[r]);
    memset(h + o_pm + 4 * n, 0, o_res + head - (o_pm + 4 * n));
    CKR(dbuf(ctx, kBufCall, o_res + results, &v));
    unsigned char* const d = (unsigned char*)v;
    *in = CallInputs{(const int*)(d + o_pm), (const uint64_t*)(d + o_pz), (const uint64_t*)(d + o_px),
                     (const double*)(d + o_cum), (const double*)(d + o_factor), d + o_plan, (const uint64_t*)(d + o_L),
                     d + o_res, h, d, o_res + head};
    return 0;
}
// Uploads them with the job tables (*djobs; larger ones go alone)
int send_inputs(csim_ctx* ctx, const CallInputs& in, const std::vector<unsigned char>& jobs, unsigned char** djobs) {
    size_t from = kCallJobs;
    if (!jobs.empty() && jobs.size() <= kCallJobs) {
        from = (kCallJobs - jobs.size()) / 256 * 256;
        memcpy(in.host + from, jobs.data(), jobs.size());
        *djobs = in.dev + from;
    } else if (!jobs.empty()) {
        CKR(staged_put(ctx, 0, kBufTreeJobs, jobs.data(), jobs.size(), djobs));
    }
    CK(cudaMemcpyAsync(in.dev + from, in.host + from, in.bytes - from, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaEventRecord(ctx->pin_ev[1], ctx->stream));
    ctx->stats.h2d_bytes += (int64_t)(in.bytes - from);
    return 0;
}

// The raw words of the next `count` states and their offsets in pinned slot 3, and their
// upload; *chain: where they end
int put_state_words(csim_ctx* ctx, int t, const double* cum, int64_t count, const uint32_t** dwords,
                    const int64_t** doffs, csim::DrawChain* chain) {
    const size_t head = (size_t)(count + 1) * 8;
    void* v;
    CKR(staged_room(ctx, 3, head + (kRawHistory + (size_t)count * state_words(t)) * 4, &v));
    RawWords w{(uint32_t*)((unsigned char*)v + head), kRawHistory, (ctx->pin_cap[3] - head) / 4};
    ctx->lr.history(w.p);
    auto grow = [&](size_t more) {
        const size_t cap = w.cap + w.cap / 2 + more;
        if (staged_grow(ctx, 3, head + cap * 4, head + w.n * 4, &v)) return false;
        w.p = (uint32_t*)((unsigned char*)v + head);
        w.cap = cap;
        return true;
    };
    for (int64_t i = 0; i < count; i++) {
        ((int64_t*)v)[i] = (int64_t)w.n;
        if (!draw_state_words(w, t, cum, grow)) return CSIM_ERR_NOMEM;
    }
    ((int64_t*)v)[count] = (int64_t)w.n;
    chain->states = count;
    memcpy(chain->history, w.p + w.n - kRawHistory, sizeof(chain->history));
    CKR(staged_send(ctx, 3, kBufWords, head + w.n * 4, &v));
    *doffs = (const int64_t*)v;
    *dwords = (const uint32_t*)((unsigned char*)v + head);
    return 0;
}

// The same on the device: *chain (device memory) counts the states that the words suffice for
int make_state_words(csim_ctx* ctx, int t, const double* cum, int64_t count, const uint32_t** dwords,
                     const int64_t** doffs, csim::DrawChain* chain) {
    csim::DrawJob j{};
    csim::draw_job(t, cum, count, ctx->draw_percent, j);
    ctx->lr.history(j.history);
    void* v;
    CKR(dbuf(ctx, kBufWords, (kRawHistory + (size_t)j.words) * 4, &v));
    j.buf = (uint32_t*)v;
    CKR(dbuf(ctx, kBufLengths, (size_t)j.padded() * 2, &v));
    j.len = (uint16_t*)v;
    CKR(dbuf(ctx, kBufChainMaps, (size_t)j.map_words() * 4, &v));
    j.map = (uint32_t*)v;
    CKR(dbuf(ctx, kBufOffsets, (size_t)(count + 1) * 8, &v));
    j.offs = (int64_t*)v;
    j.chain = chain;
    if (csim::launch_draws(launch_of(ctx), &j, 1)) return fail(ctx, CSIM_ERR_CUDA, "word launch failed");
    *dwords = j.buf;
    *doffs = j.offs;
    return 0;
}

// Draws `count` states, `batch` at a time, projects them onto P, sums their terms on the GPU, and
// returns singleProjectorSample's value for each (innerprod.c:88-144).  *done: the states whose values
// there are, also on an error (the streams stand behind them then).
int sample_batches(csim_ctx* ctx, const csim_projector* P, const uint64_t* L, int k, int exact, int64_t count,
                   int rng, uint64_t seed, int64_t batch, double* values, int64_t* done) {
    const int t = P->nqubits;
    CKR(check_code(ctx, t, exact, L, k));
    if (rng != CSIM_RNG_LIBC && rng != CSIM_RNG_PHILOX) return fail(ctx, CSIM_ERR_ARG, "unknown rng %d", rng);
    const bool tree = use_tree(ctx, t, exact, k);
    const bool tp = !exact && !tree && ctx->pair_kernel != 1;
    TpTune tn = default_tune(t);
    if (tp && count > 0) CKR(tune_for(ctx, t, &tn, P, L, k));  // before any draw: tuning leaves the streams as they are
    // the run kernel takes whole blocks of 64 runs
    if (tn.kernel == 1 && (exact || ((int64_t)1 << k) % (64 * (int64_t)tn.per_thread) != 0)) tn = default_tune(t);
    if ((tn.kernel == 2 || tn.kernel == 3) && exact) tn = default_tune(t);
    if (rng == CSIM_RNG_LIBC && seed != CSIM_SEED_CONTINUE) ctx->lr.seed((uint32_t)seed);
    if (rng == CSIM_RNG_PHILOX && seed != CSIM_SEED_CONTINUE) {
        ctx->philox_seed = seed;
        ctx->philox_next = 0;
    }
    if (count <= 0) return 0;
    const int nr = t > 32 ? 2 : 1;
    const int64_t chi = exact ? ((int64_t)1 << ((t + 1) / 2)) : ((int64_t)1 << k);
    const int P2 = 2 * t;
    const int64_t chunk = chunk_for(chi);
    const int pt = tn.per_thread;
    const int64_t shape_count = std::min(count, batch);
    if (tree) tree_plan_for(ctx, exact, L, k, t, shape_count);
    const int64_t nchunks = tree ? tree_leaf_shape(ctx->tree_plan, shape_count).parts_per_state
                                 : (tp ? csim::terms_tp_blocks(chi, pt) : (chi + chunk - 1) / chunk);

    const bool libc = rng == CSIM_RNG_LIBC;
    constexpr size_t head = 16 + (sizeof(csim::DrawChain) + 15) / 16 * 16;  // results: live states, error, chain, values
    CallInputs in;
    CKR(make_inputs(ctx, P, tree ? &ctx->tree_plan : nullptr, 16, head + (size_t)std::min(count, batch) * 8, &in));
    if (!tree) CKR(send_inputs(ctx, in, {}, nullptr));
    unsigned char* const dres = in.results;
    double hcum[CSIM_MAX_QUBITS + 1];
    cum_table(t, hcum);
    uint64_t* dcw = nullptr;
    csim_state* dphis = nullptr;
    if (!tree) CKR(stage_terms(ctx, t, exact, L, k, 0, chi, &dcw, &dphis, /*ordered=*/true, &tn));
    const int dsl = ctx->direct_slots > 0 ? std::min(t, ctx->direct_slots) : direct_slots(t);
    unsigned char* dscr = nullptr;
    size_t scr_bytes = 0;
    if (tp && tn.kernel == 1) {
        scr_bytes = csim::terms_runs_scratch_bytes(ctx->num_sms, t, std::min(t, tn.light));
        if (!scr_bytes) return fail(ctx, CSIM_ERR_CUDA, "run kernel occupancy query failed");
        void* sv;
        CKR(dbuf(ctx, kBufRunScratch, scr_bytes, &sv));
        dscr = (unsigned char*)sv;
    }

    TreeRun run;
    std::vector<unsigned char> jobs;
    std::vector<int> code;
    std::vector<__int128> acc;
    bool sent = !tree;
    bool ran_out = false;  // of the device's words: the batch runs again with the host's, and its draws' flag is cleared
    for (int64_t o = 0; o < count;) {
        const int64_t c = std::min(batch, count - o);
        void* v;
        csim::GState* dth = nullptr;  // the tree's states stay in registers
        if (!tree) {
            CKR(dbuf(ctx, kBufA, c * sizeof(csim_state), &v));
            dth = (csim::GState*)v;
        }
        CKR(dbuf(ctx, kBufCode, c * 4, &v));
        int* dcode = (int*)v;
        void* dcanon = nullptr;
        int *dcode_dir = nullptr, *dcode_rest = nullptr, *drest = nullptr;
        if (tp && tn.kernel == 3) {
            CKR(dbuf(ctx, kBufCanon, (size_t)c * csim::canon_bytes(), &dcanon));
            CKR(dbuf(ctx, kBufCodeDirect, c * 4, &v));
            dcode_dir = (int*)v;
            CKR(dbuf(ctx, kBufCodeRest, c * 4, &v));
            dcode_rest = (int*)v;
            CKR(dbuf(ctx, kBufRestCount, 4, &v));  // live states of a batch left to the block-prefix kernel
            drest = (int*)v;
        }
        const size_t nparts = (size_t)c * nchunks * 4;
        CKR(dbuf(ctx, kBufParts, nparts * sizeof(__int128), &v));
        __int128* dpart = (__int128*)v;
        CK(cudaEventRecord(ctx->ev[0], ctx->stream));
        if (!tree) CK(cudaMemsetAsync(dpart, 0, nparts * sizeof(__int128), ctx->stream));
        const bool on_host = libc && (ran_out || words_on_host(t, c));
        csim::DrawChain chain{};
        csim::TreeDraw draw{};
        if (libc) {
            const uint32_t* dw;
            const int64_t* doff;
            if (on_host) CKR(put_state_words(ctx, t, hcum, c, &dw, &doff, &chain));
            else CKR(make_state_words(ctx, t, hcum, c, &dw, &doff, (csim::DrawChain*)(dres + 16)));
            draw = csim::TreeDraw{2, P->nstabs, 0, 0, dw, doff, in.cum, in.pm, in.pz, in.px, dcode, nullptr, 0, 0};
            if (!tree && csim::launch_random_states(launch_of(ctx), t, c, 2, 0, 0, dw, doff, in.cum, dth, nullptr))
                return fail(ctx, CSIM_ERR_CUDA, "random state launch failed");
        } else {
            draw = csim::TreeDraw{0, P->nstabs, ctx->philox_seed, ctx->philox_next, nullptr, nullptr, in.cum, in.pm,
                                  in.pz, in.px, dcode, nullptr, 0, 0};
            if (!tree && csim::launch_random_states(launch_of(ctx), t, c, 0, ctx->philox_seed, ctx->philox_next,
                                                    nullptr, nullptr, in.cum, dth, nullptr))
                return fail(ctx, CSIM_ERR_CUDA, "random state launch failed");
        }
        if (!tree && csim::launch_project(launch_of(ctx), nr, dth, c, P->nstabs, in.pm, in.pz, in.px, dcode))
            return fail(ctx, CSIM_ERR_CUDA, "projection launch failed");
        if (tp && tn.kernel == 3) {
            CK(cudaMemsetAsync(drest, 0, 4, ctx->stream));
            if (csim::launch_canon(launch_of(ctx), dth, dcode, c, dsl, (unsigned char*)dcanon, dcode_dir, dcode_rest,
                                   drest))
                return fail(ctx, CSIM_ERR_CUDA, "pivot-form launch failed");
        }
        if (!tree) CK(cudaEventRecord(ctx->ev[1], ctx->stream));
        int rc = 0;
        if (tree) {
            TreeGroup g;
            g.plan = &ctx->tree_plan;
            g.dplan = in.plan;
            g.draw = draw;
            g.count = c;
            g.shape_count = shape_count;
            g.part = dpart;
            void* scratch;
            unsigned char* djobs;
            CKR(run.reserve({g}, [&](size_t bytes) { return tree_scratch(ctx, bytes, kTreeScratchMax, &scratch); }));
            run.build((unsigned char*)scratch, jobs);
            if (!sent) {
                CKR(send_inputs(ctx, in, jobs, &djobs));
                sent = true;
            } else {
                CKR(staged_put(ctx, 0, kBufTreeJobs, jobs.data(), jobs.size(), &djobs));
                CK(cudaMemsetAsync(dres, 0, 16, ctx->stream));
            }
            // the event that starts the pair kernels' time is recorded behind the first roots
            rc = run.launch(launch_of(ctx), djobs, ctx->ev[1]);
        } else if (tp && tn.kernel == 2) {
            // one launch per occupancy class; class c's launch starts at its first whole item
            const int64_t span = 64 * (int64_t)pt;
            const int nc = (int)ctx->cw_bounds.size();
            for (int cl = 0; cl < nc; cl++) {
                const int64_t a0 = cl == 0 ? 0 : (ctx->cw_starts[(size_t)cl] + span - 1) / span * span;
                const int64_t b0 = cl + 1 < nc ? (ctx->cw_starts[(size_t)cl + 1] + span - 1) / span * span : chi;
                const int64_t aa = std::min(a0, chi), bb = std::min(b0, chi);
                if (aa < bb)
                    rc |= csim::launch_terms_tp(launch_of(ctx), t, ctx->cw_bounds[(size_t)cl], dcw + aa, dth,
                                                dcode, c, aa, bb - aa, pt, P2, dpart, nchunks, aa / span,
                                                nullptr, nullptr, nullptr);
            }
        } else if (tp && tn.kernel == 1) {
            // run kernel: terms [0, jb) in heavy runs, [jb, chi) in runs whose codewords have at most
            // tn.light zeros below their run's agreed top bits
            const int64_t span = 64 * (int64_t)pt;
            const int64_t jb = ctx->cw_split;
            if (jb > 0)
                rc |= csim::launch_terms_runs(launch_of(ctx), t, t, dcw, dth, dcode, c, 0, jb, pt, P2, dpart,
                                              nchunks, 0, dscr, scr_bytes);
            if (jb < chi)
                rc |= csim::launch_terms_runs(launch_of(ctx), t, std::min(t, tn.light), dcw + jb, dth, dcode, c,
                                              jb, chi - jb, pt, P2, dpart, nchunks, jb / span, dscr, scr_bytes);
        } else if (tp) {
            // direct kernel: every term of the states it takes; the rest (or all, for kernel 0) below
            const int* rcode = dcode;
            if (tn.kernel == 3) {
                // above 32 qubits the table's heavy part [0, cw_split) holds the codewords of at most 32
                // ones (direct_light), whose pairs need 32 J rows: a launch of its own with smaller
                // per-pair memory; the rest (from its first whole item) with rows for every coordinate
                const unsigned char* cb = (const unsigned char*)dcanon;
                const int64_t span = 64 * (int64_t)pt;
                const int64_t jn = t > 32 ? std::min(chi, ctx->cw_split / span * span) : 0;
                if (jn > 0)
                    rc |= csim::launch_terms_direct(launch_of(ctx), t, 32, dsl, dcw, cb, dcode_dir, c, 0,
                                                    jn, pt, P2, dpart, nchunks, 0);
                if (jn < chi)
                    rc |= csim::launch_terms_direct(launch_of(ctx), t, t, dsl, dcw + jn, cb, dcode_dir, c,
                                                    jn, chi - jn, pt, P2, dpart, nchunks, jn / span);
                rcode = dcode_rest;
            }
            // terms [0, jb): every zero count; terms [jb, chi): at most tn.light zeros (for the direct
            // kernel's fallback, gated on the batch having a state left to it)
            const int64_t span = 64 * (int64_t)pt;
            const int64_t jb = std::min(chi, (ctx->cw_split + span - 1) / span * span);
            if (jb > 0)
                rc |= csim::launch_terms_tp(launch_of(ctx), t, t, dcw, dth, rcode, c, 0, jb, pt, P2, dpart,
                                            nchunks, 0, nullptr, nullptr, nullptr, drest);
            if (jb < chi)
                rc |= csim::launch_terms_tp(launch_of(ctx), t, tn.light, dcw + jb, dth, rcode, c, jb,
                                            chi - jb, pt, P2, dpart, nchunks, jb / span, nullptr, nullptr,
                                            nullptr, drest);
        } else {
            rc = csim::launch_terms(launch_of(ctx), nr, exact ? 1 : 0, dcw, (const csim::GState*)dphis, dth,
                                    dcode, c, 0, chi, (int)chunk, P2, dpart, nullptr, nullptr, nullptr, nullptr);
        }
        if (rc) return fail(ctx, CSIM_ERR_CUDA, "term launch failed");
        CK(cudaEventRecord(ctx->ev[2], ctx->stream));
        if (tree) {
            if (csim::launch_tree_values(launch_of(ctx), dpart, c, nchunks, t, dcode, in.factor, (double*)(dres + head),
                                         (unsigned long long*)dres))
                return fail(ctx, CSIM_ERR_CUDA, "reduce launch failed");
            CK(cudaEventRecord(ctx->ev[3], ctx->stream));
            CKR(staged_room(ctx, 2, head + (size_t)c * 8, &v));
            CKR(dget(ctx, (unsigned char*)v, dres, head + (size_t)c * 8));
            CK(cudaStreamSynchronize(ctx->stream));
            CK(cudaGetLastError());
            if (libc && !on_host) memcpy(&chain, (const unsigned char*)v + 16, sizeof(chain));
            if (libc && chain.states < c) {
                CK(cudaMemsetAsync(ctx->d_err, 0, sizeof(int), ctx->stream));
                ran_out = true;
                continue;
            }
            CKR(error_status(ctx, ((const int*)v)[2]));
            CKR(stats_batch(ctx));
            const int64_t live = *(const int64_t*)v;
            memcpy(values + o, (const unsigned char*)v + head, (size_t)c * 8);
            if (libc) ctx->lr.set_history(chain.history);
            else ctx->philox_next += c;
            ctx->stats.states += c;
            ctx->stats.states_live += live;
            ctx->stats.pairs += live * chi;
            *done = o += c;
            ran_out = false;
            continue;
        }
        CKR(dbuf(ctx, kBufAcc, (size_t)c * 4 * sizeof(__int128), &v));
        __int128* dacc = (__int128*)v;
        if (csim::launch_reduce_parts(launch_of(ctx), dpart, c, nchunks, dacc))
            return fail(ctx, CSIM_ERR_CUDA, "reduce launch failed");
        CK(cudaEventRecord(ctx->ev[3], ctx->stream));
        code.resize(c);
        acc.resize(c * 4);
        CKR(dget(ctx, code.data(), dcode, c));
        CKR(dget(ctx, acc.data(), dacc, c * 4));
        if (libc && !on_host) {
            CKR(dget(ctx, &chain, (const csim::DrawChain*)(dres + 16), 1));
            CK(cudaStreamSynchronize(ctx->stream));
            if (chain.states < c) {
                CK(cudaMemsetAsync(ctx->d_err, 0, sizeof(int), ctx->stream));
                ran_out = true;
                continue;
            }
        }
        CKR(finish(ctx));
        if (libc) ctx->lr.set_history(chain.history);
        else ctx->philox_next += c;
        CKR(stats_batch(ctx));
        const double scale = pow(2, t);
        ctx->stats.states += c;
        for (int64_t i = 0; i < c; i++) {
            if (code[i] < 0) {
                values[o + i] = 0;
                continue;
            }
            ctx->stats.states_live++;
            ctx->stats.pairs += chi;
            double re, im;
            zomega_to_complex(&acc[4 * i], P2, &re, &im);
            const double pf = sqrt_half_power(code[i]);
            const double a = re * pf, b = im * pf;
            values[o + i] = scale * (a * a + b * b);
        }
        *done = o += c;
        ran_out = false;
    }
    return 0;
}

// sample_batches with batches that there is memory for
int sample_values(csim_ctx* ctx, const csim_projector* P, const uint64_t* L, int k, int exact, int64_t count,
                  int rng, uint64_t seed, double* values) {
    int64_t o = 0;
    for (int64_t batch = std::min<int64_t>(count, 1 << 14);; batch = std::max<int64_t>(64, batch / 4)) {
        int64_t done = 0;
        const int rc = sample_batches(ctx, P, L, k, exact, count - o, rng, o ? CSIM_SEED_CONTINUE : seed, batch, values + o,
                                      &done);
        o += done;
        if (rc != CSIM_ERR_NOMEM || batch <= 64) return rc;
        CK(cudaMemsetAsync(ctx->d_err, 0, sizeof(int), ctx->stream));  // (states whose words ran out)
        CK(cudaStreamSynchronize(ctx->stream));
    }
}

}  // namespace

namespace csim_host {

namespace {

// Tuned launch parameters per device and t, shared by every context of the
// process (a property of the device model and the kernels, not of a context)
struct TuneTable {
    TpTune p[CSIM_MAX_QUBITS + 1];
    bool done[CSIM_MAX_QUBITS + 1] = {};
    double ms[CSIM_MAX_QUBITS + 1] = {};
};
std::mutex g_tune_mu;
TuneTable g_tune[64];

// One tuning pass for the t bucket [4b, 4b + 3] of t (t = 1..3 in bucket 0).
// It runs the sampler's own path (draw, project, heavy and light pair
// launches) on the workload about to run -- projector P and code L of k rows,
// when given for this t -- or on a synthetic one of the bucket's largest t
// (counter-based states projected onto ceil(0.7 t) random Pauli rows, a random
// code of min(t, 14) rows).  The states are the tuner's own counter-based
// draws, enough for about 2^25 pairs per trial (at least 16 waves of the
// largest items).  Candidates: terms per thread 16 or 32 (items of 1024 or
// 2048 pairs) and a light bound of ceil(0.5 t), ceil(0.6 t) or ceil(0.7 t)
// zeros; after one warm-up run each is timed twice (CUDA events around the
// pair launches) and the fastest time wins.  The caller's random streams and
// statistics are left as they were.
int tune_run(csim_ctx* ctx, int t, const csim_projector* Pw, const uint64_t* Lw, int kw) {
    const int b = t / 4, lo = std::max(1, 4 * b), hi = std::min(CSIM_MAX_QUBITS, 4 * b + 3);
    const bool own = Pw && Lw && kw > 0 && Pw->nqubits == t && Pw->nstabs > 0;
    const int tr = own ? t : hi;
    const csim_stats saved_stats = ctx->stats;
    const int64_t saved_l0 = ctx->stats_launch0;
    const uint64_t saved_ps = ctx->philox_seed, saved_pn = ctx->philox_next;
    const LibcRand saved_lr = ctx->lr;
    LibcRand g;
    g.seed(0x51ed + (uint32_t)tr);
    auto word = [&g](int n) {
        uint64_t w = 0;
        for (int i = 0; i < n; i++)
            if (g.next() & 1) w |= 1ull << i;
        return w;
    };
    const int nst = std::max(1, (7 * tr + 9) / 10);
    std::vector<int32_t> ph(nst);
    std::vector<uint64_t> xs(nst), zs(nst);
    for (int r = 0; r < nst; r++) {
        ph[r] = g.next() & 3;
        xs[r] = word(tr);
        zs[r] = word(tr);
    }
    const csim_projector Ps{nst, tr, ph.data(), xs.data(), zs.data()};
    const int ks = std::min(14, tr);
    std::vector<uint64_t> Ls(ks);
    for (auto& w : Ls) w = word(tr);
    const csim_projector* P = own ? Pw : &Ps;
    const uint64_t* L = own ? Lw : Ls.data();
    const int k = own ? kw : ks;
    const int64_t chi = (int64_t)1 << k;
    const int64_t count = std::max<int64_t>(128, std::min<int64_t>(4096, (((int64_t)1 << 25) + chi - 1) / chi));
    std::vector<double> vals(count);
    double best = 1e300;
    int best_pt = auto_per_thread(tr), best_pct = 60, best_kernel = 0;
    int rc = 0;
    ctx->tuning = true;
    ctx->trial = default_tune(tr);
    stats_begin(ctx);
    rc = sample_values(ctx, P, L, k, 0, count, CSIM_RNG_PHILOX, 77, vals.data());  // warm-up
    // (kernel, terms per thread, light bound in percent of t)
    struct Cand {
        int kernel, pt, pct;
    };
    // the direct kernel won at every t measured (by 2.5x to 6.5x); the block-prefix kernel stays
    // as the one alternative (the run kernel and the occupancy classes are kept for
    // CSIM_OPT_PAIR_KERNEL 3 and 4, but no longer tried)
    static const Cand cands[] = {{0, 16, 60}, {0, 32, 60}, {3, 16, 60}, {3, 32, 60}};
    for (const Cand& c : cands) {
        if (rc) break;
        if (c.kernel == 1 && chi % (64 * (int64_t)c.pt) != 0) continue;
        ctx->trial.kernel = c.kernel;
        ctx->trial.per_thread = c.pt;
        ctx->trial.light = std::min(tr, (c.pct * tr + 99) / 100);
        double tmin = 1e300;
        for (int rep = 0; rep < 2 && !rc; rep++) {
            stats_begin(ctx);
            rc = sample_values(ctx, P, L, k, 0, count, CSIM_RNG_PHILOX, 77, vals.data());
            if (!rc) tmin = std::min(tmin, ctx->stats.pair_kernel_ms);
        }
        if (!rc && tmin < best) {
            best = tmin;
            best_pt = c.pt;
            best_pct = c.pct;
            best_kernel = c.kernel;
        }
    }
    ctx->tuning = false;
    ctx->stats = saved_stats;
    ctx->stats_launch0 = saved_l0;
    ctx->philox_seed = saved_ps;
    ctx->philox_next = saved_pn;
    ctx->lr = saved_lr;
    if (rc) return rc;
    std::lock_guard<std::mutex> lock(g_tune_mu);
    TuneTable& tt = g_tune[ctx->device & 63];
    for (int u = lo; u <= hi; u++) {
        if (tt.done[u]) continue;
        tt.p[u].per_thread = best_pt;
        tt.p[u].light = std::min(u, (best_pct * u + 99) / 100);
        tt.p[u].kernel = best_kernel;
        tt.done[u] = true;
        tt.ms[u] = best;
    }
    return 0;
}

bool tuned_get(int device, int t, TpTune* out, double* ms) {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    const TuneTable& tt = g_tune[device & 63];
    if (!tt.done[t]) return false;
    if (out) *out = tt.p[t];
    if (ms) *ms = tt.ms[t];
    return true;
}

}  // namespace

int tune_for(csim_ctx* ctx, int t, TpTune* out, const csim_projector* P, const uint64_t* L, int k) {
    if (t < 1 || t > CSIM_MAX_QUBITS) return fail(ctx, CSIM_ERR_ARG, "t=%d outside 1..64", t);
    if (ctx->tuning) {
        *out = ctx->trial;
        if (out->kernel == 3) out->light = direct_light(t);
        return 0;
    }
    TpTune r = default_tune(t);
    if (ctx->autotune && !tuned_get(ctx->device, t, &r, nullptr)) {
        CKR(tune_run(ctx, t, P, L, k));
        if (!tuned_get(ctx->device, t, &r, nullptr)) r = default_tune(t);
    }
    if (ctx->pair_kernel == 2 && r.kernel != 0) {  // the block-prefix kernel, with its own light bound
        r.kernel = 0;
        r.light = light_zeros(t);
    }
    if (ctx->pair_kernel == 3 && r.kernel != 1) {  // the run kernel, with the light bound of its runs
        r.kernel = 1;
        r.light = std::min(t, (11 * t + 19) / 20);
    }
    if (ctx->pair_kernel == 4) r.kernel = 2;  // the block-prefix kernel, one launch per occupancy class
    if (ctx->pair_kernel == 5 && r.kernel != 3) {  // the direct kernel, the rest on kernel 0 with its light bound
        r.kernel = 3;
        r.light = light_zeros(t);
    }
    if (ctx->per_thread > 0) r.per_thread = ctx->per_thread;
    if (r.kernel == 3) r.light = direct_light(t);
    *out = r;
    return 0;
}

}  // namespace csim_host

extern "C" int csim_autotune(csim_ctx* ctx, int32_t t, const csim_projector* P, const uint64_t* L, int32_t k,
                             int32_t* kernel, int32_t* per_thread, int32_t* light_zeros_out, double* pair_ms) {
    if (!ctx || t < 1 || t > CSIM_MAX_QUBITS || (P && P->nqubits != t) || k < 0 || k > 30 || (k > 0 && !L))
        return fail(ctx, CSIM_ERR_ARG, "bad argument");
    cudaSetDevice(ctx->device);
    TpTune tn;
    double ms = 0;
    if (!tuned_get(ctx->device, t, &tn, &ms)) {
        if (P) CKR(check_projector(ctx, P));
        CKR(tune_run(ctx, t, P, L, k));
        if (!tuned_get(ctx->device, t, &tn, &ms)) return fail(ctx, CSIM_ERR_CUDA, "tuning left no result");
    }
    if (tn.kernel == 3) tn.light = direct_light(t);
    if (kernel) *kernel = tn.kernel;
    if (per_thread) *per_thread = tn.per_thread;
    if (light_zeros_out) *light_zeros_out = tn.light;
    if (pair_ms) *pair_ms = ms;
    return CSIM_OK;
}

extern "C" int csim_single_projector_samples(csim_ctx* ctx, const csim_projector* P, const uint64_t* L, int32_t k,
                                             int32_t exact, int64_t count, int32_t rng, uint64_t seed,
                                             double* values) {
    if (!ctx || count < 0 || (count && !values)) return fail(ctx, CSIM_ERR_ARG, "bad argument");
    cudaSetDevice(ctx->device);
    CKR(check_projector(ctx, P));
    if (P->nqubits < 1) return fail(ctx, CSIM_ERR_ARG, "singleProjectorSample needs t >= 1");
    stats_begin(ctx);
    const int r = sample_values(ctx, P, L, k, exact, count, rng, seed, values);
    stats_end(ctx);
    return r;
}

extern "C" int csim_multi_sampled_projector(csim_ctx* ctx, const csim_projector* P, const uint64_t* L, int32_t k,
                                            int32_t exact, double norm, int32_t samples, int32_t bins, int32_t rng,
                                            uint64_t seed, double* out) {
    if (!ctx || !out || bins < 1 || samples < 0) return fail(ctx, CSIM_ERR_ARG, "bad argument");
    cudaSetDevice(ctx->device);
    CKR(check_projector(ctx, P));
    stats_begin(ctx);
    // the seed takes effect even when no state is drawn: a later SEED_CONTINUE call starts from it
    if (rng == CSIM_RNG_LIBC && seed != CSIM_SEED_CONTINUE) ctx->lr.seed((uint32_t)seed);
    if (rng == CSIM_RNG_PHILOX && seed != CSIM_SEED_CONTINUE) {
        ctx->philox_seed = seed;
        ctx->philox_next = 0;
    }
    if (P->nstabs == 0) {  // sampledProjector, innerprod.c:47
        *out = pow(norm, 2);
        return CSIM_OK;
    }
    if (P->nqubits == 0) {
        *out = pow(norm, 2) * clifford_sum(P) / (1 + (double)P->nstabs);
        return CSIM_OK;
    }
    std::vector<double> v((size_t)samples * bins);
    CKR(sample_values(ctx, P, L, k, exact, (int64_t)samples * bins, rng, seed, v.data()));
    stats_end(ctx);
    *out = median_of_means(v.data(), samples, bins);
    return CSIM_OK;
}

extern "C" int csim_median_of_means(const double* values, int32_t samples, int32_t bins, double* out) {
    if (!values || !out || samples < 1 || bins < 1) return CSIM_ERR_ARG;
    *out = median_of_means(values, samples, bins);
    return CSIM_OK;
}

namespace {

// exact_rows through the tree sum: each row's state is a term, made, projected and
// put into graph form by one warp; the tree runs over all terms of the row, and the
// leaves j <= i are left out of its sum (the diagonal j = i is kept apart).
int tree_rows(csim_ctx* ctx, const csim_projector* P, const uint64_t* L, int k, int exact, int64_t i0, int64_t nrow,
              double* re_out, double* im_out) {
    const int t = P->nqubits;
    const csim::tree::Plan& plan = ctx->tree_plan;
    const int64_t chi = (int64_t)1 << plan.r, parts = tree_leaf_shape(plan, nrow).parts_per_state;
    void* v;
    CallInputs in;
    CK(cudaEventRecord(ctx->ev[0], ctx->stream));
    // results: the live rows' count, the error word, the live rows' terms, re, im
    const size_t head = 32, bytes = head + (size_t)nrow * 16;
    CKR(make_inputs(ctx, P, &plan, head, bytes, &in, exact ? nullptr : L, exact ? 0 : k));
    CKR(dbuf(ctx, kBufCode, (size_t)nrow * 4, &v));
    int* const dcode = (int*)v;
    CKR(dbuf(ctx, kBufParts, (size_t)nrow * parts * 64, &v));
    __int128* const dpart = (__int128*)v;
    CKR(dbuf(ctx, kBufPartsDiag, (size_t)nrow * 64, &v));
    __int128* const ddiag = (__int128*)v;
    CK(cudaMemsetAsync(ddiag, 0, (size_t)nrow * 64, ctx->stream));
    TreeGroup g;
    g.plan = &plan;
    g.dplan = in.plan;
    g.count = nrow;
    g.part = dpart;
    g.rows = true;
    g.row0 = i0;
    g.diag = ddiag;
    g.draw = csim::TreeDraw{3,     P->nstabs, 0,     (uint64_t)i0, nullptr, nullptr,        nullptr, in.pm,
                            in.pz, in.px,     dcode, in.L,         exact ? -1 : k, 0};
    TreeRun run;
    std::vector<unsigned char> jobs;
    void* scratch;
    unsigned char* djobs;
    CKR(run.reserve({g}, [&](size_t bytes) { return tree_scratch(ctx, bytes, kTreeScratchMax, &scratch); }));
    run.build((unsigned char*)scratch, jobs);
    CKR(send_inputs(ctx, in, jobs, &djobs));
    if (run.launch(launch_of(ctx), djobs, ctx->ev[1]))
        return fail(ctx, CSIM_ERR_CUDA, "tree launch failed");
    CK(cudaEventRecord(ctx->ev[2], ctx->stream));
    unsigned char* const dres = in.results;
    if (csim::launch_tree_rows(launch_of(ctx), dpart, ddiag, nrow, parts, t, dcode, in.factor, (double*)(dres + head),
                               (double*)(dres + head) + nrow, (unsigned long long*)dres, chi - i0))
        return fail(ctx, CSIM_ERR_CUDA, "reduce launch failed");
    CK(cudaEventRecord(ctx->ev[3], ctx->stream));
    CKR(staged_room(ctx, 2, bytes, &v));
    CKR(dget(ctx, (unsigned char*)v, dres, bytes));
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaGetLastError());
    CKR(error_status(ctx, ((const int*)v)[2]));
    CKR(stats_batch(ctx));
    const double* const res = (const double*)((const unsigned char*)v + head);
    memcpy(re_out, res, (size_t)nrow * 8);
    memcpy(im_out, res + nrow, (size_t)nrow * 8);
    ctx->stats.states = nrow;
    ctx->stats.states_live = ((const int64_t*)v)[0];
    ctx->stats.pairs += ((const int64_t*)v)[2];
    return CSIM_OK;
}

// Rows [i0, i1) of exactProjector (innerprod.c:148-261): row i adds
// 2^{-c_i/2} (diag_i + 2 Re off_i), where off_i = sum_{j>i} <Pi phi_i|phi_j> and
// c_i counts the 2^{-1/2} factors of the projection.  Each row's sum is exact
// in Z[w]; re[i - i0], im[i - i0] get the row's value in double (0 for a row
// the projector annihilates).  *chi_out receives chi.
int exact_rows(csim_ctx* ctx, const csim_projector* P, const uint64_t* L, int k, int exact, int64_t i0, int64_t i1,
               double* re_out, double* im_out, int64_t* chi_out) {
    const int t = P->nqubits;
    CKR(check_code(ctx, t, exact, L, k));
    const int64_t chi = exact ? ((int64_t)1 << ((t + 1) / 2)) : ((int64_t)1 << k);
    if (chi > ((int64_t)1 << 20)) return fail(ctx, CSIM_ERR_ARG, "chi=%lld too large for the exact projector", (long long)chi);
    if (chi_out) *chi_out = chi;
    if (i0 < 0 || i1 < i0 || i1 > chi) return fail(ctx, CSIM_ERR_ARG, "row range [%lld, %lld) outside [0, chi)",
                                                  (long long)i0, (long long)i1);
    if (i0 == i1) return CSIM_OK;
    const int64_t nrow = i1 - i0;
    if (use_tree(ctx, t, exact, k)) {
        tree_plan_for(ctx, exact, L, k, t, nrow);
        if (tree_rows_ok(ctx->tree_plan)) return tree_rows(ctx, P, L, k, exact, i0, nrow, re_out, im_out);
    }
    const int nr = t > 32 ? 2 : 1;
    const int P2 = 2 * t;
    void* v;
    CK(cudaEventRecord(ctx->ev[0], ctx->stream));
    // the terms phi_j, and theta_i = projected copies of them
    csim_state* dphis;
    if (exact) {
        uint64_t* dcw;
        CKR(stage_terms(ctx, t, 1, L, k, 0, chi, &dcw, &dphis));
    } else {
        uint64_t* dL;
        CKR(dput(ctx, kBufL, L, (size_t)k, &dL));
        CKR(dbuf(ctx, kBufCodewords, chi * 8, &v));
        uint64_t* dcw = (uint64_t*)v;
        if (csim::launch_codewords(launch_of(ctx), dL, k, 0, chi, dcw))
            return fail(ctx, CSIM_ERR_CUDA, "codeword launch failed");
        CKR(dbuf(ctx, kBufPhis, chi * sizeof(csim_state), &v));
        dphis = (csim_state*)v;
        if (csim::launch_prep(launch_of(ctx), t, 0, dcw, nullptr, chi, (csim::GState*)dphis))
            return fail(ctx, CSIM_ERR_CUDA, "prepL launch failed");
    }
    CKR(dbuf(ctx, kBufA, chi * sizeof(csim_state), &v));
    csim::GState* dth = (csim::GState*)v;
    CK(cudaMemcpyAsync(dth, dphis, chi * sizeof(csim_state), cudaMemcpyDeviceToDevice, ctx->stream));
    std::vector<int> hm(P->nstabs);
    for (int r = 0; r < P->nstabs; r++) hm[r] = phase_m(P->phase[r]);
    int* dpm;
    uint64_t *dpz, *dpx;
    CKR(dput(ctx, kBufPm, hm.data(), hm.size(), &dpm));
    CKR(dput(ctx, kBufPz, P->zs, (size_t)P->nstabs, &dpz));
    CKR(dput(ctx, kBufPx, P->xs, (size_t)P->nstabs, &dpx));
    CKR(dbuf(ctx, kBufCode, chi * 4, &v));
    int* dcode = (int*)v;
    if (csim::launch_project(launch_of(ctx), nr, dth, chi, P->nstabs, dpm, dpz, dpx, dcode))
        return fail(ctx, CSIM_ERR_CUDA, "projection launch failed");
    // rows outside [i0, i1) are marked annihilated, so the pair kernel skips them
    if (i0 > 0) CK(cudaMemsetAsync(dcode, 0xff, (size_t)i0 * 4, ctx->stream));
    if (i1 < chi) CK(cudaMemsetAsync(dcode + i1, 0xff, (size_t)(chi - i1) * 4, ctx->stream));
    const int64_t chunk = 64, nchunks = (chi + chunk - 1) / chunk;
    const size_t nparts = (size_t)chi * nchunks * 4;
    CKR(dbuf(ctx, kBufParts, nparts * sizeof(__int128), &v));
    __int128* dpart = (__int128*)v;
    CKR(dbuf(ctx, kBufPartsDiag, nparts * sizeof(__int128), &v));
    __int128* dpartd = (__int128*)v;
    CK(cudaMemsetAsync(dpart, 0, nparts * sizeof(__int128), ctx->stream));
    CK(cudaMemsetAsync(dpartd, 0, nparts * sizeof(__int128), ctx->stream));
    CK(cudaEventRecord(ctx->ev[1], ctx->stream));
    if (csim::launch_terms(launch_of(ctx), nr, 2, nullptr, (const csim::GState*)dphis, dth, dcode, chi, 0, chi,
                           (int)chunk, P2, dpart, dpartd, nullptr, nullptr, nullptr))
        return fail(ctx, CSIM_ERR_CUDA, "term launch failed");
    CK(cudaEventRecord(ctx->ev[2], ctx->stream));
    CKR(dbuf(ctx, kBufAcc, (size_t)chi * 4 * sizeof(__int128), &v));
    __int128* dacc = (__int128*)v;
    CKR(dbuf(ctx, kBufAccDiag, (size_t)chi * 4 * sizeof(__int128), &v));
    __int128* daccd = (__int128*)v;
    if (csim::launch_reduce_parts(launch_of(ctx), dpart, chi, nchunks, dacc) ||
        csim::launch_reduce_parts(launch_of(ctx), dpartd, chi, nchunks, daccd))
        return fail(ctx, CSIM_ERR_CUDA, "reduce launch failed");
    CK(cudaEventRecord(ctx->ev[3], ctx->stream));
    std::vector<int> code(nrow);
    std::vector<__int128> acc(nrow * 4), accd(nrow * 4);
    CKR(dget(ctx, code.data(), dcode + i0, nrow));
    CKR(dget(ctx, acc.data(), dacc + 4 * i0, nrow * 4));
    CKR(dget(ctx, accd.data(), daccd + 4 * i0, nrow * 4));
    CKR(finish(ctx));
    CKR(stats_batch(ctx));
    ctx->stats.states = nrow;
    for (int64_t r = 0; r < nrow; r++) {
        re_out[r] = im_out[r] = 0;
        if (code[r] < 0) continue;
        ctx->stats.states_live++;
        ctx->stats.pairs += chi - (i0 + r);
        const __int128* o = &acc[4 * r];
        const __int128* d = &accd[4 * r];
        // 2 Re(a + b w + c w^2 + d w^3) = 2a + (b - d)(w - w^3)
        const __int128 z[4] = {d[0] + 2 * o[0], d[1] + (o[1] - o[3]), d[2], d[3] - (o[1] - o[3])};
        double re, im;
        zomega_to_complex(z, P2, &re, &im);
        const double pf = sqrt_half_power(code[r]);
        re_out[r] = re * pf;
        im_out[r] = im * pf;
    }
    return CSIM_OK;
}

}  // namespace

extern "C" int csim_exact_projector(csim_ctx* ctx, const csim_projector* P, const uint64_t* L, int32_t k,
                                    int32_t exact, double norm, double* out) {
    if (!ctx || !out) return fail(ctx, CSIM_ERR_ARG, "bad argument");
    cudaSetDevice(ctx->device);
    CKR(check_projector(ctx, P));
    stats_begin(ctx);
    if (P->nstabs == 0) {  // innerprod.c:150
        *out = pow(norm, 2);
        return CSIM_OK;
    }
    if (P->nqubits == 0) {
        *out = clifford_sum(P) / (1 + (double)P->nstabs);
        return CSIM_OK;
    }
    int64_t chi = 0;
    CKR(check_code(ctx, P->nqubits, exact, L, k));
    chi = exact ? ((int64_t)1 << ((P->nqubits + 1) / 2)) : ((int64_t)1 << k);
    if (chi > ((int64_t)1 << 20)) return fail(ctx, CSIM_ERR_ARG, "chi=%lld too large for the exact projector", (long long)chi);
    std::vector<double> re(chi), im(chi);
    CKR(exact_rows(ctx, P, L, k, exact, 0, chi, re.data(), im.data(), &chi));
    stats_end(ctx);
    // rows summed in double in row order, like exactProjector's loop
    double tr = 0, ti = 0;
    for (int64_t i = 0; i < chi; i++) {
        tr += re[i];
        ti += im[i];
    }
    *out = sqrt(tr * tr + ti * ti);
    return CSIM_OK;
}

extern "C" int csim_exact_projector_rows(csim_ctx* ctx, const csim_projector* P, const uint64_t* L, int32_t k,
                                         int32_t exact, int64_t i0, int64_t i1, double* re, double* im) {
    if (!ctx || (i1 > i0 && (!re || !im))) return fail(ctx, CSIM_ERR_ARG, "bad argument");
    cudaSetDevice(ctx->device);
    CKR(check_projector(ctx, P));
    if (P->nstabs == 0 || P->nqubits == 0) return fail(ctx, CSIM_ERR_ARG, "no rows: the projector has no terms");
    stats_begin(ctx);
    const int r = exact_rows(ctx, P, L, k, exact, i0, i1, re, im, nullptr);
    stats_end(ctx);
    return r;
}

// ---------------------------------------------------------------- decompose
namespace {

int gf2_rank(const uint64_t* rows, int nrows) {
    uint64_t m[CSIM_MAX_QUBITS];
    memcpy(m, rows, sizeof(uint64_t) * (size_t)nrows);
    int rank = 0;
    for (int c = 0; c < 64 && rank < nrows; c++) {
        int piv = -1;
        for (int r = rank; r < nrows; r++)
            if ((m[r] >> c) & 1) {
                piv = r;
                break;
            }
        if (piv < 0) continue;
        std::swap(m[piv], m[rank]);
        for (int r = 0; r < nrows; r++)
            if (r != rank && ((m[r] >> c) & 1)) m[r] ^= m[rank];
        rank++;
    }
    return rank;
}

// Z(L) on the device, exactly: valid while every partial sum of the reference's
// double loop is exact, k + floor(t/2) <= 53 (terms are multiples of 2^-floor(t/2), sums < 2^k)
int fidelity_sum_gpu(csim_ctx* ctx, int t, const uint64_t* L, int k, double* Z) {
    const int S = t / 2;
    if (k < 0 || k > 40 || t < 1 || t > CSIM_MAX_QUBITS || k + S > 53)
        return fail(ctx, CSIM_ERR_ARG, "fidelity sum: k=%d t=%d beyond the exact range k + t/2 <= 53", k, t);
    uint64_t rows[CSIM_MAX_QUBITS] = {0};
    for (int i = 0; i < k; i++) rows[i] = L[i];
    uint64_t* dL;
    CKR(dput(ctx, kBufL, rows, (size_t)CSIM_MAX_QUBITS, &dL));
    void* v;
    CKR(dbuf(ctx, kBufParts, (size_t)ctx->num_sms * 8 * 16 + 16, &v));
    int nb = 0;
    if (csim::launch_fidelity_sum(launch_of(ctx), dL, k, S, (unsigned __int128*)v, &nb))
        return fail(ctx, CSIM_ERR_CUDA, "fidelity sum launch failed");
    std::vector<unsigned __int128> part(nb);
    CKR(dget(ctx, part.data(), (const unsigned __int128*)v, (size_t)nb));
    CKR(finish(ctx));
    unsigned __int128 sum = 0;
    for (int i = 0; i < nb; i++) sum += part[i];
    *Z = std::ldexp((double)(uint64_t)sum, -S);  // sum <= 2^53: exact
    return 0;
}

int decompose_impl(csim_ctx* gpu, int32_t t, double fidbound, int32_t rank, int32_t fidelity, int32_t force_l,
                   int32_t verbose, int32_t quiet, int32_t* exact, int32_t* k, double* norm, uint64_t* L_out,
                   void* rng_state, FILE* log) {
    if (!exact || !k || !norm || !L_out || !rng_state || t < 0 || t > CSIM_MAX_QUBITS) return CSIM_ERR_ARG;
    LibcRand& lr = *(LibcRand*)rng_state;
    if (t == 0) {
        *exact = 0;
        *norm = 1;
        return CSIM_OK;
    }
    const double v = cos(3.14159265358979323846 / 8);
    *norm = pow(2, floor((float)t / 2) / 2);
    if (t % 2) *norm *= 2 * v;
    if (*exact) return CSIM_OK;
    int forceK = 1;
    if (*k <= 0) {
        forceK = 0;
        *k = (int)ceil(1 - 2 * t * log2(v) - log2(fidbound));
        if (verbose && log) fprintf(log, "Autopicking k = %d to achieve delta = %f.\n", *k, fidbound);
    }
    if (*k > t / 2 && !forceK && !force_l) {
        if (verbose && log) fprintf(log, "k > t/2. Reverting to exact decomposition.\n");
        *exact = 1;
        return CSIM_OK;
    }
    if (*k > t) {
        if (forceK && !quiet && log) fprintf(log, "Can't have k > t. Setting k to %d.\n", t);
        *k = t;
    }
    if (*k > 40) return CSIM_ERR_ARG;
    double inner = 0, Z_L = 0;
    // The reference draws L until the fidelity bound holds (probability.c:355).
    // With its integer-division Z(L) the bound can be out of reach (an
    // autopicked k at larger t), and then that loop never ends; here it stops
    // after kMaxCodeDraws draws with CSIM_ERR_ARG.  Bounds that can be met take
    // hundreds to thousands of draws (411 and 2437 in the reference's seeded
    // decompose vectors).
    constexpr int kMaxCodeDraws = 1 << 16;
    int draws = 0;
    while (inner < 1 - fidbound || forceK) {
        if (++draws > kMaxCodeDraws) {
            if (log) fprintf(log, "csim: no L reached delta = %f in %d draws\n", fidbound, kMaxCodeDraws);
            return CSIM_ERR_ARG;
        }
        const int kk = *k, bytes = (kk * t + 7) / 8;
        for (int i = 0; i < kk; i++) L_out[i] = 0;
        for (int b = 0; b < bytes; b++) {  // BitMatrixSetRandom over the row-major bit array
            const int byte = lr.next() % 256;
            for (int j = 0; j < 8; j++) {
                const int g = 8 * b + j;
                if (g < kk * t && (byte & (0x80 >> j))) L_out[g / t] |= 1ull << (g % t);
            }
        }
        if (rank && gf2_rank(L_out, kk) < kk) {
            if (!quiet && log) fprintf(log, "L has insufficient rank. Sampling again...\n");
            continue;
        }
        if (fidelity) {
            // Z(L) = sum_x 2^{-|x|/2}, with the reference's integer division.  On the
            // device where that double loop is exact; beyond that its rounding is
            // reproduced by the same loop in codeword order
            if (gpu && kk + t / 2 <= 53) {
                const int rc = fidelity_sum_gpu(gpu, t, L_out, kk, &Z_L);
                if (rc) return rc;
            } else {
                Z_L = 0;
                for (int64_t i = 0; i < ((int64_t)1 << kk); i++) Z_L += pow(2, -popc(codeword(i, L_out, kk)) / 2);
            }
            inner = pow(2, kk) * pow(v, 2 * t) / Z_L;
            if (forceK) {
                if (log) fprintf(log, "delta = 1 - <H^t|L>: %lf\n", 1 - inner);
                break;
            } else if (inner < 1 - fidbound) {
                if (!quiet && log) fprintf(log, "delta = 1 - <H^t|L>: %lf - Not good enough!\n", 1 - inner);
            } else {
                if (!quiet && log) fprintf(log, "delta = 1 - <H^t|L>: %lf\n", 1 - inner);
            }
        } else {
            break;
        }
    }
    if (fidelity) *norm = sqrt(pow(2, *k) * Z_L);
    return CSIM_OK;
}

}  // namespace

extern "C" int csim_decompose(int32_t t, double fidbound, int32_t rank, int32_t fidelity, int32_t force_l,
                              int32_t verbose, int32_t quiet, int32_t* exact, int32_t* k, double* norm,
                              uint64_t* L_out, void* rng_state, FILE* log) {
    return decompose_impl(nullptr, t, fidbound, rank, fidelity, force_l, verbose, quiet, exact, k, norm, L_out,
                          rng_state, log);
}

extern "C" int csim_decompose_on(csim_ctx* ctx, int32_t t, double fidbound, int32_t rank, int32_t fidelity,
                                 int32_t force_l, int32_t verbose, int32_t quiet, int32_t* exact, int32_t* k,
                                 double* norm, uint64_t* L_out, void* rng_state, FILE* log) {
    if (!ctx) return CSIM_ERR_ARG;
    cudaSetDevice(ctx->device);
    return decompose_impl(ctx, t, fidbound, rank, fidelity, force_l, verbose, quiet, exact, k, norm, L_out,
                          rng_state, log);
}

extern "C" int csim_fidelity_sum(csim_ctx* ctx, int32_t t, const uint64_t* L, int32_t k, double* Z_L) {
    if (!ctx || !Z_L || (k > 0 && !L)) return fail(ctx, CSIM_ERR_ARG, "bad argument");
    cudaSetDevice(ctx->device);
    return fidelity_sum_gpu(ctx, t, L, k, Z_L);
}
