// Index store and range evaluation behind the C ABI (include/wahgpu.h):
// relic / bin indexes attached from the reference's (keys, offsets, bitmaps)
// triple, the host-side locate (which bitmaps a range covers wholly and which
// edge bitmaps need a row check), and batched evaluation through k_range.
#include "../../include/wahgpu.h"
#include "wah_range.cuh"
#include "wah_api_internal.h"
#include "wah_index_internal.h"

#include <cuda_runtime.h>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cmath>
#include <cstring>
#include <vector>
#include <algorithm>

using namespace wah;

#define CUDA_TRY(ctx, call)                                                            \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess)                                                         \
            return wg_fail(ctx, WAHGPU_ECUDA, "%s failed: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

// ------------------------------------------------------------------ attach
extern "C" int wahgpu_index_from_triple(wahgpu_ctx* ctx, int kind, uint64_t nrows, const double* keys,
                                        uint64_t nkeys, const int64_t* offsets, uint64_t noffsets,
                                        const uint32_t* bitmaps, uint64_t nbitmaps, wahgpu_index** out) {
    if (!ctx || !out || (kind != WAHGPU_RELIC && kind != WAHGPU_BIN) || noffsets < 1 || !offsets ||
        (nbitmaps && !bitmaps) || nrows > 0xFFFFFFFFull)
        return wg_fail(ctx, WAHGPU_EINVAL, "bad argument");
    *out = nullptr;
    const uint32_t nobs = (uint32_t)(noffsets - 1);
    if ((kind == WAHGPU_RELIC && nkeys != nobs) || (kind == WAHGPU_BIN && nkeys != 2ull * nobs) || (nkeys && !keys))
        return wg_fail(ctx, WAHGPU_EINVAL, "key count %llu does not match %u bitmaps", (unsigned long long)nkeys, nobs);
    if (offsets[0] != 0 || (uint64_t)offsets[nobs] != nbitmaps)
        return wg_fail(ctx, WAHGPU_EFORMAT, "offsets do not span the bitmap array");
    wahgpu_index* x = new wahgpu_index();
    x->ctx = ctx; x->kind = kind; x->nrows = (uint32_t)nrows;
    x->groups = (uint32_t)(nrows / MAXBITS); x->anb = (uint32_t)(nrows % MAXBITS);
    x->nobs = nobs;
    x->ntiles = (x->groups + (x->anb ? 1 : 0) + RT - 1) / RT;
    x->keys.assign(keys, keys + nkeys);
    // per bitmap: the serialized trailer (src/bitvector.cpp:54-105)
    std::vector<BitmapMeta> bm(nobs);
    x->bwords.resize(nobs);
    for (uint32_t j = 0; j < nobs; ++j) {
        const int64_t a = offsets[j], b = offsets[j + 1];
        if (b < a) { delete x; return wg_fail(ctx, WAHGPU_EFORMAT, "offsets decrease at bitmap %u", j); }
        const uint64_t len = (uint64_t)(b - a);
        BitmapMeta& m = bm[j];
        m.wstart = (uint64_t)a; m.n = 0; m.anb = 0; m.aval = 0; m.groups = 0;
        if (len > 1) {
            const uint32_t last = bitmaps[b - 1];
            if (last > 0 && last < MAXBITS) { m.anb = last; m.aval = bitmaps[b - 2]; m.n = (uint32_t)(len - 2); }
            else m.n = (uint32_t)(len - 1);
        }
        x->bwords[j] = m.n;
    }
    x->d_words = static_cast<uint32_t*>(wg_alloc(ctx, std::max<uint64_t>(nbitmaps, 1) * 4));
    x->d_bm = static_cast<BitmapMeta*>(wg_alloc(ctx, std::max<size_t>(nobs, 1) * sizeof(BitmapMeta)));
    if (!x->d_words || !x->d_bm) {
        wahgpu_index_free(x);
        return wg_fail(ctx, WAHGPU_ENOMEM, "index allocation failed");
    }
    CUDA_TRY(ctx, cudaMemcpyAsync(x->d_words, bitmaps, nbitmaps * 4, cudaMemcpyHostToDevice, ctx->stream));
    CUDA_TRY(ctx, cudaMemcpyAsync(x->d_bm, bm.data(), nobs * sizeof(BitmapMeta), cudaMemcpyHostToDevice, ctx->stream));
    int rc = wg_index_attach(x);
    if (rc) { wahgpu_index_free(x); return rc; }
    *out = x;
    return WAHGPU_OK;
}

// Cumulative rows: for a stride S, dense row k-1 = OR of bitmaps [0, k*S)
// (k = 1..K), so a range's wholly-inside span costs two dense reads per tile
// plus at most 2S edge bitmaps.  S is the smallest stride that keeps the rows
// within CUM_BUDGET bytes (or the context's WAHGPU_TUNE_CUM_STRIDE): 1, a row
// per bitmap, where that fits (a range is then its rows alone: no word of a
// bitmap is read), else at least 8.  Rows past CUM_FREELY are kept per bitmap
// only while they take less than an eighth of the device memory that is free,
// so that many indexes do not crowd out what a program holds besides.
// Indexes with fewer than two rows' worth of bitmaps keep none.  A row for the
// bitmaps past the last whole stride comes after them: the last row is then
// the OR of all bitmaps, whose 1 bits tell whether any two share a row.
static constexpr uint64_t CUM_BUDGET = 2ull << 30, CUM_FREELY = 256ull << 20;
static int cumulative_rows(wahgpu_index* x) {
    wahgpu_ctx* ctx = x->ctx;
    const uint32_t nobs = x->nobs;
    // rows are gx words rounded up to 4, so a tile's slice starts 16-byte aligned
    const uint64_t gx = ((uint64_t)x->groups + (x->anb ? 1 : 0) + 3) & ~3ull;
    x->cum_k = 0; x->cum_stride = 0;
    if (ctx->cum_stride == 1 || gx == 0) return WAHGPU_OK;
    const uint64_t fit = (nobs * gx * 4 + CUM_BUDGET - 1) / CUM_BUDGET;
    bool each = fit <= 1;
    if (each && !ctx->cum_stride && nobs * gx * 4 > CUM_FREELY) {
        size_t unused = 0, total = 0;
        each = cudaMemGetInfo(&unused, &total) == cudaSuccess && nobs * gx * 4 < unused / 8;
    }
    const uint64_t stride = ctx->cum_stride ? ctx->cum_stride : each ? 1 : std::max<uint64_t>(8, fit);
    const uint64_t K = nobs / stride;
    if (K < 2 && stride > 1) return WAHGPU_OK;
    if (K == 0) return WAHGPU_OK;
    const uint64_t bytes = (nobs + stride - 1) / stride * gx * 4;
    x->d_cum = static_cast<uint32_t*>(wg_alloc(ctx, bytes));
    if (!x->d_cum) return WAHGPU_OK;  // no room: ranges use the bitmaps alone
    CUDA_TRY(ctx, cudaMemsetAsync(x->d_cum, 0, bytes, ctx->stream));
    x->cum_k = (uint32_t)K;
    x->cum_stride = (uint32_t)stride;
    return WAHGPU_OK;
}

// Device blocks held for the duration of a call; they go back to the pool on
// exit (whoever takes them next is ordered after this call on the stream).
struct Temps {
    wahgpu_ctx* ctx;
    std::vector<void*> p;
    explicit Temps(wahgpu_ctx* c) : ctx(c) {}
    template <class T> T* get(size_t n) {
        void* q = wg_alloc(ctx, std::max<size_t>(n * sizeof(T), 16));
        if (q) p.push_back(q);
        return static_cast<T*>(q);
    }
    ~Temps() { for (void* q : p) wg_free(ctx, q); }
};

// Second half of building an index, shared by the triple upload and the
// device build: x->d_words / d_bm / bwords / keys are set; validates the
// words and computes the per-bitmap tile index and 1-bit counts, the tiles'
// bitmap lists and the cumulative rows.
int wg_index_attach(wahgpu_index* x) {
    wahgpu_ctx* ctx = x->ctx;
    const uint32_t nobs = x->nobs;
    x->ntiles = (x->groups + (x->anb ? 1 : 0) + RT - 1) / RT;
    const uint32_t nt = x->ntiles;
    Temps tmp(ctx);
    std::vector<uint32_t> choff(nobs + 1, 0);
    uint64_t nch = 0;
    for (uint32_t j = 0; j < nobs; ++j) {
        nch += std::max<uint64_t>(1, (x->bwords[j] + ICHUNK - 1) / ICHUNK);
        choff[j + 1] = (uint32_t)nch;
    }
    if (nch * 32 > 0xFFFFFFFFull) return wg_fail(ctx, WAHGPU_ERANGE, "index of %llu word chunks", (unsigned long long)nch);
    const uint32_t nchunks = (uint32_t)nch;
    x->d_tiles = static_cast<uint32_t*>(wg_alloc(ctx, std::max<size_t>((size_t)nobs * (nt + 1) * 8, 8)));
    x->d_tl_off = static_cast<uint32_t*>(wg_alloc(ctx, ((size_t)nt + 1) * 4));
    uint32_t* d_choff = tmp.get<uint32_t>((size_t)nobs + 1);
    unsigned long long* d_cg = tmp.get<unsigned long long>(nchunks);
    uint32_t* d_co = tmp.get<uint32_t>(nchunks);
    uint32_t* d_ones = tmp.get<uint32_t>(nobs);
    DevMeta* d_st = tmp.get<DevMeta>(2);
    if (!x->d_tiles || !x->d_tl_off || !d_choff || !d_cg || !d_co || !d_ones || !d_st)
        return wg_fail(ctx, WAHGPU_ENOMEM, "index allocation failed");
    const uint32_t blocks = (uint32_t)(((uint64_t)nchunks * 32 + ITHREADS - 1) / ITHREADS);
    CUDA_TRY(ctx, cudaMemsetAsync(d_st, 0, 2 * sizeof(DevMeta), ctx->stream));
    DevMeta st{};
    x->bones.resize(nobs);
    if (nobs) {
        CUDA_TRY(ctx, cudaMemcpyAsync(d_choff, choff.data(), ((size_t)nobs + 1) * 4, cudaMemcpyHostToDevice, ctx->stream));
        k_chunk_sums<<<blocks, ITHREADS, 0, ctx->stream>>>(x->d_words, x->d_bm, nobs, d_choff, nchunks, d_cg, d_co, d_st);
        k_chunk_scan<<<(uint32_t)(((uint64_t)nobs * 32 + ITHREADS - 1) / ITHREADS), ITHREADS, 0, ctx->stream>>>(
            x->d_bm, nobs, d_choff, x->nrows, d_cg, d_co, d_ones, d_st);
        ctx->launches += 2;
        CUDA_TRY(ctx, cudaGetLastError());
        CUDA_TRY(ctx, cudaMemcpyAsync(&st, d_st, sizeof(DevMeta), cudaMemcpyDeviceToHost, ctx->stream));
        CUDA_TRY(ctx, cudaMemcpyAsync(x->bones.data(), d_ones, (size_t)nobs * 4, cudaMemcpyDeviceToHost, ctx->stream));
    }
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    if (st.status == DEV_ERR_FORMAT) return wg_fail(ctx, WAHGPU_EFORMAT, "a bitmap holds a fill word of length 0");
    if (st.status) return wg_fail(ctx, WAHGPU_ERANGE, "a bitmap holds more bits than the index has rows");
    // the words are valid: every position below lies inside the index's rows
    const uint32_t tw = (nobs + 31) / 32;
    uint64_t most = 0;  // entries of the tile lists at most: a tile on a bitmap's list holds one of its 1 bits
    for (uint32_t j = 0; j < nobs; ++j) most += std::min<uint64_t>(nt, x->bones[j]);
    x->d_tl_bm = static_cast<uint32_t*>(wg_alloc(ctx, std::max<size_t>(most * 4, 16)));
    if (!x->d_tl_bm) return wg_fail(ctx, WAHGPU_ENOMEM, "index allocation failed");
    int rc = cumulative_rows(x);
    if (rc) return rc;
    if (nobs && nt) {
        uint32_t* touch = tmp.get<uint32_t>((size_t)nt * tw);
        if (!touch) return wg_fail(ctx, WAHGPU_ENOMEM, "index allocation failed");
        CUDA_TRY(ctx, cudaMemsetAsync(touch, 0, (size_t)nt * tw * 4, ctx->stream));
        PlaceArgs a;
        a.words = x->d_words; a.bm = x->d_bm; a.nobs = nobs; a.choff = d_choff; a.nchunks = nchunks; a.cstart = d_cg;
        a.ntiles = nt; a.tiles = x->d_tiles; a.touch = touch; a.tw = tw;
        a.gx = (x->groups + (x->anb ? 1u : 0u) + 3u) & ~3u;
        // without rows, the OR of all bitmaps alone
        a.cum = x->d_cum; a.cum_stride = x->cum_k ? x->cum_stride : nobs;
        if (!a.cum) {
            a.cum = tmp.get<uint32_t>(a.gx);
            if (!a.cum) return wg_fail(ctx, WAHGPU_ENOMEM, "index allocation failed");
            CUDA_TRY(ctx, cudaMemsetAsync(a.cum, 0, (size_t)a.gx * 4, ctx->stream));
        }
        const uint32_t nr = (nobs + a.cum_stride - 1) / a.cum_stride;
        k_chunk_place<<<blocks, ITHREADS, 0, ctx->stream>>>(a);
        const uint32_t nparts = (uint32_t)(((uint64_t)nt * tw + LTILE - 1) / LTILE);
        TileRec* recs; LaunchSync* sync;
        rc = wg_scratch(ctx, nparts, &recs, &sync);
        if (rc) return rc;
        k_tile_lists<<<nparts, ITHREADS, 0, ctx->stream>>>(touch, tw, nt, x->d_tl_off, x->d_tl_bm, d_st, recs, sync, nparts);
        ctx->launches += 2;
        unsigned long long* d_or = reinterpret_cast<unsigned long long*>(d_st + 1);  // 1 bits of all bitmaps OR'ed
        unsigned long long h_or = 0;
        if (nr > 1) k_cum_prefix<<<(a.gx + 255) / 256, 256, 0, ctx->stream>>>(a.cum, nr, a.gx);
        k_row_ones<<<std::min<uint32_t>((a.gx + 255) / 256, 2u * (uint32_t)ctx->sm_count), 256, 0, ctx->stream>>>(
            a.cum + (size_t)(nr - 1) * a.gx, a.gx, d_or);
        ctx->launches += nr > 1 ? 2 : 1;
        CUDA_TRY(ctx, cudaGetLastError());
        CUDA_TRY(ctx, cudaMemcpyAsync(&st, d_st, sizeof(DevMeta), cudaMemcpyDeviceToHost, ctx->stream));
        CUDA_TRY(ctx, cudaMemcpyAsync(&h_or, d_or, sizeof h_or, cudaMemcpyDeviceToHost, ctx->stream));
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        if (st.status) return wg_fail(ctx, WAHGPU_ETIMEOUT, "a device-side look-back wait gave up");
        // no row in two bitmaps: the OR holds as many 1 bits as all of them
        uint64_t ones = 0;
        for (uint32_t j = 0; j < nobs; ++j) ones += x->bones[j];
        x->disjoint = h_or == ones;
        x->partition = x->disjoint && h_or == x->nrows;
        if (!x->disjoint) {
            // rows tell a bitmap by C(j + 1) & ~C(j), which drops what it
            // shares with an earlier one: such an index goes by its words
            wg_free(ctx, x->d_cum);
            x->d_cum = nullptr;
            x->cum_k = x->cum_stride = 0;
        }
    } else {
        CUDA_TRY(ctx, cudaMemsetAsync(x->d_tl_off, 0, ((size_t)nt + 1) * 4, ctx->stream));
    }
    x->cum_words.assign(nobs + 1, 0);
    x->cum_ones.assign(nobs + 1, 0);
    for (uint32_t j = 0; j < nobs; ++j) {
        x->cum_words[j + 1] = x->cum_words[j] + x->bwords[j];
        x->cum_ones[j + 1] = x->cum_ones[j] + x->bones[j];
    }
    if (x->kind == WAHGPU_BIN) {
        x->nonempty.clear();
        x->bins_sorted = true;
        for (uint32_t j = 0; j < nobs; ++j) {
            const double mn = x->keys[j], mx = x->keys[nobs + j];
            if (x->bones[j] == 0 || !(mn <= mx)) continue;
            if (!x->nonempty.empty() && !(x->keys[nobs + x->nonempty.back()] < mn)) x->bins_sorted = false;
            x->nonempty.push_back(j);
        }
    }
    x->dev.words = x->d_words; x->dev.bm = x->d_bm; x->dev.tiles = x->d_tiles;
    x->dev.tl_off = x->d_tl_off; x->dev.tl_bm = x->d_tl_bm;
    x->dev.cum = x->d_cum; x->dev.cum_stride = x->cum_stride; x->dev.cum_k = x->cum_k;
    x->dev.gx = (x->groups + (x->anb ? 1u : 0u) + 3u) & ~3u;
    x->dev.values = nullptr; x->dev.nobs = nobs; x->dev.ntiles = x->ntiles;
    if (x->d_values) x->dev.values = x->d_values;
    return WAHGPU_OK;
}

extern "C" int wahgpu_index_set_values(wahgpu_index* x, int vtype, const void* values, uint64_t n) {
    if (!x || !values || vtype < 0 || vtype > 2) return WAHGPU_EINVAL;
    wahgpu_ctx* ctx = x->ctx;
    if (n != x->nrows) return wg_fail(ctx, WAHGPU_EINVAL, "%llu values for %u rows", (unsigned long long)n, x->nrows);
    wg_free(ctx, x->d_values);
    x->d_values = wg_alloc(ctx, std::max<uint64_t>(n, 1) * 4);
    if (!x->d_values) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    CUDA_TRY(ctx, cudaMemcpyAsync(x->d_values, values, n * 4, cudaMemcpyHostToDevice, ctx->stream));
    x->vtype = (uint32_t)vtype;
    x->dev.values = x->d_values;
    return WAHGPU_OK;
}

extern "C" int wahgpu_index_free(wahgpu_index* x) {
    if (!x) return WAHGPU_EINVAL;
    wahgpu_ctx* ctx = x->ctx;
    cudaStreamSynchronize(ctx->stream);
    wg_free(ctx, x->d_words);
    wg_free(ctx, x->d_bm);
    wg_free(ctx, x->d_tiles);
    wg_free(ctx, x->d_tl_off);
    wg_free(ctx, x->d_cum);
    wg_free(ctx, x->d_tl_bm);
    wg_free(ctx, x->d_values);
    delete x;
    return WAHGPU_OK;
}

extern "C" int64_t wahgpu_index_nbitmaps(wahgpu_index* x) { return x ? (int64_t)x->nobs : WAHGPU_EINVAL; }
extern "C" int64_t wahgpu_index_nrows(wahgpu_index* x) { return x ? (int64_t)x->nrows : WAHGPU_EINVAL; }

// estimate(count) of relic / bin (src/irelic.cpp:1843, src/ibin.cpp:6832):
// the 1 bits of all bitmaps.
extern "C" int64_t wahgpu_index_total_ones(wahgpu_index* x) {
    if (!x) return WAHGPU_EINVAL;
    uint64_t s = 0;
    for (uint32_t v : x->bones) s += v;
    return (int64_t)s;
}

// ------------------------------------------------------------------ locate
static bool pass_h(double v, int lop, double lo, int rop, double hi) {
    const bool a = lop == 0 ? true : (lop == 1 ? lo < v : lo <= v);
    const bool b = rop == 0 ? true : (rop == 1 ? v < hi : v <= hi);
    return a && b;
}

// Which bitmaps a range covers: every value of bitmaps [h0, h1) passes, the
// rows of the cand[] bitmaps must be checked, the others hold no passing
// value.  relic (src/irelic.cpp:1416-1809): a bitmap per key; bin
// (src/ibin.cpp:7596-8460): a bin whose [minval, maxval] lies inside the
// range passes whole, one that straddles an end is checked.
// Term modes: the hits (LOC_HITS); the rows certainly hit, i.e. the
// bitmaps wholly inside without the edge bins (LOC_LOWER); the candidate
// rows, the wholly-inside bitmaps and the edge bins OR'ed whole (LOC_UPPER)
// — the lower and upper bounds of bin::estimate(expr, lower, upper),
// src/ibin.cpp:6722-6829.
enum LocMode { LOC_HITS = 0, LOC_LOWER = 1, LOC_UPPER = 2 };

static int locate(wahgpu_ctx* ctx, const wahgpu_index* x, const wahgpu_term* t, DevTerm& out,
                  int mode = LOC_HITS) {
    out = DevTerm{};
    uint32_t h0 = 0, h1 = 0, nc = 0;
    if (x->kind == WAHGPU_RELIC) {
        // keys ascending: the passing keys are one interval, found by the
        // same double comparisons (qContinuousRange::inRange) as the scan
        const auto& k = x->keys;
        uint32_t a = 0, b = x->nobs;
        if (t->lop == 1) a = (uint32_t)(std::upper_bound(k.begin(), k.end(), t->lo) - k.begin());
        else if (t->lop == 2) a = (uint32_t)(std::lower_bound(k.begin(), k.end(), t->lo) - k.begin());
        if (t->rop == 1) b = (uint32_t)(std::lower_bound(k.begin(), k.end(), t->hi) - k.begin());
        else if (t->rop == 2) b = (uint32_t)(std::upper_bound(k.begin(), k.end(), t->hi) - k.begin());
        if (b > a) { h0 = a; h1 = b; }
    } else if (x->bins_sorted) {
        // bins ordered and disjoint: every test below is monotone in the bin
        // order, so binary searches over the bins holding rows find the
        // bins wholly inside and the (at most two) straddling ones
        const auto& ne = x->nonempty;
        const uint32_t nb = x->nobs, m = (uint32_t)ne.size();
        auto mn = [&](uint32_t i) { return x->keys[ne[i]]; };
        auto mx = [&](uint32_t i) { return x->keys[nb + ne[i]]; };
        auto low = [&](double v) { return t->lop == 0 || (t->lop == 1 ? t->lo < v : t->lo <= v); };
        auto high = [&](double v) { return t->rop == 0 || (t->rop == 1 ? v < t->hi : v <= t->hi); };
        auto first = [&](auto pred) {  // first i with pred(i), pred monotone false..true
            uint32_t lo = 0, hi = m;
            while (lo < hi) { const uint32_t md = (lo + hi) / 2; if (pred(md)) hi = md; else lo = md + 1; }
            return lo;
        };
        const uint32_t P = first([&](uint32_t i) { return low(mx(i)); });        // some value passes the lower side
        const uint32_t Q = first([&](uint32_t i) { return !high(mn(i)); });      // [P, Q): some value passes both
        const uint32_t I0 = first([&](uint32_t i) { return low(mn(i)); });       // every value passes the lower side
        const uint32_t I1 = first([&](uint32_t i) { return !high(mx(i)); });     // [.., I1): every value passes the upper
        const uint32_t a = std::max(P, I0), b = std::min(Q, I1);
        if (b > a) { h0 = ne[a]; h1 = ne[b - 1] + 1; }
        for (uint32_t i = P; i < Q; ++i) {
            if (i >= a && i < b) { i = b - 1; continue; }
            if (nc >= 2) return wg_fail(ctx, WAHGPU_EINVAL, "more than two bins straddle the range");
            out.cand[nc++] = ne[i];
        }
    } else {
        std::vector<uint8_t> cls(x->nobs);  // 0 none, 1 all, 2 some
        for (uint32_t j = 0; j < x->nobs; ++j) {
            const double mn = x->keys[j], mx = x->keys[x->nobs + j];
            if (x->bones[j] == 0 || !(mn <= mx)) { cls[j] = 0; continue; }
            const bool pmn = pass_h(mn, t->lop, t->lo, t->rop, t->hi), pmx = pass_h(mx, t->lop, t->lo, t->rop, t->hi);
            if (pmn && pmx) cls[j] = 1;
            else {
                // no value in [mn, mx] passes when the range lies wholly on one side
                const bool below = t->rop != 0 && (t->rop == 1 ? !(mn < t->hi) : !(mn <= t->hi));
                const bool above = t->lop != 0 && (t->lop == 1 ? !(t->lo < mx) : !(t->lo <= mx));
                cls[j] = (below || above) ? 0 : 2;
            }
        }
        h0 = x->nobs; h1 = x->nobs;
        for (uint32_t j = 0; j < x->nobs; ++j) {
            if (cls[j] == 1) { if (h0 == x->nobs) h0 = j; h1 = j + 1; }
            else if (cls[j] == 2) {
                if (nc >= 2) return wg_fail(ctx, WAHGPU_EINVAL, "more than two bins straddle the range");
                out.cand[nc++] = j;
            }
        }
        if (h0 == x->nobs) { h0 = 0; h1 = 0; }
        for (uint32_t j = h0; j < h1; ++j)
            if (cls[j] == 0 && x->bones[j] != 0)
                return wg_fail(ctx, WAHGPU_EINVAL, "bitmaps wholly inside the range are not contiguous");
            else if (cls[j] == 2)
                return wg_fail(ctx, WAHGPU_EINVAL, "bitmaps wholly inside the range are not contiguous");
    }
    if (mode == LOC_LOWER) {
        nc = 0;
    } else if (mode == LOC_UPPER && nc > 0) {
        // the edge bins join the span (they are adjacent to it: every bin
        // between two straddling bins lies wholly inside)
        uint32_t a = h1 > h0 ? h0 : out.cand[0], b = h1 > h0 ? h1 : out.cand[0] + 1u;
        for (uint32_t c = 0; c < nc; ++c) { a = std::min(a, out.cand[c]); b = std::max(b, out.cand[c] + 1u); }
        h0 = a; h1 = b; nc = 0;
    }
    if (nc > 0 && !x->d_values)
        return wg_fail(ctx, WAHGPU_EINVAL, "range needs row checks but the index has no raw values attached");
    if (nc > 0) {
        // the edge rows' comparison in the column's value keys
        const KeyMap m = key_map(x->vtype);
        out.kflip = m.flip; out.ksign = m.sign;
        if (!key_range(x->vtype, (uint32_t)t->lop, t->lo, (uint32_t)t->rop, t->hi, out.klo, out.kspan)) nc = 0;
    }
    out.h0 = h0; out.h1 = h1; out.ncand = nc;
    if (x->cum_k && x->cum_stride == 1) {
        // a row per bitmap: the span and the edge bitmaps by rows
        out.dense = 1; out.cum = x->d_cum;
        out.c0 = h1 > h0 ? h0 : 0; out.c1 = h1 > h0 ? h1 : 0;
        out.e0 = h0; out.e1 = h1;
        return WAHGPU_OK;
    }
    if (x->cum_k && h1 > h0) {
        // C(k1) & ~C(k0) covers [k0*S, k1*S); the rest are edge bitmaps
        const uint32_t S = x->cum_stride;
        const uint32_t k0 = (h0 + S - 1) / S, k1 = std::min(h1 / S, x->cum_k);
        // worth it when the span's words outweigh the dense rows read instead
        const uint64_t span = k1 > k0 ? x->cum_words[k1 * S] - x->cum_words[k0 * S] : 0;
        const uint64_t gx = ((uint64_t)x->groups + (x->anb ? 1 : 0) + 3) & ~3ull;
        if (k1 > k0 && 4 * span >= (k0 ? 2 : 1) * gx) {
            out.c0 = k0; out.c1 = k1; out.e0 = k0 * S; out.e1 = k1 * S;
            out.flip = 0;
            return WAHGPU_OK;
        }
    }
    // sumBins reads the complement when the range holds more than half the
    // index's words (src/index.cpp:6490); the bits are the same either way
    // where every row is in one bitmap
    const uint64_t in = x->cum_words[h1] - x->cum_words[h0], all = x->cum_words[x->nobs];
    out.flip = (x->partition && 2 * in > all) ? 1u : 0u;
    return WAHGPU_OK;
}

// Estimated hits of a located term (its bitmaps' 1 bits), for ordering the
// terms of a query: the most selective first, so a tile whose AND is
// already empty skips the rest.
static uint64_t term_estimate(const wahgpu_index* x, const DevTerm& d) {
    uint64_t e = x->cum_ones[d.h1] - x->cum_ones[d.h0];
    for (uint32_t c = 0; c < d.ncand; ++c) e += x->bones[d.cand[c]];
    return e;
}

// ------------------------------------------------------------------ batches
static int batch_create(wahgpu_ctx* ctx, const wahgpu_term* terms, const uint32_t* query_offsets,
                        uint32_t nq, uint64_t rid_cap, int dense_first, int mode, const uint64_t* caps,
                        wahgpu_batch** out);

extern "C" int wahgpu_batch_create(wahgpu_ctx* ctx, const wahgpu_term* terms, const uint32_t* query_offsets,
                                   uint32_t nq, uint64_t rid_cap, int dense_first, wahgpu_batch** out) {
    return batch_create(ctx, terms, query_offsets, nq, rid_cap, dense_first, LOC_HITS, nullptr, out);
}

// Row ids with a limit per query (the first rid_caps[q] of query q, in row
// order, like a LIMIT); every query's ids land in a region of its own.
extern "C" int wahgpu_batch_create_capped(wahgpu_ctx* ctx, const wahgpu_term* terms, const uint32_t* query_offsets,
                                          uint32_t nq, const uint64_t* rid_caps, wahgpu_batch** out) {
    if (!rid_caps) return wg_fail(ctx, WAHGPU_EINVAL, "rid_caps is NULL");
    uint64_t tot = 0;
    for (uint32_t q = 0; q < nq; ++q) tot += rid_caps[q];
    return batch_create(ctx, terms, query_offsets, nq, tot, 0, LOC_HITS, rid_caps, out);
}

// Does the second pass over a capped batch evaluate a quarter of its items at
// most?  A query's items are visited from the first on until its limit is
// reached, and not at all where the count pass keeps their ids.
static bool few_ids(const std::vector<double>& hits, const std::vector<DevQuery>& q, uint32_t ntiles, size_t kept_at_most) {
    const bool kept = kept_bytes(q.size() * ntiles, kept_at_most) != 0;
    double share = 0;
    for (size_t i = 0; i < q.size(); ++i)
        if (!kept || hits[i] > (double)ntiles * (RSLOT / 2)) share += std::min(1.0, (double)q[i].rid_lim / std::max(1.0, hits[i]));
    return 4 * share <= (double)q.size();
}

static int batch_create(wahgpu_ctx* ctx, const wahgpu_term* terms, const uint32_t* query_offsets,
                        uint32_t nq, uint64_t rid_cap, int dense_first, int mode, const uint64_t* caps,
                        wahgpu_batch** out) {
    if (!ctx || !out || !terms || !query_offsets || nq == 0) return wg_fail(ctx, WAHGPU_EINVAL, "bad argument");
    *out = nullptr;
    const uint32_t nt = query_offsets[nq];
    if (query_offsets[0] != 0 || nt == 0) return wg_fail(ctx, WAHGPU_EINVAL, "bad query offsets");
    const wahgpu_index* x0 = terms[0].idx;
    if (!x0) return wg_fail(ctx, WAHGPU_EINVAL, "term without an index");
    std::vector<const wahgpu_index*> idx;
    std::vector<DevTerm> dt(nt);
    uint64_t bytes = 0, min_bytes = 0;
    for (uint32_t i = 0; i < nt; ++i) {
        const wahgpu_index* x = terms[i].idx;
        if (!x || x->nrows != x0->nrows) return wg_fail(ctx, WAHGPU_EINVAL, "term %u: indexes of one batch must share their row count", i);
        int rc = locate(ctx, x, &terms[i], dt[i], mode);
        if (rc) return rc;
        auto it = std::find(idx.begin(), idx.end(), x);
        dt[i].index = (uint32_t)(it - idx.begin());
        if (it == idx.end()) idx.push_back(x);
        // bytes the term reads: the OR'ed bitmaps' words, the edge bitmaps'
        // words and the raw value of each of their rows
        const uint64_t in = x->cum_words[dt[i].h1] - x->cum_words[dt[i].h0];
        const uint64_t rowb = 4 * ((uint64_t)x->groups + (x->anb ? 1 : 0));
        if (dt[i].dense) bytes += rowb * ((dt[i].c1 ? 1 : 0) + (dt[i].c0 ? 1 : 0));
        else if (dt[i].c1)
            bytes += 4 * ((dt[i].c0 ? 2 : 1) * ((uint64_t)x->groups + (x->anb ? 1 : 0)) +
                          (x->cum_words[dt[i].e0] - x->cum_words[dt[i].h0]) +
                          (x->cum_words[dt[i].h1] - x->cum_words[dt[i].e1]));
        else
            bytes += 4 * (dt[i].flip ? x->cum_words[x->nobs] - in : in);
        for (uint32_t c = 0; c < dt[i].ncand; ++c)
            bytes += 4 * (uint64_t)x->bones[dt[i].cand[c]] +
                     (dt[i].dense ? rowb * (dt[i].cand[c] ? 2 : 1) : 4 * x->bwords[dt[i].cand[c]]);
        // what sumBins itself must read: the covered bitmaps or, when they
        // hold more than half the words, their complement
        // (src/index.cpp:6490), plus the edge bitmaps and their rows
        min_bytes += 4 * std::min(in, x->cum_words[x->nobs] - in);
        for (uint32_t c = 0; c < dt[i].ncand; ++c)
            min_bytes += 4 * (x->bwords[dt[i].cand[c]] + x->bones[dt[i].cand[c]]);
    }
    std::vector<DevQuery> dq;  // the queries k_range evaluates
    std::vector<uint64_t> base(nq, 0);  // counts known beforehand
    std::vector<uint32_t> edge_term, edge_q;  // {term, bitmap} and query of the edges counted alone
    const bool count_only = !rid_cap && !dense_first;
    std::vector<double> hits;  // capped: expected per query
    uint64_t rid_base = 0;
    bool general = false;
    for (uint32_t q = 0; q < nq; ++q) {
        if (query_offsets[q + 1] <= query_offsets[q] || query_offsets[q + 1] > nt)
            return wg_fail(ctx, WAHGPU_EINVAL, "query %u has no term", q);
        const uint32_t t0 = query_offsets[q];
        if (count_only && query_offsets[q + 1] == t0 + 1 && dt[t0].dense && terms[t0].idx->disjoint) {
            // one term over disjoint bitmaps: the wholly-inside bitmaps' 1
            // bits add up, only the edge bins' rows are left to count
            const wahgpu_index* x = terms[t0].idx;
            base[q] = x->cum_ones[dt[t0].h1] - x->cum_ones[dt[t0].h0];
            for (uint32_t c = 0; c < dt[t0].ncand; ++c) {
                edge_term.push_back(t0); edge_term.push_back(dt[t0].cand[c]);
                edge_q.push_back(q);
            }
            continue;
        }
        dq.push_back(DevQuery{});
        DevQuery& d = dq.back();
        d.q = q;
        d.t0 = t0; d.t1 = query_offsets[q + 1];
        d.rid_base = rid_base;
        d.rid_lim = caps ? caps[q] : 0;
        rid_base += caps ? caps[q] : 0;
        if (caps) {
            // hits expected, the terms taken as independent
            double h = x0->nrows;
            for (uint32_t i = d.t0; i < d.t1; ++i)
                h *= std::min(1.0, (double)term_estimate(idx[dt[i].index], dt[i]) / std::max(1u, x0->nrows));
            hits.push_back(h);
        }
        std::stable_sort(dt.begin() + d.t0, dt.begin() + d.t1, [&](const DevTerm& a, const DevTerm& b) {
            if (a.dense != b.dense) return a.dense > b.dense;
            return term_estimate(idx[a.index], a) < term_estimate(idx[b.index], b);
        });
        d.td = d.t0;
        while (d.td < d.t1 && dt[d.td].dense) ++d.td;
        general |= d.td < d.t1;
    }
    std::vector<DevIndex> di;
    for (auto* x : idx) di.push_back(x->dev);
    wahgpu_batch* B = new wahgpu_batch();
    B->ctx = ctx; B->nq = nq; B->nterms = nt; B->nidx = (uint32_t)idx.size();
    B->bytes = bytes + 8ull * nq;
    B->min_bytes = min_bytes + 8ull * nq;
    B->groups = x0->groups; B->anb = x0->anb; B->ntiles = x0->ntiles;
    B->general = general;
    B->nrange = (uint32_t)dq.size();
    B->nedges = (uint32_t)edge_q.size();
    B->etiles = x0->ntiles;
    // few items and dense terms only: smaller tiles, so that they spread
    if (!general && (uint64_t)B->nrange * B->ntiles < 2ull * (uint64_t)ctx->sm_count) {
        B->small = true;
        B->ntiles = (B->groups + (B->anb ? 1 : 0) + RT_SMALL - 1) / RT_SMALL;
    }
    B->rid_cap = rid_cap;
    B->capped = caps != nullptr;
    if (caps) B->few_ids = few_ids(hits, dq, B->ntiles, ctx->kept_at_most);
    if (caps) {
        B->h_lim.assign(caps, caps + nq);
        B->h_base.resize(nq);
        for (uint32_t q = 1; q < nq; ++q) B->h_base[q] = B->h_base[q - 1] + caps[q - 1];
    }
    if (rid_cap) B->d_rids = static_cast<uint32_t*>(wg_alloc(ctx, rid_cap * 4));
    if (dense_first) B->d_dense = static_cast<uint32_t*>(wg_alloc(ctx, ((size_t)x0->groups + 1) * 4));
    auto up16 = [](size_t v) { return (v + 15) & ~(size_t)15; };
    const size_t bi = up16(di.size() * sizeof(DevIndex)), bt = up16((size_t)nt * sizeof(DevTerm));
    const size_t bq = up16(dq.size() * sizeof(DevQuery)), be = edge_term.size() * 4, bg = edge_q.size() * 4;
    B->out_bytes = nq * 16ull + sizeof(DevMeta);
    const size_t bo = up16(B->out_bytes), all = bi + bt + bq + bo + be + bg;
    B->d_tab = static_cast<unsigned char*>(wg_alloc(ctx, all));
    B->d_counts = static_cast<unsigned long long*>(wg_alloc(ctx, B->out_bytes));
    if (!B->d_tab || !B->d_counts || (rid_cap && !B->d_rids) || (dense_first && !B->d_dense)) {
        wahgpu_batch_free(B);
        return wg_fail(ctx, WAHGPU_ENOMEM, "batch allocation failed");
    }
    B->d_idx = reinterpret_cast<DevIndex*>(B->d_tab);
    B->d_terms = reinterpret_cast<DevTerm*>(B->d_tab + bi);
    B->d_queries = reinterpret_cast<DevQuery*>(B->d_tab + bi + bt);
    B->d_init = B->d_tab + bi + bt + bq;
    B->d_start = B->d_counts + nq;
    B->d_status = reinterpret_cast<DevMeta*>(B->d_counts + 2ull * nq);
    // the tables leave from pinned staging the batch keeps until it is
    // freed, so the host does not wait for the copy
    B->h_stage = static_cast<unsigned char*>(wg_host_alloc(ctx, all));
    B->h_out = static_cast<unsigned char*>(wg_host_alloc(ctx, B->out_bytes));
    if (!B->h_stage || !B->h_out) {
        wahgpu_batch_free(B);
        return wg_fail(ctx, WAHGPU_ENOMEM, "batch staging allocation failed");
    }
    memcpy(B->h_stage, di.data(), di.size() * sizeof(DevIndex));
    memcpy(B->h_stage + bi, dt.data(), (size_t)nt * sizeof(DevTerm));
    if (!dq.empty()) memcpy(B->h_stage + bi + bt, dq.data(), dq.size() * sizeof(DevQuery));
    unsigned char* h = B->h_stage + bi + bt + bq;
    memset(h, 0, bo);
    memcpy(h, base.data(), nq * 8ull);
    if (be) { memcpy(h + bo, edge_term.data(), be); memcpy(h + bo + be, edge_q.data(), bg); }
    B->d_edges = B->d_init + bo;
    CUDA_TRY(ctx, cudaMemcpyAsync(B->d_tab, B->h_stage, all, cudaMemcpyHostToDevice, ctx->stream));
    *out = B;
    return WAHGPU_OK;
}

template <int Q, int MODE, bool GEN>
static void launch_range(const wahgpu_ctx* ctx, const RangeArgs& a) {
    static PerDeviceSetup setup;
    constexpr size_t sm = range_smem(GEN, MODE >= RM_IDS);
    const int per_sm = wg_kernel_setup(setup, ctx->device, k_range<Q, MODE, GEN>, RTHREADS, sm);
    const uint32_t ctas = ctx->range_ctas ? std::min<uint32_t>(ctx->range_ctas, (uint32_t)per_sm) : (uint32_t)per_sm;
    // the look-back takes a CTA per item
    const uint32_t grid = MODE == RM_LOOK ? a.nitems : std::min<uint32_t>(a.nitems, ctas * (uint32_t)ctx->sm_count);
    k_range<Q, MODE, GEN><<<grid, RTHREADS, sm, ctx->stream>>>(a);
}
template <int MODE>
static void launch_range_mode(const wahgpu_batch* B, const RangeArgs& a) {
    if (B->general) launch_range<RQUADS, MODE, true>(B->ctx, a);
    else if (B->small) launch_range<1, MODE, false>(B->ctx, a);
    else launch_range<RQUADS, MODE, false>(B->ctx, a);
}

extern "C" int wahgpu_batch_run(wahgpu_batch* B) {
    if (!B) return WAHGPU_EINVAL;
    wahgpu_ctx* ctx = B->ctx;
    // the counts start from those known beforehand (0 for most queries)
    CUDA_TRY(ctx, cudaMemcpyAsync(B->d_counts, B->d_init, B->out_bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    if (B->etiles == 0) return WAHGPU_OK;
    B->captured |= wg_capturing(ctx);
    if (B->nedges) {
        EdgeArgs e;
        e.idx = B->d_idx; e.terms = B->d_terms;
        e.edges = reinterpret_cast<const uint2*>(B->d_edges);
        e.edge_q = reinterpret_cast<const uint32_t*>(B->d_edges + B->nedges * 8ull);
        e.nedges = B->nedges; e.ntiles = B->etiles; e.GX = B->groups + (B->anb ? 1u : 0u);
        e.counts = B->d_counts;
        static PerDeviceSetup setup;
        const uint32_t per_sm = (uint32_t)wg_kernel_setup(setup, ctx->device, k_edge_counts, RTHREADS, 0);
        const uint64_t ctas = ((uint64_t)B->nedges * B->etiles + RWARPS - 1) / RWARPS;
        k_edge_counts<<<(uint32_t)std::min<uint64_t>(ctas, per_sm * (uint64_t)ctx->sm_count), RTHREADS, 0, ctx->stream>>>(e);
        ctx->launches++;
        CUDA_TRY(ctx, cudaGetLastError());
    }
    B->h_valid = false;
    const uint32_t nitems = B->nrange * B->ntiles;
    if (nitems == 0) return WAHGPU_OK;
    RangeArgs a;
    a.idx = B->d_idx; a.terms = B->d_terms; a.queries = B->d_queries; a.nq = B->nrange;
    a.groups = B->groups; a.anb = B->anb; a.ntiles = B->ntiles;
    a.counts = B->d_counts; a.rids = B->d_rids; a.rid_cap = B->rid_cap; a.rid_start = B->d_start;
    a.dense = B->d_dense;
    a.recs = nullptr; a.sync = nullptr; a.nitems = nitems; a.status = B->d_status;
    a.gx = (B->groups + (B->anb ? 1u : 0u) + 3u) & ~3u;
    a.item_cnt = nullptr; a.item_off = nullptr; a.item_list = nullptr; a.slots = nullptr;
    a.capped = B->capped && B->d_rids ? 1u : 0u;
    // Row ids: order 0 asks for the look-back, order 2 for two passes (of
    // several queries); order 1 takes two passes for a capped batch of many
    // items whose limits leave most of them unvisited by the second pass (few_ids()).
    // Where all ids are wanted that pass evaluates the items again, and the
    // look-back's waits cost less: ms by look-back / two passes, uncapped,
    // 2048 items of ranges over 1M rows 0.172 / 0.198, 256 conjunctions over
    // 50M rows 9.3 / 12.3; 256 ids each, 1264 items 0.113 / 0.130, 5056 0.311 /
    // 0.260, 1024 conjunctions over 10M rows (80896) 4.3 / 2.3; 2^20 ids each,
    // 256 conjunctions over 50M rows 8.4 / 10.5, 256 ranges over them 2.1 / 1.3.
    const bool ids = B->d_rids || B->d_dense;
    const bool two_pass = ids && ((ctx->range_order == 2 && B->nq > 1) ||
                                  (ctx->range_order == 1 && B->few_ids && nitems > 16u * (uint32_t)ctx->sm_count));
    a.tile_major = ((ctx->range_order != 0 && !ids) || two_pass) ? 1u : 0u;
    // items are claimed one by one where CTAs take several; with about one each
    // the claims' round trips are only added (one query of 50M rows: 46 us
    // dealt out, 66 claimed)
    if (nitems > 16u * (uint32_t)ctx->sm_count && (two_pass || !ids)) {
        const int rc = wg_scratch(ctx, 1, &a.recs, &a.sync);
        if (rc) return rc;
    }
    if (two_pass) {
        // per item its hits, its first row-id slot or list entry, and the ids
        // kept (without them every item with hits is evaluated again)
        const bool cap = wg_capturing(ctx);
        const size_t ib = (size_t)nitems * ITEM_BYTES;
        if (!a.capped && !B->scan_tmp_bytes)
            cub::DeviceScan::ExclusiveSum(nullptr, B->scan_tmp_bytes, static_cast<unsigned long long*>(nullptr),
                                          static_cast<unsigned long long*>(nullptr), (int)nitems, ctx->stream);
        const size_t tb = a.capped ? 0 : (B->scan_tmp_bytes + 127) & ~(size_t)127;
        size_t sb = B->d_dense ? 0 : kept_bytes(nitems, ctx->kept_at_most);
        if (cap && ctx->ws_bytes < ib + tb + sb) sb = 0;
        unsigned char* ws = wg_workspace(ctx, ib + tb + sb, cap);
        if (!ws && sb) { sb = 0; ws = wg_workspace(ctx, ib + tb, cap); }
        if (!ws) return wg_fail(ctx, WAHGPU_ENOMEM, "two-pass item arrays: allocation failed");
        unsigned long long* items = reinterpret_cast<unsigned long long*>(ws);
        unsigned long long* second = items + nitems;
        if (B->d_dense) CUDA_TRY(ctx, cudaMemsetAsync(B->d_dense, 0, ((size_t)B->groups + 1) * 4, ctx->stream));
        if (sb) a.slots = reinterpret_cast<uint32_t*>(ws + ib + tb);
        CUDA_TRY(ctx, cudaMemsetAsync(items, 0, (size_t)nitems * 8, ctx->stream));
        a.item_cnt = items;
        launch_range_mode<RM_ITEMS>(B, a);
        CUDA_TRY(ctx, cudaGetLastError());
        if (a.capped) {
            uint2* list = reinterpret_cast<uint2*>(second);
            k_cap_items<<<(B->nrange + RWARPS - 1) / RWARPS, RTHREADS, 0, ctx->stream>>>(a, list);
            CUDA_TRY(ctx, cudaGetLastError());
            a.item_list = list;
        } else {
            CUDA_TRY(ctx, cub::DeviceScan::ExclusiveSum(ws + ib, B->scan_tmp_bytes, items, second, (int)nitems, ctx->stream));
            a.item_off = second;
        }
        launch_range_mode<RM_IDS>(B, a);
        ctx->launches += 2;  // the count pass and the scan
    } else if (ids) {
        int rc = wg_scratch(ctx, nitems, &a.recs, &a.sync);
        if (rc) return rc;
        launch_range_mode<RM_LOOK>(B, a);
    } else {
        launch_range_mode<RM_COUNT>(B, a);
    }
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError());
    B->h_valid = false;
    return WAHGPU_OK;
}

// Results of the last run to the host; with rids, the row-id buffer too.
static int batch_fetch(wahgpu_batch* B, uint32_t* rids = nullptr) {
    if (B->h_valid) return WAHGPU_OK;
    wahgpu_ctx* ctx = B->ctx;
    CUDA_TRY(ctx, cudaMemcpyAsync(B->h_out, B->d_counts, B->out_bytes, cudaMemcpyDeviceToHost, ctx->stream));
    if (rids && B->d_rids && B->rid_cap)
        CUDA_TRY(ctx, cudaMemcpyAsync(rids, B->d_rids, B->rid_cap * 4, cudaMemcpyDeviceToHost, ctx->stream));
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    const unsigned long long* c = reinterpret_cast<const unsigned long long*>(B->h_out);
    B->h_counts.assign(c, c + B->nq);
    B->h_start.assign(c + B->nq, c + 2ull * B->nq);
    const DevMeta* st = reinterpret_cast<const DevMeta*>(c + 2ull * B->nq);
    if (st->status == DEV_ERR_TIMEOUT) return wg_fail(ctx, WAHGPU_ETIMEOUT, "a device-side look-back wait gave up");
    B->h_valid = true;
    return WAHGPU_OK;
}

extern "C" int wahgpu_batch_counts(wahgpu_batch* B, uint64_t* counts) {
    if (!B || !counts) return WAHGPU_EINVAL;
    int rc = batch_fetch(B);
    if (rc) return rc;
    for (uint32_t q = 0; q < B->nq; ++q) counts[q] = B->h_counts[q];
    return WAHGPU_OK;
}

// Row ids to the caller's memory.  A few MB of pageable memory are filled
// through two pinned pieces of the context's pool, one being copied out by the
// host while the next arrives (1.1 MB: 85 us against 120 the driver's own way).
static constexpr size_t STAGED = 8u << 20, PIECE = 256u << 10;
static int ids_to_host(wahgpu_ctx* ctx, uint32_t* out, const uint32_t* dev, size_t bytes) {
    cudaPointerAttributes at{};
    const bool pageable = cudaPointerGetAttributes(&at, out) == cudaSuccess && at.type == cudaMemoryTypeUnregistered;
    char* st = pageable && bytes <= STAGED ? static_cast<char*>(wg_host_alloc(ctx, 2 * PIECE)) : nullptr;
    cudaError_t e = cudaSuccess;
    if (!st) {
        e = cudaMemcpyAsync(out, dev, bytes, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    } else {
        const char* src = reinterpret_cast<const char*>(dev);
        char* dst = reinterpret_cast<char*>(out);
        size_t k = 0;
        e = cudaMemcpyAsync(st, src, std::min(bytes, PIECE), cudaMemcpyDeviceToHost, ctx->stream);
        for (size_t o = 0; o < bytes && e == cudaSuccess; o += PIECE, k ^= 1) {
            e = cudaStreamSynchronize(ctx->stream);
            const size_t nx = o + PIECE;
            if (e == cudaSuccess && nx < bytes)
                e = cudaMemcpyAsync(st + (k ^ 1) * PIECE, src + nx, std::min(bytes - nx, PIECE), cudaMemcpyDeviceToHost,
                                    ctx->stream);
            if (e == cudaSuccess) memcpy(dst + o, st + k * PIECE, std::min(bytes - o, PIECE));
        }
        if (e != cudaSuccess) cudaStreamSynchronize(ctx->stream);  // nothing writes the pieces any more
        wg_host_free(ctx, st);
    }
    return e == cudaSuccess ? WAHGPU_OK : wg_fail(ctx, WAHGPU_ECUDA, "row-id copy failed: %s", cudaGetErrorString(e));
}

extern "C" int64_t wahgpu_batch_rids(wahgpu_batch* B, uint32_t q, uint32_t* out, uint64_t cap) {
    if (!B || q >= B->nq || (cap && !out)) return WAHGPU_EINVAL;
    wahgpu_ctx* ctx = B->ctx;
    int rc = batch_fetch(B);
    if (rc) return rc;
    const uint64_t n = B->capped ? std::min<uint64_t>(B->h_counts[q], B->h_lim[q]) : B->h_counts[q];
    const uint64_t s = B->capped ? B->h_base[q] : B->h_start[q];
    if (!B->d_rids || s + n > B->rid_cap) return wg_fail(ctx, WAHGPU_ESIZE, "row ids exceed the batch's capacity");
    if (cap < n) return wg_fail(ctx, WAHGPU_ESIZE, "need room for %llu row ids", (unsigned long long)n);
    if (n) {
        const int r2 = ids_to_host(ctx, out, B->d_rids + s, n * 4);
        if (r2) return r2;
    }
    return (int64_t)n;
}

extern "C" const uint32_t* wahgpu_batch_device_rids(wahgpu_batch* B) { return B ? B->d_rids : nullptr; }

// Every query's count and the whole row-id buffer (rid_cap words) in one
// round trip, for a caller that answers all the queries of a capped batch
// at once: query q's ids are rids[h_base[q], h_base[q] + min(count, limit)).
int wg_batch_fetch_all(wahgpu_batch* B, uint32_t* rids) { return batch_fetch(B, rids); }

// Algorithmic bytes of one run: per term the words of the bitmaps it ORs
// (or of their complement), of its edge bitmaps and the raw values of the
// edge bitmaps' rows; 8 per query for its count.
extern "C" int64_t wahgpu_batch_bytes(wahgpu_batch* B) { return B ? (int64_t)B->bytes : WAHGPU_EINVAL; }
// Bytes any evaluation of the batch must move, whatever its index layout:
// per term the words of the bitmaps sumBins ORs (the covered set, or its
// complement when that is smaller, src/index.cpp:6490), the edge bitmaps'
// words and one raw value per edge row; 8 bytes per count.
extern "C" int64_t wahgpu_batch_min_bytes(wahgpu_batch* B) { return B ? (int64_t)B->min_bytes : WAHGPU_EINVAL; }

extern "C" int wahgpu_batch_free(wahgpu_batch* B) {
    if (!B) return WAHGPU_EINVAL;
    wahgpu_ctx* ctx = B->ctx;
    // results that have been fetched leave nothing of the batch in flight,
    // but for the replays of a graph that holds it
    if (!B->h_valid || B->captured) cudaStreamSynchronize(ctx->stream);
    wg_free(ctx, B->d_tab); wg_free(ctx, B->d_counts);
    wg_free(ctx, B->d_rids); wg_free(ctx, B->d_dense);
    wg_host_free(ctx, B->h_stage);
    wg_host_free(ctx, B->h_out);
    delete B;
    return WAHGPU_OK;
}

// One conjunctive query (countQuery::evaluate, src/countQuery.cpp:292):
// returns the hit count; row ids into host memory when out is given; the hit
// bitvector (compress()ed) when hits is given.
static int64_t evaluate_mode(wahgpu_ctx* ctx, const wahgpu_term* terms, uint32_t nterms, uint32_t* rids,
                             uint64_t cap, wahgpu_bv** hits, int mode);

extern "C" int64_t wahgpu_evaluate(wahgpu_ctx* ctx, const wahgpu_term* terms, uint32_t nterms,
                                   uint32_t* rids, uint64_t cap, wahgpu_bv** hits) {
    return evaluate_mode(ctx, terms, nterms, rids, cap, hits, LOC_HITS);
}

// index::estimate(expr, lower, upper) (src/index.h:191; relic,
// src/irelic.h:58-62: lower = the hits, upper empty; bin,
// src/ibin.cpp:6722-6829: lower = the bins wholly inside, upper = lower and
// the edge bins, empty when there is no edge bin).  An empty upper means
// lower is exact, the reference's convention.
extern "C" int wahgpu_estimate(wahgpu_ctx* ctx, const wahgpu_term* term, wahgpu_bv** lower, wahgpu_bv** upper) {
    if (!ctx || !term || !term->idx || !lower || !upper) return wg_fail(ctx, WAHGPU_EINVAL, "bad argument");
    *lower = nullptr;
    *upper = nullptr;
    DevTerm dl, du;  // no edge bin when the two spans agree
    int rc = locate(ctx, term->idx, term, dl, LOC_LOWER);
    if (!rc) rc = locate(ctx, term->idx, term, du, LOC_UPPER);
    if (rc) return rc;
    const bool exact = dl.h0 == du.h0 && dl.h1 == du.h1;
    int64_t n = evaluate_mode(ctx, term, 1, nullptr, 0, lower, LOC_LOWER);
    if (n < 0) return (int)n;
    if (exact) {
        rc = wahgpu_bv_create(ctx, 1, upper);
    } else {
        n = evaluate_mode(ctx, term, 1, nullptr, 0, upper, LOC_UPPER);
        rc = n < 0 ? (int)n : WAHGPU_OK;
    }
    if (rc) { wahgpu_bv_free(*lower); *lower = nullptr; }
    return rc;
}

// index::estimate(expr) (src/index.h:196): an upper bound of the hit count —
// relic: the exact count (src/irelic.cpp:1843-1854); bin: the 1 bits of the
// bins wholly inside and of the edge bins (src/ibin.cpp:6832-6889).  From
// the host-side per-bitmap counts; no device work.
extern "C" int64_t wahgpu_estimate_count(wahgpu_ctx* ctx, const wahgpu_term* term) {
    if (!ctx || !term || !term->idx) return wg_fail(ctx, WAHGPU_EINVAL, "bad argument");
    const wahgpu_index* x = term->idx;
    DevTerm d;
    const int rc = locate(ctx, x, term, d, LOC_UPPER);
    if (rc) return rc;
    return (int64_t)(x->cum_ones[d.h1] - x->cum_ones[d.h0]);
}

static int64_t evaluate_mode(wahgpu_ctx* ctx, const wahgpu_term* terms, uint32_t nterms, uint32_t* rids,
                             uint64_t cap, wahgpu_bv** hits, int mode) {
    if (!ctx || !terms || nterms == 0 || (cap && !rids)) return wg_fail(ctx, WAHGPU_EINVAL, "bad argument");
    const uint32_t qo[2] = {0, nterms};
    wahgpu_batch* B = nullptr;
    int rc = batch_create(ctx, terms, qo, 1, rids ? cap : 0, hits ? 1 : 0, mode, nullptr, &B);
    if (rc) return rc;
    rc = wahgpu_batch_run(B);
    uint64_t cnt = 0;
    if (!rc) rc = wahgpu_batch_counts(B, &cnt);
    if (!rc && rids) {
        int64_t n = wahgpu_batch_rids(B, 0, rids, cap);
        if (n < 0) rc = (int)n;
    }
    if (!rc && hits) {
        // the dense hit words become a bitvector; compress() gives the
        // canonical words the reference holds after compress()
        const wahgpu_index* x = terms[0].idx;
        wahgpu_bv* hv = nullptr;
        rc = wahgpu_bv_create(ctx, (uint64_t)x->groups + 1, &hv);
        if (!rc) {
            wahgpu_bv* b = hv;
            uint32_t aval = 0;
            if (x->anb) {
                uint32_t last = 0;
                cudaMemcpyAsync(&last, B->d_dense + x->groups, 4, cudaMemcpyDeviceToHost, ctx->stream);
                cudaStreamSynchronize(ctx->stream);
                aval = last >> (31u - x->anb);
            }
            cudaMemcpyAsync(b->words, B->d_dense, (size_t)x->groups * 4, cudaMemcpyDeviceToDevice, ctx->stream);
            rc = wg_scan_meta(b, x->groups, x->anb, aval);
            if (!rc) rc = wahgpu_bv_compress(b);
            if (!rc) *hits = hv; else wahgpu_bv_free(hv);
        }
    }
    wahgpu_batch_free(B);
    return rc ? rc : (int64_t)cnt;
}
