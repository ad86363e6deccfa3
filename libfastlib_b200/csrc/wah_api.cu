// C ABI of libwahgpu: contexts, device bitvectors, operators.
// Declarations and the reference interfaces they replace: include/wahgpu.h.
#include "../../include/wahgpu.h"
#include "wah_plan.h"
#include "wah_merge.cuh"
#include "wah_kernels.cuh"
#include "wah_gop.cuh"
#include "wah_fuse.cuh"
#include "wah_gone.cuh"
#include "wah_api_internal.h"

#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdarg>
#include <cstring>
#include <mutex>
#include <vector>
#include <string>

using namespace wah;

// ------------------------------------------------------------------ errors
static thread_local std::string g_tls_err;

int wg_fail(wahgpu_ctx* ctx, int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (ctx) ctx->err = buf; else g_tls_err = buf;
    return code;
}
#define CUDA_TRY(ctx, call)                                                            \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess)                                                         \
            return wg_fail(ctx, WAHGPU_ECUDA, "%s failed: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

// -------------------------------------------------------------- allocator
static void* driver_get(size_t bytes) {
    void* p = nullptr;
    if (cudaMalloc(&p, bytes) == cudaSuccess) return p;
    cudaGetLastError();
    return nullptr;
}
static void driver_put(void* p) { cudaFree(p); }
static void* driver_host_get(size_t bytes) {
    void* p = nullptr;
    if (cudaMallocHost(&p, bytes) == cudaSuccess) return p;
    cudaGetLastError();
    return nullptr;
}
static void driver_host_put(void* p) { cudaFreeHost(p); }
// Slabs of 1, 8 and then 64 MB of device memory, 64 KB .. 64 MB of pinned memory.
wahgpu_ctx::wahgpu_ctx()
    : dev(driver_get, driver_put, (size_t)1 << 20, 8, (size_t)64 << 20),
      host(driver_host_get, driver_host_put, (size_t)64 << 10, 2, (size_t)64 << 20) {}

void* wg_alloc(wahgpu_ctx* ctx, size_t bytes) {
    {
        std::lock_guard<std::mutex> g(ctx->mu);
        if (ctx->test_fail_alloc > 0 && --ctx->test_fail_alloc == 0) return nullptr;  // test hook
    }
    void* p = ctx->dev.take(bytes);
    if (!p) {
        // release cached memory and retry once
        cudaStreamSynchronize(ctx->stream);
        if (ctx->ws && !ctx->ws_captured) {
            ctx->dev.give(ctx->ws);
            ctx->ws = nullptr;
            ctx->ws_bytes = 0;
        }
        ctx->dev.trim();
        p = ctx->dev.take(bytes);
    }
    return p;
}
void wg_free(wahgpu_ctx* ctx, void* p) { ctx->dev.give(p); }

// Pinned host blocks: staging for copies that must not wait for the host (a
// block goes back to the pool only once the copies reading it are known to be
// done).
void* wg_host_alloc(wahgpu_ctx* ctx, size_t bytes) { return ctx->host.take(bytes); }
void wg_host_free(wahgpu_ctx* ctx, void* p) { ctx->host.give(p); }

// The stream's calls are being captured: they run later, and perhaps often.
bool wg_capturing(const wahgpu_ctx* ctx) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cs) != cudaSuccess) { cudaGetLastError(); return true; }
    return cs != cudaStreamCaptureStatusNone;
}
// Scratch for the look-back scans: tile records plus the launch sync words.
// A captured call's replays go on using the block that the call was given: such
// a block is kept beside the larger one that follows it (at least twice its
// size, so these come to less than the last) until the context ends.  A
// captured call takes what is there.
int wg_scratch(wahgpu_ctx* ctx, uint32_t ntiles, TileRec** recs, LaunchSync** sync) {
    const bool cap = wg_capturing(ctx);
    if (ntiles > ctx->scratch_tiles) {
        if (cap)
            return wg_fail(ctx, WAHGPU_ECUDA, "a captured call needs scratch for %u tiles: make it once before the capture", ntiles);
        const uint32_t want = std::max({ntiles + ntiles / 2, 1024u, ctx->scratch_captured ? 2 * ctx->scratch_tiles : 0u});
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        if (!ctx->scratch_captured) wg_free(ctx, ctx->scratch);
        ctx->scratch = nullptr;
        ctx->scratch_tiles = 0;
        ctx->scratch_captured = false;
        // sync words (the second's ticket for the merge's claims), TileRec
        // records, then the dense kernel's 16-byte records and the single-pass
        // kernel's (each format in a region of its own, so a stale record of
        // one is never read by the other)
        size_t bytes = sizeof(LaunchSync) * 2 + (size_t)want * (sizeof(TileRec) + 2 * sizeof(uint4));
        ctx->scratch = wg_alloc(ctx, bytes);
        if (!ctx->scratch) return wg_fail(ctx, WAHGPU_ENOMEM, "scratch allocation of %zu bytes failed", bytes);
        CUDA_TRY(ctx, cudaMemsetAsync(ctx->scratch, 0, bytes, ctx->stream));
        ctx->scratch_tiles = want;
    }
    ctx->scratch_captured |= cap;
    *sync = reinterpret_cast<LaunchSync*>(ctx->scratch);
    *recs = reinterpret_cast<TileRec*>(reinterpret_cast<char*>(ctx->scratch) + 2 * sizeof(LaunchSync));
    return WAHGPU_OK;
}
// Scratch of one call (the two-pass engine's result patterns, a batch's
// items): one block of the context that grows with its calls.  One that a
// captured call has been given is handed to nothing else until the context
// ends, so that replays write into no other object: it is kept beside the
// larger one that follows it (at least twice its size, so these come to less
// than the last).
unsigned char* wg_workspace(wahgpu_ctx* ctx, size_t bytes, bool captured) {
    if (ctx->ws_bytes < bytes) {
        const size_t want = std::max(bytes, ctx->ws_captured ? 2 * ctx->ws_bytes : ctx->ws_bytes + ctx->ws_bytes / 2);
        if (!ctx->ws_captured) wg_free(ctx, ctx->ws);
        ctx->ws = nullptr;
        ctx->ws_bytes = 0;
        ctx->ws_captured = false;
        ctx->ws = wg_alloc(ctx, want);
        if (!ctx->ws) return nullptr;
        ctx->ws_bytes = ctx->dev.size(ctx->ws);
    }
    ctx->ws_captured |= captured;
    return static_cast<unsigned char*>(ctx->ws);
}
// The dense kernel's records, after the TileRec array of the scratch block.
static uint4* wg_dense_recs(wahgpu_ctx* ctx, TileRec* recs) {
    return reinterpret_cast<uint4*>(recs + ctx->scratch_tiles);
}
// The single-pass group-space kernel's records, after the dense kernel's.
static uint4* wg_fuse_recs(wahgpu_ctx* ctx, TileRec* recs) {
    return wg_dense_recs(ctx, recs) + ctx->scratch_tiles;
}

// ------------------------------------------------------------------ context
extern "C" int wahgpu_ctx_create(int device, wahgpu_ctx** out) {
    if (!out) return wg_fail(nullptr, WAHGPU_EINVAL, "out is NULL");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        return wg_fail(nullptr, WAHGPU_ENODEV, "no CUDA device is available");
    }
    if (device < 0 || device >= ndev) return wg_fail(nullptr, WAHGPU_EINVAL, "bad device %d", device);
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess)
        return wg_fail(nullptr, WAHGPU_ENODEV, "cannot query device %d", device);
    if (prop.major != 10)
        return wg_fail(nullptr, WAHGPU_ENODEV, "device %d is sm_%d%d; this build runs on sm_100 only",
                       device, prop.major, prop.minor);
    wahgpu_ctx* c = new wahgpu_ctx();
    c->device = device;
    c->sm_count = prop.multiProcessorCount;
    cudaSetDevice(device);
    if (cudaStreamCreateWithFlags(&c->own_stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete c;
        return wg_fail(nullptr, WAHGPU_ECUDA, "stream creation failed");
    }
    c->stream = c->own_stream;
    c->h_meta_stage = wg_host_alloc(c, sizeof(DevMeta) * (META_SLOTS + 4));
    if (!c->h_meta_stage) {
        cudaStreamDestroy(c->own_stream);
        delete c;
        return wg_fail(nullptr, WAHGPU_ENOMEM, "pinned staging allocation failed");
    }
    *out = c;
    return WAHGPU_OK;
}

extern "C" int wahgpu_ctx_destroy(wahgpu_ctx* ctx) {
    if (!ctx) return WAHGPU_EINVAL;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    cudaStreamDestroy(ctx->own_stream);
    delete ctx;  // and its memory with it
    return WAHGPU_OK;
}

extern "C" int wahgpu_ctx_set_stream(wahgpu_ctx* ctx, void* stream) {
    if (!ctx) return WAHGPU_EINVAL;
    ctx->stream = stream ? reinterpret_cast<cudaStream_t>(stream) : ctx->own_stream;
    return WAHGPU_OK;
}
extern "C" int wahgpu_ctx_set_tuning(wahgpu_ctx* ctx, int key, int64_t value) {
    if (!ctx) return WAHGPU_EINVAL;
    switch (key) {
    case WAHGPU_TUNE_DENSE_TILE:
        if (value != 1024 && value != 2048 && value != 4096)
            return wg_fail(ctx, WAHGPU_EINVAL, "dense tile must be 1024, 2048 or 4096 groups, not %lld", (long long)value);
        ctx->dense_tile = (uint32_t)value;
        return WAHGPU_OK;
    case WAHGPU_TUNE_DENSE_ENGINE:
        if (value < 0 || value > 5) return wg_fail(ctx, WAHGPU_EINVAL, "dense engine must be 0 .. 5");
        ctx->dense_engine = (uint32_t)value;
        return WAHGPU_OK;
    case WAHGPU_TUNE_RANGE_ORDER:
        if (value < 0 || value > 2) return wg_fail(ctx, WAHGPU_EINVAL, "range order must be 0, 1 or 2");
        ctx->range_order = (uint32_t)value;
        return WAHGPU_OK;
    case WAHGPU_TUNE_RANGE_CTAS:
        if (value < 0 || value > 32) return wg_fail(ctx, WAHGPU_EINVAL, "range CTAs per SM must be 0..32");
        ctx->range_ctas = (uint32_t)value;
        return WAHGPU_OK;
    case WAHGPU_TEST_WITHHOLD_TILE:
        ctx->test_withhold = value < 0 ? 0xFFFFFFFFu : (uint32_t)value;
        return WAHGPU_OK;
    case WAHGPU_TEST_FAIL_ALLOC:
        if (value < 0) return wg_fail(ctx, WAHGPU_EINVAL, "allocation count must be >= 0");
        ctx->test_fail_alloc = value;
        return WAHGPU_OK;
    case WAHGPU_TUNE_MERGE_TILE:
        if (value != 0 && value != 16 && value != 32 && value != 64)
            return wg_fail(ctx, WAHGPU_EINVAL, "merge tile must be 0 (auto), 16, 32 or 64 entries, not %lld", (long long)value);
        ctx->merge_tile = (uint32_t)value;
        return WAHGPU_OK;
    case WAHGPU_TUNE_CUM_STRIDE:
        if (value < 0 || value > (1 << 30)) return wg_fail(ctx, WAHGPU_EINVAL, "cumulative stride must be 0 (auto), 1 (none) or a stride");
        ctx->cum_stride = (uint32_t)value;
        return WAHGPU_OK;
    default:
        return wg_fail(ctx, WAHGPU_EINVAL, "unknown tuning key %d", key);
    }
}
extern "C" int64_t wahgpu_ctx_get_tuning(wahgpu_ctx* ctx, int key) {
    if (!ctx) return WAHGPU_EINVAL;
    switch (key) {
    case WAHGPU_TUNE_DENSE_TILE: return ctx->dense_tile;
    case WAHGPU_TUNE_DENSE_ENGINE: return ctx->dense_engine;
    case WAHGPU_TUNE_RANGE_ORDER: return ctx->range_order;
    case WAHGPU_TUNE_RANGE_CTAS: return ctx->range_ctas;
    case WAHGPU_TUNE_CUM_STRIDE: return ctx->cum_stride;
    case WAHGPU_TUNE_MERGE_TILE: return ctx->merge_tile;
    default: return wg_fail(ctx, WAHGPU_EINVAL, "unknown tuning key %d", key);
    }
}
extern "C" void* wahgpu_ctx_stream(wahgpu_ctx* ctx) { return ctx ? (void*)ctx->stream : nullptr; }
extern "C" int wahgpu_ctx_sync(wahgpu_ctx* ctx) {
    if (!ctx) return WAHGPU_EINVAL;
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return WAHGPU_OK;
}
extern "C" const char* wahgpu_last_error(wahgpu_ctx* ctx) {
    return ctx ? ctx->err.c_str() : g_tls_err.c_str();
}
extern "C" int64_t wahgpu_ctx_launches(wahgpu_ctx* ctx) { return ctx ? (int64_t)ctx->launches : -1; }

// --------------------------------------------------------------- bitvectors
static int bv_reserve(wahgpu_bv* b, uint64_t cap) {
    wahgpu_ctx* ctx = b->ctx;
    if (cap < 1) cap = 1;
    if (cap > 0xFFFFFFFFull) return wg_fail(ctx, WAHGPU_ERANGE, "capacity %llu words too large", (unsigned long long)cap);
    if (b->words && b->cap >= cap) return WAHGPU_OK;
    wg_free(ctx, b->words);
    wg_free(ctx, b->bpos);
    b->words = static_cast<uint32_t*>(wg_alloc(ctx, cap * 4));
    b->bpos = static_cast<uint32_t*>(wg_alloc(ctx, ((cap + 31) / 32 + 2) * 4));
    if (!b->words || !b->bpos) return wg_fail(ctx, WAHGPU_ENOMEM, "device allocation of %llu words failed", (unsigned long long)cap);
    b->cap = (uint32_t)cap;
    b->gt_valid = false;
    b->rows_valid = false;
    return WAHGPU_OK;
}

// Metadata slot of a bitvector, from blocks of META_SLOTS.
static DevMeta* meta_get(wahgpu_ctx* ctx) {
    DevMeta* blk = nullptr;
    {
        std::lock_guard<std::mutex> g(ctx->mu);
        if (!ctx->meta_free.empty()) {
            DevMeta* m = ctx->meta_free.back();
            ctx->meta_free.pop_back();
            return m;
        }
    }
    blk = static_cast<DevMeta*>(wg_alloc(ctx, META_SLOTS * sizeof(DevMeta)));
    if (!blk) return nullptr;
    std::lock_guard<std::mutex> g(ctx->mu);
    ctx->meta_blocks.push_back(blk);
    for (uint32_t i = META_SLOTS; i > 1; --i) ctx->meta_free.push_back(blk + i - 1);
    return blk;
}
wahgpu_bv* wg_bv_new(wahgpu_ctx* ctx) {
    wahgpu_bv* b = new wahgpu_bv();
    b->ctx = ctx;
    b->meta = meta_get(ctx);
    if (!b->meta) { delete b; return nullptr; }
    return b;
}

static void bv_unpend(wahgpu_bv* b) {  // ctx->mu held
    if (b->pend < 0) return;
    std::vector<wahgpu_bv*>& p = b->ctx->pending;
    p[b->pend] = p.back();
    p[b->pend]->pend = b->pend;
    p.pop_back();
    b->pend = -1;
}
// b's metadata have been launched on the context's stream: the host copy is
// stale.  Work that is only being captured runs at some later time, and again
// whenever its graph does, so a result that a captured call writes is read when
// it is asked for and not along with another one, from then on.
static void bv_launched(wahgpu_bv* b) {
    wahgpu_ctx* ctx = b->ctx;
    b->h_valid = false;
    b->told = false;
    b->replayed |= wg_capturing(ctx);
    std::lock_guard<std::mutex> g(ctx->mu);
    if (b->replayed) { bv_unpend(b); return; }
    b->pend_stream = ctx->stream;
    if (b->pend < 0) {
        b->pend = (int32_t)ctx->pending.size();
        ctx->pending.push_back(b);
    }
}

// Waits for the producer of b and copies its metadata to the host, and with
// it, in the same copy, those of the other results launched on this stream
// since (a program that runs several operators and then asks for their counts
// waits once).
int wg_bv_meta(wahgpu_bv* b) {
    wahgpu_ctx* ctx = b->ctx;
    if (!b->h_valid) {
        const DevMeta* blk = nullptr;
        bool elsewhere;
        {
            std::lock_guard<std::mutex> g(ctx->mu);
            for (const DevMeta* m : ctx->meta_blocks)
                if (b->meta >= m && b->meta < m + META_SLOTS) blk = m;
            elsewhere = b->pend >= 0 && b->pend_stream != ctx->stream;
        }
        // launched before the context was given another stream: that one is
        // waited for too, by the device, for it need not be there any more
        if (elsewhere && !wg_capturing(ctx)) CUDA_TRY(ctx, cudaDeviceSynchronize());
        DevMeta* st = reinterpret_cast<DevMeta*>(ctx->h_meta_stage);
        CUDA_TRY(ctx, cudaMemcpyAsync(st, blk, META_SLOTS * sizeof(DevMeta), cudaMemcpyDeviceToHost, ctx->stream));
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        std::lock_guard<std::mutex> g(ctx->mu);
        b->h = st[b->meta - blk];
        b->h_valid = true;
        bv_unpend(b);
        for (size_t i = ctx->pending.size(); i > 0; --i) {
            wahgpu_bv* o = ctx->pending[i - 1];
            if (o->pend_stream != ctx->stream || o->meta < blk || o->meta >= blk + META_SLOTS) continue;
            o->h = st[o->meta - blk];
            o->h_valid = true;
            bv_unpend(o);
        }
    }
    if (b->told) return WAHGPU_OK;
    b->told = true;
    switch (b->h.status) {
    case 0: return WAHGPU_OK;
    case DEV_ERR_TIMEOUT: return wg_fail(ctx, WAHGPU_ETIMEOUT, "a device-side look-back wait gave up");
    case DEV_ERR_FORMAT: return wg_fail(ctx, WAHGPU_EFORMAT, "serialized bitvector holds a fill word of length 0");
    case DEV_ERR_RANGE: return wg_fail(ctx, WAHGPU_ERANGE, "bitvector holds more than 2^32-1 bits");
    default: return wg_fail(ctx, WAHGPU_ECUDA, "device status %u", b->h.status);
    }
}

// Launches the upload scan over b->words[0..n) (device data already there).
int wg_scan_meta(wahgpu_bv* b, uint32_t n, uint32_t anb, uint32_t aval) {
    wahgpu_ctx* ctx = b->ctx;
    CUDA_TRY(ctx, cudaMemsetAsync(b->meta, 0, sizeof(DevMeta), ctx->stream));
    if (n == 0) {
        k_small<<<1, 32, 0, ctx->stream>>>(0, 0, nullptr, nullptr, 0, 0, b->words, b->bpos, b->meta, anb, aval);
    } else {
        uint32_t ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
        TileRec* recs; LaunchSync* sync;
        int rc = wg_scratch(ctx, ntiles, &recs, &sync);
        if (rc) return rc;
        k_meta<<<ntiles, SCAN_THREADS, 0, ctx->stream>>>(b->words, n, b->bpos, b->meta, anb, aval, recs, sync, ntiles);
    }
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError());
    bv_launched(b);
    return WAHGPU_OK;
}

static void parse_trailer(const uint32_t* tail2, uint64_t nwords, uint32_t& n, uint32_t& anb, uint32_t& aval) {
    // src/bitvector.cpp:54-105: the last word is the active bit count when it
    // is in 1..30 (then the word before is the active value); any other last
    // word is dropped and the active word is empty
    n = 0; anb = 0; aval = 0;
    if (nwords <= 1) return;
    const uint32_t last = tail2[1];
    if (last > 0 && last < MAXBITS) { anb = last; aval = tail2[0]; n = (uint32_t)(nwords - 2); }
    else n = (uint32_t)(nwords - 1);
}

extern "C" int wahgpu_bv_from_serial(wahgpu_ctx* ctx, const uint32_t* words, uint64_t nwords, wahgpu_bv** out) {
    if (!ctx || !out || (nwords && !words)) return wg_fail(ctx, WAHGPU_EINVAL, "bad argument");
    if (nwords > 0xFFFFFFFFull) return wg_fail(ctx, WAHGPU_ERANGE, "too many words");
    *out = nullptr;
    uint32_t n, anb, aval;
    uint32_t tail[2] = {0, 0};
    if (nwords >= 2) { tail[0] = words[nwords - 2]; tail[1] = words[nwords - 1]; }
    parse_trailer(tail, nwords, n, anb, aval);
    wahgpu_bv* b = wg_bv_new(ctx);
    if (!b) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    int rc = bv_reserve(b, n);
    if (rc) { wahgpu_bv_free(b); return rc; }
    if (n) {
        cudaError_t e = cudaMemcpyAsync(b->words, words, (size_t)n * 4, cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) { wahgpu_bv_free(b); return wg_fail(ctx, WAHGPU_ECUDA, "upload failed: %s", cudaGetErrorString(e)); }
    }
    rc = wg_scan_meta(b, n, anb, aval);
    if (rc) { wahgpu_bv_free(b); return rc; }
    b->compressed_form = false;
    *out = b;
    return WAHGPU_OK;
}

extern "C" int wahgpu_bv_from_device_serial(wahgpu_ctx* ctx, const uint32_t* dev_words, uint64_t nwords,
                                            wahgpu_bv** out) {
    if (!ctx || !out || (nwords && !dev_words)) return wg_fail(ctx, WAHGPU_EINVAL, "bad argument");
    if (nwords > 0xFFFFFFFFull) return wg_fail(ctx, WAHGPU_ERANGE, "too many words");
    *out = nullptr;
    uint32_t tail[2] = {0, 0};
    if (nwords >= 2) {
        CUDA_TRY(ctx, cudaMemcpyAsync(tail, dev_words + nwords - 2, 8, cudaMemcpyDeviceToHost, ctx->stream));
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    }
    uint32_t n, anb, aval;
    parse_trailer(tail, nwords, n, anb, aval);
    wahgpu_bv* b = wg_bv_new(ctx);
    if (!b) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    int rc = bv_reserve(b, n);
    if (rc) { wahgpu_bv_free(b); return rc; }
    if (n) {
        const cudaError_t e = cudaMemcpyAsync(b->words, dev_words, (size_t)n * 4, cudaMemcpyDeviceToDevice, ctx->stream);
        if (e != cudaSuccess) {
            wahgpu_bv_free(b);
            return wg_fail(ctx, WAHGPU_ECUDA, "device copy failed: %s", cudaGetErrorString(e));
        }
    }
    rc = wg_scan_meta(b, n, anb, aval);
    if (rc) { wahgpu_bv_free(b); return rc; }
    b->compressed_form = false;
    *out = b;
    return WAHGPU_OK;
}

extern "C" int wahgpu_bv_create(wahgpu_ctx* ctx, uint64_t cap_words, wahgpu_bv** out) {
    if (!ctx || !out) return wg_fail(ctx, WAHGPU_EINVAL, "bad argument");
    wahgpu_bv* b = wg_bv_new(ctx);
    if (!b) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    int rc = bv_reserve(b, cap_words);
    if (rc) { wahgpu_bv_free(b); return rc; }
    rc = wg_scan_meta(b, 0, 0, 0);
    if (rc) { wahgpu_bv_free(b); return rc; }
    *out = b;
    return WAHGPU_OK;
}

extern "C" int wahgpu_bv_free(wahgpu_bv* b) {
    if (!b) return WAHGPU_EINVAL;
    wahgpu_ctx* ctx = b->ctx;
    // buffers go back to the context's pool; the pool never hands a block
    // to later work before earlier work on the same stream has used it
    wg_free(ctx, b->words);
    wg_free(ctx, b->bpos);
    {
        std::lock_guard<std::mutex> g(ctx->mu);
        bv_unpend(b);
        if (b->meta) ctx->meta_free.push_back(b->meta);
    }
    wg_free(ctx, b->gt);
    wg_free(ctx, b->rows);
    delete b;
    return WAHGPU_OK;
}

extern "C" int wahgpu_bv_info_get(wahgpu_bv* b, wahgpu_bv_info* info) {
    if (!b || !info) return WAHGPU_EINVAL;
    int rc = wg_bv_meta(b);
    if (rc) return rc;
    info->nwords = b->h.n;
    info->nbits = (uint64_t)b->h.groups * MAXBITS + b->h.anb;
    info->cnt = (uint64_t)b->h.nset + __builtin_popcount(b->h.aval);
    info->anb = b->h.anb;
    info->aval = b->h.aval;
    info->compressed_form = b->compressed_form ? 1u : 0u;
    return WAHGPU_OK;
}
extern "C" int64_t wahgpu_bv_size(wahgpu_bv* b) {
    wahgpu_bv_info i; int rc = wahgpu_bv_info_get(b, &i); return rc ? rc : (int64_t)i.nbits;
}
extern "C" int64_t wahgpu_bv_cnt(wahgpu_bv* b) {
    wahgpu_bv_info i; int rc = wahgpu_bv_info_get(b, &i); return rc ? rc : (int64_t)i.cnt;
}
extern "C" int64_t wahgpu_bv_serial_size(wahgpu_bv* b) {
    wahgpu_bv_info i; int rc = wahgpu_bv_info_get(b, &i);
    return rc ? rc : (int64_t)(i.nwords + 1 + (i.anb > 0));
}
extern "C" int64_t wahgpu_bv_write(wahgpu_bv* b, uint32_t* out, uint64_t cap) {
    if (!b || (cap && !out)) return WAHGPU_EINVAL;
    int rc = wg_bv_meta(b);
    if (rc) return rc;
    wahgpu_ctx* ctx = b->ctx;
    const uint64_t len = (uint64_t)b->h.n + 1 + (b->h.anb > 0);
    if (cap < len) return wg_fail(ctx, WAHGPU_ESIZE, "need %llu words", (unsigned long long)len);
    if (b->h.n) {
        CUDA_TRY(ctx, cudaMemcpyAsync(out, b->words, (size_t)b->h.n * 4, cudaMemcpyDeviceToHost, ctx->stream));
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    }
    uint64_t k = b->h.n;
    if (b->h.anb > 0) out[k++] = b->h.aval;
    out[k] = b->h.anb;
    return (int64_t)len;
}
extern "C" const uint32_t* wahgpu_bv_device_words(wahgpu_bv* b) { return b ? b->words : nullptr; }

// ---------------------------------------------------------------- operators
static uint32_t combine_active(int op, uint32_t a, uint32_t b) {
    switch (op) {
    case OP_AND: return a & b;
    case OP_OR: return a | b;
    case OP_XOR: return a ^ b;
    default: return a & ~b;
    }
}

// Launches one instantiation of the merge kernel (its shared-memory
// attribute set once per device).
template <int OP, bool FSM, bool UNARY, bool FLIP, int TB>
static void launch_k(const wahgpu_ctx* ctx, dim3 g, cudaStream_t s, const MergeArgs& a) {
    static PerDeviceSetup setup;
    const size_t sm = sizeof(TileShared<TB>);
    wg_kernel_setup(setup, ctx->device, k_merge<OP, FSM, UNARY, FLIP, TB>, MERGE_THREADS, sm);
    wg_launch_pdl(k_merge<OP, FSM, UNARY, FLIP, TB>, g.x, MERGE_THREADS, sm, s, a);
}
template <int TB>
static void launch_merge_tb(const wahgpu_ctx* ctx, int op, bool fsm, bool unary, bool flip, dim3 g, cudaStream_t s,
                            const MergeArgs& a) {
    if (unary) {
        if (flip) launch_k<0, false, true, true, TB>(ctx, g, s, a);
        else launch_k<0, false, true, false, TB>(ctx, g, s, a);
        return;
    }
#define WG_MERGE_OP(O)                                                          \
    if (fsm) launch_k<O, true, false, false, TB>(ctx, g, s, a);                 \
    else launch_k<O, false, false, false, TB>(ctx, g, s, a);
    switch (op) {
    case OP_AND: WG_MERGE_OP(OP_AND) break;
    case OP_OR: WG_MERGE_OP(OP_OR) break;
    case OP_XOR: WG_MERGE_OP(OP_XOR) break;
    default: WG_MERGE_OP(OP_MINUS) break;
    }
#undef WG_MERGE_OP
}
// Block-index entries per merge tile: the context's setting, else by the
// operands' size.  Small operands spread over the GPU in short tiles; long
// tiles share their fixed steps among more words (2^28 bits, us at 16 / 32 /
// 64 entries: 4.6 K blocks 14.8 / 13.3 / 15.4, 14 K 25.7 / 17.7 / 18.1, 45 K
// 63 / 42 / 26).
static uint32_t merge_tile_blocks(const wahgpu_ctx* ctx, uint32_t nblocks) {
    if (ctx->merge_tile) return ctx->merge_tile;
    const uint64_t sms = (uint64_t)ctx->sm_count;
    if (nblocks >= sms * 128u) return 64;
    if (nblocks >= sms * 30u) return 32;
    return 16;
}

// Merge launch: x OP y, or a (complemented) copy of x when y == nullptr.
int wg_launch_merge(wahgpu_ctx* ctx, int op, bool fsm, bool unary, bool flip,
                    const wahgpu_bv* x, const wahgpu_bv* y, uint32_t groups,
                    uint32_t anb, uint32_t aval, wahgpu_bv* res) {
    const uint32_t nx = x->h.n, ny = y ? y->h.n : 0;
    const uint32_t nbx = (nx + 31) / 32, nby = (ny + 31) / 32;
    const uint32_t need = nx + ny;
    int rc = bv_reserve(res, need);
    if (rc) return rc;
    const uint32_t nblk = unary ? nbx : nbx + nby;
    const uint32_t tb = merge_tile_blocks(ctx, nblk);
    uint32_t ntiles = (nblk + tb - 1) / tb;
    if (ntiles == 0) ntiles = 1;
    TileRec* recs; LaunchSync* sync;
    rc = wg_scratch(ctx, ntiles, &recs, &sync);
    if (rc) return rc;
    MergeArgs a;
    a.xw = x->words; a.xbp = x->bpos; a.nx = nx; a.nbx = nbx;
    a.yw = y ? y->words : x->words; a.ybp = y ? y->bpos : x->bpos; a.ny = ny; a.nby = nby;
    a.groups = groups;
    a.out = res->words; a.obp = res->bpos; a.meta = res->meta;
    a.recs = recs; a.sync = sync; a.ntiles = ntiles;
    a.aval = aval; a.anb = anb;
    a.late = ctx->test_withhold;
    ctx->test_withhold = 0xFFFFFFFFu;
    dim3 g(ntiles);
    if (tb == 16) launch_merge_tb<16>(ctx, op, fsm, unary, flip, g, ctx->stream, a);
    else if (tb == 32) launch_merge_tb<32>(ctx, op, fsm, unary, flip, g, ctx->stream, a);
    else launch_merge_tb<64>(ctx, op, fsm, unary, flip, g, ctx->stream, a);
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError());
    bv_launched(res);
    res->gt_valid = false;
    res->rows_valid = false;
    res->used = false;
    res->compressed_form = true;
    return WAHGPU_OK;
}

// Group-tile index of b (host metadata must be valid); built once.
static int wg_gtile(wahgpu_bv* b) {
    if (b->gt_valid) return WAHGPU_OK;
    wahgpu_ctx* ctx = b->ctx;
    const uint32_t nt = (b->h.groups + DT - 1) / DT;
    if (!b->gt) {
        b->gt = static_cast<uint32_t*>(wg_alloc(ctx, ((size_t)nt + 2) * 8));
        if (!b->gt) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    } else {
        // reallocate when the current block may be too small
        wg_free(ctx, b->gt);
        b->gt = static_cast<uint32_t*>(wg_alloc(ctx, ((size_t)nt + 2) * 8));
        if (!b->gt) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    }
    const uint32_t threads = 128, blocks = (nt + 1 + threads - 1) / threads;
    k_gtile<<<blocks, threads, 0, ctx->stream>>>(b->words, b->bpos, b->h.n, b->h.groups, nt, b->gt);
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError());
    b->gt_valid = !b->replayed && !wg_capturing(ctx);
    return WAHGPU_OK;
}

template <int OP, int TG, int NCW>
static void launch_dense_op(const wahgpu_ctx* ctx, uint32_t ntiles, cudaStream_t s, const DenseArgs& a) {
    static PerDeviceSetup setup;
    const size_t sm = sizeof(DShared<TG, NCW>);
    const int per_sm = wg_kernel_setup(setup, ctx->device, k_dense<OP, TG, NCW>, (NCW + 1) * 32, sm);
    // persistent: at most one wave of resident CTAs
    const uint32_t grid = std::min<uint32_t>(ntiles, (uint32_t)(per_sm * ctx->sm_count));
    k_dense<OP, TG, NCW><<<grid, (NCW + 1) * 32, sm, s>>>(a);
}
template <int OP>
static void launch_dense_tg(const wahgpu_ctx* ctx, uint32_t tg, uint32_t ntiles, cudaStream_t s, const DenseArgs& a) {
    if (tg == 1024) launch_dense_op<OP, 1024, 4>(ctx, ntiles, s, a);
    else if (tg == 4096) launch_dense_op<OP, 4096, 8>(ctx, ntiles, s, a);
    else launch_dense_op<OP, 2048, 8>(ctx, ntiles, s, a);
}

int wg_launch_dense(wahgpu_ctx* ctx, int op, wahgpu_bv* x, wahgpu_bv* y, uint32_t groups,
                    uint32_t anb, uint32_t aval, wahgpu_bv* res) {
    int rc = bv_reserve(res, (uint64_t)x->h.n + y->h.n);
    if (rc) return rc;
    rc = wg_gtile(x);
    if (rc) return rc;
    rc = wg_gtile(y);
    if (rc) return rc;
    const uint32_t tg = ctx->dense_tile;
    const uint32_t ntiles = (groups + tg - 1) / tg;
    TileRec* recs; LaunchSync* sync;
    rc = wg_scratch(ctx, ntiles, &recs, &sync);
    if (rc) return rc;
    DenseArgs a;
    a.xw = x->words; a.xgt = x->gt; a.nx = x->h.n;
    a.yw = y->words; a.ygt = y->gt; a.ny = y->h.n;
    a.groups = groups;
    a.out = res->words; a.obp = res->bpos; a.meta = res->meta;
    a.drecs = wg_dense_recs(ctx, recs); a.sync = sync; a.ntiles = ntiles;
    a.aval = aval; a.anb = anb;
    CUDA_TRY(ctx, cudaMemsetAsync(res->meta, 0, sizeof(DevMeta), ctx->stream));
    switch (op) {
    case OP_AND: launch_dense_tg<OP_AND>(ctx, tg, ntiles, ctx->stream, a); break;
    case OP_OR: launch_dense_tg<OP_OR>(ctx, tg, ntiles, ctx->stream, a); break;
    case OP_XOR: launch_dense_tg<OP_XOR>(ctx, tg, ntiles, ctx->stream, a); break;
    default: launch_dense_tg<OP_MINUS>(ctx, tg, ntiles, ctx->stream, a); break;
    }
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError());
    bv_launched(res);
    res->gt_valid = false;
    res->rows_valid = false;
    res->used = false;
    res->compressed_form = true;
    return WAHGPU_OK;
}

// Room for the row index of b over `groups` groups.
static bool rows_reserve(wahgpu_bv* b, uint32_t groups) {
    wahgpu_ctx* ctx = b->ctx;
    const uint32_t need = (uint32_t)(((uint64_t)groups + PT - 1) / PT) * TROWS;
    if (b->rows && b->rows_cap >= need) return true;
    wg_free(ctx, b->rows);
    b->rows_valid = false;
    b->rows_cap = 0;
    b->rows = static_cast<uint2*>(wg_alloc(ctx, (size_t)need * sizeof(uint2)));
    if (!b->rows) return false;
    b->rows_cap = need;
    return true;
}
// Room for a result's row index.  A result that a captured call writes keeps
// none: its replays change the words without the index.
static bool result_rows(wahgpu_bv* res, uint32_t groups) {
    return !res->replayed && !wg_capturing(res->ctx) && rows_reserve(res, groups);
}
// Row index of b (host metadata must be valid); built once, by a captured
// call on each of its replays, and for words that replays change on each use.
static int wg_rows(wahgpu_bv* b) {
    wahgpu_ctx* ctx = b->ctx;
    // positions are taken from the words: none that the upload scan refused
    if (b->h.status) return wg_fail(ctx, WAHGPU_EFORMAT, "the bitvector's words are malformed");
    if (b->rows_valid) return WAHGPU_OK;
    if (!rows_reserve(b, b->h.groups)) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    const uint32_t ntiles = (b->h.groups + PT - 1) / PT;
    k_rows<<<(ntiles + GW - 1) / GW, GCTA, 0, ctx->stream>>>(b->words, b->bpos, b->h.n, b->h.groups, ntiles, b->rows);
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError());
    b->rows_valid = !b->replayed && !wg_capturing(ctx);
    return WAHGPU_OK;
}

static constexpr uint32_t GOP_CTAS_AT_MOST = 4096;  // room for their warps' first heads
template <int OP, int KIND>
static void launch_gop_op(const wahgpu_ctx* ctx, uint32_t ntiles, cudaStream_t s, GopArgs& a) {
    static PerDeviceSetup setup;
    const size_t sm = GW * sizeof(GopWarp<(KIND >= GK_COPY)>);
    const uint32_t per_sm = (uint32_t)wg_kernel_setup(setup, ctx->device, k_gop<OP, KIND>, GCTA, sm);
    a.gop_ctas = std::min<uint32_t>({(ntiles + GW - 1) / GW, per_sm * (uint32_t)ctx->sm_count, GOP_CTAS_AT_MOST});
    wg_launch_pdl(k_gop<OP, KIND>, a.gop_ctas, GCTA, sm, s, a);
}
template <int KIND>
static void launch_gop_kind(const wahgpu_ctx* ctx, int op, uint32_t ntiles, cudaStream_t s, GopArgs& a) {
    switch (op) {
    case OP_AND: launch_gop_op<OP_AND, KIND>(ctx, ntiles, s, a); break;
    case OP_OR: launch_gop_op<OP_OR, KIND>(ctx, ntiles, s, a); break;
    case OP_XOR: launch_gop_op<OP_XOR, KIND>(ctx, ntiles, s, a); break;
    default: launch_gop_op<OP_MINUS, KIND>(ctx, ntiles, s, a); break;
    }
}

static size_t gop_bytes(uint32_t groups) {
    const size_t ntiles = ((uint64_t)groups + PT - 1) / PT;
    return ntiles * (PT * 4 + TROWS * sizeof(uint2) + 12) + std::min<size_t>((ntiles + GW - 1) / GW, GOP_CTAS_AT_MOST) * GW * 4;
}

// Two-pass group-space engine (wah_gop.cuh): the result patterns per group
// with head masks and per-CTA totals, then the words.  kind: GopKind; y is
// null for the copies.
int wg_launch_gop(wahgpu_ctx* ctx, int kind, int op, wahgpu_bv* x, wahgpu_bv* y, uint32_t groups,
                  uint32_t anb, uint32_t aval, wahgpu_bv* res) {
    int rc = bv_reserve(res, (uint64_t)x->h.n + (y ? y->h.n : 0));
    if (!rc) rc = wg_rows(x);
    if (!rc && y) rc = wg_rows(y);
    if (rc) return rc;
    const uint32_t ntiles = (uint32_t)(((uint64_t)groups + PT - 1) / PT);
    // the result keeps its head masks as its row index where a block for it
    // is at hand; else they are part of the scratch
    const bool keep = result_rows(res, groups);
    const size_t rb = (size_t)ntiles * PT * 4, hb = (size_t)ntiles * TROWS * sizeof(uint2);
    unsigned char* scr = wg_workspace(ctx, gop_bytes(groups), wg_capturing(ctx));
    if (!scr) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation of %u tiles of result patterns failed", ntiles);
    uint32_t* tot = reinterpret_cast<uint32_t*>(scr + rb + hb);
    GopArgs a;
    a.xw = x->words; a.xr = x->rows; a.xbp = x->bpos; a.nx = x->h.n;
    a.yw = y ? y->words : nullptr; a.yr = y ? y->rows : nullptr; a.ybp = y ? y->bpos : nullptr; a.ny = y ? y->h.n : 0;
    a.groups = groups; a.ntiles = ntiles;
    a.R = reinterpret_cast<uint32_t*>(scr); a.heads = tot; a.first = tot + ntiles; a.ones = tot + 2 * (size_t)ntiles;
    a.wfirst = tot + 3 * (size_t)ntiles; a.gop_ctas = 0;
    a.out = res->words; a.obp = res->bpos; a.meta = res->meta;
    a.orow = keep ? res->rows : reinterpret_cast<uint2*>(scr + rb);
    a.aval = aval; a.anb = anb;
    a.withhold = ctx->test_withhold;
    ctx->test_withhold = 0xFFFFFFFFu;
    cudaStream_t s = ctx->stream;
    if (kind == GK_CANON) launch_gop_kind<GK_CANON>(ctx, op, ntiles, s, a);
    else if (kind == GK_FSM) launch_gop_kind<GK_FSM>(ctx, op, ntiles, s, a);
    else if (kind == GK_COPY) launch_gop_op<OP_AND, GK_COPY>(ctx, ntiles, s, a);
    else launch_gop_op<OP_AND, GK_FLIP>(ctx, ntiles, s, a);
    static PerDeviceSetup setup;
    const size_t sm = GW * sizeof(PackWarp);
    const uint32_t per_sm = (uint32_t)wg_kernel_setup(setup, ctx->device, k_gpack, GCTA, sm);
    const uint32_t grid = std::max<uint32_t>(std::min<uint32_t>((ntiles + GW - 1) / GW, per_sm * (uint32_t)ctx->sm_count),
                                             (ntiles + GRANGE - 1) / GRANGE);
    wg_launch_pdl(k_gpack, grid, GCTA, sm, s, a);
    ctx->launches += 2;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return wg_fail(ctx, WAHGPU_ECUDA, "launch failed: %s", cudaGetErrorString(e));
    bv_launched(res);
    res->gt_valid = false;
    res->rows_valid = keep;
    res->used = false;
    res->compressed_form = true;
    return WAHGPU_OK;
}

// Single-pass group-space engine (wah_fuse.cuh): one launch per call,
// operands read once, words written once.  Needs 16-byte-aligned word arrays
// (every block of the allocator is); the two-pass engine runs otherwise.
static bool fuse_applies(const wahgpu_bv* x, const wahgpu_bv* y, const wahgpu_bv* res, uint32_t groups) {
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    return groups > 0 && al(x->words) && al(y->words) && al(res->words);
}
template <int OP, int FT>
static void launch_fuse_op(const wahgpu_ctx* ctx, uint32_t ntiles, cudaStream_t s, const FuseArgs& a) {
    static PerDeviceSetup setup;
    const size_t sm = sizeof(FuseShared<FT>);
    wg_kernel_setup(setup, ctx->device, k_gfuse<OP, FT>, FCfg<FT>::THREADS, sm);
    k_gfuse<OP, FT><<<ntiles, FCfg<FT>::THREADS, sm, s>>>(a);
}
template <int OP>
static void launch_fuse_tile(const wahgpu_ctx* ctx, uint32_t ft, uint32_t ntiles, cudaStream_t s, const FuseArgs& a) {
    if (ft == 1024) launch_fuse_op<OP, 1024>(ctx, ntiles, s, a);
    else if (ft == 4096) launch_fuse_op<OP, 4096>(ctx, ntiles, s, a);
    else launch_fuse_op<OP, 2048>(ctx, ntiles, s, a);
}
int wg_launch_fuse(wahgpu_ctx* ctx, int op, wahgpu_bv* x, wahgpu_bv* y, uint32_t groups,
                   uint32_t anb, uint32_t aval, wahgpu_bv* res) {
    int rc = bv_reserve(res, (uint64_t)x->h.n + y->h.n);
    if (rc) return rc;
    if (!fuse_applies(x, y, res, groups)) return wg_launch_gop(ctx, GK_CANON, op, x, y, groups, anb, aval, res);
    rc = wg_gtile(x);
    if (rc) return rc;
    rc = wg_gtile(y);
    if (rc) return rc;
    const uint32_t ft = ctx->dense_tile;  // WAHGPU_TUNE_DENSE_TILE: 1024, 2048 (default) or 4096 groups
    const uint32_t ntiles = (groups + ft - 1) / ft;
    TileRec* recs; LaunchSync* sync;
    rc = wg_scratch(ctx, ntiles, &recs, &sync);
    if (rc) return rc;
    FuseArgs a;
    a.xw = x->words; a.xgt = x->gt; a.nx = x->h.n;
    a.yw = y->words; a.ygt = y->gt; a.ny = y->h.n;
    a.groups = groups; a.ntiles = ntiles;
    a.out = res->words; a.obp = res->bpos; a.meta = res->meta; a.cap = res->cap;
    a.recs = wg_fuse_recs(ctx, recs); a.sync = sync;
    a.aval = aval; a.anb = anb;
    a.withhold = ctx->test_withhold;
    ctx->test_withhold = 0xFFFFFFFFu;
    CUDA_TRY(ctx, cudaMemsetAsync(res->meta, 0, sizeof(DevMeta), ctx->stream));
    switch (op) {
    case OP_AND: launch_fuse_tile<OP_AND>(ctx, ft, ntiles, ctx->stream, a); break;
    case OP_OR: launch_fuse_tile<OP_OR>(ctx, ft, ntiles, ctx->stream, a); break;
    case OP_XOR: launch_fuse_tile<OP_XOR>(ctx, ft, ntiles, ctx->stream, a); break;
    default: launch_fuse_tile<OP_MINUS>(ctx, ft, ntiles, ctx->stream, a); break;
    }
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError());
    bv_launched(res);
    res->gt_valid = false;
    res->rows_valid = false;
    res->used = false;
    res->compressed_form = true;
    return WAHGPU_OK;
}

// Single-pass warp-tile engine (wah_gone.cuh): one launch per call, one
// warp per 1024-group tile, operands read once, words written once.
int wg_launch_gone(wahgpu_ctx* ctx, int op, wahgpu_bv* x, wahgpu_bv* y, uint32_t groups,
                   uint32_t anb, uint32_t aval, wahgpu_bv* res) {
    int rc = bv_reserve(res, (uint64_t)x->h.n + y->h.n);
    if (rc) return rc;
    if (groups == 0) return wg_launch_gop(ctx, GK_CANON, op, x, y, groups, anb, aval, res);
    rc = wg_gtile(x);
    if (rc) return rc;
    rc = wg_gtile(y);
    if (rc) return rc;
    const uint32_t ntiles = (groups + GT - 1) / GT;
    TileRec* recs; LaunchSync* sync;
    rc = wg_scratch(ctx, ntiles, &recs, &sync);
    if (rc) return rc;
    FuseArgs a;
    a.xw = x->words; a.xgt = x->gt; a.nx = x->h.n;
    a.yw = y->words; a.ygt = y->gt; a.ny = y->h.n;
    a.groups = groups; a.ntiles = ntiles;
    a.out = res->words; a.obp = res->bpos; a.meta = res->meta; a.cap = res->cap;
    a.recs = wg_fuse_recs(ctx, recs); a.sync = sync;
    a.aval = aval; a.anb = anb;
    a.withhold = ctx->test_withhold;
    ctx->test_withhold = 0xFFFFFFFFu;
    CUDA_TRY(ctx, cudaMemsetAsync(res->meta, 0, sizeof(DevMeta), ctx->stream));
    const uint32_t grid = (ntiles + GWARPS - 1) / GWARPS;
    const size_t sm = GWARPS * sizeof(GoneWarp);
    static PerDeviceSetup setup[4];
    cudaStream_t s = ctx->stream;
    switch (op) {
    case OP_AND:
        wg_kernel_setup(setup[0], ctx->device, k_gone<OP_AND>, GTHREADS, sm);
        k_gone<OP_AND><<<grid, GTHREADS, sm, s>>>(a);
        break;
    case OP_OR:
        wg_kernel_setup(setup[1], ctx->device, k_gone<OP_OR>, GTHREADS, sm);
        k_gone<OP_OR><<<grid, GTHREADS, sm, s>>>(a);
        break;
    case OP_XOR:
        wg_kernel_setup(setup[2], ctx->device, k_gone<OP_XOR>, GTHREADS, sm);
        k_gone<OP_XOR><<<grid, GTHREADS, sm, s>>>(a);
        break;
    default:
        wg_kernel_setup(setup[3], ctx->device, k_gone<OP_MINUS>, GTHREADS, sm);
        k_gone<OP_MINUS><<<grid, GTHREADS, sm, s>>>(a);
        break;
    }
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError());
    bv_launched(res);
    res->gt_valid = false;
    res->rows_valid = false;
    res->used = false;
    res->compressed_form = true;
    return WAHGPU_OK;
}

// Group space or word space for an operator on the reference's _c2 path, and
// for copies and complements (y null): group space costs by the groups, the
// merge by the words, each at least its chain of steps.  Curves through
// measured calls of & | - at 2^16 .. 2^28 bits, d = 1e-4 .. 0.06, in us:
// group space 7.3 at 0.13M groups, 15 at 2.2M, 41 at 8.7M; merge 7.7 at 400
// words of both operands, 9.8 at 7 K, 12.3 at 63 K, 17 at 0.4M, 29 at 1.4M,
// 72 at 4M.  The row index an operand lacks is charged to its first use; an
// operand that comes back is taken to come again.  A merge tile set on the
// context asks for the merge.  A captured call may not allocate: it takes
// group space only where the call before it has left all that it needs.
static bool in_group_space(wahgpu_ctx* ctx, wahgpu_bv* x, wahgpu_bv* y, uint32_t groups) {
    if (ctx->merge_tile) return false;
    const bool fits = ctx->ws_bytes >= gop_bytes(groups);
    if ((!x->rows_valid || (y && !y->rows_valid) || !fits) && wg_capturing(ctx)) return false;
    const double g = groups * 1e-6, n = (double)x->h.n + (y ? y->h.n : 0);
    double in_groups = 6.6 + (y ? 4.0 : 3.1) * g;
    for (wahgpu_bv* b : {x, y}) {
        if (!b) continue;
        if (!b->rows_valid && (!b->used || b->replayed)) in_groups += 3.0 + 1.5 * g;
        b->used = true;
    }
    return in_groups < 7.0 + 0.5 * std::log2(1.0 + n / 200.0) + (y ? 13e-6 : 10e-6) * n;
}

// Both fall back to the merge, which needs next to no scratch, where group
// space does not find the memory.
static int launch_fsm(wahgpu_ctx* ctx, int op, wahgpu_bv* x, wahgpu_bv* y, uint32_t groups, uint32_t anb, uint32_t aval,
                      wahgpu_bv* res) {
    int rc = bv_reserve(res, (uint64_t)x->h.n + y->h.n);
    if (rc) return rc;
    if (in_group_space(ctx, x, y, groups)) {
        rc = wg_launch_gop(ctx, GK_FSM, op, x, y, groups, anb, aval, res);
        if (rc != WAHGPU_ENOMEM) return rc;
    }
    return wg_launch_merge(ctx, op, true, false, false, x, y, groups, anb, aval, res);
}
// x, or its complement, as compress() leaves it.
static int launch_copy(wahgpu_ctx* ctx, bool flip, wahgpu_bv* x, uint32_t groups, uint32_t anb, uint32_t aval,
                       wahgpu_bv* res) {
    int rc = bv_reserve(res, x->h.n);
    if (rc) return rc;
    if (groups > 0 && x->h.n > 0 && in_group_space(ctx, x, nullptr, groups)) {
        rc = wg_launch_gop(ctx, flip ? GK_FLIP : GK_COPY, 0, x, nullptr, groups, anb, aval, res);
        if (rc != WAHGPU_ENOMEM) return rc;
    }
    return wg_launch_merge(ctx, 0, false, true, flip, x, nullptr, groups, anb, aval, res);
}

// A one-word device bitvector holding the collapsed form of an all-zero
// operand (do_cnt(), src/bitvector.cpp:601-604).
static int collapsed_copy(wahgpu_ctx* ctx, const wahgpu_bv* src, wahgpu_bv** out) {
    wahgpu_bv* b = wg_bv_new(ctx);
    if (!b) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    int rc = bv_reserve(b, 1);
    if (rc) { wahgpu_bv_free(b); return rc; }
    uint32_t* st = reinterpret_cast<uint32_t*>(reinterpret_cast<DevMeta*>(ctx->h_meta_stage) + META_SLOTS);
    st[0] = HEADER0 | src->h.groups;
    st[1] = 0;
    st[2] = src->h.groups;
    CUDA_TRY(ctx, cudaMemcpyAsync(b->words, st, 4, cudaMemcpyHostToDevice, ctx->stream));
    CUDA_TRY(ctx, cudaMemcpyAsync(b->bpos, st + 1, 8, cudaMemcpyHostToDevice, ctx->stream));
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    b->h = src->h;
    b->h.n = 1;
    b->h.w0 = st[0];
    b->h.nfill = 1;
    b->h_valid = true;
    b->told = true;
    // device meta mirrors the host copy
    CUDA_TRY(ctx, cudaMemcpyAsync(b->meta, &b->h, sizeof(DevMeta), cudaMemcpyHostToDevice, ctx->stream));
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    *out = b;
    return WAHGPU_OK;
}

static OperandMeta opmeta(const wahgpu_bv* b) {
    OperandMeta m;
    m.n = b->h.n; m.groups = b->h.groups; m.anb = b->h.anb; m.aval = b->h.aval;
    m.nset = b->h.nset; m.w0 = b->h.w0;
    return m;
}

// Engine for a canonical-result operator (WAHGPU_TUNE_DENSE_ENGINE): 1 the
// pipelined group-space kernel, 2 the word-space merge, 3 the two-pass
// group-space kernels (0, the default, too), 4 / 5 the single-pass
// group-space kernels over CTA / warp tiles.
static bool dense_in_word_space(const wahgpu_ctx* ctx, const wahgpu_bv*, const wahgpu_bv*, uint32_t) {
    return ctx->dense_engine == 2;
}
static bool dense_two_pass(const wahgpu_ctx* ctx) {
    return ctx->dense_engine == 0 || ctx->dense_engine == 3;
}
static bool dense_fused(const wahgpu_ctx* ctx) {
    return ctx->dense_engine == 4;
}
static bool dense_warp_tiles(const wahgpu_ctx* ctx) {
    return ctx->dense_engine == 5;
}

// adjustSize(0, nt) of a copy of b (src/bitvector.cpp:4086-4108): the copy
// grows by appendFill(0, nt - size()) (src/bitvector.h:800-831), whose
// append_active / append_counter (699-760) may merge into b's last word, so
// the copy keeps b's words up to the last one and the rest is rebuilt here.
static int padded_copy(wahgpu_ctx* ctx, wahgpu_bv* b, uint64_t nt, wahgpu_bv** out) {
    *out = nullptr;
    const uint32_t n = b->h.n;
    std::vector<uint32_t> t;  // b's last word, then the appended words
    if (n) {
        uint32_t last = 0;
        CUDA_TRY(ctx, cudaMemcpyAsync(&last, b->words + n - 1, 4, cudaMemcpyDeviceToHost, ctx->stream));
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        t.push_back(last);
    }
    // append_active of a literal (bitvector.h:699-737)
    auto push_active = [&](uint32_t v) {
        if (t.empty()) { t.push_back(v); return; }
        uint32_t& bk = t.back();
        if (v == 0) {
            if (bk == 0) bk = HEADER0 + 2;
            else if (bk >= HEADER0 && bk < HEADER1) ++bk;
            else t.push_back(v);
        } else if (v == ALLONES) {
            if (bk == ALLONES) bk = HEADER1 | 2;
            else if (bk >= HEADER1) ++bk;
            else t.push_back(v);
        } else {
            t.push_back(v);
        }
    };
    // append_counter(0, cnt) (bitvector.h:741-760)
    auto push_zeros = [&](uint32_t cnt) {
        const uint32_t w = HEADER0 + cnt;
        if (t.empty()) { t.push_back(w); return; }
        uint32_t& bk = t.back();
        if ((bk >> 30) == 2u) bk += cnt;
        else if (bk == 0) bk = w + 1;
        else t.push_back(w);
    };
    uint32_t anb = b->h.anb, aval = b->h.aval;
    uint64_t need = nt - ((uint64_t)b->h.groups * MAXBITS + anb);
    if (anb > 0) {
        const uint32_t k = (uint32_t)std::min<uint64_t>(MAXBITS - anb, need);
        anb += k;
        aval <<= k;
        need -= k;
        if (anb >= MAXBITS) { push_active(aval); anb = 0; aval = 0; }
    }
    if (need >= MAXBITS) {
        const uint64_t cnt = need / MAXBITS;
        if (cnt > MAXCNT) return wg_fail(ctx, WAHGPU_ERANGE, "padding of %llu groups", (unsigned long long)cnt);
        if (cnt > 1) push_zeros((uint32_t)cnt);
        else push_active(0);
        need -= cnt * MAXBITS;
    }
    if (need > 0) { anb = (uint32_t)need; aval = 0; }
    const uint32_t keep = n ? n - 1 : 0;
    const uint64_t m = (uint64_t)keep + t.size();
    wahgpu_bv* p = wg_bv_new(ctx);
    if (!p) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    int rc = bv_reserve(p, m);
    if (!rc && keep && cudaMemcpyAsync(p->words, b->words, (size_t)keep * 4, cudaMemcpyDeviceToDevice, ctx->stream))
        rc = wg_fail(ctx, WAHGPU_ECUDA, "copy failed");
    if (!rc && !t.empty() && (cudaMemcpyAsync(p->words + keep, t.data(), t.size() * 4, cudaMemcpyHostToDevice,
                                              ctx->stream) || cudaStreamSynchronize(ctx->stream)))
        rc = wg_fail(ctx, WAHGPU_ECUDA, "copy failed");
    if (!rc) rc = wg_scan_meta(p, (uint32_t)m, anb, aval);
    if (!rc) rc = wg_bv_meta(p);
    if (rc) { wahgpu_bv_free(p); return rc; }
    *out = p;
    return WAHGPU_OK;
}

// Operands of different sizes (src/bitvector.cpp:1194-1838): the shorter
// one is padded with 0 bits and the operator runs in its OP= form — for
// a OP b with a longer a: res = b padded, res OP= a (& | ^) or res = a,
// res -= b padded (-); with a shorter a: res = a padded, res OP= b; for
// a OP= b: a OP= (b padded), or (a padded) OP= b.
static int binop_unequal(wahgpu_ctx* ctx, int op, bool inplace, wahgpu_bv* a, wahgpu_bv* b, wahgpu_bv* res) {
    const uint64_t sa = (uint64_t)a->h.groups * MAXBITS + a->h.anb;
    const uint64_t sb = (uint64_t)b->h.groups * MAXBITS + b->h.anb;
    wahgpu_bv* pad = nullptr;
    int rc = padded_copy(ctx, sa > sb ? b : a, sa > sb ? sa : sb, &pad);
    if (rc) return rc;
    if (sa < sb) rc = wahgpu_bv_binop_into(ctx, op, 1, pad, b, res);
    else if (inplace || op == OP_MINUS) rc = wahgpu_bv_binop_into(ctx, op, 1, a, pad, res);
    else rc = wahgpu_bv_binop_into(ctx, op, 1, pad, a, res);
    cudaStreamSynchronize(ctx->stream);
    wahgpu_bv_free(pad);
    return rc;
}

extern "C" int wahgpu_bv_binop_into(wahgpu_ctx* ctx, int op, int inplace, wahgpu_bv* a, wahgpu_bv* b,
                                    wahgpu_bv* res) {
    if (!ctx || !a || !b || !res || op < 0 || op > 3) return wg_fail(ctx, WAHGPU_EINVAL, "bad argument");
    if (res == a || res == b) return wg_fail(ctx, WAHGPU_EINVAL, "result must differ from the operands");
    int rc = wg_bv_meta(a);
    if (rc) return rc;
    rc = wg_bv_meta(b);
    if (rc) return rc;
    OperandMeta ma = effective(opmeta(a)), mb = effective(opmeta(b));
    Plan p = plan_binop(op, inplace != 0, ma, mb);
    if (p.kind == PK_UNEQUAL) {
        // pad the operands the reference would hold (an all-0 one collapsed
        // by do_cnt, src/bitvector.cpp:601-604)
        wahgpu_bv* ea = a;
        wahgpu_bv* eb = b;
        wahgpu_bv* ta = nullptr;
        wahgpu_bv* tb = nullptr;
        if (ma.n != a->h.n) { rc = collapsed_copy(ctx, a, &ta); if (rc) return rc; ea = ta; }
        if (mb.n != b->h.n) { rc = collapsed_copy(ctx, b, &tb); if (rc) { if (ta) wahgpu_bv_free(ta); return rc; } eb = tb; }
        rc = binop_unequal(ctx, op, inplace != 0, ea, eb, res);
        if (ta || tb) {
            cudaStreamSynchronize(ctx->stream);
            if (ta) wahgpu_bv_free(ta);
            if (tb) wahgpu_bv_free(tb);
        }
        return rc;
    }
    const uint32_t G = ma.groups;
    if (G >= 2 && ((ma.n == G && a->h.nfill && ma.n == a->h.n) || (mb.n == G && b->h.nfill && mb.n == b->h.n)))
        return wg_fail(ctx, WAHGPU_EDEGENERATE,
                       "an operand has one word per group and count-1 fill words; the reference "
                       "combines such fill headers as literal bits");
    const uint32_t aval = combine_active(op, a->h.aval, b->h.aval);
    const uint32_t anb = a->h.anb;
    wahgpu_bv* ca = a;
    wahgpu_bv* cb = b;
    wahgpu_bv* tmpa = nullptr;
    wahgpu_bv* tmpb = nullptr;
    if (ma.n != a->h.n) { rc = collapsed_copy(ctx, a, &tmpa); if (rc) return rc; ca = tmpa; }
    if (mb.n != b->h.n) { rc = collapsed_copy(ctx, b, &tmpb); if (rc) { if (tmpa) wahgpu_bv_free(tmpa); return rc; } cb = tmpb; }
    switch (p.kind) {
    case PK_MERGE_FSM:
        rc = launch_fsm(ctx, op, ca, cb, G, anb, aval, res);
        break;
    case PK_MERGE_CANON:
        // canonical result: the group-space kernel, or the word-space merge
        // (no step states) when the tuning asks for it
        if (dense_in_word_space(ctx, ca, cb, G))
            rc = wg_launch_merge(ctx, op, false, false, false, ca, cb, G, anb, aval, res);
        else if (dense_warp_tiles(ctx))
            rc = wg_launch_gone(ctx, op, ca, cb, G, anb, aval, res);
        else if (dense_fused(ctx))
            rc = wg_launch_fuse(ctx, op, ca, cb, G, anb, aval, res);
        else if (dense_two_pass(ctx))
            rc = wg_launch_gop(ctx, GK_CANON, op, ca, cb, G, anb, aval, res);
        else
            rc = wg_launch_dense(ctx, op, ca, cb, G, anb, aval, res);
        break;
    case PK_COPY:
    case PK_COPY_FLIP:
        rc = launch_copy(ctx, p.kind == PK_COPY_FLIP, p.src ? cb : ca, G, anb, aval, res);
        break;
    default: {
        rc = bv_reserve(res, 1);
        if (rc) break;
        int mode = p.kind == PK_EMPTY ? 0 : (p.kind == PK_RAW1 ? 1 : 2);
        cudaError_t e = cudaMemsetAsync(res->meta, 0, sizeof(DevMeta), ctx->stream);
        if (e != cudaSuccess) { rc = wg_fail(ctx, WAHGPU_ECUDA, "memset failed"); break; }
        k_small<<<1, 32, 0, ctx->stream>>>(mode, op, ca->words, cb->words, p.fill_n, G, res->words, res->bpos,
                                           res->meta, anb, aval);
        ctx->launches++;
        e = cudaGetLastError();
        if (e != cudaSuccess) { rc = wg_fail(ctx, WAHGPU_ECUDA, "launch failed: %s", cudaGetErrorString(e)); break; }
        bv_launched(res);
        res->gt_valid = false;
        res->rows_valid = false;
        res->used = false;
        res->compressed_form = true;
    }
    }
    if (tmpa || tmpb) {
        cudaStreamSynchronize(ctx->stream);
        if (tmpa) wahgpu_bv_free(tmpa);
        if (tmpb) wahgpu_bv_free(tmpb);
    }
    return rc;
}

extern "C" int wahgpu_bv_binop(wahgpu_ctx* ctx, int op, int inplace, wahgpu_bv* a, wahgpu_bv* b,
                               wahgpu_bv** res) {
    if (!res) return wg_fail(ctx, WAHGPU_EINVAL, "res is NULL");
    *res = nullptr;
    wahgpu_bv* r = wg_bv_new(ctx);
    if (!r) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    int rc = wahgpu_bv_binop_into(ctx, op, inplace, a, b, r);
    if (rc) { wahgpu_bv_free(r); return rc; }
    *res = r;
    return WAHGPU_OK;
}

// Replaces b's storage with that of tmp (both on the same context).
static void bv_take(wahgpu_bv* b, wahgpu_bv* tmp) {
    std::swap(b->words, tmp->words);
    std::swap(b->bpos, tmp->bpos);
    std::swap(b->meta, tmp->meta);
    std::swap(b->cap, tmp->cap);
    std::swap(b->h, tmp->h);
    std::swap(b->h_valid, tmp->h_valid);
    std::swap(b->told, tmp->told);
    std::swap(b->gt, tmp->gt);
    std::swap(b->gt_valid, tmp->gt_valid);
    std::swap(b->rows, tmp->rows);
    std::swap(b->rows_cap, tmp->rows_cap);
    std::swap(b->rows_valid, tmp->rows_valid);
    std::swap(b->used, tmp->used);
    std::swap(b->replayed, tmp->replayed);
    b->compressed_form = tmp->compressed_form;
}

static int unary_op(wahgpu_bv* b, bool flip) {
    wahgpu_ctx* ctx = b->ctx;
    int rc = wg_bv_meta(b);
    if (rc) return rc;
    wahgpu_bv* r = wg_bv_new(ctx);
    if (!r) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    const uint32_t aval = flip && b->h.anb ? (b->h.aval ^ ((1u << b->h.anb) - 1)) : b->h.aval;
    if (b->h.n == 0) {
        rc = bv_reserve(r, 1);
        if (!rc) rc = wg_scan_meta(r, 0, b->h.anb, aval);
    } else {
        rc = launch_copy(ctx, flip, b, b->h.groups, b->h.anb, aval, r);
    }
    // the wait for the result brings its metadata along
    if (!rc) rc = wg_bv_meta(r);
    if (rc) { wahgpu_bv_free(r); return rc; }
    bv_take(b, r);
    wahgpu_bv_free(r);
    return WAHGPU_OK;
}
extern "C" int wahgpu_bv_compress(wahgpu_bv* b) {
    if (!b) return WAHGPU_EINVAL;
    if (b->compressed_form) return WAHGPU_OK;
    return unary_op(b, false);
}
extern "C" int wahgpu_bv_flip(wahgpu_bv* b) {
    if (!b) return WAHGPU_EINVAL;
    return unary_op(b, true);
}
extern "C" int wahgpu_bv_decompress(wahgpu_bv* b) {
    if (!b) return WAHGPU_EINVAL;
    wahgpu_ctx* ctx = b->ctx;
    int rc = wg_bv_meta(b);
    if (rc) return rc;
    const uint32_t G = b->h.groups;
    if (b->h.n == G) return WAHGPU_OK;  // already uncompressed
    wahgpu_bv* r = wg_bv_new(ctx);
    if (!r) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    rc = bv_reserve(r, G);
    if (!rc) rc = wg_rows(b);  // n > 0: words without groups would be as many
    if (!rc) {
        // the groups are b's: only the words and their number change
        r->h = b->h;
        r->h.n = G;
        r->h.w0 = wpattern(b->h.w0);
        r->h.nfill = 0;
        r->h_valid = true;
        r->told = true;
        r->rows_valid = result_rows(r, G);
        const uint32_t ntiles = (uint32_t)(((uint64_t)G + PT - 1) / PT);
        k_expand<<<(ntiles + GW - 1) / GW, GCTA, 0, ctx->stream>>>(b->words, b->rows, ntiles, r->words, r->bpos,
                                                                   r->rows_valid ? r->rows : nullptr, r->meta, r->h);
        ctx->launches++;
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = wg_fail(ctx, WAHGPU_ECUDA, "launch failed: %s", cudaGetErrorString(e));
    }
    if (rc) { wahgpu_bv_free(r); return rc; }
    cudaStreamSynchronize(ctx->stream);
    bv_take(b, r);
    b->compressed_form = false;
    wahgpu_bv_free(r);
    return WAHGPU_OK;
}

int64_t wg_rids_device(wahgpu_bv* b, uint32_t* dev_out, uint64_t cap, uint64_t* total) {
    wahgpu_ctx* ctx = b->ctx;
    int rc = wg_bv_meta(b);
    if (rc) return rc;
    const uint64_t cnt = (uint64_t)b->h.nset + __builtin_popcount(b->h.anb ? b->h.aval & ((1u << b->h.anb) - 1) : 0u);
    *total = cnt;
    if (cap < cnt) return wg_fail(ctx, WAHGPU_ESIZE, "need room for %llu row ids", (unsigned long long)cnt);
    const uint32_t n = b->h.n;
    const uint32_t ntiles = n ? (n + RIDS_TILE - 1) / RIDS_TILE : 1;
    TileRec* recs; LaunchSync* sync;
    rc = wg_scratch(ctx, ntiles, &recs, &sync);
    if (rc) return rc;
    unsigned long long* dtot = reinterpret_cast<unsigned long long*>(wg_alloc(ctx, 8));
    if (!dtot) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    k_rids<<<ntiles, SCAN_THREADS, 0, ctx->stream>>>(b->words, n, b->bpos, b->h.groups, b->h.anb, b->h.aval,
                                                      dev_out, cap, dtot, b->meta, recs, sync, ntiles);
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError());
    wg_free(ctx, dtot);
    return (int64_t)cnt;
}

extern "C" int64_t wahgpu_bv_rids_device(wahgpu_bv* b, uint32_t* dev_out, uint64_t cap) {
    if (!b || (cap && !dev_out)) return WAHGPU_EINVAL;
    uint64_t total = 0;
    return wg_rids_device(b, dev_out, cap, &total);
}

extern "C" int64_t wahgpu_bv_rids(wahgpu_bv* b, uint32_t* out, uint64_t cap) {
    if (!b || (cap && !out)) return WAHGPU_EINVAL;
    wahgpu_ctx* ctx = b->ctx;
    int rc = wg_bv_meta(b);
    if (rc) return rc;
    const uint64_t cnt = (uint64_t)b->h.nset + __builtin_popcount(b->h.anb ? b->h.aval & ((1u << b->h.anb) - 1) : 0u);
    if (cap < cnt) return wg_fail(ctx, WAHGPU_ESIZE, "need room for %llu row ids", (unsigned long long)cnt);
    if (cnt == 0) return 0;
    uint32_t* d = static_cast<uint32_t*>(wg_alloc(ctx, cnt * 4));
    if (!d) return wg_fail(ctx, WAHGPU_ENOMEM, "allocation failed");
    uint64_t total = 0;
    int64_t r = wg_rids_device(b, d, cnt, &total);
    if (r < 0) { wg_free(ctx, d); return r; }
    cudaError_t e = cudaMemcpyAsync(out, d, cnt * 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    wg_free(ctx, d);
    if (e != cudaSuccess) return wg_fail(ctx, WAHGPU_ECUDA, "row-id copy failed: %s", cudaGetErrorString(e));
    rc = wg_bv_meta(b);
    return rc ? rc : (int64_t)cnt;
}
