// Internal state behind the opaque handles of include/wahgpu.h.
#ifndef WAH_API_INTERNAL_H
#define WAH_API_INTERNAL_H
#include <cuda_runtime.h>
#include <atomic>
#include <mutex>
#include <string>
#include <vector>
#include "wah_dev.cuh"
#include "wah_pool.h"
#include "wah_budget.h"

struct wahgpu_ctx {
    int device = 0;
    int sm_count = 0;
    cudaStream_t stream = nullptr;      // where work is queued
    cudaStream_t own_stream = nullptr;  // the context's own stream
    std::string err;
    std::mutex mu;
    wah::BlockPool dev, host;  // device and pinned memory
    wahgpu_ctx();
    // look-back scratch: two LaunchSync words then TileRec records
    void* scratch = nullptr;
    uint32_t scratch_tiles = 0;
    bool scratch_captured = false;      // a captured call uses it
    void* h_meta_stage = nullptr;  // pinned staging for metadata reads
    // the bitvectors' metadata live in blocks of META_SLOTS, so that one copy
    // reads those of every result launched since the last read
    std::vector<wah::DevMeta*> meta_blocks, meta_free;
    std::vector<struct wahgpu_bv*> pending;  // launched, metadata not read yet
    void* ws = nullptr;            // scratch of one call (wg_workspace())
    size_t ws_bytes = 0;
    bool ws_captured = false;      // a captured call writes to it
    size_t kept_at_most = wah::KEPT_AT_MOST;  // row ids that a batch's count pass keeps, bytes
    uint64_t launches = 0;
    uint32_t dense_tile = 2048;         // WAHGPU_TUNE_DENSE_TILE
    uint32_t dense_engine = 0;          // WAHGPU_TUNE_DENSE_ENGINE
    uint32_t range_order = 1;           // WAHGPU_TUNE_RANGE_ORDER
    uint32_t range_ctas = 0;            // WAHGPU_TUNE_RANGE_CTAS (0: as many as fit)
    uint32_t merge_tile = 0;            // WAHGPU_TUNE_MERGE_TILE (0: by operand size)
    uint32_t cum_stride = 0;            // WAHGPU_TUNE_CUM_STRIDE (0 auto, 1 none)
    // failure-path test hooks (WAHGPU_TEST_*): the tile of the next
    // single-pass operator launch that never publishes its look-back record
    // (UINT32_MAX: none), and the allocations left before one fails (0: off)
    uint32_t test_withhold = 0xFFFFFFFFu;
    int64_t test_fail_alloc = 0;
};

constexpr uint32_t META_SLOTS = 128;

struct wahgpu_bv {
    wahgpu_ctx* ctx = nullptr;
    uint32_t* words = nullptr;  // m_vec
    uint32_t* bpos = nullptr;   // block positions: group where word 32k starts
    wah::DevMeta* meta = nullptr;
    uint32_t cap = 0;           // capacity in words
    wah::DevMeta h{};           // host copy of *meta
    bool h_valid = false;
    bool told = false;          // the device status in h has been reported
    int32_t pend = -1;          // its place in ctx->pending
    cudaStream_t pend_stream = nullptr;  // where it was launched
    bool replayed = false;      // a captured call writes to it: its words may change at any time
    uint32_t* gt = nullptr;     // group-tile index (k_gtile), built on first use
    bool gt_valid = false;
    uint2* rows = nullptr;      // row index (k_rows), built on first use or with the result
    uint32_t rows_cap = 0;      // rows it has room for
    bool rows_valid = false;
    bool used = false;          // has been an operand where group and word space compete
    bool compressed_form = false;  // words are as compress() leaves them
};

// A kernel's launch setup on each device (the dynamic shared-memory limit is
// a per-device setting): resident CTAs per SM once set up, 0 before.
struct PerDeviceSetup {
    std::atomic<int> per_sm[64];
};
// Sets the kernel's dynamic shared-memory limit on the current device the
// first time it launches there; returns its resident CTAs per SM.
template <class Kernel>
int wg_kernel_setup(PerDeviceSetup& s, int device, Kernel k, int threads, size_t smem) {
    const int d = device >= 0 && device < 64 ? device : 0;
    int v = s.per_sm[d].load(std::memory_order_relaxed);
    if (v) return v;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k, threads, smem);
    if (v < 1) v = 1;
    s.per_sm[d].store(v, std::memory_order_relaxed);
    return v;
}
// Launches a kernel that calls pdl_wait() before it touches memory so that
// its CTAs may be set up while the kernel before it on the stream drains.
template <class... Args, class... Params>
void wg_launch_pdl(void (*k)(Params...), uint32_t grid, uint32_t threads, size_t smem, cudaStream_t s, const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, args...);
}
int wg_fail(wahgpu_ctx* ctx, int code, const char* fmt, ...);
bool wg_capturing(const wahgpu_ctx* ctx);
unsigned char* wg_workspace(wahgpu_ctx* ctx, size_t bytes, bool captured);
void* wg_alloc(wahgpu_ctx* ctx, size_t bytes);
void wg_free(wahgpu_ctx* ctx, void* p);
void* wg_host_alloc(wahgpu_ctx* ctx, size_t bytes);
void wg_host_free(wahgpu_ctx* ctx, void* p);
int wg_scratch(wahgpu_ctx* ctx, uint32_t ntiles, wah::TileRec** recs, wah::LaunchSync** sync);
int wg_bv_meta(wahgpu_bv* b);
wahgpu_bv* wg_bv_new(wahgpu_ctx* ctx);
int wg_scan_meta(wahgpu_bv* b, uint32_t n, uint32_t anb, uint32_t aval);
int wg_launch_merge(wahgpu_ctx* ctx, int op, bool fsm, bool unary, bool flip,
                    const wahgpu_bv* x, const wahgpu_bv* y, uint32_t groups,
                    uint32_t anb, uint32_t aval, wahgpu_bv* res);
#endif
