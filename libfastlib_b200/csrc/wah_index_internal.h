// Internal state behind the opaque index and batch handles of
// include/wahgpu.h, shared by the index store (wah_index.cu) and the device
// index builder (wah_build.cu).
#ifndef WAH_INDEX_INTERNAL_H
#define WAH_INDEX_INTERNAL_H
#include <vector>
#include "wah_range.cuh"
#include "wah_api_internal.h"

struct wahgpu_index {
    wahgpu_ctx* ctx = nullptr;
    int kind = 0;                 // WAHGPU_RELIC / WAHGPU_BIN
    uint32_t nrows = 0, groups = 0, anb = 0, nobs = 0, ntiles = 0;
    std::vector<double> keys;     // relic: distinct values; bin: minval then maxval
    std::vector<uint64_t> bwords; // m_vec words per bitmap (for the complement choice)
    std::vector<uint32_t> bones;  // 1 bits per bitmap
    std::vector<uint64_t> cum_words, cum_ones;  // prefix sums of bwords / bones
    // bin: the bins holding rows, in bitmap order, and whether their
    // [minval, maxval] are ordered and disjoint (then locate searches them)
    std::vector<uint32_t> nonempty;
    bool bins_sorted = false;
    uint32_t* d_words = nullptr;
    wah::BitmapMeta* d_bm = nullptr;
    uint32_t* d_tiles = nullptr;
    uint32_t* d_tl_off = nullptr;     // per tile: bitmaps with a 1 bit there (CSR)
    uint32_t* d_tl_bm = nullptr;
    uint32_t* d_cum = nullptr;        // cumulative dense rows (range spans in two reads)
    uint32_t cum_stride = 0, cum_k = 0;
    bool disjoint = false;            // no row in two bitmaps
    bool partition = false;           // and every row in one
    void* d_values = nullptr;
    uint32_t vtype = 0;
    wah::DevIndex dev{};
};

struct wahgpu_batch {
    wahgpu_ctx* ctx = nullptr;
    uint32_t nq = 0, nterms = 0, nidx = 0;
    uint32_t groups = 0, anb = 0, ntiles = 0;  // tiles per query
    bool general = false;             // some term is not dense
    bool small = false;               // tiles of RT_SMALL groups
    // one device block of tables: indexes, terms, queries, then what a run
    // starts from (counts known beforehand: one-term count queries over
    // disjoint bitmaps, 0 for the others; row-id starts; status), then the
    // edges to count
    unsigned char* d_tab = nullptr;
    wah::DevIndex* d_idx = nullptr;
    wah::DevTerm* d_terms = nullptr;
    wah::DevQuery* d_queries = nullptr;
    unsigned char* d_init = nullptr;
    unsigned char* d_edges = nullptr;
    // one device block of results, copied back at once: counts, row-id
    // starts, status
    unsigned long long* d_counts = nullptr;
    unsigned long long* d_start = nullptr;
    wah::DevMeta* d_status = nullptr;
    size_t out_bytes = 0;
    unsigned char* h_out = nullptr;    // pinned
    uint32_t nrange = 0;              // queries k_range evaluates
    uint32_t nedges = 0, etiles = 0;  // edges to count, RT tiles per column
    uint32_t* d_rids = nullptr;
    uint64_t rid_cap = 0;
    uint32_t* d_dense = nullptr;
    size_t scan_tmp_bytes = 0;        // two-pass order, not capped: the scan's temporary storage
    std::vector<unsigned long long> h_counts, h_start;
    uint64_t bytes = 0;               // algorithmic bytes one run reads
    uint64_t min_bytes = 0;           // the bytes sumBins itself must read (covered set or complement)
    bool capped = false;              // row ids limited per query, each query in a region of its own
    bool few_ids = false;             // its limits leave most items unvisited by a second pass
    std::vector<uint64_t> h_lim, h_base;
    bool h_valid = false;
    bool captured = false;            // a graph may hold a run of it
    unsigned char* h_stage = nullptr;  // pinned staging of the uploaded tables
};

int wg_index_attach(wahgpu_index* x);
int wg_batch_fetch_all(wahgpu_batch* B, uint32_t* rids);
#endif
