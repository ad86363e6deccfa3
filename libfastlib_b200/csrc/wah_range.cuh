// Range evaluation over equality-encoded indexes (relic: one bitmap per
// distinct value; bin: one bitmap per value bin) and the AND across columns.
//
// The reference evaluates `lo <op> x <op> hi` as
//   relic::evaluate  (src/irelic.cpp:1827): locate -> sumBins(h0, h1)
//   bin::evaluate    (src/ibin.cpp:6614):   locate -> sumBins over the bins
//                    wholly inside the range, plus the rows of the edge
//                    bins whose values pass the comparison (checkBin /
//                    doScan on the raw values, src/ibin.cpp:2057-2304)
//   index::sumBins   (src/index.cpp:6450): OR of bitmaps [h0, h1), or the
//                    complement OR'ed and flipped when that reads fewer bytes
//   countQuery::doEvaluate (src/countQuery.cpp:953-1036): AND of the terms.
// The hit set is exactly the rows whose value passes the comparison done in
// double (qContinuousRange::inRange, src/qExpr.cpp:1647-1667); the reference's
// OR order (a heap ordered by pointer values) changes only the words of its
// intermediate results, never the bits.
//
// Work item = (query, tile of groups).  Every thread owns whole quads of
// groups and keeps the query's AND over them in registers.
//
// Dense terms.  Where the index keeps a cumulative row per bitmap (stride 1),
// a range's span is C(h1) & ~C(h0), two rows read as 16-byte vectors, and an
// edge bin's bitmap is C(j+1) & ~C(j): its set rows' raw values are compared
// right there.  No word is decoded, nothing is shared between threads and a
// count needs no block barrier.
//
// Other terms (rows kept for every few bitmaps, or none): warp 0 stages the
// term and its index in shared memory; a span covering whole blocks of the
// cumulative rows starts as C(k1) & ~C(k0), and the remaining bitmaps (the
// edges of such a span, a short span, or the tile's list of bitmaps holding a
// 1 bit in it) are OR'ed into a shared-memory accumulator: a bitmap with a
// few words over the tile by one lane (32 such bitmaps per warp at once), a
// longer one and each edge bin's row check by a whole warp walking its words
// 128 at a time (positions by ballot / scan).
//
// A query's dense terms go first; an empty AND skips the rest.
//
// Counts run tile by tile (the queries of a batch share a tile's rows and
// words in L2); where the CTAs take several items each, these are claimed one
// by one.  Row ids take one pass with a decoupled look-back in query order, or,
// for limits that leave most items unvisited, two tile by tile around a list of
// the others.
#ifndef WAH_RANGE_CUH
#define WAH_RANGE_CUH
#include "wah_dev.cuh"
#include "wah_keys.h"
#include "wah_budget.h"

namespace wah {

constexpr int RT = 4096;             // groups per tile
constexpr int RTHREADS = 256;
constexpr int RWARPS = RTHREADS / 32;
constexpr uint32_t RDIRECT = 32;     // spans of at most this many bitmaps skip the tile lists
constexpr int RCHK = 2;              // raw values in flight per lane in an edge-bin row check
constexpr int RQUADS = RT / 4 / RTHREADS;  // quads of groups per thread over an RT tile
static_assert(RQUADS * 4 * RTHREADS == RT, "quads");
// Tile of a batch of few items and dense terms only: a quad per thread, so
// one query over a million rows spreads over 32 CTAs instead of 8.
constexpr int RT_SMALL = 4 * RTHREADS;

// per-bitmap metadata of an attached index
struct BitmapMeta {
    uint64_t wstart;  // first m_vec word in the index's word pool
    uint32_t n;       // m_vec words
    uint32_t anb;     // active bits
    uint32_t aval;    // active value
    uint32_t groups;  // groups covered by m_vec (set by k_chunk_scan)
};

struct DevIndex {
    const uint32_t* words;     // word pool (the bitmaps' serialized arrays)
    const BitmapMeta* bm;      // nobs entries
    const uint32_t* tiles;     // nobs x (ntiles+1) x {word index, first group}
    const uint32_t* tl_off;    // ntiles+1: tile k's bitmaps are tl_bm[tl_off[k], tl_off[k+1])
    const uint32_t* tl_bm;     // bitmaps holding a 1 bit in each tile, ascending
    const uint32_t* cum;       // cum_k dense rows, gx words apart: row k-1 = OR of bitmaps [0, k*cum_stride)
    uint32_t cum_stride, cum_k, gx, pad2;  // gx: groups incl. the active one, rounded up to 4
    const void* values;        // raw column (nrows), or null
    uint32_t nobs;
    uint32_t ntiles;
};

struct DevTerm {
    uint32_t index;       // into the DevIndex table
    uint32_t h0, h1;      // bitmaps wholly inside: [h0, h1)
    uint32_t flip;        // OR the complement [0,h0) u [h1,nobs) and flip
    // with cumulative rows: [h0, h1) = C(c1) & ~C(c0) | OR of [h0, e0) and
    // [e1, h1), C(k) = row k-1 of DevIndex::cum (C(0) empty); c1 == 0: unused
    uint32_t c0, c1, e0, e1;
    uint32_t ncand;       // edge bitmaps to check row by row (0..2)
    uint32_t cand[2];
    uint32_t klo, kspan;  // the range in value keys
    uint32_t kflip, ksign;  // the column's KeyMap
    uint32_t dense;       // the index keeps a row per bitmap: span C(c1) & ~C(c0) (c1 == 0: empty), edges by rows
    uint32_t pad;
    const uint32_t* cum;  // dense: the index's rows
};

struct DevQuery {
    uint32_t t0, t1;      // terms [t0, t1): dense ones up to td, then the others
    uint32_t td, q;       // q: the query's place in the counts
    uint64_t rid_base;    // capped batches: the query's row-id region
    uint64_t rid_lim;     // capped batches: at most this many row ids (the first ones)
};

struct RangeArgs {
    const DevIndex* idx;
    const DevTerm* terms;
    const DevQuery* queries;
    uint32_t nq;
    uint32_t groups;          // whole groups per column (nrows / 31)
    uint32_t anb;             // rows past the last whole group
    uint32_t ntiles;          // tiles per query
    unsigned long long* counts;  // per query (zeroed by the caller)
    uint32_t* rids;           // row ids, all queries back to back (or null)
    uint64_t rid_cap;
    unsigned long long* rid_start;  // per query: offset of its first row id
    uint32_t* dense;          // dense hit words of query 0 (or null)
    TileRec* recs; LaunchSync* sync; uint32_t nitems;
    DevMeta* status;
    uint32_t gx;              // words per cumulative row
    uint32_t tile_major;      // 1: items ordered tile by tile, else query by query
    // two passes: the first adds each item's hits to item_cnt (zeroed), a scan turns
    // them into item_off, the second writes the row ids; items are indexed
    // q*ntiles + k
    unsigned long long* item_cnt;
    const unsigned long long* item_off;
    // capped: {item, ids before it within its query}: the items to evaluate
    // from the front (status->n of them), those whose ids are in their slots
    // from the back (status->groups)
    const uint2* item_list;
    uint32_t* slots;             // two passes: RSLOT row ids per item, in any order (or null)
    // 1: every query writes at most rid_lim row ids into its own region at
    // rid_base (one pass: offsets within the query by a segmented look-back;
    // two: a list of the items holding ids under their query's limit)
    uint32_t capped;
};

// Row ids kept by the count pass for an item with at most so many: the id
// pass orders and copies them instead of evaluating the item again.  A
// conjunction that needs many items to fill its limit has few hits in each.
// 32: a lane each, 128 bytes of scratch per item.  When added, before the items
// were claimed: 1024 conjunctions over 10M rows, 256 ids each, 3.06 -> 2.64 ms of
// kernels (with 4 terms 1.19 -> 0.90; one term, many hits in every item, 0.35 ->
// 0.36).
constexpr uint32_t RSLOT = KEPT_IDS;
static_assert(RSLOT == 32, "a lane each");
static_assert(RECORD_BYTES == sizeof(TileRec), "what the server charges a tile");

// 64-bit sums segmented at the first item of each query: {sum lo, sum hi,
// -, head}; (f1, s1) + (f2, s2) = (f1 | f2, f2 ? s2 : s1 + s2) is
// associative, so the look-back may combine in any grouping.
struct SegSum64Comb {
    __device__ __forceinline__ uint4 operator()(uint4 a, uint4 b) const {
        if (b.w) return b;
        const uint64_t s = ((uint64_t)a.y << 32 | a.x) + ((uint64_t)b.y << 32 | b.x);
        return make_uint4((uint32_t)s, (uint32_t)(s >> 32), 0u, a.w);
    }
};

enum RangeMode : int {
    RM_COUNT = 0,   // the queries' counts
    RM_ITEMS = 1,   // two passes, first: counts per item too
    RM_IDS = 2,     // two passes, second: row ids at the items' offsets
    RM_LOOK = 3     // one pass: counts and row ids, offsets by a look-back
};
constexpr uint32_t RSTAGE = 32 * 31 + 4;  // row ids of 32 groups at most, from the output's place in 16 bytes on
struct RangeShared {
    uint32_t hdr[8];
    uint64_t base;
    uint32_t sums[2][RWARPS];
    DevTerm term;    // the term being evaluated and its index (terms that are not dense)
    DevIndex index;
    // the accumulator of a term that is not dense (RT words), then the
    // row-id staging (RWARPS * RSTAGE)
    alignas(16) uint32_t tmp[1];
};
constexpr size_t range_smem(bool general, bool ids) {
    return sizeof(RangeShared) + 4 * (size_t)(ids ? RWARPS * RSTAGE : general ? RT : 0);
}
static_assert(RT <= RWARPS * (int)RSTAGE, "the staging covers the accumulator");
constexpr uint32_t TERM_WORDS = sizeof(DevTerm) / 4, INDEX_WORDS = sizeof(DevIndex) / 4;
static_assert(sizeof(DevTerm) % 4 == 0 && TERM_WORDS <= 32, "a warp stages a term");
static_assert(sizeof(DevIndex) % 4 == 0 && INDEX_WORDS <= 32, "a warp stages an index");

#ifndef WAH_RANGE_TYPES_ONLY
// Shared-memory place of tile group l in the accumulators: bits 2-4 XOR'ed
// with bits 5-7, so groups 32 apart (a sparse bitmap's set bits often are)
// fall in different banks while every aligned quad of groups stays one
// 16-byte vector in order.  rsw4: the same for quad index l (groups 4l..).
__device__ __forceinline__ uint32_t rsw(uint32_t l) { return l ^ (((l >> 5) & 7u) << 2); }
__device__ __forceinline__ uint32_t rsw4(uint32_t l) { return l ^ ((l >> 3) & 7u); }
// Does a raw value (4 bytes of the column) pass the term's comparison?
__device__ __forceinline__ bool pass_key(uint32_t v, const DevTerm& T) {
    return value_key(v, KeyMap{T.kflip, T.ksign}) - T.klo <= T.kspan;
}

// One warp ORs bitmap b's words for the tile [g0, g1) into S.tmp (the
// virtual group G holds the active bits).
__device__ __forceinline__ void warp_or_bitmap(RangeShared& S, const DevIndex& I, uint32_t b, uint32_t k,
                                               uint32_t g0, uint32_t g1, uint32_t G, uint32_t anb) {
    const uint32_t lane = threadIdx.x & 31u;
    const BitmapMeta m = I.bm[b];
    const uint32_t* tix = I.tiles + ((size_t)b * (I.ntiles + 1) + k) * 2;
    const uint32_t i0 = __ldg(tix), s0 = __ldg(tix + 1);
    const uint32_t in1 = __ldg(tix + 2), sn1 = __ldg(tix + 3);
    const uint32_t i1 = min(sn1 < g1 ? in1 + 1u : in1, m.n);  // words covering [g0, min(g1, G))
    const uint32_t* w = I.words + m.wstart;
    uint32_t carry = s0;
    // four 32-word chunks are loaded before any is placed, so one memory
    // latency covers 128 words
    for (uint32_t base0 = i0; base0 < i1; base0 += 128) {
        uint32_t wv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t i = base0 + 32u * j + lane;
            wv[j] = i < i1 ? __ldg(w + i) : 0u;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t base = base0 + 32u * j;
            if (base >= i1) break;
            const uint32_t i = base + lane;
            const bool in = i < i1;
            const uint32_t wd = wv[j];
            const uint32_t c = in ? wgroups(wd) : 0u;
            uint32_t p;
            const uint32_t fm = __ballot_sync(0xffffffffu, in && is_fill(wd));
            if (fm == 0) {
                p = carry + lane;
                carry += __popc(__ballot_sync(0xffffffffu, in));
            } else {
                uint32_t x = c;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) { uint32_t t = __shfl_up_sync(0xffffffffu, x, d); if (lane >= (uint32_t)d) x += t; }
                p = carry + x - c;
                carry += __shfl_sync(0xffffffffu, x, 31);
            }
            if (in && wd != 0u && !(is_fill(wd) && wd < HEADER1)) {
                const uint32_t a = max(p, g0), e = min(p + c, g1);
                const uint32_t pat = wpattern(wd);
                for (uint32_t g = a; g < e; ++g) {
                    if (pat == ALLONES) S.tmp[rsw(g - g0)] = ALLONES;
                    else atomicOr(&S.tmp[rsw(g - g0)], pat);
                }
            }
        }
    }
    // the bitmap's active bits form the group after its whole words (the
    // virtual group G when the bitmap covers every row)
    const uint32_t Gb = m.groups;
    if (lane == 0 && m.anb > 0 && Gb >= g0 && Gb < g1) {
        const uint32_t pat = (m.aval & ((1u << m.anb) - 1u)) << (31u - m.anb);
        if (pat) atomicOr(&S.tmp[rsw(Gb - g0)], pat);
    }
}

// An edge bin's row check by one warp: the bin's rows in the tile [g0, g1)
// whose raw values pass the term's comparison are OR'ed into S.tmp.  The
// bin's words are taken 128 at a time; the first set row of every literal
// of the batch has its raw value loaded before any is compared (one memory
// latency per batch for the usual one-row literals of a sparse bin), the
// other rows of a literal and the rows of 1-fills RCHK at a time after.
__device__ __forceinline__ void warp_check_bitmap(RangeShared& S, const DevIndex& I, uint32_t b, uint32_t k,
                                                  uint32_t g0, uint32_t g1, const DevTerm& T) {
    const uint32_t lane = threadIdx.x & 31u;
    const BitmapMeta m = I.bm[b];
    const uint32_t* tix = I.tiles + ((size_t)b * (I.ntiles + 1) + k) * 2;
    const uint32_t i0 = __ldg(tix), s0 = __ldg(tix + 1);
    const uint32_t in1 = __ldg(tix + 2), sn1 = __ldg(tix + 3);
    const uint32_t i1 = min(sn1 < g1 ? in1 + 1u : in1, m.n);
    const uint32_t* w = I.words + m.wstart;
    const uint32_t* raw = reinterpret_cast<const uint32_t*>(I.values);  // every column type is 4 bytes a row
    uint32_t carry = s0;
    for (uint32_t base0 = i0; base0 < i1; base0 += 128) {
        uint32_t wv[4], pv[4], cv[4], v0[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t i = base0 + 32u * j + lane;
            wv[j] = i < i1 ? __ldg(w + i) : 0u;
        }
        // each row's first group per word
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t base = base0 + 32u * j;
            pv[j] = 0; cv[j] = 0;
            if (base < i1) {
                const bool in = base + lane < i1;
                const uint32_t wd = wv[j];
                const uint32_t c = in ? wgroups(wd) : 0u;
                if (__ballot_sync(0xffffffffu, in && is_fill(wd)) == 0u) {
                    pv[j] = carry + lane;
                    carry += __popc(__ballot_sync(0xffffffffu, in));
                } else {
                    uint32_t x = c;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) { uint32_t t = __shfl_up_sync(0xffffffffu, x, d); if (lane >= (uint32_t)d) x += t; }
                    pv[j] = carry + x - c;
                    carry += __shfl_sync(0xffffffffu, x, 31);
                }
                cv[j] = c;
            }
        }
        // the first set row of every literal in the tile, all loads in flight
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t wd = wv[j];
            const bool lit = cv[j] == 1u && !is_fill(wd) && wd != 0u && pv[j] >= g0 && pv[j] < g1;
            v0[j] = lit ? __ldg(raw + pv[j] * 31u + (__clz(wd) - 1u)) : 0u;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t wd = wv[j], c = cv[j], p = pv[j];
            if (c == 0u || wd == 0u || (is_fill(wd) && wd < HEADER1)) continue;
            const bool lit = c == 1u && !is_fill(wd);
            const uint32_t a = max(p, g0), e = min(p + c, g1);
            for (uint32_t g = a; g < e; ++g) {
                uint32_t bits = wpattern(wd), set = 0;
                if (lit) {
                    const uint32_t hb = 31u - __clz(bits);
                    if (pass_key(v0[j], T)) set |= 1u << hb;
                    bits &= ~(1u << hb);
                }
                while (bits) {
                    uint32_t hb[RCHK], v[RCHK];
#pragma unroll
                    for (int q = 0; q < RCHK; ++q) {
                        hb[q] = bits ? 31u - __clz(bits) : 32u;
                        if (bits) bits &= ~(1u << hb[q]);
                    }
#pragma unroll
                    for (int q = 0; q < RCHK; ++q)
                        v[q] = hb[q] < 32u ? __ldg(raw + g * 31u + (30u - hb[q])) : 0u;
#pragma unroll
                    for (int q = 0; q < RCHK; ++q)
                        if (hb[q] < 32u && pass_key(v[q], T))
                            set |= 1u << hb[q];
                }
                if (set) atomicOr(&S.tmp[rsw(g - g0)], set);
            }
        }
    }
    // the bitmap's active bits form the group after its whole words
    const uint32_t Gb = m.groups;
    if (lane == 0 && m.anb > 0 && Gb >= g0 && Gb < g1) {
        uint32_t bits = (m.aval & ((1u << m.anb) - 1u)) << (31u - m.anb), set = 0;
        while (bits) {
            const uint32_t hb = 31u - __clz(bits);
            const uint32_t row = Gb * 31u + (30u - hb);
            if (pass_key(__ldg(raw + row), T)) set |= 1u << hb;
            bits &= ~(1u << hb);
        }
        if (set) atomicOr(&S.tmp[rsw(Gb - g0)], set);
    }
}

// Bitmaps with at most LSHORT words over the tile are OR'ed by one lane
// each; longer ones (or one holding a 1-fill longer than LFILL groups of
// the tile) by the whole warp.
constexpr uint32_t LSHORT = 4, LFILL = 8;

// One lane per bitmap: lane l ORs bitmap b (valid when `have`) into S.tmp
// when its words over the tile are few: its metadata, tile-index entries
// and words are loaded by all lanes at once, so 32 sparse bitmaps cost
// three memory round trips instead of three each.  The bitmaps left over
// are OR'ed by the whole warp, one after the other.
__device__ __forceinline__ void lanes_or_bitmaps(RangeShared& S, const DevIndex& I, bool have, uint32_t b,
                                                 uint32_t k, uint32_t g0, uint32_t g1, uint32_t G, uint32_t anb) {
    uint32_t i0 = 0, i1 = 0, s0 = 0, gb = 0, banb = 0, aval = 0;
    uint64_t wstart = 0;
    if (have) {
        const BitmapMeta* m = I.bm + b;
        const uint32_t* tix = I.tiles + ((size_t)b * (I.ntiles + 1) + k) * 2;
        wstart = __ldg(&m->wstart);
        const uint32_t n = __ldg(&m->n);
        banb = __ldg(&m->anb); aval = __ldg(&m->aval); gb = __ldg(&m->groups);
        i0 = __ldg(tix); s0 = __ldg(tix + 1);
        const uint32_t in1 = __ldg(tix + 2), sn1 = __ldg(tix + 3);
        i1 = min(sn1 < g1 ? in1 + 1u : in1, n);
    }
    bool lng = have && i1 > i0 + LSHORT;
    if (have && !lng) {
        const uint32_t* w = I.words + wstart;
        uint32_t wv[LSHORT];
#pragma unroll
        for (uint32_t j = 0; j < LSHORT; ++j) wv[j] = i0 + j < i1 ? __ldg(w + i0 + j) : 0u;
        uint32_t p = s0;
#pragma unroll
        for (uint32_t j = 0; j < LSHORT; ++j) {
            if (i0 + j >= i1) break;
            const uint32_t wd = wv[j];
            const uint32_t c = wgroups(wd);
            if (!is_fill(wd)) {
                if (wd && p >= g0 && p < g1) atomicOr(&S.tmp[rsw(p - g0)], wd);
            } else if (wd >= HEADER1) {
                const uint32_t a = max(p, g0), e = min(p + c, g1);
                if (e > a + LFILL) lng = true;  // the warp paints it (OR is idempotent)
                else for (uint32_t g = a; g < e; ++g) S.tmp[rsw(g - g0)] = ALLONES;
            }
            p += c;
        }
        // the active bits form the group after the whole words
        if (!lng && banb > 0 && gb >= g0 && gb < g1) {
            const uint32_t pat = (aval & ((1u << banb) - 1u)) << (31u - banb);
            if (pat) atomicOr(&S.tmp[rsw(gb - g0)], pat);
        }
    }
    uint32_t lm = __ballot_sync(0xffffffffu, lng);
    while (lm) {
        const uint32_t src = __ffs(lm) - 1u;
        lm &= lm - 1u;
        warp_or_bitmap(S, I, __shfl_sync(0xffffffffu, b, src), k, g0, g1, G, anb);
    }
}

// Lower bound of v in the ascending list a[0, n) by a group of 16 lanes
// (lanes [gbase, gbase+16) of a full warp; every lane of the warp calls it):
// each round the 16 lanes probe evenly spaced entries of [lo, hi) and the
// count of entries below v narrows the span 16-fold.
__device__ __forceinline__ uint32_t group16_lower_bound(const uint32_t* __restrict__ a, uint32_t n, uint32_t v,
                                                         uint32_t gbase, uint32_t gl) {
    uint32_t lo = 0, hi = n;  // the answer lies in [lo, hi]
    while (__any_sync(0xffffffffu, lo < hi)) {
        uint32_t p = lo;
        bool less = false;
        if (lo < hi) {
            p = lo + (uint32_t)(((uint64_t)(hi - lo) * gl) >> 4);  // < hi
            less = __ldg(a + p) < v;
        }
        const uint32_t c = __popc((__ballot_sync(0xffffffffu, less) >> gbase) & 0xFFFFu);
        const uint32_t plast = __shfl_sync(0xffffffffu, p, gbase + (c ? c - 1u : 0u));
        const uint32_t pnext = __shfl_sync(0xffffffffu, p, gbase + (c < 16u ? c : 0u));
        if (lo < hi) {
            if (c == 0) hi = lo;  // a[lo] >= v
            else { lo = plast + 1u; if (c < 16u) hi = pnext; }
        }
    }
    return lo;
}

// A general term over the tile [g0, g1) of RT groups, left in S.tmp (whole
// CTA; ends with a block barrier).
__device__ __forceinline__ void range_term(RangeShared& S, const RangeArgs& A, uint32_t t, uint32_t k, uint32_t g0,
                                           uint32_t g1, uint32_t G, uint32_t anb, uint32_t lastmask) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t ng = g1 - g0;
    // the term and its index, staged in shared memory by warp 0
    if (warp == 0) {
        const uint32_t v = lane < TERM_WORDS ? __ldg(reinterpret_cast<const uint32_t*>(A.terms + t) + lane) : 0u;
        const uint32_t ix = __shfl_sync(0xffffffffu, v, 0);  // DevTerm::index
        if (lane < TERM_WORDS) reinterpret_cast<uint32_t*>(&S.term)[lane] = v;
        if (lane < INDEX_WORDS)
            reinterpret_cast<uint32_t*>(&S.index)[lane] = __ldg(reinterpret_cast<const uint32_t*>(A.idx + ix) + lane);
    }
    __syncthreads();
    const DevTerm& T = S.term;
    const DevIndex& I = S.index;
    uint4* t4 = reinterpret_cast<uint4*>(S.tmp);
    if (T.c1) {
        // the wholly-inside span from two cumulative rows
        // (16-byte slices: g0 is a multiple of RT and the rows'
        // padding past the last group is zero)
        const uint4* hi = reinterpret_cast<const uint4*>(I.cum + (size_t)(T.c1 - 1u) * I.gx + g0);
        const uint4* lo = reinterpret_cast<const uint4*>(T.c0 ? I.cum + (size_t)(T.c0 - 1u) * I.gx + g0 : I.cum);
        const uint32_t n4 = (ng + 3u) >> 2;
        const bool two = T.c0 != 0u;
#pragma unroll
        for (uint32_t l = tid; l < RT / 4; l += RTHREADS) {
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (l < n4) {
                const uint4 a = __ldg(hi + l);
                const uint4 b = two ? __ldg(lo + l) : v;
                v = make_uint4(a.x & ~b.x, a.y & ~b.y, a.z & ~b.z, a.w & ~b.w);
            }
            t4[rsw4(l)] = v;
        }
    } else {
#pragma unroll
        for (uint32_t l = tid; l < RT / 4; l += RTHREADS) t4[l] = make_uint4(0u, 0u, 0u, 0u);
    }
    // the bitmaps to OR, as two ranges: with cumulative rows the
    // edge spans [h0, e0) and [e1, h1), else the span [h0, h1) or
    // the complement [0, h0) and [h1, nobs).  Ranges of at most
    // RDIRECT bitmaps in all are walked directly (one that misses
    // the tile costs its tile-index lookup); wider ones take the
    // entries of the tile's list of bitmaps holding a 1 bit in it
    // that fall in the ranges (lower bounds by 16-lane searches)
    const bool flip = T.flip != 0u;
    uint32_t ra0, ra1, rb0, rb1;  // bitmap ids [ra0, ra1) u [rb0, rb1)
    if (T.c1) { ra0 = T.h0; ra1 = T.e0; rb0 = T.e1; rb1 = T.h1; }
    else if (flip) { ra0 = 0u; ra1 = T.h0; rb0 = T.h1; rb1 = I.nobs; }
    else { ra0 = T.h0; ra1 = T.h1; rb0 = rb1 = T.h1; }
    const bool direct = !flip && (ra1 - ra0) + (rb1 - rb0) <= RDIRECT;
    if (!direct && warp < 2) {
        const uint32_t o0 = __ldg(I.tl_off + k), o1 = __ldg(I.tl_off + k + 1);
        const uint32_t gbase = lane & 16u;
        const uint32_t v = warp == 0 ? (gbase ? ra1 : ra0) : (gbase ? rb1 : rb0);
        const uint32_t r = group16_lower_bound(I.tl_bm + o0, o1 - o0, v, gbase, lane & 15u);
        if ((lane & 15u) == 0) S.hdr[2 + 2 * warp + (gbase >> 4)] = o0 + r;
    }
    __syncthreads();
    // one job list per term: the edge bitmaps' row checks first
    // (the longest jobs), then the bitmaps to OR; a complement is
    // flipped before the checked rows join it
    const uint32_t nc = flip ? 0u : T.ncand;
    uint32_t sa = ra0, sb = rb0, na = ra1 - ra0, nb = rb1 - rb0;  // the two ranges' starts and sizes
    if (!direct) {  // as entries of the tile list
        sa = S.hdr[2]; na = S.hdr[3] - sa;
        sb = S.hdr[4]; nb = S.hdr[5] - sb;
    }
    const uint32_t nsel = na + nb;
    // row checks (the longest jobs) one per warp from warp 0; the
    // bitmaps to OR in batches of up to 32 per warp (one per lane),
    // spread over the warps from the one after the checks, so the
    // warps holding a check get an OR batch last
    for (uint32_t c = warp; c < nc; c += RWARPS) warp_check_bitmap(S, I, T.cand[c], k, g0, g1, T);
    const uint32_t nfree = RWARPS - min(nc, (uint32_t)RWARPS - 1u);  // warps without a check
    const uint32_t per = min(32u, (nsel + nfree - 1) / nfree);
    const uint32_t wr = (warp + RWARPS - nc % RWARPS) % RWARPS;      // the warp's place in the OR order
    for (uint32_t j0 = wr * per; j0 < nsel; j0 += RWARPS * per) {
        const uint32_t jj = j0 + lane;
        const bool have = lane < per && jj < nsel;
        uint32_t b = 0;
        if (have) {
            const uint32_t e = jj < na ? sa + jj : sb + (jj - na);
            b = direct ? e : __ldg(I.tl_bm + e);
        }
        lanes_or_bitmaps(S, I, have, b, k, g0, g1, G, anb);
    }
    if (flip) {
        __syncthreads();
        for (uint32_t l = tid; l < ng; l += RTHREADS) {
            const uint32_t msk = (g0 + l == G && anb > 0) ? lastmask : ALLONES;
            S.tmp[rsw(l)] ^= msk;
        }
        __syncthreads();
        // edge bitmaps: rows checked against the raw values
        for (uint32_t c = warp; c < T.ncand; c += RWARPS)
            warp_check_bitmap(S, I, T.cand[c], k, g0, g1, T);
    }
    __syncthreads();
}

__device__ __forceinline__ uint4 andn4(uint4 a, uint4 b) { return make_uint4(a.x & ~b.x, a.y & ~b.y, a.z & ~b.z, a.w & ~b.w); }
__device__ __forceinline__ uint4 and4(uint4 a, uint4 b) { return make_uint4(a.x & b.x, a.y & b.y, a.z & b.z, a.w & b.w); }
__device__ __forceinline__ uint4 or4(uint4 a, uint4 b) { return make_uint4(a.x | b.x, a.y | b.y, a.z | b.z, a.w | b.w); }
__device__ __forceinline__ bool any4(uint4 a) { return (a.x | a.y | a.z | a.w) != 0u; }

// The set rows of a quad's edge bits whose raw values pass the term (groups
// g .. g + 3).  Edge bits are few and scattered (a bin of 1000 holds one row
// in 32 groups), so a lane takes one row at a time, whichever group it is in:
// the warp runs as long as its fullest lane.  (Lining the warp's rows up in
// shared memory to load 32 at once took 18 % longer.)
__device__ __forceinline__ uint4 check_quad(uint4 e, uint32_t g, const uint32_t* __restrict__ raw, const DevTerm& T) {
    uint4 r = make_uint4(0u, 0u, 0u, 0u);
    while (any4(e)) {
        const uint32_t j = e.x ? 0u : e.y ? 1u : e.z ? 2u : 3u;
        const uint32_t b = e.x ? e.x : e.y ? e.y : e.z ? e.z : e.w;
        const uint32_t hb = 31u - __clz(b), bit = 1u << hb;  // highest set bit
        const uint32_t v = __ldg(raw + (g + j) * 31u + (30u - hb));
        const uint32_t keep = pass_key(v, T) ? bit : 0u;
        if (j == 0u) { e.x ^= bit; r.x |= keep; }
        else if (j == 1u) { e.y ^= bit; r.y |= keep; }
        else if (j == 2u) { e.z ^= bit; r.z |= keep; }
        else { e.w ^= bit; r.w |= keep; }
    }
    return r;
}

// The AND of a query's dense terms over one quad per lane (quad o of the tile
// at g0), starting from acc (whole warp).
__device__ __forceinline__ uint4 dense_terms(const RangeArgs& A, const DevQuery& DQ, uint4 acc, uint32_t g0,
                                             uint32_t o) {
    const uint32_t gx4 = A.gx >> 2;
    const bool in = o < gx4 - (g0 >> 2);  // rows are the groups rounded up to 4
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t t = DQ.t0; t < DQ.td; ++t) {
        const DevTerm& T = A.terms[t];
        const uint32_t c0 = T.c0, c1 = T.c1, nc = T.ncand;
        const uint4* row = reinterpret_cast<const uint4*>(T.cum) + (g0 >> 2) + o;  // + k * gx4: C(k + 1)
        uint4 v = in && c1 ? __ldg(row + (size_t)(c1 - 1u) * gx4) : zero;
        const uint4 z = in && c0 ? __ldg(row + (size_t)(c0 - 1u) * gx4) : zero;
        if (nc) {
            // an edge bitmap j is C(j + 1) & ~C(j)
            const uint32_t j0 = T.cand[0], j1 = nc > 1u ? T.cand[1] : j0;
            uint4 e = in ? __ldg(row + (size_t)j0 * gx4) : zero;
            const uint4 e0 = in && j0 ? __ldg(row + (size_t)(j0 - 1u) * gx4) : zero;
            uint4 f = in ? __ldg(row + (size_t)j1 * gx4) : zero;
            const uint4 f0 = in && j1 ? __ldg(row + (size_t)(j1 - 1u) * gx4) : zero;
            e = and4(or4(andn4(e, e0), andn4(f, f0)), acc);  // only the rows still in the AND
            v = andn4(v, z);
            if (any4(e)) {
                const DevIndex& I = A.idx[T.index];
                v = or4(v, check_quad(e, g0 + 4u * o, reinterpret_cast<const uint32_t*>(I.values), T));
            }
        } else {
            v = andn4(v, z);
        }
        acc = and4(acc, v);
        if (!__any_sync(0xffffffffu, any4(acc))) break;
    }
    return acc;
}

// The ids of a slot (c of them, unique) in ascending order to ids off, off + 1,
// ... of the query's region, those under lim (whole warp).
__device__ __forceinline__ void copy_slot(const RangeArgs& A, uint32_t item, uint32_t c, const DevQuery& DQ, uint64_t off) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t rbase0 = A.capped ? DQ.rid_base : 0ull;
    const uint64_t room = A.rid_cap > rbase0 ? A.rid_cap - rbase0 : 0ull;
    const uint64_t lim = A.capped ? min(DQ.rid_lim, room) : room;
    const uint32_t id = lane < c ? A.slots[(size_t)item * RSLOT + lane] : 0xFFFFFFFFu;
    uint32_t rank = 0;
    for (uint32_t j = 0; j < c; ++j) rank += __shfl_sync(0xffffffffu, id, j) < id ? 1u : 0u;
    if (lane < c && off + rank < lim) A.rids[rbase0 + off + rank] = id;
}

// Q quads of groups per thread: tiles of 4 * Q * RTHREADS groups.  GEN: the
// batch holds terms that are not dense (tiles of RT groups).  Dense terms are
// bound by the rows' loads (16 KB per row and tile, shared in L2) and the
// edge rows' gathers, the others by the block barriers between their steps.
// One range over 1M rows of 100 values with its row ids: 17 us on 32 CTAs,
// 93 us when 8 CTAs walked the edge bitmaps' words; 1024 conjunctions over
// 10M rows with 256 ids each: 2.2 ms against 7.7 ms.  (Asking the next item's rows into L2 ahead
// made that 3.8: most rows of later terms are never needed.)
template <int Q, int MODE, bool GEN>
__global__ void __launch_bounds__(RTHREADS, 6) k_range(RangeArgs A) {
    static_assert(!GEN || Q == RQUADS, "the tile index is over RT groups");
    constexpr uint32_t TG = 4u * Q * RTHREADS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RangeShared& S = *reinterpret_cast<RangeShared*>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t G = A.groups, anb = A.anb;
    const uint32_t GX = G + (anb > 0 ? 1u : 0u);  // groups incl. the active one
    const uint32_t lastmask = anb > 0 ? (((1u << anb) - 1u) << (31u - anb)) : ALLONES;
    uint32_t first = blockIdx.x, epoch = 0;
    if (MODE == RM_LOOK) {
        // items in claim order: an item's predecessors are running or done
        if (tid == 0) { S.hdr[0] = claim_tile(A.sync); S.hdr[1] = ld_cg(&A.sync->epoch); }
        __syncthreads();
        first = S.hdr[0];
        epoch = S.hdr[1];
    }
    uint32_t par = 0;
    const bool listed = MODE == RM_IDS && A.capped;  // the items holding ids under their query's limit
    const uint32_t nitems = listed ? A.status->n : A.nitems;
    if (listed && A.slots) {
        const uint32_t ns = A.status->groups;
        for (uint32_t i = blockIdx.x * RWARPS + warp; i < ns; i += gridDim.x * RWARPS) {
            const uint2 li = A.item_list[A.nitems - 1u - i];
            copy_slot(A, li.x, (uint32_t)A.item_cnt[li.x], A.queries[li.x / A.ntiles], li.y);
        }
    }
    // Items are claimed one by one, the next one while this one is evaluated:
    // with items dealt out by their number the CTAs drift tiles apart, and a
    // tile's rows and words leave L2 between its queries.  1024 conjunctions
    // over 10M rows, count pass 2.14 -> 1.71 ms although each item then ends
    // at a barrier; 4096 over 50M rows 88 -> 74, 1000 binned ranges over 100M
    // rows 20.2 -> 17.7.
    const bool claim = MODE != RM_LOOK && !listed && A.sync;
    uint32_t next = 0, turn = 0;
    if (claim && tid == 0) next = claim_tile(A.sync);
    for (uint32_t at = first;; at += gridDim.x) {
        if (claim) {
            turn ^= 1u;
            if (tid == 0) {
                S.hdr[turn] = next;
                if (next < nitems) next = claim_tile(A.sync);
            }
            __syncthreads();
            at = S.hdr[turn];  // not written again before the next barrier but one
        }
        if (at >= nitems) break;
        const uint2 li = listed ? A.item_list[at] : make_uint2(at, 0u);
        const uint32_t item = li.x;
        const uint32_t q = A.tile_major && !listed ? item % A.nq : item / A.ntiles;
        const uint32_t k = A.tile_major && !listed ? item / A.nq : item % A.ntiles;
        const uint32_t g0 = k * TG, g1 = min(g0 + TG, GX);
        const uint32_t ng = g1 > g0 ? g1 - g0 : 0u;
        const uint32_t qi = q * A.ntiles + k;  // the item's place in query order
        const DevQuery DQ = A.queries[q];
        if (MODE == RM_IDS && !listed) {
            if (tid == 0 && k == 0) A.rid_start[q] = A.item_off[qi];
            const unsigned long long c = A.item_cnt[qi];
            if (c == 0ull) continue;  // no hits
            if (A.slots && c <= RSLOT) {
                if (warp == 0) copy_slot(A, qi, (uint32_t)c, DQ, A.item_off[qi]);
                continue;
            }
        }
        // the thread's quads: 32 Q consecutive ones per warp, neighbouring lanes on neighbouring quads
        const uint32_t ql = warp * (32u * Q) + lane;  // + 32 i
        uint4 acc[Q];
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            acc[i] = make_uint4(ALLONES, ALLONES, ALLONES, ALLONES);
            const uint32_t l = 4u * (ql + 32u * i);
            if (l + 4u > ng || (anb > 0 && g0 + l + 4u > G)) {  // the column's end
                uint32_t m[4];
#pragma unroll
                for (uint32_t e = 0; e < 4u; ++e) m[e] = l + e >= ng ? 0u : (g0 + l + e == G ? lastmask : ALLONES);
                acc[i] = make_uint4(m[0], m[1], m[2], m[3]);
            }
        }
        // a quad at a time through all its dense terms: few registers, so that
        // many warps' loads are in flight (all quads of a term at once on 3
        // CTAs per SM: 4.0 ms for the conjunctions that take 3.1 ms so; 4 / 5 /
        // 6 CTAs of this form, spilling a little at 6: 4.0 / 3.6 / 3.3)
        bool live = false;  // the AND is not empty
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            acc[i] = dense_terms(A, DQ, acc[i], g0, ql + 32u * i);
            live |= any4(acc[i]);
        }
        if (GEN && DQ.td < DQ.t1) {
            bool on = __syncthreads_or(live);
            for (uint32_t t = DQ.td; t < DQ.t1 && on; ++t) {
                range_term(S, A, t, k, g0, g1, G, anb, lastmask);
                bool any = false;
#pragma unroll
                for (int i = 0; i < Q; ++i) {
                    const uint4 v = reinterpret_cast<const uint4*>(S.tmp)[rsw4(ql + 32u * i)];
                    acc[i] = and4(acc[i], v);
                    any |= any4(acc[i]);
                }
                // an empty AND ends the query's work on this tile (and S.tmp is read)
                on = __syncthreads_or(any);
            }
        }
        // ---- counts and row ids
        uint32_t cnt = 0;
#pragma unroll
        for (int i = 0; i < Q; ++i) cnt += __popc(acc[i].x) + __popc(acc[i].y) + __popc(acc[i].z) + __popc(acc[i].w);
        cnt = __reduce_add_sync(0xffffffffu, cnt);  // the warp's hits
        if (MODE <= RM_ITEMS) {
            if (cnt == 0u) continue;
            uint32_t o = 0;  // the item's hits counted before these
            if (lane == 0) {
                atomicAdd(&A.counts[DQ.q], (unsigned long long)cnt);
                if (MODE == RM_ITEMS) o = (uint32_t)atomicAdd(&A.item_cnt[qi], (unsigned long long)cnt);
            }
            if (MODE == RM_ITEMS && A.slots && cnt <= RSLOT) {
                o = __shfl_sync(0xffffffffu, o, 0);
                if (o + cnt <= RSLOT) {
                    uint32_t c = 0;
#pragma unroll
                    for (int i = 0; i < Q; ++i) c += __popc(acc[i].x) + __popc(acc[i].y) + __popc(acc[i].z) + __popc(acc[i].w);
                    uint32_t s = c;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const uint32_t u = __shfl_up_sync(0xffffffffu, s, d);
                        if (lane >= (uint32_t)d) s += u;
                    }
                    uint32_t* p = A.slots + (size_t)qi * RSLOT + (o + s - c);
                    if (c) {
#pragma unroll
                        for (int i = 0; i < Q; ++i) {
                            const uint32_t row = (g0 + 4u * (ql + 32u * i)) * 31u;
                            const uint32_t v[4] = {acc[i].x, acc[i].y, acc[i].z, acc[i].w};
#pragma unroll
                            for (uint32_t e = 0; e < 4u; ++e)
                                for (uint32_t bits = v[e]; bits;) {
                                    const uint32_t hb = 31u - __clz(bits);
                                    bits ^= 1u << hb;
                                    *p++ = row + e * 31u + (30u - hb);
                                }
                        }
                    }
                }
            }
            continue;
        }
        if (lane == 0) S.sums[par][warp] = cnt;
        __syncthreads();
        uint32_t before = 0, total = 0;
#pragma unroll
        for (uint32_t w = 0; w < (uint32_t)RWARPS; ++w) {
            const uint32_t c = S.sums[par][w];
            total += c;
            before += w < warp ? c : 0u;
        }
        par ^= 1u;
        uint64_t base;
        if (MODE == RM_IDS) {
            base = listed ? li.y : A.item_off[qi];
        } else {
            if (warp == 0 && A.capped) {
                // the row ids before this tile within its own query
                const uint4 mine = make_uint4(total, 0u, 0u, k == 0 ? 1u : 0u);
                uint4 pre = make_uint4(0u, 0u, 0u, 0u);
                bool ok = true;
                if (item == 0) {
                    if (lane == 0) publish(&A.recs[0], epoch, REC_INCL, mine);
                } else {
                    if (lane == 0) publish(&A.recs[item], epoch, REC_AGG, mine);
                    pre = warp_lookback(A.recs, item, epoch, make_uint4(0u, 0u, 0u, 0u), SegSum64Comb(), &ok);
                    if (lane == 0) publish(&A.recs[item], epoch, REC_INCL, SegSum64Comb()(pre, mine));
                }
                if (lane == 0) {
                    if (!ok) atomicExch(&A.status->status, DEV_ERR_TIMEOUT);
                    S.base = k == 0 ? 0ull : ((uint64_t)pre.y << 32 | pre.x);
                    if (total) atomicAdd(&A.counts[q], (unsigned long long)total);
                    if (k == 0) A.rid_start[q] = DQ.rid_base;
                }
            } else if (warp == 0) {
                uint64_t prefix; uint32_t pa, pb;
                const bool ok = lookback64(A.recs, item, epoch, total, 0, 0, prefix, pa, pb);
                if (lane == 0) {
                    if (!ok) atomicExch(&A.status->status, DEV_ERR_TIMEOUT);
                    S.base = prefix;
                    if (total) atomicAdd(&A.counts[q], (unsigned long long)total);
                    if (k == 0) A.rid_start[q] = prefix;
                }
            }
            __syncthreads();
            base = S.base;
        }
        if (A.rids && cnt) {
            // capped: offsets are within the query; ids past its limit are
            // dropped and the rest land in its region
            const uint64_t rbase0 = A.capped ? DQ.rid_base : 0ull;
            const uint64_t room = A.rid_cap > rbase0 ? A.rid_cap - rbase0 : 0ull;
            const uint64_t lim = A.capped ? min(DQ.rid_lim, room) : room;
            // 32 groups at a time: lane l takes group 32 r + l from the lane
            // owning its quad and expands it into the warp's staging, then the
            // warp stores the run of ids, neighbouring lanes on neighbouring
            // 16 bytes of the output (single ids at its ragged ends)
            uint32_t* st = S.tmp + warp * RSTAGE;
            uint64_t off = base + before;
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                if (!__any_sync(0xffffffffu, any4(acc[i]))) continue;
#pragma unroll 1
                for (uint32_t r = 0; r < 4u && off < lim; ++r) {
                    const uint32_t src = 8u * r + (lane >> 2);
                    const uint32_t x = __shfl_sync(0xffffffffu, acc[i].x, src), y = __shfl_sync(0xffffffffu, acc[i].y, src);
                    const uint32_t z = __shfl_sync(0xffffffffu, acc[i].z, src), w = __shfl_sync(0xffffffffu, acc[i].w, src);
                    uint32_t bits = (lane & 2u ? (lane & 1u ? w : z) : (lane & 1u ? y : x)) << 1;  // row 0 at bit 31
                    const uint32_t c = __popc(bits);
                    uint32_t s = c;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const uint32_t u = __shfl_up_sync(0xffffffffu, s, d);
                        if (lane >= (uint32_t)d) s += u;
                    }
                    const uint32_t rt = __shfl_sync(0xffffffffu, s, 31);
                    const uint32_t sh = (uint32_t)(rbase0 + off) & 3u;
                    uint32_t* p = st + (sh + s - c);
                    const uint32_t row = (g0 + 4u * (warp * (32u * Q) + 32u * i + 8u * r) + lane) * 31u;
                    while (bits) {
                        const uint32_t k = __clz(bits);
                        *p++ = row + k;
                        bits &= ~(0x80000000u >> k);
                    }
                    __syncwarp();
                    const uint32_t end = sh + (uint32_t)min((uint64_t)rt, lim - off);
                    uint32_t* out = A.rids + (rbase0 + off - sh);  // 16-byte aligned
                    for (uint32_t j = 4u * lane; j < end; j += 128u) {
                        if (j >= sh && j + 4u <= end) {
                            *reinterpret_cast<uint4*>(out + j) = *reinterpret_cast<const uint4*>(st + j);
                        } else {
#pragma unroll
                            for (uint32_t e = 0; e < 4u; ++e)
                                if (j + e >= sh && j + e < end) out[j + e] = st[j + e];
                        }
                    }
                    __syncwarp();
                    off += rt;
                }
            }
        }
        if (A.dense && q == 0) {
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                const uint32_t l = 4u * (ql + 32u * i);
                const uint32_t v[4] = {acc[i].x, acc[i].y, acc[i].z, acc[i].w};
#pragma unroll
                for (uint32_t e = 0; e < 4u; ++e)
                    if (l + e < ng) A.dense[g0 + l + e] = v[e];
            }
        }
        if (MODE == RM_LOOK) break;
        // the staging is free before the next item's terms use it
        if (GEN) __syncthreads();
    }
    if (MODE == RM_LOOK || claim) {
        __syncthreads();
        if (tid == 0) finish_tile(A.sync, gridDim.x);
    }
}

// Capped queries, between the passes: a warp per query scans its items' hits
// and lists those holding ids under the limit (in any order) with the ids
// before them, so that the second pass visits no item only to skip it (0.9
// ms without the list, 0.6 with it, of 81 K items).  Items of at most RSLOT
// hits are listed apart, their ids are at hand.
__global__ void __launch_bounds__(RTHREADS) k_cap_items(RangeArgs A, uint2* __restrict__ list) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t q = (blockIdx.x * RTHREADS + threadIdx.x) >> 5;
    if (q >= A.nq) return;
    const uint64_t lim = A.queries[q].rid_lim;
    if (lane == 0) A.rid_start[q] = A.queries[q].rid_base;
    uint64_t before = 0;
    for (uint32_t k0 = 0; k0 < A.ntiles && before < lim; k0 += 32u) {
        const uint32_t k = k0 + lane;
        const uint32_t c = k < A.ntiles ? (uint32_t)A.item_cnt[(size_t)q * A.ntiles + k] : 0u;
        uint32_t s = c;  // a tile holds at most RT * 31 hits
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= (uint32_t)d) s += u;
        }
        const bool on = c != 0u && before + (s - c) < lim, kept = A.slots && c <= RSLOT;
        const uint32_t me = __ballot_sync(0xffffffffu, on && !kept), mk = __ballot_sync(0xffffffffu, on && kept);
        uint32_t ae = 0, ak = 0;
        if (lane == 0 && me) ae = atomicAdd(&A.status->n, __popc(me));
        if (lane == 0 && mk) ak = atomicAdd(&A.status->groups, __popc(mk));
        ae = __shfl_sync(0xffffffffu, ae, 0) + __popc(me & ((1u << lane) - 1u));
        ak = __shfl_sync(0xffffffffu, ak, 0) + __popc(mk & ((1u << lane) - 1u));
        if (on) list[kept ? A.nitems - 1u - ak : ae] = make_uint2(q * A.ntiles + k, (uint32_t)before + (s - c));
        before += __shfl_sync(0xffffffffu, s, 31);
    }
}

// Counts of one-term queries over disjoint bitmaps: the host has added up
// the wholly-inside bitmaps' 1 bits; what is left are the edge bins' rows that
// pass the comparison.  A warp per (edge, tile of RT groups), tile by tile so
// that the queries share a tile's raw values in L2: the bin's words of the
// tile 128 at a time, the first set row of every literal loaded before any is
// compared (few literals of an edge bin hold more).  Bound by those loads'
// latency.  1000 ranges over 10M rows, 1000 bins: 0.16 ms (0.18 ms comparing in
// double: two conversions and comparisons a row); 1.1 ms reading the spans and the edges from the cumulative rows, 1.9 ms from a row per 8
// bitmaps and the other bitmaps' words.
struct EdgeArgs {
    const DevIndex* idx;
    const DevTerm* terms;
    const uint2* edges;        // {term, bitmap}
    const uint32_t* edge_q;    // the query of each edge
    uint32_t nedges, ntiles, GX;
    unsigned long long* counts;
};
__global__ void __launch_bounds__(RTHREADS) k_edge_counts(EdgeArgs A) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nw = gridDim.x * RWARPS;
    const uint64_t items = (uint64_t)A.nedges * A.ntiles;
    for (uint64_t it = (uint64_t)blockIdx.x * RWARPS + (threadIdx.x >> 5); it < items; it += nw) {
        const uint32_t k = (uint32_t)(it / A.nedges), ei = (uint32_t)(it - (uint64_t)k * A.nedges);
        const uint32_t g0 = k * (uint32_t)RT, g1 = min(g0 + (uint32_t)RT, A.GX);
        const uint2 ed = __ldg(A.edges + ei);
        const DevTerm& T = A.terms[ed.x];
        const DevIndex& I = A.idx[T.index];
        const BitmapMeta m = I.bm[ed.y];
        const uint32_t* tix = I.tiles + ((size_t)ed.y * (I.ntiles + 1) + k) * 2;
        const uint32_t i0 = __ldg(tix), s0 = __ldg(tix + 1);
        const uint32_t in1 = __ldg(tix + 2), sn1 = __ldg(tix + 3);
        const uint32_t i1 = min(sn1 < g1 ? in1 + 1u : in1, m.n);
        const uint32_t* w = I.words + m.wstart;
        const uint32_t* raw = reinterpret_cast<const uint32_t*>(I.values);
        const KeyMap km{T.kflip, T.ksign};
        const uint32_t klo = T.klo, kspan = T.kspan;
        auto pass = [&](uint32_t v) { return value_key(v, km) - klo <= kspan ? 1u : 0u; };
        uint32_t carry = s0, cnt = 0;
        for (uint32_t base0 = i0; base0 < i1; base0 += 128) {
            uint32_t wv[4], pv[4], v0[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t i = base0 + 32u * j + lane;
                wv[j] = i < i1 ? __ldg(w + i) : 0u;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t base = base0 + 32u * j;
                pv[j] = 0;
                if (base >= i1) continue;
                const uint32_t c = base + lane < i1 ? wgroups(wv[j]) : 0u;
                uint32_t x = c;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t u = __shfl_up_sync(0xffffffffu, x, d);
                    if (lane >= (uint32_t)d) x += u;
                }
                pv[j] = carry + x - c;
                carry += __shfl_sync(0xffffffffu, x, 31);
            }
            // words past i1 are 0 and hold nothing
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool lit = wv[j] - 1u < ALLONES && pv[j] >= g0 && pv[j] < g1;
                v0[j] = lit ? __ldg(raw + pv[j] * 31u + (__clz(wv[j]) - 1u)) : 0u;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t wd = wv[j], p = pv[j];
                if (wd - 1u < ALLONES) {
                    if (p >= g0 && p < g1) {
                        cnt += pass(v0[j]);
                        for (uint32_t bits = wd & ~(0x80000000u >> __clz(wd)); bits;) {
                            const uint32_t hb = 31u - __clz(bits);
                            bits &= ~(1u << hb);
                            cnt += pass(__ldg(raw + p * 31u + (30u - hb)));
                        }
                    }
                }
            }
            // 1-fills: the rows of their groups in the tile, by the warp
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t fills = __ballot_sync(0xffffffffu, wv[j] >= HEADER1);
                while (fills) {
                    const uint32_t l = __ffs(fills) - 1u;
                    fills &= fills - 1u;
                    const uint32_t p = __shfl_sync(0xffffffffu, pv[j], l);
                    const uint32_t c = __shfl_sync(0xffffffffu, wv[j], l) & MAXCNT;
                    const uint32_t a = max(p, g0) * 31u, e = min(p + c, g1) * 31u;
                    for (uint32_t r = a + lane; r < e; r += 32u)
                        cnt += pass(__ldg(raw + r));
                }
            }
        }
        // the bitmap's active bits form the group after its whole words
        if (lane == 0 && m.anb > 0 && m.groups >= g0 && m.groups < g1)
            for (uint32_t bits = (m.aval & ((1u << m.anb) - 1u)) << (31u - m.anb); bits;) {
                const uint32_t hb = 31u - __clz(bits);
                bits &= ~(1u << hb);
                cnt += pass(__ldg(raw + m.groups * 31u + (30u - hb)));
            }
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (lane == 0 && cnt) atomicAdd(&A.counts[__ldg(A.edge_q + ei)], (unsigned long long)cnt);
    }
}

// ---- attach: the passes over a new index's words
// Every bitmap's words are cut into chunks of ICHUNK words, a warp each
// (chunks choff[b] .. choff[b+1] are bitmap b's, at least one).  With a warp
// per bitmap the few heavy bitmaps of a low-cardinality column set the time:
// 100 bitmaps over 1M rows (3000 chunks) took 1430 us for the four passes
// over the words there were, and take 51 us now (sums 6, scan 7, placement
// 19, lists 9, prefix 9).  The passes are bound by their few dependent memory
// round trips.  512 words: 16 rows of 32, four loaded per memory latency,
// and still enough warps for a few bitmaps.
constexpr uint32_t ICHUNK = 512;
constexpr uint32_t ITHREADS = 256;  // threads per CTA of the attach kernels

// Bitmap of chunk c: the last b with choff[b] <= c (whole warp).
__device__ __forceinline__ uint32_t chunk_bitmap(const uint32_t* __restrict__ choff, uint32_t nobs, uint32_t c) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo = 0, hi = nobs;  // choff[lo] <= c < choff[hi]
    while (hi - lo > 1u) {
        const uint32_t step = (hi - lo + 31u) / 32u;
        const uint32_t m = lo + lane * step;
        const uint32_t k = __popc(__ballot_sync(0xffffffffu, m < hi && __ldg(choff + m) <= c));  // >= 1: lane 0
        lo += (k - 1u) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// Groups and 1 bits of every chunk; a fill word of length 0 is a format error.
__global__ void __launch_bounds__(ITHREADS)
k_chunk_sums(const uint32_t* __restrict__ words, const BitmapMeta* __restrict__ bm, uint32_t nobs,
             const uint32_t* __restrict__ choff, uint32_t nchunks, unsigned long long* __restrict__ cgroups,
             uint32_t* __restrict__ cones, DevMeta* status) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t c = (blockIdx.x * ITHREADS + threadIdx.x) >> 5;
    if (c >= nchunks) return;
    const uint32_t b = chunk_bitmap(choff, nobs, c);
    const uint32_t* w = words + bm[b].wstart;
    const uint32_t i0 = (c - __ldg(choff + b)) * ICHUNK, i1 = min(i0 + ICHUNK, bm[b].n);
    unsigned long long groups = 0;
    uint32_t ones = 0, bad = 0;
    for (uint32_t base = i0; base < i1; base += 128) {
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t i = base + 32u * j + lane;
            v[j] = i < i1 ? __ldg(w + i) : 0u;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (base + 32u * j + lane >= i1) break;
            const uint32_t cnt = wgroups(v[j]);
            groups += cnt;
            ones += v[j] > ALLONES ? (v[j] >= HEADER1 ? cnt * 31u : 0u) : __popc(v[j]);
            bad |= cnt == 0u ? 1u : 0u;
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) groups += __shfl_xor_sync(0xffffffffu, groups, d);
    ones = __reduce_add_sync(0xffffffffu, ones);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if (lane == 0) {
        cgroups[c] = groups;
        cones[c] = ones;
        if (bad) atomicExch(&status->status, DEV_ERR_FORMAT);
    }
}

// A warp per bitmap: the first group of each of its chunks (in place of the
// chunk's group count), the bitmap's groups and 1 bits; a bitmap of more bits
// than the index has rows is a range error.
__global__ void __launch_bounds__(ITHREADS)
k_chunk_scan(BitmapMeta* __restrict__ bm, uint32_t nobs, const uint32_t* __restrict__ choff, uint32_t nrows,
             unsigned long long* __restrict__ cgroups, const uint32_t* __restrict__ cones,
             uint32_t* __restrict__ bones, DevMeta* status) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t b = (blockIdx.x * ITHREADS + threadIdx.x) >> 5;
    if (b >= nobs) return;
    const uint32_t c0 = __ldg(choff + b), c1 = __ldg(choff + b + 1);
    unsigned long long carry = 0;
    uint32_t ones = 0;
    for (uint32_t base = c0; base < c1; base += 32) {
        const uint32_t c = base + lane;
        const unsigned long long g = c < c1 ? cgroups[c] : 0ull;
        if (c < c1) ones += __ldg(cones + c);
        unsigned long long x = g;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= (uint32_t)d) x += t;
        }
        if (c < c1) cgroups[c] = carry + x - g;
        carry += __shfl_sync(0xffffffffu, x, 31);
    }
    ones = __reduce_add_sync(0xffffffffu, ones);
    if (lane == 0) {
        const uint32_t anb = bm[b].anb, aval = bm[b].aval;
        bm[b].groups = (uint32_t)carry;
        bones[b] = ones + __popc(anb ? (aval & ((1u << anb) - 1u)) : 0u);
        if (carry * 31ull + anb > nrows) atomicCAS(&status->status, 0u, DEV_ERR_RANGE);
    }
}

struct PlaceArgs {
    const uint32_t* words; const BitmapMeta* bm; uint32_t nobs;
    const uint32_t* choff; uint32_t nchunks;
    const unsigned long long* cstart;  // first group of every chunk
    uint32_t ntiles;
    uint32_t* tiles;      // per-bitmap tile index: nobs x (ntiles+1) x {word, its first group}
    uint32_t* touch;      // ntiles x tw words, bit b of row k: bitmap b holds a 1 bit in tile k (zeroed)
    uint32_t tw;
    uint32_t* cum;        // block ORs for the cumulative rows (zeroed)
    uint32_t cum_stride, gx;  // bitmap b goes into row b / cum_stride
};

// Second pass over the words, from every chunk's first group: the word
// covering each multiple of RT groups, the tiles the bitmap touches, and its
// bits OR'ed into its block's cumulative row (1-fills of more than 32 groups
// by the whole warp).
__global__ void __launch_bounds__(ITHREADS) k_chunk_place(PlaceArgs A) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t ch = (blockIdx.x * ITHREADS + threadIdx.x) >> 5;
    if (ch >= A.nchunks) return;
    const uint32_t b = chunk_bitmap(A.choff, A.nobs, ch);
    const BitmapMeta m = A.bm[b];
    const uint32_t* w = A.words + m.wstart;
    const uint32_t i0 = (ch - __ldg(A.choff + b)) * ICHUNK, i1 = min(i0 + ICHUNK, m.n);
    const bool last_chunk = ch + 1u == __ldg(A.choff + b + 1);
    uint32_t* tix = A.tiles + (size_t)b * (A.ntiles + 1) * 2;
    uint32_t* tcol = A.touch + (b >> 5);  // + tile * tw
    const uint32_t tbit = 1u << (b & 31u);
    uint32_t* row = A.cum + (size_t)(b / A.cum_stride) * A.gx;
    uint32_t carry = (uint32_t)A.cstart[ch];
    uint32_t marked = 0xFFFFFFFFu;  // the last tile this chunk marked
    for (uint32_t base0 = i0; base0 < i1; base0 += 128) {
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t i = base0 + 32u * j + lane;
            v[j] = i < i1 ? __ldg(w + i) : 0u;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t base = base0 + 32u * j;
            if (base >= i1) break;
            const uint32_t i = base + lane;
            const bool in = i < i1;
            const uint32_t wd = v[j];
            const uint32_t c = in ? wgroups(wd) : 0u;
            uint32_t p;
            if (__ballot_sync(0xffffffffu, in && is_fill(wd)) == 0u) {
                p = carry + lane;
                carry += min(32u, i1 - base);
            } else {
                uint32_t x = c;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t t = __shfl_up_sync(0xffffffffu, x, d);
                    if (lane >= (uint32_t)d) x += t;
                }
                p = carry + x - c;
                carry += __shfl_sync(0xffffffffu, x, 31);
            }
            const uint32_t k0 = p / RT, k1 = c ? (p + c - 1u) / RT : k0;
            // word i covers the boundaries t * RT in [p, p + c)
            if (c) for (uint32_t t = k0 * RT == p ? k0 : k0 + 1u; t <= k1; ++t) { tix[2 * t] = i; tix[2 * t + 1] = p; }
            const bool bits = c != 0u && (wd >= HEADER1 || (wd <= ALLONES && wd != 0u));
            // positions ascend, so a tile that the nearest lane before this
            // one with bits (or the row before) marked needs no second mark:
            // few addresses, and an atomic per word would queue on them
            const uint32_t hb = __ballot_sync(0xffffffffu, bits);
            const uint32_t below = hb & ((1u << lane) - 1u);
            const uint32_t near = __shfl_sync(0xffffffffu, k1, below ? 31u - __clz(below) : lane);
            const uint32_t before = below ? near : marked;
            if (bits)
                for (uint32_t k = k0 == before ? k0 + 1u : k0; k <= k1; ++k) atomicOr(tcol + (size_t)k * A.tw, tbit);
            if (hb) marked = __shfl_sync(0xffffffffu, k1, 31u - __clz(hb));
            if (bits && wd <= ALLONES) atomicOr(row + p, wd);
            else if (bits && c <= 32u) for (uint32_t g = 0; g < c; ++g) row[p + g] = ALLONES;
            uint32_t f = __ballot_sync(0xffffffffu, bits && wd >= HEADER1 && c > 32u);
            while (f) {
                const uint32_t src = __ffs(f) - 1u;
                f &= f - 1u;
                const uint32_t fp = __shfl_sync(0xffffffffu, p, src), fc = __shfl_sync(0xffffffffu, c, src);
                for (uint32_t g = lane; g < fc; g += 32u) row[fp + g] = ALLONES;
            }
        }
    }
    if (!last_chunk) return;
    // boundaries at or past the end of the words, and the active bits, which
    // form the group after the whole words
    for (uint32_t t = (carry + RT - 1u) / RT + lane; t <= A.ntiles; t += 32u) { tix[2 * t] = m.n; tix[2 * t + 1] = carry; }
    if (lane == 0 && m.anb > 0) {
        const uint32_t pat = (m.aval & ((1u << m.anb) - 1u)) << (31u - m.anb);
        if (pat) {
            atomicOr(tcol + (size_t)(carry / RT) * A.tw, tbit);
            atomicOr(row + carry, pat);
        }
    }
}

// Per tile the ascending list of the bitmaps holding a 1 bit in it: the set
// bits of the touch matrix in order, one pass with a decoupled look-back for
// the offsets (off[k] = the first entry of tile k, off[ntiles] = their number).
constexpr uint32_t LWPT = 4;                        // matrix words per thread
constexpr uint32_t LTILE = ITHREADS * LWPT;
__global__ void __launch_bounds__(ITHREADS)
k_tile_lists(const uint32_t* __restrict__ touch, uint32_t tw, uint32_t ntiles, uint32_t* __restrict__ off,
             uint32_t* __restrict__ list, DevMeta* status, TileRec* recs, LaunchSync* sync, uint32_t nparts) {
    __shared__ uint64_t sh[ITHREADS / 32 + 1];
    __shared__ uint32_t hdr[2];
    __shared__ uint64_t part_pre;
    if (threadIdx.x == 0) { hdr[0] = claim_tile(sync); hdr[1] = ld_cg(&sync->epoch); }
    __syncthreads();
    const uint32_t t = hdr[0], epoch = hdr[1];
    const uint32_t nw = ntiles * tw;
    const uint32_t f0 = t * LTILE + threadIdx.x * LWPT;
    uint32_t v[LWPT];
    uint32_t cnt = 0;
#pragma unroll
    for (uint32_t j = 0; j < LWPT; ++j) {
        v[j] = f0 + j < nw ? __ldg(touch + f0 + j) : 0u;
        cnt += __popc(v[j]);
    }
    uint64_t total;
    const uint64_t ex = block_exscan64(cnt, sh, total);
    if (threadIdx.x < 32) {
        uint64_t prefix; uint32_t pa, pb;
        const bool ok = lookback64(recs, t, epoch, total, 0, 0, prefix, pa, pb);
        if (threadIdx.x == 0) {
            if (!ok) atomicExch(&status->status, DEV_ERR_TIMEOUT);
            part_pre = prefix;
            if (t == nparts - 1) off[ntiles] = (uint32_t)(prefix + total);
        }
    }
    __syncthreads();
    uint32_t o = (uint32_t)(part_pre + ex);
#pragma unroll
    for (uint32_t j = 0; j < LWPT; ++j) {
        const uint32_t f = f0 + j;
        if (f >= nw) break;
        const uint32_t k = f / tw, wi = f - k * tw;
        if (wi == 0u) off[k] = o;
        for (uint32_t x = v[j]; x; x &= x - 1u) list[o++] = wi * 32u + (__ffs(x) - 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) finish_tile(sync, nparts);
}

// Prefix OR down the rows: row k |= row k-1 for k = 1..nrows-1 (a thread per
// word column; neighbouring threads read neighbouring words of each row, 16
// rows loaded before any is stored).
__global__ void k_cum_prefix(uint32_t* __restrict__ rows, uint32_t nrows, uint32_t gx) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= gx) return;
    uint32_t acc = 0;
    for (uint32_t k0 = 0; k0 < nrows; k0 += 16) {
        uint32_t v[16];
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j) v[j] = k0 + j < nrows ? rows[(size_t)(k0 + j) * gx + i] : 0u;
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j) {
            acc |= v[j];
            if (k0 + j < nrows) rows[(size_t)(k0 + j) * gx + i] = acc;
        }
    }
}

// 1 bits of one cumulative row (into *total, zeroed).
__global__ void k_row_ones(const uint32_t* __restrict__ row, uint32_t gx, unsigned long long* total) {
    uint32_t c = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < gx; i += gridDim.x * blockDim.x) c += __popc(row[i]);
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31u) == 0 && c) atomicAdd(total, (unsigned long long)c);
}

#endif  // WAH_RANGE_TYPES_ONLY

}  // namespace wah
#endif
