// Two-pass group-space engine: operators, copies and complements over 31-bit
// groups, whatever the operands' words look like, with the exact words the
// reference holds after compress().
//
// Canonical results (the reference's _d2 / _d1 / _c1 / _c0 paths and the
// all-literal loops, src/bitvector.cpp:2545-2830, 2981-3278, 3354-3619,
// 3748-4079): one word per maximal run of equal all-0 / all-1 groups (a fill
// when the run holds two or more groups) and one literal per mixed group.
// The _c2 walks (src/bitvector.cpp:2419-3745) differ from that only in runs
// of one group, which may be count-1 fills; single_flag (wah_core.cuh) tells
// those from the words meeting there, and copies keep the operand's.
//
// Every operand has a row index: for each 32 groups a mask of the groups
// where a word starts and the word covering the group before them, so the
// word of group 32 k + l is base + popc(mask & bits 0..l): no decode, no scan.
// It is built once per bitvector (k_rows) and comes with every result of
// this engine, whose head masks it is.
//
// Two launches, no look-back and no waits between CTAs, a warp per tile of
// PT = 512 groups, every CTA a contiguous range of tiles:
//  * k_gop: lane l of row r owns group 32 r + l.  The tile's words of both
//    operands arrive in shared memory by bulk copies, issued one tile ahead
//    (two buffers per warp, an mbarrier each); R = a OP b is stored densely,
//    and a row's run heads come from two ballots (groups all 0, groups all 1)
//    and a shift.  Per tile: heads, first head, 1 bits.
//  * k_gpack: a tile's R arrives the same way; each head's lane writes its
//    word at the number of heads before it: the literal, or the run word
//    whose length reaches the next head.
// Bound by instruction issue (60-62 % of the slots, the integer pipe 57-61 %
// busy) and the few warps that two buffers per warp leave room for.  At 2^28
// bits, both operands of d = 0.1 / 0.5: 39 / 40 us a call against 79 / 65 for the
// form before it (a word-start marker per word and warp max-scans over 128
// groups, operands staged without prefetch, four neighbouring groups per lane;
// ~2370 + 1060 instructions per tile against 720 + 775).  Tiles of 256 groups
// double the resident warps and are slower (46 / 50 us: the per-tile work), and
// so is packing a tile's words in k_gop with k_gpack a copy (45 / 48);
// launching each kernel while the one before it drains saves 3 us a call.
#ifndef WAH_GOP_CUH
#define WAH_GOP_CUH
#include <type_traits>
#include "wah_dense.cuh"

namespace wah {

constexpr int PT = 512;                   // groups per tile of this engine, a warp's
constexpr int TROWS = PT / 32;            // rows of 32 groups per tile
constexpr int GW = 8;                     // warps per CTA of this engine
constexpr int GBUF = PT + 8;              // staged words of a tile: its own, the ones either side, 16-byte ends
constexpr int GCTA = GW * 32;
constexpr uint32_t GNONE = 0xFFFFFFFFu;   // no head
static_assert(TROWS == 16, "a half warp holds a tile's rows");

enum GopKind : int {
    GK_CANON = 0,  // x OP y, canonical words
    GK_FSM = 1,    // x OP y, the words of the reference's _c2 walk
    GK_COPY = 2,   // x, as compress() leaves it
    GK_FLIP = 3    // x complemented
};

struct GopArgs {
    const uint32_t* xw; const uint2* xr; const uint32_t* xbp; uint32_t nx;  // words, row index, block positions, words
    const uint32_t* yw; const uint2* yr; const uint32_t* ybp; uint32_t ny;
    uint32_t groups, ntiles;
    uint32_t* R;          // ntiles * PT result patterns; bit 31: as a run of one group it is a count-1 fill
    // per tile: heads (GNONE: the tile gave up), first head (GNONE: none), 1 bits
    uint32_t* heads; uint32_t* first; uint32_t* ones;
    uint32_t* wfirst;     // first head of each warp of k_gop (GNONE: none)
    uint32_t gop_ctas;    // CTAs of k_gop
    uint32_t* out; uint32_t* obp; uint2* orow; DevMeta* meta;
    uint32_t aval, anb;
    uint32_t withhold;    // test hook: this tile's wait counts as given up (UINT32_MAX: none)
};

// The word covering group g < groups and its first group (whole warp): a
// 32-way search of the block positions (bp[0] = 0, ascending), then a scan of
// the block's words.
__device__ __forceinline__ void word_of_group(const uint32_t* __restrict__ w, const uint32_t* __restrict__ bp, uint32_t n,
                                              uint32_t g, uint32_t& wi, uint32_t& start) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo = 0, hi = (n + 31u) / 32u;  // bp[lo] <= g < bp[hi]
    while (hi - lo > 1u) {
        const uint32_t step = (hi - lo + 31u) / 32u, m = lo + lane * step;
        const uint32_t k = __popc(__ballot_sync(0xffffffffu, m < hi && __ldg(bp + m) <= g));  // >= 1: lane 0
        lo += (k - 1u) * step;
        hi = min(hi, lo + step);
    }
    const uint32_t i = 32u * lo + lane;
    const uint32_t c = i < n ? wgroups(__ldg(w + i)) : 0u;
    uint32_t x = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= (uint32_t)d) x += u;
    }
    const uint32_t p = __ldg(bp + lo) + x - c;  // first group of the lane's word
    const uint32_t in = __popc(__ballot_sync(0xffffffffu, i < n && p <= g));  // >= 1: lane 0
    wi = 32u * lo + in - 1u;
    start = __shfl_sync(0xffffffffu, p, in - 1u);
}

// The row index of a bitvector (ntiles * TROWS rows; rows past the last
// group hold no start and the last word): a warp per tile finds the tile's
// first word, takes its words 32 at a time, flags the group each one starts
// at in shared memory (positions by a warp scan where a row holds a fill)
// and ballots the flags.  Bound by latency (the search's round trips); a
// launch of its own for the search (a binary search per thread) took 13 us
// at 2^28 bits beside 10 us for the rows.
__global__ void __launch_bounds__(GCTA) k_rows(const uint32_t* __restrict__ w, const uint32_t* __restrict__ bp,
                                               uint32_t n, uint32_t groups, uint32_t ntiles, uint2* __restrict__ rows) {
    __shared__ __align__(16) uint8_t mk_[GW][PT];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t t = blockIdx.x * GW + warp;
    if (t >= ntiles) return;
    uint8_t* mk = mk_[warp];
    const uint32_t g0 = t * (uint32_t)PT, g1 = min(g0 + (uint32_t)PT, groups);
    uint32_t wi0, s0;
    word_of_group(w, bp, n, g0, wi0, s0);
    reinterpret_cast<uint4*>(mk)[lane] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    uint32_t carry = s0;  // first group of the next word
    for (uint32_t base0 = wi0; base0 < n && carry < g1; base0 += 128) {
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t k = base0 + 32u * j + lane;
            v[j] = k < n ? __ldg(w + k) : 0u;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t base = base0 + 32u * j;
            if (base >= n || carry >= g1) break;
            const bool in = base + lane < n;
            uint32_t p;
            if (__ballot_sync(0xffffffffu, in && is_fill(v[j])) == 0u) {
                p = carry + lane;
                carry += min(32u, n - base);
            } else {
                const uint32_t c = in ? wgroups(v[j]) : 0u;
                uint32_t x = c;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t u = __shfl_up_sync(0xffffffffu, x, d);
                    if (lane >= (uint32_t)d) x += u;
                }
                p = carry + x - c;
                carry += __shfl_sync(0xffffffffu, x, 31);
            }
            if (in && p >= g0 && p < g1) mk[p - g0] = 1u;
        }
    }
    __syncwarp();
    uint32_t m = 0;
#pragma unroll
    for (int r = 0; r < TROWS; ++r) {
        const uint32_t b = __ballot_sync(0xffffffffu, mk[32 * r + lane] != 0u);
        if (lane == (uint32_t)r) m = b;
    }
    // words before each row: those before the tile, then the rows' starts
    uint32_t x = __popc(m);
#pragma unroll
    for (int d = 1; d < TROWS; d <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= (uint32_t)d) x += u;
    }
    const uint32_t w0 = s0 == g0 ? wi0 : wi0 + 1u;  // the first word starting in the tile
    if (lane < (uint32_t)TROWS) rows[(size_t)t * TROWS + lane] = make_uint2(m, w0 + x - __popc(m) - 1u);
}

// decompress(): every group of a bitvector as a literal word, with the
// result's block positions, row index (when orow is given) and metadata, all
// of which are known beforehand.  A warp per tile; bound by the stores.  (A
// thread per 16 words with the fills listed and written one after the other
// by the CTA took 244 us at 2^27 bits, d = 0.05, and the metadata another 23;
// this takes 12 and k_rows, where the index is not there yet, 12.)
__global__ void __launch_bounds__(GCTA) k_expand(const uint32_t* __restrict__ w, const uint2* __restrict__ rows,
                                                 uint32_t ntiles, uint32_t* __restrict__ out, uint32_t* __restrict__ obp,
                                                 uint2* __restrict__ orow, DevMeta* meta, DevMeta m) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t t = blockIdx.x * GW + (threadIdx.x >> 5);
    const uint32_t le = (2u << lane) - 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0) { *meta = m; obp[(m.groups + 31u) / 32u] = m.groups; }
    if (t >= ntiles) return;
    const uint32_t g0 = t * (uint32_t)PT;
    const uint2* xr = rows + (size_t)t * TROWS;
#pragma unroll
    for (int r0 = 0; r0 < TROWS; r0 += 8) {
        uint32_t v[8];
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(xr + r0 + j));
            v[j] = __ldg(w + (q.y + __popc(q.x & le)));
            v[j + 1] = __ldg(w + (q.w + __popc(q.z & le)));
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t g = g0 + 32u * (r0 + j) + lane;
            if (g < m.groups) out[g] = wpattern(v[j]);
        }
    }
    if (lane < (uint32_t)TROWS) {
        const uint32_t g = g0 + 32u * lane;
        const uint32_t k = m.groups > g ? m.groups - g : 0u;  // groups from the row on
        if (k) obp[g >> 5] = g;
        if (orow) orow[(size_t)t * TROWS + lane] = make_uint2(k >= 32u ? 0xFFFFFFFFu : (1u << k) - 1u, min(g, m.groups) - 1u);
    }
}

// Pattern of one group of word w in bits 0..30 (bit 31 is not part of it).
__device__ __forceinline__ uint32_t gop_pattern(uint32_t w) {
    return (int32_t)w < 0 ? (uint32_t)((int32_t)(w << 1) >> 31) : w;
}
// Result pattern of one group from its words (bit 31: a fill word of x, for
// the kinds that keep count-1 fills).
template <int OP, int KIND>
__device__ __forceinline__ uint32_t gop_value(uint32_t x, uint32_t y) {
    if (KIND == GK_COPY) return (gop_pattern(x) & ALLONES) | (x & HEADER0);
    if (KIND == GK_FLIP) return (~gop_pattern(x) & ALLONES) | (x & HEADER0);
    return op2<OP>(gop_pattern(x), gop_pattern(y)) & ALLONES;
}

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// Tiles of CTA `cta` of `n`: [lo, hi).
__device__ __forceinline__ void gop_range_of(uint32_t ntiles, uint32_t cta, uint32_t n, uint32_t& lo, uint32_t& hi) {
    const uint32_t q = (ntiles + n - 1u) / n;
    lo = min(cta * q, ntiles);
    hi = min(lo + q, ntiles);
}

// Position of the k-th set bit (from 0) of h.
__device__ __forceinline__ uint32_t nth_bit(uint32_t h, uint32_t k) {
    uint32_t pos = 0;
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
        const uint32_t c = __popc((h >> pos) & ((1u << w) - 1u));
        if (k >= c) { k -= c; pos += w; }
    }
    return pos;
}

template <bool UNARY>
struct GopWarp {
    uint32_t w[UNARY ? 1 : 2][2][GBUF];  // operand, buffer
    uint2 row[2][32];                    // per buffer: lanes 0-15 x's rows, 16-31 y's: mask, shared address of the word before
    uint2 hu[TROWS];                     // heads and uniform groups of each row
    uint64_t bar[2];
};

// A warp of k_gop marks tile t and its later ones as given up.
__device__ __noinline__ void give_up(uint32_t* heads, uint32_t t, uint32_t tend) {
    for (; t < tend; t += GW) heads[t] = GNONE;
}

template <int OP, int KIND>
__global__ void __launch_bounds__(GCTA, 3) k_gop(const __grid_constant__ GopArgs A) {
    constexpr bool UNARY = KIND >= GK_COPY;
    extern __shared__ __align__(16) unsigned char gsm[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    GopWarp<UNARY>& W = reinterpret_cast<GopWarp<UNARY>*>(gsm)[warp];
    if (lane == 0) { mbar_init(&W.bar[0], 1); mbar_init(&W.bar[1], 1); mbar_init_fence(); }
    uint32_t t, tend;
    gop_range_of(A.ntiles, blockIdx.x, gridDim.x, t, tend);
    t += warp;
    __syncwarp();
    pdl_wait();
    pdl_launch();
    if (blockIdx.x == 0 && threadIdx.x == 0) { A.meta->nfill = 0; A.meta->status = 0; }
    if (t >= tend) {
        if (lane == 0) A.wfirst[blockIdx.x * GW + warp] = GNONE;
        return;
    }
    uint32_t head0 = GNONE;  // the warp's first head
    const uint32_t le = (2u << lane) - 1u;  // lanes up to this one (lane 31: all)
    const uint32_t* __restrict__ xw = A.xw;
    const uint32_t* __restrict__ yw = A.yw;

    // rows of tile u, one per lane
    auto load_rows = [&](uint32_t u) {
        const uint2* p = lane < 16u || UNARY ? A.xr : A.yr;
        return __ldg(p + (size_t)u * TROWS + (lane & 15u));
    };
    // issues the copies of a tile's words: from the one covering the group
    // before it to the one after its last, 16-byte ends rounded outwards (the
    // word arrays are pool blocks: aligned and padded to 256 bytes)
    auto stage = [&](uint2 row, uint32_t b) {
        const uint32_t half = lane & 16u, n = half ? A.ny : A.nx;
        const uint32_t fst = __shfl_sync(0xffffffffu, row.y, half);
        const uint32_t lst = __shfl_sync(0xffffffffu, row.y + __popc(row.x), half + TROWS - 1u);
        const uint32_t lo = (fst == GNONE ? 0u : fst) & ~3u, hi = min(lst + 2u, n);
        const uint32_t bytes = ((hi - lo + 3u) & ~3u) * 4u;
        uint32_t* buf = W.w[UNARY ? 0 : half >> 4][b];
        row.y = smem_u32(buf) + (row.y - lo) * 4u;
        W.row[b][lane] = row;
        __syncwarp();
        const uint32_t both = bytes + (UNARY ? 0u : __shfl_xor_sync(0xffffffffu, bytes, 16));
        if (lane == 0) mbar_arrive_tx(&W.bar[b], both);
        __syncwarp();
        if ((lane & 15u) == 0u && (lane == 0u || !UNARY)) bulk_g2s(buf, (half ? yw : xw) + lo, bytes, &W.bar[b]);
    };

    uint2 nrow = load_rows(t);
    stage(nrow, 0);
    if (t + GW < tend) nrow = load_rows(t + GW);
    for (uint32_t k = 0; t < tend; t += GW, ++k) {
        const uint32_t b = k & 1u;
        if (t + GW < tend) {
            stage(nrow, b ^ 1u);
            if (t + 2 * GW < tend) nrow = load_rows(t + 2 * GW);
        }
        if (!__all_sync(0xffffffffu, mbar_wait(&W.bar[b], (k >> 1) & 1u)) || t == A.withhold) {
            // gave up: this tile and the warp's others say so, for k_gpack to
            // write nothing by their counts; leave once the copies in flight
            // are done or have been waited for as long again
            if (lane == 0) give_up(A.heads, t, tend);
            if (t + GW < tend) mbar_wait(&W.bar[b ^ 1u], ((k + 1u) >> 1) & 1u);
            return;
        }
        const uint32_t g0 = t * (uint32_t)PT;
        const uint32_t left = A.groups - g0;  // valid groups from g0 on
        const uint4* rows = reinterpret_cast<const uint4*>(W.row[b]);
        uint32_t* R = A.R + g0 + lane;
        uint32_t ones = 0;
        // bit 31: was the group before all 0 / all 1
        uint32_t zp = 0, op = 0;
        if (g0) {
            const uint32_t pv = gop_value<OP, KIND>(lds32(W.row[b][0].y), UNARY ? 0u : lds32(W.row[b][16].y)) & ALLONES;
            zp = pv == 0u ? 0x80000000u : 0u;
            op = pv == ALLONES ? 0x80000000u : 0u;
        }
        // FULL: every group of the tile is valid
        auto rows_of = [&](auto full_tile) {
            constexpr bool FULL = decltype(full_tile)::value;
#pragma unroll 2
            for (int r0 = 0; r0 < TROWS; r0 += 4) {
                uint32_t xv[4], yv[4];
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    const uint4 m = rows[(r0 + j) / 2];
                    xv[j] = lds32(m.y + 4u * __popc(m.x & le));
                    xv[j + 1] = lds32(m.w + 4u * __popc(m.z & le));
                    if (!UNARY) {
                        const uint4 q = rows[(TROWS + r0 + j) / 2];
                        yv[j] = lds32(q.y + 4u * __popc(q.x & le));
                        yv[j + 1] = lds32(q.w + 4u * __popc(q.z & le));
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t r = r0 + j;
                    uint32_t v = gop_value<OP, KIND>(xv[j], UNARY ? 0u : yv[j]);
                    R[32u * r] = v;
                    if (UNARY) v &= ALLONES;
                    uint32_t vm = 0xFFFFFFFFu;
                    if (!FULL) {
                        const uint32_t c = left > 32u * r ? left - 32u * r : 0u;
                        vm = c >= 32u ? 0xFFFFFFFFu : (1u << c) - 1u;
                        if (!((vm >> lane) & 1u)) v = 0u;
                    }
                    const uint32_t z = __ballot_sync(0xffffffffu, v == 0u), o = __ballot_sync(0xffffffffu, v == ALLONES);
                    // a head: mixed, or of another class than the group before
                    const uint32_t h = ~((z & __funnelshift_l(zp, z, 1)) | (o & __funnelshift_l(op, o, 1))) & vm;
                    zp = z;
                    op = o;
                    ones += __popc(v);
                    if (lane == 0) W.hu[r] = make_uint2(h, z | o);
                }
            }
        };
        if (left >= (uint32_t)PT) rows_of(std::true_type());
        else rows_of(std::false_type());
        __syncwarp();
        uint32_t H = 0, U = 0, heads = 0, first = GNONE;
        if (lane < (uint32_t)TROWS) {
            const uint2 hu = W.hu[lane];
            H = hu.x; U = hu.y;
            A.orow[(size_t)t * TROWS + lane] = hu;  // k_gpack puts the words before the row in U's place
            heads = __popc(H);
            if (H) first = g0 + 32u * lane + (__ffs(H) - 1u);
        }
        if (KIND == GK_FSM) {
            // runs of one group: a uniform head followed by a head (or the end)
            uint32_t nb = __shfl_down_sync(0xffffffffu, H, 1) & 1u;
            uint32_t xnext = 0, ynext = 0;  // starts of the row after the tile
            if (left > (uint32_t)PT) {  // the head test of the group after the tile
                const uint2* xr = A.xr + (size_t)(t + 1) * TROWS;
                const uint2* yr = A.yr + (size_t)(t + 1) * TROWS;
                const uint2 mx = __ldg(xr), my = __ldg(yr);
                xnext = mx.x; ynext = my.x;
                const uint32_t pv = gop_value<OP, KIND>(__ldg(xw + (mx.y + (mx.x & 1u))), __ldg(yw + (my.y + (my.x & 1u))));
                if (lane == TROWS - 1u) nb = !((pv == 0u && zp >> 31) || (pv == ALLONES && op >> 31));
            } else if (left == 32u * lane + 32u) {
                nb = 1u;
            }
            uint32_t S = H >> 1 | nb << 31;
            if (left > 32u * lane && left < 32u * lane + 32u) S |= 1u << (left - 32u * lane - 1u);
            S &= H & U;
            if (lane >= (uint32_t)TROWS) S = 0u;
            // the tile's one-group runs, 32 at a time whatever rows they are in
            const uint32_t ns = __popc(S);
            uint32_t before = ns;  // lane r: those before row r
#pragma unroll
            for (int d = 1; d < TROWS; d <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, before, d);
                if (lane >= (uint32_t)d) before += u;
            }
            const uint32_t nsingle = __shfl_sync(0xffffffffu, before, TROWS - 1);
            before -= ns;
            for (uint32_t k0 = 0; k0 < nsingle; k0 += 32u) {
                const uint32_t k = min(k0 + lane, nsingle - 1u);
                uint32_t r = 0;  // the last row with at most k before it
#pragma unroll
                for (uint32_t d = TROWS / 2; d > 0; d >>= 1)
                    if (__shfl_sync(0xffffffffu, before, r + d) <= k) r += d;
                const uint32_t bit = nth_bit(__shfl_sync(0xffffffffu, S, r), k - __shfl_sync(0xffffffffu, before, r));
                const uint32_t p = g0 + 32u * r + bit;
                // its words, as staged
                const uint2 mx = W.row[b][r], my = W.row[b][TROWS + r];
                const uint32_t upto = (2u << bit) - 1u;
                const uint32_t x = lds32(mx.y + 4u * __popc(mx.x & upto)), y = lds32(my.y + 4u * __popc(my.x & upto));
                // do they end at p + 1 (does the next one start there)
                bool xe = true, ye = true;
                if (p + 1u < A.groups) {
                    const uint32_t nbit = (bit + 1u) & 31u, nr = r + (bit == 31u ? 1u : 0u);
                    xe = ((nr < (uint32_t)TROWS ? W.row[b][nr].x : xnext) >> nbit) & 1u;
                    ye = ((nr < (uint32_t)TROWS ? W.row[b][TROWS + nr].x : ynext) >> nbit) & 1u;
                }
                uint32_t code = k0 + lane < nsingle
                                    ? single_flag(OP, x, y, (mx.x >> bit) & 1u, (my.x >> bit) & 1u, xe, ye) : SF_NO;
                uint32_t walk = __ballot_sync(0xffffffffu, code > SF_YES);
                while (walk) {
                    const uint32_t l = __ffs(walk) - 1u;
                    walk &= walk - 1u;
                    const uint32_t wp = __shfl_sync(0xffffffffu, p, l), wm = (2u << (wp & 31u)) - 1u;
                    const uint2 rx = __ldg(A.xr + (wp >> 5)), ry = __ldg(A.yr + (wp >> 5));
                    const bool f = walk_flag<OP>(Operands{A.xw, A.xbp, A.yw, A.ybp}, __shfl_sync(0xffffffffu, code, l), wp,
                                                 rx.y + __popc(rx.x & wm), ry.y + __popc(ry.x & wm));
                    if (lane == l) code = f ? SF_YES : SF_NO;
                }
                // over the pattern another lane stored (the warp has synchronised since)
                if (code == SF_YES) A.R[p] = gop_value<OP, KIND>(x, y) | HEADER0;
            }
        }
        ones = __reduce_add_sync(0xffffffffu, ones);
        heads = __reduce_add_sync(0xffffffffu, heads);
        first = __reduce_min_sync(0xffffffffu, first);
        if (lane == 0) { A.heads[t] = heads; A.first[t] = first; A.ones[t] = ones; }
        head0 = min(head0, first);
        __syncwarp();  // the buffer, the rows and the head masks are free again
    }
    if (lane == 0) A.wfirst[blockIdx.x * GW + warp] = head0;
}

// The first head of the tiles from i on (whole warp): of the rest of tile
// i - 1's k_gop CTA, else of the CTAs after it by their warps' first heads, 256
// at a time.  (By the tiles alone a result of one run read them all: 2^28 bits,
// 323 us a call with every tile looking, heads or not, 31 so.)
__device__ __noinline__ uint32_t head_from(const uint32_t* __restrict__ first, const uint32_t* __restrict__ wfirst,
                                           uint32_t ntiles, uint32_t gop_ctas, uint32_t i) {
    const uint32_t lane = threadIdx.x & 31u;
    if (i >= ntiles) return GNONE;
    uint32_t lo, hi, h = GNONE;
    const uint32_t cta = (i - 1u) / ((ntiles + gop_ctas - 1u) / gop_ctas);
    gop_range_of(ntiles, cta, gop_ctas, lo, hi);
    for (; h == GNONE && i < hi; i += 32u) h = __reduce_min_sync(0xffffffffu, i + lane < hi ? first[i + lane] : GNONE);
    const uint32_t nw = gop_ctas * GW;
    for (uint32_t s = (cta + 1u) * GW; h == GNONE && s < nw; s += 256u) {
        uint32_t v = GNONE;
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j)
            if (s + 32u * j + lane < nw) v = min(v, wfirst[s + 32u * j + lane]);
        h = __reduce_min_sync(0xffffffffu, v);
    }
    return h;
}

struct PackWarp {
    uint32_t r[2][PT];  // result patterns
    uint2 hu[2][TROWS];
    uint4 row[TROWS];   // heads; index of the row's first head; groups from the row's end to the head after it; heads of runs
    uint64_t bar[2];
};
constexpr uint32_t GRANGE = 1024;  // tiles of a CTA at most

// The words of one tile per warp.  The last CTA writes the metadata.
__global__ void __launch_bounds__(GCTA) k_gpack(const __grid_constant__ GopArgs A) {
    extern __shared__ __align__(16) unsigned char gsm[];
    __shared__ uint32_t sh[2][GW];
    __shared__ uint32_t pre[GRANGE + 1];  // heads before each tile of the range, from its start, and in all of it
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    PackWarp& W = reinterpret_cast<PackWarp*>(gsm)[warp];
    uint32_t tb, tend;
    gop_range_of(A.ntiles, blockIdx.x, gridDim.x, tb, tend);
    if (lane == 0) { mbar_init(&W.bar[0], 1); mbar_init(&W.bar[1], 1); mbar_init_fence(); }
    __syncwarp();
    pdl_wait();
    pdl_launch();
    if (tb >= tend) return;
    auto stage = [&](uint32_t u, uint32_t b) {
        if (lane == 0) {
            mbar_arrive_tx(&W.bar[b], sizeof W.r[0] + sizeof W.hu[0]);
            bulk_g2s(W.r[b], A.R + (size_t)u * PT, sizeof W.r[0], &W.bar[b]);
            bulk_g2s(W.hu[b], A.orow + (size_t)u * TROWS, sizeof W.hu[0], &W.bar[b]);
        }
    };
    uint32_t t = tb + warp;
    if (t < tend) stage(t, 0);
    // heads before the range; the last CTA also sums the 1 bits
    const bool last = tend == A.ntiles;
    uint32_t part = 0, ones = 0;
    uint32_t gone = 0;  // GNONE among the counts: a tile up to the range's end gave up
    for (uint32_t i = threadIdx.x; i < tb; i += GCTA) {
        const uint32_t c = A.heads[i];
        gone |= c;
        part += c;
    }
    if (last) for (uint32_t i = threadIdx.x; i < A.ntiles; i += GCTA) ones += A.ones[i];
    part = __reduce_add_sync(0xffffffffu, part);
    ones = __reduce_add_sync(0xffffffffu, ones);
    if (lane == 0) { sh[0][warp] = part; sh[1][warp] = ones; }
    if (warp == 0) {  // scan of the range's tiles
        uint32_t carry = 0;
        for (uint32_t i = tb; i < tend; i += 32u) {
            const uint32_t c = i + lane < tend ? A.heads[i + lane] : 0u;
            gone |= c;
            uint32_t x = c;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= (uint32_t)d) x += u;
            }
            if (i + lane < tend) pre[i + lane - tb] = carry + x - c;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) pre[tend - tb] = carry;
        part = carry;  // warp 0: the range's heads
    }
    if (__syncthreads_or(gone >> 31)) {
        // no word has a place; the last CTA, which has seen every tile, says so
        if (last && threadIdx.x == 0) {
            A.meta->n = A.meta->groups = A.meta->nset = A.meta->anb = A.meta->aval = A.meta->w0 = 0;
            atomicExch(&A.meta->status, DEV_ERR_TIMEOUT);
        }
        if (t < tend) mbar_wait(&W.bar[0], 0);
        return;
    }
    uint32_t base = 0;
#pragma unroll
    for (uint32_t k = 0; k < (uint32_t)GW; ++k) base += sh[0][k];
    if (last && threadIdx.x == 0) {
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t k = 0; k < (uint32_t)GW; ++k) sum += sh[1][k];
        const uint32_t n = base + part;
        A.obp[(n + 31u) / 32u] = A.groups;
        A.meta->n = n;
        A.meta->groups = A.groups;
        A.meta->nset = sum;
        A.meta->anb = A.anb;
        A.meta->aval = A.aval;
    }
    const uint32_t bit = 1u << lane, lt = bit - 1u, gt = ~(lt | bit);
    uint32_t any = 0;  // the words written, OR'ed
    for (uint32_t k = 0; t < tend; t += GW, ++k) {
        const uint32_t b = k & 1u;
        if (t + GW < tend) stage(t + GW, b ^ 1u);
        // the first head after the tile: nearly always of the 32 tiles after it
        uint32_t later;
        {
            const uint32_t i = t + 1u + lane;
            later = __reduce_min_sync(0xffffffffu, i < A.ntiles ? A.first[i] : (i == A.ntiles ? A.groups : GNONE));
        }
        const uint32_t before = pre[t - tb];
        if (later == GNONE && pre[t - tb + 1u] != before)
            later = min(head_from(A.first, A.wfirst, A.ntiles, A.gop_ctas, t + 33u), A.groups);
        if (!__all_sync(0xffffffffu, mbar_wait(&W.bar[b], (k >> 1) & 1u))) {
            if (lane == 0) atomicExch(&A.meta->status, DEV_ERR_TIMEOUT);
            if (t + GW < tend) mbar_wait(&W.bar[b ^ 1u], ((k + 1u) >> 1) & 1u);
            return;
        }
        const uint32_t g0 = t * (uint32_t)PT;
        const uint2 hu = lane < (uint32_t)TROWS ? W.hu[b][lane] : make_uint2(0u, 0u);
        const uint32_t H = hu.x, c = __popc(H);
        uint32_t x = c;
#pragma unroll
        for (int d = 1; d < TROWS; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= (uint32_t)d) x += u;
        }
        x += base + before - c;  // lane r: index of row r's first head
        const uint32_t fh = H ? g0 + 32u * lane + (__ffs(H) - 1u) : GNONE;
        uint32_t nx = __shfl_down_sync(0xffffffffu, fh, 1);
        if (lane >= TROWS - 1u) nx = later;
#pragma unroll
        for (int d = 1; d < TROWS; d <<= 1) nx = min(nx, __shfl_down_sync(0xffffffffu, nx, d));
        if (lane < (uint32_t)TROWS) {
            W.row[lane] = make_uint4(H, x, nx - (g0 + 32u * lane + 32u), hu.y & H);
            A.orow[(size_t)t * TROWS + lane].y = x - 1u;
            // block positions: a row holds at most one head of index 32 j
            const uint32_t m = (x + 31u) & ~31u;
            if (m < x + c) A.obp[m >> 5] = g0 + 32u * lane + nth_bit(H, m - x);
        }
        __syncwarp();
        const uint32_t* rl = W.r[b] + lane;
#pragma unroll 1
        for (int r0 = 0; r0 < TROWS; r0 += 4) {
            uint4 q[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) q[j] = W.row[r0 + j];
            if ((q[0].x | q[1].x | q[2].x | q[3].x) == 0u) continue;  // inside a run
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t rv = rl[32 * (r0 + j)];
                uint32_t wd = rv & ALLONES;
                if (q[j].w) {  // heads of runs among them
                    const uint32_t above = q[j].x & gt;  // the row's heads after this lane
                    // groups to the next head: in the row (its lowest bit
                    // above this lane), else past the row's end
                    const uint32_t low = 31u - __clz(above & (0u - above));  // -1: none
                    uint32_t len = low - lane;
                    if (above == 0u) len = q[j].z + (32u - lane);
                    const bool f = (q[j].w & bit) && (len >= 2u || rv >= HEADER0);
                    if (f) wd = (rv & FILLBIT) | len | HEADER0;
                }
                if (q[j].x & bit) {
                    A.out[q[j].y + __popc(q[j].x & lt)] = wd;
                    any |= wd;
                }
            }
        }
        if (t == 0 && lane == 0) A.meta->w0 = A.out[0];  // this lane's own store: group 0 is a head
        // R is read once: its lines need not be written back to memory when
        // operands, R and words outgrow L2 (2^28 bits of d = 0.5: 44 -> 40 us)
        if (lane < PT / 32u) asm volatile("discard.global.L2 [%0], 128;" ::"l"(A.R + g0 + 32u * lane) : "memory");
        __syncwarp();  // the rows and the buffer are free again
    }
    if (__any_sync(0xffffffffu, any >= HEADER0) && lane == 0) A.meta->nfill = 1u;
}

}  // namespace wah
#endif
