// Cell-tile exact kNN: the queries of one grid cell are searched together,
// one query per lane, over the cell's 3x3x3 block of candidates, which is
// staged 16 at a time in shared memory.
//
// The reference's ring search (GridKNNCuda.cu:647-743, driven level by level
// from :2322-2634) visits, for a query of level-L cell C, the points of the
// 3x3x3 block of level-L cells around C -- the same block for every query of
// C.  k_knn_plain runs one query per warp and spends ~16 warp instructions
// per candidate locating, loading and merging it.  Here each half of a warp
// takes a cell (a unit) and up to 16 of its queries, one per lane; every
// candidate of the block is loaded once per half-warp and compared by all
// of its lanes at once:
//
//   pass 1  each lane buckets its candidate distances (64 buckets, 8 per
//           octave of d^2, placed around the k-th distance that the block's
//           population suggests) and finds the bucket b* holding its (k+1)-th
//           smallest; the half records the smallest bucket of each group of
//           steps;
//   pass 2  each lane appends the candidates of buckets <= b* (at most
//           kKeep), visiting only the step groups whose smallest bucket is at
//           most the half's largest b*.  A kept candidate is one word: the
//           upper 19 bits of its distance's place in the bucket range, and its
//           13-bit position in the block;
//   sort    the words go through a sorting network in registers, the lanes side
//           by side.  Words whose 19 bits agree (distances below the bucket
//           range, and a chance pair in a hundred queries) are put in order by
//           their distances, computed again.
//
// The result is accepted only when it provably equals the ring search's list
// (the conditions of the proposal-driven box search, knn.cu): the k+1
// smallest distances are pairwise distinct; the ball of the k-th distance
// (plus a margin) lies inside the searched block, so the k kept points are
// the k nearest of the cloud; the ring search's stop step, replayed with
// decide() on that distance, visits them all; and no cell of the levels it
// visits holds max_points_in_cell points or more.  Queries whose blocks never
// reach the population that selects a level run the ring search (k_knn_plain's
// code) at the start of the same kernel; queries that fail the checks run it
// afterwards (k_knn_plain over the list of those queries).
//
// The level of a query is the first whose block around the query's cell
// holds at least kTileAlpha * (k+1) points (k_tile_assign); every cell that
// has queries at its level becomes one unit of work.
#pragma once
#include <map>
#include <mutex>
#include <utility>
#include "knn_search.cuh"
#include "proposal.cuh"

namespace egt {
namespace {

constexpr int kTileWarps = 1;    // warps per block (one: blocks pack the SM's shared memory tightly)
constexpr int kTileBins = 64;    // distance buckets per query: 8 per octave of d^2, placed by tile_unit_setup
// Forms of the search by k: list registers S of the in-kernel ring search
// (k+1 <= 32 S) and words kept per query, the query included (kKeep): k+2 and
// the rest of the last bucket, which is 9 % of the count below it on a surface.
// kWarps: warps per SM.  20 leave 96 registers a thread (4M points, k = 40: 9.23
// ms of kNN with 16 warps, 8.37 with 20, 8.69 with 23); the longest form needs
// more registers for its sorting network.
struct TileForm1 { static constexpr int S = 1, kKeep = 32, kMaxK = 22, kWarps = 20; };
struct TileForm2 { static constexpr int S = 2, kKeep = 56, kMaxK = 40, kWarps = 20; };
struct TileForm3 { static constexpr int S = 3, kKeep = 80, kMaxK = 64, kWarps = 16; };
constexpr int kTilePosBits = 13;  // block positions (kTileMaxBlock)
constexpr int kTileMaxUnsorted = 16;  // points below the bucket range a query may have (more: the ring search)
// Smallest k and cloud the tile search takes.  Below kTileMinPoints points its
// chain of launches and its long batches cost more than the ring search of
// every query (sphere, k = 16: 30,000 points 97 against 94 us, 40,000 126 against
// 139, 50,000 140 against 191; clustered clouds turn later, 100,000 to 200,000, but
// there the tiles are still 1.2 to 1.5 times as fast as with 16 warps and
// insertion sorts); k of 8 to 15 pays from kTileMinPointsLowK points
// (superquadrics, k = 8: 65,536 points 0.65 times the ring search's speed, 100,000
// 0.74, 200,000 1.05, 1M 1.8; sphere 1.7, 1.8, 1.8, 1.9), and not where more than one
// query in kTileLowShare is left to the ring search (k_tile_gather).
constexpr int kTileMinK = 8;
constexpr int kTileLowK = 16;
constexpr int64_t kTileMinPoints = 40000;
constexpr int64_t kTileMinPointsLowK = 100000;
constexpr int kTileLowShare = 16;
constexpr int64_t kTileMinCloudLowK = 5000;  // points a cloud in a batch, on average (k = 10: 64 clouds of 2,000 points
                                             // 503 against 444 us, 10 of 12,000 273 against 369)
constexpr int kTileMaxK = 64;    // largest k the cell-tile search takes
inline bool tile_takes(int64_t n, int k) {
    return k >= kTileMinK && k <= kTileMaxK && n >= (k < kTileLowK ? kTileMinPointsLowK : kTileMinPoints);
}
constexpr int kTileAlpha = 6;    // block population that selects a level, in units of k+1 (4M
                                 // superquadrics, k = 40: 8.37 ms; 5: 8.69; 4: 9.56, more rows uncertified)
constexpr int kTileEff = 24;     // smaller k select a block as if k were this: blocks of fewer points hold
                                 // fewer queries than lanes (1M points: k = 10 2.34 -> 1.96 ms, k = 16
                                 // 2.42 -> 2.30; 40 in its place: 2.02 and 2.33)
constexpr int kTileSparse = 2;       // a finer block below (k+1)/kTileSparse points: the ring search (measured
                                      // on 4M superquadrics at k = 40: (k+1)/2 and 0.6(k+1) best, 0.75(k+1)
                                      // 8 % slower, 0.45(k+1) and below 15 % slower: its long searches return)
constexpr int kTileMaxBlock = 6144;   // larger blocks: the ring search (one warp would hold the search's end)
static_assert(kTileMaxBlock <= 1 << kTilePosBits, "block positions fit their bits");
static_assert(kTileMaxBlock <= 128 * 4 * 16, "the step groups of a block fit the half's 128 bytes");
constexpr int kTileStartLevel = 3;   // the assignment's first level (the usual one on dense clouds)
constexpr int kTileClasses = 6;       // batch classes by block size (>= 4096, 2048, 1024, 512, 256, less)

struct TileArgs {
    uint8_t* lq;                      // [n] level each query is searched at (0xff: ring search)
    uint32_t* unit_bits;              // [kMaxLevels][words] cells that already have a unit
    int words;                        // words per level
    unsigned long long* units;        // [n] cloud << 40 | level << 32 | cell index
    unsigned long long* n_units;      // units written by k_tile_assign
    unsigned long long* unit_work;    // next unit to claim
    int* ring;                        // [n] queries for the ring search
    unsigned long long* n_ring;       // their count
    int maxblock;                     // kTileMaxBlock
    uint32_t* qarr;                   // [n] the units' queries, grouped by unit (k_tile_gather)
    unsigned long long* n_q;          // queries written to qarr
    uint2* batch;                     // [n + n/16 + 1 >= units + queries/16] (unit index, first query in qarr), largest blocks first
    uint8_t* bcnt;                    // [the same] queries in each batch (1..16)
    uint32_t* ucnt;                   // [n] queries of each unit
    uint8_t* ucls;                    // [n] class of each unit's block
    unsigned long long* cls_n;        // [kTileClasses] batches per class
    unsigned long long* cls_fill;     // [kTileClasses] batches written per class
    int* ring2;                       // [n] queries the tile search could not certify
    unsigned long long* n_ring2;      // their count
    unsigned long long* ring_work;    // next query of `ring` for the tile kernel's ring search
    // Several clouds (egt_batch): the search arguments of each cloud, and each
    // point's cloud.  Queries, lq and the ring lists then use indices over
    // all clouds' points; a single cloud passes its own arguments instead.
    const KnnArgs* desc;
    const uint16_t* cloud_of;
    int npts;                         // points of all clouds
    bool low_k;                       // every k the tiles take is below kTileLowK
};

// The search arguments of cloud c: the kernel's own (one cloud), or the
// cloud's descriptor.
template <bool kBatch>
__device__ __forceinline__ const KnnArgs& tile_args(const KnnArgs& a, const TileArgs& t, int c) {
    if constexpr (kBatch) return t.desc[c];
    else return a;
}

__device__ __forceinline__ unsigned long long unit_code(int c, int l, int ci) {
    return ((unsigned long long)c << 40) | ((unsigned long long)l << 32) | (unsigned)ci;
}
__device__ __forceinline__ void unit_parts(unsigned long long code, int& c, int& l, int& ci) {
    c = (int)(code >> 40);
    l = (int)((code >> 32) & 0xffu);
    ci = (int)(code & 0xffffffffu);
}

constexpr int kTileStage = 3 * 16;

// Shared memory of one warp (both halves).
// Rows of the bucket space: the buckets, then the kept words (one row each).
template <typename Form>
constexpr int tile_rows() { return kTileBins > Form::kKeep ? kTileBins : Form::kKeep; }

template <typename Form>
constexpr size_t tile_warp_bytes() {
    return (size_t)tile_rows<Form>() * 32 * 4      // bucket counts, then kept words [row][lane]
           + 2 * kTileStage * 4                    // staged candidates per half: x, y, z of 16, negated
           + 2 * 2 * 16 * 4;                       // per half: range sequence scratch at unit set-up,
                                                   // then the step groups' smallest buckets
}

// Index of level cell (cx, cy, cz) in the level's cell arrays (-1: empty).
__device__ __forceinline__ int cell_index(const LevelDev& L, int cx, int cy, int cz) {
    if (cx < 0 || cx >= L.B || cy < 0 || cy >= L.B || cz < 0 || cz >= L.B) return -1;
    const int2 rr = L.row_range[cy + cz * L.B];
    int lo = rr.x, hi = rr.y;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (L.cell_x[mid] < cx) lo = mid + 1;
        else hi = mid;
    }
    return (lo < rr.y && L.cell_x[lo] == cx) ? lo : -1;
}

// Appends the flagged values of the warp to a device list (one atomic per warp).
__device__ __forceinline__ void warp_append(bool flag, uint32_t v, uint32_t* list, unsigned long long* count,
                                            int lane) {
    const unsigned m = __ballot_sync(0xffffffffu, flag);
    if (!m) return;
    const int leader = __ffs(m) - 1;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(count, (unsigned long long)__popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (flag) list[base + __popc(m & ((1u << lane) - 1u))] = v;
}

__device__ __forceinline__ void warp_append64(bool flag, unsigned long long v, unsigned long long* list,
                                              unsigned long long* count, int lane) {
    const unsigned m = __ballot_sync(0xffffffffu, flag);
    if (!m) return;
    const int leader = __ffs(m) - 1;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(count, (unsigned long long)__popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (flag) list[base + __popc(m & ((1u << lane) - 1u))] = v;
}

// Level and unit of every query; queries that no level selects (or every
// query when the admission threshold can cut lists, or when k is outside
// [kTileMinK, kTileMaxK]) go to the ring search.  i runs over the points of
// all clouds (their sorted order).
template <bool kBatch>
__global__ void __launch_bounds__(256) k_tile_assign(KnnArgs a, TileArgs t) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool in = i < t.npts;
    const int c = (kBatch && in) ? (int)t.cloud_of[i] : 0;
    const KnnArgs& A = tile_args<kBatch>(a, t, c);
    const int q = i - (int)A.gbase;
    int lsel = -1, ci = -1;
    // thres > 4 exceeds every squared distance of the unit cube: all admitted
    if (in && A.k >= kTileMinK && A.k <= kTileMaxK && A.np->thres > 4.0f) {
        const int thr = kTileAlpha * (max(A.k, kTileEff) + 1), sparse = (A.k + 1) / kTileSparse;
        const uint32_t c0 = __float_as_uint(A.p4[q].w);
        const int cx0 = c0 & 1023u, cy0 = (c0 >> 10) & 1023u, cz0 = (c0 >> 20) & 1023u;
        // Population of the block of level l around the query's cell; the
        // blocks are nested, so it grows with l, and the first level that
        // reaches thr is found from a start near the usual one.
        auto block_pop = [&](int l) {
            const LevelDev& LV = A.lv[l];
            const int cx = cx0 >> l, cy = cy0 >> l, cz = cz0 >> l;
            int pop = 0;
#pragma unroll
            for (int r = 0; r < 9; r++) {
                const int2 g = row_points(LV, cx - 1, cx + 1, cy + r % 3 - 1, cz + r / 3 - 1);
                pop += g.y - g.x;
            }
            return pop;
        };
        int l = kTileStartLevel, pop = block_pop(l), prev = INT_MAX;  // prev: the block one level finer
        if (pop >= thr) {
            while (l > 0) {
                const int below = block_pop(l - 1);
                if (below < thr) { prev = below; break; }
                l--;
                pop = below;
            }
        } else {
            while (l + 1 < kMaxLevels && pop < thr) {
                prev = pop;
                pop = block_pop(++l);
            }
        }
        if (pop >= thr) {
            // kMaxLevels: a block too large, or a query alone in its finer
            // block -- the ring search (such a query's k nearest lie far
            // off, beyond the block, and its search climbs high)
            lsel = pop <= t.maxblock && prev >= sparse ? l : kMaxLevels;
            if (lsel == l) ci = cell_index(A.lv[l], cx0 >> l, cy0 >> l, cz0 >> l);
        }
    }
    if (lsel >= kMaxLevels || ci < 0) lsel = -1;  // ci < 0 cannot happen: the query's own cell is occupied
    // The tile kernel runs the ring search of the queries its k range takes
    // but no level selects (few, some long: they overlap the batches); the
    // clouds outside that range run it in the launch after the tile kernel,
    // at the ring search's own occupancy.
    const bool ring = in && lsel < 0;
    const bool early = A.k >= kTileMinK && A.k <= kTileMaxK;
    warp_append(ring && early, (uint32_t)i, reinterpret_cast<uint32_t*>(t.ring), t.n_ring, lane);
    warp_append(ring && !early, (uint32_t)i, reinterpret_cast<uint32_t*>(t.ring2), t.n_ring2, lane);
    if (in) t.lq[i] = lsel < 0 ? (uint8_t)0xff : (uint8_t)lsel;
    bool fresh = false;
    if (lsel >= 0) {
        // a cell is named by the first position of its points in the level's order
        const int first = (int)A.gbase + A.lv[lsel].cell_start[ci];
        const uint32_t bit = 1u << (first & 31);
        fresh = !(atomicOr(t.unit_bits + (size_t)lsel * t.words + (first >> 5), bit) & bit);
    }
    warp_append64(fresh, unit_code(c, lsel, ci), t.units, t.n_units, lane);
}

// Class of a block of `pop` candidates: larger blocks are searched first, and
// batches claimed together have blocks of similar size (the two halves of a
// warp run in step, each as long as the larger of their blocks).
__device__ __forceinline__ int tile_class(int pop) {
    return pop >= 4096 ? 0 : pop >= 2048 ? 1 : pop >= 1024 ? 2 : pop >= 512 ? 3 : pop >= 256 ? 4 : 5;
}

// Whether the search leaves every query to the launch after the tile kernel:
// with k below kTileLowK, when the assignment left more than one query in
// kTileLowShare to the ring search.  Short lists make the ring search cheap and
// the dense blocks of such clouds dear: eight clusters of widths 0.002 to 0.3, k = 8,
// 13 % left: 100,000 points 0.81 times the ring search's speed with tiles;
// 62 %: 1M 0.60.
__device__ __forceinline__ bool tile_bails(const TileArgs& t) {
    return t.low_k && *t.n_ring * kTileLowShare > (unsigned long long)t.npts;
}

// Per unit (one warp per unit, grid-stride): its query count and block class,
// and the batch count of each class.
template <bool kBatch>
__global__ void __launch_bounds__(256) k_tile_count(KnnArgs a, TileArgs t) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int nw = (int)((gridDim.x * blockDim.x) >> 5);
    if (tile_bails(t)) return;
    const unsigned long long nu = *t.n_units;
    for (unsigned long long u = gw; u < nu; u += nw) {
        int c, l, ci;
        unit_parts(t.units[u], c, l, ci);
        const KnnArgs& A = tile_args<kBatch>(a, t, c);
        const LevelDev& LV = A.lv[l];
        const int* order = l ? LV.order : nullptr;
        const int cs = LV.cell_start[ci], ce = LV.cell_start[ci + 1];
        const uint8_t* lq = t.lq + A.gbase;
        int cnt = 0;
        for (int s = cs; s < ce; s += 32) {
            bool sel = false;
            if (s + lane < ce) {
                const int qq = order ? order[s + lane] : s + lane;
                sel = lq[qq] == (uint8_t)l;
            }
            cnt += __popc(__ballot_sync(0xffffffffu, sel));
        }
        const int p0 = order ? order[cs] : cs;
        const uint32_t cc = __float_as_uint(A.p4[p0].w);
        const int cx = (int)(cc & 1023u) >> l, cy = (int)((cc >> 10) & 1023u) >> l, cz = (int)((cc >> 20) & 1023u) >> l;
        int pop = 0;
        if (lane < 9) {
            const int2 g = row_points(LV, cx - 1, cx + 1, cy + lane % 3 - 1, cz + lane / 3 - 1);
            pop = g.y - g.x;
        }
        pop = __reduce_add_sync(0xffffffffu, pop);
        const int cls = tile_class(pop);
        if (lane == 0) {
            t.ucnt[u] = (uint32_t)cnt;
            t.ucls[u] = (uint8_t)cls;
            atomicAdd(&t.cls_n[cls], (unsigned long long)((cnt + 15) >> 4));
        }
    }
}

// Compacts each unit's queries into qarr and cuts them into batches of up to
// 16 (one warp per unit, grid-stride), the batches ordered by class.
template <bool kBatch>
__global__ void __launch_bounds__(256) k_tile_gather(KnnArgs a, TileArgs t) {
    grid_dependency_wait();
    grid_dependents_launch();
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int nw = (int)((gridDim.x * blockDim.x) >> 5);
    if (tile_bails(t)) {
        for (int i = (int)(blockIdx.x * blockDim.x + threadIdx.x); i < t.npts; i += (int)(gridDim.x * blockDim.x))
            t.ring2[i] = i;
        if (blockIdx.x == 0 && threadIdx.x == 0) *t.n_ring2 = (unsigned long long)t.npts;
        return;
    }
    const unsigned long long nu = *t.n_units;
    // first batch of each class
    unsigned long long coff = 0;
    {
        unsigned long long v = lane < kTileClasses ? t.cls_n[lane] : 0ull;
        unsigned long long incl = v;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const unsigned long long w = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += w;
        }
        coff = incl - v;
    }
    for (unsigned long long u = gw; u < nu; u += nw) {
        int c, l, ci;
        unit_parts(t.units[u], c, l, ci);
        const KnnArgs& A = tile_args<kBatch>(a, t, c);
        const LevelDev& LV = A.lv[l];
        const int* order = l ? LV.order : nullptr;
        const int cs = LV.cell_start[ci], ce = LV.cell_start[ci + 1];
        const uint8_t* lq = t.lq + A.gbase;
        const int cnt = (int)t.ucnt[u], cls = (int)t.ucls[u];
        const int nbat = (cnt + 15) >> 4;
        const unsigned long long base = __shfl_sync(0xffffffffu, coff, cls);
        unsigned long long qb = 0, bb = 0;
        if (lane == 0 && cnt > 0) {
            qb = atomicAdd(t.n_q, (unsigned long long)cnt);
            bb = base + atomicAdd(&t.cls_fill[cls], (unsigned long long)nbat);
        }
        qb = __shfl_sync(0xffffffffu, qb, 0);
        bb = __shfl_sync(0xffffffffu, bb, 0);
        int w = 0;
        for (int s = cs; s < ce && w < cnt; s += 32) {
            bool sel = false;
            int qq = -1;
            if (s + lane < ce) {
                qq = order ? order[s + lane] : s + lane;
                sel = lq[qq] == (uint8_t)l;
            }
            const unsigned m = __ballot_sync(0xffffffffu, sel);
            if (sel) t.qarr[qb + w + __popc(m & ((1u << lane) - 1u))] = (uint32_t)qq;
            w += __popc(m);
        }
        for (int j = lane; j < nbat; j += 32) {
            t.batch[bb + j] = make_uint2((uint32_t)u, (uint32_t)(qb + 16 * j));
            t.bcnt[bb + j] = (uint8_t)min(16, cnt - 16 * j);
        }
    }
}

// Half-warp form of range_seq (knn_search.cuh): the ranges of a half's lanes
// (hl = lane within the half, hf = which half) as one flattened sequence.
// All 32 lanes call it; each half gets its own sequence.
__device__ __forceinline__ RangeSeq range_seq16(int sz, int cs, int hl, int hf, int* s_pref, int* s_start) {
    int incl = sz;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o, 16);
        if (hl >= o) incl += v;
    }
    const unsigned ne = (__ballot_sync(0xffffffffu, sz > 0) >> (16 * hf)) & 0xffffu;
    RangeSeq q;
    q.total = __shfl_sync(0xffffffffu, incl, 15, 16);
    q.m = __popc(ne);
    __syncwarp();
    if (sz > 0) {
        const int r = __popc(ne & ((1u << hl) - 1u));
        s_pref[r] = incl;
        s_start[r] = cs;
    }
    __syncwarp();
    q.incl = hl < q.m ? s_pref[hl] : INT_MAX;
    q.cs = hl < q.m ? s_start[hl] : 0;
    __syncwarp();
    return q;
}

// Half-warp form of seq_index: point index of candidate base + hl of the
// half's sequence (-1 past its end).  All 32 lanes call it.
__device__ __forceinline__ int seq_index16(const RangeSeq& q, int base, int hl, int hf,
                                           const int* __restrict__ order) {
    const int before = __popc((__ballot_sync(0xffffffffu, q.incl <= base) >> (16 * hf)) & 0xffffu);
    const int at = q.incl - base;
    const unsigned sb = (at > 0 && at < 16) ? (1u << at) : 0u;
    const unsigned starts = (__reduce_or_sync(0xffffffffu, sb << (16 * hf)) >> (16 * hf)) & 0xffffu;
    const int c = before + __popc(starts & ((2u << hl) - 1u));
    const int prev_end = __shfl_sync(0xffffffffu, q.incl, (c - 1) & 15, 16);
    const int cs = __shfl_sync(0xffffffffu, q.cs, c & 15, 16);
    const int j = base + hl;
    if (j >= q.total) return -1;
    const int pos = cs + (j - (c > 0 ? prev_end : 0));
    return order ? __ldg(order + pos) : pos;
}

// Distance buckets: an eighth of an octave of d^2 each, so the upper bits of
// the float (sign, exponent, three bits of the mantissa) number them; `first`
// is the number of bucket 0.  tile_clamp puts a distance into the range of the
// kTileBins buckets (NaN into the last: never kept).
constexpr int kTileShift = 20;
__device__ __forceinline__ float tile_clamp(float d, uint32_t first) {
    return fmaxf(fminf(d, __uint_as_float((first + kTileBins - 1) << kTileShift)),
                 __uint_as_float(first << kTileShift));
}
// Shared-memory address of a clamped distance's bucket; base: that of number 0
// for the lane (bucket rows are 32 words).
__device__ __forceinline__ uint32_t tile_addr(float clamped, uint32_t base) {
    return base + ((__float_as_uint(clamped) >> kTileShift) << 7);
}
__device__ __forceinline__ void shared_inc(uint32_t addr) {
    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(addr) : "memory");
}
// Squared distances of the lane's query to the half's 16 staged candidates.
__device__ __forceinline__ void tile_distances(const float* stage, float4 pq, float d[16]) {
    const float2 qx = make_float2(pq.x, pq.x), qy = make_float2(pq.y, pq.y), qz = make_float2(pq.z, pq.z);
#pragma unroll
    for (int j = 0; j < 16; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(stage + j);
        const float4 y = *reinterpret_cast<const float4*>(stage + 16 + j);
        const float4 z = *reinterpret_cast<const float4*>(stage + 32 + j);
        const float2 a = fs_dist3x2(qx, qy, qz, make_float2(x.x, x.y), make_float2(y.x, y.y), make_float2(z.x, z.y));
        const float2 b = fs_dist3x2(qx, qy, qz, make_float2(x.z, x.w), make_float2(y.z, y.w), make_float2(z.z, z.w));
        d[j] = a.x;
        d[j + 1] = a.y;
        d[j + 2] = b.x;
        d[j + 3] = b.y;
    }
}

// Batcher's merge exchange (Knuth, The Art of Computer Programming, vol. 3,
// algorithm 5.2.2M) for N elements: 32: 191 comparators, 56: 464, 80: 849.
template <int N>
struct SortNet {
    static constexpr int count() {
        int c = 0;
        for (int p = 1; p < N; p *= 2)
            for (int k = p; k >= 1; k /= 2)
                for (int j = k % p; j + k < N; j += 2 * k)
                    for (int i = 0; i < k && i + j + k < N; i++)
                        if ((i + j) / (2 * p) == (i + j + k) / (2 * p)) c++;
        return c;
    }
    struct Table { unsigned char a[count()], b[count()]; };
    static constexpr Table make() {
        Table t{};
        int c = 0;
        for (int p = 1; p < N; p *= 2)
            for (int k = p; k >= 1; k /= 2)
                for (int j = k % p; j + k < N; j += 2 * k)
                    for (int i = 0; i < k && i + j + k < N; i++)
                        if ((i + j) / (2 * p) == (i + j + k) / (2 * p)) {
                            t.a[c] = (unsigned char)(i + j);
                            t.b[c++] = (unsigned char)(i + j + k);
                        }
        return t;
    }
    static constexpr Table table = make();
    template <int A, int B>
    static __device__ __forceinline__ void exchange(uint32_t (&v)[N]) {
        const uint32_t lo = min(v[A], v[B]), hi = max(v[A], v[B]);
        v[A] = lo;
        v[B] = hi;
    }
    template <size_t... C>
    static __device__ __forceinline__ void run(uint32_t (&v)[N], std::index_sequence<C...>) {
        (exchange<table.a[C], table.b[C]>(v), ...);
    }
    static __device__ __forceinline__ void sort(uint32_t (&v)[N]) { run(v, std::make_index_sequence<count()>()); }
};

// State of one half-warp's current unit (uniform within the half).
struct TileUnit {
    RangeSeq seq;
    const int* order;
    uint32_t first;  // number of bucket 0 (tile_clamp)
    int l;         // level; -1 = no unit
    // the block's ranges r < seq.m: pref[r] = inclusive prefix end of range r
    // (INT_MAX past the last), adj[r] = its start less the positions before it
    int pref[8], adj[9];
};

// Point index of block position `pos` of a half's unit: position pos lies in
// range r, the number of ranges ending at or before it, and its level-order
// slot is pos + adj[r] (the prefix ends increase, so the last test that holds
// picks r).
__device__ __forceinline__ int tile_point(int pos, const TileUnit& U) {
    int a = U.adj[0];
#pragma unroll
    for (int t = 0; t < 8; t++) a = pos >= U.pref[t] ? U.adj[t + 1] : a;
    const int local = pos + a;
    return U.order ? __ldg(U.order + local) : local;
}

// Streams both halves' blocks through their staging buffers, 16 candidates
// per half at a time, calling f(s) for step s: the half's staged candidates
// are the block positions 16 s .. 16 s + 15 (padding past a block's end lies
// far away).
template <typename F>
__device__ __forceinline__ void tile_stream16(const TileUnit& U, bool live, int steps, const float4* __restrict__ p4,
                                              float* stage, int hl, int hf, F&& f) {
    const float4 far = make_float4(1e18f, 1e18f, 1e18f, 0.f);
    // software pipeline: the point index of step s+2 and the position of
    // step s+1 are in flight while step s is compared
    int pB = seq_index16(U.seq, 0, hl, hf, U.order);
    int pA = seq_index16(U.seq, 16, hl, hf, U.order);
    if (!live) pA = pB = -1;
    float4 vB = pB >= 0 ? __ldg(p4 + pB) : far;
    for (int s = 0; s < steps; s++) {
        __syncwarp();
        stage[hl] = -vB.x;
        stage[16 + hl] = -vB.y;
        stage[32 + hl] = -vB.z;
        __syncwarp();
        pB = pA;
        vB = pB >= 0 ? __ldg(p4 + pB) : far;
        pA = seq_index16(U.seq, (s + 2) * 16, hl, hf, U.order);
        if (!live) pA = -1;
        f(s);
    }
    __syncwarp();
}

// The same stream over a sequence of steps of each half's own: s0 its first
// step, nxt(s) the step after s (a value >= end: none left).  The warp runs
// until both halves are done; a half that is done stages padding.
template <typename N, typename F>
__device__ __forceinline__ void tile_stream16_seq(const TileUnit& U, int s0, int end, N&& nxt,
                                                  const float4* __restrict__ p4, float* stage, int hl, int hf,
                                                  F&& f) {
    const float4 far = make_float4(1e18f, 1e18f, 1e18f, 0.f);
    int s1 = nxt(s0), s2 = nxt(s1);
    int pB = seq_index16(U.seq, min(s0, end) * 16, hl, hf, U.order);
    int pA = seq_index16(U.seq, min(s1, end) * 16, hl, hf, U.order);
    if (s0 >= end) pB = -1;
    if (s1 >= end) pA = -1;
    float4 vB = pB >= 0 ? __ldg(p4 + pB) : far;
    while (__any_sync(0xffffffffu, s0 < end)) {
        __syncwarp();
        stage[hl] = -vB.x;
        stage[16 + hl] = -vB.y;
        stage[32 + hl] = -vB.z;
        __syncwarp();
        pB = pA;
        vB = pB >= 0 ? __ldg(p4 + pB) : far;
        pA = seq_index16(U.seq, min(s2, end) * 16, hl, hf, U.order);
        if (s2 >= end) pA = -1;
        f(s0);
        s0 = s1;
        s1 = s2;
        s2 = nxt(s2);
    }
    __syncwarp();
}

// Sets up a new unit for the lanes with `take` (both halves call it; a half
// with take = false keeps its unit).
__device__ __forceinline__ void tile_unit_setup(const KnnArgs& a, const NormParams& np, int l, int ci, bool take,
                                                int hl, int hf, int* s_pref, int* s_start, TileUnit& U) {
    int2 rg = make_int2(0, 0);
    int cx = 0, cy = 0, cz = 0;
    const int* order = nullptr;
    if (take) {
        const LevelDev& LV = a.lv[l];
        order = l ? LV.order : nullptr;
        const int cs = LV.cell_start[ci];
        const int p0 = order ? order[cs] : cs;
        const uint32_t cc = __float_as_uint(a.p4[p0].w);
        cx = (int)(cc & 1023u) >> l;
        cy = (int)((cc >> 10) & 1023u) >> l;
        cz = (int)((cc >> 20) & 1023u) >> l;
        if (hl < 9) rg = row_points(LV, cx - 1, cx + 1, cy + hl % 3 - 1, cz + hl / 3 - 1);
    }
    const RangeSeq seq = range_seq16(rg.y - rg.x, rg.x, hl, hf, s_pref, s_start);
    if (take) {
        U.seq = seq;
        U.order = order;
        U.l = l;
        int before = 0;  // positions of the ranges before range t
#pragma unroll
        for (int t = 0; t < 9; t++) {
            const bool in = t < seq.m;
            const int end = in ? s_pref[t] : INT_MAX;
            U.adj[t] = in ? s_start[t] - before : 0;
            if (t < 8) U.pref[t] = end;
            if (in) before = end;
        }
        // Buckets: 8 per octave of d^2, eight octaves.  The block's population on
        // a surface through it (9 h^2) puts the k-th distance at
        // (k+1) 9 h^2 / (pi pop): four octaves of buckets lie above that (three:
        // 2.4 % of 4M superquadric rows uncertified instead of 1.7 %), four
        // below, where about one point in 16 of the k is nearer than bucket 0.
        const float h = __fmul_rn(__fsub_rn(np.b, np.a), (float)(1 << l) * (1.0f / 1024.0f));
        const float top = 16.0f * 9.0f / 3.14159265f * (float)(a.k + 1) * h * h / (float)max(seq.total, 1);
        U.first = (__float_as_uint(fminf(top, 4.0f * h * h)) >> kTileShift) - (uint32_t)(kTileBins - 1);
    }
}

// Persistent: each half-warp claims batches (up to 16 queries of one unit)
// one at a time; both halves run their batches together.
//
// Bound: instruction issue (64 % busy at 20 warps per SM, 1,113 instructions a
// query of 1M superquadrics) and the latency of a block's stream (~600 candidates
// twice from shared memory, 16 at a time).  Before the kept
// candidates became one word each and were sorted by a network, 35 % of the
// time went to fetching their distances again and to insertion sorts whose
// steps differ from lane to lane, 29 % to the bucket places of pass 2.  One
// B200, kNN stage: 4M superquadrics, k = 40: 12.18 -> 8.37 ms; 4M sheets, k =
// 64: 16.73 -> 9.28; 1M superquadrics, k = 20: 2.55 -> 1.92.
template <bool kBatch, typename Form>
__global__ void __launch_bounds__(kTileWarps * 32, Form::kWarps) k_knn_tile(KnnArgs a, TileArgs t) {
    constexpr int S = Form::S, kKeep = Form::kKeep;
    constexpr size_t kWarpBytes = tile_warp_bytes<Form>();
    constexpr uint32_t kPosMask = (1u << kTilePosBits) - 1u;
    extern __shared__ __align__(16) unsigned char s_tile[];
    grid_dependency_wait();
    grid_dependents_launch();
    if (tile_bails(t)) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int hl = lane & 15, hf = lane >> 4;
    unsigned char* base = s_tile + (size_t)w * kWarpBytes;
    uint32_t* hist = reinterpret_cast<uint32_t*>(base);
    float* stages = reinterpret_cast<float*>(base + (size_t)tile_rows<Form>() * 32 * 4);
    float* stage = stages + kTileStage * hf;
    int* s_pref = reinterpret_cast<int*>(stages + 2 * kTileStage) + 32 * hf;
    int* s_start = s_pref + 16;
    uint32_t* hcol = hist + lane;
    unsigned long long evals = 0;
    unsigned maxlev = 0;
    // First the ring search (k_knn_plain's code, one query per warp) of the
    // queries no level selected, while the other warps already search
    // batches, so that the long ones do not end the search.  Its scratch lies
    // in the bucket space.  (Queries that fail the checks run it in a
    // separate launch at the ring kernel's own occupancy: measured faster than
    // running them here, between batches.)  It walks level by level: these queries
    // lie alone beside dense cells, whose points the finer levels' neighbours keep
    // out of the list; a jump meets them with an empty one (half of 200,000 points in
    // a dense ball, k = 40: 1.28 ms against 1.50 with the jump; 4M superquadrics 8.4 both).
    int* r_pref = reinterpret_cast<int*>(hist);
    int* r_start = r_pref + 32;
    float* r_md = reinterpret_cast<float*>(r_start + 32);
    int* r_mp = reinterpret_cast<int*>(r_md + 32 * S);
    unsigned reruns = 0;
    auto ring_query = [&](int i) {  // i: over all clouds' points
        const int c = kBatch ? (int)t.cloud_of[i] : 0;
        const KnnArgs& A = tile_args<kBatch>(a, t, c);
        const int q = i - (int)A.gbase;
        const NormParams np = *A.np;
        WarpList<S> L;
        bool invalid, rerun;
        const int reached = plain_query<true, false, S>(A, np, q, A.p4[q], L, invalid, lane, r_pref, r_start, r_md,
                                                        r_mp, rerun);
        write_query<S>(A, q, L, invalid, reached, lane);
        if constexpr (kBatch) {
            if (rerun && lane == 0) atomicAdd(&A.counters[kCtrExactRerun], 1ull);
        } else {
            reruns += rerun ? 1u : 0u;
            evals += L.ev;
        }
    };
    {
        const unsigned long long n_r = *t.n_ring;
        for (;;) {
            unsigned long long j = 0;
            if (lane == 0) j = atomicAdd(t.ring_work, 1ull);
            j = __shfl_sync(0xffffffffu, j, 0);
            if (j >= n_r) break;
            ring_query(t.ring[j]);
        }
        __syncwarp();
    }
    for (int b = 0; b < kTileBins; b++) hcol[b * 32] = 0u;
    TileUnit U;
    U.seq.incl = INT_MAX;
    U.seq.cs = 0;
    U.seq.m = 0;
    U.seq.total = 0;
    U.order = nullptr;
    U.first = 0u;
    U.l = -1;
#pragma unroll
    for (int t = 0; t < 9; t++) {
        U.adj[t] = 0;
        if (t < 8) U.pref[t] = INT_MAX;
    }
    unsigned long long n_batches = 0;
#pragma unroll
    for (int c = 0; c < kTileClasses; c++) n_batches += t.cls_n[c];
    for (;;) {
        // each half claims one batch: largest blocks first
        unsigned long long c = 0;
        if (hl == 0) c = atomicAdd(t.unit_work, 1ull);
        c = __shfl_sync(0xffffffffu, c, 16 * hf);
        const bool take = c < n_batches;
        if (!__any_sync(0xffffffffu, take)) break;
        const long long bi = take ? (long long)c : 0;
        const uint2 bd = take ? t.batch[bi] : make_uint2(0u, 0u);
        const int nq = take ? (int)t.bcnt[bi] : 0;
        int uc = 0, ul = 0, uci = 0;
        unit_parts(t.units[bd.x], uc, ul, uci);
        const KnnArgs& A = tile_args<kBatch>(a, t, uc);  // the half's cloud
        const NormParams np = *A.np;
        const int k = A.k;
        const float4* __restrict__ p4 = A.p4;
        tile_unit_setup(A, np, ul, uci, take, hl, hf, s_pref, s_start, U);
        const bool act = hl < nq;
        const int q = act ? (int)t.qarr[bd.y + hl] : -1;
        const float4 pq = act ? p4[q] : make_float4(3e18f, 3e18f, 3e18f, 0.f);
        const int total = take ? U.seq.total : 0;
        const int steps = (max(total, __shfl_xor_sync(0xffffffffu, total, 16)) + 15) >> 4;
        const uint32_t first = U.first;
        const uint32_t bins = (uint32_t)__cvta_generic_to_shared(hcol) - (first << 7);  // tile_addr's base
        // The smallest bucket of each group of g steps over the half's lanes
        // (one byte per group in the half's scratch, which the unit set-up no
        // longer needs): pass 2 visits only the groups that can hold a
        // candidate it keeps.  2^gs steps per byte (128 bytes cover a block
        // of up to 8192 candidates).
        const unsigned hmask = hf ? 0xffff0000u : 0x0000ffffu;
        const int steps_h = (total + 15) >> 4;
        const int gs = steps_h > 256 ? 2 : steps_h > 128 ? 1 : 0;
        uint8_t* mb = reinterpret_cast<uint8_t*>(s_pref);
        s_pref[hl] = -1;
        s_pref[hl + 16] = -1;
        __syncwarp();
        // pass 1: bucket counts (the query itself included, at distance 0)
        tile_stream16(U, take, steps, p4, stage, hl, hf, [&](int st) {
            float d[16], mnd = 3.0e38f;
            tile_distances(stage, pq, d);
#pragma unroll
            for (int j = 0; j < 16; j++) {
                d[j] = tile_clamp(d[j], first);
                mnd = fminf(mnd, d[j]);
            }
#pragma unroll
            for (int j = 0; j < 16; j++) shared_inc(tile_addr(d[j], bins));
            const uint32_t mn = (__reduce_min_sync(hmask, __float_as_uint(mnd)) >> kTileShift) - first;
            if (hl == 0 && st < steps_h) {
                const int gi = st >> gs;
                mb[gi] = (uint8_t)min((uint32_t)mb[gi], mn);
            }
        });
        // the bucket b* of the (k+1)-th distance other than the query's own
        int cum = 0, bstar = -1, m = 0;
        const int low = (int)hcol[0];  // nearer than the bucket range
#pragma unroll 8
        for (int b = 0; b < kTileBins; b++) {
            cum += (int)hcol[b * 32];
            if (bstar < 0 && cum >= k + 2) { bstar = b; m = cum; }
        }
        bool ok = act && bstar >= 0 && bstar < kTileBins - 1 && m <= kKeep && low <= kTileMaxUnsorted;
        const float T = ok ? __uint_as_float((first + (uint32_t)bstar + 1u) << kTileShift) : 0.0f;
        // pass 2: the candidates of buckets <= b* (over the spent counts), from the step
        // groups whose smallest bucket is at most the half's largest b*
        const int bmax = __reduce_max_sync(hmask, ok ? bstar : -1);
        const uint32_t lo = first << kTileShift;
        uint32_t* next = hcol;
        auto nxt = [&](int st) {
            int u = st + 1;
            while (u < steps_h) {
                const int gi = u >> gs;
                if ((int)mb[gi] <= bmax) break;
                u = (gi + 1) << gs;
            }
            return min(u, steps_h);
        };
        tile_stream16_seq(U, nxt(-1), steps_h, nxt, p4, stage, hl, hf, [&](int st) {
            float d[16];
            tile_distances(stage, pq, d);
#pragma unroll
            for (int j = 0; j < 16; j++) {
                if (d[j] < T) {
                    const uint32_t u = max(__float_as_uint(d[j]), lo) - lo;  // 26 bits
                    *next = ((u << 6) & ~kPosMask) | (uint32_t)(st * 16 + j);
                    next += 32;
                }
            }
        });
        {
            uint32_t v[kKeep];
#pragma unroll
            for (int i = 0; i < kKeep; i++) v[i] = ok && i < m ? hcol[i * 32] : 0xffffffffu;
            SortNet<kKeep>::sort(v);
#pragma unroll
            for (int i = 0; i < kKeep; i++) hcol[i * 32] = v[i];
        }
        // the point of a word, and its exact distance
        auto point = [&](uint32_t word) { return tile_point((int)(word & kPosMask), U); };
        auto exact = [&](uint32_t word) {
            const float4 v = __ldg(p4 + point(word));
            return fs_dist3(pq.x, pq.y, pq.z, v.x, v.y, v.z);
        };
        float kth = 0.0f;
        int reached = 0;
        int self = 0;  // the query's own word; entry i of the list is word i + (i >= self)
        if (ok) {
            // words that agree above the position, by (distance, block position)
            uint32_t before = hcol[0];
            for (int i = 1; i < m; i++) {
                uint32_t w = hcol[i * 32];
                if ((w ^ before) <= kPosMask) {
                    const float d = exact(w);
                    int j = i;
                    while (j > 0) {
                        const uint32_t g = hcol[(j - 1) * 32];
                        if ((g ^ w) > kPosMask) break;
                        const float e = exact(g);
                        if (e < d || (e == d && g < w)) break;
                        hcol[j * 32] = g;
                        j--;
                    }
                    hcol[j * 32] = w;
                    w = hcol[i * 32];
                }
                before = w;
            }
            // the query sits among the distance-0 entries at the front
            while (self < m - 1 && point(hcol[self * 32]) != q) self++;
            // (1) the k+1 smallest distances pairwise distinct
            uint32_t prev = hcol[(self == 0 ? 1 : 0) * 32];
            for (int i = 1; i <= k && ok; i++) {
                const uint32_t cur = hcol[(i + (i >= self)) * 32];
                if ((cur ^ prev) <= kPosMask) ok = exact(cur) != exact(prev);
                prev = cur;
            }
        }
        if (ok) {
            const int l = U.l;
            kth = exact(hcol[(k - 1 + (k - 1 >= self)) * 32]);
            const uint32_t c0 = __float_as_uint(pq.w);
            const int cq[3] = {(int)(c0 & 1023u), (int)((c0 >> 10) & 1023u), (int)((c0 >> 20) & 1023u)};
            // (2) the k-th ball inside the searched block
            int lo3[3], end3[3];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                lo3[d] = ((cq[d] >> l) - 1) << l;
                end3[d] = ((cq[d] >> l) + 2) << l;
            }
            ok = ball_in_box(np, pq, kth, lo3, end3);
            // (3) the ring search's stop step
            int sf = -1;
            if (ok) {
                for (int st = 0; st <= kMaxLevels; st++) {
                    const int Ls = st == 0 ? 0 : st - 1, o = st == 0 ? 0 : 1;
                    if (!decide(np, Ls, o, k, k, kth, false, pq, cq[0], cq[1], cq[2])) { sf = st; break; }
                }
                ok = sf >= 0;
            }
            if (ok) {
                const int Lf = sf == 0 ? 0 : sf - 1, of = sf == 0 ? 0 : 1;
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    lo3[d] = ((cq[d] >> Lf) - of) << Lf;
                    end3[d] = ((cq[d] >> Lf) + of + 1) << Lf;
                }
                if (!ball_in_box(np, pq, kth, lo3, end3)) {
                    for (int i = 0; i < k && ok; i++) {
                        const int p = point(hcol[(i + (i >= self)) * 32]);
                        ok = visit_step(__float_as_uint(p4[p].w), c0) <= sf;
                    }
                }
            }
            // (4) no oversized cell on the visited levels
            if (ok)
                for (int L = 0; L <= max(sf - 1, 0) && ok; L++)
                    ok = A.counters[kCtrMaxPop + L] < (unsigned long long)A.max_pts;
            reached = max(sf - 1, 0);
        }
        if (ok) {
            int* row = A.lists + (size_t)q * k;
#pragma unroll 4
            for (int i = 0; i < k; i++) row[i] = point(hcol[(i + (i >= self)) * 32]);
            if (A.kth_out) A.kth_out[q] = kth;
            if (A.qlevel) A.qlevel[q] = (uint8_t)reached;
            if constexpr (kBatch) {
                atomicMax(&A.counters[kCtrMaxLevel], (unsigned long long)reached);
            } else {
                maxlev = max(maxlev, (unsigned)reached);
            }
        }
        if (!kBatch && hl == 0) evals += (unsigned long long)total * nq;
        warp_append(act && !ok, (uint32_t)(A.gbase + q), reinterpret_cast<uint32_t*>(t.ring2), t.n_ring2, lane);
#pragma unroll 8
        for (int b = 0; b < kTileBins; b++) hcol[b * 32] = 0u;
    }
    if constexpr (kBatch) return;  // per-cloud counters were updated as the queries finished
    maxlev = __reduce_max_sync(0xffffffffu, maxlev);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) evals += __shfl_xor_sync(0xffffffffu, evals, o);
    if (lane == 0) {
        if (reruns) atomicAdd(&a.counters[kCtrExactRerun], (unsigned long long)reruns);
        if (evals) atomicAdd(&a.counters[kCtrEvals], evals);
        if (maxlev) atomicMax(&a.counters[kCtrMaxLevel], (unsigned long long)maxlev);
    }
}


// Working buffers of the cell-tile search for the handle's n points (all
// clouds' points for a batch).  The kNN counters are reset by the caller.
inline egt_status tile_prepare(egt_handle* h, TileArgs* t) {
    const int64_t n = h->n;
    const int words = (int)((n + 31) / 32);
    const int64_t bcap = n + n / 16 + 1;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t b_lq = al((size_t)n), b_bits = al((size_t)kMaxLevels * words * 4), b_n4 = al(4 * (size_t)n);
    const size_t b_n8 = al(8 * (size_t)n);
    const size_t b_batch = al(8 * (size_t)bcap), b_bcnt = al((size_t)bcap), b_ctr = 256;
    const size_t need = b_ctr + b_lq + b_bits + b_n8 + 4 * b_n4 + b_batch + b_bcnt + b_lq;
    if (h->tile_bytes < need) {
        dev_free(h, h->tile_mem);
        h->tile_mem = nullptr;
        h->tile_bytes = 0;
        EGT_CUDA_TRY(dev_alloc(h, &h->tile_mem, need));
        h->tile_bytes = need;
    }
    unsigned char* m = static_cast<unsigned char*>(h->tile_mem);
    unsigned long long* tctr = reinterpret_cast<unsigned long long*>(m);  // class counts and fills
    t->cls_n = tctr;
    t->cls_fill = tctr + kTileClasses;
    m += b_ctr;
    t->unit_bits = reinterpret_cast<uint32_t*>(m);
    m += b_bits;
    t->words = words;
    t->lq = m;
    m += b_lq;
    t->units = reinterpret_cast<unsigned long long*>(m);
    m += b_n8;
    t->ring = reinterpret_cast<int*>(m);
    m += b_n4;
    t->ring2 = reinterpret_cast<int*>(m);
    m += b_n4;
    t->qarr = reinterpret_cast<uint32_t*>(m);
    m += b_n4;
    t->ucnt = reinterpret_cast<uint32_t*>(m);
    m += b_n4;
    t->batch = reinterpret_cast<uint2*>(m);
    m += b_batch;
    t->bcnt = m;
    m += b_bcnt;
    t->ucls = m;
    t->n_units = h->d_counters + kCtrTileUnits;
    t->unit_work = h->d_counters + kCtrTileWork;
    t->n_ring = h->d_counters + kCtrSelFallback;
    t->n_q = h->d_counters + kCtrTileQ;
    t->n_ring2 = h->d_counters + kCtrTileRing2;
    t->ring_work = h->d_counters + kCtrTileRingWork1;
    t->maxblock = kTileMaxBlock;
    t->desc = nullptr;
    t->cloud_of = nullptr;
    t->npts = (int)n;
    cudaStream_t st = h->stream;
    EGT_CUDA_TRY(cudaMemsetAsync(tctr, 0, b_ctr + b_bits, st));  // class counters and unit bits
    return EGT_OK;
}

// Assignment, batching and the tile kernel (with the ring search of the
// queries no level selected); the uncertified queries are left in t.ring2.
template <bool kBatch, typename Form>
egt_status tile_kernel_launch(const KnnArgs& a, const TileArgs& t, cudaStream_t st) {
    constexpr size_t smem = tile_warp_bytes<Form>() * kTileWarps;
    static std::mutex mu;
    static std::map<int, unsigned> waves;  // per device: blocks of one resident wave
    int dev = 0;
    EGT_CUDA_TRY(cudaGetDevice(&dev));
    unsigned G = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = waves.find(dev);
        if (it != waves.end()) G = it->second;
    }
    if (!G) {
        EGT_CUDA_TRY(cudaFuncSetAttribute(k_knn_tile<kBatch, Form>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
        int sms = 0, per = 0;
        EGT_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        EGT_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_knn_tile<kBatch, Form>, kTileWarps * 32,
                                                                    smem));
        G = (unsigned)std::max(1, sms * std::max(per, 1));
        std::lock_guard<std::mutex> lock(mu);
        waves[dev] = G;
    }
    return launch_dependent(k_knn_tile<kBatch, Form>, dim3(G), dim3(kTileWarps * 32), smem, st, a, t);
}

// kmax: the largest k among the queries the tile search takes.
template <bool kBatch>
egt_status tile_launch(const KnnArgs& a, TileArgs t, int kmax, cudaStream_t st) {
    t.low_k = kmax < kTileLowK;
    const unsigned T = 256;
    const int64_t npts = t.npts;
    EGT_TRY(launch_dependent(k_tile_assign<kBatch>, dim3((unsigned)((npts + T - 1) / T)), dim3(T), 0, st, a, t));
    const unsigned Gu = (unsigned)std::min<int64_t>(4096, (npts + T - 1) / T);
    EGT_TRY(launch_dependent(k_tile_count<kBatch>, dim3(Gu), dim3(T), 0, st, a, t));
    EGT_TRY(launch_dependent(k_tile_gather<kBatch>, dim3(Gu), dim3(T), 0, st, a, t));
    if (kmax <= TileForm1::kMaxK) return tile_kernel_launch<kBatch, TileForm1>(a, t, st);
    if (kmax <= TileForm2::kMaxK) return tile_kernel_launch<kBatch, TileForm2>(a, t, st);
    return tile_kernel_launch<kBatch, TileForm3>(a, t, st);
}

}  // namespace
}  // namespace egt
