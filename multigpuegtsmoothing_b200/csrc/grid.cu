// Grid build: normalisation, level-0 cell sort and the cell hierarchy.
//
// Reference: GridStructure::InitStructure (GridKNNCuda.cu:1023-1133),
// getBuckets / InitializeLevel (GridKNNCuda.cu:898-946).
//
// Layout produced in HBM (all in cell-sorted order):
//   p4[n]      float4 (x,y,z,c) normalised positions; c = the packed level-0
//              cell coordinates (bit pattern), read together with the position
//   x/y/z[n]   SoA mirror                              -- KNNInterface views
//   cell0[n]   packed level-0 cell coords x|y<<10|z<<20
//   perm[n]    sorted slot -> original index
//   per level L (B = 1024 >> L):
//     order[n]          sorted indices grouped by level-L cell, ascending in a
//                       cell (level 0: identity, not stored)
//     cell_start[C+1]   cell -> [start,end) into order
//     cell_x[C]         x coordinate of the cell
//     row_range[B*B]    (y,z) row -> [first,last) cell, so a cell lookup is one
//                       row load plus a short binary search over x.
// Level-L cell = level-0 cell >> L exactly, because u*B_L = (u*1024)/2^L has no
// rounding; the hierarchy therefore never re-reads positions.
//
// The build is a chain of 12 launches for a small cloud: extents, keys, four
// radix passes (radix.cuh), gather, four passes that sort every level, and one
// that writes every level's tables (head flags, cell numbering by look-back, row
// ranges and largest population).
// The levels of clouds of up to 2.4M points share their launches (kGroupBytes
// of buffers), so that one level's waits are filled by the others' work; larger
// clouds sort fewer at a time (4M points 1.40 ms so, 1.36 ms with all levels
// together; one at a time 1.60 ms; 20M points 6.8 ms one at a time, 6.6 ms three
// at a time with a gigabyte of buffers).  Launches are programmatic dependents, so
// each one's start-up overlaps the end of the one before it.
//
// Measured on one B200 against a library sort per level (75 launches and
// memsets): 2,000 points 325 -> 76 us (host-bound before), 36K 603 -> 99 us, 1M
// 836 -> 410 us, 4M 1.77 -> 1.40 ms, 20M 6.89 -> 6.77 ms.
#include <algorithm>
#include <cub/cub.cuh>
#include "egt_internal.cuh"
#include "grid_common.cuh"
#include "radix.cuh"

namespace egt {
namespace {

constexpr int kT = 256;              // threads per block
constexpr int kL0Bits = 8;           // digits of the level-0 sort (30-bit keys)
constexpr int kL0Passes = 4;
constexpr int kLevelBits = kRadixBits;     // widest digit of the upper levels' sorts
constexpr int kMaxPasses = 4;
// Clouds of more points sort with the library after the first pass of each level,
// as every cloud did before the shared passes: its passes move 2 TB/s of pairs there
// against 1.6 (the votes of radix_peers bound a large pass), while the first
// pass still forms the keys and the tables come from k_tables.  Build time, library
// / this / own passes alone: sheets 20M 6.80 / 6.72 / 6.72 ms, 30M 9.95 / 9.70 / 10.19,
// 40M 12.9 / 12.9 / 13.7, 80M 24.8 / 25.8 / 27.6.
constexpr int64_t kLibrarySort = 24 << 20;
constexpr int64_t kGroupBytes = 256 << 20;  // (key, value) pairs in and out of the levels sorted together

// Digits of a level's sort: 3 (10 - L) key bits in passes of near-equal width.
constexpr int level_bits(int L) { return 3 * (10 - L); }
constexpr int level_passes(int L) { return (level_bits(L) + kLevelBits - 1) / kLevelBits; }
constexpr int pass_bits(int L, int p) {
    const int per = (level_bits(L) + level_passes(L) - 1) / level_passes(L);
    return p + 1 < level_passes(L) ? per : level_bits(L) - per * (level_passes(L) - 1);
}
constexpr int pass_shift(int L, int p) {
    return p * ((level_bits(L) + level_passes(L) - 1) / level_passes(L));
}
constexpr int kLevelHists = 4 + 3 + 3 + 3 + 2 + 2 + 2;  // passes of levels 1..7
constexpr int hist_slot(int L, int p) {
    int s = p;
    for (int l = 1; l < L; l++) s += level_passes(l);
    return s;
}
static_assert(hist_slot(kMaxLevels - 1, level_passes(kMaxLevels - 1)) == kLevelHists, "one histogram per pass");

// Per-axis min/max over AoS xyz (the six thrust::reduce calls of
// GridKNNCuda.cu:1042-1065 fused into one pass) and, in the last block to
// finish, the scalar cube.  vec: xyz is 16-byte aligned, read four points at a
// time.
__global__ void __launch_bounds__(kT) k_extents(const float* __restrict__ xyz, int64_t n, int vec, float eps,
                                                float thres0, float* __restrict__ part, uint32_t* __restrict__ ticket,
                                                NormParams* __restrict__ out,
                                                unsigned long long* __restrict__ counters) {
    __shared__ float s_red[kT / 32][6];
    __shared__ uint32_t s_last;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    auto take = [&](float v, int d) { lo[d] = fminf(lo[d], v); hi[d] = fmaxf(hi[d], v); };
    const int64_t t0 = blockIdx.x * (int64_t)kT + threadIdx.x, stride = (int64_t)gridDim.x * kT;
    const int64_t quads = vec ? n / 4 : 0;
    const float4* v4 = reinterpret_cast<const float4*>(xyz);
    for (int64_t i = t0; i < quads; i += stride) {
        const float4 a = v4[3 * i], b = v4[3 * i + 1], c = v4[3 * i + 2];
        take(a.x, 0); take(a.y, 1); take(a.z, 2); take(a.w, 0); take(b.x, 1); take(b.y, 2);
        take(b.z, 0); take(b.w, 1); take(c.x, 2); take(c.y, 0); take(c.z, 1); take(c.w, 2);
    }
    for (int64_t i = 4 * quads + t0; i < n; i += stride) {
#pragma unroll
        for (int d = 0; d < 3; d++) take(xyz[3 * i + d], d);
    }
    // block reduction of lo/hi, the result in threads 0..5 (lo x y z, hi x y z)
    auto reduce = [&]() {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            for (int o = 16; o > 0; o >>= 1) {
                lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
                hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
            }
            if ((threadIdx.x & 31) == 0) {
                s_red[threadIdx.x >> 5][d] = lo[d];
                s_red[threadIdx.x >> 5][3 + d] = hi[d];
            }
        }
        __syncthreads();
        float v = 0.0f;
        if (threadIdx.x < 6) {
            v = s_red[0][threadIdx.x];
            for (int w = 1; w < kT / 32; w++)
                v = threadIdx.x < 3 ? fminf(v, s_red[w][threadIdx.x]) : fmaxf(v, s_red[w][threadIdx.x]);
        }
        return v;
    };
    const float v = reduce();
    if (threadIdx.x < 6) {
        part[blockIdx.x * 6 + threadIdx.x] = v;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
#pragma unroll
    for (int d = 0; d < 3; d++) { lo[d] = INFINITY; hi[d] = -INFINITY; }
    for (unsigned b = threadIdx.x; b < gridDim.x; b += kT) {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            lo[d] = fminf(lo[d], __ldcg(part + b * 6 + d));
            hi[d] = fmaxf(hi[d], __ldcg(part + b * 6 + 3 + d));
        }
    }
    const float r = reduce();
    if (threadIdx.x < 6) s_red[0][threadIdx.x] = r;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t acc[6];
        for (int d = 0; d < 6; d++) acc[d] = f2ord(s_red[0][d]);
        *out = finalize_norm(acc, eps, thres0, n);
    }
    if (threadIdx.x < kMaxLevels) counters[kCtrMaxPop + threadIdx.x] = 0ull;  // k_tables fills them
}

// GRIDCUDAKNNSELF_COMPACT's threshold scaling (GridKNNCuda.cu:2324-2325):
// thres /= (maxExtent - minExtent); thres *= thres.
__global__ void k_set_thres(float thres0, NormParams* np) {
    float t = __fdiv_rn(thres0, __fsub_rn(np->mx, np->mn));
    np->thres = __fmul_rn(t, t);
}

// normalize_points (GridKNNCuda.cu:840-849).
__device__ __forceinline__ float4 normalized(const float* __restrict__ xyz, int64_t i, const NormParams& p) {
    const float d = __fsub_rn(p.mx, p.mn);
    return make_float4(__fdiv_rn(__fsub_rn(xyz[3 * i], p.mn), d), __fdiv_rn(__fsub_rn(xyz[3 * i + 1], p.mn), d),
                       __fdiv_rn(__fsub_rn(xyz[3 * i + 2], p.mn), d), 0.f);
}

// Level-0 keys (get_buckets_no_binary at B=1024, GridKNNCuda.cu:74-88) and
// the counts of their first digit.
__global__ void __launch_bounds__(kT) k_keys(const float* __restrict__ xyz, int64_t n,
                                             const NormParams* __restrict__ np, uint32_t* __restrict__ key,
                                             uint32_t* __restrict__ hist) {
    __shared__ uint32_t s_hist[1 << kL0Bits];
    for (int i = threadIdx.x; i < 1 << kL0Bits; i += kT) s_hist[i] = 0u;
    __syncthreads();
    grid_dependency_wait();
    grid_dependents_launch();
    const NormParams p = *np;
    for (int64_t i = blockIdx.x * (int64_t)kT + threadIdx.x; i < n; i += (int64_t)gridDim.x * kT) {
        const float4 v = normalized(xyz, i, p);
        const int xi = cell_coord(v.x, p.a, p.b, 1024), yi = cell_coord(v.y, p.a, p.b, 1024),
                  zi = cell_coord(v.z, p.a, p.b, 1024);
        const uint32_t k = ((uint32_t)xi + (uint32_t)yi * 1024u + (uint32_t)zi * 1024u * 1024u) & 0x3fffffffu;
        key[i] = k;
        atomicAdd(&s_hist[k & ((1u << kL0Bits) - 1u)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 1 << kL0Bits; i += kT)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// thrust::gather into sorted order (GridKNNCuda.cu:1114-1125) + SoA mirror.
// The positions are normalised again from the input: 12 bytes gathered per
// point against 16 written and 16 gathered for a stored copy.  Counts the
// first digit of every upper level's sort (hist of pass 0 of level L at
// hist_slot(L, 0); nullptr: no upper levels).
__global__ void __launch_bounds__(kT) k_gather_sorted(const float* __restrict__ xyz, const int* __restrict__ perm,
                                                      const uint32_t* __restrict__ key, int64_t n,
                                                      float4* __restrict__ p4, float* __restrict__ x,
                                                      float* __restrict__ y, float* __restrict__ z,
                                                      uint32_t* __restrict__ cell0,
                                                      const NormParams* __restrict__ np, uint32_t* __restrict__ hist) {
    __shared__ uint32_t s_hist[(kMaxLevels - 1) << kLevelBits];
    for (int i = threadIdx.x; i < (kMaxLevels - 1) << kLevelBits; i += kT) s_hist[i] = 0u;
    __syncthreads();
    grid_dependency_wait();
    grid_dependents_launch();
    const NormParams p = *np;
    for (int64_t s = blockIdx.x * (int64_t)kT + threadIdx.x; s < n; s += (int64_t)gridDim.x * kT) {
        const uint32_t packed = key[s];  // x + y*1024 + z*1024^2 is the packed form
        float4 v = normalized(xyz, perm[s], p);
        x[s] = v.x; y[s] = v.y; z[s] = v.z;
        cell0[s] = packed;
        v.w = __uint_as_float(packed);  // the kNN reads a candidate's cell with its position
        p4[s] = v;
        if (hist) {
#pragma unroll
            for (int L = 1; L < kMaxLevels; L++)
                atomicAdd(&s_hist[((L - 1) << kLevelBits) + (level_key(packed, L) & ((1u << pass_bits(L, 0)) - 1u))],
                          1u);
        }
    }
    if (!hist) return;
    __syncthreads();
#pragma unroll
    for (int L = 1; L < kMaxLevels; L++)
        for (int i = threadIdx.x; i < 1 << pass_bits(L, 0); i += kT) {
            const uint32_t c = s_hist[((L - 1) << kLevelBits) + i];
            if (c) atomicAdd(&hist[(hist_slot(L, 0) << kLevelBits) + i], c);
        }
}

// Cell tables of one level from its sorted keys.
struct TableJob {
    const uint32_t* key;
    int* cell_start;
    int* cell_x;
    int2* row_range;
    unsigned long long* state;  // [tiles], zero
    uint32_t* ticket;           // zero
    int L;
};
struct TableBatch {
    TableJob job[kMaxLevels];
    int n;
    int polls;
    unsigned long long* counters;
};
constexpr int kTableItems = 16;
constexpr int kTableTile = kT * kTableItems;
// Look-back word: state (2 bits), heads (31 bits), 1 + position of the last head (31 bits; 0: none).
constexpr unsigned long long kWordSum = 1ull << 62, kWordFull = 2ull << 62, kLow31 = (1ull << 31) - 1;

// unique_by_key + cell starts (GridKNNCuda.cu:915-925), plus the row index:
// the head of cell c closes the row of cell c-1 when the rows differ.  Cells
// are numbered by decoupled look-back over the tiles' head counts (radix.cuh);
// the words also carry the last head's position, which gives every cell's
// population where the next one starts.
__global__ void __launch_bounds__(kT) k_tables(const __grid_constant__ TableBatch b) {
    __shared__ uint32_t s_tile, s_cnt[kT / 32], s_lst[kT / 32], s_prev, s_plast, s_pop[kT / 32];
    grid_dependency_wait();
    grid_dependents_launch();
    const TableJob& j = b.job[blockIdx.y];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    if (threadIdx.x == 0) s_tile = atomicAdd(j.ticket, 1u);
    __syncthreads();
    const int tile = (int)s_tile;
    const int64_t first = (int64_t)tile * kTableTile;
    const uint32_t* __restrict__ key = j.key;
    auto is_head = [&](int64_t i) { return i == 0 || key[i] != key[i - 1]; };
    uint32_t k[kTableItems];
    unsigned heads[kTableItems];
    uint32_t cnt = 0, lst = 0;  // the warp's heads, 1 + position of its last one
#pragma unroll
    for (int i = 0; i < kTableItems; i++) {
        const int64_t at = first + w * (32 * kTableItems) + i * 32 + lane;
        k[i] = at < b.n ? key[at] : 0u;
    }
#pragma unroll
    for (int i = 0; i < kTableItems; i++) {
        const int64_t at = first + w * (32 * kTableItems) + i * 32 + lane;
        uint32_t pk = __shfl_up_sync(0xffffffffu, k[i], 1);
        if (lane == 0 && at > 0 && at < b.n) pk = key[at - 1];
        heads[i] = __ballot_sync(0xffffffffu, at < b.n && (at == 0 || k[i] != pk));
        cnt += __popc(heads[i]);
        if (heads[i]) lst = (uint32_t)(at - lane + (31 - __clz(heads[i])) + 1);
    }
    if (lane == 0) { s_cnt[w] = cnt; s_lst[w] = lst; }
    __syncthreads();
    uint32_t tcnt = 0, tlst = 0, before = 0, carry = 0;
#pragma unroll
    for (int u = 0; u < kT / 32; u++) {
        if (u < w) { before += s_cnt[u]; carry = max(carry, s_lst[u]); }
        tcnt += s_cnt[u];
        tlst = max(tlst, s_lst[u]);
    }
    auto store = [&](int t, unsigned long long v) {
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(j.state + t), "l"(v) : "memory");
    };
    auto load = [&](int t) {
        unsigned long long v;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(j.state + t) : "memory");
        return v;
    };
    bool lost = false;
    if (w == 0) {
        if (lane == 0)
            store(tile, (tile ? kWordSum : kWordFull) | ((unsigned long long)tcnt << 31) | tlst);
        uint32_t prev = 0, plast = 0;
        for (int t0 = tile - 1; t0 >= 0 && !lost; t0 -= 32) {  // 32 words at a time, nearest on lane 0
            const int t = t0 - lane;
            unsigned long long v = kWordFull;
            if (t >= 0) {
                v = load(t);
                for (int tries = 0; v == 0ull && tries < b.polls; tries++) v = load(t);
            }
            const unsigned full = __ballot_sync(0xffffffffu, (v & kWordFull) != 0ull);
            const int stop = full ? __ffs(full) - 1 : 31;  // words past the nearest full one are not needed
            lost = __any_sync(0xffffffffu, lane <= stop && v == 0ull);
            uint32_t c = lane <= stop ? (uint32_t)((v >> 31) & kLow31) : 0u;
            uint32_t l = lane <= stop ? (uint32_t)(v & kLow31) : 0u;
            prev += __reduce_add_sync(0xffffffffu, c);
            plast = max(plast, __reduce_max_sync(0xffffffffu, l));
            if (full) break;
        }
        if (lane == 0) { s_prev = prev; s_plast = plast; }
    }
    if (__syncthreads_or(lost)) {  // a predecessor did not answer: count its heads here
        if (threadIdx.x == 0) atomicAdd(&b.counters[kCtrRecounts], 1ull);
        uint32_t c = 0, l = 0;
        for (int64_t i = threadIdx.x; i < first; i += kT)
            if (is_head(i)) { c++; l = (uint32_t)i + 1u; }
        c = __reduce_add_sync(0xffffffffu, c);
        l = __reduce_max_sync(0xffffffffu, l);
        if (threadIdx.x == 0) { s_prev = 0u; s_plast = 0u; }
        __syncthreads();
        if (lane == 0) { atomicAdd(&s_prev, c); atomicMax(&s_plast, l); }
        __syncthreads();
    }
    const uint32_t prev = s_prev, plast = s_plast;
    if (threadIdx.x == 0 && tile)
        store(tile, kWordFull | ((unsigned long long)(prev + tcnt) << 31) | max(tlst, plast));
    const int bits = 10 - j.L;
    int c0 = (int)(prev + before);     // cells before this warp's
    uint32_t head = max(carry, plast);  // 1 + position of the last head before
    uint32_t pop = 0;
#pragma unroll
    for (int i = 0; i < kTableItems; i++) {
        const int64_t at = first + w * (32 * kTableItems) + i * 32 + lane;
        const unsigned lower = heads[i] & below;
        const uint32_t base = (uint32_t)(at - lane);
        const uint32_t ph = lower ? base + (31 - __clz(lower)) + 1u : head;
        const int c = c0 + __popc(lower);
        if ((heads[i] >> lane) & 1u) {
            j.cell_start[c] = (int)at;
            j.cell_x[c] = (int)(k[i] & ((1u << bits) - 1u));
            const uint32_t row = k[i] >> bits;
            if (c == 0) {
                j.row_range[row].x = 0;
            } else {
                pop = max(pop, (uint32_t)at + 1u - ph);
                const uint32_t prow = key[at - 1] >> bits;
                if (prow != row) {
                    j.row_range[prow].y = c;
                    j.row_range[row].x = c;
                }
            }
        }
        if (at == b.n - 1) {  // the last point closes the last cell
            const bool mine = (heads[i] >> lane) & 1u;
            const int nc = c + (mine ? 1 : 0);
            b.counters[kCtrNcells + j.L] = (unsigned long long)nc;
            j.cell_start[nc] = b.n;
            j.row_range[k[i] >> bits].y = nc;
            pop = max(pop, mine ? 1u : (uint32_t)b.n + 1u - ph);
        }
        c0 += __popc(heads[i]);
        if (heads[i]) head = base + (31 - __clz(heads[i])) + 1u;
    }
    pop = __reduce_max_sync(0xffffffffu, pop);
    if (lane == 0) s_pop[w] = pop;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int u = 1; u < kT / 32; u++) pop = max(pop, s_pop[u]);
        if (pop) atomicMax(&b.counters[kCtrMaxPop + j.L], (unsigned long long)pop);
    }
}

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

// The level tables of h: one allocation, kept with the handle.
egt_status level_memory(egt_handle* h, int levels) {
    if (h->levels_built >= levels) return EGT_OK;
    const size_t n = (size_t)h->n;
    size_t total = 0;
    auto take = [&](size_t bytes) { const size_t at = total; total += align256(bytes); return at; };
    size_t rows[kMaxLevels], start[kMaxLevels], cx[kMaxLevels], order[kMaxLevels];
    for (int L = 0; L < levels; L++) rows[L] = take(sizeof(int2) * (size_t)(1024 >> L) * (1024 >> L));
    const size_t row_bytes = total;
    for (int L = 0; L < levels; L++) {
        start[L] = take(sizeof(int) * (n + 1));
        cx[L] = take(sizeof(int) * n);
        order[L] = L ? take(sizeof(int) * n) : 0;
    }
    dev_free(h, h->grid_mem);
    h->grid_mem = nullptr;
    EGT_CUDA_TRY(dev_alloc(h, &h->grid_mem, total));
    char* m = static_cast<char*>(h->grid_mem);
    h->row_bytes = row_bytes;
    for (int L = 0; L < levels; L++) {
        LevelDev& lv = h->lv[L];
        lv.B = 1024 >> L;
        lv.row_range = reinterpret_cast<int2*>(m + rows[L]);
        lv.cell_start = reinterpret_cast<int*>(m + start[L]);
        lv.cell_x = reinterpret_cast<int*>(m + cx[L]);
        lv.order = L ? reinterpret_cast<int*>(m + order[L]) : nullptr;
    }
    return EGT_OK;
}

}  // namespace

egt_status scratch_reserve(egt_handle* h, size_t bytes, void** out) {
    if (h->scratch.bytes < bytes) {
        if (h->scratch.ptr) {
            dev_free(h, h->scratch.ptr);  // stream-ordered: pending work keeps it until done
            h->scratch.ptr = nullptr;
            h->scratch.bytes = 0;
        }
        size_t want = bytes + bytes / 4 + 256;
        EGT_CUDA_TRY(dev_alloc(h, &h->scratch.ptr, want));
        h->scratch.bytes = want;
    }
    *out = h->scratch.ptr;
    return EGT_OK;
}

// Full grid build from device AoS xyz (n points).  levels = number of
// hierarchy levels to build (8 for point clouds, 1 for meshes).  Enqueued
// only: fetch_norm waits for it.
egt_status build_grid(egt_handle* h, const float* xyz, int levels) {
    const int64_t n = h->n;
    cudaStream_t st = h->stream;
    EGT_TRY(level_memory(h, levels));
    h->levels_built = levels;
    const int64_t tiles = radix_tiles(n), ttiles = (n + kTableTile - 1) / kTableTile;
    const bool library = n > kLibrarySort;
    const int group =
        library ? 1 : (int)std::max<int64_t>(1, std::min<int64_t>(kMaxLevels - 1, kGroupBytes / (16 * n)));
    // scratch: what starts at zero (digit counts, look-back words, tickets), then the sorts' buffers
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t a = at; at += align256(bytes); return a; };
    const size_t o_hist0 = take(sizeof(uint32_t) * (kL0Passes << kL0Bits));
    const size_t o_hist = take(sizeof(uint32_t) * (kLevelHists << kLevelBits));
    const size_t o_ticket = take(sizeof(uint32_t) * 64);
    size_t o_state0[kL0Passes], o_state[kMaxLevels][kMaxPasses], o_tstate[kMaxLevels];
    for (int p = 0; p < kL0Passes; p++) o_state0[p] = take(sizeof(uint32_t) * ((size_t)tiles << kL0Bits));
    for (int L = 1; L < levels; L++)
        for (int p = 0; p < level_passes(L); p++)
            o_state[L][p] = take(sizeof(uint32_t) * ((size_t)tiles << pass_bits(L, p)));
    for (int L = 0; L < levels; L++) o_tstate[L] = take(sizeof(unsigned long long) * ttiles);
    const size_t zero = at;
    const unsigned ge = (unsigned)std::min<int64_t>((n + 4 * kT - 1) / (4 * kT), 148 * 4);
    const size_t o_part = take(sizeof(float) * 6 * ge);
    const size_t o_key0 = take(sizeof(uint32_t) * n);
    const size_t o_buf = take(0), stride = align256(sizeof(uint32_t) * n);
    take(stride * 4 * group);
    size_t t_sort = 0;
    if (library)
        EGT_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, t_sort, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                                     (const int*)nullptr, (int*)nullptr, (int)n, 0, 30, st));
    const size_t o_sort = take(t_sort);
    void* mem = nullptr;
    EGT_TRY(scratch_reserve(h, at, &mem));
    char* m = static_cast<char*>(mem);
    auto U = [&](size_t o) { return reinterpret_cast<uint32_t*>(m + o); };
    auto buf = [&](int g, int which) { return m + o_buf + stride * (4 * g + which); };  // keys A, B, values A, B
    auto keys = [&](int g, int w) { return reinterpret_cast<uint32_t*>(buf(g, w)); };
    auto vals = [&](int g, int w) { return reinterpret_cast<int*>(buf(g, 2 + w)); };
    uint32_t* ticket = U(o_ticket);

    EGT_CUDA_TRY(cudaEventRecord(h->ev[0], st));
    EGT_CUDA_TRY(cudaMemsetAsync(m, 0, zero, st));
    EGT_CUDA_TRY(cudaMemsetAsync(h->grid_mem, 0, h->row_bytes, st));
    const int vec = (reinterpret_cast<uintptr_t>(xyz) & 15) == 0;
    k_extents<<<ge, kT, 0, st>>>(xyz, n, vec, h->cfg.eps, h->cfg.threshold, reinterpret_cast<float*>(m + o_part),
                                 ticket++, h->d_norm, h->d_counters);
    EGT_LAUNCH_CHECK();
    const unsigned gk = (unsigned)std::min<int64_t>((n + kT - 1) / kT, 148 * 8);
    EGT_TRY(launch_dependent(k_keys, dim3(gk), dim3(kT), 0, st, xyz, n, h->d_norm, keys(0, 0), U(o_hist0)));
    RadixBatch rb{};
    rb.n = (int)n;
    rb.polls = h->lookback_polls >= 0 ? h->lookback_polls : kRadixPolls;
    rb.recounts = h->d_counters + kCtrRecounts;
    // the digits from bit `from` on of keys sorted by the digits below (a large cloud)
    auto rest = [&](const uint32_t* key_in, uint32_t* key_out, const int* val_in, int* val_out, int from,
                    int to) -> egt_status {
        EGT_CUDA_TRY(cub::DeviceRadixSort::SortPairs(m + o_sort, t_sort, key_in, key_out, val_in, val_out, (int)n, from,
                                                     to, st));
        return EGT_OK;
    };
    for (int p = 0; p < (library ? 1 : kL0Passes); p++) {
        RadixJob& j = rb.job[0];
        j.key_in = keys(0, p & 1);
        j.val_in = p ? vals(0, p & 1) : nullptr;
        j.key_out = p + 1 < kL0Passes ? keys(0, (p & 1) ^ 1) : U(o_key0);
        j.val_out = p + 1 < kL0Passes ? vals(0, (p & 1) ^ 1) : h->perm;
        j.hist = U(o_hist0) + (p << kL0Bits);
        j.state = U(o_state0[p]);
        j.ticket = ticket++;
        j.shift = p * kL0Bits;
        j.bits = kL0Bits;
        j.xf = kKeyRaw;
        j.next_hist = p + 1 < kL0Passes && !library ? U(o_hist0) + ((p + 1) << kL0Bits) : nullptr;
        j.next_shift = j.shift + kL0Bits;
        j.next_bits = kL0Bits;
        EGT_TRY(radix_pass(rb, 1, st));
    }
    if (library) EGT_TRY(rest(keys(0, 1), U(o_key0), vals(0, 1), h->perm, kL0Bits, 30));
    EGT_TRY(launch_dependent(k_gather_sorted, dim3(gk), dim3(kT), 0, st, xyz, h->perm, U(o_key0), n, h->p4, h->x, h->y,
                             h->z, h->cell0, h->d_norm, levels > 1 ? U(o_hist) : nullptr));
    TableBatch tb{};
    tb.n = (int)n;
    tb.polls = rb.polls;
    tb.counters = h->d_counters;
    auto table = [&](int L, const uint32_t* key) {
        const LevelDev& lv = h->lv[L];
        return TableJob{key, lv.cell_start, lv.cell_x, lv.row_range,
                        reinterpret_cast<unsigned long long*>(m + o_tstate[L]), ticket++, L};
    };
    int tjobs = 0;
    tb.job[tjobs++] = table(0, U(o_key0));
    for (int L0 = 1; L0 < levels || tjobs; L0 += group) {
        const int L1 = std::min(levels, L0 + group);  // levels [L0, L1) are sorted together
        for (int p = 0; p < (library ? 1 : kMaxPasses); p++) {
            int jobs = 0;
            for (int L = L0; L < L1 && level_passes(L) > p; L++) {
                const int g = L - L0, last = library ? kMaxPasses : level_passes(L) - 1;  // the pass that ends in the tables
                RadixJob& j = rb.job[jobs++];
                // A, B, A...: a pass never writes what it reads
                j.key_in = p ? keys(g, (p - 1) & 1) : h->cell0;
                j.val_in = p ? vals(g, (p - 1) & 1) : nullptr;
                j.key_out = keys(g, p & 1);
                j.val_out = p == last ? h->lv[L].order : vals(g, p & 1);
                j.hist = U(o_hist) + ((size_t)hist_slot(L, p) << kLevelBits);
                j.state = U(o_state[L][p]);
                j.ticket = ticket++;
                j.shift = pass_shift(L, p);
                j.bits = pass_bits(L, p);
                j.xf = p ? kKeyRaw : L;
                j.next_hist = p < last && !library ? U(o_hist) + ((size_t)hist_slot(L, p + 1) << kLevelBits) : nullptr;
                j.next_shift = j.next_hist ? pass_shift(L, p + 1) : 0;
                j.next_bits = j.next_hist ? pass_bits(L, p + 1) : 0;
                if (p == last) tb.job[tjobs++] = table(L, keys(g, p & 1));
            }
            if (jobs) EGT_TRY(radix_pass(rb, jobs, st));
        }
        if (library && L0 < levels) {  // one level at a time
            EGT_TRY(rest(keys(0, 0), keys(0, 1), vals(0, 0), h->lv[L0].order, pass_bits(L0, 0), level_bits(L0)));
            tb.job[tjobs++] = table(L0, keys(0, 1));
        }
        EGT_TRY(launch_dependent(k_tables, dim3((unsigned)ttiles, (unsigned)tjobs), dim3(kT), 0, st, tb));
        tjobs = 0;
    }
    EGT_CUDA_TRY(cudaEventRecord(h->ev[1], st));
    return EGT_OK;
}

// The host's copy of the normalisation cube; waits for the grid build.
egt_status fetch_norm(egt_handle* h) {
    EGT_CUDA_TRY(cudaMemcpyAsync(&h->norm, h->d_norm, sizeof(NormParams), cudaMemcpyDeviceToHost, h->stream));
    EGT_CUDA_TRY(cudaStreamSynchronize(h->stream));
    return EGT_OK;
}

egt_status set_threshold(egt_handle* h, float thres) {
    k_set_thres<<<1, 1, 0, h->stream>>>(thres, h->d_norm);
    EGT_LAUNCH_CHECK();
    h->cfg.threshold = thres;
    return EGT_OK;
}

}  // namespace egt
