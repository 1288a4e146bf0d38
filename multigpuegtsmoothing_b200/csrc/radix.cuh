// Stable least-significant-digit radix passes over (key, value) pairs, for
// several sorts of the same n elements in one launch (the hierarchy levels of
// a grid).
//
// One pass reads every element once and writes it once.  A block takes a tile
// of consecutive elements, ranks them by digit (votes, and counters of each
// warp's own), gets the number of equal digits in the tiles before it
// by decoupled look-back (Merrill & Garland, "Single-pass Parallel Prefix Scan
// with Decoupled Look-back", 2016; one word per tile and digit holding a count
// and its state), reorders the tile by digit in shared memory and stores it in
// runs.  A pass needs the whole input's counts of its digit: the caller counts
// the first one while it forms what is sorted, and each pass counts the next
// one (counting all digits of the seven hierarchy levels beforehand took 89 us
// for 4M points: in the sorted order the upper digits of neighbours fall into
// one counter).
//
// Bound: the latency of a pass (load, rank, look-back, scatter): 7 us for 36K
// pairs, 45 us for 4M (1.4 TB/s) on their own, 42 us each when several sorts
// share a launch and fill one another's waits; from tens of millions of pairs on
// issue (55 to 65 % busy, DRAM a quarter of its peak; 1.6 TB/s).
//
// A look-back that waits too long (kRadixPolls) stops waiting: the block then
// counts the elements before its tile from the pass's input, which no block
// writes, so the pass ends with the same result whatever the other blocks do.
#pragma once
#include "egt_internal.cuh"

namespace egt {
namespace {

constexpr int kRadixThreads = 256;
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kRadixBits = 8;  // widest digit: one per thread
constexpr int kRadixBins = 1 << kRadixBits;
constexpr int kRadixJobs = 8;
constexpr int kRadixPolls = 1 << 20;     // look-back polls of one word before the tile counts for itself
constexpr uint32_t kStateSum = 1u << 30;   // the word holds the tile's own count
constexpr uint32_t kStateFull = 2u << 30;  // the word holds the count up to and including the tile
constexpr uint32_t kStateValue = kStateSum - 1;

// Key x + y*B + z*B^2 of the level-L cell of a packed level-0 cell.
__device__ __forceinline__ uint32_t level_key(uint32_t c, int L) {
    const int b = 10 - L;
    return ((c & 1023u) >> L) | ((((c >> 10) & 1023u) >> L) << b) | (((c >> 20) & 1023u) >> L) << (2 * b);
}

constexpr int kKeyRaw = -1;  // the keys themselves (1..7: packed level-0 cells, sorted by their level-L cell)

__device__ __forceinline__ uint32_t radix_key(uint32_t v, int xf) { return xf == kKeyRaw ? v : level_key(v, xf); }

struct RadixJob {
    const uint32_t* key_in;  // keys, or what they are formed from (xf)
    const int* val_in;       // nullptr: 0 .. n-1
    uint32_t* key_out;
    int* val_out;
    const uint32_t* hist;    // [1 << bits] elements per digit
    uint32_t* next_hist;     // the next pass's, zero (nullptr: the last pass)
    uint32_t* state;         // [tiles << bits], zero
    uint32_t* ticket;        // zero
    int shift, bits, xf;
    int next_shift, next_bits;
};
struct RadixBatch {
    RadixJob job[kRadixJobs];
    int n;
    int polls;                    // kRadixPolls
    unsigned long long* recounts;  // tiles that counted for themselves
};

// Exclusive prefix of one value per thread over the block.  s: kRadixWarps
// words of shared memory.
__device__ __forceinline__ uint32_t radix_block_prefix(uint32_t v, uint32_t* s) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) s[w] = incl;
    __syncthreads();
    uint32_t before = 0;
#pragma unroll
    for (int i = 0; i < kRadixWarps; i++) before += i < w ? s[i] : 0u;
    return before + incl - v;
}

__device__ __forceinline__ uint32_t load_state(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_state(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Lanes that hold the same digit (valid lanes only), by one vote per bit.  (The
// match instruction instead: 75 us for a pass over 4M pairs, against 45.)
__device__ __forceinline__ unsigned radix_peers(uint32_t d, bool valid) {
    unsigned m = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int i = 0; i < kRadixBits; i++) {
        const unsigned v = __ballot_sync(0xffffffffu, (d >> i) & 1u);
        m &= ((d >> i) & 1u) ? v : ~v;
    }
    return m;
}

// One pass of job blockIdx.y.
template <int ITEMS>
__global__ void __launch_bounds__(kRadixThreads, 4) k_radix_pass(const __grid_constant__ RadixBatch b) {
    constexpr int kTile = kRadixThreads * ITEMS;
    __shared__ uint16_t s_cnt[kRadixWarps][kRadixBins];  // digits seen by each warp, then the warps' offsets
    __shared__ uint32_t s_key[kTile];
    __shared__ int s_val[kTile];
    __shared__ uint32_t s_off[kRadixBins];  // first slot of each digit in the tile, then its place in the output
    __shared__ uint32_t s_next[kRadixBins];  // the tile's counts of the next pass's digit
    __shared__ uint32_t s_scan[kRadixWarps];
    __shared__ uint32_t s_tile;
    grid_dependency_wait();
    grid_dependents_launch();
    const RadixJob& j = b.job[blockIdx.y];
    const int n = b.n;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t mask = (1u << j.bits) - 1u;
    const int shift = j.shift, xf = j.xf;
    // tiles in the order in which blocks start, so that a tile's predecessors are running or done
    if (threadIdx.x == 0) s_tile = atomicAdd(j.ticket, 1u);
    for (int i = threadIdx.x; i < kRadixWarps * kRadixBins / 2; i += kRadixThreads)
        reinterpret_cast<uint32_t*>(&s_cnt[0][0])[i] = 0u;
    s_next[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t first = (int64_t)tile * kTile;
    const int count = (int)min((int64_t)kTile, n - first);
    const int at0 = w * 32 * ITEMS + lane;  // the thread's elements: at0, at0 + 32, ...
    uint32_t key[ITEMS];
    uint32_t rank[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; i++)
        key[i] = at0 + 32 * i < count ? radix_key(j.key_in[first + at0 + 32 * i], xf) : 0u;
    if (j.next_hist) {
        const uint32_t next_mask = (1u << j.next_bits) - 1u;
#pragma unroll
        for (int i = 0; i < ITEMS; i++)
            if (at0 + 32 * i < count) atomicAdd(&s_next[(key[i] >> j.next_shift) & next_mask], 1u);
    }
    // rank of each element among the warp's elements of its digit
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        const bool valid = at0 + 32 * i < count;
        const uint32_t d = (key[i] >> shift) & mask;
        const unsigned peers = radix_peers(d, valid);
        const uint32_t before = s_cnt[w][d];
        rank[i] = before + __popc(peers & ((1u << lane) - 1u));
        __syncwarp();
        if (valid && (peers >> lane) == 1u) s_cnt[w][d] = (uint16_t)(rank[i] + 1);  // the last of its peers
        __syncwarp();
    }
    __syncthreads();
    // thread d: digit d's offsets per warp, count and first place in the output
    const int d = (int)threadIdx.x;
    const bool used = d <= (int)mask;
    uint32_t tot = 0;
#pragma unroll
    for (int u = 0; u < kRadixWarps; u++) {
        const uint32_t c = s_cnt[u][d];
        s_cnt[u][d] = (uint16_t)tot;
        tot += c;
    }
    uint32_t* state = j.state + d;
    if (used) store_state(state + ((size_t)tile << j.bits), (tile ? kStateSum : kStateFull) | tot);
    if (j.next_hist && s_next[d]) atomicAdd(&j.next_hist[d], s_next[d]);
    const uint32_t whole = used ? j.hist[d] : 0u;
    const uint32_t slot = radix_block_prefix(tot, s_scan);
    const uint32_t base = radix_block_prefix(whole, s_scan);
    s_off[d] = slot;
    __syncthreads();
    // the tile by digit, in shared memory
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        if (at0 + 32 * i < count) {
            const uint32_t e = (key[i] >> shift) & mask;
            const uint32_t to = rank[i] + s_off[e] + s_cnt[w][e];
            s_key[to] = key[i];
            s_val[to] = j.val_in ? j.val_in[first + at0 + 32 * i] : (int)(first + at0 + 32 * i);
        }
    }
    // Look back: equal digits in the tiles before this one.  kAhead words are
    // in flight: a wave of blocks that start together walks back over one
    // another, and the walk's length is what a pass of a few million elements
    // waits for.
    uint32_t prev = 0;
    bool lost = false;
    if (used) {
        constexpr int kAhead = 16;
        bool full = false;
        for (int t = (int)tile - 1; t >= 0 && !lost && !full; t -= kAhead) {
            uint32_t s[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; u++)
                s[u] = t >= u ? load_state(state + ((size_t)(t - u) << j.bits)) : kStateFull;
#pragma unroll
            for (int u = 0; u < kAhead; u++) {
                if (full || lost) continue;
                for (int tries = 0; s[u] == 0u && tries < b.polls; tries++)
                    s[u] = load_state(state + ((size_t)(t - u) << j.bits));
                lost = s[u] == 0u;
                prev += s[u] & kStateValue;
                full = s[u] & kStateFull;
            }
        }
    }
    if (__syncthreads_or(lost)) {  // a predecessor did not answer: count its elements here
        if (d == 0) atomicAdd(b.recounts, 1ull);
        uint32_t* all = reinterpret_cast<uint32_t*>(&s_cnt[0][0]);
        all[d] = 0u;
        __syncthreads();
        for (int64_t i = threadIdx.x; i < first; i += kRadixThreads)
            atomicAdd(&all[(radix_key(j.key_in[i], xf) >> shift) & mask], 1u);
        __syncthreads();
        prev = all[d];
    }
    if (used && tile) store_state(state + ((size_t)tile << j.bits), kStateFull | (prev + tot));
    s_off[d] = base + prev - slot;  // output place of the digit's elements, less their slot (mod 2^32)
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += kRadixThreads) {
        const uint32_t k = s_key[i];
        const uint32_t to = s_off[(k >> shift) & mask] + (uint32_t)i;
        j.key_out[to] = k;
        j.val_out[to] = s_val[i];
    }
}

// Elements per thread: four while the tiles do not fill the chip, else twelve
// (registers: sixteen spill at four blocks per SM; grid build of 4M points 1.39
// ms with 12, 1.43 with 8).
constexpr int kRadixSmall = 4, kRadixLarge = 12;
inline int radix_items(int64_t n) { return n <= 262144 ? kRadixSmall : kRadixLarge; }
inline int64_t radix_tiles(int64_t n) {
    const int64_t t = (int64_t)kRadixThreads * radix_items(n);
    return (n + t - 1) / t;
}

// One pass of the first `jobs` jobs of b.
inline egt_status radix_pass(const RadixBatch& b, int jobs, cudaStream_t st) {
    const dim3 g((unsigned)radix_tiles(b.n), (unsigned)jobs);
    if (radix_items(b.n) == kRadixSmall)
        return launch_dependent(k_radix_pass<kRadixSmall>, g, dim3(kRadixThreads), 0, st, b);
    return launch_dependent(k_radix_pass<kRadixLarge>, g, dim3(kRadixThreads), 0, st, b);
}

}  // namespace
}  // namespace egt
