// Normal orientation over a minimum spanning forest.
//
// Reference: Normal_CUDA::GetNormals (Normal_CUDA.cu:329-711) with CUDA_MST.cu
// (Borůvka, :296-418) and bfs.cu (level-synchronous BFS with a host loop per
// level, :63-110).  The reference builds undirected edges (min,max) from the
// filtered lists with weight max(0, 1 - |n_u . n_v|), removes duplicates by the
// key u*n+v, sorts by weight (stable, so ties stay in key order), takes a
// minimum spanning forest and walks each tree breadth-first from a root,
// negating a child's normal when its dot product with its parent's (already
// oriented) normal is negative.  The first root is the first vertex of the
// lightest edge (Normal_CUDA.cu:438-440).
//
// Along a tree path the BFS rule makes the sign of every vertex a product of
// the edge signs sign(n_u . n_v) from the root, so no traversal order is
// needed: this file runs a deterministic Borůvka that carries that sign parity
// through its component merges (each vertex stores its sign relative to its
// component representative, merged by pointer jumping), then re-bases every
// tree on its root.  Edges are totally ordered by (weight, key) -- the
// reference's sort order -- so the forest is the unique minimum one for that
// order.  Every tree is rooted at the first vertex of its lightest edge (for
// the first tree this is the reference's root; the reference picks later roots
// by a racy last-writer search, Normal_CUDA.cu:232-240).  An exactly zero dot
// product is treated as a same-sign link (the reference re-seeds the child from
// its raw sign there).  Component sign votes (Normal_CUDA.cu:517-711) only act
// on list edges that join different trees; the trees are the connected
// components of the list graph, so there are none to act on.
//
// The host waits once per few rounds (kRoundsPerSync): every kernel of a round
// reads its sizes from the device, and ends at once when nothing is left.
#include <cub/cub.cuh>
#include <numeric>
#include <vector>
#include "egt_internal.cuh"
#include "radix.cuh"

namespace egt {
namespace {

constexpr unsigned long long kNone = ~0ull;

constexpr int kTB = 256;  // threads per block

// Block-aggregated counter increment.  Every thread of the block must call it
// (pred false for threads without an item).
__device__ __forceinline__ void block_count(unsigned long long* ctr, bool pred) {
    const int c = __syncthreads_count(pred);
    if (threadIdx.x == 0 && c) atomicAdd(ctr, (unsigned long long)c);
}

// ---- the undirected edges of the lists, in key order ----
// Every edge {u, v}, u < v, belongs to the bucket of u.  Row u's own entries
// above u go there directly; an entry u of a row v > u only if row u does not
// list v (most do, so few entries need an atomic).  A bucket is then ordered
// by v and repeated entries dropped, which puts the edges in (u, v) order: the
// reference's key order, without sorting 64-bit keys (1M points, 16M list entries:
// 1.03 ms with a radix sort).  The order comes from counting, quadratic in a
// bucket, whose length is the rows that list u; buckets of more than kLongBucket
// entries (equal points all list the same few of them) are sorted first.

constexpr int kRowLanes = 16;  // lanes per row
constexpr int kLongBucket = 1024;

// keep[e]: 1 = bucket of its own row, 2 = bucket of the other end.  own[i]:
// entries of kind 1; cnt[u]: entries of bucket u (zero before).
__global__ void __launch_bounds__(kTB) k_bucket_count(const int* __restrict__ off, const int* __restrict__ col, int n,
                                                      unsigned char* __restrict__ keep, int* __restrict__ own,
                                                      int* __restrict__ cnt) {
    const int i = (int)((blockIdx.x * (int64_t)kTB + threadIdx.x) / kRowLanes);
    const int l = threadIdx.x & (kRowLanes - 1);
    const int e0 = i < n ? off[i] : 0, e1 = i < n ? off[i + 1] : 0;
    int mine = 0;
    for (int e = e0 + l; e < e1; e += kRowLanes) {
        const int m = col[e];
        unsigned char kind = 0;
        if (m > i) {
            kind = 1;
            mine++;
        } else if (m < i) {
            const int f0 = off[m], f1 = off[m + 1];
            kind = 2;
            for (int f = f0; f < f1; f++)
                if (col[f] == i) { kind = 0; break; }
            if (kind) atomicAdd(&cnt[m], 1);
        }
        keep[e] = kind;
    }
#pragma unroll
    for (int o = kRowLanes / 2; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if (l == 0 && i < n) {
        own[i] = mine;
        if (mine) atomicAdd(&cnt[i], mine);
    }
}

// Fills the buckets (boff: their starts).  own[u] becomes bucket u's next free
// place after its own row's entries.  longs [*n_long]: the buckets to sort.
__global__ void __launch_bounds__(kTB) k_bucket_fill(const int* __restrict__ off, const int* __restrict__ col, int n,
                                                     int bits, const unsigned char* __restrict__ keep,
                                                     const int* __restrict__ boff, int* __restrict__ own,
                                                     unsigned long long* __restrict__ key, int* __restrict__ longs,
                                                     int* __restrict__ n_long) {
    const int i = (int)((blockIdx.x * (int64_t)kTB + threadIdx.x) / kRowLanes);
    const int l = threadIdx.x & (kRowLanes - 1);
    const int e0 = i < n ? off[i] : 0, e1 = i < n ? off[i + 1] : 0;
    const unsigned gmask = 0xffffu << (threadIdx.x & 16);
    int at = i < n ? boff[i] : 0;
    if (l == 0 && i < n && boff[i + 1] - at > kLongBucket) longs[atomicAdd(n_long, 1)] = i;
    const int rounds = (e1 - e0 + kRowLanes - 1) / kRowLanes;
    for (int r = 0; r < rounds; r++) {  // uniform over the row's lanes
        const int e = e0 + r * kRowLanes + l;
        const int kind = e < e1 ? keep[e] : 0;
        const unsigned b = __ballot_sync(gmask, kind == 1) & gmask;
        if (kind) {
            const int m = col[e];
            if (kind == 1) {
                key[at + __popc(b & ((1u << (threadIdx.x & 31)) - 1u))] = ((unsigned long long)i << bits) | (unsigned)m;
            } else {
                key[boff[m] + atomicAdd(&own[m], 1)] = ((unsigned long long)m << bits) | (unsigned)i;
            }
        }
        at += __popc(b);
    }
}

// Sorts the long buckets by v, a block per bucket: least-significant-digit passes
// between key and tmp (the same places), digits of 8 bits, the last pass ending in
// key.  A pass takes the bucket in chunks and keeps each digit's next place.
// 200,000 points, 50,000 of them equal, orientation: k = 16 23.1 ms by counting
// alone, 2.0 with a sort of all keys, 0.99 so; k = 40 54.5, 3.5 and 1.44.
constexpr int kSortItems = 8;
__global__ void __launch_bounds__(kRadixThreads) k_bucket_sort(unsigned long long* key, unsigned long long* tmp,
                                                               const int* __restrict__ boff,
                                                               const int* __restrict__ longs,
                                                               const int* __restrict__ n_long, int bits) {
    __shared__ uint16_t s_cnt[kRadixWarps][kRadixBins];  // digits seen by each warp, then the warps' offsets
    __shared__ uint32_t s_next[kRadixBins];              // next place of each digit
    __shared__ uint32_t s_scan[kRadixWarps];
    constexpr int kChunk = kRadixThreads * kSortItems;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, d = threadIdx.x;
    for (int b = blockIdx.x; b < *n_long; b += gridDim.x) {
        const int b0 = boff[longs[b]], m = boff[longs[b] + 1] - b0;
        unsigned long long *src = key + b0, *dst = tmp + b0;
        for (int shift = 0; shift < bits; shift += kRadixBits) {
            s_next[d] = 0u;
            __syncthreads();
            for (int i = threadIdx.x; i < m; i += kRadixThreads)
                atomicAdd(&s_next[(uint32_t)(src[i] >> shift) & (kRadixBins - 1u)], 1u);
            __syncthreads();
            const uint32_t base = radix_block_prefix(s_next[d], s_scan);
            s_next[d] = base;
            for (int c0 = 0; c0 < m; c0 += kChunk) {
                for (int i = threadIdx.x; i < kRadixWarps * kRadixBins / 2; i += kRadixThreads)
                    reinterpret_cast<uint32_t*>(&s_cnt[0][0])[i] = 0u;
                __syncthreads();
                unsigned long long k[kSortItems];
                uint32_t rank[kSortItems];
                const int at0 = c0 + w * 32 * kSortItems + lane;
#pragma unroll
                for (int i = 0; i < kSortItems; i++) k[i] = at0 + 32 * i < m ? src[at0 + 32 * i] : 0ull;
#pragma unroll
                for (int i = 0; i < kSortItems; i++) {
                    const bool valid = at0 + 32 * i < m;
                    const uint32_t e = (uint32_t)(k[i] >> shift) & (kRadixBins - 1u);
                    const unsigned peers = radix_peers(e, valid);
                    rank[i] = s_cnt[w][e] + __popc(peers & ((1u << lane) - 1u));
                    __syncwarp();
                    if (valid && (peers >> lane) == 1u) s_cnt[w][e] = (uint16_t)(rank[i] + 1);  // the last of its peers
                    __syncwarp();
                }
                __syncthreads();
                uint32_t tot = 0;
#pragma unroll
                for (int u = 0; u < kRadixWarps; u++) {
                    const uint32_t c = s_cnt[u][d];
                    s_cnt[u][d] = (uint16_t)tot;
                    tot += c;
                }
                __syncthreads();
#pragma unroll
                for (int i = 0; i < kSortItems; i++) {
                    const uint32_t e = (uint32_t)(k[i] >> shift) & (kRadixBins - 1u);
                    if (at0 + 32 * i < m) dst[s_next[e] + s_cnt[w][e] + rank[i]] = k[i];
                }
                __syncthreads();
                s_next[d] += tot;
            }
            __syncthreads();  // the pass is written before the next one reads it
            unsigned long long* t = src;
            src = dst;
            dst = t;
        }
        if (src != key + b0)
            for (int i = threadIdx.x; i < m; i += kRadixThreads) dst[i] = src[i];
        __syncthreads();
    }
}

// Orders every bucket and gives its edges their places: ukey[p] the edge at
// place p, act[p] its order key (weight bits, p) -- p grows with the vertex key,
// so this is the reference's (weight, key) order -- and sgn[p] the sign of its
// dot product.  The place of a repeated entry stays empty (kNone).
__global__ void __launch_bounds__(kTB) k_bucket_edges(const unsigned long long* __restrict__ key,
                                                      const int* __restrict__ boff, int n, int bits,
                                                      const float* __restrict__ nrm,
                                                      unsigned long long* __restrict__ ukey,
                                                      unsigned long long* __restrict__ act,
                                                      signed char* __restrict__ sgn) {
    const int64_t e = blockIdx.x * (int64_t)kTB + threadIdx.x;
    if (e >= boff[n]) return;
    const unsigned long long k = key[e];
    const int u = (int)(k >> bits), v = (int)(k & ((1ull << bits) - 1ull));
    const int b0 = boff[u], b1 = boff[u + 1];
    int p = b0;
    bool again = false;
    if (b1 - b0 > kLongBucket) {  // sorted (k_bucket_sort)
        p = (int)e;
        again = e > b0 && key[e - 1] == k;
    } else {
        for (int f = b0; f < b1; f++) {
            const unsigned long long o = key[f];
            p += (o < k || (o == k && f < e)) ? 1 : 0;
            again |= o == k && f < e;
        }
    }
    ukey[p] = k;
    if (again) { act[p] = kNone; return; }
    const float d = fs_dot3(nrm[u], nrm[n + u], nrm[2 * (size_t)n + u], nrm[v], nrm[n + v], nrm[2 * (size_t)n + v]);
    const float w = fmaxf(0.0f, __fsub_rn(1.0f, fabsf(d)));
    act[p] = ((unsigned long long)__float_as_uint(w) << 32) | (unsigned)p;
    sgn[p] = d < 0.0f ? -1 : 1;
}

// 1 for the first copy of each edge key in the sorted array (self-loop
// sentinels excluded).
__global__ void k_first_copy(const unsigned long long* __restrict__ key, int64_t m, int bits,
                             unsigned char* __restrict__ flag) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= m) return;
    const unsigned long long k = key[e];
    flag[e] = (k != (1ull << (2 * bits)) - 1ull) && (e == 0 || key[e - 1] != k);
}

// State of a forest computation on the device.
struct ForestState {
    int live[2];               // edges of the two edge lists
    unsigned long long linked;  // links of the last round
};

__global__ void k_init_comp(int n, const int* __restrict__ edges, int max_edges, int* __restrict__ comp,
                            signed char* __restrict__ sig, unsigned long long* __restrict__ best,
                            ForestState* __restrict__ fs) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v == 0) {
        fs->live[0] = edges ? *edges : max_edges;
        fs->live[1] = 0;
        fs->linked = 0;
    }
    if (v >= n) return;
    comp[v] = v;
    sig[v] = 1;
    best[v] = kNone;
}

// Lightest live edge of every component.  in: the edges that joined two
// components when the last round began; those that still do are copied to out,
// so dead edges are read once more and no pass of its own drops them.  Most
// edges are not lighter than what their component has seen, which a read
// tells without an atomic (1M points, 9M edges, first round: 245 us with two
// atomics per edge).  One count atomic per block.
constexpr int kSelItems = 8;
__global__ void __launch_bounds__(kTB) k_select(const unsigned long long* __restrict__ in,
                                                unsigned long long* __restrict__ out, int side,
                                                const unsigned long long* __restrict__ ukey, int bits,
                                                const int* __restrict__ comp, unsigned long long* best,
                                                ForestState* __restrict__ fs) {
    __shared__ int s_cnt[kTB / 32], s_base;
    const int live = fs->live[side];
    if (blockIdx.x == 0 && threadIdx.x == 0) fs->linked = 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int64_t i0 = (int64_t)blockIdx.x * kTB * kSelItems; i0 < live; i0 += (int64_t)gridDim.x * kTB * kSelItems) {
        unsigned long long c[kSelItems];
        unsigned mask[kSelItems];
        int cnt = 0;
#pragma unroll
        for (int j = 0; j < kSelItems; j++) {
            const int64_t i = i0 + j * kTB + threadIdx.x;
            c[j] = i < live ? in[i] : kNone;
        }
#pragma unroll
        for (int j = 0; j < kSelItems; j++) {
            bool joins = false;
            if (c[j] != kNone) {
                const unsigned long long k = ukey[c[j] & 0xffffffffull];
                const int cu = comp[(int)(k >> bits)], cv = comp[(int)(k & ((1ull << bits) - 1ull))];
                joins = cu != cv;
                if (joins) {
                    if (c[j] < *(volatile unsigned long long*)&best[cu]) atomicMin(&best[cu], c[j]);
                    if (c[j] < *(volatile unsigned long long*)&best[cv]) atomicMin(&best[cv], c[j]);
                }
            }
            mask[j] = __ballot_sync(0xffffffffu, joins);
            cnt += __popc(mask[j]);
        }
        if (lane == 0) s_cnt[w] = cnt;
        __syncthreads();
        if (threadIdx.x == 0) {
            int total = 0;
            for (int u = 0; u < kTB / 32; u++) { const int t = s_cnt[u]; s_cnt[u] = total; total += t; }
            s_base = total ? atomicAdd(&fs->live[side ^ 1], total) : 0;
        }
        __syncthreads();
        int at = s_base + s_cnt[w];
#pragma unroll
        for (int j = 0; j < kSelItems; j++) {
            if ((mask[j] >> lane) & 1u) out[at + __popc(mask[j] & ((1u << lane) - 1u))] = c[j];
            at += __popc(mask[j]);
        }
        __syncthreads();
    }
}

// Hooks every component to the one across its lightest edge: link[c] = (that
// component << 1) | (1 when the signs across differ); a root links to itself.
// A pair that chose each other links only the larger representative.  Counts
// the links (= forest edges added).  first (optional): the round's choices.
__global__ void __launch_bounds__(kTB) k_hook(const unsigned long long* __restrict__ ukey,
                                              const signed char* __restrict__ sgn, int n, int bits, int side,
                                              const int* __restrict__ comp, const signed char* __restrict__ sig,
                                              const unsigned long long* __restrict__ best, unsigned* __restrict__ link,
                                              unsigned long long* __restrict__ first, ForestState* __restrict__ fs,
                                              unsigned long long* __restrict__ ctr, unsigned char* __restrict__ msf) {
    const int c = blockIdx.x * kTB + threadIdx.x;
    bool linked = false;
    if (c == 0) fs->live[side] = 0;  // the list this round read: the next round's output
    if (c < n) {
        const unsigned long long b = comp[c] == c ? best[c] : kNone;
        if (first) first[c] = b;
        unsigned to = (unsigned)c << 1;
        if (b != kNone) {
            const int e = (int)(b & 0xffffffffull);
            const unsigned long long k = ukey[e];
            const int u = (int)(k >> bits), v = (int)(k & ((1ull << bits) - 1ull));
            const int x = comp[u] == c ? u : v;
            const int y = x == u ? v : u;
            const int c2 = comp[y];
            if (!(best[c2] == b && c < c2)) {  // mutual choice: the smaller representative stays a root
                to = ((unsigned)c2 << 1) | (sig[x] * sgn[e] * sig[y] < 0 ? 1u : 0u);
                linked = true;
                if (msf) msf[e] = 1;
            }
        }
        link[c] = to;
    }
    const int t = __syncthreads_count(linked);
    if (threadIdx.x == 0 && t) {
        atomicAdd(&fs->linked, (unsigned long long)t);
        atomicAdd(&ctr[kCtrMsf], (unsigned long long)t);
    }
}

// Shortens the link chains in place: a component follows the links it finds,
// which other threads shorten meanwhile (target and sign are one word, and
// every word is a true path of its component, old or new).
constexpr int kJumps = 32;
__global__ void __launch_bounds__(kTB) k_jump(unsigned* link, int n, const int* __restrict__ comp,
                                              const ForestState* __restrict__ fs) {
    const int c = blockIdx.x * kTB + threadIdx.x;
    if (c >= n || fs->linked == 0 || comp[c] != c) return;
    unsigned w = link[c];
    for (int it = 0; it < kJumps; it++) {
        const unsigned l = w >> 1;
        const unsigned wl = *(volatile unsigned*)&link[l];
        if ((wl >> 1) == l) break;
        w = (wl & ~1u) | ((w ^ wl) & 1u);
        *(volatile unsigned*)&link[c] = w;
    }
}

// Every vertex to its component's root (the rest of a chain that k_jump did
// not finish is followed here).
__global__ void __launch_bounds__(kTB) k_relabel(int n, const unsigned* __restrict__ link, int* __restrict__ comp,
                                                 signed char* __restrict__ sig, unsigned long long* __restrict__ best,
                                                 const ForestState* __restrict__ fs) {
    const int v = blockIdx.x * kTB + threadIdx.x;
    if (v >= n || fs->linked == 0) return;
    unsigned w = link[comp[v]];
    for (;;) {
        const unsigned wl = link[w >> 1];
        if ((wl >> 1) == (w >> 1)) break;
        w = (wl & ~1u) | ((w ^ wl) & 1u);
    }
    comp[v] = (int)(w >> 1);
    if (w & 1u) sig[v] = (signed char)-sig[v];
    best[v] = kNone;
}

// Lightest edge of every tree.  It is the lightest edge at one of its ends, so
// it is the minimum of the first round's choices (first) over the tree's
// vertices.  Lanes of a warp that share a tree combine before the atomic.
__global__ void k_roots(int n, const int* __restrict__ comp, const unsigned long long* __restrict__ first,
                        unsigned long long* __restrict__ rootkey) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = v < n ? comp[v] : -1;
    unsigned long long b = v < n ? first[v] : kNone;
    if (__match_any_sync(0xffffffffu, c) == 0xffffffffu) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long t = __shfl_xor_sync(0xffffffffu, b, o);
            b = t < b ? t : b;
        }
        if ((threadIdx.x & 31) == 0 && c >= 0 && b != kNone) atomicMin(&rootkey[c], b);
    } else if (c >= 0 && b != kNone) {
        atomicMin(&rootkey[c], b);
    }
}

__global__ void k_apply(int n, int bits, const int* __restrict__ comp, const signed char* __restrict__ sig,
                        const unsigned long long* __restrict__ rootkey, const unsigned long long* __restrict__ ukey,
                        float* __restrict__ nrm, unsigned long long* __restrict__ ctr) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    bool root = false;
    if (v < n) {
        const int c = comp[v];
        const unsigned long long rk = rootkey[c];
        if (rk != kNone) {  // else: no edge, keeps its unoriented normal
            const int e = (int)(rk & 0xffffffffull);
            const int R = (int)(ukey[e] >> bits);
            root = v == c;
            if (sig[v] * sig[R] < 0) {
                nrm[v] = -nrm[v];
                nrm[n + v] = -nrm[n + v];
                nrm[2 * (size_t)n + v] = -nrm[2 * (size_t)n + v];
            }
        }
    }
    block_count(&ctr[kCtrComps], root);
}

// ---- orient_kruskal (MST.cpp:399-423): the reference's CPU orienter ----

// Vertex keys (min << bits | max) of the first k_use entries of every row
// (rows of k ints); empty entries (< 0) and self pairs get the sentinel
// that sorts last.  An entry >= n sets ctr[kCtrFlag].
__global__ void k_kr_keys(const int* __restrict__ knn, int n, int k, int k_use, int bits,
                          unsigned long long* __restrict__ key, unsigned long long* __restrict__ ctr) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)n * k_use) return;
    const int i = (int)(t / k_use);
    const int m = knn[(int64_t)i * k + (int)(t - (int64_t)i * k_use)];
    const unsigned long long sentinel = (1ull << (2 * bits)) - 1ull;
    if (m >= n) {
        ctr[kCtrFlag] = 1;
        key[t] = sentinel;
        return;
    }
    if (m < 0 || m == i) { key[t] = sentinel; return; }
    const unsigned u = (unsigned)min(i, m), v = (unsigned)max(i, m);
    key[t] = ((unsigned long long)u << bits) | v;
}

// Edge weight max(0, 1 - |d|) in double, d the float dot product
// nx_u*nx_v + ny_u*ny_v + nz_u*nz_v summed left to right with every product
// and sum rounded separately (the reference's host arithmetic, MST.cpp:408-409);
// the weight's bit pattern orders like the weight (it is never negative).
// sgn = -1 for d < 0; zero = 1 for d == 0.
__global__ void k_kr_weights(const unsigned long long* __restrict__ ukey, int E, int bits, const float* __restrict__ nrm,
                             int n, unsigned long long* __restrict__ wkey, int* __restrict__ eidx,
                             signed char* __restrict__ sgn, unsigned char* __restrict__ zero) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    const unsigned long long k = ukey[e];
    const int u = (int)(k >> bits), v = (int)(k & ((1ull << bits) - 1ull));
    const float* X = nrm;
    const float* Y = nrm + n;
    const float* Z = nrm + 2 * (size_t)n;
    const float d = __fadd_rn(__fadd_rn(__fmul_rn(X[u], X[v]), __fmul_rn(Y[u], Y[v])), __fmul_rn(Z[u], Z[v]));
    const double w1 = __dsub_rn(1.0, fabs((double)d));
    const double w = w1 > 0.0 ? w1 : 0.0;  // std::max(0.0, w1): +0 for -0 and NaN
    wkey[e] = (unsigned long long)__double_as_longlong(w);
    eidx[e] = e;
    sgn[e] = d < 0.0f ? -1 : 1;
    zero[e] = d == 0.0f;
}

// Order keys (rank << 32 | edge) from the edges sorted by (weight, u, v).
__global__ void k_kr_rank(const int* __restrict__ order, int E, unsigned long long* __restrict__ act) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= E) return;
    act[r] = ((unsigned long long)r << 32) | (unsigned)order[r];
}

// Per rank: the edge's vertex key, and flags for forest edges (f1), forest
// edges with a non-zero dot product (f2, with their order keys in okey) and
// forest edges with a zero dot product (f3).
__global__ void k_kr_forest_lists(const int* __restrict__ order, int E, const unsigned long long* __restrict__ ukey,
                                  const unsigned char* __restrict__ msf, const unsigned char* __restrict__ zero,
                                  unsigned long long* __restrict__ vkey, unsigned long long* __restrict__ okey,
                                  unsigned char* __restrict__ f1, unsigned char* __restrict__ f2,
                                  unsigned char* __restrict__ f3) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= E) return;
    const int e = order[r];
    vkey[r] = ukey[e];
    okey[r] = ((unsigned long long)r << 32) | (unsigned)e;
    const bool in = msf[e] != 0;
    f1[r] = in;
    f2[r] = in && !zero[e];
    f3[r] = in && zero[e];
}

// ref[comp[s]] = s for every walk start s (one per component of comp).
__global__ void k_kr_starts(const int* __restrict__ starts, int ns, const int* __restrict__ comp,
                            int* __restrict__ ref) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ns) return;
    const int s = starts[i];
    ref[comp[s]] = s;
}

// Final signs: s_v = sig[v] * sig[r], r = ref[comp[v]] the vertex whose sign
// the reference's walk leaves unchanged at the start of v's part of the tree.
__global__ void k_kr_apply(int n, const int* __restrict__ comp, const int* __restrict__ ref,
                           const signed char* __restrict__ sig, float* __restrict__ nrm) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    if (sig[v] * sig[ref[comp[v]]] < 0) {
        nrm[v] = -nrm[v];
        nrm[n + v] = -nrm[n + v];
        nrm[2 * (size_t)n + v] = -nrm[2 * (size_t)n + v];
    }
}

// Device buffers of one spanning-forest computation over n vertices.
struct Forest {
    int* comp = nullptr;
    unsigned* link = nullptr;
    signed char* sig = nullptr;
    unsigned long long* best = nullptr;
    unsigned long long* first = nullptr;
    ForestState* state = nullptr;

    cudaError_t alloc(int n, cudaStream_t st) {
        cudaError_t e = cudaSuccess;
        auto A = [&](auto** p, size_t bytes) {
            if (e == cudaSuccess) e = cudaMallocAsync((void**)p, bytes, st);
        };
        A(&comp, sizeof(int) * n); A(&link, sizeof(unsigned) * n); A(&sig, n);
        A(&best, sizeof(unsigned long long) * n); A(&first, sizeof(unsigned long long) * n);
        A(&state, sizeof(ForestState));
        return e;
    }
    void release(cudaStream_t st) {
        for (void* p : {(void*)comp, (void*)link, (void*)sig, (void*)best, (void*)first, (void*)state})
            if (p) cudaFreeAsync(p, st);
    }
};

constexpr int kRoundsPerSync = 4;

// Borůvka minimum spanning forest with sign parity.  act[0..E): order keys
// (rank << 32 | edge; kNone: no edge), the low half indexing ukey (u << bits |
// v) and sgn (+-1); edges (optional): their number on the device, at most E.
// act and act2 (E entries) take turns as the list of edges between components.
// On return f.comp[v] is v's component representative, f.sig[v] the product of
// the edge signs on the forest path from the representative to v, and
// f.first[v] the order key of v's lightest edge.  msf (optional): msf[edge] =
// 1 for every forest edge.  ctr: device counters (kCtrMsf is used).
egt_status spanning_forest(int n, int E, int bits, const unsigned long long* ukey, unsigned long long* act,
                           unsigned long long* act2, const int* edges, const signed char* sgn,
                           unsigned long long* ctr, Forest& f, unsigned char* msf, cudaStream_t st) {
    auto G = [&](int64_t m) { return (unsigned)((m + kTB - 1) / kTB); };
    k_init_comp<<<G(n), kTB, 0, st>>>(n, edges, E, f.comp, f.sig, f.best, f.state);
    EGT_LAUNCH_CHECK();
    if (E == 0) {  // every vertex is its own component
        EGT_CUDA_TRY(cudaMemsetAsync(f.first, 0xff, sizeof(unsigned long long) * n, st));
        return EGT_OK;
    }
    // each round at least halves the non-trivial components
    int64_t live = E;  // upper bound of the list's length
    unsigned long long* list[2] = {act, act2};
    for (int round = 0;; round++) {
        if (round > 64) { set_error("orientation: spanning forest did not converge"); return EGT_ERR_CAP_EXCEEDED; }
        const int side = round & 1;
        const unsigned gs = (unsigned)std::max<int64_t>(
            1, std::min<int64_t>((live + kTB * kSelItems - 1) / (kTB * kSelItems), 148 * 8));
        k_select<<<gs, kTB, 0, st>>>(list[side], list[side ^ 1], side, ukey, bits, f.comp, f.best, f.state);
        EGT_LAUNCH_CHECK();
        k_hook<<<G(n), kTB, 0, st>>>(ukey, sgn, n, bits, side, f.comp, f.sig, f.best, f.link,
                                     round == 0 ? f.first : nullptr, f.state, ctr, msf);
        EGT_LAUNCH_CHECK();
        k_jump<<<G(n), kTB, 0, st>>>(f.link, n, f.comp, f.state);
        EGT_LAUNCH_CHECK();
        k_relabel<<<G(n), kTB, 0, st>>>(n, f.link, f.comp, f.sig, f.best, f.state);
        EGT_LAUNCH_CHECK();
        if (round % kRoundsPerSync == kRoundsPerSync - 1) {
            ForestState s;
            EGT_CUDA_TRY(cudaMemcpyAsync(&s, f.state, sizeof(s), cudaMemcpyDeviceToHost, st));
            EGT_CUDA_TRY(cudaStreamSynchronize(st));
            if (s.linked == 0) break;
            live = s.live[side ^ 1];
        }
    }
    return EGT_OK;
}

}  // namespace

egt_status run_orient(egt_handle* h) {
    cudaStream_t st = h->stream;
    const int n = (int)h->n;
    int64_t nnz = 0;
    EGT_TRY(csr_nnz(h, &nnz));
    EGT_CUDA_TRY(cudaEventRecord(h->ev[10], st));
    EGT_CUDA_TRY(cudaMemsetAsync(h->d_counters + kCtrMsf, 0, 2 * sizeof(unsigned long long), st));
    if (nnz == 0 || n < 2) {
        EGT_CUDA_TRY(cudaEventRecord(h->ev[11], st));
        return EGT_OK;
    }
    int bits = 1;
    while ((1ll << bits) < (int64_t)n) bits++;
    auto G = [&](int64_t m) { return (unsigned)((m + kTB - 1) / kTB); };
    // 1. undirected edges in key order, with their order keys and signs
    size_t t_scan = 0;
    EGT_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, t_scan, (int*)nullptr, (int*)nullptr, n + 1, st));
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t a = at; at += (bytes + 255) & ~(size_t)255; return a; };
    const size_t o_key = take(sizeof(unsigned long long) * nnz), o_ukey = take(sizeof(unsigned long long) * nnz),
                 o_act = take(sizeof(unsigned long long) * nnz), o_sgn = take(nnz), o_keep = take(nnz),
                 o_cnt = take(sizeof(int) * (n + 2)), o_boff = take(sizeof(int) * (n + 1)),
                 o_own = take(sizeof(int) * n), o_scan = take(t_scan),
                 o_longs = take(sizeof(int) * (nnz / kLongBucket + 1));
    char* m = nullptr;
    EGT_CUDA_TRY(cudaMallocAsync((void**)&m, at, st));
    auto* key = reinterpret_cast<unsigned long long*>(m + o_key);
    auto* ukey = reinterpret_cast<unsigned long long*>(m + o_ukey);
    auto* act = reinterpret_cast<unsigned long long*>(m + o_act);
    auto* sgn = reinterpret_cast<signed char*>(m + o_sgn);
    auto* keep = reinterpret_cast<unsigned char*>(m + o_keep);
    auto* cnt = reinterpret_cast<int*>(m + o_cnt);
    auto* boff = reinterpret_cast<int*>(m + o_boff);
    auto* own = reinterpret_cast<int*>(m + o_own);
    auto* longs = reinterpret_cast<int*>(m + o_longs);
    int* n_long = cnt + n + 1;
    EGT_CUDA_TRY(cudaMemsetAsync(cnt, 0, sizeof(int) * (n + 2), st));
    k_bucket_count<<<G((int64_t)n * kRowLanes), kTB, 0, st>>>(h->csr_off, h->csr_col, n, keep, own, cnt);
    EGT_LAUNCH_CHECK();
    EGT_CUDA_TRY(cub::DeviceScan::ExclusiveSum(m + o_scan, t_scan, cnt, boff, n + 1, st));
    k_bucket_fill<<<G((int64_t)n * kRowLanes), kTB, 0, st>>>(h->csr_off, h->csr_col, n, bits, keep, boff, own, key, longs,
                                                               n_long);
    EGT_LAUNCH_CHECK();
    if (nnz > kLongBucket) {
        const unsigned gl = (unsigned)std::min<int64_t>(nnz / kLongBucket, 148);
        k_bucket_sort<<<gl, kRadixThreads, 0, st>>>(key, ukey, boff, longs, n_long, bits);
        EGT_LAUNCH_CHECK();
    }
    k_bucket_edges<<<G(nnz), kTB, 0, st>>>(key, boff, n, bits, h->nrm, ukey, act, sgn);
    EGT_LAUNCH_CHECK();
    // 2. Borůvka rounds (the unordered edges' buffer is free again)
    Forest f;
    EGT_CUDA_TRY(f.alloc(n, st));
    egt_status status =
        spanning_forest(n, (int)nnz, bits, ukey, act, key, boff + n, sgn, h->d_counters, f, nullptr, st);
    if (status == EGT_OK) {
        // 3. roots (first vertex of each tree's lightest edge) and signs
        EGT_CUDA_TRY(cudaMemsetAsync(f.best, 0xff, sizeof(unsigned long long) * n, st));
        k_roots<<<G(n), kTB, 0, st>>>(n, f.comp, f.first, f.best);
        EGT_LAUNCH_CHECK();
        k_apply<<<G(n), kTB, 0, st>>>(n, bits, f.comp, f.sig, f.best, ukey, h->nrm, h->d_counters);
        EGT_LAUNCH_CHECK();
    }
    cudaFreeAsync(m, st);
    f.release(st);
    EGT_CUDA_TRY(cudaEventRecord(h->ev[11], st));
    return status;
}

// orient_kruskal (MST.cpp:399-423) with Graph::kruskalMST (:297-376),
// DisjointSets (:185-229) and orientSpanningTree (:262-279), the reference's
// CPU orienter, on the GPU.  The reference keeps each undirected list edge
// once, sorts the edges by (weight, u, v) with weight max(0, 1 - |n_u . n_v|)
// in double, runs Kruskal with a union-find (union by rank, the second root
// winning ties), and walks every tree depth-first from its union-find root,
// negating a child whose float dot product with its (final) parent normal is
// negative.  Here:
//   1. the edge keys are sorted and deduplicated, the weights computed with
//      the reference's rounding, and the edges ranked by a stable sort on the
//      weight bits -- the reference's (weight, u, v) order;
//   2. Borůvka over that total order gives the same (unique) forest, with each
//      vertex's sign parity relative to its component;
//   3. the union-find roots depend on the order of the unions, so the forest
//      edges are replayed on the host in Kruskal order (n - components unions,
//      no sorting, no edge scan) with the reference's rank rule;
//   4. along a tree path the walk's rule multiplies the edge signs, except
//      across an edge whose dot product is exactly zero: the child is then
//      left as it is and its subtree follows from it.  So each vertex's sign is
//      its parity relative to the start of its part of the tree: the root, or
//      the child end of the last zero edge above it.  Parts are found (only
//      when zero edges exist) by a second forest pass without the zero edges
//      and a walk over the few zero edges on the host.
// knn: n rows of k ints (device), the first k_use of each read; nrm: [3n] SoA
// normals (device), in place.
egt_status run_orient_kruskal(const int* knn, float* nrm, int n, int k, int k_use, cudaStream_t st) {
    if (n < 2 || k_use < 1) return EGT_OK;
    const int64_t slots = (int64_t)n * k_use;
    if (slots > INT32_MAX) { set_error("orient_kruskal: n * k_use exceeds 2^31 - 1 list entries"); return EGT_ERR_CAP_EXCEEDED; }
    int bits = 1;
    while ((1ll << bits) < (int64_t)n) bits++;
    const unsigned TB = 256;
    auto G = [&](int64_t m) { return (unsigned)((m + TB - 1) / TB); };
    std::vector<void*> owned;
    auto D = [&](auto** p, size_t bytes) {
        const cudaError_t e = cudaMallocAsync((void**)p, std::max<size_t>(bytes, 16), st);
        if (e == cudaSuccess) owned.push_back((void*)*p);
        return e;
    };
    struct Releaser {
        std::vector<void*>& v;
        cudaStream_t st;
        ~Releaser() { for (void* p : v) cudaFreeAsync(p, st); }
    } releaser{owned, st};
    unsigned long long *ctr = nullptr, *bufA = nullptr, *bufB = nullptr;
    unsigned char* flag = nullptr;
    int* d_num = nullptr;
    EGT_CUDA_TRY(D(&ctr, sizeof(unsigned long long) * kCtrWords));
    EGT_CUDA_TRY(D(&bufA, sizeof(unsigned long long) * slots));
    EGT_CUDA_TRY(D(&bufB, sizeof(unsigned long long) * slots));
    EGT_CUDA_TRY(D(&flag, slots));
    EGT_CUDA_TRY(D(&d_num, sizeof(int)));
    EGT_CUDA_TRY(cudaMemsetAsync(ctr, 0, sizeof(unsigned long long) * kCtrWords, st));
    k_kr_keys<<<G(slots), TB, 0, st>>>(knn, n, k, k_use, bits, bufA, ctr);
    EGT_LAUNCH_CHECK();
    // 1. unique edges in (u, v) order
    cub::DoubleBuffer<unsigned long long> keys(bufA, bufB);
    size_t t_sort = 0, t_flag = 0;
    EGT_CUDA_TRY(cub::DeviceRadixSort::SortKeys(nullptr, t_sort, keys, (int)slots, 0, 2 * bits, st));
    EGT_CUDA_TRY(cub::DeviceSelect::Flagged(nullptr, t_flag, bufA, flag, d_num, (int)slots, st));
    void* tmp = nullptr;
    EGT_CUDA_TRY(D(&tmp, std::max(t_sort, t_flag)));
    EGT_CUDA_TRY(cub::DeviceRadixSort::SortKeys(tmp, t_sort, keys, (int)slots, 0, 2 * bits, st));
    unsigned long long* ukey = keys.Current();
    unsigned long long* act = keys.Alternate();
    k_first_copy<<<G(slots), TB, 0, st>>>(ukey, slots, bits, flag);
    EGT_LAUNCH_CHECK();
    EGT_CUDA_TRY(cub::DeviceSelect::Flagged(tmp, t_flag, ukey, flag, d_num, (int)slots, st));
    int E = 0;
    unsigned long long bad = 0;
    EGT_CUDA_TRY(cudaMemcpyAsync(&E, d_num, sizeof(int), cudaMemcpyDeviceToHost, st));
    EGT_CUDA_TRY(cudaMemcpyAsync(&bad, ctr + kCtrFlag, sizeof(bad), cudaMemcpyDeviceToHost, st));
    EGT_CUDA_TRY(cudaStreamSynchronize(st));
    if (bad) { set_error("orient_kruskal: a list entry is >= n"); return EGT_ERR_ARG; }
    if (E == 0) return EGT_OK;
    // weights, signs, and the rank of every edge in (weight, u, v) order
    unsigned long long *wkey = nullptr, *wkey2 = nullptr;
    int *eidx = nullptr, *order = nullptr;
    signed char* sgn = nullptr;
    unsigned char *zero = nullptr, *msf = nullptr;
    EGT_CUDA_TRY(D(&wkey, sizeof(unsigned long long) * E));
    EGT_CUDA_TRY(D(&wkey2, sizeof(unsigned long long) * E));
    EGT_CUDA_TRY(D(&eidx, sizeof(int) * E));
    EGT_CUDA_TRY(D(&order, sizeof(int) * E));
    EGT_CUDA_TRY(D(&sgn, E));
    EGT_CUDA_TRY(D(&zero, E));
    EGT_CUDA_TRY(D(&msf, E));
    k_kr_weights<<<G(E), TB, 0, st>>>(ukey, E, bits, nrm, n, wkey, eidx, sgn, zero);
    EGT_LAUNCH_CHECK();
    unsigned long long *vkey = nullptr, *okey = nullptr, *sel = nullptr;
    EGT_CUDA_TRY(D(&vkey, sizeof(unsigned long long) * E));
    EGT_CUDA_TRY(D(&okey, sizeof(unsigned long long) * E));
    EGT_CUDA_TRY(D(&sel, sizeof(unsigned long long) * E));
    unsigned char *f1 = nullptr, *f2 = nullptr, *f3 = nullptr;
    EGT_CUDA_TRY(D(&f1, E));
    EGT_CUDA_TRY(D(&f2, E));
    EGT_CUDA_TRY(D(&f3, E));
    size_t t_pairs = 0, t_sel = 0;
    EGT_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, t_pairs, wkey, wkey2, eidx, order, E, 0, 64, st));
    EGT_CUDA_TRY(cub::DeviceSelect::Flagged(nullptr, t_sel, vkey, f1, sel, d_num, E, st));
    void* tmp2 = nullptr;
    EGT_CUDA_TRY(D(&tmp2, std::max(t_pairs, t_sel)));
    EGT_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp2, t_pairs, wkey, wkey2, eidx, order, E, 0, 64, st));
    k_kr_rank<<<G(E), TB, 0, st>>>(order, E, act);
    EGT_LAUNCH_CHECK();
    EGT_CUDA_TRY(cudaMemsetAsync(msf, 0, E, st));
    // 2. the minimum spanning forest for that order, with sign parities
    Forest f;
    struct ForestReleaser {
        Forest& f;
        cudaStream_t st;
        ~ForestReleaser() { f.release(st); }
    } fr{f, st};
    EGT_CUDA_TRY(f.alloc(n, st));
    // (the second edge list: the unsorted weights are no longer needed)
    EGT_TRY(spanning_forest(n, E, bits, ukey, act, wkey, nullptr, sgn, ctr, f, msf, st));
    // forest edges in Kruskal order, and the zero-dot ones among them
    k_kr_forest_lists<<<G(E), TB, 0, st>>>(order, E, ukey, msf, zero, vkey, okey, f1, f2, f3);
    EGT_LAUNCH_CHECK();
    int m = 0;
    EGT_CUDA_TRY(cub::DeviceSelect::Flagged(tmp2, t_sel, vkey, f1, sel, d_num, E, st));
    EGT_CUDA_TRY(cudaMemcpyAsync(&m, d_num, sizeof(int), cudaMemcpyDeviceToHost, st));
    EGT_CUDA_TRY(cudaStreamSynchronize(st));
    std::vector<unsigned long long> tree((size_t)m);
    if (m) EGT_CUDA_TRY(cudaMemcpyAsync(tree.data(), sel, sizeof(unsigned long long) * m, cudaMemcpyDeviceToHost, st));
    EGT_CUDA_TRY(cudaStreamSynchronize(st));
    // 3. the reference's union-find, replayed over the forest edges in order
    // (union by rank, the second root winning ties; path halving in place of
    // the reference's full compression, which changes no root or rank; the
    // next edges' entries are prefetched, the accesses being random)
    const unsigned long long mask = (1ull << bits) - 1ull;
    std::vector<int> par((size_t)n);
    std::vector<unsigned char> rnk((size_t)n, 0);
    std::iota(par.begin(), par.end(), 0);
    auto find = [&](int x) {
        while (par[x] != x) {
            par[x] = par[par[x]];
            x = par[x];
        }
        return x;
    };
    constexpr size_t kAhead = 16;
    for (size_t i = 0; i < tree.size(); i++) {
        if (i + kAhead < tree.size()) {
            const unsigned long long t2 = tree[i + kAhead];
            __builtin_prefetch(&par[(int)(t2 >> bits)]);
            __builtin_prefetch(&par[(int)(t2 & mask)]);
        }
        const unsigned long long t = tree[i];
        const int a = find((int)(t >> bits)), b = find((int)(t & mask));
        if (a == b) continue;  // cannot happen for a forest; kept for safety
        if (rnk[a] > rnk[b]) par[b] = a;
        else par[a] = b;
        if (rnk[a] == rnk[b]) rnk[b]++;
    }
    // where each tree's walk starts: its union-find root (a root is a vertex
    // that is its own parent)
    std::vector<int> starts;
    // 4. zero-dot forest edges split the trees into parts
    int z = 0;
    EGT_CUDA_TRY(cub::DeviceSelect::Flagged(tmp2, t_sel, vkey, f3, sel, d_num, E, st));
    EGT_CUDA_TRY(cudaMemcpyAsync(&z, d_num, sizeof(int), cudaMemcpyDeviceToHost, st));
    EGT_CUDA_TRY(cudaStreamSynchronize(st));
    const int* comp_for_sign = f.comp;
    const signed char* sig_for_sign = f.sig;
    Forest g;
    struct ForestReleaser gr{g, st};
    if (z == 0) {
        for (int r = 0; r < n; r++)
            if (par[r] == r) starts.push_back(r);
    } else {
        std::vector<unsigned long long> zedges((size_t)z);
        EGT_CUDA_TRY(cudaMemcpyAsync(zedges.data(), sel, sizeof(unsigned long long) * z, cudaMemcpyDeviceToHost, st));
        EGT_CUDA_TRY(cudaStreamSynchronize(st));
        // parts: the forest without its zero edges
        int e2 = 0;
        EGT_CUDA_TRY(cub::DeviceSelect::Flagged(tmp2, t_sel, okey, f2, sel, d_num, E, st));
        EGT_CUDA_TRY(cudaMemcpyAsync(&e2, d_num, sizeof(int), cudaMemcpyDeviceToHost, st));
        EGT_CUDA_TRY(cudaStreamSynchronize(st));
        EGT_CUDA_TRY(g.alloc(n, st));
        EGT_TRY(spanning_forest(n, e2, bits, ukey, sel, wkey, nullptr, sgn, ctr, g, nullptr, st));
        std::vector<int> part((size_t)n);
        EGT_CUDA_TRY(cudaMemcpyAsync(part.data(), g.comp, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
        EGT_CUDA_TRY(cudaStreamSynchronize(st));
        // walk the parts from each tree's root part across the zero edges: the
        // part entered through zero edge (a, b) from a's side starts at b
        std::vector<std::vector<int>> by_part;
        std::vector<int> part_id((size_t)n, -1), start;
        auto pid = [&](int v) {
            int& p = part_id[part[v]];
            if (p < 0) { p = (int)start.size(); start.push_back(-1); by_part.emplace_back(); }
            return p;
        };
        for (int i = 0; i < z; i++) {
            const int a = (int)(zedges[i] >> bits), b = (int)(zedges[i] & mask);
            by_part[pid(a)].push_back(i);
            by_part[pid(b)].push_back(i);
        }
        std::vector<int> queue;
        for (int r = 0; r < n; r++) {
            if (par[r] != r) continue;
            const int p0 = part_id[part[r]];
            if (p0 < 0) {  // a tree without zero edges: one part
                starts.push_back(r);
                continue;
            }
            if (start[p0] >= 0) continue;
            start[p0] = r;
            queue.assign(1, p0);
            for (size_t qi = 0; qi < queue.size(); qi++) {
                const int p = queue[qi];
                for (int i : by_part[p]) {
                    const int a = (int)(zedges[i] >> bits), b = (int)(zedges[i] & mask);
                    const int pa = part_id[part[a]], pb = part_id[part[b]];
                    const int other = pa == p ? pb : pa;
                    if (start[other] >= 0) continue;
                    start[other] = pa == p ? b : a;
                    queue.push_back(other);
                }
            }
        }
        starts.insert(starts.end(), start.begin(), start.end());
        comp_for_sign = g.comp;
        sig_for_sign = g.sig;
    }
    // every vertex takes the sign parity relative to its part's start
    int *d_starts = nullptr, *d_ref = nullptr;
    const int ns = (int)starts.size();
    EGT_CUDA_TRY(D(&d_starts, sizeof(int) * ns));
    EGT_CUDA_TRY(D(&d_ref, sizeof(int) * n));
    EGT_CUDA_TRY(cudaMemcpyAsync(d_starts, starts.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, st));
    k_kr_starts<<<G(ns), TB, 0, st>>>(d_starts, ns, comp_for_sign, d_ref);
    EGT_LAUNCH_CHECK();
    k_kr_apply<<<G(n), TB, 0, st>>>(n, comp_for_sign, d_ref, sig_for_sign, nrm);
    EGT_LAUNCH_CHECK();
    EGT_CUDA_TRY(cudaStreamSynchronize(st));  // host vectors above are read by pending copies
    return EGT_OK;
}

}  // namespace egt
