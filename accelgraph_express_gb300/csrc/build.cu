/*
 * CSR and CSC built on the device from an edge list.
 *
 * The reference builds its CSR with the OpenGraph pair sortRunAlgorithms +
 * graphCSRAssignEdgeList (call sites SSSP.c:552-565, bellmanFord.c:737-744;
 * the OpenGraph sources are absent from the snapshot).  The host build here,
 * graphCSRFromEdgeList, sorts the edges by (row, neighbour) with a stable
 * radix sort, so each row lists its neighbours in ascending id and duplicate
 * edges keep their input order.  This file sorts them into the same order on
 * the GPU, so every array it produces is identical to the host build's.
 *
 * The edges are three arrays (source, destination, weight).  The CSR is a
 * stable sort by destination, then by source; the CSC a stable sort of that
 * order by destination (duplicates still in input order).  Each is a least
 * significant digit radix sort on the b bits of the ids, in digits of 8 bits
 * or, spread evenly, fewer:
 *   k_sort_count    per-tile digit counts, tile-major (counts[tile][d]), by
 *                   shared atomics (one per warp when its keys share a digit)
 *   column scan     k_col_one, or k_col_reduce / k_col_top / k_col_down:
 *                   counts[tile][d] becomes the first output slot of digit
 *                   d's keys of that tile (keys of smaller digits, then of
 *                   digit d in earlier tiles); every access is a coalesced row
 *   k_sort_scatter  stable rank within the tile (per-warp digit counters;
 *                   lanes with equal digits found by ballots), then one array
 *                   after the other is put in digit order in shared memory
 *                   and written out in runs
 * The first pass reads the caller's arrays, checks the ids and takes the
 * largest weight; the last pass of a direction writes the mapping's neighbour
 * and weight arrays, and k_offsets finds the rows in the sorted ids.
 *
 * A pass reads the sorted field twice, the others once and writes all once
 * (the reduce-then-scan form: no block waits on another).  67M weighted edges,
 * V = 2^22: 340-360 us a scatter (4.6 TB/s), 55 a count, 35 the scan; the build
 * 4.2 ms (6.4 when the words (row << b | neighbour) were sorted).  Tiles of
 * 4,096 keys by 256 threads, four blocks an SM; 8,192 by 512 threads 4.7 ms, 3,072
 * in five blocks 4.35, 2,048 in eight 4.75.
 */
#include <cuda_runtime.h>

#include <cstring>
#include <utility>

#include "gg_internal.h"

namespace {

constexpr int SORT_BINS = 256; /* most digit values of a pass */
constexpr int SORT_THREADS = 256;
constexpr int SORT_CTAS = 4; /* resident per SM: 64 registers a thread */
constexpr int SORT_ITEMS = 16;
constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;
constexpr int SORT_WARPS = SORT_THREADS / 32;

constexpr uint32_t COL_TILES = 64;      /* tiles per block of the column scan */
constexpr uint32_t COL_ONE_TILES = 256; /* tiles that k_col_one scans */

/* one pass: the arrays in and out (p1, p2: as many as PAYS), the first output
 * slots from the column scan, and, for the first pass over a caller's edges,
 * V and flags: [0] set when an id is >= V, [1] the largest weight above 0 */
template <class KEY>
struct SortPass
{
    const KEY *key;
    const uint32_t *p1, *p2;
    KEY *okey;
    uint32_t *op1, *op2;
    const uint32_t *first;
    uint32_t n;
    int shift;
    uint32_t V;
    uint32_t *flags;
};

template <int BITS, class KEY>
__device__ __forceinline__ uint32_t digit_of(KEY k, int shift)
{
    return (uint32_t)(k >> shift) & ((1u << BITS) - 1u);
}

/* lanes of `among` holding a key with the same digit (warp multisplit: one
 * ballot per digit bit, ALU work instead of a match instruction) */
template <int BITS>
__device__ __forceinline__ uint32_t digit_peers(uint32_t among, uint32_t d)
{
    uint32_t m = among;
#pragma unroll
    for (int b = 0; b < BITS; b++)
    {
        const bool bit = (d >> b) & 1u;
        const uint32_t v = __ballot_sync(0xffffffffu, bit);
        m &= bit ? v : ~v;
    }
    return m;
}

/* tile elements: warp w takes the 32 * SORT_ITEMS consecutive keys from tile
 * base + w * 32 * SORT_ITEMS, lane-interleaved per step; the same map in both
 * kernels */
template <class KEY, int BITS>
__global__ void __launch_bounds__(SORT_THREADS) k_sort_count(const KEY *__restrict__ keys, uint32_t n, int shift,
                                                             uint32_t *__restrict__ counts)
{
    constexpr uint32_t BINS = 1u << BITS;
    __shared__ uint32_t h[BINS];
    const uint32_t lane = threadIdx.x & 31, tile = blockIdx.x;
    const KEY *t = keys + (size_t)tile * SORT_TILE;
    const uint32_t cnt = min(n - tile * (uint32_t)SORT_TILE, (uint32_t)SORT_TILE);
    const uint32_t base = (threadIdx.x >> 5) * 32u * SORT_ITEMS + lane;
    for (uint32_t i = threadIdx.x; i < BINS; i += SORT_THREADS) h[i] = 0u;
    __syncthreads();
    KEY k[SORT_ITEMS];
#pragma unroll
    for (int it = 0; it < SORT_ITEMS; it++) k[it] = base + it * 32 < cnt ? t[base + it * 32] : KEY(0);
#pragma unroll
    for (int it = 0; it < SORT_ITEMS; it++)
    {
        const bool valid = base + it * 32 < cnt;
        const uint32_t d = digit_of<BITS>(k[it], shift);
        /* a warp whose keys all share one digit (frequent in the skewed
         * high digits of row ids) adds 32 at once; otherwise every key adds
         * itself.  Every lane takes part in the shuffle and the vote */
        const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);
        if (__all_sync(0xffffffffu, valid && d == d0))
        {
            if (lane == 0) atomicAdd(&h[d], 32u);
        }
        else if (valid)
            atomicAdd(&h[d], 1u);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < BINS; i += SORT_THREADS) counts[(size_t)tile * BINS + i] = h[i];
}

/* shared memory of k_sort_scatter: two staging arrays, the per-warp digit
 * counts, and for each digit its first output slot less its place in the tile */
/* the value, of which the compiler keeps no derived form in registers */
__device__ __forceinline__ uint32_t opaque(uint32_t x)
{
    asm volatile("" : "+r"(x));
    return x;
}

template <class KEY, int BITS, int PAYS>
constexpr size_t sort_smem()
{
    return (size_t)SORT_TILE * (sizeof(KEY) + (PAYS ? 4 : 0)) + ((size_t)SORT_WARPS * 4 + 4) * (1u << BITS) + SORT_WARPS * 4;
}

/* Bounded by the shared-memory and global wavefronts of the digit order (each
 * array is stored at random in the tile once) and by issue: the arrays go
 * through shared memory one after the other, 4 bytes a key and two buffers in
 * turn, so that SORT_CTAS blocks fit an SM with their ranks in registers. */
template <class KEY, int BITS, int PAYS, bool FIRST>
__global__ void __launch_bounds__(SORT_THREADS, SORT_CTAS) k_sort_scatter(const SortPass<KEY> a)
{
    constexpr uint32_t BINS = 1u << BITS;
    static_assert(BINS >= 32 && BINS <= SORT_THREADS, "a thread per digit, whole warps");
    extern __shared__ __align__(16) unsigned char smem[];
    KEY *skey = reinterpret_cast<KEY *>(smem);
    uint32_t *s1 = reinterpret_cast<uint32_t *>(skey + SORT_TILE);
    uint32_t *s2 = reinterpret_cast<uint32_t *>(smem);
    uint32_t *wcnt = s1 + (PAYS ? SORT_TILE : 0); /* [SORT_WARPS][BINS] */
    uint32_t *gofs = wcnt + SORT_WARPS * BINS;
    uint32_t *wtot = gofs + BINS;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, tile = blockIdx.x;
    const size_t t0 = (size_t)tile * SORT_TILE;
    const uint32_t cnt = min(a.n - tile * (uint32_t)SORT_TILE, (uint32_t)SORT_TILE);
    const uint32_t base = w * 32u * SORT_ITEMS + lane;
    uint32_t *mine = wcnt + w * BINS;
    KEY k[SORT_ITEMS];
    if (cnt == SORT_TILE)
    {
#pragma unroll
        for (int it = 0; it < SORT_ITEMS; it++) k[it] = a.key[t0 + base + it * 32];
    }
    else
    {
#pragma unroll
        for (int it = 0; it < SORT_ITEMS; it++) k[it] = base + it * 32 < cnt ? a.key[t0 + base + it * 32] : KEY(0);
    }
    uint32_t slot = 0;
    if (threadIdx.x < BINS) slot = a.first[(size_t)tile * BINS + threadIdx.x];
#pragma unroll
    for (uint32_t i = lane; i < BINS; i += 32) mine[i] = 0u;
    __syncwarp();
    /* rank among the warp's earlier keys of the same digit, in element
     * order: every lane reads the warp's counter of its digit, and the
     * group's lowest lane advances it by the group's size */
    uint32_t at[SORT_ITEMS / 2] = {}; /* 16 bits each */
    static_assert(SORT_TILE <= 65536, "places in the tile in 16 bits");
#pragma unroll
    for (int it = 0; it < SORT_ITEMS; it++)
    {
        const uint32_t d = digit_of<BITS>(k[it], a.shift);
        uint32_t among = 0xffffffffu;
        if (cnt != SORT_TILE) among = __ballot_sync(0xffffffffu, base + it * 32 < cnt);
        const uint32_t peers = digit_peers<BITS>(among, d);
        const uint32_t before = (uint32_t)__popc(peers & ((1u << lane) - 1u));
        const uint32_t seen = mine[d];
        at[it / 2] |= (seen + before) << (it % 2 * 16);
        __syncwarp();
        if (before == 0u && (among >> lane & 1u)) mine[d] = seen + (uint32_t)__popc(peers);
        __syncwarp();
    }
    __syncthreads();
    /* thread t = digit t: exclusive prefix over warps on top of the tile's
     * digit start, which a block scan of the digit totals gives */
    uint32_t run = 0, incl = 0;
    if (threadIdx.x < BINS)
    {
#pragma unroll
        for (int ww = 0; ww < SORT_WARPS; ww++) run += wcnt[ww * BINS + threadIdx.x];
        incl = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        if (lane == 31) wtot[w] = incl;
    }
    __syncthreads();
    if (threadIdx.x < BINS)
    {
        uint32_t start = incl - run;
        for (uint32_t ww = 0; ww < w; ww++) start += wtot[ww];
        gofs[threadIdx.x] = slot - start;
#pragma unroll
        for (int ww = 0; ww < SORT_WARPS; ww++)
        {
            const uint32_t c = wcnt[ww * BINS + threadIdx.x];
            wcnt[ww * BINS + threadIdx.x] = start;
            start += c;
        }
    }
    __syncthreads();
    uint32_t v[SORT_ITEMS];
    auto load = [&](const uint32_t *__restrict__ p) {
        if (cnt == SORT_TILE)
        {
#pragma unroll
            for (int it = 0; it < SORT_ITEMS; it++) v[it] = p[t0 + base + it * 32];
        }
        else
        {
#pragma unroll
            for (int it = 0; it < SORT_ITEMS; it++) v[it] = base + it * 32 < cnt ? p[t0 + base + it * 32] : 0u;
        }
    };
    auto stage = [&](uint32_t *sm) {
#pragma unroll
        for (int it = 0; it < SORT_ITEMS; it++)
            if (base + it * 32 < cnt) sm[opaque(at[it / 2]) >> (it % 2 * 16) & 0xffffu] = v[it];
    };
    if (PAYS > 0) load(a.p1);
    /* the keys in digit order */
#pragma unroll
    for (int it = 0; it < SORT_ITEMS; it++)
    {
        at[it / 2] += mine[digit_of<BITS>(k[it], a.shift)] << (it % 2 * 16);
        if (base + it * 32 < cnt) skey[at[it / 2] >> (it % 2 * 16) & 0xffffu] = k[it];
        if (FIRST && base + it * 32 < cnt && (k[it] >= a.V || v[it] >= a.V)) atomicOr(a.flags, 1u);
    }
    __syncthreads();
    /* runs of one digit go to consecutive output slots */
    uint32_t to[SORT_ITEMS];
#pragma unroll
    for (int it = 0; it < SORT_ITEMS; it++)
    {
        const uint32_t j = threadIdx.x + it * SORT_THREADS;
        if (j < cnt)
        {
            const KEY key = skey[j];
            to[it] = gofs[digit_of<BITS>(key, a.shift)] + j;
            a.okey[to[it]] = key;
        }
    }
    if (PAYS > 0)
    {
        stage(s1);
        if (PAYS > 1) load(a.p2);
        __syncthreads();
#pragma unroll
        for (int it = 0; it < SORT_ITEMS; it++)
        {
            const uint32_t j = threadIdx.x + it * SORT_THREADS;
            if (j < cnt) a.op1[opaque(to[it])] = s1[j];
        }
    }
    if (PAYS > 1)
    {
        if (FIRST)
        {
            /* the largest weight above 0 (none: 0), as the edge-list readers
             * record it: such floats order as their bits, and NaN fails > */
            float m = 0.0f;
#pragma unroll
            for (int it = 0; it < SORT_ITEMS; it++)
                if (__uint_as_float(v[it]) > m) m = __uint_as_float(v[it]);
            const uint32_t all = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
            if (lane == 0 && all > __ldcg(a.flags + 1)) atomicMax(a.flags + 1, all);
        }
        stage(s2);
        __syncthreads();
#pragma unroll
        for (int it = 0; it < SORT_ITEMS; it++)
        {
            const uint32_t j = threadIdx.x + it * SORT_THREADS;
            if (j < cnt) a.op2[opaque(to[it])] = s2[j];
        }
    }
}

/* ---- column scan of the [tile][digit] counts (thread = digit) ---- */

/* the column sums of each block of COL_TILES tiles (the loads of a block's
 * rows are independent: unrolled so they are in flight together) */
__global__ void __launch_bounds__(SORT_BINS) k_col_reduce(const uint32_t *__restrict__ counts, uint32_t ntiles,
                                                          uint32_t *csum)
{
    const uint32_t bins = blockDim.x, t0 = blockIdx.x * COL_TILES, t1 = min(t0 + COL_TILES, ntiles);
    uint32_t t = 0;
#pragma unroll 8
    for (uint32_t tile = t0; tile < t1; tile++) t += counts[(size_t)tile * bins + threadIdx.x];
    csum[(size_t)blockIdx.x * bins + threadIdx.x] = t;
}

/* one block of COL_SPLIT threads per digit: c[r][d] becomes the first output
 * slot of digit d in row r (the keys of all smaller digits plus digit d in
 * earlier rows); each digit's rows are split over COL_SPLIT threads, combined
 * through shared memory.  Rows are block sums, or, up to COL_ONE_TILES, the
 * tiles themselves (one launch instead of three) */
constexpr uint32_t COL_SPLIT = 4;

__global__ void __launch_bounds__(COL_SPLIT * SORT_BINS) k_col_one(uint32_t *c, uint32_t rows)
{
    __shared__ uint32_t part[COL_SPLIT][SORT_BINS];
    __shared__ uint32_t wtot[SORT_BINS / 32];
    const uint32_t bins = blockDim.x / COL_SPLIT, d = threadIdx.x % bins, q = threadIdx.x / bins;
    const uint32_t b0 = (uint32_t)((uint64_t)rows * q / COL_SPLIT);
    const uint32_t b1 = (uint32_t)((uint64_t)rows * (q + 1) / COL_SPLIT);
    uint32_t run = 0;
#pragma unroll 8
    for (uint32_t b = b0; b < b1; b++) run += c[(size_t)b * bins + d];
    part[q][d] = run;
    __syncthreads();
    /* digit d's total and the start of quarter q within it */
    uint32_t before = 0, total = 0;
    for (uint32_t k = 0; k < COL_SPLIT; k++)
    {
        if (k < q) before += part[k][d];
        total += part[k][d];
    }
    /* exclusive scan of the digit totals (the first `bins` threads) */
    uint32_t base = 0;
    if (q == 0)
    {
        const uint32_t lane = d & 31, w = d >> 5;
        uint32_t incl = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        if (lane == 31) wtot[w] = incl;
        base = incl - total;
    }
    __syncthreads();
    if (q == 0)
    {
        for (uint32_t k = 0; k < (d >> 5); k++) base += wtot[k];
        part[0][d] = base;
    }
    __syncthreads();
    uint32_t at = part[0][d] + before, b = b0;
    /* eight rows loaded together, then their running prefix written */
    for (; b + 8 <= b1; b += 8)
    {
        uint32_t n[8];
#pragma unroll
        for (int k = 0; k < 8; k++) n[k] = c[(size_t)(b + k) * bins + d];
#pragma unroll
        for (int k = 0; k < 8; k++)
        {
            c[(size_t)(b + k) * bins + d] = at;
            at += n[k];
        }
    }
    for (; b < b1; b++)
    {
        const uint32_t n = c[(size_t)b * bins + d];
        c[(size_t)b * bins + d] = at;
        at += n;
    }
}

__global__ void __launch_bounds__(SORT_BINS) k_col_down(uint32_t *counts, uint32_t ntiles,
                                                        const uint32_t *__restrict__ csum)
{
    const uint32_t bins = blockDim.x, t0 = blockIdx.x * COL_TILES, t1 = min(t0 + COL_TILES, ntiles);
    uint32_t run = csum[(size_t)blockIdx.x * bins + threadIdx.x];
    uint32_t tile = t0;
    /* eight rows loaded together, then their running prefix written */
    for (; tile + 8 <= t1; tile += 8)
    {
        uint32_t c[8];
#pragma unroll
        for (int k = 0; k < 8; k++) c[k] = counts[(size_t)(tile + k) * bins + threadIdx.x];
#pragma unroll
        for (int k = 0; k < 8; k++)
        {
            counts[(size_t)(tile + k) * bins + threadIdx.x] = run;
            run += c[k];
        }
    }
    for (; tile < t1; tile++)
    {
        uint32_t *p = counts + (size_t)tile * bins + threadIdx.x;
        const uint32_t c = *p;
        *p = run;
        run += c;
    }
}

/* off[v] = the first slot whose key is >= v (off[V] = n): slot i writes the
 * offsets of the rows between its predecessor's key and its own.  A thread
 * takes four slots, so that the keys are read once, in 16-byte loads */
__global__ void k_offsets(const uint32_t *__restrict__ keys, uint32_t n, uint32_t V, uint32_t *__restrict__ off)
{
    const uint64_t groups = (uint64_t)n / 4 + 1; /* the last one writes off[..V] = n */
    for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < groups; q += (uint64_t)gridDim.x * blockDim.x)
    {
        const uint64_t i0 = q * 4;
        uint32_t k[4];
        if (i0 + 4 <= n)
        {
            const uint4 v = *reinterpret_cast<const uint4 *>(keys + i0);
            k[0] = v.x;
            k[1] = v.y;
            k[2] = v.z;
            k[3] = v.w;
        }
        else
        {
#pragma unroll
            for (int j = 0; j < 4; j++) k[j] = i0 + j < n ? keys[i0 + j] : V;
        }
        /* rows 0 .. next - 1 have their offsets from earlier slots */
        uint64_t next = i0 ? (uint64_t)min(keys[i0 - 1], V) + 1u : 0u;
#pragma unroll
        for (int j = 0; j < 4; j++)
        {
            if (i0 + j > n) break;
            const uint32_t cur = min(k[j], V); /* above V: only an id >= V, which is reported */
            for (; next <= cur; next++) off[next] = (uint32_t)(i0 + j);
        }
    }
}

__global__ void k_degrees(const uint32_t *__restrict__ off, uint32_t V, uint32_t *deg)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        deg[v] = off[v + 1] - off[v];
}

int bits_for(uint32_t V)
{
    int b = 1;
    while (b < 32 && (1ull << b) < V) b++;
    return b;
}

int grid_for(uint64_t n, int threads)
{
    const uint64_t b = (n + threads - 1) / threads, cap = (uint64_t)gg_sm_count() * 8;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

uint32_t sort_tiles(uint64_t n) { return (uint32_t)((n + SORT_TILE - 1) / SORT_TILE); }

/* bytes of the counts and of the block sums of sorts of n keys */
size_t sort_counts_bytes(uint64_t n) { return (size_t)SORT_BINS * (sort_tiles(n) + 1) * 4; }
size_t sort_sums_bytes(uint64_t n) { return ((size_t)sort_tiles(n) / COL_TILES + 2) * SORT_BINS * 4; }

template <class KEY, int BITS, int PAYS, bool FIRST>
gg_status sort_pass_run(const SortPass<KEY> &a, uint32_t *counts, uint32_t *sums, cudaStream_t s)
{
    constexpr uint32_t BINS = 1u << BITS;
    constexpr size_t smem = sort_smem<KEY, BITS, PAYS>();
    GG_CUDA(cudaFuncSetAttribute(k_sort_scatter<KEY, BITS, PAYS, FIRST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    const uint32_t nt = sort_tiles(a.n), nb = (nt + COL_TILES - 1) / COL_TILES;
    k_sort_count<KEY, BITS><<<nt, SORT_THREADS, 0, s>>>(a.key, a.n, a.shift, counts);
    if (nt <= COL_ONE_TILES)
        k_col_one<<<1, COL_SPLIT * BINS, 0, s>>>(counts, nt);
    else
    {
        k_col_reduce<<<nb, BINS, 0, s>>>(counts, nt, sums);
        k_col_one<<<1, COL_SPLIT * BINS, 0, s>>>(sums, nb);
        k_col_down<<<nb, BINS, 0, s>>>(counts, nt, sums);
    }
    SortPass<KEY> b = a;
    b.first = counts;
    k_sort_scatter<KEY, BITS, PAYS, FIRST><<<nt, SORT_THREADS, smem, s>>>(b);
    GG_CUDA(cudaGetLastError());
    return GG_OK;
}

template <class KEY, int PAYS, bool FIRST>
gg_status sort_pass_bits(const SortPass<KEY> &a, int bits, uint32_t *counts, uint32_t *sums, cudaStream_t s)
{
    switch (bits)
    {
    case 8: return sort_pass_run<KEY, 8, PAYS, FIRST>(a, counts, sums, s);
    case 7: return sort_pass_run<KEY, 7, PAYS, FIRST>(a, counts, sums, s);
    case 6: return sort_pass_run<KEY, 6, PAYS, FIRST>(a, counts, sums, s);
    default: return sort_pass_run<KEY, 5, PAYS, FIRST>(a, counts, sums, s);
    }
}

/* edges, and which of the fields is sorted */
struct Edges
{
    uint32_t *src = nullptr, *dst = nullptr;
    float *w = nullptr; /* null when unweighted */
};

struct SortBufs
{
    Edges set[2];
    uint32_t *counts, *sums, *flags;
};

gg_status edges_pass(const Edges &in, const Edges &out, bool by_src, bool first, uint32_t n, uint32_t V, int shift,
                     int bits, const SortBufs &B, cudaStream_t s)
{
    SortPass<uint32_t> a{};
    a.key = by_src ? in.src : in.dst;
    a.p1 = by_src ? in.dst : in.src;
    a.p2 = (const uint32_t *)in.w;
    a.okey = by_src ? out.src : out.dst;
    a.op1 = by_src ? out.dst : out.src;
    a.op2 = (uint32_t *)out.w;
    a.n = n;
    a.shift = shift;
    a.V = V;
    a.flags = B.flags;
    if (out.w)
        return first ? sort_pass_bits<uint32_t, 2, true>(a, bits, B.counts, B.sums, s)
                     : sort_pass_bits<uint32_t, 2, false>(a, bits, B.counts, B.sums, s);
    return first ? sort_pass_bits<uint32_t, 1, true>(a, bits, B.counts, B.sums, s)
                 : sort_pass_bits<uint32_t, 1, false>(a, bits, B.counts, B.sums, s);
}

/* stable sort of the edges `in` by one field on its b bits; the last pass
 * writes `last`, in whose place a null array stands for the scratch array.
 * `in` and the returned place of every array may be scratch: a pass writes the
 * scratch set that holds nothing it reads */
gg_status sort_field(Edges in, Edges last, bool by_src, bool caller, uint32_t n, uint32_t V, const SortBufs &B, int &set,
                     Edges *out, cudaStream_t s)
{
    int rem = bits_for(V), shift = 0;
    for (int left = (rem + 7) / 8; left > 0; left--)
    {
        const int bits = (rem + left - 1) / left;
        Edges o = B.set[set];
        if (!in.w) o.w = nullptr;
        if (left == 1)
        {
            if (last.src) o.src = last.src;
            if (last.dst) o.dst = last.dst;
            if (last.w && in.w) o.w = last.w;
        }
        if (n) GG_CHECK(edges_pass(in, o, by_src, caller && shift == 0, n, V, shift, bits, B, s));
        in = o;
        set ^= 1;
        shift += bits;
        rem -= bits;
    }
    *out = in;
    return GG_OK;
}

/* device arrays of one direction: offsets from the sorted field */
gg_status offsets_alloc(gg_graph *g, const uint32_t *keys, uint32_t **off, cudaStream_t s)
{
    GG_CHECK(gg_dev_alloc(g, (void **)off, ((size_t)g->V + 1) * 4));
    k_offsets<<<grid_for((uint64_t)g->E / 4 + 1, 256), 256, 0, s>>>(keys, g->E, g->V, *off);
    GG_CUDA(cudaGetLastError());
    return GG_OK;
}

/* an edge array of the mapping, its pad cleared */
gg_status edge_alloc(gg_graph *g, void **p, cudaStream_t s)
{
    GG_CHECK(gg_dev_alloc(g, p, ((size_t)g->E + GG_EDGE_PAD) * 4));
    GG_CUDA(cudaMemsetAsync((uint32_t *)*p + g->E, 0, GG_EDGE_PAD * 4, s));
    return GG_OK;
}

/* both directions into g's arrays; see the head of the file */
gg_status build_directions(gg_graph *g, const SortBufs &B, const Edges &input, bool need_out, bool need_in, bool out_w,
                           bool in_w, cudaStream_t s)
{
    const uint32_t V = g->V, E = g->E;
    int set = 0;
    Edges e = input, last;
    if (!out_w && !in_w) e.w = nullptr;
    GG_CHECK(sort_field(e, Edges(), false, true, E, V, B, set, &e, s));
    if (need_out)
    {
        GG_CHECK(edge_alloc(g, (void **)&g->out_adj, s));
        last.dst = g->out_adj;
        if (out_w)
        {
            GG_CHECK(edge_alloc(g, (void **)&g->out_w, s));
            last.w = g->out_w;
        }
    }
    GG_CHECK(sort_field(e, last, true, false, E, V, B, set, &e, s));
    /* the out-degrees come from the CSR */
    GG_CHECK(offsets_alloc(g, e.src, &g->out_off, s));
    GG_CHECK(gg_dev_alloc(g, (void **)&g->out_deg, (size_t)V * 4 + 16));
    k_degrees<<<grid_for(V, 256), 256, 0, s>>>(g->out_off, V, g->out_deg);
    GG_CUDA(cudaGetLastError());
    if (!need_in) return GG_OK;
    last = Edges();
    GG_CHECK(edge_alloc(g, (void **)&g->in_adj, s));
    last.src = g->in_adj;
    if (in_w)
    {
        GG_CHECK(edge_alloc(g, (void **)&g->in_w, s));
        last.w = g->in_w;
    }
    else
        e.w = nullptr;
    GG_CHECK(sort_field(e, last, false, false, E, V, B, set, &e, s));
    return offsets_alloc(g, e.dst, &g->in_off, s);
}

} // namespace

gg_status gg_build_arrays(gg_graph *g, const uint32_t *src, const uint32_t *dst, const float *w, uint32_t what,
                          cudaStream_t s)
{
    GgRange range("gg_build_csr");
    const uint32_t V = g->V, E = g->E;
    if (V == 0) return gg_fail(GG_ERR_INVALID, "a graph needs at least one vertex");
    /* weights given and asked for; without given weights a _W request gets
     * the reference's constant 0.0001f, as gg_graph_map does */
    const bool weighted = w != nullptr && (what & (GG_MAP_OUT_W | GG_MAP_IN_W));
    const bool need_out = what & (GG_MAP_OUT | GG_MAP_OUT_W), need_in = what & (GG_MAP_IN | GG_MAP_IN_W);
    SortBufs B{};
    const size_t bytes = (size_t)E * 4 + 16, counts_bytes = sort_counts_bytes(E), sums_bytes = sort_sums_bytes(E);
    gg_status st = GG_OK;
    do
    {
        for (Edges &e : B.set)
        {
            if (st == GG_OK) st = gg_dev_alloc(g, (void **)&e.src, bytes);
            if (st == GG_OK) st = gg_dev_alloc(g, (void **)&e.dst, bytes);
            if (st == GG_OK && weighted) st = gg_dev_alloc(g, (void **)&e.w, bytes);
        }
        if (st == GG_OK) st = gg_dev_alloc(g, (void **)&B.counts, counts_bytes);
        if (st == GG_OK) st = gg_dev_alloc(g, (void **)&B.sums, sums_bytes);
        if (st == GG_OK) st = gg_dev_alloc(g, (void **)&B.flags, 16);
        if (st != GG_OK) break;
        if (cudaMemsetAsync(B.flags, 0, 16, s) != cudaSuccess)
        {
            st = gg_fail(GG_ERR_CUDA, "cudaMemsetAsync");
            break;
        }
        Edges input;
        input.src = const_cast<uint32_t *>(src);
        input.dst = const_cast<uint32_t *>(dst);
        input.w = weighted ? const_cast<float *>(w) : nullptr;
        if ((st = build_directions(g, B, input, need_out, need_in, weighted && (what & GG_MAP_OUT_W),
                                   weighted && (what & GG_MAP_IN_W), s)) != GG_OK)
            break;
        if (!need_out)
        {
            /* the CSR was only the degree source */
            if (cudaStreamSynchronize(s) != cudaSuccess)
            {
                st = gg_fail(GG_ERR_CUDA, "cudaStreamSynchronize");
                break;
            }
            gg_dev_free(g, g->out_off, ((size_t)V + 1) * 4);
            g->out_off = nullptr;
        }
        unsigned int flags[2] = {0u, 0u};
        if ((st = gg_wait(s)) != GG_OK) break; /* bounded, before a copy to pageable memory */
        if (cudaMemcpyAsync(flags, B.flags, 8, cudaMemcpyDeviceToHost, s) != cudaSuccess)
        {
            st = gg_fail(GG_ERR_CUDA, "cudaMemcpyAsync");
            break;
        }
        if ((st = gg_wait(s)) != GG_OK) break;
        if (flags[0])
            st = gg_fail(GG_ERR_INVALID, "edge list has a vertex id >= num_vertices");
        else if (weighted)
            memcpy(&g->max_weight, &flags[1], 4); /* for the host copy's max_weight */
    } while (false);
    gg_wait(s);
    for (Edges &e : B.set)
    {
        gg_dev_free(g, e.src, bytes);
        gg_dev_free(g, e.dst, bytes);
        gg_dev_free(g, e.w, bytes);
    }
    gg_dev_free(g, B.counts, counts_bytes);
    gg_dev_free(g, B.sums, sums_bytes);
    gg_dev_free(g, B.flags, 16);
    if (st == GG_OK && !weighted)
    {
        if (what & GG_MAP_OUT_W) st = gg_fill_constant_weights(g, &g->out_w, E, s);
        if (st == GG_OK && (what & GG_MAP_IN_W)) st = gg_fill_constant_weights(g, &g->in_w, E, s);
        if (st == GG_OK) st = gg_wait(s);
    }
    if (st == GG_OK) g->what = what | (g->in_off ? GG_MAP_IN : 0u) | (g->out_off ? GG_MAP_OUT : 0u);
    return st;
}

/* ---- degree-based relabelling (the reference's -l modes) ------------------
 *
 * The reference lists its relabelling modes (README.md:362-378: 1
 * out-degree, 2 in-degree, 3 (in+out)-degree, 4/5 DBG out/in, 6/7 HUBSort
 * out/in, 8/9 HUBCluster out/in, 10 random, 11 load from file); their code is
 * in the absent OpenGraph submodule.  Each mode here is the published
 * algorithm as one sort key per vertex, (key << b) | id, sorted by the radix
 * sort above, so ties keep the original order:
 *   degree (1-3)    descending degree
 *   DBG (4/5)       degree-based grouping (Faldu et al., IISWC 2019): eight
 *                   groups, group k >= 1 holding degrees in
 *                   [avg/2 * 2^(k-1), avg/2 * 2^k) (the last one open), group
 *                   0 the rest; hotter groups first, original order inside
 *   HUBSort (6/7)   hubs (degree > avg) by descending degree, then the other
 *                   vertices in original order (Zhang et al., 2017)
 *   HUBCluster (8/9) hubs first, then the others, both in original order
 *   random (10)     SplitMix64(seed ^ id), ties by id
 * avg = E / V.  The result is label[orig] = new. */

namespace {

__global__ void k_degree_count(const uint32_t *__restrict__ ids, uint64_t n, uint32_t V, uint32_t *deg, uint32_t *bad)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    {
        const uint32_t v = ids[i];
        if (v < V)
            atomicAdd(deg + v, 1u);
        else
            atomicOr(bad, 1u);
    }
}

__device__ __forceinline__ uint64_t mode_degree(uint32_t mode, const uint32_t *dout, const uint32_t *din, uint32_t v)
{
    switch (mode)
    {
    case 1: case 4: case 6: case 8: return dout[v];
    case 2: case 5: case 7: case 9: return din[v];
    case 3: return (uint64_t)dout[v] + din[v];
    default: return 0;
    }
}

__global__ void k_degree_max(const uint32_t *__restrict__ dout, const uint32_t *__restrict__ din, uint32_t V,
                             uint32_t mode, unsigned long long *out)
{
    unsigned long long m = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    {
        const unsigned long long d = mode_degree(mode, dout, din, v);
        m = d > m ? d : m;
    }
    for (int o = 16; o > 0; o >>= 1)
    {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, m, o);
        m = y > m ? y : m;
    }
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

__device__ __forceinline__ uint64_t relabel_key(uint32_t mode, uint64_t d, uint64_t dmax, uint64_t avg, uint64_t seed,
                                                uint32_t v)
{
    switch (mode)
    {
    case 1: case 2: case 3: return dmax - d;
    case 4: case 5:
    {
        const uint64_t r = 2 * d / (avg ? avg : 1);
        const uint32_t group = r ? min(7u, 64u - (uint32_t)__clzll((long long)r)) : 0u;
        return 7u - group;
    }
    case 6: case 7: return d > avg ? dmax - d : dmax + 1;
    case 8: case 9: return d > avg ? 0u : 1u;
    case 10:
    {
        uint64_t z = seed ^ v;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return (z ^ (z >> 31)) & 0xffffffffull;
    }
    default: return 0;
    }
}

__global__ void k_relabel_keys(const uint32_t *__restrict__ dout, const uint32_t *__restrict__ din, uint32_t V,
                               uint32_t mode, uint64_t dmax, uint64_t avg, uint64_t seed, int b, uint64_t *keys)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        keys[v] = (relabel_key(mode, mode_degree(mode, dout, din, v), dmax, avg, seed, v) << b) | v;
}

__global__ void k_labels_from_order(const uint64_t *__restrict__ keys, uint32_t V, uint64_t mask, uint32_t *label)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x)
        label[keys[i] & mask] = i;
}

/* checks label is a permutation of 0..V-1 (every new id hit once) */
__global__ void k_perm_hits(const uint32_t *__restrict__ label, uint32_t V, uint32_t *hits, uint32_t *bad)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    {
        const uint32_t l = label[v];
        if (l >= V || atomicAdd(hits + l, 1u) != 0u) atomicOr(bad, 1u);
    }
}

/* out may be ids (in place: each slot is read, then written, by one thread);
 * an id >= V stays as it is, for the build to report */
__global__ void k_apply_labels(const uint32_t *ids, uint64_t n, const uint32_t *__restrict__ label, uint32_t V, uint32_t *out)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    {
        const uint32_t v = ids[i];
        out[i] = v < V ? label[v] : v;
    }
}

int bits_for64(uint64_t x)
{
    int b = 0;
    while (b < 64 && (x >> b)) b++;
    return b;
}

/* a device scratch allocation freed at scope exit */
struct Scratch
{
    gg_graph *g;
    void *p = nullptr;
    size_t bytes = 0;
    Scratch(gg_graph *g_) : g(g_) {}
    gg_status alloc(size_t n)
    {
        bytes = n;
        return gg_dev_alloc(g, &p, n);
    }
    ~Scratch() { gg_dev_free(g, p, bytes); }
};

} // namespace

/* label[orig] = new for `mode` (1..10; 0 = identity) over device edge ids */
gg_status gg_relabel_device(gg_graph *g, uint32_t V, uint64_t E, const uint32_t *src, const uint32_t *dst,
                            uint32_t mode, uint64_t seed, uint32_t *label, cudaStream_t s)
{
    GgRange range("gg_relabel");
    if (mode > 10) return gg_fail(GG_ERR_INVALID, "relabelling mode must be 0..10 (11 takes labels from the caller)");
    Scratch degs(g), keys(g), tmp(g), counts(g), sums(g), flag(g);
    GG_CHECK(degs.alloc((size_t)V * 8 + 64));
    GG_CHECK(flag.alloc(64));
    uint32_t *dout = (uint32_t *)degs.p, *din = dout + V;
    GG_CUDA(cudaMemsetAsync(degs.p, 0, (size_t)V * 8 + 64, s));
    GG_CUDA(cudaMemsetAsync(flag.p, 0, 64, s));
    uint32_t *bad = (uint32_t *)flag.p;
    unsigned long long *dmax_d = (unsigned long long *)((char *)flag.p + 8);
    k_degree_count<<<grid_for(E, 256), 256, 0, s>>>(src, E, V, dout, bad);
    k_degree_count<<<grid_for(E, 256), 256, 0, s>>>(dst, E, V, din, bad);
    k_degree_max<<<grid_for(V, 256), 256, 0, s>>>(dout, din, V, mode, dmax_d);
    GG_CUDA(cudaGetLastError());
    unsigned long long hf[2] = {0, 0};
    GG_CHECK(gg_wait(s)); /* bounded, before a copy to pageable memory */
    GG_CUDA(cudaMemcpyAsync(hf, flag.p, 16, cudaMemcpyDeviceToHost, s));
    GG_CHECK(gg_wait(s));
    if (hf[0] & 0xffffffffull) return gg_fail(GG_ERR_INVALID, "edge list has a vertex id >= num_vertices");
    const uint64_t dmax = hf[1], avg = V ? E / V : 0;
    const int b = bits_for(V);
    int hi_bits = 0;
    switch (mode)
    {
    case 0: hi_bits = 0; break;
    case 1: case 2: case 3: hi_bits = bits_for64(dmax); break;
    case 4: case 5: hi_bits = 3; break;
    case 6: case 7: hi_bits = bits_for64(dmax + 1); break;
    case 8: case 9: hi_bits = 1; break;
    default: hi_bits = 32; break;
    }
    if (hi_bits + b > 64) return gg_fail(GG_ERR_INVALID, "degrees and ids do not fit one 64-bit sort key");
    GG_CHECK(keys.alloc((size_t)V * 8 + 16));
    GG_CHECK(tmp.alloc((size_t)V * 8 + 16));
    GG_CHECK(counts.alloc(sort_counts_bytes(V)));
    GG_CHECK(sums.alloc(sort_sums_bytes(V)));
    k_relabel_keys<<<grid_for(V, 256), 256, 0, s>>>(dout, din, V, mode, dmax, avg, seed, b, (uint64_t *)keys.p);
    GG_CUDA(cudaGetLastError());
    /* the words start in id order, so a stable sort of the key bits alone
     * leaves equal keys in id order */
    uint64_t *order = (uint64_t *)keys.p, *spare = (uint64_t *)tmp.p;
    for (int shift = b; V > 1 && shift < hi_bits + b; shift += 8)
    {
        SortPass<uint64_t> a{};
        a.key = order;
        a.okey = spare;
        a.n = V;
        a.shift = shift;
        GG_CHECK((sort_pass_run<uint64_t, 8, 0, false>(a, (uint32_t *)counts.p, (uint32_t *)sums.p, s)));
        std::swap(order, spare);
    }
    k_labels_from_order<<<grid_for(V, 256), 256, 0, s>>>(order, V, (1ull << b) - 1ull, label);
    GG_CUDA(cudaGetLastError());
    return gg_wait(s);
}

gg_status gg_check_permutation(gg_graph *g, const uint32_t *label, uint32_t V, cudaStream_t s)
{
    Scratch hits(g), flag(g);
    GG_CHECK(hits.alloc((size_t)V * 4 + 16));
    GG_CHECK(flag.alloc(16));
    GG_CUDA(cudaMemsetAsync(hits.p, 0, (size_t)V * 4 + 16, s));
    GG_CUDA(cudaMemsetAsync(flag.p, 0, 16, s));
    k_perm_hits<<<grid_for(V, 256), 256, 0, s>>>(label, V, (uint32_t *)hits.p, (uint32_t *)flag.p);
    GG_CUDA(cudaGetLastError());
    uint32_t bad = 0;
    GG_CHECK(gg_wait(s)); /* bounded, before a copy to pageable memory */
    GG_CUDA(cudaMemcpyAsync(&bad, flag.p, 4, cudaMemcpyDeviceToHost, s));
    GG_CHECK(gg_wait(s));
    if (bad) return gg_fail(GG_ERR_INVALID, "label array is not a permutation of 0..V-1");
    return GG_OK;
}

gg_status gg_apply_labels(const uint32_t *ids, uint64_t n, const uint32_t *label, uint32_t V, uint32_t *out, cudaStream_t s)
{
    k_apply_labels<<<grid_for(n, 256), 256, 0, s>>>(ids, n, label, V, out);
    GG_CUDA(cudaGetLastError());
    return GG_OK;
}
