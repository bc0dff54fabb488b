/*
 * Hot-vertex table of the pull gather: the GPU counterpart of the reference
 * FPGA's vertex cache (cu_vertex_cache_reuse_control.sv keeps frequently
 * read vertices on chip, marked through heat bits that EXTRACT_VALUE masks
 * off the neighbour ids).  Here the H vertices with the most out-edges -- the
 * contributions a pull gather reads most often -- get slots 0..H-1, and a
 * copy of the CSC neighbour ids carries them as 0x80000000 | slot, so a
 * gather kernel can serve those reads from a table in shared memory filled
 * per launch.  On R-MAT graphs in natural order the 32K hottest of 16.7M
 * vertices receive 37% of all gathers, the 64K hottest 48%.
 *
 * Preparation, once per mapping, without a wait on the host: a histogram of
 * out-degrees (clamped at 65535) gives the threshold degree T; vertices above
 * T and, up to H, vertices at T take slots by atomics (which of the ties win
 * does not matter: the table holds exact copies); one pass over the CSC
 * writes the encoded ids.  The gather (gg_hot.cuh) finds rows through the ids
 * themselves: passes over the row offsets list the rows that have edges, mark
 * each one's last edge in the encoded ids, and note for every tile of edges which
 * row end comes first in it.
 */
#include <cuda_runtime.h>

#include "gg_hot.cuh"

namespace {

constexpr uint32_t NO_SLOT = 0xffffffffu;

using gg::hot_taken;

/* out-degree histogram (clamped at 65535): degrees below 4096 -- nearly all
 * of them on skewed graphs, so global atomics on those bins would serialise
 * -- are counted in shared memory per CTA and flushed once */
__global__ void __launch_bounds__(256) k_deg_hist(const uint32_t *__restrict__ outdeg, uint32_t V, uint32_t *hist)
{
    constexpr uint32_t LOW = 4096;
    __shared__ uint32_t s[LOW];
    for (uint32_t i = threadIdx.x; i < LOW; i += blockDim.x) s[i] = 0;
    __syncthreads();
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    {
        const uint32_t d = min(outdeg[v], 65535u);
        if (d < LOW)
            atomicAdd(&s[d], 1u);
        else
            atomicAdd(&hist[d], 1u);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < LOW; i += blockDim.x)
        if (s[i]) atomicAdd(&hist[i], s[i]);
}

/* cnt[0] = vertices above T, cnt[1] = at T, cnt[2] = T, cnt[3] = vertices
 * above T by the histogram: T is the degree with fewer than H vertices above
 * it.  One block: its warps sum 2,048 bins each, then the chunk in which the
 * count from the top reaches H is scanned bin by bin.  (Read back and
 * scanned on the host, with a second read for the slots taken, preparation
 * took 160 us longer than its kernels: 247 -> 89 us at R-MAT-20.) */
__global__ void __launch_bounds__(1024) k_hot_threshold(const uint32_t *__restrict__ hist, uint32_t H, uint32_t *cnt)
{
    __shared__ uint32_t s_sum[32], s_chunk, s_before;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    /* chunk c holds bins 65535 - 2048 c downwards */
    uint32_t n = 0;
#pragma unroll 8
    for (uint32_t k = 0; k < 64; k++) n += hist[65535u - (w * 2048u + k * 32u + lane)];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (lane == 0) s_sum[w] = n;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        uint32_t c = 0, before = 0;
        while (c < 31u && before + s_sum[c] < H) before += s_sum[c++];
        s_chunk = c;
        s_before = before;
    }
    __syncthreads();
    const uint32_t top = 65535u - s_chunk * 2048u - threadIdx.x * 2u; /* this thread's bins: top, top - 1 */
    const uint32_t n0 = hist[top], n1 = hist[top - 1u];
    uint32_t incl = n0 + n1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) s_sum[w] = incl;
    __syncthreads();
    uint32_t before = s_before;
    for (uint32_t k = 0; k < w; k++) before += s_sum[k];
    before += incl - n0 - n1;
    /* the first bin from the top at which the count reaches H; bin 0 if none */
    if (before < H && before + n0 >= H)
    {
        cnt[2] = top;
        cnt[3] = before;
    }
    else if (before + n0 < H && (before + n0 + n1 >= H || top == 1u))
    {
        cnt[2] = top - 1u;
        cnt[3] = before + n0;
    }
}

__global__ void k_hot_mark(const uint32_t *__restrict__ outdeg, uint32_t V, uint32_t H, uint32_t *slot_of,
                           uint32_t *hot_list, uint32_t *cnt)
{
    const uint32_t T = cnt[2], above = cnt[3];
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    {
        const uint32_t d = min(outdeg[v], 65535u);
        uint32_t slot = NO_SLOT;
        if (d > T)
            slot = atomicAdd(&cnt[0], 1u);
        else if (d == T && T > 0)
        {
            const uint32_t k = atomicAdd(&cnt[1], 1u);
            if (above + k < H) slot = above + k;
        }
        slot_of[v] = slot;
        if (slot != NO_SLOT) hot_list[slot] = v;
    }
}

/* ids -> encoded ids.  Every CTA first puts the hot vertices into a Bloom
 * filter in shared memory (BLOOM_BITS bits, two hashes): an id whose two
 * bits are not both set is not hot and is copied as it is, and only the
 * others (the hot ones, 37-48% of the edges of R-MAT-24, and rare false
 * positives) read their slot.  Reading the slot of every id at random had
 * made the pass ~0.9 ms of L2 requests at R-MAT-24.  The ids stream in
 * 16-byte loads, four in flight per thread. */
constexpr uint32_t BLOOM_LOG2 = 20;
constexpr uint32_t BLOOM_BITS = 1u << BLOOM_LOG2; /* 128 KB: 1.4% false positives at 64K hot vertices */

__device__ __forceinline__ uint32_t bloom_h1(uint32_t u) { return (u * 0x9E3779B1u) >> (32 - BLOOM_LOG2); }
__device__ __forceinline__ uint32_t bloom_h2(uint32_t u) { return (u * 0x85EBCA77u + 0x165667B1u) >> (32 - BLOOM_LOG2); }

__global__ void __launch_bounds__(1024) k_hot_encode(const uint32_t *__restrict__ adj, uint64_t n,
                                                     const uint32_t *__restrict__ slot_of,
                                                     const uint32_t *__restrict__ hot_list,
                                                     const uint32_t *__restrict__ counters, uint32_t H, uint32_t cap,
                                                     uint32_t *__restrict__ out)
{
    extern __shared__ uint32_t bloom[];
    for (uint32_t i = threadIdx.x; i < BLOOM_BITS / 32; i += blockDim.x) bloom[i] = 0u;
    __syncthreads();
    const uint32_t nh = hot_taken(counters, H);
    for (uint32_t i = threadIdx.x; i < nh; i += blockDim.x)
    {
        const uint32_t u = hot_list[i], b1 = bloom_h1(u), b2 = bloom_h2(u);
        atomicOr(&bloom[b1 >> 5], 1u << (b1 & 31));
        atomicOr(&bloom[b2 >> 5], 1u << (b2 & 31));
    }
    __syncthreads();
    auto enc = [&](uint32_t u) -> uint32_t {
        const uint32_t b1 = bloom_h1(u), b2 = bloom_h2(u);
        if (!((bloom[b1 >> 5] >> (b1 & 31)) & (bloom[b2 >> 5] >> (b2 & 31)) & 1u)) return u;
        const uint32_t sl = slot_of[u];
        return sl == NO_SLOT ? u : (GG_HOT_FLAG | sl);
    };
    const uint64_t nv = n / 4, stride = (uint64_t)gridDim.x * blockDim.x;
    const uint4 *a4 = reinterpret_cast<const uint4 *>(adj);
    uint4 *o4 = reinterpret_cast<uint4 *>(out);
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    for (; i + 3 * stride < nv; i += 4 * stride)
    {
        uint4 v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = __ldcs(a4 + i + k * stride);
#pragma unroll
        for (int k = 0; k < 4; k++)
        {
            v[k].x = enc(v[k].x);
            v[k].y = enc(v[k].y);
            v[k].z = enc(v[k].z);
            v[k].w = enc(v[k].w);
            o4[i + k * stride] = v[k];
        }
    }
    for (; i < nv; i += stride)
    {
        uint4 v = __ldcs(a4 + i);
        v.x = enc(v.x);
        v.y = enc(v.y);
        v.z = enc(v.z);
        v.w = enc(v.w);
        o4[i] = v;
    }
    /* the last n % 4 ids */
    if (blockIdx.x == 0 && threadIdx.x < n - nv * 4)
    {
        const uint64_t e = nv * 4 + threadIdx.x;
        out[e] = enc(adj[e]);
    }
    /* the pads after the last id read the table's zero entry */
    if (blockIdx.x == 0 && threadIdx.x < GG_EDGE_PAD) out[n + threadIdx.x] = GG_HOT_FLAG | cap;
}

/* What the choice between the gathers turns on (gg_hot_choose): SAMPLE_WINDOWS
 * windows of consecutive edges, evenly spaced.  out[0] += 32-byte sectors of the
 * values in each window (L1 misses of a CTA of the plain gather, whose warps take
 * about that many consecutive edges), out[1] += edges that the table would serve
 * (threshold degree in cnt[2]). */
constexpr uint32_t SAMPLE_WINDOWS = 304, SAMPLE_EDGES = GG_TILE_ITEMS * GG_TILE_WARPS, SAMPLE_SLOTS = 4096;
constexpr uint32_t SAMPLE_PER = 3, SAMPLE_NT = SAMPLE_EDGES / SAMPLE_PER;
static_assert(SAMPLE_NT * SAMPLE_PER == SAMPLE_EDGES && SAMPLE_NT % 32 == 0, "whole warps");

/* E is at least GG_HOT_MIN_E: the windows do not overlap */
__global__ void __launch_bounds__(SAMPLE_NT) k_hot_sample(const uint32_t *__restrict__ adj, uint32_t E,
                                                    const uint32_t *__restrict__ outdeg,
                                                    const uint32_t *__restrict__ cnt, uint32_t shift, uint32_t *out)
{
    __shared__ uint32_t seen[SAMPLE_SLOTS];
    const uint32_t T = cnt[2], e0 = (uint32_t)((uint64_t)E * blockIdx.x / gridDim.x) + threadIdx.x;
    uint32_t u[SAMPLE_PER], fresh = 0, served = 0;
#pragma unroll
    for (uint32_t k = 0; k < SAMPLE_PER; k++) u[k] = adj[e0 + k * SAMPLE_NT];
    for (uint32_t i = threadIdx.x; i < SAMPLE_SLOTS; i += SAMPLE_NT) seen[i] = NO_SLOT; /* no sector: ids are below 2^30 */
#pragma unroll
    for (uint32_t k = 0; k < SAMPLE_PER; k++) served += min(outdeg[u[k]], 65535u) > T;
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < SAMPLE_PER; k++)
    {
        const uint32_t sector = u[k] >> shift;
        uint32_t at = (sector * 0x9E3779B1u) >> 20;
        for (;;) /* at most SAMPLE_EDGES of SAMPLE_SLOTS are taken */
        {
            const uint32_t was = atomicCAS(&seen[at], NO_SLOT, sector);
            fresh += was == NO_SLOT;
            if (was == NO_SLOT || was == sector) break;
            at = (at + 1u) & (SAMPLE_SLOTS - 1u);
        }
    }
    fresh = __reduce_add_sync(0xffffffffu, fresh);
    served = __reduce_add_sync(0xffffffffu, served);
    if ((threadIdx.x & 31) == 0)
    {
        atomicAdd(out, fresh);
        atomicAdd(out + 1, served);
    }
}

/* ---- rows with edges ---- */

constexpr uint32_t ROW_BLOCK = 256, ROW_PER = 8, ROW_TILE = ROW_BLOCK * ROW_PER;

/* inclusive sum over the block of one value per thread; total in *all */
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t *all)
{
    __shared__ uint32_t part[ROW_BLOCK / 32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (uint32_t)o) v += y;
    }
    if (lane == 31) part[w] = v;
    __syncthreads();
    uint32_t base = 0, total = 0;
    for (uint32_t k = 0; k < ROW_BLOCK / 32; k++)
    {
        if (k < w) base += part[k];
        total += part[k];
    }
    __syncthreads();
    *all = total;
    return v + base;
}

/* thread t of a block takes rows first + t, first + t + 256, ... so that the
 * offsets are read coalesced; bit k of the result: row first + t + 256 k has
 * edges */
__device__ __forceinline__ uint32_t rows_with_edges(const uint32_t *__restrict__ off, uint32_t V, uint32_t first)
{
    uint32_t bits = 0;
#pragma unroll
    for (uint32_t k = 0; k < ROW_PER; k++)
    {
        const uint32_t v = first + k * ROW_BLOCK + threadIdx.x;
        if (v < V && off[v + 1] > off[v]) bits |= 1u << k;
    }
    return bits;
}

/* rows with edges per block of ROW_TILE rows; the block that finishes last
 * turns the counts into their exclusive prefix, in place, and stores the total
 * (ticket: zeroed before the launch) */
__global__ void __launch_bounds__(ROW_BLOCK) k_rows_count(const uint32_t *__restrict__ off, uint32_t V,
                                                          uint32_t *counts, uint32_t *ticket, uint32_t *total)
{
    __shared__ bool s_last;
    uint32_t all;
    block_scan((uint32_t)__popc(rows_with_edges(off, V, blockIdx.x * ROW_TILE)), &all);
    if (threadIdx.x == 0)
    {
        counts[blockIdx.x] = all;
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const uint32_t n = gridDim.x;
    uint32_t base = 0;
    for (uint32_t at = 0; at < n; at += ROW_TILE)
    {
        uint32_t c[ROW_PER], sum = 0;
#pragma unroll
        for (uint32_t k = 0; k < ROW_PER; k++)
        {
            const uint32_t i = at + threadIdx.x * ROW_PER + k;
            c[k] = i < n ? __ldcg(counts + i) : 0u;
            sum += c[k];
        }
        uint32_t run = base + block_scan(sum, &all) - sum;
#pragma unroll
        for (uint32_t k = 0; k < ROW_PER; k++)
        {
            const uint32_t i = at + threadIdx.x * ROW_PER + k;
            if (i < n) counts[i] = run;
            run += c[k];
        }
        base += all;
    }
    if (threadIdx.x == 0) *total = base;
}

/* tiles whose first edge lies in row r = [a, b) (r-th with edges) */
__device__ __forceinline__ void row_tiles(uint32_t a, uint32_t b, uint32_t r, uint32_t tile, uint32_t *seg0)
{
    for (uint64_t t = ((uint64_t)a + tile - 1) / tile; t * tile < b; t++) seg0[t] = r | (t * tile > a ? 0x80000000u : 0u);
}

/* rows[r] = the r-th row with edges, then the pads; seg0 of every tile */
__global__ void __launch_bounds__(ROW_BLOCK) k_rows_write(const uint32_t *__restrict__ off, uint32_t V,
                                                          const uint32_t *__restrict__ base, uint32_t *__restrict__ rows,
                                                          uint32_t *__restrict__ seg0, uint32_t tile)
{
    const uint32_t first = blockIdx.x * ROW_TILE;
    uint32_t r0 = base[blockIdx.x];
    for (uint32_t k = 0; k < ROW_PER; k++)
    {
        const uint32_t v = first + k * ROW_BLOCK + threadIdx.x;
        uint32_t a = 0, b = 0;
        if (v < V)
        {
            a = off[v];
            b = off[v + 1];
        }
        uint32_t all;
        const uint32_t r = r0 + block_scan(b > a ? 1u : 0u, &all) - 1u;
        if (b > a)
        {
            rows[r] = v;
            row_tiles(a, b, r, tile, seg0);
        }
        r0 += all;
    }
    const uint32_t total = rows[V + GG_ROW_PAD];
    if (blockIdx.x == 0 && threadIdx.x < GG_ROW_PAD) rows[total + threadIdx.x] = V;
}

/* seg0 alone, for another tile size */
__global__ void k_rows_seg0(const uint32_t *__restrict__ off, uint32_t V, const uint32_t *__restrict__ rows,
                            uint32_t *__restrict__ seg0, uint32_t tile)
{
    const uint32_t n = rows[V + GG_ROW_PAD];
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
        row_tiles(off[rows[r]], off[rows[r] + 1], r, tile, seg0);
}

/* the last edge of every row in the encoded ids */
__global__ void k_rows_mark(const uint32_t *__restrict__ off, uint32_t V, uint32_t *__restrict__ ids)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    {
        const uint32_t a = off[v], b = off[v + 1];
        if (b > a) ids[b - 1] |= GG_HOT_END;
    }
}

} // namespace

gg_status gg_rows_tiles(gg_graph *g, cudaStream_t s, uint32_t tile, uint32_t **seg0, uint32_t *ntiles,
                        uint32_t *launches)
{
    const uint32_t V = g->V, E = g->E;
    const uint32_t nt = (uint32_t)(((uint64_t)E + tile - 1) / tile), nb = (uint32_t)(((uint64_t)V + ROW_TILE - 1) / ROW_TILE);
    /* all that is allocated here, before any of it is set on the mapping */
    const bool list = !g->rows_list;
    const size_t seg_bytes = (size_t)nt * 4;
    void *counts = nullptr, *seg = nullptr, *rows = g->rows_list;
    if (list) GG_CHECK(gg_work(g, 33, ((size_t)nb + 4) * 4, &counts));
    GG_CHECK(gg_dev_alloc(g, &seg, seg_bytes));
    if (list)
    {
        const gg_status st = gg_dev_alloc(g, &rows, ((size_t)V + GG_ROW_PAD + 4) * 4);
        if (st != GG_OK)
        {
            gg_dev_free(g, seg, seg_bytes);
            return st;
        }
    }
    cudaError_t e = cudaSuccess;
    uint32_t *r = (uint32_t *)rows;
    if (list)
    {
        uint32_t *ticket = (uint32_t *)counts + nb;
        e = cudaMemsetAsync(ticket, 0, 4, s);
        if (e == cudaSuccess)
        {
            k_rows_count<<<nb, ROW_BLOCK, 0, s>>>(g->in_off, V, (uint32_t *)counts, ticket, r + V + GG_ROW_PAD);
            k_rows_write<<<nb, ROW_BLOCK, 0, s>>>(g->in_off, V, (const uint32_t *)counts, r, (uint32_t *)seg, tile);
        }
    }
    else
        k_rows_seg0<<<gg_sm_count() * 8, 256, 0, s>>>(g->in_off, V, r, (uint32_t *)seg, tile);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess)
    {
        gg_dev_free(g, seg, seg_bytes);
        if (list) gg_dev_free(g, rows, ((size_t)V + GG_ROW_PAD + 4) * 4);
        return gg_cuda_fail(e, "rows and tiles");
    }
    g->rows_list = r;
    *seg0 = (uint32_t *)seg;
    *ntiles = nt;
    *launches += list ? 2 : 1;
    return GG_OK;
}

/* edges per tile: the tiles are dealt round robin to 32 warps on every SM, so
 * a few tiles per warp leave the last round nearly empty (R-MAT-20, 3,450
 * edges per warp: 49 us with tiles of 2048) and many cost an atomic add each.
 * At least eight tiles per warp, from 256 to GG_HOT_TILE_MAX edges. */
static uint32_t hot_tile_for(uint32_t E)
{
    uint32_t tile = 256;
    while (tile < GG_HOT_TILE_MAX && (uint64_t)tile * 2 * 8 * 32 * (uint32_t)gg_sm_count() <= E) tile *= 2;
    return tile;
}

/* threshold degree of a table of `cap` entries, behind the hot list */
static gg_status hot_threshold(gg_graph *g, cudaStream_t s, uint32_t cap)
{
    if (g->hot_threshold == cap) return GG_OK;
    const uint32_t V = g->V, H = V < cap ? V : cap;
    void *hist;
    GG_CHECK(gg_work(g, 25, 65536 * 4, &hist));
    if (!g->hot_list) GG_CHECK(gg_dev_alloc(g, (void **)&g->hot_list, GG_HOT_LIST_BYTES));
    g->hot_threshold = 0;
    GG_CUDA(cudaMemsetAsync(hist, 0, 65536 * 4, s));
    k_deg_hist<<<gg_sm_count() * 2, 256, 0, s>>>(g->out_deg, V, (uint32_t *)hist);
    k_hot_threshold<<<1, 1024, 0, s>>>((const uint32_t *)hist, H, g->hot_list + GG_HOT_ENTRIES);
    GG_CUDA(cudaGetLastError());
    g->hot_threshold = cap;
    return GG_OK;
}

/* the rows with edges and the first row end of every tile */
static gg_status hot_rows(gg_graph *g, cudaStream_t s)
{
    uint32_t launches = 0;
    if (g->hot_seg0) return GG_OK;
    g->hot_tile = hot_tile_for(g->E);
    return gg_rows_tiles(g, s, g->hot_tile, &g->hot_seg0, &g->hot_ntiles, &launches);
}

/* the encoded ids' memory, and a slot per vertex */
static gg_status hot_memory(gg_graph *g, void **slot_of)
{
    GG_CHECK(gg_work(g, 26, (size_t)g->V * 4, slot_of));
    if (!g->hot_adj) GG_CHECK(gg_dev_alloc(g, (void **)&g->hot_adj, ((size_t)g->E + GG_EDGE_PAD) * 4));
    return GG_OK;
}

/* the table's encoded ids and list, and the rows and tiles of its gathers */
static gg_status hot_prepare(gg_graph *g, cudaStream_t s, uint32_t cap)
{
    const uint32_t V = g->V, E = g->E, H = V < cap ? V : cap;
    GG_CHECK(hot_rows(g, s));
    if (g->hot_adj && g->hot_cap == cap) return GG_OK;
    GG_CHECK(hot_threshold(g, s, cap));
    void *slot_of;
    GG_CHECK(hot_memory(g, &slot_of));
    uint32_t *cnt = g->hot_list + GG_HOT_ENTRIES;
    g->hot_cap = 0; /* until the list and the ids are written */
    GG_CUDA(cudaMemsetAsync(cnt, 0, 8, s));
    const int grid = gg_sm_count() * 8;
    k_hot_mark<<<grid, 256, 0, s>>>(g->out_deg, V, H, (uint32_t *)slot_of, g->hot_list, cnt);
    /* one CTA of 1024 threads per SM (60 registers a thread); adj and out are
     * whole allocations, 16-byte aligned for the vector loads */
    GG_CUDA(cudaFuncSetAttribute(k_hot_encode, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(BLOOM_BITS / 8)));
    k_hot_encode<<<gg_sm_count(), 1024, BLOOM_BITS / 8, s>>>(g->in_adj, (uint64_t)E, (const uint32_t *)slot_of,
                                                              g->hot_list, cnt, H, cap, g->hot_adj);
    k_rows_mark<<<grid, 256, 0, s>>>(g->in_off, V, g->hot_adj);
    GG_CUDA(cudaGetLastError());
    g->plain_its = 0;
    g->hot_slots = H;
    g->hot_cap = cap;
    return GG_OK;
}

/* Whether the plain gather is the faster one on this graph.  It reads through L1,
 * the table's does not (gg_hot.cuh), so it wins where most neighbours of nearby
 * rows lie close together: meshes, orders with locality, unions of small graphs.
 * With h the share of a window's edges that find their sector read already and s
 * the share that the table serves, a gather takes, in ps per edge (PageRank /
 * SpMV),
 *     plain   2.55 / 2.9  +  4.0 / 4.5 V / E  +  1.8 / 2.3 (1 - h)^2
 *     table   3.73 / 4.0 (1 - s)  +  0.52 / 0 h
 * Measured us per gather of 67M edges between 4.2M vertices, plain : table.
 * PageRank: neighbours within 1,000 ids (h 0.78) 191 : 271, 3,000 (0.49) 220 : 251,
 * 10,000 (0.20) 265 : 250, uniform random (0) 295 : 252, R-MAT (0.14, s 0.48) 232 :
 * 139, half R-MAT half within 1,000 (0.40, 0.25) 225 : 194.  SpMV: within 1,000 215 :
 * 269, blocks of 4,096 (0.60) 226 : 266, within 10,000 312 : 266; a mesh of 16.7M
 * vertices (0.90) 267 : 252. */
static bool plain_is_faster(double V, double E, double h, double s, bool weighted)
{
    const double miss = (1.0 - h) * (1.0 - h);
    return weighted ? 2.9 + 4.5 * V / E + 2.3 * miss < 4.0 * (1.0 - s)
                    : 2.55 + 4.0 * V / E + 1.8 * miss < 3.73 * (1.0 - s) + 0.52 * h;
}

gg_status gg_hot_choose(gg_graph *g, cudaStream_t s, const gg_hot_ask &ask, gg_pull_shape *shape, bool *use)
{
    *use = false;
    if ((ask.flags & GG_PR_HOT_OFF) || !gg_hot_fits(g->V, g->E)) return GG_OK;
    if (!(ask.flags & GG_PR_HOT_ON) && shape->hot == 0) return GG_OK;
    const bool by_rule = !(ask.flags & GG_PR_HOT_ON) && shape->hot == 2;
    if (by_rule && g->E < GG_HOT_MIN_E) return GG_OK;
    if (!g->in_adj || !g->out_deg) return gg_fail(GG_ERR_INVALID, "the hot-vertex table needs GG_MAP_IN");
    if (by_rule)
    {
        uint32_t shift = 5; /* ids to sectors of 32 bytes */
        while ((32u >> shift) < ask.bytes) shift--;
        uint8_t &choice = g->hot_choice[ask.weighted ? 1 : 0][shift];
        if (choice != GG_HOT_PLAIN && !(g->hot_adj && g->hot_cap == ask.cap))
        {
            const uint64_t its = g->plain_its + ask.iterations;
            if (its <= 2 || (its - 2) * g->E < GG_HOT_PAYS)
            {
                g->plain_its = its;
                return GG_OK;
            }
        }
        if (choice == GG_HOT_UNKNOWN)
        {
            /* the host allocates, and waits for the sample, beside the passes over
             * the degrees and rows */
            void *pin, *slot_of;
            const bool had = g->hot_adj != nullptr;
            GG_CHECK(gg_pinned(g, 64, &pin));
            GG_CHECK(hot_threshold(g, s, ask.cap));
            uint32_t *cnt = g->hot_list + GG_HOT_ENTRIES, *out = cnt + 4;
            GG_CUDA(cudaMemsetAsync(out, 0, 8, s));
            k_hot_sample<<<SAMPLE_WINDOWS, SAMPLE_NT, 0, s>>>(g->in_adj, g->E, g->out_deg, cnt, shift, out);
            GG_CUDA(cudaGetLastError());
            GG_CUDA(cudaMemcpyAsync(pin, out, 8, cudaMemcpyDeviceToHost, s));
            GG_CUDA(cudaEventRecord(g->ev_begin, s));
            GG_CHECK(hot_rows(g, s));
            GG_CHECK(hot_memory(g, &slot_of));
            GG_CHECK(gg_wait_event(g->ev_begin));
            const volatile uint32_t *got = (const volatile uint32_t *)pin;
            const double n = (double)SAMPLE_WINDOWS * SAMPLE_EDGES;
            choice = plain_is_faster(g->V, g->E, 1.0 - got[0] / n, got[1] / n, ask.weighted) ? GG_HOT_PLAIN : GG_HOT_TABLE;
            if (choice == GG_HOT_PLAIN && !had)
            {
                gg_dev_free(g, g->hot_adj, ((size_t)g->E + GG_EDGE_PAD) * 4);
                g->hot_adj = nullptr;
            }
        }
        if (choice == GG_HOT_PLAIN)
        {
            shape->ctas = GG_PULL_CTAS_LOCAL;
            return GG_OK;
        }
    }
    GG_CHECK(hot_prepare(g, s, ask.cap));
    *use = true;
    return GG_OK;
}
