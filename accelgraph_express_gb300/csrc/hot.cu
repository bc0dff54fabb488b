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

bool gg_hot_wanted(gg_graph *g, uint32_t flags, uint32_t hot, uint32_t cap, uint32_t iterations)
{
    if (flags & GG_PR_HOT_OFF) return false;
    if (flags & GG_PR_HOT_ON) return true;
    if (hot != 2) return hot == 1;
    if (g->E < GG_HOT_MIN_E) return false;
    if (g->hot_adj && g->hot_cap == cap) return true;
    const uint64_t its = g->plain_its + iterations;
    if (its > 2 && (its - 2) * g->E >= GG_HOT_PAYS) return true;
    g->plain_its = its;
    return false;
}

gg_status gg_hot_prepare(gg_graph *g, cudaStream_t s, uint32_t cap)
{
    if (!g->in_adj || !g->out_deg) return gg_fail(GG_ERR_INVALID, "the hot-vertex table needs GG_MAP_IN");
    const uint32_t V = g->V, E = g->E;
    if (!gg_hot_fits(V, E)) return gg_fail(GG_ERR_INVALID, "graph too large for flag-encoded ids");
    if (cap < 1 || cap > GG_HOT_ENTRIES) return gg_fail(GG_ERR_INVALID, "hot table capacity out of range");
    if (!g->hot_seg0)
    {
        uint32_t launches = 0;
        g->hot_tile = hot_tile_for(E);
        GG_CHECK(gg_rows_tiles(g, s, g->hot_tile, &g->hot_seg0, &g->hot_ntiles, &launches));
    }
    if (g->hot_adj && g->hot_cap == cap) return GG_OK;
    const uint32_t H = V < cap ? V : cap;
    void *hist, *slot_of;
    GG_CHECK(gg_work(g, 25, 65536 * 4, &hist));
    GG_CHECK(gg_work(g, 26, (size_t)V * 4, &slot_of));
    if (!g->hot_list) GG_CHECK(gg_dev_alloc(g, (void **)&g->hot_list, GG_HOT_LIST_BYTES));
    if (!g->hot_adj) GG_CHECK(gg_dev_alloc(g, (void **)&g->hot_adj, ((size_t)E + GG_EDGE_PAD) * 4));
    uint32_t *cnt = g->hot_list + GG_HOT_ENTRIES;
    g->hot_cap = 0; /* until the list and the ids are written */
    GG_CUDA(cudaMemsetAsync(hist, 0, 65536 * 4, s));
    GG_CUDA(cudaMemsetAsync(cnt, 0, 16, s));
    const int grid = gg_sm_count() * 8;
    k_deg_hist<<<gg_sm_count() * 2, 256, 0, s>>>(g->out_deg, V, (uint32_t *)hist);
    k_hot_threshold<<<1, 1024, 0, s>>>((const uint32_t *)hist, H, cnt);
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
