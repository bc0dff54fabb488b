/*
 * PageRank pull (FP32) of a small graph: every iteration in one launch, on one
 * SM or on one thread-block cluster of eight.
 *
 * A graph of a few thousand vertices needs well under a microsecond of work per
 * iteration, and two dependent launches take ~6 us for it.  Here the whole graph
 * sits in shared memory: each CTA holds an equal share of the in-neighbour ids
 * (16 bits, bit 15 marking the last edge of a row), a copy of all
 * contributions, and the sums, ranks and out-degrees of its share of the
 * vertices.  Per iteration:
 *   gather   every thread sums its own run of edges, ending rows as it meets
 *            their marks; one segmented scan per warp joins the runs.  A row's
 *            sum goes to the CTA that owns the vertex (distributed shared
 *            memory): stored when the row lies within one warp's edges, added
 *            otherwise
 *   barrier
 *   update   pageRank.c:1055-1069 and the contribution pass :1026-1033; the new
 *            contribution is stored into every CTA's copy
 *   barrier; the active count decides alike in all CTAs whether to stop
 * Bound by instruction issue (about ten instructions per edge and lane) and, in
 * a cluster, by its two barriers: one CTA up to SM_ONE edges, eight above.
 *
 * Measured per call of 20 iterations, R-MAT with 16 edges per vertex, against
 * the launches: 1.6K edges 144 -> 60 us, 16K 163 -> 96,
 * 64K 169 -> 116, 128K 176 -> 153 (some 43 us of each are the call's host work).
 */
#include <cuda_runtime.h>

#include <algorithm>

#include "gg_device.cuh"

namespace {

using namespace gg;

constexpr uint32_t SM_THREADS = 1024, SM_WARPS = SM_THREADS / 32;
constexpr uint32_t SM_END = 0x8000u, SM_ID = 0x7fffu;
constexpr size_t SM_LIMIT = 220 * 1024;

/* per-iteration record, as the launches of pr.cu write it */
struct SmallRec
{
    double err;
    uint32_t active, maxbits;
    float qinv;
    uint32_t pad;
};

struct SmallArgs
{
    const uint32_t *off, *adj, *outdeg;
    float *rank;
    SmallRec *rec;
    double *sum;
    uint32_t V, E, iterations;
    uint32_t run, eq, vq; /* edges per thread, edges and vertices per CTA */
    uint32_t rows_cap;  /* entries of the row list */
    float base, damp, init, eps_f;
    int divide;
};

/* shared memory of the run: this CTA's own, or the cluster's */
template <bool MULTI>
struct Mem
{
    static __device__ __forceinline__ uint32_t rank()
    {
        if constexpr (!MULTI) return 0u;
        uint32_t r;
        asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
        return r;
    }
    static __device__ __forceinline__ void sync()
    {
        if constexpr (MULTI)
            asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory");
        else
            __syncthreads();
    }
    /* this CTA's shared `addr` as an address in CTA `rank` */
    static __device__ __forceinline__ uint32_t at(uint32_t addr, uint32_t rank)
    {
        if constexpr (!MULTI) return addr;
        uint32_t r;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
        return r;
    }
    static __device__ __forceinline__ void store(uint32_t addr, float v)
    {
        if constexpr (MULTI)
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
        else
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
    }
    static __device__ __forceinline__ void add(uint32_t addr, float v)
    {
        if constexpr (MULTI)
            asm volatile("red.relaxed.cluster.shared::cluster.add.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
        else
            asm volatile("red.relaxed.cta.shared.add.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
    }
    static __device__ __forceinline__ void add(uint32_t addr, uint32_t v)
    {
        if constexpr (MULTI)
            asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
        else
            asm volatile("red.relaxed.cta.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
    }
};

/* exclusive sum over the block; total in *all (every thread calls it) */
__device__ __forceinline__ uint32_t block_excl(uint32_t v, uint32_t *all)
{
    __shared__ uint32_t part[SM_WARPS];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) part[w] = incl;
    __syncthreads();
    if (w == 0)
    {
        const uint32_t own = part[lane];
        uint32_t x = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        part[lane] = x - own;
        if (lane == 31) *all = x;
    }
    __syncthreads();
    const uint32_t r = part[w] + incl - v;
    __syncthreads();
    return r;
}

struct SmallShape
{
    size_t ids, rows, c, sums, rank, deg, total;
};
__host__ __device__ inline SmallShape small_shape(uint32_t V, uint32_t eq, uint32_t vq, uint32_t rows_cap)
{
    SmallShape s;
    s.c = 0;
    s.sums = s.c + ((size_t)V + 4) / 4 * 16;
    s.rank = s.sums + (size_t)vq * 4;
    s.deg = s.rank + (size_t)vq * 4;
    s.ids = (s.deg + (size_t)vq * 4 + 15) / 16 * 16;
    s.rows = (s.ids + (size_t)eq * 2 + 15) / 16 * 16;
    s.total = (s.rows + (size_t)rows_cap * 4 + 15) / 16 * 16;
    return s;
}

template <bool MULTI>
__global__ void __launch_bounds__(SM_THREADS, 1) k_pr_small(SmallArgs a)
{
    typedef Mem<MULTI> M;
    extern __shared__ __align__(1024) unsigned char gg_dyn[];
    __shared__ uint32_t s_total;
    __shared__ uint32_t s_act[3]; /* active counts of the run, iteration mod 3 */
    __shared__ bool s_open;       /* this CTA's first edge continues a row of the CTA before */
    const SmallShape sh = small_shape(a.V, a.eq, a.vq, a.rows_cap);
    float *c = reinterpret_cast<float *>(gg_dyn + sh.c);
    float *sums = reinterpret_cast<float *>(gg_dyn + sh.sums);
    float *rank = reinterpret_cast<float *>(gg_dyn + sh.rank);
    uint32_t *deg = reinterpret_cast<uint32_t *>(gg_dyn + sh.deg);
    uint16_t *ids = reinterpret_cast<uint16_t *>(gg_dyn + sh.ids);
    uint32_t *rows = reinterpret_cast<uint32_t *>(gg_dyn + sh.rows); /* addresses of the rows' sums */
    const uint32_t C = MULTI ? gridDim.x : 1u, me = M::rank();
    const uint32_t tid = threadIdx.x, lane = tid & 31, lt = (1u << lane) - 1u;
    const uint32_t e0 = min(me * a.eq, a.E), e1 = min(e0 + a.eq, a.E), ne = e1 - e0;
    const uint32_t v0 = min(me * a.vq, a.V), v1 = min(v0 + a.vq, a.V);
    /* the warps with edges; their threads' runs are padded with the id V,
     * whose contribution is 0 */
    const uint32_t wedges = 32 * a.run, nwork = (ne + wedges - 1) / wedges;
    const bool work = (tid >> 5) < nwork;

    for (uint32_t i = tid; i < nwork * wedges; i += SM_THREADS) ids[i] = (uint16_t)(i < ne ? a.adj[e0 + i] : a.V);
    for (uint32_t v = tid; v <= a.V; v += SM_THREADS)
    {
        const uint32_t d = v < a.V ? a.outdeg[v] : 0u;
        c[v] = d ? __fdiv_rn(a.init, __uint2float_rn(d)) : 0.0f;
        if (v >= v0 && v < v1)
        {
            deg[v - v0] = d;
            rank[v - v0] = a.init;
            sums[v - v0] = 0.0f;
        }
    }
    __syncthreads();
    /* the rows whose last edge is here, in order (the address of their sum),
     * and the marks of their last edges; a row still open at the end of this
     * CTA's edges follows them.  A thread looks at a run of consecutive rows */
    const uint32_t sums_at = (uint32_t)__cvta_generic_to_shared(sums), c_at = (uint32_t)__cvta_generic_to_shared(c);
    const uint32_t act_at = (uint32_t)__cvta_generic_to_shared(s_act);
    const uint32_t per = (a.V + SM_THREADS - 1) / SM_THREADS, r0 = min(tid * per, a.V), r1 = min(r0 + per, a.V);
    /* nonempty row [s, e) with edges here: it ends here, or is open at the end */
    auto here = [&](uint32_t s, uint32_t e) { return e > s && e > e0 && s < e1; };
    uint32_t mine = 0;
    for (uint32_t v = r0; v < r1; v++) mine += here(a.off[v], a.off[v + 1]);
    if (tid == 0) s_open = false;
    if (tid < 3) s_act[tid] = 0u;
    uint32_t at_row = block_excl(mine, &s_total);
    const uint32_t found = s_total;
    for (uint32_t v = r0; v < r1; v++)
    {
        const uint32_t s = a.off[v], e = a.off[v + 1];
        if (!here(s, e)) continue;
        if (e <= e1) ids[e - 1 - e0] |= (uint16_t)SM_END;
        if (s < e0) s_open = true; /* only the first row of the list */
        const uint32_t own = v / a.vq;
        rows[at_row++] = M::at(sums_at + (v - own * a.vq) * 4, own);
    }
    __syncthreads();
    /* the row ends before this thread's run, and whether the row of its
     * warp's first edge began before the warp */
    const uint16_t *run = ids + (size_t)tid * a.run;
    uint32_t n = 0;
    if (work)
        for (uint32_t j = 0; j < a.run; j++) n += run[j] >> 15;
    const uint32_t seg0 = block_excl(n, &s_total);
    bool open = false;
    if (work)
    {
        const uint32_t first = (tid & ~31u) * a.run;
        open = first ? !(ids[first - 1] & SM_END) : s_open;
    }
    M::sync();

    Sum2 err;
    uint32_t it = 0, total = 0;
    for (; it < a.iterations; it++)
    {
        if (work)
        {
            uint32_t seg = seg0;
            float sum = 0.0f, head = 0.0f; /* head: the sum at the first row end */
            bool ended = false;
            for (uint32_t j = 0; j < a.run; j += 4)
            {
                const uint2 q = *reinterpret_cast<const uint2 *>(run + j);
                const uint32_t u[4] = {q.x & 0xffffu, q.x >> 16, q.y & 0xffffu, q.y >> 16};
                float v[4];
#pragma unroll
                for (int i = 0; i < 4; i++) v[i] = c[u[i] & SM_ID];
#pragma unroll
                for (int i = 0; i < 4; i++)
                {
                    sum = __fadd_rn(sum, v[i]);
                    if (u[i] & SM_END)
                    {
                        /* the first one waits for what earlier lanes have of it */
                        if (ended)
                            M::store(rows[seg], sum);
                        else
                            head = sum;
                        ended = true;
                        seg++;
                        sum = 0.0f;
                    }
                }
            }
            /* open sums carried across lanes up to the next lane with a row end */
            const uint32_t ends = __ballot_sync(0xffffffffu, ended), le = ends & (lt | (1u << lane));
            const int hd = le ? 31 - __clz((int)le) : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const float y = __shfl_up_sync(0xffffffffu, sum, o);
                if ((int)lane - o >= hd) sum = __fadd_rn(sum, y);
            }
            const float before = __shfl_up_sync(0xffffffffu, sum, 1);
            if (ended)
            {
                const float s = lane ? __fadd_rn(head, before) : head;
                if (open && !(ends & lt))
                    M::add(rows[seg0], s);
                else
                    M::store(rows[seg0], s);
            }
            /* what the warp has of the row it leaves open; after the graph's
             * last edge there is none (only pads follow the last row end) */
            if (lane == 31 && seg < found && !(run[a.run - 1] & SM_END)) M::add(rows[seg], sum);
        }
        M::sync();
        err = Sum2();
        uint32_t act = 0;
        for (uint32_t i = tid; i < v1 - v0; i += SM_THREADS)
        {
            const float s = sums[i];
            sums[i] = 0.0f;
            const float nr = __fadd_rn(a.base, __fmul_rn(a.damp, s));
            const float e = fabsf(__fsub_rn(nr, rank[i]));
            rank[i] = nr;
            err.add(e);
            if (e >= a.eps_f) act++;
            const uint32_t d = deg[i];
            const float x = d ? __fdiv_rn(nr, __uint2float_rn(d)) : 0.0f;
            for (uint32_t k = 0; k < C; k++) M::store(M::at(c_at + (v0 + i) * 4, k), x);
        }
        /* counted in every CTA's own word; the word of the iteration after
         * next is cleared here, between its last reads (before the barrier
         * above) and its first adds (after the one below) */
        act = __reduce_add_sync(0xffffffffu, act);
        if (act && lane < C) M::add(M::at(act_at + (it % 3) * 4, lane), act);
        if (tid == 0) s_act[(it + 1) % 3] = 0u;
        M::sync();
        total = s_act[it % 3];
        if (me == 0 && tid == 0) a.rec[it].active = total;
        if (total == 0u)
        {
            it++;
            break;
        }
    }
    /* the residual is only wanted of the last iteration run */
    double e_sum;
    uint32_t none;
    block_sum2<SM_THREADS>(err, 0u, e_sum, none);
    if (tid == 0 && it > 0) atomicAdd(&a.rec[it - 1].err, e_sum);
    Sum2 rs;
    for (uint32_t i = tid; i < v1 - v0; i += SM_THREADS)
    {
        float r = rank[i];
        if (a.divide) r = __fdiv_rn(r, __uint2float_rn(a.V));
        a.rank[v0 + i] = r;
        rs.add(r);
    }
    double t_sum;
    block_sum2<SM_THREADS>(rs, 0u, t_sum, none);
    if (tid == 0 && t_sum != 0.0) atomicAdd(a.sum, t_sum);
    M::sync(); /* no CTA leaves while another may still write its memory */
}

/* One CTA up to this many edges, a cluster of eight above: a cluster's two
 * barriers and remote stores cost about a microsecond per iteration, one SM's
 * issue slots as much per 8K edges.  Per call of 20 iterations, one CTA /
 * clusters of 2 / 4 / 8: 4.8K edges 74 / 88 / 85 / 85 us, 16K 96 / 103 / 101 /
 * 98, 32K 163 (the launches) / 121 / 109 / 117, 64K - / 165 / 134 / 120. */
constexpr uint32_t SM_ONE = 16384, SM_CLUSTER = 8;
/* Edges per thread above which the launches are faster: 128K edges (20 per
 * thread) 155 us against 168, 192K (28) 183 against 178. */
constexpr uint32_t SM_RUN_MAX = 20;

/* the CTAs and shares for a graph, or false when it does not fit or is better
 * left to the launches */
bool small_plan(uint32_t V, uint32_t E, SmallArgs &a, uint32_t &C, size_t &smem)
{
    if (V == 0 || V >= SM_ID || E == 0 || E > SM_CLUSTER * SM_THREADS * SM_RUN_MAX) return false;
    C = E <= SM_ONE ? 1 : SM_CLUSTER;
    /* 4, 12, 20, ...: threads read their runs four ids at a time, and an odd
     * number of 8-byte words between threads spreads them over the banks */
    const uint32_t need = (E + C * SM_THREADS - 1) / (C * SM_THREADS);
    a.run = need <= 4 ? 4 : 4 + (need - 4 + 7) / 8 * 8;
    if (a.run > SM_RUN_MAX) return false;
    /* whole warps' worth of edges per CTA */
    const uint32_t wedges = 32 * a.run;
    a.eq = ((E + C - 1) / C + wedges - 1) / wedges * wedges;
    a.vq = ((V + C - 1) / C + 3) / 4 * 4;
    a.rows_cap = std::min(V, a.eq) + 1;
    smem = small_shape(V, a.eq, a.vq, a.rows_cap).total;
    return smem <= SM_LIMIT;
}

} // namespace

bool gg_small_fits(const gg_graph *g)
{
    SmallArgs a{};
    uint32_t C;
    size_t smem;
    return small_plan(g->V, g->E, a, C, smem);
}

gg_status gg_small_pagerank(gg_graph *g, const gg_pr_params *p, float *rank, void *rec, double *sum, float base,
                            float init, float eps_f, cudaStream_t s)
{
    SmallArgs a{};
    uint32_t C;
    size_t smem;
    if (!small_plan(g->V, g->E, a, C, smem)) return gg_fail(GG_ERR_INVALID, "graph too large for the cluster kernel");
    a.off = g->in_off; a.adj = g->in_adj; a.outdeg = g->out_deg;
    a.rank = rank; a.rec = (SmallRec *)rec; a.sum = sum;
    a.V = g->V; a.E = g->E; a.iterations = p->max_iterations;
    a.base = base; a.damp = p->damp; a.init = init; a.eps_f = eps_f;
    a.divide = p->init_one_over_n ? 0 : 1;
    void (*fn)(SmallArgs) = C > 1 ? k_pr_small<true> : k_pr_small<false>;
    GG_CUDA(cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM_LIMIT));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(SM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GG_CUDA(cudaLaunchKernelEx(&cfg, fn, a));
    return GG_OK;
}
