/*
 * PageRank pull (FP32) of a small graph: every iteration in one launch, on one
 * SM, on one thread-block cluster of eight or, further down, on the whole chip.
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
 * Measured per call of 20 iterations, R-MAT with 16 edges per vertex, ranks left on
 * the device, against the launches: 1.6K edges 137 -> 43 us, 16K 140 -> 76, 32K 142 ->
 * 101, 64K 144 -> 101, 96K 146 -> 126 (some 30 us of each are the call's host work).
 */
#include <cuda_runtime.h>

#include <algorithm>

#include "gg_device.cuh"

namespace {

using namespace gg;

constexpr uint32_t SM_THREADS = 1024, SM_WARPS = SM_THREADS / 32;
constexpr uint32_t SM_END = 0x8000u, SM_ID = 0x7fffu;
constexpr size_t SM_LIMIT = 220 * 1024; /* graphs up to this are taken */
constexpr size_t SM_MOST = 226 * 1024;  /* dynamic shared memory beside 1 KB of static */

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
    uint32_t keep;      /* 1: the ranks an iteration began with stay in shared memory */
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

/* four ids of a thread's run */
__device__ __forceinline__ void load4(const uint16_t *p, uint32_t *u)
{
    const uint2 q = *reinterpret_cast<const uint2 *>(p);
    u[0] = q.x & 0xffffu;
    u[1] = q.x >> 16;
    u[2] = q.y & 0xffffu;
    u[3] = q.y >> 16;
}
__device__ __forceinline__ void load4(const uint32_t *p, uint32_t *u)
{
    const uint4 q = *reinterpret_cast<const uint4 *>(p);
    u[0] = q.x;
    u[1] = q.y;
    u[2] = q.z;
    u[3] = q.w;
}

/* a warp's sums: every thread adds up its run of n ids (the top bit marks a
 * row's last edge), storing rows that begin and end in it; a segmented scan
 * joins the runs.  seg0: the first row that ends in the thread's run or later.
 * The warp's first row end goes to first(row, sum of the warp's edges); lane 31
 * calls tail(any row end in the warp, the row after the last, its sum so far) */
template <class ID, class Load, class Store, class First, class Tail>
__device__ __forceinline__ void gather_run(const ID *run, uint32_t n, uint32_t seg0, Load load, Store store,
                                           First first, Tail tail)
{
    constexpr uint32_t END = (uint32_t)1 << (sizeof(ID) * 8 - 1);
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    uint32_t seg = seg0;
    float sum = 0.0f, head = 0.0f; /* head: the sum at the first row end */
    bool ended = false;
    for (uint32_t j = 0; j < n; j += 4)
    {
        uint32_t u[4];
        float v[4];
        load4(run + j, u);
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = load(u[i] & (END - 1u));
#pragma unroll
        for (int i = 0; i < 4; i++)
        {
            sum = __fadd_rn(sum, v[i]);
            if (u[i] & END)
            {
                /* the first one waits for what earlier lanes have of it */
                if (ended)
                    store(seg, sum);
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
        if (ends & lt)
            store(seg0, s);
        else
            first(seg0, s);
    }
    if (lane == 31) tail(ends != 0u, seg, sum);
}

/* shared memory in which small_finish joins the threads' sums */
constexpr uint32_t SM_JOIN = 2 * 3 * (SM_THREADS / 4) * 4;

/* the ranks of this CTA's vertices, their sum, and the residual of the last
 * iteration run, which began with the ranks in `old`.  The sums stay in FP32 words
 * (gg_device.cuh) up to one lane: a conversion to FP64 takes the SM about 64 clocks
 * per warp (a call on 3,000 vertices lost 8 us to two per vertex).  join: SM_JOIN
 * bytes, which nothing else uses any more */
__device__ __forceinline__ void small_finish(const SmallArgs &a, const float *rank, const float *old, uint32_t v0,
                                             uint32_t v1, uint32_t it, float *join)
{
    constexpr uint32_t SLOTS = SM_THREADS / 4;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    double *to[2] = {&a.rec[it ? it - 1 : 0].err, a.sum};
    LongSum s[2];
    for (uint32_t i = tid; i < v1 - v0; i += SM_THREADS)
    {
        float r = rank[i];
        if (it > 0) s[0].add(fabsf(__fsub_rn(r, old[i])), to[0]);
        if (a.divide) r = __fdiv_rn(r, __uint2float_rn(a.V));
        a.rank[v0 + i] = r;
        s[1].add(r, to[1]);
    }
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < 2; k++)
    {
        LongSum t = k ? s[1] : s[0];
        t.spill(SM_THREADS, k ? to[1] : to[0]);
#pragma unroll 1
        for (int o = 16; o >= 8; o >>= 1) t.merge_down(o);
        float *p = join + k * 3 * SLOTS + w * 8 + lane;
        if (lane < 8)
        {
            p[0] = t.hi;
            p[SLOTS] = t.mid;
            p[2 * SLOTS] = t.lo;
        }
    }
    __syncthreads();
    if (w < 2)
    {
        LongSum all;
        const float *p = join + w * 3 * SLOTS + lane;
#pragma unroll 1
        for (uint32_t k = 0; k < SLOTS; k += 32) all.merge(p[k], p[SLOTS + k], p[2 * SLOTS + k]);
#pragma unroll 1
        for (int o = 16; o > 0; o >>= 1) all.merge_down(o);
        if (lane == 0 && (w || it > 0)) atomicAdd(w ? to[1] : to[0], all.value());
    }
}

struct SmallShape
{
    size_t ids, rows, c, sums, rank, deg, old, join, total;
};
/* keep: with the ranks that an iteration began with */
__host__ __device__ inline SmallShape small_shape(uint32_t V, uint32_t eq, uint32_t vq, uint32_t rows_cap, uint32_t keep)
{
    SmallShape s;
    s.c = 0;
    s.sums = s.c + ((size_t)V + 4) / 4 * 16;
    s.rank = s.sums + (size_t)vq * 4;
    s.deg = s.rank + (size_t)vq * 4;
    s.old = s.deg + (size_t)vq * 4;
    s.ids = (s.old + (size_t)vq * 4 * keep + 15) / 16 * 16;
    s.rows = (s.ids + (size_t)eq * 2 + 15) / 16 * 16;
    s.total = (s.rows + (size_t)rows_cap * 4 + 15) / 16 * 16;
    /* the sums are joined over the contributions, or behind everything */
    s.join = ((size_t)V + 1) * 4 >= SM_JOIN ? s.c : s.total;
    if (s.join) s.total += SM_JOIN;
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
    const SmallShape sh = small_shape(a.V, a.eq, a.vq, a.rows_cap, a.keep);
    float *c = reinterpret_cast<float *>(gg_dyn + sh.c);
    float *sums = reinterpret_cast<float *>(gg_dyn + sh.sums);
    float *rank = reinterpret_cast<float *>(gg_dyn + sh.rank);
    uint32_t *deg = reinterpret_cast<uint32_t *>(gg_dyn + sh.deg);
    uint16_t *ids = reinterpret_cast<uint16_t *>(gg_dyn + sh.ids);
    uint32_t *rows = reinterpret_cast<uint32_t *>(gg_dyn + sh.rows); /* addresses of the rows' sums */
    const uint32_t C = MULTI ? gridDim.x : 1u, me = M::rank();
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const uint32_t e0 = min(me * a.eq, a.E), e1 = min(e0 + a.eq, a.E), ne = e1 - e0;
    const uint32_t v0 = min(me * a.vq, a.V), v1 = min(v0 + a.vq, a.V);
    float *old = a.keep ? reinterpret_cast<float *>(gg_dyn + sh.old) : a.rank + v0;
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

    uint32_t it = 0, total = 0;
    for (; it < a.iterations; it++)
    {
        if (work)
            gather_run(
                run, a.run, seg0, [&](uint32_t u) { return c[u]; },
                [&](uint32_t r, float v) { M::store(rows[r], v); },
                [&](uint32_t r, float v) {
                    if (open)
                        M::add(rows[r], v);
                    else
                        M::store(rows[r], v);
                },
                /* after the graph's last edge no row is open (only pads
                 * follow the last row end) */
                [&](bool, uint32_t r, float v) {
                    if (r < found && !(run[a.run - 1] & SM_END)) M::add(rows[r], v);
                });
        M::sync();
        uint32_t act = 0;
        for (uint32_t i = tid; i < v1 - v0; i += SM_THREADS)
        {
            const float s = sums[i];
            sums[i] = 0.0f;
            const float nr = __fadd_rn(a.base, __fmul_rn(a.damp, s));
            const float e = fabsf(__fsub_rn(nr, rank[i]));
            old[i] = rank[i];
            rank[i] = nr;
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
    small_finish(a, rank, old, v0, v1, it, reinterpret_cast<float *>(gg_dyn + sh.join));
    M::sync(); /* no CTA leaves while another may still write its memory */
}

/* ---- the whole chip ---------------------------------------------------------
 *
 * The same run for graphs past a cluster's reach, in one cooperative launch of
 * a CTA per SM: each holds its share of the in-neighbour ids in shared memory
 * for all iterations; contributions and row sums are in global memory, read
 * through the L1 that the ids leave, and the barriers are grid barriers, whose
 * fences make each iteration's reads new.
 *
 * Bound by the two barriers (1.7 us each with the block's own) and, from 1M
 * edges, by the gather's L2 requests.  Measured per call of 20 iterations, R-MAT
 * with 16 edges per vertex, launches -> here: 128K edges 151 -> 129 us (the
 * cluster 140), 262K 156 -> 140, 524K 175 -> 151, 1M 212 -> 179, 1.6M 239 -> 215;
 * uniform random, 1.9M 336 -> 286. */
struct GridArgs
{
    SmallArgs a;
    float *c, *sums; /* V + 1 contributions, the last 0; V row sums */
    unsigned long long *words; /* barriers: after each gather, then the one before the first */
    uint32_t *failed;
    unsigned long long limit_ns;
};

struct GridShape
{
    size_t rows, rank, deg, total;
};
__host__ __device__ inline GridShape grid_shape(uint32_t eq, uint32_t vq, uint32_t rows_cap)
{
    GridShape s;
    s.rows = (size_t)eq * 4;
    s.rank = s.rows + (size_t)rows_cap * 4;
    if (s.rank < SM_JOIN) s.rank = SM_JOIN; /* the sums are joined over the ids and rows */
    s.deg = s.rank + (size_t)vq * 4;
    s.total = (s.deg + (size_t)vq * 4 + 15) / 16 * 16;
    return s;
}

/* the last r in [0, V] with off[r] <= e (a whole warp calls it) */
__device__ __forceinline__ uint32_t last_row(const uint32_t *__restrict__ off, uint32_t V, uint32_t e)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, n = V + 1; /* the answer is in [lo, lo + n); off[0] = 0 */
    while (n > 1)
    {
        const uint32_t step = (n + 31) / 32, at = lo + lane * step;
        const uint32_t in = __ballot_sync(0xffffffffu, lane * step < n && off[at] <= e);
        const uint32_t k = 31u - (uint32_t)__clz((int)in); /* bit 0 is always set */
        lo += k * step;
        n = min(step, n - k * step);
    }
    return lo;
}

/* Grid barrier of k_pr_grid on a 64-bit word, zero at first: arrivals in the
 * high half, the sum of `add` in the low one, which is returned in *sum.  One
 * release add per CTA and acquire loads of the one word: two memory round
 * trips, as the barrier of gg_device.cuh, which has sixteen words for 900 blocks
 * and returns no sum.  False when the wait reached its limit, which sets
 * *failed: the other CTAs then leave at their next barrier. */
__device__ __forceinline__ bool counted_barrier(unsigned long long *word, uint32_t add, uint32_t *failed,
                                                unsigned long long limit_ns, uint32_t *sum)
{
    __shared__ unsigned long long s_word;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(((unsigned long long)1 << 32) | add)
                     : "memory");
        const unsigned long long t0 = global_ns();
        unsigned long long v = 0;
        for (;;)
        {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(word) : "memory");
            if ((uint32_t)(v >> 32) == gridDim.x) break;
            if (global_ns() - t0 > limit_ns)
            {
                atomicExch(failed, 1u);
                v = ~0ull;
                break;
            }
        }
        s_word = v;
    }
    __syncthreads();
    const unsigned long long v = s_word;
    *sum = (uint32_t)v;
    return v != ~0ull;
}

__global__ void __launch_bounds__(SM_THREADS, 1) k_pr_grid(GridArgs ga)
{
    const SmallArgs &a = ga.a;
    extern __shared__ __align__(1024) unsigned char gg_dyn[];
    __shared__ uint32_t s_total, s_row;
    __shared__ bool s_open; /* this CTA's first edge continues a row of the CTA before */
    __shared__ float s_first[SM_WARPS], s_tail[SM_WARPS]; /* per warp, see gather_run */
    __shared__ uint32_t s_seg[SM_WARPS];
    __shared__ bool s_ended[SM_WARPS];
    const GridShape sh = grid_shape(a.eq, a.vq, a.rows_cap);
    uint32_t *ids = reinterpret_cast<uint32_t *>(gg_dyn);
    uint32_t *rows = reinterpret_cast<uint32_t *>(gg_dyn + sh.rows);
    float *rank = reinterpret_cast<float *>(gg_dyn + sh.rank);
    uint32_t *deg = reinterpret_cast<uint32_t *>(gg_dyn + sh.deg);
    float *c = ga.c, *sums = ga.sums; /* written here: never read as constants */
    const uint32_t me = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const uint32_t e0 = (uint32_t)min((uint64_t)me * a.eq, (uint64_t)a.E), e1 = min(e0 + a.eq, a.E), ne = e1 - e0;
    const uint32_t v0 = (uint32_t)min((uint64_t)me * a.vq, (uint64_t)a.V), v1 = min(v0 + a.vq, a.V);
    /* the ranks that an iteration began with (in shared memory: 150K vertices, 750K
     * edges 241 us a call against 226) */
    float *old = a.rank + v0;
    const uint32_t wedges = 32 * a.run, nwork = (ne + wedges - 1) / wedges;
    const bool work = (tid >> 5) < nwork;

    for (uint32_t i = tid; i < nwork * wedges; i += SM_THREADS) ids[i] = i < ne ? a.adj[e0 + i] : a.V;
    for (uint32_t i = tid; i < v1 - v0; i += SM_THREADS)
    {
        const uint32_t d = a.outdeg[v0 + i];
        c[v0 + i] = d ? __fdiv_rn(a.init, __uint2float_rn(d)) : 0.0f;
        deg[i] = d;
        rank[i] = a.init;
        sums[v0 + i] = 0.0f;
    }
    if (me == 0 && tid == 0) c[a.V] = 0.0f;
    if (tid == 0) s_open = false;
    /* the rows with edges here, in order, and the marks of the last edges of
     * those that end here; 1,024 rows a step, runs of empty ones skipped */
    uint32_t found = 0;
    bool more = ne > 0, seek = true;
    uint32_t rb = 0, at_e = e0;
    while (more)
    {
        if (seek)
        {
            if (tid < 32)
            {
                const uint32_t r = last_row(a.off, a.V, at_e);
                if (lane == 0) s_row = r;
            }
            __syncthreads();
            rb = s_row;
            __syncthreads();
        }
        const uint32_t v = rb + tid;
        uint32_t s = 0, e = 0;
        if (v < a.V)
        {
            s = a.off[v];
            e = a.off[v + 1];
        }
        const bool here = v < a.V && e > s && e > e0 && s < e1;
        const uint32_t idx = found + block_excl(here ? 1u : 0u, &s_total);
        if (here)
        {
            rows[idx] = v;
            if (e <= e1) ids[e - 1 - e0] |= 0x80000000u;
            if (s < e0) s_open = true; /* only the first row of the list */
        }
        found += s_total;
        rb += SM_THREADS;
        if (rb >= a.V)
            more = false;
        else
        {
            const uint32_t next = a.off[rb];
            more = next < e1;
            seek = next == a.off[rb - SM_THREADS];
            at_e = next;
        }
        __syncthreads();
    }
    const uint32_t *run = ids + (size_t)tid * a.run;
    uint32_t n = 0;
    if (work)
        for (uint32_t j = 0; j < a.run; j++) n += run[j] >> 31;
    const uint32_t seg0 = block_excl(n, &s_total), ended_rows = s_total;
    uint32_t total;
    bool ok = counted_barrier(ga.words + a.iterations, 0u, ga.failed, ga.limit_ns, &total);

    uint32_t it = 0;
    for (; ok && it < a.iterations; it++)
    {
        if (work)
            gather_run(
                run, a.run, seg0, [&](uint32_t u) { return c[u]; }, [&](uint32_t r, float v) { sums[rows[r]] = v; },
                [&](uint32_t r, float v) {
                    s_first[tid >> 5] = v;
                    s_seg[tid >> 5] = r;
                },
                [&](bool ended, uint32_t, float v) {
                    s_ended[tid >> 5] = ended;
                    s_tail[tid >> 5] = v;
                });
        __syncthreads();
        /* warp 0 joins the warps as each joined its lanes: a row in one CTA is
         * stored, one over several gets an addition from each (at most one per
         * SM, fewer than the launches' one per 352 edges) */
        if (tid < 32 && nwork)
        {
            const bool used = lane < nwork, ended = used && s_ended[lane];
            float sum = used ? s_tail[lane] : 0.0f;
            const uint32_t ends = __ballot_sync(0xffffffffu, ended), le = ends & (((1u << lane) - 1u) | (1u << lane));
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
                const float v = lane ? __fadd_rn(s_first[lane], before) : s_first[lane];
                float *to = &sums[rows[s_seg[lane]]];
                if (s_open && le == (1u << lane))
                    atomicAdd(to, v);
                else
                    *to = v;
            }
            if (lane == 31 && found > ended_rows) atomicAdd(&sums[rows[ended_rows]], sum);
        }
        if (tid == 0) s_total = 0u;
        if (!(ok = counted_barrier(ga.words + it, 0u, ga.failed, ga.limit_ns, &total))) break;
        uint32_t act = 0;
        for (uint32_t i = tid; i < v1 - v0; i += SM_THREADS)
        {
            const float s = sums[v0 + i];
            sums[v0 + i] = 0.0f;
            const float nr = __fadd_rn(a.base, __fmul_rn(a.damp, s));
            const float e = fabsf(__fsub_rn(nr, rank[i]));
            old[i] = rank[i];
            rank[i] = nr;
            if (e >= a.eps_f) act++;
            const uint32_t d = deg[i];
            c[v0 + i] = d ? __fdiv_rn(nr, __uint2float_rn(d)) : 0.0f;
        }
        act = __reduce_add_sync(0xffffffffu, act);
        if (act && lane == 0) atomicAdd(&s_total, act);
        __syncthreads();
        /* the record's active count and the word after it */
        if (!(ok = counted_barrier(reinterpret_cast<unsigned long long *>(&a.rec[it].active), s_total, ga.failed,
                                   ga.limit_ns, &total)))
            break;
        if (total == 0u)
        {
            it++;
            break;
        }
    }
    if (!ok) return; /* the host reports it */
    small_finish(a, rank, old, v0, v1, it, reinterpret_cast<float *>(gg_dyn));
}

/* Edges per thread (of 152 SMs: 2.5M edges) and vertices above which the
 * launches are faster.  One launch against launches, us per call of 20 iterations:
 * R-MAT with 2.0M edges 253 : 273, 2.4M 301 : 310 -- the ids leave the L1 less room.
 * By vertices (a thread has a second one from 156K), uniform random with 5 or 8
 * edges each / R-MAT with 5 or 8: 150K 224 : 239, 249 : 278 / 225 : 215, 237 : 239;
 * 200K 274 : 273, 312 : 333 / 254 : 249, 298 : 284; 219K 335 : 285, 360 : 346 / 323 :
 * 255, 362 : 297. */
constexpr uint32_t GRID_RUN_MAX = 16, GRID_MAX_V = 200000;
constexpr size_t GRID_LIMIT = 220 * 1024;

/* the shares of a graph of one CTA per SM, or false when it does not fit */
bool grid_plan(uint32_t V, uint32_t E, SmallArgs &a, uint32_t &C, size_t &smem)
{
    C = (uint32_t)gg_sm_count();
    if (V == 0 || V > GRID_MAX_V || E == 0 || E > (uint64_t)C * SM_THREADS * GRID_RUN_MAX) return false;
    const uint32_t need = (E + C * SM_THREADS - 1) / (C * SM_THREADS);
    a.run = (need + 3) / 4 * 4;
    if (a.run > GRID_RUN_MAX) return false;
    const uint32_t wedges = 32 * a.run;
    a.eq = ((E + C - 1) / C + wedges - 1) / wedges * wedges;
    a.vq = (V + C - 1) / C;
    a.rows_cap = std::min(V, a.eq) + 1;
    smem = grid_shape(a.eq, a.vq, a.rows_cap).total;
    return smem <= GRID_LIMIT;
}

/* One CTA up to this many edges, a cluster of eight above: a cluster's two
 * barriers and remote stores cost about a microsecond per iteration, one SM's
 * issue slots as much per 8K edges.  Per call of 20 iterations, one CTA /
 * clusters of 2 / 4 / 8: 4.8K edges 74 / 88 / 85 / 85 us, 16K 96 / 103 / 101 /
 * 98, 32K 163 (the launches) / 121 / 109 / 117, 64K - / 165 / 134 / 120. */
constexpr uint32_t SM_ONE = 16384, SM_CLUSTER = 8;
/* Edges per thread of a cluster above which the whole chip is faster: 96K edges (12 per
 * thread) 138 us in a cluster against 151, 128K (20) 163 against 151.  A cluster
 * of 16 takes 149 where one of 8 takes 124 (64K edges). */
constexpr uint32_t SM_RUN_MAX = 12;

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
    if (C > 1 && a.run > SM_RUN_MAX) return false;
    /* whole warps' worth of edges per CTA */
    const uint32_t wedges = 32 * a.run;
    a.eq = ((E + C - 1) / C + wedges - 1) / wedges * wedges;
    a.vq = ((V + C - 1) / C + 3) / 4 * 4;
    a.rows_cap = std::min(V, a.eq) + 1;
    smem = small_shape(V, a.eq, a.vq, a.rows_cap, 0).total;
    if (smem > SM_LIMIT) return false;
    /* without the room, the ranks that an iteration began with go to global memory
     * (a call on 3,000 vertices with 15K edges: 101 us there, 92 in shared) */
    const size_t with = small_shape(V, a.eq, a.vq, a.rows_cap, 1).total;
    a.keep = with <= SM_MOST ? 1u : 0u;
    if (a.keep) smem = with;
    return true;
}

} // namespace

bool gg_small_fits(const gg_graph *g)
{
    SmallArgs a{};
    uint32_t C;
    size_t smem;
    return small_plan(g->V, g->E, a, C, smem) || grid_plan(g->V, g->E, a, C, smem);
}

gg_status gg_small_pagerank(gg_graph *g, const gg_pr_params *p, float *rank, void *rec, double *sum, float base,
                            float init, float eps_f, cudaStream_t s, bool *launched)
{
    *launched = false;
    SmallArgs a{};
    uint32_t C;
    size_t smem;
    const bool small = small_plan(g->V, g->E, a, C, smem);
    if (!small && !grid_plan(g->V, g->E, a, C, smem)) return gg_fail(GG_ERR_INVALID, "graph too large for one launch");
    a.off = g->in_off; a.adj = g->in_adj; a.outdeg = g->out_deg;
    a.rank = rank; a.rec = (SmallRec *)rec; a.sum = sum;
    a.V = g->V; a.E = g->E; a.iterations = p->max_iterations;
    a.base = base; a.damp = p->damp; a.init = init; a.eps_f = eps_f;
    a.divide = p->init_one_over_n ? 0 : 1;
    if (!small)
    {
        GridArgs ga{};
        void *c, *sums, *words;
        GG_CHECK(gg_work(g, 2, ((size_t)g->V + 16) * 4, &c));
        GG_CHECK(gg_work(g, 5, ((size_t)g->V + 16) * 4, &sums));
        GG_CHECK(gg_work(g, 34, ((size_t)a.iterations + 1) * 8, &words));
        GG_CUDA(cudaMemsetAsync(words, 0, ((size_t)a.iterations + 1) * 8, s));
        ga.a = a;
        ga.c = (float *)c; ga.sums = (float *)sums; ga.words = (unsigned long long *)words;
        ga.failed = &a.rec[a.iterations + 1].pad;
        ga.limit_ns = gg_barrier_limit_ns();
        GG_CUDA(cudaFuncSetAttribute((const void *)k_pr_grid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GRID_LIMIT));
        void *args[] = {&ga};
        *launched = cudaLaunchCooperativeKernel((const void *)k_pr_grid, dim3(C), dim3(SM_THREADS), args, smem, s) == cudaSuccess;
        if (!*launched) cudaGetLastError();
        return GG_OK;
    }
    void (*fn)(SmallArgs) = C > 1 ? k_pr_small<true> : k_pr_small<false>;
    GG_CUDA(cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM_MOST));
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
    *launched = cudaLaunchKernelEx(&cfg, fn, a) == cudaSuccess;
    if (!*launched) cudaGetLastError();
    return GG_OK;
}
