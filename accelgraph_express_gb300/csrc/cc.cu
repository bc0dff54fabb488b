/*
 * Connected components on CSR (connectedComponents.c:337-720) on one GPU.
 *
 * Every algorithm ends with each vertex labelled by the smallest vertex id
 * of its weakly connected component; the labels are deterministic, the
 * iteration counts (as in the reference) depend on the order of concurrent
 * updates.  Edge passes walk the CSR in merge-path tiles (warp_push), so a
 * hub's edges are spread over many warps.
 *
 *   Shiloach-Vishkin (pushpull 0; :362-468 with the FPGA hook step of
 *     cu_ConnectedComponents/.../cu_update_kernel_control.sv:171-190):
 *     repeat { k_cc_hook: for every out-edge, the higher of the two labels,
 *     if it is still a root, is pointed at the lower one; k_cc_compress:
 *     pointer jumping to the root } while any hook happened
 *   Afforest (pushpull 1 and default; :470-626): `neighbor_rounds` rounds of
 *     k_cc_link_round (link u with its r-th out-neighbour) + compression; a
 *     sample of labels picks the largest component (k_cc_pick), whose vertices
 *     skip the final link (k_cc_link_rest over the remaining out-edges and,
 *     when the CSC is mapped, every in-edge); compression
 *   weakly connected components (pushpull 2; :628-720): repeat k_cc_minprop
 *     (both endpoints of every out-edge take the smaller label by atomicMin)
 *     while any label fell
 *
 * cc_link is the reference's linkNodes (:249-269): union by the lower label
 * with a compare-and-swap on the higher root, retried while the roots move.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "gg_device.cuh"

namespace {

using namespace gg;

struct CcFlags
{
    unsigned int changed;
    unsigned int err;
    unsigned int roots;
    unsigned int skip;   /* Afforest: the label left out of the final link, or ~0 */
    unsigned int nheavy; /* rows deferred to k_cc_link_heavy (may exceed CC_MAX_HEAVY) */
    unsigned int pad[3];
};

/* rows of the final link above CC_HEAVY edges are spread over the whole grid,
 * up to CC_MAX_HEAVY of them (further ones stay with their warp) */
constexpr uint32_t CC_HEAVY = 2048, CC_MAX_HEAVY = 4096;

constexpr uint32_t LINK_RETRIES = 1u << 16;

__device__ __forceinline__ uint32_t ld_comp(const uint32_t *comp, uint32_t i)
{
    return *(const volatile uint32_t *)(comp + i);
}

/* A label through L1.  It may be older than another warp's update in the same
 * launch; an old label of a vertex is still a node of its tree, and a node once
 * seen under another stays in its tree, so it serves wherever a later check
 * reads the label anew (ld_comp) or only tree membership matters. */
__device__ __forceinline__ uint32_t ld_old(const uint32_t *comp, uint32_t i)
{
    uint32_t v;
    asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(comp + i) : "memory");
    return v;
}

/* unite the trees of nodes a and b (labels read earlier, or the vertices) */
__device__ __forceinline__ void cc_unite(uint32_t a, uint32_t b, uint32_t *comp, CcFlags *f)
{
    for (uint32_t tries = 0; a != b; tries++)
    {
        if (tries == LINK_RETRIES)
        {
            atomicOr(&f->err, 1u);
            return;
        }
        const uint32_t hi = a > b ? a : b, lo = a > b ? b : a;
        const uint32_t ph = ld_comp(comp, hi);
        if (ph == lo) return;
        if (ph == hi && atomicCAS(comp + hi, hi, lo) == hi) return;
        a = ld_comp(comp, ld_comp(comp, hi));
        b = ld_comp(comp, lo);
    }
}

__global__ void k_cc_init(uint32_t *comp, uint32_t V)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) comp[v] = v;
}

__device__ __forceinline__ void cc_link(uint32_t u, uint32_t v, uint32_t *comp, CcFlags *f)
{
    cc_unite(ld_old(comp, u), ld_old(comp, v), comp, f);
}

/* pointer jumping until every vertex points at its root (labels only
 * decrease along a chain, so each loop ends); with COUNT also the number of
 * roots.  Bound by the random reads of the chains: they go through L1 (most
 * chains end at a few roots, and an older pointer leads to the same root, which
 * no compression moves), a thread follows four vertices' chains together, and
 * only labels that moved are written (6M vertices: 77 us one chain at a time
 * through L2, 15 now). */
template <bool COUNT>
__global__ void __launch_bounds__(256) k_cc_compress(uint32_t *comp, uint32_t V, CcFlags *f)
{
    const uint32_t Q = V >> 2, stride = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t roots = 0;
    for (uint32_t q = tid; q < Q; q += stride)
    {
        const uint4 own = reinterpret_cast<const uint4 *>(comp)[q];
        uint32_t c[4] = {own.x, own.y, own.z, own.w}, n[4];
        bool go[4] = {true, true, true, true};
        do
        {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (go[k]) n[k] = ld_old(comp, c[k]);
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (go[k])
                {
                    go[k] = n[k] != c[k];
                    c[k] = n[k];
                }
        } while (go[0] | go[1] | go[2] | go[3]);
        if (c[0] != own.x) comp[4 * q] = c[0];
        if (c[1] != own.y) comp[4 * q + 1] = c[1];
        if (c[2] != own.z) comp[4 * q + 2] = c[2];
        if (c[3] != own.w) comp[4 * q + 3] = c[3];
        if (COUNT)
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) roots += c[k] == 4 * q + k;
    }
    if (tid < (V & 3u))
    {
        const uint32_t v = 4 * Q + tid;
        uint32_t c = ld_old(comp, v), n;
        while ((n = ld_old(comp, c)) != c) c = n;
        comp[v] = c;
        if (COUNT) roots += c == v;
    }
    if (COUNT)
    {
        __shared__ uint32_t s_roots;
        if (threadIdx.x == 0) s_roots = 0u;
        __syncthreads();
        roots = warp_sum(roots);
        if ((threadIdx.x & 31) == 0 && roots) atomicAdd(&s_roots, roots);
        __syncthreads();
        if (threadIdx.x == 0 && s_roots) atomicAdd(&f->roots, s_roots);
    }
}

/* note that a pass changed a label: one store per block (one per changed label
 * had the L2 take millions to one address: R-MAT with 16M edges, Shiloach-Vishkin
 * 556 -> 402 us, minimum propagation 729 -> 371) */
__device__ __forceinline__ void cc_changed(bool changed, CcFlags *f)
{
    if (__syncthreads_or(changed) && threadIdx.x == 0) *(volatile unsigned int *)&f->changed = 1u;
}

__global__ void __launch_bounds__(GG_TILE_NT) k_cc_hook(const uint32_t *__restrict__ off,
                                                        const uint32_t *__restrict__ adj, const uint2 *__restrict__ coord,
                                                        uint32_t ntiles, uint32_t V, uint32_t *comp, CcFlags *f)
{
    /* the row's label is read once per row segment; a label read here may
     * be older than another warp's hook in the same pass, which costs at most
     * a repeat in the next pass (a pass that hooks nothing reads no stale
     * value, so the stop test is exact) */
    struct Op
    {
        typedef uint32_t RowVal;
        uint32_t *comp;
        bool changed;
        __device__ __forceinline__ uint32_t row_value(uint32_t r) const { return comp[r]; }
        __device__ __forceinline__ void scatter(uint32_t cu, uint32_t, uint32_t v)
        {
            const uint32_t cv = comp[v];
            if (cu == cv) return;
            const uint32_t hi = cu > cv ? cu : cv, lo = cu > cv ? cv : cu;
            if (comp[hi] == hi)
            {
                comp[hi] = lo;
                changed = true;
            }
        }
    } op{comp, false};
    warp_push<GG_TILE_IPT, GG_TILE_WARPS>(off, adj, V, coord, ntiles, op);
    cc_changed(op.changed, f);
}

__global__ void __launch_bounds__(GG_TILE_NT) k_cc_minprop(const uint32_t *__restrict__ off,
                                                           const uint32_t *__restrict__ adj,
                                                           const uint2 *__restrict__ coord, uint32_t ntiles,
                                                           uint32_t V, uint32_t *comp, CcFlags *f)
{
    /* the row's label is read once per row segment (a stale, larger label
     * only propagates less in this pass) */
    struct Row
    {
        uint32_t u, cu;
    };
    struct Op
    {
        typedef Row RowVal;
        uint32_t *comp;
        bool changed;
        __device__ __forceinline__ Row row_value(uint32_t r) const { return Row{r, comp[r]}; }
        __device__ __forceinline__ void scatter(Row &rv, uint32_t, uint32_t v)
        {
            const uint32_t cv = comp[v];
            if (rv.cu < cv)
            {
                if (atomicMin(comp + v, rv.cu) > rv.cu) changed = true;
            }
            else if (cv < rv.cu)
            {
                if (atomicMin(comp + rv.u, cv) > cv) changed = true;
                rv.cu = cv; /* the segment's next edges go on from it */
            }
        }
    } op{comp, false};
    warp_push<GG_TILE_IPT, GG_TILE_WARPS>(off, adj, V, coord, ntiles, op);
    cc_changed(op.changed, f);
}

/* link every vertex with its r-th out-neighbour: four vertices per thread,
 * their offsets, neighbours and labels loaded together before the links.  In
 * the first round every label is its vertex, so none is read: the higher end is
 * pointed at the lower by one compare-and-swap, and only where another edge
 * came first does the general link take over, from the label that the swap
 * returned.  (6M vertices, two rounds: 162 us reading each label,
 * 94 now.) */
template <bool FIRST>
__global__ void __launch_bounds__(256) k_cc_link_round(const uint32_t *__restrict__ off,
                                                       const uint32_t *__restrict__ adj, uint32_t V, uint32_t r,
                                                       uint32_t *comp, CcFlags *f)
{
    const uint32_t Q = V >> 2, stride = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t q = tid; q < Q; q += stride)
    {
        const uint4 o = reinterpret_cast<const uint4 *>(off)[q];
        const uint32_t s[5] = {o.x, o.y, o.z, o.w, off[4 * q + 4]};
        uint32_t v[4], a[4], b[4];
        bool has[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
        {
            has[k] = r < s[k + 1] - s[k];
            v[k] = has[k] ? adj[s[k] + r] : 0u;
        }
        if (FIRST)
        {
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
                const uint32_t u = 4 * q + k, hi = max(u, v[k]), lo = min(u, v[k]);
                a[k] = b[k] = lo;
                if (has[k] && hi != lo)
                {
                    const uint32_t seen = atomicCAS(comp + hi, hi, lo);
                    if (seen != hi) a[k] = seen;
                }
            }
        }
        else
        {
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
                a[k] = b[k] = 0u;
                if (has[k])
                {
                    a[k] = ld_old(comp, 4 * q + k);
                    b[k] = ld_old(comp, v[k]);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (a[k] != b[k]) cc_unite(a[k], b[k], comp, f);
    }
    if (tid < (V & 3u))
    {
        const uint32_t u = 4 * Q + tid;
        if (r < off[u + 1] - off[u]) cc_link(u, adj[off[u] + r], comp, f);
    }
}

/* the final link: every edge of the vertices whose label is not f->skip -- the
 * out-edges from `skip_head` on (the rounds linked the others) and, with
 * in_off, every in-edge.  Most vertices of a graph with a giant component are
 * skipped, and so are nearly all edges: the labels are read first, 32 vertices
 * per warp, and only the rows left are touched (reading the adjacency of every
 * row had cost 213 us per direction at 96M edges; 76 now for both).
 * The rows a warp is left with are concatenated and taken 32 edges at a time;
 * rows above CC_HEAVY edges go to k_cc_link_heavy. */
__global__ void __launch_bounds__(256) k_cc_link_rest(const uint32_t *__restrict__ out_off,
                                                      const uint32_t *__restrict__ out_adj,
                                                      const uint32_t *__restrict__ in_off,
                                                      const uint32_t *__restrict__ in_adj, uint32_t V,
                                                      uint32_t skip_head, uint32_t *comp, CcFlags *f, uint4 *heavy)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t words = (uint32_t)(((uint64_t)V + 31) / 32), skip = f->skip;
    for (uint32_t w = warp; w < words; w += nwarps)
    {
        const uint32_t u = w * 32 + lane;
        const bool act = u < V && ld_comp(comp, u) != skip;
        if (__ballot_sync(0xffffffffu, act) == 0u) continue;
        for (int dir = 0; dir < (in_off ? 2 : 1); dir++)
        {
            const uint32_t *off = dir ? in_off : out_off, *adj = dir ? in_adj : out_adj;
            uint32_t s = 0, len = 0;
            if (act)
            {
                const uint32_t s0 = off[u], deg = off[u + 1] - s0, head = dir ? 0u : skip_head;
                if (deg > head)
                {
                    s = s0 + head;
                    len = deg - head;
                }
                if (len > CC_HEAVY)
                {
                    const uint32_t at = atomicAdd(&f->nheavy, 1u);
                    if (at < CC_MAX_HEAVY)
                    {
                        heavy[at] = make_uint4(u, s, s + len, (uint32_t)dir);
                        len = 0;
                    }
                }
            }
            uint32_t left = len;
            while (__ballot_sync(0xffffffffu, left != 0u))
            {
                /* items 0..31 of the concatenated remaining rows; a row gives
                 * at most 32 per round, so the running totals stay small */
                const uint32_t give = min(left, 32u);
                uint32_t incl = give;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1)
                {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= (uint32_t)o) incl += y;
                }
                const uint32_t excl = incl - give, total = __shfl_sync(0xffffffffu, incl, 31);
                uint32_t owner = 0;
#pragma unroll
                for (uint32_t step = 16; step >= 1; step >>= 1)
                    if (__shfl_sync(0xffffffffu, incl, owner + step - 1) <= lane) owner += step;
                const uint32_t o_excl = __shfl_sync(0xffffffffu, excl, owner & 31);
                const uint32_t o_s = __shfl_sync(0xffffffffu, s, owner & 31);
                const uint32_t o_u = __shfl_sync(0xffffffffu, u, owner & 31);
                if (lane < total) cc_link(o_u, adj[o_s + (lane - o_excl)], comp, f);
                __syncwarp();
                const uint32_t used = incl <= 32u ? give : (excl < 32u ? 32u - excl : 0u);
                s += used;
                left -= used;
            }
        }
    }
}

__global__ void __launch_bounds__(256) k_cc_link_heavy(const uint32_t *__restrict__ out_adj,
                                                       const uint32_t *__restrict__ in_adj, uint32_t *comp, CcFlags *f,
                                                       const uint4 *__restrict__ heavy)
{
    const uint32_t n = min(f->nheavy, CC_MAX_HEAVY);
    const uint32_t stride = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t i = 0; i < n; i++)
    {
        const uint4 h = heavy[i];
        const uint32_t *adj = h.w ? in_adj : out_adj;
        for (uint64_t j = (uint64_t)h.y + tid; j < h.z; j += stride) cc_link(h.x, adj[j], comp, f);
    }
}

/* the i-th sampled label (SplitMix64 of seed + i) */
__device__ __forceinline__ uint32_t cc_sample(const uint32_t *comp, uint32_t V, uint64_t seed, uint32_t i)
{
    uint64_t z = seed + i;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return comp[z % V];
}

__global__ void k_cc_sample(const uint32_t *__restrict__ comp, uint32_t V, uint64_t seed, uint32_t n, uint32_t *out)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = cc_sample(comp, V, seed, i);
}

/* the most frequent of n <= 1024 sampled labels (ties to the smaller) into
 * f->skip, counted in an open-addressing table of the block's shared memory:
 * no read-back and sort on the host between the rounds and the final link */
__global__ void __launch_bounds__(1024) k_cc_pick(const uint32_t *__restrict__ comp, uint32_t V, uint64_t seed,
                                                  uint32_t n, CcFlags *f)
{
    constexpr uint32_t SLOTS = 2048, FREE = 0xffffffffu; /* no label is ~0: labels are below V */
    __shared__ uint32_t key[SLOTS], count[SLOTS];
    __shared__ unsigned long long best;
    for (uint32_t i = threadIdx.x; i < SLOTS; i += blockDim.x)
    {
        key[i] = FREE;
        count[i] = 0u;
    }
    if (threadIdx.x == 0) best = 0ull;
    __syncthreads();
    if (threadIdx.x < n)
    {
        const uint32_t l = cc_sample(comp, V, seed, threadIdx.x);
        uint32_t at = (l * 0x9E3779B1u) >> 21;
        for (;;) /* at most 1024 keys in 2048 slots: a free one is found */
        {
            const uint32_t seen = atomicCAS(&key[at], FREE, l);
            if (seen == FREE || seen == l) break;
            at = (at + 1u) & (SLOTS - 1u);
        }
        atomicAdd(&count[at], 1u);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < SLOTS; i += blockDim.x)
        if (count[i]) atomicMax(&best, (unsigned long long)count[i] << 32 | (0xffffffffu - key[i]));
    __syncthreads();
    if (threadIdx.x == 0) f->skip = 0xffffffffu - (uint32_t)best;
}

__global__ void k_cc_roots(const uint32_t *__restrict__ comp, uint32_t V, CcFlags *f)
{
    uint32_t n = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) n += comp[v] == v;
    n = warp_sum(n);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(&f->roots, n);
}

int grid_for(uint32_t n)
{
    const uint32_t b = (n + 255) / 256, cap = (uint32_t)gg_sm_count() * 8;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

struct Cc
{
    gg_graph *g;
    cudaStream_t s;
    uint32_t *comp;
    CcFlags *f, *h;
    uint32_t launches = 0;
    int profile = 0;
    std::vector<cudaEvent_t> evs;
};

gg_status mark(Cc &C)
{
    if (!C.profile) return GG_OK;
    cudaEvent_t e;
    GG_CHECK(gg_event_at(C.g, (uint32_t)C.evs.size(), &e));
    GG_CUDA(cudaEventRecord(e, C.s));
    C.evs.push_back(e);
    return GG_OK;
}

gg_status read_flags(Cc &C)
{
    GG_CUDA(cudaMemcpyAsync(C.h, C.f, sizeof(CcFlags), cudaMemcpyDeviceToHost, C.s));
    GG_CHECK(gg_wait(C.s));
    if (C.h->err) return gg_fail(GG_ERR_KERNEL, "connected components: a link gave up after its retry limit");
    return GG_OK;
}

gg_status compress(Cc &C, bool count = false)
{
    if (count)
        k_cc_compress<true><<<grid_for(C.g->V), 256, 0, C.s>>>(C.comp, C.g->V, C.f);
    else
        k_cc_compress<false><<<grid_for(C.g->V), 256, 0, C.s>>>(C.comp, C.g->V, C.f);
    C.launches++;
    GG_CUDA(cudaGetLastError());
    return GG_OK;
}

/* repeat one edge pass + (for SV) compression while a label changed */
template <class Launch>
gg_status until_stable(Cc &C, uint32_t max_iterations, bool with_compress, uint32_t *iterations, Launch launch)
{
    uint32_t it = 0;
    for (;;)
    {
        GG_CUDA(cudaMemsetAsync(&C.f->changed, 0, 4, C.s));
        GG_CHECK(mark(C));
        launch();
        C.launches++;
        if (with_compress) GG_CHECK(compress(C));
        GG_CHECK(mark(C));
        GG_CUDA(cudaGetLastError());
        it++;
        GG_CHECK(read_flags(C));
        if (!C.h->changed) break;
        if (it >= max_iterations) return gg_fail(GG_ERR_KERNEL, "connected components did not settle");
    }
    *iterations = it;
    return GG_OK;
}

} // namespace

extern "C" gg_status gg_cc(gg_graph *g, const gg_cc_params *p, uint32_t *components, gg_cc_result *r, void *stream)
{
    GgRange range("gg_cc");
    if (!g || !p) return gg_fail(GG_ERR_INVALID, "NULL argument");
    if (p->algorithm > 2) return gg_fail(GG_ERR_INVALID, "unknown connected-components algorithm");
    if (!g->out_off) return gg_fail(GG_ERR_INVALID, "connected components need GG_MAP_OUT");
    if (p->algorithm == GG_CC_AFFOREST && p->use_in_edges == 1 && !g->in_off)
        return gg_fail(GG_ERR_INVALID, "use_in_edges needs GG_MAP_IN");
    const uint32_t V = g->V;
    Cc C;
    C.g = g;
    C.s = gg_stream(g, stream);
    C.profile = (int)p->profile;
    void *ptr;
    GG_CHECK(gg_work(g, 0, ((size_t)V + 64) * 4, &ptr));
    C.comp = (uint32_t *)ptr;
    GG_CHECK(gg_work(g, 7, 256, &ptr));
    C.f = (CcFlags *)ptr;
    GG_CHECK(gg_pinned(g, 256, &ptr));
    C.h = (CcFlags *)ptr;
    GG_CUDA(cudaMemsetAsync(C.f, 0, sizeof(CcFlags), C.s));
    k_cc_init<<<grid_for(V), 256, 0, C.s>>>(C.comp, V);
    C.launches++;
    GG_CUDA(cudaGetLastError());

    gg_cc_result res{};
    const uint32_t max_it = p->max_iterations ? p->max_iterations : V + 1;
    gg_tiles *t = nullptr;
    int tgrid = 0;
    if (p->algorithm != GG_CC_AFFOREST)
    {
        GG_CHECK(gg_tiles_get(g, 0, C.s, &t));
        tgrid = gg_persistent_grid((const void *)k_cc_hook, t->ntiles);
    }
    if (p->algorithm == 0)
    {
        GG_CHECK(until_stable(C, max_it, true, &res.iterations, [&] {
            k_cc_hook<<<tgrid, GG_TILE_NT, 0, C.s>>>(g->out_off, g->out_adj, t->coord, t->ntiles, V, C.comp, C.f);
        }));
    }
    else if (p->algorithm == 2)
    {
        GG_CHECK(until_stable(C, max_it, false, &res.iterations, [&] {
            k_cc_minprop<<<tgrid, GG_TILE_NT, 0, C.s>>>(g->out_off, g->out_adj, t->coord, t->ntiles, V, C.comp, C.f);
        }));
    }
    else
    {
        const uint32_t rounds = p->neighbor_rounds ? p->neighbor_rounds : 2;
        GG_CHECK(mark(C));
        for (uint32_t rr = 0; rr < rounds; rr++)
        {
            if (rr == 0)
                k_cc_link_round<true><<<grid_for(V), 256, 0, C.s>>>(g->out_off, g->out_adj, V, rr, C.comp, C.f);
            else
                k_cc_link_round<false><<<grid_for(V), 256, 0, C.s>>>(g->out_off, g->out_adj, V, rr, C.comp, C.f);
            C.launches++;
            GG_CHECK(compress(C));
        }
        /* the skipped component: the most frequent label among the samples
         * (ties to the smaller label); none when in-edges are not linked and
         * the caller has not declared the graph symmetric */
        const bool use_in = p->use_in_edges == 1 || (p->use_in_edges == 2 && g->in_off);
        const bool may_skip = use_in || p->use_in_edges == 0;
        const uint32_t ns = p->samples ? (p->samples < V ? p->samples : V) : (V < 1024 ? V : 1024);
        GG_CUDA(cudaMemsetAsync(&C.f->skip, 0xff, 4, C.s));
        if (may_skip && ns && ns <= 1024)
        {
            k_cc_pick<<<1, 1024, 0, C.s>>>(C.comp, V, p->seed, ns, C.f);
            C.launches++;
        }
        else if (may_skip && ns)
        {
            void *sp;
            GG_CHECK(gg_work(g, 1, (size_t)ns * 4, &sp));
            k_cc_sample<<<grid_for(ns), 256, 0, C.s>>>(C.comp, V, p->seed, ns, (uint32_t *)sp);
            C.launches++;
            std::vector<uint32_t> smp(ns);
            GG_CHECK(gg_wait(C.s)); /* bounded, before a copy to pageable memory */
            GG_CUDA(cudaMemcpyAsync(smp.data(), sp, (size_t)ns * 4, cudaMemcpyDeviceToHost, C.s));
            GG_CHECK(gg_wait(C.s));
            std::sort(smp.begin(), smp.end());
            uint32_t best = 0, skip = 0xffffffffu;
            for (size_t i = 0; i < smp.size();)
            {
                size_t k = i;
                while (k < smp.size() && smp[k] == smp[i]) k++;
                if (k - i > best)
                {
                    best = (uint32_t)(k - i);
                    skip = smp[i];
                }
                i = k;
            }
            C.h->skip = skip;
            GG_CUDA(cudaMemcpyAsync(&C.f->skip, &C.h->skip, 4, cudaMemcpyHostToDevice, C.s));
        }
        void *hv;
        GG_CHECK(gg_work(g, 8, (size_t)CC_MAX_HEAVY * sizeof(uint4), &hv));
        k_cc_link_rest<<<gg_sm_count() * 8, 256, 0, C.s>>>(g->out_off, g->out_adj, use_in ? g->in_off : nullptr,
                                                          g->in_adj, V, rounds, C.comp, C.f, (uint4 *)hv);
        k_cc_link_heavy<<<gg_sm_count() * 8, 256, 0, C.s>>>(g->out_adj, g->in_adj, C.comp, C.f, (const uint4 *)hv);
        C.launches += 2;
        GG_CHECK(compress(C, true));
        GG_CHECK(mark(C));
        GG_CUDA(cudaGetLastError());
        res.iterations = rounds;
    }
    if (p->algorithm != GG_CC_AFFOREST) /* its last compression counted them */
    {
        k_cc_roots<<<grid_for(V), 256, 0, C.s>>>(C.comp, V, C.f);
        C.launches++;
        GG_CUDA(cudaGetLastError());
    }
    if (components) GG_CHECK(gg_copy_d2h(components, C.comp, (size_t)V * 4, C.s));
    GG_CHECK(read_flags(C));
    res.components = C.h->roots;
    if (p->algorithm == GG_CC_AFFOREST) res.skipped_label = C.h->skip;
    res.launches = C.launches;
    if (C.profile)
        for (size_t i = 0; i + 1 < C.evs.size(); i += 2) res.kernel_ms += gg_event_ms(C.evs[i], C.evs[i + 1]);
    if (r) *r = res;
    return GG_OK;
}

extern "C" gg_status gg_cc_device_labels(const gg_graph *g, const uint32_t **components)
{
    if (!g || !g->work[0].ptr) return gg_fail(GG_ERR_INVALID, "no connected-components run on this mapping");
    if (components) *components = (const uint32_t *)g->work[0].ptr;
    return GG_OK;
}
