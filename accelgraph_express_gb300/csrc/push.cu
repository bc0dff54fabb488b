/*
 * The frequent destinations of the push scatters.
 *
 * A push adds every edge's value to its destination with an atomic at the L2,
 * 183 G/s over the chip -- but one address takes an addition every 5 ns only,
 * and the L2 slices that hold the hubs' lines are busy while the others wait: on
 * R-MAT graphs, where the first vertex has 1% of the edges, that bounds a
 * scatter.  The kernels add the most frequent destinations up in shared memory
 * (PushTable, gg_device.cuh), PUSH_SLOTS of them, found by their hash.
 *
 * Which they are is estimated once per mapping, on the device, from up to
 * SAMPLES edges: of the destinations with one hash the one sampled most often
 * has the slot.  The highest sampled count decides whether the table is used.
 */
#include <cuda_runtime.h>

#include "gg_device.cuh"

namespace {

using namespace gg;

constexpr uint32_t SAMPLES = 1u << 18;

/* every 32 consecutive edges of `every` * 32 */
__global__ void k_push_sample(const uint32_t *__restrict__ adj, uint32_t E, uint32_t groups, uint32_t every,
                              uint32_t *counts)
{
    const uint32_t lane = threadIdx.x & 31, warps = gridDim.x * blockDim.x / 32;
    for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) / 32; k < groups; k += warps)
    {
        const uint64_t e = (uint64_t)k * every * 32 + lane;
        if (e < E) atomicAdd(&counts[adj[e]], 1u);
    }
}

/* best[slot] = count and id of the destination sampled most often; one seen
 * once is no better than any */
__global__ void k_push_pick(const uint32_t *__restrict__ counts, uint32_t V, unsigned long long *best)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    {
        const uint32_t n = counts[v];
        if (n > 1) atomicMax(&best[push_slot(v)], (unsigned long long)n << 32 | v);
    }
}

__global__ void __launch_bounds__(1024) k_push_tags(const unsigned long long *__restrict__ best, uint32_t *tags)
{
    __shared__ uint32_t s_most;
    if (threadIdx.x == 0) s_most = 0u;
    __syncthreads();
    uint32_t most = 0;
    for (uint32_t i = threadIdx.x; i < PUSH_SLOTS; i += 1024)
    {
        const unsigned long long b = best[i];
        most = max(most, (uint32_t)(b >> 32));
        tags[i] = b ? (uint32_t)b : 0xffffffffu; /* no vertex */
    }
    atomicMax(&s_most, most);
    __syncthreads();
    if (threadIdx.x == 0) tags[PUSH_SLOTS] = s_most;
}

} // namespace

gg_status gg_push_tags(gg_graph *g, uint32_t iterations, cudaStream_t s, const uint32_t **tags)
{
    *tags = nullptr;
    const uint32_t V = g->V, E = g->E;
    if (!g->push_tags)
    {
        /* looking for them takes some 40 us, with the wait */
        if (E < (1u << 16)) return GG_OK;
        g->push_edges += (uint64_t)iterations * E;
        if (g->push_edges < (1u << 21)) return GG_OK;
        void *w;
        GG_CHECK(gg_work(g, 25, (size_t)PUSH_SLOTS * 8 > 65536 * 4 ? (size_t)PUSH_SLOTS * 8 : 65536 * 4, &w));
        unsigned long long *best = (unsigned long long *)w;
        GG_CHECK(gg_work(g, 26, (size_t)V * 4, &w));
        uint32_t *counts = (uint32_t *)w;
        GG_CHECK(gg_dev_alloc(g, (void **)&g->push_tags, (PUSH_SLOTS + 4) * 4));
        GG_CUDA(cudaMemsetAsync(best, 0, (size_t)PUSH_SLOTS * 8, s));
        GG_CUDA(cudaMemsetAsync(counts, 0, (size_t)V * 4, s));
        const uint32_t all = E / 32 + (E % 32 ? 1u : 0u), every = (all + SAMPLES / 32 - 1) / (SAMPLES / 32);
        const uint32_t groups = (all + every - 1) / every;
        const int grid = gg_sm_count() * 8;
        k_push_sample<<<grid, 256, 0, s>>>(g->out_adj, E, groups, every, counts);
        k_push_pick<<<grid, 256, 0, s>>>(counts, V, best);
        k_push_tags<<<1, 1024, 0, s>>>(best, g->push_tags);
        GG_CUDA(cudaGetLastError());
        void *pin;
        GG_CHECK(gg_pinned(g, 64, &pin));
        GG_CUDA(cudaMemcpyAsync(pin, g->push_tags + PUSH_SLOTS, 4, cudaMemcpyDeviceToHost, s));
        GG_CHECK(gg_wait(s));
        const uint32_t most = *(const volatile uint32_t *)pin;
        /* the additions to one address, 5 ns each, against half of what the
         * others take (183 G/s, 8 us of latency and launch).  Far below the
         * line the table only costs: uniform random graphs of 75K edges 9.4 ->
         * 12.6 us an iteration, 1M 14.0 -> 16.1, 2.5M 20.4 -> 23.1 */
        const double same = 5e-3 * (double)most / (groups * 32.0) * E, others = (double)E / 183e3 + 8.0;
        g->push_hubs = same >= 0.5 * others;
    }
    if (g->push_hubs) *tags = g->push_tags;
    return GG_OK;
}
