/*
 * SpMV on CSR (02_capi_graph/src/algorithms/capi/SPMV.c:594-1135) on one GPU.
 *
 *   pull  (mode 0): y[v] = sum over in-edges (u,v) of w(u,v)*x[u]; the
 *                   merge-path tile gather over the CSC, recomputed every
 *                   iteration like the FPGA CU run per iteration (:712-718)
 *   push  (mode 1): y[dst] += w*x[src] over out-edges with FP32 atomics,
 *                   accumulating across iterations (:795-820)
 *   pull fixed (2): Q16.16 operands, (x*w) >> 16 summed in 64 bits
 *                   (cu_SPMV/CSR/PULL/FixedPoint/cu/cu_sum_kernel_control.sv:155-184)
 *   push fixed (3): Q32.32, y64 += (w*x) >> 32 (:1080-1093)
 * x and the weights may be stored as BF16/FP16 (FP32 products and sums).
 */
#include <cuda_runtime.h>
#include <cmath>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstring>
#include <string>
#include <vector>

#include "gg_hot.cuh"

namespace {

using namespace gg;

/* the edge term of the pull product: w[e] * x[u] (SPMV.c:735-760) */
template <class T>
struct SpmvGather
{
    typedef float Acc;
    typedef float Sum;
    struct Raw { T w, x; };
    const T *w;
    const T *x;
    __device__ __forceinline__ Raw load(uint32_t e, uint32_t u) const { return Raw{ldg_val(w + e), ldg_val(x + u)}; }
    __device__ __forceinline__ float value(const Raw &r) const { return __fmul_rn(to_f32(r.w), to_f32(r.x)); }
};

/* y of the next product: the gathers add the partials of rows that span tiles,
 * so each clears the other one of two buffers, V floats (null: none follows).
 * The plain gather does it at its end, beside the warps still at work: before the
 * gather it took 29 us of 257 (4.2M vertices, 67M edges between near ids; the gather
 * with the table loads that in the meantime and lost 3 us the other way round) */
__device__ __forceinline__ void clear_next(float *__restrict__ next, uint32_t V)
{
    if (!next) return;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) next[v] = 0.0f;
}

template <class T>
__global__ void __launch_bounds__(GG_TILE_NT) k_spmv_pull(const uint32_t *__restrict__ off, const uint32_t *__restrict__ adj,
                                                          const uint2 *__restrict__ coord, uint32_t ntiles, uint32_t V,
                                                          float *y, float *next, SpmvGather<T> op)
{
    pdl_wait();
    warp_pull_sums<GG_TILE_IPT, GG_TILE_WARPS>(off, adj, V, coord, ntiles, y, op);
    clear_next(next, V);
    pdl_trigger();
}

/* x of the hot vertices, contiguous (once per call: x does not change) */
template <class T>
__global__ void k_spmv_hot_fill(const T *__restrict__ x, const uint32_t *__restrict__ hot_list, uint32_t H,
                                uint32_t cap, T *__restrict__ out)
{
    hot_table_fill(x, hot_list, H, cap, out);
}

/* the pull product through the hot-vertex table (gg_hot.cuh) */
template <class T>
__global__ void __launch_bounds__(GG_HOT_WARPS * 32, 1)
    k_spmv_pull_hot(HotArgs a, const T *__restrict__ x, const T *__restrict__ w, const T *__restrict__ table_src,
                    float *y, float *next, uint32_t V)
{
    pdl_wait();
    clear_next(next, V);
    extern __shared__ __align__(1024) unsigned char gg_dyn[];
    const uint32_t warps = blockDim.x >> 5, wid = threadIdx.x >> 5;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(gg_dyn), table = ring + warps * HOT_RING;
    hot_pull_sums<T, float, float, true>(ring + wid * HOT_RING, table, hot_cap<T>(), a,
                           wid * gridDim.x + blockIdx.x, gridDim.x * warps, x, w, y, [&] {
                               hot_table_load(table, table_src, hot_table_bytes<T>());
                               return true;
                           });
    pdl_trigger();
}

/* one CTA of `warps` warps per SM */
template <class T>
int spmv_hot_grid(uint32_t ntiles, uint32_t warps)
{
    static int ok = -1;
    if (ok < 0)
    {
        cudaError_t e = cudaFuncSetAttribute(k_spmv_pull_hot<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)hot_smem_bytes<T>(GG_HOT_WARPS));
        ok = e == cudaSuccess ? 1 : 0;
        if (!ok) cudaGetLastError();
    }
    if (!ok) return 0;
    const uint32_t need = (ntiles + warps - 1) / warps;
    const uint32_t cap = (uint32_t)gg_sm_count();
    return (int)(need < cap ? (need ? need : 1) : cap);
}

/* fixed-point pull (SPMV.c:775-815): x in Q16.16, weights converted per
 * edge, products truncated to Q16.16 and summed exactly in 64 bits */
struct SpmvFxGather
{
    typedef unsigned long long Acc;
    typedef unsigned long long Sum;
    struct Raw { float w; uint32_t x; };
    const float *w;
    const uint32_t *x32;
    __device__ __forceinline__ Raw load(uint32_t e, uint32_t u) const { return Raw{ldg_val(w + e), ldg_val(x32 + u)}; }
    __device__ __forceinline__ unsigned long long value(const Raw &r) const
    {
        return ((unsigned long long)r.x * fx_from_float(r.w, 65536.0f, 0xffffffffu)) >> 16;
    }
};

__global__ void __launch_bounds__(GG_TILE_NT) k_spmv_pull_fx(const uint32_t *__restrict__ off, const uint32_t *__restrict__ adj,
                                                             const uint2 *__restrict__ coord, uint32_t ntiles, uint32_t V,
                                                             unsigned long long *y64, SpmvFxGather op)
{
    warp_pull_sums<GG_TILE_IPT, GG_TILE_WARPS>(off, adj, V, coord, ntiles, y64, op);
}

/* y = Q16.16 sums as float; clears the sums for the next product */
__global__ void k_spmv_fx_pull_out(unsigned long long *y64, float *y, uint32_t V)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    {
        const unsigned long long s = y64[v];
        y[v] = fx_to_float(s, 1.0f / 65536.0f);
        clear_after_read(&y64[v], s);
    }
}

/* TABLE: with the frequent destinations in shared memory (push.cu) */
template <class T, bool TABLE>
__global__ void __launch_bounds__(TABLE ? PUSH_NT : GG_TILE_NT)
    k_spmv_push(const uint32_t *__restrict__ off, const uint32_t *__restrict__ adj, const uint2 *__restrict__ coord,
                uint32_t ntiles, uint32_t V, const uint32_t *__restrict__ tags, const T *w, const T *x, float *y)
{
    push_scatter<TABLE>(
        off, adj, V, coord, ntiles, tags, y, [=](uint32_t r) -> float { return to_f32(x[r]); },
        [=](float xv, uint32_t e) { return __fmul_rn(to_f32(w[e]), xv); });
}

template <bool TABLE>
__global__ void __launch_bounds__(TABLE ? PUSH_NT : GG_TILE_NT)
    k_spmv_push_fx(const uint32_t *__restrict__ off, const uint32_t *__restrict__ adj, const uint2 *__restrict__ coord,
                   uint32_t ntiles, uint32_t V, const uint32_t *__restrict__ tags, const float *w,
                   const unsigned long long *x64, unsigned long long *y64)
{
    push_scatter<TABLE>(
        off, adj, V, coord, ntiles, tags, y64, [=](uint32_t r) -> unsigned long long { return x64[r]; },
        [=](unsigned long long xv, uint32_t e) { return fx64_mul(fx64_from_float(w[e]), xv); });
}

/* x[v] = 1/outdeg(v), or 0.001 when 0 (SPMV.c:696-701), unless given; the
 * stored copy in the chosen storage and the fixed-point copies */
template <class T>
__global__ void k_spmv_x(const uint32_t *__restrict__ outdeg, const float *xin, float *xf, T *xs, uint32_t *x32,
                         unsigned long long *x64, float *y, uint32_t V)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    {
        float xv;
        if (xin)
            xv = xin[v];
        else
        {
            uint32_t d = outdeg[v];
            xv = d ? __fdiv_rn(1.0f, __uint2float_rn(d)) : 0.001f;
        }
        xf[v] = xv;
        if (xs) xs[v] = from_f32<T>(xv);
        if (x32) x32[v] = fx_from_float(xv, 65536.0f, 0xffffffffu);
        if (x64) x64[v] = fx64_from_float(xv);
        y[v] = 0.0f;
    }
}

__global__ void k_spmv_fx64_out(const unsigned long long *y64, float *y, uint32_t V)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        y[v] = fx_to_float(y64[v], 1.0f / 4294967296.0f);
}

/* (int)(x * 100 + 0.5) in FP64, as the reference's round2 takes it; below
 * 2^22 from the exact fraction of the FP32 product, without FP64 */
__device__ __forceinline__ int round2_int(float y)
{
    const float f = __fmul_rn(y, 100.0f), a = fabsf(f);
    if (!(a < 4194304.0f)) return (int)__dadd_rn((double)f, 0.5);
    const int i = __float2int_rz(a);
    const bool up = __fsub_rn(a, (float)i) >= 0.5f;
    if (f >= 0.0f) return up ? i + 1 : i;
    const int n = up ? i : i - 1; /* truncation towards zero of f + 0.5 */
    return n > 0 ? -n : 0;
}

/* sum of round2(y) as the reference prints it (SPMV.c:727-730), in
 * hundredths: whole numbers, summed exactly (an FP64 division per vertex had
 * made this pass 197 us at 5M vertices; 31 now) */
__global__ void k_spmv_checksum(const float *__restrict__ y, uint32_t V, unsigned long long *out)
{
    long long s = 0;
    const uint32_t P = V >> 2, stride = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t p = tid; p < P; p += stride)
    {
        const float4 v = reinterpret_cast<const float4 *>(y)[p];
        s += (long long)round2_int(v.x) + round2_int(v.y) + round2_int(v.z) + round2_int(v.w);
    }
    if (tid < (V & 3u)) s += round2_int(y[P * 4 + tid]);
    __shared__ long long part[8];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (int k = 1; k < 8; k++) s += part[k];
        if (s) atomicAdd(out, (unsigned long long)s);
    }
}

int grid_v(uint32_t V) { int b = (int)((V + 255) / 256); int cap = gg_sm_count() * 8; return b < 1 ? 1 : (b > cap ? cap : b); }

template <class T>
gg_status spmv_fp(gg_graph *g, const gg_spmv_params *p, const float *x_dev, float *xf, float *y, cudaStream_t s,
                  uint32_t &launches, uint32_t &timed, std::vector<cudaEvent_t> &evs)
{
    const uint32_t V = g->V;
    const bool pull = p->mode == GG_SPMV_PULL;
    gg_tiles *t;
    GG_CHECK(gg_tiles_get(g, pull ? 1 : 0, s, &t));
    void *xs = nullptr;
    const T *w;
    if constexpr (sizeof(T) == 4)
    {
        w = (const T *)(pull ? g->in_w : g->out_w);
    }
    else
    {
        const void *w16;
        GG_CHECK(gg_weights16(g, pull ? 1 : 0, p->storage, s, &w16));
        w = (const T *)w16;
        GG_CHECK(gg_work(g, 12, ((size_t)V + 16) * sizeof(T), &xs));
    }
    const T *xv = sizeof(T) == 4 ? (const T *)xf : (const T *)xs;
    /* the products of a pull go to two buffers in turn, the last to y: a memset
     * before each was a launch more (20 products: 128K edges 266 -> 180 us, 1M
     * 397 -> 304, 3.2M 552 -> 493) */
    void *other = nullptr;
    if (pull && p->iterations > 1) GG_CHECK(gg_work(g, 14, ((size_t)V + 16) * 4, &other));
    float *ys[2] = {y, (float *)other};
    const uint32_t last = p->iterations ? p->iterations - 1 : 0;
    k_spmv_x<T><<<grid_v(V), 256, 0, s>>>(g->out_deg, x_dev, xf, (T *)xs, nullptr, nullptr, pull ? ys[last & 1] : y, V);
    launches++;
    /* the hot-vertex table, as for the PageRank pull */
    bool use_hot = false;
    void *hot_tab = nullptr;
    gg_tune_lookup(g, s);
    gg_pull_shape shape = g->spmv_shape;
    if (pull)
        GG_CHECK(gg_hot_choose(g, s, gg_hot_ask{p->flags, hot_cap<T>(), (uint32_t)sizeof(T), p->iterations, true}, &shape, &use_hot));
    if (use_hot)
    {
        GG_CHECK(gg_work(g, 32, GG_HOT_TABLE_BYTES + 16, &hot_tab));
        k_spmv_hot_fill<T><<<(hot_cap<T>() + 255) / 256, 256, 0, s>>>(xv, g->hot_list, g->hot_slots, hot_cap<T>(), (T *)hot_tab);
        launches++;
    }
    const uint32_t *tags = nullptr;
    if (!pull) GG_CHECK(gg_push_tags(g, p->iterations, s, &tags));
    for (uint32_t it = 0; it < p->iterations; it++)
    {
        if (p->profile)
        {
            cudaEvent_t e;
            GG_CHECK(gg_event_at(g, (uint32_t)evs.size(), &e));
            GG_CUDA(cudaEventRecord(e, s));
            evs.push_back(e);
        }
        if (pull)
        {
            float *yi = ys[(last - it) & 1], *next = it < last ? ys[(last - it - 1) & 1] : nullptr;
            const int hg = use_hot ? spmv_hot_grid<T>(g->hot_ntiles, shape.hot_warps) : 0;
            /* dependent launches, timed runs apart: 20 products of 16K edges
             * 170 -> 120 us, of 1M 304 -> 249 */
            if (hg)
            {
                const HotArgs ha{g->hot_adj, g->rows_list, g->hot_seg0, g->E, g->hot_ntiles, g->hot_tile};
                const dim3 grid(hg), block(shape.hot_warps * 32);
                const size_t smem = hot_smem_bytes<T>(shape.hot_warps);
                if (p->profile)
                    k_spmv_pull_hot<T><<<grid, block, smem, s>>>(ha, xv, w, (const T *)hot_tab, yi, next, V);
                else
                    GG_CUDA(gg_launch_pdl(k_spmv_pull_hot<T>, grid, block, smem, s, ha, xv, w, (const T *)hot_tab, yi, next, V));
            }
            else
            {
                size_t pad;
                const dim3 grid(gg_persistent_grid((const void *)k_spmv_pull<T>, t->ntiles, (int)shape.ctas, &pad)), block(GG_TILE_NT);
                const SpmvGather<T> op{w, xv};
                if (p->profile)
                    k_spmv_pull<T><<<grid, block, 0, s>>>(g->in_off, g->in_adj, t->coord, t->ntiles, V, yi, next, op);
                else
                    GG_CUDA(gg_launch_pdl(k_spmv_pull<T>, grid, block, pad, s, g->in_off, g->in_adj, t->coord, t->ntiles, V, yi,
                                          next, op));
            }
        }
        else
        {
            if (tags)
                k_spmv_push<T, true><<<gg_push_grid((const void *)k_spmv_push<T, true>, t->ntiles, push_smem<float>()), PUSH_NT,
                                       push_smem<float>(), s>>>(g->out_off, g->out_adj, t->coord, t->ntiles, V, tags, w, xv, y);
            else
                k_spmv_push<T, false><<<gg_persistent_grid((const void *)k_spmv_push<T, false>, t->ntiles), GG_TILE_NT, 0, s>>>(
                    g->out_off, g->out_adj, t->coord, t->ntiles, V, tags, w, xv, y);
        }
        if (p->profile)
        {
            cudaEvent_t e;
            GG_CHECK(gg_event_at(g, (uint32_t)evs.size(), &e));
            GG_CUDA(cudaEventRecord(e, s));
            evs.push_back(e);
        }
        launches++;
        timed++;
    }
    GG_CUDA(cudaGetLastError());
    return GG_OK;
}

} // namespace

extern "C" gg_status gg_spmv(gg_graph *g, const gg_spmv_params *p, const float *x, float *x_out, float *y,
                             gg_spmv_result *r, void *stream)
{
    GgRange range("gg_spmv");
    if (!g || !p) return gg_fail(GG_ERR_INVALID, "NULL argument");
    if (p->mode > 3) return gg_fail(GG_ERR_INVALID, "unknown SpMV mode");
    if (p->storage > 2) return gg_fail(GG_ERR_INVALID, "unknown storage");
    const bool pull = p->mode == GG_SPMV_PULL || p->mode == GG_SPMV_PULL_FX;
    if (pull && (!g->in_off || !g->in_w)) return gg_fail(GG_ERR_INVALID, "pull SpMV needs GG_MAP_IN|GG_MAP_IN_W");
    if (!pull && (!g->out_off || !g->out_w)) return gg_fail(GG_ERR_INVALID, "push SpMV needs GG_MAP_OUT|GG_MAP_OUT_W");
    if (!g->out_deg) return gg_fail(GG_ERR_INVALID, "mapping has no out-degrees");
    cudaStream_t s = gg_stream(g, stream);
    const uint32_t V = g->V;
    gg_spmv_result res;
    memset(&res, 0, sizeof(res));
    void *xf, *yv, *xin = nullptr, *chk, *pin;
    GG_CHECK(gg_pinned(g, GG_STAGE_VALUES * 8 + 64, &pin)); /* before the launches: allocating it may wait for them */
    GG_CHECK(gg_work(g, 0, ((size_t)V + 16) * 4, &xf));
    GG_CHECK(gg_work(g, 11, ((size_t)V + 16) * 4, &yv));
    GG_CHECK(gg_work(g, 10, 64, &chk));
    GG_CUDA(cudaMemsetAsync(chk, 0, 64, s));
    if (x)
    {
        GG_CHECK(gg_work(g, 13, ((size_t)V + 16) * 4, &xin));
        GG_CUDA(cudaMemcpyAsync(xin, x, (size_t)V * 4, cudaMemcpyHostToDevice, s));
    }
    std::vector<cudaEvent_t> evs;
    uint32_t launches = 0, timed = 0;
    if (V > 0)
    {
        if (p->mode == GG_SPMV_PULL || p->mode == GG_SPMV_PUSH)
        {
            gg_status st = p->storage == GG_STORE_BF16
                               ? spmv_fp<__nv_bfloat16>(g, p, (const float *)xin, (float *)xf, (float *)yv, s, launches, timed, evs)
                           : p->storage == GG_STORE_F16
                               ? spmv_fp<__half>(g, p, (const float *)xin, (float *)xf, (float *)yv, s, launches, timed, evs)
                               : spmv_fp<float>(g, p, (const float *)xin, (float *)xf, (float *)yv, s, launches, timed, evs);
            if (st != GG_OK) return st;
        }
        else
        {
            gg_tiles *t;
            GG_CHECK(gg_tiles_get(g, pull ? 1 : 0, s, &t));
            void *xq, *y64 = nullptr;
            GG_CHECK(gg_work(g, 12, ((size_t)V + 16) * 8, &xq));
            GG_CHECK(gg_work(g, 14, ((size_t)V + 16) * 8, &y64));
            GG_CUDA(cudaMemsetAsync(y64, 0, ((size_t)V + 16) * 8, s));
            k_spmv_x<float><<<grid_v(V), 256, 0, s>>>(g->out_deg, (const float *)xin, (float *)xf, nullptr,
                                                      pull ? (uint32_t *)xq : nullptr,
                                                      pull ? nullptr : (unsigned long long *)xq, (float *)yv, V);
            launches++;
            const uint32_t *tags = nullptr;
            if (!pull) GG_CHECK(gg_push_tags(g, p->iterations, s, &tags));
            for (uint32_t it = 0; it < p->iterations; it++)
            {
                if (p->profile)
                {
                    cudaEvent_t e;
                    GG_CHECK(gg_event_at(g, (uint32_t)evs.size(), &e));
                    GG_CUDA(cudaEventRecord(e, s));
                    evs.push_back(e);
                }
                if (pull)
                {
                    k_spmv_pull_fx<<<gg_persistent_grid((const void *)k_spmv_pull_fx, t->ntiles, GG_PULL_CTAS_PER_SM), GG_TILE_NT, 0, s>>>(
                        g->in_off, g->in_adj, t->coord, t->ntiles, V, (unsigned long long *)y64,
                        SpmvFxGather{g->in_w, (const uint32_t *)xq});
                    k_spmv_fx_pull_out<<<grid_v(V), 256, 0, s>>>((unsigned long long *)y64, (float *)yv, V);
                    launches++;
                }
                else
                {
                    constexpr size_t smem = push_smem<unsigned long long>();
                    if (tags)
                        k_spmv_push_fx<true><<<gg_push_grid((const void *)k_spmv_push_fx<true>, t->ntiles, smem), PUSH_NT, smem, s>>>(
                            g->out_off, g->out_adj, t->coord, t->ntiles, V, tags, g->out_w, (const unsigned long long *)xq,
                            (unsigned long long *)y64);
                    else
                        k_spmv_push_fx<false><<<gg_persistent_grid((const void *)k_spmv_push_fx<false>, t->ntiles), GG_TILE_NT, 0, s>>>(
                            g->out_off, g->out_adj, t->coord, t->ntiles, V, tags, g->out_w, (const unsigned long long *)xq,
                            (unsigned long long *)y64);
                }
                if (p->profile)
                {
                    cudaEvent_t e;
                    GG_CHECK(gg_event_at(g, (uint32_t)evs.size(), &e));
                    GG_CUDA(cudaEventRecord(e, s));
                    evs.push_back(e);
                }
                launches++;
                timed++;
            }
            if (!pull)
            {
                k_spmv_fx64_out<<<grid_v(V), 256, 0, s>>>((const unsigned long long *)y64, (float *)yv, V);
                launches++;
            }
        }
        k_spmv_checksum<<<grid_v(V), 256, 0, s>>>((const float *)yv, V, (unsigned long long *)chk);
        launches++;
        GG_CUDA(cudaGetLastError());
    }
    long long hundredths = 0;
    /* small results through the page-locked scratch, with one wait */
    const bool stage = V <= GG_STAGE_VALUES;
    float *pin_y = (float *)((char *)pin + 64), *pin_x = pin_y + GG_STAGE_VALUES;
    GG_CUDA(cudaMemcpyAsync(pin, chk, 8, cudaMemcpyDeviceToHost, s));
    if (stage && y && V) GG_CUDA(cudaMemcpyAsync(pin_y, yv, (size_t)V * 4, cudaMemcpyDeviceToHost, s));
    if (stage && x_out && V) GG_CUDA(cudaMemcpyAsync(pin_x, xf, (size_t)V * 4, cudaMemcpyDeviceToHost, s));
    GG_CHECK(gg_wait(s));
    memcpy(&hundredths, pin, 8);
    if (stage)
    {
        if (y && V) memcpy(y, pin_y, (size_t)V * 4);
        if (x_out && V) memcpy(x_out, pin_x, (size_t)V * 4);
    }
    else
    {
        if (y) GG_CHECK(gg_copy_d2h(y, yv, (size_t)V * 4, s));
        if (x_out) GG_CHECK(gg_copy_d2h(x_out, xf, (size_t)V * 4, s));
    }
    res.checksum = (double)hundredths / 100.0;
    res.launches = launches;
    res.spmv_launches = timed;
    if (p->profile)
        for (size_t i = 0; i + 1 < evs.size(); i += 2) res.spmv_ms += gg_event_ms(evs[i], evs[i + 1]);
    if (r) *r = res;
    return GG_OK;
}

/* ---- allocation-free SpMV pull -------------------------------------------------
 *
 * For callers that must not allocate GPU memory: code running inside an
 * allocator-free section (a host memory manager or plugin host that owns
 * every device allocation and forbids cudaMalloc/cudaFree from plugins, a
 * real-time loop where an allocation could block or fragment, or a process
 * whose device memory is fully reserved up front).  gg_spmv needs a
 * gg_graph mapping and work buffers that the runtime allocates; this entry
 * point instead takes the caller's device arrays and keeps its scratch (the
 * merge-path tile coordinates) in the file-scope array below, which exists
 * on every GPU that loads the library until the process exits; partial sums
 * of rows spanning tiles accumulate in the caller's y.
 */
#define GG_NOALLOC_SCRATCH_BYTES (4u << 20)

static __device__ __align__(256) unsigned char g_noalloc_scratch[GG_NOALLOC_SCRATCH_BYTES];

namespace {

size_t noalloc_coord_bytes(uint32_t ntiles) { return (((size_t)ntiles + 1) * sizeof(uint2) + 255) / 256 * 256; }

/* [a, a + an) and [b, b + bn) share a byte */
bool noalloc_overlap(const void *a, size_t an, const void *b, size_t bn)
{
    const uintptr_t pa = (uintptr_t)a, pb = (uintptr_t)b;
    return an && bn && pa < pb + bn && pb < pa + an;
}

} // namespace

extern "C" uint64_t gg_spmv_pull_noalloc_max_items(void)
{
    /* the largest V + E whose tile coordinates fit: (ntiles+1) of 8 bytes,
     * rounded to 256 */
    uint64_t lo = 0, hi = (uint64_t)GG_NOALLOC_SCRATCH_BYTES / 8 * GG_TILE_ITEMS;
    while (lo < hi)
    {
        const uint64_t mid = (lo + hi + 1) / 2;
        const uint64_t nt = (mid + GG_TILE_ITEMS - 1) / GG_TILE_ITEMS;
        if (noalloc_coord_bytes((uint32_t)nt) <= GG_NOALLOC_SCRATCH_BYTES)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

extern "C" gg_status gg_spmv_pull_noalloc(uint32_t V, uint32_t E, const uint32_t *in_off, const uint32_t *in_src,
                                          const float *w, const float *x, float *y, void *stream)
{
    if (V == 0) return GG_OK;
    if (!in_off || !x || !y || !w || (E && !in_src)) return gg_fail(GG_ERR_INVALID, "NULL device array");
    const uint64_t items = (uint64_t)V + E;
    const uint64_t max_items = gg_spmv_pull_noalloc_max_items();
    if (items > max_items)
        return gg_fail(GG_ERR_INVALID, "gg_spmv_pull_noalloc: V + E = " + std::to_string(items) +
                                           " exceeds the scratch limit of " + std::to_string(max_items) +
                                           " (4 MiB of tile scratch); use gg_spmv");
    /* y is written while the others are read (x through the read-only
     * path): an overlap would silently corrupt the product */
    const size_t vb = (size_t)V * sizeof(float), eb = (size_t)E * sizeof(float);
    if (noalloc_overlap(y, vb, x, vb) || noalloc_overlap(y, vb, w, eb) || noalloc_overlap(y, vb, in_src, eb) ||
        noalloc_overlap(y, vb, in_off, vb + sizeof(uint32_t)))
        return gg_fail(GG_ERR_INVALID, "gg_spmv_pull_noalloc: y overlaps x, w, in_off or in_src");
    /* The host-side name of the array is not a device address: ask the
     * runtime for it on every call, in the context current now.  A cached
     * address would go stale when the context it came from is reset or when
     * the caller switches to another context of the same device; the lookup
     * is host-side and queues no work.  The first call in a context loads the
     * library's kernels into it. */
    void *base = nullptr;
    GG_CUDA(cudaGetSymbolAddress(&base, g_noalloc_scratch));
    const uint32_t ntiles = (uint32_t)((items + GG_TILE_ITEMS - 1) / GG_TILE_ITEMS);
    uint2 *coord = (uint2 *)base;
    cudaStream_t s = (cudaStream_t)stream;
    /* the coordinates are rewritten on every call; y is the row-sum array
     * and starts at zero (rows spanning tiles are added into it) */
    GG_CHECK(gg_launch_tile_coords(in_off, V, E, ntiles, coord, s));
    GG_CUDA(cudaMemsetAsync(y, 0, (size_t)V * sizeof(float), s));
    k_spmv_pull<float><<<gg_persistent_grid((const void *)k_spmv_pull<float>, ntiles, GG_PULL_CTAS_PER_SM), GG_TILE_NT, 0, s>>>(
        in_off, in_src, coord, ntiles, V, y, nullptr, SpmvGather<float>{w, x});
    GG_CUDA(cudaGetLastError());
    return GG_OK;
}
