/*
 * Device-side helpers shared by the kernels: storage conversions, the
 * fixed-point formats, warp/block reductions, and the merge-path tile
 * engine that every pull gather and push scatter is built on.
 */
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cstdint>

#include "gg_internal.h"

namespace gg {

/* ---- storage types of gathered values ------------------------------------ */

template <class T> __device__ __forceinline__ float to_f32(T x);
template <> __device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <> __device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }

template <class T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }

/* ---- fixed point (Q32.32 / Q16.16 / Q4.12 / Q2.6), same as the oracle ---- */

__device__ __forceinline__ double fx64_to_double(uint64_t f) { return __dmul_rn(__ull2double_rn(f), 1.0 / 4294967296.0); }
__device__ __forceinline__ uint64_t fx64_mul(uint64_t a, uint64_t b)
{
    /* (a*b) >> 32 of the 128-bit product */
    uint64_t lo = a * b;
    uint64_t hi = __umul64hi(a, b);
    return (hi << 32) | (lo >> 32);
}
/* The conversions below use no FP64: sm_103a issues FP64 at about 1/64 of the
 * FP32 rate, and a few FP64 operations per vertex or edge were what the
 * passes that call them spent their time on.  The scales are powers of two,
 * so the FP32 products are exact and the results are those of the FP64 form. */

/* trunc(x * 2^32) in 64 bits, saturating; NaN and negatives give 0 */
__device__ __forceinline__ uint64_t fx64_from_float(float x)
{
    if (!(x > 0.0f)) return 0ull;
    if (x >= 4294967296.0f) return ~0ull;
    return __float2ull_rz(__fmul_rn(x, 4294967296.0f));
}
/* trunc(x * scale), at most maxv; scale a power of two */
__device__ __forceinline__ uint32_t fx_from_float(float x, float scale, uint32_t maxv)
{
    const float t = __fmul_rn(x, scale);
    if (!(t > 0.0f)) return 0u;
    return min(__float2uint_rz(t), maxv);
}
/* f * inv_scale rounded once to FP32; inv_scale a power of two.  From 2^53 on
 * the FP64 form rounds twice, which is kept. */
__device__ __forceinline__ float fx_to_float(uint64_t f, float inv_scale)
{
    if (f >> 53) return __double2float_rn(__dmul_rn(__ull2double_rn(f), (double)inv_scale));
    return __fmul_rn(f >> 32 ? __ull2float_rn(f) : __uint2float_rn((uint32_t)f), inv_scale);
}

/* Clear a sum slot that was just read.  The store is made to wait for the
 * load (a branch on the value read): on GB300 a store issued to a sector
 * whose L2 read miss is still outstanding stalls that sector, and a pass
 * that read and cleared 64 MB with an independent store ran 7x slower than
 * with this dependent one.  Slots already zero are left alone (-0.0 stays;
 * the atomics that later add into it give the same sums). */
__device__ __forceinline__ void clear_after_read(float *p, float seen)
{
    if (seen != 0.0f) *p = 0.0f;
}
__device__ __forceinline__ void clear_after_read(unsigned long long *p, unsigned long long seen)
{
    if (seen != 0ull) *p = 0ull;
}

/* ---- reductions --------------------------------------------------------- */

template <class T> __device__ __forceinline__ T warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

/* Programmatic dependent launch: a kernel launched with
 * cudaLaunchAttributeProgrammaticStreamSerialization (gg_launch_pdl) may be
 * launched while the kernel before it on the stream still runs; it calls
 * pdl_wait before its first access to memory that kernel writes, which
 * returns once that kernel has completed and its writes are visible (at
 * once for a kernel launched without the attribute).  pdl_trigger lets the
 * next such kernel launch before this one has ended. */
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

/* two FP32 additions or subtractions in one instruction, each rounded as FADD */
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    float2 r;
    asm("{\n\t.reg .b64 ra, rb, rc;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rc, ra, rb;\n\tmov.b64 {%0, %1}, rc;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    float2 r;
    asm("{\n\t.reg .b64 ra, rb, rc;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "sub.rn.f32x2 rc, ra, rb;\n\tmov.b64 {%0, %1}, rc;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

/* A running sum of floats in three of them: hi takes the sum, mid the rounding
 * errors of hi, lo those of mid (Knuth's two-sum), about 72 bits, in FP32
 * operations: one FP64 addition per vertex bounds the passes that sum a residual
 * (k_pr_update of a 16.7M-vertex graph: 78 us in FP64, 60 in FP32).  Where FP32
 * ends -- sums past SUM_MAX, infinities, NaN -- the sum so far is added to the
 * FP64 total `over` instead. */
struct LongSum
{
    static constexpr float SUM_MAX = 8.507059173e37f; /* 2^126 */
    float hi = 0.0f, mid = 0.0f, lo = 0.0f;
    static __device__ __forceinline__ float two_sum(float &s, float x)
    {
        const float t = __fadd_rn(s, x), z = __fsub_rn(t, s);
        const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(x, z));
        s = t;
        return e;
    }
    __device__ __forceinline__ void add(float x, double *over)
    {
        if (fabsf(__fadd_rn(hi, x)) <= SUM_MAX)
            lo = __fadd_rn(lo, two_sum(mid, two_sum(hi, x)));
        else
        {
            /* keeps the conversions to FP64 in this branch */
            asm volatile("" : "+f"(hi), "+f"(mid), "+f"(lo), "+f"(x));
            atomicAdd(over, value() + (double)x);
            hi = mid = lo = 0.0f;
        }
    }
    /* neither sum past SUM_MAX / 2 */
    __device__ __forceinline__ void merge(float h, float m, float l)
    {
        const float e = two_sum(mid, two_sum(hi, h));
        lo = __fadd_rn(__fadd_rn(lo, l), __fadd_rn(e, two_sum(mid, m)));
    }
    __device__ __forceinline__ double value() const { return (double)hi + ((double)mid + (double)lo); }
    /* lane l: with lane l + o */
    __device__ __forceinline__ void merge_down(int o)
    {
        merge(__shfl_down_sync(0xffffffffu, hi, o), __shfl_down_sync(0xffffffffu, mid, o),
              __shfl_down_sync(0xffffffffu, lo, o));
    }
    /* to `over` if n sums of this size could leave FP32 */
    __device__ __forceinline__ void spill(int n, double *over)
    {
        if (fabsf(hi) <= SUM_MAX / (2 * n)) return;
        asm volatile("" : "+f"(hi), "+f"(mid), "+f"(lo));
        atomicAdd(over, value());
        hi = mid = lo = 0.0f;
    }
};

/* the same for the even and the odd vertex of a pair, by packed instructions */
struct PairSum
{
    float2 hi = {0.0f, 0.0f}, mid = {0.0f, 0.0f}, lo = {0.0f, 0.0f};
    static __device__ __forceinline__ float2 two_sum(float2 &s, float2 x, float2 t)
    {
        const float2 z = sub2(t, s), e = add2(sub2(s, sub2(t, z)), sub2(x, z));
        s = t;
        return e;
    }
    __device__ __forceinline__ void add(float x, float y, double *over)
    {
        float2 v = make_float2(x, y), t = add2(hi, v);
        if (fabsf(t.x) <= LongSum::SUM_MAX && fabsf(t.y) <= LongSum::SUM_MAX)
        {
            const float2 e = two_sum(hi, v, t);
            lo = add2(lo, two_sum(mid, e, add2(mid, e)));
        }
        else
        {
            asm volatile("" : "+f"(v.x), "+f"(v.y));
            atomicAdd(over, part(0).value() + part(1).value() + (double)v.x + (double)v.y);
            hi = mid = lo = make_float2(0.0f, 0.0f);
        }
    }
    __device__ __forceinline__ LongSum part(int odd) const
    {
        LongSum s;
        s.hi = odd ? hi.y : hi.x;
        s.mid = odd ? mid.y : mid.x;
        s.lo = odd ? lo.y : lo.x;
        return s;
    }
    /* both together */
    __device__ __forceinline__ LongSum total(double *over) const
    {
        LongSum s = part(0);
        if (fabsf(hi.x) <= LongSum::SUM_MAX / 2 && fabsf(hi.y) <= LongSum::SUM_MAX / 2)
            s.merge(hi.y, mid.y, lo.y);
        else
            atomicAdd(over, part(1).value());
        return s;
    }
};

/* sum over the warp; the result is valid in lane 0 */
__device__ __forceinline__ double warp_sum(LongSum s)
{
    if (__any_sync(0xffffffffu, fabsf(s.hi) > LongSum::SUM_MAX / 64)) return warp_sum(s.value());
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s.merge_down(o);
    return s.value();
}

/* Block-wide sum of (LongSum, uint32) pairs, once per kernel; the result is valid in
 * thread 0.  Groups of four lanes are joined in their warps, the rest by one
 * warp: all of it in every warp took 1.5 us of a vertex pass, and a slot per
 * thread (3 KB) kept the blocks off SMs whose shared memory the gather before
 * them had sized for itself (a call on 7M edges 1.01 -> 1.10 ms). */
template <int NT>
__device__ __forceinline__ void block_sum2(LongSum s, uint32_t b, double &a, uint32_t &n)
{
    constexpr uint32_t SLOTS = NT / 4;
    __shared__ float part[3][SLOTS];
    __shared__ uint32_t sb[NT / 32];
    __shared__ double s_wide; /* sums near the end of FP32 */
    const uint32_t t = threadIdx.x, l = t & 31;
    if (t == 0) s_wide = 0.0;
    __syncthreads();
    s.spill(NT, &s_wide);
#pragma unroll
    for (int o = 16; o >= 8; o >>= 1) s.merge_down(o);
    b = __reduce_add_sync(0xffffffffu, b);
    if (l < 8)
    {
        const uint32_t k = (t >> 5) * 8 + l;
        part[0][k] = s.hi;
        part[1][k] = s.mid;
        part[2][k] = s.lo;
    }
    if (l == 0) sb[t >> 5] = b;
    __syncthreads();
    a = 0.0;
    n = 0u;
    if (t >= 32) return;
    LongSum all;
#pragma unroll
    for (uint32_t k = l; k < SLOTS; k += 32) all.merge(part[0][k], part[1][k], part[2][k]);
    a = warp_sum(all) + s_wide;
    n = __reduce_add_sync(0xffffffffu, l < NT / 32 ? sb[l] : 0u);
}

/* Asynchronous 4-byte global -> shared copy (cp.async, cached in L1): the
 * issuing thread holds no register for it and does not stall until
 * cp_async_wait_all.  Both addresses must be 4-byte aligned. */
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem)
{
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
/* Asynchronous 16-byte copy through L2 only (cp.async.cg), so staged
 * streams do not displace the L1-resident gather data.  Both addresses must
 * be 16-byte aligned. */
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
/* Wait for this thread's cp.async copies; a __syncwarp after it makes every
 * lane's copies visible to the whole warp. */
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

/* Streaming 4-byte load that does not allocate in L1 (the neighbour ids are
 * read once per launch). */
__device__ __forceinline__ uint32_t ldg_stream(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

/*
 * One warp copies src[i0 .. i0+n) into shared memory asynchronously, word
 * i0+k landing at dst[(i0 & 3) + k]; dst must be 16-byte aligned with room
 * for n + 3 words.  From a 16-byte-aligned src the body moves in 16-byte
 * chunks starting at the aligned word at or below i0 (words before i0 are
 * copied too, never words at or past i0+n); the last 1-3 words and any
 * unaligned src go word by word.  Returns i0 & 3.
 */
__device__ __forceinline__ uint32_t stage_words(uint32_t *dst, const uint32_t *src, uint32_t i0, uint32_t n,
                                                uint32_t lane)
{
    const uint32_t first = i0 & 3u;
    if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0)
    {
        const uint32_t base = i0 - first, total = first + n, full = total >> 2;
        for (uint32_t c = lane; c < full; c += 32) cp_async16(dst + 4u * c, src + base + 4u * c);
        if (lane < (total & 3u)) cp_async4(dst + 4u * full + lane, src + base + 4u * full + lane);
    }
    else
        for (uint32_t k = lane; k < n; k += 32) cp_async4(dst + first + k, src + i0 + k);
    return first;
}

__device__ __forceinline__ void atomic_add_acc(float *p, float v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_acc(unsigned long long *p, unsigned long long v) { atomicAdd(p, v); }

/* ---- merge-path tiles ------------------------------------------------------
 *
 * A CSR with V rows and E edges is the merge of two lists: the V row-end
 * offsets and the E edge slots.  Cutting that merge into tiles of
 * GG_TILE_ITEMS items balances work whatever the degree distribution
 * (Merrill & Garland, "Merge-based parallel sparse matrix-vector
 * multiplication", SC'16).  coord[t] = (rows ended, edges consumed) at
 * diagonal t*GG_TILE_ITEMS.  Each tile is consumed by one warp.
 *
 * A row whose items fall in more than one tile gets each tile's partial
 * sum added atomically; a row lying wholly in one tile is stored by that
 * tile.  No tile waits for another.
 */

__device__ __forceinline__ uint2 merge_path_search(uint32_t diag, const uint32_t *row_end, uint32_t nrows,
                                                   uint32_t nedges, uint32_t edge_base)
{
    /* row_end[i] is the (absolute) end offset of local row i; edges are
     * numbered from edge_base.  Returns (rows consumed, edges consumed). */
    uint32_t lo = diag > nedges ? diag - nedges : 0;
    uint32_t hi = diag < nrows ? diag : nrows;
    while (lo < hi)
    {
        uint32_t mid = (lo + hi) >> 1;
        if ((row_end[mid] - edge_base) + mid < diag)
            lo = mid + 1;
        else
            hi = mid;
    }
    return make_uint2(lo, diag - lo);
}

/* Per-warp tile geometry shared by the pull and push engines. */
struct TileGeom
{
    uint32_t i0, j0, i1, j1, nrows, nedges, nitems;
    __device__ __forceinline__ void load(const uint2 *coord, uint32_t tile, uint32_t V)
    {
        const uint2 c0 = coord[tile], c1 = coord[tile + 1];
        i0 = c0.x; j0 = c0.y; i1 = c1.x; j1 = c1.y;
        /* rows touched: i0 .. last_row; row i1 (if < V) may have edges here
         * but its end item lies in a later tile */
        const uint32_t last_row = i1 < V ? i1 : V - 1;
        nrows = (i1 < V || i0 < V) ? last_row - i0 + 1 : 0;
        nedges = j1 - j0;
        nitems = (i1 - i0) + nedges;
    }
};

/* Gather loads issued where they are written (inline PTX is not moved), so a
 * tile's loads stay in flight while the previous tile is reduced; the
 * values are read-only for the launch (non-coherent path). */
__device__ __forceinline__ float ldg_val(const float *p)
{
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg_val(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned long long ldg_val(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.global.nc.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint16_t ldg_val(const uint16_t *p)
{
    uint16_t v;
    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint8_t ldg_val(const uint8_t *p)
{
    uint32_t v;
    asm volatile("ld.global.nc.u8 %0, [%1];" : "=r"(v) : "l"(p));
    return (uint8_t)v;
}
__device__ __forceinline__ __nv_bfloat16 ldg_val(const __nv_bfloat16 *p)
{
    return __ushort_as_bfloat16(ldg_val(reinterpret_cast<const uint16_t *>(p)));
}
__device__ __forceinline__ __half ldg_val(const __half *p) { return __ushort_as_half(ldg_val(reinterpret_cast<const uint16_t *>(p))); }

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
/* wait until at most one committed group of this thread is still pending */
__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

template <int IPT>
__device__ __forceinline__ void load_ids(uint32_t (&id)[IPT], const uint32_t *adj, uint32_t j0, uint32_t j1,
                                         uint32_t lane)
{
#pragma unroll
    for (int g = 0; g < IPT; g++)
    {
        const uint32_t e = j0 + lane + 32u * g;
        if (e < j1) id[g] = ldg_stream(adj + e);
    }
}

/* rows of a tile with at least one item in it: i0 .. last row (row i1 when
 * i1 < V has items here but ends in a later tile) */
__device__ __forceinline__ uint32_t tile_rows(uint2 c0, uint2 c1, uint32_t V)
{
    const uint32_t last_row = c1.x < V ? c1.x : V - 1;
    return (c1.x < V || c0.x < V) ? last_row - c0.x + 1 : 0;
}

/*
 * The pull engine: sums[r] = sum over the CSC row r of op's edge terms, for
 * every row, by persistent warps over merge-path tiles.  Op supplies:
 *   typedef Acc;                       float, uint32_t or unsigned long long:
 *                                      sums within a tile
 *   typedef Sum;                       the type of sums[] (Acc, or 64 bits
 *                                      where a tile's sums fit 32: 8- and
 *                                      16-bit formats, whose tile of at most
 *                                      2^10 edges sums to less than 2^26)
 *   typedef Raw;                       what one edge's gather loads
 *   Raw load(uint32_t e, uint32_t u) const;
 *                                      issue the loads of edge e with
 *                                      neighbour u (ldg_val)
 *   Acc value(const Raw &r) const;     the edge term, computed where the
 *                                      loads are first used
 * sums must be zero on entry for rows whose items span tiles: a row lying in
 * one tile is stored, the partials of a spanning row are added atomically
 * (the row epilogues that read sums clear it again).
 *
 * Each warp runs its tiles as a software pipeline: while tile A is reduced,
 * tile B's gathers and tile C's neighbour ids are in flight and tile B's row
 * offsets are landing in shared memory (cp.async, double-buffered), so a
 * tile's dependent load chain (ids, then values) overlaps the reduction of
 * the tile before it.  A tile is reduced along the merge path
 * (GG_TILE_IPT items per lane): a row ended inside a lane is stored
 * directly; the partial sum of the row open at the end of each lane is
 * combined across lanes by a warp-shuffle segmented scan.  Only __syncwarp
 * orders the phases.
 */
/* Per-warp shared staging of the pull engine: two buffers of row offsets
 * (each holding up to 3 words before the tile's first row, see stage_words,
 * 16-byte aligned), the tile's values and its row sums. */
template <int IPT, class Acc>
struct PullStage
{
    static constexpr uint32_t TW = 32 * IPT;
    static constexpr uint32_t OFFW = TW + 8;
    static constexpr size_t OFF_BYTES = (size_t)2 * OFFW * 4;
    static constexpr size_t VAL_BYTES = ((size_t)TW * sizeof(Acc) + 15) / 16 * 16;
    static constexpr size_t ROW_BYTES = ((size_t)(TW + 1) * sizeof(Acc) + 15) / 16 * 16;
    static constexpr size_t BYTES = OFF_BYTES + VAL_BYTES + ROW_BYTES;
};

/* The engine proper: this warp's tiles are tile, tile + nw, ...; s_offs
 * (2 * OFFW words), s_val (TW) and s_row (TW + 1) are its staging. */
template <int IPT, class Op>
__device__ __forceinline__ void warp_pull_sums_core(uint32_t *s_offs, typename Op::Acc *s_val,
                                                    typename Op::Acc *s_row, uint32_t tile, uint32_t nw,
                                                    const uint32_t *__restrict__ off, const uint32_t *__restrict__ adj,
                                                    uint32_t V, const uint2 *__restrict__ coord, uint32_t ntiles,
                                                    typename Op::Sum *sums, const Op &op)
{
    typedef typename Op::Acc Acc;
    typedef typename Op::Sum Sum;
    typedef typename Op::Raw Raw;
    constexpr uint32_t TW = PullStage<IPT, Acc>::TW;
    constexpr uint32_t OFFW = PullStage<IPT, Acc>::OFFW;
    const uint32_t lane = threadIdx.x & 31;
    if (tile >= ntiles) return;

    /* pipeline state: A = tile (gathers in flight in val, offsets staged in
     * buffer buf), B = tile + nw (ids in flight in id, offsets staged in
     * buf ^ 1), C = tile + 2nw (coordinates only) */
    const uint2 zero2 = make_uint2(0, 0);
    uint2 a0 = coord[tile], a1 = coord[tile + 1];
    uint2 b0 = zero2, b1 = zero2, c0 = zero2, c1 = zero2;
    if (tile + nw < ntiles) { b0 = coord[tile + nw]; b1 = coord[tile + nw + 1]; }
    if (tile + 2 * nw < ntiles) { c0 = coord[tile + 2 * nw]; c1 = coord[tile + 2 * nw + 1]; }
    uint32_t id[IPT];
    Raw val[IPT];
    load_ids<IPT>(id, adj, a0.y, a1.y, lane);
    uint32_t buf = 0;
    uint32_t shA = stage_words(s_offs, off, a0.x, tile_rows(a0, a1, V) + 1, lane);
    cp_async_commit();
    uint32_t shB = 0;
    if (tile + nw < ntiles) shB = stage_words((s_offs + OFFW), off, b0.x, tile_rows(b0, b1, V) + 1, lane);
    cp_async_commit();
#pragma unroll
    for (int g = 0; g < IPT; g++)
    {
        const uint32_t e = a0.y + lane + 32u * g;
        if (e < a1.y) val[g] = op.load(e, id[g]);
    }
    if (tile + nw < ntiles) load_ids<IPT>(id, adj, b0.y, b1.y, lane);

    for (; tile < ntiles; tile += nw)
    {
        const bool hasB = tile + nw < ntiles, hasC = tile + 2 * nw < ntiles;
        /* B's gathers, C's ids, D's coordinates */
        Raw nv[IPT];
        if (hasB)
        {
#pragma unroll
            for (int g = 0; g < IPT; g++)
            {
                const uint32_t e = b0.y + lane + 32u * g;
                if (e < b1.y) nv[g] = op.load(e, id[g]);
            }
        }
        if (hasC) load_ids<IPT>(id, adj, c0.y, c1.y, lane);
        uint2 d0 = zero2, d1 = zero2;
        if (tile + 3 * nw < ntiles)
        {
            d0 = coord[tile + 3 * nw];
            d1 = coord[tile + 3 * nw + 1];
        }

        /* tile A */
        const uint32_t i0 = a0.x, j0 = a0.y, i1 = a1.x, j1 = a1.y;
        const uint32_t nedges = j1 - j0;
        const uint32_t nend = i1 - i0; /* local rows whose end item is in this tile */
        const uint32_t nitems = nend + nedges;
#pragma unroll
        for (int g = 0; g < IPT; g++)
        {
            const uint32_t e = j0 + lane + 32u * g;
            if (e < j1) s_val[e - j0] = op.value(val[g]);
        }
        cp_async_wait_one();
        __syncwarp();
        const uint32_t *s_off = (s_offs + buf * OFFW) + shA;

        /* merge-path consumption; the first row a lane ends may have begun
         * in earlier lanes, so its sum waits for the carry scan */
        const uint32_t d = lane * IPT;
        uint32_t first_row = 0xffffffffu, key = 0xffffffffu;
        Acc first_sum = Acc(0), carry = Acc(0);
        bool first_done = false;
        if (d < nitems)
        {
            uint2 p = merge_path_search(d, s_off + 1, nend, nedges, j0);
            uint32_t ri = p.x, ej = p.y;
            first_row = ri;
            uint32_t rend = ri < nend ? s_off[ri + 1] - j0 : 0xffffffffu;
            Acc sum = Acc(0);
            const uint32_t dend = min(d + IPT, nitems);
            for (uint32_t k = d; k < dend; k++)
            {
                if (ej < rend)
                {
                    sum += s_val[ej];
                    ej++;
                }
                else
                {
                    if (!first_done)
                    {
                        first_sum = sum;
                        first_done = true;
                    }
                    else
                        s_row[ri] = sum;
                    sum = Acc(0);
                    ri++;
                    rend = ri < nend ? s_off[ri + 1] - j0 : 0xffffffffu;
                }
            }
            key = ri;
            carry = sum;
        }
        /* segmented inclusive scan of the open-row partials, keyed by row
         * (keys are non-decreasing across lanes) */
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t k2 = __shfl_up_sync(0xffffffffu, key, o);
            const Acc v2 = __shfl_up_sync(0xffffffffu, carry, o);
            if (lane >= (uint32_t)o && k2 == key) carry += v2;
        }
        {
            const uint32_t kp = __shfl_up_sync(0xffffffffu, key, 1);
            const Acc vp = __shfl_up_sync(0xffffffffu, carry, 1);
            if (first_done) s_row[first_row] = first_sum + ((lane > 0 && kp == first_row) ? vp : Acc(0));
            /* the row left open at the end of the tile (row i1) */
            if (i1 < V)
            {
                const uint32_t m = __ballot_sync(0xffffffffu, key == nend);
                const Acc tot = m ? __shfl_sync(0xffffffffu, carry, 31 - __clz((int)m)) : Acc(0);
                if (lane == 0) s_row[nend] = tot;
            }
        }
        __syncwarp();

        /* rows ending here are stored, except row i0 when it began in an
         * earlier tile (off[i0] < j0); that one and the open row i1 add
         * their partials to sums */
        for (uint32_t k = lane; k < nend; k += 32)
        {
            if (k == 0 && s_off[0] < j0)
            {
                if (s_off[1] > j0) atomic_add_acc(&sums[i0], (Sum)s_row[0]);
            }
            else
                sums[i0 + k] = s_row[k];
        }
        if (lane == 0 && i1 < V && s_off[nend] < j1) atomic_add_acc(&sums[i1], (Sum)s_row[nend]);
        __syncwarp();

        /* C's offsets into A's buffer; rotate */
        uint32_t shC = 0;
        if (hasC) shC = stage_words((s_offs + buf * OFFW), off, c0.x, tile_rows(c0, c1, V) + 1, lane);
        cp_async_commit();
#pragma unroll
        for (int g = 0; g < IPT; g++) val[g] = nv[g];
        a0 = b0; a1 = b1; b0 = c0; b1 = c1; c0 = d0; c1 = d1;
        shA = shB; shB = shC;
        buf ^= 1u;
    }
    cp_async_wait_all();
}

/* the engine with static per-warp staging, WARPS warps per CTA */
template <int IPT, int WARPS, class Op>
__device__ __forceinline__ void warp_pull_sums(const uint32_t *__restrict__ off, const uint32_t *__restrict__ adj,
                                               uint32_t V, const uint2 *__restrict__ coord, uint32_t ntiles,
                                               typename Op::Sum *sums, const Op &op)
{
    typedef typename Op::Acc Acc;
    constexpr uint32_t TW = PullStage<IPT, Acc>::TW, OFFW = PullStage<IPT, Acc>::OFFW;
    __shared__ __align__(16) uint32_t sm_off[WARPS][2 * OFFW];
    __shared__ Acc sm_val[WARPS][TW];
    __shared__ Acc sm_row[WARPS][TW + 1];
    const uint32_t w = threadIdx.x >> 5;
    warp_pull_sums_core<IPT>(sm_off[w], sm_val[w], sm_row[w], blockIdx.x * WARPS + w, gridDim.x * WARPS, off, adj,
                             V, coord, ntiles, sums, op);
}

/*
 * The push engine: the same warp tiles over the out-CSR; every edge
 * (row -> dst) applies op.scatter(row value, edge, dst).  Per-row data is
 * fetched once per lane segment through op.row_value(row).
 */
template <int IPT, int WARPS, class Op>
__device__ __forceinline__ void warp_push_staged(uint32_t *sm_off, uint32_t *sm_adj, const uint32_t *__restrict__ off,
                                                 const uint32_t *__restrict__ adj, uint32_t V,
                                                 const uint2 *__restrict__ coord, uint32_t ntiles, Op &op)
{
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nw = gridDim.x * WARPS;
    for (uint32_t tile = blockIdx.x * WARPS + w; tile < ntiles; tile += nw)
    {
        TileGeom t;
        t.load(coord, tile, V);
        /* edge j0+i at s_adj[i], row i0+k's offset at s_off[k] */
        const uint32_t *s_adj = sm_adj + stage_words(sm_adj, adj, t.j0, t.nedges, lane);
        const uint32_t *s_off = sm_off + stage_words(sm_off, off, t.i0, t.nrows + 1, lane);
        cp_async_wait_all();
        __syncwarp();
        const uint32_t d = lane * IPT;
        if (d < t.nitems)
        {
            const uint32_t nend = t.i1 - t.i0;
            uint2 p = merge_path_search(d, s_off + 1, nend, t.nedges, t.j0);
            uint32_t ri = p.x, ej = p.y;
            const uint32_t *ids = s_adj;
            uint32_t rend = ri < nend ? s_off[ri + 1] - t.j0 : 0xffffffffu;
            const uint32_t dend = min(d + IPT, t.nitems);
            bool have = false;
            typename Op::RowVal rv{};
            for (uint32_t k = d; k < dend; k++)
            {
                if (ej < rend)
                {
                    if (!have) { rv = op.row_value(t.i0 + ri); have = true; }
                    op.scatter(rv, t.j0 + ej, ids[ej]);
                    ej++;
                }
                else
                {
                    ri++;
                    have = false;
                    rend = ri < nend ? s_off[ri + 1] - t.j0 : 0xffffffffu;
                }
            }
        }
        __syncwarp();
    }
}

template <int IPT, int WARPS, class Op>
__device__ __forceinline__ void warp_push(const uint32_t *__restrict__ off, const uint32_t *__restrict__ adj,
                                          uint32_t V, const uint2 *__restrict__ coord, uint32_t ntiles, Op &op)
{
    constexpr uint32_t TW = 32 * IPT;
    __shared__ __align__(16) uint32_t sm_off[WARPS][TW + 8];
    __shared__ __align__(16) uint32_t sm_adj[WARPS][TW + 4];
    const uint32_t w = threadIdx.x >> 5;
    warp_push_staged<IPT, WARPS>(sm_off[w], sm_adj[w], off, adj, V, coord, ntiles, op);
}

/*
 * Table of the push scatters: the most frequent destinations (push.cu) are
 * added up in shared memory, one table per block, and each block adds them to
 * global memory once, at its end (shared-memory additions of FP32 run at 1 T/s
 * over random slots and 10 ns apart on one).  Per scatter, without -> with, R-MAT
 * with 16 edges per vertex: 1M edges 57 -> 22 us, 8M 204 -> 72; 33M (11 per
 * vertex) 541 -> 236.  Half the slots: 22, 81, 259; twice: 24, 66, 228.
 */
__device__ __forceinline__ uint32_t push_slot(uint32_t dst) { return (dst * GG_PUSH_HASH) >> (32 - PUSH_LOG); }

template <class T>
struct PushTable
{
    uint32_t *tag; /* the destination of each slot */
    T *val;
    T *out;
    /* smem: PUSH_SLOTS values, then as many tags */
    __device__ __forceinline__ PushTable(unsigned char *smem, const uint32_t *__restrict__ tags, T *o) : out(o)
    {
        val = reinterpret_cast<T *>(smem);
        tag = reinterpret_cast<uint32_t *>(val + PUSH_SLOTS);
        for (uint32_t i = threadIdx.x; i < PUSH_SLOTS; i += PUSH_NT)
        {
            tag[i] = tags[i];
            val[i] = T(0);
        }
        __syncthreads();
    }
    __device__ __forceinline__ void add(uint32_t dst, T v) const
    {
        const uint32_t slot = push_slot(dst);
        if (tag[slot] == dst)
            atomicAdd(&val[slot], v);
        else
            atomicAdd(&out[dst], v);
    }
    __device__ __forceinline__ void flush() const
    {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < PUSH_SLOTS; i += PUSH_NT)
        {
            const T v = val[i];
            if (v != T(0)) atomicAdd(&out[tag[i]], v);
        }
    }
};

/* warp_push for blocks of PUSH_WARPS warps, staged in dynamic shared memory */
constexpr size_t PUSH_STAGE = (size_t)PUSH_WARPS * (2 * GG_TILE_ITEMS + 12) * 4;
template <class T>
constexpr size_t push_smem()
{
    return PUSH_STAGE + (size_t)PUSH_SLOTS * (sizeof(T) + 4);
}

template <class T>
struct PushDirect
{
    T *out;
    __device__ __forceinline__ void add(uint32_t dst, T v) const { atomicAdd(&out[dst], v); }
};

template <class T, class Sink, class Row, class Term>
struct PushOp
{
    typedef T RowVal;
    Sink sink;
    Row row;
    Term term;
    __device__ __forceinline__ T row_value(uint32_t r) const { return row(r); }
    __device__ __forceinline__ void scatter(T rv, uint32_t e, uint32_t dst) const { sink.add(dst, term(rv, e)); }
};

/* out[dst] += term(row(r), e) over all edges e of every row r, by blocks of
 * PUSH_NT threads with push_smem<T>() bytes of dynamic shared memory and the
 * table, or of GG_TILE_NT threads without */
template <bool TABLE, class T, class Row, class Term>
__device__ __forceinline__ void push_scatter(const uint32_t *__restrict__ off, const uint32_t *__restrict__ adj, uint32_t V,
                                             const uint2 *__restrict__ coord, uint32_t ntiles,
                                             const uint32_t *__restrict__ tags, T *out, Row row, Term term)
{
    if constexpr (TABLE)
    {
        extern __shared__ __align__(1024) unsigned char gg_dyn[];
        const PushTable<T> table(gg_dyn + PUSH_STAGE, tags, out);
        PushOp<T, PushTable<T>, Row, Term> op{table, row, term};
        uint32_t *st = reinterpret_cast<uint32_t *>(gg_dyn) + (threadIdx.x >> 5) * (2 * GG_TILE_ITEMS + 12);
        warp_push_staged<GG_TILE_IPT, PUSH_WARPS>(st, st + GG_TILE_ITEMS + 8, off, adj, V, coord, ntiles, op);
        table.flush();
    }
    else
    {
        PushOp<T, PushDirect<T>, Row, Term> op{PushDirect<T>{out}, row, term};
        warp_push<GG_TILE_IPT, GG_TILE_WARPS>(off, adj, V, coord, ntiles, op);
    }
}

/*
 * Grid-wide barrier over the co-resident blocks of a cooperative launch, on
 * a control block `ctl` of GG_BAR_BYTES zeroed before the launch: an arrival
 * counter per group of blocks, at 1024 + 128 g (a 128-byte line each: one
 * address takes an addition every 5 ns).  A block adds to its group's counter
 * and the lanes of its first warp each poll one group's: two memory round trips
 * (through a root counter and a release word per group it was five: a search of
 * 1,000 vertices 71 -> 63 us, of R-MAT-22 207 -> 190).  The counters only grow (barrier `gen` completes a group
 * at (gen + 1) * group size arrivals), so no arrival waits for a counter to be
 * reset.  Ordering: the addition releases the block's writes, which the block
 * barrier before it has gathered; the polls acquire, and the block barrier
 * after them hands that on.  A wait gives up after limit_ns (globaltimer) and
 * sets *err; the block then reports false and the caller leaves, so the other
 * blocks give up at their next barrier and the launch ends with *err set, the
 * context intact.  Bytes 0..1023 of ctl are the caller's.
 */
constexpr unsigned int GG_BAR_GROUPS = 16;

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool grid_barrier(char *ctl, unsigned int *err, unsigned long long limit_ns,
                                             unsigned int &gen)
{
    __shared__ unsigned int s_ok;
    __syncthreads();
    if (threadIdx.x < 32)
    {
        const unsigned int lane = threadIdx.x;
        const unsigned int G = gridDim.x < GG_BAR_GROUPS ? gridDim.x : GG_BAR_GROUPS;
        if (lane == 0)
            asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(ctl + 1024 + 128 * (blockIdx.x % G)), "r"(1u)
                         : "memory");
        const char *word = ctl + 1024 + 128 * lane;
        const unsigned int want = lane < G ? (gen + 1) * ((gridDim.x - lane + G - 1) / G) : 0u;
        bool ok = true;
        const unsigned long long t0 = global_ns();
        /* the polls of 900 blocks hold the arrivals up at the L2 (a search of 30K
         * vertices: 77 us with 20 ns between polls, 69 with 150, 67 with 300 to
         * 800), those of 300 do not (a batched PageRank: 618 against 635) */
        const unsigned int pause = gridDim.x > 512u ? 400u : 20u;
        for (;;)
        {
            unsigned int v = want;
            if (lane < G) asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
            /* a counter past `want` has arrivals at the next barrier already */
            if (__all_sync(0xffffffffu, (int)(v - want) >= 0)) break;
            __nanosleep(pause);
            if (__shfl_sync(0xffffffffu, global_ns() - t0, 0) > limit_ns)
            {
                if (lane == 0) atomicExch(err, 1u);
                ok = false;
                break;
            }
        }
        if (lane == 0) s_ok = ok ? 1u : 0u;
    }
    __syncthreads();
    gen++;
    return s_ok != 0u;
}

} // namespace gg
