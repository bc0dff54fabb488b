/*
 * Batched personalised PageRank: K rank vectors over one graph, all advanced
 * by one pull gather per iteration.  There is no counterpart in the
 * reference's C API; per vector the arithmetic is the reference's pull
 * PageRank (pageRank.c:1026-1069: contribution = rank / outdeg, 0 for
 * outdeg 0, no dangling redistribution) with the uniform teleport replaced
 * by a teleport to the vector's seed set S_k:
 *     rank_0[v][k]  = c_k(v) / |S_k|              (c_k(v): occurrences of v in S_k)
 *     contrib[v][k] = rank[v][k] / outdeg(v)
 *     rank'[v][k]   = (1-d) c_k(v) / |S_k| + d * sum over in-edges (u,v) of contrib[u][k]
 *
 * Layout: contributions vertex-major, [V][KP] with KP = K rounded up to 16,
 * 32 or 64, stored in FP32 or BF16 and summed in FP32, so an edge gathers one
 * contiguous row of 32 to 256 bytes.
 *
 * The gather.  Little's law bounds it: at ~1 us under load an SM needs 50 KB
 * and more of rows in flight, and a warp that holds rows in registers has room
 * for a few (four to six were in flight per half warp, 25 KB per SM).  So rows
 * land in shared memory: a warp owns a tile of edges, asks for the rows of a
 * chunk of up to 32 edges with 16-byte asynchronous copies (cp.async.cg: L2
 * only, so rows rewritten inside the persistent launch are read fresh), and
 * sums a chunk while the next ones arrive; up to 8 KB of landing space per warp
 * (4 KB for 32-byte rows), 20 warps per SM.  The half warps take alternate edges, each lane KP / 16
 * columns, so one shared-memory read serves two edges and the additions are
 * packed (add.f32x2): issue slots are what is left to bound the loop.  The two
 * halves' sums are exchanged and added where the row ends, for every KP: the
 * order of a vector's additions does not depend on the vectors batched with it.
 *
 * Rows are finished where they end: rank = teleport + d * sum (the teleport
 * row comes through a per-vertex seed index), contribution = rank *
 * (1 / outdeg) with the reciprocal computed once per vertex (within an ulp of
 * the division); FP32 ranks are only written by the last iteration.  The rows
 * with edges are listed once per mapping (hot.cu); a warp keeps the next 64
 * rows' ends, seed indices and reciprocals in registers and turns the ends
 * into one bit mask per chunk.  A row spanning tiles leaves its partial sum in
 * per-tile slots (the tile where it began or that it crosses: `tail`; the tile
 * where it ends: `head`) and the fix-up adds them in tile order, so every
 * vector's result is deterministic.  The fix-up also writes the rows without
 * in-edges.
 *
 * Landing rows must be 128-byte aligned in shared memory: 16 bytes off, the
 * asynchronous copies ran at half the rate.
 *
 * Measured, 20 iterations, K = 64 BF16 / FP32 and K = 16 FP32, against rows held
 * in registers: R-MAT-20 17.2 / 20.3 / 15.1 -> 7.3 / 8.6 / 6.0 ms; R-MAT-16
 * 3.6 / 3.6 / 5.6 -> 1.6 / 1.8 / 1.2 ms.
 */
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <unordered_map>
#include <vector>

#include "gg_device.cuh"

namespace {

using namespace gg;

constexpr uint32_t NO_SEED = 0xffffffffu;

/* the gather kernels: two CTAs of ten warps per SM (96 registers a thread;
 * 24 warps at 80 registers spilled in the persistent kernel's loop) */
constexpr int PPR_THREADS = 320, PPR_CTAS = 2, PPR_WARPS = PPR_THREADS / 32;

/* a pair of FP32 sums, added in one instruction (each sum rounded as FADD) */
struct F2
{
    float x, y;
};
__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    const float2 r = gg::add2(make_float2(a.x, a.y), make_float2(b.x, b.y));
    return F2{r.x, r.y};
}

/* One row of KP stored values, seen by a half warp: lane l of 16 reads the
 * columns from l * VPL on.  At a row's end the lane keeps OUT of them: the
 * lower half the first OUT, the upper half the rest (nothing at KP = 16). */
template <class CT, int KP>
struct PprRow
{
    static constexpr uint32_t BYTES = KP * sizeof(CT);
    static constexpr uint32_t VPL = KP / 16;
    static constexpr uint32_t OUT = VPL == 1 ? 1 : VPL / 2;
    static constexpr uint32_t CHUNK = 4096 / BYTES < 32 ? 4096 / BYTES : 32; /* edges per chunk */
    static constexpr uint32_t STAGE = CHUNK * BYTES;
    static constexpr uint32_t DEPTH = 8192 / STAGE < 4 ? 8192 / STAGE : 4;   /* chunks in flight */
    static constexpr uint32_t RING = DEPTH * STAGE;               /* landing bytes per warp */
    static constexpr uint32_t LPR = BYTES / 16;                   /* lanes that copy one row */
    static constexpr uint32_t RPI = 32 / LPR;                     /* rows per copy instruction */
    static constexpr uint32_t F2S = (VPL + 1) / 2;

    /* first column this lane keeps at a row's end, and whether it keeps any */
    static __device__ __forceinline__ uint32_t out_col(uint32_t lane)
    {
        return (lane & 15) * VPL + (VPL > 1 ? (lane >> 4) * OUT : 0);
    }
    static __device__ __forceinline__ bool keeps(uint32_t lane) { return VPL > 1 || lane < 16; }

    /* this lane's columns of the row landed at shared address `at` (the
     * lane's own offset included); BF16 -> FP32 is exact, the low half is the
     * lower column */
    static __device__ __forceinline__ void read(uint32_t at, F2 *v)
    {
        if constexpr (sizeof(CT) == 4 && VPL == 4)
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[1].x), "=f"(v[1].y) : "r"(at) : "memory");
        else if constexpr (sizeof(CT) == 4 && VPL == 2)
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v[0].x), "=f"(v[0].y) : "r"(at) : "memory");
        else if constexpr (sizeof(CT) == 4)
        {
            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v[0].x) : "r"(at) : "memory");
            v[0].y = 0.0f;
        }
        else if constexpr (VPL == 4)
        {
            uint32_t a, b;
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "r"(at) : "memory");
            v[0] = F2{__uint_as_float(a << 16), __uint_as_float(a & 0xffff0000u)};
            v[1] = F2{__uint_as_float(b << 16), __uint_as_float(b & 0xffff0000u)};
        }
        else if constexpr (VPL == 2)
        {
            uint32_t a;
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(a) : "r"(at) : "memory");
            v[0] = F2{__uint_as_float(a << 16), __uint_as_float(a & 0xffff0000u)};
        }
        else
        {
            uint16_t a;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(a) : "r"(at) : "memory");
            v[0] = F2{__uint_as_float((uint32_t)a << 16), 0.0f};
        }
    }
    static __device__ __forceinline__ void store(CT *p, const float *c)
    {
        if constexpr (sizeof(CT) == 4 && OUT == 2)
            *reinterpret_cast<float2 *>(p) = make_float2(c[0], c[1]);
        else if constexpr (OUT == 2)
            *reinterpret_cast<__nv_bfloat162 *>(p) = __floats2bfloat162_rn(c[0], c[1]);
        else
            *p = from_f32<CT>(c[0]);
    }
};

template <uint32_t N>
__device__ __forceinline__ void load_f32(const float *p, float *v)
{
    if constexpr (N == 2)
    {
        const float2 t = *reinterpret_cast<const float2 *>(p);
        v[0] = t.x;
        v[1] = t.y;
    }
    else
        v[0] = *p;
}
template <uint32_t N>
__device__ __forceinline__ void store_f32(float *p, const float *v)
{
    if constexpr (N == 2)
        *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
    else
        *p = v[0];
}

template <class CT>
struct PprArgs
{
    const uint32_t *off, *adj, *seed_idx;
    const float *inv_deg; /* 1 / out-degree, 0 for out-degree 0 */
    const uint32_t *rows; /* the rows with edges, padded with V */
    const uint32_t *seg0; /* per tile: its first row end; bit 31: the row began earlier */
    uint32_t ntiles, V, E;
    uint32_t tile; /* edges per tile (gg_ppr_tile): a power of two, at least a chunk's; below 256 every
                    * tile needs a resident warp of its own (ppr_tiles_fit) */
    const CT *cin;
    CT *cout;
    float *rank;       /* [V][rs]: ranks of the vectors in rank_mask are written here */
    unsigned long long rank_mask; /* vectors whose ranks this iteration writes (their last) */
    unsigned long long zero_mask; /* vectors whose contributions are stored as zero (a freed slot) */
    const float *tele; /* [nseeds][rs]: (1-d) c_k(v) / |S_k| of seed vertex i */
    float *head;       /* [ntiles][KP]: partial of the row that ends in the tile but began before it */
    float *tail;       /* [ntiles][KP]: partial of the row left open at the tile's end */
    float damp;
};

/* what changes from one iteration to the next: the contributions read and
 * written, and the vectors whose ranks this iteration writes (kept apart
 * from PprArgs so that the persistent kernel reads PprArgs from its
 * parameter space instead of copying it into registers) */
template <class CT>
struct PprIter
{
    const CT *cin;
    CT *cout;
    unsigned long long rank_mask;
};

/* the stores of a row end in an iteration where some vectors write their
 * ranks or retire (rare: the loops have an instance of their own for it) */
template <int KP, class CT>
__device__ __forceinline__ void ppr_store_masked(CT *cout, float *rank, unsigned long long rank_mask,
                                              unsigned long long zero_mask, size_t o, const float *r, float *c,
                                              uint32_t col)
{
    constexpr uint32_t VPL = PprRow<CT, KP>::OUT;
    const uint32_t zero = (uint32_t)(zero_mask >> col) & ((1u << VPL) - 1u);
    const uint32_t want = (uint32_t)(rank_mask >> col) & ((1u << VPL) - 1u);
#pragma unroll
    for (uint32_t k = 0; k < VPL; k++)
        if (zero >> k & 1u) c[k] = 0.0f;
    PprRow<CT, KP>::store(cout + o, c);
#pragma unroll
    for (uint32_t k = 0; k < VPL; k++)
        if (want >> k & 1u) rank[o + k] = r[k];
}

/* rank and contribution of row r from its sums (this lane's columns, from
 * `col`; every lane of the warp calls it, at KP = 16 the upper half stores
 * nothing): contribution = rank * (1 / out-degree).  RS: values per vertex
 * row of cin / cout / rank / tele -- KP, or 64 when only the first KP of
 * wider rows are run (the server's continuous batch).  MASKED: some vectors
 * write their ranks or retire in this iteration */
template <int KP, int RS, bool MASKED, class CT>
__device__ __forceinline__ void ppr_finish(const PprArgs<CT> &a, const PprIter<CT> &it, uint32_t r, const float *s,
                                           uint32_t si, float inv, uint32_t col, bool mine)
{
    constexpr uint32_t VPL = PprRow<CT, KP>::OUT;
    float rr[VPL], c[VPL];
#pragma unroll
    for (uint32_t k = 0; k < VPL; k++) rr[k] = __fmul_rn(a.damp, s[k]);
    if (si != NO_SEED)
    {
        float t[VPL];
        load_f32<VPL>(a.tele + (size_t)si * RS + col, t);
#pragma unroll
        for (uint32_t k = 0; k < VPL; k++) rr[k] = __fadd_rn(t[k], rr[k]);
    }
#pragma unroll
    for (uint32_t k = 0; k < VPL; k++) c[k] = __fmul_rn(rr[k], inv);
    const size_t o = (size_t)r * RS + col;
    if constexpr (MASKED)
    {
        if (mine) ppr_store_masked<KP, CT>(it.cout, a.rank, it.rank_mask, a.zero_mask, o, rr, c, col);
    }
    else if (mine)
        PprRow<CT, KP>::store(it.cout + o, c);
}

/* the next rows with edges, one per lane: id, end offset, seed index, 1 / out-degree */
struct PprWindow
{
    uint32_t row, end, seed;
    float inv;
};
template <class CT>
__device__ __forceinline__ PprWindow ppr_window(const PprArgs<CT> &a, uint32_t row)
{
    PprWindow w{row, 0xffffffffu, NO_SEED, 0.0f};
    if (row < a.V)
    {
        w.end = a.off[row + 1];
        w.seed = a.seed_idx[row];
        w.inv = a.inv_deg[row];
    }
    return w;
}

/* `next`: hands out the tiles after each warp's first (zero on entry) -- a
 * tile of one-edge rows takes several times as long as one of a hub's edges,
 * and dealt round robin the slowest warp held the others up by a third */
template <int KP, int RS, bool MASKED, class CT>
__device__ __forceinline__ void ppr_gather_tiles(const PprArgs<CT> &a, const PprIter<CT> &it, uint32_t ring,
                                                 uint32_t *next)
{
    typedef PprRow<CT, KP> R;
    constexpr uint32_t CH = R::CHUNK, D = R::DEPTH, OUT = R::OUT, F2S = R::F2S;
    const uint32_t lane = threadIdx.x & 31, half = lane >> 4;
    const uint32_t col = R::out_col(lane);
    const bool mine = R::keeps(lane);
    const uint32_t nw = gridDim.x * (blockDim.x >> 5);
    uint32_t tile = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    if (tile >= a.ntiles) return;
    /* positions count chunks: 32 bits hold them for any E */
    const uint32_t per = a.tile / CH, pmask = per - 1u;
    const uint32_t nchunks = (a.E - 1u) / CH + 1u;
    /* the chunk after c: in the same tile, or the first of the next one, which
     * lane 0 took from the counter when the current one began */
    uint32_t taken = 0, ntile = 0;
    auto take = [&]() {
        if (lane == 0) taken = nw + atomicAdd(next, 1u);
    };
    auto after = [&](uint32_t c) -> uint32_t {
        const uint32_t n = c + 1u;
        if (n & pmask) return n;
        ntile = __shfl_sync(0xffffffffu, taken, 0);
        return ntile * per;
    };
    take();
    auto ids_at = [&](uint32_t c) -> uint32_t {
        const uint32_t i = c * CH + lane;
        return (lane < CH && c < nchunks && i < a.E) ? ldg_stream(a.adj + i) : 0u;
    };
    /* ask for the rows of chunk c into landing slot `slot`; rows past E land
     * as zeros */
    const uint32_t sub = lane / R::LPR;
    const unsigned char *src0 = reinterpret_cast<const unsigned char *>(it.cin) + (lane % R::LPR) * 16;
    auto ask = [&](uint32_t c, uint32_t ids, uint32_t slot) {
        const uint32_t dst = ring + slot * R::STAGE + lane * 16;
        if (c + 1u < nchunks)
        {
#pragma unroll
            for (uint32_t i = 0; i < CH / R::RPI; i++)
            {
                const uint32_t u = __shfl_sync(0xffffffffu, ids, i * R::RPI + sub);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + i * 512u),
                             "l"(src0 + (uint64_t)u * (uint32_t)(RS * sizeof(CT))) : "memory");
            }
        }
        else if (c < nchunks)
        {
            const uint32_t n = a.E - c * CH;
#pragma unroll 1
            for (uint32_t i = 0; i < CH / R::RPI; i++)
            {
                const uint32_t r = i * R::RPI + sub, u = __shfl_sync(0xffffffffu, ids, r);
                if (r < n)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + i * 512u),
                                 "l"(src0 + (uint64_t)u * (uint32_t)(RS * sizeof(CT))) : "memory");
                else
                    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};\n" ::"r"(dst + i * 512u), "r"(0u) : "memory");
            }
        }
        cp_async_commit();
    };

    uint32_t c = tile * per;
    uint32_t ahead = c; /* the chunk whose rows are asked for next, its ids in idn */
    uint32_t idn = ids_at(ahead);
#pragma unroll
    for (uint32_t d = 0; d < D; d++)
    {
        const uint32_t n = after(ahead), ids = idn;
        idn = ids_at(n);
        ask(ahead, ids, d);
        ahead = n;
    }
    uint32_t s0 = a.seg0[tile];
    uint32_t seg = s0 & 0x7fffffffu, wb = seg;
    bool open = s0 >> 31;
    PprWindow cur = ppr_window(a, a.rows[wb + lane]), nxt = ppr_window(a, a.rows[wb + 32 + lane]);
    uint32_t row2 = a.rows[wb + 64 + lane];
    uint32_t seeded = __ballot_sync(0xffffffffu, cur.seed != NO_SEED);
    F2 acc[F2S];
#pragma unroll
    for (uint32_t k = 0; k < F2S; k++) acc[k] = F2{0.0f, 0.0f};

    /* the row's sum in the columns this lane keeps */
    auto total = [&](float *t) {
        if constexpr (R::VPL == 4)
        {
            const F2 give = half ? acc[0] : acc[1], keep = half ? acc[1] : acc[0];
            t[0] = __fadd_rn(keep.x, __shfl_xor_sync(0xffffffffu, give.x, 16));
            t[1] = __fadd_rn(keep.y, __shfl_xor_sync(0xffffffffu, give.y, 16));
        }
        else if constexpr (R::VPL == 2)
        {
            const float give = half ? acc[0].x : acc[0].y, keep = half ? acc[0].y : acc[0].x;
            t[0] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, 16));
        }
        else
            t[0] = __fadd_rn(acc[0].x, __shfl_xor_sync(0xffffffffu, acc[0].x, 16));
    };
    auto finish = [&]() {
        float t[OUT];
        total(t);
        const uint32_t k = seg - wb;
        if (open)
        {
            if (mine) store_f32<OUT>(a.head + (size_t)tile * KP + col, t);
            open = false;
        }
        else
        {
            uint32_t si = NO_SEED;
            if (seeded >> k & 1u) si = __shfl_sync(0xffffffffu, cur.seed, k);
            ppr_finish<KP, RS, MASKED, CT>(a, it, __shfl_sync(0xffffffffu, cur.row, k), t, si,
                                           __shfl_sync(0xffffffffu, cur.inv, k), col, mine);
        }
        seg++;
        if (k == 31u)
        {
            wb += 32;
            cur = nxt;
            seeded = __ballot_sync(0xffffffffu, cur.seed != NO_SEED);
            nxt = ppr_window(a, row2);
            row2 = a.rows[wb + 64 + lane];
        }
    };

    const uint32_t read0 = ring + half * R::BYTES + (lane & 15) * (R::VPL * (uint32_t)sizeof(CT));
    uint32_t slot = 0;
    for (;;)
    {
        /* row ends of the chunk: bit i = its edge i is the last of its row */
        const uint32_t b0 = cur.end - 1u - c * CH, b1 = nxt.end - 1u - c * CH;
        const uint32_t m = __reduce_or_sync(0xffffffffu, (cur.row < a.V && b0 < CH ? 1u << b0 : 0u) |
                                                             (nxt.row < a.V && b1 < CH ? 1u << b1 : 0u));
        asm volatile("cp.async.wait_group %0;\n" ::"n"((int)D - 1) : "memory");
        __syncwarp();
        const uint32_t at = read0 + slot * R::STAGE;
        constexpr uint32_t B = 8; /* edges per step: four pairs */
#pragma unroll 1
        for (uint32_t i0 = 0; i0 < CH; i0 += B)
        {
            F2 v[B / 2][F2S];
#pragma unroll
            for (uint32_t i = 0; i < B / 2; i++) R::read(at + (i0 + 2 * i) * R::BYTES, v[i]);
            const uint32_t mm = (m >> i0) & 0xffu;
            if (mm == 0u)
            {
#pragma unroll
                for (uint32_t i = 0; i < B / 2; i++)
#pragma unroll
                    for (uint32_t k = 0; k < F2S; k++) acc[k] = add2(acc[k], v[i][k]);
            }
            else
            {
#pragma unroll
                for (uint32_t i = 0; i < B / 2; i++)
                {
                    /* row ends after the even and the odd edge of the pair;
                     * selects, not branches, keep the half warps together
                     * (x + 0 is x: sums here are never -0) */
                    const uint32_t two = (mm >> (2 * i)) & 3u;
                    if (two & 1u)
                    {
#pragma unroll
                        for (uint32_t k = 0; k < F2S; k++)
                            acc[k] = add2(acc[k], half ? F2{0.0f, 0.0f} : v[i][k]);
                        finish();
#pragma unroll
                        for (uint32_t k = 0; k < F2S; k++) acc[k] = half ? v[i][k] : F2{0.0f, 0.0f};
                    }
                    else
#pragma unroll
                        for (uint32_t k = 0; k < F2S; k++) acc[k] = add2(acc[k], v[i][k]);
                    if (two & 2u)
                    {
                        finish();
#pragma unroll
                        for (uint32_t k = 0; k < F2S; k++) acc[k] = F2{0.0f, 0.0f};
                    }
                }
            }
        }
        __syncwarp(); /* every lane has read the slot that is asked for again */
        {
            const uint32_t n = after(ahead), ids = idn;
            idn = ids_at(n);
            ask(ahead, ids, slot);
            ahead = n;
        }
        slot = slot + 1 == D ? 0 : slot + 1;
        if (((c + 1u) & pmask) == 0u || c + 1u >= nchunks)
        {
            /* a row open at the tile's end leaves what the tile had of it
             * (edge E - 1 ends its row) */
            if (c + 1u < nchunks && !(m >> (CH - 1) & 1u))
            {
                float t[OUT];
                total(t);
                if (mine) store_f32<OUT>(a.tail + (size_t)tile * KP + col, t);
#pragma unroll
                for (uint32_t k = 0; k < F2S; k++) acc[k] = F2{0.0f, 0.0f};
            }
            if (c + 1u >= nchunks) break; /* the last tile may be short of a full one */
            tile = ntile; /* set when the chunks asked for reached it */
            if (tile >= a.ntiles) break;
            take();
            s0 = a.seg0[tile];
            seg = wb = s0 & 0x7fffffffu;
            open = s0 >> 31;
            cur = ppr_window(a, a.rows[wb + lane]);
            nxt = ppr_window(a, a.rows[wb + 32 + lane]);
            row2 = a.rows[wb + 64 + lane];
            seeded = __ballot_sync(0xffffffffu, cur.seed != NO_SEED);
            c = tile * per;
        }
        else
            c++;
    }
    cp_async_wait_all();
}

template <int KP, int RS, bool MASKED, class CT>
__global__ void __launch_bounds__(PPR_THREADS, PPR_CTAS) k_ppr_pull(PprArgs<CT> a, uint32_t *next)
{
    extern __shared__ __align__(1024) unsigned char gg_dyn[];
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(gg_dyn) + (threadIdx.x >> 5) * PprRow<CT, KP>::RING;
    ppr_gather_tiles<KP, RS, MASKED, CT>(a, PprIter<CT>{a.cin, a.cout, a.rank_mask}, ring, next);
}

/* finish the rows spanning tiles: the row that begins in tile t and is
 * still open at t's end sums tail[t], the tails of the tiles it crosses and
 * the head of the tile where it ends, in tile order; and, with `empty`, the
 * rows without in-edges (their sum is zero).  One warp per row, one row at a
 * time: four at once, or a function of its own, made the persistent kernel's
 * gather spill (R-MAT-20, K = 64 BF16, 7.3 -> 8.0 and 7.6 ms). */
template <int KP, int RS, bool MASKED, class CT>
__device__ __forceinline__ void ppr_fixup_tiles(const PprArgs<CT> &a, const PprIter<CT> &it, bool empty)
{
    typedef PprRow<CT, KP> R;
    constexpr uint32_t VPL = R::OUT, B = 16 / VPL; /* tails in flight per lane */
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t col = R::out_col(lane);
    const bool mine = R::keeps(lane);
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    /* the tiles are spread over all warps, at most 32 per warp and round; a
     * lane looks at one, with what its row's end needs, and the warp then
     * takes the spanning rows found */
    const uint32_t group = min(32u, (a.ntiles + nw - 1) / nw);
    for (uint32_t t0 = warp * group; t0 + 1 < a.ntiles; t0 += nw * group)
    {
        const uint32_t t = t0 + lane;
        uint32_t row = a.V, last = 0, seed = NO_SEED;
        float inv = 0.0f;
        if (lane < group && t + 1 < a.ntiles)
        {
            const uint32_t s = a.seg0[t + 1];
            if (s >> 31)
            {
                const uint32_t r = a.rows[s & 0x7fffffffu];
                if (a.off[r] / a.tile == t)
                {
                    row = r;
                    last = (a.off[r + 1] - 1u) / a.tile;
                    seed = a.seed_idx[r];
                    inv = a.inv_deg[r];
                }
            }
        }
        for (uint32_t todo = __ballot_sync(0xffffffffu, row < a.V); todo; todo &= todo - 1)
        {
            const int src = __ffs(todo) - 1;
            const uint32_t r = __shfl_sync(0xffffffffu, row, src), tt = t0 + src;
            const uint32_t t_last = __shfl_sync(0xffffffffu, last, src);
            float tot[VPL], h[VPL];
            load_f32<VPL>(a.tail + (size_t)tt * KP + col, tot);
            load_f32<VPL>(a.head + (size_t)t_last * KP + col, h);
            for (uint32_t m = tt + 1; m < t_last; m += B)
            {
                float v[B][VPL];
#pragma unroll
                for (uint32_t i = 0; i < B; i++)
                    if (m + i < t_last) load_f32<VPL>(a.tail + (size_t)(m + i) * KP + col, v[i]);
#pragma unroll
                for (uint32_t i = 0; i < B; i++)
                    if (m + i < t_last)
#pragma unroll
                        for (uint32_t k = 0; k < VPL; k++) tot[k] += v[i][k];
            }
#pragma unroll
            for (uint32_t k = 0; k < VPL; k++) tot[k] += h[k];
            ppr_finish<KP, RS, MASKED, CT>(a, it, r, tot, __shfl_sync(0xffffffffu, seed, src),
                                           __shfl_sync(0xffffffffu, inv, src), col, mine);
        }
    }
    if (!empty) return;
    for (uint64_t v0 = (uint64_t)warp * 32; v0 < a.V; v0 += (uint64_t)nw * 32)
    {
        const uint32_t v = (uint32_t)v0 + lane;
        bool none = false;
        uint32_t si = NO_SEED;
        float inv = 0.0f;
        if (v0 + lane < a.V && a.off[v] == a.off[v + 1])
        {
            none = true;
            si = a.seed_idx[v];
            inv = a.inv_deg[v];
        }
        for (uint32_t todo = __ballot_sync(0xffffffffu, none); todo; todo &= todo - 1)
        {
            const int src = __ffs(todo) - 1;
            float zero[VPL];
#pragma unroll
            for (uint32_t k = 0; k < VPL; k++) zero[k] = 0.0f;
            ppr_finish<KP, RS, MASKED, CT>(a, it, (uint32_t)v0 + src, zero, __shfl_sync(0xffffffffu, si, src),
                                   __shfl_sync(0xffffffffu, inv, src), col, mine);
        }
    }
}

/* `next` is the gather's tile counter, cleared for the next gather */
template <int KP, int RS, bool MASKED, class CT>
__global__ void __launch_bounds__(256) k_ppr_fixup(PprArgs<CT> a, uint32_t *next)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) *next = 0u;
    ppr_fixup_tiles<KP, RS, MASKED, CT>(a, PprIter<CT>{a.cin, a.cout, a.rank_mask}, true);
}

/* every iteration in one cooperative launch: gather, grid barrier, fix-up
 * of the spanning rows, grid barrier.  The control block (GG_BAR_BYTES,
 * zeroed before the launch) holds the barrier; a barrier wait that runs out
 * sets *err and the launch ends (gg_set_barrier_limit_us). */
template <class CT>
struct PprLoop
{
    CT *cb0, *cb1;
    uint32_t iterations;
    char *ctl;
    unsigned int *err;
    uint32_t *next; /* a zeroed tile counter per iteration */
    unsigned long long limit_ns;
};

template <int KP, class CT>
__global__ void __launch_bounds__(PPR_THREADS, PPR_CTAS) k_ppr_persist(const __grid_constant__ PprArgs<CT> a,
                                                        const __grid_constant__ PprLoop<CT> L)
{
    extern __shared__ __align__(1024) unsigned char gg_dyn[];
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(gg_dyn) + (threadIdx.x >> 5) * PprRow<CT, KP>::RING;
    unsigned int gen = 0;
    for (uint32_t i = 0; i < L.iterations; i++)
    {
        const PprIter<CT> it{(i & 1) ? L.cb1 : L.cb0, (i & 1) ? L.cb0 : L.cb1, i + 1 == L.iterations ? ~0ull : 0ull};
        const bool last = i + 1 == L.iterations; /* writes the ranks */
        if (last)
            ppr_gather_tiles<KP, KP, true, CT>(a, it, ring, L.next + i);
        else
            ppr_gather_tiles<KP, KP, false, CT>(a, it, ring, L.next + i);
        if (!grid_barrier(L.ctl, L.err, L.limit_ns, gen)) return;
        /* a row without in-edges keeps its contribution: both buffers hold it
         * after two iterations, and the last one writes the ranks */
        if (last)
            ppr_fixup_tiles<KP, KP, true, CT>(a, it, true);
        else
            ppr_fixup_tiles<KP, KP, false, CT>(a, it, i < 2);
        if (!last && !grid_barrier(L.ctl, L.err, L.limit_ns, gen)) return;
    }
}

/* dynamic shared memory of the gather kernels: the warps' landing space */
template <int KP, class CT> constexpr size_t ppr_smem() { return (size_t)PPR_WARPS * PprRow<CT, KP>::RING; }

/* allow a kernel its dynamic shared memory (once per kernel) */
gg_status ppr_allow(const void *kernel, size_t smem)
{
    GG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return GG_OK;
}

/* contributions of the seed vertices at iteration 0 (the rest is zero), and
 * their seed indices; rows of rs values, of which vectors in `fresh` are
 * written (all of them for gg_ppr; the newly admitted slots for the
 * server, whose other columns hold running vectors) */
/* with `inv`, also inv[v] = 1 / out-degree (correctly rounded), 0 without
 * out-edges */
template <class CT>
__global__ void k_ppr_seed_init(const uint32_t *__restrict__ seed_vertex, uint32_t nseeds,
                                const float *__restrict__ init, const uint32_t *__restrict__ outdeg, CT *cin,
                                uint32_t *seed_idx, uint32_t rs, unsigned long long fresh, uint32_t V, float *inv)
{
    if (inv)
        for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        {
            const uint32_t d = outdeg[v];
            inv[v] = d ? __frcp_rn(__uint2float_rn(d)) : 0.0f;
        }
    const uint64_t n = (uint64_t)nseeds * (rs / 2);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    {
        const uint32_t s = (uint32_t)(i / (rs / 2)), gl = (uint32_t)(i % (rs / 2));
        const uint32_t v = seed_vertex[s];
        if (gl == 0) seed_idx[v] = s;
        const uint32_t pair = (uint32_t)(fresh >> (2 * gl)) & 3u;
        if (!pair) continue;
        const uint32_t deg = outdeg[v];
        const float2 r = *reinterpret_cast<const float2 *>(init + (size_t)s * rs + 2 * gl);
        float c0 = 0.0f, c1 = 0.0f;
        if (deg)
        {
            const float fd = __uint2float_rn(deg);
            c0 = __fdiv_rn(r.x, fd);
            c1 = __fdiv_rn(r.y, fd);
        }
        CT *dst = cin + (size_t)v * rs + 2 * gl;
        /* only the fresh columns: the others belong to running vectors */
        if (pair & 1u) dst[0] = from_f32<CT>(c0);
        if (pair & 2u) dst[1] = from_f32<CT>(c1);
    }
}

/* inv[v] = 1 / out-degree (correctly rounded), 0 without out-edges */
__global__ void k_ppr_inv_deg(const uint32_t *__restrict__ outdeg, uint32_t V, float *inv)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
    {
        const uint32_t d = outdeg[v];
        inv[v] = d ? __frcp_rn(__uint2float_rn(d)) : 0.0f;
    }
}

gg_status ppr_inv_deg(gg_graph *g, cudaStream_t s, const float **out)
{
    void *inv;
    GG_CHECK(gg_work(g, 15, (size_t)g->V * 4 + 16, &inv));
    k_ppr_inv_deg<<<gg_sm_count() * 4, 256, 0, s>>>(g->out_deg, g->V, (float *)inv);
    GG_CUDA(cudaGetLastError());
    *out = (const float *)inv;
    return GG_OK;
}

/* persistent grid of a kernel with one warp per work item */
int occupancy_grid(const void *kernel, int threads, size_t smem, size_t warps)
{
    int bps = gg_occupancy(kernel, threads, smem);
    if (bps < 1) bps = 1;
    const size_t need = (warps + threads / 32 - 1) / (threads / 32), cap = (size_t)gg_sm_count() * bps;
    const size_t g = need < cap ? need : cap;
    return (int)(g < 1 ? 1 : g);
}

/* seg0 of the mapping for its PPR tile size */
gg_status ppr_tiles(gg_graph *g, cudaStream_t s, uint32_t *launches)
{
    const uint32_t tile = gg_ppr_tile(g);
    if (g->ppr_seg0 && g->ppr_tiles_items == tile) return GG_OK;
    if (g->ppr_seg0) gg_dev_free(g, g->ppr_seg0, (size_t)g->ppr_ntiles * 4);
    g->ppr_seg0 = nullptr;
    g->ppr_tiles_items = 0;
    GG_CHECK(gg_rows_tiles(g, s, tile, &g->ppr_seg0, &g->ppr_ntiles, launches));
    g->ppr_tiles_items = tile;
    return GG_OK;
}

/* tiles below 256 edges need a warp each (gg_ppr_tile) */
gg_status ppr_tiles_fit(uint32_t tile, uint32_t ntiles, int grid)
{
    if (tile < 256u && (uint64_t)grid * PPR_WARPS < ntiles)
        return gg_fail(GG_ERR_CUDA, "the batched gather has fewer resident warps than its tiles were made for");
    return GG_OK;
}

/* one gather / fix-up as a launch of its own */
template <int KP, int RS, class CT>
gg_status launch_pull(const PprArgs<CT> &a, uint32_t *next, cudaStream_t s)
{
    if (!a.ntiles) return GG_OK;
    constexpr size_t smem = ppr_smem<KP, CT>();
    const bool masked = (a.rank_mask | a.zero_mask) != 0ull;
    const void *fn = masked ? (const void *)k_ppr_pull<KP, RS, true, CT> : (const void *)k_ppr_pull<KP, RS, false, CT>;
    GG_CHECK(ppr_allow(fn, smem));
    void *args[] = {(void *)&a, &next};
    const int grid = occupancy_grid(fn, PPR_THREADS, smem, a.ntiles);
    GG_CHECK(ppr_tiles_fit(a.tile, a.ntiles, grid));
    GG_CUDA(cudaLaunchKernel(fn, dim3(grid), dim3(PPR_THREADS), args, smem, s));
    return GG_OK;
}
template <int KP, int RS, class CT>
gg_status launch_fixup(const PprArgs<CT> &a, uint32_t *next, cudaStream_t s)
{
    const bool masked = (a.rank_mask | a.zero_mask) != 0ull;
    const void *fn = masked ? (const void *)k_ppr_fixup<KP, RS, true, CT> : (const void *)k_ppr_fixup<KP, RS, false, CT>;
    void *args[] = {(void *)&a, &next};
    GG_CUDA(cudaLaunchKernel(fn, dim3(occupancy_grid(fn, 256, 0, ((size_t)a.V + 31) / 32)), dim3(256), args, 0, s));
    return GG_OK;
}

template <int KP, class CT>
gg_status run_ppr(gg_graph *g, const gg_ppr_params *p, uint32_t nseedv, const uint32_t *d_seedv, const float *d_init,
                  const float *d_tele, uint32_t *d_seed_idx, float *d_rank, cudaStream_t s, gg_ppr_result &res,
                  std::vector<cudaEvent_t> &evs, void **ctl_out)
{
    const uint32_t V = g->V;
    GG_CHECK(ppr_tiles(g, s, &res.launches));
    const uint32_t ntiles = g->ppr_ntiles;
    void *c0, *c1, *slots;
    GG_CHECK(gg_work(g, 16, (size_t)V * KP * sizeof(CT), &c0));
    GG_CHECK(gg_work(g, 17, (size_t)V * KP * sizeof(CT), &c1));
    GG_CHECK(gg_work(g, 18, ((size_t)ntiles * KP * 2 + 4) * sizeof(float), &slots));
    uint32_t *next = (uint32_t *)((float *)slots + (size_t)ntiles * KP * 2);
    void *inv;
    GG_CHECK(gg_work(g, 15, (size_t)V * 4 + 16, &inv));
    GG_CUDA(cudaMemsetAsync(c0, 0, (size_t)V * KP * sizeof(CT), s));
    GG_CUDA(cudaMemsetAsync(d_seed_idx, 0xff, (size_t)V * sizeof(uint32_t), s));
    k_ppr_seed_init<CT><<<gg_sm_count() * 4, 256, 0, s>>>(d_seedv, nseedv, d_init, g->out_deg, (CT *)c0, d_seed_idx,
                                                          KP, ~0ull, V, (float *)inv);
    res.launches++;

    PprArgs<CT> a;
    a.off = g->in_off; a.adj = g->in_adj; a.seed_idx = d_seed_idx;
    a.inv_deg = (const float *)inv;
    a.rows = g->rows_list; a.seg0 = g->ppr_seg0; a.ntiles = ntiles; a.V = V; a.E = g->E; a.tile = g->ppr_tiles_items;
    a.rank = d_rank; a.rank_mask = 0; a.zero_mask = 0;
    a.tele = d_tele; a.damp = p->damp;
    a.head = (float *)slots;
    a.tail = (float *)slots + (size_t)ntiles * KP;
    constexpr size_t smem = ppr_smem<KP, CT>();
    CT *cb[2] = {(CT *)c0, (CT *)c1};
    if (!p->profile)
    {
        /* all iterations in one cooperative launch: every block resident */
        const void *fn = (const void *)k_ppr_persist<KP, CT>;
        GG_CHECK(ppr_allow(fn, smem));
        const int per_sm = gg_occupancy(fn, PPR_THREADS, smem);
        if (per_sm < 1) return gg_fail(GG_ERR_CUDA, "k_ppr_persist cannot be resident");
        /* a warp per tile, or per 32 vertices (the rows without in-edges) */
        const int grid = occupancy_grid(fn, PPR_THREADS, smem, std::max<size_t>(ntiles, ((size_t)V + 31) / 32));
        GG_CHECK(ppr_tiles_fit(a.tile, ntiles, grid));
        void *ctl;
        const size_t ctl_bytes = GG_BAR_BYTES + (size_t)p->iterations * 4;
        GG_CHECK(gg_work(g, 30, ctl_bytes, &ctl));
        GG_CUDA(cudaMemsetAsync(ctl, 0, ctl_bytes, s));
        PprLoop<CT> L;
        L.cb0 = cb[0]; L.cb1 = cb[1]; L.iterations = p->iterations;
        L.ctl = (char *)ctl; L.err = (unsigned int *)ctl; L.limit_ns = gg_barrier_limit_ns();
        L.next = (uint32_t *)((char *)ctl + GG_BAR_BYTES);
        void *args[] = {&a, &L};
        GG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(PPR_THREADS), args, smem, s));
        res.launches++;
        res.gather_launches = p->iterations;
        res.persistent = 1;
        *ctl_out = ctl;
        GG_CUDA(cudaGetLastError());
        return GG_OK;
    }
    GG_CUDA(cudaMemsetAsync(next, 0, 4, s));
    for (uint32_t it = 0; it < p->iterations; it++)
    {
        a.cin = cb[it & 1];
        a.cout = cb[(it + 1) & 1];
        a.rank_mask = it + 1 == p->iterations ? ~0ull : 0ull;
        if (p->profile)
        {
            cudaEvent_t e;
            GG_CHECK(gg_event_at(g, (uint32_t)evs.size(), &e));
            GG_CUDA(cudaEventRecord(e, s));
            evs.push_back(e);
        }
        GG_CHECK((launch_pull<KP, KP, CT>(a, next, s)));
        if (p->profile)
        {
            cudaEvent_t e;
            GG_CHECK(gg_event_at(g, (uint32_t)evs.size(), &e));
            GG_CUDA(cudaEventRecord(e, s));
            evs.push_back(e);
        }
        GG_CHECK((launch_fixup<KP, KP, CT>(a, next, s)));
        res.launches += 2;
        res.gather_launches++;
    }
    GG_CUDA(cudaGetLastError());
    return GG_OK;
}

} // namespace

/* ---- one iteration on caller-held state (the server's continuous batch) ----- */

namespace {

template <int KP, class CT>
gg_status round_run(gg_graph *g, const gg_ppr_round_args &r, cudaStream_t s)
{
    const uint32_t ntiles = g->ppr_ntiles;
    PprArgs<CT> a;
    a.off = g->in_off; a.adj = g->in_adj; a.seed_idx = r.seed_idx;
    void *inv;
    GG_CHECK(gg_work(g, 15, (size_t)g->V * 4 + 16, &inv)); /* filled by gg_ppr_round_prepare */
    a.inv_deg = (const float *)inv;
    a.rows = g->rows_list; a.seg0 = g->ppr_seg0; a.ntiles = ntiles; a.V = g->V; a.E = g->E;
    a.tile = g->ppr_tiles_items;
    a.cin = (const CT *)r.cin; a.cout = (CT *)r.cout; a.rank = r.rank;
    a.rank_mask = r.rank_mask; a.zero_mask = r.zero_mask;
    a.tele = r.tele; a.damp = r.damp;
    a.head = r.slots;
    a.tail = r.slots + (size_t)ntiles * KP;
    uint32_t *next = (uint32_t *)(r.slots + (size_t)ntiles * 64 * 2); /* cleared by gg_ppr_round_prepare */
    GG_CHECK((launch_pull<KP, 64, CT>(a, next, s)));
    GG_CHECK((launch_fixup<KP, 64, CT>(a, next, s)));
    GG_CUDA(cudaGetLastError());
    return GG_OK;
}

} // namespace

/* edges per tile: the tuned size, or by the graph's.  A tile runs on one warp,
 * so a graph of few tiles per warp (3,040 resident) ends with the slowest:
 * 256 below four 512-edge tiles per warp (R-MAT-16, K = 64
 * BF16: 96 -> 78 us an iteration), 512 above (fewer rows
 * span tiles).  Down to 32 while every warp has one tile at most (K = 16 FP32, 20
 * iterations: 32K R-MAT edges 351 us, 320K 962 -> 722): the gather asks for rows a
 * few chunks ahead, past a next tile of so few only if there is none. */
uint32_t gg_ppr_tile(const gg_graph *g)
{
    const uint32_t warps = (uint32_t)(PPR_CTAS * PPR_WARPS) * (uint32_t)gg_sm_count();
    uint32_t tile = g->ppr_tile;
    if (tile)
    {
        /* a size from a file may be any: the gather needs a power of two, no less
         * than a chunk */
        uint32_t pow2 = 32u;
        while (pow2 <= tile / 2) pow2 *= 2;
        tile = pow2;
    }
    else
    {
        tile = g->E < 4u * 512u * warps ? 256u : 512u;
        while (tile > 32u && (uint64_t)(tile / 2) * warps >= g->E) tile /= 2;
    }
    /* below 256 only while every warp has one tile at most */
    if (tile < 256u && (uint64_t)tile * warps < g->E) tile = 256u;
    return tile;
}

gg_status gg_ppr_round_prepare(gg_graph *g, uint32_t rs, int bf16, void **cb0, void **cb1, float **slots,
                               cudaStream_t s)
{
    const uint32_t V = g->V;
    uint32_t launches = 0;
    GG_CHECK(ppr_tiles(g, s, &launches));
    const size_t cb = (size_t)V * rs * (bf16 ? 2 : 4);
    GG_CHECK(gg_work(g, 16, cb, cb0));
    GG_CHECK(gg_work(g, 17, cb, cb1));
    GG_CHECK(gg_work(g, 18, ((size_t)g->ppr_ntiles * rs * 2 + 4) * sizeof(float), (void **)slots));
    GG_CUDA(cudaMemsetAsync(*slots + (size_t)g->ppr_ntiles * rs * 2, 0, 4, s));
    GG_CUDA(cudaMemsetAsync(*cb0, 0, cb, s));
    GG_CUDA(cudaMemsetAsync(*cb1, 0, cb, s));
    const float *inv;
    GG_CHECK(ppr_inv_deg(g, s, &inv));
    return GG_OK;
}

gg_status gg_ppr_round_seed(gg_graph *g, uint32_t rs, int bf16, void *cin, const uint32_t *d_seedv, uint32_t nseedv,
                            const float *d_init, uint32_t *d_seed_idx, unsigned long long fresh, cudaStream_t s)
{
    if (!nseedv) return GG_OK;
    if (bf16)
        k_ppr_seed_init<__nv_bfloat16><<<gg_sm_count() * 2, 256, 0, s>>>(d_seedv, nseedv, d_init, g->out_deg,
                                                                         (__nv_bfloat16 *)cin, d_seed_idx, rs, fresh, 0, nullptr);
    else
        k_ppr_seed_init<float><<<gg_sm_count() * 2, 256, 0, s>>>(d_seedv, nseedv, d_init, g->out_deg, (float *)cin,
                                                                 d_seed_idx, rs, fresh, 0, nullptr);
    GG_CUDA(cudaGetLastError());
    return GG_OK;
}

gg_status gg_ppr_round(gg_graph *g, const gg_ppr_round_args &r, cudaStream_t s)
{
    if (r.bf16)
        return r.kp == 16 ? round_run<16, __nv_bfloat16>(g, r, s)
               : r.kp == 32 ? round_run<32, __nv_bfloat16>(g, r, s) : round_run<64, __nv_bfloat16>(g, r, s);
    return r.kp == 16 ? round_run<16, float>(g, r, s) : r.kp == 32 ? round_run<32, float>(g, r, s)
                                                                : round_run<64, float>(g, r, s);
}

extern "C" gg_status gg_ppr(gg_graph *g, const gg_ppr_params *p, const uint32_t *seed_off, const uint32_t *seeds,
                            float *ranks, gg_ppr_result *r, void *stream)
{
    GgRange range("gg_ppr");
    if (!g || !p || !seed_off) return gg_fail(GG_ERR_INVALID, "NULL argument");
    const uint32_t K = p->num_vectors;
    if (K < 1 || K > 64) return gg_fail(GG_ERR_INVALID, "num_vectors must be 1..64");
    if (p->iterations < 1) return gg_fail(GG_ERR_INVALID, "iterations must be at least 1");
    if (p->storage != GG_STORE_F32 && p->storage != GG_STORE_BF16)
        return gg_fail(GG_ERR_INVALID, "batched PageRank stores FP32 or BF16 contributions");
    if (!g->in_off || !g->out_deg) return gg_fail(GG_ERR_INVALID, "batched PageRank needs GG_MAP_IN");
    if (seed_off[0] != 0) return gg_fail(GG_ERR_INVALID, "seed_off[0] must be 0");
    for (uint32_t k = 0; k < K; k++)
        if (seed_off[k + 1] < seed_off[k]) return gg_fail(GG_ERR_INVALID, "seed_off must be non-decreasing");
    const uint32_t nseeds = seed_off[K];
    if (nseeds && !seeds) return gg_fail(GG_ERR_INVALID, "NULL seeds");
    const uint32_t V = g->V;
    for (uint32_t i = 0; i < nseeds; i++)
        if (seeds[i] >= V) return gg_fail(GG_ERR_INVALID, "seed vertex out of range");
    const uint32_t KP = K <= 16 ? 16 : (K <= 32 ? 32 : 64);
    cudaStream_t s = gg_stream(g, stream);
    gg_tune_lookup(g, s);
    gg_ppr_result res;
    memset(&res, 0, sizeof(res));
    res.padded_vectors = KP;

    /* seed vertices, each with its initial-rank and teleport rows */
    std::vector<uint32_t> verts;
    std::unordered_map<uint32_t, uint32_t> index;
    for (uint32_t i = 0; i < nseeds; i++)
        if (index.emplace(seeds[i], (uint32_t)verts.size()).second) verts.push_back(seeds[i]);
    const uint32_t nv = (uint32_t)verts.size();
    std::vector<double> share((size_t)nv * KP, 0.0);
    for (uint32_t k = 0; k < K; k++)
    {
        const uint32_t n = seed_off[k + 1] - seed_off[k];
        for (uint32_t i = seed_off[k]; i < seed_off[k + 1]; i++)
            share[(size_t)index[seeds[i]] * KP + k] += 1.0 / (double)n;
    }
    std::vector<float> tables((size_t)nv * KP * 2);
    for (size_t i = 0; i < share.size(); i++)
    {
        tables[i] = (float)share[i];
        tables[share.size() + i] = (float)((1.0 - (double)p->damp) * share[i]);
    }
    void *d_seedv = nullptr, *d_tab = nullptr, *d_idx, *d_rank;
    if (V > 0)
    {
        GG_CHECK(gg_work(g, 19, ((size_t)nv + 1) * 4, &d_seedv));
        GG_CHECK(gg_work(g, 20, (tables.size() + 4) * sizeof(float), &d_tab));
        GG_CHECK(gg_work(g, 21, (size_t)V * 4, &d_idx));
        GG_CHECK(gg_work(g, 22, (size_t)V * KP * sizeof(float), &d_rank));
        if (nv)
        {
            GG_CUDA(cudaMemcpyAsync(d_seedv, verts.data(), (size_t)nv * 4, cudaMemcpyHostToDevice, s));
            GG_CUDA(cudaMemcpyAsync(d_tab, tables.data(), tables.size() * sizeof(float), cudaMemcpyHostToDevice, s));
        }
        std::vector<cudaEvent_t> evs;
        void *ctl = nullptr;
        const float *d_init = (const float *)d_tab, *d_tele = (const float *)d_tab + (size_t)nv * KP;
        gg_status st;
#define GG_PPR_RUN(KPV, CTV)                                                                                          \
    run_ppr<KPV, CTV>(g, p, nv, (const uint32_t *)d_seedv, d_init, d_tele, (uint32_t *)d_idx, (float *)d_rank, s,     \
                      res, evs, &ctl)
        if (p->storage == GG_STORE_BF16)
            st = KP == 16 ? GG_PPR_RUN(16, __nv_bfloat16) : KP == 32 ? GG_PPR_RUN(32, __nv_bfloat16) : GG_PPR_RUN(64, __nv_bfloat16);
        else
            st = KP == 16 ? GG_PPR_RUN(16, float) : KP == 32 ? GG_PPR_RUN(32, float) : GG_PPR_RUN(64, float);
#undef GG_PPR_RUN
        if (st != GG_OK) return st;
        GG_CHECK(gg_wait(s)); /* bounded, before a copy to pageable memory */
        if (ranks)
            GG_CUDA(cudaMemcpy2DAsync(ranks, (size_t)K * sizeof(float), d_rank, (size_t)KP * sizeof(float),
                                      (size_t)K * sizeof(float), V, cudaMemcpyDeviceToHost, s));
        uint32_t *h_err = nullptr;
        if (ctl)
        {
            GG_CHECK(gg_pinned(g, 64, (void **)&h_err));
            GG_CUDA(cudaMemcpyAsync(h_err, ctl, 4, cudaMemcpyDeviceToHost, s));
        }
        GG_CHECK(gg_wait(s));
        if (h_err && *h_err) return gg_fail(GG_ERR_KERNEL, "batched PageRank grid barrier timed out");
        for (size_t i = 0; i + 1 < evs.size(); i += 2) res.gather_ms += gg_event_ms(evs[i], evs[i + 1]);
        g->ppr_ranks = (const float *)d_rank;
        g->ppr_stride = KP;
    }
    if (r) *r = res;
    return GG_OK;
}

extern "C" const float *gg_ppr_device_ranks(const gg_graph *g, uint32_t *stride)
{
    if (!g) return nullptr;
    if (stride) *stride = g->ppr_stride;
    return g->ppr_ranks;
}
