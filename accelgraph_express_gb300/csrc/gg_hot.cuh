/*
 * The pull gather through the hot-vertex table (hot.cu prepares the table
 * and the encoded ids).
 *
 * What bounds it.  A gather of 4-byte values at random ids costs one L1->L2
 * request per id, and an SM issues one request per clock: 297 G/s over the
 * chip, whatever the size of the array (measured with loads, and with
 * 4- and 16-byte asynchronous copies).  The id stream, the sums and the
 * arithmetic all fit beside that.  So the only way to go faster is to send
 * fewer requests: serve as many ids as possible from shared memory.
 *
 * Why the values go through 16-byte asynchronous copies.  A load keeps a
 * line of the L1 array for every request in flight; with more than ~160 KB
 * of the 256 KB array given to shared memory the same loads fall from 293 to
 * 142 G/s (111 at 64 MB).  cp.async.cg of the 16 bytes that hold the value
 * lands in shared memory without an L1 line and keeps 297 G/s with 225 KB of
 * shared memory.  That leaves 160 KB for the table (40K FP32 or 80K 16-bit
 * values; 8K / 16K fitted beside the staging of the merge-path engine) next
 * to 2 KB of landing slots per warp.
 *
 * Why the ids carry row ends.  The merge-path engine stages row offsets,
 * values and row sums, 3.6 KB per warp.  Here bit 30 of an id marks the last
 * edge of its row, so rows need no staging: a step is 128 edges, four
 * consecutive ones per lane; a lane sums its edges in order, a warp-shuffle
 * segmented scan carries open sums across lanes, and the count of row ends so
 * far indexes the list of the rows that have edges.  Tiles of 2048 edges are
 * dealt to the warps round robin; the sum of a row that spans tiles is added
 * atomically, every other row is stored.
 *
 * Per step a warp takes the values of step s, sends the gathers of step s + 1
 * (whose ids arrived during step s - 1), loads the ids of step s + 2 and then
 * reduces step s, so gathers are always in flight; 32 warps of one step each
 * are about 2,600 requests per SM, four times what its latency needs.
 *
 * Measured, per launch, against the merge-path engine with an 8K (FP32) / 16K
 * (16-bit) table: R-MAT-24 FP32 896 -> 631 us (425 G edges/s; L1 89% busy),
 * R-MAT-22 BF16 209 -> 150 us, weighted SpMV of 5M vertices and 80M edges
 * 330 -> 202 us.
 */
#pragma once

#include <type_traits>

#include "gg_device.cuh"

namespace gg {

constexpr uint32_t HOT_STEP = 128;      /* edges per warp step */
constexpr uint32_t HOT_RING = 32 * 4 * 16; /* landing slots of one warp, bytes */

__device__ __forceinline__ uint4 ldg_ids4(const uint32_t *p)
{
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

template <class T> __device__ __forceinline__ T lds_at(uint32_t a);
template <> __device__ __forceinline__ float lds_at<float>(uint32_t a)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
template <> __device__ __forceinline__ uint16_t lds_at<uint16_t>(uint32_t a)
{
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
    return v;
}
template <> __device__ __forceinline__ uint8_t lds_at<uint8_t>(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return (uint8_t)v;
}
template <> __device__ __forceinline__ uint32_t lds_at<uint32_t>(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
template <> __device__ __forceinline__ unsigned long long lds_at<unsigned long long>(uint32_t a)
{
    unsigned long long v;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    return v;
}
template <> __device__ __forceinline__ __nv_bfloat16 lds_at<__nv_bfloat16>(uint32_t a)
{
    return __ushort_as_bfloat16(lds_at<uint16_t>(a));
}
template <> __device__ __forceinline__ __half lds_at<__half>(uint32_t a)
{
    return __ushort_as_half(lds_at<uint16_t>(a));
}

/* a stored value as a term of the sums: FP32, or the integer itself */
template <class Acc, class CT>
__device__ __forceinline__ Acc hot_value(CT x)
{
    if constexpr (std::is_same<Acc, float>::value)
        return to_f32(x);
    else
        return (Acc)x;
}
/* FP32 additions are never contracted or reordered */
__device__ __forceinline__ float hot_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ uint32_t hot_add(uint32_t a, uint32_t b) { return a + b; }
__device__ __forceinline__ unsigned long long hot_add(unsigned long long a, unsigned long long b) { return a + b; }

/* four consecutive edge weights of a lane; the array is 16-byte aligned and
 * padded past E */
struct Weights4
{
    float v[4];
};
__device__ __forceinline__ Weights4 ldg_weights4(const float *w, uint32_t e)
{
    Weights4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]) : "l"(w + e));
    return r;
}
template <class T>
__device__ __forceinline__ Weights4 ldg_weights4(const T *w, uint32_t e)
{
    static_assert(sizeof(T) == 2, "16-bit weights");
    T h[4];
    uint2 u;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(u.x), "=r"(u.y) : "l"(w + e));
    *reinterpret_cast<uint2 *>(h) = u;
    Weights4 r;
#pragma unroll
    for (int i = 0; i < 4; i++) r.v[i] = to_f32(h[i]);
    return r;
}

/* What a launch reads: ids (encoded, E of them), the rows with edges in
 * order, each tile's first row end (bit 31: that row began in an earlier
 * tile), and the table, whose entry `cap` stays zero. */
struct HotArgs
{
    const uint32_t *ids, *row_of, *seg0;
    uint32_t E, ntiles, tile_edges; /* tile_edges: a power of two, at least HOT_STEP */
};

/* sums[r] += over the edges of row r of (weight *) x[id], for the rows with
 * edges; sums must be zero on entry for the rows that span tiles.  `ring`:
 * this warp's landing slots, `table` / `cap`: the filled table.  READY is
 * called once, before the first access to x or the table, and returns false
 * to leave without any.  Acc sums within a tile (at most GG_HOT_TILE_MAX
 * edges: 32 bits hold those of 16-bit integers), Sum across tiles. */
template <class CT, class Acc, class Sum, bool HAS_W, class Ready>
__device__ __forceinline__ void hot_pull_sums(uint32_t ring, uint32_t table, uint32_t cap, const HotArgs &a,
                                              uint32_t warp, uint32_t nwarps, const CT *__restrict__ x,
                                              const CT *__restrict__ w, Sum *sums, Ready ready)
{
    constexpr uint32_t PER = 16 / sizeof(CT); /* values per landing slot */
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    const uint32_t pad = GG_HOT_FLAG | cap; /* reads the table's zero */
    const uint4 pad4 = make_uint4(pad, pad, pad, pad);
    const uint32_t slot = ring + lane * 16;
    uint32_t tile = warp;
    const uint32_t tmask = a.tile_edges - 1u;
    uint32_t e = tile * a.tile_edges; /* below 2^32: E <= GG_HOT_MAX_E */
    const bool any = tile < a.ntiles;

    auto load = [&](uint32_t at) -> uint4 {
        const uint32_t i = at + 4 * lane;
        /* the ids past E up to the next multiple of four are pads too */
        return i < a.E ? ldg_ids4(a.ids + i) : pad4;
    };
    /* the step after the one at `at`: in the same tile, or in this warp's next */
    auto after = [&](uint32_t at) -> uint32_t {
        const uint32_t n = at + HOT_STEP;
        return (n & tmask) ? n : n + (nwarps - 1) * a.tile_edges;
    };
    auto send = [&](const uint4 &id) {
        const uint32_t u[4] = {id.x, id.y, id.z, id.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (!(u[i] & GG_HOT_FLAG))
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(slot + i * 512),
                             "l"(x + (u[i] & (GG_HOT_ID & ~(PER - 1)))) : "memory");
    };

    uint4 ida = pad4, idb = pad4;
    uint32_t s0 = 0, s1 = 0, e1 = 0;
    if (any)
    {
        ida = load(e);
        e1 = after(e);
        idb = e1 < a.E ? load(e1) : pad4;
        s0 = a.seg0[tile];
        if (tile + nwarps < a.ntiles) s1 = a.seg0[tile + nwarps];
    }
    if (!ready() || !any) return;
    uint32_t seg = s0 & 0x7fffffffu;
    bool open = s0 >> 31; /* the next row end closes a row begun in an earlier tile */
    uint32_t win = a.row_of[seg + lane];
    Acc carry = Acc(0);
    Weights4 wa = {};
    if constexpr (HAS_W)
        if (e + 4 * lane < a.E) wa = ldg_weights4(w, e + 4 * lane);
    send(ida);
    for (;;)
    {
        cp_async_wait_all();
        Acc v[4];
        uint32_t f[4];
        {
            const uint32_t u[4] = {ida.x, ida.y, ida.z, ida.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
            {
                const uint32_t at = (u[i] & GG_HOT_FLAG) ? table + (u[i] & GG_HOT_SLOT) * (uint32_t)sizeof(CT)
                                                         : slot + i * 512 + (u[i] & (PER - 1)) * (uint32_t)sizeof(CT);
                v[i] = hot_value<Acc>(lds_at<CT>(at));
                f[i] = (u[i] >> 30) & 1u;
            }
        }
        if constexpr (HAS_W)
        {
            /* past E the value is the table's zero; its weight is not read */
            const uint32_t left = a.E - e - 4 * lane; /* meaningful when e + 4 * lane < E */
            const bool in = e + 4 * lane < a.E;
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = in && (uint32_t)i < left ? __fmul_rn(wa.v[i], v[i]) : 0.0f;
        }
        ida = idb;
        const bool more = e1 < a.E;
        if (more)
        {
            send(ida);
            if constexpr (HAS_W)
                if (e1 + 4 * lane < a.E) wa = ldg_weights4(w, e1 + 4 * lane);
        }
        const uint32_t e2 = after(e1);
        idb = more && e2 < a.E ? load(e2) : pad4;

        /* row ends: ballots per edge position; this lane's rank among them */
        uint32_t m[4], pre = 0, cnt = 0;
#pragma unroll
        for (int i = 0; i < 4; i++)
        {
            m[i] = __ballot_sync(0xffffffffu, f[i] != 0u);
            pre += __popc(m[i] & lt);
            cnt += __popc(m[i]);
        }
        const uint32_t wcur = win, seg_at = seg;
        const bool tile_end = ((e + HOT_STEP) & tmask) == 0 || e + HOT_STEP >= a.E;
        /* the rows of the next step, which may open this warp's next tile */
        win = a.row_of[(tile_end ? s1 & 0x7fffffffu : seg + cnt) + lane];

        /* sums along the lane's edges; p[i] = sum since its last row end */
        Acc p[4];
        p[0] = v[0];
#pragma unroll
        for (int i = 1; i < 4; i++) p[i] = f[i - 1] ? v[i] : hot_add(p[i - 1], v[i]);
        Acc run = f[3] ? Acc(0) : p[3];
        const uint32_t ends = m[0] | m[1] | m[2] | m[3]; /* lanes with a row end */
        /* segmented inclusive scan of the lanes' open sums: lane `hd` is the
         * last one at or before this lane that has a row end */
        const uint32_t le = ends & (lt | (1u << lane));
        const int hd = le ? 31 - __clz((int)le) : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const Acc y = __shfl_up_sync(0xffffffffu, run, o);
            if ((int)lane - o >= hd) run = hot_add(run, y);
        }
        Acc cin = __shfl_up_sync(0xffffffffu, run, 1);
        if (lane == 0) cin = Acc(0);
        if (!(ends & lt)) cin = hot_add(cin, carry);
        const Acc last = __shfl_sync(0xffffffffu, run, 31);
        carry = ends ? last : hot_add(carry, last);

        uint32_t k = pre;
        bool first = true;
#pragma unroll
        for (int i = 0; i < 4; i++)
        {
            if (!m[i]) continue;
            uint32_t row = __shfl_sync(0xffffffffu, wcur, k & 31);
            if (f[i])
            {
                if (k >= 32) row = a.row_of[seg_at + k];
                const Acc s = first ? hot_add(p[i], cin) : p[i];
                if (k == 0 && open)
                    atomicAdd(&sums[row], (Sum)s);
                else
                    sums[row] = (Sum)s;
                first = false;
                k++;
            }
        }
        seg += cnt;
        if (cnt) open = false;
        if (tile_end)
        {
            /* a row still open at the tile's end adds what this tile had of
             * it; past E there is none (edge E - 1 ends its row) */
            const bool pend = e + HOT_STEP < a.E && !(m[3] >> 31);
            if (pend && lane == 0) atomicAdd(&sums[a.row_of[seg]], (Sum)carry);
            if (!more) break;
            tile += nwarps;
            s0 = s1;
            seg = s0 & 0x7fffffffu;
            open = s0 >> 31;
            carry = Acc(0);
            if (tile + nwarps < a.ntiles) s1 = a.seg0[tile + nwarps];
        }
        e = e1;
        e1 = e2;
    }
}

/* slots in use of the H there are, from the counts behind the hot list:
 * vertices above the threshold degree and at it */
__device__ __forceinline__ uint32_t hot_taken(const uint32_t *__restrict__ cnt, uint32_t H)
{
    return min(cnt[0] + cnt[1], H);
}

/* table[i] = x[hot_list[i]], zero from the slots in use to cap and in the pad entry, padded
 * to 16 bytes: the contiguous copy that every CTA of the gather reads (each
 * CTA gathering its own had cost 32K requests per SM and launch) */
template <class CT>
__device__ __forceinline__ void hot_table_fill(const CT *__restrict__ x, const uint32_t *__restrict__ hot_list,
                                               uint32_t H, uint32_t cap, CT *__restrict__ out)
{
    const uint32_t n = hot_taken(hot_list + GG_HOT_ENTRIES, H);
    const uint32_t all = cap + 16 / sizeof(CT);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < all; i += gridDim.x * blockDim.x)
        out[i] = i < n ? x[hot_list[i]] : CT(0);
}
template <class CT>
__host__ __device__ constexpr uint32_t hot_cap()
{
    return GG_HOT_TABLE_BYTES / sizeof(CT) < GG_HOT_ENTRIES ? (uint32_t)(GG_HOT_TABLE_BYTES / sizeof(CT))
                                                            : GG_HOT_ENTRIES;
}
template <class CT>
__host__ __device__ constexpr uint32_t hot_table_bytes()
{
    return hot_cap<CT>() * (uint32_t)sizeof(CT) + 16;
}
/* dynamic shared memory of a gather of `warps` warps: table, landing slots */
template <class CT>
__host__ __device__ constexpr size_t hot_smem_bytes(uint32_t warps)
{
    return (size_t)hot_table_bytes<CT>() + (size_t)warps * HOT_RING;
}

/* the table into shared memory: `bytes` of the contiguous copy in 16-byte
 * pieces, by the whole block */
__device__ __forceinline__ void hot_table_load(uint32_t table, const void *src, uint32_t bytes)
{
    for (uint32_t i = threadIdx.x * 16; i < bytes; i += blockDim.x * 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(table + i),
                     "l"((const unsigned char *)src + i) : "memory");
    cp_async_wait_all();
    __syncthreads();
}

} // namespace gg
