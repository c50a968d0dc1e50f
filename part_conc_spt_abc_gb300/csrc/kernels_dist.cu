/*
 * kernels_dist.cu -- fused 2-D prefix sum + cumulative distance.
 *
 * Follows cusim::K_distance (src/gpu/cusim/kernel-distance.inl:81-241), which
 * runs one 32x32 block per proposal over the whole R x B histogram twice
 * (row scans, then column scans accumulating (cum - ref)^2) and zeroes the
 * histogram for reuse.  Here one CTA per proposal streams the histogram in
 * strips of 32 DE columns through a shared-memory tile:
 *   k_distance_strip (up to 1664 rows, 512 threads): the whole strip height
 *            sits in a swizzled tile filled by TMA box copies; phase A
 *            builds its 2-D prefix sums (zeros written back by box stores,
 *            per-lane column and row passes, per-row carry across strips
 *            in shared memory), phase B reads columns c0+2w, c0+2w+1 for
 *            logical warps 2w, 2w+1 while lane l accumulates
 *            (float(cum) - float(ref))^2 for rows l, l+32, ..., the observed
 *            cumulative histogram read from its column-major copy (coalesced);
 *   k_distance_cluster (histograms of up to 256 bins, where they are tall
 *            or each has a cluster): a thread-block cluster per histogram,
 *            one strip per CTA, the row carries and per-lane sums
 *            exchanged through distributed shared memory;
 *   k_distance_rows (up to 1024 bins, many or wide histograms): a warp per
 *            128 columns, the rows stream past it;
 *   k_distance (taller histograms, 1024 threads): the same in blocks of
 *            256 rows (tile row pitch 33 words), with the column carry in a
 *            register.
 * Warp w / lane l therefore own exactly the columns and rows they own in the
 * reference launch, so the per-lane sums, the shfl_down trees of reduce0
 * (:69-78) and the final per-warp tree reproduce the reference's float
 * result bit for bit (each operation is an explicit round-to-nearest
 * intrinsic, as in a build without FMA contraction).  The exact integer sum
 * of squares and a double-precision sum are accumulated alongside on request.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <map>
#include <mutex>
#include <tuple>

#include "pcs_common.h"
#include "pcs_kernels.h"

namespace pcs {

namespace {

const uint32_t kPad = 33; /* shared tile row pitch: conflict-free column reads */

__device__ __forceinline__ uint32_t warp_scan_(uint32_t v, uint32_t lane)
{
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        uint32_t t = __shfl_up_sync(0xFFFFFFFFu, v, d);
        if (lane >= d) v += t;
    }
    return v;
}

__device__ __forceinline__ float reduce0_(float v)
{
    v = __fadd_rn(v, __shfl_down_sync(0xFFFFFFFFu, v, 16));
    v = __fadd_rn(v, __shfl_down_sync(0xFFFFFFFFu, v, 8));
    v = __fadd_rn(v, __shfl_down_sync(0xFFFFFFFFu, v, 4));
    v = __fadd_rn(v, __shfl_down_sync(0xFFFFFFFFu, v, 2));
    v = __fadd_rn(v, __shfl_down_sync(0xFFFFFFFFu, v, 1));
    return v;
}

__device__ __forceinline__ double reduce0_(double v)
{
    v = __dadd_rn(v, __shfl_down_sync(0xFFFFFFFFu, v, 16));
    v = __dadd_rn(v, __shfl_down_sync(0xFFFFFFFFu, v, 8));
    v = __dadd_rn(v, __shfl_down_sync(0xFFFFFFFFu, v, 4));
    v = __dadd_rn(v, __shfl_down_sync(0xFFFFFFFFu, v, 2));
    v = __dadd_rn(v, __shfl_down_sync(0xFFFFFFFFu, v, 1));
    return v;
}

/* what the row kernel leaves as the distance of a histogram that the kernel
 * launched after it shall take: a quiet NaN that no sum of squares is */
const uint32_t kRedo = 0x7FC5EED0u;

__device__ __forceinline__ void add128_(uint64_t& hi, uint64_t& lo, uint64_t bhi, uint64_t blo)
{
    uint64_t n = lo + blo;
    hi += bhi + (n < lo ? 1u : 0u);
    lo = n;
}

} // namespace

template <bool F64>
__global__ void __launch_bounds__(1024, 1) k_distance(DistArgs a, uint32_t redo)
{
    extern __shared__ uint32_t s_mem[];
    uint32_t* carry = s_mem;            /* [max_rows] */
    uint32_t* T = s_mem + a.max_rows;   /* [kDistRowBlock][kPad] */
    __shared__ float s_tot[32];
    __shared__ double s_tot64[32];
    __shared__ uint64_t s_hi[32], s_lo[32];

    const uint32_t tid = threadIdx.x;
    const uint32_t w = tid >> 5, l = tid & 31u;
    const uint32_t M = *a.n_props;

    for (uint32_t p = blockIdx.x; p < M; p += gridDim.x) {
        if (redo && __float_as_uint(a.dist_f32[p]) != kRedo) continue; /* the row kernel's */
        const uint32_t job = a.props[p].job;
        const uint64_t hoff = a.props[p].hist_off;
        const uint32_t R = a.jobs[job].R, B = a.jobs[job].B;
        const uint32_t* refT = a.jobs[job].ref_sat_t;
        uint32_t* hist = a.hist + hoff;
        uint32_t* cum = a.cum_out ? a.cum_out + hoff : nullptr;
        if (R > a.max_rows) {
            if (tid == 0) {
                atomicOr(a.err, PCS_ERRBIT_ROWS);
                a.dist_f32[p] = __int_as_float(0x7fc00000);
            }
            continue;
        }
        for (uint32_t r = tid; r < R; r += blockDim.x) carry[r] = 0u;
        __syncthreads();

        float acc = 0.0f;
        double acc64 = 0.0;
        uint64_t shi = 0, slo = 0;
        for (uint32_t c0 = 0; c0 < B; c0 += 32u) {
            const uint32_t col = c0 + w;
            uint32_t colcarry = 0u;
            float a2 = 0.0f;
            double a2d = 0.0;
            for (uint32_t r0 = 0; r0 < R; r0 += kDistRowBlock) {
                const uint32_t rows = min(kDistRowBlock, R - r0);
                /* phase A: prefix along DE within each row of the strip */
                for (uint32_t rr = w; rr < rows; rr += 32u) {
                    const uint32_t r = r0 + rr;
                    const uint32_t c = c0 + l;
                    uint32_t v = 0u;
                    if (c < B) {
                        uint32_t* h = hist + (uint64_t)r * B + c;
                        v = *h;
                        *h = 0u;
                    }
                    const uint32_t cr = carry[r];
                    const uint32_t s = warp_scan_(v, l) + cr;
                    T[rr * kPad + l] = s;
                    __syncwarp();
                    if (l == 31u) carry[r] = s;
                }
                __syncthreads();
                /* phase B: prefix along K down column c0 + w, distance terms */
                if (col < B) {
                    for (uint32_t rr0 = 0; rr0 < rows; rr0 += 32u) {
                        const uint32_t rr = rr0 + l;
                        const bool valid = rr < rows;
                        const uint32_t v = valid ? T[rr * kPad + w] : 0u;
                        const uint32_t s = warp_scan_(v, l) + colcarry;
                        colcarry = __shfl_sync(0xFFFFFFFFu, s, 31);
                        if (valid) {
                            const uint32_t r = r0 + rr;
                            const uint32_t ref = __ldg(refT + pcs_sat_t_index(r, col, R, B));
                            const float dd = __fsub_rn(__uint2float_rn(s), __uint2float_rn(ref));
                            a2 = __fadd_rn(a2, __fmul_rn(dd, dd));
                            if (F64) {
                                const double d64 = __dsub_rn((double)s, (double)ref);
                                a2d = __dadd_rn(a2d, __dmul_rn(d64, d64));
                            }
                            const uint64_t ad = (s >= ref) ? (uint64_t)(s - ref) : (uint64_t)(ref - s);
                            add128_(shi, slo, 0u, ad * ad);
                            if (cum) cum[(uint64_t)r * B + col] = s;
                        }
                    }
                }
                __syncthreads();
            }
            if (col < B) {
                acc = __fadd_rn(acc, a2);
                if (F64) acc64 = __dadd_rn(acc64, a2d);
            }
        }

        /* reduce0 per warp, then over the 32 warp totals (kernel-distance.inl:210-229) */
        const float wsum = reduce0_(acc);
        double wsum64 = 0.0;
        if (F64) wsum64 = reduce0_(acc64);
        for (uint32_t d = 16; d >= 1; d >>= 1) {
            uint64_t ohi = __shfl_down_sync(0xFFFFFFFFu, shi, d);
            uint64_t olo = __shfl_down_sync(0xFFFFFFFFu, slo, d);
            if (l + d < 32u) add128_(shi, slo, ohi, olo);
        }
        if (l == 0) {
            s_tot[w] = wsum;
            s_tot64[w] = wsum64;
            s_hi[w] = shi;
            s_lo[w] = slo;
        }
        __syncthreads();
        if (w == 0) {
            const float fin = reduce0_(s_tot[l]);
            double fin64 = 0.0;
            if (F64) fin64 = reduce0_(s_tot64[l]);
            uint64_t thi = s_hi[l], tlo = s_lo[l];
            for (uint32_t d = 16; d >= 1; d >>= 1) {
                uint64_t ohi = __shfl_down_sync(0xFFFFFFFFu, thi, d);
                uint64_t olo = __shfl_down_sync(0xFFFFFFFFu, tlo, d);
                if (l + d < 32u) add128_(thi, tlo, ohi, olo);
            }
            if (l == 0) {
                a.dist_f32[p] = fin;
                if (F64 && a.dist_f64) a.dist_f64[p] = fin64;
                if (a.ssd) {
                    a.ssd[2 * (uint64_t)p] = thi;
                    a.ssd[2 * (uint64_t)p + 1] = tlo;
                }
            }
        }
        __syncthreads();
    }
}

/* Strip kernel: 16 warps, full-height strips of 32 DE columns, a persistent
 * CTA walking the (proposal, strip) sequence blockIdx.x, blockIdx.x + grid,
 * ... strip by strip.
 *
 * Tile: rows of 32 cells (128 bytes) whose 16-byte chunks are permuted by
 * XOR with (row mod 8) -- the TMA 128-byte swizzle -- so row-wise 128-bit
 * accesses by lanes on consecutive rows, and column-wise accesses, are free
 * of bank conflicts; 1024-byte aligned; rows up to the next multiple of 32.
 * Copy: with a tensor map for the job (B x R x histograms, boxes of 32 x 32
 * cells), one thread issues ceil(R/32) box copies (cp.async.bulk.tensor, the
 * TMA unit) completing on the tile's mbarrier; rows past R and columns past
 * B are outside the tensor and arrive as zeros.  Without one (B not a
 * multiple of 4, R or B below 32, callers without maps), every lane copies
 * its cells with 4-byte cp.async into the swizzled positions, zero-filling
 * past R and B.  Every thread arrives on the tile's mbarrier once per fill,
 * so a waiter passes only when all copies of the strip have landed; the
 * wait is bounded (error bit 0x80 and a clean exit when it runs out).  With
 * two tiles (db) the copies of the next strip -- or of the next proposal's
 * first strip -- are issued after the current strip's first barrier (every
 * warp is then past the strip before, whose tile they fill) and are in
 * flight while the current strip is computed: two CTA barriers per strip.
 * With one tile (tall histograms) the copies of a strip are issued together
 * after a third barrier.
 * Rows are split into 16 warp segments of a multiple of 8 rows (the
 * segments reach the next multiple of 8 past R; those rows hold zeros), so
 * a lane's swizzled column offset within each group of 8 rows is fixed.
 * Phase A1: lane l runs down column c0+l of its warp's segment (column
 * prefix within the segment, in place) and keeps the segment's column total;
 * the strip is zeroed in the histogram, as K_distance does, by box stores
 * of a zero box (one thread), or by the lanes cell by cell without a map.
 * Phase A2: lane l adds the totals of the segments above (the column carry
 * into the segment) and a warp scan turns the 32 carries into their prefix
 * across the strip; lane j then runs across row rb+j from the row's carry
 * of the strips to its left (128-bit shared loads and stores), adding the
 * scanned column carry: the tile holds the 2-D prefix sums.
 * Phase B: warp w reads columns c0+2w and c0+2w+1 -- logical warps 2w and
 * 2w+1 of the reference's 32x32 launch -- with one 8-byte shared load per
 * row, and the observed cumulative histogram of the same two columns with
 * one coalesced 8-byte load per row (pair-interleaved copy), so every lane
 * keeps the reference's per-lane sums in two accumulators.  When every
 * cumulative count of the strip and of the observed histogram is below
 * 2^22 (the largest is the last row's last cell: prefix sums of counts
 * are monotone), float(s) - float(o) is the exact integer s - o, and it is
 * formed as the float whose bits are 0x4B400000 + s - o (1.5 * 2^23 + s - o,
 * exact in [2^23, 2^24)) minus 1.5 * 2^23: the same value the reference's
 * two conversions and subtraction give, in two instructions.
 * F64: also the distance accumulated in double, SSD: the exact integer sum of
 * squares (128-bit).  Below 2^22 a lane's squares of a strip (at most 52 rows)
 * sum to less than 2^50, so every partial sum of the reference's double chain
 * is that integer exactly: one 32 x 32 + 64 bit multiply-add per cell and one
 * conversion per strip give the same double.  GB300's FP64 rate is a small
 * fraction of its FP32 rate: three FP64 operations and two conversions per
 * cell set the pace before (a short round of 201 x 1000: 398 -> 136 us;
 * 16 of 1001 x 256 with both sums and the prefix sums: 433 -> 114 us).
 * The standalone calls that ask for these take any counts, also an observed
 * array that falls somewhere or prefix sums that wrap: the lane looks at all
 * it has read and takes the conversions after all where some count is 2^22 or
 * more.  (Calls for the float alone trust the last cells.) */
const uint32_t kStripThreads = 512;
const uint32_t kBox = 32;                     /* rows and columns of a tensor-map box */
const uint32_t kBoxBytes = kBox * kBox * 4u;  /* 4096 */
const uint32_t kMbarWaitLimit = 1u << 22;     /* try_wait rounds before a wait is given up */
const uint32_t kExactBelow = 1u << 22;        /* cumulative counts below this take the integer difference */

__host__ __device__ __forceinline__ uint32_t strip_cap_rows(uint32_t max_rows) { return (max_rows + 31u) & ~31u; }

__device__ __forceinline__ uint32_t round8_(uint32_t x) { return (x + 7u) & ~7u; }

/* word of (row r, column c) in a swizzled strip tile */
__device__ __forceinline__ uint32_t sw_(uint32_t r, uint32_t c)
{
    return (r << 5) | ((((c >> 2) ^ (r & 7u)) << 2) | (c & 3u));
}

__device__ __forceinline__ uint32_t smem_u32_(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init_(uint64_t* m, uint32_t count)
{
    asm volatile("mbarrier.init.shared.b64 [%0], %1;\n" ::"r"(smem_u32_(m)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_init_fence_() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive_expect_tx_(uint64_t* m, uint32_t bytes)
{
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}\n" ::"r"(smem_u32_(m)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait_(uint64_t* m, uint32_t parity)
{
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(done)
                 : "r"(smem_u32_(m)), "r"(parity)
                 : "memory");
    return done != 0u;
}

/* bounded wait for a phase of the mbarrier */
__device__ __forceinline__ bool mbar_wait_(uint64_t* m, uint32_t parity)
{
    for (uint32_t it = 0; it < kMbarWaitLimit; ++it)
        if (mbar_try_wait_(m, parity)) return true;
    return false;
}

/* the tensor map as written through global memory, for this thread's box copies */
__device__ __forceinline__ void tmap_acquire_(const TmapDev* map)
{
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" ::"l"(map) : "memory");
}

/* box (x, y, z) of a 3-D tensor map -> shared memory, completing on an mbarrier */
__device__ __forceinline__ void tma_load_3d_(uint32_t* dst, const TmapDev* map, uint32_t x, uint32_t y, uint32_t z,
                                             uint64_t* m)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
            smem_u32_(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32_(m))
        : "memory");
}

/* shared memory -> box (x, y, z) of a 3-D tensor map (cells outside the tensor are dropped) */
__device__ __forceinline__ void tma_store_3d_(const TmapDev* map, uint32_t x, uint32_t y, uint32_t z, const uint32_t* src)
{
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];\n" ::"l"(map),
                 "r"(x), "r"(y), "r"(z), "r"(smem_u32_(src))
                 : "memory");
}

__device__ __forceinline__ void bulk_commit_() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }

/* this thread's box stores have completed */
__device__ __forceinline__ void bulk_wait_all_() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }

/* orders this thread's earlier generic shared-memory accesses before later
 * async-proxy (tensor copy) accesses to the same memory */
__device__ __forceinline__ void fence_proxy_async_() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

__device__ __forceinline__ void cp_async4_(uint32_t* dst, const uint32_t* src, bool valid)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = valid ? 4 : 0; /* 0: the destination is zero-filled, src is not read */
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}

__device__ __forceinline__ void cp_async_commit_() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait_() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

/* thread-block cluster: this CTA's rank, the cluster's index and count */
__device__ __forceinline__ uint32_t cluster_rank_()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t cluster_id_()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%clusterid.x;\n" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t cluster_count_()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%nclusterid.x;\n" : "=r"(r));
    return r;
}

/* every thread of every CTA of the cluster; shared-memory writes before it
 * are visible to shared::cluster reads after it */
__device__ __forceinline__ void cluster_sync_()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

/* the word at `p` (this CTA's shared memory) in the shared memory of the
 * cluster's CTA `rank` */
__device__ __forceinline__ uint32_t ld_cluster_(const void* p, uint32_t rank)
{
    uint32_t ra, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(smem_u32_(p)), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v) : "r"(ra) : "memory");
    return v;
}

/* warp w's segment of rows: [rb, re), multiples of 8, up to round8(R) */
struct Seg {
    uint32_t rb, re;
};

__device__ __forceinline__ Seg seg_(uint32_t R, uint32_t w)
{
    const uint32_t R8 = round8_(R);
    const uint32_t n = round8_((R8 + 15u) / 16u);
    Seg s;
    s.rb = min(R8, w * n);
    s.re = min(R8, s.rb + n);
    return s;
}

/* proposal p's tensor map and its index along the map, or null (cell-by-cell copies) */
__device__ __forceinline__ const TmapDev* prop_tmap_(const DistArgs& a, uint32_t p, uint32_t job, uint32_t& z)
{
    z = 0u;
    if (!a.tmaps) return nullptr;
    const uint32_t depth = a.jobs[job].tmap_depth;
    z = a.props[p].hist_z;
    return (depth != 0u && z < depth) ? a.tmaps + job : nullptr;
}

/* This thread's part of filling tile T with strip c0 of proposal p, and its
 * one arrival on the tile's mbarrier. */
__device__ __forceinline__ void strip_fill_(const DistArgs& a, uint32_t p, uint32_t c0, uint32_t* T, uint32_t tid,
                                            uint64_t* mbar)
{
    const uint32_t job = a.props[p].job;
    const uint32_t R = a.jobs[job].R, B = a.jobs[job].B;
    if (R > a.max_rows) {
        mbar_arrive_expect_tx_(mbar, 0u);
        return;
    }
    uint32_t z;
    const TmapDev* map = prop_tmap_(a, p, job, z);
    if (map) {
        if (tid == 0u) {
            const uint32_t nbox = (R + kBox - 1u) / kBox;
            tmap_acquire_(map);
            mbar_arrive_expect_tx_(mbar, nbox * kBoxBytes);
            for (uint32_t b = 0; b < nbox; ++b) tma_load_3d_(T + b * kBox * 32u, map, c0, b * kBox, z, mbar);
        } else {
            mbar_arrive_expect_tx_(mbar, 0u);
        }
        return;
    }
    mbar_arrive_expect_tx_(mbar, 0u);
    const uint32_t w = tid >> 5, l = tid & 31u;
    const Seg sg = seg_(R, w);
    const uint32_t* hist = a.hist + a.props[p].hist_off;
    const uint32_t c = c0 + l, lc = l >> 2, lo = l & 3u;
    for (uint32_t r8 = sg.rb; r8 < sg.re; r8 += 8u)
#pragma unroll
        for (uint32_t k = 0; k < 8u; ++k) {
            const uint32_t r = r8 + k;
            const bool v = r < R && c < B;
            cp_async4_(T + (r << 5) + (((lc ^ k) << 2) | lo), v ? hist + (uint64_t)r * B + c : hist, v);
        }
}

/* one distance term, general form: the reference's conversions, and on
 * request the FP64 and exact integer sums */
template <bool F64, bool SSD>
__device__ __forceinline__ void term_(uint32_t s, uint32_t o, float& a2, double& a2d, uint64_t& shi,
                                      uint64_t& slo)
{
    const float dd = __fsub_rn(__uint2float_rn(s), __uint2float_rn(o));
    a2 = __fadd_rn(a2, __fmul_rn(dd, dd));
    if (SSD) {
        const uint64_t ad = (s >= o) ? (uint64_t)(s - o) : (uint64_t)(o - s);
        add128_(shi, slo, 0u, ad * ad);
    }
    if (F64) {
        const double d64 = __dsub_rn((double)s, (double)o);
        a2d = __dadd_rn(a2d, __dmul_rn(d64, d64));
    }
}

/* float(s) - float(o) for s, o < 2^22 (exact integer difference) */
__device__ __forceinline__ float exact_diff_(uint32_t s, uint32_t o)
{
    return __fsub_rn(__uint_as_float(0x4B400000u + s - o), 12582912.0f);
}

/* (s - o)^2 for s, o < 2^22: below 2^44 */
__device__ __forceinline__ uint64_t square_(uint32_t s, uint32_t o)
{
    const int32_t d = (int32_t)(s - o);
    return (uint64_t)((int64_t)d * d);
}

/* Cluster mode (k_distance_cluster), for launches where walking each
 * histogram's strips one after another in one CTA leaves SMs idle or takes
 * long: few histograms, or tall ones.  A cluster of `cl` CTAs takes one
 * histogram at a time, CTA k its strip k (columns
 * 32k..32k+31; cl is at least the strips of every job).  Each CTA builds
 * its strip's 2-D prefix sums as if the strip stood alone (row carry 0) and
 * publishes the last column, P_k(r) = the cells of rows <= r in the strip;
 * after a cluster barrier CTA k's row carry is sum_{j<k} P_j(r), read from
 * the other CTAs' shared memory (integers, so the prefix sums are the strip
 * walk's exactly).  Each CTA then forms its strip's per-lane sums for
 * logical warps 2w, 2w+1 as the strip walk does and publishes them; after
 * the next barrier CTA 0 adds each (logical warp, lane)'s strip sums in
 * strip order -- the strip walk's per-lane accumulation, operation for
 * operation -- and reduces them with the same trees: the same float, bit
 * for bit.  One barrier per histogram: P and the per-lane sums alternate
 * between two buffers, and CTA 0 reduces histogram i while the cluster
 * computes histogram i + 1.  The next histogram's strip is copied in while
 * the current one is computed (two tiles), or, with one tile (tall
 * histograms), as soon as phase B has read it.  A copy wait that runs out ends
 * the loop on every CTA of the cluster together (each reads all CTAs' flags
 * after the barrier), so no CTA is left waiting at a cluster barrier.
 * With F64 and SSD each CTA also publishes its strip's per-lane double sums
 * and its warps' exact sums, as the strip kernel forms them, and CTA 0 adds
 * them likewise; the prefix sums leave with the row carry added.  (16 of 1001
 * x 256 with all of these: strip by strip 114 us, here 46.) */
__device__ __forceinline__ void cluster_fill_(const DistArgs& a, uint32_t p, uint32_t k, uint32_t cl, uint32_t* T,
                                              uint32_t tid, uint64_t* mbar)
{
    const uint32_t ns = (a.jobs[a.props[p].job].B + 31u) / 32u;
    if (k < ns && ns <= cl) strip_fill_(a, p, 32u * k, T, tid, mbar);
    else mbar_arrive_expect_tx_(mbar, 0u);
}

/* the double at `p` (this CTA's shared memory) in the cluster's CTA `rank` */
__device__ __forceinline__ double ld_cluster_f64_(const void* p, uint32_t rank)
{
    uint32_t ra;
    double v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(smem_u32_(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f64 %0, [%1];\n" : "=d"(v) : "r"(ra) : "memory");
    return v;
}

/* what a CTA publishes of its strip: per-lane sums, and with SSD each warp's
 * exact sum of squares */
struct ClusterSums {
    float* f;       /* [32][32] */
    double* d;      /* [32][32] with F64 */
    uint64_t* sq;   /* [16] (hi, lo) with SSD */
    /* the one of two that histogram number `it` of the cluster uses */
    __device__ __forceinline__ ClusterSums of(uint32_t it) const
    {
        const uint32_t b = it & 1u;
        return {f + b * 1024u, d + b * 1024u, sq + b * (kStripThreads / 16u)};
    }
};

/* CTA 0: histogram p's distance from every strip's per-lane sums */
template <bool F64, bool SSD>
__device__ __forceinline__ void cluster_reduce_(const DistArgs& a, uint32_t p, uint32_t cl, const ClusterSums& part,
                                                float* s_tot, double* s_tot64)
{
    const uint32_t tid = threadIdx.x, w = tid >> 5, l = tid & 31u;
    const uint32_t job = a.props[p].job;
    const uint32_t B = a.jobs[job].B;
    if (!(a.jobs[job].R <= a.max_rows && (B + 31u) / 32u <= cl)) {
        if (tid == 0u) {
            atomicOr(a.err, PCS_ERRBIT_ROWS);
            a.dist_f32[p] = __int_as_float(0x7fc00000);
        }
        return;
    }
    const uint32_t ns = (B + 31u) / 32u;
#pragma unroll
    for (uint32_t h = 0; h < 2u; ++h) {
        const uint32_t lw = 2u * w + h;
        float acc = 0.0f;
        double acc64 = 0.0;
        for (uint32_t j = 0; j < ns; ++j)
            if (32u * j + lw < B) {
                acc = __fadd_rn(acc, __uint_as_float(ld_cluster_(part.f + lw * 32u + l, j)));
                if (F64) acc64 = __dadd_rn(acc64, ld_cluster_f64_(part.d + lw * 32u + l, j));
            }
        const float ws = reduce0_(acc);
        const double wd = F64 ? reduce0_(acc64) : 0.0;
        if (l == 0u) {
            s_tot[lw] = ws;
            if (F64) s_tot64[lw] = wd;
        }
    }
    __syncthreads();
    if (w == 0u) {
        const float fin = reduce0_(s_tot[l]);
        const double fin64 = F64 ? reduce0_(s_tot64[l]) : 0.0;
        uint64_t hi = 0u, lo = 0u;
        if (SSD) {
            if (l < kStripThreads / 32u)
                for (uint32_t j = 0; j < ns; ++j) {
                    uint64_t v[2];
#pragma unroll
                    for (uint32_t i = 0; i < 2u; ++i)
                        v[i] = (uint64_t)ld_cluster_(part.sq + 2u * l + i, j) |
                               (uint64_t)ld_cluster_(reinterpret_cast<const uint32_t*>(part.sq + 2u * l + i) + 1, j) << 32;
                    add128_(hi, lo, v[0], v[1]);
                }
            for (uint32_t d = 16; d >= 1; d >>= 1) {
                const uint64_t ohi = __shfl_down_sync(0xFFFFFFFFu, hi, d), olo = __shfl_down_sync(0xFFFFFFFFu, lo, d);
                if (l + d < 32u) add128_(hi, lo, ohi, olo);
            }
        }
        if (l == 0u) {
            a.dist_f32[p] = fin;
            if (F64 && a.dist_f64) a.dist_f64[p] = fin64;
            if (SSD && a.ssd) {
                a.ssd[2 * (uint64_t)p] = hi;
                a.ssd[2 * (uint64_t)p + 1] = lo;
            }
        }
    }
}

template <bool F64, bool SSD>
__device__ __forceinline__ void strip_cluster_(const DistArgs& a, uint32_t db, uint32_t cl, uint32_t M,
                                               uint32_t* tiles, uint32_t tile_words, const uint32_t* zero,
                                               uint32_t* carry, uint32_t* P2, const ClusterSums& part2, float* s_tot, double* s_tot64,
                                               uint32_t (*s_col)[32], uint32_t (*s_K)[32], uint64_t* s_mbar,
                                               uint32_t* s_abort)
{
    const uint32_t tid = threadIdx.x;
    const uint32_t w = tid >> 5, l = tid & 31u;
    const uint32_t k = cluster_rank_(), ncl = cluster_count_();
    const uint32_t prow = strip_cap_rows(a.max_rows);
    uint32_t p = cluster_id_();
    cluster_sync_(); /* every CTA of the cluster runs before shared::cluster reads */
    uint32_t cur = 0, parity = 0u, pending = 1u, it = 0u, ab = 0u;
    uint32_t p_prev = 0u;
    cluster_fill_(a, p, k, cl, tiles, tid, &s_mbar[0]);
    cp_async_commit_();
    for (;;) {
        const uint32_t job = a.props[p].job;
        const uint32_t R = a.jobs[job].R, B = a.jobs[job].B;
        const uint32_t ns = (B + 31u) / 32u;
        const bool ok = R <= a.max_rows && ns <= cl;
        const bool act = ok && k < ns;
        const uint32_t c0 = 32u * k;
        const uint32_t pn = p + ncl;
        const bool has_next = pn < M;
        uint32_t* P = P2 + (it & 1u) * prow;
        const ClusterSums part = part2.of(it);
        cp_async_wait_<0>();
        if (!mbar_wait_(&s_mbar[cur], (parity >> cur) & 1u)) {
            atomicOr(a.err, PCS_ERRBIT_TIMEOUT);
            *s_abort = 1u;
        }
        parity ^= 1u << cur;
        pending &= ~(1u << cur);
        __syncwarp();
        uint32_t* T = tiles + cur * tile_words;
        const Seg sg = seg_(R, w);
        const uint32_t lc = l >> 2, lo = l & 3u;
        if (act) {
            /* phase A1 as in the strip walk, and the strip zeroed */
            uint32_t run = 0u;
            for (uint32_t r8 = sg.rb; r8 < sg.re; r8 += 8u) {
                uint32_t* t = T + (r8 << 5);
#pragma unroll
                for (uint32_t j = 0; j < 8u; ++j) {
                    uint32_t* q = t + (j << 5) + (((lc ^ j) << 2) | lo);
                    run += *q;
                    *q = run;
                }
            }
            s_col[w][l] = run;
            uint32_t z;
            const TmapDev* map = prop_tmap_(a, p, job, z);
            if (map) {
                if (tid == 0u) {
                    const uint32_t nbox = (R + kBox - 1u) / kBox;
                    for (uint32_t b = 0; b < nbox; ++b) tma_store_3d_(map, c0, b * kBox, z, zero);
                    bulk_commit_();
                }
            } else if (c0 + l < B) {
                uint32_t* hist = a.hist + a.props[p].hist_off;
                for (uint32_t r = sg.rb; r < min(sg.re, R); ++r) __stcs(hist + (uint64_t)r * B + c0 + l, 0u);
            }
        }
        __syncthreads();
        if (db && has_next && !*s_abort) {
            cluster_fill_(a, pn, k, cl, tiles + (cur ^ 1u) * tile_words, tid, &s_mbar[cur ^ 1u]);
            pending |= 1u << (cur ^ 1u);
            cp_async_commit_();
        }
        if (act) {
            /* phase A2 with row carry 0: the strip's own 2-D prefix sums */
            uint32_t cc = 0u;
            for (uint32_t q = 0; q < w; ++q) cc += s_col[q][l];
            s_K[w][l] = warp_scan_(cc, l);
            __syncwarp();
            const uint4* K4 = reinterpret_cast<const uint4*>(s_K[w]);
            for (uint32_t r = sg.rb + l; r < sg.re; r += 32u) {
                uint4* row4 = reinterpret_cast<uint4*>(T + (r << 5));
                const uint32_t m = r & 7u;
                uint32_t acc = 0u;
                uint4 o = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (uint32_t j = 0; j < 8u; ++j) {
                    const uint4 v = row4[j ^ m];
                    const uint4 kk = K4[j];
                    acc += v.x;
                    o.x = acc + kk.x;
                    acc += v.y;
                    o.y = acc + kk.y;
                    acc += v.z;
                    o.z = acc + kk.z;
                    acc += v.w;
                    o.w = acc + kk.w;
                    row4[j ^ m] = o;
                }
                P[r] = o.w;
            }
        }
        /* this histogram's last columns, and the previous one's per-lane sums, published */
        cluster_sync_();
        for (uint32_t j = 0; j < cl; ++j) ab |= ld_cluster_(s_abort, j);
        if (ab) break; /* a copy wait ran out somewhere in the cluster (error word set) */
        if (act) {
            /* row carry from the strips to the left */
            for (uint32_t r = tid; r < R; r += kStripThreads) {
                uint32_t c = 0u;
                for (uint32_t j = 0; j < k; ++j) c += ld_cluster_(P + r, j);
                carry[r] = c;
            }
            __syncthreads();
            uint32_t* cum = a.cum_out ? a.cum_out + a.props[p].hist_off : nullptr;
            if (cum && c0 + l < B)
                for (uint32_t r = w; r < R; r += kStripThreads / 32u) __stcs(cum + (uint64_t)r * B + c0 + l, T[sw_(r, l)] + carry[r]);
            /* phase B as in the strip walk, the row carry added to each cell */
            const uint32_t colA = c0 + 2u * w;
            float a2A = 0.0f, a2B = 0.0f;
            double a2dA = 0.0, a2dB = 0.0;
            uint64_t shi = 0u, slo = 0u;
            if (colA < B) {
                const bool inB = colA + 1u < B;
                const uint32_t* Tl = T + ((((w >> 1) ^ (l & 7u)) << 2) | ((2u * w) & 3u));
                const uint32_t* __restrict__ refT = a.jobs[job].ref_sat_t;
                const uint32_t* refc = refT + (uint64_t)colA * R;
                bool exact = (F64 || SSD || !cum) && T[sw_(R - 1u, 31u)] + carry[R - 1u] < kExactBelow &&
                             __ldg(refT + pcs_sat_t_index(R - 1u, B - 1u, R, B)) < kExactBelow;
                uint64_t iA = 0u, iB = 0u;
                uint32_t seen = 0u;
                if (exact && inB) {
                    const uint2* ref2 = reinterpret_cast<const uint2*>(refc);
#pragma unroll 4
                    for (uint32_t r = l; r < R; r += 32u) {
                        const uint2 v = *reinterpret_cast<const uint2*>(Tl + (r << 5));
                        const uint32_t c = carry[r];
                        const uint2 o = __ldg(ref2 + r);
                        const float dA = exact_diff_(v.x + c, o.x);
                        const float dB = exact_diff_(v.y + c, o.y);
                        a2A = __fadd_rn(a2A, __fmul_rn(dA, dA));
                        a2B = __fadd_rn(a2B, __fmul_rn(dB, dB));
                        if (F64 || SSD) {
                            iA += square_(v.x + c, o.x);
                            iB += square_(v.y + c, o.y);
                            seen |= (v.x + c) | (v.y + c) | o.x | o.y;
                        }
                    }
                } else if (exact) {
                    for (uint32_t r = l; r < R; r += 32u) {
                        const uint32_t v = Tl[r << 5] + carry[r], o = __ldg(refc + r);
                        const float dA = exact_diff_(v, o);
                        a2A = __fadd_rn(a2A, __fmul_rn(dA, dA));
                        if (F64 || SSD) {
                            iA += square_(v, o);
                            seen |= v | o;
                        }
                    }
                }
                if (F64 || SSD) exact = exact && seen < kExactBelow;
                if (!exact) {
                    a2A = a2B = 0.0f;
                    for (uint32_t r = l; r < R; r += 32u) {
                        const uint32_t c = carry[r];
                        if (inB) {
                            const uint2 v = *reinterpret_cast<const uint2*>(Tl + (r << 5));
                            const uint2 o = __ldg(reinterpret_cast<const uint2*>(refc) + r);
                            term_<F64, SSD>(v.x + c, o.x, a2A, a2dA, shi, slo);
                            term_<F64, SSD>(v.y + c, o.y, a2B, a2dB, shi, slo);
                        } else {
                            term_<F64, SSD>(Tl[r << 5] + c, __ldg(refc + r), a2A, a2dA, shi, slo);
                        }
                    }
                }
                if (exact) {
                    if (F64) {
                        a2dA = (double)iA;
                        a2dB = (double)iB;
                    }
                    if (SSD) {
                        add128_(shi, slo, 0u, iA);
                        add128_(shi, slo, 0u, iB);
                    }
                }
            }
            part.f[(2u * w) * 32u + l] = a2A;
            part.f[(2u * w + 1u) * 32u + l] = a2B;
            if (F64) {
                part.d[(2u * w) * 32u + l] = a2dA;
                part.d[(2u * w + 1u) * 32u + l] = a2dB;
            }
            if (SSD) {
                for (uint32_t d = 16; d >= 1; d >>= 1) {
                    const uint64_t ohi = __shfl_down_sync(0xFFFFFFFFu, shi, d), olo = __shfl_down_sync(0xFFFFFFFFu, slo, d);
                    if (l + d < 32u) add128_(shi, slo, ohi, olo);
                }
                if (l == 0u) {
                    part.sq[2u * w] = shi;
                    part.sq[2u * w + 1u] = slo;
                }
            }
        }
        /* this tile's generic accesses before its next box fill */
        fence_proxy_async_();
        if (!db && has_next) {
            __syncthreads(); /* the one tile is free: refill it before CTA 0's reduction */
            cluster_fill_(a, pn, k, cl, tiles, tid, &s_mbar[0]);
            pending |= 1u;
            cp_async_commit_();
        }
        /* CTA 0: the previous histogram, whose sums every CTA published before the barrier */
        if (k == 0u && it > 0u) cluster_reduce_<F64, SSD>(a, p_prev, cl, part2.of(it - 1u), s_tot, s_tot64);
        if (!has_next) break;
        if (db) cur ^= 1u;
        p_prev = p;
        p = pn;
        ++it;
    }
    cluster_sync_(); /* the last histogram's per-lane sums published */
    if (!ab && k == 0u) cluster_reduce_<F64, SSD>(a, p, cl, part2.of(it), s_tot, s_tot64);
    cluster_sync_(); /* no CTA leaves while CTA 0 reads its sums */
    cp_async_wait_<0>();
    for (uint32_t b = 0; b < 2u; ++b)
        if ((pending >> b) & 1u) mbar_wait_(&s_mbar[b], (parity >> b) & 1u);
    bulk_wait_all_();
}

/* Cluster mode, clusters of cl CTAs. */
template <bool F64, bool SSD>
__global__ void __launch_bounds__(512, 2) k_distance_cluster(DistArgs a, uint32_t db, uint32_t cl)
{
    extern __shared__ __align__(16) uint32_t s_mem[];
    const uint32_t M = *a.n_props;
    if (cluster_id_() >= M) return; /* whole clusters return */
    const uint32_t prow = strip_cap_rows(a.max_rows), tile_words = prow * 32u;
    /* [1 + db][cap rows][32] tiles (1024-byte aligned), a zero box, the row
     * carries, two last-column arrays, two 32 x 32 per-lane sum arrays, with
     * F64 two of doubles */
    uint32_t* tiles = s_mem + ((1024u - (smem_u32_(s_mem) & 1023u)) & 1023u) / 4u;
    uint32_t* zero = tiles + (1u + db) * tile_words;
    uint32_t* carry = zero + kBox * kBox;
    uint32_t* P2 = carry + prow;
    float* f2 = reinterpret_cast<float*>(P2 + 2u * prow);
    double* d2 = reinterpret_cast<double*>(f2 + 2u * 1024u);
    __shared__ float s_tot[32];
    __shared__ double s_tot64[32];
    __shared__ uint64_t s_sq[2u * (kStripThreads / 16u)];
    __shared__ uint32_t s_col[16][32];
    __shared__ __align__(16) uint32_t s_K[16][32];
    __shared__ __align__(8) uint64_t s_mbar[2];
    __shared__ uint32_t s_abort;
    const uint32_t tid = threadIdx.x;
    if (tid == 0) {
        mbar_init_(&s_mbar[0], kStripThreads);
        mbar_init_(&s_mbar[1], kStripThreads);
        mbar_init_fence_();
        s_abort = 0u;
    }
    for (uint32_t i = tid; i < kBox * kBox; i += kStripThreads) zero[i] = 0u;
    fence_proxy_async_(); /* the zero box, before box stores read it */
    __syncthreads();
    const ClusterSums part2 = {f2, d2, s_sq};
    strip_cluster_<F64, SSD>(a, db, cl, M, tiles, tile_words, zero, carry, P2, part2, s_tot, s_tot64, s_col, s_K, s_mbar,
                             &s_abort);
}

/* Row kernel: a CTA takes one histogram at a time, a warp 128 of its columns
 * (lane l columns 4l..4l+3), and the rows stream past.  Rows come in blocks of
 * 8 through a ring of three blocks per warp in shared memory, filled two
 * blocks ahead by each lane's own cp.async (16 bytes where the rows are
 * 16-byte aligned, else cell by cell), so no lane waits for another's copy.
 * A lane keeps its columns' running sums; one warp scan per row (eight rows'
 * step by step together) turns them into the row's 2-D prefix sums.  With
 * more than 128 columns the warps exchange each row's last prefix sum once
 * per block (one CTA barrier).  The reference's per-lane sums, one for every
 * (row mod 32, column) of a strip of 32 columns, live in shared memory as
 * [32][128] floats per warp, one 16-byte read and write per row and lane; at
 * the end the strips' are added in order and the reference's trees follow.
 *
 * 65 warp instructions per 128 cells, where the strip kernel, passing over
 * its tile three times, has about 150; of 8 warps per SM (shared memory: 28 KB
 * each, 64 KB of loads in flight) the two per scheduler issue in 32 % of the
 * cycles, between waits for shared memory, scans and the observed cells.
 * 1024 of 301 x 128: 88 us (strips) -> 52 us.  One lane per column instead
 * (7 KB per warp, 32 warps per SM) has 48 instructions per 32 cells: 86 us.
 * A walk down few rows at a time costs a fixed 90 ns per row, so few
 * histograms of few columns stay with the strips (use_rows_).
 *
 * Where every value of a block of rows is below 2^22 the differences are exact
 * integers (see k_distance_strip); other blocks take the reference's
 * conversions.  All of the block's counts are looked at, not its last row's:
 * an observed array passed to a standalone call need not grow down the rows.
 * The vote comes after the integer form's terms, which are dropped where it
 * fails, so nothing waits for it (device time of whole device calls: 304 of
 * 1001 x 256 144 us, 143 without the look at every count, 146 with the vote
 * before the terms; 152 of 1700 x 256 202, 201, 214).  F64 needs exact
 * differences and an exact sum of squares below 2^53, where the reference's
 * chain of double additions is exact in any order.  Whether that holds is
 * known when the last row has passed: a histogram for which it does not is
 * left as it was (with F64 the zeroing waits for the verdict) with kRedo as
 * its distance, and the strip kernel launched after it takes it. */
const uint32_t kRowsBlock = 8u, kRowsRing = 3u, kRowsWarps = 8u;
const uint32_t kRowsAccBytes = 32u * 128u * 4u, kRowsRingBytes = kRowsRing * kRowsBlock * 512u;
const uint32_t kRowsWarpBytes = kRowsAccBytes + kRowsRingBytes;

/* 16 bytes where `valid`, else zeros, without reading src */
__device__ __forceinline__ void cp_async16z_(void* dst, const void* src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32_(dst)), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}

/* a warp's inclusive scans of eight values, step by step together */
__device__ __forceinline__ void warp_scan8_(uint32_t* t)
{
#define PCS_SCAN_STEP(d)                                                                                       \
    _Pragma("unroll") for (uint32_t i = 0; i < kRowsBlock; ++i)                                                 \
        asm volatile("{\n\t.reg .u32 u;\n\t.reg .pred p;\n\tshfl.sync.up.b32 u|p, %0, " #d                     \
                     ", 0x0, 0xffffffff;\n\t@p add.u32 %0, %0, u;\n\t}\n"                                       \
                     : "+r"(t[i]));
    PCS_SCAN_STEP(1)
    PCS_SCAN_STEP(2)
    PCS_SCAN_STEP(4)
    PCS_SCAN_STEP(8)
    PCS_SCAN_STEP(16)
#undef PCS_SCAN_STEP
}

/* One warp's walk down its 128 columns of a histogram. */
template <bool F64, bool SSD, bool VEC>
struct RowsWalk {
    const uint32_t* hist; /* this lane's first column (or column 0), row 0 */
    const uint32_t* next; /* the same, the next row to fill (16-byte rows) */
    const uint32_t* ref;  /* of the next row of the observed histogram */
    uint32_t* gone;       /* the next row to zero */
    uint32_t* cum;        /* or null */
    uint4* ring;          /* [3][8] steps of 32 */
    float4* acc;          /* [32] steps of 32 */
    uint32_t (*P)[kRowsWarps][kRowsBlock];
    uint32_t R, B, nc, w, l, NP;
    uint4 col, o[kRowsBlock];
    bool high;            /* a value of 2^22 or more has passed */
    uint64_t hi, lo;      /* exact sum of squares */

    /* this lane's copies of block b (one group); rows and columns past the last arrive as zeros */
    __device__ __forceinline__ void fill(uint32_t b)
    {
        uint4* to = ring + (b % kRowsRing) * (kRowsBlock * 32u);
        const bool full = (b + 1u) * kRowsBlock <= R;
        if (VEC && full) {
            if (nc) {
#pragma unroll
                for (uint32_t i = 0; i < kRowsBlock; ++i, next += B) cp_async16z_(to + i * 32u, next, true);
            }
        } else {
#pragma unroll
            for (uint32_t i = 0; i < kRowsBlock; ++i) {
                const uint32_t r = b * kRowsBlock + i;
                const uint32_t* from = hist + (uint64_t)min(r, R - 1u) * B;
                if (VEC) {
                    cp_async16z_(to + i * 32u, from, r < R && nc != 0u);
                } else {
#pragma unroll
                    for (uint32_t x = 0; x < 4u; ++x)
                        cp_async4_(reinterpret_cast<uint32_t*>(to + i * 32u) + x, from + (x < nc ? x : 0u), r < R && x < nc);
                }
            }
        }
        cp_async_commit_();
    }

    /* the observed histogram's cells at q in this lane's columns */
    __device__ __forceinline__ uint4 observed(const uint32_t* q) const
    {
        if (VEC) return __ldg(reinterpret_cast<const uint4*>(q));
        return make_uint4(__ldg(q), __ldg(q + (1u < nc ? 1u : 0u)), __ldg(q + (2u < nc ? 2u : 0u)), __ldg(q + (3u < nc ? 3u : 0u)));
    }

    /* those of block b; rows past the last take the last row's */
    __device__ __forceinline__ void observe(uint32_t b)
    {
        if ((b + 1u) * kRowsBlock <= R) {
#pragma unroll
            for (uint32_t i = 0; i < kRowsBlock; ++i, ref += B) o[i] = observed(ref);
        } else if (b * kRowsBlock < R) {
#pragma unroll
            for (uint32_t i = 0; i < kRowsBlock; ++i) {
                o[i] = observed(ref);
                if (b * kRowsBlock + i + 1u < R) ref += B;
            }
        }
    }

    /* one row's cells zeroed, as K_distance does */
    __device__ __forceinline__ void zero_row()
    {
        if (VEC) {
            if (nc) __stcs(reinterpret_cast<uint4*>(gone), make_uint4(0u, 0u, 0u, 0u));
        } else {
            if (nc > 0u) __stcs(gone, 0u);
            if (nc > 1u) __stcs(gone + 1, 0u);
            if (nc > 2u) __stcs(gone + 2, 0u);
            if (nc > 3u) __stcs(gone + 3, 0u);
        }
        gone += B;
    }

    /* the rows' terms added to the sums (columns past the last too: they are not read) */
    template <bool FULL, typename Diff>
    __device__ __forceinline__ void terms(uint32_t b, const uint4* s, float4* v, Diff diff) const
    {
#pragma unroll
        for (uint32_t i = 0; i < kRowsBlock; ++i) {
            if (!FULL && b * kRowsBlock + i >= R) break;
            const float dx = diff(s[i].x, o[i].x), dy = diff(s[i].y, o[i].y);
            const float dz = diff(s[i].z, o[i].z), dw = diff(s[i].w, o[i].w);
            v[i].x = __fadd_rn(v[i].x, __fmul_rn(dx, dx));
            v[i].y = __fadd_rn(v[i].y, __fmul_rn(dy, dy));
            v[i].z = __fadd_rn(v[i].z, __fmul_rn(dz, dz));
            v[i].w = __fadd_rn(v[i].w, __fmul_rn(dw, dw));
        }
    }

    __device__ __forceinline__ void wide_square_(uint32_t s, uint32_t o)
    {
        const uint64_t d = s >= o ? s - o : o - s;
        add128_(hi, lo, 0u, d * d);
    }

    template <bool FULL>
    __device__ __forceinline__ void block(uint32_t b)
    {
        fill(b + 2u);
        cp_async_wait_<2>();
        const uint4* in = ring + (b % kRowsRing) * (kRowsBlock * 32u);
        uint4 s[kRowsBlock];
#pragma unroll
        for (uint32_t i = 0; i < kRowsBlock; ++i) {
            const uint4 v = in[i * 32u];
            col.x += v.x;
            col.y += v.y;
            col.z += v.z;
            col.w += v.w;
            s[i].x = col.x;
            s[i].y = col.x + col.y;
            s[i].z = s[i].y + col.z;
            s[i].w = s[i].z + col.w;
            if (!F64 && (FULL || b * kRowsBlock + i < R)) zero_row();
        }
        uint32_t t[kRowsBlock];
#pragma unroll
        for (uint32_t i = 0; i < kRowsBlock; ++i) t[i] = s[i].w;
        warp_scan8_(t);
#pragma unroll
        for (uint32_t i = 0; i < kRowsBlock; ++i) {
            const uint32_t before = t[i] - s[i].w;
            s[i].x += before;
            s[i].y += before;
            s[i].z += before;
            s[i].w = t[i];
        }
        if (NP > 1u) {
            uint32_t (*Pb)[kRowsBlock] = P[b & 1u];
            if (l == 31u) {
#pragma unroll
                for (uint32_t i = 0; i < kRowsBlock; ++i) Pb[w][i] = s[i].w;
            }
            __syncthreads();
            uint32_t left = 0u;
            for (uint32_t j = 0; j < w; ++j) left += Pb[j][l & (kRowsBlock - 1u)];
#pragma unroll
            for (uint32_t i = 0; i < kRowsBlock; ++i) {
                const uint32_t add = __shfl_sync(0xFFFFFFFFu, left, i);
                s[i].x += add;
                s[i].y += add;
                s[i].z += add;
                s[i].w += add;
            }
        }
        float4* at = acc + (b & 3u) * (kRowsBlock * 32u);
        float4 v[kRowsBlock];
#pragma unroll
        for (uint32_t i = 0; i < kRowsBlock; ++i) v[i] = at[i * 32u];
        terms<FULL>(b, s, v, [](uint32_t t, uint32_t q) { return exact_diff_(t, q); });
        /* every bit that a count of the block has (rows past the last repeat it) */
        uint32_t part[kRowsBlock];
#pragma unroll
        for (uint32_t i = 0; i < kRowsBlock; ++i) {
            uint32_t q = o[i].x | o[i].y | o[i].z;
            part[i] = s[i].x | s[i].y | s[i].z;
            asm("" : "+r"(q), "+r"(part[i])); /* a tree, not one chain of all */
            part[i] |= s[i].w | q;
            asm("" : "+r"(part[i]));
            part[i] |= o[i].w;
        }
        const uint32_t seen = ((part[0] | part[1] | part[2]) | (part[3] | part[4] | part[5])) | part[6] | part[7];
        const bool exact = !__any_sync(0xFFFFFFFFu, seen >= kExactBelow);
        if (!exact) {
            high = true;
            if (!F64) { /* the sums are as they were in shared memory */
#pragma unroll
                for (uint32_t i = 0; i < kRowsBlock; ++i) v[i] = at[i * 32u];
                terms<FULL>(b, s, v, [](uint32_t t, uint32_t q) { return __fsub_rn(__uint2float_rn(t), __uint2float_rn(q)); });
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < kRowsBlock; ++i) at[i * 32u] = v[i];
        if (F64 || SSD) {
            /* With F64 the sum counts only where every block is exact: below
             * 2^44 a cell, no carry.  Else a block's is below 2^49. */
            uint64_t sq = 0u;
            uint64_t& sum = F64 ? lo : sq;
#pragma unroll
            for (uint32_t i = 0; i < kRowsBlock; ++i) {
                if (!FULL && b * kRowsBlock + i >= R) break;
                if (F64 || exact) {
                    if (VEC || nc > 0u) sum += square_(s[i].x, o[i].x);
                    if (VEC || nc > 1u) sum += square_(s[i].y, o[i].y);
                    if (VEC || nc > 2u) sum += square_(s[i].z, o[i].z);
                    if (VEC || nc > 3u) sum += square_(s[i].w, o[i].w);
                } else {
                    if (VEC || nc > 0u) wide_square_(s[i].x, o[i].x);
                    if (VEC || nc > 1u) wide_square_(s[i].y, o[i].y);
                    if (VEC || nc > 2u) wide_square_(s[i].z, o[i].z);
                    if (VEC || nc > 3u) wide_square_(s[i].w, o[i].w);
                }
            }
            if (!F64) add128_(hi, lo, 0u, sq);
        }
        observe(b + 1u);
        if (cum) {
#pragma unroll
            for (uint32_t i = 0; i < kRowsBlock; ++i) {
                const uint32_t r = b * kRowsBlock + i;
                if (r < R && nc) {
                    uint32_t* q = cum + (uint64_t)r * B;
                    if (VEC) {
                        __stcs(reinterpret_cast<uint4*>(q), s[i]);
                    } else {
                        q[0] = s[i].x;
                        if (nc > 1u) q[1] = s[i].y;
                        if (nc > 2u) q[2] = s[i].z;
                        if (nc > 3u) q[3] = s[i].w;
                    }
                }
            }
        }
    }

    __device__ __forceinline__ void walk()
    {
        if (VEC && !nc) /* filled by no copy */
#pragma unroll
            for (uint32_t i = 0; i < kRowsRing * kRowsBlock; ++i) ring[i * 32u] = make_uint4(0u, 0u, 0u, 0u);
        next = hist;
        fill(0u);
        fill(1u);
        observe(0u);
#pragma unroll
        for (uint32_t k = 0; k < 32u; ++k) acc[k * 32u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        col = make_uint4(0u, 0u, 0u, 0u);
        high = false;
        hi = lo = 0u;
        uint32_t b = 0u;
        for (; (b + 1u) * kRowsBlock <= R; ++b) block<true>(b);
        if (b * kRowsBlock < R) block<false>(b);
        cp_async_wait_<0>();
    }
};

/* histogram p by the CTA's warps; false: left as it was */
template <bool F64, bool SSD, bool VEC>
__device__ __forceinline__ bool rows_hist_(const DistArgs& a, uint32_t p, const JobDev& jd, uint32_t* hist,
                                           unsigned char* s_rows, uint32_t (*s_P)[kRowsWarps][kRowsBlock],
                                           uint64_t* s_hi, uint64_t* s_lo)
{
    RowsWalk<F64, SSD, VEC> k;
    k.w = threadIdx.x >> 5;
    k.l = threadIdx.x & 31u;
    k.NP = blockDim.x >> 5;
    k.R = jd.R;
    k.B = jd.B;
    const uint32_t c = 128u * k.w + 4u * k.l, w = k.w, l = k.l, NP = k.NP;
    k.nc = c < k.B ? min(k.B - c, 4u) : 0u;
    const uint32_t c1 = k.nc ? c : 0u;
    k.hist = k.gone = hist + c1;
    k.ref = jd.ref_sat + c1;
    k.cum = a.cum_out ? a.cum_out + a.props[p].hist_off + c1 : nullptr;
    k.acc = reinterpret_cast<float4*>(s_rows + w * kRowsWarpBytes) + l;
    k.ring = reinterpret_cast<uint4*>(s_rows + w * kRowsWarpBytes + kRowsAccBytes) + l;
    k.P = s_P;
    k.walk();

    uint64_t hi = k.nc ? k.hi : 0u, lo = k.nc ? k.lo : 0u;
    if (F64 || SSD) {
        for (uint32_t d = 16; d >= 1; d >>= 1) {
            const uint64_t ohi = __shfl_down_sync(0xFFFFFFFFu, hi, d);
            const uint64_t olo = __shfl_down_sync(0xFFFFFFFFu, lo, d);
            if (l + d < 32u) add128_(hi, lo, ohi, olo);
        }
        if (l == 0u) {
            s_hi[w] = hi;
            s_lo[w] = lo;
        }
    }
    const bool over = __syncthreads_or(k.high) != 0;
    if (F64 || SSD) {
        hi = lo = 0u;
        for (uint32_t j = 0; j < NP; ++j) add128_(hi, lo, s_hi[j], s_lo[j]);
    }
    if (F64) {
        if (over || hi != 0u || (lo >> 53) != 0u) return false;
#pragma unroll 8
        for (uint32_t r = 0; r < k.R; ++r) k.zero_row();
    }
    /* (logical warp l, lane i): its strips' sums in order; then the trees */
    float* sums = reinterpret_cast<float*>(s_rows + kRowsAccBytes); /* [32][33], over warp 0's ring */
    const uint32_t ns = (k.B + 31u) / 32u;
    for (uint32_t i = w; i < 32u; i += NP) {
        float v = 0.0f;
        for (uint32_t j = 0; j < ns; ++j)
            if (32u * j + l < k.B)
                v = __fadd_rn(v, reinterpret_cast<const float*>(s_rows + (j >> 2) * kRowsWarpBytes)[i * 128u + (j & 3u) * 32u + l]);
        sums[l * 33u + i] = v;
    }
    __syncthreads();
    if (w == 0u) {
        float v[32];
#pragma unroll
        for (uint32_t i = 0; i < 32u; ++i) v[i] = sums[l * 33u + i];
#pragma unroll
        for (uint32_t d = 16; d >= 1; d >>= 1)
#pragma unroll
            for (uint32_t i = 0; i < d; ++i) v[i] = __fadd_rn(v[i], v[i + d]);
        const float fin = reduce0_(v[0]);
        if (l == 0u) {
            a.dist_f32[p] = fin;
            if (F64 && a.dist_f64) a.dist_f64[p] = (double)lo;
            if (SSD && a.ssd) {
                a.ssd[2 * (uint64_t)p] = hi;
                a.ssd[2 * (uint64_t)p + 1] = lo;
            }
        }
    }
    return true;
}

template <bool F64, bool SSD>
__global__ void __launch_bounds__(32 * kRowsWarps) k_distance_rows(DistArgs a)
{
    extern __shared__ __align__(128) unsigned char s_rows[]; /* per warp: float sums [32][128], ring [3][8][128] */
    __shared__ uint32_t s_P[2][kRowsWarps][kRowsBlock];      /* each warp's last prefix sum of a row */
    __shared__ uint64_t s_hi[kRowsWarps], s_lo[kRowsWarps];
    const uint32_t M = *a.n_props;
    for (uint32_t p = blockIdx.x; p < M; p += gridDim.x) {
        const JobDev& jd = a.jobs[a.props[p].job];
        uint32_t* hist = a.hist + a.props[p].hist_off;
        bool done = false;
        if (jd.R > a.max_rows || jd.B > 4u * blockDim.x) {
            if (threadIdx.x == 0u) {
                atomicOr(a.err, PCS_ERRBIT_ROWS);
                a.dist_f32[p] = __int_as_float(0x7fc00000);
            }
            done = true;
        } else {
            const uintptr_t at = reinterpret_cast<uintptr_t>(hist) | reinterpret_cast<uintptr_t>(jd.ref_sat) |
                                 reinterpret_cast<uintptr_t>(a.cum_out ? a.cum_out + a.props[p].hist_off : nullptr);
            if (((jd.B * 4u) & 15u) == 0u && (at & 15u) == 0u)
                done = rows_hist_<F64, SSD, true>(a, p, jd, hist, s_rows, s_P, s_hi, s_lo);
            else
                done = rows_hist_<F64, SSD, false>(a, p, jd, hist, s_rows, s_P, s_hi, s_lo);
        }
        if (!done && threadIdx.x == 0u) a.dist_f32[p] = __uint_as_float(kRedo);
        __syncthreads(); /* the sums are read */
    }
}

/* the first histogram from p on in this CTA's sequence that is the strip
 * kernel's: all of them, or (REDO) those that the row kernel left */
template <bool REDO>
__device__ __forceinline__ uint32_t strip_next_(const DistArgs& a, uint32_t p, uint32_t M)
{
    if (REDO)
        while (p < M && __float_as_uint(a.dist_f32[p]) != kRedo) p += gridDim.x;
    return p;
}

template <bool F64, bool SSD, bool REDO>
__global__ void __launch_bounds__(512, 2) k_distance_strip(DistArgs a, uint32_t db)
{
    extern __shared__ __align__(16) uint32_t s_mem[];
    const uint32_t tile_words = strip_cap_rows(a.max_rows) * 32u;
    /* [1 + db][cap rows][32] tiles, 1024-byte aligned (the launch reserves
     * 1024 bytes for this), a zero box, the row carries */
    uint32_t* tiles = s_mem + ((1024u - (smem_u32_(s_mem) & 1023u)) & 1023u) / 4u;
    uint32_t* zero = tiles + (1u + db) * tile_words;
    uint32_t* carry = zero + kBox * kBox;
    __shared__ float s_tot[32];
    __shared__ double s_tot64[32];
    __shared__ uint64_t s_hi[32], s_lo[32];
    __shared__ uint32_t s_col[16][32];             /* column totals of each warp's row segment */
    __shared__ __align__(16) uint32_t s_K[16][32]; /* per segment: prefix across the strip of its column carries */
    __shared__ __align__(8) uint64_t s_mbar[2];
    __shared__ uint32_t s_abort;

    const uint32_t tid = threadIdx.x;
    const uint32_t w = tid >> 5, l = tid & 31u;
    const uint32_t M = *a.n_props;
    uint32_t p = strip_next_<REDO>(a, blockIdx.x, M);
    if (p >= M) return;
    if (tid == 0) {
        mbar_init_(&s_mbar[0], kStripThreads);
        mbar_init_(&s_mbar[1], kStripThreads);
        mbar_init_fence_();
        s_abort = 0u;
    }
    for (uint32_t i = tid; i < kBox * kBox; i += kStripThreads) zero[i] = 0u;
    fence_proxy_async_(); /* the zero box, before box stores read it */
    __syncthreads();

    uint32_t c0 = 0, cur = 0, parity = 0u; /* parity bit b: the phase of tile b's next fill */
    uint32_t pending = 1u;                  /* bit b: tile b has a fill in flight */
    strip_fill_(a, p, 0u, tiles, tid, &s_mbar[0]);
    cp_async_commit_();

    float acc0 = 0.0f, acc1 = 0.0f;
    double accd0 = 0.0, accd1 = 0.0;
    uint64_t shi = 0, slo = 0;
    for (;;) {
        const uint32_t job = a.props[p].job;
        const uint64_t hoff = a.props[p].hist_off;
        const uint32_t R = a.jobs[job].R, B = a.jobs[job].B;
        const bool ok = R <= a.max_rows;
        /* the (proposal, strip) after this one */
        uint32_t pn = p, cn = c0 + 32u;
        if (!ok || cn >= B) {
            pn = strip_next_<REDO>(a, p + gridDim.x, M);
            cn = 0u;
        }
        const bool has_next = pn < M;
        cp_async_wait_<0>(); /* this thread's cell copies of the current strip have landed */
        /* the current strip's box copies (all threads' arrivals and bytes) */
        if (!mbar_wait_(&s_mbar[cur], (parity >> cur) & 1u)) {
            atomicOr(a.err, PCS_ERRBIT_TIMEOUT);
            s_abort = 1u;
        }
        parity ^= 1u << cur;
        pending &= ~(1u << cur);
        __syncwarp(); /* cells copied by other lanes of this warp */
        uint32_t* T = tiles + cur * tile_words;
        if (!ok) {
            if (tid == 0) {
                atomicOr(a.err, PCS_ERRBIT_ROWS);
                a.dist_f32[p] = __int_as_float(0x7fc00000);
            }
            __syncthreads();
            if (s_abort) break; /* a copy wait ran out (error word set) */
            if (db && has_next) {
                strip_fill_(a, pn, cn, tiles + (cur ^ 1u) * tile_words, tid, &s_mbar[cur ^ 1u]);
                pending |= 1u << (cur ^ 1u);
                cp_async_commit_();
            }
        } else {
            const uint32_t* __restrict__ refT = a.jobs[job].ref_sat_t;
            uint32_t* hist = a.hist + hoff;
            uint32_t* cum = a.cum_out ? a.cum_out + hoff : nullptr;
            const Seg sg = seg_(R, w);
            const uint32_t lc = l >> 2, lo = l & 3u;
            /* phase A1: column prefix within the segment, segment totals */
            uint32_t run = 0u;
            for (uint32_t r8 = sg.rb; r8 < sg.re; r8 += 8u) {
                uint32_t* t = T + (r8 << 5);
#pragma unroll
                for (uint32_t k = 0; k < 8u; ++k) {
                    uint32_t* q = t + (k << 5) + (((lc ^ k) << 2) | lo);
                    run += *q;
                    *q = run;
                }
            }
            s_col[w][l] = run;
            /* ... and the strip is zeroed in the histogram */
            uint32_t z;
            const TmapDev* map = prop_tmap_(a, p, job, z);
            if (map) {
                if (tid == 0u) {
                    const uint32_t nbox = (R + kBox - 1u) / kBox;
                    for (uint32_t b = 0; b < nbox; ++b) tma_store_3d_(map, c0, b * kBox, z, zero);
                    bulk_commit_();
                }
            } else if (c0 + l < B) {
                for (uint32_t r = sg.rb; r < min(sg.re, R); ++r) __stcs(hist + (uint64_t)r * B + c0 + l, 0u);
            }
            __syncthreads();
            if (s_abort) break; /* a copy wait ran out (error word set) */
            /* every warp is past the previous strip, whose tile the next
             * strip's copies now fill (with two tiles) */
            if (db && has_next) {
                strip_fill_(a, pn, cn, tiles + (cur ^ 1u) * tile_words, tid, &s_mbar[cur ^ 1u]);
                pending |= 1u << (cur ^ 1u);
                cp_async_commit_();
            }
            /* phase A2: column carry into the segment, scanned across the
             * strip; then the row prefix from the left strips' row carry */
            uint32_t cc = 0u;
            for (uint32_t q = 0; q < w; ++q) cc += s_col[q][l];
            s_K[w][l] = warp_scan_(cc, l);
            __syncwarp();
            const uint4* K4 = reinterpret_cast<const uint4*>(s_K[w]);
            for (uint32_t r = sg.rb + l; r < sg.re; r += 32u) {
                uint4* row4 = reinterpret_cast<uint4*>(T + (r << 5));
                const uint32_t m = r & 7u;
                uint32_t acc = c0 ? carry[r] : 0u;
                uint4 o = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (uint32_t j = 0; j < 8u; ++j) {
                    const uint4 v = row4[j ^ m];
                    const uint4 k = K4[j];
                    acc += v.x;
                    o.x = acc + k.x;
                    acc += v.y;
                    o.y = acc + k.y;
                    acc += v.z;
                    o.z = acc + k.z;
                    acc += v.w;
                    o.w = acc + k.w;
                    row4[j ^ m] = o;
                }
                carry[r] = o.w;
            }
            __syncthreads();
            /* the strip's prefix sums, a row segment of 128 bytes per warp (the
             * lanes of phase B hold columns, whose cells lie B apart) */
            if (cum && c0 + l < B)
                for (uint32_t r = w; r < R; r += kStripThreads / 32u) cum[(uint64_t)r * B + c0 + l] = T[sw_(r, l)];
            /* phase B: columns c0 + 2w and c0 + 2w + 1; lane l reads rows
             * l, l + 32, ..., all congruent to l mod 8, so its swizzled
             * offset within a row is fixed */
            const uint32_t colA = c0 + 2u * w;
            if (colA < B) {
                const bool inB = colA + 1u < B;
                const uint32_t* Tl = T + ((((w >> 1) ^ (l & 7u)) << 2) | ((2u * w) & 3u));
                const uint32_t* refc = refT + (uint64_t)colA * R; /* this column pair (or lone last column) */
                float a2A = 0.0f, a2B = 0.0f;
                double a2dA = 0.0, a2dB = 0.0;
                /* the largest cumulative counts: the strip's and the observed histogram's last cells */
                bool exact = (F64 || SSD || !cum) && T[sw_(R - 1u, 31u)] < kExactBelow &&
                             __ldg(refT + pcs_sat_t_index(R - 1u, B - 1u, R, B)) < kExactBelow;
                uint64_t iA = 0u, iB = 0u; /* exact sums of squares of the lane's rows */
                uint32_t seen = 0u;        /* every bit that a count of them has */
                if (exact && inB) {
                    const uint2* ref2 = reinterpret_cast<const uint2*>(refc);
#pragma unroll 4
                    for (uint32_t r = l; r < R; r += 32u) {
                        const uint2 s = *reinterpret_cast<const uint2*>(Tl + (r << 5));
                        const uint2 o = __ldg(ref2 + r);
                        const float dA = exact_diff_(s.x, o.x);
                        const float dB = exact_diff_(s.y, o.y);
                        a2A = __fadd_rn(a2A, __fmul_rn(dA, dA));
                        a2B = __fadd_rn(a2B, __fmul_rn(dB, dB));
                        if (F64 || SSD) {
                            iA += square_(s.x, o.x);
                            iB += square_(s.y, o.y);
                            seen |= s.x | s.y | o.x | o.y;
                        }
                    }
                } else if (exact) {
#pragma unroll 4
                    for (uint32_t r = l; r < R; r += 32u) {
                        const uint32_t s = Tl[r << 5], o = __ldg(refc + r);
                        const float dA = exact_diff_(s, o);
                        a2A = __fadd_rn(a2A, __fmul_rn(dA, dA));
                        if (F64 || SSD) {
                            iA += square_(s, o);
                            seen |= s | o;
                        }
                    }
                }
                if (F64 || SSD) exact = exact && seen < kExactBelow;
                if (!exact) {
                    a2A = a2B = 0.0f;
                    for (uint32_t r = l; r < R; r += 32u) {
                        if (inB) {
                            const uint2 s = *reinterpret_cast<const uint2*>(Tl + (r << 5));
                            const uint2 o = __ldg(reinterpret_cast<const uint2*>(refc) + r);
                            term_<F64, SSD>(s.x, o.x, a2A, a2dA, shi, slo);
                            term_<F64, SSD>(s.y, o.y, a2B, a2dB, shi, slo);
                        } else {
                            term_<F64, SSD>(Tl[r << 5], __ldg(refc + r), a2A, a2dA, shi, slo);
                        }
                    }
                }
                if (exact) {
                    if (F64) {
                        a2dA = (double)iA;
                        a2dB = (double)iB;
                    }
                    if (SSD) {
                        add128_(shi, slo, 0u, iA);
                        add128_(shi, slo, 0u, iB);
                    }
                }
                acc0 = __fadd_rn(acc0, a2A);
                if (F64) accd0 = __dadd_rn(accd0, a2dA);
                if (inB) {
                    acc1 = __fadd_rn(acc1, a2B);
                    if (F64) accd1 = __dadd_rn(accd1, a2dB);
                }
            }
        }
        /* this tile's generic accesses before its next box fill, which
         * follows the next strip's first barrier (with one tile, the
         * barrier before the refill below) */
        fence_proxy_async_();

        if (ok && c0 + 32u >= B) {
            /* last strip: reduce0 per logical warp (2w and 2w + 1), then over
             * the 32 totals */
            const float ws0 = reduce0_(acc0), ws1 = reduce0_(acc1);
            double wd0 = 0.0, wd1 = 0.0;
            if (F64) {
                wd0 = reduce0_(accd0);
                wd1 = reduce0_(accd1);
            }
            if (SSD) {
                for (uint32_t d = 16; d >= 1; d >>= 1) {
                    uint64_t ohi = __shfl_down_sync(0xFFFFFFFFu, shi, d);
                    uint64_t olo = __shfl_down_sync(0xFFFFFFFFu, slo, d);
                    if (l + d < 32u) add128_(shi, slo, ohi, olo);
                }
            }
            if (l == 0) {
                s_tot[2u * w] = ws0;
                s_tot[2u * w + 1u] = ws1;
                s_tot64[2u * w] = wd0;
                s_tot64[2u * w + 1u] = wd1;
                s_hi[2u * w] = shi;
                s_lo[2u * w] = slo;
                s_hi[2u * w + 1u] = 0u;
                s_lo[2u * w + 1u] = 0u;
            }
            __syncthreads();
            if (w == 0) {
                const float fin = reduce0_(s_tot[l]);
                double fin64 = 0.0;
                if (F64) fin64 = reduce0_(s_tot64[l]);
                uint64_t thi = s_hi[l], tlo = s_lo[l];
                if (SSD) {
                    for (uint32_t d = 16; d >= 1; d >>= 1) {
                        uint64_t ohi = __shfl_down_sync(0xFFFFFFFFu, thi, d);
                        uint64_t olo = __shfl_down_sync(0xFFFFFFFFu, tlo, d);
                        if (l + d < 32u) add128_(thi, tlo, ohi, olo);
                    }
                }
                if (l == 0) {
                    a.dist_f32[p] = fin;
                    if (F64 && a.dist_f64) a.dist_f64[p] = fin64;
                    if (SSD && a.ssd) {
                        a.ssd[2 * (uint64_t)p] = thi;
                        a.ssd[2 * (uint64_t)p + 1] = tlo;
                    }
                }
            }
            __syncthreads();
            acc0 = acc1 = 0.0f;
            accd0 = accd1 = 0.0;
            shi = slo = 0u;
        }
        if (!has_next) break;
        if (!db) {
            __syncthreads(); /* the one tile is free */
            strip_fill_(a, pn, cn, tiles, tid, &s_mbar[0]);
            pending |= 1u;
            cp_async_commit_();
        } else {
            cur ^= 1u;
        }
        p = pn;
        c0 = cn;
    }
    cp_async_wait_<0>();
    /* after a given-up wait: let the fills still in flight land (bounded) */
    for (uint32_t b = 0; b < 2u; ++b)
        if ((pending >> b) & 1u) mbar_wait_(&s_mbar[b], (parity >> b) & 1u);
    bulk_wait_all_(); /* the zero box stores have read the zero box before the CTA's shared memory goes */
}

static const size_t kStripSmemMax = 220u * 1024u;

/* 1024 bytes to align the tiles, one or two tiles, the zero box, the row
 * carries; for cluster launches two of each strip's last column and of its
 * 32 x 32 per-lane sums (with F64 also double ones) */
static size_t strip_smem_bytes(uint32_t max_rows, bool db, uint32_t cl, bool f64 = false)
{
    const size_t rows = strip_cap_rows(max_rows);
    size_t n = 1024u + (db ? 2u : 1u) * rows * 32u * sizeof(uint32_t) + kBoxBytes + rows * sizeof(uint32_t);
    if (cl > 1u) n += 2u * (rows * sizeof(uint32_t) + 32u * 32u * (sizeof(float) + (f64 ? sizeof(double) : 0u)));
    return n;
}

static bool use_strip(uint32_t max_rows, uint32_t cl) { return strip_smem_bytes(max_rows, false, cl) <= kStripSmemMax; }
static bool strip_db(uint32_t max_rows, uint32_t cl) { return strip_smem_bytes(max_rows, true, cl) <= kStripSmemMax; }

uint32_t distance_cluster_size(uint32_t max_rows, uint32_t max_bins)
{
    const uint32_t strips = (max_bins + 31u) / 32u;
    if (strips < 2u || strips > kMaxDistCluster) return 0u;
    return use_strip(max_rows, strips) ? strips : 0u;
}

size_t distance_smem_bytes(uint32_t max_rows, uint32_t cl)
{
    if (use_strip(max_rows, cl)) return strip_smem_bytes(max_rows, strip_db(max_rows, cl), cl);
    return ((size_t)max_rows + (size_t)kDistRowBlock * kPad) * sizeof(uint32_t);
}

uint32_t distance_block_threads(uint32_t max_rows) { return use_strip(max_rows, 0u) ? kStripThreads : 1024u; }

static const size_t kSmemPerSm = 228u * 1024u; /* of which 1 KB per resident CTA is not the CTA's */

/* From the launch bounds and shared memory: two strip CTAs where both fit
 * (5.25 KB each besides the dynamic part), one of the others.  (Asking the
 * driver took 3 us of a 50 us call, between its two launches.) */
int distance_ctas_per_sm(uint32_t max_rows, uint32_t cl)
{
    return use_strip(max_rows, cl) && 2u * (distance_smem_bytes(max_rows, cl) + 5376u) <= kSmemPerSm ? 2 : 1;
}

/* Clusters of cl CTAs of k_distance_cluster that fit at once with `smem`
 * bytes of shared memory each, on the current device; queried once per
 * (device, kernel, cl, smem), since the plain form launches per proposal. */
static cudaError_t cluster_fit_(void (*k)(DistArgs, uint32_t, uint32_t), cudaLaunchConfig_t& cfg, uint32_t cl, size_t smem,
                                int& fit)
{
    static std::mutex mu;
    static std::map<std::tuple<int, const void*, uint32_t, size_t>, int> cache;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const auto key = std::make_tuple(dev, (const void*)k, cl, smem);
    {
        std::lock_guard<std::mutex> g(mu);
        const auto it = cache.find(key);
        if (it != cache.end()) {
            fit = it->second;
            return cudaSuccess;
        }
    }
    e = cudaOccupancyMaxActiveClusters(&fit, (const void*)k, &cfg);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> g(mu);
    cache[key] = fit;
    return cudaSuccess;
}

/* Device-side set-up of a standalone distance launch: the descriptors of
 * `count` consecutive histograms sharing one job, and the observed
 * histogram's column-major copy (pairs of columns interleaved,
 * pcs_sat_t_index) through tiles of 16 rows x 32 columns in shared memory,
 * read in 128-byte rows and written in 128-byte runs of a pair (done cell by
 * cell on the host it took 0.4 ms for 1001 x 256).  Two cells per thread, and
 * the job and its map by a block of their own: a launch of few cells is a
 * chain of latencies (tiles of 32 x 64 took 5.5 us, a cell per thread written
 * one by one 3.8). */
constexpr uint32_t kPropWords = sizeof(PropDev) / 4u;

__global__ void __launch_bounds__(256) k_distance_setup(DistSetup d, const __grid_constant__ TmapDev map)
{
    __shared__ uint32_t s_t[16][33];
    const uint32_t tid = threadIdx.x, blocks = gridDim.x - 1u;
    const uint32_t R = d.rows, B = d.bins;
    if (blockIdx.x == blocks) { /* the last block */
        if (tid == 0u) {
            JobDev j;
            memset(&j, 0, sizeof j);
            j.R = R;
            j.B = B;
            j.ref_sat = d.ref;
            j.ref_sat_t = d.ref_t;
            j.tmap_depth = d.map_depth;
            *d.job = j;
            *d.n_props = d.count;
            if (d.err) *d.err = 0u;
        } else if (tid == 32u && d.map_depth) {
            *d.map = map;
            /* the map, for the tensor copies of the kernel that follows (which acquires it) */
            asm volatile("fence.proxy.tensormap::generic.release.gpu;\n" ::: "memory");
        }
        return;
    }
    /* the histograms' descriptors, word by word across the threads */
    for (uint64_t i = (uint64_t)blockIdx.x * 256u + tid; i < (uint64_t)d.count * kPropWords; i += (uint64_t)blocks * 256u) {
        const uint32_t q = (uint32_t)(i / kPropWords), k = (uint32_t)(i % kPropWords);
        const uint64_t off = (uint64_t)q * R * B;
        uint32_t v = 0u;
        if (k == offsetof(PropDev, hist_z) / 4u) v = q;
        if (k == offsetof(PropDev, hist_off) / 4u) v = (uint32_t)off;
        if (k == offsetof(PropDev, hist_off) / 4u + 1u) v = (uint32_t)(off >> 32);
        reinterpret_cast<uint32_t*>(d.props)[i] = v;
    }
    const uint32_t tc = (B + 31u) / 32u, tr = (R + 15u) / 16u;
    for (uint64_t t = blockIdx.x; t < (uint64_t)tc * tr; t += blocks) {
        const uint32_t r0 = (uint32_t)(t / tc) * 16u, c0 = (uint32_t)(t % tc) * 32u;
#pragma unroll
        for (uint32_t i = tid; i < 512u; i += 256u) {
            const uint32_t r = r0 + i / 32u, c = c0 + i % 32u;
            if (r < R && c < B) s_t[i / 32u][i % 32u] = d.ref[(uint64_t)r * B + c];
        }
        __syncthreads();
#pragma unroll
        for (uint32_t i = tid; i < 512u; i += 256u) {
            const uint32_t k = i % 32u, x = 2u * (i / 32u) + (k & 1u);
            const uint32_t r = r0 + k / 2u, c = c0 + x;
            if (r < R && c < B) d.ref_t[pcs_sat_t_index(r, c, R, B)] = s_t[k / 2u][x];
        }
        __syncthreads();
    }
}

cudaError_t launch_distance_setup(const DistSetup& d, const TmapDev& map, cudaStream_t st)
{
    const uint64_t tiles = (uint64_t)((d.bins + 31u) / 32u) * ((d.rows + 15u) / 16u);
    const uint64_t blocks = std::max<uint64_t>(tiles, ((uint64_t)d.count * kPropWords + 1023u) / 1024u);
    k_distance_setup<<<(unsigned)std::min<uint64_t>(blocks, 4096u) + 1u, 256, 0, st>>>(d, map);
    return cudaGetLastError();
}

/* Rows or strips.  The row kernel takes one walk down the rows (10 us + 90 ns
 * per row) for any number of columns and histograms until its warps fill the
 * SMs; the strip kernels take 2.2 us + 9.5 ns per row for every strip (or
 * cluster's histogram) that a CTA (cluster slot) has in turn.  The lines
 * cross at 5 turns for 33 rows, 7 for 201 and 8.5 for 1001.  Measured, strips
 * -> rows in us: 4 turns (201 x 100 x 213) 21.9 -> 24.5, 8 turns (201 x 100 x
 * 608) 40.9 -> 27.1 and (201 x 256 x 100) 33.3 -> 26.4, 32 turns (201 x 1000
 * x 152) 122 -> 52; clusters at 6 turns (1001 x 256 x 76) 83 -> 102, at 8
 * (x 120) 115 -> 104, at 21 (x 304) 281 -> 131; 16 turns (301 x 128 x 1024)
 * 89.6 -> 51.1.
 * With double sums the walk zeroes in a second pass and a launch for the
 * histograms left over follows: 8 turns (1001 x 256 x 152) 114 -> 138, 16
 * (x 304) 228 -> 166, 32 (201 x 1000 x 20) 126 -> 63.
 * Where rows are not 16-byte aligned (in a round of several jobs: the widest
 * one's, which has the most of the work) the lanes copy cell by cell: 8 turns
 * (201 x 255 x 100) 39.4 -> 43, 12 (201 x 99 x 912) 75.9 -> 57.8, 32 (201 x
 * 999 x 38) 145 -> 90; and a warp has to replace three strips: with one (51 x
 * 31 x 3000) 44.6 -> 57, with two (329 x 49 x 2036, whole calls) 203 -> 235.
 * Histograms too tall for a strip in shared memory (above 1664 rows), whose
 * kernel works through blocks of rows: 2 turns (1800 x 40 x 2) 154 -> 157,
 * 4 (x 200) 836 -> 146, 16 (1800 x 256 x 200) 5409 -> 195. */
static bool use_rows_(const DistArgs& a, uint32_t turns)
{
    uint32_t from = 8u;
    if (a.dist_f64) from += 4u;
    if (a.max_bins & 3u) from += 4u;
    const bool strips = use_strip(a.max_rows, 0u);
    if (!strips) from = 3u;
    if (strips && (a.max_bins & 3u) != 0u && (a.max_bins + 31u) / 32u < 3u * ((a.max_bins + 127u) / 128u)) return false;
    if (strips && a.mostly_narrow) return false;
    return a.max_bins <= 128u * kRowsWarps && turns >= from;
}

/* CTAs of the row kernel that fit on an SM */
static uint32_t rows_per_sm_(uint32_t max_bins)
{
    const size_t smem = (size_t)((max_bins + 127u) / 128u) * kRowsWarpBytes;
    return std::max<uint32_t>(1u, (uint32_t)(kSmemPerSm / (smem + 2048u)));
}

/* A round of several jobs: every CTA of the row kernel has the warps that the
 * widest job needs, and a narrow histogram takes one of them for as long as a
 * wide one, where strips take turns by each histogram's own width.  The lines
 * cross at 12 strips on average where one CTA fits on an SM, 6 where two do, 4
 * where three do (for 61 rows at 6.4, 3.2 and 2.1).
 * Served jobs of 256 bins (three CTAs fit), 400 (two) and 1024 (one) beside
 * narrow ones, distance time of all rounds, strips -> rows in ms, 201 rows: 256,
 * 64, 64, 64 (3.5 strips) 2.85 -> 3.29, 256, 64, 64 (4) 2.35 -> 2.31, 256, 256,
 * 64, 64 (5) 3.41 -> 2.87; 320, 128, 128, 64 (5) 3.48 -> 3.86, 320, 320, 64, 64
 * (6) 4.26 -> 4.08; 1024, 64, 64, 64 (9.5) 8.50 -> 10.3, 1024, 256, 128, 64
 * (11.5) 8.72 -> 8.73, 1024, 512, 256, 128 (15) 10.4 -> 8.8; 61 rows: 1024 and
 * seven of 33 (5.75) 4.50 -> 5.46, 320, 32, 32 (4) 1.93 -> 1.52; 451 rows: 320,
 * 128, 128, 64 (5) 4.05 -> 4.13, 1024, 256, 128, 64 9.9 -> 9.6. */
bool distance_mostly_narrow(uint32_t max_rows, uint32_t max_bins, uint32_t strips16)
{
    const uint32_t line = std::min(12u, 4u + max_rows / 25u);
    return strips16 * rows_per_sm_(max_bins) < 16u * line;
}

static cudaError_t launch_rows_(const DistArgs& a, uint32_t sms, cudaStream_t st)
{
    void (*k)(DistArgs);
    if (a.dist_f64) k = a.ssd ? k_distance_rows<true, true> : k_distance_rows<true, false>;
    else k = a.ssd ? k_distance_rows<false, true> : k_distance_rows<false, false>;
    const cudaError_t e = allow_smem(k, kRowsWarps * kRowsWarpBytes);
    if (e != cudaSuccess) return e;
    const uint32_t warps = (a.max_bins + 127u) / 128u;
    const size_t smem = (size_t)warps * kRowsWarpBytes;
    k<<<std::min(a.max_count, rows_per_sm_(a.max_bins) * sms), 32u * warps, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_distance(const DistArgs& a, uint32_t grid, cudaStream_t st, uint32_t cl, uint32_t* launched)
{
    /* a caller that leaves these unset would get some kernel, but not the one that suits it */
    if (!a.max_rows || !a.max_bins || !a.max_count) return cudaErrorInvalidValue;
    int dev = 0, n_sm = 0;
    cudaError_t e0 = cudaGetDevice(&dev);
    if (e0 == cudaSuccess) e0 = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    if (e0 != cudaSuccess) return e0;
    const uint32_t sms = (uint32_t)n_sm, strips = (a.max_bins + 31u) / 32u;
    const size_t smem = distance_smem_bytes(a.max_rows, 0u);
    if (smem > 227u * 1024u) return cudaErrorInvalidValue;
    const uint32_t count = std::max(1u, a.min_count);
    const uint32_t slots = sms * (uint32_t)distance_ctas_per_sm(a.max_rows, 0u);
    uint32_t turns = strips * ((count + slots - 1u) / slots);

    const bool f64 = a.dist_f64 != nullptr;
    const size_t csmem1 = strip_smem_bytes(a.max_rows, false, cl, f64), csmem2 = strip_smem_bytes(a.max_rows, true, cl, f64);
    if (a.strips_only || cl > kMaxDistCluster || csmem1 > kStripSmemMax) cl = 0u;
    const bool tall = strip_cap_rows(a.max_rows) >= kClusterRowsMin;
    if (cl > 1u && !tall && grid > 2u * sms / cl) cl = 0u; /* more histograms than clusters ever fit */
    const bool two = csmem2 <= kStripSmemMax;
    void (*kcl)(DistArgs, uint32_t, uint32_t);
    if (f64) kcl = a.ssd ? k_distance_cluster<true, true> : k_distance_cluster<true, false>;
    else kcl = a.ssd ? k_distance_cluster<false, true> : k_distance_cluster<false, false>;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    int fit = 0; /* clusters that fit at once */
    if (cl > 1u) {
        const cudaError_t e = allow_smem(kcl, kStripSmemMax);
        if (e != cudaSuccess) return e;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cl;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.blockDim = dim3(kStripThreads);
        cfg.dynamicSmemBytes = two ? csmem2 : csmem1;
        cfg.stream = st;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cfg.gridDim = dim3(cl);
        const cudaError_t f = cluster_fit_(kcl, cfg, cl, cfg.dynamicSmemBytes, fit);
        if (f != cudaSuccess) return f;
    }
    /* clusters of cl CTAs where the histograms are tall, or where every histogram of
     * the launch has a cluster to itself, if that takes clearly fewer turns than
     * strips by single CTAs do.  A turn is a strip's time, 2.2 us + 9.5 ns per row
     * (see use_rows_), that is (230 + rows) x 9.5 ns, and with clusters a fifth more,
     * hence the 6 to 5 (152 of 1001 x 256 with double sums 178 us in 11 turns of
     * clusters, 114 in 8 of strips; 152 of 601 x 128 34 in 4 of strips, 120 of them 41
     * in 4 of clusters; 476 of 645 x 63, whole calls, 150 in 7 of clusters, 142 in 8
     * of strips); and the turns saved have to be more than a cluster launch's own 3.5
     * us, with a margin 400 x 9.5 ns (kernel alone, strips and clusters: 108 of 107 x
     * 61 11.5 and 12.9 us, 71 of 153 x 34 11.3 and 11.7, 5 of 261 x 48 14.5 and 12.1);
     * as many clusters as fit at once, at most one per histogram slot */
    const uint32_t cturns = fit > 0 ? (count + (uint32_t)fit - 1u) / (uint32_t)fit : 0u;
    const bool clusters = fit > 0 && (tall || grid <= (uint32_t)fit) && 6u * cturns < 5u * turns &&
                          (turns - cturns) * (230u + a.max_rows) > 400u;
    if (clusters) turns = cturns;
    const bool rows = !a.strips_only && use_rows_(a, turns);
    if (launched) *launched = rows && f64 ? 2u : 1u;
    last_kernel(kFamilyDistance) = rows                        ? "k_distance_rows"
                                   : clusters                  ? "k_distance_cluster"
                                   : use_strip(a.max_rows, 0u) ? "k_distance_strip"
                                                               : "k_distance";
    if (rows) {
        const cudaError_t e = launch_rows_(a, sms, st);
        if (e != cudaSuccess || !f64) return e;
    } else if (clusters) {
        cfg.gridDim = dim3(std::min<uint32_t>(grid, (uint32_t)fit) * cl);
        return cudaLaunchKernelEx(&cfg, kcl, a, two ? 1u : 0u, cl);
    }
    if (use_strip(a.max_rows, 0u)) {
        void (*k)(DistArgs, uint32_t);
        if (rows) k = a.ssd ? k_distance_strip<true, true, true> : k_distance_strip<true, false, true>;
        else if (f64) k = a.ssd ? k_distance_strip<true, true, false> : k_distance_strip<true, false, false>;
        else k = a.ssd ? k_distance_strip<false, true, false> : k_distance_strip<false, false, false>;
        cudaError_t e = allow_smem(k, kStripSmemMax);
        if (e != cudaSuccess) return e;
        k<<<grid, kStripThreads, smem, st>>>(a, strip_db(a.max_rows, 0u) ? 1u : 0u);
        return cudaGetLastError();
    }
    if (a.dist_f64) {
        cudaError_t e = allow_smem(k_distance<true>, kDynSmemMax);
        if (e != cudaSuccess) return e;
        k_distance<true><<<grid, 1024, smem, st>>>(a, rows ? 1u : 0u);
    } else {
        cudaError_t e = allow_smem(k_distance<false>, kDynSmemMax + 256u);
        if (e != cudaSuccess) return e;
        k_distance<false><<<grid, 1024, smem, st>>>(a, 0u);
    }
    return cudaGetLastError();
}

} // namespace pcs
