/*
 * kernels_sim.cu -- the fused forward model: simulate + summarise.
 *
 * One persistent launch walks the particles of every proposal in a round
 * (cusim::K_simulate_system, src/gpu/cusim/kernel-simulate.inl:106-185, and
 * its unrolled twin kernel-simulate-unroll.inl:69-298, do one proposal per
 * launch with one warp per video).  Work items are (proposal, range of
 * particles) pulled from a device counter, so proposals with uneven Poisson
 * particle counts pack densely onto all SMs.  Per particle the walk state
 * lives in registers.  k_simulate_walk, the default, records tracks by global
 * atomics and screens out the particles that are never detected;
 * k_simulate_few spreads the particles of small standalone calls over four or
 * eight lanes each; k_simulate (a tile of histogram rows privatised in shared
 * memory, several walkers per thread, replayed draws) walks an item per CTA,
 * and k_simulate_split is the slab-split walk.
 *
 * Arithmetic contract: the walk, DE and binning use explicit round-to-nearest
 * intrinsics (__fmul_rn/__fadd_rn/__fdiv_rn) in the reference's evaluation
 * order, so given the same draws the histogram is bit-exact with the
 * reference kernel built without FMA contraction.
 *
 * Random draws: Philox4x32-10, counter (particle, tag|block, slot,
 * generation|trial) with the job seed folded into words 2 and 3; the rounds'
 * work on the words that stay fixed for a particle is done once per particle
 * (pcs_philox_prepare); block 0 = position and
 * component, block 1 = size, blocks 2+3g..4+3g = the 12 normals of walk steps
 * 4g+1..4g+4 (Box-Muller on word pairs).  In replay mode the same kernel
 * reads pre-generated draws instead.
 */
#include <cuda_runtime.h>

#include <algorithm>

#include "pcs_common.h"
#include "pcs_kernels.h"

namespace pcs {

namespace {

__device__ __forceinline__ float wrap_(float v, float m, float two_m)
{
    /* periodic_bounds_ (kernel-simulate.inl:95-103): one wrap, v -= 2 copysign(m, v) */
    return (fabsf(v) > m) ? __fsub_rn(v, copysignf(two_m, v)) : v;
}

/* The three wraps of one step.  A step is much shorter than the box, so a
 * wrap is rare: one combined test skips the three selects on the common
 * path (same values as three wrap_ calls). */
__device__ __forceinline__ void wrap3_(float& x, float& y, float& z, float hx, float hy, float hz)
{
    if (__builtin_expect(fabsf(x) > hx || fabsf(y) > hy || fabsf(z) > hz, 0)) {
        x = wrap_(x, hx, 2.0f * hx);
        y = wrap_(y, hy, 2.0f * hy);
        z = wrap_(z, hz, 2.0f * hz);
    }
}

/* The PTX approximate instructions in their flush-to-zero forms.  Box-Muller
 * never gives them a subnormal operand (u >= 2^-33; -2 ln u is 0 or above
 * 5e-8; the angle is 0 or above 1e-7 in magnitude), so they return what the
 * non-flushing forms (__log2f, __sincosf in a build without -ftz) return,
 * without the subnormal handling those carry: ~10% fewer instructions per
 * particle-step for the same normals. */
__device__ __forceinline__ float lg2_ftz_(float x)
{
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float sqrt_ftz_(float x)
{
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float sin_ftz_(float x)
{
    float y;
    asm("sin.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float cos_ftz_(float x)
{
    float y;
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

const float kSqrt2Ln2 = 1.1774100225154747f; /* sqrt(2 ln 2): sqrt(-2 ln u) = sqrt(2 ln 2) sqrt(-log2 u) */

/* Box-Muller on two 32-bit words: u1 in (0,1], angle uniform on [-pi, pi);
 * both normals times scale = rscale / sqrt(2 ln 2).  The radius is
 * rscale sqrt(-log2 u): a caller that scales every pair by the same factor
 * (the walk: its particle's step sd, so its steps take the normals as they
 * are) folds sqrt(2 ln 2) into it once, one multiply per pair fewer. */
__device__ __forceinline__ void box_muller_r_(uint32_t ra, uint32_t rb, float& n0, float& n1, float rscale)
{
    float u = __fmaf_rn(__uint2float_rn(ra), 2.3283064365386963e-10f, 1.1641532182693481e-10f);
    float rad = rscale * sqrt_ftz_(-lg2_ftz_(u));
    float t = __fmaf_rn(__uint2float_rn(rb), 1.4629180792671596e-09f, -3.14159265358979f);
    n0 = rad * sin_ftz_(t);
    n1 = rad * cos_ftz_(t);
}

/* unit normals */
__device__ __forceinline__ void box_muller_(uint32_t ra, uint32_t rb, float& n0, float& n1)
{
    box_muller_r_(ra, rb, n0, n1, kSqrt2Ln2);
}

struct Walker {
    float x, y, z, de, sd, haz; /* sd: the step sd, or (fresh-draw walk) sd x sqrt(2 ln 2) for box_muller_r_ */
    uint32_t k, F, n;  /* n: particle index within the proposal */
    pcs_philox_pre ph; /* the particle's stream with its fixed counter words folded in */
};

struct ItemCtx {
    float hlx, hly, hlz, two_hlx, two_hly, two_hlz, hax, hay, four_dt, dde;
    uint32_t kmin, B, RB, tile_words_used, tile_rows;
    uint32_t* hist; /* global histogram of the proposal */
    uint32_t* err;
};

/* HistogramRecorder::record (histogram2d.inl:313-321) into the privatised
 * tile or the global histogram. */
template <bool AGG>
__device__ __noinline__ void record_out_(float four_dt, float dde, uint32_t B, uint32_t RB,
                                         uint32_t tile_rows, uint32_t* hist, uint32_t* err,
                                         uint32_t* tile, uint32_t k, float de)
{
    float denom = __fmul_rn(__uint2float_rn(k - 1u), four_dt);
    float DE = __fdiv_rn(de, denom);
    float q = __fdiv_rn(DE, dde);
    uint32_t bin = __float2uint_rz(q); /* tCount(aDE / mDDE): truncating, saturating, NaN -> 0 */
    if (bin >= B) return;
    uint64_t idx = (uint64_t)k * B + bin;
    if (idx >= RB) {
        atomicOr(err, PCS_ERRBIT_HIST_BOUNDS);
        return;
    }
    if (k < tile_rows) {
        if (AGG) {
            unsigned mask = __activemask();
            unsigned peers = __match_any_sync(mask, (unsigned)idx);
            int leader = __ffs(peers) - 1;
            if ((int)(threadIdx.x & 31u) == leader) atomicAdd(&tile[idx], (uint32_t)__popc(peers));
        } else {
            atomicAdd(&tile[idx], 1u);
        }
    } else {
        atomicAdd(&hist[idx], 1u);
    }
}

template <bool AGG>
__device__ __forceinline__ void record_(const ItemCtx& c, uint32_t* tile, uint32_t k, float de)
{
    record_out_<AGG>(c.four_dt, c.dde, c.B, c.RB, c.tile_rows, c.hist, c.err, tile, k, de);
}

/* Where a walk's tracks go: the item's tile (and the histogram past it). */
template <bool AGG>
struct TileSink {
    uint32_t* tile;
    __device__ __forceinline__ void record(const ItemCtx& c, uint32_t k, float de) const { record_<AGG>(c, tile, k, de); }
};

/* One frame of the walk.  CHECK: the frame may lie past the particle's
 * last one (s >= F) and is then skipped; full groups of four frames call it
 * without the test.  SCALED: the normals already carry the step sd (fresh
 * Philox draws); replayed normals are unit normals, scaled here as the
 * reference scales them. */
template <class SINK, bool CHECK = true, bool SCALED = false>
__device__ __forceinline__ void step_(const ItemCtx& c, const SINK& sink, Walker& w, uint32_t s,
                                      float n0, float n1, float n2)
{
    if (CHECK && s >= w.F) return;
    float dx = SCALED ? n0 : __fmul_rn(w.sd, n0);
    float dy = SCALED ? n1 : __fmul_rn(w.sd, n1);
    float dz = SCALED ? n2 : __fmul_rn(w.sd, n2);
    w.x = __fadd_rn(w.x, dx);
    w.y = __fadd_rn(w.y, dy);
    w.z = __fadd_rn(w.z, dz);
    wrap3_(w.x, w.y, w.z, c.hlx, c.hly, c.hlz);
    /* kernel-simulate.inl:70-93: a detected step extends the track (DE from
     * its second frame on), an undetected one closes it (recorded if K >=
     * kmin).  (Updating the track state by selects instead keeps all lanes
     * together but executes ~6% more instructions: no faster.) */
    bool det = fabsf(w.z) <= w.haz && fabsf(w.x) <= c.hax && fabsf(w.y) <= c.hay;
    if (det) {
        uint32_t kp = w.k + 1u;
        if (kp >= 2u) w.de = __fadd_rn(w.de, __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)));
        w.k = kp;
    } else {
        if (w.k >= c.kmin) sink.record(c, w.k, w.de);
        w.k = 0u;
        w.de = 0.0f;
    }
}

/* wrand_index (utility.inl:8-57). */
__device__ __forceinline__ uint32_t wrand_index_(float u, uint32_t C, const float* pre)
{
    if (C == 2u) return (pre[0] >= u) ? 0u : 1u;
    uint32_t bot = 0, top = C;
    while (bot != top) {
        uint32_t mid = (top + bot) >> 1;
        if (pre[mid] <= u)
            bot = mid + 1u;
        else
            top = mid;
    }
    return bot;
}

__device__ __forceinline__ uint32_t video_of_(const uint32_t* prefix, uint32_t V, uint32_t n)
{
    /* largest v with prefix[v] <= n (prefix[0] = 0, prefix[V] = total) */
    uint32_t lo = 0, hi = V;
    while (hi - lo > 1u) {
        uint32_t mid = (lo + hi) >> 1;
        if (__ldg(prefix + mid) <= n)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

/* Item context of proposal s_prop (of job s_job). */
__device__ __forceinline__ ItemCtx item_ctx_(const SimArgs& a, const JobDev& s_job, const PropDev& s_prop)
{
    ItemCtx c;
    c.hlx = s_job.half_lx;
    c.hly = s_job.half_ly;
    c.hlz = s_job.half_lz;
    c.two_hlx = 2.0f * s_job.half_lx;
    c.two_hly = 2.0f * s_job.half_ly;
    c.two_hlz = 2.0f * s_job.half_lz;
    c.hax = s_job.half_ax;
    c.hay = s_job.half_ay;
    c.four_dt = s_job.four_delta_t;
    c.dde = s_job.dde;
    c.kmin = s_job.kmin;
    c.B = s_job.B;
    c.RB = s_job.R * s_job.B;
    c.tile_rows = min(s_job.R, a.tile_words / max(s_job.B, 1u));
    c.tile_words_used = c.tile_rows * s_job.B;
    c.hist = a.hist + s_prop.hist_off;
    c.err = a.err;
    return c;
}

/* Loads work item `item`'s proposal and job blocks into shared memory. */
__device__ __forceinline__ void load_item_(const SimArgs& a, uint32_t item, PropDev& s_prop, JobDev& s_job)
{
    const uint32_t tid = threadIdx.x;
    const uint32_t p = a.item_prop[item];
    if (tid < sizeof(PropDev) / 4) reinterpret_cast<uint32_t*>(&s_prop)[tid] = reinterpret_cast<const uint32_t*>(a.props + p)[tid];
    __syncthreads();
    if (tid < sizeof(JobDev) / 4) reinterpret_cast<uint32_t*>(&s_job)[tid] = reinterpret_cast<const uint32_t*>(a.jobs + s_prop.job)[tid];
    __syncthreads();
}

/* Initial state of particle n (make_particle, utility.inl:60-99, and the
 * particle's step sd): position, component, half depth, step sd, K.
 * BM_SD: q.sd carries sd x sqrt(2 ln 2), the scale box_muller_r_ takes. */
template <bool REPLAY, bool BM_SD = false>
__device__ __forceinline__ void init_walker_(const SimArgs& a, const ItemCtx& c, const JobDev& s_job,
                                             const PropDev& s_prop, const uint32_t* prefix, uint32_t n,
                                             uint32_t slot, uint32_t gt, uint32_t k0, uint32_t k1, Walker& q)
{
    const uint32_t V = s_job.V, C = s_job.C, model = s_job.model;
    const uint32_t v = video_of_(prefix, V, n);
    q.F = __ldg(s_job.frames + v);
    float u0, u1, u2, u3;
    if (REPLAY) {
        const float* u = a.rp_uniforms + 4ull * n;
        u0 = u[0];
        u1 = u[1];
        u2 = u[2];
        u3 = u[3];
    } else {
        q.ph = pcs_philox_prepare(n, slot, gt, k0, k1);
        pcs_u4 r = pcs_draw_pre(q.ph, pcs_ctr_tag(PCS_STREAM_PARTICLE, 0u));
        u0 = pcs_u01_24(r.x);
        u1 = pcs_u01_24(r.y);
        u2 = pcs_u01_24(r.z);
        u3 = pcs_u01_24(r.w);
    }
    /* make_particle (utility.inl:60-99): halfL * (2u - 1) */
    q.x = __fmul_rn(c.hlx, __fsub_rn(2.0f * u0, 1.0f));
    q.y = __fmul_rn(c.hly, __fsub_rn(2.0f * u1, 1.0f));
    q.z = __fmul_rn(c.hlz, __fsub_rn(2.0f * u2, 1.0f));
    uint32_t comp = (C > 1u) ? wrand_index_(u3, C, s_prop.pre_comp_prob) : 0u;
    if (comp >= C) {
        atomicOr(a.err, PCS_ERRBIT_COMPONENT);
        comp = C - 1u;
    }
    q.haz = (model == PCS_DEV_MODEL_VARIABLE_Z) ? s_prop.half_az[comp] : s_prop.half_az[0];
    if (model == PCS_DEV_MODEL_LOGNORMAL) {
        if (REPLAY) {
            q.sd = a.rp_sigmas[n];
        } else {
            pcs_u4 r = pcs_draw_pre(q.ph, pcs_ctr_tag(PCS_STREAM_PARTICLE, 1u));
            float z0, z1;
            box_muller_(r.x, r.y, z0, z1);
            q.sd = s_prop.sd_scale[comp] * expf(s_prop.sd_shape[comp] * z0);
        }
    } else {
        q.sd = s_prop.sd_scale[comp];
    }
    if (BM_SD) q.sd = __fmul_rn(q.sd, kSqrt2Ln2);
    const bool det = fabsf(q.z) <= q.haz && fabsf(q.x) <= c.hax && fabsf(q.y) <= c.hay;
    q.k = det ? 1u : 0u;
}

/* The 12 normals of the group of frames s0 .. s0+3: Philox blocks
 * 2+3g .. 4+3g through Box-Muller, times the particle's step sd (q.sd holds
 * sd x sqrt(2 ln 2) on this path); or the replayed unit normals (zeros past
 * F). */
template <bool REPLAY>
__device__ __forceinline__ void group_normals_(const SimArgs& a, const Walker& q, uint32_t s0, float* nn)
{
    if (REPLAY) {
        const float* src = a.rp_normals + ((uint64_t)q.n * a.rp_stride + (s0 - 1u)) * 3u;
        const uint32_t rem = min(4u, q.F - s0);
#pragma unroll
        for (int t = 0; t < 12; ++t) nn[t] = ((uint32_t)t < rem * 3u) ? src[t] : 0.0f;
    } else {
        const uint32_t g = (s0 - 1u) >> 2;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            pcs_u4 r = pcs_draw_pre(q.ph, pcs_ctr_tag(PCS_STREAM_PARTICLE, 2u + 3u * g + (uint32_t)b));
            box_muller_r_(r.x, r.y, nn[4 * b + 0], nn[4 * b + 1], q.sd);
            box_muller_r_(r.z, r.w, nn[4 * b + 2], nn[4 * b + 3], q.sd);
        }
    }
}

/* Frames 1 .. F-1 of one walker, four per group: the full groups skip the
 * per-frame end test, the tail group keeps it. */
template <bool REPLAY, class SINK>
__device__ __forceinline__ void walk_single_(const SimArgs& a, const ItemCtx& c, const SINK& sink, Walker& q)
{
    uint32_t s0 = 1;
    for (; s0 + 3u < q.F; s0 += 4u) {
        float nn[12];
        group_normals_<REPLAY>(a, q, s0, nn);
        step_<SINK, false, !REPLAY>(c, sink, q, s0 + 0u, nn[0], nn[1], nn[2]);
        step_<SINK, false, !REPLAY>(c, sink, q, s0 + 1u, nn[3], nn[4], nn[5]);
        step_<SINK, false, !REPLAY>(c, sink, q, s0 + 2u, nn[6], nn[7], nn[8]);
        step_<SINK, false, !REPLAY>(c, sink, q, s0 + 3u, nn[9], nn[10], nn[11]);
    }
    if (s0 < q.F) {
        float nn[12];
        group_normals_<REPLAY>(a, q, s0, nn);
        step_<SINK, true, !REPLAY>(c, sink, q, s0 + 0u, nn[0], nn[1], nn[2]);
        step_<SINK, true, !REPLAY>(c, sink, q, s0 + 1u, nn[3], nn[4], nn[5]);
        step_<SINK, true, !REPLAY>(c, sink, q, s0 + 2u, nn[6], nn[7], nn[8]);
        step_<SINK, true, !REPLAY>(c, sink, q, s0 + 3u, nn[9], nn[10], nn[11]);
    }
}

} // namespace

/* Launch bound by walkers per thread: one walker keeps 64 registers for
 * 1024-thread CTAs; 2, 4 and 8 interleaved walkers get 128 (512 threads) and
 * 255 (256 threads) registers, so their walk state stays out of local
 * memory. */
template <int PPT, bool REPLAY, bool AGG>
__global__ void __launch_bounds__(sim_max_block(PPT)) k_simulate(SimArgs a)
{
    extern __shared__ uint32_t s_tile[];
    __shared__ uint32_t s_item;
    __shared__ PropDev s_prop;
    __shared__ JobDev s_job;

    const uint32_t tid = threadIdx.x, bd = blockDim.x;
    for (uint32_t i = tid; i < a.tile_words; i += bd) s_tile[i] = 0u;
    const uint32_t n_items = *a.n_items;

    for (;;) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(a.queue_head, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= n_items) break;
        load_item_(a, item, s_prop, s_job);
        const ItemCtx c = item_ctx_(a, s_job, s_prop);
        const TileSink<AGG> sink = {s_tile};

        const uint32_t V = s_job.V;
        const uint32_t* prefix = a.counts + s_prop.counts_off + V; /* [V+1] */
        const uint32_t k0 = s_job.seed_lo, k1 = s_job.seed_hi;
        const uint32_t slot = s_prop.slot;
        const uint32_t gt = pcs_ctr_gen_trial(s_prop.gen, s_prop.trial);

        const uint32_t chunk_idx = item - s_prop.item_begin;
        const uint32_t a0 = chunk_idx * a.chunk;
        const uint32_t a1 = min(a0 + a.chunk, s_prop.total_particles);

        for (uint32_t base = a0; base < a1; base += bd * PPT) {
            Walker w[PPT];
            uint32_t fmax = 0;
#pragma unroll
            for (int j = 0; j < PPT; ++j) {
                const uint32_t n = base + tid + (uint32_t)j * bd;
                Walker& q = w[j];
                q.n = n;
                q.F = 0;
                q.k = 0;
                q.de = 0.0f;
                q.x = q.y = q.z = 0.0f;
                q.sd = 0.0f;
                q.haz = 0.0f;
                if (n < a1) {
                    init_walker_<REPLAY, !REPLAY>(a, c, s_job, s_prop, prefix, n, slot, gt, k0, k1, q);
                    fmax = max(fmax, q.F);
                }
            }

            /* frames 1 .. F-1, four per group; one walker per thread: the
             * full groups skip the per-frame end test, the tail group keeps it */
            if (PPT == 1) {
                walk_single_<REPLAY>(a, c, sink, w[0]);
            } else
            for (uint32_t s0 = 1; s0 < fmax; s0 += 4u) {
#pragma unroll
                for (int j = 0; j < PPT; ++j) {
                    Walker& q = w[j];
                    if (s0 >= q.F) continue;
                    float nn[12];
                    group_normals_<REPLAY>(a, q, s0, nn);
                    step_<TileSink<AGG>, true, !REPLAY>(c, sink, q, s0 + 0u, nn[0], nn[1], nn[2]);
                    step_<TileSink<AGG>, true, !REPLAY>(c, sink, q, s0 + 1u, nn[3], nn[4], nn[5]);
                    step_<TileSink<AGG>, true, !REPLAY>(c, sink, q, s0 + 2u, nn[6], nn[7], nn[8]);
                    step_<TileSink<AGG>, true, !REPLAY>(c, sink, q, s0 + 3u, nn[9], nn[10], nn[11]);
                }
            }
#pragma unroll
            for (int j = 0; j < PPT; ++j) {
                if (w[j].F > 0u && w[j].k >= c.kmin) record_<AGG>(c, s_tile, w[j].k, w[j].de);
            }
        }

        __syncthreads();
        /* flush the privatised rows into the proposal's histogram */
        for (uint32_t i = tid; i < c.tile_words_used; i += bd) {
            const uint32_t v = s_tile[i];
            if (v) {
                atomicAdd(c.hist + i, v);
                s_tile[i] = 0u;
            }
        }
    }
}

/* ----------------------------------------------------------------------- */
/* The walk without a shared-memory histogram tile (k_simulate_walk).
 *
 * Every record is a global atomic, so nothing ties a CTA's warps to one work
 * item: each warp takes 32-particle slices of the items from the device
 * queue (slice s is part s % slices of item s / slices).
 *
 * Screening.  A particle is recorded only if some frame finds all three
 * coordinates in the detection region, which is a tenth of the box's depth
 * and a quarter of its area in the benchmark configurations: most particles
 * of a video are never detected, and nothing of their walk reaches the
 * histogram.  So a particle that starts far enough from the region along one
 * coordinate is first walked along that coordinate alone, unwrapped: if it
 * provably stays outside the region's images all along, it is done.  This
 * costs the same Philox draws as the walk (a coordinate's normals lie in all
 * three blocks of a group) but a third of the Box-Muller trigonometry, no
 * wraps, no detection tests and no divergence.  A particle that comes too
 * near is walked in full from its start, as are those that start too near:
 * the histogram is the same, count for count.
 *
 * The screen walk's sums differ from the walk's own positions by rounding
 * only.  With k = sd sqrt(2 ln 2) and the box half length h (6k <= h is
 * required), per step: the trigonometric approximations and their arguments
 * differ by less than 6e-5 (their documented error is far smaller), times
 * the largest radius sqrt(33) k; the products' roundings, 7e-7 k; the
 * position's additions and wraps, below 4 (h + 6k) 2^-24; the sum's own
 * addition, below 2h 2^-24 while the particle is inside the interval.
 * screen_margin_ bounds their total by 4e-4 k + 1e-6 h per frame, and the
 * interval is narrowed by it on both sides.
 *
 * Screened and full walks go to full warps through a queue per CTA (entries
 * (proposal, particle), guarded by a lock that is held for ~100 cycles): a
 * warp takes 32 candidates to screen if there are as many, else 32 full
 * walks, else a new slice, whose particles it sorts into the queue -- or
 * walks at once where none is a candidate.  What is left in the queue at the
 * end is walked in full.  The lock is taken only to add or where there is
 * something to take (short videos of 31 frames, which are never sorted, lost
 * 5% to it; configuration 0's rounds 2%).
 *
 * Measured (forward model alone, before -> after): 1e10 particle-steps of
 * configuration 3 in one proposal 28.1 -> 21.5 ms; configuration 1, prior
 * pass and three generations (5.6e10 particle-steps) 158 -> 120 ms;
 * configuration 0, a whole job's 66 short rounds 24.7 -> 20.3 ms.  The bound
 * is the FMA-heavy pipe, where a Philox round's 32 x 32 -> 64 bit product
 * takes four cycles: 48 products a group, 192 of the ~440 cycles per warp
 * and group of a full walk and of the ~290 of a screen walk. */

constexpr uint32_t kScreenQueue = 96;     /* entries of each queue: at most 62 stay between visits, 32 more during one */
constexpr uint32_t kLockLimit = 1u << 22; /* tries before a wait for the queue's lock is given up */
/* What is screened, and where.  A screen walk costs about 0.65 of a walk, so
 * a particle is a candidate where it is likely to pass: its distance to the
 * region is above kScreenSigmas standard deviations of its whole walk (0.7,
 * 0.9, 1.1, 1.2 and 1.5 were timed; 1.1 and 1.2 are best, and flat).  Videos
 * shorter than kScreenMinFrames are walked at once: sorting and starting
 * their particles twice would weigh too much.  A launch of fewer than
 * kScreenSlices slices per warp is over after a walk or two, which screening
 * first would only lengthen; and the last slices, one for
 * every kScreenTail-th warp, are walked at once so that no screened particle
 * starts its full walk when the other warps are done (configuration 0's
 * short rounds: 21.8 -> 20.9 ms of walks per job). */
constexpr float kScreenSigmas = 1.1f;
constexpr uint32_t kScreenMinFrames = 48;
constexpr uint32_t kScreenSlices = 2;
constexpr uint32_t kScreenTail = 2;

struct ScreenQueue {
    uint32_t lock, nc, nf;
    uint2 c[kScreenQueue]; /* candidates to screen */
    uint2 f[kScreenQueue]; /* full walks */
};

namespace {

enum Visit { kVisitNone = 0, kVisitScreen = 1, kVisitFull = 2, kVisitAbort = 3, kVisitSort = 4 };

/* One visit of a warp to its CTA's queue: lanes with push 1 or 2 add their
 * entry to the candidates or the full walks; then the warp takes 32 of one
 * kind (entry 0xFFFFFFFF: none for this lane).  `sorting`: more entries will
 * come, so fewer than 32 stay; then they are taken, all for full walks.  After a visit at most 62 entries are left:
 * 32 are taken whenever one queue holds that many. */
__device__ __forceinline__ Visit queue_visit_(ScreenQueue& s, uint2& e, uint32_t push, bool sorting, uint32_t* err)
{
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    uint32_t held = 0u;
    if (lane == 0u) {
        for (uint32_t it = 0; it < kLockLimit && !held; ++it) {
            held = atomicCAS(&s.lock, 0u, 1u) == 0u ? 1u : 0u;
            if (!held) __nanosleep(40);
        }
        if (!held) atomicOr(err, PCS_ERRBIT_TIMEOUT);
    }
    if (!__shfl_sync(0xFFFFFFFFu, held, 0)) return kVisitAbort;
    __threadfence_block();
    volatile ScreenQueue& q = s;
    uint32_t nc = q.nc, nf = q.nf;
    const unsigned mc = __ballot_sync(0xFFFFFFFFu, push == 1u), mf = __ballot_sync(0xFFFFFFFFu, push == 2u);
    if (push == 1u) {
        q.c[nc + __popc(mc & lt)].x = e.x;
        q.c[nc + __popc(mc & lt)].y = e.y;
    } else if (push == 2u) {
        q.f[nf + __popc(mf & lt)].x = e.x;
        q.f[nf + __popc(mf & lt)].y = e.y;
    }
    nc += __popc(mc);
    nf += __popc(mf);
    __threadfence_block();
    __syncwarp();
    Visit v = kVisitNone;
    e.x = 0xFFFFFFFFu;
    if (nc >= 32u) {
        v = kVisitScreen;
        nc -= 32u;
        e.x = q.c[nc + lane].x;
        e.y = q.c[nc + lane].y;
    } else if (nf >= 32u || (!sorting && nf + nc > 0u)) {
        v = kVisitFull;
        const uint32_t tf = min(nf, 32u), tc = min(nc, 32u - tf);
        nf -= tf;
        if (lane < tf) {
            e.x = q.f[nf + lane].x;
            e.y = q.f[nf + lane].y;
        }
        if (!sorting) { /* the last ones: candidates are walked in full, too */
            nc -= tc;
            if (lane >= tf && lane < tf + tc) {
                e.x = q.c[nc + lane - tf].x;
                e.y = q.c[nc + lane - tf].y;
            }
        }
    }
    __syncwarp();
    if (lane == 0u) {
        q.nc = nc;
        q.nf = nf;
        __threadfence_block();
        atomicExch(&s.lock, 0u);
    }
    __syncwarp();
    return v;
}

/* Whether a visit adds or may take something: a look without the lock.  (A
 * count that another warp raises just after is that warp's to see: it visits
 * after every push.) */
__device__ __forceinline__ bool queue_worth_(const ScreenQueue& s, uint32_t push, bool sorting)
{
    const volatile ScreenQueue& q = s;
    const uint32_t from = sorting ? 32u : 1u;
    return __any_sync(0xFFFFFFFFu, push != 0u || q.nc >= from || q.nf >= from);
}

/* Tracks closed by a warp's walks, kept until 32 of them can be binned at
 * once: a record's two divisions and its atomic would otherwise run for the
 * one lane whose track ended.  32 lanes close at most 128 tracks in a group
 * of four frames. */
constexpr uint32_t kTrackBuf = 160; /* 31 left over, 128 more */

struct TrackBuf {
    uint32_t p[kTrackBuf], k[kTrackBuf]; /* proposal, frames */
    float de[kTrackBuf];
};

/* adds the track (k, de) of proposal p of the lanes with `rec` */
__device__ __forceinline__ void track_push_(TrackBuf& b, uint32_t& n, bool rec, uint32_t p, uint32_t k, float de)
{
    const unsigned m = __ballot_sync(0xFFFFFFFFu, rec);
    if (m) {
        if (rec) {
            const uint32_t at = n + __popc(m & ((1u << (threadIdx.x & 31u)) - 1u));
            b.p[at] = p;
            b.k[at] = k;
            b.de[at] = de;
        }
        n += __popc(m);
    }
}

/* bins the last `m` <= 32 of the n tracks */
__device__ __forceinline__ void track_flush_(const SimArgs& a, TrackBuf& b, uint32_t& n, uint32_t m)
{
    const uint32_t lane = threadIdx.x & 31u;
    __syncwarp();
    n -= m;
    if (lane < m) {
        const PropDev& prop = a.props[b.p[n + lane]];
        const JobDev& job = a.jobs[prop.job];
        record_out_<false>(job.four_delta_t, job.dde, job.B, job.R * job.B, 0u, a.hist + prop.hist_off, a.err, nullptr,
                           b.k[n + lane], b.de[n + lane]);
    }
    __syncwarp();
}

/* Four frames of 32 walks in step, one straight line of code: the tracks'
 * state is updated by selects, and only where some lane's track has closed
 * are the four frames gone through again to collect it.  (Branches on
 * detection, as step_ has them, execute fewer instructions but leave each
 * warp's next instruction waiting on the last: with this form 24 warps per SM
 * do what 32 did, each walk takes less time and launches end sooner.)
 * CHECK: lanes whose particle has no frame s0 + t stay as they are.  XY: x
 * and y may leave the box within the group. */
template <bool CHECK, bool XY>
__device__ __forceinline__ void group_warp_(const ItemCtx& c, TrackBuf& b, uint32_t& nb, Walker& w, uint32_t p,
                                            uint32_t s0, const float* nn)
{
    const uint32_t k0 = w.k;
    const float de0 = w.de;
    bool det[4], on[4], closed = false;
    float dd[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        on[t] = !CHECK || s0 + (uint32_t)t < w.F;
        const float dx = nn[3 * t], dy = nn[3 * t + 1];
        float x = __fadd_rn(w.x, dx), y = __fadd_rn(w.y, dy);
        if (XY) {
            x = wrap_(x, c.hlx, 2.0f * c.hlx);
            y = wrap_(y, c.hly, 2.0f * c.hly);
        }
        const float z = wrap_(__fadd_rn(w.z, nn[3 * t + 2]), c.hlz, 2.0f * c.hlz);
        det[t] = fabsf(z) <= w.haz && fabsf(x) <= c.hax && fabsf(y) <= c.hay;
        dd[t] = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
        if (on[t]) {
            w.x = x;
            w.y = y;
            w.z = z;
            closed |= !det[t] && w.k >= c.kmin;
            w.de = det[t] && w.k != 0u ? __fadd_rn(w.de, dd[t]) : 0.0f; /* from the track's second frame on */
            w.k = det[t] ? w.k + 1u : 0u;
        }
    }
    if (__any_sync(0xFFFFFFFFu, closed)) {
        uint32_t k = k0;
        float de = de0;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            track_push_(b, nb, on[t] && !det[t] && k >= c.kmin, p, k, de);
            if (on[t]) {
                de = det[t] && k != 0u ? __fadd_rn(de, dd[t]) : 0.0f;
                k = det[t] ? k + 1u : 0u;
            }
        }
    }
}

/* Frames 1 .. F-1 of a warp's 32 particles (lanes without one have F = 0),
 * and their last tracks. */
__device__ __forceinline__ void walk_warp_(const SimArgs& a, const ItemCtx& c, TrackBuf& b, uint32_t& nb, Walker& q,
                                           uint32_t p)
{
    const uint32_t f_max = __reduce_max_sync(0xFFFFFFFFu, q.F);
    const uint32_t f_min = __reduce_min_sync(0xFFFFFFFFu, q.F ? q.F : f_max); /* 0 where no lane has one */
    /* Four steps are at most 4 sqrt(33) k < 23 k long and their additions round
     * by less than 1e-6 half box lengths; and what is left of the particles
     * after screening mostly starts around the detection area.  Where that
     * lies farther than this from the box's edge, one vote per group spares
     * the x and y wraps (-2% on configuration 3, -0.7% on configuration 1; a
     * vote that always says no costs 1%). */
    const float far = 23.2f * fabsf(q.sd); /* a negative sd mirrors the steps */
    const float in_x = c.hlx * (1.0f - 1.0e-6f) - far, in_y = c.hly * (1.0f - 1.0e-6f) - far;
    const bool vote = __all_sync(0xFFFFFFFFu, q.F == 0u || (c.hax < in_x && c.hay < in_y));
    uint32_t s0 = 1;
    for (; s0 + 3u < f_min; s0 += 4u) {
        float nn[12];
        group_normals_<false>(a, q, s0, nn);
        if (vote && __all_sync(0xFFFFFFFFu, q.F == 0u || (fabsf(q.x) < in_x && fabsf(q.y) < in_y)))
            group_warp_<false, false>(c, b, nb, q, p, s0, nn);
        else
            group_warp_<false, true>(c, b, nb, q, p, s0, nn);
        while (nb >= 32u) track_flush_(a, b, nb, 32u);
    }
#pragma unroll 1
    for (; s0 < f_max; s0 += 4u) {
        float nn[12];
        group_normals_<false>(a, q, s0, nn);
        group_warp_<true, true>(c, b, nb, q, p, s0, nn);
        while (nb >= 32u) track_flush_(a, b, nb, 32u);
    }
    track_push_(b, nb, q.F > 0u && q.k >= c.kmin, p, q.k, q.de);
    while (nb >= 32u) track_flush_(a, b, nb, 32u);
}

/* a position's distance from its detection region, along one coordinate:
 * from the near edge, or 0.8 of that from the next image's edge */
__device__ __forceinline__ float screen_room_(float v, float half_l, float half_a)
{
    const float u = fabsf(v);
    return fminf(u - half_a, 0.8f * (2.0f * half_l - half_a - u));
}

__device__ __forceinline__ float screen_margin_(float k, float half_l, uint32_t F)
{
    return (__uint2float_rn(F) + 8.0f) * (4.0e-4f * k + 1.0e-6f * half_l);
}

/* the coordinate along which q has the most room (0 x, 1 y, 2 z) */
__device__ __forceinline__ uint32_t screen_axis_(const Walker& q, const ItemCtx& c, float& room, float& half_l)
{
    const float rx = screen_room_(q.x, c.hlx, c.hax), ry = screen_room_(q.y, c.hly, c.hay);
    const float rz = screen_room_(q.z, c.hlz, q.haz);
    uint32_t axis = 0u;
    room = rx;
    half_l = c.hlx;
    if (ry > room) {
        axis = 1u;
        room = ry;
        half_l = c.hly;
    }
    if (rz > room) {
        axis = 2u;
        room = rz;
        half_l = c.hlz;
    }
    return axis;
}

/* Whether to screen q (q.sd holds k).  Any NaN or infinity says no. */
__device__ __forceinline__ bool screen_wanted_(const Walker& q, const ItemCtx& c)
{
    float room, half_l;
    screen_axis_(q, c, room, half_l);
    const float reach = kScreenSigmas / kSqrt2Ln2 * q.sd * sqrtf(__uint2float_rn(q.F));
    return q.F >= kScreenMinFrames && c.kmin >= 1u && q.sd > 0.0f && 6.0f * q.sd <= half_l &&
           room > reach + screen_margin_(q.sd, half_l, q.F);
}

/* The screen walk: true if q is certainly never detected.  The coordinate's
 * normals of a group's four steps (group_normals_: numbers 0..11 in step
 * order x, y, z, pairs sine then cosine) by axis:
 *   x  r0.xy sin, r0.zw cos, r1.zw sin, r2.xy cos
 *   y  r0.xy cos, r1.xy sin, r1.zw cos, r2.zw sin
 *   z  r0.zw sin, r1.xy cos, r2.xy sin, r2.zw cos
 * and cos(t) is taken as sin(t + pi/2), so all lanes run the same code. */
__device__ __forceinline__ bool screen_walk_(const Walker& q, const ItemCtx& c)
{
    float room, half_l;
    const uint32_t axis = screen_axis_(q, c, room, half_l);
    const bool ax = axis == 0u, az = axis == 2u;
    const float pi = 3.14159265358979f;
    const float off0 = axis == 1u ? -0.5f * pi : -pi, off1 = axis == 1u ? -pi : -0.5f * pi;
    float S = 0.0f, lo = 0.0f, hi = 0.0f; /* displacement over k, its extremes */
    const uint32_t f_max = __reduce_max_sync(0xFFFFFFFFu, q.F);
    for (uint32_t s0 = 1u, blk = 2u; s0 < f_max; s0 += 4u, blk += 3u) {
        /* without this the lanes of a warp, whose axes differ, do not stay
         * together: 20% more warp instructions per screened particle */
        __syncwarp();
        const pcs_u4 r0 = pcs_draw_pre(q.ph, pcs_ctr_tag(PCS_STREAM_PARTICLE, blk));
        const pcs_u4 r1 = pcs_draw_pre(q.ph, pcs_ctr_tag(PCS_STREAM_PARTICLE, blk + 1u));
        const pcs_u4 r2 = pcs_draw_pre(q.ph, pcs_ctr_tag(PCS_STREAM_PARTICLE, blk + 2u));
        const uint32_t ra[4] = {az ? r0.z : r0.x, ax ? r0.z : r1.x, az ? r2.x : r1.z, ax ? r2.x : r2.z};
        const uint32_t rb[4] = {az ? r0.w : r0.y, ax ? r0.w : r1.y, az ? r2.y : r1.w, ax ? r2.y : r2.w};
        float d[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float u = __fmaf_rn(__uint2float_rn(ra[i]), 2.3283064365386963e-10f, 1.1641532182693481e-10f);
            const float t = __fmaf_rn(__uint2float_rn(rb[i]), 1.4629180792671596e-09f, (i & 1) ? off1 : off0);
            S = __fmaf_rn(sqrt_ftz_(-lg2_ftz_(u)), sin_ftz_(t), S);
            d[i] = S;
        }
        if (s0 < q.F) {
            lo = fminf(fminf(lo, fminf(d[0], d[1])), fminf(d[2], d[3]));
            hi = fmaxf(fmaxf(hi, fmaxf(d[0], d[1])), fmaxf(d[2], d[3]));
        }
    }
    /* the interval between the region and its next image, seen from u0 >= 0 */
    const float v0 = ax ? q.x : (az ? q.z : q.y), half_a = ax ? c.hax : (az ? q.haz : c.hay);
    const float u0 = fabsf(v0), m = screen_margin_(q.sd, half_l, q.F);
    const float down = v0 < 0.0f ? hi : -lo, up = v0 < 0.0f ? -lo : hi; /* both >= 0 */
    return u0 - q.sd * down > half_a + m && u0 + q.sd * up < 2.0f * half_l - half_a - m;
}

} // namespace

/* Registers: at most 80 a thread in CTAs of up to 256 threads (it uses 71; 24
 * warps per SM; 64 and 32 warps, or 128 and 16, were slower by 1-4%).  CTAs of
 * 512 threads also use 71, so one fits on an SM (16 warps), and CTAs of 1024
 * have 64 (32 warps, some spills); the autotuner times all three. */
template <uint32_t BLOCK>
__global__ void __launch_bounds__(BLOCK, BLOCK <= 256u ? 3 : 1) k_simulate_walk(const __grid_constant__ SimArgs a)
{
    __shared__ ScreenQueue s_queue;
    extern __shared__ TrackBuf s_tracks[]; /* one per warp */
    TrackBuf& tracks = s_tracks[threadIdx.x / 32u];
    uint32_t n_tracks = 0u;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t slices = (a.chunk + 31u) / 32u;
    const uint32_t n_slices = *a.n_items * slices, warps = gridDim.x * (blockDim.x / 32u);
    const bool screening = n_slices / warps >= kScreenSlices;
    const uint32_t n_sort = n_slices - min(n_slices, warps / kScreenTail);
    if (threadIdx.x == 0u) s_queue.lock = s_queue.nc = s_queue.nf = 0u;
    __syncthreads();

    bool more = true, sorting = screening; /* slices are left; they go into the queue */
    uint32_t push = 0u;
    uint2 e = make_uint2(0xFFFFFFFFu, 0u); /* this lane's particle: (proposal, particle) */
    for (;;) {
        __syncwarp();
        Visit v = kVisitNone;
        if (screening && queue_worth_(s_queue, push, sorting)) v = queue_visit_(s_queue, e, push, sorting, a.err);
        push = 0u;
        if (v == kVisitAbort) break;
        if (v == kVisitNone) {
            if (!more) break;
            uint32_t sl = 0u;
            if (lane == 0u) sl = atomicAdd(a.queue_head, 1u);
            sl = __shfl_sync(0xFFFFFFFFu, sl, 0);
            if (sl >= n_slices) {
                more = sorting = false;
                continue;
            }
            if (sl >= n_sort) sorting = false;
            const uint32_t item = sl / slices, part = sl - item * slices;
            const uint32_t p = a.item_prop[item];
            const PropDev& prop = a.props[p];
            const uint32_t i0 = (item - prop.item_begin) * a.chunk;
            const uint32_t n = i0 + part * 32u + lane;
            e = make_uint2(n < min(i0 + a.chunk, prop.total_particles) ? p : 0xFFFFFFFFu, n);
            v = sorting && a.jobs[prop.job].frames_max >= kScreenMinFrames ? kVisitSort : kVisitFull;
        }
        Walker q;
        ItemCtx c;
        q.n = e.y;
        q.F = q.k = 0u;
        q.de = 0.0f;
        if (e.x != 0xFFFFFFFFu) {
            const PropDev& prop = a.props[e.x];
            const JobDev& job = a.jobs[prop.job];
            c = item_ctx_(a, job, prop);
            init_walker_<false, true>(a, c, job, prop, a.counts + prop.counts_off + job.V, e.y, prop.slot,
                                      pcs_ctr_gen_trial(prop.gen, prop.trial), job.seed_lo, job.seed_hi, q);
        } else { /* never detected, never recorded */
            c.hlx = c.hly = c.hlz = 1.0f;
            c.hax = c.hay = q.haz = -1.0f;
            c.kmin = 0xFFFFFFFFu;
            q.x = q.y = q.z = q.sd = 0.0f;
            q.ph = pcs_philox_prepare(0u, 0u, 0u, 0u, 0u);
        }
        __syncwarp();
        if (v == kVisitSort) {
            const bool screen = e.x != 0xFFFFFFFFu && screen_wanted_(q, c);
            if (__any_sync(0xFFFFFFFFu, screen))
                push = screen ? 1u : (e.x != 0xFFFFFFFFu ? 2u : 0u);
            else
                v = kVisitFull; /* a short video's, or all too near: at once, as they were started */
        }
        if (v == kVisitScreen) {
            if (!screen_walk_(q, c)) push = 2u;
        } else if (v == kVisitFull) {
            walk_warp_(a, c, tracks, n_tracks, q, e.x);
        }
    }
    if (n_tracks) track_flush_(a, tracks, n_tracks, n_tracks);
}

/* ----------------------------------------------------------------------- */
/* Few particles (k_simulate_few): L lanes per particle, 4 or 8.
 *
 * A launch of a few slices per scheduler takes as long as one walk's chain of
 * Philox rounds, Box-Muller and steps, group after group, whatever its size.
 * Here lane j of a particle's L draws the normals of frames 4j .. 4j+3 of a
 * block of 4L, and then walks one coordinate (lane 0 x, 1 y, the others z)
 * through all of them, the steps transposed through shared memory; the next
 * block's normals are drawn meanwhile.  Each lane keeps a bit per frame for
 * its coordinate lying in the detection region; two exchanges give the frames
 * that find the particle, and only where there are any does the first lane
 * extend and close tracks.  Every value is computed as in the other walks:
 * the histogram is the same, count for count.
 *
 * Only the z coordinate's steps are repeated, so with 4 lanes a particle's
 * frames take ~1.3 times the issue slots of a walk by one lane, with 8 ~1.5
 * times; a group of four frames takes a lone warp 0.23 us (0.18) and not 0.8.
 * Measured, k_simulate_walk -> 4 lanes -> 8 lanes in us, 200 frames: 2560
 * particles 45 -> 22.8 -> 18.1, 8000 54 -> 25.9 -> 24.8, 16000 56 -> 29.3 ->
 * 34.3, 48000 77 -> 54, 64000 77 -> 69, 96000 79 -> 93; 1000 frames: 2560
 * 202 -> 75 -> 58, 8000 239 -> 87 -> 75, 64000 354 -> 281, 96000 354 -> 388;
 * 50 frames: 2560 16.9 -> 11.0 -> 10.8, 64000 26.4 -> 26.8.  Hence the lines:
 * 8 lanes to 8192 particles, 4 lanes to 65536.  The host has to know the
 * number: standalone calls only. */
constexpr uint32_t kFewItems = 65536u / kFewChunk, kFewItems8 = 8192u / kFewChunk;
constexpr uint32_t kFewThreads = 64;

/* frames s0 .. s0+nv-1 of the particle's track (bit t of `det`: found in frame s0 + t) */
__device__ __forceinline__ void few_tracks_(const ItemCtx& c, uint32_t det, uint32_t nv, const float* dd, uint32_t& k, float& de)
{
    uint32_t f = 0u;
    while (f < nv) {
        uint32_t rest = det >> f;
        if (!(rest & 1u)) { /* closed, up to the next frame that finds it */
            if (k >= c.kmin) record_out_<false>(c.four_dt, c.dde, c.B, c.RB, 0u, c.hist, c.err, nullptr, k, de);
            k = 0u;
            de = 0.0f;
            if (!rest) break;
            f += (uint32_t)__ffs(rest) - 1u;
            rest = det >> f;
        }
        const uint32_t end = min(f + (uint32_t)__clz((int)__brev(~rest)), nv);
        if (k == 0u) { /* from the track's second frame on */
            k = 1u;
            ++f;
        }
        k += end - f;
#pragma unroll 4
        for (; f < end; ++f) de = __fadd_rn(de, dd[f]);
    }
}

template <uint32_t L>
__global__ void __launch_bounds__(kFewThreads, 12) k_simulate_few(const __grid_constant__ SimArgs a)
{
    /* a particle's x, y, z steps and squared displacements of a block's
     * frames: rows of 4L + 4, free of bank conflicts either way */
    constexpr uint32_t kParticles = 32u / L, kFrames = 4u * L, kRow = kFrames + 4u;
    __shared__ __align__(16) float s_steps[kFewThreads / 32u][kParticles * 4u * kRow];
    const uint32_t lane = threadIdx.x & 31u, j = lane % L;
    const uint32_t slices = (a.chunk + kParticles - 1u) / kParticles;
    const uint32_t sl = blockIdx.x * (kFewThreads / 32u) + (threadIdx.x >> 5);
    const uint32_t item = sl / slices, part = sl - item * slices;
    if (item >= *a.n_items) return; /* whole warp */
    const PropDev& prop = a.props[a.item_prop[item]];
    const JobDev& job = a.jobs[prop.job];
    const uint32_t i0 = (item - prop.item_begin) * a.chunk;
    const uint32_t n = i0 + part * kParticles + lane / L;
    const bool real = part * kParticles + lane / L < a.chunk && n < prop.total_particles;
    if (!__any_sync(0xFFFFFFFFu, real)) return;
    const ItemCtx c = item_ctx_(a, job, prop);
    Walker q;
    q.F = q.k = 0u;
    q.x = q.y = q.z = q.sd = q.haz = 0.0f;
    if (real) {
        init_walker_<false, true>(a, c, job, prop, a.counts + prop.counts_off + job.V, n, prop.slot,
                                  pcs_ctr_gen_trial(prop.gen, prop.trial), job.seed_lo, job.seed_hi, q);
    } else {
        q.ph = pcs_philox_prepare(0u, 0u, 0u, 0u, 0u);
    }
    float v = j == 0u ? q.x : (j == 1u ? q.y : q.z);
    const float half_l = j == 0u ? c.hlx : (j == 1u ? c.hly : c.hlz);
    const float half_a = j == 0u ? c.hax : (j == 1u ? c.hay : q.haz);
    float* mine = s_steps[threadIdx.x >> 5] + lane / L * 4u * kRow;
    const float* walk = mine + min(j, 2u) * kRow;
    uint32_t k = j == 0u ? q.k : 0u;
    float de = 0.0f;
    const uint32_t f_max = __reduce_max_sync(0xFFFFFFFFu, q.F);
    float nn[12];
    group_normals_<false>(a, q, 1u + 4u * j, nn);
    for (uint32_t s0 = 1u; s0 < f_max; s0 += kFrames) {
        __syncwarp(); /* the block before is read */
#pragma unroll
        for (int x = 0; x < 3; ++x)
            *reinterpret_cast<float4*>(mine + x * (int)kRow + 4u * j) = make_float4(nn[x], nn[3 + x], nn[6 + x], nn[9 + x]);
        float dd[4];
#pragma unroll
        for (int t = 0; t < 4; ++t)
            dd[t] = __fadd_rn(__fmul_rn(nn[3 * t], nn[3 * t]), __fmul_rn(nn[3 * t + 1], nn[3 * t + 1]));
        *reinterpret_cast<float4*>(mine + 3u * kRow + 4u * j) = make_float4(dd[0], dd[1], dd[2], dd[3]);
        __syncwarp();
        group_normals_<false>(a, q, s0 + kFrames + 4u * j, nn); /* past the last frame: not used */
        uint32_t in = 0u;
#pragma unroll
        for (uint32_t g = 0; g < L; ++g) {
            const float4 d = *reinterpret_cast<const float4*>(walk + 4u * g);
            const float step[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
            for (uint32_t t = 0; t < 4u; ++t) {
                v = wrap_(__fadd_rn(v, step[t]), half_l, 2.0f * half_l);
                in |= fabsf(v) <= half_a ? 1u << (4u * g + t) : 0u;
            }
        }
        in &= __shfl_xor_sync(0xFFFFFFFFu, in, 1);
        in &= __shfl_xor_sync(0xFFFFFFFFu, in, 2); /* all three coordinates', in lanes 0 .. 3 */
        const uint32_t nv = q.F > s0 ? min(q.F - s0, kFrames) : 0u;
        in &= nv < 32u ? (1u << nv) - 1u : 0xFFFFFFFFu;
        /* the vote keeps the warp together where no lane has any */
        if (__any_sync(0xFFFFFFFFu, j == 0u && (in | k) != 0u)) {
            if (j == 0u) few_tracks_(c, in, nv, mine + 3u * kRow, k, de);
            __syncwarp();
        }
    }
    if (j == 0u && q.F > 0u && k >= c.kmin) record_out_<false>(c.four_dt, c.dde, c.B, c.RB, 0u, c.hist, c.err, nullptr, k, de);
}

/* The slab-split walk (k_simulate_split).
 *
 * Same model as k_simulate, fewer draws: a particle can only be detected
 * while its z lies in the detection slab (|z| <= half depth), and the x, y
 * steps taken while z is outside it matter only through their sum.  Steps
 * go in groups of four (m <= 4 in the last group).  The CTA (256 threads,
 * one particle each) works in chunks of kSplitG groups, in three phases
 * separated by barriers:
 *   Z  every thread walks z step by step exactly (four normals per group)
 *      and moves x, y by the group's summed displacement S = sd sqrt(m) n;
 *      a group with any z in the slab becomes a task in the CTA's queue;
 *   T  the CTA's threads take the queued tasks densely: a task draws its
 *      group's x, y steps conditioned on their sum (Gaussian bridge,
 *      d_i = S/m + sd (n_i - mean n), exactly i.i.d. N(0, sd^2) again),
 *      walks them from the group's start and stores each step's detection
 *      bit and dx^2 + dy^2;
 *   S  each thread runs the reference's track bookkeeping
 *      (kernel-simulate.inl:70-93) over its groups in time order; a group
 *      without a task is undetected from its first step.
 * The joint law of the positions at every frame is the per-step walk's, so
 * the histograms have the same distribution (from different draws); the
 * CPU oracle's orc_simulate_philox_split follows the same blocks and
 * arithmetic.  Philox blocks of particle n per group pair h (groups 2h,
 * 2h+1): 2+8h z(2h), 3+8h z(2h+1), 4+8h both groups' sums, 5+8h..6+8h the
 * x, y steps of group 2h, 7+8h..8+8h those of group 2h+1. */

constexpr uint32_t kSplitThreads = 256;
constexpr uint32_t kSplitG = 6; /* groups per chunk: even, so group pairs stay in one chunk */
constexpr uint32_t kSplitCap = kSplitThreads * kSplitG;

struct SplitShared {
    float xs[kSplitCap], ys[kSplitCap], sx[kSplitCap], sy[kSplitCap]; /* in; out: dx^2 + dy^2 per step */
    float sd[kSplitCap];
    uint32_t meta[kSplitCap]; /* owner << 16 | group-in-chunk << 8 | m << 4 | in-slab bits (detection bits out) */
    uint16_t idx[kSplitG][kSplitThreads]; /* task of (group-in-chunk, thread) */
    uint32_t count;
};

namespace {

__device__ __forceinline__ float split_sqrt_m_(uint32_t m)
{
    return m == 4u ? 2.0f : (m == 3u ? 1.73205080757f : (m == 2u ? 1.41421356237f : 1.0f));
}

__device__ __forceinline__ float split_inv_m_(uint32_t m)
{
    return m == 4u ? 0.25f : (m == 3u ? 0.333333333333f : (m == 2u ? 0.5f : 1.0f));
}

template <bool AGG>
__device__ __forceinline__ void close_track_(const ItemCtx& c, uint32_t* tile, Walker& q)
{
    if (q.k >= c.kmin) record_<AGG>(c, tile, q.k, q.de);
    q.k = 0u;
    q.de = 0.0f;
}

} // namespace

template <bool AGG>
__global__ void __launch_bounds__(kSplitThreads, 4) k_simulate_split(SimArgs a)
{
    extern __shared__ uint32_t s_tile[];
    __shared__ uint32_t s_item, s_gmax;
    __shared__ PropDev s_prop;
    __shared__ JobDev s_job;

    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    SplitShared& sh = *reinterpret_cast<SplitShared*>(s_tile + a.tile_words);
    for (uint32_t i = tid; i < a.tile_words; i += kSplitThreads) s_tile[i] = 0u;
    const uint32_t n_items = *a.n_items;
    unsigned long long tasks_total = 0ull;

    for (;;) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(a.queue_head, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= n_items) break;
        load_item_(a, item, s_prop, s_job);
        const ItemCtx c = item_ctx_(a, s_job, s_prop);
        const uint32_t* prefix = a.counts + s_prop.counts_off + s_job.V; /* [V+1] */
        const uint32_t k0 = s_job.seed_lo, k1 = s_job.seed_hi;
        const uint32_t slot = s_prop.slot;
        const uint32_t gt = pcs_ctr_gen_trial(s_prop.gen, s_prop.trial);
        const uint32_t chunk_idx = item - s_prop.item_begin;
        const uint32_t a0 = chunk_idx * a.chunk;
        const uint32_t a1 = min(a0 + a.chunk, s_prop.total_particles);

        for (uint32_t base = a0; base < a1; base += kSplitThreads) {
            const uint32_t n = base + tid;
            Walker q;
            q.n = n;
            q.F = 0u;
            q.k = 0u;
            q.de = 0.0f;
            q.x = q.y = q.z = 0.0f;
            q.sd = 0.0f;
            q.haz = 0.0f;
            if (n < a1) init_walker_<false>(a, c, s_job, s_prop, prefix, n, slot, gt, k0, k1, q);
            const uint32_t steps = q.F > 0u ? q.F - 1u : 0u;
            const uint32_t groups = (steps + 3u) >> 2;
            if (tid == 0) {
                s_gmax = 0u;
                sh.count = 0u;
            }
            __syncthreads();
            atomicMax(&s_gmax, groups);
            __syncthreads();
            const uint32_t gmax = s_gmax;

            for (uint32_t g0 = 0; g0 < gmax; g0 += kSplitG) {
                /* ---- phase Z: z per step, x, y per group, tasks queued ---- */
                uint32_t fullmask = 0u;
#pragma unroll 1
                for (uint32_t gl = 0; gl < kSplitG; gl += 2u) {
                    const uint32_t g = g0 + gl; /* even */
                    float nz[8], ag[4];
                    if (g < groups) {
                        const uint32_t blk0 = 2u + 8u * (g >> 1);
                        const pcs_u4 r0 = pcs_draw_pre(q.ph, pcs_ctr_tag(PCS_STREAM_PARTICLE, blk0));
                        const pcs_u4 r1 = pcs_draw_pre(q.ph, pcs_ctr_tag(PCS_STREAM_PARTICLE, blk0 + 1u));
                        const pcs_u4 r2 = pcs_draw_pre(q.ph, pcs_ctr_tag(PCS_STREAM_PARTICLE, blk0 + 2u));
                        box_muller_(r0.x, r0.y, nz[0], nz[1]);
                        box_muller_(r0.z, r0.w, nz[2], nz[3]);
                        box_muller_(r1.x, r1.y, nz[4], nz[5]);
                        box_muller_(r1.z, r1.w, nz[6], nz[7]);
                        box_muller_(r2.x, r2.y, ag[0], ag[1]);
                        box_muller_(r2.z, r2.w, ag[2], ag[3]);
                    }
#pragma unroll
                    for (uint32_t h = 0; h < 2u; ++h) {
                        const uint32_t gg = g + h;
                        uint32_t zbits = 0u, m = 0u;
                        float xs = 0.0f, ys = 0.0f, sx = 0.0f, sy = 0.0f;
                        if (gg < groups) {
                            m = min(4u, steps - 4u * gg);
#pragma unroll
                            for (uint32_t i = 0; i < 4u; ++i) {
                                if (i < m) {
                                    const float dz = __fmul_rn(q.sd, nz[4u * h + i]);
                                    q.z = wrap_(__fadd_rn(q.z, dz), c.hlz, c.two_hlz);
                                    if (fabsf(q.z) <= q.haz) zbits |= 1u << i;
                                }
                            }
                            const float sds = __fmul_rn(q.sd, split_sqrt_m_(m));
                            sx = __fmul_rn(sds, ag[2u * h]);
                            sy = __fmul_rn(sds, ag[2u * h + 1u]);
                            xs = q.x;
                            ys = q.y;
                            q.x = wrap_(__fadd_rn(q.x, sx), c.hlx, c.two_hlx);
                            q.y = wrap_(__fadd_rn(q.y, sy), c.hly, c.two_hly);
                        }
                        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, zbits != 0u);
                        if (bal) {
                            uint32_t wbase = 0u;
                            if (lane == 0u) wbase = atomicAdd(&sh.count, (uint32_t)__popc(bal));
                            wbase = __shfl_sync(0xFFFFFFFFu, wbase, 0);
                            if (zbits) {
                                const uint32_t e = wbase + (uint32_t)__popc(bal & lt_mask);
                                sh.xs[e] = xs;
                                sh.ys[e] = ys;
                                sh.sx[e] = sx;
                                sh.sy[e] = sy;
                                sh.sd[e] = q.sd;
                                sh.meta[e] = (tid << 16) | ((gl + h) << 8) | (m << 4) | zbits;
                                sh.idx[gl + h][tid] = (uint16_t)e;
                                fullmask |= 1u << (gl + h);
                            }
                        }
                    }
                }
                __syncthreads();
                /* ---- phase T: the queued tasks, densely ---- */
                const uint32_t cnt = sh.count;
                for (uint32_t e = tid; e < cnt; e += kSplitThreads) {
                    const uint32_t meta = sh.meta[e];
                    const uint32_t owner = meta >> 16, gl = (meta >> 8) & 0xFFu, m = (meta >> 4) & 7u;
                    const uint32_t zbits = meta & 15u, g = g0 + gl;
                    const float xs = sh.xs[e], ys = sh.ys[e], sxv = sh.sx[e], syv = sh.sy[e], sd = sh.sd[e];
                    const pcs_philox_pre ph = pcs_philox_prepare(base + owner, slot, gt, k0, k1);
                    const uint32_t blk = 2u + 8u * (g >> 1) + 3u + 2u * (g & 1u);
                    float nx[4], ny[4];
                    pcs_u4 r = pcs_draw_pre(ph, pcs_ctr_tag(PCS_STREAM_PARTICLE, blk));
                    box_muller_(r.x, r.y, nx[0], ny[0]);
                    box_muller_(r.z, r.w, nx[1], ny[1]);
                    r = pcs_draw_pre(ph, pcs_ctr_tag(PCS_STREAM_PARTICLE, blk + 1u));
                    box_muller_(r.x, r.y, nx[2], ny[2]);
                    box_muller_(r.z, r.w, nx[3], ny[3]);
                    const float im = split_inv_m_(m);
                    float mx = 0.0f, my = 0.0f;
#pragma unroll
                    for (uint32_t i = 0; i < 4u; ++i) {
                        if (i < m) {
                            mx = __fadd_rn(mx, nx[i]);
                            my = __fadd_rn(my, ny[i]);
                        }
                    }
                    mx = __fmul_rn(mx, im);
                    my = __fmul_rn(my, im);
                    const float cx = __fmul_rn(sxv, im), cy = __fmul_rn(syv, im);
                    float xx = xs, yy = ys, dv[4];
                    uint32_t det = 0u;
#pragma unroll
                    for (uint32_t i = 0; i < 4u; ++i) {
                        dv[i] = 0.0f;
                        if (i < m) {
                            const float dx = __fadd_rn(cx, __fmul_rn(sd, __fsub_rn(nx[i], mx)));
                            const float dy = __fadd_rn(cy, __fmul_rn(sd, __fsub_rn(ny[i], my)));
                            xx = wrap_(__fadd_rn(xx, dx), c.hlx, c.two_hlx);
                            yy = wrap_(__fadd_rn(yy, dy), c.hly, c.two_hly);
                            if (((zbits >> i) & 1u) && fabsf(xx) <= c.hax && fabsf(yy) <= c.hay) det |= 1u << i;
                            dv[i] = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
                        }
                    }
                    sh.xs[e] = dv[0];
                    sh.ys[e] = dv[1];
                    sh.sx[e] = dv[2];
                    sh.sy[e] = dv[3];
                    sh.meta[e] = (meta & ~15u) | det;
                }
                tasks_total += cnt;
                __syncthreads();
                if (tid == 0) sh.count = 0u;
                /* ---- phase S: track bookkeeping over this thread's groups ---- */
                const uint32_t have = groups > g0 ? min(groups - g0, kSplitG) : 0u; /* groups of this chunk */
                uint32_t bits = fullmask, pos = 0u;
                while (bits) {
                    const uint32_t gl = (uint32_t)__ffs(bits) - 1u;
                    bits &= bits - 1u;
                    if (gl > pos) close_track_<AGG>(c, s_tile, q); /* groups without a task before it */
                    const uint32_t e = sh.idx[gl][tid];
                    const uint32_t meta = sh.meta[e];
                    const uint32_t m = (meta >> 4) & 7u;
                    const float dv[4] = {sh.xs[e], sh.ys[e], sh.sx[e], sh.sy[e]};
#pragma unroll
                    for (uint32_t i = 0; i < 4u; ++i) {
                        if (i < m) {
                            if ((meta >> i) & 1u) {
                                const uint32_t kp = q.k + 1u;
                                if (kp >= 2u) q.de = __fadd_rn(q.de, dv[i]);
                                q.k = kp;
                            } else {
                                close_track_<AGG>(c, s_tile, q);
                            }
                        }
                    }
                    pos = gl + 1u;
                }
                if (have > pos) close_track_<AGG>(c, s_tile, q); /* groups without a task after the last */
                __syncthreads();
            }
            if (q.F > 0u && q.k >= c.kmin) record_<AGG>(c, s_tile, q.k, q.de);
        }

        __syncthreads();
        /* flush the privatised rows into the proposal's histogram */
        for (uint32_t i = tid; i < c.tile_words_used; i += kSplitThreads) {
            const uint32_t v = s_tile[i];
            if (v) {
                atomicAdd(c.hist + i, v);
                s_tile[i] = 0u;
            }
        }
    }
    if (a.tasks && tid == 0u && tasks_total) atomicAdd(a.tasks, tasks_total);
}

/* ----------------------------------------------------------------------- */

namespace {
template <int PPT, bool REPLAY, bool AGG>
cudaError_t launch_sim_(const SimArgs& a, uint32_t grid, uint32_t block, size_t smem, cudaStream_t st)
{
    auto fn = k_simulate<PPT, REPLAY, AGG>;
    cudaError_t e = allow_smem(fn, kDynSmemMax);
    if (e != cudaSuccess) return e;
    fn<<<grid, block, smem, st>>>(a);
    return cudaGetLastError();
}

template <int PPT, bool REPLAY, bool AGG>
int occupancy_(uint32_t block, size_t smem)
{
    int n = 0;
    auto fn = k_simulate<PPT, REPLAY, AGG>;
    allow_smem(fn, kDynSmemMax);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, (int)block, smem) != cudaSuccess) return 0;
    return n;
}

/* the tile-less walk's build for `block` threads */
auto walk_kernel_(uint32_t block) -> void (*)(SimArgs)
{
    return block <= 256u ? k_simulate_walk<256> : (block <= 512u ? k_simulate_walk<512> : k_simulate_walk<1024>);
}

size_t walk_smem_(uint32_t block) { return (block / 32u) * sizeof(TrackBuf); }

template <bool AGG>
cudaError_t launch_split_(const SimArgs& a, uint32_t grid, size_t smem, cudaStream_t st)
{
    auto fn = k_simulate_split<AGG>;
    cudaError_t e = allow_smem(fn, kDynSmemMax);
    if (e != cudaSuccess) return e;
    fn<<<grid, kSplitThreads, smem, st>>>(a);
    return cudaGetLastError();
}

template <bool AGG>
int occupancy_split_(size_t smem)
{
    int n = 0;
    auto fn = k_simulate_split<AGG>;
    allow_smem(fn, kDynSmemMax);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, (int)kSplitThreads, smem) != cudaSuccess) return 0;
    return n;
}

/* The split walk's task queue follows the histogram tile in shared memory;
 * the tile gives way so that both fit in 220 KB. */
uint32_t split_tile_words_(uint32_t tile_words)
{
    const size_t cap = (220u * 1024u - sizeof(SplitShared)) / 4u;
    return (uint32_t)(tile_words < cap ? tile_words : cap);
}

bool walk_launch_(const SimLaunch& l, uint32_t tile_words) { return !l.replay && l.ppt == 1 && tile_words == 0u; }
} // namespace

cudaError_t launch_simulate(const SimArgs& a_in, const SimLaunch& l, cudaStream_t st)
{
    if (l.split) {
        if (l.replay) return cudaErrorInvalidValue;
        SimArgs a = a_in;
        a.tile_words = split_tile_words_(a.tile_words);
        const size_t smem = (size_t)a.tile_words * 4u + sizeof(SplitShared);
        last_kernel(kFamilyForward) = "k_simulate_split";
        return l.aggregate ? launch_split_<true>(a, l.grid, smem, st) : launch_split_<false>(a, l.grid, smem, st);
    }
    const SimArgs& a = a_in;
    if (l.few_items) {
        if (a.chunk != kFewChunk) return cudaErrorInvalidValue;
        const uint32_t per = kFewThreads / 32u;
        last_kernel(kFamilyForward) = "k_simulate_few";
        if (l.few_items <= kFewItems8)
            k_simulate_few<8><<<(l.few_items * (kFewChunk / 4u) + per - 1u) / per, kFewThreads, 0, st>>>(a);
        else
            k_simulate_few<4><<<(l.few_items * (kFewChunk / 8u) + per - 1u) / per, kFewThreads, 0, st>>>(a);
        return cudaGetLastError();
    }
    if (walk_launch_(l, a.tile_words)) {
        const auto fn = walk_kernel_(l.block);
        const size_t tracks = walk_smem_(l.block);
        const cudaError_t e = allow_smem(fn, walk_smem_(1024u));
        if (e != cudaSuccess) return e;
        last_kernel(kFamilyForward) = "k_simulate_walk";
        fn<<<l.grid, l.block, tracks, st>>>(a);
        return cudaGetLastError();
    }
    const size_t smem = (size_t)a.tile_words * 4u;
    last_kernel(kFamilyForward) = "k_simulate";
#define PCS_SIM_CASE(P, R, G)                                                               \
    if (l.ppt == P && l.replay == R && l.aggregate == G) return launch_sim_<P, R, G>(a, l.grid, l.block, smem, st);
    PCS_SIM_CASE(1, false, false)
    PCS_SIM_CASE(1, false, true)
    PCS_SIM_CASE(2, false, false)
    PCS_SIM_CASE(2, false, true)
    PCS_SIM_CASE(4, false, false)
    PCS_SIM_CASE(4, false, true)
    PCS_SIM_CASE(8, false, false)
    PCS_SIM_CASE(8, false, true)
    PCS_SIM_CASE(1, true, false)
    PCS_SIM_CASE(1, true, true)
#undef PCS_SIM_CASE
    return cudaErrorInvalidValue;
}

bool simulate_few(const SimLaunch& l, uint32_t tile_words, uint32_t kmin, uint64_t items)
{
    /* kmin 0 records an empty track for every frame that does not find the
     * particle, which the runs of few_tracks_ do not see */
    return !l.split && walk_launch_(l, tile_words) && kmin >= 1u && items <= kFewItems;
}

int simulate_occupancy(const SimLaunch& l, uint32_t tile_words)
{
    if (l.split) {
        const size_t smem = (size_t)split_tile_words_(tile_words) * 4u + sizeof(SplitShared);
        return l.aggregate ? occupancy_split_<true>(smem) : occupancy_split_<false>(smem);
    }
    if (walk_launch_(l, tile_words)) {
        int n = 0;
        const auto fn = walk_kernel_(l.block);
        const size_t tracks = walk_smem_(l.block);
        allow_smem(fn, walk_smem_(1024u));
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, (int)l.block, tracks) == cudaSuccess ? n : 0;
    }
    const size_t smem = (size_t)tile_words * 4u;
#define PCS_SIM_OCC(P, R, G) \
    if (l.ppt == P && l.replay == R && l.aggregate == G) return occupancy_<P, R, G>(l.block, smem);
    PCS_SIM_OCC(1, false, false)
    PCS_SIM_OCC(1, false, true)
    PCS_SIM_OCC(2, false, false)
    PCS_SIM_OCC(2, false, true)
    PCS_SIM_OCC(4, false, false)
    PCS_SIM_OCC(4, false, true)
    PCS_SIM_OCC(8, false, false)
    PCS_SIM_OCC(8, false, true)
    PCS_SIM_OCC(1, true, false)
    PCS_SIM_OCC(1, true, true)
#undef PCS_SIM_OCC
    return 0;
}

/* Raw stream words for the counter-layout check. */
__global__ void k_debug_stream(uint32_t k0, uint32_t k1, uint32_t slot, uint32_t gt, uint32_t n,
                               uint32_t j, uint32_t* out)
{
    pcs_u4 r = pcs_draw(n, pcs_ctr_tag(PCS_STREAM_PARTICLE, j), slot, gt, k0, k1);
    out[0] = r.x;
    out[1] = r.y;
    out[2] = r.z;
    out[3] = r.w;
}

cudaError_t launch_debug_stream(uint64_t seed, uint32_t slot, uint32_t gen, uint32_t trial,
                                uint32_t particle, uint32_t block, uint32_t* d_out, cudaStream_t st)
{
    uint32_t m0 = 0, m1 = 0;
    pcs_seed_masks(seed, &m0, &m1);
    k_debug_stream<<<1, 1, 0, st>>>(m0, m1, slot, pcs_ctr_gen_trial(gen, trial), particle, block, d_out);
    return cudaGetLastError();
}

} // namespace pcs
