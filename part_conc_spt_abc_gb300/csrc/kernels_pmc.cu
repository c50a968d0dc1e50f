/*
 * kernels_pmc.cu -- the ABC-PMC step on the device.
 *
 * The reference runs the population Monte Carlo loop on the host in double
 * (SimulationT::run, src/gpu/detail/simulation_impl.inl:178-455): per slot it
 * picks a parent by weight (wrand_idx_ :54-62), perturbs every parameter with
 * a reflected Gaussian (displace_ :64-79), sorts components by m to avoid
 * label switching (:276-303), draws Poisson particle counts (:307-317), ships
 * one proposal per launch and retries the slot until dist <= gamma; at the
 * end of a generation it reweights (:832-887), updates tau (:733-749) and
 * lowers gamma.  Here the same steps run as kernels over all pending slots of
 * all jobs in a round:
 *
 *   k_round_plan   shares the round's proposal capacity among the jobs
 *                  (trials per pending slot k = capacity / pending, clamped)
 *   k_propose      two warps per proposal: parent pick, perturbation,
 *                  label sort, per-proposal forward-model arguments, Poisson
 *                  counts per video (transformed rejection, Hoermann 1993)
 *   k_items        scan of work items and the item -> proposal map
 *   k_accept       per job: first accepted trial of every slot, trial
 *                  accounting, compaction of the pending list
 *   k_whiten       coordinates of old/new populations in the metric of the
 *                  perturbation kernel (double -> float, centred)
 *   k_kernel_sum   pmc-standard importance weights: log-sum-exp over the old
 *                  population in FP32
 *   k_finalize     per job: weight normalisation (FP64), commit, tau or
 *                  weighted covariance + Cholesky (FP64), gamma update
 *
 * Every random draw is Philox keyed by (seed, generation, slot, trial), so a
 * job's result does not depend on the round capacity or on which other jobs
 * share its rounds.
 */
#include <cuda_runtime.h>
#include <math.h>

#include "pcs_common.h"
#include "pcs_kernels.h"
#include "pcs_proposal.h"

namespace pcs {

namespace {

/* the job whose range of the round's proposals holds q (a warp's lanes look
 * at two jobs each) */
__device__ __forceinline__ uint32_t job_of_(const RoundDev* rd, uint32_t q, uint32_t lane)
{
    static_assert(kMaxRoundJobs <= 64u, "two jobs per lane");
    const uint32_t n = rd->n_jobs;
    uint32_t found = 0u;
#pragma unroll
    for (uint32_t h = 0; h < 2u; ++h) {
        const uint32_t i = lane + 32u * h;
        if (i < n && q >= rd->job_base[i] && q - rd->job_base[i] < rd->job_count[i]) found |= 1u << h;
    }
    const unsigned m0 = __ballot_sync(0xFFFFFFFFu, found & 1u), m1 = __ballot_sync(0xFFFFFFFFu, found & 2u);
    return m0 ? (uint32_t)__ffs(m0) - 1u : (m1 ? 31u + (uint32_t)__ffs(m1) : 0u);
}

} // namespace

/* ----------------------------------------------------------------------- */
/* One thread per job computes the job's share (divisions and dependent loads
 * of 64 jobs side by side instead of one after another: 4 jobs 20 -> 9 us);
 * thread 0 adds up what depends on the jobs before. */
__global__ void __launch_bounds__(kMaxRoundJobs) k_round_plan(PmcArgs a)
{
    __shared__ double s_planned[kMaxRoundJobs], s_key[kMaxRoundJobs];
    __shared__ uint64_t s_rb[kMaxRoundJobs], s_hbase[kMaxRoundJobs];
    __shared__ uint32_t s_pend[kMaxRoundJobs], s_k[kMaxRoundJobs], s_base[kMaxRoundJobs], s_cnt[kMaxRoundJobs];
    __shared__ uint8_t s_ord[kMaxRoundJobs], s_spec[kMaxRoundJobs];
    __shared__ uint32_t s_kmax;
    __shared__ double s_fill;
    const uint32_t j = threadIdx.x;
    RoundDev* rd = a.round;
    const uint32_t nj = min(rd->n_jobs, kMaxRoundJobs);
    const bool have = j < nj;
    const JobPmcDev& pm = a.pmc[have ? j : 0u];
    const bool live = have && !pm.done;
    const uint32_t pend = live ? pm.pending_count : 0u, gen = pm.generation;
    const double accepted = (double)pm.accepted_gen, trials = (double)pm.trials;
    const double sims = (double)pm.simulations, steps = (double)pm.particle_steps;
    s_pend[j] = pend;
    s_rb[j] = have ? (uint64_t)a.jobs[j].R * a.jobs[j].B : 0u;
    const double fmax_j = (double)max(have ? a.jobs[j].frames_max : 1u, 1u);
    __syncthreads();
    if (j == 0u) {
        uint64_t total_pending = 0;
        for (uint32_t i = 0; i < nj; ++i) total_pending += s_pend[i];
        uint32_t k = total_pending ? (uint32_t)(rd->capacity / total_pending) : 1u;
        if (k < 1u) k = 1u;
        if (k > rd->max_spec) k = rd->max_spec;
        s_kmax = k;
    }
    __syncthreads();
    const uint32_t k = s_kmax;
    /* trials per pending slot: enough to fill the round, but not many more
     * than ~0.3 / (acceptance rate so far), so that few trials are simulated
     * after a slot's first acceptance -- unless the round's proposals would
     * then carry fewer than `fill` particles (one wave of the simulate
     * launch; at the end of a generation few slots are left and the GPU
     * would idle), in which case the slots get proportionally more trials,
     * up to k.  Particles per proposal are estimated from the job's history. */
    const double pacc = (accepted + 1.0) / (trials + 2.0);
    uint32_t kj = k;
    if (gen == 0u) {
        kj = 1u; /* prior pass: one simulation per slot */
    } else {
        const double kw = ceil(0.3 / pacc);
        if (kw < (double)kj) kj = (uint32_t)(kw < 1.0 ? 1.0 : kw);
    }
    /* particles per proposal so far (steps over the longest video) */
    const double spp = steps / sims;
    const double ppp = pm.simulations ? spp / fmax_j : (double)rd->fill;
    s_planned[j] = (double)pend * kj * ppp;
    s_spec[j] = live && gen > 0u && pend > 0u;
    /* the order in which jobs take the round's capacity: admission order, or
     * (order == 1) jobs in their prior pass first, then the least estimated
     * remaining work first -- (pending slots + slots of the generations left)
     * x particle-steps per proposal / acceptance rate -- which lets short
     * jobs finish early instead of waiting behind long ones */
    double kv = (double)j;
    if (rd->order == 1u && gen > 0u && live) {
        const double gens_left =
            pm.max_generations ? fmax(0.0, (double)pm.max_generations - (double)pm.iterations) : 8.0;
        kv = 1e6 + ((double)pend + (double)pm.N * gens_left) * (pm.simulations ? spp : 1.0) / pacc;
    }
    s_key[j] = kv;
    s_ord[j] = (uint8_t)j;
    __syncthreads();
    if (j == 0u) {
        double planned = 0.0;
        bool spec = false;
        for (uint32_t i = 0; i < nj; ++i) {
            if (s_pend[i]) planned += s_planned[i];
            spec |= s_spec[i] != 0u;
        }
        /* the factor of a round to be topped up, else 0 */
        s_fill = rd->fill && planned < (double)rd->fill && spec
                     ? (planned > 0.0 ? (double)rd->fill / planned : (double)k)
                     : 0.0;
    }
    uint32_t rank = 0u; /* of this job's key, equal keys in admission order */
    for (uint32_t i = 0; i < nj; ++i) rank += s_key[i] < kv || (s_key[i] == kv && i < j) ? 1u : 0u;
    if (have) s_ord[rank] = (uint8_t)j;
    __syncthreads();
    if (s_fill > 0.0 && gen > 0u && live)
        kj = (uint32_t)min((double)k, fmax((double)kj, ceil((double)kj * s_fill)));
    s_k[j] = have ? kj : 1u;
    __syncthreads();
    if (j == 0u) {
        uint32_t base = 0;
        uint64_t hbase = 0, cells = 0;
        for (uint32_t o = 0; o < nj; ++o) {
            const uint32_t i = s_ord[o];
            const uint32_t ki = s_k[i];
            uint64_t want = (uint64_t)s_pend[i] * ki;
            uint64_t room = rd->capacity - base;
            const uint64_t rb = s_rb[i];
            if (rb) {
                /* each job's histograms start at a multiple of R x B words, so
                 * one tensor map (B x R x histograms over the whole area) reaches
                 * every histogram of the job */
                hbase = (hbase + rb - 1u) / rb * rb;
                const uint64_t hroom = hbase < rd->hist_cap ? (rd->hist_cap - hbase) / rb : 0u;
                if (hroom < room) room = hroom;
            }
            uint32_t cnt = (uint32_t)(want < room ? want : room);
            cnt -= cnt % ki; /* whole slots only */
            s_base[i] = base;
            s_cnt[i] = cnt;
            s_hbase[i] = hbase;
            base += cnt;
            hbase += cnt * rb;
            cells += cnt * rb;
        }
        rd->n_props = base;
        rd->n_items = 0u;
        rd->queue_head = 0u;
        rd->round_steps = 0ull;
        rd->round_cells = cells;
    }
    __syncthreads();
    if (j < rd->n_jobs) {
        rd->job_base[j] = have ? s_base[j] : 0u;
        rd->job_k[j] = s_k[j];
        rd->job_count[j] = have ? s_cnt[j] : 0u;
        rd->job_hist_base[j] = have ? s_hbase[j] : 0u;
    }
}

/* ----------------------------------------------------------------------- */
/* First index i < N with !(wcum[i] < u) (std::lower_bound on a
 * non-decreasing array), clamped to N - 1, as pcs_pick: a 32-way search, each
 * lane probing one split point per round (2 dependent loads for N = 1024
 * instead of 10). */
__device__ __forceinline__ uint32_t warp_pick_(const double* wcum, uint32_t N, double u, uint32_t lane)
{
    uint32_t lo = 0, hi = N; /* the answer lies in [lo, hi]; hi == N: none found yet */
    for (int round = 0; round < 8 && hi > lo; ++round) {
        const uint32_t span = hi - lo;
        uint32_t idx;
        bool valid;
        if (span <= 32u) {
            idx = lo + lane;
            valid = lane < span;
        } else {
            idx = lo + (uint32_t)(((uint64_t)(lane + 1u) * span) / 32u) - 1u;
            valid = true;
        }
        const bool ge = valid && !(wcum[idx] < u);
        const unsigned m = __ballot_sync(0xFFFFFFFFu, ge);
        if (m == 0u) {
            lo = hi;
            break;
        }
        const uint32_t f = (uint32_t)(__ffs(m) - 1);
        const uint32_t idx_f = __shfl_sync(0xFFFFFFFFu, idx, f);
        if (span <= 32u) {
            lo = hi = idx_f;
            break;
        }
        const uint32_t prev = __shfl_sync(0xFFFFFFFFu, idx, f > 0u ? f - 1u : 0u);
        lo = f > 0u ? prev + 1u : lo;
        hi = idx_f;
    }
    return lo < N ? lo : N - 1u;
}

/* Two warps per proposal.  The FP64 work is spread over the lanes: lane i
 * draws perturbation normal pair i, lane p perturbs and reflects parameter p,
 * lane c computes component c's arguments (10^log10c, step sd); the Poisson
 * constants are computed once and the lanes draw the per-video counts in
 * parallel (each count has its own Philox counter) and scan them into the
 * video prefix.  Every value is the one pcs_build_theta / pcs_build_args /
 * pcs_draw_counts compute (same functions, same operation order).
 *
 * Bound by one proposal's chain of FP64 operations (a dependent one every ~60
 * cycles, a warp instruction per ~16 cycles and SM), so what is independent
 * goes side by side: warp 0 draws the normals' radii, perturbs and sorts, and
 * has the concentrations, the Poisson constants and the counts; warp 1 picks
 * the parent, draws the normals' angles, and has the step sds, the logarithm
 * of the Poisson mean and the descriptor.  (One warp for all of it: 33000
 * cycles, 25.7 us a launch; two: 21.4.)  A round's warps are spread over all
 * SMs: pair w of CTA b takes proposal w x CTAs + b.  The parameters and the
 * descriptor are put together in shared memory and written by a whole warp,
 * not in each lane's local memory. */
constexpr uint32_t kProposePairs = 2;

struct ProposePair {
    double th[PCS_MAX_P], nrm[PCS_MAX_P], sn[PCS_MAX_P / 2 + 1], cs[PCS_MAX_P / 2 + 1];
    double lambda, loglam;
    CompArgs ca[PCS_MAX_C];
    PropDev pd;
    uint32_t parent;
};

/* a pair's barriers: 0 both wait; 1 warp 1 waits for warp 0, 2 warp 0 for warp 1 */
__device__ __forceinline__ void pair_sync_(uint32_t pair, uint32_t which)
{
    __syncwarp();
    asm volatile("bar.sync %0, 64;\n" ::"r"(1u + 3u * pair + which) : "memory");
}

__device__ __forceinline__ void pair_arrive_(uint32_t pair, uint32_t which)
{
    __syncwarp();
    __threadfence_block();
    asm volatile("bar.arrive %0, 64;\n" ::"r"(1u + 3u * pair + which) : "memory");
}

__global__ void __launch_bounds__(64 * kProposePairs) k_propose(PmcArgs a)
{
    __shared__ ProposePair s_pair[kProposePairs];
    RoundDev* rd = a.round;
    const uint32_t lane = threadIdx.x & 31u, pair = threadIdx.x >> 6;
    const bool first = (threadIdx.x & 32u) == 0u; /* warp 0 of the pair */
    const uint32_t q = pair * gridDim.x + blockIdx.x;
    if (q >= rd->n_props) return; /* both warps */
    ProposePair& w = s_pair[pair];
    const uint32_t j = job_of_(rd, q, lane);
    JobPmcDev& pm = a.pmc[j];
    const JobDev& jd = a.jobs[j];
    const uint32_t k = rd->job_k[j];
    const uint32_t local = q - rd->job_base[j];
    const uint32_t pend_idx = local / k, rep = local % k;
    const uint32_t slot = pm.pending[pend_idx];
    const uint32_t trial = pm.next_trial[slot] + rep;
    const uint32_t gen = pm.generation;
    const uint32_t k0 = jd.seed_lo, k1 = jd.seed_hi;
    const uint32_t P = pm.P;
    const uint32_t gt = pcs_ctr_gen_trial(gen, trial);

    /* parameters: lane p computes parameter p */
    if (gen == 0u) {
        if (first && lane < P) w.th[lane] = pm.theta[(uint64_t)slot * P + lane];
    } else {
        pcs_u4 rr = {0u, 0u, 0u, 0u};
        if (2u * lane < P) rr = pcs_draw(lane, pcs_ctr_tag(PCS_STREAM_PERTURB, 0u), slot, gt, k0, k1);
        double rad = 0.0;
        if (first) {
            if (2u * lane < P) rad = pcs_normal_radius(rr);
        } else {
            const pcs_u4 r = pcs_draw(0u, pcs_ctr_tag(PCS_STREAM_PICK, 0u), slot, gt, k0, k1);
            const uint32_t parent = warp_pick_(pm.wcum, pm.N, pcs_u01_53(r.x, r.y), lane);
            if (lane == 0u) w.parent = parent;
            if (2u * lane < P) pcs_normal_angle(rr, w.sn[lane], w.cs[lane]);
        }
        pair_sync_(pair, 0u);
        if (first) {
            if (2u * lane < P) {
                w.nrm[2u * lane] = rad * w.sn[lane];
                if (2u * lane + 1u < PCS_MAX_P) w.nrm[2u * lane + 1u] = rad * w.cs[lane];
            }
            __syncwarp();
            const double* tp = pm.theta + (uint64_t)w.parent * P;
            if (lane < P) w.th[lane] = pcs_perturb_one(pm, tp, pm.factor, w.nrm, lane);
            __syncwarp();
            if (lane == 0u) pcs_sort_components(pm, w.th);
        }
    }
    pair_sync_(pair, 0u);

    /* per-component arguments: lane c computes component c */
    const uint64_t coff = (uint64_t)q * (2u * rd->v_max + 1u);
    if (first) {
        if (lane < pm.C) w.ca[lane].powc = pcs_comp_power(pm, w.th, lane);
        __syncwarp();
        const double lambda = pcs_lambda(pm, w.ca);
        if (lane == 0u) w.lambda = lambda;
        pair_arrive_(pair, 1u);
        if (lane < P) a.theta_prop[(uint64_t)q * PCS_MAX_P + lane] = w.th[lane];

        PoissonSetup ps = pcs_poisson_setup<false>(lambda);
        ps.logfact = a.logfact;
        ps.logfact_n = a.logfact_n;
        pair_sync_(pair, 2u);
        if (pcs_poisson_takes_log(lambda)) pcs_poisson_set_log(ps, w.loglam);
        uint32_t* cnt = a.counts + coff;
        uint32_t* pre = cnt + jd.V;
        uint64_t run = 0, steps = 0;
        if (lane == 0u) pre[0] = 0u;
        for (uint32_t v0 = 0; v0 < jd.V; v0 += 32u) {
            const uint32_t v = v0 + lane;
            uint32_t c = 0u;
            if (v < jd.V) {
                c = pcs_poisson_draw(ps, v, slot, gt, k0, k1);
                cnt[v] = c;
                steps += (uint64_t)c * jd.frames[v];
            }
            uint64_t incl = c;
            for (int d = 1; d < 32; d <<= 1) {
                const uint64_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                if ((int)lane >= d) incl += t;
            }
            const uint64_t tot = run + incl;
            if (v < jd.V) pre[v + 1] = (uint32_t)(tot < 0xFFFFFFFFull ? tot : 0xFFFFFFFFull);
            run += __shfl_sync(0xFFFFFFFFu, incl, 31);
        }
        for (int d = 16; d >= 1; d >>= 1) steps += __shfl_xor_sync(0xFFFFFFFFu, steps, d);
        if (lane == 0u) {
            const uint64_t total = run;
            if (total > 0xFFFFFFFFull) atomicOr(a.err, PCS_ERRBIT_COUNTS);
            w.pd.total_particles = (uint32_t)min(total, (uint64_t)0xFFFFFFFFu);
            w.pd.item_count = (w.pd.total_particles + rd->chunk - 1u) / rd->chunk;
            w.pd.item_begin = 0u;
            atomicAdd((unsigned long long*)&pm.particle_steps, (unsigned long long)steps);
            atomicAdd(&a.round->round_steps, (unsigned long long)steps);
        }
    } else {
        if (lane < pm.C) pcs_comp_sd(pm, w.th, lane, w.ca[lane]);
        pair_sync_(pair, 1u); /* the concentrations and the mean */
        if (lane == 0u && pcs_poisson_takes_log(w.lambda)) w.loglam = log(w.lambda);
        pair_arrive_(pair, 2u);
        if (lane == 0u) {
            const uint64_t rb = (uint64_t)jd.R * jd.B;
            w.pd.job = j;
            w.pd.slot = slot;
            w.pd.trial = trial;
            w.pd.gen = gen;
            pcs_assemble_args(pm, w.th, w.ca, gen, w.pd);
            w.pd.counts_off = coff;
            w.pd.hist_off = rd->job_hist_base[j] + (uint64_t)local * rb;
            /* the job's histograms start at a multiple of R x B words (k_round_plan) */
            w.pd.hist_z = (uint32_t)(w.pd.hist_off / max(1ull, (unsigned long long)rb));
        }
    }
    pair_sync_(pair, 0u);
    if (first)
        for (uint32_t i = lane; i < sizeof(PropDev) / 4u; i += 32u)
            reinterpret_cast<uint32_t*>(a.props + q)[i] = reinterpret_cast<const uint32_t*>(&w.pd)[i];
}

/* ----------------------------------------------------------------------- */
/* item scan: one block */
__global__ void __launch_bounds__(1024) k_items(PmcArgs a)
{
    __shared__ uint32_t s_part[32]; /* each warp's items */
    RoundDev* rd = a.round;
    const uint32_t M = rd->n_props;
    const uint32_t per = (M + blockDim.x - 1) / blockDim.x;
    const uint32_t b = threadIdx.x * per, e = min(b + per, M);
    uint32_t sum = 0;
    for (uint32_t q = b; q < e; ++q) sum += a.props[q].item_count;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t incl = sum, part = 0u;
    for (uint32_t d = 1; d < 32u; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += t;
    }
    if (lane == 31u) s_part[warp] = incl;
    __syncthreads();
    part = lane < nw ? s_part[lane] : 0u; /* every warp scans the warps' */
    for (uint32_t d = 1; d < 32u; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, part, d);
        if (lane >= d) part += t;
    }
    const uint32_t before = __shfl_sync(0xFFFFFFFFu, part, warp ? warp - 1u : 0u);
    uint32_t run = (warp ? before : 0u) + incl - sum;
    for (uint32_t q = b; q < e; ++q) {
        a.props[q].item_begin = run;
        run += a.props[q].item_count;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, part, 31);
    const uint32_t cap = rd->items_cap;
    __syncthreads(); /* every proposal's item_begin is written */
    if (threadIdx.x == 0) {
        if (total > cap) atomicOr(a.err, PCS_ERRBIT_ITEMS);
        rd->n_items = min(total, cap);
        rd->queue_head = 0u;
    }
    /* the item -> proposal map: a warp per proposal, its lanes on
     * consecutive items (coalesced stores) */
    for (uint32_t q = warp; q < M; q += nw) {
        const uint32_t ib = a.props[q].item_begin, ic = a.props[q].item_count;
        for (uint32_t i = lane; i < ic; i += 32u)
            if (ib + i < cap) a.item_prop[ib + i] = q;
    }
}

/* ----------------------------------------------------------------------- */
/* accept: one block per job */
__global__ void __launch_bounds__(1024) k_accept(PmcArgs a)
{
    __shared__ uint32_t s_keep, s_exhausted;
    __shared__ unsigned long long s_trials, s_acc;
    __shared__ double s_sure, s_never;
    const uint32_t j = blockIdx.x;
    RoundDev* rd = a.round;
    if (j >= rd->n_jobs) return;
    JobPmcDev& pm = a.pmc[j];
    if (pm.done) return;
    const uint32_t k = rd->job_k[j];
    const uint32_t cnt = rd->job_count[j];
    const uint32_t base = rd->job_base[j];
    const uint32_t nprop_slots = cnt / k;
    const uint32_t npend = pm.pending_count;
    const uint32_t P = pm.P;
    if (threadIdx.x == 0) {
        s_keep = 0u;
        s_exhausted = 0u;
        s_trials = 0ull;
        s_acc = 0ull;
        pm.gen_ended = 0u;
        const double edge = exp10(pm.gamma); /* one warp's FP64, not the block's */
        s_sure = edge * (1.0 - 1e-11);
        s_never = edge * (1.0 + 1e-11);
    }
    __syncthreads();
    /* decide every pending slot; kept slots go to scratch (as u32 bits).  A
     * group of lanes (as many as the trials per slot, at most a warp) looks at
     * a slot's trials side by side: at a generation's end few slots have many
     * trials each.  log10(d) <= gamma is decided by d against 10^gamma but for
     * a margin far above both functions' errors, in which log10 is taken: on
     * this GPU's FP64 rate it would otherwise set the pace for every trial. */
    uint32_t* keep_list = reinterpret_cast<uint32_t*>(pm.scratch);
    uint32_t g = 1u;
    while (g < 32u && g < k) g <<= 1;
    const uint32_t lane = threadIdx.x & 31u, gl = lane & (g - 1u), g0 = lane & ~(g - 1u);
    const unsigned gmask = g == 32u ? 0xFFFFFFFFu : (1u << g) - 1u;
    const bool prior = pm.generation == 0u;
    /* the job's own choice: another job's in the round may have the doubles formed */
    const bool f64 = a.jobs[j].distance_double && a.use_f64_distance && a.dist_f64;
    const double gamma = pm.gamma, sure = s_sure, never = s_never;
    unsigned long long trials = 0ull, accepted = 0ull;
    for (uint32_t i0 = 0; i0 < npend; i0 += blockDim.x / g) {
        const uint32_t i = i0 + threadIdx.x / g;
        const bool in = i < npend && i < nprop_slots;
        const uint32_t slot = i < npend ? pm.pending[i] : 0u;
        uint32_t first = k;
        for (uint32_t r0 = 0; r0 < k; r0 += g) {
            const uint32_t r = r0 + gl;
            bool ok = false;
            if (in && first == k && r < k) {
                const uint32_t q = base + i * k + r;
                const double df = f64 ? a.dist_f64[q] : (double)a.dist_f32[q];
                ok = prior || df <= sure || (!(df >= never) && log10(df) <= gamma);
            }
            const unsigned m = (__ballot_sync(0xFFFFFFFFu, ok) >> g0) & gmask;
            if (m) first = r0 + (uint32_t)__ffs(m) - 1u;
            if (!__any_sync(0xFFFFFFFFu, in && first == k)) break;
        }
        if (in && first < k) {
            const uint32_t q = base + i * k + first;
            for (uint32_t p = gl; p < P; p += g)
                pm.theta_new[(uint64_t)slot * P + p] = a.theta_prop[(uint64_t)q * PCS_MAX_P + p];
        }
        if (i < npend && gl == 0u) {
            if (in && first < k) {
                const uint32_t q = base + i * k + first;
                pm.dist_new[slot] = log10(f64 ? a.dist_f64[q] : (double)a.dist_f32[q]);
                pm.accepted[slot] = 1u;
                trials += first + 1u;
                accepted += 1u;
            } else {
                if (in) {
                    pm.next_trial[slot] += k;
                    trials += k;
                    /* the trial ordinal has 20 bits in the random-stream counter:
                     * a slot that exhausts them ends the generation like the
                     * trial cap does (converged) */
                    if (pm.next_trial[slot] + rd->max_spec >= (1u << 20)) s_exhausted = 1u;
                }
                keep_list[atomicAdd(&s_keep, 1u)] = slot;
            }
        }
    }
    for (int d = 16; d >= 1; d >>= 1) {
        trials += __shfl_xor_sync(0xFFFFFFFFu, trials, d);
        accepted += __shfl_xor_sync(0xFFFFFFFFu, accepted, d);
    }
    if (lane == 0u && trials) {
        atomicAdd(&s_trials, trials);
        atomicAdd(&s_acc, accepted);
    }
    __syncthreads();
    const uint32_t nk = s_keep;
    for (uint32_t i = threadIdx.x; i < nk; i += blockDim.x) pm.pending[i] = keep_list[i];
    if (threadIdx.x == 0) {
        pm.pending_count = nk;
        pm.trials += s_trials;
        pm.simulations += cnt;
        pm.accepted_total += s_acc;
        pm.accepted_gen += s_acc;
        if (s_exhausted && pm.generation > 0u) pm.trials = (uint64_t)pm.avg_trials * pm.N;
        const bool cap = pm.generation > 0u &&
                         (double)pm.trials >= (double)pm.avg_trials * (double)pm.N;
        if (nk == 0u || cap) pm.gen_ended = 1u;
    }
}

/* ----------------------------------------------------------------------- */
/* whitened coordinates for the kernel density: y = A^-1 (theta - mean),
 * A = diag(tau) or the Cholesky factor; fixed parameters dropped.  Output
 * float [2][N][P] in the job's ybuf (old population, then new). */
__device__ __forceinline__ bool needs_kernel_sum_(const JobPmcDev& pm)
{
    return !(pm.done || !pm.gen_ended || pm.generation == 0u || pm.weighting != 0u) &&
           !((double)pm.trials >= (double)pm.avg_trials * (double)pm.N);
}

/* y_i = L^-1 (theta_i - lo) (Cholesky) or (theta_i - lo) / tau: point i of
 * the committed (i < N) or new (i >= N) population, whitened. */
__device__ __forceinline__ void whiten_one_(const JobPmcDev& pm, uint32_t i)
{
    const uint32_t N = pm.N, P = pm.P;
    const double* th = (i < N) ? pm.theta + (uint64_t)i * P : pm.theta_new + (uint64_t)(i - N) * P;
    float* y = pm.ybuf + (uint64_t)i * P;
    double v[PCS_MAX_P];
    for (uint32_t p = 0; p < P; ++p) v[p] = th[p] - pm.lo[p];
    if (pm.perturbation == 1u) {
        for (uint32_t p = 0; p < P; ++p) {
            if (pm.fixed[p]) {
                v[p] = 0.0;
                continue;
            }
            double s = v[p];
            for (uint32_t q = 0; q < p; ++q)
                if (!pm.fixed[q]) s -= pm.factor[p * P + q] * v[q];
            v[p] = s / pm.factor[p * P + p];
        }
    } else {
        for (uint32_t p = 0; p < P; ++p) v[p] = pm.fixed[p] ? 0.0 : v[p] / pm.factor[p * P + p];
    }
    for (uint32_t p = 0; p < P; ++p) y[p] = (float)v[p];
}

/* The grid covers one job's 2N points and strides over the round's jobs, so
 * rounds that end no generation launch a few blocks that return at once. */
__global__ void k_whiten(PmcArgs a)
{
    const uint32_t n_jobs = a.round->n_jobs;
    for (uint32_t j = 0; j < n_jobs; ++j) {
        const JobPmcDev& pm = a.pmc[j];
        if (!needs_kernel_sum_(pm)) continue;
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 2u * pm.N; i += gridDim.x * blockDim.x)
            whiten_one_(pm, i);
    }
}


/* pmc-standard (simulation_impl.inl:832-871): log w*_a = -log sum_i w_i
 * exp(-0.5 |y*_a - y_i|^2) (the Gaussian normalising constants cancel in
 * the normalisation).  One warp per new particle a. */
__device__ __forceinline__ void kernel_sum_one_(const JobPmcDev& pm, uint32_t an, uint32_t lane);

__global__ void __launch_bounds__(256) k_kernel_sum(PmcArgs a)
{
    const uint32_t n_jobs = a.round->n_jobs;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t j = 0; j < n_jobs; ++j) {
        const JobPmcDev& pm = a.pmc[j];
        if (!needs_kernel_sum_(pm)) continue;
        for (uint32_t an = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; an < pm.N; an += warps)
            kernel_sum_one_(pm, an, lane);
    }
}

/* log w*_an for new particle an, one warp */
__device__ __forceinline__ void kernel_sum_one_(const JobPmcDev& pm, uint32_t an, uint32_t lane)
{
    const uint32_t N = pm.N, P = pm.P;
    const float* yb = pm.ybuf;
    const float* ya = yb + (uint64_t)(N + an) * P;
    float yl[PCS_MAX_P];
    for (uint32_t p = 0; p < P; ++p) yl[p] = ya[p];
    /* pass 1: max exponent; pass 2: scaled sum */
    float mx = -INFINITY;
    for (uint32_t i = lane; i < N; i += 32u) {
        if (!(pm.w[i] > 0.0)) continue;
        const float* yi = yb + (uint64_t)i * P;
        float s = 0.0f;
        for (uint32_t p = 0; p < P; ++p) {
            float d = yl[p] - yi[p];
            s = fmaf(d, d, s);
        }
        mx = fmaxf(mx, -0.5f * s);
    }
    for (int d = 16; d >= 1; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, d));
    float acc = 0.0f;
    for (uint32_t i = lane; i < N; i += 32u) {
        const float wi = (float)pm.w[i];
        if (!(wi > 0.0f)) continue;
        const float* yi = yb + (uint64_t)i * P;
        float s = 0.0f;
        for (uint32_t p = 0; p < P; ++p) {
            float d = yl[p] - yi[p];
            s = fmaf(d, d, s);
        }
        acc = fmaf(wi, __expf(-0.5f * s - mx), acc);
    }
    for (int d = 16; d >= 1; d >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, d);
    if (lane == 0) pm.scratch[an] = -(double)mx - log((double)acc); /* log w*_a */
}

/* ----------------------------------------------------------------------- */
/* Order-preserving map of a double to an unsigned key (negative values:
 * all bits flipped; others: the sign bit set), and back. */
__device__ __forceinline__ unsigned long long order_key_(double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

__device__ __forceinline__ double from_order_key_(unsigned long long k)
{
    const unsigned long long b = (k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
    return __longlong_as_double((long long)b);
}

struct SelectShared {
    uint32_t hist[256];
    unsigned long long prefix, mask;
    uint32_t target;
};

/* The value at position `target` (0-based) of x[0..N) in ascending order
 * (nth_element's result, simulation_impl.inl:819-829), by one block: a
 * radix select over the order-preserving keys, eight passes of 8-bit
 * digits from the top; each pass counts the candidates' digits in shared
 * memory (warp-aggregated atomics) and keeps the digit whose bucket holds
 * the target rank.  O(8 N) work instead of comparing all pairs. */
__device__ double select_rank_(const double* x, uint32_t N, uint32_t target, SelectShared& sh)
{
    const uint32_t tid = threadIdx.x, bd = blockDim.x, lane = tid & 31u;
    if (tid == 0) {
        sh.prefix = 0ull;
        sh.mask = 0ull;
        sh.target = target;
    }
    for (int shift = 56; shift >= 0; shift -= 8) {
        for (uint32_t b = tid; b < 256u; b += bd) sh.hist[b] = 0u;
        __syncthreads();
        const unsigned long long prefix = sh.prefix, mask = sh.mask;
        for (uint32_t base = 0; base < N; base += bd) { /* the same trip count for every thread */
            const uint32_t i = base + tid;
            uint32_t digit = 256u; /* no candidate */
            if (i < N) {
                const unsigned long long k = order_key_(x[i]);
                if ((k & mask) == prefix) digit = (uint32_t)(k >> shift) & 255u;
            }
            const unsigned peers = __match_any_sync(0xFFFFFFFFu, digit);
            if (digit < 256u && lane == (uint32_t)(__ffs(peers) - 1)) atomicAdd(&sh.hist[digit], (uint32_t)__popc(peers));
        }
        __syncthreads();
        if (tid < 32u) {
            /* warp 0: lane l owns digits 8l .. 8l+7; find the digit holding the target */
            uint32_t c[8], own = 0u;
            for (int t = 0; t < 8; ++t) {
                c[t] = sh.hist[8u * lane + t];
                own += c[t];
            }
            uint32_t incl = own;
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                if ((int)lane >= d) incl += v;
            }
            const uint32_t tgt = sh.target, excl = incl - own;
            if (tgt >= excl && tgt < incl) { /* exactly one lane */
                uint32_t run = excl, dsel = 8u * lane;
                for (int t = 0; t < 8; ++t) {
                    if (tgt < run + c[t]) {
                        dsel = 8u * lane + (uint32_t)t;
                        break;
                    }
                    run += c[t];
                }
                sh.target = tgt - run;
                sh.prefix |= (unsigned long long)dsel << shift;
                sh.mask |= 255ull << shift;
            }
        }
        __syncthreads();
    }
    return from_order_key_(sh.prefix);
}

__device__ double block_sum_(double v, double* s_red)
{
    for (int d = 16; d >= 1; d >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
    const uint32_t w = threadIdx.x >> 5, l = threadIdx.x & 31u;
    __syncthreads();
    if (l == 0) s_red[w] = v;
    __syncthreads();
    double t = 0.0;
    const uint32_t nw = blockDim.x >> 5;
    if (w == 0) {
        t = (l < nw) ? s_red[l] : 0.0;
        for (int d = 16; d >= 1; d >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, d);
        if (l == 0) s_red[0] = t;
    }
    __syncthreads();
    t = s_red[0];
    __syncthreads();
    return t;
}

__device__ double block_max_(double v, double* s_red)
{
    for (int d = 16; d >= 1; d >>= 1) v = fmax(v, __shfl_xor_sync(0xFFFFFFFFu, v, d));
    const uint32_t w = threadIdx.x >> 5, l = threadIdx.x & 31u;
    __syncthreads();
    if (l == 0) s_red[w] = v;
    __syncthreads();
    const uint32_t nw = blockDim.x >> 5;
    if (w == 0) {
        double t = (l < nw) ? s_red[l] : -INFINITY;
        for (int d = 16; d >= 1; d >>= 1) t = fmax(t, __shfl_xor_sync(0xFFFFFFFFu, t, d));
        if (l == 0) s_red[0] = t;
    }
    __syncthreads();
    double t = s_red[0];
    __syncthreads();
    return t;
}

/* start of a main iteration (simulation_impl.inl:202-222): count it, stop
 * once -S is exceeded (the count then stays at max + 1, as the reference's
 * meta reports), lower gamma on the delta schedule */
__device__ void start_generation_(JobPmcDev& pm)
{
    pm.iterations += 1u;
    if ((pm.max_generations && pm.iterations > pm.max_generations) || pm.generation >= PCS_MAX_GENERATION) {
        pm.done = 1u;
        return;
    }
    if (pm.schedule == 0u) pm.gamma -= pm.delta_gamma;
    pm.generation += 1u;
    pm.pending_count = pm.N;
    pm.trials = 0ull;
    pm.accepted_gen = 0ull;
    pm.gen_ended = 0u;
}

/* block_sum_ of K values at once, to s_out: the same sums in the same order,
 * with one pair of barriers, the second stages by K warps.  Threads from n
 * on hold zeros, so warps past n only write theirs (FP64 runs at one warp
 * instruction per ~16 cycles and SM: 32 warps' trees take 2600 cycles). */
template <uint32_t K>
__device__ void block_sums_(const double* v, uint32_t n, double (*s_part)[32], double* s_out)
{
    const uint32_t w = threadIdx.x >> 5, l = threadIdx.x & 31u, nw = blockDim.x >> 5;
    static_assert(K <= 32u, "a warp per value");
    __syncthreads(); /* s_part and s_out are read */
#pragma unroll
    for (uint32_t k = 0; k < K; ++k) {
        double t = v[k];
        if (32u * w < n)
            for (int d = 16; d >= 1; d >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, d);
        if (l == 0u) s_part[k][w] = t;
    }
    __syncthreads();
    if (w < K) {
        double t = l < nw ? s_part[w][l] : 0.0;
        for (int d = 16; d >= 1; d >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, d);
        if (l == 0u) s_out[w] = t;
    }
    __syncthreads();
}

/* finalize: a cluster of 8 CTAs per job whose generation ended this round.
 * What does not depend on one another runs at the same time: CTA 0 has the
 * weights and their cumulative sums (a serial chain), CTAs 1-6 the
 * perturbation factor's moments, CTA 7 the next epsilon (selection), the
 * population's commit and the slots' reset.  The moments with weights start
 * when the weights are there (one cluster barrier); after the last barrier
 * CTA 0 factorises the covariance and starts the next generation.  Bound by
 * chains of FP64 operations (a dependent addition every ~60 cycles, a warp
 * instruction per ~16 cycles and SM).  In one CTA, one after another: N = 256,
 * P = 4 52 us, N = 840, P = 7 119 us, N = 1024, P = 7 with the covariance
 * 195 us; here 22, 48 and 76
 * us (rounds' PMC kernels of a job: configuration 0 1.63 -> 1.29 ms,
 * configuration 1 1.57 -> 1.06 ms, four served jobs 2.30 -> 1.65 ms). */
constexpr uint32_t kWcumChunk = 1024;
constexpr uint32_t kFinCtas = 8, kFinMoments = 6; /* CTAs per cluster; of these for the moments */

__device__ __forceinline__ void fin_cluster_sync_()
{
    __syncwarp(); /* the barrier is the whole warp's */
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

/* s_wc[0 .. m) and acc become cumulative sums, by one thread in order; eight
 * values are read ahead of the chain (a load behind a store to the same array
 * waits for it: 110 cycles per value) */
__device__ __forceinline__ void wcum_chain_(double* s_wc, uint32_t m, double& acc)
{
    constexpr uint32_t U = 8;
    double v[U];
    uint32_t i = 0;
    if (m >= U)
#pragma unroll
        for (uint32_t t = 0; t < U; ++t) v[t] = s_wc[t];
    for (; i + U <= m; i += U) {
        double nx[U];
#pragma unroll
        for (uint32_t t = 0; t < U; ++t) nx[t] = s_wc[min(i + U + t, m - 1u)];
#pragma unroll
        for (uint32_t t = 0; t < U; ++t) {
            acc += v[t];
            s_wc[i + t] = acc;
        }
#pragma unroll
        for (uint32_t t = 0; t < U; ++t) v[t] = nx[t];
    }
    for (; i < m; ++i) {
        acc += s_wc[i];
        s_wc[i] = acc;
    }
}

/* pm.w: the new population's normalised weights */
__device__ __forceinline__ void fin_weights_(JobPmcDev& pm, double* s_red)
{
    const uint32_t N = pm.N, tid = threadIdx.x, bd = blockDim.x;
    double s = 0.0;
    if (pm.weighting == 0u) {
        double mx = -INFINITY;
        for (uint32_t i = tid; i < N; i += bd) mx = fmax(mx, pm.scratch[i]);
        mx = block_max_(mx, s_red);
        for (uint32_t i = tid; i < N; i += bd) {
            const double e = exp(pm.scratch[i] - mx);
            pm.scratch[i] = e;
            s += e;
        }
    } else {
        /* inverse-distance-squared (:872-887) */
        for (uint32_t i = tid; i < N; i += bd) {
            const double d = pm.dist_new[i];
            const double wv = 1.0 / (d * d);
            pm.scratch[i] = wv;
            s += wv;
        }
    }
    s = block_sum_(s, s_red);
    for (uint32_t i = tid; i < N; i += bd) pm.w[i] = pm.scratch[i] / s;
    __syncthreads();
}

/* cumulative weights (partial_sum, :222): one thread adds them in the
 * reference's order, from a shared-memory copy of each 1024-weight chunk */
__device__ __forceinline__ void fin_wcum_(JobPmcDev& pm, double* s_wc)
{
    const uint32_t N = pm.N, tid = threadIdx.x, bd = blockDim.x;
    double acc = 0.0; /* thread 0's running sum across chunks */
    for (uint32_t base = 0; base < N; base += kWcumChunk) {
        const uint32_t m = min(kWcumChunk, N - base);
        for (uint32_t i = tid; i < m; i += bd) s_wc[i] = pm.w[base + i];
        __syncthreads();
        if (tid == 0) wcum_chain_(s_wc, m, acc);
        __syncthreads();
        for (uint32_t i = tid; i < m; i += bd) pm.wcum[base + i] = s_wc[i];
        __syncthreads();
    }
}

/* compute_tau_ (:733-749) of parameters first, first + kFinMoments, ...:
 * tau = sqrt(2 var), uncorrected 1/N variance */
__device__ __forceinline__ void fin_tau_(JobPmcDev& pm, const double* theta, uint32_t first, double (*s_part)[32], double* s_out)
{
    const uint32_t N = pm.N, P = pm.P, tid = threadIdx.x, bd = blockDim.x;
    for (uint32_t p = first; p < P; p += kFinMoments) {
        double s = 0.0;
        for (uint32_t i = tid; i < N; i += bd) s += theta[(uint64_t)i * P + p];
        block_sums_<1>(&s, N, s_part, s_out);
        const double mean = s_out[0] / (double)N;
        double v = 0.0;
        for (uint32_t i = tid; i < N; i += bd) {
            const double x = theta[(uint64_t)i * P + p] - mean;
            v += x * x;
        }
        block_sums_<1>(&v, N, s_part, s_out);
        for (uint32_t q = tid; q < P; q += bd)
            pm.factor[p * P + q] = q == p ? sqrt(2.0 * (s_out[0] / (double)N)) : 0.0;
    }
}

/* 2 x weighted covariance (Beaumont et al. 2009), entries first, first +
 * kFinMoments, ... of the lower triangle row by row, into pm.factor */
__device__ __forceinline__ void fin_covariance_(JobPmcDev& pm, const double* theta, uint32_t first, double (*s_part)[32],
                                                double* s_out, double* s_mean)
{
    const uint32_t N = pm.N, P = pm.P, tid = threadIdx.x, bd = blockDim.x;
    constexpr uint32_t K = 4;
    for (uint32_t p0 = 0; p0 < P; p0 += K) { /* every CTA has all the means */
        double s[K] = {0.0, 0.0, 0.0, 0.0};
        for (uint32_t i = tid; i < N; i += bd) {
            const double wi = pm.w[i];
#pragma unroll
            for (uint32_t k = 0; k < K; ++k)
                if (p0 + k < P) s[k] += wi * theta[(uint64_t)i * P + p0 + k];
        }
        block_sums_<K>(s, N, s_part, s_out);
        if (tid < K && p0 + tid < P) s_mean[p0 + tid] = s_out[tid];
    }
    __syncthreads();
    const uint32_t pairs = P * (P + 1u) / 2u;
    for (uint32_t e0 = first; e0 < pairs; e0 += K * kFinMoments) {
        double s[K] = {0.0, 0.0, 0.0, 0.0};
        uint32_t pk[K], qk[K];
#pragma unroll
        for (uint32_t k = 0; k < K; ++k) {
            const uint32_t e = min(e0 + k * kFinMoments, pairs - 1u);
            uint32_t p = 0;
            while ((p + 1u) * (p + 2u) / 2u <= e) ++p;
            pk[k] = p;
            qk[k] = e - p * (p + 1u) / 2u;
        }
        for (uint32_t i = tid; i < N; i += bd) {
            const double* t = theta + (uint64_t)i * P;
            const double wi = pm.w[i];
#pragma unroll
            for (uint32_t k = 0; k < K; ++k)
                if (e0 + k * kFinMoments < pairs) s[k] += wi * (t[pk[k]] - s_mean[pk[k]]) * (t[qk[k]] - s_mean[qk[k]]);
        }
        block_sums_<K>(s, N, s_part, s_out);
        if (tid < K && e0 + tid * kFinMoments < pairs) {
            const uint32_t e = e0 + tid * kFinMoments;
            uint32_t p = 0;
            while ((p + 1u) * (p + 2u) / 2u <= e) ++p;
            const uint32_t q = e - p * (p + 1u) / 2u;
            pm.factor[p * P + q] = pm.factor[q * P + p] = 2.0 * s_out[tid];
        }
    }
}

/* pm.factor, a covariance, becomes its lower Cholesky factor (one thread) */
__device__ void fin_cholesky_(JobPmcDev& pm, double* s_cov)
{
    const uint32_t P = pm.P;
    for (uint32_t x = 0; x < P * P; ++x) {
        s_cov[x] = pm.factor[x];
        pm.factor[x] = 0.0;
    }
    for (uint32_t c = 0; c < P; ++c) {
        if (pm.fixed[c]) continue;
        double d = s_cov[c * P + c];
        for (uint32_t t = 0; t < c; ++t)
            if (!pm.fixed[t]) d -= pm.factor[c * P + t] * pm.factor[c * P + t];
        const double lv = sqrt(fmax(d, 1e-300));
        pm.factor[c * P + c] = lv;
        for (uint32_t r = c + 1; r < P; ++r) {
            if (pm.fixed[r]) continue;
            double s = s_cov[r * P + c];
            for (uint32_t t = 0; t < c; ++t)
                if (!pm.fixed[t]) s -= pm.factor[r * P + t] * pm.factor[c * P + t];
            pm.factor[r * P + c] = s / lv;
        }
    }
}

/* x, as this CTA's threads left it, to pinned host memory: the host reads it
 * when the round has ended (three copies behind the kernel took 10 us a round;
 * this takes 2.5) */
template <typename T>
__device__ __forceinline__ void report_(T& host, const T& x)
{
    static_assert(sizeof(T) % 4u == 0u, "words");
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < sizeof(T) / 4u; i += blockDim.x)
        reinterpret_cast<volatile uint32_t*>(&host)[i] = reinterpret_cast<const volatile uint32_t*>(&x)[i];
}

__global__ void __cluster_dims__(kFinCtas, 1, 1) __launch_bounds__(1024) k_finalize(PmcArgs a)
{
    __shared__ double s_red[32];
    __shared__ double s_wc[kWcumChunk];
    __shared__ double s_part[4][32], s_out[4];
    __shared__ double s_mean[PCS_MAX_P];
    __shared__ double s_cov[PCS_MAX_P * PCS_MAX_P];
    __shared__ SelectShared s_select;
    const uint32_t rank = blockIdx.x % kFinCtas, tid = threadIdx.x, bd = blockDim.x;
    const uint32_t n_jobs = a.round->n_jobs;
    for (uint32_t j = blockIdx.x / kFinCtas; j < n_jobs; j += gridDim.x / kFinCtas) {
        JobPmcDev& pm = a.pmc[j];
        if (pm.done || !pm.gen_ended) {
            if (rank == kFinCtas - 1u) report_(a.h_pmc[j], pm);
            continue;
        }
        const uint32_t N = pm.N, P = pm.P;
        /* generation 0: the prior pass's population stays as it was drawn */
        const bool commit = pm.generation != 0u, covariance = pm.perturbation != 0u;
        if (commit && (double)pm.trials >= (double)pm.avg_trials * (double)pm.N) {
            /* trial cap: converged, discard this generation (:425-428); the
             * other CTAs pass the job by whether they see this or not */
            if (rank == kFinCtas - 1u) {
                __syncthreads(); /* the CTA has read them */
                if (tid == 0) {
                    pm.converged = 1u;
                    pm.done = 1u;
                }
                report_(a.h_pmc[j], pm);
            }
            continue;
        }
        const double* theta = commit ? pm.theta_new : pm.theta;
        double gamma = pm.gamma; /* CTA 0: the old one */
        if (rank == 0u) {
            if (commit) fin_weights_(pm, s_red);
            if (covariance) fin_cluster_sync_();
            fin_wcum_(pm, s_wc);
        } else if (rank <= kFinMoments) {
            if (covariance) {
                fin_cluster_sync_(); /* the weights */
                fin_covariance_(pm, theta, rank - 1u, s_part, s_out, s_mean);
            } else {
                fin_tau_(pm, theta, rank - 1u, s_part, s_out);
            }
        } else {
            if (covariance) fin_cluster_sync_();
            /* gamma_0 from the median distance (compute_initial_gamma_
             * :819-829), or the next epsilon of the quantile schedule */
            if (!commit || pm.schedule == 1u) {
                const uint32_t target = pm.schedule == 1u ? min(N - 1u, (uint32_t)floor(pm.quantile * N)) : N / 2u;
                gamma = select_rank_(pm.dist_new, N, target, s_select);
            }
            /* commit the new population (:434-450); the quantile schedule
             * keeps the prior pass's distances as the generation-0 distances */
            if (commit)
                for (uint64_t i = tid; i < (uint64_t)N * P; i += bd) pm.theta[i] = pm.theta_new[i];
            for (uint32_t i = tid; i < N; i += bd) {
                pm.dist[i] = commit || pm.schedule == 1u ? pm.dist_new[i] : 0.0;
                pm.pending[i] = i;
                pm.next_trial[i] = 0u;
                pm.accepted[i] = 0u;
            }
        }
        fin_cluster_sync_();
        if (rank == 0u && tid == 0 && covariance) fin_cholesky_(pm, s_cov);
        if (rank == kFinCtas - 1u) {
            if (tid == 0) {
                pm.gamma = gamma;
                start_generation_(pm);
            }
            report_(a.h_pmc[j], pm);
        }
        __syncthreads(); /* s_cov, s_out and the rest are free */
    }
    if (blockIdx.x == 0u) { /* no kernel from here on changes these */
        report_(*a.h_round, *a.round);
        report_(*a.h_err, *a.err);
    }
}

/* ----------------------------------------------------------------------- */
/* observed cumulative histogram (simulation_impl.inl:605-629) */
__global__ void k_observed_bin(const uint32_t* K, const double* DE, size_t n, uint32_t rows,
                               uint32_t bins, double ub_de, uint32_t* sat, uint32_t* err)
{
    const double width = ub_de / (double)bins;
    const uint64_t total = (uint64_t)rows * bins;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double de = DE[i];
        if (de >= ub_de) continue;
        const long long idx = (long long)(de / width);
        const long long flat = (long long)K[i] * bins + idx;
        if (flat < 0 || (unsigned long long)flat >= total) {
            atomicOr(err, PCS_ERRBIT_HIST_BOUNDS);
            continue;
        }
        atomicAdd(sat + flat, 1u);
    }
}

/* the Julia path's observed histogram (src/cpu/estimate.jl:32-40): kmax
 * rows for K = 1..kmax, bin ceil(DE / width) kept when in 1..bins, i.e.
 * (0, w] bins; a K outside 1..kmax sets the bounds bit (Julia throws). */
__global__ void k_observed_bin_julia(const uint32_t* K, const double* DE, size_t n, uint32_t kmax,
                                     uint32_t bins, double ub_de, uint32_t* sat, uint32_t* err)
{
    const double width = ub_de / (double)bins;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double q = ceil(DE[i] / width);
        if (!(q >= 1.0 && q <= (double)bins)) continue;
        const uint32_t k = K[i];
        if (k < 1u || k > kmax) {
            atomicOr(err, PCS_ERRBIT_HIST_BOUNDS);
            continue;
        }
        atomicAdd(sat + (uint64_t)(k - 1u) * bins + (uint64_t)q - 1u, 1u);
    }
}

/* Row-wise, then column-wise inclusive sums in place; the column pass also
 * writes the column-major copy (pairs of columns interleaved,
 * pcs_sat_t_index).  A few MB: what counts is how many loads are in flight.
 * Rows: a warp each, 32 cells (128 bytes) at a time, eight such loads issued
 * before the first is summed.  Columns: eight of them (one 32-byte sector)
 * per CTA, 128 threads down each: a thread sums its share of the rows, the
 * shares are scanned in shared memory, and the rows are read again (from L2)
 * with their running sums.  One thread per column and one per row, each
 * waiting for its loads in turn, took 430 and 114 us for 1001 x 1000 cells;
 * these take 7 and 6 us. */
constexpr uint32_t kSatRowWarps = 8;
constexpr uint32_t kSatCols = 8, kSatParts = 128;

__global__ void __launch_bounds__(32 * kSatRowWarps) k_observed_rows(uint32_t rows, uint32_t bins, uint32_t* sat)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t r = blockIdx.x * kSatRowWarps + (threadIdx.x >> 5);
    if (r >= rows) return; /* whole warp */
    uint32_t* row = sat + (uint64_t)r * bins;
    uint32_t run = 0u;
    for (uint32_t c0 = 0; c0 < bins; c0 += 256u) {
        uint32_t v[8];
#pragma unroll
        for (uint32_t i = 0; i < 8u; ++i) v[i] = c0 + 32u * i + lane < bins ? row[c0 + 32u * i + lane] : 0u;
#pragma unroll
        for (uint32_t i = 0; i < 8u; ++i) {
            uint32_t s = v[i];
            for (uint32_t d = 1; d < 32u; d <<= 1) {
                const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, s, d);
                if (lane >= d) s += t;
            }
            s += run;
            run = __shfl_sync(0xFFFFFFFFu, s, 31);
            if (c0 + 32u * i + lane < bins) row[c0 + 32u * i + lane] = s;
        }
    }
}

__global__ void __launch_bounds__(kSatCols * kSatParts) k_observed_cols(uint32_t rows, uint32_t bins, uint32_t* sat,
                                                                         uint32_t* sat_t)
{
    __shared__ uint32_t s_part[kSatParts][kSatCols];
    const uint32_t x = threadIdx.x % kSatCols, y = threadIdx.x / kSatCols;
    const uint32_t c = blockIdx.x * kSatCols + x;
    const uint32_t per = (rows + kSatParts - 1u) / kSatParts;
    const uint32_t r0 = min(rows, y * per), r1 = min(rows, r0 + per);
    uint32_t sum = 0u;
    if (c < bins) {
#pragma unroll 8
        for (uint32_t r = r0; r < r1; ++r) sum += sat[(uint64_t)r * bins + c];
    }
    s_part[y][x] = sum;
    __syncthreads();
    for (uint32_t d = 1; d < kSatParts; d <<= 1) { /* inclusive scan of the shares */
        const uint32_t t = y >= d ? s_part[y - d][x] : 0u;
        __syncthreads();
        s_part[y][x] += t;
        __syncthreads();
    }
    uint32_t acc = s_part[y][x] - sum;
    if (c >= bins) return;
#pragma unroll 4
    for (uint32_t r = r0; r < r1; ++r) {
        acc += sat[(uint64_t)r * bins + c];
        sat[(uint64_t)r * bins + c] = acc;
        if (sat_t) sat_t[pcs_sat_t_index(r, c, rows, bins)] = acc;
    }
}

static void launch_sat_sums_(uint32_t rows, uint32_t bins, uint32_t* sat, uint32_t* sat_t, cudaStream_t st)
{
    k_observed_rows<<<(rows + kSatRowWarps - 1) / kSatRowWarps, 32 * kSatRowWarps, 0, st>>>(rows, bins, sat);
    k_observed_cols<<<(bins + kSatCols - 1) / kSatCols, kSatCols * kSatParts, 0, st>>>(rows, bins, sat, sat_t);
}

/* ----------------------------------------------------------------------- */
cudaError_t launch_round_plan(const PmcArgs& a, cudaStream_t st)
{
    k_round_plan<<<1, kMaxRoundJobs, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_propose(const PmcArgs& a, uint32_t capacity, cudaStream_t st)
{
    k_propose<<<(capacity + kProposePairs - 1) / kProposePairs, 64 * kProposePairs, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_items(const PmcArgs& a, cudaStream_t st)
{
    k_items<<<1, 1024, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_accept(const PmcArgs& a, uint32_t n_jobs, cudaStream_t st)
{
    k_accept<<<n_jobs, 1024, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_finalize(const PmcArgs& a, uint32_t n_jobs, uint32_t max_n, cudaStream_t st)
{
    /* grids for one job's points; the kernels stride over the round's jobs */
    k_whiten<<<(2u * max_n + 255) / 256, 256, 0, st>>>(a);
    k_kernel_sum<<<(max_n * 32u + 255) / 256, 256, 0, st>>>(a);
    k_finalize<<<(n_jobs + kFinCtas - 1u) / kFinCtas * kFinCtas, 1024, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_observed_sat(const uint32_t* K, const double* DE, size_t n, uint32_t rows,
                                uint32_t bins, double ub_de, uint32_t* sat, uint32_t* sat_t,
                                uint32_t* err, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(sat, 0, sizeof(uint32_t) * (size_t)rows * bins, st);
    if (e != cudaSuccess) return e;
    if (n) k_observed_bin<<<(unsigned)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096), 256, 0, st>>>(K, DE, n, rows, bins, ub_de, sat, err);
    launch_sat_sums_(rows, bins, sat, sat_t, st);
    return cudaGetLastError();
}

cudaError_t launch_observed_sat_julia(const uint32_t* K, const double* DE, size_t n, uint32_t kmax,
                                      uint32_t bins, double ub_de, uint32_t* sat, uint32_t* err, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(sat, 0, sizeof(uint32_t) * (size_t)kmax * bins, st);
    if (e != cudaSuccess) return e;
    if (n) k_observed_bin_julia<<<(unsigned)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096), 256, 0, st>>>(K, DE, n, kmax, bins, ub_de, sat, err);
    launch_sat_sums_(kmax, bins, sat, nullptr, st);
    return cudaGetLastError();
}

} // namespace pcs
