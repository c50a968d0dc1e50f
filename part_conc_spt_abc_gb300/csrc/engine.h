/*
 * engine.h -- host runtime of the GB300 ABC-PMC engine (C++17).
 *
 * Replaces the reference's SimulationT orchestration
 * (src/gpu/simulation_impl.cuh:135-374, detail/simulation_impl.inl) with a
 * device-resident design: a job's population, weights and observed
 * histogram live in one device arena; the host only plans rounds, launches a
 * captured CUDA graph per round and reads a small status table back.
 */
#ifndef PCS_ENGINE_H
#define PCS_ENGINE_H

#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <cstdint>
#include <deque>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/pcs.h"
#include "pcs_common.h"
#include "pcs_kernels.h"

namespace pcs {

/* Error carried to the C ABI as a status + message. */
struct Error : std::runtime_error {
    pcs_status status;
    Error(pcs_status s, const std::string& m) : std::runtime_error(m), status(s) {}
};

void cuda_check(cudaError_t e, const char* what);
#define PCS_CUDA(x) ::pcs::cuda_check((x), #x)

/* device allocation owned by the engine */
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void alloc(size_t n);
    void release();
    template <class T> T* as() const { return static_cast<T*>(p); }
};

/* Memory that the standalone entry points keep between calls: device memory
 * up to kKeep bytes (allocating and freeing nine buffers took 30-40 us of a
 * 90 us call) and a pinned page for small transfers.  One call at a time
 * holds it (Lease); a call that finds it taken by another thread, or needs
 * more, allocates its own for the call.  Given back at pcs_close, and when
 * another allocation of the context fails: its jobs', the plain form's
 * (alloc) or that of a call which needs more.  Under a cap on the serve
 * loop's memory, which does not count it, nothing is kept. */
struct Workspace {
    static const size_t kKeep = 64ull << 20, kPinned = 64ull << 10;
    std::mutex mu;
    DevBuf dev;
    char* pinned = nullptr;
    std::atomic<bool> keep{true};

    /* false: what is kept is given back, at once or at the end of the call
     * that holds it, and calls allocate their own from then on */
    void set_keep(bool k);
    /* frees the device memory; false if there is none or a call holds it */
    bool give_back();
    /* b.alloc(n); if that fails, once more after give_back() */
    void alloc(DevBuf& b, size_t n);
};

class Lease {
public:
    /* bytes: the sum of need<T>(n) over the get<T>(n) that follow */
    Lease(Workspace& ws, cudaStream_t stream, size_t bytes);
    ~Lease();
    Lease(const Lease&) = delete;
    Lease& operator=(const Lease&) = delete;
    template <class T> static size_t need(size_t n) { return (n * sizeof(T) + 255u) / 256u * 256u; }
    template <class T> T* get(size_t n) { return static_cast<T*>(take(need<T>(n))); }
    /* pinned memory for `n` bytes of this call, or NULL (none left, or taken) */
    char* stage(size_t n);
    /* the call's work on the stream has completed */
    void done() { done_ = true; }

private:
    void* take(size_t bytes);
    void own_alloc_();
    Workspace& ws_;
    cudaStream_t stream_;
    std::unique_lock<std::mutex> held_;
    DevBuf own_;
    char* base_ = nullptr;
    size_t size_ = 0, used_ = 0, staged_ = 0;
    bool done_ = false;
};

struct Tuning {
    uint32_t block = 256;
    uint32_t ppt = 1;
    uint32_t tile_rows = 0; /* 0: no shared-memory tile, warps take their own slices of the items */
    uint32_t aggregate = 0;
    uint32_t chunk = 256;
    uint32_t capacity = 2048;
    uint32_t max_spec = 4096;
    uint32_t use_graphs = 1;
    uint32_t plain_launch = 1; /* 1 reference geometry, 2 persistent grid */
    uint32_t round_fill = 0; /* particles a round is topped up to (0: none); set to one wave at open */
    uint32_t walk = 2; /* forward-model walk on Philox streams: 1 slab-split, 2 per step */
    uint32_t job_order = 2; /* capacity order among jobs: 1 admission, 2 least remaining work first */
};

struct Job;

/* Round buffers shared by all jobs of a round (sized by capacity). */
struct RoundBufs {
    uint32_t capacity = 0, items_cap = 0, v_max = 0, max_rows = 0, max_n = 0;
    uint64_t counts_cap = 0, hist_cap = 0, ystride = 0;
    DevBuf round, props, theta_prop, counts, item_prop, hist, dist32, dist64, jobs, pmc;
    DevBuf tmaps; /* [kMaxRoundJobs] TmapDev: each job's histogram tensor map over hist */
};

struct Ctx {
    int device = 0;
    int sm_count = 0;
    int inflight = 1;
    cudaStream_t stream = nullptr;
    Tuning tune;
    DevBuf err;              /* device error word */
    DevBuf sim_tasks;        /* slab-split task counter (u64, cumulative) */
    DevBuf logfact;          /* [kLogFactEntries] log(k!) from the host's lgamma */
    uint64_t sim_tasks_base = 0;
    Workspace ws;
    uint32_t* h_err = nullptr;
    RoundBufs rb;
    JobPmcDev* h_status = nullptr; /* pinned: the jobs' states, written by k_finalize */
    RoundDev* h_round = nullptr;   /* pinned */
    cudaGraphExec_t graph = nullptr;
    bool graph_dirty = true;
    std::vector<Job*> table;       /* jobs in the round table (index = table slot) */
    std::deque<Job*> queue;        /* serve: submitted, not yet admitted */
    uint32_t rb_max_b_ = 0;        /* widest histogram row among admitted jobs */
    bool rb_f64_ = false;          /* some admitted job's distances are double */
    bool rb_narrow_ = false;       /* distance_mostly_narrow of the admitted jobs */
    uint64_t mem_cap = 0;
    uint64_t mem_used = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEvent_t ev_sim0 = nullptr, ev_sim1 = nullptr, ev_dist0 = nullptr, ev_dist1 = nullptr;
    cudaEvent_t ev_pmc0 = nullptr, ev_pmc1 = nullptr;
    cudaEvent_t ev_t0 = nullptr, ev_t1 = nullptr;
    RoundDev* h_round_out = nullptr; /* pinned: the round counters, written by k_finalize */
    pcs_kernel_stats stats{};
    static const uint32_t kKernelsPerRound = 8; /* besides the distance's */
    uint32_t distance_kernels_ = 1;
    std::mutex mu;

    explicit Ctx(int dev, int inflight);
    ~Ctx();

    /* round machinery */
    void ensure_round_buffers(uint32_t v_max, uint32_t max_rows, uint32_t max_n, uint64_t rb_max);
    void upload_table();
    void look_at_widths();
    void enqueue_round();
    void run_round(double* ms_out);
    void admit(Job* j);
    void retire(Job* j);
    uint32_t sim_grid(uint32_t block, uint32_t ppt, bool agg, uint32_t tile_words, bool split = false) const;
    bool split_walk() const { return tune.walk == 1u; }
    uint64_t read_sim_tasks();
};

struct Job {
    Ctx* ctx = nullptr;
    pcs_params p{};
    double ax = 0, ay = 0, deltat = 0;
    std::vector<uint32_t> frames;
    std::vector<uint32_t> K;
    std::vector<double> DE;
    uint64_t seed = 0;
    uint32_t N = 0, P = 0, C = 0, Z = 0, V = 0, R = 0, B = 0;
    DevBuf arena;
    JobDev jd{};
    JobPmcDev pm{};        /* initial state uploaded at admission */
    JobPmcDev status{};    /* last status read back */
    int slot = -1;         /* index in the round table, -1 when not admitted */
    bool initialised = false;
    bool finished = false;
    bool in_serve = false;
    bool mem_counted = false; /* its arena is counted in the context's serve memory use */
    double device_ms = 0.0;
    std::chrono::steady_clock::time_point t_submit, t_done;

    Job(Ctx* c, const pcs_params& prm, const pcs_observed& obs, uint64_t sd);
    uint64_t arena_bytes() const;
    void build_device_state(); /* allocate arena, observed histogram, prior population */
    void output(double* m, double* s, double* c, double* az, double* dist, double* w) const;
    /* checkpoint.cpp: the job's state between rounds as a byte blob, and back */
    size_t checkpoint_bytes() const;
    void save_state(void* buf) const;
    void load_state(const void* buf, size_t bytes);
};

/* shared-memory histogram words for a tile of tile_rows rows of `bins` bins */
uint32_t tile_words_for(uint32_t tile_rows, uint32_t bins);

/* validates and normalises parameters; throws Error */
void validate(const pcs_params& p, const pcs_observed& o);

} // namespace pcs

struct pcs_ctx {
    std::unique_ptr<pcs::Ctx> impl;
};
struct pcs_job {
    std::unique_ptr<pcs::Job> impl;
};

#endif
