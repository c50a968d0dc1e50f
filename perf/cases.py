"""Performance cases: the work a user of this framework has it do, through its
public entry points, over the range of sizes it is used on.

Kinds of case
  forward          simulate_hist: the forward model of `count` proposals (host
                   arguments in, host histograms out)
  distance         scan_distance: cumulative histogram distances of host
                   histograms, optionally with the double sum, the exact
                   integer sum and the prefix sums
  distance_device  pcs_scan_distance_noalloc: the same distances for histograms
                   that are on the GPU already (a caller with its own
                   allocator); the call consumes its histograms, so a pass
                   first copies them into the work buffer
  observed         observed_sat: the observed cumulative histogram of track lists
  job              make_simulation(...).run().output(): one whole estimation
                   (prior pass and generations) from host data to host population
  serve            Server: several jobs sharing batched rounds until all are done

Shapes are those of part_conc_spt_abc_gb300.workloads (configurations 0, 1, 3
and the serving stream), of the reference's input file as the posterior
fixtures state it (discrete mixtures, 1000 DE bins, delta schedule) and ranges
around them.  Everything that is drawn comes from the seed.
"""
import ctypes
import math

import numpy as np
import torch

import part_conc_spt_abc_gb300 as P
from part_conc_spt_abc_gb300 import workloads as W

OPS_PER_STEP = 105.0  # algorithmic operations of one particle-step: draws, Box-Muller, step, detection

_CTX = []


def _ctx():
    """The one context that a user's program opens on its GPU."""
    if not _CTX:
        _CTX.append(P.Context(0))
    return _CTX[0]


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def listed():
    return [
        # one proposal of configuration 0 (20 videos x 200 frames, 128 particles per video): a
        # user trying parameters by hand; half a million particle-steps, launches and copies count
        dict(name="forward-one", kind="forward", model="lognormal", C=1, videos=20, frames=200, ragged=False,
             bins=100, particles=128, count=1),
        # one proposal of configuration 3, the largest forward model that is used: 1e5 particles
        # per video, 100 videos x 1000 frames, 1e10 particle-steps
        dict(name="forward-large", kind="forward", model="lognormal", C=3, videos=100, frames=1000, ragged=False,
             bins=256, particles=100000, count=1),
        # the reference's discrete mixture with a depth per component, videos of differing
        # lengths, 1000 DE bins: a handful of proposals checked against measured data
        dict(name="forward-ragged", kind="forward", model="variable", C=3, videos=25, frames=397, ragged=True,
             bins=1000, particles=333, count=7),
        # one histogram of configuration 0 from the host: the smallest call there is
        dict(name="distance-one", kind="distance", rows=201, bins=100, count=1, f64=False, ssd=False, cum=False),
        # tall histograms with every sum and the prefix sums: parity and inspection work
        dict(name="distance-full", kind="distance", rows=1001, bins=256, count=16, f64=True, ssd=True, cum=True),
        # a round of configuration 1 (population 1024, 301 x 128) on the device
        dict(name="distance-round", kind="distance_device", rows=301, bins=128, count=1024),
        # tall, odd-sized histograms, fewer than SMs, on the device
        dict(name="distance-tall", kind="distance_device", rows=997, bins=255, count=61),
        # the reference's own data file in size: 38302 tracks into 1001 x 1000 cells
        dict(name="observed", kind="observed", rows=1001, bins=1000, tracks=38302, julia=False),
        # configuration 0 from start to end: short rounds, where launches and the PMC step count
        dict(name="job-short", kind="job", model="lognormal", C=1, videos=20, frames=200, bins=100, pop=256,
             generations=8, weighting=0, cholesky=False, double=False),
        # configuration 1's prior pass and three generations: full rounds
        dict(name="job-full", kind="job", model="lognormal", C=2, videos=50, frames=300, bins=128, pop=1024,
             generations=3, weighting=0, cholesky=True, double=False),
        # the reference's discrete fixed-depth model, delta schedule, 1000 DE bins,
        # inverse-distance-squared weights, double distance (accel -dt d)
        dict(name="job-discrete", kind="job", model="fixed", C=2, videos=25, frames=200, bins=1000, pop=1000,
             generations=3, weighting=1, cholesky=False, double=True),
        # four jobs of the serving stream's sizes sharing rounds
        dict(name="serve-mix", kind="serve", jobs=4, frames=200, bins=160, pop=700, generations=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "distance", "distance_device", "observed", "job", "job", "serve"])
    if kind == "forward":
        frames, videos, count = _log_int(rng, 20, 1000), _log_int(rng, 5, 100), _log_int(rng, 1, 64)
        most = min(1e5, 5e9 / (frames * videos * count))
        return dict(kind=kind, model=rng.choice(["lognormal", "fixed", "variable"]), C=rng.randint(1, 3), videos=videos,
                    frames=frames, ragged=rng.random() < 0.3, bins=_log_int(rng, 48, 1000),
                    particles=_log_int(rng, 30, max(31.0, most)), count=count)
    if kind == "distance":
        rows, bins = _log_int(rng, 40, 2001), _log_int(rng, 33, 1000)
        count = _log_int(rng, 1, max(1.01, min(60.0, 4.2e6 / (rows * bins))))
        more = rng.random() < 0.5
        return dict(kind=kind, rows=rows, bins=bins, count=count, f64=more, ssd=more, cum=more and rng.random() < 0.5)
    if kind == "distance_device":
        rows, bins = _log_int(rng, 40, 1400), _log_int(rng, 33, 700)
        return dict(kind=kind, rows=rows, bins=bins, count=_log_int(rng, 1, max(1.01, min(4096.0, 8e7 / (rows * bins)))))
    if kind == "observed":
        return dict(kind=kind, rows=_log_int(rng, 40, 1200), bins=_log_int(rng, 48, 1000),
                    tracks=_log_int(rng, 500, 400000), julia=rng.random() < 0.3)
    if kind == "job":
        model = rng.choice(["lognormal", "lognormal", "fixed", "variable"])
        return dict(kind=kind, model=model, C=rng.randint(1, 3), videos=_log_int(rng, 5, 30), frames=_log_int(rng, 50, 300),
                    bins=_log_int(rng, 48, 300), pop=_log_int(rng, 64, 800), generations=rng.randint(1, 3),
                    weighting=int(rng.random() < 0.25), cholesky=rng.random() < 0.25, double=rng.random() < 0.25)
    return dict(kind=kind, jobs=rng.randint(2, 4), frames=_log_int(rng, 100, 250), bins=rng.randint(64, 256),
                pop=_log_int(rng, 256, 600), generations=rng.randint(1, 3))


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

# the reference's input and data files, as the posterior fixtures state them
REF_BOX, REF_AREA, REF_DT, REF_UB_DE, REF_KMIN = (80.0, 80.0, 20.0), (61.6448, 61.6448), 0.068, 5.0, 3
REF_VOLUME_ML = REF_BOX[0] * REF_BOX[1] * REF_BOX[2] / 1e12
LOG_VOLUME_ML = W.BOX[0] * W.BOX[1] * W.BOX[2] / 1e12


def _forward(case, rng):
    """Setup and runs of a forward case: proposals as an estimation makes them,
    their parameters spread around the configurations' truths."""
    C, V, F = case["C"], case["videos"], case["frames"]
    frames = rng.integers(1, F + 1, V).astype(np.uint32) if case["ragged"] else np.full(V, F, np.uint32)
    frames[0] = F
    w = rng.dirichlet(np.full(C, 4.0))
    runs = []
    if case["model"] == "lognormal":
        setup = W.forward_setup(frames, case["bins"], C=C)
        for q in range(case["count"]):
            mu = np.sort(rng.uniform(100.0, 600.0, C))
            parts = rng.poisson(case["particles"] * rng.uniform(0.8, 1.25) if case["count"] > 1 else case["particles"], V)
            runs.append(W.lognormal_run(parts, mu, 0.05 * mu, w, slot=q, trial=1, generation=1))
    else:
        variable = case["model"] == "variable"
        setup = P.ForwardSetup(P.MODEL_DISCRETE_VARIABLE_DEPTH if variable else P.MODEL_DISCRETE_FIXED_DEPTH, C, frames,
                               REF_KMIN, float(np.float32(4.0) * np.float32(REF_DT)),
                               tuple(float(np.float32(0.5 * x)) for x in REF_BOX),
                               tuple(float(np.float32(0.5 * x)) for x in REF_AREA),
                               float(np.float32(REF_UB_DE / case["bins"])), F + 1, case["bins"])
        for q in range(case["count"]):
            m = np.sort(rng.uniform(0.3, 4.5, C))
            pre = np.cumsum(w).astype(np.float32)
            pre[-1] = 2.0
            half_az = 0.5 * rng.uniform(1.5, 2.5, C if variable else 1)
            parts = rng.poisson(case["particles"] * rng.uniform(0.8, 1.25), V)
            runs.append(P.ForwardRun(parts.astype(np.uint32), half_az.astype(np.float32), pre,
                                     np.sqrt(2.0 * m * REF_DT).astype(np.float32), None, q, 1, 1))
    return setup, runs


def _track_hist(rows, bins, count, tracks, seed, tail):
    """Histograms [count, rows, bins] (int32, GPU) of about `tracks` tracks: lengths fall off
    geometrically, DE is spread around the middle of its range and narrows with the length."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.arange(rows, device="cuda", dtype=torch.float32)
    b = (torch.arange(bins, device="cuda", dtype=torch.float32) + 0.5) / bins
    pk = torch.exp(-k / tail)
    width = 0.05 + 0.2 / torch.sqrt(k + 1.0)
    pb = torch.exp(-0.5 * ((b[None, :] - 0.2) / width[:, None]) ** 2)
    rate = pk[:, None] * pb
    rate[:2] = 0.0  # kmin 2
    rate *= tracks / rate.sum()
    out = torch.empty((count, rows, bins), dtype=torch.int32, device="cuda")
    for q0 in range(0, count, 64):
        n = min(64, count - q0)
        s = torch.rand(n, generator=g, device="cuda") + 0.5
        out[q0:q0 + n] = torch.poisson(rate[None] * s[:, None, None], generator=g).to(torch.int32)
    return out


def _distance_data(case, seed):
    rows, bins = case["rows"], case["bins"]
    hist = _track_hist(rows, bins, case["count"], 9000.0, 2 * seed + 1, 12.0)
    ref = _track_hist(rows, bins, 1, 9000.0, 2 * seed + 2, 14.0)[0]
    return hist, torch.cumsum(torch.cumsum(ref, 0), 1).to(torch.int32)


def _observed_data(case, seed):
    rng = np.random.default_rng(seed)
    kmax = case["rows"] if case["julia"] else case["rows"] - 1
    K = np.minimum(rng.geometric(0.08, case["tracks"]) + 1, kmax).astype(np.uint32)
    return K, rng.gamma(2.0, 0.6, case["tracks"])


def _job_input(case, seed):
    """An Input whose observed data is the forward model's own output at parameters drawn from the seed."""
    ctx, rng = _ctx(), np.random.default_rng(seed)
    C = case["C"]
    w = (np.array([0.6, 0.4, 0.3])[:C] if C > 1 else np.ones(1)) * rng.uniform(0.9, 1.1, C)
    if case["model"] == "lognormal":
        mu = np.sort(np.array([175.0, 500.0, 300.0])[:C] * rng.uniform(0.9, 1.1, C)).tolist()
        sd = [0.055 * m for m in mu]
        conc = (2e14 if C == 1 else 5e14) * rng.uniform(0.9, 1.1)
        inp, _ = W.make_problem(ctx, mu, sd, conc, w.tolist(), case["videos"], case["frames"], case["bins"], case["pop"],
                                case["generations"], seed=seed)
    else:
        f = dict(kind="forward", model=case["model"], C=C, videos=case["videos"], frames=case["frames"], ragged=False,
                 bins=case["bins"], particles=1.2e9 * C * REF_VOLUME_ML, count=1)
        setup, runs = _forward(f, rng)
        K, DE = W.observed_from_hist(P.simulate_hist(ctx, setup, runs, seed=seed)[0], REF_UB_DE)
        p = P.params_defaults()
        p.model, p.component_count, p.kmin, p.de_bin_count = setup.model, C, REF_KMIN, case["bins"]
        p.abc_sample_count, p.avg_trial_count, p.gamma_adaptive = case["pop"], 500, 1
        p.Lx, p.Ly, p.Lz = REF_BOX
        p.ub_de, p.lb_m, p.ub_m, p.lb_c, p.ub_c = REF_UB_DE, 0.1, 5.0, 5e8, 5e9
        p.lb_az, p.ub_az = (1.0, 3.0) if case["model"] == "variable" else (2.0, 2.0)
        p.delta_gamma, p.max_generations = 0.2, case["generations"]
        inp = P.Input(p, REF_AREA[0], REF_AREA[1], REF_DT, np.full(case["videos"], case["frames"], np.uint64), K, DE)
    inp.params.weighting_scheme = case["weighting"]
    if case["cholesky"]:
        inp.params.perturbation = P.PERTURB_CHOLESKY
    inp.params.distance_double = int(case["double"])
    return inp


def _serve_jobs(case, seed):
    """Jobs around the case's sizes, as the serving stream draws them."""
    rng, jobs = np.random.default_rng(seed), []
    scale = np.linspace(0.7, 1.2, case["jobs"])  # the sizes differ from job to job, not from seed to seed
    for j in range(case["jobs"]):
        C = 1 + j % 2
        mu = np.sort(rng.uniform(150.0, 700.0, C)).tolist()
        inp, _ = W.make_problem(_ctx(), mu, [0.05 * m for m in mu], rng.uniform(2e14, 5e14), [1.0] * C, 20,
                                int(case["frames"] * scale[j]), int(case["bins"] * scale[-1 - j]),
                                int(case["pop"] * scale[j]), case["generations"], seed=seed + j, prior_mu=(100.0, 800.0))
        jobs.append(inp)
    return jobs


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, kind=kind, seed=seed, ctx=_ctx())
    if kind == "forward":
        s["setup"], s["runs"] = _forward(case, np.random.default_rng(seed))
    elif kind in ("distance", "distance_device"):
        hist, ref = _distance_data(case, seed)
        if kind == "distance":
            s["hist"], s["ref"] = hist.cpu().numpy().view(np.uint32), ref.cpu().numpy().view(np.uint32)
        else:
            s["hist"], s["ref"] = hist, ref
            s["work"] = torch.zeros_like(hist)
            s["dist"] = torch.zeros(case["count"], dtype=torch.float32, device="cuda")
    elif kind == "observed":
        s["K"], s["DE"] = _observed_data(case, seed)
    elif kind == "job":
        s["input"] = _job_input(case, seed)
    else:
        s["jobs"] = _serve_jobs(case, seed)
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------

def _population(sim):
    o, i = sim.output(), sim.info()
    r = dict(m=o.m, c=o.c, az=o.az, dist=o.dist, w=o.w, gamma=float(i.gamma), iterations=int(i.iterations),
             converged=bool(i.converged), trials=int(i.trials), accepted=int(i.accepted))
    if o.s is not None:
        r["s"] = o.s
    return r


def run(state):
    kind, case, ctx = state["kind"], state["case"], state["ctx"]
    if kind == "forward":
        # counts are uint32; the same bits as int32, which every consumer of numpy arrays takes
        return P.simulate_hist(ctx, state["setup"], state["runs"], seed=state["seed"]).view(np.int32)
    if kind == "distance":
        r = P.scan_distance(ctx, state["hist"], state["ref"], want_cum=case["cum"], want_f64=case["f64"],
                            want_ssd=case["ssd"])
        if case["cum"]:
            r["cum"] = r["cum"].view(np.int32)
        return r
    if kind == "distance_device":
        state["work"].copy_(state["hist"])
        P._lib.check(P.lib().pcs_scan_distance_noalloc(
            ctypes.c_void_p(state["work"].data_ptr()), ctypes.c_void_p(state["ref"].data_ptr()), case["rows"], case["bins"],
            case["count"], ctypes.c_void_p(state["dist"].data_ptr()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "pcs_scan_distance_noalloc")
        return dict(dist=state["dist"], hist=state["work"])
    if kind == "observed":
        return P.observed_sat(ctx, state["K"], state["DE"], case["rows"], case["bins"], REF_UB_DE,
                              julia=case["julia"]).view(np.int32)
    if kind == "job":
        sim = P.make_simulation(ctx, state["input"], state["seed"])
        sim.run()
        r = _population(sim)
        sim.close()
        return r
    srv = P.Server(ctx)
    sims = [P.make_simulation(ctx, inp, state["seed"] + j) for j, inp in enumerate(state["jobs"])]
    for sim in sims:
        srv.submit(sim)
    while srv.step():
        pass
    r = [_population(sim) for sim in sims]
    for sim in sims:
        sim.close()
    return r


# --------------------------------------------------------------------------
# what a pass cannot do without, and the outputs in 64 bits
# --------------------------------------------------------------------------

def _job_work(case):
    """At least one proposal per population slot and generation, the prior pass included: its
    particle-steps at the prior's mean concentration, its histogram written, read and compared once."""
    lo, hi, vol = (1e7, 1e9, LOG_VOLUME_ML) if case["model"] == "lognormal" else (5e8, 5e9, REF_VOLUME_ML)
    lam = case["C"] * (hi - lo) / math.log(hi / lo) * vol
    proposals = case["pop"] * (case["generations"] + 1)
    steps = proposals * lam * case["videos"] * case["frames"]
    cells = proposals * (case["frames"] + 1) * case["bins"]
    return dict(bytes=8.0 * cells, flops=OPS_PER_STEP * steps + 5.0 * cells)


def work(case):
    kind = case["kind"]
    if kind == "forward":
        frames = (case["frames"] + 1) / 2 if case["ragged"] else case["frames"]
        steps = float(case["particles"]) * case["videos"] * frames * case["count"]
        return dict(bytes=4.0 * (case["frames"] + 1) * case["bins"] * case["count"] + 4.0 * case["videos"] * case["count"],
                    flops=OPS_PER_STEP * steps)
    cells = float(case.get("rows", 0)) * case.get("bins", 0)
    if kind == "distance":
        n = case["count"]
        return dict(bytes=4.0 * cells * (n + 1 + (n if case["cum"] else 0)), flops=5.0 * cells * n)
    if kind == "distance_device":  # the work buffer filled, then read and reset
        return dict(bytes=4.0 * cells * (4 * case["count"] + 1), flops=5.0 * cells * case["count"])
    if kind == "observed":
        return dict(bytes=4.0 * cells + 12.0 * case["tracks"], flops=2.0 * cells)
    if kind == "job":
        return _job_work(case)
    total = dict(bytes=0.0, flops=0.0)
    scale = np.linspace(0.7, 1.2, case["jobs"])
    for j in range(case["jobs"]):
        w = _job_work(dict(model="lognormal", C=1 + j % 2, videos=20, frames=int(case["frames"] * scale[j]),
                           bins=int(case["bins"] * scale[-1 - j]), pop=int(case["pop"] * scale[j]),
                           generations=case["generations"]))
        total = {k: total[k] + w[k] for k in total}
    return total


def exact(case, seed):
    """Distances in 64 bits.  Histograms and prefix sums are whole numbers; an
    estimation's population follows from random draws and has no such value."""
    if case["kind"] not in ("distance", "distance_device"):
        return None
    hist, ref = _distance_data(case, seed)
    d = torch.empty(case["count"], dtype=torch.float64, device="cuda")
    for q in range(case["count"]):
        cum = torch.cumsum(torch.cumsum(hist[q].to(torch.int64), 0), 1)
        d[q] = (cum - ref).to(torch.float64).square().sum()
    if case["kind"] == "distance_device":
        return dict(dist=d, hist=None)
    d = d.cpu().numpy()
    out = dict(dist_f32=d)
    if case["cum"]:
        out["cum"] = None
    if case["f64"]:
        out["dist_f64"] = d
    if case["ssd"]:
        out["ssd"] = [None] * case["count"]
    return out
