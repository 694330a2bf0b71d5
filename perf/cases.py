"""The work users have this package do, as measurable cases.

`listed()` names the cases, `draw(rng)` gives further ones of the same ranges; `prepare`
makes what a program has in hand before the call, `run` is one pass through the public
entry points, `work` the bytes and operations the pass cannot do without.  Every result of
the package is reproducible bit for bit (fp64 in one fixed operation order), so the
tolerance is "exact".

Kinds of cases:

  score     PlacementEvaluator.get_scores, or get_stats as the greedy steps call it, on a list
            of candidate placements (random ones, or "grown": all one step away from a
            half-filled placement, as a search layer makes)
  search    a serving case whose placement comes from a whole search (greedy or beam: hundreds
            of small dependent batches), then evaluated
  one       one placement on one trace with all per-request outputs, the drop-in for
            approximate_one_case_one_placement; mixed or one clock per group
  stats     approximate_one_case, statistics of the whole trace or with the warm-up cut off,
            one placement or a schedule of three, with or without batching
  batching  a list of placements through the batching simulator
  sweep     one placement scored on many traces, uploaded and simulated
  dense     the low-level drop-ins on the reference's dense tables
"""
import math
from functools import partial

import numpy as np

from mms_b200 import cases, engine, search, simulator
from mms_b200.placement import (ClusterEnv, ModelPlacement, ModelPlacementWithReplacement,
                                PlacementEvaluator, TraceSweep)
from mms_b200.profiling import GB, ParallelConfig

BATCH_SIZES = (1, 2, 4, 8)
MEM_BUDGET = 13 * GB


def _case(name, kind, devices, models, requests, rate, cv, slo, **more):
    c = {"kind": kind, "devices": devices, "models": models, "requests": requests,
         "rate": rate, "cv": cv, "slo": slo}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one step of a greedy chain on a toy cluster with a short trace: pure latency
        _case("score-one", "score", 4, 4, 2000, 12.0, 3.0, 5.0, candidates=1, shape="random",
              stats=True),
        # a small hand-made comparison on a training trace of ordinary length, odd count
        _case("score-37", "score", 16, 8, 30000, 30.0, 3.0, 5.0, candidates=37, shape="random",
              stats=True),
        # one generation of the evolutionary search
        _case("score-1025", "score", 16, 8, 30000, 30.0, 4.0, 5.0, candidates=1025,
              shape="random", stats=False),
        # the headline: 64 devices, 32 models, an hour-long trace, 4096 random placements
        _case("score-4096", "score", 64, 32, 180000, 50.0, 3.0, 5.0, candidates=4096,
              shape="random", stats=False),
        # one layer of the beam search on 64 devices and 56 models
        _case("layer-64", "score", 64, 56, 144000, 80.0, 4.0, 5.0, candidates=2343,
              shape="grown", stats=False),
        # a whole model-parallel placement search on 16 devices
        _case("search-16", "search", 16, 8, 30000, 30.0, 3.0, 5.0, policy="mp-search"),
        # 8 devices as pipelines of two, hour-long trace, per-request outputs
        _case("one-hour", "one", 8, 8, 57600, 16.0, 4.0, 5.0, mixed=True, batching=False),
        # final evaluation of a placement schedule: latency statistics, warm-up cut off
        _case("stats-schedule", "stats", 16, 8, 27000, 30.0, 3.0, 5.0, schedule=True,
              fast=False, batching=False),
        # final evaluation with dynamic batching
        _case("stats-batching", "stats", 16, 8, 27000, 30.0, 3.0, 5.0, schedule=False,
              fast=True, batching=True),
        # candidate placements compared under dynamic batching
        _case("batching-256", "batching", 64, 32, 45000, 50.0, 3.0, 5.0, candidates=256),
        # robustness of one placement: 48 traces of four rate scales and four CVs
        _case("sweep-48", "sweep", 64, 32, 83400, 278.0, 1.0, 5.0, traces=48),
        # the reference's kernel call itself, odd length
        _case("dense-10007", "dense", 16, 8, 10007, 30.0, 3.0, 5.0, batching=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("score", "score", "score", "search", "one", "stats", "batching", "sweep",
                       "dense"))
    devices = rng.choice((4, 8, 16, 32, 64))
    models = rng.randint(4, {4: 8, 8: 16, 16: 24, 32: 40, 64: 56}[devices])
    rate = round(devices * rng.uniform(0.6, 2.0), 2)
    cv, slo = rng.choice((1.0, 2.0, 3.0, 4.0)), rng.choice((2.0, 3.0, 5.0, 8.0))
    if kind == "score":
        requests = _log(rng, 1000, 180000)
        candidates = min(_log(rng, 1, 4096), max(1, 250_000_000 // requests))
        return _case(None, kind, devices, models, requests, rate, cv, slo,
                     candidates=candidates, shape=rng.choice(("random", "grown")),
                     stats=candidates <= 256 and rng.random() < 0.5)
    if kind == "search":
        devices = min(devices, 16)
        return _case(None, kind, devices, min(models, 8), _log(rng, 2000, 30000),
                     round(devices * rng.uniform(0.6, 2.0), 2), cv, slo,
                     policy=rng.choice(("mp-search", "mp-greedy", "sr-greedy", "sr-search")))
    if kind == "one":
        mixed = rng.random() < 0.75
        return _case(None, kind, devices, models, _log(rng, 1000, 150000), rate, cv, slo,
                     mixed=mixed, batching=mixed and rng.random() < 0.25)
    if kind == "stats":
        batching = rng.random() < 0.3
        return _case(None, kind, devices, models, _log(rng, 2000, 60000 if batching else 150000),
                     rate, cv, slo, schedule=rng.random() < 0.4, fast=rng.random() < 0.5,
                     batching=batching)
    if kind == "batching":
        return _case(None, kind, devices, models, _log(rng, 2000, 45000), rate, cv, slo,
                     candidates=_log(rng, 2, 256))
    if kind == "sweep":
        return _case(None, kind, devices, models, _log(rng, 5000, 60000),
                     round(devices * rng.uniform(0.6, 4.3), 2), 1.0, slo,
                     traces=rng.randint(5, 48))
    batching = rng.random() < 0.25
    return _case(None, kind, devices, models, _log(rng, 100, 20000 if batching else 60000), rate,
                 cv, slo, batching=batching)


def _models(case):
    bs = BATCH_SIZES if case["kind"] in ("batching", "dense") or case.get("batching") else (1,)
    return cases.mixed_models(case["models"], case["rate"], case["cv"], case["slo"], bs)


def _trace(datas, case, seed):
    """A merged Gamma trace of exactly case["requests"] requests."""
    duration = 1.2 * case["requests"] / case["rate"]
    while True:
        w = cases.merged_gamma_trace(datas, duration, (seed * 7919 + 17) % (1 << 31))
        if len(w) >= case["requests"]:
            return w[:case["requests"]]
        duration *= 1.5


def _placements(datas, case, seed, count):
    return cases.random_placements(datas, case["devices"], MEM_BUDGET, count,
                                   (seed * 104729 + 5) % (1 << 31))


def _half_filled(datas, devices, pp, rng):
    """Equal pipeline groups about half full: the model with the most requests per replica
    first, each to the emptiest group that takes it.  Returns (placement, model sizes)."""
    config = ParallelConfig(1, 1, pp)
    mem = [max(d.profiling_result.para_dict[config].weight_mem) for d in datas]
    load = np.array([d.rate for d in datas]) * rng.uniform(0.7, 1.4, len(datas))
    groups = [[] for _ in range(devices // pp)]
    used = np.zeros(len(groups))
    replicas = np.ones(len(datas))
    while used.sum() < 0.5 * MEM_BUDGET * len(groups):
        for m in np.argsort(-load / replicas):
            fits = [g for g in np.argsort(used, kind="stable")
                    if m not in groups[g] and used[g] + mem[m] < MEM_BUDGET]
            if fits:
                break
        else:
            break
        groups[fits[0]].append(int(m))
        used[fits[0]] += mem[m]
        replicas[m] += 1
    return ModelPlacement([config] * len(groups), groups).normalize(), mem


def _grown(datas, case, seed):
    """A layer of a search over equal pipeline groups: every partition of the cluster about
    half filled, and each candidate adds one model to one group."""
    rng = np.random.RandomState((seed * 15485863 + 3) % (1 << 31))
    out, count = [], case["candidates"]
    for _ in range(8):                 # the beams of a wide search, until there are enough
        for pp in (1, 2, 4, 8):
            if pp > case["devices"]:
                continue
            base, mem = _half_filled(datas, case["devices"], pp, rng)
            seen = set()
            for g, ms in enumerate(base.group_models):
                used = sum(mem[m] for m in ms)
                for m in range(len(datas)):
                    if m not in ms and used + mem[m] < MEM_BUDGET:
                        nxt = base.add_model(g, m).normalize()
                        if nxt.group_models not in seen:
                            seen.add(nxt.group_models)
                            out.append(nxt)
        if len(out) >= count:
            break
    rng.shuffle(out)
    return (out * (count // len(out) + 1))[:count]


def _serving_case(datas, workload, place):
    """The reference's ServingCase triple."""
    def register_models(controller):
        for d in datas:
            controller.register_model.remote(d.name, partial(object, d.profiling_result))

    return register_models, lambda: workload, place


POLICIES = {"mp-search": partial(search.ModelParallelismSearch, max_op=1),
            "mp-greedy": partial(search.ModelParallelismGreedy, group_size=2),
            "sr-greedy": search.SelectiveReplicationGreedy,
            "sr-search": search.SelectiveReplicationSearch}


def prepare(case, seed):
    kind = case["kind"]
    datas = _models(case)
    env = ClusterEnv(case["devices"], MEM_BUDGET)
    s = {"kind": kind, "case": case, "datas": datas, "env": env}
    if kind == "sweep":
        # trace t is in cell t mod 16: four rate scales by four CVs
        sweep = cases.SweepCase(datas, env, _placements(datas, case, seed, 1)[0],
                                case["requests"] / case["rate"], case["rate"])
        first = (seed * 6271) % (1 << 20) * 16
        s["workloads"] = [sweep.trace(first + t) for t in range(case["traces"])]
        s["sweep"] = TraceSweep(datas, env, sweep.placement, cells=16)
        return s
    workload = s["workload"] = _trace(datas, case, seed)
    if kind == "score":
        s["list"] = (_placements(datas, case, seed, case["candidates"])
                     if case["shape"] == "random" else _grown(datas, case, seed))
        s["evaluator"] = PlacementEvaluator(datas, env, workload)
        return s
    if kind == "search":
        policy = POLICIES[case["policy"]]()
        s["serving"] = _serving_case(
            datas, workload, lambda c: policy.solve_placement(datas, env, workload)[0])
        return s
    if case.get("batching") or kind == "batching":
        simulator.batchsize_config[:] = BATCH_SIZES
    names = tuple(d.name for d in datas)
    ids, slos = simulator.workload_arrays(workload, names)
    profiles = tuple(d.profiling_result for d in datas)
    if kind == "batching":
        s["list"] = _placements(datas, case, seed, case["candidates"])
        s["trace"] = engine.DeviceTrace(workload.arrivals, ids, slos, len(names))
        s["table"] = engine.LatencyTable(profiles, BATCH_SIZES)
    elif kind == "one":
        s["args"] = (_placements(datas, case, seed, 1)[0], names, profiles, ids, slos,
                     workload.arrivals)
    elif kind == "stats":
        if case["schedule"]:
            end = float(workload.arrivals[-1])
            # the same groups all along; each change shifts the models within their size class
            first = _placements(datas, case, seed, 1)[0]
            shifted = [ModelPlacement(first.group_configs,
                                      [[(m + 3 * k) % len(datas) for m in ms]
                                       for ms in first.group_models]) for k in range(3)]
            placement = ModelPlacementWithReplacement([0.0, end / 3, 2 * end / 3], shifted)
        else:
            placement = _placements(datas, case, seed, 1)[0]
        s["serving"] = _serving_case(datas, workload, lambda controller: placement)
    else:
        s["args"] = _dense_tables(datas, _placements(datas, case, seed, 1)[0], case["batching"])
        s["inputs"] = (workload.arrivals, ids, slos)
    return s


def _dense_tables(datas, placement, batching):
    """(m_id2g_id, g_id2m_id, num_stages, stage_latency) as the reference's callers make them."""
    M, G = len(datas), len(placement.group_configs)
    S = max(c.pp for c in placement.group_configs)
    sizes = BATCH_SIZES if batching else (1,)
    m2g = np.full((M, G + 1), -1, np.int32)
    g2m = np.full((G, M + 1), -1, np.int32)
    lat = np.zeros((M, G, S, len(sizes)), np.float32)
    fill = [0] * M
    for g, (c, ms) in enumerate(zip(placement.group_configs, placement.group_models)):
        for k, m in enumerate(sorted(ms)):
            m2g[m, fill[m]] = g
            fill[m] += 1
            g2m[g, k] = m
        for m, d in enumerate(datas):
            entry = d.profiling_result.para_dict[c]
            for j, b in enumerate(sizes):
                lat[m, g, :c.pp, j] = np.array(entry.latency[b]) * (1 + 0.009 * c.pp)
    stages = np.array([c.pp for c in placement.group_configs], np.int32)
    return m2g, g2m, stages, lat if batching else np.ascontiguousarray(lat[..., 0])


def _wide(counts, devices):
    """Per-group counters with one column per device (placements differ in groups)."""
    counts = np.asarray(counts)
    out = np.zeros(counts.shape[:-1] + (devices,), counts.dtype)
    out[..., :counts.shape[-1]] = counts
    return out


def _stats_arrays(stats, names, devices):
    """A StatsResult as arrays, one row per registered model."""
    fields = ("num_requests", "goodput", "throughput", "latency_mean", "latency_std",
              "latency_p90", "latency_p99")
    rows = {m.name: [getattr(m, f) for f in fields] for m in stats.per_model_stats}
    return {"models": np.array([rows.get(n, [0] * len(fields)) for n in names], np.float64),
            "groups": _wide(stats.group_num_requests, devices),
            "whole": np.array([stats.goodput, stats.latency_mean, stats.num_requests,
                               stats.request_rate], np.float64)}


def run(s):
    kind, case = s["kind"], s["case"]
    names, devices = [d.name for d in s["datas"]], case["devices"]
    if kind == "score" and case["stats"]:
        rows = s["evaluator"].get_stats(s["list"])
        return {"goodput": np.array([r[0] for r in rows]),
                "per_model": np.array([r[1] for r in rows]),
                "groups": np.array([_wide(r[2], devices) for r in rows]),
                "latency_mean": np.array([r[3].latency_mean for r in rows])}
    if kind == "score":
        return np.array(s["evaluator"].get_scores(s["list"]))
    if kind == "search":
        stats, sol = simulator.approximate_one_case(s["serving"], fast_stats=True)
        table = np.full((devices, 3 + len(names)), -1, np.int32)
        for g, (c, ms) in enumerate(zip(sol.group_configs, sol.group_models)):
            table[g, :3] = c
            table[g, 3:3 + len(ms)] = ms
        return table, _stats_arrays(stats, names, devices)
    if kind == "one":
        _, finish, good, mreq, mgood, greq, ggood = simulator.approximate_one_case_one_placement(
            *s["args"], mixed=case["mixed"], enable_batching=case["batching"])
        return finish, good, mreq, mgood, _wide(greq, devices), _wide(ggood, devices)
    if kind == "stats":
        stats, _ = simulator.approximate_one_case(s["serving"], fast_stats=case["fast"],
                                                  enable_batching=case["batching"])
        return _stats_arrays(stats, names, devices)
    if kind == "batching":
        enc = engine.encode_placements(s["list"], s["table"], len(s["datas"]))
        res = engine.run_batch_batching(s["trace"], enc, s["table"], rows_on_device=True,
                                        per_request=False)
        return [res.finish_device, res.good_device, res.model_num_good,
                _wide(res.group_num_requests, devices), res.good_total, res.latency_sum]
    if kind == "sweep":
        rows, tally = s["sweep"].evaluate_tally(s["workloads"])
        return {"goodput": np.array([r[0] for r in rows]),
                "per_model": np.array([r[1] for r in rows]),
                "groups": _wide(np.array([r[2] for r in rows]), devices), "tally": tally}
    arrivals, ids, slos = s["inputs"]
    m2g, g2m, stages, lat = s["args"]
    n = len(arrivals)
    finish, good = np.empty(n, np.float64), np.empty(n, bool)
    if case["batching"]:
        counters = simulator.simulate_requests_mixed_batching(finish, good, arrivals, ids, slos,
                                                              m2g, g2m, stages, lat, n)
    else:
        counters = simulator.simulate_requests_mixed(finish, good, arrivals, ids, slos, m2g,
                                                     stages, lat, n)
    mreq, mgood, greq, ggood = counters
    return finish, good, mreq, mgood, _wide(greq, devices), _wide(ggood, devices)


def work(case):
    """Inputs once (16 bytes a request: arrival f64, model i32, SLO f32; 4 bytes per placed
    model and group), outputs once, and per simulated request about 12 fp64 operations: the
    comparison of the replicas' clocks, a max and an add per pipeline stage, the SLO test."""
    kind, n = case["kind"], case["requests"]
    placed = 8 * case["devices"]
    runs = case.get("candidates", 1)
    if kind == "search":
        # a search adds about two models per device; a partition search runs four chains
        runs = 2 * case["devices"] * (4 if case["policy"] == "mp-search" else 1)
    if kind == "sweep":
        runs = case["traces"]
        total = 1.875 * n * runs                     # rate scales 0.5, 1, 2 and 4
        return {"bytes": 16 * total + 4 * runs * (case["models"] + case["devices"]),
                "flops": 12 * total}
    rows = {"one": 9, "dense": 9, "batching": 9}.get(kind, 0) * n * runs
    return {"bytes": 16 * n + runs * (placed + 8) + rows, "flops": 12 * n * runs}


def tolerance(case):
    return "exact"
