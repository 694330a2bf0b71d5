"""GPU tests of the batching simulator's two forms: the one with a group per lane, in which
interchangeable groups may change places and ties between them are noted, and the one with
lists, for everything beyond 64 groups or models and for traces and tables with oddities."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(placements, profs, ts, ids, slos, sizes=(1, 2, 4, 8), full_heap=False):
    """Every placement against the CPU checker.  full_heap: room for one pending event per group of the
    largest placement and no more."""
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from mms_b200 import engine
    from oracle import tables
    trace = engine.DeviceTrace(ts, ids, slos, len(profs))
    table = engine.LatencyTable(profs, list(sizes))
    enc = engine.encode_placements(placements, table, len(profs))
    res = engine.run_batch_batching(trace, enc, table, heap_capacity=enc.G if full_heap else 0)
    for b, p in enumerate(placements):
        fin, good, mreq, mgood, greq, ggood = tables.one_placement(p, profs, ids, slos, ts,
                                                                   batchsize_config=sizes)
        assert res.finish[b].tobytes() == fin.tobytes(), b
        assert np.array_equal(res.good[b], good), b
        assert np.array_equal(res.model_num_requests[b], mreq), b
        assert np.array_equal(res.model_num_good[b], mgood), b
        assert np.array_equal(res.group_num_requests[b, :len(greq)], greq), b
        assert np.array_equal(res.group_num_good[b, :len(ggood)], ggood), b
        assert res.good_total[b] == np.count_nonzero(good)
        assert res.latency_sum[b] == float(np.add.reduce(fin - ts)), b
    return res


def _trace(n, models, rate, grid, seed):
    """Bursty arrivals, rounded to `grid`; the last model is rare, some requests are of none."""
    rng = np.random.RandomState(seed)
    ts = np.cumsum(rng.gamma(0.2, 5.0 / rate, size=n))
    if grid:
        ts = np.floor(ts / grid) * grid
    ids = np.minimum(rng.geometric(0.35, size=n) - 1, models).astype(np.int32)
    ids[ids == models] = -1
    return ts, ids


def _placement(groups):
    from mms_b200.placement import ModelPlacement
    from mms_b200.profiling import ParallelConfig
    return ModelPlacement([ParallelConfig(1, 1, p) for p, _ in groups], [ms for _, ms in groups])


def _profiles(models, slo=3.0):
    from mms_b200 import cases
    datas = cases.mixed_models(models, 10.0, 2.0, slo, (1, 2, 4, 8))
    return [d.profiling_result for d in datas], np.array([d.slo for d in datas] + [1.0], np.float32)


@pytest.mark.parametrize("grid", [0.0, 0.01, 0.2])
@pytest.mark.parametrize("rate", [3.0, 20.0, 120.0])
def test_interchangeable_groups_that_take_turns(rate, grid):
    """Pairs, triples and eight of a kind that serve one or two models alone, in and out of
    order: a speculative run often has them the wrong way round for the rest of the trace, and on a
    grid the group number decides every other choice."""
    profs, slo = _profiles(6)
    ts, ids = _trace(6000, 6, rate, grid, int(rate))
    pairs = [(1, [4]), (1, [4]), (2, [5]), (2, [5])]
    sols = [_placement(pairs + [(1, [0, 1]), (2, [1, 2]), (4, [3])]),
            _placement([(1, [0]), (2, [1, 5]), (1, [0]), (1, [4]), (2, [1, 5]), (1, [0]), (1, [4])]),
            _placement([(1, [0, 1, 2])] * 8 + pairs),
            _placement([(1, [3]), (1, [3, 4]), (1, [3]), (1, [4, 3]), (2, [3])])]
    _check(sols, profs, ts, ids, slo[ids])


@pytest.mark.parametrize("rate", [3.0, 20.0])
def test_labels_spare_walks(rate):
    """Two placements that do the same: in the second the groups of a pair are not interchangeable, because
    one of each also has a model that is never asked for.  There a run with the pair the wrong way round is
    simulated again; the first takes it over."""
    profs, slo = _profiles(7)
    ts, ids = _trace(24000, 6, rate, 0.0, 9)
    alike = _placement([(1, [4]), (1, [4]), (2, [5]), (2, [5]), (1, [0]), (1, [0]), (4, [1, 2, 3])])
    told_apart = _placement([(1, [4]), (1, [4, 6]), (2, [5]), (2, [5, 6]), (1, [0]), (1, [0, 6]), (4, [1, 2, 3])])
    res = _check([alike, told_apart], profs, ts, ids, slo[ids])
    assert np.array_equal(res.finish[0], res.finish[1])
    assert 4 * res.resimulated[0] < res.resimulated[1]


@pytest.mark.parametrize("rate", [60.0, 400.0])
def test_room_for_one_pending_event_per_group(rate):
    """Bursts on a grid, in which groups have several events pending at a time: with room for one per group
    a run is right or reports that it was not enough, as it does for some; by default there is enough."""
    profs, slo = _profiles(6)
    ts, ids = _trace(6000, 6, rate, 0.05, 4)
    overflows = 0
    for groups in (3, 31, 32, 40):
        sols = [_placement([(1, [k % 6, (k + 1) % 6]) for k in range(groups)])]
        try:
            _check(sols, profs, ts, ids, slo[ids], full_heap=True)
        except RuntimeError as e:
            assert "heap overflow" in str(e)
            overflows += 1
        _check(sols, profs, ts, ids, slo[ids])
    assert overflows


@pytest.mark.parametrize("seed", [1, 3, 4, 6, 7, 9, 11])
def test_events_without_room_are_reported_alike(seed):
    """One event more pending than there is room for is an overflow, whether its group has one already or
    not: the form with a group per lane says so for the same capacities as the lists do (which take the
    same placements with 60 more models that nobody asks for)."""
    from mms_b200 import engine
    profs, slo = _profiles(66)
    rng = np.random.RandomState(seed)
    rate, n = (20, 60, 150, 400)[seed % 4], (700, 6000)[seed // 4 % 2]
    ts = np.cumsum(rng.gamma(0.2, 5.0 / rate, size=n))
    if seed % 3:
        ts = np.floor(ts / 0.05) * 0.05
    ids = np.minimum(rng.geometric(0.35, size=n) - 1, 5).astype(np.int32)
    forms = []
    for models in (6, 66):
        forms.append((models, engine.DeviceTrace(ts, ids, slo[ids], models),
                      engine.LatencyTable(profs[:models], [1, 2, 4, 8])))

    def overflows(form, sol, capacity):
        models, trace, table = form
        try:
            engine.run_batch_batching(trace, engine.encode_placements([sol], table, models), table,
                                      heap_capacity=capacity)
        except RuntimeError as e:
            assert "heap overflow" in str(e)
            return True
        return False
    for groups in (1, 2, 3, 5, 8, 16, 31, 40):
        sol = _placement([((1, 2)[k % 2], sorted(set(rng.choice(6, 3).tolist()))) for k in range(groups)])
        lanes, lists = ([overflows(form, sol, groups + k) for k in range(8)] for form in forms)
        assert lanes == lists, groups
        assert lanes == sorted(lanes, reverse=True)


@pytest.mark.parametrize("groups", [31, 32, 33, 64, 65, 130])
def test_groups_around_a_lane_each(groups):
    profs, slo = _profiles(5)
    ts, ids = _trace(3000, 5, 40.0, 0.01, groups)
    kinds = [(1, [0, 1]), (1, [2]), (2 if groups < 100 else 1, [1, 3]), (1, [4]), (1, [0])]
    sols = [_placement([kinds[k % 5] for k in range(groups)]),
            _placement([kinds[k * 5 // groups] for k in range(groups)])]
    _check(sols, profs, ts, ids, slo[ids])


@pytest.mark.parametrize("models", [1, 32, 33, 64, 65])
def test_models_around_a_lane_each(models):
    profs, slo = _profiles(models)
    rng = np.random.RandomState(models)
    ts, _ = _trace(3000, models, 30.0, 0.0, models)
    ids = rng.randint(-1, models, 3000).astype(np.int32)
    groups = [(int(rng.choice([1, 2, 4, 8])), sorted(set(rng.randint(0, models, 12).tolist())))
              for _ in range(12)]
    _check([_placement(groups), _placement(sorted(groups))], profs, ts, ids, slo[ids])


@pytest.mark.parametrize("odd", ["unsorted", "negative", "infinite"])
def test_odd_traces_and_tables(odd):
    """An arrival out of order, negative arrival times, or a model without a profile (latency
    +inf) under an SLO without end."""
    from mms_b200.profiling import ParallelConfig
    profs, slo = _profiles(4)
    ts, ids = _trace(4000, 4, 30.0, 0.0, 5)
    slos = slo[ids]
    if odd == "unsorted":
        ts[2000:2002] = ts[2000:2002][::-1].copy()
    elif odd == "negative":
        ts = ts - ts[1500]
    else:
        del profs[1].para_dict[ParallelConfig(1, 1, 2)]
        slos = np.full(len(ts), np.inf, np.float32)
    sols = [_placement([(1, [0, 1]), (2, [1, 2]), (2, [1, 2]), (1, [3]), (1, [3])])] * 3
    _check(sols, profs, ts, ids, slos)


def test_lists_of_replicas_in_any_order():
    """A caller's own tables may list a model's replicas in any order; the first of equal clocks
    is the first of the list."""
    from mms_b200 import simulator
    from oracle import cpu
    rng = np.random.RandomState(3)
    n, M, G, S = 6000, 3, 6, 2
    ts = np.floor(np.cumsum(rng.gamma(0.2, 0.2, size=n)) / 0.05) * 0.05
    ids = rng.randint(0, M, size=n).astype(np.int32)
    slo = np.full(n, 1.5, np.float32)
    m2g = np.array([[3, 1, 2, -1, -1, -1, -1], [5, 4, 0, -1, -1, -1, -1], [2, 0, 4, 1, -1, -1, -1]], np.int32)
    g2m = np.full((G, M + 1), -1, np.int32)
    for g in range(G):
        ms = [m for m in range(M) if g in m2g[m]]
        g2m[g, :len(ms)] = ms
    ns = np.array([1, 1, 1, 2, 2, 1], np.int32)
    lat = np.full((M, G, S, 4), 0.08, np.float32) * np.array([1.0, 1.2, 1.6, 2.4], np.float32)
    fin = np.empty(n); good = np.empty(n, bool)
    efin = np.empty(n); egood = np.empty(n, bool)
    sizes, old = [1, 2, 4, 8], list(simulator.batchsize_config)
    simulator.batchsize_config[:] = sizes
    try:
        got = simulator.simulate_requests_mixed_batching(fin, good, ts, ids, slo, m2g, g2m, ns, lat, n)
        exp = cpu.simulate_requests_mixed_batching(efin, egood, ts, ids, slo, m2g, g2m, ns, lat, n, sizes)
    finally:
        simulator.batchsize_config[:] = old
    assert fin.tobytes() == efin.tobytes() and np.array_equal(good, egood)
    for x, y in zip(got, exp):
        assert np.array_equal(x, y)
