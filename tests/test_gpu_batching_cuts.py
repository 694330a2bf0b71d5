"""GPU tests of the batching simulator around the lengths at which a trace is
cut and at the chunk counts its last pass goes through, and of traces stored
one after the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,count", [(20.0, 1), (60.0, 1), (60.0, 24), (60.0, 33)])
@pytest.mark.parametrize("n", [1, 255, 1023, 1024, 4095, 4096, 4097, 9001])
def test_batching_where_the_trace_is_cut(rate, count, n):
    """One placement and 24 or 33, a warp for every chunk of each, on traces just
    below, at and above the lengths from which chunks are simulated in parallel;
    at the higher rate requests queue across the cuts."""
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from mms_b200 import cases, engine
    from mms_b200.simulator import workload_arrays
    from oracle import tables
    case = cases.candidate_batch_case(num_candidates=count, duration=9600.0 / rate,
                                      batching=True, placement_seed=3, total_rate=rate, cv=3.0)
    names = [d.name for d in case.model_datas]
    profs = [d.profiling_result for d in case.model_datas]
    mids, slos = workload_arrays(case.workload, names)
    arr, mids, slos = (np.ascontiguousarray(x[:n]) for x in (case.workload.arrivals, mids, slos))
    assert len(arr) == min(n, len(case.workload.arrivals))
    trace = engine.DeviceTrace(arr, mids, slos, len(names))
    table = engine.LatencyTable(profs, [1, 2, 4, 8])
    enc = engine.encode_placements(case.placements, table, len(names))
    res = engine.run_batch_batching(trace, enc, table)
    for b in {0, count // 2, count - 1}:
        fin, good, mreq, mgood, greq, ggood = tables.one_placement(
            case.placements[b], profs, mids, slos, arr, batchsize_config=(1, 2, 4, 8))
        assert res.finish[b].tobytes() == fin.tobytes(), b
        assert np.array_equal(res.good[b], good)
        assert np.array_equal(res.model_num_good[b], mgood)
        assert np.array_equal(res.group_num_requests[b, :len(greq)], greq)
        assert res.latency_sum[b] == float(np.add.reduce(fin - arr))


@pytest.mark.parametrize("count,walks", [(24, True), (320, False)])
@pytest.mark.parametrize("grid", [0.0, 0.02])
def test_batching_chunks_shorter_and_longer_than_the_run_in(count, walks, grid):
    """Few placements are cut into chunks shorter than the run-in and failed ones walked beside one
    another; of many the chunks are longer and the last pass alone puts them together.  Half of
    the placements have interchangeable groups; some are cut behind 8 000 requests, at a load where queues
    cross the cuts."""
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from mms_b200 import _native as nat
    from mms_b200 import cases, engine
    from mms_b200.placement import ModelPlacement
    from mms_b200.profiling import ParallelConfig
    from oracle import tables
    n, M = 8000, 6
    datas = cases.mixed_models(M, 10.0, 2.0, 3.0, (1, 2, 4, 8))
    profs = [d.profiling_result for d in datas]
    rng = np.random.RandomState(31)
    ts = np.cumsum(rng.gamma(0.3, 1 / (0.3 * 25.0), size=n))
    if grid:
        ts = np.floor(ts / grid) * grid
    ids = np.minimum(rng.geometric(0.35, size=n) - 1, M - 1).astype(np.int32)
    slos = np.array([d.slo for d in datas], np.float32)[ids]
    placements = []
    for k in range(count):
        degrees = [(1, 1, 2, 2, 2, 4, 4), (1, 1, 1, 1, 4, 8), (2,) * 8, (1,) * 16][k % 4]
        models = [sorted(rng.choice(M, size=int(rng.randint(1, 4)), replace=False).tolist()) for _ in degrees]
        if k % 2:
            for g in range(1, len(degrees), 2):          # pairs alike
                models[g] = models[g - 1]
        placements.append(ModelPlacement([ParallelConfig(1, 1, p) for p in degrees], models))
    trace = engine.DeviceTrace(ts, ids, slos, M)
    table = engine.LatencyTable(profs, [1, 2, 4, 8])
    enc = engine.encode_placements(placements, table, M)
    nat.profile_begin()
    res = engine.run_batch_batching(trace, enc, table)
    rounds = int(np.count_nonzero(nat.profile_end()[1] == nat.PROFILE_BATCH_REPAIR))
    assert rounds == (2 if walks else 1)                 # spans: each round of walks, and the last judgement
    assert (res.resimulated > 0).sum() > count // 4
    worst = np.argsort(res.resimulated)[-8:].tolist()
    for b in sorted({0, 1, 2, 3, 31, 32, count - 1, *worst} & set(range(count))):
        fin, good, mreq, mgood, greq, ggood = tables.one_placement(
            placements[b], profs, ids, slos, ts, batchsize_config=(1, 2, 4, 8))
        assert res.finish[b].tobytes() == fin.tobytes(), b
        assert np.array_equal(res.good[b], good), b
        assert np.array_equal(res.model_num_requests[b], mreq), b
        assert np.array_equal(res.model_num_good[b], mgood), b
        assert np.array_equal(res.group_num_requests[b, :len(greq)], greq), b
        assert np.array_equal(res.group_num_good[b, :len(ggood)], ggood), b
        assert res.latency_sum[b] == float(np.add.reduce(fin - ts)), b


@pytest.mark.parametrize("lengths", [[5], [0, 3], [8192, 0, 8193, 1], [31, 32, 33, 40000]])
def test_traces_one_after_the_other(lengths):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from mms_b200 import engine
    rng = np.random.default_rng(len(lengths))
    arrivals = [np.sort(rng.random(n) * 50.0) for n in lengths]
    mids = [rng.integers(0, 5, n).astype(np.int32) for n in lengths]
    slos = [(rng.random(n) + 0.5).astype(np.float32) for n in lengths]
    if max(lengths) > 40:                                  # one arrival out of order
        arrivals[-1][:2] = arrivals[-1][:2][::-1].copy() if lengths[-1] > 1 else arrivals[-1][:2]
    rows = engine.DeviceTraceRows(arrivals, mids, slos, 5)
    by_request = engine.DeviceTraceBatch(arrivals, mids, slos, 5)
    for name in ("arrivals", "model_ids", "slos"):
        got, want = (getattr(x, name).cpu().numpy() for x in (rows, by_request))
        assert got.tobytes() == np.ascontiguousarray(want.T).tobytes(), name
    assert np.array_equal(rows.model_hist.cpu().numpy(), by_request.model_hist.cpu().numpy())
