"""Host side of the GPU simulator: trace upload, placement encoding, launch.

The three steps mirror what the reference does per candidate in
alpa_serve/simulator/controller.py:410-503 (approximate_one_case_one_placement
builds m_id2g_id / num_stages / stage_latency, then calls the numba kernel),
but for a whole list of candidates at once and in the compact form that
include/mms_sim.h describes.  PyTorch is used for device memory and streams
only; all compute goes through the C ABI in libmms_sim.so.
"""
import ctypes
import functools
import operator
import threading
from contextlib import nullcontext
from itertools import chain, permutations, product
from math import factorial, prod
from typing import List, Sequence

import numpy as np
import torch

from . import _native as nat
from .profiling import ParallelConfig

inf = 1e100      # alpa_serve/util.py:23
_PP = operator.itemgetter(2)     # pipeline degree of a ParallelConfig(dp, op, pp)


def _require_cuda():
    if torch.cuda.is_initialized():       # (there was a device, and it is cheaper to ask)
        return
    if not torch.cuda.is_available():
        raise RuntimeError("mms_b200 needs a CUDA device: the simulator has no CPU path")


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None and t.numel() > 0 else ctypes.c_void_p(0)


def _raw_stream(index=None):
    """The current stream of a device (None: the current one) as CUDA's handle, 0 for the default one
    (torch.cuda.current_stream() makes an object of it, which takes longer than a launch; the name in
    torch._C is private, and a torch without it goes that way)."""
    if index is None:
        index = torch.cuda.current_device()
    try:
        ask = torch._C._cuda_getCurrentRawStream
    except AttributeError:
        return torch.cuda.current_stream(index).cuda_stream
    return ask(index)


def _stream_ptr():
    return ctypes.c_void_p(_raw_stream())


def _layout(fields):
    """{name: (offset, bytes, dtype, shape)} of arrays one behind the other, each 16-byte aligned, and
    the bytes of all; a field without a shape is left out."""
    at, total = {}, 0
    for name, dtype, shape in fields:
        if shape is not None:
            size = prod(shape) * _ITEM_BYTES[dtype]
            at[name] = (total, size, dtype, shape)
            total += (size + 15) & ~15
    return at, max(total, 16)


_ITEM_BYTES = {t: np.dtype(t).itemsize for t in (np.int32, np.uint32, np.int64, np.float64)}


_NO_CONTEXT = nullcontext()


def _on(dev):
    """`dev` as the current device (entering torch.cuda.device for the device that is current
    anyway costs as much as a kernel launch)."""
    return _NO_CONTEXT if dev.index == torch.cuda.current_device() else torch.cuda.device(dev)


def _to_device(arr: np.ndarray, device, pinned=False):
    t = torch.from_numpy(np.ascontiguousarray(arr))
    if pinned:
        t = t.pin_memory()
    return t.to(device, non_blocking=pinned)


# Uploads up to this size go straight from pageable memory: the driver takes such a copy into
# a buffer of its own before the call returns, and nothing waits for the GPU.
_SMALL_UPLOAD = 64 << 10
_TORCH_TYPE = {np.dtype(k): v for k, v in (
    (np.uint8, torch.uint8), (np.uint16, torch.uint16), (np.int32, torch.int32),
    (np.uint32, torch.uint32), (np.int64, torch.int64), (np.float32, torch.float32),
    (np.float64, torch.float64))}
_STAGED_UPLOAD = 128 << 20       # larger ones are not worth holding that much page-locked memory


def _to_device_many(arrays, device):
    """Several host arrays to the device as ONE transfer: a launch uploads half a
    dozen small tables, and each transfer costs tens of microseconds whatever its
    size.  Small ones are packed in pageable memory, larger ones in page-locked
    memory from torch's host allocator (which keeps a block until the copies
    from it are done).  Returns device tensors that are views of one buffer, each
    16-byte aligned."""
    arrays = [np.ascontiguousarray(a) for a in arrays]
    buf, offsets = _pack(arrays, device)
    if buf is None:
        return [_to_device(a, device) for a in arrays]
    return [buf[o:o + a.nbytes].view(_TORCH_TYPE[a.dtype]).reshape(a.shape)
            for a, o in zip(arrays, offsets)]


def _upload(arrays, device):
    """_to_device_many for callers that only need addresses: (what to keep, [pointer, ...])."""
    arrays = [np.ascontiguousarray(a) for a in arrays]
    buf, offsets = _pack(arrays, device)
    if buf is None:
        keep = [_to_device(a, device) for a in arrays]
        return keep, [_ptr(t) for t in keep]
    base = buf.data_ptr()
    return buf, [ctypes.c_void_p(base + o if a.size else 0) for a, o in zip(arrays, offsets)]


def _pack(arrays, device):
    """The transfer of _to_device_many: (buffer, offsets), or (None, None) where the arrays are so large
    that they go one by one."""
    offsets, total = [], 0
    for a in arrays:
        offsets.append(total)
        total += (a.nbytes + 15) & ~15
    total = max(total, 16)
    if total > _STAGED_UPLOAD:
        return None, None
    small = total <= _SMALL_UPLOAD
    stage = torch.empty(total, dtype=torch.uint8, pin_memory=not small)
    host = stage.numpy()
    for a, o in zip(arrays, offsets):
        if a.nbytes:
            host[o:o + a.nbytes] = a.reshape(-1).view(np.uint8)
    buf = torch.empty(total, dtype=torch.uint8, device=device)
    buf.copy_(stage, non_blocking=True)
    return buf, offsets


@functools.lru_cache(maxsize=64)
def _sum_plan(n):
    """(leaf starts i32[leaves + 1], merges u8[max(leaves, 1)]) of numpy's pairwise sum of n
    elements (mms_sum_plan)."""
    L = nat.lib()
    n_leaves = L.mms_sum_plan_leaves(n)
    if n_leaves < 0:
        nat.check(n_leaves, "mms_sum_plan_leaves")
    leaf_start = np.zeros(n_leaves + 1, np.int32)
    leaf_merges = np.zeros(max(n_leaves, 1), np.uint8)
    nat.check(L.mms_sum_plan_fill(n, leaf_start.ctypes.data, leaf_merges.ctypes.data),
              "mms_sum_plan_fill")
    leaf_start.setflags(write=False)
    leaf_merges.setflags(write=False)
    return leaf_start, leaf_merges


class DeviceTrace:
    """A request trace resident on one GPU: arrivals f64[N], model ids i32[N]
    (-1 = unknown model), SLOs f32[N] — the arrays controller.py:335-336
    caches per workload — plus what depends on the trace alone: the per-model
    request counts (controller.py:587) and numpy's summation plan for N."""

    def __init__(self, arrivals, model_ids, slos, num_models: int, device=None):
        _require_cuda()
        self.device = torch.device("cuda", torch.cuda.current_device()) if device is None \
            else torch.device(device)
        arrivals = np.ascontiguousarray(arrivals, dtype=np.float64)
        model_ids = np.ascontiguousarray(model_ids, dtype=np.int32)
        slos = np.ascontiguousarray(slos, dtype=np.float32)
        if not (len(arrivals) == len(model_ids) == len(slos)):
            raise ValueError("arrivals, model_ids and slos must have one entry per request")
        self.num_requests = int(len(arrivals))
        self.num_models = int(num_models)
        self.host_arrivals = arrivals
        self.h2d_bytes = arrivals.nbytes + model_ids.nbytes + slos.nbytes
        L = nat.lib()
        leaf_start, leaf_merges = _sum_plan(self.num_requests)
        self.num_leaves = len(leaf_start) - 1
        with _on(self.device):
            (self.arrivals, self.model_ids, self.slos, self.leaf_start,
             self.leaf_merges) = _to_device_many(
                (arrivals, model_ids, slos, leaf_start, leaf_merges), self.device)
            self.model_hist = torch.empty(self.num_models + 1, dtype=torch.int32,
                                          device=self.device)
            tr = self.c_trace()
            nat.check(L.mms_trace_model_histogram(ctypes.byref(tr), self.num_models,
                                                  _ptr(self.model_hist), _stream_ptr()),
                      "mms_trace_model_histogram")

    def next_same_model(self):
        """i32[N] on the device: index of the next request with the same model, -1 if there is none
        (a model's FIFO queue is a run of this list)."""
        if getattr(self, "_next_same", None) is None:
            with _on(self.device):
                buf = torch.empty(max(self.num_requests, 1), dtype=torch.int32,
                                  device=self.device)
                tr = self.c_trace()
                nat.check(nat.lib().mms_trace_next_same_model(
                    ctypes.byref(tr), self.num_models, _ptr(buf), _stream_ptr()),
                    "mms_trace_next_same_model")
            self._next_same = buf
        return self._next_same

    def c_trace(self):
        return nat.Trace(self.num_requests, _ptr(self.arrivals), _ptr(self.model_ids),
                         _ptr(self.slos))

    def c_plan(self):
        return nat.SumPlan(self.num_leaves, 0, _ptr(self.leaf_start), _ptr(self.leaf_merges))


class LazyArray:
    """A host array that is produced piece by piece, straight into an upload
    buffer: fill(out, lo, hi) writes elements [lo, hi) into `out` (a numpy view
    of hi - lo elements of `dtype`).  Saves the pass that would materialise it."""

    def __init__(self, size, dtype, fill):
        self.size, self.dtype, self.fill = int(size), np.dtype(dtype), fill

    def __len__(self):
        return self.size

    def materialize(self):
        out = np.empty(self.size, self.dtype)
        self.fill(out, 0, self.size)
        return out


class PinnedStager:
    """Uploads many host arrays through pinned staging buffers: a few threads
    copy pieces of the arrays into page-locked buffers (numpy copies run
    outside the interpreter lock) and enqueue the transfers from there, each on
    a stream of its own.  Pageable memory goes to the device at about a third
    of the rate of page-locked memory, whatever the number of threads that
    ask; staging by hand is what lets the threads help.  One instance per
    device is kept (page-locked allocations are slow); uploads from several
    threads take turns, since they share its buffers."""

    _instances = {}

    @classmethod
    def get(cls, dev, threads=8, piece_bytes=16 << 20):
        key = (torch.device(dev), threads, piece_bytes)
        if key not in cls._instances:
            cls._instances[key] = cls(*key)
        return cls._instances[key]

    def __init__(self, dev, threads, piece_bytes):
        from concurrent.futures import ThreadPoolExecutor
        self.device, self.threads, self.piece = torch.device(dev), int(threads), int(piece_bytes)
        self.pool = ThreadPoolExecutor(self.threads)
        self.turn = threading.Lock()
        # of high priority, which torch takes from a pool of their own: a stream that kernels are
        # queued on (torch has 32 per priority and hands them out in turn) would hold the copies up
        self.streams = [torch.cuda.Stream(device=self.device, priority=-1)
                        for _ in range(self.threads)]
        self.buffers = [[torch.empty(self.piece, dtype=torch.uint8).pin_memory() for _ in range(2)]
                        for _ in range(self.threads)]

    def upload(self, tasks):
        """tasks: [(device tensor, numpy array or LazyArray)] of equal byte sizes
        pairwise, contiguous.  Returns when every transfer has been enqueued;
        the current stream waits for them."""
        pieces = [[] for _ in range(self.threads)]
        load = [0] * self.threads
        for dst, src in tasks:
            d8 = dst.reshape(-1).view(torch.uint8)
            lazy = isinstance(src, LazyArray)
            if lazy:
                item, count = src.dtype.itemsize, src.size
            else:
                src = np.ascontiguousarray(src).reshape(-1)
                item, count = src.dtype.itemsize, src.size
            if d8.numel() != item * count:
                raise ValueError("upload: sizes differ")
            step = max(self.piece // item, 1)
            for lo in range(0, count, step):
                k = load.index(min(load))
                hi = min(lo + step, count)
                pieces[k].append((d8[lo * item:hi * item], src, lo, hi))
                load[k] += (hi - lo) * item
        main = torch.cuda.current_stream(self.device)

        def work(k):
            stream, bufs = self.streams[k], self.buffers[k]
            events = [None, None]
            stream.wait_stream(main)            # the destinations are free to write there
            with torch.cuda.device(self.device), torch.cuda.stream(stream):
                for j, (d8, src, lo, hi) in enumerate(pieces[k]):
                    if events[j & 1] is not None:
                        events[j & 1].synchronize()      # the buffer's last transfer is done
                    buf = bufs[j & 1][:d8.numel()]
                    view = buf.numpy().view(src.dtype)
                    if isinstance(src, LazyArray):
                        src.fill(view, lo, hi)
                    else:
                        np.copyto(view, src[lo:hi])
                    d8.copy_(buf, non_blocking=True)
                    ev = torch.cuda.Event()
                    ev.record(stream)
                    events[j & 1] = ev
            for ev in events:                   # the buffers are free for the next upload
                if ev is not None:
                    ev.synchronize()

        with self.turn:
            list(self.pool.map(work, [k for k in range(self.threads) if pieces[k]]))
        for k in range(self.threads):
            if pieces[k]:
                main.wait_stream(self.streams[k])


class DeviceTraceBatch:
    """T request traces resident on one GPU for runs in which every candidate
    has a trace of its own (one placement scored on many traces).  The traces
    are stored request-major ([N][T]: the 32 candidates of a warp read
    consecutive addresses) and padded to the longest one with requests of
    model -1 at the last arrival time, which change no clock and no counter.
    The host uploads every trace as it is, one after the other; the
    request-major batch is made on the device (mms_trace_pack).
    Duck-type compatible with DeviceTrace where launches are concerned."""

    flags = 0

    def __init__(self, arrivals: Sequence, model_ids: Sequence, slos: Sequence, num_models: int,
                 device=None, staged=False, owner=None):
        """staged: upload through PinnedStager (worth it from about a gigabyte).
        owner: the stream from whose memory the traces are taken (None: the current one, on which
        they are uploaded and counted in any case)."""
        _require_cuda()
        self.owner = owner
        self.device = torch.device("cuda", torch.cuda.current_device()) if device is None \
            else torch.device(device)
        T = len(arrivals)
        if T == 0 or not (len(model_ids) == len(slos) == T):
            raise ValueError("need one (arrivals, model_ids, slos) triple per trace")
        self.lengths = np.fromiter((len(a) for a in arrivals), np.int64, T)
        for t in range(T):
            if not (len(model_ids[t]) == len(slos[t]) == int(self.lengths[t])):
                raise ValueError(f"trace {t}: arrays differ in length")
        N = int(self.lengths.max())
        self.num_traces, self.num_requests, self.num_models = T, N, int(num_models)
        self.h2d_bytes = int(self.lengths.sum()) * 16 + (T + 1) * 8
        with torch.cuda.device(self.device):
            self._store((arrivals, model_ids, slos), staged)
            leaf_start, leaf_merges = _sum_plan(N)
            self.num_leaves = len(leaf_start) - 1
            self.leaf_start, self.leaf_merges = _to_device_many((leaf_start, leaf_merges),
                                                                self.device)
            # [T][M + 1] counts, then the total of unsorted positions (T == 1: plain [M + 1])
            cells = T * (self.num_models + 1) + (1 if T > 1 else 0)
            self.model_hist = torch.zeros(cells, dtype=torch.int32, device=self.device)
            self._count()

    def _upload(self, sources, staged, place):
        """Copies array k of trace t to place(k, t), every trace as it is."""
        tasks = []
        for t in range(self.num_traces):
            if not self.lengths[t]:
                continue
            for k, dtype in enumerate((np.float64, np.int32, np.float32)):
                src = sources[k][t]
                if isinstance(src, LazyArray):
                    if src.dtype != dtype:
                        raise ValueError("lazy trace array of the wrong type")
                    src = src if staged else src.materialize()
                else:
                    src = np.ascontiguousarray(src, dtype)
                tasks.append((place(k, t), src))
        if staged:
            PinnedStager.get(self.device).upload(tasks)
        else:
            for dst, src in tasks:
                dst.copy_(torch.from_numpy(src), non_blocking=True)

    def _empty(self, shape):
        here = torch.cuda.current_stream(self.device)
        owner = here if self.owner is None else self.owner
        with torch.cuda.stream(owner):
            new = tuple(torch.empty(shape, dtype=t, device=self.device)
                        for t in (torch.float64, torch.int32, torch.float32))
        if owner != here:
            here.wait_stream(owner)         # what used the memory before is in order there
            for t in new:
                t.record_stream(here)       # and it is not handed out again before `here` is done
        return new

    def _store(self, sources, staged):
        N, T = self.num_requests, self.num_traces
        offsets = np.concatenate(([0], np.cumsum(self.lengths))).astype(np.int64)
        cat = self._empty(max(int(offsets[-1]), 1))
        self._upload(sources, staged, lambda k, t: cat[k][int(offsets[t]):int(offsets[t + 1])])
        d_off = _to_device(offsets, self.device)
        self.arrivals, self.model_ids, self.slos = self._empty((max(N, 1), T))
        nat.check(nat.lib().mms_trace_pack(
            *(_ptr(x) for x in cat), _ptr(d_off), T, N, _ptr(self.arrivals),
            _ptr(self.model_ids), _ptr(self.slos), _stream_ptr()), "mms_trace_pack")

    def _count(self):
        tr = self.c_trace()
        nat.check(nat.lib().mms_trace_model_histogram(
            ctypes.byref(tr), self.num_models, _ptr(self.model_hist), _stream_ptr()),
            "mms_trace_model_histogram")

    def c_trace(self):
        return nat.Trace(self.num_requests, _ptr(self.arrivals), _ptr(self.model_ids),
                         _ptr(self.slos), self.num_traces)

    def c_plan(self):
        return nat.SumPlan(self.num_leaves, 0, _ptr(self.leaf_start), _ptr(self.leaf_merges))


class DeviceTraceRows(DeviceTraceBatch):
    """The same traces stored one after the other ([T][N]): a warp that
    simulates one candidate reads 32 consecutive requests of its trace at a
    time.  Every trace is uploaded straight to its place, so that nothing is
    copied again on the device."""

    flags = nat.FLAG_TRACE_ROWS

    def _store(self, sources, staged):
        N, T = self.num_requests, self.num_traces
        self.arrivals, self.model_ids, self.slos = self._empty((T, max(N, 1)))
        rows = (self.arrivals, self.model_ids, self.slos)
        self._upload(sources, staged, lambda k, t: rows[k][t, :int(self.lengths[t])])
        if np.any(self.lengths < N):
            d_len = _to_device(self.lengths, self.device)
            nat.check(nat.lib().mms_trace_pad_rows(_ptr(d_len), T, N, *(_ptr(x) for x in rows),
                                                   _stream_ptr()), "mms_trace_pad_rows")

    def _count(self):
        if self.num_traces == 1:                     # one trace: both layouts are the same
            return super()._count()
        nat.check(nat.lib().mms_trace_rows_histogram(
            _ptr(self.arrivals), _ptr(self.model_ids), self.num_traces, self.num_requests,
            self.num_models, _ptr(self.model_hist), _stream_ptr()), "mms_trace_rows_histogram")


class LatencyTable:
    """stage latency per (model, parallel config, stage) in f32, with the
    0.9 %-per-stage penalty of controller.py:467-476 folded in.  Column c is
    the parallel config `configs[c]`; a config a model has no profile for is
    +inf (the f32 cast of 1e100), so such a replica never meets an SLO."""

    def __init__(self, prof_ress: Sequence, batch_sizes=None):
        """batch_sizes None: one latency per stage (batch size 1, table
        [M][C][S]); else the table gets a last axis over those batch sizes
        ([M][C][S][NB], controller.py:451-461)."""
        self.prof_ress = list(prof_ress)
        self.batch_sizes = None if batch_sizes is None else [int(b) for b in batch_sizes]
        self.configs: List = []
        self.column = {}
        self.max_stages = 1
        tail = () if batch_sizes is None else (len(self.batch_sizes),)
        self._host = np.zeros((len(self.prof_ress), 0, 1) + tail, np.float32)
        self._device = None

    def columns_for(self, configs) -> None:
        new = [c for c in dict.fromkeys(configs) if c not in self.column]
        if not new:
            return
        for c in new:
            self.column[c] = len(self.configs)
            self.configs.append(c)
        S = max([self.max_stages] + [int(c.pp) for c in new])
        M, C = len(self.prof_ress), len(self.configs)
        old = self._host
        tab = np.zeros((M, C, S) + old.shape[3:], np.float32)
        tab[:, :old.shape[1], :old.shape[2]] = old
        # the new columns as one list of numbers: 1 + the penalty times each latency in f64, rounded
        # to f32 once, as controller.py:467-476 does it array by array
        sizes = (1,) if self.batch_sizes is None else self.batch_sizes
        rows = []
        for prof in self.prof_ress:
            for c in new:
                value, pp = prof.para_dict.get(c, None), int(c.pp)
                if value:
                    factor = 1 + 0.009 * len(value.latency[1])
                    lats = [list(value.latency[b][:pp]) for b in sizes]
                    lats = [lat * pp if len(lat) == 1 else lat for lat in lats]   # one for all stages
                    if any(len(lat) != pp for lat in lats):
                        raise ValueError(f"fewer latencies than stages of {c}")
                    rows += [float(lat[k]) * factor for k in range(pp) for lat in lats]
                    rows += [0.0] * ((S - pp) * len(sizes))
                else:
                    rows += [inf] * (S * len(sizes))
        with np.errstate(over="ignore"):
            tab[:, len(self.configs) - len(new):] = np.array(rows, np.float64).reshape(
                (M, len(new), S) + old.shape[3:])
        self._host = tab
        self.max_stages = S
        self._device = None

    @property
    def host(self):
        return self._host

    def device(self, dev):
        """The table on `dev`; uploaded on the current stream when it changed,
        and any stream that asks for it waits for that upload."""
        with _on(torch.device(dev)):
            here = _raw_stream()
            if self._device is None or self._device.device != dev:
                self._device = _to_device(self._host, dev)
                self._ready = torch.cuda.Event()
                self._ready.record()
                self._uploaded_on = here
            elif here or self._uploaded_on:           # (the default stream is in order with itself)
                torch.cuda.current_stream().wait_event(self._ready)
        return self._device


class EncodedBatch:
    """Host arrays of a placement batch in the layout of mms_placements."""

    def __init__(self, B, M, G, P, T, S, C, model_off, model_rep, group_info, num_groups,
                 num_replicas, twins=None, has_twins=None):
        self.B, self.M, self.G, self.P, self.T, self.S, self.C = B, M, G, P, T, S, C
        self.model_off = model_off        # u16[B][M+1]
        self.model_rep = model_rep        # u32[B][P]
        self.group_info = group_info      # u32[B][G]
        self.num_groups = num_groups      # i64[B]
        self.num_replicas = num_replicas  # i64[B]: sum of len(group_models)
        self._twins = twins               # see twins; or a function that makes it
        # bool[B]: the placement has interchangeable groups at all (None: not known)
        self.has_twins = has_twins
        self._mirror_table = None         # see mirror_table()
        self._depth = None                # u8[B], or 0: see by_depth()

    @property
    def twins(self):
        """[(candidate index, [[group ids of one class of interchangeable groups], ...])]
        for every placement that has such groups, see twin_groups().  Made when somebody
        asks: running a batch only needs has_twins."""
        if callable(self._twins):
            self._twins = self._twins()
        return self._twins

    def may_have_twins(self):
        return self.has_twins is None or bool(np.any(self.has_twins))

    def mirror_table(self):
        """(counts i64[len(twins)], words u64[sum(counts)]): the exchange lists of
        every placement's mirrors (mirror_swaps), placement after placement in the
        order of `twins`; made once, for all placements of one class pattern together."""
        if self._mirror_table is None:
            self._mirror_table = mirror_swaps_batch([classes for _, classes in (self.twins or [])])
        return self._mirror_table

    def by_depth(self, index=None):
        """`index` (None: all placements) ordered by the depth of their pipelines, in lists that mix
        partitions of a cluster.  32 neighbours share a warp in large batches and wait for one
        another: partitions into single devices have up to 30 replicas of a model to choose from,
        those into eight none of that but long pipelines."""
        count = self.B if index is None else len(index)
        if count < MIN_BY_DEPTH or self.G == 0:
            return index
        if self._depth is None:
            def stages(rows):             # the second byte of group_info; 0: no group
                return rows.view(np.uint8).reshape(len(rows), -1, 4)[:, :, 1]

            # worth it where most placements have pipelines of one depth, as those of a search
            info = np.ascontiguousarray(self.group_info)
            sample = stages(np.ascontiguousarray(info[::max(self.B // 64, 1)]))
            alike = np.where(sample == 0, 255, sample).min(axis=1) == sample.max(axis=1)
            self._depth = stages(info).max(axis=1) if 2 * np.count_nonzero(alike) > len(alike) else 0
        if isinstance(self._depth, int):
            return index
        depth = self._depth if index is None else self._depth[index]
        if depth.min() == depth.max():
            return index
        order = np.argsort(depth, kind="stable")
        return order if index is None else index[order]

    def take(self, index):
        """The sub-batch of the placements `index`."""
        index = np.asarray(index, np.int64)

        def kept():
            new_id = np.full(self.B, -1, np.int64)
            new_id[index] = np.arange(len(index))
            keep = [k for k, (b, _) in enumerate(self.twins or []) if new_id[b] >= 0]
            return keep, [(int(new_id[self.twins[k][0]]), self.twins[k][1]) for k in keep]

        sub = EncodedBatch(len(index), self.M, self.G, self.P, self.T, self.S, self.C,
                           self.model_off[index], self.model_rep[index], self.group_info[index],
                           self.num_groups[index], self.num_replicas[index], lambda: kept()[1],
                           None if self.has_twins is None else self.has_twins[index])
        if self._mirror_table is not None:
            counts, words = self._mirror_table
            keep = np.asarray(kept()[0], np.int64)
            start = np.concatenate(([0], np.cumsum(counts)))[:-1]
            sub_counts = counts[keep]
            # the kept placements' stretches of `words`, one after the other
            pos = np.repeat(start[keep] - (np.cumsum(sub_counts) - sub_counts), sub_counts) \
                + np.arange(int(sub_counts.sum()))
            sub._mirror_table = (sub_counts, words[pos])
        return sub

    def repeat(self, count: int):
        """This batch `count` times over (placement 0 .. B-1, then again ...):
        the tables of one placement for `count` traces."""
        B = self.B

        def twins():
            return [(b + k * B, classes) for k in range(count) for b, classes in (self.twins or [])]

        return EncodedBatch(B * count, self.M, self.G, self.P, self.T, self.S, self.C,
                            np.tile(self.model_off, (count, 1)), np.tile(self.model_rep, (count, 1)),
                            np.tile(self.group_info, (count, 1)), np.tile(self.num_groups, count),
                            np.tile(self.num_replicas, count), twins,
                            None if self.has_twins is None else np.tile(self.has_twins, count))

    def with_mirrors(self):
        """The tables with mirror candidates appended for every placement
        that has interchangeable groups (see "Mirrors" in include/mms_sim.h),
        one per way of permuting them: (model_off, model_rep, group_info,
        partner i32[B'], mirror_swap u32[B'][2]) or None when no placement
        has any."""
        if not self.twins:
            return None
        counts, words = self.mirror_table()
        total = int(counts.sum())
        if total == 0:
            return None
        twin_b = np.fromiter((b for b, _ in self.twins), np.int64, len(self.twins))
        has = counts > 0
        first = self.B + np.cumsum(counts) - counts
        owners = np.repeat(twin_b, counts)
        at = self.B + total
        partner = np.full(at, -1, np.int32)
        partner[twin_b[has]] = first[has]
        partner[self.B:] = owners
        swap = np.full((at, 2), NO_SWAP, np.uint32)
        swap[self.B:] = words.view(np.uint32).reshape(-1, 2)
        return (np.concatenate((self.model_off, self.model_off[owners])),
                np.concatenate((self.model_rep, self.model_rep[owners])),
                np.concatenate((self.group_info, self.group_info[owners])), partner, swap)

    @property
    def nbytes(self):
        return self.model_off.nbytes + self.model_rep.nbytes + self.group_info.nbytes


NO_SWAP = np.uint32(0xFFFFFFFF)
_MODEL_KEYS = {}


MAX_MIRRORS = 15          # per placement
_PERM_CACHE = {}


def _perm_swaps(sizes):
    """Every non-identity way of permuting classes of the given sizes among
    themselves, each as a list of exchanges (i, j) of positions in the
    concatenated classes, at most four per permutation."""
    if sizes not in _PERM_CACHE:
        offsets = np.concatenate(([0], np.cumsum(sizes)))[:-1]
        per_class = []
        for off, n in zip(offsets, sizes):
            options = []
            for perm in permutations(range(n)):
                # exchanges that turn the identity arrangement into `perm`
                cur, ex = list(range(n)), []
                for i in range(n):
                    if cur[i] != perm[i]:
                        k = cur.index(perm[i])
                        cur[i], cur[k] = cur[k], cur[i]
                        ex.append((int(off) + i, int(off) + k))
                options.append(ex)
            per_class.append(options)
        out = []
        for combo in product(*per_class):
            ex = [e for part in combo for e in part]
            if ex and len(ex) <= 4:
                out.append(ex)
        _PERM_CACHE[sizes] = out
    return _PERM_CACHE[sizes]


def mirror_swaps(classes):
    """64-bit exchange lists (see mirror_swap in include/mms_sim.h) of the
    mirrors for one placement whose interchangeable groups are `classes`: one
    per permutation, or none at all when there are more than MAX_MIRRORS
    (covering only some would cost throughput without removing the serial
    repairs of the rest)."""
    sizes = tuple(len(c) for c in classes)
    count = 1
    for n in sizes:
        count *= factorial(n) if n < 5 else MAX_MIRRORS + 2
    if count - 1 > MAX_MIRRORS:
        return []
    groups = [g for c in classes for g in c]
    words = []
    for ex in _perm_swaps(sizes):
        w = 0xFFFFFFFFFFFFFFFF
        for k, (i, j) in enumerate(ex):
            w &= ~(0xFFFF << (16 * k))
            w |= (groups[i] | (groups[j] << 8)) << (16 * k)
        words.append(w)
    return words


def mirror_swaps_batch(class_lists):
    """mirror_swaps for many placements at once: (counts i64[n], words u64[sum])
    with the words of placement k at [sum(counts[:k]), sum(counts[:k + 1])), in
    the order mirror_swaps gives them.  Placements with the same class sizes
    share their permutations, so their words are formed together."""
    n = len(class_lists)
    counts = np.zeros(n, np.int64)
    by_sizes = {}
    for k, classes in enumerate(class_lists):
        by_sizes.setdefault(tuple(map(len, classes)), []).append(k)
    made = {}
    for sizes, members in by_sizes.items():
        ways = 1
        for size in sizes:
            ways *= factorial(size) if size < 5 else MAX_MIRRORS + 2
        if ways - 1 > MAX_MIRRORS:
            continue
        perms = _perm_swaps(sizes)
        if not perms:
            continue
        groups = np.array([[g for c in class_lists[k] for g in c] for k in members], np.uint64)
        words = np.empty((len(members), len(perms)), np.uint64)
        for q, ex in enumerate(perms):
            w = np.full(len(members), 0xFFFFFFFFFFFFFFFF, np.uint64)
            for t, (i, j) in enumerate(ex):
                w &= np.uint64(~(0xFFFF << (16 * t)) & 0xFFFFFFFFFFFFFFFF)
                w |= (groups[:, i] | (groups[:, j] << np.uint64(8))) << np.uint64(16 * t)
            words[:, q] = w
        counts[members] = len(perms)
        made[sizes] = (np.asarray(members, np.int64), words)
    out = np.empty(int(counts.sum()), np.uint64)
    start = np.cumsum(counts) - counts
    for members, words in made.values():
        pos = start[members][:, None] + np.arange(words.shape[1])[None, :]
        out[pos] = words
    return counts, out


def _arrangements(classes) -> int:
    count = 1
    for cls in classes:
        count *= factorial(len(cls)) if len(cls) < 5 else MAX_MIRRORS + 2
    return count


def twin_groups(B, M, grp_b, grp_g, cfg_col, n_in_group, placed_model):
    """Classes of groups of one placement with the same parallel config and
    the same set of models (flat arrays as in encode_placements).  Such groups
    are interchangeable: which of them is ahead after a stretch of the trace
    depends on history long past, and a speculative chunk may come out with
    their roles permuted.  Returns [(placement index, [[group ids], ...])] for
    the placements that have any and at most MAX_MIRRORS + 1 ways of arranging
    them.  The sets are compared through a 64-bit sum
    of random per-model keys; a collision could only cost speed, never
    exactness."""
    tot_groups = len(grp_b)
    if tot_groups < 2 or len(placed_model) == 0:
        return []
    if M not in _MODEL_KEYS:
        _MODEL_KEYS[M] = np.random.RandomState(20240229).randint(
            1, 2 ** 62, size=max(M, 1), dtype=np.int64).astype(np.uint64)
    with np.errstate(over="ignore"):
        csum = np.concatenate((np.zeros(1, np.uint64),
                               np.cumsum(_MODEL_KEYS[M][placed_model], dtype=np.uint64)))
        ends = np.cumsum(n_in_group)
        key = (csum[ends] - csum[ends - n_in_group]) * np.uint64(0x9E3779B97F4A7C15) \
            + cfg_col.astype(np.uint64) * np.uint64(0xC2B2AE3D27D4EB4F) + n_in_group.astype(np.uint64)
    # keys as a [B][G] matrix (unused cells and empty groups get keys of their own: top bit
    # set, which no hash has), each row sorted on its own: equal neighbours are a class
    G = int(grp_g.max()) + 1
    mat = (np.arange(B * G, dtype=np.uint64) | np.uint64(1 << 63)).reshape(B, G)
    live = n_in_group > 0
    mat[grp_b[live], grp_g[live]] = key[live] & np.uint64((1 << 63) - 1)
    order = np.argsort(mat, axis=1)
    srt = np.take_along_axis(mat, order, axis=1)
    same = srt[:, 1:] == srt[:, :-1]
    rows, cols = np.nonzero(same)                     # sorted by row, then column
    lo_ids = order[rows, cols].tolist()
    hi_ids = order[rows, cols + 1].tolist()
    out = []
    prev_b, prev_c = -1, -2
    for b, c, g_lo, g_hi in zip(rows.tolist(), cols.tolist(), lo_ids, hi_ids):
        if b != prev_b:
            out.append((b, []))
        if b == prev_b and c == prev_c + 1:
            out[-1][1][-1].append(g_hi)                # the run of equal keys goes on
        else:
            out[-1][1].append([g_lo, g_hi])
        prev_b, prev_c = b, c
    for _, classes in out:
        for cls in classes:
            cls.sort()
    # placements with more arrangements than get mirrors are of no use to anyone
    return [(b, classes) for b, classes in out if _arrangements(classes) <= MAX_MIRRORS + 1]


def _flatten(placements):
    """(groups per placement i64[B], configs i64[groups][3] = (dp, op, pp),
    models per group i64[groups], the models of all groups i64[pairs]) in
    placement order: by the C helper when it is built, else by passes over the
    Python objects."""
    B = len(placements)
    H = nat.host_lib()
    if H is not None and isinstance(placements, (list, tuple)):
        n_groups = np.zeros(B, np.int64)
        n_pairs = np.zeros(B, np.int64)
        # one pass with room for 96 groups and 256 (group, model) pairs per placement
        # (untouched room costs nothing) ...
        cap_g, cap_p = 96 * B + 64, 256 * B + 256
        cfg = np.empty((cap_g, 3), np.int64)
        n_in_group = np.empty(cap_g, np.int64)
        placed_model = np.empty(cap_p, np.int64)
        totals = np.zeros(2, np.int64)
        rc = H.mms_host_flatten_once(placements, n_groups.ctypes.data, n_pairs.ctypes.data,
                                     cfg.ctypes.data, n_in_group.ctypes.data,
                                     placed_model.ctypes.data, cap_g, cap_p, totals.ctypes.data)
        if rc == 0:
            tg, tp = int(totals[0]), int(totals[1])
            return n_groups, cfg[:tg], n_in_group[:tg], placed_model[:tp]
        if rc != -2:
            raise RuntimeError("mms_host_flatten_once failed")   # a Python exception is normally set
        # ... else count first, then fill
        if H.mms_host_scan(placements, n_groups.ctypes.data, n_pairs.ctypes.data) != 0:
            raise RuntimeError("mms_host_scan failed")
        tot_groups, tot_placed = int(n_groups.sum()), int(n_pairs.sum())
        cfg = np.zeros((tot_groups, 3), np.int64)
        n_in_group = np.zeros(tot_groups, np.int64)
        placed_model = np.zeros(tot_placed, np.int64)
        if H.mms_host_flatten(placements, cfg.ctypes.data, n_in_group.ctypes.data,
                              placed_model.ctypes.data, tot_groups, tot_placed) != 0:
            raise RuntimeError("mms_host_flatten failed")
        return n_groups, cfg, n_in_group, placed_model
    all_cfgs = list(chain.from_iterable(p.group_configs for p in placements))
    all_groups = list(chain.from_iterable(p.group_models for p in placements))
    n_groups = np.fromiter(map(len, (p.group_configs for p in placements)), np.int64, B)
    tot_groups = len(all_cfgs)
    if len(all_groups) != tot_groups:
        raise ValueError("group_configs and group_models differ in length")
    cfg = np.fromiter(chain.from_iterable(c[:3] for c in all_cfgs), np.int64,
                      3 * tot_groups).reshape(tot_groups, 3)
    n_in_group = np.fromiter(map(len, all_groups), np.int64, tot_groups)
    placed_model = np.fromiter(chain.from_iterable(all_groups), np.int64, int(n_in_group.sum()))
    return n_groups, cfg, n_in_group, placed_model


def _too_large(G, T, S, C):
    if G > nat.MAX_GROUPS or T > nat.MAX_SLOTS or S > nat.MAX_STAGES or C > nat.MAX_COLUMNS:
        raise NotImplementedError(
            f"placement too large for the kernels: {G} groups (max {nat.MAX_GROUPS}), "
            f"{T} pipeline stages in total (max {nat.MAX_SLOTS}), {C} parallel configs "
            f"(max {nat.MAX_COLUMNS})")


def _encode_native(H, B, M, table, n_groups, cfg, n_in_group, placed_model) -> EncodedBatch:
    """encode_placements behind the flattening, by csrc/encode_host.c."""
    tot_groups = len(n_in_group)
    cfg = np.ascontiguousarray(cfg)
    uniq = np.zeros((nat.MAX_COLUMNS + 1, 3), np.int64)
    cfg_index = np.zeros(max(tot_groups, 1), np.int32)
    n_uniq = H.mms_host_configs(cfg.ctypes.data, tot_groups, uniq.ctypes.data, len(uniq),
                                cfg_index.ctypes.data)
    if n_uniq < 0:
        raise NotImplementedError(f"more than {nat.MAX_COLUMNS} parallel configs in one batch")
    # new columns are handed out in ascending (dp, op, pp)
    found = [ParallelConfig(*map(int, row)) for row in uniq[:n_uniq]]
    table.columns_for(sorted(found))
    column_of = np.fromiter(map(table.column.__getitem__, found), np.int64, n_uniq)
    G = int(n_groups.max()) if B else 0
    S, C = int(table.max_stages), len(table.configs)
    _too_large(G, 0, S, C)
    # pairs per placement: the sums of n_in_group over each placement's groups
    ends = np.cumsum(n_groups)
    csum = np.concatenate(([0], np.cumsum(n_in_group)))
    placed_per_b = csum[ends] - csum[ends - n_groups] if B else np.zeros(0, np.int64)
    P = int(placed_per_b.max()) if B else 0
    if P > nat.MAX_PLACED:
        raise NotImplementedError(f"{P} (group, model) pairs in one placement (max {nat.MAX_PLACED})")
    Gc, Pc = max(G, 1), max(P, 1)
    model_off = np.zeros((B, M + 1), np.uint16)
    model_rep = np.zeros((B, Pc), np.uint32)
    group_info = np.zeros((B, Gc), np.uint32)
    slots = np.zeros(max(B, 1), np.int64)
    items = np.empty((max(tot_groups, 1), 3), np.int32)
    n_items = np.zeros(1, np.int64)
    has_twins = np.zeros(max(B, 1), np.uint8)
    counts = np.zeros(M + 1, np.int64)
    mark = np.zeros(max(M, 1), np.int64)
    n_groups = np.ascontiguousarray(n_groups, np.int64)
    rc = H.mms_host_encode(B, M, Gc, Pc, n_groups.ctypes.data, cfg.ctypes.data,
                           cfg_index.ctypes.data, column_of.ctypes.data, n_in_group.ctypes.data,
                           placed_model.ctypes.data, model_off.ctypes.data, model_rep.ctypes.data,
                           group_info.ctypes.data, slots.ctypes.data, items.ctypes.data,
                           n_items.ctypes.data, has_twins.ctypes.data, counts.ctypes.data, mark.ctypes.data,
                           MAX_MIRRORS + 1)
    if rc == 1:
        raise IndexError("model id in group_models is out of range")
    T = int(slots[:B].max()) if B else 0
    _too_large(G, T, S, C)

    def twins():
        out = []
        prev_b, prev_c = -1, -1
        for b, c, g in items[:int(n_items[0])].tolist():
            if b != prev_b:
                out.append((b, []))
                prev_c = -1
            if c != prev_c:
                out[-1][1].append([])
            out[-1][1][-1].append(g)
            prev_b, prev_c = b, c
        return out

    return EncodedBatch(B, M, Gc, Pc, max(T, 1), S, C, model_off, model_rep, group_info,
                        n_groups, placed_per_b.astype(np.int64), twins, has_twins[:B].astype(bool))


def encode_placements(placements: Sequence, table: LatencyTable, num_models: int,
                      native: bool = True) -> EncodedBatch:
    """List of ModelPlacement -> compact tables.  Each placement is taken as
    given: group order decides dispatch ties (controller.py:596 is a strict
    '<' over groups in ascending id), so nothing is re-sorted.  With the host
    helper built (and `native`), one C pass makes the tables; else numpy does."""
    B = len(placements)
    M = int(num_models)
    n_groups, cfg, n_in_group, placed_model = _flatten(placements)
    tot_groups, tot_placed = len(n_in_group), len(placed_model)
    H = nat.host_lib() if native else None
    if H is not None:
        return _encode_native(H, B, M, table, n_groups, cfg, n_in_group, placed_model)
    # distinct (dp, op, pp) rows -> columns of the latency table
    cfg_key = (cfg[:, 0] << 40) | (cfg[:, 1] << 20) | cfg[:, 2]
    uniq, inverse = np.unique(cfg_key, return_inverse=True)
    uniq_cfgs = [ParallelConfig(int(k >> 40), int((k >> 20) & 0xFFFFF), int(k & 0xFFFFF))
                 for k in uniq]
    table.columns_for(uniq_cfgs)
    cfg_col = np.fromiter(map(table.column.__getitem__, uniq_cfgs), np.int64,
                          len(uniq_cfgs))[inverse] if tot_groups else np.zeros(0, np.int64)
    cfg_pp = cfg[:, 2].copy()
    if tot_placed and (placed_model.min() < 0 or placed_model.max() >= M):
        raise IndexError("model id in group_models is out of range")

    G = int(n_groups.max()) if B else 0
    grp_first = np.concatenate(([0], np.cumsum(n_groups)))[:-1]     # first flat group of b
    grp_b = np.repeat(np.arange(B), n_groups)                       # candidate of flat group
    grp_g = np.arange(tot_groups) - grp_first[grp_b]                # group id inside b
    # clock slots: exclusive prefix sum of stages inside each candidate
    csum = np.cumsum(cfg_pp)
    base = np.concatenate(([0], csum))[grp_first]
    slot_first = (csum - cfg_pp) - base[grp_b]
    slots_per_b = np.bincount(grp_b, weights=cfg_pp, minlength=B).astype(np.int64)
    T = int(slots_per_b.max()) if B else 0
    S = int(table.max_stages)
    C = len(table.configs)
    _too_large(G, T, S, C)

    # (candidate, model, group) triples, ordered by model then group inside b
    pl_grp = np.repeat(np.arange(tot_groups), n_in_group)           # flat group of each pair
    pl_b = grp_b[pl_grp]
    pl_g = grp_g[pl_grp]
    # one composite key: by candidate, then model, then group id
    order = np.argsort((pl_b * max(M, 1) + placed_model) * (G + 1) + pl_g)      # keys are unique
    pl_b, pl_g, pl_m, pl_grp = pl_b[order], pl_g[order], placed_model[order], pl_grp[order]
    placed_per_b = np.bincount(pl_b, minlength=B) if tot_placed else np.zeros(B, np.int64)
    P = int(placed_per_b.max()) if B else 0
    if P > nat.MAX_PLACED:
        raise NotImplementedError(f"{P} (group, model) pairs in one placement (max {nat.MAX_PLACED})")
    pair_first = np.concatenate(([0], np.cumsum(placed_per_b)))[:-1]
    pos = np.arange(tot_placed) - pair_first[pl_b]
    model_rep = np.zeros((B, max(P, 1)), np.uint32)
    model_rep[pl_b, pos] = (pl_g | (slot_first[pl_grp] << 8) | (cfg_pp[pl_grp] << 16)
                            | (cfg_col[pl_grp] << 24)).astype(np.uint32)
    counts = np.bincount(pl_b * (M + 1) + pl_m + 1, minlength=B * (M + 1)).reshape(B, M + 1)
    model_off = np.cumsum(counts, axis=1).astype(np.uint16)
    # a group is contested when one of its models has more than one replica
    replicas = counts[pl_b, pl_m + 1]
    contested = (np.bincount(pl_grp, weights=(replicas > 1), minlength=tot_groups) > 0
                 ).astype(np.int64)
    group_info = np.zeros((B, max(G, 1)), np.uint32)
    group_info[grp_b, grp_g] = (slot_first | (cfg_pp << 8) | (contested << 16)).astype(np.uint32)

    twins = twin_groups(B, M, grp_b, grp_g, cfg_col, n_in_group, placed_model)
    return EncodedBatch(B, M, max(G, 1), max(P, 1), max(T, 1), S, C, model_off, model_rep,
                        group_info, n_groups, placed_per_b.astype(np.int64), twins)


class BatchResult:
    """Outputs of one launch, as numpy arrays on the host."""
    __slots__ = ("model_num_requests", "model_num_good", "group_num_requests",
                 "group_num_good", "good_total", "latency_sum", "status", "finish", "good",
                 "resimulated", "finish_device", "good_device")

    def __init__(self):
        # per-request outputs left on the GPU (f64[B][N], u8[B][N]) when a caller asked for that
        self.finish_device = self.good_device = None

    @staticmethod
    def concatenate(parts):
        """Results of consecutive sub-batches as one (per-request outputs are
        not carried); group columns are padded to the widest part."""
        res = BatchResult()
        G = max(p.group_num_requests.shape[1] for p in parts)

        def wide(a):
            return np.pad(a, ((0, 0), (0, G - a.shape[1])))
        res.model_num_requests = np.concatenate([p.model_num_requests for p in parts])
        res.model_num_good = np.concatenate([p.model_num_good for p in parts])
        res.group_num_requests = np.concatenate([wide(p.group_num_requests) for p in parts])
        res.group_num_good = (np.concatenate([wide(p.group_num_good) for p in parts])
                              if parts[0].group_num_good is not None else None)
        for name in ("good_total", "latency_sum", "status", "resimulated"):
            setattr(res, name, np.concatenate([getattr(p, name) for p in parts]))
        res.finish = res.good = None
        return res


class BatchSummary:
    """What callers read from an encoded batch after evaluation, for a batch
    that was encoded and launched in several parts."""

    def __init__(self, encs):
        self.parts = encs
        self.B = sum(e.B for e in encs)
        self.num_groups = np.concatenate([e.num_groups for e in encs])
        self.num_replicas = np.concatenate([e.num_replicas for e in encs])


def sim_options(chunk_requests=0, warmup_requests=0, repair_rounds=0, repair_segments=0):
    """How the trace is cut for time-parallel execution (mms_sim_options):
    0 lets the library choose, chunk_requests < 0 forces one chunk.  Results
    never depend on these numbers, only the run time does."""
    return nat.SimOptions(int(chunk_requests), int(warmup_requests), int(repair_rounds),
                          int(repair_segments))


class _Pending:
    """A submitted launch: device tensors and what collect() needs."""
    __slots__ = ("keep", "buf", "fields", "rows", "B", "M", "N", "full", "h2d", "stream",
                 "scratch", "call", "trace")

    def field(self, name):
        """One output as a device tensor (a view of the launch's output buffer)."""
        at, size, dtype, shape = self.fields[name]
        return self.buf[at:at + size].view(_TORCH_TYPE[np.dtype(dtype)]).reshape(shape)


# Scratch buffers of finished launches, per device, kept for the next ones: a
# search scores batch after batch of slowly changing size, and a fresh
# cudaMalloc for each would cost more than the kernels.  A buffer is handed to
# one launch at a time (taken in _submit, returned in _collect).
_SCRATCH_POOL = {}


def _take_scratch(dev, need):
    pool = _SCRATCH_POOL.setdefault(dev, [])
    fits = [k for k, t in enumerate(pool) if t.numel() >= need]
    if fits:
        return pool.pop(min(fits, key=lambda k: pool[k].numel()))
    if pool:                       # grow instead of hoarding: drop the largest idle one
        pool.pop(max(range(len(pool)), key=lambda k: pool[k].numel()))
    return torch.empty(max(int(need * 1.25), 1 << 20), dtype=torch.uint8, device=dev)


def _return_scratch(dev, t):
    pool = _SCRATCH_POOL.setdefault(dev, [])
    if len(pool) < 8:
        pool.append(t)


def _submit(trace: DeviceTrace, B, M, G, P, T, S, C, model_off, model_rep, group_info,
            latency, latency_stride, flags, want_group_good, pinned=False,
            options=None) -> _Pending:
    """Uploads the tables and enqueues mms_sim_mixed on the current stream;
    nothing waits for the GPU."""
    job = _prepare(trace, B, M, G, P, T, S, C, model_off, model_rep, group_info, latency,
                   latency_stride, flags, want_group_good, pinned, options)
    _enqueue(job)
    return job


def _enqueue(job: _Pending):
    """The C call of a prepared launch, on the current stream (again and
    again, if the caller wishes: everything it reads stays on the device)."""
    trace = job.trace
    cands, opts, ws, out, flags = job.call
    with _on(trace.device):
        tr, plan = trace.c_trace(), trace.c_plan()
        rc = nat.lib().mms_sim_mixed(ctypes.byref(tr), ctypes.byref(cands), ctypes.byref(plan),
                                     _ptr(trace.model_hist), ctypes.byref(opts), ctypes.byref(ws),
                                     ctypes.byref(out), flags, _stream_ptr())
        nat.check(rc, "mms_sim_mixed")
        # None: the default stream
        job.stream = torch.cuda.current_stream() if _raw_stream() else None


def _prepare(trace: DeviceTrace, B, M, G, P, T, S, C, model_off, model_rep, group_info,
             latency, latency_stride, flags, want_group_good, pinned=False,
             options=None) -> _Pending:
    """Uploads the tables and allocates scratch and outputs of one launch."""
    _require_cuda()
    L = nat.lib()
    dev = trace.device
    N = trace.num_requests
    opts = options if options is not None else sim_options()
    flags |= getattr(trace, "flags", 0)
    if not want_group_good:
        flags |= nat.FLAG_NO_GROUP_GOOD
    job = _Pending()
    with _on(dev):
        h2d = model_off.nbytes + model_rep.nbytes + group_info.nbytes
        tables = (model_off, model_rep, group_info)
        host_latency = not isinstance(latency, torch.Tensor)
        if host_latency:
            tables += (latency,)
        if pinned:
            d_tables = [_to_device(t, dev, pinned) for t in tables]
            at_tables = [_ptr(t) for t in d_tables]
        else:
            d_tables, at_tables = _upload(tables, dev)
        cands = nat.Placements(B, M, G, P, T, S, C, 0, *at_tables[:3],
                               at_tables[3] if host_latency else _ptr(latency), int(latency_stride),
                               None, None)
        need = L.mms_sim_workspace_bytes(N, ctypes.byref(cands), ctypes.byref(opts), flags)
        if need == 0 and B > 0:
            raise NotImplementedError("placement batch outside the kernel limits "
                                      "(see MMS_MAX_* in include/mms_sim.h)")
        ws_t = _take_scratch(dev, max(need, 256))
        ws = nat.Workspace(_ptr(ws_t), need)
        # the outputs in one buffer: one allocation here, one transfer when they are read
        rows = max(B, 1)
        fields, total = _layout((
            ("good_total", np.int64, (rows,)), ("latency_sum", np.float64, (rows,)),
            ("model_num_requests", np.int32, (rows, max(M, 1))),
            ("model_num_good", np.int32, (rows, max(M, 1))),
            ("group_num_requests", np.int32, (rows, G)),
            ("group_num_good", np.int32, (rows, G) if want_group_good else None),
            ("status", np.uint32, (rows,)), ("resimulated", np.int32, (rows,))))
        buf = torch.empty(total, dtype=torch.uint8, device=dev)
        full = bool(flags & nat.FLAG_PER_REQUEST)
        o_fin = torch.empty((rows, max(N, 1)), dtype=torch.float64, device=dev) if full else None
        o_good = torch.empty((rows, max(N, 1)), dtype=torch.uint8, device=dev) if full else None
        base = buf.data_ptr()

        def at(name):
            return ctypes.c_void_p(base + fields[name][0] if name in fields else 0)
        out = nat.Results(at("model_num_requests"), at("model_num_good"), at("group_num_requests"),
                          at("group_num_good"), at("good_total"), at("latency_sum"), at("status"),
                          _ptr(o_fin), _ptr(o_good), at("resimulated"))
    job.stream = None
    job.call = (cands, opts, ws, out, flags)
    job.trace = trace
    job.keep = (d_tables, latency)
    job.scratch = ws_t
    job.buf, job.fields, job.rows = buf, fields, (o_fin, o_good)
    job.B, job.M, job.N, job.full = B, M, N, full
    job.h2d = h2d
    return job


def _to_host(t):
    """A device tensor as a numpy array of its own.  Larger ones pass through page-locked
    memory (torch's host allocator keeps such blocks): the transfer runs at several
    times the rate of one into pageable memory."""
    if t.numel() * t.element_size() < (256 << 10):
        return t.cpu().numpy()
    stage = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    stage.copy_(t, non_blocking=True)
    torch.cuda.current_stream(t.device).synchronize()
    return stage.numpy().copy()


def _on_stream(stream, dev):
    """`dev` as the current device and `stream` (None: the default one) as its current stream, where they
    are not."""
    if _raw_stream(dev.index) == (stream.cuda_stream if stream is not None else 0):
        return _on(dev)
    return torch.cuda.stream(stream if stream is not None else torch.cuda.default_stream(dev))


def _download(job: _Pending, rows_on_device=False):
    """Waits for the launch and copies its results to the host.  Returns
    (BatchResult, d2h_bytes).  rows_on_device: the per-request outputs are not
    downloaded; the result carries the device tensors instead."""
    B, M, N, full = job.B, job.M, job.N, job.full
    o_fin, o_good = job.rows
    res = BatchResult()
    host_rows = full and not rows_on_device
    with _on_stream(job.stream, job.buf.device):
        host = _to_host(job.buf)
        for name, (at, size, dtype, shape) in job.fields.items():
            setattr(res, name, host[at:at + size].view(dtype).reshape(shape)[:B])
        res.model_num_requests = res.model_num_requests[:, :M]
        res.model_num_good = res.model_num_good[:, :M]
        if "group_num_good" not in job.fields:
            res.group_num_good = None
        res.finish = _to_host(o_fin[:B, :N]) if host_rows else None
        res.good = _to_host(o_good[:B, :N]).view(bool) if host_rows else None
        if full and rows_on_device:
            res.finish_device, res.good_device = o_fin[:B, :N], o_good[:B, :N]
    d2h = sum(x.nbytes for x in (res.model_num_requests, res.model_num_good,
                                 res.group_num_requests, res.good_total, res.latency_sum,
                                 res.status))
    if host_rows:
        d2h += res.finish.nbytes + res.good.nbytes
    return res, d2h


def _release(job: _Pending):
    """Hands the scratch buffer back; every kernel that used it has finished."""
    job.keep = job.buf = job.rows = job.call = None
    if job.scratch is not None:
        _return_scratch(job.scratch.device, job.scratch)
        job.scratch = None


def _check_status(res):
    if np.any(res.status):
        bad = int(np.flatnonzero(res.status)[0])
        raise RuntimeError(f"simulator kernel reported status {int(res.status[bad])} "
                           f"for candidate {bad} (bad table index or capacity overflow)")


def _collect(job, rows_on_device=False):
    """Waits for a submitted launch and downloads its results.  Returns
    (BatchResult, h2d_bytes, d2h_bytes)."""
    if isinstance(job, ResidentBatch):
        res, d2h = job.results()
        h2d = job.h2d_bytes
        job.release()
        _check_status(res)
        return res, h2d, d2h
    res, d2h = _download(job, rows_on_device)
    h2d = job.h2d
    _release(job)
    _check_status(res)
    return res, h2d, d2h


def _launch(*args, rows_on_device=False, **kwargs):
    """_submit + _collect: uploads the tables, runs mms_sim_mixed on the current
    stream, downloads the results.  Returns (BatchResult, h2d_bytes, d2h_bytes)."""
    return _collect(_submit(*args, **kwargs), rows_on_device)


# Placements from which a list is ordered by depth (by_depth): below, making the copies costs more
# than neighbours that wait less for one another give.
MIN_BY_DEPTH = 128

# A batch is split when it has at least so many placements without interchangeable groups ...
SPLIT_MIN_EASY = 512
# ... or so many, when all its placements together simulate so many requests: a second launch costs
# 0.15 to 0.2 ms, and one whose launches are short of candidates cuts both finer.  As one call and as
# two, ms: 442 on 8 devices over 3 300 requests 1.24 and 1.41, 420 random ones over 100 000 on 16 devices
# 5.48 and 4.54, on 64 6.20 and 6.84, 500 over 180 000 on 64 9.8 and 8.5; 1000 grown ones over 100 000,
# 650 of them with interchangeable groups, on 16 devices 9.32 and 8.53, on 64 29.4 and 26.2.  With fewer
# than 256: 700 grown ones over 100 000, on 32 devices 10.4 and 12.2, on 64 23.2 and 32.7.
SPLIT_MIN_EASY_LONG = 256
SPLIT_LONG = 64e6
SPLIT_MIN_HARD = 32       # ... and so many with such groups
_SIDE_STREAMS = {}


def _side_streams(main):
    """Two side streams per calling stream, so that batches launched from
    different streams do not queue up behind each other."""
    key = (main.device, main.cuda_stream)
    if key not in _SIDE_STREAMS:
        _SIDE_STREAMS[key] = (torch.cuda.Stream(device=main.device),
                              torch.cuda.Stream(device=main.device))
    return _SIDE_STREAMS[key]


def _calls_of(trace, enc, split, mirrors):
    """The calls a batch is simulated in: [placement indices in the order of simulation, or None for all
    as they are].  Where every placement has a trace of its own, placement k is simulated on trace k,
    so such a batch is one call and stays in order."""
    if getattr(trace, "num_traces", 1) > 1:
        return [None]
    parts = [None]
    if split and mirrors and enc.has_twins is not None:
        hard = np.flatnonzero(enc.has_twins)
        least = SPLIT_MIN_EASY
        if trace.num_requests * enc.B >= SPLIT_LONG:
            least = min(least, SPLIT_MIN_EASY_LONG)
        if len(hard) >= SPLIT_MIN_HARD and enc.B - len(hard) >= least:
            parts = [hard, np.flatnonzero(~enc.has_twins)]
    return [enc.by_depth(index) for index in parts]


class StreamLease:
    """`count` streams of a device that nobody else has, until give_back() (or the end of this
    object).  torch.cuda.Stream() hands out 32 streams in turn: of streams made for each call two
    soon are one, and what was to run beside a kernel of 40 ms waits behind it; and torch keeps
    freed memory by stream, so each new one begins with none."""

    _lock = threading.RLock()       # (give_back may be called by the garbage collector)
    _known, _free = {}, {}          # per device: handles that were ever lent, streams at hand

    def __init__(self, count, main):
        """main: the calling stream, which is not among them."""
        dev = main.device
        self.device, self.streams = dev, []
        with self._lock:
            known, free = self._known.setdefault(dev, set()), self._free.setdefault(dev, [])
            while len(self.streams) < count:
                spare = [s for s in free if s.cuda_stream != main.cuda_stream]
                if spare:
                    stream = spare[-1]
                    free.remove(stream)
                else:
                    for _ in range(32):         # beyond that many there are no others: shared
                        stream = torch.cuda.Stream(device=dev)
                        if stream.cuda_stream not in known and stream != main:
                            break
                    known.add(stream.cuda_stream)
                self.streams.append(stream)

    def give_back(self):
        with self._lock:
            free = self._free[self.device]
            # (in the order in which they go out again)
            free.extend(s for s in reversed(self.streams) if s not in free)
            self.streams = []

    __del__ = give_back


class ResidentBatch:
    """An encoded batch with its tables, scratch and outputs on the GPU, ready
    to be launched (any number of times).

    A batch whose placements partly have interchangeable groups is launched as
    TWO calls of mms_sim_mixed on two side streams: those placements first, and
    the rest, for which the library then needs no bookkeeping of such groups
    (FLAG_NO_TWINS), beside them.  The first are few and finish their
    speculative pass early; their repairs — serial re-simulations that leave
    the GPU almost idle — run while the rest are still in theirs.  Results
    are the same as from one call."""

    def __init__(self, trace, enc: EncodedBatch, table: LatencyTable, group_good=False,
                 pinned=False, options=None, mirrors=True, split=True, crowded=False,
                 hard_options=None, launch_now=False):
        """mirrors: False = the library does not look for interchangeable groups
        (slower on placements that have them).
        crowded: another batch is to run beside this one (MMS_FLAG_CROWDED, a hint; passed
        for a split batch in any case).
        hard_options: sim_options for the launch that holds the placements with
        interchangeable groups, when the batch is split (default: `options`).
        launch_now: every call is enqueued as soon as its tables are uploaded
        (as launch() would afterwards), so that the GPU starts on the first
        while the host prepares the second."""
        self.trace, self.enc = trace, enc
        dev = trace.device
        parts = [(index, enc if index is None else enc.take(index))
                 for index in _calls_of(trace, enc, split, mirrors)]
        self.index = [p[0] for p in parts]
        self.jobs = []
        self.h2d_bytes = 0
        self.launched = False
        lat = table.device(dev)
        main = sides = None
        if launch_now and len(parts) > 1:
            main = torch.cuda.current_stream(dev)
            sides = _side_streams(main)
        for k, (_, e) in enumerate(parts):
            flags = nat.FLAG_CROWDED if crowded or len(parts) > 1 else 0
            if not mirrors or not e.may_have_twins():
                flags |= nat.FLAG_NO_TWINS
            opts_k = hard_options if len(parts) > 1 and k == 0 and hard_options is not None else options
            job = _prepare(trace, e.B, e.M, e.G, e.P, e.T, e.S, e.C, e.model_off, e.model_rep,
                           e.group_info, lat, 0, flags, group_good, pinned, opts_k)
            self.jobs.append(job)
            self.h2d_bytes += job.h2d
            if launch_now:              # the GPU starts on this call while the next is prepared
                if sides is None:
                    _enqueue(job)
                else:
                    sides[k].wait_stream(main)
                    with torch.cuda.stream(sides[k]):
                        _enqueue(job)
        if launch_now:
            if sides is not None:
                for side in sides:
                    main.wait_stream(side)
                for job in self.jobs:   # results are read in order behind the join
                    job.stream = main
            self.launched = True

    def launch(self):
        """Enqueues the call(s); stream-ordered with respect to the current
        stream on both sides, nothing waits for the GPU."""
        if len(self.jobs) == 1:
            _enqueue(self.jobs[0])
            return self
        main = torch.cuda.current_stream(self.trace.device)
        sides = _side_streams(main)
        for job, side in zip(self.jobs, sides):
            side.wait_stream(main)
            with torch.cuda.stream(side):
                _enqueue(job)
        for side in sides:
            main.wait_stream(side)
        for job in self.jobs:           # results are read in order behind the join
            job.stream = main
        return self

    def device_outputs(self):
        """[(candidate indices or None, good_total i64[.], latency_sum f64[.])] per call, on the
        device."""
        return [(idx, job.field("good_total")[:job.B], job.field("latency_sum")[:job.B])
                for idx, job in zip(self.index, self.jobs)]

    def results(self):
        """Waits and downloads: (BatchResult in the order of the batch, d2h bytes)."""
        done = [_download(job) for job in self.jobs]
        d2h = sum(d[1] for d in done)
        if self.index[0] is None:
            return done[0][0], d2h
        res = BatchResult()
        B = self.enc.B
        for name in BatchResult.__slots__:
            first = getattr(done[0][0], name)
            if first is None:
                setattr(res, name, None)
                continue
            whole = np.zeros((B,) + first.shape[1:], first.dtype)
            for idx, (part, _) in zip(self.index, done):
                whole[idx] = getattr(part, name)
            setattr(res, name, whole)
        return res, d2h

    def release(self):
        for job in self.jobs:
            _release(job)


def submit_batch(trace: DeviceTrace, enc: EncodedBatch, table: LatencyTable, group_good=False,
                 pinned=False, options=None, mirrors=True, split=True,
                 crowded=False) -> ResidentBatch:
    """run_batch without waiting: returns a handle for collect_batch."""
    return ResidentBatch(trace, enc, table, group_good, pinned, options, mirrors, split,
                         crowded, launch_now=True)


collect_batch = _collect


def run_batch(trace: DeviceTrace, enc: EncodedBatch, table: LatencyTable,
              per_request=False, group_good=False, pinned=False, options=None, mirrors=True,
              split=True, crowded=False, rows_on_device=False):
    """Simulates every placement of `enc` against `trace`
    (simulate_requests_mixed, controller.py:561-628).  `mirrors`: the library
    may take over speculative runs in which interchangeable groups have changed
    places (a speed-up of the time-parallel execution; results are the same
    with and without).
    `crowded`: passes MMS_FLAG_CROWDED, a hint that another batch is to run beside this one.
    `rows_on_device` (with per_request): finish and good stay on the GPU, as
    BatchResult.finish_device / .good_device."""
    if not per_request:
        return _collect(submit_batch(trace, enc, table, group_good, pinned, options, mirrors,
                                     split, crowded))
    return _collect(_submit_rows(trace, enc, table, group_good, pinned, options, mirrors, crowded),
                    rows_on_device)


def _submit_rows(trace, enc, table, group_good, pinned, options, mirrors, crowded):
    """One launch with per-request outputs."""
    flags = (nat.FLAG_PER_REQUEST | (nat.FLAG_CROWDED if crowded else 0)
             | (0 if mirrors and enc.may_have_twins() else nat.FLAG_NO_TWINS))
    return _submit(trace, enc.B, enc.M, enc.G, enc.P, enc.T, enc.S, enc.C, enc.model_off,
                   enc.model_rep, enc.group_info, table.device(trace.device), 0, flags, group_good,
                   pinned, options)


def begin_batch_rows(trace: DeviceTrace, enc: EncodedBatch, table: LatencyTable, group_good=False,
                     options=None, rows_on_device=False):
    """run_batch(per_request=True) in two steps: enqueues and returns the function that waits."""
    job = _submit_rows(trace, enc, table, group_good, False, options, True, False)
    return lambda: _collect(job, rows_on_device)[0]


def encode_dense(m_id2g_id, num_stages, num_models):
    """One candidate given as the reference's dense tables (m_id2g_id [M][*]
    with -1 ending a row, num_stages [G]) -> (model_off, model_rep,
    group_info, T) with latency column = group id."""
    m2g = np.asarray(m_id2g_id, dtype=np.int64).reshape(num_models, -1)
    ns = np.asarray(num_stages, dtype=np.int64)
    G = len(ns)
    if G > nat.MAX_COLUMNS or (G and ns.max() > nat.MAX_STAGES) or ns.sum() > nat.MAX_SLOTS:
        raise NotImplementedError("placement too large for the kernels")
    slot_first = np.cumsum(ns) - ns
    rows, offs = [], [0]
    contested = np.zeros(G, np.int64)
    for m in range(num_models):
        row = m2g[m]
        stop = np.flatnonzero(row < 0)
        row = row[:stop[0]] if len(stop) else row
        if len(row) and (row.max() >= G):
            raise IndexError("group id in m_id2g_id is out of range")
        if len(row) > 1:
            contested[row] = 1
        rows.append(row | (slot_first[row] << 8) | (ns[row] << 16) | (row << 24))
        offs.append(offs[-1] + len(row))
    if offs[-1] > nat.MAX_PLACED:
        raise NotImplementedError("too many (group, model) pairs")
    rep = np.concatenate(rows).astype(np.uint32) if rows and offs[-1] else np.zeros(0, np.uint32)
    rep = rep.reshape(1, -1) if len(rep) else np.zeros((1, 1), np.uint32)
    off = np.asarray(offs, dtype=np.uint16).reshape(1, -1)
    info = (slot_first | (ns << 8) | (contested << 16)).astype(np.uint32).reshape(1, -1)
    if info.shape[1] == 0:
        info = np.zeros((1, 1), np.uint32)
    return off, rep, info, max(int(ns.sum()), 1)


def group_lists(model_off, model_rep, group_info, G):
    """g_id2m_id of controller.py:424-430 as CSR per candidate, from the
    compact tables: (group_off u16[B][G+1], group_mod u16[B][P], group_cfg
    u32[B][G] = first slot | stages << 8 | column << 16)."""
    B, P = model_rep.shape
    M = model_off.shape[1] - 1
    group_mod = np.zeros((B, P), np.uint16)
    counts = np.diff(model_off.astype(np.int64), axis=1)
    n = model_off[:, M].astype(np.int64)
    total = int(n.sum())
    b = np.repeat(np.arange(B), n)                       # candidate of each (model, group) pair
    first = np.cumsum(n) - n
    pos = np.arange(total) - first[b]
    ents = model_rep[b, pos].astype(np.int64)
    g = ents & 0xFF
    m = np.repeat(np.tile(np.arange(M), B), counts.reshape(-1))
    order = np.lexsort((m, g, b))                        # by candidate, group, models ascending
    group_mod[b, pos] = m[order]                         # (b[order] is b)
    per_group = np.bincount(b * G + g, minlength=B * G).reshape(B, G)
    group_off = np.zeros((B, G + 1), np.uint16)
    group_off[:, 1:] = np.cumsum(per_group, axis=1)
    col = np.zeros((B, G), np.int64)
    col[b, g] = ents >> 24
    group_cfg = ((group_info[:, :G].astype(np.int64) & 0xFFFF) | (col << 16)).astype(np.uint32)
    return group_off, group_mod, group_cfg


class ResidentBatching:
    """A placement batch for the batching simulator with its tables, scratch
    and outputs on the GPU, ready to be launched (any number of times) on the
    current stream."""

    def __init__(self, trace: DeviceTrace, B, M, G, P, T, S, C, model_off, model_rep, group_info,
                 latency, latency_stride, batch_sizes, heap_capacity=0):
        _require_cuda()
        L = nat.lib()
        dev = trace.device
        N = trace.num_requests
        self.trace, self.B, self.M, self.G, self.N = trace, B, M, G, N
        goff, gmod, gcfg = group_lists(model_off, model_rep, group_info, G)
        self.h2d_bytes = sum(x.nbytes for x in (model_off, model_rep, goff, gmod, gcfg))
        with _on(dev):
            tables = (model_off, model_rep, goff, gmod, gcfg)
            host_latency = not isinstance(latency, torch.Tensor)
            d_tables, at_tables = _upload(tables + ((latency,) if host_latency else ()), dev)
            self.cands = nat.Placements(B, M, G, P, T, S, C, 0, *at_tables[:2], None,
                                        at_tables[5] if host_latency else _ptr(latency),
                                        int(latency_stride))
            self.bat = nat.Batching(*at_tables[2:5], len(batch_sizes), int(heap_capacity),
                                    (ctypes.c_int32 * 8)(*list(batch_sizes)))
            need = L.mms_sim_batching_workspace_bytes(N, ctypes.byref(self.cands),
                                                      ctypes.byref(self.bat))
            ws_t = torch.empty(max(need, 256), dtype=torch.uint8, device=dev)
            self.ws = nat.Workspace(_ptr(ws_t), need)
            self.fields, total = _layout((
                ("good_total", np.int64, (B,)), ("latency_sum", np.float64, (B,)),
                ("model_num_requests", np.int32, (B, max(M, 1))),
                ("model_num_good", np.int32, (B, max(M, 1))),
                ("group_num_requests", np.int32, (B, G)), ("group_num_good", np.int32, (B, G)),
                ("status", np.uint32, (B,)), ("resimulated", np.int32, (B,))))
            self.buf = torch.zeros(total, dtype=torch.uint8, device=dev)
            o_fin = torch.empty((B, max(N, 1)), dtype=torch.float64, device=dev)
            o_good = torch.empty((B, max(N, 1)), dtype=torch.uint8, device=dev)
            base = self.buf.data_ptr()
            at = {name: ctypes.c_void_p(base + f[0]) for name, f in self.fields.items()}
            self.res = nat.Results(at["model_num_requests"], at["model_num_good"],
                                   at["group_num_requests"], at["group_num_good"],
                                   at["good_total"], at["latency_sum"], at["status"], _ptr(o_fin),
                                   _ptr(o_good), at["resimulated"])
        self.keep = (d_tables, latency, ws_t)
        self.rows = (o_fin, o_good)

    def launch(self):
        trace = self.trace
        with _on(trace.device):
            tr, plan = trace.c_trace(), trace.c_plan()
            rc = nat.lib().mms_sim_batching(ctypes.byref(tr), ctypes.byref(self.cands),
                                            ctypes.byref(self.bat), None,
                                            ctypes.byref(plan), ctypes.byref(self.ws),
                                            ctypes.byref(self.res), _stream_ptr())
            nat.check(rc, "mms_sim_batching")
        return self

    def results(self, per_request=True, rows_on_device=False):
        """Waits and downloads: (BatchResult, d2h bytes).  rows_on_device: the
        result carries the per-request outputs as device tensors."""
        o_fin, o_good = self.rows
        M, N = self.M, self.N
        res = BatchResult()
        host = _to_host(self.buf)
        for name, (at, size, dtype, shape) in self.fields.items():
            setattr(res, name, host[at:at + size].view(dtype).reshape(shape))
        res.model_num_requests = res.model_num_requests[:, :M]
        res.model_num_good = res.model_num_good[:, :M]
        res.finish = _to_host(o_fin[:, :N]) if per_request else None
        res.good = _to_host(o_good[:, :N]).view(bool) if per_request else None
        if rows_on_device:
            res.finish_device, res.good_device = o_fin[:, :N], o_good[:, :N]
        d2h = sum(x.nbytes for x in (res.model_num_requests, res.model_num_good,
                                     res.group_num_requests, res.group_num_good, res.good_total,
                                     res.latency_sum, res.status))
        if per_request:
            d2h += res.finish.nbytes + res.good.nbytes
        return res, d2h


def launch_batching(trace: DeviceTrace, B, M, G, P, T, S, C, model_off, model_rep, group_info,
                    latency, latency_stride, batch_sizes, heap_capacity=0, per_request=True,
                    rows_on_device=False):
    """simulate_requests_mixed_batching (controller.py:630-798) for every
    candidate.  The kernel always writes per-request outputs (the latency sums
    are formed from them); per_request=False does not download them."""
    return _begin_batching(trace, B, M, G, P, T, S, C, model_off, model_rep, group_info, latency,
                           latency_stride, batch_sizes, heap_capacity, per_request,
                           rows_on_device)()


def _begin_batching(trace, B, M, G, P, T, S, C, model_off, model_rep, group_info, latency,
                    latency_stride, batch_sizes, heap_capacity, per_request, rows_on_device):
    """launch_batching in two steps: enqueues and returns the function that waits."""
    def begin(capacity):
        return ResidentBatching(trace, B, M, G, P, T, S, C, model_off, model_rep, group_info,
                                latency, latency_stride, batch_sizes, capacity).launch()
    job = begin(heap_capacity)

    def collect():
        res, _ = job.results(per_request, rows_on_device)
        if heap_capacity == 0 and np.any(res.status & nat.STATUS_HEAP_OVERFLOW):
            # the default capacity (G + 16 pending events) is what the simulation was seen to
            # need; nothing bounds it, so a run that overflowed is repeated with room to spare
            res, _ = begin(8 * G + 64).results(per_request, rows_on_device)
        if np.any(res.status):
            bad = int(np.flatnonzero(res.status)[0])
            what = {nat.STATUS_HEAP_OVERFLOW: "event heap overflow (raise heap_capacity)",
                    nat.STATUS_QUEUE_LEFT: "a request was left queued",
                    nat.STATUS_BAD_INDEX: "bad table index"}
            raise RuntimeError(f"batching simulator reported status {int(res.status[bad])} for "
                               f"candidate {bad}: " + ", ".join(v for k, v in what.items()
                                                                if res.status[bad] & k))
        return res
    return collect


def resident_batching(trace: DeviceTrace, enc: EncodedBatch, table: LatencyTable,
                      heap_capacity=0) -> ResidentBatching:
    """ResidentBatching for an encoded batch and a table built with batch sizes."""
    if table.batch_sizes is None:
        raise ValueError("the latency table has no batch-size axis")
    return ResidentBatching(trace, enc.B, enc.M, enc.G, enc.P, enc.T, enc.S, enc.C,
                            enc.model_off, enc.model_rep, enc.group_info,
                            table.device(trace.device), 0, table.batch_sizes, heap_capacity)


def run_batch_batching(trace: DeviceTrace, enc: EncodedBatch, table: LatencyTable,
                       heap_capacity=0, per_request=True, rows_on_device=False):
    """Batching simulation of every placement of `enc`; `table` must have been
    built with batch sizes.  per_request=False leaves the per-request outputs
    (9 bytes per candidate and request) on the device."""
    return begin_batch_batching(trace, enc, table, heap_capacity, per_request, rows_on_device)()


def begin_batch_batching(trace: DeviceTrace, enc: EncodedBatch, table: LatencyTable,
                         heap_capacity=0, per_request=True, rows_on_device=False):
    """run_batch_batching in two steps: enqueues and returns the function that waits."""
    if table.batch_sizes is None:
        raise ValueError("the latency table has no batch-size axis")
    return _begin_batching(trace, enc.B, enc.M, enc.G, enc.P, enc.T, enc.S, enc.C, enc.model_off,
                           enc.model_rep, enc.group_info, table.device(trace.device), 0,
                           table.batch_sizes, heap_capacity, per_request, rows_on_device)


STATS_FIELDS = ("num_good", "first_start", "last_start", "latency_mean", "latency_std",
                "latency_p90", "latency_p99")


def device_compute_stats(arrivals, model_ids, num_models: int, finish, good, first: int,
                         window: int):
    """Workload.compute_stats (alpa_serve/simulator/workload.py:308-354) on the
    GPU, through mms_compute_stats: statistics of the requests [first, first +
    window) of per-request outputs that are already on the device.  arrivals
    f64[N], model_ids i32[N] (index into the WORKLOAD's names), finish f64[B][N],
    good u8[B][N]: torch tensors on one GPU.  Returns a dict of numpy arrays:
    num_requests i32[M]; num_good, first_start, last_start, latency_mean,
    latency_std, latency_p90, latency_p99 [B][M]; good_total i64[B],
    latency_sum f64[B]; and "d2h_bytes"."""
    _require_cuda()
    L = nat.lib()
    dev = finish.device
    if finish.dim() != 2 or good.shape != finish.shape or finish.stride(1) != 1 \
            or good.stride(1) != 1 or finish.stride(0) != good.stride(0):
        raise ValueError("finish and good must be [B][N] rows of one pitch")
    if finish.dtype != torch.float64 or good.dtype != torch.uint8:
        raise ValueError("finish must be float64 and good uint8")
    B, N = finish.shape
    M = int(num_models)
    first, window = int(first), int(window)
    if first < 0 or window < 0 or first + window > N or arrivals.numel() < N \
            or model_ids.numel() < N:
        raise ValueError("window outside the trace")
    with torch.cuda.device(dev):
        need = L.mms_compute_stats_workspace_bytes(window, M, B)
        if need == 0:
            raise NotImplementedError("statistics outside the kernel limits")
        ws_t = _take_scratch(dev, max(need, 256))
        ws = nat.Workspace(_ptr(ws_t), need)
        fields, total = _layout(
            [("good_total", np.int64, (B,)), ("latency_sum", np.float64, (B,))]
            + [(k, np.float64, (B, max(M, 1))) for k in STATS_FIELDS[1:]]
            + [("num_good", np.int32, (B, max(M, 1))), ("num_requests", np.int32, (max(M, 1),))])
        buf = torch.zeros(total, dtype=torch.uint8, device=dev)
        out = nat.StatsOut(*[ctypes.c_void_p(buf.data_ptr() + fields[k][0])
                             for k in ("num_requests",) + STATS_FIELDS + ("good_total", "latency_sum")])
        rc = L.mms_compute_stats(_ptr(arrivals), _ptr(model_ids), M, _ptr(finish), _ptr(good),
                                 finish.stride(0), B, first, window, ctypes.byref(ws),
                                 ctypes.byref(out), _stream_ptr())
        nat.check(rc, "mms_compute_stats")
        host = _to_host(buf)                                  # waits for the kernels
        _return_scratch(dev, ws_t)
    res = {k: host[at:at + size].view(dtype).reshape(shape)
           for k, (at, size, dtype, shape) in fields.items()}
    res["d2h_bytes"] = sum(v.nbytes for v in res.values())
    res["num_requests"] = res["num_requests"][:M]
    for name in STATS_FIELDS:
        res[name] = res[name][:, :M]
    return res
