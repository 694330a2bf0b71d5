// sim_batching.cuh — the batching simulator, one candidate per warp.
//
// Restates simulate_requests_mixed_batching
// (alpa_serve/simulator/controller.py:630-798; pure Python in the reference:
// closures, list queues and heapq).  Requests wait in one FIFO queue per
// MODEL; a group serves, when its first stage frees up, the model whose
// oldest queued request arrived first, batching as many of that model's
// queued requests as still meet the head request's deadline.
//
// A model's queue always holds a run of consecutive requests of that model.
// batch_order_kernel sorts the trace by model (stable), so a queue is a pair
// (position of its head, length) and the requests behind a head are its
// neighbours: nothing is stored per queued request, and 32 deadlines are one load.
//
// Arrivals are a serial chain; what a warp does in parallel is what each of
// them asks: the last-stage clocks of the model's replicas, the queue heads of
// a group's models and the pending events are compared by 32 lanes at a time,
// and the finish times of all batch sizes are worked out beside each other, a batch
// size per lane (batch_groups.cuh; batch_lists.cuh where that does not fit).  What bounds it is
// the latency of those steps, 1.0 us an arrival; 16 warps to an SM hide one another's.
// (One lane going through the reference's loops took 1.5 us an arrival; 32 candidates to a
// warp in step, each lane with its own control flow, 9 us for the 32 with room for two
// warps on an SM: 256 placements on 64 devices over 45 000 requests 28 ms, then 8.0, and the whole
// call 62 and 12.3; 1024 over 180 715 203 and 119 ms.)
//
// Like the unbatched path, the trace is cut into chunks that are simulated
// speculatively at the same time (idle start, a run-in, then the chunk; a
// snapshot of the state after every segment) and stitched exactly afterwards:
//   batch_validate_kernel  does the run of a chunk continue the run of the one before it
//                          (batch_equivalent)?  Lists those that do not, with the state they
//                          should have started from as far as known
//   batch_walk_kernel      simulates the listed chunks again, until the state meets the
//                          stored one or the chunk ends
//   batch_chain_kernel     goes through a candidate's chunks in order and simulates again,
//                          from the true state, what still does not fit, as far as it does not;
//                          runs in which interchangeable groups have changed places count as well
// A request that is queued at a chunk boundary is served by the NEXT chunk's
// run; a run that did not start from the true state does not write the outputs
// of such carried requests (a wrong guess would clobber what the chunk before it
// wrote) but lists them, and the chain kernel applies the list when it
// accepts the chunk.  The groups' counters are kept per segment.
#pragma once
#include "sim_core.cuh"

namespace mms {

constexpr int kBatchWarps = 8;          // warps of a block (they share the latency table), at most
constexpr int kBatchBlocksPerSm = 2;    // register budget: 128 per thread
constexpr int kMaxCarry = 120;          // carried requests a speculative chunk may list
constexpr int kGroupLimit = 64;          // groups, and models, of the kernels with a group per lane
constexpr int kOutRing = 64;            // outputs gathered on chip before they are written
constexpr int kBatchDepth = 8;          // stages whose times stay in registers
constexpr int kTallyThreads = 256;
constexpr int kTallyLeaves = kTallyThreads / 8;   // leaves of numpy's sum per tally block
constexpr double kNoHead = 2e100;       // head time of an empty queue: not below kInf
constexpr uint64_t kNoEvent = ~0ull;
constexpr uint32_t kNoCarry = 0xFFFFFFFFu;        // a carry list that overflowed
constexpr uint32_t kDropped = 0x80000000u;        // out ring: finish is the arrival time

struct Carried { double fin; uint32_t req, good; };
// A choice that the group number decided between interchangeable groups in the same state, and
// what those had counted since their last one (see other_labels).
constexpr int kSwapGroups = 4, kSwapCap = 64;
struct Swap {
    uint64_t groups;
    int32_t seg;
    uint32_t picked;
    uint16_t requests[kSwapGroups], good[kSwapGroups];    // of the groups in ascending order
};
constexpr uint8_t kLinkSame = 1, kLinkOther = 2;

// Shared memory of a warp of the kernels with a group per lane (GroupWarp); indices, each in the
// entry's own size, from the warp's first byte.
struct GroupSmem {
    uint32_t orders;                    // bytes
    uint32_t clk, head_ts, head_dl, extra, out_fin;      // f64
    uint32_t queue, serves, served;     // u64: position | length << 32; models of a group; groups of a model
    uint32_t info, out_pos;             // u32
    uint32_t extra_g, labels;           // u8
    size_t bytes;
};

struct __align__(16) BatchOrder {       // an arrival of the window at work
    double ts, dl;
    int32_t pos, m;
    uint64_t served;                    // its model's replicas: a list (first entry | count << 16) or
                                        //   a set of groups; 0: none
};

__host__ __device__ inline GroupSmem group_smem(int M, int T, int H)
{
    GroupSmem L;
    size_t off = 0;
    const auto take = [&](size_t size, size_t n) {
        const uint32_t at = (uint32_t)(off / size);
        off += size * n;
        return at;
    };
    L.orders = take(1, sizeof(BatchOrder) * kLanes);
    L.clk = take(8, T);
    L.head_ts = take(8, M);
    L.head_dl = take(8, M);
    L.extra = take(8, H);
    L.out_fin = take(8, kOutRing);
    L.queue = take(8, M);
    L.serves = take(8, kGroupLimit);
    L.served = take(8, M);
    L.info = take(4, kGroupLimit);
    L.out_pos = take(4, kOutRing);
    L.labels = take(1, kGroupLimit);
    L.extra_g = take(1, H);
    L.bytes = (off + 15) & ~(size_t)15;
    return L;
}

struct BatchArgs {
    const double *arrivals;
    const int32_t *model_ids;
    const float *slos;
    int64_t N;
    int32_t B, M, G, P, T, S, C, NB, H;
    int32_t event_rows;           // rows of 32 event slots: H rounded up
    uint32_t spare;               // H - G: events there is room for besides one of each group
    int32_t batch_sizes[8];
    int32_t batch_cols[8];        // log2 of the batch size: the column the reference reads
    const uint16_t *model_off;    // [B][M+1]
    const uint32_t *model_rep;    // [B][P]   group | first slot<<8 | stages<<16 | column<<24
    const uint16_t *group_off;    // [B][G+1]
    const uint16_t *group_mod;    // [B][P]   models of each group, ascending
    const uint32_t *group_cfg;    // [B][G]   first slot | stages<<8 | column<<16
    const float *latency;         // [M][C][S][NB]
    int64_t latency_stride;
    int32_t table_elems;          // entries of the on-chip latency table; 0: off chip
    GroupSmem at;                 // shared memory of the kernels with a group per lane: a warp's,
    uint32_t warp0, warp_bytes;   //   where the first warp's is, and its size
    double *finish;               // [B][N]
    uint8_t *good;                // [B][N]
    uint32_t *status;             // [B]
    int32_t *resimulated;         // [B] or null: chunks simulated again
    // the trace sorted by model
    int32_t *first_of;            // [M + 1] where each model's requests begin
    int32_t *pos;                 // [N] position of request i (of a known model)
    int32_t *req;                 // [.] request at a position, and its arrival time and deadline
    double *pos_ts, *pos_dl;
    // time-parallel execution
    int32_t K, NS;                // chunks, segments
    int32_t seg_len, seg_per_chunk;
    int32_t warmup;               // run-in arrivals of a speculative chunk
    const int32_t *odd;           // != 0: arrival times not sorted, not finite or negative, or a
                                  //   latency not >= 0 -> lists, one chunk
    bool only_odd;                // the list kernels run in that case alone
    size_t state_bytes;
    unsigned char *chunk_start;   // [K][B] state a chunk was started from
    unsigned char *seg_end;       // [NS][B] state after the segment's last arrival
    Carried *carry;               // [K][B][kMaxCarry] outputs of carried requests, in order
    uint32_t *carry_n;            // [K][B] how many (kNoCarry: too many)
    uint8_t *carry_seg;           // [NS][B] how many of them were listed in the segment
    Carried *walk_carry;          // [warps of a walk grid][kMaxCarry]
    uint32_t *run_status;         // [K][B] status word of the chunk's run
    uint8_t *link;                // [K][B]: the chunk's stored run continues that of the one before
                                  //   (kLinkSame), or does under other labels (kLinkOther)
    uint8_t *perm;                // [K][B][kGroupLimit], kLinkOther: label in this run -> label in that
                                  //   of the chunk before
    uint64_t *tie;                // [NS][B] groups that a group number decided about in the segment
    Swap *swaps;                  // [K][B][kSwapCap], in order
    uint32_t *swap_n;             // [K][B]
    Swap *walk_swaps;             // [warps of a walk grid][kSwapCap]
    uint32_t *seg_counts;         // [NS][B][2][G] requests and good ones of each label (but those in `swaps`)
    uint8_t *stamp;               // [K][B]: 1 + the last round in which the chunk was walked
    uint32_t *work_count;         // [rounds]
    uint32_t *work_next;          // [rounds]
    uint32_t *work_items;         // [K * B]: chunk * B + candidate
    int32_t round, rounds;
};

// Saved state: clocks f64[T], events u64[slots], queue positions i32[M], queue lengths i32[M],
// event count u32, groups of the events u8[slots].
__host__ __device__ inline size_t batch_state_bytes(int M, int T, int event_rows)
{
    return (8 * (size_t)T + 9 * (size_t)event_rows * kLanes + 8 * (size_t)M + 4 + 15) & ~(size_t)15;
}

struct StateView {
    double *clk;
    uint64_t *ev;
    int32_t *qpos, *qlen;
    uint32_t *ev_n;
    uint8_t *ev_g;
};

__device__ inline StateView state_view(const BatchArgs &a, unsigned char *p)
{
    StateView v;
    v.clk = reinterpret_cast<double *>(p);
    v.ev = reinterpret_cast<uint64_t *>(v.clk + a.T);
    v.qpos = reinterpret_cast<int32_t *>(v.ev + (size_t)a.event_rows * kLanes);
    v.qlen = v.qpos + a.M;
    v.ev_n = reinterpret_cast<uint32_t *>(v.qlen + a.M);
    v.ev_g = reinterpret_cast<uint8_t *>(v.ev_n + 1);
    return v;
}

// An integer that orders times as `<` does.
__device__ __forceinline__ uint64_t time_key(double t)
{
    const uint64_t bits = (uint64_t)__double_as_longlong(t);
    return bits ^ ((uint64_t)((int64_t)bits >> 63) | 0x8000000000000000ull);
}

// The lanes with the smallest key; 0 when no lane has one.
__device__ __forceinline__ uint32_t warp_least(uint64_t key)
{
    const uint32_t hi = (uint32_t)(key >> 32);
    const uint32_t least = __reduce_min_sync(0xFFFFFFFFu, hi);
    uint32_t who = __ballot_sync(0xFFFFFFFFu, hi == least);
    if (who & (who - 1)) {
        if (least == 0xFFFFFFFFu) return 0;
        const uint32_t lo = hi == least ? (uint32_t)key : 0xFFFFFFFFu;
        const uint32_t low = __reduce_min_sync(0xFFFFFFFFu, lo);
        who = __ballot_sync(0xFFFFFFFFu, hi == least && lo == low);
    }
    return least == 0xFFFFFFFFu ? 0u : who;
}

// ---- outputs -----------------------------------------------------------------------------
__device__ __forceinline__ void write_output(const BatchArgs &a, int64_t b, uint32_t r, double fin,
                                             uint32_t good)
{
    const size_t at = (size_t)b * a.N + r;
    a.finish[at] = fin;
    a.good[at] = (uint8_t)good;
}

// Writes (or lists, see ListWarp::direct) the outputs gathered on chip.  Returns how many are
// listed by now.  Everything by value: a ListWarp whose address is taken lives in memory.
__device__ __noinline__ uint32_t outputs_write(const BatchArgs &a, int64_t b, uint32_t out_fin,
                                               uint32_t out_pos, uint32_t out_n, int32_t own_begin,
                                               Carried *carry, uint32_t carry_n)
{
    const int lane = threadIdx.x & (kLanes - 1);
    __syncwarp();
    for (uint32_t base = 0; base < out_n; base += kLanes) {
        const uint32_t k = base + lane;
        const bool is = k < out_n;
        uint32_t r = 0, good = 0;
        double fin = 0.0;
        if (is) {
            const uint32_t at = SM_U32(out_pos + k);
            good = !(at & kDropped);
            r = (uint32_t)a.req[at & ~kDropped];
            fin = good ? SM_F64(out_fin + k) : a.pos_ts[at & ~kDropped];
        }
        const bool own = is && (int32_t)r >= own_begin;
        if (own) write_output(a, b, r, fin, good);
        const uint32_t listed = __ballot_sync(0xFFFFFFFFu, is && !own);
        if (listed && carry_n != kNoCarry) {
            const uint32_t at = carry_n + __popc(listed & ((1u << lane) - 1u));
            if (is && !own && at < (uint32_t)kMaxCarry) carry[at] = Carried{fin, r, good};
            carry_n += __popc(listed);
            if (carry_n > (uint32_t)kMaxCarry) carry_n = kNoCarry;
        }
    }
    __syncwarp();
    return carry_n;
}

template <class W>
__device__ __forceinline__ void outputs_flush(const BatchArgs &a, W &w)
{
    w.carry_n = outputs_write(a, w.b, w.ring_fin(a), w.ring_pos(a), w.out_n, w.direct ? 0 : w.own_begin,
                              w.carry, w.carry_n);
    w.out_n = 0;
}

// Outputs of the `n` (at most 32) requests from position `pos` on; dropped: 0 or kDropped.
template <class W>
__device__ __forceinline__ void outputs_add(const BatchArgs &a, W &w, int32_t n, int32_t pos,
                                            double fin, uint32_t dropped)
{
    if (!w.record) return;
    const int lane = threadIdx.x & (kLanes - 1);
    if (lane < n) {
        const uint32_t k = w.out_n + lane;
        SM_F64(w.ring_fin(a) + k) = fin;
        SM_U32(w.ring_pos(a) + k) = (uint32_t)(pos + lane) | dropped;
    }
    w.out_n += n;
    if (w.out_n >= (uint32_t)kLanes) outputs_flush(a, w);
}

}  // namespace mms

#include "batch_lists.cuh"
#include "batch_groups.cuh"

namespace mms {

// The latency table on chip, as doubles.
template <class W>
__device__ inline void batch_stage(const BatchArgs &a)
{
    if constexpr (W::kDoubles) {
        const int real = a.M * a.C * a.S * a.NB;
        for (int i = threadIdx.x; i < a.table_elems; i += blockDim.x)
            SM_F64(i) = i < real ? (double)__ldg(a.latency + i) : 0.0;
        __syncthreads();
    } else {
        batch_stage_table(a);
    }
}

// ---- chunks -----------------------------------------------------------------------------------
__device__ inline bool batch_can_chunk(const BatchArgs &a) { return a.K > 1 && *a.odd == 0; }

// First arrival of segment q (q == NS: one past the last arrival).
__device__ inline int64_t segment_begin(const BatchArgs &a, int32_t q)
{
    return q >= a.NS ? a.N : (int64_t)q * a.seg_len;
}

// First arrival of chunk j.
__device__ inline int64_t chunk_begin(const BatchArgs &a, int32_t j)
{
    return segment_begin(a, j * a.seg_per_chunk < a.NS ? j * a.seg_per_chunk : a.NS);
}

// Simulates arrivals [begin, end of the run): the run-in up to `first` (nothing recorded), then
// the segments [q, q1), after each of which the state is saved (`snapshots`).  A walk
// replaces a stored run and ends where its state meets the stored one, with kMeetOther under other
// labels as well (they are then the warp's).  Returns the first segment that was not simulated.
enum BatchMeet { kMeetNever, kMeetSame, kMeetOther };
template <class W>
__device__ inline int32_t batch_run(const BatchArgs &a, W &w, int64_t begin, int64_t first,
                                    int32_t q, int32_t q1, bool snapshots, BatchMeet meet,
                                    unsigned char *start = nullptr)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const int64_t end = segment_begin(a, q1);
    BatchOrder *orders = w.window(a);
    // the window behind the one at work
    double ts = 0.0; float slo = 0.0f; int32_t m = -1, pos = 0;
    const auto fetch = [&](int64_t base) {
        const int64_t i = base + lane < a.N ? base + lane : a.N - 1;
        ts = __ldg(a.arrivals + i);
        slo = __ldg(a.slos + i);
        m = __ldg(a.model_ids + i);
        pos = a.pos[i];
    };
    if (begin < end) fetch(begin);
    int64_t i = begin, window_end = begin;
    w.record = begin >= first;
    w.seg = q;
    int64_t stop = w.record ? segment_begin(a, q + 1) : first;
    uint32_t listed = 0;                       // carried requests up to the segment's begin
    for (;;) {
        while (i < stop) {
            if (i == window_end) {
                BatchOrder o;
                o.ts = ts;
                o.dl = ts + (double)slo;
                if (m >= a.M) { w.status |= MMS_STATUS_BAD_INDEX; m = -1; }
                o.pos = pos;
                o.m = m;
                o.served = m < 0 ? 0ull : replicas_of(a, w, m);
                // :748-757 unknown model or no replica
                const int64_t at = i + lane;
                if (!o.served && at >= first && at < end) write_output(a, w.b, (uint32_t)at, ts, 0u);
                __syncwarp();
                orders[lane] = o;
                __syncwarp();
                window_end = i + kLanes;
                fetch(window_end);
            }
            const int64_t to = stop < window_end ? stop : window_end;
            const int k = (int)(i - (window_end - kLanes));
            batch_arrivals(a, w, k, k + (int)(to - i));
            i = to;
        }
        if (!w.record) {
            w.record = true;
            w.status &= MMS_STATUS_BAD_INDEX;            // overflows of the run-in are not the chunk's
            w.tie = 0;
            counts_store(a, w, nullptr);
            if (snapshots) state_save(a, w, start);
            stop = segment_begin(a, q + 1);
            continue;
        }
        if (i == a.N) batch_drain(a, w);
        outputs_flush(a, w);
        counts_store(a, w, a.seg_counts + ((size_t)q * a.B + w.b) * 2 * a.G);
        if (snapshots) {
            const size_t cell = (size_t)q * a.B + w.b;
            unsigned char *p = a.seg_end + cell * a.state_bytes;
            bool same = false;
            if (meet != kMeetNever && q + 1 < q1) {
                const double tau = __ldg(a.arrivals + i);
                same = batch_equivalent(a, w, p, tau);
                if constexpr (W::kOrderly)
                    if (!same && meet == kMeetOther) {
                        int to[W::kGroups];
                        same = other_labels(a, w, p, tau, to);
                        if (same) labels_set(a, w, to);
                    }
            }
            if constexpr (W::kOrderly) {
                if (lane == 0) a.tie[cell] = w.tie;
                w.tie = 0;
            }
            // (the entries of a list that overflowed are never used)
            const uint32_t now = w.carry_n == kNoCarry ? listed : w.carry_n;
            if (lane == 0) a.carry_seg[cell] = (uint8_t)(now - listed);
            listed = now;
            if (same) return q + 1;
            state_save(a, w, p);
        }
        if (++q >= q1) return q;
        w.seg = q;
        stop = segment_begin(a, q + 1);
    }
}


// The speculative pass: one warp per (chunk, candidate).  Chunk 0 starts from the true
// (idle) state; the others start idle `warmup` arrivals early and store the state they
// have at their first arrival.
template <class W>
__global__ void __launch_bounds__(kBatchWarps * kLanes, kBatchBlocksPerSm)
batch_stream_kernel(const __grid_constant__ BatchArgs a)
{
    if (W::kOrderly ? *a.odd != 0 : a.only_odd && *a.odd == 0) return;
    batch_stage<W>(a);
    const int lane = threadIdx.x & (kLanes - 1);
    const bool chunked = batch_can_chunk(a);
    const int64_t items = (int64_t)a.B * (chunked ? a.K : 1);
    const int64_t step = (int64_t)gridDim.x * (blockDim.x / kLanes);
    for (int64_t it = (int64_t)blockIdx.x * (blockDim.x / kLanes) + threadIdx.x / kLanes; it < items; it += step) {
        const int32_t j = (int32_t)(it / a.B);
        const int64_t b = it % a.B;
        W w;
        batch_setup(a, w, b);
        if (w.bad) {
            if (j == 0 && lane == 0) atomicOr(&a.status[b], MMS_STATUS_BAD_INDEX);
            continue;
        }
        batch_zero_state(a, w);
        const size_t cell = (size_t)j * a.B + b;
        const int32_t q = j * a.seg_per_chunk;
        const int32_t q1 = chunked && q + a.seg_per_chunk < a.NS ? q + a.seg_per_chunk : a.NS;
        const int64_t first = chunk_begin(a, j);
        if (j > 0) {
            w.direct = false;
            w.own_begin = (int32_t)first;
            w.carry = a.carry + cell * kMaxCarry;
        }
        if constexpr (W::kOrderly)
            if (chunked) w.swaps = a.swaps + cell * kSwapCap;
        batch_run(a, w, j > 0 && first > a.warmup ? first - a.warmup : 0, first, q, q1, chunked, kMeetNever,
                  a.chunk_start + cell * a.state_bytes);
        const uint32_t status = __reduce_or_sync(0xFFFFFFFFu, w.status);
        if (lane == 0) {
            if (chunked) {
                a.carry_n[cell] = w.carry_n;
                a.run_status[cell] = status;
                if constexpr (W::kOrderly) a.swap_n[cell] = w.swap_n;
            } else if (status) {
                atomicOr(&a.status[b], status);
            }
        }
    }
}

// One warp per boundary whose sides the round before changed (all in round 0): does the state
// the chunk's stored run started from continue the state the run of the chunk before it ended
// in?  If not, that end state becomes the chunk's start state and the chunk goes on the
// round's work list.  The end state may itself be wrong still (its chunk is on the list too);
// then the next round, or the chain kernel, catches what follows from it.  A last pass
// (round == rounds) only judges, for the chain kernel.
template <class W>
__global__ void __launch_bounds__(kBatchWarps * kLanes)
batch_validate_kernel(const __grid_constant__ BatchArgs a)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const int64_t t = (int64_t)blockIdx.x * (blockDim.x / kLanes) + threadIdx.x / kLanes;
    if (!batch_can_chunk(a) || t >= (int64_t)a.B * (a.K - 1)) return;
    if (a.round > 0 && a.work_count[a.round - 1] == 0) return;      // nothing changed since
    const int32_t j = (int32_t)(t / a.B) + 1;
    const int64_t b = t % a.B;
    const size_t cell = (size_t)j * a.B + b;
    if (a.round > 0 && a.stamp[cell] != (uint8_t)a.round && a.stamp[cell - a.B] != (uint8_t)a.round) return;
    W w;
    batch_setup(a, w, b);
    if (w.bad) return;
    unsigned char *start = a.chunk_start + cell * a.state_bytes;
    state_load(a, w, a.seg_end + ((size_t)(j * a.seg_per_chunk - 1) * a.B + b) * a.state_bytes);
    const double tau = a.arrivals[chunk_begin(a, j)];
    uint8_t how = batch_equivalent(a, w, start, tau) ? kLinkSame : 0;
    if constexpr (W::kOrderly) {
        int to[W::kGroups];
        if (!how && other_labels(a, w, start, tau, to)) {
            how = kLinkOther;
#pragma unroll
            for (int h = 0; h < W::kGroups; ++h) a.perm[cell * kGroupLimit + lane + h * kLanes] = (uint8_t)to[h];
        }
    }
    if (lane == 0) a.link[cell] = how;
    if (how || a.round == a.rounds) return;
    state_save(a, w, start);
    if (lane == 0) {
        a.stamp[cell] = (uint8_t)(a.round + 1);
        a.work_items[atomicAdd(&a.work_count[a.round], 1u)] = (uint32_t)cell;
        if (a.resimulated) atomicAdd(&a.resimulated[b], 1);
    }
}

// How many outputs the stored run of a chunk listed in segments [q, q1).
__device__ inline uint32_t carried_from(const BatchArgs &a, int64_t b, int32_t q, int32_t q1)
{
    uint32_t n = 0;
    for (int32_t s = q + (int32_t)(threadIdx.x & (kLanes - 1)); s < q1; s += kLanes)
        n += a.carry_seg[(size_t)s * a.B + b];
    return __reduce_add_sync(0xFFFFFFFFu, n);
}

// What a swap had set apart, back to its segment's counters.
__device__ inline void counts_give_back(const BatchArgs &a, int64_t b, const Swap &s)
{
    if ((threadIdx.x & (kLanes - 1)) == 0) {
        uint32_t *counts = a.seg_counts + ((size_t)s.seg * a.B + b) * 2 * a.G;
        int k = 0;
        for (uint64_t rest = s.groups; rest; rest &= rest - 1, ++k) {
            const int g = (int)__ffsll((long long)rest) - 1;
            counts[g] += s.requests[k];
            counts[a.G + g] += s.good[k];
        }
    }
    __syncwarp();
}

// The listed chunks, one to a warp, taken from the list as warps become free: simulated again
// from the start state batch_validate_kernel stored.  That state is not known to be the true
// one yet, so the outputs of carried requests are listed, not written, like in a speculative run.
template <class W>
__global__ void __launch_bounds__(kBatchWarps * kLanes, kBatchBlocksPerSm)
batch_walk_kernel(const __grid_constant__ BatchArgs a)
{
    if (!batch_can_chunk(a)) return;
    const uint32_t count = a.work_count[a.round];
    if ((uint64_t)blockIdx.x * (blockDim.x / kLanes) >= count) return;
    batch_stage<W>(a);
    const int lane = threadIdx.x & (kLanes - 1);
    Carried *list = a.walk_carry + ((size_t)blockIdx.x * (blockDim.x / kLanes) + threadIdx.x / kLanes) * kMaxCarry;
    for (;;) {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&a.work_next[a.round], 1u);
        at = __shfl_sync(0xFFFFFFFFu, at, 0);
        if (at >= count) return;
        const size_t cell = a.work_items[at];
        const int32_t j = (int32_t)(cell / (uint32_t)a.B);
        const int64_t b = (int64_t)(cell % (uint32_t)a.B);
        W w;
        batch_setup(a, w, b);
        const int64_t first = chunk_begin(a, j);
        const int32_t q0 = j * a.seg_per_chunk;
        const int32_t q1 = q0 + a.seg_per_chunk < a.NS ? q0 + a.seg_per_chunk : a.NS;
        w.direct = false;
        w.own_begin = (int32_t)first;
        w.carry = list;
        Swap *swaps = nullptr;
        if constexpr (W::kOrderly)
            w.swaps = swaps = a.walk_swaps + (list - a.walk_carry) / kMaxCarry * kSwapCap;
        state_load(a, w, a.chunk_start + cell * a.state_bytes);
        const uint32_t stored = a.carry_n[cell];
        // (a run that overflowed something is replaced as a whole)
        const int32_t q = batch_run(a, w, first, first, q0, q1, true,
                                    stored != kNoCarry && a.run_status[cell] == 0 ? kMeetSame : kMeetNever);
        const uint32_t status = __reduce_or_sync(0xFFFFFFFFu, w.status);
        uint32_t n = w.carry_n;
        Carried *kept = a.carry + cell * kMaxCarry;
        __syncwarp();
        if (q < q1 && n != kNoCarry) {       // the stored run takes over: its outputs from there on
            const uint32_t more = carried_from(a, b, q, q1);
            if (n + more > (uint32_t)kMaxCarry) {
                n = kNoCarry;
            } else {
                for (uint32_t k = lane; k < more; k += kLanes) list[n + k] = kept[stored - more + k];
                n += more;
            }
        }
        __syncwarp();
        if (n != kNoCarry)
            for (uint32_t k = lane; k < n; k += kLanes) kept[k] = list[k];
        if constexpr (W::kOrderly) {
            // the same for the swaps; those that find no place are ties
            Swap *old = a.swaps + cell * kSwapCap;
            uint32_t count = w.swap_n;
            if (q < q1) {
                const uint32_t had = a.swap_n[cell];
                for (uint32_t k = 0; k < had; ++k) {
                    if (old[k].seg < q) continue;
                    if (count < (uint32_t)kSwapCap) {
                        if (lane == 0) swaps[count] = old[k];
                        ++count;
                    } else {               // counted for its labels
                        if (lane == 0) a.tie[(size_t)old[k].seg * a.B + b] |= old[k].groups;
                        counts_give_back(a, b, old[k]);
                    }
                }
            }
            __syncwarp();
            for (uint32_t k = lane; k < count; k += kLanes) old[k] = swaps[k];
            if (lane == 0) a.swap_n[cell] = count;
        }
        if (lane == 0) {
            a.carry_n[cell] = n;
            a.run_status[cell] = status;
        }
        __syncwarp();
    }
}

// Writes entries [from, to) of a chunk's list of carried requests.
__device__ inline void apply_carried(const BatchArgs &a, int64_t b, size_t cell, uint32_t from, uint32_t to)
{
    const Carried *list = a.carry + cell * kMaxCarry;
    for (uint32_t k = from + (threadIdx.x & (kLanes - 1)); k < to; k += kLanes)
        write_output(a, b, list[k].req, list[k].fin, list[k].good);
    __syncwarp();
}

// Translates the counters of segment q of chunk j and follows the labels through its swaps; `k`: the
// first swap of the chunk that is not behind it.
template <int kPer>
__device__ inline void name_counts(const BatchArgs &a, const GroupWarp<kPer> &w, int32_t j, int32_t q, uint32_t &k)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const size_t cell = (size_t)j * a.B + w.b;
    const Swap *list = a.swaps + cell * kSwapCap;
    const uint32_t count = a.swap_n[cell];
    uint32_t *counts = a.seg_counts + ((size_t)q * a.B + w.b) * 2 * a.G;
    uint32_t n[2 * kPer], add[2 * kPer];               // of LABELS and of GROUPS lane and lane + 32
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const int g = lane + h * kLanes;
        n[2 * h] = g < a.G ? counts[g] : 0u;
        n[2 * h + 1] = g < a.G ? counts[a.G + g] : 0u;
        add[2 * h] = add[2 * h + 1] = 0;
    }
    __syncwarp();
    while (k < count && list[k].seg < q) ++k;
    // what was counted before a swap belongs to the labels before it
    for (; k < count && list[k].seg == q; ++k) {
        const Swap s = list[k];
        int at = 0;
        uint32_t least = 0xFFFFFFFFu;                  // group << 8 | label
        for (uint64_t rest = s.groups; rest; rest &= rest - 1, ++at) {
            const uint32_t label = (uint32_t)__ffsll((long long)rest) - 1u, g = smem[AT1(labels) + label];
            least = min(least, (g << 8) | label);
#pragma unroll
            for (int h = 0; h < kPer; ++h)
                if ((uint32_t)(lane + h * kLanes) == g) {
                    add[2 * h] += s.requests[at];
                    add[2 * h + 1] += s.good[at];
                }
        }
        __syncwarp();
        if (lane == 0) {                               // the picked label stands for the smallest group
            smem[AT1(labels) + (least & 0xFFu)] = smem[AT1(labels) + s.picked];
            smem[AT1(labels) + s.picked] = (uint8_t)(least >> 8);
        }
        __syncwarp();
    }
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const int label = lane + h * kLanes;
        if (label < a.G) {
            const uint32_t g = smem[AT1(labels) + label];
            counts[g] = n[2 * h];
            counts[a.G + g] = n[2 * h + 1];
        }
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const int g = lane + h * kLanes;
        if (g < a.G) {
            counts[g] += add[2 * h];
            counts[a.G + g] += add[2 * h + 1];
        }
    }
    __syncwarp();
}

// One warp per candidate: goes through the chunks in order.  A chunk whose start state is
// equivalent to the true state, under the same or other labels, is kept (and the outputs of the
// requests it carried over are written), any other is simulated again from the true state, as
// far as it differs.
template <class W>
__global__ void __launch_bounds__(kBatchWarps * kLanes, kBatchBlocksPerSm)
batch_chain_kernel(const __grid_constant__ BatchArgs a)
{
    if (!batch_can_chunk(a)) return;
    const int lane = threadIdx.x & (kLanes - 1);
    const int64_t b = (int64_t)blockIdx.x * (blockDim.x / kLanes) + threadIdx.x / kLanes;
    const size_t B = (size_t)a.B;
    const bool mine = b < a.B && a.status[b] == 0;           // else: bad tables
    bool open = false, other = false;
    if (mine)
        for (int32_t j = 1 + lane; j < a.K; j += kLanes) {
            const uint8_t link = a.link[(size_t)j * B + b];
            open |= !link || a.carry_n[(size_t)j * B + b] == kNoCarry;
            other |= link == kLinkOther;
        }
    // (labels may turn out not to be usable)
    if (__syncthreads_or(open || other)) batch_stage<W>(a);
    if (!mine) return;
    W w;
    if (__any_sync(0xFFFFFFFFu, open || other)) batch_setup(a, w, b);
    // Chunk 0 ran from the true state.  While stored runs continue one another (judged by
    // batch_validate_kernel) their states need not come on chip.
    bool live = false;                     // the true state before chunk j is on chip; else the stored
    uint64_t moved = 0;                    //   run before it counts, under labels that move these groups
    uint32_t status = a.run_status[b];
    int32_t redone = 0;
    for (int32_t j = 1; j < a.K; ++j) {
        if (!live) {
            // up to 32 chunks in which nothing happens but outputs to be written
            const int32_t s = j + lane;
            const bool in = s < a.K;
            const uint32_t many = in ? a.carry_n[(size_t)s * B + b] : 0u;
            const uint32_t stops = __ballot_sync(0xFFFFFFFFu, in && (moved || many == kNoCarry ||
                                                                     a.link[(size_t)s * B + b] != kLinkSame));
            const int32_t quiet = stops ? __ffs((int)stops) - 1 : a.K - j < kLanes ? a.K - j : kLanes;
            if (lane < quiet) status |= a.run_status[(size_t)s * B + b];
            for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, lane < quiet && many > 0); todo; todo &= todo - 1) {
                const int k = __ffs((int)todo) - 1;
                apply_carried(a, b, (size_t)(j + k) * B + b, 0, __shfl_sync(0xFFFFFFFFu, many, k));
            }
            if (quiet) { j += quiet - 1; continue; }
        }
        const size_t cell = (size_t)j * B + b;
        const uint32_t n = a.carry_n[cell], was = a.run_status[cell];
        const int32_t q0 = j * a.seg_per_chunk;
        const int32_t q1 = q0 + a.seg_per_chunk < a.NS ? q0 + a.seg_per_chunk : a.NS;
        // does the stored run of chunk j count?
        bool valid;
        if (live) {
            unsigned char *start = a.chunk_start + cell * a.state_bytes;
            const double tau = a.arrivals[chunk_begin(a, j)];
            valid = n != kNoCarry && batch_equivalent(a, w, start, tau);
            if constexpr (W::kOrderly) {
                int to[W::kGroups];
                if (!valid && n != kNoCarry && other_labels(a, w, start, tau, to)) {
                    valid = true;
                    labels_set(a, w, to);
                    moved = labels_moved(a, w);
                }
            }
        } else {
            const uint8_t link = a.link[cell];
            valid = link && n != kNoCarry;
            if (!valid) {
                state_load(a, w, a.seg_end + ((size_t)(q0 - 1) * B + b) * a.state_bytes);
                labels_reset(a, w);
                moved = 0;
            } else if constexpr (W::kOrderly) {
                if (link == kLinkOther) labels_through(a, w, a.perm + cell * kGroupLimit);
                moved = labels_moved(a, w);
            }
        }
        uint32_t swap = 0;                 // of the chunk's swaps, see name_counts
        bool touched = false;
        for (int32_t q = q0; q < q1;) {
            if (valid) {
                const uint32_t from = n - carried_from(a, b, q, q1);
                status |= was;
                if (!moved) {              // the rest of the chunk as it is
                    apply_carried(a, b, cell, from, n);
                    if constexpr (W::kOrderly)
                        for (uint32_t k = touched ? 0u : 0xFFFFFFFFu; k < a.swap_n[cell]; ++k)
                            if (a.swaps[cell * kSwapCap + k].seg >= q) counts_give_back(a, b, a.swaps[cell * kSwapCap + k]);
                    break;
                }
                touched = true;
                if constexpr (W::kOrderly) {
                    if (!(moved_class(a, w, moved) & a.tie[(size_t)q * B + b])) {
                        apply_carried(a, b, cell, from, n - carried_from(a, b, q + 1, q1));
                        name_counts(a, w, j, q, swap);
                        moved = labels_moved(a, w);
                        ++q;
                        continue;
                    }
                }
                // a group number decided about a group that is another one: from the true state
                // (in front of the chunk the state its run started from, which is under the run's labels)
                state_load(a, w, q == q0 ? a.chunk_start + cell * a.state_bytes
                                         : a.seg_end + ((size_t)(q - 1) * B + b) * a.state_bytes);
                labels_reset(a, w);
                moved = 0;
                valid = false;
            }
            touched = true;
            ++redone;
            w.status = 0;
            const int64_t at = segment_begin(a, q);
            q = batch_run(a, w, at, at, q, q1, true, n != kNoCarry && was == 0 ? kMeetOther : kMeetNever);
            status |= w.status;
            valid = q < q1;
            if constexpr (W::kOrderly) moved = valid ? labels_moved(a, w) : 0;
        }
        if constexpr (W::kOrderly)
            if (touched && lane == 0) a.swap_n[cell] = 0;
        __syncwarp();
        live = !valid;
    }
    status = __reduce_or_sync(0xFFFFFFFFu, status);
    if (lane == 0) {
        if (a.resimulated && redone) atomicAdd(&a.resimulated[b], redone);
        if (status) atomicOr(&a.status[b], status);
    }
}

// In one launch: the trace sorted by model (the first M blocks, one per model: its warps
// take a stretch of the trace each, count the model's requests and those of smaller models in it,
// then go through it again and place them), and, by the blocks behind them, what a call clears
// and the positions where the arrival times are not finite or go backwards and the latencies that
// are not >= 0 (batch_equivalent needs clocks that an accepted request leaves at or behind its
// arrival, see kIrregularLatency), added to *odd (zero on entry).
struct BatchClear {
    int32_t *odd;
    int32_t *model_num_good;
};
constexpr int kOrderWarps = 16;

__global__ void __launch_bounds__(kOrderWarps * kLanes)
batch_order_kernel(const BatchArgs a, const BatchClear c)
{
    const int lane = threadIdx.x & (kLanes - 1), warp = threadIdx.x / kLanes;
    if ((int)blockIdx.x >= a.M) {
        const int64_t nth = (int64_t)(gridDim.x - a.M) * blockDim.x;
        const int64_t tid = (int64_t)(blockIdx.x - a.M) * blockDim.x + threadIdx.x;
        for (int64_t i = tid; i < (int64_t)a.B * a.M; i += nth) c.model_num_good[i] = 0;
        for (int64_t i = tid; i < a.B; i += nth) {
            a.status[i] = 0;
            if (a.resimulated) a.resimulated[i] = 0;
        }
        if (a.K > 1) {
            for (int64_t i = tid; i < (int64_t)a.K * a.B; i += nth) a.stamp[i] = 0;
            for (int64_t i = tid; i < 2 * (a.rounds + 1); i += nth) a.work_count[i] = 0;
        }
        int32_t bad = 0;
        for (int64_t i = tid; i < a.N; i += nth) {
            const double t = a.arrivals[i];
            if (!(t - t == 0.0) || __double2hiint(t) < 0 || (i > 0 && !(a.arrivals[i - 1] <= t))) ++bad;
        }
        const int64_t entries = (int64_t)a.M * a.C * a.S * a.NB;
        for (int64_t i = tid; i < (a.latency_stride ? a.B * entries : entries); i += nth)
            bad += !(a.latency[i / entries * a.latency_stride + i % entries] >= 0.0f);
        if (bad) atomicAdd(c.odd, bad);
        return;
    }
    __shared__ int32_t equal[kOrderWarps], less[kOrderWarps];
    constexpr int kAhead = 8;                      // loads in flight
    const int m = blockIdx.x;
    const int64_t tiles = (a.N + kLanes - 1) / kLanes;
    const int64_t t0 = tiles * warp / kOrderWarps, t1 = tiles * (warp + 1) / kOrderWarps;
    int32_t n_equal = 0, n_less = 0;
    for (int64_t t = t0; t < t1; t += kAhead) {
        int32_t id[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int64_t i = (t + u) * kLanes + lane;
            id[u] = t + u < t1 && i < a.N ? a.model_ids[i] : -1;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            n_equal += id[u] == m;
            n_less += id[u] >= 0 && id[u] < m;
        }
    }
    n_equal = (int32_t)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)n_equal);
    n_less = (int32_t)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)n_less);
    if (lane == 0) { equal[warp] = n_equal; less[warp] = n_less; }
    __syncthreads();
    int32_t at = 0, total = 0;
    for (int w = 0; w < kOrderWarps; ++w) {
        at += less[w] + (w < warp ? equal[w] : 0);
        total += less[w] + equal[w];
    }
    if (threadIdx.x == 0) {
        a.first_of[m] = at;                        // (warp 0: nothing of the model is before it)
        if (m == a.M - 1) a.first_of[a.M] = total;
    }
    for (int64_t t = t0; t < t1; t += kAhead) {
        int32_t id[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int64_t i = (t + u) * kLanes + lane;
            id[u] = t + u < t1 && i < a.N ? a.model_ids[i] : -1;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const uint32_t has = __ballot_sync(0xFFFFFFFFu, id[u] == m);
            if (id[u] == m) {
                const int64_t i = (t + u) * kLanes + lane;
                const int32_t k = at + __popc(has & ((1u << lane) - 1u));
                const double ts = a.arrivals[i];
                a.pos[i] = k;
                a.req[k] = (int32_t)i;
                a.pos_ts[k] = ts;
                a.pos_dl[k] = ts + (double)a.slos[i];
            }
            at += __popc(has);
        }
    }
}

// Counts the good requests of each model and, of finish - arrival, makes the leaf sums of numpy's
// pairwise order.  A block takes the requests of kTallyLeaves leaves of one candidate; request k of
// a leaf goes to partial sum k mod 8, eight lanes to a leaf.
__global__ void __launch_bounds__(kTallyThreads)
batch_tally_kernel(const BatchArgs a, int32_t num_leaves, const int32_t *leaf_start,
                   int32_t *model_num_good, double *leaf_sums)
{
    extern __shared__ uint32_t tally[];            // [M]
    const int32_t slices = (num_leaves + kTallyLeaves - 1) / kTallyLeaves;
    const int64_t b = blockIdx.x / slices;
    const int32_t l0 = (int32_t)(blockIdx.x % slices) * kTallyLeaves;
    const int32_t l1 = l0 + kTallyLeaves < num_leaves ? l0 + kTallyLeaves : num_leaves;
    for (int c = threadIdx.x; c < a.M; c += blockDim.x) tally[c] = 0;
    __syncthreads();
    const size_t row = (size_t)b * a.N;
    const int64_t i1 = leaf_start[l1];
    for (int64_t i = leaf_start[l0] + threadIdx.x; i < i1; i += blockDim.x)
        // (a run that failed leaves requests without an outcome: what stands there may be anything)
        if (a.good[row + i] == 1) {
            const uint32_t m = (uint32_t)a.model_ids[i];
            if (m < (uint32_t)a.M) atomicAdd(&tally[m], 1u);
        }
    __syncthreads();
    for (int c = threadIdx.x; c < a.M; c += blockDim.x)
        if (tally[c]) atomicAdd(model_num_good + (size_t)b * a.M + c, (int32_t)tally[c]);
    const int32_t leaf = l0 + (int32_t)threadIdx.x / 8;
    const int part = threadIdx.x & 7;
    const bool is = leaf < l1;
    const int64_t s = is ? leaf_start[leaf] : 0, e = is ? leaf_start[leaf + 1] : 0;
    const int64_t body = s + ((e - s) & ~(int64_t)7);
    const double *f = a.finish + row;
    double p = 0.0;
    for (int64_t i = s + part; i < body; i += 8) p += f[i] - a.arrivals[i];
    p = p + __shfl_xor_sync(0xFFFFFFFFu, p, 1);
    p = p + __shfl_xor_sync(0xFFFFFFFFu, p, 2);
    p = p + __shfl_xor_sync(0xFFFFFFFFu, p, 4);
    if (is && part == 0) {
        for (int64_t i = body; i < e; ++i) p += f[i] - a.arrivals[i];
        leaf_sums[(size_t)leaf * a.B + b] = p;
    }
}

// The groups' counters: a warp per candidate and 32 of its counters adds those of the segments and
// of the swaps that are left.
__global__ void __launch_bounds__(4 * kLanes)
batch_count_kernel(const BatchArgs a, int32_t *group_num_requests, int32_t *group_num_good)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const int32_t parts = (2 * a.G + kLanes - 1) / kLanes;
    const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
    const int64_t b = t / parts;
    if (b >= a.B) return;
    const int c = (int)(t % parts) * kLanes + lane;
    const bool is = c < 2 * a.G;
    int32_t n = 0;
    if (a.status[b] & MMS_STATUS_BAD_INDEX) {          // nothing was simulated, perhaps
        if (is) (c < a.G ? group_num_requests : group_num_good)[(size_t)b * a.G + (c < a.G ? c : c - a.G)] = 0;
        return;
    }
    constexpr int kAhead = 8;
    for (int32_t q = 0; q < a.NS; q += kAhead)
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            n += is && q + u < a.NS ? a.seg_counts[((size_t)(q + u) * a.B + b) * 2 * a.G + c] : 0u;
    if (a.swap_n && batch_can_chunk(a))
        for (int32_t j = 0; j < a.K; ++j) {
            const size_t cell = (size_t)j * a.B + b;
            const uint32_t count = a.swap_n[cell];
            for (uint32_t k = 0; k < count; ++k) {
                const Swap *s = a.swaps + cell * kSwapCap + k;
                const uint64_t groups = s->groups;
                const int g = c < a.G ? c : c - a.G;
                if (!is || !((groups >> g) & 1u)) continue;
                const int at = __popcll(groups & ((1ull << g) - 1u));
                n += c < a.G ? s->requests[at] : s->good[at];
            }
        }
    if (is) (c < a.G ? group_num_requests : group_num_good)[(size_t)b * a.G + (c < a.G ? c : c - a.G)] = n;
}

// next_same[i] = next request with request i's model, -1 if none.  One block per model; its
// warps take a stretch of the trace each, look for the first request of the model in it (what
// the stretch before it ends with), then go through the stretch backwards, 32 requests to a
// vote.  (One thread per model walking the whole trace: 1.2 ms for 27 000 requests.)
constexpr int kNextWarps = 16;

__global__ void __launch_bounds__(kNextWarps * kLanes)
next_same_kernel(const int32_t *model_ids, int64_t N, int32_t *next_same)
{
    __shared__ int32_t first[kNextWarps];
    constexpr int kAhead = 8;                      // loads in flight
    const int m = blockIdx.x, lane = threadIdx.x & (kLanes - 1), warp = threadIdx.x / kLanes;
    const int64_t tiles = (N + kLanes - 1) / kLanes;
    const int64_t t0 = tiles * warp / kNextWarps, t1 = tiles * (warp + 1) / kNextWarps;
    int32_t found = 0x7FFFFFFF;
    for (int64_t t = t0; t < t1; t += kAhead) {
        int32_t id[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int64_t i = (t + u) * kLanes + lane;
            id[u] = t + u < t1 && i < N ? model_ids[i] : -1;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const uint32_t has = __ballot_sync(0xFFFFFFFFu, id[u] == m);
            if (has && found == 0x7FFFFFFF) found = (int32_t)((t + u) * kLanes) + __ffs((int)has) - 1;
        }
        if (found != 0x7FFFFFFF) break;
    }
    if (lane == 0) first[warp] = found;
    __syncthreads();
    int32_t carry = 0x7FFFFFFF;
    for (int w = warp + 1; w < kNextWarps; ++w) carry = first[w] < carry ? first[w] : carry;
    if (carry == 0x7FFFFFFF) carry = -1;
    for (int64_t t = t1; t > t0; t -= kAhead) {    // tiles t - 1, t - 2, ...
        int32_t id[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int64_t i = (t - 1 - u) * kLanes + lane;
            id[u] = t - 1 - u >= t0 && i < N ? model_ids[i] : -1;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const uint32_t has = __ballot_sync(0xFFFFFFFFu, id[u] == m);
            const int32_t base = (int32_t)((t - 1 - u) * kLanes);
            const uint32_t later = has & ~((2u << lane) - 1u);
            if (id[u] == m) next_same[base + lane] = later ? base + __ffs((int)later) - 1 : carry;
            if (has) carry = base + __ffs((int)has) - 1;
        }
    }
}

}  // namespace mms
