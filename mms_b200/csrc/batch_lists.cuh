// batch_lists.cuh — the batching simulator on lists of any length (see sim_batching.cuh).
//
// For what has no group and no model to a lane: more than 64 of either, a latency table that does
// not fit on chip, and traces and tables with oddities (arrival times out of order, negative or
// not finite, latencies that are not >= 0), which are simulated in one piece.  Times are mapped to integers
// that keep their order, and compared by 32 lanes at a time, the high word first, the low word only on a tie.
// About 550 instructions an arrival, which is what it costs.
#pragma once
#include "sim_core.cuh"

namespace mms {

struct BatchSmem {
    size_t warp0, warp_bytes, clocks, head_ts, head_dl, events, out_fin, orders, out_pos, counts,
        qpos, qlen, mrep, mlist, gcfg, glist, gmod, event_g, total;
};

// Shared memory of a block of `warps` warps: the latency table, then per warp the state and
// (not lean) the candidate's tables.  Lean: tables and the queue heads' times are read
// from global memory, for shapes that would not fit otherwise.
__host__ __device__ inline BatchSmem batch_smem(int M, int G, int P, int T, int event_rows,
                                                int table_elems, bool lean, int warps)
{
    BatchSmem L;
    L.warp0 = (sizeof(float) * (size_t)table_elems + 15) & ~(size_t)15;
    const size_t slots = (size_t)event_rows * kLanes, full = lean ? 0 : 1;
    size_t off = 0;
    L.orders = off;   off += sizeof(BatchOrder) * kLanes;
    L.clocks = off;   off += 8 * (size_t)T;
    L.head_ts = off;  off += 8 * full * M;
    L.head_dl = off;  off += 8 * full * M;
    L.events = off;   off += 8 * slots;
    L.out_fin = off;  off += 8 * (size_t)kOutRing;
    L.out_pos = off;  off += 4 * (size_t)kOutRing;
    L.counts = off;   off += 8 * (size_t)G;
    L.qpos = off;     off += 4 * (size_t)M;
    L.qlen = off;     off += 4 * (size_t)M;
    L.mrep = off;     off += 4 * full * P;
    L.mlist = off;    off += 4 * full * M;
    L.gcfg = off;     off += 4 * full * G;
    L.glist = off;    off += 4 * full * G;
    L.gmod = off;     off += 2 * full * P;
    L.event_g = off;  off += slots;
    L.warp_bytes = (off + 15) & ~(size_t)15;
    L.total = L.warp0 + (size_t)warps * L.warp_bytes;
    return L;
}

// A warp's view of its candidate, tables as lists; uniform over the warp except where noted.
template <bool kLean>
struct ListWarp {
    static constexpr bool kDoubles = false;
    static constexpr bool kOrderly = false;
    __device__ uint32_t ring_fin(const BatchArgs &) const { return out_fin; }
    __device__ uint32_t ring_pos(const BatchArgs &) const { return out_pos; }
    __device__ BatchOrder *window(const BatchArgs &) const { return reinterpret_cast<BatchOrder *>(smem + orders); }
    uint32_t clk, head_ts, head_dl, events, out_fin;     // f64 indices into shared memory
    uint32_t out_pos, counts, qpos, qlen, mrep, mlist, gcfg, glist;   // u32; counts: [2][G]
    uint32_t gmod, event_g, orders;                      // u16, byte, byte
    int64_t b;
    bool bad;                          // a table index is bad: nothing is simulated
    uint32_t status;                   // per lane
    // pending events: lane l owns the slots l, l + 32, ..., filled from the first on
    uint32_t ev_n;                     // of all lanes
    double top;                        // the earliest one, its group and its lane
    uint32_t top_g;
    int top_lane;
    uint64_t my_key;                   // per lane: its earliest, that one's group and row
    uint32_t my_g, my_row, my_n;       //   and how many it has
    int32_t queued;                    // requests in all queues
    // outputs
    bool record, direct;               // direct: carried requests are written, not listed
    int32_t own_begin;
    uint32_t out_n, carry_n;
    uint64_t tie;                      // not kept
    int32_t seg;
    Carried *carry;
    uint32_t my_bs, my_col;            // per lane: batch size and latency column
};

// ---- the candidate's tables --------------------------------------------------------
template <bool kLean>
__device__ __forceinline__ uint32_t replica_at(const BatchArgs &a, const ListWarp<kLean> &w, uint32_t e)
{
    return kLean ? __ldg(a.model_rep + (size_t)w.b * a.P + e) : SM_U32(w.mrep + e);
}
template <bool kLean>
__device__ __forceinline__ uint32_t replica_list(const BatchArgs &a, const ListWarp<kLean> &w, int32_t m)
{
    if (!kLean) return SM_U32(w.mlist + m);
    const uint16_t *off = a.model_off + (size_t)w.b * (a.M + 1) + m;
    const uint32_t lo = __ldg(off), hi = __ldg(off + 1);
    return lo | ((hi - lo) << 16);
}
template <bool kLean>
__device__ __forceinline__ uint32_t group_config(const BatchArgs &a, const ListWarp<kLean> &w, uint32_t g)
{
    return kLean ? __ldg(a.group_cfg + (size_t)w.b * a.G + g) : SM_U32(w.gcfg + g);
}
template <bool kLean>
__device__ __forceinline__ uint32_t group_list(const BatchArgs &a, const ListWarp<kLean> &w, uint32_t g)
{
    if (!kLean) return SM_U32(w.glist + g);
    const uint16_t *off = a.group_off + (size_t)w.b * (a.G + 1) + g;
    const uint32_t lo = __ldg(off), hi = __ldg(off + 1);
    return lo | ((hi - lo) << 16);
}
template <bool kLean>
__device__ __forceinline__ uint32_t group_model(const BatchArgs &a, const ListWarp<kLean> &w, uint32_t e)
{
    return kLean ? __ldg(a.group_mod + (size_t)w.b * a.P + e) : SM_U16(w.gmod + e);
}

// This lane's replica of a list (first entry | count << 16), as far as there is one.
template <bool kLean>
__device__ __forceinline__ uint32_t own_replica(const BatchArgs &a, const ListWarp<kLean> &w, uint32_t list)
{
    const uint32_t lane = threadIdx.x & (kLanes - 1);
    return lane < list >> 16 ? replica_at<kLean>(a, w, (list & 0xFFFFu) + lane) : 0u;
}

// All threads of the block, before any of them leaves.
__device__ inline void batch_stage_table(const BatchArgs &a)
{
    const int real = a.M * a.C * a.S * a.NB;
    for (int i = threadIdx.x; i < a.table_elems; i += blockDim.x)
        SM_F32(i) = i < real ? __ldg(a.latency + i) : 0.0f;
    __syncthreads();
}

// Idle clocks, empty queues, no events.
template <bool kLean>
__device__ inline void batch_zero_state(const BatchArgs &a, ListWarp<kLean> &w)
{
    const int lane = threadIdx.x & (kLanes - 1);
    for (int t = lane; t < a.T; t += kLanes) SM_F64(w.clk + t) = 0.0;
    for (int m = lane; m < a.M; m += kLanes) {
        SM_U32(w.qpos + m) = 0;
        SM_U32(w.qlen + m) = 0;
        if (!kLean) SM_F64(w.head_ts + m) = kNoHead;
    }
    for (int r = 0; r < a.event_rows; ++r)
        reinterpret_cast<uint64_t *>(smem)[w.events + r * kLanes + lane] = kNoEvent;
    w.ev_n = 0;
    w.my_n = 0;
    w.my_key = kNoEvent;
    w.queued = 0;
    __syncwarp();
}

// Candidate b's tables, every index checked: a bad one is reported and nothing is simulated.
template <bool kLean>
__device__ inline void batch_setup(const BatchArgs &a, ListWarp<kLean> &w, int64_t b)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const BatchSmem L = batch_smem(a.M, a.G, a.P, a.T, a.event_rows, a.table_elems, kLean, 1);
    const size_t base = L.warp0 + (size_t)(threadIdx.x / kLanes) * L.warp_bytes;
    w.orders = (uint32_t)(base + L.orders);
    w.clk = (uint32_t)((base + L.clocks) / 8);
    w.head_ts = (uint32_t)((base + L.head_ts) / 8);
    w.head_dl = (uint32_t)((base + L.head_dl) / 8);
    w.events = (uint32_t)((base + L.events) / 8);
    w.out_fin = (uint32_t)((base + L.out_fin) / 8);
    w.out_pos = (uint32_t)((base + L.out_pos) / 4);
    w.counts = (uint32_t)((base + L.counts) / 4);
    w.qpos = (uint32_t)((base + L.qpos) / 4);
    w.qlen = (uint32_t)((base + L.qlen) / 4);
    w.mrep = (uint32_t)((base + L.mrep) / 4);
    w.mlist = (uint32_t)((base + L.mlist) / 4);
    w.gcfg = (uint32_t)((base + L.gcfg) / 4);
    w.glist = (uint32_t)((base + L.glist) / 4);
    w.gmod = (uint32_t)((base + L.gmod) / 2);
    w.event_g = (uint32_t)(base + L.event_g);
    w.b = b;
    w.status = 0;
    w.record = w.direct = true;
    w.own_begin = 0;
    w.out_n = w.carry_n = 0;
    w.carry = nullptr;
    w.my_bs = (uint32_t)a.batch_sizes[lane < a.NB ? lane : 0];
    w.my_col = (uint32_t)a.batch_cols[lane < a.NB ? lane : 0];
    __syncwarp();
    bool bad = false;
    const uint16_t *moff = a.model_off + (size_t)b * (a.M + 1), *goff = a.group_off + (size_t)b * (a.G + 1);
    for (int g = lane; g < a.G; g += kLanes) {
        const uint32_t cfg = a.group_cfg[(size_t)b * a.G + g];
        const uint32_t slot = cfg & 0xFFu, ns = (cfg >> 8) & 0xFFu;
        bad |= slot + ns > (uint32_t)a.T || ns > (uint32_t)a.S || (cfg >> 16) >= (uint32_t)a.C;
        const uint32_t lo = goff[g], hi = goff[g + 1];
        bad |= lo > hi || hi > (uint32_t)a.P;
        if (!kLean) {
            SM_U32(w.gcfg + g) = cfg;
            SM_U32(w.glist + g) = lo | ((hi - lo) << 16);
        }
    }
    for (int m = lane; m < a.M; m += kLanes) {
        const uint32_t lo = moff[m], hi = moff[m + 1];
        bad |= lo > hi || hi > (uint32_t)a.P;
        if (!kLean) SM_U32(w.mlist + m) = lo | ((hi - lo) << 16);
    }
    const uint32_t n_rep = a.M > 0 ? moff[a.M] : 0u, n_mod = a.G > 0 ? goff[a.G] : 0u;
    for (uint32_t e = lane; e < (uint32_t)a.P; e += kLanes) {
        if (e < n_rep) {
            const uint32_t ent = a.model_rep[(size_t)b * a.P + e], g = ent & 0xFFu;
            if (g >= (uint32_t)a.G) bad = true;
            else {
                const uint32_t cfg = a.group_cfg[(size_t)b * a.G + g];
                bad |= ((ent >> 8) & 0xFFFFu) != (cfg & 0xFFFFu) || ((ent >> 16) & 0xFFu) == 0;
            }
            if (!kLean) SM_U32(w.mrep + e) = ent;
        }
        if (e < n_mod) {
            const uint32_t m = a.group_mod[(size_t)b * a.P + e];
            bad |= m >= (uint32_t)a.M;
            if (!kLean) SM_U16(w.gmod + e) = (uint16_t)m;
        }
    }
    for (int c = lane; c < 2 * a.G; c += kLanes) SM_U32(w.counts + c) = 0;
    w.bad = __any_sync(0xFFFFFFFFu, bad);
    __syncwarp();
}

// ---- pending events ------------------------------------------------------------------
#define BATCH_EVENT(w, row, lane) (reinterpret_cast<uint64_t *>(smem)[(w).events + (row) * kLanes + (lane)])
#define BATCH_EVENT_G(w, row, lane) (smem[(w).event_g + (row) * kLanes + (lane)])

// This lane's earliest event: (time, group) in order, like the tuples the reference pushes (:728).
template <bool kLean>
__device__ inline void events_scan(ListWarp<kLean> &w)
{
    const int lane = threadIdx.x & (kLanes - 1);
    w.my_key = kNoEvent;
    w.my_g = 0;
    w.my_row = 0;
    for (uint32_t r = 0; r < w.my_n; ++r) {
        const uint64_t key = BATCH_EVENT(w, r, lane);
        const uint32_t g = BATCH_EVENT_G(w, r, lane);
        if (key < w.my_key || (key == w.my_key && g < w.my_g)) { w.my_key = key; w.my_g = g; w.my_row = r; }
    }
}

// The earliest event of all lanes.
template <bool kLean>
__device__ __forceinline__ void events_top(ListWarp<kLean> &w)
{
    if (w.ev_n == 0) return;
    uint32_t who = warp_least(w.my_key);
    if (who & (who - 1)) {
        const bool in = (who >> (threadIdx.x & (kLanes - 1))) & 1u;
        const uint32_t g = __reduce_min_sync(0xFFFFFFFFu, in ? w.my_g : 0xFFFFFFFFu);
        who = __ballot_sync(0xFFFFFFFFu, in && w.my_g == g);
    }
    // (a NaN time, which only a table with one can lead to, may have every bit set)
    w.top_lane = who ? __ffs((int)who) - 1 : __ffs((int)__ballot_sync(0xFFFFFFFFu, w.my_n != 0)) - 1;
    const uint64_t key = __shfl_sync(0xFFFFFFFFu, w.my_key, w.top_lane);
    w.top_g = __shfl_sync(0xFFFFFFFFu, w.my_g, w.top_lane);
    w.top = __longlong_as_double((long long)(key ^ ((key >> 63) ? 0x8000000000000000ull : ~0ull)));
}

template <bool kLean>
__device__ __forceinline__ void event_pop(ListWarp<kLean> &w)
{
    const int lane = threadIdx.x & (kLanes - 1);
    if (lane == w.top_lane) {
        const uint32_t last = --w.my_n;
        if (w.my_row != last) {
            BATCH_EVENT(w, w.my_row, lane) = BATCH_EVENT(w, last, lane);
            BATCH_EVENT_G(w, w.my_row, lane) = BATCH_EVENT_G(w, last, lane);
        }
        BATCH_EVENT(w, last, lane) = kNoEvent;
        events_scan(w);
    }
    __syncwarp();
    --w.ev_n;
    events_top(w);
}

template <bool kLean>
__device__ __forceinline__ void event_push(const BatchArgs &a, ListWarp<kLean> &w, double t, uint32_t g)
{
    const int lane = threadIdx.x & (kLanes - 1);
    if (w.ev_n >= (uint32_t)a.H) { w.status |= MMS_STATUS_HEAP_OVERFLOW; return; }
    const uint32_t room = __ballot_sync(0xFFFFFFFFu, w.my_n < (uint32_t)a.event_rows);
    int to = (int)(g & (kLanes - 1));
    if (!((room >> to) & 1u)) to = __ffs((int)room) - 1;
    const uint64_t key = time_key(t);
    if (lane == to) {
        BATCH_EVENT(w, w.my_n, lane) = key;
        BATCH_EVENT_G(w, w.my_n, lane) = (uint8_t)g;
        if (key < w.my_key || (key == w.my_key && g < w.my_g) || w.my_n == 0) {
            w.my_key = key;
            w.my_g = g;
            w.my_row = w.my_n;
        }
        ++w.my_n;
    }
    const uint64_t top = time_key(w.top);
    if (w.ev_n == 0 || key < top || (key == top && g < w.top_g)) {
        w.top = t;
        w.top_g = g;
        w.top_lane = to;
    }
    ++w.ev_n;
}

// ---- the groups' counters -------------------------------------------------------------------
template <bool kLean>
__device__ __forceinline__ void count_add(const BatchArgs &a, const ListWarp<kLean> &w, uint32_t g, int32_t n,
                                          int32_t good)
{
    if ((threadIdx.x & (kLanes - 1)) == 0) {
        SM_U32(w.counts + g) += (uint32_t)n;
        SM_U32(w.counts + a.G + g) += (uint32_t)good;
    }
}

// Into `to` (null: nowhere), and from zero again.
template <bool kLean>
__device__ inline void counts_store(const BatchArgs &a, ListWarp<kLean> &w, uint32_t *to)
{
    __syncwarp();
    for (int c = threadIdx.x & (kLanes - 1); c < 2 * a.G; c += kLanes) {
        if (to) to[c] = SM_U32(w.counts + c);
        SM_U32(w.counts + c) = 0;
    }
    __syncwarp();
}

// ---- the simulation ------------------------------------------------------------------------
// select_model, :654-664: the group's model whose queue head arrived first; -1: nothing queued.
template <bool kLean>
__device__ __forceinline__ int32_t pick_model(const BatchArgs &a, const ListWarp<kLean> &w, uint32_t g)
{
    const int lane = threadIdx.x & (kLanes - 1);
    if (w.queued == 0) return -1;
    const uint32_t list = group_list<kLean>(a, w, g), lo = list & 0xFFFFu, n = list >> 16;
    uint64_t key = kNoEvent;
    uint32_t m = 0, at = 0;
    for (uint32_t e = lane; e < n; e += kLanes) {
        const uint32_t me = group_model<kLean>(a, w, lo + e);
        double ts;
        if (kLean) ts = (int32_t)SM_U32(w.qlen + me) > 0 ? a.pos_ts[SM_U32(w.qpos + me)] : kNoHead;
        else ts = SM_F64(w.head_ts + me);
        const uint64_t k = ts < kInf ? time_key(ts) : kNoEvent;
        if (k < key) { key = k; m = me; at = e; }
    }
    uint32_t who = warp_least(key);
    if (!who) return -1;
    if (n > (uint32_t)kLanes && (who & (who - 1))) {       // the first of the list
        const bool in = (who >> lane) & 1u;
        const uint32_t first = __reduce_min_sync(0xFFFFFFFFu, in ? at : 0xFFFFFFFFu);
        who = __ballot_sync(0xFFFFFFFFu, in && at == first);
    }
    return (int32_t)__shfl_sync(0xFFFFFFFFu, m, __ffs((int)who) - 1);
}

// handle_batched_requests with get_max_batch_under_slo, :674-732: group g serves model m at time
// ts; the queue of m is `len` requests from position `pos` on, the first one due at `dl`.
// The reference recurses when a model's whole queue was dropped; the loop is the same tail
// call.  Lane j works out what a batch of size j would do: `adm` as the admission check has it
// (:667-672: the overhead behind the stages), `run` as the dispatch has it (:715-719: before
// them).
template <bool kLean>
__device__ __forceinline__ void serve_group(const BatchArgs &a, ListWarp<kLean> &w, double ts, int32_t m,
                                            uint32_t g, int32_t pos, int32_t len, double dl)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const uint32_t cfg = group_config<kLean>(a, w, g);
    const uint32_t slot = cfg & 0xFFu, ns = (cfg >> 8) & 0xFFu, col = cfg >> 16;
    const uint32_t clk = w.clk + slot;
    for (;;) {
        const uint32_t row = (((uint32_t)m * a.C + col) * a.S) * a.NB + w.my_col;
        const float *lat_gl = a.latency + (size_t)w.b * a.latency_stride + row;
        const auto lat = [&](uint32_t k) {
            return (double)(a.table_elems ? SM_F32(row + k * a.NB) : __ldg(lat_gl + (size_t)k * a.NB));
        };
        double adm = ts, run = ts + kOverhead, t[kBatchDepth];
#pragma unroll
        for (uint32_t k = 0; k < kBatchDepth; ++k) {
            if (k >= ns) break;
            const double c = SM_F64(clk + k), l = lat(k);
            adm = tmax(c, adm) + l;
            run = tmax(run, c) + l;
            t[k] = run;
        }
        for (uint32_t k = kBatchDepth; k < ns; ++k) {
            const double c = SM_F64(clk + k), l = lat(k);
            adm = tmax(c, adm) + l;
            run = tmax(run, c) + l;
        }
        adm = adm + kOverhead;
        // :693-702 sizes whose requests are there and for which the head's deadline still holds
        uint32_t ok = __ballot_sync(0xFFFFFFFFu, lane < a.NB && (int32_t)w.my_bs <= len && adm <= dl);
        if (!(ok & 1u)) {
            // :677-686 drop queue heads that cannot make their deadline even alone
            const double alone = __shfl_sync(0xFFFFFFFFu, adm, 0);
            uint32_t pass;
            int32_t n;
            double due;
            do {
                due = lane < len ? a.pos_dl[pos + lane] : 0.0;
                pass = __ballot_sync(0xFFFFFFFFu, lane < len && alone <= due);
                n = pass ? __ffs((int)pass) - 1 : len < kLanes ? len : kLanes;
                outputs_add(a, w, n, pos, 0.0, kDropped);
                count_add(a, w, g, n, 0);
                pos += n;
                len -= n;
                w.queued -= n;
            } while (!pass && len > 0);
            if (len == 0) {                                // :709-713
                if (lane == 0) {
                    SM_U32(w.qlen + m) = 0;
                    if (!kLean) SM_F64(w.head_ts + m) = kNoHead;
                }
                __syncwarp();
                m = pick_model<kLean>(a, w, g);
                if (m < 0) return;
                pos = (int32_t)SM_U32(w.qpos + m);
                len = (int32_t)SM_U32(w.qlen + m);
                dl = kLean ? a.pos_dl[pos] : SM_F64(w.head_dl + m);
                continue;
            }
            dl = __shfl_sync(0xFFFFFFFFu, due, n);
            ok = __ballot_sync(0xFFFFFFFFu, lane < a.NB && (int32_t)w.my_bs <= len && adm <= dl);
        }
        const int j = __ffs((int)~ok) - 2;
        const int32_t bs = a.batch_sizes[j];
        if (lane == j) {
#pragma unroll
            for (uint32_t k = 0; k < kBatchDepth; ++k)
                if (k < ns) SM_F64(clk + k) = t[k];
            if (ns > kBatchDepth) {                        // the same chain again, stored
                double cur = t[kBatchDepth - 1];
                for (uint32_t k = kBatchDepth; k < ns; ++k) {
                    cur = tmax(cur, SM_F64(clk + k)) + lat(k);
                    SM_F64(clk + k) = cur;
                }
            }
        }
        const double fin = __shfl_sync(0xFFFFFFFFu, run, j), free_at = __shfl_sync(0xFFFFFFFFu, t[0], j);
        for (int32_t k = 0; k < bs; k += kLanes)
            outputs_add(a, w, bs - k < kLanes ? bs - k : kLanes, pos + k, fin, 0u);
        pos += bs;
        len -= bs;
        w.queued -= bs;
        double head_ts = kNoHead, head_dl = 0.0;
        if (!kLean && len > 0) { head_ts = a.pos_ts[pos]; head_dl = a.pos_dl[pos]; }
        count_add(a, w, g, bs, bs);
        event_push(a, w, free_at, g);
        if (lane == 0) {
            SM_U32(w.qpos + m) = (uint32_t)pos;
            SM_U32(w.qlen + m) = (uint32_t)len;
            if (!kLean) {
                SM_F64(w.head_ts + m) = head_ts;
                SM_F64(w.head_dl + m) = head_dl;
            }
        }
        __syncwarp();
        return;
    }
}

// Arrival o, :736-778; `ent`: per lane, the first 32 replicas of its model.  (One call of
// serve_group, so that the loop stays small.)
template <bool kLean>
__device__ __forceinline__ void batch_arrival(const BatchArgs &a, ListWarp<kLean> &w, const BatchOrder &o,
                                              uint32_t ent)
{
    const int lane = threadIdx.x & (kLanes - 1);
    bool events = true;
    for (;;) {
        double ts = o.ts, dl = o.dl;
        int32_t m = o.m, pos = o.pos, len;
        uint32_t g;
        const bool event = events && w.ev_n > 0 && w.top <= o.ts;
        if (event) {
            // :739-744 a group whose first stage became free before this arrival
            ts = w.top;
            g = w.top_g;
            event_pop(w);
            m = pick_model<kLean>(a, w, g);
            if (m < 0) { events = false; continue; }       // the reference breaks here, not continues
            pos = (int32_t)SM_U32(w.qpos + m);
            len = (int32_t)SM_U32(w.qlen + m);
            dl = kLean ? a.pos_dl[pos] : SM_F64(w.head_dl + m);
        } else {
            const uint32_t lo = (uint32_t)o.served & 0xFFFFu, n = (uint32_t)o.served >> 16;
            if (n == 0) return;                            // :748-757, see batch_run
            // :759-770 the replica whose last-stage clock is strictly smallest
            uint64_t key = kNoEvent;
            uint32_t at = 0, mine = ent;
            if ((uint32_t)lane < n) {
                const double c = SM_F64(w.clk + ((ent >> 8) & 0xFFu) + ((ent >> 16) & 0xFFu) - 1);
                if (c < kInf) key = time_key(c);
                at = lane;
            }
            for (uint32_t e = lane + kLanes; e < n; e += kLanes) {
                const uint32_t x = replica_at<kLean>(a, w, lo + e);
                const double c = SM_F64(w.clk + ((x >> 8) & 0xFFu) + ((x >> 16) & 0xFFu) - 1);
                const uint64_t k = c < kInf ? time_key(c) : kNoEvent;
                if (k < key) { key = k; mine = x; at = e; }
            }
            uint32_t who = warp_least(key);
            if (n > (uint32_t)kLanes && (who & (who - 1))) {       // the first of the list
                const bool in = (who >> lane) & 1u;
                const uint32_t first = __reduce_min_sync(0xFFFFFFFFu, in ? at : 0xFFFFFFFFu);
                who = __ballot_sync(0xFFFFFFFFu, in && at == first);
            }
            const uint32_t pick = __shfl_sync(0xFFFFFFFFu, mine, who ? __ffs((int)who) - 1 : 0);
            g = pick & 0xFFu;
            // :772-773 the request joins its MODEL's queue
            len = (int32_t)SM_U32(w.qlen + m) + 1;
            ++w.queued;
            // :776-778 (a group's idle time is the clock of its first stage: :727 stores it in both)
            if (!(who && ts >= SM_F64(w.clk + ((pick >> 8) & 0xFFu)))) {
                if (lane == 0) {
                    SM_U32(w.qlen + m) = (uint32_t)len;
                    if (len == 1) {
                        SM_U32(w.qpos + m) = (uint32_t)pos;
                        if (!kLean) {
                            SM_F64(w.head_ts + m) = ts;
                            SM_F64(w.head_dl + m) = dl;
                        }
                    }
                }
                __syncwarp();
                return;
            }
            if (len > 1) {
                pos = (int32_t)SM_U32(w.qpos + m);
                dl = kLean ? a.pos_dl[pos] : SM_F64(w.head_dl + m);
            }
        }
        serve_group<kLean>(a, w, ts, m, g, pos, len, dl);
        if (!event) return;
    }
}

// Arrivals [k, k1) of the window at work.
template <bool kLean>
__device__ __forceinline__ void batch_arrivals(const BatchArgs &a, ListWarp<kLean> &w, int k, int k1)
{
    const BatchOrder *orders = reinterpret_cast<const BatchOrder *>(smem + w.orders);
    BatchOrder o = orders[k];
    uint32_t ent = own_replica<kLean>(a, w, (uint32_t)o.served);
    while (k < k1) {
        ++k;
        const BatchOrder next = orders[k < kLanes ? k : kLanes - 1];
        const uint32_t next_ent = own_replica<kLean>(a, w, (uint32_t)next.served);
        batch_arrival<kLean>(a, w, o, ent);
        o = next;
        ent = next_ent;
    }
}

template <bool kLean>
__device__ __forceinline__ uint64_t replicas_of(const BatchArgs &a, const ListWarp<kLean> &w, int32_t m)
{
    const uint32_t list = replica_list<kLean>(a, w, m);
    return list >> 16 ? list : 0u;
}

// After the last arrival, :781-790.
template <bool kLean>
__device__ inline void batch_drain(const BatchArgs &a, ListWarp<kLean> &w)
{
    while (w.ev_n > 0) {
        const double te = w.top;
        const uint32_t ge = w.top_g;
        event_pop(w);
        const int32_t m = pick_model<kLean>(a, w, ge);
        if (m < 0) continue;
        const int32_t pos = (int32_t)SM_U32(w.qpos + m);
        serve_group<kLean>(a, w, te, m, ge, pos, (int32_t)SM_U32(w.qlen + m),
                           kLean ? a.pos_dl[pos] : SM_F64(w.head_dl + m));
    }
    if (w.queued != 0) w.status |= MMS_STATUS_QUEUE_LEFT;
}

// ---- states ----------------------------------------------------------------------------------
template <bool kLean>
__device__ inline void state_save(const BatchArgs &a, const ListWarp<kLean> &w, unsigned char *p)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const StateView v = state_view(a, p);
    __syncwarp();
    for (int t = lane; t < a.T; t += kLanes) v.clk[t] = SM_F64(w.clk + t);
    for (int r = 0; r < a.event_rows; ++r) {
        v.ev[r * kLanes + lane] = BATCH_EVENT(w, r, lane);
        v.ev_g[r * kLanes + lane] = BATCH_EVENT_G(w, r, lane);
    }
    for (int m = lane; m < a.M; m += kLanes) {
        v.qpos[m] = (int32_t)SM_U32(w.qpos + m);
        v.qlen[m] = (int32_t)SM_U32(w.qlen + m);
    }
    if (lane == 0) *v.ev_n = w.ev_n;
    __syncwarp();
}

template <bool kLean>
__device__ inline void state_load(const BatchArgs &a, ListWarp<kLean> &w, unsigned char *p)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const StateView v = state_view(a, p);
    __syncwarp();
    for (int t = lane; t < a.T; t += kLanes) SM_F64(w.clk + t) = v.clk[t];
    w.my_n = 0;
    for (int r = 0; r < a.event_rows; ++r) {
        const uint64_t key = v.ev[r * kLanes + lane];
        BATCH_EVENT(w, r, lane) = key;
        BATCH_EVENT_G(w, r, lane) = v.ev_g[r * kLanes + lane];
        w.my_n += key != kNoEvent;
    }
    int32_t queued = 0;
    for (int m = lane; m < a.M; m += kLanes) {
        const int32_t len = v.qlen[m], pos = v.qpos[m];
        SM_U32(w.qlen + m) = (uint32_t)len;
        SM_U32(w.qpos + m) = (uint32_t)pos;
        if (!kLean) {
            SM_F64(w.head_ts + m) = len > 0 ? a.pos_ts[pos] : kNoHead;
            SM_F64(w.head_dl + m) = len > 0 ? a.pos_dl[pos] : 0.0;
        }
        queued += len;
    }
    w.queued = (int32_t)__reduce_add_sync(0xFFFFFFFFu, (uint32_t)queued);
    w.ev_n = *v.ev_n;
    events_scan(w);
    __syncwarp();
    events_top(w);
}

// The state on chip and a saved one, both taken just before the arrival at time tau, lead to
// identical futures when
//  - every queue has the same length and, if not empty, the same head (a queue is a run of
//    consecutive requests of its model);
//  - the pending events are the same (they are taken in the order of (time, group));
//  - every clock is equal in both or < theta in both, theta = the earlier of tau and the
//    first pending event: a clock only ever enters max(clock, t) with t an arrival time or a
//    pending event's time (:669, :719), or (the first stage's, a group's idle time) is compared
//    with arrival times >= tau (:776);
//  - the last-stage clocks that differ (both < theta) of groups serving a replicated model
//    are in the same order (ties included) relative to those of all groups they share a
//    model with: dispatch compares them with '<' (:764).
// Sufficient, not necessary: a failed check only costs a re-simulation.
template <bool kLean>
__device__ inline bool batch_equivalent(const BatchArgs &a, const ListWarp<kLean> &w, unsigned char *saved,
                                        double tau)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const StateView v = state_view(a, saved);
    __syncwarp();
    if (*v.ev_n != w.ev_n) return false;
    bool bad = false;
    for (int m = lane; m < a.M; m += kLanes) {
        const uint32_t n = SM_U32(w.qlen + m);
        bad |= n != (uint32_t)v.qlen[m] || (n > 0 && SM_U32(w.qpos + m) != (uint32_t)v.qpos[m]);
    }
    if (__any_sync(0xFFFFFFFFu, bad)) return false;
    const double theta = w.ev_n > 0 && w.top < tau ? w.top : tau;
    bool differ = false;
    for (int t = lane; t < a.T; t += kLanes) {
        const double x = SM_F64(w.clk + t), y = v.clk[t];
        bad |= !(x == y || (x < theta && y < theta));
        differ |= x != y;
    }
    if (__any_sync(0xFFFFFFFFu, bad)) return false;
    // every event as often in the one as in the other
    bool moved = false;
    for (int r = 0; r < a.event_rows; ++r) {
        const uint64_t x = BATCH_EVENT(w, r, lane), y = v.ev[r * kLanes + lane];
        moved |= x != y || (x != kNoEvent && BATCH_EVENT_G(w, r, lane) != v.ev_g[r * kLanes + lane]);
    }
    if (__any_sync(0xFFFFFFFFu, moved)) {
        for (int s = 0; s < a.event_rows; ++s)
            for (int l = 0; l < kLanes; ++l) {
                const uint64_t key = BATCH_EVENT(w, s, l);
                if (key == kNoEvent) continue;
                const uint32_t g = BATCH_EVENT_G(w, s, l);
                int here = 0, there = 0;
                for (int r = 0; r < a.event_rows; ++r) {
                    here += __popc(__ballot_sync(0xFFFFFFFFu, BATCH_EVENT(w, r, lane) == key &&
                                                                  BATCH_EVENT_G(w, r, lane) == g));
                    there += __popc(__ballot_sync(0xFFFFFFFFu, v.ev[r * kLanes + lane] == key &&
                                                                   v.ev_g[r * kLanes + lane] == g));
                }
                if (here != there) return false;
            }
    }
    if (!__any_sync(0xFFFFFFFFu, differ)) return true;
    for (int m = lane; m < a.M; m += kLanes) {
        const uint32_t list = replica_list<kLean>(a, w, m), lo = list & 0xFFFFu, hi = lo + (list >> 16);
        for (uint32_t e = lo; e + 1 < hi; ++e) {
            const uint32_t eu = replica_at<kLean>(a, w, e);
            const uint32_t su = ((eu >> 8) & 0xFFu) + ((eu >> 16) & 0xFFu) - 1;
            const double xu = SM_F64(w.clk + su), yu = v.clk[su];
            for (uint32_t f = e + 1; f < hi; ++f) {
                const uint32_t ev = replica_at<kLean>(a, w, f);
                const uint32_t sv = ((ev >> 8) & 0xFFu) + ((ev >> 16) & 0xFFu) - 1;
                const double xv = SM_F64(w.clk + sv), yv = v.clk[sv];
                bad |= (xu < xv) != (yu < yv) || (xu > xv) != (yu > yv);
            }
        }
    }
    return !__any_sync(0xFFFFFFFFu, bad);
}

// The lists know no labels.
template <bool kLean>
__device__ inline void labels_reset(const BatchArgs &, const ListWarp<kLean> &) {}

}  // namespace mms
