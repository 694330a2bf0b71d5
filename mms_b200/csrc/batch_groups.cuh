// batch_groups.cuh — the batching simulator with a group per lane (see sim_batching.cuh).
//
// For candidates of up to 64 groups and 64 models whose latency table fits on chip, on a trace
// without oddities (BatchArgs::odd): lane g keeps, in registers, the earliest pending event of group g, its
// idle time and its last-stage clock, and sets of groups and of models are bit masks.  What an arrival
// costs is its instructions, at 6 to 7 cycles each for a lone warp: 255 to 330 of them (550 with lists, nearly
// as many as one lane that goes through the reference's loops), branches most of all, whose conditions the
// compiler cannot see to be the same in all lanes.  A lone warp takes 1.0 us an arrival, and four
// on its scheduler take no longer.
//
// Events of one group come in ascending order (its first clock never goes back), so a group's
// other pending ones, which are rare, wait in a list (`extra`) behind its earliest.
#pragma once
#include "sim_core.cuh"

namespace mms {

template <int kPer>
struct GroupWarp {
    static constexpr bool kDoubles = true;               // the table on chip
    static constexpr bool kOrderly = true;               // needs a trace and table without oddities
    static constexpr int kGroups = kPer;                 // per lane
    __device__ uint32_t ring_fin(const BatchArgs &a) const { return (base >> 3) + a.at.out_fin; }
    __device__ uint32_t ring_pos(const BatchArgs &a) const { return (base >> 2) + a.at.out_pos; }
    __device__ BatchOrder *window(const BatchArgs &a) const { return reinterpret_cast<BatchOrder *>(smem + base + a.at.orders); }
    uint32_t base;                       // of the warp's shared memory, in bytes
    int64_t b;
    bool bad;                            // a table index is bad: nothing is simulated
    uint32_t status;                     // per lane
    double ev[kPer], idle[kPer], last[kPer];             // per lane: of groups lane and lane + 32
    uint32_t extra_n;
    uint64_t waiting;                    // models with a queue
    uint64_t tie;                        // groups that a group number decided about
    bool plain;                          // the candidate's lists are in ascending order
    uint32_t requests[kPer], good[kPer]; // per lane: counted since the segment's begin
    Swap *swaps;                         // null: not noted
    uint32_t swap_n;
    int32_t seg;                         // the segment at work
    bool record, direct;
    int32_t own_begin;
    uint32_t out_n, carry_n;
    Carried *carry;
    int32_t my_bs;                       // per lane: batch size (none: longer than any queue)
    uint32_t my_col;                     //   and latency column
};

#define SM_U64(i) (reinterpret_cast<uint64_t *>(smem)[(i)])

// No event: not a number, and as an integer above every time.
__device__ __forceinline__ double no_event() { return __longlong_as_double(0x7FFFFFFFFFFFFFFFll); }

// Where things are in a warp's shared memory, an index in the entry's own size.
#define AT8(field) ((w.base >> 3) + a.at.field)
#define AT4(field) ((w.base >> 2) + a.at.field)
#define AT1(field) (w.base + a.at.field)

template <int kPer>
__device__ inline void batch_setup(const BatchArgs &a, GroupWarp<kPer> &w, int64_t b)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const uint32_t base = a.warp0 + (uint32_t)(threadIdx.x / kLanes) * a.warp_bytes;
    w.base = base;
    w.b = b;
    w.status = 0;
    w.record = w.direct = true;
    w.own_begin = 0;
    w.out_n = w.carry_n = 0;
    w.carry = nullptr;
    w.my_bs = lane < a.NB ? a.batch_sizes[lane] : 0x7FFFFFFF;
    w.my_col = (uint32_t)a.batch_cols[lane < a.NB ? lane : 0];
    __syncwarp();
    bool bad = false, unordered = false;
    const uint16_t *moff = a.model_off + (size_t)b * (a.M + 1), *goff = a.group_off + (size_t)b * (a.G + 1);
    for (int g = lane; g < kGroupLimit; g += kLanes) {
        uint32_t cfg = 0;
        uint64_t models = 0;
        if (g < a.G) {
            cfg = a.group_cfg[(size_t)b * a.G + g];
            const uint32_t slot = cfg & 0xFFu, ns = (cfg >> 8) & 0xFFu;
            bad |= slot + ns > (uint32_t)a.T || ns > (uint32_t)a.S || (cfg >> 16) >= (uint32_t)a.C;
            const uint32_t lo = goff[g], hi = goff[g + 1];
            bad |= lo > hi || hi > (uint32_t)a.P;
            for (uint32_t e = lo; e < hi && e < (uint32_t)a.P; ++e) {
                const uint32_t m = a.group_mod[(size_t)b * a.P + e];
                if (m >= (uint32_t)a.M) { bad = true; continue; }
                unordered |= models >> m != 0;
                models |= 1ull << m;
            }
        }
        SM_U32(AT4(info) + g) = cfg;
        SM_U64(AT8(serves) + g) = models;
    }
    for (int m = lane; m < a.M; m += kLanes) {
        uint64_t groups = 0;
        const uint32_t lo = moff[m], hi = moff[m + 1];
        bad |= lo > hi || hi > (uint32_t)a.P;
        for (uint32_t e = lo; e < hi && e < (uint32_t)a.P; ++e) {
            const uint32_t ent = a.model_rep[(size_t)b * a.P + e], g = ent & 0xFFu;
            if (g >= (uint32_t)a.G) { bad = true; continue; }
            const uint32_t cfg = a.group_cfg[(size_t)b * a.G + g];
            bad |= ((ent >> 8) & 0xFFFFu) != (cfg & 0xFFFFu) || ((ent >> 16) & 0xFFu) == 0;
            unordered |= groups >> g != 0;
            groups |= 1ull << g;
        }
        SM_U64(AT8(served) + m) = groups;
    }
    w.bad = __any_sync(0xFFFFFFFFu, bad);
    w.plain = !__any_sync(0xFFFFFFFFu, unordered);
    w.tie = 0;
    w.swaps = nullptr;
    w.swap_n = 0;
#pragma unroll
    for (int h = 0; h < kPer; ++h) w.requests[h] = w.good[h] = 0;
    for (int g = lane; g < kGroupLimit; g += kLanes) smem[AT1(labels) + g] = (uint8_t)g;
    __syncwarp();
}

template <int kPer>
__device__ __forceinline__ void count_add(const BatchArgs &, GroupWarp<kPer> &w, int32_t g, int32_t n, int32_t good)
{
#pragma unroll
    for (int h = 0; h < kPer; ++h)
        if ((int)(threadIdx.x & (kLanes - 1)) + h * kLanes == g) {
            w.requests[h] += n;
            w.good[h] += good;
        }
}

template <int kPer>
__device__ inline void counts_store(const BatchArgs &a, GroupWarp<kPer> &w, uint32_t *to)
{
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const int g = (int)(threadIdx.x & (kLanes - 1)) + h * kLanes;
        if (to && g < a.G) {
            to[g] = w.requests[h];
            to[a.G + g] = w.good[h];
        }
        w.requests[h] = w.good[h] = 0;
    }
}

template <int kPer>
__device__ inline void batch_zero_state(const BatchArgs &a, GroupWarp<kPer> &w)
{
    const int lane = threadIdx.x & (kLanes - 1);
    for (int t = lane; t < a.T; t += kLanes) SM_F64(AT8(clk) + t) = 0.0;
#pragma unroll
    for (int h = 0; h < kPer; ++h) { w.ev[h] = no_event(); w.idle[h] = w.last[h] = 0.0; }
    w.extra_n = 0;
    w.waiting = 0;
    w.tie = 0;
    __syncwarp();
}

// The groups of `in` (per lane: groups lane, lane + 32) with the smallest value, none of which is
// negative.
template <int kPer>
__device__ __forceinline__ uint64_t least_groups(const bool (&in)[kPer], const double (&value)[kPer])
{
    uint32_t who[kPer];
    const auto several = [&]() {
        uint32_t more = who[0] & (who[0] - 1);
        if constexpr (kPer == 2) more |= (who[1] & (who[1] - 1)) | (who[0] ? who[1] : 0u);
        return more != 0;
    };
#pragma unroll
    for (int h = 0; h < kPer; ++h) who[h] = __ballot_sync(0xFFFFFFFFu, in[h]);
    if (several()) {
        uint32_t hi[kPer], least = 0xFFFFFFFFu;
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            hi[h] = in[h] ? (uint32_t)__double2hiint(value[h]) : 0xFFFFFFFFu;
            least = hi[h] < least ? hi[h] : least;
        }
        least = __reduce_min_sync(0xFFFFFFFFu, least);
#pragma unroll
        for (int h = 0; h < kPer; ++h) who[h] = __ballot_sync(0xFFFFFFFFu, hi[h] == least);
        if (several()) {
            uint32_t lo[kPer], low = 0xFFFFFFFFu;
#pragma unroll
            for (int h = 0; h < kPer; ++h) {
                lo[h] = hi[h] == least ? (uint32_t)__double2loint(value[h]) : 0xFFFFFFFFu;
                low = lo[h] < low ? lo[h] : low;
            }
            low = __reduce_min_sync(0xFFFFFFFFu, low);
#pragma unroll
            for (int h = 0; h < kPer; ++h) who[h] = __ballot_sync(0xFFFFFFFFu, hi[h] == least && lo[h] == low);
        }
    }
    if constexpr (kPer == 2) return who[0] | ((uint64_t)who[1] << 32);
    else return who[0];
}

// Of several equally good groups of a model (kOfModel) or models of a group: the first in the
// caller's list.
template <bool kOfModel>
__device__ __noinline__ int32_t first_listed(const BatchArgs &a, int64_t b, int32_t of, uint64_t among)
{
    const uint16_t *off = kOfModel ? a.model_off + (size_t)b * (a.M + 1) : a.group_off + (size_t)b * (a.G + 1);
    const uint32_t lo = off[of], hi = off[of + 1];
    for (uint32_t base = lo; base < hi; base += kLanes) {
        const uint32_t e = base + (threadIdx.x & (kLanes - 1));
        uint32_t id = 0;
        if (e < hi) id = kOfModel ? a.model_rep[(size_t)b * a.P + e] & 0xFFu : a.group_mod[(size_t)b * a.P + e];
        const uint32_t is = __ballot_sync(0xFFFFFFFFu, e < hi && ((among >> id) & 1u));
        if (is) return (int32_t)__shfl_sync(0xFFFFFFFFu, id, __ffs((int)is) - 1);
    }
    return -1;
}

// The model among `models`, of which several wait, whose queue head arrived first.
template <int kPer>
__device__ __forceinline__ int32_t earliest_head(const BatchArgs &a, const GroupWarp<kPer> &w, int32_t g,
                                                 uint64_t models)
{
    const int lane = threadIdx.x & (kLanes - 1);
    bool in[2];
    double ts[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        in[h] = (models >> (lane + h * kLanes)) & 1u;
        ts[h] = in[h] ? SM_F64(AT8(head_ts) + lane + h * kLanes) : 0.0;
        in[h] = in[h] && ts[h] < kInf;
    }
    const uint64_t who = least_groups<2>(in, ts);
    return who & (who - 1) ? first_listed<false>(a, w.b, g, who) : (int32_t)__ffsll((long long)who) - 1;
}

// An event of group g at time t, behind one that is pending already.
template <int kPer>
__device__ __forceinline__ void extra_push(const BatchArgs &a, GroupWarp<kPer> &w, double t, int32_t g)
{
    uint32_t pending = w.extra_n;
#pragma unroll
    for (int h = 0; h < kPer; ++h) pending += __popc(__ballot_sync(0xFFFFFFFFu, w.ev[h] == w.ev[h]));
    if (pending >= (uint32_t)a.H) { w.status |= MMS_STATUS_HEAP_OVERFLOW; return; }
    if ((threadIdx.x & (kLanes - 1)) == 0) {
        SM_F64(AT8(extra) + w.extra_n) = t;
        smem[AT1(extra_g) + w.extra_n] = (uint8_t)g;
    }
    ++w.extra_n;
    __syncwarp();
}

// Are more events pending than there is room for?  A group's earliest has a place of its own and is not
// refused one, but counts.  Events only go when they are taken, so asking before that finds every
// excess: 0.8 % of the simulation (256 placements over 45 538 requests 8.36 -> 8.42 ms), as a function that is called, here
// or in extra_pop, 2 %, at each dispatch 1.3 %.
template <int kPer>
__device__ __forceinline__ void room_check(const BatchArgs &a, GroupWarp<kPer> &w)
{
    uint32_t pending = w.extra_n;
#pragma unroll
    for (int h = 0; h < kPer; ++h) pending += __popc(__ballot_sync(0xFFFFFFFFu, w.ev[h] == w.ev[h]));
    if (pending > (uint32_t)a.H) w.status |= MMS_STATUS_HEAP_OVERFLOW;
}

// The next event of group g, taken out of the list; no_event() if there is none.
__device__ __noinline__ double extra_pop(uint32_t extra, uint32_t extra_g, uint32_t n, int32_t g)
{
    const int lane = threadIdx.x & (kLanes - 1);
    uint64_t best = ~0ull;
    uint32_t at = 0;
    for (uint32_t e = lane; e < n; e += kLanes) {
        const uint64_t key = smem[extra_g + e] == (uint32_t)g ? (uint64_t)__double_as_longlong(SM_F64(extra + e)) : ~0ull;
        if (key < best) { best = key; at = e; }
    }
    const uint32_t who = warp_least(best);
    if (!who) return no_event();
    const int from = __ffs((int)who) - 1;
    const double t = __longlong_as_double((long long)__shfl_sync(0xFFFFFFFFu, best, from));
    at = __shfl_sync(0xFFFFFFFFu, at, from);
    __syncwarp();
    if (lane == 0) {
        SM_F64(extra + at) = SM_F64(extra + n - 1);
        smem[extra_g + at] = smem[extra_g + n - 1];
    }
    __syncwarp();
    return t;
}

// A choice of `picked` among the groups `who`, alike in what was compared, that the group number
// decided.  Those that are interchangeable with the picked one and in its state (every clock, and
// the pending event) are the result's `swap`, if there are any besides itself; `tie`: the groups of the others
// that matter, and itself with them (not those that come behind all of the picked one's class: then the
// true choice is among the picked one's class as well, whatever the labels).
struct BatchTie { uint64_t swap, tie; };
template <int kPer>
__device__ __noinline__ BatchTie judge_tie(const BatchArgs &a, const uint32_t base, const uint64_t who,
                                           const int32_t picked, const double ev0, const double ev1)
{
    struct { uint32_t base; } w = {base};              // for AT4, AT8
    const int lane = threadIdx.x & (kLanes - 1);
    const uint32_t cfg = SM_U32(AT4(info) + picked), ns = (cfg >> 8) & 0xFFu;
    const uint64_t models = SM_U64(AT8(serves) + picked);
    const double ev = __shfl_sync(0xFFFFFFFFu, kPer == 2 && picked >= kLanes ? ev1 : ev0, picked & (kLanes - 1));
    uint64_t cls = 0, same = 0;
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const int g = lane + h * kLanes;
        const uint32_t mine = SM_U32(AT4(info) + g);
        const bool twin = mine >> 8 == cfg >> 8 && SM_U64(AT8(serves) + g) == models;
        bool alike = twin && ((who >> g) & 1u) &&
                     __double_as_longlong(ev) == __double_as_longlong(h ? ev1 : ev0);
        for (uint32_t k = 0; alike && k < ns; ++k)
            alike = SM_F64(AT8(clk) + (cfg & 0xFFu) + k) == SM_F64(AT8(clk) + (mine & 0xFFu) + k);
        cls |= (uint64_t)__ballot_sync(0xFFFFFFFFu, twin) << (32 * h);
        same |= (uint64_t)__ballot_sync(0xFFFFFFFFu, alike) << (32 * h);
    }
    BatchTie t;
    t.swap = same & (same - 1) ? same : 0;
    t.tie = 0;
    for (uint64_t rest = who & ~same; rest; rest &= rest - 1) {
        const int o = (int)__ffsll((long long)rest) - 1;
        const uint32_t other = SM_U32(AT4(info) + o) >> 8;
        const uint64_t set = SM_U64(AT8(serves) + o);
        uint64_t ocls = 0;
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            const int g = lane + h * kLanes;
            ocls |= (uint64_t)__ballot_sync(0xFFFFFFFFu, SM_U32(AT4(info) + g) >> 8 == other &&
                                                             SM_U64(AT8(serves) + g) == set) << (32 * h);
        }
        const bool behind = !(ocls & cls) && 63 - __clzll((long long)cls) < (int)__ffsll((long long)ocls) - 1;
        if (!behind) t.tie |= (1ull << o) | (1ull << picked);
    }
    return t;
}

template <int kPer>
__device__ __forceinline__ void note_tie(const BatchArgs &a, GroupWarp<kPer> &w, uint64_t who, int32_t picked)
{
    if (!w.record || !w.swaps) return;
    if (w.extra_n) { w.tie |= who; return; }
    const BatchTie t = judge_tie<kPer>(a, w.base, who, picked, w.ev[0], w.ev[kPer - 1]);
    w.tie |= t.tie;
    if (!t.swap) return;
    bool large = false;
#pragma unroll
    for (int h = 0; h < kPer; ++h) large |= w.requests[h] > 0xFFFFu;
    if (w.swap_n >= (uint32_t)kSwapCap || __popcll(t.swap) > kSwapGroups || __any_sync(0xFFFFFFFFu, large)) {
        w.tie |= t.swap;
        return;
    }
    Swap *to = w.swaps + w.swap_n;
    const int lane = threadIdx.x & (kLanes - 1);
    if (lane == 0) {
        to->groups = t.swap;
        to->seg = w.seg;
        to->picked = (uint32_t)picked;
    }
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const int g = lane + h * kLanes;
        if ((t.swap >> g) & 1u) {
            const int k = __popcll(t.swap & ((1ull << g) - 1u));
            to->requests[k] = (uint16_t)w.requests[h];
            to->good[k] = (uint16_t)w.good[h];
            w.requests[h] = w.good[h] = 0;
        }
    }
    ++w.swap_n;
}

// Takes the earliest of the due events (a.ts) of `in`: its group and time.
template <int kPer>
__device__ __forceinline__ int32_t event_take(const BatchArgs &a, GroupWarp<kPer> &w, const bool (&in)[kPer], double &te)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const uint64_t who = least_groups<kPer>(in, w.ev);
    const int32_t g = (int32_t)__ffsll((long long)who) - 1;      // of equal times the lowest group
    if (who & (who - 1)) note_tie(a, w, who, g);
    double t = w.ev[0];
    if constexpr (kPer == 2) t = g >= kLanes ? w.ev[1] : w.ev[0];
    te = __shfl_sync(0xFFFFFFFFu, t, g & (kLanes - 1));
    double next = no_event();
    if (w.extra_n) {
        if (w.extra_n > a.spare) room_check(a, w);
        next = extra_pop(AT8(extra), AT1(extra_g), w.extra_n, g);
        w.extra_n -= next == next;
    }
#pragma unroll
    for (int h = 0; h < kPer; ++h)
        if (lane + h * kLanes == g) w.ev[h] = next;
    return g;
}

// serve_group above.
template <int kPer>
__device__ __forceinline__ void serve_group(const BatchArgs &a, GroupWarp<kPer> &w, double ts, int32_t m,
                                            int32_t g, int32_t pos, int32_t len, double dl)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const uint32_t cfg = SM_U32(AT4(info) + g);
    const uint32_t slot = cfg & 0xFFu, ns = (cfg >> 8) & 0xFFu, col = cfg >> 16;
    const uint32_t clk = AT8(clk) + slot;
    for (;;) {
        const uint32_t row = (((uint32_t)m * a.C + col) * a.S) * a.NB + w.my_col;
        double adm = ts, run = ts + kOverhead, t[kBatchDepth];
#pragma unroll
        for (uint32_t k = 0; k < kBatchDepth; ++k) {
            const double c = SM_F64(clk + k), l = SM_F64(row + k * a.NB);
            adm = tmax(c, adm) + l;
            run = tmax(run, c) + l;
            t[k] = run;
            if (k + 1 >= ns) break;
        }
        for (uint32_t k = kBatchDepth; k < ns; ++k) {
            const double c = SM_F64(clk + k), l = SM_F64(row + k * a.NB);
            adm = tmax(c, adm) + l;
            run = tmax(run, c) + l;
        }
        adm = adm + kOverhead;
        // :693-702 sizes whose requests are there and for which the head's deadline still holds
        uint32_t ok = __ballot_sync(0xFFFFFFFFu, w.my_bs <= len && adm <= dl);
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
            } while (!pass && len > 0);
            if (len == 0) {                                // :709-713
                w.waiting &= ~(1ull << m);
                const uint64_t models = SM_U64(AT8(serves) + g) & w.waiting;
                if (!models) return;
                m = models & (models - 1) ? earliest_head(a, w, g, models) : (int32_t)__ffsll((long long)models) - 1;
                if (m < 0) return;
                const uint64_t q = SM_U64(AT8(queue) + m);
                pos = (int32_t)q;
                len = (int32_t)(q >> 32);
                dl = SM_F64(AT8(head_dl) + m);
                continue;
            }
            dl = __shfl_sync(0xFFFFFFFFu, due, n);
            ok = __ballot_sync(0xFFFFFFFFu, w.my_bs <= len && adm <= dl);
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
                    cur = tmax(cur, SM_F64(clk + k)) + SM_F64(row + k * a.NB);
                    SM_F64(clk + k) = cur;
                }
            }
        }
        const double fin = __shfl_sync(0xFFFFFFFFu, run, j), free_at = __shfl_sync(0xFFFFFFFFu, t[0], j);
        for (int32_t k = 0; k < bs; k += kLanes)
            outputs_add(a, w, bs - k < kLanes ? bs - k : kLanes, pos + k, fin, 0u);
        bool behind = false;
#pragma unroll
        for (int h = 0; h < kPer; ++h)
            if (lane + h * kLanes == g) {
                w.last[h] = fin;
                w.idle[h] = free_at;
                behind = w.ev[h] == w.ev[h];
                w.ev[h] = behind ? w.ev[h] : free_at;
                w.requests[h] += bs;
                w.good[h] += bs;
            }
        if (__any_sync(0xFFFFFFFFu, behind)) extra_push(a, w, free_at, g);
        if (len > bs) {
            pos += bs;
            const double head_ts = a.pos_ts[pos], head_dl = a.pos_dl[pos];
            if (lane == 0) {
                SM_U64(AT8(queue) + m) = (uint32_t)pos | ((uint64_t)(uint32_t)(len - bs) << 32);
                SM_F64(AT8(head_ts) + m) = head_ts;
                SM_F64(AT8(head_dl) + m) = head_dl;
            }
            w.waiting |= 1ull << m;
        } else {
            w.waiting &= ~(1ull << m);
        }
        __syncwarp();
        return;
    }
}

// Arrivals [k, k1) of the window at work, :736-778.
template <int kPer>
__device__ __forceinline__ void batch_arrivals(const BatchArgs &a, GroupWarp<kPer> &w, int k, int k1)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const BatchOrder *orders = reinterpret_cast<const BatchOrder *>(smem + AT1(orders));
    BatchOrder o = orders[k], next = o;
    bool events = true;
    for (;;) {
        double ts = o.ts, dl = o.dl;
        int32_t m = o.m, pos = o.pos, len = 1, g;
        bool due[kPer];
        uint32_t any = 0;
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            due[h] = w.ev[h] <= ts;
            any |= __ballot_sync(0xFFFFFFFFu, due[h]);
        }
        const bool event = events && any;
        if (event) {
            // :739-744 a group whose first stage became free before this arrival
            g = event_take(a, w, due, ts);
            const uint64_t models = SM_U64(AT8(serves) + g) & w.waiting;
            if (!models) { events = false; continue; }     // the reference breaks here, not continues
            m = models & (models - 1) ? earliest_head(a, w, g, models) : (int32_t)__ffsll((long long)models) - 1;
            if (m < 0) { events = false; continue; }
            const uint64_t q = SM_U64(AT8(queue) + m);
            pos = (int32_t)q;
            len = (int32_t)(q >> 32);
            dl = SM_F64(AT8(head_dl) + m);
        } else {
            next = orders[k + 1 < kLanes ? k + 1 : k];
            bool serve = false;
            if (o.served) {                                // :748-757, see batch_run
                // :759-770 the replica whose last-stage clock is strictly smallest
                bool in[kPer];
                uint32_t idle[kPer];
#pragma unroll
                for (int h = 0; h < kPer; ++h) {
                    in[h] = ((uint32_t)(o.served >> (32 * h)) >> lane) & 1u && w.last[h] < kInf;
                    idle[h] = __ballot_sync(0xFFFFFFFFu, ts >= w.idle[h]);
                }
                const uint64_t who = least_groups<kPer>(in, w.last);
                g = (int32_t)__ffsll((long long)who) - 1;
                if (who & (who - 1)) {
                    g = first_listed<true>(a, w.b, m, who);
                    note_tie(a, w, who, g);
                }
                // :776-778 (a group's idle time is the clock of its first stage: :727 stores it in both)
                uint64_t idles = idle[0];
                if constexpr (kPer == 2) idles |= (uint64_t)idle[1] << 32;
                serve = g >= 0 && ((idles >> g) & 1u);
                // :772-773 the request joins its MODEL's queue
                if ((w.waiting >> m) & 1u) {
                    const uint64_t q = SM_U64(AT8(queue) + m);
                    len = (int32_t)(q >> 32) + 1;
                    pos = (int32_t)q;
                    if (serve) dl = SM_F64(AT8(head_dl) + m);
                    else {
                        if (lane == 0) SM_U64(AT8(queue) + m) = q + (1ull << 32);
                        __syncwarp();
                    }
                } else if (!serve) {
                    if (lane == 0) {
                        SM_U64(AT8(queue) + m) = (uint32_t)pos | (1ull << 32);
                        SM_F64(AT8(head_ts) + m) = ts;
                        SM_F64(AT8(head_dl) + m) = dl;
                    }
                    w.waiting |= 1ull << m;
                    __syncwarp();
                }
            }
            if (!serve) {
                if (++k >= k1) return;
                o = next;
                events = true;
                continue;
            }
        }
        serve_group(a, w, ts, m, g, pos, len, dl);
        if (!event) {
            if (++k >= k1) return;
            o = next;
            events = true;
        }
    }
}

template <int kPer>
__device__ __forceinline__ uint64_t replicas_of(const BatchArgs &a, const GroupWarp<kPer> &w, int32_t m)
{
    return SM_U64(AT8(served) + m);
}

// After the last arrival, :781-790.
template <int kPer>
__device__ inline void batch_drain(const BatchArgs &a, GroupWarp<kPer> &w)
{
    for (;;) {
        bool in[kPer];
        uint32_t any = 0;
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            in[h] = w.ev[h] == w.ev[h];
            any |= __ballot_sync(0xFFFFFFFFu, in[h]);
        }
        if (!any) break;
        double te;
        const int32_t g = event_take(a, w, in, te);
        const uint64_t models = SM_U64(AT8(serves) + g) & w.waiting;
        if (!models) continue;
        const int32_t m = models & (models - 1) ? earliest_head(a, w, g, models) : (int32_t)__ffsll((long long)models) - 1;
        if (m < 0) continue;
        const uint64_t q = SM_U64(AT8(queue) + m);
        serve_group(a, w, te, m, g, (int32_t)q, (int32_t)(q >> 32), SM_F64(AT8(head_dl) + m));
    }
    if (w.waiting) w.status |= MMS_STATUS_QUEUE_LEFT;
}

// A saved state's slots: rows 0 to kPer - 1 the groups' earliest events, then the extra ones,
// whose number is ev_n.
template <int kPer>
__device__ inline void state_save(const BatchArgs &a, const GroupWarp<kPer> &w, unsigned char *p)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const StateView v = state_view(a, p);
    __syncwarp();
    for (int t = lane; t < a.T; t += kLanes) v.clk[t] = SM_F64(AT8(clk) + t);
#pragma unroll
    for (int h = 0; h < kPer; ++h) v.ev[h * kLanes + lane] = (uint64_t)__double_as_longlong(w.ev[h]);
    for (uint32_t e = lane; e < w.extra_n; e += kLanes) {
        v.ev[kPer * kLanes + e] = (uint64_t)__double_as_longlong(SM_F64(AT8(extra) + e));
        v.ev_g[kPer * kLanes + e] = smem[AT1(extra_g) + e];
    }
    for (int m = lane; m < a.M; m += kLanes) {
        const bool some = (w.waiting >> m) & 1u;
        const uint64_t q = some ? SM_U64(AT8(queue) + m) : 0ull;
        v.qpos[m] = (int32_t)q;
        v.qlen[m] = (int32_t)(q >> 32);
    }
    if (lane == 0) *v.ev_n = w.extra_n;
    __syncwarp();
}

// The state under the warp's labels (what stands at label g is group labels[g]'s).
template <int kPer>
__device__ inline void state_load(const BatchArgs &a, GroupWarp<kPer> &w, unsigned char *p)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const StateView v = state_view(a, p);
    __syncwarp();
    for (int label = lane; label < a.G; label += kLanes) {
        const uint32_t from = SM_U32(AT4(info) + label), to = SM_U32(AT4(info) + smem[AT1(labels) + label]);
        for (uint32_t k = 0; k < ((from >> 8) & 0xFFu); ++k)
            SM_F64(AT8(clk) + (to & 0xFFu) + k) = v.clk[(from & 0xFFu) + k];
    }
    w.extra_n = *v.ev_n;
    for (uint32_t e = lane; e < w.extra_n; e += kLanes) {
        SM_F64(AT8(extra) + e) = __longlong_as_double((long long)v.ev[kPer * kLanes + e]);
        smem[AT1(extra_g) + e] = smem[AT1(labels) + v.ev_g[kPer * kLanes + e]];
    }
    // the label of groups lane and lane + 32
    int label[kPer];
#pragma unroll
    for (int h = 0; h < kPer; ++h) label[h] = lane + h * kLanes;
    for (int x = 0; x < a.G; ++x)
#pragma unroll
        for (int h = 0; h < kPer; ++h)
            if (smem[AT1(labels) + x] == lane + h * kLanes) label[h] = x;
    w.waiting = 0;
    for (int h = 0; h * kLanes < a.M; ++h) {
        const int m = lane + h * kLanes;
        const int32_t len = m < a.M ? v.qlen[m] : 0, pos = m < a.M ? v.qpos[m] : 0;
        if (len > 0) {
            SM_U64(AT8(queue) + m) = (uint32_t)pos | ((uint64_t)(uint32_t)len << 32);
            SM_F64(AT8(head_ts) + m) = a.pos_ts[pos];
            SM_F64(AT8(head_dl) + m) = a.pos_dl[pos];
        }
        w.waiting |= (uint64_t)__ballot_sync(0xFFFFFFFFu, len > 0) << (32 * h);
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        w.ev[h] = __longlong_as_double((long long)v.ev[label[h]]);
        const uint32_t cfg = SM_U32(AT4(info) + lane + h * kLanes), slot = cfg & 0xFFu, ns = (cfg >> 8) & 0xFFu;
        w.idle[h] = ns ? SM_F64(AT8(clk) + slot) : 0.0;
        w.last[h] = ns ? SM_F64(AT8(clk) + slot + ns - 1) : 0.0;
    }
}

// batch_equivalent above, of the state on chip and the saved one with its groups moved: what
// stands at label from[h] (per lane, of groups lane and lane + 32) there is this group's.
template <int kPer>
__device__ inline bool group_equivalent(const BatchArgs &a, const GroupWarp<kPer> &w, unsigned char *saved,
                                        double tau, const int (&from)[kPer])
{
    const int lane = threadIdx.x & (kLanes - 1);
    const StateView v = state_view(a, saved);
    __syncwarp();
    if (*v.ev_n != w.extra_n) return false;
    bool bad = false;
    for (int m = lane; m < a.M; m += kLanes) {
        const uint64_t q = (w.waiting >> m) & 1u ? SM_U64(AT8(queue) + m) : 0ull;
        bad |= q != ((uint32_t)v.qpos[m] | ((uint64_t)(uint32_t)v.qlen[m] << 32));
    }
    bool in[kPer];
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        bad |= v.ev[from[h]] != (uint64_t)__double_as_longlong(w.ev[h]);
        in[h] = w.ev[h] == w.ev[h];
    }
    if (__any_sync(0xFFFFFFFFu, bad)) return false;
    // theta: the earliest pending event (a group's other ones are behind its first) or tau
    double theta = tau;
    const uint64_t who = least_groups<kPer>(in, w.ev);
    if (who) {
        const int g = (int)__ffsll((long long)who) - 1;
        double t = w.ev[0];
        if constexpr (kPer == 2) t = g >= kLanes ? w.ev[1] : w.ev[0];
        t = __shfl_sync(0xFFFFFFFFu, t, g & (kLanes - 1));
        theta = t < tau ? t : tau;
    }
    double y[kPer];
    uint64_t differ = 0;
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const uint32_t cfg = SM_U32(AT4(info) + lane + h * kLanes), ns = (cfg >> 8) & 0xFFu;
        const uint32_t here = AT8(clk) + (cfg & 0xFFu), there = SM_U32(AT4(info) + from[h]) & 0xFFu;
        y[h] = 0.0;
        for (uint32_t k = 0; k < ns; ++k) {
            const double x = SM_F64(here + k);
            y[h] = v.clk[there + k];
            bad |= !(x == y[h] || (x < theta && y[h] < theta));
        }
        differ |= (uint64_t)__ballot_sync(0xFFFFFFFFu, y[h] != w.last[h]) << (32 * h);
    }
    if (__any_sync(0xFFFFFFFFu, bad)) return false;
    // the extra events, each as often in the one as in the other (not looked at under other labels)
    for (uint32_t e = 0; e < w.extra_n; ++e) {
        const double t = SM_F64(AT8(extra) + e);
        const uint32_t g = smem[AT1(extra_g) + e];
        int here = 0, there = 0;
        for (uint32_t base = 0; base < w.extra_n; base += kLanes) {
            const uint32_t x = base + lane;
            const bool is = x < w.extra_n;
            here += __popc(__ballot_sync(0xFFFFFFFFu, is && SM_F64(AT8(extra) + x) == t && smem[AT1(extra_g) + x] == g));
            there += __popc(__ballot_sync(0xFFFFFFFFu, is && __longlong_as_double((long long)v.ev[kPer * kLanes + x]) == t &&
                                                           v.ev_g[kPer * kLanes + x] == g));
        }
        if (here != there) return false;
    }
    // the order of the last-stage clocks
    if (!differ) return true;
    for (int m = 0; m < a.M; ++m) {
        const uint64_t groups = SM_U64(AT8(served) + m);
        if (!(groups & (groups - 1))) continue;
        for (uint64_t todo = groups & differ; todo; todo &= todo - 1) {
            const int u = (int)__ffsll((long long)todo) - 1;
            double xs = w.last[0], ys = y[0];
            if constexpr (kPer == 2)
                if (u >= kLanes) { xs = w.last[1]; ys = y[1]; }
            const double xu = __shfl_sync(0xFFFFFFFFu, xs, u & (kLanes - 1));
            const double yu = __shfl_sync(0xFFFFFFFFu, ys, u & (kLanes - 1));
#pragma unroll
            for (int h = 0; h < kPer; ++h)
                bad |= ((groups >> (lane + h * kLanes)) & 1u) &&
                       ((xu < w.last[h]) != (yu < y[h]) || (xu > w.last[h]) != (yu > y[h]));
        }
        if (__any_sync(0xFFFFFFFFu, bad)) return false;
    }
    return true;
}

template <int kPer>
__device__ inline bool batch_equivalent(const BatchArgs &a, const GroupWarp<kPer> &w, unsigned char *saved,
                                        double tau)
{
    int from[kPer];
#pragma unroll
    for (int h = 0; h < kPer; ++h) from[h] = (int)(threadIdx.x & (kLanes - 1)) + h * kLanes;
    return group_equivalent<kPer>(a, w, saved, tau, from);
}

// OTHER LABELS.  Groups with the same stages, column and models are interchangeable, and which of
// them is ahead depends on history long past: two that serve one model alone take turns, and
// a run that starts them the wrong way round never finds back (of 22 boundaries of 60 placements on
// 64 devices over 45 000 requests that failed, 20 were such pairs, and the chain walked half the trace of a
// placement because of one).  Such a run is the true one with the groups' roles exchanged, choice by choice, except where a
// group number decides, between replicas with equal last-stage clocks or events of one time
// (bursts of requests with one arrival time do that).  Mostly those are interchangeable and in the
// same state: then any can stand for any other, and the labels are exchanged, from there on, so that the
// run's choice is the true one's (`Swap`).  Others are noted (`tie`), and a run is not taken over
// under labels that move any of their class.  What a run counts, it counts for its labels; the chain kernel
// translates.
//
// Is the state on chip equivalent to the saved one under other labels?  Within a class they have to
// keep the order of the last-stage clocks, so both are sorted by it.  Out: per lane, to[h] = the group that
// label lane + 32 h of the saved state stands for.
template <int kPer>
__device__ inline bool other_labels(const BatchArgs &a, const GroupWarp<kPer> &w, unsigned char *saved,
                                    double tau, int (&to)[kPer])
{
    const int lane = threadIdx.x & (kLanes - 1);
    const StateView v = state_view(a, saved);
    if (!w.plain || w.extra_n || *v.ev_n) return false;
    uint64_t cls[kPer];                  // the groups interchangeable with this one, and itself
    double z[kPer];                      // its last-stage clock in the saved state
    uint32_t mine[kPer];
    uint64_t models[kPer];
    bool any = false;
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const uint32_t cfg = SM_U32(AT4(info) + lane + h * kLanes);
        mine[h] = cfg >> 8;
        models[h] = SM_U64(AT8(serves) + lane + h * kLanes);
        cls[h] = 0;
        z[h] = (cfg >> 8) & 0xFFu ? v.clk[(cfg & 0xFFu) + ((cfg >> 8) & 0xFFu) - 1] : 0.0;
    }
    for (int g = 0; g < a.G; ++g) {
        const uint32_t cfg = SM_U32(AT4(info) + g) >> 8;
        const uint64_t set = SM_U64(AT8(serves) + g);
#pragma unroll
        for (int h = 0; h < kPer; ++h)
            if (set && cfg == mine[h] && set == models[h]) cls[h] |= 1ull << g;
    }
#pragma unroll
    for (int h = 0; h < kPer; ++h) any |= (cls[h] & (cls[h] - 1)) != 0;
    if (!__any_sync(0xFFFFFFFFu, any)) return false;
    uint32_t rx[kPer], rz[kPer];         // ranks within the class, here and there
#pragma unroll
    for (int h = 0; h < kPer; ++h) { rx[h] = rz[h] = 0; to[h] = lane + h * kLanes; }
    const auto of = [&](const double (&x)[kPer], int g) {
        double t = x[0];
        if constexpr (kPer == 2) t = g >= kLanes ? x[1] : x[0];
        return __shfl_sync(0xFFFFFFFFu, t, g & (kLanes - 1));
    };
    for (int g = 0; g < a.G; ++g) {
        const double xg = of(w.last, g), zg = of(z, g);
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            const bool in = (cls[h] >> g) & 1u, before = g < lane + h * kLanes;
            rx[h] += in && (xg < w.last[h] || (xg == w.last[h] && before));
            rz[h] += in && (zg < z[h] || (zg == z[h] && before));
        }
    }
    int from[kPer];
#pragma unroll
    for (int h = 0; h < kPer; ++h) from[h] = lane + h * kLanes;
    for (int g = 0; g < a.G; ++g) {
        uint32_t x = rx[0], y = rz[0];
        if constexpr (kPer == 2)
            if (g >= kLanes) { x = rx[1]; y = rz[1]; }
        const uint32_t rxg = __shfl_sync(0xFFFFFFFFu, x, g & (kLanes - 1));
        const uint32_t rzg = __shfl_sync(0xFFFFFFFFu, y, g & (kLanes - 1));
#pragma unroll
        for (int h = 0; h < kPer; ++h)
            if ((cls[h] >> g) & 1u) {
                if (rxg == rz[h]) to[h] = g;
                if (rzg == rx[h]) from[h] = g;
            }
    }
    bool moves = false;
#pragma unroll
    for (int h = 0; h < kPer; ++h) moves |= to[h] != lane + h * kLanes;
    return __any_sync(0xFFFFFFFFu, moves) && group_equivalent<kPer>(a, w, saved, tau, from);
}

// The labels of the run at hand (u8[kGroupLimit] on chip): labels[g] is the group that label g stands for.
template <int kPer>
__device__ inline void labels_reset(const BatchArgs &a, const GroupWarp<kPer> &w)
{
    __syncwarp();
    for (int g = threadIdx.x & (kLanes - 1); g < kGroupLimit; g += kLanes) smem[AT1(labels) + g] = (uint8_t)g;
    __syncwarp();
}

template <int kPer>
__device__ inline void labels_set(const BatchArgs &a, const GroupWarp<kPer> &w, const int (&to)[kPer])
{
    __syncwarp();
#pragma unroll
    for (int h = 0; h < kPer; ++h)
        smem[AT1(labels) + (threadIdx.x & (kLanes - 1)) + h * kLanes] = (uint8_t)to[h];
    __syncwarp();
}

// The groups that the labels move.
template <int kPer>
__device__ inline uint64_t labels_moved(const BatchArgs &a, const GroupWarp<kPer> &w)
{
    uint64_t moved = 0;
    __syncwarp();
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const int g = (int)(threadIdx.x & (kLanes - 1)) + h * kLanes;
        moved |= (uint64_t)__ballot_sync(0xFFFFFFFFu, smem[AT1(labels) + g] != g) << (32 * h);
    }
    return moved;
}

// Labels behind `perm` (label -> label of the run before).
template <int kPer>
__device__ inline void labels_through(const BatchArgs &a, const GroupWarp<kPer> &w, const uint8_t *perm)
{
    int to[kPer];
    __syncwarp();
#pragma unroll
    for (int h = 0; h < kPer; ++h)
        to[h] = smem[AT1(labels) + perm[(threadIdx.x & (kLanes - 1)) + h * kLanes]];
    labels_set(a, w, to);
}

// All groups of the classes of `moved` ones.
template <int kPer>
__device__ inline uint64_t moved_class(const BatchArgs &a, const GroupWarp<kPer> &w, uint64_t moved)
{
    uint64_t all = moved;
    for (int g = 0; g < a.G && moved; ++g) {
        bool in = false;
        const uint32_t cfg = SM_U32(AT4(info) + g) >> 8;
        const uint64_t set = SM_U64(AT8(serves) + g);
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            const int x = (int)(threadIdx.x & (kLanes - 1)) + h * kLanes;
            in |= ((moved >> x) & 1u) && SM_U32(AT4(info) + x) >> 8 == cfg && SM_U64(AT8(serves) + x) == set;
        }
        if (__any_sync(0xFFFFFFFFu, in)) all |= 1ull << g;
    }
    return all;
}

}  // namespace mms
