// sim_window.cuh — one candidate per warp, a WINDOW of 32 requests at a time.
//
// The recurrence of one candidate (controller.py:579-622) is sequential only
// where requests meet: a request reads the clocks of the groups that serve its
// model and, if it is accepted, writes those of one of them.  Two requests
// whose models share no group do not see each other, and a request that is
// dropped changes nothing.  So a warp takes 32 consecutive requests, one per
// lane, and works through them in rounds: every request that is left is
// evaluated against the current clocks, and the outcome is FINAL for a lane
// when every earlier request it shares a group with is done or was found
// dropped, finally, in this round.  Final lanes store their clocks and leave.
// The first request left is always final, so a window takes at most 32 rounds;
// measured over the package's cases 8 to 12 where a cluster has about twenty
// groups, 20 to 27 with five groups (bursts of one model are a chain), fewer
// under overload, where most requests are dropped.
//
// What bounds it: the latency of a round (replica clocks, choice, stage clocks,
// max/add chain, two votes), not issue slots or memory.  It is the engine of
// everything that is short of candidates — small batches, where the chunks of
// each candidate are the parallelism, the repairs and the chain kernel.
#pragma once
#include "sim_chunk.cuh"

namespace mms {

constexpr int kWindowWarps = 4;        // warps of a window-kernel block (they share the table)
constexpr int kWindowBlocksPerSm = 3;
constexpr size_t kOrderBytes = 32;     // see window_groups
// Longest pipelines that window_groups serves.  Both ways cost about the same from four stages on
// (170 ns a request by groups, 145 ns in rounds, 4 groups of 4; 199 and 234 ns, 6 mixed ones); with
// eight the rounds win (22 mixed groups: 199 and 183 ns; a sweep of 48 overloaded traces: 86 and
// 62 ms), with one the groups (16 groups under overload: layers of a search 84 and 277 ms).
constexpr int kGroupDepth = 4;
constexpr int kWindowList = 1024;      // (group, model) pairs of a candidate kept on chip, at most

// Depth the on-chip tables are laid out for: the batch's deepest pipeline rounded up to a
// power of two, or 0 when it is deeper than 8 (tables as the caller gives them then).
__host__ __device__ inline int window_depth(int S) { return S <= 1 ? 1 : S <= 2 ? 2 : S <= 4 ? 4 : S <= 8 ? 8 : 0; }

// Shared memory of a window block: the latency table as doubles (when it is on
// chip), then per warp the clocks, a second state to compare with, the window's
// latencies, the candidate's group table and where its clock slots are.
//
// Pipelines are laid out RIGHT-ALIGNED at a fixed pitch of D stages, clocks and
// latencies alike: a group of fewer stages begins with virtual ones whose
// clock is in the past and whose latency is 0.0 (max(t, past) + 0.0 is t, exactly).  The
// chain then always runs over D stages and ends in the same register, and the
// stores need no test per stage: a round takes about a third fewer instructions than with
// a finish time picked by depth, and instructions are what a lone warp's round
// consists of (5.5 cycles each).
struct WindowLayout {
    size_t warp0, warp_bytes, clocks, old_state, last, ring, info, slot_at, cls, list, perm, labels, rank, orders, total;
};

__host__ __device__ inline size_t window_table_elems(int M, int C, int S, bool legacy)
{
    const int D = legacy ? 2 : window_depth(S);
    return (size_t)M * C * (D ? D : S) + 8;
}

__host__ __device__ inline WindowLayout window_layout(int T, int G, int S, int P, size_t table_elems)
{
    WindowLayout L;
    L.warp0 = (sizeof(double) * table_elems + 15) & ~(size_t)15;
    const size_t D = (size_t)window_depth(S);
    size_t clocks = (size_t)(T + kClockPad);
    if (D * (size_t)G + 1 > clocks) clocks = D * (size_t)G + 1;
    size_t off = 0;
    L.clocks = off;    off += sizeof(double) * clocks;
    L.old_state = off; off += sizeof(double) * (size_t)T;
    L.last = off;      off += sizeof(double) * (size_t)G;
    L.ring = off;      off += sizeof(double) * kLanes;
    off = (off + 15) & ~(size_t)15;
    L.orders = off;    off += kOrderBytes * kLanes;
    L.info = off;      off += sizeof(uint32_t) * (size_t)G;
    L.slot_at = off;   off += sizeof(uint16_t) * (size_t)T;
    off = (off + 3) & ~(size_t)3;
    L.cls = off;       off += sizeof(uint32_t) * (size_t)G;
    L.list = off;      off += P <= kWindowList ? sizeof(uint32_t) * (size_t)P : 0;
    L.perm = off;      off += (size_t)G;
    L.labels = off;    off += (size_t)G;
    L.rank = off;      off += 2 * (size_t)G;
    L.warp_bytes = (off + 15) & ~(size_t)15;
    L.total = L.warp0 + (size_t)kWindowWarps * L.warp_bytes;
    return L;
}

// A warp's view of its candidate; uniform over the warp except where noted.
struct Window {
    uint32_t clk, ring, info;                // f64, f64, u32 indices into shared memory
    RelabelScratch re;                       // re.z: the state to compare with
    uint32_t labels;                         // u8 index (G), see Labels
    uint32_t slot_at;                        // u16 index: where clock slot t is, behind clk
    bool lat_on_chip;
    const float *lat_gl;
    int64_t b;
    const uint4 *rows;
    const uint16_t *off;                     // the candidate's model_off
    uint32_t list;                           // u32 index of its replica list, if it is on chip
    uint32_t cls;                            // u32 index of its classes of twins
    uint32_t orders;                         // byte offset, see window_groups
    bool by_group;                           // window_groups can be used
    uint32_t column;                         // per lane: latency columns of groups lane and lane + 32
    int32_t depth;                           // pitch of the pipelines: 1, 2, 4 or 8; 0: slots as given
    const double *arrivals; const int32_t *model_ids; const float *slos;
    uint32_t pitch;
    int32_t last;                            // highest request index
    uint32_t status;                         // per lane
};

// All threads of the block, before any of them leaves.
template <bool kLegacy>
__device__ inline void window_stage_table(const KernelArgs &a)
{
    if (a.win_table_elems) {
        const int real = a.M * a.C;
        const int D = window_depth(a.S);
        if (kLegacy || D == 0 || *a.irregular || *a.unsorted != 0) {   // as given
            const int pitch = kLegacy ? 2 : D ? D : a.S;
            for (int i = threadIdx.x; i < a.win_table_elems; i += blockDim.x) {
                const int s = i % pitch;
                SM_F64(i) = i / pitch < real && s < a.S ? (double)__ldg(a.latency + (size_t)(i / pitch) * a.S + s) : 0.0;
            }
        } else {                                        // right-aligned
            for (int i = threadIdx.x; i < a.win_table_elems; i += blockDim.x) {
                const int row = i / D;
                int s = -1;
                if (row < real) s = i % D - (D - (int)a.column_stages[row % a.C]);
                SM_F64(i) = s >= 0 && s < a.S ? (double)__ldg(a.latency + (size_t)row * a.S + s) : 0.0;
            }
        }
    }
    __syncthreads();
}

// Clock slot t of the candidate.
#define WIN_CLOCK(w, t) SM_F64((w).clk + SM_U16((w).slot_at + (t)))

template <bool kLegacy, bool kTwins>
__device__ inline void window_setup(const KernelArgs &a, Window &w, int64_t b)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const WindowLayout L = window_layout(a.T, a.G, a.S, a.P, a.win_table_elems);
    const size_t base = L.warp0 + (size_t)(threadIdx.x / kLanes) * L.warp_bytes;
    w.clk = (uint32_t)((base + L.clocks) / sizeof(double));
    w.re.z = (uint32_t)((base + L.old_state) / sizeof(double));
    w.re.last = (uint32_t)((base + L.last) / sizeof(double));
    w.re.perm = (uint32_t)(base + L.perm);
    w.re.rank = (uint32_t)(base + L.rank);
    w.labels = (uint32_t)(base + L.labels);
    w.ring = (uint32_t)((base + L.ring) / sizeof(double));
    w.info = (uint32_t)((base + L.info) / sizeof(uint32_t));
    w.slot_at = (uint32_t)((base + L.slot_at) / sizeof(uint16_t));
    w.lat_on_chip = a.win_table_elems != 0;
    w.lat_gl = a.latency + (size_t)b * a.latency_stride;
    w.b = b;
    w.rows = reinterpret_cast<const uint4 *>(a.rep_rows) + row_index(a, b, 0);
    w.off = a.model_off + (size_t)b * (a.M + 1);
    w.list = (uint32_t)((base + L.list) / sizeof(uint32_t));
    w.cls = (uint32_t)((base + L.cls) / sizeof(uint32_t));
    w.orders = (uint32_t)(base + L.orders);
    const size_t tb = trace_base(a, b);
    w.arrivals = a.arrivals + tb; w.model_ids = a.model_ids + tb; w.slos = a.slos + tb;
    w.pitch = (uint32_t)a.trace_pitch;
    w.last = (int32_t)(a.N - 1);
    w.status = 0;
    __syncwarp();
    uint32_t depth = 1;
    for (int g = lane; g < a.G; g += kLanes) {
        const uint32_t info = a.group_info[(size_t)b * a.G + g];
        SM_U32(w.info + g) = info;
        if (kTwins) SM_U32(w.cls + g) = a.twin_class[(size_t)b * a.G + g];
        const uint32_t ns = (info >> 8) & 0xFFu;
        depth = ns > depth ? ns : depth;
    }
    depth = __reduce_max_sync(0xFFFFFFFFu, depth);
    // virtual stages are overwritten with arrival times, which are in the past for the requests
    // behind them only where the trace is sorted
    const bool plain = kLegacy || *a.irregular || *a.unsorted != 0 || window_depth(a.S) == 0;
    w.depth = plain ? 0 : window_depth((int)depth);
    if (a.P <= kWindowList)
        for (int e = lane; e < a.P; e += kLanes)
            SM_U32(w.list + e) = rep_to_last(a.model_rep[(size_t)b * a.P + e]);
    // lane g's groups, for window_groups
    w.by_group = w.depth > 0 && w.depth <= kGroupDepth &&
                 (a.G <= kLanes || (a.G <= 2 * kLanes && w.depth <= 2)) && w.lat_on_chip &&
                 a.P <= kWindowList && w.arrivals[0] >= 0.0;
    w.column = 0;
    for (int h = 0; h < 2; ++h) {
        const int g = lane + h * kLanes;
        const uint32_t col = g < a.G ? a.group_column[(size_t)b * a.G + g] : 0u;
        if (col < (uint32_t)a.C) w.column |= col << (16 * h);    // (a group without models has none)
    }
    const int cells = w.depth ? w.depth * a.G + 1 : a.T + kClockPad;
    for (int t = lane; t < cells; t += kLanes) SM_F64(w.clk + t) = w.depth ? -kInf : 0.0;
    for (int t = lane; t < a.T; t += kLanes) SM_U16(w.slot_at + t) = (uint16_t)(w.depth ? w.depth * a.G : t);   // no group's: a spare cell
    __syncwarp();
    if (w.depth) {
        for (int g = lane; g < a.G; g += kLanes) {
            const uint32_t info = SM_U32(w.info + g);
            const uint32_t slot = info & 0xFFu, ns = (info >> 8) & 0xFFu;
            for (uint32_t k = 0; k < ns; ++k) {
                const uint32_t at = (uint32_t)((g + 1) * w.depth) - ns + k;
                SM_U16(w.slot_at + slot + k) = (uint16_t)at;
                SM_F64(w.clk + at) = 0.0;
            }
        }
        __syncwarp();
    }
}

// Is the live state equivalent to a saved one (entries `pitch` apart), as it is (1) or under
// other labels (2: the permutation is in w.re.perm)?  0: it is not.
template <bool kTwins>
__device__ inline int window_equivalent(const KernelArgs &a, const Window &w, const double *saved,
                                        size_t pitch, double tau)
{
    const int lane = threadIdx.x & (kLanes - 1);
    __syncwarp();
    for (int t = lane; t < a.T; t += kLanes) SM_F64(w.re.z + t) = saved[(size_t)t * pitch];
    __syncwarp();
    const auto info = [&](int g) { return SM_U32(w.info + g); };
    const auto X = [&](uint32_t t) { return WIN_CLOCK(w, t); };
    const auto Z = [&](uint32_t t) { return SM_F64(w.re.z + t); };
    if (warp_equivalent(a.G, info, X, Z, tau)) return 1;
    if (!kTwins || !a.twins[w.b]) return 0;
    if (!warp_relabel(a.G, a.T, a.twin_class + (size_t)w.b * a.G, info, X, saved, pitch, w.re)) return 0;
    return warp_equivalent(a.G, info, X, Z, tau) ? 2 : 0;
}

// A request as its lane holds it.
struct WinRequest {
    double ts; float slo; int32_t m;
    uint4 r;                  // the first four replicas
    uint32_t lo, n;           // where the model's replica list begins; its length
};

__device__ __forceinline__ void window_element(const Window &w, int32_t block, double &ts,
                                               float &slo, int32_t &m)
{
    const int64_t want = (int64_t)block * kLanes + (threadIdx.x & (kLanes - 1));
    const size_t o = (size_t)(want < w.last ? want : (int64_t)w.last) * w.pitch;
    ts = __ldg(w.arrivals + o);
    slo = __ldg(w.slos + o);
    m = __ldg(w.model_ids + o);
}

__device__ __forceinline__ void window_rows(const KernelArgs &a, Window &w, WinRequest &q)
{
    if (q.m >= a.M) { w.status |= MMS_STATUS_BAD_INDEX; q.m = -1; }
    const size_t at = (size_t)(q.m < 0 ? a.M : q.m) * kLanes;
    q.r = __ldg(w.rows + at);
    q.lo = q.m < 0 ? 0u : w.off[q.m];
    q.n = q.m < 0 ? 0u : w.off[q.m + 1] - q.lo;
}

// Replica `at` of the candidate's list.
__device__ __forceinline__ uint32_t window_replica(const KernelArgs &a, const Window &w, uint32_t at)
{
    return a.P <= kWindowList ? SM_U32(w.list + at)
                              : rep_to_last(__ldg(a.model_rep + (size_t)w.b * a.P + at));
}

// The choices of `need` (lanes of the window) that the group number decided, between replicas
// whose last-stage clock is the lane's `best`: see warp_relabel.  `swap`: the twins of
// the picked one in its state, as a mask of their ranks in the class; `classes`: those of the
// others that matter (tie_matters), and its own with them.  Lanes of one model saw the same clocks: the warp looks at each model once, replica r in
// lane r.
struct WindowTies { uint64_t classes; uint32_t swap; };

template <int kDepth>
__device__ __noinline__ WindowTies window_ties(uint32_t need, uint32_t clk, uint32_t cls, uint32_t list,
                                               const uint32_t *list_gl, uint32_t lo, uint32_t n,
                                               int32_t m, uint32_t pick, double best, double ts)
{
    const int lane = threadIdx.x & (kLanes - 1);
    WindowTies mine;
    mine.classes = 0;
    mine.swap = 0;
    while (need) {
        const int k = __ffs((int)need) - 1;
        const int32_t mk = __shfl_sync(0xFFFFFFFFu, m, k);
        const uint32_t lok = __shfl_sync(0xFFFFFFFFu, lo, k), nk = __shfl_sync(0xFFFFFFFFu, n, k);
        const uint32_t pk = __shfl_sync(0xFFFFFFFFu, pick, k);
        const double bk = __shfl_sync(0xFFFFFFFFu, best, k), tk = __shfl_sync(0xFFFFFFFFu, ts, k);
        const bool alike_m = ((need >> lane) & 1u) && m == mk;
        need &= ~__ballot_sync(0xFFFFFFFFu, alike_m);
        auto last_at = [&](uint32_t e) {
            return clk + (kDepth > 0 ? rep_group(e) * (uint32_t)kDepth + (kDepth - 1) : rep_last(e));
        };
        const uint32_t own = SM_U32(cls + rep_group(pk));
        uint32_t swap = 0;
        uint64_t classes = 0;
        for (uint32_t r = lane; r < nk; r += kLanes) {
            const uint32_t e = list_gl ? rep_to_last(__ldg(list_gl + lok + r)) : SM_U32(list + lok + r);
            if (!(SM_F64(last_at(e)) == bk)) continue;
            const uint32_t other = SM_U32(cls + rep_group(e));
            bool same = class_first(other) == class_first(own) && class_rank(other) < 32;
            for (uint32_t s = 1; s < rep_stages(pk) && same; ++s) {
                const double x = SM_F64(last_at(pk) - s), y = SM_F64(last_at(e) - s);
                same = x == y || (x < tk && y < tk);
            }
            if (same) swap |= 1u << class_rank(other);
            else if (tie_matters(own, other)) classes |= class_bit(own) | class_bit(other);
        }
        swap = __reduce_or_sync(0xFFFFFFFFu, swap);
        const uint32_t c0 = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)classes);
        const uint32_t c1 = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)(classes >> 32));
        if (alike_m) {
            mine.swap = (swap & (swap - 1)) ? swap : 0u;      // more than the picked one
            mine.classes = ((uint64_t)c1 << 32) | c0;
        }
    }
    __syncwarp();
    return mine;
}

// The requests `todo` of the window (lanes), one after the other, with a GROUP per lane: lane g
// keeps the clocks of group g in registers and works out, for every request, when group g would
// finish it; the group whose last-stage clock is smallest among the model's replicas is found
// by the warp (clocks are not negative — neither the first arrival nor a latency is, see by_group
// and kIrregularLatency — so doubles are compared as integers, high word first), and its lane takes the request.  A request costs the same whatever the number of
// replicas and whoever else is waiting, and nothing of it passes through shared memory: the
// orders — arrival time, SLO, the model's groups as a mask, its latency row — are laid out there
// beforehand.  For candidates of up to 32 groups, or 64 in pipelines of one or two stages (two
// groups to a lane), and pipelines of up to kGroupDepth stages.
//
// Out: fin, rec, tie, swap of the requests in their lanes, as window_rounds leaves them.
struct __align__(16) WindowOrder {
    double ts, slo;           // slo: then the finish time
    uint64_t groups;
    uint32_t row, rec;        // rec: the decision record, when it is done
};
static_assert(sizeof(WindowOrder) == kOrderBytes, "order size");

template <int kDepth, int kPer, bool kTwins>
__device__ __forceinline__ void window_groups(const KernelArgs &a, const Window &w, uint32_t todo,
                                              double &fin, uint32_t &rec, uint64_t &tie,
                                              uint32_t &swap)
{
    const int lane = threadIdx.x & (kLanes - 1);
    if (!todo) return;
    WindowOrder *orders = reinterpret_cast<WindowOrder *>(smem + w.orders);
    const uint32_t D = (uint32_t)window_depth(a.S);
    const uint32_t yes = a.dec_wide ? 0x8000u : 0x80u;
    const uint32_t done = todo;
    // lane g has groups g and, with kPer == 2, g + 32
    double c[kPer][kDepth], l[kPer][kDepth];
    uint32_t ck[kPer], lat[kPer];
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const int g = lane + h * kLanes;
        ck[h] = w.clk + (uint32_t)(g < a.G ? g : 0) * kDepth;
        lat[h] = ((w.column >> (16 * h)) & 0xFFFFu) * D + (D - kDepth);
#pragma unroll
        for (int s = 0; s < kDepth; ++s) c[h][s] = SM_F64(ck[h] + s);
    }
    // the order at hand and its latencies, the order behind it
    int k = __ffs((int)todo) - 1;
    todo &= todo - 1;
    double ts = orders[k].ts, slo = orders[k].slo;
    uint64_t groups = orders[k].groups;
    uint32_t row = orders[k].row;
#pragma unroll
    for (int h = 0; h < kPer; ++h)
#pragma unroll
        for (int s = 0; s < kDepth; ++s) l[h][s] = SM_F64(row + lat[h] + s);
    for (;;) {
        const int k1 = todo ? __ffs((int)todo) - 1 : k;
        const double ts1 = orders[k1].ts, slo1 = orders[k1].slo;
        const uint64_t groups1 = orders[k1].groups;
        const uint32_t row1 = orders[k1].row;
        // :605-613 what this lane's groups would make of the request
        double t[kPer][kDepth], f[kPer];
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            double cur = ts;
#pragma unroll
            for (int s = 0; s < kDepth; ++s) {
                cur = tmax(cur, c[h][s]) + l[h][s];
                t[h][s] = cur;
            }
            f[h] = cur + kOverhead;
        }
        // :589-598 the first group with the smallest last-stage clock: `win` are the groups that
        // have it
        uint32_t win[kPer];
#pragma unroll
        for (int h = 0; h < kPer; ++h) win[h] = (uint32_t)(groups >> (32 * h));
        auto several = [&]() {
            uint32_t any = 0;
            int n = 0;
#pragma unroll
            for (int h = 0; h < kPer; ++h) { any |= win[h] & (win[h] - 1); n += win[h] != 0; }
            return any != 0 || n > 1;
        };
        if (several()) {
            uint32_t hi[kPer], low[kPer], least = 0xFFFFFFFFu;
#pragma unroll
            for (int h = 0; h < kPer; ++h) {
                const uint64_t key = (uint64_t)__double_as_longlong(c[h][kDepth - 1]);
                hi[h] = (win[h] >> lane) & 1u ? (uint32_t)(key >> 32) : 0xFFFFFFFFu;
                low[h] = (uint32_t)key;
                least = hi[h] < least ? hi[h] : least;
            }
            least = __reduce_min_sync(0xFFFFFFFFu, least);
#pragma unroll
            for (int h = 0; h < kPer; ++h)
                win[h] &= __ballot_sync(0xFFFFFFFFu, hi[h] == least);
            if (several()) {
                uint32_t low_least = 0xFFFFFFFFu;
#pragma unroll
                for (int h = 0; h < kPer; ++h) {
                    low[h] = (win[h] >> lane) & 1u ? low[h] : 0xFFFFFFFFu;
                    low_least = low[h] < low_least ? low[h] : low_least;
                }
                low_least = __reduce_min_sync(0xFFFFFFFFu, low_least);
#pragma unroll
                for (int h = 0; h < kPer; ++h)
                    win[h] &= __ballot_sync(0xFFFFFFFFu, low[h] == low_least);
                if (kTwins && several()) {      // the group number decides, see warp_relabel
                    const int ph = win[0] ? 0 : kPer - 1, p = __ffs((int)win[ph]) - 1;
                    const uint32_t picked = SM_U32(w.cls + p + ph * kLanes);
                    uint32_t alike = 0;
#pragma unroll
                    for (int h = 0; h < kPer; ++h) {
                        const int g = lane + h * kLanes;
                        const uint32_t own = g < a.G ? SM_U32(w.cls + g) : 0u;
                        bool same = class_first(own) == class_first(picked) && class_rank(own) < 32;
#pragma unroll
                        for (int s = 0; s + 1 < kDepth; ++s) {
                            const double x = __shfl_sync(0xFFFFFFFFu, kPer == 2 && ph ? c[kPer - 1][s] : c[0][s], p);
                            same = same && (x == c[h][s] || (x < ts && c[h][s] < ts));
                        }
                        const bool in = (win[h] >> lane) & 1u;
                        if (in && same) alike |= 1u << class_rank(own);
                        if (in && !same && tie_matters(picked, own)) tie |= class_bit(own) | class_bit(picked);
                    }
                    alike = __reduce_or_sync(0xFFFFFFFFu, alike);
                    if (lane == k) swap = (alike & (alike - 1)) ? alike : 0u;
                }
            }
        }
        const int wh = kPer == 1 || win[0] ? 0 : kPer - 1;
        const bool winner = lane == __ffs((int)win[wh]) - 1;
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            const bool mine = winner && wh == h;
            const bool found = c[h][kDepth - 1] < kInf;
            const bool accept = mine && found && f[h] - ts <= slo;
#pragma unroll
            for (int s = 0; s < kDepth; ++s) {
                c[h][s] = accept ? t[h][s] : c[h][s];
                l[h][s] = SM_F64(row1 + lat[h] + s);
            }
            if (mine) {
                orders[k].slo = accept ? f[h] : ts;
                orders[k].rec = found ? (uint32_t)(lane + h * kLanes + 1) | (accept ? yes : 0u) : 0u;
            }
        }
        if (!todo) break;
        todo &= todo - 1;
        k = k1; ts = ts1; slo = slo1; groups = groups1; row = row1;
    }
#pragma unroll
    for (int h = 0; h < kPer; ++h)
#pragma unroll
        for (int s = 0; s < kDepth; ++s)
            if (lane + h * kLanes < a.G) SM_F64(ck[h] + s) = c[h][s];
    __syncwarp();
    if ((done >> lane) & 1u) {
        fin = orders[lane].slo;
        rec = orders[lane].rec;
    }
}

// Executes the requests of `active` (lanes of the window), in order of their
// lane number as far as they depend on one another.  Out: fin (finish time, or
// the arrival time of a request that was not accepted) and the decision record,
// per lane.  kDepth: pitch of the pipelines (1, 2, 4, 8), 0 = slots and table as given.
// kTwins: the candidate has interchangeable groups, choices that the group number decides are
// noted (tie, swap); a variant of its own, because the rounds are short and every instruction
// in them counts.
template <bool kLegacy, int kDepth, bool kTwins>
__device__ __forceinline__ void window_rounds(const KernelArgs &a, const Window &w,
                                              const WinRequest &q, uint32_t conf, bool serves,
                                              uint32_t active, double &fin, uint32_t &rec, uint64_t &tie,
                                              uint32_t &swap)
{
    constexpr int kRegs = kDepth > 0 ? kDepth : 1;
    const int lane = threadIdx.x & (kLanes - 1);
    const uint32_t e0 = q.r.x, e1 = q.r.y, e2 = q.r.z, e3 = q.r.w;
    const double ts = q.ts, slo = (double)q.slo;
    const bool in = (active >> lane) & 1u;
    const uint32_t yes = a.dec_wide ? 0x8000u : 0x80u;
    if (in) { fin = ts; rec = 0; swap = 0; }
    uint32_t undone = __ballot_sync(0xFFFFFFFFu, in && serves);
    // what the window's requests need at most (uniform)
    const bool four = __any_sync(0xFFFFFFFFu, in && e2 < kMoreReplicas);
    const uint32_t most = four ? __reduce_max_sync(0xFFFFFFFFu, in && serves ? q.n : 0u) : 0u;
    // f64 index of a replica's last-stage clock
    auto last_at = [&](uint32_t e) {
        return w.clk + (kDepth > 0 ? rep_group(e) * (uint32_t)kRegs + (kRegs - 1) : rep_last(e));
    };
    // latency row of the request's model in column c
    const uint32_t mrow = (uint32_t)(q.m < 0 ? 0 : q.m) * a.C;
    const uint32_t D = kLegacy ? 2u : (uint32_t)window_depth(a.S);
    const uint32_t row_pitch = w.lat_on_chip && D ? D : (uint32_t)a.S;
    double l[kRegs];
    auto latencies = [&](uint32_t e) {
        const uint32_t row = (mrow + rep_column(e)) * row_pitch;
        if (w.lat_on_chip) {
#pragma unroll
            for (int s = 0; s < kRegs; ++s) l[s] = SM_F64(row + D - kRegs + s);
        } else {
            const int skip = kRegs - (int)rep_stages(e);
#pragma unroll
            for (int s = 0; s < kRegs; ++s)
                l[s] = s >= skip ? (double)__ldg(w.lat_gl + row + (s - skip)) : 0.0;
        }
    };
    // latencies that do not depend on the choice are read once, before the rounds
    bool one_column = true;
    if constexpr (kDepth > 0) {
        const uint32_t col = e0 >> 24;
        one_column = !__any_sync(0xFFFFFFFFu,
                                 in && serves && ((e1 < kMoreReplicas && e1 >> 24 != col) ||
                                                  (e2 < kMoreReplicas && e2 >> 24 != col) ||
                                                  (e3 < kMoreReplicas && e3 >> 24 != col)));
        for (uint32_t r = 4; r < most && one_column; ++r)
            one_column = !__any_sync(0xFFFFFFFFu, in && serves && r < q.n &&
                                                      window_replica(a, w, q.lo + r) >> 24 != col);
        latencies(e0 < kMoreReplicas ? e0 : 0x00010000u);
    }
    while (undone) {
        const bool mine = (undone >> lane) & 1u;
        // :589-598 replica whose last-stage clock is strictly smallest
        double best = kInf;
        uint32_t pick = 0x00010000u;          // group 0, slot 0, one stage, column 0
        {
            const double c0 = SM_F64(last_at(e0 < kMoreReplicas ? e0 : pick));
            if (e0 < kMoreReplicas && c0 < best) { best = c0; pick = e0; }
        }
        bool tied = false;                    // the group number decided, see warp_relabel
        auto consider = [&](uint32_t e) {
            const bool is = e < kMoreReplicas;
            const double c = SM_F64(last_at(is ? e : 0x00010000u));
            if (kTwins && is && c == best && e != pick) tied = true;
            if (is && c < best) { best = c; pick = e; tied = false; }
        };
        consider(e1);
        if (four) { consider(e2); consider(e3); }
        for (uint32_t r = 4; r < most; r += 4) {
            uint32_t e[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                e[k] = serves && r + k < q.n ? window_replica(a, w, q.lo + r + k) : kNoReplica;
#pragma unroll
            for (int k = 0; k < 4; ++k) consider(e[k]);
        }
        const bool found = best < kInf;
        double t[kRegs], f;
        uint32_t ck, row = 0, ns = 1;
        if constexpr (kDepth > 0) {
            ck = w.clk + rep_group(pick) * (uint32_t)kRegs;
            if (!one_column) latencies(pick);
            double cur = ts;
#pragma unroll
            for (int s = 0; s < kRegs; ++s) t[s] = SM_F64(ck + s);
#pragma unroll
            for (int s = 0; s < kRegs; ++s) {                // :605-608
                cur = tmax(cur, t[s]) + l[s];
                t[s] = cur;
            }
            f = cur + kOverhead;                             // :610
        } else {
            row = (mrow + rep_column(pick)) * row_pitch;
            auto lat = [&](uint32_t s) {
                return w.lat_on_chip ? SM_F64(row + s) : (double)__ldg(w.lat_gl + row + s);
            };
            if constexpr (kLegacy) {
                // :543-544 one clock per group; latency row = {sum, max}
                ck = w.clk + rep_last(pick);
                const double start = tmax(SM_F64(ck), ts);
                f = start + lat(0) + kOverhead;
                t[0] = start + lat(1);
            } else {
                ns = rep_stages(pick);
                ck = w.clk + rep_last(pick) + 1 - ns;
                double cur = ts;
                for (uint32_t s = 0; s < ns; ++s) cur = tmax(cur, SM_F64(ck + s)) + lat(s);
                f = cur + kOverhead;
            }
        }
        const bool accept = mine && found && f - ts <= slo;     // :613
        // which outcomes are final: no earlier unfinished request of a shared group was
        // accepted just now, or is itself not final
        const uint32_t accepted = __ballot_sync(0xFFFFFFFFu, accept);
        const uint32_t before = conf & undone;
        // ("Not final" spreads from request to request: two votes, and where the second one still
        // adds some, everything from the first of those on waits for the next round.)
        const uint32_t first = __ballot_sync(0xFFFFFFFFu, mine && (before & accepted));
        uint32_t open = __ballot_sync(0xFFFFFFFFu, mine && (before & (accepted | first)));
        const uint32_t late = open & ~first;
        open |= late ? ~((late & (0u - late)) - 1u) & undone : 0u;
        const bool final = mine && !((open >> lane) & 1u);
        const bool store = final && accept;
        if constexpr (kTwins) {
            const uint32_t need = __ballot_sync(0xFFFFFFFFu, final && tied);
            if (need) {
                const WindowTies ties = window_ties<kLegacy ? 0 : kDepth>(
                    need, w.clk, w.cls, w.list,
                    a.P <= kWindowList ? nullptr : a.model_rep + (size_t)w.b * a.P, q.lo, q.n, q.m, pick,
                    best, ts);
                if (final && tied) {
                    tie |= ties.classes;
                    swap = ties.swap;
                }
            }
        }
        if constexpr (kLegacy || kDepth > 0) {
#pragma unroll
            for (int s = 0; s < kRegs; ++s)
                if (store) SM_F64(ck + s) = t[s];
        } else if (store) {                                  // the same chain again, stored
            double cur = ts;
            for (uint32_t s = 0; s < ns; ++s) {
                cur = tmax(cur, SM_F64(ck + s)) +
                      (w.lat_on_chip ? SM_F64(row + s) : (double)__ldg(w.lat_gl + row + s));
                SM_F64(ck + s) = cur;
            }
        }
        fin = store ? f : fin;
        rec = final ? (found ? (rep_group(pick) + 1u) | (accept ? yes : 0u) : 0u) : rec;
        undone &= open;
        __syncwarp();                // the stores, before the next round's loads
    }
}

// Simulates requests of the warp's candidate by windows, in one of two ways.  The windows
// are aligned to 32 requests; one that a segment's end or the run-in's end falls
// into is worked through in two parts.
//
//   speculative (walk == kNoWalk): chunk j from idle clocks at `begin`, as run_chunk
//       does it for 32 candidates a warp.
//   walk: the warp's clocks hold the state at `begin`, the first request of segment
//       q_begin of chunk j.  The stored run is replaced segment by segment until what is stored
//       can take over: after a segment inside a chunk the state is compared with the one
//       the stored run had there, before a chunk with the one the stored run of that chunk
//       started from — as they are, or under other labels (warp_relabel; the permutation is then
//       noted in front of the segment the stored run takes over from).  A walk also stops,
//       without that, before a chunk that is on this round's work list (kWalkRound: another warp
//       is at work there) and at the end of the trace.  Comparing is optional: while it fails it
//       is tried less and less often (a group that is busy for thousands of requests keeps its
//       state different all along).
// Returns the first segment the walk did not run.
enum WalkMode { kNoWalk = 0, kWalkRound = 1, kWalkChain = 2 };
constexpr int32_t kMaxPause = 1024;    // requests between two comparisons, at most

//
// kTwins: stored runs may be compared under other labels.  kLog: choices that the group number
// decides are noted (tie, swap_mask) for those who compare later.
template <bool kLegacy, int kDepth, bool kTwins, bool kLog>
__device__ inline int32_t window_run_depth(const KernelArgs &a, Window &w, WalkMode walk, int32_t j,
                                           int32_t begin, bool snapshots, int32_t q_begin)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const int64_t b = w.b;
    const size_t B = (size_t)a.B;
    int32_t q = q_begin;
    int32_t q1 = (j + 1) * a.seg_per_chunk < a.NS ? (j + 1) * a.seg_per_chunk : a.NS;
    int32_t pause = 0, next_pause = 0;         // segments to skip comparing; and after the next failure
    const int32_t max_pause = kMaxPause / a.seg_len - 1;
    uint64_t tie = 0;
    int32_t leaf = seg_leaf(a, q);
    int32_t seg_stop = seg_leaf(a, q + 1);
    const int32_t first = leaf < a.num_leaves ? a.leaf_start[leaf] : (int32_t)a.N;
    int32_t leaf_end = leaf < a.num_leaves ? a.leaf_start[leaf + 1] : (int32_t)a.N;
    int32_t seg_end_i = seg_stop < a.num_leaves ? a.leaf_start[seg_stop] : (int32_t)a.N;
    bool record = begin >= first;
    int32_t stop = record ? seg_end_i : first;     // where this stretch ends
    double part = 0.0;                             // lanes 0-7: partial sum (lane) of the leaf

    // requests in flight: the window at work, the next one with its rows, the one behind it
    int32_t block = begin >> 5;
    WinRequest cur, nxt;
    double ts2; float slo2; int32_t m2;
    window_element(w, block, nxt.ts, nxt.slo, nxt.m);
    window_element(w, block + 1, ts2, slo2, m2);
    window_rows(a, w, nxt);
    int32_t i = begin;
    uint32_t conf = 0;
    bool serves = false;
    double fin = 0.0;
    uint32_t rec = 0, swap = 0;
    int32_t swap_n = 0;                            // entries of segment q's list of swaps
    int32_t decoded = -1;
    // a stretch that is empty (no run-in, or an empty segment) falls straight through
    for (;;) {
        while (i < stop) {
            if (decoded != (i >> 5)) {
                // ---- the next window: its rows have arrived; fetch for the two behind it --
                cur = nxt;
                nxt.ts = ts2; nxt.slo = slo2; nxt.m = m2;
                window_rows(a, w, nxt);
                decoded = i >> 5;
                window_element(w, decoded + 2, ts2, slo2, m2);
                // groups of the request's replicas, folded to 64 bits (a false clash only
                // costs a round)
                uint64_t groups = 0;
                const uint32_t e[4] = {cur.r.x, cur.r.y, cur.r.z, cur.r.w};
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (e[k] < kMoreReplicas) groups |= 1ull << (rep_group(e[k]) & 63u);
                if (groups)
                    for (uint32_t r = 4; r < cur.n; ++r)
                        groups |= 1ull << (rep_group(window_replica(a, w, cur.lo + r)) & 63u);
                serves = groups != 0;
                if (kDepth > 0 && w.by_group) {
                    WindowOrder *order = reinterpret_cast<WindowOrder *>(smem + w.orders) + lane;
                    __syncwarp();
                    order->ts = cur.ts;
                    order->slo = (double)cur.slo;
                    order->groups = groups;
                    order->row = (uint32_t)(cur.m < 0 ? 0 : cur.m) * a.C * (uint32_t)window_depth(a.S);
                }
                conf = 0;
                auto clashes = [&](uint32_t half) {      // over the groups that occur in the window
                    for (uint32_t occur = __reduce_or_sync(0xFFFFFFFFu, half); occur; occur &= occur - 1) {
                        const bool has = half & (occur & (0u - occur));
                        const uint32_t with = __ballot_sync(0xFFFFFFFFu, has);
                        if (has) conf |= with;
                    }
                };
                if (!(kDepth > 0 && w.by_group)) clashes((uint32_t)groups);
                if (a.G > 32 && !(kDepth > 0 && w.by_group)) clashes((uint32_t)(groups >> 32));
                conf &= (1u << lane) - 1u;
            }
            const int32_t base = decoded << 5;
            const int32_t to = stop < base + kLanes ? stop : base + kLanes;
            const uint32_t upto = to - base >= kLanes ? 0xFFFFFFFFu : (1u << (to - base)) - 1u;
            const uint32_t active = upto & ~((1u << (i - base)) - 1u);
            bool rounds = true;
            if constexpr (kDepth > 0 && kDepth <= kGroupDepth) {
                if (w.by_group) {
                    rounds = false;
                    const bool in = (active >> lane) & 1u;
                    if (in) { fin = cur.ts; rec = 0; swap = 0; }
                    __syncwarp();
                    const uint32_t todo = __ballot_sync(0xFFFFFFFFu, in && serves);
                    if (kDepth > 2 || a.G <= kLanes)
                        window_groups<kDepth, 1, kLog>(a, w, todo, fin, rec, tie, swap);
                    else if constexpr (kDepth <= 2)
                        window_groups<kDepth, 2, kLog>(a, w, todo, fin, rec, tie, swap);
                }
            }
            if (rounds)
                window_rounds<kLegacy, kDepth, kLog>(a, w, cur, conf, serves, active, fin, rec, tie, swap);
            if (record) {
                const bool in = (active >> lane) & 1u;
                const int32_t at = base + lane;
                // decision records: see sim_step
                if (a.dec_wide) {
                    if (in)
                        static_cast<uint16_t *>(a.decisions)
                            [(((size_t)(at >> 2) * a.dec_pitch) + b) * 4 + (at & 3)] = (uint16_t)rec;
                } else {
                    uint32_t word = (in ? rec : 0u) << (8 * (lane & 3));
                    word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1);
                    word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2);
                    if (in && (lane & 3) == 0)
                        static_cast<uint32_t *>(a.decisions)[(size_t)(at >> 2) * a.dec_pitch + b] = word;
                }
                if constexpr (kLog) {        // which choices the group number decided
                    const bool some = in && swap && rec;
                    const uint32_t who = __ballot_sync(0xFFFFFFFFu, some);
                    if (who) {
                        const int32_t k = swap_n + __popc(who & ((1u << lane) - 1u));
                        if (some && k < a.swap_cap) {
                            const size_t cell = ((size_t)q * a.swap_cap + k) * B + b;
                            a.swap_mask[cell] = swap;
                            a.swap_at[cell] = (uint16_t)(at - a.leaf_start[seg_leaf(a, q)]);
                        } else if (some) {
                            tie |= class_bit(SM_U32(w.cls + (rec & (a.dec_wide ? 0x7FFFu : 0x7Fu)) - 1u));
                        }
                        swap_n += __popc(who);
                    }
                }
                if (a.finish && in) {
                    a.finish[(size_t)b * a.N + at] = fin;
                    a.good[(size_t)b * a.N + at] = rec & (a.dec_wide ? 0x8000u : 0x80u) ? 1 : 0;
                }
                // latency sums: request k of a leaf goes to partial sum k mod 8, as numpy's
                // pairwise sum does; leaves start at multiples of 8
                SM_F64(w.ring + lane) = fin - cur.ts;
                __syncwarp();
                auto leaf_done = [&](int32_t tail) {     // [tail, leaf_end): behind the last full eight
                    double r = part + __shfl_xor_sync(0xFFFFFFFFu, part, 1);
                    r = r + __shfl_xor_sync(0xFFFFFFFFu, r, 2);
                    r = r + __shfl_xor_sync(0xFFFFFFFFu, r, 4);
                    for (int32_t x = tail; x < leaf_end; ++x) r += SM_F64(w.ring + (x - base));
                    if (lane == 0) a.leaf_sums[(size_t)leaf * B + b] = r;
                    part = 0.0;
                    ++leaf;
                    if (leaf < a.num_leaves) leaf_end = a.leaf_start[leaf + 1];
                };
                if (i == base && to == base + kLanes && to <= leaf_end) {
                    const uint32_t at8 = w.ring + (lane & 7);
                    part += SM_F64(at8);
                    part += SM_F64(at8 + 8);
                    part += SM_F64(at8 + 16);
                    part += SM_F64(at8 + 24);
                    if (to == leaf_end) leaf_done(leaf_end);
                } else {
                    for (int32_t o = i; o < to; o += 8) {
                        if (o + 8 <= leaf_end) part += SM_F64(w.ring + (o - base) + (lane & 7));
                        if (o + 8 >= leaf_end) leaf_done(o + 8 > leaf_end ? o : leaf_end);
                    }
                }
                __syncwarp();
            }
            i = to;
        }
        if (!record) {
            if (snapshots)             // the state this speculative chunk starts from
                for (int t = lane; t < a.T; t += kLanes)
                    a.chunk_start[((size_t)j * a.T + t) * B + b] = WIN_CLOCK(w, t);
            record = true;
            tie = 0;
            stop = seg_end_i;
            continue;
        }
        // ---- segment q is complete --------------------------------------------------
        if (snapshots) {
            const bool compare = walk && pause == 0 && i < a.N;
            if (pause > 0) --pause;
            if constexpr (kLog) {
                const uint32_t lo = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)tie);
                const uint32_t hi = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)(tie >> 32));
                tie = 0;
                if (lane == 0) {
                    a.tie[(size_t)q * B + b] = ((uint64_t)hi << 32) | lo;
                    a.swap_count[(size_t)q * B + b] = (uint8_t)(swap_n < a.swap_cap ? swap_n : a.swap_cap);
                }
                swap_n = 0;
            }
            const bool inside = q + 1 < q1;
            int same = 0;
            // a stored run under other labels can only take over where no choice in the rest of
            // the chunk was decided by a group number between different states
            auto usable = [&](int how, int32_t from, int32_t to_seg) {
                if (how != 2) return how;
                const uint32_t *cls = a.twin_class + (size_t)b * a.G;
                const uint64_t moved = moved_classes(cls, a.G, [&](int g) { return smem[w.re.perm + g]; });
                bool some = false;
                for (int32_t s = from + lane; s < to_seg; s += kLanes)
                    some |= (a.tie[(size_t)s * B + b] & moved) != 0;
                return __any_sync(0xFFFFFFFFu, some) ? 0 : how;
            };
            if (compare && inside) {
                same = window_equivalent<kTwins>(a, w, a.seg_end + (size_t)q * a.T * B + b, B, arrival_at(a, b, i));
                same = usable(same, q + 1, q1);
            }
            __syncwarp();              // (read above, written below)
            for (int t = lane; t < a.T; t += kLanes)
                a.seg_end[((size_t)q * a.T + t) * B + b] = WIN_CLOCK(w, t);
            ++q;
            if (walk && !inside && q < a.NS) {
                // ---- the next chunk -------------------------------------------------------
                const size_t cell = (size_t)(j + 1) * B + b;
                if (walk == kWalkRound && a.stamp[cell] == (uint8_t)(a.round + 1)) return q;
                const int32_t q2 = q1 + a.seg_per_chunk < a.NS ? q1 + a.seg_per_chunk : a.NS;
                if (compare) {
                    same = window_equivalent<kTwins>(a, w, a.chunk_start + (size_t)(j + 1) * a.T * B + b, B,
                                             arrival_at(a, b, i));
                    same = usable(same, q1, q2);
                }
                __syncwarp();
                if (!same) {
                    ++j;
                    q1 = q2;
                    for (int t = lane; t < a.T; t += kLanes)
                        a.chunk_start[((size_t)j * a.T + t) * B + b] = WIN_CLOCK(w, t);
                    if (lane == 0) {
                        a.stamp[cell] = (uint8_t)(a.round + 1);
                        a.link[cell] = 1;
                        if (a.resimulated) atomicAdd(&a.resimulated[b], 1);
                    }
                } else if (lane == 0) {
                    a.link[cell] = 1;
                    a.rel[(size_t)q * B + b] = 0;    // replaced below, if at all
                }
            }
            if (same) {                // what is stored takes over from segment q
                const size_t cell = (size_t)q * B + b;
                if (same == 2) {
                    // inside a chunk the labels may change in front of segment q already
                    const bool had = a.rel[cell] != 0;
                    __syncwarp();
                    uint8_t *perm = a.perm + cell * a.G;
                    for (int g = lane; g < a.G; g += kLanes)
                        perm[g] = smem[w.re.perm + (had && inside ? perm[g] : (uint8_t)g)];
                    if (lane == 0) {
                        a.rel[cell] = kRelOther;
                        a.relabelled[b] = 1;
                    }
                }
                __syncwarp();
                return q;
            }
            if (compare) {
                pause = next_pause;
                next_pause = 2 * next_pause + 1 < max_pause ? 2 * next_pause + 1 : max_pause;
            }
            if (walk && lane == 0 && q < a.NS) a.rel[(size_t)q * B + b] = 0;
        } else {
            ++q;
        }
        if (q >= (walk ? a.NS : q1)) return q;
        seg_stop = seg_leaf(a, q + 1);
        seg_end_i = seg_stop < a.num_leaves ? a.leaf_start[seg_stop] : (int32_t)a.N;
        stop = seg_end_i;
    }
}

template <bool kLegacy, bool kTwins, bool kLog = kTwins>
__device__ inline int32_t window_run(const KernelArgs &a, Window &w, WalkMode walk, int32_t j,
                                     int32_t begin, bool snapshots, int32_t q_begin)
{
#define MMS_WINDOW_DEPTH(D) window_run_depth<kLegacy, D, kTwins, kLog>(a, w, walk, j, begin, snapshots, q_begin)
    if constexpr (!kLegacy) {
        switch (w.depth) {
            case 1: return MMS_WINDOW_DEPTH(1);
            case 2: return MMS_WINDOW_DEPTH(2);
            case 4: return MMS_WINDOW_DEPTH(4);
            case 8: return MMS_WINDOW_DEPTH(8);
            default: break;
        }
    }
    return MMS_WINDOW_DEPTH(0);
#undef MMS_WINDOW_DEPTH
}

}  // namespace mms
