// sim_chunk.cuh — kernel arguments, trace geometry and the chunk runner.
//
// Geometry.  The trace is cut at leaf boundaries of numpy's pairwise sum into
// SEGMENTS of about seg_len requests (the last one takes the remainder); a
// CHUNK is seg_per_chunk consecutive segments.  Per (candidate, segment) the
// kernels keep the clock vector at the segment's end and the decisions of the
// segment; per (candidate, chunk) the clock vector the chunk was started
// from.  All of it is laid out [..][entry][candidate] so that the 32
// candidates of a warp touch consecutive addresses.
#pragma once
#include "sim_core.cuh"

namespace mms {

// What build_tables_kernel finds in a call's tables (KernelArgs::irregular).
// The layout the window kernels make of them would not do: a column is used with different
// numbers of stages, a replica's slots are not its group's, a group has several columns, or a
// replica list is not in ascending group order.
constexpr uint32_t kIrregularLayout = 1;
// A latency is negative or not a number.  An accepted request may then leave a clock BEFORE its
// arrival time, and neither cutting in time (states_equivalent) nor comparing clocks by their bits
// (window_groups) is sound: such a call is simulated in one piece, in the layout as given.
constexpr uint32_t kIrregularLatency = 2;

constexpr uint8_t kRelOther = 1, kRelNamed = 2;       // KernelArgs::rel

struct KernelArgs {
    // trace
    const double *arrivals;
    const int32_t *model_ids;
    const float *slos;
    int64_t N;
    int64_t trace_pitch, trace_stride;    // request i of candidate b's trace is element i *
                                  //   trace_pitch + b * trace_stride: 1, 0 with one trace for all
                                  //   candidates; T, 1 with T traces stored request-major ([N][T]);
                                  //   1, N with T traces stored one after the other ([T][N])
    bool many_traces;             // candidate b simulates trace b
    const int32_t *model_hist;    // [M + 1] request counts per model ([T][M + 1] with T traces)
    const int32_t *unsorted;      // number of unsorted / non-finite positions in the trace(s)
    // placements
    int32_t B, M, G, P, T, S, C;
    const uint16_t *model_off;
    const uint32_t *model_rep;
    const uint32_t *group_info;
    const float *latency;
    int64_t latency_stride;
    int32_t lat_smem_elems;
    int32_t lat_f64;              // the on-chip latency table holds doubles (the f32 values widened)
    int32_t block_warps;          // warps per block of the stream kernel
    // geometry
    int32_t K;                    // chunks
    int32_t NS;                   // segments
    int32_t seg_len;              // requests per segment (nominal)
    int32_t seg_per_chunk;
    int32_t warmup;               // run-in requests before a speculative chunk
    // summation plan
    int32_t num_leaves;
    const int32_t *leaf_start;
    // scratch
    uint32_t *rep_rows;           // [row_planes][ceil(B/32)][M + 1][32][4]: replica rows built from
                                  //   model_off/model_rep (first four replicas of each model,
                                  //   then the next four, then those behind), see row_index()
    int32_t row_planes;           // 2: models with more than eight replicas have no further rows
    double *leaf_sums;            // [num_leaves][B]
    double *seg_end;              // [NS][T][B]   clock vector after each segment
    double *chunk_start;          // [K][T][B]    clock vector each chunk started from
    int64_t dec_pitch;            // elements per request row of `decisions`: B rounded up to 32,
                                  //   so that a warp's records of one request fill whole sectors
    void *decisions;              // [ceil(N/4)][dec_pitch][4] u8 (up to 126 groups) or u16: 0 = not
                                  //   dispatched, else (group + 1) | accepted << 7 (or << 15),
                                  //   see count_kernel
    bool dec_wide;
    uint32_t *work_count;         // [kMaxRepairRounds] entries per round
    uint32_t *work_next;          // [kMaxRepairRounds] next list entry to be taken, per round
    uint32_t *work_items;         // [B * K]: chunk * B + candidate
    uint8_t *stamp;               // [K][B]: 1 + the last round in which the chunk was walked
    uint8_t *link;                // [K][B]: the run of chunk j continues the run of chunk j-1
    uint8_t *open;                // [B]: some boundary of the candidate does not
    // relabelling, see warp_relabel
    const uint32_t *twin_class;   // [B][G]: smallest group interchangeable with the group | the
                                  //   group's rank among those << 8 | the largest one << 16
    const uint8_t *twins;         // [B]: some group has an interchangeable one
    uint8_t *rel;                 // [NS][B]: segment q is written in other labels than segment q-1
                                  //   (kRelOther); its records are to be named (kRelNamed)
    uint8_t *perm;                // [NS][B][G]: label in segment q -> label in segment q-1; behind
                                  //   finish_kernel, where name_from says so: -> group number
    int32_t *name_from;           // [NS][B], where rel is kRelNamed: segment with the labels to use
    uint64_t *tie;                // [NS][B]: classes of twins (class_bit) for which a group number
                                  //   decided a choice in segment q between different states
    // choices that a group number decided between twins in the same state: per segment and
    // candidate a list, in order, of at most swap_cap.  Null: no candidate has twins
    uint32_t *swap_mask;          // [NS][swap_cap][B]: those twins (bit k: rank k of the class)
    uint16_t *swap_at;            // [NS][swap_cap][B]: the request, counted from the segment's first
    uint8_t *swap_count;          // [NS][B]
    int32_t swap_cap;
    uint8_t *relabelled;          // [B]: some segment has one
    int32_t *seg_first_leaf;      // [NS + 1]: first leaf of each segment
    int32_t win_table_elems;      // entries of the window kernels' on-chip latency table; 0: off chip
    const uint32_t *column_stages, *irregular, *group_column;    // see ClearArgs, kIrregularLayout
    bool window;                  // the speculative pass is window_stream_kernel's
    int32_t round;
    // outputs
    uint32_t *status;             // [B]
    double *finish;               // [B][N], or null: no per-request outputs wanted
    uint8_t *good;                // [B][N] or null
    int32_t *resimulated;         // [B] or null
};

// First leaf whose first request is at or after request index `pos`.
__device__ inline int32_t leaf_lower_bound(const int32_t *leaf_start, int32_t num_leaves,
                                           int64_t pos)
{
    int32_t lo = 0, hi = num_leaves;
    while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if ((int64_t)leaf_start[mid] < pos) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// First leaf of segment q (q == NS: one past the last leaf).
__device__ inline int32_t seg_leaf(const KernelArgs &a, int32_t q)
{
    if (q <= 0) return 0;
    if (q >= a.NS) return a.num_leaves;
    return a.seg_first_leaf[q];
}

// Where the replica row of (candidate b, model m) is, in 16-byte units: the
// rows of 32 consecutive candidates for one model are contiguous.
__device__ inline size_t row_index(const KernelArgs &a, int64_t b, int m)
{
    return ((size_t)(b / kLanes) * (a.M + 1) + m) * kLanes + (size_t)(b % kLanes);
}

// 16-byte units between a model's replica rows.
__device__ inline size_t row_plane(const KernelArgs &a)
{
    return (size_t)((a.B + kLanes - 1) / kLanes) * (a.M + 1) * kLanes;
}

// True when the trace can be cut (sorted, finite arrival times; no negative latencies).
__device__ inline bool can_chunk(const KernelArgs &a)
{
    return a.K > 1 && *a.unsorted == 0 && !(*a.irregular & kIrregularLatency);
}

// Offset of request 0 of the trace candidate b simulates.
__device__ inline size_t trace_base(const KernelArgs &a, int64_t b)
{
    return (size_t)(b * a.trace_stride);
}

// Arrival time of request i in candidate b's trace.
__device__ inline double arrival_at(const KernelArgs &a, int64_t b, int64_t i)
{
    return a.arrivals[(size_t)i * a.trace_pitch + trace_base(a, b)];
}

// Two clock vectors X and Y, taken at a point where every later arrival is
// >= tau, lead to identical futures (every later finish time, good flag and
// counter) when
//  (1) each slot holds the same value in both, or a value < tau in both — a
//      clock that is already in the past only ever enters max(t, clock) with
//      t >= tau, so its exact value cannot matter — EXCEPT
//  (2) the last-stage clock of a group that serves a model with several
//      replicas: dispatch compares those clocks with '<' (controller.py:595-598),
//      so for the ones in the past the ORDER among them (ties included) must
//      agree as well.  A clock in the past is below every clock that is not,
//      in both vectors, so mixed comparisons agree by (1).
// Each accepted request overwrites clocks with values >= tau (latencies are not
// negative, see kIrregularLatency) that are equal in both runs, so the relation is preserved step by step, and it is
// transitive.  LoadX / LoadY map a clock slot to its value.
template <typename LoadX, typename LoadY, typename Stale>
__device__ inline bool states_equivalent(const KernelArgs &a, int64_t b, LoadX X, LoadY Y,
                                         double tau, Stale stale)
{
    int n_stale = 0;
    for (int g = 0; g < a.G; ++g) {
        const uint32_t info = a.group_info[(size_t)b * a.G + g];
        const uint32_t slot = info & 0xFFu, ns = (info >> 8) & 0xFFu;
        const bool contested = (info >> 16) & 1u;
        for (uint32_t k = 0; k < ns; ++k) {
            const double x = X(slot + k), y = Y(slot + k);
            const bool past = x < tau && y < tau;
            if (!(x == y || past)) return false;
            if (past && contested && k == ns - 1 && x != y) stale(n_stale++) = (uint8_t)(slot + k);
        }
    }
    // Order of every past last-stage clock that differs between X and Y
    // against the last-stage clocks of all contested groups.
    for (int u = 0; u < n_stale; ++u) {
        const uint32_t su = stale(u);
        const double xu = X(su), yu = Y(su);
        for (int g = 0; g < a.G; ++g) {
            const uint32_t info = a.group_info[(size_t)b * a.G + g];
            const uint32_t ns = (info >> 8) & 0xFFu;
            if (ns == 0 || !((info >> 16) & 1u)) continue;
            const uint32_t sv = (info & 0xFFu) + ns - 1;
            const double xv = X(sv), yv = Y(sv);
            if ((xu < xv) != (yu < yv) || (xu > xv) != (yu > yv)) return false;
        }
    }
    return true;
}

// The same with the lanes of a warp over the groups: X(slot) and Z(slot) give the two
// states, info(g) the group table.  The answer is the same in all lanes.
template <typename Info, typename LoadX, typename LoadZ>
__device__ inline bool warp_equivalent(int G, Info info, LoadX X, LoadZ Z, double tau)
{
    const int lane = threadIdx.x & (kLanes - 1);
    uint32_t any_stale = 0;
    for (int g0 = 0; g0 < G; g0 += kLanes) {
        const int g = g0 + lane;
        const uint32_t in = g < G ? info(g) : 0u;
        const uint32_t slot = in & 0xFFu, ns = (in >> 8) & 0xFFu;
        bool bad = false, stale = false;
        for (uint32_t k = 0; k < ns; ++k) {
            const double x = X(slot + k), z = Z(slot + k);
            const bool past = x < tau && z < tau;
            bad |= !(x == z || past);
            if (k == ns - 1) stale = past && x != z && ((in >> 16) & 1u);
        }
        if (__any_sync(0xFFFFFFFFu, bad)) return false;
        any_stale |= __ballot_sync(0xFFFFFFFFu, stale);
    }
    if (!any_stale) return true;
    for (int u = 0; u < G; ++u) {
        const uint32_t iu = info(u);
        const uint32_t nu = (iu >> 8) & 0xFFu;
        if (nu == 0 || !((iu >> 16) & 1u)) continue;
        const uint32_t su = (iu & 0xFFu) + nu - 1;
        const double xu = X(su), zu = Z(su);
        if (xu == zu || !(xu < tau && zu < tau)) continue;
        bool bad = false;
        for (int g = lane; g < G; g += kLanes) {
            const uint32_t in = info(g);
            const uint32_t ns = (in >> 8) & 0xFFu;
            if (ns == 0 || !((in >> 16) & 1u)) continue;
            const uint32_t sv = (in & 0xFFu) + ns - 1;
            const double xv = X(sv), zv = Z(sv);
            bad |= (xu < xv) != (zu < zv) || (xu > xv) != (zu > zv);
        }
        if (__any_sync(0xFFFFFFFFu, bad)) return false;
    }
    return true;
}

// RELABELLING.  Groups with the same parallel config and the same models (twins, found
// on the device: twins_kernel) are interchangeable, and which of them is ahead depends on
// history long past: a speculative run often comes out with their roles exchanged.
// Such a run is the true one under other labels.  Let Z be the state it starts
// from, X the true state, and p a permutation within the classes of twins with X ~ p(Z) (equivalent
// in the sense above after p has moved every group's clocks).  Then the run makes, request by
// request, the choice p would translate into the true one — the replicas of a model are
// closed under p, their latencies are the same, the smallest last-stage clock is the
// same — EXCEPT where the smallest clock belongs to several replicas and the group number
// decides (bursts of requests with one arrival time do that all the time).  Mostly those are
// twins in the same state, all clocks alike: then any of them can stand for any other, and p
// is replaced, from that request on, by the permutation with two of them exchanged that
// translates the run's choice into the true one.  The simulation notes these requests in a list
// per segment (`swap_mask`, `swap_at`; a word per request instead was five sixths of a call's
// scratch, nearly all of it zero).  Where the replicas are not in the same state and that matters
// (tie_matters), or the list is full, it notes their classes for the segment (`tie`), and a segment
// is only taken over under labels that leave those classes alone.
// name_kernel translates the decision records into group numbers; nothing else has labels.
//
// p has to keep the order of the last-stage clocks within a class (every group of a class serves
// a replicated model), so it is the one that sorts them, equal ones by group number.
//
// Writes p (label of Z -> label of X; u8[G], and the identity for groups without twins) and
// p(Z) to shared memory; `last` (f64[G]) and `rank` (u8[2G]) are scratch there.  Y is the saved
// state, entries `pitch` apart.  Returns whether p is not the identity.
struct RelabelScratch { uint32_t z, last, perm, rank; };       // f64, f64, u8, u8 indices

template <typename Info, typename LoadX>
__device__ inline bool warp_relabel(int G, int T, const uint32_t *cls, Info info, LoadX X,
                                    const double *Y, size_t pitch, const RelabelScratch &s)
{
    const int lane = threadIdx.x & (kLanes - 1);
    __syncwarp();
    for (int g = lane; g < G; g += kLanes) {
        const uint32_t in = info(g);
        const uint32_t ns = (in >> 8) & 0xFFu;
        SM_F64(s.last + g) = ns ? Y[(size_t)((in & 0xFFu) + ns - 1) * pitch] : 0.0;
    }
    __syncwarp();
    for (int g = lane; g < G; g += kLanes) {
        const uint32_t in = info(g);
        const uint32_t ns = (in >> 8) & 0xFFu;
        const uint32_t c = class_first(cls[g]);
        const double x = ns ? X((in & 0xFFu) + ns - 1) : 0.0, y = SM_F64(s.last + g);
        uint32_t rx = 0, ry = 0;
        for (int h = (int)c; h < G; ++h) {                // members of the class: c is its smallest
            if (class_first(cls[h]) != c || h == g) continue;
            const uint32_t ih = info(h);
            const double xh = X((ih & 0xFFu) + ((ih >> 8) & 0xFFu) - 1), yh = SM_F64(s.last + h);
            rx += xh < x || (xh == x && h < g);
            ry += yh < y || (yh == y && h < g);
        }
        smem[s.rank + g] = (uint8_t)rx;
        smem[s.rank + G + g] = (uint8_t)ry;
    }
    __syncwarp();
    bool moved = false;
    for (int g = lane; g < G; g += kLanes) {
        const uint32_t c = class_first(cls[g]), r = smem[s.rank + G + g];
        int to = g;
        for (int h = (int)c; h < G; ++h)
            if (class_first(cls[h]) == c && smem[s.rank + h] == r) { to = h; break; }
        smem[s.perm + g] = (uint8_t)to;
        moved |= to != g;
        const uint32_t ig = info(g), it = info(to);
        for (uint32_t k = 0; k < ((ig >> 8) & 0xFFu); ++k)
            SM_F64(s.z + (it & 0xFFu) + k) = Y[(size_t)((ig & 0xFFu) + k) * pitch];
    }
    (void)T;
    __syncwarp();
    return __any_sync(0xFFFFFFFFu, moved);
}

// Does it matter, under labels that move the class `picked` or the class `other`, that a group number
// decided between a picked group of the former and one of the latter?  Not if all of the
// former's numbers are smaller than all of the latter's: then the true choice is among the picked one's
// twins as well, whatever the labels.  (Placements that a search has normalized have their twins
// side by side, where this is always so; of random ones on 64 devices 0.001 % of the requests are
// such a choice, 0.03 % on 16.  Without the test 0.01 to 1.6 % were, and the last pass walked most
// candidates with twins from end to end because of them.)
__device__ __forceinline__ bool tie_matters(uint32_t picked, uint32_t other)
{
    return class_first(picked) == class_first(other) || class_last(picked) > class_first(other);
}

// Bit of a class of twins in a tie mask (more than 64 classes share bits, which only costs
// re-simulations).
__device__ __forceinline__ uint64_t class_bit(uint32_t twin_class) { return 1ull << (twin_class & 63u); }

// Classes that a permutation moves, by a warp: perm(g) is the image of group g.
template <typename Perm>
__device__ inline uint64_t moved_classes(const uint32_t *twin_class, int G, Perm perm)
{
    uint64_t moved = 0;
    for (int g = threadIdx.x & (kLanes - 1); g < G; g += kLanes)
        if (perm(g) != (uint8_t)g) moved |= class_bit(twin_class[g]);
    const uint32_t lo = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)moved);
    const uint32_t hi = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)(moved >> 32));
    return ((uint64_t)hi << 32) | lo;
}

template <int kStride>
__device__ Tie note_tie(const KernelArgs *args, int32_t b, int32_t q, int32_t swaps, int32_t i,
                        const uint32_t *twin_class, const uint32_t *list, int n, uint32_t clk,
                        double best, uint32_t pick, double ts)
{
    const KernelArgs &a = *args;
    Tie t;
    t.classes = 0;
    t.noted = 0;
    const uint32_t pns = rep_stages(pick), p0 = clk + (rep_last(pick) + 1 - pns) * kStride;
    const uint32_t own = twin_class[rep_group(pick)];
    uint32_t swap = 0;
    for (int r = 0; r < n; ++r) {
        const uint32_t e = rep_to_last(__ldg(list + r));
        if (!(SM_F64(clk + rep_last(e) * kStride) == best)) continue;
        const uint32_t other = twin_class[rep_group(e)];
        bool same = class_first(other) == class_first(own) && class_rank(other) < 32;
        const uint32_t e0 = clk + (rep_last(e) + 1 - pns) * kStride;
        for (uint32_t k = 0; k + 1 < pns && same; ++k) {
            const double x = SM_F64(p0 + k * kStride), y = SM_F64(e0 + k * kStride);
            same = x == y || (x < ts && y < ts);
        }
        if (same) swap |= 1u << class_rank(other);
        else if (tie_matters(own, other)) t.classes |= class_bit(own) | class_bit(other);
    }
    if (swap & (swap - 1)) {                 // more than the picked one
        if (swaps < a.swap_cap) {
            const size_t cell = ((size_t)q * a.swap_cap + swaps) * a.B + b;
            a.swap_mask[cell] = swap;
            a.swap_at[cell] = (uint16_t)(i - a.leaf_start[seg_leaf(a, q)]);
            t.noted = 1;
        } else {
            t.classes |= class_bit(own);
        }
    }
    return t;
}

// Runs chunk j of candidate b on this lane, speculatively: requests [begin, first)
// as run-in (nothing recorded; `first` is the chunk's first request), then the
// chunk's segments, recording decisions, per-request outputs (kFull) and one latency
// sum per leaf.  With `snapshots` the clock vector after the run-in is stored as the
// chunk's start state, and every segment's end state.  Within a leaf the latency
// of request k goes to partial sum k mod 8, as numpy's pairwise sum does.
template <bool kFull, bool kLegacy, bool kTwins>
__device__ inline void run_chunk(const KernelArgs &a, Lane &ln, Pipe &p, int64_t b, int32_t j,
                                 int32_t begin, bool snapshots)
{
    double *fin_out = kFull ? a.finish + (size_t)b * a.N : nullptr;
    uint8_t *good_out = kFull ? a.good + (size_t)b * a.N : nullptr;
    int32_t q = j * a.seg_per_chunk;
    const int32_t q1 = (j + 1) * a.seg_per_chunk < a.NS ? (j + 1) * a.seg_per_chunk : a.NS;
    int32_t leaf = seg_leaf(a, q);
    int32_t seg_stop = seg_leaf(a, q + 1);
    const int32_t first = leaf < a.num_leaves ? a.leaf_start[leaf] : (int32_t)a.N;
    leaf -= 1;                      // the run-in counts as a leaf that is not recorded
    int32_t i = begin, span_end = first;
    bool record = false;
    ln.q = q;
    pipe_prime(ln, p, begin);
    for (;;) {
        // Within a leaf the latency of request k goes to partial sum k mod 8
        // (leaves start at multiples of 8).  The latencies of eight requests
        // are parked in the eight spare clock slots behind the lane's clock
        // vector (read only as don't-care stages otherwise) and added to the
        // partial sums together.
        const int32_t body_end = record ? i + ((span_end - i) & ~7) : i;
        const uint32_t ring = ln.clk + (uint32_t)a.T * kLanes;
        double p0 = 0.0, p1 = 0.0, p2 = 0.0, p3 = 0.0, p4 = 0.0, p5 = 0.0, p6 = 0.0, p7 = 0.0;
        double r = 0.0;
        auto one = [&](int32_t ii) {
            const double d = sim_step<kFull, kLegacy, kTwins>(ln, p, ii, record, fin_out, good_out);
            if (ii < body_end) {
                SM_F64(ring + (uint32_t)(ii & 7) * kLanes) = d;
                if ((ii & 7) == 7) {
                    p0 += SM_F64(ring); p1 += SM_F64(ring + kLanes);
                    p2 += SM_F64(ring + 2 * kLanes); p3 += SM_F64(ring + 3 * kLanes);
                    p4 += SM_F64(ring + 4 * kLanes); p5 += SM_F64(ring + 5 * kLanes);
                    p6 += SM_F64(ring + 6 * kLanes); p7 += SM_F64(ring + 7 * kLanes);
                    if (ii + 1 == body_end)
                        r = ((p0 + p1) + (p2 + p3)) + ((p4 + p5) + (p6 + p7));
                }
            } else {
                r += d;
            }
        };
        // three requests per turn: the values fetched ahead rotate through three sets of
        // registers, and after three steps every set is back where it was — no moves (two
        // dozen per request otherwise: stream kernel 17.0 -> 16.1 ms)
        for (; i + 3 <= span_end; i += 3) { one(i); one(i + 1); one(i + 2); }
#pragma unroll 1
        for (; i < span_end; ++i) one(i);
        if (!record) {
            ln.tie = 0;
            if (snapshots)   // the state this speculative chunk starts from
                for (int t = 0; t < a.T; ++t)
                    a.chunk_start[((size_t)j * a.T + t) * a.B + b] = SM_F64(ln.clk + t * kLanes);
        } else {
            a.leaf_sums[(size_t)leaf * a.B + b] = r;
            if (leaf + 1 == seg_stop) {             // segment q is complete
                if (snapshots) {
                    if constexpr (kTwins) {
                        a.tie[(size_t)q * a.B + b] = ln.tie;
                        a.swap_count[(size_t)q * a.B + b] = (uint8_t)ln.swaps;
                        ln.tie = 0;
                        ln.swaps = 0;
                        ln.q = q + 1;
                    }
                    for (int t = 0; t < a.T; ++t)
                        a.seg_end[((size_t)q * a.T + t) * a.B + b] = SM_F64(ln.clk + t * kLanes);
                }
                if (++q >= q1) return;
                seg_stop = seg_leaf(a, q + 1);
            }
        }
        ++leaf;
        if (leaf >= a.num_leaves) return;        // only an empty trace gets here
        record = true;
        span_end = a.leaf_start[leaf + 1];
    }
}

}  // namespace mms
