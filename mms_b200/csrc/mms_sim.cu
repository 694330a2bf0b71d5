// mms_sim.cu — sm_100a kernels of the placement-evaluation simulator.
//
// What is simulated: AlpaServe's per-request FIFO pipeline model with SLO
// dropping (alpa_serve/simulator/controller.py:561-628, and :506-558 for the
// one-clock-per-group variant) for a batch of candidate placements against
// one request trace, followed by the fast_stats reductions of
// controller.py:393-403.
//
// The recurrence over requests is sequential per candidate.  Parallelism
// comes from (a) the candidates of the batch and (b) cutting each candidate's
// trace into chunks that are simulated SPECULATIVELY at the same time:
//
//   stream kernel   the speculative pass.  A chunk starts from idle clocks some
//                   requests before its first one (run-in, nothing recorded), stores the
//                   clock vector it has when the chunk proper begins and after
//                   every segment, and records its decisions and latency sums.  Large
//                   batches: one thread per (candidate, chunk), 32 candidates to a
//                   warp (sim_stream_kernel); small ones: one warp (sim_window.cuh).
//   link kernel     one thread per chunk boundary: does the chunk's run start from a state
//                   EQUIVALENT to the one the run before it ended in (states_equivalent:
//                   equal futures, provably), as it is or under other labels of
//                   interchangeable groups (warp_relabel)?
//   restart or      lists the chunks behind failed boundaries, all of them or the first of each
//   resolve kernel  failed stretch.
//   walk kernel     one warp per listed chunk re-simulates it, and what follows, from the state
//                   the chunk before it ended in until the stored run can take over.
//                   (A walk that started from a wrong state has to be done again.)
//   finish kernel   one warp per candidate that is still open, or has relabelled segments,
//                   goes through them in order, re-simulates whatever the rounds
//                   left and follows the labels — it makes the result exact
//                   whatever the chunking and the rounds.
//   name kernel     translates labels into group numbers, a warp per few segments.
//   count kernel    tallies the recorded decisions into the counters and combines the
//                   per-leaf latency sums in numpy's pairwise order.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "mms_sim.h"
#include "sim_batching.cuh"
#include "sim_chunk.cuh"
#include "sim_window.cuh"

namespace mms {

constexpr int kMaxSumDepth = 48;        // pair-sum stack of the numpy order
constexpr int kLatSmemBytes = 32 * 1024;
constexpr int kMaxRepairRounds = 16;
constexpr int kTwinModels = 256;        // models a launch with interchangeable groups may have
// One round of parallel walks: what it leaves open finish_kernel walks in any case, all candidates
// beside each other, and each further round is three launches and waits for its longest walk
// (a second one: 1000 placements on 64 devices 18.6 -> 15.7 ms, but 500 9.7 -> 10.5, grown ones on
// 64 devices 73 -> 86 and 37.4 -> 36.6, a layer of 2343 47 -> 50, 4096 placements the same).
constexpr int kDefaultRepairRounds = 1;

// What a call clears before its kernels run, in one launch (grid-stride): the
// work lists and marks of the time-parallel machinery, the outputs
// the tally adds into, the status words — and the kernels' own copy of
// group_info, bounds-checked (a bad entry becomes an empty group) and with the
// "contested" bit (bit 16) cleared: build_tables_kernel derives that bit from
// the replica lists, so exactness never rests on what the caller put there.
struct ClearArgs {
    const uint32_t *group_info_in;    // the caller's [B][G]
    uint32_t *group_info;             // scratch copy the kernels read
    int32_t *model_num_good;          // [B][M]
    int32_t *model_num_requests;      // [B][M]
    int32_t *group_num_requests;      // [B][G]
    int32_t *group_num_good;          // [B][G] or null
    int64_t *good_total;              // [B]
    // for twins_kernel
    int32_t group_words;              // 64-bit words of a group's model set; 0: too many models
    uint64_t *group_models;           // [B][G][group_words]
    uint32_t *group_column;           // [B][G] latency column of the group; 0xFFFFFFFF: no model
    uint32_t *twin_class;             // see KernelArgs
    uint8_t *twins;
    uint32_t *column_stages;          // [C] stages of the groups that use the column
    uint32_t *irregular;              // kIrregularLayout | kIrregularLatency
};

__device__ inline bool group_info_valid(const KernelArgs &a, uint32_t info)
{
    const uint32_t slot = info & 0xFFu, ns = (info >> 8) & 0xFFu;
    return slot + ns <= (uint32_t)a.T && ns <= (uint32_t)a.S;
}

__global__ void clear_kernel(const KernelArgs a, const ClearArgs c)
{
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    if (a.K > 1) {
        for (int64_t i = tid; i < (int64_t)a.NS * a.B; i += nth) a.rel[i] = 0;
        for (int64_t i = tid; i < (int64_t)a.K * a.B; i += nth) a.stamp[i] = 0;
        for (int64_t i = tid; i < (int64_t)a.B * a.G; i += nth) {
            for (int k = 0; k < c.group_words; ++k) c.group_models[i * c.group_words + k] = 0;
        }
        for (int64_t i = tid; i < a.B; i += nth) { c.twins[i] = 0; a.open[i] = 0; a.relabelled[i] = 0; }
    }
    for (int64_t i = tid; i < (int64_t)a.B * a.G; i += nth) {
        c.group_column[i] = 0xFFFFFFFFu;
        const uint32_t info = c.group_info_in[i];
        c.group_info[i] = group_info_valid(a, info) ? (info & ~0x10000u) : 0u;
    }
    // model_num_requests (controller.py:587) does not depend on the placement: the trace's histogram
    for (int64_t i = tid; i < (int64_t)a.B * a.M; i += nth) {
        c.model_num_good[i] = 0;
        c.model_num_requests[i] = a.model_hist[(a.many_traces ? i / a.M * (a.M + 1) : 0) + i % a.M];
    }
    for (int64_t i = tid; i < (int64_t)a.B * a.G; i += nth) {
        c.group_num_requests[i] = 0;
        if (c.group_num_good) c.group_num_good[i] = 0;
    }
    for (int64_t i = tid; i < a.B; i += nth) {
        c.good_total[i] = 0;
        a.status[i] = 0;
        if (a.resimulated) a.resimulated[i] = 0;
    }
    for (int64_t i = tid; i < a.C; i += nth) c.column_stages[i] = 0;
    if (tid == 0) *c.irregular = 0;
    for (int64_t i = tid; i < kMaxRepairRounds; i += nth) { a.work_count[i] = 0; a.work_next[i] = 0; }
}

// Builds, in one launch behind clear_kernel, the tables the simulation kernels
// read: (1) one thread per (candidate, model or the extra empty row) checks the
// model's replica list, writes its two 16-byte rows (see Lane::rows) and marks
// the groups of a list with more than one replica as contested; a list with a
// bad index is reported in the status word and emptied.  (2) One thread per
// (candidate, group) reports a group_info entry that clear_kernel had to empty.
// (3) One thread per segment finds the segment's first leaf.  (4) The latency tables are looked
// through for entries that are not >= 0 (kIrregularLatency).  Each is a chain of loads: each part
// begins at another quarter of the grid, so that the four run beside each other in a small call.
constexpr int kTableBlocks = 4;              // blocks of build_tables_kernel, at least
__global__ void build_tables_kernel(const KernelArgs a, const ClearArgs c)
{
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const auto next_quarter = [&] { tid = tid >= nth / 4 ? tid - nth / 4 : tid + nth - nth / 4; };
    for (int64_t q = tid; q <= a.NS; q += nth)
        a.seg_first_leaf[q] = q == 0 ? 0 : q == a.NS ? a.num_leaves
            : leaf_lower_bound(a.leaf_start, a.num_leaves, q * a.seg_len);
    const int64_t entries = (int64_t)a.M * a.C * a.S;
    bool odd = false;
    next_quarter();
    for (int64_t i = tid; i < (a.latency_stride ? a.B * entries : entries); i += nth)
        odd |= !(a.latency[i / entries * a.latency_stride + i % entries] >= 0.0f);
    if (odd) atomicOr(c.irregular, kIrregularLatency);
    next_quarter();
    for (int64_t i = tid; i < (int64_t)a.B * a.G; i += nth)
        if (!group_info_valid(a, c.group_info_in[i]))
            atomicOr(&a.status[i / a.G], MMS_STATUS_BAD_INDEX);
    next_quarter();
    for (int64_t t = tid; t < (int64_t)a.B * (a.M + 1); t += nth) {
        const int64_t b = t / (a.M + 1);
        const int m = (int)(t % (a.M + 1));
        uint32_t e[8] = {kNoReplica, kNoReplica, kNoReplica, kNoReplica,
                         kNoReplica, kNoReplica, kNoReplica, kNoReplica};
        if (m < a.M) {
            const uint32_t lo = a.model_off[(size_t)b * (a.M + 1) + m];
            const uint32_t hi = a.model_off[(size_t)b * (a.M + 1) + m + 1];
            bool bad = lo > hi || hi > (uint32_t)a.P;
            if (!bad) {
                for (uint32_t r = lo; r < hi; ++r) {
                    const uint32_t ent = a.model_rep[(size_t)b * a.P + r];
                    const uint32_t ns = (ent >> 16) & 0xFFu, first = (ent >> 8) & 0xFFu;
                    if ((ent & 0xFFu) >= (uint32_t)a.G || ns == 0 || first + ns > (uint32_t)a.T ||
                        ns > (uint32_t)a.S || (ent >> 24) >= (uint32_t)a.C) {
                        bad = true;
                        continue;
                    }
                    // the window kernels lay pipelines out by group and by column
                    const uint32_t was = atomicCAS(&c.column_stages[ent >> 24], 0u, ns);
                    if ((was != 0 && was != ns) ||
                        ((c.group_info_in[(size_t)b * a.G + (ent & 0xFFu)] & 0xFFFFu) != (first | (ns << 8))))
                        atomicOr(c.irregular, kIrregularLayout);
                    const size_t gg = (size_t)b * a.G + (ent & 0xFFu);
                    const uint32_t col = atomicCAS(&c.group_column[gg], 0xFFFFFFFFu, ent >> 24);
                    if (col != 0xFFFFFFFFu && col != ent >> 24) atomicOr(c.irregular, kIrregularLayout);
                    // ... and take the first of the smallest clocks for the lowest group number
                    if (r > lo && (a.model_rep[(size_t)b * a.P + r - 1] & 0xFFu) >= (ent & 0xFFu))
                        atomicOr(c.irregular, kIrregularLayout);
                    if (a.K > 1 && c.group_words)
                        atomicOr((unsigned long long *)&c.group_models[gg * c.group_words + (m >> 6)], 1ull << (m & 63));
                    if (r - lo < 8)
                        e[r - lo] = rep_to_last(ent);
                }
                if (hi - lo > 8) {
                    // the eighth and those behind, four to a row, up to a row that is not full
                    e[7] = kMoreReplicas;
                    uint4 *more = reinterpret_cast<uint4 *>(a.rep_rows) + row_index(a, b, m);
                    uint32_t r = lo + 7;
                    for (int p = 2; p < a.row_planes && r <= hi && !bad; ++p, r += 4) {
                        uint32_t x[4];
                        for (uint32_t k = 0; k < 4; ++k)
                            x[k] = r + k < hi ? rep_to_last(a.model_rep[(size_t)b * a.P + r + k]) : kNoReplica;
                        if (p + 1 == a.row_planes && r + 4 <= hi) x[3] = kMoreReplicas;
                        more[(size_t)p * row_plane(a)] = make_uint4(x[0], x[1], x[2], x[3]);
                    }
                }
            }
            if (bad) {
                atomicOr(&a.status[b], MMS_STATUS_BAD_INDEX);
                for (int k = 0; k < 8; ++k) e[k] = kNoReplica;
            } else if (hi - lo > 1) {
                // dispatch compares the last-stage clocks of these groups with '<'
                for (uint32_t r = lo; r < hi; ++r)
                    atomicOr(&c.group_info[(size_t)b * a.G + (a.model_rep[(size_t)b * a.P + r] & 0xFFu)],
                             0x10000u);
            }
        }
        uint4 *rows = reinterpret_cast<uint4 *>(a.rep_rows);
        rows[row_index(a, b, m)] = make_uint4(e[0], e[1], e[2], e[3]);
        rows[row_plane(a) + row_index(a, b, m)] = make_uint4(e[4], e[5], e[6], e[7]);
    }
}

// This lane's view of candidate b: offsets of its shared-memory state (clocks
// zeroed) and pointers to its tables in global memory.
__device__ inline Lane setup_lane(const KernelArgs &a, int64_t b, int lane, int warp = 0)
{
    const SmemLayout L = smem_layout(a.T, a.S, a.lat_smem_elems, a.lat_f64 != 0);
    const size_t base = L.warp0 + (size_t)warp * L.warp_bytes;
    Lane ln;
    ln.clk = (uint32_t)((base + L.clocks) / sizeof(double)) + lane;
    ln.tmp = (uint32_t)((base + L.stage_tmp) / sizeof(double)) + lane;
    ln.lat_sm = (uint32_t)(L.latency / sizeof(float));
    ln.dec_wide = a.dec_wide;
    ln.dec = a.dec_wide ? static_cast<void *>(static_cast<uint16_t *>(a.decisions) + 4 * b)
                        : static_cast<void *>(static_cast<uint8_t *>(a.decisions) + 4 * b);
    ln.dec_pitch = (uint32_t)a.dec_pitch;
    ln.dec_word = 0;
    ln.rows = reinterpret_cast<const uint4 *>(a.rep_rows) + row_index(a, b, 0);
    ln.plane = (uint32_t)row_plane(a);
    ln.rows_b = ln.rows + ln.plane;
    ln.rows_c = a.row_planes > 2 ? ln.rows_b + ln.plane : nullptr;
    ln.rep_raw = a.model_rep + (size_t)b * a.P;
    ln.rep_off = a.model_off + (size_t)b * (a.M + 1);
    ln.lat_gl = a.latency + (size_t)b * a.latency_stride;
    ln.lat_on_chip = a.lat_smem_elems != 0;
    ln.lat_f64 = a.lat_f64 != 0;
    ln.M = a.M; ln.C = a.C; ln.S = a.S;
    ln.status = 0;
    ln.tie = 0;
    ln.args = &a;
    ln.b = (int32_t)b;
    ln.q = ln.swaps = 0;
    ln.twin_class = a.swap_mask && a.twins[b] ? a.twin_class + (size_t)b * a.G : nullptr;
    for (int t = 0; t < a.T + kClockPad; ++t) SM_F64(ln.clk + t * kLanes) = 0.0;
    return ln;
}

// The batch's shared latency table goes on chip (f32; widened to f64, exactly,
// when it is used), loaded by all threads of the block: call it before any
// thread returns.
__device__ inline void stage_latency_table(const KernelArgs &a, const SmemLayout &L)
{
    if (a.lat_smem_elems) {
        const int real = a.M * a.C * a.S;
        if (a.lat_f64) {        // widened once here instead of at every use
            const uint32_t base = (uint32_t)(L.latency / sizeof(double));
            for (int i = threadIdx.x; i < a.lat_smem_elems; i += blockDim.x)
                SM_F64(base + i) = i < real ? (double)__ldg(a.latency + i) : 0.0;
        } else {
            const uint32_t base = (uint32_t)(L.latency / sizeof(float));
            for (int i = threadIdx.x; i < a.lat_smem_elems; i += blockDim.x)
                SM_F32(base + i) = i < real ? __ldg(a.latency + i) : 0.0f;
        }
    }
    __syncthreads();
}

__device__ inline void init_pipe(const KernelArgs &a, Pipe &p, int64_t b)
{
    const size_t base = trace_base(a, b);
    p.arrivals = a.arrivals + base; p.model_ids = a.model_ids + base; p.slos = a.slos + base;
    p.pitch = (uint32_t)a.trace_pitch;
    p.last = (int32_t)(a.N - 1);
}

// Blocks of block_warps warps (they share the latency table and nothing else).
template <bool kFull, bool kLegacy, bool kTwins>
__global__ void __launch_bounds__(kLanes * kMaxBlockWarps, 1)
sim_stream_kernel(const __grid_constant__ KernelArgs a)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const int warp = threadIdx.x / kLanes;
    stage_latency_table(a, smem_layout(a.T, a.S, a.lat_smem_elems, a.lat_f64 != 0));
    const bool chunked = can_chunk(a);
    const int64_t stream = ((int64_t)blockIdx.x * a.block_warps + warp) * kLanes + lane;
    if (stream >= (int64_t)a.B * a.K) return;   // lanes never wait for each other below
    const int32_t j = (int32_t)(stream / a.B);
    const int64_t b = stream % a.B;
    if (a.N == 0 || (!chunked && j > 0)) return;
    Lane ln = setup_lane(a, b, lane, warp);
    Pipe p;
    init_pipe(a, p, b);
    // not chunked: one chunk holding every segment, plain sequential simulation
    KernelArgs ka = a;
    int32_t begin = 0;
    if (!chunked) {
        ka.seg_per_chunk = a.NS;
    } else if (j > 0) {
        const int32_t first = a.leaf_start[seg_leaf(a, j * a.seg_per_chunk)];
        begin = first - a.warmup > 0 ? first - a.warmup : 0;
    }
    run_chunk<kFull, kLegacy, kTwins>(ka, ln, p, b, j, begin, chunked);
    if (ln.status) atomicOr(&a.status[b], ln.status);
}

// Classes of interchangeable groups (warp_relabel): same stages, same latency column, same
// set of models.  One thread per (candidate, group); behind build_tables_kernel, which
// collects every group's models as a bit set (a launch with more than kTwinModels models has
// no classes).
__global__ void twins_kernel(const KernelArgs a, const ClearArgs c)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)a.B * a.G || *a.irregular) return;
    const int64_t b = t / a.G;
    const int g = (int)(t % a.G);
    const int W = c.group_words;
    const uint64_t *mine = c.group_models + (size_t)t * W;
    uint64_t some = 0;
    for (int k = 0; k < W; ++k) some |= mine[k];
    const uint32_t ns = (a.group_info[t] >> 8) & 0xFFu, column = c.group_column[t];
    int cls = g, rank = 0, last = g;
    if (some && ns && column < (uint32_t)a.C) {
        for (int h = 0; h < a.G; ++h) {
            if (h == g) continue;
            const size_t u = (size_t)b * a.G + h;
            if (((a.group_info[u] >> 8) & 0xFFu) != ns || c.group_column[u] != column) continue;
            const uint64_t *other = c.group_models + u * W;
            bool same = true;
            for (int k = 0; k < W && same; ++k) same = mine[k] == other[k];
            if (!same) continue;
            if (h > g) last = h;
            else { if (cls == g) cls = h; ++rank; }
        }
    }
    c.twin_class[t] = (uint32_t)(cls | (rank << 8) | (last << 16));
    if (cls != g) c.twins[b] = 1;
}

// Does the run of chunk j of candidate b continue the run of the chunk before it, in the
// same labels (states_equivalent: equal futures, provably)?
__device__ inline bool continues(const KernelArgs &a, int32_t j, int64_t b)
{
    const int32_t q_prev = j * a.seg_per_chunk - 1;
    const double tau = arrival_at(a, b, a.leaf_start[seg_leaf(a, q_prev + 1)]);
    const size_t B = (size_t)a.B;
    const double *X = a.seg_end + (size_t)q_prev * a.T * B + b;
    const double *Y = a.chunk_start + (size_t)j * a.T * B + b;
    uint8_t stale[MMS_MAX_GROUPS];
    return states_equivalent(a, b, [&](uint32_t s) { return X[s * B]; },
                             [&](uint32_t s) { return Y[s * B]; }, tau,
                             [&](int w) -> uint8_t & { return stale[w]; });
}

// A round that walked nothing left every state as it was.
__device__ inline bool nothing_changed(const KernelArgs &a)
{
    return a.round > 0 && a.work_count[a.round - 1] == 0;
}

constexpr int kLinkWarps = 4;

// Shared memory of a link_kernel warp: two states, last-stage clocks, permutation, ranks.
__host__ __device__ inline size_t link_warp_bytes(int T, int G)
{
    return (sizeof(double) * (2 * (size_t)T + (size_t)G) + 3 * (size_t)G + 15) & ~(size_t)15;
}

// Judges the chunk boundaries whose sides the round before changed (all of them in round 0), of
// candidates without interchangeable groups: one thread per boundary.
constexpr int64_t kLinkAlone = 148 * 64;     // boundaries that all have a warp at once

__global__ void __launch_bounds__(128)
link_kernel(const __grid_constant__ KernelArgs a)
{
    if (!can_chunk(a) || nothing_changed(a)) return;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)a.B * (a.K - 1)) return;
    const int64_t b = t % a.B;
    const int32_t j = (int32_t)(t / a.B) + 1;
    const size_t cell = (size_t)j * a.B + b;
    if (a.round != 0 && a.stamp[cell - a.B] != (uint8_t)a.round && a.stamp[cell] != (uint8_t)a.round) return;
    a.link[cell] = continues(a, j, b);
    a.rel[(size_t)(j * a.seg_per_chunk) * a.B + b] = 0;
}

// The same with a warp per boundary, its lanes over the groups, and under other labels: for calls with few boundaries, where a
// thread's way through two states is what takes the time (70 boundaries of one placement on 16 devices
// 27 to 46 us, by warps 9; 3 700 of 37 placements 32 and 10), and for candidates with interchangeable
// groups, whose failed boundaries are compared under other labels by a warp in any case (46 000 of a layer on 64
// devices 498 and 190, the second time 305 and 74).
__global__ void __launch_bounds__(kLinkWarps * kLanes)
link_warp_kernel(const __grid_constant__ KernelArgs a)
{
    if (!can_chunk(a) || nothing_changed(a)) return;
    const int lane = threadIdx.x & (kLanes - 1), warp = threadIdx.x / kLanes;
    const int64_t t = (int64_t)blockIdx.x * kLinkWarps + warp;
    if (t >= (int64_t)a.B * (a.K - 1)) return;
    const size_t B = (size_t)a.B;
    const int64_t b = t % a.B;
    const int32_t j = (int32_t)(t / a.B) + 1;
    const size_t cell = (size_t)j * B + b;
    if (a.round != 0 && a.stamp[cell - B] != (uint8_t)a.round && a.stamp[cell] != (uint8_t)a.round) return;
    const size_t base = (size_t)warp * link_warp_bytes(a.T, a.G);
    const uint32_t x = (uint32_t)(base / sizeof(double));
    RelabelScratch s;
    s.z = x + a.T;
    s.last = s.z + a.T;
    s.perm = (uint32_t)(base + sizeof(double) * (2 * (size_t)a.T + (size_t)a.G));
    s.rank = s.perm + a.G;
    const int32_t q0 = j * a.seg_per_chunk;
    const double *Y = a.chunk_start + (size_t)j * a.T * B + b;
    const double tau = arrival_at(a, b, a.leaf_start[seg_leaf(a, q0)]);
    for (int k = lane; k < a.T; k += kLanes) {
        SM_F64(x + k) = a.seg_end[((size_t)(q0 - 1) * a.T + k) * B + b];
        SM_F64(s.z + k) = Y[(size_t)k * B];
    }
    __syncwarp();
    const auto info = [&](int g) { return a.group_info[(size_t)b * a.G + g]; };
    const auto X = [&](uint32_t k) { return SM_F64(x + k); };
    const auto Z = [&](uint32_t k) { return SM_F64(s.z + k); };
    bool ok = warp_equivalent(a.G, info, X, Z, tau), other = false;
    if (!ok && a.twins[b] &&
        warp_relabel(a.G, a.T, a.twin_class + (size_t)b * a.G, info, X, Y, B, s))
        ok = other = warp_equivalent(a.G, info, X, Z, tau);
    const size_t at = (size_t)q0 * B + b;
    if (other)
        for (int g = lane; g < a.G; g += kLanes) a.perm[at * a.G + g] = smem[s.perm + g];
    if (lane == 0) {
        a.link[cell] = ok;
        a.rel[at] = other ? kRelOther : 0;
        if (other) a.relabelled[b] = 1;
    }
}

// One thread per boundary, the first round where chunks are at least as long as the run-in: lists
// EVERY chunk behind a failed boundary, to be simulated again from the state that the run before
// it ended in, as stored.  That state has a run-in and a whole chunk of history and is usually the
// true one, although the one that the listed chunk's speculative run started from was not.  (While
// only the first chunk of each failed stretch was walked, and none of a candidate a third of
// whose boundaries fail, the rest was left to finish_kernel, one chunk after the other: 1500
// placements with 1 in 60 boundaries failing 9.1 ms, all at once 7.3; 700 grown ones on 32 devices,
// 1 in 4 failing, 17.8 and 13.3; a layer of 2343 59 and 47; 4096 on 64 devices 25.7 and 24.)
__global__ void restart_kernel(const __grid_constant__ KernelArgs a)
{
    if (!can_chunk(a)) return;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t B = (size_t)a.B;
    const size_t cell = (size_t)t + B;                   // chunk 0 is the true run
    const bool failed = t < (int64_t)a.B * (a.K - 1) && !a.link[cell];
    const uint32_t all = __ballot_sync(0xFFFFFFFFu, failed);
    if (!all) return;
    const int lane = threadIdx.x & (kLanes - 1);
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&a.work_count[a.round], (uint32_t)__popc(all));
    at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(all & ((1u << lane) - 1u));
    if (!failed) return;
    const int64_t b = t % a.B;
    const int32_t j = (int32_t)(t / a.B) + 1;
    a.work_items[at] = (uint32_t)cell;
    a.stamp[cell] = (uint8_t)(a.round + 1);
    a.open[b] = 1;
    if (a.resimulated) atomicAdd(&a.resimulated[b], 1);
    const double *X = a.seg_end + (size_t)(j * a.seg_per_chunk - 1) * a.T * B + b;
    double *Y = a.chunk_start + (size_t)j * a.T * B + b;
    for (int s = 0; s < a.T; ++s) Y[s * B] = X[s * B];
}

// One warp per candidate, the other rounds: lists the chunks behind a failed boundary that itself
// has a good one before it, and copies the state they start from.  The walk from there goes
// through the failed boundaries behind it.  A candidate a third of whose boundaries fail is left
// to finish_kernel: its walks would start from states that are wrong as well, and the call would
// wait for the longest of them twice.  (With them: 321 grown placements on 32 devices 5.5 -> 7.9
// ms, 450 on 64 24.6 -> 31, 42 on 64 6.6 -> 7.8, a sweep of 18 traces 24 -> 26.5, a search on 16 devices
// 71 -> 82; lists of random placements the same.)
__global__ void resolve_kernel(const __grid_constant__ KernelArgs a)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
    if (!can_chunk(a) || b >= a.B || nothing_changed(a)) return;
    const size_t B = (size_t)a.B;
    int32_t fails = 0;
    for (int32_t j = 1 + lane; j < a.K; j += kLanes) fails += !a.link[(size_t)j * B + b];
    fails = __reduce_add_sync(0xFFFFFFFFu, fails);
    if (lane == 0) a.open[b] = fails != 0;
    if (fails == 0 || (a.K > 8 && (int64_t)fails * 3 >= (int64_t)(a.K - 1))) return;
    int32_t listed = 0;
    for (int32_t j0 = 1; j0 < a.K; j0 += kLanes) {
        const int32_t j = j0 + lane;
        const bool head = j < a.K && !a.link[(size_t)j * B + b] && (j == 1 || a.link[(size_t)(j - 1) * B + b]);
        if (head) {
            a.work_items[atomicAdd(&a.work_count[a.round], 1u)] = (uint32_t)((int64_t)j * a.B + b);
            a.stamp[(size_t)j * B + b] = (uint8_t)(a.round + 1);
        }
        for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, head); todo; todo &= todo - 1, ++listed) {
            const int32_t k = j0 + __ffs((int)todo) - 1;
            const double *X = a.seg_end + (size_t)(k * a.seg_per_chunk - 1) * a.T * B + b;
            double *Y = a.chunk_start + (size_t)k * a.T * B + b;
            for (int s = lane; s < a.T; s += kLanes) Y[s * B] = X[s * B];
        }
    }
    if (a.resimulated && lane == 0 && listed) atomicAdd(&a.resimulated[b], listed);
}

// The speculative pass of a small batch: one warp per (chunk, candidate), by windows.
template <bool kLegacy, bool kTwins>
__global__ void __launch_bounds__(kWindowWarps * kLanes, kWindowBlocksPerSm)
window_stream_kernel(const __grid_constant__ KernelArgs a)
{
    window_stage_table<kLegacy>(a);
    if (a.N == 0) return;
    const bool chunked = can_chunk(a);
    // not chunked: one chunk holding every segment, plain sequential simulation
    KernelArgs ka = a;
    if (!chunked) ka.seg_per_chunk = a.NS;
    const int64_t items = (int64_t)a.B * (chunked ? a.K : 1);
    const int64_t step = (int64_t)gridDim.x * kWindowWarps;
    for (int64_t it = (int64_t)blockIdx.x * kWindowWarps + threadIdx.x / kLanes; it < items; it += step) {
        const int32_t j = (int32_t)(it / a.B);
        const int64_t b = it % a.B;
        Window w;
        window_setup<kLegacy, kTwins>(a, w, b);
        int32_t begin = 0;
        if (j > 0) {
            const int32_t first = a.leaf_start[seg_leaf(a, j * a.seg_per_chunk)];
            begin = first - a.warmup > 0 ? first - a.warmup : 0;
        }
        window_run<kLegacy, kTwins>(ka, w, kNoWalk, j, begin, chunked, j * a.seg_per_chunk);
        if (w.status) atomicOr(&a.status[b], w.status);
    }
}

// The chunks on the work list of this round, one to a warp, taken from the
// list as warps become free: each is re-simulated from the state the chunk before it ended in,
// and the chunks behind it as well, until the stored run can take over or the next listed
// chunk comes.  A round lasts as long as its longest walk, so what counts is how fast ONE
// candidate gets through its requests: a lane of the 32-candidate step takes 0.5 to 0.9 us a
// request, windows 0.1 to 0.4 us.
template <bool kLegacy, bool kTwins>
__global__ void __launch_bounds__(kWindowWarps * kLanes, kWindowBlocksPerSm)
walk_kernel(const __grid_constant__ KernelArgs a)
{
    const uint32_t count = a.work_count[a.round];
    if ((uint64_t)blockIdx.x * kWindowWarps >= count) return;
    window_stage_table<kLegacy>(a);
    const int lane = threadIdx.x & (kLanes - 1);
    for (;;) {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&a.work_next[a.round], 1u);
        at = __shfl_sync(0xFFFFFFFFu, at, 0);
        if (at >= count) return;
        const uint32_t item = a.work_items[at];
        const int32_t j = (int32_t)(item / (uint32_t)a.B);
        const int64_t b = item % (uint32_t)a.B;
        Window w;
        window_setup<kLegacy, kTwins>(a, w, b);
        const double *src = a.chunk_start + (size_t)j * a.T * a.B + b;
        for (int t = lane; t < a.T; t += kLanes) WIN_CLOCK(w, t) = src[(size_t)t * a.B];
        __syncwarp();
        const int32_t q0 = j * a.seg_per_chunk;
        window_run<kLegacy, kTwins>(a, w, kWalkRound, j, a.leaf_start[seg_leaf(a, q0)], true, q0);
        if (w.status) atomicOr(&a.status[b], w.status);
    }
}

// The labels of a candidate's segments, followed from one to the next by a warp: `pi` (u8[G] in
// shared memory) translates the labels of the segment at hand into group numbers.
struct Labels {
    uint32_t pi, tmp;                        // u8 indices; tmp: scratch of the same size
    const uint32_t *cls;                     // the candidate's classes of twins
    uint64_t moved;                          // classes in which pi is not the identity
};

__device__ inline void labels_reset(Labels &l, int G)
{
    __syncwarp();
    for (int g = threadIdx.x & (kLanes - 1); g < G; g += kLanes) smem[l.pi + g] = (uint8_t)g;
    l.moved = 0;
    __syncwarp();
}

// Into tmp: the translation behind `perm` (label -> label of the segment before).  Returns
// the classes in which it is not the identity.
__device__ inline uint64_t labels_through(const Labels &l, int G, const uint8_t *perm)
{
    __syncwarp();
    for (int g = threadIdx.x & (kLanes - 1); g < G; g += kLanes) smem[l.tmp + g] = smem[l.pi + perm[g]];
    __syncwarp();
    return moved_classes(l.cls, G, [&](int g) { return smem[l.tmp + g]; });
}

__device__ inline void labels_take(Labels &l, int G, uint64_t moved)
{
    __syncwarp();
    for (int g = threadIdx.x & (kLanes - 1); g < G; g += kLanes) smem[l.pi + g] = smem[l.tmp + g];
    l.moved = moved;
    __syncwarp();
}

// The list of swaps of a segment (KernelArgs::swap_mask), an entry per lane at a time.
struct Swaps {
    size_t cell;                             // entry 0
    int32_t count, base, next;               // base: entry in lane 0; next: the one peeked at
    int32_t first, at;                       // the segment's first request; this lane's entry
    uint32_t mask;
};

__device__ inline void swaps_load(const KernelArgs &a, Swaps &s, int32_t from)
{
    const int32_t k = from + (int32_t)(threadIdx.x & (kLanes - 1));
    s.base = from;
    s.at = 0x7FFFFFFF;
    s.mask = 0;
    if (k < s.count) {
        s.mask = a.swap_mask[s.cell + (size_t)k * a.B];
        s.at = s.first + a.swap_at[s.cell + (size_t)k * a.B];
    }
}

__device__ inline Swaps swaps_of(const KernelArgs &a, int64_t b, int32_t q, int32_t first)
{
    Swaps s;
    s.cell = (size_t)q * a.swap_cap * a.B + b;
    s.count = a.swap_count[(size_t)q * a.B + b];
    s.first = first;
    s.next = 0;
    swaps_load(a, s, 0);
    return s;
}

// The request of the next swap (behind the last one: 0x7FFFFFFF) and its mask.
__device__ inline int32_t swaps_peek(const KernelArgs &a, Swaps &s, uint32_t &mask)
{
    if (s.next - s.base == kLanes) swaps_load(a, s, s.next);
    mask = __shfl_sync(0xFFFFFFFFu, s.mask, s.next - s.base);
    return __shfl_sync(0xFFFFFFFFu, s.at, s.next - s.base);
}

// A choice between twins in the same state: the true one is the smallest group number among the
// labels of `mask` (ranks in the class of `mine`, the picked one); the label that has it changes
// places with the picked one.  Returns whether they did.
__device__ inline bool labels_swap(const KernelArgs &a, Labels &l, uint32_t mine, uint32_t mask)
{
    uint32_t key = 0xFFFFFFFFu;              // group << 8 | label
    for (int g = threadIdx.x & (kLanes - 1); g < a.G; g += kLanes)
        if (class_first(l.cls[g]) == class_first(l.cls[mine]) && class_rank(l.cls[g]) < 32 &&
            ((mask >> class_rank(l.cls[g])) & 1u)) {
            const uint32_t mapped = ((uint32_t)smem[l.pi + g] << 8) | (uint32_t)g;
            key = mapped < key ? mapped : key;
        }
    key = __reduce_min_sync(0xFFFFFFFFu, key);
    const uint32_t other = key & 0xFFu;
    if (other == mine) return false;
    __syncwarp();
    if ((threadIdx.x & (kLanes - 1)) == 0) {
        const uint8_t g = smem[l.pi + mine];
        smem[l.pi + mine] = (uint8_t)(key >> 8);
        smem[l.pi + other] = g;
    }
    __syncwarp();
    return true;
}

// First request of segment q.
__device__ inline int32_t segment_first(const KernelArgs &a, int32_t q)
{
    return seg_leaf(a, q) < a.num_leaves ? a.leaf_start[seg_leaf(a, q)] : (int32_t)a.N;
}

// Where the decision record of request i is.
__device__ inline size_t record_at(const KernelArgs &a, int64_t b, int32_t i)
{
    return ((size_t)(i >> 2) * a.dec_pitch + b) * 4 + (size_t)(i & 3);
}

// Follows the labels through segment q, which has swaps.  Returns whether they changed.
__device__ inline bool labels_follow(const KernelArgs &a, int64_t b, Labels &l, int32_t q)
{
    Swaps s = swaps_of(a, b, q, segment_first(a, q));
    bool changed = false;
    for (;; ++s.next) {
        uint32_t mask;
        const int32_t i = swaps_peek(a, s, mask);
        if (i == 0x7FFFFFFF) break;
        const uint32_t rec = a.dec_wide ? static_cast<uint16_t *>(a.decisions)[record_at(a, b, i)] & 0x7FFFu
                                        : static_cast<uint8_t *>(a.decisions)[record_at(a, b, i)] & 0x7Fu;
        if (rec && (class_bit(l.cls[rec - 1]) & l.moved)) changed |= labels_swap(a, l, rec - 1, mask);
    }
    if (changed) l.moved = moved_classes(l.cls, a.G, [&](int g) { return smem[l.pi + g]; });
    return changed;
}

// Translates the decision records of segment q into group numbers, 32 requests at a time, and
// follows the labels through the choices between twins in the same state (see warp_relabel).
// The records are strided over memory: what bounds this is the latency of the loads, so they are
// fetched four windows ahead (10 ms -> 1 ms for the 389 placements with twins of a list of 4096).
__device__ inline void name_segment(const KernelArgs &a, int64_t b, Labels &l, int32_t q)
{
    constexpr int kAhead = 4;
    const int lane = threadIdx.x & (kLanes - 1);
    const int32_t i0 = segment_first(a, q), i1 = segment_first(a, q + 1);
    const uint32_t flag = a.dec_wide ? 0x8000u : 0x80u;
    auto fetch = [&](int32_t base, uint32_t &rec) {
        const int32_t i = base + lane;
        rec = 0;
        if (i < i1)
            rec = a.dec_wide ? static_cast<uint16_t *>(a.decisions)[record_at(a, b, i)]
                             : static_cast<uint8_t *>(a.decisions)[record_at(a, b, i)];
    };
    Swaps swaps = swaps_of(a, b, q, i0);
    auto window = [&](int32_t base, uint32_t rec) {
        const uint32_t label = rec ? (rec & (flag - 1)) - 1 : 0u;
        const bool moves = rec && (class_bit(l.cls[label]) & l.moved);
        const uint32_t movers = __ballot_sync(0xFFFFFFFFu, moves);
        uint32_t group = label;
        int from = 0;
        bool changed = false;
        for (;;) {
            uint32_t mask;
            const int32_t i = swaps_peek(a, swaps, mask);
            const int k = i - base < kLanes ? i - base : kLanes;
            if (k < kLanes) ++swaps.next;
            if (k < kLanes && !((movers >> k) & 1u)) continue;
            if (lane >= from && lane < k && moves) group = smem[l.pi + label];
            if (k == kLanes) break;
            from = k;
            changed |= labels_swap(a, l, __shfl_sync(0xFFFFFFFFu, label, k), mask);
        }
        if (moves && group != label) {
            rec = (rec & flag) | (group + 1);
            const size_t at = record_at(a, b, base + lane);
            if (a.dec_wide) static_cast<uint16_t *>(a.decisions)[at] = (uint16_t)rec;
            else static_cast<uint8_t *>(a.decisions)[at] = (uint8_t)rec;
        }
        if (changed) {
            __syncwarp();
            l.moved = moved_classes(l.cls, a.G, [&](int g) { return smem[l.pi + g]; });
        }
    };
    uint32_t rec[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) fetch(i0 + u * kLanes, rec[u]);
    for (int32_t base = i0; base < i1 && l.moved; base += kAhead * kLanes) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const uint32_t r = rec[u];
            fetch(base + (u + kAhead) * kLanes, rec[u]);
            if (l.moved) window(base + u * kLanes, r);
        }
    }
}

constexpr int kNameWarps = 4;
constexpr int kNameSegments = 8;             // segments to a warp, at most 32
// Segments of a call up to which each has a warp of its own: they all run at once then.
constexpr int64_t kNameAlone = 148 * 64;

// The segments that finish_kernel left to be named: a warp per stretch of `segments`, each
// with the labels noted for its start.  (finish_kernel did this itself, in order: 27 ns a request
// and candidate, 4 ms for one placement over 150 000 requests; it now follows the labels through
// the lists of swaps alone.)
__global__ void __launch_bounds__(kNameWarps * kLanes)
name_kernel(const __grid_constant__ KernelArgs a, const int32_t segments)
{
    const int lane = threadIdx.x & (kLanes - 1);
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
    const int32_t parts = (a.NS + segments - 1) / segments;
    const int64_t b = w / parts;
    if (!can_chunk(a) || b >= a.B || !a.relabelled[b]) return;
    const size_t B = (size_t)a.B;
    const int32_t q0 = (int32_t)(w % parts) * segments, s = q0 + lane;
    const bool mine = lane < segments && s < a.NS && a.rel[(size_t)s * B + b] == kRelNamed;
    Labels l;
    l.pi = (threadIdx.x / kLanes) * (uint32_t)a.G;
    l.tmp = l.pi;
    l.cls = a.twin_class + (size_t)b * a.G;
    for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, mine); todo; todo &= todo - 1) {
        const int32_t q = q0 + __ffs((int)todo) - 1;
        const uint8_t *pi = a.perm + ((size_t)a.name_from[(size_t)q * B + b] * B + b) * a.G;
        __syncwarp();
        for (int g = lane; g < a.G; g += kLanes) smem[l.pi + g] = pi[g];
        __syncwarp();
        l.moved = moved_classes(l.cls, a.G, [&](int g) { return smem[l.pi + g]; });
        name_segment(a, b, l, q);
    }
}

// One warp per candidate that has an open boundary or relabelled segments: goes through the
// segments in order with the translation of their labels into group numbers, and notes it where
// name_kernel is to translate their records.  At a failed boundary, and at a segment in other labels in which a group number
// decided between different states, it walks from the true state (under the true labels)
// until what is stored can take over.  After it, every segment was simulated from a state
// equivalent to the true one under a translation that is exact for it: the result does
// not depend on the chunking or the rounds.
//
// kBlocks: blocks an SM has registers for.  The walk wants more than the 168 that three leave a
// thread: with two, 31 traces of 16 devices are walked in 13.4 ms instead of 14.5, 137 placements on 64
// devices in 26.4 instead of 27.7.  Where not all blocks find a place then, a second wave is slower
// (a layer of 2343: 7.2 ms instead of 5.0), and without labels and a group per lane 168 are enough
// (40 traces of 32 devices 35.3 and 36.2 ms).
constexpr int kFinishBlocksPerSm = 2;
template <bool kLegacy, bool kTwins, int kBlocks>
__global__ void __launch_bounds__(kWindowWarps * kLanes, kBlocks)
finish_kernel(const __grid_constant__ KernelArgs a)
{
    if (!can_chunk(a) || a.N == 0) return;
    const int lane = threadIdx.x & (kLanes - 1);
    const int64_t b = (int64_t)blockIdx.x * kWindowWarps + threadIdx.x / kLanes;
    const bool mine = b < a.B && (a.open[b] || a.relabelled[b]);
    if (!__syncthreads_or(mine)) return;
    window_stage_table<kLegacy>(a);
    if (!mine) return;
    const size_t B = (size_t)a.B;
    Window w;
    window_setup<kLegacy, kTwins>(a, w, b);
    Labels l;
    l.pi = w.labels;
    l.tmp = w.re.perm;
    // (window_setup's copy on chip as well, but through a pointer into shared memory the whole kernel
    // is 3 % slower: 256 traces of 64 devices 54.5 ms instead of 52.9)
    l.cls = a.twin_class + (size_t)b * a.G;
    labels_reset(l, a.G);
    int32_t q = a.seg_per_chunk;             // chunk 0 is the true run
    int32_t noted = -1;                      // segment in whose `perm` l.pi is noted
    // segments [q, q + n) are to be named with l.pi at their start
    auto note = [&](int32_t n) {
        if (!kTwins || !l.moved) return;
        __syncwarp();
        if (noted < 0) {
            noted = q;
            for (int g = lane; g < a.G; g += kLanes) a.perm[((size_t)q * B + b) * a.G + g] = smem[l.pi + g];
        }
        if (lane < n) {
            a.rel[(size_t)(q + lane) * B + b] = kRelNamed;
            a.name_from[(size_t)(q + lane) * B + b] = noted;
        }
        __syncwarp();
    };
    while (q < a.NS) {
        // the first of 32 segments in which something happens; those before it keep the labels
        // (each lane keeps what it loads: an event is a chain of loads as it is)
        const int32_t s = q + lane;
        bool event = false, linked = true;
        uint8_t rel = 0, swap_count = 0;
        uint64_t tie = 0;
        if (s < a.NS) {
            const size_t at = (size_t)s * B + b;
            linked = s % a.seg_per_chunk != 0 || a.link[(size_t)(s / a.seg_per_chunk) * B + b];
            event = !linked;
            if constexpr (kTwins) {
                rel = a.rel[at];
                swap_count = a.swap_count[at];
                tie = a.tie[at];
                event |= rel || (l.moved && (swap_count || (tie & l.moved)));
            }
        }
        const uint32_t todo = __ballot_sync(0xFFFFFFFFu, event);
        int32_t quiet = todo ? __ffs((int)todo) - 1 : kLanes;
        if (quiet > a.NS - q) quiet = a.NS - q;
        if (quiet) note(quiet);              // (the labels in front of an event are still to be read)
        q += quiet;
        if (!todo) continue;
        const size_t cell = (size_t)q * B + b;
        const int32_t j = q / a.seg_per_chunk;
        const bool first = q % a.seg_per_chunk == 0;
        if (__shfl_sync(0xFFFFFFFFu, linked, quiet)) {
            uint64_t moved = l.moved;
            const bool other = __shfl_sync(0xFFFFFFFFu, rel, quiet) != 0;
            if (other) moved = labels_through(l, a.G, a.perm + cell * a.G);
            if (!(moved & __shfl_sync(0xFFFFFFFFu, tie, quiet))) {
                if (other) {
                    labels_take(l, a.G, moved);
                    noted = -1;
                }
                note(1);
                if (l.moved && __shfl_sync(0xFFFFFFFFu, swap_count, quiet) && labels_follow(a, b, l, q)) noted = -1;
                ++q;
                continue;
            }
        }
        // from the true state, under the true labels (l.pi is still that of segment q - 1)
        for (int g = lane; g < a.G; g += kLanes) {
            const uint32_t from = SM_U32(w.info + g), to = SM_U32(w.info + smem[l.pi + g]);
            for (uint32_t k = 0; k < ((from >> 8) & 0xFFu); ++k)
                WIN_CLOCK(w, (to & 0xFFu) + k) =
                    a.seg_end[((size_t)(q - 1) * a.T + (from & 0xFFu) + k) * B + b];
        }
        __syncwarp();
        if (first)
            for (int t = lane; t < a.T; t += kLanes)
                a.chunk_start[((size_t)j * a.T + t) * B + b] = WIN_CLOCK(w, t);
        if (lane == 0) {
            a.rel[cell] = 0;
            if (a.resimulated) atomicAdd(&a.resimulated[b], 1);
        }
        __syncwarp();
        // (nothing is noted about choices between twins: nobody compares with these segments again)
        const int32_t e = window_run<kLegacy, kTwins, false>(a, w, kWalkChain, j, a.leaf_start[seg_leaf(a, q)], true, q);
        labels_reset(l, a.G);
        noted = -1;
        q = e;
    }
    if (w.status) atomicOr(&a.status[b], w.status);
}

// Stack machine over leaves [l0, l1) of candidate b: their sums combined in numpy's
// pairing order as far as the merges stay inside the range (a subtree).
__device__ inline double sum_subtree(const KernelArgs &a, int64_t b, const uint8_t *leaf_merges,
                                     int32_t l0, int32_t l1, bool &bad)
{
    double stack[kMaxSumDepth];
    int sp = 0;
    for (int32_t base = l0; base < l1; base += 8) {
        double v[8];
        uint8_t mg[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {            // fetched together, so that the loads overlap
            const int32_t leaf = base + u < l1 ? base + u : l1 - 1;
            v[u] = a.leaf_sums[(size_t)leaf * a.B + b];
            mg[u] = leaf_merges[leaf];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (base + u >= l1) break;
            if (sp < kMaxSumDepth) stack[sp] = v[u];
            ++sp;
            // the merges behind a subtree's last leaf that reach beyond it are its parents'
            for (int k = mg[u]; k > 0 && sp >= 2; --k) {
                --sp;
                if (sp < kMaxSumDepth) stack[sp - 1] = stack[sp - 1] + stack[sp];
            }
        }
    }
    bad |= sp > kMaxSumDepth;
    return sp > 0 ? stack[0] : 0.0;
}

// The latency sum of candidate b in numpy's pairing order (controller.py:402 consumes the
// mean), by the lanes of a warp: numpy splits n elements at n / 2 rounded down to a multiple
// of eight while there are more than 128, so the first levels of the tree are known from N
// alone and lane k sums the k-th of up to 32 subtrees; the levels above are left + right.
// (One thread alone took 125 us for 256 leaves: a dependent chain of loads.)
__device__ inline void sum_leaves(const KernelArgs &a, int64_t b, const uint8_t *leaf_merges,
                                  double *latency_sum)
{
    const int lane = threadIdx.x & (kLanes - 1);
    int depth = 0;                                   // every node above this level is split
    while (depth < 5 && (a.N >> (depth + 1)) > 160) ++depth;
    int64_t base = 0, n = a.N;
    for (int d = depth - 1; d >= 0; --d) {
        int64_t half = n / 2;
        half -= half % 8;
        if ((lane >> d) & 1) { base += half; n -= half; } else n = half;
    }
    bool bad = false;
    double v = 0.0;
    if (lane < (1 << depth)) {
        const int32_t l0 = leaf_lower_bound(a.leaf_start, a.num_leaves, base);
        const int32_t l1 = leaf_lower_bound(a.leaf_start, a.num_leaves, base + n);
        v = sum_subtree(a, b, leaf_merges, l0, l1, bad);
    }
    for (int d = 0; d < depth; ++d) {
        const double right = __shfl_down_sync(0xFFFFFFFFu, v, 1 << d);
        if ((lane & ((2 << d) - 1)) == 0) v = v + right;
    }
    if (bad) atomicOr(&a.status[b], MMS_STATUS_BAD_INDEX);
    if (lane == 0) latency_sum[b] = v;
}

// The batching simulator's reductions, one warp per candidate: the latency sum, the total
// of the good requests (controller.py:401) from the per-model counts, and the requests of each
// model that has a replica.
__global__ void finalize_kernel(const KernelArgs a, const uint8_t *leaf_merges, const int32_t *first_of,
                                const int32_t *model_num_good, int32_t *model_num_requests,
                                int64_t *good_total, double *latency_sum)
{
    const int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
    if (b >= a.B) return;
    sum_leaves(a, b, leaf_merges, latency_sum);
    int32_t total = 0;
    const uint16_t *off = a.model_off + (size_t)b * (a.M + 1);
    for (int m = threadIdx.x & (kLanes - 1); m < a.M; m += kLanes) {
        total += model_num_good[(size_t)b * a.M + m];
        model_num_requests[(size_t)b * a.M + m] = a.N > 0 && off[m + 1] > off[m] ? first_of[m + 1] - first_of[m] : 0;
    }
    total = __reduce_add_sync(0xFFFFFFFFu, total);
    if ((threadIdx.x & (kLanes - 1)) == 0) good_total[b] = total;
}

// Tallies the recorded decisions of the runs that count (controller.py:587,
// 611, 617-618).  A warp handles 32 consecutive scored candidates (one per
// lane, so their decisions of one request are one 64-byte access) over a
// range of at most 32 segments (fewer than 65 536 requests); each lane counts
// in its own 16-bit shared-memory histograms and adds them to the
// outputs (good_total among them), which must be zero on entry.  32 more rows
// of blocks (the first ones) form the candidates' latency sums beside the tally, a warp each.
template <typename Dec>
__global__ void __launch_bounds__(kLanes)
count_kernel(const KernelArgs a, int32_t seg_per_block, bool group_good, int32_t *model_num_good,
             int32_t *group_num_requests, int32_t *group_num_good, int64_t *good_total,
             const uint8_t *leaf_merges, double *latency_sum)
{
    if (blockIdx.y < kLanes) {
        const int64_t c = (int64_t)blockIdx.x * kLanes + blockIdx.y;
        if (c < a.B) sum_leaves(a, c, leaf_merges, latency_sum);
        return;
    }
    constexpr int kAcceptedBit = 8 * sizeof(Dec) - 1;
    constexpr uint32_t kAccepted = 1u << kAcceptedBit;
    // per lane: a 32-bit word per group (requests in the low half, good ones in
    // the high half: one update per record) at [group][lane], and 16-bit counts
    // of good requests per model at [model / 2][lane][model % 2] — every lane
    // stays in a bank of its own whatever it counts
    extern __shared__ uint32_t hist[];
    uint32_t *grp = hist;
    uint32_t *modw = hist + (size_t)a.G * kLanes;          // two 16-bit counts to a word
    uint16_t *mod = reinterpret_cast<uint16_t *>(modw);
    const int lane = threadIdx.x;
    const int64_t b = (int64_t)blockIdx.x * kLanes + lane;
    for (int g = 0; g < a.G; ++g) grp[g * kLanes + lane] = 0;
    for (int h = 0; h < (a.M + 1) / 2; ++h)
        reinterpret_cast<uint32_t *>(mod)[h * kLanes + lane] = 0;
    if (b >= a.B || a.num_leaves == 0) return;
    const size_t tb = trace_base(a, b);
    const int32_t q0 = (blockIdx.y - kLanes) * seg_per_block;
    const int32_t q1 = q0 + seg_per_block < a.NS ? q0 + seg_per_block : a.NS;
    for (int32_t q = q0; q < q1; ++q) {
        // four consecutive requests of a candidate are one aligned group of records
        struct alignas(4 * sizeof(Dec)) Quad { Dec r[4]; };
        const Quad *col = static_cast<const Quad *>(a.decisions) + b;
        const int32_t i_begin = a.leaf_start[seg_leaf(a, q)];
        const int32_t i1 = seg_leaf(a, q + 1) < a.num_leaves ? a.leaf_start[seg_leaf(a, q + 1)]
                                                             : (int32_t)a.N;
        // four groups (sixteen requests) at a time, so that their loads are in flight
        // together; segments start at multiples of 8
        constexpr int kQuads = 4;
        for (int32_t i0 = i_begin; i0 < i1; i0 += 4 * kQuads) {
            Quad d[kQuads];
            int32_t m[4 * kQuads];
#pragma unroll
            for (int u = 0; u < kQuads; ++u) {
                const int32_t i = i0 + 4 * u < i1 ? i0 + 4 * u : i0;
                d[u] = col[(size_t)(i >> 2) * a.dec_pitch];
            }
#pragma unroll
            for (int u = 0; u < 4 * kQuads; ++u) {
                const int32_t i = i0 + u < i1 ? i0 + u : i1 - 1;
                m[u] = a.model_ids[(size_t)i * a.trace_pitch + tb];
            }
            const int32_t valid = i1 - i0;
#pragma unroll
            for (int u = 0; u < 4 * kQuads; ++u) {
                const uint32_t rec = d[u >> 2].r[u & 3];
                if (u >= valid || rec == 0) continue;
                const uint32_t g = (rec & (kAccepted - 1)) - 1;
                const uint32_t accepted = rec >> kAcceptedBit;
                // shared-memory atomics whose result nobody reads: one instruction each and
                // nothing to wait for, where load + add + store was a dependent chain (a lane
                // only ever meets its own words, so there is no contention)
                atomicAdd(&grp[g * kLanes + lane], 1u + (accepted << 16));
                if (accepted)
                    atomicAdd(&modw[((uint32_t)m[u] >> 1) * kLanes + lane], 1u << (16 * (m[u] & 1)));
            }
        }
    }
    uint32_t accepted = 0;
    for (int m = 0; m < a.M; ++m) {
        const uint32_t k = mod[((m >> 1) * kLanes + lane) * 2 + (m & 1)];
        if (k) {
            atomicAdd(&model_num_good[(size_t)b * a.M + m], (int32_t)k);
            accepted += k;
        }
    }
    if (accepted)
        atomicAdd(reinterpret_cast<unsigned long long *>(good_total + b), (unsigned long long)accepted);
    for (int g = 0; g < a.G; ++g) {
        const uint32_t r = grp[g * kLanes + lane] & 0xFFFFu, k = grp[g * kLanes + lane] >> 16;
        if (r) atomicAdd(&group_num_requests[(size_t)b * a.G + g], (int32_t)r);
        if (group_good && k) atomicAdd(&group_num_good[(size_t)b * a.G + g], (int32_t)k);
    }
}

// The same for few candidates, whose lanes count_kernel would leave idle: a block takes 1024
// consecutive requests of one, four to a thread.  The first B blocks form the latency sums.  A thread
// reads 4 bytes of a sector, which is why this is for few: 57 600 requests of one candidate 55 -> 10 us,
// 30 000 of 37 46 -> 8 us.
constexpr int kCountThreads = 256;
constexpr int kCountFew = 64;
template <typename Dec>
__global__ void __launch_bounds__(kCountThreads)
count_few_kernel(const KernelArgs a, bool group_good, int32_t *model_num_good, int32_t *group_num_requests,
                 int32_t *group_num_good, int64_t *good_total, const uint8_t *leaf_merges, double *latency_sum)
{
    if ((int)blockIdx.x < a.B) {
        if (threadIdx.x < kLanes) sum_leaves(a, blockIdx.x, leaf_merges, latency_sum);
        return;
    }
    constexpr int kAcceptedBit = 8 * sizeof(Dec) - 1;
    extern __shared__ uint32_t hist[];               // [G] requests, [G] good, [M] good, good in all
    const int cells = 2 * a.G + a.M + 1;
    for (int c = threadIdx.x; c < cells; c += blockDim.x) hist[c] = 0;
    __syncthreads();
    const int64_t block = blockIdx.x - a.B;
    const int64_t b = block % a.B;
    const int64_t i0 = (block / a.B * kCountThreads + threadIdx.x) * 4;
    if (i0 < a.N) {
        struct alignas(4 * sizeof(Dec)) Quad { Dec r[4]; };
        const Quad d = static_cast<const Quad *>(a.decisions)[(size_t)(i0 >> 2) * a.dec_pitch + b];
        const size_t tb = trace_base(a, b);
        uint32_t good = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t rec = i0 + u < a.N ? d.r[u] : 0u;
            if (!rec) continue;
            const uint32_t g = (rec & ((1u << kAcceptedBit) - 1)) - 1;
            atomicAdd(&hist[g], 1u);
            if (rec >> kAcceptedBit) {
                atomicAdd(&hist[a.G + g], 1u);
                atomicAdd(&hist[2 * a.G + a.model_ids[(size_t)(i0 + u) * a.trace_pitch + tb]], 1u);
                ++good;
            }
        }
        if (good) atomicAdd(&hist[cells - 1], good);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < cells; c += blockDim.x) {
        const uint32_t n = hist[c];
        if (!n) continue;
        if (c < a.G) atomicAdd(&group_num_requests[(size_t)b * a.G + c], (int32_t)n);
        else if (c < 2 * a.G) { if (group_good) atomicAdd(&group_num_good[(size_t)b * a.G + (c - a.G)], (int32_t)n); }
        else if (c < 2 * a.G + a.M) atomicAdd(&model_num_good[(size_t)b * a.M + (c - 2 * a.G)], (int32_t)n);
        else atomicAdd(reinterpret_cast<unsigned long long *>(good_total + b), (unsigned long long)n);
    }
}

// Per-model request counts, plus the number of positions where the arrival
// times are not finite or go backwards (hist[M]).
__global__ void histogram_kernel(const double *arrivals, const int32_t *model_ids, int64_t N,
                                 int32_t M, int32_t *hist)
{
    extern __shared__ int32_t local[];
    for (int m = threadIdx.x; m <= M; m += blockDim.x) local[m] = 0;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += stride) {
        const int32_t m = model_ids[i];
        if (m >= 0 && m < M) atomicAdd(&local[m], 1);
        const double t = arrivals[i];
        const bool bad = !(t - t == 0.0) || (i > 0 && !(arrivals[i - 1] <= t));
        if (bad) atomicAdd(&local[M], 1);
    }
    __syncthreads();
    for (int m = threadIdx.x; m <= M; m += blockDim.x)
        if (local[m]) atomicAdd(&hist[m], local[m]);
}

// The same for T traces stored request-major ([N][T]): hist[t][M + 1], and the
// total of the bad positions of all traces in hist[T * (M + 1)].  A block
// covers 32 traces (threadIdx.x) and a slice of the requests (blockIdx.y).
__global__ void histogram_traces_kernel(const double *arrivals, const int32_t *model_ids, int64_t N,
                                        int32_t T, int32_t M, int32_t *hist)
{
    extern __shared__ int32_t local[];      // [32][M + 1]
    const int lane = threadIdx.x, row = threadIdx.y;
    for (int k = row * 32 + lane; k < 32 * (M + 1); k += 32 * blockDim.y) local[k] = 0;
    __syncthreads();
    const int64_t t = (int64_t)blockIdx.x * 32 + lane;
    const int64_t step = (int64_t)gridDim.y * blockDim.y;
    if (t < T) {
        for (int64_t i = (int64_t)blockIdx.y * blockDim.y + row; i < N; i += step) {
            const int32_t m = model_ids[(size_t)i * T + t];
            if (m >= 0 && m < M) atomicAdd(&local[lane * (M + 1) + m], 1);
            const double x = arrivals[(size_t)i * T + t];
            const bool bad = !(x - x == 0.0) || (i > 0 && !(arrivals[(size_t)(i - 1) * T + t] <= x));
            if (bad) atomicAdd(&local[lane * (M + 1) + M], 1);
        }
    }
    __syncthreads();
    for (int k = row * 32 + lane; k < 32 * (M + 1); k += 32 * blockDim.y) {
        const int64_t tt = (int64_t)blockIdx.x * 32 + k / (M + 1);
        if (local[k] && tt < T) {
            atomicAdd(&hist[tt * (M + 1) + k % (M + 1)], local[k]);
            if (k % (M + 1) == M) atomicAdd(&hist[(size_t)T * (M + 1)], local[k]);
        }
    }
}

// The same for T traces stored one after the other ([T][N]): a block covers a slice of
// one trace.
__global__ void histogram_rows_kernel(const double *arrivals, const int32_t *model_ids, int64_t N,
                                      int32_t T, int32_t M, int32_t *hist)
{
    extern __shared__ int32_t local[];
    for (int m = threadIdx.x; m <= M; m += blockDim.x) local[m] = 0;
    __syncthreads();
    const int64_t t = blockIdx.x;
    const double *at = arrivals + t * N;
    const int32_t *id = model_ids + t * N;
    const int64_t step = (int64_t)gridDim.y * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; i < N; i += step) {
        const int32_t m = id[i];
        if (m >= 0 && m < M) atomicAdd(&local[m], 1);
        const double x = at[i];
        if (!(x - x == 0.0) || (i > 0 && !(at[i - 1] <= x))) atomicAdd(&local[M], 1);
    }
    __syncthreads();
    for (int m = threadIdx.x; m <= M; m += blockDim.x)
        if (local[m]) {
            atomicAdd(&hist[t * (M + 1) + m], local[m]);
            if (m == M) atomicAdd(&hist[(size_t)T * (M + 1)], local[m]);
        }
}

// Pads trace t of T traces stored one after the other ([T][N]) behind its lengths[t] requests,
// as pack_traces_kernel does.
__global__ void pad_traces_kernel(const int64_t *lengths, int64_t N, double *arrivals,
                                  int32_t *model_ids, float *slos)
{
    const int64_t t = blockIdx.x, n = lengths[t];
    const double last = n > 0 ? arrivals[t * N + n - 1] : 0.0;
    for (int64_t i = n + (int64_t)blockIdx.y * blockDim.x + threadIdx.x; i < N;
         i += (int64_t)gridDim.y * blockDim.x) {
        arrivals[t * N + i] = last;
        model_ids[t * N + i] = -1;
        slos[t * N + i] = 0.0f;
    }
}

// T traces given one after the other (trace t = elements [offsets[t],
// offsets[t + 1]) of the three arrays) -> the request-major batch the kernels
// read ([N][T], see mms_trace.num_traces), shorter traces padded with requests
// of model -1 that repeat the trace's last arrival time.  A block moves a tile
// of 32 requests x 32 traces through shared memory, so that both the reads
// (along a trace) and the writes (across traces) are coalesced.
__global__ void __launch_bounds__(32 * 8)
pack_traces_kernel(const double *arrivals, const int32_t *model_ids, const float *slos,
                   const int64_t *offsets, int64_t T, int64_t N, double *out_arrivals,
                   int32_t *out_model_ids, float *out_slos)
{
    __shared__ double s_arr[32][33];
    __shared__ int32_t s_mid[32][33];
    __shared__ float s_slo[32][33];
    const int64_t i0 = (int64_t)blockIdx.x * 32, t0 = (int64_t)blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += 8) {          // row r of the tile: trace t0 + r
        const int64_t t = t0 + r, i = i0 + threadIdx.x;
        double a = 0.0;
        int32_t m = -1;
        float s = 0.0f;
        if (t < T) {
            const int64_t lo = offsets[t], n = offsets[t + 1] - lo;
            if (i < n) { a = arrivals[lo + i]; m = model_ids[lo + i]; s = slos[lo + i]; }
            else if (n > 0) a = arrivals[lo + n - 1];
        }
        s_arr[r][threadIdx.x] = a; s_mid[r][threadIdx.x] = m; s_slo[r][threadIdx.x] = s;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8) {          // request i0 + r, trace t0 + threadIdx.x
        const int64_t i = i0 + r, t = t0 + threadIdx.x;
        if (i < N && t < T) {
            out_arrivals[i * T + t] = s_arr[threadIdx.x][r];
            out_model_ids[i * T + t] = s_mid[threadIdx.x][r];
            out_slos[i * T + t] = s_slo[threadIdx.x][r];
        }
    }
}

// The search's selection over one shard of candidates: the score of
// base_policy.py:225-226 from the reductions (goodput - latency_mean / 10000 +
// num_replicas / 1000000, the same fp64 operations in the same order as the
// host forms it), and the FIRST maximum as np.argmax returns it
// (model_parallelism.py:349-351).  One block; best = {score, global index as a
// double}.  With `accumulate` the pair already in `best` competes too (a batch
// scored in several calls), the smaller index winning a tie.
constexpr int kArgmaxThreads = 256;

__global__ void __launch_bounds__(kArgmaxThreads)
argmax_scores_kernel(const int64_t *good_total, const double *latency_sum,
                     const int64_t *num_replicas, int64_t N, int32_t B, const int64_t *index_map,
                     int64_t index_base, bool accumulate, double *best)
{
    __shared__ double s_score[kArgmaxThreads];
    __shared__ double s_index[kArgmaxThreads];
    double top = -kInf, top_i = 9007199254740992.0;     // 2^53: behind every real index
    for (int32_t b = threadIdx.x; b < B; b += kArgmaxThreads) {
        const double n = (double)N;
        const double goodput = (double)good_total[b] / n;
        const double latency_mean = latency_sum[b] / n;
        double score = goodput - latency_mean / 10000.0;
        if (num_replicas) score = score + (double)num_replicas[b] / 1000000.0;
        const double idx = (double)(index_base + (index_map ? index_map[b] : (int64_t)b));
        if (score > top || (score == top && idx < top_i)) { top = score; top_i = idx; }
    }
    s_score[threadIdx.x] = top;
    s_index[threadIdx.x] = top_i;
    __syncthreads();
    for (int w = kArgmaxThreads / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            const double o = s_score[threadIdx.x + w], oi = s_index[threadIdx.x + w];
            if (o > s_score[threadIdx.x] || (o == s_score[threadIdx.x] && oi < s_index[threadIdx.x])) {
                s_score[threadIdx.x] = o;
                s_index[threadIdx.x] = oi;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        double sc = s_score[0], si = s_index[0];
        if (accumulate && (best[0] > sc || (best[0] == sc && best[1] < si))) { sc = best[0]; si = best[1]; }
        best[0] = sc;
        best[1] = si;
    }
}

}  // namespace mms

#include "mms_abi.inl"
