// mms_abi.inl — host side of the C ABI (included at the end of mms_sim.cu).
namespace mms {

thread_local char g_last_error[256] = "";

static int cuda_fail(cudaError_t e, const char *what)
{
    snprintf(g_last_error, sizeof(g_last_error), "%s: %s", what, cudaGetErrorString(e));
    return MMS_ERR_CUDA;
}

#define MMS_CUDA(call)                                             \
    do {                                                           \
        cudaError_t e_ = (call);                                   \
        if (e_ != cudaSuccess) return mms::cuda_fail(e_, #call);   \
    } while (0)

// numpy's pairwise split of n elements starting at `base`.
static void plan_rec(int64_t base, int64_t n, int32_t *leaf_start, uint8_t *merges, int32_t &count)
{
    if (n <= 128) {
        if (leaf_start) { leaf_start[count] = (int32_t)base; merges[count] = 0; }
        ++count;
        return;
    }
    int64_t half = n / 2;
    half -= half % 8;
    plan_rec(base, half, leaf_start, merges, count);
    plan_rec(base + half, n - half, leaf_start, merges, count);
    if (merges) merges[count - 1] += 1;
}

static int32_t plan_leaves(int64_t n)
{
    if (n <= 0) return 0;
    int32_t count = 0;
    plan_rec(0, n, nullptr, nullptr, count);
    return count;
}

struct Geometry {
    int32_t K, NS, seg_len, seg_per_chunk, warmup, lat_smem_elems, rounds,
        block_warps, lat_f64, window_blocks, win_table_elems;
    bool window, restart, finish_at_once;     // finish_at_once: see kFinishBlocksPerSm
    size_t smem_stream, smem_window;
    size_t off_leaf, off_seg_end, off_chunk_start, off_decisions, off_work_count, off_work_items,
        off_rows, off_seg_leaf, off_group_info, off_columns, off_stamp, off_link, off_flags, off_rel,
        off_tie, off_swap_mask, off_swap_at, off_swap_count, off_name_from, off_perm, off_twin_class, off_group_column, off_group_models;
    int32_t group_words, swap_cap, row_planes;
    size_t smem_count;        // shared memory of count_kernel
    size_t total;
};

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Is the call faster with one candidate per warp in the speculative pass than with 32?  A warp of
// the former takes 0.15 to 0.2 us a request when it is alone on its scheduler and up to 0.4
// us beside two others; a warp of the latter 0.5 us alone and 0.9 us beside eleven on its SM, but
// for 32 candidates: one candidate per warp pays while the GPU is short of candidates.
// Estimated microseconds of both passes.
//
// What follows the pass counts too: `worth`, below.
static bool window_pays(int64_t N, int64_t B, int64_t K_wide, int64_t K_win, int64_t warm, int sm_count,
                        double worth)
{
    const double n_win = (double)N / K_win + (K_win > 1 ? warm : 0);
    const double n_wide = (double)N / K_wide + (K_wide > 1 ? warm : 0);
    const double warps_win = (double)B * K_win / (4.0 * sm_count);
    const double t_win = n_win * (warps_win <= 1.0 ? 0.18 : 0.18 + 0.11 * (warps_win - 1.0));
    double share = (double)((B + 31) / 32) * K_wide / (12.0 * sm_count);
    if (share > 1.0) share = 1.0;
    return t_win < worth * n_wide * (0.5 + 0.4 * share);
}

// How many times as long the pass with one candidate per warp may take, by that estimate.  It goes with
// longer chunks, so fewer boundaries fail, and with a longer run-in where there are many groups (plan_call),
// and the walks behind failed boundaries are often most of the call; by how much depends on how
// many groups there are to get out of order, and the more candidates, the less a failed one stands alone.
// Where single devices are among the groups ("whole": as many groups as slots, the lists a search makes over all
// partitions) that is most, in a few deep pipelines least.
//
// Measured: 3 664 lists of 1 to 800 placements (random, grown over all partitions and over one; 4 to 32
// devices, 2 000 to 150 000 requests), both passes for each, 32 to a warp / one.  In geometric
// mean, lists slower than 0.95 times: up to four stages, whole, fewer than 128 placements 1.87 and 1 %, more of them
// 1.56 and 1 %; more than a group to three slots 1.48 and 1 %, fewer 1.29 and 2 %; deeper ones, whole
// 1.51 and 2 %; on up to 8 slots 1.34 and 4 %.  Just behind these lines, up to half as much again, 25 to 50 % of
// the lists are slower: 445 placements of two pipelines of four over 10 000 requests 0.47 / 1.17 ms, 262 random ones
// on 16 devices over 12 000 3.4 / 7.1 (deep, 12 groups: no line at all, as in general on 16 slots and more).
// (Of 2 267 further lists 1 211 are inside these lines: 1.57 times as fast in the mean, 0.8 % of them slower than
// 0.95 times, the slowest 0.81.)
// Not on more than 32 slots (280 grown placements on 64 devices, 30 000 requests 14.1 / 18.5) and not
// in the two calls of a list that is split (1025 placements on 16 devices 3.7 / 4.7), which pass
// MMS_FLAG_CROWDED.  The two parts of a list that goes out pipelined, and the groups of a sweep, do
// not pass it: 754 such lists on 4 to 32 devices are 0.74 to 1.04 times as fast with it, 0.99 in the mean, 143
// sweeps 0.75 to 1.04.
static double window_worth(const mms_placements *c, int64_t B, uint32_t flags)
{
    const int32_t T = c->max_slots, G = c->max_groups;
    if (flags & MMS_FLAG_CROWDED || T > 32) return 1.0;
    const bool whole = G >= T, few = B < 128;
    if (c->max_stages <= kGroupDepth) {
        if (whole) return few ? 4.0 : c->max_stages == 1 || T > 8 ? 3.0 : 2.0;
        return 3 * G > T ? (few ? 2.5 : 2.0) : 1.5;
    }
    if (whole) return few || T > 8 ? 2.0 : 1.5;
    if (T > 8) return 1.0;
    return few && 2 * G > T ? 2.0 : 1.25;
}

// Chunking, shared-memory and scratch geometry of one call.  `thrift` > 0 asks for less scratch at
// the price of speed (never of results): 1 = long segments and chunks, 2 = also no bookkeeping of
// interchangeable groups, 3 = also few chunks.
constexpr int kMaxThrift = 3;
constexpr int kMaxRowReplicas = 64;      // of a model in the replica rows
static int plan_call(int64_t N, const mms_placements *c, const mms_sim_options *opts,
                     uint32_t flags, bool group_good, int thrift, Geometry *g)
{
    *g = Geometry();
    if (!c || N < 0 || c->num_candidates < 0 || c->num_models < 0 || c->max_groups < 0 ||
        c->max_placed < 0 || c->max_slots < 0 || c->max_stages < 1 || c->num_columns < 0)
        return MMS_ERR_ARG;
    if (N > 0x7FFFFFFF) return MMS_ERR_UNSUPPORTED;
    if (c->max_groups > MMS_MAX_GROUPS || c->max_slots > MMS_MAX_SLOTS ||
        c->max_placed > MMS_MAX_PLACED || c->max_stages > MMS_MAX_STAGES ||
        c->num_columns > MMS_MAX_COLUMNS)
        return MMS_ERR_UNSUPPORTED;
    if ((flags & MMS_FLAG_LEGACY_CLOCK) && c->max_stages != 2) return MMS_ERR_ARG;
    if (c->num_scored < 0 || c->num_scored > c->num_candidates) return MMS_ERR_ARG;
    const bool mirrors = c->num_scored != 0 && c->num_scored != c->num_candidates;
    // per-request outputs come from one run per candidate; mirrors need the partner list
    if (mirrors && ((flags & MMS_FLAG_PER_REQUEST) || !c->partner || !c->mirror_swap))
        return MMS_ERR_ARG;

    // mirrors are accepted and not needed any more
    const int64_t B = c->num_scored ? c->num_scored : c->num_candidates;
    // blocks that fit an SM at once, from the kernel's shared-memory use
    const size_t lat_elems0 = (size_t)c->num_models * c->num_columns * c->max_stages + 8;
    const int lat_on_chip0 = (c->latency_stride == 0 && lat_elems0 * sizeof(float) <= (size_t)kLatSmemBytes)
                                 ? (int)lat_elems0 : 0;
    const SmemLayout L0 = smem_layout(c->max_slots, c->max_stages, lat_on_chip0);
    int sm_count = 148, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        (void)cudaGetLastError();
        sm_count = 148;
    }
    // Warps per block: blocks share the latency table among their warps, so the
    // size that fits the most warps on an SM (233472 bytes, 1024 reserved per
    // block; 232448 at most in one block) wins, the smaller one on a tie.
    int64_t per_sm = 1;
    int block_warps = 1;
    auto fit = [&](const SmemLayout &L, int64_t &best_per_sm, int &best_w) {
        best_per_sm = 1;
        best_w = 1;
        for (int w = 1; w <= kMaxBlockWarps; ++w) {
            const size_t bytes = L.warp0 + (size_t)w * L.warp_bytes;
            if (bytes > 232448) break;
            int64_t warps = (int64_t)(233472 / (bytes + 1024)) * w;
            if (warps > kMaxWarpsPerSm) warps = kMaxWarpsPerSm;
            if (warps >= best_per_sm) { best_per_sm = warps; best_w = w; }
        }
    };
    fit(L0, per_sm, block_warps);
    // The table goes on chip as doubles (no conversion per use) when that costs
    // no resident warp.
    g->lat_f64 = 0;
    if (lat_on_chip0) {
        const SmemLayout L64 = smem_layout(c->max_slots, c->max_stages, lat_on_chip0, true);
        int64_t per_sm64;
        int block_warps64;
        fit(L64, per_sm64, block_warps64);
        if (per_sm64 >= per_sm) { g->lat_f64 = 1; block_warps = block_warps64; }
    }
    const int64_t resident_slots = (int64_t)sm_count * per_sm;
    // the window kernels: blocks resident on an SM, from their shared memory (the table as
    // doubles) and their register budget
    size_t table = window_table_elems(c->num_models, c->num_columns, c->max_stages,
                                      (flags & MMS_FLAG_LEGACY_CLOCK) != 0);
    if (c->latency_stride != 0 || table * sizeof(double) > 2 * (size_t)kLatSmemBytes) table = 0;
    g->win_table_elems = (int32_t)table;
    g->smem_window = window_layout(c->max_slots, c->max_groups, c->max_stages, c->max_placed, table).total;
    if (g->smem_window > 227 * 1024) return MMS_ERR_UNSUPPORTED;
    int64_t window_per_sm = 233472 / (int64_t)(g->smem_window + 1024);
    if (window_per_sm > kWindowBlocksPerSm) window_per_sm = kWindowBlocksPerSm;
    g->window_blocks = (int32_t)(window_per_sm * sm_count);
    const int64_t chunk = opts ? opts->chunk_requests : 0;
    int64_t warm = opts ? opts->warmup_requests : 0;
    // Run-in: enough requests for every group to have had an idle moment and every replicated
    // model a request, most of the time.  Both grow with the cluster.  Chunks simulated again, of
    // those of lists of 500 to 2000 placements at 0.6 to 2 requests a second and device, and the
    // call, with 32 requests per clock slot and with 64:
    //     8 slots    random  1.6 and 0.4 %   5.0 and 4.3 ms    grown   3 and 0.3 %   5.7 and 5.6 ms
    //    16 slots    random  1.2 and 0.3 %   6.1 and 6.0 ms    grown   9 and 1 %     7.7 and 7.0 ms
    //    32 slots    random  1.8 and 0.2 %   6.5 and 7.7 ms    grown  22 and 9 %    13.3 and 15.2 ms
    //    64 slots    random  1.1 and 0.1 %   9.8 and 12.1 ms   grown  22 and 8 %    36.6 and 42 ms
    // What fails is repaired in parallel (restart_kernel), at less than a longer run-in costs all
    // chunks: 4096 placements on 64 devices 24 and 27 ms, a layer of 2343 on 64 47 and 48.
    if (warm <= 0) {
        warm = 32 * (int64_t)c->max_slots;
        if (warm < 128) warm = 128;
        if (warm > 2048) warm = 2048;
    }
    // Segments are the unit of state snapshots and repairs, chunks (runs of segments) the unit
    // of parallel work.  The 32-candidate kernel takes as many chunks as fill nine tenths of
    // ONE wave of the resident warps (SMs x warps per SM at its shared-memory use; a second
    // wave would pay the run-in twice), but none shorter than min_chunk.
    struct Cut { int64_t seg, NS, spc, K; };
    auto cut_trace = [&](int64_t seg, int64_t lanes, int64_t min_chunk) {
        Cut x;
        x.seg = seg;
        x.NS = N / seg > 0 ? N / seg : 1;
        if (chunk < 0 || N < 4 * seg || B == 0) {
            x.spc = x.NS;
        } else if (chunk > 0) {
            x.spc = (chunk + seg / 2) / seg;
        } else {
            // the ideal length rounded to the nearest number of segments, or the next longer
            // one when the chunks would not fit the wave any more
            x.spc = (20 * x.NS * B + 9 * lanes) / (18 * lanes);
            if (x.spc * seg < min_chunk) x.spc = (min_chunk + seg - 1) / seg;
            if (x.spc < 1) x.spc = 1;
            if (x.spc < x.NS && ((x.NS + x.spc - 1) / x.spc) * B > lanes) x.spc += 1;
        }
        if (x.spc < 1) x.spc = 1;
        if (x.spc > x.NS) x.spc = x.NS;
        x.K = (x.NS + x.spc - 1) / x.spc;
        return x;
    };
    // Segments of 128 requests where the snapshots are few (they are 8 bytes per clock slot,
    // candidate and segment), of 1024 in the large batches, whose chunks then have at least three.
    // Calls with the line at 64, 256 and 1024 MB of snapshots at 128: 600 random placements on 16
    // devices (90 MB) 5.0, 3.9 and 3.9 ms, 1500 on 32 (180) 8.1, 7.3, 7.4; 500 on 64 (360) 9.8, 9.8,
    // 8.0, 1536 (670) 11.4, 11.4, 12.8; grown ones: 1000 on 32 devices (300) 14.6, 14.6, 16.7, 1000 on
    // 64 (400) 29, 29, 36.
    const int64_t seg = !thrift && (double)N * (double)c->max_slots * (double)B * 8.0 / 128.0 <= 256e6 ? 128 : 1024;
    const int64_t thrifty = thrift == 0 ? 0 : thrift < 3 ? 3 * seg : 12 * seg;     // shortest chunk
    const Cut wide = cut_trace(seg, resident_slots * kLanes,
                               thrifty ? thrifty : seg == 1024 ? 3 * seg : warm / 2);
    const Cut win = cut_trace(seg, (int64_t)g->window_blocks * kWindowWarps, thrifty ? thrifty : seg);
    // Which speculative pass: see window_pays.
    g->window = window_pays(N, B, wide.K, win.K, warm, sm_count, window_worth(c, B, flags));
    // Few candidates cut into many chunks wait for the walks behind failed boundaries, one after the
    // other for each candidate, and those of many groups of few stages fail most (9 % of grown
    // ones on 16 devices with 32 requests a slot, 1 % with 64: the order in which idle replicas were
    // used).  A search on 16 devices over 30 000 requests, four traces, with 32 a slot and with 64 a
    // group: 77, 84, 81, 108 and 64, 64, 65, 69 ms; a search over 5 600 35 and 36, three placements over
    // 11 900 0.78 and 0.86: there the longer pass costs more than the walks.  Random placements have a
    // third as many groups as slots.
    if (g->window && !(opts && opts->warmup_requests > 0) && 2 * c->max_groups > c->max_slots &&
        N >= 128 * 128) {
        warm = 64 * (int64_t)c->max_groups;
        if (warm > 2048) warm = 2048;
    }
    const Cut &x = g->window ? win : wide;
    const int64_t NS = x.NS, spc = x.spc, K = x.K;
    if (K * (B > 0 ? B : 1) >= 0x7FFFFFFFLL) return MMS_ERR_UNSUPPORTED;   // work-list encoding
    // A launch that fills less than half of the GPU goes out in smaller
    // blocks, one per SM: a warp that shares its SM with two others runs
    // faster than one that shares it with eleven while most SMs stand idle.
    // (A nearly full launch keeps the large blocks: the SMs they leave free
    // serve the small kernels of a launch running beside it.)
    const int64_t total_warps = ((B + kLanes - 1) / kLanes) * K;
    if (2 * total_warps <= (int64_t)sm_count * block_warps) {
        block_warps = (int)((total_warps + sm_count - 1) / sm_count);
        if (block_warps < 1) block_warps = 1;
    }
    g->block_warps = block_warps;
    int rounds = opts ? opts->repair_rounds : 0;
    if (rounds <= 0) rounds = kDefaultRepairRounds;
    if (rounds > kMaxRepairRounds) rounds = kMaxRepairRounds;
    g->rounds = rounds;
    // Where a chunk is shorter than the run-in, one more chunk of history changes little and walks
    // are better done in order.  With the line at half the run-in: 1500 placements on 32 devices, of
    // which 61 with interchangeable groups have chunks of 512 behind 1024, 7.3 -> 8.3 ms, 1025 on 16
    // (256 behind 512) 3.8 -> 4.25, but 200 grown ones on 32 (512 behind 1024) 5.6 -> 4.9.
    g->restart = spc * x.seg >= warm;
    g->K = (int32_t)K; g->NS = (int32_t)NS; g->seg_len = (int32_t)x.seg;
    g->seg_per_chunk = (int32_t)spc; g->warmup = (int32_t)warm;

    // the shared table goes on chip (f32), with 8 readable entries of padding
    const size_t lat_elems = (size_t)c->num_models * c->num_columns * c->max_stages + 8;
    g->lat_smem_elems = (c->latency_stride == 0 && lat_elems * sizeof(float) <= (size_t)kLatSmemBytes)
                            ? (int32_t)lat_elems : 0;
    const SmemLayout L = smem_layout(c->max_slots, c->max_stages, g->lat_smem_elems,
                                     g->lat_smem_elems != 0 && g->lat_f64 != 0);
    g->smem_stream = L.warp0 + (size_t)g->block_warps * L.warp_bytes;
    // the tally's per-lane histograms (count_kernel)
    g->smem_count = sizeof(uint32_t) * (size_t)(c->max_groups + (c->num_models + 1) / 2) * kLanes;
    if (g->smem_count > 227 * 1024) return MMS_ERR_UNSUPPORTED;
    size_t off = 0;
    // Replica rows: two of four, and for a model of more than eight replicas as many more as
    // there can be, up to kMaxRowReplicas, with one that is not full and one to spare for reading ahead.
    g->row_planes = 2;
    if (!thrift && c->max_groups > 8 && c->max_placed > 8) {
        const int32_t most = c->max_groups < c->max_placed ? c->max_groups : c->max_placed;
        g->row_planes = 3 + (most < kMaxRowReplicas ? most : kMaxRowReplicas) / 4;
    }
    g->off_rows = off;
    off += align256((g->row_planes + (g->row_planes > 2)) * sizeof(uint32_t) * kRowWords *
                        (size_t)((B + kLanes - 1) / kLanes * kLanes) * (c->num_models + 1) + 256);
    g->off_leaf = off;        off += align256(sizeof(double) * (size_t)plan_leaves(N) * B);
    g->off_decisions = off;   off += align256((c->max_groups > 126 ? 2 : 1) * (size_t)((N + 3) / 4 * 4 + 4) *
                                               (size_t)((B + 31) / 32 * 32));
    g->off_work_count = off;  off += align256(2 * sizeof(uint32_t) * kMaxRepairRounds);
    g->off_work_items = off;  off += align256(sizeof(uint32_t) * (size_t)K * B);
    g->off_seg_leaf = off;    off += align256(sizeof(int32_t) * (size_t)(NS + 1));
    g->off_group_info = off;  off += align256(sizeof(uint32_t) * (size_t)B * c->max_groups + 4);
    g->off_group_column = off; off += align256(sizeof(uint32_t) * (size_t)B * c->max_groups + 4);
    g->off_columns = off;     off += align256(sizeof(uint32_t) * ((size_t)c->num_columns + 1));
    g->off_flags = off;       off += align256(3 * (size_t)B + 4);      // relabelled, open, twins
    g->group_words = 0;
    // Entries of a segment's list of swaps.  Of placements with twins 0.05 to 4 % of the requests
    // are one, in bursts: of the segments of 128 requests of an hour on 64 devices at most 12, of
    // bursts on 16 devices 0.1 % have more than 34; of those of 1024 requests 43, and 0.1 % have
    // more than 123.  Arrival times on a grid make it 20 to 45 % (of 117 chunks of such a trace 77
    // are simulated again with room for 24 of 128, 10 with 48, 8 with 64, 1 with 96).  A full list
    // costs walks, never results.
    g->swap_cap = seg == 128 ? 64 : 160;
    if (K > 1) {
        const size_t G = (size_t)c->max_groups;
        g->off_stamp = off;        off += align256((size_t)K * B);
        g->off_link = off;         off += align256((size_t)K * B);
        g->off_rel = off;          off += align256((size_t)NS * B);
        if (c->num_models <= kTwinModels && !(flags & MMS_FLAG_NO_TWINS) && thrift < 2)
            g->group_words = (c->num_models + 63) / 64;
        if (g->group_words) {
            const size_t cells = (size_t)NS * B;
            g->off_twin_class = off;  off += align256(sizeof(uint32_t) * (size_t)B * G + 4);
            g->off_tie = off;         off += align256(sizeof(uint64_t) * cells);
            g->off_perm = off;        off += align256(cells * G + 4);
            g->off_swap_count = off;  off += align256(cells);
            g->off_name_from = off;   off += align256(sizeof(int32_t) * cells);
            g->off_swap_mask = off;   off += align256(sizeof(uint32_t) * cells * g->swap_cap);
            g->off_swap_at = off;     off += align256(sizeof(uint16_t) * cells * g->swap_cap);
            g->off_group_models = off;
            off += align256(sizeof(uint64_t) * (size_t)B * G * (size_t)g->group_words);
        }
        g->off_seg_end = off;     off += align256(sizeof(double) * (size_t)NS * c->max_slots * B);
        g->off_chunk_start = off; off += align256(sizeof(double) * (size_t)K * c->max_slots * B);
    }
    g->finish_at_once = (B + kWindowWarps - 1) / kWindowWarps <= (int64_t)kFinishBlocksPerSm * sm_count &&
                        (g->group_words || c->max_stages <= kGroupDepth);
    g->total = off;
    return MMS_OK;
}

// Events around the dominant kernels, see mms_profile_begin().
constexpr int kProfileSlots = 2048;
static cudaEvent_t g_prof_ev[2 * kProfileSlots];
static int32_t g_prof_tag[kProfileSlots];
static int g_prof_created = 0;      // events exist
static int g_prof_on = 0;
static int g_prof_count = 0;

// Brackets what is enqueued between its construction and stop() with two events.
struct ProfileSpan {
    int slot;
    cudaStream_t st;
    ProfileSpan(int32_t tag, cudaStream_t s) : slot(-1), st(s)
    {
        if (g_prof_on && g_prof_count < kProfileSlots) {
            slot = g_prof_count++;
            g_prof_tag[slot] = tag;
            (void)cudaEventRecord(g_prof_ev[2 * slot], st);
        }
    }
    void stop()
    {
        if (slot >= 0) (void)cudaEventRecord(g_prof_ev[2 * slot + 1], st);
        slot = -1;
    }
};

// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) is sticky per function and
// device and not cheap; it is issued only when a call needs more than any
// earlier one asked for.
struct SmemGrant { const void *func; int device; size_t bytes; };
constexpr int kMaxGrants = 128;
static SmemGrant g_grants[kMaxGrants];
static int g_num_grants = 0;
static std::mutex g_grant_mutex;

static int allow_smem(const void *func, size_t bytes)
{
    int dev = 0;
    MMS_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_grant_mutex);
    SmemGrant *slot = nullptr;
    for (int i = 0; i < g_num_grants; ++i)
        if (g_grants[i].func == func && g_grants[i].device == dev) { slot = &g_grants[i]; break; }
    if (slot && slot->bytes >= bytes) return MMS_OK;
    MMS_CUDA(cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    if (!slot && g_num_grants < kMaxGrants) slot = &g_grants[g_num_grants++];
    if (slot) { slot->func = func; slot->device = dev; slot->bytes = bytes; }
    return MMS_OK;
}

#define MMS_TRY(call)                  \
    do {                               \
        const int rc_ = (call);        \
        if (rc_ != MMS_OK) return rc_; \
    } while (0)

template <bool kFull, bool kLegacy>
static int launch_sim(KernelArgs &ka, const ClearArgs &ca, const Geometry &g, cudaStream_t st)
{
    // everything a call clears, then the tables its kernels read: two launches
    {
        int64_t cells = (int64_t)ka.NS * ka.B;
        if ((int64_t)ka.B * (ka.M + 1) > cells) cells = (int64_t)ka.B * (ka.M + 1);
        int64_t blocks = (cells + 255) / 256;
        if (blocks > 148 * 8) blocks = 148 * 8;
        if (blocks < 1) blocks = 1;
        clear_kernel<<<(unsigned)blocks, 256, 0, st>>>(ka, ca);
        MMS_CUDA(cudaGetLastError());
        if (blocks < kTableBlocks) blocks = kTableBlocks;
        build_tables_kernel<<<(unsigned)blocks, 256, 0, st>>>(ka, ca);
        MMS_CUDA(cudaGetLastError());
    }
    if (ka.K > 1 && ca.group_words && ka.G > 0) {
        const int64_t groups = (int64_t)ka.B * ka.G;
        twins_kernel<<<(unsigned)((groups + 127) / 128), 128, 0, st>>>(ka, ca);
        MMS_CUDA(cudaGetLastError());
    }
    ProfileSpan stream_span(MMS_PROFILE_STREAM, st);
    const int64_t streams = (int64_t)ka.B * ka.K;
    const auto window_blocks = [&](int64_t warps) {
        const int64_t blocks = (warps + kWindowWarps - 1) / kWindowWarps;
        return (unsigned)(blocks < g.window_blocks ? blocks : g.window_blocks);
    };
    if (g.window) {
        auto stream_k = ka.swap_mask ? window_stream_kernel<kLegacy, true> : window_stream_kernel<kLegacy, false>;
        MMS_TRY(allow_smem((const void *)stream_k, g.smem_window));
        stream_k<<<window_blocks(streams), kWindowWarps * kLanes, g.smem_window, st>>>(ka);
    } else {
        auto stream_k = ka.swap_mask ? sim_stream_kernel<kFull, kLegacy, true> : sim_stream_kernel<kFull, kLegacy, false>;
        MMS_TRY(allow_smem((const void *)stream_k, g.smem_stream));
        const int64_t per_block = (int64_t)kLanes * g.block_warps;
        stream_k<<<(unsigned)((streams + per_block - 1) / per_block), (unsigned)per_block,
                   g.smem_stream, st>>>(ka);
    }
    MMS_CUDA(cudaGetLastError());
    stream_span.stop();
    if (ka.K > 1) {
        auto walk_k = ka.swap_mask ? walk_kernel<kLegacy, true> : walk_kernel<kLegacy, false>;
        auto finish_k = g.finish_at_once
                            ? (ka.swap_mask ? finish_kernel<kLegacy, true, kFinishBlocksPerSm>
                                            : finish_kernel<kLegacy, false, kFinishBlocksPerSm>)
                            : (ka.swap_mask ? finish_kernel<kLegacy, true, kWindowBlocksPerSm>
                                            : finish_kernel<kLegacy, false, kWindowBlocksPerSm>);
        MMS_TRY(allow_smem((const void *)walk_k, g.smem_window));
        MMS_TRY(allow_smem((const void *)finish_k, g.smem_window));
        const int64_t bounds = (int64_t)ka.B * (ka.K - 1);
        const size_t link_smem = kLinkWarps * link_warp_bytes(ka.T, ka.G);
        // round g.rounds only judges the boundaries, for finish_kernel
        for (int r = 0; r <= g.rounds; ++r) {
            ka.round = r;
            if (ka.swap_mask || bounds <= kLinkAlone)
                link_warp_kernel<<<(unsigned)((bounds + kLinkWarps - 1) / kLinkWarps), kLinkWarps * kLanes,
                                   link_smem, st>>>(ka);
            else
                link_kernel<<<(unsigned)((bounds + 127) / 128), 128, 0, st>>>(ka);
            MMS_CUDA(cudaGetLastError());
            if (r == g.rounds) break;
            if (r == 0 && g.restart)
                restart_kernel<<<(unsigned)((bounds + 127) / 128), 128, 0, st>>>(ka);
            else
                resolve_kernel<<<(unsigned)((ka.B + 3) / 4), 4 * kLanes, 0, st>>>(ka);
            MMS_CUDA(cudaGetLastError());
            // sized for the worst case; blocks past the work list return at once
            walk_k<<<window_blocks(bounds), kWindowWarps * kLanes, g.smem_window, st>>>(ka);
            MMS_CUDA(cudaGetLastError());
        }
        ProfileSpan chain_span(MMS_PROFILE_CHAIN, st);
        finish_k<<<(unsigned)((ka.B + kWindowWarps - 1) / kWindowWarps), kWindowWarps * kLanes,
                   g.smem_window, st>>>(ka);
        MMS_CUDA(cudaGetLastError());
        if (ka.swap_mask) {
            const int32_t segments = (int64_t)ka.B * ka.NS <= kNameAlone ? 1 : kNameSegments;
            const int64_t warps = (int64_t)ka.B * ((ka.NS + segments - 1) / segments);
            name_kernel<<<(unsigned)((warps + kNameWarps - 1) / kNameWarps), kNameWarps * kLanes,
                          (size_t)kNameWarps * ka.G, st>>>(ka, segments);
            MMS_CUDA(cudaGetLastError());
        }
        chain_span.stop();
    }
    return MMS_OK;
}

}  // namespace mms

extern "C" {

int mms_abi_version(void) { return 10; }

const char *mms_last_error(void) { return mms::g_last_error; }

int mms_profile_begin(void)
{
    using namespace mms;
    if (!g_prof_created) {
        for (int i = 0; i < 2 * kProfileSlots; ++i) MMS_CUDA(cudaEventCreate(&g_prof_ev[i]));
        g_prof_created = 1;
    }
    g_prof_count = 0;
    g_prof_on = 1;
    return MMS_OK;
}

int mms_profile_end(int32_t *launches, float *each_ms, int32_t *each_tag, int32_t capacity)
{
    using namespace mms;
    g_prof_on = 0;
    for (int i = 0; i < g_prof_count; ++i) {
        float ms = 0.0f;
        MMS_CUDA(cudaEventSynchronize(g_prof_ev[2 * i + 1]));
        MMS_CUDA(cudaEventElapsedTime(&ms, g_prof_ev[2 * i], g_prof_ev[2 * i + 1]));
        if (each_ms && i < capacity) each_ms[i] = ms;
        if (each_tag && i < capacity) each_tag[i] = g_prof_tag[i];
    }
    if (launches) *launches = g_prof_count;
    g_prof_count = 0;
    return MMS_OK;
}

int32_t mms_sum_plan_leaves(int64_t num_requests)
{
    if (num_requests > 0x7FFFFFFF) return MMS_ERR_UNSUPPORTED;
    return mms::plan_leaves(num_requests);
}

int mms_sum_plan_fill(int64_t num_requests, int32_t *leaf_start, uint8_t *leaf_merges)
{
    if (num_requests < 0 || !leaf_start || !leaf_merges) return MMS_ERR_ARG;
    if (num_requests > 0x7FFFFFFF) return MMS_ERR_UNSUPPORTED;
    int32_t count = 0;
    if (num_requests > 0) mms::plan_rec(0, num_requests, leaf_start, leaf_merges, count);
    leaf_start[count] = (int32_t)num_requests;
    return MMS_OK;
}

int mms_trace_model_histogram(const mms_trace *trace, int32_t num_models, int32_t *hist,
                              void *stream)
{
    if (!trace || !hist || num_models < 0 || trace->num_requests < 0 || trace->num_traces < 0)
        return MMS_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (trace->num_traces > 1) {
        const int64_t T = trace->num_traces;
        if (T > 0x7FFFFFFF) return MMS_ERR_UNSUPPORTED;
        const size_t cells = (size_t)T * (num_models + 1) + 1;
        MMS_CUDA(cudaMemsetAsync(hist, 0, sizeof(int32_t) * cells, st));
        if (trace->num_requests == 0) return MMS_OK;
        if (!trace->model_ids || !trace->arrivals) return MMS_ERR_ARG;
        const size_t smem = sizeof(int32_t) * 32 * ((size_t)num_models + 1);
        if (smem > 48 * 1024) return MMS_ERR_UNSUPPORTED;
        const dim3 block(32, 8);
        int64_t slices = (trace->num_requests + 8 * 256 - 1) / (8 * 256);
        if (slices > 64) slices = 64;
        const dim3 grid((unsigned)((T + 31) / 32), (unsigned)slices);
        mms::histogram_traces_kernel<<<grid, block, smem, st>>>(
            trace->arrivals, trace->model_ids, trace->num_requests, (int32_t)T, num_models, hist);
        MMS_CUDA(cudaGetLastError());
        return MMS_OK;
    }
    MMS_CUDA(cudaMemsetAsync(hist, 0, sizeof(int32_t) * ((size_t)num_models + 1), st));
    if (trace->num_requests == 0) return MMS_OK;
    if (!trace->model_ids || !trace->arrivals) return MMS_ERR_ARG;
    if (((size_t)num_models + 1) * sizeof(int32_t) > 48 * 1024) return MMS_ERR_UNSUPPORTED;
    const int threads = 256;
    int64_t want = (trace->num_requests + threads - 1) / threads;
    const int blocks = (int)(want < 592 ? want : 592);   // 4 blocks per SM on 148 SMs
    mms::histogram_kernel<<<blocks, threads, sizeof(int32_t) * ((size_t)num_models + 1), st>>>(
        trace->arrivals, trace->model_ids, trace->num_requests, num_models, hist);
    MMS_CUDA(cudaGetLastError());
    return MMS_OK;
}

size_t mms_sim_workspace_bytes(int64_t num_requests, const mms_placements *cands,
                               const mms_sim_options *opts, uint32_t flags)
{
    // enough with and without MMS_FLAG_CROWDED, which callers need not pass here
    mms::Geometry g;
    size_t most = 0;
    for (const uint32_t crowded : {0u, (uint32_t)MMS_FLAG_CROWDED}) {
        if (mms::plan_call(num_requests, cands, opts, (flags & ~MMS_FLAG_CROWDED) | crowded,
                           !(flags & MMS_FLAG_NO_GROUP_GOOD), 0, &g) != MMS_OK)
            return 0;
        if (g.total > most) most = g.total;
    }
    return most;
}

}  // extern "C"

namespace mms {

static int sim_mixed(const mms_trace *trace, const mms_placements *cands, const mms_sum_plan *plan,
                     const int32_t *model_hist, const mms_sim_options *opts, const mms_workspace *ws,
                     const mms_results *out, uint32_t flags, int thrift, void *stream)
{
    if (!trace || !cands || !plan || !ws || !out) return MMS_ERR_ARG;
    if (flags & ~(MMS_FLAG_PER_REQUEST | MMS_FLAG_LEGACY_CLOCK | MMS_FLAG_NO_GROUP_GOOD |
                  MMS_FLAG_CROWDED | MMS_FLAG_NO_TWINS | MMS_FLAG_TRACE_ROWS))
        return MMS_ERR_ARG;
    const int64_t N = trace->num_requests;
    const bool gg = !(flags & MMS_FLAG_NO_GROUP_GOOD);
    if (gg && !out->group_num_good) return MMS_ERR_ARG;
    Geometry g;
    int rc = plan_call(N, cands, opts, flags, gg, thrift, &g);
    if (rc) return rc;
    const int32_t B = cands->num_scored ? cands->num_scored : cands->num_candidates;
    if (B == 0) return MMS_OK;
    if (!out->model_num_requests || !out->model_num_good || !out->group_num_requests ||
        !out->good_total || !out->latency_sum || !out->status || !model_hist)
        return MMS_ERR_ARG;
    if (N > 0 && (!trace->arrivals || !trace->model_ids || !trace->slos)) return MMS_ERR_ARG;
    if (trace->num_traces < 0 || trace->num_traces > 0x7FFFFFFF) return MMS_ERR_ARG;
    if (trace->num_traces > 1 && B > trace->num_traces)
        return MMS_ERR_ARG;                 // every scored candidate needs a trace of its own
    if (!cands->model_off || !cands->group_info || !cands->model_rep || !cands->latency)
        return MMS_ERR_ARG;
    const bool full = (flags & MMS_FLAG_PER_REQUEST) != 0;
    if (full && N > 0 && (!out->finish || !out->good)) return MMS_ERR_ARG;
    if (plan->num_leaves != plan_leaves(N)) return MMS_ERR_ARG;
    if (plan->num_leaves > 0 && (!plan->leaf_start || !plan->leaf_merges)) return MMS_ERR_ARG;
    if (g.total > 0 && (!ws->ptr || ws->bytes < g.total)) return MMS_ERR_ARG;

    cudaStream_t st = (cudaStream_t)stream;
    unsigned char *scratch = (unsigned char *)ws->ptr;
    KernelArgs ka;
    memset(&ka, 0, sizeof(ka));
    ka.arrivals = trace->arrivals; ka.model_ids = trace->model_ids; ka.slos = trace->slos;
    ka.N = N; ka.model_hist = model_hist;
    ka.many_traces = trace->num_traces > 1;
    const bool rows = (flags & MMS_FLAG_TRACE_ROWS) != 0;
    ka.trace_pitch = ka.many_traces && !rows ? trace->num_traces : 1;
    ka.trace_stride = ka.many_traces ? (rows ? N : 1) : 0;
    ka.unsorted = trace->num_traces > 1
                      ? model_hist + (size_t)trace->num_traces * (cands->num_models + 1)
                      : model_hist + cands->num_models;
    ka.B = B;
    ka.M = cands->num_models; ka.G = cands->max_groups; ka.P = cands->max_placed;
    ka.T = cands->max_slots; ka.S = cands->max_stages; ka.C = cands->num_columns;
    ka.model_off = cands->model_off; ka.model_rep = cands->model_rep;
    ka.group_info = cands->group_info; ka.latency = cands->latency;
    ka.latency_stride = cands->latency_stride;
    ka.lat_smem_elems = g.lat_smem_elems; ka.block_warps = g.block_warps;
    ka.lat_f64 = g.lat_smem_elems != 0 ? g.lat_f64 : 0;
    ka.K = g.K; ka.NS = g.NS; ka.seg_len = g.seg_len; ka.seg_per_chunk = g.seg_per_chunk;
    ka.warmup = g.warmup;
    ka.num_leaves = plan->num_leaves; ka.leaf_start = plan->leaf_start;
    ka.rep_rows = (uint32_t *)(scratch + g.off_rows);
    ka.row_planes = g.row_planes;
    ka.leaf_sums = (double *)(scratch + g.off_leaf);
    ka.decisions = scratch + g.off_decisions;
    ka.dec_wide = cands->max_groups > 126;
    ka.dec_pitch = ((int64_t)B + 31) / 32 * 32;
    ka.work_count = (uint32_t *)(scratch + g.off_work_count);
    ka.work_next = ka.work_count + kMaxRepairRounds;
    ka.work_items = (uint32_t *)(scratch + g.off_work_items);
    ka.stamp = scratch + g.off_stamp; ka.link = scratch + g.off_link;
    ka.relabelled = scratch + g.off_flags; ka.open = ka.relabelled + B;
    ka.rel = scratch + g.off_rel; ka.tie = (uint64_t *)(scratch + g.off_tie); ka.perm = scratch + g.off_perm;
    ka.swap_mask = g.group_words ? (uint32_t *)(scratch + g.off_swap_mask) : nullptr;
    ka.swap_at = (uint16_t *)(scratch + g.off_swap_at); ka.swap_count = scratch + g.off_swap_count;
    ka.swap_cap = g.swap_cap;
    ka.name_from = (int32_t *)(scratch + g.off_name_from);
    ka.seg_first_leaf = (int32_t *)(scratch + g.off_seg_leaf);
    ka.window = g.window;
    ka.seg_end = (double *)(scratch + g.off_seg_end);
    ka.chunk_start = (double *)(scratch + g.off_chunk_start);
    ka.status = out->status;
    ka.finish = full ? out->finish : nullptr; ka.good = full ? out->good : nullptr;
    ka.resimulated = out->resimulated;

    ClearArgs ca;
    ca.group_info_in = cands->group_info;
    ca.group_info = (uint32_t *)(scratch + g.off_group_info);
    ca.model_num_good = out->model_num_good;
    ca.model_num_requests = out->model_num_requests;
    ca.group_num_requests = out->group_num_requests;
    ca.group_num_good = gg ? out->group_num_good : nullptr;
    ca.good_total = out->good_total;
    ca.column_stages = (uint32_t *)(scratch + g.off_columns);
    ca.irregular = ca.column_stages + cands->num_columns;
    ca.group_words = g.group_words;
    ca.group_models = (uint64_t *)(scratch + g.off_group_models);
    ca.group_column = (uint32_t *)(scratch + g.off_group_column);
    ca.twin_class = (uint32_t *)(scratch + g.off_twin_class); ca.twins = ka.open + B;
    ka.group_column = ca.group_column;
    ka.twin_class = ca.twin_class; ka.twins = ca.twins;
    ka.column_stages = ca.column_stages; ka.irregular = ca.irregular;
    ka.win_table_elems = g.win_table_elems;
    ka.group_info = ca.group_info;       // the checked copy, contested bits derived on the device
    ProfileSpan call_span(MMS_PROFILE_CALL, st);
    const bool legacy = (flags & MMS_FLAG_LEGACY_CLOCK) != 0;
    if (full) rc = legacy ? launch_sim<true, true>(ka, ca, g, st) : launch_sim<true, false>(ka, ca, g, st);
    else rc = legacy ? launch_sim<false, true>(ka, ca, g, st) : launch_sim<false, false>(ka, ca, g, st);
    if (rc) return rc;

    // tally the recorded decisions (outputs were cleared up front)
    const size_t few_bytes = sizeof(uint32_t) * (size_t)(2 * ka.G + ka.M + 1);
    if (ka.B <= kCountFew && few_bytes <= 48 * 1024) {
        auto count_k = ka.dec_wide ? count_few_kernel<uint16_t> : count_few_kernel<uint8_t>;
        const int64_t slices = (N + 4 * kCountThreads - 1) / (4 * kCountThreads);
        count_k<<<(unsigned)(ka.B * (1 + slices)), kCountThreads, few_bytes, st>>>(
            ka, gg, out->model_num_good, out->group_num_requests, out->group_num_good, out->good_total,
            plan->leaf_merges, out->latency_sum);
        MMS_CUDA(cudaGetLastError());
        call_span.stop();
        return MMS_OK;
    }
    const size_t hist_bytes = g.smem_count;
    auto count_k = ka.dec_wide ? count_kernel<uint16_t> : count_kernel<uint8_t>;
    MMS_TRY(allow_smem((const void *)count_k, hist_bytes));
    int32_t seg_per_block = ka.NS / 96 > 0 ? ka.NS / 96 : 1;   // 16-bit counts: at most 32 segments
    if (seg_per_block > 32) seg_per_block = 32;
    // 32 more rows of blocks (the first) form the latency sums
    const dim3 count_grid((unsigned)((ka.B + kLanes - 1) / kLanes),
                          (unsigned)((ka.NS + seg_per_block - 1) / seg_per_block) + kLanes);
    count_k<<<count_grid, kLanes, hist_bytes, st>>>(ka, seg_per_block, gg, out->model_num_good,
                                                    out->group_num_requests, out->group_num_good,
                                                    out->good_total, plan->leaf_merges,
                                                    out->latency_sum);
    MMS_CUDA(cudaGetLastError());
    call_span.stop();
    return MMS_OK;
}

}  // namespace mms

extern "C" {

int mms_sim_mixed(const mms_trace *trace, const mms_placements *cands, const mms_sum_plan *plan,
                  const int32_t *model_hist, const mms_sim_options *opts, const mms_workspace *ws,
                  const mms_results *out, uint32_t flags, void *stream)
{
    return mms::sim_mixed(trace, cands, plan, model_hist, opts, ws, out, flags, 0, stream);
}

int mms_trace_pack(const double *arrivals, const int32_t *model_ids, const float *slos,
                   const int64_t *offsets, int64_t num_traces, int64_t padded_requests,
                   double *out_arrivals, int32_t *out_model_ids, float *out_slos, void *stream)
{
    if (num_traces < 0 || padded_requests < 0) return MMS_ERR_ARG;
    if (num_traces == 0 || padded_requests == 0) return MMS_OK;
    if (!arrivals || !model_ids || !slos || !offsets || !out_arrivals || !out_model_ids || !out_slos)
        return MMS_ERR_ARG;
    const int64_t bx = (padded_requests + 31) / 32, by = (num_traces + 31) / 32;
    if (bx > 0x7FFFFFFF || by > 65535) return MMS_ERR_UNSUPPORTED;
    mms::pack_traces_kernel<<<dim3((unsigned)bx, (unsigned)by), dim3(32, 8), 0,
                              (cudaStream_t)stream>>>(arrivals, model_ids, slos, offsets,
                                                      num_traces, padded_requests, out_arrivals,
                                                      out_model_ids, out_slos);
    MMS_CUDA(cudaGetLastError());
    return MMS_OK;
}

int mms_trace_pad_rows(const int64_t *lengths, int64_t num_traces, int64_t num_requests,
                       double *arrivals, int32_t *model_ids, float *slos, void *stream)
{
    if (num_traces < 0 || num_requests < 0) return MMS_ERR_ARG;
    if (num_traces == 0 || num_requests == 0) return MMS_OK;
    if (!lengths || !arrivals || !model_ids || !slos) return MMS_ERR_ARG;
    if (num_traces > 0x7FFFFFFF) return MMS_ERR_UNSUPPORTED;
    mms::pad_traces_kernel<<<dim3((unsigned)num_traces, 8), 256, 0, (cudaStream_t)stream>>>(
        lengths, num_requests, arrivals, model_ids, slos);
    MMS_CUDA(cudaGetLastError());
    return MMS_OK;
}

int mms_trace_rows_histogram(const double *arrivals, const int32_t *model_ids, int64_t num_traces,
                             int64_t num_requests, int32_t num_models, int32_t *hist, void *stream)
{
    if (num_traces < 1 || num_requests < 0 || num_models < 0 || !hist) return MMS_ERR_ARG;
    if (num_traces > 0x7FFFFFFF || ((size_t)num_models + 1) * sizeof(int32_t) > 48 * 1024)
        return MMS_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    MMS_CUDA(cudaMemsetAsync(hist, 0, sizeof(int32_t) * ((size_t)num_traces * (num_models + 1) + 1), st));
    if (num_requests == 0) return MMS_OK;
    if (!arrivals || !model_ids) return MMS_ERR_ARG;
    int64_t slices = (num_requests + 8191) / 8192;
    if (slices > 64) slices = 64;
    mms::histogram_rows_kernel<<<dim3((unsigned)num_traces, (unsigned)slices), 256,
                                 sizeof(int32_t) * ((size_t)num_models + 1), st>>>(
        arrivals, model_ids, num_requests, (int32_t)num_traces, num_models, hist);
    MMS_CUDA(cudaGetLastError());
    return MMS_OK;
}

int mms_argmax_scores(const int64_t *good_total, const double *latency_sum,
                      const int64_t *num_replicas, int64_t num_requests, int32_t num_candidates,
                      const int64_t *index_map, int64_t index_base, int32_t accumulate,
                      double *best, void *stream)
{
    if (num_candidates < 0 || num_requests < 0 || !best) return MMS_ERR_ARG;
    if (num_candidates > 0 && (!good_total || !latency_sum)) return MMS_ERR_ARG;
    mms::argmax_scores_kernel<<<1, mms::kArgmaxThreads, 0, (cudaStream_t)stream>>>(
        good_total, latency_sum, num_replicas, num_requests, num_candidates, index_map,
        index_base, accumulate != 0, best);
    MMS_CUDA(cudaGetLastError());
    return MMS_OK;
}

}  // extern "C"

namespace mms {

// Scratch of mms_sim_mixed_static.  In host code this name is only a handle
// for cudaGetSymbolAddress, never an address a kernel can use.
static __device__ __align__(256) unsigned char g_static_scratch[MMS_STATIC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
static void *g_static_scratch_ptr[kMaxDevices];   // device address, per device ordinal
static std::mutex g_static_scratch_mutex;

}  // namespace mms

extern "C" {

int mms_sim_mixed_static(const mms_trace *trace, const mms_placements *cands,
                         const mms_sum_plan *plan, const int32_t *model_hist,
                         const mms_sim_options *opts, const mms_results *out,
                         uint32_t flags, void *stream)
{
    if (!trace || !cands) return MMS_ERR_ARG;
    // the same shape checks as mms_sim_mixed, with the same return codes; only a
    // shape that is fine but needs more scratch than the array holds, however thrifty the plan, is new
    mms::Geometry geo;
    int thrift = 0;
    for (;; ++thrift) {
        const int rc = mms::plan_call(trace->num_requests, cands, opts, flags,
                                      !(flags & MMS_FLAG_NO_GROUP_GOOD), thrift, &geo);
        if (rc != MMS_OK) return rc;
        if (thrift == mms::kMaxThrift || geo.total <= (size_t)MMS_STATIC_SCRATCH_BYTES)
            break;
    }
    if (geo.total > (size_t)MMS_STATIC_SCRATCH_BYTES) {
        snprintf(mms::g_last_error, sizeof(mms::g_last_error),
                 "mms_sim_mixed_static: needs %zu bytes of scratch, the built-in array holds %u; "
                 "use fewer candidates per call or mms_sim_mixed with a caller workspace",
                 geo.total, (unsigned)MMS_STATIC_SCRATCH_BYTES);
        return MMS_ERR_UNSUPPORTED;
    }
    int dev = -1;
    MMS_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= mms::kMaxDevices) return MMS_ERR_NO_DEVICE;
    {
        // once per device, with that device current (under a lock: two host
        // threads may make the first call together)
        std::lock_guard<std::mutex> lock(mms::g_static_scratch_mutex);
        if (!mms::g_static_scratch_ptr[dev]) {
            void *p = nullptr;
            MMS_CUDA(cudaGetSymbolAddress(&p, mms::g_static_scratch));
            mms::g_static_scratch_ptr[dev] = p;
        }
    }
    mms_workspace ws;
    ws.ptr = mms::g_static_scratch_ptr[dev];
    ws.bytes = (size_t)MMS_STATIC_SCRATCH_BYTES;
    return mms::sim_mixed(trace, cands, plan, model_hist, opts, &ws, out, flags, thrift, stream);
}

int mms_trace_next_same_model(const mms_trace *trace, int32_t num_models, int32_t *next_same,
                              void *stream)
{
    if (!trace || num_models < 0 || trace->num_requests < 0) return MMS_ERR_ARG;
    if (trace->num_requests > 0x7FFFFFFF) return MMS_ERR_UNSUPPORTED;
    if (trace->num_requests == 0 || num_models == 0) return MMS_OK;
    if (!trace->model_ids || !next_same) return MMS_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    // requests of unknown models (-1) are never queued; give them a defined value
    MMS_CUDA(cudaMemsetAsync(next_same, 0xFF, sizeof(int32_t) * (size_t)trace->num_requests, st));
    mms::next_same_kernel<<<(unsigned)num_models, mms::kNextWarps * mms::kLanes, 0, st>>>(
        trace->model_ids, trace->num_requests, next_same);
    MMS_CUDA(cudaGetLastError());
    return MMS_OK;
}

}  // extern "C"

namespace mms {

struct BatchGeometry {
    int32_t per_lane;         // groups per lane of the kernels with a group per lane; 0: lists
    int32_t H, event_rows, K, NS, seg_len, seg_per_chunk, warmup, table_elems, warps, blocks;
    bool lean;
    int32_t list_elems, list_warps, list_blocks;      // the list kernels beside the others
    size_t list_smem;
    size_t smem, smem_judge, state_bytes;
    size_t off_leaf, off_start, off_end, off_carry, off_carry_n, off_carry_seg, off_walk_carry,
        off_run_status, off_perm, off_tie, off_swaps, off_swap_n, off_walk_swaps, off_counts, off_flag, off_work, off_items, off_marks, off_first, off_pos, off_req, off_ts, off_dl,
        total;
    int32_t rounds;
};

constexpr size_t kBatchSnapshotBytes = 256u << 20;

// Chunking and scratch layout of one mms_sim_batching call.
static int plan_batching(int64_t N, const mms_placements *c, const mms_batching *bt,
                         BatchGeometry *g)
{
    *g = BatchGeometry();
    if (!c || !bt || N < 0 || N > 0x7FFFFFFF || c->num_candidates < 0) return MMS_ERR_ARG;
    const int64_t B = c->num_candidates;
    g->H = bt->heap_capacity > 0 ? bt->heap_capacity : c->max_groups + 16;
    g->event_rows = (g->H + kLanes - 1) / kLanes;
    g->state_bytes = batch_state_bytes(c->num_models, c->max_slots, g->event_rows);
    int sm_count = 148, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        (void)cudaGetLastError();
        sm_count = 148;
    }
    // Shared memory: the latency table on chip where it takes little of it; the candidate's tables
    // too, unless they would not fit; as many warps to a block as fit.
    const size_t table = (size_t)c->num_models * c->num_columns * c->max_stages * bt->num_batch_sizes;
    const auto layout = [&](int32_t elems, int warps) {
        if (g->per_lane)
            return ((sizeof(double) * (size_t)elems + 15) & ~(size_t)15) +
                   warps * group_smem(c->num_models, c->max_slots, g->H).bytes;
        return batch_smem(c->num_models, c->max_groups, c->max_placed, c->max_slots, g->event_rows, elems,
                          g->lean, warps).total;
    };
    // A group per lane where groups and models fit masks, the table as doubles fits beside the
    // warps, and more events than groups may be pending; else lists, with the candidate's tables
    // on chip unless they would not fit.
    const auto list_plan = [&]() {
        g->per_lane = 0;
        g->table_elems = c->latency_stride == 0 && table * sizeof(float) <= 2 * (size_t)kLatSmemBytes ? (int32_t)table : 0;
        g->lean = false;
        g->lean = layout(0, 1) > 227 * 1024;
        if (g->lean && layout(0, 1) > 227 * 1024) return false;
        if (layout(g->table_elems, 1) > 227 * 1024) g->table_elems = 0;
        g->warps = kBatchWarps;
        while (g->warps > 1 && layout(g->table_elems, g->warps) > 227 * 1024) --g->warps;
        g->smem = layout(g->table_elems, g->warps);
        return true;
    };
    if (!list_plan()) return MMS_ERR_UNSUPPORTED;
    g->list_elems = g->table_elems; g->list_warps = g->warps; g->list_smem = g->smem;
    int64_t per_sm = 1;
    const auto resident = [&]() {
        per_sm = (int64_t)(233472 / (g->smem + 1024));
        const int64_t most = (kBatchWarps * kBatchBlocksPerSm) / g->warps;     // registers
        if (per_sm > most) per_sm = most;
        if (per_sm < 1) per_sm = 1;
        g->blocks = (int32_t)(per_sm * sm_count);
    };
    resident();
    g->list_blocks = g->blocks;
    if (c->max_groups <= kGroupLimit && c->num_models <= kGroupLimit && g->H >= c->max_groups &&
        c->latency_stride == 0 && table > 0 && table * sizeof(double) <= 3 * (size_t)kLatSmemBytes) {
        g->per_lane = c->max_groups <= kLanes ? 1 : 2;
        g->table_elems = (int32_t)table + kBatchDepth * bt->num_batch_sizes;
        g->warps = kBatchWarps;
        g->event_rows = g->per_lane + (g->H + kLanes - 1) / kLanes;
        g->smem = layout(g->table_elems, g->warps);
        if (g->smem <= 227 * 1024) resident();
        else if (list_plan()) { g->event_rows = (g->H + kLanes - 1) / kLanes; resident(); }
    }
    g->state_bytes = batch_state_bytes(c->num_models, c->max_slots, g->event_rows);
    g->smem_judge = layout(0, g->warps);
    // Run-in as in plan_call; as many chunks as there are resident warps, none shorter than half
    // the run-in (one placement on 16 devices, 27 000 requests, two traces, speculative pass and repairs:
    // chunks of 128 0.80 + 2.5 and 0.61 + 0.1 ms, 256 0.93 + 1.1 and 0.71 + 0.1, 512 1.31 + 0.9 and 1.04 +
    // 0.04), and no cut at all when that leaves fewer than two.
    int64_t warm = 32 * (int64_t)c->max_slots;
    if (warm < 128) warm = 128;
    if (warm > 2048) warm = 2048;
    g->warmup = (int32_t)warm;
    int64_t seg = 128;
    while (seg < N && (size_t)(N / seg) * (size_t)B * g->state_bytes > kBatchSnapshotBytes) seg *= 2;
    int64_t NS = N / seg > 0 ? N / seg : 1, spc = NS;
    if (B > 0 && N >= 1024) {
        const int64_t K = (int64_t)g->blocks * g->warps / B, least = (warm / 2 + seg - 1) / seg;
        if (K >= 2) spc = (NS + K - 1) / K;
        if (spc < least) spc = least;
        if (spc > NS) spc = NS;
    }
    g->K = (int32_t)((NS + spc - 1) / spc);
    g->seg_len = (int32_t)seg;
    g->NS = (int32_t)NS;
    g->seg_per_chunk = (int32_t)spc;
    const size_t b = (size_t)(B > 0 ? B : 1), cells = (size_t)g->K * b, segs = (size_t)NS * b;
    if (cells >= 0x7FFFFFFF) return MMS_ERR_UNSUPPORTED;
    size_t off = 0;
    const auto take = [&](size_t bytes) { const size_t at = off; off += align256(bytes + 8); return at; };
    g->off_leaf = take(sizeof(double) * (size_t)plan_leaves(N) * b);
    g->off_flag = take(256);
    g->off_first = take(sizeof(int32_t) * ((size_t)c->num_models + 1));
    g->off_pos = take(sizeof(int32_t) * (size_t)N);
    g->off_req = take(sizeof(int32_t) * (size_t)N);
    g->off_ts = take(sizeof(double) * (size_t)N);
    g->off_dl = take(sizeof(double) * (size_t)N);
    g->off_counts = take(2 * sizeof(uint32_t) * segs * c->max_groups);
    // A round of walks beside each other takes as long as a chunk: it pays where chunks are short
    // (the trace of above, chunks of 128: 0.34 + 1.5 instead of 2.1 ms), not where the chain has
    // little to do (256 placements on 64 devices, 45 000 requests, chunks of 5 000: 4.6 + 1.8
    // instead of 1.8 ms; with twice as many chunks 12.3 -> 16).
    g->rounds = g->seg_per_chunk * g->seg_len <= g->warmup ? 1 : 0;
    if (g->K > 1) {
        g->off_start = take(cells * g->state_bytes);
        g->off_end = take(segs * g->state_bytes);
        g->off_carry = take(cells * sizeof(Carried) * kMaxCarry);
        g->off_carry_n = take(cells * sizeof(uint32_t));
        g->off_carry_seg = take(segs);
        g->off_walk_carry = take((size_t)g->blocks * g->warps * sizeof(Carried) * kMaxCarry);
        g->off_run_status = take(cells * sizeof(uint32_t));
        if (g->per_lane) {
            g->off_perm = take(cells * kGroupLimit);
            g->off_tie = take(segs * sizeof(uint64_t));
            g->off_swaps = take(cells * sizeof(Swap) * kSwapCap);
            g->off_swap_n = take(cells * sizeof(uint32_t));
            g->off_walk_swaps = take((size_t)g->blocks * g->warps * sizeof(Swap) * kSwapCap);
        }
        g->off_work = take(2 * sizeof(uint32_t) * (size_t)(g->rounds + 1));
        g->off_items = take(cells * sizeof(uint32_t));
        g->off_marks = take(2 * cells);
    }
    g->total = off;
    return MMS_OK;
}

}  // namespace mms

extern "C" {

size_t mms_sim_batching_workspace_bytes(int64_t num_requests, const mms_placements *cands,
                                        const mms_batching *batching)
{
    mms::BatchGeometry g;
    if (mms::plan_batching(num_requests, cands, batching, &g) != MMS_OK) return 0;
    return g.total;
}

int mms_sim_batching(const mms_trace *trace, const mms_placements *cands,
                     const mms_batching *batching, const int32_t *next_same,
                     const mms_sum_plan *plan, const mms_workspace *ws, const mms_results *out,
                     void *stream)
{
    using namespace mms;
    if (!trace || !cands || !batching || !plan || !ws || !out) return MMS_ERR_ARG;
    const int64_t N = trace->num_requests;
    const int32_t B = cands->num_candidates;
    if (N < 0 || B < 0 || cands->num_models < 0 || cands->max_groups < 0 ||
        cands->max_placed < 0 || cands->max_slots < 0 || cands->max_stages < 1 ||
        cands->num_columns < 0)
        return MMS_ERR_ARG;
    if (N > 0x7FFFFFFF || cands->max_groups > MMS_MAX_GROUPS || cands->max_slots > MMS_MAX_SLOTS ||
        cands->max_placed > MMS_MAX_PLACED || cands->max_stages > MMS_MAX_STAGES ||
        cands->num_columns > MMS_MAX_COLUMNS)
        return MMS_ERR_UNSUPPORTED;
    if (trace->num_traces > 1) return MMS_ERR_UNSUPPORTED;   // one shared trace only
    const int NB = batching->num_batch_sizes;
    if (NB < 1 || NB > 8 || batching->batch_sizes[0] != 1) return MMS_ERR_ARG;
    if (B == 0) return MMS_OK;
    if (!out->model_num_requests || !out->model_num_good || !out->group_num_requests ||
        !out->group_num_good || !out->good_total || !out->latency_sum || !out->status)
        return MMS_ERR_ARG;
    (void)next_same;                       // accepted and not needed any more
    if (N > 0 && (!trace->arrivals || !trace->model_ids || !trace->slos || !out->finish || !out->good))
        return MMS_ERR_ARG;
    if (!cands->model_off || !cands->model_rep || !cands->latency || !batching->group_off ||
        !batching->group_mod || !batching->group_cfg)
        return MMS_ERR_ARG;
    if (plan->num_leaves != plan_leaves(N)) return MMS_ERR_ARG;
    if (plan->num_leaves > 0 && (!plan->leaf_start || !plan->leaf_merges)) return MMS_ERR_ARG;
    BatchGeometry geo;
    {
        const int rc = plan_batching(N, cands, batching, &geo);
        if (rc != MMS_OK) return rc;
    }
    if (!ws->ptr || ws->bytes < geo.total) return MMS_ERR_ARG;

    BatchArgs a;
    memset(&a, 0, sizeof(a));
    a.arrivals = trace->arrivals; a.model_ids = trace->model_ids; a.slos = trace->slos;
    a.N = N;
    a.B = B; a.M = cands->num_models; a.G = cands->max_groups; a.P = cands->max_placed;
    a.T = cands->max_slots; a.S = cands->max_stages; a.C = cands->num_columns; a.NB = NB;
    a.H = geo.H; a.event_rows = geo.event_rows;
    a.spare = geo.H > a.G ? (uint32_t)(geo.H - a.G) : 0u;
    for (int j = 0; j < NB; ++j) {
        const int32_t bs = batching->batch_sizes[j];
        if (bs < 1 || (bs & (bs - 1)) || (j > 0 && bs <= batching->batch_sizes[j - 1]))
            return MMS_ERR_ARG;
        int col = 0;
        while ((1 << col) < bs) ++col;
        if (col >= NB) return MMS_ERR_ARG;   // the reference would index past the table
        a.batch_sizes[j] = bs;
        a.batch_cols[j] = col;
    }
    a.model_off = cands->model_off; a.model_rep = cands->model_rep;
    a.group_off = batching->group_off; a.group_mod = batching->group_mod;
    a.group_cfg = batching->group_cfg;
    a.latency = cands->latency; a.latency_stride = cands->latency_stride;
    a.table_elems = geo.table_elems;
    a.at = group_smem(a.M, a.T, a.H);
    a.warp0 = (uint32_t)((sizeof(double) * (size_t)a.table_elems + 15) & ~(size_t)15);
    a.warp_bytes = (uint32_t)a.at.bytes;
    a.finish = out->finish; a.good = out->good;
    a.status = out->status;
    a.resimulated = out->resimulated;
    unsigned char *scratch = (unsigned char *)ws->ptr;
    a.K = geo.K; a.NS = geo.NS; a.seg_len = geo.seg_len; a.seg_per_chunk = geo.seg_per_chunk;
    a.warmup = geo.warmup; a.state_bytes = geo.state_bytes; a.rounds = geo.rounds;
    a.odd = (const int32_t *)(scratch + geo.off_flag);
    a.first_of = (int32_t *)(scratch + geo.off_first);
    a.pos = (int32_t *)(scratch + geo.off_pos);
    a.req = (int32_t *)(scratch + geo.off_req);
    a.pos_ts = (double *)(scratch + geo.off_ts);
    a.pos_dl = (double *)(scratch + geo.off_dl);
    a.seg_counts = (uint32_t *)(scratch + geo.off_counts);
    if (a.K > 1) {
        a.chunk_start = scratch + geo.off_start;
        a.seg_end = scratch + geo.off_end;
        a.carry = (Carried *)(scratch + geo.off_carry);
        a.carry_n = (uint32_t *)(scratch + geo.off_carry_n);
        a.carry_seg = scratch + geo.off_carry_seg;
        a.walk_carry = (Carried *)(scratch + geo.off_walk_carry);
        a.run_status = (uint32_t *)(scratch + geo.off_run_status);
        a.perm = scratch + geo.off_perm;
        a.tie = (uint64_t *)(scratch + geo.off_tie);
        if (geo.per_lane) {
            a.swaps = (Swap *)(scratch + geo.off_swaps);
            a.swap_n = (uint32_t *)(scratch + geo.off_swap_n);
            a.walk_swaps = (Swap *)(scratch + geo.off_walk_swaps);
        }
        a.work_count = (uint32_t *)(scratch + geo.off_work);
        a.work_next = a.work_count + a.rounds + 1;
        a.work_items = (uint32_t *)(scratch + geo.off_items);
        a.link = scratch + geo.off_marks;
        a.stamp = a.link + (size_t)a.K * B;
    }

    cudaStream_t st = (cudaStream_t)stream;
    const unsigned threads = (unsigned)(geo.warps * kLanes);
    const auto blocks_for = [&](int64_t warps, bool resident) {
        const int64_t blocks = (warps + geo.warps - 1) / geo.warps;
        return (unsigned)(resident && blocks > geo.blocks ? geo.blocks : blocks);
    };
    MMS_CUDA(cudaMemsetAsync(scratch + geo.off_flag, 0, 256, st));
    {
        BatchClear c;
        c.odd = (int32_t *)(scratch + geo.off_flag);
        c.model_num_good = out->model_num_good;
        int64_t cells = N > (int64_t)a.K * B ? N : (int64_t)a.K * B;
        if ((int64_t)B * a.M > cells) cells = (int64_t)B * a.M;
        int64_t blocks = (cells + kOrderWarps * kLanes - 1) / (kOrderWarps * kLanes);
        if (blocks > 148) blocks = 148;
        batch_order_kernel<<<(unsigned)(a.M + blocks), kOrderWarps * kLanes, 0, st>>>(a, c);
        MMS_CUDA(cudaGetLastError());
    }
    struct Kernels { void (*stream)(BatchArgs), (*judge)(BatchArgs), (*walk)(BatchArgs), (*chain)(BatchArgs); };
#define MMS_BATCH_KERNELS(W) \
    Kernels{batch_stream_kernel<W>, batch_validate_kernel<W>, batch_walk_kernel<W>, batch_chain_kernel<W>}
    const Kernels lists = geo.lean ? MMS_BATCH_KERNELS(ListWarp<true>) : MMS_BATCH_KERNELS(ListWarp<false>);
    const Kernels kern = geo.per_lane == 1 ? MMS_BATCH_KERNELS(GroupWarp<1>)
                         : geo.per_lane == 2 ? MMS_BATCH_KERNELS(GroupWarp<2>) : lists;
#undef MMS_BATCH_KERNELS
    if (N > 0) {
        ProfileSpan stream_span(MMS_PROFILE_BATCH_STREAM, st);
        MMS_TRY(allow_smem((const void *)kern.stream, geo.smem));
        kern.stream<<<blocks_for((int64_t)B * a.K, true), threads, geo.smem, st>>>(a);
        MMS_CUDA(cudaGetLastError());
        if (geo.per_lane) {                // ... and where the trace is odd
            BatchArgs odd = a;
            odd.table_elems = geo.list_elems;
            odd.event_rows = (geo.H + kLanes - 1) / kLanes;
            odd.only_odd = true;
            MMS_TRY(allow_smem((const void *)lists.stream, geo.list_smem));
            const int64_t blocks = (B + geo.list_warps - 1) / geo.list_warps;
            lists.stream<<<(unsigned)(blocks < geo.list_blocks ? blocks : geo.list_blocks),
                           (unsigned)(geo.list_warps * kLanes), geo.list_smem, st>>>(odd);
            MMS_CUDA(cudaGetLastError());
        }
        stream_span.stop();
    }
    if (N > 0 && a.K > 1) {
        MMS_TRY(allow_smem((const void *)kern.judge, geo.smem_judge));
        MMS_TRY(allow_smem((const void *)kern.walk, geo.smem));
        MMS_TRY(allow_smem((const void *)kern.chain, geo.smem));
        const int64_t bounds = (int64_t)B * (a.K - 1);
        // round a.rounds only judges the boundaries, for batch_chain_kernel
        for (int r = 0; r <= a.rounds; ++r) {
            ProfileSpan repair_span(MMS_PROFILE_BATCH_REPAIR, st);
            a.round = r;
            BatchArgs judge = a;
            judge.table_elems = 0;
            judge.warp0 = 0;
            kern.judge<<<blocks_for(bounds, false), threads, geo.smem_judge, st>>>(judge);
            MMS_CUDA(cudaGetLastError());
            if (r < a.rounds) {
                kern.walk<<<blocks_for(bounds, true), threads, geo.smem, st>>>(a);
                MMS_CUDA(cudaGetLastError());
            }
            repair_span.stop();
        }
        ProfileSpan chain_span(MMS_PROFILE_BATCH_CHAIN, st);
        kern.chain<<<blocks_for(B, false), threads, geo.smem, st>>>(a);
        MMS_CUDA(cudaGetLastError());
        chain_span.stop();
    }
    double *leaf_sums = (double *)(scratch + geo.off_leaf);
    if (plan->num_leaves > 0) {
        const int64_t slices = (plan->num_leaves + kTallyLeaves - 1) / kTallyLeaves;
        const size_t bytes = sizeof(uint32_t) * (size_t)a.M;
        if (bytes > 227 * 1024 || slices * B > 0x7FFFFFFF) return MMS_ERR_UNSUPPORTED;
        MMS_TRY(allow_smem((const void *)batch_tally_kernel, bytes));
        batch_tally_kernel<<<(unsigned)(slices * B), kTallyThreads, bytes, st>>>(
            a, plan->num_leaves, plan->leaf_start, out->model_num_good, leaf_sums);
        MMS_CUDA(cudaGetLastError());
    }
    if (a.G > 0) {
        if (N == 0) a.NS = 0;              // nothing was simulated
        const int64_t warps = (int64_t)B * ((2 * a.G + kLanes - 1) / kLanes);
        batch_count_kernel<<<(unsigned)((warps + 3) / 4), 4 * kLanes, 0, st>>>(
            a, out->group_num_requests, out->group_num_good);
        MMS_CUDA(cudaGetLastError());
    }
    KernelArgs fa;                         // what finalize_kernel reads; one run per candidate
    memset(&fa, 0, sizeof(fa));
    fa.B = B; fa.M = a.M; fa.num_leaves = plan->num_leaves; fa.N = N;
    fa.leaf_start = plan->leaf_start; fa.model_off = a.model_off;
    fa.leaf_sums = leaf_sums; fa.status = out->status;
    finalize_kernel<<<(B + 3) / 4, 4 * kLanes, 0, st>>>(
        fa, plan->leaf_merges, a.first_of, out->model_num_good, out->model_num_requests,
        out->good_total, out->latency_sum);
    MMS_CUDA(cudaGetLastError());
    return MMS_OK;
}

}  // extern "C"
