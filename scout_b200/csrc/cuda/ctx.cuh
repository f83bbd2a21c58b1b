// ctx.cuh -- the engine context (struct scout_ctx) and host-side helpers shared by the
// .cu translation units.
#pragma once

#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>
#include <cuda_runtime.h>

#include "../../../include/scout_gpu.h"
#include "common.cuh"

// Per-batch device counters, copied back once per batch.
struct DevCounters {
    // update phase
    int n_ins;          // edits classified as insertions
    int n_del;          // edits classified as deletions
    int n_half;         // applied half-edits (2 per applied edit)
    int n_aff;          // vertices whose row changed
    int n_one, n_short;       // short rows with one half-edit / with several
    int n_slices, n_rest;     // merge slices / rows that are not of the first kind
    int n_long;               // long rows compacted in place (tiered store)
    int plan_ticket, merge_ticket;   // tiles of the plan, items of the merge handed out so far
    long long new_elems;      // elements written to the pool this batch (HBM part when split)
    long long new_elems_host; // tiered store, split batch: elements written to the host pool
    long long nnz_delta;      // inserted minus deleted entries
    long long update_bytes;   // algorithmic bytes of the row merge
    // repair
    int q_count[12];          // queue counters (BFS: three rotating ones per phase, queue i lies in buffer i % 3)
    int list_count[4];        // auxiliary list counters
    int tick[4];              // work handed out in a round (BFS invalidation, rotating)
    int rounds;
    int changed;
    int affected;
    int conflicts;
    int noop;
    int recomputes;
    int splits;
    int searches;
    int overflow;             // a device list hit its capacity (results invalid)
    int pad;                  // CC: an edge joins two labels (inconsistent uploaded labelling)
    int ins_eff;              // BFS: insertions that lowered a level; CC: insertions that merged classes
    int del_eff;              // BFS: deletions of shortest-path tree edges
    long long hbm_bytes;      // algorithmic bytes of the repair
    long long aux64[4];
    unsigned long long phase_ns[8];   // %globaltimer marks written by the repair kernels
    // scheduler: feature accumulators, the 24 features, the model's 4 outputs, its decision
    int sched_hist[16];       // affected rows by floor(log2(1 + new degree))
    int sched_del_hit;        // deletion half-edits meeting the problem's structural test
    int sched_del;            // deletion half-edits
    int decision;             // repair variant the kernels run (read on the device)
    int sort_err;             // 1: a sort look-back wait timed out, 2: a sort position out of range,
                              // 4: a look-back wait of a scan or of the merge plan timed out
    int sched_flags;          // 1 features computed, 2 model applied
    int pairs_ok;             // the repair left its changed entries in DevBatch::pairs (when they fit)
    float feat[24];
    float pred[4];
};

// What a batch zeroes at its start and copies back at its end, in one piece: the counters, the
// barriers of the update and of the repair, and the changed entries when they are few (then
// the commit needs no launch and no copy of its own; not zeroed).
constexpr int COMMIT_PAIRS = 2048;
struct DevBatch {
    DevCounters ctr;
    scout::GridBar bar[2];
    int32_t pairs[2 * COMMIT_PAIRS];   // (id, value)
};

struct scout_ctx {
    int device = 0;
    int sm_count = 0;
    cudaStream_t s_main = nullptr;
    cudaStream_t s_copy[2] = {nullptr, nullptr};
    cudaEvent_t ev_copy[2] = {nullptr, nullptr};
    cudaEvent_t ev_t[8] = {nullptr};
    uint64_t budget = 0;
    uint64_t held = 0;
    std::string err;
    char name[256] = {0};

    // ---- graph store ----
    int64_t n = 0;
    int64_t nnz = 0;           // live entries (host view, exact after each batch)
    scout::Row* row = nullptr;
    int32_t* pool = nullptr;
    int64_t pool_cap = 0;
    int64_t tail = 0;          // first free pool element (host view)
    int32_t* spare = nullptr;  // previous pool, next compaction target
    int64_t spare_cap = 0;
    // tiered store (device budget smaller than the graph): cold rows live in mapped page-locked
    // host memory and are read in place by the kernels; a row is HBM-resident iff
    // 0 <= start < pool_cap, otherwise start is its element offset from `pool` into host_pool
    bool tiered = false;
    int32_t* host_pool = nullptr;   // host pointer (also the device pointer: unified addressing)
    int64_t host_cap = 0;
    int64_t host_tail = 0;
    int64_t evictions = 0;          // rows moved from HBM to the host pool by compactions
    int64_t evicted_entries = 0;
    int batch_dest = 0;             // where this batch's rewritten rows go: 0 HBM tail, 1 host
                                    // tail, 2 split (rows from HBM to HBM, host rows to host)
    int64_t host_batches = 0;       // batches whose rows were rewritten into the host pool
    int64_t compactions = 0;
    long long merge_tail = 0;       // HBM tail once the current batch's merge is done
    // gather of the next batch's cold rows (tiered store; scout_prefetch, gather.cu)
    bool pf_pending = false;        // a hint waits for the next repair's merge
    int64_t pf_m = 0;
    const scout_edge* pf_host = nullptr;   // where the hinted edits are read from (page-locked)
    void* h_pf_edits = nullptr;  int64_t cap_h_pf_edits = 0;   // pinned copy of pageable hinted edits
    scout_edge* d_pf_edits[2] = {nullptr, nullptr};  int64_t cap_pf_edits[2] = {0, 0};
    int pf_slot = 0;                // slot of the latest copy of hinted edits
    bool pf_ready = false;          // that slot holds (once ev_pf completes) a batch not yet used
    int64_t pf_ready_m = 0;
    bool pf_use = false;            // this call's edits are the hinted batch (scout_sched.prefetched)
    cudaEvent_t ev_pf = nullptr;    // the hinted edits' copy is done (copy stream)
    cudaEvent_t ev_union = nullptr; // fused repair rounds: this store's merge / the repair is done
    int32_t* gather_stamp = nullptr;   // n: last gather that took the vertex's row
    uint32_t gather_tag = 0;
    void* d_gctr = nullptr;
    void* h_gctr = nullptr;            // pinned
    int32_t* d_gather_list = nullptr;  int64_t cap_gather_list = 0;
    long long* d_gather_dst = nullptr; int64_t cap_gather_dst = 0;
    cudaEvent_t ev_gather0 = nullptr, ev_gather1 = nullptr;   // start / end of the gather (copy stream)
    long long gather_base = 0;
    bool gather_active = false;
    int64_t gathered_rows = 0, gathered_bytes = 0;
    bool reserved = false;
    bool sealed = false;
    int32_t* d_tmp_rows = nullptr;   // staging target for rows of one slot
    int64_t staged_rows = 0;

    // ---- per-problem state ----
    int32_t* level = nullptr;
    int32_t* color = nullptr;
    int32_t* label = nullptr;
    int32_t* mis = nullptr;
    int32_t source = 0;
    int32_t* d_sources = nullptr;   // BFS roots of a union of graphs (nsrc > 0), else `source`
    int nsrc = 0;
    int last_problem = -1;

    // ---- persistent per-vertex scratch (stamped with a batch epoch; never cleared) ----
    int32_t* stamp_a = nullptr;   // e.g. invalid / queued marks
    int32_t* stamp_b = nullptr;
    int32_t* stamp_c = nullptr;
    int32_t* stamp_d = nullptr;
    int32_t* aux_v = nullptr;     // per-vertex int scratch (label canonicalisation)
    uint32_t epoch = 0;

    // ---- per-batch workspace: one allocation, carved per batch size (grow-only) ----
    void* ws = nullptr;
    int64_t ws_bytes = 0;
    int64_t ws_m = 0;               // edits the workspace is carved for
    scout_edge* d_edits = nullptr;
    uint8_t* d_ops = nullptr;
    uint8_t* d_eflag = nullptr;
    unsigned long long* d_keys = nullptr;       // half-edit keys (2m)
    unsigned long long* d_keys_alt = nullptr;   // radix ping-pong (2m)
    unsigned long long* d_hkeys = nullptr;      // sorted half-edits of the current batch
    long long* d_mdp = nullptr;     // matched deletions before every half-edit (2m int32; room for 2m int64)
    int32_t* d_aff = nullptr;       // affected vertex ids (2m)
    int32_t* d_seg_b = nullptr;     // their segments' begins in the half-edits (2m + 1)
    int32_t* d_seg_d = nullptr;     // their segments' first deletions (2m)
    int32_t* d_longs = nullptr;     // long affected rows compacted in place (2m)
    int32_t* d_shorts = nullptr;    // short affected rows of several half-edits (2m)
    scout::MergeRow* d_mrow = nullptr;   // merge records: short rows of one half-edit from the front, others from the back (2m)
    int64_t* d_slices = nullptr;  int64_t cap_slices = 0;   // merge items (row << 32 | slice)
    void* d_update = nullptr;       // scratch of the one-launch update
    int64_t* d_coff = nullptr;      // compaction offsets (n + 1)
    int key_bits = 0;

    // ---- per-vertex work lists (n-sized, allocated on first repair) ----
    void* d_qbuf[3] = {nullptr, nullptr, nullptr};   // queues (uint64 items), qcap each
    int64_t qcap = 0;
    int32_t* d_list[2] = {nullptr, nullptr};         // touched / invalid lists, n each
    int32_t* d_commit = nullptr;                     // (id, value) pairs for the commit (2n)
    uint32_t qtag = 1;                               // per-round dedupe tags, never reused
    unsigned int* d_sort_hist = nullptr; int64_t cap_hist = 0;   // one-sweep control + look-back
    int64_t* d_scan_tmp = nullptr;  int64_t cap_scan = 0;
    void* d_misc = nullptr;         int64_t cap_misc = 0;   // colouring proposal markers
    int32_t* d_cc = nullptr;        // component scratch (7 n int32)
    int32_t* bfs_lv = nullptr;      // levels of a full BFS traversal before the diff (n int32)

    // ---- scheduler ----
    void* model[4] = {nullptr, nullptr, nullptr, nullptr};   // bf16 cost model per problem
    double prev_repair_ms[4] = {0, 0, 0, 0};                  // last batch's repair time per problem
    int32_t* probe_buf = nullptr;   // probe: pre-repair state, first variant's result, mismatch counter
    DevCounters* d_ctr_snap = nullptr;

    DevBatch* d_batch = nullptr;
    DevBatch* h_batch = nullptr;     // pinned
    DevCounters* d_ctr = nullptr;    // d_batch's and h_batch's counters
    DevCounters* h_ctr = nullptr;
    scout::GridBar* d_bar = nullptr; // the repair's barrier (d_batch->bar[1])
    bool bar_used = false;           // a kernel has used it since the batch began
    bool fetched = false;            // the last counters_fetch read them (they may hold an error)
    bool pairs_ready = false;        // h_batch->pairs holds the last repair's changed entries
    int* d_flags = nullptr;          // staging / seal error flags (int[16])

    // ---- pinned staging ----
    void* h_pin_edits = nullptr;  int64_t cap_pin_edits = 0;
    void* h_pin_commit = nullptr; int64_t cap_pin_commit = 0;
    void* h_slab[2] = {nullptr, nullptr}; int64_t cap_slab = 0;   // int32 elements
    int64_t* h_slab_off[2] = {nullptr, nullptr}; int32_t* h_slab_ids[2] = {nullptr, nullptr};
    int64_t cap_slab_rows = 0;
    int32_t* d_stage_ids[2] = {nullptr, nullptr};
    int64_t* d_stage_off[2] = {nullptr, nullptr};
    int64_t cap_stage_rows = 0;

    // ---- last batch bookkeeping ----
    int64_t last_changed = 0;
    int64_t last_half = 0;
    int64_t last_aff = 0;
    int32_t coop_blocks = 0;   // resident blocks of the persistent kernels
    // tuning knobs of the current call (scout_sched.blocks_per_sm / chunk_log2)
    int tune_blocks_per_sm = 0;   // 256-thread quarters of a repair block (0: all four)
    int tune_chunk_log2 = 10;     // BFS queue item = 2^chunk_log2 row entries
    int tune_share = 0;           // most warps sharing one BFS queue item (0: as many as useful)
    int64_t nlaunch = 0;       // kernels launched (running count)

    int fail(int code, const std::string& msg) { err = msg; return code; }
};

namespace scout {

// Allocation against the context's HBM budget.
int dev_alloc(scout_ctx* c, void** p, size_t bytes, const char* what);
void dev_free(scout_ctx* c, void* p, size_t bytes);
template <typename T>
int dev_grow(scout_ctx* c, T** p, int64_t* cap, int64_t need, const char* what) {
    if (*cap >= need && *p) return SCOUT_OK;
    int64_t nc = need + need / 4 + 1024;
    if (*p) dev_free(c, *p, (size_t)*cap * sizeof(T));
    *p = nullptr;
    *cap = 0;
    int rc = dev_alloc(c, (void**)p, (size_t)nc * sizeof(T), what);
    if (rc != SCOUT_OK) return rc;
    *cap = nc;
    return SCOUT_OK;
}
int pin_grow(scout_ctx* c, void** p, int64_t* cap_bytes, int64_t need_bytes);

int cuda_fail(scout_ctx* c, cudaError_t e, const char* where);
int host_fail(int code, const std::string& msg);   // thread-local message for calls without a context
#define SCOUT_CU(c, call)                                                  \
    do {                                                                   \
        cudaError_t e_ = (call);                                           \
        if (e_ != cudaSuccess) return ::scout::cuda_fail((c), e_, #call);  \
    } while (0)
#define SCOUT_LAUNCH(c, what)                                              \
    do {                                                                   \
        cudaError_t e_ = cudaGetLastError();                               \
        if (e_ != cudaSuccess) return ::scout::cuda_fail((c), e_, what);   \
    } while (0)
#define SCOUT_RC(x)                          \
    do {                                     \
        int rc_ = (x);                       \
        if (rc_ != SCOUT_OK) return rc_;     \
    } while (0)

// End of a repair, after a grid barrier that follows the last change: the changed entries, when
// they are few, beside the counters that the host copies next.
__device__ __forceinline__ void commit_pairs(const int32_t* touched, const int32_t* val, DevCounters* ctr, int32_t* pairs) {
    const int n = ld_volatile(&ctr->changed);
    if (n <= COMMIT_PAIRS)
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            const int32_t v = ld_volatile(touched + i);
            ((int2*)pairs)[i] = make_int2(v, ld_volatile(val + v));
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) ctr->pairs_ok = 1;
}

inline DGraph dgraph(const scout_ctx* c) { return DGraph{c->row, c->pool, (int32_t)c->n}; }
inline int blocks_for(int64_t items, int threads, int cap = 148 * 32) {
    int64_t b = (items + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > cap) b = cap;
    return (int)b;
}

// sort.cu
int sort_keys(scout_ctx* c, unsigned long long* keys, unsigned long long* alt, int64_t n, int bits,
              unsigned long long** sorted_out);
// scan.cu: exclusive scan of int64 values in place; *total receives the sum (device ptr or null)
int scan_i64(scout_ctx* c, int64_t* data, int64_t n, int64_t* d_total);
int sort_reserve(scout_ctx* c, int64_t nkeys);
unsigned next_stamp();   // sort.cu: look-back stamps, unique across the process
// graph.cu: every buffer a batch of up to m edits can grow, allocated now
int graph_reserve_batch(scout_ctx* c, int64_t m);
// problem scratch allocated on first use, or ahead of time by scout_reserve
int cc_ensure(scout_ctx* c);
int coloring_ensure(scout_ctx* c);
// graph.cu
// A merge's row plan (k_row_plan) and a store's update in one launch (k_update)
struct RowPlan {
    Row* row;
    DevCounters* ctr;
    const int32_t* aff;
    const int32_t* seg_b;
    const int32_t* seg_d;
    const int32_t* E;
    const uint32_t* epos;
    MergeRow* mrow;        // short rows of one half-edit from the front, the others from the back
    int64_t mcap;
    int32_t* shorts;       // records of the other short rows
    int64_t* slices;       // (record << 32 | slice, or an insertion item)
    int64_t slice_cap;
    int32_t* longs;        // records of long rows compacted in place
    bool long_in_place;
    bool split;            // rows whose old version is not in HBM go to the second destination
    long long hbm_cap;     // in HBM: 0 <= start < hbm_cap
    long long base_hbm, base_host;
};

struct UpdateParams {
    DGraph g;
    int32_t* pool;
    const scout_edge* e;
    const uint8_t* ops;
    int m, B;
    unsigned long long* raw;    // half-edits as classified (2m)
    unsigned long long* tmp;    // half-edits by bucket (may share E's memory, written later)
    unsigned long long* keys;   // sorted
    uint8_t* eflag;
    uint32_t* epos;             // may share `raw`'s memory: written after the sort
    unsigned long long* split;  // UPDATE_SPLIT
    int* bucket;                // UPDATE_BUCKETS counts
    unsigned long long* cnt;    // heads << 32 | matches per block
    int rows;                   // 0: stop after the plan (tiered store: the host decides where rows go)
    RowPlan rp;                 // its aff, seg_b, seg_d and E are written here
    int32_t *aff, *seg_b, *seg_d, *E;
    GridBar* bar;
};

constexpr int SIDE_MAX = 4;
struct UpdateRound { UpdateParams p[SIDE_MAX]; };
// With `later`, an update of one launch is left to the caller: its parameters in *later, whose m is
// unchanged if the update has been launched (or the batch is empty).
int graph_update(scout_ctx* c, const scout_edge* edits, const uint8_t* ops, int64_t m, scout_batch_stats* st,
                 UpdateParams* later = nullptr);
// k stores' updates in one launch on c's stream, side by side: each on 1/k of the SMs
int update_side(scout_ctx* c, const UpdateRound& r, int k);
int graph_ensure_scratch(scout_ctx* c);
int graph_compact(scout_ctx* c, int64_t min_free, bool nnz_exact = false);
int ws_ensure(scout_ctx* c, int64_t m);
int lists_ensure(scout_ctx* c);
int batch_begin(scout_ctx* c);   // zeroes the counters and the barrier for a new batch
int counters_fetch(scout_ctx* c); // copies the device counters into c->h_ctr (synchronous)
// problem kernels (their .cu files)
// BFS repair variants: 0 incremental, 1 top-down traversal, 2 direction-optimizing
// traversal; mode_dev (device int) overrides mode when the scheduler decides on the device.
constexpr int BFS_MODE_INCREMENTAL = 0, BFS_MODE_TOP_DOWN = 1, BFS_MODE_DIRECTION_OPT = 2;
int bfs_repair(scout_ctx* c, int mode, const int* mode_dev, scout_batch_stats* st);
int bfs_recompute(scout_ctx* c, int32_t source, scout_batch_stats* st);
// CC repair variants: 0 incremental, 1 recompute of every class, 2 recompute of every class
// with an unsettled deletion; mode_dev as for BFS.
int cc_repair(scout_ctx* c, const scout_sched* sched, int variant, const int* mode_dev, scout_batch_stats* st);
int cc_recompute(scout_ctx* c, scout_batch_stats* st);
int coloring_repair(scout_ctx* c, scout_batch_stats* st);
int mis_repair(scout_ctx* c, scout_batch_stats* st);
// sched.cu: features + on-device inference of the installed model; writes ctr->decision.
// Returns SCOUT_OK and sets *mode_dev to the decision's device address when the learned
// policy applies to the problem, else leaves it null (plain policy).
int sched_decide(scout_ctx* c, int problem, int64_t m, bool use_model, const int** mode_dev);
void sched_release(scout_ctx* c);
int sched_variants(int problem);   // repair variants a problem has (BFS 3, CC 2, others 1)
// api.cu: the last repair's (id, value) pairs in page-locked memory (valid until the next call)
int commit_gather(scout_ctx* c, int problem, const int32_t** pairs, int64_t* count);
// Block size of the persistent repair kernels: one block of up to REPAIR_THREADS threads per SM.
// A grid barrier then has 148 arrivals instead of 592 (1.3 against 2.1 us), and the component
// repair, whose hash sets take half an SM's shared memory, runs 1,024 threads per SM instead of
// one 256-thread block (recompute of 2 M vertices: 544 -> 339 us; 50,000-edit batch at scale 20:
// 1,187 -> 1,016 us with its merge). The blocks_per_sm knob takes fewer 256-thread quarters.
// While the tiered store gathers the next batch's rows, a repair takes at most three, whatever the
// knob says, so that the gather's blocks run beside it: four quarters of 64 registers a thread (BFS,
// colouring) hold all of an SM's, and of 56 (components, MIS) leave exactly a gather block's, which
// then started beside the components repair in some runs and after it in others. BFS, 1,000-edit batches
// on 300,000 vertices: the gather ends 70 us after the merge beside three quarters, 118 to 127 beside
// four. The repairs lose nothing by it where the rows lie across the host link (20,000 edits at scale
// 20, three and four quarters: components 1,406 and 1,408 us, MIS 185 and 189; BFS 300 and 215, within
// a call of 3.3 ms that is no shorter for it).
constexpr int REPAIR_THREADS = 1024;
inline int repair_threads(const scout_ctx* c) {
    const int quarters = c->tune_blocks_per_sm > 0 ? c->tune_blocks_per_sm : 4;
    return 256 * (c->tiered && c->gather_active && quarters > 3 ? 3 : quarters);
}
// persistent launch helpers: a launch that waits on d_bar (cleared when it was used before), one
// on a barrier of its own
int coop_launch(scout_ctx* c, const void* fn, int threads, void** args, size_t smem);
int coop_launch_own(scout_ctx* c, const void* fn, int threads, void** args, size_t smem);
int bar_clear(scout_ctx* c, cudaStream_t s);
// gather.cu: the hinted next batch's edits to the device and (tiered store) its cold rows into
// free HBM from `base` on a copy stream, after the current merge is queued; gather_finish waits
// for the gather (main stream and host) and moves the tail.
int prefetch_launch(scout_ctx* c, long long base);
// union.cu: one cooperative launch of the repairs of ne union stores of distinct problems whose
// batches are merged (queued); api.cu: the whole round (merges, launch, counters, stats)
int union_launch(scout_ctx* const* cs, const int* problems, const scout_sched* sds, const int* variants, int ne,
                 const UpdateRound& round, int later, bool side);
bool union_side(scout_ctx* const* cs, const int64_t* counts, int ne);
int union_run(scout_ctx* const* cs, const int* problems, const scout_edge* const* edits, const uint8_t* const* ops,
              const int64_t* counts, int ne, const scout_sched* sched, scout_batch_stats* stats);
// graph.cu: host copy into page-locked staging, over the host threads for large copies
void stage_copy(void* dst, const void* src, size_t bytes);
int gather_finish(scout_ctx* c, double* ms, int64_t* rows, int64_t* bytes);
int gather_reserve(scout_ctx* c, int64_t max_edits);

}  // namespace scout
