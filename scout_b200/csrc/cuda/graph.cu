// graph.cu -- the HBM graph store: row table + element pool, staging from pinned host slabs,
// toggle classification and the per-batch merge of edits into the rows.
//
// Layout. row[v] = {start, len, cap} indexes the int32 pool; every row is kept sorted
// ascending (a sorted multiset: a pair inserted twice in one batch appears twice, as the
// reference's scratchpad appends it twice, core/FlashGraph.h:227-234). A row that gains
// entries, or a long one, is merged into new space at the pool tail and its descriptor
// switched; a short row whose half-edits are all deletions is compacted where it lies (its
// survivors only move towards the row start; only the warp merging it touches it). The host
// compacts the pool when the free space could not hold a full rewrite plus the batch.
//
// Batch merge (replaces DeltaOverlay::insertEdge / removeEdge + neighbors_into,
// core/FlashGraph.h:227-265, done on the device for every affected row at once):
//   k_classify        toggle -> insert/delete by binary search in the shorter row
//                     (HybridGraph::isAdjacent, FlashGraph.h:356-366); emits two half-edit
//                     keys (u, op, v) and (v, op, u) per applied edit
//   sort_keys         groups half-edits by vertex; inserts before deletes; neighbours sorted
//   k_plan            one pass over the sorted half-edits: one search of each in its old row (an
//                     insertion's position, the old entry a deletion cancels by the multiset
//                     rule), the affected rows and their segments, and the running count of
//                     matched deletions (decoupled look-back)
//   k_row_plan        per affected row: its new space (old length + insertions; none for a row
//                     that only loses entries and is short), its new descriptor, its record in
//                     the list of short rows or of slices of longer ones
//   k_merge           the new rows: survivors and insertions of short rows (a few rows per warp)
//                     and of slices of SLICE old entries (a warp each, so a hub row is spread
//                     over many warps), positions taken from the sorted edit events; rows whose
//                     events crowd have their insertions placed by items of their own
//   k_merge_long_inplace  tiered store: rows longer than IN_PLACE_LEN that only lose entries
#include "ctx.cuh"

#include <omp.h>

#include <algorithm>
#include <cstddef>
#include <cstring>

namespace scout {

constexpr int SLICE = 2048;          // old-row entries merged by one warp at a time
constexpr int SMALL_LEN = 128;       // rows up to this length (and 32 half-edits) are short
constexpr int IN_PLACE_LEN = 4096;   // longest deletion-only row compacted in place by one warp
constexpr int HEAVY = 1024;          // half-edits from which a row may be heavy (heavy_row), and the insertions
                                     // of one merge item of such a row
constexpr int64_t INS_ITEM = 1ll << 31;     // in the slice list: such an item,
constexpr int64_t HEAVY_ITEM = 1ll << 30;   // a slice of a heavy row

// A row whose half-edits are all deletions is rewritten in place: its survivors only move
// towards the row start, it keeps its start and capacity, and it takes no pool space (one warp
// merges the whole row). A longer one is compacted in place by one block (k_merge_long_inplace:
// its slices would overlap) only when `long_in_place` is set, in the tiered store, whose HBM
// room is scarce; in the all-HBM store it is rewritten at the pool tail, spread over many warps.
__host__ __device__ __forceinline__ bool in_place_row(long long insertions, int old_len, bool long_in_place) {
    return insertions == 0 && (old_len <= IN_PLACE_LEN || long_in_place);
}

__device__ __forceinline__ bool in_hbm(const Row& r, long long cap) { return r.start >= 0 && r.start < cap; }

// ---------------------------------------------------------------------------------------
// Staging
// ---------------------------------------------------------------------------------------
__global__ void k_rows_from_offsets(Row* __restrict__ row, const int64_t* __restrict__ off, int64_t n, long long base) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        long long s = off[v], e = off[v + 1];
        row[v] = Row{base + s, (int)(e - s), (int)(e - s)};
    }
}

__global__ void k_rows_from_stage(Row* __restrict__ row, const int32_t* __restrict__ ids, const int64_t* __restrict__ off,
                                  int64_t nrows, long long base, int32_t n, int* __restrict__ bad) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nrows; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t v = ids[i];
        if (v < 0 || v >= n) { atomicExch(bad, 1); continue; }
        long long s = off[i] - off[0], e = off[i + 1] - off[0];
        row[v] = Row{base + s, (int)(e - s), (int)(e - s)};
    }
}

// One warp per row: flags rows that are not ascending and counts entries out of range.
__global__ void k_check_rows(const Row* __restrict__ row, const int32_t* __restrict__ pool, int32_t n,
                             int32_t* __restrict__ unsorted, int* __restrict__ n_unsorted, int* __restrict__ bad) {
    for (int v = gwarp_id(); v < n; v += gwarp_count()) {
        Row r = row[v];
        bool ok = true, range_ok = true;
        for (long long i = lane_id(); i < r.len; i += WARP) {
            int32_t x = pool[r.start + i];
            if (x < 0 || x >= n) range_ok = false;
            if (i + 1 < r.len && pool[r.start + i + 1] < x) ok = false;
        }
        ok = __all_sync(0xffffffffu, ok);
        range_ok = __all_sync(0xffffffffu, range_ok);
        if (!range_ok && lane_id() == 0) atomicExch(bad, 1);
        if (!ok && lane_id() == 0) unsorted[atomicAdd(n_unsorted, 1)] = v;
    }
}

// Sort of one unsorted row by one block (bitonic in shared memory, rows up to 8192).
__global__ void k_sort_rows_small(const Row* __restrict__ row, int32_t* __restrict__ pool,
                                  const int32_t* __restrict__ list, int count, int* __restrict__ too_big) {
    __shared__ int32_t s[8192];
    for (int k = blockIdx.x; k < count; k += gridDim.x) {
        Row r = row[list[k]];
        if (r.len > 8192) { if (threadIdx.x == 0) atomicExch(too_big, 1); continue; }
        int p = 1;
        while (p < r.len) p <<= 1;
        for (int i = threadIdx.x; i < p; i += blockDim.x) s[i] = i < r.len ? pool[r.start + i] : INT32_MAX;
        __syncthreads();
        for (int size = 2; size <= p; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int i = threadIdx.x; i < p; i += blockDim.x) {
                    int j = i ^ stride;
                    if (j > i) {
                        bool up = (i & size) == 0;
                        int32_t a = s[i], b = s[j];
                        if ((a > b) == up) { s[i] = b; s[j] = a; }
                    }
                }
                __syncthreads();
            }
        for (int i = threadIdx.x; i < r.len; i += blockDim.x) pool[r.start + i] = s[i];
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------
// Classification and half-edit keys
// ---------------------------------------------------------------------------------------
// Key layout: (u << (B + 1)) | (op << B) | v, op 0 = insert, 1 = delete; B = bits(n), so the
// all-ones sentinel sorts after every real key.
__device__ __forceinline__ unsigned long long pack_key(uint32_t u, uint32_t op, uint32_t v, int B) {
    return ((unsigned long long)u << (B + 1)) | ((unsigned long long)op << B) | v;
}

// One edit's classification: bit 0 valid, bit 1 insertion, bit 2 applied. WIDE as in plan_search.
template <bool WIDE>
__device__ __forceinline__ int classify_edit(const DGraph& g, int32_t u, int32_t v, int op) {
    if (!(u >= 0 && u < g.n && v >= 0 && v < g.n && u != v)) return 0;
    const bool adj = WIDE ? dg_adjacent_wide(g, u, v) : dg_adjacent(g, u, v);
    bool ins = op == SCOUT_OP_INSERT, applied = op == SCOUT_OP_INSERT ? !adj : adj;
    if (op != SCOUT_OP_INSERT && op != SCOUT_OP_DELETE) { ins = !adj; applied = true; }
    return 1 | (ins ? 2 : 0) | (applied ? 4 : 0);
}

__global__ void k_classify(DGraph g, const scout_edge* __restrict__ e, const uint8_t* __restrict__ ops, int64_t m,
                           int B, unsigned long long* __restrict__ keys, uint8_t* __restrict__ eflag,
                           DevCounters* __restrict__ ctr, int emit) {
    const unsigned long long SENT = (B + B + 1) >= 64 ? ~0ull : ((1ull << (B + B + 1)) - 1);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t u = e[i].u, v = e[i].v;
        const int f = classify_edit<false>(g, u, v, ops ? ops[i] : SCOUT_OP_TOGGLE);
        const bool valid = f & 1, ins = f & 2, applied = f & 4;
        eflag[i] = (uint8_t)f;
        unsigned mi = __ballot_sync(__activemask(), valid && ins);
        unsigned md = __ballot_sync(__activemask(), valid && !ins);
        unsigned ma = __ballot_sync(__activemask(), valid && applied);
        if (ctr && lane_id() == (unsigned)(__ffs(__activemask()) - 1)) {
            if (mi) atomicAdd(&ctr->n_ins, __popc(mi));
            if (md) atomicAdd(&ctr->n_del, __popc(md));
            if (ma) atomicAdd(&ctr->n_half, 2 * __popc(ma));
        }
        if (emit) {
            if (valid && applied) {
                uint32_t op = ins ? 0u : 1u;
                keys[2 * i] = pack_key((uint32_t)u, op, (uint32_t)v, B);
                keys[2 * i + 1] = pack_key((uint32_t)v, op, (uint32_t)u, B);
            } else {
                keys[2 * i] = SENT;
                keys[2 * i + 1] = SENT;
            }
        }
    }
}

__device__ __forceinline__ int32_t key_u(unsigned long long k, int B) { return (int32_t)(k >> (B + 1)); }
__device__ __forceinline__ int32_t key_v(unsigned long long k, int B) { return (int32_t)(k & ((1ull << B) - 1)); }
__device__ __forceinline__ int key_op(unsigned long long k, int B) { return (int)((k >> B) & 1ull); }

constexpr int PLAN_THREADS = 256;
constexpr int PLAN_WARPS = PLAN_THREADS / WARP;
constexpr int PLAN_STEPS = 4;                          // half-edits per thread, their searches interleaved
constexpr int PLAN_TILE = PLAN_THREADS * PLAN_STEPS;
constexpr uint64_t PLAN_WAIT_LIMIT_NS = 1000000000ull;   // 1 s
constexpr unsigned long long PLAN_TAG = 0x5Aull << 56;

// One pass over the sorted half-edits. Each is searched once in its old row:
//   insertion y   position = number of old entries <= y; it is placed before that entry
//   deletion d    multiset rule: the r-th copy of d among a row's deletions cancels the r-th copy
//                 of d in the old row (DeltaOverlay::removeEdge forgets one added copy or
//                 tombstones the base edge, FlashGraph.h:236-243); position = the cancelled
//                 entry, or the end of d's copies when none is left (not matched)
// epos[k] = position << 1 | matched, non-decreasing along a row's insertions and along its
// deletions; E[k] = matched deletions before half-edit k (E[n_half] the total); the affected
// rows in id order with their segments (seg_b[a], seg_b[a + 1]) and first deletions seg_d[a].
// The running counts of heads and matched deletions go from tile to tile by a decoupled
// look-back (state: three words per tile, as in the single-pass scan).
//
// What bounds it: dependent reads of the binary searches (a thread keeps PLAN_STEPS searches
// in flight, and neighbouring threads search the same rows). 10^6 edits at scale 22: 123 us; the
// launches it replaces (segment heads and tails, two searches of every half-edit, a scan and its
// clears) took 300 us, and on small batches most of their time was the seven launches.
//
// plan_search: the searches of a thread's half-edits k0 + STRIDE s (`at(k)` reads sorted half-edit
// k), their positions, and the warps' head and match ballots. Warps converge on return.
// WIDE: three probes per step (a quarter of the range is left) where the chain of dependent
// reads is all there is, on batches too small to fill the memory system; one probe (half) else.
template <int STEPS, int STRIDE, bool WIDE, typename At>
__device__ __forceinline__ void plan_search(const Row* __restrict__ row, const int32_t* __restrict__ pool,
                                            const unsigned long long (&key)[STEPS], int B, int nh, int k0, At at,
                                            uint32_t* __restrict__ epos, unsigned (&hm)[STEPS], unsigned (&mm)[STEPS]) {
    const int32_t* O[STEPS];
    int lo[STEPS], hi[STEPS], len[STEPS];
#pragma unroll
    for (int s = 0; s < STEPS; s++) {
        lo[s] = hi[s] = len[s] = 0;
        O[s] = pool;
        if (k0 + s * STRIDE < nh) {
            const Row r = row[key_u(key[s], B)];
            O[s] = pool + r.start;
            len[s] = hi[s] = r.len;
        }
    }
    // lower bounds, one step of every search per turn
    while (true) {
        bool more = false;
        int32_t x[STEPS], x1[STEPS], x3[STEPS];
#pragma unroll
        for (int s = 0; s < STEPS; s++)
            if (lo[s] < hi[s]) {
                const int n = hi[s] - lo[s];
                x[s] = O[s][lo[s] + (n >> 1)];
                if (WIDE) {
                    x1[s] = O[s][lo[s] + (n >> 2)];
                    x3[s] = O[s][lo[s] + (n >> 1) + (n >> 2)];
                }
            }
#pragma unroll
        for (int s = 0; s < STEPS; s++)
            if (lo[s] < hi[s]) {
                const int32_t y = key_v(key[s], B);
                const int n = hi[s] - lo[s], mid = lo[s] + (n >> 1), q1 = lo[s] + (n >> 2), q3 = mid + (n >> 2);
                if (x[s] < y) lo[s] = mid + 1; else hi[s] = mid;
                if (WIDE) {   // q1 <= mid <= q3 < the old hi
                    if (x1[s] >= y) hi[s] = min(hi[s], q1); else lo[s] = max(lo[s], q1 + 1);
                    if (x3[s] < y) lo[s] = max(lo[s], q3 + 1); else hi[s] = min(hi[s], q3);
                }
                more |= lo[s] < hi[s];
            }
        if (!more) break;
    }
#pragma unroll
    for (int s = 0; s < STEPS; s++) {
        const int k = k0 + s * STRIDE;
        bool matched = false, head = false;
        if (k < nh) {
            const unsigned long long kk = key[s];
            const int32_t y = key_v(kk, B);
            const unsigned long long pk = k > 0 ? at(k - 1) : ~kk;
            head = k == 0 || key_u(pk, B) != key_u(kk, B);
            int pos = lo[s];
            const bool here = pos < len[s] && O[s][pos] == y;
            if (key_op(kk, B) == 0) {
                if (here) pos += (int)upper_bound_i32(O[s] + pos, len[s] - pos, y);
            } else {
                int rank = 0;   // copies of this deletion before it: doubling steps back, then a search
                if (pk == kk) {
                    int j = k - 1, step = 1;   // j is a copy, lo2 lies before the first one (or at -1)
                    while (j - step >= 0 && at(j - step) == kk) {
                        j -= step;
                        step <<= 1;
                    }
                    int lo2 = max(j - step, -1);
                    while (j - lo2 > 1) {
                        const int mid = (lo2 + j) >> 1;
                        if (at(mid) == kk) j = mid; else lo2 = mid;
                    }
                    rank = k - j;
                }
                matched = here && pos + rank < len[s] && O[s][pos + rank] == y;
                if (matched) pos += rank;
                else if (here) pos += (int)upper_bound_i32(O[s] + pos, len[s] - pos, y);
            }
            epos[k] = ((uint32_t)pos << 1) | (matched ? 1u : 0u);
        }
        hm[s] = __ballot_sync(0xffffffffu, head);
        mm[s] = __ballot_sync(0xffffffffu, matched);
    }
}

// plan_finish: the segments and running counts, given the heads << 32 | matches before the warp.
template <int STEPS, typename At>
__device__ __forceinline__ void plan_finish(const unsigned long long (&key)[STEPS], int B, int nh, int k0, At at,
                                            const unsigned (&hm)[STEPS], const unsigned (&mm)[STEPS],
                                            unsigned long long base, DevCounters* __restrict__ ctr,
                                            int32_t* __restrict__ aff, int32_t* __restrict__ seg_b,
                                            int32_t* __restrict__ seg_d, int32_t* __restrict__ E) {
    const unsigned l = lane_id(), lt = (1u << l) - 1;
    int heads = (int)(base >> 32), match = (int)(base & 0xffffffffu);
#pragma unroll
    for (int s = 0; s < STEPS; s++) {
        const int k = k0 + s * WARP;
        if (k < nh) {
            const unsigned long long kk = key[s];
            const int32_t u = key_u(kk, B);
            const bool head = (hm[s] >> l) & 1u;
            const int a = heads + __popc(hm[s] & lt) + (head ? 1 : 0) - 1;
            const int e = match + __popc(mm[s] & lt);
            E[k] = e;
            if (head) {
                aff[a] = u;
                seg_b[a] = k;
            }
            const int op = key_op(kk, B);
            if (op == 1) {
                if (head || key_op(at(k - 1), B) == 0) seg_d[a] = k;
            } else if (k == nh - 1 || key_u(at(k + 1), B) != u) {
                seg_d[a] = k + 1;
            }
            if (k == nh - 1) {
                E[nh] = e + (int)((mm[s] >> l) & 1u);
                seg_b[a + 1] = nh;
                ctr->n_aff = a + 1;
            }
        }
        heads += __popc(hm[s]);
        match += __popc(mm[s]);
    }
}

template <int STEPS>
__device__ __forceinline__ unsigned long long plan_count(const unsigned (&hm)[STEPS], const unsigned (&mm)[STEPS]) {
    unsigned long long c = 0;
#pragma unroll
    for (int s = 0; s < STEPS; s++) c += ((unsigned long long)__popc(hm[s]) << 32) | (unsigned)__popc(mm[s]);
    return c;
}

__global__ void __launch_bounds__(PLAN_THREADS) k_plan(const Row* __restrict__ row, const int32_t* __restrict__ pool,
                                                       const unsigned long long* __restrict__ keys, int B,
                                                       DevCounters* __restrict__ ctr, int32_t* __restrict__ aff,
                                                       int32_t* __restrict__ seg_b, int32_t* __restrict__ seg_d,
                                                       uint32_t* __restrict__ epos, int32_t* __restrict__ E,
                                                       unsigned long long* __restrict__ st, unsigned stamp) {
    __shared__ int s_tile;
    __shared__ unsigned long long s_cnt[PLAN_WARPS];
    __shared__ unsigned long long s_prefix;
    const int nh = ctr->n_half;
    const int w = threadIdx.x / WARP;
    const unsigned l = lane_id();
    if (threadIdx.x == 0) s_tile = atomicAdd(&ctr->plan_ticket, 1);
    __syncthreads();
    const int tile = s_tile;
    if (tile * (long long)PLAN_TILE >= nh) return;   // whole block; no tile after it has work either
    const int k0 = tile * PLAN_TILE + w * (PLAN_STEPS * WARP) + (int)l;
    auto at = [&](int k) { return keys[k]; };
    unsigned long long key[PLAN_STEPS];
#pragma unroll
    for (int s = 0; s < PLAN_STEPS; s++) {
        const int k = k0 + s * WARP;
        key[s] = k < nh ? keys[k] : ~0ull;
    }
    unsigned hm[PLAN_STEPS], mm[PLAN_STEPS];
    plan_search<PLAN_STEPS, WARP, false>(row, pool, key, B, nh, k0, at, epos, hm, mm);
    if (l == 0) s_cnt[w] = plan_count<PLAN_STEPS>(hm, mm);
    __syncthreads();
    if (w == 0) {   // publish, look back 32 tiles per step, publish the prefix
        unsigned long long tot = 0;
        for (int j = 0; j < PLAN_WARPS; j++) tot += s_cnt[j];
        const unsigned long long want = PLAN_TAG | ((unsigned long long)stamp << 2);
        unsigned long long* me = st + 3 * (int64_t)tile;
        unsigned long long prefix = 0;
        if (tile > 0) {
            if (l == 0) {
                me[1] = tot;
                __threadfence();
                *(volatile unsigned long long*)me = want | 1ull;
            }
            const uint64_t t0 = globaltimer_ns();
            for (int end = tile - 1;; end -= WARP) {
                const int j = end - (int)l;           // lane 0 looks at the nearest tile
                unsigned long long sw = want | 2ull;  // tiles before the first: a prefix of 0
                bool ok = true;
                if (j >= 0) {
                    const unsigned long long* pj = st + 3 * (int64_t)j;
                    sw = ld_volatile(pj);
                    for (unsigned it = 1; (sw & ~3ull) != want || (sw & 3ull) == 0; it++) {
                        if ((it & 63) == 0 && globaltimer_ns() - t0 > PLAN_WAIT_LIMIT_NS) { ok = false; break; }
                        sw = ld_volatile(pj);
                    }
                }
                if (!__all_sync(0xffffffffu, ok)) {
                    if (l == 0) atomicCAS(&ctr->sort_err, 0, 4);
                    break;
                }
                __threadfence();
                const bool pre = (sw & 3ull) == 2;
                unsigned long long v = 0;
                if (j >= 0) v = ld_volatile(st + 3 * (int64_t)j + (pre ? 2 : 1));
                const unsigned pm = __ballot_sync(0xffffffffu, pre);
                const int f = pm ? __ffs(pm) - 1 : WARP;   // nearest tile with an inclusive prefix
                if ((int)l > f) v = 0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                prefix += v;
                if (pm) break;
            }
        }
        if (l == 0) {
            me[2] = prefix + tot;
            __threadfence();
            *(volatile unsigned long long*)me = want | 2ull;
            s_prefix = prefix;
        }
    }
    __syncthreads();
    unsigned long long base = s_prefix;
    for (int j = 0; j < w; j++) base += s_cnt[j];
    plan_finish<PLAN_STEPS>(key, B, nh, k0, at, hm, mm, base, ctr, aff, seg_b, seg_d, E);
}

// Per affected row: the space of its new version (old length + insertions: slots of matched
// deletions stay unused until the next compaction), its new descriptor and its merge record.
// Space and list slots are taken by one set of atomics per block (the order of rows in the pool
// does not matter).
constexpr int ROW_THREADS = 256;

// Exclusive scans of two values over the block (at most 32 warps) at once, and their totals.
__device__ __forceinline__ void block_scan2(long long& x, long long& y, long long* tx, long long* ty) {
    __shared__ long long ws[2][WARP + 1];
    const int w = threadIdx.x / WARP, l = (int)lane_id();
    const long long ix = warp_incl_scan(x), iy = warp_incl_scan(y);
    if (l == WARP - 1) { ws[0][w] = ix; ws[1][w] = iy; }
    __syncthreads();
    if (w < 2) {
        const long long v = l < (int)(blockDim.x / WARP) ? ws[w][l] : 0;
        const long long iv = warp_incl_scan(v);
        ws[w][l] = iv - v;
        if (l == WARP - 1) ws[w][WARP] = iv;
    }
    __syncthreads();
    x = ws[0][w] + ix - x;
    y = ws[1][w] + iy - y;
    *tx = ws[0][WARP];
    *ty = ws[1][WARP];
}

// Tiered store: the growth of each destination, before anything is placed.
__global__ void __launch_bounds__(ROW_THREADS) k_row_sizes(RowPlan p) {
    const int A = p.ctr->n_aff;
    long long nh = 0, nc = 0;
    for (int a = blockIdx.x * ROW_THREADS + threadIdx.x; a < A; a += gridDim.x * ROW_THREADS) {
        const Row r = p.row[p.aff[a]];
        const int ins = p.seg_d[a] - p.seg_b[a];
        if (in_place_row(ins, r.len, p.long_in_place)) continue;
        if (p.split && !in_hbm(r, p.hbm_cap)) nc += (long long)r.len + ins;
        else nh += (long long)r.len + ins;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        nh += __shfl_xor_sync(0xffffffffu, nh, o);
        nc += __shfl_xor_sync(0xffffffffu, nc, o);
    }
    if (lane_id() == 0 && nh) atomicAdd((unsigned long long*)&p.ctr->new_elems, (unsigned long long)nh);
    if (lane_id() == 0 && nc) atomicAdd((unsigned long long*)&p.ctr->new_elems_host, (unsigned long long)nc);
}

// Rows whose events crowd: more than twice as many as old entries, or HEAVY in a row (of insertions, or
// of deletions) within HEAVY / 2 entries. A warp walks a slice's events 32 at a time, which is the
// faster where they are spread (64 streams of small graphs under batches of up to a quarter of
// their entries: updates of all their batches 11.8 ms, 13.2 when every row of more than HEAVY half-edits
// was searched).
__device__ __forceinline__ bool heavy_row(const uint32_t* epos, int len, int b, int d, int e) {
    if (e - b <= HEAVY) return false;
    bool crowd = (long long)(e - b) > 2LL * len;
    for (int k = b; !crowd && k + HEAVY < d; k += HEAVY) crowd = (epos[k + HEAVY] >> 1) - (epos[k] >> 1) < HEAVY / 2;
    for (int k = d; !crowd && k + HEAVY < e; k += HEAVY) crowd = (epos[k + HEAVY] >> 1) - (epos[k] >> 1) < HEAVY / 2;
    return crowd;
}

// BLOCK: rows are taken a block's threads at a time, with one set of atomics on the counters;
// else 32 at a time by a warp, with no barrier (few rows, nothing to save on atomics).
template <bool BLOCK>
__device__ __forceinline__ void row_plan(const RowPlan& p, int A, int group, int groups) {
    const int ROWS = BLOCK ? (int)blockDim.x : WARP;
    __shared__ long long s_base[7];
    const int t = BLOCK ? (int)threadIdx.x : (int)lane_id();
    long long nnz_delta = 0, bytes = 0;
    for (int a0 = group * ROWS; a0 < A; a0 += groups * ROWS) {
        const int a = a0 + t;
        const bool ok = a < A;
        Row r{0, 0, 0};
        int32_t u = 0;
        int b = 0, d = 0, e = 0, nl = 0, ns = 0, ni = 0;   // ns old slices, ni insertion items
        bool ip = false, cold = false, one = false, sm = false, lip = false, heavy = false;
        if (ok) {
            u = p.aff[a];
            b = p.seg_b[a];
            d = p.seg_d[a];
            e = p.seg_b[a + 1];
            r = p.row[u];
            nl = r.len + (d - b) - (p.E[e] - p.E[d]);
            ip = in_place_row(d - b, r.len, p.long_in_place);
            cold = p.split && !in_hbm(r, p.hbm_cap);
            lip = ip && r.len > IN_PLACE_LEN;
            one = r.len <= SMALL_LEN && e - b == 1;
            sm = !one && r.len <= SMALL_LEN && e - b <= WARP;
            ns = one || sm || lip ? 0 : ip ? 1 : max(1, (r.len + SLICE - 1) / SLICE);
            heavy = ns > 0 && heavy_row(p.epos, r.len, b, d, e);
            if (heavy) ni = (d - b + HEAVY - 1) / HEAVY;
            nnz_delta += nl - r.len;
            bytes += 4LL * ((long long)r.len + nl) + 8LL * (e - b) + 16;
        }
        const long long need = ok && !ip ? (long long)r.len + (d - b) : 0;
        // counts packed: slices 30 bits, rows of one half-edit, other rows, short ones 11 bits each
        long long th, tc = 0, tn, tl = 0, oh = cold ? 0 : need, oc = 0, ol = lip;
        long long on = (long long)(ns + ni) | ((long long)(ok && one) << 30) | ((long long)(ok && !one) << 41) | ((long long)sm << 52);
        auto scan2 = [](long long& x, long long& y, long long* tx, long long* ty) {
            if (BLOCK) {
                block_scan2(x, y, tx, ty);
            } else {
                const long long ix = warp_incl_scan(x), iy = warp_incl_scan(y);
                x = ix - x;
                y = iy - y;
                *tx = __shfl_sync(0xffffffffu, ix, WARP - 1);
                *ty = __shfl_sync(0xffffffffu, iy, WARP - 1);
            }
        };
        scan2(oh, on, &th, &tn);
        if (p.long_in_place) {   // tiered store: the second destination, the long rows in place
            oc = cold ? need : 0;
            if (BLOCK) __syncthreads();   // the first scan's sums are read
            scan2(oc, ol, &tc, &tl);
        }
        // one thread per counter: the atomics' latencies overlap
        long long base = 0;
        if (t < 2) {
            const long long x = t ? tc : th;
            if (x)
                base = (long long)atomicAdd((unsigned long long*)(t ? &p.ctr->new_elems_host : &p.ctr->new_elems),
                                            (unsigned long long)x);
        } else if (t < 7) {
            int* to = t == 2 ? &p.ctr->n_slices : t == 3 ? &p.ctr->n_one : t == 4 ? &p.ctr->n_rest
                      : t == 5 ? &p.ctr->n_short : &p.ctr->n_long;
            const int x = t == 6 ? (int)tl : t == 2 ? (int)(tn & ((1ll << 30) - 1)) : (int)(tn >> (30 + 11 * (t - 3))) & 2047;
            if (x) base = atomicAdd(to, x);
        }
        long long bs[7];
        if (BLOCK) {
            if (t < 7) s_base[t] = base;
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < 7; j++) bs[j] = BLOCK ? s_base[j] : __shfl_sync(0xffffffffu, base, j);
        if (ok) {
            long long dst = r.start;
            if (!ip) dst = cold ? p.base_host + bs[1] + oc : p.base_hbm + bs[0] + oh;
            const long long at = one ? bs[3] + ((on >> 30) & 2047) : p.mcap - 1 - (bs[4] + ((on >> 41) & 2047));
            p.mrow[at] = MergeRow{r.start, dst, r.len, b, d, e};
            p.row[u] = ip ? Row{r.start, nl, r.cap} : Row{dst, nl, r.len + (d - b)};
            if (sm) p.shorts[bs[5] + ((on >> 52) & 2047)] = (int32_t)at;
            if (lip) p.longs[bs[6] + ol] = (int32_t)at;
            const long long s0 = bs[2] + (on & ((1ll << 30) - 1));
            if (s0 + ns + ni > p.slice_cap) {
                if (ns + ni) atomicExch(&p.ctr->overflow, 1);
            } else {
                for (int s = 0; s < ns; s++) p.slices[s0 + s] = (at << 32) | (heavy ? HEAVY_ITEM : 0) | s;
                for (int s = 0; s < ni; s++) p.slices[s0 + ns + s] = (at << 32) | INS_ITEM | s;
            }
        }
        if (BLOCK) __syncthreads();   // the bases and sums are read before the next rows overwrite them
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        nnz_delta += __shfl_xor_sync(0xffffffffu, nnz_delta, o);
        bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
    }
    if (lane_id() == 0 && (nnz_delta || bytes)) {
        atomicAdd((unsigned long long*)&p.ctr->nnz_delta, (unsigned long long)nnz_delta);
        atomicAdd((unsigned long long*)&p.ctr->update_bytes, (unsigned long long)bytes);
    }
}

__global__ void __launch_bounds__(ROW_THREADS) k_row_plan(RowPlan p) {
    row_plan<true>(p, p.ctr->n_aff, (int)blockIdx.x, (int)gridDim.x);
}

// ---- the merge -------------------------------------------------------------------------------
// A row's new version is its old one with every entry moved by a count: old entry e that is not
// cancelled lands at e + (insertions at positions <= e) - (matched deletions before e), and
// insertion j of position i at i + j - (matched deletions before i). Between two events of the
// row's sorted edit list the shift is constant, so the merge compares no values: a warp enters
// the events of 1,024 old entries into bitmaps, a lane per event, and copies the entries 32 at a
// time, each finding its shift by counting bits.
// Rows go three ways: short ones of one half-edit (most rows of a batch) by eight lanes each, other
// rows of at most 32 half-edits with a lane per event, the rest slice by slice with their
// events entered chunk by chunk.
// What bounds it: on large graphs reads of rows scattered over the pool (10^6 preferential edits
// at scale 22, 0.92 GB of rows: 328 us; 10^4 there, 0.25 GB: 58 us), on smaller ones the
// instructions per event (500,000 edits at scale 20: 120 us, 186 with every event of a slice
// searched on its own). The three kernels before it and the scan they waited on, which searched
// the insertions for every surviving entry, took 680 and 122 us at scale 22.
constexpr int MERGE_THREADS = 256;
constexpr int MERGE_WARPS = MERGE_THREADS / WARP;
constexpr int MERGE_U = 8;                 // 32-entry groups of a slice in flight
constexpr int MERGE_ROWS = 4;              // short rows in flight per warp

// The events of MERGE_CHUNK old entries of a row, in shared memory (one per warp).
constexpr int MERGE_CHUNK = 32 * WARP;
// Word w of a chunk's 32: x a bit per cancelled entry, y a bit per entry that insertions go
// before, z insertions before the word (bit 30: several go before one entry), w cancelled
// entries before the word.
typedef uint4 ChunkEvents[WARP];

// First half-edit in [b, e) whose position is >= x (positions ascending), 32 probes per step;
// every lane calls it and gets the same answer.
__device__ __forceinline__ int warp_lb_event(const uint32_t* epos, int b, int e, int x) {
    int lo = b, hi = e;
    while (hi - lo > WARP) {
        const int step = (hi - lo + WARP - 1) / WARP;
        const int at = lo + (int)lane_id() * step;
        const int c = __popc(__ballot_sync(0xffffffffu, at < hi && (int)(epos[at] >> 1) < x));   // probes below x
        if (c == 0) { hi = lo; break; }
        const int nlo = lo + (c - 1) * step + 1;
        hi = min(hi, lo + c * step);
        lo = nlo;
    }
    const int at = lo + (int)lane_id();
    return lo + __popc(__ballot_sync(0xffffffffu, at < hi && (int)(epos[at] >> 1) < x));
}

// The events in [c0, c1) of the row (half-edits from *ii and *id on) are entered, a lane each:
// insertions written to their places, the words left for the entries. Both cursors move past
// the chunk. Returns the chunk's cancelled entries.
static __device__ __forceinline__ int chunk_events(int32_t* __restrict__ N, const unsigned long long* __restrict__ keys,
                                                   int B, const uint32_t* __restrict__ epos, const MergeRow& r, int c0,
                                                   int c1, int* ii, int* id, bool any_ins, bool any_del, int gone,
                                                   ChunkEvents& ev) {
    const int l = (int)lane_id();
    __syncwarp();   // the previous chunk's words are read
    ev[l] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    int dtot = 0;
    if (any_del) {
        for (int k = *id;; k += WARP) {
            const uint32_t e = k + l < r.e ? epos[k + l] : ~0u;
            const int pos = (int)(e >> 1);
            const bool in = pos < c1;
            if (in && (e & 1u)) atomicOr(&ev[(pos - c0) >> 5].x, 1u << ((pos - c0) & 31));
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (m != 0xffffffffu) { *id = k + __popc(m); break; }
        }
        __syncwarp();
        const int mine = __popc(ev[l].x);
        const int inc = warp_incl_scan_i(mine);
        dtot = __shfl_sync(0xffffffffu, inc, WARP - 1);
        ev[l].w = (unsigned)(inc - mine);
        __syncwarp();
    }
    if (any_ins) {
        for (int k = *ii;; k += WARP) {
            const int pos = k + l < r.d ? (int)(epos[k + l] >> 1) : INT32_MAX;
            const bool in = pos < c1;
            if (in) {
                const int w = (pos - c0) >> 5;
                const unsigned bit = 1u << ((pos - c0) & 31);
                atomicOr(&ev[w].y, bit);
                atomicAdd(&ev[w].z, 1u);
                N[pos + (k + l - r.b) - gone - (int)ev[w].w - __popc(ev[w].x & (bit - 1))] = key_v(keys[k + l], B);
            }
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (m != 0xffffffffu) { *ii = k + __popc(m); break; }
        }
        __syncwarp();
        const int cnt = (int)ev[l].z;
        const int inc = warp_incl_scan_i(cnt);
        ev[l].z = (unsigned)(inc - cnt) | (__popc(ev[l].y) != cnt ? 1u << 30 : 0u);
        __syncwarp();
    }
    return dtot;
}

// Old entries [s0, s1) of one row, by one warp.
static __device__ __forceinline__ void merge_slice(int32_t* __restrict__ pool, const unsigned long long* __restrict__ keys,
                                                   int B, const uint32_t* __restrict__ epos, const int32_t* __restrict__ E,
                                                   const MergeRow& r, int s0, int s1, ChunkEvents& ev) {
    constexpr int STEP = MERGE_U * WARP;
    const int l = (int)lane_id();
    const unsigned lt = (1u << l) - 1, le = lt | (1u << l);
    const int32_t* O = pool + r.start + l;   // this lane's entry of a group at 0
    int32_t* N = pool + r.dst;
    int32_t x[MERGE_U];
#pragma unroll
    for (int u = 0; u < MERGE_U; u++) x[u] = s0 + u * WARP + l < s1 ? O[s0 + u * WARP] : 0;
    int id = r.d, ii = r.b;   // events not below the chunk
    if (s0 > 0) {
        ii = warp_lb_event(epos, r.b, r.d, s0);
        id = warp_lb_event(epos, r.d, r.e, s0);
    }
    int gone = id > r.d ? E[id] - E[r.d] : 0;   // matched deletions before the chunk
    for (int c0 = s0; c0 < s1; c0 += MERGE_CHUNK) {
        const int c1 = min(c0 + MERGE_CHUNK, s1);
        const int shift = (ii - r.b) - gone;
        const int ni = ii < r.d ? (int)(epos[ii] >> 1) : INT32_MAX, nd = id < r.e ? (int)(epos[id] >> 1) : INT32_MAX;
        const int ib = ii;
        const bool quiet = ni >= c1 && nd >= c1;   // no event among the chunk's entries
        if (!quiet) gone += chunk_events(N, keys, B, epos, r, c0, c1, &ii, &id, ni < c1, nd < c1, gone, ev);
        for (int b0 = c0; b0 < c1; b0 += STEP) {
            int32_t nx[MERGE_U];
            if (b0 + 2 * STEP <= s1) {
#pragma unroll
                for (int u = 0; u < MERGE_U; u++) nx[u] = O[b0 + STEP + u * WARP];
            } else {
#pragma unroll
                for (int u = 0; u < MERGE_U; u++) nx[u] = b0 + STEP + u * WARP + l < s1 ? O[b0 + STEP + u * WARP] : 0;
            }
            __syncwarp();   // a row compacted where it lies: these loads precede the stores below
            int32_t* M = N + b0 + shift + l;
            if (quiet && b0 + STEP <= c1) {
#pragma unroll
                for (int u = 0; u < MERGE_U; u++) M[u * WARP] = x[u];
            } else if (quiet) {
#pragma unroll
                for (int u = 0; u < MERGE_U; u++)
                    if (b0 + u * WARP + l < c1) M[u * WARP] = x[u];
            } else {
#pragma unroll
                for (int u = 0; u < MERGE_U; u++) {
                    const uint4 w = ev[(b0 - c0) / WARP + u];
                    int to = (int)(w.z & ~(1u << 30)) - (int)w.w - __popc(w.x & lt);
                    if (w.z >> 30) {   // uniform: several insertions before one entry, counted one by one
                        for (int k = ib + (int)(w.z & ~(1u << 30)); k < r.d; k++) {
                            const int pos = (int)(epos[k] >> 1);
                            if (pos >= b0 + (u + 1) * WARP) break;
                            to += pos <= b0 + u * WARP + l;
                        }
                    } else {
                        to += __popc(w.y & le);
                    }
                    if (b0 + u * WARP + l < c1 && !((w.x >> l) & 1u)) M[u * WARP + to] = x[u];
                }
            }
#pragma unroll
            for (int u = 0; u < MERGE_U; u++) x[u] = nx[u];
        }
    }
    if (s1 == r.len)   // insertions past the last entry
        for (int k = ii + l; k < r.d; k += WARP) N[r.len + (k - r.b) - gone] = key_v(keys[k], B);
}

// First half-edit in [lo, hi) whose position is >= x, by one lane.
__device__ __forceinline__ int lb_event(const uint32_t* __restrict__ epos, int lo, int hi, int x) {
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((int)(epos[mid] >> 1) < x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Heavy rows. Their events may all lie in one gap of a short row (a vertex that gains its neighbours in
// one batch) or repeat one pair, so nothing walks them: insertions are items of HEAVY of them, each
// placed by a lane (merge_insertions), and old entries [s0, s1) find their own shift by searching the
// slice's events (merge_heavy). A warp that walked them took a turn per 32 events, on one word of its
// chunk: update of 10^6 edits at one vertex of three neighbours, on 2^20 vertices, 101.8 ms; so 0.46
// (random pairs: 0.51).
static __device__ __forceinline__ void merge_insertions(int32_t* __restrict__ pool,
                                                        const unsigned long long* __restrict__ keys, int B,
                                                        const uint32_t* __restrict__ epos, const int32_t* __restrict__ E,
                                                        const MergeRow& r, int item) {
    const int k0 = r.b + item * HEAVY, k1 = min(r.d, k0 + HEAVY);
    int dlo = r.d, dhi = r.e;   // the deletions among these insertions' positions
    if (r.d < r.e) {
        dlo = warp_lb_event(epos, r.d, r.e, (int)(epos[k0] >> 1));
        dhi = warp_lb_event(epos, dlo, r.e, (int)(epos[k1 - 1] >> 1));
    }
    const int before = r.d < r.e ? E[r.d] : 0;
    for (int k = k0 + (int)lane_id(); k < k1; k += WARP) {
        const int pos = (int)(epos[k] >> 1);
        const int gone = r.d < r.e ? E[lb_event(epos, dlo, dhi, pos)] - before : 0;
        pool[r.dst + pos + (k - r.b) - gone] = key_v(keys[k], B);
    }
}

static __device__ __forceinline__ void merge_heavy(int32_t* __restrict__ pool, const uint32_t* __restrict__ epos,
                                                   const int32_t* __restrict__ E, const MergeRow& r, int s0, int s1) {
    constexpr int U = 4;
    const int l = (int)lane_id();
    const int ilo = warp_lb_event(epos, r.b, r.d, s0), ihi = warp_lb_event(epos, ilo, r.d, s1);
    const int dlo = warp_lb_event(epos, r.d, r.e, s0), dhi = warp_lb_event(epos, dlo, r.e, s1);
    const int before = r.d < r.e ? E[r.d] : 0;
    for (int b0 = s0; b0 < s1; b0 += U * WARP) {
        int32_t x[U];
        int to[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = b0 + u * WARP + l;
            x[u] = 0;
            to[u] = -1;
            if (i >= s1) continue;
            x[u] = pool[r.start + i];
            const int ins = lb_event(epos, ilo, ihi, i + 1) - r.b;   // insertions before it
            int gone = 0;
            bool keep = true;
            if (r.d < r.e) {
                const int j = lb_event(epos, dlo, dhi, i);
                gone = E[j] - before;
                // (deletions that cancel nothing may share its position)
                keep = j == dhi || (int)(epos[j] >> 1) != i || E[lb_event(epos, j, dhi, i + 1)] - before == gone;
            }
            if (keep) to[u] = i + ins - gone;
        }
        __syncwarp();   // a row compacted where it lies: these loads precede the stores below
#pragma unroll
        for (int u = 0; u < U; u++)
            if (to[u] >= 0) pool[r.dst + to[u]] = x[u];
        __syncwarp();   // ... and these stores the next loads
    }
}

// A whole row of at most 32 half-edits: a lane holds each event, no chunk is prepared.
static __device__ __forceinline__ void merge_mid(int32_t* __restrict__ pool, const unsigned long long* __restrict__ keys,
                                                 int B, const uint32_t* __restrict__ epos, const MergeRow& r) {
    constexpr int STEP = MERGE_U * WARP;
    const int l = (int)lane_id(), len = r.len;
    const unsigned lt = (1u << l) - 1, le = lt | (1u << l);
    const int32_t* O = pool + r.start + l;
    int32_t* N = pool + r.dst;
    int32_t x[MERGE_U];
#pragma unroll
    for (int u = 0; u < MERGE_U; u++) x[u] = u * WARP + l < len ? O[u * WARP] : 0;
    const uint32_t ev = r.b + l < r.e ? epos[r.b + l] : 0u;
    const int pos = (int)(ev >> 1);
    const bool ins = r.b + l < r.d, del = (ev & 1u) != 0;
    const int32_t y = ins ? key_v(keys[r.b + l], B) : 0;
    int shift = 0, gone = 0;
    for (int b0 = 0; b0 < len; b0 += STEP) {
        int32_t nx[MERGE_U];
        if (b0 + 2 * STEP <= len) {
#pragma unroll
            for (int u = 0; u < MERGE_U; u++) nx[u] = O[b0 + STEP + u * WARP];
        } else {
#pragma unroll
            for (int u = 0; u < MERGE_U; u++) nx[u] = b0 + STEP + u * WARP + l < len ? O[b0 + STEP + u * WARP] : 0;
        }
        __syncwarp();   // a row compacted where it lies: these loads precede the stores below
        int32_t* M = N + b0 + l;
        if (!__any_sync(0xffffffffu, (ins || del) && (unsigned)(pos - b0) < STEP)) {
            if (b0 + STEP <= len) {
#pragma unroll
                for (int u = 0; u < MERGE_U; u++) M[u * WARP + shift] = x[u];
            } else {
#pragma unroll
                for (int u = 0; u < MERGE_U; u++)
                    if (b0 + u * WARP + l < len) M[u * WARP + shift] = x[u];
            }
        } else {
#pragma unroll
            for (int u = 0; u < MERGE_U; u++) {
                const int at = pos - b0 - u * WARP;
                const bool here = (unsigned)at < WARP;
                const unsigned bit = 1u << (at & 31);
                const unsigned dm = __reduce_or_sync(0xffffffffu, del && here ? bit : 0u);
                const bool in = ins && here && pos < len;
                const unsigned mi = __ballot_sync(0xffffffffu, in);
                int to = shift - __popc(dm & lt);
                if (mi) {
                    const unsigned im = __reduce_or_sync(0xffffffffu, in ? bit : 0u);
                    if (__popc(im) == __popc(mi)) {
                        to += __popc(im & le);
                    } else {
                        for (unsigned q = mi; q; q &= q - 1) to += __shfl_sync(0xffffffffu, at, __ffs(q) - 1) <= l;
                    }
                    if (in) N[pos + l - gone - __popc(dm & (bit - 1))] = y;
                }
                if (b0 + u * WARP + l < len && !((dm >> l) & 1u)) M[u * WARP + to] = x[u];
                shift += __popc(mi) - __popc(dm);
                gone += __popc(dm);
            }
        }
#pragma unroll
        for (int u = 0; u < MERGE_U; u++) x[u] = nx[u];
    }
    if (ins && pos == len) N[len + l - gone] = y;   // past the last entry
}

// Short rows (at most SMALL_LEN entries and 32 half-edits): all events of a row fit one warp.
static __device__ __forceinline__ void merge_short(int32_t* __restrict__ pool, const unsigned long long* __restrict__ keys,
                                                   int B, const uint32_t* __restrict__ epos,
                                                   const MergeRow* __restrict__ mrow,
                                                   const int32_t* __restrict__ shorts, int i0, int cnt) {
    const int l = (int)lane_id();
    const unsigned lt = (1u << l) - 1, le = lt | (1u << l);
    MergeRow r{0, 0, 0, 0, 0, 0};
    if (l < cnt) r = mrow[shorts[i0 + l]];
    for (int j0 = 0; j0 < cnt; j0 += MERGE_ROWS) {
        long long st[MERGE_ROWS], ds[MERGE_ROWS];
        int len[MERGE_ROWS], pos[MERGE_ROWS];
        int32_t x0[MERGE_ROWS], x1[MERGE_ROWS], y[MERGE_ROWS];
        bool ins[MERGE_ROWS], del[MERGE_ROWS];
#pragma unroll
        for (int u = 0; u < MERGE_ROWS; u++) {   // the loads of MERGE_ROWS rows
            const int j = (j0 + u) & (WARP - 1);
            const bool have = j0 + u < cnt;
            st[u] = __shfl_sync(0xffffffffu, r.start, j);
            ds[u] = __shfl_sync(0xffffffffu, r.dst, j);
            len[u] = __shfl_sync(0xffffffffu, r.len, j);
            const int b = __shfl_sync(0xffffffffu, r.b, j);
            int p = __shfl_sync(0xffffffffu, r.d, j) - b;
            int ne = __shfl_sync(0xffffffffu, r.e, j) - b;
            if (!have) { len[u] = 0; p = 0; ne = 0; }
            const uint32_t e = l < ne ? epos[b + l] : 0u;
            pos[u] = (int)(e >> 1);
            del[u] = (e & 1u) != 0;   // matched deletions only
            ins[u] = l < p;
            y[u] = l < p ? key_v(keys[b + l], B) : 0;
            x0[u] = l < len[u] ? pool[st[u] + l] : 0;
            x1[u] = WARP + l < len[u] ? pool[st[u] + WARP + l] : 0;
        }
        __syncwarp();   // rows compacted where they lie: these loads precede the stores
#pragma unroll
        for (int u = 0; u < MERGE_ROWS; u++) {
            int32_t* N = pool + ds[u];
            const int32_t* O = pool + st[u];
            int32_t x = x0[u], xn = x1[u];
            int shift = 0, gone = 0;   // insertions minus cancelled entries, and cancelled entries, before the group
            for (int e0 = 0; e0 < len[u]; e0 += WARP) {
                int32_t xnn = 0;
                if (e0 + 2 * WARP < len[u]) xnn = e0 + 2 * WARP + l < len[u] ? O[e0 + 2 * WARP + l] : 0;
                const int at = pos[u] - e0;
                const bool here = (unsigned)at < WARP;
                const unsigned bit = 1u << (at & 31);
                const unsigned dm = __reduce_or_sync(0xffffffffu, del[u] && here ? bit : 0u);
                const bool in = ins[u] && here && pos[u] < len[u];
                const unsigned mi = __ballot_sync(0xffffffffu, in);
                int to = e0 + l + shift - __popc(dm & lt);
                if (mi) {
                    const unsigned im = __reduce_or_sync(0xffffffffu, in ? bit : 0u);
                    if (__popc(im) == __popc(mi)) {
                        to += __popc(im & le);
                    } else {
                        for (unsigned q = mi; q; q &= q - 1)
                            to += __shfl_sync(0xffffffffu, at, __ffs(q) - 1) <= l;
                    }
                    if (in) N[pos[u] + l - gone - __popc(dm & (bit - 1))] = y[u];
                }
                __syncwarp();
                if (e0 + l < len[u] && !((dm >> l) & 1u)) N[to] = x;
                shift += __popc(mi) - __popc(dm);
                gone += __popc(dm);
                x = xn;
                xn = xnn;
            }
            if (ins[u] && pos[u] == len[u]) N[pos[u] + l - gone] = y[u];   // past the last entry
        }
    }
}

// Short rows of one half-edit (most of a batch's rows): eight lanes each, four rows at a time, 32
// entries of each in flight. Every entry past the event moves by one place.
static __device__ __forceinline__ void merge_one(int32_t* __restrict__ pool, const unsigned long long* __restrict__ keys,
                                                 int B, const uint32_t* __restrict__ epos,
                                                 const MergeRow* __restrict__ mrow, int i0, int cnt) {
    const int l = (int)lane_id(), q = l & 7;
    MergeRow r{0, 0, 0, 0, 0, 0};
    auto load_row = [&](int j) { return j < cnt ? mrow[i0 + j] : MergeRow{0, 0, 0, 0, 0, 0}; };
    MergeRow nr = load_row(l >> 3);
    for (int j = l >> 3; j - (l >> 3) < cnt; j += 4) {
        r = nr;
        nr = load_row(j + 4);
        const bool ok = j < cnt;
        const int32_t* O = pool + r.start;
        int32_t* N = pool + r.dst;
        const uint32_t ev = ok ? epos[r.b] : 0u;
        const bool in = r.d > r.b, cut = (ev & 1u) != 0;   // an insertion, a matched deletion, or neither
        const int32_t y = in ? key_v(keys[r.b], B) : 0;
        const int at = (int)(ev >> 1);
        for (int b0 = 0; __any_sync(0xffffffffu, b0 < r.len); b0 += 32) {
            int32_t x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) x[u] = b0 + 8 * u + q < r.len ? O[b0 + 8 * u + q] : 0;
            __syncwarp();   // rows compacted where they lie: these loads precede the stores
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int e = b0 + 8 * u + q;
                if (e < r.len && !(cut && e == at)) N[e + (in && e >= at) - (cut && e > at)] = x[u];
            }
        }
        if (in && q == 0) N[at] = y;
    }
}

// The batch's rows, by every warp of the grid; `ev`: the warp's chunk events.
struct MergeList {
    const MergeRow* mrow;
    const int64_t* slices;
    int64_t slice_cap;
    const int32_t* shorts;
};
static __device__ __forceinline__ void merge_rows(int32_t* __restrict__ pool, const unsigned long long* __restrict__ keys,
                                                  int B, DevCounters* __restrict__ ctr, const uint32_t* __restrict__ epos,
                                                  const int32_t* __restrict__ E, const MergeList& m, ChunkEvents& ev) {
    const int over = ld_volatile(&ctr->overflow), sl = ld_volatile(&ctr->n_slices), none = ld_volatile(&ctr->n_one),
              nsh = ld_volatile(&ctr->n_short);
    if (over) return;   // the slice list did not fit (the host reports it)
    const int nsl = (int)min((int64_t)sl, m.slice_cap);
    // short rows of a warp's turn: up to 32, fewer while that leaves warps without any
    const int W = gwarp_count();
    const int per_s = min(WARP, max(MERGE_ROWS, (nsh + W - 1) / W)), per_o = min(WARP, max(MERGE_ROWS, (none + W - 1) / W));
    const int it_s = nsl + (nsh + per_s - 1) / per_s, items = it_s + (none + per_o - 1) / per_o;
    int it = gwarp_id();   // the first item of every warp; the rest are handed out
    while (it < items) {
        int nx = 0;
        if (lane_id() == 0) nx = W + atomicAdd(&ctr->merge_ticket, 1);
        if (it < nsl) {
            const int64_t item = m.slices[it];
            const MergeRow r = m.mrow[item >> 32];
            const int s = (int)(item & (HEAVY_ITEM - 1));
            const bool whole = r.dst == r.start;   // compacted where it lies: one warp, front to back
            if (r.e - r.b <= WARP && (whole || r.len <= SLICE)) {
                merge_mid(pool, keys, B, epos, r);
            } else if (item & INS_ITEM) {
                merge_insertions(pool, keys, B, epos, E, r, s);
            } else {
                const int s0 = whole ? 0 : s * SLICE, s1 = whole ? r.len : min(r.len, s0 + SLICE);
                if (item & HEAVY_ITEM) merge_heavy(pool, epos, E, r, s0, s1);
                else merge_slice(pool, keys, B, epos, E, r, s0, s1, ev);
            }
        } else if (it < it_s) {
            const int i0 = (it - nsl) * per_s;
            merge_short(pool, keys, B, epos, m.mrow, m.shorts, i0, min(per_s, nsh - i0));
        } else {
            const int i0 = (it - it_s) * per_o;
            merge_one(pool, keys, B, epos, m.mrow, i0, min(per_o, none - i0));
        }
        it = __shfl_sync(0xffffffffu, nx, 0);
    }
}

__global__ void __launch_bounds__(MERGE_THREADS, 4) k_merge(
        int32_t* __restrict__ pool, const unsigned long long* __restrict__ keys, int B, DevCounters* __restrict__ ctr,
        const uint32_t* __restrict__ epos, const int32_t* __restrict__ E, MergeList m) {
    __shared__ ChunkEvents s_ev[MERGE_WARPS];
    merge_rows(pool, keys, B, ctr, epos, E, m, s_ev[threadIdx.x / WARP]);
}

// ---- up to UPDATE_MAX edits: the whole update in one launch ------------------------------------
// A cooperative kernel, one block per SM, of the phases that larger batches launch one by one,
// with the bounded grid barrier between them: classification; the sort; the plan, a stretch of
// consecutive half-edits per block, its running counts added up from the blocks before; the
// rows' plan; the merge. The sort is one of two:
//   up to UPDATE_PAIRS half-edits   every key's place is the number of smaller keys: a warp per
//                                   key against all of them in shared memory
//   more                            sample sort: 2,048 or 4,096 keys are ranked that way and split
//                                   the others into buckets (10 to 64 keys on average), whose keys
//                                   are ranked among themselves. The sample takes one key of every
//                                   stretch at a hashed place: an edit's two half-edits lie side by
//                                   side, and an even stride would sample one orientation alone
//                                   (pairs written low id first, or all of one vertex, then fall into
//                                   few buckets). Keys equal to a splitter have a bucket of their
//                                   own and are not ranked, so a pair that is repeated costs nothing.
//
// What bounds it: the latency of two searches in rows, the barriers (6 to 9 of them) and the
// merge's traffic. Up to UPDATE_MAX edits it is faster than the launches it replaces (each about
// 4 us on the host, and the radix sort's passes wait on one another): whole call with them and
// so: 1,000 edits on 65,536 vertices 203 -> 180 us, 10,000 at scale 22 409 -> 363, 100,003 on
// 1.5 M vertices 466 -> 438. Beyond it a thread would hold more than two keys and the buckets'
// quadratic ranking overtakes the radix passes.
constexpr int UPDATE_THREADS = 1024;
constexpr int UPDATE_WARPS = UPDATE_THREADS / WARP;
constexpr int64_t UPDATE_MAX = 131072;
constexpr int UPDATE_PAIRS = 4096;
constexpr int UPDATE_SPLIT = 4096;   // splitters; half of them up to UPDATE_FEW half-edits
constexpr int UPDATE_FEW = 65536;
constexpr int UPDATE_ROWS = 16384;   // more affected rows are planned by blocks, fewer by warps
constexpr int UPDATE_BUCKETS = 2 * UPDATE_SPLIT + 1;   // between the splitters, and equal to each
// device scratch: splitters, the blocks' plan counts, bucket counts
constexpr int64_t UPDATE_SCRATCH = UPDATE_SPLIT * 8 + 1024 * 8 + (UPDATE_BUCKETS + 63) * 4;

constexpr int UPDATE_SMEM = (UPDATE_BUCKETS + 1) * 4 + 8;   // the buckets' first places and the end: 32 KB and 16 bytes
static_assert(UPDATE_SMEM % 16 == 0, "aligned");

// First index of the ascending a[0, n) whose value is above x.
template <typename T>
__device__ __forceinline__ int first_above(const T* a, int n, T x) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] <= x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// The half-edits p.raw[0, n) in ascending order into p.keys, all blocks; `smem`: UPDATE_SMEM. Returns
// false when a barrier failed. Ends before a barrier: the caller's next one publishes the order.
static __device__ bool update_sort(const UpdateParams& p, int n, unsigned long long SENT, unsigned char* smem) {
    const int t = threadIdx.x, l = (int)lane_id();
    const int G = (int)gridDim.x, wid = gwarp_id(), W = gwarp_count();
    const int tid = (int)blockIdx.x * UPDATE_THREADS + t, T = G * UPDATE_THREADS;
    unsigned long long* k = (unsigned long long*)smem;
    if (n <= UPDATE_PAIRS) {
        for (int i = t; i < n; i += UPDATE_THREADS) k[i] = ld_volatile(p.raw + i);
        __syncthreads();
        for (int j = wid; j < n; j += W) {
            const unsigned long long x = k[j];
            if (x == SENT) continue;   // past the half-edits; no one reads it
            int c = 0;
            for (int i = l; i < n; i += WARP) c += k[i] < x || (k[i] == x && i < j);
            c = __reduce_add_sync(0xffffffffu, c);
            if (l == 0) p.keys[c] = x;
        }
        return true;
    }
    const int S = n <= UPDATE_FEW ? UPDATE_SPLIT / 2 : UPDATE_SPLIT;   // 2,048 or 4,096
    // the sample, ranked like that
    for (int i = t; i < S; i += UPDATE_THREADS)
        k[i] = ld_volatile(p.raw + (long long)i * n / S + (((unsigned)i * 2654435761u) >> 16) % (unsigned)(n / S));
    __syncthreads();
    for (int j = wid; j < S; j += W) {
        const unsigned long long x = k[j];
        int c = 0;
        for (int i = l; i < S; i += WARP) c += k[i] < x || (k[i] == x && i < j);
        c = __reduce_add_sync(0xffffffffu, c);
        if (l == 0) p.split[c] = x;
    }
    if (!grid_sync(p.bar, 65)) return false;
    // every key's bucket and its place there (in the order the atomics came)
    for (int i = t; i < S; i += UPDATE_THREADS) k[i] = ld_volatile(p.split + i);
    __syncthreads();
    unsigned long long key[2] = {SENT, SENT};   // n <= 2 T
    int b[2] = {0, 0}, at[2] = {0, 0};
#pragma unroll
    for (int s = 0; s < 2; s++) {
        const int i = tid + s * T;
        if (i < n) key[s] = ld_volatile(p.raw + i);
        // bucket 2 q: between splitters q - 1 and q; 2 q + 1: equal to splitter q (to the first of equals)
        bool eq = false;
        if (key[s] != SENT) {
            int q = 0, hi = S;
            while (q < hi) {
                const int mid = (q + hi) >> 1;
                if (k[mid] < key[s]) q = mid + 1; else hi = mid;
            }
            eq = q < S && k[q] == key[s];
            b[s] = 2 * q + (eq ? 1 : 0);
        }
        // equal keys of a warp take their places by one atomic (a pair may be repeated all batch long)
        const unsigned em = __ballot_sync(0xffffffffu, eq);
        const int first = em ? __ffs(em) - 1 : 0;
        const int b1 = __shfl_sync(0xffffffffu, b[s], first);   // (every lane takes part)
        const bool same = eq && b[s] == b1;
        const unsigned sm = __ballot_sync(0xffffffffu, same);
        if (key[s] != SENT && (!same || l == first)) at[s] = atomicAdd(p.bucket + b[s], same ? __popc(sm) : 1);
        const int base = __shfl_sync(0xffffffffu, at[s], first);
        if (same) at[s] = base + __popc(sm & ((1u << l) - 1));
    }
    if (!grid_sync(p.bar, 66)) return false;
    int* off = (int*)smem;   // the buckets' first places, and the end
    {
        const int per = 2 * S / UPDATE_THREADS;   // 4 or 8 buckets per thread, and the last one
        const int4* mine = (const int4*)(p.bucket + per * t);   // (from L2: other blocks counted them)
        const int4 ca = __ldcg(mine), cb = per == 8 ? __ldcg(mine + 1) : make_int4(0, 0, 0, 0);
        const int c[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
        long long x = 0, y = 0, tx, ty;
#pragma unroll
        for (int q = 0; q < 8; q++) x += c[q];
        block_scan2(x, y, &tx, &ty);   // its barriers are past the splitters' last reader
#pragma unroll
        for (int q = 0; q < 8; q++) {
            if (q < per) off[per * t + q] = (int)x;
            x += c[q];
        }
        if (t == 0) {
            off[2 * S] = (int)tx;
            off[2 * S + 1] = (int)tx + ld_volatile(p.bucket + 2 * S);
        }
        __syncthreads();
    }
#pragma unroll
    for (int s = 0; s < 2; s++)
        if (key[s] != SENT) p.tmp[off[b[s]] + at[s]] = key[s];
    if (!grid_sync(p.bar, 67)) return false;
    const int total = off[2 * S + 1];
    for (int i = tid; i < total; i += T) {
        const unsigned long long x = ld_volatile(p.tmp + i);
        const int q = first_above(off, 2 * S + 2, i) - 1;   // the bucket of place i
        if (q & 1) {   // equal keys: in order as they lie
            p.keys[i] = x;
            continue;
        }
        const int q0 = off[q], q1 = off[q + 1];
        int c = 0;
        for (int j = q0; j < q1; j++) {
            const unsigned long long y = p.tmp[j];
            c += y < x || (y == x && j < i);
        }
        p.keys[q0 + c] = x;
    }
    return true;
}

static __device__ __forceinline__ void update_body(const UpdateParams& p) {
    __shared__ __align__(16) unsigned char s_mem[UPDATE_SMEM];   // the sort's, later the warps' chunk events
    static_assert(sizeof(s_mem) >= UPDATE_WARPS * sizeof(ChunkEvents) && sizeof(s_mem) >= UPDATE_SPLIT * 8 &&
                  sizeof(s_mem) >= UPDATE_PAIRS * 8, "fits");
    const int t = threadIdx.x, w = t / WARP, l = (int)lane_id();
    const int G = (int)gridDim.x, T = G * UPDATE_THREADS;
    const int B = p.B;
    DevCounters* ctr = p.rp.ctr;
    // classification; neighbouring edits on different SMs
    const unsigned long long SENT = (B + B + 1) >= 64 ? ~0ull : ((1ull << (B + B + 1)) - 1);
    if (2 * p.m > UPDATE_PAIRS)
        for (int i = (int)blockIdx.x * UPDATE_THREADS + t; i < UPDATE_BUCKETS; i += T) p.bucket[i] = 0;
    for (int i0 = t * G; i0 - l * G < p.m; i0 += T) {   // uniform per warp
        const int i = i0 + (int)blockIdx.x;
        int f = 0;
        if (i < p.m) {
            const int32_t u = p.e[i].u, v = p.e[i].v;
            f = classify_edit<true>(p.g, u, v, p.ops ? p.ops[i] : SCOUT_OP_TOGGLE);
            p.eflag[i] = (uint8_t)f;
            const bool half = (f & 5) == 5;
            const uint32_t op = f & 2 ? 0u : 1u;
            p.raw[2 * i] = half ? pack_key((uint32_t)u, op, (uint32_t)v, B) : SENT;
            p.raw[2 * i + 1] = half ? pack_key((uint32_t)v, op, (uint32_t)u, B) : SENT;
        }
        const unsigned mi = __ballot_sync(0xffffffffu, (f & 3) == 3), md = __ballot_sync(0xffffffffu, (f & 3) == 1);
        const unsigned ma = __ballot_sync(0xffffffffu, (f & 5) == 5);
        if (l == 0) {
            if (mi) atomicAdd(&ctr->n_ins, __popc(mi));
            if (md) atomicAdd(&ctr->n_del, __popc(md));
            if (ma) atomicAdd(&ctr->n_half, 2 * __popc(ma));
        }
    }
    if (!grid_sync(p.bar, 60)) return;
    if (!update_sort(p, 2 * p.m, SENT, s_mem)) return;
    if (!grid_sync(p.bar, 61)) return;
    // the plan: per block a stretch of whole 32-groups, at most 2,048 half-edits
    const int nh = ld_volatile(&ctr->n_half);
    const int groups = (nh + WARP - 1) / WARP;
    const int stretch = (groups + G - 1) / G * WARP;
    const int first = (int)blockIdx.x * stretch, end = min(nh, first + stretch);
    const int k0 = first + t;
    auto at = [&](int k) { return ld_volatile(p.keys + k); };
    unsigned long long key[2];
#pragma unroll
    for (int s = 0; s < 2; s++) key[s] = k0 + s * UPDATE_THREADS < end ? at(k0 + s * UPDATE_THREADS) : ~0ull;
    unsigned hm[2], mm[2];
    plan_search<2, UPDATE_THREADS, true>(p.g.row, p.g.pool, key, B, end, k0, at, p.epos, hm, mm);
    // counts of the warp's two groups: the first groups of all warps come before the second ones
    long long c0 = 0, c1 = 0, t0, t1;
    if (l == 0) {
        c0 = ((long long)__popc(hm[0]) << 32) | __popc(mm[0]);
        c1 = ((long long)__popc(hm[1]) << 32) | __popc(mm[1]);
    }
    block_scan2(c0, c1, &t0, &t1);
    if (t == 0) p.cnt[blockIdx.x] = (unsigned long long)(t0 + t1);
    if (!grid_sync(p.bar, 62)) return;
    __shared__ long long s_all, s_before;
    if (w == 0) {
        long long all = 0, before = 0;
        for (int j = l; j < G; j += WARP) {
            const long long c = (long long)ld_volatile(p.cnt + j);
            all += c;
            before += j < (int)blockIdx.x ? c : 0;
        }
        all = warp_incl_scan(all);
        before = warp_incl_scan(before);
        if (l == WARP - 1) { s_all = all; s_before = before; }
    }
    __syncthreads();
    const long long all = s_all, before = s_before;
#pragma unroll
    for (int s = 0; s < 2; s++) {   // lane 0's exclusive counts are those before the group
        const long long base = before + (s ? t0 : 0) + __shfl_sync(0xffffffffu, s ? c1 : c0, 0);
        const unsigned long long kk[1] = {key[s]};
        const unsigned h1[1] = {hm[s]}, m1[1] = {mm[s]};
        const int k = k0 + s * UPDATE_THREADS;
        plan_finish<1>(kk, B, k < end ? nh : 0, k, at, h1, m1, (unsigned long long)base, ctr, p.aff, p.seg_b, p.seg_d, p.E);
    }
    if (!p.rows) return;
    if (!grid_sync(p.bar, 63)) return;
    const int A = (int)(all >> 32);
    if (A > UPDATE_ROWS) row_plan<true>(p.rp, A, (int)blockIdx.x, G);
    else row_plan<false>(p.rp, A, gwarp_id(), gwarp_count());
    if (!grid_sync(p.bar, 64)) return;
    merge_rows(p.pool, p.keys, B, ctr, p.epos, p.E, MergeList{p.rp.mrow, p.rp.slices, p.rp.slice_cap, p.rp.shorts},
               ((ChunkEvents*)s_mem)[w]);
}

__global__ void __launch_bounds__(UPDATE_THREADS, 1) k_update(UpdateParams p) { update_body(p); }

// Several stores' updates side by side: grid row y runs the y-th (at most 2 keys per thread of its
// blocks: the callers' limit is far below).
__global__ void __launch_bounds__(UPDATE_THREADS, 1) k_update_side(const __grid_constant__ UpdateRound r) {
    update_body(r.p[blockIdx.y]);
}

int update_side(scout_ctx* c, const UpdateRound& r, int k) {
    void* args[] = {(void*)&r};
    SCOUT_CU(c, cudaLaunchCooperativeKernel((const void*)k_update_side, dim3((unsigned)(c->sm_count / k), (unsigned)k),
                                            dim3(UPDATE_THREADS), args, 0, c->s_main));
    c->nlaunch += 1;
    return SCOUT_OK;
}

// Long rows that only lose entries, compacted in place: one block per row streams it front to
// back in chunks of LIP_CHUNK entries, marking the chunk's cancelled entries from the row's
// sorted events; every entry of a chunk is loaded before any survivor of that chunk is stored,
// and a survivor's new position (survivors before it in the row) never exceeds its old one, so
// no store lands on an entry still to be read.
constexpr int LIP_THREADS = 256;
constexpr int LIP_U = 4;
constexpr int LIP_CHUNK = LIP_THREADS * LIP_U;
constexpr int LIP_TURNS = 2 * LIP_U;   // a chunk's own deletions take LIP_U + 1 turns at most, the rest are copies

__global__ void __launch_bounds__(LIP_THREADS) k_merge_long_inplace(int32_t* __restrict__ pool,
                                                                    const DevCounters* __restrict__ ctr,
                                                                    const uint32_t* __restrict__ epos,
                                                                    const int32_t* __restrict__ E,
                                                                    const int32_t* __restrict__ longs,
                                                                    const MergeRow* __restrict__ mrow) {
    __shared__ int s_warp[LIP_U][LIP_THREADS / WARP];
    __shared__ unsigned s_gone[LIP_CHUNK / WARP];
    __shared__ int s_next;
    const int t = threadIdx.x, w = t / WARP;
    const unsigned lt = (1u << lane_id()) - 1;
    const int nl = ctr->n_long;
    for (int li = blockIdx.x; li < nl; li += gridDim.x) {
        const MergeRow r = mrow[longs[li]];
        int32_t* O = pool + r.start;
        long long run = 0;
        int k = r.d;   // first event not below the chunk
        for (int b = 0; b < r.len; b += LIP_CHUNK) {
            const int lim = b > INT32_MAX - LIP_CHUNK ? INT32_MAX : b + LIP_CHUNK;
            if (t < LIP_CHUNK / WARP) s_gone[t] = 0;
            if (t == 0) s_next = r.e;
            __syncthreads();
            bool more = true;
            for (int turn = 0; more && turn < LIP_TURNS; turn++) {
                const int i = k + t;
                const uint32_t e = i < r.e ? epos[i] : 0u;
                const bool in = i < r.e && (int)(e >> 1) < lim;
                if (in && (e & 1u)) atomicOr(&s_gone[((e >> 1) - b) >> 5], 1u << (((e >> 1) - b) & 31));
                if (i < r.e && !in) atomicMin(&s_next, i);
                more = __syncthreads_and(in) != 0;
                if (more) k += LIP_THREADS;
            }
            if (more) {   // many copies of some pair: every entry searches the events that are left
                const int end = lb_event(epos, k, r.e, lim);
                for (int rel = t; rel < LIP_CHUNK && b + rel < r.len; rel += LIP_THREADS) {
                    const int j = lb_event(epos, k, end, b + rel), j1 = lb_event(epos, j, end, b + rel + 1);
                    if (E[j1] != E[j]) atomicOr(&s_gone[rel >> 5], 1u << (rel & 31));
                }
                if (t == 0) s_next = end;
                __syncthreads();
            }
            k = s_next;
            int32_t x[LIP_U];
            unsigned m[LIP_U];
#pragma unroll
            for (int u = 0; u < LIP_U; u++) {
                const int rel = u * LIP_THREADS + t;
                const long long i = (long long)b + rel;
                const bool keep = i < r.len && !((s_gone[rel >> 5] >> (rel & 31)) & 1u);
                x[u] = keep ? O[i] : -1;
                m[u] = __ballot_sync(0xffffffffu, keep);
                if (lane_id() == 0) s_warp[u][w] = __popc(m[u]);
            }
            __syncthreads();   // every load of the chunk is done; the warp counts are visible
            long long base = run;
#pragma unroll
            for (int u = 0; u < LIP_U; u++) {
                int before = 0, total = 0;
#pragma unroll
                for (int q = 0; q < LIP_THREADS / WARP; q++) {
                    const int cnt = s_warp[u][q];
                    before += q < w ? cnt : 0;
                    total += cnt;
                }
                if (x[u] >= 0) O[base + before + __popc(m[u] & lt)] = x[u];
                base += total;
            }
            run = base;
            __syncthreads();   // the counts are read before the next chunk overwrites them
        }
    }
}

// ---------------------------------------------------------------------------------------
// Compaction and download
// ---------------------------------------------------------------------------------------
__global__ void k_row_lens(const Row* __restrict__ row, int64_t n, int64_t* __restrict__ out) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        out[v] = row[v].len;
}

// Merge-path tiles: row r costs one unit and each of its entries one more, so row r starts
// at unit r + off[r] and entry e of row r sits at unit r + 1 + e. One block copies the
// entries of COPY_UNITS units: at most COPY_UNITS + 1 rows and COPY_UNITS entries, whatever
// mix of hubs, short rows and empty rows the range holds. The rows are found with a warp
// search and indexed in shared memory (output and source begin per row); every thread then
// copies COPY_UNITS / COPY_THREADS entries, finding each entry's row by a search of the
// index, with all its loads in flight before the stores.
constexpr int COPY_UNITS = 2048;
constexpr int COPY_THREADS = 256;

// first r in [0, n) with r + off[r] > x (n if none), 32 probes per step (all lanes call)
__device__ __forceinline__ long long warp_first_unit_above(const int64_t* off, long long n, long long x) {
    long long lo = 0, hi = n;
    while (hi - lo > WARP) {
        const long long step = (hi - lo + WARP - 1) / WARP;
        const long long pos = lo + (long long)lane_id() * step;
        const bool le = pos < hi && pos + off[pos] <= x;
        const int c = __popc(__ballot_sync(0xffffffffu, le));
        const long long nlo = c == 0 ? lo : lo + (long long)(c - 1) * step + 1;
        const long long nhi = c == 0 ? lo : min(hi, lo + (long long)c * step);
        lo = nlo;
        hi = max(nlo, nhi);
        if (c == 0) break;
    }
    const long long pos = lo + lane_id();
    const bool le = pos < hi && pos + off[pos] <= x;
    return lo + __popc(__ballot_sync(0xffffffffu, le));
}

__global__ void __launch_bounds__(COPY_THREADS) k_copy_rows(const Row* __restrict__ row, const int32_t* __restrict__ src,
                                                            int32_t* __restrict__ dst, const int64_t* __restrict__ off,
                                                            int32_t n, long long live) {
    __shared__ long long s_ra, s_rb;
    __shared__ int s_ob[COPY_UNITS + 2];
    __shared__ long long s_sb[COPY_UNITS + 2];
    const long long units = (long long)n + live;
    for (long long d0 = (long long)blockIdx.x * COPY_UNITS; d0 < units; d0 += (long long)gridDim.x * COPY_UNITS) {
        const long long d1 = min(units, d0 + COPY_UNITS);
        if (threadIdx.x < WARP) {
            const long long ra = warp_first_unit_above(off, n, d0) - 1;       // last row starting at or before d0
            const long long rb = warp_first_unit_above(off, n, d1 - 1) - 1;   // last row starting before d1
            if (threadIdx.x == 0) { s_ra = ra; s_rb = rb; }
        }
        __syncthreads();
        const long long ra = s_ra;
        const int nr = (int)(s_rb - ra + 1);
        const long long ef = max((long long)off[ra], d0 - ra - 1);            // first entry of the tile
        long long el = min((long long)off[s_rb + 1], d1 - s_rb - 1);          // one past the last
        if (el < ef) el = ef;
        for (int i = threadIdx.x; i < nr; i += COPY_THREADS) {
            const long long r = ra + i;
            const long long b = off[r];
            const long long eb = max(b, d0 - r - 1);
            s_ob[i] = (int)(min(eb, el) - ef);
            s_sb[i] = row[r].start + (eb - b);
        }
        __syncthreads();
        const int span = (int)(el - ef);
        constexpr int U = COPY_UNITS / COPY_THREADS;
        int32_t v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int rel = threadIdx.x + u * COPY_THREADS;
            v[u] = 0;
            if (rel < span) {
                int lo = 0, hi = nr - 1;   // last row whose output begin is <= rel
                while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (s_ob[mid] <= rel) lo = mid; else hi = mid - 1; }
                v[u] = src[s_sb[lo] + (rel - s_ob[lo])];
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int rel = threadIdx.x + u * COPY_THREADS;
            if (rel < span) dst[ef + rel] = v[u];
        }
        __syncthreads();
    }
}

__global__ void k_rows_compacted(Row* __restrict__ row, const int64_t* __restrict__ off, int32_t n) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        long long s = off[v];
        int len = row[v].len;
        row[v] = Row{s, len, len};
    }
}

// ---- tiered store ---------------------------------------------------------------------------
__device__ __forceinline__ int len_bin(int len) { return 31 - __clz(len + 1); }

__global__ void k_row_lens_hbm(const Row* __restrict__ row, int64_t n, long long cap, int64_t* __restrict__ out) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const Row r = row[v];
        out[v] = in_hbm(r, cap) ? r.len : 0;
    }
}

// HBM entries by floor(log2(1 + row length)) (32 bins), for the eviction threshold.
__global__ void k_hbm_hist(const Row* __restrict__ row, int64_t n, long long cap, unsigned long long* __restrict__ hist) {
    __shared__ unsigned long long sh[32];
    if (threadIdx.x < 32) sh[threadIdx.x] = 0;
    __syncthreads();
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const Row r = row[v];
        if (in_hbm(r, cap) && r.len > 0) atomicAdd(&sh[len_bin(r.len)], (unsigned long long)r.len);
    }
    __syncthreads();
    if (threadIdx.x < 32 && sh[threadIdx.x]) atomicAdd(&hist[threadIdx.x], sh[threadIdx.x]);
}

__global__ void k_row_lens_evict(const Row* __restrict__ row, int64_t n, long long cap, int bins,
                                 int64_t* __restrict__ out) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const Row r = row[v];
        out[v] = (in_hbm(r, cap) && r.len > 0 && len_bin(r.len) < bins) ? r.len : 0;
    }
}

__global__ void k_rows_evicted(Row* __restrict__ row, const int64_t* __restrict__ off, int64_t n, long long cap,
                               int bins, long long host_base) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const Row r = row[v];
        if (in_hbm(r, cap) && r.len > 0 && len_bin(r.len) < bins) row[v] = Row{host_base + off[v], r.len, r.len};
    }
}

// ---- host pool compaction ---------------------------------------------------------------------
// The host rows are put into HOST_BUCKETS buckets by address (entry >> sh), their lengths and
// numbers counted per bucket; a row's new place is its bucket's first one plus the room that
// rows of the bucket took before it (any order inside a bucket will do).
constexpr int HOST_BUCKETS = 4096;

__global__ void k_host_count(const Row* __restrict__ row, int64_t n, long long cap, long long rel, int sh,
                             unsigned long long* __restrict__ len, unsigned long long* __restrict__ cnt) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const Row r = row[v];
        if (in_hbm(r, cap) || r.len <= 0) continue;
        const long long b = (r.start - rel) >> sh;
        atomicAdd(&len[b], (unsigned long long)r.len);
        atomicAdd(&cnt[b], 1ull);
    }
}

// len and cnt hold the buckets' next free places now.
__global__ void k_host_place(const Row* __restrict__ row, int64_t n, long long cap, long long rel, int sh,
                             unsigned long long* __restrict__ len, unsigned long long* __restrict__ cnt,
                             int32_t* __restrict__ list, long long* __restrict__ to) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const Row r = row[v];
        if (in_hbm(r, cap) || r.len <= 0) continue;
        const long long b = (r.start - rel) >> sh;
        list[atomicAdd(&cnt[b], 1ull)] = (int32_t)v;
        to[v] = (long long)atomicAdd(&len[b], (unsigned long long)r.len);
    }
}

// Rows list[i0, i1) into the staging buffer (which starts at new place `base`), a warp per row, and
// their descriptors to where the buffer is copied next.
__global__ void __launch_bounds__(256) k_host_stage(Row* __restrict__ row, const int32_t* __restrict__ pool,
                                                    const int32_t* __restrict__ list, int i0, int i1,
                                                    const long long* __restrict__ to, long long base, long long rel,
                                                    int32_t* __restrict__ stage) {
    constexpr int U = 8;   // loads in flight per lane (they cross the host link)
    for (int k = i0 + gwarp_id(); k < i1; k += gwarp_count()) {
        const int32_t v = list[k];
        const Row r = row[v];
        const int32_t* s = pool + r.start;
        int32_t* d = stage + (to[v] - base);
        for (int j0 = 0; j0 < r.len; j0 += U * WARP) {
            int32_t x[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int j = j0 + u * WARP + (int)lane_id();
                x[u] = j < r.len ? s[j] : 0;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int j = j0 + u * WARP + (int)lane_id();
                if (j < r.len) d[j] = x[u];
            }
        }
        __syncwarp();
        if (lane_id() == 0) row[v] = Row{rel + to[v], r.len, r.len};
    }
}

// After the HBM rows were copied to the new pool: HBM rows point at their copies, host rows
// keep their address (their offset is re-based on the new pool).
__global__ void k_rows_compacted_tiered(Row* __restrict__ row, const int64_t* __restrict__ off, int32_t n,
                                        long long cap, long long rebase) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const Row r = row[v];
        if (in_hbm(r, cap)) row[v] = Row{(long long)off[v], r.len, r.len};
        else row[v] = Row{r.start + rebase, r.len, r.cap};
    }
}

// ---------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------
static int key_bits_for(int64_t n) {
    int B = 1;
    while ((1ll << B) < n + 1) B++;
    return B;
}

static inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

int ws_ensure(scout_ctx* c, int64_t m) {
    int64_t M = std::max<int64_t>(m, 1024);
    if (c->ws && c->ws_m >= M) return SCOUT_OK;
    M = M + M / 2;
    const int64_t H = 2 * M;
    size_t sz[] = {
        (size_t)M * sizeof(scout_edge), (size_t)M, (size_t)M,
        (size_t)H * 8, (size_t)H * 8, (size_t)(H + 1) * 8,
        (size_t)H * 4, (size_t)(H + 1) * 4, (size_t)H * 4, (size_t)H * 4, (size_t)H * 4, (size_t)H * sizeof(MergeRow)};
    size_t total = 0;
    for (size_t s : sz) total += align256(s);
    if (c->ws) dev_free(c, c->ws, (size_t)c->ws_bytes);
    c->ws = nullptr;
    c->ws_m = 0;
    SCOUT_RC(dev_alloc(c, &c->ws, total, "batch workspace"));
    c->ws_bytes = (int64_t)total;
    c->ws_m = M;
    char* p = (char*)c->ws;
    auto take = [&](size_t s) { char* q = p; p += align256(s); return (void*)q; };
    c->d_edits = (scout_edge*)take(sz[0]);
    c->d_ops = (uint8_t*)take(sz[1]);
    c->d_eflag = (uint8_t*)take(sz[2]);
    c->d_keys = (unsigned long long*)take(sz[3]);
    c->d_keys_alt = (unsigned long long*)take(sz[4]);
    c->d_mdp = (long long*)take(sz[5]);
    c->d_aff = (int32_t*)take(sz[6]);
    c->d_seg_b = (int32_t*)take(sz[7]);
    c->d_seg_d = (int32_t*)take(sz[8]);
    c->d_longs = (int32_t*)take(sz[9]);
    c->d_shorts = (int32_t*)take(sz[10]);
    c->d_mrow = (MergeRow*)take(sz[11]);
    c->d_hkeys = c->d_keys;
    return SCOUT_OK;
}

// Merge items of a batch of m edits: the long rows' ceil(len / SLICE) sum to at most nnz / SLICE +
// Amax, the heavy rows' ceil(insertions / HEAVY) to at most twice their half-edits / HEAVY.
static int64_t slices_for(int64_t nnz, int64_t m, int64_t Amax) { return nnz / SLICE + Amax + 4 * m / HEAVY + 1024; }

static int update_ensure(scout_ctx* c) {   // scratch of the one-launch update
    if (c->d_update) return SCOUT_OK;
    return dev_alloc(c, &c->d_update, (size_t)UPDATE_SCRATCH, "update scratch");
}

int graph_reserve_batch(scout_ctx* c, int64_t m) {
    SCOUT_RC(lists_ensure(c));
    SCOUT_RC(ws_ensure(c, m));
    SCOUT_RC(update_ensure(c));
    const int64_t Amax = std::min<int64_t>(2 * m, c->n);
    SCOUT_RC(dev_grow(c, &c->d_slices, &c->cap_slices, slices_for(c->pool_cap, m, Amax), "merge slices"));
    SCOUT_RC(sort_reserve(c, std::max<int64_t>(2 * c->ws_m, c->n + 1)));
    if (!c->d_coff) SCOUT_RC(dev_alloc(c, (void**)&c->d_coff, (size_t)(c->n + 1) * sizeof(int64_t), "compaction offsets"));
    // the compaction target, when the budget leaves room for a second pool
    if (!c->spare && c->held + (uint64_t)c->pool_cap * 4 <= c->budget / 100 * 85) {
        SCOUT_RC(dev_alloc(c, (void**)&c->spare, (size_t)c->pool_cap * 4, "element pool"));
        c->spare_cap = c->pool_cap;
    }
    SCOUT_RC(pin_grow(c, &c->h_pin_edits, &c->cap_pin_edits, m * (int64_t)sizeof(scout_edge) + m + 1));
    return SCOUT_OK;
}

int lists_ensure(scout_ctx* c) {
    SCOUT_RC(graph_ensure_scratch(c));
    if (c->d_list[0]) return SCOUT_OK;
    // Queue items are (chunk << 32 | vertex); a vertex pushed once per round occupies at most
    // ceil(len / chunk) items with chunk >= 256 entries, so n + nnz / 256 + slack bounds a round.
    c->qcap = c->n + (c->pool_cap / 256) + 4096;
    for (int i = 0; i < 3; i++) SCOUT_RC(dev_alloc(c, &c->d_qbuf[i], (size_t)c->qcap * 8, "work queues"));
    for (int i = 0; i < 2; i++) SCOUT_RC(dev_alloc(c, (void**)&c->d_list[i], (size_t)c->n * 4, "vertex lists"));
    SCOUT_RC(dev_alloc(c, (void**)&c->d_commit, (size_t)c->n * 8, "commit pairs"));
    return SCOUT_OK;
}

int batch_begin(scout_ctx* c) {
    SCOUT_RC(gather_finish(c, nullptr, nullptr, nullptr));   // no graph work while a gather runs
    SCOUT_CU(c, cudaMemsetAsync(c->d_batch, 0, offsetof(DevBatch, pairs), c->s_main));
    c->bar_used = false;
    c->pairs_ready = false;
    c->last_changed = 0;   // counted again when the batch has run; until then there is nothing to commit
    return SCOUT_OK;
}

int counters_fetch(scout_ctx* c) {
    c->fetched = false;
    SCOUT_CU(c, cudaMemcpyAsync(c->h_batch, c->d_batch, sizeof(DevBatch), cudaMemcpyDeviceToHost, c->s_main));
    SCOUT_CU(c, cudaStreamSynchronize(c->s_main));
    c->fetched = true;
    for (const GridBar& b : c->h_batch->bar)
        if (b.err & 1)
            return c->fail(SCOUT_E_TIMEOUT, "a device grid barrier timed out (tag " + std::to_string(b.where) + ")");
    if (c->h_ctr->pad)
        return c->fail(SCOUT_E_STATE, "the component labels do not describe the components of the graph "
                                      "(an edge joins two labels); upload a consistent labelling");
    if (c->h_ctr->sort_err == 1) return c->fail(SCOUT_E_TIMEOUT, "a sort look-back wait timed out");
    if (c->h_ctr->sort_err == 4) return c->fail(SCOUT_E_TIMEOUT, "a scan or merge-plan look-back wait timed out");
    if (c->h_ctr->sort_err) return c->fail(SCOUT_E_STATE, "the sort computed a position out of range");
    if (c->h_batch->bar[0].err != 0 || c->h_batch->bar[1].err != 0 || c->h_ctr->overflow)
        return c->fail(SCOUT_E_CAPACITY, "a device work list overflowed its capacity");
    c->pairs_ready = c->h_ctr->pairs_ok && c->h_ctr->changed <= COMMIT_PAIRS;
    return SCOUT_OK;
}

int graph_ensure_scratch(scout_ctx* c) {
    if (c->stamp_a) return SCOUT_OK;
    size_t bytes = (size_t)c->n * sizeof(int32_t);
    int32_t** arrs[] = {&c->stamp_a, &c->stamp_b, &c->stamp_c, &c->stamp_d, &c->aux_v};
    for (auto a : arrs) {
        SCOUT_RC(dev_alloc(c, (void**)a, bytes, "per-vertex scratch"));
        SCOUT_CU(c, cudaMemsetAsync(*a, 0, bytes, c->s_main));
    }
    return SCOUT_OK;
}

// Rewrites the pool so rows are contiguous and leaves at least min_free free elements
// (the on-device half of compact_flash_graph). With nnz_exact the host's live count is used
// and nothing waits for the device; otherwise (after staging) the live count is read back.
static inline long long elem_delta(const int32_t* a, const int32_t* b) {
    return (long long)(((intptr_t)a - (intptr_t)b) / (intptr_t)sizeof(int32_t));
}

// Host pool compaction (tiered store) by the host: the host rows are moved down in order of
// their position (memmove, every destination at or below its source), and the row table is
// rewritten. Only for stores whose host pool has a bucket longer than the staging buffer.
static int host_compact_serial(scout_ctx* c) {
    const int64_t n = c->n;
    SCOUT_CU(c, cudaStreamSynchronize(c->s_main));
    std::vector<Row> rows((size_t)n);
    SCOUT_CU(c, cudaMemcpy(rows.data(), c->row, (size_t)n * sizeof(Row), cudaMemcpyDeviceToHost));
    const long long rel = elem_delta(c->host_pool, c->pool);
    std::vector<int32_t> ids;
    for (int64_t v = 0; v < n; v++) {
        const Row& r = rows[v];
        if (!(r.start >= 0 && r.start < c->pool_cap) && r.len > 0) ids.push_back((int32_t)v);
    }
    std::sort(ids.begin(), ids.end(), [&](int32_t a, int32_t b) { return rows[a].start < rows[b].start; });
    int64_t pos = 0;
    for (int32_t v : ids) {
        Row& r = rows[v];
        const int64_t from = r.start - rel;
        if (from != pos) std::memmove(c->host_pool + pos, c->host_pool + from, (size_t)r.len * 4);
        r.start = rel + pos;
        r.cap = r.len;
        pos += r.len;
    }
    SCOUT_CU(c, cudaMemcpy(c->row, rows.data(), (size_t)n * sizeof(Row), cudaMemcpyHostToDevice));
    c->host_tail = pos;
    return SCOUT_OK;
}

// Host pool compaction (tiered store) by the device, through a staging buffer in HBM (the repair's
// work queues, free outside a repair): address buckets in order, as many at a time as fit the
// buffer, are gathered into it over the host link and copied back to their new place in one
// piece. Rows are disjoint, so the new place of a group of buckets ends at or before the first
// row of any later bucket: nothing is overwritten before it was read.
// What bounds it: the host link, the live rows crossing it twice. About 5 ms for 24 M live entries at
// scale 20 against 68 ms for the host's sort and memmove; a stream of 20,000-edit batches,
// which waited on it every fourth batch or so, 18.8 -> 4.5 ms per batch.
static int host_compact(scout_ctx* c) {
    const int64_t n = c->n;
    SCOUT_RC(lists_ensure(c));
    const long long rel = elem_delta(c->host_pool, c->pool);
    int sh = 0;
    while (((c->host_tail + 1) >> sh) >= HOST_BUCKETS) sh++;
    int32_t* stage = (int32_t*)c->d_qbuf[0];
    const int64_t stage_cap = 2 * c->qcap;
    long long* to = (long long*)c->d_qbuf[1];
    int64_t* len = (int64_t*)c->d_qbuf[2];   // qcap >= 4096 + n items: two arrays of HOST_BUCKETS + 1 fit
    int64_t* cnt = len + HOST_BUCKETS + 1;
    if (2 * (HOST_BUCKETS + 1) > c->qcap) return host_compact_serial(c);
    const int nb = blocks_for(n, 256);
    SCOUT_CU(c, cudaMemsetAsync(len, 0, 2 * (HOST_BUCKETS + 1) * 8, c->s_main));
    k_host_count<<<nb, 256, 0, c->s_main>>>(c->row, n, (long long)c->pool_cap, rel, sh, (unsigned long long*)len,
                                            (unsigned long long*)cnt);
    SCOUT_LAUNCH(c, "k_host_count");
    SCOUT_RC(scan_i64(c, len, HOST_BUCKETS + 1, nullptr));
    SCOUT_RC(scan_i64(c, cnt, HOST_BUCKETS + 1, nullptr));
    std::vector<int64_t> first(2 * (HOST_BUCKETS + 1));   // the buckets' first places, then their first rows
    SCOUT_CU(c, cudaMemcpyAsync(first.data(), len, first.size() * 8, cudaMemcpyDeviceToHost, c->s_main));
    SCOUT_CU(c, cudaStreamSynchronize(c->s_main));
    const int64_t* rows = first.data() + HOST_BUCKETS + 1;
    for (int b = 0; b < HOST_BUCKETS; b++)
        if (first[b + 1] - first[b] > stage_cap) return host_compact_serial(c);
    k_host_place<<<nb, 256, 0, c->s_main>>>(c->row, n, (long long)c->pool_cap, rel, sh, (unsigned long long*)len,
                                            (unsigned long long*)cnt, c->d_list[1], to);
    SCOUT_LAUNCH(c, "k_host_place");
    c->nlaunch += 2;
    for (int b = 0; b < HOST_BUCKETS;) {
        int e = b + 1;
        while (e < HOST_BUCKETS && first[e + 1] - first[b] <= stage_cap) e++;
        const int64_t cntr = rows[e] - rows[b], ne = first[e] - first[b];
        if (cntr > 0) {
            k_host_stage<<<blocks_for(cntr * WARP, 256, 8 * c->sm_count), 256, 0, c->s_main>>>(
                c->row, c->pool, c->d_list[1], (int)rows[b], (int)rows[e], to, first[b], rel, stage);
            SCOUT_LAUNCH(c, "k_host_stage");
            c->nlaunch += 1;
            SCOUT_CU(c, cudaMemcpyAsync(c->host_pool + first[b], stage, (size_t)ne * 4, cudaMemcpyDeviceToHost, c->s_main));
        }
        b = e;
    }
    c->host_tail = first[HOST_BUCKETS];
    return SCOUT_OK;
}

// Tiered compaction: only HBM rows move. When they and min_free do not fit the HBM pool, the
// shortest ones (whole log2 length classes, shortest first) are evicted to the host pool.
static int graph_compact_tiered(scout_ctx* c, int64_t min_free) {
    const int64_t n = c->n;
    if (!c->d_coff) SCOUT_RC(dev_alloc(c, (void**)&c->d_coff, (size_t)(n + 1) * sizeof(int64_t), "compaction offsets"));
    int64_t* off = c->d_coff;
    const int nb = blocks_for(n, 256);
    auto hbm_live = [&](int64_t* live) -> int {
        k_row_lens_hbm<<<nb, 256, 0, c->s_main>>>(c->row, n, (long long)c->pool_cap, off);
        SCOUT_LAUNCH(c, "k_row_lens_hbm");
        SCOUT_RC(scan_i64(c, off, n, off + n));
        SCOUT_CU(c, cudaMemcpyAsync(live, off + n, 8, cudaMemcpyDeviceToHost, c->s_main));
        SCOUT_CU(c, cudaStreamSynchronize(c->s_main));
        return SCOUT_OK;
    };
    int64_t live = 0;
    SCOUT_RC(hbm_live(&live));
    if (live + min_free > c->pool_cap) {
        // 32 histogram slots in the scan partials (free between scans)
        SCOUT_RC(dev_grow(c, &c->d_scan_tmp, &c->cap_scan, 64, "scan partials"));
        unsigned long long* hist = (unsigned long long*)c->d_scan_tmp;
        SCOUT_CU(c, cudaMemsetAsync(hist, 0, 32 * 8, c->s_main));
        k_hbm_hist<<<nb, 256, 0, c->s_main>>>(c->row, n, (long long)c->pool_cap, hist);
        SCOUT_LAUNCH(c, "k_hbm_hist");
        unsigned long long h[32];
        SCOUT_CU(c, cudaMemcpyAsync(h, hist, sizeof(h), cudaMemcpyDeviceToHost, c->s_main));
        SCOUT_CU(c, cudaStreamSynchronize(c->s_main));
        int bins = 0;
        int64_t keep = live;
        while (bins < 32 && keep + min_free > c->pool_cap) keep -= (int64_t)h[bins++];
        if (keep + min_free > c->pool_cap)
            return c->fail(SCOUT_E_CAPACITY, "tiered store: the HBM pool cannot hold the rows of one batch");
        k_row_lens_evict<<<nb, 256, 0, c->s_main>>>(c->row, n, (long long)c->pool_cap, bins, off);
        SCOUT_LAUNCH(c, "k_row_lens_evict");
        SCOUT_RC(scan_i64(c, off, n, off + n));
        int64_t ev = 0;
        SCOUT_CU(c, cudaMemcpyAsync(&ev, off + n, 8, cudaMemcpyDeviceToHost, c->s_main));
        SCOUT_CU(c, cudaStreamSynchronize(c->s_main));
        if (c->host_tail + ev > c->host_cap) {   // the HBM rows and their offsets stay as they are
            SCOUT_RC(host_compact(c));
            if (c->host_tail + ev > c->host_cap) return c->fail(SCOUT_E_CAPACITY, "tiered store: the host pool is full");
        }
        const int64_t tiles = (n + ev + COPY_UNITS - 1) / COPY_UNITS;
        k_copy_rows<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(tiles, 32 * c->sm_count)), COPY_THREADS, 0,
                      c->s_main>>>(c->row, c->pool, c->host_pool + c->host_tail, off, (int32_t)n, (long long)ev);
        k_rows_evicted<<<nb, 256, 0, c->s_main>>>(c->row, off, n, (long long)c->pool_cap, bins,
                                                  elem_delta(c->host_pool, c->pool) + c->host_tail);
        SCOUT_LAUNCH(c, "eviction");
        c->host_tail += ev;
        c->evictions++;
        c->evicted_entries += ev;
        c->nlaunch += 8;
        SCOUT_RC(hbm_live(&live));
    }
    int64_t cap = c->pool_cap;
    int32_t* np = nullptr;
    if (c->spare && c->spare_cap >= cap) {
        np = c->spare;
        cap = c->spare_cap;
        c->spare = nullptr;
        c->spare_cap = 0;
    } else {
        if (c->spare) { dev_free(c, c->spare, (size_t)c->spare_cap * 4); c->spare = nullptr; c->spare_cap = 0; }
        SCOUT_RC(dev_alloc(c, (void**)&np, (size_t)cap * sizeof(int32_t), "element pool"));
    }
    const int64_t tiles = (n + live + COPY_UNITS - 1) / COPY_UNITS;
    k_copy_rows<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(tiles, 32 * c->sm_count)), COPY_THREADS, 0,
                  c->s_main>>>(c->row, c->pool, np, off, (int32_t)n, (long long)live);
    k_rows_compacted_tiered<<<nb, 256, 0, c->s_main>>>(c->row, off, (int32_t)n, (long long)c->pool_cap,
                                                       elem_delta(c->pool, np));
    SCOUT_LAUNCH(c, "tiered compaction");
    c->nlaunch += 6;
    if (c->held <= c->budget / 100 * 85) {
        c->spare = c->pool;
        c->spare_cap = c->pool_cap;
    } else {
        dev_free(c, c->pool, (size_t)c->pool_cap * sizeof(int32_t));
    }
    c->compactions++;
    c->pool = np;
    c->pool_cap = cap;
    c->tail = live;
    return SCOUT_OK;
}

int graph_compact(scout_ctx* c, int64_t min_free, bool nnz_exact) {
    if (c->tiered) return graph_compact_tiered(c, min_free);
    const int64_t n = c->n;
    if (!c->d_coff) SCOUT_RC(dev_alloc(c, (void**)&c->d_coff, (size_t)(n + 1) * sizeof(int64_t), "compaction offsets"));
    int64_t* off = c->d_coff;
    int nb = blocks_for(n, 256);
    k_row_lens<<<nb, 256, 0, c->s_main>>>(c->row, n, off);
    SCOUT_LAUNCH(c, "k_row_lens");
    SCOUT_RC(scan_i64(c, off, n, off + n));
    int64_t live = c->nnz;
    if (!nnz_exact) {
        SCOUT_CU(c, cudaMemcpyAsync(&live, off + n, sizeof(int64_t), cudaMemcpyDeviceToHost, c->s_main));
        SCOUT_CU(c, cudaStreamSynchronize(c->s_main));
    }
    int64_t cap = std::max<int64_t>(c->pool_cap, live + min_free);
    // Ping-pong: the previous pool is kept as the next compaction's target, so steady-state
    // compactions allocate nothing. Without budget room for two pools the old one is freed.
    int32_t* np = nullptr;
    if (c->spare && c->spare_cap >= cap) {
        np = c->spare;
        cap = c->spare_cap;
        c->spare = nullptr;
        c->spare_cap = 0;
    } else {
        if (c->spare) { dev_free(c, c->spare, (size_t)c->spare_cap * 4); c->spare = nullptr; c->spare_cap = 0; }
        SCOUT_RC(dev_alloc(c, (void**)&np, (size_t)cap * sizeof(int32_t), "element pool"));
    }
    const int64_t tiles = (n + live + COPY_UNITS - 1) / COPY_UNITS;
    k_copy_rows<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(tiles, 32 * c->sm_count)), COPY_THREADS, 0,
                  c->s_main>>>(c->row, c->pool, np, off, (int32_t)n, (long long)live);
    k_rows_compacted<<<nb, 256, 0, c->s_main>>>(c->row, off, (int32_t)n);
    SCOUT_LAUNCH(c, "compaction");
    c->nlaunch += 6;
    if (c->held <= c->budget / 100 * 85) {   // keep the old pool as the next target
        c->spare = c->pool;
        c->spare_cap = c->pool_cap;
    } else {
        dev_free(c, c->pool, (size_t)c->pool_cap * sizeof(int32_t));
    }
    c->compactions++;
    c->pool = np;
    c->pool_cap = cap;
    c->tail = live;
    c->nnz = live;
    return SCOUT_OK;
}

static bool is_pinned(const void* p) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeHost;
}

// Host memcpy into the pinned staging buffer, shared by a few host threads from 256 KB on (one
// thread moves about 15 GB/s: an 800 KB batch reached the device in 67 us, with up to eight
// threads in 36).
void stage_copy(void* dst, const void* src, size_t bytes) {
    constexpr size_t PART = (size_t)1 << 17;
    if (bytes < 2 * PART) {
        std::memcpy(dst, src, bytes);
        return;
    }
    const int64_t parts = (int64_t)((bytes + PART - 1) / PART);
    const int threads = (int)std::min<int64_t>(std::min<int64_t>(parts, 8), std::max(1, omp_get_max_threads()));
#pragma omp parallel for schedule(static) num_threads(threads)
    for (int64_t i = 0; i < parts; i++) {
        size_t o = (size_t)i * PART;
        std::memcpy((char*)dst + o, (const char*)src + o, std::min(PART, bytes - o));
    }
}

// Edits in pinned host memory are copied to the device directly; pageable ones go through the
// context's pinned staging buffer.
// Edits hinted by scout_prefetch and declared by this call are already on their way to the
// device (copy stream, ev_pf): the main stream waits for that copy and reads them there.
static int upload_edits(scout_ctx* c, const scout_edge* edits, const uint8_t* ops, int64_t m,
                        const scout_edge** d_src) {
    const bool hinted = c->pf_use && c->pf_ready && c->pf_ready_m == m && !ops;
    c->pf_use = false;
    if (c->pf_ready) c->pf_ready = false;   // consumed now, or stale (the next hint replaces it)
    if (hinted) {
        SCOUT_CU(c, cudaStreamWaitEvent(c->s_main, c->ev_pf, 0));
        *d_src = c->d_pf_edits[c->pf_slot];
        return SCOUT_OK;
    }
    *d_src = c->d_edits;
    const size_t eb = (size_t)m * sizeof(scout_edge);
    const bool pe = is_pinned(edits), po = !ops || is_pinned(ops);
    if (!pe || !po) {
        int64_t bytes = (int64_t)((pe ? 0 : eb) + (po ? 0 : (size_t)m));
        SCOUT_RC(pin_grow(c, &c->h_pin_edits, &c->cap_pin_edits, std::max<int64_t>(bytes, 1)));
    }
    const void* se = edits;
    if (!pe) {
        stage_copy(c->h_pin_edits, edits, eb);
        se = c->h_pin_edits;
    }
    SCOUT_CU(c, cudaMemcpyAsync(c->d_edits, se, eb, cudaMemcpyHostToDevice, c->s_main));
    if (ops) {
        const void* so = ops;
        if (!po) {
            char* dst = (char*)c->h_pin_edits + (pe ? 0 : eb);
            stage_copy(dst, ops, (size_t)m);
            so = dst;
        }
        SCOUT_CU(c, cudaMemcpyAsync(c->d_ops, so, (size_t)m, cudaMemcpyHostToDevice, c->s_main));
    }
    return SCOUT_OK;
}

int graph_update(scout_ctx* c, const scout_edge* edits, const uint8_t* ops, int64_t m, scout_batch_stats* st,
                 UpdateParams* later) {
    const int64_t n = c->n;
    const int B = key_bits_for(n);
    c->key_bits = B;
    // Free space must hold a rewrite of every live entry plus two entries per edit (tiered
    // store: the batch's exact growth is checked after the row allocation instead).
    int64_t need = c->tiered ? 2 * m + 1024 : c->nnz + 2 * m + 1024;
    SCOUT_CU(c, cudaEventRecord(c->ev_t[6], c->s_main));
    if (c->pool_cap - c->tail < need) SCOUT_RC(graph_compact(c, need, true));
    SCOUT_CU(c, cudaEventRecord(c->ev_t[7], c->s_main));
    SCOUT_RC(ws_ensure(c, m));
    SCOUT_RC(graph_ensure_scratch(c));
    if (st) st->h2d_bytes += m * (int64_t)sizeof(scout_edge) + (ops ? m : 0);
    c->merge_tail = c->tail;
    if (m == 0) {
        c->d_hkeys = c->d_keys;
        SCOUT_CU(c, cudaEventRecord(c->ev_t[3], c->s_main));
        return SCOUT_OK;
    }
    const scout_edge* d_src = nullptr;
    SCOUT_RC(upload_edits(c, edits, ops, m, &d_src));
    SCOUT_CU(c, cudaEventRecord(c->ev_t[3], c->s_main));
    DGraph g = dgraph(c);
    const int64_t H = 2 * m;
    const int64_t Amax = std::min<int64_t>(H, n);
    SCOUT_RC(dev_grow(c, &c->d_slices, &c->cap_slices, slices_for(c->nnz, m, Amax), "merge slices"));
    int32_t* E = (int32_t*)c->d_mdp;
    RowPlan rp;
    rp.row = c->row;
    rp.ctr = c->d_ctr;
    rp.aff = c->d_aff;
    rp.seg_b = c->d_seg_b;
    rp.seg_d = c->d_seg_d;
    rp.E = E;
    rp.mrow = c->d_mrow;
    rp.mcap = 2 * c->ws_m;
    rp.slices = c->d_slices;
    rp.slice_cap = c->cap_slices;
    rp.longs = c->d_longs;
    rp.shorts = c->d_shorts;
    rp.long_in_place = c->tiered;
    rp.hbm_cap = c->pool_cap;
    rp.split = c->tiered;   // rows whose old version lives in HBM are rewritten into HBM, host rows into the host pool
    rp.base_hbm = c->tail;
    rp.base_host = 0;
    c->batch_dest = c->tiered ? 2 : 0;
    unsigned long long* sorted = c->d_keys;
    uint32_t* epos = (uint32_t*)c->d_keys_alt;
    rp.epos = epos;
    const int64_t sms = later ? c->sm_count / SIDE_MAX : c->sm_count;
    const bool one = m <= UPDATE_MAX && H <= 2 * sms * UPDATE_THREADS;
    if (one) {
        SCOUT_RC(update_ensure(c));
        UpdateParams up;
        up.g = g;
        up.pool = c->pool;
        up.e = d_src;
        up.ops = ops ? c->d_ops : nullptr;
        up.m = (int)m;
        up.B = B;
        up.raw = c->d_keys_alt;
        up.tmp = (unsigned long long*)c->d_mdp;
        up.keys = sorted;
        up.eflag = c->d_eflag;
        up.epos = epos;
        up.split = (unsigned long long*)c->d_update;
        up.cnt = up.split + UPDATE_SPLIT;
        up.bucket = (int*)(up.cnt + 1024);
        up.rows = c->tiered ? 0 : 1;
        up.rp = rp;
        up.aff = c->d_aff;
        up.seg_b = c->d_seg_b;
        up.seg_d = c->d_seg_d;
        up.E = E;
        up.bar = &c->d_batch->bar[0];
        if (later && !c->tiered) {   // the caller launches it (update_side)
            *later = up;
        } else {
            void* args[] = {&up};
            SCOUT_RC(coop_launch_own(c, (const void*)k_update, UPDATE_THREADS, args, 0));
        }
    } else {
        k_classify<<<blocks_for(m, 256), 256, 0, c->s_main>>>(g, d_src, ops ? c->d_ops : nullptr, m, B, c->d_keys,
                                                             c->d_eflag, c->d_ctr, 1);
        SCOUT_LAUNCH(c, "k_classify");
        c->nlaunch += 1;
        SCOUT_RC(sort_keys(c, c->d_keys, c->d_keys_alt, 2 * m, 2 * B + 1, &sorted));
        epos = (uint32_t*)(sorted == c->d_keys ? c->d_keys_alt : c->d_keys);   // the free ping-pong half
        rp.epos = epos;
        const int64_t tiles = (H + PLAN_TILE - 1) / PLAN_TILE;
        SCOUT_RC(dev_grow(c, &c->d_scan_tmp, &c->cap_scan, std::max<int64_t>(64, 1 + 3 * tiles), "scan look-back"));
        k_plan<<<(unsigned)tiles, PLAN_THREADS, 0, c->s_main>>>(c->row, c->pool, sorted, B, c->d_ctr, c->d_aff, c->d_seg_b,
                                                                c->d_seg_d, epos, E,
                                                                (unsigned long long*)c->d_scan_tmp + 1, next_stamp());
        SCOUT_LAUNCH(c, "k_plan");
        c->nlaunch += 1;
    }
    c->d_hkeys = sorted;
    const int nbr = blocks_for(Amax, ROW_THREADS, 8 * c->sm_count);
    if (c->tiered) {
        // the exact growth, before anything is written. HBM part too large: compact (evicting
        // short rows to the host pool); larger than three quarters of the HBM pool: the whole
        // batch goes to the host pool. Host pool full: compacted (host_compact, by the device).
        long long grow[2] = {0, 0};   // HBM, host
        auto read_grow = [&](bool again) -> int {
            if (again) SCOUT_CU(c, cudaMemsetAsync(&c->d_ctr->new_elems, 0, 16, c->s_main));
            rp.hbm_cap = c->pool_cap;
            k_row_sizes<<<nbr, ROW_THREADS, 0, c->s_main>>>(rp);
            SCOUT_LAUNCH(c, "k_row_sizes");
            c->nlaunch += 1;
            SCOUT_CU(c, cudaMemcpyAsync(grow, &c->d_ctr->new_elems, 16, cudaMemcpyDeviceToHost, c->s_main));
            SCOUT_CU(c, cudaStreamSynchronize(c->s_main));
            return SCOUT_OK;
        };
        SCOUT_RC(read_grow(false));
        // a hinted next batch is gathered into the free HBM above this merge: keep room for about
        // its endpoint rows at the average degree (two per edit), at most a quarter of the pool.
        // More room means evicting more rows to the host pool on every compaction, which costs
        // more over the host link than the merge saves on the gathered rows.
        long long headroom = 0;
        if (c->pf_pending && c->pf_m > 0) {
            const long long avg = c->n > 0 ? (c->nnz + c->n - 1) / c->n : 1;
            headroom = std::min<long long>(c->pool_cap / 4, 2 * c->pf_m * avg + 4096);
        }
        if (c->tail + grow[0] + 1024 + headroom > c->pool_cap) {
            if (grow[0] + 1024 + headroom <= c->pool_cap / 4 * 3) {
                SCOUT_RC(graph_compact(c, grow[0] + 1024 + headroom, true));
            } else if (c->tail + grow[0] + 1024 <= c->pool_cap) {
                // the gather gets what is left
            } else if (grow[0] + 1024 <= c->pool_cap / 4 * 3) {
                SCOUT_RC(graph_compact(c, grow[0] + 1024, true));
            } else {
                c->batch_dest = 1;
                c->host_batches++;
            }
            rp.split = c->batch_dest == 2;
            SCOUT_RC(read_grow(true));
        }
        const long long host_need = c->batch_dest == 1 ? grow[0] : grow[1];
        if (c->host_tail + host_need > c->host_cap) {
            SCOUT_RC(host_compact(c));
            if (c->host_tail + host_need > c->host_cap)
                return c->fail(SCOUT_E_CAPACITY, "tiered store: the host pool cannot take this batch's rows");
        }
        c->merge_tail = c->tail + (c->batch_dest == 1 ? 0 : grow[0]);
        const long long host_base = elem_delta(c->host_pool, c->pool) + c->host_tail;
        SCOUT_CU(c, cudaMemsetAsync(&c->d_ctr->new_elems, 0, 16, c->s_main));   // counted again by the allocation
        rp.hbm_cap = c->pool_cap;
        rp.base_hbm = c->batch_dest == 1 ? host_base : c->tail;
        rp.base_host = host_base;
    }
    if (!one || c->tiered) {
        k_row_plan<<<nbr, ROW_THREADS, 0, c->s_main>>>(rp);
        SCOUT_LAUNCH(c, "k_row_plan");
        k_merge<<<(unsigned)std::min<int64_t>(4 * c->sm_count, (Amax + c->nnz / SLICE) / MERGE_WARPS + 1), MERGE_THREADS, 0,
                  c->s_main>>>(c->pool, sorted, B, c->d_ctr, epos, E,
                               MergeList{c->d_mrow, c->d_slices, c->cap_slices, c->d_shorts});
        SCOUT_LAUNCH(c, "k_merge");
        c->nlaunch += 2;
    }
    if (c->tiered) {
        k_merge_long_inplace<<<(unsigned)std::min<int64_t>(std::max<int64_t>(1, Amax), 8 * (int64_t)c->sm_count),
                               LIP_THREADS, 0, c->s_main>>>(c->pool, c->d_ctr, epos, E, c->d_longs, c->d_mrow);
        SCOUT_LAUNCH(c, "k_merge_long_inplace");
        c->nlaunch += 1;
    }
    return SCOUT_OK;
}

}  // namespace scout

using namespace scout;

extern "C" {

// ---- graph store ---------------------------------------------------------------------------
int scout_graph_reserve(scout_ctx* c, int64_t n, int64_t nnz) {
    if (!c || n < 1 || n >= INT32_MAX || nnz < 0) return c ? c->fail(SCOUT_E_INVALID, "bad graph size") : SCOUT_E_INVALID;
    if (c->reserved) return c->fail(SCOUT_E_STATE, "graph already reserved");
    cudaSetDevice(c->device);
    c->n = n;
    SCOUT_RC(dev_alloc(c, (void**)&c->row, (size_t)n * sizeof(Row), "row table"));
    SCOUT_CU(c, cudaMemsetAsync(c->row, 0, (size_t)n * sizeof(Row), c->s_main));
    // Room for several batches of rewritten rows between compactions: a compaction copies every
    // live row whatever the garbage, so the larger the pool, the rarer they are. HBM is
    // plentiful (the pool and its compaction spare at eight times a 128 M-entry graph are
    // 8.6 GB); a budget that cannot hold that falls back to four, then two times the graph.
    const int64_t mult[3] = {8, 4, 2};
    for (int i = 0; i < 3; i++) {
        c->pool_cap = mult[i] * nnz + (i < 2 ? (1 << 26) : (1 << 22));
        if ((uint64_t)c->pool_cap * 4 * 2 + c->held <= c->budget) break;
    }
    SCOUT_RC(dev_alloc(c, (void**)&c->pool, (size_t)c->pool_cap * sizeof(int32_t), "element pool"));
    c->tail = 0;
    c->nnz = 0;
    c->reserved = true;
    c->sealed = false;
    return SCOUT_OK;
}

static int ensure_slabs(scout_ctx* c, int64_t elems, int64_t rows) {
    if (c->cap_slab < elems) {
        for (int i = 0; i < 2; i++) {
            if (c->h_slab[i]) { cudaEventSynchronize(c->ev_copy[i]); cudaFreeHost(c->h_slab[i]); c->h_slab[i] = nullptr; }
            SCOUT_CU(c, cudaMallocHost(&c->h_slab[i], (size_t)elems * 4));
        }
        c->cap_slab = elems;
    }
    if (c->cap_stage_rows < rows) {
        for (int i = 0; i < 2; i++) {
            if (c->h_slab_ids[i]) { cudaEventSynchronize(c->ev_copy[i]); cudaFreeHost(c->h_slab_ids[i]); cudaFreeHost(c->h_slab_off[i]); }
            if (c->d_stage_ids[i]) { dev_free(c, c->d_stage_ids[i], (size_t)c->cap_stage_rows * 4); dev_free(c, c->d_stage_off[i], (size_t)(c->cap_stage_rows + 1) * 8); }
            SCOUT_CU(c, cudaMallocHost((void**)&c->h_slab_ids[i], (size_t)rows * 4));
            SCOUT_CU(c, cudaMallocHost((void**)&c->h_slab_off[i], (size_t)(rows + 1) * 8));
            SCOUT_RC(dev_alloc(c, (void**)&c->d_stage_ids[i], (size_t)rows * 4, "staging ids"));
            SCOUT_RC(dev_alloc(c, (void**)&c->d_stage_off[i], (size_t)(rows + 1) * 8, "staging offsets"));
        }
        c->cap_stage_rows = rows;
    }
    return SCOUT_OK;
}

// One slab's worth of rows: bounce through pinned memory, async copy on the slot's stream,
// then a kernel points the row descriptors at the copied elements.
static int stage_chunk(scout_ctx* c, int slot, const int32_t* ids, const int64_t* offs, const int32_t* elems,
                       int64_t r0, int64_t r1) {
    int64_t e0 = offs[r0], e1 = offs[r1];
    int64_t ne = e1 - e0, nr = r1 - r0;
    if (c->tail + ne > c->pool_cap) return c->fail(SCOUT_E_CAPACITY, "element pool full while staging rows");
    SCOUT_CU(c, cudaEventSynchronize(c->ev_copy[slot]));
    std::memcpy(c->h_slab[slot], elems + e0, (size_t)ne * 4);
    std::memcpy(c->h_slab_ids[slot], ids + r0, (size_t)nr * 4);
    std::memcpy(c->h_slab_off[slot], offs + r0, (size_t)(nr + 1) * 8);
    cudaStream_t s = c->s_copy[slot];
    SCOUT_CU(c, cudaMemcpyAsync(c->pool + c->tail, c->h_slab[slot], (size_t)ne * 4, cudaMemcpyHostToDevice, s));
    SCOUT_CU(c, cudaMemcpyAsync(c->d_stage_ids[slot], c->h_slab_ids[slot], (size_t)nr * 4, cudaMemcpyHostToDevice, s));
    SCOUT_CU(c, cudaMemcpyAsync(c->d_stage_off[slot], c->h_slab_off[slot], (size_t)(nr + 1) * 8, cudaMemcpyHostToDevice, s));
    k_rows_from_stage<<<blocks_for(nr, 256), 256, 0, s>>>(c->row, c->d_stage_ids[slot], c->d_stage_off[slot], nr,
                                                          (long long)c->tail, (int32_t)c->n, c->d_flags);
    SCOUT_LAUNCH(c, "k_rows_from_stage");
    SCOUT_CU(c, cudaEventRecord(c->ev_copy[slot], s));
    c->tail += ne;
    return SCOUT_OK;
}

int scout_stage_rows(scout_ctx* c, int slot, const int32_t* ids, const int64_t* offs, const int32_t* elems,
                     int64_t nrows, int64_t nelems) {
    if (!c || !ids || !offs || (slot != 0 && slot != 1) || nrows < 0) return c ? c->fail(SCOUT_E_INVALID, "bad staging arguments") : SCOUT_E_INVALID;
    if (!c->reserved) return c->fail(SCOUT_E_STATE, "scout_graph_reserve first");
    if (nrows == 0) return SCOUT_OK;
    if (offs[nrows] - offs[0] != nelems || (!elems && nelems > 0)) return c->fail(SCOUT_E_INVALID, "offsets do not match nelems");
    cudaSetDevice(c->device);
    const int64_t SLAB = 1 << 24;
    int64_t maxrow = 0;
    for (int64_t i = 0; i < nrows; i++) {
        int64_t d = offs[i + 1] - offs[i];
        if (d < 0) return c->fail(SCOUT_E_INVALID, "offsets must be monotone");
        maxrow = std::max(maxrow, d);
    }
    SCOUT_RC(ensure_slabs(c, std::max(SLAB, maxrow), std::min<int64_t>(nrows, 1 << 20)));
    int64_t r = 0;
    int s = slot;
    while (r < nrows) {
        int64_t r1 = r;
        while (r1 < nrows && r1 - r < c->cap_stage_rows && offs[r1 + 1] - offs[r] <= c->cap_slab) r1++;
        SCOUT_RC(stage_chunk(c, s, ids, offs, elems, r, r1));
        r = r1;
        s ^= 1;
    }
    c->sealed = false;
    return SCOUT_OK;
}

int scout_graph_seal(scout_ctx* c) {
    if (!c) return SCOUT_E_INVALID;
    if (!c->reserved) return c->fail(SCOUT_E_STATE, "scout_graph_reserve first");
    cudaSetDevice(c->device);
    for (int i = 0; i < 2; i++) SCOUT_CU(c, cudaStreamWaitEvent(c->s_main, c->ev_copy[i], 0));
    // Rows must be ascending and in range; unsorted rows are sorted here (the reference keeps
    // rows in file order; every rule of this engine is order independent).
    int32_t* list = nullptr;
    int* flags = nullptr;
    SCOUT_RC(dev_alloc(c, (void**)&list, (size_t)c->n * 4, "seal list"));
    int rc = dev_alloc(c, (void**)&flags, 16, "seal flags");
    if (rc != SCOUT_OK) { dev_free(c, list, (size_t)c->n * 4); return rc; }
    cudaMemsetAsync(flags, 0, 16, c->s_main);
    k_check_rows<<<blocks_for(c->n * WARP, 256), 256, 0, c->s_main>>>(c->row, c->pool, (int32_t)c->n, list, flags, flags + 1);
    int h[4] = {0, 0, 0, 0};
    cudaMemcpyAsync(h, flags, 16, cudaMemcpyDeviceToHost, c->s_main);
    int bad_id = 0;
    cudaMemcpyAsync(&bad_id, c->d_flags, 4, cudaMemcpyDeviceToHost, c->s_main);
    cudaError_t e = cudaStreamSynchronize(c->s_main);
    if (e != cudaSuccess) { dev_free(c, list, (size_t)c->n * 4); dev_free(c, flags, 16); return cuda_fail(c, e, "seal"); }
    if (h[1] || bad_id) {
        dev_free(c, list, (size_t)c->n * 4);
        dev_free(c, flags, 16);
        cudaMemsetAsync(c->d_flags, 0, 16, c->s_main);
        return c->fail(SCOUT_E_INVALID, "staged rows hold vertex ids outside [0, n)");
    }
    if (h[0] > 0) {
        k_sort_rows_small<<<blocks_for(h[0], 1, 4096), 512, 0, c->s_main>>>(c->row, c->pool, list, h[0], flags + 2);
        int big = 0;
        cudaMemcpyAsync(&big, flags + 2, 4, cudaMemcpyDeviceToHost, c->s_main);
        cudaStreamSynchronize(c->s_main);
        if (big) {   // rows longer than 8192 entries: sorted on the host
            std::vector<int32_t> ids((size_t)h[0]);
            cudaMemcpy(ids.data(), list, (size_t)h[0] * 4, cudaMemcpyDeviceToHost);
            std::vector<int32_t> tmp;
            for (int32_t v : ids) {
                Row r;
                cudaMemcpy(&r, c->row + v, sizeof(Row), cudaMemcpyDeviceToHost);
                if (r.len <= 8192) continue;
                tmp.resize((size_t)r.len);
                cudaMemcpy(tmp.data(), c->pool + r.start, (size_t)r.len * 4, cudaMemcpyDeviceToHost);
                std::sort(tmp.begin(), tmp.end());
                cudaMemcpy(c->pool + r.start, tmp.data(), (size_t)r.len * 4, cudaMemcpyHostToDevice);
            }
        }
    }
    dev_free(c, list, (size_t)c->n * 4);
    dev_free(c, flags, 16);
    SCOUT_LAUNCH(c, "seal");
    // Contiguous rows, exact nnz and tail (a tiered load lays its rows out contiguously).
    if (!c->tiered) SCOUT_RC(graph_compact(c, std::max<int64_t>(c->pool_cap - c->tail, 1 << 22)));
    c->sealed = true;
    return SCOUT_OK;
}

int scout_graph_load_csr(scout_ctx* c, int64_t n, const int64_t* off, const int32_t* adj) {
    if (!c || !off || n < 1) return c ? c->fail(SCOUT_E_INVALID, "bad CSR") : SCOUT_E_INVALID;
    int64_t nnz = off[n];
    if (off[0] != 0 || nnz < 0 || (nnz > 0 && !adj)) return c->fail(SCOUT_E_INVALID, "bad CSR offsets");
    for (int64_t v = 0; v < n; v++)
        if (off[v + 1] < off[v]) return c->fail(SCOUT_E_INVALID, "CSR offsets must be monotone");
    // A budget that cannot hold the smallest single-tier store (row table, two pools of
    // 2 nnz + 4M entries, about 160 B of per-vertex state) gets the tiered store.
    const uint64_t single = (uint64_t)(16 * n + 160 * n) + 2ull * 4ull * (uint64_t)(2 * nnz + (1 << 22));
    if (c->held + single > c->budget) return scout_graph_load_tiered(c, n, off, adj, 0);
    SCOUT_RC(scout_graph_reserve(c, n, nnz));
    // Elements: contiguous pinned-slab copies on two streams.
    const int64_t SLAB = 1 << 24;
    SCOUT_RC(ensure_slabs(c, SLAB, 1024));
    int s = 0;
    for (int64_t e0 = 0; e0 < nnz; e0 += SLAB) {
        int64_t ne = std::min(SLAB, nnz - e0);
        SCOUT_CU(c, cudaEventSynchronize(c->ev_copy[s]));
        std::memcpy(c->h_slab[s], adj + e0, (size_t)ne * 4);
        SCOUT_CU(c, cudaMemcpyAsync(c->pool + e0, c->h_slab[s], (size_t)ne * 4, cudaMemcpyHostToDevice, c->s_copy[s]));
        SCOUT_CU(c, cudaEventRecord(c->ev_copy[s], c->s_copy[s]));
        s ^= 1;
    }
    int64_t* d_off = nullptr;
    SCOUT_RC(dev_alloc(c, (void**)&d_off, (size_t)(n + 1) * 8, "load offsets"));
    SCOUT_CU(c, cudaMemcpyAsync(d_off, off, (size_t)(n + 1) * 8, cudaMemcpyHostToDevice, c->s_main));
    k_rows_from_offsets<<<blocks_for(n, 256), 256, 0, c->s_main>>>(c->row, d_off, n, 0);
    SCOUT_LAUNCH(c, "k_rows_from_offsets");
    SCOUT_CU(c, cudaStreamSynchronize(c->s_main));
    dev_free(c, d_off, (size_t)(n + 1) * 8);
    c->tail = nnz;
    return scout_graph_seal(c);
}

// Tiered load: the highest-degree rows (up to half the HBM pool, the rest of it left for rows
// the batches rewrite) are copied to HBM; every other row goes to a mapped page-locked host
// pool that the kernels read in place. Rows are sorted here, on the host.
int scout_graph_load_tiered(scout_ctx* c, int64_t n, const int64_t* off, const int32_t* adj, int64_t hbm_entries) {
    if (!c || !off || n < 1 || n >= INT32_MAX) return c ? c->fail(SCOUT_E_INVALID, "bad CSR") : SCOUT_E_INVALID;
    if (c->reserved) return c->fail(SCOUT_E_STATE, "graph already reserved");
    const int64_t nnz = off[n];
    if (off[0] != 0 || nnz < 0 || (nnz > 0 && !adj)) return c->fail(SCOUT_E_INVALID, "bad CSR offsets");
    for (int64_t v = 0; v < n; v++)
        if (off[v + 1] < off[v] || off[v + 1] - off[v] > INT32_MAX) return c->fail(SCOUT_E_INVALID, "CSR offsets must be monotone");
    cudaSetDevice(c->device);
    if (hbm_entries <= 0) {
        // what the budget leaves after the row table and about 160 B of per-vertex state, for
        // two HBM pools (the pool and its compaction target)
        const int64_t fixed = (int64_t)c->held + 16 * n + 160 * n;
        hbm_entries = std::max<int64_t>(1 << 20, ((int64_t)c->budget - fixed) / 8);
    }
    c->n = n;
    SCOUT_RC(dev_alloc(c, (void**)&c->row, (size_t)n * sizeof(Row), "row table"));
    c->pool_cap = hbm_entries;
    SCOUT_RC(dev_alloc(c, (void**)&c->pool, (size_t)c->pool_cap * sizeof(int32_t), "element pool"));
    // after a host compaction the pool holds at most the live graph, and one batch adds at
    // most a rewrite of every row it touches: 2 nnz (plus slack for insertions)
    c->host_cap = 2 * nnz + (1 << 22);
    {
        void* hp = nullptr;
        cudaError_t e = cudaHostAlloc(&hp, (size_t)c->host_cap * 4, cudaHostAllocMapped | cudaHostAllocPortable);
        if (e != cudaSuccess) { cudaGetLastError(); return c->fail(SCOUT_E_CAPACITY, std::string("host pool: ") + cudaGetErrorString(e)); }
        void* dp = nullptr;
        SCOUT_CU(c, cudaHostGetDevicePointer(&dp, hp, 0));
        if (dp != hp) return c->fail(SCOUT_E_NODEV, "tiered store needs unified addressing of page-locked memory");
        c->host_pool = (int32_t*)hp;
    }
    c->tiered = true;
    // placement: hot rows by descending degree while they fit half the HBM pool
    std::vector<int32_t> order(n);
    for (int64_t v = 0; v < n; v++) order[v] = (int32_t)v;
    std::sort(order.begin(), order.end(), [&](int32_t a, int32_t b) {
        const int64_t da = off[a + 1] - off[a], db = off[b + 1] - off[b];
        return da != db ? da > db : a < b;
    });
    std::vector<Row> rows(n);
    std::vector<char> hot(n, 0);
    int64_t hbm_used = 0;
    for (int64_t i = 0; i < n; i++) {
        const int32_t v = order[i];
        const int64_t d = off[v + 1] - off[v];
        if (hbm_used + d > hbm_entries / 2) break;
        rows[v] = Row{hbm_used, (int)d, (int)d};
        hot[v] = 1;
        hbm_used += d;
    }
    const long long host_rel = elem_delta(c->host_pool, c->pool);
    int64_t host_used = 0;
    std::vector<int64_t> hpos(n, -1);
    for (int64_t v = 0; v < n; v++) {
        if (hot[v]) continue;
        const int64_t d = off[v + 1] - off[v];
        hpos[v] = host_used;
        rows[v] = Row{host_rel + host_used, (int)d, (int)d};
        host_used += d;
    }
#pragma omp parallel for schedule(dynamic, 4096)
    for (int64_t v = 0; v < n; v++) {
        if (hpos[v] < 0) continue;
        int32_t* dst = c->host_pool + hpos[v];
        const int64_t d = off[v + 1] - off[v];
        std::memcpy(dst, adj + off[v], (size_t)d * 4);
        if (!std::is_sorted(dst, dst + d)) std::sort(dst, dst + d);
    }
    // hot rows: gathered in HBM order into the pinned slabs, sorted, copied on two streams
    const int64_t SLAB = 1 << 24;
    SCOUT_RC(ensure_slabs(c, SLAB, 1024));
    int s = 0;
    int64_t i = 0, pos = 0;
    while (pos < hbm_used) {
        SCOUT_CU(c, cudaEventSynchronize(c->ev_copy[s]));
        int32_t* slab = (int32_t*)c->h_slab[s];
        const int64_t p0 = pos;
        while (i < n && hot[order[i]]) {
            const int32_t v = order[i];
            const int64_t d = off[v + 1] - off[v];
            if (pos - p0 + d > SLAB) {
                if (pos == p0) return c->fail(SCOUT_E_CAPACITY, "a row is longer than the staging slab");
                break;
            }
            int32_t* dst = slab + (pos - p0);
            std::memcpy(dst, adj + off[v], (size_t)d * 4);
            if (!std::is_sorted(dst, dst + d)) std::sort(dst, dst + d);
            pos += d;
            i++;
        }
        SCOUT_CU(c, cudaMemcpyAsync(c->pool + p0, slab, (size_t)(pos - p0) * 4, cudaMemcpyHostToDevice, c->s_copy[s]));
        SCOUT_CU(c, cudaEventRecord(c->ev_copy[s], c->s_copy[s]));
        s ^= 1;
    }
    SCOUT_CU(c, cudaMemcpy(c->row, rows.data(), (size_t)n * sizeof(Row), cudaMemcpyHostToDevice));
    c->tail = hbm_used;
    c->host_tail = host_used;
    c->nnz = nnz;
    c->reserved = true;
    c->sealed = false;
    return scout_graph_seal(c);
}

int scout_graph_tier_info(scout_ctx* c, int64_t* hbm_cap, int64_t* hbm_used, int64_t* host_cap, int64_t* host_used,
                          int64_t* evictions, int64_t* host_batches) {
    if (!c) return SCOUT_E_INVALID;
    if (host_batches) *host_batches = c->host_batches;
    if (hbm_cap) *hbm_cap = c->pool_cap;
    if (hbm_used) *hbm_used = c->tail;
    if (host_cap) *host_cap = c->tiered ? c->host_cap : 0;
    if (host_used) *host_used = c->tiered ? c->host_tail : 0;
    if (evictions) *evictions = c->evicted_entries;
    return SCOUT_OK;
}

int scout_graph_info(scout_ctx* c, int64_t* n, int64_t* nnz, int64_t* used, int64_t* cap) {
    if (!c) return SCOUT_E_INVALID;
    if (n) *n = c->n;
    if (nnz) *nnz = c->nnz;
    if (used) *used = c->tail;
    if (cap) *cap = c->pool_cap;
    return SCOUT_OK;
}

int scout_graph_download(scout_ctx* c, int64_t* off, int32_t* adj, int64_t cap) {
    if (!c || !off) return SCOUT_E_INVALID;
    if (!c->sealed) return c->fail(SCOUT_E_STATE, "graph not sealed");
    cudaSetDevice(c->device);
    SCOUT_RC(gather_finish(c, nullptr, nullptr, nullptr));
    const int64_t n = c->n;
    int64_t* d_off = nullptr;
    SCOUT_RC(dev_alloc(c, (void**)&d_off, (size_t)(n + 1) * 8, "download offsets"));
    k_row_lens<<<blocks_for(n, 256), 256, 0, c->s_main>>>(c->row, n, d_off);
    int rc = scan_i64(c, d_off, n, d_off + n);
    if (rc == SCOUT_OK && cudaMemcpyAsync(off, d_off, (size_t)(n + 1) * 8, cudaMemcpyDeviceToHost, c->s_main) != cudaSuccess) rc = SCOUT_E_CUDA;
    if (rc == SCOUT_OK && cudaStreamSynchronize(c->s_main) != cudaSuccess) rc = cuda_fail(c, cudaGetLastError(), "download");
    if (rc != SCOUT_OK) { dev_free(c, d_off, (size_t)(n + 1) * 8); return rc; }
    int64_t total = off[n];
    if (!adj || cap < total) { dev_free(c, d_off, (size_t)(n + 1) * 8); return c->fail(SCOUT_E_CAPACITY, "adjacency buffer too small"); }
    int32_t* tmp = nullptr;
    rc = dev_alloc(c, (void**)&tmp, (size_t)std::max<int64_t>(total, 1) * 4, "download buffer");
    if (rc != SCOUT_OK) { dev_free(c, d_off, (size_t)(n + 1) * 8); return rc; }
    k_copy_rows<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((n + total + COPY_UNITS - 1) / COPY_UNITS,
                                                                    32 * c->sm_count)),
                  COPY_THREADS, 0, c->s_main>>>(c->row, c->pool, tmp, d_off, (int32_t)n, (long long)total);
    cudaMemcpyAsync(adj, tmp, (size_t)total * 4, cudaMemcpyDeviceToHost, c->s_main);
    cudaError_t e = cudaStreamSynchronize(c->s_main);
    dev_free(c, tmp, (size_t)std::max<int64_t>(total, 1) * 4);
    dev_free(c, d_off, (size_t)(n + 1) * 8);
    if (e != cudaSuccess) return cuda_fail(c, e, "download");
    return SCOUT_OK;
}

int scout_graph_compact(scout_ctx* c) {
    if (!c) return SCOUT_E_INVALID;
    if (!c->sealed) return c->fail(SCOUT_E_STATE, "graph not sealed");
    cudaSetDevice(c->device);
    SCOUT_RC(gather_finish(c, nullptr, nullptr, nullptr));
    return graph_compact(c, std::max<int64_t>(c->nnz, 1 << 22), true);
}

int scout_classify(scout_ctx* c, const scout_edge* e, int64_t m, uint8_t* out) {
    if (!c || (m > 0 && (!e || !out)) || m < 0) return c ? c->fail(SCOUT_E_INVALID, "bad arguments") : SCOUT_E_INVALID;
    if (!c->sealed) return c->fail(SCOUT_E_STATE, "graph not sealed");
    if (m == 0) return SCOUT_OK;
    cudaSetDevice(c->device);
    SCOUT_RC(ws_ensure(c, m));
    // (no batch begins: the last repair's counters and changed entries stay, for its commit)
    SCOUT_RC(gather_finish(c, nullptr, nullptr, nullptr));
    SCOUT_RC(pin_grow(c, &c->h_pin_edits, &c->cap_pin_edits, m * (int64_t)sizeof(scout_edge) + m));
    std::memcpy(c->h_pin_edits, e, (size_t)m * sizeof(scout_edge));
    SCOUT_CU(c, cudaMemcpyAsync(c->d_edits, c->h_pin_edits, (size_t)m * sizeof(scout_edge), cudaMemcpyHostToDevice, c->s_main));
    k_classify<<<blocks_for(m, 256), 256, 0, c->s_main>>>(dgraph(c), c->d_edits, nullptr, m, 1, nullptr, c->d_eflag, nullptr, 0);
    SCOUT_LAUNCH(c, "k_classify");
    uint8_t* pf = (uint8_t*)c->h_pin_edits + m * sizeof(scout_edge);
    SCOUT_CU(c, cudaMemcpyAsync(pf, c->d_eflag, (size_t)m, cudaMemcpyDeviceToHost, c->s_main));
    SCOUT_CU(c, cudaStreamSynchronize(c->s_main));
    for (int64_t i = 0; i < m; i++) out[i] = (pf[i] & 1) ? (uint8_t)((pf[i] >> 1) & 1) : (uint8_t)0xFF;
    return SCOUT_OK;
}

}  // extern "C"
