// seed.cu -- initial solutions computed on the device from the resident graph.
//
// The reference seeds its streams with offline host tools: greedy MIS in vertex-id order
// (tools/compute_initial_mis.py:32-43), greedy smallest-free colouring in vertex-id order
// (tools/greedy_color.cpp:37-52), BFS levels (tools/bfs_ground_truth.cu:39-151) and min-id
// component labels (tools/excc_src/excc_v1.cu:520-531). scout_seed computes the same solutions
// on the GPU: BFS and CC by the engine's own full traversal and recompute, the two greedy
// rules by persistent kernels of rounds. A vertex decides once every lower-id neighbour has
// decided (rows are sorted, so those neighbours are a prefix of its row):
//   MIS       in iff no lower-id neighbour is in
//   colouring the smallest colour no lower-id neighbour has
// Decisions only go from undecided to final, so reading neighbours that decide during the same
// round cannot change any outcome: the result is the sequential greedy one whatever the timing.
// The number of rounds is the longest chain of vertices each waiting on a lower-id neighbour
// (about 900 on an R-MAT graph of 500,000 vertices, edge factor 16).
//
// Both rules begin with rounds that look at every open vertex (k_seed_rounds). That settles graphs of
// short chains alone: a greedy MIS decides a vertex as soon as any lower neighbour joins (6 to 13
// rounds on R-MAT graphs of 2,000 to 2 M vertices and on random graphs, where waiting in lists takes
// 35 to 233, as a waiter hears of a joined neighbour only when the one it waits for decides), and so
// are a colouring's chains on shuffled grids or with a few hubs. What is open after SEED_ROUNDS rounds
// (a colouring: after SEED_FIRST, once a round leaves more than 7/8 open; its prefixes of more than
// SEED_BIG entries at once) is finished by waiter lists. Whole calls, lists alone and so: MIS,
// R-MAT of edge factor 16, 8,000 vertices 424 and 249 us, 100,000 917 and 447, 2 M 4,950 and 2,180;
// grid of 700 x 700 numbered in order 9.2 and 9.7 ms (17.4 by rounds alone); colouring, the same grid
// shuffled 644 and 187 us, 300,000 vertices on 60 hubs 1,850 and 286, R-MAT of 500,000 11.1 and
// 11.2 ms.
//
// The lists (k_seed_greedy). What bounds it: the latency of a round (a few hundred open vertices
// decide in each), so a round only touches vertices that can move. An open vertex waits on ONE
// undecided neighbour, the highest-id one (it tends to decide last, so few waits follow one
// another), in that neighbour's list of waiters; a vertex that decides closes its list and queues
// the waiters for the next round. The list of w holds at most as many waiters as w has higher-id neighbours; a
// vertex that finds it full (rows that are not symmetric, or no memory for the lists) is queued
// again itself and simply looks again next round. One grid barrier per round.
// Greedy colouring of 500,009 vertices (edge factor 16): 1,073 ms with every open vertex
// rescanning its row by one thread in every round, 11.2 ms so (902 rounds; a round costs about
// 7 us of dependent L2 accesses and one barrier on small graphs, 12 us here, where long
// prefixes are scanned).
#include "ctx.cuh"

#include <algorithm>
#include <cstring>

namespace scout {

constexpr int SEED_THREADS = 1024;
constexpr int32_t UNDECIDED = -1;
constexpr int SEED_ROUNDS = 32;             // MIS rounds before the lists take over
constexpr int SEED_FIRST = 7;               // colouring rounds whatever they decide
constexpr int SEED_ASK = 16384;             // vertices from which a colouring's rounds are waited for
constexpr int SEED_BIG = 1024;              // longer prefixes are scanned by a whole block
constexpr int SEED_WORDS = 32;              // bitmap window: 1024 colours
constexpr int SEED_CLOSED = 0x40000000;     // a closed waiter list's count
constexpr int32_t SLOT_CLOSED = -2;         // a slot whose list closed before it was filled

struct SeedParams {
    DGraph g;
    int32_t* out;       // MIS: 1 in / 0 out; colouring: colour; UNDECIDED while open
    int mode;           // 0 MIS, 1 colouring
    int32_t* wl[2];     // vertices to look at in this and the next round (n each)
    int32_t* pre;       // lower-id entries of every row
    int32_t* open;      // entries below this index may still be undecided
    int32_t* nwait;     // waiters in a vertex's list
    int32_t* waiters;   // every list's slots (-1), list v at [off[v], off[v + 1]); null: no lists
    const int64_t* off;
    DevCounters* ctr;   // list_count[0..2]: rotating sizes of wl; rounds
    GridBar* bar;
};

// Rounds over all open vertices, one thread each, until none is open, SEED_ROUNDS are done or
// (colouring) a round has left more than 7/8 of them open. ctr->affected: the vertices left open.
__global__ void __launch_bounds__(SEED_THREADS, 1) k_seed_rounds(SeedParams p) {
    const int64_t n = p.g.n;
    const int64_t tid = lthread_id();
    const int64_t T = (int64_t)gridDim.x * blockDim.x;
    const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
    for (int64_t v = tid; v < n; v += T) p.out[v] = UNDECIDED;
    if (!grid_sync(p.bar, 50)) return;
    int cur = 2, rounds = 0, cnt = (int)n, before = INT32_MAX;
    long long bytes = 0;
    while (cnt > 0 && rounds < SEED_ROUNDS && (p.mode == 0 || rounds < SEED_FIRST || cnt <= before - before / 8)) {
        const int nxt = (cur + 1) % 3, zer = (cur + 2) % 3;
        const int32_t* wl = p.wl[rounds & 1];
        int32_t* wn = p.wl[(rounds & 1) ^ 1];
        if (leader) p.ctr->list_count[zer] = 0;
        for (int64_t b = tid - (tid & (WARP - 1)); b < cnt; b += T) {
            const int64_t i = b + lane_id();
            bool open = false;
            int32_t v = 0;
            if (i < cnt) {
                v = rounds ? wl[i] : (int32_t)i;   // every vertex in the first round
                const Row r = p.g.row[v];
                const int32_t* row = p.g.pool + r.start;
                const int k = (int)lower_bound_i32(row, r.len, v);
                bytes += 16 + 4LL * k * 2;
                bool any_in = false, all_done = true;
                if (p.mode == 0) {
                    for (int j = 0; j < k && !any_in; j++) {
                        const int32_t s = ld_volatile(p.out + row[j]);
                        any_in = s == 1;
                        all_done &= s != UNDECIDED;
                    }
                    open = !any_in && !all_done;
                    if (!open) p.out[v] = any_in ? 0 : 1;
                } else {
                    if (k > SEED_BIG) all_done = false;   // left to the lists' blocks
                    for (int j = 0; j < k && all_done; j++) all_done = ld_volatile(p.out + row[j]) != UNDECIDED;
                    open = !all_done;
                    if (!open) {
                        int32_t colour = 0;
                        for (int32_t base = 0;; base += 64) {   // smallest colour absent below
                            unsigned long long used = 0;
                            for (int j = 0; j < k; j++) {
                                const int32_t c = ld_volatile(p.out + row[j]) - base;
                                if (c >= 0 && c < 64) used |= 1ull << c;
                            }
                            if (~used) { colour = base + __ffsll((long long)~used) - 1; break; }
                        }
                        p.out[v] = colour;
                    }
                }
            }
            const int at = warp_append(open, &p.ctr->list_count[nxt]);
            if (open) wn[at] = v;
        }
        rounds++;
        if (!grid_sync(p.bar, 51)) return;
        cur = nxt;
        before = cnt;
        cnt = ld_volatile(&p.ctr->list_count[cur]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
    if (lane_id() == 0) atomicAdd((unsigned long long*)&p.ctr->hbm_bytes, (unsigned long long)bytes);
    if (leader) {
        p.ctr->rounds = rounds;
        p.ctr->affected = cnt;
    }
}

// Per vertex: the row prefix of neighbours below it, the slots its waiter list gets. The list of a vertex
// that the rounds have decided is closed.
__global__ void k_seed_prep(DGraph g, const int32_t* __restrict__ out, int32_t* __restrict__ pre,
                            int32_t* __restrict__ open, int32_t* __restrict__ nwait, int64_t* __restrict__ slots) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < g.n; v += (int64_t)gridDim.x * blockDim.x) {
        const Row r = g.row[v];
        const int32_t* row = g.pool + r.start;
        const int k = (int)lower_bound_i32(row, r.len, (int32_t)v);
        pre[v] = k;
        open[v] = k;
        nwait[v] = out[v] != UNDECIDED ? SEED_CLOSED : 0;
        slots[v] = r.len - k;   // a loop's own entry only adds a slot
    }
}

// Every lane with `pred` appends v to the next round's queue (all 32 lanes call).
__device__ __forceinline__ void seed_queue(const SeedParams& p, bool pred, int32_t v, int nxt, int32_t* wl) {
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (!m) return;
    int base = 0;
    if (lane_id() == 0) base = atomicAdd(&p.ctr->list_count[nxt], __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (pred) wl[base + __popc(m & ((1u << lane_id()) - 1))] = v;
}

// v waits for w. 0: it does; 1: no room, look again next round; 2: w has decided meanwhile.
__device__ __forceinline__ int seed_wait(const SeedParams& p, int32_t v, int32_t w) {
    if (!p.waiters) return ld_volatile(p.out + w) == UNDECIDED ? 1 : 2;
    const int64_t o = p.off[w];
    const int cap = (int)(p.off[w + 1] - o);
    const int at = atomicAdd(p.nwait + w, 1);
    int res = 1;
    if (at >= SEED_CLOSED) res = 2;
    else if (at < cap) res = atomicExch(p.waiters + o + at, v) == SLOT_CLOSED ? 2 : 0;
    if (res == 2) __threadfence();   // w's value is read after its closed list was seen
    return res;
}

// v has its value: it is written, then v's list is closed (who sees the list closed sees the
// value). Returns the number of waiters.
__device__ __forceinline__ int seed_close(const SeedParams& p, int32_t v, int32_t val) {
    p.out[v] = val;
    __threadfence();
    return atomicOr(p.nwait + v, SEED_CLOSED);
}

// The waiters of a closed list go to the next round's queue; `lanes` threads of one
// group (a warp, or a block in warps of which each calls this with its own tid) share the list.
__device__ __forceinline__ void seed_release(const SeedParams& p, int32_t v, int cnt, int tid, int lanes, int nxt,
                                             int32_t* wl) {
    if (!p.waiters) return;
    const int64_t o = p.off[v];
    const int c = min(cnt, (int)(p.off[v + 1] - o));
    for (int b = tid - (int)lane_id(); b < c; b += lanes) {
        const int i = b + (int)lane_id();
        int32_t x = -1;
        if (i < c) x = atomicExch(p.waiters + o + i, SLOT_CLOSED);   // -1: its waiter sees the mark
        seed_queue(p, x >= 0, x, nxt, wl);
    }
}

// The colouring's bitmap of 1024 colours from `base`: entries [0, k) of the row, by `lanes`
// threads; the smallest absent colour is found by the caller after its group's barrier.
__device__ __forceinline__ void seed_mark(const SeedParams& p, const int32_t* row, int k, int tid, int lanes, int base,
                                          unsigned* bm) {
    constexpr int U = 8;
    for (int b = tid; b < k; b += U * lanes) {
        int32_t c[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = b + u * lanes;
            c[u] = i < k ? ld_volatile(p.out + row[i]) - base : -1;
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c[u] >= 0 && c[u] < SEED_WORDS * 32) atomicOr(&bm[c[u] >> 5], 1u << (c[u] & 31));
    }
}

// One warp: v's value if it can be decided now (UNDECIDED otherwise; *on: the neighbour it
// waits for). MIS looks at the whole prefix: one member settles it whatever is undecided.
__device__ __forceinline__ int32_t seed_decide(const SeedParams& p, const int32_t* row, int k, int32_t v, int32_t* on,
                                               unsigned* bm, long long& bytes) {
    const int l = (int)lane_id();
    constexpr int U = 8;   // entries per lane and step: their loads are in flight together
    const int o = p.open[v];
    int32_t wait = -1;
    for (int hi = o; hi > 0; hi -= U * WARP) {   // from the top, lane 31 of u = 0 first
        int32_t x[U], s[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = hi - (u + 1) * WARP + l;
            x[u] = i >= 0 ? row[i] : -1;
        }
        bool in = false;
#pragma unroll
        for (int u = 0; u < U; u++) {
            s[u] = x[u] >= 0 ? ld_volatile(p.out + x[u]) : 0;
            in |= x[u] >= 0 && s[u] == 1;
        }
        if (p.mode == 0 && __any_sync(0xffffffffu, in)) return 0;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const unsigned um = __ballot_sync(0xffffffffu, x[u] >= 0 && s[u] == UNDECIDED);
            if (um && wait < 0) {
                const int top = 31 - __clz(um);
                wait = __shfl_sync(0xffffffffu, x[u], top);
                if (l == 0) p.open[v] = hi - (u + 1) * WARP + top + 1;
            }
        }
        if (wait >= 0 && p.mode != 0) break;
    }
    if (l == 0) bytes += 16 + 8LL * o;
    if (wait >= 0) { *on = wait; return UNDECIDED; }
    if (p.mode == 0) return 1;   // the entries above `open` were seen decided and out
    if (l == 0) bytes += 8LL * k;
    for (int base = 0;; base += SEED_WORDS * 32) {
        bm[l] = 0;
        __syncwarp();
        seed_mark(p, row, k, l, WARP, base, bm);
        __syncwarp();
        const unsigned fr = ~bm[l];
        const unsigned any = __ballot_sync(0xffffffffu, fr != 0);
        if (any) {
            const int w = __ffs(any) - 1;
            return base + w * 32 + __ffs(__shfl_sync(0xffffffffu, fr, w)) - 1;
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(SEED_THREADS, 1) k_seed_greedy(SeedParams p) {
    __shared__ unsigned s_bm[SEED_THREADS / WARP][SEED_WORDS];
    __shared__ int32_t s_list[SEED_THREADS / WARP];
    __shared__ int s_big, s_top, s_in, s_col, s_cnt, s_act;
    const int64_t n = p.g.n;
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t T = (int64_t)gridDim.x * blockDim.x;
    const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
    const int W = gwarp_count(), t = threadIdx.x, wl_ = threadIdx.x / WARP;
    long long bytes = 0;
    // round 0, one lane per vertex: without a lower neighbour it decides, else it waits for the
    // highest one
    for (int64_t b = tid - (tid & (WARP - 1)); b < n; b += T) {
        const int64_t v = b + lane_id();
        bool again = false;
        int cnt = 0;
        if (v < n && ld_volatile(p.nwait + v) < SEED_CLOSED) {   // (closed: decided by the rounds before)
            const int k = p.pre[v];
            bytes += 24;
            if (k == 0) {
                cnt = seed_close(p, (int32_t)v, p.mode == 0 ? 1 : 0);
            } else {
                again = seed_wait(p, (int32_t)v, p.g.pool[p.g.row[v].start + k - 1]) != 0;
            }
        }
        seed_queue(p, again, (int32_t)v, 0, p.wl[0]);
        unsigned m = __ballot_sync(0xffffffffu, cnt > 0);
        while (m) {
            const int j = __ffs(m) - 1;
            m &= m - 1;
            seed_release(p, (int32_t)(b + j), __shfl_sync(0xffffffffu, cnt, j), (int)lane_id(), WARP, 0, p.wl[0]);
        }
    }
    if (!grid_sync(p.bar, 50)) return;
    int cur = 0, rounds = 1;
    while (true) {
        const int cnt = ld_volatile(&p.ctr->list_count[cur]);
        if (cnt == 0) break;
        const int nxt = (cur + 1) % 3, zer = (cur + 2) % 3;
        const int32_t* wl = p.wl[rounds & 1 ? 0 : 1];
        int32_t* wn = p.wl[rounds & 1 ? 1 : 0];
        if (leader) p.ctr->list_count[zer] = 0;
        // a block takes one vertex per warp at a time; those with a long prefix are set aside and
        // shared among all its warps
        for (int i0 = blockIdx.x * (blockDim.x / WARP); i0 < cnt; i0 += W) {
            const int i = i0 + wl_;
            const int32_t v = i < cnt ? wl[i] : -1;
            const int k = v >= 0 ? p.pre[v] : 0;
            if (t == 0) s_big = 0;
            __syncthreads();
            if (k > SEED_BIG) {
                if (lane_id() == 0) s_list[atomicAdd(&s_big, 1)] = v;
            } else if (v >= 0) {
                const int32_t* row = p.g.pool + p.g.row[v].start;
                while (true) {
                    int32_t on = -1;
                    const int32_t val = seed_decide(p, row, k, v, &on, s_bm[wl_], bytes);
                    int res = 0;
                    if (lane_id() == 0) {
                        if (val == UNDECIDED) {
                            res = seed_wait(p, v, on);
                        } else {
                            res = seed_close(p, v, val);
                        }
                    }
                    res = __shfl_sync(0xffffffffu, res, 0);
                    if (val != UNDECIDED) { seed_release(p, v, res, (int)lane_id(), WARP, nxt, wn); break; }
                    if (res == 2) continue;   // its neighbour decided meanwhile: look again
                    seed_queue(p, res == 1 && lane_id() == 0, v, nxt, wn);
                    break;
                }
            }
            __syncthreads();
            const int nbig = s_big;
            for (int j = 0; j < nbig; j++) {
                const int32_t v = s_list[j];
                const int k = p.pre[v];
                const int32_t* row = p.g.pool + p.g.row[v].start;
                while (true) {
                    if (t == 0) { s_top = -1; s_in = 0; }
                    __syncthreads();
                    const int o = p.mode == 0 ? k : p.open[v];
                    constexpr int U = 4;
                    int mine = -1;   // this thread's highest undecided entry
                    for (int b = t; b < o; b += U * blockDim.x) {
                        int32_t s[U];
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const int x = b + u * (int)blockDim.x;
                            s[u] = x < o ? ld_volatile(p.out + row[x]) : 0;
                        }
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            if (s[u] == UNDECIDED) mine = b + u * (int)blockDim.x;
                            else if (s[u] == 1 && p.mode == 0) s_in = 1;
                        }
                    }
                    mine = __reduce_max_sync(0xffffffffu, mine);
                    if (lane_id() == 0 && mine >= 0) atomicMax(&s_top, mine);
                    if (t == 0) bytes += 16 + 8LL * o;
                    __syncthreads();
                    const int top = s_top;
                    const bool in = s_in != 0;
                    int32_t val = UNDECIDED;
                    if (p.mode == 0) {
                        if (in) val = 0;
                        else if (top < 0) val = 1;
                    } else if (top < 0) {
                        for (int base = 0; val == UNDECIDED; base += SEED_WORDS * 32) {
                            if (t < SEED_WORDS) s_bm[0][t] = 0;
                            if (t == 0) s_col = INT32_MAX;
                            __syncthreads();
                            seed_mark(p, row, k, t, blockDim.x, base, s_bm[0]);
                            __syncthreads();
                            if (t < SEED_WORDS && ~s_bm[0][t]) atomicMin(&s_col, t * 32 + __ffs(~s_bm[0][t]) - 1);
                            __syncthreads();
                            if (s_col != INT32_MAX) val = base + s_col;
                            __syncthreads();
                        }
                        if (t == 0) bytes += 8LL * k;
                    }
                    if (t == 0) {
                        if (val == UNDECIDED) {
                            p.open[v] = top + 1;
                            s_act = seed_wait(p, v, row[top]);
                            s_cnt = 0;
                        } else {
                            s_cnt = seed_close(p, v, val);
                            s_act = 0;
                        }
                    }
                    __syncthreads();
                    const int act = s_act, c = s_cnt;
                    __syncthreads();
                    if (val != UNDECIDED) seed_release(p, v, c, t, blockDim.x, nxt, wn);
                    if (act == 2) continue;
                    if (t < WARP) seed_queue(p, act == 1 && t == 0, v, nxt, wn);
                    break;
                }
            }
            __syncthreads();   // the list is read before the next vertices fill it
        }
        rounds++;
        if (!grid_sync(p.bar, 51)) return;
        cur = nxt;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
    if (lane_id() == 0) atomicAdd((unsigned long long*)&p.ctr->hbm_bytes, (unsigned long long)bytes);
    if (leader) p.ctr->rounds += rounds;
}

// The lists' scratch and kernel, and the counters.
static int seed_lists(scout_ctx* c, SeedParams p) {
    const int64_t n = c->n;
    if (!c->d_coff) SCOUT_RC(dev_alloc(c, (void**)&c->d_coff, (size_t)(n + 1) * sizeof(int64_t), "compaction offsets"));
    p.pre = (int32_t*)c->d_qbuf[0];    // the work queues are free outside a repair (qcap >= n items)
    p.open = (int32_t*)c->d_qbuf[1];
    p.nwait = (int32_t*)c->d_qbuf[2];
    p.off = c->d_coff;
    k_seed_prep<<<blocks_for(n, 256), 256, 0, c->s_main>>>(p.g, p.out, p.pre, p.open, p.nwait, c->d_coff);
    SCOUT_LAUNCH(c, "k_seed_prep");
    SCOUT_RC(scan_i64(c, c->d_coff, n, c->d_coff + n));
    // the waiter lists hold at most nnz slots in all: the compaction spare's memory (its contents
    // are dead between compactions), or an allocation of its own if the budget has room
    const int64_t slots = std::max<int64_t>(c->nnz, 1);
    int32_t* own = nullptr;
    if (c->spare && c->spare_cap >= slots) {
        p.waiters = c->spare;
    } else {
        const std::string before = c->err;
        if (dev_alloc(c, (void**)&own, (size_t)slots * 4, "waiter lists") != SCOUT_OK) { own = nullptr; c->err = before; }
        p.waiters = own;
    }
    void* args[] = {&p};
    int rc = SCOUT_OK;
    if (p.waiters && cudaMemsetAsync(p.waiters, 0xff, (size_t)slots * 4, c->s_main) != cudaSuccess)
        rc = cuda_fail(c, cudaGetLastError(), "seed");
    if (rc == SCOUT_OK) rc = coop_launch(c, (const void*)k_seed_greedy, SEED_THREADS, args, 0);
    c->nlaunch += 1;
    if (rc == SCOUT_OK && cudaEventRecord(c->ev_t[2], c->s_main) != cudaSuccess) rc = cuda_fail(c, cudaGetLastError(), "seed");
    if (rc == SCOUT_OK) rc = counters_fetch(c);
    if (own) dev_free(c, own, (size_t)slots * 4);
    return rc;
}

}  // namespace scout

using namespace scout;

extern "C" int scout_recompute_bfs(scout_ctx*, int32_t, scout_batch_stats*);
extern "C" int scout_recompute_cc(scout_ctx*, scout_batch_stats*);

extern "C" {

int scout_seed(scout_ctx* c, int problem, int32_t source, scout_batch_stats* st) {
    if (!c) return SCOUT_E_INVALID;
    if (!c->sealed) return c->fail(SCOUT_E_STATE, "graph not sealed");
    if (problem < SCOUT_MIS || problem > SCOUT_CC) return c->fail(SCOUT_E_INVALID, "unknown problem");
    cudaSetDevice(c->device);
    scout_batch_stats local;
    if (!st) st = &local;
    std::memset(st, 0, sizeof(*st));
    int32_t** slot = problem == SCOUT_MIS ? &c->mis : problem == SCOUT_COLORING ? &c->color
                     : problem == SCOUT_BFS ? &c->level : &c->label;
    if (!*slot) {
        SCOUT_RC(dev_alloc(c, (void**)slot, (size_t)c->n * 4, "solution state"));
        // a fresh state: BFS unreached everywhere, CC every vertex its own label (the full
        // traversal and recompute overwrite every entry)
        SCOUT_CU(c, cudaMemsetAsync(*slot, problem == SCOUT_BFS ? 0xff : 0, (size_t)c->n * 4, c->s_main));
    }
    if (problem == SCOUT_BFS) {
        if (source < 0 || source >= c->n) return c->fail(SCOUT_E_INVALID, "source out of range");
        return scout_recompute_bfs(c, source, st);
    }
    if (problem == SCOUT_CC) return scout_recompute_cc(c, st);
    SCOUT_RC(lists_ensure(c));
    SCOUT_RC(batch_begin(c));
    SeedParams p;
    p.g = dgraph(c);
    p.out = *slot;
    p.mode = problem == SCOUT_MIS ? 0 : 1;
    p.wl[0] = c->d_list[0];
    p.wl[1] = c->d_list[1];
    p.ctr = c->d_ctr;
    p.bar = c->d_bar;
    p.pre = p.open = p.nwait = p.waiters = nullptr;
    p.off = nullptr;
    c->last_problem = problem;
    SCOUT_CU(c, cudaEventRecord(c->ev_t[1], c->s_main));
    void* args[] = {&p};
    SCOUT_RC(coop_launch(c, (const void*)k_seed_rounds, SEED_THREADS, args, 0));
    // Whether vertices are open is read back before the lists are prepared, a wait of 20 us; on a small
    // graph the lists of a colouring, which nearly always needs them, follow without it (with
    // nothing open they take about as long there).
    bool lists = true;
    if (p.mode == 0 || c->n >= SEED_ASK) {
        SCOUT_CU(c, cudaEventRecord(c->ev_t[2], c->s_main));
        SCOUT_RC(counters_fetch(c));
        lists = c->h_ctr->affected > 0;
    }
    if (lists) {
        SCOUT_CU(c, cudaMemsetAsync(c->d_ctr->list_count, 0, sizeof(c->d_ctr->list_count), c->s_main));
        SCOUT_RC(seed_lists(c, p));
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev_t[1], c->ev_t[2]);
    st->ms_repair = ms;
    st->rounds = c->h_ctr->rounds;
    st->hbm_bytes = c->h_ctr->hbm_bytes;
    st->changed = c->n;
    c->last_changed = 0;   // nothing to commit: download the state
    return SCOUT_OK;
}

}  // extern "C"
