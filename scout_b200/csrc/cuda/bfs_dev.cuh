// bfs_dev.cuh -- device code of the bfs repair kernel (k_bfs): its parameters, helpers and
// body, shared by bfs.cu (the kernel and its host launcher) and union.cu (the one persistent
// kernel that runs several problems' repairs of a round).
#pragma once

#include "ctx.cuh"

namespace scout {

constexpr int BFS_Q_REST = 9;    // invalidation: the other chunks of long candidates (buffers 0, 1, 2)
constexpr int BFS_Q_SEED = 5;    // queue of the rows that seed invalidated vertices (buffer 2)
constexpr int BFS_Q_RELAX = 6;   // first of the relax rounds' three queues (buffers 0, 1, 2)
constexpr int CHECK_ITEMS = 8;   // candidates a warp checks at a time (invalidation)
constexpr int PSCAN = 4;   // row entries per lane and step in the seed scan

struct BfsParams {
    DGraph g;
    int32_t* level;
    int32_t source;
    const unsigned long long* hkeys;
    int B;
    unsigned long long* q[3];
    int64_t qcap;
    int32_t* inval;
    int32_t* touched;
    int32_t* st_inval;
    int32_t* st_touch;
    uint32_t* st_q;
    int32_t* found;     // == tag: a chunk of a long candidate found a valid parent this round
    int32_t epoch;
    uint32_t qtag0;
    DevCounters* ctr;
    GridBar* bar;
    int mode;             // 0 incremental, 1 top-down traversal, 2 direction-optimizing traversal
    const int* mode_dev;  // when set, the mode is read here (written on the device by the scheduler)
    int32_t* lv_new;      // n: levels of a full traversal before they are diffed into `level`
    long long nnz_pre;    // directed entries before this batch (the batch's delta is in ctr)
    int chunk, chunk_log2;    // row entries per queue item (a power of two, 256 .. 8192)
    const int32_t* sources;   // when nsrc > 0: every listed vertex is a level-0 root (a union of
    int nsrc;                 // disjoint graphs, one source each); else `source` alone
    int32_t* pairs;           // commit_pairs
    int max_share;            // most warps that share one queue item (lanes_per_vertex / 32)
};

__device__ __forceinline__ int32_t ld_level(const int32_t* p) { return ld_volatile(p); }
// A level that no one writes before the next grid barrier: read through L1 (rows repeat the same
// hubs), where a volatile read always goes to L2.
__device__ __forceinline__ int32_t ld_fixed(const int32_t* p) { return *p; }

// Warp-cooperative push (all 32 lanes call): lanes with `pred` push vertex y into queue qn
// once per round (tag), split into chunk-sized items; first touches of the batch are
// appended to the touched list.
__device__ __forceinline__ void push_vertex(const BfsParams& p, bool pred, int32_t y, int qi, uint32_t tag,
                                            bool chunked, bool touch) {
    bool first = false;
    if (pred) first = atomicExch(&p.st_q[y], tag) != tag;
    if (touch) {
        bool nt = false;
        if (pred) nt = atomicExch(&p.st_touch[y], p.epoch) != p.epoch;
        int ti = warp_append(nt, &p.ctr->changed);
        if (nt) p.touched[ti] = y;
    }
    int nit = 0;
    if (first) {
        if (chunked) {
            int len = p.g.row[y].len;
            nit = max(1, (len + p.chunk - 1) >> p.chunk_log2);   // an empty row still gets its item
        } else {
            nit = 1;
        }
    }
    int incl = warp_incl_scan_i(nit);
    int tot = __shfl_sync(0xffffffffu, incl, WARP - 1);
    if (tot == 0) return;
    int base = 0;
    if (lane_id() == WARP - 1) base = atomicAdd(&p.ctr->q_count[qi], tot);
    base = __shfl_sync(0xffffffffu, base, WARP - 1);
    long long start = (long long)base + incl - nit;
    for (int k = 0; k < nit; k++) {
        long long pos = start + k;
        if (pos < p.qcap) p.q[qi % 3][pos] = ((unsigned long long)k << 32) | (uint32_t)y;
        else atomicExch(&p.ctr->overflow, 1);
    }
}

// push_vertex (one item per vertex, no touch list) of two vertices per lane at once: the dedupe
// atomics of both are in flight together, and one atomicAdd reserves both's items.
__device__ __forceinline__ void push_vertex2(const BfsParams& p, bool pa, int32_t ya, bool pb, int32_t yb, int qi,
                                             uint32_t tag) {
    bool fa = false, fb = false;
    if (pa) fa = atomicExch(&p.st_q[ya], tag) != tag;
    if (pb) fb = atomicExch(&p.st_q[yb], tag) != tag;   // ya == yb: only the first push counts
    const int na = fa, nit = (int)fa + (int)fb;
    const int incl = warp_incl_scan_i(nit);
    const int tot = __shfl_sync(0xffffffffu, incl, WARP - 1);
    if (tot == 0) return;
    int base = 0;
    if (lane_id() == WARP - 1) base = atomicAdd(&p.ctr->q_count[qi], tot);
    base = __shfl_sync(0xffffffffu, base, WARP - 1);
    const long long start = (long long)base + incl - nit;
    if (start + nit > p.qcap) { if (nit) atomicExch(&p.ctr->overflow, 1); return; }
    if (fa) p.q[qi % 3][start] = (uint32_t)ya;
    if (fb) p.q[qi % 3][start + na] = (uint32_t)yb;
}

// Every chunk but the first of row y (`chunks` of them in all) into queue qi; one warp, all lanes.
__device__ __forceinline__ void push_rest(const BfsParams& p, int32_t y, int chunks, int qi) {
    int base = 0;
    if (lane_id() == 0) base = atomicAdd(&p.ctr->q_count[qi], chunks - 1);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (int k = 1 + (int)lane_id(); k < chunks; k += WARP) {
        const long long pos = (long long)base + k - 1;
        if (pos < p.qcap) p.q[qi % 3][pos] = ((unsigned long long)k << 32) | (uint32_t)y;
        else atomicExch(&p.ctr->overflow, 1);
    }
}

// Has one of the entries rw[0, n) a valid parent level (lc - 1)? The warp, 256 entries at a time: a
// chunk is two dependent reads, not sixteen.
static __device__ __forceinline__ bool parent_among(const BfsParams& p, const int32_t* rw, int n, int lc, long long& bytes) {
    constexpr int U = 8;
    for (int b0 = 0; b0 < n; b0 += U * WARP) {
        int32_t w[U];
        int lw[U];
        bool ok = false;
#pragma unroll
        for (int u = 0; u < U; u++) w[u] = b0 + u * WARP + (int)lane_id() < n ? rw[b0 + u * WARP + (int)lane_id()] : -1;
#pragma unroll
        for (int u = 0; u < U; u++) lw[u] = w[u] >= 0 ? ld_fixed(p.level + w[u]) : -2;
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (lw[u] == lc - 1 && w[u] >= 0) ok = ok || ld_volatile(p.st_inval + w[u]) != p.epoch;
            if (w[u] >= 0) bytes += 8;
        }
        if (__any_sync(0xffffffffu, ok)) return true;
    }
    return false;
}

// The children (level lc + 1) among rw[0, n) of an invalidated vertex are queued for a check.
static __device__ __forceinline__ void push_children(const BfsParams& p, const int32_t* rw, int n, int lc, int qi,
                                                     uint32_t tag, long long& bytes) {
    constexpr int U = 4;
    for (int b0 = 0; b0 < n; b0 += U * WARP) {
        int32_t w[U];
        int lw[U];
#pragma unroll
        for (int u = 0; u < U; u++) w[u] = b0 + u * WARP + (int)lane_id() < n ? rw[b0 + u * WARP + (int)lane_id()] : -1;
#pragma unroll
        for (int u = 0; u < U; u++) lw[u] = w[u] >= 0 ? ld_fixed(p.level + w[u]) : -2;
        for (int u = 0; u < U; u++) {
            const bool ch = w[u] >= 0 && lw[u] == lc + 1 && ld_volatile(p.st_inval + w[u]) != p.epoch;
            if (__any_sync(0xffffffffu, ch)) push_vertex(p, ch, w[u], qi, tag, false, false);
        }
    }
    if (lane_id() == 0) bytes += 8LL * max(n, 0);
}

__device__ __forceinline__ int qcount(const BfsParams& p, int qi) {
    int c = ld_volatile(&p.ctr->q_count[qi]);
    return (long long)c > p.qcap ? (int)p.qcap : c;
}

// Work split of a round over `cnt` queue items (each at most `chunk` row entries) among the
// grid's W warps. With at least W / 2 items, a warp takes per = ceil(cnt / W) consecutive
// items per pass (one per lane, at most 32) and expands their entries together. With fewer
// items, g warps share every item (g a power of two with g * cnt <= W and at least 32 entries
// per share), each expanding its own contiguous 1/g of the item's entries: a round of a few
// hub chunks then spreads over the whole grid instead of over a handful of warps.
__device__ __forceinline__ int items_per_warp(int cnt, int W) {
    const int per = (int)(((long long)cnt + W - 1) / W);
    return per < 1 ? 1 : (per > WARP ? WARP : per);
}
__device__ __forceinline__ int warps_per_item(int cnt, int W, int chunk, int max_share) {
    int g = 1;
    while ((long long)g * 2 * cnt <= W && g * 2 * WARP <= chunk && g * 2 <= max_share) g *= 2;
    return g;
}

// Expansion of one item share [b, e) of a row segment starting at s, 32 entries at a time;
// every lane calls it (the pushes are warp-collective). Levels only decrease during the relax
// rounds, so a neighbour whose level (read without an atomic, possibly stale and then larger)
// is already at most lv + 1 needs no atomicMin.
__device__ __forceinline__ void relax_share(const BfsParams& p, long long s, int b, int e, int lv, int nxt,
                                            uint32_t tag) {
    const unsigned cand = (unsigned)(lv + 1);
    for (int k0 = b; k0 < e; k0 += WARP) {
        const int k = k0 + (int)lane_id();
        bool dec = false;
        int32_t y = 0;
        if (k < e) {
            y = p.g.pool[s + k];
            if ((unsigned)ld_level(p.level + y) > cand) dec = atomicMin((unsigned*)(p.level + y), cand) > cand;
        }
        push_vertex(p, dec, y, nxt, tag, true, true);
    }
}

// One relax round over queue `cur` into `nxt` (warp-level load-balanced expansion).
static __device__ void relax_round(const BfsParams& p, int cur, int nxt, uint32_t tag, long long& bytes) {
    const int cnt = qcount(p, cur);
    const int W = gwarp_count();
    if ((long long)cnt * 2 <= W) {
        const int g = warps_per_item(cnt, W, p.chunk, p.max_share);
        for (long long wv = gwarp_id(); wv < (long long)cnt * g; wv += W) {
            const int item = (int)(wv / g), part = (int)(wv % g);
            const unsigned long long it = p.q[cur % 3][item];
            const int32_t v = (int32_t)(it & 0xffffffffu);
            const int chunk = (int)(it >> 32);
            const Row r = p.g.row[v];
            const int lv = ld_level(p.level + v);
            const int len = lv < 0 ? 0 : max(0, min(p.chunk, r.len - (chunk << p.chunk_log2)));
            const int b = (int)((long long)len * part / g), e = (int)((long long)len * (part + 1) / g);
            if (lane_id() == 0) bytes += 8LL * (e - b) + (part == 0 ? 24 : 0);
            relax_share(p, r.start + ((long long)chunk << p.chunk_log2), b, e, lv, nxt, tag);
        }
        return;
    }
    const int per = items_per_warp(cnt, W);
    for (long long gbase = (long long)gwarp_id() * per; gbase < cnt; gbase += (long long)W * per) {
        long long idx = gbase + lane_id();
        bool valid = (int)lane_id() < per && idx < cnt;
        unsigned long long item = valid ? p.q[cur % 3][idx] : 0ull;
        int32_t v = (int32_t)(item & 0xffffffffu);
        int chunk = (int)(item >> 32);
        long long s = 0;
        int len = 0, lv = -1;
        if (valid) {
            Row r = p.g.row[v];
            s = r.start + ((long long)chunk << p.chunk_log2);
            len = min(p.chunk, r.len - (chunk << p.chunk_log2));
            if (len < 0) len = 0;
            lv = ld_level(p.level + v);
            if (lv < 0) len = 0;
        }
        int incl = warp_incl_scan_i(len);
        int total = __shfl_sync(0xffffffffu, incl, WARP - 1);
        int excl = incl - len;
        bytes += (long long)len * 8 + (valid ? 24 : 0);
        for (int e0 = 0; e0 < total; e0 += WARP) {
            int e = e0 + (int)lane_id();
            int lo = 0, hi = WARP - 1;
#pragma unroll
            for (int it = 0; it < 5; it++) {
                int mid = (lo + hi + 1) >> 1;
                int em = __shfl_sync(0xffffffffu, excl, mid);
                if (em <= e) lo = mid; else hi = mid - 1;
            }
            long long so = __shfl_sync(0xffffffffu, s, lo);
            int eo = __shfl_sync(0xffffffffu, excl, lo);
            int lo_lv = __shfl_sync(0xffffffffu, lv, lo);
            bool dec = false;
            int32_t y = 0;
            if (e < total) {
                y = p.g.pool[so + (e - eo)];
                unsigned cand = (unsigned)(lo_lv + 1);
                if ((unsigned)ld_level(p.level + y) > cand) dec = atomicMin((unsigned*)(p.level + y), cand) > cand;
            }
            push_vertex(p, dec, y, nxt, tag, true, true);
        }
    }
}

// ---- full traversals (modes 1 and 2) ---------------------------------------------------------
// Frontier bookkeeping rotates over three slots like the queues: list_count[s] holds the
// vertices and aux64[s] the adjacency entries of the frontier in q[s].
constexpr int DO_ALPHA = 14;   // top-down -> bottom-up once frontier entries > unexplored / 14
constexpr int DO_BETA = 24;    // bottom-up -> top-down once the frontier has < n / 24 vertices

// Warp-cooperative push of newly levelled vertices (each pushed by exactly one lane, so no
// dedupe tag is needed): chunk items into q[qi], vertex and entry counts into slot qi.
__device__ __forceinline__ void push_new(const BfsParams& p, bool pred, int32_t y, int len, int qi) {
    int nit = pred ? max(1, (len + p.chunk - 1) >> p.chunk_log2) : 0;
    int incl = warp_incl_scan_i(nit);
    int tot = __shfl_sync(0xffffffffu, incl, WARP - 1);
    if (tot == 0) return;
    long long deg = pred ? len : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) deg += __shfl_xor_sync(0xffffffffu, deg, o);
    const int nv = __popc(__ballot_sync(0xffffffffu, pred));
    int base = 0;
    if (lane_id() == WARP - 1) {
        base = atomicAdd(&p.ctr->q_count[qi], tot);
        atomicAdd(&p.ctr->list_count[qi], nv);
        atomicAdd((unsigned long long*)&p.ctr->aux64[qi], (unsigned long long)deg);
    }
    base = __shfl_sync(0xffffffffu, base, WARP - 1);
    long long start = (long long)base + incl - nit;
    for (int k = 0; k < nit; k++) {
        long long pos = start + k;
        if (pos < p.qcap) p.q[qi % 3][pos] = ((unsigned long long)k << 32) | (uint32_t)y;
        else atomicExch(&p.ctr->overflow, 1);
    }
}

// Top-down step: every entry of every frontier item claims its unlevelled neighbours (the
// same work split as the relax rounds).
__device__ __forceinline__ void td_share(const BfsParams& p, int32_t* lv, long long s, int b, int e, int d, int nxt) {
    for (int k0 = b; k0 < e; k0 += WARP) {
        const int k = k0 + (int)lane_id();
        bool got = false;
        int32_t y = 0;
        int ylen = 0;
        if (k < e) {
            y = p.g.pool[s + k];
            if (ld_volatile(lv + y) < 0) got = atomicCAS(lv + y, -1, d + 1) == -1;
            if (got) ylen = p.g.row[y].len;
        }
        push_new(p, got, y, ylen, nxt);
    }
}

static __device__ void td_step(const BfsParams& p, int32_t* lv, int cur, int nxt, int d, long long& bytes) {
    const int cnt = qcount(p, cur);
    const int W = gwarp_count();
    if ((long long)cnt * 2 <= W) {
        const int g = warps_per_item(cnt, W, p.chunk, p.max_share);
        for (long long wv = gwarp_id(); wv < (long long)cnt * g; wv += W) {
            const int item = (int)(wv / g), part = (int)(wv % g);
            const unsigned long long it = p.q[cur % 3][item];
            const int32_t v = (int32_t)(it & 0xffffffffu);
            const int chunk = (int)(it >> 32);
            const Row r = p.g.row[v];
            const int len = max(0, min(p.chunk, r.len - (chunk << p.chunk_log2)));
            const int b = (int)((long long)len * part / g), e = (int)((long long)len * (part + 1) / g);
            if (lane_id() == 0) bytes += 8LL * (e - b) + (part == 0 ? 24 : 0);
            td_share(p, lv, r.start + ((long long)chunk << p.chunk_log2), b, e, d, nxt);
        }
        return;
    }
    const int per = items_per_warp(cnt, W);
    for (long long gbase = (long long)gwarp_id() * per; gbase < cnt; gbase += (long long)W * per) {
        long long idx = gbase + lane_id();
        bool valid = (int)lane_id() < per && idx < cnt;
        unsigned long long item = valid ? p.q[cur % 3][idx] : 0ull;
        int32_t v = (int32_t)(item & 0xffffffffu);
        int chunk = (int)(item >> 32);
        long long s = 0;
        int len = 0;
        if (valid) {
            Row r = p.g.row[v];
            s = r.start + ((long long)chunk << p.chunk_log2);
            len = max(0, min(p.chunk, r.len - (chunk << p.chunk_log2)));
        }
        int incl = warp_incl_scan_i(len);
        int total = __shfl_sync(0xffffffffu, incl, WARP - 1);
        int excl = incl - len;
        bytes += (long long)len * 8 + (valid ? 24 : 0);
        for (int e0 = 0; e0 < total; e0 += WARP) {
            int e = e0 + (int)lane_id();
            int lo = 0, hi = WARP - 1;
#pragma unroll
            for (int it = 0; it < 5; it++) {
                int mid = (lo + hi + 1) >> 1;
                int em = __shfl_sync(0xffffffffu, excl, mid);
                if (em <= e) lo = mid; else hi = mid - 1;
            }
            long long so = __shfl_sync(0xffffffffu, s, lo);
            int eo = __shfl_sync(0xffffffffu, excl, lo);
            bool got = false;
            int32_t y = 0;
            int ylen = 0;
            if (e < total) {
                y = p.g.pool[so + (e - eo)];
                if (ld_volatile(lv + y) < 0) got = atomicCAS(lv + y, -1, d + 1) == -1;
                if (got) ylen = p.g.row[y].len;
            }
            push_new(p, got, y, ylen, nxt);
        }
    }
}

// Bottom-up step: every unlevelled vertex looks for a neighbour on level d and stops at the
// first one. Short rows are scanned by their own lane, longer ones by the whole warp.
static __device__ void bu_step(const BfsParams& p, int32_t* lv, int nxt, int d, long long& bytes) {
    const int64_t n = p.g.n;
    const int W = gwarp_count();
    for (int64_t base = (int64_t)gwarp_id() * WARP; base < n; base += (int64_t)W * WARP) {
        const int64_t v = base + lane_id();
        bool un = v < n && ld_volatile(lv + v) < 0;
        Row r{0, 0, 0};
        if (un) r = p.g.row[v];
        bool found = false;
        const bool big = un && r.len > WARP;
        long long scanned = un ? 4 + 16 : (v < n ? 4 : 0);
        if (un && !big) {
            for (int k = 0; k < r.len; k++) {
                scanned += 8;
                if (ld_volatile(lv + p.g.pool[r.start + k]) == d) { found = true; break; }
            }
        }
        unsigned bigm = __ballot_sync(0xffffffffu, big);
        while (bigm) {
            const int j = __ffs(bigm) - 1;
            bigm &= bigm - 1;
            const long long js = __shfl_sync(0xffffffffu, r.start, j);
            const int jl = __shfl_sync(0xffffffffu, r.len, j);
            bool hit = false;
            for (int b0 = 0; b0 < jl && !hit; b0 += WARP) {
                int k = b0 + (int)lane_id();
                bool ok = k < jl && ld_volatile(lv + p.g.pool[js + k]) == d;
                if (k < jl) scanned += 8;
                hit = __any_sync(0xffffffffu, ok);
            }
            if ((int)lane_id() == j) found = hit;
        }
        if (found) lv[v] = d + 1;
        bytes += scanned;
        push_new(p, found, (int32_t)v, found ? r.len : 0, nxt);
    }
}

// Full traversal into lv_new, then the diff into level. Returns false when a barrier failed.
static __device__ bool full_bfs(const BfsParams& p, int mode, long long& bytes, int& rounds) {
    int32_t* lv = p.lv_new;
    const int64_t n = p.g.n;
    const int64_t tid = lthread_id();
    const int64_t T = (int64_t)gridDim.x * blockDim.x;
    const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
    for (int64_t v = tid; v < n; v += T) lv[v] = -1;
    if (tid == 0) bytes += 4LL * n;
    if (!grid_sync(p.bar, 22)) return false;
    if (leader) {
        const int ns = p.nsrc > 0 ? p.nsrc : 1;
        int items = 0;
        long long deg = 0;
        for (int i = 0; i < ns; i++) {
            const int32_t s = p.nsrc > 0 ? p.sources[i] : p.source;
            lv[s] = 0;
            const int len = p.g.row[s].len;
            const int nit = max(1, (len + p.chunk - 1) >> p.chunk_log2);
            for (int k = 0; k < nit && items + k < p.qcap; k++)
                p.q[0][items + k] = ((unsigned long long)k << 32) | (uint32_t)s;
            items += nit;
            deg += len;
        }
        if (items > p.qcap) { p.ctr->overflow = 1; items = (int)p.qcap; }
        p.ctr->q_count[0] = items;
        p.ctr->list_count[0] = ns;
        p.ctr->aux64[0] = deg;
        p.ctr->q_count[1] = p.ctr->list_count[1] = 0;
        p.ctr->q_count[2] = p.ctr->list_count[2] = 0;
        p.ctr->aux64[1] = p.ctr->aux64[2] = 0;
    }
    if (!grid_sync(p.bar, 20)) return false;
    const long long total = p.nnz_pre + ld_volatile(&p.ctr->nnz_delta);
    long long visited = 0;
    bool bottom_up = false;
    int cur = 0;
    for (int d = 0;; d++) {
        const int nf = ld_volatile(&p.ctr->list_count[cur]);
        if (nf == 0) break;
        const long long mf = ld_volatile(&p.ctr->aux64[cur]);
        visited += mf;
        if (mode == 2) {
            if (!bottom_up && mf > (total - visited) / DO_ALPHA) bottom_up = true;
            else if (bottom_up && (long long)nf * DO_BETA < n) bottom_up = false;
        }
        const int nxt = (cur + 1) % 3, zer = (cur + 2) % 3;
        if (leader) { p.ctr->q_count[zer] = 0; p.ctr->list_count[zer] = 0; p.ctr->aux64[zer] = 0; }
        if (bottom_up) bu_step(p, lv, nxt, d, bytes);
        else td_step(p, lv, cur, nxt, d, bytes);
        rounds++;
        if (!grid_sync(p.bar, 21)) return false;
        cur = nxt;
    }
    // diff: store and list the levels that changed
    for (int64_t b = tid - (tid & (WARP - 1)); b < n; b += T) {
        const int64_t v = b + lane_id();
        bool ch = false;
        int32_t nv = 0;
        if (v < n) {
            nv = lv[v];
            ch = nv != p.level[v];
            if (ch) p.level[v] = nv;
        }
        int ti = warp_append(ch, &p.ctr->changed);
        if (ch) p.touched[ti] = (int32_t)v;
    }
    if (tid == 0) bytes += 12LL * n;
    return true;
}

__device__ __forceinline__ void bfs_body(const BfsParams& p) {
    const int W = gwarp_count();
    const int wid = gwarp_id();
    const int64_t tid = gthread_id();
    const int64_t T = (int64_t)gridDim.x * blockDim.x;
    const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
    long long bytes = 0;
    int rounds = 0;
    uint32_t tag = p.qtag0;
    int cur = 0;
    if (update_failed(p.bar)) return;
    phase_mark(&p.ctr->phase_ns[0]);

    const int mode = p.mode_dev ? *p.mode_dev : p.mode;
    if (mode != 0) {
        if (!full_bfs(p, mode, bytes, rounds)) return;
        phase_mark(&p.ctr->phase_ns[3]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
        if (lane_id() == 0) atomicAdd((unsigned long long*)&p.ctr->hbm_bytes, (unsigned long long)bytes);
        if (leader) {
            p.ctr->rounds = rounds;
            p.ctr->affected = p.g.n;
            p.ctr->recomputes = 1;
        }
        return;
    }
    {
        // ---- A: invalidation -------------------------------------------------------------
        // A candidate is queued once; a warp looks for a valid parent in its row's first chunk, where
        // nearly every candidate has one. A candidate of a single chunk is settled there (children
        // pushed if it has none). The other chunks of a longer one are queued only if the first
        // holds no parent: after a barrier they are checked side by side (any chunk with one marks
        // found = tag), after another the candidate is decided, and after a third every chunk
        // of an invalidated candidate pushes its children, so a hub's row is spread over many
        // warps. (With every chunk queued at once, a 10^6-edit batch at scale 22 checked 422,000
        // items in the first rounds, most of them of rows whose first chunk settles them.)
        const int nh = ld_volatile(&p.ctr->n_half);
        tag++;
        // two half-edits per thread and step (k and k + T): their loads overlap, and both
        // candidates go out in one warp-collective push
        for (int64_t b = tid - (tid & (WARP - 1)); b < nh; b += 2 * T) {
            bool cand[2] = {false, false};
            int32_t y[2] = {0, 0};
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int64_t k = b + h * T + lane_id();
                if (k < nh) {
                    const unsigned long long key = p.hkeys[k];
                    const int op = (int)((key >> p.B) & 1ull);
                    const int32_t x = (int32_t)(key >> (p.B + 1));
                    y[h] = (int32_t)(key & ((1ull << p.B) - 1));
                    if (op == 1) {
                        const int lx = ld_fixed(p.level + x), ly = ld_fixed(p.level + y[h]);
                        cand[h] = lx >= 0 && ly == lx + 1;
                    }
                }
            }
            const int nc = __popc(__ballot_sync(0xffffffffu, cand[0])) + __popc(__ballot_sync(0xffffffffu, cand[1]));
            if (lane_id() == 0 && nc) atomicAdd(&p.ctr->del_eff, nc);   // tree-edge deletions
            push_vertex2(p, cand[0], y[0], cand[1], y[1], 0, tag);
        }
        if (!grid_sync(p.bar, 2)) return;
        cur = 0;
        while (true) {
            const int cnt = qcount(p, cur);
            if (cnt == 0) break;
            const int nxt = (cur + 1) % 3, zer = (cur + 2) % 3;
            const int rest = BFS_Q_REST + zer;   // its items lie in the buffer that is free this round
            if (leader) {
                p.ctr->q_count[zer] = 0;
                p.ctr->q_count[BFS_Q_REST + (zer + 1) % 3] = 0;   // the next round's
                p.ctr->tick[nxt] = 0;
            }
            tag++;
            // A warp takes up to CHECK_ITEMS candidates at a time (fewer while that leaves warps
            // without any): a lane each holds their vertex, row, level and invalidation mark,
            // loaded while the previous candidates are checked; their first entries, and those
            // entries' levels, are in flight together. None of what is loaded ahead changes
            // during this pass: levels are fixed in this phase, and a candidate is queued once
            // per round and invalidated only by its own warp (a long one after the barriers
            // below). What bounds it: the random reads of levels (32 bytes of L2 traffic each). The
            // invalidation of a 10^6-edit batch at scale 22 (174,000 candidates in the first round)
            // took 315 us with a warp per candidate, 32 entries at a time and every chunk of
            // long rows queued; 275 us without the latter; 215 us with eight entries first.
            const int per = min(CHECK_ITEMS, max(1, (cnt + W - 1) / W));
            const int l = (int)lane_id();
            // (the queue holds vertices alone here: chunk 0; -1 marks a lane without one)
            auto load_item = [&](long long i) { return l < per && i + l < cnt ? (int32_t)p.q[cur % 3][i + l] : -1; };
            struct Cand { Row r; int lc, si; };
            auto load_cand = [&](int32_t c) {
                Cand d{Row{0, 0, 0}, 0, 0};
                if (c >= 0) {
                    d.r = p.g.row[c];
                    d.lc = ld_fixed(p.level + c);
                    d.si = ld_volatile(p.st_inval + c);
                }
                return d;
            };
            // a candidate without a valid parent in its first chunk (the warp, all lanes)
            auto invalidate = [&](int32_t c, const Row& r, int lc) {
                if (r.len > p.chunk) {
                    push_rest(p, c, (r.len + p.chunk - 1) >> p.chunk_log2, rest);
                    return;
                }
                if (l == 0) {
                    p.st_inval[c] = p.epoch;
                    int at = atomicAdd(&p.ctr->list_count[0], 1);
                    p.inval[at] = c;
                }
                __syncwarp();
                push_children(p, p.g.pool + r.start, r.len, lc, nxt, tag, bytes);
                if (l == 0) bytes += 24;
            };
            // No more candidates than warps: a cascade that is bound by the latency of its rounds, one
            // candidate per warp and its whole chunk at once (eight entries first, and turns handed
            // out, made the rounds of a narrow cascade a fifth longer).
            if (per == 1 && wid < cnt) {
                const int32_t c = (int32_t)p.q[cur % 3][wid];
                const Cand d = load_cand(c);
                if (c != p.source && d.lc > 0 && d.si != p.epoch &&
                    !parent_among(p, p.g.pool + d.r.start, min(p.chunk, d.r.len), d.lc, bytes))
                    invalidate(c, d.r, d.lc);
            }
            // the first two turns of every warp are fixed, the rest handed out (rows take unequal time)
            long long i = per == 1 ? cnt : (long long)wid * per, i_n = i + (long long)W * per;
            int32_t it_n = load_item(i);
            Cand cd_n = load_cand(it_n);
            int32_t it_nn = load_item(i_n);
            while (i < cnt) {
                int tk = 0;
                if (l == 0) tk = atomicAdd(&p.ctr->tick[cur], 1);
                const int32_t it_c = it_n;
                const Cand cd = cd_n;
                it_n = it_nn;   // arrived during the previous candidates' waits
                cd_n = load_cand(it_n);
                const bool live = it_c >= 0 && it_c != p.source && cd.lc > 0 && cd.si != p.epoch;
                const int clen = live ? min(p.chunk, cd.r.len) : 0;
                // the first eight entries of every candidate, eight lanes each: nearly all have a
                // parent there, and the random reads of levels are what this pass costs
                unsigned none = __ballot_sync(0xffffffffu, live);   // without a parent so far
                {
                    int32_t w[CHECK_ITEMS / 4];
                    int lw[CHECK_ITEMS / 4];
#pragma unroll
                    for (int h = 0; h < CHECK_ITEMS / 4; h++) {
                        const int u = 4 * h + (l >> 3);
                        const long long st = __shfl_sync(0xffffffffu, cd.r.start, u);
                        const int len = __shfl_sync(0xffffffffu, clen, u);
                        w[h] = (l & 7) < len ? p.g.pool[st + (l & 7)] : -1;
                    }
#pragma unroll
                    for (int h = 0; h < CHECK_ITEMS / 4; h++) lw[h] = w[h] >= 0 ? ld_fixed(p.level + w[h]) : -2;
#pragma unroll
                    for (int h = 0; h < CHECK_ITEMS / 4; h++) {
                        const int lc = __shfl_sync(0xffffffffu, cd.lc, 4 * h + (l >> 3));
                        const bool at = w[h] >= 0 && lw[h] == lc - 1;
                        const unsigned m = __ballot_sync(0xffffffffu, at), group = 0xffu << (l & 24);
                        // the first of a candidate's parents is checked (another, below, if it is invalid)
                        const bool ok = at && !(m & group & ((1u << l) - 1)) && ld_volatile(p.st_inval + w[h]) != p.epoch;
                        const unsigned f = __ballot_sync(0xffffffffu, ok);
#pragma unroll
                        for (int g = 0; g < 4; g++)
                            if (f & (0xffu << (8 * g))) none &= ~(1u << (4 * h + g));
                        if (w[h] >= 0) bytes += 8;
                    }
                }
                // the others 32 entries per step, until each has a valid parent or no entries left
                unsigned open = none;
                auto load_entries = [&](int u, int b0) {   // (0 entries where there is no candidate)
                    const long long st = __shfl_sync(0xffffffffu, cd.r.start, u);
                    const int len = __shfl_sync(0xffffffffu, clen, u);
                    return ((open >> u) & 1u) && b0 + l < len ? p.g.pool[st + b0 + l] : -1;
                };
                int32_t w[CHECK_ITEMS];
#pragma unroll
                for (int u = 0; u < CHECK_ITEMS; u++) w[u] = load_entries(u, 0);
                for (int b0 = 0; open; b0 += WARP) {
                    int32_t nx[CHECK_ITEMS];   // the next step's, loaded while these are checked
                    int lw[CHECK_ITEMS];
#pragma unroll
                    for (int u = 0; u < CHECK_ITEMS; u++) {
                        lw[u] = w[u] >= 0 ? ld_fixed(p.level + w[u]) : -2;
                        nx[u] = load_entries(u, b0 + WARP);
                    }
                    unsigned hit = 0;
#pragma unroll
                    for (int u = 0; u < CHECK_ITEMS; u++) {
                        const int lc = __shfl_sync(0xffffffffu, cd.lc, u);
                        const bool ok = w[u] >= 0 && lw[u] == lc - 1 && ld_volatile(p.st_inval + w[u]) != p.epoch;
                        if (w[u] >= 0) bytes += 8;
                        if (__any_sync(0xffffffffu, ok)) hit |= 1u << u;
                    }
                    none &= ~hit;
                    open = none & __ballot_sync(0xffffffffu, b0 + WARP < clen);
#pragma unroll
                    for (int u = 0; u < CHECK_ITEMS; u++) w[u] = (open >> u) & 1u ? nx[u] : -1;
                }
                const long long i_nn = ((long long)2 * W + __shfl_sync(0xffffffffu, tk, 0)) * per;
                it_nn = load_item(i_nn);
                i = i_n;
                i_n = i_nn;
                for (; none; none &= none - 1) {
                    const int u = __ffs(none) - 1;
                    const int32_t c = __shfl_sync(0xffffffffu, it_c, u);
                    Row r;
                    r.start = __shfl_sync(0xffffffffu, cd.r.start, u);
                    r.len = __shfl_sync(0xffffffffu, cd.r.len, u);
                    r.cap = 0;
                    invalidate(c, r, __shfl_sync(0xffffffffu, cd.lc, u));
                }
            }
            if (!grid_sync(p.bar, 3)) return;
            const int nrest = qcount(p, rest);
            if (nrest) {
                // long candidates without a parent in their first chunk: the others
                for (int i = wid; i < nrest; i += W) {
                    const unsigned long long item = p.q[rest % 3][i];
                    const int32_t c = (int32_t)(item & 0xffffffffu);
                    const Row r = p.g.row[c];
                    const int lc = ld_fixed(p.level + c);
                    const long long c0 = ((long long)(item >> 32) << p.chunk_log2);
                    const int clen = (int)min((long long)p.chunk, (long long)r.len - c0);
                    const int32_t* rw = p.g.pool + r.start + c0;
                    if (ld_volatile(p.found + c) == (int32_t)tag) continue;   // another chunk has one
                    if (parent_among(p, rw, clen, lc, bytes) && l == 0) p.found[c] = (int32_t)tag;
                }
                if (!grid_sync(p.bar, 10)) return;
                // decide on a candidate's first item here (chunk 1)
                for (int64_t b = tid - (tid & (WARP - 1)); b < nrest; b += T) {
                    const int64_t i = b + lane_id();
                    bool nt = false;
                    int32_t c = 0;
                    if (i < nrest) {
                        const unsigned long long item = p.q[rest % 3][i];
                        c = (int32_t)(item & 0xffffffffu);
                        if ((item >> 32) == 1 && ld_volatile(p.found + c) != (int32_t)tag)
                            nt = atomicExch(&p.st_inval[c], p.epoch) != p.epoch;
                    }
                    int at = warp_append(nt, &p.ctr->list_count[0]);
                    if (nt) p.inval[at] = c;
                }
                if (!grid_sync(p.bar, 8)) return;
                for (int i = wid; i < nrest; i += W) {
                    const unsigned long long item = p.q[rest % 3][i];
                    const int32_t c = (int32_t)(item & 0xffffffffu);
                    if (ld_volatile(p.found + c) == (int32_t)tag || ld_volatile(p.st_inval + c) != p.epoch) continue;
                    const Row r = p.g.row[c];
                    const int lc = ld_fixed(p.level + c);
                    const int chunk = (int)(item >> 32);
                    const long long c0 = chunk == 1 ? 0 : ((long long)chunk << p.chunk_log2);   // chunk 1 with chunk 0
                    const int clen = (int)(min((long long)r.len, (long long)(chunk + 1) << p.chunk_log2) - c0);
                    const int32_t* rw = p.g.pool + r.start + c0;
                    push_children(p, rw, clen, lc, nxt, tag, bytes);
                }
                if (!grid_sync(p.bar, 9)) return;
            }
            rounds++;
            cur = nxt;
        }
        phase_mark(&p.ctr->phase_ns[1]);
        // ---- B: reset and seed --------------------------------------------------------------
        // Every invalidated vertex restarts at +inf and queues its row's chunks in q[2]; each
        // chunk then offers (min level of its valid neighbours) + 1. Inserted edges seed their
        // endpoints. Both push into the relax rounds' first queue. The queues of this phase and of
        // the relax rounds have counters of their own (zero since the batch began), so that no
        // barrier clears the invalidation's; without an invalidated vertex the reset and its
        // barrier fall away.
        const int ninv = ld_volatile(&p.ctr->list_count[0]);
        tag++;
        for (int64_t b = tid - (tid & (WARP - 1)); b < ninv; b += T) {
            int64_t i = b + lane_id();
            bool ok = i < ninv;
            int32_t c = ok ? p.inval[i] : 0;
            bool nt = false;
            if (ok) {
                nt = atomicExch(&p.st_touch[c], p.epoch) != p.epoch;
                p.level[c] = -1;
            }
            int ti = warp_append(nt, &p.ctr->changed);
            if (nt) p.touched[ti] = c;
            push_vertex(p, ok, c, BFS_Q_SEED, tag, true, false);
        }
        if (ninv > 0 && !grid_sync(p.bar, 5)) return;
        tag++;
        // boundary seeds: warp per chunk of an invalidated vertex's row
        const int nseed = ninv > 0 ? qcount(p, BFS_Q_SEED) : 0;
        for (int i = wid; i < nseed; i += W) {
            const unsigned long long item = p.q[BFS_Q_SEED % 3][i];
            const int32_t c = (int32_t)(item & 0xffffffffu);
            const Row r = p.g.row[c];
            const long long c0 = ((long long)(item >> 32) << p.chunk_log2);
            const int clen = (int)min((long long)p.chunk, (long long)r.len - c0);
            const int32_t* rw = p.g.pool + r.start + c0;
            unsigned best = 0xffffffffu;
            for (int b0 = 0; b0 < clen; b0 += PSCAN * WARP) {   // both loads of PSCAN entries in flight
                int32_t w[PSCAN];
#pragma unroll
                for (int u = 0; u < PSCAN; u++) {
                    const int k = b0 + u * WARP + (int)lane_id();
                    w[u] = k < clen ? rw[k] : -1;
                }
#pragma unroll
                for (int u = 0; u < PSCAN; u++) {
                    if (w[u] < 0) continue;
                    const int32_t si = ld_volatile(p.st_inval + w[u]);
                    const int lw = ld_level(p.level + w[u]);
                    if (si != p.epoch && lw >= 0) best = min(best, (unsigned)lw);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
            if (lane_id() == 0) bytes += 8LL * max(clen, 0) + 24;
            bool dec = false;
            if (lane_id() == 0 && best != 0xffffffffu) {
                unsigned cand = best + 1;
                unsigned old = atomicMin((unsigned*)(p.level + c), cand);
                dec = old > cand;
            }
            push_vertex(p, dec, c, BFS_Q_RELAX, tag, true, false);
        }
        // insertion seeds: thread per half-edit
        for (int64_t b = tid - (tid & (WARP - 1)); b < nh; b += T) {
            int64_t k = b + lane_id();
            bool dec = false;
            int32_t y = 0;
            if (k < nh) {
                unsigned long long key = p.hkeys[k];
                int op = (int)((key >> p.B) & 1ull);
                int32_t x = (int32_t)(key >> (p.B + 1));
                y = (int32_t)(key & ((1ull << p.B) - 1));
                if (op == 0) {
                    int lx = ld_level(p.level + x);
                    if (lx >= 0) {
                        unsigned cand = (unsigned)lx + 1;
                        unsigned old = atomicMin((unsigned*)(p.level + y), cand);
                        dec = old > cand;
                    }
                }
            }
            const unsigned md = __ballot_sync(0xffffffffu, dec);   // insertions that lowered a level
            if (lane_id() == 0 && md) atomicAdd(&p.ctr->ins_eff, __popc(md));
            push_vertex(p, dec, y, BFS_Q_RELAX, tag, true, true);
        }
        if (!grid_sync(p.bar, 6)) return;
        cur = BFS_Q_RELAX;
    }
    phase_mark(&p.ctr->phase_ns[2]);
    // ---- C: relax rounds -------------------------------------------------------------------
    while (true) {
        const int cnt = qcount(p, cur);
        if (cnt == 0) break;
        const int nxt = BFS_Q_RELAX + (cur + 1) % 3, zer = BFS_Q_RELAX + (cur + 2) % 3;
        if (leader) p.ctr->q_count[zer] = 0;
        tag++;
        relax_round(p, cur, nxt, tag, bytes);
        rounds++;
        if (!grid_sync(p.bar, 7)) return;
        cur = nxt;
    }
    phase_mark(&p.ctr->phase_ns[3]);
    commit_pairs(p.touched, p.level, p.ctr, p.pairs);
    // ---- counters ----------------------------------------------------------------------------
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
    if (lane_id() == 0) atomicAdd((unsigned long long*)&p.ctr->hbm_bytes, (unsigned long long)bytes);
    if (leader) {
        p.ctr->rounds = rounds;
        p.ctr->affected = p.ctr->changed;
    }
}
// host: the kernel parameters of the context's current batch (bfs.cu)
int bfs_params(scout_ctx* c, int mode, const int* mode_dev, BfsParams* out);

}  // namespace scout
