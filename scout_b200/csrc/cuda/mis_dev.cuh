// mis_dev.cuh -- device code of the mis repair kernel (k_mis): its parameters, helpers and
// body, shared by mis.cu (the kernel and its host launcher) and union.cu (the one persistent
// kernel that runs several problems' repairs of a round).
#pragma once

#include "ctx.cuh"

namespace scout {

struct MisParams {
    DGraph g;
    int32_t* mis;
    const unsigned long long* hkeys;
    int B;
    int32_t* list[2];      // undecided candidates (n each)
    int32_t* removed;      // dropped vertices (n)
    int32_t* touched;
    int32_t* st_cand;      // == epoch: candidate this batch
    int32_t* st_done;      // == epoch: decided this batch
    int32_t* st_touch;
    int32_t epoch;
    int32_t* pairs;        // commit_pairs
    DevCounters* ctr;
    GridBar* bar;
};

constexpr int MIS_ITEMS = 4;   // candidates a warp decides at a time, half-edits a thread reads at a time

__device__ __forceinline__ void mis_touch(const MisParams& p, bool pred, int32_t v) {
    bool nt = false;
    if (pred) nt = atomicExch(&p.st_touch[v], p.epoch) != p.epoch;
    int at = warp_append(nt, &p.ctr->changed);
    if (nt) p.touched[at] = v;
}

// Warp-cooperative: lanes with pred add v to the candidate list once per batch.
__device__ __forceinline__ void mis_candidate(const MisParams& p, bool pred, int32_t v) {
    bool first = false;
    if (pred) first = atomicExch(&p.st_cand[v], p.epoch) != p.epoch;
    int at = warp_append(first, &p.ctr->list_count[0]);
    if (first) p.list[0][at] = v;
}

__device__ __forceinline__ void mis_body(const MisParams& p) {
    const int W = gwarp_count(), wid = gwarp_id();
    const int64_t tid = gthread_id();
    const int64_t T = (int64_t)gridDim.x * blockDim.x;
    const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
    const int nh = ld_volatile(&p.ctr->n_half);
    long long bytes = 0;
    int rounds = 0;

    if (update_failed(p.bar)) return;
    // ---- 1: conflicts of inserted edges, evaluated on the pre-batch set ----------------
    for (int64_t b = tid - (tid & (WARP - 1)); b < nh; b += MIS_ITEMS * T) {
        int32_t x[MIS_ITEMS], y[MIS_ITEMS];
        bool mx[MIS_ITEMS], my[MIS_ITEMS];
#pragma unroll
        for (int u = 0; u < MIS_ITEMS; u++) {
            const int64_t k = b + u * T + lane_id();
            const unsigned long long key = k < nh ? p.hkeys[k] : ~0ull;
            x[u] = (int32_t)(key >> (p.B + 1));
            y[u] = (int32_t)(key & ((1ull << p.B) - 1));
            if (k >= nh || ((key >> p.B) & 1ull) || x[u] >= y[u]) x[u] = -1;   // insertions, once each
        }
#pragma unroll
        for (int u = 0; u < MIS_ITEMS; u++) {
            mx[u] = x[u] >= 0 && ld_volatile(p.mis + x[u]) != 0;
            my[u] = x[u] >= 0 && ld_volatile(p.mis + y[u]) != 0;
        }
#pragma unroll
        for (int u = 0; u < MIS_ITEMS; u++) {
            bool drop = false;
            if (mx[u] && my[u]) {
                drop = atomicExch(&p.st_done[y[u]], p.epoch) != p.epoch;
                atomicAdd(&p.ctr->conflicts, 1);
            }
            const int at = warp_append(drop, &p.ctr->list_count[2]);
            if (drop) p.removed[at] = y[u];
        }
    }
    if (!grid_sync(p.bar, 20)) return;
    // ---- 2: drop them; candidates = dropped vertices, their neighbours, deletion endpoints ---
    const int nrem = ld_volatile(&p.ctr->list_count[2]);
    for (int64_t b = tid - (tid & (WARP - 1)); b < nrem; b += T) {
        int64_t i = b + lane_id();
        bool ok = i < nrem;
        int32_t r = ok ? p.removed[i] : 0;
        if (ok) p.mis[r] = 0;
        mis_touch(p, ok, r);
    }
    if (!grid_sync(p.bar, 21)) return;
    for (int i = wid; i < nrem; i += W) {
        int32_t r = p.removed[i];
        Row rr = p.g.row[r];
        const int32_t* rw = p.g.pool + rr.start;
        mis_candidate(p, lane_id() == 0, r);
        for (int b0 = 0; b0 < rr.len; b0 += WARP) {
            int k = b0 + (int)lane_id();
            mis_candidate(p, k < rr.len, k < rr.len ? rw[k] : 0);
        }
        if (lane_id() == 0) bytes += 4LL * rr.len + 16;
    }
    for (int64_t b = tid - (tid & (WARP - 1)); b < nh; b += MIS_ITEMS * T) {
        int32_t x[MIS_ITEMS];
        bool first[MIS_ITEMS];
#pragma unroll
        for (int u = 0; u < MIS_ITEMS; u++) {
            const int64_t k = b + u * T + lane_id();
            const unsigned long long key = k < nh ? p.hkeys[k] >> p.B : 0ull;
            // (sorted: a vertex's deletions are consecutive, the first one speaks for them)
            const bool del = (key & 1ull) && (k == 0 || (p.hkeys[k - 1] >> p.B) != key);
            x[u] = del ? (int32_t)(key >> 1) : -1;
        }
#pragma unroll
        for (int u = 0; u < MIS_ITEMS; u++) first[u] = x[u] >= 0 && atomicExch(&p.st_cand[x[u]], p.epoch) != p.epoch;
#pragma unroll
        for (int u = 0; u < MIS_ITEMS; u++) {
            const int at = warp_append(first[u], &p.ctr->list_count[0]);
            if (first[u]) p.list[0][at] = x[u];
        }
    }
    if (!grid_sync(p.bar, 22)) return;
    if (leader) p.ctr->affected = ld_volatile(&p.ctr->list_count[0]);
    // ---- 3: id-priority rounds --------------------------------------------------------------
    int cur = 0;
    while (true) {
        const int cnt = ld_volatile(&p.ctr->list_count[cur]);
        if (cnt == 0) break;
        const int nxt = cur ^ 1;
        if (leader) p.ctr->list_count[nxt] = 0;
        if (!grid_sync(p.bar, 23)) return;
        // st_done: == epoch marks a vertex dropped in step 1 (still undecided); DONE_IN / DONE_OUT
        // a vertex decided in these rounds. The decision and its value live in one word, so a
        // neighbour read once is either undecided or decided with its final membership (a
        // separate flag read after the set entry could pair a new flag with a stale entry).
        const int32_t DONE_IN = p.epoch + 0x40000000, DONE_OUT = p.epoch + 0x20000000;
        // A set entry is one read per neighbour and settles most candidates: an entry of 1 is final
        // here. Only if a row shows none are the decision words and candidate marks read. A warp
        // reads the last 32 entries of up to MIS_ITEMS candidates side by side, longer rows then one
        // by one towards the front. What bounds it: chains of dependent reads, 22 candidates per warp
        // one after the other (three reads per neighbour) when 300,007 edits on 10^6 vertices leave
        // 104,000 of them: that repair took 165 us, so 95 (108 with eight at a time).
        const int per = min(MIS_ITEMS, max(1, (cnt + W - 1) / W));
        for (int i0 = wid * per; i0 < cnt; i0 += W * per) {
            int32_t cv[MIS_ITEMS], w[MIS_ITEMS];
            Row r[MIS_ITEMS];
            bool in[MIS_ITEMS], m[MIS_ITEMS];
#pragma unroll
            for (int u = 0; u < MIS_ITEMS; u++) cv[u] = u < per && i0 + u < cnt ? p.list[cur][i0 + u] : -1;
#pragma unroll
            for (int u = 0; u < MIS_ITEMS; u++) {
                r[u] = cv[u] >= 0 ? p.g.row[cv[u]] : Row{0, 0, 0};
                in[u] = cv[u] >= 0 && ld_volatile(p.mis + cv[u]) != 0;
            }
#pragma unroll
            for (int u = 0; u < MIS_ITEMS; u++) {
                const int k = r[u].len - 1 - (int)lane_id();
                w[u] = !in[u] && k >= 0 ? p.g.pool[r[u].start + k] : -1;
            }
#pragma unroll
            for (int u = 0; u < MIS_ITEMS; u++) m[u] = w[u] >= 0 && ld_volatile(p.mis + w[u]) != 0;
#pragma unroll
            for (int u = 0; u < MIS_ITEMS; u++) {
                if (cv[u] < 0) continue;   // uniform per warp
                const int32_t c = cv[u];
                const bool was_in = in[u];
                bool member_nb = __any_sync(0xffffffffu, m[u]), lower_undecided = false;
                if (w[u] >= 0) bytes += 8;
                if (!was_in && !member_nb) {
                    int32_t x = w[u];
                    for (int k = r[u].len - 1 - (int)lane_id();;) {
                        bool mm = false, l = false;
                        if (x >= 0) {
                            const int32_t sd = ld_volatile(p.st_done + x);
                            mm = sd == DONE_IN;
                            l = !mm && sd != DONE_OUT && x < c && ld_volatile(p.st_cand + x) == p.epoch;
                        }
                        member_nb = __any_sync(0xffffffffu, mm);
                        lower_undecided = lower_undecided || __any_sync(0xffffffffu, l);
                        k -= WARP;
                        if (member_nb || k + (int)lane_id() < 0) break;
                        x = k >= 0 ? p.g.pool[r[u].start + k] : -1;
                        member_nb = __any_sync(0xffffffffu, x >= 0 && ld_volatile(p.mis + x) != 0);
                        if (x >= 0) bytes += 8;
                        if (member_nb) break;
                    }
                }
                const bool joined = !was_in && !member_nb && !lower_undecided;
                if (lane_id() == 0) {
                    if (was_in) {
                        p.st_done[c] = DONE_IN;    // kept
                    } else if (member_nb) {
                        p.st_done[c] = DONE_OUT;
                    } else if (joined) {
                        p.mis[c] = 1;
                        p.st_done[c] = DONE_IN;
                    } else {
                        p.list[nxt][atomicAdd(&p.ctr->list_count[nxt], 1)] = c;   // wait
                    }
                }
                mis_touch(p, lane_id() == 0 && joined, c);
            }
        }
        rounds++;
        if (!grid_sync(p.bar, 24)) return;
        cur = nxt;
    }
    commit_pairs(p.touched, p.mis, p.ctr, p.pairs);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
    if (lane_id() == 0) atomicAdd((unsigned long long*)&p.ctr->hbm_bytes, (unsigned long long)bytes);
    if (leader) p.ctr->rounds = rounds;
}
// host: the kernel parameters of the context's current batch (mis.cu)
int mis_params(scout_ctx* c, MisParams* out);

}  // namespace scout
