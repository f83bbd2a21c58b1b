// common.cuh -- shared device infrastructure of the sm_100a engine.
//
//   Row        per-vertex row descriptor in HBM: (start, len) into the element pool; rows
//              are kept sorted ascending so adjacency tests are binary searches.
//   GridBar    bounded grid-wide barrier for the persistent cooperative kernels: every wait
//              is limited by %globaltimer; a timeout sets a sticky error flag that makes all
//              blocks leave, and the host reads it back as SCOUT_E_TIMEOUT.
//   Counters   small device block of per-batch counters (copied back once per batch).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace scout {

constexpr int WARP = 32;
constexpr uint32_t UNREACHED_U = 0xFFFFFFFFu;   // level -1 seen as unsigned: +infinity

struct __align__(16) Row {
    long long start;   // element index in the pool
    int len;           // degree
    int cap;           // reserved elements at start (>= len)
};

// One affected row of a batch's merge: its old version, where the new one goes (the same place
// for a row compacted where it lies), and its half-edits [b, d) insertions, [d, e) deletions.
struct __align__(16) MergeRow {
    long long start, dst;
    int len;
    int b, d, e;
};

// Device-resident graph handle passed by value to kernels.
struct DGraph {
    const Row* row;
    const int32_t* pool;
    int32_t n;
};

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & (WARP - 1); }

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

template <typename T>
__device__ __forceinline__ T ld_volatile(const T* p) { return *(const volatile T*)p; }

// Inclusive warp scan of 64-bit values.
__device__ __forceinline__ long long warp_incl_scan(long long x) {
#pragma unroll
    for (int o = 1; o < WARP; o <<= 1) {
        long long y = __shfl_up_sync(0xffffffffu, x, o);
        if ((int)lane_id() >= o) x += y;
    }
    return x;
}
__device__ __forceinline__ int warp_incl_scan_i(int x) {
#pragma unroll
    for (int o = 1; o < WARP; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if ((int)lane_id() >= o) x += y;
    }
    return x;
}

// The lanes whose low 8 bits of d equal this lane's, by eight ballots.
__device__ __forceinline__ unsigned match_digit(unsigned d) {
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 8; b++) {
        const bool one = (d >> b) & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, one);
        peers &= one ? m : ~m;
    }
    return peers;
}

// Warp-aggregated append: every lane with `pred` gets a distinct slot of `q` through one
// atomicAdd per warp. Returns the slot (or -1); slots beyond cap are not written and the
// caller sees the overflow in the counter.
__device__ __forceinline__ int warp_append(bool pred, int* counter) {
    unsigned m = __ballot_sync(__activemask(), pred);
    if (!m) return -1;
    int leader = __ffs(m) - 1;
    int base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(counter, __popc(m));
    base = __shfl_sync(__activemask(), base, leader);
    if (!pred) return -1;
    return base + __popc(m & ((1u << lane_id()) - 1));
}

// Binary search helpers over sorted int32 spans.
__device__ __forceinline__ long long lower_bound_i32(const int32_t* a, long long n, int32_t x) {
    long long lo = 0, hi = n;
    while (lo < hi) {
        long long mid = (lo + hi) >> 1;
        if (a[mid] < x) lo = mid + 1; else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ long long upper_bound_i32(const int32_t* a, long long n, int32_t x) {
    long long lo = 0, hi = n;
    while (lo < hi) {
        long long mid = (lo + hi) >> 1;
        if (a[mid] <= x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Adjacency test on sorted rows: binary search in the shorter of the two rows.
__device__ __forceinline__ bool dg_adjacent(const DGraph& g, int32_t u, int32_t v) {
    Row ru = g.row[u], rv = g.row[v];
    if (rv.len < ru.len) { Row t = ru; ru = rv; rv = t; int32_t s = u; u = v; v = s; }
    const int32_t* a = g.pool + ru.start;
    long long k = lower_bound_i32(a, ru.len, v);
    return k < ru.len && a[k] == v;
}

// The same with three probes per step: half the dependent reads, for calls that are bound by their
// latency alone.
__device__ __forceinline__ bool dg_adjacent_wide(const DGraph& g, int32_t u, int32_t v) {
    Row ru = g.row[u], rv = g.row[v];
    if (rv.len < ru.len) { Row t = ru; ru = rv; rv = t; int32_t s = u; u = v; v = s; }
    const int32_t* a = g.pool + ru.start;
    int lo = 0, hi = ru.len;
    bool hit = false;
    while (lo < hi) {
        const int n = hi - lo, mid = lo + (n >> 1), q1 = lo + (n >> 2), q3 = mid + (n >> 2);
        const int32_t x1 = a[q1], x2 = a[mid], x3 = a[q3];
        hit = x1 == v || x2 == v || x3 == v;
        if (hit) break;
        if (x1 > v) hi = q1;
        else if (x2 > v) { lo = q1 + 1; hi = mid; }
        else if (x3 > v) { lo = mid + 1; hi = q3; }
        else lo = q3 + 1;
    }
    return hit;
}

// ---------------------------------------------------------------------------------------
// Bounded grid barrier (cooperative launch guarantees co-residency of all blocks).
// `count` only grows within a launch: the k-th barrier is complete once it reaches k * blocks,
// so the last block's own arrival releases the others (no reset and no second counter to bump).
// Every block passes the same sequence of barriers, so a block arriving at barrier k sees
// old in [(k - 1) * blocks, k * blocks). The host zeroes the block before each launch.
// `count` and `err` are the halves of ONE 64-bit word, and a launch touches it by 64-bit
// operations only: an arrival and the poll that sees it order memory between blocks because
// both are strong operations on the same eight bytes (a 32-bit arrival under a 64-bit poll would
// overlap it in part and order nothing).
// ---------------------------------------------------------------------------------------
struct __align__(16) GridBar {
    unsigned int count; // low half of the barrier's word
    int err;            // its high half: 0 ok, bit 0 barrier timeout, bit 1 capacity overflow inside a kernel
    int where;          // tag of the barrier that timed out
    unsigned int pad;
};
static_assert(offsetof(GridBar, count) == 0 && offsetof(GridBar, err) == 4, "one word, count below err");

constexpr uint64_t GRID_WAIT_LIMIT_NS = 4000000000ull;   // 4 s

__device__ __forceinline__ unsigned long long ld_acquire_gpu(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long atom_add_release_gpu(unsigned long long* p, unsigned long long x) {
    unsigned long long old;
    asm volatile("atom.add.release.gpu.global.u64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(x) : "memory");
    return old;
}

// The first error of a launch (true for the thread that set it): every wait ends on it.
__device__ __forceinline__ bool grid_error(GridBar* b, unsigned code) {
    return (atomicOr((unsigned long long*)b, (unsigned long long)code << 32) >> 32) == 0;
}

// What bounds it: the latency of one arrival (a release atomic) and of the poll that sees the
// last one. A poll is one acquire load of {count, err}; the clock is read every 64th poll only.
// On a B200, over 1,000 barriers: 1.32 us with one block of 1,024 threads per SM (148 arrivals),
// 2.14 us with four of 256 threads (592 arrivals); reading the clock and the error flag and
// sleeping on every poll made that 2.47 us (2.00 us with 148 arrivals).
__device__ __forceinline__ bool grid_sync(GridBar* b, int tag = 0) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long* word = (unsigned long long*)b;
        const unsigned nb = gridDim.x;   // (rows of a two-dimensional grid have barriers of their own)
        const unsigned old = (unsigned)atom_add_release_gpu(word, 1ull);
        const unsigned target = (old / nb + 1) * nb;
        uint64_t t0 = 0;
        unsigned long long w;
        for (unsigned it = 1;; it++) {
            w = ld_acquire_gpu(word);
            if ((int)((unsigned)w - target) >= 0 || (w >> 32) != 0) break;
            if ((it & 63u) == 0) {
                const uint64_t t = globaltimer_ns();
                if (t0 == 0) {
                    t0 = t;
                } else if (t - t0 > GRID_WAIT_LIMIT_NS) {
                    if (grid_error(b, 1)) b->where = tag;
                    w |= 1ull << 32;
                    break;
                }
            }
        }
        s_ok = (w >> 32) == 0;
    }
    __syncthreads();
    return s_ok != 0;
}

// A batch has two barriers side by side: the update kernel's, then the repair kernel's. The
// repair (given its own) does not start on a store whose update gave up.
__device__ __forceinline__ bool update_failed(const GridBar* repair_bar) { return ld_volatile(&(repair_bar - 1)->err) != 0; }


// Phase timestamp written by one thread right after a grid barrier (profiling aid).
__device__ __forceinline__ void phase_mark(unsigned long long* slot) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *slot = globaltimer_ns();
}

// Global warp index / count for grid-stride warp loops: neighbouring indices lie in different
// blocks, so that a few items go to as many SMs. gthread_id numbers the threads the same way;
// lthread_id numbers a block's threads together, for passes over whole arrays (what they list
// comes out in stretches of consecutive ids, which the host's commit loop walks faster).
__device__ __forceinline__ int gwarp_id() { return (int)(threadIdx.x / WARP * gridDim.x + blockIdx.x); }
__device__ __forceinline__ int64_t gthread_id() { return (int64_t)gwarp_id() * WARP + lane_id(); }
__device__ __forceinline__ int64_t lthread_id() { return blockIdx.x * (int64_t)blockDim.x + threadIdx.x; }
__device__ __forceinline__ int gwarp_count() { return (int)((gridDim.x * blockDim.x) / WARP); }

}  // namespace scout
