// union.cu -- one persistent kernel for a round of several problems' union stores.
//
// The batched engine (multi.cu) keeps many streams of ONE problem as a disjoint union in one
// store, so a round over streams of all four problems would be four merges and four
// cooperative repair launches. Here ONE cooperative launch runs the repairs, each over its own
// store and work queues, with its own counters and its own bounded grid barrier (zeroed before
// the launch). Rounds of ordinary batches run side by side: the updates in one launch
// (update_side), then the repairs (k_union_side), each problem on its share of the SMs. Larger
// ones queue the stores' merges first, each on its own context's stream, and then run the repairs
// one after the other, every block taking part in each (k_union_round). The kernels' register
// counts are the largest of the four bodies', within the 64 per thread a 1,024-thread block
// allows.
#include "ctx.cuh"
#include "bfs_dev.cuh"
#include "cc_dev.cuh"
#include "coloring_dev.cuh"
#include "mis_dev.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>

namespace scout {

struct UnionRound {
    int has_bfs, has_cc, has_col, has_mis;
    BfsParams bfs;
    CcParams cc;
    ColParams col;
    MisParams mis;
    int order[SIDE_MAX];   // side by side: the problem of each grid row
};

__global__ void __launch_bounds__(REPAIR_THREADS, 1) k_union_round(UnionRound u) {
    if (u.has_bfs) bfs_body(u.bfs);
    if (u.has_cc) cc_body(u.cc);
    if (u.has_col) coloring_body(u.col);
    if (u.has_mis) mis_body(u.mis);
}

// Grid row y runs the repair of problem order[y] on its share of the SMs.
__global__ void __launch_bounds__(REPAIR_THREADS, 1) k_union_side(const __grid_constant__ UnionRound u) {
    switch (u.order[blockIdx.y]) {
    case SCOUT_BFS: bfs_body(u.bfs); break;
    case SCOUT_CC: cc_body(u.cc); break;
    case SCOUT_COLORING: coloring_body(u.col); break;
    default: mis_body(u.mis); break;
    }
}

// What bounds a round of ordinary batches is latency: a repair is a chain of barriers and dependent
// reads that leaves most of 148 SMs idle, and the repairs (and updates) of four stores one after the
// other take the sum of their chains. Side by side, each on its share of the SMs and with a grid
// barrier of its own blocks (gridDim.x), they take about the longest one. Measured with four stores of
// scale 16 (16 edges per vertex), whole round, one after the other -> side by side: 64 edits each
// 466 -> 311 us, 1,000 529 -> 333, 16,000 775 -> 432. One large batch beside three of 64 edits has
// only a share of the chip: of 16,000 edits at scale 17 the closest case (CC) still gains, 525 -> 415
// us, at scale 20 it is even (619 -> 615, 655 -> 669 with most deletions at low degrees), and 32,000
// there lose (657 -> 740). Hence the limits: up to SIDE_EDITS edits in every batch, and up to
// SIDE_VERTICES vertices (what a recompute or a wide cascade reads grows with the store, not with
// the batch).
constexpr int64_t SIDE_EDITS = 16384, SIDE_VERTICES = 1 << 19;

bool union_side(scout_ctx* const* cs, const int64_t* counts, int ne) {
    if (ne < 2 || ne > SIDE_MAX || cs[0]->sm_count < ne) return false;
    for (int i = 0; i < ne; i++)
        if (cs[i]->tiered || counts[i] > SIDE_EDITS || cs[i]->n > SIDE_VERTICES) return false;
    return true;
}

// cs[i] holds the union store of problems[i] (distinct problems, one device) with its batch
// merged (queued on its stream), or its parameters in `round` (the first `later`; their launch comes
// first). Launches the fused repair on cs[0]'s stream once every merge is done; every context's stream then waits for the repair. variants[i]: the repair variant
// (BFS mode, CC variant). cs[0]'s ev_t[4] / ev_t[5] bracket the launch.
int union_launch(scout_ctx* const* cs, const int* problems, const scout_sched* sds, const int* variants, int ne,
                 const UpdateRound& round, int later, bool side) {
    UnionRound u;
    std::memset(&u, 0, sizeof(u));
    scout_ctx* c0 = cs[0];
    size_t smem = 0;
    for (int i = 0; i < ne; i++) {
        scout_ctx* c = cs[i];
        u.order[i] = problems[i];
        switch (problems[i]) {
        case SCOUT_BFS: SCOUT_RC(bfs_params(c, variants[i], nullptr, &u.bfs)); u.has_bfs = 1; break;
        case SCOUT_CC:
            SCOUT_RC(cc_params(c, &sds[i], variants[i], nullptr, &u.cc));
            u.has_cc = 1;
            smem = CC_SMEM;
            break;
        case SCOUT_COLORING: SCOUT_RC(coloring_params(c, &u.col)); u.has_col = 1; break;
        case SCOUT_MIS: SCOUT_RC(mis_params(c, &u.mis)); u.has_mis = 1; break;
        default: return c->fail(SCOUT_E_INVALID, "unknown problem");
        }
    }
    for (int i = 1; i < ne; i++) {   // the launch stream waits for every other store's merge
        SCOUT_CU(cs[i], cudaEventRecord(cs[i]->ev_union, cs[i]->s_main));
        SCOUT_CU(c0, cudaStreamWaitEvent(c0->s_main, cs[i]->ev_union, 0));
    }
    if (later > 0) {
        SCOUT_RC(update_side(c0, round, later));
        for (int i = 0; i < ne; i++) SCOUT_CU(cs[i], cudaEventRecord(cs[i]->ev_t[1], c0->s_main));
    }
    for (int i = 0; i < ne; i++)   // every repair's grid barrier starts at zero
        SCOUT_RC(bar_clear(cs[i], c0->s_main));
    const void* fn = side ? (const void*)k_union_side : (const void*)k_union_round;
    if (smem) {   // the dynamic shared-memory opt-in: once per device
        static std::atomic<unsigned long long> attr_done[2];
        const unsigned long long bit = 1ull << (c0->device & 63);
        if (!(attr_done[side].load() & bit)) {
            SCOUT_CU(c0, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            attr_done[side].fetch_or(bit);
        }
    }
    const int threads = repair_threads(c0);
    int per_sm = 0;
    SCOUT_CU(c0, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
    if (per_sm < 1) return c0->fail(SCOUT_E_CUDA, "fused repair kernel does not fit on an SM");
    void* args[] = {&u};
    SCOUT_CU(c0, cudaEventRecord(c0->ev_t[4], c0->s_main));
    const dim3 grid(side ? (unsigned)(c0->sm_count / ne) : (unsigned)c0->sm_count, side ? (unsigned)ne : 1u);
    SCOUT_CU(c0, cudaLaunchCooperativeKernel(fn, grid, dim3((unsigned)threads), args, smem, c0->s_main));
    SCOUT_CU(c0, cudaEventRecord(c0->ev_t[5], c0->s_main));
    c0->nlaunch += 1;
    SCOUT_CU(c0, cudaEventRecord(c0->ev_union, c0->s_main));
    for (int i = 1; i < ne; i++) SCOUT_CU(cs[i], cudaStreamWaitEvent(cs[i]->s_main, c0->ev_union, 0));
    return SCOUT_OK;
}

}  // namespace scout
