// Slot arrays and kernel argument blocks of the search kernels.
#pragma once

#include "common.cuh"

namespace ddp {

struct SearchCtl;

// Memory of `nslots` independent search slots (one per concurrent query).
struct SlotArrays {
    int32_t n = 0;
    int nslots = 0;
    int words = 1;        // 64-bit state words per node: 1, or 4 (paired slots: a 32-byte record)
    int64_t sstride = 0;  // state words per slot
    int hbits = 0;        // hashed paired slots: log2 of the records per slot
    bool pair = false;    // bidirectional layout (no queues, 8-byte units of far memory)
    int64_t cap_q = 0, cap_f = 0;
    unsigned long long *state = nullptr;  // nslots x n x words
    int32_t *touched = nullptr;           // nslots x n (null for paired slots)
    uint32_t *hops = nullptr;             // nslots x n (per-target heuristic) or null
    uint2 *q = nullptr;                   // nslots x 2 x cap_q (null for paired slots)
    uint4 *f = nullptr;                   // nslots x 2 x cap_f {node, g, f, 0}
    SearchCtl *ctl = nullptr;             // nslots
    uint32_t *epoch = nullptr;            // nslots: per-query tag counter of the hop array
};

// Graph maintenance jobs of a serving launch, run by its service CTA (or by
// k_svc when no serving kernel runs).  Lists live in host memory mapped into
// the device.  Kinds (k elements):
//   SVC_SCATTER_ARCS  ((uint2 *)p0)[((long long *)p2)[i]] = ((uint2 *)p3)[i]
//   SVC_SCATTER_ROWS  r = ((int4 *)p2)[i]: ((int *)p0)[r.x] = r.y, ((int *)p1)[r.x] = r.z
//   SVC_GATHER_ARCS   j = ((long long *)p2)[i]: ((uint2 *)p0)[j] = ((uint2 *)p1)[j]
//   SVC_GATHER_INTS   j = ((int *)p2)[i]: ((int *)p0)[j] = ((int *)p1)[j]
//   SVC_COPY_WORDS    ((uint32_t *)p0)[i] = ((uint32_t *)p1)[i]
enum { SVC_SCATTER_ARCS = 0, SVC_SCATTER_ROWS, SVC_GATHER_ARCS, SVC_GATHER_INTS, SVC_COPY_WORDS };
struct SvcSub {
    int kind, pad;
    long long k;
    unsigned long long p0, p1, p2, p3;
};
constexpr int SVC_MAX_SUB = 8;
// The host fills nsub, sub[], wait_buf and claim (= the job's number) and
// publishes seq.  The service CTA waits for the buffer, claims the job (claim:
// its number -> 0), runs the subs in order and marks done = seq.  A host that
// gives up waiting takes the job back by the same step, so that a job it has
// reported as failed never runs on lists that are written again.
struct SvcJob {
    int seq, claim, done, nsub;
    int wait_buf, pad;  // version buffer that no search may run on first (-1: none)
    SvcSub sub[SVC_MAX_SUB];
};
// Polls of a busy buffer after which the service CTA looks at its launch
// again (closing, pause) before it waits on, and how long the host waits for
// a job.  (A build with small numbers lets a test see both run out.)
#ifndef DDP_SVC_POLLS
#define DDP_SVC_POLLS (1u << 21)
#endif
#ifndef DDP_SVC_WAIT_NS
#define DDP_SVC_WAIT_NS 30000000000LL
#endif
constexpr uint32_t SVC_POLLS = DDP_SVC_POLLS;
constexpr long long SVC_WAIT_NS = DDP_SVC_WAIT_NS;

struct BatchArgs {
    const int32_t *S, *T;
    int32_t nq;
    int32_t *cost, *plen, *paths;
    int32_t path_cap;
    int32_t *qstatus;
    long long *stats, *tstart, *tend;
    int *work, *status;
    int32_t *order;  // non-null: the queries in the order they are claimed (k_order)
    uint32_t delta;
    int32_t K;
    int64_t bfs_budget;  // capped heuristic BFS (0 = run to completion)
    int64_t lazy_budget;   // entries a search may expand before it starts again with eager labels
    uint32_t eager_delta;  // bucket width of that second start
    bool skewed;           // the graph has hubs (skewed_rows)
    int group;           // CTAs per query slot
    int sync_engine;     // 1: phase-synchronous engine even for one-CTA slots
    // serving mode (continuous batching): requests are published in host
    // memory mapped into the device; slots wait for them
    int serve;
    const volatile int *pub;    // published request count
    const volatile int *pause;  // non-zero: stop claiming, exit
    int idle_limit;             // polls (~1 us each) before a slot votes to exit
    int *seen, *tokens;         // published count as the slots know it; requests free to claim
    int *idle_votes;            // slots that found no work for idle_limit polls
    int *closing;               // set once every slot voted: all slots exit
    int serve_slots;            // search slots in the launch
    volatile SvcJob *svc;       // non-null: CTA serve_slots is the service CTA
    volatile int *done;         // per request: 1 once cost/ver are written
    int32_t *ver;               // per request: graph version it ran on
    int version;
    // versioned graphs (serving): version v lives in vtab[v % nver]
    const DevGraph *vtab;         // host memory, rewritten while the kernel runs
    int nver;
    const volatile int *cur_ver;  // latest published version (host memory)
    int *inflight;                // per buffer: searches running on it
};

// The bidirectional batch kinds, and their k_batch instances (5: no
// potential, 6: Euclidean, 7: Manhattan potentials).
inline bool is_bidir_kind(int k) {
    return k == DDP_H_BIDIR || k == DDP_H_BIDIR_EUCLID || k == DDP_H_BIDIR_MANHATTAN;
}
// 8: DDP_H_BIDIR with hashed records (DDP_OPT_HASH); 9: DDP_H_BIDIR with
// 16-byte pairs (graphs with coordinates); 10: landmark potentials
constexpr bool bidir_hk(int hk) { return hk >= 5 && hk <= 10; }
constexpr bool pair16_hk(int hk) { return hk == 9; }
// Whether slots of `group` CTAs answer a batch kind by the bidirectional
// search: the bidirectional kinds always; one-CTA slots also for no bound,
// hop bounds (without them: a one-directional search under so weak a bound
// expands orders of magnitude more; 300 queries, 100,000 nodes: a reverse BFS
// of the whole graph and 45k expansions per query, 9.86 ms, against 0.8k
// expansions, 0.20 ms) and landmarks (as average potentials).  These bounds
// are admissible on every graph, so the costs are the same.  Wider slots and
// DDP_OPT_SYNC keep the A* engine.
inline bool batch_bidir(int hkind, int group, int flags) {
    if (is_bidir_kind(hkind)) return true;
    return group <= 1 && !(flags & DDP_OPT_SYNC) &&
           (hkind == DDP_H_ZERO || hkind == DDP_H_BFS_HOPS || hkind == DDP_H_BFS_CAPPED || hkind == DDP_H_LANDMARK);
}
// Far memory (8-byte units per half, slot_bytes) of a bidirectional slot: the
// bucket lists want 4 MB however small the graph or the caller's capacity.
inline int64_t bidir_cap_f(int64_t want) { return want > (1 << 18) ? want : (int64_t)(1 << 18) + 4096; }
int kernel_hk(int hkind, bool has_xy, bool hash, int group, int flags);
int hk_slot_kind(int hk);

// Slot kinds (bits): a per-target hop array; paired forward/reverse state;
// paired records in a hash table of 2^hbits records instead of one per node.
// SLOT_PAIR16: 16-byte pairs (one 64-bit word per direction), a touched
// log of 2n entries and the paired queue layout.
enum { SLOT_HOPS = 1, SLOT_PAIR = 2, SLOT_HASH = 4, SLOT_PAIR16 = 8 };
size_t slot_bytes(int32_t n, int64_t cap_q, int64_t cap_f, int kind, int hbits = 0);
// log2 of the hashed records per slot for an n-node graph
int hash_bits(int32_t n);
// Runs maintenance subs with ordinary launches on st (no serving kernel runs).
cudaError_t svc_run_direct(const SvcSub *subs, int nsub, cudaStream_t st);
int slots_alloc(SlotArrays &sa, int32_t n, int nslots, int64_t cap_q, int64_t cap_f, int kind,
                cudaStream_t st, int hbits = 0);
void slots_free(SlotArrays &sa);
uint32_t *heuristic_hops_ptr(const ddp_heuristic *h);
int heuristic_build_locked(ddp_graph *g, int32_t target, int32_t kind, const int32_t *user_h, int32_t *out_h,
                           ddp_heuristic **out);
cudaError_t launch_slots(int hk, int grid, int block, bool coop, DevGraph G, SlotArrays sa, BatchArgs A,
                         cudaStream_t st);
int slots_per_sm(int hk, int block, bool grouped);
int device_sms();
uint32_t auto_delta(const ddp_graph *g);
uint32_t loose_delta(const ddp_graph *g);  // SearchParams::delta_loose
uint32_t auto_delta_bidir(const ddp_graph *g);
// Fills the bucket widths and the budget of a bidirectional launch.
void bidir_args(const ddp_graph *g, int32_t delta, BatchArgs *A);
int64_t bfs_budget(int32_t n);
// Whether queues of cap entries are worth a try: they begin at about the number
// of nodes and are doubled when one overflows.  A phase pushes an entry for
// each arc that improves its head at most, so that hubs whose rows name the
// nodes many times over want far more entries than nodes, but never many more
// than arcs.
bool queue_cap_ok(const ddp_graph *g, int64_t cap);

}  // namespace ddp
