// GA* search engine: device code shared by the single-query (whole grid)
// and batched (one CTA per query slot) kernels.
//
// What it replaces (lkoshale/DDP, LIB/include/kernels/a_star_kernels.cu):
//   extractMin  (:7-61)   K threads pop K heap tops
//   A_star_expand (:67-133) one thread per node, spin lock per child
//   keepHeapPQ + setNV + insertPQ (:138-237) heap repair, O(N) flag scan,
//                                           round-robin re-insert
//   checkMIN (:243-254)   stop when no heap top has f < f(t)
//
// How it works here:
//   * Open list = threshold buckets on f (near-far): `near` holds entries
//     with f < T, `far` the rest.  One iteration expands up to K entries of
//     near (all of it when K = 0); improved children go to `next` when
//     f < T, else to `far`.  When near and next are empty the far pile is
//     split at T' = T + delta (or at its smallest f + delta): f < T' moves to
//     near, the rest is compacted.  Stale entries (g changed since the push)
//     and entries with f >= f(t) are dropped at every pop and split.
//   * Termination (the GA* test of checkMIN, made exact): the search ends
//     when near, next and far are all empty after pruning, i.e. no open
//     node has f < f(t).  With an admissible heuristic g(t) is then optimal.
//   * Expansion is warp-cooperative: 32 popped nodes per warp, their rows are
//     concatenated by a warp prefix sum and walked 32 arcs at a time, so arc
//     loads are 8-byte {head, w} reads of consecutive row slices.
//   * Relaxation is lock-free: one 64-bit word per node packs (g << 32 |
//     parent); a plain L2 read filters the (common) non-improving arcs, then
//     a CAS loop installs strictly smaller g.  No spin locks (the reference's
//     `while(!leaveLoop)` lock with __syncthreads inside divergent code is
//     gone).
//   * Pushes are warp-aggregated: one atomic per warp per target queue.
//   * Every loop bound is data-driven; the only wait is the group barrier,
//     which is bounded (common.cuh).
#pragma once

#include "common.cuh"
#include "rules.h"

namespace ddp {

constexpr unsigned FULL = 0xffffffffu;

// Control block of one search slot (global memory).  Push counters rotate
// over 4 phases so that a counter is reset two phases before it is used
// again, with a single barrier per phase.  One phase's counters are 16
// bytes, read together after the phase's barrier.
struct __align__(16) PhaseWords {
    int nq;            // pushes into near/next (or BFS frontier) this phase
    int fq;            // pushes into far this phase
    unsigned int mf;   // min f kept in far during a split phase
    int err;           // ST_* raised during the phase (read after its barrier)
};
struct SearchCtl {
    PhaseWords ph[4];
    int ck[4];            // chunks claimed so far in the phase, beyond one per warp
    int touched;          // nodes whose state left the initial value
    int status;           // ST_* bits
    int iters;            // phases run
    int pad;
    unsigned long long expanded, scanned, relaxed, pad2;
    unsigned long long bfs_reached, bfs_scanned;  // heuristic BFS work
    unsigned long long far_scanned;               // far entries read by splits
    unsigned int tag;     // hop-array tag of the current query (batch)
    unsigned int hcap;    // hop cap of the last BFS
    int cur_q;            // query the slot is working on (batch)
    int far_n, far_sel;   // far pile left by the last run (dynamic resume)
    int cur_ver;          // graph version of the current search (serving)
    int path_len;         // single query: the path as walked before the labels go (walk_path)
    unsigned int bar_count, bar_gen;  // grid barrier (single-query form)
    int cold_n;           // entries in the far pile's cold tier (keep mode) ...
    unsigned int cold_x;  // ... all with g >= cold_x
    // what CTA 0 hands back after running phases alone (run_search)
    int loc_near, loc_far, loc_waves, loc_flip, loc_done;
    uint32_t loc_T;
};

// Buffers of one slot.
struct SlotBufs {
    unsigned long long *state;  // n, (g << 32) | parent; all-ones = unreached
    uint2 *q0, *q1;             // near / next ping-pong, cap_q entries {node, g}
    uint4 *f0, *f1;             // far ping-pong, cap_f entries {node, g, f, 0}
    int32_t *touched;           // n: nodes whose state must be reset
    uint32_t *hops;             // n: per-target hop heuristic (may be null)
    SearchCtl *ctl;
    int64_t cap_q, cap_f;
    int64_t swords;  // 64-bit words of the state array
    int hbits;       // hashed records: log2 of the table size (0: one record per node)
};

// ---- groups ------------------------------------------------------------------
struct CtaGroup {
    int *status;
    __device__ int rank() const { return threadIdx.x; }
    __device__ int size() const { return blockDim.x; }
    __device__ int warp() const { return threadIdx.x >> 5; }
    __device__ int nwarps() const { return blockDim.x >> 5; }
    __device__ void sync() const { __syncthreads(); }
    template <class F>
    __device__ void sync_fetch(F fetch) const {  // see grid_sync_fetch
        __syncthreads();
        if (threadIdx.x == 0) fetch();
        __syncthreads();
    }
    static constexpr bool multi = false;  // more than one CTA
    __device__ bool first_cta() const { return true; }
};

struct GridGroup {
    GridBarrier bar;
    int *status;
    __device__ int rank() const { return blockIdx.x * blockDim.x + threadIdx.x; }
    __device__ int size() const { return gridDim.x * blockDim.x; }
    __device__ int warp() const { return (blockIdx.x * blockDim.x + threadIdx.x) >> 5; }
    __device__ int nwarps() const { return (gridDim.x * blockDim.x) >> 5; }
    __device__ void sync() const { grid_sync(bar, gridDim.x, status); }
    template <class F>
    __device__ void sync_fetch(F fetch) const { grid_sync_fetch(bar, gridDim.x, status, fetch); }
    static constexpr bool multi = true;
    __device__ bool first_cta() const { return blockIdx.x == 0; }
};

// G consecutive CTAs of a cooperative launch working on one query.
struct SubGridGroup {
    GridBarrier bar;
    int *status;
    int G;
    __device__ int rank() const { return (blockIdx.x % G) * blockDim.x + threadIdx.x; }
    __device__ int size() const { return G * blockDim.x; }
    __device__ int warp() const { return rank() >> 5; }
    __device__ int nwarps() const { return size() >> 5; }
    __device__ void sync() const { grid_sync(bar, (unsigned)G, status); }
    template <class F>
    __device__ void sync_fetch(F fetch) const { grid_sync_fetch(bar, (unsigned)G, status, fetch); }
    static constexpr bool multi = true;
    __device__ bool first_cta() const { return blockIdx.x % G == 0; }
};

// ---- heuristics (h(v) as uint32, INF_G = "cannot reach the target") -------
struct HeurZero {
    __device__ uint32_t operator()(int32_t) const { return 0; }
};

struct HeurHops {  // reverse-BFS hop count x scale (GA_star/bfs_hx.cu)
    const uint32_t *hops;
    uint32_t scale;
    uint32_t cap;  // hops assumed for unreached nodes (HOPS_INF = cannot reach t)
    uint32_t tag;  // 0: plain levels; else epoch-tagged words (run_bfs_hops)
    __device__ uint32_t operator()(int32_t v) const {
        const uint32_t x = __ldcg(hops + v);
        uint32_t hv;
        if (tag) hv = ((x & 0xFFFFFF00u) == tag) ? (x & 0xFFu) : cap;
        else hv = (x == HOPS_INF) ? cap : x;
        if (hv == HOPS_INF) return INF_G;
        unsigned long long p = (unsigned long long)hv * scale;
        return p >= INF_G ? INF_G : (uint32_t)p;
    }
};

struct HeurArray {  // caller-supplied h; negative = cannot reach the target
    const int32_t *h;
    __device__ uint32_t operator()(int32_t v) const {
        int32_t x = __ldg(h + v);
        return x < 0 ? INF_G : (uint32_t)x;
    }
};

struct HeurManhattan {
    const int32_t *xy;
    int32_t tx, ty;
    uint32_t scale;
    __device__ uint32_t operator()(int32_t v) const {
        int2 p = __ldg(reinterpret_cast<const int2 *>(xy) + v);
        unsigned long long d = (unsigned long long)(abs(p.x - tx)) + (unsigned long long)(abs(p.y - ty));
        d *= scale;
        return d >= INF_G ? INF_G : (uint32_t)d;
    }
};

// ALT lower bound: max over landmarks L of d(L,t) - d(L,v) and d(v,L) - d(t,L)
// (triangle inequality, so admissible, and consistent when s = 1).  The
// table holds q = floor(d / s); d(a) - d(b) >= s (q_a - q_b) - (s - 1),
// which is the exact difference when s = 1.  The engines need
// admissibility only: a node reached again with a smaller g is re-expanded.  A landmark that reaches v but not t, or is
// reached from t but not from v, proves that v cannot reach t.
// unroll factor of the landmark row loops (row loads issued ahead of use).
// More row loads in flight cost registers that the one-CTA engine spills:
// 500 queries on 400,000 nodes, 64 landmarks of 8 bits: 8 -> 9.21 ms,
// 4 -> 8.59, 2 -> 8.37.
constexpr int ALT_UNROLL = 2;
struct HeurALT {
    const uint2 *tab;  // DevGraph::lm: rows of 2L entries
    int32_t L;         // landmarks, a multiple of 4 (16-bit) or 8 (8-bit)
    int32_t s;         // DevGraph::lm_scale
    int32_t t;
    int32_t mode;      // DevGraph::lm_bits (16 or 8) + 256 lm_cut
    __device__ __forceinline__ bool bytes() const { return (mode & 255) == 8; }
    __device__ __forceinline__ bool cut() const { return mode >= 256; }
    // One packed word of B-bit entries, a from the row that must be larger:
    // the lanes' a - b, saturated at 0, fold into the lane-wise maximum m (the
    // marker counts as an entry: as b it leaves nothing, as a it stands for a
    // distance of at least that many scales, so the bound stays one, and stays
    // consistent, where a distance was too long for the table); lanes where a
    // is the marker and b is not (the landmark relates v and t one way
    // only, so v cannot reach t if every finite distance is in the table:
    // cut) fold into the cut mask cm.  Since s >= 1,
    // the maximum over terms of s (a - b) - (s - 1), floored at 0, is
    // s max(a - b) - (s - 1) when that maximum is positive, else 0.
    template <int B>
    __device__ __forceinline__ void word(uint32_t a, uint32_t b, uint32_t &m, uint32_t &cm) const {
        if (B == 8) {
            const uint32_t ea = __vcmpeq4(a, 0xFFFFFFFFu), eb = __vcmpeq4(b, 0xFFFFFFFFu);
            cm |= ea & ~eb;
            m = __vmaxu4(m, __vsubus4(a, b));
        } else {
            const uint32_t ea = __vcmpeq2(a, 0xFFFFFFFFu), eb = __vcmpeq2(b, 0xFFFFFFFFu);
            cm |= ea & ~eb;
            m = __vmaxu2(m, __vsubus2(a, b));
        }
    }
    template <int B>
    __device__ __forceinline__ void terms(uint2 a, uint2 b, uint32_t &m, uint32_t &cm) const {
        word<B>(a.x, b.x, m, cm);
        word<B>(a.y, b.y, m, cm);
    }
    template <int B>
    __device__ __forceinline__ uint32_t eval(int32_t v) const {
        const int W = L / (64 / B);  // 8-byte words per half row
        const uint2 *rv = tab + (size_t)v * (2 * W);
        const uint2 *rt = tab + (size_t)t * (2 * W);
        uint32_t m = 0, cm = 0;
        if ((W & 1) == 0) {
            // both halves start on a 16-byte boundary: 16-byte loads
            const uint4 *qv = reinterpret_cast<const uint4 *>(rv), *qt = reinterpret_cast<const uint4 *>(rt);
            const int W2 = W >> 1;
#pragma unroll ALT_UNROLL
            for (int i = 0; i < W2; i++) {
                const uint4 fv = __ldg(qv + i), ft = __ldg(qt + i);
                terms<B>(make_uint2(ft.x, ft.y), make_uint2(fv.x, fv.y), m, cm);
                terms<B>(make_uint2(ft.z, ft.w), make_uint2(fv.z, fv.w), m, cm);
            }
#pragma unroll ALT_UNROLL
            for (int i = W2; i < 2 * W2; i++) {
                const uint4 bv = __ldg(qv + i), bt = __ldg(qt + i);
                terms<B>(make_uint2(bv.x, bv.y), make_uint2(bt.x, bt.y), m, cm);
                terms<B>(make_uint2(bv.z, bv.w), make_uint2(bt.z, bt.w), m, cm);
            }
        } else {
            for (int i = 0; i < W; i++) {
                const uint2 fv = __ldg(rv + i), ft = __ldg(rt + i);
                const uint2 bv = __ldg(rv + W + i), bt = __ldg(rt + W + i);
                terms<B>(ft, fv, m, cm);
                terms<B>(bv, bt, m, cm);
            }
        }
        return cm && cut() ? INF_G : top<B>(m);
    }
    // the bound of the lane-wise maximum m
    template <int B>
    __device__ __forceinline__ uint32_t top(uint32_t m) const {
        const uint32_t mx = B == 8 ? max(max(m & 0xFFu, (m >> 8) & 0xFFu), max((m >> 16) & 0xFFu, m >> 24))
                                   : max(m & 0xFFFFu, m >> 16);
        // mx s is at most the marker times s, at most INF_G
        return mx ? mx * (uint32_t)s - (uint32_t)(s - 1) : 0u;
    }
    __device__ uint32_t operator()(int32_t v) const { return bytes() ? eval<8>(v) : eval<16>(v); }
};

// floor(sqrt(x)) for x < 2^62, exact: a float estimate, then integer fix-up
__host__ __device__ __forceinline__ uint64_t isqrt_floor(uint64_t x) {
    uint64_t r = (uint64_t)sqrt((double)x);
    while (r * r > x) r--;
    while ((r + 1) * (r + 1) <= x) r++;
    return r;
}

struct HeurEuclid {  // floor(rho * floor(dist)), rho <= w / length on every arc
    const int32_t *xy;
    int32_t tx, ty;
    uint32_t rho_fp;  // 16.16
    __device__ uint32_t operator()(int32_t v) const {
        int2 p = __ldg(reinterpret_cast<const int2 *>(xy) + v);
        const int64_t dx = (int64_t)p.x - tx, dy = (int64_t)p.y - ty;
        const uint64_t r = isqrt_floor((uint64_t)(dx * dx + dy * dy));
        const uint64_t h = (r * rho_fp) >> 16;
        return h >= INF_G ? INF_G - 1 : (uint32_t)h;
    }
};

// Heuristics computed from registers and one small load (coordinates): the
// one-CTA engine evaluates them speculatively, beside the relaxation's
// atomic, instead of after it.  Table heuristics (hops, landmarks, arrays)
// are read only for relaxations that improve g.
template <class H>
struct heur_cheap {
    static constexpr bool value = false;
};
template <>
struct heur_cheap<HeurZero> {
    static constexpr bool value = true;
};
template <>
struct heur_cheap<HeurManhattan> {
    static constexpr bool value = true;
};
template <>
struct heur_cheap<HeurEuclid> {
    static constexpr bool value = true;
};

// ---- warp helpers ----------------------------------------------------------
__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// Returns this lane's slot in a warp-aggregated append (or -1 when !pred).
__device__ __forceinline__ int warp_append(bool pred, int *counter) {
    unsigned m = __ballot_sync(FULL, pred);
    if (m == 0) return -1;
    int lane = lane_id();
    int leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counter, __popc(m));
    base = __shfl_sync(FULL, base, leader);
    return pred ? base + __popc(m & ((1u << lane) - 1u)) : -1;
}

__device__ __forceinline__ int warp_excl_scan(int x, int *total) {
    int lane = lane_id();
    int v = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v += y;
    }
    *total = __shfl_sync(FULL, v, 31);
    return v - x;
}

// Chunks of a phase over `cnt` entries: warp w takes chunk w, and only a
// phase with more chunks than warps claims the rest from a counter (dynamic
// balance: warps that finish early take more).  A narrow phase then costs no
// claim atomics (they serialise on one L2 line: two per warp of a full grid
// took 5-10 us a phase), and its entries are spread over the warps instead
// of filling the first few.
struct Chunks {
    int size;      // entries per chunk, at most 32
    int64_t first; // this warp's first chunk
    bool more;     // further chunks are claimed
    int nw;
    int *counter;
    __device__ Chunks(int64_t cnt, int warp, int nwarps, int *ck) : first(warp), nw(nwarps), counter(ck) {
        const int64_t per = (cnt + nwarps - 1) / nwarps;
        size = per >= 32 ? 32 : per < 1 ? 1 : (int)per;
        more = cnt > (int64_t)size * nwarps;
    }
    // the chunk after c (a count past the end when there is none)
    __device__ int64_t next(int64_t cnt) const {
        if (!more) return cnt;
        int c = 0;
        if ((threadIdx.x & 31) == 0) c = atomicAdd(counter, 1);
        return (int64_t)nw + __shfl_sync(0xffffffffu, c, 0);
    }
};

// Records an error for phase `ph` (consistent control flow after the
// barrier) and in the sticky status word (reporting).
__device__ __forceinline__ void raise_err(SearchCtl *ctl, int ph, int bit) {
    atomicOr(&ctl->ph[ph].err, bit);
    atomicOr(&ctl->status, bit);
}

__device__ __forceinline__ uint32_t sat_add(uint32_t a, uint32_t b) {
    uint32_t c = a + b;
    return c < a ? 0xFFFFFFFFu : c;
}

// Per-warp shared memory: staging of 32 popped rows, and staging buffers
// for queue pushes (flushed with one atomic per >= 32 entries, so the L2
// round trip of a queue reservation is paid once per flush instead of once
// per 32 arcs, and the stores are coalesced).
struct WarpRows {
    int excl[32];
    int rb[32];      // first arc of the base row
    int bdeg[32];    // base-row length (diff arcs follow)
    int drb[32];     // first arc of the diff row
    uint32_t g[32];
    int u[32];
    uint2 sn[64];    // staged near/next pushes
    int2 snr[64];    // one-CTA engine: row bounds of the staged own children
    uint4 sf[64];    // staged far pushes
    int st[64];      // staged first touches / BFS frontier pushes
};

// Copies a warp's staged entries to dst[base + reserved ..] (all lanes).
template <class T>
__device__ __forceinline__ void stage_flush(T *buf, int &cnt, int *counter, T *dst, int64_t base,
                                            int64_t cap, SearchCtl *ctl, int ph);

template <class T>
__device__ __forceinline__ void stage_push(bool pred, T val, T *buf, int &cnt, int *counter, T *dst,
                                           int64_t base, int64_t cap, SearchCtl *ctl, int ph) {
    const unsigned m = __ballot_sync(FULL, pred);
    if (pred) buf[cnt + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))] = val;
    cnt += __popc(m);
    if (cnt >= 32) stage_flush(buf, cnt, counter, dst, base, cap, ctl, ph);
}

template <class T>
__device__ __forceinline__ void stage_flush(T *buf, int &cnt, int *counter, T *dst, int64_t base,
                                            int64_t cap, SearchCtl *ctl, int ph) {
    if (cnt == 0) return;  // warp-uniform
    __syncwarp();
    int b = 0;
    if ((threadIdx.x & 31) == 0) b = atomicAdd(counter, cnt);
    b = __shfl_sync(FULL, b, 0);
    for (int i = threadIdx.x & 31; i < cnt; i += 32) {
        const int64_t pos = base + b + i;
        if (pos < cap) dst[pos] = buf[i];
        else raise_err(ctl, ph, ST_OVERFLOW);
    }
    __syncwarp();
    cnt = 0;
}

// What a phase leaves in a warp's staging buffers, for the three pushes a
// search makes, copied out CTA-wide: one reservation per queue and CTA
// instead of one per queue and warp.
struct CtaFlush {
    int cnt[3][32];   // entries per warp, then the warp's offset
};
// near, far and touched entries of this warp; call from every thread.
template <class TN, class TF>
__device__ __forceinline__ void cta_flush(CtaFlush *cf, WarpRows &wr, const TN *bn, int c_n, int *k_n, TN *d_n,
                                          int64_t base_n, int64_t cap_n, const TF *bf, int c_f, int *k_f, TF *d_f,
                                          int64_t base_f, int64_t cap_f, int c_t, int *k_t, int32_t *d_t,
                                          int64_t cap_t, SearchCtl *ctl, int ph) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)((blockDim.x + 31) >> 5);
    if (lane == 0) {
        cf->cnt[0][warp] = c_n;
        cf->cnt[1][warp] = c_f;
        cf->cnt[2][warp] = c_t;
    }
    __syncthreads();
    for (int q = warp; q < 3; q += nw) {
        const int x = lane < nw ? cf->cnt[q][lane] : 0;
        int total;
        const int ex = warp_excl_scan(x, &total);
        int b = 0;
        if (lane == 0 && total) b = atomicAdd(q == 0 ? k_n : q == 1 ? k_f : k_t, total);
        b = __shfl_sync(FULL, b, 0);
        if (lane < nw) cf->cnt[q][lane] = b + ex;
    }
    __syncthreads();
    const int64_t on = base_n + cf->cnt[0][warp], of = base_f + cf->cnt[1][warp], ot = cf->cnt[2][warp];
    for (int i = lane; i < c_n; i += 32) {
        if (on + i < cap_n) d_n[on + i] = bn[i];
        else raise_err(ctl, ph, ST_OVERFLOW);
    }
    for (int i = lane; i < c_f; i += 32) {
        if (of + i < cap_f) d_f[of + i] = bf[i];
        else raise_err(ctl, ph, ST_OVERFLOW);
    }
    for (int i = lane; i < c_t; i += 32) {
        if (ot + i < cap_t) d_t[ot + i] = wr.st[i];
        else raise_err(ctl, ph, ST_OVERFLOW);
    }
}

__device__ __forceinline__ int row_owner(const WarpRows &wr, int k) {
    int o = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
        if (wr.excl[o + step] <= k) o += step;
    return o;
}

__device__ __forceinline__ uint2 row_arc(const DevGraph &G, const WarpRows &wr, int o, int k,
                                         bool fwd) {
    int j = k - wr.excl[o];
    if (j < wr.bdeg[o]) {
        if (G.oend) return fwd ? __ldcg(G.arc + wr.rb[o] + j) : __ldcg(G.rarc + wr.rb[o] + j);
        return fwd ? __ldg(G.arc + wr.rb[o] + j) : __ldg(G.rarc + wr.rb[o] + j);
    }
    j -= wr.bdeg[o];
    return fwd ? __ldcg(G.darc + wr.drb[o] + j) : __ldcg(G.drarc + wr.drb[o] + j);
}

// ---- search parameters -------------------------------------------------------
struct SearchParams {
    int32_t s, t;
    uint32_t delta;
    int32_t K;     // 0 = whole near bucket per iteration
    int resume;    // keep mode: continue from the slot's far pile instead of starting at s
    int no_touch_log;  // do not log first touches (slots that are never reset)
    // t < 0: no target, the search settles everything reachable from s
    // Keep mode, resumed searches: cold tier of the far pile.  A first split
    // moves live entries with g >= cold_x (their f is at least g) to `cold`
    // unexamined; they stay there from one resumed search to the next, with
    // the threshold they went in under, until min(f(t), threshold) of a
    // split passes it and takes them back.  On 1M nodes the tier held 671,300
    // of 671,400 open entries: carried through every search (read, set aside,
    // appended again) they took 25 us of an update's 220.  cold_x =
    // 0xFFFFFFFF: no new tier.
    uint2 *cold = nullptr;
    int64_t cold_cap = 0;
    uint32_t cold_x = 0xFFFFFFFFu;
    // A* searches on a grid: the bucket width when h(s) is below it (0: always
    // delta).  Under so weak a bound, less than an arc, the search is little
    // but rounds over buckets, and wider ones save more rounds than they
    // repeat expansions: hop bounds and none at half the weight range instead
    // of a quarter, 250k nodes of 10 arcs 353 -> 331 us, of 4 arcs 400 -> 312,
    // 1M points 9.8 -> 7.2 ms.  Tight bounds keep the quarter (200k points,
    // Euclidean: 1.01 against 1.06 ms).
    uint32_t delta_loose = 0;
    bool long_rows = true;  // A* searches on a grid: there may be rows of more than LOCAL_ROW arcs
    int64_t budget = 0;  // bidirectional search: entries it may expand (0: any number)
    bool skewed = false;  // ... and the graph has hubs (skewed_rows)
};

struct SearchResult {
    uint32_t cost;  // g(t) + h(t), >= INF_G when unreachable
    int iters;
};

// ---- narrow phases on one CTA -------------------------------------------------
// A phase of a few hundred entries gives a grid little to do and still costs
// its barrier and four dependent trips to memory.  While the near list holds
// at most LOCAL_IN entries, CTA 0 runs the search's phases alone: the list
// lives in shared memory, an entry carries its row bounds (read beside the
// relaxation that pushed it), eight lanes walk one row, and a phase ends with
// a block barrier.  It hands the list back when it outgrows LOCAL_OUT entries
// or after LOCAL_WAVES phases (the other CTAs wait in a bounded barrier).
// While the far pile is small (LOCAL_FAR, LOCAL_FAR_KEEP) it splits it too, and while the
// list is narrow (LOCAL_FILL) it takes the next bucket in early, so that the
// floods of successive buckets overlap instead of running one after the other
// (at most LOCAL_AHEAD buckets before the list empties; not in keep mode,
// where it tripled the expansions of a maze's update batches and cost 20 %).
// A phase of a 511 x 511 maze query (20-70 entries) takes about 2.5 us so, on
// the grid it took 23, and overlapping buckets halve their number (16, 32 or 64
// entries alike; wider buckets instead expand nodes again and again).
// LOCAL_FAR: one CTA takes about 20 us over a pile of 4,096 entries, a grid
// split 4.  Single queries, 4,096, 2,048, 1,024 and 512 entries: 1M points
// without bounds 26.8, 18.1, 14.8, 14.8 ms, 200,000 points under hop bounds
// 3.04, 3.04, 2.63, 2.42, a 2,047 x 2,047 maze without bounds 8.8, 8.8, 6.9,
// 7.1, a 700 x 700 one 2.04, 2.04, 2.04, 2.21, 511 x 511 and 250,000 random
// nodes alike.  Keep mode rarely splits and then needs the far pile's minimum
// at once: updates of 1M nodes at 1,024, 4,096, 16,384 entries 202, 199, 211 us.
constexpr int LOCAL_IN = 256, LOCAL_OUT = 512;
constexpr int LOCAL_FAR = 1024, LOCAL_FAR_KEEP = 4096;
constexpr int LOCAL_FILL = 32, LOCAL_AHEAD = 16;
constexpr int LOCAL_WAVES = 4096;
// Where rows may be long (SearchParams::long_rows), arcs decide too.  A row of
// more than LOCAL_LONG arcs goes to the next phase in segments, one a team (the
// entry's row end carries SEG_END).  A phase whose arcs (in rows of more than
// LOCAL_ROW) outnumber LOCAL_ARCS is the grid's, unless most are in one row: a
// grid phase gives that to one warp, 64 arcs a step, CTA 0 walks it with all its
// threads.  After LOCAL_WORK arcs the grid may pass its barrier, whose wait is
// bounded.  400,000 nodes with 20 hubs of 100,000 arcs, a caller's bound: 28 ms
// with every phase on the grid, 33 with eight lanes a row whatever its length, 17
// so; 200,000 nodes with degrees by a power law: 5.0, 5.3, 4.2 ms.  The code costs
// the 511 x 511 maze 1 % (1,445 -> 1,464 us), 250,000 nodes nothing.
constexpr int LOCAL_ROW = 32, LOCAL_ARCS = 8192, LOCAL_LONG = 256;
constexpr unsigned int LOCAL_WORK = 1u << 24, SEG_END = 0x80000000u;

// entries that the warp rows (16 per CTA in every search kernel) hold as two
// lists of uint4
constexpr int LOCAL_CAP = (int)(16 * sizeof(WarpRows) / (2 * sizeof(uint4)));
static_assert(LOCAL_CAP >= LOCAL_IN && LOCAL_CAP >= LOCAL_OUT, "local lists hold a whole phase");

// near: nnear entries in qcur (rewritten on return with the entries left);
// cold_x: no entry of the cold tier has a smaller f (0xFFFFFFFF: no tier).
// Results go to ctl->loc_*; far pushes and first touches are appended as a
// grid phase does.
template <bool KEEP, class Heur>
__device__ void local_phases(const DevGraph &G, const SlotBufs &B, const Heur &H, const SearchParams &P,
                             WarpRows *wrows, uint2 *qcur, int nnear, uint4 *fcur, uint4 *falt, int64_t nfar0,
                             uint32_t T, uint32_t ht, uint32_t cold_x, unsigned long long &n_exp,
                             unsigned long long &n_scan, unsigned long long &n_rel) {
    SearchCtl *ctl = B.ctl;
    // {node, g, row begin, row end}
    uint4 *buf = reinterpret_cast<uint4 *>(wrows);
    constexpr int cap = LOCAL_CAP;
    __shared__ int cnt[3];  // entries per wave, rotating
    __shared__ int c_far, c_touch, c_alt;
    __shared__ unsigned int tg, far_min;  // far_min: no far entry has a smaller f
    __shared__ unsigned int arcs[3], longest[3];  // of a wave's rows of more than LOCAL_ROW arcs
    const bool rows = P.long_rows;
    // a row of len arcs joins wave w (rows of more than 2^21 count as that: no sum overflows)
    auto count_row = [&](int w, int len) {
        if (len <= LOCAL_ROW) return;
        atomicAdd(&arcs[w], (unsigned int)min(len, 1 << 21));
        atomicMax(&longest[w], (unsigned int)min(len, 1 << 21));
    };
    auto wide = [&](int w) { return rows && arcs[w] > LOCAL_ARCS + 8 * longest[w]; };
    // lanes per entry: four for rows of four arcs or fewer on average
    const int lanes = G.e <= 4 * (int64_t)G.n ? 4 : 8;
    const int sub = threadIdx.x & (lanes - 1);
    const int team = threadIdx.x / lanes, teams = blockDim.x / lanes;
    const int touch0 = *(volatile int *)&ctl->touched;
    if (threadIdx.x == 0) {
        cnt[0] = nnear;
        cnt[1] = cnt[2] = 0;
        for (int w = 0; w < 3; w++) arcs[w] = longest[w] = 0;
        c_far = c_touch = 0;
        far_min = 0;
        tg = P.t >= 0 ? st_g(__ldcg(B.state + P.t)) : 0xFFFFFFFFu;
    }
    if (rows) __syncthreads();
    for (int i = threadIdx.x; i < nnear; i += blockDim.x) {
        const uint2 en = __ldcg(qcur + i);
        const int rb = row_begin(G.off, G.oend, (int)en.x), re = row_end(G.off, G.oend, (int)en.x);
        buf[i] = make_uint4(en.x, en.y, (uint32_t)rb, (uint32_t)re);
        if (rows) count_row(0, re - rb);
    }
    __syncthreads();
    int m = nnear, wv = 0, ahead = 0, flip = 0, done = 0;
    bool recheck = KEEP;
    if (!KEEP) cold_x = 0xFFFFFFFFu;
    unsigned long long n_far = 0;
    unsigned int work = 0;  // arcs in long rows so far
    uint4 *cur = buf, *nxt = buf + cap;
    while (wv || !wide(0)) {  // (a wide list goes back at once)
        if (m < (KEEP ? 1 : LOCAL_FILL)) {
            // the list is empty or narrow: the far pile's turn
            const int64_t nf = nfar0 + c_far;
            const uint64_t ft64 = (uint64_t)tg + ht;
            const uint32_t ft = ft64 >= 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)ft64;
            const uint32_t fm = far_min;
            __syncthreads();  // every thread has read the words the branches below depend on
            if (m == 0) ahead = 0;
            if ((nf == 0 ? cold_x : min(fm, cold_x)) >= ft) {
                if (m == 0) {
                    done = 1;  // no open node with f < f(t)
                    break;
                }
            } else if (nf > 0 && nf <= (KEEP ? LOCAL_FAR_KEEP : LOCAL_FAR) && (m == 0 || ahead < LOCAL_AHEAD) &&
                       min(ft, sat_add(max(fm, T), P.delta)) <= cold_x) {
                T = sat_add(max(fm, T), P.delta);  // above the smallest f: something moves
                ahead++;
                n_far += (unsigned long long)nf;
                if (threadIdx.x == 0) {
                    c_alt = 0;
                    far_min = 0xFFFFFFFFu;
                }
                __syncthreads();
                auto split = [&](const uint4 &e) {
                    if (e.z < T && (!KEEP || e.z < ft)) {
                        const int p = atomicAdd(&cnt[wv % 3], 1);
                        if (p < cap) {
                            const int rb = row_begin(G.off, G.oend, (int)e.x), re = row_end(G.off, G.oend, (int)e.x);
                            cur[p] = make_uint4(e.x, e.y, (uint32_t)rb, (uint32_t)re);
                            if (rows) count_row(wv % 3, re - rb);
                            return;
                        }
                    }
                    falt[atomicAdd(&c_alt, 1)] = e;  // no more than were read
                    atomicMin(&far_min, e.z);
                };
                if (KEEP && recheck) {
                    // keep mode, once: h may have changed since the push, f is
                    // re-derived (entries that go stale later are dropped when
                    // they are popped); a pile of a few thousand entries, four
                    // of them in flight a lane
                    constexpr int U = 4;
                    for (int64_t base = threadIdx.x; base < nf; base += (int64_t)U * blockDim.x) {
                        uint4 e[U];
                        uint64_t se[U];
                        uint32_t h[U];
#pragma unroll
                        for (int k = 0; k < U; k++) {
                            const int64_t i = base + k * (int)blockDim.x;
                            e[k] = __ldcg(fcur + (i < nf ? i : base));
                        }
#pragma unroll
                        for (int k = 0; k < U; k++) {
                            se[k] = __ldcg(B.state + e[k].x);
                            h[k] = H((int)e[k].x);
                        }
#pragma unroll
                        for (int k = 0; k < U; k++) {
                            e[k].z = sat_add(e[k].y, h[k]);
                            if (base + k * (int)blockDim.x < nf && st_g(se[k]) == e[k].y) split(e[k]);
                        }
                    }
                    recheck = false;
                } else {
                    for (int64_t i = threadIdx.x; i < nf; i += blockDim.x) {
                        const uint4 e = __ldcg(fcur + i);
                        if (KEEP || e.z < ft) split(e);
                    }
                }
                __syncthreads();
                nfar0 = c_alt;
                m = min(cnt[wv % 3], cap);
                uint4 *t = fcur;
                fcur = falt;
                falt = t;
                flip ^= 1;
                if (threadIdx.x == 0) c_far = 0;
                __syncthreads();
                if (m == 0) continue;  // far_min is known now: the next split moves something
                if (wide(wv % 3)) break;
            } else if (m == 0) {
                break;  // a large pile, or the cold tier's turn: the grid splits it
            }
        }
        int *push = &cnt[(wv + 1) % 3];
        if (threadIdx.x == 0) {
            cnt[(wv + 2) % 3] = 0;
            if (rows) arcs[(wv + 2) % 3] = longest[(wv + 2) % 3] = 0;
        }
        const uint64_t ft64 = (uint64_t)(*(volatile unsigned int *)&tg) + ht;
        const uint32_t ft = ft64 >= 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)ft64;
        auto to_far = [&](uint32_t v, uint32_t g, uint32_t f) {
            const int64_t p = nfar0 + atomicAdd(&c_far, 1);
            atomicMin(&far_min, f);
            if (p < B.cap_f) fcur[p] = make_uint4(v, g, f, 0u);
            else atomicOr(&ctl->status, ST_OVERFLOW);
        };
        for (int i = team; i < m; i += teams) {
            const uint4 en = cur[i];
            const int u = (int)en.x;
            const uint32_t gu = en.y;
            int j = (int)en.z + sub;
            const int r1 = (int)(en.w & ~SEG_END);
            // the first arcs load beside the label that decides about them
            uint2 a = j < r1 ? (G.oend ? __ldcg(G.arc + j) : __ldg(G.arc + j)) : make_uint2(0xFFFFFFFFu, 0u);
            const uint64_t su = __ldcg(B.state + u);
            const uint32_t hu = (ft < T || (KEEP && ft != 0xFFFFFFFFu)) ? H(u) : 0u;
            if (st_g(su) != gu || u == P.t) continue;
            if ((uint64_t)gu + hu >= ft) {
                // keep mode: stays open beyond f(t)
                if (KEEP && sub == 0) to_far((uint32_t)u, gu, sat_add(gu, hu));
                continue;
            }
            if ((int)en.w - (int)en.z > LOCAL_LONG && rows) {
                // (a segment's end is negative here)
                const int len = (int)en.w - (int)en.z, seg = max(LOCAL_LONG, (len + teams - 1) / teams);
                for (int k = sub; k * seg < len; k += lanes) {
                    const int b = (int)en.z + k * seg, p = atomicAdd(push, 1);
                    count_row((wv + 1) % 3, min(seg, r1 - b));
                    if (p < cap) nxt[p] = make_uint4(en.x, gu, (uint32_t)b, (uint32_t)min(b + seg, r1) | SEG_END);
                    else if (p < B.cap_q) qcur[p] = make_uint2(en.x, gu);  // (the grid walks the whole row)
                    else atomicOr(&ctl->status, ST_OVERFLOW);
                }
                if (sub == 0) {
                    n_exp++;
                    atomicMax(&longest[(wv + 1) % 3], (unsigned int)min(len, 1 << 21));
                }
                continue;
            }
            if (sub == 0) {
                n_exp += (int)en.w >= 0;  // (a row in segments was counted when it was cut)
                n_scan += (unsigned long long)(r1 - (int)en.z);
            }
            for (;;) {
                const int v = (int)a.x;
                const uint64_t ng64 = (uint64_t)gu + a.y;
                if (v >= 0 && ng64 < INF_G) {
                    const uint32_t ng = (uint32_t)ng64;
                    const uint64_t nv = st_make(ng, u);
                    uint64_t c0;
                    bool inst = false, first = false;
                    const int rb = row_begin(G.off, G.oend, v), re = row_end(G.off, G.oend, v);
                    uint32_t hv;
                    if (!KEEP && a.y != 0) {
                        // one atomic per arc (the asynchronous engine's latency
                        // form: over a positive arc a tie may swap the parent
                        // for an equal-cost one)
                        hv = H(v);
                        c0 = atomicMin(B.state + v, nv);
                        inst = ng < st_g(c0);
                    } else {
                        c0 = __ldcg(B.state + v);
                        hv = H(v);
                        if (KEEP ? hv < INF_G : (uint64_t)ng + hv < ft) {
                            while (ng < st_g(c0)) {
                                const uint64_t got = atomicCAS(B.state + v, c0, nv);
                                if (got == c0) {
                                    inst = true;
                                    break;
                                }
                                c0 = got;
                            }
                        }
                    }
                    if (inst) {
                        first = !P.no_touch_log && st_g(c0) >= INF_G;
                        if (v == P.t) atomicMin(&tg, ng);
                        const uint64_t fv = (uint64_t)ng + hv;
                        if (fv < T) {
                            n_rel++;
                            if (rows) count_row((wv + 1) % 3, re - rb);
                            const int p = atomicAdd(push, 1);
                            if (p < cap) nxt[p] = make_uint4((uint32_t)v, ng, (uint32_t)rb, (uint32_t)re);
                            else if (p < B.cap_q) qcur[p] = make_uint2((uint32_t)v, ng);  // past shared memory
                            else atomicOr(&ctl->status, ST_OVERFLOW);
                        } else if (KEEP || fv < ft) {
                            n_rel++;
                            to_far((uint32_t)v, ng, fv >= 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)fv);
                        }
                        if (first) {
                            const int p = touch0 + atomicAdd(&c_touch, 1);
                            if (p < G.n) B.touched[p] = v;
                            else atomicOr(&ctl->status, ST_OVERFLOW);
                        }
                    }
                }
                j += lanes;
                if (j >= r1) break;
                a = G.oend ? __ldcg(G.arc + j) : __ldg(G.arc + j);
            }
        }
        __syncthreads();
        wv++;
        m = cnt[wv % 3];
        uint4 *t = cur;
        cur = nxt;
        nxt = t;
        if (m > LOCAL_OUT || wv >= LOCAL_WAVES || nfar0 + c_far > B.cap_f / 2) break;
        if (rows) {
            work += arcs[wv % 3];
            if (wide(wv % 3) || work > LOCAL_WORK) break;
        }
        __syncthreads();  // every thread has read the counters
    }
    __syncthreads();
    // the entries left go back to the near list (those past the shared list
    // are there already)
    const int back = local_handback(m, cap, B.cap_q);
    for (int i = threadIdx.x; i < back; i += blockDim.x) {
        const uint4 en = cur[i];
        // of a row in segments (all of them are here) the first goes back as
        // the node, the others with a label that no node has
        const bool dead = (en.w & SEG_END) && (int)en.z != row_begin(G.off, G.oend, (int)en.x);
        qcur[i] = make_uint2(en.x, dead ? INF_G : en.y);
    }
    if (threadIdx.x == 0) {
        if (m > B.cap_q) atomicOr(&ctl->status, ST_OVERFLOW);
        ctl->loc_near = m;
        ctl->loc_far = (int)(nfar0 + c_far);
        ctl->loc_waves = wv;
        ctl->loc_T = T;
        ctl->loc_flip = flip;
        ctl->loc_done = done;
        ctl->far_scanned += n_far;
        ctl->touched = touch0 + c_touch;
    }
}

// One A* run on one slot, executed collectively by every thread of `grp`.
// KEEP: keep mode, every generated node stays open (no f(t) pruning), so that
// the state can be resumed after graph updates.  It is a template argument:
// as a word of P its code beside the plain mode's cost a maze query 4%
// (1.73 -> 1.80 ms).
// Precondition: slot state is all-ones (unreached) for every node.
template <bool KEEP = false, class Grp, class Heur>
__device__ SearchResult run_search(const Grp &grp, const DevGraph &G, const SlotBufs &B,
                                   const Heur &H, const SearchParams &P0, WarpRows *wrows) {
    SearchCtl *ctl = B.ctl;
    const int lane = lane_id();
    SearchParams P = P0;
    const uint32_t hs = H(P.s);
    if (hs < P.delta_loose) P.delta = P.delta_loose;
    const bool resume = KEEP && P.resume;
    WarpRows &wr = wrows[threadIdx.x >> 5];
    const bool has_diff = G.doff != nullptr;
    // words every thread needs after a barrier, read by one thread per CTA
    __shared__ struct {
        PhaseWords w;
        int status;
        uint32_t tg;
        int loc_near, loc_far, loc_waves, loc_flip, loc_done;
        uint32_t loc_T;
    } pc;
    __shared__ CtaFlush cf;

    if (grp.rank() == 0) {
        for (int i = 0; i < 4; i++) {
            ctl->ph[i] = PhaseWords{0, 0, 0xFFFFFFFFu, 0};
            ctl->ck[i] = 0;
        }
        ctl->iters = 0;
        ctl->expanded = ctl->scanned = ctl->relaxed = 0;
        ctl->far_scanned = 0;
        if (!resume) {
            ctl->cold_n = 0;
            ctl->touched = 1;
            B.state[P.s] = st_make(0, -1);
            B.touched[0] = P.s;
            B.q0[0] = make_uint2((uint32_t)P.s, 0u);
        }
    }
    const int64_t far_resume = resume ? (int64_t)(*(volatile int *)&ctl->far_n) : 0;
    const bool far_in_f1 = resume && (*(volatile int *)&ctl->far_sel) != 0;
    // cold tier (keep mode, resumed), as the last search left it
    int64_t ncold = resume && P.cold ? min((int64_t)*(volatile int *)&ctl->cold_n, P.cold_cap) : 0;
    uint32_t cold_x = ncold > 0 ? *(volatile unsigned int *)&ctl->cold_x : 0xFFFFFFFFu;
    auto read_tg = [&]() -> uint32_t { return P.t >= 0 ? st_g(__ldcg(B.state + P.t)) : 0xFFFFFFFFu; };
    grp.sync_fetch([&] { pc.tg = read_tg(); });

    uint2 *qcur = B.q0, *qnxt = B.q1;
    uint4 *fcur = far_in_f1 ? B.f1 : B.f0, *falt = far_in_f1 ? B.f0 : B.f1;
    int64_t nnear = resume ? 0 : 1, head = 0, nnext = 0, nfar = far_resume;
    uint32_t T = sat_add(hs, P.delta);
    uint32_t Tsplit = T;
    bool splitting = resume;
    if (resume) {
        T = 0;
        Tsplit = 0;  // the first split only measures the far pile's minimum f
    }
    // compaction: a split pass at the current T that only drops stale and
    // pruned far entries, run when the far pile fills up between splits
    bool compacting = false;
    int64_t far_after_compact = 0;
    unsigned long long n_exp = 0, n_scan = 0, n_rel = 0;
    int it = 0;
    int64_t waves = 0;  // phases that CTA 0 ran alone
    int status = 0;
    const int64_t max_phases = 4 * (int64_t)G.n + (1 << 22);
    const uint32_t ht = P.t >= 0 ? H(P.t) : 0u;
    uint32_t tg = pc.tg;  // g(t): only decreases, so a stale value only prunes less
    // phases that CTA 0 may run alone
    const bool local_ok = Grp::multi && !has_diff && (P.K <= 0 || P.K >= LOCAL_OUT);
    // the first split of a resumed search: it takes the tier back when the two
    // piles hold half of what one can (their stale entries are dropped), moves
    // entries to the tier when the pile is more than CTA 0 can split, and is
    // CTA 0's otherwise
    bool cold_take = false, cold_pass = false;
    if (resume && P.cold) {
        cold_take = ncold > 0 && ncold + nfar > B.cap_f / 2;
        if (!cold_take && nfar > LOCAL_FAR_KEEP) {
            if (ncold == 0) cold_x = P.cold_x;
            cold_pass = cold_x != 0xFFFFFFFFu;
        }
    }
    if (resume && !cold_take && !cold_pass && local_ok && nfar <= LOCAL_FAR_KEEP) splitting = false;
    uint2 *cold_stage = reinterpret_cast<uint2 *>(wr.snr);

    for (;;) {
        if constexpr (Grp::multi) {
            if (!splitting && head == 0 && nnext == 0 && local_ok && nnear <= LOCAL_IN && nfar <= B.cap_f / 2) {
                if (grp.first_cta())
                    local_phases<KEEP>(G, B, H, P, wrows, qcur, (int)nnear, fcur, falt, nfar, T, ht,
                                 ncold > 0 ? cold_x : 0xFFFFFFFFu, n_exp, n_scan, n_rel);
                grp.sync_fetch([&] {
                    pc.loc_near = *(volatile int *)&ctl->loc_near;
                    pc.loc_far = *(volatile int *)&ctl->loc_far;
                    pc.loc_waves = *(volatile int *)&ctl->loc_waves;
                    pc.loc_flip = *(volatile int *)&ctl->loc_flip;
                    pc.loc_done = *(volatile int *)&ctl->loc_done;
                    pc.loc_T = *(volatile uint32_t *)&ctl->loc_T;
                    pc.status = *(volatile int *)&ctl->status;
                    pc.tg = read_tg();
                });
                nnear = pc.loc_near;
                nfar = pc.loc_far;
                T = pc.loc_T;
                if (pc.loc_flip) {
                    uint4 *t2 = fcur;
                    fcur = falt;
                    falt = t2;
                }
                waves += pc.loc_waves;
                status = pc.status;
                tg = pc.tg;
                if (status & (ST_OVERFLOW | ST_TIMEOUT)) break;
                if (pc.loc_done) break;  // no open node with f < f(t)
                if (it + waves > max_phases) {
                    if (grp.rank() == 0) atomicOr(&ctl->status, ST_TIMEOUT);
                    break;
                }
                if (nnear == 0) {
                    splitting = true;
                    Tsplit = sat_add(T, P.delta);
                } else if (nfar > B.cap_f / 2 && nfar - far_after_compact > B.cap_f / 8) {
                    compacting = true;
                    splitting = true;
                }
            }
        }
        const int PH = (it + 1) & 3, RS = (it + 3) & 3;
        const uint64_t ft64 = (uint64_t)tg + ht;
        const uint32_t ft = ft64 >= 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)ft64;
        int64_t end = 0;
        if (!splitting) {
            end = (P.K > 0) ? min(nnear, head + (int64_t)P.K) : nnear;
            int c_n = 0, c_f = 0, c_t = 0;  // staged pushes of this warp
            const Chunks ch(end - head, grp.warp(), grp.nwarps(), &ctl->ck[PH]);
            // claims are made one chunk ahead to hide their round trip
            int64_t cnext = ch.first;
            for (int64_t base = head + ch.size * cnext; base < end; base = head + ch.size * cnext) {
                cnext = ch.next(end);
                const int64_t idx = base + lane;
                int u = -1, rb = 0, bdeg = 0, drb = 0, deg = 0;
                uint32_t gu = 0;
                bool requeue = false;
                if (lane < ch.size && idx < end) {
                    const uint2 en = __ldcg(qcur + idx);
                    u = (int)en.x;
                    gu = en.y;
                    // independent loads issued together (speculatively for
                    // entries that turn out stale)
                    const uint64_t su = __ldcg(B.state + u);
                    // every near entry was pushed with f = g + h(u) < T
                    // (relaxations, split and compaction moves alike; T only
                    // grows), so while f(t) >= T the pop test f < f(t)
                    // passes without reading h again; keep mode re-derives it
                    const uint32_t hu = (ft < T || (KEEP && ft != 0xFFFFFFFFu)) ? H(u) : 0u;
                    const int r0 = row_begin(G.off, G.oend, u), r1 = row_end(G.off, G.oend, u);
                    int d0 = 0, d1 = 0;
                    if (has_diff) {
                        d0 = __ldcg(G.doff + u);
                        d1 = __ldcg(G.doff + u + 1);
                    }
                    if (st_g(su) == gu && u != P.t) {
                        if ((uint64_t)gu + hu < ft) {
                            rb = r0;
                            bdeg = r1 - r0;
                            drb = d0;
                            deg = bdeg + (d1 - d0);
                            n_exp++;
                        } else if (KEEP) {
                            requeue = true;  // stays open beyond f(t)
                        }
                    }
                }
                stage_push(requeue, make_uint4((uint32_t)u, gu, 0u, 0u), wr.sf, c_f, &ctl->ph[PH].fq,  // keep mode: f re-derived
                           fcur, nfar, B.cap_f, ctl, PH);
                int total;
                int ex = warp_excl_scan(deg, &total);
                wr.excl[lane] = ex;
                wr.rb[lane] = rb;
                wr.bdeg[lane] = bdeg;
                wr.drb[lane] = drb;
                wr.g[lane] = gu;
                wr.u[lane] = u;
                __syncwarp();
                n_scan += (lane == 0) ? (unsigned long long)total : 0ull;
                // ARCS arcs per lane per step; every stage issues all of its
                // loads / atomics before consuming any result
#ifndef DDP_ARCS
#define DDP_ARCS 2
#endif
                constexpr int ARCS = DDP_ARCS;
                for (int kb = 0; kb < total; kb += 32 * ARCS) {
                    int v[ARCS], o[ARCS];
                    uint32_t ng[ARCS], hv[ARCS];
                    uint64_t sv[ARCS], prev[ARCS];
                    bool live[ARCS], go[ARCS];
#pragma unroll
                    for (int r = 0; r < ARCS; r++) {
                        const int k = kb + 32 * r + lane;
                        live[r] = false;
                        v[r] = 0;
                        ng[r] = 0;
                        o[r] = 0;
                        if (k < total) {
                            o[r] = row_owner(wr, k);
                            const uint2 a = row_arc(G, wr, o[r], k, true);
                            v[r] = (int)a.x;
                            const uint64_t ng64 = (uint64_t)wr.g[o[r]] + a.y;
                            live[r] = v[r] >= 0 && ng64 < INF_G;
                            ng[r] = (uint32_t)ng64;
                        }
                    }
#pragma unroll
                    for (int r = 0; r < ARCS; r++) sv[r] = live[r] ? __ldcg(B.state + v[r]) : 0ull;
#pragma unroll
                    for (int r = 0; r < ARCS; r++) {
                        live[r] = live[r] && ng[r] < st_g(sv[r]);
                        hv[r] = live[r] ? H(v[r]) : 0u;
                    }
#pragma unroll
                    for (int r = 0; r < ARCS; r++) {
                        go[r] = live[r] && (KEEP ? hv[r] < INF_G : (uint64_t)ng[r] + hv[r] < ft);
                        prev[r] = go[r] ? atomicCAS(B.state + v[r], sv[r], st_make(ng[r], wr.u[o[r]])) : sv[r];
                    }
#pragma unroll
                    for (int r = 0; r < ARCS; r++) {
                        bool to_near = false, to_far = false, first = false;
                        if (go[r]) {
                            uint64_t cur = sv[r];
                            uint64_t got = prev[r];
                            bool won = got == cur;
                            // retry only when another relaxation got in between;
                            // one that is no longer better pushes nothing: entries
                            // pushed twice are expanded by two warps at once and
                            // would double again at every node they reach
                            while (!won && ng[r] < st_g(got)) {
                                cur = got;
                                got = atomicCAS(B.state + v[r], cur, st_make(ng[r], wr.u[o[r]]));
                                won = got == cur;
                            }
                            if (won) {
                                first = !P.no_touch_log && st_g(cur) >= INF_G;
                                const uint64_t fv = (uint64_t)ng[r] + hv[r];
                                if (fv < T) to_near = true;
                                else to_far = true;
                            }
                        }
                        if (to_near || to_far) n_rel++;
                        const uint2 en = make_uint2((uint32_t)v[r], ng[r]);
                        stage_push(to_near, en, wr.sn, c_n, &ctl->ph[PH].nq, qnxt, nnext, B.cap_q, ctl, PH);
                        stage_push(to_far, make_uint4(en.x, en.y, sat_add(ng[r], hv[r]), 0u), wr.sf, c_f,
                                   &ctl->ph[PH].fq, fcur, nfar, B.cap_f, ctl, PH);
                        // at most n first touches: the touched log never overflows
                        stage_push(first, v[r], wr.st, c_t, &ctl->touched, B.touched, 0, (int64_t)G.n, ctl, PH);
                    }
                }
                __syncwarp();
            }
            cta_flush(&cf, wr, wr.sn, c_n, &ctl->ph[PH].nq, qnxt, nnext, B.cap_q, wr.sf, c_f, &ctl->ph[PH].fq, fcur,
                      nfar, B.cap_f, c_t, &ctl->touched, B.touched, (int64_t)G.n, ctl, PH);
        } else {
            // split the far pile at Tsplit (or compact it at T).  Entries
            // carry f from their push: a split reads no node state, stale
            // entries are dropped when they are popped.  Keep mode (h may
            // have changed since the push) and compaction (which must drop
            // stale entries) re-check the state and h.
            const uint32_t thr = compacting ? T : Tsplit;
            const bool recheck = KEEP || compacting;
            // cold tier: added to here (first split of a resumed search), or
            // scanned with the pile once min(f(t), threshold) passes cold_x
            const bool to_cold = cold_pass && !compacting;
            const bool merge_cold = !compacting && ncold > 0 && (cold_take || (!to_cold && min(ft, thr) > cold_x));
            const int64_t nscan = nfar + (merge_cold ? ncold : 0);
            if (grp.rank() == 0) ctl->far_scanned += (unsigned long long)nscan;
            uint2 *dst = compacting ? qnxt : qcur;
            const int64_t dbase = compacting ? nnext : 0;
            unsigned int local_min = 0xFFFFFFFFu;
            int c_n = 0, c_f = 0, c_c = 0;
            // uniform work per entry: a fixed stride, no claims
            for (int64_t base = 32 * (int64_t)grp.warp(); base < nscan; base += 32 * (int64_t)grp.nwarps()) {
                const int64_t idx = base + lane;
                bool to_near = false, keep = false, cold = false;
                uint4 en = make_uint4(0u, 0u, 0u, 0u);
                if (idx < nscan) {
                    if (idx < nfar) {
                        en = __ldcg(fcur + idx);
                    } else {
                        const uint2 c = __ldcg(P.cold + (idx - nfar));
                        en = make_uint4(c.x, c.y, 0u, 0u);  // f re-derived below (keep mode)
                    }
                    bool live = true;
                    uint64_t f = en.z;
                    if (recheck) {
                        live = st_g(__ldcg(B.state + en.x)) == en.y;
                        if (live && to_cold && en.y >= cold_x) {
                            cold = true;  // f >= g >= cold_x: h is not read
                            live = false;
                        } else {
                            f = (uint64_t)en.y + H((int)en.x);
                            en.z = f >= 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)f;
                        }
                    }
                    if (live) {
                        if (f < ft && f < thr) {
                            to_near = true;
                        } else if (f < ft || (KEEP && f < INF_G)) {
                            keep = true;
                            local_min = min(local_min, (uint32_t)f);
                        }
                    }
                }
                stage_push(to_near, make_uint2(en.x, en.y), wr.sn, c_n, &ctl->ph[PH].nq, dst, dbase, B.cap_q, ctl, PH);
                // compaction never grows the pile
                stage_push(keep, en, wr.sf, c_f, &ctl->ph[PH].fq, falt, 0, B.cap_f, ctl, PH);
                if (to_cold)
                    stage_push(cold, make_uint2(en.x, en.y), cold_stage, c_c, &ctl->cold_n, P.cold, 0, P.cold_cap,
                               ctl, PH);
            }
            cta_flush(&cf, wr, wr.sn, c_n, &ctl->ph[PH].nq, dst, dbase, B.cap_q, wr.sf, c_f, &ctl->ph[PH].fq, falt, 0,
                      B.cap_f, 0, &ctl->touched, B.touched, (int64_t)G.n, ctl, PH);
            if (to_cold) stage_flush(cold_stage, c_c, &ctl->cold_n, P.cold, 0, P.cold_cap, ctl, PH);
            if (merge_cold) {
                ncold = 0;  // every cold entry was examined: none is left
                cold_x = 0xFFFFFFFFu;
                cold_take = false;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) local_min = min(local_min, __shfl_xor_sync(FULL, local_min, o));
            if (lane == 0 && local_min != 0xFFFFFFFFu) atomicMin(&ctl->ph[PH].mf, local_min);
        }

        grp.sync_fetch([&] {
            const int4 x = __ldcg(reinterpret_cast<const int4 *>(&ctl->ph[PH]));
            pc.w = PhaseWords{x.x, x.y, (unsigned int)x.z, x.w};
            pc.status = *(volatile int *)&ctl->status;
            pc.tg = read_tg();
        });
        if (grp.rank() == 0) {
            ctl->ph[RS] = PhaseWords{0, 0, 0xFFFFFFFFu, 0};
            ctl->ck[RS] = 0;
        }
        const int a = pc.w.nq, b = pc.w.fq;
        const unsigned int m = pc.w.mf;
        const int perr = pc.w.err;
        status = pc.status;
        tg = pc.tg;
        it++;
        if ((perr & ST_OVERFLOW) || (status & ST_TIMEOUT)) break;
        if (it + waves > max_phases) {
            // a search never needs this many phases; stop instead of spinning
            if (grp.rank() == 0) atomicOr(&ctl->status, ST_TIMEOUT);
            break;
        }
        if (compacting) {
            uint4 *t2 = fcur;
            fcur = falt;
            falt = t2;
            nfar = b;
            nnext += a;
            far_after_compact = nfar;
            compacting = false;
            splitting = false;
        } else if (!splitting) {
            nnext += a;
            nfar += b;
            head = end;
            if (head >= nnear) {
                uint2 *t2 = qcur;
                qcur = qnxt;
                qnxt = t2;
                nnear = nnext;
                nnext = 0;
                head = 0;
                if (nnear == 0) {
                    splitting = true;
                    Tsplit = sat_add(T, P.delta);
                }
            }
            if (!splitting && nfar > B.cap_f / 2 && nfar - far_after_compact > B.cap_f / 8) {
                compacting = true;
                splitting = true;  // the split code path runs the compaction
            }
        } else {
            uint4 *t2 = fcur;
            fcur = falt;
            falt = t2;
            nfar = b;
            nnear = a;
            head = 0;
            nnext = 0;
            if (cold_pass) {
                // pushes past the buffer raised an overflow (the loop ends below)
                ncold = min((int64_t)*(volatile int *)&ctl->cold_n, P.cold_cap);
                cold_pass = false;
            }
            // cold entries have f >= cold_x
            const uint32_t mall = ncold > 0 ? min(m, cold_x) : m;
            if (nnear > 0) {
                T = Tsplit;
                splitting = false;
            } else if ((nfar == 0 && ncold == 0) || mall >= ft) {
                break;  // no open node with f < f(t): done
            } else {
                Tsplit = sat_add(mall, P.delta);
            }
        }
        if (nnear > B.cap_q || nfar > B.cap_f) {
            if (grp.rank() == 0) atomicOr(&ctl->status, ST_OVERFLOW);
            break;  // uniform: every thread computed the same counts
        }
    }

    // fold per-thread counters
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        n_exp += __shfl_xor_sync(FULL, n_exp, o);
        n_rel += __shfl_xor_sync(FULL, n_rel, o);
        n_scan += __shfl_xor_sync(FULL, n_scan, o);
    }
    if (lane == 0) {
        if (n_scan) atomicAdd(&ctl->scanned, n_scan);
        if (n_exp) atomicAdd(&ctl->expanded, n_exp);
        if (n_rel) atomicAdd(&ctl->relaxed, n_rel);
    }
    if (grp.rank() == 0) {
        ctl->far_n = (int)nfar;
        ctl->far_sel = fcur == B.f1 ? 1 : 0;
        ctl->cold_n = (int)ncold;
        ctl->cold_x = cold_x;
    }
    grp.sync();
    SearchResult r;
    const uint64_t st_t = P.t >= 0 ? __ldcg(B.state + P.t) : ~0ull;
    const uint64_t c = (uint64_t)st_g(st_t) + (P.t >= 0 ? H(P.t) : 0u);
    r.cost = (st_g(st_t) >= INF_G || c >= INF_G) ? 0xFFFFFFFFu : (uint32_t)c;
    r.iters = (int)(it + waves);
    if (grp.rank() == 0) ctl->iters = r.iters;
    return r;
}

// Reverse BFS from `t` (hop counts to t), executed collectively by `grp`.
// Replaces GA_star/bfs_hx.cu: the level loop runs on the device (no per-level
// D2H of the frontier size), frontier expansion is warp-cooperative over
// reverse-CSR rows, and each node is claimed once with a CAS.
//
// tag == 0: hops[] is first filled with HOPS_INF and then holds plain levels.
// tag != 0: hops[] is not cleared; a word is valid for this run when its high
//   24 bits equal tag >> 8, its low 8 bits hold the level (so levels stop at
//   254).  This lets a batch slot reuse the array per query without a fill.
// budget > 0: the BFS stops after the first level at which it has reached
//   `budget` nodes.  Returns the cap for unreached nodes in hop units:
//   HOPS_INF when the BFS ran to completion (unreached = cannot reach t),
//   else L+1 with L the last level claimed (unreached nodes are at least
//   L+1 hops away), so min(hops, cap) x wmin stays admissible and consistent.
template <class Grp>
__device__ uint32_t run_bfs_hops(const Grp &grp, const DevGraph &G, const SlotBufs &B, int32_t t,
                                 WarpRows *wrows, uint32_t tag, int64_t budget, bool spare_q0 = false) {
    SearchCtl *ctl = B.ctl;
    const int lane = lane_id();
    WarpRows &wr = wrows[threadIdx.x >> 5];
    const bool has_diff = G.doff != nullptr;
    // frontier ping-pong: the two near queues, or (when q0 is the
    // asynchronous ring that must stay clean) q1 and the second far pile
    int *fa = spare_q0 ? reinterpret_cast<int *>(B.f1) : reinterpret_cast<int *>(B.q0);
    int *fb = reinterpret_cast<int *>(B.q1);
    const int64_t capf = 2 * (spare_q0 ? min(B.cap_q, B.cap_f) : B.cap_q);  // uint2 slots reused as ints
    const uint32_t max_lvl = tag ? 254u : 0xFFFFFFF0u;
    __shared__ struct {
        int nf, err, status;
    } pc;
    __shared__ CtaFlush cf;

    if (!tag)
        for (int64_t i = grp.rank(); i < G.n; i += grp.size()) B.hops[i] = HOPS_INF;
    if (grp.rank() == 0) {
        for (int i = 0; i < 4; i++) {
            ctl->ph[i] = PhaseWords{0, 0, 0xFFFFFFFFu, 0};
            ctl->ck[i] = 0;
        }
        ctl->bfs_scanned = 0;
        ctl->bfs_reached = 0;
    }
    grp.sync();
    if (grp.rank() == 0) {
        B.hops[t] = tag;  // level 0
        fa[0] = t;
    }
    grp.sync();
    int64_t nf = 1;
    uint32_t lvl = 0;
    int it = 0;
    unsigned long long b_reached = 1, b_scanned = 0;
    bool complete = true;
    while (nf > 0) {
        if (lvl >= max_lvl || (budget > 0 && (int64_t)b_reached >= budget)) {
            complete = false;
            break;
        }
        const int PH = (it + 1) & 3, RS = (it + 3) & 3;
        const uint32_t claim_val = tag | (lvl + 1);
        int c_b = 0;
        const Chunks ch(nf, grp.warp(), grp.nwarps(), &ctl->ck[PH]);
        int64_t cnext = ch.first;
        for (int64_t base = ch.size * cnext; base < nf; base = ch.size * cnext) {
            cnext = ch.next(nf);
            const int64_t idx = base + lane;
            int rb = 0, bdeg = 0, drb = 0, deg = 0;
            if (lane < ch.size && idx < nf) {
                int u = __ldcg(fa + idx);
                rb = row_begin(G.roff, G.roend, u);
                bdeg = row_end(G.roff, G.roend, u) - rb;
                deg = bdeg;
                if (has_diff) {
                    drb = __ldcg(G.droff + u);
                    deg += __ldcg(G.droff + u + 1) - drb;
                }
            }
            int total;
            int ex = warp_excl_scan(deg, &total);
            wr.excl[lane] = ex;
            wr.rb[lane] = rb;
            wr.bdeg[lane] = bdeg;
            wr.drb[lane] = drb;
            __syncwarp();
            if (lane == 0) b_scanned += (unsigned long long)total;
            for (int kb = 0; kb < total; kb += 32) {
                const int k = kb + lane;
                bool claim = false;
                int p = -1;
                if (k < total) {
                    const int o = row_owner(wr, k);
                    p = (int)row_arc(G, wr, o, k, false).x;
                    if (p >= 0) {
                        const uint32_t x = __ldcg(B.hops + p);
                        const bool seen = tag ? ((x & 0xFFFFFF00u) == tag) : (x != HOPS_INF);
                        if (!seen) claim = atomicCAS(B.hops + p, x, claim_val) == x;
                    }
                }
                stage_push(claim, p, wr.st, c_b, &ctl->ph[PH].nq, fb, 0, capf, ctl, PH);
            }
            __syncwarp();
        }
        cta_flush(&cf, wr, wr.st, c_b, &ctl->ph[PH].nq, fb, 0, capf, wr.sf, 0, &ctl->ph[PH].fq, B.f0, 0, B.cap_f, 0,
                  &ctl->touched, B.touched, (int64_t)G.n, ctl, PH);
        grp.sync_fetch([&] {
            pc.nf = *(volatile int *)&ctl->ph[PH].nq;
            pc.err = *(volatile int *)&ctl->ph[PH].err;
            pc.status = *(volatile int *)&ctl->status;
        });
        if (grp.rank() == 0) {
            ctl->ph[RS] = PhaseWords{0, 0, 0xFFFFFFFFu, 0};
            ctl->ck[RS] = 0;
        }
        nf = pc.nf;
        b_reached += (unsigned long long)nf;
        const int perr = pc.err, status = pc.status;
        it++;
        lvl++;
        int *tmp = fa;
        fa = fb;
        fb = tmp;
        if ((perr & ST_OVERFLOW) || (status & ST_TIMEOUT)) break;
    }
    if (lane == 0 && b_scanned) atomicAdd(&ctl->bfs_scanned, b_scanned);
    if (grp.rank() == 0) ctl->bfs_reached = b_reached;
    grp.sync();
    return complete ? HOPS_INF : lvl + 1;
}

// Parent walk t -> s into buf[0..bcap), t first; returns the length (0 when
// unreachable, -1 when the path is longer than buf).  One thread.
__device__ inline int32_t walk_path(const SlotBufs &B, int32_t s, int32_t t, int32_t *buf, int32_t bcap) {
    uint64_t st = __ldcg(B.state + t);
    if (st_g(st) >= INF_G) return 0;
    int32_t len = 0;
    for (int32_t c = t; c >= 0;) {
        if (len == bcap) return -1;
        buf[len++] = c;
        if (c == s) break;
        c = st_parent(st);
        if (c >= 0) st = __ldcg(B.state + c);
    }
    return len;
}

// Path of a finished search into path[0..cap) in s..t order, by one CTA;
// returns the length.  len: what walk_path left in buf (bcap ids in shared
// memory), copied out by all threads (reversing it in place took as long again
// as the walk); -1: too long for buf, one thread walks it twice.
__device__ inline int32_t write_path_cta(const SlotBufs &B, int32_t s, int32_t t, int32_t *path, int32_t cap,
                                         int32_t n, int *status, const int32_t *buf, int32_t len) {
    __shared__ int32_t s_len;
    if (len < 0) {
        if (threadIdx.x == 0) {
            int32_t l = 0;
            for (int32_t c = t; c >= 0 && l <= n; c = c == s ? -1 : st_parent(__ldcg(B.state + c))) l++;
            if (l > cap) atomicOr(status, ST_PATH_TRUNC);
            int32_t c = t;
            for (int32_t i = l - 1; i >= 0 && c >= 0; i--) {
                if (i < cap) path[i] = c;
                c = st_parent(__ldcg(B.state + c));
            }
            s_len = l;
        }
        __syncthreads();
        return s_len;
    }
    if (len > cap && threadIdx.x == 0) atomicOr(status, ST_PATH_TRUNC);
    for (int32_t i = threadIdx.x; i < len; i += blockDim.x)
        if (len - 1 - i < cap) path[len - 1 - i] = buf[i];
    __syncthreads();
    return len;
}

// Parent walk t -> s into path[0..cap) in s..t order; returns the length
// (0 when unreachable).  One thread.
__device__ inline int32_t write_path(const SlotBufs &B, int32_t s, int32_t t, int32_t *path,
                                     int32_t cap, int32_t n, int *status) {
    uint64_t st = __ldcg(B.state + t);
    if (st_g(st) >= INF_G) return 0;
    int32_t len = 0;
    int32_t c = t;
    while (c >= 0 && len <= n) {
        if (len < cap) path[len] = c;
        len++;
        if (c == s) break;
        c = st_parent(__ldcg(B.state + c));
    }
    if (len <= cap) {
        for (int32_t i = 0, j = len - 1; i < j; i++, j--) {
            int32_t x = path[i];
            path[i] = path[j];
            path[j] = x;
        }
    } else {
        // too long: second walk keeps the first `cap` ids in s..t order
        atomicOr(status, ST_PATH_TRUNC);
        c = t;
        for (int32_t i = len - 1; i >= 0 && c >= 0; i--) {
            if (i < cap) path[i] = c;
            c = st_parent(__ldcg(B.state + c));
        }
    }
    return len;
}

}  // namespace ddp
