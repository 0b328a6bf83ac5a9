// Bidirectional one-CTA search: a forward search from s over the CSR and a
// reverse search from t over the reverse CSR, run together by one CTA until
// they meet.  No per-graph table: the plain kind keys both searches by g,
// so on graphs of small hop diameter two balls of half the radius replace
// one ball of the full radius (orders of magnitude fewer nodes on random
// digraphs); on graphs with coordinates the searches may key by g plus the
// average of two coordinate potentials (bidirectional A*, section
// "potentials" below).
//
// Labels: each node has a record of two units, forward then reverse, each a
// (g, parent) label (reverse: successor toward t).  Loading v's record gives
// the label being relaxed and the other side's label for the meeting test;
// a label changes by one compare-and-swap of its unit.  Three layouts
// (section "record layouts" below):
//   RecDense   32 bytes per node (one DRAM sector), 16-byte units
//              {epoch, g, parent, 0}.  A unit whose epoch is not the current
//              query's reads as unreached, so a slot is never reset between
//              queries: each query only advances the slot's epoch.
//   RecPair16  16 bytes per node, a 64-bit (g << 32 | parent) word per
//              direction; two nodes share a sector, which pays where node
//              ids have spatial locality.  Needs a touched log and a reset.
//   RecHash    an open-addressing table of epoch-tagged records sized to the
//              settled set instead of n.
//
// Open set: a window of 32 bucket lists per direction (bucket = key / width)
// in the slot's far memory, written once per push and read once per pop, and
// a pile for entries past the window or past a list's room, which are put
// into lists when the window reaches them.  The search runs in waves.  A wave
// expands the children of the last one that fell into buckets already opened
// (kept in shared memory) and, while these are fewer than the CTA can expand
// at once, opens the smallest bucket of the advancing direction(s) as well.
// A small team of lanes expands one entry, so a wave costs the dependent
// loads of one entry (row bounds and record together, then arcs) however
// many it holds; draining each bucket to the end before the next is opened
// spent most waves on a few last children.
//
// Lazy labels (LAZY; graphs without coordinates): a relaxation pushes
// {node, g, parent} without touching the node's record; the label is
// installed when the entry is popped and found smaller.  A search of a random
// digraph pushes eight entries for each one it pops (35k against 4.5k at 4M
// nodes), so seven eighths of the random record reads and writes are never
// made.  The meeting test needs only the nodes that the other side settled:
// a bit filter per direction in shared memory answers "not settled" for most
// arcs, and only its hits read the record.  On graphs with coordinates nodes
// are reached from several sides and most relaxations do not improve, so
// labels are installed at once there (eager).
//
// Meeting: relaxing arc (u, v) in direction dir with v's other-side label
// finite offers mu = g(u) + w + g_other(v), kept with the arc's forward-side
// tail x (u forward, v reverse) in one 64-bit atomicMin (mu << 32 | x).
// Labels only decrease, so at the end some arc (x, y) of x's forward row
// has g_f(x) + w + g_r(y) == mu, and the path is s .. x (forward parents),
// y .. t (reverse successors).
//
// Balance: each direction keeps its own position, and a wave opens a bucket
// of direction d only while its open set is at most twice the other's (plus a
// little), so the search grows the smaller ball, as bidirectional Dijkstra
// expands the side with the smaller queue.  A query whose source has only
// heavy out-arcs then advances the forward side alone instead of letting the
// reverse ball grow far past the meeting radius.
//
// Stop rule (bidirectional Dijkstra; stated here for keys equal to g, and
// with 2 mu in place of mu for potential keys): between waves, every node
// with a forward distance below a (the smallest key of the next wave's
// children, or the edge of the smallest bucket not opened) is final and
// expanded, and likewise below b in reverse.  When
// a + b >= mu, a shorter s-t path P would hold an arc (x, y) with d_s(x) < a and
// d_t(y) < b; both ends were expanded with final labels, and whichever
// expansion came second saw the other's final label (a label, and its filter
// bit, are installed by atomics that complete before the node's arcs are
// walked, each install setting the bit itself, and records are read from L2),
// so mu <= len(P): no shorter path exists.  An empty direction also ends the
// search.  Within a wave the same bound prunes: an entry with key + (the other
// side's bound) >= mu is dropped, since a path through it either ends at a node
// the other side has yet to settle (length >= mu) or meets a settled node,
// which its arc offered.
#pragma once

#include "engine_async.cuh"

namespace ddp {

constexpr uint32_t DIR_BIT = 0x80000000u;
constexpr uint32_t NODE_MASK = 0x7FFFFFFFu;

constexpr int WAVE_LISTS = 32;     // bucket lists per direction (a power of two, one per lane)
constexpr int WAVE_NEAR = 1024;    // entries of one wave held in shared memory
constexpr int WAVE_ROOM = 4096;    // entries per list at most
// A wave of fewer children also opens a bucket.  4M nodes, 4,096 pairs: 16 ->
// 22 waves a query, 32 -> 20, 64 -> 18 but 7 % more expansions; 2048 x 2048
// maze, longest of 16: 16 -> 5,886 waves and 470k expansions, 32 -> 3,285 and
// 591k, 64 -> 2,530 and 792k (29.4, 20.0, 21.9 ms); buckets drained one by
// one: 12,949 waves, 524k, 42.6 ms.
constexpr int WAVE_FILL = 32;
// How many buckets past its smallest unexpanded key a direction may open.
// Without a limit a search that starts along a chain of single arcs opens a
// bucket per wave, and when its ball grows at last all of it counts as
// opened (4M nodes: 472k expansions and 33 ms for one such query, 15k and
// 1.3 ms with 2).  Frontiers on graphs with coordinates grow slowly and
// profit from more overlap (maze, 2 -> 25.9 ms, 8 -> 19.4, 16 -> 19.1).  On
// graphs with hubs (skewed_rows) none are opened ahead: once a hub is reached,
// its children up to the last bucket opened are expanded in one wave, and the
// other hubs with them (the digraph above, 2,000 pairs: up to 206,000 expansions
// for a query, 37 ms; 3,800 and 2.5 ms with none).
constexpr uint32_t WAVE_AHEAD = 2, WAVE_AHEAD_XY = 16;
constexpr int WAVE_FILTER = 1024;  // words of a direction's settled filter (32,768 bits)
// Long rows: a wave's teams are a few lanes, chosen for the number of its
// entries.  A row that would take its team more than LONG_STEPS steps goes to
// the next wave in segments instead, which are entries like others there, so
// that no wave waits for a hub.  With the rule on opening ahead below, a digraph
// of 200,000 nodes with degrees by a power law (rows up to 19,000 arcs): 300
// pairs 44.1 -> 1.08 ms, 2,000 81.4 -> 2.5, 500 requests served 53 -> 1.2.  On
// graphs without long rows it costs 1 % (4,096 pairs on 4M nodes 3.43 -> 3.47 ms);
// walking such rows in a pass of their own behind the wave cost 8-20 %, its code
// taking registers and instruction fetches from the wave loop.
constexpr int LONG_STEPS = 16;
constexpr int LONG_SEG = 256;   // arcs of a segment (more for rows of more than LONG_SEGS segments)
constexpr int LONG_SEGS = 1024;
constexpr uint32_t SEG_BIT = 0x40000000u;  // in an entry's node: a segment (graphs of at most 2^30 nodes)

// What a wave expands, decided between two waves by the CTA's first warp.
struct WavePlan {
    int m;                // children of the last wave
    int n[2];             // entries of the buckets opened now
    uint32_t c[2];        // last bucket opened, per direction
    uint32_t lo[2];       // first bucket of the lists' window
    uint32_t lim[2];      // keys below belong to opened buckets
    uint32_t lb[2];       // keys below are settled and expanded
    int act;              // 0: expand, 1: done, 2: the pile's turn
};

// Shared memory of one search.
struct WaveQ {
    unsigned long long mu;           // (best s-t length << 32) | forward-side tail of its arc
    WavePlan plan;
    int lcnt[2][WAVE_LISTS];         // entries pushed per bucket list (those past its room went to the pile)
    int near[3];                     // children per wave, rotating
    unsigned int near_min[3][2];     // their smallest key per direction
    int pile_n, pile_alt;            // entries in the pile; kept by the pass over it
    int pile_dir[2];                 // pile entries per direction
    unsigned int pile_min[2];        // their smallest key
    int status;
    int touched;
    int no_path;  // table potentials: t is known to be out of s's reach, the search starts empty
    long long spent;                 // entries expanded or dropped
    unsigned long long edge_mul;     // 2^64 / (2^32 / bucket width)
    uint32_t settled[2][WAVE_FILTER];  // lazy labels: filter over settled nodes
    uint4 list[2][WAVE_NEAR];
};

// Unit of node v in direction dir of a paired slot's records.
__device__ __forceinline__ uint4 *unit_ptr(unsigned long long *st, int v, uint32_t dir) {
    return reinterpret_cast<uint4 *>(st) + 2 * (size_t)v + dir;
}

// g of a unit, or INF_G when it belongs to another query.
__device__ __forceinline__ uint32_t unit_g(const uint4 &u, uint32_t ep) { return u.x == ep ? u.y : INF_G; }

__device__ __forceinline__ bool unit_eq(const uint4 &a, const uint4 &b) {
    return a.x == b.x && a.y == b.y && a.z == b.z && a.w == b.w;
}

// 128-bit compare-and-swap (PTX atom.cas.b128, sm_90 and later) on a
// 16-byte aligned unit; returns the unit's old value.  The first 64-bit
// operand of each pair is the low half ({x, y}), the second the high half.
__device__ __forceinline__ uint4 cas_unit(uint4 *addr, const uint4 &cmp, const uint4 &val) {
    const unsigned long long c0 = ((unsigned long long)cmp.y << 32) | cmp.x;
    const unsigned long long c1 = ((unsigned long long)cmp.w << 32) | cmp.z;
    const unsigned long long v0 = ((unsigned long long)val.y << 32) | val.x;
    const unsigned long long v1 = ((unsigned long long)val.w << 32) | val.z;
    unsigned long long o0, o1;
    asm volatile(
        "{\n\t.reg .b128 cc, vv, oo;\n\t"
        "mov.b128 cc, {%2, %3};\n\t"
        "mov.b128 vv, {%4, %5};\n\t"
        "atom.global.cas.b128 oo, [%6], cc, vv;\n\t"
        "mov.b128 {%0, %1}, oo;\n\t}"
        : "=l"(o0), "=l"(o1)
        : "l"(c0), "l"(c1), "l"(v0), "l"(v1), "l"(addr)
        : "memory");
    return make_uint4((uint32_t)o0, (uint32_t)(o0 >> 32), (uint32_t)o1, (uint32_t)(o1 >> 32));
}

// ---- record layouts ----------------------------------------------------------
// A layout maps node v to its record (two units, forward then reverse).
// find(v) returns the record or null when v has none this query; claim(v)
// returns it, creating it if needed (null when the table is full).
// keyw(v) is the forward unit's w field: 0 for dense records, the node id
// for hashed ones.

// Unit operations shared by the epoch-tagged layouts (16-byte units).
struct UnitOps16 {
    using U = uint4;
    static constexpr bool logs = false;  // no touched log: epochs retire the records
    __device__ static U ld(const U *p) { return __ldcg(p); }
    __device__ static void ld2(const U *p, U &f, U &r) {
        f = __ldcg(p);
        r = __ldcg(p + 1);
    }
    __device__ static uint32_t g(const U &u, uint32_t ep) { return unit_g(u, ep); }
    __device__ static int32_t link(const U &u) { return (int32_t)u.z; }
    __device__ static U make(uint32_t ep, uint32_t g, uint32_t parent, uint32_t keyw) {
        return make_uint4(ep, g, parent, keyw);
    }
    __device__ static U cas(U *p, const U &cmp, const U &val) { return cas_unit(p, cmp, val); }
    __device__ static bool eq(const U &a, const U &b) { return unit_eq(a, b); }
};

// One record per node, at index v (the slot's state array holds n).
struct RecDense : UnitOps16 {
    static constexpr bool hashed = false;
    unsigned long long *st;
    __device__ uint4 *find(int v, uint32_t) const { return unit_ptr(st, v, 0); }
    __device__ uint4 *claim(int v, uint32_t) const { return unit_ptr(st, v, 0); }
    __device__ uint32_t keyw(int) const { return 0u; }
};

// One 16-byte pair per node: a 64-bit (g << 32 | parent) word per direction,
// all-ones = unreached.  Two nodes share a 32-byte sector, which pays where
// node ids have spatial locality (grids in row order, points in Morton
// order): a search's neighbours are then often in the same sector.  The
// price is a touched log and a reset pass after each query (full-sector
// stores of the logged nodes' sectors).
struct RecPair16 {
    using U = unsigned long long;
    static constexpr bool hashed = false;
    static constexpr bool logs = true;
    unsigned long long *st;
    __device__ U *find(int v, uint32_t) const { return st + 2 * (size_t)v; }
    __device__ U *claim(int v, uint32_t) const { return st + 2 * (size_t)v; }
    __device__ uint32_t keyw(int) const { return 0u; }
    __device__ static U ld(const U *p) { return __ldcg(p); }
    __device__ static void ld2(const U *p, U &f, U &r) {
        const ulonglong2 x = __ldcg(reinterpret_cast<const ulonglong2 *>(p));
        f = x.x;
        r = x.y;
    }
    __device__ static uint32_t g(const U &u, uint32_t) { return min(st_g(u), INF_G); }
    __device__ static int32_t link(const U &u) { return st_parent(u); }
    __device__ static U make(uint32_t, uint32_t g, uint32_t parent, uint32_t) {
        return st_make(g, (int32_t)parent);
    }
    __device__ static U cas(U *p, const U &cmp, const U &val) { return atomicCAS(p, cmp, val); }
    __device__ static bool eq(const U &a, const U &b) { return a == b; }
};

// Open addressing: 2^bits records, multiplicative hashing, linear probing.
// A record belongs to this query when its forward unit carries the epoch,
// and to node v when that unit's w field is v; records of other epochs are
// free.  A record is claimed by one 128-bit CAS of its forward unit to
// {epoch, unreached, no parent, v}; within a query records are never freed,
// so a probe for v ends at v's record or at the first free one.  This is the
// closed set of a search that touches far fewer nodes than the graph holds:
// the table is sized to the touched set, not to n.
constexpr int HASH_PROBES = 256;  // probe limit before the table counts as full
struct RecHash : UnitOps16 {
    static constexpr bool hashed = true;
    unsigned long long *st;
    uint32_t mask;
    int shift;  // 32 - bits
    __device__ uint32_t home(int v) const { return ((uint32_t)v * 0x9E3779B1u) >> shift; }
    __device__ uint4 *rec(uint32_t i) const { return unit_ptr(st, (int)i, 0); }
    __device__ uint4 *find(int v, uint32_t ep) const {
        uint32_t i = home(v);
        for (int k = 0; k < HASH_PROBES; k++, i = (i + 1) & mask) {
            const uint4 f = __ldcg(rec(i));
            if (f.x != ep) return nullptr;
            if (f.w == (uint32_t)v) return rec(i);
        }
        return nullptr;
    }
    __device__ uint4 *claim(int v, uint32_t ep) const {
        uint32_t i = home(v);
        for (int k = 0; k < HASH_PROBES; k++, i = (i + 1) & mask) {
            uint4 f = __ldcg(rec(i));
            if (f.x != ep) {
                const uint4 got = cas_unit(rec(i), f, make_uint4(ep, INF_G, 0xFFFFFFFFu, (uint32_t)v));
                if (unit_eq(got, f)) return rec(i);
                f = got;  // another thread claimed it meanwhile
            }
            if (f.x == ep && f.w == (uint32_t)v) return rec(i);
        }
        return nullptr;
    }
    __device__ uint32_t keyw(int v) const { return (uint32_t)v; }
};

// Path s..t from the meeting word; returns its length (0 when no path).
// Called by the CTA's first warp.  buf: two arrays of PATH_BUF node ids in
// shared memory.  The lanes test the arcs of the meeting row together, then
// lane 0 walks to s and lane 1 to t at the same time, once: a walk is a chain
// of dependent loads (three walks by one thread took 10-17 us a query on
// random digraphs, a tenth of its service time).
constexpr int PATH_BUF = 4096;
template <class Rec>
__device__ inline int32_t write_path_bidir(const DevGraph &G, const Rec &R, uint32_t ep, int32_t s, int32_t t,
                                           unsigned long long mu, int32_t *path, int32_t cap, int *status,
                                           int32_t *buf) {
    const uint32_t cost = uint32_t(mu >> 32);
    const int lane = lane_id();
    if (cost >= INF_G) return 0;
    if (s == t) {
        if (cap > 0 && lane == 0) path[0] = s;
        return 1;
    }
    // label of node v in direction dir (unit absent: unreached) and its
    // parent / successor
    auto lab = [&](int v, uint32_t dir, int32_t *link) -> uint32_t {
        const typename Rec::U *r = R.find(v, ep);
        if (!r) {
            *link = -1;
            return INF_G;
        }
        const typename Rec::U u = Rec::ld(r + dir);
        *link = Rec::link(u);
        return Rec::g(u, ep);
    };
    const int32_t x = int32_t(uint32_t(mu));
    int32_t lk;
    const uint32_t gx = lab(x, 0, &lk);
    int32_t y = -1;
    const int r1 = row_end(G.off, G.oend, x);
    for (int k0 = row_begin(G.off, G.oend, x); k0 < r1 && y < 0; k0 += 32) {
        const int k = k0 + lane;
        const uint2 a = k < r1 ? (G.oend ? __ldcg(G.arc + k) : __ldg(G.arc + k)) : make_uint2(0xFFFFFFFFu, 0u);
        bool hit = false;
        if ((int)a.x >= 0) {
            const uint32_t gr = lab((int)a.x, 1, &lk);
            hit = gr < INF_G && (uint64_t)gx + a.y + gr == cost;
        }
        const unsigned m = __ballot_sync(FULL, hit);
        if (m) y = __shfl_sync(FULL, (int)a.x, __ffs(m) - 1);
    }
    if (y < 0) {
        if (lane == 0) atomicOr(status, ST_TIMEOUT);  // no meeting arc: report the query failed
        return 0;
    }
    // Arcs of weight 0: the halves may share nodes (of a cycle of weight 0
    // through the meeting arc), each with both labels adding up to the cost.
    // The path leaves the forward half at the one nearest to s: no node before
    // it has such labels, so none is on its reverse half.
    int32_t jx = x, jy = y;  // where the halves join: jx -> jy
    if (G.wmin == 0) {
        int32_t len = 0, up;
        for (int32_t c = x; c >= 0 && len <= G.n; c = c == s ? -1 : up, len++) {
            const uint32_t gf = lab(c, 0, &up);
            if ((uint64_t)gf + lab(c, 1, &lk) == cost) {
                jx = c;
                jy = c == t ? -1 : lk;
            }
        }
    }
    // jx..s by forward parents (lane 0) and jy..t by reverse successors (lane 1)
    int32_t len = 0;
    if (lane < 2) {
        const int32_t end = lane ? t : s;
        for (int32_t c = lane ? jy : jx; c >= 0 && len <= G.n;) {
            if (len < PATH_BUF) buf[lane * PATH_BUF + len] = c;
            len++;
            if (c == end) break;
            lab(c, (uint32_t)lane, &lk);
            c = lk;
        }
    }
    __syncwarp();
    const int32_t lf = __shfl_sync(FULL, len, 0), lr = __shfl_sync(FULL, len, 1);
    if (lf + lr > cap && lane == 0) atomicOr(status, ST_PATH_TRUNC);
    if (lf <= PATH_BUF && lr <= PATH_BUF) {
        for (int32_t i = lane; i < lf; i += 32)
            if (lf - 1 - i < cap) path[lf - 1 - i] = buf[i];
        for (int32_t i = lane; i < lr; i += 32)
            if (lf + i < cap) path[lf + i] = buf[PATH_BUF + i];
    } else if (lane < 2) {
        // longer than the buffer: a second walk writes it
        int32_t i = lane ? lf : lf - 1;
        for (int32_t c = lane ? jy : jx; c >= 0 && i >= 0 && i < lf + lr; i += lane ? 1 : -1) {
            if (i < cap) path[i] = c;
            lab(c, (uint32_t)lane, &lk);
            c = lk;
        }
    }
    return lf + lr;
}

// ---- potentials (bidirectional A*) ------------------------------------------
// A potential pair gives, for node v, lower bounds pt(v) <= d(v, t) and
// ps(v) <= d(s, v), each consistent (|p(u) - p(v)| <= w(u, v) on every arc).
// The searches key their buckets by K_f(v) = 2 g_f(v) + pt(v) - ps(v) and
// K_r(v) = 2 g_r(v) + ps(v) - pt(v) (the average potentials, doubled to stay
// integral): both are non-negative and grow along arcs, so every proof of
// the plain engine holds on the keys, with the stop rule a + b >= 2 mu and
// pruning of a label g at v when g + pt(v) >= mu (forward) or
// g + ps(v) >= mu (reverse).  PotNone keeps the keys equal to g.
//
// slack: by how much a key may exceed the key of some consistent potential
// pair.  The proofs hold on the consistent keys, so the stop rule and the
// pruning allow for it on both sides: a + b >= 2 mu + 2 slack.
// table: the potentials are read from a table row per node, so they are
// evaluated only for relaxations that improve the label.
struct PotNone {
    static constexpr bool on = false, table = false;
    __device__ uint32_t slack() const { return 0u; }
    __device__ uint2 at(int) const { return make_uint2(0u, 0u); }
};

// floor(rho * |v - p|) in double precision: rho (16.16 fixed point, below
// min w / length over live arcs) makes the exact real potential consistent,
// and the rounding error (far below 1) cannot push a floor difference past
// an integer weight.
struct PotEuclid {
    static constexpr bool on = true, table = false;
    __device__ uint32_t slack() const { return 0u; }
    const int32_t *xy;
    int2 s, t;
    double rho;  // rho_fp / 65536
    __device__ uint32_t d1(const int2 &q, const int2 &p) const {
        const double dx = (double)q.x - p.x, dy = (double)q.y - p.y;
        const double h = floor(rho * sqrt(dx * dx + dy * dy));
        return h >= (double)(INF_G - 1) ? INF_G - 1 : (uint32_t)h;
    }
    __device__ uint2 at(int v) const {  // {pt(v), ps(v)}
        const int2 q = __ldg(reinterpret_cast<const int2 *>(xy) + v);
        return make_uint2(d1(q, t), d1(q, s));
    }
};

// wmin x Manhattan distance: consistent on grids whose arcs join
// 4-neighbours (length 1) with weights >= wmin.
struct PotManhattan {
    static constexpr bool on = true, table = false;
    __device__ uint32_t slack() const { return 0u; }
    const int32_t *xy;
    int2 s, t;
    uint32_t wmin;
    __device__ uint32_t d1(const int2 &q, const int2 &p) const {
        const uint64_t h = (uint64_t)wmin * (uint64_t)(abs(q.x - p.x) + abs(q.y - p.y));
        return h >= INF_G - 1 ? INF_G - 1 : (uint32_t)h;
    }
    __device__ uint2 at(int v) const {
        const int2 q = __ldg(reinterpret_cast<const int2 *>(xy) + v);
        return make_uint2(d1(q, t), d1(q, s));
    }
};

// Landmark bounds (HeurALT) to t and from s, from one read of v's row.  With
// table entries floor(d / sc) each bound lies at most 2 (sc - 1) below the
// exact landmark bound, which is consistent, and never above it: a key
// exceeds its consistent one by at most the error of the bound it subtracts.
//
// What an evaluation costs is its instructions.  With 8-bit entries the bytes
// of a row are spread into 16-bit halves and each difference is one
// add-and-maximum per pair (256 + a - b, floored at 256); the rows of t and s
// are prepared in shared memory in the form that the sums want (query_row).
// The unreachable marker (255, 65535) needs no test: as the subtracted entry it gives
// a negative difference, and as the one subtracted from it says that there is
// no path, for which every bound holds, or one of at least 255 scales.  The per-byte compare, subtract and
// maximum intrinsics, which the hardware does not have, took 2,000
// instructions per evaluation of 64 landmarks instead of 300.
struct PotALT {
    static constexpr bool on = true, table = true;
    HeurALT alt;  // alt.t: the target
    int32_t s;
    const uint4 *cf, *cb;  // 8-bit entries: the query's words (query_row)
    __device__ uint32_t slack() const { return 2u * (uint32_t)(alt.s - 1); }
    static constexpr uint32_t C256 = 0x01000100u;
    static __device__ __forceinline__ uint32_t lo16(uint32_t x) { return __byte_perm(x, 0u, 0x4140); }  // bytes 0, 1
    static __device__ __forceinline__ uint32_t hi16(uint32_t x) { return __byte_perm(x, 0u, 0x4342); }  // bytes 2, 3
    // Fills words (two per four landmarks: forward, then backward half):
    // {t, 256 - s} forward, {256 - t, s} backward.  All threads of a CTA; sets
    // *cut when a landmark proves that s cannot reach t (it reaches s and not
    // t, or t reaches it and s does not).
    static __device__ void query_row(const HeurALT &alt, int32_t s, uint4 *words, int *cut) {
        const int n4 = alt.L / 4;  // 4-byte words per half row
        const uint32_t *rt = reinterpret_cast<const uint32_t *>(alt.tab) + (size_t)alt.t * (2 * n4);
        const uint32_t *rs = reinterpret_cast<const uint32_t *>(alt.tab) + (size_t)s * (2 * n4);
        for (int i = threadIdx.x; i < 2 * n4; i += blockDim.x) {
            const uint32_t t = __ldg(rt + i), x = __ldg(rs + i);
            const uint32_t neg = i < n4 ? x : t, pos = i < n4 ? t : x;
            if (alt.cut() && (__vcmpeq4(pos, 0xFFFFFFFFu) & ~__vcmpeq4(neg, 0xFFFFFFFFu))) *cut = 1;
            words[i] = make_uint4(lo16(pos), hi16(pos), C256 - lo16(neg), C256 - hi16(neg));
        }
    }
    // four landmarks: f, b the row's forward and backward bytes
    __device__ __forceinline__ void word8(uint32_t f, uint32_t b, int i, uint32_t &mt, uint32_t &ms) const {
        const uint4 kf = cf[i], kb = cb[i];
        const uint32_t f0 = lo16(f), f1 = hi16(f), b0 = lo16(b), b1 = hi16(b);
        mt = __viaddmax_s16x2(kf.x, C256 - f0, mt);  // d(L, t) - d(L, v)
        mt = __viaddmax_s16x2(kf.y, C256 - f1, mt);
        ms = __viaddmax_s16x2(f0, kf.z, ms);         // d(L, v) - d(L, s)
        ms = __viaddmax_s16x2(f1, kf.w, ms);
        mt = __viaddmax_s16x2(b0, kb.z, mt);         // d(v, L) - d(t, L)
        mt = __viaddmax_s16x2(b1, kb.w, mt);
        ms = __viaddmax_s16x2(kb.x, C256 - b0, ms);  // d(s, L) - d(v, L)
        ms = __viaddmax_s16x2(kb.y, C256 - b1, ms);
    }
    __device__ __forceinline__ uint32_t bound8(uint32_t m) const {
        const uint32_t d = max(m & 0xFFFFu, m >> 16) - 256u;
        return d ? d * (uint32_t)alt.s - (uint32_t)(alt.s - 1) : 0u;
    }
    __device__ __forceinline__ uint2 eval8(int32_t v) const {
        const int n8 = alt.L / 8;  // 8-byte words per half row
        const uint2 *rv = alt.tab + (size_t)v * (2 * n8);
        uint32_t mt = C256, ms = C256;
        if ((n8 & 1) == 0) {
            const uint4 *qv = reinterpret_cast<const uint4 *>(rv);
#pragma unroll 2
            for (int i = 0; i < n8 / 2; i++) {
                const uint4 f = __ldg(qv + i), b = __ldg(qv + n8 / 2 + i);
                word8(f.x, b.x, 4 * i, mt, ms);
                word8(f.y, b.y, 4 * i + 1, mt, ms);
                word8(f.z, b.z, 4 * i + 2, mt, ms);
                word8(f.w, b.w, 4 * i + 3, mt, ms);
            }
        } else {
            for (int i = 0; i < n8; i++) {
                const uint2 f = __ldg(rv + i), b = __ldg(rv + n8 + i);
                word8(f.x, b.x, 2 * i, mt, ms);
                word8(f.y, b.y, 2 * i + 1, mt, ms);
            }
        }
        return make_uint2(bound8(mt), bound8(ms));
    }
    __device__ __forceinline__ uint2 eval16(int32_t v) const {
        const int W = alt.L / 4;  // 8-byte words per half row
        const uint2 *rv = alt.tab + (size_t)v * (2 * W);
        const uint2 *rt = alt.tab + (size_t)alt.t * (2 * W), *rs = alt.tab + (size_t)s * (2 * W);
        uint32_t mt = 0, ms = 0;
        auto fold = [](uint2 a, uint2 b, uint32_t &m) {
            m = __vmaxu2(m, __vsubus2(a.x, b.x));
            m = __vmaxu2(m, __vsubus2(a.y, b.y));
        };
#pragma unroll 2
        for (int i = 0; i < W; i++) {
            const uint2 f = __ldg(rv + i), b = __ldg(rv + W + i);
            fold(__ldg(rt + i), f, mt);
            fold(b, __ldg(rt + W + i), mt);
            fold(f, __ldg(rs + i), ms);
            fold(__ldg(rs + W + i), b, ms);
        }
        return make_uint2(alt.top<16>(mt), alt.top<16>(ms));
    }
    __device__ uint2 at(int v) const { return alt.bytes() ? eval8(v) : eval16(v); }
};

// Bucket key of label g in direction dir, with pot = {pt(v), ps(v)}.
template <class Pot>
__device__ __forceinline__ uint32_t bi_key(uint32_t g, uint32_t dir, uint2 pot) {
    if constexpr (!Pot::on) {
        return g;
    } else {
        const int64_t k = 2 * (int64_t)g + (dir ? (int64_t)pot.y - (int64_t)pot.x : (int64_t)pot.x - (int64_t)pot.y);
        return k <= 0 ? 0u : k >= 0xFFFFFFFFll ? 0xFFFFFFFFu : (uint32_t)k;
    }
}

// The key every open key must stay below to matter (keys of labels at or
// above mu's bound cannot lead to a shorter path).
template <class Pot>
__device__ __forceinline__ uint64_t bi_key_bound(uint32_t mu) {
    return Pot::on ? 2 * (uint64_t)mu : (uint64_t)mu;
}

// What an open entry holds: {node | dir << 31, key} and, with lazy labels, the
// parent, with potentials, the label g that the key was made from.
// Segment k of a long row: the entry with SEG_BIT, and k in the place of what
// it can do without: the parent with lazy labels (installed by now), the key
// in the short form (the label is read from the record).
template <bool LAZY, bool POT>
struct WaveEntry {
    using T = uint4;
    __device__ static T make(uint32_t vd, uint32_t key, uint32_t x) { return make_uint4(vd, key, x, 0u); }
    __device__ static uint32_t extra(const T &e) { return e.z; }
    __device__ static T segment(const T &e, uint32_t k) {
        return LAZY ? make_uint4(e.x | SEG_BIT, e.y, k, 0u) : make_uint4(e.x | SEG_BIT, e.y, e.z, k);
    }
    __device__ static uint32_t segment(const T &e) { return LAZY ? e.z : e.w; }
};
template <>
struct WaveEntry<false, false> {
    using T = uint2;
    __device__ static T make(uint32_t vd, uint32_t key, uint32_t) { return make_uint2(vd, key); }
    __device__ static uint32_t extra(const T &e) { return e.y; }  // no potentials: the key is g
    __device__ static T segment(const T &e, uint32_t k) { return make_uint2(e.x | SEG_BIT, k); }
    __device__ static uint32_t segment(const T &e) { return e.y; }
};

// Arcs of one segment of a row of len arcs.
__device__ __forceinline__ int long_seg(int len) {
    return len <= LONG_SEG * LONG_SEGS ? LONG_SEG : (len + LONG_SEGS - 1) / LONG_SEGS;
}

// ep: the slot's epoch for this query (never 0; units of other epochs read
// as unreached).
template <bool LAZY, class Pot, class Rec>
__device__ __forceinline__ SearchResult run_bidir_cta(const DevGraph &G, const SlotBufs &B, const SearchParams &P, uint32_t ep,
                                      WaveQ *q, const Pot &pot, const Rec &R) {
    static_assert(!(LAZY && Pot::on), "lazy labels are keyed by g");
    using WE = WaveEntry<LAZY, Pot::on>;
    using E = typename WE::T;
    SearchCtl *ctl = B.ctl;
    const int lane = lane_id();
    // arcs per lane whose loads are in flight together
    // (two 32-byte records per lane would not fit the registers)
    constexpr int AU = LAZY ? 4 : Pot::on || !Rec::logs ? 1 : 2;
    // (eager labels without potentials: coordinates, or a flooding search)
    const uint32_t seg_bit = G.n <= (int)SEG_BIT ? SEG_BIT : 0u, node_mask = NODE_MASK & ~seg_bit;
    const uint32_t ahead = P.skewed ? 0u : G.xy || (!LAZY && !Pot::on) ? WAVE_AHEAD_XY : WAVE_AHEAD;
    // the slot's far memory: 2 x 32 lists (at most a quarter), two halves of a
    // pile, two spill areas for waves that outgrow shared memory (a sixteenth
    // each)
    const int64_t total = 2 * B.cap_f * (int64_t)sizeof(uint2) / (int64_t)sizeof(E);
    const int room = (int)min(total / (8 * WAVE_LISTS), (int64_t)WAVE_ROOM);  // entries per list
    const int scap = (int)min(total / 16, (int64_t)0x0FFFFFFF);
    const int pcap = (int)min((total - (int64_t)2 * WAVE_LISTS * room - 2 * (int64_t)scap) / 2, (int64_t)0x3FFFFFFF);
    E *lists = reinterpret_cast<E *>(B.f0);
    E *pile0 = lists + (int64_t)2 * WAVE_LISTS * room;
    E *spill0 = pile0 + 2 * (int64_t)pcap;
    E *near0 = reinterpret_cast<E *>(q->list[0]);
    constexpr int NEAR_STRIDE = (int)(sizeof(q->list[0]) / sizeof(E));
    // keys are doubled with potentials: so is the bucket width
    const uint32_t dk = Pot::on ? 2 * P.delta : P.delta;
    constexpr uint32_t NONE = 0xFFFFFFFFu;
    // bucket of a key: one multiplication by 2^32 / width (buckets then are a
    // little wider than the width: what counts is that they grow with the
    // key and that edge(b) is the smallest key of bucket b)
    const uint32_t rec_dk = dk <= 1 ? NONE : (uint32_t)(0x100000000ull / dk);
    auto bucket = [&](uint32_t key) -> uint32_t { return __umulhi(key, rec_dk); };
    // ceil(b 2^32 / rec_dk): two multiplications by 2^64 / rec_dk come out at
    // most a few below it.  With a 64-bit division here, four in each plan,
    // the CTA waited about a microsecond longer for every wave: 16 maze pairs
    // 18 % longer, 200 pairs on 1M points 5, 4,096 on 4M nodes 3, 500 landmark
    // queries 7.
    if (threadIdx.x == 0) q->edge_mul = ~0ull / rec_dk;
    auto edge = [&](uint32_t b) -> uint32_t {
        const unsigned long long M = q->edge_mul;
        uint64_t k = (uint64_t)b * (uint32_t)(M >> 32) + (((uint64_t)b * (uint32_t)M) >> 32);
        while (k < NONE && bucket((uint32_t)k) < b) k++;
        return k >= NONE ? NONE : (uint32_t)k;
    };

    for (int i = threadIdx.x; i < 2 * WAVE_LISTS; i += blockDim.x) q->lcnt[0][i] = 0;
    if constexpr (LAZY)
        for (int i = threadIdx.x; i < 2 * WAVE_FILTER; i += blockDim.x) q->settled[0][i] = 0u;
    __syncthreads();
    if (threadIdx.x == 0) {
        ctl->iters = 0;
        ctl->expanded = ctl->scanned = ctl->relaxed = 0;
        ctl->far_scanned = 0;
        ctl->touched = 0;
        for (int i = 0; i < 3; i++) {
            q->near[i] = 0;
            q->near_min[i][0] = q->near_min[i][1] = NONE;
        }
        q->pile_n = 0;
        q->pile_dir[0] = q->pile_dir[1] = 0;
        q->pile_min[0] = q->pile_min[1] = NONE;
        q->status = room < 1 ? ST_OVERFLOW : 0;
        q->touched = 0;
        q->spent = 0;
        if (P.s == P.t) {
            q->mu = (unsigned long long)(uint32_t)P.s;  // length 0
        } else {
            q->mu = ~0ull;
            if constexpr (!LAZY) {
                typename Rec::U *rs = R.claim(P.s, ep);
                typename Rec::U *rt = R.claim(P.t, ep);
                rs[0] = Rec::make(ep, 0u, NONE, R.keyw(P.s));
                rt[1] = Rec::make(ep, 0u, NONE, 0u);
                if constexpr (Rec::logs) {
                    B.touched[0] = P.s;
                    B.touched[1] = P.t;
                }
                q->touched = 2;
            }
            const uint32_t ks = bi_key<Pot>(0u, 0u, pot.at(P.s)), kt = bi_key<Pot>(0u, 1u, pot.at(P.t));
            q->plan.lo[0] = bucket(ks);
            q->plan.lo[1] = bucket(kt);
            q->plan.c[0] = q->plan.lo[0] - 1;  // nothing opened yet
            q->plan.c[1] = q->plan.lo[1] - 1;
            if (room >= 1 && !(Pot::table && q->no_path)) {
                // lazy: no parent; else the label
                const uint32_t x = LAZY ? NONE : 0u;
                const int l0 = (int)(q->plan.lo[0] % WAVE_LISTS), l1 = (int)(q->plan.lo[1] % WAVE_LISTS);
                lists[(int64_t)l0 * room] = WE::make((uint32_t)P.s, ks, x);
                lists[(int64_t)(WAVE_LISTS + l1) * room] = WE::make((uint32_t)P.t | DIR_BIT, kt, x);
                q->lcnt[0][l0] = 1;
                q->lcnt[1][l1] = 1;
            }
        }
    }
    __syncthreads();
    if (P.s == P.t) {
        SearchResult r0;
        r0.cost = 0;
        r0.iters = 0;
        return r0;
    }

    bool flip = false;  // which half the pile is in
    unsigned long long n_exp = 0, n_scan = 0, n_rel = 0, n_far = 0;
    unsigned int n_first = 0;
    int wv = 0;
    const int64_t max_waves = 4 * (int64_t)G.n + (1 << 22);
    uint32_t lb0 = 0, lb1 = 0;

    // the length in mu (its high word: one 32-bit read)
    auto mu_now = [&]() -> uint32_t { return reinterpret_cast<volatile uint32_t *>(&q->mu)[1]; };
    const uint32_t slack2 = 2u * pot.slack();
    // the bound that a key must stay below, given the other side's lb
    auto key_limit = [&](uint32_t mu, uint32_t lbo) -> uint32_t {
        if constexpr (!Pot::on) return mu > lbo ? mu - lbo : 0u;
        const uint64_t kb = bi_key_bound<Pot>(mu) + slack2;
        return kb <= lbo ? 0u : (uint32_t)min(kb - lbo, (uint64_t)NONE);
    };
    uint32_t lim0 = 0, lim1 = 0, lo0 = 0, lo1 = 0;  // the wave's plan
    auto to_pile = [&](const E e, uint32_t key, uint32_t dir, int *count, E *pile) {
        const int p = atomicAdd(count, 1);
        if (p < pcap) pile[p] = e;
        else atomicOr(&q->status, ST_OVERFLOW);
        atomicAdd(&q->pile_dir[dir], 1);
        atomicMin(&q->pile_min[dir], key);
    };
    // appends e to bucket b's list, or (past the window, past its room) to the pile
    auto to_lists = [&](const E e, uint32_t key, uint32_t dir, uint32_t b, int *count, E *pile) {
        if (b - (dir ? lo1 : lo0) < (uint32_t)WAVE_LISTS) {
            const int l = (int)(dir * WAVE_LISTS + (b & (WAVE_LISTS - 1)));
            const int p = atomicAdd(&q->lcnt[0][l], 1);
            if (p < room) {
                lists[(int64_t)l * room + p] = e;
                return;
            }
        }
        to_pile(e, key, dir, count, pile);
    };
    // an entry of an opened bucket: wave w expands it
    auto to_near = [&](const E e, uint32_t key, uint32_t dir, int w) -> bool {
        const int p = atomicAdd(&q->near[w % 3], 1);
        if (p >= WAVE_NEAR + scap) return false;
        atomicMin(&q->near_min[w % 3][dir], key);
        if (p < WAVE_NEAR) near0[(w & 1) * NEAR_STRIDE + p] = e;
        else spill0[(int64_t)(w & 1) * scap + (p - WAVE_NEAR)] = e;
        return true;
    };
    auto push = [&](uint32_t vd, uint32_t key, uint32_t x) {
        const uint32_t dir = vd >> 31;
        const E e = WE::make(vd, key, x);
        if (key >= (dir ? lim1 : lim0)) to_lists(e, key, dir, bucket(key), &q->pile_n, pile0 + (flip ? pcap : 0));
        else if (!to_near(e, key, dir, wv + 1)) atomicOr(&q->status, ST_OVERFLOW);
    };
    // eager labels: installs label ng of v (seen with unit c) reached from u
    // and pushes its entry
    auto install = [&](uint32_t dir, int u, int v, uint32_t ng, uint2 pv, typename Rec::U c, uint32_t lbo) {
        const uint32_t nk = bi_key<Pot>(ng, dir, pv);
        if (ng >= Rec::g(c, ep) || nk >= key_limit(mu_now(), lbo)) return;
        const typename Rec::U nv = Rec::make(ep, ng, (uint32_t)u, dir ? 0u : R.keyw(v));
        typename Rec::U *rv = R.claim(v, ep);
        for (;;) {
            const typename Rec::U got = Rec::cas(rv + dir, c, nv);
            if (Rec::eq(got, c)) break;
            c = got;
            if (ng >= Rec::g(c, ep)) return;
        }
        n_rel++;
        if (Rec::g(c, ep) >= INF_G) {
            if constexpr (Rec::logs) {
                // first touches of either direction (a node may be logged
                // twice; the reset takes it twice)
                const int p = atomicAdd(&q->touched, 1);
                if ((int64_t)p < 2 * (int64_t)G.n) B.touched[p] = v;
            } else {
                n_first++;
            }
        }
        push((uint32_t)v | (dir << 31), nk, ng);
    };
    // whether a team of 2^tsh lanes leaves a row of len arcs to the next wave
    auto too_long = [&](int len, int tsh) -> bool {
        return len > max(2 * LONG_SEG, LONG_STEPS * AU << tsh) && seg_bit;
    };
    // lane sub of tw: its share of the segments of entry en (key, dir), a row of len arcs
    auto to_segments = [&](const E en, uint32_t key, uint32_t dir, int len, int sub, int tw) {
        const int seg = long_seg(len);
        for (int k = sub; k * (int64_t)seg < len; k += tw)
            if (!to_near(WE::segment(en, (uint32_t)k), key, dir, wv + 1)) atomicOr(&q->status, ST_OVERFLOW);
    };
    // expands one entry with a team of 2^tsh lanes
    auto expand = [&](const E en, const int tsh) {
        const int tw = 1 << tsh, sub = lane & (tw - 1);
        const uint32_t vd = en.x, key = en.y;
        const uint32_t dir = vd >> 31;
        const int u = (int)(vd & node_mask);
        const bool segment = (vd & seg_bit) != 0;
        const uint32_t lbo = dir ? lb0 : lb1;
        // row bounds load beside the record
        int r0 = dir ? row_begin(G.roff, G.roend, u) : row_begin(G.off, G.oend, u);
        int r1 = dir ? row_end(G.roff, G.roend, u) : row_end(G.off, G.oend, u);
        const uint2 *arcs = dir ? G.rarc : G.arc;
        uint2 a[AU];
        // (here, after the record's load: looking at the bounds any earlier
        // would wait for them first)
        auto cut = [&] {
            if (!segment) return;
            const int seg = long_seg(r1 - r0);
            r0 += (int)WE::segment(en) * seg;
            r1 = min(r1, r0 + seg);
        };
        auto load_arcs = [&](int j) {
#pragma unroll
            for (int k = 0; k < AU; k++)
                a[k] = j + k * tw < r1 ? (G.oend ? __ldcg(arcs + j + k * tw) : __ldg(arcs + j + k * tw))
                                       : make_uint2(NONE, 0u);
        };
        uint32_t gu;
        bool ok = false;
        if constexpr (LAZY) {
            gu = key;
            typename Rec::U *w = nullptr;
            typename Rec::U c{};
            if (segment) {
                ok = true;  // installed when the row was set aside
            } else if (sub == 0 && key < key_limit(mu_now(), lbo)) {
                typename Rec::U *rv = R.claim(u, ep);
                if (rv) {
                    w = rv + dir;
                    c = Rec::ld(w);
                } else {
                    atomicOr(&q->status, ST_OVERFLOW);  // the slot's table is full
                }
            }
            cut();
            load_arcs(r0 + sub);  // beside the label's compare-and-swap
            if (w) {
                const typename Rec::U nv = Rec::make(ep, gu, WE::extra(en), dir ? 0u : R.keyw(u));
                while (gu < Rec::g(c, ep)) {
                    const typename Rec::U got = Rec::cas(w, c, nv);
                    if (Rec::eq(got, c)) {
                        ok = true;
                        n_first += Rec::g(c, ep) >= INF_G;
                        // every install sets the bit, not the first alone:
                        // the thread of the first may not have come to it
                        // when a second, smaller label is installed and
                        // walked, and the other side would miss that one
                        const uint32_t h = ((uint32_t)u * 0x9E3779B1u) >> 17;
                        atomicOr(&q->settled[dir][h >> 5], 1u << (h & 31));
                        break;
                    }
                    c = got;
                }
                // label, then filter bit, then the walk over the arcs
                __threadfence_block();
            }
            ok = __shfl_sync(((1u << tw) - 1u) << (lane & ~(tw - 1)), (int)ok, lane & ~(tw - 1)) != 0;
        } else {
            gu = WE::extra(en);
            const typename Rec::U *ru = R.find(u, ep);
            const uint32_t gl = Rec::g(Rec::ld(ru + dir), ep);
            cut();
            load_arcs(r0 + sub);
            // current, and a path through it may still be shorter
            ok = gl == gu && key < key_limit(mu_now(), lbo);
        }
        if (!ok) return;
        if (too_long(r1 - r0, tsh) && !segment) {
            to_segments(en, key, dir, r1 - r0, sub, tw);
            return;
        }
        if (sub == 0) {
            n_exp++;
            n_scan += (unsigned long long)(r1 - r0);
        }
        for (int j = r0 + sub;;) {
            const uint32_t mu = mu_now();
            // weights below room keep g below min(mu, unreached)
            const uint32_t top = min(mu, INF_G), room_w = top > gu ? top - gu : 0u;
            const uint32_t lim = key_limit(mu, lbo);
            if constexpr (LAZY) {
#pragma unroll
                for (int k = 0; k < AU; k++) {
                    const int v = (int)a[k].x;
                    if (v < 0 || a[k].y >= room_w) continue;
                    const uint32_t ng = gu + a[k].y;
                    const uint32_t h = ((uint32_t)v * 0x9E3779B1u) >> 17;
                    const uint32_t f0 = *(volatile uint32_t *)&q->settled[0][h >> 5];
                    const uint32_t f1 = *(volatile uint32_t *)&q->settled[1][h >> 5];
                    if (((f0 | f1) >> (h & 31)) & 1u) {
                        // v may be settled: by this side (no need to come
                        // again) or by the other (the searches meet here)
                        const typename Rec::U *rv = R.find(v, ep);
                        if (rv) {
                            typename Rec::U uf, ur;
                            Rec::ld2(rv, uf, ur);
                            // both below 2^31
                            const uint32_t c = ng + Rec::g(dir ? uf : ur, ep);
                            if (c < mu) atomicMin(&q->mu, ((unsigned long long)c << 32) | (dir ? (uint32_t)v : (uint32_t)u));
                            if (Rec::g(dir ? ur : uf, ep) <= ng) continue;
                        }
                    }
                    if (ng >= lim) continue;
                    n_rel++;
                    push((uint32_t)v | (dir << 31), ng, (uint32_t)u);
                }
            } else {
                typename Rec::U uf[AU], ur[AU];
                uint2 pv[AU];  // {pt(v), ps(v)}
                bool live[AU];
                // every load of the step before any is used
#pragma unroll
                for (int k = 0; k < AU; k++) {
                    live[k] = (int)a[k].x >= 0 && a[k].y < room_w;
                    pv[k] = make_uint2(0u, 0u);
                    uf[k] = typename Rec::U{};
                    ur[k] = typename Rec::U{};
                    if (live[k]) {
                        Rec::ld2(R.find((int)a[k].x, ep), uf[k], ur[k]);
                        if constexpr (Pot::on && !Pot::table) pv[k] = pot.at((int)a[k].x);
                    }
                }
#pragma unroll
                for (int k = 0; k < AU; k++) {
                    const int v = (int)a[k].x;
                    const uint32_t ng = gu + a[k].y;
                    // a path through v is at least g + the bound of the other side
                    if (!live[k] || (Pot::on && !Pot::table && (uint64_t)ng + (dir ? pv[k].y : pv[k].x) >= (uint64_t)mu))
                        continue;
                    const uint64_t mc = (uint64_t)ng + Rec::g(dir ? uf[k] : ur[k], ep);
                    if (mc < mu) atomicMin(&q->mu, (mc << 32) | (dir ? (uint32_t)v : (uint32_t)u));
                    if constexpr (Pot::table) {
                        if (ng >= Rec::g(dir ? ur[k] : uf[k], ep)) continue;
                        pv[k] = pot.at(v);
                        const uint32_t hb = dir ? pv[k].y : pv[k].x;
                        if (hb >= INF_G || (uint64_t)ng + hb >= (uint64_t)mu) continue;
                    }
                    install(dir, u, v, ng, pv[k], dir ? ur[k] : uf[k], lbo);
                }
            }
            j += AU * tw;
            if (j >= r1) break;
            load_arcs(j);
        }
    };

    // Eager labels without potentials: the warp's entries together, one per
    // team (have: this lane's team has one).  Most relaxations fail, so the
    // teams' walks diverge: apart, 14 of 32 lanes were active and the compiler
    // could make it a fifth worse (200 pairs on 1M points: 30.8 or 37.4 ms);
    // stage by stage, with a step's compare-and-swaps in flight together, 26.9
    // ms.  Lazy labels and potentials lose by it (4M nodes: 3.68 -> 4.09 ms,
    // maze 18.6 -> 19.9 ms): their stages are short or rare.
    auto expand_warp = [&](const bool have, const E en, const int tsh) {
        const int tw = 1 << tsh, sub = lane & (tw - 1);
        const uint32_t dir = en.x >> 31;
        const int u = (int)(en.x & node_mask);
        const bool segment = (en.x & seg_bit) != 0;
        const uint32_t lbo = dir ? lb0 : lb1;
        const uint2 *arcs = dir ? G.rarc : G.arc;
        int r0 = 0, r1 = 0;
        uint32_t gl = 0;
        if (have) {
            // row bounds load beside the record
            r0 = dir ? row_begin(G.roff, G.roend, u) : row_begin(G.off, G.oend, u);
            r1 = dir ? row_end(G.roff, G.roend, u) : row_end(G.off, G.oend, u);
            gl = Rec::g(Rec::ld(R.find(u, ep) + dir), ep);
            if (segment) {
                const int seg = long_seg(r1 - r0);
                r0 += (int)WE::segment(en) * seg;
                r1 = min(r1, r0 + seg);
            }
        }
        const uint32_t gu = segment ? gl : WE::extra(en);  // a segment goes by the label as it is now
        uint2 a[AU];
        auto load_arcs = [&](int j) {
#pragma unroll
            for (int k = 0; k < AU; k++)
                a[k] = j + k * tw < r1 ? (G.oend ? __ldcg(arcs + j + k * tw) : __ldg(arcs + j + k * tw))
                                       : make_uint2(NONE, 0u);
        };
        load_arcs(r0 + sub);
        // current, and a path through it may still be shorter
        bool ok = have && gl == gu && gu < key_limit(mu_now(), lbo);
        if (ok && too_long(r1 - r0, tsh) && !segment) {
            to_segments(en, gu, dir, r1 - r0, sub, tw);
            ok = false;
        }
        if (ok && sub == 0) {
            n_exp++;
            n_scan += (unsigned long long)(r1 - r0);
        }
        for (int j = r0 + sub;; j += AU * tw) {
            const uint32_t mu = mu_now();
            const uint32_t top = min(mu, INF_G), room_w = ok && top > gu ? top - gu : 0u;
            const uint32_t lim = key_limit(mu, lbo);
            typename Rec::U uf[AU], ur[AU], got[AU];
            bool live[AU];
            // every load of the step before any is used
#pragma unroll
            for (int k = 0; k < AU; k++) {
                live[k] = (int)a[k].x >= 0 && a[k].y < room_w;
                uf[k] = typename Rec::U{};
                ur[k] = typename Rec::U{};
                if (live[k]) Rec::ld2(R.find((int)a[k].x, ep), uf[k], ur[k]);
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < AU; k++) {
                const uint32_t ng = gu + a[k].y;
                const uint32_t mc = ng + Rec::g(dir ? uf[k] : ur[k], ep);  // both below 2^31
                if (live[k] && mc < mu)
                    atomicMin(&q->mu, ((unsigned long long)mc << 32) | (dir ? a[k].x : (uint32_t)u));
                live[k] = live[k] && ng < Rec::g(dir ? ur[k] : uf[k], ep) && ng < lim;
            }
            // the step's atomics fly together.  Pairs: a minimum on (g, parent)
            // needs no second try (a tie may put an equal-cost parent in);
            // over an arc of weight 0 a tie could close a cycle of parents, so
            // those compare and swap, as the wider units do.  (Swaps with a
            // retry vote per arc, and the key limit in 64 bits per arc: 200
            // pairs on 1M points 20.4 -> 21.9 ms.)
#pragma unroll
            for (int k = 0; k < AU; k++) {
                got[k] = typename Rec::U{};
                if (!live[k]) continue;
                typename Rec::U *rv = R.claim((int)a[k].x, ep) + dir;
                const typename Rec::U nv = Rec::make(ep, gu + a[k].y, (uint32_t)u, 0u);
                if constexpr (Rec::logs) {
                    if (a[k].y != 0) {
                        got[k] = atomicMin(rv, nv);
                        continue;
                    }
                }
                got[k] = Rec::cas(rv, dir ? ur[k] : uf[k], nv);
            }
            bool again[AU], any = false;  // another relaxation came first
#pragma unroll
            for (int k = 0; k < AU; k++) {
                again[k] = live[k] && (!Rec::logs || a[k].y == 0) && !Rec::eq(got[k], dir ? ur[k] : uf[k]);
                any |= again[k];
            }
            if (__any_sync(FULL, any)) {
#pragma unroll
                for (int k = 0; k < AU; k++) {
                    // ends with the word that was replaced, or one that is no worse
                    while (again[k] && gu + a[k].y < Rec::g(got[k], ep)) {
                        const typename Rec::U c = got[k];
                        got[k] = Rec::cas(R.claim((int)a[k].x, ep) + dir, c,
                                          Rec::make(ep, gu + a[k].y, (uint32_t)u, 0u));
                        again[k] = !Rec::eq(got[k], c);
                    }
                    __syncwarp();
                }
            }
#pragma unroll
            for (int k = 0; k < AU; k++) {
                const int v = (int)a[k].x;
                const uint32_t ng = gu + a[k].y;
                const typename Rec::U c = got[k];
                const bool inst = live[k] && ng < Rec::g(c, ep);
                if (inst) {
                    n_rel++;
                    if (Rec::g(c, ep) >= INF_G) {
                        if constexpr (Rec::logs) {
                            // first touches of either direction (a node may be
                            // logged twice; the reset takes it twice)
                            const int p = atomicAdd(&q->touched, 1);
                            if ((int64_t)p < 2 * (int64_t)G.n) B.touched[p] = v;
                        } else {
                            n_first++;
                        }
                    }
                    push((uint32_t)v | (dir << 31), ng, ng);
                }
                __syncwarp();
            }
            const bool more = ok && j - sub + AU * tw < r1;
            if (!__any_sync(FULL, more)) break;
            load_arcs(more ? j + AU * tw : r1);
        }
    };

    for (;;) {
        __syncthreads();  // the last wave's pushes are in place
        if (threadIdx.x < 32) {
            // ---- plan the next wave ------------------------------------------
            // even lanes decide for the forward direction, odd lanes for the
            // backward one: the CTA waits, and an instruction that comes by
            // once a wave costs several cycles to fetch
            const uint32_t dir = lane & 1;
            const int cur = wv % 3;
            const int m = min(q->near[cur], WAVE_NEAR + scap);
            // the buckets opened are no longer in the window
            const uint32_t b0 = q->plan.c[0] + 1, b1 = q->plan.c[1] + 1;
            uint32_t lo = dir ? b1 : b0, c = lo - 1;
            int n = 0, act = 0;
            const int x0 = min(q->lcnt[0][(b0 + lane) & (WAVE_LISTS - 1)], room);
            const int x1 = min(q->lcnt[1][(b1 + lane) & (WAVE_LISTS - 1)], room);
            const unsigned m0 = __ballot_sync(FULL, x0 > 0), m1 = __ballot_sync(FULL, x1 > 0);
            const int first = __ffs(dir ? m1 : m0) - 1;
            const int pd = q->pile_dir[dir];
            const uint32_t nb = first >= 0 ? lo + (uint32_t)first : NONE;
            const uint32_t pm = pd ? q->pile_min[dir] : NONE;
            const uint32_t k = q->near_min[cur][dir];
            const uint32_t e = nb == NONE ? NONE : edge(nb);
            const uint32_t lb = min(min(k, pm), e), lbo = __shfl_xor_sync(FULL, lb, 1);
            const bool piled = __any_sync(FULL, pm < e);
            // an empty direction, or nothing open that could be shorter: mu is the distance
            if (lb == NONE || lbo == NONE || (uint64_t)lb + lbo >= bi_key_bound<Pot>(mu_now()) + slack2 || q->status) {
                act = 1;
            } else if (m >= WAVE_FILL) {
                // enough to do
            } else if (piled) {
                // the pile holds a direction's smallest bucket (a bucket whose
                // list was full leaves the rest there)
                act = 2;
                if (nb == NONE && pd && pm >= edge(lo)) lo = bucket(pm);  // nothing listed below
                c = lo - 1;
            } else {
                // open the next bucket of the direction(s) whose open set is
                // not much larger than the other's
                const int o0 = (int)__reduce_add_sync(FULL, (unsigned)x0), o1 = (int)__reduce_add_sync(FULL, (unsigned)x1);
                const int o = (dir ? o1 : o0) + pd, oo = __shfl_xor_sync(FULL, o, 1);
                const uint32_t nbo = __shfl_xor_sync(FULL, nb, 1);
                const int y0 = __shfl_sync(FULL, x0, first & 31), y1 = __shfl_sync(FULL, x1, first & 31);
                if (nb != NONE && ((int64_t)o <= 2 * (int64_t)oo + 64 || nbo == NONE) &&
                    (k == NONE || nb - bucket(k) <= ahead)) {
                    c = lo = nb;
                    n = dir ? y1 : y0;
                }
            }
            const int nn = (wv + 2) % 3;  // the counters of the wave after the next
            if (lane < 2) {
                q->plan.c[dir] = c;
                q->plan.lo[dir] = lo;
                q->plan.lb[dir] = lb;
                q->plan.lim[dir] = edge(c + 1);
                q->plan.n[dir] = n;
                // a bucket opened gives its list back after this wave: lo
                // keeps the bucket that would reuse it out of the window
                if (n) q->lcnt[dir][c & (WAVE_LISTS - 1)] = 0;
                q->near_min[nn][dir] = NONE;
            }
            const int n_both = n + __shfl_xor_sync(FULL, n, 1);
            if (lane == 0) {
                if (act == 0) {
                    q->spent += m + n_both;
                    if (P.budget > 0 && q->spent > P.budget) {
                        act = 1;
                        q->status = ST_BUDGET;
                    }
                }
                q->near[nn] = 0;
                q->plan.m = m;
                q->plan.act = act;
            }
        }
        __syncthreads();
        const int act = q->plan.act;
        lb0 = q->plan.lb[0];
        lb1 = q->plan.lb[1];
        lim0 = q->plan.lim[0];
        lim1 = q->plan.lim[1];
        lo0 = q->plan.lo[0];
        lo1 = q->plan.lo[1];
        if (act == 1) break;
        if (act == 2) {
            // put what the window covers of the pile into the lists, and
            // what belongs to buckets already opened into this wave
            const int n = min(q->pile_n, pcap);
            const uint32_t mu = mu_now();
            __syncthreads();
            if (threadIdx.x == 0) {
                q->pile_alt = 0;
                q->pile_dir[0] = q->pile_dir[1] = 0;
                q->pile_min[0] = q->pile_min[1] = NONE;
                n_far += (unsigned long long)n;
            }
            __syncthreads();
            const E *src = pile0 + (flip ? pcap : 0);
            E *dst = pile0 + (flip ? 0 : pcap);
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                const E e = __ldcg(src + i);
                const uint32_t dir = e.x >> 31;
                if (e.y >= key_limit(mu, dir ? lb0 : lb1)) continue;
                if (e.y >= (dir ? lim1 : lim0)) to_lists(e, e.y, dir, bucket(e.y), &q->pile_alt, dst);
                else if (!to_near(e, e.y, dir, wv)) to_pile(e, e.y, dir, &q->pile_alt, dst);
            }
            __syncthreads();
            if (threadIdx.x == 0) q->pile_n = q->pile_alt;
            flip = !flip;
            continue;  // plan again
        }
        if (wv >= max_waves) {
            if (threadIdx.x == 0) atomicOr(&ctl->status, ST_TIMEOUT);
            break;
        }
        // ---- the wave ---------------------------------------------------------
        const int m = q->plan.m, n0 = q->plan.n[0], n1 = q->plan.n[1];
        const E *l0 = lists + (int64_t)(q->plan.c[0] & (WAVE_LISTS - 1)) * room;
        const E *l1 = lists + (int64_t)(WAVE_LISTS + (q->plan.c[1] & (WAVE_LISTS - 1))) * room;
        const E *cur = near0 + (wv & 1) * NEAR_STRIDE;
        if (threadIdx.x == 0) n_far += (unsigned long long)(n0 + n1);
        const int W = m + n0 + n1;
        auto entry = [&](int i) -> E {
            if (i < m) return i < WAVE_NEAR ? cur[i] : __ldcg(spill0 + (int64_t)(wv & 1) * scap + (i - WAVE_NEAR));
            return i - m < n0 ? __ldcg(l0 + (i - m)) : __ldcg(l1 + (i - m - n0));
        };
        // lanes per entry: the wave's entries spread over the CTA, at least
        // two lanes each with lazy labels (a lane filters four arcs at once),
        // four otherwise (each arc is a record read and maybe a
        // compare-and-swap).  4M nodes, 4,096 pairs: 2 lanes 3.74 ms, 4 lanes
        // 4.36 ms, 1 lane 3.75 ms; 1M points, 200 pairs: 4 lanes 42.9 ms, 2
        // lanes 53.5 ms
        const int nt = (int)blockDim.x;
        const int tsh = W * 16 <= nt ? 4 : W * 8 <= nt ? 3 : (!LAZY || W * 4 <= nt) ? 2 : 1;
        const int teams = nt >> tsh;
        int i = (int)threadIdx.x >> tsh;
        const int lead = (int)(threadIdx.x & ~31u) >> tsh;  // the warp's first entry
        if constexpr (LAZY || Pot::on) {
            if (i < W) {
                E e = entry(i);
                for (;;) {
                    E en = e;
                    if (i + teams < W) en = entry(i + teams);  // loads while this one expands
                    expand(e, tsh);
                    i += teams;
                    if (i >= W) break;
                    e = en;
                }
            }
        } else if (lead < W) {
            E e{};
            if (i < W) e = entry(i);
            for (int b = lead; b < W; b += teams, i += teams) {
                E en{};
                if (i + teams < W) en = entry(i + teams);
                expand_warp(i < W, e, tsh);
                e = en;
            }
        }
        wv++;
    }
    if (threadIdx.x == 0 && q->status) atomicOr(&ctl->status, q->status);

#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        n_exp += __shfl_xor_sync(FULL, n_exp, o);
        n_scan += __shfl_xor_sync(FULL, n_scan, o);
        n_rel += __shfl_xor_sync(FULL, n_rel, o);
        n_first += __shfl_xor_sync(FULL, n_first, o);
    }
    if (lane == 0) {
        if (n_exp) atomicAdd(&ctl->expanded, n_exp);
        if (n_scan) atomicAdd(&ctl->scanned, n_scan);
        if (n_rel) atomicAdd(&ctl->relaxed, n_rel);
        if (n_first) atomicAdd(&ctl->touched, (int)n_first);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        ctl->iters = wv;
        ctl->far_scanned = n_far;
        if constexpr (Rec::logs) ctl->touched = (int)min((int64_t)q->touched, 2 * (int64_t)G.n);
    }
    __syncthreads();
    SearchResult r;
    const unsigned long long mw = *(volatile unsigned long long *)&q->mu;
    r.cost = uint32_t(mw >> 32) >= INF_G ? 0xFFFFFFFFu : uint32_t(mw >> 32);
    r.iters = wv;
    return r;
}

}  // namespace ddp
