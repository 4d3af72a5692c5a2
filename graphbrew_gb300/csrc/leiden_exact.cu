// leiden_exact.cu -- local moving with the reference's serial semantics.
//
// localMovingPhase<false> (bench/include/graphbrew/reorder/reorder_graphbrew.h:1588-1734)
// with one thread is a Gauss-Seidel sweep in vertex-id order: vertex u sees
// every move of the vertices before it.  This engine reproduces that sweep
// exactly with a sliding window of speculative decisions:
//
//   * the window [P, E) holds decisions D_prev from the previous round
//     (unknown for vertices that just entered);
//   * each round re-evaluates every window vertex u against the committed
//     state plus the D_prev moves of window vertices before u (neighbour
//     communities, affected flags and community totals at "time u");
//   * the first vertex x whose new decision differs from D_prev bounds the
//     exact prefix: all of [P, x] was evaluated from exact inputs (induction
//     from P), so it is committed; the rest carries its new decisions forward.
//
// Community totals at time u come from an event table rebuilt every round:
// each speculative move contributes (old, -k) and (new, +k) at its time, hashed
// by community.  A lookup adds up the community's events before u; the few
// communities with many events have theirs sorted by time and prefix-summed.
// All totals are exact integers, so every Delta-modularity equals the serial
// one whatever the order of the sums.
//
// Vertices above kBigMaxDeg ("hubs") are split into 1024-edge segments, each
// accumulated by its own CTA into the hub's global table, whose occupied slots
// are then scored in segments; the last CTA of a hub reduces the partial maxima.
// The whole round reads its window bounds from a device control block, so an
// iteration's rounds are one graph launch, or enqueued without waiting.
//
// The iteration's totalDelta decides the tolerance break; it is summed in a
// fixed tree order with a rigorous error bound and re-summed serially in
// vertex order only when the bound cannot settle the comparison.
#include <algorithm>
#include <cstdlib>
#include <cmath>
#include <vector>

#include "gb_common.cuh"
#include "gb_leiden_internal.cuh"

namespace gb {

namespace {

constexpr int kT = 256;
// Decision word of a window vertex: the community it moves to, or kNoMove, and
// whether the last evaluation changed it (vertex ids are below 2^31 - 1).
constexpr uint32_t kNoMove = 0x7FFFFFFFu;
constexpr uint32_t kChanged = 0x80000000u;
constexpr int kWindowMax = 65536;             // window vertices
constexpr int kEventsMax = 2 * kWindowMax;    // a departure and an arrival each
constexpr int kSlotBits = 18;
constexpr int kTableSlots = 1 << kSlotBits;   // hash slots, >= 2 x events
constexpr int kTbThreads = 256;               // table insert: one window vertex per thread
constexpr int kSortThreads = 512;             // sorting of the slots with many events
constexpr int kSortCtas = 2 * kNumSMs;
constexpr uint32_t kPadSlot = 0xFFFFFFFFu;
// Events of a slot: up to kInline of them lie at the slot, in any order (their
// sum is what a lookup wants), the others in blocks of kInline at slots of the
// same table, under names of their own: 1 << 31 | slot << kBlockBits | block.
constexpr int kInline = 16;
constexpr int kBlockBits = 13;
constexpr int kWarpSort = 64;                 // events of a slot that one warp sorts
static_assert(kTableSlots >= 2 * (kEventsMax + kEventsMax / kInline) * 15 / 16, "hash load factor near 1/2");
static_assert(kSlotBits + kBlockBits <= 31 && (kEventsMax / kInline) <= (1 << kBlockBits), "block names fit");
// Slots with many events ("hot": a community that many window vertices join
// or leave) get an index by time: a bit per window offset that has an event,
// and the events before each 32 offsets.
constexpr int kHotMin = 128;                  // events that make a slot hot
constexpr int kHotMax = kEventsMax / kHotMin;
constexpr int kHotWords = kWindowMax / 32;
constexpr int kBucketV = 16;                  // window vertices per bucket of a dense row
constexpr int kBucketStride = kWindowMax / kBucketV + 1;
// Designated communities: the few communities with the most events (on RMAT
// the one most vertices join) leave the table.  Each gets a dense row
// over the window (the signed degree of every window offset's move into or
// out of it) and the prefix of its 16-offset bucket sums, so a lookup is one
// prefix load plus one 64-byte read, and no slot of the table holds a giant
// community.  Chosen each round from the previous table's counts.
constexpr int kZMax = 8;                      // designated communities at most
constexpr int kZKeep = 64;                    // events a designated community needs to stay / be chosen
constexpr int kZCand = 128;                   // hot slots of the table considered
// CommRec.slotw: where the community's events of the current table are -- low
// bits of the table's generation, then a designated index or a hash slot.
constexpr int kSlotwTagShift = kSlotBits + 1;
constexpr uint32_t kSlotwDesig = 1u << kSlotBits;
constexpr int kHubThreads2 = 256;             // threads of the hub kernels
constexpr int kSmallMaxDeg = 32;              // rows up to this: a lane per neighbour
constexpr int kMidMaxDeg = 128;               // rows above that up to this: one warp each
constexpr int kLongThreads = 128;             // rows above that up to kWarpMaxDeg: one CTA of this size each
constexpr int kBigMaxDeg = 2048;              // rows above kWarpMaxDeg up to this: one CTA each
constexpr int kBigThreads = 512;
constexpr int kHubSeg = 4 * kHubThreads2;     // edges per hub-accumulation CTA (4 per thread)
constexpr int kTabSeg = 2 * kHubThreads2 - 1; // occupied slots per hub-selection CTA (2 per thread, one for the hub's own)
constexpr unsigned long long kNoChange = ~0ull;
constexpr int kIndexV = 64;                   // vertices per entry of the lists' index
constexpr int kIndexLists = 5;

struct Ctl {
    long long P, E, n;
    long long B, b_min;       // window length: at most B, at least b_min
    long long progress;       // mean of the vertices committed a round, x 64
    unsigned long long first_change;
    long long es0, es1;       // hub edge-segment range of the window
    long long ts0, ts1;       // hub table-segment range of the window
    long long ms0, ms1;       // mid-degree list range of the window
    long long ls0, ls1;       // long-row list range of the window
    long long bs0, bs1;       // big-row list range of the window
    long long c_bs0, c_bs1;   // big-row range of the last decided window
    long long round;
    long long evals;          // window vertices evaluated in this iteration
    long long cP, cX;         // committed range of the last decided window
    long long c_es0, c_es1;   // its hub edge-segment range
    long long c_ts0, c_ts1;   // its hub table-segment range
    long long pE;             // end of the last decided window: vertices from here on are new to this one
    long long max_rounds;     // bound on rounds per iteration (n + 1 always suffices)
    long long error;          // nonzero: the round loop stopped without finishing
    unsigned long long tag;   // generation of the event table (slots of older tags are empty)
    unsigned int nhot;        // hot slots of the current table
    unsigned int nmany[2];     // slots with more than kInline / more than kWarpSort events
    unsigned int sorted;       // events placed in the sorted arrays
    unsigned int nz;                 // designated communities of the current table
    unsigned int zc[kZMax];          // their ids
    unsigned int zcount[kZMax];      // events each received in the current table
};

// A slot's name, generation and count share one word, so that a claim is one
// compare-and-swap and an event's place one add.  The generation is the
// table's modulo 2^14 - 1, plus 1: the advance clears kClearSlots slots a round,
// the whole table in a fraction of that cycle, and 0 is no generation.
constexpr int kCountBits = 18;
constexpr int kClearSlots = 128;
struct __align__(16) SlotMeta {
    unsigned long long word;  // community id << 32 | generation << kCountBits | events
    int32_t start;            // more than kInline events: the first in the sorted arrays
    uint32_t hot;             // hot index + 1, 0 = search by time
};
static_assert(kEventsMax < (1 << kCountBits), "counts fit");
static_assert(2 * (kTableSlots / kClearSlots) < (1 << (32 - kCountBits)) - 1, "cleared before a generation returns");

// What an evaluation needs of a community, in one 16-byte load: its committed
// total, where its events of the current table are (if it has any) and the last
// round in which those events differ from the round before's.
struct __align__(16) CommRec {
    unsigned long long total;
    uint32_t slotw;
    uint32_t cver;
};

struct HubSeg {
    int32_t hub;      // index into the hub arrays
    int32_t part;     // segment number within the hub
};

struct ExactState {
    const int64_t* rp;
    const int32_t* col;
    const uint32_t* vcob;  // refinement bounds (localMovingPhase<true>), null otherwise
    uint32_t* vcom;
    CommRec* rec;         // per community
    uint8_t* vaff;
    uint8_t* mv;          // committed vertex moved (read by the affected-flag kernels)
    Ctl* ctl;
    uint32_t* dec[2];     // decision words, double-buffered by round parity
    double* delta;        // delta of the current decision (movers)
    double* final_delta;
    // event table
    SlotMeta* slots;      // kTableSlots
    uint2* ev;            // kTableSlots x kInline events: window offset, signed degree
    uint32_t* many[2];    // slots with more than kInline / more than kWarpSort events
    uint32_t* stime;      // slots with more than kInline events: times (vertex ids), sorted by time within the slot
    long long* epre;      // inclusive prefix of the signed degrees within the slot
    int32_t* sdeg;        // signed degrees (slots sorted by a CTA)
    uint2* hot_row;       // kHotMax x kHotWords: offsets with an event, events before the word
    uint8_t* zof;             // per community: designated index + 1, 0 = in the table
    int32_t* zcontrib;        // [2 parities][kZMax][kWindowMax] signed degree per window offset
    long long* zbsum;         // [2][kZMax][kBucketStride] 16-offset bucket sums
    long long* zpre;          // [2][kZMax][kBucketStride] exclusive prefix of the bucket sums
    unsigned long long* zcand;  // hot slots of the table: events << 32 | community
    // hubs
    const uint32_t* hub_v;        // hub vertex ids (ascending)
    const int64_t* hub_toff;      // table offset
    const uint32_t* hub_tcap;     // table capacity (pow2)
    const int32_t* hub_tfirst;    // first table segment index of each hub
    const int32_t* hub_tcount;    // table segments of each hub
    const HubSeg* eseg;           // edge segments (hub id order)
    const uint32_t* eseg_v;       // hub vertex of each edge segment
    long long n_eseg;
    const HubSeg* tseg;           // table segments
    const uint32_t* tseg_v;
    long long n_tseg;
    uint32_t* tkeys;              // hub tables (pool)
    uint32_t* tvals;
    int32_t* hub_any;
    int32_t* hub_done;
    uint32_t* hub_kud;            // edges of the hub into its own community (accumulated)
    uint32_t* hub_occ;            // per hub (pool offsets): slots of its table in insertion order
    uint32_t* hub_occn;           // per hub: occupied slots
    int32_t* hub_clr;             // per hub: table segments cleared this round
    double* part_d;               // per table segment
    uint32_t* part_c;
    const uint32_t* mid_v;        // vertices with kSmallMaxDeg < degree <= kMidMaxDeg (ascending)
    long long n_mid;
    const uint32_t* long_v;       // vertices with kMidMaxDeg < degree <= kWarpMaxDeg (ascending)
    long long n_long;
    const int32_t* list_index;    // per list of window_ranges: entries before each kIndexV-th vertex
    long long index_len;
    const uint32_t* big_v;        // vertices with kWarpMaxDeg < degree <= kBigMaxDeg (ascending)
    long long n_big;
    cudaGraphConditionalHandle cond;  // while-node condition (graph-driven rounds)
    int use_cond;
    double M, R;
    DqConst dq;
};

__device__ __forceinline__ uint32_t slot_hash(uint32_t c) {
    return (uint32_t)(((uint64_t)c * 0x9E3779B97F4A7C15ull) >> 40);
}

// The part of a slot's word above the count.
__device__ __forceinline__ unsigned long long slot_name(unsigned long long tag, uint32_t id) {
    constexpr uint32_t kCycle = (1u << (32 - kCountBits)) - 1u;
    return (unsigned long long)id << (32 - kCountBits) | ((uint32_t)tag % kCycle + 1u);
}

__device__ __forceinline__ CommRec load_rec(const ExactState& a, uint32_t c) {
    const uint4 v = *reinterpret_cast<const uint4*>(a.rec + c);
    CommRec r;
    r.total = (unsigned long long)v.y << 32 | v.x;
    r.slotw = v.z;
    r.cver = v.w;
    return r;
}

// Community totals at time u for K communities: the committed total plus the
// speculative events of c before u.  The community's record says whether it has
// events in this table at all -- most candidates have none, and their total is
// this one load (probing the hash for each cost a 16-byte read per candidate
// more, and the total and the designated index one read each: uniform 2^23
// took 225 us a round so) -- and where they are: a slot's few events, added up
// where they lie before u; a slot's time-sorted events, the last before u found
// by the hot index or by search; or a designated community's dense row.
// The K chains advance in lockstep so their loads are in flight together.  The
// record's generation is cut to its low bits, so what it points at is checked
// against the slot's name.  valid[k] = false entries return 0.
template <int K>
__device__ __forceinline__ void sigma_at_k(const ExactState& a, unsigned long long tag, long long P, int par,
                                           const uint32_t (&c)[K], const bool (&valid)[K], const CommRec (&rec)[K],
                                           uint32_t u, long long (&out)[K]) {
    int lo[K], l[K], r[K];
    int zd[K];
    SlotMeta sm[K];
    bool slot[K];
    bool any = false;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        out[k] = valid[k] ? (long long)rec[k].total : 0;
        const bool ev = valid[k] && (rec[k].slotw >> kSlotwTagShift) ==
                                        ((uint32_t)tag & ((1u << (32 - kSlotwTagShift)) - 1u));
        zd[k] = ev && (rec[k].slotw & kSlotwDesig) ? (int)(rec[k].slotw & (kZMax - 1)) : -1;
        slot[k] = ev && zd[k] < 0;
        any = any || ev;
    }
    if (!any) return;
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (slot[k]) sm[k] = a.slots[rec[k].slotw & (kTableSlots - 1)];
    const uint32_t off = (uint32_t)((long long)u - P);
    any = false;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        lo[k] = l[k] = r[k] = 0;
        if (slot[k] && sm[k].word >> kCountBits == slot_name(tag, c[k])) {
            const int cnt = (int)(sm[k].word & ((1u << kCountBits) - 1u));
            if (cnt <= kInline) {
                const uint4* q = reinterpret_cast<const uint4*>(
                    a.ev + (size_t)(rec[k].slotw & (kTableSlots - 1)) * kInline);
#pragma unroll 1
                for (int m = 0; m < cnt; m += 2) {
                    const uint4 x = q[m >> 1];
                    if (x.x < off) out[k] += (int32_t)x.y;
                    if (m + 1 < cnt && x.z < off) out[k] += (int32_t)x.w;
                }
            } else {
                lo[k] = sm[k].start;
                if (sm[k].hot > (uint32_t)kHotMax) {   // never written by a finished table
                    a.ctl->error = 2;
                } else if (sm[k].hot) {
                    const uint2 w = a.hot_row[(size_t)(sm[k].hot - 1) * kHotWords + (off >> 5)];
                    l[k] = r[k] = lo[k] + (int)w.y + __popc(w.x & ((1u << (off & 31)) - 1u));
                } else {
                    l[k] = lo[k];
                    r[k] = lo[k] + cnt;
                    any = true;
                }
            }
        }
        if (zd[k] >= 0 && (zd[k] >= (int)a.ctl->nz || a.ctl->zc[zd[k]] != c[k])) zd[k] = -1;
    }
    while (any) {
        uint32_t t[K];
        int mid[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            mid[k] = (l[k] + r[k]) >> 1;
            if (l[k] < r[k]) t[k] = a.stime[mid[k]];
        }
        any = false;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (l[k] < r[k]) {
                if (t[k] < u) l[k] = mid[k] + 1; else r[k] = mid[k];
                any = any || l[k] < r[k];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (l[k] > lo[k]) out[k] += a.epre[l[k] - 1];
    // Designated communities: bucket prefix + the bucket's offsets before u.
    const int bk = (int)(off >> 4), rem = (int)(off & 15u);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (zd[k] < 0) continue;
        const size_t row = (size_t)(par * kZMax + zd[k]);
        const int4* q = reinterpret_cast<const int4*>(a.zcontrib + row * kWindowMax + ((size_t)bk << 4));
        long long sum = a.zpre[row * kBucketStride + bk];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int4 v = q[m];
            if (4 * m + 0 < rem) sum += v.x;
            if (4 * m + 1 < rem) sum += v.y;
            if (4 * m + 2 < rem) sum += v.z;
            if (4 * m + 3 < rem) sum += v.w;
        }
        out[k] += sum;
    }
}

struct Round {
    long long P, E;
    long long cP, pE;     // start and end of the window before
    unsigned long long tag;
    int par;              // parity of the round (decision buffers and dense rows)
    const uint32_t* pdec;
    uint32_t* ndec;
};

__device__ __forceinline__ Round round_view(const ExactState& a, const Ctl* c) {
    Round r;
    r.P = c->P;
    r.E = c->E;
    r.cP = c->cP;
    r.pE = c->pE;
    r.tag = c->tag;
    const int par = (int)(c->round & 1);
    r.par = par;
    r.pdec = a.dec[par];
    r.ndec = a.dec[par ^ 1];
    return r;
}

// What u sees of its neighbour v: v's community at time u, whether v moves
// before u in this window, and whether v's decision is another one than in the
// round before (v may have been committed since: the window before reaches
// back to cP).
struct Seen {
    uint32_t c;
    bool moved, changed;
};

__device__ __forceinline__ Seen see(const ExactState& a, const Round& r, int64_t v, int64_t u) {
    Seen s{a.vcom[v], false, false};
    if (v >= r.cP && v < u) {
        const uint32_t w = r.pdec[v], to = w & kNoMove;
        s.changed = (w & kChanged) != 0;
        if (v >= r.P && to != kNoMove) {
            s.moved = true;
            s.c = to;
        }
    }
    return s;
}

__device__ __forceinline__ bool prev_mover(const ExactState& a, const Round& r, int64_t v) {
    return (r.pdec[v] & kNoMove) != kNoMove;
}

// Vertices that enter with this window (from pE on) have no decision yet: the
// insert kernel marks them, beside the hub accumulation.
__device__ __forceinline__ bool decided_before(const Round& r, int64_t v, int64_t u) {
    return v >= r.P && v < u && v < r.pE;
}

__device__ __forceinline__ uint32_t comm_at(const ExactState& a, const Round& r, int64_t v, int64_t u) {
    if (decided_before(r, v, u)) {
        const uint32_t to = r.pdec[v] & kNoMove;
        if (to != kNoMove) return to;
    }
    return a.vcom[v];
}

// Totals of each candidate lane's community c and of the group's own community
// d, one lookup per lane: a lane without a candidate (`idle`: those of the
// group; the same in its lanes) looks d up beside the others.  Only groups that
// have none take a second turn.  Every lane of the warp calls; `group` is the
// lane's group.
__device__ __forceinline__ void sigma_with_own(const ExactState& a, const Round& r, uint32_t u, bool cand, uint32_t c,
                                               const CommRec& rc, uint32_t d, const CommRec& rd, unsigned idle,
                                               unsigned group, long long& sc, long long& sd) {
    const int lane = threadIdx.x & 31;
    const int own = __ffs(idle ? idle : group) - 1;
    const bool first = idle != 0 && lane == own && d != kNone;
    long long o[1];
    {
        const uint32_t cc[1] = {cand ? c : d};
        const bool vv[1] = {cand || first};
        const CommRec rr[1] = {cand ? rc : rd};
        sigma_at_k<1>(a, r.tag, r.P, r.par, cc, vv, rr, u, o);
        sc = o[0];
    }
    long long mine = sc;
    if (__any_sync(0xFFFFFFFFu, idle == 0)) {
        const uint32_t cc[1] = {d};
        const bool vv[1] = {idle == 0 && lane == own};
        const CommRec rr[1] = {rd};
        sigma_at_k<1>(a, r.tag, r.P, r.par, cc, vv, rr, u, o);
        if (vv[0]) mine = o[0];
    }
    sd = __shfl_sync(0xFFFFFFFFu, mine, own);
}

// Whether the events of a community differ from the round before's (a mark of
// this round for the next may be there already: then once too often).
__device__ __forceinline__ bool comm_changed(const Round& r, const CommRec& rec) { return rec.cver >= (uint32_t)r.tag; }

// A vertex that the round before evaluated, with unchanged neighbours and
// unchanged communities, decides as it did: every input is the same, as a
// commit only turns decisions into state.
__device__ __forceinline__ void keep_decision(const Round& r, int64_t u) { r.ndec[u] = r.pdec[u] & kNoMove; }

// Refinement (scanCommunities<true>, RG:1392-1437): only neighbours inside
// u's bound count; ub = vcob[u] (0 when not refining).
__device__ __forceinline__ uint32_t bound_of(const ExactState& a, uint32_t u) { return a.vcob ? a.vcob[u] : 0u; }
__device__ __forceinline__ bool counts(const ExactState& a, int32_t v, uint32_t u, uint32_t ub) {
    return v != (int32_t)u && (a.vcob == nullptr || a.vcob[v] == ub);
}
// localMovingPhase<true> (RG:1663-1666): a vertex whose community already
// holds more than itself stays.
__device__ __forceinline__ bool refine_stays(const ExactState& a, double sigma_d, double ku) {
    return a.vcob != nullptr && sigma_d > __dmul_rn(ku, 1.001);
}

// Marks c as changed for the next round.  Designated communities change in
// nearly every round and are marked once by the advance (every mover storing
// to the one record of RMAT-22's giant community cost 80 us a round).
__device__ __forceinline__ void mark_changed(const ExactState& a, const Round& r, uint32_t c) {
    const uint32_t next = (uint32_t)r.tag + 1u;
    if (a.rec[c].cver != next && a.zof[c] == 0) a.rec[c].cver = next;
}

// cur: u's committed community; to: the community it moves to, or kNoMove.
__device__ __forceinline__ void record(const ExactState& a, const Round& r, int64_t u, uint32_t cur, uint32_t to,
                                       double delta) {
    // Only the move itself is visible to later vertices: "inactive",
    // "evaluated, stays" and "not yet evaluated" are the same input to them,
    // so only a different move is a change.
    const uint32_t prev = r.pdec[u] & kNoMove;
    const bool changed = to != prev;
    r.ndec[u] = to | (changed ? kChanged : 0u);
    if (to != kNoMove) a.delta[u] = delta;
    if (changed) {
        atomicMin(&a.ctl->first_change, (unsigned long long)u);
        // The events of these differ in the next table.
        if (to == kNoMove || prev == kNoMove) mark_changed(a, r, cur);
        if (to != kNoMove) mark_changed(a, r, to);
        if (prev != kNoMove) mark_changed(a, r, prev);
    }
}

__device__ __forceinline__ long long lower_bound_u32(const uint32_t* a, long long n, uint32_t key) {
    long long lo = 0, hi = n;
    while (lo < hi) {
        const long long mid = (lo + hi) >> 1;
        if (a[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// First index i in the ascending array a[0, n) with a[i] >= key, searched by
// one warp: 32 samples per step narrow the range 32-fold (4 steps for 2^20).
__device__ __forceinline__ long long warp_lower_bound_u32(const uint32_t* a, long long n, uint32_t key,
                                                         int lane) {
    long long lo = 0, hi = n;   // a[0, lo) < key; a[hi] >= key or hi == n
    while (hi - lo > 32) {
        const long long step = (hi - lo + 31) / 32;
        const long long p = lo + (long long)lane * step;
        const bool ge = p < hi ? a[p] >= key : true;
        const unsigned b = __ballot_sync(0xFFFFFFFFu, ge);   // lanes at or past hi vote true
        if (b == 0) {   // every sample < key: the bound lies past the last sample
            lo = lo + 31 * step + 1;
            continue;
        }
        const int f = __ffs(b) - 1;
        if (f == 0) return lo;
        const long long pf = lo + (long long)f * step;
        lo = lo + (long long)(f - 1) * step + 1;
        hi = min(hi, pf);
    }
    const long long p = lo + lane;
    const bool ge = p < hi ? a[p] >= key : true;
    const unsigned b = __ballot_sync(0xFFFFFFFFu, ge);
    return b ? lo + (__ffs(b) - 1) : hi;
}

// Window ranges of the hub segment lists and the mid, long and big-row lists
// for the window [P, E): ten searches on warps 0-9, within the entries of a block of
// kIndexV vertices (over the whole lists they took five dependent loads each, of an
// advance that every round waits for).
__device__ __forceinline__ void window_ranges(const ExactState& a, Ctl* c, long long P, long long E) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w >= 10) return;
    const uint32_t* arr = w < 2 ? a.eseg_v : (w < 4 ? a.tseg_v : (w < 6 ? a.mid_v : (w < 8 ? a.big_v : a.long_v)));
    const long long v = (w & 1) ? E : P;
    const long long len = w < 2 ? a.n_eseg : (w < 4 ? a.n_tseg : (w < 6 ? a.n_mid : (w < 8 ? a.n_big : a.n_long)));
    long long pos = 0;
    if (len) {
        const int32_t* ix = a.list_index + (size_t)(w >> 1) * a.index_len + (v / kIndexV);
        const long long lo = ix[0], hi = ix[1];
        pos = lo + warp_lower_bound_u32(arr + lo, hi - lo, (uint32_t)v, lane);
    }
    if (lane == 0) {
        switch (w) {
            case 0: c->es0 = pos; break;
            case 1: c->es1 = pos; break;
            case 2: c->ts0 = pos; break;
            case 3: c->ts1 = pos; break;
            case 4: c->ms0 = pos; break;
            case 5: c->ms1 = pos; break;
            case 6: c->bs0 = pos; break;
            case 7: c->bs1 = pos; break;
            case 8: c->ls0 = pos; break;
            default: c->ls1 = pos; break;
        }
    }
}

// ---------------------------------------------------------------------------
// Event table.  Each D_prev mover w of the window contributes two events at
// time w: (old community, -deg w) and (new community, +deg w).  A lookup needs,
// per community, the sum of its events before a time: no order, unless there
// are too many to read.  Built in two kernels:
//   insert: one thread per window vertex; movers find both communities' slots
//           in the generation-tagged hash (no clearing between rounds), take
//           their events' numbers there by one add per slot and warp, and
//           write the events to their places;
//   sort:   slots with more than kInline events: a warp each up to kWarpSort,
//           else a CTA, sorts them by time and prefix-sums them.
// Chains of a few dependent L2 round trips, 65,536 threads of them, bound both.
// (Grouping all events by slot first, stably, by a histogram, a scatter and a
// sort per bucket of slots, took 37 us a round where this takes 10 on a grid and 13 on planted communities
// of 300 K vertices.)
// ---------------------------------------------------------------------------
// Slot of `name` in the table, claiming one if absent (`claimed`); h: where to
// look first, cur: the word there.
__device__ __forceinline__ uint32_t table_slot(const ExactState& a, unsigned long long name, uint32_t h,
                                               unsigned long long cur, bool& claimed) {
    constexpr unsigned long long kGen = (1ull << (32 - kCountBits)) - 1ull;
    claimed = false;
    while (true) {
        const unsigned long long at = cur >> kCountBits;
        if (at == name) return h;
        if ((at ^ name) & kGen) {   // of an older generation: free
            const unsigned long long prev = atomicCAS(&a.slots[h].word, cur, name << kCountBits);
            claimed = prev == cur;
            if (claimed || prev >> kCountBits == name) return h;
            cur = prev;             // another community took the slot
        } else {
            h = (h + 1) & (kTableSlots - 1);
            cur = *(volatile unsigned long long*)&a.slots[h].word;
        }
    }
}

__device__ __forceinline__ uint32_t home_slot(uint32_t id) { return slot_hash(id) & (kTableSlots - 1); }

__device__ __forceinline__ uint32_t block_id(uint32_t slot, uint32_t number) {
    return 0x80000000u | slot << kBlockBits | (number - kInline) / kInline;
}

// Numbers of a warp's events in their slots (kPadSlot: none): one add per slot.
__device__ __forceinline__ uint32_t slot_number(const ExactState& a, uint32_t slot) {
    const int lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, slot);
    const int lead = __ffs(peers) - 1;
    uint32_t first = 0;
    if (slot != kPadSlot && lane == lead)
        first = (uint32_t)atomicAdd(&a.slots[slot].word, (unsigned long long)__popc(peers)) & ((1u << kCountBits) - 1u);
    first = __shfl_sync(0xFFFFFFFFu, first, lead);
    return first + __popc(peers & ((1u << lane) - 1u));
}

__device__ __forceinline__ void put_event(const ExactState& a, unsigned long long tag, uint32_t slot, uint32_t number,
                                          uint32_t off, int32_t sdeg) {
    uint32_t at = slot;
    if (number >= kInline) {
        const uint32_t id = block_id(slot, number), h = home_slot(id);
        bool claimed;
        at = table_slot(a, slot_name(tag, id), h, *(volatile unsigned long long*)&a.slots[h].word, claimed);
        if (number == kInline) a.many[0][atomicAdd(&a.ctl->nmany[0], 1u)] = slot;
        if (number == kWarpSort) a.many[1][atomicAdd(&a.ctl->nmany[1], 1u)] = slot;
    }
    a.ev[(size_t)at * kInline + number % kInline] = make_uint2(off, (uint32_t)sdeg);
}

__global__ void __launch_bounds__(kTbThreads) k_tb_insert(ExactState a) {
    const Ctl* c = a.ctl;
    const long long P = c->P, E = c->E;
    if (P >= c->n) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl->first_change = kNoChange;
    const Round r = round_view(a, c);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int W = (int)(E - P);
    if ((i & ~31) >= W) return;   // whole warps
    const int nz = (int)c->nz;
    uint32_t z0 = 0, z1 = 0;   // designated index + 1 of the departure / arrival community
    uint32_t s0 = kPadSlot, s1 = kPadSlot;
    int dg = 0;
    if (i < W) {
        const int64_t wv = P + i;
        const bool enters = wv >= r.pE;
        if (enters) a.dec[r.par][wv] = kNoMove;
        const uint32_t pb = enters ? kNoMove : r.pdec[wv] & kNoMove, vc = a.vcom[wv];
        const int64_t r0 = a.rp[wv], r1 = a.rp[wv + 1];
        if (pb != kNoMove) {
            dg = (int)(r1 - r0);
            const uint32_t h0 = home_slot(vc), h1 = home_slot(pb);
            const unsigned long long w0 = *(volatile unsigned long long*)&a.slots[h0].word;
            const unsigned long long w1 = *(volatile unsigned long long*)&a.slots[h1].word;
            if (nz) {
                z0 = a.zof[vc];
                z1 = a.zof[pb];
            }
            // The thread that claims a slot notes it in the community's record.
            bool claimed;
            if (!z0) {
                s0 = table_slot(a, slot_name(r.tag, vc), h0, w0, claimed);
                if (claimed) a.rec[vc].slotw = (uint32_t)r.tag << kSlotwTagShift | s0;
            }
            if (!z1) {
                s1 = table_slot(a, slot_name(r.tag, pb), h1, w1, claimed);
                if (claimed) a.rec[pb].slotw = (uint32_t)r.tag << kSlotwTagShift | s1;
            }
        }
    }
    const uint32_t n0 = slot_number(a, s0), n1 = slot_number(a, s1);
    if (s0 != kPadSlot) put_event(a, r.tag, s0, n0, (uint32_t)i, -dg);
    if (s1 != kPadSlot) put_event(a, r.tag, s1, n1, (uint32_t)i, dg);
    // Dense rows: every window offset writes its signed degree for each
    // designated community (zero when it does not move into or out of it), and
    // each 16-offset bucket (a half-warp) its sum; warp-aggregated event counts.
    for (int j = 0; j < nz; ++j) {
        const int v = (z1 == (uint32_t)j + 1 ? dg : 0) - (z0 == (uint32_t)j + 1 ? dg : 0);
        const size_t row = (size_t)(r.par * kZMax + j);
        if (i < W) a.zcontrib[row * kWindowMax + i] = v;
        long long sum = v;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
        if ((i & 15) == 0 && i < W) a.zbsum[row * kBucketStride + (i >> 4)] = sum;
        const int evs = __popc(__ballot_sync(0xFFFFFFFFu, z0 == (uint32_t)j + 1)) +
                        __popc(__ballot_sync(0xFFFFFFFFu, z1 == (uint32_t)j + 1));
        if ((i & 31) == 0 && evs) atomicAdd(&a.ctl->zcount[j], (unsigned)evs);
    }
}

// Event `number` of a slot of the finished table.
__device__ __forceinline__ uint2 get_event(const ExactState& a, unsigned long long tag, uint32_t slot,
                                           uint32_t number) {
    uint32_t at = slot;
    if (number >= kInline) {
        const uint32_t id = block_id(slot, number);
        const unsigned long long name = slot_name(tag, id);
        at = home_slot(id);
        int steps = 0;
        while (a.slots[at].word >> kCountBits != name && steps < kTableSlots) {
            at = (at + 1) & (kTableSlots - 1);
            ++steps;
        }
        if (steps == kTableSlots) a.ctl->error = 2;   // never in a finished table
    }
    uint2 e = a.ev[(size_t)at * kInline + number % kInline];
    e.x &= kWindowMax - 1;
    return e;
}

template <typename T>
__device__ __forceinline__ T warp_incl(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// Exclusive prefix of the CTA's values by thread; every thread calls.
__device__ __forceinline__ long long cta_excl(long long v, long long* warp_sum) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long incl = warp_incl(v);
    __syncthreads();
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    long long before = 0;
    for (int k = 0; k < w; ++k) before += warp_sum[k];
    return before + incl - v;
}

// Up to kWarpSort events of a slot by one warp: each lane counts the events
// before its two.
__device__ __forceinline__ void sort_slot_warp(const ExactState& a, const Round& r, uint32_t slot, int cnt,
                                               uint2* buf) {
    const int lane = threadIdx.x & 31;
    uint2 e[2];
    int pos[2] = {0, 0};
#pragma unroll
    for (int k = 0; k < 2; ++k)
        e[k] = lane + 32 * k < cnt ? get_event(a, r.tag, slot, lane + 32 * k) : make_uint2(0xFFFFFFFFu, 0u);
    int start = 0;
    if (lane == 0) start = (int)atomicAdd(&a.ctl->sorted, (unsigned)cnt);
    start = __shfl_sync(0xFFFFFFFFu, start, 0);
#pragma unroll 8
    for (int j = 0; j < 32; ++j) {
        const uint32_t x = __shfl_sync(0xFFFFFFFFu, e[0].x, j), y = __shfl_sync(0xFFFFFFFFu, e[1].x, j);
        pos[0] += (x < e[0].x) + (y < e[0].x);
        pos[1] += (x < e[1].x) + (y < e[1].x);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
        if (lane + 32 * k < cnt) buf[pos[k]] = e[k];   // a vertex is in a slot once
    __syncwarp();
    long long before = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int i = lane + 32 * k;
        const uint2 x = i < cnt ? buf[i] : make_uint2(0u, 0u);
        const long long incl = before + warp_incl((long long)(int32_t)x.y);
        if (i < cnt) {
            a.stime[start + i] = (uint32_t)(r.P + x.x);
            a.epre[start + i] = incl;
        }
        before = __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
    if (lane == 0) {
        a.slots[slot].start = start;
        a.slots[slot].hot = 0;
    }
    __syncwarp();
}

// Any number of events of a slot by one CTA: offsets with an event set their
// bit, and an event's place is the bits before its own.
__device__ __forceinline__ void sort_slot_cta(const ExactState& a, const Round& r, int words, uint32_t slot, int cnt,
                                              uint32_t* bits, uint32_t* before, long long* warp_sum) {
    __shared__ int s_start;
    __shared__ uint32_t s_hot;
    const int tid = threadIdx.x;
    constexpr int kPer = kHotWords / kSortThreads;
    for (int k = tid; k < words; k += kSortThreads) bits[k] = 0;
    if (tid == 0) {
        s_start = (int)atomicAdd(&a.ctl->sorted, (unsigned)cnt);
        s_hot = 0;
        if (cnt >= kHotMin) {
            const unsigned id = atomicAdd(&a.ctl->nhot, 1u);
            if (id < (unsigned)kHotMax) s_hot = id + 1;
            if (id < (unsigned)kZCand)
                a.zcand[id] = (unsigned long long)cnt << 32 | (uint32_t)(a.slots[slot].word >> 32);
        }
    }
    __syncthreads();
#pragma unroll 4
    for (int k = tid; k < cnt; k += kSortThreads) {
        const uint32_t off = get_event(a, r.tag, slot, k).x;
        atomicOr(&bits[off >> 5], 1u << (off & 31));
    }
    __syncthreads();
    uint32_t own = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k)
        if (tid * kPer + k < words) own += __popc(bits[tid * kPer + k]);
    uint32_t run = (uint32_t)cta_excl(own, warp_sum);
#pragma unroll
    for (int k = 0; k < kPer; ++k)
        if (tid * kPer + k < words) {
            before[tid * kPer + k] = run;
            run += __popc(bits[tid * kPer + k]);
        }
    __syncthreads();
    const int start = s_start;
    const uint32_t hot = s_hot;
#pragma unroll 4
    for (int k = tid; k < cnt; k += kSortThreads) {
        const uint2 e = get_event(a, r.tag, slot, k);
        const int at = start + (int)before[e.x >> 5] + __popc(bits[e.x >> 5] & ((1u << (e.x & 31)) - 1u));
        a.stime[at] = (uint32_t)(r.P + e.x);
        a.sdeg[at] = (int32_t)e.y;
    }
    if (hot)
        for (int k = tid; k < words; k += kSortThreads)
            a.hot_row[(size_t)(hot - 1) * kHotWords + k] = make_uint2(bits[k], before[k]);
    if (tid == 0) {
        a.slots[slot].start = start;
        a.slots[slot].hot = hot;
    }
    __syncthreads();
    long long carry = 0;
    for (int k0 = 0; k0 < cnt; k0 += 4 * kSortThreads) {
        int v[4];
        long long sum = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + 4 * tid + j;
            v[j] = k < cnt ? a.sdeg[start + k] : 0;
            sum += v[j];
        }
        const long long ex = cta_excl(sum, warp_sum);
        long long x = carry + ex;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + 4 * tid + j;
            x += v[j];
            if (k < cnt) a.epre[start + k] = x;
        }
        for (int k = 0; k < kSortThreads / 32; ++k) carry += warp_sum[k];
    }
    __syncthreads();
}

// Grid: kZMax designated-community prefixes, then kSortCtas over the slots with
// many events.
__global__ void __launch_bounds__(kSortThreads) k_tb_sort(ExactState a) {
    __shared__ uint32_t bits[kHotWords], before[kHotWords];
    __shared__ uint2 buf[kSortThreads / 32][kWarpSort];
    __shared__ long long warp_sum[kSortThreads / 32];
    static_assert(kHotWords % kSortThreads == 0, "bitmap words split evenly");
    const Ctl* c = a.ctl;
    if (c->P >= c->n) return;
    const Round r = round_view(a, c);
    const int tid = threadIdx.x, w = tid >> 5;
    if (blockIdx.x < kZMax) {
        // Designated community j: exclusive prefix of its bucket sums (one
        // extra entry holds the total).
        const int j = blockIdx.x;
        if (j >= (int)c->nz) return;
        const int nbk = (int)((r.E - r.P + kBucketV - 1) / kBucketV);
        const size_t row = ((size_t)r.par * kZMax + j) * kBucketStride;
        constexpr int kPer = kWindowMax / kBucketV / kSortThreads;
        long long v[kPer], own = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            v[k] = tid * kPer + k < nbk ? a.zbsum[row + tid * kPer + k] : 0;
            own += v[k];
        }
        long long run = cta_excl(own, warp_sum);
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            if (tid * kPer + k < nbk) a.zpre[row + tid * kPer + k] = run;
            run += v[k];
        }
        if (tid == kSortThreads - 1) a.zpre[row + nbk] = run;
        return;
    }
    const int words = (int)((r.E - r.P + 31) / 32);
    const unsigned n1 = c->nmany[1], n0 = c->nmany[0];
    const unsigned cta = blockIdx.x - kZMax, ctas = gridDim.x - kZMax;
    for (unsigned q = cta; q < n1; q += ctas) {
        const uint32_t slot = a.many[1][q];
        sort_slot_cta(a, r, words, slot, (int)(a.slots[slot].word & ((1u << kCountBits) - 1u)), bits, before, warp_sum);
    }
    for (unsigned q = w * ctas + cta; q < n0; q += ctas * (kSortThreads / 32)) {
        const uint32_t slot = a.many[0][q];
        const int cnt = (int)(a.slots[slot].word & ((1u << kCountBits) - 1u));
        if (cnt <= kWarpSort) sort_slot_warp(a, r, slot, cnt, buf[w]);
    }
}

constexpr int kMidWarpsPerBlock = 4;
constexpr int kSmallWarpsPerBlock = 8;

// Row of up to 32 neighbours by a warp: c is the lane's neighbour's community
// (kNone: none that counts), d the vertex's own; lanes of a community are ranked by
// __match_any_sync.
__device__ __forceinline__ void decide_small(const ExactState& a, const Round& r, int64_t u, int deg, uint32_t d,
                                             uint32_t c) {
    const int lane = threadIdx.x & 31;
    const CommRec rd = load_rec(a, d);
    const CommRec rc = c != kNone ? load_rec(a, c) : rd;
    if (a.vcob) {
        long long sg1 = 0;
        if (lane == 0) {
            const uint32_t cc[1] = {d};
            const bool vv[1] = {true};
            const CommRec rr[1] = {rd};
            long long o[1];
            sigma_at_k<1>(a, r.tag, r.P, r.par, cc, vv, rr, (uint32_t)u, o);
            sg1 = o[0];
        }
        sg1 = __shfl_sync(0xFFFFFFFFu, sg1, 0);
        if (refine_stays(a, (double)sg1, (double)deg)) {
            if (lane == 0) record(a, r, u, d, kNoMove, 0.0);
            return;
        }
    }
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, c);
    const int kud = __popc(__ballot_sync(0xFFFFFFFFu, c == d));
    const bool cand = c != kNone && c != d && lane == __ffs(peers) - 1;
    const unsigned idle = ~__ballot_sync(0xFFFFFFFFu, cand);
    long long sc = 0, sd = 0;
    sigma_with_own(a, r, (uint32_t)u, cand, c, rc, d, rd, idle, 0xFFFFFFFFu, sc, sd);
    double best_d = 0.0;
    uint32_t best_c = kNone;
    if (cand) {
        const double dl = delta_qi(a.dq, __popc(peers), kud, deg, sc, sd);
        if (dpos(dl)) { best_d = dl; best_c = c; }
    }
    warp_argmax_pos(best_d, best_c);
    if (lane == 0) {
        if (best_d > 0.0 && best_c != kNone && best_c != d) record(a, r, u, d, best_c, best_d);
        else record(a, r, u, d, kNoMove, 0.0);
    }
}

// Mid row (kSmallMaxDeg < degree <= kMidMaxDeg) by one warp: its neighbours'
// communities in one gather of up to four a lane, which also says whether anything
// that the vertex sees has changed; then a count per community in the warp's shared
// table.  One warp's chain of dependent loads bounds it, so the tables are small
// enough (2 KB) for the registers to limit the warps in flight, and longer rows go
// to CTAs: with 8 KB tables, up to three gathers and rows of up to 512, R-MAT-22's
// rounds spent 90 us here, now 33, and 26 on the longer rows beside it.
constexpr int kMidSlots = 2 * kMidMaxDeg;
__device__ __forceinline__ void eval_mid(const ExactState& a, const Round& r, int64_t u, int lane, uint32_t* tk,
                                         uint32_t* tv) {
    const int64_t rb = a.rp[u];
    const int deg = (int)(a.rp[u + 1] - rb);
    const bool aff = a.vaff[u] != 0;
    const uint32_t d = a.vcom[u], ub = bound_of(a, (uint32_t)u);
    int32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = 32 * k + lane < deg ? a.col[rb + 32 * k + lane] : -1;
    const CommRec rd = load_rec(a, d);
    bool dirty = u >= r.pE || comm_changed(r, rd), moved = false;
    uint32_t c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        c[k] = kNone;
        if (v[k] >= 0) {
            const Seen sv = see(a, r, v[k], u);
            moved |= sv.moved;
            dirty |= sv.changed;
            if (counts(a, v[k], (uint32_t)u, ub)) c[k] = sv.c;
        }
    }
    if (!__any_sync(0xFFFFFFFFu, dirty)) {
        uint32_t ver[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) ver[k] = c[k] != kNone ? a.rec[c[k]].cver : 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) dirty |= ver[k] >= (uint32_t)r.tag;
        if (!__any_sync(0xFFFFFFFFu, dirty)) {
            if (lane == 0) keep_decision(r, u);
            return;
        }
    }
    if (!aff && !__any_sync(0xFFFFFFFFu, moved)) {
        if (lane == 0) record(a, r, u, d, kNoMove, 0.0);
        return;
    }
    uint32_t H = 64;
    while (H < 2u * (uint32_t)deg) H <<= 1;
    const uint32_t mask = H - 1;
    for (uint32_t i = lane; i < H; i += 32) { tk[i] = kNone; tv[i] = 0; }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (32 * k >= deg) break;
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, c[k]);
        if (c[k] != kNone && lane == __ffs(peers) - 1) table_add(tk, tv, mask, c[k], (uint32_t)__popc(peers));
    }
    __syncwarp();
    const uint32_t kud = table_get(tk, tv, mask, d);
    // The candidate communities (c != d) to the front of the table, so that the
    // selection takes ceil((candidates + 1) / 32) lookup steps.
    uint32_t cnt = 0;
    for (uint32_t i0 = 0; i0 < H; i0 += 32) {
        const uint32_t x = tk[i0 + lane], y = tv[i0 + lane];
        const bool occ = x != kNone && x != d;
        const unsigned bal = __ballot_sync(0xFFFFFFFFu, occ);
        __syncwarp();
        if (occ) {
            const uint32_t pos = cnt + __popc(bal & ((1u << lane) - 1u));
            tk[pos] = x;
            tv[pos] = y;
        }
        cnt += __popc(bal);
        __syncwarp();
    }
    // One lookup per lane per step: lane 31 of the first step takes d's, the
    // other 31 candidates; every later step 32 (a second lookup per lane, for
    // d, doubled the step's instructions and registers).
    long long sd = 0;
    double best_d = 0.0;
    uint32_t best_c = kNone;
    for (uint32_t i0 = 0;; i0 += 32) {
        const bool own = i0 == 0 && lane == 31;
        const uint32_t i = i0 == 0 ? lane : i0 - 1 + lane;
        const bool valid = !own && i < cnt;
        const uint32_t cc[1] = {valid ? tk[i] : d};
        const bool vv[1] = {valid || own};
        const CommRec rr[1] = {valid ? load_rec(a, cc[0]) : rd};
        long long sg[1];
        sigma_at_k<1>(a, r.tag, r.P, r.par, cc, vv, rr, (uint32_t)u, sg);
        if (i0 == 0) sd = __shfl_sync(0xFFFFFFFFu, sg[0], 31);
        if (valid) {
            const double dl = delta_qi(a.dq, tv[i], kud, deg, sg[0], sd);
            if (dpos(dl) && better_pos(dl, cc[0], best_d, best_c)) { best_d = dl; best_c = cc[0]; }
        }
        if (i0 + 31 >= cnt) break;
    }
    __syncwarp();
    if (refine_stays(a, (double)sd, (double)deg)) best_c = kNone;   // every lane holds the same sd
    warp_argmax_pos(best_d, best_c);
    if (lane == 0) {
        if (best_d > 0.0 && best_c != kNone && best_c != d) record(a, r, u, d, best_c, best_d);
        else record(a, r, u, d, kNoMove, 0.0);
    }
}

// Small rows.  A warp takes four consecutive window vertices: rows of degree
// <= 8 are evaluated together by four 8-lane groups (one neighbour per lane).
// Of rows of degree 9..32 the neighbours' communities are gathered for all four at
// once, a lane per neighbour, and those that see a change are then decided one
// after another by the whole warp.  (Gathered one after another, with the change to mid
// rows: 8 M uniform vertices 268 ms, now 220.)
constexpr int kTinyDeg = 8;

__device__ __forceinline__ void eval_small_body(const ExactState& a, const Ctl* c) {
    const Round r = round_view(a, c);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane >> 3, j = lane & 7;
    const unsigned gmask = 0xFFu << (g * 8);
    const int wpb = (int)(blockDim.x >> 5);
    __shared__ uint32_t wide_c[kSmallWarpsPerBlock][4][32];
    const int64_t nw = (int64_t)gridDim.x * wpb;
    for (int64_t u0 = r.P + 4 * ((int64_t)blockIdx.x * wpb + w); u0 < r.E; u0 += 4 * nw) {
        const int64_t u = u0 + g;
        const bool inwin = u < r.E;
        int64_t rb = 0;
        int deg = 0;
        if (inwin) {
            rb = a.rp[u];
            deg = (int)(a.rp[u + 1] - rb);
        }
        const bool tiny = inwin && deg <= kTinyDeg, wide = inwin && !tiny && deg <= kSmallMaxDeg;
        // One load round for the row and its vertex state, one for its
        // neighbours' states, one for the communities they are in.
        int32_t v = -1;
        uint32_t d = kNone;
        bool aff = false;
        uint32_t ub = 0;
        if (tiny || wide) {
            if (tiny && j < deg) v = a.col[rb + j];
            d = a.vcom[u];
            aff = a.vaff[u] != 0;
            ub = bound_of(a, (uint32_t)u);
        }
        bool fresh = u >= r.pE;
        bool pm = false;
        uint32_t cv = kNone;
        CommRec rc{0ull, 0u, 0u}, rd = rc;
        if (tiny || wide) {
            rd = load_rec(a, d);
            fresh = fresh || comm_changed(r, rd);
        }
        bool dirty = tiny && fresh;
        if (v >= 0) {
            const Seen sv = see(a, r, v, u);
            pm = sv.moved;
            dirty = dirty || sv.changed;
            if (counts(a, v, (uint32_t)u, ub)) {   // not self loops (nor, refining, other bounds)
                cv = sv.c;
                rc = load_rec(a, cv);
                dirty = dirty || comm_changed(r, rc);
            }
        }
        const unsigned dirtyb = __ballot_sync(0xFFFFFFFFu, dirty);
        const bool redo = tiny && (dirtyb & gmask) != 0;
        if (tiny && !redo && j == 0) keep_decision(r, u);
        const unsigned pmb = __ballot_sync(0xFFFFFFFFu, pm);
        const bool act = redo && (aff || (pmb & gmask) != 0);
        // Refinement: the group's vertex stays when its community already holds more.
        bool stays = false;
        if (a.vcob) {
            long long sg1 = 0;
            if (redo && j == 0) {
                const uint32_t cc[1] = {d};
                const bool vv[1] = {true};
                const CommRec rr[1] = {rd};
                long long o[1];
                sigma_at_k<1>(a, r.tag, r.P, r.par, cc, vv, rr, (uint32_t)u, o);
                sg1 = o[0];
            }
            sg1 = __shfl_sync(0xFFFFFFFFu, sg1, lane & ~7);
            stays = redo && refine_stays(a, (double)sg1, (double)deg);
        }
        const uint32_t c = act ? cv : kNone;
        double best_d = 0.0;
        uint32_t best_c = kNone;
        if (dirtyb) {
            const unsigned peers = __match_any_sync(0xFFFFFFFFu, ((unsigned long long)g << 32) | c);
            const unsigned eqd = __ballot_sync(0xFFFFFFFFu, act && c != kNone && c == d) & gmask;
            const bool cand = act && c != kNone && c != d && lane == __ffs(peers) - 1;
            const unsigned idle = ~__ballot_sync(0xFFFFFFFFu, cand) & gmask;
            long long sc = 0, sd = 0;
            sigma_with_own(a, r, (uint32_t)u, cand, c, rc, act ? d : kNone, rd, act ? idle : gmask, gmask, sc, sd);
            if (cand) {
                const double dl = delta_qi(a.dq, __popc(peers), __popc(eqd), deg, sc, sd);
                if (dpos(dl)) { best_d = dl; best_c = c; }
            }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {   // argmax inside each 8-lane group
            const double od = __shfl_xor_sync(0xFFFFFFFFu, best_d, o);
            const uint32_t oc = __shfl_xor_sync(0xFFFFFFFFu, best_c, o);
            if (better_pos(od, oc, best_d, best_c)) { best_d = od; best_c = oc; }
        }
        if (redo && j == 0) {
            if (act && !stays && best_d > 0.0 && best_c != kNone && best_c != d) record(a, r, u, d, best_c, best_d);
            else record(a, r, u, d, kNoMove, 0.0);
        }
        // Rows of degree 9..32.
        if (!__any_sync(0xFFFFFFFFu, wide)) continue;
        uint32_t ck[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int dk = __shfl_sync(0xFFFFFFFFu, wide ? deg : 0, k * 8);
            const int64_t rk = __shfl_sync(0xFFFFFFFFu, rb, k * 8);
            ck[k] = lane < dk ? (uint32_t)a.col[rk + lane] : kNone;
        }
        unsigned flags = 0;   // bit k: a neighbour of row k moved; bit 4 + k: something it sees changed
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (ck[k] == kNone) continue;
            const int32_t vk = (int32_t)ck[k];
            const int64_t uk = u0 + k;
            const Seen sv = see(a, r, vk, uk);
            flags |= (sv.moved ? 1u << k : 0u) | (sv.changed ? 16u << k : 0u);
            ck[k] = counts(a, vk, (uint32_t)uk, bound_of(a, (uint32_t)uk)) ? sv.c : kNone;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (ck[k] != kNone && a.rec[ck[k]].cver >= (uint32_t)r.tag) flags |= 16u << k;
            wide_c[w][k][lane] = ck[k];
        }
        __syncwarp();
        flags = __reduce_or_sync(0xFFFFFFFFu, flags);
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            const int dk = __shfl_sync(0xFFFFFFFFu, wide ? deg : 0, k * 8);
            const bool freshk = __shfl_sync(0xFFFFFFFFu, fresh, k * 8), affk = __shfl_sync(0xFFFFFFFFu, aff, k * 8);
            const uint32_t dcom = __shfl_sync(0xFFFFFFFFu, d, k * 8);
            if (dk == 0) continue;
            if (!freshk && !(flags >> (4 + k) & 1u)) {
                if (lane == 0) keep_decision(r, u0 + k);
            } else if (!affk && !(flags >> k & 1u)) {
                if (lane == 0) record(a, r, u0 + k, dcom, kNoMove, 0.0);
            } else {
                decide_small(a, r, u0 + k, dk, dcom, wide_c[w][k][lane]);
            }
        }
        __syncwarp();
    }
}

// Four CTAs per SM (registers capped at 64; a few bytes spill): measured
// faster than three CTAs at 68 registers.
__global__ void __launch_bounds__(kSmallWarpsPerBlock * 32, 4) k_ex_eval_small(ExactState a) {
    if (a.ctl->P >= a.ctl->n) return;
    eval_small_body(a, a.ctl);
}

// Long and big rows (kMidMaxDeg < degree <= kWarpMaxDeg, up to kBigMaxDeg): one
// CTA per row, table in shared memory, candidates compacted, one candidate per thread per step (its
// lookup interleaved with d's in the first step; wider interleaving spilled
// under the register cap).  Three CTAs per SM (registers capped near 80).
template <int kMaxDeg>
constexpr int row_smem() { return (2 * 2 * kMaxDeg + 2 * (kMaxDeg + 1)) * (int)sizeof(uint32_t); }

template <int kMaxDeg>
__device__ __forceinline__ void eval_row_cta(const ExactState& a, const Ctl* c, const uint32_t* rows, long long b0,
                                             long long b1) {
    extern __shared__ uint32_t big_smem[];
    uint32_t* tk = big_smem;                      // 2 kMaxDeg keys
    uint32_t* tv = tk + 2 * kMaxDeg;              // 2 kMaxDeg counts
    uint32_t* cand_c = tv + 2 * kMaxDeg;          // d and up to kMaxDeg compacted candidates
    uint32_t* cand_w = cand_c + kMaxDeg + 1;
    __shared__ int s_any;
    __shared__ uint32_t s_cnt;
    __shared__ long long s_own;
    __shared__ double red_d[32];
    __shared__ uint32_t red_c[32];
    const Round r = round_view(a, c);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (long long bi = b0 + blockIdx.x; bi < b1; bi += gridDim.x) {
        const uint32_t u = rows[bi];
        const int64_t rb = a.rp[u], re = a.rp[u + 1];
        const int deg = (int)(re - rb);
        const uint32_t d = a.vcom[u];
        const uint32_t ub = bound_of(a, u);
        uint32_t H = 64;
        while (H < 2u * (uint32_t)deg) H <<= 1;
        const uint32_t mask = H - 1;
        for (uint32_t i = tid; i < H; i += blockDim.x) { tk[i] = kNone; tv[i] = 0; }
        if (tid == 0) {
            s_any = a.vaff[u] != 0;
            s_cnt = 1;
            cand_c[0] = d;
        }
        __syncthreads();
        bool any = false;
        for (int64_t base = rb; base < re; base += 4 * (int64_t)blockDim.x) {
            uint32_t c[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int64_t e = base + k * (int64_t)blockDim.x + tid;
                c[k] = kNone;
                if (e < re) {
                    const int32_t v = a.col[e];
                    any = any || (decided_before(r, v, u) && prev_mover(a, r, v));
                    if (counts(a, v, u, ub)) c[k] = comm_at(a, r, v, u);
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const unsigned peers = __match_any_sync(0xFFFFFFFFu, c[k]);
                if (c[k] != kNone && lane == __ffs(peers) - 1) table_add(tk, tv, mask, c[k], (uint32_t)__popc(peers));
            }
        }
        if (any) s_any = 1;
        __syncthreads();
        if (!s_any) {
            if (tid == 0) record(a, r, u, d, kNoMove, 0.0);
            __syncthreads();
            continue;
        }
        const double ku = (double)deg;
        const uint32_t kud = table_get(tk, tv, mask, d);
        // Compact the candidates (c != d) behind d itself; their order does not
        // matter, the selection is a total order.
        for (uint32_t i0 = 0; i0 < H; i0 += blockDim.x) {
            const uint32_t i = i0 + tid;
            const uint32_t c = i < H ? tk[i] : kNone;
            const bool occ = c != kNone && c != d;
            const unsigned bal = __ballot_sync(0xFFFFFFFFu, occ);
            uint32_t base = 0;
            if (lane == 0 && bal) base = atomicAdd(&s_cnt, (uint32_t)__popc(bal));
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if (occ) {
                const uint32_t pos = base + __popc(bal & ((1u << lane) - 1u));
                cand_c[pos] = c;
                cand_w[pos] = tv[i];
            }
        }
        __syncthreads();
        const uint32_t cnt = s_cnt;
        double best_d = 0.0;
        uint32_t best_c = kNone;
        long long sd = 0;
        for (uint32_t i0 = 0;; i0 += blockDim.x) {
            const uint32_t i = i0 + tid;
            const uint32_t cc[1] = {i < cnt ? cand_c[i] : kNone};
            const bool vv[1] = {i < cnt};
            CommRec rr[1] = {CommRec{0ull, 0u, 0u}};
            if (vv[0]) rr[0] = load_rec(a, cc[0]);
            long long sg[1];
            sigma_at_k<1>(a, r.tag, r.P, r.par, cc, vv, rr, u, sg);
            if (i0 == 0) {   // thread 0 looked d up
                if (tid == 0) s_own = sg[0];
                __syncthreads();
                sd = s_own;
            }
            if (vv[0] && i > 0) {
                const double dl = delta_qi(a.dq, cand_w[i], kud, deg, sg[0], sd);
                if (dpos(dl) && better_pos(dl, cc[0], best_d, best_c)) { best_d = dl; best_c = cc[0]; }
            }
            if (i0 + blockDim.x >= cnt) break;
        }
        warp_argmax_pos(best_d, best_c);
        if (lane == 0) { red_d[w] = best_d; red_c[w] = best_c; }
        __syncthreads();
        if (tid == 0) {
            double bd = red_d[0];
            uint32_t bc = red_c[0];
            for (int k = 1; k < (int)(blockDim.x / 32); ++k)
                if (better_pos(red_d[k], red_c[k], bd, bc)) { bd = red_d[k]; bc = red_c[k]; }
            if (!refine_stays(a, (double)sd, ku) && bd > 0.0 && bc != kNone && bc != d) record(a, r, u, d, bc, bd);
            else record(a, r, u, d, kNoMove, 0.0);
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kBigThreads, 2) k_ex_eval_big(ExactState a) {
    if (a.ctl->P >= a.ctl->n) return;
    eval_row_cta<kBigMaxDeg>(a, a.ctl, a.big_v, a.ctl->bs0, a.ctl->bs1);
}

__global__ void __launch_bounds__(kLongThreads, 8) k_ex_eval_long(ExactState a) {
    if (a.ctl->P >= a.ctl->n) return;
    eval_row_cta<kWarpMaxDeg>(a, a.ctl, a.long_v, a.ctl->ls0, a.ctl->ls1);
}

// Mid rows of the window (from the ascending list of mid-degree vertices).
__device__ __forceinline__ void eval_mid_body(const ExactState& a, const Ctl* c) {
    extern __shared__ uint32_t ex_smem[];
    const Round r = round_view(a, c);
    const long long m0 = c->ms0, m1 = c->ms1;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int wpb = (int)(blockDim.x >> 5);
    uint32_t* tk = ex_smem + (size_t)w * 2 * kMidSlots;
    uint32_t* tv = tk + kMidSlots;
    const long long nw = (long long)gridDim.x * wpb;
    for (long long i = m0 + (long long)blockIdx.x * wpb + w; i < m1; i += nw)
        eval_mid(a, r, a.mid_v[i], lane, tk, tv);
}

__global__ void __launch_bounds__(kMidWarpsPerBlock * 32) k_ex_eval_mid(ExactState a) {
    if (a.ctl->P >= a.ctl->n) return;
    eval_mid_body(a, a.ctl);
}

__global__ void k_degree_flags(const int64_t* __restrict__ rp, int64_t n, int64_t above, int64_t most,
                               int32_t* __restrict__ flag) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int64_t d = rp[v + 1] - rp[v];
        flag[v] = d > above && d <= most;
    }
}

__global__ void k_degree_scatter(const int32_t* __restrict__ flag, const int64_t* __restrict__ pos, int64_t n,
                                 uint32_t* __restrict__ out) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        if (flag[v]) out[pos[v]] = (uint32_t)v;
}

// Entries of an ascending list before each kIndexV-th vertex; the last one: all.
__global__ void k_list_index(const uint32_t* __restrict__ list, int64_t len, int64_t entries,
                             int32_t* __restrict__ out) {
    for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b < entries; b += (int64_t)gridDim.x * blockDim.x)
        out[b] = (int32_t)(b == entries - 1 ? len : lower_bound_u32(list, len, (uint32_t)(b * kIndexV)));
}

// Hub accumulation: one CTA per kHubSeg-edge segment of a window hub, four
// edges per thread in flight, and their first probes (one edge after another took
// R-MAT-22's rounds 38 us here, now 21; counting a segment in shared memory first
// costs more than it saves, as most keys are different).  Needs no event table: it runs while the
// previous window commits its affected flags and the event table is built.
__device__ __forceinline__ void hub_accum_body(const ExactState& a, const Ctl* c) {
    const Round r = round_view(a, c);
    const long long q0 = c->es0, q1 = c->es1;
    const int lane = threadIdx.x & 31;
    __shared__ int s_any;
    for (long long q = q0 + blockIdx.x; q < q1; q += gridDim.x) {
        const HubSeg sg = a.eseg[q];
        const uint32_t h = a.hub_v[sg.hub];
        const int64_t rb = a.rp[h], re = a.rp[h + 1];
        const int64_t e0 = rb + (int64_t)sg.part * kHubSeg, e1 = min(re, e0 + kHubSeg);
        uint32_t* tk = a.tkeys + a.hub_toff[sg.hub];
        uint32_t* tv = a.tvals + a.hub_toff[sg.hub];
        const uint32_t mask = a.hub_tcap[sg.hub] - 1;
        uint32_t* occ = a.hub_occ + a.hub_toff[sg.hub];
        uint32_t* occn = a.hub_occn + sg.hub;
        const uint32_t d = a.vcom[h];
        const uint32_t ub = bound_of(a, h);
        if (threadIdx.x == 0) s_any = 0;
        __syncthreads();
        bool any = false;
        uint32_t c[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int64_t e = e0 + k * (int64_t)blockDim.x + threadIdx.x;
            c[k] = kNone;
            if (e < e1) {
                const int32_t v = a.col[e];
                any = any || (decided_before(r, v, h) && prev_mover(a, r, v));
                if (counts(a, v, h, ub)) c[k] = comm_at(a, r, v, h);
            }
        }
        // Insert-or-add, the four first probes in flight together; keys that are
        // new also go on the hub's occupied list, one reservation per warp.
        uint32_t own = 0;
        uint32_t at[4], prev[4], cnt[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned peers = __match_any_sync(0xFFFFFFFFu, c[k]);
            own += __popc(__ballot_sync(0xFFFFFFFFu, c[k] == d));
            cnt[k] = c[k] != kNone && lane == __ffs(peers) - 1 ? (uint32_t)__popc(peers) : 0u;
            at[k] = hash_u32(c[k]) & mask;
            if (cnt[k]) prev[k] = atomicCAS(&tk[at[k]], kNone, c[k]);
        }
        unsigned fresh = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (!cnt[k]) continue;
            while (prev[k] != kNone && prev[k] != c[k]) {
                at[k] = (at[k] + 1) & mask;
                prev[k] = atomicCAS(&tk[at[k]], kNone, c[k]);
            }
            atomicAdd(&tv[at[k]], cnt[k]);
            if (prev[k] == kNone) fresh |= 1u << k;
        }
        const int nfresh = __popc(fresh);
        int incl = nfresh;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += y;
        }
        uint32_t pos = 0;
        if (lane == 31 && incl) pos = atomicAdd(occn, (uint32_t)incl);
        pos = __shfl_sync(0xFFFFFFFFu, pos, 31) + (uint32_t)(incl - nfresh);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (fresh >> k & 1u) occ[pos++] = at[k];
        if (lane == 0 && own) atomicAdd(&a.hub_kud[sg.hub], own);
        if (any) s_any = 1;
        __syncthreads();
        if (threadIdx.x == 0 && s_any) atomicOr(&a.hub_any[sg.hub], 1);
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kHubThreads2) k_ex_hub_accum(ExactState a) {
    if (a.ctl->P >= a.ctl->n) return;
    hub_accum_body(a, a.ctl);
}

// Hub selection: one CTA per kTabSeg occupied slots of a window hub's table, two
// per thread, in flight together; the last CTA of a hub reduces the partial maxima and
// records the decision.  Three CTAs per SM, as for the big rows.
__device__ __forceinline__ void hub_select_body(const ExactState& a, const Ctl* c) {
    const Round r = round_view(a, c);
    const long long q0 = c->ts0, q1 = c->ts1;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __shared__ double red_d[32];
    __shared__ uint32_t red_c[32];
    __shared__ int s_last;
    __shared__ long long s_own;
    for (long long q = q0 + blockIdx.x; q < q1; q += gridDim.x) {
        const HubSeg sg = a.tseg[q];
        const int j = sg.hub;
        const uint32_t h = a.hub_v[j];
        const uint32_t* tk = a.tkeys + a.hub_toff[j];
        const uint32_t* tv = a.tvals + a.hub_toff[j];
        const uint32_t* occ = a.hub_occ + a.hub_toff[j];
        const uint32_t nocc = a.hub_occn[j];
        const int parts = max(1, (int)((nocc + kTabSeg - 1) / kTabSeg));
        if (sg.part >= parts) continue;   // block-uniform
        const uint32_t d = a.vcom[h];
        const long long ku = a.rp[h + 1] - a.rp[h];
        const uint32_t kud = a.hub_kud[j];
        double best_d = 0.0;
        uint32_t best_c = kNone;
        // Occupied slots [s0, s0 + kTabSeg); thread 0's first lookup is d's.
        uint32_t cc[2], wt[2], slot[2];
        bool vv[2];
        CommRec rr[2];
        const uint32_t s0 = (uint32_t)sg.part * kTabSeg, s1 = min(nocc, s0 + kTabSeg);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t i = s0 + k * kHubThreads2 + threadIdx.x - 1u;
            vv[k] = (k > 0 || threadIdx.x > 0) && i < s1;
            slot[k] = vv[k] ? occ[i] : 0u;
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            cc[k] = vv[k] ? tk[slot[k]] : d;
            wt[k] = vv[k] ? tv[slot[k]] : 0u;
            vv[k] = vv[k] && cc[k] != d;
        }
        vv[0] = vv[0] || threadIdx.x == 0;
#pragma unroll
        for (int k = 0; k < 2; ++k) rr[k] = vv[k] ? load_rec(a, cc[k]) : CommRec{0ull, 0u, 0u};
        long long sgm[2];
        sigma_at_k<2>(a, r.tag, r.P, r.par, cc, vv, rr, h, sgm);
        if (threadIdx.x == 0) s_own = sgm[0];
        __syncthreads();
        const long long sd = s_own;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (!vv[k] || cc[k] == d) continue;
            const double dl = delta_qi(a.dq, wt[k], kud, ku, sgm[k], sd);
            if (dpos(dl) && better_pos(dl, cc[k], best_d, best_c)) { best_d = dl; best_c = cc[k]; }
        }
        warp_argmax_pos(best_d, best_c);
        if (lane == 0) { red_d[w] = best_d; red_c[w] = best_c; }
        __syncthreads();
        if (threadIdx.x == 0) {
            double bd = red_d[0];
            uint32_t bc = red_c[0];
            for (int k = 1; k < (int)(blockDim.x / 32); ++k)
                if (better_pos(red_d[k], red_c[k], bd, bc)) { bd = red_d[k]; bc = red_c[k]; }
            a.part_d[q] = bd;
            a.part_c[q] = bc;
            __threadfence();
            s_last = atomicAdd(&a.hub_done[j], 1) == parts - 1;
        }
        __syncthreads();
        if (s_last) {
            // The whole CTA reduces the hub's partial maxima.
            __threadfence();
            double bd = 0.0;
            uint32_t bc = kNone;
            const int f = a.hub_tfirst[j];
            for (int k = threadIdx.x; k < parts; k += blockDim.x) {
                const double pd = ((volatile double*)a.part_d)[f + k];
                const uint32_t pc = ((volatile uint32_t*)a.part_c)[f + k];
                if (better_pos(pd, pc, bd, bc)) { bd = pd; bc = pc; }
            }
            warp_argmax_pos(bd, bc);
            __syncthreads();
            if (lane == 0) { red_d[w] = bd; red_c[w] = bc; }
            __syncthreads();
            if (threadIdx.x == 0) {
                bd = red_d[0];
                bc = red_c[0];
                for (int k = 1; k < (int)(blockDim.x / 32); ++k)
                    if (better_pos(red_d[k], red_c[k], bd, bc)) { bd = red_d[k]; bc = red_c[k]; }
                const bool act = a.vaff[h] != 0 || ((volatile int32_t*)a.hub_any)[j] != 0;
                const bool stays = refine_stays(a, (double)sd, (double)ku);
                if (act && !stays && bd > 0.0 && bc != kNone && bc != d) record(a, r, h, d, bc, bd);
                else record(a, r, h, d, kNoMove, 0.0);
                a.hub_done[j] = 0;
                a.hub_any[j] = 0;
                a.hub_kud[j] = 0;
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kHubThreads2, 3) k_ex_hub_select(ExactState a) {
    if (a.ctl->P >= a.ctl->n) return;
    hub_select_body(a, a.ctl);
}

// First change of the decided window (global, written by record()).
__device__ __forceinline__ unsigned long long first_change_of(const ExactState& a) {
    return *(volatile unsigned long long*)&a.ctl->first_change;
}

__device__ __forceinline__ long long commit_end(const ExactState& a, const Ctl* c) {
    const unsigned long long f = first_change_of(a);
    const long long E = c->E;
    return f == kNoChange ? E - 1 : min((long long)f, E - 1);
}

// The window just decided, as the commit kernels see it after the advance:
// [cP, cX] is committed (empty when cX < cP); the decisions are the new
// round's "previous" buffers.
struct CommitView {
    long long P, x;
    const uint32_t* dec;
};

__device__ __forceinline__ CommitView commit_view(const ExactState& a, const Ctl* ct) {
    CommitView c;
    c.P = ct->cP;
    c.x = ct->cX;
    c.dec = a.dec[ct->round & 1];
    return c;
}

// Commit [cP, cX]: totals and memberships of movers, final deltas, processed
// flags cleared, move flags for the affected-flag kernels; and the decided
// window's hub tables cleared for the next round.
// Adds (or, with neg, subtracts) v to the key's total once per distinct key of the
// warp (kNone = no update); every lane of the warp calls it.  Degrees are
// below 2^31, so the 16-bit halves of 32 of them sum without overflow.
__device__ __forceinline__ void warp_add_total(CommRec* rec, uint32_t key, uint32_t v, bool neg) {
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, key);
    unsigned lo = v & 0xFFFFu, hi = v >> 16;
    // A sum per key costs its own turn, so keys that are alone take none (uniform
    // 2^23: the commit's 9.1 us a round, now 6.0).
    if (key != kNone && (peers & (peers - 1))) {
        lo = __reduce_add_sync(peers, lo);
        hi = __reduce_add_sync(peers, hi);
    }
    if (key != kNone && (threadIdx.x & 31) == __ffs(peers) - 1) {
        const long long sum = ((long long)hi << 16) + (long long)lo;
        if (sum) atomicAdd(&rec[key].total, (unsigned long long)(neg ? -sum : sum));
    }
}

__device__ __forceinline__ void commit_a_body(const ExactState& a, const Ctl* ct) {
    const CommitView c = commit_view(a, ct);
    if (c.x < c.P) return;
    // Warp-uniform loop: the total updates are summed per community inside
    // the warp first (many movers of a window join the same few communities,
    // and their atomics on one total would serialise).
    const int lane = threadIdx.x & 31;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long base = c.P + ((blockIdx.x * (long long)blockDim.x + threadIdx.x) & ~31ll); base <= c.x;
         base += stride) {
        const long long u = base + lane;
        bool moves = false;
        uint32_t cur = kNone, nb = kNone;
        uint32_t deg = 0;
        if (u <= c.x) {
            double dl = 0.0;
            cur = a.vcom[u];
            nb = c.dec[u] & kNoMove;
            moves = nb != kNoMove;
            if (moves) {
                deg = (uint32_t)(a.rp[u + 1] - a.rp[u]);
                dl = a.delta[u];
                a.vcom[u] = nb;
            }
            a.mv[u] = moves;
            a.final_delta[u] = dl;
            a.vaff[u] = 0;
        }
        warp_add_total(a.rec, moves ? cur : kNone, deg, true);
        warp_add_total(a.rec, moves ? nb : kNone, deg, false);
    }
    const long long q0 = ct->c_ts0, q1 = ct->c_ts1;
    __shared__ int s_last;
    for (long long q = q0 + blockIdx.x; q < q1; q += gridDim.x) {
        const HubSeg sg = a.tseg[q];
        const int j = sg.hub;
        uint32_t* tk = a.tkeys + a.hub_toff[j];
        uint32_t* tv = a.tvals + a.hub_toff[j];
        const uint32_t* occ = a.hub_occ + a.hub_toff[j];
        const uint32_t s0 = (uint32_t)sg.part * kTabSeg, s1 = min(a.hub_occn[j], s0 + kTabSeg);
        for (uint32_t i = s0 + threadIdx.x; i < s1; i += blockDim.x) {
            const uint32_t slot = occ[i];
            tk[slot] = kNone;
            tv[slot] = 0;
        }
        __syncthreads();
        // The hub's last clearing CTA empties its occupied list (every CTA has
        // read the count before it arrives here).
        if (threadIdx.x == 0) s_last = atomicAdd(&a.hub_clr[j], 1) == a.hub_tcount[j] - 1;
        __syncthreads();
        if (s_last && threadIdx.x == 0) {
            a.hub_occn[j] = 0;
            a.hub_clr[j] = 0;
        }
    }
}

__global__ void k_ex_commit_a(ExactState a) { commit_a_body(a, a.ctl); }

// Affected flags from committed movers: every neighbour outside [cP, cX] and
// every neighbour in [cP, cX] processed before the mover.  Non-hub movers
// here, hub movers in k_ex_commit_hub.
__device__ __forceinline__ void commit_b_body(const ExactState& a, const Ctl* ct) {
    const CommitView c = commit_view(a, ct);
    if (c.x < c.P) return;
    // A thread per window vertex: rows of up to kOwnRow entries are flagged
    // by their own thread (four entries in flight), longer ones by the whole
    // warp, four rows at a time (one after another: 17 us a round on 8 M uniform
    // vertices, now 11, beside a table of 13).
    constexpr int kOwnRow = 16;
    const int lane = threadIdx.x & 31;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long base = c.P + ((blockIdx.x * (long long)blockDim.x + threadIdx.x) & ~31ll); base <= c.x;
         base += stride) {
        const long long w = base + lane;
        int64_t rb = 0, re = 0;
        if (w <= c.x && a.mv[w]) {
            rb = a.rp[w];
            re = a.rp[w + 1];
            if (re - rb > kWarpMaxDeg) re = rb;   // hubs and big rows: k_ex_commit_hub
        }
        if (re - rb <= kOwnRow) {
            for (int64_t e0 = rb; e0 < re; e0 += 4) {
                int32_t v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = e0 + k < re ? a.col[e0 + k] : -1;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (v[k] >= 0 && (v[k] < c.P || v[k] > c.x || v[k] < w)) a.vaff[v[k]] = 1;
            }
        }
        unsigned longer = __ballot_sync(0xFFFFFFFFu, re - rb > kOwnRow);
        while (longer) {
            // The next four rows' first 32 entries in flight together.
            int32_t v[4];
            int64_t e[4], end[4];
            long long ws[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int src = longer ? __ffs(longer) - 1 : 0;
                const bool row = longer != 0;
                longer &= longer - 1;
                ws[k] = __shfl_sync(0xFFFFFFFFu, w, src);
                e[k] = __shfl_sync(0xFFFFFFFFu, rb, src) + lane;
                end[k] = row ? __shfl_sync(0xFFFFFFFFu, re, src) : 0;
                v[k] = e[k] < end[k] ? a.col[e[k]] : -1;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (v[k] >= 0 && (v[k] < c.P || v[k] > c.x || v[k] < ws[k])) a.vaff[v[k]] = 1;
                for (int64_t f = e[k] + 32; f < end[k]; f += 32) {
                    const int32_t x = a.col[f];
                    if (x < c.P || x > c.x || x < ws[k]) a.vaff[x] = 1;
                }
            }
        }
    }
}

__global__ void k_ex_commit_b(ExactState a) { commit_b_body(a, a.ctl); }

__device__ __forceinline__ void commit_hub_body(const ExactState& a, const Ctl* ct) {
    const CommitView c = commit_view(a, ct);
    if (c.x < c.P) return;
    // Work items: the decided window's hub edge segments, then its big rows.
    const long long q0 = ct->c_es0, q1 = ct->c_es1;
    const long long g0 = ct->c_bs0, g1 = ct->c_bs1;
    const long long nseg = q1 - q0, items = nseg + (g1 - g0);
    for (long long q = blockIdx.x; q < items; q += gridDim.x) {
        uint32_t h;
        int64_t e0, e1;
        if (q < nseg) {
            const HubSeg sg = a.eseg[q0 + q];
            h = a.hub_v[sg.hub];
            e0 = a.rp[h] + (int64_t)sg.part * kHubSeg;
            e1 = min(a.rp[h + 1], e0 + kHubSeg);
        } else {
            h = a.big_v[g0 + (q - nseg)];
            e0 = a.rp[h];
            e1 = a.rp[h + 1];
        }
        if ((long long)h > c.x || !a.mv[h]) continue;   // block-uniform
        for (int64_t e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
            const int32_t v = a.col[e];
            if (v < c.P || v > c.x || v < (int64_t)h) a.vaff[v] = 1;
        }
    }
}

__global__ void __launch_bounds__(kHubThreads2) k_ex_commit_hub(ExactState a) { commit_hub_body(a, a.ctl); }

// Re-choose the designated communities of the next table from the counts of
// the table just used: the designated ones' event counts and the table's
// hot slots, largest first, at least kZKeep events each.  Keeps the
// set when nothing in the table was hot and every member kept its
// events.  Called by every thread of one CTA.
__device__ __forceinline__ void designate(const ExactState& a, Ctl* c) {
    __shared__ unsigned long long cand[kZMax + kZCand];
    __shared__ int s_change;
    const int tid = threadIdx.x;
    const int nz = (int)c->nz;
    const int nh = min((int)a.ctl->nhot, kZCand);
    if (tid == 0) {
        int change = nh > 0;
        for (int j = 0; j < nz; ++j) change |= c->zcount[j] < (unsigned)kZKeep;
        s_change = change;
    }
    __syncthreads();
    if (!s_change) {
        if (tid < kZMax) c->zcount[tid] = 0;
        __syncthreads();
        return;
    }
    if (tid < nz) cand[tid] = (unsigned long long)c->zcount[tid] << 32 | c->zc[tid];
    if (tid < nh) cand[nz + tid] = a.zcand[tid];
    __syncthreads();
    if (tid < 32) {
        const int total = nz + nh;
        uint32_t chosen[kZMax];
        int nc = 0;
#pragma unroll 1
        for (int pick = 0; pick < kZMax; ++pick) {
            unsigned long long best = 0;
            int bi = -1;
            for (int t = tid; t < total; t += 32) {
                const unsigned long long v = cand[t];
                if ((v >> 32) >= (unsigned long long)kZKeep && v > best) {
                    best = v;
                    bi = t;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long ob = __shfl_xor_sync(0xFFFFFFFFu, best, o);
                const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
                if (ob > best) {
                    best = ob;
                    bi = oi;
                }
            }
            if (best == 0) break;
            if (tid == 0) {
                chosen[nc] = (uint32_t)best;
                cand[bi] = 0;
            }
            ++nc;
            __syncwarp();
        }
        if (tid == 0) {
            for (int j = 0; j < nz; ++j) a.zof[c->zc[j]] = 0;
            for (int j = 0; j < nc; ++j) {
                a.zof[chosen[j]] = (uint8_t)(j + 1);
                c->zc[j] = chosen[j];
            }
            c->nz = (unsigned)nc;
            for (int j = 0; j < kZMax; ++j) c->zcount[j] = 0;
        }
    }
    __syncthreads();
}

// Length of the next window: kSpan rounds' worth of progress, from the mean of
// the last sixteen or so, between b_min and B.  What lies further ahead is decided
// again many times before its turn comes (a grid of 300 K vertices commits some
// 400 a round, however long the window: 73 ms with always 65,536 of them, 67 so);
// where a window is committed in three or four rounds, a shorter one only adds
// rounds (8 M uniform vertices: 268 ms with 65,536, 345 with always 16,384).
// A span of 4 left planted communities 3 percent slower, 8 nothing faster.  The
// floor stands above what the span asks for on a grid (2,400): decisions far ahead
// are made again, but a round costs nearly the same and moves on further (511 x 601
// grid, local moving with windows of 4,096 / 8,192 / 12,288 / 16,384: 89.2 / 69.9 /
// 63.2 / 59.7 ms in 4,626 / 3,524 / 3,095 / 2,812 rounds; R-MAT scale 16: 4.6 / 3.6 /
// 3.5 / 3.4 ms).
constexpr long long kSpan = 6;
constexpr long long kWindowMin = 16384;

__device__ __forceinline__ long long window_length(const Ctl* c, long long progress) {
    return min(c->B, max(c->b_min, kSpan * progress / 64));
}

// After the window's decisions: fix the committed prefix [P, x] for the commit
// kernels, slide the window (the new decisions become D_prev) and tell the graph's loop whether to go on.  The next
// window's event table and this window's commits then run concurrently: they
// touch disjoint vertices.  Ends with a CTA barrier, so every thread sees the
// updated block.
__device__ __forceinline__ void advance_ctl(const ExactState& a, Ctl* c, bool set_cond) {
    const long long P = c->P, E = c->E, n = c->n;
    if (P >= n) {
        __syncthreads();
        if (threadIdx.x == 0) {
            c->cP = 1;   // nothing to commit
            c->cX = 0;
            if (set_cond) cudaGraphSetConditional(a.cond, 0u);
        }
        __syncthreads();
        return;
    }
    const long long x = commit_end(a, c);
    const long long nP = x + 1;
    const long long progress = c->progress + (64 * (nP - P) - c->progress) / 16;
    // May end before E: what is dropped enters again as new.
    const long long nE = min(n, nP + window_length(c, progress));
    if (threadIdx.x == 0) {
        c->c_es0 = c->es0;
        c->c_es1 = c->es1;
        c->c_ts0 = c->ts0;
        c->c_ts1 = c->ts1;
        c->c_bs0 = c->bs0;
        c->c_bs1 = c->bs1;
    }
    __syncthreads();
    window_ranges(a, c, nP, nE);
    // Designated communities: their records point the next table's lookups at
    // the dense rows, and count as changed -- the old set's too, which a
    // change of the set moves between the dense rows and the table.
    const uint32_t ntag = (uint32_t)c->tag + 1u;
    // This round's table is done with.
    if (threadIdx.x < kClearSlots)
        a.slots[((uint32_t)c->tag * kClearSlots + threadIdx.x) & (kTableSlots - 1)].word = 0;
    if (threadIdx.x < c->nz) a.rec[c->zc[threadIdx.x]].cver = ntag;
    designate(a, c);
    if (threadIdx.x < c->nz) {
        CommRec* z = a.rec + c->zc[threadIdx.x];
        z->cver = ntag;
        z->slotw = ntag << kSlotwTagShift | kSlotwDesig | threadIdx.x;
    }
    if (threadIdx.x == 0) {
        const long long rnd = c->round + 1;
        c->cP = P;
        c->cX = x;
        c->pE = E;
        c->progress = progress;
        c->evals = c->evals + (E - P);
        c->P = nP;
        c->E = nE;
        c->round = rnd;
        c->tag = c->tag + 1;
        c->nmany[0] = c->nmany[1] = c->sorted = c->nhot = 0;
        // Every round commits at least vertex P, so the loop ends within n
        // rounds; the bound only guards against a broken invariant.
        bool more = nP < n;
        if (nP <= P || (more && rnd >= c->max_rounds)) {
            c->error = 1;
            c->P = n;
            more = false;
        }
        if (set_cond) cudaGraphSetConditional(a.cond, more ? 1u : 0u);
    }
    __syncthreads();
}

__global__ void __launch_bounds__(1024) k_ex_advance(ExactState a) {
    advance_ctl(a, a.ctl, a.use_cond != 0);
}

// The first window of an iteration.
__device__ __forceinline__ void init_ctl(const ExactState& a, Ctl* c) {
    const long long n = c->n;
    const long long E = min(n, window_length(c, c->progress));
    window_ranges(a, c, 0, E);
    // The generation that the last advance left without a table: its share of the slots.
    if (threadIdx.x < kClearSlots)
        a.slots[((uint32_t)c->tag * kClearSlots + threadIdx.x) & (kTableSlots - 1)].word = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
        c->P = 0;
        c->E = E;
        c->round = 0;
        c->evals = 0;
        c->cP = n;   // no window before: nothing to commit, nothing changed
        c->cX = 0;
        c->pE = 0;
        c->tag = c->tag + 1;
        c->nmany[0] = c->nmany[1] = c->sorted = c->nhot = 0;
        for (int j = 0; j < kZMax; ++j) c->zcount[j] = 0;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(1024) k_ex_init_iter(ExactState a) {
    init_ctl(a, a.ctl);
}

// Deterministic tree sum of the iteration's committed deltas (and count).
__global__ void k_sum_deltas(const double* __restrict__ d, int64_t n, double* __restrict__ partial,
                             unsigned long long* __restrict__ cnt) {
    double s = 0.0;
    unsigned long long c = 0;
    const int64_t per = (n + gridDim.x - 1) / gridDim.x;
    const int64_t b = blockIdx.x * per, e = min(n, b + per);
    for (int64_t i = b + threadIdx.x; i < e; i += blockDim.x) {
        s += d[i];
        c += d[i] != 0.0;
    }
    __shared__ double sh[kT];
    __shared__ unsigned long long shc[kT];
    sh[threadIdx.x] = s;
    shc[threadIdx.x] = c;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            sh[threadIdx.x] += sh[threadIdx.x + o];
            shc[threadIdx.x] += shc[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = sh[0];
        atomicAdd(cnt, shc[0]);
    }
}

// Exact left-to-right sum in vertex order (only when the bound is inconclusive).
__global__ void k_sum_serial(const double* __restrict__ d, int64_t n, double* __restrict__ out) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        double s = 0.0;
        for (int64_t i = 0; i < n; ++i) s += d[i];
        *out = s;
    }
}

__global__ void k_rec_from_totals(const unsigned long long* __restrict__ ctot, int64_t n, CommRec* __restrict__ rec) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x)
        rec[c] = CommRec{ctot[c], 0u, 0u};
}

__global__ void k_totals_from_rec(const CommRec* __restrict__ rec, int64_t n, unsigned long long* __restrict__ ctot) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x)
        ctot[c] = rec[c].total;
}

__global__ void k_hub_degrees(const int64_t* __restrict__ rp, const uint32_t* __restrict__ hubs, int64_t nh,
                              int64_t* __restrict__ deg) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nh; j += (int64_t)gridDim.x * blockDim.x)
        deg[j] = rp[hubs[j] + 1] - rp[hubs[j]];
}

template <typename T>
T read_dev(const T* p, cudaStream_t s) {
    T h;
    GB_CUDA(cudaMemcpyAsync(&h, p, sizeof(T), cudaMemcpyDeviceToHost, s));
    GB_CUDA(cudaStreamSynchronize(s));
    return h;
}

template <typename T>
DevBuf<T> upload(const std::vector<T>& v, cudaStream_t s) {
    DevBuf<T> d(v.empty() ? 1 : v.size(), s);
    if (!v.empty()) GB_CUDA(cudaMemcpyAsync(d.get(), v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    return d;
}

}  // namespace

// A graph's rows above kSmallMaxDeg by length, with the segments of the longest:
// what local moving needs to know of the graph, the same in every pass (R-MAT-22:
// 1 ms of host work and copies).
struct RowLists {
    int64_t nh = 0, n_big = 0, n_mid = 0, n_long = 0, n_eseg = 0, n_tseg = 0;
    int64_t pool = 0;        // slots of the hubs' tables
    int64_t index_len = 0;
    DevBuf<int64_t> toff;
    DevBuf<uint32_t> tcap;
    DevBuf<int32_t> tfirst, tcount, index;
    DevBuf<HubSeg> eseg, tseg;
    DevBuf<uint32_t> eseg_v, tseg_v, hub_v, big_v, mid_v, long_v;
};

static std::shared_ptr<RowLists> list_rows(const LocalMoveContext& ctx, cudaStream_t s) {
    const int64_t n = ctx.g.n;
    auto rows = std::make_shared<RowLists>();
    RowLists& L = *rows;
    // Rows above kWarpMaxDeg: up to kBigMaxDeg one CTA each ("big"), above
    // that segmented over CTAs ("hubs").
    const int64_t nh_all = (int64_t)ctx.hubs_h.size();
    std::vector<int64_t> hdeg_all(nh_all);
    if (nh_all) {
        DevBuf<int64_t> dd(nh_all, s);
        k_hub_degrees<<<grid_for(nh_all, kT), kT, 0, s>>>(ctx.g.row_ptr, ctx.hubs, nh_all, dd);
        GB_LAUNCH_CHECK();
        GB_CUDA(cudaMemcpyAsync(hdeg_all.data(), dd.get(), nh_all * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
        GB_CUDA(cudaStreamSynchronize(s));
    }
    std::vector<uint32_t> big_h, hub_h;
    std::vector<int64_t> hdeg;
    for (int64_t j = 0; j < nh_all; ++j) {
        if (hdeg_all[j] <= kBigMaxDeg) {
            big_h.push_back(ctx.hubs_h[j]);
        } else {
            hub_h.push_back(ctx.hubs_h[j]);
            hdeg.push_back(hdeg_all[j]);
        }
    }
    const int64_t nh = (int64_t)hub_h.size();
    L.nh = nh;
    L.n_big = (int64_t)big_h.size();
    std::vector<int64_t> toff(nh);
    std::vector<uint32_t> tcap(nh);
    std::vector<int32_t> tfirst(nh), tcount(nh);
    std::vector<HubSeg> eseg, tseg;
    std::vector<uint32_t> eseg_v, tseg_v;
    for (int64_t j = 0; j < nh; ++j) {
        uint32_t cap = 64;
        while ((int64_t)cap < 2 * hdeg[j]) cap <<= 1;
        tcap[j] = cap;
        toff[j] = L.pool;
        L.pool += cap;
        const int ne = (int)ceil_div(hdeg[j], kHubSeg);
        for (int k = 0; k < ne; ++k) {
            eseg.push_back({(int32_t)j, k});
            eseg_v.push_back(hub_h[j]);
        }
        const int nt = (int)std::max<int64_t>(1, ceil_div(hdeg[j], kTabSeg));   // occupied slots <= degree
        tfirst[j] = (int32_t)tseg.size();
        tcount[j] = nt;
        for (int k = 0; k < nt; ++k) {
            tseg.push_back({(int32_t)j, k});
            tseg_v.push_back(hub_h[j]);
        }
    }
    L.toff = upload(toff, s);
    L.tcap = upload(tcap, s);
    L.tfirst = upload(tfirst, s);
    L.tcount = upload(tcount, s);
    L.eseg = upload(eseg, s);
    L.tseg = upload(tseg, s);
    L.eseg_v = upload(eseg_v, s);
    L.tseg_v = upload(tseg_v, s);
    L.hub_v = upload(hub_h, s);
    L.big_v = upload(big_h, s);
    L.n_eseg = (int64_t)eseg.size();
    L.n_tseg = (int64_t)tseg.size();

    // Mid and long rows: both counts in one look at the device.
    {
        DevBuf<int32_t> flag(2 * n, s);
        DevBuf<int64_t> pos(2 * n, s), tot(2, s);
        const int64_t above[2] = {kSmallMaxDeg, kMidMaxDeg}, most[2] = {kMidMaxDeg, kWarpMaxDeg};
        for (int k = 0; k < 2; ++k) {
            k_degree_flags<<<grid_for(n, kT), kT, 0, s>>>(ctx.g.row_ptr, n, above[k], most[k], flag.get() + k * n);
            GB_LAUNCH_CHECK();
            exclusive_scan_i32_to_i64(flag.get() + k * n, pos.get() + k * n, n, tot.get() + k, s);
        }
        int64_t counts[2];
        GB_CUDA(cudaMemcpyAsync(counts, tot.get(), sizeof(counts), cudaMemcpyDeviceToHost, s));
        GB_CUDA(cudaStreamSynchronize(s));
        DevBuf<uint32_t>* out[2] = {&L.mid_v, &L.long_v};
        for (int k = 0; k < 2; ++k) {
            out[k]->alloc(counts[k] > 0 ? counts[k] : 1, s);
            if (counts[k] == 0) continue;
            k_degree_scatter<<<grid_for(n, kT), kT, 0, s>>>(flag.get() + k * n, pos.get() + k * n, n, out[k]->get());
            GB_LAUNCH_CHECK();
        }
        L.n_mid = counts[0];
        L.n_long = counts[1];
    }

    L.index_len = n / kIndexV + 2;
    L.index.alloc(kIndexLists * L.index_len, s);
    const uint32_t* lists[kIndexLists] = {L.eseg_v.get(), L.tseg_v.get(), L.mid_v.get(), L.big_v.get(),
                                          L.long_v.get()};
    const int64_t lens[kIndexLists] = {L.n_eseg, L.n_tseg, L.n_mid, L.n_big, L.n_long};
    for (int k = 0; k < kIndexLists; ++k) {
        if (lens[k] == 0) continue;   // window_ranges does not look
        k_list_index<<<grid_for(L.index_len, kT), kT, 0, s>>>(lists[k], lens[k], L.index_len,
                                                             L.index.get() + k * L.index_len);
        GB_LAUNCH_CHECK();
    }
    return rows;
}

int local_move_exact(LocalMoveContext& ctx, double tolerance, int max_iterations, int64_t window,
                     cudaStream_t s, int64_t* launches, int64_t* rounds_out, int64_t* evals_out) {
    const int64_t n = ctx.g.n;
    const int64_t B = std::max<int64_t>(32, std::min<int64_t>(std::min<int64_t>(window, kWindowMax), n));

    if (!ctx.rows) ctx.rows = list_rows(ctx, s);
    const RowLists& L = *ctx.rows;
    const int64_t nh = L.nh, n_big = L.n_big, n_mid = L.n_mid, n_long = L.n_long, pool = L.pool;

    // ---- hub tables ----
    DevBuf<uint32_t> tkeys(pool > 0 ? pool : 1, s), tvals(pool > 0 ? pool : 1, s);
    GB_CUDA(cudaMemsetAsync(tkeys, 0xFF, (pool > 0 ? pool : 1) * sizeof(uint32_t), s));
    GB_CUDA(cudaMemsetAsync(tvals, 0, (pool > 0 ? pool : 1) * sizeof(uint32_t), s));
    DevBuf<int32_t> hub_any(nh > 0 ? nh : 1, s), hub_done(nh > 0 ? nh : 1, s);
    GB_CUDA(cudaMemsetAsync(hub_any, 0, (nh > 0 ? nh : 1) * sizeof(int32_t), s));
    GB_CUDA(cudaMemsetAsync(hub_done, 0, (nh > 0 ? nh : 1) * sizeof(int32_t), s));
    DevBuf<uint32_t> hub_kud(nh > 0 ? nh : 1, s), hub_occn(nh > 0 ? nh : 1, s);
    DevBuf<int32_t> hub_clr(nh > 0 ? nh : 1, s);
    DevBuf<uint32_t> hub_occ(pool > 0 ? pool : 1, s);
    GB_CUDA(cudaMemsetAsync(hub_occn, 0, (nh > 0 ? nh : 1) * sizeof(uint32_t), s));
    GB_CUDA(cudaMemsetAsync(hub_clr, 0, (nh > 0 ? nh : 1) * sizeof(int32_t), s));
    GB_CUDA(cudaMemsetAsync(hub_kud, 0, (nh > 0 ? nh : 1) * sizeof(uint32_t), s));
    DevBuf<double> part_d(L.n_tseg > 0 ? L.n_tseg : 1, s);
    DevBuf<uint32_t> part_c(L.n_tseg > 0 ? L.n_tseg : 1, s);

    // ---- round state ----
    DevBuf<uint32_t> dec0(n, s), dec1(n, s);
    DevBuf<double> delta(n, s), final_delta(n, s);
    DevBuf<CommRec> rec(n, s);
    k_rec_from_totals<<<grid_for(n, kT), kT, 0, s>>>(ctx.ctot, n, rec);
    GB_LAUNCH_CHECK();
    DevBuf<uint8_t> mv(n, s);
    DevBuf<SlotMeta> slots(kTableSlots, s);
    GB_CUDA(cudaMemsetAsync(slots, 0, kTableSlots * sizeof(SlotMeta), s));   // no generation yet
    DevBuf<uint2> ev((size_t)kTableSlots * kInline, s), hot_row((size_t)kHotMax * kHotWords, s);
    DevBuf<uint32_t> many0(kEventsMax / kInline, s), many1(kEventsMax / kWarpSort, s), stime(kEventsMax, s);
    DevBuf<long long> epre(kEventsMax, s);
    DevBuf<int32_t> sdeg(kEventsMax, s);
    DevBuf<uint8_t> zof(n > 0 ? n : 1, s);
    GB_CUDA(cudaMemsetAsync(zof, 0, (n > 0 ? n : 1), s));
    DevBuf<int32_t> zcontrib((size_t)2 * kZMax * kWindowMax, s);
    DevBuf<long long> zbsum((size_t)2 * kZMax * kBucketStride, s), zpre((size_t)2 * kZMax * kBucketStride, s);
    DevBuf<unsigned long long> zcand(kZCand, s);
    DevBuf<Ctl> ctl(1, s);
    Ctl* hctl = nullptr;
    GB_CUDA(cudaMallocHost(&hctl, sizeof(Ctl)));
    *hctl = Ctl{};
    hctl->n = n;
    hctl->B = B;
    hctl->b_min = std::min(B, (int64_t)kWindowMin);
    hctl->progress = 64 * hctl->b_min / kSpan;
    hctl->max_rounds = n + 2;
    GB_CUDA(cudaMemcpyAsync(ctl.get(), hctl, sizeof(Ctl), cudaMemcpyHostToDevice, s));
    DevBuf<double> partial(1024, s), dsum(1, s);
    DevBuf<unsigned long long> nmov(1, s);

    ExactState a{};
    a.rp = ctx.g.row_ptr;
    a.col = ctx.g.col;
    a.vcom = ctx.vcom;
    a.rec = rec.get();
    a.vaff = ctx.vaff;
    a.vcob = ctx.vcob;
    a.mv = mv.get();
    a.ctl = ctl.get();
    a.dec[0] = dec0.get();
    a.dec[1] = dec1.get();
    a.delta = delta.get();
    a.final_delta = final_delta.get();
    a.slots = slots.get();
    a.ev = ev.get();
    a.many[0] = many0.get();
    a.many[1] = many1.get();
    a.sdeg = sdeg.get();
    a.hot_row = hot_row.get();
    a.zof = zof.get();
    a.zcontrib = zcontrib.get();
    a.zbsum = zbsum.get();
    a.zpre = zpre.get();
    a.zcand = zcand.get();
    a.stime = stime.get();
    a.epre = epre.get();
    a.hub_v = L.hub_v.get();
    a.big_v = L.big_v.get();
    a.n_big = n_big;
    a.hub_toff = L.toff.get();
    a.hub_tcap = L.tcap.get();
    a.hub_tfirst = L.tfirst.get();
    a.hub_tcount = L.tcount.get();
    a.eseg = L.eseg.get();
    a.eseg_v = L.eseg_v.get();
    a.n_eseg = L.n_eseg;
    a.tseg = L.tseg.get();
    a.tseg_v = L.tseg_v.get();
    a.n_tseg = L.n_tseg;
    a.tkeys = tkeys.get();
    a.tvals = tvals.get();
    a.hub_any = hub_any.get();
    a.hub_kud = hub_kud.get();
    a.hub_occ = hub_occ.get();
    a.hub_occn = hub_occn.get();
    a.hub_clr = hub_clr.get();
    a.hub_done = hub_done.get();
    a.part_d = part_d.get();
    a.part_c = part_c.get();
    a.mid_v = L.mid_v.get();
    a.n_mid = n_mid;
    a.long_v = L.long_v.get();
    a.n_long = n_long;
    a.list_index = L.index.get();
    a.index_len = L.index_len;
    a.M = ctx.M;
    a.R = ctx.R;
    a.dq = ctx.dq;

    const int tb_grid = (int)ceil_div(B, kTbThreads);
    auto enqueue_table = [&](cudaStream_t st) {
        k_tb_insert<<<tb_grid, kTbThreads, 0, st>>>(a);
        k_tb_sort<<<kZMax + kSortCtas, kSortThreads, 0, st>>>(a);
    };
    const int mid_smem = kMidWarpsPerBlock * 2 * kMidSlots * (int)sizeof(uint32_t);
    GB_CUDA(cudaFuncSetAttribute(k_ex_eval_mid, cudaFuncAttributeMaxDynamicSharedMemorySize, mid_smem));
    const int small_grid = (int)std::max<int64_t>(1, ceil_div(B, 4 * kSmallWarpsPerBlock));
    // Grid-stride kernels: one resident wave (blocks per SM from the occupancy
    // of the compiled kernel x the SM count).
    auto resident = [&](const void* fn, int threads, int smem) {
        int per_sm = 0;
        GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
        int dev = 0, sms = kNumSMs;
        GB_CUDA(cudaGetDevice(&dev));
        GB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        return std::max(1, per_sm) * sms;
    };
    const int mid_grid = resident((const void*)k_ex_eval_mid, kMidWarpsPerBlock * 32, mid_smem);
    const int select_grid = resident((const void*)k_ex_hub_select, kHubThreads2, 0);
    const int big_smem = row_smem<kBigMaxDeg>(), long_smem = row_smem<kWarpMaxDeg>();
    GB_CUDA(cudaFuncSetAttribute(k_ex_eval_big, cudaFuncAttributeMaxDynamicSharedMemorySize, big_smem));
    const int big_grid = resident((const void*)k_ex_eval_big, kBigThreads, big_smem);
    const int long_grid = resident((const void*)k_ex_eval_long, kLongThreads, long_smem);
    const int hub_grid = resident((const void*)k_ex_hub_accum, kHubThreads2, 0);
    const int commit_grid = (int)std::max<int64_t>(1, ceil_div(B, kT));
    const int commit_b_grid = (int)std::max<int64_t>(1, ceil_div(B, kT));
    // eval_small, advance, 2 table kernels, commit_a, commit_b; eval_mid;
    // eval_long; eval_big; hub_select + hub_accum; commit_hub (hubs or big rows).
    const int per_round = 6 + (n_mid ? 1 : 0) + (n_long ? 1 : 0) + (n_big ? 1 : 0) + (nh ? 2 : 0) + ((nh || n_big) ? 1 : 0);
    const int commit_a_grid = std::max(commit_grid, nh ? hub_grid : 0);
    // Side streams and events for the fork/join shape of a captured round:
    struct Fork {
        cudaStream_t s1 = nullptr, s2 = nullptr, s3 = nullptr, s4 = nullptr;
        cudaEvent_t ev[10] = {};
        ~Fork() {
            for (cudaEvent_t e : ev)
                if (e) cudaEventDestroy(e);
            if (s1) cudaStreamDestroy(s1);
            if (s2) cudaStreamDestroy(s2);
            if (s3) cudaStreamDestroy(s3);
            if (s4) cudaStreamDestroy(s4);
        }
    } fk;
    // One round: decide the window, advance, then prepare the next window
    // while this one commits.  Forked shape (graph capture):
    //   { eval_small | eval_mid | eval_long | eval_big | hub_select } -> advance
    //   -> { table(next) | commit_a -> { commit_b | commit_hub | hub_accum(next) } }
    // hub_accum needs the committed memberships but no event table; the
    // round before the first needs the first window's table and accumulation.
    auto enqueue_round = [&](cudaStream_t st, bool fork) {
        cudaStream_t sm = fork ? fk.s1 : st, sh = fork ? fk.s2 : st, sa = fork ? fk.s3 : st,
                     sl = fork ? fk.s4 : st;
        if (fork) {
            GB_CUDA(cudaEventRecord(fk.ev[0], st));
            GB_CUDA(cudaStreamWaitEvent(sm, fk.ev[0], 0));
            GB_CUDA(cudaStreamWaitEvent(sh, fk.ev[0], 0));
        }
        if (fork) GB_CUDA(cudaStreamWaitEvent(sa, fk.ev[0], 0));
        if (fork && n_long) GB_CUDA(cudaStreamWaitEvent(sl, fk.ev[0], 0));
        k_ex_eval_small<<<small_grid, kSmallWarpsPerBlock * 32, 0, st>>>(a);
        if (n_mid) k_ex_eval_mid<<<mid_grid, kMidWarpsPerBlock * 32, mid_smem, sm>>>(a);
        if (nh) k_ex_hub_select<<<select_grid, kHubThreads2, 0, sh>>>(a);
        if (n_long) k_ex_eval_long<<<long_grid, kLongThreads, long_smem, sl>>>(a);
        if (n_big) k_ex_eval_big<<<big_grid, kBigThreads, big_smem, sa>>>(a);
        if (fork) {
            GB_CUDA(cudaEventRecord(fk.ev[1], sm));
            GB_CUDA(cudaEventRecord(fk.ev[2], sh));
            GB_CUDA(cudaEventRecord(fk.ev[8], sa));
            if (n_long) {
                GB_CUDA(cudaEventRecord(fk.ev[9], sl));
                GB_CUDA(cudaStreamWaitEvent(st, fk.ev[9], 0));
            }
            GB_CUDA(cudaStreamWaitEvent(st, fk.ev[1], 0));
            GB_CUDA(cudaStreamWaitEvent(st, fk.ev[2], 0));
            GB_CUDA(cudaStreamWaitEvent(st, fk.ev[8], 0));
        }
        k_ex_advance<<<1, 1024, 0, st>>>(a);
        if (fork) {
            GB_CUDA(cudaEventRecord(fk.ev[3], st));
            GB_CUDA(cudaStreamWaitEvent(sm, fk.ev[3], 0));
        }
        enqueue_table(sm);
        k_ex_commit_a<<<commit_a_grid, kT, 0, st>>>(a);
        if (fork) {
            GB_CUDA(cudaEventRecord(fk.ev[4], st));
            GB_CUDA(cudaStreamWaitEvent(sh, fk.ev[4], 0));
            GB_CUDA(cudaStreamWaitEvent(sa, fk.ev[4], 0));
        }
        k_ex_commit_b<<<commit_b_grid, kT, 0, st>>>(a);
        if (nh || n_big) k_ex_commit_hub<<<hub_grid, kHubThreads2, 0, sh>>>(a);
        if (nh) k_ex_hub_accum<<<hub_grid, kHubThreads2, 0, sa>>>(a);
        if (fork) {
            GB_CUDA(cudaEventRecord(fk.ev[5], sm));
            GB_CUDA(cudaEventRecord(fk.ev[6], sh));
            GB_CUDA(cudaEventRecord(fk.ev[7], sa));
            GB_CUDA(cudaStreamWaitEvent(st, fk.ev[5], 0));
            GB_CUDA(cudaStreamWaitEvent(st, fk.ev[6], 0));
            GB_CUDA(cudaStreamWaitEvent(st, fk.ev[7], 0));
        }
        GB_LAUNCH_CHECK();
    };
    auto enqueue_first = [&](cudaStream_t st) {
        k_ex_init_iter<<<1, 1024, 0, st>>>(a);
        enqueue_table(st);
        if (nh) k_ex_hub_accum<<<hub_grid, kHubThreads2, 0, st>>>(a);
    };

    // One local-moving iteration as one graph: the init kernel, then a
    // device-side while loop over rounds whose condition the advance kernel
    // sets.  GBGPU_EXACT_GRAPH=0 enqueues rounds from the host instead.
    const char* genv = std::getenv("GBGPU_EXACT_GRAPH");
    const bool use_graph = !(genv && genv[0] == '0');
    struct GraphGuard {
        cudaGraph_t g = nullptr;
        cudaGraphExec_t e = nullptr;
        cudaStream_t cs = nullptr;
        ~GraphGuard() {
            if (e) cudaGraphExecDestroy(e);
            if (g) cudaGraphDestroy(g);
            if (cs) cudaStreamDestroy(cs);
        }
    } gg;
    if (use_graph) {
        GB_CUDA(cudaStreamCreateWithFlags(&gg.cs, cudaStreamNonBlocking));
        GB_CUDA(cudaGraphCreate(&gg.g, 0));
        cudaGraphConditionalHandle cond;
        GB_CUDA(cudaGraphConditionalHandleCreate(&cond, gg.g, 1, cudaGraphCondAssignDefault));
        a.cond = cond;
        a.use_cond = 1;
        // init -> first window's table (captured) -> while(rounds)
        GB_CUDA(cudaStreamBeginCaptureToGraph(gg.cs, gg.g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        enqueue_first(gg.cs);
        GB_LAUNCH_CHECK();
        GB_CUDA(cudaStreamEndCapture(gg.cs, &gg.g));
        // The captured chain's last node (the one no other node depends on).
        cudaGraphNode_t init_node = nullptr;
        {
            size_t nn = 0;
            GB_CUDA(cudaGraphGetNodes(gg.g, nullptr, &nn));
            std::vector<cudaGraphNode_t> nodes(nn);
            GB_CUDA(cudaGraphGetNodes(gg.g, nodes.data(), &nn));
            for (cudaGraphNode_t nd : nodes) {
                size_t nd_out = 0;
                GB_CUDA(cudaGraphNodeGetDependentNodes(nd, nullptr, nullptr, &nd_out));
                if (nd_out == 0) init_node = nd;
            }
            if (!init_node) throw Error(GBGPU_E_CUDA, "serial-order local moving: empty init graph");
        }
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = cond;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        cudaGraphNode_t loop_node;
        GB_CUDA(cudaGraphAddNode(&loop_node, gg.g, &init_node, nullptr, 1, &cp));
        cudaGraph_t body = cp.conditional.phGraph_out[0];
        GB_CUDA(cudaStreamCreateWithFlags(&fk.s1, cudaStreamNonBlocking));
        GB_CUDA(cudaStreamCreateWithFlags(&fk.s2, cudaStreamNonBlocking));
        GB_CUDA(cudaStreamCreateWithFlags(&fk.s3, cudaStreamNonBlocking));
        GB_CUDA(cudaStreamCreateWithFlags(&fk.s4, cudaStreamNonBlocking));
        for (cudaEvent_t& e : fk.ev) GB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        GB_CUDA(cudaStreamBeginCaptureToGraph(gg.cs, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        enqueue_round(gg.cs, true);
        GB_CUDA(cudaStreamEndCapture(gg.cs, &body));
        // Node priorities: the event-table chain that every round waits for
        // (and the advance before it) first; the affected-flag branch, which
        // runs beside the table with time to spare, last; the evaluations in
        // between.  Honoured through cudaGraphInstantiateFlagUseNodePriority
        // (RMAT-22 local moving 105 -> 100 ms: the table's CTAs no longer wait
        // behind the commit branch's).
        {
            int least = 0, greatest = 0;
            GB_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
            const int mid = (least + greatest) / 2;
            size_t nn = 0;
            GB_CUDA(cudaGraphGetNodes(body, nullptr, &nn));
            std::vector<cudaGraphNode_t> nodes(nn);
            GB_CUDA(cudaGraphGetNodes(body, nodes.data(), &nn));
            for (cudaGraphNode_t nd : nodes) {
                cudaGraphNodeType ty;
                GB_CUDA(cudaGraphNodeGetType(nd, &ty));
                if (ty != cudaGraphNodeTypeKernel) continue;
                cudaKernelNodeParams kp;
                GB_CUDA(cudaGraphKernelNodeGetParams(nd, &kp));
                const void* f = kp.func;
                int pr = mid;
                if (f == (const void*)k_tb_insert || f == (const void*)k_tb_sort || f == (const void*)k_ex_advance)
                    pr = greatest;
                else if (f == (const void*)k_ex_commit_b || f == (const void*)k_ex_commit_hub ||
                         f == (const void*)k_ex_hub_accum)
                    pr = least;
                cudaKernelNodeAttrValue v = {};
                v.priority = pr;
                GB_CUDA(cudaGraphKernelNodeSetAttribute(nd, cudaKernelNodeAttributePriority, &v));
            }
        }
        GB_CUDA(cudaGraphInstantiate(&gg.e, gg.g, cudaGraphInstantiateFlagUseNodePriority));
    }
    const int kBatch = 8;

    int iterations = 0;
    int64_t rounds = 0, nl = 0, evals = 0;
    for (int it = 0; it < max_iterations; ++it) {
        if (use_graph) {
            GB_CUDA(cudaGraphLaunch(gg.e, s));
            GB_CUDA(cudaMemcpyAsync(hctl, ctl.get(), sizeof(Ctl), cudaMemcpyDeviceToHost, s));
            GB_CUDA(cudaStreamSynchronize(s));
        } else {
            enqueue_first(s);
            GB_LAUNCH_CHECK();
            while (true) {
                for (int b = 0; b < kBatch; ++b) enqueue_round(s, false);
                GB_CUDA(cudaMemcpyAsync(hctl, ctl.get(), sizeof(Ctl), cudaMemcpyDeviceToHost, s));
                GB_CUDA(cudaStreamSynchronize(s));
                if (hctl->P >= n) break;
            }
        }
        if (hctl->error == 2)
            throw Error(GBGPU_E_CUDA, "serial-order local moving: event table slot with an invalid hot index");
        if (hctl->error)
            throw Error(GBGPU_E_CUDA, "serial-order local moving: round loop stopped without progress");
        nl += 3 + (nh ? 1 : 0) + hctl->round * per_round;
        rounds += hctl->round;
        evals += hctl->evals;
        ++iterations;
        // totalDelta <= tolerance, decided exactly.
        const int sb = 1024;
        GB_CUDA(cudaMemsetAsync(nmov, 0, sizeof(unsigned long long), s));
        k_sum_deltas<<<sb, kT, 0, s>>>(final_delta, n, partial, nmov);
        GB_LAUNCH_CHECK();
        std::vector<double> hp(sb);
        GB_CUDA(cudaMemcpyAsync(hp.data(), partial.get(), sb * sizeof(double), cudaMemcpyDeviceToHost, s));
        const unsigned long long movers = read_dev(nmov.get(), s);
        double total = 0.0;
        for (double v : hp) total += v;
        // All terms are >= 0: any summation order is within (k-1) u sum of the exact value.
        const double bound = (double)(movers + 1) * 2.220446049250313e-16 * total;
        bool stop;
        if (std::fabs(total - tolerance) > 2.0 * bound) {
            stop = total <= tolerance;
        } else {
            k_sum_serial<<<1, 1, 0, s>>>(final_delta, n, dsum);
            GB_LAUNCH_CHECK();
            stop = read_dev(dsum.get(), s) <= tolerance;
            ++nl;
        }
        nl += 2;
        if (stop) break;
    }
    k_totals_from_rec<<<grid_for(n, kT), kT, 0, s>>>(rec, n, ctx.ctot);
    GB_LAUNCH_CHECK();
    nl += 2;
    cudaFreeHost(hctl);
    if (launches) *launches += nl;
    if (rounds_out) *rounds_out += rounds;
    if (evals_out) *evals_out += evals;
    return iterations;
}

}  // namespace gb
