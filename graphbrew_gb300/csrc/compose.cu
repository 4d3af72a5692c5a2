// compose.cu -- COMPOSE placement and intra-community ordering on the device.
//
// Follows graphbrew::orderCompose (bench/include/graphbrew/reorder/reorder_graphbrew.h:6286-7087)
// with super-graph order "none":
//   * vertices of degree 0 go to the global tail in id order (:6336-6386);
//   * communities are stable-sorted by the community-order key (:6438-6502);
//   * each community's vertices keep vertex-id order (commVertices, :6373-6386);
//   * intra order: Gorder with window w for 4..fallback vertices
//     (intraGorderGreedy, :4420-4587), BFS from the hub above the fallback
//     (intraBFSFromHub, :3929-3984), identity for <= 3 vertices; or reverse
//     Cuthill-McKee for every community (intraRCM, :4000-4134);
//   * newIds[v] = offset(community) + localId[v] (:7003-7017).
//
// Layout in HBM (n vertices): one stable radix sort of (rank(community), v)
// gives the whole placement skeleton: position p in [0, n) holds the vertex
// placed p-th before intra ordering, isolated vertices last.  Every later
// kernel indexes communities by their contiguous position range.
#include <algorithm>
#include <type_traits>

#include "gb_common.cuh"
#include "gb_stages.h"

namespace gb {

namespace {

enum CommunityOrderOrd { kSizeDesc = 0, kSizeAsc = 1, kDegreeDesc = 2, kDegreeAsc = 3, kIdentity = 6 };
enum IntraOrd { kIntraBFS = 0, kIntraRCM = 1, kIntraRCMpp = 2, kIntraDendrogram = 3, kIntraGorder = 4, kIntraRandom = 10 };

constexpr int kT = 256;

__global__ void k_max_u32(const uint32_t* __restrict__ a, int64_t n, uint32_t* __restrict__ out) {
    uint32_t m = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        m = max(m, a[i]);
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Community sizes over non-isolated vertices, optional degree totals.
__global__ void k_comm_sizes(const int64_t* __restrict__ rp, const uint32_t* __restrict__ memb, int64_t n,
                             uint32_t* __restrict__ csize, unsigned long long* __restrict__ cdeg) {
    const int lane = threadIdx.x & 31;
    for (int64_t v0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; v0 < n;
         v0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = v0 + lane;
        const int64_t d = v < n ? rp[v + 1] - rp[v] : 0;
        const uint32_t c = d ? memb[v] : 0u;
        warp_add_u32(csize, c, 1u, d != 0);
        if (cdeg) warp_add_u64(cdeg, c, (unsigned long long)d, d != 0);
    }
}

__global__ void k_max_u32_u64(const uint32_t* __restrict__ a, const unsigned long long* __restrict__ b, int64_t n,
                              uint32_t* __restrict__ out_a, unsigned long long* __restrict__ out_b) {
    uint32_t ma = 0;
    unsigned long long mb = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        ma = max(ma, a[i]);
        if (b) mb = max(mb, b[i]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        ma = max(ma, __shfl_xor_sync(0xFFFFFFFFu, ma, o));
        mb = max(mb, __shfl_xor_sync(0xFFFFFFFFu, mb, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(out_a, ma);
        if (b) atomicMax(out_b, mb);
    }
}

// stage1, when given (a super-graph order), places community c at position
// stage1[c] before the stable sort, so equal keys keep stage1's order.
__global__ void k_comm_keys(int order, const uint32_t* __restrict__ csize, const unsigned long long* __restrict__ cdeg,
                            int64_t C, uint32_t max_size, unsigned long long max_deg,
                            const uint32_t* __restrict__ stage1, uint64_t* __restrict__ keys,
                            uint32_t* __restrict__ ids) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < C; c += (int64_t)gridDim.x * blockDim.x) {
        uint64_t k = 0;
        switch (order) {
            case kSizeDesc: k = (uint64_t)(max_size - csize[c]); break;
            case kSizeAsc: k = csize[c]; break;
            case kDegreeDesc: k = max_deg - cdeg[c]; break;
            case kDegreeAsc: k = cdeg[c]; break;
            default: k = 0; break;
        }
        const int64_t at = stage1 ? (int64_t)stage1[c] : c;
        keys[at] = k;
        ids[at] = (uint32_t)c;
    }
}

// rank[c] and sorted sizes.
__global__ void k_rank(const uint32_t* __restrict__ order, const uint32_t* __restrict__ csize, int64_t C,
                       uint32_t* __restrict__ rank, int64_t* __restrict__ ssize) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < C; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t c = order[i];
        rank[c] = (uint32_t)i;
        ssize[i] = csize[c];
    }
}

// Sort keys for the placement skeleton: rank of the vertex's community, or C
// for isolated vertices (they sort last, in id order).
__global__ void k_vertex_keys(const int64_t* __restrict__ rp, const uint32_t* __restrict__ memb,
                              const uint32_t* __restrict__ rank, int64_t n, uint32_t C,
                              uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        keys[v] = (rp[v + 1] == rp[v]) ? C : rank[memb[v]];
        vals[v] = (uint32_t)v;
    }
}

// pos_of[v], local index (identity intra order) per vertex.
__global__ void k_positions(const uint32_t* __restrict__ order_v, const uint32_t* __restrict__ keys_sorted,
                            const int64_t* __restrict__ offs, int64_t n, uint32_t C,
                            int64_t* __restrict__ pos_of, uint32_t* __restrict__ local) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t v = order_v[p];
        const uint32_t r = keys_sorted[p];
        pos_of[v] = p;
        local[v] = (r < C) ? (uint32_t)(p - offs[r]) : 0u;
    }
}

// Community classes.  Gorder communities by size: a thread, a warp or a CTA
// over a scan heap in shared memory, and a warp over a global workspace for the
// sizes whose scan heap shared memory does not hold.  Lists hold ranks.
enum Class { kClsThread = 1, kClsWarp = 2, kClsCta = 3, kClsBfs = 4, kClsGlobal = 5, kClasses = 6 };

struct ClassCounts {
    int32_t n[kClasses];
    unsigned long long gorder_communities, gorder_vertices, fallback_communities, fallback_vertices;
    uint32_t gorder_max, largest;
};

constexpr int kThreadGorderMax = 32;
constexpr int kWarpGorderMax = 1024;    // a lane scans up to 32 vertices
constexpr int kCtaGorderMax = 16384;    // 256 threads; up to 12 bytes of shared memory a vertex
constexpr int kMaxGorderWindow = 100;   // the thread variant's bound (kMaxB) too

// Counters are added once per warp (millions of tiny communities share them).
__global__ void k_classify(const int64_t* __restrict__ ssize, int64_t C, int intra, int fallback,
                           int32_t* __restrict__ lists, ClassCounts* __restrict__ cc) {
    const int lane = threadIdx.x & 31;
    for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; i0 < C;
         i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + lane;
        const int64_t sz = i < C ? ssize[i] : 0;
        const uint32_t sz32 = (uint32_t)sz;
        int cls = 0;
        bool gorder = false, fell = false;
        if (sz > 0) {
            if (intra == kIntraGorder) {
                fell = fallback > 0 && sz > fallback;
                gorder = !fell && sz > 3;
                if (fell) cls = kClsBfs;
                else if (gorder)
                    cls = sz <= kThreadGorderMax ? kClsThread
                          : sz <= kWarpGorderMax ? kClsWarp
                          : sz <= kCtaGorderMax  ? kClsCta : kClsGlobal;
            } else {
                cls = sz >= 2 ? kClsBfs : 0;
            }
        }
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, cls);
        const int leader = __ffs(peers) - 1;
        int32_t slot = 0;
        if (cls && lane == leader) slot = atomicAdd(&cc->n[cls], __popc(peers));
        slot = __shfl_sync(0xFFFFFFFFu, slot, leader) + __popc(peers & ((1u << lane) - 1u));
        if (cls) lists[(int64_t)cls * C + slot] = (int32_t)i;
        const uint32_t largest = __reduce_max_sync(0xFFFFFFFFu, sz32);
        const uint32_t gmax = __reduce_max_sync(0xFFFFFFFFu, gorder ? sz32 : 0u);
        const unsigned gb = __ballot_sync(0xFFFFFFFFu, gorder), fb = __ballot_sync(0xFFFFFFFFu, fell);
        unsigned long long gv = gorder ? (unsigned long long)sz : 0ull, fv = fell ? (unsigned long long)sz : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            gv += __shfl_xor_sync(0xFFFFFFFFu, gv, o);
            fv += __shfl_xor_sync(0xFFFFFFFFu, fv, o);
        }
        if (lane == 0) {
            if (largest) atomicMax(&cc->largest, largest);
            if (gb) {
                atomicAdd(&cc->gorder_communities, (unsigned long long)__popc(gb));
                atomicAdd(&cc->gorder_vertices, gv);
                atomicMax(&cc->gorder_max, gmax);
            }
            if (fb) {
                atomicAdd(&cc->fallback_communities, (unsigned long long)__popc(fb));
                atomicAdd(&cc->fallback_vertices, fv);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Local adjacency for Gorder communities: for each position p, the local
// indices of in-community neighbours in row order.  A vertex is not its own
// neighbour here: a placed vertex is never moved again, and the scan heap writes
// its word while it bumps the rest of its row.
// ---------------------------------------------------------------------------
__global__ void k_mark_gorder_positions(const int32_t* __restrict__ list, const int32_t* __restrict__ count_p,
                                        const int64_t* __restrict__ offs, const int64_t* __restrict__ ssize,
                                        uint8_t* __restrict__ mark) {
    const int32_t count = *count_p;
    for (int32_t j = blockIdx.x; j < count; j += gridDim.x) {
        const int32_t r = list[j];
        const int64_t b = offs[r], sz = ssize[r];
        for (int64_t k = threadIdx.x; k < sz; k += blockDim.x) mark[b + k] = 1;
    }
}

// Both passes: eight lanes a row (four rows per warp), rows above kOctetRow
// entries by the whole warp afterwards, so that neither the many short rows
// idle a warp nor a hub's row waits on one thread (a thread a row took 224 us
// for the two passes on RMAT scale 12, where one row has 800 entries).
constexpr int kOctetRow = 64;

template <typename Short, typename Long>
__device__ __forceinline__ void for_marked_rows(const int64_t* __restrict__ rp, const uint32_t* __restrict__ memb,
                                                const uint32_t* __restrict__ order_v,
                                                const uint8_t* __restrict__ mark, int64_t nn, Short&& short_row,
                                                Long&& long_row) {
    const int lane = threadIdx.x & 31, g = lane >> 3;
    const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t p0 = 4 * w; p0 < nn; p0 += 4 * nw) {
        const int64_t p = p0 + g;
        int64_t b = 0, e = 0;
        uint32_t u = 0, cu = 0;
        if (p < nn && mark[p]) {
            u = order_v[p];
            b = rp[u];
            e = rp[u + 1];
            cu = memb[u];
        }
        const bool is_long = e - b > kOctetRow;
        short_row(p, b, is_long ? b : e, u, cu, is_long);
        unsigned todo = __ballot_sync(0xFFFFFFFFu, is_long && (lane & 7) == 0);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            long_row(p0 + (src >> 3), __shfl_sync(0xFFFFFFFFu, b, src), __shfl_sync(0xFFFFFFFFu, e, src),
                     __shfl_sync(0xFFFFFFFFu, u, src), __shfl_sync(0xFFFFFFFFu, cu, src));
        }
    }
}

__global__ void k_local_count(const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                              const uint32_t* __restrict__ memb, const uint32_t* __restrict__ order_v,
                              const uint8_t* __restrict__ mark, int64_t nn, int64_t* __restrict__ cnt) {
    const int lane = threadIdx.x & 31, j = lane & 7;
    auto counts = [&](int32_t w, uint32_t u, uint32_t cu) { return memb[w] == cu && (uint32_t)w != u; };
    for_marked_rows(
        rp, memb, order_v, mark, nn,
        [&](int64_t p, int64_t b, int64_t e, uint32_t u, uint32_t cu, bool is_long) {
            int c = 0;
            for (int64_t x = b + j; x < e; x += 8) c += counts(col[x], u, cu);
            c += __shfl_xor_sync(0xFFFFFFFFu, c, 4);
            c += __shfl_xor_sync(0xFFFFFFFFu, c, 2);
            c += __shfl_xor_sync(0xFFFFFFFFu, c, 1);
            if (j == 0 && p < nn && !is_long) cnt[p] = c;
        },
        [&](int64_t p, int64_t b, int64_t e, uint32_t u, uint32_t cu) {
            int c = 0;
            for (int64_t x = b + lane; x < e; x += 32) c += counts(col[x], u, cu);
            c = __reduce_add_sync(0xFFFFFFFFu, c);
            if (lane == 0) cnt[p] = c;
        });
}

__global__ void k_local_fill(const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                             const uint32_t* __restrict__ memb, const uint32_t* __restrict__ order_v,
                             const uint8_t* __restrict__ mark, const uint32_t* __restrict__ local,
                             const int64_t* __restrict__ loff, int64_t nn, uint16_t* __restrict__ ladj16,
                             uint32_t* __restrict__ ladj32) {
    const int lane = threadIdx.x & 31, j = lane & 7;
    auto put = [&](int64_t o, int32_t w) {
        if (ladj32) ladj32[o] = local[w];
        else ladj16[o] = (uint16_t)local[w];
    };
    for_marked_rows(
        rp, memb, order_v, mark, nn,
        [&](int64_t p, int64_t b, int64_t e, uint32_t u, uint32_t cu, bool) {
            int64_t o = e > b ? loff[p] : 0;
            for (int64_t x = b + j; __any_sync(0xFFFFFFFFu, x < e); x += 8) {
                const int32_t w = x < e ? col[x] : -1;
                const bool keep = w >= 0 && memb[w] == cu && (uint32_t)w != u;
                const unsigned bal = (__ballot_sync(0xFFFFFFFFu, keep) >> (lane & 24)) & 0xFFu;
                if (keep) put(o + __popc(bal & ((1u << j) - 1u)), w);
                o += __popc(bal);
            }
        },
        [&](int64_t p, int64_t b, int64_t e, uint32_t u, uint32_t cu) {
            int64_t o = loff[p];
            for (int64_t x0 = b; x0 < e; x0 += 32) {
                const int64_t x = x0 + lane;
                const int32_t w = x < e ? col[x] : -1;
                const bool keep = w >= 0 && memb[w] == cu && (uint32_t)w != u;
                const unsigned bal = __ballot_sync(0xFFFFFFFFu, keep);
                if (keep) put(o + __popc(bal & ((1u << lane) - 1u)), w);
                o += __popc(bal);
            }
        });
}

// ---------------------------------------------------------------------------
// UnitHeap replica (intraGorderGreedy).  The list keeps buckets contiguous in
// descending key order; insertion is at the bucket front; extract-max takes
// the front of the highest non-empty bucket.  Storage is abstracted so one
// body serves thread-private arrays, shared memory and global workspaces.
// ---------------------------------------------------------------------------
struct HeapView {
    int* key;
    int* prev;
    int* next;
    int* bfirst;
    int* bsecond;
    int max_key;

    __device__ __forceinline__ void unlink(int idx) {
        const int p = prev[idx], nx = next[idx];
        if (p >= 0) next[p] = nx;
        if (nx >= 0) prev[nx] = p;
        const int k = key[idx];
        if (bfirst[k] == idx && bsecond[k] == idx) {
            bfirst[k] = bsecond[k] = -1;
        } else if (bfirst[k] == idx) {
            bfirst[k] = nx;
        } else if (bsecond[k] == idx) {
            bsecond[k] = p;
        }
    }
    __device__ __forceinline__ void link_front(int idx, int k) {
        key[idx] = k;
        if (bfirst[k] < 0) {
            int after = -1;
            for (int bk = k - 1; bk >= 0; --bk)
                if (bfirst[bk] >= 0) { after = bfirst[bk]; break; }
            int before = -1;
            for (int bk = k + 1; bk <= max_key; ++bk)
                if (bsecond[bk] >= 0) { before = bsecond[bk]; break; }
            prev[idx] = before;
            next[idx] = after;
            if (before >= 0) next[before] = idx;
            if (after >= 0) prev[after] = idx;
            bfirst[k] = bsecond[k] = idx;
        } else {
            const int old_first = bfirst[k];
            const int before_old = prev[old_first];
            prev[idx] = before_old;
            next[idx] = old_first;
            prev[old_first] = idx;
            if (before_old >= 0) next[before_old] = idx;
            bfirst[k] = idx;
        }
        if (k > max_key) max_key = k;
    }
    __device__ __forceinline__ void remove(int idx) {
        unlink(idx);
        prev[idx] = next[idx] = -1;
        key[idx] = -1;
        while (max_key > 0 && bfirst[max_key] < 0) --max_key;
    }
    __device__ __forceinline__ int extract_max() {
        while (max_key > 0 && bfirst[max_key] < 0) --max_key;
        const int idx = bfirst[max_key];
        if (idx >= 0) remove(idx);
        return idx;
    }
    __device__ __forceinline__ void bump(int idx, int delta) {
        const int old = key[idx];
        if (old < 0) return;
        if (delta < 0 && old <= 0) return;
        unlink(idx);
        link_front(idx, old + delta);
    }
};

// Runs the greedy placement of one community of sz vertices (local indices
// 0..sz-1 in vertex-id order).  ladj/loff give local adjacency; seed_deg the
// degrees for seeding; out_local receives local ids by local index.
template <typename LAdj>
__device__ void gorder_run(HeapView& h, int sz, int nbuckets, int window, const LAdj* __restrict__ ladj,
                           const int64_t* __restrict__ loff, const uint32_t* __restrict__ degs,
                           int* __restrict__ placed, uint32_t* __restrict__ out_local) {
    for (int i = 0; i < sz; ++i) {
        h.key[i] = 0;
        h.prev[i] = i - 1;
        h.next[i] = (i + 1 < sz) ? i + 1 : -1;
    }
    for (int b = 0; b < nbuckets; ++b) h.bfirst[b] = h.bsecond[b] = -1;
    h.bfirst[0] = 0;
    h.bsecond[0] = sz - 1;
    h.max_key = 0;
    int seed = 0;
    uint32_t seed_deg = degs[0];
    for (int i = 1; i < sz; ++i)
        if (degs[i] > seed_deg) { seed_deg = degs[i]; seed = i; }
    h.remove(seed);
    int nplaced = 0;
    placed[nplaced++] = seed;
    out_local[seed] = 0;
    for (int64_t k = loff[seed]; k < loff[seed + 1]; ++k) h.bump((int)ladj[k], +1);
    for (int lid = 1; lid < sz; ++lid) {
        const int best = h.extract_max();
        if (best < 0) {
            for (int i = 0; i < sz && lid < sz; ++i) {
                if (h.key[i] >= 0) {
                    h.remove(i);
                    out_local[i] = (uint32_t)lid++;
                }
            }
            break;
        }
        placed[nplaced++] = best;
        out_local[best] = (uint32_t)lid;
        for (int64_t k = loff[best]; k < loff[best + 1]; ++k) h.bump((int)ladj[k], +1);
        if (nplaced > window) {
            const int old_v = placed[nplaced - 1 - window];
            for (int64_t k = loff[old_v]; k < loff[old_v + 1]; ++k) h.bump((int)ladj[k], -1);
        }
    }
}

// One thread per community of 4..32 vertices; state in thread-private arrays.
template <typename LAdj>
__global__ void k_gorder_thread(const int32_t* __restrict__ list, const int32_t* __restrict__ count_p,
                                const int64_t* __restrict__ offs, const int64_t* __restrict__ ssize,
                                const uint32_t* __restrict__ order_v, const int64_t* __restrict__ rp,
                                const LAdj* __restrict__ ladj, const int64_t* __restrict__ loff,
                                int window, uint32_t* __restrict__ local_by_pos) {
    constexpr int kMaxB = 102 + 8;  // window <= 100
    const int32_t count = *count_p;
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < count; j += gridDim.x * blockDim.x) {
        const int32_t r = list[j];
        const int64_t base = offs[r];
        const int sz = (int)ssize[r];
        int key[kThreadGorderMax], prev[kThreadGorderMax], next[kThreadGorderMax], placed[kThreadGorderMax];
        int bf[kMaxB], bs[kMaxB];
        uint32_t degs[kThreadGorderMax];
        for (int i = 0; i < sz; ++i) {
            const uint32_t u = order_v[base + i];
            degs[i] = (uint32_t)(rp[u + 1] - rp[u]);
        }
        HeapView h{key, prev, next, bf, bs, 0};
        const int nb = min(window + 2, kMaxB);
        gorder_run<LAdj>(h, sz, nb, window, ladj, loff + base, degs, placed, local_by_pos + base);
    }
}

// ---------------------------------------------------------------------------
// The same UnitHeap, held so that a warp can apply a placed vertex's bumps
// together.  Each bucket is a stack in a push log: a bump pushes the vertex
// onto its new bucket's stack; an entry is live while it is its vertex's
// latest push and the vertex is unplaced; a bucket's front (extract-max,
// bucket-front insertion) is its newest live entry.  That is the linked
// list's order exactly: a bucket lists the vertices moved into it, newest
// first, then -- bucket 0 only -- the untouched vertices in local order (the
// initial pushes, vertex 0 last).  A batch of bumps by one placed vertex
// touches distinct vertices, so it is applied a warp at a time, pushes
// ordered as the reference processes the adjacency: entries are allocated in
// that order and each links to the previous push onto the same bucket (a
// __match_any_sync group).  Stale entries are skipped when a front is taken;
// when the log is full, a compaction keeps each live vertex's latest entry in
// push order and relinks the stacks.
// ---------------------------------------------------------------------------
struct LazyHeap {
    int* key;        // [S] bucket of each local vertex, -1 once placed
    int* lastpush;   // [S] log entry of its latest push
    int* log_v;      // [L] pushed vertex
    int* log_next;   // [L] entry below it in the same bucket (-1: bottom)
    int* top;        // [nb] newest entry of each bucket (-1: empty)
    int* last;       // [nb] compaction scratch
    int* ring;       // [window + 1] the last placed vertices
    uint32_t* degs;  // [S] degrees (seed choice)
    int L;
};

__host__ __device__ constexpr int lazy_log_cap(int S) { return 2 * S + 64; }
__host__ __device__ constexpr int64_t lazy_ws_ints(int64_t S, int nb, int window) {
    return 3 * S + 2 * (int64_t)lazy_log_cap((int)S) + 2 * nb + window + 1;
}

__device__ __forceinline__ LazyHeap lazy_view(int* ws, int64_t S, int nb, int window) {
    LazyHeap h;
    h.L = lazy_log_cap((int)S);
    h.key = ws;
    h.lastpush = h.key + S;
    h.log_v = h.lastpush + S;
    h.log_next = h.log_v + h.L;
    h.top = h.log_next + h.L;
    h.last = h.top + nb;
    h.ring = h.last + nb;
    h.degs = reinterpret_cast<uint32_t*>(h.ring + window + 1);
    return h;
}

template <typename LAdj>
__device__ void gorder_lazy_warp(const LazyHeap& h, int sz, int nb, int window, const LAdj* __restrict__ ladj,
                                 const int64_t* __restrict__ loff, uint32_t* __restrict__ out_local) {
    const int lane = threadIdx.x & 31;
    constexpr unsigned kFull = 0xFFFFFFFFu;
    const unsigned lower_lanes = (1u << lane) - 1u;
    // Bucket 0 lists 0..sz-1 with 0 in front: pushed sz-1 first, 0 last.
    for (int e = lane; e < sz; e += 32) {
        const int v = sz - 1 - e;
        h.log_v[e] = v;
        h.log_next[e] = e - 1;
        h.key[v] = 0;
        h.lastpush[v] = e;
    }
    for (int b = lane; b < nb; b += 32) h.top[b] = b == 0 ? sz - 1 : -1;
    // Seed: largest degree, first in local order.
    uint32_t bd = 0;
    int bi = -1;
    for (int i = lane; i < sz; i += 32)
        if (bi < 0 || h.degs[i] > bd) {
            bd = h.degs[i];
            bi = i;
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const uint32_t od = __shfl_xor_sync(kFull, bd, o);
        const int oi = __shfl_xor_sync(kFull, bi, o);
        if (oi >= 0 && (bi < 0 || od > bd || (od == bd && oi < bi))) {
            bd = od;
            bi = oi;
        }
    }
    const int seed = bi;
    int len = sz, max_key = 0;
    __syncwarp();
    if (lane == 0) {
        h.key[seed] = -1;
        out_local[seed] = 0;
        h.ring[0] = seed;
    }
    __syncwarp();

    auto compact = [&]() {
        for (int b = lane; b < nb; b += 32) h.last[b] = -1;
        __syncwarp();
        int nl = 0;
        for (int c0 = 0; c0 < len; c0 += 32) {
            const int e = c0 + lane;
            int v = -1, b = -1;
            bool keep = false;
            if (e < len) {
                v = h.log_v[e];
                b = h.key[v];
                keep = b >= 0 && h.lastpush[v] == e;
            }
            const unsigned kb = __ballot_sync(kFull, keep);
            const int ne = nl + __popc(kb & lower_lanes);
            const unsigned peers = __match_any_sync(kFull, keep ? b : -1 - lane);
            const unsigned below = peers & lower_lanes;
            const int ne_below = __shfl_sync(kFull, ne, below ? 31 - __clz(below) : lane);
            const int prev = keep ? (below ? ne_below : h.last[b]) : -1;
            __syncwarp();
            if (keep) {
                h.log_v[ne] = v;
                h.log_next[ne] = prev;
                h.lastpush[v] = ne;
                if ((peers >> lane) == 1u) h.last[b] = ne;
            }
            nl += __popc(kb);
            __syncwarp();
        }
        for (int b = lane; b < nb; b += 32) h.top[b] = h.last[b];
        len = nl;
        __syncwarp();
    };

    // bump(n, delta) for every neighbour n of v, in adjacency order.
    auto bump_all = [&](int v, int delta) {
        const int64_t e0 = loff[v], e1 = loff[v + 1];
        if (len + (e1 - e0) > h.L) compact();
        for (int64_t base = e0; base < e1; base += 32) {
            const int64_t idx = base + lane;
            int n = -1, k = -1;
            if (idx < e1) {
                n = (int)ladj[idx];
                k = h.key[n];
            }
            const bool app = k >= 0 && !(delta < 0 && k <= 0);
            const int t = k + delta;
            const unsigned ab = __ballot_sync(kFull, app);
            const int e = len + __popc(ab & lower_lanes);
            const unsigned peers = __match_any_sync(kFull, app ? t : -1 - lane);
            const unsigned below = peers & lower_lanes;
            const int e_below = __shfl_sync(kFull, e, below ? 31 - __clz(below) : lane);
            const int prev = app ? (below ? e_below : h.top[t]) : -1;
            __syncwarp();
            if (app) {
                h.log_v[e] = n;
                h.log_next[e] = prev;
                h.key[n] = t;
                h.lastpush[n] = e;
                if ((peers >> lane) == 1u) h.top[t] = e;
            }
            len += __popc(ab);
            int tm = app ? t : 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) tm = max(tm, __shfl_xor_sync(kFull, tm, o));
            max_key = max(max_key, tm);
            __syncwarp();
        }
    };

    bump_all(seed, +1);
    int nplaced = 1;
    for (int lid = 1; lid < sz; ++lid) {
        // extract-max: newest live entry of the highest non-empty bucket.
        int best = -1, b = max_key;
        if (lane == 0) {
            while (true) {
                int e = h.top[b];
                while (e >= 0) {
                    const int v = h.log_v[e];
                    if (h.key[v] == b && h.lastpush[v] == e) break;
                    e = h.log_next[e];
                }
                if (e >= 0) {
                    best = h.log_v[e];
                    h.top[b] = h.log_next[e];
                    h.key[best] = -1;
                    break;
                }
                h.top[b] = -1;
                if (b == 0) break;
                --b;
            }
        }
        best = __shfl_sync(kFull, best, 0);
        max_key = __shfl_sync(kFull, b, 0);
        if (best < 0) {   // no live vertex left: the rest in local order
            if (lane == 0)
                for (int i = 0; i < sz && lid < sz; ++i)
                    if (h.key[i] >= 0) {
                        h.key[i] = -1;
                        out_local[i] = (uint32_t)lid++;
                    }
            break;
        }
        if (lane == 0) {
            out_local[best] = (uint32_t)lid;
            h.ring[nplaced % (window + 1)] = best;
        }
        ++nplaced;
        __syncwarp();
        bump_all(best, +1);
        if (nplaced > window) {
            int old_v = 0;
            if (lane == 0) old_v = h.ring[(nplaced - 1 - window) % (window + 1)];
            old_v = __shfl_sync(kFull, old_v, 0);
            bump_all(old_v, -1);
        }
    }
    __syncwarp();
}

// One warp per community above kCtaGorderMax vertices, its workspace in
// global memory (one slice per CTA).
template <typename LAdj>
__global__ void k_gorder_warp(const int32_t* __restrict__ list, const int32_t* __restrict__ count_p,
                              const int64_t* __restrict__ offs, const int64_t* __restrict__ ssize,
                              const uint32_t* __restrict__ order_v, const int64_t* __restrict__ rp,
                              const LAdj* __restrict__ ladj, const int64_t* __restrict__ loff, int window,
                              uint32_t* __restrict__ local_by_pos, int* __restrict__ gws, int64_t cap) {
    const int32_t count = *count_p;
    const int lane = threadIdx.x & 31;
    const int nb = window + 2;
    const LazyHeap h = lazy_view(gws + (int64_t)blockIdx.x * lazy_ws_ints(cap, nb, window), cap, nb, window);
    for (int32_t j = blockIdx.x; j < count; j += gridDim.x) {
        const int32_t r = list[j];
        const int64_t base = offs[r];
        const int sz = (int)ssize[r];
        for (int i = lane; i < sz; i += 32) {
            const uint32_t u = order_v[base + i];
            h.degs[i] = (uint32_t)(rp[u + 1] - rp[u]);
        }
        __syncwarp();
        gorder_lazy_warp<LAdj>(h, sz, nb, window, ladj, loff + base, local_by_pos + base);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// The same greedy order without linked buckets (33..kCtaGorderMax vertices).
//
// The UnitHeap's next vertex is the unplaced one of the highest key that was
// moved into its bucket last.  A placed vertex moves its neighbours in
// adjacency order, and adjacency rows ascend in local index, so "last" is the
// larger (placement, bump sign) stamp and, within one stamp, the larger local
// index; vertices never moved stand in local order behind all others of bucket
// 0, which initial stamps sz - i below every later one express.  So a vertex is
// one word, key | stamp | index (0 once placed), a bump rewrites one word, and
// the next vertex is the largest word.
//
// Per placement: the vertex leaving the window lowers its neighbours, the
// placed one raises its own (each row's vertices are distinct, so plain stores;
// the lowering first but with the later stamp, which leaves the same words, as
// an unplaced neighbour of a leaving vertex has key >= 1: that vertex raised it
// when it was placed), then the maximum over all words, by one hardware
// reduction per level, gives the next vertex.  Short rows are bumped by the
// first warp alone, long ones by the CTA.
//
// What bounds it is that chain's latency, one placement after another, so the
// code is laid out for it: one warp without a barrier up to 1,024 vertices
// (eight vector loads a lane), 256 threads above; rows in shared memory; no
// branch on the chain (a lane without an entry bumps the dummy word, which is 0
// and stays so); the leaving vertex's row kept by the ring and fetched a
// placement ahead.  3,267 vertices of an RMAT graph of scale 12 took 9.5 ms with
// linked buckets (a warp, push stacks with lazy deletion), 3.3 ms with key and
// stamp in two arrays bumped by atomics over 512 threads, and 1.8 ms so.
// ---------------------------------------------------------------------------
constexpr int kShortRow = 128;              // rows the first warp bumps alone
constexpr int kMaxSmem = 226 * 1024;        // dynamic shared memory of a CTA (227 KB less the static part)

// Words padded to whole vector loads of the CTA; the dummy word follows.
__host__ __device__ constexpr int64_t scan_words(int64_t cap, int threads) {
    return (cap + 4 * threads - 1) / (4 * threads) * (4 * threads);
}
__host__ __device__ constexpr int64_t scan_smem_bytes(int64_t cap, int threads, int window, int word) {
    return (((scan_words(cap, threads) + 4) * word + (cap + 2) / 2 * 8 + (window + 1) * 8) + 15) & ~15ll;
}

__device__ __forceinline__ uint32_t warp_max_word(uint32_t v) { return __reduce_max_sync(0xFFFFFFFFu, v); }
__device__ __forceinline__ unsigned long long warp_max_word(unsigned long long v) {
    const uint32_t hi = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(v >> 32));
    const uint32_t lo = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(v >> 32) == hi ? (uint32_t)v : 0u);
    return (unsigned long long)hi << 32 | lo;
}

// Maximum over the CTA, in every thread (wm: a slot per warp).
template <int T, typename W>
__device__ __forceinline__ W cta_max_word(W v, W* wm) {
    v = warp_max_word(v);
    if (T > 32) {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        if (lane == 0) wm[w] = v;
        __syncthreads();
        v = warp_max_word(wm[lane & (T / 32 - 1)]);
    }
    return v;
}

// Maximum of four consecutive words.
__device__ __forceinline__ uint32_t quad_max(const uint32_t* p) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    return max(max(v.x, v.y), max(v.z, v.w));
}
__device__ __forceinline__ unsigned long long quad_max(const unsigned long long* p) {
    const ulonglong2 v = reinterpret_cast<const ulonglong2*>(p)[0], w = reinterpret_cast<const ulonglong2*>(p)[1];
    return max(max(v.x, v.y), max(w.x, w.y));
}

// One community's placements; row(i) is entry i of its local adjacency.  ib /
// sb: bits of the index and stamp fields of a word (the key above them).
template <typename LAdj, int T, typename W>
struct GorderScan {
    static constexpr int kW = T / 32;
    W *word, *wm;
    uint32_t* off;        // adjacency offsets relative to the community's first
    uint2* ring;          // rows of the last window + 1 placed vertices
    uint32_t* out;
    int sz, window, ib, sb;

    template <typename Row>
    __device__ __forceinline__ void run(int best, Row row) const {
        const int tid = threadIdx.x, lane = tid & 31;
        const bool first_warp = T == 32 || tid < 32;
        const W unit = (W)1 << (ib + sb), imask = ((W)1 << ib) - 1, smask = (((W)1 << sb) - 1) << ib;
        const int nwords = (int)scan_words(sz, T), dummy = nwords;
        auto bumped = [&](W v, W delta, W st) {   // the later stamp of this placement stays
            return v ? ((v & ~smask) + delta) | max(v & smask, st) : (W)0;
        };
        auto bump = [&](int n, W delta, W st) { word[n] = bumped(word[n], delta, st); };
        uint2 leave = make_uint2(0, 0);   // row of the vertex that leaves the window
        int m = dummy;                    // its entry of this lane (first warp)
        int wpos = 0;                     // ring slot of this placement
        W st = (W)(sz + 1) << ib;
        const W one = (W)1 << ib;
        W top = 0;
        for (int lid = 0;; ++lid, st += 2 * one) {
            // Here every thread has scanned; top: this warp's maximum (lid > 0).
            const uint32_t olen = leave.y - leave.x;
            const bool olong = T > 32 && olen > (uint32_t)kShortRow;
            if (olong) {
                for (uint32_t i = leave.x + tid; i < leave.y; i += T) bump(row(i), (W)0 - unit, st + one);
            } else if (first_warp) {
                bump(m, (W)0 - unit, st + one);
                if (olen > 32u)
                    for (uint32_t i = leave.x + lane + 32; i < leave.y; i += 32) bump(row(i), (W)0 - unit, st + one);
            }
            if (lid > 0) {
                if (T > 32) top = warp_max_word(wm[lane & (kW - 1)]);
                best = (int)(top & imask);
            }
            const uint32_t e0 = off[best], e1 = off[best + 1], elen = e1 - e0;
            const bool elong = T > 32 && elen > (uint32_t)kShortRow;
            if (tid == 0) {
                out[best] = (uint32_t)lid;
                ring[wpos] = make_uint2(e0, e1);
            }
            if (lid + 1 == sz) break;
            if (olong || elong) __syncthreads(); else __syncwarp();
            if (tid == 0) word[best] = 0;
            if (elong) {
                for (uint32_t i = e0 + tid; i < e1; i += T) bump(row(i), unit, st);
            } else if (first_warp) {
                bump((uint32_t)lane < elen ? row(e0 + lane) : dummy, unit, st);
                if (elen > 32u)
                    for (uint32_t i = e0 + lane + 32; i < e1; i += 32) bump(row(i), unit, st);
            }
            if (T > 32) __syncthreads(); else __syncwarp();
            // The next placement's leaving vertex is known: its row is fetched
            // while the maximum is formed.
            if (++wpos > window) wpos = 0;
            if (lid + 1 >= window) {
                leave = ring[wpos == window ? 0 : wpos + 1];
                m = first_warp && leave.x + lane < leave.y ? row(leave.x + lane) : dummy;
            }
            top = 0;
#pragma unroll 4
            for (int i = 4 * tid; i < nwords; i += 4 * T) top = max(top, quad_max(word + i));
            top = warp_max_word(top);
            if (T > 32) {
                if (lane == 0) wm[tid >> 5] = top;
                __syncthreads();
            }
        }
    }
};

template <typename LAdj, int T, typename W>
__global__ void __launch_bounds__(T)
k_gorder_scan(const int32_t* __restrict__ list, const int64_t* __restrict__ offs, const int64_t* __restrict__ ssize,
              const uint32_t* __restrict__ order_v, const int64_t* __restrict__ rp, const LAdj* __restrict__ ladj,
              const int64_t* __restrict__ loff, int window, int cap, int ib, int sb, uint32_t sadj_cap,
              uint32_t* __restrict__ local_by_pos) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned long long wm64[T / 32];
    GorderScan<LAdj, T, W> h;
    const int tid = threadIdx.x;
    const int32_t r = list[blockIdx.x];
    const int64_t base = offs[r];
    h.sz = (int)ssize[r];
    h.window = window;
    h.ib = ib;
    h.sb = sb;
    h.wm = reinterpret_cast<W*>(wm64);
    h.word = reinterpret_cast<W*>(smem_raw);
    h.ring = reinterpret_cast<uint2*>(h.word + scan_words(cap, T) + 4);
    h.off = reinterpret_cast<uint32_t*>(h.ring + window + 1);
    h.out = local_by_pos + base;
    LAdj* sadj = reinterpret_cast<LAdj*>(smem_raw + scan_smem_bytes(cap, T, window, sizeof(W)));
    const int sz = h.sz;
    const int64_t l0 = loff[base];
    const LAdj* adj = ladj + l0;
    // Seed: largest degree, first in local order.
    unsigned long long seed = 0;
    for (int i = tid; i < (int)scan_words(sz, T) + 4; i += T) {
        h.word[i] = i < sz ? (W)(sz - i) << ib | (W)i : (W)0;
        if (i < sz) {
            const uint32_t u = order_v[base + i];
            const unsigned long long d = (unsigned long long)(rp[u + 1] - rp[u]) << 32 | (uint32_t)(sz - i);
            seed = d > seed ? d : seed;
        }
    }
    for (int i = tid; i <= sz; i += T) h.off[i] = (uint32_t)(loff[base + i] - l0);
    const uint32_t total = (uint32_t)(loff[base + sz] - l0);
    const bool staged = total <= sadj_cap;
    if (staged)
        for (uint32_t i = tid; i < total; i += T) sadj[i] = adj[i];
    const int first = sz - (int)(uint32_t)cta_max_word<T, unsigned long long>(seed, wm64);
    if (T > 32) __syncthreads(); else __syncwarp();
    if (staged) h.run(first, [&](uint32_t i) { return (int)sadj[i]; });
    else h.run(first, [&](uint32_t i) { return (int)adj[i]; });
}

// ---------------------------------------------------------------------------
// Exact-order BFS from the hub (intraBFSFromHub), level-synchronous over all
// BFS communities at once.  Within one community the reference's FIFO order
// is reproduced: a vertex is discovered by the earliest frontier vertex (queue
// position) that reaches it and, within that parent, in row order.
//
// claim[w] is 0 once w is visited, else 1 + the smallest frontier index that
// has reached it in this level (all ones: none): the row offset within the
// parent needs no place in it, as a row names w once.  So a pass over the
// frontier's edges asks one 4-byte word per neighbour, and only a smaller
// frontier index looks at the community and claims; the edge that finds its own
// index there afterwards is w's.  Edges are dealt in runs of eight to a thread:
// a run's discoveries are one byte of bits, the children's positions a scan of
// the counts of 256 runs each.  (A 64-bit claim, a visited byte and the community per edge
// in both passes and an offset per edge took 0.73, 0.83 and 0.27 ms over the
// 21 levels of RCM on RMAT scale 19.)
// ---------------------------------------------------------------------------
__global__ void k_bfs_slots(const int32_t* __restrict__ list, const int32_t* __restrict__ count_p,
                            const uint32_t* __restrict__ order_v, const int64_t* __restrict__ offs,
                            const uint32_t* __restrict__ memb, int32_t* __restrict__ slot_of_comm,
                            int64_t* __restrict__ slot_base, int64_t* __restrict__ slot_size,
                            const int64_t* __restrict__ ssize) {
    const int32_t count = *count_p;
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < count; j += gridDim.x * blockDim.x) {
        const int32_t r = list[j];
        const uint32_t c = memb[order_v[offs[r]]];
        slot_of_comm[c] = j;
        slot_base[j] = offs[r];
        slot_size[j] = ssize[r];
    }
}

// Per slot the best (degree, tie) over its positions: the largest degree,
// first in position order (kMin = false), or the smallest, ties to the smaller id
// (kMin).  A thread per position; a block inside one community, as most are,
// reduces before its one atomic.
template <bool kMin>
__global__ void __launch_bounds__(kT)
k_slot_extreme(const uint32_t* __restrict__ order_v, int64_t nn, const uint32_t* __restrict__ memb,
               const int32_t* __restrict__ slot_of_comm, const int64_t* __restrict__ slot_base,
               const int64_t* __restrict__ rp, unsigned long long* __restrict__ key) {
    __shared__ unsigned long long s_best;
    __shared__ int32_t s_first;
    const unsigned long long none = kMin ? ~0ull : 0ull;
    auto better = [](unsigned long long x, unsigned long long y) { return kMin ? (x < y ? x : y) : (x > y ? x : y); };
    for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x; p0 < nn; p0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = p0 + threadIdx.x;
        int32_t j = -1;
        unsigned long long k = none;
        if (p < nn) {
            const uint32_t u = order_v[p];
            j = slot_of_comm[memb[u]];
            if (j >= 0) {
                const unsigned long long d = (unsigned long long)(rp[u + 1] - rp[u]);
                k = kMin ? d << 32 | u : d << 32 | (0xFFFFFFFFull - (unsigned long long)(p - slot_base[j]));
            }
        }
        if (threadIdx.x == 0) {
            s_first = j;
            s_best = none;
        }
        __syncthreads();
        const bool same = __syncthreads_and(j == s_first || p >= nn);
        if (same) {
            for (int o = 16; o > 0; o >>= 1) k = better(k, __shfl_xor_sync(0xFFFFFFFFu, k, o));
            if ((threadIdx.x & 31) == 0) {
                if (kMin) atomicMin(&s_best, k); else atomicMax(&s_best, k);
            }
            __syncthreads();
            if (threadIdx.x == 0 && s_first >= 0) {
                if (kMin) atomicMin(&key[s_first], s_best); else atomicMax(&key[s_first], s_best);
            }
        } else if (j >= 0) {
            if (kMin) atomicMin(&key[j], k); else atomicMax(&key[j], k);
        }
        __syncthreads();
    }
}

__global__ void k_bfs_init(const unsigned long long* __restrict__ hubkey, const int64_t* __restrict__ slot_base,
                           int32_t nslots, const uint32_t* __restrict__ order_v, int32_t* __restrict__ frontier,
                           uint32_t* __restrict__ claim, uint32_t* __restrict__ local, int64_t* __restrict__ qlen,
                           int64_t* __restrict__ fs, int64_t* __restrict__ fe) {
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nslots; j += gridDim.x * blockDim.x) {
        const int64_t k = (int64_t)(0xFFFFFFFFull - (hubkey[j] & 0xFFFFFFFFull));
        const uint32_t hub = order_v[slot_base[j] + k];
        frontier[j] = (int32_t)hub;
        claim[hub] = 0;
        local[hub] = 0;
        qlen[j] = 1;
        fs[j] = j;
        fe[j] = j + 1;
    }
}

__global__ void k_frontier_degrees(const int32_t* __restrict__ F, int64_t nf, const int64_t* __restrict__ rp,
                                   int64_t* __restrict__ fdeg) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nf; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t u = F[i];
        fdeg[i] = rp[u + 1] - rp[u];
    }
}

__device__ __forceinline__ int64_t upper_index(const int64_t* __restrict__ D, int64_t nf, int64_t e) {
    // largest i in [0, nf) with D[i] <= e
    int64_t lo = 0, hi = nf - 1;
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        if (D[mid] <= e) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Frontier edges in runs of kEdgeRun consecutive edge indices per thread: one
// binary search for the run's first edge, then the owning frontier vertex
// advances with the edge index.  nbr, idx: the run's neighbours (-1 past the last
// edge, T) and their frontier indices, all read together.
constexpr int kEdgeRun = 8;

__device__ __forceinline__ void edge_run(int64_t run, const int32_t* __restrict__ F, int64_t nf,
                                         const int64_t* __restrict__ D, int64_t T, const int64_t* __restrict__ rp,
                                         const int32_t* __restrict__ col, int32_t (&nbr)[kEdgeRun],
                                         int32_t (&idx)[kEdgeRun]) {
    const int64_t e0 = run * kEdgeRun;
    int64_t i = upper_index(D, nf, e0), next = D[i + 1];
    int64_t row = rp[F[i]] - D[i];
#pragma unroll
    for (int k = 0; k < kEdgeRun; ++k) {
        const int64_t e = e0 + k;
        nbr[k] = -1;
        idx[k] = 0;
        if (e < T) {
            if (e >= next) {
                do {
                    ++i;
                    next = D[i + 1];
                } while (e >= next);
                row = rp[F[i]] - D[i];
            }
            nbr[k] = col[row + e];
            idx[k] = (int32_t)i;
        }
    }
}

template <typename Skip, typename Fn>
__device__ __forceinline__ void for_edge_runs(const int32_t* __restrict__ F, int64_t nf, const int64_t* __restrict__ D,
                                              const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                                              Skip&& skip, Fn&& fn) {
    const int64_t T = D[nf];
    for (int64_t run = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; run * kEdgeRun < T;
         run += (int64_t)gridDim.x * blockDim.x) {
        if (skip(run)) continue;
        int32_t nbr[kEdgeRun], idx[kEdgeRun];
        edge_run(run, F, nf, D, T, rp, col, nbr, idx);
        fn(run, nbr, idx);
    }
}

inline int edge_grid(int64_t T) { return grid_for(ceil_div(T, kEdgeRun), 256); }

__global__ void __launch_bounds__(256)
k_bfs_claim(const int32_t* __restrict__ F, int64_t nf, const int64_t* __restrict__ D, const int64_t* __restrict__ rp,
            const int32_t* __restrict__ col, const uint32_t* __restrict__ memb, uint32_t* __restrict__ claim) {
    for_edge_runs(F, nf, D, rp, col, [](int64_t) { return false; },
                  [&](int64_t, const int32_t* nbr, const int32_t* idx) {
                      uint32_t c[kEdgeRun];
#pragma unroll
                      for (int k = 0; k < kEdgeRun; ++k) c[k] = nbr[k] >= 0 ? claim[nbr[k]] : 0u;
#pragma unroll
                      for (int k = 0; k < kEdgeRun; ++k)
                          if (c[k] > (uint32_t)idx[k] + 1u && memb[nbr[k]] == memb[F[idx[k]]])
                              atomicMin(&claim[nbr[k]], (uint32_t)idx[k] + 1u);
                  });
}

// Discoveries of the frontier's edges.  A CTA takes kRunBlock runs at a time:
// bits and first[run], the discoveries before the run within its block; count[]
// gets the block's.  Blocks past the last edge count none.
constexpr int kRunBlock = 256;

struct Discoveries {
    uint8_t* bits;      // per run: which of its edges discovered their neighbour
    uint16_t* first;
    int64_t* count;     // per block, then its exclusive scan (and the total behind)
    int64_t blocks;
};

__global__ void __launch_bounds__(kRunBlock)
k_bfs_flag(const int32_t* __restrict__ F, int64_t nf, const int64_t* __restrict__ D, const int64_t* __restrict__ rp,
           const int32_t* __restrict__ col, const uint32_t* __restrict__ claim, Discoveries d) {
    __shared__ int wsum[kRunBlock / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t T = D[nf];
    for (int64_t blk = blockIdx.x; blk < d.blocks; blk += gridDim.x) {
        const int64_t run = blk * kRunBlock + threadIdx.x;
        uint32_t b = 0;
        if (run * kEdgeRun < T) {
            int32_t nbr[kEdgeRun], idx[kEdgeRun];
            edge_run(run, F, nf, D, T, rp, col, nbr, idx);
            uint32_t c[kEdgeRun];
#pragma unroll
            for (int k = 0; k < kEdgeRun; ++k) c[k] = nbr[k] >= 0 ? claim[nbr[k]] : 0u;
#pragma unroll
            for (int k = 0; k < kEdgeRun; ++k) b |= c[k] == (uint32_t)idx[k] + 1u ? 1u << k : 0u;
        }
        const int mine = __popc(b);
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += x;
        }
        if (lane == 31) wsum[w] = incl;
        __syncthreads();
        int before = 0;
        for (int q = 0; q < w; ++q) before += wsum[q];
        d.bits[run] = (uint8_t)b;
        d.first[run] = (uint16_t)(before + incl - mine);
        if (threadIdx.x == kRunBlock - 1) d.count[blk] = before + incl;
        __syncthreads();
    }
}

__device__ __forceinline__ int64_t run_first(const Discoveries& d, int64_t run) {
    return d.count[run / kRunBlock] + d.first[run];
}

// Children found by the edges before edge e.
__device__ __forceinline__ int64_t children_before(int64_t e, const Discoveries& d) {
    const int64_t run = e / kEdgeRun;
    if (run >= d.blocks * kRunBlock) return d.count[d.blocks];
    return run_first(d, run) + __popc(d.bits[run] & ((1u << (e % kEdgeRun)) - 1u));
}

// Per community: where its children start in the next frontier this level.
__global__ void k_bfs_bases(int32_t nslots, const int64_t* __restrict__ fs, const int64_t* __restrict__ fe,
                            const int64_t* __restrict__ D, Discoveries d, int64_t* __restrict__ base,
                            int64_t* __restrict__ end) {
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nslots; j += gridDim.x * blockDim.x) {
        base[j] = children_before(D[fs[j]], d);
        end[j] = children_before(D[fe[j]], d);
    }
}

__device__ __forceinline__ void warp_add_sum(unsigned long long* out, unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(out, v);
}

// degree_sum: the entries of the next frontier.
__global__ void __launch_bounds__(256)
k_bfs_write(const int32_t* __restrict__ F, int64_t nf, const int64_t* __restrict__ D, const int64_t* __restrict__ rp,
            const int32_t* __restrict__ col, const uint32_t* __restrict__ memb, Discoveries d,
            const int32_t* __restrict__ slot_of_comm,
            const int64_t* __restrict__ qlen, const int64_t* __restrict__ base, int32_t* __restrict__ nextF,
            uint32_t* __restrict__ claim, uint32_t* __restrict__ local, unsigned long long* __restrict__ degree_sum) {
    unsigned long long sum = 0;
    for_edge_runs(F, nf, D, rp, col, [&](int64_t run) { return d.bits[run] == 0; },
                  [&](int64_t run, const int32_t* nbr, const int32_t*) {
                      const uint32_t b = d.bits[run];
                      int64_t p = run_first(d, run);
#pragma unroll
                      for (int k = 0; k < kEdgeRun; ++k) {
                          if (!((b >> k) & 1u)) continue;
                          const int32_t w = nbr[k], j = slot_of_comm[memb[w]];
                          nextF[p] = w;
                          claim[w] = 0;
                          local[w] = (uint32_t)(qlen[j] + (p - base[j]));
                          sum += (unsigned long long)(rp[w + 1] - rp[w]);
                          ++p;
                      }
                  });
    warp_add_sum(degree_sum, sum);
}

__global__ void k_bfs_advance(int32_t nslots, int64_t* __restrict__ qlen, int64_t* __restrict__ fs,
                              int64_t* __restrict__ fe, const int64_t* __restrict__ base,
                              const int64_t* __restrict__ end) {
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nslots; j += gridDim.x * blockDim.x) {
        qlen[j] += end[j] - base[j];
        fs[j] = base[j];
        fe[j] = end[j];
    }
}

// Unreached vertices of BFS communities, in vertex order after the BFS order.
__global__ void k_bfs_left_flags(const uint32_t* __restrict__ order_v, int64_t nn, const uint32_t* __restrict__ memb,
                                 const int32_t* __restrict__ slot_of_comm, const uint32_t* __restrict__ claim,
                                 int32_t* __restrict__ flag) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < nn; p += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t v = order_v[p];
        flag[p] = (slot_of_comm[memb[v]] >= 0 && claim[v] != 0) ? 1 : 0;
    }
}

__global__ void k_bfs_left_assign(const uint32_t* __restrict__ order_v, int64_t nn, const uint32_t* __restrict__ memb,
                                  const int32_t* __restrict__ slot_of_comm, const int32_t* __restrict__ flag,
                                  const int64_t* __restrict__ R, const int64_t* __restrict__ slot_base,
                                  const int64_t* __restrict__ qlen, uint32_t* __restrict__ local) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < nn; p += (int64_t)gridDim.x * blockDim.x) {
        if (!flag[p]) continue;
        const uint32_t v = order_v[p];
        const int32_t j = slot_of_comm[memb[v]];
        local[v] = (uint32_t)(qlen[j] + (R[p] - R[slot_base[j]]));
    }
}

// ---------------------------------------------------------------------------
// Reverse Cuthill-McKee (intraRCM, :4000-4134) over all communities at once,
// level-synchronous like the BFS above:
//   * start: minimum degree, ties to the smaller id;
//   * communities above 32 vertices: up to three George-Liu sweeps, each a
//     BFS from the current node whose start is *not* marked visited (so it
//     reappears on level 2, as in the reference); while the eccentricity
//     grows, the next node is the minimum-degree vertex of the last level,
//     first in level order;
//   * Cuthill-McKee BFS: a level's children are ordered by (parent position,
//     degree, id) -- claims give (parent, row offset) order, a stable sort by
//     (parent, degree) finishes it;
//   * the reached part is reversed, unreached vertices follow in id order.
// ---------------------------------------------------------------------------
// Frontier of a sweep: one start per participating slot, in slot order.
__global__ void k_rcm_frontier(int32_t nslots, const int32_t* __restrict__ part, const int64_t* __restrict__ pos,
                               const uint32_t* __restrict__ start, int mark, int32_t* __restrict__ F,
                               uint32_t* __restrict__ claim, int64_t* __restrict__ fs, int64_t* __restrict__ fe,
                               int64_t* __restrict__ qlen, int32_t* __restrict__ ecc,
                               unsigned long long* __restrict__ cand) {
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nslots; j += gridDim.x * blockDim.x) {
        fs[j] = pos[j];
        fe[j] = pos[j] + part[j];
        qlen[j] = part[j];
        ecc[j] = 0;
        cand[j] = ~0ull;
        if (part[j]) {
            F[pos[j]] = (int32_t)start[j];
            if (mark) claim[start[j]] = 0;
        }
    }
}

// Children in (parent, row offset) order with their parent's frontier index,
// and the largest of their degrees and their sum.
__global__ void __launch_bounds__(256)
k_rcm_write(const int32_t* __restrict__ F, int64_t nf, const int64_t* __restrict__ D, const int64_t* __restrict__ rp,
            const int32_t* __restrict__ col, Discoveries d, int32_t* __restrict__ nextF, int32_t* __restrict__ parent, uint32_t* __restrict__ claim,
            unsigned long long* __restrict__ max_deg, unsigned long long* __restrict__ degree_sum) {
    unsigned long long m = 0, sum = 0;
    for_edge_runs(F, nf, D, rp, col, [&](int64_t run) { return d.bits[run] == 0; },
                  [&](int64_t run, const int32_t* nbr, const int32_t* idx) {
                      const uint32_t b = d.bits[run];
                      int64_t p = run_first(d, run);
#pragma unroll
                      for (int k = 0; k < kEdgeRun; ++k) {
                          if (!((b >> k) & 1u)) continue;
                          const int32_t w = nbr[k];
                          nextF[p] = w;
                          parent[p] = idx[k];
                          claim[w] = 0;
                          const unsigned long long deg = (unsigned long long)(rp[w + 1] - rp[w]);
                          m = max(m, deg);
                          sum += deg;
                          ++p;
                      }
                  });
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(max_deg, m);
    warp_add_sum(degree_sum, sum);
}

// Last level of a slot whose next level is empty: minimum degree, first in
// level order (RCM) or smallest id (RCM++).
__global__ void k_rcm_last_level(const int32_t* __restrict__ F, int64_t nf, const int64_t* __restrict__ rp,
                                 const uint32_t* __restrict__ memb, const int32_t* __restrict__ slot_of_comm,
                                 const int64_t* __restrict__ bbase, const int64_t* __restrict__ bend, int by_id,
                                 unsigned long long* __restrict__ cand) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nf; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t u = F[i];
        const int32_t j = slot_of_comm[memb[u]];
        if (bend[j] != bbase[j]) continue;
        const unsigned long long tie = by_id ? (unsigned long long)(uint32_t)u : (unsigned long long)i;
        atomicMin(&cand[j], ((unsigned long long)(rp[u + 1] - rp[u]) << 32) | tie);
    }
}

__global__ void k_rcm_level_done(int32_t nslots, const int64_t* __restrict__ fs, const int64_t* __restrict__ fe,
                                 const int64_t* __restrict__ bbase, const int64_t* __restrict__ bend,
                                 const int32_t* __restrict__ F, int by_id, unsigned long long* __restrict__ cand,
                                 uint32_t* __restrict__ last_node, int32_t* __restrict__ ecc) {
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nslots; j += gridDim.x * blockDim.x) {
        if (fe[j] == fs[j]) continue;
        if (bend[j] > bbase[j]) {
            ++ecc[j];
        } else if (cand[j] != ~0ull) {
            const uint32_t lo = (uint32_t)(cand[j] & 0xFFFFFFFFull);
            last_node[j] = by_id ? lo : (uint32_t)F[lo];
            cand[j] = ~0ull;
        }
    }
}

// RCM++ start (RG:4185-4256): depth of each reached vertex from the seed.
__global__ void k_rcm_depth(const int32_t* __restrict__ F, int64_t nf, uint32_t level, uint32_t* __restrict__ depth) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nf; i += (int64_t)gridDim.x * blockDim.x)
        depth[F[i]] = level;
}

// Rank keys over the placement skeleton: (community rank, degree) or
// (community rank, ~depth); a stable sort keeps vertex order for ties.
__global__ void k_rcmpp_keys(const uint32_t* __restrict__ order_v, const uint32_t* __restrict__ ranks, int64_t nn,
                             const int64_t* __restrict__ rp, const uint32_t* __restrict__ depth, int low_bits,
                             uint32_t max_depth, int by_depth, uint64_t* __restrict__ keys,
                             uint32_t* __restrict__ pos) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < nn; p += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t v = order_v[p];
        const uint64_t low = by_depth ? (uint64_t)(max_depth - depth[v]) : (uint64_t)(rp[v + 1] - rp[v]);
        keys[p] = ((uint64_t)ranks[p] << low_bits) | low;
        pos[p] = (uint32_t)p;
    }
}

__global__ void k_rcmpp_rank(const uint32_t* __restrict__ sorted_pos, const uint32_t* __restrict__ ranks,
                             const int64_t* __restrict__ offs, int64_t nn, int64_t* __restrict__ score) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nn; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t p = sorted_pos[i];
        score[p] += i - offs[ranks[p]];
    }
}

// Least degree rank + depth rank per participating slot, ties to the smaller id.
__global__ void k_rcmpp_pick(const uint32_t* __restrict__ order_v, int64_t nn, const uint32_t* __restrict__ memb,
                             const int32_t* __restrict__ slot_of_comm, const int32_t* __restrict__ part,
                             const int64_t* __restrict__ score, unsigned long long* __restrict__ best) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < nn; p += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t v = order_v[p];
        const int32_t j = slot_of_comm[memb[v]];
        if (j < 0 || !part[j]) continue;
        atomicMin(&best[j], ((unsigned long long)score[p] << 32) | v);
    }
}

__global__ void k_rcmpp_start(int32_t nslots, const int32_t* __restrict__ part,
                              const unsigned long long* __restrict__ best, uint32_t* __restrict__ start) {
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nslots; j += gridDim.x * blockDim.x)
        if (part[j] && best[j] != ~0ull) start[j] = (uint32_t)(best[j] & 0xFFFFFFFFull);
}

// George-Liu step: keep sweeping while the eccentricity grows.
__global__ void k_rcm_gl_step(int32_t nslots, int32_t* __restrict__ part, const int32_t* __restrict__ ecc,
                              int32_t* __restrict__ prev_ecc, const uint32_t* __restrict__ last_node,
                              uint32_t* __restrict__ start, int32_t* __restrict__ still) {
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nslots; j += gridDim.x * blockDim.x) {
        if (!part[j]) continue;
        if (ecc[j] <= prev_ecc[j]) {
            part[j] = 0;
            continue;
        }
        prev_ecc[j] = ecc[j];
        start[j] = last_node[j];
        atomicAdd(still, 1);
    }
}

__global__ void k_rcm_keys(const int32_t* __restrict__ NF, const int32_t* __restrict__ parent, int64_t cnt,
                           const int64_t* __restrict__ rp, int degbits, uint64_t* __restrict__ keys,
                           uint32_t* __restrict__ vals) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < cnt; p += (int64_t)gridDim.x * blockDim.x) {
        const int32_t w = NF[p];
        keys[p] = ((uint64_t)parent[p] << degbits) | (uint64_t)(rp[w + 1] - rp[w]);
        vals[p] = (uint32_t)w;
    }
}

__global__ void k_rcm_assign(const uint32_t* __restrict__ sorted, int64_t cnt, const uint32_t* __restrict__ memb,
                             const int32_t* __restrict__ slot_of_comm, const int64_t* __restrict__ qlen,
                             const int64_t* __restrict__ bbase, int32_t* __restrict__ NF,
                             uint32_t* __restrict__ local) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < cnt; p += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t w = sorted[p];
        const int32_t j = slot_of_comm[memb[w]];
        NF[p] = (int32_t)w;
        local[w] = (uint32_t)(qlen[j] + (p - bbase[j]));
    }
}

// Reverse the reached part: local = reached - 1 - Cuthill-McKee position.
__global__ void k_rcm_reverse(const uint32_t* __restrict__ order_v, int64_t nn, const uint32_t* __restrict__ memb,
                              const int32_t* __restrict__ slot_of_comm, const uint32_t* __restrict__ claim,
                              const int64_t* __restrict__ qlen, uint32_t* __restrict__ local) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < nn; p += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t v = order_v[p];
        const int32_t j = slot_of_comm[memb[v]];
        if (j >= 0 && claim[v] == 0) local[v] = (uint32_t)(qlen[j] - 1 - local[v]);
    }
}

__global__ void k_rcm_init_slots(int32_t nslots, const int64_t* __restrict__ slot_size,
                                 const unsigned long long* __restrict__ key, uint32_t* __restrict__ start,
                                 int32_t* __restrict__ part, int32_t* __restrict__ prev_ecc) {
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nslots; j += gridDim.x * blockDim.x) {
        start[j] = (uint32_t)(key[j] & 0xFFFFFFFFull);
        part[j] = slot_size[j] > 32 ? 1 : 0;
        prev_ecc[j] = 0;
    }
}

__global__ void k_max_degree_of(const int32_t* __restrict__ list, int64_t cnt, const int64_t* __restrict__ rp,
                                unsigned long long* __restrict__ out) {
    unsigned long long m = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t u = list[i];
        const unsigned long long d = (unsigned long long)(rp[u + 1] - rp[u]);
        m = d > m ? d : m;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xFFFFFFFFu, m, o);
        m = t > m ? t : m;
    }
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

__global__ void k_fill_i32(int32_t* p, int64_t n, int32_t v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = v;
}

__global__ void k_gather_local(const uint32_t* __restrict__ order_v, const uint32_t* __restrict__ local_by_pos,
                               const uint8_t* __restrict__ mark, int64_t nn, uint32_t* __restrict__ local) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < nn; p += (int64_t)gridDim.x * blockDim.x)
        if (mark[p]) local[order_v[p]] = local_by_pos[p];
}

__global__ void k_final_assign(const uint32_t* __restrict__ order_v, const uint32_t* __restrict__ keys_sorted,
                               const int64_t* __restrict__ offs, const uint32_t* __restrict__ local, int64_t n,
                               uint32_t C, int32_t* __restrict__ new_ids) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t v = order_v[p];
        const uint32_t r = keys_sorted[p];
        new_ids[v] = (r < C) ? (int32_t)(offs[r] + local[v]) : (int32_t)p;
    }
}

template <typename T>
T read_dev(const T* p, cudaStream_t s) {
    T h;
    GB_CUDA(cudaMemcpyAsync(&h, p, sizeof(T), cudaMemcpyDeviceToHost, s));
    GB_CUDA(cudaStreamSynchronize(s));
    return h;
}

// The discoveries of one BFS level, in device memory sized for the graph.  A level
// needs no look at the device before its kernels are enqueued, and one after (two or
// three a level were a third of RCM's time): its number of edges comes with the
// children of the level before.  A first level's is bounded by its vertices and the
// largest degree; with that bound for every level, one hub had 1,500 levels of 40
// vertices pass over all of 142 M entries' runs (196.7 ms, 134.9 with the looks).
struct LevelBufs {
    DevBuf<uint8_t> bits;
    DevBuf<uint16_t> first;
    DevBuf<int64_t> count;
    DevBuf<unsigned long long> out;   // children, the largest of their degrees, the degrees' sum
    int64_t max_deg = 0, bound = 0, blocks = 0;
    int64_t edges = -1;               // the next frontier's entries, -1: not known
    static int64_t blocks_for(int64_t edges) { return ceil_div(ceil_div(edges, kEdgeRun), kRunBlock); }
    LevelBufs(const DeviceCSR& g, int64_t nn, const int32_t* order_v, cudaStream_t s)
        : bits(blocks_for(g.nnz) * kRunBlock, s), first(blocks_for(g.nnz) * kRunBlock, s),
          count(blocks_for(g.nnz) + 1, s), out(3, s) {
        GB_CUDA(cudaMemsetAsync(out, 0, 3 * sizeof(unsigned long long), s));
        k_max_degree_of<<<grid_for(nn, kT), kT, 0, s>>>(order_v, nn, g.row_ptr, out);
        GB_LAUNCH_CHECK();
        max_deg = (int64_t)read_dev(out.get(), s);
    }
    unsigned long long* max_child() const { return out.get() + 1; }
    unsigned long long* degree_sum() const { return out.get() + 2; }
    Discoveries view() const { return {bits.get(), first.get(), count.get(), blocks}; }
    // A frontier that is not the last level's children comes next.
    void restart() { edges = -1; }
    // Claims and discoveries of the frontier F[0, nf); D receives its edge offsets.
    void find(const DeviceCSR& g, const int32_t* F, int64_t nf, int64_t* D, const uint32_t* memb, uint32_t* claim,
              cudaStream_t s) {
        bound = edges >= 0 ? edges : nf > g.nnz / std::max<int64_t>(max_deg, 1) ? g.nnz : nf * max_deg;
        blocks = blocks_for(bound);
        GB_CUDA(cudaMemsetAsync(out, 0, 3 * sizeof(unsigned long long), s));
        k_frontier_degrees<<<grid_for(nf, kT), kT, 0, s>>>(F, nf, g.row_ptr, D);
        GB_LAUNCH_CHECK();
        exclusive_scan_i64_total(D, D, nf, D + nf, s);
        k_bfs_claim<<<edge_grid(bound), 256, 0, s>>>(F, nf, D, g.row_ptr, g.col, memb, claim);
        GB_LAUNCH_CHECK();
        if (blocks > 0) {
            k_bfs_flag<<<grid_for(blocks, 1), kRunBlock, 0, s>>>(F, nf, D, g.row_ptr, g.col, claim, view());
            GB_LAUNCH_CHECK();
        }
        exclusive_scan_i64_total(count, count, blocks, count.get() + blocks, s);
    }
    // Children of the level (after the kernels that write them).
    int64_t children(unsigned long long* max_child_deg, cudaStream_t s) {
        GB_CUDA(cudaMemcpyAsync(out, count.get() + blocks, sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
        unsigned long long h[3];
        GB_CUDA(cudaMemcpyAsync(h, out.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
        GB_CUDA(cudaStreamSynchronize(s));
        if (max_child_deg) *max_child_deg = h[1];
        edges = (int64_t)h[2];
        return (int64_t)h[0];
    }
};

}  // namespace

// Reverse Cuthill-McKee for the listed communities (see the kernels above).
// Returns the number of BFS levels run.
int64_t rcm_communities(const DeviceCSR& g, const uint32_t* memb, const int32_t* blist, const int32_t* count_p,
                        int32_t nslots, const uint32_t* order_v, const uint32_t* ranks, const int64_t* offs,
                        const int64_t* ssize, int64_t C, int64_t nn, bool pp, uint32_t* local,
                        cudaStream_t s, int64_t* launches) {
    const int64_t n = g.n;
    DevBuf<int32_t> slot_of_comm(C, s);
    GB_CUDA(cudaMemsetAsync(slot_of_comm, 0xFF, C * sizeof(int32_t), s));
    DevBuf<int64_t> slot_base(nslots, s), slot_size(nslots, s), qlen(nslots, s), fs(nslots, s), fe(nslots, s),
        bbase(nslots, s), bend(nslots, s), pos(nslots + 1, s);
    k_bfs_slots<<<grid_for(nslots, kT), kT, 0, s>>>(blist, count_p, order_v, offs, memb, slot_of_comm, slot_base,
                                                    slot_size, ssize);
    GB_LAUNCH_CHECK();
    DevBuf<unsigned long long> key(nslots, s), cand(nslots, s);
    GB_CUDA(cudaMemsetAsync(key, 0xFF, nslots * sizeof(unsigned long long), s));
    k_slot_extreme<true><<<grid_for(nn, kT), kT, 0, s>>>(order_v, nn, memb, slot_of_comm, slot_base, g.row_ptr, key);
    GB_LAUNCH_CHECK();
    DevBuf<uint32_t> start(nslots, s), last_node(nslots, s);
    DevBuf<int32_t> part(nslots, s), prev_ecc(nslots, s), ecc(nslots, s), still(1, s);
    k_rcm_init_slots<<<grid_for(nslots, kT), kT, 0, s>>>(nslots, slot_size, key, start, part, prev_ecc);
    GB_LAUNCH_CHECK();
    *launches += 4;
    DevBuf<uint32_t> claim(n, s);
    DevBuf<int32_t> F(nn + 1, s), NF(nn + 1, s), parent(nn + 1, s);
    DevBuf<int64_t> D(nn + 1, s);
    LevelBufs lv(g, nn, reinterpret_cast<const int32_t*>(order_v), s);
    int64_t levels = 0;
    DevBuf<uint32_t> depth(pp ? n : 0, s);
    // One BFS over the participating slots: a George-Liu sweep, the
    // Cuthill-McKee order (cm), or the RCM++ depths from the seed (dep).
    auto sweep = [&](bool cm, bool dep = false) -> void {
        exclusive_scan_i32_to_i64(part, pos, nslots, pos.get() + nslots, s);
        const int64_t np = read_dev(pos.get() + nslots, s);
        GB_CUDA(cudaMemsetAsync(claim, 0xFF, n * sizeof(uint32_t), s));
        k_rcm_frontier<<<grid_for(nslots, kT), kT, 0, s>>>(nslots, part, pos, start, (cm || dep) ? 1 : 0, F,
                                                           claim, fs, fe, qlen, ecc, cand);
        GB_LAUNCH_CHECK();
        *launches += 4;
        if (cm) {
            // the start is Cuthill-McKee position 0 of its community
            DevBuf<uint32_t> sorted(np > 0 ? np : 1, s);
            GB_CUDA(cudaMemsetAsync(bbase, 0, nslots * sizeof(int64_t), s));
            GB_CUDA(cudaMemcpyAsync(sorted, F.get(), np * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
            DevBuf<int64_t> zero(nslots, s);
            GB_CUDA(cudaMemsetAsync(zero, 0, nslots * sizeof(int64_t), s));
            k_rcm_assign<<<grid_for(np, kT), kT, 0, s>>>(sorted, np, memb, slot_of_comm, zero, pos, F, local);
            GB_LAUNCH_CHECK();
            *launches += 1;
        }
        int64_t nf = np;
        uint32_t level = 0;
        lv.restart();
        while (nf > 0) {
            ++levels;
            if (dep) {
                k_rcm_depth<<<grid_for(nf, kT), kT, 0, s>>>(F, nf, level, depth);
                GB_LAUNCH_CHECK();
                ++*launches;
            }
            ++level;
            lv.find(g, F, nf, D, memb, claim, s);
            k_bfs_bases<<<grid_for(nslots, kT), kT, 0, s>>>(nslots, fs, fe, D, lv.view(), bbase, bend);
            GB_LAUNCH_CHECK();
            k_rcm_write<<<edge_grid(lv.bound), 256, 0, s>>>(F, nf, D, g.row_ptr, g.col, lv.view(), NF, parent, claim,
                                                           lv.max_child(), lv.degree_sum());
            GB_LAUNCH_CHECK();
            unsigned long long md = 0;
            const int64_t next = lv.children(&md, s);
            if (!cm && !dep) {
                k_rcm_last_level<<<grid_for(nf, kT), kT, 0, s>>>(F, nf, g.row_ptr, memb, slot_of_comm, bbase, bend,
                                                                 pp ? 1 : 0, cand);
                GB_LAUNCH_CHECK();
                k_rcm_level_done<<<grid_for(nslots, kT), kT, 0, s>>>(nslots, fs, fe, bbase, bend, F, pp ? 1 : 0, cand,
                                                                     last_node, ecc);
                GB_LAUNCH_CHECK();
            } else if (cm && next > 0) {
                // Children of one parent by (degree, id): stable sort by (parent, degree).
                const int degbits = bits_for(md);
                const int pbits = bits_for((uint64_t)(nf > 1 ? nf - 1 : 1));
                DevBuf<uint64_t> keys(next, s);
                DevBuf<uint32_t> vals(next, s);
                k_rcm_keys<<<grid_for(next, kT), kT, 0, s>>>(NF, parent, next, g.row_ptr, degbits, keys, vals);
                GB_LAUNCH_CHECK();
                *launches += 3 + radix_sort_pairs_u64(keys, vals, next, degbits + pbits, s);
                k_rcm_assign<<<grid_for(next, kT), kT, 0, s>>>(vals, next, memb, slot_of_comm, qlen, bbase, NF,
                                                               local);
                GB_LAUNCH_CHECK();
            }
            k_bfs_advance<<<grid_for(nslots, kT), kT, 0, s>>>(nslots, qlen, fs, fe, bbase, bend);
            GB_LAUNCH_CHECK();
            *launches += 8;
            std::swap(F.ptr, NF.ptr);
            nf = next;
        }
    };
    if (pp) {
        // RCM++ start for the communities above 32 vertices: BFS depths from
        // the seed, ranks by (degree, id) and (depth descending, id), least sum.
        int32_t np_host = 0;
        {
            DevBuf<int64_t> tot(1, s);
            exclusive_scan_i32_to_i64(part, pos, nslots, tot, s);
            np_host = (int32_t)read_dev(tot.get(), s);
        }
        if (np_host > 0) {
            GB_CUDA(cudaMemsetAsync(depth, 0, n * sizeof(uint32_t), s));
            sweep(false, true);
            DevBuf<unsigned long long> mx(1, s);
            GB_CUDA(cudaMemsetAsync(mx, 0, sizeof(unsigned long long), s));
            k_max_degree_of<<<grid_for(nn, kT), kT, 0, s>>>(reinterpret_cast<const int32_t*>(order_v), nn, g.row_ptr,
                                                            mx);
            GB_LAUNCH_CHECK();
            const int degbits = bits_for(read_dev(mx.get(), s));
            const uint32_t max_depth = (uint32_t)std::max<int64_t>(0, levels);   // depth < levels run so far
            const int dbits = bits_for(max_depth);
            const int rbits = bits_for((uint64_t)(C > 1 ? C - 1 : 1));
            DevBuf<int64_t> score(nn, s);
            GB_CUDA(cudaMemsetAsync(score, 0, nn * sizeof(int64_t), s));
            DevBuf<uint64_t> keys(nn, s);
            DevBuf<uint32_t> sp(nn, s);
            for (int by_depth = 0; by_depth < 2; ++by_depth) {
                const int low = by_depth ? dbits : degbits;
                k_rcmpp_keys<<<grid_for(nn, kT), kT, 0, s>>>(order_v, ranks, nn, g.row_ptr, depth.get(), low, max_depth,
                                                            by_depth, keys, sp);
                GB_LAUNCH_CHECK();
                *launches += 2 + radix_sort_pairs_u64(keys, sp, nn, low + rbits, s);
                k_rcmpp_rank<<<grid_for(nn, kT), kT, 0, s>>>(sp, ranks, offs, nn, score);
                GB_LAUNCH_CHECK();
            }
            DevBuf<unsigned long long> best(nslots, s);
            GB_CUDA(cudaMemsetAsync(best, 0xFF, nslots * sizeof(unsigned long long), s));
            k_rcmpp_pick<<<grid_for(nn, kT), kT, 0, s>>>(order_v, nn, memb, slot_of_comm, part, score, best);
            GB_LAUNCH_CHECK();
            k_rcmpp_start<<<grid_for(nslots, kT), kT, 0, s>>>(nslots, part, best, start);
            GB_LAUNCH_CHECK();
            *launches += 3;
        }
    }
    // George-Liu sweeps (communities above 32 vertices), at most three.
    for (int it = 0; it < 3; ++it) {
        int32_t np_host = 0;
        {
            DevBuf<int64_t> tot(1, s);
            exclusive_scan_i32_to_i64(part, pos, nslots, tot, s);
            np_host = (int32_t)read_dev(tot.get(), s);
        }
        if (np_host == 0) break;
        sweep(false);
        GB_CUDA(cudaMemsetAsync(still, 0, sizeof(int32_t), s));
        k_rcm_gl_step<<<grid_for(nslots, kT), kT, 0, s>>>(nslots, part, ecc, prev_ecc, last_node, start, still);
        GB_LAUNCH_CHECK();
        *launches += 2;
        if (read_dev(still.get(), s) == 0) break;
    }
    // Cuthill-McKee BFS from the final starts, all communities.
    k_fill_i32<<<grid_for(nslots, kT), kT, 0, s>>>(part, nslots, 1);
    GB_LAUNCH_CHECK();
    sweep(true);
    // Reverse the reached part; unreached vertices follow in vertex order.
    k_rcm_reverse<<<grid_for(nn, kT), kT, 0, s>>>(order_v, nn, memb, slot_of_comm, claim, qlen, local);
    GB_LAUNCH_CHECK();
    DevBuf<int32_t> lflag(nn, s);
    DevBuf<int64_t> R(nn + 1, s);
    k_bfs_left_flags<<<grid_for(nn, kT), kT, 0, s>>>(order_v, nn, memb, slot_of_comm, claim, lflag);
    GB_LAUNCH_CHECK();
    exclusive_scan_i32_to_i64(lflag, R, nn, R.get() + nn, s);
    k_bfs_left_assign<<<grid_for(nn, kT), kT, 0, s>>>(order_v, nn, memb, slot_of_comm, lflag, R, slot_base, qlen,
                                                      local);
    GB_LAUNCH_CHECK();
    *launches += 7;
    return levels;
}

void compose_device(const DeviceCSR& g, const uint32_t* memb, const ComposeParams& p, int32_t* new_ids,
                    gbgpu_stats* st, cudaStream_t s) {
    const int64_t n = g.n;
    if (n == 0) return;
    int intra = p.intra_order;
    if (intra == kIntraDendrogram) intra = kIntraBFS;  // Leiden has no Rabbit dendrogram (:6668-6677)
    const bool sorted_intra = is_sorted_intra_order(intra);
    const bool random_intra = intra == kIntraRandom;
    GB_REQUIRE(intra == kIntraBFS || intra == kIntraGorder || intra == kIntraRCM || intra == kIntraRCMpp ||
                   sorted_intra || random_intra,
               GBGPU_E_UNSUPPORTED, "intra-community order not available on the GPU path");
    const int co = p.community_order;
    GB_REQUIRE(co == kSizeDesc || co == kSizeAsc || co == kDegreeDesc || co == kDegreeAsc || co == kIdentity,
               GBGPU_E_UNSUPPORTED, "community order not available on the GPU path");
    GB_REQUIRE(intra != kIntraGorder || p.gorder_window > 0, GBGPU_E_INVALID,
               "Local Gorder requires a positive window");
    GB_REQUIRE(p.gorder_window <= 100, GBGPU_E_INVALID, "Gorder window above 100");
    int64_t launches = 0;
    cudaEvent_t ev0, ev1;
    GB_CUDA(cudaEventCreate(&ev0));
    GB_CUDA(cudaEventCreate(&ev1));
    GB_CUDA(cudaEventRecord(ev0, s));

    // numComm = max(membership) + 1 (:6338-6343).
    DevBuf<uint32_t> scal(4, s);
    GB_CUDA(cudaMemsetAsync(scal, 0, 4 * sizeof(uint32_t), s));
    k_max_u32<<<grid_for(n, kT), kT, 0, s>>>(memb, n, scal.get());
    GB_LAUNCH_CHECK();
    const int64_t C = (int64_t)read_dev(scal.get(), s) + 1;
    GB_REQUIRE(C <= n, GBGPU_E_INVALID, "membership ids must be < n");

    DevBuf<uint32_t> csize(C, s);
    GB_CUDA(cudaMemsetAsync(csize, 0, C * sizeof(uint32_t), s));
    const bool need_deg = (co == kDegreeDesc || co == kDegreeAsc);
    DevBuf<unsigned long long> cdeg(need_deg ? C : 0, s);
    if (need_deg) GB_CUDA(cudaMemsetAsync(cdeg, 0, C * sizeof(unsigned long long), s));
    k_comm_sizes<<<grid_for(n, kT), kT, 0, s>>>(g.row_ptr, memb, n, csize, need_deg ? cdeg.get() : nullptr);
    GB_LAUNCH_CHECK();

    // Community order: stable sort of 0..C-1 by the order key.
    DevBuf<uint32_t> comm_order(C, s);
    {
        DevBuf<unsigned long long> maxdeg(1, s);
        GB_CUDA(cudaMemsetAsync(scal, 0, sizeof(uint32_t), s));
        GB_CUDA(cudaMemsetAsync(maxdeg, 0, sizeof(unsigned long long), s));
        k_max_u32_u64<<<grid_for(C, kT), kT, 0, s>>>(csize, need_deg ? cdeg.get() : nullptr, C, scal.get(), maxdeg.get());
        GB_LAUNCH_CHECK();
        const uint32_t max_size = read_dev(scal.get(), s);
        const unsigned long long max_deg = read_dev(maxdeg.get(), s);
        DevBuf<uint32_t> stage1;
        if (p.super_order != 0) {
            stage1.alloc(C, s);
            super_order_device(g, memb, csize, C, p.super_order, p.super_gamma, stage1, s, &launches);
        }
        DevBuf<uint64_t> keys(C, s);
        k_comm_keys<<<grid_for(C, kT), kT, 0, s>>>(co, csize, need_deg ? cdeg.get() : nullptr, C, max_size, max_deg,
                                                   stage1.get(), keys, comm_order);
        GB_LAUNCH_CHECK();
        int kbits = 0;
        if (co == kSizeDesc || co == kSizeAsc) kbits = bits_for(max_size);
        else if (co == kDegreeDesc || co == kDegreeAsc) kbits = bits_for(max_deg);
        launches += 4 + radix_sort_pairs_u64(keys, comm_order, C, kbits, s);
    }
    DevBuf<uint32_t> rank(C, s);
    DevBuf<int64_t> ssize(C, s);
    DevBuf<int64_t> offs(C + 1, s);
    k_rank<<<grid_for(C, kT), kT, 0, s>>>(comm_order, csize, C, rank, ssize);
    GB_LAUNCH_CHECK();
    exclusive_scan_i64_total(ssize, offs, C, offs.get() + C, s);
    const int64_t nn = read_dev(offs.get() + C, s);  // non-isolated vertices

    // Placement skeleton: stable sort of (rank(community) | C for isolated, v).
    DevBuf<uint32_t> vkeys(n, s), order_v(n, s);
    k_vertex_keys<<<grid_for(n, kT), kT, 0, s>>>(g.row_ptr, memb, rank, n, (uint32_t)C, vkeys, order_v);
    GB_LAUNCH_CHECK();
    const int vbits = bits_for((uint64_t)C);
    launches += 6 + radix_sort_pairs_u32(vkeys, order_v, n, vbits, s);
    DevBuf<int64_t> pos_of(n, s);
    DevBuf<uint32_t> local(n, s);
    k_positions<<<grid_for(n, kT), kT, 0, s>>>(order_v, vkeys, offs, n, (uint32_t)C, pos_of, local);
    GB_LAUNCH_CHECK();

    // Classify communities.
    DevBuf<int32_t> lists(kClasses * C, s);
    DevBuf<ClassCounts> cc(1, s);
    GB_CUDA(cudaMemsetAsync(cc, 0, sizeof(ClassCounts), s));
    k_classify<<<grid_for(C, kT), kT, 0, s>>>(ssize, C, intra, p.gorder_fallback, lists, cc);
    GB_LAUNCH_CHECK();
    ClassCounts hc = read_dev(cc.get(), s);
    launches += 1;

    cudaEvent_t ev_intra0, ev_intra1;
    GB_CUDA(cudaEventCreate(&ev_intra0));
    GB_CUDA(cudaEventCreate(&ev_intra1));
    GB_CUDA(cudaEventRecord(ev_intra0, s));

    // ---- Gorder communities ----
    const int32_t ng = hc.n[kClsThread] + hc.n[kClsWarp] + hc.n[kClsCta] + hc.n[kClsGlobal];
    if (ng > 0) {
        DevBuf<uint8_t> mark(nn, s);
        GB_CUDA(cudaMemsetAsync(mark, 0, nn, s));
        for (int cls = 1; cls < kClasses; ++cls) {
            if (cls == kClsBfs || hc.n[cls] == 0) continue;
            k_mark_gorder_positions<<<kNumSMs * 8, kT, 0, s>>>(lists.get() + cls * C, cc.get()->n + cls, offs, ssize, mark);
            GB_LAUNCH_CHECK();
            ++launches;
        }
        DevBuf<int64_t> loff(nn + 1, s);
        k_local_count<<<grid_for(nn * 8, kT), kT, 0, s>>>(g.row_ptr, g.col, memb, order_v, mark, nn, loff);
        GB_LAUNCH_CHECK();
        exclusive_scan_i64_total(loff, loff, nn, loff.get() + nn, s);
        const int64_t ltot = read_dev(loff.get() + nn, s);
        const bool wide = hc.gorder_max > 65535;
        DevBuf<uint16_t> l16(wide ? 0 : (ltot > 0 ? ltot : 1), s);
        DevBuf<uint32_t> l32(wide ? (ltot > 0 ? ltot : 1) : 0, s);
        k_local_fill<<<grid_for(nn * 8, kT), kT, 0, s>>>(g.row_ptr, g.col, memb, order_v, mark, local, loff, nn,
                                                     l16.get(), wide ? l32.get() : nullptr);
        GB_LAUNCH_CHECK();
        DevBuf<uint32_t> local_by_pos(nn, s);
        GB_CUDA(cudaMemsetAsync(local_by_pos, 0, nn * sizeof(uint32_t), s));
        launches += 5;
        auto run = [&](auto* ladj) {
            using LT = std::remove_pointer_t<decltype(ladj)>;
            // Largest communities first: theirs is the longest chain.
            auto scan = [&](auto threads, auto word, int cls, int max_size) {
                constexpr int T = decltype(threads)::value;
                using W = decltype(word);
                if (hc.n[cls] == 0) return;
                // Shared memory: the words of this call's largest community of
                // the class, and an equal share of what an SM has for the
                // adjacency, as far as all communities still run at once.  The
                // attribute is a constant, so concurrent callers never race on it.
                const int cap = (int)std::min<int64_t>(max_size, hc.gorder_max);
                const int ib = bits_for((uint64_t)cap - 1), sb = bits_for(3 * (uint64_t)cap + 2);
                const int64_t need = scan_smem_bytes(cap, T, p.gorder_window, sizeof(W));
                const int64_t per_sm = ceil_div(hc.n[cls], kNumSMs);
                const int64_t share = std::min<int64_t>(kMaxSmem, kMaxSmem / per_sm - 1024) - need;
                const int64_t sadj = std::max<int64_t>(0, std::min<int64_t>(share / (int64_t)sizeof(LT), ltot));
                const auto fn = k_gorder_scan<LT, T, W>;
                GB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
                fn<<<(unsigned)hc.n[cls], T, need + sadj * (int64_t)sizeof(LT), s>>>(
                    lists.get() + cls * C, offs, ssize, order_v, g.row_ptr, ladj, loff, p.gorder_window, cap, ib, sb,
                    (uint32_t)sadj, local_by_pos);
                GB_LAUNCH_CHECK();
                ++launches;
            };
            if (hc.n[kClsGlobal] > 0) {
                const int grid = std::min<int>(hc.n[kClsGlobal], kNumSMs * 4);
                const int64_t cap = hc.gorder_max;
                const int nb = p.gorder_window + 2;
                DevBuf<int> gws((int64_t)grid * lazy_ws_ints(cap, nb, p.gorder_window), s);
                k_gorder_warp<LT><<<grid, 32, 0, s>>>(lists.get() + kClsGlobal * C, cc.get()->n + kClsGlobal, offs,
                                                      ssize, order_v, g.row_ptr, ladj, loff, p.gorder_window,
                                                      local_by_pos, gws, cap);
                GB_LAUNCH_CHECK();
                ++launches;
            }
            // One 32-bit word holds key, stamp and index of the warp class at any
            // window and of 5,000 vertices at the default one; else 64 bits.
            const uint64_t cap = std::min<uint64_t>(kCtaGorderMax, hc.gorder_max);
            if (bits_for(cap - 1) + bits_for(3 * cap + 2) + bits_for(p.gorder_window + 1) <= 32)
                scan(std::integral_constant<int, 256>{}, uint32_t{}, kClsCta, kCtaGorderMax);
            else
                scan(std::integral_constant<int, 256>{}, (unsigned long long){}, kClsCta, kCtaGorderMax);
            scan(std::integral_constant<int, 32>{}, uint32_t{}, kClsWarp, kWarpGorderMax);
            if (hc.n[kClsThread] > 0) {
                k_gorder_thread<LT><<<grid_for(hc.n[kClsThread], 64), 64, 0, s>>>(
                    lists.get() + kClsThread * C, cc.get()->n + kClsThread, offs, ssize, order_v, g.row_ptr, ladj,
                    loff, p.gorder_window, local_by_pos);
                GB_LAUNCH_CHECK();
                ++launches;
            }
        };
        if (wide) run(l32.get()); else run(l16.get());
        k_gather_local<<<grid_for(nn, kT), kT, 0, s>>>(order_v, local_by_pos, mark, nn, local);
        GB_LAUNCH_CHECK();
        ++launches;
    }

    // ---- RCM: every community of two or more vertices ----
    const int32_t nbfs = hc.n[kClsBfs];
    int64_t levels = 0;
    if (nbfs > 0 && (intra == kIntraRCM || intra == kIntraRCMpp)) {
        levels = rcm_communities(g, memb, lists.get() + kClsBfs * C, cc.get()->n + kClsBfs, nbfs, order_v, vkeys, offs, ssize, C,
                                 nn, intra == kIntraRCMpp, local, s, &launches);
    }
    // ---- sorted orders: every community ----
    if (sorted_intra) sorted_communities(g, memb, intra, order_v, vkeys, offs, ssize, nn, local, s, &launches);
    // ---- intra_random: every community of two or more vertices ----
    if (random_intra)
        random_communities(memb, order_v, vkeys, offs, ssize, lists.get() + kClsBfs * C, cc.get()->n + kClsBfs, nbfs, nn, local, s,
                           &launches);
    // ---- BFS communities ----
    if (nbfs > 0 && intra != kIntraRCM && intra != kIntraRCMpp && !sorted_intra && !random_intra) {
        const int32_t* blist = lists.get() + kClsBfs * C;
        DevBuf<int32_t> slot_of_comm(C, s);
        GB_CUDA(cudaMemsetAsync(slot_of_comm, 0xFF, C * sizeof(int32_t), s));
        DevBuf<int64_t> slot_base(nbfs, s), slot_size(nbfs, s), qlen(nbfs, s), fs(nbfs, s), fe(nbfs, s),
            bbase(nbfs, s), bend(nbfs, s);
        k_bfs_slots<<<grid_for(nbfs, kT), kT, 0, s>>>(blist, cc.get()->n + kClsBfs, order_v, offs, memb, slot_of_comm,
                                                      slot_base, slot_size, ssize);
        GB_LAUNCH_CHECK();
        DevBuf<unsigned long long> hubkey(nbfs, s);
        GB_CUDA(cudaMemsetAsync(hubkey, 0, nbfs * sizeof(unsigned long long), s));
        k_slot_extreme<false><<<grid_for(nn, kT), kT, 0, s>>>(order_v, nn, memb, slot_of_comm, slot_base, g.row_ptr,
                                                              hubkey);
        GB_LAUNCH_CHECK();
        DevBuf<uint32_t> claim(n, s);
        GB_CUDA(cudaMemsetAsync(claim, 0xFF, n * sizeof(uint32_t), s));
        DevBuf<int32_t> F(nn + 1, s), NF(nn + 1, s);
        k_bfs_init<<<grid_for(nbfs, kT), kT, 0, s>>>(hubkey, slot_base, nbfs, order_v, F, claim, local, qlen, fs, fe);
        GB_LAUNCH_CHECK();
        launches += 4;
        int64_t nf = nbfs;
        DevBuf<int64_t> D(nn + 1, s);
        LevelBufs lv(g, nn, reinterpret_cast<const int32_t*>(order_v.get()), s);
        while (nf > 0) {
            ++levels;
            lv.find(g, F, nf, D, memb, claim, s);
            if (lv.bound == 0) break;
            k_bfs_bases<<<grid_for(nbfs, kT), kT, 0, s>>>(nbfs, fs, fe, D, lv.view(), bbase, bend);
            GB_LAUNCH_CHECK();
            k_bfs_write<<<edge_grid(lv.bound), 256, 0, s>>>(F, nf, D, g.row_ptr, g.col, memb, lv.view(),
                                                           slot_of_comm, qlen, bbase, NF, claim, local, lv.degree_sum());
            GB_LAUNCH_CHECK();
            k_bfs_advance<<<grid_for(nbfs, kT), kT, 0, s>>>(nbfs, qlen, fs, fe, bbase, bend);
            GB_LAUNCH_CHECK();
            const int64_t next = lv.children(nullptr, s);
            launches += 10;
            std::swap(F.ptr, NF.ptr);
            nf = next;
        }
        // Unreached vertices keep vertex order after the BFS order (:3978-3983).
        DevBuf<int32_t> lflag(nn, s);
        DevBuf<int64_t> R(nn + 1, s);
        k_bfs_left_flags<<<grid_for(nn, kT), kT, 0, s>>>(order_v, nn, memb, slot_of_comm, claim, lflag);
        GB_LAUNCH_CHECK();
        exclusive_scan_i32_to_i64(lflag, R, nn, R.get() + nn, s);
        k_bfs_left_assign<<<grid_for(nn, kT), kT, 0, s>>>(order_v, nn, memb, slot_of_comm, lflag, R, slot_base, qlen,
                                                          local);
        GB_LAUNCH_CHECK();
        launches += 5;
    }
    GB_CUDA(cudaEventRecord(ev_intra1, s));

    k_final_assign<<<grid_for(n, kT), kT, 0, s>>>(order_v, vkeys, offs, local, n, (uint32_t)C, new_ids);
    GB_LAUNCH_CHECK();
    launches += 1;
    GB_CUDA(cudaEventRecord(ev1, s));
    GB_CUDA(cudaEventSynchronize(ev1));
    if (st) {
        float ms = 0, ims = 0;
        cudaEventElapsedTime(&ms, ev0, ev1);
        cudaEventElapsedTime(&ims, ev_intra0, ev_intra1);
        st->compose_ms += ms;
        st->intra_ms += ims;
        st->num_communities = C;
        st->isolated = n - nn;
        st->gorder_communities = (int64_t)hc.gorder_communities;
        st->gorder_vertices = (int64_t)hc.gorder_vertices;
        st->gorder_max_community = hc.gorder_max;
        st->fallback_communities = (int64_t)hc.fallback_communities;
        st->fallback_vertices = (int64_t)hc.fallback_vertices;
        st->largest_community = hc.largest;
        st->bfs_levels = levels;
        st->kernel_launches += launches;
    }
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    cudaEventDestroy(ev_intra0);
    cudaEventDestroy(ev_intra1);
}

}  // namespace gb
