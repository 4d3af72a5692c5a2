// kernels.cu -- the graph kernels timed after a mapping, and the DBG arm.
//
// "Map + kernel" end-to-end time (README.md:127-129 of the reference) is the
// mapping plus r runs of a benchmark kernel on the relabelled graph.  These are
// the GPU counterparts of the reference's timed consumers:
//   PageRank, pull form with damping 0.85 (bench/src/pr.cc:40-90), Jacobi
//     sweeps until the L1 change falls below epsilon or max_iters;
//   BFS depths from a source, direction-optimising (bench/src/bfs.cc);
//   connected components as minimum vertex id per component (bench/src/cc.cc);
// and the selector's fallback arm, DBG (algorithm 5,
// bench/include/graphbrew/reorder/reorder_hub.h:267-342): vertices grouped
// into 8 degree buckets (avg/2, avg, 2avg .. 32avg, inf), highest bucket
// first, vertex-id order inside a bucket -- the order the reference's static
// OpenMP schedule produces for any thread count.
#include <algorithm>
#include <vector>

#include "gb_chunks.cuh"
#include "gb_common.cuh"
#include "gb_stages.h"

namespace gb {

namespace {

constexpr int kT = 256;
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kHubRow = 1024;   // frontier rows above this go to CTAs

// ---- PageRank ----
__global__ void k_pr_full(const int64_t* __restrict__ rp, int64_t n, uint8_t* __restrict__ full) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        full[v] = rp[v] != rp[v + 1];
}

// id: the rows with entries, in order, then n (n + 1 places in all); pos: how many
// come before a row.  And the rows that hold each chunk's first and last entry, in
// first and last, with their places in id.
struct PrChunks {
    int32_t *first, *last, *first_place, *last_place;
};

__global__ void k_pr_rows(const int64_t* __restrict__ rp, int64_t n, int64_t nnz, const int64_t* __restrict__ pos,
                          int32_t* __restrict__ id, PrChunks chunk) {
    const int lane = threadIdx.x & 31;
    auto go_on = [] { return false; };
    for (int64_t v0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; v0 < n;
         v0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = v0 + lane;
        const int64_t b = v < n ? rp[v] : 0, e = v < n ? rp[v + 1] : 0, p = v < n ? pos[v] : 0;
        if (b < e) id[p] = (int32_t)v;
        else if (v < n) id[n - (v - p)] = (int32_t)n;   // v - p empty rows before this one
        if (v == n - 1) id[p + (b < e)] = (int32_t)n;   // the place behind the last row
        note_chunk_first(b, e, (int32_t)v, chunk.first, go_on);
        note_chunk_first(b, e, (int32_t)p, chunk.first_place, go_on);
        note_chunk_last(b, e, (int32_t)v, nnz, chunk.last);
        note_chunk_last(b, e, (int32_t)p, nnz, chunk.last_place);
    }
}

__global__ void k_pr_init(const int64_t* __restrict__ rp, int64_t n, float init, float* __restrict__ score,
                          float* __restrict__ contrib, float* __restrict__ other) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int64_t d = rp[v + 1] - rp[v];
        score[v] = init;
        contrib[v] = d ? init / (float)d : 0.f;
        other[v] = 0.f;   // rows without entries are never written again
    }
}

// Sweep `it` of a batch does nothing once an earlier one has converged (err
// holds each sweep's L1 change, 0 for sweeps not run).
__device__ __forceinline__ bool pr_done(const double* err, int it, double epsilon) {
    return it > 0 && err[it - 1] < epsilon;
}

// L1 change added up over the CTA, one atomic each.
__device__ __forceinline__ void pr_add_change(double e, double* err) {
    __shared__ double ws[kT / 32];
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(kFull, e, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kT / 32; ++k) e += ws[k];
        if (e != 0.0) atomicAdd(err, e);
    }
}

struct PrArgs {
    const int64_t* rp;
    const int32_t* col;
    int64_t n, nnz;
    const int32_t* id;          // the rows with entries (k_pr_rows)
    const int32_t* chunk_row;   // row of the chunk's first entry, or the complement of its place in id
    float base, damp;
    const float* cin;
    float* cout;
    float* score;
    float* head;          // per chunk: sum of the row that began in an earlier chunk
    float* tail;          // per chunk: sum so far of the row that goes on in the next
    int32_t* tail_row;    // that row, or -1
    double* err;
    double epsilon;
};

__device__ __forceinline__ double pr_put(const PrArgs& a, int64_t u, float s, int64_t d) {
    const float ns = a.base + a.damp * s;
    const double e = fabsf(ns - a.score[u]);
    a.score[u] = ns;
    a.cout[u] = ns / (float)d;
    return e;
}

// One Jacobi sweep, score[u] = base + damp * sum contrib_in[v], over chunks of
// kEdgeChunk entries: a CTA gathers its chunk's contributions into shared
// memory (coalesced neighbour reads, sixteen gathers a thread in flight whatever
// the row lengths), then adds up the rows in it by a thread, eight lanes or a
// warp.  Rows that cross chunks leave partial sums to k_pr_join.
// Bound by the gather of contributions from L2, 4 bytes wanted of each 32-byte
// sector.  RMAT scale 20, 33 M entries: a warp per row 1.43 ms a sweep (nearly
// all of it the largest row's), lanes, warps and CTAs by row length 0.48 ms.
// Rows without entries keep the score that k_pr_first gives them.
// A lane adds its entries up with the rounding errors kept beside the sum (Knuth's
// two-sum), so that 24 of them in a row are no further off than a tree over a warp.
constexpr int kPrOwn = 24;      // rows up to this long by a thread
constexpr int kPrOctet = 256;   // up to this long by eight lanes, longer ones by a warp

struct PrSum {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float t = __fadd_rn(s, x), z = __fsub_rn(t, s);
        c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(x, z)));
        s = t;
    }
    __device__ __forceinline__ float value() const { return s + c; }
};

__global__ void __launch_bounds__(kT, 6) k_pr_sweep(PrArgs a, int it) {
    if (pr_done(a.err, it, a.epsilon)) return;
    __shared__ float val[kEdgeChunkPadded];
    __shared__ int32_t s_more, s_listed;
    __shared__ int sb[kT], se[kT];
    __shared__ float sums[kT];
    __shared__ uint8_t list[kT];   // rows left to more lanes
    static_assert(kT <= 256, "list entries");
    const int t = threadIdx.x, lane = t & 31;
    double err = 0.0;
    const int64_t chunks = (a.nnz + kEdgeChunk - 1) / kEdgeChunk;
    for (int64_t c = blockIdx.x; c < chunks; c += gridDim.x) {
        const int64_t e0 = c * kEdgeChunk, e1 = min(a.nnz, e0 + kEdgeChunk);
        const int len = (int)(e1 - e0);
        const int32_t row0 = a.chunk_row[c];
        {
            int32_t v[kEdgeChunk / kT];
#pragma unroll
            for (int k = 0; k < kEdgeChunk / kT; ++k) v[k] = k * kT + t < len ? a.col[e0 + k * kT + t] : -1;
#pragma unroll
            for (int k = 0; k < kEdgeChunk / kT; ++k)
                if (v[k] >= 0) val[chunk_pad(k * kT + t)] = a.cin[v[k]];
        }
        if (t == 0) {
            a.tail_row[c] = -1;
            s_listed = 0;
        }
        __syncthreads();
        // Rows from the one that holds entry e0, 256 at a time, until one starts past the chunk.
        const bool gaps = row0 < 0;
        for (int64_t u0 = gaps ? ~row0 : row0;; u0 += kT) {
            const int64_t u = gaps ? (int64_t)a.id[min(u0 + t, a.n)] : u0 + t;
            const int64_t rb = u < a.n ? a.rp[u] : e1, re = u < a.n ? a.rp[u + 1] : e1;
            const int b = (int)(max(rb, e0) - e0), e = rb < e1 ? (int)(min(re, e1) - e0) : b;
            if (t == kT - 1) s_more = rb < e1;
            float s = 0.f;
            if (e - b <= kPrOwn) {
                PrSum x;
                for (int i = b; i < e; ++i) x.add(val[chunk_pad(i)]);
                s = x.value();
            } else {
                list[atomicAdd(&s_listed, 1)] = (uint8_t)t;
                sb[t] = b;
                se[t] = e;
            }
            __syncthreads();
            const int listed = s_listed;
            for (int q = t >> 3; q - (t >> 3) < listed; q += kT / 8) {
                const int w = q < listed ? list[q] : 0;
                const bool mine = q < listed && se[w] - sb[w] <= kPrOctet;
                PrSum p;
                if (mine)
                    for (int i = sb[w] + (lane & 7); i < se[w]; i += 8) p.add(val[chunk_pad(i)]);
                float x = p.value();
                for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
                if (mine && (lane & 7) == 0) sums[w] = x;
            }
            for (int q = t >> 5; q < listed; q += kT / 32) {
                const int w = list[q];
                if (se[w] - sb[w] <= kPrOctet) continue;
                PrSum p;
                for (int i = sb[w] + lane; i < se[w]; i += 32) p.add(val[chunk_pad(i)]);
                float x = p.value();
                for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
                if (lane == 0) sums[w] = x;
            }
            __syncthreads();
            if (e - b > kPrOwn) s = sums[t];
            if (e > b) {
                if (rb < e0) a.head[c] = s;
                else if (re > e1) {
                    a.tail[c] = s;
                    a.tail_row[c] = (int32_t)u;
                } else err += pr_put(a, u, s, re - rb);
            }
            const bool more = s_more;
            if (t == 0) s_listed = 0;
            __syncthreads();
            if (!more) break;
        }
    }
    pr_add_change(err, a.err + it);
}

// Rows that cross chunks: the chunk where one begins adds up its parts, a warp
// each (the largest row of RMAT scale 22 has some hundred).
__global__ void __launch_bounds__(kT) k_pr_join(PrArgs a, int it) {
    if (pr_done(a.err, it, a.epsilon)) return;
    const int lane = threadIdx.x & 31;
    const int64_t chunks = (a.nnz + kEdgeChunk - 1) / kEdgeChunk;
    double err = 0.0;
    for (int64_t c = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; c < chunks;
         c += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int32_t u = a.tail_row[c];
        if (u < 0) continue;
        const int64_t rb = a.rp[u], re = a.rp[u + 1];
        const int64_t last = (re - 1) / kEdgeChunk;
        PrSum p;
        for (int64_t k = c + 1 + lane; k <= last; k += 32) p.add(a.head[k]);
        float s = p.value();
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
        if (lane == 0) err += pr_put(a, u, a.tail[c] + s, re - rb);
    }
    pr_add_change(err, a.err + it);
}

// Before the first sweep.  Rows without entries: the base score from here on.  In a
// graph with gaps, chunks of which more than a fifth of the rows are empty walk the
// rows with entries: first[c] becomes the complement of the first one's place.  (By
// their ids a gap of 4 M in one chunk took 6.6 ms a sweep.  Graphs without gaps are
// spared the list: 30 us for a 517 x 1023 grid.)
__global__ void __launch_bounds__(kT) k_pr_first(PrArgs a, PrChunks chunk) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t chunks = (a.nnz + kEdgeChunk - 1) / kEdgeChunk;
    for (int64_t c = tid; chunk.first_place && c < chunks; c += stride) {
        const int32_t place = chunk.first_place[c];
        const int32_t rows = chunk.last[c] - chunk.first[c] + 1, held = chunk.last_place[c] - place + 1;
        if (rows - held > rows / 5) chunk.first[c] = ~place;
    }
    double err = 0.0;
    for (int64_t v = tid; v < a.n; v += stride) {
        if (a.rp[v] != a.rp[v + 1]) continue;
        const float ns = a.base + a.damp * 0.f;
        err += fabsf(ns - a.score[v]);
        a.score[v] = ns;
    }
    pr_add_change(err, a.err);
}

// ---- BFS ----
struct BfsCtl {
    int32_t nf;                  // frontier vertices
    int32_t level;               // their depth
    unsigned long long edges;    // sum of their degrees
    int32_t nhub;                // frontier rows left to k_bfs_td_hub
};

// Appends v to the queue and its degree to the edge count, one atomic each per
// warp; every lane calls.
__device__ __forceinline__ void bfs_push(bool add, int32_t v, int64_t deg, int32_t* __restrict__ next, BfsCtl* ctl) {
    const int lane = threadIdx.x & 31;
    const unsigned bal = __ballot_sync(kFull, add);
    if (!bal) return;
    unsigned long long d = add ? (unsigned long long)deg : 0ull;
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(kFull, d, o);
    int32_t at = 0;
    if (lane == 0) {
        at = atomicAdd(&ctl->nf, __popc(bal));
        atomicAdd(&ctl->edges, d);
    }
    at = __shfl_sync(kFull, at, 0);
    if (add) next[at + __popc(bal & ((1u << lane) - 1u))] = v;
}

// Levels with a small frontier, all by one CTA: a level is a neighbour read, a
// claim, the claimed vertices' row offsets and two barriers, where a launch and
// the host's look at the counters cost 27 us (a 517 x 1023 grid has 1,533
// levels).  Runs until the frontier is empty or outgrows Q vertices /
// kSmallEdges entries; leaves the frontier in q.  With kBits the visited set is
// a bitmap in shared memory (zero but for the source on the first launch, else
// copied from `visited`), which takes the claim's L2 round trip out of the
// level: 3.1 us a level on that grid without it.
constexpr int kSmallEdges = 32768;
constexpr int kSmallT = 1024;
constexpr int kSmallOwn = 8;         // rows up to this long by their own thread
constexpr int kSmallPlain = 4096;    // frontiers of more entries ask for their rows' mean length
constexpr int kBitsQ = 2048;         // queue beside a bitmap
constexpr int kPlainQ = 4096;
constexpr int64_t kBitsMax = 160 * 1024 * 8;   // vertices whose bitmap shared memory holds

struct SmallEntry {
    int64_t b;      // the vertex's row
    int32_t deg;
    int32_t v;
};

template <bool kBits>
__global__ void __launch_bounds__(kSmallT)
k_bfs_small(const int64_t* __restrict__ rp, const int32_t* __restrict__ col, int32_t* __restrict__ depth,
            int32_t* __restrict__ q, const uint32_t* __restrict__ visited, int64_t words, int fresh,
            BfsCtl* __restrict__ ctl) {
    constexpr int kSmallQ = kBits ? kBitsQ : kPlainQ;
    extern __shared__ __align__(16) unsigned char bfs_smem[];
    SmallEntry* cur = reinterpret_cast<SmallEntry*>(bfs_smem);
    SmallEntry* nxt = cur + kSmallQ;
    uint32_t* bits = reinterpret_cast<uint32_t*>(nxt + kSmallQ);
    __shared__ int s_n[2];
    __shared__ unsigned s_edges[2];   // degrees cut at 2^16, below 2^31 for kSmallEdges claims
    __shared__ int s_warp[kSmallT / 32];
    const int tid = threadIdx.x, lane = tid & 31;
    int nf = ctl->nf, level = ctl->level;
    if (nf > kSmallQ || ctl->edges > (unsigned long long)kSmallEdges) return;
    unsigned edges = (unsigned)ctl->edges;
    if (kBits) {
        for (int64_t w = tid; w < words; w += kSmallT) bits[w] = fresh ? 0u : visited[w];
        __syncthreads();
        if (fresh && tid == 0) bits[q[0] >> 5] |= 1u << (q[0] & 31);
    }
    for (int i = tid; i < nf; i += kSmallT) {
        const int32_t v = q[i];
        cur[i] = SmallEntry{rp[v], (int32_t)(rp[v + 1] - rp[v]), v};
    }
    int par = 0;
    if (tid < 2) {
        s_n[tid] = 0;
        s_edges[tid] = 0;
    }
    __syncthreads();
    // Up to four neighbours of each lane at once: their claims and their rows
    // are in flight together, so a level waits for two round trips, and the
    // queue's counters take one shared-memory atomic a warp (one per vertex
    // serialised: 3.2 us a level).  Every lane of the warp calls.
    auto claim4 = [&](const int32_t* nbr, int count, bool look) {
        int32_t v[4];
        int old[4];
        int64_t b[4], e[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = k < count ? nbr[k] : -1;
        if (!kBits && look) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (v[k] >= 0 && depth[v[k]] >= 0) v[k] = -1;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            old[k] = 0;
            b[k] = e[k] = 0;
            if (v[k] >= 0) {
                if (kBits) {
                    const uint32_t bit = 1u << (v[k] & 31);
                    old[k] = (atomicOr(&bits[v[k] >> 5], bit) & bit) ? 0 : -1;
                    if (old[k] == 0) continue;
                    depth[v[k]] = level + 1;
                } else {
                    old[k] = atomicCAS(&depth[v[k]], -1, level + 1);
                }
                b[k] = rp[v[k]];
                e[k] = rp[v[k] + 1];
            }
        }
        int mine = 0;
        unsigned deg = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (old[k] == -1) {
                ++mine;
                deg += (unsigned)min(e[k] - b[k], (int64_t)65536);
            }
        if (!__any_sync(kFull, mine != 0)) return;
        int at = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(kFull, at, o);
            if (lane >= o) at += x;
        }
        deg = __reduce_add_sync(kFull, deg);
        int base = 0;
        if (lane == 31) {
            base = atomicAdd(&s_n[par], at);
            atomicAdd(&s_edges[par], deg);
        }
        at += __shfl_sync(kFull, base, 31) - mine;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (old[k] == -1) {
                if (at < kSmallQ) nxt[at] = SmallEntry{b[k], (int32_t)(e[k] - b[k]), v[k]};
                else q[at] = v[k];
                ++at;
            }
    };
    // A level of rows above kSmallOwn entries on average: entries dealt to the lanes one
    // by one, 192 a warp at a time, whatever the rows.  Degrees become their inclusive
    // prefix, where an entry's row is searched for; the next frontier's rows are looked
    // up once a level.  Row after row by a warp, 500 levels of 2,000 vertices with 16
    // neighbours took 27.8 ms, where a launch and a look a level had taken 17.1; so
    // 9.1.  Without a bitmap, 700 levels: 46.0, 24.3 and 17.7.
    auto flat_level = [&]() {
        constexpr int kPer = kSmallQ / kSmallT, kLane = 6, kRows = 2;
        const int i0 = tid * kPer;
        int sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) sum += i0 + k < nf ? cur[i0 + k].deg : 0;
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += x;
        }
        if (lane == 31) s_warp[tid >> 5] = incl;
        __syncthreads();
        int run = incl - sum + __reduce_add_sync(kFull, lane < tid >> 5 ? s_warp[lane] : 0);
#pragma unroll
        for (int k = 0; k < kPer; ++k)
            if (i0 + k < nf) cur[i0 + k].deg = run += cur[i0 + k].deg;
        __syncthreads();
        const int total = cur[nf - 1].deg;
        int top = 1;
        while (top < nf) top <<= 1;
        // The first entry's row by search, the later ones' by walking on: a search for
        // each took most of the level's instructions.
        auto fetch = [&](int k0, int32_t (&v)[kLane]) {
            int at = 0;
            for (int half = top >> 1; half > 0; half >>= 1)
                if (at + half < nf && cur[at + half - 1].deg <= k0 + lane) at += half;
#pragma unroll
            for (int k = 0; k < kLane; ++k) {
                const int e = k0 + 32 * k + lane;
                v[k] = -1;
                if (e < total) {
                    while (cur[at].deg <= e) ++at;
                    v[k] = col[cur[at].b + (e - (at ? cur[at - 1].deg : 0))];
                }
            }
        };
        int32_t ahead[kLane];
        int k0 = (tid - lane) * kLane;
        fetch(k0, ahead);
        while (k0 < total) {
            int32_t v[kLane];
#pragma unroll
            for (int k = 0; k < kLane; ++k) v[k] = ahead[k];
            k0 += kSmallT * kLane;
            if (k0 < total) fetch(k0, ahead);   // in flight during the claims
            if (!kBits) {
#pragma unroll
                for (int k = 0; k < kLane; ++k)
                    if (v[k] >= 0 && depth[v[k]] >= 0) v[k] = -1;
            }
            // Claims in flight together.
            int32_t old[kLane];
#pragma unroll
            for (int k = 0; k < kLane; ++k) {
                old[k] = 0;
                if (v[k] < 0) continue;
                if (kBits) old[k] = (int32_t)(atomicOr(&bits[v[k] >> 5], 1u << (v[k] & 31)) >> (v[k] & 31) & 1u) - 1;
                else old[k] = atomicCAS(&depth[v[k]], -1, level + 1);
            }
            int mine = 0;
#pragma unroll
            for (int k = 0; k < kLane; ++k) {
                if (old[k] != -1) continue;
                if (kBits) depth[v[k]] = level + 1;
                ++mine;
            }
            if (!__any_sync(kFull, mine != 0)) continue;
            int put = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(kFull, put, o);
                if (lane >= o) put += x;
            }
            int base = 0;
            if (lane == 31) base = atomicAdd(&s_n[par], put);
            put += __shfl_sync(kFull, base, 31) - mine;
#pragma unroll
            for (int k = 0; k < kLane; ++k)
                if (old[k] == -1) {
                    if (put < kSmallQ) nxt[put].v = v[k];
                    else q[put] = v[k];
                    ++put;
                }
        }
        __syncthreads();
        const int found = s_n[par];
        unsigned deg = 0;
        for (int i0 = tid; i0 < found; i0 += kRows * kSmallT) {
            int32_t u[kRows];
            int64_t b[kRows], e[kRows];
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                const int i = i0 + k * kSmallT;
                u[k] = i < min(found, kSmallQ) ? nxt[i].v : i < found ? q[i] : -1;
            }
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                b[k] = u[k] >= 0 ? rp[u[k]] : 0;
                e[k] = u[k] >= 0 ? rp[u[k] + 1] : 0;
            }
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                const int i = i0 + k * kSmallT;
                if (i < min(found, kSmallQ)) nxt[i] = SmallEntry{b[k], (int32_t)(e[k] - b[k]), u[k]};
                deg += (unsigned)min(e[k] - b[k], (int64_t)65536);
            }
        }
        deg = __reduce_add_sync(kFull, deg);
        if (lane == 0) atomicAdd(&s_edges[par], deg);
    };
    auto next_level = [&]() {
        __syncthreads();
        nf = s_n[par];
        edges = s_edges[par];
        par ^= 1;
        if (tid == 0) {
            s_n[par] = 0;
            s_edges[par] = 0;
        }
        ++level;
        SmallEntry* t = cur;
        cur = nxt;
        nxt = t;
        __syncthreads();
    };
    while (nf > 0 && nf <= kSmallQ && edges <= (unsigned)kSmallEdges) {
        if (edges > (unsigned)(kSmallOwn * nf)) {
            flat_level();
            next_level();
            continue;
        }
        // Asked again after a level of many entries; smaller ones go on without.
        const unsigned most = edges <= (unsigned)kSmallPlain ? kSmallPlain : 0;
        do {
            for (int i0 = tid - lane; i0 < nf; i0 += kSmallT) {
                const int i = i0 + lane;
                SmallEntry u{0, 0, 0};
                if (i < nf) u = cur[i];
                const int own = u.deg <= kSmallOwn ? u.deg : 0;
                for (int k = 0; __any_sync(kFull, k < own); k += 4) claim4(col + u.b + k, own - k, false);
                unsigned todo = __ballot_sync(kFull, u.deg > kSmallOwn);
                while (todo) {
                    const int src = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const int64_t b = __shfl_sync(kFull, u.b, src);
                    const int d = __shfl_sync(kFull, u.deg, src);
                    for (int k = 0; k < d; k += 128) claim4(col + b + k + 4 * lane, d - k - 4 * lane, true);
                }
            }
            next_level();
        } while (nf > 0 && nf <= kSmallQ && edges <= most);
    }
    for (int i = tid; i < min(nf, kSmallQ); i += kSmallT) q[i] = cur[i].v;
    if (tid == 0) {
        ctl->nf = nf;
        ctl->level = level;
        ctl->edges = edges;
    }
}

// Top-down step: a warp per frontier vertex, rows above kHubRow to the hub
// list.  The counters of the next frontier start at zero.
__global__ void __launch_bounds__(kT)
k_bfs_td(const int64_t* __restrict__ rp, const int32_t* __restrict__ col, const int32_t* __restrict__ frontier,
         int64_t nf, int32_t* __restrict__ depth, int32_t level, int32_t* __restrict__ next, int32_t* __restrict__ hubs,
         BfsCtl* __restrict__ ctl) {
    const int lane = threadIdx.x & 31;
    const int64_t wid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = wid; i < nf; i += nw) {
        const int32_t u = frontier[i];
        const int64_t b = rp[u], e = rp[u + 1];
        if (e - b > kHubRow) {
            if (lane == 0) hubs[atomicAdd(&ctl->nhub, 1)] = u;
            continue;
        }
        for (int64_t x0 = b; x0 < e; x0 += 32) {
            const int64_t x = x0 + lane;
            const int32_t v = x < e ? col[x] : -1;
            const bool add = v >= 0 && depth[v] < 0 && atomicCAS(&depth[v], -1, level + 1) == -1;
            bfs_push(add, v, add ? rp[v + 1] - rp[v] : 0, next, ctl);
        }
    }
}

__global__ void __launch_bounds__(kT)
k_bfs_td_hub(const int64_t* __restrict__ rp, const int32_t* __restrict__ col, const int32_t* __restrict__ hubs,
             int32_t* __restrict__ depth, int32_t level, int32_t* __restrict__ next, BfsCtl* __restrict__ ctl) {
    const int nh = ctl->nhub;
    int64_t turn = 0;   // chunks of all hubs dealt to the CTAs in turn
    for (int i = 0; i < nh; ++i) {
        const int32_t u = hubs[i];
        const int64_t b = rp[u], e = rp[u + 1];
        const int64_t chunks = (e - b + kT - 1) / kT;
        int64_t c = ((int64_t)blockIdx.x - turn) % gridDim.x;
        if (c < 0) c += gridDim.x;
        for (; c < chunks; c += gridDim.x) {
            const int64_t x = b + c * kT + threadIdx.x;
            const int32_t v = x < e ? col[x] : -1;
            const bool add = v >= 0 && depth[v] < 0 && atomicCAS(&depth[v], -1, level + 1) == -1;
            bfs_push(add, v, add ? rp[v + 1] - rp[v] : 0, next, ctl);
        }
        turn = (turn + chunks) % gridDim.x;
    }
}

// Bitmaps of the visited vertices and of the frontier.
__global__ void k_bfs_bits(const int32_t* __restrict__ depth, int64_t n, int32_t level, uint32_t* __restrict__ visited,
                           uint32_t* __restrict__ front) {
    const int lane = threadIdx.x & 31;
    const int64_t words = (n + 31) / 32;
    for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < words;
         w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t v = w * 32 + lane;
        const int32_t d = v < n ? depth[v] : 0;
        const unsigned vis = __ballot_sync(kFull, d >= 0), fr = __ballot_sync(kFull, v < n && d == level);
        if (lane == 0) {
            visited[w] = vis;
            front[w] = fr;
        }
    }
}

// Bottom-up step: a warp owns 32 consecutive vertices and their bitmap words.
// Most unvisited vertices meet the frontier within a few neighbours, so a
// vertex first looks through kBuOwn entries by itself; the rest of a longer row
// is the warp's.  The frontier is read as bits (128 KB at 2^20 vertices, mostly
// L1 hits) where the depths were a 4 MB gather.
constexpr int kBuOwn = 16;

__global__ void __launch_bounds__(kT)
k_bfs_bu(const int64_t* __restrict__ rp, const int32_t* __restrict__ col, int64_t n, int32_t* __restrict__ depth,
         int32_t level, uint32_t* __restrict__ visited, const uint32_t* __restrict__ front,
         uint32_t* __restrict__ next, BfsCtl* __restrict__ ctl) {
    const int lane = threadIdx.x & 31;
    const int64_t words = (n + 31) / 32;
    auto in_front = [&](int64_t x) {
        const uint32_t v = (uint32_t)col[x];
        return (front[v >> 5] >> (v & 31)) & 1u;
    };
    int32_t found = 0;
    unsigned long long edges = 0;
    for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < words;
         w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const uint32_t vis = visited[w];
        if (vis == kFull) {
            if (lane == 0) next[w] = 0;
            continue;
        }
        const int64_t v = w * 32 + lane;
        int64_t b = 0, e = 0;
        if (!((vis >> lane) & 1u)) {   // v < n: bits past the end are set
            b = rp[v];
            e = rp[v + 1];
        }
        bool hit = false;
        const int64_t own = min(e, b + kBuOwn);
        for (int64_t x = b; x < own && !hit; ++x) hit = in_front(x);
        unsigned todo = __ballot_sync(kFull, !hit && e > own);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const int64_t es = __shfl_sync(kFull, e, src);
            bool any = false;
            for (int64_t x0 = __shfl_sync(kFull, own, src); x0 < es && !any; x0 += 128) {
                bool h = false;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (x0 + 32 * k + lane < es) h |= in_front(x0 + 32 * k + lane) != 0;
                any = __any_sync(kFull, h);
            }
            if (lane == src) hit = any;
        }
        const unsigned bal = __ballot_sync(kFull, hit);
        if (hit) {
            depth[v] = level + 1;
            ++found;
            edges += (unsigned long long)(e - b);
        }
        if (lane == 0) {
            next[w] = bal;
            visited[w] = vis | bal;
        }
    }
    __shared__ int32_t s_found;
    __shared__ unsigned long long s_edges;
    if (threadIdx.x == 0) {
        s_found = 0;
        s_edges = 0;
    }
    __syncthreads();
    for (int o = 16; o > 0; o >>= 1) {
        found += __shfl_xor_sync(kFull, found, o);
        edges += __shfl_xor_sync(kFull, edges, o);
    }
    if (lane == 0 && found) {
        atomicAdd(&s_found, found);
        atomicAdd(&s_edges, edges);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_found) {
        atomicAdd(&ctl->nf, s_found);
        atomicAdd(&ctl->edges, s_edges);
    }
}

// The frontier of a level as a queue.
__global__ void k_bfs_collect(const int32_t* __restrict__ depth, int64_t n, int32_t level, int32_t* __restrict__ q,
                              int32_t* __restrict__ nq) {
    const int lane = threadIdx.x & 31;
    for (int64_t v0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; v0 < n;
         v0 += (int64_t)gridDim.x * blockDim.x) {
        const bool in = v0 + lane < n && depth[v0 + lane] == level;
        const unsigned bal = __ballot_sync(kFull, in);
        if (!bal) continue;
        int32_t at = 0;
        if (lane == 0) at = atomicAdd(nq, __popc(bal));
        at = __shfl_sync(kFull, at, 0);
        if (in) q[at + __popc(bal & ((1u << lane) - 1u))] = (int32_t)(v0 + lane);
    }
}

// ---- connected components ----
// Union-find whose links always point to the smaller id, so a component's root
// is its smallest vertex.  Every vertex starts under its smallest neighbour
// (rows ascend) if that is smaller; then one pass over all entries joins what
// is still apart, most entries costing one read of their neighbour's parent.
// (Rounds of label hooking over all entries until nothing changed, a warp per
// row, took 3 x 1.7 ms on RMAT scale 20.)
//
// Searches read through L1: a stale parent is still an ancestor, and every
// search for the giant component's root at L2 would queue on its one sector (a
// sampling pass over 10^6 vertices took 0.96 ms so).  Only the larger root, the
// one to be linked, is checked at L2; the smaller may be linked to even if it is
// no root any more, as links point to smaller ids either way.
__device__ __forceinline__ int32_t cc_find(int32_t* parent, int32_t v) {
    int32_t p = parent[v];
    while (p != v) {
        const int32_t g = parent[p];
        if (g != p) parent[v] = g;   // halve the path; any ancestor is a valid parent
        v = p;
        p = g;
    }
    return v;
}

__device__ __forceinline__ void cc_union(int32_t* parent, int32_t a, int32_t b) {
    while (true) {
        a = cc_find(parent, a);
        b = cc_find(parent, b);
        if (a == b) return;
        if (a < b) {
            const int32_t t = a;
            a = b;
            b = t;
        }
        const int32_t p = __ldcg(&parent[a]);
        if (p != a) {
            a = p;   // linked meanwhile: smaller, so this ends
            continue;
        }
        const int32_t old = atomicCAS(&parent[a], a, b);
        if (old == a) return;
        a = old;
    }
}

__global__ void k_cc_init(const int64_t* __restrict__ rp, const int32_t* __restrict__ col, int64_t n,
                          int32_t* __restrict__ parent) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = rp[v];
        parent[v] = b < rp[v + 1] ? min((int32_t)v, col[b]) : (int32_t)v;
    }
}

// kFinal: every vertex ends under its root.  Its search then only reads: a
// halving store of a search that passed through v could land after v's own
// store and leave an ancestor that is not the root.
template <bool kFinal>
__global__ void k_cc_flatten(int64_t n, int32_t* parent) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        int32_t r = (int32_t)v;
        if (kFinal) {
            for (int32_t p = parent[r]; p != r; p = parent[r]) r = p;
        } else {
            r = cc_find(parent, r);
        }
        parent[v] = r;
    }
}

// Joins every step-th vertex with its second and its last neighbour: on graphs
// with a giant component nearly all of it is one tree before the pass over all
// entries.
__global__ void k_cc_sample(const int64_t* __restrict__ rp, const int32_t* __restrict__ col, int64_t n, int step,
                            int32_t* parent) {
    for (int64_t v = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) * step; v < n;
         v += (int64_t)gridDim.x * blockDim.x * step) {
        const int64_t b = rp[v], e = rp[v + 1];
        if (e - b < 2) continue;
        cc_union(parent, (int32_t)v, col[b + 1]);
        if (e - b > 2) cc_union(parent, (int32_t)v, col[e - 1]);
    }
}

// All entries, in chunks with their rows known: coalesced neighbour reads and
// eight pairs of parent reads a thread in flight.  The parents come through L1: a
// stale one is still an ancestor, and only sends its entry to the union.
__global__ void __launch_bounds__(kT)
k_cc_link(const int64_t* __restrict__ rp, const int32_t* __restrict__ col, int64_t n, int64_t nnz,
          const int32_t* __restrict__ chunk_row, const int32_t* __restrict__ chunk_last, int32_t* parent) {
    __shared__ int32_t srow[kEdgeChunkPadded], wmax[kT / 32];
    constexpr int kStep = 8;
    const int64_t chunks = (nnz + kEdgeChunk - 1) / kEdgeChunk;
    for (int64_t c = blockIdx.x; c < chunks; c += gridDim.x) {
        const int64_t e0 = c * kEdgeChunk, e1 = min(nnz, e0 + kEdgeChunk);
        const int len = (int)(e1 - e0);
        chunk_entry_rows<kT>(rp, n, chunk_row[c], e0, e1, srow, wmax, chunk_last[c]);
        for (int i0 = threadIdx.x; i0 < len; i0 += kStep * kT) {
            int32_t u[kStep], v[kStep], pu[kStep], pv[kStep];
#pragma unroll
            for (int k = 0; k < kStep; ++k) {
                const int i = i0 + k * kT;
                u[k] = i < len ? srow[chunk_pad(i)] : 0;
                v[k] = i < len ? col[e0 + i] : 0;
            }
#pragma unroll
            for (int k = 0; k < kStep; ++k) {
                pu[k] = parent[u[k]];
                pv[k] = parent[v[k]];
            }
#pragma unroll
            for (int k = 0; k < kStep; ++k)
                if (pu[k] != pv[k]) cc_union(parent, u[k], v[k]);
        }
        __syncthreads();
    }
}

// ---- DBG ----
__global__ void k_dbg_keys(const int64_t* __restrict__ rp, int64_t n, uint64_t avg, uint32_t* __restrict__ keys,
                           uint32_t* __restrict__ vals) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t d = (uint64_t)(rp[v + 1] - rp[v]);
        const uint64_t th[7] = {avg / 2, avg, avg * 2, avg * 4, avg * 8, avg * 16, avg * 32};
        int b = 7;
        for (int j = 0; j < 7; ++j)
            if (d <= th[j]) { b = j; break; }
        keys[v] = (uint32_t)(7 - b);  // highest bucket first
        vals[v] = (uint32_t)v;
    }
}

__global__ void k_scatter_rank(const uint32_t* __restrict__ order, int64_t n, int32_t* __restrict__ new_ids) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        new_ids[order[i]] = (int32_t)i;
}

float ev_ms(cudaEvent_t a, cudaEvent_t b) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    return ms;
}

}  // namespace

double pagerank_device(const DeviceCSR& g, int max_iters, double epsilon, float* score, int* iters_out,
                       cudaStream_t s) {
    const int64_t n = g.n;
    if (n == 0) return 0.0;
    constexpr int kBatch = 8;   // sweeps enqueued between two looks at the change
    const int64_t chunks = edge_chunks(g.nnz);
    DevBuf<float> contrib(2 * n, s), sums(2 * chunks, s);
    DevBuf<int32_t> rows(g.gaps ? n + 1 + 5 * chunks : 2 * chunks, s);
    DevBuf<double> err(kBatch, s);
    float *ca = contrib.get(), *cb = ca + n, *head = sums.get(), *tail = head + chunks;
    int32_t *tail_row = rows.get(), *id = g.gaps ? tail_row + 5 * chunks : nullptr;
    PrChunks chunk{tail_row + chunks, nullptr, nullptr, nullptr};
    cudaEvent_t e0, e1;
    GB_CUDA(cudaEventCreate(&e0));
    GB_CUDA(cudaEventCreate(&e1));
    GB_CUDA(cudaEventRecord(e0, s));
    const float init = 1.0f / (float)n, damp = 0.85f, base = (1.0f - damp) / (float)n;
    if (g.gaps) {
        // The scores and contributions lend their place to the rows' flags and positions.
        uint8_t* full = reinterpret_cast<uint8_t*>(score);
        int64_t* pos = reinterpret_cast<int64_t*>(contrib.get());
        chunk.last = chunk.first + chunks;
        chunk.first_place = chunk.last + chunks;
        chunk.last_place = chunk.first_place + chunks;
        k_pr_full<<<grid_for(n, kT), kT, 0, s>>>(g.row_ptr, n, full);
        GB_LAUNCH_CHECK();
        exclusive_scan_u8_to_i64(full, pos, n, nullptr, s);
        k_pr_rows<<<grid_for(n, kT), kT, 0, s>>>(g.row_ptr, n, g.nnz, pos, id, chunk);
        GB_LAUNCH_CHECK();
    } else {
        chunk_rows_device(g.row_ptr, n, g.nnz, chunk.first, s);
    }
    k_pr_init<<<grid_for(n, kT), kT, 0, s>>>(g.row_ptr, n, init, score, ca, cb);
    GB_LAUNCH_CHECK();
    PrArgs a{g.row_ptr, g.col, n,    g.nnz, id,   chunk.first, base, damp,   ca,
             cb,        score, head, tail,  tail_row, err,     epsilon};
    const int grid = grid_for(chunks, 1), join_grid = grid_for(chunks * 32, kT);
    int it = 0;
    for (bool done = false; it < max_iters && !done;) {
        const int count = std::min(kBatch, max_iters - it);
        GB_CUDA(cudaMemsetAsync(err, 0, kBatch * sizeof(double), s));
        for (int k = 0; k < count; ++k) {
            if (it + k == 0) k_pr_first<<<grid_for(n, kT), kT, 0, s>>>(a, chunk);
            if (chunks > 0) {
                k_pr_sweep<<<grid, kT, 0, s>>>(a, k);
                k_pr_join<<<join_grid, kT, 0, s>>>(a, k);
            }
            float* next = a.cout;
            a.cout = const_cast<float*>(a.cin);
            a.cin = next;
        }
        GB_LAUNCH_CHECK();
        double h[kBatch];
        GB_CUDA(cudaMemcpyAsync(h, err.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
        GB_CUDA(cudaStreamSynchronize(s));
        for (int k = 0; k < count && !done; ++k) {
            ++it;
            done = h[k] < epsilon;
        }
    }
    GB_CUDA(cudaEventRecord(e1, s));
    GB_CUDA(cudaEventSynchronize(e1));
    if (iters_out) *iters_out = it;
    const double ms = ev_ms(e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return ms;
}

double bfs_device(const DeviceCSR& g, int64_t source, int32_t* depth, cudaStream_t s) {
    const int64_t n = g.n;
    if (n == 0) return 0.0;
    GB_REQUIRE(source >= 0 && source < n, GBGPU_E_INVALID, "BFS source out of range");
    const int64_t words = ceil_div(n, 32);
    DevBuf<int32_t> qa(n, s), qb(n, s), hubs(g.nnz / kHubRow + 1, s);
    DevBuf<uint32_t> visited(words, s), front(words, s), next(words, s);
    DevBuf<BfsCtl> ctl(1, s);
    cudaEvent_t e0, e1;
    GB_CUDA(cudaEventCreate(&e0));
    GB_CUDA(cudaEventCreate(&e1));
    GB_CUDA(cudaEventRecord(e0, s));
    GB_CUDA(cudaMemsetAsync(depth, 0xFF, n * sizeof(int32_t), s));
    const int32_t zero = 0, src = (int32_t)source;
    GB_CUDA(cudaMemcpyAsync(depth + source, &zero, sizeof(int32_t), cudaMemcpyHostToDevice, s));
    GB_CUDA(cudaMemcpyAsync(qa.get(), &src, sizeof(int32_t), cudaMemcpyHostToDevice, s));
    BfsCtl c{1, 0, 0, 0};
    {
        int64_t h[2];
        GB_CUDA(cudaMemcpyAsync(h, g.row_ptr + source, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
        GB_CUDA(cudaStreamSynchronize(s));
        c.edges = (unsigned long long)(h[1] - h[0]);
    }
    auto put = [&] { GB_CUDA(cudaMemcpyAsync(ctl.get(), &c, sizeof(c), cudaMemcpyHostToDevice, s)); };
    auto get = [&] {
        GB_CUDA(cudaMemcpyAsync(&c, ctl.get(), sizeof(c), cudaMemcpyDeviceToHost, s));
        GB_CUDA(cudaStreamSynchronize(s));
    };
    const bool bits = n <= kBitsMax;
    const int small_q = bits ? kBitsQ : kPlainQ;
    const int small_smem = 2 * small_q * (int)sizeof(SmallEntry) + (bits ? (int)words * 4 : 0);
    GB_CUDA(cudaFuncSetAttribute(k_bfs_small<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 2 * kBitsQ * (int)sizeof(SmallEntry) + (int)(kBitsMax / 8)));
    GB_CUDA(cudaFuncSetAttribute(k_bfs_small<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 2 * kPlainQ * (int)sizeof(SmallEntry)));
    bool fresh = true;   // only the source is visited
    bool bottom_up = false;
    while (c.nf > 0) {
        const int32_t level = c.level;
        const int64_t nf = c.nf;
        // Beamer's heuristic: go bottom-up when the frontier's edges exceed
        // nnz / 14, back to top-down when the frontier is below n / 24.
        if (!bottom_up && c.edges > (unsigned long long)g.nnz / 14 && c.edges > (unsigned long long)kSmallEdges) {
            bottom_up = true;
            k_bfs_bits<<<grid_for(n, kT), kT, 0, s>>>(depth, n, level, visited, front);
            GB_LAUNCH_CHECK();
        } else if (bottom_up && nf < n / 24) {
            bottom_up = false;
            int32_t* nq = &ctl.get()->nhub;   // scratch counter of the rebuilt queue
            GB_CUDA(cudaMemsetAsync(nq, 0, sizeof(int32_t), s));
            k_bfs_collect<<<grid_for(n, kT), kT, 0, s>>>(depth, n, level, qa, nq);
            GB_LAUNCH_CHECK();
        }
        if (!bottom_up && nf <= small_q && c.edges <= (unsigned long long)kSmallEdges) {
            put();
            if (bits && !fresh) k_bfs_bits<<<grid_for(n, kT), kT, 0, s>>>(depth, n, level, visited, front);
            (bits ? k_bfs_small<true> : k_bfs_small<false>)<<<1, kSmallT, small_smem, s>>>(
                g.row_ptr, g.col, depth, qa, visited, words, fresh ? 1 : 0, ctl);
            GB_LAUNCH_CHECK();
            get();
            fresh = false;
            continue;
        }
        fresh = false;
        c = BfsCtl{0, level + 1, 0, 0};
        put();
        if (bottom_up) {
            k_bfs_bu<<<grid_for(n, kT), kT, 0, s>>>(g.row_ptr, g.col, n, depth, level, visited, front, next, ctl);
            GB_LAUNCH_CHECK();
            std::swap(front.ptr, next.ptr);
        } else {
            k_bfs_td<<<grid_for(nf * 32, kT), kT, 0, s>>>(g.row_ptr, g.col, qa, nf, depth, level, qb, hubs, ctl);
            GB_LAUNCH_CHECK();
            k_bfs_td_hub<<<kNumSMs * 8, kT, 0, s>>>(g.row_ptr, g.col, hubs, depth, level, qb, ctl);
            GB_LAUNCH_CHECK();
            std::swap(qa.ptr, qb.ptr);
        }
        get();
    }
    GB_CUDA(cudaEventRecord(e1, s));
    GB_CUDA(cudaEventSynchronize(e1));
    const double ms = ev_ms(e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return ms;
}

double cc_device(const DeviceCSR& g, int32_t* comp, cudaStream_t s) {
    const int64_t n = g.n;
    if (n == 0) return 0.0;
    cudaEvent_t e0, e1;
    GB_CUDA(cudaEventCreate(&e0));
    GB_CUDA(cudaEventCreate(&e1));
    GB_CUDA(cudaEventRecord(e0, s));
    k_cc_init<<<grid_for(n, kT), kT, 0, s>>>(g.row_ptr, g.col, n, comp);
    GB_LAUNCH_CHECK();
    k_cc_flatten<false><<<grid_for(n, kT), kT, 0, s>>>(n, comp);
    GB_LAUNCH_CHECK();
    if (g.nnz > 0) {
        // Every 32nd vertex first: the large trees meet with few threads asking
        // for the same roots (all vertices at once: 0.56 ms on RMAT scale 20).
        for (const int step : {32, 1}) {
            k_cc_sample<<<grid_for(ceil_div(n, step), kT), kT, 0, s>>>(g.row_ptr, g.col, n, step, comp);
            k_cc_flatten<false><<<grid_for(n, kT), kT, 0, s>>>(n, comp);
        }
        GB_LAUNCH_CHECK();
        const int64_t chunks = edge_chunks(g.nnz);
        DevBuf<int32_t> chunk_row(2 * chunks, s);
        int32_t* chunk_last = chunk_row.get() + chunks;
        chunk_rows_device(g.row_ptr, n, g.nnz, chunk_row, s, chunk_last);
        k_cc_link<<<grid_for(chunks, 1), kT, 0, s>>>(g.row_ptr, g.col, n, g.nnz, chunk_row, chunk_last, comp);
        GB_LAUNCH_CHECK();
    }
    k_cc_flatten<false><<<grid_for(n, kT), kT, 0, s>>>(n, comp);
    k_cc_flatten<true><<<grid_for(n, kT), kT, 0, s>>>(n, comp);
    GB_LAUNCH_CHECK();
    GB_CUDA(cudaEventRecord(e1, s));
    GB_CUDA(cudaEventSynchronize(e1));
    const double ms = ev_ms(e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return ms;
}

double dbg_mapping_device(const DeviceCSR& g, int32_t* new_ids, cudaStream_t s) {
    const int64_t n = g.n;
    if (n == 0) return 0.0;
    cudaEvent_t e0, e1;
    GB_CUDA(cudaEventCreate(&e0));
    GB_CUDA(cudaEventCreate(&e1));
    GB_CUDA(cudaEventRecord(e0, s));
    DevBuf<uint32_t> keys(n, s), vals(n, s);
    k_dbg_keys<<<grid_for(n, kT), kT, 0, s>>>(g.row_ptr, n, (uint64_t)(g.nnz / n), keys, vals);
    GB_LAUNCH_CHECK();
    radix_sort_pairs_u32(keys, vals, n, 3, s);
    k_scatter_rank<<<grid_for(n, kT), kT, 0, s>>>(vals, n, new_ids);
    GB_LAUNCH_CHECK();
    GB_CUDA(cudaEventRecord(e1, s));
    GB_CUDA(cudaEventSynchronize(e1));
    const double ms = ev_ms(e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return ms;
}

}  // namespace gb
