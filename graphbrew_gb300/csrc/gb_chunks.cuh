// gb_chunks.cuh -- entry-parallel sweeps over a CSR graph.
//
// A sweep splits the nnz adjacency entries into chunks of kEdgeChunk
// consecutive entries, one chunk per CTA iteration.  chunk_rows_device fills
// chunk_row[c] = the row holding entry c * kEdgeChunk (one thread per row,
// no search).  Inside the CTA, chunk_entry_rows expands that into the row of
// every entry of the chunk: the rows that start inside the chunk are
// scattered to their start offsets in shared memory and a prefix maximum
// fills the gaps.  Entries are then read in coalesced order with their row
// known, whatever the degree distribution: no warp idles on a short row and
// no long row serialises one warp.
#pragma once

#include "gb_common.cuh"

namespace gb {

constexpr int kEdgeChunk = 4096;
// One padding word per 32 entries keeps the per-thread runs of the prefix
// scan off a single bank.
constexpr int kEdgeChunkPadded = kEdgeChunk + kEdgeChunk / 32;

__device__ __forceinline__ int chunk_pad(int i) { return i + (i >> 5); }

// chunk_row has ceil(nnz / kEdgeChunk) entries, and so has chunk_last where it is
// given: the row that holds the chunk's last entry.  The CSR must be valid
// (row_ptr non-decreasing from 0 to nnz).
void chunk_rows_device(const int64_t* row_ptr, int64_t n, int64_t nnz, int32_t* chunk_row, cudaStream_t s,
                       int32_t* chunk_last = nullptr);

inline int64_t edge_chunks(int64_t nnz) { return ceil_div(nnz, kEdgeChunk); }

// fn(c, u) for the chunks c of [c0, c1), this lane's row u being what is noted in
// them (c0 >= c1: nothing).  More than kOwn of them are the whole warp's work, whose
// lanes all call; they are left out once stop() holds.
template <typename Fn, typename Stop>
__device__ __forceinline__ void for_chunks(int64_t c0, int64_t c1, int32_t u, Fn&& fn, Stop&& stop) {
    constexpr int kOwn = 64;   // some 0.3 us of stores; the question of stop() alone is a read of L2
    const int lane = threadIdx.x & 31;
    unsigned longer = __ballot_sync(0xFFFFFFFFu, c1 - c0 > kOwn);
    if (c1 - c0 <= kOwn)
        for (int64_t c = c0; c < c1; ++c) fn(c, u);
    while (longer && !__any_sync(0xFFFFFFFFu, stop())) {
        const int src = __ffs(longer) - 1;
        longer &= longer - 1;
        const int64_t end = __shfl_sync(0xFFFFFFFFu, c1, src);
        const int32_t row = __shfl_sync(0xFFFFFFFFu, u, src);
        for (int64_t c = __shfl_sync(0xFFFFFFFFu, c0, src) + lane; c < end; c += 32) fn(c, row);
    }
}

// first[c] = u for the chunks whose first entry is in [b, e), the entries of this
// lane's row u (b == e: none); last[c] likewise for the last entry.
template <typename Stop>
__device__ __forceinline__ void note_chunk_first(int64_t b, int64_t e, int32_t u, int32_t* first, Stop&& stop) {
    const uint64_t up = kEdgeChunk - 1;
    for_chunks((int64_t)(((uint64_t)b + up) / kEdgeChunk), (int64_t)(((uint64_t)e + up) / kEdgeChunk), u,
               [&](int64_t c, int32_t row) { first[c] = row; }, stop);
}

__device__ __forceinline__ void note_chunk_last(int64_t b, int64_t e, int32_t u, int64_t nnz, int32_t* last) {
    const uint64_t up = b < e && e == nnz ? kEdgeChunk - 1 : 0;   // the last chunk may be a short one
    for_chunks((int64_t)((uint64_t)b / kEdgeChunk), (int64_t)(((uint64_t)e + up) / kEdgeChunk), u,
               [&](int64_t c, int32_t row) { last[c] = row; }, [] { return false; });
}

// Rows that a CTA walks between a chunk's first and last.  Where there are more,
// nearly all of them empty, every entry's row is searched for instead: some 0.1 ms,
// which is what a walk over 64 K rows takes (4 M isolated ids in one chunk: 3.1 ms).
constexpr int64_t kChunkWalk = 65536;

// srow[chunk_pad(i)] = the largest row of [u0, last] that begins at or before e0 + i.
template <int kThreads>
__device__ __forceinline__ void chunk_search_rows(const int64_t* __restrict__ rp, int32_t u0, int32_t last, int64_t e0,
                                                  int64_t e1, int32_t* srow) {
    constexpr int kStep = 4;   // searches of a thread in flight
    const int len = (int)(e1 - e0);
    int64_t top = 1;
    while (top <= last - u0) top <<= 1;
    for (int i0 = threadIdx.x; i0 < len; i0 += kStep * kThreads) {
        int64_t u[kStep];
#pragma unroll
        for (int k = 0; k < kStep; ++k) u[k] = u0;
        for (int64_t half = top >> 1; half > 0; half >>= 1) {
#pragma unroll
            for (int k = 0; k < kStep; ++k) {
                const int64_t at = u[k] + half;
                if (at <= last && rp[at] <= e0 + i0 + k * kThreads) u[k] = at;
            }
        }
#pragma unroll
        for (int k = 0; k < kStep; ++k)
            if (i0 + k * kThreads < len) srow[chunk_pad(i0 + k * kThreads)] = (int32_t)u[k];
    }
    __syncthreads();
}

// srow (kEdgeChunkPadded ints of shared memory) receives, at chunk_pad(i),
// the row of entry e0 + i for i < e1 - e0.  warp_max: kThreads / 32 ints of
// shared memory; last: the row of entry e1 - 1, where it is known.  Every thread
// of the CTA calls it; it ends with a barrier.
template <int kThreads>
__device__ __forceinline__ void chunk_entry_rows(const int64_t* __restrict__ rp, int64_t n, int32_t u0,
                                                 int64_t e0, int64_t e1, int32_t* srow, int32_t* warp_max,
                                                 int32_t last = -1) {
    static_assert(kEdgeChunk % kThreads == 0 && kThreads % 32 == 0, "chunk / CTA shape");
    if (last - u0 > kChunkWalk) {
        chunk_search_rows<kThreads>(rp, u0, last, e0, e1, srow);
        return;
    }
    constexpr int kPer = kEdgeChunk / kThreads;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int i = t; i < kEdgeChunk; i += kThreads) srow[chunk_pad(i)] = -1;
    __syncthreads();
    if (t == 0) srow[0] = u0;
    // Rows after u0 begin strictly after e0; empty rows share their start
    // with the next non-empty row, which has the larger id.
    for (int64_t u = (int64_t)u0 + 1 + t; u < n; u += kThreads) {
        const int64_t r = rp[u];
        if (r >= e1) break;
        atomicMax(&srow[chunk_pad((int)(r - e0))], (int32_t)u);
    }
    __syncthreads();
    int m = -1;
#pragma unroll
    for (int k = 0; k < kPer; ++k) m = max(m, srow[chunk_pad(t * kPer + k)]);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xFFFFFFFFu, m, o);
        if (lane >= o) m = max(m, x);
    }
    if (lane == 31) warp_max[warp] = m;
    __syncthreads();
    int run = __shfl_up_sync(0xFFFFFFFFu, m, 1);
    if (lane == 0) run = -1;
    for (int w = 0; w < warp; ++w) run = max(run, warp_max[w]);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int p = chunk_pad(t * kPer + k);
        run = max(run, srow[p]);
        srow[p] = run;
    }
    __syncthreads();
}

}  // namespace gb
