// primitives.cu -- scan, stable radix sort and fill kernels used by every stage.
//
// All of these are bandwidth-bound integer passes: tiles of 2,048 (scans, 256
// threads) or 4,096 elements (radix passes, 512 threads) per CTA, coalesced loads,
// shared-memory staging, grid sizes set by the element count; short scans and sorts
// by one CTA.
#include <algorithm>

#include "gb_chunks.cuh"
#include "gb_common.cuh"

namespace gb {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ int64_t warp_incl_scan(int64_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int64_t t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Exclusive scan across the CTA; returns this thread's exclusive prefix and
// writes the CTA total to *total.
__device__ __forceinline__ int64_t block_excl_scan(int64_t v, int64_t* total) {
    __shared__ int64_t warp_sums[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    int64_t incl = warp_incl_scan(v);
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int64_t w = lane < nwarps ? warp_sums[lane] : 0;
        int64_t wi = warp_incl_scan(w);
        if (lane < nwarps) warp_sums[lane] = wi - w;
        if (lane == nwarps - 1) warp_sums[31] = wi;
    }
    __syncthreads();
    int64_t res = warp_sums[warp] + incl - v;
    if (total) *total = warp_sums[31];
    __syncthreads();
    return res;
}

template <typename Tin>
__global__ void k_tile_reduce(const Tin* __restrict__ in, int64_t n, int64_t* __restrict__ partial) {
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    int64_t sum = 0;
    for (int i = threadIdx.x; i < kScanTile; i += kScanThreads) {
        const int64_t idx = base + i;
        if (idx < n) sum += (int64_t)in[idx];
    }
    int64_t total;
    block_excl_scan(sum, &total);
    if (threadIdx.x == 0) partial[blockIdx.x] = total;
}

template <typename Tin>
__global__ void k_tile_scan(const Tin* __restrict__ in, int64_t* __restrict__ out, int64_t n,
                            const int64_t* __restrict__ tile_offset, int64_t* __restrict__ total_out) {
    __shared__ int64_t s[kScanTile];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    for (int i = threadIdx.x; i < kScanTile; i += kScanThreads) {
        const int64_t idx = base + i;
        s[i] = idx < n ? (int64_t)in[idx] : 0;
    }
    __syncthreads();
    int64_t local[kScanItems];
    int64_t tsum = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        local[j] = s[threadIdx.x * kScanItems + j];
        tsum += local[j];
    }
    int64_t total;
    int64_t run = block_excl_scan(tsum, &total) + (tile_offset ? tile_offset[blockIdx.x] : 0);
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        s[threadIdx.x * kScanItems + j] = run;
        run += local[j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kScanTile; i += kScanThreads) {
        const int64_t idx = base + i;
        if (idx < n) out[idx] = s[i];
    }
    if (total_out && blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanThreads - 1) {
        *total_out = run;  // prefix of the last tile's end = grand total
    }
}

// Up to kScanOneMax values by one CTA, tile after tile with a running offset:
// one launch of 3 to 7 us where reduce, scan of the partials and scan are three
// launches of 4 us each and the gaps between them.  A tile's values are read
// before any of it is written, so out may alias in.
constexpr int kScanOneThreads = 512;   // block_excl_scan keeps a slot of its 32 for the total
constexpr int kScanOneItems = 16;
constexpr int kScanOneTile = kScanOneThreads * kScanOneItems;
constexpr int64_t kScanOneMax = 4 * kScanOneTile;

template <typename Tin>
__global__ void __launch_bounds__(kScanOneThreads)
k_scan_one(const Tin* __restrict__ in, int64_t* __restrict__ out, int64_t n, int64_t* __restrict__ total_out) {
    int64_t carry = 0;
    for (int64_t base = 0; base < n; base += kScanOneTile) {
        int64_t v[kScanOneItems], sum = 0;
#pragma unroll
        for (int j = 0; j < kScanOneItems; ++j) {
            const int64_t i = base + (int64_t)threadIdx.x * kScanOneItems + j;
            v[j] = i < n ? (int64_t)in[i] : 0;
            sum += v[j];
        }
        int64_t total;
        int64_t run = carry + block_excl_scan(sum, &total);
#pragma unroll
        for (int j = 0; j < kScanOneItems; ++j) {
            const int64_t i = base + (int64_t)threadIdx.x * kScanOneItems + j;
            if (i < n) out[i] = run;
            run += v[j];
        }
        carry += total;
    }
    if (total_out && threadIdx.x == 0) *total_out = carry;
}

// Returns its kernel launches.
template <typename Tin>
int exclusive_scan_impl(const Tin* in, int64_t* out, int64_t n, int64_t* total_dev, cudaStream_t s) {
    if (n <= 0) {
        if (total_dev) GB_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(int64_t), s));
        return 0;
    }
    const int64_t tiles = ceil_div(n, kScanTile);
    if (tiles == 1) {
        k_tile_scan<Tin><<<1, kScanThreads, 0, s>>>(in, out, n, nullptr, total_dev);
        GB_LAUNCH_CHECK();
        return 1;
    }
    if (n <= kScanOneMax) {
        k_scan_one<Tin><<<1, kScanOneThreads, 0, s>>>(in, out, n, total_dev);
        GB_LAUNCH_CHECK();
        return 1;
    }
    DevBuf<int64_t> partial(tiles, s);
    k_tile_reduce<Tin><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, partial);
    GB_LAUNCH_CHECK();
    const int partials = exclusive_scan_impl<int64_t>(partial, partial, tiles, nullptr, s);
    k_tile_scan<Tin><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, out, n, partial, total_dev);
    GB_LAUNCH_CHECK();
    return 2 + partials;
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort, 8-bit digits.
// Tile = 16 warps x 256 consecutive keys; each warp walks its 256 keys in 8
// steps of 32, ranking equal digits by a ballot multisplit, so ranks follow
// input order (stable).  The tile is put in digit order in shared memory first
// and written from there: a digit's 16 keys or so leave as one run, where each
// thread writing its own keys filled sectors piecemeal (230 M 64-bit keys: 4.2 ms
// a pass, 0.9 TB/s; this way 1.74 ms, 2.1 TB/s).
// ---------------------------------------------------------------------------
constexpr int kRadixThreads = 512;
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kRadixSteps = 8;
constexpr int kRadixPerWarp = 32 * kRadixSteps;
constexpr int kRadixTile = kRadixWarps * kRadixPerWarp;  // 4096

template <typename K>
__global__ void __launch_bounds__(kRadixThreads)
k_radix_hist(const K* __restrict__ keys, int64_t n, int shift, int64_t num_tiles, int32_t* __restrict__ hist) {
    __shared__ int32_t counts[256];
    if (threadIdx.x < 256) counts[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kRadixTile;
    K k[kRadixSteps];
#pragma unroll
    for (int j = 0; j < kRadixSteps; ++j) {
        const int64_t idx = base + j * kRadixThreads + threadIdx.x;
        k[j] = idx < n ? keys[idx] : 0;
    }
#pragma unroll
    for (int j = 0; j < kRadixSteps; ++j)
        if (base + j * kRadixThreads + threadIdx.x < n) atomicAdd(&counts[(unsigned)((k[j] >> shift) & 0xFF)], 1);
    __syncthreads();
    if (threadIdx.x < 256) hist[(int64_t)threadIdx.x * num_tiles + blockIdx.x] = counts[threadIdx.x];
}

template <typename K, bool kHasValues>
constexpr int radix_scatter_smem() {
    return kRadixTile * (int)(sizeof(K) + (kHasValues ? sizeof(uint32_t) : 0));
}

template <typename K, bool kHasValues>
__global__ void __launch_bounds__(kRadixThreads)
k_radix_scatter(const K* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                K* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int64_t n,
                int shift, int64_t num_tiles, const int64_t* __restrict__ offsets) {
    extern __shared__ __align__(16) unsigned char radix_smem[];
    K* skeys = reinterpret_cast<K*>(radix_smem);
    uint32_t* svals = reinterpret_cast<uint32_t*>(skeys + kRadixTile);
    __shared__ uint16_t wrun[kRadixWarps][258];
    __shared__ int64_t gbase[256];
    __shared__ int wsum[8];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int i = t; i < kRadixWarps * 258; i += kRadixThreads) (&wrun[0][0])[i] = 0;
    __syncthreads();
    const int64_t tile = (int64_t)blockIdx.x * kRadixTile, base = tile + (int64_t)warp * kRadixPerWarp;
    K k_reg[kRadixSteps];
    uint32_t v_reg[kRadixSteps];
    uint16_t d_reg[kRadixSteps], r_reg[kRadixSteps];
#pragma unroll
    for (int st = 0; st < kRadixSteps; ++st) {
        const int64_t idx = base + st * 32 + lane;
        k_reg[st] = idx < n ? keys_in[idx] : 0;
        v_reg[st] = kHasValues && idx < n ? vals_in[idx] : 0u;
    }
    const unsigned lt_mask = (1u << lane) - 1u;
#pragma unroll
    for (int st = 0; st < kRadixSteps; ++st) {
        const bool in = base + st * 32 + lane < n;
        const int d = in ? (int)((k_reg[st] >> shift) & 0xFF) : 256;
        unsigned peers = __ballot_sync(0xFFFFFFFFu, in);
        if (!in) peers = ~peers;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const bool bit = (d >> b) & 1;
            const unsigned bal = __ballot_sync(0xFFFFFFFFu, bit);
            peers &= bit ? bal : ~bal;
        }
        const int before = wrun[warp][d];
        __syncwarp();
        if (lane == __ffs(peers) - 1) wrun[warp][d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
        d_reg[st] = (uint16_t)d;
        r_reg[st] = (uint16_t)(before + __popc(peers & lt_mask));
    }
    __syncthreads();
    // Per digit: exclusive prefix over warps (warps cover consecutive keys),
    // then over the digits of the tile.
    int total = 0;
    if (t < 256) {
#pragma unroll
        for (int w = 0; w < kRadixWarps; ++w) {
            const int c = wrun[w][t];
            wrun[w][t] = (uint16_t)total;
            total += c;
        }
    }
    int incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += x;
    }
    if (t < 256 && lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (t < 256) {
        int first = incl - total;
        for (int w = 0; w < warp; ++w) first += wsum[w];
        gbase[t] = offsets[(int64_t)t * num_tiles + blockIdx.x] - first;
#pragma unroll
        for (int w = 0; w < kRadixWarps; ++w) wrun[w][t] = (uint16_t)(wrun[w][t] + first);
    }
    __syncthreads();
#pragma unroll
    for (int st = 0; st < kRadixSteps; ++st) {
        const int d = d_reg[st];
        if (d < 256) {
            const int at = wrun[warp][d] + r_reg[st];
            skeys[at] = k_reg[st];
            if (kHasValues) svals[at] = v_reg[st];
        }
    }
    __syncthreads();
    const int cnt = (int)min((int64_t)kRadixTile, n - tile);
    for (int i = t; i < cnt; i += kRadixThreads) {
        const K k = skeys[i];
        const int64_t pos = gbase[(unsigned)((k >> shift) & 0xFF)] + i;
        keys_out[pos] = k;
        if (kHasValues) vals_out[pos] = svals[i];
    }
}

// Up to kSmallSort pairs by one CTA: a bitonic sort in shared memory by (key,
// input position), so it is stable too.  One launch of a few microseconds where a
// radix sort takes three to five a pass and up to eight passes.
constexpr int kSmallSort = 4096;
constexpr int kSmallSortThreads = 1024;

template <typename K, bool kHasValues>
__global__ void __launch_bounds__(kSmallSortThreads)
k_sort_small(K* __restrict__ keys, uint32_t* __restrict__ values, int n, int padded, K mask) {
    extern __shared__ __align__(16) unsigned char sort_smem[];
    K* k = reinterpret_cast<K*>(sort_smem);
    uint16_t* at = reinterpret_cast<uint16_t*>(k + padded);
    for (int i = threadIdx.x; i < padded; i += blockDim.x) {
        k[i] = i < n ? keys[i] & mask : (K)~(K)0;   // the padding's positions are the largest, too
        at[i] = (uint16_t)i;
    }
    __syncthreads();
    for (int run = 2; run <= padded; run <<= 1) {
        for (int d = run >> 1; d > 0; d >>= 1) {
            for (int t = threadIdx.x; t < padded / 2; t += blockDim.x) {
                const int i = 2 * t - (t & (d - 1)), j = i + d;
                const K x = k[i], y = k[j];
                const uint16_t p = at[i], q = at[j];
                const bool after = x > y || (x == y && p > q);
                if (after == ((i & run) == 0)) {
                    k[i] = y;
                    k[j] = x;
                    at[i] = q;
                    at[j] = p;
                }
            }
            __syncthreads();
        }
    }
    // Keys and values as given, moved: every read before the first write.
    constexpr int kPer = kSmallSort / kSmallSortThreads;
    K kk[kPer];
    uint32_t vv[kPer];
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
        const int i = threadIdx.x + r * blockDim.x;
        if (i < n) {
            kk[r] = keys[at[i]];
            if (kHasValues) vv[r] = values[at[i]];
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
        const int i = threadIdx.x + r * blockDim.x;
        if (i < n) {
            keys[i] = kk[r];
            if (kHasValues) values[i] = vv[r];
        }
    }
}

template <typename K, bool kHasValues>
int radix_sort_impl(K* keys, uint32_t* values, int64_t n, int key_bits, cudaStream_t s) {
    if (n <= 1 || key_bits <= 0) return 0;
    const int passes = (key_bits + 7) / 8;
    if (n <= kSmallSort) {
        int padded = 2;
        while (padded < n) padded <<= 1;
        const K mask = 8 * passes >= (int)(8 * sizeof(K)) ? (K)~(K)0 : (((K)1 << (8 * passes)) - 1);
        const int smem = padded * (int)(sizeof(K) + sizeof(uint16_t));
        k_sort_small<K, kHasValues><<<1, std::min(kSmallSortThreads, std::max(32, padded / 2)), smem, s>>>(
            keys, values, (int)n, padded, mask);
        GB_LAUNCH_CHECK();
        return 1;
    }
    const int64_t tiles = ceil_div(n, kRadixTile);
    constexpr int smem = radix_scatter_smem<K, kHasValues>();
    if (smem > 24 * 1024)   // beside some 10 KB of static shared memory; the limit without it is 48 KB in all
        GB_CUDA(cudaFuncSetAttribute(k_radix_scatter<K, kHasValues>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    DevBuf<K> kbuf(n, s);
    DevBuf<uint32_t> vbuf(kHasValues ? n : 0, s);
    DevBuf<int32_t> hist(256 * tiles, s);
    DevBuf<int64_t> offs(256 * tiles, s);
    K* kin = keys;
    K* kout = kbuf.get();
    uint32_t* vin = values;
    uint32_t* vout = vbuf.get();
    int launches = 0;
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        k_radix_hist<K><<<(unsigned)tiles, kRadixThreads, 0, s>>>(kin, n, shift, tiles, hist);
        GB_LAUNCH_CHECK();
        launches += 2 + exclusive_scan_impl<int32_t>(hist, offs, 256 * tiles, nullptr, s);
        k_radix_scatter<K, kHasValues><<<(unsigned)tiles, kRadixThreads, smem, s>>>(
            kin, vin, kout, vout, n, shift, tiles, offs);
        GB_LAUNCH_CHECK();
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    if (kin != keys) {
        GB_CUDA(cudaMemcpyAsync(keys, kin, n * sizeof(K), cudaMemcpyDeviceToDevice, s));
        if (kHasValues)
            GB_CUDA(cudaMemcpyAsync(values, vin, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
    }
    return launches;
}

__global__ void k_fill_u32(uint32_t* p, uint32_t v, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = v;
}
__global__ void k_fill_i64(int64_t* p, int64_t v, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = v;
}
__global__ void k_iota_u32(uint32_t* p, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = (uint32_t)i;
}
__global__ void k_degrees(const int64_t* __restrict__ rp, int64_t* __restrict__ deg, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        deg[i] = rp[i + 1] - rp[i];
}

__global__ void k_chunk_rows(const int64_t* __restrict__ rp, int64_t n, int64_t nnz, int32_t* __restrict__ chunk_row,
                             int32_t* __restrict__ chunk_last) {
    const int lane = threadIdx.x & 31;
    for (int64_t u0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; u0 < n;
         u0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t u = u0 + lane;
        const int64_t b = u < n ? rp[u] : 0, e = u < n ? rp[u + 1] : 0;
        note_chunk_first(b, e, (int32_t)u, chunk_row, [] { return false; });
        if (chunk_last) note_chunk_last(b, e, (int32_t)u, nnz, chunk_last);
    }
}

}  // namespace

void chunk_rows_device(const int64_t* row_ptr, int64_t n, int64_t nnz, int32_t* chunk_row, cudaStream_t s,
                       int32_t* chunk_last) {
    if (n <= 0 || nnz <= 0) return;
    k_chunk_rows<<<grid_for(n, 256), 256, 0, s>>>(row_ptr, n, nnz, chunk_row, chunk_last);
    GB_LAUNCH_CHECK();
}

void exclusive_scan_i64(const int64_t* in, int64_t* out, int64_t n, cudaStream_t s) {
    exclusive_scan_impl<int64_t>(in, out, n, nullptr, s);
}

void exclusive_scan_i64_total(const int64_t* in, int64_t* out, int64_t n, int64_t* total_dev,
                              cudaStream_t s) {
    exclusive_scan_impl<int64_t>(in, out, n, total_dev, s);
}

void exclusive_scan_i32_to_i64(const int32_t* in, int64_t* out, int64_t n, int64_t* total_dev,
                               cudaStream_t s) {
    exclusive_scan_impl<int32_t>(in, out, n, total_dev, s);
}

void exclusive_scan_u8_to_i64(const uint8_t* in, int64_t* out, int64_t n, int64_t* total_dev, cudaStream_t s) {
    exclusive_scan_impl<uint8_t>(in, out, n, total_dev, s);
}

int radix_sort_pairs_u32(uint32_t* keys, uint32_t* values, int64_t n, int key_bits, cudaStream_t s) {
    return radix_sort_impl<uint32_t, true>(keys, values, n, key_bits, s);
}
int radix_sort_pairs_u64(uint64_t* keys, uint32_t* values, int64_t n, int key_bits, cudaStream_t s) {
    return radix_sort_impl<uint64_t, true>(keys, values, n, key_bits, s);
}
int radix_sort_keys_u64(uint64_t* keys, int64_t n, int key_bits, cudaStream_t s) {
    return radix_sort_impl<uint64_t, false>(keys, nullptr, n, key_bits, s);
}

void fill_u32(uint32_t* p, uint32_t v, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    k_fill_u32<<<grid_for(n, 256), 256, 0, s>>>(p, v, n);
    GB_LAUNCH_CHECK();
}
void fill_i64(int64_t* p, int64_t v, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    k_fill_i64<<<grid_for(n, 256), 256, 0, s>>>(p, v, n);
    GB_LAUNCH_CHECK();
}
void iota_u32(uint32_t* p, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    k_iota_u32<<<grid_for(n, 256), 256, 0, s>>>(p, n);
    GB_LAUNCH_CHECK();
}
void degrees_i64(const int64_t* row_ptr, int64_t* deg, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    k_degrees<<<grid_for(n, 256), 256, 0, s>>>(row_ptr, deg, n);
    GB_LAUNCH_CHECK();
}

}  // namespace gb
