// selector.cu -- Tier-0 graph features on the device and the learned selector's MLP.
//
// Tier-0 features follow ComputeTier0SampledGraphFeatures
// (bench/include/graphbrew/reorder/reorder_types.h:6066-6186): a strided
// sample of s = clamp(sqrt(n), 1024, 8192) vertices (vertex (2i+1)n/(2s)),
// sample mean degree and coefficient of variation (n-1 denominator, summed in
// sample order like the reference), hub concentration of the top 10% of the
// sample, packing factor of the hubs over 8-vertex property lines, normalised
// edge span and window-neighbour overlap over the sampled rows.  The degree
// statistics and hub terms are summed in the reference's order, so the inputs
// of the frozen rule are exact; the span sums use a tree order.
//
// The learned selector is a float32 MLP in -> 64 -> 64 -> 3 (ReLU) predicting
// log end-to-end times of the three arms (GraphBrew algorithm 12, DBG, original
// order).  Forward, backward (mean squared error) and Adam are hand-written
// kernels with a fixed summation order per output element.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "gb_common.cuh"
#include "gb_selector.h"

namespace gb {

namespace {

constexpr int kSampleMax = 8192;
constexpr int kSortThreads = 1024;

struct SampleEntry {
    long long deg;
    long long node;
};

__device__ __forceinline__ bool entry_before(const SampleEntry& a, const SampleEntry& b) {
    // degree descending, vertex id ascending; padding (deg < 0) last
    if (a.deg != b.deg) return a.deg > b.deg;
    return a.node < b.node;
}

__global__ void __launch_bounds__(kSortThreads)
k_tier0(const int64_t* __restrict__ rp, const int32_t* __restrict__ col, int64_t n, int64_t nnz, int s,
        double* __restrict__ out) {
    extern __shared__ unsigned char smem_raw[];
    SampleEntry* e = reinterpret_cast<SampleEntry*>(smem_raw);
    __shared__ double s_span[kSortThreads / 32];
    __shared__ unsigned long long s_edges[kSortThreads / 32], s_window[kSortThreads / 32];
    __shared__ double s_degsum, s_avg;
    int P = 1;
    while (P < s) P <<= 1;
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
        if (i < s) {
            const uint64_t node = ((2ull * (uint64_t)i + 1ull) * (uint64_t)n) / (2ull * (uint64_t)s);
            e[i].node = (long long)node;
            e[i].deg = (long long)(rp[node + 1] - rp[node]);
        } else {
            e[i].node = 0x7FFFFFFFFFFFFFFFll;
            e[i].deg = -1;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int i = 0; i < s; ++i) sum += (double)e[i].deg;
        const double avg = sum / s;
        double var = 0.0;
        for (int i = 0; i < s; ++i) {
            // explicit rounding: no fused multiply-add, as in the reference's sum
            const double d = __dsub_rn((double)e[i].deg, avg);
            var = __dadd_rn(var, __dmul_rn(d, d));
        }
        const double variance = s > 1 ? var / (s - 1) : 0.0;
        out[0] = (double)n;
        out[1] = (double)nnz;
        out[2] = avg;
        out[3] = avg > 0.0 ? sqrt(variance) / avg : 0.0;
        out[4] = n > 1 ? avg / (double)(n - 1) : 0.0;
        s_degsum = sum;
        s_avg = avg;
    }
    __syncthreads();
    // Bitonic sort of the padded sample.
    for (int k = 2; k <= P; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < P; i += blockDim.x) {
                const int ixj = i ^ j;
                if (ixj > i) {
                    const bool asc = (i & k) == 0;
                    const SampleEntry a = e[i], b = e[ixj];
                    const bool swap = asc ? entry_before(b, a) : entry_before(a, b);
                    if (swap) { e[i] = b; e[ixj] = a; }
                }
            }
            __syncthreads();
        }
    }
    const int hub_count = max(1, s / 10);
    if (threadIdx.x == 0) {
        double hub_sum = 0.0;
        for (int i = 0; i < hub_count; ++i) hub_sum += (double)e[i].deg;
        out[5] = s_degsum > 0.0 ? hub_sum / s_degsum : 0.0;
        // Hubs on distinct 8-vertex property lines (sizeof(double) = 8 bytes per vertex).
        int distinct = 0;
        for (int i = 0; i < hub_count; ++i) {
            const long long line = e[i].node / 8;
            bool seen = false;
            for (int j = 0; j < i && !seen; ++j) seen = (e[j].node / 8) == line;
            distinct += !seen;
        }
        out[6] = distinct ? (double)hub_count / distinct : 0.0;
    }
    // Span and window overlap over the sampled rows (warp per sampled vertex).
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double denom = (double)(n - 1 > 1 ? n - 1 : 1);
    double span = 0.0;
    unsigned long long edges = 0, window = 0;
    for (int i = w; i < s; i += blockDim.x / 32) {
        const long long node = e[i].node;
        const long long nline = node / 8;
        for (int64_t q = rp[node] + lane; q < rp[node + 1]; q += 32) {
            const long long dst = col[q];
            span += (double)llabs(dst - node) / denom;
            ++edges;
            window += llabs(dst / 8 - nline) <= 1;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        span += __shfl_xor_sync(0xFFFFFFFFu, span, o);
        edges += __shfl_xor_sync(0xFFFFFFFFu, edges, o);
        window += __shfl_xor_sync(0xFFFFFFFFu, window, o);
    }
    if (lane == 0) { s_span[w] = span; s_edges[w] = edges; s_window[w] = window; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double sp = 0.0;
        unsigned long long ed = 0, wi = 0;
        for (int i = 0; i < (int)(blockDim.x / 32); ++i) { sp += s_span[i]; ed += s_edges[i]; wi += s_window[i]; }
        out[7] = ed ? sp / (double)ed : 0.0;
        out[8] = ed ? (double)wi / (double)ed : 0.0;
    }
}

// ---- MLP ----
__global__ void k_dense_fwd(const float* __restrict__ X, const float* __restrict__ W, const float* __restrict__ b,
                            float* __restrict__ Y, int B, int I, int O, int relu) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= B * O) return;
    const int r = idx / O, o = idx % O;
    float acc = b[o];
    for (int i = 0; i < I; ++i) acc += X[r * I + i] * W[i * O + o];
    Y[idx] = relu ? fmaxf(acc, 0.f) : acc;
}

// dX[r,i] = sum_o dY[r,o] W[i,o], masked by the ReLU of the forward output X.
__global__ void k_dense_bwd_x(const float* __restrict__ dY, const float* __restrict__ W,
                              const float* __restrict__ Xfwd, float* __restrict__ dX, int B, int I, int O) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= B * I) return;
    const int r = idx / I, i = idx % I;
    float acc = 0.f;
    for (int o = 0; o < O; ++o) acc += dY[r * O + o] * W[i * O + o];
    dX[idx] = Xfwd[idx] > 0.f ? acc : 0.f;
}

// dW[i,o] = sum_r X[r,i] dY[r,o]; db[o] = sum_r dY[r,o].
__global__ void k_dense_bwd_w(const float* __restrict__ X, const float* __restrict__ dY, float* __restrict__ dW,
                              float* __restrict__ db, int B, int I, int O) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < I * O) {
        const int i = idx / O, o = idx % O;
        float acc = 0.f;
        for (int r = 0; r < B; ++r) acc += X[r * I + i] * dY[r * O + o];
        dW[idx] = acc;
    } else if (idx < I * O + O) {
        const int o = idx - I * O;
        float acc = 0.f;
        for (int r = 0; r < B; ++r) acc += dY[r * O + o];
        db[o] = acc;
    }
}

// Mean squared error over B x O outputs: dY = 2 (Y - T) / (B O); loss summed per row.
__global__ void k_mse(const float* __restrict__ Y, const float* __restrict__ T, float* __restrict__ dY,
                      float* __restrict__ row_loss, int B, int O) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= B) return;
    float l = 0.f;
    for (int o = 0; o < O; ++o) {
        const float d = Y[r * O + o] - T[r * O + o];
        dY[r * O + o] = 2.f * d / (float)(B * O);
        l += d * d;
    }
    row_loss[r] = l;
}

__device__ __forceinline__ void adam_step(float& p, float g, float& m, float& v, float lr, float b1, float b2,
                                          float eps, float c1, float c2) {
    // Contracted by name: the same rounding in every kernel that steps.
    m = fmaf(b1, m, (1.f - b1) * g);
    v = fmaf(b2, v, (1.f - b2) * g * g);
    p -= lr * (m / c1) / (sqrtf(v / c2) + eps);
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    adam_step(p[i], g[i], m[i], v[i], lr, b1, b2, eps, c1, c2);
}

__global__ void k_gather_rows(const float* __restrict__ src, const int32_t* __restrict__ idx, int rows, int cols,
                              float* __restrict__ dst) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= rows * cols) return;
    dst[t] = src[(int64_t)idx[t / cols] * cols + t % cols];
}

// ---------------------------------------------------------------------------
// One epoch of training in one launch.
//
// A minibatch of 128 rows is 1.9 M multiply-adds, so as a dozen launches with a
// copy back and a wait each it was all latency: 98 us a minibatch.  Here one
// cluster of eight CTAs runs the epoch's minibatches with two cluster barriers
// each: every CTA takes an eighth of the rows through the forward pass and the
// activations' gradients (weights in its shared memory), then owns a block of
// the weights: it fetches the activation columns that those need from the
// others through L2, forms their gradients and Adam steps with parameter and
// moments in registers, and leaves the new weights in L2 for all eight.  (Through
// distributed shared memory, element by element, the two exchanges were half of
// a minibatch's 14.5 us.)
//
// Every sum runs in the order of the kernels above (inputs, outputs or rows
// ascending, one fused multiply-add each), so the parameters are the same bit for
// bit: training amplifies a changed rounding some thousandfold.
// ---------------------------------------------------------------------------
constexpr int kTrCtas = 8;
constexpr int kTrThreads = 512;
constexpr int kTrMaxIn = 32;      // the single-output threads cover in * 8 + 67 outputs
constexpr int kTrMaxBatch = 256;  // activations and column copies in shared memory
constexpr int kTrW2Stride = kMlpHidden + 1;   // W2 is read along both axes

struct TrainArgs {
    float *params, *m, *v;    // 16-byte aligned
    float* act;               // a minibatch's activations and gradients, TrainExchange
    const float *X, *T;
    const int32_t* order;     // this epoch's rows
    const float2* corr;       // per minibatch: Adam's 1 - b1^t, 1 - b2^t
    float* row_loss;
    int n, in, batch;
    float lr, b1, b2, eps;
};

// Offsets (floats) into the exchange buffer: row-major, a row per minibatch row.
struct TrainExchange {
    int h1, h2, d2, d1, dy, x, total;
};

__host__ __device__ inline TrainExchange train_exchange(int in, int batch) {
    TrainExchange e;
    e.h1 = 0;
    e.h2 = e.h1 + batch * kMlpHidden;
    e.d2 = e.h2 + batch * kMlpHidden;
    e.d1 = e.d2 + batch * kMlpHidden;
    e.dy = e.d1 + batch * kMlpHidden;
    e.x = e.dy + batch * 4;
    e.total = e.x + batch * in;
    return e;
}

// Offsets (floats) into a CTA's shared memory.
struct TrainLayout {
    int w1, b1, w2, b2, w3, b3;             // weights
    int x, h1, h2, d2, d1, dy;              // this CTA's rows
    int cx, ch1, ch2, cd2, cd1, cdy;        // columns of all rows
    int one;                                // 1.0: the input of a bias
    int total;
};

__host__ __device__ inline TrainLayout train_layout(int in, int batch) {
    const int rows = (batch + kTrCtas - 1) / kTrCtas, all = rows * kTrCtas;
    TrainLayout l;
    int at = 0;
    auto take = [&](int floats) {
        const int here = at;
        at += (floats + 3) & ~3;
        return here;
    };
    l.w1 = take(in * kMlpHidden);
    l.b1 = take(kMlpHidden);
    l.w2 = take(kMlpHidden * kTrW2Stride);
    l.b2 = take(kMlpHidden);
    l.w3 = take(kMlpHidden * kMlpOut);
    l.b3 = take(kMlpOut);
    l.x = take(rows * in);
    l.h1 = take(rows * kMlpHidden);
    l.h2 = take(rows * kMlpHidden);
    l.d2 = take(rows * kMlpHidden);
    l.d1 = take(rows * kMlpHidden);
    l.dy = take(rows * 4);
    l.cx = take(all * in);
    l.ch1 = take(all * 16);
    l.ch2 = take(all * 8);
    l.cd2 = take(all * 32);
    l.cd1 = take(all * 8);
    l.cdy = take(all * 4);
    l.one = take(1);
    l.total = at;
    return l;
}

__global__ void __cluster_dims__(kTrCtas, 1, 1) __launch_bounds__(kTrThreads) k_mlp_epoch(TrainArgs a) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) float sm[];
    constexpr int H = kMlpHidden, O = kMlpOut;
    const int t = threadIdx.x, rank = (int)cluster.block_rank(), in = a.in;
    const TrainLayout L = train_layout(in, a.batch);
    const TrainExchange E = train_exchange(in, a.batch);
    const int gw1 = 0, gb1 = in * H, gw2 = gb1 + H, gb2 = gw2 + H * H, gw3 = gb2 + H, gb3 = gw3 + H * O;
    // Packed parameters -> shared memory (read at L2: other CTAs write them).
    auto load_weights = [&]() {
        for (int i = 4 * t; i < gb3; i += 4 * kTrThreads) {   // every part but the last is a multiple of 4
            const float4 w = __ldcg(reinterpret_cast<const float4*>(a.params + i));
            const bool in_w2 = i >= gw2 && i < gb2;
            const int at = in_w2 ? L.w2 + (i - gw2) / H * kTrW2Stride + (i - gw2) % H
                           : i < gb1 ? L.w1 + i : i < gw2 ? L.b1 + i - gb1 : i < gw3 ? L.b2 + i - gb2 : L.w3 + i - gw3;
            sm[at] = w.x;
            sm[at + 1] = w.y;
            sm[at + 2] = w.z;
            sm[at + 3] = w.w;
        }
        if (t < O) sm[L.b3 + t] = __ldcg(a.params + gb3 + t);
    };
    load_weights();
    if (t == 0) sm[L.one] = 1.f;
    // Parameters that this thread owns: the first 128 threads a 1 x 4 piece of
    // the CTA's 16 x 32 block of W2, each other thread one of the rest.
    const int bi = (rank >> 1) * 16, bo = (rank & 1) * 32;
    const int wi = t >> 3, wo = (t & 7) * 4;
    const int q = t - 128;
    int own = 0, pg = 0;                    // how many, packed index
    int ax = L.one, as = 0, bx = 0, bs = 0; // its gradient: sum over rows of sm[ax + r as] sm[bx + r bs]
    if (q < 0) {
        own = 4;
        pg = gw2 + (bi + wi) * H + bo + wo;
    } else if (q < in * 8) {
        own = 1, pg = gw1 + (q >> 3) * H + rank * 8 + (q & 7);
        ax = L.cx + (q >> 3), as = in, bx = L.cd1 + (q & 7), bs = 8;
    } else if (q < in * 8 + 8) {
        const int j = q - in * 8;
        own = 1, pg = gb1 + rank * 8 + j;
        bx = L.cd1 + j, bs = 8;
    } else if (q < in * 8 + 32) {
        const int j = q - in * 8 - 8;
        own = 1, pg = gw3 + (rank * 8 + j / O) * O + j % O;
        ax = L.ch2 + j / O, as = 8, bx = L.cdy + j % O, bs = 4;
    } else if (q < in * 8 + 64 && rank < 2) {   // bo = rank * 32 for these
        const int j = q - in * 8 - 32;
        own = 1, pg = gb2 + bo + j;
        bx = L.cd2 + j, bs = 32;
    } else if (q >= in * 8 + 64 && q < in * 8 + 64 + O && rank == 0) {
        const int j = q - in * 8 - 64;
        own = 1, pg = gb3 + j;
        bx = L.cdy + j, bs = 4;
    }
    float p[4], m[4], v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        p[k] = m[k] = v[k] = 0.f;
        if (k < own) {
            p[k] = a.params[pg + k];
            m[k] = a.m[pg + k];
            v[k] = a.v[pg + k];
        }
    }
    const int o = t & (H - 1), rg = t >> 6;   // column and row group of the row phase
    // A minibatch's inputs and this thread's target are read a minibatch ahead:
    // the row number and the row are two round trips.
    constexpr int kXPer = kTrMaxBatch / kTrCtas * kTrMaxIn / kTrThreads;
    float nx[kXPer], ntarget = 0.f;
    auto read_ahead = [&](int b0) {
        const int B = min(a.batch, a.n - b0), R = (B + kTrCtas - 1) / kTrCtas;
        const int r0 = rank * R, rows = max(0, min(R, B - r0));
#pragma unroll
        for (int k = 0; k < kXPer; ++k) {
            const int i = t + k * kTrThreads;
            nx[k] = i < rows * in ? a.X[(int64_t)a.order[b0 + r0 + i / in] * in + i % in] : 0.f;
        }
        if (t < rows * 4 && (t & 3) < O) ntarget = a.T[(int64_t)a.order[b0 + r0 + (t >> 2)] * O + (t & 3)];
    };
    read_ahead(0);
    for (int b0 = 0, step = 0; b0 < a.n; b0 += a.batch, ++step) {
        const int B = min(a.batch, a.n - b0), R = (B + kTrCtas - 1) / kTrCtas;
        const int r0 = rank * R, rows = max(0, min(R, B - r0));
        const float2 corr = a.corr[step];
        const float target = ntarget;
#pragma unroll
        for (int k = 0; k < kXPer; ++k) {
            const int i = t + k * kTrThreads;
            if (i < rows * in) sm[L.x + i] = nx[k];
        }
        __syncthreads();
        // ---- this CTA's rows: forward (rows rg, rg + 8, ..., two at a time) ----
        for (int r = rg; r < rows; r += 16) {
            const int r2 = r + 8 < rows ? r + 8 : r;
            float x = sm[L.b1 + o], y = x;
            for (int i = 0; i < in; ++i) {
                const float w = sm[L.w1 + i * H + o];
                x = fmaf(sm[L.x + r * in + i], w, x);
                y = fmaf(sm[L.x + r2 * in + i], w, y);
            }
            sm[L.h1 + r * H + o] = fmaxf(x, 0.f);
            sm[L.h1 + r2 * H + o] = fmaxf(y, 0.f);
        }
        __syncthreads();
        for (int r = rg; r < rows; r += 16) {
            const int r2 = r + 8 < rows ? r + 8 : r;
            float x = sm[L.b2 + o], y = x;
#pragma unroll 4
            for (int i = 0; i < H; i += 4) {
                const float4 f = *reinterpret_cast<const float4*>(&sm[L.h1 + r * H + i]);
                const float4 g = *reinterpret_cast<const float4*>(&sm[L.h1 + r2 * H + i]);
                const float w0 = sm[L.w2 + i * kTrW2Stride + o], w1 = sm[L.w2 + (i + 1) * kTrW2Stride + o];
                const float w2 = sm[L.w2 + (i + 2) * kTrW2Stride + o], w3 = sm[L.w2 + (i + 3) * kTrW2Stride + o];
                x = fmaf(f.w, w3, fmaf(f.z, w2, fmaf(f.y, w1, fmaf(f.x, w0, x))));
                y = fmaf(g.w, w3, fmaf(g.z, w2, fmaf(g.y, w1, fmaf(g.x, w0, y))));
            }
            sm[L.h2 + r * H + o] = fmaxf(x, 0.f);
            sm[L.h2 + r2 * H + o] = fmaxf(y, 0.f);
        }
        __syncthreads();
        // Outputs: four threads a row, three of them with an output; the mean
        // squared error's gradient and the row's loss.  The shuffles' lanes are named
        // before any of them part.
        const unsigned mask = __ballot_sync(0xFFFFFFFFu, t < rows * 4);
        if (t < rows * 4) {
            const int r = t >> 2, c = t & 3;
            const int cc = c < O ? c : 0;
            float y = sm[L.b3 + cc];
#pragma unroll 8
            for (int i = 0; i < H; ++i) y = fmaf(sm[L.h2 + r * H + i], sm[L.w3 + i * O + cc], y);
            const float d = y - target;
            if (c < O) sm[L.dy + r * 4 + c] = 2.f * d / (float)(B * O);
            const int q0 = (t & 31) & ~3;
            const float d0 = __shfl_sync(mask, d, q0), d1 = __shfl_sync(mask, d, q0 + 1),
                        d2 = __shfl_sync(mask, d, q0 + 2);
            if (c == 0) a.row_loss[b0 + r0 + r] = fmaf(d2, d2, fmaf(d1, d1, fmaf(d0, d0, 0.f)));
        }
        __syncthreads();
        // Gradients of the activations.
        for (int r = rg; r < rows; r += 8) {
            float x = 0.f;
#pragma unroll
            for (int c = 0; c < O; ++c) x = fmaf(sm[L.dy + r * 4 + c], sm[L.w3 + o * O + c], x);
            sm[L.d2 + r * H + o] = sm[L.h2 + r * H + o] > 0.f ? x : 0.f;
        }
        __syncthreads();
        for (int r = rg; r < rows; r += 16) {
            const int r2 = r + 8 < rows ? r + 8 : r;
            float x = 0.f, y = 0.f;
#pragma unroll 4
            for (int c = 0; c < H; c += 4) {
                const float4 f = *reinterpret_cast<const float4*>(&sm[L.d2 + r * H + c]);
                const float4 g = *reinterpret_cast<const float4*>(&sm[L.d2 + r2 * H + c]);
                const float* w = &sm[L.w2 + o * kTrW2Stride + c];
                x = fmaf(f.w, w[3], fmaf(f.z, w[2], fmaf(f.y, w[1], fmaf(f.x, w[0], x))));
                y = fmaf(g.w, w[3], fmaf(g.z, w[2], fmaf(g.y, w[1], fmaf(g.x, w[0], y))));
            }
            sm[L.d1 + r * H + o] = sm[L.h1 + r * H + o] > 0.f ? x : 0.f;
            sm[L.d1 + r2 * H + o] = sm[L.h1 + r2 * H + o] > 0.f ? y : 0.f;
        }
        // This CTA's rows to the exchange.
        __syncthreads();
        for (int i = t; i < rows * (H / 4); i += kTrThreads) {
            const int at = (r0 * H) / 4 + i;
            reinterpret_cast<float4*>(a.act + E.h1)[at] = reinterpret_cast<const float4*>(&sm[L.h1])[i];
            reinterpret_cast<float4*>(a.act + E.h2)[at] = reinterpret_cast<const float4*>(&sm[L.h2])[i];
            reinterpret_cast<float4*>(a.act + E.d2)[at] = reinterpret_cast<const float4*>(&sm[L.d2])[i];
            reinterpret_cast<float4*>(a.act + E.d1)[at] = reinterpret_cast<const float4*>(&sm[L.d1])[i];
        }
        for (int i = t; i < rows * 4; i += kTrThreads) a.act[E.dy + r0 * 4 + i] = sm[L.dy + i];
        for (int i = t; i < rows * in; i += kTrThreads) a.act[E.x + r0 * in + i] = sm[L.x + i];
        cluster.sync();
        // ---- columns of all rows that this CTA's parameters need ----
        auto fetch = [&](int from, int stride, int col, int to, auto width) {   // float4s a row
            constexpr int kW = decltype(width)::value;
            for (int i = t; i < B * kW; i += kTrThreads)
                reinterpret_cast<float4*>(&sm[to])[i] = __ldcg(
                    reinterpret_cast<const float4*>(a.act + from + (i / kW) * stride + col + 4 * (i % kW)));
        };
        fetch(E.h1, H, bi, L.ch1, std::integral_constant<int, 4>{});
        fetch(E.d2, H, bo, L.cd2, std::integral_constant<int, 8>{});
        fetch(E.h2, H, rank * 8, L.ch2, std::integral_constant<int, 2>{});
        fetch(E.d1, H, rank * 8, L.cd1, std::integral_constant<int, 2>{});
        fetch(E.dy, 4, 0, L.cdy, std::integral_constant<int, 1>{});
        for (int i = t; i < B * in; i += kTrThreads) sm[L.cx + i] = __ldcg(a.act + E.x + i);
        if (b0 + a.batch < a.n) read_ahead(b0 + a.batch);
        __syncthreads();
        // ---- gradients, rows ascending ----
        float g[4] = {0.f, 0.f, 0.f, 0.f};
        if (q < 0) {
#pragma unroll 8
            for (int r = 0; r < B; ++r) {
                const float h = sm[L.ch1 + r * 16 + wi];
                const float4 d = *reinterpret_cast<const float4*>(&sm[L.cd2 + r * 32 + wo]);
                g[0] = fmaf(h, d.x, g[0]);
                g[1] = fmaf(h, d.y, g[1]);
                g[2] = fmaf(h, d.z, g[2]);
                g[3] = fmaf(h, d.w, g[3]);
            }
        } else if (own) {
            // A bias multiplies by 1: the product and so the sum are exact copies.
#pragma unroll 8
            for (int r = 0; r < B; ++r) g[0] = fmaf(sm[ax + r * as], sm[bx + r * bs], g[0]);
        }
        // ---- Adam, and the new weights into every CTA's copy ----
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < own) adam_step(p[k], g[k], m[k], v[k], a.lr, a.b1, a.b2, a.eps, corr.x, corr.y);
        if (own == 4) *reinterpret_cast<float4*>(a.params + pg) = make_float4(p[0], p[1], p[2], p[3]);
        else if (own) a.params[pg] = p[0];
        cluster.sync();
        load_weights();   // the next minibatch's barrier follows its inputs
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (k < own) {
            a.m[pg + k] = m[k];
            a.v[pg + k] = v[k];
        }
}

inline int blocks(int64_t work) { return (int)((work + 255) / 256); }

}  // namespace

void tier0_features_device(const DeviceCSR& g, double* out9_host, cudaStream_t s) {
    const int64_t n = g.n;
    if (n == 0) {
        for (int i = 0; i < 9; ++i) out9_host[i] = 0.0;
        return;
    }
    int sample = (int)std::max<int64_t>(1024, std::min<int64_t>((int64_t)std::sqrt((double)n), kSampleMax));
    sample = (int)std::min<int64_t>(sample, n);
    int P = 1;
    while (P < sample) P <<= 1;
    const int smem = P * (int)sizeof(SampleEntry);
    GB_CUDA(cudaFuncSetAttribute(k_tier0, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    DevBuf<double> out(9, s);
    k_tier0<<<1, kSortThreads, smem, s>>>(g.row_ptr, g.col, n, g.nnz, sample, out);
    GB_LAUNCH_CHECK();
    GB_CUDA(cudaMemcpyAsync(out9_host, out.get(), 9 * sizeof(double), cudaMemcpyDeviceToHost, s));
    GB_CUDA(cudaStreamSynchronize(s));
}

int mlp_param_count(int in_dim) {
    return in_dim * kMlpHidden + kMlpHidden + kMlpHidden * kMlpHidden + kMlpHidden + kMlpHidden * kMlpOut + kMlpOut;
}

namespace {
struct MlpView {
    const float *W1, *b1, *W2, *b2, *W3, *b3;
};
MlpView view(const float* p, int in) {
    MlpView v;
    v.W1 = p;
    v.b1 = v.W1 + in * kMlpHidden;
    v.W2 = v.b1 + kMlpHidden;
    v.b2 = v.W2 + kMlpHidden * kMlpHidden;
    v.W3 = v.b2 + kMlpHidden;
    v.b3 = v.W3 + kMlpHidden * kMlpOut;
    return v;
}
}  // namespace

void mlp_forward_device(const float* params, const float* X, int B, int in, float* Y, float* H1, float* H2,
                        cudaStream_t s) {
    const MlpView v = view(params, in);
    k_dense_fwd<<<blocks((int64_t)B * kMlpHidden), 256, 0, s>>>(X, v.W1, v.b1, H1, B, in, kMlpHidden, 1);
    k_dense_fwd<<<blocks((int64_t)B * kMlpHidden), 256, 0, s>>>(H1, v.W2, v.b2, H2, B, kMlpHidden, kMlpHidden, 1);
    k_dense_fwd<<<blocks((int64_t)B * kMlpOut), 256, 0, s>>>(H2, v.W3, v.b3, Y, B, kMlpHidden, kMlpOut, 0);
    GB_LAUNCH_CHECK();
}

float mlp_grad_device(const float* params, const float* X, const float* T, int B, int in, float* grad,
                      cudaStream_t s) {
    DevBuf<float> H1((int64_t)B * kMlpHidden, s), H2((int64_t)B * kMlpHidden, s), Y((int64_t)B * kMlpOut, s),
        dY((int64_t)B * kMlpOut, s), dH2((int64_t)B * kMlpHidden, s), dH1((int64_t)B * kMlpHidden, s),
        row_loss(B, s);
    mlp_forward_device(params, X, B, in, Y, H1, H2, s);
    k_mse<<<blocks(B), 256, 0, s>>>(Y, T, dY, row_loss, B, kMlpOut);
    const MlpView v = view(params, in);
    float* gW1 = grad;
    float* gb1 = gW1 + in * kMlpHidden;
    float* gW2 = gb1 + kMlpHidden;
    float* gb2 = gW2 + kMlpHidden * kMlpHidden;
    float* gW3 = gb2 + kMlpHidden;
    float* gb3 = gW3 + kMlpHidden * kMlpOut;
    k_dense_bwd_w<<<blocks((int64_t)kMlpHidden * kMlpOut + kMlpOut), 256, 0, s>>>(H2, dY, gW3, gb3, B, kMlpHidden,
                                                                                  kMlpOut);
    k_dense_bwd_x<<<blocks((int64_t)B * kMlpHidden), 256, 0, s>>>(dY, v.W3, H2, dH2, B, kMlpHidden, kMlpOut);
    k_dense_bwd_w<<<blocks((int64_t)kMlpHidden * kMlpHidden + kMlpHidden), 256, 0, s>>>(H1, dH2, gW2, gb2, B,
                                                                                        kMlpHidden, kMlpHidden);
    k_dense_bwd_x<<<blocks((int64_t)B * kMlpHidden), 256, 0, s>>>(dH2, v.W2, H1, dH1, B, kMlpHidden, kMlpHidden);
    k_dense_bwd_w<<<blocks((int64_t)in * kMlpHidden + kMlpHidden), 256, 0, s>>>(X, dH1, gW1, gb1, B, in,
                                                                                kMlpHidden);
    GB_LAUNCH_CHECK();
    std::vector<float> rl(B);
    GB_CUDA(cudaMemcpyAsync(rl.data(), row_loss.get(), B * sizeof(float), cudaMemcpyDeviceToHost, s));
    GB_CUDA(cudaStreamSynchronize(s));
    double tot = 0.0;
    for (float x : rl) tot += x;
    return (float)(tot / ((double)B * kMlpOut));
}

float mlp_train_device(float* params, const float* X, const float* T, int n, int in, int epochs, int batch,
                       float lr, uint64_t seed, cudaStream_t s) {
    const int P = mlp_param_count(in);
    DevBuf<float> grad(P, s), m(P, s), v(P, s), Xb((int64_t)batch * in, s), Tb((int64_t)batch * kMlpOut, s);
    DevBuf<int32_t> idx(batch, s);
    GB_CUDA(cudaMemsetAsync(m, 0, P * sizeof(float), s));
    GB_CUDA(cudaMemsetAsync(v, 0, P * sizeof(float), s));
    std::vector<int32_t> order(n);
    for (int i = 0; i < n; ++i) order[i] = i;
    uint64_t state = seed ^ 0x9E3779B97F4A7C15ull;
    auto next = [&]() {
        state += 0x9E3779B97F4A7C15ull;
        uint64_t z = state;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    };
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    int t = 0;
    float last = 0.f;
    // Minibatches and inputs that the fused kernel's shared memory holds take
    // one launch an epoch (the next epoch is shuffled meanwhile).
    if (in <= kTrMaxIn && batch <= kTrMaxBatch) {
        const int nb = (int)ceil_div(n, batch), smem = train_layout(in, batch).total * (int)sizeof(float);
        GB_CUDA(cudaFuncSetAttribute(k_mlp_epoch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     train_layout(kTrMaxIn, kTrMaxBatch).total * (int)sizeof(float)));
        DevBuf<int32_t> rows(n, s);
        DevBuf<float2> corr(nb, s);
        DevBuf<float> row_loss(n, s), act(train_exchange(in, batch).total, s), own_params(P, s);
        GB_CUDA(cudaMemcpyAsync(own_params, params, P * sizeof(float), cudaMemcpyDeviceToDevice, s));
        // Two staging copies, reused once their transfer is over.
        struct Stage {
            std::vector<int32_t> rows;
            std::vector<float2> corr;
            cudaEvent_t done = nullptr;
            ~Stage() {
                if (done) cudaEventDestroy(done);
            }
        } stage[2];
        for (Stage& st : stage) {
            st.corr.resize(nb);
            GB_CUDA(cudaEventCreateWithFlags(&st.done, cudaEventDisableTiming));
        }
        for (int ep = 0; ep < epochs; ++ep) {
            Stage& st = stage[ep & 1];
            for (int i = n - 1; i > 0; --i) std::swap(order[i], order[next() % (uint64_t)(i + 1)]);
            GB_CUDA(cudaEventSynchronize(st.done));
            st.rows = order;
            for (float2& c : st.corr) {
                ++t;
                c = make_float2(1.f - std::pow(b1, (float)t), 1.f - std::pow(b2, (float)t));
            }
            GB_CUDA(cudaMemcpyAsync(rows, st.rows.data(), n * sizeof(int32_t), cudaMemcpyHostToDevice, s));
            GB_CUDA(cudaMemcpyAsync(corr, st.corr.data(), nb * sizeof(float2), cudaMemcpyHostToDevice, s));
            GB_CUDA(cudaEventRecord(st.done, s));
            k_mlp_epoch<<<kTrCtas, kTrThreads, smem, s>>>(
                TrainArgs{own_params, m, v, act, X, T, rows, corr, row_loss, n, in, batch, lr, b1, b2, eps});
            GB_LAUNCH_CHECK();
        }
        GB_CUDA(cudaMemcpyAsync(params, own_params, P * sizeof(float), cudaMemcpyDeviceToDevice, s));
        if (epochs > 0) {
            std::vector<float> rl(n);
            GB_CUDA(cudaMemcpyAsync(rl.data(), row_loss.get(), n * sizeof(float), cudaMemcpyDeviceToHost, s));
            GB_CUDA(cudaStreamSynchronize(s));
            double ep_loss = 0.0;
            for (int b0 = 0; b0 < n; b0 += batch) {
                const int B = std::min(batch, n - b0);
                double tot = 0.0;
                for (int r = 0; r < B; ++r) tot += rl[b0 + r];
                ep_loss += (float)(tot / ((double)B * kMlpOut));
            }
            last = (float)(ep_loss / std::max(1, nb));
        }
        GB_CUDA(cudaStreamSynchronize(s));
        return last;
    }
    for (int ep = 0; ep < epochs; ++ep) {
        for (int i = n - 1; i > 0; --i) std::swap(order[i], order[next() % (uint64_t)(i + 1)]);
        double ep_loss = 0.0;
        int nb = 0;
        for (int b0 = 0; b0 < n; b0 += batch) {
            const int B = std::min(batch, n - b0);
            GB_CUDA(cudaMemcpyAsync(idx.get(), order.data() + b0, B * sizeof(int32_t), cudaMemcpyHostToDevice, s));
            k_gather_rows<<<blocks((int64_t)B * in), 256, 0, s>>>(X, idx, B, in, Xb);
            k_gather_rows<<<blocks((int64_t)B * kMlpOut), 256, 0, s>>>(T, idx, B, kMlpOut, Tb);
            ep_loss += mlp_grad_device(params, Xb, Tb, B, in, grad, s);
            ++nb;
            ++t;
            const float c1 = 1.f - std::pow(b1, (float)t), c2 = 1.f - std::pow(b2, (float)t);
            k_adam<<<blocks(P), 256, 0, s>>>(params, grad, m, v, P, lr, b1, b2, eps, c1, c2);
            GB_LAUNCH_CHECK();
        }
        last = (float)(ep_loss / std::max(1, nb));
    }
    GB_CUDA(cudaStreamSynchronize(s));
    return last;
}

}  // namespace gb
