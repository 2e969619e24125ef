// GroupNorm + ReLU over (batch, channels, particles) feature tensors, forward and backward.
//
// The reference's network blocks apply torch.nn.GroupNorm followed by ReLU to every convolution
// output (apr_models/apr_models/unet/unet_parts.py:18-26), with one group per channel by default.  On a
// (B, C, N) tensor with N in the tens of millions that is B*G rows of C/G*N elements; the stock
// kernels reduce one row per thread block, so a handful of blocks walk gigabytes serially.  Here the
// statistics are a two-stage reduction (many blocks per row, double-precision partial sums, fixed
// order: deterministic), normalisation and ReLU are one fused pass, and the backward pass is one
// reduction pass plus one elementwise pass; the ReLU mask is recomputed from the input instead of
// being stored.  Same arithmetic as torch: biased variance, eps inside the square root, statistics
// over the whole (padded) particle axis.
#include "apr_device.cuh"
#include <cuda_bf16.h>
#include <algorithm>

namespace {

typedef long long ll;
constexpr int GN_TPB = 256;
constexpr int GN_MAX_CHUNKS = 512;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// block-wide sum of two doubles; result valid in thread 0
__device__ __forceinline__ void block_sum2(double& a, double& b) {
    __shared__ double sa[GN_TPB / 32], sb[GN_TPB / 32];
    a = warp_sum(a); b = warp_sum(b);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { sa[w] = a; sb[w] = b; }
    __syncthreads();
    if (w == 0) {
        a = l < GN_TPB / 32 ? sa[l] : 0.0;
        b = l < GN_TPB / 32 ? sb[l] : 0.0;
        a = warp_sum(a); b = warp_sum(b);
    }
    __syncthreads();
}

// Entries of a batch item that hold values.  AllEntries: the whole row; ItemEntries: the first n[item] of them, behind which the row counts as zeros that are
// not read (the particles of an item among those of the largest one of its batch; inference over four images of 0.3 to 1.8 M particles: statistics 1.93 -> 1.37, apply
// 3.34 -> 3.03 ms, and 0.9 ms of zeros that need not be written).
struct AllEntries { __device__ __forceinline__ ll of(ll, ll n) const { return n; } };
constexpr int GN_ITEMS = 64;
struct ItemEntries { ll n[GN_ITEMS]; __device__ __forceinline__ ll of(ll item, ll) const { return n[item]; } };

// stage 1 of the statistics: partial[row][chunk] = (sum x, sum x^2) over the chunk
template<typename T, typename Entries>
__global__ void __launch_bounds__(GN_TPB) gn_partial_stats_kernel(const T* __restrict__ x, ll n, ll chunk_len, double* __restrict__ partial, int nchunks, int C,
                                                                  const __grid_constant__ Entries entries) {
    const ll row = blockIdx.y;
    const ll b0 = (ll) blockIdx.x * chunk_len, b1 = min(entries.of(row / C, n), b0 + chunk_len);
    const T* xr = x + row * n;
    double s = 0.0, ss = 0.0;
    ll i = b0 + threadIdx.x;
    for (; i + 3 * GN_TPB < b1; i += 4 * GN_TPB) {        // four independent loads in flight; same summation order
        T v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = xr[i + u * GN_TPB];
#pragma unroll
        for (int u = 0; u < 4; ++u) { const double d = (double) v[u]; s += d; ss += d * d; }
    }
    for (; i < b1; i += GN_TPB) { const double v = (double) xr[i]; s += v; ss += v * v; }
    block_sum2(s, ss);
    if (threadIdx.x == 0) { partial[(row * nchunks + blockIdx.x) * 2] = s; partial[(row * nchunks + blockIdx.x) * 2 + 1] = ss; }
}

// Sums of `count` pairs in ascending order, by a block: the pairs come into shared memory together, then thread 0 adds the first and thread 1 the second values.
// (A thread that added them from memory took 16 us for 37 pairs, now 4.)
constexpr int GN_SUM_TPB = 64, GN_SUM_PAIRS = 128;
__device__ __forceinline__ double sum_pairs(const double* __restrict__ pairs, int count, double* buf) {
    double acc = 0.0;
    for (int i0 = 0; i0 < count; i0 += GN_SUM_PAIRS) {
        const int n = min(GN_SUM_PAIRS, count - i0);
        for (int i = threadIdx.x; i < 2 * n; i += GN_SUM_TPB) buf[i] = pairs[2 * i0 + i];
        __syncthreads();
        if (threadIdx.x < 2) for (int i = 0; i < n; ++i) acc += buf[2 * i + threadIdx.x];
        __syncthreads();
    }
    return acc;
}

// stage 2, a block per (batch item, group): mean and 1/sqrt(var + eps)
template<typename T>
__global__ void __launch_bounds__(GN_SUM_TPB) gn_finalize_stats_kernel(const double* __restrict__ partial, int nchunks, int rows_per_group, ll n,
                                                                       double eps, T* __restrict__ mean, T* __restrict__ rstd) {
    __shared__ double buf[2 * GN_SUM_PAIRS];
    const int g = blockIdx.x;
    const double s = sum_pairs(partial + (ll) g * rows_per_group * nchunks * 2, rows_per_group * nchunks, buf);
    if (threadIdx.x >= 32) return;
    const double ss = __shfl_sync(0xffffffffu, s, 1);
    if (threadIdx.x > 0) return;
    const double m = (double) rows_per_group * (double) n;
    const double mu = s / m;
    const double var = fmax(ss / m - mu * mu, 0.0);
    mean[g] = (T) mu;
    rstd[g] = (T) (1.0 / sqrt(var + eps));
}

// Sums of the first stage, ascending (the order of gn_finalize_stats_kernel / gn_backward_rows_kernel): short rows have so few chunks
// that every block of the apply kernels adds them by itself and the kernels in between are not launched.
constexpr int GN_FUSE = 32;             // chunks of a group at most
__device__ __forceinline__ void sum_chunks(const double* __restrict__ partial, int count, double* buf, double& a, double& b) {
    for (int i = threadIdx.x; i < 2 * count; i += GN_TPB) buf[i] = partial[i];
    __syncthreads();
    a = 0.0; b = 0.0;
    for (int i = 0; i < count; ++i) { a += buf[2 * i]; b += buf[2 * i + 1]; }
}

// The apply kernels walk their row in tiles of GN_TILE entries, shifted so that a warp's stores cover whole 128-byte lines of the
// output (rows start at any element); four loads are in flight per thread and tensor.
constexpr int GN_UNROLL = 4, GN_TILE = GN_UNROLL * GN_TPB;
template<typename T> __device__ __forceinline__ ll first_of(const T* row) {
    return (ll) blockIdx.x * GN_TILE + threadIdx.x - (ll) ((reinterpret_cast<uintptr_t>(row) & 127) / sizeof(T));
}
// all threads of the block have all entries of the tile: no condition per access then (forward in a batch of four 3.43 -> 3.34 ms)
__device__ __forceinline__ bool whole_tile(ll i0, ll n) { const ll b = i0 - threadIdx.x; return b >= 0 && b + GN_TILE <= n; }
// Their blocks per row: four waves over the chip, so that a block's statistics (sums of the partials, a division and a square root in double
// precision, about 1 us) are spread over many tiles, but at least two tiles.  With 2048 entries per block whatever the row, the forward kernel took 4.92 ms
// in a batch of four tensors of 1.8 M locations (2.5 times the statistics, which read what it reads and writes), now 3.43; on one of 3.5 M locations
// forward 2.08 -> 1.82 and backward 2.89 -> 2.50 ms.
inline int apply_blocks(ll n, ll rows) {
    return (int) std::max<ll>(1, std::min<ll>((n + 127) / (2 * GN_TILE) + 1, (148ll * 8 * 4 + rows - 1) / rows));
}

// partial (null: mean / rstd are given): [row][nchunks][2] of the first stage; the first block of a group's first row stores its statistics
// y = max((x - mean) * rstd * gamma + beta, 0)
template<typename T, typename Entries>
__global__ void __launch_bounds__(GN_TPB) gn_relu_apply_kernel(const T* __restrict__ x, ll n, int C, int ch_per_group, const T* __restrict__ gamma,
                                                               const T* __restrict__ beta, T* mean, T* rstd, const double* __restrict__ partial,
                                                               int nchunks, double eps, T* __restrict__ y, int relu, const __grid_constant__ Entries entries) {
    __shared__ double buf[2 * GN_FUSE];
    const ll row = blockIdx.y;                       // b * C + c
    const int c = (int) (row % C);
    const ll g = row / ch_per_group;                 // (b * C + c) / ch_per_group = b * G + c / ch_per_group
    T mu, rs;
    if (partial) {
        double s, ss;
        sum_chunks(partial + g * ch_per_group * nchunks * 2, ch_per_group * nchunks, buf, s, ss);
        const double m = (double) ch_per_group * (double) n;
        const double mud = s / m, var = fmax(ss / m - mud * mud, 0.0);
        mu = (T) mud; rs = (T) (1.0 / sqrt(var + eps));
        if (blockIdx.x == 0 && threadIdx.x == 0 && row % ch_per_group == 0) { mean[g] = mu; rstd[g] = rs; }
    } else { mu = mean[g]; rs = rstd[g]; }
    const T ga = gamma ? gamma[c] : T(1), be = beta ? beta[c] : T(0);
    const T* xr = x + row * n;
    T* yr = y + row * n;
    const ll nv = entries.of(row / C, n);
    for (ll i0 = first_of(yr); i0 < n; i0 += (ll) gridDim.x * GN_TILE) {
        T v[GN_UNROLL];
        if (whole_tile(i0, nv)) {
#pragma unroll
            for (int u = 0; u < GN_UNROLL; ++u) v[u] = xr[i0 + u * GN_TPB];
#pragma unroll
            for (int u = 0; u < GN_UNROLL; ++u) {
                const T r = (v[u] - mu) * rs * ga + be;
                yr[i0 + u * GN_TPB] = (relu && r < T(0)) ? T(0) : r;
            }
            continue;
        }
#pragma unroll
        for (int u = 0; u < GN_UNROLL; ++u) { const ll i = i0 + u * GN_TPB; v[u] = i >= 0 && i < nv ? xr[i] : T(0); }
#pragma unroll
        for (int u = 0; u < GN_UNROLL; ++u) {
            const ll i = i0 + u * GN_TPB;
            if (i < 0 || i >= n) continue;
            const T r = (v[u] - mu) * rs * ga + be;        // same expression as the backward pass uses for the ReLU mask
            yr[i] = (relu && r < T(0)) ? T(0) : r;
        }
    }
}

// backward stage 1: partial[row][chunk] = (sum dy_eff, sum dy_eff * xhat), dy_eff = dy * [y > 0]
template<typename T>
__global__ void __launch_bounds__(GN_TPB) gn_backward_partial_kernel(const T* __restrict__ x, const T* __restrict__ dy, ll n, ll chunk_len, int C,
                                                                     int ch_per_group, const T* __restrict__ gamma, const T* __restrict__ beta,
                                                                     const T* __restrict__ mean, const T* __restrict__ rstd,
                                                                     double* __restrict__ partial, int nchunks, int relu) {
    const ll row = blockIdx.y;
    const int c = (int) (row % C);
    const ll g = row / ch_per_group;
    const T mu = mean[g], rs = rstd[g];
    const T ga = gamma ? gamma[c] : T(1), be = beta ? beta[c] : T(0);
    const ll b0 = (ll) blockIdx.x * chunk_len, b1 = min(n, b0 + chunk_len);
    const T* xr = x + row * n;
    const T* dr = dy + row * n;
    double s = 0.0, sx = 0.0;
    auto add = [&](T xv, T d) {
        const T xh = (xv - mu) * rs;
        if (relu && xh * ga + be <= T(0)) d = T(0);
        s += (double) d; sx += (double) d * (double) xh;
    };
    ll i = b0 + threadIdx.x;
    for (; i + 3 * GN_TPB < b1; i += 4 * GN_TPB) {        // eight independent loads in flight; same summation order
        T xv[4], dv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) { xv[u] = xr[i + u * GN_TPB]; dv[u] = dr[i + u * GN_TPB]; }
#pragma unroll
        for (int u = 0; u < 4; ++u) add(xv[u], dv[u]);
    }
    for (; i < b1; i += GN_TPB) add(xr[i], dr[i]);
    block_sum2(s, sx);
    if (threadIdx.x == 0) { partial[(row * nchunks + blockIdx.x) * 2] = s; partial[(row * nchunks + blockIdx.x) * 2 + 1] = sx; }
}

// backward stage 2a, a block per row: A = sum dy_eff, Bx = sum dy_eff * xhat  (row_sums[row] = (A, Bx))
__global__ void __launch_bounds__(GN_SUM_TPB) gn_backward_rows_kernel(const double* __restrict__ partial, int nchunks, double* __restrict__ row_sums) {
    __shared__ double buf[2 * GN_SUM_PAIRS];
    const double v = sum_pairs(partial + (ll) blockIdx.x * nchunks * 2, nchunks, buf);
    if (threadIdx.x < 2) row_sums[(ll) blockIdx.x * 2 + threadIdx.x] = v;
}

// backward stage 2b: dgamma[c] = sum_b Bx, dbeta[c] = sum_b A; group terms mA, mB per (b, g)
template<typename T>
__global__ void gn_backward_finalize_kernel(const double* __restrict__ row_sums, int B, int C, int ch_per_group, ll n, const T* __restrict__ gamma,
                                            T* __restrict__ dgamma, T* __restrict__ dbeta, T* __restrict__ group_terms) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int G = C / ch_per_group;
    if (i < C) {
        double a = 0.0, b = 0.0;
        for (int bb = 0; bb < B; ++bb) { a += row_sums[((ll) bb * C + i) * 2]; b += row_sums[((ll) bb * C + i) * 2 + 1]; }
        if (dbeta) dbeta[i] = (T) a;
        if (dgamma) dgamma[i] = (T) b;
    }
    if (i < B * G) {
        const int bb = i / G, g = i % G;
        double a = 0.0, b = 0.0;
        for (int k = 0; k < ch_per_group; ++k) {
            const int c = g * ch_per_group + k;
            const double ga = gamma ? (double) gamma[c] : 1.0;
            a += ga * row_sums[((ll) bb * C + c) * 2]; b += ga * row_sums[((ll) bb * C + c) * 2 + 1];
        }
        const double m = (double) ch_per_group * (double) n;
        group_terms[2 * i] = (T) (a / m); group_terms[2 * i + 1] = (T) (b / m);
    }
}

// backward stage 3: dx = rstd * (dy_eff * gamma - mA - xhat * mB).  partial (null: group_terms are given): sums of stage 1 of ONE batch item;
// every block adds those of its group as stages 2a and 2b do, the first block of a row stores its dgamma and dbeta
template<typename T>
__global__ void __launch_bounds__(GN_TPB) gn_backward_apply_kernel(const T* __restrict__ x, const T* __restrict__ dy, ll n, int C, int ch_per_group,
                                                                   const T* __restrict__ gamma, const T* __restrict__ beta, const T* __restrict__ mean,
                                                                   const T* __restrict__ rstd, const T* __restrict__ group_terms, const double* __restrict__ partial,
                                                                   int nchunks, T* __restrict__ dgamma, T* __restrict__ dbeta, T* __restrict__ dx, int relu) {
    __shared__ double buf[2 * GN_FUSE];
    const ll row = blockIdx.y;
    const int c = (int) (row % C);
    const ll g = row / ch_per_group;
    const T mu = mean[g], rs = rstd[g];
    const T ga = gamma ? gamma[c] : T(1), be = beta ? beta[c] : T(0);
    T mA, mB;
    if (partial) {
        const int count = ch_per_group * nchunks;
        const double* p = partial + g * count * 2;
        for (int i = threadIdx.x; i < 2 * count; i += GN_TPB) buf[i] = p[i];
        __syncthreads();
        double a = 0.0, b = 0.0;
        for (int k = 0; k < ch_per_group; ++k) {
            double ra = 0.0, rb = 0.0;
            for (int i = k * nchunks; i < (k + 1) * nchunks; ++i) { ra += buf[2 * i]; rb += buf[2 * i + 1]; }
            const int ck = (int) (g * ch_per_group) + k;
            const double gk = gamma ? (double) gamma[ck] : 1.0;
            a += gk * ra; b += gk * rb;
            if (ck == c && blockIdx.x == 0 && threadIdx.x == 0) { if (dbeta) dbeta[c] = (T) ra; if (dgamma) dgamma[c] = (T) rb; }
        }
        const double m = (double) ch_per_group * (double) n;
        mA = (T) (a / m); mB = (T) (b / m);
    } else { mA = group_terms[2 * g]; mB = group_terms[2 * g + 1]; }
    const T* xr = x + row * n;
    const T* dr = dy + row * n;
    T* o = dx + row * n;
    for (ll i0 = first_of(o); i0 < n; i0 += (ll) gridDim.x * GN_TILE) {
        T xv[GN_UNROLL], dv[GN_UNROLL];
        if (whole_tile(i0, n)) {
#pragma unroll
            for (int u = 0; u < GN_UNROLL; ++u) { xv[u] = xr[i0 + u * GN_TPB]; dv[u] = dr[i0 + u * GN_TPB]; }
#pragma unroll
            for (int u = 0; u < GN_UNROLL; ++u) {
                const T xh = (xv[u] - mu) * rs;
                T d = dv[u];
                if (relu && xh * ga + be <= T(0)) d = T(0);
                o[i0 + u * GN_TPB] = rs * (d * ga - mA - xh * mB);
            }
            continue;
        }
#pragma unroll
        for (int u = 0; u < GN_UNROLL; ++u) { const ll i = i0 + u * GN_TPB; if (i >= 0 && i < n) { xv[u] = xr[i]; dv[u] = dr[i]; } }
#pragma unroll
        for (int u = 0; u < GN_UNROLL; ++u) {
            const ll i = i0 + u * GN_TPB;
            if (i < 0 || i >= n) continue;
            const T xh = (xv[u] - mu) * rs;
            T d = dv[u];
            if (relu && xh * ga + be <= T(0)) d = T(0);
            o[i] = rs * (d * ga - mA - xh * mB);
        }
    }
}

// Stage 3 for a convolution in front of the normalisation whose backward pass works from packed bf16 rows of its output's gradient: the same
// dx, rounded and written as rows [0, n_rows) of cpad channels, row n_rows zero, instead of a channel-major tensor that would be read once
// more to be packed (12 + 6 bytes per value; here 10: 2.1 + 1.35 ms in two passes where one now takes 2.00).  One batch item; a block has 32 channels x 128 entries at a time.
// A block walks its tiles, the next one's loads in flight while a tile is stored: with a tile per block nothing of another was under way between its loads and its
// stores, and each block added up its partial sums for one tile: the 13 layers of a
// training step on 3.5 M locations 2.28 ms, now 2.00 (8C + 2C bytes per row at 0.87 of the copy rate).
constexpr int GN_ROWS_BLOCKS = 4;       // blocks per SM
__global__ void __launch_bounds__(256, GN_ROWS_BLOCKS) gn_backward_apply_rows_kernel(const float* __restrict__ x, const float* __restrict__ dy, ll n, ll n_rows, int C, int ch_per_group,
                                                                     const float* __restrict__ gamma, const float* __restrict__ beta, const float* __restrict__ mean,
                                                                     const float* __restrict__ rstd, const float* __restrict__ group_terms, const double* __restrict__ partial,
                                                                     int nchunks, float* __restrict__ dgamma, float* __restrict__ dbeta, int relu, int cpad,
                                                                     __nv_bfloat16* __restrict__ out) {
    __shared__ float tile[2][32][129], par[32][6];         // par: mean, rstd, gamma, beta, mA, mB
    const int c0 = blockIdx.y * 32, lane = threadIdx.x & 31, wrp = __shfl_sync(0xffffffffu, (int) threadIdx.x >> 5, 0);
    if (threadIdx.x < 32 && c0 + (int) threadIdx.x < C) {
        const int c = c0 + threadIdx.x, g = c / ch_per_group;
        float mA, mB;
        if (partial) {                                     // sums of stage 1, as gn_backward_apply_kernel adds them
            double a = 0.0, b = 0.0;
            for (int k = 0; k < ch_per_group; ++k) {
                const int ck = g * ch_per_group + k;
                double ra = 0.0, rb = 0.0;
                for (int i = 0; i < nchunks; ++i) { ra += partial[((ll) ck * nchunks + i) * 2]; rb += partial[((ll) ck * nchunks + i) * 2 + 1]; }
                const double gk = gamma ? (double) gamma[ck] : 1.0;
                a += gk * ra; b += gk * rb;
                if (ck == c && blockIdx.x == 0) { dbeta[c] = (float) ra; dgamma[c] = (float) rb; }
            }
            const double m = (double) ch_per_group * (double) n;
            mA = (float) (a / m); mB = (float) (b / m);
        } else { mA = group_terms[2 * g]; mB = group_terms[2 * g + 1]; }
        float* p = par[threadIdx.x];
        p[0] = mean[g]; p[1] = rstd[g]; p[2] = gamma ? gamma[c] : 1.f; p[3] = beta ? beta[c] : 0.f; p[4] = mA; p[5] = mB;
    }
    const ll tiles = n_rows / 128 + 1;                     // with the row of zeros
    float xv[4][4], dv[4][4];
    auto request = [&](ll r0) {
        if (r0 + 128 <= n_rows) {                          // one condition per channel, the same for a warp
            const ll at = (ll) (c0 + wrp) * n + r0 + lane;
#pragma unroll
            for (int cc = 0; cc < 4; ++cc)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const bool in = c0 + wrp + 8 * cc < C;
                    xv[cc][k] = in ? x[at + 8 * cc * n + 32 * k] : 0.f; dv[cc][k] = in ? dy[at + 8 * cc * n + 32 * k] : 0.f;
                }
            return;
        }
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
            const int ch = c0 + wrp + 8 * cc;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const ll r = r0 + lane + 32 * k;
                const bool in = ch < C && r < n_rows;
                xv[cc][k] = in ? x[(ll) ch * n + r] : 0.f;
                dv[cc][k] = in ? dy[(ll) ch * n + r] : 0.f;
            }
        }
    };
    request((ll) blockIdx.x * 128);
    __syncthreads();                                       // par
    int buf = 0;
    for (ll t = blockIdx.x; t < tiles; t += gridDim.x, buf ^= 1) {
        const ll r0 = t * 128;
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
            const int ch = wrp + 8 * cc;
            const float mu = par[ch][0], rs = par[ch][1], ga = par[ch][2], be = par[ch][3], mA = par[ch][4], mB = par[ch][5];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float xh = (xv[cc][k] - mu) * rs;
                float d = dv[cc][k];
                if (relu && xh * ga + be <= 0.f) d = 0.f;
                tile[buf][ch][lane + 32 * k] = c0 + ch < C && r0 + lane + 32 * k < n_rows ? rs * (d * ga - mA - xh * mB) : 0.f;
            }
        }
        __syncthreads();                                   // (the other buffer is written after the next one)
        if (t + gridDim.x < tiles) request((t + gridDim.x) * 128);      // in flight while this tile is stored
#pragma unroll
        for (int e = threadIdx.x; e < 128 * 4; e += 256) { // consecutive threads take consecutive 8-channel pieces of a row
            const int rr = e >> 2, piece = e & 3;
            const ll r = r0 + rr;
            if (r <= n_rows && c0 + piece * 8 < cpad) {
                __nv_bfloat162 h[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(tile[buf][piece * 8 + 2 * i][rr], tile[buf][piece * 8 + 2 * i + 1][rr]);
                *reinterpret_cast<uint4*>(out + r * cpad + c0 + piece * 8) = *reinterpret_cast<uint4*>(h);
            }
        }
    }
}

inline int gn_chunks(ll n, ll rows) {
    ll want = std::max<ll>(1, (148ll * 8 + rows - 1) / rows);
    want = std::min<ll>(want, (n + 4095) / 4096);
    return (int) std::max<ll>(1, std::min<ll>(GN_MAX_CHUNKS, want));
}

template<typename T, typename Entries = AllEntries>
int gn_forward(int B, int C, ll n, int groups, const T* x, const T* gamma, const T* beta, double eps, T* y, T* mean, T* rstd, double* ws, int relu, cudaStream_t st,
               const Entries& entries = Entries()) {
    const ll rows = (ll) B * C;
    const int cpg = C / groups;
    const int nchunks = gn_chunks(n, rows);
    const ll chunk_len = (n + nchunks - 1) / nchunks;
    const bool fused = cpg * nchunks <= GN_FUSE;
    { AprnetProfScope _p("groupnorm_stats", st);
    gn_partial_stats_kernel<T, Entries><<<dim3(nchunks, (unsigned) rows), GN_TPB, 0, st>>>(x, n, chunk_len, ws, nchunks, C, entries);
    if (!fused) gn_finalize_stats_kernel<T><<<(unsigned) (B * groups), GN_SUM_TPB, 0, st>>>(ws, nchunks, cpg, n, eps, mean, rstd);
    }
    const int gx = apply_blocks(n, rows);
    { AprnetProfScope _p("groupnorm_relu_apply", st);
    gn_relu_apply_kernel<T, Entries><<<dim3(gx, (unsigned) rows), GN_TPB, 0, st>>>(x, n, C, cpg, gamma, beta, mean, rstd, fused ? ws : nullptr, nchunks, eps, y, relu, entries);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

template<typename T>
int gn_backward(int B, int C, ll n, int groups, const T* x, const T* dy, const T* gamma, const T* beta, const T* mean, const T* rstd,
                T* dx, T* dgamma, T* dbeta, double* ws, int relu, cudaStream_t st) {
    const ll rows = (ll) B * C;
    const int cpg = C / groups;
    const int nchunks = gn_chunks(n, rows);
    const ll chunk_len = (n + nchunks - 1) / nchunks;
    double* row_sums = ws + rows * nchunks * 2;
    T* group_terms = reinterpret_cast<T*>(row_sums + rows * 2);
    const bool fused = B == 1 && cpg * nchunks <= GN_FUSE;
    { AprnetProfScope _p("groupnorm_bwd_reduce", st);
    gn_backward_partial_kernel<T><<<dim3(nchunks, (unsigned) rows), GN_TPB, 0, st>>>(x, dy, n, chunk_len, C, cpg, gamma, beta, mean, rstd, ws, nchunks, relu);
    if (!fused) gn_backward_rows_kernel<<<(unsigned) rows, GN_SUM_TPB, 0, st>>>(ws, nchunks, row_sums);
    if (!fused) gn_backward_finalize_kernel<T><<<aprnet_ceil_div(std::max<ll>(C, (ll) B * groups), 128), 128, 0, st>>>(row_sums, B, C, cpg, n, gamma, dgamma, dbeta, group_terms);
    }
    const int gx = apply_blocks(n, rows);
    { AprnetProfScope _p("groupnorm_bwd_apply", st);
    gn_backward_apply_kernel<T><<<dim3(gx, (unsigned) rows), GN_TPB, 0, st>>>(x, dy, n, C, cpg, gamma, beta, mean, rstd, group_terms, fused ? ws : nullptr, nchunks, dgamma, dbeta, dx, relu);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

} // namespace

// backward pass of one batch item whose dx leaves as packed bf16 rows [n_rows + 1][cpad] (the first n_rows entries of each channel, then a row of zeros)
int aprnet_groupnorm_relu_backward_rows(int C, ll n, ll n_rows, int groups, const float* x, const float* dy, const float* gamma, const float* beta,
                                        const float* mean, const float* rstd, float* dgamma, float* dbeta, int cpad, void* rows_out, double* ws, int relu, cudaStream_t st) {
    APRNET_ARG_CHECK(C > 0 && n > 0 && n_rows >= 0 && n_rows <= n && groups > 0 && C % groups == 0 && x && dy && mean && rstd && dgamma && dbeta && rows_out && ws &&
                     cpad >= C && cpad % 16 == 0, "bad argument");
    const int cpg = C / groups, nchunks = gn_chunks(n, C);
    const ll chunk_len = (n + nchunks - 1) / nchunks;
    double* row_sums = ws + (ll) C * nchunks * 2;
    float* group_terms = reinterpret_cast<float*>(row_sums + (ll) C * 2);
    const bool fused = cpg * nchunks <= GN_FUSE;
    { AprnetProfScope _p("groupnorm_bwd_reduce", st);
    gn_backward_partial_kernel<float><<<dim3(nchunks, (unsigned) C), GN_TPB, 0, st>>>(x, dy, n, chunk_len, C, cpg, gamma, beta, mean, rstd, ws, nchunks, relu);
    if (!fused) gn_backward_rows_kernel<<<(unsigned) C, GN_SUM_TPB, 0, st>>>(ws, nchunks, row_sums);
    if (!fused) gn_backward_finalize_kernel<float><<<aprnet_ceil_div(C, 128), 128, 0, st>>>(row_sums, 1, C, cpg, n, gamma, dgamma, dbeta, group_terms);
    }
    { AprnetProfScope _p("groupnorm_bwd_apply_rows", st);
    const int gy = aprnet_ceil_div(cpad, 32);
    gn_backward_apply_rows_kernel<<<dim3((unsigned) std::min<ll>(aprnet_ceil_div(n_rows + 1, 128), aprnet_ceil_div(148 * GN_ROWS_BLOCKS, gy)), (unsigned) gy), 256, 0, st>>>(
        x, dy, n, n_rows, C, cpg, gamma, beta, mean, rstd, group_terms, fused ? ws : nullptr, nchunks, dgamma, dbeta, relu, cpad, (__nv_bfloat16*) rows_out);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

// bytes of workspace for either direction
extern "C" int64_t aprnet_groupnorm_workspace_bytes(int batch, int channels, int groups) {
    const ll rows = (ll) batch * channels;
    return (int64_t) ((rows * GN_MAX_CHUNKS * 2 + rows * 2) * sizeof(double) + (ll) batch * groups * 2 * sizeof(double) + 256);
}

extern "C" int aprnet_groupnorm_relu_forward(int dtype, int batch, int channels, int64_t n, int groups, const void* x, const void* gamma,
                                             const void* beta, double eps, void* y, void* mean, void* rstd, void* workspace, int relu, void* stream) {
    APRNET_ARG_CHECK(batch > 0 && channels > 0 && n > 0 && groups > 0 && channels % groups == 0 && x && y && mean && rstd && workspace, "bad argument");
    cudaStream_t st = (cudaStream_t) stream;
    if (dtype == APRNET_F32) return gn_forward<float>(batch, channels, n, groups, (const float*) x, (const float*) gamma, (const float*) beta, eps, (float*) y, (float*) mean, (float*) rstd, (double*) workspace, relu, st);
    if (dtype == APRNET_F64) return gn_forward<double>(batch, channels, n, groups, (const double*) x, (const double*) gamma, (const double*) beta, eps, (double*) y, (double*) mean, (double*) rstd, (double*) workspace, relu, st);
    aprnet_set_error("aprnet_groupnorm_relu_forward: unknown dtype %d", dtype);
    return APRNET_ERR_ARG;
}

// forward pass over a batch whose items hold fewer than n entries: host_valid[item] of them; what lies behind counts as zeros and is not read
extern "C" int aprnet_groupnorm_relu_forward_valid(int dtype, int batch, int channels, int64_t n, const int64_t* host_valid, int groups, const void* x, const void* gamma,
                                                   const void* beta, double eps, void* y, void* mean, void* rstd, void* workspace, int relu, void* stream) {
    APRNET_ARG_CHECK(batch > 0 && channels > 0 && n > 0 && host_valid && groups > 0 && channels % groups == 0 && x && y && mean && rstd && workspace, "bad argument");
    if (batch > GN_ITEMS) { aprnet_set_error("%s: at most %d batch items", __func__, GN_ITEMS); return APRNET_ERR_UNSUPPORTED; }
    ItemEntries e;
    for (int b = 0; b < batch; ++b) {
        APRNET_ARG_CHECK(host_valid[b] >= 0 && host_valid[b] <= n, "more valid entries than the row holds");
        e.n[b] = host_valid[b];
    }
    cudaStream_t st = (cudaStream_t) stream;
    if (dtype == APRNET_F32) return gn_forward<float, ItemEntries>(batch, channels, n, groups, (const float*) x, (const float*) gamma, (const float*) beta, eps, (float*) y, (float*) mean, (float*) rstd, (double*) workspace, relu, st, e);
    if (dtype == APRNET_F64) return gn_forward<double, ItemEntries>(batch, channels, n, groups, (const double*) x, (const double*) gamma, (const double*) beta, eps, (double*) y, (double*) mean, (double*) rstd, (double*) workspace, relu, st, e);
    aprnet_set_error("%s: unknown dtype %d", __func__, dtype);
    return APRNET_ERR_ARG;
}

extern "C" int aprnet_groupnorm_relu_backward(int dtype, int batch, int channels, int64_t n, int groups, const void* x, const void* grad_y,
                                              const void* gamma, const void* beta, const void* mean, const void* rstd, void* grad_x,
                                              void* grad_gamma, void* grad_beta, void* workspace, int relu, void* stream) {
    APRNET_ARG_CHECK(batch > 0 && channels > 0 && n > 0 && groups > 0 && channels % groups == 0 && x && grad_y && mean && rstd && grad_x && workspace, "bad argument");
    cudaStream_t st = (cudaStream_t) stream;
    if (dtype == APRNET_F32) return gn_backward<float>(batch, channels, n, groups, (const float*) x, (const float*) grad_y, (const float*) gamma, (const float*) beta, (const float*) mean, (const float*) rstd, (float*) grad_x, (float*) grad_gamma, (float*) grad_beta, (double*) workspace, relu, st);
    if (dtype == APRNET_F64) return gn_backward<double>(batch, channels, n, groups, (const double*) x, (const double*) grad_y, (const double*) gamma, (const double*) beta, (const double*) mean, (const double*) rstd, (double*) grad_x, (double*) grad_gamma, (double*) grad_beta, (double*) workspace, relu, st);
    aprnet_set_error("aprnet_groupnorm_relu_backward: unknown dtype %d", dtype);
    return APRNET_ERR_ARG;
}

// ---- split forms: the caller combines the sums of several devices before the statistics are applied --------
// (one z-slab of an APR per GPU: every rank sums over the particles it owns, the sums are all-reduced, every rank
// applies the same mean / rstd).  row_sums: double [batch * channels][2].
template<typename T>
static int gn_row_sums(int B, int C, ll n, const T* x, double* ws, double* row_sums, cudaStream_t st) {
    const ll rows = (ll) B * C;
    const int nchunks = gn_chunks(n, rows);
    const ll chunk_len = (n + nchunks - 1) / nchunks;
    { AprnetProfScope _p("groupnorm_stats", st);
    gn_partial_stats_kernel<T, AllEntries><<<dim3(nchunks, (unsigned) rows), GN_TPB, 0, st>>>(x, n, chunk_len, ws, nchunks, C, AllEntries());
    gn_backward_rows_kernel<<<(unsigned) rows, GN_SUM_TPB, 0, st>>>(ws, nchunks, row_sums);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

template<typename T>
static int gn_apply(int B, int C, ll n, int groups, const T* x, const T* gamma, const T* beta, const T* mean, const T* rstd, T* y, int relu, cudaStream_t st) {
    const ll rows = (ll) B * C;
    const int gx = apply_blocks(n, rows);
    { AprnetProfScope _p("groupnorm_relu_apply", st);
    gn_relu_apply_kernel<T, AllEntries><<<dim3(gx, (unsigned) rows), GN_TPB, 0, st>>>(x, n, C, C / groups, gamma, beta, const_cast<T*>(mean), const_cast<T*>(rstd), nullptr, 0, 0.0, y, relu, AllEntries());
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

template<typename T>
static int gn_bwd_row_sums(int B, int C, ll n, int groups, const T* x, const T* dy, const T* gamma, const T* beta, const T* mean, const T* rstd,
                           double* ws, double* row_sums, int relu, cudaStream_t st) {
    const ll rows = (ll) B * C;
    const int nchunks = gn_chunks(n, rows);
    const ll chunk_len = (n + nchunks - 1) / nchunks;
    { AprnetProfScope _p("groupnorm_bwd_reduce", st);
    gn_backward_partial_kernel<T><<<dim3(nchunks, (unsigned) rows), GN_TPB, 0, st>>>(x, dy, n, chunk_len, C, C / groups, gamma, beta, mean, rstd, ws, nchunks, relu);
    gn_backward_rows_kernel<<<(unsigned) rows, GN_SUM_TPB, 0, st>>>(ws, nchunks, row_sums);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

template<typename T>
static int gn_bwd_apply(int B, int C, ll n, int groups, const T* x, const T* dy, const T* gamma, const T* beta, const T* mean, const T* rstd,
                        const T* group_terms, T* dx, int relu, cudaStream_t st) {
    const ll rows = (ll) B * C;
    const int gx = apply_blocks(n, rows);
    { AprnetProfScope _p("groupnorm_bwd_apply", st);
    gn_backward_apply_kernel<T><<<dim3(gx, (unsigned) rows), GN_TPB, 0, st>>>(x, dy, n, C, C / groups, gamma, beta, mean, rstd, group_terms, nullptr, 0, nullptr, nullptr, dx, relu);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

#define GN_DISPATCH(F32_CALL, F64_CALL)                                               \
    if (dtype == APRNET_F32) return F32_CALL;                                         \
    if (dtype == APRNET_F64) return F64_CALL;                                         \
    aprnet_set_error("%s: unknown dtype %d", __func__, dtype);                       \
    return APRNET_ERR_ARG;

extern "C" int aprnet_groupnorm_row_sums(int dtype, int batch, int channels, int64_t n, const void* x, void* workspace, double* row_sums, void* stream) {
    APRNET_ARG_CHECK(batch > 0 && channels > 0 && n > 0 && x && workspace && row_sums, "bad argument");
    cudaStream_t st = (cudaStream_t) stream;
    GN_DISPATCH(gn_row_sums<float>(batch, channels, n, (const float*) x, (double*) workspace, row_sums, st),
                gn_row_sums<double>(batch, channels, n, (const double*) x, (double*) workspace, row_sums, st))
}

extern "C" int aprnet_groupnorm_relu_apply(int dtype, int batch, int channels, int64_t n, int groups, const void* x, const void* gamma, const void* beta,
                                           const void* mean, const void* rstd, void* y, int relu, void* stream) {
    APRNET_ARG_CHECK(batch > 0 && channels > 0 && n > 0 && groups > 0 && channels % groups == 0 && x && y && mean && rstd, "bad argument");
    cudaStream_t st = (cudaStream_t) stream;
    GN_DISPATCH(gn_apply<float>(batch, channels, n, groups, (const float*) x, (const float*) gamma, (const float*) beta, (const float*) mean, (const float*) rstd, (float*) y, relu, st),
                gn_apply<double>(batch, channels, n, groups, (const double*) x, (const double*) gamma, (const double*) beta, (const double*) mean, (const double*) rstd, (double*) y, relu, st))
}

extern "C" int aprnet_groupnorm_backward_row_sums(int dtype, int batch, int channels, int64_t n, int groups, const void* x, const void* grad_y,
                                                  const void* gamma, const void* beta, const void* mean, const void* rstd, void* workspace,
                                                  double* row_sums, int relu, void* stream) {
    APRNET_ARG_CHECK(batch > 0 && channels > 0 && n > 0 && groups > 0 && channels % groups == 0 && x && grad_y && mean && rstd && workspace && row_sums, "bad argument");
    cudaStream_t st = (cudaStream_t) stream;
    GN_DISPATCH(gn_bwd_row_sums<float>(batch, channels, n, groups, (const float*) x, (const float*) grad_y, (const float*) gamma, (const float*) beta, (const float*) mean, (const float*) rstd, (double*) workspace, row_sums, relu, st),
                gn_bwd_row_sums<double>(batch, channels, n, groups, (const double*) x, (const double*) grad_y, (const double*) gamma, (const double*) beta, (const double*) mean, (const double*) rstd, (double*) workspace, row_sums, relu, st))
}

extern "C" int aprnet_groupnorm_backward_apply(int dtype, int batch, int channels, int64_t n, int groups, const void* x, const void* grad_y,
                                               const void* gamma, const void* beta, const void* mean, const void* rstd, const void* group_terms,
                                               void* grad_x, int relu, void* stream) {
    APRNET_ARG_CHECK(batch > 0 && channels > 0 && n > 0 && groups > 0 && channels % groups == 0 && x && grad_y && mean && rstd && group_terms && grad_x, "bad argument");
    cudaStream_t st = (cudaStream_t) stream;
    GN_DISPATCH(gn_bwd_apply<float>(batch, channels, n, groups, (const float*) x, (const float*) grad_y, (const float*) gamma, (const float*) beta, (const float*) mean, (const float*) rstd, (const float*) group_terms, (float*) grad_x, relu, st),
                gn_bwd_apply<double>(batch, channels, n, groups, (const double*) x, (const double*) grad_y, (const double*) gamma, (const double*) beta, (const double*) mean, (const double*) rstd, (const double*) group_terms, (double*) grad_x, relu, st))
}
