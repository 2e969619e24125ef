// Stencil weights of the 3x3x3 convolution: restriction of the given stencils to one per level (and its transpose), and packing
// of the level stencils into the operand layouts of the gather kernels.
//
// All move blocks of whole filters (27 contiguous values) through shared memory, so that both sides of memory are read and
// written in whole lines.  One thread per filter or per packed element, as before, read four bytes of every line: 2.0 ms of an 8.1 ms
// training step on a 64 x 128 x 128 patch, whatever the number of particles.
// Arithmetic of the restriction: pyapr/aprnet/src/kernel.hpp:54-224.
#include "apr_device.cuh"
#include <cuda_bf16.h>
#include <algorithm>

namespace {

typedef long long ll;
constexpr int FB = 128;                // filters per block, one per thread
constexpr int CROW = 28;               // row of the coefficient table, a whole number of 16-byte vectors

// Slots < S are copied; slot k >= S is the last given stencil box-averaged onto a grid 2^(k-S+1) times coarser (overlap lengths per
// axis, divided by step^3).  Overlap weight between fine tap ti and coarse tap to along one axis, for a grid `step` times coarser:
__device__ __forceinline__ float restrict_overlap(int step, int fine_tap, int coarse_tap) {
    const int off = step - 1;
    return fmaxf(0.f, (float) (min((coarse_tap + 1) * step, off + fine_tap + step) - max(coarse_tap * step, off + fine_tap)));
}

// coef[to][ti]: share of fine tap ti in coarse tap to of slot k (products of small integers times a power of two: exact)
template<typename T>
__device__ __forceinline__ void restrict_table(int S, int k, T (*coef)[CROW]) {
    const int step = 1 << (k - (S - 1));
    const float inv = 1.0f / ((float) step * (float) step * (float) step);
    float ov[3][3];
#pragma unroll
    for (int t = 0; t < 9; ++t) ov[t / 3][t % 3] = restrict_overlap(step, t % 3, t / 3);      // [coarse][fine]
    if (threadIdx.x < 27) {              // thread = coarse tap; its row of 27 products is unrolled
        const int z = threadIdx.x / 9, x = (threadIdx.x / 3) % 3, y = threadIdx.x % 3;
        float oz[3], ox[3], oy[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            oz[i] = z == 0 ? ov[0][i] : (z == 1 ? ov[1][i] : ov[2][i]);
            ox[i] = x == 0 ? ov[0][i] : (x == 1 ? ov[1][i] : ov[2][i]);
            oy[i] = y == 0 ? ov[0][i] : (y == 1 ? ov[1][i] : ov[2][i]);
        }
#pragma unroll
        for (int t = 0; t < 27; ++t) coef[threadIdx.x][t] = (T) (ox[(t / 3) % 3] * oy[t % 3] * oz[t / 9] * inv);
    }
}

// The grid of an extra slot is at least twice coarser, so along an axis the middle fine tap lies in the middle coarse tap and an outer
// one in the middle and in its own: 125 of the 729 pairs overlap.  The others are left out, not multiplied by zero: a value that is not
// finite stays in the taps that it belongs to.
__host__ __device__ constexpr bool restrict_axis(int fine, int coarse) { return coarse == 1 || (fine != 1 && fine == coarse); }
__host__ __device__ constexpr bool restrict_overlaps(int fine, int coarse) {
    return restrict_axis(fine / 9, coarse / 9) && restrict_axis(fine / 3 % 3, coarse / 3 % 3) && restrict_axis(fine % 3, coarse % 3);
}

// grid (filter blocks, level slots).  A thread holds the 27 values of its filter and adds the products of a result in ascending order
// of the fine taps; the coefficients are broadcast reads.
template<typename T>
__global__ void __launch_bounds__(FB) restrict333_forward_kernel(int S, ll filters, const T* __restrict__ src, T* __restrict__ dst) {
    __shared__ T stage[FB * 27];
    __shared__ __align__(16) T coef[27][CROW];
    const int k = blockIdx.y;
    const ll f0 = (ll) blockIdx.x * FB;
    const int n = (int) min((ll) FB, filters - f0) * 27;
    const T* from = src + ((ll) min(k, S - 1) * filters + f0) * 27;
    T* to = dst + ((ll) k * filters + f0) * 27;
    if (k < S) {
#pragma unroll 9
        for (int e = threadIdx.x; e < n; e += FB) to[e] = from[e];
        return;
    }
#pragma unroll 9
    for (int e = threadIdx.x; e < n; e += FB) stage[e] = from[e];
    restrict_table<T>(S, k, coef);
    __syncthreads();
    T fine[27];
#pragma unroll
    for (int t = 0; t < 27; ++t) fine[t] = stage[threadIdx.x * 27 + t];
#pragma unroll
    for (int o = 0; o < 27; ++o) {
        T acc = 0;
#pragma unroll
        for (int t = 0; t < 27; ++t) if (restrict_overlaps(t, o)) acc += coef[o][t] * fine[t];
        stage[threadIdx.x * 27 + o] = acc;             // this thread's own values
    }
    __syncthreads();
#pragma unroll 9
    for (int e = threadIdx.x; e < n; e += FB) to[e] = stage[e];
}

// transpose: every extra slot is folded into slot S-1, slots, then coarse taps, in ascending order
template<typename T>
__global__ void __launch_bounds__(FB) restrict333_backward_kernel(int S, int L, ll filters, const T* __restrict__ src, T* __restrict__ dst) {
    __shared__ T stage[FB * 27];
    __shared__ __align__(16) T coef[27][CROW];
    const int s = blockIdx.y;
    const ll f0 = (ll) blockIdx.x * FB;
    const int n = (int) min((ll) FB, filters - f0) * 27;
    const T* from = src + ((ll) s * filters + f0) * 27;
    T* to = dst + ((ll) s * filters + f0) * 27;
    if (s < S - 1) {
#pragma unroll 9
        for (int e = threadIdx.x; e < n; e += FB) to[e] = from[e];
        return;
    }
#pragma unroll 9
    for (int e = threadIdx.x; e < n; e += FB) stage[e] = from[e];
    __syncthreads();
    T acc[27];
#pragma unroll
    for (int t = 0; t < 27; ++t) acc[t] = stage[threadIdx.x * 27 + t];
    T next[27];                          // the next slot's values, requested while this one's are used
    auto request = [&](int k) {
#pragma unroll
        for (int i = 0; i < 27; ++i) { const int e = threadIdx.x + i * FB; next[i] = e < n ? src[((ll) k * filters + f0) * 27 + e] : T(0); }
    };
    if (S < L) request(S);
    for (int k = S; k < L; ++k) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 27; ++i) stage[threadIdx.x + i * FB] = next[i];
        restrict_table<T>(S, k, coef);
        __syncthreads();
        if (k + 1 < L) request(k + 1);
#pragma unroll
        for (int o = 0; o < 27; ++o) {
            const T c = stage[threadIdx.x * 27 + o];
#pragma unroll
            for (int t = 0; t < 27; ++t) if (restrict_overlaps(t, o)) acc[t] += coef[o][t] * c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 27; ++t) stage[threadIdx.x * 27 + t] = acc[t];
    __syncthreads();
#pragma unroll 9
    for (int e = threadIdx.x; e < n; e += FB) to[e] = stage[e];
}

template<typename T>
int restrict333(int S, int L, ll filters, const T* src, T* dst, bool backward, cudaStream_t st) {
    const unsigned gx = (unsigned) aprnet_ceil_div(filters, FB);
    if (backward) restrict333_backward_kernel<T><<<dim3(gx, (unsigned) S), FB, 0, st>>>(S, L, filters, src, dst);
    else restrict333_forward_kernel<T><<<dim3(gx, (unsigned) L), FB, 0, st>>>(S, filters, src, dst);
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

// ---- packing --------------------------------------------------------------------------------------------
// Block = 32 result channels (n) x 8 source channels (k) of one slot, all 27 taps.  transposed == 0: n = co, k = ci (forward);
// 1: n = ci, k = co (input gradient; the same-level part reads the taps mirrored).  Channels beyond their extents are zeros.
//   bf16: [slot][tap][n tile][k / 8][nt][8]       (canonical K-major operand of the tensor cores per slot, tap and n tile)
//   fp32: [slot][tap][n tile][k][nt]
struct UsedSlots { int n; int slot[APRNET_MAX_LEVELS]; };
constexpr int PK_N = 32, PK_ROW = 8 * 27 + 1;

template<bool BF16>
__global__ void __launch_bounds__(256) pack_weights_kernel(const float* __restrict__ w, UsedSlots used, int cin, int cout, int transposed,
                                                           int nt, int n_tiles, int kpad, void* __restrict__ out) {
    __shared__ float tile[PK_N][PK_ROW];      // [n][k][tap]; the odd row length spreads the n of a warp over the banks
    const int slot = used.slot[blockIdx.z], k0 = blockIdx.x * 8, n0 = blockIdx.y * PK_N;
    const int n_dim = transposed ? cin : cout, k_dim = transposed ? cout : cin;
    const float* ws = w + (ll) slot * cout * cin * 27;
#pragma unroll
    for (int i = 0; i < PK_N * 8 * 27 / 256; ++i) {          // 27: all requested before any is stored
        const int e = threadIdx.x + i * 256;
        int n, k, tap;
        if (transposed) { k = e / (PK_N * 27); n = (e / 27) % PK_N; tap = e % 27; }        // ci (n) and tap are contiguous in memory
        else { n = e / (8 * 27); k = (e / 27) % 8; tap = e % 27; }                         // ci (k) and tap
        float v = 0.f;
        if (n0 + n < n_dim && k0 + k < k_dim) {
            const int co = transposed ? k0 + k : n0 + n, ci = transposed ? n0 + n : k0 + k;
            v = ws[((ll) co * cin + ci) * 27 + tap];
        }
        tile[n][k * 27 + tap] = v;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, n = n0 + lane;
    if (n >= n_tiles * nt) return;
    const int ntile = n / nt, nn = n - ntile * nt;
    for (int tap = threadIdx.x >> 5; tap < 27; tap += 8) {
        const ll base = ((ll) slot * 27 + tap) * n_tiles + ntile;
        if (BF16) {
            __nv_bfloat162 h[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(tile[lane][2 * i * 27 + tap], tile[lane][(2 * i + 1) * 27 + tap]);
            *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(out) + ((base * (kpad / 8) + blockIdx.x) * nt + nn) * 8) = *reinterpret_cast<const uint4*>(h);
        } else {
            float* o = reinterpret_cast<float*>(out) + (base * kpad + k0) * nt + nn;
#pragma unroll
            for (int k = 0; k < 8; ++k) if (k0 + k < kpad) o[k * nt] = tile[lane][k * 27 + tap];
        }
    }
}

} // namespace

// Packs the stencils of the slots that the locations of level delta dl use (the others of the expanded set meet no location).
int aprnet_pack_weights(const aprnet_apr* a, int dl, bool bf16, const float* w, int slots, int cin, int cout, int transposed, int nt, int n_tiles, int kpad,
                        void* out, cudaStream_t st) {
    UsedSlots used;
    used.n = 0;
    for (const Segment& sg : aprnet_segments(a, dl, slots, false))
        if (used.n == 0 || used.slot[used.n - 1] != sg.slot) used.slot[used.n++] = sg.slot;      // coarse to fine: equal slots are neighbours
    if (used.n == 0) return APRNET_OK;
    const dim3 grid((unsigned) aprnet_ceil_div(kpad, 8), (unsigned) aprnet_ceil_div((ll) n_tiles * nt, PK_N), (unsigned) used.n);
    AprnetProfScope _prof(bf16 ? "pack_weights_bf16" : "pack_weights_f32", st);
    if (bf16) pack_weights_kernel<true><<<grid, 256, 0, st>>>(w, used, cin, cout, transposed, nt, n_tiles, kpad, out);
    else pack_weights_kernel<false><<<grid, 256, 0, st>>>(w, used, cin, cout, transposed, nt, n_tiles, kpad, out);
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

extern "C" int aprnet_restrict333_forward(int dtype, int S, int L, int64_t filters, const void* w, void* expanded, void* stream) {
    APRNET_ARG_CHECK(w && expanded && S > 0 && L >= S && filters > 0, "requires num_levels >= num_stencils");
    cudaStream_t st = (cudaStream_t) stream;
    if (dtype == APRNET_F32) return restrict333<float>(S, L, filters, (const float*) w, (float*) expanded, false, st);
    if (dtype == APRNET_F64) return restrict333<double>(S, L, filters, (const double*) w, (double*) expanded, false, st);
    aprnet_set_error("%s: unknown dtype %d", __func__, dtype);
    return APRNET_ERR_ARG;
}

extern "C" int aprnet_restrict333_backward(int dtype, int S, int L, int64_t filters, const void* gexp, void* gw, void* stream) {
    APRNET_ARG_CHECK(gexp && gw && S > 0 && L >= S && filters > 0, "requires num_stencils <= expanded levels");
    cudaStream_t st = (cudaStream_t) stream;
    if (dtype == APRNET_F32) return restrict333<float>(S, L, filters, (const float*) gexp, (float*) gw, true, st);
    if (dtype == APRNET_F64) return restrict333<double>(S, L, filters, (const double*) gexp, (double*) gw, true, st);
    aprnet_set_error("%s: unknown dtype %d", __func__, dtype);
    return APRNET_ERR_ARG;
}
