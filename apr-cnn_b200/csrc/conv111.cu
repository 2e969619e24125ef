// 1x1x1 particle convolution (per-level channel mixing).
//
// Replaces pyapr/aprnet/cuda/src/conv111_gpu.cu:9-232.  The reference
// splits input channels over grid.z and combines them with atomicAdd into a zero-filled output; here
// one thread owns a particle and a block of output channels, loops over all input channels and
// writes each output once (no atomics, deterministic).  Weight gradients are block-local partial
// sums followed by a fixed-order second pass.
#include "apr_device.cuh"
#include <algorithm>

namespace {

typedef long long ll;
constexpr int MAX_SEGS = APRNET_MAX_LEVELS;

struct SegTable {
    int n;
    ll begin[MAX_SEGS], end[MAX_SEGS];
    int slot[MAX_SEGS];
    int tile_begin[MAX_SEGS + 1];     // cumulative tile counts
};

inline SegTable make_seg_table(const std::vector<Segment>& segs, int tile) {
    SegTable t;
    t.n = (int) segs.size();
    t.tile_begin[0] = 0;
    for (int i = 0; i < t.n; ++i) {
        t.begin[i] = segs[i].begin; t.end[i] = segs[i].end; t.slot[i] = segs[i].slot;
        t.tile_begin[i + 1] = t.tile_begin[i] + aprnet_ceil_div(segs[i].end - segs[i].begin, tile);
    }
    return t;
}

// 16-byte vector of T (4 floats / 2 doubles): the staged weights are read from shared memory in such pieces, so that
// one shared-memory instruction feeds several multiply-adds (with scalar reads the kernel is bound by the
// shared-memory pipe, one broadcast read per multiply-add).
template<typename T> struct Vec16;
template<> struct Vec16<float> { typedef float4 type; static constexpr int N = 4; };
template<> struct Vec16<double> { typedef double2 type; static constexpr int N = 2; };

// out[o][p] = sum_i w[slot][o][i] * in[i][p]; weight element (s, o, i) at w[s*ws + o*wo + i*wi]
// (forward: wo = Cin, wi = 1; input gradient: roles of the channel axes swapped, wo = 1, wi = Cin_fwd).
// A thread owns PPT locations (p, p + TPB, ...) and OB output channels: every 16-byte weight read from shared memory
// feeds 4 * PPT multiply-adds.  (With one location per thread the kernel ran at 84 % of the load/store pipe and 32 % of
// DRAM: bound by the broadcast weight reads.)
template<typename T, int OB, int TPB, int PPT>
__global__ void __launch_bounds__(TPB, sizeof(T) == 4 ? 2 : 1) conv111_kernel(SegTable segs, const T* __restrict__ in, ll ld_in,
                                                      const T* __restrict__ w, ll ws, ll wo, ll wi,
                                                      const T* __restrict__ bias, T* __restrict__ out, ll ld_out, int n_in, int n_out) {
    typedef typename Vec16<T>::type V;
    constexpr int VN = Vec16<T>::N;
    static_assert(OB % VN == 0, "output block is a whole number of 16-byte vectors");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* wsm = reinterpret_cast<T*>(smem_raw);              // [n_in][OB]
    int seg = 0;
    while (seg + 1 < segs.n && (int) blockIdx.x >= segs.tile_begin[seg + 1]) ++seg;
    const ll p0 = segs.begin[seg] + (ll) (blockIdx.x - segs.tile_begin[seg]) * (TPB * PPT) + threadIdx.x;
    const ll pend = segs.end[seg];
    const int o0 = blockIdx.y * OB;
    const T* wslot = w + (ll) segs.slot[seg] * ws;
    for (int e = threadIdx.x; e < n_in * OB; e += TPB) {
        const int i = e / OB, o = e % OB;
        wsm[e] = (o0 + o < n_out) ? wslot[(ll) (o0 + o) * wo + (ll) i * wi] : T(0);
    }
    __syncthreads();
    if (p0 >= pend) return;
    T acc[PPT][OB];
#pragma unroll
    for (int q = 0; q < PPT; ++q)
#pragma unroll
        for (int o = 0; o < OB; ++o) acc[q][o] = 0;
    constexpr int IU = PPT == 1 ? 8 : 4;     // input channels whose loads are in flight together
    auto mix = [&](const T (&v)[PPT], const int i) {
        const V* wr = reinterpret_cast<const V*>(wsm + i * OB);
#pragma unroll
        for (int o = 0; o < OB / VN; ++o) {
            const V wv = wr[o];
            const T* we = reinterpret_cast<const T*>(&wv);
#pragma unroll
            for (int e = 0; e < VN; ++e)
#pragma unroll
                for (int q = 0; q < PPT; ++q) acc[q][o * VN + e] = fma(v[q], we[e], acc[q][o * VN + e]);
        }
    };
    int i = 0;
    for (; i + IU <= n_in; i += IU) {
        T v[IU][PPT];
#pragma unroll
        for (int k = 0; k < IU; ++k)
#pragma unroll
            for (int q = 0; q < PPT; ++q) v[k][q] = (p0 + (ll) q * TPB < pend) ? in[(ll) (i + k) * ld_in + p0 + (ll) q * TPB] : T(0);
#pragma unroll
        for (int k = 0; k < IU; ++k) mix(v[k], i + k);
    }
    for (; i < n_in; ++i) {
        T v[PPT];
#pragma unroll
        for (int q = 0; q < PPT; ++q) v[q] = (p0 + (ll) q * TPB < pend) ? in[(ll) i * ld_in + p0 + (ll) q * TPB] : T(0);
        mix(v, i);
    }
    if (bias) {
#pragma unroll
        for (int o = 0; o < OB; ++o) {
            const T b = o0 + o < n_out ? bias[o0 + o] : T(0);
#pragma unroll
            for (int q = 0; q < PPT; ++q) acc[q][o] += b;
        }
    }
#pragma unroll
    for (int q = 0; q < PPT; ++q) {
        const ll p = p0 + (ll) q * TPB;
        if (p >= pend) break;
#pragma unroll
        for (int o = 0; o < OB; ++o)
            if (o0 + o < n_out) out[(ll) (o0 + o) * ld_out + p] = acc[q][o];
    }
}

// Weight gradient of one segment: partial[chunk][o][i] = sum over the chunk's particles of
// gout[o][p] * in[i][p].  Block tile 64 (o) x 64 (i), 256 threads, 4x4 outputs per thread: per particle a thread
// reads 4 + 4 values from shared memory (two 16-byte reads for floats) for 16 multiply-adds.
template<typename T>
__global__ void __launch_bounds__(256) conv111_dw_partial_kernel(ll seg_begin, ll seg_end, ll chunk_len,
                                                                 const T* __restrict__ in, ll ld_in,
                                                                 const T* __restrict__ gout, ll ld_out,
                                                                 T* __restrict__ partial, int cin, int cout) {
    constexpr int TILE = 64, KC = 32;
    // [particle][channel]: a thread's four channels are contiguous; rows padded by 4 so that the transposing stores of a
    // warp (32 particles of one channel) spread over 8 banks instead of one
    __shared__ __align__(16) T gs[KC][TILE + 4];
    __shared__ __align__(16) T xs[KC][TILE + 4];
    const int nib = (cin + TILE - 1) / TILE;
    const int ob = blockIdx.y / nib, ib = blockIdx.y % nib;
    const ll pb = seg_begin + (ll) blockIdx.x * chunk_len;
    const ll pe = min(seg_end, pb + chunk_len);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;          // 4 input channels, 4 output channels
    T acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0;
    for (ll p0 = pb; p0 < pe; p0 += KC) {
        // consecutive threads read consecutive particles of one channel row (coalesced), stored transposed
        for (int e = threadIdx.x; e < TILE * KC; e += 256) {
            const int r = e / KC, k = e % KC;
            const bool inr = p0 + k < pe;
            const int o = ob * TILE + r, i = ib * TILE + r;
            gs[k][r] = (inr && o < cout) ? gout[(ll) o * ld_out + p0 + k] : T(0);
            xs[k][r] = (inr && i < cin) ? in[(ll) i * ld_in + p0 + k] : T(0);
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < KC; ++k) {
            T g[4], x[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) { g[a] = gs[k][4 * ty + a]; x[a] = xs[k][4 * tx + a]; }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] = fma(g[a], x[b], acc[a][b]);
        }
        __syncthreads();
    }
    T* dst = partial + (ll) blockIdx.x * cout * cin;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int o = ob * TILE + 4 * ty + a, i = ib * TILE + 4 * tx + b;
            if (o < cout && i < cin) dst[(ll) o * cin + i] = acc[a][b];
        }
}

// Weight gradient for few output channels (CO <= 4, e.g. a classification head): a lane owns one particle
// of a 32-particle strip and keeps the CO x 32 products of one block of 32 input channels; strips are
// visited in a fixed order, lanes and warps are combined in a fixed order.
template<typename T, int CO>
__global__ void __launch_bounds__(256) conv111_dw_small_kernel(ll seg_begin, ll seg_end, ll chunk_len,
                                                               const T* __restrict__ in, ll ld_in,
                                                               const T* __restrict__ gout, ll ld_out,
                                                               T* __restrict__ partial, int cin, int cout) {
    __shared__ T red[8][CO * 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i0 = blockIdx.y * 32;
    const ll pb = seg_begin + (ll) blockIdx.x * chunk_len;
    const ll pe = min(seg_end, pb + chunk_len);
    T acc[CO][32];
#pragma unroll
    for (int o = 0; o < CO; ++o)
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[o][i] = 0;
    for (ll p = pb + warp * 32 + lane; p < pe; p += 256) {
        T g[CO];
#pragma unroll
        for (int o = 0; o < CO; ++o) g[o] = o < cout ? gout[(ll) o * ld_out + p] : T(0);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const T x = i0 + i < cin ? in[(ll) (i0 + i) * ld_in + p] : T(0);
#pragma unroll
            for (int o = 0; o < CO; ++o) acc[o][i] = fma(g[o], x, acc[o][i]);
        }
    }
#pragma unroll
    for (int o = 0; o < CO; ++o)
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            T v = acc[o][i];
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
            if (lane == 0) red[warp][o * 32 + i] = v;
        }
    __syncthreads();
    T* dst = partial + (ll) blockIdx.x * cout * cin;
    for (int e = threadIdx.x; e < CO * 32; e += 256) {
        const int o = e / 32, i = i0 + e % 32;
        T v = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[w][e];
        if (o < cout && i < cin) dst[(ll) o * cin + i] = v;
    }
}

// dst[e] += the chunks' sums of entry e in a fixed order: a block has 32 entries, warp w adds every eighth chunk (one thread for all of them waited for the 100 to 500
// loads of an entry)
template<typename T>
__global__ void __launch_bounds__(256) reduce_partial_kernel(const T* __restrict__ partial, int nchunks, ll elems, T* __restrict__ dst) {
    __shared__ T part[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const ll e = (ll) blockIdx.x * 32 + lane;
    T s = 0;
    if (e < elems)
#pragma unroll 8
        for (int c = w; c < nchunks; c += 8) s += partial[(ll) c * elems + e];
    part[w][lane] = s;
    __syncthreads();
    if (w == 0 && e < elems) {
        for (int k = 1; k < 8; ++k) s += part[k][lane];
        dst[e] += s;
    }
}

// block partials of the weight gradient: many chunks for small filters (parallelism), fewer for large ones (workspace)
inline int dw_max_chunks(int cin, int cout) { return (int) std::max<ll>(128, std::min<ll>(2048, (16ll << 20) / ((ll) cin * cout))); }

template<typename T, int OB, int TPB, int PPT>
int conv111_launch(const aprnet_apr* a, int dl, int S, const T* in, ll ld_in, const T* w, ll ws, ll wo, ll wi, const T* bias, T* out, ll ld_out,
                   int n_in, int n_out, cudaStream_t st) {
    const SegTable segs = make_seg_table(aprnet_segments(a, dl, S, true), TPB * PPT);
    const int tiles = segs.tile_begin[segs.n];
    if (tiles == 0) return APRNET_OK;
    const size_t smem = (size_t) n_in * OB * sizeof(T);
    if (smem > 48 * 1024)
        APRNET_CUDA_CHECK(cudaFuncSetAttribute(conv111_kernel<T, OB, TPB, PPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    dim3 grid((unsigned) tiles, (unsigned) aprnet_ceil_div(n_out, OB));
    { AprnetProfScope _prof("conv111", st);
    conv111_kernel<T, OB, TPB, PPT><<<grid, TPB, smem, st>>>(segs, in, ld_in, w, ws, wo, wi, bias, out, ld_out, n_in, n_out);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

template<typename T>
int conv111_apply(const aprnet_apr* a, int dl, int n_in, int n_out, int S, const T* in, ll ld_in, const T* w,
                  ll ws, ll wo, ll wi, const T* bias, T* out, ll ld_out, cudaStream_t st) {
    constexpr int TPB = 256;
    if (n_out <= 4) return conv111_launch<T, 4, TPB, 4>(a, dl, S, in, ld_in, w, ws, wo, wi, bias, out, ld_out, n_in, n_out, st);      // e.g. a classification head
    if (n_out <= 16) return conv111_launch<T, 16, TPB, 2>(a, dl, S, in, ld_in, w, ws, wo, wi, bias, out, ld_out, n_in, n_out, st);
    // the input is read once per 32 outputs; two locations per thread (fp32) halve the shared-memory reads per multiply-add
    if (sizeof(T) == 4) return conv111_launch<T, 32, TPB, 2>(a, dl, S, in, ld_in, w, ws, wo, wi, bias, out, ld_out, n_in, n_out, st);
    return conv111_launch<T, 32, TPB, 1>(a, dl, S, in, ld_in, w, ws, wo, wi, bias, out, ld_out, n_in, n_out, st);
}

template<typename T>
int conv111_dw(const aprnet_apr* a, int dl, int cin, int cout, int S, const T* in, ll ld_in, const T* gout, ll ld_out,
               T* gw, T* partial, cudaStream_t st) {
    const std::vector<Segment> segs = aprnet_segments(a, dl, S, true);
    const ll elems = (ll) cin * cout;
    for (const Segment& s : segs) {
        const ll len = s.end - s.begin;
        // few outputs: blocks of 32 input channels (conv111_dw_small_kernel); else 64 x 64 tiles
        const unsigned gy = cout <= 4 ? (unsigned) aprnet_ceil_div(cin, 32) : (unsigned) (aprnet_ceil_div(cout, 64) * aprnet_ceil_div(cin, 64));
        // chunks of 1024 locations, shorter ones where those leave SMs without a block, down to 128: fp32 training steps on 9.7 k, 26 k and 503 k
        // locations 7.5 -> 7.3, 9.8 -> 9.4 and 43.0 -> 42.6 ms, with the sums added by eight warps
        const ll fill = std::min<ll>((len + 127) / 128, (3 * 148 + gy - 1) / gy);
        const int nchunks = (int) std::min<ll>(dw_max_chunks(cin, cout), std::max<ll>((len + 1023) / 1024, fill));
        const ll chunk_len = ((len + nchunks - 1) / nchunks + 31) / 32 * 32;
        dim3 grid((unsigned) nchunks, gy);
        { AprnetProfScope _prof("conv111_dw", st);
        if (cout <= 4) conv111_dw_small_kernel<T, 4><<<grid, 256, 0, st>>>(s.begin, s.end, chunk_len, in, ld_in, gout, ld_out, partial, cin, cout);
        else conv111_dw_partial_kernel<T><<<grid, 256, 0, st>>>(s.begin, s.end, chunk_len, in, ld_in, gout, ld_out, partial, cin, cout);
        }
        { AprnetProfScope _prof("conv111_dw_reduce", st);
        reduce_partial_kernel<T><<<(unsigned) aprnet_ceil_div(elems, 32), 256, 0, st>>>(partial, nchunks, elems, gw + (ll) s.slot * elems);
        }
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

} // namespace

#define DISPATCH(dtype, CALL_F, CALL_D)                                                   \
    switch (dtype) {                                                                      \
        case APRNET_F32: return CALL_F;                                                   \
        case APRNET_F64: return CALL_D;                                                   \
        default: aprnet_set_error("%s: unknown dtype %d", __func__, dtype); return APRNET_ERR_ARG; \
    }

extern "C" int aprnet_conv111_forward_bias(const aprnet_apr* a, int dl, int dtype, int cin, int cout, int S, const void* in,
                                           int64_t ld_in, const void* w, const void* bias, void* out, int64_t ld_out, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && in && w && out && cin > 0 && cout > 0 && S > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl), "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    const ll ws = (ll) cin * cout;
    DISPATCH(dtype, conv111_apply<float>(a, dl, cin, cout, S, (const float*) in, ld_in, (const float*) w, ws, cin, 1, (const float*) bias, (float*) out, ld_out, st),
             conv111_apply<double>(a, dl, cin, cout, S, (const double*) in, ld_in, (const double*) w, ws, cin, 1, (const double*) bias, (double*) out, ld_out, st));
}

extern "C" int aprnet_conv111_forward(const aprnet_apr* a, int dl, int dtype, int cin, int cout, int S, const void* in,
                                      int64_t ld_in, const void* w, void* out, int64_t ld_out, void* stream) {
    return aprnet_conv111_forward_bias(a, dl, dtype, cin, cout, S, in, ld_in, w, nullptr, out, ld_out, stream);
}

extern "C" int aprnet_conv111_backward_input(const aprnet_apr* a, int dl, int dtype, int cin, int cout, int S,
                                             const void* gout, int64_t ld_out, const void* w, void* gin, int64_t ld_in,
                                             void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && gout && w && gin && cin > 0 && cout > 0 && S > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl), "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    const ll ws = (ll) cin * cout;
    DISPATCH(dtype, conv111_apply<float>(a, dl, cout, cin, S, (const float*) gout, ld_out, (const float*) w, ws, 1, cin, nullptr, (float*) gin, ld_in, st),
             conv111_apply<double>(a, dl, cout, cin, S, (const double*) gout, ld_out, (const double*) w, ws, 1, cin, nullptr, (double*) gin, ld_in, st));
}

extern "C" int64_t aprnet_conv111_partial_elems(int cin, int cout) { return (int64_t) dw_max_chunks(cin, cout) * cin * cout; }

extern "C" int aprnet_conv111_backward_weights(const aprnet_apr* a, int dl, int dtype, int cin, int cout, int S,
                                               const void* in, int64_t ld_in, const void* gout, int64_t ld_out,
                                               void* gw, void* partial, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && in && gout && gw && partial && cin > 0 && cout > 0 && S > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl), "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    DISPATCH(dtype, conv111_dw<float>(a, dl, cin, cout, S, (const float*) in, ld_in, (const float*) gout, ld_out, (float*) gw, (float*) partial, st),
             conv111_dw<double>(a, dl, cin, cout, S, (const double*) in, ld_in, (const double*) gout, ld_out, (double*) gw, (double*) partial, st));
}
