// Tree fill (mean / max), max pooling and constant up-sampling.
//
// All four are child <-> parent transfers along the APR tree.  They run as index-driven gathers over
// the cached child table: one thread per parent tree node, eight child slots, channels looped inside
// the thread so the indices are read once.  Consecutive threads hold consecutive nodes of a sparse
// row, whose children are consecutive in the child rows, so the value accesses coalesce.  The adjoint of the
// tree mean is the exception: it runs child-centric over cached parent tables (see its kernel).
// Arithmetic follows pyapr/aprnet/src/helpers.hpp:156-350 (tree mean and its adjoint),
// pyapr/aprnet/src/maxpool.hpp:70-230 and pyapr/aprnet/src/upsample.hpp:70-236.
#include "apr_device.cuh"
#include <algorithm>
#include <cmath>

namespace {

typedef long long ll;
constexpr int TPB = 256;                 // threads (= parent nodes) per block
constexpr int CH_PER_BLOCK = 8;          // channels a block loops over with the child slots resolved once

template<typename T> struct DT;
template<> struct DT<float> { static constexpr int id = APRNET_F32; };
template<> struct DT<double> { static constexpr int id = APRNET_F64; };

// One tree level: node t = scale[t] * sum(children) (MAX: their maximum).  A thread owns a node and CH channels; the
// block's channel group is the fast grid axis, so that the groups of the same nodes run together and find the 36-byte
// table entries of a node in L2.  All CH x 8 child values are requested before any is used.
// The levels are a chain of short launches, each of which reads what the one before wrote: a launch starts behind the running one and has its table entries when that one
// ends (8 channels on 256 x 512 x 512, mean and maximum of all levels: 122 -> 104 us; one launch after the other, each began with a gap and the latency of the table).
template<typename T, int CH, bool MAX, bool BEHIND = false>
__device__ __forceinline__ void tree_node(const int32_t* __restrict__ child, const float* __restrict__ scale, ll n_tree, ll t,
                                          const T* __restrict__ in, ll ld_in, T* tree, ll ld_tree, int c0, int nch, ll up_off, int use_up) {
    int32_t v[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) v[s] = __ldg(child + (ll) s * n_tree + t);
    const T f = MAX ? T(1) : (T) __ldg(scale + t);
    if (BEHIND) wait_for_grid_before();         // for the finer level's nodes
    const T* xin = in + (ll) c0 * ld_in;
    const T* xtree = use_up ? xin + up_off : tree + (ll) c0 * ld_tree;     // coded children: upgraded nodes in the features, else the tree scratch
    const ll ld_coded = use_up ? ld_in : ld_tree;
    T vals[CH][8];
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const T* src = v[s] >= 0 ? xin + v[s] : xtree + aprnet_dec_tree(v[s]);
        const ll ld = v[s] >= 0 ? ld_in : ld_coded;
#pragma unroll
        for (int k = 0; k < CH; ++k) vals[k][s] = (v[s] != APRNET_NONE && k < nch) ? src[k * ld] : (MAX ? T(-INFINITY) : T(0));
    }
    int first = 8;
    if (MAX) {
#pragma unroll
        for (int s = 7; s >= 0; --s) if (v[s] != APRNET_NONE) first = s;
    }
    T* dst = tree + (ll) c0 * ld_tree + t;
#pragma unroll
    for (int k = 0; k < CH; ++k) {
        if (k >= nch) break;
        if (MAX) {              // the first child's value, then what exceeds it (an absent child is -infinity); 0 where there is none
            T best = 0;
#pragma unroll
            for (int s = 0; s < 8; ++s)
                if (vals[k][s] > best || s == first) best = vals[k][s];
            dst[(ll) k * ld_tree] = best;
        } else {
            T s_part = 0, s_tree = 0;       // particles first, then tree children (fixed order)
#pragma unroll
            for (int s = 0; s < 8; ++s) { if (v[s] < 0) s_tree += vals[k][s]; else s_part += vals[k][s]; }
            dst[(ll) k * ld_tree] = f * (s_part + s_tree);
        }
    }
}

// channels [0, split) of the features, then those of a second tensor (a concatenation that is not written out, 1.46 of 25.6 ms of an inference batch of four); split is a
// multiple of a thread's channels
template<typename T>
struct Features {
    const T* in0; ll ld0;
    const T* in1; ll ld1;
    int split;
    // row 0 as if the channels of c0's tensor began at channel 0
    __device__ __forceinline__ const T* base(int c0) const { return c0 < split ? in0 : in1 - split * ld1; }
    __device__ __forceinline__ ll ld(int c0) const { return c0 < split ? ld0 : ld1; }
};

template<typename T, int CH, bool MAX>
__global__ void __launch_bounds__(TPB) tree_level_kernel(const int32_t* __restrict__ child, const float* __restrict__ scale, ll n_tree,
                                                         ll tb, ll te, const Features<T> in, T* tree,
                                                         ll ld_tree, int C, ll up_off, int use_up) {
    const ll t = tb + (ll) blockIdx.y * TPB + threadIdx.x;
    const int c0 = blockIdx.x * CH;
    let_next_grid_start();
    if (t < te) tree_node<T, CH, MAX, true>(child, scale, n_tree, t, in.base(c0), in.ld(c0), tree, ld_tree, c0, min(CH, C - c0), up_off, use_up);
}

// The coarse end of the tree in one launch: a cluster of blocks owns CH channels and walks the levels [0, n) of `lv` (fine to
// coarse).  A level reads what the cluster has written for the finer ones: the cluster barrier orders the blocks' global writes.  It
// costs about 2 us, so levels of at most ALONE_NODES nodes are left to the cluster's first block, between barriers of its own.
// PAIR: two feature tensors, a kernel of its own: with their choice in it, the chain of small levels took 2 to 4 us more (mean and maximum on 2 k to 10 k nodes, float64 33 to 39 us instead of 29 to 35).
struct LevelList { int n; ll begin[APRNET_MAX_LEVELS], end[APRNET_MAX_LEVELS]; int use_up[APRNET_MAX_LEVELS]; };
constexpr int COARSE_TPB = 512, CLUSTER = 8;
constexpr ll ALONE_NODES = 1024;

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;\n" ::: "memory");
}

template<typename T, int CH, bool MAX, bool PAIR>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(COARSE_TPB) tree_coarse_kernel(const int32_t* __restrict__ child, const float* __restrict__ scale, ll n_tree,
                                                                 LevelList lv, const Features<T> in, T* tree, ll ld_tree, int C, ll up_off) {
    const int c0 = (int) (blockIdx.x / CLUSTER) * CH, first = (int) (blockIdx.x % CLUSTER) * COARSE_TPB + threadIdx.x;
    const T* x = PAIR ? in.base(c0) : in.in0;
    const ll ld_x = PAIR ? in.ld(c0) : in.ld0;
    int i = 0;
    wait_for_grid_before();
    for (; i < lv.n && lv.end[i] - lv.begin[i] > ALONE_NODES; ++i) {
        for (ll t = lv.begin[i] + first; t < lv.end[i]; t += CLUSTER * COARSE_TPB)
            tree_node<T, CH, MAX>(child, scale, n_tree, t, x, ld_x, tree, ld_tree, c0, min(CH, C - c0), up_off, lv.use_up[i]);
        cluster_barrier();
    }
    if (first >= COARSE_TPB) return;
    for (; i < lv.n; ++i) {
        for (ll t = lv.begin[i] + first; t < lv.end[i]; t += COARSE_TPB)
            tree_node<T, CH, MAX>(child, scale, n_tree, t, x, ld_x, tree, ld_tree, c0, min(CH, C - c0), up_off, lv.use_up[i]);
        __syncthreads();
    }
}

// Adjoint, child-centric: entry u of `dst` (a tree node of one level, or a feature location) receives
// scale[t] * grad_tree[t] of its parent node t = parent[u].  One thread per child and CH_PER_BLOCK channels: the child
// axis is streamed (coalesced read-modify-write, one writer per entry), the parents' values come from a few cache lines
// per warp.  The parent-centric form (one thread per parent, eight scattered children) touched every sector of the
// gradient half at a time and ran at half this speed.  dst and gtree may be the same array (node levels): a level only
// reads the level above it.  A launch starts behind the one before it and has its table entries and the old values by the time the parents are there.
template<typename T, bool BEHIND = false>
__device__ __forceinline__ void tree_backward_child(const int32_t* __restrict__ parent, const float* __restrict__ scale, ll u, T* dst, ll ld_dst,
                                                    const T* gtree, ll ld_tree, int c0, int C) {
    T old[CH_PER_BLOCK];
#pragma unroll
    for (int k = 0; k < CH_PER_BLOCK; ++k) old[k] = dst[(ll) min(c0 + k, C - 1) * ld_dst + u];        // independent of the parent
    const int32_t t = parent[u];
    const T f = t < 0 ? T(0) : (T) scale[t];
    if (BEHIND) wait_for_grid_before();         // for the parents' gradients
    if (t < 0) return;
    T g[CH_PER_BLOCK];
#pragma unroll
    for (int k = 0; k < CH_PER_BLOCK; ++k) g[k] = gtree[(ll) min(c0 + k, C - 1) * ld_tree + t];
#pragma unroll
    for (int k = 0; k < CH_PER_BLOCK; ++k)
        if (c0 + k < C) dst[(ll) (c0 + k) * ld_dst + u] = old[k] + f * g[k];
}

template<typename T>
__global__ void __launch_bounds__(TPB) tree_mean_backward_children_kernel(const int32_t* __restrict__ parent, const float* __restrict__ scale,
                                                                          ll ub, ll ue, T* dst, ll ld_dst, const T* gtree, ll ld_tree, int C) {
    const ll u = ub + (ll) blockIdx.x * blockDim.x + threadIdx.x;
    let_next_grid_start();
    if (u < ue) tree_backward_child<T, true>(parent, scale, u, dst, ld_dst, gtree, ld_tree, blockIdx.y * CH_PER_BLOCK, C);
}

// the coarse tree levels of `lv` (coarse to fine) in one launch, a cluster per channel group (see tree_coarse_kernel)
template<typename T>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(COARSE_TPB) tree_mean_backward_coarse_kernel(const int32_t* __restrict__ parent, const float* __restrict__ scale,
                                                                               LevelList lv, T* gtree, ll ld_tree, int C) {
    const int c0 = (int) (blockIdx.x / CLUSTER) * CH_PER_BLOCK, first = (int) (blockIdx.x % CLUSTER) * COARSE_TPB + threadIdx.x;
    int i = 0;
    for (; i < lv.n && lv.end[i] - lv.begin[i] <= ALONE_NODES; ++i) {
        if (first < COARSE_TPB) {
            for (ll u = lv.begin[i] + first; u < lv.end[i]; u += COARSE_TPB)
                tree_backward_child<T>(parent, scale, u, gtree, ld_tree, gtree, ld_tree, c0, C);
            __syncthreads();
        }
    }
    for (; i < lv.n; ++i) {
        cluster_barrier();
        for (ll u = lv.begin[i] + first; u < lv.end[i]; u += CLUSTER * COARSE_TPB)
            tree_backward_child<T>(parent, scale, u, gtree, ld_tree, gtree, ld_tree, c0, C);
    }
}

// ---- pooling and up-sampling ---------------------------------------------------------------------------
// One thread per tree node and CH_PER_BLOCK channels.  Bound by HBM once enough loads are in flight: the loads carry no conditions (a
// child outside the volume stands for entry 0 and its value is not used) and those of several channels are requested before the first
// value is looked at; one conditional load after the other, the adjoint of the
// up-sampling took 4.9 ms in a training step on 28 M particles instead of 2.3, the max pooling 3.0 instead of 2.6.

// where child s of a node is stored: particles as they are, tree nodes from `off` on; 0 where there is none
template<typename T>
struct Children {
    ll at[8];
    unsigned particle = 0, node = 0;             // which of the eight are particles / tree nodes
    __device__ Children(const int32_t* __restrict__ child, ll n_tree, ll t, ll off) {
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const int32_t v = child[(ll) s * n_tree + t];
            at[s] = v >= 0 ? v : (v == APRNET_NONE ? 0 : aprnet_dec_tree(v) + off);
            particle |= (v >= 0 ? 1u : 0u) << s;
            node |= (v < APRNET_NONE ? 1u : 0u) << s;
        }
    }
    __device__ void load(const T* __restrict__ x, T (&v)[8]) const {
#pragma unroll
        for (int s = 0; s < 8; ++s) v[s] = x[at[s]];
    }
};

// Max pooling: tree nodes of level cml-1.  Visiting order = APR-particle children in
// slot order (dz, dx, dy), then upgraded-node children in slot order; strict '>' against an initial
// -1e17 with index 0 (pyapr/aprnet/src/maxpool.hpp:51-52,105-142).
template<typename T>
__global__ void maxpool_kernel(const int32_t* __restrict__ child, ll n_tree, ll tb, ll te, ll out_off,
                               const T* __restrict__ in, ll ld_in, T* __restrict__ out, long long* __restrict__ idx,
                               ll ld_out, int C, ll up_off) {
    constexpr int CB = 2;
    const ll t = tb + (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= te) return;
    const Children<T> ch(child, n_tree, t, up_off);
    const int c0 = blockIdx.y * CH_PER_BLOCK, c1 = min(C, c0 + CH_PER_BLOCK);
    for (int c = c0; c < c1; c += CB) {
        T v[CB][8];
#pragma unroll
        for (int k = 0; k < CB; ++k) ch.load(in + (ll) min(c + k, C - 1) * ld_in, v[k]);
#pragma unroll
        for (int k = 0; k < CB; ++k) {
            if (c + k >= c1) break;
            T best = (T) -1e17f;
            ll arg = 0;
#pragma unroll
            for (int s = 0; s < 8; ++s)
                if ((ch.particle >> s & 1) && v[k][s] > best) { best = v[k][s]; arg = ch.at[s]; }
#pragma unroll
            for (int s = 0; s < 8; ++s)
                if ((ch.node >> s & 1) && v[k][s] > best) { best = v[k][s]; arg = ch.at[s]; }
            out[(ll) (c + k) * ld_out + t + out_off] = best;
            if (idx) idx[(ll) (c + k) * ld_out + t + out_off] = arg;
        }
    }
}

template<typename T>
__global__ void maxpool_backward_kernel(const T* __restrict__ gout, const long long* __restrict__ idx, ll ld_out,
                                        T* __restrict__ gin, ll ld_in, ll nfixed, ll m, int C) {
    constexpr int CB = 4;
    const ll i = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const int c0 = blockIdx.y * CH_PER_BLOCK, c1 = min(C, c0 + CH_PER_BLOCK);
    const bool fixed = i < nfixed;
    for (int c = c0; c < c1; c += CB) {
        T g[CB];
        ll dst[CB];
#pragma unroll
        for (int k = 0; k < CB; ++k) {
            const ll at = (ll) min(c + k, C - 1) * ld_out + i;
            g[k] = gout[at];
            dst[k] = fixed ? i : idx[at];
        }
#pragma unroll
        for (int k = 0; k < CB; ++k)
            if (c + k < c1) gin[(ll) (c + k) * ld_in + dst[k]] = g[k];
    }
}

// Up-sampling: one thread per tree node t of the input's max level; its stored value sits at
// t + in_off; children are APR particles of the next level or its tree nodes (stored at + out_off).
template<typename T, bool BACKWARD>
__global__ void upsample_kernel(const int32_t* __restrict__ child, ll n_tree, ll tb, ll te, ll in_off, ll out_off,
                                const T* __restrict__ src, ll ld_src, T* __restrict__ dst, ll ld_dst, int C) {
    constexpr int CB = BACKWARD ? 2 : 4;
    const ll t = tb + (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= te) return;
    const Children<T> ch(child, n_tree, t, out_off);
    const int c0 = blockIdx.y * CH_PER_BLOCK, c1 = min(C, c0 + CH_PER_BLOCK);
    for (int c = c0; c < c1; c += CB) {
        if (!BACKWARD) {        // src = input (coarse), dst = output (fine)
            T v[CB];
#pragma unroll
            for (int k = 0; k < CB; ++k) v[k] = src[(ll) min(c + k, C - 1) * ld_src + t + in_off];
#pragma unroll
            for (int k = 0; k < CB; ++k) {
                if (c + k >= c1) break;
                T* o = dst + (ll) (c + k) * ld_dst;
#pragma unroll
                for (int s = 0; s < 8; ++s)
                    if ((ch.particle | ch.node) >> s & 1) o[ch.at[s]] = v[k];
            }
        } else {                // src = grad_output (fine), dst = grad_input (coarse)
            T v[CB][8];
#pragma unroll
            for (int k = 0; k < CB; ++k) ch.load(src + (ll) min(c + k, C - 1) * ld_src, v[k]);
#pragma unroll
            for (int k = 0; k < CB; ++k) {
                if (c + k >= c1) break;
                T s_part = 0, s_tree = 0;
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    if (ch.particle >> s & 1) s_part += v[k][s];
                    if (ch.node >> s & 1) s_tree += v[k][s];
                }
                dst[(ll) (c + k) * ld_dst + t + in_off] = s_part + s_tree;
            }
        }
    }
}

inline dim3 node_grid(ll count, int C) { return dim3((unsigned) aprnet_ceil_div(count, TPB), (unsigned) aprnet_ceil_div(C, CH_PER_BLOCK)); }

// The particles that pooling and up-sampling leave as they are: `count` leading entries of C rows.  Rows start at any multiple of the
// element, each side at its own; a warp's stores cover whole 128-byte lines, eight loads are in flight per thread.  HBM-bound: the 1.2 GB of a
// pooling (32 channels) and an up-sampling (64) of 3.5 M locations take 183 us; two strided copies by the runtime took 626.
constexpr int COPY_PER_THREAD = 8;
template<typename T>
__global__ void __launch_bounds__(TPB) copy_rows_kernel(T* __restrict__ dst, ll ld_dst, const T* __restrict__ src, ll ld_src, ll count) {
    T* d = dst + (ll) blockIdx.y * ld_dst;
    const T* s = src + (ll) blockIdx.y * ld_src;
    const int skew = (int) ((reinterpret_cast<uintptr_t>(d) & 127) / sizeof(T));
    const ll i0 = (ll) blockIdx.x * (TPB * COPY_PER_THREAD) + threadIdx.x - skew;
    T v[COPY_PER_THREAD];
#pragma unroll
    for (int k = 0; k < COPY_PER_THREAD; ++k) { const ll i = i0 + k * TPB; if (i >= 0 && i < count) v[k] = s[i]; }
#pragma unroll
    for (int k = 0; k < COPY_PER_THREAD; ++k) { const ll i = i0 + k * TPB; if (i >= 0 && i < count) d[i] = v[k]; }
}

template<typename T>
int copy_rows(T* dst, ll ld_dst, const T* src, ll ld_src, ll count, int C, cudaStream_t st) {
    if (count <= 0 || C <= 0) return APRNET_OK;
    AprnetProfScope _prof("copy_rows", st);
    for (int c0 = 0; c0 < C; c0 += 65535) {                 // grid.y holds 65535 blocks
        const dim3 grid((unsigned) aprnet_ceil_div(count + 127, TPB * COPY_PER_THREAD), (unsigned) std::min(C - c0, 65535));
        copy_rows_kernel<T><<<grid, TPB, 0, st>>>(dst + c0 * ld_dst, ld_dst, src + c0 * ld_src, ld_src, count);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

// Fills the tree bottom-up.  The coarsest levels, as long as they have at most COARSE_NODES nodes each, share one launch: a launch
// costs the host 4 us, which is what small structures wait for, and the device about 2 us; inside the shared one a level costs about
// 2 us per CLUSTER * COARSE_TPB nodes.  Every finer level is a launch of its own, also one with few nodes: where fine cells are
// rare, a level below it has many, and one cluster would walk them with 8 of the SMs.
constexpr ll COARSE_NODES = 2 * CLUSTER * COARSE_TPB;

// last level of the shared launch (level_min - 2: none)
int last_coarse_level(const LevelMeta& m, int cml) {
    int l = m.level_min - 1;
    while (l <= cml - 1 && m.tlvl_begin[l + 1] - m.tlvl_begin[l] <= COARSE_NODES) ++l;
    return l - 1;
}

template<typename T, bool MAX>
int fill_tree(const aprnet_apr* a, int dl, int C, const Features<T>& in, T* tree, ll ld_tree, const char* pname, cudaStream_t st) {
    constexpr int CH = 4;
    const LevelMeta& m = a->meta;
    const int cml = a->cml(dl);
    const ll up = (dl > 0) ? a->tree_offset(cml) : 0;
    const unsigned gx = (unsigned) aprnet_ceil_div(C, CH);
    LevelList coarse;
    coarse.n = 0;
    const int last = last_coarse_level(m, cml);
    bool behind = false;
    for (int lp = cml - 1; lp >= m.level_min - 1; --lp) {
        const ll tb = m.tlvl_begin[lp], te = m.tlvl_begin[lp + 1];
        if (te <= tb) continue;
        const int use_up = (dl > 0 && lp + 1 == cml) ? 1 : 0;
        if (lp <= last) {
            coarse.begin[coarse.n] = tb; coarse.end[coarse.n] = te; coarse.use_up[coarse.n] = use_up;
            ++coarse.n;
            continue;
        }
        for (ll b = tb; b < te; b += 65535ll * TPB) {              // grid.y holds 65535 blocks
            AprnetProfScope _prof(pname, st);
            const ll e = std::min(te, b + 65535ll * TPB);
            aprnet_launch(behind, tree_level_kernel<T, CH, MAX>, dim3(gx, (unsigned) aprnet_ceil_div(e - b, TPB)), TPB, 0, st, a->child, a->tree_scale, a->n_tree, b, e, in,
                          tree, ld_tree, C, up, use_up);
            behind = true;
        }
    }
    if (coarse.n > 0) {
        AprnetProfScope _prof(pname, st);
        auto kern = in.split < C ? tree_coarse_kernel<T, CH, MAX, true> : tree_coarse_kernel<T, CH, MAX, false>;
        aprnet_launch(behind, kern, gx * CLUSTER, COARSE_TPB, 0, st, a->child, a->tree_scale, a->n_tree, coarse, in, tree, ld_tree, C, up);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

template<typename T>
inline Features<T> one_tensor(const T* in, ll ld, int C) { return Features<T>{in, ld, in, ld, C}; }

template<typename T>
int fill_tree_mean_bwd(const aprnet_apr* a, int dl, int C, T* gin, ll ld_in, T* gtree, ll ld_tree, cudaStream_t st) {
    const LevelMeta& m = a->meta;
    const int cml = a->cml(dl);
    const int32_t* node_parent = aprnet_node_parent_table(a, st);
    const int32_t* loc_parent = aprnet_loc_parent_table(a, dl, st);
    if (!node_parent || !loc_parent) return APRNET_ERR_CUDA;
    // tree nodes, coarse to fine: level l receives from level l - 1, whose gradient is complete by then
    LevelList coarse;
    coarse.n = 0;
    int l = m.level_min;
    for (; l <= cml - 1 && m.tlvl_begin[l + 1] - m.tlvl_begin[l] <= COARSE_NODES; ++l)
        if (m.tlvl_begin[l + 1] > m.tlvl_begin[l]) { coarse.begin[coarse.n] = m.tlvl_begin[l]; coarse.end[coarse.n] = m.tlvl_begin[l + 1]; ++coarse.n; }
    if (coarse.n > 0) {
        AprnetProfScope _prof("tree_mean_bwd", st);
        aprnet_launch(false, tree_mean_backward_coarse_kernel<T>, (unsigned) aprnet_ceil_div(C, CH_PER_BLOCK) * CLUSTER, COARSE_TPB, 0, st, node_parent, a->tree_scale, coarse, gtree, ld_tree, C);
    }
    bool behind = coarse.n > 0;
    for (; l <= cml - 1; ++l) {
        const ll ub = m.tlvl_begin[l], ue = m.tlvl_begin[l + 1];
        if (ue <= ub) continue;
        AprnetProfScope _prof("tree_mean_bwd", st);
        aprnet_launch(behind, tree_mean_backward_children_kernel<T>, node_grid(ue - ub, C), TPB, 0, st, node_parent, a->tree_scale, ub, ue, gtree, ld_tree, gtree, ld_tree, C);
        behind = true;
    }
    // then every feature location (particles of all levels, upgraded nodes) from its parent node
    const ll n = a->number_parts(dl);
    if (n > 0) {
        AprnetProfScope _prof("tree_mean_bwd", st);
        aprnet_launch(behind, tree_mean_backward_children_kernel<T>, node_grid(n, C), TPB, 0, st, loc_parent, a->tree_scale, 0, n, gin, ld_in, gtree, ld_tree, C);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

template<typename T>
int maxpool_fwd(const aprnet_apr* a, int dl, int C, const T* in, ll ld_in, T* out, long long* idx, ll ld_out, cudaStream_t st) {
    const LevelMeta& m = a->meta;
    const int cml = a->cml(dl);
    const ll ncopy = m.lvl_begin[cml];                       // particles of levels <= cml-1
    int rc = copy_rows(out, ld_out, in, ld_in, ncopy, C, st);
    if (rc) return rc;
    const ll tb = m.tlvl_begin[cml - 1], te = m.tlvl_begin[cml];
    if (te > tb) {
        const ll up = (dl > 0) ? a->tree_offset(cml) : 0;
        { AprnetProfScope _prof("maxpool_fwd", st);
        maxpool_kernel<T><<<node_grid(te - tb, C), TPB, 0, st>>>(a->child, a->n_tree, tb, te, a->tree_offset(cml - 1), in,
                                                                  ld_in, out, idx, ld_out, C, up);
        }
        APRNET_LAUNCH_CHECK();
    }
    return APRNET_OK;
}

template<typename T>
int maxpool_bwd(const aprnet_apr* a, int dl, int C, const T* gout, const long long* idx, ll ld_out, T* gin, ll ld_in, cudaStream_t st) {
    const ll mcount = a->number_parts(dl + 1);
    const ll nfixed = a->meta.lvl_begin[a->cml(dl)];
    if (mcount > 0) {
        { AprnetProfScope _prof("maxpool_bwd", st);
        maxpool_backward_kernel<T><<<node_grid(mcount, C), TPB, 0, st>>>(gout, idx, ld_out, gin, ld_in, nfixed, mcount, C);
        }
        APRNET_LAUNCH_CHECK();
    }
    return APRNET_OK;
}

template<typename T, bool BACKWARD>
int upsample_impl(const aprnet_apr* a, int dl, int C, const T* src, ll ld_src, T* dst, ll ld_dst, cudaStream_t st) {
    const LevelMeta& m = a->meta;
    const int in_max = a->cml(dl), out_max = in_max + 1;
    const ll ncopy = m.lvl_begin[in_max + 1];                // particles of levels <= in_max
    int rc = copy_rows(dst, ld_dst, src, ld_src, ncopy, C, st);
    if (rc) return rc;
    const ll tb = m.tlvl_begin[in_max], te = m.tlvl_begin[in_max + 1];
    if (te > tb) {
        const ll out_off = (out_max <= m.level_max - 1) ? a->tree_offset(out_max) : 0;
        { AprnetProfScope _prof("upsample", st);
        upsample_kernel<T, BACKWARD><<<node_grid(te - tb, C), TPB, 0, st>>>(a->child, a->n_tree, tb, te, a->tree_offset(in_max),
                                                                             out_off, src, ld_src, dst, ld_dst, C);
        }
        APRNET_LAUNCH_CHECK();
    }
    return APRNET_OK;
}

} // namespace

#define DISPATCH(dtype, CALL_F, CALL_D)                                                   \
    switch (dtype) {                                                                      \
        case APRNET_F32: return CALL_F;                                                   \
        case APRNET_F64: return CALL_D;                                                   \
        default: aprnet_set_error("%s: unknown dtype %d", __func__, dtype); return APRNET_ERR_ARG; \
    }

// tree means of the concatenation of two float32 tensors of c0 and C - c0 channels (c0 a multiple of four)
int aprnet_fill_tree_mean_pair(const aprnet_apr* a, int dl, int C, const float* in0, ll ld0, int c0, const float* in1, ll ld1, float* tree, ll ld_tree, cudaStream_t st) {
    return fill_tree<float, false>(a, dl, C, Features<float>{in0, ld0, in1, ld1, c0}, tree, ld_tree, "tree_mean_fwd", st);
}

extern "C" int aprnet_fill_tree_mean_forward(const aprnet_apr* a, int dl, int dtype, int C, const void* in, int64_t ld_in,
                                             void* tree, int64_t ld_tree, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && in && tree && C > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_tree >= a->tree_size(dl), "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    DISPATCH(dtype, (fill_tree<float, false>(a, dl, C, one_tensor((const float*) in, ld_in, C), (float*) tree, ld_tree, "tree_mean_fwd", st)),
             (fill_tree<double, false>(a, dl, C, one_tensor((const double*) in, ld_in, C), (double*) tree, ld_tree, "tree_mean_fwd", st)));
}

extern "C" int aprnet_fill_tree_mean_full(const aprnet_apr* a, int dtype, int C, const void* in, int64_t ld_in, void* tree,
                                          int64_t ld_tree, void* stream) {
    return aprnet_fill_tree_mean_forward(a, 0, dtype, C, in, ld_in, tree, ld_tree, stream);
}

extern "C" int aprnet_fill_tree_mean_backward(const aprnet_apr* a, int dl, int dtype, int C, void* gin, int64_t ld_in,
                                              void* gtree, int64_t ld_tree, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && gin && gtree && C > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_tree >= a->tree_size(dl), "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    DISPATCH(dtype, fill_tree_mean_bwd<float>(a, dl, C, (float*) gin, ld_in, (float*) gtree, ld_tree, st),
             fill_tree_mean_bwd<double>(a, dl, C, (double*) gin, ld_in, (double*) gtree, ld_tree, st));
}

extern "C" int aprnet_fill_tree_max(const aprnet_apr* a, int dtype, int C, const void* in, int64_t ld_in, void* tree,
                                    int64_t ld_tree, void* stream) {
    APRNET_ARG_CHECK(a && in && tree && C > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->n_particles && ld_tree >= a->n_tree, "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    DISPATCH(dtype, (fill_tree<float, true>(a, 0, C, one_tensor((const float*) in, ld_in, C), (float*) tree, ld_tree, "tree_max", st)),
             (fill_tree<double, true>(a, 0, C, one_tensor((const double*) in, ld_in, C), (double*) tree, ld_tree, "tree_max", st)));
}

extern "C" int aprnet_maxpool_forward(const aprnet_apr* a, int dl, int dtype, int C, const void* in, int64_t ld_in,
                                      void* out, int64_t* idx, int64_t ld_out, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && a->valid_dl(dl + 1) && in && out && idx && C > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl + 1), "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    DISPATCH(dtype, maxpool_fwd<float>(a, dl, C, (const float*) in, ld_in, (float*) out, (long long*) idx, ld_out, st),
             maxpool_fwd<double>(a, dl, C, (const double*) in, ld_in, (double*) out, (long long*) idx, ld_out, st));
}

// the same without indices, where no backward pass follows
extern "C" int aprnet_maxpool_forward_values(const aprnet_apr* a, int dl, int dtype, int C, const void* in, int64_t ld_in, void* out, int64_t ld_out, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && a->valid_dl(dl + 1) && in && out && C > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl + 1), "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    DISPATCH(dtype, maxpool_fwd<float>(a, dl, C, (const float*) in, ld_in, (float*) out, nullptr, ld_out, st),
             maxpool_fwd<double>(a, dl, C, (const double*) in, ld_in, (double*) out, nullptr, ld_out, st));
}

extern "C" int aprnet_maxpool_backward(const aprnet_apr* a, int dl, int dtype, int C, const void* gout, const int64_t* idx,
                                       int64_t ld_out, void* gin, int64_t ld_in, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && a->valid_dl(dl + 1) && gout && gin && idx && C > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl + 1), "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    DISPATCH(dtype, maxpool_bwd<float>(a, dl, C, (const float*) gout, (const long long*) idx, ld_out, (float*) gin, ld_in, st),
             maxpool_bwd<double>(a, dl, C, (const double*) gout, (const long long*) idx, ld_out, (double*) gin, ld_in, st));
}

extern "C" int aprnet_upsample_forward(const aprnet_apr* a, int dl, int dtype, int C, const void* in, int64_t ld_in, void* out,
                                       int64_t ld_out, void* stream) {
    APRNET_ARG_CHECK(a && dl > 0 && a->valid_dl(dl) && in && out && C > 0, "bad argument (level_delta must be > 0)");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl - 1), "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    DISPATCH(dtype, (upsample_impl<float, false>(a, dl, C, (const float*) in, ld_in, (float*) out, ld_out, st)),
             (upsample_impl<double, false>(a, dl, C, (const double*) in, ld_in, (double*) out, ld_out, st)));
}

extern "C" int aprnet_upsample_backward(const aprnet_apr* a, int dl, int dtype, int C, const void* gout, int64_t ld_out,
                                        void* gin, int64_t ld_in, void* stream) {
    APRNET_ARG_CHECK(a && dl > 0 && a->valid_dl(dl) && gout && gin && C > 0, "bad argument (level_delta must be > 0)");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl - 1), "leading dimension too small");
    cudaStream_t st = (cudaStream_t) stream;
    DISPATCH(dtype, (upsample_impl<float, true>(a, dl, C, (const float*) gout, ld_out, (float*) gin, ld_in, st)),
             (upsample_impl<double, true>(a, dl, C, (const double*) gout, ld_out, (double*) gin, ld_in, st)));
}
