// Cross-level part of the 3x3x3 input gradient without atomics.
//
// A tap of an output location p whose source is a coarser particle or a tree node ("cross-level edge")
// contributes W[tap]^T dO[p] to that source.  The reference scatters these with atomicAdd
// (pyapr/aprnet/cuda/src/conv333_gpu_backward.cu:184-192,417,643).  Here the edges of a level_delta are
// enumerated once (cached in the APR handle) and grouped by (target, tap): all edges of one group meet
// the same weight matrix (their locations lie on one level), so their dO rows are summed first
// ("virtual row", pass 1: a segmented sum in ascending location order) and the contraction becomes an
// ordinary 27-tap gather GEMM over the targets that have edges (pass 2, on the tensor cores), whose
// result is added to the gradient of the particle / tree node by exactly one thread.  Both passes are
// deterministic, and the work is proportional to the number of (target, tap) groups, not edges.
#include "apr_device.cuh"
#include <cub/cub.cuh>
#include <cuda_bf16.h>
#include <algorithm>
#include <cstring>

namespace {

typedef long long ll;

struct LevelRanges { int n; ll begin[APRNET_MAX_LEVELS], end[APRNET_MAX_LEVELS]; };

// flag[f] = 1 when entry f = tap * N + p of the neighbour table is a cross-level source
__global__ void edge_flag_kernel(const int32_t* __restrict__ nbr, ll N, LevelRanges lr, int32_t* __restrict__ flag) {
    const ll f = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (f > 27 * N) return;
    int32_t v = 0;
    if (f < 27 * N) {
        const ll p = f % N;
        const int32_t q = nbr[f];
        if (q < APRNET_NONE) v = 1;
        else if (q >= 0) {
            ll lo = 0;
            for (int i = 0; i < lr.n; ++i) if (p >= lr.begin[i] && p < lr.end[i]) lo = lr.begin[i];
            v = q < lo;
        }
    }
    flag[f] = v;
}

__global__ void edge_emit_kernel(const int32_t* __restrict__ nbr, ll N, const int32_t* __restrict__ scan,
                                 int32_t* __restrict__ src, int32_t* __restrict__ tgt, int32_t* __restrict__ count) {
    const ll f = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= 27 * N) return;
    const int32_t e = scan[f];
    if (scan[f + 1] == e) return;
    const int32_t q = nbr[f];
    const int32_t t = q >= 0 ? q : (int32_t) (N + aprnet_dec_tree(q));
    src[e] = (int32_t) (f % N);
    tgt[e] = t;
    atomicAdd(count + t, 1);
}

__global__ void edge_fill_kernel(const int32_t* __restrict__ tgt, ll E, int32_t* __restrict__ cursor, int32_t* __restrict__ tgt_edge) {
    const ll e = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    tgt_edge[atomicAdd(cursor + tgt[e], 1)] = (int32_t) e;
}

// ascending edge order inside every target's list (the fill order above depends on scheduling)
__global__ void edge_sort_kernel(const int32_t* __restrict__ ptr, ll n_targets, int32_t* __restrict__ tgt_edge, int32_t* __restrict__ is_active) {
    const ll t = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (t > n_targets) return;
    if (t == n_targets) { is_active[t] = 0; return; }
    const int32_t b = ptr[t], e = ptr[t + 1];
    is_active[t] = e > b;
    for (int32_t i = b + 1; i < e; ++i) {
        const int32_t v = tgt_edge[i];
        int32_t j = i - 1;
        while (j >= b && tgt_edge[j] > v) { tgt_edge[j + 1] = tgt_edge[j]; --j; }
        tgt_edge[j + 1] = v;
    }
}

__global__ void edge_compact_active_kernel(const int32_t* __restrict__ pos, ll n_targets, int32_t* __restrict__ active) {
    const ll t = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_targets) return;
    if (pos[t + 1] != pos[t]) active[pos[t]] = (int32_t) t;
}

struct TapBegin { int32_t b[28]; };      // first edge id of every tap (edge ids are tap-major)

// virtual rows of one active target = runs of equal tap, of more than one edge, in its ascending edge list
template<typename F>
__device__ __forceinline__ void for_each_run(const int32_t* __restrict__ tgt_edge, int begin, int end, const TapBegin& tb, F f) {
    int tap = 0;
    for (int i = begin; i < end;) {
        while (tgt_edge[i] >= tb.b[tap + 1]) ++tap;
        int j = i + 1;
        while (j < end && tgt_edge[j] < tb.b[tap + 1]) ++j;
        f(tap, i, j);
        i = j;
    }
}

__global__ void vrow_count_kernel(const int32_t* __restrict__ active, ll n_active, const int32_t* __restrict__ ptr,
                                  const int32_t* __restrict__ tgt_edge, TapBegin tb, int32_t* __restrict__ nruns, int32_t* __restrict__ nedges) {
    const ll a = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (a > n_active) return;
    int runs = 0, edges = 0;
    if (a < n_active) {
        const int t = active[a];
        for_each_run(tgt_edge, ptr[t], ptr[t + 1], tb, [&](int, int i, int j) { if (j - i > 1) { ++runs; edges += j - i; } });
    }
    nruns[a] = runs;
    nedges[a] = edges;
}

__global__ void vrow_fill_kernel(const int32_t* __restrict__ active, ll n_active, const int32_t* __restrict__ ptr,
                                 const int32_t* __restrict__ tgt_edge, const int32_t* __restrict__ src, TapBegin tb,
                                 const int32_t* __restrict__ vfirst, const int32_t* __restrict__ efirst, int32_t* __restrict__ vstart,
                                 int32_t* __restrict__ vnbr, int32_t* __restrict__ vsrc) {
    const ll a = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n_active) return;
    if (a == 0) vstart[vfirst[n_active]] = efirst[n_active];
    const int t = active[a];
    int32_t v = vfirst[a], at = efirst[a];
    for_each_run(tgt_edge, ptr[t], ptr[t + 1], tb, [&](int tap, int i, int j) {
        if (j - i == 1) { vnbr[(ll) tap * n_active + a] = aprnet_enc_tree(src[tgt_edge[i]]); return; }
        vstart[v] = at;
        vnbr[(ll) tap * n_active + a] = v++;
        for (; i < j; ++i) vsrc[at++] = src[tgt_edge[i]];
    });
}

// out[k] = first index i of sorted[0, n) with sorted[i] >= key[k]; value (may be null): sorted[out[k]], readable up to sorted[n]
__global__ void lower_bound_kernel(const int32_t* __restrict__ sorted, ll n, const ll* __restrict__ key, int nkeys, ll* __restrict__ out, ll* __restrict__ value) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nkeys) return;
    ll lo = 0, hi = n;
    while (lo < hi) { const ll m = (lo + hi) >> 1; if ((ll) sorted[m] < key[k]) lo = m + 1; else hi = m; }
    out[k] = lo;
    if (value) value[k] = sorted[lo];
}

// pass 1: thread = (VPT consecutive virtual rows, 8-channel chunk); sums the dO rows of each row's locations in
// ascending order (fp32) and writes the bf16 row v - v0 of the workspace.  The three
// dependent accesses (row starts -> source locations -> dO rows) are each requested for all VPT rows and up to four
// locations per row before any is used (runs are 2-4 locations long; longer ones continue in a loop).
// What bounds it is the issue of instructions (57 % of the slots with 41 % of the warps active, DRAM at 20 %), so a block divides its
// threads among rows and chunks in 32 bits and adds channels in pairs.  Before, with a 64-bit division per thread and single additions: 242 us
// for the 32 channels of 3.5 M locations, 181 us for 64 channels at level delta 1 (1.86 M); now 197 and 147.
constexpr int VROW_VPT = 2;          // measured: 2 rows per thread 20 % faster than 1, 4 slower (registers)
constexpr int VROW_CHUNKS = 32;      // chunks of a row that a block takes at most; the others are another blockIdx.y

__device__ __forceinline__ void add_pair(unsigned long long& acc, uint32_t bf16x2) {       // acc.{x,y} += the two values, which are exact in fp32
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(bf16x2 << 16), "r"(bf16x2 & 0xffff0000u));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(v));
}

template<int VPT>
__global__ void __launch_bounds__(256) vrow_reduce_kernel(const int32_t* __restrict__ vstart, const int32_t* __restrict__ vsrc, ll v0, ll v1,
                                                          const __nv_bfloat16* __restrict__ grows, int gpad, __nv_bfloat16* __restrict__ out) {
    const unsigned nch = min((gpad >> 3) - (int) blockIdx.y * VROW_CHUNKS, VROW_CHUNKS), rows = 256 / nch, r = threadIdx.x / nch;
    const ll vb = v0 + ((ll) blockIdx.x * rows + r) * VPT;
    if (r >= rows || vb >= v1) return;
    const int c = blockIdx.y * VROW_CHUNKS + threadIdx.x - r * nch;
    int s[VPT + 1];
#pragma unroll
    for (int u = 0; u <= VPT; ++u) s[u] = __ldg(vstart + min(vb + u, v1));
    int32_t src[VPT][4];
#pragma unroll
    for (int u = 0; u < VPT; ++u)
#pragma unroll
        for (int k = 0; k < 4; ++k) src[u][k] = s[u] + k < s[u + 1] ? __ldg(vsrc + s[u] + k) : -1;
    uint4 q[VPT][4];
#pragma unroll
    for (int u = 0; u < VPT; ++u)
#pragma unroll
        for (int k = 0; k < 4; ++k)
            q[u][k] = src[u][k] >= 0 ? __ldg(reinterpret_cast<const uint4*>(grows + (ll) src[u][k] * gpad + c * 8)) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
        if (vb + u >= v1) break;
        unsigned long long acc[4] = {0ull, 0ull, 0ull, 0ull};
        auto add = [&](const uint4& w) { add_pair(acc[0], w.x); add_pair(acc[1], w.y); add_pair(acc[2], w.z); add_pair(acc[3], w.w); };
#pragma unroll
        for (int k = 0; k < 4; ++k) add(q[u][k]);              // ascending location order (absent entries add zeros)
        for (int i = s[u] + 4; i < s[u + 1]; ++i)
            add(__ldg(reinterpret_cast<const uint4*>(grows + (ll) __ldg(vsrc + i) * gpad + c * 8)));
        __nv_bfloat162 o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float2 f;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(acc[k]));
            o[k] = __floats2bfloat162_rn(f.x, f.y);
        }
        *reinterpret_cast<uint4*>(out + (vb + u - v0) * gpad + c * 8) = *reinterpret_cast<const uint4*>(o);
    }
}

template<typename T>
int dev_alloc(T** p, size_t n, long long* bytes, cudaStream_t st) {
    const int rc = aprnet_pool_alloc((void**) p, std::max<size_t>(n, 1) * sizeof(T), st);
    if (!rc && bytes) *bytes += (long long) (std::max<size_t>(n, 1) * sizeof(T));
    return rc;
}

} // namespace

void aprnet_free_edge_plan(EdgePlan& ep, cudaStream_t st) {
    aprnet_pool_free(ep.vsrc, st); aprnet_pool_free(ep.vstart, st); aprnet_pool_free(ep.active, st); aprnet_pool_free(ep.vnbr, st);
    ep = EdgePlan();
}

static int build_edge_plan(aprnet_apr* a, int dl, const AprPlan* plan, EdgePlan& ep, cudaStream_t st) {
    const ll N = plan->n, T = plan->tree_size, NT = N + T;
    const ll F = 27 * N;
    if (F + 1 >= (1ll << 31)) { aprnet_set_error("edge plan: neighbour table too large for 32-bit edge ids"); return APRNET_ERR_UNSUPPORTED; }
    const std::vector<Segment> segs = aprnet_segments(a, dl, 1, false);
    LevelRanges lr;
    lr.n = (int) segs.size();
    for (int i = 0; i < lr.n; ++i) { lr.begin[i] = segs[i].begin; lr.end[i] = segs[i].end; }

    // temporaries: flags / scan, per-edge source and target, per-target lists
    int32_t *scan = nullptr, *src = nullptr, *tgt = nullptr, *count = nullptr, *tgt_ptr = nullptr, *tgt_edge = nullptr, *vfirst = nullptr, *efirst = nullptr;
    ll *keys = nullptr, *found = nullptr;
    void* temp = nullptr;
    int rc = APRNET_OK;
    auto cleanup = [&]() { void* all[] = {scan, src, tgt, count, tgt_ptr, tgt_edge, vfirst, efirst, keys, found, temp}; for (void* p : all) aprnet_pool_free(p, st); };
#define EP_ALLOC(p, n) do { if ((rc = dev_alloc(&(p), (size_t) (n), nullptr, st))) { cleanup(); return rc; } } while (0)
#define EP_CHECK(expr) do { cudaError_t _e = (expr); if (_e != cudaSuccess) { aprnet_set_error("%s failed: %s", #expr, cudaGetErrorString(_e)); cleanup(); return APRNET_ERR_CUDA; } } while (0)

    EP_ALLOC(scan, F + 1);
    edge_flag_kernel<<<aprnet_ceil_div(F + 1, 256), 256, 0, st>>>(plan->nbr, N, lr, scan);
    size_t temp_bytes = 0, temp2 = 0;
    EP_CHECK(cub::DeviceScan::ExclusiveSum(nullptr, temp_bytes, scan, scan, (int) (F + 1), st));
    EP_CHECK(cub::DeviceScan::ExclusiveSum(nullptr, temp2, scan, scan, (int) (NT + 2), st));
    temp_bytes = std::max(temp_bytes, temp2);
    if ((rc = aprnet_pool_alloc(&temp, std::max<size_t>(temp_bytes, 1), st))) { cleanup(); return rc; }
    EP_CHECK(cub::DeviceScan::ExclusiveSum(temp, temp_bytes, scan, scan, (int) (F + 1), st));

    // first edge id of every tap
    TapBegin tb;
    if (N > 0) EP_CHECK(cudaMemcpy2DAsync(tb.b, sizeof(int32_t), scan, (size_t) N * sizeof(int32_t), sizeof(int32_t), 28, cudaMemcpyDeviceToHost, st));
    else memset(&tb, 0, sizeof(tb));
    EP_CHECK(cudaStreamSynchronize(st));
    const ll E = tb.b[27];
    ep.n_edges = E; ep.n_targets = NT;

    // per-edge source and target, per-target ascending edge lists, active targets
    EP_ALLOC(src, E);
    EP_ALLOC(tgt, E);
    EP_ALLOC(tgt_edge, E);
    EP_ALLOC(tgt_ptr, NT + 1);
    EP_ALLOC(count, NT + 1);
    EP_CHECK(cudaMemsetAsync(count, 0, (size_t) (NT + 1) * sizeof(int32_t), st));
    edge_emit_kernel<<<aprnet_ceil_div(F, 256), 256, 0, st>>>(plan->nbr, N, scan, src, tgt, count);
    EP_CHECK(cub::DeviceScan::ExclusiveSum(temp, temp_bytes, count, tgt_ptr, (int) (NT + 1), st));
    EP_CHECK(cudaMemcpyAsync(count, tgt_ptr, (size_t) (NT + 1) * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));   // cursors
    if (E) edge_fill_kernel<<<aprnet_ceil_div(E, 256), 256, 0, st>>>(tgt, E, count, tgt_edge);
    edge_sort_kernel<<<aprnet_ceil_div(NT + 1, 128), 128, 0, st>>>(tgt_ptr, NT, tgt_edge, count);     // also flags active targets in `count`
    EP_CHECK(cub::DeviceScan::ExclusiveSum(temp, temp_bytes, count, count, (int) (NT + 1), st));
    int32_t n_active = 0;
    EP_CHECK(cudaMemcpyAsync(&n_active, count + NT, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    EP_CHECK(cudaStreamSynchronize(st));
    ep.n_active = n_active;
    if ((rc = dev_alloc(&ep.active, (size_t) n_active, &a->device_bytes, st))) { cleanup(); return rc; }
    if (NT) edge_compact_active_kernel<<<aprnet_ceil_div(NT, 256), 256, 0, st>>>(count, NT, ep.active);
    aprnet_pool_free(scan, st); scan = nullptr;
    aprnet_pool_free(tgt, st); tgt = nullptr;

    // virtual rows: runs of equal tap in every active target's list
    EP_ALLOC(vfirst, n_active + 1);
    EP_ALLOC(efirst, n_active + 1);
    vrow_count_kernel<<<aprnet_ceil_div((ll) n_active + 1, 128), 128, 0, st>>>(ep.active, n_active, tgt_ptr, tgt_edge, tb, vfirst, efirst);
    EP_CHECK(cub::DeviceScan::ExclusiveSum(temp, temp_bytes, vfirst, vfirst, n_active + 1, st));
    EP_CHECK(cub::DeviceScan::ExclusiveSum(temp, temp_bytes, efirst, efirst, n_active + 1, st));
    int32_t n_vrows = 0, n_summed = 0;
    EP_CHECK(cudaMemcpyAsync(&n_vrows, vfirst + n_active, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    EP_CHECK(cudaMemcpyAsync(&n_summed, efirst + n_active, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    EP_CHECK(cudaStreamSynchronize(st));
    ep.n_vrows = n_vrows;
    if ((rc = dev_alloc(&ep.vsrc, (size_t) n_summed, &a->device_bytes, st)) || (rc = dev_alloc(&ep.vstart, (size_t) n_vrows + 1, &a->device_bytes, st)) ||
        (rc = dev_alloc(&ep.vnbr, (size_t) 27 * std::max(n_active, 1), &a->device_bytes, st))) { cleanup(); return rc; }
    EP_CHECK(cudaMemsetAsync(ep.vnbr, 0xFF, (size_t) 27 * std::max(n_active, 1) * sizeof(int32_t), st));       // APRNET_NONE
    EP_CHECK(cudaMemsetAsync(ep.vstart, 0, ((size_t) n_vrows + 1) * sizeof(int32_t), st));
    if (n_active) vrow_fill_kernel<<<aprnet_ceil_div(n_active, 128), 128, 0, st>>>(ep.active, n_active, tgt_ptr, tgt_edge, src, tb, vfirst, efirst,
                                                                                  ep.vstart, ep.vnbr, ep.vsrc);

    // ranges of active[] by level of the locations their edges come from, and the chunk map
    const int cml = a->cml(dl);
    std::vector<ll> key_h;
    std::vector<int> key_level;
    for (int l = a->meta.level_min; l <= cml; ++l) {        // particle targets of level l <- locations of level l + 1
        key_h.push_back(a->meta.lvl_begin[l]); key_level.push_back(l + 1);
    }
    for (int l = a->meta.level_min - 1; l <= cml - 1; ++l) {    // tree targets of level l <- locations of level l
        key_h.push_back(N + a->meta.tlvl_begin[l]); key_level.push_back(l);
    }
    key_h.push_back(NT); key_level.push_back(-1);
    const int nkeys = (int) key_h.size();
    const int nchunk = (int) (n_vrows / APRNET_VROW_GRANULE) + 1, nk = std::max(nkeys, nchunk + 1);
    EP_ALLOC(keys, nk);
    EP_ALLOC(found, 2 * nk);                                  // indices, values
    std::vector<ll> found_h(2 * nk);
    EP_CHECK(cudaMemcpyAsync(keys, key_h.data(), nkeys * sizeof(ll), cudaMemcpyHostToDevice, st));
    lower_bound_kernel<<<1, 64, 0, st>>>(ep.active, n_active, keys, nkeys, found, nullptr);
    EP_CHECK(cudaMemcpyAsync(found_h.data(), found, nkeys * sizeof(ll), cudaMemcpyDeviceToHost, st));
    EP_CHECK(cudaStreamSynchronize(st));
    ep.segs.clear();
    for (int k = 0; k + 1 < nkeys; ++k) {
        ActiveSeg sg; sg.begin = found_h[k]; sg.end = found_h[k + 1]; sg.location_level = key_level[k];
        if (sg.end > sg.begin && sg.location_level >= a->meta.level_min && sg.location_level <= cml) ep.segs.push_back(sg);
        else if (sg.end > sg.begin) { aprnet_set_error("edge plan: edges from level %d outside [%d, %d]", sg.location_level, a->meta.level_min, cml); cleanup(); return APRNET_ERR_CUDA; }
    }
    std::vector<ll> ckey(nchunk + 1);
    for (int k = 0; k < nchunk; ++k) ckey[k] = (ll) k * APRNET_VROW_GRANULE;
    ckey[nchunk] = (ll) n_vrows + 1;        // beyond the last value: maps to n_active
    EP_CHECK(cudaMemcpyAsync(keys, ckey.data(), (nchunk + 1) * sizeof(ll), cudaMemcpyHostToDevice, st));
    lower_bound_kernel<<<aprnet_ceil_div(nchunk + 1, 64), 64, 0, st>>>(vfirst, n_active, keys, nchunk + 1, found, found + nk);
    EP_CHECK(cudaMemcpyAsync(found_h.data(), found, 2 * nk * sizeof(ll), cudaMemcpyDeviceToHost, st));
    EP_CHECK(cudaStreamSynchronize(st));
    ep.chunk_a.clear(); ep.chunk_v.clear();
    for (int k = 0; k <= nchunk; ++k) {
        const ll ca = found_h[k];
        if (!ep.chunk_a.empty() && ep.chunk_a.back() == ca) continue;
        ep.chunk_a.push_back(ca); ep.chunk_v.push_back(found_h[nk + k]);
    }
    if (ep.chunk_a.back() != n_active) { ep.chunk_a.push_back(n_active); ep.chunk_v.push_back(n_vrows); }
    EP_CHECK(cudaGetLastError());
    EP_CHECK(cudaStreamSynchronize(st));
#undef EP_CHECK
#undef EP_ALLOC
    cleanup();
    return APRNET_OK;
}

EdgePlan* aprnet_get_edge_plan(aprnet_apr* a, int dl, cudaStream_t st) {
    auto it = a->edge_plans.find(dl);
    if (it != a->edge_plans.end()) return &it->second;
    const AprPlan* plan = aprnet_get_plan(a, dl, st);
    if (!plan) return nullptr;
    EdgePlan ep;
    if (build_edge_plan(a, dl, plan, ep, st) != APRNET_OK) { aprnet_free_edge_plan(ep, st); return nullptr; }
    auto res = a->edge_plans.emplace(dl, ep);
    return &res.first->second;
}

// Builds (once; cached) the cross-level edge lists of a level delta.  Allocates; call it up front.
extern "C" int aprnet_edge_plan_build(aprnet_apr* a, int dl, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl), "bad handle or level_delta");
    APRNET_DEVICE_CHECK(a);
    return aprnet_get_edge_plan(a, dl, (cudaStream_t) stream) ? APRNET_OK : APRNET_ERR_CUDA;
}

extern "C" int64_t aprnet_edge_workspace_bytes(const aprnet_apr* a, int dl, int cout) {
    if (!a || !a->valid_dl(dl)) return -1;
    const auto it = a->edge_plans.find(dl);
    return (int64_t) aprnet_vrow_workspace_bytes(it != a->edge_plans.end() ? it->second.n_vrows : 27 * a->number_parts(dl), (ll) aprnet_tc_pad(cout) * 2);
}

// Cross-level part of the input gradient (added to grad_input, which holds the same-level part, and to
// grad_tree, which the call zero-fills) followed by the tree adjoint.  packed_grad_output_rows:
// channels-last bf16 dO rows; weights fp32 (slots, Cout, Cin, 27); wp_ws: the packed transposed
// weights; edge_ws: aprnet_edge_workspace_bytes() bytes.
int aprnet_cross_level_tc(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* grows, int gpad, const float* w, float* gin,
                          long long ld_in, float* gtree, long long ld_tree, void* wp_ws, void* edge_ws, long long edge_ws_bytes, void* stream,
                          bool tree_adjoint) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && cin > 0 && cout > 0 && slots > 0 && grows && w && gin && gtree && wp_ws && edge_ws, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(gpad == aprnet_tc_pad(cout), "packed row width does not match the padded channel count");
    cudaStream_t st = (cudaStream_t) stream;
    EdgePlan* ep = aprnet_get_edge_plan(a, dl, st);
    if (!ep) return APRNET_ERR_CUDA;
    const ll ts = a->tree_size(dl);
    if (ts > 0) APRNET_CUDA_CHECK(cudaMemset2DAsync(gtree, (size_t) ld_tree * sizeof(float), 0, (size_t) ts * sizeof(float), (size_t) cin, st));
    if (ep->n_active > 0) {
        int rc = APRNET_OK;
        // virtual rows lie a whole number of rows behind the first dO row, so that the gather addresses both from there
        const ll row = (ll) gpad * 2, n = a->number_parts(dl);
        StreamScratch joint(st);
        const char *g0 = (const char*) grows, *e0 = (const char*) edge_ws, *e1 = e0 + edge_ws_bytes;
        if (e0 < g0 + (n + 1) * row || (e1 - g0) / row >= (1ll << 31) - 2) {      // separate buffers of a caller: one joint copy
            const ll rows = (n + 1) * row;
            if ((rc = joint.get((size_t) (rows + edge_ws_bytes)))) return rc;
            APRNET_CUDA_CHECK(cudaMemcpyAsync(joint.p, grows, (size_t) rows, cudaMemcpyDeviceToDevice, st));
            g0 = (const char*) joint.p; e0 = g0 + rows; e1 = e0 + edge_ws_bytes;
        }
        const ll off = (e0 - g0 + row - 1) / row, cap_rows = (e1 - g0) / row - off;
        __nv_bfloat16* vrows = (__nv_bfloat16*) (g0 + off * row);
        const int nk = (int) ep->chunk_a.size() - 1;
        int k0 = 0;
        while (k0 < nk) {
            const int k1 = aprnet_vrow_pass_end(ep->chunk_v, k0, cap_rows);
            const ll v0 = ep->chunk_v[k0], v1 = ep->chunk_v[k1], a0 = ep->chunk_a[k0], a1 = ep->chunk_a[k1];
            if (v1 - v0 > cap_rows) { aprnet_set_error("edge workspace too small for %lld virtual rows", v1 - v0); return APRNET_ERR_ARG; }
            if (v1 > v0) {
                AprnetProfScope _prof("edge_reduce", st);
                // rows per block of the widest column of blocks; a narrower last column has more, and its last blocks find nothing
                const int nch = gpad / 8;
                const dim3 grid((unsigned) aprnet_ceil_div(v1 - v0, VROW_VPT * (256 / std::min(nch, VROW_CHUNKS))), (unsigned) aprnet_ceil_div(nch, VROW_CHUNKS));
                vrow_reduce_kernel<VROW_VPT><<<grid, 256, 0, st>>>(ep->vstart, ep->vsrc, v0, v1, (const __nv_bfloat16*) g0, gpad, vrows);
                APRNET_LAUNCH_CHECK();
            }
            if (a1 > a0 && (rc = aprnet_tc_gather_targets(a, dl, cin, cout, slots, g0, gpad, off - v0, wp_ws, ep, a0, a1, gin, ld_in, gtree, ld_tree, st))) return rc;
            k0 = k1;
        }
    }
    if (!tree_adjoint) return APRNET_OK;
    return aprnet_fill_tree_mean_backward(a, dl, APRNET_F32, cin, gin, ld_in, gtree, ld_tree, st);
}

extern "C" int aprnet_conv333_backward_input_cross_level_tc(aprnet_apr* a, int dl, int cin, int cout, int slots,
                                                            const void* grows, int gpad, const float* w, float* gin,
                                                            int64_t ld_in, float* gtree, int64_t ld_tree, void* wp_ws,
                                                            void* edge_ws, int64_t edge_ws_bytes, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && cin > 0 && cout > 0 && slots > 0 && w && wp_ws, "bad argument");
    APRNET_DEVICE_CHECK(a);
    const int rc = aprnet_tc_pack_weights(a, dl, w, slots, cin, cout, 1, wp_ws, (cudaStream_t) stream);
    return rc ? rc : aprnet_cross_level_tc(a, dl, cin, cout, slots, grows, gpad, w, gin, ld_in, gtree, ld_tree, wp_ws, edge_ws, edge_ws_bytes, stream, true);
}
