// 3x3x3 convolution for very few input channels (Cin <= 4: the first layer of a network) on CUDA cores,
// fp32, used in either arithmetic instead of the implicit GEMM: with Cin = 1 a packed bf16 row would
// carry one useful value in 32 bytes and the 27 x Cin x Cout products per location are far too few to
// amortise a gathered operand tile.  Values are read from a channel-major buffer
//     vals[ci][r],  r in [0, N) particles, [N, N + T) tree means, r = N + T: zero
// through the run plan (forward) or the cached neighbour table (weight gradient), one 4-byte load per entry and input channel.
// Arithmetic: pyapr/aprnet/src/helpers.hpp:505-575 (forward) and :624-702 (weight gradient).
#include "apr_device.cuh"
#include <algorithm>

namespace {

typedef long long ll;
constexpr int MAX_SEGS = APRNET_MAX_LEVELS;

struct SegTable {
    int n;
    ll begin[MAX_SEGS], end[MAX_SEGS];
    int slot[MAX_SEGS];
    int tile_begin[MAX_SEGS + 1];
};

inline SegTable make_seg_table(const std::vector<Segment>& segs, ll tile) {
    SegTable t;
    t.n = (int) segs.size();
    t.tile_begin[0] = 0;
    for (int i = 0; i < t.n; ++i) {
        t.begin[i] = segs[i].begin; t.end[i] = segs[i].end; t.slot[i] = segs[i].slot;
        t.tile_begin[i + 1] = t.tile_begin[i] + aprnet_ceil_div(segs[i].end - segs[i].begin, tile);
    }
    return t;
}

constexpr int SMALL_STEP = 4 * 30;       // slots whose results a block of the forward kernel yields per tile

struct alignas(16) F4 { float a[4]; };

__device__ __forceinline__ ll resolve_row(int32_t v, ll n, ll zero_row) {
    return v >= 0 ? (ll) v : (v == APRNET_NONE ? zero_row : n + aprnet_dec_tree(v));
}

// vals[ci][0, n) = x[ci], vals[ci][n, n + t) = tree[ci], vals[ci][n + t] = 0
__global__ void small_stage_kernel(const float* __restrict__ x, ll ld_x, ll n, const float* __restrict__ tree, ll ld_tree, ll t,
                                   int cin, float* __restrict__ vals) {
    const ll R = n + t + 1;
    const ll r = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= R) return;
    for (int ci = 0; ci < cin; ++ci)
        vals[(ll) ci * R + r] = r < n ? x[(ll) ci * ld_x + r] : (r < n + t ? tree[(ll) ci * ld_tree + (r - n)] : 0.f);
}

// forward: thread = slot of the run plan x block of 32 output channels; weights of the level's stencil in shared memory as [tap][ci][32],
// read four at a time.  A lane loads the 9 values that lie beside its cell (dz, dx) and gets those of the y neighbours from the lanes next to it, so a warp
// yields 30 slots and gathers 9 values per slot where the neighbour table needs 27 entries and 27 values per location.  What bounds it is the latency of
// these gathers: the table entries of the next tile are on their way during the multiply-adds, and a block takes up to eight tiles with one
// staging of the weights.  (They are requested behind a block's last tile too: a condition costs registers, 1 -> 16 on 3.5 M locations
// 303 -> 320 us, and is no faster with one tile per block, on 7 k and 64 k locations.)  1 -> 32 channels on 3.5 M locations 522 -> 311 us against one thread per
// location and the neighbour table, 2 -> 32 889 -> 596, 4 -> 40 on 1.9 M 1415 -> 1124; 1 -> 16 on 7 k locations 10.7 -> 6.1.  (Paired multiply-adds: 0 to 10 % slower.)
// The chain of multiply-adds of a result is channel by channel, tap by tap.
template<int CIN>
__global__ void __launch_bounds__(128) conv333_small_forward_kernel(SegTable segs, int tiles, const int32_t* __restrict__ src, ll S, const int32_t* __restrict__ loc,
                                                                    ll N, ll T, const float* __restrict__ vals, const float* __restrict__ w,
                                                                    int cout, const float* __restrict__ bias, float* __restrict__ out, ll ld_out) {
    __shared__ F4 ws[27 * CIN * 8];
    __shared__ float bias_s[32];
    int seg = 0;
    while (seg + 1 < segs.n && (int) blockIdx.x >= segs.tile_begin[seg + 1]) ++seg;
    const int co0 = blockIdx.y * 32;
    const float* wslot = w + (ll) segs.slot[seg] * cout * CIN * 27;
    for (int e = threadIdx.x; e < 27 * CIN * 32; e += 128) {
        const int co = e & 31, ci = (e >> 5) % CIN, tap = e / (32 * CIN);
        reinterpret_cast<float*>(ws)[e] = co0 + co < cout ? wslot[((ll) (co0 + co) * CIN + ci) * 27 + tap] : 0.f;
    }
    if (threadIdx.x < 32) bias_s[threadIdx.x] = bias && co0 + (int) threadIdx.x < cout ? bias[co0 + threadIdx.x] : 0.f;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const ll R = N + T + 1, begin = segs.begin[seg], end = segs.end[seg];
    // the warp's first tile: lane 0 is the slot in front of its 30; consecutive tiles of a block are SMALL_STEP slots apart
    ll s = begin + (ll) (blockIdx.x - segs.tile_begin[seg]) * SMALL_STEP * tiles + (threadIdx.x >> 5) * 30 - 1 + lane;
    const int nco = min(32, cout - co0);
    int32_t rows[9], p_next;
    auto request = [&]() {                             // row numbers fit 32 bits (aprnet_rows_overflow)
        const bool in = s >= begin && s < end;
#pragma unroll
        for (int d = 0; d < 9; ++d) rows[d] = in ? __ldg(src + d * S + s) : APRNET_NONE;
        p_next = in && lane > 0 && lane < 31 ? __ldg(loc + s) : -1;
    };
    request();
    for (int i = 0; i < tiles && s - lane + 1 < end; ++i) {
        float acc[32];
#pragma unroll
        for (int o = 0; o < 32; ++o) acc[o] = 0.f;
        int32_t at[9];
#pragma unroll
        for (int d = 0; d < 9; ++d) at[d] = (int32_t) resolve_row(rows[d], N, N + T);
        const int32_t p = p_next;
        s += SMALL_STEP;
        float v[9];
#pragma unroll
        for (int d = 0; d < 9; ++d) v[d] = __ldg(vals + at[d]);
        request();
#pragma unroll 1
        for (int ci = 0; ci < CIN; ++ci) {
#pragma unroll
            for (int d = 0; d < 9; ++d) {
                const float beside[3] = {__shfl_up_sync(0xffffffffu, v[d], 1), v[d], __shfl_down_sync(0xffffffffu, v[d], 1)};
                if (ci + 1 < CIN) v[d] = __ldg(vals + (ll) (ci + 1) * R + at[d]);
#pragma unroll
                for (int dy = 0; dy < 3; ++dy) {
                    const F4* wr = ws + ((d * 3 + dy) * CIN + ci) * 8;
#pragma unroll
                    for (int o4 = 0; o4 < 8; ++o4) {
                        const F4 q = wr[o4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) acc[4 * o4 + k] = fmaf(beside[dy], q.a[k], acc[4 * o4 + k]);
                    }
                }
            }
        }
        if (bias) {
#pragma unroll
            for (int o = 0; o < 32; ++o) acc[o] += bias_s[o];
        }
        if (p < 0) continue;
        float* dst = out + (ll) co0 * ld_out + p;
        if (nco == 32) {
#pragma unroll
            for (int o = 0; o < 32; ++o) dst[(ll) o * ld_out] = acc[o];
        } else {
#pragma unroll
            for (int o = 0; o < 32; ++o)
                if (o < nco) dst[(ll) o * ld_out] = acc[o];
        }
    }
}

// weight gradient: block = range of locations of one level x block of 32 output channels, one launch over all levels.  The 27 x CIN
// gathered values and the 32 dO values of KP locations are staged in shared memory; the staging is bound by the latency of its loads, so the table
// entries and the dO of a step are requested before the products of the step before it, its values together (1 -> 32 channels on 3.5 M
// locations 661 -> 375 us, 2 -> 32 1995 -> 832, 1 -> 16 on 7 k locations 22 -> 15).  A thread owns a 4 x 4
// tile of (tap, ci) x co products; the 4 thread groups of a block take different quarters of every staged
// step and are combined in a fixed order.  The products of a quarter (8 or 16 locations) are summed before they are added to the
// thread's sums: short chains of additions whatever the length of the range.  partial[range][tap][co][ci].
struct SmallRanges { int n; ll begin[MAX_SEGS], end[MAX_SEGS], len[MAX_SEGS]; int first[MAX_SEGS + 1]; };

template<int CIN>
__global__ void __launch_bounds__(256) conv333_small_dw_kernel(SmallRanges rg, const int32_t* __restrict__ nbr, ll N, ll T,
                                                               const float* __restrict__ vals, const float* __restrict__ gout, ll ld_out,
                                                               int cout, float* __restrict__ partial) {
    constexpr int ROWS = 27 * CIN, RQ = (ROWS + 3) / 4;                 // (tap, ci) rows, row quads
    constexpr int KP = CIN <= 2 ? 64 : 32;                              // staged locations per step
    constexpr int XSTRIDE = RQ | 1;                                     // odd: consecutive locations fall on different banks
    __shared__ F4 xs[KP][XSTRIDE];
    __shared__ F4 gs[KP][8 + 1];
    __shared__ float red[RQ * 4 * 32];
    const int co0 = blockIdx.y * 32;
    int seg = 0;
    while (seg + 1 < rg.n && (int) blockIdx.x >= rg.first[seg + 1]) ++seg;
    const ll pb = rg.begin[seg] + (ll) ((int) blockIdx.x - rg.first[seg]) * rg.len[seg], pe = min(rg.end[seg], pb + rg.len[seg]);
    const ll R = N + T + 1;
    const int grp = threadIdx.x >> 6, t64 = threadIdx.x & 63;
    const int rq = t64 >> 3, cq = t64 & 7;                             // 8 row quads per pass of 64 threads
    constexpr int PASSES = (RQ + 7) / 8;
    float acc[PASSES][4][4];
#pragma unroll
    for (int ps = 0; ps < PASSES; ++ps)
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[ps][a][b] = 0.f;
    constexpr int NX = (KP * RQ * 4 + 255) / 256, NG = KP * 32 / 256;           // consecutive threads take consecutive locations of one row
    int32_t at[NX];
    float gv[NG];
    auto request = [&](ll p0) {                    // table entries and dO of a step: they come from DRAM, one step ahead
#pragma unroll
        for (int i = 0; i < NX; ++i) {
            const int e = threadIdx.x + i * 256, k = e % KP, row = e / KP;
            at[i] = row < ROWS && p0 + k < pe ? __ldg(nbr + (ll) (row / CIN) * N + p0 + k) : APRNET_NONE;
        }
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            const int e = threadIdx.x + i * 256, k = e % KP, co = e / KP;
            gv[i] = (p0 + k < pe && co0 + co < cout) ? gout[(ll) (co0 + co) * ld_out + p0 + k] : 0.f;
        }
    };
    request(pb);
    for (ll p0 = pb; p0 < pe; p0 += KP) {
        float xv[NX];
#pragma unroll
        for (int i = 0; i < NX; ++i) {
            const int row = (threadIdx.x + i * 256) / KP;
            xv[i] = row < RQ * 4 ? __ldg(vals + (ll) (row % CIN) * R + resolve_row(at[i], N, N + T)) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < NX; ++i) {
            const int e = threadIdx.x + i * 256, k = e % KP, row = e / KP;
            if (row < RQ * 4) xs[k][row >> 2].a[row & 3] = xv[i];
        }
#pragma unroll
        for (int i = 0; i < NG; ++i) { const int e = threadIdx.x + i * 256, k = e % KP, co = e / KP; gs[k][co >> 2].a[co & 3] = gv[i]; }
        __syncthreads();
        request(p0 + KP);                          // (beyond the range: nothing is read)
#pragma unroll
        for (int ps = 0; ps < PASSES; ++ps) {
            if (ps * 8 + rq >= RQ) continue;
            float part[4][4];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) part[a][b] = 0.f;
#pragma unroll 4
            for (int k = grp * (KP / 4); k < (grp + 1) * (KP / 4); ++k) {
                const F4 g = gs[k][cq], x = xs[k][ps * 8 + rq];
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b < 4; ++b) part[a][b] = fmaf(x.a[a], g.a[b], part[a][b]);
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[ps][a][b] += part[a][b];
        }
        __syncthreads();
    }
    // the four groups add their tiles one after the other: fixed order
    for (int gsel = 0; gsel < 4; ++gsel) {
        if (grp == gsel) {
#pragma unroll
            for (int ps = 0; ps < PASSES; ++ps)
                if (ps * 8 + rq < RQ)
#pragma unroll
                    for (int a = 0; a < 4; ++a)
#pragma unroll
                        for (int b = 0; b < 4; ++b) {
                            float* r = red + ((ps * 8 + rq) * 4 + a) * 32 + cq * 4 + b;
                            *r = gsel == 0 ? acc[ps][a][b] : *r + acc[ps][a][b];
                        }
        }
        __syncthreads();
    }
    float* dst = partial + (ll) blockIdx.x * cout * CIN * 27;
    for (int e = threadIdx.x; e < ROWS * 32; e += 256) {
        const int row = e >> 5, co = co0 + (e & 31);
        if (co < cout) dst[((ll) (row / CIN) * cout + co) * CIN + row % CIN] = red[e];
    }
}

} // namespace

bool aprnet_small_cin(int cin) { return cin <= 4; }

int aprnet_small_stage(const float* x, ll ld_x, ll n, const float* tree, ll ld_tree, ll t, int cin, float* vals, cudaStream_t st) {
    AprnetProfScope _prof("small_stage", st);
    small_stage_kernel<<<aprnet_ceil_div(n + t + 1, 256), 256, 0, st>>>(x, ld_x, n, tree, ld_tree, t, cin, vals);
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

int aprnet_small_forward(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* vals, const float* w, const float* bias, float* out, ll ld_out, cudaStream_t st) {
    const RunPlan* rp = aprnet_get_run_plan(a, dl, st);
    if (!rp) return APRNET_ERR_CUDA;
    std::vector<Segment> list = aprnet_segments(a, dl, slots, false);
    for (Segment& g : list) { g.begin = rp->level_begin[g.level]; g.end = rp->level_begin[g.level + 1]; }
    // several tiles per block once eight blocks per SM have one each
    const ll tiles = aprnet_ceil_div(rp->n_slots, SMALL_STEP), groups = aprnet_ceil_div(cout, 32);
    const int per_block = (int) std::min<ll>(8, std::max<ll>(1, tiles * groups / (148 * 8)));
    const SegTable segs = make_seg_table(list, SMALL_STEP * per_block);
    if (segs.tile_begin[segs.n] == 0) return APRNET_OK;
    dim3 grid((unsigned) segs.tile_begin[segs.n], (unsigned) groups);
    char pname[64];
    snprintf(pname, sizeof(pname), "conv333_small_fwd:ci%d:co%d:dl%d", cin, cout, dl);
    AprnetProfScope _prof(pname, st);
#define SMALL_CASE(CIN_) case CIN_: conv333_small_forward_kernel<CIN_><<<grid, 128, 0, st>>>(segs, per_block, rp->src, rp->n_slots, rp->loc, a->number_parts(dl), \
        a->tree_size(dl), vals, w, cout, bias, out, ld_out); break;
    switch (cin) {
        SMALL_CASE(1) SMALL_CASE(2) SMALL_CASE(3) SMALL_CASE(4)
        default: aprnet_set_error("small-Cin path called with cin = %d", cin); return APRNET_ERR_ARG;
    }
#undef SMALL_CASE
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

// partial: aprnet_conv333_tc_dw_partial_elems() floats
int aprnet_small_backward_weights(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* vals, const float* gout, ll ld_out,
                                  float* gw, int accumulate, float* partial, cudaStream_t st) {
    const AprPlan* plan = aprnet_get_plan(a, dl, st);
    if (!plan) return APRNET_ERR_CUDA;
    const ll max_ranges = aprnet_conv333_tc_dw_partial_elems(cin, cout) / ((ll) 27 * cin * cout);
    char pname[64];
    snprintf(pname, sizeof(pname), "conv333_small_dw:ci%d:co%d:dl%d", cin, cout, dl);
    const std::vector<Segment> segs = aprnet_segments(a, dl, slots, false);
    SmallRanges rg;
    SlotRanges sr;
    rg.n = (int) segs.size();
    sr.n = 0;
    ll total = 0;
    for (const Segment& s : segs) total += s.end - s.begin;
    // at least 512 locations per block, at most eight blocks per SM or what the partial buffer holds
    const ll budget = std::max<ll>(rg.n, std::min<ll>(max_ranges, 1184) - rg.n);
    ll len = std::max<ll>(512, (total + budget - 1) / budget + 63) / 64 * 64;
    auto blocks = [&]() { ll b = 0; for (const Segment& s : segs) b += (s.end - s.begin + len - 1) / len; return b; };
    while (blocks() > std::max<ll>(max_ranges, rg.n)) len *= 2;
    rg.first[0] = 0;
    for (int i = 0; i < rg.n; ++i) {
        rg.begin[i] = segs[i].begin; rg.end[i] = segs[i].end; rg.len[i] = len;
        rg.first[i + 1] = rg.first[i] + aprnet_ceil_div(segs[i].end - segs[i].begin, len);
        if (sr.n == 0 || sr.slot[sr.n - 1] != segs[i].slot) { sr.first[sr.n] = rg.first[i]; sr.slot[sr.n++] = segs[i].slot; }
        sr.first[sr.n] = rg.first[i + 1];
    }
    const int nranges = rg.n ? rg.first[rg.n] : 0;
    if (nranges > max_ranges) { aprnet_set_error("first-layer weight gradient: %d ranges exceed the partial buffer", nranges); return APRNET_ERR_ARG; }
    if (nranges > 0) {
        dim3 grid((unsigned) nranges, (unsigned) aprnet_ceil_div(cout, 32));
        AprnetProfScope _prof(pname, st);
        switch (cin) {
            case 1: conv333_small_dw_kernel<1><<<grid, 256, 0, st>>>(rg, plan->nbr, plan->n, plan->tree_size, vals, gout, ld_out, cout, partial); break;
            case 2: conv333_small_dw_kernel<2><<<grid, 256, 0, st>>>(rg, plan->nbr, plan->n, plan->tree_size, vals, gout, ld_out, cout, partial); break;
            case 3: conv333_small_dw_kernel<3><<<grid, 256, 0, st>>>(rg, plan->nbr, plan->n, plan->tree_size, vals, gout, ld_out, cout, partial); break;
            case 4: conv333_small_dw_kernel<4><<<grid, 256, 0, st>>>(rg, plan->nbr, plan->n, plan->tree_size, vals, gout, ld_out, cout, partial); break;
            default: aprnet_set_error("small-Cin path called with cin = %d", cin); return APRNET_ERR_ARG;
        }
        APRNET_LAUNCH_CHECK();
    }
    return aprnet_dw_reduce(partial, sr, slots, accumulate, cin, cout, gw, st);
}
