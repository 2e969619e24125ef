// Run plan of a level delta: the output locations of every level in runs along y, for gathers that stage a row of cells once
// and use it for the three y taps of the stencil.
//
// The cells of a level are listed row by row (z, x, then y), every cell that holds an output location plus the cells one step
// below and above it (a "slot" each; slots without a location are the ends of the runs).  Neighbouring slots of a run are
// neighbouring cells, so the y neighbours of the location in slot s sit in slots s - 1 and s + 1 of whatever row of cells
// (z + dz, x + dx) was gathered for the slots: 9 gathered rows per slot instead of 27 per location.  Runs of an APR are 5 to 30
// cells long (fine cells come in pairs, the refined regions are compact): 1.07 to 1.27 slots per location.
#include "apr_device.cuh"
#include <cub/cub.cuh>
#include <algorithm>

namespace {

typedef long long ll;

// rows of all levels of the level delta, level by level
struct RunLevels { int lmin, cml, dl; ll begin[APRNET_MAX_LEVELS + 2]; ll tree_off; };

__device__ __forceinline__ int level_of_row(const RunLevels& R, ll row) {
    int l = R.lmin;
    while (l < R.cml && row >= R.begin[l + 1]) ++l;
    return l;
}

struct RunRow {                 // the sorted y coordinates of one row: particles, and at the finest level of a pooled tensor tree nodes
    const uint16_t *a, *b;
    ll ia, ea, ib, eb;
    __device__ bool next(int* y, ll* index, bool* from_b) {
        const int ya = ia < ea ? (int) a[ia] : 1 << 30, yb = ib < eb ? (int) b[ib] : 1 << 30;
        if (ya == 1 << 30 && yb == 1 << 30) return false;
        *from_b = yb < ya;
        *y = min(ya, yb);
        *index = *from_b ? ib++ : ia++;
        return true;
    }
};

__device__ __forceinline__ RunRow run_row(const LevelMeta& m, const ll* row_ptr, const uint16_t* y, const ll* trow_ptr, const uint16_t* ty, int l, ll row, int with_tree) {
    RunRow r;
    r.a = y; r.b = ty;
    r.ia = row_ptr[m.row_off[l] + row]; r.ea = row_ptr[m.row_off[l] + row + 1];
    r.ib = r.eb = 0;
    if (with_tree) { r.ib = trow_ptr[m.trow_off[l] + row]; r.eb = trow_ptr[m.trow_off[l] + row + 1]; }
    return r;
}

// one thread per row; first pass (slot_y == null): count[row] = slots of the row, *total = slots of all rows; second pass: the slots
// from first[row] on
__global__ void run_slots_kernel(LevelMeta m, RunLevels R, const ll* __restrict__ row_ptr, const uint16_t* __restrict__ y, const ll* __restrict__ trow_ptr,
                                 const uint16_t* __restrict__ ty, int32_t* __restrict__ count, const int32_t* __restrict__ first,
                                 int32_t* __restrict__ slot_y, int32_t* __restrict__ slot_loc, unsigned long long* __restrict__ total) {
    const ll g = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    const bool inside = g < R.begin[R.cml + 1];
    const int l = inside ? level_of_row(R, g) : R.cml;
    const ll row = g - R.begin[l], tree_off = R.tree_off;
    const int with_tree = R.dl > 0 && l == R.cml;
    RunRow r = {};
    if (inside) r = run_row(m, row_ptr, y, trow_ptr, ty, l, row, with_tree);
    int last = -3, n = 0, yy;
    ll index;
    bool from_b;
    const ll base = slot_y && inside ? first[g] : 0;
    while (r.next(&yy, &index, &from_b)) {
        for (int c = max(yy - 1, last + 1); c <= yy + 1; ++c) {
            if (slot_y) { slot_y[base + n] = c; slot_loc[base + n] = -1; }
            ++n;
        }
        last = yy + 1;
        if (slot_y) slot_loc[base + n - 2] = (int32_t) (from_b ? index + tree_off : index);
    }
    if (slot_y) return;
    if (inside) count[g] = n;
    const unsigned sum = __reduce_add_sync(0xffffffffu, (unsigned) n);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(total, (unsigned long long) sum);
}

__device__ __forceinline__ ll find_cell(const uint16_t* __restrict__ y, ll b, ll e, int target) {
    ll lo = b, hi = e;
    while (lo < hi) { const ll mid = (lo + hi) >> 1; if ((int) y[mid] < target) lo = mid + 1; else hi = mid; }
    return (lo < e && (int) y[lo] == target) ? lo : -1;
}

// one warp per row: what fills cell (z + dz, x + dx, y) for every slot of the row; binary search of the neighbour row in particles, coarser particles and tree nodes
__global__ void run_sources_kernel(LevelMeta m, RunLevels R, const ll* __restrict__ row_ptr, const uint16_t* __restrict__ y, const ll* __restrict__ trow_ptr,
                                   const uint16_t* __restrict__ ty, const int32_t* __restrict__ first, const int32_t* __restrict__ slot_y, ll S,
                                   int32_t* __restrict__ src) {
    const ll g = ((ll) blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (g >= R.begin[R.cml + 1]) return;
    const int l = level_of_row(R, g), cml = R.cml;
    const ll row = g - R.begin[l], tree_off = R.tree_off;
    const int xn = m.x_num[l], zn = m.z_num[l], yn = m.y_num[l];
    const ll sb = first[g], se = first[g + 1];
    if (sb == se) return;
    const int z = (int) (row / xn), x = (int) (row % xn);
    for (int d = 0; d < 9; ++d) {
        const int nz = z + d / 3 - 1, nx = x + d % 3 - 1;
        const bool inside = nz >= 0 && nx >= 0 && nz < zn && nx < xn;
        ll pb = 0, pe = 0, cb = 0, ce = 0, tb = 0, te = 0;
        if (inside) {
            const ll r = m.row_off[l] + (ll) nz * xn + nx;
            pb = row_ptr[r]; pe = row_ptr[r + 1];
            if (l > m.level_min) {
                const ll cr = m.row_off[l - 1] + (ll) (nz >> 1) * m.x_num[l - 1] + (nx >> 1);
                cb = row_ptr[cr]; ce = row_ptr[cr + 1];
            }
            if (l <= m.level_max - 1) {
                const ll tr = m.trow_off[l] + (ll) nz * xn + nx;
                tb = trow_ptr[tr]; te = trow_ptr[tr + 1];
            }
        }
        for (ll s = sb + lane; s < se; s += 32) {
            const int yq = slot_y[s];
            int32_t v = APRNET_NONE;
            if (inside && yq >= 0 && yq < yn) {
                ll f = find_cell(y, pb, pe, yq);
                if (f < 0) f = find_cell(y, cb, ce, yq >> 1);
                if (f >= 0) v = (int32_t) f;
                else {
                    f = find_cell(ty, tb, te, yq);
                    if (f >= 0) v = l == cml ? (int32_t) (f + tree_off) : aprnet_enc_tree(f);
                }
            }
            src[(ll) d * S + s] = v;
        }
    }
}

// the neighbour table from the run plan: the three y neighbours of a location are its slot and the slots beside it, in the nine rows
__global__ void nbr_from_runs_kernel(const int32_t* __restrict__ loc, const int32_t* __restrict__ src, ll S, int32_t* __restrict__ nbr, ll N) {
    const ll s = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const int32_t p = loc[s];
    if (p < 0) return;                 // a location has a slot on either side, so s - 1 and s + 1 exist
    int32_t v[27];
#pragma unroll
    for (int t = 0; t < 27; ++t) v[t] = src[(ll) (t / 3) * S + s + t % 3 - 1];
#pragma unroll
    for (int t = 0; t < 27; ++t) nbr[(ll) t * N + p] = v[t];
}

struct Picks { ll at[APRNET_MAX_LEVELS + 2]; };
__global__ void pick_kernel(const int32_t* __restrict__ v, Picks at, int n, int32_t* __restrict__ out) { if ((int) threadIdx.x < n) out[threadIdx.x] = v[at.at[threadIdx.x]]; }

int build_run_plan(aprnet_apr* a, int dl, RunPlan& rp, cudaStream_t st) {
    const LevelMeta& m = a->meta;
    const int cml = a->cml(dl);
    RunLevels R;
    R.lmin = m.level_min; R.cml = cml; R.dl = dl; R.tree_off = dl > 0 ? a->tree_offset(cml) : 0;
    ll rows = 0;
    for (int l = m.level_min; l <= cml; ++l) { R.begin[l] = rows; rows += (ll) m.z_num[l] * m.x_num[l]; }
    R.begin[cml + 1] = rows;
    int32_t *first = nullptr, *slot_y = nullptr, *picked = nullptr;
    unsigned long long* total = nullptr;
    int rc = APRNET_OK;
    void* temp = nullptr;
    size_t temp_bytes = 0;
    auto cleanup = [&]() { aprnet_pool_free(first, st); aprnet_pool_free(slot_y, st); aprnet_pool_free(picked, st); aprnet_pool_free(temp, st); aprnet_pool_free(total, st); };
#define RP_ALLOC(p, bytes) do { if ((rc = aprnet_pool_alloc((void**) &(p), (bytes), st))) { cleanup(); return rc; } } while (0)
#define RP_CHECK(expr) do { cudaError_t _e = (expr); if (_e != cudaSuccess) { aprnet_set_error("%s failed: %s", #expr, cudaGetErrorString(_e)); cudaGetLastError(); cleanup(); return APRNET_ERR_CUDA; } } while (0)
    // rows of packed operands and slots are 32-bit in the kernels
    if (aprnet_rows_overflow(a, dl)) return APRNET_ERR_UNSUPPORTED;
    RP_ALLOC(total, sizeof(ll));
    RP_CHECK(cudaMemsetAsync(total, 0, sizeof(ll), st));
    RP_ALLOC(first, (size_t) (rows + 1) * sizeof(int32_t));
    RP_CHECK(cudaMemsetAsync(first + rows, 0, sizeof(int32_t), st));
    run_slots_kernel<<<aprnet_ceil_div(rows, 128), 128, 0, st>>>(m, R, a->row_ptr, a->y, a->tree_row_ptr, a->tree_y, first, nullptr, nullptr, nullptr, total);
    RP_CHECK(cub::DeviceScan::ExclusiveSum(nullptr, temp_bytes, first, first, rows + 1, st));
    RP_ALLOC(temp, std::max<size_t>(temp_bytes, 1));
    RP_CHECK(cub::DeviceScan::ExclusiveSum(temp, temp_bytes, first, first, rows + 1, st));
    std::vector<int32_t> at(cml + 2, 0);
    Picks picks;
    for (int l = m.level_min; l <= cml + 1; ++l) picks.at[l - m.level_min] = R.begin[l];
    RP_ALLOC(picked, sizeof(int32_t) * (APRNET_MAX_LEVELS + 2));
    pick_kernel<<<1, 32, 0, st>>>(first, picks, cml + 2 - m.level_min, picked);
    RP_CHECK(cudaMemcpyAsync(at.data() + m.level_min, picked, sizeof(int32_t) * (cml + 2 - m.level_min), cudaMemcpyDeviceToHost, st));
    unsigned long long all = 0;
    RP_CHECK(cudaMemcpyAsync(&all, total, sizeof(all), cudaMemcpyDeviceToHost, st));
    RP_CHECK(cudaStreamSynchronize(st));
    if (all >= (1ull << 31) - 256) { aprnet_set_error("run plan: %llu slots exceed the 32-bit tables", all); cleanup(); return APRNET_ERR_UNSUPPORTED; }
    const ll S = at[cml + 1];
    rp.n_slots = S;
    rp.level_begin.assign(at.begin(), at.end());
    RP_ALLOC(slot_y, (size_t) std::max<ll>(S, 1) * sizeof(int32_t));
    RP_ALLOC(rp.loc, (size_t) std::max<ll>(S, 1) * sizeof(int32_t));
    RP_ALLOC(rp.src, (size_t) std::max<ll>(S, 1) * 9 * sizeof(int32_t));
    run_slots_kernel<<<aprnet_ceil_div(rows, 128), 128, 0, st>>>(m, R, a->row_ptr, a->y, a->tree_row_ptr, a->tree_y, nullptr, first, slot_y, rp.loc, nullptr);
    run_sources_kernel<<<aprnet_ceil_div(rows * 32, 128), 128, 0, st>>>(m, R, a->row_ptr, a->y, a->tree_row_ptr, a->tree_y, first, slot_y, S, rp.src);
    RP_CHECK(cudaGetLastError());
    RP_CHECK(cudaStreamSynchronize(st));
#undef RP_CHECK
#undef RP_ALLOC
    cleanup();
    return APRNET_OK;
}

} // namespace

const RunPlan* aprnet_get_run_plan(aprnet_apr* a, int dl, cudaStream_t st) {
    auto it = a->run_plans.find(dl);
    if (it != a->run_plans.end()) return &it->second;
    if (aprnet_check_device(a) != APRNET_OK) return nullptr;
    RunPlan rp;
    if (build_run_plan(a, dl, rp, st) != APRNET_OK) { aprnet_pool_free(rp.loc, st); aprnet_pool_free(rp.src, st); return nullptr; }
    a->device_bytes += std::max<ll>(rp.n_slots, 1) * 10 * (ll) sizeof(int32_t);
    return &a->run_plans.emplace(dl, rp).first->second;
}

// nbr: [27][n].  Nine searches per slot and a copy instead of 27 searches per location; a run plan that is not cached is built for it.
int aprnet_fill_nbr_table(aprnet_apr* a, int dl, int32_t* nbr, ll n, cudaStream_t st) {
    const auto it = a->run_plans.find(dl);
    RunPlan own;
    const RunPlan* rp = it != a->run_plans.end() ? &it->second : &own;
    int rc = APRNET_OK;
    if (rp == &own) rc = build_run_plan(a, dl, own, st);
    if (!rc && rp->n_slots > 0) {
        nbr_from_runs_kernel<<<aprnet_ceil_div(rp->n_slots, 256), 256, 0, st>>>(rp->loc, rp->src, rp->n_slots, nbr, n);
        if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) { aprnet_set_error("aprnet_fill_nbr_table: kernel failed"); rc = APRNET_ERR_CUDA; }
    }
    aprnet_pool_free(own.loc, st); aprnet_pool_free(own.src, st);
    return rc;
}

// Builds (once; cached) the run plan of a level delta.  Allocates; call it up front.
extern "C" int aprnet_run_plan_build(aprnet_apr* a, int dl, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl), "bad handle or level_delta");
    APRNET_DEVICE_CHECK(a);
    return aprnet_get_run_plan(a, dl, (cudaStream_t) stream) ? APRNET_OK : APRNET_ERR_CUDA;
}
