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

// one thread per row; first pass (slot_y == null): count[row] = slots of the row; second pass: the slots from first[row] on
__global__ void run_slots_kernel(LevelMeta m, const ll* __restrict__ row_ptr, const uint16_t* __restrict__ y, const ll* __restrict__ trow_ptr,
                                 const uint16_t* __restrict__ ty, int l, int with_tree, ll tree_off, int32_t* __restrict__ count,
                                 const int32_t* __restrict__ first, int32_t* __restrict__ slot_y, int32_t* __restrict__ slot_loc) {
    const ll row = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= (ll) m.z_num[l] * m.x_num[l]) return;
    RunRow r = run_row(m, row_ptr, y, trow_ptr, ty, l, row, with_tree);
    int last = -3, n = 0, yy;
    ll index;
    bool from_b;
    const ll base = slot_y ? first[row] : 0;
    while (r.next(&yy, &index, &from_b)) {
        for (int c = max(yy - 1, last + 1); c <= yy + 1; ++c) {
            if (slot_y) { slot_y[base + n] = c; slot_loc[base + n] = -1; }
            ++n;
        }
        last = yy + 1;
        if (slot_y) slot_loc[base + n - 2] = (int32_t) (from_b ? index + tree_off : index);
    }
    if (!slot_y) count[row] = n;
}

__device__ __forceinline__ ll find_cell(const uint16_t* __restrict__ y, ll b, ll e, int target) {
    ll lo = b, hi = e;
    while (lo < hi) { const ll mid = (lo + hi) >> 1; if ((int) y[mid] < target) lo = mid + 1; else hi = mid; }
    return (lo < e && (int) y[lo] == target) ? lo : -1;
}

// one warp per row: what fills cell (z + dz, x + dx, y) for every slot of the row; resolution as in build_nbr_table_kernel
__global__ void run_sources_kernel(LevelMeta m, const ll* __restrict__ row_ptr, const uint16_t* __restrict__ y, const ll* __restrict__ trow_ptr,
                                   const uint16_t* __restrict__ ty, int l, int cml, ll tree_off, const int32_t* __restrict__ first,
                                   const int32_t* __restrict__ slot_y, ll S, int32_t* __restrict__ src) {
    const ll row = ((ll) blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int xn = m.x_num[l], zn = m.z_num[l], yn = m.y_num[l];
    if (row >= (ll) zn * xn) return;
    const ll sb = first[row], se = first[row + 1];
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

int build_run_plan(aprnet_apr* a, int dl, RunPlan& rp, cudaStream_t st) {
    const LevelMeta& m = a->meta;
    const int cml = a->cml(dl);
    const ll toff = dl > 0 ? a->tree_offset(cml) : 0;
    ll rows = 0;
    std::vector<ll> row_begin(cml + 2, 0);
    for (int l = m.level_min; l <= cml; ++l) { row_begin[l] = rows; rows += (ll) m.z_num[l] * m.x_num[l]; }
    row_begin[cml + 1] = rows;
    int32_t *first = nullptr, *slot_y = nullptr;
    void* temp = nullptr;
    size_t temp_bytes = 0;
    auto cleanup = [&]() { cudaFree(first); cudaFree(slot_y); cudaFree(temp); };
#define RP_CHECK(expr) do { cudaError_t _e = (expr); if (_e != cudaSuccess) { aprnet_set_error("%s failed: %s", #expr, cudaGetErrorString(_e)); cudaGetLastError(); cleanup(); return APRNET_ERR_CUDA; } } while (0)
    RP_CHECK(cudaMalloc((void**) &first, (size_t) (rows + 1) * sizeof(int32_t)));
    RP_CHECK(cudaMemsetAsync(first + rows, 0, sizeof(int32_t), st));
    for (int l = m.level_min; l <= cml; ++l)
        run_slots_kernel<<<aprnet_ceil_div((ll) m.z_num[l] * m.x_num[l], 128), 128, 0, st>>>(m, a->row_ptr, a->y, a->tree_row_ptr, a->tree_y, l, dl > 0 && l == cml, toff,
                                                                                       first + row_begin[l], nullptr, nullptr, nullptr);
    RP_CHECK(cub::DeviceScan::ExclusiveSum(nullptr, temp_bytes, first, first, (int) (rows + 1), st));
    RP_CHECK(cudaMalloc(&temp, std::max<size_t>(temp_bytes, 1)));
    RP_CHECK(cub::DeviceScan::ExclusiveSum(temp, temp_bytes, first, first, (int) (rows + 1), st));
    std::vector<int32_t> at(cml + 2, 0);
    for (int l = m.level_min; l <= cml + 1; ++l)
        RP_CHECK(cudaMemcpyAsync(&at[l], first + row_begin[l], sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    RP_CHECK(cudaStreamSynchronize(st));
    const ll S = at[cml + 1];
    rp.n_slots = S;
    rp.level_begin.assign(at.begin(), at.end());
    RP_CHECK(cudaMalloc((void**) &slot_y, (size_t) std::max<ll>(S, 1) * sizeof(int32_t)));
    RP_CHECK(cudaMalloc((void**) &rp.loc, (size_t) std::max<ll>(S, 1) * sizeof(int32_t)));
    RP_CHECK(cudaMalloc((void**) &rp.src, (size_t) std::max<ll>(S, 1) * 9 * sizeof(int32_t)));
    a->device_bytes += std::max<ll>(S, 1) * 10 * (ll) sizeof(int32_t);
    for (int l = m.level_min; l <= cml; ++l) {
        const ll n = (ll) m.z_num[l] * m.x_num[l];
        run_slots_kernel<<<aprnet_ceil_div(n, 128), 128, 0, st>>>(m, a->row_ptr, a->y, a->tree_row_ptr, a->tree_y, l, dl > 0 && l == cml, toff, nullptr,
                                                                 first + row_begin[l], slot_y, rp.loc);
        run_sources_kernel<<<aprnet_ceil_div(n * 32, 128), 128, 0, st>>>(m, a->row_ptr, a->y, a->tree_row_ptr, a->tree_y, l, cml, toff, first + row_begin[l], slot_y, S, rp.src);
    }
    RP_CHECK(cudaGetLastError());
    RP_CHECK(cudaStreamSynchronize(st));
#undef RP_CHECK
    cleanup();
    return APRNET_OK;
}

} // namespace

const RunPlan* aprnet_get_run_plan(aprnet_apr* a, int dl, cudaStream_t st) {
    auto it = a->run_plans.find(dl);
    if (it != a->run_plans.end()) return &it->second;
    if (aprnet_check_device(a) != APRNET_OK) return nullptr;
    RunPlan rp;
    if (build_run_plan(a, dl, rp, st) != APRNET_OK) { cudaFree(rp.loc); cudaFree(rp.src); return nullptr; }
    return &a->run_plans.emplace(dl, rp).first->second;
}

// Builds (once; cached) the run plan of a level delta.  Allocates; call it up front.
extern "C" int aprnet_run_plan_build(aprnet_apr* a, int dl, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl), "bad handle or level_delta");
    return aprnet_get_run_plan(a, dl, (cudaStream_t) stream) ? APRNET_OK : APRNET_ERR_CUDA;
}
