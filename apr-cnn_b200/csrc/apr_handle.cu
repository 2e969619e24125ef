// Device-side APR access structure, tree child table and per-level_delta neighbour tables.
//
// The reference re-derives "which rows hold anything" and re-stages dense (z, x, y) patches on every
// forward and backward call (pyapr/aprnet/cuda/src/nonempty_rows.cu:26-230,
// conv333_gpu.cu:63-118, fill_tree_gpu.cu:1098).  Here the sparse-row searches run once per APR
// (child table) and once per (APR, level_delta) (neighbour table); the hot kernels are pure
// index-driven gathers.
#include "apr_device.cuh"
#include <cstring>
#include <mutex>
#include <algorithm>

static thread_local std::string g_last_error;

void aprnet_set_error(const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_last_error = buf;
}

extern "C" const char* aprnet_last_error(void) { return g_last_error.c_str(); }

// ---- memory of the cached tables and of their construction ------------------------------------------
// One stream-ordered pool per device, shared by all handles.  cudaMalloc / cudaFree cost about 0.9 and 0.5 ms per table, which was
// most of the time it took to prepare an access structure.  What is freed (temporaries, the tables of a destroyed handle) stays for
// the next structure up to POOL_SPARE bytes above what is in use; the driver gives the rest back at the next synchronisation.  When a
// device's last structure is destroyed, all but POOL_IDLE goes back.
// The driver's allocator is safe with several threads and streams.
namespace {
constexpr unsigned long long POOL_SPARE = 2ull << 30, POOL_IDLE = 256ull << 20;
constexpr int POOL_DEVICES = 64;
std::mutex g_pool_mutex;
cudaMemPool_t g_pools[POOL_DEVICES] = {};
int g_structures[POOL_DEVICES] = {};           // alive on the device

cudaMemPool_t pool_of_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= POOL_DEVICES) { cudaGetLastError(); return nullptr; }
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (!g_pools[dev]) {
        cudaMemPoolProps props;
        memset(&props, 0, sizeof(props));
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        if (cudaMemPoolCreate(&g_pools[dev], &props) != cudaSuccess) { cudaGetLastError(); g_pools[dev] = nullptr; }
    }
    return g_pools[dev];
}

void pool_keep(cudaMemPool_t pool) {          // reserved memory the pool may hold: what is in use and POOL_SPARE on top
    unsigned long long used = 0;
    if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) { cudaGetLastError(); return; }
    used += POOL_SPARE;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &used);
}
}

static void count_structure(int device, int change) {
    if (device < 0 || device >= POOL_DEVICES) return;
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    g_structures[device] += change;
    if (g_structures[device] > 0 || change > 0 || !g_pools[device]) return;
    if (cudaStreamSynchronize(0) != cudaSuccess || cudaMemPoolTrimTo(g_pools[device], POOL_IDLE) != cudaSuccess) cudaGetLastError();
}

int aprnet_pool_alloc(void** p, size_t bytes, cudaStream_t st) {
    *p = nullptr;
    cudaMemPool_t pool = pool_of_device();
    if (!pool) { aprnet_set_error("no memory pool on this device"); return APRNET_ERR_CUDA; }
    const cudaError_t e = cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 16), pool, st);
    if (e != cudaSuccess) { *p = nullptr; cudaGetLastError(); aprnet_set_error("allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e)); return APRNET_ERR_CUDA; }
    pool_keep(pool);
    return APRNET_OK;
}

void aprnet_pool_free(void* p, cudaStream_t st) {
    if (!p) return;
    cudaFreeAsync(p, st);
    if (cudaMemPool_t pool = pool_of_device()) pool_keep(pool);
}

// ---- per-kernel event timing -----------------------------------------------------------------
namespace {
struct ProfRecord { std::string name; cudaEvent_t start, stop; };
bool g_prof_on = false;
std::vector<ProfRecord> g_prof_records;
}

AprnetProfScope::AprnetProfScope(const char* name, cudaStream_t st) : slot(-1), stream(st) {
    if (!g_prof_on) return;
    ProfRecord r;
    r.name = name;
    if (cudaEventCreate(&r.start) != cudaSuccess || cudaEventCreate(&r.stop) != cudaSuccess) return;
    cudaEventRecord(r.start, st);
    g_prof_records.push_back(r);
    slot = (int) g_prof_records.size() - 1;
}

AprnetProfScope::~AprnetProfScope() {
    if (slot >= 0) cudaEventRecord(g_prof_records[slot].stop, stream);
}

extern "C" void aprnet_profile_enable(int on) { g_prof_on = on != 0; }

extern "C" int64_t aprnet_profile_read(char* buf, int64_t buflen) {
    std::map<std::string, std::pair<long long, double>> agg;
    for (ProfRecord& r : g_prof_records) {
        float ms = 0;
        if (cudaEventSynchronize(r.stop) == cudaSuccess && cudaEventElapsedTime(&ms, r.start, r.stop) == cudaSuccess) {
            agg[r.name].first += 1;
            agg[r.name].second += ms;
        }
        cudaEventDestroy(r.start);
        cudaEventDestroy(r.stop);
    }
    g_prof_records.clear();
    std::string out;
    for (auto& kv : agg) {
        char line[256];
        snprintf(line, sizeof(line), "%s %lld %.6f\n", kv.first.c_str(), kv.second.first, kv.second.second);
        out += line;
    }
    if (buf && buflen > 0) {
        const size_t n = std::min<size_t>(out.size(), (size_t) buflen - 1);
        memcpy(buf, out.data(), n);
        buf[n] = 0;
    }
    return (int64_t) out.size();
}

namespace {

typedef long long ll;

// first position in [b, e) whose y is >= target
__device__ __forceinline__ ll lower_bound_y(const uint16_t* __restrict__ y, ll b, ll e, int target) {
    while (b < e) {
        const ll mid = (b + e) >> 1;
        if ((int) y[mid] < target) b = mid + 1; else e = mid;
    }
    return b;
}

// One warp per tree row of level `l`; lanes stride over the row's nodes.
__global__ void build_child_table_kernel(LevelMeta m, const ll* __restrict__ row_ptr, const uint16_t* __restrict__ y,
                                         const ll* __restrict__ trow_ptr, const uint16_t* __restrict__ ty,
                                         int32_t* __restrict__ child, float* __restrict__ scale, ll n_tree, int l) {
    const ll row = ((ll) blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const ll rows = (ll) m.z_num[l] * m.x_num[l];
    if (row >= rows) return;
    const int z = (int) (row / m.x_num[l]), x = (int) (row % m.x_num[l]);
    const ll tr = m.trow_off[l] + row;
    const ll tb = trow_ptr[tr], te = trow_ptr[tr + 1];
    const int cl = l + 1;
    const int bx = ((2 * m.x_num[l]) != m.x_num[cl]) && (x == m.x_num[l] - 1);
    const int bz = ((2 * m.z_num[l]) != m.z_num[cl]) && (z == m.z_num[l] - 1);
    const float f_xz = fmaxf(2.0f * (float) (bx + bz), 1.0f) / 8.0f;
    const bool y_odd = (2 * m.y_num[l]) != m.y_num[cl];
    const bool child_tree = cl <= m.level_max - 1;

    for (ll t = tb + lane; t < te; t += 32) {
        const int yp = ty[t];
        scale[t] = (y_odd && yp == m.y_num[l] - 1) ? 2.0f * f_xz : f_xz;
        for (int s4 = 0; s4 < 4; ++s4) {
            const int cz = 2 * z + (s4 >> 1), cx = 2 * x + (s4 & 1);
            int32_t v0 = APRNET_NONE, v1 = APRNET_NONE;
            if (cz < m.z_num[cl] && cx < m.x_num[cl]) {
                const ll crow = (ll) cz * m.x_num[cl] + cx;
                const ll pr = m.row_off[cl] + crow;
                const ll pb = row_ptr[pr], pe = row_ptr[pr + 1];
                ll p = lower_bound_y(y, pb, pe, 2 * yp);
                if (p < pe && (int) y[p] == 2 * yp) { v0 = (int32_t) p; ++p; }
                if (p < pe && (int) y[p] == 2 * yp + 1) v1 = (int32_t) p;
                if (child_tree && (v0 == APRNET_NONE || v1 == APRNET_NONE)) {
                    const ll ctr = m.trow_off[cl] + crow;
                    const ll cb = trow_ptr[ctr], ce = trow_ptr[ctr + 1];
                    ll q = lower_bound_y(ty, cb, ce, 2 * yp);
                    if (q < ce && (int) ty[q] == 2 * yp) { if (v0 == APRNET_NONE) v0 = aprnet_enc_tree(q); ++q; }
                    if (q < ce && (int) ty[q] == 2 * yp + 1 && v1 == APRNET_NONE) v1 = aprnet_enc_tree(q);
                }
            }
            child[(ll) (2 * s4) * n_tree + t] = v0;
            child[(ll) (2 * s4 + 1) * n_tree + t] = v1;
        }
    }
}

template<typename T>
int upload(T** dst, const T* src, size_t n, long long* bytes) {
    const int rc = aprnet_pool_alloc((void**) dst, std::max<size_t>(n, 1) * sizeof(T), 0);
    if (rc) return rc;
    if (n) APRNET_CUDA_CHECK(cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice));
    *bytes += (long long) (std::max<size_t>(n, 1) * sizeof(T));
    return APRNET_OK;
}

} // namespace

std::vector<Segment> aprnet_segments(const aprnet_apr* apr, int dl, int num_slots, bool merge) {
    std::vector<Segment> segs;
    const int cml = apr->cml(dl);
    const long long N = apr->number_parts(dl);
    for (int l = apr->meta.level_min; l <= cml; ++l) {
        Segment s;
        s.begin = apr->meta.lvl_begin[l];
        s.end = (l == cml) ? N : apr->meta.lvl_begin[l + 1];
        s.slot = std::min(cml - l, num_slots - 1);
        s.level = l;
        if (s.end <= s.begin) continue;
        if (merge && !segs.empty() && segs.back().slot == s.slot && segs.back().end == s.begin) segs.back().end = s.end;
        else segs.push_back(s);
    }
    return segs;
}

extern "C" int aprnet_apr_create(aprnet_apr** out, int level_min, int level_max, const int* dims,
                                 const int64_t* row_ptr, const uint16_t* y,
                                 const int64_t* tree_row_ptr, const uint16_t* tree_y, int device) {
    APRNET_ARG_CHECK(out && dims && row_ptr && tree_row_ptr, "null argument");
    APRNET_ARG_CHECK(level_min >= 1 && level_max >= level_min && level_max < APRNET_MAX_LEVELS - 1, "bad level range");
    // the structure is built on `device`; the caller's current device is restored on every way out
    struct DeviceRestore { int prev = -1; ~DeviceRestore() { if (prev >= 0) cudaSetDevice(prev); } } restore;
    if (cudaGetDevice(&restore.prev) != cudaSuccess) { restore.prev = -1; cudaGetLastError(); }
    APRNET_CUDA_CHECK(cudaSetDevice(device));
    aprnet_apr* a = new aprnet_apr();
    a->device = device;
    LevelMeta& m = a->meta;
    memset(&m, 0, sizeof(m));
    m.level_min = level_min; m.level_max = level_max;
    for (int l = 0; l <= level_max; ++l) { m.z_num[l] = dims[3 * l]; m.x_num[l] = dims[3 * l + 1]; m.y_num[l] = dims[3 * l + 2]; }
    for (int l = 0; l <= level_max; ++l) {
        m.row_off[l + 1] = m.row_off[l] + (l >= level_min ? (long long) m.z_num[l] * m.x_num[l] : 0);
        m.trow_off[l + 1] = m.trow_off[l] + ((l >= level_min - 1 && l <= level_max - 1) ? (long long) m.z_num[l] * m.x_num[l] : 0);
    }
    for (int l = level_max + 1; l < APRNET_MAX_LEVELS; ++l) { m.row_off[l + 1] = m.row_off[l]; m.trow_off[l + 1] = m.trow_off[l]; }
    a->n_rows = m.row_off[level_max + 1];
    a->n_tree_rows = m.trow_off[level_max];
    for (int l = 0; l <= APRNET_MAX_LEVELS; ++l) {
        m.lvl_begin[l] = row_ptr[std::min(m.row_off[std::min(l, APRNET_MAX_LEVELS)], a->n_rows)];
        m.tlvl_begin[l] = tree_row_ptr[std::min(m.trow_off[std::min(l, APRNET_MAX_LEVELS)], a->n_tree_rows)];
    }
    a->n_particles = row_ptr[a->n_rows];
    a->n_tree = tree_row_ptr[a->n_tree_rows];
    if (a->n_particles >= (1ll << 31) - 2 || a->n_tree >= (1ll << 31) - 2) {
        delete a;
        aprnet_set_error("aprnet_apr_create: more than 2^31 particles are not supported by the 32-bit tables");
        return APRNET_ERR_UNSUPPORTED;
    }
    static_assert(sizeof(long long) == sizeof(int64_t), "int64 layout");
    count_structure(device, +1);
    int rc;
    if ((rc = upload(&a->row_ptr, (const long long*) row_ptr, (size_t) a->n_rows + 1, &a->device_bytes))) { aprnet_apr_destroy(a); return rc; }
    if ((rc = upload(&a->y, y, (size_t) a->n_particles, &a->device_bytes))) { aprnet_apr_destroy(a); return rc; }
    if ((rc = upload(&a->tree_row_ptr, (const long long*) tree_row_ptr, (size_t) a->n_tree_rows + 1, &a->device_bytes))) { aprnet_apr_destroy(a); return rc; }
    if ((rc = upload(&a->tree_y, tree_y, (size_t) a->n_tree, &a->device_bytes))) { aprnet_apr_destroy(a); return rc; }

    const size_t nt = (size_t) std::max<long long>(a->n_tree, 1);
    if ((rc = aprnet_pool_alloc((void**) &a->child, 8 * nt * sizeof(int32_t), 0)) || (rc = aprnet_pool_alloc((void**) &a->tree_scale, nt * sizeof(float), 0))) {
        aprnet_apr_destroy(a);
        return rc;
    }
    a->device_bytes += (long long) (8 * nt * sizeof(int32_t) + nt * sizeof(float));
    for (int l = level_min - 1; l <= level_max - 1; ++l) {
        const long long rows = (long long) m.z_num[l] * m.x_num[l];
        const int blocks = aprnet_ceil_div(rows * 32, 128);
        build_child_table_kernel<<<blocks, 128>>>(m, a->row_ptr, a->y, a->tree_row_ptr, a->tree_y, a->child,
                                                  a->tree_scale, a->n_tree, l);
    }
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        aprnet_set_error("aprnet_apr_create: child table: %s", cudaGetErrorString(e));
        aprnet_apr_destroy(a);
        return APRNET_ERR_CUDA;
    }
    *out = a;
    return APRNET_OK;
}

extern "C" void aprnet_apr_destroy(aprnet_apr* a) {
    if (!a) return;
    int prev = -1;
    if (cudaGetDevice(&prev) != cudaSuccess) { prev = -1; cudaGetLastError(); }
    cudaSetDevice(a->device);
    cudaDeviceSynchronize();          // no stream uses the tables any more
    void* owned[] = {a->row_ptr, a->y, a->tree_row_ptr, a->tree_y, a->child, a->tree_scale, a->node_parent};
    for (void* p : owned) aprnet_pool_free(p, 0);
    for (auto& kv : a->plans) aprnet_pool_free(kv.second.nbr, 0);
    for (auto& kv : a->loc_parent) aprnet_pool_free(kv.second, 0);
    for (auto& kv : a->edge_plans) aprnet_free_edge_plan(kv.second, 0);
    for (auto& kv : a->run_plans) { aprnet_pool_free(kv.second.loc, 0); aprnet_pool_free(kv.second.src, 0); }
    count_structure(a->device, -1);
    delete a;
    if (prev >= 0) cudaSetDevice(prev);
}

// Every entry point launches on the current device with pointers that live on the handle's device: a mismatch is
// an argument error here instead of an illegal address inside a kernel.
int aprnet_check_device(const aprnet_apr* a) {
    int cur = -1;
    if (cudaGetDevice(&cur) != cudaSuccess) { cudaGetLastError(); aprnet_set_error("no current CUDA device"); return APRNET_ERR_CUDA; }
    if (a && cur != a->device) {
        aprnet_set_error("the access structure lives on device %d but the current device is %d", a->device, cur);
        return APRNET_ERR_ARG;
    }
    return APRNET_OK;
}

extern "C" int64_t aprnet_number_parts(const aprnet_apr* a, int dl) { return (a && a->valid_dl(dl)) ? a->number_parts(dl) : -1; }
extern "C" int64_t aprnet_tree_size(const aprnet_apr* a, int dl) { return (a && a->valid_dl(dl)) ? a->tree_size(dl) : -1; }
extern "C" int64_t aprnet_total_tree_nodes(const aprnet_apr* a) { return a ? a->n_tree : -1; }
extern "C" int64_t aprnet_device_bytes(const aprnet_apr* a) { return a ? a->device_bytes : -1; }

const AprPlan* aprnet_get_plan(aprnet_apr* a, int dl, cudaStream_t stream) {
    if (aprnet_check_device(a) != APRNET_OK) return nullptr;
    auto it = a->plans.find(dl);
    if (it != a->plans.end()) return &it->second;
    if (aprnet_rows_overflow(a, dl)) return nullptr;
    AprPlan p;
    p.level_delta = dl;
    p.n = a->number_parts(dl);
    p.tree_size = a->tree_size(dl);
    const size_t bytes = 27 * (size_t) std::max<long long>(p.n, 1) * sizeof(int32_t);
    if (aprnet_pool_alloc((void**) &p.nbr, bytes, stream)) return nullptr;
    if (aprnet_fill_nbr_table(a, dl, p.nbr, p.n, stream)) { aprnet_pool_free(p.nbr, stream); return nullptr; }
    a->device_bytes += (long long) bytes;
    auto res = a->plans.emplace(dl, p);
    return &res.first->second;
}

// Parent tables from the child table: every child slot of tree node t names a particle (v >= 0), a tree node (coded) or,
// from the node up_from on (the finest tree level of a level delta > 0), an upgraded node that lives in the feature vector at
// up_off + index.  Either output may be null.
__global__ void build_parent_tables_kernel(const int32_t* __restrict__ child, long long n_tree, long long tb, long long te,
                                           long long up_off, long long up_from, int32_t* __restrict__ loc_parent, int32_t* __restrict__ node_parent) {
    const long long t = tb + (long long) blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= te) return;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const int32_t v = child[(long long) s * n_tree + t];
        if (v >= 0) { if (loc_parent) loc_parent[v] = (int32_t) t; }
        else if (v != APRNET_NONE) {
            if (t >= up_from) { if (loc_parent) loc_parent[aprnet_dec_tree(v) + up_off] = (int32_t) t; }
            else if (node_parent) node_parent[aprnet_dec_tree(v)] = (int32_t) t;
        }
    }
}

static int32_t* alloc_minus_one(const aprnet_apr* a, long long n, cudaStream_t stream) {
    int32_t* p = nullptr;
    n = std::max<long long>(n, 1);
    if (aprnet_pool_alloc((void**) &p, (size_t) n * sizeof(int32_t), stream)) return nullptr;
    a->device_bytes += n * (long long) sizeof(int32_t);
    cudaMemsetAsync(p, 0xFF, (size_t) n * sizeof(int32_t), stream);
    return p;
}

const int32_t* aprnet_node_parent_table(const aprnet_apr* a, cudaStream_t stream) {
    if (a->node_parent) return a->node_parent;
    int32_t* tab = alloc_minus_one(a, a->n_tree, stream);
    if (!tab) return nullptr;
    if (a->n_tree > 0) build_parent_tables_kernel<<<aprnet_ceil_div(a->n_tree, 256), 256, 0, stream>>>(a->child, a->n_tree, 0, a->n_tree, 0, a->n_tree, nullptr, tab);
    if (cudaGetLastError() != cudaSuccess) { aprnet_set_error("aprnet_node_parent_table: kernel launch failed"); aprnet_pool_free(tab, stream); return nullptr; }
    if (cudaStreamSynchronize(stream) != cudaSuccess) return nullptr;          // usable on any stream from here on
    a->node_parent = tab;
    return tab;
}

const int32_t* aprnet_loc_parent_table(const aprnet_apr* a, int dl, cudaStream_t stream) {
    auto it = a->loc_parent.find(dl);
    if (it != a->loc_parent.end()) return it->second;
    int32_t* tab = alloc_minus_one(a, a->number_parts(dl), stream);
    if (!tab) return nullptr;
    const LevelMeta& m = a->meta;
    const int cml = a->cml(dl);
    const long long te = m.tlvl_begin[cml];          // nodes of levels below cml
    if (te > 0) build_parent_tables_kernel<<<aprnet_ceil_div(te, 256), 256, 0, stream>>>(a->child, a->n_tree, 0, te, dl > 0 ? a->tree_offset(cml) : 0,
                                                                                       dl > 0 ? m.tlvl_begin[cml - 1] : te, tab, nullptr);
    if (cudaGetLastError() != cudaSuccess) { aprnet_set_error("aprnet_loc_parent_table: kernel launch failed"); aprnet_pool_free(tab, stream); return nullptr; }
    if (cudaStreamSynchronize(stream) != cudaSuccess) return nullptr;
    a->loc_parent.emplace(dl, tab);
    return tab;
}

extern "C" int aprnet_plan_build(aprnet_apr* a, int dl, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl), "bad handle or level_delta");
    APRNET_DEVICE_CHECK(a);
    if (!aprnet_get_run_plan(a, dl, (cudaStream_t) stream)) return APRNET_ERR_CUDA;          // first: the neighbour table is derived from it
    if (!aprnet_get_plan(a, dl, (cudaStream_t) stream)) return APRNET_ERR_CUDA;
    if (!aprnet_node_parent_table(a, (cudaStream_t) stream) || !aprnet_loc_parent_table(a, dl, (cudaStream_t) stream)) return APRNET_ERR_CUDA;
    return APRNET_OK;
}

extern "C" int aprnet_plan_copy_nbr_table(aprnet_apr* a, int dl, int32_t* host_out) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && host_out, "bad argument");
    const AprPlan* p = aprnet_get_plan(a, dl, 0);
    if (!p) return APRNET_ERR_CUDA;
    APRNET_CUDA_CHECK(cudaDeviceSynchronize());
    APRNET_CUDA_CHECK(cudaMemcpy(host_out, p->nbr, 27 * (size_t) p->n * sizeof(int32_t), cudaMemcpyDeviceToHost));
    return APRNET_OK;
}

extern "C" int aprnet_copy_child_table(aprnet_apr* a, int32_t* host_out) {
    APRNET_ARG_CHECK(a && host_out, "bad argument");
    APRNET_CUDA_CHECK(cudaMemcpy(host_out, a->child, 8 * (size_t) a->n_tree * sizeof(int32_t), cudaMemcpyDeviceToHost));
    return APRNET_OK;
}
