// Internal definitions shared by the CUDA translation units of libaprnet_b200.
#pragma once

#include <cstdint>
#include <cstdio>
#include <cstdarg>
#include <string>
#include <vector>
#include <map>
#include <algorithm>
#include <cuda_runtime.h>
#include "../../include/aprnet_b200.h"

#define APRNET_MAX_LEVELS 20

// Encoding of neighbour / child table entries:
//   v >= 0 : index into the feature vector (APR particle, or upgraded tree node stored behind them)
//   v == -1: nothing there (outside the domain) -> value 0
//   v <= -2: tree node t = -2 - v (value comes from the tree scratch)
#define APRNET_NONE (-1)
__host__ __device__ inline int32_t aprnet_enc_tree(long long t) { return (int32_t) (-2 - t); }
__host__ __device__ inline long long aprnet_dec_tree(int32_t v) { return -2 - (long long) v; }

// Per-level geometry and index ranges; passed to kernels by value.
struct LevelMeta {
    int level_min, level_max;                    // particle levels; the tree spans level_min-1 .. level_max-1
    int z_num[APRNET_MAX_LEVELS], x_num[APRNET_MAX_LEVELS], y_num[APRNET_MAX_LEVELS];
    long long row_off[APRNET_MAX_LEVELS + 1];    // first particle row of each level
    long long trow_off[APRNET_MAX_LEVELS + 1];   // first tree row of each level
    long long lvl_begin[APRNET_MAX_LEVELS + 1];  // first particle index of each level ([l+1] = end of l)
    long long tlvl_begin[APRNET_MAX_LEVELS + 1]; // first tree node index of each level
};

struct AprPlan {                 // cached per level_delta
    int level_delta = 0;
    long long n = 0;             // number of output locations (= number_parts)
    long long tree_size = 0;
    int32_t* nbr = nullptr;      // [27][n]
};

// Cross-level edges of one level_delta: every (output location p, tap) whose source ("target" of the
// gradient) is a coarser particle or a tree node.  Targets are numbered as particle index, or
// N + tree index.  The edges of one (target, tap) meet the same weight matrix: where there are several, their dO rows are summed
// before the contraction into a "virtual row"; a single one (every tap of a tree node, most of a particle's) is that location's row
// itself.  Virtual rows are numbered by ascending target, then tap; vsrc[vstart[v] .. vstart[v + 1]) lists the locations p of row v in
// ascending order.  active[] lists the targets that have at least one edge (ascending), vnbr[tap][a] is the virtual row of
// (active[a], tap), the location encoded like a tree node (<= -2), or -1.
struct ActiveSeg { long long begin, end; int location_level; };     // range of active[] whose edges come from one level
struct EdgePlan {
    long long n_edges = 0, n_targets = 0, n_active = 0, n_vrows = 0;
    int32_t* vsrc = nullptr;       // [locations of all virtual rows]
    int32_t* vstart = nullptr;     // [n_vrows + 1]
    int32_t* active = nullptr;     // [n_active]
    int32_t* vnbr = nullptr;       // [27][n_active]
    std::vector<ActiveSeg> segs;   // by level, in active[] order
    // coarse map for splitting the work when the virtual rows do not fit the workspace: chunk k starts at
    // active index chunk_a[k] and virtual row chunk_v[k]; a chunk holds at most APRNET_VROW_CHUNK rows
    std::vector<long long> chunk_a, chunk_v;
};

// A chunk ends with the target that reaches the granule, which adds at most 27 rows.  The workspace of the virtual rows is bounded by
// 8 GiB, but never smaller than one chunk, whatever the width of a row; one pass takes as many chunks as fit.
constexpr long long APRNET_VROW_GRANULE = 64ll << 10, APRNET_VROW_CHUNK = APRNET_VROW_GRANULE + 27;
inline long long aprnet_vrow_workspace_bytes(long long n_vrows, long long row_bytes) {
    const long long cap = std::max(8ll << 30, (APRNET_VROW_CHUNK + 2) * row_bytes);
    return std::max<long long>(256, std::min(cap, (n_vrows + 2) * row_bytes));
}
// first chunk that no longer fits a pass of cap_rows rows from chunk k0 on
inline int aprnet_vrow_pass_end(const std::vector<long long>& chunk_v, int k0, long long cap_rows) {
    int k1 = k0 + 1;
    while (k1 + 1 < (int) chunk_v.size() && chunk_v[k1 + 1] - chunk_v[k0] <= cap_rows) ++k1;
    return k1;
}

// Output locations of a level delta in runs along y (run_plan.cu): slot s is a cell of its level, loc[s] the location it holds
// (-1: none), src[d][s] what fills the cell (dz, dx) = (d / 3 - 1, d % 3 - 1) away (encoded like the neighbour table).
struct RunPlan {
    long long n_slots = 0;
    std::vector<long long> level_begin;      // first slot of each level ([l + 1] = end of l)
    int32_t* loc = nullptr;                  // [n_slots]
    int32_t* src = nullptr;                  // [9][n_slots]
};

struct aprnet_apr {
    int device = 0;
    LevelMeta meta;
    long long n_particles = 0, n_tree = 0, n_rows = 0, n_tree_rows = 0;
    long long* row_ptr = nullptr;        // device
    uint16_t* y = nullptr;
    long long* tree_row_ptr = nullptr;
    uint16_t* tree_y = nullptr;
    int32_t* child = nullptr;            // [8][n_tree]
    float* tree_scale = nullptr;         // [n_tree] weight of each child in its parent's mean
    std::map<int, AprPlan> plans;
    std::map<int, EdgePlan> edge_plans;
    std::map<int, RunPlan> run_plans;
    // parent tree node of every tree node (-1: none) and, per level delta, of every feature location (particle or
    // upgraded node); built on first use by the tree-mean adjoint (aprnet_node_parent_table / aprnet_loc_parent_table)
    mutable int32_t* node_parent = nullptr;
    mutable std::map<int, int32_t*> loc_parent;
    mutable long long device_bytes = 0;

    int cml(int dl) const { return meta.level_max - dl; }
    long long number_parts(int dl) const {
        const int c = cml(dl);
        long long n = meta.lvl_begin[c + 1];
        if (c <= meta.level_max - 1) n += meta.tlvl_begin[c + 1] - meta.tlvl_begin[c];
        return n;
    }
    long long tree_size(int dl) const { return meta.tlvl_begin[cml(dl)]; }   // nodes of levels <= cml-1
    long long tree_offset(int level) const { return meta.lvl_begin[level + 1] - meta.tlvl_begin[level]; }
    bool valid_dl(int dl) const { return dl >= 0 && cml(dl) >= meta.level_min; }
};

void aprnet_set_error(const char* fmt, ...);

// Packed operands have a row per location, per tree node and one of zeros; the kernels hold row numbers in 32 bits.
inline bool aprnet_rows_overflow(const aprnet_apr* a, int dl) {
    if (a->number_parts(dl) + a->tree_size(dl) + 1 < (1ll << 31)) return false;
    aprnet_set_error("%lld locations and %lld tree nodes exceed the 32-bit row numbers of the convolutions", a->number_parts(dl), a->tree_size(dl));
    return true;
}
int aprnet_check_device(const aprnet_apr* a);      // APRNET_OK when the current device is the handle's device

#define APRNET_CUDA_CHECK(expr)                                                                     \
    do {                                                                                            \
        cudaError_t _e = (expr);                                                                    \
        if (_e != cudaSuccess) {                                                                    \
            aprnet_set_error("%s failed at %s:%d: %s", #expr, __FILE__, __LINE__, cudaGetErrorString(_e)); \
            return APRNET_ERR_CUDA;                                                                 \
        }                                                                                           \
    } while (0)

#define APRNET_LAUNCH_CHECK() APRNET_CUDA_CHECK(cudaGetLastError())

// Chains of short kernels: a kernel launched with `behind` starts while the launch before it on the stream still runs, once all blocks of that one have started and called
// let_next_grid_start() or have ended.  Up to wait_for_grid_before() it may only read what was there before the chain's first launch, which is an ordinary one: tables and
// inputs, not what the chain writes; it writes nothing up to there.  Every block of such a kernel waits, so that the end of one launch is the end of all before it.
// (Reads behind the wait go through pointers without __restrict__: loads of what the compiler takes for constant are free to move.)
template<typename... P, typename... A>
inline void aprnet_launch(bool behind, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cfg.attrs = &attr; cfg.numAttrs = behind ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);             // (an error stays for APRNET_LAUNCH_CHECK)
}
#ifdef __CUDACC__
__device__ __forceinline__ void let_next_grid_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_grid_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

#define APRNET_ARG_CHECK(cond, msg)                                                                 \
    do { if (!(cond)) { aprnet_set_error("%s: %s", __func__, msg); return APRNET_ERR_ARG; } } while (0)

#define APRNET_DEVICE_CHECK(a)                                                                      \
    do { const int _rc = aprnet_check_device(a); if (_rc != APRNET_OK) return _rc; } while (0)

inline int aprnet_ceil_div(long long a, long long b) { return (int) ((a + b - 1) / b); }

// A contiguous range of output locations that shares one stencil slot.
struct Segment { long long begin, end; int slot; int level; };
// Segments of level_delta dl for a filter bank with `num_slots` slots: level l -> slot
// min(cml - l, num_slots - 1); the upgraded tree nodes ride with the level-cml particles.
// With merge=true, consecutive levels that share a slot are fused into one range (1x1x1 conv).
std::vector<Segment> aprnet_segments(const aprnet_apr* apr, int dl, int num_slots, bool merge);

// memory of the cached tables and of their construction (one pool per device)
int aprnet_pool_alloc(void** p, size_t bytes, cudaStream_t st);
void aprnet_pool_free(void* p, cudaStream_t st);

int aprnet_fill_nbr_table(aprnet_apr* a, int dl, int32_t* nbr, long long n, cudaStream_t st);
const AprPlan* aprnet_get_plan(aprnet_apr* apr, int dl, cudaStream_t stream);
const int32_t* aprnet_node_parent_table(const aprnet_apr* apr, cudaStream_t stream);            // nullptr on failure
const int32_t* aprnet_loc_parent_table(const aprnet_apr* apr, int dl, cudaStream_t stream);     // nullptr on failure

// Optional per-kernel timing (aprnet_profile_enable): brackets a launch site with two CUDA events on
// the launching stream.  Costs nothing when profiling is off.
struct AprnetProfScope {
    int slot;
    cudaStream_t stream;
    AprnetProfScope(const char* name, cudaStream_t st);
    ~AprnetProfScope();
};

// tensor-core helpers shared between translation units (conv333_tc.cu / conv333_tc_dw.cu)
int* aprnet_tc_error_flag_device();
extern "C" int aprnet_conv333_backward_weights_tc(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* xrows, int xpad,
                                                  const void* grows, int gpad, float* gw, float* partial, void* stream);
extern "C" int64_t aprnet_conv333_tc_dw_partial_elems(int cin, int cout);
extern "C" int aprnet_conv333_backward_input_cross_level(aprnet_apr* a, int dl, int dtype, int cin, int cout, int slots,
                                                         const void* gout, int64_t ld_out, const void* w, void* gin,
                                                         int64_t ld_in, void* gtree, int64_t ld_tree, void* stream);

// cross-level part by atomic adds (fp32; grad_tree is zero-filled and, with tree_adjoint, folded into grad_input)
int aprnet_cross_level_scatter(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* gout, long long ld_out, const float* w, float* gin, long long ld_in,
                               float* gtree, long long ld_tree, bool tree_adjoint, cudaStream_t st);
const RunPlan* aprnet_get_run_plan(aprnet_apr* apr, int dl, cudaStream_t stream);                // nullptr on failure
EdgePlan* aprnet_get_edge_plan(aprnet_apr* apr, int dl, cudaStream_t stream);
void aprnet_free_edge_plan(EdgePlan& ep, cudaStream_t st);
// gather GEMM over the active targets [a0, a1) of an edge plan: grad[target] += sum over taps of W[slot][:, :, tap]^T times the row
// of vnbr[tap][a]; rows are addressed from grows: location p at row p (zeros at row n_split = N), virtual row v at row v + v_shift
int aprnet_tc_gather_targets(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* grows, int gpad, long long v_shift,
                             const void* wp_packed, const EdgePlan* ep, long long a0, long long a1,
                             float* gin, long long ld_in, float* gtree, long long ld_tree, cudaStream_t st);
// CUDA-core fp32 kernels for Cin <= 4 (conv333_small.cu), used in either arithmetic for such layers:
// vals = channel-major staging buffer [cin][N + T + 1] (particles, tree means, zero)
bool aprnet_small_cin(int cin);
int aprnet_small_stage(const float* x, long long ld_x, long long n, const float* tree, long long ld_tree, long long t, int cin, float* vals, cudaStream_t st);
int aprnet_small_forward(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* vals, const float* w, const float* bias, float* out, long long ld_out, cudaStream_t st);
int aprnet_small_backward_weights(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* vals, const float* gout, long long ld_out,
                                  float* gw, int accumulate, float* partial, cudaStream_t st);
// fp32 gather kernel (conv333_f32.cu): blocks of four locations per lane up to which the form with one location per lane, four times as many blocks, is the faster
// one.  Its time grows with the blocks it puts on an SM.  Time of one location per lane / of four, where it puts 1, 2, 3 and 4 blocks on an SM (up to 37, 74, 111 and 148
// blocks of four): tiles of 64 result channels, forward pass 0.6, 0.77, 0.92, 1.1 to 1.25, same-level input gradient 0.65, 0.95, 1.26, 1.43, cross-level 0.62, 0.9, 1.16, 1.35; 32
// channels, forward pass and same-level input gradient, 0.47, 0.65, 0.77, 1.0 and 0.56, 0.77, 0.97, 1.2; 16 channels 0.5, 0.6, 0.72, 0.85 and 0.6, 0.78, 0.9, 1.08; 8 channels 0.55, 0.61, 0.7, 0.75 and 0.8, 0.9, 1.0, 1.1.
inline int aprnet_f32_few_blocks(int tile_channels, bool forward) { return 37 * ((tile_channels == 64 ? 2 : 3) + (forward ? 1 : 0)); }
// Blocks of four locations per lane from which 512 threads per SM are faster than 384 (forward pass of 64 result channels, same-level input gradient of 32): beyond the three blocks per
// SM that 384 threads hold.  Time with 384 / with 512 threads up to 148, 296 and 444 blocks and beyond 900: 64 channels 0.96, 0.98, 0.98 and 1.01; 32 channels, 32 and more source
// channels, 0.87, 0.98, 1.01 and 1.05; 24 0.81, 0.93, 0.95 and 1.01; 16 0.87, 0.95, 0.95 and 0.98; 8 0.86, 0.87, 0.89 and 0.88.
inline bool aprnet_f32_many_blocks(int tile_channels, int source_channels, long long blocks) { return blocks > 3 * 148 && (tile_channels == 64 || source_channels > 16); }
// tensor-core gather over runs (conv333_tc_runs.cu)
inline int aprnet_run_max_height(int nt) { return nt >= 64 ? 2 : 4; }      // blocks of 128 rows in a tile of nt result channels, at most (pick_h has the times)
constexpr int APRNET_TAP_KERNEL = 1;      // of aprnet_tc_run_conv: nothing was launched, the kernel that gathers every tap is the faster one
int aprnet_tc_runs_order(int backward, int kpad, int nt_order, int nt, int ks);
int aprnet_tc_run_conv(aprnet_apr* a, int dl, int backward, int slots, int nt, int order, const void* rows, int kpad, long long tree_base, long long zero_row, const void* wp,
                       const float* bias, float* out, long long ld_out, int n_dim, int* error_flag, cudaStream_t st, const char* pname);
int aprnet_pack_weights(const aprnet_apr* a, int dl, bool bf16, const float* w, int slots, int cin, int cout, int transposed, int nt, int n_tiles, int kpad,
                        void* out, cudaStream_t st);
int aprnet_tc_pack_weights(const aprnet_apr* a, int dl, const float* w, int slots, int cin, int cout, int transposed, void* wp, cudaStream_t st);
size_t aprnet_tc_weight_bytes(int k_dim, int n_dim, int slots);
size_t aprnet_tc_rows_bytes(long long rows, int channels);
int aprnet_tc_pad(int channels);
extern "C" int64_t aprnet_edge_workspace_bytes(const aprnet_apr* a, int dl, int cout);
extern "C" int aprnet_conv333_backward_input_cross_level_tc(aprnet_apr* a, int dl, int cin, int cout, int slots,
                                                            const void* grows, int gpad, const float* w, float* gin,
                                                            int64_t ld_in, float* gtree, int64_t ld_tree, void* wp_ws,
                                                            void* edge_ws, int64_t edge_ws_bytes, void* stream);
// same, with the final tree adjoint (grad_tree folded into grad_input) optional
int aprnet_cross_level_tc(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* grows, int gpad, const float* w, float* gin,
                          long long ld_in, float* gtree, long long ld_tree, void* wp_ws, void* edge_ws, long long edge_ws_bytes, void* stream,
                          bool tree_adjoint);

// fp32 path (conv333_f32.cu): the same steps over packed fp32 rows
size_t aprnet_f32_rows_bytes(const aprnet_apr* a, int dl, int cin);
size_t aprnet_f32_forward_bytes(const aprnet_apr* a, int dl, int cin, int cout, int slots);        // packed input rows + packed weights
size_t aprnet_f32_backward_bytes(const aprnet_apr* a, int dl, int cin, int cout, int slots);       // packed grad_output rows, weights, edge sums
int64_t aprnet_f32_partial_elems(int cin, int cout);
int aprnet_f32_pack_input(const aprnet_apr* a, int dl, int cin, const float* in, long long ld_in, const float* tree, long long ld_tree, void* rows, cudaStream_t st);
int aprnet_f32_pack_grad(const aprnet_apr* a, int dl, int cout, const float* gout, long long ld_out, void* grows, cudaStream_t st);
int aprnet_f32_forward(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* w, const float* bias, float* out, long long ld_out, void* workspace, cudaStream_t st);
int aprnet_f32_backward_weights(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* rows, const float* gout, long long ld_out, const void* grows,
                                float* gw, int accumulate, float* partial, cudaStream_t st);
int aprnet_f32_backward_input(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* gout, long long ld_out, const float* w, float* gin, long long ld_in,
                              float* gtree, long long ld_tree, void* workspace, bool tree_adjoint, cudaStream_t st);

// ranges of block partial sums [range][27][cout][cin] per stencil slot: slot[g] owns [first[g], first[g + 1]), g < n
struct SlotRanges { int n; int first[APRNET_MAX_LEVELS + 1]; int slot[APRNET_MAX_LEVELS]; unsigned empty; };      // empty: slots to zero (bit per slot)
// grad_weights (slots, Cout, Cin, 27) += sums in a fixed order; without `accumulate` all of it is written (zeros in slots without ranges)
int aprnet_dw_reduce(const float* partial, SlotRanges sr, int slots, int accumulate, int cin, int cout, float* gw, cudaStream_t st);
int aprnet_tc_backward_weights(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* xrows, int xpad, const void* grows, int gpad, float* gw, int accumulate,
                               float* partial, cudaStream_t st);

// stream-ordered scratch of one call, for entry points whose signature has no workspace
struct StreamScratch {
    void* p = nullptr;
    cudaStream_t st;
    explicit StreamScratch(cudaStream_t s) : st(s) {}
    ~StreamScratch() { if (p) cudaFreeAsync(p, st); }
    int get(size_t bytes) {
        const cudaError_t e = cudaMallocAsync(&p, bytes, st);
        if (e != cudaSuccess) { p = nullptr; cudaGetLastError(); aprnet_set_error("allocation of %zu bytes of scratch failed: %s", bytes, cudaGetErrorString(e)); return APRNET_ERR_CUDA; }
        return APRNET_OK;
    }
};
