// 3x3x3 particle convolution on the tensor cores over runs of cells (bf16 operands, fp32 accumulation): forward pass of layers with at
// most 128 result channels (above 64 and with several chunks of source channels by a kernel of its own, see there), same-level input gradient of any width.
//
// The kernel of conv333_tc.cu gathers every source row once per tap, 27 rows per location.  Here the M dimension of a tile is not
// 128 locations but 128 * H consecutive slots of the run plan (run_plan.cu).  For each of the 9 rows of cells (dz, dx) the tile's
// sources are gathered once, one row per slot, and the three y taps read the same staged rows shifted by one: the A descriptor of
// tap dy starts dy rows further.  (The swizzle of a K-major operand is a function of the shared-memory address, so a start address
// inside the pattern is an ordinary one.)  That is 9 x 1.07 .. 1.27 gathered rows per location instead of 27; slots without a
// location are the price, 7 to 27 % more multiply-adds.  Each weight tile that is fetched meets H blocks of 128 rows.
// What bounds it: operand reads.  Shares of each unit's own peak for 32 -> 32 and 64 -> 64 channels, which overlap: operand reads of the tensor
// core (l1tex__data_pipe_tc_wavefronts) 71 and 80 %, load-store unit (copies, whose sectors land one by one, shuffles, stores of the results;
// l1tex__data_pipe_lsu_wavefronts) 67 and 60 %, issue slots 34 and 30 %, tensor pipe 31 and 54 %; 16 -> 16: 52, 61, 38 and 23 %.  (All rows by tile::gather4 instead of cp.async took 6.6 cycles per row: 0.96 ms for a
// 32 -> 32 layer that takes 0.48.)
//
// Every result of the forward pass is the same sequence of MMAs (neighbour row, channel block, dy, 16 channels) as in
// conv333_tc.cu, so the two kernels agree bit for bit: what follows a convolution (rounding to bf16, ReLU, max-pooling) turns a
// difference in the last bit into another gate.
#include "apr_device.cuh"
#include "tc_ptx.cuh"
#include <cuda_bf16.h>
#include <algorithm>
#include <cstring>

namespace {

using namespace tcptx;
typedef long long ll;
constexpr int MAX_SEGS = APRNET_MAX_LEVELS;
constexpr int MAX_STAGES = 16;
constexpr int MAX_ACC = 4;
constexpr int MAX_N = 256;                               // result channels of all tiles, where a bias is added
constexpr int NPROD = 8;                                 // producer warps
constexpr int MMA_WARP = NPROD, EPI_WARP = NPROD + 2;    // two MMA warps, two sets of four epilogue warps
constexpr int THREADS = (NPROD + 2 + 8) * 32;

struct RunParams {
    int n_segs;
    ll slot_begin[MAX_SEGS], slot_end[MAX_SEGS];         // slots of the level
    ll lo[MAX_SEGS], hi[MAX_SEGS];                       // its locations (same-level mask of the input gradient)
    int wslot[MAX_SEGS];
    int tile_begin[MAX_SEGS + 1];
    const int32_t* src; ll S;                            // run plan: [9][S] sources, [S] locations
    const int32_t* loc;
    const __nv_bfloat16* rows; int kpad;
    ll tree_base, zero_row;
    const __nv_bfloat16* wp;                             // packed weights [slot][tap][n tile][k chunk][NT][8]
    float* out; ll ld_out; int n_dim, n_tiles;           // results, tiles of NT channels
    const float* bias;
    int same_level_only;                                 // input gradient: sources of the tile's own level, taps mirrored
    int* error_flag;
};

template<int KS> __device__ __forceinline__ int swizzled_chunk(int row, int c) {      // position of 16-byte chunk c of row `row`
    return KS == 64 ? (c ^ (row & 7)) : (KS == 32 ? (c ^ ((row >> 1) & 3)) : (c ^ ((row >> 2) & 1)));
}

// The tiles of a block, one after the other: work items blockIdx.x, + gridDim.x, ... over (tile, result tile).  The segment is found by going
// on from the previous tile's: searching the parameters' table for every tile in every role cost some 500 cycles of dependent reads each time.
struct TileWalk {
    int tile, ntile, seg = -1, seg_first = 0, seg_end = 0, wslot = 0;
    int32_t lo = 0, hi = 0;                 // locations of the tile's level
    const int dt, dn;                       // step of (tile, result tile) from one work item to the next
    ll sb = 0, se = 0;                      // its slots
    __device__ __forceinline__ explicit TileWalk(const RunParams& P)
        : tile(blockIdx.x / P.n_tiles), ntile(blockIdx.x % P.n_tiles), dt(gridDim.x / P.n_tiles), dn(gridDim.x % P.n_tiles) { settle(P); }
    __device__ __forceinline__ void settle(const RunParams& P) {
        while (tile >= seg_end && seg + 1 < P.n_segs) {
            ++seg;
            seg_first = P.tile_begin[seg]; seg_end = P.tile_begin[seg + 1];
            sb = P.slot_begin[seg]; se = P.slot_end[seg]; lo = (int32_t) P.lo[seg]; hi = (int32_t) P.hi[seg]; wslot = P.wslot[seg];
        }
    }
    __device__ __forceinline__ void next(const RunParams& P) {
        tile += dt; ntile += dn;
        if (ntile >= P.n_tiles) { ntile -= P.n_tiles; ++tile; }
        settle(P);
    }
    // slot of staged row 0; the first and the last of the `rows` rows have no neighbour on one side.  The rows [first, end) are slots of the level
    __device__ __forceinline__ ll s0(int rows) const { return sb - 1 + (ll) (tile - seg_first) * (rows - 2); }
    __device__ __forceinline__ int first() const { return tile == seg_first ? 1 : 0; }
    __device__ __forceinline__ int end(int rows) const { return (int) min(se - s0(rows), (ll) rows); }
};

// Roles of the warps of the persistent block:
//   0-7         producers, in groups of WPS; a stage (neighbour row x KS channels x 128 H slots, and the weights of its three taps) belongs to one
//               group, each warp copies its share of the rows with 16-byte cp.async into the swizzled K-major operand and attaches its
//               arrival to the stage's barrier; a lane holds the table entries of its rows, requested one stage of the group ahead, and
//               hands them round by shuffles; one lane streams the weights with bulk copies;
//   8, 9        one thread each issues the MMAs of every second block of 128 rows (two issuers: a narrow MMA costs its thread more
//               cycles than it costs the tensor pipe) and commits the stage's free barrier;
//   10-17       epilogue, four warps per issuer: TMEM -> registers -> global;
// All waits are bounded and poll the block's abort flag (see conv333_tc.cu).
//
// KUSE: channels of a stage that exist, the others of its KS-wide rows are neither copied nor multiplied.  48 channels (33 to 48, padded) in stages of 16 took three
// stages per neighbour row, each with rows of 32 bytes: 48 -> 48 on 3.5 M locations 1.04 ms, now 0.76; 96 -> 48, input gradient at level delta 1, 1.40 -> 0.53.
template<int NT, int KS, int KUSE, int KORD, int H, int WPS>
__global__ void __launch_bounds__(THREADS, 1) conv333_tc_runs_kernel(const RunParams P, const int stages) {
    constexpr int NG = NPROD / WPS;                          // stages in issue at once
    constexpr int CH = KS / 8;                               // 16-byte chunks per row piece
    constexpr int RW = 32 / CH;                              // rows per copy instruction of a warp
    constexpr int ROWS = 128 * H, WROWS = ROWS / WPS;        // slots of a tile, rows a producer warp copies
    constexpr int NI = WROWS / RW, LR = (WROWS + 31) / 32;   // its copy instructions per stage, table entries per lane
    constexpr int NB = NI < 8 ? NI : 8;                      // copies whose rows are handed round together
    constexpr int NACC = 512 / (H * NT) < MAX_ACC ? 512 / (H * NT) : MAX_ACC;      // accumulators in flight per block of 128 rows
    constexpr int ISSUERS = H < 2 ? 1 : 2;
    constexpr int ROW_BYTES = KS * 2;
    constexpr uint32_t A_LAYOUT = KS == 64 ? 2u : (KS == 32 ? 4u : 6u);     // SWIZZLE_128B / 64B / 32B
    constexpr int A_BYTES = ROWS * ROW_BYTES;
    constexpr int B_TAP = NT * KUSE * 2;
    constexpr int STAGE_BYTES = A_BYTES + 3 * B_TAP;
    constexpr uint32_t IDESC = make_idesc(NT, false, false);
    static_assert(STAGE_BYTES % 1024 == 0 && H * NT <= 512 && WROWS % 32 == 0 && NI % NB == 0, "stages keep the swizzle alignment; accumulators fit TMEM");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ float bias_s[MAX_N];
    // ring at a multiple of 1024 bytes, with 1024 bytes in front of it (row -1 of the first stage is read, its results are not used)
    unsigned char* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u) + 1024;
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring + (size_t) stages * STAGE_BYTES + 1024);
    uint64_t* full = bars;                                   // [stages] copies of the stage landed
    uint64_t* empty = bars + MAX_STAGES;                     // [stages] all MMAs that read the stage completed
    uint64_t* tmem_full = empty + MAX_STAGES;                // [2][NACC] accumulators of an issuer complete
    uint64_t* tmem_empty = tmem_full + 2 * MAX_ACC;          // [2][NACC] read back
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2 * MAX_ACC);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = warp_number(), lane = tid & 31;
    const int kchunks = P.kpad / KUSE, steps = 9 * kchunks;
    const int total_tiles = P.tile_begin[P.n_segs] * P.n_tiles;
    const int my_tiles = (int) blockIdx.x < total_tiles ? (total_tiles - (int) blockIdx.x + (int) gridDim.x - 1) / (int) gridDim.x : 0;
    const int ngroups = min(NG, stages);

    if (P.bias) for (int c = tid; c < min(MAX_N, P.n_tiles * NT); c += THREADS) bias_s[c] = c < P.n_dim ? P.bias[c] : 0.f;
    if (tid == 0) {
        for (int i = 0; i < stages; ++i) { mbar_init(smem_u32(full + i), WPS * 32 + 1); mbar_init(smem_u32(empty + i), ISSUERS); }
        for (int i = 0; i < 2 * MAX_ACC; ++i) { mbar_init(smem_u32(tmem_full + i), 1); mbar_init(smem_u32(tmem_empty + i), 4); }
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == MMA_WARP) { tmem_alloc(smem_u32(tmem_slot), H * NACC * NT); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = *tmem_slot;
    bool failed = false, bulk_issued = false;

    if (warp < NPROD) {
        // ---------------- producers ----------------
        const int grp = warp / WPS, sub = warp % WPS;
        if (grp < ngroups) {
            const int j = lane % CH, rsub = lane / CH;
            const uint32_t total = (uint32_t) my_tiles * (uint32_t) steps;
            const ll w_tile = (ll) P.kpad * NT * 2, w_tap_stride = P.n_tiles * w_tile;
            uint32_t slot = grp, use = 0;
            uint32_t left = grp < (int) total ? (total - grp + ngroups - 1) / ngroups : 0;       // stages of this group
            TileWalk walk(P);
            int d = 0, kc = grp;                             // the stage's neighbour row and channels
            auto locate = [&]() {
                while (kc >= kchunks) { kc -= kchunks; ++d; }
                while (d >= 9) { d -= 9; walk.next(P); }
            };
            int32_t raw[LR], cur[LR];
            auto request = [&]() {                           // table entries of this lane's rows
                const int first = walk.first(), end = walk.end(ROWS);
                const int32_t* src = P.src + (ll) d * P.S + walk.s0(ROWS) + sub * WROWS + lane;
#pragma unroll
                for (int i = 0; i < LR; ++i) {
                    const int row = sub * WROWS + 32 * i + lane;
                    raw[i] = row >= first && row < end ? __ldg(src + 32 * i) : APRNET_NONE;
                }
            };
            const int32_t zero = (int32_t) P.zero_row, tree = (int32_t) P.tree_base - 2;       // row numbers fit 32 bits
            if (left > 0) { locate(); request(); }
            for (; left > 0; --left) {
#pragma unroll
                for (int i = 0; i < LR; ++i) {
                    const int32_t v = raw[i];
                    if (P.same_level_only) cur[i] = v >= walk.lo && v < walk.hi ? v : zero;
                    else cur[i] = v >= 0 ? v : (v != APRNET_NONE ? tree - v : zero);
                }
                const unsigned char* wsrc = reinterpret_cast<const unsigned char*>(P.wp) + ((ll) walk.wslot * 27 + (P.same_level_only ? 26 - 3 * d : 3 * d)) * w_tap_stride + walk.ntile * w_tile + (ll) kc * KUSE * NT * 2;
                const __nv_bfloat16* src0 = P.rows + kc * KUSE + j * 8;
                kc += ngroups;
                if (left > 1) { locate(); request(); }       // in flight while this stage is copied
                if (use > 0 && !mbar_wait_warp(smem_u32(empty + slot), (use - 1) & 1, abort_flag)) { failed = true; break; }
                unsigned char* a_s = ring + (size_t) slot * STAGE_BYTES;
                if (sub == 0 && elect_one()) {
                    mbar_expect_tx(smem_u32(full + slot), 3 * B_TAP);
#pragma unroll
                    for (int dy = 0; dy < 3; ++dy)
                        bulk_copy_g2s(smem_u32(a_s + A_BYTES + dy * B_TAP), wsrc + (P.same_level_only ? -dy : dy) * w_tap_stride, B_TAP, smem_u32(full + slot));
                    bulk_issued = true;
                }
#pragma unroll
                for (int i0 = 0; i0 < NI; i0 += NB) {        // copies and shuffles keep their order: the rows of several copies are handed round first
                    int32_t r[NB];
#pragma unroll
                    for (int i = 0; i < NB; ++i) r[i] = __shfl_sync(0xffffffffu, cur[(i0 + i) * RW / 32], ((i0 + i) * RW + rsub) & 31);
#pragma unroll
                    for (int i = 0; i < NB; ++i) {
                        const int row = sub * WROWS + (i0 + i) * RW + rsub;
                        if (KUSE == KS || j < KUSE / 8) cp_async16(smem_u32(a_s + row * ROW_BYTES + (swizzled_chunk<KS>(row, j) << 4)), src0 + (ll) r[i] * P.kpad);
                    }
                }
                cp_async_arrive_noinc(smem_u32(full + slot));        // this thread's arrival when its copies have landed
                slot += ngroups;
                if (slot >= (uint32_t) stages) { slot -= stages; ++use; }
            }
            cp_async_commit();
            cp_async_wait<0>();
        }
    } else if (warp < EPI_WARP) {
        // ---------------- MMA issue, every second block of 128 rows ----------------
        const int h0 = warp - MMA_WARP;
        if (h0 < ISSUERS && elect_one()) {
            constexpr int MMAS = 3 * (KUSE / 16);
            uint32_t slot = 0, use = 0;
            bool ready = false;                   // the next stage is known to be there
            for (int it = 0; it < my_tiles && !failed; ++it) {
                const uint32_t acc = (uint32_t) it % NACC, acc_use = (uint32_t) it / NACC;
                if (acc_use > 0 && !mbar_wait(smem_u32(tmem_empty + h0 * MAX_ACC + acc), (acc_use - 1) & 1, abort_flag)) { failed = true; break; }
                tc_fence_after();
                for (int step = 0; step < steps; ++step) {
                    if (!ready && !mbar_wait(smem_u32(full + slot), use & 1, abort_flag)) { failed = true; break; }
                    fence_proxy_async();          // generic-proxy writes of the cp.async copies -> tensor-core (async proxy) reads
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(ring + (size_t) slot * STAGE_BYTES);
                    const uint64_t db0 = make_desc(a_addr + A_BYTES, NT * 16, 128, 0);
                    const uint32_t used = slot;
                    if (++slot == (uint32_t) stages) { slot = 0; ++use; }
#pragma unroll
                    for (int h = 0; h < H; h += ISSUERS) {
                        const uint64_t da0 = make_desc(a_addr + (h + h0) * 128 * ROW_BYTES - ROW_BYTES, 16, 8 * ROW_BYTES, A_LAYOUT);      // dy = -1
                        const uint32_t d_addr = tmem_d + ((h + h0) * NACC + acc) * NT;
#pragma unroll
                        for (int m = 0; m < MMAS; ++m) {          // blocks of KORD channels, dy, 16 channels
                            const int ko = m / (3 * (KORD / 16)), dy = m / (KORD / 16) % 3, k = ko * (KORD / 16) + m % (KORD / 16);
                            if (h + ISSUERS >= H && m == MMAS / 2) ready = mbar_test(smem_u32(full + slot), use & 1);
                            umma_bf16(d_addr, da0 + (uint64_t) ((dy * ROW_BYTES + k * 32) >> 4), db0 + (uint64_t) ((dy * B_TAP + k * 2 * (NT * 16)) >> 4),
                                      IDESC, (step > 0 || m > 0) ? 1u : 0u);
                        }
                    }
                    umma_commit(smem_u32(empty + used));
                }
                if (!failed) umma_commit(smem_u32(tmem_full + h0 * MAX_ACC + acc));
            }
        }
    } else if ((warp - EPI_WARP) / 4 < ISSUERS) {
        // ---------------- epilogue of one issuer's blocks ----------------
        const int h0 = (warp - EPI_WARP) >> 2, q = warp & 3;         // q: TMEM lanes this warp may read
        TileWalk walk(P);                                            // the tile after the one that is read back
        auto location = [&](int it, int h) {
            const int m = h * 128 + q * 32 + lane;
            if (it >= my_tiles || m == 0 || m == ROWS - 1) return (int32_t) -1;
            return m >= walk.first() && m < walk.end(ROWS) ? __ldg(P.loc + walk.s0(ROWS) + m) : -1;
        };
        constexpr int BLOCKS = H / ISSUERS;
        int32_t p_next[BLOCKS];
#pragma unroll
        for (int b = 0; b < BLOCKS; ++b) p_next[b] = location(0, h0 + b * ISSUERS);
        for (int it = 0; it < my_tiles; ++it) {
            const int n0 = walk.ntile * NT;
            walk.next(P);
            int32_t p_cur[BLOCKS];
#pragma unroll
            for (int b = 0; b < BLOCKS; ++b) { p_cur[b] = p_next[b]; p_next[b] = location(it + 1, h0 + b * ISSUERS); }
            const uint32_t acc = (uint32_t) it % NACC, acc_use = (uint32_t) it / NACC;
            if (!mbar_wait_warp(smem_u32(tmem_full + h0 * MAX_ACC + acc), acc_use & 1, abort_flag)) { failed = true; break; }
            tc_fence_after();
#pragma unroll
            for (int b = 0; b < BLOCKS; ++b) {
                const int32_t p = p_cur[b];
#pragma unroll 1
                for (int c0 = 0; c0 < NT; c0 += 32) {
                    uint32_t r[32];
                    tmem_ld32(tmem_d + ((uint32_t) (q * 32) << 16) + ((h0 + b * ISSUERS) * NACC + acc) * NT + c0, r);
                    tmem_ld_wait();
                    if (P.bias) {
#pragma unroll
                        for (int jj = 0; jj < 32; ++jj)
                            r[jj] = __float_as_uint(__uint_as_float(r[jj]) + bias_s[n0 + c0 + jj]);
                    }
                    if (p >= 0) {
                        float* dst = P.out + (ll) (n0 + c0) * P.ld_out + p;
#pragma unroll
                        for (int jj = 0; jj < 32; ++jj)
                            if (n0 + c0 + jj < P.n_dim) dst[(ll) jj * P.ld_out] = __uint_as_float(r[jj]);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(tmem_empty + h0 * MAX_ACC + acc));
        }
    }

    // teardown (also the error path): the gather copies were drained above; after a failure the bulk copies still in flight get
    // time to land before the block's shared memory is released
    if (failed) {
        *abort_flag = 1;
        if (P.error_flag) *P.error_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (bulk_issued && *abort_flag) for (int i = 0; i < 2000; ++i) __nanosleep(100);
    if (warp == MMA_WARP) tmem_dealloc(tmem_d, H * NACC * NT);
}

// Forward pass of layers with 65 to 128 result channels and several chunks of 64 source channels, over runs of cells, in the order of conv333_tc.cu for them: one tap
// after the other, each over all chunks.  A tap's products run through all source channels before the next tap's, so all chunks of a neighbour row
// have to be there before its first tap is finished: the rows (pieces of 128 H slots x 64 channels) and the weights (tiles of one tap and chunk) have rings of
// their own; a piece is given back after the last of its row's three taps, a weight tile after its MMAs.  Gathering every tap by itself the layers were
// bound by the gather (27 rows per location past L1): 128 -> 128 on 553 k locations 0.52 ms, now 0.45; 256 -> 128 0.99, now 0.86.
// Roles of the warps: 0-7 producers of pieces, in two groups of four; 8 weights (bulk copies of one thread); 9 MMA issue (one thread); 10-17 epilogue, one set of four warps
// for every block of 128 rows (H = 1: the first set).
constexpr int WIDE_MAX_PIECES = 14, WIDE_MAX_TILES = 8;
template<int NT, int H>
__global__ void __launch_bounds__(THREADS, 1) conv333_tc_wide_kernel(const RunParams P, const int pieces, const int tiles) {
    constexpr int KS = 64, CH = 8, RW = 4, WPS = 4;
    constexpr int ROWS = 128 * H, WROWS = ROWS / WPS, NI = WROWS / RW, LR = WROWS / 32;
    constexpr int NACC = 512 / (H * NT) < MAX_ACC ? 512 / (H * NT) : MAX_ACC;
    constexpr int ROW_BYTES = 128, PIECE = ROWS * ROW_BYTES, B_TILE = NT * KS * 2;
    constexpr uint32_t IDESC = make_idesc(NT, false, false);
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ float bias_s[MAX_N];
    // the ring of pieces at a multiple of 1024 bytes, with 1024 bytes in front of it and behind it (rows that are read next to a piece's first and last, for results that are not used)
    unsigned char* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u) + 1024;
    unsigned char* b_ring = ring + (size_t) pieces * PIECE + 1024;
    uint64_t* bars = reinterpret_cast<uint64_t*>(b_ring + (size_t) tiles * B_TILE);
    uint64_t* full = bars;                                   // [pieces] rows landed
    uint64_t* empty = full + WIDE_MAX_PIECES;                // [pieces] the last tap's MMAs completed
    uint64_t* w_full = empty + WIDE_MAX_PIECES;              // [tiles]  weights landed
    uint64_t* w_empty = w_full + WIDE_MAX_TILES;             // [tiles]  MMAs that read them completed
    uint64_t* tmem_full = w_empty + WIDE_MAX_TILES;          // [NACC]   accumulators of a tile complete
    uint64_t* tmem_empty = tmem_full + MAX_ACC;              // [NACC]   read back (four warps per block of 128 rows)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + MAX_ACC);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = warp_number(), lane = tid & 31;
    const int kchunks = P.kpad / KS, steps = 9 * kchunks;    // pieces of a tile
    const int total_tiles = P.tile_begin[P.n_segs] * P.n_tiles;
    const int my_tiles = (int) blockIdx.x < total_tiles ? (total_tiles - (int) blockIdx.x + (int) gridDim.x - 1) / (int) gridDim.x : 0;

    if (P.bias) for (int c = tid; c < min(MAX_N, P.n_tiles * NT); c += THREADS) bias_s[c] = c < P.n_dim ? P.bias[c] : 0.f;
    if (tid == 0) {
        for (int i = 0; i < pieces; ++i) { mbar_init(smem_u32(full + i), WPS * 32); mbar_init(smem_u32(empty + i), 1); }
        for (int i = 0; i < tiles; ++i) { mbar_init(smem_u32(w_full + i), 1); mbar_init(smem_u32(w_empty + i), 1); }
        for (int i = 0; i < NACC; ++i) { mbar_init(smem_u32(tmem_full + i), 1); mbar_init(smem_u32(tmem_empty + i), 4 * H); }
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == MMA_WARP + 1) { tmem_alloc(smem_u32(tmem_slot), H * NACC * NT); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = *tmem_slot;
    bool failed = false, bulk_issued = false;

    if (warp < NPROD) {
        // ---------------- rows ----------------
        const int grp = warp / WPS, sub = warp % WPS, j = lane % CH, rsub = lane / CH;
        const uint32_t total = (uint32_t) my_tiles * (uint32_t) steps;
        uint32_t slot = grp, use = 0;                        // (two groups, at least three pieces)
        uint32_t left = grp < (int) total ? (total - grp + 1) / 2 : 0;
        TileWalk walk(P);
        int d = 0, kc = grp;                                 // the piece's neighbour row and channels
        auto locate = [&]() {
            while (kc >= kchunks) { kc -= kchunks; ++d; }
            while (d >= 9) { d -= 9; walk.next(P); }
        };
        int32_t raw[LR], cur[LR];
        auto request = [&]() {                               // table entries of this lane's rows
            const int first = walk.first(), end = walk.end(ROWS);
            const int32_t* src = P.src + (ll) d * P.S + walk.s0(ROWS) + sub * WROWS + lane;
#pragma unroll
            for (int i = 0; i < LR; ++i) {
                const int row = sub * WROWS + 32 * i + lane;
                raw[i] = row >= first && row < end ? __ldg(src + 32 * i) : APRNET_NONE;
            }
        };
        const int32_t zero = (int32_t) P.zero_row, tree = (int32_t) P.tree_base - 2;       // row numbers fit 32 bits
        if (left > 0) { locate(); request(); }
        for (; left > 0; --left) {
#pragma unroll
            for (int i = 0; i < LR; ++i) { const int32_t v = raw[i]; cur[i] = v >= 0 ? v : (v != APRNET_NONE ? tree - v : zero); }
            const __nv_bfloat16* src0 = P.rows + kc * KS + j * 8;
            kc += 2;
            if (left > 1) { locate(); request(); }           // in flight while this piece is copied
            if (use > 0 && !mbar_wait_warp(smem_u32(empty + slot), (use - 1) & 1, abort_flag)) { failed = true; break; }
            unsigned char* a_s = ring + (size_t) slot * PIECE;
#pragma unroll
            for (int i0 = 0; i0 < NI; i0 += 8) {             // copies and shuffles keep their order: the rows of several copies are handed round first
                int32_t r[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) r[i] = __shfl_sync(0xffffffffu, cur[(i0 + i) * RW / 32], ((i0 + i) * RW + rsub) & 31);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int row = sub * WROWS + (i0 + i) * RW + rsub;
                    cp_async16(smem_u32(a_s + row * ROW_BYTES + (swizzled_chunk<KS>(row, j) << 4)), src0 + (ll) r[i] * P.kpad);
                }
            }
            cp_async_arrive_noinc(smem_u32(full + slot));
            slot += 2;
            if (slot >= (uint32_t) pieces) { slot -= pieces; ++use; }
        }
        cp_async_commit();
        cp_async_wait<0>();
    } else if (warp == MMA_WARP) {
        // ---------------- weights: tap by tap, chunk by chunk ----------------
        if (elect_one()) {
            const ll w_tile = (ll) P.kpad * NT * 2, w_tap = P.n_tiles * w_tile;
            TileWalk walk(P);
            uint32_t slot = 0, use = 0;
            for (int it = 0; it < my_tiles && !failed; ++it, walk.next(P)) {
                const unsigned char* src = reinterpret_cast<const unsigned char*>(P.wp) + (ll) walk.wslot * 27 * w_tap + walk.ntile * w_tile;
                for (int tap = 0; tap < 27 && !failed; ++tap, src += w_tap)
                    for (int kc = 0; kc < kchunks; ++kc) {
                        if (use > 0 && !mbar_wait(smem_u32(w_empty + slot), (use - 1) & 1, abort_flag)) { failed = true; break; }
                        mbar_expect_tx(smem_u32(w_full + slot), B_TILE);
                        bulk_copy_g2s(smem_u32(b_ring + (size_t) slot * B_TILE), src + (ll) kc * B_TILE, B_TILE, smem_u32(w_full + slot));
                        bulk_issued = true;
                        if (++slot == (uint32_t) tiles) { slot = 0; ++use; }
                    }
            }
        }
    } else if (warp == MMA_WARP + 1) {
        // ---------------- MMA issue ----------------
        if (elect_one()) {
            uint32_t p0 = 0, p0_use = 0, ws = 0, wu = 0;     // first piece of the neighbour row; weight tile
            for (int it = 0; it < my_tiles && !failed; ++it) {
                const uint32_t acc = (uint32_t) it % NACC, acc_use = (uint32_t) it / NACC;
                if (acc_use > 0 && !mbar_wait(smem_u32(tmem_empty + acc), (acc_use - 1) & 1, abort_flag)) { failed = true; break; }
                tc_fence_after();
                for (int d = 0; d < 9 && !failed; ++d) {
                    for (int dy = 0; dy < 3 && !failed; ++dy) {
                        uint32_t p = p0, pu = p0_use;
                        for (int kc = 0; kc < kchunks; ++kc) {
                            if (dy == 0 && !mbar_test(smem_u32(full + p), pu & 1) && !mbar_wait(smem_u32(full + p), pu & 1, abort_flag)) { failed = true; break; }
                            if (!mbar_test(smem_u32(w_full + ws), wu & 1) && !mbar_wait(smem_u32(w_full + ws), wu & 1, abort_flag)) { failed = true; break; }
                            if (dy == 0) fence_proxy_async();        // generic-proxy writes of the cp.async copies -> tensor-core (async proxy) reads
                            tc_fence_after();
                            const uint64_t db0 = make_desc(smem_u32(b_ring + (size_t) ws * B_TILE), NT * 16, 128, 0);
#pragma unroll
                            for (int h = 0; h < H; ++h) {
                                const uint64_t da0 = make_desc(smem_u32(ring + (size_t) p * PIECE) + (h * 128 + dy - 1) * ROW_BYTES, 16, 8 * ROW_BYTES, 2u);
#pragma unroll
                                for (int k = 0; k < 4; ++k)
                                    umma_bf16(tmem_d + (h * NACC + acc) * NT, da0 + (uint64_t) ((k * 32) >> 4), db0 + (uint64_t) ((k * 2 * (NT * 16)) >> 4), IDESC, (d > 0 || dy > 0 || kc > 0 || k > 0) ? 1u : 0u);
                            }
                            umma_commit(smem_u32(w_empty + ws));
                            if (dy == 2) umma_commit(smem_u32(empty + p));
                            if (++ws == (uint32_t) tiles) { ws = 0; ++wu; }
                            if (++p == (uint32_t) pieces) { p = 0; ++pu; }
                        }
                        if (dy == 2) { p0 = p; p0_use = pu; }
                    }
                }
                if (!failed) umma_commit(smem_u32(tmem_full + acc));
            }
        }
    } else if ((warp - EPI_WARP) / 4 < H) {
        // ---------------- epilogue of one block of 128 rows ----------------
        const int h = (warp - EPI_WARP) >> 2, q = warp & 3;          // q: TMEM lanes this warp may read
        TileWalk walk(P);                                            // the tile after the one that is read back
        auto location = [&](int it) {
            const int m = h * 128 + q * 32 + lane;
            if (it >= my_tiles || m == 0 || m == ROWS - 1) return (int32_t) -1;
            return m >= walk.first() && m < walk.end(ROWS) ? __ldg(P.loc + walk.s0(ROWS) + m) : -1;
        };
        int32_t next = location(0);
        for (int it = 0; it < my_tiles; ++it) {
            const int n0 = walk.ntile * NT;
            walk.next(P);
            const int32_t p = next;
            next = location(it + 1);
            const uint32_t acc = (uint32_t) it % NACC, acc_use = (uint32_t) it / NACC;
            if (!mbar_wait_warp(smem_u32(tmem_full + acc), acc_use & 1, abort_flag)) { failed = true; break; }
            tc_fence_after();
#pragma unroll 1
            for (int c0 = 0; c0 < NT; c0 += 32) {
                uint32_t r[32];
                tmem_ld32(tmem_d + ((uint32_t) (q * 32) << 16) + (h * NACC + acc) * NT + c0, r);
                tmem_ld_wait();
                if (P.bias) {
#pragma unroll
                    for (int jj = 0; jj < 32; ++jj) r[jj] = __float_as_uint(__uint_as_float(r[jj]) + bias_s[n0 + c0 + jj]);
                }
                if (p >= 0) {
                    float* dst = P.out + (ll) (n0 + c0) * P.ld_out + p;
#pragma unroll
                    for (int jj = 0; jj < 32; ++jj)
                        if (n0 + c0 + jj < P.n_dim) dst[(ll) jj * P.ld_out] = __uint_as_float(r[jj]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(tmem_empty + acc));
        }
    }

    // teardown as in conv333_tc_runs_kernel
    if (failed) {
        *abort_flag = 1;
        if (P.error_flag) *P.error_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (bulk_issued && *abort_flag) for (int i = 0; i < 2000; ++i) __nanosleep(100);
    if (warp == MMA_WARP + 1) tmem_dealloc(tmem_d, H * NACC * NT);
}

// ---- host side ----------------------------------------------------------------------------------------
constexpr size_t FIXED = (2 * MAX_STAGES + 4 * MAX_ACC) * 8 + 16 + 2048 + 1024;      // barriers, the rows in front of and behind the ring, alignment

inline size_t stage_bytes(int nt, int ks, int kuse, int h) { return (size_t) 128 * h * ks * 2 + 3 * (size_t) nt * kuse * 2; }
inline int run_stages(int nt, int ks, int kuse, int h) { return (int) std::min<size_t>(MAX_STAGES, (226 * 1024 - FIXED) / stage_bytes(nt, ks, kuse, h)); }

template<int NT, int KS, int KUSE, int KORD, int H, int WPS>
int launch_runs(RunParams& P, int sms, cudaStream_t st, const char* pname) {
    auto kern = conv333_tc_runs_kernel<NT, KS, KUSE, KORD, H, WPS>;
    const int stages = run_stages(NT, KS, KUSE, H);
    const size_t smem = (size_t) stages * stage_bytes(NT, KS, KUSE, H) + FIXED;
    APRNET_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    for (int i = 0; i < P.n_segs; ++i) P.tile_begin[i + 1] = P.tile_begin[i] + aprnet_ceil_div(P.slot_end[i] - P.slot_begin[i], 128 * H - 2);
    if (P.tile_begin[P.n_segs] == 0) return APRNET_OK;
    AprnetProfScope _prof(pname, st);
    kern<<<std::min(P.tile_begin[P.n_segs] * P.n_tiles, sms), THREADS, smem, st>>>(P, stages);
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

// Blocks of 128 rows per tile.  Cycles of a stage as fitted to the measurements below: the MMAs read their operands from shared
// memory at 128 bytes per clock (32 cycles for A, nt / 4 for B each), the copies write it, and about 550 cycles pass between the
// roles whatever the stage holds.  Tall tiles spread that and the weights over more rows; few rows want short tiles on all SMs.
// (16 -> 16, 32 -> 32, 64 -> 32 at level delta 0 and 64 -> 64 at level delta 1 of 1.8 M particles, forward: H = 2: 0.22, 0.30,
// 0.45, 0.26 ms; H = 4: 0.16, 0.24, 0.39, 0.25 ms; conv333_tc.cu: 0.52 for 32 -> 32, 0.48 for 64 -> 64.)  Since the roles branch per warp, result tiles of
// 64 channels are 6 % faster with H = 2 and its deeper ring (64 -> 64 at level delta 1 0.52 -> 0.49 ms, input gradient 64 -> 32 0.45 -> 0.41), those of 32 stay at 4
// (32 -> 32 0.38 against 0.44).  Stages of 16 channels had 8 until then: 16 -> 16 forward on 3.5 M and 263 k locations 306 and 38 us with 8, 267 and 31 with 4, input gradient 252 and 234; only
// input gradients of up to 8 channels on millions of locations lose, 3 to 5 % (8 -> 8 219 and 229).
inline int pick_h(const RunParams& P, int nt, int ks, int kuse, int max_h, int sms) {
    int best = 1;
    double cost = 0;
    for (int h = 1; h <= max_h; h *= 2) {
        ll tiles = 0;
        for (int i = 0; i < P.n_segs; ++i) tiles += aprnet_ceil_div(P.slot_end[i] - P.slot_begin[i], 128 * h - 2);
        const double stage = 550 + h * 3 * (kuse / 16) * (32 + nt / 4) + 1.3 * stage_bytes(nt, ks, kuse, h) / 128;
        const double c = (double) ((tiles * P.n_tiles + sms - 1) / sms) * (9 * P.kpad / kuse) * stage;
        if (h == 1 || c < cost) { cost = c; best = h; }
    }
    return best;
}

constexpr size_t WIDE_FIXED = (2 * WIDE_MAX_PIECES + 2 * WIDE_MAX_TILES + 2 * MAX_ACC) * 8 + 16 + 2048 + 1024;
constexpr size_t WIDE_SMEM = 227 * 1024 - 1024;          // (the biases are static)

// Rings of a layer of kpad source channels: all pieces of a neighbour row and one more, and three weight tiles; what is left goes to the pieces of a second row, then to the weights.
// false: they do not fit
inline bool wide_shape(int nt, int h, int kpad, int* pieces, int* tiles) {
    const size_t piece = (size_t) 128 * h * 128, tile = (size_t) nt * 128, room = WIDE_SMEM - WIDE_FIXED;
    const int kchunks = kpad / 64;
    if (kchunks + 1 > WIDE_MAX_PIECES || (kchunks + 1) * piece + 3 * tile > room) return false;
    *tiles = 3;
    *pieces = (int) std::min<size_t>(std::min(2 * kchunks, WIDE_MAX_PIECES), (room - 3 * tile) / piece);
    *pieces = std::max(*pieces, kchunks + 1);
    *tiles = (int) std::min<size_t>(WIDE_MAX_TILES, (room - *pieces * piece) / tile);
    return *pieces >= 3;
}

template<int NT, int H>
int launch_wide(RunParams& P, int sms, cudaStream_t st, const char* pname) {
    int pieces, tiles;
    if (!wide_shape(NT, H, P.kpad, &pieces, &tiles)) return APRNET_ERR_UNSUPPORTED;
    auto kern = conv333_tc_wide_kernel<NT, H>;
    const size_t smem = (size_t) pieces * 128 * H * 128 + (size_t) tiles * NT * 128 + WIDE_FIXED;
    APRNET_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    for (int i = 0; i < P.n_segs; ++i) P.tile_begin[i + 1] = P.tile_begin[i] + aprnet_ceil_div(P.slot_end[i] - P.slot_begin[i], 128 * H - 2);
    if (P.tile_begin[P.n_segs] == 0) return APRNET_OK;
    AprnetProfScope _prof(pname, st);
    kern<<<std::min(P.tile_begin[P.n_segs] * P.n_tiles, sms), THREADS, smem, st>>>(P, pieces, tiles);
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

} // namespace

// Channels between two changes of dy (the order of the products) of this kernel for kpad source channels; 0: not this kernel.
// nt_order, ks: tile width and channels per stage that conv333_tc.cu takes for the layer.  The forward pass keeps its order: stages of
// `ks` channels that hold three taps for nt_order <= 64, and for 128 where ks < 64 (the same order as here); one tap at a time for 128 and ks = 64 (the same only when all
// channels are in one stage), pairs of taps for 256.  The input gradient is free: nothing that follows depends on its last bit.
// -1: one tap after the other over all channels, in the kernel for that (APRNET_TAP_KERNEL where the tap kernel is the faster one; result tiles narrower than 128, that is few
// locations, are 10 to 15 % faster in the tap kernel: 9 k locations 42 against 37 us).
int aprnet_tc_runs_order(int backward, int kpad, int nt_order, int nt, int ks) {
    if (backward) return kpad % 32 == 0 ? 32 : 16;
    if (nt_order <= 64) return ks;
    if (nt_order == 128 && ks == 64 && kpad > 64) { int pieces, tiles; return nt == 128 && wide_shape(nt, 1, kpad, &pieces, &tiles) ? -1 : 0; }
    return nt_order == 128 && (ks < 64 || kpad == ks) ? ks : 0;
}

int aprnet_tc_run_conv(aprnet_apr* a, int dl, int backward, int slots, int nt, int order, const void* rows, int kpad, ll tree_base, ll zero_row, const void* wp,
                       const float* bias, float* out, ll ld_out, int n_dim, int* error_flag, cudaStream_t st, const char* pname) {
    const RunPlan* rp = aprnet_get_run_plan(a, dl, st);
    if (!rp) return APRNET_ERR_CUDA;
    RunParams P;
    memset(&P, 0, sizeof(P));
    for (const Segment& sg : aprnet_segments(a, dl, slots, false)) {
        const int i = P.n_segs++;
        P.slot_begin[i] = rp->level_begin[sg.level]; P.slot_end[i] = rp->level_begin[sg.level + 1];
        P.lo[i] = sg.begin; P.hi[i] = sg.end; P.wslot[i] = sg.slot;
    }
    if (P.n_segs == 0) return APRNET_OK;
    P.src = rp->src; P.S = rp->n_slots; P.loc = rp->loc;
    P.rows = (const __nv_bfloat16*) rows; P.kpad = kpad; P.tree_base = tree_base; P.zero_row = zero_row;
    P.wp = (const __nv_bfloat16*) wp; P.out = out; P.ld_out = ld_out; P.n_dim = n_dim; P.n_tiles = (n_dim + nt - 1) / nt; P.bias = bias; P.same_level_only = backward;
    P.error_flag = error_flag;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (order < 0) {
        // Microseconds of a wave of tiles for 128 source channels, and before the first one, of this kernel with two and with one block of 128 rows per tile and of the tap kernel,
        // as fitted to 128 -> 128 layers: 553 k locations 455, 538, 522; 170 k 158, 177, 186; 61 k 80, 85, 83; 33 k 55, 53, 49; 32 k (fewer tiles of two than SMs) -, 39, 49.
        // The choice against the tap kernel at other widths, 9 k to 2 M locations: 192 and 256 source channels 0 to 30 % faster, 320 to 512 (whose rows leave room for tiles of one block only) 0 to 20 %.
        ll t2 = 0, t1 = 0, taps = 0;
        for (int i = 0; i < P.n_segs; ++i) {
            const ll slots_ = P.slot_end[i] - P.slot_begin[i];
            t2 += aprnet_ceil_div(slots_, 254); t1 += aprnet_ceil_div(slots_, 126); taps += aprnet_ceil_div(P.hi[i] - P.lo[i], 128);
        }
        const double k = kpad / 128.0;
        auto time = [&](ll tiles, double wave, double start) { return (double) ((tiles + sms - 1) / sms) * wave * k + start; };
        int pieces, wtiles;
        const double two = wide_shape(nt, 2, kpad, &pieces, &wtiles) ? time(t2, 27.0, 3.0) : 1e30, one = time(t1, 15.8, 7.0);
        if (std::min(one, two) > time(taps, 17.4, 14.0)) return APRNET_TAP_KERNEL;
        return two < one ? launch_wide<128, 2>(P, sms, st, pname) : launch_wide<128, 1>(P, sms, st, pname);
    }
    // channels per stage: whole 128-byte rows where the width allows (64 -> 64: 0.25 instead of 0.29 ms with 32)
    const int kuse = kpad == 48 && order == 16 ? 48 : (kpad % 64 == 0 && order >= 32 ? 64 : order), ks = kuse == 48 ? 64 : kuse;
    const int h = pick_h(P, nt, ks, kuse, aprnet_run_max_height(nt), sms);
#define RUN_CASE(NT_, KS_, KORD_, H_, WPS_) if (nt == NT_ && kuse == KS_ && order == KORD_ && h == H_) return launch_runs<NT_, KS_ == 48 ? 64 : KS_, KS_, KORD_, H_, WPS_>(P, sms, st, pname);
    // warps per stage: two, so that four stages are in issue at once; four where the ring holds only two or three stages
    RUN_CASE(32, 16, 16, 1, 2) RUN_CASE(32, 16, 16, 2, 2) RUN_CASE(32, 16, 16, 4, 2)
    RUN_CASE(32, 32, 32, 1, 2) RUN_CASE(32, 32, 32, 2, 2) RUN_CASE(32, 32, 32, 4, 2)
    RUN_CASE(32, 64, 64, 1, 2) RUN_CASE(32, 64, 64, 2, 2) RUN_CASE(32, 64, 64, 4, 4)
    RUN_CASE(32, 64, 32, 1, 2) RUN_CASE(32, 64, 32, 2, 2) RUN_CASE(32, 64, 32, 4, 4) RUN_CASE(64, 64, 64, 1, 2) RUN_CASE(64, 64, 64, 2, 4)
    RUN_CASE(64, 16, 16, 1, 2) RUN_CASE(64, 16, 16, 2, 2)
    RUN_CASE(64, 32, 32, 1, 2) RUN_CASE(64, 32, 32, 2, 2)
    RUN_CASE(64, 64, 32, 1, 2) RUN_CASE(64, 64, 32, 2, 4)
    RUN_CASE(128, 16, 16, 1, 2) RUN_CASE(128, 16, 16, 2, 2) RUN_CASE(128, 32, 32, 1, 2) RUN_CASE(128, 32, 32, 2, 2)
    RUN_CASE(32, 48, 16, 1, 2) RUN_CASE(32, 48, 16, 2, 2) RUN_CASE(32, 48, 16, 4, 4)
    RUN_CASE(64, 48, 16, 1, 2) RUN_CASE(64, 48, 16, 2, 4) RUN_CASE(128, 48, 16, 1, 4) RUN_CASE(128, 48, 16, 2, 4)
    RUN_CASE(128, 64, 32, 1, 4) RUN_CASE(128, 64, 32, 2, 4) RUN_CASE(128, 64, 64, 1, 4) RUN_CASE(128, 64, 64, 2, 4)
#undef RUN_CASE
    aprnet_set_error("conv333 tensor-core path: unsupported run geometry nt=%d ks=%d order=%d h=%d", nt, ks, order, h);
    return APRNET_ERR_UNSUPPORTED;
}
