// Weight gradient of the 3x3x3 particle convolution on the tensor cores (tcgen05 + TMEM), bf16
// operands with fp32 accumulation, deterministic.
//
//     dW[d, dy][ci][co] = sum over locations p of  X[cell (dz, dx, dy) of p][ci] * dO[p][co]
//                       = sum over slots s of      X_d[s][ci] * dO[location of slot s - dy][co]
//
// with the slots of the run plan (run_plan.cu): X_d[s] is what fills the cell one step of d = (dz, dx) beside slot s, and the cell of
// slot s is the y neighbour of slot s - dy.  So every neighbour row is gathered once per slot (9 x 1.07 .. 1.27 rows per location)
// and meets dO three times, shifted by one slot each.  The product contracts over the slots; both operands are MN-major with a hardware
// swizzle, rows of channels in shared memory as they lie in global memory.  M = TPT = 128 / CIB neighbours x CIB input channels; the
// three shifts lie side by side in N: the B operand's blocks of NCOL columns start one slot (one row) further each (their stride in
// the descriptor is a row), which makes one MMA of 3 * NCOL <= 192 columns; for NCOL = 128 they are three MMAs.
// A block owns every cnt-th chunk of 128 slots of one level, a group of neighbours, CIB input and NCOL output channels; its
// accumulators stay in the 512 TMEM columns for all its chunks.  Blocks that run together walk through the level side by side, so the
// rows one of them gathers for the neighbouring z planes are still in L2 for the others.
//
// What bounds it: rows arriving from L2 (6 to 7 TB/s).  Gathering all 27 taps of a location by themselves, as this kernel did before,
// took 1.15 ms for 64 -> 64 channels at level delta 1 (1.86 M locations) and 1.03 ms for 32 -> 32 at level delta 0 (3.5 M).
//
// Warp roles: 16 producer warps (four stages in issue at once, four warps of 32 slots each per stage; table entries are loaded by the
// lane that owns the slot, one stage ahead, and passed between lanes by shuffles; arrival on the stage barrier is asynchronous), one
// MMA thread, epilogue by warps 0-3 after the last MMA.  Each block writes its partial sums once; a second pass adds the ranges in
// a fixed order (no atomics).
// Reference arithmetic: pyapr/aprnet/src/helpers.hpp:624-702 (accumulate_convolution_backward, dW part).
#include "apr_device.cuh"
#include "tc_ptx.cuh"
#include <cuda_bf16.h>
#include <algorithm>
#include <cmath>

extern int g_dw_waves_override;

namespace {

using namespace tcptx;
typedef long long ll;
constexpr int PT = 128;                       // slots per stage (K extent of one stage)
constexpr int NGROUP = 4;                     // producer groups of four warps = stages in issue at once
constexpr int MMA_WARP = 4 * NGROUP;
constexpr int DW_THREADS = (4 * NGROUP + 1) * 32;
constexpr int DW_MAX_STAGES = 6;
constexpr int A_STAGE = 2 * PT * 128;         // 128 accumulator rows = two 64-element swizzle atoms per slot
constexpr int G_ROWS = PT + 8;                // dO of slots -1 .. 128 of the chunk, whole 8-row groups
constexpr int DO_PHASES = NGROUP;             // "dO chunk read" barriers: chunk modulo DO_PHASES (the buffers alternate between two)

constexpr int DW_MAX_SEGS = APRNET_MAX_LEVELS;
struct DwParams {
    // the levels of the level delta, each cut into chunks of PT slots that its blocks take in turn: block r with
    // range_first[i] <= r < range_first[i + 1] belongs to level i and takes that level's chunks r - range_first[i], + cnt, + 2 cnt, ...
    int n_segs;
    ll seg_begin[DW_MAX_SEGS], seg_end[DW_MAX_SEGS];
    int range_first[DW_MAX_SEGS + 1];
    const int32_t* src; ll S;              // run plan
    const int32_t* loc;
    const __nv_bfloat16* xrows; int xpad;  // packed inputs [N + T + 1][xpad]; tree rows start at tree_base, zeros at zero_row
    ll tree_base, zero_row;
    const __nv_bfloat16* grows; int gpad;  // packed dO [N + 1][gpad], zeros at row g_zero_row
    ll g_zero_row;
    float* partial;                        // [range][27][cout][cin]
    int cin, cout, ci_blocks, groups, d_per_group;
    int* error_flag;
};

template<int CIB, int NCOL>
__global__ void __launch_bounds__(DW_THREADS, 1) conv333_tc_dw_kernel(const DwParams P, const int nstage) {
    constexpr int TPT = 128 / CIB;                      // neighbours per 128-row accumulator tile
    constexpr int PC = CIB / 8;                         // 16-byte chunks per gathered row piece
    constexpr int PB = PC < 8 ? PC : 8;                 // copies whose rows are handed round together
    constexpr int G_ROW = NCOL == 32 ? 64 : 128;        // bytes of a dO row in one swizzle atom
    constexpr int G_ATOM = G_ROWS * G_ROW;              // one atom (32 or 64 columns) of a dO chunk
    constexpr int G_BYTES = (G_ATOM * (NCOL == 128 ? 2 : 1) + 1023) / 1024 * 1024;
    constexpr int COLS = 3 * NCOL;                      // accumulator columns of a tile
    constexpr int MMAS = NCOL == 128 ? 3 : 1;
    constexpr uint32_t IDESC = make_idesc(COLS / MMAS, true, true);
    constexpr uint32_t ATOM_STRIDE = PT * 128;          // between 64-element atoms along M

    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char* a_ring = smem;                                               // nstage * A_STAGE
    unsigned char* g_ring = a_ring + (size_t) nstage * A_STAGE;                 // 2 * G_BYTES
    uint64_t* bars = reinterpret_cast<uint64_t*>(g_ring + 2 * G_BYTES);
    uint64_t* full = bars;                       // [nstage] gathered rows landed (4 warps x 32 lanes)
    uint64_t* empty = bars + DW_MAX_STAGES;      // [nstage] MMAs that read the stage completed
    uint64_t* dfull = empty + DW_MAX_STAGES;     // [2] dO chunk landed
    uint64_t* dempty = dfull + 2;                // [4] MMAs that read the dO chunk completed, by chunk modulo 4
    uint64_t* done = dempty + DO_PHASES;         // all MMAs of the range completed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = warp_number(), lane = tid & 31;
    const int grp = blockIdx.y % P.groups, cib = (blockIdx.y / P.groups) % P.ci_blocks, cob = blockIdx.y / (P.groups * P.ci_blocks);
    const int d0 = grp * P.d_per_group;
    const int nd = min(P.d_per_group, 9 - d0);
    const int MT = (nd + TPT - 1) / TPT;                // accumulator tiles of this block
    int seg = 0;
    while (seg + 1 < P.n_segs && (int) blockIdx.x >= P.range_first[seg + 1]) ++seg;
    const int rl = (int) blockIdx.x - P.range_first[seg], cnt = P.range_first[seg + 1] - P.range_first[seg];
    const ll sb = P.seg_begin[seg], se = P.seg_end[seg];
    const ll seg_chunks = (se - sb + PT - 1) / PT;
    const int nchunks = rl < seg_chunks ? (int) ((seg_chunks - rl + cnt - 1) / cnt) : 0;
    const int total_stages = nchunks * MT;
    const int cpieces = min(PC, (P.xpad - cib * CIB) / 8);            // 16-byte pieces that exist of a row (the others are never used)
    const int gpieces = min(NCOL, P.gpad - cob * NCOL) / 8;

    if (tid == 0) {
        for (int i = 0; i < nstage; ++i) { mbar_init(smem_u32(full + i), 128); mbar_init(smem_u32(empty + i), 1); }
        for (int i = 0; i < 2; ++i) mbar_init(smem_u32(dfull + i), 128);
        for (int i = 0; i < DO_PHASES; ++i) mbar_init(smem_u32(dempty + i), 1);
        mbar_init(smem_u32(done), 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == MMA_WARP) { tmem_alloc(smem_u32(tmem_slot), 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = *tmem_slot;
    bool failed = false;

    if (warp < MMA_WARP && total_stages > 0) {
        // ---------------- producers ----------------
        const int gq = warp >> 2, wq = warp & 3;        // stage (modulo NGROUP) / 32-slot quarter of the stage
        const int c = lane % PC, r0 = lane / PC;
        constexpr int RPI = 32 / PC;                    // slots covered by one copy instruction
        int32_t rows_cur[TPT], raw_nxt[TPT];
        int32_t loc_nxt = -1, loc_extra = -1, g_row = 0, g_extra = 0;
        // table entries of this lane's slot for stage s: requested here, decoded only when the stage is issued, so that the load
        // latency overlaps the copies of the stage in between; with a chunk's first stage also the locations of its dO rows (row r of
        // the dO chunk is slot r - 1; the last two rows belong to the last quarter)
        auto request = [&](int chunk, int mt) {
            const ll c0 = sb + ((ll) rl + (ll) chunk * cnt) * PT, slot = c0 + wq * 32 + lane;
#pragma unroll
            for (int tl = 0; tl < TPT; ++tl) {
                const int d = mt * TPT + tl;
                raw_nxt[tl] = (slot < se && d < nd) ? __ldg(P.src + (ll) (d0 + d) * P.S + slot) : APRNET_NONE;
            }
            if (mt == 0) {
                const ll p = slot - 1, q = c0 + PT - 1 + lane;
                loc_nxt = p >= sb && p < se ? __ldg(P.loc + p) : -1;
                loc_extra = wq == 3 && lane < 2 && q < se ? __ldg(P.loc + q) : -1;
            }
        };
        const int32_t zero = (int32_t) P.zero_row, tree = (int32_t) P.tree_base - 2;      // row numbers fit 32 bits
        auto decode = [&]() {
#pragma unroll
            for (int tl = 0; tl < TPT; ++tl) {
                const int32_t v = raw_nxt[tl];
                rows_cur[tl] = v >= 0 ? v : (v == APRNET_NONE ? zero : tree - v);
            }
            g_row = loc_nxt >= 0 ? loc_nxt : (int32_t) P.g_zero_row;
            g_extra = loc_extra >= 0 ? loc_extra : (int32_t) P.g_zero_row;
        };
        int chunk_nxt = 0, mt_nxt = gq;                    // chunk and accumulator tile of the next stage of this group
        auto advance = [&]() { while (mt_nxt >= MT) { mt_nxt -= MT; ++chunk_nxt; } };
        advance();
        if (gq < total_stages) { request(chunk_nxt, mt_nxt); decode(); }
        uint32_t slot = gq, use = 0;                       // (the ring has at least NGROUP stages)
        for (int s = gq; s < total_stages; s += NGROUP, slot += NGROUP) {
            if (slot >= (uint32_t) nstage) { slot -= nstage; ++use; }
            const int chunk = chunk_nxt, mt = mt_nxt;
            mt_nxt += NGROUP;
            advance();
            const bool more = s + NGROUP < total_stages;
            if (more) request(chunk_nxt, mt_nxt);          // in flight while this stage is issued
            if (use > 0 && !mbar_wait_warp(smem_u32(empty + slot), (use - 1) & 1, abort_flag)) { failed = true; break; }
            if (mt == 0) {
                // this warp's rows of the dO chunk, into the buffer of chunk - 2.  A wait by parity must know the phase before the awaited
                // one complete: the group that fills chunk c also filled c - 4 (groups take the stages modulo four), so with a barrier per
                // chunk modulo four every warp waits for all phases of the barriers it uses, one after the other.
                const uint32_t db = chunk & 1, before = (uint32_t) chunk - 2;
                if (chunk >= 2 && !mbar_wait_warp(smem_u32(dempty + before % DO_PHASES), (before / DO_PHASES) & 1, abort_flag)) { failed = true; break; }
                unsigned char* g_s = g_ring + db * G_BYTES;
                constexpr int GP = NCOL / 8;                           // 16-byte pieces of a dO row
                const int cc = lane % GP;
#pragma unroll
                for (int i = 0; i < GP; ++i) {
                    const int pl = i * (32 / GP) + lane / GP, r = wq * 32 + pl;
                    const int32_t a = __shfl_sync(0xffffffffu, g_row, pl);
                    const uint32_t off = NCOL == 32 ? r * 64 + ((cc ^ ((r >> 1) & 3)) << 4) : (cc >> 3) * G_ATOM + r * 128 + (((cc & 7) ^ (r & 7)) << 4);
                    if (cc < gpieces) cp_async16_or_zero(smem_u32(g_s) + off, P.grows + (ll) a * P.gpad + cob * NCOL + cc * 8, a != (int32_t) P.g_zero_row);
                }
                if (wq == 3) {                                         // rows 128 and 129
                    const int pl = lane / GP, r = PT + pl;
                    const int32_t a = __shfl_sync(0xffffffffu, g_extra, pl & 1);
                    const uint32_t off = NCOL == 32 ? r * 64 + ((cc ^ ((r >> 1) & 3)) << 4) : (cc >> 3) * G_ATOM + r * 128 + (((cc & 7) ^ (r & 7)) << 4);
                    if (pl < 2 && cc < gpieces) cp_async16_or_zero(smem_u32(g_s) + off, P.grows + (ll) a * P.gpad + cob * NCOL + cc * 8, a != (int32_t) P.g_zero_row);
                }
                cp_async_arrive_noinc(smem_u32(dfull + db));
            }
            unsigned char* a_s = a_ring + (size_t) slot * A_STAGE;
            const __nv_bfloat16* src0 = P.xrows + cib * CIB + c * 8;
#pragma unroll
            for (int tl = 0; tl < TPT; ++tl) {
                if (mt * TPT + tl >= nd) break;
                const int m = tl * CIB + c * 8;                        // accumulator row of this chunk's first channel
                const uint32_t dst0 = smem_u32(a_s + (m >> 6) * ATOM_STRIDE);
                const int cc = (m & 63) >> 3;
#pragma unroll
                for (int p0 = 0; p0 < PC; p0 += PB) {      // copies and shuffles keep their order: the rows of several copies are handed round first
                    int32_t r[PB];
#pragma unroll
                    for (int pi = 0; pi < PB; ++pi) r[pi] = __shfl_sync(0xffffffffu, rows_cur[tl], (p0 + pi) * RPI + r0);
#pragma unroll
                    for (int pi = 0; pi < PB; ++pi) {
                        const int k = wq * 32 + (p0 + pi) * RPI + r0;
                        if (c < cpieces) cp_async16_or_zero(dst0 + k * 128 + ((cc ^ (k & 7)) << 4), src0 + (ll) r[pi] * P.xpad, r[pi] != zero);
                    }
                }
            }
            // the stage's barrier receives this thread's arrival when the copies above have landed
            cp_async_arrive_noinc(smem_u32(full + slot));
            if (more) decode();
        }
        cp_async_commit();
        cp_async_wait<0>();
    } else if (warp == MMA_WARP && total_stages > 0) {
        // ---------------- MMA issue ----------------
        if (elect_one()) {
            uint32_t slot = 0, use = 0;
            bool ready = false;                   // the next stage is known to be there
            for (int chunk = 0; chunk < nchunks && !failed; ++chunk) {
                const uint32_t db = chunk & 1, duse = chunk >> 1;
                const uint32_t b_addr = smem_u32(g_ring + db * G_BYTES);
                for (int mt = 0; mt < MT; ++mt) {
                    if (!ready && !mbar_wait(smem_u32(full + slot), use & 1, abort_flag)) { failed = true; break; }
                    if (mt == 0 && !mbar_test(smem_u32(dfull + db), duse & 1) && !mbar_wait(smem_u32(dfull + db), duse & 1, abort_flag)) { failed = true; break; }
                    fence_proxy_async();          // generic-proxy writes of the cp.async copies -> tensor-core (async proxy) reads
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(a_ring + (size_t) slot * A_STAGE), used = slot;
                    if (++slot == (uint32_t) nstage) { slot = 0; ++use; }
#pragma unroll
                    for (int k = 0; k < PT / 16; ++k) {
                        // 16 slots = two 8-row groups; atoms along M are ATOM_STRIDE apart, along N one row (the next shift) or, for
                        // 128 columns, one atom
                        const uint64_t da = make_desc(a_addr + k * 2048, ATOM_STRIDE, 1024, 2);
                        if (k == PT / 32) ready = mbar_test(smem_u32(full + slot), use & 1);
#pragma unroll
                        for (int i = 0; i < MMAS; ++i) {
                            const uint64_t dbd = NCOL == 32 ? make_desc(b_addr + k * 1024, 64, 512, 4)
                                                            : make_desc(b_addr + k * 2048 + i * 128, NCOL == 64 ? 128 : G_ATOM, 1024, 2);
                            umma_bf16(tmem_d + mt * COLS + i * NCOL, da, dbd, IDESC, (chunk > 0 || k > 0) ? 1u : 0u);
                        }
                    }
                    umma_commit(smem_u32(empty + used));
                    if (mt == MT - 1) umma_commit(smem_u32(dempty + chunk % DO_PHASES));
                }
            }
            if (!failed) umma_commit(smem_u32(done));
        }
    }

    // ---------------- epilogue: warps 0-3 ----------------
    float* dst = P.partial + (ll) blockIdx.x * P.cout * P.cin * 27;
    if (warp < 4 && total_stages > 0 && !failed) {
        if (!mbar_wait_warp(smem_u32(done), 0, abort_flag)) failed = true;
        if (!failed) {
            tc_fence_after();
            const int row = warp * 32 + lane;                 // accumulator row = (neighbour within tile) * CIB + ci
            const int tl = row / CIB, ci = cib * CIB + row % CIB;
            for (int mt = 0; mt < MT; ++mt) {
                const int d = mt * TPT + tl;
#pragma unroll 1
                for (int c0 = 0; c0 < COLS; c0 += 32) {
                    uint32_t r[32];
                    tmem_ld32(tmem_d + ((uint32_t) (warp * 32) << 16) + mt * COLS + c0, r);
                    tmem_ld_wait();
                    if (d < nd && ci < P.cin) {
                        const int tap = (d0 + d) * 3 + 2 - c0 / NCOL;      // block i of the columns holds dy = 1 - i
                        const int co0 = cob * NCOL + c0 % NCOL;
                        float* o = dst + ((ll) tap * P.cout + co0) * P.cin + ci;         // the lanes lie along ci
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (co0 + j < P.cout) o[(ll) j * P.cin] = __uint_as_float(r[j]);
                    }
                }
            }
        }
    }

    if (failed) {
        *abort_flag = 1;
        if (P.error_flag) *P.error_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) tmem_dealloc(tmem_d, 512);
}

template<int CIB, int NCOL>
int launch_dw(const DwParams& P, int nranges, int blocks_y, cudaStream_t st, const char* pname) {
    constexpr size_t G_BYTES = ((size_t) G_ROWS * (NCOL == 32 ? 64 : 128) * (NCOL == 128 ? 2 : 1) + 1023) / 1024 * 1024;
    const size_t fixed = 2 * G_BYTES + (2 * DW_MAX_STAGES + 2 + DO_PHASES + 1) * 8 + 16 + 1024;
    // A wait for a ring slot must find the phase before the awaited one complete (its parity test cannot tell two phases apart): with at
    // least NGROUP stages the group has by then seen a later stage of that round read.  The dO buffers have barriers of their own.
    const int nstage = (int) std::min<size_t>(DW_MAX_STAGES, (227 * 1024 - fixed) / A_STAGE);
    if (nstage < NGROUP) { aprnet_set_error("conv333 tensor-core weight gradient: ring of %d stages", nstage); return APRNET_ERR_UNSUPPORTED; }
    const size_t smem = (size_t) nstage * A_STAGE + fixed;
    auto kern = conv333_tc_dw_kernel<CIB, NCOL>;
    APRNET_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    dim3 grid((unsigned) nranges, (unsigned) blocks_y);
    { AprnetProfScope _prof(pname, st);
    kern<<<grid, DW_THREADS, smem, st>>>(P, nstage);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

} // namespace

int g_dw_waves_override = 0;     // aprnet_tc_set_option("dw_waves", n): waves of blocks of the weight gradient, measurement switch

extern "C" int64_t aprnet_conv333_tc_dw_partial_elems(int cin, int cout) {
    const ll per = (ll) 27 * cin * cout;
    const ll ranges = std::max<ll>(32, std::min<ll>(1024, (64ll << 20) / per));     // at least one per level plus room for a wave
    return (int64_t) (ranges * per);
}

// xrows / grows: channels-last bf16 copies of the input (+ tree means + zero row) and of grad_output
// (+ zero row) as produced by aprnet_pack_rows_bf16.  grad_weights (slots, Cout, Cin, 27) fp32 is
// accumulated into or written.
int aprnet_tc_backward_weights(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* xrows, int xpad, const void* grows, int gpad, float* gw, int accumulate,
                               float* partial, cudaStream_t st) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && cin > 0 && cout > 0 && slots > 0 && xrows && grows && gw && partial, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(xpad % 16 == 0 && gpad % 16 == 0 && xpad >= cin && gpad >= cout, "packed row widths must be multiples of 16");
    const RunPlan* rp = aprnet_get_run_plan(a, dl, st);
    if (!rp) return APRNET_ERR_CUDA;
    const ll n = a->number_parts(dl), t = a->tree_size(dl);
    // one block of input channels where they fit (rows are then gathered once per neighbour), 128 at a time beyond
    const int cib = xpad <= 16 ? 16 : (xpad <= 32 ? 32 : (xpad <= 64 ? 64 : 128));
    const int ncol = gpad <= 32 ? 32 : (gpad <= 64 ? 64 : 128);
    const int ci_blocks = (xpad + cib - 1) / cib, co_blocks = (gpad + ncol - 1) / ncol;
    const int max_d = 512 / (3 * ncol) * (128 / cib);                      // neighbours whose accumulators fit the 512 TMEM columns
    const int groups = (9 + max_d - 1) / max_d, d_per_group = (9 + groups - 1) / groups;
    const int blocks_y = groups * ci_blocks * co_blocks;
    const ll elems = (ll) 27 * cin * cout;
    const ll max_ranges = aprnet_conv333_tc_dw_partial_elems(cin, cout) / elems;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    char pname[64];
    snprintf(pname, sizeof(pname), "conv333_tc_dw:ci%d:co%d:dl%d", cin, cout, dl);
    // one launch over all levels, blocks for `waves` waves of one block per SM where the partial buffer and the number
    // of levels allow it: every level gets blocks in proportion to its chunks (at most `per_block` chunks each); a level's partial
    // sums are added into the slot of that level afterwards
    const std::vector<Segment> segs = aprnet_segments(a, dl, slots, false);
    DwParams P;
    P.n_segs = 0;
    SlotRanges sr;
    sr.n = 0;
    ll total_chunks = 0;
    for (const Segment& sg : segs) {
        P.seg_begin[P.n_segs] = rp->level_begin[sg.level]; P.seg_end[P.n_segs] = rp->level_begin[sg.level + 1];
        total_chunks += (P.seg_end[P.n_segs] - P.seg_begin[P.n_segs] + PT - 1) / PT;
        ++P.n_segs;
    }
    if (total_chunks == 0) return accumulate ? APRNET_OK : aprnet_dw_reduce(partial, sr, slots, 0, cin, cout, gw, st);
    // How many ranges: the tensor cores truncate their sums, so the error of a result grows with the products that one accumulator takes
    // one after the other (32 -> 64 channels on 2 M locations, relative error of the sums: 1.5e-5 with 148 ranges, 5e-6 with 370).  At
    // least as many ranges per location as two waves of blocks give whose accumulators fill TMEM (65536 each) without gaps, then whole
    // waves of the blocks at hand, so that the last one is not nearly empty.
    const ll full = ((ll) 27 * xpad * ((gpad + 63) / 64 * 64) + 65535) / 65536;
    const ll need = (ll) std::ceil(2.0 * sms * ((double) total_chunks * PT / (double) std::max<ll>(n, 1)) / (double) full);
    const ll waves = g_dw_waves_override > 0 ? g_dw_waves_override : (need * blocks_y + sms - 1) / sms;
    ll budget = std::max<ll>(P.n_segs, std::min<ll>(waves * sms / blocks_y, max_ranges));
    auto blocks_of = [&](int i, ll per_block) { return ((P.seg_end[i] - P.seg_begin[i] + PT - 1) / PT + per_block - 1) / per_block; };
    auto blocks_for = [&](ll per_block) { ll b = 0; for (int i = 0; i < P.n_segs; ++i) b += blocks_of(i, per_block); return b; };
    // (at least four chunks per block: the block sums of 256 x 256 channels are 7 MB per range)
    ll per_block = std::max<ll>(4, (total_chunks + budget - 1) / budget);
    while (blocks_for(per_block) > budget) ++per_block;
    P.range_first[0] = 0;
    for (int i = 0; i < P.n_segs; ++i) {
        P.range_first[i + 1] = P.range_first[i] + (int) blocks_of(i, per_block);
        // levels are listed coarse to fine, so those that share a slot (the last one) are neighbours
        if (sr.n == 0 || sr.slot[sr.n - 1] != segs[i].slot) { sr.first[sr.n] = P.range_first[i]; sr.slot[sr.n++] = segs[i].slot; }
        sr.first[sr.n] = P.range_first[i + 1];
    }
    const int nranges = P.range_first[P.n_segs];
    if (nranges > max_ranges) { aprnet_set_error("conv333 tensor-core weight gradient: %d ranges exceed the partial buffer", nranges); return APRNET_ERR_ARG; }
    P.src = rp->src; P.S = rp->n_slots; P.loc = rp->loc;
    P.xrows = (const __nv_bfloat16*) xrows; P.xpad = xpad; P.tree_base = n; P.zero_row = n + t;
    P.grows = (const __nv_bfloat16*) grows; P.gpad = gpad; P.g_zero_row = n;
    P.partial = partial; P.cin = cin; P.cout = cout; P.ci_blocks = ci_blocks; P.groups = groups; P.d_per_group = d_per_group;
    P.error_flag = aprnet_tc_error_flag_device();
    int rc;
#define DW_CASE(CIB_, NCOL_) if (cib == CIB_ && ncol == NCOL_) rc = launch_dw<CIB_, NCOL_>(P, nranges, blocks_y, st, pname); else
    DW_CASE(16, 32) DW_CASE(16, 64) DW_CASE(16, 128)
    DW_CASE(32, 32) DW_CASE(32, 64) DW_CASE(32, 128)
    DW_CASE(64, 32) DW_CASE(64, 64) DW_CASE(64, 128)
    DW_CASE(128, 32) DW_CASE(128, 64) DW_CASE(128, 128)
    { aprnet_set_error("conv333 tensor-core weight gradient: unsupported blocking"); return APRNET_ERR_UNSUPPORTED; }
#undef DW_CASE
    return rc ? rc : aprnet_dw_reduce(partial, sr, slots, accumulate, cin, cout, gw, st);
}

extern "C" int aprnet_conv333_backward_weights_tc(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* xrows, int xpad,
                                                  const void* grows, int gpad, float* gw, float* partial, void* stream) {
    return aprnet_tc_backward_weights(a, dl, cin, cout, slots, xrows, xpad, grows, gpad, gw, 1, partial, (cudaStream_t) stream);
}
