// 1x1x1 particle convolution on the tensor cores (bf16 operands, fp32 accumulate).
//
// Replaces pyapr/aprnet/cuda/src/conv111_gpu.cu:9-232 for float32 tensors when the layer's precision is "bf16".
// out[o][p] = sum_i w[slot(level of p)][o][i] * in[i][p] is a plain [locations x Cin] . [Cin x Cout] product per
// level; with 2 * Cin * Cout flops against 4 * (Cin + Cout) bytes per location the CUDA-core kernel sits at the
// fp32 multiply-add bound, the tensor-core kernel at the HBM bound.
//
// One persistent block per SM, 21 warps:
//   warps 0-11  producers, three groups of 128 threads that take the tiles of 128 locations in turn (a fourth leaves 72 registers per
//               thread, and the epilogue spills).  A thread owns one location:
//               it requests up to 32 input channels at a time (4-byte loads, coalesced across the warp along the location
//               axis of the channel-major tensor), rounds them to bf16 and writes them as 16-byte pieces of the K-major,
//               hardware-swizzled A operand (the transposition happens in registers), then one arrival per warp on the
//               stage's barrier;
//   warp 12     one thread waits for the stage, fences the generic-proxy writes against the tensor core's reads and
//               issues the Cin / 16 tcgen05.mma (M = 128, N = padded Cout) of each tile and commits the
//               stage's "slot free" barrier and the accumulator's "complete" barrier;
//   warps 13-20 epilogue, two sets of four warps on the two tiles of a unit: TMEM -> registers (+ bias) -> shared memory ->
//               fp32 stores of out[o][p].  The rows of the channel-major tensor start at any multiple of four bytes, and a store that
//               straddles two 128-byte lines costs two partial writes: writing 128 rows of 3.5 M locations from 64 ran at 3.3 TB/s, with
//               aligned rows at 5.  So two neighbouring tiles (256 locations) are written together, 16 channels at a time, and every store
//               covers what one line holds of them: 64 -> 128 channels on 3.5 M locations 0.85 -> 0.55 ms
//               (0.42 ms at the HBM rate; the chain TMEM -> shared memory -> line is what is left).
// The weights of one level (B operand, bf16, all of Cin x Cout) stay in shared memory; the block walks the levels one
// after the other and converts the next level's weights from the fp32 tensor between two block-wide barriers.
// Every wait is bounded and polls a block-wide abort flag; after an expiry the block raises the library's error flag,
// skips the remaining work (all block-wide barriers are still reached) and returns.
#include "apr_device.cuh"
#include "tc_ptx.cuh"
#include <cuda_bf16.h>
#include <algorithm>

int* aprnet_tc_error_flag_device();

namespace {

using namespace tcptx;
typedef long long ll;
constexpr int TILE_M = 128;
constexpr int C1_GROUPS = 3, C1_MMA = 4 * C1_GROUPS;
constexpr int C1_THREADS = (C1_MMA + 9) * 32;
constexpr int DW_GROUPS = 2, DW_MMA = 8 * DW_GROUPS;
constexpr int C1_THREADS_DW = (DW_MMA + 5) * 32;
constexpr int C1_MAX_STAGES = 8;
constexpr int C1_MAX_ACC = 4;
constexpr int C1_OUT_CH = 16, C1_OUT_BYTES = 2 * C1_OUT_CH * 2 * TILE_M * 4;    // staged output: two buffers of 16 channels x 256 locations
constexpr int C1_SMEM = 227 * 1024 - 1024;                                       // (the biases are static)
constexpr int C1_MAX_SEGS = APRNET_MAX_LEVELS;

struct C1Params {
    int n_segs;
    ll seg_begin[C1_MAX_SEGS], seg_end[C1_MAX_SEGS];
    int seg_slot[C1_MAX_SEGS];
    const float* in; ll ld_in; int n_in;           // K = n_in channels
    const float* w; ll ws, wo, wi;                 // element (slot, o, i) at w[slot * ws + o * wo + i * wi]
    float* out; ll ld_out; int n_out;
    const float* bias;                             // added to every output channel (null: none)
    int kpad;                                      // n_in padded to 16, 32 or a multiple of 64
    int* error_flag;
};

template<int KS> __device__ __forceinline__ int swz_chunk(int row, int c) {      // position of 16-byte chunk c of row `row`
    return KS == 64 ? (c ^ (row & 7)) : (KS == 32 ? (c ^ ((row >> 1) & 3)) : (c ^ ((row >> 2) & 1)));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// One unit (two neighbouring tiles, 256 locations) of the channel-major result from its accumulators, by the eight epilogue warps: TMEM -> shared memory ->
// stores that each cover what one line holds.  w8: the warp among the eight, which are two sets of four; has: this set's tile exists; piece: 16-channel pieces staged so far.  (A failed warp keeps the pace of the barriers.)
__device__ __forceinline__ void store_unit(float* __restrict__ out, ll ld_out, int n_out, const float* bias_s, ll p0, int cnt, bool has, uint32_t acc_addr, uint32_t full_bar, uint32_t full_parity,
                                           uint32_t empty_bar, float* out_s, int w8, int& piece, bool& failed, volatile int* abort_flag) {
    constexpr int LINES = 2 * TILE_M / 32 + 1;
    const int lane = threadIdx.x & 31, q = (threadIdx.x >> 5) & 3, set = w8 >> 2;         // q: TMEM lane group this warp may read
    if (has && !failed && !mbar_wait_warp(full_bar, full_parity, abort_flag)) failed = true;
    const bool live = has && !failed;
    tc_fence_after();
    const uint32_t taddr = acc_addr + ((uint32_t) (q * 32) << 16);
    uint32_t r[C1_OUT_CH];
    if (live) tmem_ld16(taddr, r);
#pragma unroll 1
    for (int c0 = 0; c0 < n_out; c0 += C1_OUT_CH) {
        float* buf = out_s + (piece++ & 1 ? C1_OUT_CH * 2 * TILE_M : 0);
        if (live) {
            tmem_ld_wait();
            float* dst = buf + set * TILE_M + q * 32 + lane;
#pragma unroll
            for (int jj = 0; jj < C1_OUT_CH; ++jj) dst[jj * 2 * TILE_M] = __uint_as_float(r[jj]);
            if (c0 + C1_OUT_CH < n_out) tmem_ld16(taddr + c0 + C1_OUT_CH, r);      // read while this piece is stored
        }
        // the buffer is written again after the barrier of the other one
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (failed) continue;
#pragma unroll
        for (int k = 0; k < C1_OUT_CH / 8; ++k) {
            const int c = k * 8 + w8;
            if (c0 + c >= n_out) break;
            float* o = out + (ll) (c0 + c) * ld_out + p0;
            const int e0 = lane - (int) ((reinterpret_cast<uintptr_t>(o) >> 2) & 31);
            const float* src = buf + c * 2 * TILE_M + e0;
            float v[LINES];
#pragma unroll
            for (int i = 0; i < LINES; ++i) v[i] = e0 + i * 32 >= 0 && e0 + i * 32 < 2 * TILE_M ? src[i * 32] : 0.f;
            if (bias_s) {
                const float bias = bias_s[c0 + c];
#pragma unroll
                for (int i = 0; i < LINES; ++i) v[i] += bias;
            }
            o += e0;
#pragma unroll
            for (int i = 0; i < LINES; ++i)
                if (e0 + i * 32 >= 0 && e0 + i * 32 < cnt) o[i * 32] = v[i];
        }
    }
    tc_fence_before();
    __syncwarp();
    if (live && lane == 0) mbar_arrive(empty_bar);
}

template<int NT, int KS>
__global__ void __launch_bounds__(C1_THREADS, 1) conv111_tc_kernel(const C1Params P, const int stages) {
    constexpr int ACC_COLS = NT < 32 ? 32 : NT;                 // TMEM columns per accumulator
    constexpr int NACC = NT <= 128 ? 4 : 2;
    constexpr int ROW_BYTES = KS * 2;
    constexpr int A_SUB = TILE_M * ROW_BYTES;                   // one K chunk of KS channels
    constexpr uint32_t A_LAYOUT = KS == 64 ? 2u : (KS == 32 ? 4u : 6u);
    constexpr uint32_t IDESC = make_idesc(NT, false, false);
    constexpr int KB = KS < 32 ? KS : 32;                       // channels a producer thread requests together

    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ float bias_s[ACC_COLS];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int kchunks = P.kpad / KS;
    const int a_stage = kchunks * A_SUB;
    unsigned char* a_ring = smem;                                                   // stages x [kchunks][128][KS] bf16, swizzled
    unsigned char* b_s = a_ring + (size_t) stages * a_stage;                        // [kpad / 8][NT][8] bf16
    float* out_s = reinterpret_cast<float*>(b_s + (size_t) NT * P.kpad * 2);        // [2][C1_OUT_CH][256]
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_s + C1_OUT_BYTES / 4);
    uint64_t* full = bars;                              // [stages] operand written (4 producer warps)
    uint64_t* empty = bars + C1_MAX_STAGES;             // [stages] MMAs that read the stage completed
    uint64_t* tmem_full = empty + C1_MAX_STAGES;        // [NACC]   accumulator complete
    uint64_t* tmem_empty = tmem_full + C1_MAX_ACC;      // [NACC]   accumulator read back (4 epilogue warps)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + C1_MAX_ACC);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = warp_number(), lane = tid & 31;
    for (int c = tid; c < ACC_COLS; c += C1_THREADS) bias_s[c] = P.bias && c < P.n_out ? P.bias[c] : 0.f;
    if (tid == 0) {
        for (int i = 0; i < stages; ++i) { mbar_init(smem_u32(full + i), 4); mbar_init(smem_u32(empty + i), 1); }
        for (int i = 0; i < NACC; ++i) { mbar_init(smem_u32(tmem_full + i), 1); mbar_init(smem_u32(tmem_empty + i), 4); }
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == C1_MMA) { tmem_alloc(smem_u32(tmem_slot), NACC * ACC_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = *tmem_slot;
    bool failed = false;
    const int ngroups = min(C1_GROUPS, stages);      // (a ring at least as long as the groups keeps the phases that a wait can meet apart)
    int piece = 0;                          // 16-channel pieces the epilogue has staged
    const int w8 = warp - C1_MMA - 1, set = w8 >> 2;       // epilogue: two sets of four warps on the two tiles of a unit
    uint32_t j_base = 0;                    // tiles this block has been given in the levels before the current one

    for (int seg = 0; seg < P.n_segs; ++seg) {
        const ll sb = P.seg_begin[seg], se = P.seg_end[seg];
        const int seg_tiles = (int) ((se - sb + TILE_M - 1) / TILE_M);
        // units of two neighbouring tiles, of one where every block gets at most one tile
        const int pair = seg_tiles > (int) gridDim.x ? 1 : 0;
        const int seg_units = (seg_tiles + pair) >> pair;
        const int units = (int) blockIdx.x < seg_units ? (seg_units - (int) blockIdx.x + (int) gridDim.x - 1) / (int) gridDim.x : 0;
        const int mine = (units << pair) - (units > 0 && (seg_tiles & pair) && (seg_units - 1) % (int) gridDim.x == (int) blockIdx.x ? 1 : 0);
        auto tile_begin = [&](int it) { return sb + ((((ll) blockIdx.x + (ll) (it >> pair) * gridDim.x) << pair) + (it & pair)) * TILE_M; };
        // ---- the level's weights -> B operand (every accumulator of the previous level has been read back) ----
        __syncthreads();
        {
            const float* wslot = P.w + (ll) P.seg_slot[seg] * P.ws;
            const int nk8 = P.kpad / 8;
            for (int e = tid; e < NT * nk8; e += C1_THREADS) {
                const int n = e % NT, k8 = e / NT;
                float v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int k = k8 * 8 + q;
                    v[q] = (n < P.n_out && k < P.n_in) ? __ldg(wslot + (ll) n * P.wo + (ll) k * P.wi) : 0.f;
                }
                uint4 pk;
                pk.x = pack_bf16x2(v[0], v[1]); pk.y = pack_bf16x2(v[2], v[3]); pk.z = pack_bf16x2(v[4], v[5]); pk.w = pack_bf16x2(v[6], v[7]);
                *reinterpret_cast<uint4*>(b_s + ((size_t) k8 * NT + n) * 16) = pk;
            }
            fence_proxy_async();
        }
        __syncthreads();
        tc_fence_after();

        if (warp < C1_MMA) {
            // ---------------- producers ----------------
            const int grp = warp >> 2, row = tid & 127;
            for (int it = grp; grp < ngroups && it < mine && !failed; it += ngroups) {
                const uint32_t j = j_base + (uint32_t) it, slot = j % (uint32_t) stages, use = j / (uint32_t) stages;
                const float* src = P.in + min(tile_begin(it) + row, se - 1);     // rows past the end repeat the last location and are not stored
                float v[KB];
                auto request = [&](int kb) {
                    const float* s = src + (ll) kb * P.ld_in;
                    if (kb + KB <= P.n_in) {                                     // no condition per load
#pragma unroll
                        for (int q = 0; q < KB; ++q) { v[q] = *s; s += P.ld_in; }
                    } else {
#pragma unroll
                        for (int q = 0; q < KB; ++q) v[q] = kb + q < P.n_in ? s[(ll) q * P.ld_in] : 0.f;
                    }
                };
                request(0);             // in flight while this warp waits for the ring slot
                if (use > 0 && !mbar_wait_warp(smem_u32(empty + slot), (use - 1) & 1, abort_flag)) { failed = true; break; }
                unsigned char* a_s = a_ring + (size_t) slot * a_stage;
                for (int kb = 0; kb < P.kpad; kb += KB) {
                    if (kb > 0) request(kb);
                    unsigned char* sub = a_s + (size_t) (kb / KS) * A_SUB + row * ROW_BYTES;
                    const int c0 = (kb % KS) / 8;
#pragma unroll
                    for (int q8 = 0; q8 < KB / 8; ++q8) {
                        uint4 pk;
                        pk.x = pack_bf16x2(v[q8 * 8 + 0], v[q8 * 8 + 1]); pk.y = pack_bf16x2(v[q8 * 8 + 2], v[q8 * 8 + 3]);
                        pk.z = pack_bf16x2(v[q8 * 8 + 4], v[q8 * 8 + 5]); pk.w = pack_bf16x2(v[q8 * 8 + 6], v[q8 * 8 + 7]);
                        *reinterpret_cast<uint4*>(sub + (swz_chunk<KS>(row, c0 + q8) << 4)) = pk;
                    }
                }
                // (no proxy fence here: the MMA thread fences after its wait)
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(full + slot));
            }
        } else if (warp == C1_MMA) {
            // ---------------- MMA issue ----------------
            if (elect_one()) {
                for (int it = 0; it < mine && !failed; ++it) {
                    const uint32_t j = j_base + (uint32_t) it, slot = j % (uint32_t) stages, use = j / (uint32_t) stages;
                    const uint32_t acc = j % NACC, acc_use = j / NACC;
                    if (acc_use > 0 && !mbar_wait(smem_u32(tmem_empty + acc), (acc_use - 1) & 1, abort_flag)) { failed = true; break; }
                    if (!mbar_wait(smem_u32(full + slot), use & 1, abort_flag)) { failed = true; break; }
                    fence_proxy_async();          // generic-proxy writes of the producers -> tensor-core (async proxy) reads
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(a_ring + (size_t) slot * a_stage);
                    const uint64_t db0 = make_desc(smem_u32(b_s), NT * 16, 128, 0);
                    for (int kc = 0; kc < kchunks; ++kc) {
                        const uint64_t da0 = make_desc(a_addr + kc * A_SUB, 16, 8 * ROW_BYTES, A_LAYOUT);
#pragma unroll
                        for (int k = 0; k < KS / 16; ++k)
                            umma_bf16(tmem_d + acc * ACC_COLS, da0 + (uint64_t) ((k * 32) >> 4),
                                      db0 + (uint64_t) (((kc * (KS / 16) + k) * 2 * (NT * 16)) >> 4), IDESC, (kc > 0 || k > 0) ? 1u : 0u);
                    }
                    umma_commit(smem_u32(empty + slot));
                    umma_commit(smem_u32(tmem_full + acc));
                }
            }
        } else {
            // ---------------- epilogue ----------------
            for (int u = 0; u < units; ++u) {
                const int it = (u << pair) + set;
                const uint32_t j = j_base + (uint32_t) it;
                store_unit(P.out, P.ld_out, P.n_out, P.bias ? bias_s : nullptr, tile_begin(u << pair), (int) min(se - tile_begin(u << pair), (ll) (TILE_M << pair)), set <= pair && it < mine,
                           tmem_d + (j % NACC) * ACC_COLS, smem_u32(tmem_full + j % NACC), (j / NACC) & 1, smem_u32(tmem_empty + j % NACC), out_s, w8, piece, failed, abort_flag);
            }
        }
        if (failed) *abort_flag = 1;
        j_base += (uint32_t) mine;
    }

    if (failed) {
        *abort_flag = 1;
        if (P.error_flag) *P.error_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == C1_MMA) tmem_dealloc(tmem_d, NACC * ACC_COLS);
}

inline int pad_k(int c) { return c <= 16 ? 16 : (c <= 32 ? 32 : (c + 63) / 64 * 64); }
inline int pick_nt(int n) { return n <= 16 ? 16 : (n <= 32 ? 32 : (n <= 64 ? 64 : (n <= 128 ? 128 : 256))); }

template<int NT, int KS>
int launch_c1(const C1Params& P, ll total_tiles, cudaStream_t st, const char* pname) {
    const size_t a_stage = (size_t) TILE_M * P.kpad * 2, b_bytes = (size_t) NT * P.kpad * 2;
    const size_t fixed = b_bytes + C1_OUT_BYTES + (2 * C1_MAX_STAGES + 2 * C1_MAX_ACC) * 8 + 16 + 1024;
    if (fixed + 2 * a_stage > C1_SMEM) return APRNET_ERR_UNSUPPORTED;
    const int stages = (int) std::min<size_t>(C1_MAX_STAGES, (C1_SMEM - fixed) / a_stage);
    const size_t smem = (size_t) stages * a_stage + fixed;
    auto kern = conv111_tc_kernel<NT, KS>;
    APRNET_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int grid = (int) std::min<ll>(total_tiles, sms);
    { AprnetProfScope _prof(pname, st);
    kern<<<grid, C1_THREADS, smem, st>>>(P, stages);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

// out[o][p] = sum_i w[slot][o][i] in[i][p] over the locations of level delta dl
int run_conv111_tc(const aprnet_apr* a, int dl, int n_in, int n_out, int slots, const float* in, ll ld_in, const float* w, ll ws, ll wo, ll wi,
                   const float* bias, float* out, ll ld_out, cudaStream_t st, const char* pname) {
    // narrow layers (a classifier head) are bound by their one wide tensor either way and run faster on the CUDA cores
    if (n_out > 256 || n_in > 256 || n_in < 8 || n_out < 8) return APRNET_ERR_UNSUPPORTED;
    const std::vector<Segment> segs = aprnet_segments(a, dl, slots, true);
    C1Params P;
    P.n_segs = 0;
    ll total_tiles = 0;
    for (const Segment& s : segs) {
        if (s.end <= s.begin) continue;
        if (P.n_segs >= C1_MAX_SEGS) return APRNET_ERR_UNSUPPORTED;
        P.seg_begin[P.n_segs] = s.begin; P.seg_end[P.n_segs] = s.end; P.seg_slot[P.n_segs] = s.slot;
        total_tiles = std::max<ll>(total_tiles, (s.end - s.begin + TILE_M - 1) / TILE_M);
        ++P.n_segs;
    }
    if (P.n_segs == 0) return APRNET_OK;
    P.in = in; P.ld_in = ld_in; P.n_in = n_in; P.w = w; P.ws = ws; P.wo = wo; P.wi = wi; P.out = out; P.ld_out = ld_out; P.n_out = n_out; P.bias = bias;
    P.kpad = pad_k(n_in);
    P.error_flag = aprnet_tc_error_flag_device();
    const int nt = pick_nt(n_out), ks = std::min(64, P.kpad);
#define C1_CASE(NT_, KS_) if (nt == NT_ && ks == KS_) return launch_c1<NT_, KS_>(P, total_tiles, st, pname);
    C1_CASE(16, 16) C1_CASE(16, 32) C1_CASE(16, 64) C1_CASE(32, 16) C1_CASE(32, 32) C1_CASE(32, 64)
    C1_CASE(64, 16) C1_CASE(64, 32) C1_CASE(64, 64) C1_CASE(128, 16) C1_CASE(128, 32) C1_CASE(128, 64)
    C1_CASE(256, 16) C1_CASE(256, 32) C1_CASE(256, 64)
#undef C1_CASE
    return APRNET_ERR_UNSUPPORTED;
}


// ---- weight gradient -----------------------------------------------------------------------------------
// gw[slot][o][i] += sum over the locations p of the slot's levels of gout[o][p] * in[i][p]: M = output channels (padded
// to 128 per accumulator), N = input channels, K = locations.  Both tensors are channel-major, i.e. K-major operands
// as they lie in memory; they only have to be rounded to bf16.  One persistent block per SM walks its share of the
// 128-location tiles of ONE level range and keeps the accumulators in TMEM until the end:
//   warps 0-15  producers, two groups of eight warps on alternate tiles: a warp takes channel rows of both tensors in turn, 32 consecutive locations per load
//               instruction (coalesced), and writes each value as a 2-byte piece of the swizzled K-major operand row
//               (conflict-free: the 32 lanes fill 64 bytes of one 128-byte row); locations past the end are zeros;
//   warp 16     one thread issues 8 tcgen05.mma per accumulator and stage;
//   warps 17-20 after the last tile: TMEM -> partial sums of this block; a second kernel adds the blocks in fixed order.
struct C1DwParams {
    ll seg_begin, seg_end;
    const float* in; ll ld_in; int cin;
    const float* gout; ll ld_out; int cout;
    float* partial;                         // [block][cout][cin]
    int* error_flag;
};

template<int NT>
__global__ void __launch_bounds__(C1_THREADS_DW, 1) conv111_tc_dw_kernel(const C1DwParams P, const int stages, const int mtiles) {
    constexpr int SUB = 64;                                  // locations per swizzle atom row (128 bytes)
    constexpr uint32_t IDESC = make_idesc(NT, false, false);
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int a_rows = mtiles * 128;
    const int stage_bytes = (a_rows + NT) * 256;             // two 64-location halves of 128 bytes per channel row
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t) stages * stage_bytes);
    uint64_t* full = bars;                                   // [stages] operands written (the eight warps of a group)
    uint64_t* empty = bars + C1_MAX_STAGES;                  // [stages] MMAs that read the stage completed
    uint64_t* done = empty + C1_MAX_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = warp_number(), lane = tid & 31;
    const uint32_t tmem_cols = mtiles * NT <= 32 ? 32u : (mtiles * NT <= 64 ? 64u : (mtiles * NT <= 128 ? 128u : (mtiles * NT <= 256 ? 256u : 512u)));
    if (tid == 0) {
        for (int i = 0; i < stages; ++i) { mbar_init(smem_u32(full + i), 8); mbar_init(smem_u32(empty + i), 1); }
        mbar_init(smem_u32(done), 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == DW_MMA) { tmem_alloc(smem_u32(tmem_slot), tmem_cols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = *tmem_slot;
    bool failed = false;
    const ll sb = P.seg_begin, se = P.seg_end;
    const int seg_tiles = (int) ((se - sb + TILE_M - 1) / TILE_M);
    const int mine = (int) blockIdx.x < seg_tiles ? (seg_tiles - (int) blockIdx.x + (int) gridDim.x - 1) / (int) gridDim.x : 0;

    if (warp < DW_MMA) {
        // ---------------- producers ----------------
        const int nrows = P.cout + P.cin;                    // channel rows of a stage: gout rows, then in rows
        for (int it = warp >> 3; it < mine && !failed; it += DW_GROUPS) {
            const uint32_t slot = (uint32_t) it % (uint32_t) stages, use = (uint32_t) it / (uint32_t) stages;
            const ll p0 = sb + ((ll) blockIdx.x + (ll) it * gridDim.x) * TILE_M;
            if (use > 0 && !mbar_wait_warp(smem_u32(empty + slot), (use - 1) & 1, abort_flag)) { failed = true; break; }
            unsigned char* st = smem + (size_t) slot * stage_bytes;
            const bool whole = p0 + TILE_M <= se;
            for (int r0 = warp & 7; r0 < nrows; r0 += 8 * 8) {   // 8 rows of this warp x 4 quarters of 32 locations in flight
                float v[8][4];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int r = min(r0 + u * 8, nrows - 1);     // (the rows that repeat are not stored)
                    const float* src = (r < P.cout ? P.gout + (ll) r * P.ld_out : P.in + (ll) (r - P.cout) * P.ld_in) + p0 + lane;
                    if (whole) {                                  // no condition per load: a branch each cost more than the load
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[u][q] = src[q * 32];
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[u][q] = p0 + q * 32 + lane < se ? src[q * 32] : 0.f;
                    }
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int r = r0 + u * 8;
                    if (r >= nrows) break;
                    // operand row: gout rows first (accumulator rows), in rows after a_rows
                    const int orow = r < P.cout ? r : a_rows + (r - P.cout);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int pl = q * 32 + lane;                     // location within the tile
                        const int half = pl / SUB, k = pl % SUB;
                        unsigned char* dst = st + (size_t) half * ((size_t) (a_rows + NT) * 128) + (size_t) orow * 128
                                           + ((((k >> 3) ^ (orow & 7)) << 4) | ((k & 7) << 1));
                        *reinterpret_cast<__nv_bfloat16*>(dst) = __float2bfloat16(v[u][q]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(full + slot));   // the MMA thread fences the generic-proxy writes after its wait
        }
    } else if (warp == DW_MMA) {
        // ---------------- MMA issue ----------------
        if (elect_one()) {
            for (int it = 0; it < mine && !failed; ++it) {
                const uint32_t slot = (uint32_t) it % (uint32_t) stages, use = (uint32_t) it / (uint32_t) stages;
                if (!mbar_wait(smem_u32(full + slot), use & 1, abort_flag)) { failed = true; break; }
                fence_proxy_async();
                tc_fence_after();
                const uint32_t base = smem_u32(smem + (size_t) slot * stage_bytes);
                for (int half = 0; half < 2; ++half) {
                    const uint32_t hb = base + half * ((a_rows + NT) * 128);
                    const uint64_t db0 = make_desc(hb + a_rows * 128, 16, 1024, 2);
                    for (int mt = 0; mt < mtiles; ++mt) {
                        const uint64_t da0 = make_desc(hb + mt * 128 * 128, 16, 1024, 2);
#pragma unroll
                        for (int k = 0; k < SUB / 16; ++k)
                            umma_bf16(tmem_d + mt * NT, da0 + (uint64_t) ((k * 32) >> 4), db0 + (uint64_t) ((k * 32) >> 4), IDESC,
                                      (it > 0 || half > 0 || k > 0) ? 1u : 0u);
                    }
                }
                umma_commit(smem_u32(empty + slot));
            }
            if (!failed) umma_commit(smem_u32(done));
        }
    }
    // ---------------- epilogue: the last four warps ----------------
    float* dst = P.partial + (ll) blockIdx.x * P.cout * P.cin;
    if (warp > DW_MMA && mine > 0 && !failed) {
        if (!mbar_wait_warp(smem_u32(done), 0, abort_flag)) failed = true;
        if (!failed) {
            tc_fence_after();
            const int q = warp & 3, row = q * 32 + lane;
            for (int mt = 0; mt < mtiles; ++mt) {
                const int o = mt * 128 + row;
#pragma unroll
                for (int c0 = 0; c0 < NT; c0 += 32) {
                    uint32_t r[32];
                    tmem_ld32(tmem_d + ((uint32_t) (q * 32) << 16) + mt * NT + c0, r);
                    tmem_ld_wait();
                    if (o < P.cout) {
#pragma unroll
                        for (int jj = 0; jj < 32; ++jj)
                            if (c0 + jj < P.cin) dst[(ll) o * P.cin + c0 + jj] = __uint_as_float(r[jj]);
                    }
                }
            }
        }
    } else if (mine == 0) {
        for (int e = tid; e < P.cout * P.cin; e += C1_THREADS_DW) dst[e] = 0.f;       // this block still owns its slice
    }
    if (failed) {
        *abort_flag = 1;
        if (P.error_flag) *P.error_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == DW_MMA) tmem_dealloc(tmem_d, tmem_cols);
}

// ---- both gradients in one pass ----------------------------------------------------------------------------
// grad_in[i][p] = sum_o w[slot][o][i] * gout[o][p] and gw[slot][o][i] = sum_p gout[o][p] * in[i][p], and the sums of gout over the locations (the gradient of a
// bias), from one reading of gout and in.  The three passes apart read gout three times and round it twice: 64 -> 128 channels on 3.5 M locations 0.69 + 0.51 + 0.32 ms,
// 0.81 together (0.56 at the rate of a copy).
// One persistent block per SM, 25 warps, over tiles of 128 locations, the weights of one level in shared memory:
//   warps 0-15  producers in groups of 2, 4 or 8 warps (8 channel rows a warp, so that narrow layers have as much under way), which take the tiles in turn.  A warp reads
//               whole rows, 128 locations of a channel, rounds them to bf16 and leaves, as conv111_tc_dw_kernel does, rows of channels whose locations lie in two
//               swizzled halves: K-major operands of the weight gradient, and as MN-major operand that of the input gradient, so that one rounding and one
//               write to shared memory serve both.  (A thread that owns a location and reads 32 of its channels, as in conv111_tc_kernel, has its warp fetch 128
//               bytes of 32 rows, whose lines, at any multiple of four bytes, its neighbours fetch again: the pass took 1.03 ms; row pieces by bulk copies, which are
//               issued one after the other, 1.5.)  The sums of gout add the fp32 values before they are rounded, those of a tile by halving in fp32, the tiles in
//               double precision, each by an addition in L2 that nobody waits for (fp32 chains lost up to 1e-6 of a sum on 2.1 M locations and more with the volume; doubles in shared
//               memory, 1 KB more, cost 64 -> 128 and 128 -> 128 channels 12 %: beyond 196 KB an SM's L1 shrinks);
//   warp 16     one thread issues the tcgen05.mma of a tile: cout / 16 for the input gradient, 8 for every 128 rows of the weight gradient, whose accumulators
//               (mtiles x nt columns) stay in TMEM over all tiles of a level range, next to those of the input gradient, two or four tiles in flight;
//   warps 17-24 epilogue as in conv111_tc_kernel, and the weight sums at the end of a level range.
struct C1JointParams {
    int n_segs;
    ll seg_begin[C1_MAX_SEGS], seg_end[C1_MAX_SEGS];
    int seg_slot[C1_MAX_SEGS];
    const float* in; ll ld_in; int cin;
    const float* gout; ll ld_out; int cout;
    const float* w;                                // [slot][cout][cin]
    float* gin; ll ld_gin;
    float* partial;                                // [segment][block][cout][cin]
    double* sums;                                  // [block][group][cout] (null: not wanted)
    int stages, nt, mtiles, nacc;                  // ring; cin padded; 128-row accumulators of the weight gradient; accumulators of the input gradient
    uint32_t idesc_x, idesc_w;
    int* error_flag;
};

constexpr int C1J_PROD = 16, C1J_MMA = C1J_PROD, C1J_EPI = C1J_PROD + 1, C1J_THREADS = (C1J_EPI + 8) * 32;

template<int WPG>
__global__ void __launch_bounds__(C1J_THREADS, 1) conv111_tc_joint_kernel(const __grid_constant__ C1JointParams P) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int nt = P.nt, nacc = P.nacc, stages = P.stages;
    const int kpad = (P.cout + 15) / 16 * 16, half_bytes = (kpad + nt) * 128, stage_bytes = 2 * half_bytes;
    unsigned char* b_s = smem + (size_t) stages * stage_bytes;                      // [kpad / 8][nt][8] bf16
    float* out_s = reinterpret_cast<float*>(b_s + (size_t) nt * kpad * 2);          // [2][C1_OUT_CH][256]
    constexpr int groups = C1J_PROD / WPG;
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_s + C1_OUT_BYTES / 4);
    uint64_t* full = bars;                              // [stages] operands written (the warps of a group)
    uint64_t* empty = bars + C1_MAX_STAGES;             // [stages] MMAs that read the stage completed
    uint64_t* tmem_full = empty + C1_MAX_STAGES;        // [nacc]   accumulator of the input gradient complete
    uint64_t* tmem_empty = tmem_full + C1_MAX_ACC;      // [nacc]   read back (4 epilogue warps)
    uint64_t* done = tmem_empty + C1_MAX_ACC;           //          all MMAs of the level range completed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = warp_number(), lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < stages; ++i) { mbar_init(smem_u32(full + i), WPG); mbar_init(smem_u32(empty + i), 1); }
        for (int i = 0; i < nacc; ++i) { mbar_init(smem_u32(tmem_full + i), 1); mbar_init(smem_u32(tmem_empty + i), 4); }
        mbar_init(smem_u32(done), 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    // the rows that pad the contraction are zeros that nobody writes again
    const int pad_rows = kpad - P.cout;
    for (int e = tid; e < stages * 2 * pad_rows * 8; e += C1J_THREADS)
        *reinterpret_cast<uint4*>(smem + (e / (pad_rows * 8)) * half_bytes + P.cout * 128 + e % (pad_rows * 8) * 16) = make_uint4(0, 0, 0, 0);
    // sums of gout: an entry belongs to one lane of the group, which sets it to zero and adds each tile of the group in turn
    if (P.sums && warp < C1J_PROD && lane < 8)
        for (int r = warp % WPG + lane * WPG; r < P.cout; r += 8 * WPG) P.sums[((ll) blockIdx.x * groups + warp / WPG) * P.cout + r] = 0.0;
    if (warp == C1J_MMA) { tmem_alloc(smem_u32(tmem_slot), 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_w = *tmem_slot, tmem_x = tmem_w + P.mtiles * nt;
    bool failed = false;
    int piece = 0;
    const int w8 = warp - C1J_EPI, set = w8 >> 2;
    uint32_t j_base = 0;                                // tiles of the level ranges before
    uint32_t done_phase = 0;

    for (int seg = 0; seg < P.n_segs; ++seg) {
        const ll sb = P.seg_begin[seg], se = P.seg_end[seg];
        const int seg_tiles = (int) ((se - sb + TILE_M - 1) / TILE_M);
        const int pair = seg_tiles > (int) gridDim.x ? 1 : 0;
        const int seg_units = (seg_tiles + pair) >> pair;
        const int units = (int) blockIdx.x < seg_units ? (seg_units - (int) blockIdx.x + (int) gridDim.x - 1) / (int) gridDim.x : 0;
        const int mine = (units << pair) - (units > 0 && (seg_tiles & pair) && (seg_units - 1) % (int) gridDim.x == (int) blockIdx.x ? 1 : 0);
        auto tile_begin = [&](int it) { return sb + ((((ll) blockIdx.x + (ll) (it >> pair) * gridDim.x) << pair) + (it & pair)) * TILE_M; };
        // ---- the level's weights -> B operand (every accumulator of the previous level range has been read back) ----
        tc_fence_before();
        __syncthreads();
        {
            const float* wslot = P.w + (ll) P.seg_slot[seg] * P.cout * P.cin;
            for (int e = tid; e < nt * kpad / 8; e += C1J_THREADS) {
                const int n = e % nt, k8 = e / nt;
                float v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int k = k8 * 8 + q;
                    v[q] = (n < P.cin && k < P.cout) ? __ldg(wslot + (ll) k * P.cin + n) : 0.f;
                }
                uint4 pk;
                pk.x = pack_bf16x2(v[0], v[1]); pk.y = pack_bf16x2(v[2], v[3]); pk.z = pack_bf16x2(v[4], v[5]); pk.w = pack_bf16x2(v[6], v[7]);
                *reinterpret_cast<uint4*>(b_s + ((size_t) k8 * nt + n) * 16) = pk;
            }
            fence_proxy_async();
        }
        __syncthreads();
        tc_fence_after();

        if (warp < C1J_PROD) {
            // ---------------- producers ----------------
            const int grp = warp / WPG, sub = warp % WPG, used = min(groups, stages);      // (a ring at least as long as the groups keeps the phases that a wait can meet apart)
            const int nrows = P.cout + P.cin;      // channel rows of a tile
            for (int it = grp; grp < used && it < mine && !failed; it += used) {
                const uint32_t j = j_base + (uint32_t) it, slot = j % (uint32_t) stages, use = j / (uint32_t) stages;
                const ll p0 = tile_begin(it);
                if (use > 0 && !mbar_wait_warp(smem_u32(empty + slot), (use - 1) & 1, abort_flag)) { failed = true; break; }
                unsigned char* st = smem + (size_t) slot * stage_bytes;
                const bool whole = p0 + TILE_M <= se;
                for (int r0 = sub; r0 < nrows; r0 += 8 * WPG) {      // 8 rows of this warp x 4 quarters of 32 locations in flight
                    float v[8][4];
                    auto source = [&](int r) { return (r < P.cout ? P.gout + (ll) r * P.ld_out : P.in + (ll) (r - P.cout) * P.ld_in) + p0 + lane; };
                    if (whole) {                                     // no condition per load: a branch each costs more than the loads
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            const float* src = source(min(r0 + u * WPG, nrows - 1));      // (the rows that repeat are not stored)
#pragma unroll
                            for (int q = 0; q < 4; ++q) v[u][q] = src[q * 32];
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            const float* src = source(min(r0 + u * WPG, nrows - 1));
#pragma unroll
                            for (int q = 0; q < 4; ++q) v[u][q] = p0 + q * 32 + lane < se ? src[q * 32] : 0.f;       // locations past the end are zeros
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const int r = r0 + u * WPG;
                        if (r >= nrows) break;
                        const int orow = r < P.cout ? r : kpad + (r - P.cout);
                        unsigned char* dst = st + (size_t) orow * 128 + ((lane & 7) << 1);
#pragma unroll
                        for (int q = 0; q < 4; ++q)                  // location 32 q + lane: half q >> 1, 16-byte piece 4 (q & 1) + lane / 8, swizzled
                            *reinterpret_cast<__nv_bfloat16*>(dst + (q >> 1) * half_bytes + (((((q & 1) << 2) + (lane >> 3)) ^ (orow & 7)) << 4)) = __float2bfloat16(v[u][q]);
                    }
                    if (P.sums && r0 < P.cout) {                     // the fp32 values, before they are rounded: 8 rows in 9 shuffles
                        float s[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) s[u] = (v[u][0] + v[u][1]) + (v[u][2] + v[u][3]);       // (of rows that repeat or are not of gout, not used)
#pragma unroll
                        for (int h = 4; h > 0; h >>= 1)              // lane l keeps the rows whose bit h is that of l
#pragma unroll
                            for (int u = 0; u < h; ++u) { const float x = s[u], y = s[u + h]; s[u] = ((lane & h) ? y : x) + __shfl_xor_sync(0xffffffffu, (lane & h) ? x : y, h); }
                        s[0] += __shfl_xor_sync(0xffffffffu, s[0], 8);
                        s[0] += __shfl_xor_sync(0xffffffffu, s[0], 16);
                        const int r = r0 + lane * WPG;
                        if (lane < 8 && r < P.cout) atomicAdd(P.sums + ((ll) blockIdx.x * groups + grp) * P.cout + r, (double) s[0]);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(full + slot));   // the MMA thread fences the generic-proxy writes after its wait
            }
        } else if (warp == C1J_MMA) {
            // ---------------- MMA issue ----------------
            if (elect_one()) {
                const uint64_t dw0 = make_desc(smem_u32(b_s), nt * 16, 128, 0);
                const int ksteps = kpad / 16;
                for (int it = 0; it < mine && !failed; ++it) {
                    const uint32_t j = j_base + (uint32_t) it, slot = j % (uint32_t) stages, use = j / (uint32_t) stages;
                    const uint32_t acc = j % (uint32_t) nacc, acc_use = j / (uint32_t) nacc;
                    if (acc_use > 0 && !mbar_wait(smem_u32(tmem_empty + acc), (acc_use - 1) & 1, abort_flag)) { failed = true; break; }
                    if (!mbar_wait(smem_u32(full + slot), use & 1, abort_flag)) { failed = true; break; }
                    fence_proxy_async();          // generic-proxy writes of the producers -> tensor-core (async proxy) reads
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + (size_t) slot * stage_bytes);
                    const uint64_t da0 = make_desc(a_addr, half_bytes, 1024, 2);                 // 128 locations = two halves, 16 channels = 16 rows
                    for (int k = 0; k < ksteps; ++k)
                        umma_bf16(tmem_x + acc * nt, da0 + (uint64_t) ((k * 2048) >> 4), dw0 + (uint64_t) ((k * 2 * nt * 16) >> 4), P.idesc_x, k > 0 ? 1u : 0u);
                    umma_commit(smem_u32(tmem_full + acc));
                    for (int half = 0; half < 2; ++half) {
                        const uint32_t hb = a_addr + half * half_bytes;
                        const uint64_t db = make_desc(hb + kpad * 128, 16, 1024, 2);
                        for (int mt = 0; mt < P.mtiles; ++mt) {
                            // (128 rows: behind those of gout lies what follows them in shared memory, and results that nobody reads)
                            const uint64_t da = make_desc(hb + mt * 128 * 128, 16, 1024, 2);
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                umma_bf16(tmem_w + mt * nt, da + (uint64_t) ((k * 32) >> 4), db + (uint64_t) ((k * 32) >> 4), P.idesc_w, (it > 0 || half > 0 || k > 0) ? 1u : 0u);
                        }
                    }
                    umma_commit(smem_u32(empty + slot));
                }
                if (!failed && mine > 0) umma_commit(smem_u32(done));
            }
        } else {
            // ---------------- epilogue ----------------
            for (int u = 0; u < units; ++u) {
                const int it = (u << pair) + set;
                const uint32_t j = j_base + (uint32_t) it, acc = j % (uint32_t) nacc;
                store_unit(P.gin, P.ld_gin, P.cin, nullptr, tile_begin(u << pair), (int) min(se - tile_begin(u << pair), (ll) (TILE_M << pair)), set <= pair && it < mine,
                           tmem_x + acc * nt, smem_u32(tmem_full + acc), (j / (uint32_t) nacc) & 1, smem_u32(tmem_empty + acc), out_s, w8, piece, failed, abort_flag);
            }
            // weight sums of the level range: set 0 the even, set 1 the odd pieces of 16 columns
            float* dst = P.partial + ((ll) seg * gridDim.x + blockIdx.x) * P.cout * P.cin;
            if (mine == 0) {
                for (int e = tid - C1J_EPI * 32; e < P.cout * P.cin; e += 256) dst[e] = 0.f;     // this block still owns its slice
            } else if (!failed && mbar_wait_warp(smem_u32(done), done_phase & 1, abort_flag)) {
                tc_fence_after();
                const int q = warp & 3;
#pragma unroll 1
                for (int mt = 0; mt < P.mtiles; ++mt) {
                    const int o = mt * 128 + q * 32 + lane;
#pragma unroll 1
                    for (int c0 = set * 16; c0 < P.cin; c0 += 32) {
                        uint32_t r[16];
                        tmem_ld16(tmem_w + ((uint32_t) (q * 32) << 16) + mt * nt + c0, r);
                        tmem_ld_wait();
                        if (o < P.cout) {
#pragma unroll
                            for (int jj = 0; jj < 16; ++jj)
                                if (c0 + jj < P.cin) dst[(ll) o * P.cin + c0 + jj] = __uint_as_float(r[jj]);
                        }
                    }
                }
            } else failed = true;
        }
        if (mine > 0) ++done_phase;
        if (failed) *abort_flag = 1;
        j_base += (uint32_t) mine;
    }

    if (failed) {
        *abort_flag = 1;
        if (P.error_flag) *P.error_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == C1J_MMA) tmem_dealloc(tmem_w, 512);
}

// dst[slot of segment y][e] += the blocks' partial sums; the last y (bias): dst_bias[e] = the `nbias` sums of the bias.  A block has 32 entries, warp w adds
// every eighth of the sums (in T); the warps' sums are added in order.
struct C1Reduce { int n_segs; int slot[C1_MAX_SEGS]; };
template<typename T>
__device__ __forceinline__ T c1_sums(const T* __restrict__ from, int count, int n, int e) {      // valid in warp 0
    __shared__ T sums[8][32];
    const int lane = threadIdx.x & 31, wrp = threadIdx.x >> 5;
    T s = 0;
    if (e < n)
#pragma unroll 4
        for (int b = wrp; b < count; b += 8) s += from[(ll) b * n + e];
    sums[wrp][lane] = s;
    __syncthreads();
    if (wrp == 0) for (int k = 1; k < 8; ++k) s += sums[k][lane];
    return s;
}
__global__ void __launch_bounds__(256) c1_reduce_kernel(const float* __restrict__ partial, const double* __restrict__ bias_partial, C1Reduce R, int nblocks, int nbias, int elems, int cout,
                                                        float* __restrict__ gw, float* __restrict__ gbias) {
    const int e = blockIdx.x * 32 + (threadIdx.x & 31), seg = blockIdx.y;
    const bool bias = seg == R.n_segs;
    const int n = bias ? cout : elems;
    if ((int) blockIdx.x * 32 >= n) return;
    const bool writes = threadIdx.x < 32 && e < n;
    if (bias) {
        const double s = c1_sums(bias_partial, nbias, n, e);
        if (writes) gbias[e] = (float) s;
    } else {
        const float s = c1_sums(partial + (ll) seg * nblocks * elems, nblocks, n, e);
        if (writes) gw[(ll) R.slot[seg] * elems + e] += s;
    }
}

template<int WPG>
int launch_c1_joint(const C1JointParams& P, int grid, size_t smem, cudaStream_t st) {
    auto kern = conv111_tc_joint_kernel<WPG>;
    APRNET_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    AprnetProfScope _prof("conv111_tc_dw:joint", st);
    kern<<<grid, C1J_THREADS, smem, st>>>(P);
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

template<int NT>
int launch_c1_dw(const C1DwParams& P, int grid, int mtiles, cudaStream_t st) {
    const size_t stage = (size_t) (mtiles * 128 + NT) * 256;
    const size_t fixed = (2 * C1_MAX_STAGES + 1) * 8 + 16 + 1024;
    if (fixed + 2 * stage > 227 * 1024 - 1024) return APRNET_ERR_UNSUPPORTED;
    const int stages = (int) std::min<size_t>(C1_MAX_STAGES, (227 * 1024 - 1024 - fixed) / stage);
    const size_t smem = (size_t) stages * stage + fixed;
    auto kern = conv111_tc_dw_kernel<NT>;
    APRNET_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    kern<<<grid, C1_THREADS_DW, smem, st>>>(P, stages, mtiles);
    return APRNET_OK;
}

} // namespace

extern "C" int aprnet_conv111_forward_tc_bias(const aprnet_apr* a, int dl, int cin, int cout, int S, const float* in, int64_t ld_in,
                                              const float* w, const float* bias, float* out, int64_t ld_out, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && in && w && out && cin > 0 && cout > 0 && S > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl), "leading dimension too small");
    char pname[64];
    snprintf(pname, sizeof(pname), "conv111_tc:ci%d:co%d:dl%d", cin, cout, dl);
    return run_conv111_tc(a, dl, cin, cout, S, in, ld_in, w, (ll) cin * cout, cin, 1, bias, out, ld_out, (cudaStream_t) stream, pname);
}

extern "C" int aprnet_conv111_forward_tc(const aprnet_apr* a, int dl, int cin, int cout, int S, const float* in, int64_t ld_in,
                                         const float* w, float* out, int64_t ld_out, void* stream) {
    return aprnet_conv111_forward_tc_bias(a, dl, cin, cout, S, in, ld_in, w, nullptr, out, ld_out, stream);
}

extern "C" int aprnet_conv111_backward_input_tc(const aprnet_apr* a, int dl, int cin, int cout, int S, const float* gout, int64_t ld_out,
                                                const float* w, float* gin, int64_t ld_in, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && gout && w && gin && cin > 0 && cout > 0 && S > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl), "leading dimension too small");
    char pname[64];
    snprintf(pname, sizeof(pname), "conv111_tc:ci%d:co%d:dl%d", cout, cin, dl);
    return run_conv111_tc(a, dl, cout, cin, S, gout, ld_out, w, (ll) cin * cout, 1, cin, nullptr, gin, ld_in, (cudaStream_t) stream, pname);
}

extern "C" int aprnet_conv111_backward_weights_tc(const aprnet_apr* a, int dl, int cin, int cout, int S, const float* in, int64_t ld_in,
                                                  const float* gout, int64_t ld_out, float* gw, float* partial, int64_t partial_elems,
                                                  void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && in && gout && gw && partial && cin > 0 && cout > 0 && S > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld_in >= a->number_parts(dl) && ld_out >= a->number_parts(dl), "leading dimension too small");
    if (cin > 256 || cout > 256) return APRNET_ERR_UNSUPPORTED;      // (narrow layers included: the padding costs no memory traffic)
    cudaStream_t st = (cudaStream_t) stream;
    const ll elems = (ll) cin * cout;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int max_blocks = (int) std::min<ll>(sms, partial_elems / elems);
    if (max_blocks < 1) return APRNET_ERR_UNSUPPORTED;
    const int nt = pick_nt(cin), mtiles = (cout + 127) / 128;
    if (mtiles * nt > 512) return APRNET_ERR_UNSUPPORTED;
    for (const Segment& sg : aprnet_segments(a, dl, S, true)) {
        if (sg.end <= sg.begin) continue;
        C1DwParams P;
        P.seg_begin = sg.begin; P.seg_end = sg.end; P.in = in; P.ld_in = ld_in; P.cin = cin; P.gout = gout; P.ld_out = ld_out; P.cout = cout;
        P.partial = partial; P.error_flag = aprnet_tc_error_flag_device();
        const int grid = (int) std::min<ll>(max_blocks, (sg.end - sg.begin + TILE_M - 1) / TILE_M);
        int rc = APRNET_ERR_UNSUPPORTED;
        { AprnetProfScope _prof("conv111_tc_dw", st);
        switch (nt) {
            case 16: rc = launch_c1_dw<16>(P, grid, mtiles, st); break;
            case 32: rc = launch_c1_dw<32>(P, grid, mtiles, st); break;
            case 64: rc = launch_c1_dw<64>(P, grid, mtiles, st); break;
            case 128: rc = launch_c1_dw<128>(P, grid, mtiles, st); break;
            case 256: rc = launch_c1_dw<256>(P, grid, mtiles, st); break;
        }
        }
        if (rc) return rc;
        { AprnetProfScope _prof("conv111_dw_reduce", st);
        C1Reduce R;
        R.n_segs = 1; R.slot[0] = sg.slot;
        c1_reduce_kernel<<<(unsigned) aprnet_ceil_div(elems, 32), 256, 0, st>>>(partial, nullptr, R, grid, 0, (int) elems, cout, gw, nullptr);
        }
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

// All gradients of a layer in one pass: grad_input (written), grad_weights (accumulated into) and, where grad_bias is not null, the sums of grad_output over the
// structure's locations (written).  APRNET_ERR_UNSUPPORTED where a channel count is below 8 or above 256, cin above 4 cout, the operands of two tiles do not fit shared memory or the
// accumulators TMEM: the passes apart then.
extern "C" int aprnet_conv111_backward_tc(const aprnet_apr* a, int dl, int cin, int cout, int S, const float* in, int64_t ld_in, const float* gout, int64_t ld_out,
                                          const float* w, float* gin, int64_t ld_gin, float* gw, float* gbias, float* partial, int64_t partial_elems, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && in && gout && w && gin && gw && partial && cin > 0 && cout > 0 && S > 0, "bad argument");
    APRNET_DEVICE_CHECK(a);
    const ll n = a->number_parts(dl), elems = (ll) cin * cout;
    APRNET_ARG_CHECK(ld_in >= n && ld_out >= n && ld_gin >= n, "leading dimension too small");
    if (cin < 8 || cout < 8 || cin > 256 || cout > 256) return APRNET_ERR_UNSUPPORTED;
    // what is saved is reading gout twice more: 16 -> 16 channels 0.21 ms instead of 0.33, 64 -> 32 0.59 instead of 0.67, but 128 -> 8 0.97 instead of 0.94
    if (4 * cout < cin) return APRNET_ERR_UNSUPPORTED;
    C1JointParams P;
    C1Reduce R;
    ll tiles = 0;
    P.n_segs = 0;
    for (const Segment& sg : aprnet_segments(a, dl, S, true)) {
        if (P.n_segs >= C1_MAX_SEGS) return APRNET_ERR_UNSUPPORTED;
        P.seg_begin[P.n_segs] = sg.begin; P.seg_end[P.n_segs] = sg.end; P.seg_slot[P.n_segs] = R.slot[P.n_segs] = sg.slot;
        tiles = std::max<ll>(tiles, (sg.end - sg.begin + TILE_M - 1) / TILE_M);
        ++P.n_segs;
    }
    if (P.n_segs == 0) return APRNET_ERR_UNSUPPORTED;
    R.n_segs = P.n_segs;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int wpg = cin + cout <= 16 ? 2 : (cin + cout <= 32 ? 4 : 8), groups = C1J_PROD / wpg;
    // (behind the partial weight gradients the sums of gout, doubles at a multiple of eight bytes)
    const int blocks = (int) std::min<ll>(tiles, sms), grid = (int) std::min<ll>(blocks, (partial_elems - 1) / (P.n_segs * elems + (gbias ? 2 * groups * cout : 0)));
    if (grid < 1 || grid < blocks / 2) return APRNET_ERR_UNSUPPORTED;            // too little workspace
    P.in = in; P.ld_in = ld_in; P.cin = cin; P.gout = gout; P.ld_out = ld_out; P.cout = cout; P.w = w; P.gin = gin; P.ld_gin = ld_gin;
    P.partial = partial; P.sums = gbias ? reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(partial + (ll) grid * P.n_segs * elems) + 7) & ~(uintptr_t) 7) : nullptr;
    P.nt = pick_nt(cin); P.mtiles = (cout + 127) / 128; P.nacc = P.nt <= 64 ? 4 : 2;
    P.idesc_x = make_idesc(P.nt, true, false); P.idesc_w = make_idesc(P.nt, false, false);
    P.error_flag = aprnet_tc_error_flag_device();
    const int kpad = (cout + 15) / 16 * 16;
    const size_t stage = (size_t) (kpad + P.nt) * 256, smem_max = 227 * 1024;
    const size_t fixed = (size_t) P.nt * kpad * 2 + C1_OUT_BYTES + (2 * C1_MAX_STAGES + 2 * C1_MAX_ACC + 1) * 8 + 16 + 1024;
    if ((P.mtiles + P.nacc) * P.nt > 512 || fixed + 2 * stage > smem_max) return APRNET_ERR_UNSUPPORTED;
    P.stages = (int) std::min<size_t>(C1_MAX_STAGES, (smem_max - fixed) / stage);
    const size_t smem = P.stages * stage + fixed;
    cudaStream_t st = (cudaStream_t) stream;
    const int rc = wpg == 2 ? launch_c1_joint<2>(P, grid, smem, st) : (wpg == 4 ? launch_c1_joint<4>(P, grid, smem, st) : launch_c1_joint<8>(P, grid, smem, st));
    if (rc) return rc;
    { AprnetProfScope _prof("conv111_dw_reduce", st);
    c1_reduce_kernel<<<dim3((unsigned) aprnet_ceil_div(std::max<ll>(elems, gbias ? cout : 0), 32), (unsigned) (P.n_segs + (gbias ? 1 : 0))), 256, 0, st>>>(
        partial, P.sums, R, grid, grid * groups, (int) elems, cout, gw, gbias);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}
