// 3x3x3 particle convolution in exact fp32 on the CUDA cores, as tiled matrix products over gathered rows.
//
// Same formulation as the tensor-core path (conv333_tc.cu): the features are repacked channels-last, so that the
// neighbour of a location is one contiguous row; a tile of output locations is a matrix product
//     D[locations][Cout] += X[nbr(tap, location)][Cin] * W[tap][Cin][Cout]          over the 27 taps,
// the same-level input gradient is the same product over the rows of grad_output with mirrored, transposed weights, the
// cross-level part gathers per-(target, tap) sums of those rows over the edge plan, and the weight gradient contracts over
// the locations.  Multiply-adds are fp32 throughout.
//
// What bounds it: the fp32 pipe (128 multiply-adds per clock and SM, 72 TFLOP/s measured) and, next to it, the shared-memory
// pipe: a 16-byte read of a warp takes one pass per eight lanes unless all 32 lanes read the same address.  So the 32 lanes
// of a warp lie along the gathered dimension (32 different rows per read: every pass carries 128 useful bytes) and share
// their TN columns of the other operand (one pass per read); a thread's 4 x TN results take 16 + TN passes per 16 * TN
// multiply-adds of the warp.  With an 8 x 4 arrangement of the lanes and 8 x 8 results per thread (48 passes instead of 32 per
// 256 multiply-adds) the kernels stayed at 45 to 49 TFLOP/s, both pipes at about 65 %.  The gathered rows come in by asynchronous
// 16-byte copies several stages ahead.
// Arithmetic: pyapr/aprnet/src/conv.hpp:83-195,289-481 and helpers.hpp:358-478,505-704.
#include "apr_device.cuh"
#include "tc_ptx.cuh"
#include <algorithm>
#include <cstring>

namespace {

using tcptx::smem_u32;
using tcptx::cp_async16;
using tcptx::cp_async_commit;
using tcptx::cp_async_wait;
typedef long long ll;
constexpr int MAX_SEGS = APRNET_MAX_LEVELS;
constexpr int KS = 16;                   // channels (gather) or locations (weight gradient) per ring slot

struct SegTable {
    int n;
    ll begin[MAX_SEGS], end[MAX_SEGS];
    int slot[MAX_SEGS];
    int tile_begin[MAX_SEGS + 1];
};

inline SegTable make_seg_table(const std::vector<Segment>& segs, int tile) {
    SegTable t;
    t.n = (int) segs.size();
    t.tile_begin[0] = 0;
    for (int i = 0; i < t.n; ++i) {
        t.begin[i] = segs[i].begin; t.end[i] = segs[i].end; t.slot[i] = segs[i].slot;
        t.tile_begin[i + 1] = t.tile_begin[i] + aprnet_ceil_div(segs[i].end - segs[i].begin, tile);
    }
    return t;
}

// 16-byte asynchronous copy, or 16 zero bytes when `valid` is false (nothing is read then)
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// two multiply-adds in one instruction: acc.{x,y} += a * b.{x,y}.  A single FFMA reads three registers for one product, and with
// the 8 x 8 register tile its operand reads held the scheduler back (0.75 instructions per cycle issued, 62 % of the fp32 pipe);
// the paired form issues and reads half as often.
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ void add2(unsigned long long& acc, unsigned long long a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(a)); }
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// ---- operand packing --------------------------------------------------------------------------------
// rows [0, n): x[:, p], with PAIR from channel `split` on x1[:, p] (a kernel of its own: the choice cost one tensor's packing 12 %); rows [n, n + t): tree[:, p - n]; row n + t: zeros.  Channels padded with zeros to cpad (multiple of 4).
template<bool PAIR>
__global__ void __launch_bounds__(256) pack_rows_f32_kernel(const float* __restrict__ x, ll ld_x, int split, const float* __restrict__ x1, ll ld_x1, ll n, const float* __restrict__ tree, ll ld_tree, ll t,
                                                            int c, int cpad, float* __restrict__ out) {
    // tile: 32 channels x 64 rows, read along the particle axis, written as 16-byte pieces of the rows
    __shared__ float tile[32][65];
    const ll r0 = (ll) blockIdx.x * 64;
    const int c0 = blockIdx.y * 32;
    const ll rows = n + t + 1;
    const int lane = threadIdx.x & 31, wrp = threadIdx.x >> 5;
    float v[4][2];
#pragma unroll
    for (int cc = 0; cc < 4; ++cc)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int ch = c0 + wrp + 8 * cc;
            const ll r = r0 + lane + 32 * k;
            const float* from = PAIR && ch >= split ? x1 + (ll) (ch - split) * ld_x1 : x + (ll) ch * ld_x;
            v[cc][k] = (ch < c && r < n + t) ? (r < n ? from[r] : tree[(ll) ch * ld_tree + (r - n)]) : 0.f;
        }
#pragma unroll
    for (int cc = 0; cc < 4; ++cc)
#pragma unroll
        for (int k = 0; k < 2; ++k) tile[wrp + 8 * cc][lane + 32 * k] = v[cc][k];
    __syncthreads();
    const int pieces = min(8, (cpad - c0) / 4);
    for (int e = threadIdx.x; e < 64 * pieces; e += 256) {
        const int rr = e / pieces, piece = e - rr * pieces;
        const ll r = r0 + rr;
        if (r < rows)
            *reinterpret_cast<float4*>(out + r * cpad + c0 + piece * 4) =
                make_float4(tile[piece * 4][rr], tile[piece * 4 + 1][rr], tile[piece * 4 + 2][rr], tile[piece * 4 + 3][rr]);
    }
}

// ---- gather product ---------------------------------------------------------------------------------
struct F32Params {
    SegTable segs;
    const int32_t* nbr; ll N;              // neighbour table [27][N]
    const float* rows; int kpad;           // packed source rows [R][kpad]
    ll tree_base, zero_row;                // row of tree node 0 and of the zero row
    const float* wp; int mirror;           // packed weights (weights.cu); mirror: tap t meets the weights of tap 26 - t
    int n_dim, n_tiles;
    int same_level_only;                   // mask table entries outside the tile's own level (as a constant of the mode: 16 -> 16 3.5 % slower)
    float* out; ll ld_out;
    const float* bias;                     // added to every output channel (null: none)
    // target mode (cross-level input gradient): location a stands for target out_map[a]; the result is added to
    // out[:, t] for t < out_split and to out2[:, t - out_split] otherwise
    const int32_t* out_map; ll out_split;
    float* out2; ll ld_out2;
    ll v_shift;                            // added to table entries >= 0 (virtual rows)
};

enum { FORWARD, SAME_LEVEL, TARGETS };        // forward pass, the two parts of the input gradient

// Block = 32 * R * WM locations x NT = TN * WN output channels, WM x WN warps; a thread owns the locations lane + 32 i (i < R) of its
// warp's 32 R and TN channels.  R = 4 where the blocks fill the chip; few blocks are a serial chain of slots each, and with R = 1 a slot takes a quarter of the
// multiply-adds and four times the blocks share the work: gathers of 64-wide tiles in a training step on 9.7 k locations 7.3 -> 4.2 ms.  Each result is the same chain.  A ring slot holds 16 channels of the tile's rows for one tap and the matching weights; 16-byte
// pieces of a row are exchanged so that eight consecutive rows read at the same channel fall on different banks.  Table
// entries are requested one tap ahead of the copies that need them.
//
// Order of the products.  Input gradient: taps outer, 16 channels of one tap per slot.  KMAJOR (forward pass): blocks of
// 8 channels outer, taps inner, a slot holds two consecutive (block, tap) pairs.  A result is then the same chain of
// multiply-adds whatever the tile (blocks of 8 channels, tap by tap, channel by channel): ReLU and max-pooling behind a
// convolution turn a difference in its last bit into another gate or another child, so the forward pass keeps one order.
//
// ZEROS: absent neighbours are zeros that are not read instead of the row of zeros in L1.  In the cross-level part, where most taps have none, that
// takes 4 to 25 % off (32 -> 32 on 1.2 M locations 522 -> 465 us, with the sums below), in the same-level part up to 7 % where the tile is at most 32 channels wide
// (32 -> 32 1805 -> 1753) and minus 3 to 10 % where it is 64 (33 -> 33 3220 -> 3333, 64 -> 64 at level delta 1 2595 -> 2663: the test costs more than
// the reads).  The forward pass has next to none (neighbours outside the volume).
// Threads per SM and ring slots.  16 warps of 128 registers instead of 12 of 168 give little, because the register file bounds the loop (paired multiply-adds read
// four registers a cycle): input gradient of 32 channels 4.94 -> 4.56 ms (32 -> 32, 3.5 M locations, three slots), forward pass of 64 9.01 -> 8.90 ms (64 -> 64 at level
// delta 1), weight gradient of 16 x 32 tiles 8.16 -> 7.98 (33 -> 24); the other shapes lose 1 to 14 %, and so do these where the blocks do not need the room (MANY: aprnet_f32_many_blocks).
template<int WM, int TN, int MODE> constexpr bool MORE_THREADS = TN == 16 && ((MODE == FORWARD && WM == 1) || (MODE == SAME_LEVEL && WM == 2));
template<int WM, int R, bool MANY> struct GatherShape {
    static constexpr int THREADS = R == 1 ? 768 : (MANY ? 512 : 384), RING = MANY && WM == 2 ? 3 : 4;
};
template<int WM, int WN, int TN, int R, int MODE, bool MANY>
__global__ void __launch_bounds__(32 * WM * WN, GatherShape<WM, R, MANY>::THREADS / (32 * WM * WN)) conv333_f32_gather_kernel(const F32Params P) {
    constexpr int RING = GatherShape<WM, R, MANY>::RING;
    constexpr int T = 32 * WM * WN, M = 32 * R * WM, NT = TN * WN;
    constexpr bool KMAJOR = MODE == FORWARD, ZEROS = MODE == TARGETS || (MODE == SAME_LEVEL && NT < 64);
    constexpr int RPT = M * (KS / 4) / T;          // row pieces a thread copies per slot
    constexpr int RSTEP = T / (KS / 4);            // distance of their rows
    constexpr int A_ELEMS = M * KS, B_ELEMS = KS * NT, SLOT = A_ELEMS + B_ELEMS;
    extern __shared__ __align__(16) float ring[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp % WM, wn = warp / WM;
    const int tile = blockIdx.x / P.n_tiles, nt = blockIdx.x - tile * P.n_tiles;
    int seg = 0;
    while (seg + 1 < P.segs.n && tile >= P.segs.tile_begin[seg + 1]) ++seg;
    const ll lo = P.segs.begin[seg], hi = P.segs.end[seg];
    const ll p0 = lo + (ll) (tile - P.segs.tile_begin[seg]) * M;
    const int kchunks = KMAJOR ? (P.kpad + 7) / 8 : (P.kpad + KS - 1) / KS;
    const int total = KMAJOR ? (27 * kchunks + 1) / 2 : 27 * kchunks;
    const float* wtile = P.wp + ((ll) P.segs.slot[seg] * 27 * P.n_tiles + nt) * ((ll) P.kpad * NT);
    const ll wtap = (ll) P.n_tiles * P.kpad * NT;

    // producer side of the thread
    const int piece = tid & (KS / 4 - 1), prow = tid / (KS / 4);
    int32_t raw[RPT], src[RPT];
    auto request = [&](int tap) {
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const ll p = p0 + prow + i * RSTEP;
            raw[i] = (tap < 27 && p < hi) ? __ldg(P.nbr + (ll) tap * P.N + p) : APRNET_NONE;
        }
    };
    auto decode = [&]() {
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int32_t v = raw[i];
            ll r = P.zero_row;
            if (P.same_level_only) { if (v >= lo && v < hi) r = v; }
            else if (v >= 0) r = v + P.v_shift;
            else if (v != APRNET_NONE) r = P.tree_base + aprnet_dec_tree(v);
            src[i] = (int32_t) r;
        }
    };
    auto copy_rows = [&](float* a_s, int k) {      // channels [k, k + 4) of the rows src[]; beyond the row: zeros
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int row = prow + i * RSTEP;
            cp_async16_zfill(smem_u32(a_s + row * KS + ((piece ^ ((row >> 1) & 3)) << 2)), P.rows + (ll) src[i] * P.kpad + k, k < P.kpad && (!ZEROS || src[i] != (int32_t) P.zero_row));
        }
    };
    int itap = KMAJOR ? piece >> 1 : 0, ikc = 0, islot = 0, is = 0;       // KMAJOR: the (block, tap) pair of this thread's half of a slot
    auto issue = [&]() {                           // next slot of the ring
        if (is >= total) return;
        float* a_s = ring + islot * SLOT;
        if (KMAJOR) {
            decode();
            copy_rows(a_s, ikc < kchunks ? ikc * 8 + (piece & 1) * 4 : P.kpad);
            for (int e = tid; e < KS * (NT / 4); e += T) {
                const int row = e / (NT / 4), pair = 2 * is + (row >> 3), kc = pair / 27, tap = pair - kc * 27, k = kc * 8 + (row & 7);
                cp_async16_zfill(smem_u32(a_s + A_ELEMS + e * 4), wtile + tap * wtap + (ll) k * NT + (e % (NT / 4)) * 4, k < P.kpad);
            }
            itap += 2;
            if (itap >= 27) { itap -= 27; ++ikc; }
            request(ikc < kchunks ? itap : 27);
        } else {
            if (ikc == 0) { decode(); request(itap + 1); }
            copy_rows(a_s, ikc * KS + piece * 4);
            const float* w = wtile + (P.mirror ? 26 - itap : itap) * wtap + (ll) ikc * KS * NT;
            const int wpieces = min(KS, P.kpad - ikc * KS) * (NT / 4);
            for (int e = tid; e < wpieces; e += T) cp_async16(smem_u32(a_s + A_ELEMS + e * 4), w + e * 4);
            if (++ikc == kchunks) { ikc = 0; ++itap; }
        }
        ++is;
        if (++islot == RING) islot = 0;
    };

    unsigned long long acc[R][TN / 2];             // pairs of output channels
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int n = 0; n < TN / 2; ++n) acc[i][n] = 0ull;

    request(itap);
#pragma unroll
    for (int s = 0; s < RING - 1; ++s) { issue(); cp_async_commit(); }
    const int sw = (lane >> 1) & 3, arow = (wm * 32 * R + lane) * KS, n_off = wn * TN;
    int slot = 0, kc = 0;
    for (int s = 0; s < total; ++s) {
        cp_async_wait<RING - 2>();
        __syncthreads();                           // slot s has landed for everybody, slot s - 1 has been read by everybody
        issue();
        cp_async_commit();
        const float* a_s = ring + slot * SLOT + arow;
        const float* b_s = ring + slot * SLOT + A_ELEMS + n_off;
        auto quad = [&](int q) {                   // four channels
            float4 a[R];
#pragma unroll
            for (int i = 0; i < R; ++i) a[i] = *reinterpret_cast<const float4*>(a_s + i * 32 * KS + ((q ^ sw) << 2));
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const float* bk = b_s + (q * 4 + kk) * NT;
                unsigned long long a2[R];
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    const float av = kk == 0 ? a[i].x : (kk == 1 ? a[i].y : (kk == 2 ? a[i].z : a[i].w));
                    a2[i] = pack2(av, av);
                }
#pragma unroll
                for (int h = 0; h < TN / 4; ++h) {
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bk + h * 4);
#pragma unroll
                    for (int i = 0; i < R; ++i) fma2(acc[i][2 * h], a2[i], b.x);
#pragma unroll
                    for (int i = 0; i < R; ++i) fma2(acc[i][2 * h + 1], a2[i], b.y);
                }
            }
        };
        const int quads = KMAJOR ? KS / 4 : (P.kpad - kc * KS) >> 2;
        if (quads >= KS / 4) {                     // straight-line code: the reads of a quad move ahead of the previous one's multiply-adds
#pragma unroll
            for (int q = 0; q < KS / 4; ++q) quad(q);
        } else {
            for (int q = 0; q < quads; ++q) quad(q);
        }
        if (++slot == RING) slot = 0;
        if (++kc == kchunks) kc = 0;
    }
    cp_async_wait<0>();

#pragma unroll
    for (int i = 0; i < R; ++i) {
        const ll p = p0 + wm * 32 * R + lane + i * 32;
        if (p >= hi) continue;
        float* dst = P.out + p;
        ll ld = P.ld_out;
        if (MODE == TARGETS) {
            const ll t = P.out_map[p];
            dst = t < P.out_split ? P.out + t : P.out2 + (t - P.out_split);
            ld = t < P.out_split ? P.ld_out : P.ld_out2;
            // adds to what is there (this thread is the only writer of its target in this launch): all of it is requested before any is
            // written, an addition after the other waited TN times for scattered accesses.  (In a kernel shared with the other parts this cost
            // their epilogues up to 9 %: 8 -> 33, forward, on 1.2 M locations 814 -> 875 us, now 805.)
            float held[TN];
#pragma unroll
            for (int n = 0; n < TN; ++n) held[n] = nt * NT + n_off + n < P.n_dim ? dst[(ll) (nt * NT + n_off + n) * ld] : 0.f;
#pragma unroll
            for (int n = 0; n < TN; ++n) {
                const int co = nt * NT + n_off + n;
                const float2 pair = unpack2(acc[i][n / 2]);
                if (co < P.n_dim) dst[(ll) co * ld] = (n & 1 ? pair.y : pair.x) + held[n];
            }
            continue;
        }
        auto store = [&](bool bias) {
#pragma unroll
            for (int n = 0; n < TN; ++n) {
                const int co = nt * NT + n_off + n;
                if (co >= P.n_dim) continue;
                const float2 pair = unpack2(acc[i][n / 2]);
                const float v = n & 1 ? pair.y : pair.x;
                dst[(ll) co * ld] = bias ? v + P.bias[co] : v;
            }
        };
        if (MODE == FORWARD && P.bias) store(true); else store(false);
    }
}

// per-(target, tap) sums of dO rows: virtual row v of [v0, v1) -> row v - v0.  A thread owns one
// row and four channels and requests up to four locations before it adds them in ascending order (runs are 2 to 4 long).
__global__ void __launch_bounds__(256) vrow_reduce_f32_kernel(const int32_t* __restrict__ vstart, const int32_t* __restrict__ vsrc, ll v0, ll v1,
                                                              const float* __restrict__ grows, int gpad, float* __restrict__ out) {
    const int nch = gpad >> 2;
    const ll e = (ll) blockIdx.x * blockDim.x + threadIdx.x;
    const ll v = v0 + e / nch;
    if (v >= v1) return;
    const int c = (int) (e % nch) * 4;
    const int b = __ldg(vstart + v), n = __ldg(vstart + v + 1) - b;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k0 = 0; k0 < n; k0 += 4) {
        float4 q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            q[k] = k0 + k < n ? __ldg(reinterpret_cast<const float4*>(grows + (ll) __ldg(vsrc + b + k0 + k) * gpad + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 4; ++k) { acc.x += q[k].x; acc.y += q[k].y; acc.z += q[k].z; acc.w += q[k].w; }
    }
    *reinterpret_cast<float4*>(out + (v - v0) * gpad + c) = acc;
}

// ---- weight gradient ----------------------------------------------------------------------------------
// dW[tap][ci][co] = sum over locations p of X[nbr(tap, p)][ci] * dO[p][co]: a product that contracts over the locations.
// Block = (range of one level, M = 128 * WM rows (tap, ci) = M / CIB taps x CIB channels, NT = TN * WN output channels); a
// ring slot holds 16 locations of both operands as they lie in memory (rows of channels), which is the order in which a
// thread's 4 x TN results want them.  The blocks of a level take its units of 64 locations in turn, so that blocks that run
// together gather from neighbouring rows.  Block sums go to a workspace and are added in a fixed order.
//
// A result of the block would be one chain of additions, and its rounding error grows with the chain.  So the chain starts again
// after seg_flush slots: narrow tiles (TN <= 8) keep the sum of the finished chains in registers; wide ones, whose accumulators take
// them, add it to the block's sum in the workspace (only one thread ever touches a sum, so its reductions are applied in program order:
// one order of summation).  Relative error against float64 on 2 M locations, one chain / chains: 16 -> 16 6.6e-7 / 2.3e-7, 33 -> 33
// 15e-7 / 8.1e-7, 128 -> 128 34e-7 / 8.6e-7; it costs 0 (16 -> 16) to 4 % (64 -> 64) of the kernel's time.
constexpr int DW_UNIT = 64;

struct F32DwParams {
    int n_segs;
    ll seg_begin[MAX_SEGS], seg_end[MAX_SEGS];
    int range_first[MAX_SEGS + 1];
    int seg_flush[MAX_SEGS];               // ring slots per chain of additions
    const int32_t* nbr; ll N;
    const float* xrows; int xpad; ll tree_base, zero_row;
    const float* grows; int gpad; ll g_zero_row;
    float* partial;                        // [range][27][cout][cin]
    int cin, cout, ci_blocks, groups;
};

template<int CIB, int WM, int TN> struct DwShape {
    static constexpr bool MORE = CIB == 16 && WM == 2 && TN == 16;
    static constexpr int THREADS = MORE ? 512 : 384, RING = MORE ? 3 : 4;
};
template<int CIB, int WM, int WN, int TN>
__global__ void __launch_bounds__(32 * WM * WN, DwShape<CIB, WM, TN>::THREADS / (32 * WM * WN)) conv333_f32_dw_kernel(const F32DwParams P) {
    constexpr int RING = DwShape<CIB, WM, TN>::RING;
    constexpr int T = 32 * WM * WN, M = 128 * WM, NT = TN * WN;
    constexpr int TS = M / CIB;                    // taps of a block
    constexpr int PC = CIB / 4;                    // 16-byte pieces of a gathered row
    constexpr int RPT = M * (KS / 4) / T;          // pieces a thread copies per slot
    constexpr int RSTEP = T / PC;
    constexpr int TAP_STRIDE = KS * CIB + (CIB < 32 ? CIB : 0);      // taps that one warp reads together start on different banks
    constexpr int A_ELEMS = TS * TAP_STRIDE, SLOT = A_ELEMS + KS * NT;
    extern __shared__ __align__(16) float ring[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp % WM, wn = warp / WM;
    const int grp = blockIdx.y % P.groups, cib = (blockIdx.y / P.groups) % P.ci_blocks, cob = blockIdx.y / (P.groups * P.ci_blocks);
    const int tap0 = grp * TS, c0 = cib * CIB, o0 = cob * NT;
    int seg = 0;
    while (seg + 1 < P.n_segs && (int) blockIdx.x >= P.range_first[seg + 1]) ++seg;
    const int rl = (int) blockIdx.x - P.range_first[seg], cnt = P.range_first[seg + 1] - P.range_first[seg];
    const ll sb = P.seg_begin[seg], se = P.seg_end[seg];
    const ll units = (se - sb + DW_UNIT - 1) / DW_UNIT;
    const int my_units = rl < units ? (int) ((units - rl + cnt - 1) / cnt) : 0;
    const int total = my_units * (DW_UNIT / KS);

    const int piece = tid % PC, prow = tid / PC;   // gathered row = (tap slot, location of the slot) = prow + i * RSTEP
    int32_t raw[RPT];
    auto location = [&](int s) { return sb + ((ll) rl + (ll) (s / (DW_UNIT / KS)) * cnt) * DW_UNIT + (s % (DW_UNIT / KS)) * KS; };
    auto request = [&](int s) {
        const ll pb = location(s);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int row = prow + i * RSTEP, tap = tap0 + row / KS;
            const ll p = pb + row % KS;
            raw[i] = (s < total && tap < 27 && p < se) ? __ldg(P.nbr + (ll) tap * P.N + p) : APRNET_NONE;
        }
    };
    int is = 0, islot = 0;
    auto issue = [&]() {
        if (is >= total) return;
        float* a_s = ring + islot * SLOT;
        const int c = c0 + piece * 4;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int row = prow + i * RSTEP;
            const int32_t v = raw[i];
            const ll r = v >= 0 ? (ll) v : (v == APRNET_NONE ? P.zero_row : P.tree_base + aprnet_dec_tree(v));
            cp_async16_zfill(smem_u32(a_s + (row / KS) * TAP_STRIDE + (row % KS) * CIB + piece * 4), P.xrows + r * P.xpad + c, c < P.xpad);
        }
        const ll pb = location(is);
        for (int e = tid; e < KS * (NT / 4); e += T) {
            const int k = e / (NT / 4), o = o0 + (e % (NT / 4)) * 4;
            const ll p = pb + k;
            cp_async16_zfill(smem_u32(a_s + A_ELEMS + e * 4), P.grows + (p < se ? p : P.g_zero_row) * P.gpad + o, o < P.gpad);
        }
        ++is;
        request(is);
        if (++islot == RING) islot = 0;
    };

    constexpr bool IN_REGISTERS = TN <= 8;
    unsigned long long acc[4][TN / 2], done[IN_REGISTERS ? 4 : 1][IN_REGISTERS ? TN / 2 : 1];
    if (IN_REGISTERS) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int n = 0; n < TN / 2; ++n) done[i][n] = 0ull;
    }

    request(0);
#pragma unroll
    for (int s = 0; s < RING - 1; ++s) { issue(); cp_async_commit(); }
    const int m0 = wm * 128 + lane * 4;            // this thread's rows: m0 .. m0 + 3
    const int a_off = (m0 / CIB) * TAP_STRIDE + m0 % CIB, n_off = wn * TN;
    int slot = 0, s = 0;
    do {
        const int s0 = s, s1 = min(total, s + P.seg_flush[seg]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int n = 0; n < TN / 2; ++n) acc[i][n] = 0ull;
        for (; s < s1; ++s) {
            cp_async_wait<RING - 2>();
            __syncthreads();
            issue();
            cp_async_commit();
            const float* a_s = ring + slot * SLOT;
            const float* b_s = a_s + A_ELEMS + n_off;
#pragma unroll
            for (int k = 0; k < KS; ++k) {
                const float4 a = *reinterpret_cast<const float4*>(a_s + a_off + k * CIB);
                const unsigned long long a2[4] = {pack2(a.x, a.x), pack2(a.y, a.y), pack2(a.z, a.z), pack2(a.w, a.w)};
#pragma unroll
                for (int h = 0; h < TN / 4; ++h) {
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(b_s + k * NT + h * 4);
#pragma unroll
                    for (int i = 0; i < 4; ++i) { fma2(acc[i][2 * h], a2[i], b.x); fma2(acc[i][2 * h + 1], a2[i], b.y); }
                }
            }
            if (++slot == RING) slot = 0;
        }
        if (IN_REGISTERS) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int n = 0; n < TN / 2; ++n) add2(done[i][n], acc[i][n]);
        }
        if (IN_REGISTERS && s < total) continue;
        // a thread's four rows are four input channels of one tap, the lanes of a warp lie along them (opaque to the compiler, so that
        // it keeps no addresses in registers during the main loop)
        int m = m0;
        asm volatile("" : "+r"(m));
        const int tap = tap0 + m / CIB, ci = c0 + m % CIB;
        if (tap >= 27) continue;
        float* dst = P.partial + (((ll) blockIdx.x * 27 + tap) * P.cout + o0 + n_off) * P.cin + ci;
#pragma unroll
        for (int n = 0; n < TN; ++n, dst += P.cin) {
            if (o0 + n_off + n >= P.cout) break;
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { const float2 pair = unpack2(IN_REGISTERS ? done[IN_REGISTERS ? i : 0][IN_REGISTERS ? n / 2 : 0] : acc[i][n / 2]); v[i] = n & 1 ? pair.y : pair.x; }
            if (!IN_REGISTERS && s0 > 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i) if (ci + i < P.cin) asm volatile("red.global.add.f32 [%0], %1;" ::"l"(dst + i), "f"(v[i]) : "memory");
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) if (ci + i < P.cin) dst[i] = v[i];
            }
        }
    } while (s < total);
    cp_async_wait<0>();
}

// grad_weights[slot][filter][tap] = (+=) the block sums [range][tap][filter] of the slot's ranges, filter = co * cin + ci.  Block = 32
// filters of one slot: warp y takes every eighth range, 27 independent coalesced loads at a time; the warps' sums are combined in a
// fixed order and leave transposed, as contiguous filters.
__global__ void __launch_bounds__(256) dw_reduce_kernel(const float* __restrict__ partial, SlotRanges sr, int accumulate, ll filters, float* __restrict__ gw) {
    __shared__ float sums[8][27][33];
    const int lane = threadIdx.x & 31, y = threadIdx.x >> 5;
    const ll f0 = (ll) blockIdx.x * 32, f = f0 + lane;
    int slot, r0 = 0, r1 = 0;
    if ((int) blockIdx.y < sr.n) { slot = sr.slot[blockIdx.y]; r0 = sr.first[blockIdx.y]; r1 = sr.first[blockIdx.y + 1]; }
    else {                                     // the k-th slot without ranges
        unsigned left = sr.empty;
        for (int k = (int) blockIdx.y - sr.n; k > 0; --k) left &= left - 1;
        slot = __ffs(left) - 1;
    }
    const int ny = min(8, r1 - r0);
    float s[27];
#pragma unroll
    for (int t = 0; t < 27; ++t) s[t] = 0.f;
    if (f < filters) {
        for (int r = r0 + y; r < r1; r += 8) {
            const float* p = partial + r * 27 * filters + f;
#pragma unroll
            for (int t = 0; t < 27; ++t) s[t] += __ldg(p + t * filters);
        }
    }
    if (y < ny) {
#pragma unroll
        for (int t = 0; t < 27; ++t) sums[y][t][lane] = s[t];
    }
    __syncthreads();
    const int n = (int) min((ll) 32, filters - f0) * 27;
    float* dst = gw + ((ll) slot * filters + f0) * 27;
    for (int e = threadIdx.x; e < n; e += 256) {
        const int c = e / 27, t = e - c * 27;
        float v = 0.f;
        for (int k = 0; k < ny; ++k) v += sums[k][t][c];
        dst[e] = accumulate ? dst[e] + v : v;
    }
}

// ---- host side ----------------------------------------------------------------------------------------
inline int pad4(int c) { return (c + 3) / 4 * 4; }
inline size_t align256(size_t b) { return (b + 255) / 256 * 256; }
inline size_t rows_bytes(ll rows, int channels) { return align256((size_t) rows * pad4(channels) * sizeof(float)); }

// tile width of `n` channels among `count` candidates: the least time, taking each one's measured rate relative to the widest
inline int pick_width(int n, const int* width, const double* rate, int count) {
    int best = 0;
    double cost = 0;
    for (int i = 0; i < count; ++i) {
        const double c = (n + width[i] - 1) / width[i] * width[i] / rate[i];
        if (i == 0 || c < cost) { best = i; cost = c; }
    }
    return width[best];
}

// output channels per tile (forward and input gradient 16 -> 16: 29 to 31, 32 -> 32: 37 to 39, 64 -> 64: 48 to 49, 8 -> 8: 13 to 15 TFLOP/s)
inline int pick_nt(int n) {
    static const int width[4] = {64, 32, 16, 8};
    static const double rate[4] = {1.0, 0.8, 0.62, 0.33};
    return pick_width(n, width, rate, 4);
}

inline size_t weight_bytes(int k_dim, int n_dim, int slots) {
    const int nt = pick_nt(n_dim);
    return align256((size_t) slots * 27 * ((n_dim + nt - 1) / nt * nt) * pad4(k_dim) * sizeof(float));
}

int run_pack_rows(const float* x, ll ld_x, int split, const float* x1, ll ld_x1, ll n, const float* tree, ll ld_tree, ll t, int c, float* out, cudaStream_t st) {
    dim3 grid((unsigned) aprnet_ceil_div(n + t + 1, 64), (unsigned) aprnet_ceil_div(pad4(c), 32));
    AprnetProfScope _prof("pack_rows_f32", st);
    if (split < c) pack_rows_f32_kernel<true><<<grid, 256, 0, st>>>(x, ld_x, split, x1, ld_x1, n, tree, ld_tree, t, c, pad4(c), out);
    else pack_rows_f32_kernel<false><<<grid, 256, 0, st>>>(x, ld_x, split, x1, ld_x1, n, tree, ld_tree, t, c, pad4(c), out);
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

int run_pack_weights(const aprnet_apr* a, int dl, const float* w, int slots, int cin, int cout, int transposed, float* wp, cudaStream_t st) {
    const int n_dim = transposed ? cin : cout, nt = pick_nt(n_dim);
    return aprnet_pack_weights(a, dl, false, w, slots, cin, cout, transposed, nt, (n_dim + nt - 1) / nt, pad4(transposed ? cout : cin), wp, st);
}

template<int WM, int WN, int TN, int R, int MODE, bool MANY = false>
int launch_gather(F32Params& P, const std::vector<Segment>& segs, cudaStream_t st, const char* pname) {
    constexpr int M = 32 * R * WM, NT = TN * WN;
    constexpr size_t smem = (size_t) GatherShape<WM, R, MANY>::RING * (M + NT) * KS * sizeof(float);
    auto kern = conv333_f32_gather_kernel<WM, WN, TN, R, MODE, MANY>;
    APRNET_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    P.segs = make_seg_table(segs, M);
    P.n_tiles = (P.n_dim + NT - 1) / NT;
    const int tiles = P.segs.tile_begin[P.segs.n];
    if (tiles == 0) return APRNET_OK;
    AprnetProfScope _prof(pname, st);
    kern<<<(unsigned) (tiles * P.n_tiles), 32 * WM * WN, smem, st>>>(P);
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

// One location per lane where four leave SMs without work: training steps on 9.7 k and 26 k locations 10.7 -> 7.5 and 12.0 -> 9.8 ms.  Up to which number of blocks: aprnet_f32_few_blocks.
template<int WM, int WN, int TN, int MODE>
int launch_tiles(F32Params& P, const std::vector<Segment>& segs, cudaStream_t st, const char* pname) {
    ll blocks = 0;
    for (const Segment& s : segs) blocks += aprnet_ceil_div(s.end - s.begin, 128 * WM);
    blocks *= (P.n_dim + TN * WN - 1) / (TN * WN);
    if (blocks <= aprnet_f32_few_blocks(TN * WN, MODE == FORWARD)) return launch_gather<WM, WN, TN, 1, MODE>(P, segs, st, pname);
    if constexpr (MORE_THREADS<WM, TN, MODE>)
        if (aprnet_f32_many_blocks(TN * WN, P.kpad, blocks)) return launch_gather<WM, WN, TN, 4, MODE, true>(P, segs, st, pname);
    return launch_gather<WM, WN, TN, 4, MODE>(P, segs, st, pname);
}

template<int MODE>
int run_gather(F32Params& P, const std::vector<Segment>& segs, cudaStream_t st, const char* pname) {
    switch (pick_nt(P.n_dim)) {
        case 64: return launch_tiles<1, 4, 16, MODE>(P, segs, st, pname);
        case 32: return launch_tiles<2, 2, 16, MODE>(P, segs, st, pname);
        case 16: return launch_tiles<2, 2, 8, MODE>(P, segs, st, pname);
        default: return launch_tiles<2, 2, 4, MODE>(P, segs, st, pname);
    }
}

struct DwGeom { int cib, nt, m, groups, ci_blocks, co_blocks; };

inline DwGeom dw_geometry(int cin, int cout) {
    DwGeom g;
    g.nt = pick_nt(cout);
    g.m = g.nt == 64 ? 128 : 256;
    static const int width[3] = {32, 16, 8};          // narrower pieces of a row cost more copies per byte
    static const double rate[3] = {1.0, 0.85, 0.5};
    g.cib = pick_width(cin, width, rate, 3);
    const int ts = g.m / g.cib;
    g.groups = (27 + ts - 1) / ts;
    g.ci_blocks = (cin + g.cib - 1) / g.cib;
    g.co_blocks = (cout + g.nt - 1) / g.nt;
    return g;
}

// ring slots (16 locations) per chain of a block, for a level of `len` locations and tiles of nt output channels.  In registers: 128
// locations.  In the workspace, where the end of a chain writes the block's sums: at least 512 locations, and 1 / 256 of the level.
inline int dw_flush_slots(ll len, int nt) { return nt <= 16 ? 128 / KS : (int) std::max<ll>(512 / KS, (len / 256 + KS - 1) / KS); }

// ranges of the whole launch: enough blocks for four waves of three per SM, bounded by 64 Mi partial sums
inline int dw_max_ranges(int cin, int cout) {
    const DwGeom g = dw_geometry(cin, cout);
    const ll per = (ll) 27 * cin * cout, blocks_y = (ll) g.groups * g.ci_blocks * g.co_blocks;
    const ll want = (4 * 3 * 148 + blocks_y - 1) / blocks_y;
    return (int) std::max<ll>(MAX_SEGS, std::min<ll>(want, (64ll << 20) / per));
}

template<int CIB, int WM, int WN, int TN>
int launch_dw(const F32DwParams& P, int nranges, int blocks_y, cudaStream_t st, const char* pname) {
    constexpr int TS = 128 * WM / CIB, TAP_STRIDE = KS * CIB + (CIB < 32 ? CIB : 0);
    constexpr size_t smem = (size_t) DwShape<CIB, WM, TN>::RING * (TS * TAP_STRIDE + KS * TN * WN) * sizeof(float);
    auto kern = conv333_f32_dw_kernel<CIB, WM, WN, TN>;
    APRNET_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    AprnetProfScope _prof(pname, st);
    kern<<<dim3((unsigned) nranges, (unsigned) blocks_y), 32 * WM * WN, smem, st>>>(P);
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

int run_dw(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* xrows, const float* grows, float* gw, int accumulate, float* partial, cudaStream_t st) {
    const AprPlan* plan = aprnet_get_plan(a, dl, st);
    if (!plan) return APRNET_ERR_CUDA;
    const DwGeom g = dw_geometry(cin, cout);
    const std::vector<Segment> segs = aprnet_segments(a, dl, slots, false);
    if (segs.empty()) return accumulate ? APRNET_OK : (cudaMemsetAsync(gw, 0, (size_t) slots * 27 * cin * cout * sizeof(float), st), APRNET_OK);
    const int budget = dw_max_ranges(cin, cout);
    F32DwParams P;
    P.n_segs = (int) segs.size();
    ll total_units = 0;
    for (const Segment& sg : segs) total_units += (sg.end - sg.begin + DW_UNIT - 1) / DW_UNIT;
    // every level gets blocks in proportion to its units, at least two units each where the budget allows
    auto blocks_for = [&](ll per_block) { ll b = 0; for (const Segment& sg : segs) b += ((sg.end - sg.begin + DW_UNIT - 1) / DW_UNIT + per_block - 1) / per_block; return b; };
    ll per_block = std::max<ll>(2, (total_units + budget - 1) / budget);
    while (blocks_for(per_block) > budget) ++per_block;
    SlotRanges sr;
    sr.n = 0;
    P.range_first[0] = 0;
    for (int i = 0; i < P.n_segs; ++i) {
        P.seg_begin[i] = segs[i].begin; P.seg_end[i] = segs[i].end; P.seg_flush[i] = dw_flush_slots(segs[i].end - segs[i].begin, g.nt);
        P.range_first[i + 1] = P.range_first[i] + (int) (((segs[i].end - segs[i].begin + DW_UNIT - 1) / DW_UNIT + per_block - 1) / per_block);
        // levels are listed coarse to fine, so those that share a slot (the last one) are neighbours
        if (sr.n == 0 || sr.slot[sr.n - 1] != segs[i].slot) { sr.first[sr.n] = P.range_first[i]; sr.slot[sr.n++] = segs[i].slot; }
        sr.first[sr.n] = P.range_first[i + 1];
    }
    P.nbr = plan->nbr; P.N = plan->n;
    P.xrows = xrows; P.xpad = pad4(cin); P.tree_base = plan->n; P.zero_row = plan->n + plan->tree_size;
    P.grows = grows; P.gpad = pad4(cout); P.g_zero_row = plan->n;
    P.partial = partial; P.cin = cin; P.cout = cout; P.ci_blocks = g.ci_blocks; P.groups = g.groups;
    const int nranges = P.range_first[P.n_segs], blocks_y = g.groups * g.ci_blocks * g.co_blocks;
    char pname[64];
    snprintf(pname, sizeof(pname), "conv333_dw:ci%d:co%d:dl%d", cin, cout, dl);
    int rc = APRNET_ERR_UNSUPPORTED;
#define DW_CASE(CIB_, NT_, WM_, WN_, TN_) if (g.cib == CIB_ && g.nt == NT_) rc = launch_dw<CIB_, WM_, WN_, TN_>(P, nranges, blocks_y, st, pname);
    DW_CASE(32, 64, 1, 4, 16) DW_CASE(32, 32, 2, 2, 16) DW_CASE(32, 16, 2, 2, 8) DW_CASE(32, 8, 2, 2, 4)
    DW_CASE(16, 64, 1, 4, 16) DW_CASE(16, 32, 2, 2, 16) DW_CASE(16, 16, 2, 2, 8) DW_CASE(16, 8, 2, 2, 4)
    DW_CASE(8, 64, 1, 4, 16) DW_CASE(8, 32, 2, 2, 16) DW_CASE(8, 16, 2, 2, 8) DW_CASE(8, 8, 2, 2, 4)
#undef DW_CASE
    return rc ? rc : aprnet_dw_reduce(partial, sr, slots, accumulate, cin, cout, gw, st);
}

// cross-level part of the input gradient (see edge_plan.cu; wp: the transposed weights as packed for the same-level part): sums per (target, tap), then the gather over the targets
int run_cross(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* grows, float* gin, ll ld_in, float* gtree, ll ld_tree,
              float* wp, float* vrows, ll vrow_bytes, cudaStream_t st) {
    EdgePlan* ep = aprnet_get_edge_plan(a, dl, st);
    if (!ep) return APRNET_ERR_CUDA;
    if (ep->n_active == 0) return APRNET_OK;
    const int gpad = pad4(cout), cml = a->cml(dl);
    int rc = APRNET_OK;
    // virtual rows lie a whole number of rows behind the first dO row, so that the gather addresses both from there
    const ll row = (ll) gpad * 4, off = ((char*) vrows - (char*) grows + row - 1) / row, cap_rows = ((char*) vrows + vrow_bytes - (char*) grows) / row - off;
    vrows = const_cast<float*>(grows) + off * gpad;
    const int nk = (int) ep->chunk_a.size() - 1;
    char pname[64];
    snprintf(pname, sizeof(pname), "conv333_bwd_cross_pull:ci%d:co%d:dl%d", cin, cout, dl);
    for (int k0 = 0, k1; k0 < nk; k0 = k1) {
        k1 = aprnet_vrow_pass_end(ep->chunk_v, k0, cap_rows);
        const ll v0 = ep->chunk_v[k0], v1 = ep->chunk_v[k1], a0 = ep->chunk_a[k0], a1 = ep->chunk_a[k1];
        if (v1 - v0 > cap_rows) { aprnet_set_error("edge workspace too small for %lld virtual rows", v1 - v0); return APRNET_ERR_ARG; }
        if (v1 > v0) {
            AprnetProfScope _prof("edge_reduce", st);
            vrow_reduce_f32_kernel<<<aprnet_ceil_div((v1 - v0) * (gpad / 4), 256), 256, 0, st>>>(ep->vstart, ep->vsrc, v0, v1, grows, gpad, vrows);
        }
        std::vector<Segment> segs;
        for (const ActiveSeg& sg : ep->segs) {
            Segment s;
            s.begin = std::max(sg.begin, a0); s.end = std::min(sg.end, a1);
            s.level = sg.location_level; s.slot = std::min(cml - sg.location_level, slots - 1);
            if (s.end > s.begin) segs.push_back(s);
        }
        if (segs.empty()) continue;
        F32Params P;
        memset(&P, 0, sizeof(P));
        P.nbr = ep->vnbr; P.N = ep->n_active; P.rows = grows; P.kpad = gpad; P.zero_row = a->number_parts(dl); P.tree_base = 0; P.v_shift = off - v0;
        P.wp = wp; P.n_dim = cin;
        P.out = gin; P.ld_out = ld_in; P.out_map = ep->active; P.out_split = a->number_parts(dl); P.out2 = gtree; P.ld_out2 = ld_tree;
        if ((rc = run_gather<TARGETS>(P, segs, st, pname))) return rc;
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

inline size_t edge_bytes(const aprnet_apr* a, int dl, int cout) {
    const auto it = a->edge_plans.find(dl);
    return align256((size_t) aprnet_vrow_workspace_bytes(it != a->edge_plans.end() ? it->second.n_vrows : 27 * a->number_parts(dl), (ll) pad4(cout) * 4));
}

} // namespace

int aprnet_dw_reduce(const float* partial, SlotRanges sr, int slots, int accumulate, int cin, int cout, float* gw, cudaStream_t st) {
    int nz = sr.n;
    sr.empty = 0;
    if (!accumulate) {
        if (slots > 32) { APRNET_CUDA_CHECK(cudaMemsetAsync(gw, 0, (size_t) slots * 27 * cin * cout * sizeof(float), st)); accumulate = 1; }      // (more slots than any structure has levels)
        else {
            sr.empty = slots == 32 ? ~0u : (1u << slots) - 1;
            for (int i = 0; i < sr.n; ++i) sr.empty &= ~(1u << sr.slot[i]);
            nz += __builtin_popcount(sr.empty);
        }
    }
    if (nz == 0) return APRNET_OK;
    AprnetProfScope _prof("conv333_dw_reduce", st);
    const ll filters = (ll) cin * cout;
    dw_reduce_kernel<<<dim3((unsigned) aprnet_ceil_div(filters, 32), (unsigned) nz), 256, 0, st>>>(partial, sr, accumulate, filters, gw);
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

// bytes of the packed rows of the input (particles, tree means, zero row), which a forward call leaves at the start of its workspace
size_t aprnet_f32_rows_bytes(const aprnet_apr* a, int dl, int cin) {
    const ll rows = a->number_parts(dl) + a->tree_size(dl) + 1;
    // first-layer widths keep a channel-major copy instead (conv333_small.cu)
    return aprnet_small_cin(cin) ? align256((size_t) rows * cin * sizeof(float)) : rows_bytes(rows, cin);
}

size_t aprnet_f32_forward_bytes(const aprnet_apr* a, int dl, int cin, int cout, int slots) {
    return aprnet_f32_rows_bytes(a, dl, cin) + (aprnet_small_cin(cin) ? 0 : weight_bytes(cin, cout, slots));
}

size_t aprnet_f32_backward_bytes(const aprnet_apr* a, int dl, int cin, int cout, int slots) {
    return rows_bytes(a->number_parts(dl) + 1, cout) + weight_bytes(cout, cin, slots) + edge_bytes(a, dl, cout);
}

int64_t aprnet_f32_partial_elems(int cin, int cout) {
    return (int64_t) std::max<ll>((ll) dw_max_ranges(cin, cout) * 27 * cin * cout, aprnet_small_cin(cin) ? aprnet_conv333_tc_dw_partial_elems(cin, cout) : 0);
}

int aprnet_f32_pack_input(const aprnet_apr* a, int dl, int cin, const float* in, ll ld_in, const float* tree, ll ld_tree, void* rows, cudaStream_t st) {
    const ll n = a->number_parts(dl), t = a->tree_size(dl);
    if (aprnet_small_cin(cin)) return aprnet_small_stage(in, ld_in, n, tree, ld_tree, t, cin, (float*) rows, st);
    return run_pack_rows(in, ld_in, cin, in, ld_in, n, tree, ld_tree, t, cin, (float*) rows, st);
}

int aprnet_f32_pack_pair(const aprnet_apr* a, int dl, int cin, const float* in0, ll ld0, int c0, const float* in1, ll ld1, const float* tree, ll ld_tree, void* rows, cudaStream_t st) {
    return run_pack_rows(in0, ld0, c0, in1, ld1, a->number_parts(dl), tree, ld_tree, a->tree_size(dl), cin, (float*) rows, st);
}

int aprnet_f32_pack_grad(const aprnet_apr* a, int dl, int cout, const float* gout, ll ld_out, void* grows, cudaStream_t st) {
    return run_pack_rows(gout, ld_out, cout, gout, ld_out, a->number_parts(dl), nullptr, 0, 0, cout, (float*) grows, st);
}

// forward from the packed input rows at the start of `workspace` (aprnet_f32_forward_bytes)
int aprnet_f32_forward(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* w, const float* bias, float* out, ll ld_out, void* workspace, cudaStream_t st) {
    if (aprnet_small_cin(cin)) return aprnet_small_forward(a, dl, cin, cout, slots, (const float*) workspace, w, bias, out, ld_out, st);
    const AprPlan* plan = aprnet_get_plan(a, dl, st);
    if (!plan) return APRNET_ERR_CUDA;
    float* wp = (float*) ((char*) workspace + aprnet_f32_rows_bytes(a, dl, cin));
    int rc = run_pack_weights(a, dl, w, slots, cin, cout, 0, wp, st);
    if (rc) return rc;
    F32Params P;
    memset(&P, 0, sizeof(P));
    P.nbr = plan->nbr; P.N = plan->n; P.rows = (const float*) workspace; P.kpad = pad4(cin);
    P.tree_base = plan->n; P.zero_row = plan->n + plan->tree_size;
    P.wp = wp; P.n_dim = cout; P.out = out; P.ld_out = ld_out; P.bias = bias;
    char pname[64];
    snprintf(pname, sizeof(pname), "conv333_fwd:ci%d:co%d:dl%d", cin, cout, dl);
    return run_gather<FORWARD>(P, aprnet_segments(a, dl, slots, false), st, pname);
}

int aprnet_f32_backward_weights(aprnet_apr* a, int dl, int cin, int cout, int slots, const void* rows, const float* gout, ll ld_out, const void* grows,
                                float* gw, int accumulate, float* partial, cudaStream_t st) {
    if (aprnet_small_cin(cin)) return aprnet_small_backward_weights(a, dl, cin, cout, slots, (const float*) rows, gout, ld_out, gw, accumulate, partial, st);
    return run_dw(a, dl, cin, cout, slots, (const float*) rows, (const float*) grows, gw, accumulate, partial, st);
}

// input gradient from the packed grad_output rows at the start of `workspace` (aprnet_f32_backward_bytes): grad_input is written,
// grad_tree zero-filled and, with tree_adjoint, folded into it
int aprnet_f32_backward_input(aprnet_apr* a, int dl, int cin, int cout, int slots, const float* gout, ll ld_out, const float* w, float* gin, ll ld_in, float* gtree, ll ld_tree,
                              void* workspace, bool tree_adjoint, cudaStream_t st) {
    const AprPlan* plan = aprnet_get_plan(a, dl, st);
    if (!plan) return APRNET_ERR_CUDA;
    const ll n = plan->n, ts = plan->tree_size;
    float* grows = (float*) workspace;
    float* wp = (float*) ((char*) workspace + rows_bytes(n + 1, cout));
    float* vrows = (float*) ((char*) wp + weight_bytes(cout, cin, slots));
    int rc = run_pack_weights(a, dl, w, slots, cin, cout, 1, wp, st);
    if (rc) return rc;
    F32Params P;
    memset(&P, 0, sizeof(P));
    P.nbr = plan->nbr; P.N = n; P.rows = grows; P.kpad = pad4(cout); P.tree_base = n; P.zero_row = n; P.same_level_only = 1; P.mirror = 1;
    P.wp = wp; P.n_dim = cin; P.out = gin; P.ld_out = ld_in;
    char pname[64];
    snprintf(pname, sizeof(pname), "conv333_bwd_input:ci%d:co%d:dl%d", cin, cout, dl);
    if ((rc = run_gather<SAME_LEVEL>(P, aprnet_segments(a, dl, slots, false), st, pname))) return rc;
    if (27 * n + 1 >= (1ll << 31)) {
        // more than 79.5 M locations: the 32-bit edge ids of the edge plan run out; the cross-level part is scattered with
        // atomic adds instead (correct, but the summation order is no longer fixed)
        return aprnet_cross_level_scatter(a, dl, cin, cout, slots, gout, ld_out, w, gin, ld_in, gtree, ld_tree, tree_adjoint, st);
    }
    if (ts > 0) APRNET_CUDA_CHECK(cudaMemset2DAsync(gtree, (size_t) ld_tree * sizeof(float), 0, (size_t) ts * sizeof(float), (size_t) cin, st));
    if ((rc = run_cross(a, dl, cin, cout, slots, grows, gin, ld_in, gtree, ld_tree, wp, vrows, (ll) edge_bytes(a, dl, cout), st))) return rc;
    return tree_adjoint ? aprnet_fill_tree_mean_backward(a, dl, APRNET_F32, cin, gin, ld_in, gtree, ld_tree, st) : APRNET_OK;
}
