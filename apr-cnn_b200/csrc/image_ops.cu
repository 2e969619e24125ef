// Particle features <-> dense image at the resolution of level cml = level_max - level_delta.
//
//   reconstruct:       image[c][z][x][y] = value of the particle (or upgraded tree node) whose cell covers
//                      the voxel (piecewise-constant reconstruction); adjoint: sum of the image over the cell
//   sample_particles:  particle = mean of the image over its cell (cells are clipped at the volume border,
//                      the divisor is the clipped volume); adjoint: every voxel of the cell gets value / volume
//
// Arithmetic follows pyapr/aprnet/cuda/src/reconstruct_gpu.cu:5-157 and sample_particles_gpu.cu:5-170.  The
// reference launches one block per (image row, level) and combines the rows of a coarse cell with atomicAdd.
// Here every value has one writer and a fixed order of summation:
//   to the image:    one launch, one warp per row of the image.  The particles tile the volume, so a row is put together from the cells of all levels that cover
//                    it, each voxel once, in shared memory, and stored in whole lines.  (A pyramid of dense images, each level painted over the two-fold enlarged
//                    coarser one, wrote and read the voxels of subdivided cells once per level and took a launch per level: 157 us for two channels of
//                    256 x 320 x 384 voxels, now 91; 39 us at the rate of a copy.)
//   from the image:  level by level over a pyramid of sums: a particle of level l is one cell of S_l, and S_(l - 1) = sums of 2x2x2 cells of S_l (S of the
//                    last level is the image), clipped at the border like the cells are.  Level l has 1/8 of the cells of level l + 1, so the
//                    pyramid costs 1/7 of the image in traffic and scratch.  The image is read once, in whole rows, by one warp per row (pairs of
//                    voxels where rows are aligned to them: 113 -> 97 us for the same two channels).
// (One warp per particle sweeping its own cell, the first kernel, touched the rows of an image 8 to 32 bytes at a time: 4.0 ms for image -> particles ->
// image with both gradients on these two channels, 6 % of the HBM rate.)
#include "apr_device.cuh"
#include <algorithm>

namespace {

typedef long long ll;
constexpr int WARPS = 8;                 // rows per block
constexpr int TPB = WARPS * 32;
constexpr int ROW_BYTES = 4096;          // of its row that a warp holds in shared memory at a time, for all channels that are painted together
constexpr int PAINT_CH = 2;              // channels that are painted together, with their cells looked up once
constexpr int CH_PER_BLOCK = 4;          // channels a warp loops over with its row pointers resolved once

// the cells that hold a value at one level: particles, and at the last level of a pooled tensor its upgraded tree nodes
struct CellRows {
    const ll* row_ptr;      // CSR row pointers of the level (already offset to its first row)
    const uint16_t* y;
    ll index_offset;        // feature index = structure index + index_offset
};

struct ImageLevel {
    CellRows rows[2];
    int n_rows_sets;
    int z_num, x_num, y_num;        // extents of the level
    int k;                          // cell edge = 2^k voxels of the image
    int Z, X, Y;                    // image extents
    int mean;                       // divide by the (clipped) cell volume
};

__device__ __forceinline__ ll first_at_or_after(const uint16_t* __restrict__ y, ll b, ll e, int target) {
    while (b < e) { const ll m = (b + e) >> 1; if ((int) y[m] < target) b = m + 1; else e = m; }
    return b;
}

// voxels of cell (z, x, y): cells at the border are clipped
__device__ __forceinline__ ll cell_volume(const ImageLevel& L, int z, int x, int y) {
    const int s = 1 << L.k;
    return (ll) (min((z + 1) * s, L.Z) - z * s) * (min((x + 1) * s, L.X) - x * s) * (min((y + 1) * s, L.Y) - y * s);
}

// the cells of every level (and, behind them, the upgraded nodes of a pooled tensor), which together tile the image
struct PaintLevels {
    int n, Z, X, Y, mean;
    CellRows rows[APRNET_MAX_LEVELS + 1];
    int k[APRNET_MAX_LEVELS + 1], x_num[APRNET_MAX_LEVELS + 1];
};

template<typename T> __device__ __forceinline__ void store_equal(T* p, T v, int count) {      // `count` values from an address that is aligned to them (1, 2 or 4)
    if (count == 1) { *p = v; return; }
    if (sizeof(T) == 8) {
        *reinterpret_cast<double2*>(p) = make_double2(v, v);
        if (count == 4) *reinterpret_cast<double2*>(p + 2) = make_double2(v, v);
    } else if (count == 4) *reinterpret_cast<float4*>(p) = make_float4(v, v, v, v);
    else *reinterpret_cast<float2*>(p) = make_float2(v, v);
}

// CH channels together.  PIECES: rows longer than a warp holds, painted piece by piece; the cells of a piece are looked for in all levels at once, a lane per level.  (Each level in
// turn and from both ends, 20 loads one after the other, 256 x 512 x 1024 voxels took 551 and 571 us for one and two float32 channels, 256 x 512 x 512 442 and 464 for float64: more
// than a pyramid; now 210 and 355, 170 and 313.)
template<typename T, int CH, bool PIECES>
__global__ void __launch_bounds__(TPB) paint_rows_kernel(const __grid_constant__ PaintLevels L, const T* __restrict__ parts, ll ld, T* __restrict__ image, int C) {
    constexpr int CHUNK = ROW_BYTES / CH / sizeof(T), VEC = 16 / sizeof(T);
    __shared__ __align__(16) T buf_s[WARPS][CH][CHUNK];
    const int lane = threadIdx.x & 31, w = __shfl_sync(0xffffffffu, (int) threadIdx.x >> 5, 0);      // (one value per warp, also to the compiler)
    const ll r = (ll) blockIdx.x * WARPS + w;
    if (r >= (ll) L.Z * L.X) return;
    const int z = (int) (r / L.X), x = (int) (r % L.X);
    // the row pointers of all levels at once, a lane per level
    ll first = 0, last = 0;
    if (lane < L.n) {
        const int k = L.k[lane];
        const ll* rp = L.rows[lane].row_ptr + (ll) (z >> k) * L.x_num[lane] + (x >> k);
        first = rp[0]; last = rp[1];
    }
    const ll stride = (ll) L.Z * L.X * L.Y;
    const int c0 = blockIdx.y * CH, nc = min(CH, C - c0);
    for (int y0 = 0; y0 < L.Y; y0 += CHUNK) {
        const int len = PIECES ? min(CHUNK, L.Y - y0) : L.Y;
        ll end = last, next = last;
        if (PIECES && first < last) {       // the cells that reach into this piece; the next one begins with the last of them or behind it
            const int k = L.k[lane], behind = ((y0 + len - 1) >> k) + 1;
            const uint16_t* __restrict__ ys = L.rows[lane].y;
            end = first_at_or_after(ys, first, min(last, first + behind - (y0 >> k)), behind);
            next = end > first && ((int) ys[end - 1] + 1) << k > y0 + len ? end - 1 : end;
        }
        for (int i = 0; i < L.n; ++i) {
            const ll pb = __shfl_sync(0xffffffffu, first, i), pe = __shfl_sync(0xffffffffu, end, i);
            const int k = L.k[i];
            const uint16_t* __restrict__ ys = L.rows[i].y;
            const T* __restrict__ src = parts + (ll) c0 * ld + L.rows[i].index_offset;
            // a lane writes `width` equal voxels of a cell; 2^shift lanes share a cell
            const int shift = max(k - 2, 0), width = k == 0 ? 1 : (k == 1 ? 2 : 4);
            const ll total = (pe - pb) << shift;
#pragma unroll 1
            for (ll e = lane; e < total; e += 32) {
                const ll p = pb + (e >> shift);
                const int cell = ys[p], at = (cell << k) + (((int) e & ((1 << shift) - 1)) << 2) - y0;
                T v[CH];
#pragma unroll
                for (int c = 0; c < CH; ++c) v[c] = src[min(c, nc - 1) * ld + p];
                if (PIECES ? (unsigned) at >= (unsigned) len : at >= len) continue;
                if (L.mean && k > 0) {
                    const int s = 1 << k, cz = z >> k, cx = x >> k;
                    const T inv = T(1) / (T) ((ll) (min((cz + 1) * s, L.Z) - cz * s) * (min((cx + 1) * s, L.X) - cx * s) * (min((cell + 1) * s, L.Y) - cell * s));
#pragma unroll
                    for (int c = 0; c < CH; ++c) v[c] *= inv;
                }
#pragma unroll
                for (int c = 0; c < CH; ++c) store_equal(&buf_s[w][c][at], v[c], width);      // (what a clipped cell writes behind the row stays in the buffer)
            }
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            if (c >= nc) break;
            T* dst = image + (c0 + c) * stride + r * L.Y + y0;
            const T* b = buf_s[w][c];
            int e = lane;
            if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
                for (int q = lane; q < len / VEC; q += 32) reinterpret_cast<int4*>(dst)[q] = reinterpret_cast<const int4*>(b)[q];
                e += len / VEC * VEC;
            }
#pragma unroll 4
            for (; e < len; e += 32) dst[e] = b[e];
        }
        __syncwarp();
        if (PIECES) first = next;
    }
}

template<typename T> struct Pair;
template<> struct Pair<float> { typedef float2 type; };
template<> struct Pair<double> { typedef double2 type; };

// S_(l - 1) = 2x2x2 sums of S_l, and the level's particles read from S_l.  One warp per row of the parent level (up to four
// rows of the level, which the particles then find in L1); parent == nullptr: only the particles are wanted.
template<typename T>
__global__ void __launch_bounds__(TPB) gather_level_kernel(const __grid_constant__ ImageLevel L, T* __restrict__ parts, ll ld, const T* __restrict__ dense,
                                                           T* __restrict__ parent, int parent_z, int parent_x, int parent_y, int C) {
    const int lane = threadIdx.x & 31;
    const ll pr = (ll) blockIdx.x * WARPS + (threadIdx.x >> 5);
    if (pr >= (ll) parent_z * parent_x) return;
    const int z0 = (int) (pr / parent_x) * 2, x0 = (int) (pr % parent_x) * 2;
    const int nz = min(2, L.z_num - z0), nx = min(2, L.x_num - x0);
    const ll stride = (ll) L.z_num * L.x_num * L.y_num, parent_stride = (ll) parent_z * parent_x * parent_y;
    const int c0 = blockIdx.y * CH_PER_BLOCK, c1 = min(C, c0 + CH_PER_BLOCK);
    if (parent) {
        for (int c = c0; c < c1; ++c) {
            const T* src = dense + c * stride + ((ll) z0 * L.x_num + x0) * L.y_num;
            T* dst = parent + c * parent_stride + pr * parent_y;
            const ll off[4] = {0, (ll) L.y_num, (ll) L.x_num * L.y_num, ((ll) L.x_num + 1) * L.y_num};
            if (nz == 2 && nx == 2 && L.y_num % 2 == 0 && (reinterpret_cast<uintptr_t>(src) & (2 * sizeof(T) - 1)) == 0) {       // rows of whole pairs
                typedef typename Pair<T>::type P2;
#pragma unroll 4
                for (int e = lane; e < parent_y; e += 32) {
                    P2 v[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = reinterpret_cast<const P2*>(src + off[q])[e];
                    dst[e] = ((v[0].x + v[0].y) + (v[1].x + v[1].y)) + ((v[2].x + v[2].y) + (v[3].x + v[3].y));
                }
                continue;
            }
#pragma unroll 2
            for (int e = lane; e < parent_y; e += 32) {
                const bool two = 2 * e + 1 < L.y_num;
                T v[8];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const bool in = (q >> 1) < nz && (q & 1) < nx;
                    v[2 * q] = in ? src[off[q] + 2 * e] : T(0);
                    v[2 * q + 1] = in && two ? src[off[q] + 2 * e + 1] : T(0);
                }
                dst[e] = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
            }
        }
    }
    for (int q = 0; q < 4; ++q) {
        if ((q >> 1) >= nz || (q & 1) >= nx) continue;
        const int z = z0 + (q >> 1), x = x0 + (q & 1);
        const ll r = (ll) z * L.x_num + x;
        for (int s = 0; s < L.n_rows_sets; ++s) {
            const ll pe = L.rows[s].row_ptr[r + 1];
            for (ll p = L.rows[s].row_ptr[r] + lane; p < pe; p += 32) {
                const int y = L.rows[s].y[p];
                const T inv = L.mean && L.k > 0 ? T(1) / (T) cell_volume(L, z, x, y) : T(1);
                for (int c = c0; c < c1; ++c) parts[c * ld + p + L.rows[s].index_offset] = dense[c * stride + r * L.y_num + y] * inv;
            }
        }
    }
}

// coarsest level that holds particles: the pyramid starts there
int first_level(const aprnet_apr* a, int cml) {
    const LevelMeta& m = a->meta;
    int l = m.level_min;
    while (l < cml && m.lvl_begin[l + 1] == m.lvl_begin[l]) ++l;
    return l;
}

// elements per channel of the pyramid below the image: levels first_level .. cml - 1
ll pyramid_elems(const aprnet_apr* a, int dl) {
    const LevelMeta& m = a->meta;
    ll n = 0;
    for (int l = first_level(a, a->cml(dl)); l < a->cml(dl); ++l) n += (ll) m.z_num[l] * m.x_num[l] * m.y_num[l];
    return n;
}

// the cells of level l, and at the last level of a pooled tensor the upgraded tree nodes behind the particles
int cell_rows(const aprnet_apr* a, int dl, int l, CellRows (&rows)[2]) {
    const LevelMeta& m = a->meta;
    rows[0].row_ptr = a->row_ptr + m.row_off[l]; rows[0].y = a->y; rows[0].index_offset = 0;
    rows[1] = rows[0];
    if (l < a->cml(dl) || dl == 0) return 1;
    rows[1].row_ptr = a->tree_row_ptr + m.trow_off[l]; rows[1].y = a->tree_y; rows[1].index_offset = a->tree_offset(l);
    return 2;
}

template<typename T>
int run_paint(const aprnet_apr* a, int dl, int C, const T* parts, ll ld, T* image, int mean, cudaStream_t st) {
    const LevelMeta& m = a->meta;
    const int cml = a->cml(dl);
    PaintLevels L;
    L.n = 0; L.Z = m.z_num[cml]; L.X = m.x_num[cml]; L.Y = m.y_num[cml]; L.mean = mean;
    for (int l = first_level(a, cml); l <= cml; ++l) {
        CellRows rows[2];
        const int sets = cell_rows(a, dl, l, rows);
        for (int i = 0; i < sets; ++i) { L.rows[L.n] = rows[i]; L.k[L.n] = cml - l; L.x_num[L.n] = m.x_num[l]; ++L.n; }
    }
    const unsigned gx = (unsigned) aprnet_ceil_div((ll) L.Z * L.X, WARPS);
    const ll voxels = (ll) L.Z * L.X * L.Y;
    AprnetProfScope _prof("cells_to_image", st);
    for (int c0 = 0, n; c0 < C; c0 += n) {                     // grid.y holds 65535 blocks
        n = std::min(C - c0, 65535 * PAINT_CH);
        const T* src = parts + c0 * ld;
        T* dst = image + c0 * voxels;
        const int pairs = n / PAINT_CH * PAINT_CH;
        if (L.Y * (ll) (PAINT_CH * sizeof(T)) <= ROW_BYTES) {
            paint_rows_kernel<T, PAINT_CH, false><<<dim3(gx, (unsigned) aprnet_ceil_div(n, PAINT_CH)), TPB, 0, st>>>(L, src, ld, dst, n);
            continue;
        }
        // longer rows: a channel that has no other beside it has the whole of the warp's shared memory
        if (pairs) paint_rows_kernel<T, PAINT_CH, true><<<dim3(gx, (unsigned) (pairs / PAINT_CH)), TPB, 0, st>>>(L, src, ld, dst, pairs);
        if (pairs == n) continue;
        src += pairs * ld; dst += pairs * voxels;
        if (L.Y * (ll) sizeof(T) <= ROW_BYTES) paint_rows_kernel<T, 1, false><<<gx, TPB, 0, st>>>(L, src, ld, dst, 1);
        else paint_rows_kernel<T, 1, true><<<gx, TPB, 0, st>>>(L, src, ld, dst, 1);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

template<typename T>
int run_gather(const aprnet_apr* a, int dl, int C, T* parts, ll ld, const T* image, int mean, T* scratch, cudaStream_t st) {
    const int cml = a->cml(dl), l0 = first_level(a, cml);
    const LevelMeta& m = a->meta;
    std::vector<T*> sums(cml + 1, nullptr);
    for (int l = l0; l < cml; ++l) { sums[l] = scratch; scratch += (ll) C * m.z_num[l] * m.x_num[l] * m.y_num[l]; }
    for (int l = cml; l >= l0; --l) {
        ImageLevel L;
        L.n_rows_sets = cell_rows(a, dl, l, L.rows);
        L.z_num = m.z_num[l]; L.x_num = m.x_num[l]; L.y_num = m.y_num[l]; L.k = cml - l;
        L.Z = m.z_num[cml]; L.X = m.x_num[cml]; L.Y = m.y_num[cml];
        L.mean = mean;
        const int pz = (L.z_num + 1) / 2, px = (L.x_num + 1) / 2, py = (L.y_num + 1) / 2;
        AprnetProfScope _prof("image_to_cells", st);
        gather_level_kernel<T><<<dim3((unsigned) aprnet_ceil_div((ll) pz * px, WARPS), (unsigned) aprnet_ceil_div(C, CH_PER_BLOCK)), TPB, 0, st>>>(
            L, parts, ld, l == cml ? image : sums[l], l == l0 ? nullptr : sums[l - 1], pz, px, py, C);
    }
    APRNET_LAUNCH_CHECK();
    return APRNET_OK;
}

template<bool TO_IMAGE>
int dispatch(const aprnet_apr* a, int dl, int dtype, int C, void* parts, ll ld, void* image, int mean, void* workspace, void* stream) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && C > 0 && parts && image, "bad argument");
    APRNET_DEVICE_CHECK(a);
    APRNET_ARG_CHECK(ld >= a->number_parts(dl), "leading dimension too small");
    if (dtype != APRNET_F32 && dtype != APRNET_F64) { aprnet_set_error("unsupported dtype %d", dtype); return APRNET_ERR_ARG; }
    cudaStream_t st = (cudaStream_t) stream;
    if (TO_IMAGE) return dtype == APRNET_F32 ? run_paint<float>(a, dl, C, (const float*) parts, ld, (float*) image, mean, st)
                                             : run_paint<double>(a, dl, C, (const double*) parts, ld, (double*) image, mean, st);
    void* own = nullptr;                 // without a workspace from the caller: stream-ordered allocation for the call
    if (!workspace) {
        APRNET_CUDA_CHECK(cudaMallocAsync(&own, (size_t) aprnet_image_workspace_bytes(a, dl, dtype, C), st));
        workspace = own;
    }
    const int rc = dtype == APRNET_F32 ? run_gather<float>(a, dl, C, (float*) parts, ld, (const float*) image, mean, (float*) workspace, st)
                                       : run_gather<double>(a, dl, C, (double*) parts, ld, (const double*) image, mean, (double*) workspace, st);
    if (own) cudaFreeAsync(own, st);
    return rc;
}

} // namespace

extern "C" int64_t aprnet_image_workspace_bytes(const aprnet_apr* a, int dl, int dtype, int C) {
    if (!a || !a->valid_dl(dl) || C <= 0) return -1;
    return std::max<int64_t>(256, (int64_t) C * pyramid_elems(a, dl) * (dtype == APRNET_F64 ? 8 : 4));
}

extern "C" int aprnet_image_dims(const aprnet_apr* a, int dl, int* z, int* x, int* y) {
    APRNET_ARG_CHECK(a && a->valid_dl(dl) && z && x && y, "bad argument");
    const int cml = a->cml(dl);
    *z = a->meta.z_num[cml]; *x = a->meta.x_num[cml]; *y = a->meta.y_num[cml];
    return APRNET_OK;
}

// image (C, Z, X, Y) of aprnet_image_dims(); every voxel is written (the cells tile the volume)
extern "C" int aprnet_reconstruct_forward(const aprnet_apr* a, int dl, int dtype, int C, const void* input, int64_t ld_in, void* image, void* stream) {
    return dispatch<true>(a, dl, dtype, C, const_cast<void*>(input), ld_in, image, 0, nullptr, stream);
}
extern "C" int aprnet_reconstruct_backward(const aprnet_apr* a, int dl, int dtype, int C, const void* grad_image, void* grad_input, int64_t ld_in, void* stream) {
    return dispatch<false>(a, dl, dtype, C, grad_input, ld_in, const_cast<void*>(grad_image), 0, nullptr, stream);
}
extern "C" int aprnet_sample_particles_forward(const aprnet_apr* a, int dl, int dtype, int C, const void* image, void* output, int64_t ld_out, void* stream) {
    return dispatch<false>(a, dl, dtype, C, output, ld_out, const_cast<void*>(image), 1, nullptr, stream);
}
extern "C" int aprnet_sample_particles_backward(const aprnet_apr* a, int dl, int dtype, int C, const void* grad_output, int64_t ld_out, void* grad_image, void* stream) {
    return dispatch<true>(a, dl, dtype, C, const_cast<void*>(grad_output), ld_out, grad_image, 1, nullptr, stream);
}

// the same two transfers with the caller's workspace (aprnet_image_workspace_bytes), which only image -> particles uses
extern "C" int aprnet_cells_to_image(const aprnet_apr* a, int dl, int dtype, int C, const void* cells, int64_t ld, void* image, int mean, void*, void* stream) {
    return dispatch<true>(a, dl, dtype, C, const_cast<void*>(cells), ld, image, mean, nullptr, stream);
}
extern "C" int aprnet_image_to_cells(const aprnet_apr* a, int dl, int dtype, int C, const void* image, void* cells, int64_t ld, int mean, void* workspace, void* stream) {
    APRNET_ARG_CHECK(workspace, "null workspace");
    return dispatch<false>(a, dl, dtype, C, cells, ld, const_cast<void*>(image), mean, workspace, stream);
}
