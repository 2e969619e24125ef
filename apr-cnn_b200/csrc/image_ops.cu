// Particle features <-> dense image at the resolution of level cml = level_max - level_delta.
//
//   reconstruct:       image[c][z][x][y] = value of the particle (or upgraded tree node) whose cell covers
//                      the voxel (piecewise-constant reconstruction); adjoint: sum of the image over the cell
//   sample_particles:  particle = mean of the image over its cell (cells are clipped at the volume border,
//                      the divisor is the clipped volume); adjoint: every voxel of the cell gets value / volume
//
// Arithmetic follows pyapr/aprnet/cuda/src/reconstruct_gpu.cu:5-157 and sample_particles_gpu.cu:5-170.  The
// reference launches one block per (image row, level) and combines the rows of a coarse cell with atomicAdd.
// Here both directions run level by level over a pyramid of dense images (level l has 1/8 of the cells of level
// l + 1, so the whole pyramid costs 1/7 of the image in traffic and scratch):
//   to the image:    dense_l = the level's particles painted over the two-fold enlarged dense_(l - 1); cells that are
//                    subdivided hold whatever lies above them and are always painted over further down, because the
//                    particles tile the volume.  The last level is the image itself.
//   from the image:  a particle of level l is one cell of S_l, and S_(l - 1) = sums of 2x2x2 cells of S_l (S of the
//                    last level is the image), clipped at the border like the cells are.
// The image is written / read exactly once, in whole rows, by one warp per row; every value has one writer and a
// fixed order of summation.  (One warp per particle sweeping its own cell, the former kernel, touched the rows of an
// image 8 to 32 bytes at a time: 4.0 ms for image -> particles -> image with both gradients on two channels of
// 256 x 320 x 384 voxels, 6 % of the HBM rate.)
#include "apr_device.cuh"
#include <algorithm>

namespace {

typedef long long ll;
constexpr int WARPS = 8;                 // rows per block
constexpr int TPB = WARPS * 32;
constexpr int CHUNK = 512;               // cells of a row that a warp holds in shared memory at a time
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

// dense[c][z][x][:] = the parent level's row enlarged two-fold, then the row's own cells over it
template<typename T>
__global__ void __launch_bounds__(TPB) paint_level_kernel(ImageLevel L, const T* __restrict__ parts, ll ld, const T* __restrict__ parent,
                                                          int parent_x, int parent_y, ll parent_stride, T* __restrict__ dense, int C) {
    __shared__ T buf_s[WARPS][CHUNK];
    const int lane = threadIdx.x & 31;
    T* buf = buf_s[threadIdx.x >> 5];
    const ll r = (ll) blockIdx.x * WARPS + (threadIdx.x >> 5);
    if (r >= (ll) L.z_num * L.x_num) return;
    const int z = (int) (r / L.x_num), x = (int) (r % L.x_num);
    const ll stride = (ll) L.z_num * L.x_num * L.y_num;
    const int c0 = blockIdx.y * CH_PER_BLOCK, c1 = min(C, c0 + CH_PER_BLOCK);
    ll rb[2] = {0, 0}, re[2] = {0, 0};
    for (int s = 0; s < L.n_rows_sets; ++s) { rb[s] = L.rows[s].row_ptr[r]; re[s] = L.rows[s].row_ptr[r + 1]; }
    const T* prow = parent ? parent + ((ll) (z >> 1) * parent_x + (x >> 1)) * parent_y : nullptr;
    for (int y0 = 0; y0 < L.y_num; y0 += CHUNK) {
        const int len = min(CHUNK, L.y_num - y0);
        ll pb[2], pe[2];
        for (int s = 0; s < 2; ++s) {
            pb[s] = rb[s]; pe[s] = re[s];
            if (L.y_num > CHUNK && pe[s] > pb[s]) {
                pb[s] = first_at_or_after(L.rows[s].y, rb[s], re[s], y0);
                pe[s] = first_at_or_after(L.rows[s].y, pb[s], re[s], y0 + CHUNK);
            }
        }
        for (int c = c0; c < c1; ++c) {
            if (prow) {
                const T* ps = prow + c * parent_stride + (y0 >> 1);
#pragma unroll 4
                for (int e = lane; e < (len + 1) >> 1; e += 32) {       // CHUNK is even: one parent value covers cells 2e and 2e + 1
                    const T v = ps[e];
                    buf[2 * e] = v; buf[2 * e + 1] = v;
                }
            }
            __syncwarp();
            for (int s = 0; s < L.n_rows_sets; ++s) {
                const T* src = parts + c * ld + L.rows[s].index_offset;
                for (ll p = pb[s] + lane; p < pe[s]; p += 32) {
                    const int y = L.rows[s].y[p];
                    T v = src[p];
                    if (L.mean && L.k > 0) v *= T(1) / (T) cell_volume(L, z, x, y);
                    buf[y - y0] = v;
                }
            }
            __syncwarp();
            T* dst = dense + c * stride + r * L.y_num + y0;
#pragma unroll 4
            for (int e = lane; e < len; e += 32) dst[e] = buf[e];
            __syncwarp();
        }
    }
}

// S_(l - 1) = 2x2x2 sums of S_l, and the level's particles read from S_l.  One warp per row of the parent level (up to four
// rows of the level, which the particles then find in L1); parent == nullptr: only the particles are wanted.
template<typename T>
__global__ void __launch_bounds__(TPB) gather_level_kernel(ImageLevel L, T* __restrict__ parts, ll ld, const T* __restrict__ dense,
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

template<typename T, bool TO_IMAGE>
int run_levels(const aprnet_apr* a, int dl, int C, T* parts, ll ld, T* image, int mean, T* scratch, cudaStream_t st) {
    const int cml = a->cml(dl), l0 = first_level(a, cml);
    const LevelMeta& m = a->meta;
    std::vector<T*> dense(cml + 1, nullptr);
    T* next = scratch;
    for (int l = l0; l < cml; ++l) { dense[l] = next; next += (ll) C * m.z_num[l] * m.x_num[l] * m.y_num[l]; }
    dense[cml] = image;
    auto level = [&](int l) {
        ImageLevel L;
        L.rows[0].row_ptr = a->row_ptr + m.row_off[l]; L.rows[0].y = a->y; L.rows[0].index_offset = 0;
        L.rows[1] = L.rows[0];
        L.n_rows_sets = 1;
        if (l == cml && dl > 0) {      // upgraded tree nodes, stored behind the particles
            L.rows[1].row_ptr = a->tree_row_ptr + m.trow_off[l]; L.rows[1].y = a->tree_y; L.rows[1].index_offset = a->tree_offset(l);
            L.n_rows_sets = 2;
        }
        L.z_num = m.z_num[l]; L.x_num = m.x_num[l]; L.y_num = m.y_num[l]; L.k = cml - l;
        L.Z = m.z_num[cml]; L.X = m.x_num[cml]; L.Y = m.y_num[cml];
        L.mean = mean;
        return L;
    };
    const unsigned gy = (unsigned) aprnet_ceil_div(C, CH_PER_BLOCK);
    if (TO_IMAGE) {
        for (int l = l0; l <= cml; ++l) {
            const ImageLevel L = level(l);
            const bool top = l == l0;
            AprnetProfScope _prof("cells_to_image", st);
            paint_level_kernel<T><<<dim3((unsigned) aprnet_ceil_div((ll) L.z_num * L.x_num, WARPS), gy), TPB, 0, st>>>(
                L, parts, ld, top ? nullptr : dense[l - 1], top ? 0 : m.x_num[l - 1], top ? 0 : m.y_num[l - 1],
                top ? 0 : (ll) m.z_num[l - 1] * m.x_num[l - 1] * m.y_num[l - 1], dense[l], C);
        }
    } else {
        for (int l = cml; l >= l0; --l) {
            const ImageLevel L = level(l);
            const int pz = (L.z_num + 1) / 2, px = (L.x_num + 1) / 2, py = (L.y_num + 1) / 2;
            AprnetProfScope _prof("image_to_cells", st);
            gather_level_kernel<T><<<dim3((unsigned) aprnet_ceil_div((ll) pz * px, WARPS), gy), TPB, 0, st>>>(
                L, parts, ld, dense[l], l == l0 ? nullptr : dense[l - 1], pz, px, py, C);
        }
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
    void* own = nullptr;                 // without a workspace from the caller: stream-ordered allocation for the call
    if (!workspace) {
        APRNET_CUDA_CHECK(cudaMallocAsync(&own, (size_t) aprnet_image_workspace_bytes(a, dl, dtype, C), st));
        workspace = own;
    }
    const int rc = dtype == APRNET_F32 ? run_levels<float, TO_IMAGE>(a, dl, C, (float*) parts, ld, (float*) image, mean, (float*) workspace, st)
                                       : run_levels<double, TO_IMAGE>(a, dl, C, (double*) parts, ld, (double*) image, mean, (double*) workspace, st);
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

// the same two transfers with the caller's workspace (aprnet_image_workspace_bytes)
extern "C" int aprnet_cells_to_image(const aprnet_apr* a, int dl, int dtype, int C, const void* cells, int64_t ld, void* image, int mean, void* workspace, void* stream) {
    APRNET_ARG_CHECK(workspace, "null workspace");
    return dispatch<true>(a, dl, dtype, C, const_cast<void*>(cells), ld, image, mean, workspace, stream);
}
extern "C" int aprnet_image_to_cells(const aprnet_apr* a, int dl, int dtype, int C, const void* image, void* cells, int64_t ld, int mean, void* workspace, void* stream) {
    APRNET_ARG_CHECK(workspace, "null workspace");
    return dispatch<false>(a, dl, dtype, C, cells, ld, const_cast<void*>(image), mean, workspace, stream);
}
