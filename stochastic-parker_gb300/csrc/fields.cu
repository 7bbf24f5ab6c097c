// Field preparation kernels: raw 8-variable frames -> 32-variable arrays
// with gradients (mhd_data_parallel.f90:504-610) -> packed mover records.
#include "device_common.cuh"
#include "fp64_exact.cuh"

namespace gpat {

// Slot order of the packed records, as indices into the 32-variable cell
// (vars 0-7: vx vy vz rho bx by bz |B|; gradient of var v along d at 8+3v+d).
__constant__ int kPack2D[kRec2D] = {0, 1, 4, 5, 6, 8, 12, 20, 21, 23, 24, 26, 27, 29, 30, 3};
__constant__ int kPack3D[kRec3D] = {0, 1, 2, 4, 5, 6, 8, 12, 16, 20, 21, 22,
                                    23, 24, 25, 26, 27, 28, 29, 30, 31, 3, 7, -1};

// One 16-byte chunk of the 32-variable record per thread: HBM streaming (32 B
// read, 128 B written per cell) with full lines written.
__global__ void scatter_raw_kernel(const float4 *__restrict__ raw, float4 *__restrict__ full,
                                   size_t ncells) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < 8 * ncells; t += stride) {
        const int q = (int)(t & 7);
        full[t] = q < 2 ? raw[2 * (t >> 3) + q] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

cudaError_t launch_scatter_raw_fields(const float *raw, float *full, size_t ncells,
                                      cudaStream_t s) {
    const int threads = 256;
    const size_t blocks = (8 * ncells + threads - 1) / threads;
    scatter_raw_kernel<<<(unsigned)(blocks < 65535 * 16 ? blocks : 65535 * 16), threads, 0, s>>>(
        reinterpret_cast<const float4 *>(raw), reinterpret_cast<float4 *>(full), ncells);
    return cudaGetLastError();
}

// One-sided / centred difference exactly as the reference evaluates it:
// single-precision differences, scaled by the double 0.5/d, rounded to float.
__device__ __forceinline__ float grad_lo(float a0, float a1, float a2, double ih) {
    float t = -__fmul_rn(3.0f, a0);
    t = __fadd_rn(t, __fmul_rn(4.0f, a1));
    t = __fsub_rn(t, a2);
    return (float)__dmul_rn((double)t, ih);
}
__device__ __forceinline__ float grad_hi(float an, float an1, float an2, double ih) {
    float t = __fmul_rn(3.0f, an);
    t = __fsub_rn(t, __fmul_rn(4.0f, an1));
    t = __fadd_rn(t, an2);
    return (float)__dmul_rn((double)t, ih);
}
__device__ __forceinline__ float grad_c(float ap, float am, double ih) {
    return (float)__dmul_rn((double)__fsub_rn(ap, am), ih);
}

// Gradients of the fluctuation records {db2_slab, db2_2d, lc_slab, lc_2d}, 16 floats
// a node: value v at 4 v, its d/dx d/dy d/dz behind it; the z component only in 3D.
// ihx/ihy/ihz: per-node inverse spans of a non-uniform grid (idxh_grid of
// set_local_grid_positions, mhd_data_parallel.f90:2153-2190, as used by
// calc_fields_gradients_nonuniform :612-764), or null for 0.5 / d.  odd_found: set
// where a value or a gradient is subnormal, infinite or NaN; the values are looked
// at where the x differences have read them, node i + 1 at node i.
__global__ void aux_gradients_kernel(float *__restrict__ a, int ndim, int nxg, int nyg, int nzg,
                                     double idxh, double idyh, double idzh,
                                     const double *__restrict__ ihx, const double *__restrict__ ihy,
                                     const double *__restrict__ ihz, unsigned int *odd_found) {
    const size_t ncells = (size_t)nxg * nyg * nzg;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t sx = 16, sy = 16 * (size_t)nxg, sz = 16 * (size_t)nxg * nyg;
    bool odd = false;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += stride) {
        const int i = (int)(c % nxg);
        const int j = (int)((c / nxg) % nyg);
        const int k = (int)(c / ((size_t)nxg * nyg));
        const double hx = ihx ? ihx[i] : idxh;
        const double hy = ihy ? ihy[j] : idyh;
        const double hz = ihz ? ihz[k] : idzh;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            float *cell = a + 16 * c + 4 * v, d;
            if (i == 0) {
                d = grad_lo(cell[0], cell[sx], cell[2 * sx], hx);
                odd |= odd_float(cell[0]) | odd_float(cell[sx]);
            } else if (i == nxg - 1) {
                d = grad_hi(cell[0], *(cell - sx), *(cell - 2 * sx), hx);
            } else {
                d = grad_c(cell[sx], *(cell - sx), hx);
                odd |= odd_float(cell[sx]);
            }
            cell[1] = d;
            odd |= odd_float(d);
            if (nyg > 1) {
                if (j == 0) d = grad_lo(cell[0], cell[sy], cell[2 * sy], hy);
                else if (j == nyg - 1) d = grad_hi(cell[0], *(cell - sy), *(cell - 2 * sy), hy);
                else d = grad_c(cell[sy], *(cell - sy), hy);
                cell[2] = d;
                odd |= odd_float(d);
            }
            if (nzg > 1 && ndim == 3) {
                if (k == 0) d = grad_lo(cell[0], cell[sz], cell[2 * sz], hz);
                else if (k == nzg - 1) d = grad_hi(cell[0], *(cell - sz), *(cell - 2 * sz), hz);
                else d = grad_c(cell[sz], *(cell - sz), hz);
                cell[3] = d;
                odd |= odd_float(d);
            }
        }
    }
    if (odd) *odd_found = 1u;
}

// (float)((double)t * ih), the reference's rounding to double and then to
// float, from ih = hi + lo in floats: t * hi in two floats plus t * lo is within
// 2^-46 of the product, and gives the same float wherever it lies clearly
// inside that float's rounding interval.  Elsewhere (one value in 2^13, powers
// of two, very small or large ones) the double product decides.
__device__ __forceinline__ float scale_diff(float t, double ih, float hi, float lo) {
    const float p = __fmul_rn(t, hi);
    const float e = __fmaf_rn(t, lo, __fmaf_rn(t, hi, -p));
    const float r = __fadd_rn(p, e);
    const float d = __fadd_rn(__fsub_rn(p, r), e);
    const unsigned b = __float_as_uint(r) & 0x7fffffffu, ex = b & 0x7f800000u;
    const float half_ulp = __uint_as_float(ex - (24u << 23));
    if (ex - (70u << 23) < (120u << 23) && b != ex && fabsf(d) < half_ulp * 0.9999f) return r;
    return (float)__dmul_rn((double)t, ih);
}

// The three differences grad_lo, grad_c, grad_hi take, before scaling.
__device__ __forceinline__ float axis_diff(const float *v, size_t stride, int at, int n) {
    if (at == 0) {
        const float t = __fadd_rn(-__fmul_rn(3.0f, v[0]), __fmul_rn(4.0f, v[stride]));
        return __fsub_rn(t, v[2 * stride]);
    }
    if (at == n - 1) {
        const float t = __fsub_rn(__fmul_rn(3.0f, v[0]), __fmul_rn(4.0f, *(v - stride)));
        return __fadd_rn(t, *(v - 2 * stride));
    }
    return __fsub_rn(v[stride], *(v - stride));
}

struct GradArgs {
    int ndim, nxg, nyg, nzg;
    double idh[3];
    float hi[3], lo[3];
    const double *ih[3];   // per-node inverse spans, or null
};

// Gradients (GRAD) and packed records, eight lanes per cell: lane v takes the
// derivatives of variable v, the cell's 32 values meet in shared memory, and
// each lane then writes one 16-byte chunk of the gradients and of the record.
// HBM streaming: 32 B read and 96 + 64 (2D) or 96 (3D) B written per cell.
// One thread per cell with scalar stores at a stride of 128 bytes took 1055 us
// for the gradients of 132^3 cells, 564 us for the records.
template <int R, bool GRAD>
__global__ void __launch_bounds__(256) fields_kernel(float *full, float *rec, size_t ncells,
                                                     const GradArgs g, unsigned int *odd_found) {
    __shared__ __align__(16) float cells[32][32];
    const int v = threadIdx.x & 7, slot = threadIdx.x >> 3;
    bool odd = false;
    const size_t sx = 32, sy = 32 * (size_t)g.nxg, sz = 32 * (size_t)g.nxg * g.nyg;
    for (size_t c0 = 32 * (size_t)blockIdx.x; c0 < ncells; c0 += 32 * (size_t)gridDim.x) {
        const size_t c = c0 + slot;
        if (c < ncells) {
            float *cell = full + 32 * c;
            if (GRAD) {
                const unsigned row = (unsigned)(c / (unsigned)g.nxg);
                const int i = (int)(c - (size_t)row * (unsigned)g.nxg);
                const int k = (int)(row / (unsigned)g.nyg), j = (int)(row - (unsigned)k * (unsigned)g.nyg);
                const int at[3] = {i, j, k}, n[3] = {g.nxg, g.nyg, g.nzg};
                const size_t st[3] = {sx, sy, sz};
                const float x = cell[v];
                cells[slot][v] = x;
                odd |= odd_float(x);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    float y;
                    if (d == 0 || (n[d] > 1 && (d == 1 || g.ndim == 3))) {
                        const float t = axis_diff(cell + v, st[d], at[d], n[d]);
                        y = g.ih[d] ? (float)__dmul_rn((double)t, g.ih[d][at[d]])
                                    : scale_diff(t, g.idh[d], g.hi[d], g.lo[d]);
                    } else {
                        y = cell[8 + 3 * v + d];   // not resolved: kept
                    }
                    cells[slot][8 + 3 * v + d] = y;
                    odd |= odd_float(y);
                }
            } else {
                const float4 x = reinterpret_cast<const float4 *>(cell)[v];
                reinterpret_cast<float4 *>(cells[slot])[v] = x;
                odd |= odd_float(x.x) | odd_float(x.y) | odd_float(x.z) | odd_float(x.w);
            }
        }
        __syncwarp();
        if (c < ncells) {
            if (GRAD && v >= 2)
                reinterpret_cast<float4 *>(full + 32 * c)[v] =
                    reinterpret_cast<const float4 *>(cells[slot])[v];
            if (v < R / 4) {
                float o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int from = (R == kRec2D) ? kPack2D[4 * v + e] : kPack3D[4 * v + e];
                    o[e] = from >= 0 ? cells[slot][from] : 0.0f;
                }
                reinterpret_cast<float4 *>(rec + (size_t)R * c)[v] =
                    make_float4(o[0], o[1], o[2], o[3]);
            }
        }
        __syncwarp();
    }
    if (odd) *odd_found = 1u;
}

template <bool GRAD>
cudaError_t launch_fields(float *full, float *rec, int ndim, size_t ncells, const GradArgs &g,
                          unsigned int *odd, cudaStream_t s) {
    const cudaError_t e = cudaMemsetAsync(odd, 0, sizeof(unsigned int), s);
    if (e != cudaSuccess) return e;
    const size_t want = (ncells + 31) / 32;
    const unsigned blocks = (unsigned)(want < 65535 * 16 ? want : 65535 * 16);
    if (ndim == 2) fields_kernel<kRec2D, GRAD><<<blocks, 256, 0, s>>>(full, rec, ncells, g, odd);
    else fields_kernel<kRec3D, GRAD><<<blocks, 256, 0, s>>>(full, rec, ncells, g, odd);
    return cudaGetLastError();
}

cudaError_t launch_calc_fields_gradients(float *full, float *rec, int ndim, int nxg, int nyg,
                                         int nzg, double dx, double dy, double dz,
                                         const double *const *ih, unsigned int *odd,
                                         cudaStream_t s) {
    GradArgs g{};
    g.ndim = ndim;
    g.nxg = nxg; g.nyg = nyg; g.nzg = nzg;
    const double d[3] = {0.5 / dx, 0.5 / dy, 0.5 / dz};
    for (int k = 0; k < 3; ++k) {
        g.idh[k] = d[k];
        g.hi[k] = (float)d[k];
        g.lo[k] = (float)(d[k] - (double)g.hi[k]);
        g.ih[k] = ih ? ih[k] : nullptr;
    }
    return launch_fields<true>(full, rec, ndim, (size_t)nxg * nyg * nzg, g, odd, s);
}

cudaError_t launch_pack_records(const float *full, float *rec, int ndim, size_t ncells,
                                unsigned int *odd, cudaStream_t s) {
    return launch_fields<false>(const_cast<float *>(full), rec, ndim, ncells, GradArgs{}, odd, s);
}

cudaError_t launch_calc_aux_gradients(float *aux, int ndim, int nxg, int nyg, int nzg, double dx,
                                      double dy, double dz, cudaStream_t s,
                                      const double *const *ih, unsigned int *odd) {
    const cudaError_t e = cudaMemsetAsync(odd, 0, sizeof(unsigned int), s);
    if (e != cudaSuccess) return e;
    const size_t ncells = (size_t)nxg * nyg * nzg;
    const int threads = 256;
    size_t blocks = (ncells + threads - 1) / threads;
    if (blocks > 65535 * 16) blocks = 65535 * 16;
    aux_gradients_kernel<<<(unsigned)blocks, threads, 0, s>>>(
        aux, ndim, nxg, nyg, nzg, 0.5 / dx, 0.5 / dy, 0.5 / dz, ih ? ih[0] : nullptr,
        ih ? ih[1] : nullptr, ih ? ih[2] : nullptr, odd);
    return cudaGetLastError();
}

// One scalar field (nzg, nyg, nxg) into component `comp` of the 16-float
// fluctuation records.
__global__ void scatter_aux_kernel(const float *__restrict__ src, float *__restrict__ aux,
                                   int comp, size_t ncells) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += stride)
        aux[16 * c + comp] = src[c];
}

__global__ void fill_kernel(float *__restrict__ a, float v, size_t n) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += stride) a[c] = v;
}

cudaError_t launch_scatter_aux(const float *src, float *aux, int comp, size_t ncells,
                               cudaStream_t s) {
    const int threads = 256;
    size_t blocks = (ncells + threads - 1) / threads;
    if (blocks > 65535 * 16) blocks = 65535 * 16;
    scatter_aux_kernel<<<(unsigned)blocks, threads, 0, s>>>(src, aux, comp, ncells);
    return cudaGetLastError();
}

cudaError_t launch_fill(float *a, float v, size_t n, cudaStream_t s) {
    const int threads = 256;
    size_t blocks = (n + threads - 1) / threads;
    if (blocks > 65535 * 16) blocks = 65535 * 16;
    if (blocks == 0) return cudaSuccess;
    fill_kernel<<<(unsigned)blocks, threads, 0, s>>>(a, v, n);
    return cudaGetLastError();
}

}  // namespace gpat

namespace gpat {
namespace {

// Chunk-planar copy of the packed records: float4 chunk j of every node
// contiguous, planes[j * ncells + c] = rec[c * R + 4 j .. 4 j + 3].  The
// tile mover stages these planes, so neighbouring nodes of one chunk sit in
// neighbouring shared-memory bank groups.
template <int R>
__global__ void planarize_kernel(const float4 *__restrict__ rec, float4 *__restrict__ planes,
                                 size_t ncells) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += stride) {
#pragma unroll
        for (int j = 0; j < R / 4; ++j) planes[(size_t)j * ncells + c] = rec[c * (R / 4) + j];
    }
}

}  // namespace

cudaError_t launch_planarize_records(const float *rec, float *planes, int ndim, size_t ncells,
                                     cudaStream_t s) {
    const int threads = 256;
    size_t blocks = (ncells + threads - 1) / threads;
    if (blocks > 65535 * 8) blocks = 65535 * 8;
    const float4 *r = reinterpret_cast<const float4 *>(rec);
    float4 *o = reinterpret_cast<float4 *>(planes);
    if (ndim == 2) planarize_kernel<kRec2D><<<(unsigned)blocks, threads, 0, s>>>(r, o, ncells);
    else planarize_kernel<kRec3D><<<(unsigned)blocks, threads, 0, s>>>(r, o, ncells);
    return cudaGetLastError();
}

}  // namespace gpat
