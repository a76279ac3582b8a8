// Elementwise and stencil steps of the SART/motion loop: the reference's
// cu_add.cu, cu_initial.cu, cu_division.cu, cu_multiple.cu, cu_update_udvf.cu
// and mex_diff.cu kernels (drop-in forms), plus the fused motion-pass kernels
// the engine's driver uses instead of chains of them.
#pragma once

#include <algorithm>

#include "backprojector.cuh"
#include "common.cuh"
#include "warp.cuh"

namespace mcsart {

#define MC_GRID_STRIDE(n)                                                                      \
    for (int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; id < (n);                \
         id += (int64_t)gridDim.x * blockDim.x)

// The pointwise kernels (bound by memory): VEC, four elements per load and
// store, for arrays that all begin on 16 bytes; otherwise one.  At 512x512x256
// host_add took 175 us with one element per load and 130 us with four (806 MB,
// 6.2 TB/s), host_division 195 and 146 us.
template <bool VEC, typename F> __device__ __forceinline__ void pointwise(int64_t n, F f) {
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    if (VEC) {
        for (int64_t i = t0; i < n / 4; i += step) f.four(i);
        const int64_t id = n / 4 * 4 + t0;
        if (id < n) f.one(id);
    } else {
        for (int64_t id = t0; id < n; id += step) f.one(id);
    }
}
__device__ __forceinline__ float4 ld4(const float *p, int64_t i) {
    return reinterpret_cast<const float4 *>(p)[i];
}
__device__ __forceinline__ void st4(float *p, int64_t i, float4 v) {
    reinterpret_cast<float4 *>(p)[i] = v;
}

// Forward difference along ind, 0 on the last plane (cu_add.cu:37-57).
template <typename T>
__device__ __forceinline__ float fwd_diff(const T *img0, int64_t id, const Vox &v, int nx, int ny,
                                          int nz, int ind) {
    switch (ind) {
        case 1: return (v.ix == nx - 1) ? 0.0f : ldv(img0, id + 1) - ldv(img0, id);
        case 2: return (v.iy == ny - 1) ? 0.0f : ldv(img0, id + nx) - ldv(img0, id);
        case 3: return (v.iz == nz - 1) ? 0.0f : ldv(img0, id + (int64_t)nx * ny) - ldv(img0, id);
        default: return 0.0f;
    }
}

// The stencil kernels (bound by memory) go through the volume's voxels in memory
// order (Grid3), so that every lane has a voxel whatever the slices' shape.  With
// 32 x 32 tiles of a slice (event time of a call, tiles against this): diff 21 and
// 11 us at 1x4096x64, 179 and 140 us at 512x512x256; initial2 24 and 12 us, 181 and
// 146 us.
// A block is 256 threads of N voxels each, 256 apart, all read before the first is
// stored: N = 4, or 1 where the GPU holds a thread for every voxel (diff in a
// chain of launches, N = 4 against 1: 2.3 and 1.8 us at 64x64x64, 2.5 and 2.5 us
// at 100x90x64).
constexpr unsigned STENCIL_SMALL = 148 * 2048;
template <unsigned N, typename F> __device__ __forceinline__ void stencil(const Grid3 &g, F f) {
    for (unsigned b = blockIdx.x * (256 * N) + threadIdx.x; b < g.n; b += gridDim.x * (256 * N)) {
        float v[N];
#pragma unroll
        for (unsigned k = 0; k < N; k++)
            if (const unsigned id = b + 256 * k; id < g.n) v[k] = f.value(id, g.at(id), g);
#pragma unroll
        for (unsigned k = 0; k < N; k++)
            if (const unsigned id = b + 256 * k; id < g.n) f.store(id, v[k]);
    }
}
template <unsigned N, typename F>
static __global__ void __launch_bounds__(256) stencil_kernel(const Grid3 g, const F op) {
    stencil<N>(g, op);
}
template <typename F>
int launch_stencil(mcsart_ctx *ctx, const char *name, const Grid3 &g, const F &op) {
    ctx->label = name;
    if (g.n <= STENCIL_SMALL)
        MC_LAUNCH(ctx, (stencil_kernel<1, F>), div_up(g.n, 256), 256, 0, g, op);
    else
        MC_LAUNCH(ctx, (stencil_kernel<4, F>), std::min(div_up(g.n, 1024), 148u * 8), 256, 0, g, op);
    return MCSART_OK;
}

// cu_add.cu:9-18
struct AddOp {
    float *img1;
    const float *img;
    float weight;
    __device__ void one(int64_t id) const { img1[id] = __fmaf_rn(img[id], weight, img1[id]); }
    __device__ void four(int64_t i) const {
        const float4 a = ld4(img, i), b = ld4(img1, i);
        st4(img1, i, make_float4(__fmaf_rn(a.x, weight, b.x), __fmaf_rn(a.y, weight, b.y),
                                 __fmaf_rn(a.z, weight, b.z), __fmaf_rn(a.w, weight, b.w)));
    }
};
template <bool VEC>
static __global__ void __launch_bounds__(256) add_kernel(float *img1, const float *img, int64_t n,
                                                         float weight) {
    pointwise<VEC>(n, AddOp{img1, img, weight});
}

// cu_add.cu:28-59: img1[id] += img[iy + ix*ny + iz*nx*ny] * weight * d_ind img0
struct Add2Op {
    float *img1;
    const float *img, *img0;
    float weight;
    int ind;
    __device__ float value(unsigned id, const Vox &v, const Grid3 &g) const {
        const unsigned plane = (unsigned)g.nx * g.ny;
        return __fmaf_rn(img[v.iy + (unsigned)v.ix * g.ny + v.iz * plane] * weight,
                         fwd_diff(img0, id, v, g.nx, g.ny, g.nz, ind), img1[id]);
    }
    __device__ void store(unsigned id, float v) const { img1[id] = v; }
};
// The same with img read through a 32 x 32 tile of a slice, its memory order along
// the lanes (blockDim (32, 8), four voxels per thread; the other arrays' values
// are loaded before the barrier, so that a block waits on memory once).  For
// slices of ADD2_TILE_MIN and more a side: narrower ones leave the tile's lanes
// idle (8x8x20000: 38 us, Add2Op in a stencil kernel 13), and volumes of at most
// ADD2_ROWS_MAX fill too few blocks (in a chain of launches, tiles against rows:
// 3.1 and 1.9 us at 36x36x100, 2.7 and 2.8 us at 64x64x64).
constexpr int ADD2_TILE_MIN = 16;
constexpr unsigned ADD2_ROWS_MAX = 148 * 1024;
inline dim3 add2_grid(int nx, int ny, int nz) {
    return dim3(div_up(nx, 32), std::min(div_up(ny, 32), 65535u), std::min((unsigned)nz, 65535u));
}
static __global__ void __launch_bounds__(256) add2_kernel(float *img1, const float *img, int nx,
                                                          int ny, int nz, const float *img0,
                                                          float weight, int ind) {
    __shared__ float tile[32][33];
    const int x0 = blockIdx.x * 32, ix = x0 + threadIdx.x;
    const int64_t step = ind == 1 ? 1 : ind == 2 ? nx : (int64_t)nx * ny;
    for (int iz = blockIdx.z; iz < nz; iz += gridDim.z)
        for (int y0 = blockIdx.y * 32; y0 < ny; y0 += gridDim.y * 32) {
            const int64_t slice = (int64_t)iz * nx * ny;
            float t[4], df[4], old[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int tx = x0 + threadIdx.y + 8 * k, ty = y0 + threadIdx.x;
                t[k] = tx < nx && ty < ny ? img[ty + (int64_t)tx * ny + slice] : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (const int iy = y0 + threadIdx.y + 8 * k; ix < nx && iy < ny) {
                    const int64_t id = ix + (int64_t)iy * nx + slice;
                    const bool last = ind == 1 ? ix == nx - 1 : ind == 2 ? iy == ny - 1 : iz == nz - 1;
                    df[k] = last ? 0.0f : img0[id + step] - img0[id];  // fwd_diff
                    old[k] = img1[id];
                }
#pragma unroll
            for (int k = 0; k < 4; k++) tile[threadIdx.y + 8 * k][threadIdx.x] = t[k];
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (const int iy = y0 + threadIdx.y + 8 * k; ix < nx && iy < ny) {
                    const int64_t id = ix + (int64_t)iy * nx + slice;
                    img1[id] = __fmaf_rn(tile[threadIdx.x][iy - y0] * weight, df[k], old[k]);
                }
            __syncthreads();
        }
}

// cu_initial.cu:10-17
struct InitialOp {
    float *img;
    float value;
    __device__ void one(int64_t id) const { img[id] = value; }
    __device__ void four(int64_t i) const { st4(img, i, make_float4(value, value, value, value)); }
};
template <bool VEC>
static __global__ void __launch_bounds__(256) initial_kernel(float *img, int64_t n, float value) {
    pointwise<VEC>(n, InitialOp{img, value});
}

// cu_initial.cu:27-49
struct Initial2Op {
    float *img;
    const float *img0;
    float s;  // volume + flow
    __device__ float value(unsigned id, const Vox &v, const Grid3 &g) const {
        const float dfx = fwd_diff(img0, id, v, g.nx, g.ny, g.nz, 1);
        const float dfy = fwd_diff(img0, id, v, g.nx, g.ny, g.nz, 2);
        const float dfz = fwd_diff(img0, id, v, g.nx, g.ny, g.nz, 3);
        return (dfx + dfy + dfz) * s;
    }
    __device__ void store(unsigned id, float v) const { img[id] = v; }
};

// cu_division.cu:11-25
struct DivisionOp {
    float *img1;
    const float *img;
    static __device__ float ratio(float a, float b) {
        const float q = a / b;
        return (isnan(q) || isinf(q)) ? 0.0f : q;
    }
    __device__ void one(int64_t id) const { img1[id] = ratio(img1[id], img[id]); }
    __device__ void four(int64_t i) const {
        const float4 a = ld4(img1, i), b = ld4(img, i);
        st4(img1, i, make_float4(ratio(a.x, b.x), ratio(a.y, b.y), ratio(a.z, b.z), ratio(a.w, b.w)));
    }
};
template <bool VEC>
static __global__ void __launch_bounds__(256) division_kernel(float *img1, const float *img,
                                                              int64_t n) {
    pointwise<VEC>(n, DivisionOp{img1, img});
}

// cu_multiple.cu:11-43
struct MultipleOp {
    float *img1;
    const float *img0;
    float weight;
    int ind;
    __device__ float value(unsigned id, const Vox &v, const Grid3 &g) const {
        return img1[id] * (weight * fwd_diff(img0, id, v, g.nx, g.ny, g.nz, ind));
    }
    __device__ void store(unsigned id, float v) const { img1[id] = v; }
};

// cu_update_udvf.cu:11-62.  b pairs alpha_y/beta_y with the x gradient and
// alpha_x/beta_x with the y gradient (:45-50) while the update adds the x
// component to alpha_x (:55), exactly as the reference does.  One voxel at a time:
// each field is read again behind the stores before it, as there.
static __global__ void __launch_bounds__(256) update_udvf_kernel(
    const Grid3 g, float *ax, float *ay, float *az, float *bx, float *by, float *bz,
    const float *img, const float *img0, float volume_diff, float flow_diff) {
    for (unsigned id = blockIdx.x * 256 + threadIdx.x; id < g.n; id += gridDim.x * 256) {
        const Vox v = g.at(id);
        const float dfI = img0[id] - img[id];
        const float dfx = fwd_diff(img, id, v, g.nx, g.ny, g.nz, 1);
        const float dfy = fwd_diff(img, id, v, g.nx, g.ny, g.nz, 2);
        const float dfz = fwd_diff(img, id, v, g.nx, g.ny, g.nz, 3);
        const float cax = dfx * volume_diff, cay = dfy * volume_diff, caz = dfz * volume_diff;
        const float cbx = dfx * flow_diff, cby = dfy * flow_diff, cbz = dfz * flow_diff;
        const float w = cax * cax + cay * cay + caz * caz + cbx * cbx + cby * cby + cbz * cbz;
        const float a_x = ay[id], a_y = ax[id], a_z = az[id];
        const float b_x = by[id], b_y = bx[id], b_z = bz[id];
        float b = dfI - cax * a_x - cay * a_y - caz * a_z - cbx * b_x - cby * b_y - cbz * b_z;
        if (w == 0) continue;
        b /= w;
        ax[id] += 1.0f / 6 * b * cax;
        ay[id] += 1.0f / 6 * b * cay;
        az[id] += 1.0f / 6 * b * caz;
        bx[id] += 1.0f / 6 * b * cbx;
        by[id] += 1.0f / 6 * b * cby;
        bz[id] += 1.0f / 6 * b * cbz;
    }
}

// mex_diff.cu:75-113: backward difference, 0 on both faces.
struct DiffOp {
    float *img1;
    const float *img;
    int ind;
    __device__ float value(unsigned id, const Vox &v, const Grid3 &g) const {
        const int i = ind == 1 ? v.ix : ind == 2 ? v.iy : v.iz;
        const int m = ind == 1 ? g.nx : ind == 2 ? g.ny : g.nz;
        const unsigned step = ind == 1 ? 1 : ind == 2 ? g.nx : (unsigned)g.nx * g.ny;
        return (i == m - 1 || i == 0) ? 0.0f : img[id] - img[id - step];
    }
    __device__ void store(unsigned id, float v) const { img1[id] = v; }
};

// --------------------------------------------------------- fused kernels
// z-fastest copy of an x-fastest volume: dst[iz + (ix + iy*nx)*nzp] =
// src[ix + iy*nx + iz*nx*ny], zero for nz <= iz < nzp (zf_pitch).  blockDim
// (32, 8); a block turns a tile of 32 columns of row iy by ZF_Z slices; gridDim
// (ceil(nx/32) * ny, ceil(nz/ZF_Z)).  Eight loads a thread in flight;
// with 32-slice tiles and four, 512x512x256 took 123 us, now 92 (5.8 TB/s), and
// 256x256x160 27, now 24.
constexpr int ZF_Z = 64;
template <typename ST, typename DT>
static __global__ void __launch_bounds__(256) zfast_kernel(DT *dst, const ST *src, int nx, int ny,
                                                           int nz, int nzp) {
    __shared__ float tile[ZF_Z][33];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const unsigned gx = (nx + 31) / 32, iy = blockIdx.x / gx;
    const int x0 = (int)(blockIdx.x - iy * gx) * 32, z0 = blockIdx.y * ZF_Z;
    const int64_t plane = (int64_t)nx * ny, row = (int64_t)iy * nx;
    const int ix = x0 + tx;
    const ST *const p = src + ix + row + (z0 + ty) * plane;
#pragma unroll
    for (int k = 0; k < ZF_Z / 8; k++)
        tile[ty + 8 * k][tx] =
            (ix < nx && z0 + ty + 8 * k < nz) ? ldv(p, 8 * k * plane) : 0.0f;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int lx = ty + 8 * k;
#pragma unroll
        for (int h = 0; h < ZF_Z; h += 32) {
            const int iz = z0 + h + tx;
            if (x0 + lx < nx && iz < nzp) dst[iz + (row + x0 + lx) * nzp] = cvt<DT>(tile[h + tx][lx]);
        }
    }
}
inline dim3 zfast_grid(int nx, int ny, int nz) {
    return dim3(div_up(nx, 32) * (unsigned)ny, div_up(nz, ZF_Z));
}
// The same with a column per thread, for volumes of at most ZF_THIN slices (a
// multiple of 2), which leave most of a tile's threads idle (512x512x4: 19 us,
// this 7.  Grid ceil(nx * ny / 256).
constexpr int ZF_THIN = 8;
template <typename ST, typename DT>
static __global__ void __launch_bounds__(256) zfast_thin_kernel(DT *dst, const ST *src, int plane,
                                                                int nz, int nzp) {
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= plane) return;
    float v[ZF_THIN];
#pragma unroll
    for (int k = 0; k < ZF_THIN; k++) v[k] = k < nz ? ldv(src, c + (int64_t)k * plane) : 0.0f;
#pragma unroll
    for (int k = 0; k < ZF_THIN; k++)
        if (k < nzp) dst[c * nzp + k] = cvt<DT>(v[k]);
}
// The launch of either (not a context's: mcsart_projection_noalloc has none).
template <typename ST, typename DT>
void zfast_launch(cudaStream_t stream, DT *dst, const ST *src, int nx, int ny, int nz, int nzp) {
    if (nz <= ZF_THIN)
        zfast_thin_kernel<ST, DT><<<div_up((int64_t)nx * ny, 256), 256, 0, stream>>>(dst, src, nx * ny,
                                                                                    nz, nzp);
    else
        zfast_kernel<ST, DT><<<zfast_grid(nx, ny, nz), dim3(32, 8), 0, stream>>>(dst, src, nx, ny, nz,
                                                                                nzp);
}
template <typename ST, typename DT>
int zfast(mcsart_ctx *ctx, DT *dst, const ST *src, const Geom &g) {
    if (ctx->profiling) MC_TRY(prof_before(ctx, "zfast_kernel"));
    zfast_launch(ctx->stream, dst, src, g.nx, g.ny, g.nz, g.nzp);
    ctx->launches++;
    MC_TRY(check_launch("zfast_kernel"));
    if (ctx->profiling) MC_TRY(prof_after(ctx));
    ctx->label = nullptr;
    return MCSART_OK;
}

// Loads the 32x32 tile of a field read at the transposed index
// t = iy + ix*ny + iz*nx*ny for the block's (x, y) tile into tile[lx][ly].
template <typename T>
__device__ __forceinline__ void load_tile_T(float (*tile)[33], const T *src, int x0, int y0,
                                            int nx, int ny, int64_t slice) {
    const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int lx = ty + 8 * k, ix = x0 + lx, iy = y0 + tx;
        tile[lx][tx] = (ix < nx && iy < ny) ? ldv(src, iy + (int64_t)ix * ny + slice) : 0.0f;
    }
}

// The DVF pass's per-view kernels work on tiles of MP_T x MP_T (x, y) columns
// and MP_Z slices, one column per thread, so that a thread ends with MP_Z
// consecutive slices of its column, a 32-byte piece of the z-fastest img0 and
// initial2 volumes the projector reads.  16 x 16 columns keep the x-fastest
// rows of the fields in whole 64-byte pieces.
constexpr int MP_T = 16, MP_Z = 4;
inline dim3 motion_grid(int nx, int ny, int nz) {
    return dim3(div_up(nx, MP_T), div_up(ny, MP_T), div_up(nz, MP_Z));
}

// Eight consecutive floats as one 32-byte store (p 32-byte aligned), and
// eight consecutive 16-bit values as one 16-byte store (p 16-byte aligned).
__device__ __forceinline__ void st8(float *p, const float *v) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]),
                 "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}
template <typename T> __device__ __forceinline__ void st8(T *p, const float *v) {
    union {
        T h[8];
        uint4 u;
    } w;
#pragma unroll
    for (int i = 0; i < 8; i++) w.h[i] = cvt<T>(v[i]);
    *reinterpret_cast<uint4 *>(p) = w.u;
}

// Stores slices z0 .. z0 + MP_Z - 1 (those below nzp, zero from nz on) of column
// c: PAIR, img0 and ones interleaved in img0; otherwise apart.  Interleaved
// pairs of a pitch that is a multiple of 4 go out as one store: lanes are different columns,
// so every store of a warp touches 32 lines, and one whole-sector store in
// place of four 8-byte ones takes a quarter of the write transactions.
template <typename VT, bool PAIR>
__device__ __forceinline__ void store_column(VT *img0, VT *ones, int64_t c, int z0, int nz,
                                             int nzp, float *a, float *b) {
    const int64_t i = c * nzp + z0;
#pragma unroll
    for (int k = 0; k < MP_Z; k++)
        if (z0 + k >= nz) a[k] = b[k] = 0.0f;
    if (PAIR && nzp % MP_Z == 0) {
        const float v[8] = {a[0], b[0], a[1], b[1], a[2], b[2], a[3], b[3]};
        st8(img0 + 2 * i, v);
        return;
    }
#pragma unroll
    for (int k = 0; k < MP_Z; k++) {
        if (z0 + k >= nzp) break;
        if (PAIR) {
            stv2(img0, i + k, a[k], b[k]);
        } else {
            img0[i + k] = cvt<VT>(a[k]);
            ones[i + k] = cvt<VT>(b[k]);
        }
    }
}

// AUMISART.cu:252-258 and :267 for slices z0 .. of column (ix, iy): img0 =
// the sum over the six (field, gradient) pairs of F*w*d img in the
// reference's order (host_initial(img0, 0), then six host_add2) and ones =
// (dx + dy + dz img) * (-vd + -fd) (cu_initial.cu:48).  ft[c][k]: the six
// fields' values for slice z0 + k of this column, read at the reference's
// transposed index.
__device__ __forceinline__ void motion_column(const float *img, int ix, int iy, int z0, int nx,
                                              int ny, int nz, float vd, float fd,
                                              const float (*ft)[MP_Z], float *a, float *b) {
    const float s_ones = (-vd) + (-fd);
    const int64_t plane = (int64_t)nx * ny, id = ix + (int64_t)iy * nx + z0 * plane;
    float cur = ldv(img, id);
#pragma unroll
    for (int k = 0; k < MP_Z; k++) {
        if (z0 + k >= nz) break;
        const int64_t i = id + k * plane;
        const float up = z0 + k == nz - 1 ? 0.0f : ldv(img, i + plane);
        // fwd_diff along x, y and z
        const float dfx = ix == nx - 1 ? 0.0f : ldv(img, i + 1) - cur;
        const float dfy = iy == ny - 1 ? 0.0f : ldv(img, i + nx) - cur;
        const float dfz = z0 + k == nz - 1 ? 0.0f : up - cur;
        float s = 0.0f;
        s = __fmaf_rn(ft[0][k] * vd, dfx, s);
        s = __fmaf_rn(ft[1][k] * vd, dfy, s);
        s = __fmaf_rn(ft[2][k] * vd, dfz, s);
        s = __fmaf_rn(ft[3][k] * fd, dfx, s);
        s = __fmaf_rn(ft[4][k] * fd, dfy, s);
        s = __fmaf_rn(ft[5][k] * fd, dfz, s);
        a[k] = s;
        b[k] = (dfx + dfy + dfz) * s_ones;
        cur = up;
    }
}

// Motion pass, AUMISART.cu:252-258 and :267 fused: for the current view the
// img0 and initial2 volumes (motion_column), z-fastest for the projector.
// PAIR: interleaved in img0 (img0[2i], img0[2i + 1]) for the projector's
// paired load, ones unused.  blockDim (MP_T, MP_T), motion_grid.
template <typename FT, typename VT, bool PAIR = false>
static __global__ void __launch_bounds__(256) motion_prep_kernel(VT *img0, VT *ones,
                                                                 const float *img, Fields<FT> f,
                                                                 int nx, int ny, int nz, int nzp,
                                                                 float vd, float fd) {
    __shared__ float sm[6][MP_Z][MP_T][MP_T + 1];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x0 = blockIdx.x * MP_T, y0 = blockIdx.y * MP_T, z0 = blockIdx.z * MP_Z;
    const int64_t plane = (int64_t)nx * ny;
    // the fields at the transposed index iy + ix*ny, lanes along iy
    const bool in_t = x0 + ty < nx && y0 + tx < ny;
    const int64_t it = (y0 + tx) + (int64_t)(x0 + ty) * ny + z0 * plane;
#pragma unroll
    for (int k = 0; k < MP_Z; k++) {
        const bool in = in_t && z0 + k < nz;
        const int64_t i = it + k * plane;
        sm[0][k][ty][tx] = in ? ldv(f.ay, i) : 0.0f;
        sm[1][k][ty][tx] = in ? ldv(f.ax, i) : 0.0f;
        sm[2][k][ty][tx] = in ? ldv(f.az, i) : 0.0f;
        sm[3][k][ty][tx] = in ? ldv(f.by, i) : 0.0f;
        sm[4][k][ty][tx] = in ? ldv(f.bx, i) : 0.0f;
        sm[5][k][ty][tx] = in ? ldv(f.bz, i) : 0.0f;
    }
    __syncthreads();
    const int ix = x0 + tx, iy = y0 + ty;
    if (ix >= nx || iy >= ny) return;
    float ft[6][MP_Z], a[MP_Z], b[MP_Z];
#pragma unroll
    for (int c = 0; c < 6; c++)
#pragma unroll
        for (int k = 0; k < MP_Z; k++) ft[c][k] = sm[c][k][tx][ty];
    motion_column(img, ix, iy, z0, nx, ny, nz, vd, fd, ft, a, b);
    store_column<VT, PAIR>(img0, ones, ix + (int64_t)iy * nx, z0, nz, nzp, a, b);
}

// Motion pass field update, AUMISART.cu:272-277 fused: with q = img_temp read
// at the transposed index, alpha_y += q*nvd*dx img, alpha_x += q*nvd*dy img,
// alpha_z += q*nvd*dz img, and the same for beta with nfd.
template <typename FT>
static __global__ void __launch_bounds__(256) field_update_kernel(FT *ax, FT *ay, FT *az, FT *bx, FT *by,
                                                           FT *bz, const float *img_temp,
                                                           const float *img, int nx, int ny,
                                                           int nz, float nvd, float nfd) {
    __shared__ float qt[32][33];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32, iz = blockIdx.z;
    const int64_t slice = (int64_t)iz * nx * ny;
    load_tile_T(qt, img_temp, x0, y0, nx, ny, slice);
    __syncthreads();
    const int ix = x0 + tx;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int ly = ty + 8 * k, iy = y0 + ly;
        if (ix < nx && iy < ny) {
            const int64_t id = ix + (int64_t)iy * nx + slice;
            const Vox v{ix, iy, iz};
            const float dfx = fwd_diff(img, id, v, nx, ny, nz, 1);
            const float dfy = fwd_diff(img, id, v, nx, ny, nz, 2);
            const float dfz = fwd_diff(img, id, v, nx, ny, nz, 3);
            const float q = qt[tx][ly];
            ay[id] = cvt<FT>(__fmaf_rn(q * nvd, dfx, ldv(ay, id)));
            ax[id] = cvt<FT>(__fmaf_rn(q * nvd, dfy, ldv(ax, id)));
            az[id] = cvt<FT>(__fmaf_rn(q * nvd, dfz, ldv(az, id)));
            by[id] = cvt<FT>(__fmaf_rn(q * nfd, dfx, ldv(by, id)));
            bx[id] = cvt<FT>(__fmaf_rn(q * nfd, dfy, ldv(bx, id)));
            bz[id] = cvt<FT>(__fmaf_rn(q * nfd, dfz, ldv(bz, id)));
        }
    }
}

// field_update_kernel for view v followed by motion_prep_kernel for the next
// view, in one pass over the fields (square slices, nx == ny).  The block of
// output tile A = (x0, y0) updates the fields on the transposed memory tile
// A^T, which is exactly the set motion_prep reads for A, keeps the updated
// values in shared memory and then computes img0 / ones of tile A for the
// next view.  Every field voxel is updated by exactly one block, and the
// arithmetic is that of the two kernels, so the results are bitwise theirs.
// EARLY (a launch shape the driver's tuning may choose): every thread loads
// its MP_Z x 6 field values first, before the ratio tile and its barrier, so
// that 24 loads per thread are in flight at once (more registers, fewer
// resident blocks); otherwise the fields are loaded voxel by voxel.
// PAIR: img0 and ones interleaved, as in motion_prep_kernel.
// BP: the view's backprojection ratio of tile A (the DVF pass's
// host_backprojection and host_division, src/AUMISART.cu:95-100 / :265-270) is
// computed here from `bp` (its (residual, initial2-projection) pairs and
// column data) with the backprojector's own per-voxel code, instead of being
// read from img_temp: the field update of a tile needs the ratio of that tile
// only, so the ratio never goes to memory, and blocks gathering from the
// detector (bound by instruction issue) share the SMs with blocks streaming
// the fields (bound by memory latency).  PROVEN: as in bp_kernel.  The
// ratio's bits are the backprojector kernel's.  blockDim (MP_T, MP_T),
// motion_grid.
template <typename FT, typename VT, bool EARLY = false, bool PAIR = false, bool BP = false,
          bool PROVEN = false>
static __global__ void __launch_bounds__(256) field_update_prep_kernel(
    FT *ax, FT *ay, FT *az, FT *bx, FT *by, FT *bz, const float *img_temp, const float *img,
    int nx, int ny, int nz, int nzp, float nvd, float nfd, VT *img0, VT *ones, float vd, float fd,
    const BPArgs bp) {
    __shared__ float sm[6][MP_Z][MP_T][MP_T + 1];
    __shared__ float rt[MP_Z][MP_T][MP_T + 1];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x0 = blockIdx.x * MP_T, y0 = blockIdx.y * MP_T, z0 = blockIdx.z * MP_Z;
    const int64_t plane = (int64_t)nx * ny;
    if (BP) {
        // The block's own field rows (tile A^T) and volume rows (A^T and A)
        // are prefetched into L2 before the backprojection gather, which
        // then covers their memory latency: rows of MP_T voxels, two per
        // thread (7 x MP_T x MP_Z rows of A^T and MP_T x MP_Z of A).
        const int t = ty * MP_T + tx;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int e = t + 256 * h, w = e / (MP_T * MP_Z), r = e % MP_T, z = z0 + e / MP_T % MP_Z;
            const void *p = nullptr;
            if (z < nz && w < 7 && x0 + r < ny && y0 < nx) {
                const int64_t i = y0 + (int64_t)(x0 + r) * nx + z * plane;
                switch (w) {
                    case 0: p = ax + i; break;
                    case 1: p = ay + i; break;
                    case 2: p = az + i; break;
                    case 3: p = bx + i; break;
                    case 4: p = by + i; break;
                    case 5: p = bz + i; break;
                    default: p = img + i;
                }
            } else if (z < nz && w == 7 && y0 + r < ny && x0 < nx) {
                p = img + x0 + (int64_t)(y0 + r) * nx + z * plane;
            }
            if (p) asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
        }
    }
    // this thread's column of A^T: (xp, yp) = (y0 + tx, x0 + ty)
    const int xp = y0 + tx, yp = x0 + ty;
    const bool in_t = xp < nx && yp < ny;
    const int64_t it = xp + (int64_t)yp * nx + z0 * plane;
    float fe[EARLY ? MP_Z : 1][6];  // its field values (EARLY)
    if (EARLY) {
#pragma unroll
        for (int k = 0; k < MP_Z; k++) {
            const bool in = in_t && z0 + k < nz;
            const int64_t id = in ? it + k * plane : 0;
            fe[k][0] = in ? ldv(ay, id) : 0.0f;
            fe[k][1] = in ? ldv(ax, id) : 0.0f;
            fe[k][2] = in ? ldv(az, id) : 0.0f;
            fe[k][3] = in ? ldv(by, id) : 0.0f;
            fe[k][4] = in ? ldv(bx, id) : 0.0f;
            fe[k][5] = in ? ldv(bz, id) : 0.0f;
        }
    }
    // ratio on tile A: this thread's column (ix, iy), two slices at a time
    const int ix = x0 + tx, iy = y0 + ty;
    const bool in_a = ix < nx && iy < ny;
#pragma unroll 1
    for (int k = 0; k < MP_Z; k += 2) {
        float q[2] = {0.0f, 0.0f};
        if (in_a) {
            if (BP) {
                float a0[2] = {0.0f, 0.0f}, a1[2] = {0.0f, 0.0f};
                if (z0 + k < nz)
                    bp_gather_view<2, PROVEN, 2>(bp, bp.angle, nullptr, bp.pair, ix, iy, z0 + k,
                                                 a0, a1);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    q[h] = a0[h] / a1[h];                           // cu_division.cu:20
                    if (isnan(q[h]) || isinf(q[h])) q[h] = 0.0f;    // :21-24
                }
            } else {
#pragma unroll
                for (int h = 0; h < 2; h++)
                    if (z0 + k + h < nz) q[h] = img_temp[ix + (int64_t)iy * nx + (z0 + k + h) * plane];
            }
        }
        rt[k][ty][tx] = q[0];
        rt[k + 1][ty][tx] = q[1];
    }
    __syncthreads();
    // field update on A^T: voxel (xp, yp)'s q is the ratio at the transposed
    // index, i.e. at (x0 + ty, y0 + tx) of tile A
    if (in_t) {
        float cur = ldv(img, it);
#pragma unroll
        for (int k = 0; k < MP_Z; k++) {
            if (z0 + k >= nz) break;
            const int64_t id = it + k * plane;
            const float up = z0 + k == nz - 1 ? 0.0f : ldv(img, id + plane);
            const float dfx = xp == nx - 1 ? 0.0f : ldv(img, id + 1) - cur;
            const float dfy = yp == ny - 1 ? 0.0f : ldv(img, id + nx) - cur;
            const float dfz = z0 + k == nz - 1 ? 0.0f : up - cur;
            cur = up;
            const float q = rt[k][tx][ty];
            const float fay = EARLY ? fe[k % (EARLY ? MP_Z : 1)][0] : ldv(ay, id);
            const float fax = EARLY ? fe[k % (EARLY ? MP_Z : 1)][1] : ldv(ax, id);
            const float faz = EARLY ? fe[k % (EARLY ? MP_Z : 1)][2] : ldv(az, id);
            const float fby = EARLY ? fe[k % (EARLY ? MP_Z : 1)][3] : ldv(by, id);
            const float fbx = EARLY ? fe[k % (EARLY ? MP_Z : 1)][4] : ldv(bx, id);
            const float fbz = EARLY ? fe[k % (EARLY ? MP_Z : 1)][5] : ldv(bz, id);
            const FT nay = cvt<FT>(__fmaf_rn(q * nvd, dfx, fay));
            const FT nax = cvt<FT>(__fmaf_rn(q * nvd, dfy, fax));
            const FT naz = cvt<FT>(__fmaf_rn(q * nvd, dfz, faz));
            const FT nby = cvt<FT>(__fmaf_rn(q * nfd, dfx, fby));
            const FT nbx = cvt<FT>(__fmaf_rn(q * nfd, dfy, fbx));
            const FT nbz = cvt<FT>(__fmaf_rn(q * nfd, dfz, fbz));
            ay[id] = nay; ax[id] = nax; az[id] = naz;
            by[id] = nby; bx[id] = nbx; bz[id] = nbz;
            sm[0][k][ty][tx] = tof(nay);
            sm[1][k][ty][tx] = tof(nax);
            sm[2][k][ty][tx] = tof(naz);
            sm[3][k][ty][tx] = tof(nby);
            sm[4][k][ty][tx] = tof(nbx);
            sm[5][k][ty][tx] = tof(nbz);
        }
    }
    __syncthreads();
    // motion_prep_kernel for tile A with the next view's weights
    if (!in_a) return;
    float ft[6][MP_Z], a[MP_Z], b[MP_Z];
#pragma unroll
    for (int c = 0; c < 6; c++)
#pragma unroll
        for (int k = 0; k < MP_Z; k++) ft[c][k] = sm[c][k][tx][ty];
    motion_column(img, ix, iy, z0, nx, ny, nz, vd, fd, ft, a, b);
    store_column<VT, PAIR>(img0, ones, ix + (int64_t)iy * nx, z0, nz, nzp, a, b);
}

// Norm ratios ||r_v|| / ||b_v|| from per-block partials (fixed order); one
// warp per view.  Replaces the two cublasSnrm2 calls per view.
static __global__ void norm_finalize_kernel(float *norm_out, const double2 *part, int n_blocks,
                                     const int *views, int n) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= n) return;
    const double2 *p = part + (int64_t)w * n_blocks;
    double sb = 0.0, sr = 0.0;
    for (int i = lane; i < n_blocks; i += 32) {
        sb += p[i].x;
        sr += p[i].y;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        sb += __shfl_down_sync(0xffffffffu, sb, off);
        sr += __shfl_down_sync(0xffffffffu, sr, off);
    }
    if (lane == 0) norm_out[views[w]] = (float)(sqrt(sr) / sqrt(sb));
}

}  // namespace mcsart
