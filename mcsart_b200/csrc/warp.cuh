// 5DCT deformation d(x,t) = a(t) v(x) + b(t) f(x) applied to a volume
// (the reference's host_deform / kernel_forwardDVF / kernel_deformation,
// src/cu_deform.cu:3-47,66-90, and the first-order host_deform2, :49-64,92-113).
//
// The displacement m = alpha*volume + beta*flow is formed in registers
// (kernel_forwardDVF's three scratch volumes and their cudaMalloc/cudaFree per
// call disappear).  The trilinear gather reads either a persistent 3D texture
// (SrcTex: the texture unit's linear filtering, bit-identical to the
// reference, whose filter weights are not plain products of 8-bit fractions)
// or the linear volume in software with FP32 weights (SrcLinear, the EXACT
// model).  The output keeps the reference's in-slice transposed indexing:
// voxel (ix, iy, iz) of the sampling grid is written at iy + ix*ny + iz*nx*ny
// and samples the source at texture coordinates (iy + my, ix + mx, iz + mz)
// + 0.5 (:85-89).
#pragma once

#include <algorithm>

#include "common.cuh"

namespace mcsart {

template <typename FT> struct Fields {
    const FT *ax, *ay, *az, *bx, *by, *bz;
};

// Sample of `src` for output memory index id (any id in [0, nx*ny*nz)).
// The reference indexes the warp's output in-slice transposed
// (cu_deform.cu:82-85): memory position r = x + y*nx of a slice is treated as
// (ix, iy) = (r / ny, r % ny).  For square slices that is (y, x).
__device__ __forceinline__ void warp_coords(int x, int y, int nx, int ny, int &ix, int &iy) {
    if (nx == ny) {
        ix = y;
        iy = x;
    } else {
        const int r = x + y * nx;
        ix = r / ny;
        iy = r - ix * ny;
    }
}

// Sample of voxel id, whose in-slice transposed coordinates are (ix, iy, iz),
// given its field values.
template <typename SRC>
__device__ __forceinline__ float warp_sample_at(const SRC &src, float fax, float fay, float faz,
                                                float fbx, float fby, float fbz, int ix, int iy,
                                                int iz, int nx, int ny, int nz, float volume,
                                                float flow) {
    // kernel_forwardDVF, cu_deform.cu:74-76
    const float mx = fax * volume + fbx * flow;
    const float my = fay * volume + fby * flow;
    const float mz = faz * volume + fbz * flow;
    // kernel_deformation, cu_deform.cu:86-89
    const float xi = iy + 1.0f + my;
    const float yi = ix + 1.0f + mx;
    const float zi = iz + 1.0f + mz;
    return src.fetch(xi - 0.5f, yi - 0.5f, zi - 0.5f, nx, ny, nz);
}

// N consecutive values of a storage type at element i (aligned to N of them)
// as floats, and their store.
template <int N, typename T> __device__ __forceinline__ void ldn(const T *p, int64_t i, float *v) {
    if constexpr (N == 1) {
        v[0] = ldv(p, i);
    } else if constexpr (sizeof(T) == 4) {
        const float4 a = __ldg(reinterpret_cast<const float4 *>(p + i));
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    } else {
        const uint2 a = __ldg(reinterpret_cast<const uint2 *>(p + i));
        union {
            uint2 u;
            T h[4];
        } w;
        w.u = a;
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = tof(w.h[k]);
    }
}
template <int N, typename T> __device__ __forceinline__ void stn(T *p, int64_t i, const float *v) {
    if constexpr (N == 1) {
        p[i] = cvt<T>(v[0]);
    } else if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4 *>(p + i) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
        union {
            uint2 u;
            T h[4];
        } w;
#pragma unroll
        for (int k = 0; k < 4; k++) w.h[k] = cvt<T>(v[k]);
        *reinterpret_cast<uint2 *>(p + i) = w.u;
    }
}

// The warp of N neighbouring voxels (x .. x + N - 1, y, iz), id the first one's
// memory position: the six fields as N-element loads, so that a thread has
// 6 N values in flight before its N dependent gathers.  N = 4 needs rows that
// begin on four elements (warp_vec).
template <int N, typename SRC, typename FT>
__device__ __forceinline__ void warp_sample_n(const SRC &src, const Fields<FT> &f, int64_t id, int x,
                                              int y, int iz, int nx, int ny, int nz, float volume,
                                              float flow, float *out) {
    float a[6][N];
    ldn<N>(f.ax, id, a[0]);
    ldn<N>(f.bx, id, a[3]);
    ldn<N>(f.ay, id, a[1]);
    ldn<N>(f.by, id, a[4]);
    ldn<N>(f.az, id, a[2]);
    ldn<N>(f.bz, id, a[5]);
#pragma unroll
    for (int k = 0; k < N; k++) {
        int ix, iy;
        warp_coords(x + k, y, nx, ny, ix, iy);
        out[k] = warp_sample_at(src, a[0][k], a[1][k], a[2][k], a[3][k], a[4][k], a[5][k], ix, iy, iz,
                                nx, ny, nz, volume, flow);
    }
}

// Whether the warps may take four voxels per thread: rows and arrays begin on
// four elements (16 bytes for FP32, 8 for 16 bits).
template <typename FT>
inline bool warp_vec(int nx, const Fields<FT> &f, const void *p0 = nullptr, const void *p1 = nullptr) {
    const uintptr_t m = 4 * sizeof(FT) - 1;
    const uintptr_t fields = (uintptr_t)f.ax | (uintptr_t)f.ay | (uintptr_t)f.az | (uintptr_t)f.bx |
                             (uintptr_t)f.by | (uintptr_t)f.bz;
    return nx % 4 == 0 && (fields & m) == 0 && (((uintptr_t)p0 | (uintptr_t)p1) & 15) == 0;
}

// Drop-in kernel_deformation.  FT: the fields' and the output's storage type.
// N neighbouring voxels per thread (4 only where warp_vec holds), in memory order
// (Grid3): blocks of 32 * N columns of 8 rows left most lanes idle in narrow
// volumes, and had more blocks along y than a grid takes for ny above 524280.  In a
// chain of launches, such blocks against this, exact weights: 111 and 8.6 us at
// 8x8x20000, 4.8 and 3.3 at 64x64x64, 433 and 402 at 512x512x256.  Grid:
// warp_blocks<N>.
template <int N, typename SRC, typename FT>
static __global__ void __launch_bounds__(256) deform_kernel(FT *out, const SRC src, Fields<FT> f,
                                                            const Grid3 g, float volume,
                                                            float flow) {
    const unsigned id = (blockIdx.x * 256 + threadIdx.x) * N;
    if (id >= g.n) return;
    const Vox p = g.at(id);
    float v[N];
    warp_sample_n<N>(src, f, id, p.ix, p.iy, p.iz, g.nx, g.ny, g.nz, volume, flow, v);
    stn<N>(out, id, v);
}
template <int N> inline unsigned warp_blocks(const Grid3 &g) { return div_up(g.n, 256 * N); }

// Drop-in kernel_forwardDVF (bound by memory; VEC: four voxels per thread, all fields
// read before the first component is stored).
template <bool VEC>
static __global__ void __launch_bounds__(256) forward_dvf_kernel(float *mx, float *my, float *mz,
                                                                 Fields<float> f, int64_t n,
                                                                 float volume, float flow) {
    constexpr int N = VEC ? 4 : 1;
    const int64_t step = (int64_t)gridDim.x * blockDim.x * N;
    auto one = [&](int64_t id) {
        mx[id] = f.ax[id] * volume + f.bx[id] * flow;
        my[id] = f.ay[id] * volume + f.by[id] * flow;
        mz[id] = f.az[id] * volume + f.bz[id] * flow;
    };
    for (int64_t id = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) * N; id < n; id += step) {
        if (VEC && id + 4 <= n) {
            float a[6][4], m[3][4];
            ldn<4>(f.ax, id, a[0]);
            ldn<4>(f.ay, id, a[1]);
            ldn<4>(f.az, id, a[2]);
            ldn<4>(f.bx, id, a[3]);
            ldn<4>(f.by, id, a[4]);
            ldn<4>(f.bz, id, a[5]);
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int k = 0; k < 4; k++) m[c][k] = a[c][k] * volume + a[3 + c][k] * flow;
            stn<4>(mx, id, m[0]);
            stn<4>(my, id, m[1]);
            stn<4>(mz, id, m[2]);
        } else {
            for (int64_t i = id; i < n && i < id + N; i++) one(i);
        }
    }
}
// The displacement as one float4 (mx, my, mz, 0) per voxel, for invert_dvf_kernel.
static __global__ void __launch_bounds__(256) forward_dvf4_kernel(float4 *m, Fields<float> f,
                                                                  int64_t n, float volume,
                                                                  float flow) {
    for (int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; id < n;
         id += (int64_t)gridDim.x * blockDim.x)
        m[id] = make_float4(ldv(f.ax, id) * volume + ldv(f.bx, id) * flow,
                            ldv(f.ay, id) * volume + ldv(f.by, id) * flow,
                            ldv(f.az, id) * volume + ldv(f.bz, id) * flow, 0.0f);
}

// Drop-in host_deform2 (first-order warp).  Neighbour reads that fall past
// the end of the volume (the +nx neighbour of the last rows of the last slice
// under the transposed index) read 0; the reference reads out of bounds there.
// A voxel per thread, in memory order; grid warp_blocks<1>.
static __global__ void __launch_bounds__(256) deform2_kernel(float *out, const float *in,
                                                             Fields<float> f, const Grid3 g,
                                                             float volume, float flow) {
    const unsigned id = blockIdx.x * 256 + threadIdx.x, plane = (unsigned)g.nx * g.ny;
    if (id >= g.n) return;
    const Vox p = g.at(id);
    int ix, iy;
    warp_coords(p.ix, p.iy, g.nx, g.ny, ix, iy);
    const float mx = f.ax[id] * volume + f.bx[id] * flow;
    const float my = f.ay[id] * volume + f.by[id] * flow;
    const float mz = f.az[id] * volume + f.bz[id] * flow;
    const float c = in[id];
    auto at = [&](unsigned j) { return j < g.n ? in[j] : 0.0f; };
    float dx, dy, dz;
    if (ix == g.nx - 1) dx = 0; else dx = at(id + 1) - c;
    if (iy == g.ny - 1) dy = 0; else dy = at(id + g.nx) - c;
    if (p.iz == g.nz - 1) dz = 0; else dz = at(id + plane) - c;
    out[id] = c + dy * mx + dx * my + dz * mz;  // cu_deform.cu:112
}

// The image pass's warps are bound by the latency of each voxel's field loads
// and the dependent texture fetch.  With four voxels per thread (six 16-byte
// loads, four fetches) enough bytes are in flight by themselves; the scalar
// form, for rows that do not begin on four elements, keeps the L2 prefetch of
// the rows of the tile WARP_PREFETCH_AHEAD blocks later in dispatch order.
constexpr int WARP_PREFETCH_AHEAD = 600;
// Slices (warp_fwd) or rows (warp_back_add) per thread: the launch shape the
// driver's tuning may choose; the same bits for every value.
constexpr int WARP_ROWS = 2;

// The prefetch for a block of a grid of 32 x TH tiles (gridDim.x x gridDim.y
// per slice, gridDim.z slices); t = the thread's index in the block.
template <typename FT>
__device__ __forceinline__ void prefetch_tile_rows(const Fields<FT> &f, const float *extra,
                                                   int TH, int nx, int ny, int nz, int t) {
    const int64_t gx = gridDim.x, gy = gridDim.y;
    const int64_t b = blockIdx.x + gx * (blockIdx.y + gy * blockIdx.z) + WARP_PREFETCH_AHEAD;
    if (t >= 7 * TH || b >= gx * gy * gridDim.z) return;
    const int bx = (int)(b % gx), by = (int)((b / gx) % gy), bz = (int)(b / (gx * gy));
    const int a = t / TH, y = by * TH + t % TH, x = bx * 32;
    if (y >= ny || x >= nx || bz >= nz) return;
    const int64_t i = x + (int64_t)y * nx + (int64_t)bz * nx * ny;
    const void *p;
    switch (a) {
        case 0: p = f.ax + i; break;
        case 1: p = f.ay + i; break;
        case 2: p = f.az + i; break;
        case 3: p = f.bx + i; break;
        case 4: p = f.by + i; break;
        case 5: p = f.bz + i; break;
        default: p = extra + i;
    }
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// The prefetch for a block of warp_fwd_kernel's grid of 32 x TZ (x, z) tiles
// (x tiles of row 0, of row 1, ... along gridDim.x, z tiles along gridDim.y).
template <typename FT>
__device__ __forceinline__ void prefetch_xz_rows(const Fields<FT> &f, int TZ, int nx, int ny,
                                                 int nz, int t) {
    const unsigned nxy = gridDim.x;
    unsigned b = blockIdx.x + WARP_PREFETCH_AHEAD, bz = blockIdx.y;
    while (b >= nxy) {  // the tile WARP_PREFETCH_AHEAD blocks later may be in a later z tile row
        b -= nxy;
        bz++;
    }
    if (t >= 6 * TZ) return;
    const unsigned gx = (nx + 31) / 32, y = b / gx;
    const int a = t / TZ, z = (int)bz * TZ + t % TZ, x = (int)(b - y * gx) * 32;
    if (z >= nz) return;
    const int64_t i = x + (int64_t)y * nx + (int64_t)z * nx * ny;
    const void *p;
    switch (a) {
        case 0: p = f.ax + i; break;
        case 1: p = f.ay + i; break;
        case 2: p = f.az + i; break;
        case 3: p = f.bx + i; break;
        case 4: p = f.by + i; break;
        default: p = f.bz + i;
    }
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// SART image pass, forward warp of the current volume into the view's phase,
// z-fastest for the projector: dst[iz + (x + y*nx)*nzp] = warp(src) at memory
// position x + y*nx + iz*nx*ny, stored in VT.
// blockDim (32, 8); a block covers a 32 * N x (8 * WR) (x, z) tile of row y,
// gridDim (ceil(nx/(32*N)) * ny, ceil(nz/(8*WR))).
template <int N, typename SRC, typename FT, typename VT, int WR = WARP_ROWS>
static __global__ void __launch_bounds__(256) warp_fwd_kernel(VT *dst, const SRC src, Fields<FT> f,
                                                              int nx, int ny, int nz, int nzp,
                                                              float volume, float flow) {
    constexpr int TZ = 8 * WR, TX = 32 * N;
    // column c of a row at place(c): with N = 4, 33 apart, so that the lanes'
    // stores of column i, and the turned reads, fall on different banks
    __shared__ float tile[TZ][N == 1 ? 33 : 4 * 33 + 1];
    const auto place = [](int c) { return N == 1 ? c : c % N * 33 + c / N; };
    const int tx = threadIdx.x, ty = threadIdx.y;
    if (N == 1) prefetch_xz_rows(f, TZ, nx, ny, nz, ty * 32 + tx);
    const unsigned gx = (nx + TX - 1) / TX, ym = blockIdx.x / gx;
    const int x0 = (int)(blockIdx.x - ym * gx) * TX, z0 = blockIdx.y * TZ;
    const int64_t plane = (int64_t)nx * ny, row = (int64_t)ym * nx;
    const int xm = x0 + tx * N;
#pragma unroll
    for (int k = 0; k < WR; k++) {
        const int lz = ty + 8 * k, iz = z0 + lz;
        if (xm < nx && iz < nz) {
            float v[N];
            warp_sample_n<N>(src, f, xm + row + iz * plane, xm, (int)ym, iz, nx, ny, nz, volume, flow,
                             v);
#pragma unroll
            for (int i = 0; i < N; i++) tile[lz][place(tx * N + i)] = v[i];
        }
    }
    __syncthreads();
    // turned store: runs of TZ consecutive slices per column
    const int t = ty * 32 + tx;
#pragma unroll
    for (int k = 0; k < WR * N; k++) {
        const int e = t + 256 * k, lx = e / TZ, lz = e % TZ;
        if (x0 + lx < nx && z0 + lz < nzp)
            dst[z0 + lz + (row + x0 + lx) * nzp] =
                cvt<VT>(z0 + lz < nz ? tile[lz][place(lx)] : 0.0f);
    }
}
template <int N, int WR> inline dim3 warp_fwd_grid(int nx, int ny, int nz) {
    return dim3(div_up(nx, 32 * N) * (unsigned)ny, div_up(nz, 8 * WR));
}

// SART image pass, backward warp of the normalised correction and update:
// img[id] += lambda * warp(src)[id]  (AUMISART.cu:222-223).  With a surface,
// the updated voxel is also written to the 3D array the next forward warp
// samples through the texture unit.
// blockDim (32, 8), 32 * N x (8 * WR) tiles of slice blockIdx.z.
template <int N, typename SRC, typename FT, int WR = WARP_ROWS>
static __global__ void __launch_bounds__(256) warp_back_add_kernel(
    float *img, cudaSurfaceObject_t img_surf, const SRC src, Fields<FT> f, int nx, int ny,
    int nz, float volume, float flow, float lambda) {
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int xm = (blockIdx.x * 32 + tx) * N, iz = blockIdx.z;
    const int64_t slice = (int64_t)iz * nx * ny;
    if (N == 1) prefetch_tile_rows(f, img, 8 * WR, nx, ny, nz, ty * 32 + tx);
    if (xm >= nx) return;
#pragma unroll
    for (int k = 0; k < WR; k++) {
        const int ym = blockIdx.y * (8 * WR) + ty + 8 * k;
        if (ym >= ny) break;
        const int64_t id = xm + (int64_t)ym * nx + slice;
        float w[N], v[N];
        ldn<N>(img, id, v);
        warp_sample_n<N>(src, f, id, xm, ym, iz, nx, ny, nz, volume, flow, w);
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = __fmaf_rn(w[i], lambda, v[i]);  // cu_add.cu:17
        stn<N>(img, id, v);
        if (img_surf) {
            if constexpr (N == 4)
                surf3Dwrite(make_float4(v[0], v[1], v[2], v[3]), img_surf, xm * (int)sizeof(float), ym,
                            iz, cudaBoundaryModeZero);
            else
                surf3Dwrite(v[0], img_surf, xm * (int)sizeof(float), ym, iz, cudaBoundaryModeZero);
        }
    }
}

// Inverse of the warp's displacement, for square slices (nx == ny), where
// the reference's warp (cu_deform.cu:79-90) samples memory position
// q = (X, Y, Z) of its source at q + D(q) with D = (my, mx, mz)(q) (the
// in-slice transposed index swaps the first two components).  The inverse
// N(q) = -D(q + N(q)) is found by fixed-point iteration from N = 0 with exact
// FP32 trilinear samples of m (clamped at the edges, as the texture), and
// returned in the forward layout: ox = N_Y, oy = N_X, oz = N_Z, so that a
// warp with displacement (ox, oy, oz) undoes the warp with (mx, my, mz).
// blockDim (32, 8), 32x8 tiles of slice blockIdx.z.
// SRC: the displacement's corners.  DispPacked, as float4 (mx, my, mz, 0) per voxel,
// so that the three components of a corner are one load; DispPlanes, three arrays,
// where there is no memory for the fourth component (688 us against 430 at
// 256x256x160 and 8 steps).
struct DispPacked {
    const float4 *m;
    __device__ __forceinline__ float4 at(int i) const { return __ldg(m + i); }
};
struct DispPlanes {
    const float *x, *y, *z;
    __device__ __forceinline__ float4 at(int i) const {
        return make_float4(__ldg(x + i), __ldg(y + i), __ldg(z + i), 0.0f);
    }
};
__device__ __forceinline__ float lerp8(float t000, float t100, float t010, float t110, float t001,
                                       float t101, float t011, float t111, float a, float b,
                                       float c) {
    // SrcLinear's order: along x, then y, then z
    const float c00 = fmaf(a, t100 - t000, t000), c10 = fmaf(a, t110 - t010, t010);
    const float c01 = fmaf(a, t101 - t001, t001), c11 = fmaf(a, t111 - t011, t011);
    const float c0 = fmaf(b, c10 - c00, c00), c1 = fmaf(b, c11 - c01, c01);
    return fmaf(c, c1 - c0, c0);
}
template <typename SRC>
static __global__ void __launch_bounds__(256) invert_dvf_kernel(float *ox, float *oy, float *oz,
                                                                const SRC m, int nx, int ny,
                                                                int nz, int iters) {
    const int X = blockIdx.x * 32 + threadIdx.x, Y = blockIdx.y * 8 + threadIdx.y, Z = blockIdx.z;
    if (X >= nx || Y >= ny) return;
    float NX = 0.0f, NY = 0.0f, NZ = 0.0f;
    for (int k = 0; k < iters; k++) {
        const float px = (float)X + 0.5f + NX, py = (float)Y + 0.5f + NY, pz = (float)Z + 0.5f + NZ;
        int x0, x1, y0, y1, z0, z1;
        float a, b, c;
        lin_axis(px, nx, x0, x1, a);
        lin_axis(py, ny, y0, y1, b);
        lin_axis(pz, nz, z0, z1, c);
        const int sz = nx * ny;  // fits: volumes hold fewer than 2^31 voxels
        const int r00 = y0 * nx + z0 * sz, r10 = y1 * nx + z0 * sz;
        const int r01 = y0 * nx + z1 * sz, r11 = y1 * nx + z1 * sz;
        const float4 t000 = m.at(r00 + x0), t100 = m.at(r00 + x1), t010 = m.at(r10 + x0),
                     t110 = m.at(r10 + x1), t001 = m.at(r01 + x0), t101 = m.at(r01 + x1),
                     t011 = m.at(r11 + x0), t111 = m.at(r11 + x1);
#define MC_LERP(q) lerp8(t000.q, t100.q, t010.q, t110.q, t001.q, t101.q, t011.q, t111.q, a, b, c)
        // D = (my, mx, mz): the in-slice transposed index swaps the first two
        const float dX = MC_LERP(y), dY = MC_LERP(x), dZ = MC_LERP(z);
#undef MC_LERP
        NX = -dX;
        NY = -dY;
        NZ = -dZ;
    }
    const int64_t id = X + (int64_t)Y * nx + (int64_t)Z * nx * ny;
    ox[id] = NY;
    oy[id] = NX;
    oz[id] = NZ;
}

// warp_back_add_kernel with an explicit displacement (mx, my, mz) instead of
// alpha * volume + beta * flow: img += lambda * src sampled at the warped
// position (square slices).  blockDim (32, 8), 32x32 tiles of slice blockIdx.z.
template <typename SRC>
static __global__ void __launch_bounds__(256) warp_back_add_disp_kernel(
    float *img, cudaSurfaceObject_t img_surf, const SRC src, const float *mx, const float *my,
    const float *mz, int nx, int ny, int nz, float lambda) {
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int xm = blockIdx.x * 32 + tx, iz = blockIdx.z;
    const int64_t slice = (int64_t)iz * nx * ny;
    if (xm >= nx) return;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int ym = blockIdx.y * 32 + ty + 8 * k;
        if (ym >= ny) break;
        const int64_t id = xm + (int64_t)ym * nx + slice;
        int ix, iy;
        warp_coords(xm, ym, nx, ny, ix, iy);
        const float xi = iy + 1.0f + my[id], yi = ix + 1.0f + mx[id], zi = iz + 1.0f + mz[id];
        const float w = src.fetch(xi - 0.5f, yi - 0.5f, zi - 0.5f, nx, ny, nz);
        const float v = __fmaf_rn(w, lambda, img[id]);  // cu_add.cu:17
        img[id] = v;
        if (img_surf)
            surf3Dwrite(v, img_surf, xm * (int)sizeof(float), ym, iz, cudaBoundaryModeZero);
    }
}

}  // namespace mcsart
