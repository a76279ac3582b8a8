// mcsart_backprojection_adjoint: the exact adjoint (transpose) of the engine's
// distance-driven projector (mcsart_projection, the reference's
// kernel_projection, src/cu_projection.cu:7-145).  The reference's own
// backprojector (src/cu_backprojection.cu) is a different operator: it maps
// voxel boundaries onto the detector, while the projector maps detector cell
// boundaries onto slab planes.  A matched pair makes SART's update a true
// gradient step and lets dot-product tests hold.
//
// Deterministic gather, no floating-point atomics.  Per view:
//  1. every ray's geometry (ray_geom): the column's in-plane part and the
//     ray's axial ratios rz0, rz1, stored with its value, rows fastest;
//  2. every column's in-plane footprint per slab (slab_u) and, for each
//     (driving axis, slab, in-plane voxel), the range of columns whose
//     footprint covers it (integer min / max atomics, order-independent);
//  3. per voxel: for the covering columns and the rows whose axial footprint
//     can reach the voxel (the footprint centre is linear in the row), the
//     projector's own weights w_u, w_z, recomputed with the same operations,
//     and acc = fma(p * w_u, w_z, acc) in a fixed order (x-driven columns,
//     then y-driven; columns, then rows, ascending).
#include <climits>

#include "common.cuh"
#include "projector.cuh"

#define MC_EXPORT extern "C" __attribute__((visibility("default")))

namespace mcsart {

// What a column's rows share, for the gather: the centre of row 0's axial ratios
// and its increment per row, half the ratios' distance, and the driving axis.
struct __align__(16) AdjColumn {
    float q0, qs, half;
    int axis;  // 1: x-driven
};
// d_half and src_d (RayGeom) of each driving axis; general: set where some ray is
// not narrow (ray_axial).
struct AdjAxes {
    float d_half[2], src_d[2];
    int general;
};

// A ray for the gather: its axial ratios and its value; RowNarrow, the ratios alone,
// the value read where the projection is (where there is no memory for RowWide).
struct __align__(16) RowWide {
    float rz0, rz1, value, pad;
    __device__ __forceinline__ void set(float a, float b, float v) {
        *reinterpret_cast<float4 *>(this) = make_float4(a, b, v, 0.0f);
    }
};
struct __align__(8) RowNarrow {
    float rz0, rz1;
    __device__ __forceinline__ void set(float a, float b, float) {
        *reinterpret_cast<float2 *>(this) = make_float2(a, b);
    }
};
__device__ __forceinline__ float4 adj_row(const RowWide *row, int ib, const float *, int) {
    return __ldg(reinterpret_cast<const float4 *>(row + ib));
}
__device__ __forceinline__ float4 adj_row(const RowNarrow *row, int ib, const float *proj, int na) {
    const float2 q = __ldg(reinterpret_cast<const float2 *>(row + ib));
    return make_float4(q.x, q.y, __ldg(proj + (int64_t)ib * na), 0.0f);
}

// blockDim (32, 32): 32 x 32 rays, a thread each (four each in 32 x 8 threads took
// 4 us more where the blocks are few), turned through shared memory.
// rows[ib + ia*nb]
template <typename ROW>
static __global__ void __launch_bounds__(1024) adj_rays_kernel(RayGeom *cols, AdjColumn *colz,
                                                               AdjAxes *axes, ROW *rows,
                                                               const float *proj, float angle, Geom g) {
    __shared__ float tile[32][33];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int a0 = blockIdx.x * 32, b0 = blockIdx.y * 32, ib = b0 + tx, ia = a0 + ty;
    if (a0 + tx < g.na && b0 + ty < g.nb) tile[ty][tx] = proj[a0 + tx + (int64_t)(b0 + ty) * g.na];
    __syncthreads();
    if (ib >= g.nb || ia >= g.na) return;
    const float cphi = cosf(angle), sphi = sinf(angle);  // as the projector
    const RayGeom r = ray_geom(cphi, sphi, ia, ib, g);
    rows[ib + (int64_t)ia * g.nb].set(r.rz0, r.rz1, tile[tx][ty]);
    if (!ray_axial(r, (float)(g.nz / 2), g.nz).narrow) axes->general = 1;
    if (ib != 0) return;
    cols[ia] = r;
    const RayGeom l = ray_geom(cphi, sphi, ia, g.nb - 1, g);
    AdjColumn c;
    c.q0 = 0.5f * (r.rz0 + r.rz1);
    c.qs = g.nb > 1 ? (0.5f * (l.rz0 + l.rz1) - c.q0) / (float)(g.nb - 1) : 0.0f;
    c.half = 0.5f * fabsf(r.rz1 - r.rz0);
    c.axis = r.xdrive ? 1 : 0;
    colz[ia] = c;
    if (ia == 0) {
        axes->d_half[1] = __fdiv_rn((float)g.nx, 2.0f);
        axes->d_half[0] = __fdiv_rn((float)g.ny, 2.0f);
        axes->src_d[1] = -__fmul_rn(g.SO, cphi);
        axes->src_d[0] = -__fmul_rn(g.SO, sphi);
    }
}

static __global__ void adj_range_init_kernel(int2 *range, int64_t n, AdjAxes *axes) {
    if (blockIdx.x == 0 && threadIdx.x == 0) axes->general = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        range[i] = make_int2(INT_MAX, -1);
}

// range[(axis * nmax + d) * nmax + u] = (first, last) column covering in-plane
// voxel u of slab d, axis 1 = x-driven columns.
static __global__ void adj_slabs_kernel(const RayGeom *cols, SlabU *slabs, int2 *range, Geom g,
                                        int nmax) {
    const int ia = blockIdx.x * blockDim.x + threadIdx.x, d = blockIdx.y;
    if (ia >= g.na) return;
    const RayGeom r = cols[ia];
    if (d >= r.nd) return;
    const SlabU e = slab_u(r, d);
    slabs[(int64_t)ia * nmax + d] = e;
    const int axis = r.xdrive ? 1 : 0;
    const int u0 = max(0, e.U1), u1 = min(r.nu - 1, e.U2);
    for (int u = u0; u <= u1; u++) {
        int2 *c = range + ((int64_t)axis * nmax + d) * nmax + u;
        atomicMin(&c->x, ia);
        atomicMax(&c->y, ia);
    }
}

// Voxel (x, y, z) of the gather.  NARROW: every ray is (AdjAxes): the axial edges
// are in order, and the branch-free division is exact (ray_axial, fp_pair_staged).
template <bool NARROW, typename ROW>
__device__ __forceinline__ float adj_voxel(const ROW *rows, const float *proj,
                                           const AdjColumn *colz, const AdjAxes &axes, const SlabU *slabs,
                                           const int2 *range, const Geom &g, int nmax, int x, int y,
                                           int z) {
    const float z_half = (float)(g.nz / 2), fz = (float)z;
    const int nb = g.nb;
    float acc = 0.0f;
    for (int axis = 1; axis >= 0; axis--) {
        const int d = axis ? x : y, u = axis ? y : x, nu = axis ? g.ny : g.nx;
        const int2 cr = range[((int64_t)axis * nmax + d) * nmax + u];
        const float dc =
            __fsub_rn(__fsub_rn(__fadd_rn((float)d, 0.5f), axes.d_half[axis]), axes.src_d[axis]);
        for (int ia = cr.x; ia <= cr.y; ia++) {
            const AdjColumn c = colz[ia];
            if (c.axis != axis) continue;
            const SlabU e = slabs[(int64_t)ia * nmax + d];
            if (u < max(0, e.U1) || u > min(nu - 1, e.U2)) continue;
            // the projector's in-plane weight of voxel u (slab_u, fp_slab_general)
            float wu;
            if (e.U2 - e.U1 <= 1) {
                wu = u == e.U1 ? e.a : e.b;
            } else {
                const float ui1 = e.a, ui2 = e.b;
                wu = __fdiv_rn(__fsub_rn(fminf(__fadd_rn((float)u, 1.0f), ui2), fmaxf((float)u, ui1)),
                               __fsub_rn(ui2, ui1));
            }
            // rows whose axial footprint can reach z: its centre c0 + s * row is
            // linear in the row; tol (slices) covers the rounding of these
            // floats and of the ratios (2^-21 of the distance from the centre
            // plane, at most nz/2 within the volume), and every candidate is
            // tested exactly
            int ib_lo = 0, ib_hi = nb - 1;
            const float c0 = c.q0 * dc + z_half, s = c.qs * dc;
            if (fabsf(s) > 1e-6f) {
                const float tol = 1e-3f + 0x1p-18f * (fabsf(c0) + fabsf(s) * (float)nb + z_half);
                const float h = c.half * fabsf(dc) + 0.5f + tol, m = fz + 0.5f - c0, y = 1.0f / s;
                const float ta = (m - h) * y, tb = (m + h) * y;
                const float lo = fminf(ta, tb), hi = fmaxf(ta, tb);
                if (hi < 0.0f || lo > (float)(nb - 1)) continue;
                ib_lo = max(0, (int)ceilf(fmaxf(lo, 0.0f)));
                ib_hi = min(nb - 1, (int)floorf(fminf(hi, (float)(nb - 1))));
            }
            const ROW *const row = rows + (int64_t)ia * nb;
            for (int ib = ib_lo; ib <= ib_hi; ib++) {
                const float4 q = adj_row(row, ib, proj + ia, g.na);
                // the projector's axial footprint (fp_slab_general)
                const float cz0 = __fadd_rn(__fmul_rn(q.x, dc), z_half);
                const float cz1 = __fadd_rn(__fmul_rn(q.y, dc), z_half);
                const float zi1 = NARROW ? cz0 : fminf(cz0, cz1);
                const float zi2 = NARROW ? cz1 : fmaxf(cz0, cz1);
                // floor(zi1) <= z <= floor(zi2)
                const float fz1 = __fadd_rn(fz, 1.0f);
                if (!(zi1 < fz1 && zi2 >= fz)) continue;
                const float n = __fsub_rn(fminf(fz1, zi2), fmaxf(fz, zi1));
                const float dz = __fsub_rn(zi2, zi1);
                const float wz = NARROW ? mk_div(n, dz, mk_recip(dz)) : __fdiv_rn(n, dz);
                acc = __fmaf_rn(__fmul_rn(q.z, wu), wz, acc);
            }
        }
    }
    return acc;
}

// A block is adj_x<ZL>() (or fewer, X) voxel columns of one row y and ZL slices of them; the lanes
// of a warp are the ZL slices of 32 / ZL columns.  The slices of a column share its
// detector columns and their in-plane weights, and neighbouring slices read
// neighbouring rows.  Bound by instruction issue.  With a voxel per thread, lanes
// along x, every lane fetched its own columns and rows: one view of a projector
// and adjoint pair at 256x256x160, 512x384, 909 us, now 394
// (the gather 529, now 267; 240 with the branch-free division).
// Volumes of up to four slices take no more lanes than those along z: 512x512x1
// with a 1024x1 detector 44-46 us by eight, 16-29 by one.
constexpr int ADJ_THREADS = 256;
template <int ZL> constexpr int adj_x() { return ZL >= 8 ? 32 : ADJ_THREADS / ZL; }
// X: the block's columns; with 32 a warp goes through one after another, with 8 (small
// volumes, which do not fill the GPU with such blocks) it has one or two.
template <int ZL, typename ROW, int X>
static __global__ void __launch_bounds__(ADJ_THREADS) adj_gather_kernel(
    float *img, const ROW *rows, const float *proj, const AdjColumn *colz, const AdjAxes *axes, const SlabU *slabs,
    const int2 *range, Geom g, int nmax) {
    constexpr int XL = 32 / ZL, ADJ_X = X;
    __shared__ float tile[ZL][ADJ_X + 1];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const unsigned gx = (g.nx + ADJ_X - 1) / ADJ_X, y = blockIdx.x / gx;
    const int x0 = (int)(blockIdx.x - y * gx) * ADJ_X, zb = blockIdx.y * ZL;
    const int lz = lane % ZL;
    const AdjAxes ax = *axes;
    for (int cx = warp * XL + lane / ZL; cx < ADJ_X; cx += ADJ_THREADS / ZL)
        if (x0 + cx < g.nx && zb + lz < g.nz)
            tile[lz][cx] = ax.general ? adj_voxel<false>(rows, proj, colz, ax, slabs, range, g, nmax,
                                                         x0 + cx, (int)y, zb + lz)
                                      : adj_voxel<true>(rows, proj, colz, ax, slabs, range, g, nmax,
                                                        x0 + cx, (int)y, zb + lz);
    __syncthreads();
    for (int i = t; i < ZL * ADJ_X; i += ADJ_THREADS) {
        const int x = x0 + i % ADJ_X, z = zb + i / ADJ_X;
        if (x < g.nx && z < g.nz)
            img[x + (int64_t)y * g.nx + (int64_t)z * g.nx * g.ny] = tile[i / ADJ_X][i % ADJ_X];
    }
}

// Blocks of 32 columns below which 8 are taken: two an SM (32x32x32: 17-19 and 11 us).
constexpr int ADJ_FEW_BLOCKS = 148 * 2;
template <int ZL, typename ROW, int X = adj_x<ZL>()>
static int launch_adj_gather(mcsart_ctx *ctx, float *img, const ROW *rows, const float *proj,
                             const AdjColumn *colz, const AdjAxes *axes, const SlabU *slabs,
                             const int2 *range, const Geom &g, int nmax) {
    const dim3 grid(div_up(g.nx, X) * (unsigned)g.ny, div_up(g.nz, ZL));
    if constexpr (X == 32)
        if ((int64_t)grid.x * grid.y < ADJ_FEW_BLOCKS)
            return launch_adj_gather<ZL, ROW, 8>(ctx, img, rows, proj, colz, axes, slabs, range, g, nmax);
    MC_LAUNCH(ctx, (adj_gather_kernel<ZL, ROW, X>), grid, ADJ_THREADS, 0, img, rows, proj, colz, axes,
              slabs, range, g, nmax);
    return MCSART_OK;
}

// The passes of a view, with the scratch laid out.
template <typename ROW>
static int launch_adjoint(mcsart_ctx *ctx, float *img, const float *proj, float angle, const Geom &g,
                          RayGeom *cols, AdjColumn *colz, AdjAxes *axes, ROW *rows, SlabU *slabs,
                          int2 *range) {
    const int nx = g.nx, ny = g.ny, nz = g.nz, na = g.na, nb = g.nb, nmax = std::max(nx, ny);
    const int64_t n_range = 2LL * nmax * nmax;
    MC_LAUNCH(ctx, adj_range_init_kernel, (unsigned)std::min<int64_t>(div_up(n_range, 256), 4096),
              256, 0, range, n_range, axes);
    MC_LAUNCH(ctx, adj_rays_kernel<ROW>, dim3(div_up(na, 32), div_up(nb, 32)), dim3(32, 32), 0, cols, colz,
              axes, rows, proj, angle, g);
    MC_LAUNCH(ctx, adj_slabs_kernel, dim3(div_up(na, 128), nmax), 128, 0, cols, slabs, range, g,
              nmax);
    // 32 slices a warp, 8 where a quarter or more of its lanes would have none, as
    // many as there are below that
    if (nz == 1)
        MC_TRY(launch_adj_gather<1>(ctx, img, rows, proj, colz, axes, slabs, range, g, nmax));
    else if (nz == 2)
        MC_TRY(launch_adj_gather<2>(ctx, img, rows, proj, colz, axes, slabs, range, g, nmax));
    else if (nz <= 4)
        MC_TRY(launch_adj_gather<4>(ctx, img, rows, proj, colz, axes, slabs, range, g, nmax));
    else if (div_up(nz, 32) * 32 - nz < nz / 4)
        MC_TRY(launch_adj_gather<32>(ctx, img, rows, proj, colz, axes, slabs, range, g, nmax));
    else
        MC_TRY(launch_adj_gather<8>(ctx, img, rows, proj, colz, axes, slabs, range, g, nmax));
    return MCSART_OK;
}

}  // namespace mcsart

using namespace mcsart;

MC_EXPORT int mcsart_backprojection_adjoint(mcsart_ctx *ctx, float *d_img, const float *d_proj,
                                            float angle, float SO, float SD, float da, int na,
                                            float ai, float db, int nb, float bi, int nx, int ny,
                                            int nz) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_REQUIRE(d_proj && d_img, "d_proj and d_img must be non-NULL");
    Geom g;
    g.SO = SO; g.SD = SD; g.da = da; g.ai = ai; g.db = db; g.bi = bi;
    g.na = na; g.nb = nb; g.nx = nx; g.ny = ny; g.nz = nz;
    MC_TRY(validate_geom(g));
    const int nmax = std::max(nx, ny);
    void *w_cols, *w_rows, *w_slabs, *w_range;
    // the columns' tables in one workspace
    MC_TRY(workspace(ctx, "adj_cols",
                     (size_t)na * (sizeof(AdjColumn) + sizeof(RayGeom)) + sizeof(AdjAxes), &w_cols));
    MC_TRY(workspace(ctx, "adj_slabs", (size_t)na * nmax * sizeof(SlabU), &w_slabs));
    const int64_t n_range = 2LL * nmax * nmax;
    MC_TRY(workspace(ctx, "adj_range", (size_t)n_range * sizeof(int2), &w_range));
    int rc = workspace(ctx, "adj_rows", (size_t)na * nb * sizeof(RowWide), &w_rows);
    const bool narrow = rc == MCSART_ERR_OUT_OF_MEMORY;
    if (narrow) {
        (void)cudaGetLastError();
        clear_error();
        rc = workspace(ctx, "adj_rows", (size_t)na * nb * sizeof(RowNarrow), &w_rows);
    }
    MC_TRY(rc);
    AdjColumn *colz = (AdjColumn *)w_cols;
    RayGeom *cols = (RayGeom *)(colz + na);
    AdjAxes *axes = (AdjAxes *)(cols + na);
    SlabU *slabs = (SlabU *)w_slabs;
    int2 *range = (int2 *)w_range;
    if (narrow)
        MC_TRY(launch_adjoint(ctx, d_img, d_proj, angle, g, cols, colz, axes, (RowNarrow *)w_rows, slabs,
                              range));
    else
        MC_TRY(launch_adjoint(ctx, d_img, d_proj, angle, g, cols, colz, axes, (RowWide *)w_rows, slabs,
                              range));
    return finish(ctx, "mcsart_backprojection_adjoint");
}
