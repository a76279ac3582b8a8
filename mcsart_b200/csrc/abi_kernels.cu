// Kernel-level C ABI: one entry point per reference launcher (include/mcsart.h).
#include <algorithm>
#include <cmath>
#include <initializer_list>

#include "backprojector.cuh"
#include "common.cuh"
#include "elementwise.cuh"
#include "projector.cuh"
#include "sart.cuh"
#include "warp.cuh"

#define MC_EXPORT extern "C" __attribute__((visibility("default")))

namespace mcsart {

// Slab groups per ray: enough warps for ~4 waves of 48 warps on 148 SMs,
// at least 8 slabs per group, at most 8 groups.
int fp_auto_groups(int64_t ray_blocks, int n_slabs) {
    const int64_t target = 148LL * 48 * 2;
    int s = 1;
    while (s < 8 && ray_blocks * s < target && n_slabs / (2 * s) >= 8) s *= 2;
    return s;
}

template <int K>
int launch_fp_plain(mcsart_ctx *ctx, float *d_proj, const float *d_imgZ, float angle,
                    const float *d_angles, int n_views, const Geom &g) {
    FPArgs<float, K> a{};
    a.vol.zf[0] = d_imgZ;
    a.g = g;
    a.angle = angle;
    a.angles = d_angles;
    a.mode = FP_PLAIN;
    a.out = d_proj;
    // the reference's summation order: bitwise the reference kernel's output
    const dim3 grid(div_up(g.na, FPC_COLS), div_up(g.nb, FPC_ROWS), n_views);
    // several views (mcsart_projection_views): the multi-view instantiation
    if (n_views > 1) return launch_fp_ref<K, false, float, float, true>(ctx, grid, a);
    return launch_fp_ref<K, false, float>(ctx, grid, a);
}

// The z-fastest copy of a volume the projector reads, in a workspace; in a
// captured call in memory of the graph's own (*owned, given back by zfast_free
// behind the projector), so that the graph keeps no address that a later call
// may give back and a first call can be captured.
template <typename VT>
int zfast_copy(mcsart_ctx *ctx, const char *name, const VT *src, const Geom &g, const VT **out,
               void **owned) {
    const size_t bytes = nvox(g.nx, g.ny, g.nzp) * sizeof(VT);
    void *ws;
    *owned = nullptr;
    if (capturing(ctx->stream)) {
        MC_CHECK_CUDA(cudaMallocAsync(&ws, bytes, ctx->stream));
        *owned = ws;
    } else {
        MC_TRY(workspace(ctx, name, bytes, &ws));
    }
    MC_TRY(zfast(ctx, (VT *)ws, src, g));
    *out = (const VT *)ws;
    return MCSART_OK;
}

int zfast_free(mcsart_ctx *ctx, void *owned) {
    if (owned) MC_CHECK_CUDA(cudaFreeAsync(owned, ctx->stream));
    return MCSART_OK;
}

unsigned stream_blocks(int64_t n) {
    const int64_t b = (n + 255) / 256;
    return (unsigned)std::min<int64_t>(b, 148LL * 16);
}

// Whether every array begins on 16 bytes (four elements per load and store).
static bool aligned16(std::initializer_list<const void *> ptrs) {
    for (const void *p : ptrs)
        if ((uintptr_t)p % 16 != 0) return false;
    return true;
}
// Blocks of a pointwise kernel over n elements.
static unsigned pointwise_blocks(int64_t n, bool vec) { return stream_blocks(vec ? (n + 3) / 4 : n); }

}  // namespace mcsart

using namespace mcsart;

static Geom make_geom(float SO, float SD, float da, int na, float ai, float db, int nb, float bi,
                      int nx, int ny, int nz) {
    Geom g;
    g.SO = SO; g.SD = SD; g.da = da; g.ai = ai; g.db = db; g.bi = bi;
    g.na = na; g.nb = nb; g.nx = nx; g.ny = ny; g.nz = nz;
    g.nzp = zf_pitch(nx, ny, nz);
    return g;
}

MC_EXPORT int mcsart_projection(mcsart_ctx *ctx, float *d_proj, const float *d_img, float angle,
                                float SO, float SD, float da, int na, float ai, float db, int nb,
                                float bi, int nx, int ny, int nz) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_REQUIRE(d_proj && d_img, "d_proj and d_img must be non-NULL");
    const Geom g = make_geom(SO, SD, da, na, ai, db, nb, bi, nx, ny, nz);
    MC_TRY(validate_geom(g));
    const float *imgZ;
    void *owned;
    const int rc = zfast_copy(ctx, "fp_volZ", d_img, g, &imgZ, &owned);
    if (rc == MCSART_ERR_OUT_OF_MEMORY) {
        (void)cudaGetLastError();
        clear_error();
        MC_LAUNCH(ctx, fp_nocopy_kernel, dim3(div_up(na, 128), nb), 128, 0, d_proj, d_img, angle, g);
        return finish(ctx, "mcsart_projection");
    }
    MC_TRY(rc);
    MC_TRY(launch_fp_plain<1>(ctx, d_proj, imgZ, angle, nullptr, 1, g));
    MC_TRY(zfast_free(ctx, owned));
    return finish(ctx, "mcsart_projection");
}

MC_EXPORT int mcsart_projection_views(mcsart_ctx *ctx, float *d_proj, const float *d_img,
                                      const float *h_angles, int n_views, float SO, float SD,
                                      float da, int na, float ai, float db, int nb, float bi,
                                      int nx, int ny, int nz) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_REQUIRE(d_proj && d_img && h_angles, "d_proj, d_img and h_angles must be non-NULL");
    MC_REQUIRE(n_views > 0 && n_views <= 65535, "n_views must be in [1, 65535]");
    const Geom g = make_geom(SO, SD, da, na, ai, db, nb, bi, nx, ny, nz);
    MC_TRY(validate_geom(g));
    void *wsA;
    const float *imgZ;
    MC_TRY(workspace(ctx, "fp_angles", (size_t)n_views * sizeof(float), &wsA));
    MC_CHECK_CUDA(cudaMemcpyAsync(wsA, h_angles, (size_t)n_views * sizeof(float),
                                  cudaMemcpyHostToDevice, ctx->stream));
    void *owned;
    MC_TRY(zfast_copy(ctx, "fp_volZ", d_img, g, &imgZ, &owned));
    MC_TRY(launch_fp_plain<1>(ctx, d_proj, imgZ, 0.0f, (const float *)wsA, n_views, g));
    MC_TRY(zfast_free(ctx, owned));
    // the angle staging buffer must outlive the launch before the host array is reused
    MC_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
    return finish(ctx, "mcsart_projection_views");
}

// Scratch of the slice-lane backprojector, or none where there is no memory for
// it or the stream is being captured (a graph must not keep an address that a
// later call may give back): bp_kernel needs none.
static int bp_cells_workspace(mcsart_ctx *ctx, const Geom &g, float **cells) {
    if (capturing(ctx->stream)) return MCSART_OK;
    void *ws = nullptr;
    const int rc = workspace(ctx, "bp_cells", bp_cells(g.na, g.nb) * sizeof(float), &ws);
    if (rc == MCSART_ERR_OUT_OF_MEMORY) {
        (void)cudaGetLastError();
        clear_error();
        return MCSART_OK;
    }
    *cells = (float *)ws;
    return rc;
}

MC_EXPORT int mcsart_backprojection(mcsart_ctx *ctx, float *d_img, const float *d_proj,
                                    float angle, float SO, float SD, float da, int na, float ai,
                                    float db, int nb, float bi, int nx, int ny, int nz) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_REQUIRE(d_proj && d_img, "d_proj and d_img must be non-NULL");
    const Geom g = make_geom(SO, SD, da, na, ai, db, nb, bi, nx, ny, nz);
    MC_TRY(validate_geom(g));
    const bool proven = bp_geom_proven(g);
    float *cells = nullptr;
    if (nvox(nx, ny, nz) >= BP_SLICE_LANES_MIN) MC_TRY(bp_cells_workspace(ctx, g, &cells));
    if (cells != nullptr) {
        MC_LAUNCH(ctx, bp_cells_kernel, dim3(div_up(na, 32), div_up(nb, 32)), dim3(32, 8), 0, cells,
                  d_proj, na, nb);
        // 16 slices per tile where the last 32 would be at most half full
        if ((nz - 1) % 32 < 16)
            MC_LAUNCH(ctx, (proven ? &bp_slice_kernel<true, 16> : &bp_slice_kernel<false, 16>),
                      bp_slice_grid<16>(g), BP_THREADS, 0, d_img, cells, angle, g);
        else
            MC_LAUNCH(ctx, (proven ? &bp_slice_kernel<true, 32> : &bp_slice_kernel<false, 32>),
                      bp_slice_grid<32>(g), BP_THREADS, 0, d_img, cells, angle, g);
        return finish(ctx, "mcsart_backprojection");
    }
    BPArgs a{};
    a.proj = d_proj;
    a.g = g;
    a.angle = angle;
    a.out = d_img;
    const dim3 grid = bp_grid<BP_NZ, BP_ROWS>(g, BP_PLAIN), block(32, BP_ROWS);
    if (proven)
        MC_LAUNCH(ctx, (bp_kernel<1, BP_PLAIN, false, true>), grid, block, 0, a);
    else
        MC_LAUNCH(ctx, (bp_kernel<1, BP_PLAIN>), grid, block, 0, a);
    return finish(ctx, "mcsart_backprojection");
}

// The warp of a volume given as a texture or in memory: four voxels per thread
// where rows and arrays allow (warp_vec).
template <typename SRC, typename FT>
static int launch_deform(mcsart_ctx *ctx, FT *out, const SRC &src, const Fields<FT> &f, int nx,
                         int ny, int nz, float volume, float flow) {
    const Grid3 g(nx, ny, nz);
    if (warp_vec(nx, f) && (uintptr_t)out % (4 * sizeof(FT)) == 0)
        MC_LAUNCH(ctx, (deform_kernel<4, SRC, FT>), warp_blocks<4>(g), 256, 0, out, src, f, g, volume,
                  flow);
    else
        MC_LAUNCH(ctx, (deform_kernel<1, SRC, FT>), warp_blocks<1>(g), 256, 0, out, src, f, g, volume,
                  flow);
    return MCSART_OK;
}

static int deform_common(mcsart_ctx *ctx, bool first_order, float *d_img1, const float *d_img,
                         int nx, int ny, int nz, float volume, float flow, const float *ax,
                         const float *ay, const float *az, const float *bx, const float *by,
                         const float *bz) {
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(d_img1 && d_img && ax && ay && az && bx && by && bz,
               "volume and field pointers must be non-NULL");
    const int64_t n = nvox(nx, ny, nz);
    const Fields<float> f{ax, ay, az, bx, by, bz};
    if (!first_order && ctx->interp == MCSART_INTERP_TEXTURE) {
        // the reference samples a texture over a copy of the input
        // (cu_deform.cu:13-38); here the 3D array persists across calls
        if (!ctx->driver) ctx->driver.reset(new DriverState());
        TexVol &tv = ctx->driver->tv_deform;
        MC_TRY(scratch_begin(ctx));
        MC_TRY(tv.ensure(nx, ny, nz));
        MC_TRY(tv.upload(d_img, ctx->stream));
        return launch_deform(ctx, d_img1, SrcTex{tv.tex}, f, nx, ny, nz, volume, flow);
    }
    const float *src = d_img;
    if (d_img1 == d_img) {  // the reference samples a copy (cu_deform.cu:13-23)
        void *ws;
        MC_TRY(workspace(ctx, "deform_src", n * sizeof(float), &ws));
        MC_CHECK_CUDA(cudaMemcpyAsync(ws, d_img, n * sizeof(float), cudaMemcpyDeviceToDevice,
                                      ctx->stream));
        src = (const float *)ws;
    }
    if (first_order) {
        const Grid3 g(nx, ny, nz);
        MC_LAUNCH(ctx, deform2_kernel, warp_blocks<1>(g), 256, 0, d_img1, src, f, g, volume, flow);
        return MCSART_OK;
    }
    return launch_deform(ctx, d_img1, SrcLinear<float>{src}, f, nx, ny, nz, volume, flow);
}

MC_EXPORT int mcsart_deform(mcsart_ctx *ctx, float *d_img1, const float *d_img, int nx, int ny,
                            int nz, float volume, float flow, const float *ax, const float *ay,
                            const float *az, const float *bx, const float *by, const float *bz) {
    clear_error();
    MC_TRY(deform_common(ctx, false, d_img1, d_img, nx, ny, nz, volume, flow, ax, ay, az, bx, by,
                         bz));
    return finish(ctx, "mcsart_deform");
}

MC_EXPORT int mcsart_deform2(mcsart_ctx *ctx, float *d_img1, const float *d_img, int nx, int ny,
                             int nz, float volume, float flow, const float *ax, const float *ay,
                             const float *az, const float *bx, const float *by, const float *bz) {
    clear_error();
    MC_TRY(deform_common(ctx, true, d_img1, d_img, nx, ny, nz, volume, flow, ax, ay, az, bx, by,
                         bz));
    return finish(ctx, "mcsart_deform2");
}

MC_EXPORT int mcsart_forward_dvf(mcsart_ctx *ctx, float *mx, float *my, float *mz,
                                 const float *ax, const float *ay, const float *az,
                                 const float *bx, const float *by, const float *bz, float volume,
                                 float flow, int nx, int ny, int nz) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(mx && my && mz && ax && ay && az && bx && by && bz, "pointers must be non-NULL");
    const int64_t n = nvox(nx, ny, nz);
    const Fields<float> f{ax, ay, az, bx, by, bz};
    // (a component computed in place of a later one's field is read back there, as
    // the reference's kernel does, voxel by voxel)
    const bool shared = mx == ay || mx == by || mx == az || mx == bz || my == az || my == bz;
    const bool vec = !shared && aligned16({mx, my, mz, ax, ay, az, bx, by, bz});
    MC_LAUNCH(ctx, (vec ? &forward_dvf_kernel<true> : &forward_dvf_kernel<false>),
              pointwise_blocks(n, vec), 256, 0, mx, my, mz, f, n, volume, flow);
    return finish(ctx, "mcsart_forward_dvf");
}

MC_EXPORT int mcsart_invert_dvf(mcsart_ctx *ctx, float *inv_x, float *inv_y, float *inv_z,
                                const float *ax, const float *ay, const float *az,
                                const float *bx, const float *by, const float *bz, float volume,
                                float flow, int nx, int ny, int nz, int n_iter) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(inv_x && inv_y && inv_z && ax && ay && az && bx && by && bz,
               "pointers must be non-NULL");
    MC_REQUIRE(nx == ny, "the warp is a displacement field only for square slices (nx == ny)");
    MC_REQUIRE(n_iter >= 1 && n_iter <= 64, "n_iter must be in [1, 64]");
    const int64_t n = nvox(nx, ny, nz);
    const Fields<float> f{ax, ay, az, bx, by, bz};
    const dim3 grid(div_up(nx, 32), div_up(ny, 8), nz), block(32, 8);
    void *ws;
    const int rc = workspace(ctx, "inv_m", n * sizeof(float4), &ws);
    if (rc == MCSART_ERR_OUT_OF_MEMORY) {
        (void)cudaGetLastError();
        clear_error();
        MC_TRY(workspace(ctx, "inv_m", n * 3 * sizeof(float), &ws));
        float *const m = (float *)ws;
        MC_LAUNCH(ctx, forward_dvf_kernel<false>, stream_blocks(n), 256, 0, m, m + n, m + 2 * n, f, n,
                  volume, flow);
        MC_LAUNCH(ctx, invert_dvf_kernel, grid, block, 0, inv_x, inv_y, inv_z,
                  (DispPlanes{m, m + n, m + 2 * n}), nx, ny, nz, n_iter);
        return finish(ctx, "mcsart_invert_dvf");
    }
    MC_TRY(rc);
    float4 *m = (float4 *)ws;
    MC_LAUNCH(ctx, forward_dvf4_kernel, stream_blocks(n), 256, 0, m, f, n, volume, flow);
    MC_LAUNCH(ctx, invert_dvf_kernel, grid, block, 0, inv_x, inv_y, inv_z, DispPacked{m}, nx, ny, nz,
              n_iter);
    return finish(ctx, "mcsart_invert_dvf");
}

MC_EXPORT int mcsart_add(mcsart_ctx *ctx, float *img1, const float *img, int nx, int ny, int nz,
                         float weight) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(img1 && img, "pointers must be non-NULL");
    const int64_t n = nvox(nx, ny, nz);
    const bool vec = aligned16({img1, img});
    MC_LAUNCH(ctx, (vec ? &add_kernel<true> : &add_kernel<false>), pointwise_blocks(n, vec), 256, 0,
              img1, img, n, weight);
    return finish(ctx, "mcsart_add");
}

MC_EXPORT int mcsart_add2(mcsart_ctx *ctx, float *img1, const float *img, int nx, int ny, int nz,
                          const float *img0, float weight, int ind) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(img1 && img && img0, "pointers must be non-NULL");
    MC_REQUIRE(ind >= 1 && ind <= 3, "ind must be 1, 2 or 3 (got %d)", ind);
    const Grid3 g(nx, ny, nz);
    if (nx >= ADD2_TILE_MIN && ny >= ADD2_TILE_MIN && g.n > ADD2_ROWS_MAX) {
        MC_LAUNCH(ctx, add2_kernel, add2_grid(nx, ny, nz), dim3(32, 8), 0, img1, img, nx, ny, nz,
                  img0, weight, ind);
    } else {
        MC_TRY(launch_stencil(ctx, "add2_kernel", g, Add2Op{img1, img, img0, weight, ind}));
    }
    return finish(ctx, "mcsart_add2");
}

MC_EXPORT int mcsart_initial(mcsart_ctx *ctx, float *img, int nx, int ny, int nz, float value) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(img, "img must be non-NULL");
    const int64_t n = nvox(nx, ny, nz);
    const bool vec = aligned16({img});
    MC_LAUNCH(ctx, (vec ? &initial_kernel<true> : &initial_kernel<false>), pointwise_blocks(n, vec), 256, 0,
              img, n, value);
    return finish(ctx, "mcsart_initial");
}

MC_EXPORT int mcsart_initial2(mcsart_ctx *ctx, float *img, int nx, int ny, int nz,
                              const float *img0, float volume, float flow) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(img && img0, "pointers must be non-NULL");
    MC_TRY(launch_stencil(ctx, "initial2_kernel", Grid3(nx, ny, nz), Initial2Op{img, img0, volume + flow}));
    return finish(ctx, "mcsart_initial2");
}

MC_EXPORT int mcsart_division(mcsart_ctx *ctx, float *img1, const float *img, int nx, int ny,
                              int nz) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(img1 && img, "pointers must be non-NULL");
    const int64_t n = nvox(nx, ny, nz);
    const bool vec = aligned16({img1, img});
    MC_LAUNCH(ctx, (vec ? &division_kernel<true> : &division_kernel<false>), pointwise_blocks(n, vec), 256, 0,
              img1, img, n);
    return finish(ctx, "mcsart_division");
}

MC_EXPORT int mcsart_multiple(mcsart_ctx *ctx, float *img1, int nx, int ny, int nz,
                              const float *img0, float weight, int ind) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(img1 && img0, "pointers must be non-NULL");
    MC_REQUIRE(ind >= 1 && ind <= 3, "ind must be 1, 2 or 3 (got %d)", ind);
    MC_TRY(launch_stencil(ctx, "multiple_kernel", Grid3(nx, ny, nz), MultipleOp{img1, img0, weight, ind}));
    return finish(ctx, "mcsart_multiple");
}

MC_EXPORT int mcsart_update_udvf(mcsart_ctx *ctx, float *ax, float *ay, float *az, float *bx,
                                 float *by, float *bz, const float *img, const float *img0,
                                 float volume_diff, float flow_diff, int nx, int ny, int nz,
                                 int iter) {
    clear_error();
    (void)iter;  // unused by the reference kernel too (cu_update_udvf.cu:11)
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(ax && ay && az && bx && by && bz && img && img0, "pointers must be non-NULL");
    const Grid3 g(nx, ny, nz);
    MC_LAUNCH(ctx, update_udvf_kernel, stream_blocks(g.n), 256, 0, g, ax, ay, az, bx, by, bz, img, img0,
              volume_diff, flow_diff);
    return finish(ctx, "mcsart_update_udvf");
}

MC_EXPORT int mcsart_diff(mcsart_ctx *ctx, float *img1, const float *img, int nx, int ny, int nz,
                          int ind) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(img1 && img, "pointers must be non-NULL");
    MC_REQUIRE(ind >= 1 && ind <= 3, "ind must be 1, 2 or 3 (got %d)", ind);
    MC_TRY(launch_stencil(ctx, "diff_kernel", Grid3(nx, ny, nz), DiffOp{img1, img, ind}));
    return finish(ctx, "mcsart_diff");
}

namespace mcsart {
__global__ void sumsq_kernel(const float *x, int64_t n, double *part) {
    double s = 0.0;
    MC_GRID_STRIDE(n) { s += (double)x[id] * (double)x[id]; }
    __shared__ double red[8];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
        part[blockIdx.x] = t;
    }
}
}  // namespace mcsart

MC_EXPORT int mcsart_snrm2(mcsart_ctx *ctx, int n, const float *d_x, float *h_result) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_REQUIRE(n >= 0 && h_result, "n must be >= 0 and h_result non-NULL");
    if (n == 0) {
        *h_result = 0.0f;
        return MCSART_OK;
    }
    MC_REQUIRE(d_x, "d_x must be non-NULL");
    const unsigned blocks = std::min<unsigned>(div_up(n, 256), 1184u);
    void *ws;
    MC_TRY(workspace(ctx, "snrm2", blocks * sizeof(double), &ws));
    MC_LAUNCH(ctx, sumsq_kernel, blocks, 256, 0, d_x, (int64_t)n, (double *)ws);
    double host[1184];
    MC_CHECK_CUDA(cudaMemcpyAsync(host, ws, blocks * sizeof(double), cudaMemcpyDeviceToHost,
                                  ctx->stream));
    MC_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
    double s = 0.0;
    for (unsigned i = 0; i < blocks; i++) s += host[i];
    *h_result = (float)sqrt(s);
    return MCSART_OK;
}

// ------------------------------------------------- mixed-precision kernels
namespace {

template <typename VT>
int projection_ex_launch(mcsart_ctx *ctx, float *d_proj, const VT *zf, int fp_sum, int geom64,
                         float angle, const Geom &g) {
    FPArgs<VT, 1, VT> a{};
    a.vol.zf[0] = zf;
    a.g = g;
    a.angle = angle;
    a.mode = FP_PLAIN;
    a.out = d_proj;
    if (fp_sum == SUM_REF)
        return launch_fp_ref<1, false, VT>(
            ctx, dim3(div_up(g.na, FPC_COLS), div_up(g.nb, FPC_ROWS), 1), a);
    a.cos64 = cos((double)angle);
    a.sin64 = sin((double)angle);
    const int groups = fp_auto_groups((int64_t)div_up(g.na, 32) * g.nb, std::max(g.nx, g.ny));
    return fp_sum == SUM_PLAIN ? launch_fp_split<1, false, SUM_PLAIN>(ctx, groups, geom64 != 0, a)
                               : launch_fp_split<1, false, SUM_KAHAN>(ctx, groups, geom64 != 0, a);
}

template <typename VT>
int projection_ex_typed(mcsart_ctx *ctx, float *d_proj, const VT *d_img, int fp_sum, int geom64,
                        float angle, const Geom &g) {
    const VT *zf;
    void *owned;
    MC_TRY(zfast_copy(ctx, "fp_volZ_ex", d_img, g, &zf, &owned));
    MC_TRY(projection_ex_launch(ctx, d_proj, zf, fp_sum, geom64, angle, g));
    return zfast_free(ctx, owned);
}

template <typename FT>
int deform_ex_typed(mcsart_ctx *ctx, FT *d_img1, const float *d_img, int nx, int ny, int nz,
                    float volume, float flow, const FT *fields, int interp) {
    const int64_t V = nvox(nx, ny, nz);
    const Fields<FT> f{fields, fields + V, fields + 2 * V, fields + 3 * V, fields + 4 * V,
                       fields + 5 * V};
    if (interp == MCSART_INTERP_TEXTURE) {
        if (!ctx->driver) ctx->driver.reset(new DriverState());
        TexVol &tv = ctx->driver->tv_deform;
        MC_TRY(scratch_begin(ctx));
        MC_TRY(tv.ensure(nx, ny, nz));
        MC_TRY(tv.upload(d_img, ctx->stream));
        return launch_deform(ctx, d_img1, SrcTex{tv.tex}, f, nx, ny, nz, volume, flow);
    }
    return launch_deform(ctx, d_img1, SrcLinear<float>{d_img}, f, nx, ny, nz, volume, flow);
}

}  // namespace

MC_EXPORT int mcsart_projection_ex(mcsart_ctx *ctx, float *d_proj, const void *d_img,
                                   int storage, int fp_sum, int geom64, float angle, float SO,
                                   float SD, float da, int na, float ai, float db, int nb,
                                   float bi, int nx, int ny, int nz) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_REQUIRE(d_proj && d_img, "d_proj and d_img must be non-NULL");
    MC_REQUIRE(storage >= MCSART_F32 && storage <= MCSART_F16, "unknown storage type %d", storage);
    MC_REQUIRE(fp_sum >= SUM_REF && fp_sum <= SUM_KAHAN, "fp_sum must be 0, 1 or 2");
    MC_REQUIRE(geom64 == 0 || geom64 == 1, "geom64 must be 0 or 1");
    MC_REQUIRE(geom64 == 0 || fp_sum != SUM_REF,
               "FP64 geometry (geom64) needs a split summation projector (fp_sum 1 or 2)");
    const Geom g = make_geom(SO, SD, da, na, ai, db, nb, bi, nx, ny, nz);
    MC_TRY(validate_geom(g));
    if (storage == MCSART_F32)
        MC_TRY(projection_ex_typed(ctx, d_proj, (const float *)d_img, fp_sum, geom64, angle, g));
    else if (storage == MCSART_BF16)
        MC_TRY(projection_ex_typed(ctx, d_proj, (const __nv_bfloat16 *)d_img, fp_sum, geom64,
                                   angle, g));
    else
        MC_TRY(projection_ex_typed(ctx, d_proj, (const __half *)d_img, fp_sum, geom64, angle, g));
    return finish(ctx, "mcsart_projection_ex");
}

MC_EXPORT int mcsart_backprojection_ex(mcsart_ctx *ctx, float *d_img, const float *d_proj,
                                       int geom64, float angle, float SO, float SD, float da,
                                       int na, float ai, float db, int nb, float bi, int nx,
                                       int ny, int nz) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_REQUIRE(d_proj && d_img, "d_proj and d_img must be non-NULL");
    MC_REQUIRE(geom64 == 0 || geom64 == 1, "geom64 must be 0 or 1");
    if (!geom64)
        return mcsart_backprojection(ctx, d_img, d_proj, angle, SO, SD, da, na, ai, db, nb, bi,
                                     nx, ny, nz);
    const Geom g = make_geom(SO, SD, da, na, ai, db, nb, bi, nx, ny, nz);
    MC_TRY(validate_geom(g));
    BPArgs a{};
    a.proj = d_proj;
    a.g = g;
    a.angle = angle;
    a.cos64 = cos((double)angle);
    a.sin64 = sin((double)angle);
    a.out = d_img;
    const dim3 grid = bp_grid<BP_NZ, BP_ROWS>(g, BP_PLAIN), block(32, BP_ROWS);
    MC_LAUNCH(ctx, (bp_kernel<1, BP_PLAIN, false, false, true>), grid, block, 0, a);
    return finish(ctx, "mcsart_backprojection_ex");
}

MC_EXPORT int mcsart_deform_ex(mcsart_ctx *ctx, void *d_img1, const float *d_img, int nx, int ny,
                               int nz, float volume, float flow, const void *d_fields, int storage,
                               int interp) {
    clear_error();
    MC_TRY(validate_ctx(ctx));
    MC_TRY(validate_dims(nx, ny, nz));
    MC_REQUIRE(d_img1 && d_img && d_fields, "volume and field pointers must be non-NULL");
    MC_REQUIRE(d_img1 != (const void *)d_img, "d_img1 must not alias d_img");
    MC_REQUIRE(storage >= MCSART_F32 && storage <= MCSART_F16, "unknown storage type %d", storage);
    MC_REQUIRE(interp == MCSART_INTERP_TEXTURE || interp == MCSART_INTERP_EXACT,
               "unknown interpolation model %d", interp);
    if (storage == MCSART_F32)
        MC_TRY(deform_ex_typed(ctx, (float *)d_img1, d_img, nx, ny, nz, volume, flow,
                               (const float *)d_fields, interp));
    else if (storage == MCSART_BF16)
        MC_TRY(deform_ex_typed(ctx, (__nv_bfloat16 *)d_img1, d_img, nx, ny, nz, volume, flow,
                               (const __nv_bfloat16 *)d_fields, interp));
    else
        MC_TRY(deform_ex_typed(ctx, (__half *)d_img1, d_img, nx, ny, nz, volume, flow,
                               (const __half *)d_fields, interp));
    return finish(ctx, "mcsart_deform_ex");
}
