// Distance-driven forward projector (the reference's kernel_projection,
// src/cu_projection.cu:15-145), restructured for B200.
//
// Reference semantics kept exactly: per-ray driving axis |x21| > |y21| (:39);
// the four in-plane edge ratios yl/xl, yl/xr, yr/xl, yr/xr and their min/max
// (:54-64); axial edges zl/x21, zr/x21 (:71-77); integer ny/2, nz/2 offsets
// against float nx/2 (:52,55,72); overlap weights normalised by the footprint
// width (:83,86); loops clamped to the volume.
//
// Restructured for the hardware:
//   * one thread per ray (the reference runs 4 redundant threads per ray that
//     race on a non-atomic +=), the 32 lanes of a warp being 32 consecutive
//     detector rows of one detector column;
//   * every volume is read through a z-fastest copy
//     zf[iz + (ix + iy*nx)*nzp]: a warp's rays meet each slab in the same one
//     or two in-plane voxel columns and in neighbouring slices, so one copy
//     serves both driving axes, a ray's two axial voxels are neighbours in
//     memory, and everything in-plane (weights, which columns are visited,
//     their addresses) is the same for the whole warp;
//   * the loop-invariant ratios are hoisted out of the slab loop;
//   * up to three volumes are projected with one set of weights, the
//     projection of a ones-volume (sum of weights) comes for free, and the
//     SART residual, its norm partial sums and the packing for the
//     backprojector are done in the epilogue;
//   * in the split summation modes the slabs of a ray are split across
//     `groups` warps of a block and recombined in a fixed order through shared
//     memory (deterministic).
#pragma once

#include "backprojector.cuh"
#include "common.cuh"

namespace mcsart {

enum FPMode { FP_PLAIN = 0, FP_IMAGE = 1, FP_MOTION = 2 };

struct RayGeom {
    float r0, r1, r2, r3;  // in-plane edge ratios
    float rz0, rz1;        // axial edge ratios
    float u_off;           // source coordinate along the in-plane axis (y1 or x1)
    float u_half;          // (float)(nu/2), integer division
    float d_half;          // (float)nd/2, float division
    float src_d;           // source coordinate along the driving axis (x1 or y1)
    int nd, nu;
    bool xdrive;
};

// src/cu_projection.cu:23-39,48-51,67-68,101-104,120-121 for ray (ia, ib).
// Every operation is pinned with an explicit rounding intrinsic: which
// products the compiler fuses into fma's otherwise depends on the surrounding
// code.  The fused forms below are the ones whose results equal the
// reference kernel's bit for bit; they were selected by running every
// combination of candidate forms against the rebuilt reference on ~300k rays
// (3 geometries, 30 angles, both driving axes): x2 and y2 fuse the product
// with cos, the edge offsets (da/2)*sin, (da/2)*cos fuse into the edges, the
// axial edges are z2 -+ db/2 after rounding z2, the source offset is
// subtracted unfused.
__device__ __forceinline__ RayGeom ray_geom(float cphi, float sphi, int ia, int ib,
                                            const Geom &g) {
    const float x1 = -__fmul_rn(g.SO, cphi), y1 = -__fmul_rn(g.SO, sphi);
    const float x20 = __fsub_rn(g.SD, g.SO);
    const float y20 = __fmul_rn(__fadd_rn((float)ia, g.ai), g.da);
    const float x2 = __fmaf_rn(x20, cphi, -__fmul_rn(y20, sphi));
    const float y2 = __fmaf_rn(y20, cphi, __fmul_rn(x20, sphi));
    const float z2 = __fmul_rn(__fadd_rn((float)ib, g.bi), g.db);  // z21 = z2 - z1, z1 = 0
    const float x21 = __fsub_rn(x2, x1), y21 = __fsub_rn(y2, y1);
    RayGeom r;
    r.xdrive = fabsf(x21) > fabsf(y21);
    const float hda = __fdiv_rn(g.da, 2.0f), hdb = __fdiv_rn(g.db, 2.0f);
    const float xl = __fmaf_rn(-hda, sphi, x21), xr = __fmaf_rn(hda, sphi, x21);
    const float yl = __fmaf_rn(-hda, cphi, y21), yr = __fmaf_rn(hda, cphi, y21);
    const float zl = __fsub_rn(z2, hdb), zr = __fadd_rn(z2, hdb);
    if (r.xdrive) {
        r.r0 = __fdiv_rn(yl, xl); r.r1 = __fdiv_rn(yl, xr);
        r.r2 = __fdiv_rn(yr, xl); r.r3 = __fdiv_rn(yr, xr);
        r.rz0 = __fdiv_rn(zl, x21); r.rz1 = __fdiv_rn(zr, x21);
        r.u_off = y1; r.u_half = (float)(g.ny / 2);
        r.d_half = __fdiv_rn((float)g.nx, 2.0f); r.src_d = x1;
        r.nd = g.nx; r.nu = g.ny;
    } else {
        r.r0 = __fdiv_rn(xl, yl); r.r1 = __fdiv_rn(xl, yr);
        r.r2 = __fdiv_rn(xr, yl); r.r3 = __fdiv_rn(xr, yr);
        r.rz0 = __fdiv_rn(zl, y21); r.rz1 = __fdiv_rn(zr, y21);
        r.u_off = x1; r.u_half = (float)(g.nx / 2);
        r.d_half = __fdiv_rn((float)g.ny, 2.0f); r.src_d = y1;
        r.nd = g.ny; r.nu = g.nx;
    }
    return r;
}

// z-fastest volumes: zf[k][iz + (ix + iy*nx)*nzp], zero for nz <= iz < nzp (zf_pitch)
template <typename VT, int K> struct FPVolumes {
    const VT *zf[K];
};

// Distance in a z-fastest volume between in-plane neighbours along the
// in-plane axis (su) and along the driving axis (sd) of a ray.
__device__ __forceinline__ void zf_strides(bool xdrive, const Geom &g, int &su, int &sd) {
    const int row = g.nx * g.nzp;  // fits: the copies hold fewer than 2^31 elements
    su = xdrive ? row : g.nzp;
    sd = xdrive ? g.nzp : row;
}

// The K volumes' values at voxel offset a into t[0..K-1]: one load per
// volume, or (PAIR, three volumes) the second and third interleaved in one
// array, base[1][2a], base[1][2a + 1], read with one two-element load.
template <int K, bool PAIR, typename VT>
__device__ __forceinline__ void fp_voxel(const VT *const *base, int64_t a, float *t) {
    static_assert(!PAIR || K == 3, "paired volumes come with three volumes");
    if (PAIR) {
        t[0] = ldv(base[0], a);
        const float2 q = ldv2(base[1], a);
        t[1] = q.x;
        t[2] = q.y;
    } else {
#pragma unroll
        for (int k = 0; k < K; k++) t[k] = ldv(base[k], a);
    }
}
// Ray-sum order.  SUM_REF accumulates every voxel term straight into the ray
// sum in the reference's order (slabs, then in-plane, then axial index,
// acc = fma(v*w_u, w_z, acc), cu_projection.cu:81-88), so that results are
// bitwise those of the reference kernel.  SUM_PLAIN / SUM_KAHAN first sum the
// (at most a few) terms of one slab and then add the slab sum to the ray sum,
// plainly or with Kahan compensation; they allow the slabs of a ray to be
// split across warps.
enum SumMode { SUM_REF = 0, SUM_PLAIN = 1, SUM_KAHAN = 2 };

// ------------------------------------------------------------------------
// FP64 geometry (options.geom64, with the split summation modes): the same
// footprint formulas as ray_geom / slab_u (src/cu_projection.cu:23-144),
// every boundary coordinate and overlap weight in FP64; the volume terms
// v * w are accumulated in FP32 (plainly or Kahan-compensated), the weight
// sum (the projection of a ones-volume, the SART row normaliser) in FP64.
struct RayGeom64 {
    double r0, r1, r2, r3, rz0, rz1;
    double u_off, u_half, d_half, src_d;
    int nd, nu;
    bool xdrive;
};

__device__ __forceinline__ RayGeom64 ray_geom64(double cphi, double sphi, int ia, int ib,
                                                const Geom &g) {
    const double SO = g.SO, SD = g.SD, da = g.da, db = g.db;
    const double x1 = -SO * cphi, y1 = -SO * sphi;  // :25-26
    const double x20 = SD - SO, y20 = ((double)ia + (double)g.ai) * da;
    const double x2 = x20 * cphi - y20 * sphi, y2 = y20 * cphi + x20 * sphi;
    const double z2 = ((double)ib + (double)g.bi) * db;
    const double x21 = x2 - x1, y21 = y2 - y1;
    RayGeom64 r;
    r.xdrive = fabs(x21) > fabs(y21);  // :39
    const double hda = da / 2.0, hdb = db / 2.0;
    const double xl = x21 - hda * sphi, xr = x21 + hda * sphi;
    const double yl = y21 - hda * cphi, yr = y21 + hda * cphi;
    const double zl = z2 - hdb, zr = z2 + hdb;
    if (r.xdrive) {
        r.r0 = yl / xl; r.r1 = yl / xr; r.r2 = yr / xl; r.r3 = yr / xr;
        r.rz0 = zl / x21; r.rz1 = zr / x21;
        r.u_off = y1; r.u_half = (double)(g.ny / 2);
        r.d_half = (double)g.nx / 2.0; r.src_d = x1;
        r.nd = g.nx; r.nu = g.ny;
    } else {
        r.r0 = xl / yl; r.r1 = xl / yr; r.r2 = xr / yl; r.r3 = xr / yr;
        r.rz0 = zl / y21; r.rz1 = zr / y21;
        r.u_off = x1; r.u_half = (double)(g.nx / 2);
        r.d_half = (double)g.ny / 2.0; r.src_d = y1;
        r.nd = g.ny; r.nu = g.nx;
    }
    return r;
}

template <typename VT, int K, typename MT = VT> struct FPArgs {
    FPVolumes<VT, K> vol;
    Geom g;
    float angle;            // used when angles == nullptr
    double cos64, sin64;    // of the angle (single views with FP64 geometry)
    const float *angles;    // per-view angles (device), view = blockIdx.z
    int mode;
    // FP_PLAIN: out[view*na*nb + ia + ib*na] = s0
    float *out;
    // FP_IMAGE / FP_MOTION
    const MT *meas;     // measured projection of this view
    float *resid;       // residual output (nullable)
    float2 *bp_in;      // (residual, ones-projection) pairs for the backprojector
    double2 *norm_part; // per-block (sum b^2, sum r^2)
    // several views per launch (fp_ref_kernel, view = blockIdx.z): meas,
    // resid and bp_in advance by na*nb per view, norm_part by the blocks of
    // one view, and the volumes by vol_stride elements per view (0: every
    // view projects the same volumes)
    int64_t vol_stride;
    // when set, also write each view's backprojector column data (bp_column
    // for every (ix, iy), index ix + iy*nx, view j of a several-view launch at
    // + j*nx*ny) for the backprojector launch that follows
    float4 *bpcolA;  // amin, amax, rl, rr
    float *bpcolB;   // r0
};

// ------------------------------------------------------------------------
// Row-lane projector for the reference summation order (SUM_REF).
//
// A warp is 32 consecutive detector rows of one detector column.  Every ray
// of a column has the same in-plane geometry (driving axis, edge ratios and
// so, per slab, the in-plane voxels and weights w_u); only the axial part
// depends on the row, through z2.  So the warp's lanes compute the in-plane
// part of 32 slabs at a time, one slab each, into a table of the warp's own in
// shared memory, and then walk the slabs together: the in-plane weights, the
// addresses of the voxel columns and whether there are one or two of them are
// the same for all lanes, and each lane adds its ray's axial part and terms in
// the reference's order.  The axial weights of two slabs are computed at once
// with packed FP32 instructions (each half rounds as the scalar one).
//
// The rays of a warp meet a slab within some 20 neighbouring slices of one or
// two voxel columns (32 rows of less than a voxel each), so the lanes copy
// both windows, two slices each, into shared memory with one cp.async, S slabs
// at a time and a stage ahead: no ray waits on the L2, and every voxel is
// requested once per warp instead of once per ray.  Warps share nothing; the
// slab loop has no block barrier.
//
// What bounds it: instruction issue (66-72 % of the slots at 256x256x160 with
// a 512x384 detector) and, with three volumes, shared-memory bandwidth (80 %).
// Two thirds of a slab's instructions are the axial footprint's correctly
// rounded weights and the terms, which the reference's bits require of every
// ray and slab.  Measured there, one view: 107 us with one volume and the
// weights' sum (77 M warp instructions), 160 us with three; with 16 columns x
// 2 rows per warp reading x- or y-fastest copies straight from L2 they took
// 199 us (126 M) and 229 us.  128x128x96, 256x192: 25 and 34 us (43 and 50).
// Also measured, same bits: direct loads instead of the windows 128 / 197 us
// (L2 latency), two rows per lane with the packed operations across the rows
// 117 / 180 us (half the warps), 1 or 2 columns per block no difference.
constexpr int FPC_COLS = 4;                    // detector columns (warps) per block
constexpr int FPC_ROWS = 32;                   // detector rows per block: a warp's lanes
constexpr int FPC_THREADS = FPC_COLS * 32;

// In-plane footprint of one slab.  U2 - U1 <= 1: (a, b) = weights of voxels
// U1 and U1 + 1; otherwise (a, b) = (ui1, ui2), the footprint edges.
struct SlabU {
    int U1, U2;
    float a, b;
};

// :52 / :105: distance of slab d's centre from the source along the driving
// axis (d < 2^20, validate_geom: mk_i2f is exact).
__device__ __forceinline__ float slab_dc(const RayGeom &r, int d) {
    return __fsub_rn(__fsub_rn(__fadd_rn(mk_i2f(d), 0.5f), r.d_half), r.src_d);
}

// :52-63 / :105-116 for slab d of the ray's column.
__device__ __forceinline__ SlabU slab_u(const RayGeom &r, int d) {
    const float dc = slab_dc(r, d);
    const float c0 = __fadd_rn(__fmaf_rn(r.r0, dc, r.u_off), r.u_half);
    const float c1 = __fadd_rn(__fmaf_rn(r.r1, dc, r.u_off), r.u_half);
    const float c2 = __fadd_rn(__fmaf_rn(r.r2, dc, r.u_off), r.u_half);
    const float c3 = __fadd_rn(__fmaf_rn(r.r3, dc, r.u_off), r.u_half);
    const float ui1 = fminf(fminf(c0, c1), fminf(c2, c3));
    const float ui2 = fmaxf(fmaxf(c0, c1), fmaxf(c2, c3));
    SlabU e;
    float fu0, fu1;
    if (fabsf(ui1) < MK_MAGIC_RANGE && fabsf(ui2) < MK_MAGIC_RANGE) {
        e.U1 = mk_floor(ui1, fu0);
        e.U2 = mk_floor_i(ui2);
        fu1 = __fadd_rn(fu0, 1.0f);  // (float)(U1 + 1), exact below 2^22
    } else {
        e.U1 = (int)floorf(ui1);
        e.U2 = (int)floorf(ui2);
        fu0 = (float)e.U1;
        fu1 = (float)(e.U1 + 1);
    }
    if (e.U2 - e.U1 <= 1) {
        const float du = __fsub_rn(ui2, ui1);  // :83 / :136
        const float n0 = __fsub_rn(fminf(__fadd_rn(fu0, 1.0f), ui2), fmaxf(fu0, ui1));
        const float n1 = __fsub_rn(fminf(__fadd_rn(fu1, 1.0f), ui2), fmaxf(fu1, ui1));
        const float y = mk_recip(du);
        e.a = mk_div(n0, du, y);
        e.b = mk_div(n1, du, y);
        if (!(mk_den_ok(du) && mk_num_ok(n0) && mk_num_ok(n1))) {
            e.a = __fdiv_rn(n0, du);
            e.b = __fdiv_rn(n1, du);
        }
    } else {
        e.a = ui1;
        e.b = ui2;
    }
    return e;
}

// Per-ray facts about the axial footprint over all the ray's slabs, bounded
// from the ray's constants with rounding margins: the slab distance dc runs
// monotonically over [dc(0), dc(nd - 1)] and cz = rz * dc + nz/2 is linear in
// it, computed with an error below 2^-23 * max|cz|.
//  zsafe:  |cz| < 2^19, inside the magic-number floor's range, so that also
//          dz = zi2 - zi1 < 2^20;
//  narrow: additionally dc keeps one sign, x21 or y21 the same one, so that
//          cz0 and cz1 grow with the detector row (products, quotients and
//          sums round monotonically) and cz0 <= cz1 are the minimum and the
//          maximum themselves; and dz is in [2^-19, 0.99], so the footprint
//          spans at most the two slices Z1 and Z1 + 1.  With one slice nz/2 is
//          0, and each edge is 0 or at least 2^-79 in magnitude.
// On a narrow ray's slabs with 0 <= Z1 every division's operands are in
// mk_div's checked range: dz is; n0 is dz or (Z1 + 1) - zi1 with
// 0 <= zi1 < Z1 + 1, at least 2^-24 and positive; n1, used only when
// Z2 = Z1 + 1, is zi2 - (Z1 + 1), +0 or at least an ulp of 1.  With Z1 = -1, n1 is
// cz1 itself, a sum with nz/2, so +0 or at least 2^-24 for nz/2 >= 1, and +0 or at
// least 2^-79 with one slice (a product and a sum with +0, never -0).
struct RayAxial {
    bool zsafe, narrow;
};
__device__ __forceinline__ RayAxial ray_axial(const RayGeom &r, float z_half, int nz) {
    const float dc_lo = __fsub_rn(__fsub_rn(0.5f, r.d_half), r.src_d) - 1.0f;
    const float dc_hi = __fsub_rn(__fsub_rn((float)r.nd - 0.5f, r.d_half), r.src_d) + 1.0f;
    const float dmax = fmaxf(fabsf(dc_lo), fabsf(dc_hi));
    const float rmax = fmaxf(fabsf(r.rz0), fabsf(r.rz1));
    const float zmax = rmax * dmax + fabsf(z_half) + 1.0f;
    const float err = zmax * 0x1p-21f;  // >= 4 ulp of any cz, covers these bounds' rounding
    RayAxial a;
    a.zsafe = zmax + err < 0x1p19f;
    // rz = (z2 -+ db/2) / x21: rz0 < rz1 exactly when x21 > 0
    const bool ordered = (dc_lo > 0.0f && r.rz0 < r.rz1) || (dc_hi < 0.0f && r.rz0 > r.rz1);
    const float dmin = fminf(fabsf(dc_lo), fabsf(dc_hi));
    const float drz = fabsf(r.rz1 - r.rz0);
    const float dz_min = (drz * dmin - 2.0f * err) * (1.0f - 0x1p-20f);
    const float dz_max = (drz * dmax + 2.0f * err) * (1.0f + 0x1p-20f);
    a.narrow = a.zsafe && ordered && dz_min >= 0x1p-19f && dz_max <= 0.99f;
    if (nz < 2) {
        // (a factor of 2 for the rounding of these products)
        const float e0 = fabsf(r.rz0) * dmin, e1 = fabsf(r.rz1) * dmin;
        a.narrow = a.narrow && (r.rz0 == 0.0f || e0 >= 0x1p-78f) && (r.rz1 == 0.0f || e1 >= 0x1p-78f);
    }
    return a;
}

// The slabs d of a ray whose axial footprint can meet the volume: a superset
// of {d : max(cz0, cz1) >= 0 and min(cz0, cz1) < nz}, outside which the
// reference's axial loop over max(0, Z1) .. min(nz-1, Z2) is empty
// (:80-82 / :133-135) and the slab adds nothing.  Worked from the exact lines
// c_k(dc) = rz_k * dc + nz/2 of the ray's own (float) constants with a
// tolerance of 1/16 voxel, far above the difference of their float evaluation
// (a few ulp of values below 2^16 at the faces); each condition's set of dc is
// a union of half-lines whose hull is taken, and the intersection of the hulls
// is mapped to slab indices with a margin of one slab plus the rounding of
// these float expressions (2^-19 of the largest magnitude, four times the sum
// of their relative errors).  Returns lo > hi when no slab can contribute.
__device__ __forceinline__ void ray_zrange(const RayGeom &r, float zh, int nz, int &lo, int &hi) {
    const float tol = 1.0f / 16.0f, inf = __int_as_float(0x7f800000);
    const float rz[2] = {r.rz0, r.rz1};
    // hulls of U_k {rz_k dc >= -tol - zh} and U_k {rz_k dc < nz + tol - zh}
    float lo1 = inf, hi1 = -inf, lo2 = inf, hi2 = -inf;
    const float t1 = -tol - zh, t2 = (float)nz + tol - zh;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float a = rz[k];
        float y;  // 1 / a to 2^-22
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
        if (a > 0.0f) {
            lo1 = fminf(lo1, t1 * y); hi1 = inf;    // [t1, inf)
            lo2 = -inf; hi2 = fmaxf(hi2, t2 * y);   // (-inf, t2)
        } else if (a < 0.0f) {
            lo1 = -inf; hi1 = fmaxf(hi1, t1 * y);   // (-inf, t1]
            lo2 = fminf(lo2, t2 * y); hi2 = inf;    // (t2, inf)
        } else {  // constant zh: inside [0, nz)
            lo1 = -inf; hi1 = inf;
            lo2 = -inf; hi2 = inf;
        }
    }
    // slab d has dc = d + 0.5 - d_half - src_d (up to the rounding of those floats)
    const float off = r.d_half + r.src_d - 0.5f, fn = (float)r.nd;
    const float m = 1.0f + 0x1p-19f * (fn + fabsf(off) + 2.0f);
    const float a = fmaxf(fmaxf(lo1, lo2) + off - m, -1.0f);
    const float b = fminf(fminf(hi1, hi2) + off + m, fn);
    if (a <= b) {
        lo = max(0, (int)floorf(a));
        hi = min(r.nd - 1, (int)ceilf(b));
    } else {  // also NaN
        lo = INT_MAX;
        hi = INT_MIN;
    }
}

// A slab of a warp's table: what its rays share.  In-plane, for a footprint
// of at most two voxels, the voxels the reference's loop visits (:80-82 /
// :133-135), in its order, a single one always first: the offset o of the
// warp's window in the first one's column of the z-fastest volume (the second
// one's is su further) and the weights a, b (zero for a voxel not visited).
// The window begins at slice zlo, the even one at or below the first ray's Z1;
// pairs: bit l is set where one of its slices 2l, 2l + 1 is needed and in the
// volume (the other is too, or is the zero behind an odd depth), bit 16 + l
// where moreover the second voxel is visited.
struct __align__(8) SlabCopy {
    int o;
    unsigned pairs;
};
// The rest of two neighbouring slabs, side by side for the packed operations.
struct __align__(16) SlabPair {
    float a[2], b[2];
    float dc[2];  // the slabs' distances (slab_dc)
    int zb[2];    // MK_MAGIC_BITS + zlo: a ray's place in the window is (bits
                  // of its magic-number sum) - zb
};
// SC_ANY: some ray can meet the volume in the slab; SC_FAST: the in-plane
// footprint is at most two voxels wide, and o, a, b are valid; SC_TWO: it
// visits two voxels; SC_STAGE: additionally all rays are narrow and the window
// holds every slice they need; SC_IN: additionally every ray's slices Z1 and
// Z1 + 1 are in the volume.
constexpr int SC_ANY = 1, SC_FAST = 2, SC_TWO = 4, SC_STAGE = 8, SC_IN = 16;
constexpr int FPW = 32;  // slices per window

// The table entry of slab d; rz_first, rz_last: rz0 of the warp's first and
// last row; narrow: every ray of the warp is (ray_axial).
__device__ __forceinline__ void slab_entry(const RayGeom &r, int d, int su, int sd, float rz_first,
                                           float rz_last, bool narrow, float z_half, int nz,
                                           SlabCopy &c, int &flags, float &a, float &b, float &dc,
                                           int &zb) {
    const SlabU e = slab_u(r, d);
    const bool two_wide = e.U2 - e.U1 <= 1;
    const bool u0 = e.U1 >= 0 && e.U1 <= r.nu - 1;
    const bool u1 = e.U1 + 1 <= e.U2 && e.U1 + 1 >= 0 && e.U1 + 1 <= r.nu - 1;
    const bool any = e.U2 >= 0 && e.U1 <= r.nu - 1;
    int f = (any ? SC_ANY : 0) | (two_wide && (u0 || u1) ? SC_FAST : 0) |
            (two_wide && u0 && u1 ? SC_TWO : 0);
    dc = slab_dc(r, d);
    c.pairs = 0;
    int zlo = 0;
    if (narrow) {
        // cz0 as every ray computes it (:71 / :124); rows in order, so these
        // are the warp's smallest and largest Z1
        const int zf = mk_floor_i(__fadd_rn(__fmul_rn(rz_first, dc), z_half));
        const int zl = mk_floor_i(__fadd_rn(__fmul_rn(rz_last, dc), z_half)) + 1;
        zlo = zf & ~1;
        const int lo = max(0, -zlo), hi = min(zl, nz - 1) - zlo;
        if (lo > hi) f = 0;  // no ray meets a slice of the volume here
        if ((f & SC_FAST) && zl - zlo < FPW) {
            f |= SC_STAGE | (zf >= 0 && zl <= nz - 1 ? SC_IN : 0);
            c.pairs = (0xffffu >> (15 - (hi >> 1))) & (0xffffu << (lo >> 1));
            if (f & SC_TWO) c.pairs |= c.pairs << 16;
        }
    }
    flags = f;
    const int U = u0 ? e.U1 : u1 ? e.U1 + 1 : 0;  // the first visited voxel
    c.o = U * su + d * sd + zlo;
    a = f & SC_FAST ? (u0 ? e.a : e.b) : 0.0f;
    b = f & SC_TWO ? e.b : 0.0f;
    zb = MK_MAGIC_BITS + zlo;
}

// One slab of one ray by the reference's loops, any footprint (:80-88 /
// :133-141), of volumes with strides su, sd and sz (below 2^31 elements).
template <int K, bool ONES, typename VT, bool PAIR>
__device__ __forceinline__ void fp_slab_loops(const RayGeom &r, const Geom &g, int d,
                                              const VT *const *base, int su, int sd, int sz,
                                              float z_half, float *acc, float &accw) {
    const SlabU e = slab_u(r, d);
    const float dc = slab_dc(r, d);
    // :71-77 / :124-130 ("ratio * xc + z1 + nz / 2", z1 = 0)
    const float cz0 = __fadd_rn(__fmul_rn(r.rz0, dc), z_half);
    const float cz1 = __fadd_rn(__fmul_rn(r.rz1, dc), z_half);
    const float zi1 = fminf(cz0, cz1), zi2 = fmaxf(cz0, cz1);
    const int Z1 = (int)floorf(zi1), Z2 = (int)floorf(zi2);
    const float dz = __fsub_rn(zi2, zi1);
    const int U1 = e.U1, U2 = e.U2;
    const bool narrow = U2 - U1 <= 1;
    const int u_lo = max(0, U1), u_hi = min(r.nu - 1, U2);
    const int z_lo = max(0, Z1), z_hi = min(g.nz - 1, Z2);
    const float ui1 = e.a, ui2 = e.b;
    const float du = narrow ? 0.0f : __fsub_rn(ui2, ui1);
    for (int u = u_lo; u <= u_hi; u++) {
        const float wu = narrow ? (u == U1 ? e.a : e.b)
                                : __fdiv_rn(__fsub_rn(fminf(__fadd_rn((float)u, 1.0f), ui2),
                                                      fmaxf((float)u, ui1)), du);
        const int row = u * su + d * sd;
        for (int z = z_lo; z <= z_hi; z++) {
            const float wz = __fdiv_rn(__fsub_rn(fminf(__fadd_rn((float)z, 1.0f), zi2),
                                                 fmaxf((float)z, zi1)), dz);
            float t[K];
            fp_voxel<K, PAIR>(base, row + z * sz, t);
#pragma unroll
            for (int k = 0; k < K; k++) acc[k] = __fmaf_rn(__fmul_rn(t[k], wu), wz, acc[k]);
            if (ONES) accw = __fmaf_rn(wu, wz, accw);
        }
    }
}
template <int K, bool ONES, typename VT, bool PAIR>
__device__ __forceinline__ void fp_slab_general(const RayGeom &r, const Geom &g, int d,
                                                const VT *const *base, float z_half, float *acc,
                                                float &accw) {
    int su, sd;
    zf_strides(r.xdrive, g, su, sd);
    fp_slab_loops<K, ONES, VT, PAIR>(r, g, d, base, su, sd, 1, z_half, acc, accw);
}

// One slab of one ray straight from memory, for slabs of narrow warps that are not
// staged: at most two slices Z1, Z1 + 1, with the operand ranges tested; false,
// with nothing added, where a lane's footprint does not fit.
template <int K, bool ONES, typename VT, bool PAIR>
__device__ __forceinline__ bool fp_slab_direct(float rz0, float rz1, float dc, float a, float b,
                                               int o, int su, bool two_u, const VT *const *base,
                                               int nz, float z_half, float *acc, float &accw) {
    // :71-77 / :124-130 ("ratio * xc + z1 + nz / 2", z1 = 0)
    const float cz0 = __fadd_rn(__fmul_rn(rz0, dc), z_half);
    const float cz1 = __fadd_rn(__fmul_rn(rz1, dc), z_half);
    const float zi1 = fminf(cz0, cz1), zi2 = fmaxf(cz0, cz1);
    float fz0;
    const int Z1 = mk_floor(zi1, fz0);
    const float fz1 = __fadd_rn(fz0, 1.0f), dz = __fsub_rn(zi2, zi1);
    // Z2 = floor(zi2) is Z1 (zi2 < Z1 + 1) or Z1 + 1 (zi2 < Z1 + 2): compared
    // against the exact floats
    const bool two = zi2 >= fz1, narrow = zi2 < __fadd_rn(fz1, 1.0f);
    // :86 / :139: min(Z1 + 1, zi2) - max(Z1, zi1), where Z1 <= zi1; and, when
    // Z2 = Z1 + 1, min(Z1 + 2, zi2) - max(Z1 + 1, zi1) = zi2 - (Z1 + 1)
    const float n0 = __fsub_rn(fminf(fz1, zi2), zi1);
    const float n1 = __fsub_rn(zi2, fz1);
    const bool outside = zi2 < 0.0f || zi1 >= (float)nz;
    const bool ok = outside || (narrow && mk_den_ok(dz) && mk_num_ok(n0) && mk_num_ok(n1));
    if (!__all_sync(0xffffffffu, ok)) return false;
    const float y = mk_recip(dz);
    const float wz0 = mk_div(n0, dz, y), wz1 = mk_div(n1, dz, y);
    const bool p0 = (unsigned)Z1 < (unsigned)nz, p1 = two && (unsigned)(Z1 + 1) < (unsigned)nz;
    const int z0 = min(max(Z1, 0), nz - 1), z1 = min(max(Z1 + 1, 0), nz - 1);
    for (int u = 0; u < (two_u ? 2 : 1); u++) {
        const float wu = u ? b : a;
        float v0[K], v1[K];
        fp_voxel<K, PAIR>(base, o + u * su + z0, v0);
        fp_voxel<K, PAIR>(base, o + u * su + z1, v1);
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (p0) acc[k] = __fmaf_rn(__fmul_rn(v0[k], wu), wz0, acc[k]);
            if (p1) acc[k] = __fmaf_rn(__fmul_rn(v1[k], wu), wz1, acc[k]);
        }
        if (ONES) {
            if (p0) accw = __fmaf_rn(wu, wz0, accw);
            if (p1) accw = __fmaf_rn(wu, wz1, accw);
        }
    }
    return true;
}

// One slab of one ray straight from memory, for warps whose rays are not narrow:
// axial footprints of at most three slices Z1 .. Z1 + 2, with the operand ranges
// tested; false, with nothing added, where a lane's does not fit.  The in-plane
// footprint is the table entry's (fast: voxels at o and, if two_u, o + su with
// weights a, b) or, of any width, worked out again; either is the same for the
// whole warp.  All of a slab's loads are issued before its terms.
template <int K, bool ONES, typename VT, bool PAIR>
__device__ __forceinline__ bool fp_slab_wide(const RayGeom &r, int d, bool fast, float dc, float a,
                                               float b, int o, int su, int sd, bool two_u,
                                               const VT *const *base, int nz, float z_half,
                                               float *acc, float &accw) {
    // :71-77 / :124-130 ("ratio * xc + z1 + nz / 2", z1 = 0)
    const float cz0 = __fadd_rn(__fmul_rn(r.rz0, dc), z_half);
    const float cz1 = __fadd_rn(__fmul_rn(r.rz1, dc), z_half);
    const float zi1 = fminf(cz0, cz1), zi2 = fmaxf(cz0, cz1);
    float fz0;
    const int Z1 = mk_floor(zi1, fz0);
    const float fz1 = __fadd_rn(fz0, 1.0f), fz2 = __fadd_rn(fz0, 2.0f), dz = __fsub_rn(zi2, zi1);
    // Z2 = floor(zi2), compared against the exact floats
    const bool two = zi2 >= fz1, three = zi2 >= fz2;
    // :86 / :139, the overlaps of slices Z1 (Z1 <= zi1), Z1 + 1 and Z1 + 2
    const float n0 = __fsub_rn(fminf(fz1, zi2), zi1);
    const float n1 = __fsub_rn(fminf(fz2, zi2), fz1);
    const float n2 = __fsub_rn(zi2, fz2);
    const bool outside = zi2 < 0.0f || zi1 >= (float)nz;
    const bool ok = outside || (zi2 < __fadd_rn(fz0, 3.0f) && mk_den_ok(dz) && mk_num_ok(n0) &&
                                (!two || mk_num_ok(n1)) && (!three || mk_num_ok(n2)));
    if (!__all_sync(0xffffffffu, ok)) return false;
    const float y = mk_recip(dz);
    const float wz0 = mk_div(n0, dz, y), wz1 = mk_div(n1, dz, y), wz2 = mk_div(n2, dz, y);
    const bool p0 = (unsigned)Z1 < (unsigned)nz, p1 = two && (unsigned)(Z1 + 1) < (unsigned)nz;
    const bool p2 = three && (unsigned)(Z1 + 2) < (unsigned)nz;
    // (slices outside the volume read 0, and nothing is added for them)
    const auto load = [&](int at, float (*v)[K]) {
#pragma unroll
        for (int j = 0; j < 3; j++)
            if (j == 0 ? p0 : j == 1 ? p1 : p2) fp_voxel<K, PAIR>(base, at + Z1 + j, v[j]);
    };
    const auto add = [&](const float (*v)[K], float wu) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (p0) acc[k] = __fmaf_rn(__fmul_rn(v[0][k], wu), wz0, acc[k]);
            if (p1) acc[k] = __fmaf_rn(__fmul_rn(v[1][k], wu), wz1, acc[k]);
            if (p2) acc[k] = __fmaf_rn(__fmul_rn(v[2][k], wu), wz2, acc[k]);
        }
        if (ONES) {
            if (p0) accw = __fmaf_rn(wu, wz0, accw);
            if (p1) accw = __fmaf_rn(wu, wz1, accw);
            if (p2) accw = __fmaf_rn(wu, wz2, accw);
        }
    };
    float v0[3][K], v1[3][K];
    if (fast) {
        load(o, v0);
        if (two_u) load(o + su, v1);
        add(v0, a);
        if (two_u) add(v1, b);
        return true;
    }
    const SlabU e = slab_u(r, d);
    const bool narrow = e.U2 - e.U1 <= 1;
    const float du = narrow ? 0.0f : __fsub_rn(e.b, e.a);
    const int u_lo = max(0, e.U1), u_hi = min(r.nu - 1, e.U2);
    const auto weight = [&](int u) {  // :83 / :136
        return narrow ? (u == e.U1 ? e.a : e.b)
                      : __fdiv_rn(__fsub_rn(fminf(__fadd_rn((float)u, 1.0f), e.b),
                                            fmaxf((float)u, e.a)), du);
    };
    for (int u = u_lo; u <= u_hi; u += 2) {
        const int at = u * su + d * sd;
        load(at, v0);
        if (u < u_hi) load(at + su, v1);
        add(v0, weight(u));
        if (u < u_hi) add(v1, weight(u + 1));
    }
    return true;
}

// ---- the warp's windows in shared memory
// One window: FPW slices of one voxel column and of the paired volumes' (PAIR),
// zeros in the place of slices outside the volume, and behind each a zero.
template <typename VT, bool PAIR> struct FPWindow {
    static constexpr unsigned ES = sizeof(VT);              // bytes per slice
    static constexpr unsigned PAIRS = FPW * ES + 16;        // offset of the paired volumes
    static constexpr unsigned BYTES = PAIRS + (PAIR ? 2 * FPW * ES + 16 : 0);
};

// An N-byte asynchronous copy, or N zeros where !in (nothing is read then); both
// addresses on N bytes either way.
#ifndef MCSART_ON_COPY
#define MCSART_ON_COPY(dst, src, n)  // a test program's check of the addresses
#endif
#ifndef MCSART_ON_FORM
#define MCSART_ON_FORM(form)  // and its count of the forms that warps take
#endif
template <int N> __device__ __forceinline__ void cp_async(unsigned dst, const void *src, bool in) {
    MCSART_ON_COPY(dst, src, N);
    const int n = in ? N : 0;
    if (N == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;" ::"r"(dst), "l"(src), "r"(n),
                     "n"(N)
                     : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void sts_zero4(unsigned a) {
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(0) : "memory");
}

// This lane's part of a slab's two windows at dst (shared memory), the second
// one all zeros where the slab visits one in-plane voxel: slices 2j and 2j + 1
// of window h as one copy, lane = 16 h + j, lane_off and lane_dst that place in
// the volume and the windows (which begin on even elements: the pitch is even).
template <typename VT, bool PAIR>
__device__ __forceinline__ void window_copy(unsigned dst, const VT *const *base, const int2 c,
                                            int lane, int bit, int64_t lane_off,
                                            unsigned lane_dst) {
    using W = FPWindow<VT, PAIR>;
    constexpr int ES = sizeof(VT);
    const bool in = c.y & bit;
    cp_async<2 * ES>(dst + lane_dst, base[0] + lane_off + c.x, in);
    if constexpr (PAIR)
        cp_async<4 * ES>(dst + lane_dst + W::PAIRS + 2 * ES * (lane & 15),
                         base[1] + 2 * (lane_off + c.x), in);
}

// The K volumes' values of slice z of both windows of the slab at w.
template <int K, typename VT, bool PAIR>
__device__ __forceinline__ void window_read(const unsigned char *w, int z, float (*v)[K]) {
    using W = FPWindow<VT, PAIR>;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        v[i][0] = tof(reinterpret_cast<const VT *>(w + i * W::BYTES)[z]);
        if constexpr (PAIR) {
            const unsigned char *q = w + i * W::BYTES + W::PAIRS;
            if constexpr (sizeof(VT) == 4) {
                const float2 a = reinterpret_cast<const float2 *>(q)[z];
                v[i][1] = a.x;
                v[i][2] = a.y;
            } else {
                union {
                    unsigned u;
                    VT h[2];
                } a;
                a.u = reinterpret_cast<const unsigned *>(q)[z];
                v[i][1] = tof(a.h[0]);
                v[i][2] = tof(a.h[1]);
            }
        }
    }
}

// Two neighbouring staged slabs (narrow rays).  The branch-free division is exact
// wherever its quotient is used (ray_axial).
// What the reference's loops do not visit is read as zero, so its terms add a
// zero to the sums: slices outside the volume and a second in-plane voxel that
// is not visited are zeros in the window, and slice Z1 + 1 of a ray whose Z2 is
// Z1 is read behind it; for the weights' sum their weights are set to zero.
// Without branches the slabs of a stage are one straight line of code, whose
// long chains (reciprocal, divisions, sums) overlap.
// IN: every ray's slices Z1 and Z1 + 1 are in the volume; otherwise on tells
// whether a slab is a staged one at all (its weights a, b are zero if not).
// w: the first slab's windows.
template <int K, bool ONES, bool IN, typename VT, bool PAIR>
__device__ __forceinline__ void fp_pair_staged(float rz0, float rz1, const SlabPair &y, bool on_a,
                                               bool on_b, const unsigned char *w, int nz,
                                               float z_half, float *acc, float &accw) {
    using W = FPWindow<VT, PAIR>;
    const ulonglong2 ab = *reinterpret_cast<const ulonglong2 *>(&y.a);
    const ulonglong2 dcz = *reinterpret_cast<const ulonglong2 *>(&y.dc);
    const f32x2 dc = dcz.x;
    const int zb[2] = {(int)(unsigned)dcz.y, (int)(unsigned)(dcz.y >> 32)};
    const f32x2 zh = f2_pack(z_half, z_half);
    // :71-77 / :124-130 ("ratio * xc + z1 + nz / 2", z1 = 0)
    // (scalar products: ptxas contracts a packed product and sum, both .rn,
    // into one fma, whose single rounding is not the reference's)
    float d[2];
    f2_unpack(dc, d[0], d[1]);
    const f32x2 zi1 = f2_add(f2_pack(__fmul_rn(rz0, d[0]), __fmul_rn(rz0, d[1])), zh);
    const f32x2 zi2 = f2_add(f2_pack(__fmul_rn(rz1, d[0]), __fmul_rn(rz1, d[1])), zh);
    // floor(zi1) and floor(zi1) + 1 as a float from one magic-number sum (exact)
    const f32x2 tm = f2_add_rd(zi1, f2_pack(MK_MAGIC, MK_MAGIC));
    const f32x2 fz1 = f2_add(tm, f2_pack(1.0f - MK_MAGIC, 1.0f - MK_MAGIC));
    const f32x2 ndz = f2_sub(zi1, zi2);  // -dz, exactly negated
    float t[2], e2[2], f1[2], nd[2], wu[2][2];
    f2_unpack(tm, t[0], t[1]);
    f2_unpack(zi2, e2[0], e2[1]);
    f2_unpack(fz1, f1[0], f1[1]);
    f2_unpack(ndz, nd[0], nd[1]);
    f2_unpack(ab.x, wu[0][0], wu[0][1]);
    f2_unpack(ab.y, wu[1][0], wu[1][1]);
    // :86 / :139: min(Z1 + 1, zi2) - max(Z1, zi1), where Z1 <= zi1; and, when
    // Z2 = Z1 + 1, min(Z1 + 2, zi2) - max(Z1 + 1, zi1) = zi2 - (Z1 + 1)
    const f32x2 n0 = f2_sub(f2_pack(fminf(f1[0], e2[0]), fminf(f1[1], e2[1])), zi1);
    const f32x2 n1 = f2_sub(zi2, fz1);
    // mk_recip and mk_div, packed
    float y0[2];
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0[0]) : "f"(-nd[0]));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0[1]) : "f"(-nd[1]));
    const f32x2 ys = f2_pack(y0[0], y0[1]);
    const f32x2 yr = f2_fma(ys, f2_fma(ndz, ys, f2_pack(1.0f, 1.0f)), ys);
    const f32x2 q0 = f2_mul(n0, yr), q1 = f2_mul(n1, yr);
    float wz[2][2];  // [slice][slab]
    f2_unpack(f2_fma(f2_fma(ndz, q0, n0), yr, q0), wz[0][0], wz[0][1]);
    f2_unpack(f2_fma(f2_fma(ndz, q1, n1), yr, q1), wz[1][0], wz[1][1]);
    float v[2][2][2][K];  // [slab][slice][in-plane voxel][volume]
    float ow[2][2];       // weights of the weights' sum
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const unsigned char *const wh = w + h * 2 * W::BYTES;
        // Z2 = floor(zi2) is Z1 (zi2 < Z1 + 1) or Z1 + 1: a narrow footprint,
        // compared against the exact float
        const bool two = e2[h] >= f1[h];
        int z = (int)(__float_as_uint(t[h]) - (unsigned)zb[h]);  // place in the window
        if (!IN) z = (h ? on_b : on_a) ? z : 0;
        const int z1 = two ? z : FPW - 1;  // slice Z1 + 1, or the zero behind the window
        window_read<K, VT, PAIR>(wh, z, v[h][0]);
        window_read<K, VT, PAIR>(wh, z1 + 1, v[h][1]);
        if (ONES) {
            bool p0 = true, p2 = two;
            if (!IN) {
                const int Z1 = (int)(__float_as_uint(t[h]) - (unsigned)MK_MAGIC_BITS);
                p0 = (unsigned)Z1 < (unsigned)nz;
                p2 = two && (unsigned)(Z1 + 1) < (unsigned)nz;
            }
            ow[0][h] = p0 ? wz[0][h] : 0.0f;
            ow[1][h] = p2 ? wz[1][h] : 0.0f;
        }
    }
    // v * w_u of both slabs, then the terms in the reference's order: slab,
    // in-plane voxel, slice
    float m[2][2][2][K];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            f2_unpack(f2_mul(f2_pack(v[0][j][i][0], v[1][j][i][0]), i ? ab.y : ab.x), m[0][j][i][0],
                      m[1][j][i][0]);
#pragma unroll
            for (int k = 1; k < K; k++)
#pragma unroll
                for (int h = 0; h < 2; h++) m[h][j][i][k] = __fmul_rn(v[h][j][i][k], wu[i][h]);
        }
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
#pragma unroll
                for (int k = 0; k < K; k++) acc[k] = __fmaf_rn(m[h][j][i][k], wz[j][h], acc[k]);
                if (ONES) accw = __fmaf_rn(wu[i][h], ow[j][h], accw);
            }
}

// Shared memory of a warp of fp_ref_kernel: NST * S slabs of two windows, two
// tables of 32 slabs, their masks and the column's constants.
template <typename VT, bool PAIR, int S, int NST> struct FPShared {
    SlabPair pairs[32];
    SlabCopy copy[64];
    int flags[64];  // SC_*
    uint4 mask[2];  // bit i: slab i of a table is SC_IN, SC_STAGE, neither staged nor empty
    RayGeom ray;
    float rz_last;
    __align__(16) unsigned char win[NST * S][2][FPWindow<VT, PAIR>::BYTES];
};

// Slabs i0 .. i0 + 31 of a warp that is not narrow (slab i is wlo + i, n in all): a
// table of them, one by each lane, and then one slab after another.
template <int K, bool ONES, typename VT, bool PAIR, typename Shared>
__device__ __forceinline__ void fp_slabs_wide(Shared &sm, const Geom &g, int wlo, int i0, int n,
                                              float rz0, float rz1, bool safe, const VT *const *base,
                                              int nz, float z_half, float *acc, float &accw) {
    const int lane = threadIdx.x & 31;
    RayGeom r = sm.ray;
    int su, sd;
    zf_strides(r.xdrive, g, su, sd);
    {
        SlabCopy c;
        SlabPair &y = sm.pairs[lane >> 1];
        int f;
        float a, b, dc;
        int zb;
        slab_entry(r, wlo + min(i0 + lane, n - 1), su, sd, rz0, rz1, false, z_half, nz, c, f, a, b,
                   dc, zb);
        sm.copy[lane] = c;
        sm.flags[lane] = f;
        y.a[lane & 1] = a;
        y.b[lane & 1] = b;
        y.dc[lane & 1] = dc;
    }
    __syncwarp();
    r.rz0 = rz0;
    r.rz1 = rz1;
#pragma unroll 1
    for (int q = 0; q < min(32, n - i0); q++) {
        const int f = sm.flags[q];
        if (!(f & SC_ANY)) continue;
        const SlabPair &y = sm.pairs[q >> 1];
        if (safe && fp_slab_wide<K, ONES, VT, PAIR>(r, wlo + i0 + q, (f & SC_FAST) != 0, y.dc[q & 1],
                                                    y.a[q & 1], y.b[q & 1], sm.copy[q].o, su, sd,
                                                    (f & SC_TWO) != 0, base, nz, z_half, acc, accw)) {
            MCSART_ON_FORM(4);
            continue;
        }
        MCSART_ON_FORM(5);
        fp_slab_general<K, ONES, VT, PAIR>(r, g, wlo + i0 + q, base, z_half, acc, accw);
    }
    __syncwarp();  // the table may be overwritten now
}

// Row block i of n in dispatch order, from the middle of the detector
// outwards (m, m+1, m-1, m+2, ...): central rays cross the whole volume,
// outer ones fewer slabs (ray_zrange), so the longest blocks start first and
// the short ones fill the last wave.
__device__ __forceinline__ int middle_out(int i, int n) {
    const int m = (n - 1) / 2;
    return (i & 1) ? m + (i + 1) / 2 : m - i / 2;
}

// blockDim = FPC_THREADS: warp w is detector column blockIdx.x*FPC_COLS + w,
// lane l row 32*(row block) + l; gridDim = (ceil(na/FPC_COLS),
// ceil(nb/FPC_ROWS), views); dynamic shared memory fp_ref_smem.
// MULTI = true: several views per launch (ordered subsets, kernel-level
// multi-view projection), view = blockIdx.z with the per-view offsets of
// FPArgs; false: one view per launch without them.
// S: slabs per stage; NST: stages, NST - 1 of them in flight; MINB: resident
// blocks per SM the register budget must allow (the launch shape the driver's
// tuning may choose; every choice gives the same bits).
// PAIR (three volumes): the second and third volumes interleaved in one
// array, vol.zf[1] (fp_voxel).
// WIDE: warps that are not narrow take a loop of their own (fp_slabs_wide): at
// 256x256x160 with 256x192 cells 1.03 slices high 206 us a call, 354 by the stages'
// one-by-one form; with cells 1.55 high 250 and 463.  Its code beside the stages
// costs the narrow warps 0 to 1.5 %, so that launches leave it out where cells are
// low (fp_wide).  The bits are the same.
template <int K> constexpr int fp_stage() { return K >= 3 ? 4 : 8; }
template <int K> constexpr int fp_min_blocks() { return K >= 3 ? 5 : 6; }
template <int K, bool ONES, typename VT, typename MT = VT, bool MULTI = false,
          int S = fp_stage<K>(), int NST = 2, int MINB = fp_min_blocks<K>(), bool PAIR = false,
          bool WIDE = false>
__global__ void __launch_bounds__(FPC_THREADS, MINB) fp_ref_kernel(const FPArgs<VT, K, MT> p) {
    static_assert(K == 1 || PAIR, "one volume, or three with the last two paired");
    static_assert(32 % S == 0 && S % 2 == 0 && (NST - 1) * S <= 32, "a table holds whole stages");
    using W = FPWindow<VT, PAIR>;
    using Shared = FPShared<VT, PAIR, S, NST>;
    extern __shared__ __align__(16) unsigned char sm_warps[];
    __shared__ float sm_s[K + (ONES ? 1 : 0)][FPC_ROWS][FPC_COLS + 1];
    __shared__ double2 sm_norm[FPC_THREADS / 32];
    const Geom &g = p.g;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int by = middle_out(blockIdx.y, gridDim.y);  // this block's row block
    const float angle = p.angles ? p.angles[blockIdx.z] : p.angle;
    {
        const int ia = blockIdx.x * FPC_COLS + warp, ib = by * FPC_ROWS + lane;
        float acc[K], accw = 0.0f;
#pragma unroll
        for (int k = 0; k < K; k++) acc[k] = 0.0f;
        if (ia < g.na) {  // the same for the whole warp
            Shared &sm = reinterpret_cast<Shared *>(sm_warps)[warp];
            const VT *base[K];
            const int64_t voff = MULTI ? (int64_t)blockIdx.z * p.vol_stride : 0;
#pragma unroll
            for (int k = 0; k < K; k++)
                base[k] = PAIR && k == 2 ? nullptr : p.vol.zf[k] + (PAIR && k == 1 ? 2 : 1) * voff;
            const float z_half = (float)(g.nz / 2);
            const int nz = g.nz;
            float rz0, rz1;
            int wlo, whi;
            bool w_safe, w_narrow;
            {
                const float cphi = cosf(angle), sphi = sinf(angle);  // :23-24
                // lanes past the last row repeat its ray; nothing of them is stored
                const RayGeom r = ray_geom(cphi, sphi, ia, min(ib, g.nb - 1), g);
                const RayAxial ax = ray_axial(r, z_half, nz);
                w_safe = __all_sync(0xffffffffu, ax.zsafe);
                w_narrow = __all_sync(0xffffffffu, ax.narrow) && g.nzp % 2 == 0;
                // the warp's slabs: those where some ray meets the volume
                int lo, hi;
                ray_zrange(r, z_half, nz, lo, hi);
                wlo = __reduce_min_sync(0xffffffffu, lo);
                whi = __reduce_max_sync(0xffffffffu, hi);
                // the column's constants live in shared memory, read again
                // per table, so that the slab loop's registers hold the ray's own
                if (lane == 0) sm.ray = r;
                if (lane == 31) sm.rz_last = r.rz0;
                rz0 = r.rz0;
                rz1 = r.rz1;
            }
            const unsigned win0 = (unsigned)__cvta_generic_to_shared(&sm.win[0][0][0]);
            // the zeros behind the windows
            for (int i = lane; i < NST * S * 2; i += 32) {
                sts_zero4(win0 + i * W::BYTES + FPW * W::ES);
                if (PAIR) {
                    sts_zero4(win0 + i * W::BYTES + W::PAIRS + 2 * FPW * W::ES);
                    sts_zero4(win0 + i * W::BYTES + W::PAIRS + 2 * FPW * W::ES + 4);
                }
            }
            __syncwarp();
            const int bit = 1 << lane;
            int su_;
            {
                int sd;
                zf_strides(sm.ray.xdrive, g, su_, sd);
            }
            const int su = su_;
            const int64_t lane_off = (lane >> 4) * (int64_t)su + 2 * (lane & 15);
            const unsigned lane_dst = (lane >> 4) * W::BYTES + 2 * W::ES * (lane & 15);
            const int n = wlo <= whi ? whi - wlo + 1 : 0;  // slab i of the warp is wlo + i
            // a warp that is not narrow has no staged slab
            if (WIDE) {
#pragma unroll 1
                for (int i0 = 0; !w_narrow && i0 < n; i0 += 32)
                    fp_slabs_wide<K, ONES, VT, PAIR>(sm, g, wlo, i0, n, rz0, rz1, w_safe, base, nz,
                                                     z_half, acc, accw);
            }
            const int stages = !WIDE || w_narrow ? (n + S - 1) / S : 0;

            // Copies the windows of stage s (slabs s*S ..), filling the table
            // of 32 slabs first where the stage begins one.
            auto issue = [&](int s) {
                if (s < stages) {
                    const int i0 = s * S;
                    if (i0 % 32 == 0) {
                        const int i = i0 + lane;
                        const RayGeom rc = sm.ray;
                        int su, sd;
                        zf_strides(rc.xdrive, g, su, sd);
                        SlabCopy c;
                        int f;
                        float a, b, dc;
                        int zb;
                        slab_entry(rc, wlo + min(i, n - 1), su, sd, rc.rz0, sm.rz_last,
                                   WIDE || w_narrow, z_half, nz, c, f, a, b, dc, zb);
                        if (i >= n) {
                            f = 0;
                            c.pairs = 0;
                            a = b = 0.0f;
                        }
                        const unsigned in = __ballot_sync(0xffffffffu, (f & SC_IN) != 0);
                        const unsigned st = __ballot_sync(0xffffffffu, (f & SC_STAGE) != 0);
                        const unsigned slow = __ballot_sync(
                            0xffffffffu, (f & (SC_ANY | SC_STAGE)) == SC_ANY);
                        sm.copy[i & 63] = c;
                        sm.flags[i & 63] = f;
                        SlabPair &y = sm.pairs[(i & 63) >> 1];
                        y.a[i & 1] = a;
                        y.b[i & 1] = b;
                        y.dc[i & 1] = dc;
                        y.zb[i & 1] = zb;
                        if (lane == 0) sm.mask[(i0 >> 5) & 1] = make_uint4(in, st, slow, 0);
                        __syncwarp();
                    }
                    // no window of a warp that is not narrow is read (SC_STAGE), and
                    // at an odd pitch its copies would not be aligned
                    if (WIDE || w_narrow) {
                        const SlabCopy *const c = sm.copy + (i0 & 63);
                        const unsigned dst = win0 + s % NST * (S * 2 * W::BYTES);
#pragma unroll
                        for (int q = 0; q < S; q++)
                            window_copy<VT, PAIR>(dst + q * 2 * W::BYTES, base,
                                                  *reinterpret_cast<const int2 *>(c + q), lane,
                                                  bit, lane_off, lane_dst);
                    }
                }
                cp_async_commit();
            };

#pragma unroll 1
            for (int s = 0; s < NST - 1; s++) issue(s);
#pragma unroll 1
            for (int s = 0; s < stages; s++) {
                issue(s + NST - 1);
                cp_async_wait<NST - 1>();
                __syncwarp();
                const int i0 = s * S;
                const unsigned char(*const w)[2][W::BYTES] = sm.win + s % NST * S;
                const SlabPair *const y = sm.pairs + ((i0 & 63) >> 1);
                // the stage's bits of the table's masks (in, staged, slow)
                uint4 m = sm.mask[(i0 >> 5) & 1];
                constexpr unsigned ALL = (1u << S) - 1;
                m.x = m.x >> (i0 & 31) & ALL;
                m.y = m.y >> (i0 & 31) & ALL;
                m.z = m.z >> (i0 & 31) & ALL;
                if (m.x == ALL) {
                    MCSART_ON_FORM(0);
#pragma unroll
                    for (int q = 0; q < S; q += 2)
                        fp_pair_staged<K, ONES, true, VT, PAIR>(rz0, rz1, y[q / 2], true, true,
                                                                w[q][0], nz, z_half, acc, accw);
                } else if (m.z == 0) {
                    if (m.y == 0) continue;  // no staged slab: no ray meets the volume
                    MCSART_ON_FORM(1);
#pragma unroll
                    for (int q = 0; q < S; q += 2)
                        fp_pair_staged<K, ONES, false, VT, PAIR>(rz0, rz1, y[q / 2], m.y >> q & 1u,
                                                                 m.y >> (q + 1) & 1u, w[q][0], nz,
                                                                 z_half, acc, accw);
                } else {
#pragma unroll 1
                    for (int q = 0; q < S; q++) {
                        const int o = sm.copy[(i0 + q) & 63].o, f = sm.flags[(i0 + q) & 63];
                        if (!(f & SC_ANY)) continue;
                        const SlabPair &yq = y[q / 2];
                        RayGeom rc = sm.ray;
                        rc.rz0 = rz0;
                        rc.rz1 = rz1;
                        if ((WIDE || w_safe) && (f & SC_FAST) &&
                            fp_slab_direct<K, ONES, VT, PAIR>(
                                rz0, rz1, yq.dc[q & 1], yq.a[q & 1], yq.b[q & 1],
                                o - (yq.zb[q & 1] - MK_MAGIC_BITS), su, (f & SC_TWO) != 0,
                                base, nz, z_half, acc, accw)) {
                            MCSART_ON_FORM(2);
                            continue;
                        }
                        MCSART_ON_FORM(3);
                        fp_slab_general<K, ONES, VT, PAIR>(rc, g, wlo + i0 + q, base, z_half, acc,
                                                           accw);
                    }
                }
                __syncwarp();  // the stage's windows may be overwritten now
            }
        }
#pragma unroll
        for (int k = 0; k < K; k++) sm_s[k][lane][warp] = acc[k];
        if (ONES) sm_s[K][lane][warp] = accw;
    }

    if (p.bpcolA != nullptr) {
        // the following backprojector's per-column part, with its own sine
        // and cosine of the angle (src/cu_backprojection.cu:62-63): the same
        // device code, so the same bits as computing it there; spread over
        // all threads of the view's blocks
        const float bs = __sinf(angle), bc = __cosf(angle);
        const int64_t ncol = (int64_t)g.nx * g.ny;  // below 2^31
        const int64_t coff = MULTI ? (int64_t)blockIdx.z * ncol : 0;
        const int64_t nthr = (int64_t)gridDim.x * gridDim.y * FPC_THREADS;
        for (int64_t c = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * FPC_THREADS + t; c < ncol;
             c += nthr) {
            const unsigned cu = (unsigned)c, cy = cu / (unsigned)g.nx, cx = cu - cy * (unsigned)g.nx;
            const BPColumn col = bp_column<false>((int)cx, (int)cy, bc, bs, g);
            p.bpcolA[coff + c] = make_float4(col.amin, col.amax, col.rl, col.rr);
            p.bpcolB[coff + c] = col.r0;
        }
    }
    __syncthreads();

    // epilogue with the block's columns along the lanes, as the detector is stored
    double nb2 = 0.0, nr2 = 0.0;
#pragma unroll
    for (int e = t; e < FPC_ROWS * FPC_COLS; e += FPC_THREADS) {
        const int ecol = e % FPC_COLS, erow = e / FPC_COLS;
        const int ia = blockIdx.x * FPC_COLS + ecol, ib = by * FPC_ROWS + erow;
        if (ia >= g.na || ib >= g.nb) continue;
        const int64_t pix = ia + (int64_t)ib * g.na;
        // this view's cell
        const int64_t vpix = MULTI ? pix + (int64_t)blockIdx.z * g.na * g.nb : pix;
        const float s0 = sm_s[0][erow][ecol];
        if (p.mode == FP_PLAIN) {
            p.out[vpix] = s0;
            continue;
        }
        const float b = ldv(p.meas, vpix);
        // AUMISART.cu:206 host_add(proj, proj_temp, -1): proj += proj_temp * -1
        float res = __fmaf_rn(s0, -1.0f, b);
        float ones = ONES ? sm_s[ONES ? K : 0][erow][ecol] : 0.0f;
        if (p.mode == FP_MOTION) {
            // AUMISART.cu:260, + FP(img0)
            res = __fmaf_rn(sm_s[K > 1 ? 1 : 0][erow][ecol], 1.0f, res);
            if (K >= 3) ones = sm_s[K - 1][erow][ecol];  // FP(initial2(...)), :267-268
        }
        if (p.resid) p.resid[vpix] = res;
        // the backprojector's operands as the reference's texture reads
        // them; resid and the norms keep the residual itself
        p.bp_in[vpix] = make_float2(tex_texel(res), tex_texel(ones));
        nb2 += (double)b * (double)b;
        nr2 += (double)res * (double)res;
    }
    if (p.mode == FP_PLAIN) return;
    // block partial of the two squared norms, fixed-order reduction
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        nb2 += __shfl_down_sync(0xffffffffu, nb2, off);
        nr2 += __shfl_down_sync(0xffffffffu, nr2, off);
    }
    if (lane == 0) sm_norm[warp] = make_double2(nb2, nr2);
    __syncthreads();
    if (t == 0) {
        double tb = 0.0, tr = 0.0;
        for (int w = 0; w < FPC_THREADS / 32; w++) {
            tb += sm_norm[w].x;
            tr += sm_norm[w].y;
        }
        const int64_t vblk = MULTI ? (int64_t)blockIdx.z * gridDim.x * gridDim.y : 0;
        p.norm_part[vblk + by * gridDim.x + blockIdx.x] = make_double2(tb, tr);
    }
}

// Whether a call gains by the loop for warps that are not narrow: cells higher than
// ray_axial's bound at the volume's far side.
inline bool fp_wide(const Geom &g) {
    const float far = g.SO + 0.5f * (float)(g.nx > g.ny ? g.nx : g.ny);
    return g.db * far > 0.99f * g.SD;
}

// Launch of fp_ref_kernel, one block per FPC_COLS x FPC_ROWS detector cells and
// view.
template <typename VT, bool PAIR, int S, int NST> constexpr size_t fp_ref_smem() {
    return FPC_COLS * sizeof(FPShared<VT, PAIR, S, NST>);
}
template <int K, bool ONES, typename VT, typename MT, bool MULTI, int S, int NST, int MINB, bool PAIR,
          bool WIDE>
int launch_fp_form(mcsart_ctx *ctx, dim3 grid, const FPArgs<VT, K, MT> &a) {
    constexpr size_t smem = fp_ref_smem<VT, PAIR, S, NST>();
    const auto kernel = fp_ref_kernel<K, ONES, VT, MT, MULTI, S, NST, MINB, PAIR, WIDE>;
    // with the kernel's static arrays within the 48 KB of any launch
    static_assert(smem <= 44 * 1024, "a shape of more shared memory needs the limit raised");
    if (!ctx->label) ctx->label = "fp_ref_kernel";
    MC_LAUNCH(ctx, kernel, grid, dim3(FPC_THREADS), smem, a);
    return MCSART_OK;
}
// (the wide form in the built-in shape: its loop has no stages)
template <int K, bool ONES, typename VT, typename MT = VT, bool MULTI = false,
          int S = fp_stage<K>(), int NST = 2, int MINB = fp_min_blocks<K>(), bool PAIR = false>
int launch_fp_ref(mcsart_ctx *ctx, dim3 grid, const FPArgs<VT, K, MT> &a) {
    if (fp_wide(a.g))
        return launch_fp_form<K, ONES, VT, MT, MULTI, fp_stage<K>(), 2, fp_min_blocks<K>(), PAIR, true>(
            ctx, grid, a);
    return launch_fp_form<K, ONES, VT, MT, MULTI, S, NST, MINB, PAIR, false>(ctx, grid, a);
}

// ------------------------------------------------------------------------
// The projector from the x-fastest volume itself, a ray per thread, where there is
// no memory for the z-fastest copy: the plain loops, so the same bits (256x256x160,
// 512x384: 370-380 us against 113-119).  Grid (ceil(na / 128), nb).
static __global__ void __launch_bounds__(128) fp_nocopy_kernel(float *out, const float *img,
                                                               float angle, const Geom g) {
    const int ia = blockIdx.x * 128 + threadIdx.x, ib = blockIdx.y;
    if (ia >= g.na) return;
    const RayGeom r = ray_geom(cosf(angle), sinf(angle), ia, ib, g);  // :23-24
    const float z_half = (float)(g.nz / 2);
    int lo, hi;
    ray_zrange(r, z_half, g.nz, lo, hi);
    float acc[1] = {0.0f}, accw = 0.0f;
    const float *base[1] = {img};
    for (int d = lo; d <= hi; d++)
        fp_slab_loops<1, false, float, false>(r, g, d, base, r.xdrive ? g.nx : 1, r.xdrive ? 1 : g.nx,
                                              g.nx * g.ny, z_half, acc, accw);
    out[ia + (int64_t)ib * g.na] = acc[0];
}

// ------------------------------------------------------------------------
// Projector of the split summation modes: blockDim (32, groups), threadIdx.y =
// slab group of the same 32 rays.  The 32 lanes are 32 consecutive detector rows
// of one column (gridDim (na, ceil(nb/32), views)): they compute the column's
// in-plane footprint of 32 slabs at a time, one slab each, into a table of the
// warp's own, and then walk the slabs together, each lane adding its ray's axial
// part.  RAYS: 32 consecutive columns of one row (gridDim (ceil(na/32), nb,
// views)), each lane with its own footprints, for detectors whose rows would not
// fill the warps (split_rays).  Each slab's terms are summed first (in-plane
// voxel, then slice) and the slab sums added, plainly or with Kahan compensation.
// GEO64: FP64 geometry and weight sum (ray_geom64): every coordinate, box edge
// and overlap weight in FP64, the weights summed one by one; volume terms in FP32.
// Bound by instruction issue: FP64 operations, and divisions in FP32 geometry.
// 128x128x96, 256x192 detector, Kahan, FP64 geometry: 146 us with a thread
// computing its ray's footprints by itself, now 65; 256x256x160, 512x384, FP32
// geometry: 387, now 338.

// Whether the split-sum projector's lanes are columns: where rows would leave lanes
// idle and the shared footprints do not make up for it.  A ray with footprints of
// its own costs 1.3 times one without in FP32 geometry and twice in FP64 (each
// measured with full warps).  The kernel by events, rows against columns:
// 512x512x1 with a 1024x1 detector 97 and 42 us, 512x512x4 with 1024x4 130 and 56;
// a call at 256x256x160 with 512x33 87 and 64 us, and in FP64, which keeps the
// rows there, 100 against 123.
inline bool split_rays(const Geom &g, bool geom64) {
    const int64_t rows = (g.nb + 31) / 32 * 32, cols = (g.na + 31) / 32 * 32;
    return g.nb * cols * (geom64 ? 20 : 13) < rows * g.na * 10;
}
inline dim3 split_grid(const Geom &g, bool rays) {
    return rays ? dim3(div_up(g.na, 32), g.nb) : dim3(g.na, div_up(g.nb, 32));
}

// In-plane footprint of one slab: voxels u_lo .. u_lo + n - 1 (in the volume)
// with the first one's column at element `row`, the edges, the reciprocal width
// (GEO64; the width itself otherwise) and the first two weights.
template <typename R> struct SlabSplit {
    R lo, hi, inv, dc;
    R w0, w1;
    int row, u_lo, n;
};
__device__ __forceinline__ double overlap(double i, double lo, double hi) {
    return fmin(i + 1.0, hi) - fmax(i, lo);
}
__device__ __forceinline__ float overlap(float i, float lo, float hi) {
    return __fsub_rn(fminf(__fadd_rn(i, 1.0f), hi), fmaxf(i, lo));
}
// The quotient by the width, correctly rounded in both (inv: SlabSplit's).
__device__ __forceinline__ double split_weight(double i, double lo, double hi, double inv) {
    return mk_div64(overlap(i, lo, hi), hi - lo, inv);
}
__device__ __forceinline__ float split_weight(float i, float lo, float hi, float width) {
    return __fdiv_rn(overlap(i, lo, hi), width);
}

// (without the weights)
__device__ __forceinline__ SlabSplit<double> slab_edges(const RayGeom64 &r, int d, int su, int sd) {
    SlabSplit<double> e;
    e.dc = ((double)d + 0.5) - r.d_half - r.src_d;  // :52 / :105
    const double c0 = r.r0 * e.dc + r.u_off + r.u_half, c1 = r.r1 * e.dc + r.u_off + r.u_half;
    const double c2 = r.r2 * e.dc + r.u_off + r.u_half, c3 = r.r3 * e.dc + r.u_off + r.u_half;
    e.lo = fmin(fmin(c0, c1), fmin(c2, c3));
    e.hi = fmax(fmax(c0, c1), fmax(c2, c3));
    e.inv = 1.0 / (e.hi - e.lo);
    e.u_lo = max(0, __double2int_rd(e.lo));
    e.n = max(0, min(r.nu - 1, __double2int_rd(e.hi)) - e.u_lo + 1);
    e.row = e.u_lo * su + d * sd;
    return e;
}
__device__ __forceinline__ SlabSplit<float> slab_edges(const RayGeom &r, int d, int su, int sd) {
    SlabSplit<float> e;
    e.dc = __fsub_rn(__fsub_rn(__fadd_rn((float)d, 0.5f), r.d_half), r.src_d);  // :52 / :105
    // :54-63 / :107-116
    const float c0 = __fadd_rn(__fmaf_rn(r.r0, e.dc, r.u_off), r.u_half);
    const float c1 = __fadd_rn(__fmaf_rn(r.r1, e.dc, r.u_off), r.u_half);
    const float c2 = __fadd_rn(__fmaf_rn(r.r2, e.dc, r.u_off), r.u_half);
    const float c3 = __fadd_rn(__fmaf_rn(r.r3, e.dc, r.u_off), r.u_half);
    e.lo = fminf(fminf(c0, c1), fminf(c2, c3));
    e.hi = fmaxf(fmaxf(c0, c1), fmaxf(c2, c3));
    e.inv = __fsub_rn(e.hi, e.lo);
    e.u_lo = max(0, (int)floorf(e.lo));
    e.n = max(0, min(r.nu - 1, (int)floorf(e.hi)) - e.u_lo + 1);
    e.row = e.u_lo * su + d * sd;
    return e;
}

// The weight of the footprint's voxel i (:83 / :136).
template <typename R> __device__ __forceinline__ R slab_weight(const SlabSplit<R> &e, int i) {
    return split_weight((R)(e.u_lo + i), e.lo, e.hi, e.inv);
}

// Axial edges of a slab (:71-77 / :124-130, "ratio * xc + z1 + nz / 2", z1 = 0)
// and their slices, clamped to the volume; inv as SlabSplit's.
template <typename R> struct SplitZ {
    R lo, hi, inv;
    int z0, z1;
};
__device__ __forceinline__ SplitZ<double> split_z(double rz0, double rz1, double dc, double z_half,
                                                  int nz) {
    const double a = rz0 * dc + z_half, b = rz1 * dc + z_half;
    SplitZ<double> z;
    z.lo = fmin(a, b);
    z.hi = fmax(a, b);
    z.inv = 1.0 / (z.hi - z.lo);
    z.z0 = max(0, __double2int_rd(z.lo));
    z.z1 = min(nz - 1, __double2int_rd(z.hi));
    return z;
}
__device__ __forceinline__ SplitZ<float> split_z(float rz0, float rz1, float dc, float z_half, int nz) {
    const float a = __fadd_rn(__fmul_rn(rz0, dc), z_half), b = __fadd_rn(__fmul_rn(rz1, dc), z_half);
    SplitZ<float> z;
    z.lo = fminf(a, b);
    z.hi = fmaxf(a, b);
    z.inv = __fsub_rn(z.hi, z.lo);
    z.z0 = max(0, (int)floorf(z.lo));
    z.z1 = min(nz - 1, (int)floorf(z.hi));
    return z;
}

// One voxel's terms: FP32, or the FP64 weight rounded to FP32 and its sum in FP64.
template <int K, bool ONES, typename VT>
__device__ __forceinline__ void split_term(const VT *const *zf, int a, float wu, float wz, float *ss,
                                           float &sw) {
#pragma unroll
    for (int k = 0; k < K; k++) ss[k] = __fmaf_rn(__fmul_rn(ldv(zf[k], a), wu), wz, ss[k]);
    if (ONES) sw = __fmaf_rn(wu, wz, sw);
}
template <int K, bool ONES, typename VT>
__device__ __forceinline__ void split_term(const VT *const *zf, int a, double wu, double wz, float *ss,
                                           double &sw) {
    const double w = wu * wz;
    const float wf = (float)w;
#pragma unroll
    for (int k = 0; k < K; k++) ss[k] = __fmaf_rn(ldv(zf[k], a), wf, ss[k]);
    if (ONES) sw += w;
}

// Adds slab sum x to sum s, plainly or with Kahan compensation c.
template <int SUM> __device__ __forceinline__ void split_add(float &s, float &c, float x) {
    if (SUM == SUM_KAHAN) {
        const float y = x - c, t = s + y;
        c = (t - s) - y;
        s = t;
    } else {
        s += x;
    }
}

template <bool GEO64> struct SplitReal { using R = float; using Ray = RayGeom; };
template <> struct SplitReal<true> { using R = double; using Ray = RayGeom64; };

// Slabs [d0, d1) of the lane's ray: s[k], and sw (FP32 slab sums of FP32 weights,
// FP64 sum of FP64 weights); tab (not RAYS): 32 entries of the warp's own, whose
// rays have the same slabs.
template <int K, bool ONES, int SUM, bool GEO64, bool RAYS, typename VT>
__device__ __forceinline__ void split_slabs(const typename SplitReal<GEO64>::Ray &r,
                                            const FPVolumes<VT, K> &v, const Geom &g, int d0, int d1,
                                            SlabSplit<typename SplitReal<GEO64>::R> *tab, float *s,
                                            typename SplitReal<GEO64>::R &sw) {
    using R = typename SplitReal<GEO64>::R;
    static_assert(SUM != SUM_REF, "the reference order is fp_ref_kernel's");
    const int lane = threadIdx.x;
    int su, sd;
    zf_strides(r.xdrive, g, su, sd);
    const R z_half = (R)(g.nz / 2);
    float acc[K], cmp[K], cmpw = 0.0f;
    R accw = 0;
#pragma unroll
    for (int k = 0; k < K; k++) { acc[k] = 0.0f; cmp[k] = 0.0f; }
    for (int c0 = d0; c0 < d1; c0 += RAYS ? 1 : 32) {
        SlabSplit<R> own;
        if (RAYS) {
            own = slab_edges(r, c0, su, sd);
        } else {
            __syncwarp();
            if (c0 + lane < d1) {
                SlabSplit<R> e = slab_edges(r, c0 + lane, su, sd);
                e.w0 = slab_weight(e, 0);
                e.w1 = slab_weight(e, 1);
                tab[lane] = e;
            }
            __syncwarp();
        }
        const int m = RAYS ? 1 : min(32, d1 - c0);
        for (int j = 0; j < m; j++) {
            const SlabSplit<R> &e = RAYS ? own : tab[j];
            if (e.n == 0) continue;  // (not RAYS: the same for the whole warp)
            const SplitZ<R> z = split_z(r.rz0, r.rz1, e.dc, z_half, g.nz);
            if (z.z0 > z.z1) continue;
            const R wz0 = split_weight((R)z.z0, z.lo, z.hi, z.inv);  // :86 / :139
            const R wz1 = z.z1 > z.z0 ? split_weight((R)(z.z0 + 1), z.lo, z.hi, z.inv) : (R)0;
            float ss[K];
            R ssw = GEO64 ? accw : (R)0;  // FP64: straight on
#pragma unroll
            for (int k = 0; k < K; k++) ss[k] = 0.0f;
            for (int i = 0; i < e.n; i++) {
                const R wu = !RAYS && i == 0 ? e.w0 : !RAYS && i == 1 ? e.w1 : slab_weight(e, i);
                const int a = e.row + i * su;
                split_term<K, ONES>(v.zf, a + z.z0, wu, wz0, ss, ssw);
                if (z.z1 > z.z0) split_term<K, ONES>(v.zf, a + z.z0 + 1, wu, wz1, ss, ssw);
                for (int q = z.z0 + 2; q <= z.z1; q++)
                    split_term<K, ONES>(v.zf, a + q, wu, split_weight((R)q, z.lo, z.hi, z.inv), ss, ssw);
            }
#pragma unroll
            for (int k = 0; k < K; k++) split_add<SUM>(acc[k], cmp[k], ss[k]);
            if constexpr (ONES) {
                if constexpr (GEO64)
                    accw = ssw;
                else
                    split_add<SUM>(accw, cmpw, ssw);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < K; k++) s[k] = acc[k];
    sw = accw;
}

template <int K, bool ONES, int SUM, typename VT, typename MT = VT, bool GEO64 = false,
          bool RAYS = false>
__global__ void __launch_bounds__(256) fp_kernel(const FPArgs<VT, K, MT> p) {
    constexpr int NS = K + (ONES ? 1 : 0);
    extern __shared__ float sm_fp[];  // [groups][NS][32]
    __shared__ double sm_w64[GEO64 ? 8 : 1][32];  // GEO64: the groups' FP64 weight sums
    __shared__ SlabSplit<typename SplitReal<GEO64>::R> sm_tab[RAYS ? 1 : 8][32];
    const int lane = threadIdx.x;
    const Geom &g = p.g;
    const int ia = RAYS ? blockIdx.x * 32 + lane : blockIdx.x;
    const int ib = RAYS ? blockIdx.y : blockIdx.y * 32 + lane;
    const bool active = ia < g.na && ib < g.nb;
    const int groups = blockDim.y, grp = threadIdx.y;
    float s[K], sw = 0.0f;
    double sw64 = 0.0;
    {
        // lanes past the last row or column repeat its ray; nothing of them is stored
        const int row = min(ib, g.nb - 1), col = min(ia, g.na - 1);
        auto *const tab = sm_tab[RAYS ? 0 : grp];
        if constexpr (GEO64) {
            const RayGeom64 r = ray_geom64(p.cos64, p.sin64, col, row, g);
            const int per = (r.nd + groups - 1) / groups, d0 = grp * per, d1 = min(r.nd, d0 + per);
            split_slabs<K, ONES, SUM, true, RAYS, VT>(r, p.vol, g, d0, d1, tab, s, sw64);
        } else {
            const float angle = p.angles ? p.angles[blockIdx.z] : p.angle;
            const RayGeom r = ray_geom(cosf(angle), sinf(angle), col, row, g);  // :23-24
            const int per = (r.nd + groups - 1) / groups, d0 = grp * per, d1 = min(r.nd, d0 + per);
            split_slabs<K, ONES, SUM, false, RAYS, VT>(r, p.vol, g, d0, d1, tab, s, sw);
        }
    }
#pragma unroll
    for (int k = 0; k < K; k++) sm_fp[(grp * NS + k) * 32 + lane] = s[k];
    if (ONES) sm_fp[(grp * NS + K) * 32 + lane] = sw;
    if (GEO64) sm_w64[grp][lane] = sw64;
    __syncthreads();
    if (grp != 0) return;
    // fixed-order combination of the slab groups
    for (int q = 1; q < groups; q++) {
#pragma unroll
        for (int k = 0; k < K; k++) s[k] += sm_fp[(q * NS + k) * 32 + lane];
        if (ONES) sw += sm_fp[(q * NS + K) * 32 + lane];
        if (GEO64) sw64 += sm_w64[q][lane];
    }
    if (GEO64) sw = (float)sw64;
    const int64_t pix = ia + (int64_t)ib * g.na;
    double nb2 = 0.0, nr2 = 0.0;
    if (active) {
        if (p.mode == FP_PLAIN) {
            p.out[pix + (int64_t)blockIdx.z * g.na * g.nb] = s[0];
        } else {
            const float b = ldv(p.meas, pix);
            // AUMISART.cu:206 host_add(proj, proj_temp, -1): proj += proj_temp * -1
            float res = __fmaf_rn(s[0], -1.0f, b);
            float ones = ONES ? sw : 0.0f;
            if (p.mode == FP_MOTION) {
                res = __fmaf_rn(s[K > 1 ? 1 : 0], 1.0f, res);  // AUMISART.cu:260, + FP(img0)
                if (K >= 3) ones = s[K - 1];                   // FP(initial2(...)), :267-268
            }
            if (p.resid) p.resid[pix] = res;
            p.bp_in[pix] = make_float2(tex_texel(res), tex_texel(ones));
            nb2 = (double)b * (double)b;
            nr2 = (double)res * (double)res;
        }
    }
    if (p.mode == FP_PLAIN) return;
    // the block's partial of the two squared norms (one warp is left)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        nb2 += __shfl_down_sync(0xffffffffu, nb2, off);
        nr2 += __shfl_down_sync(0xffffffffu, nr2, off);
    }
    if (lane == 0) p.norm_part[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = make_double2(nb2, nr2);
}

// Launch of fp_kernel for one view, in FP32 or FP64 geometry (a: cos64, sin64 set).
template <int K, bool ONES, int SUM, typename VT, typename MT>
int launch_fp_split(mcsart_ctx *ctx, int groups, bool geom64, const FPArgs<VT, K, MT> &a) {
    const bool rays = split_rays(a.g, geom64);
    const dim3 grid = split_grid(a.g, rays), block(32, groups);
    const size_t smem = (size_t)groups * (K + 1) * 32 * sizeof(float);
    if (!ctx->label) ctx->label = "fp_kernel";
    if (geom64 && rays)
        MC_LAUNCH(ctx, (fp_kernel<K, ONES, SUM, VT, MT, true, true>), grid, block, smem, a);
    else if (geom64)
        MC_LAUNCH(ctx, (fp_kernel<K, ONES, SUM, VT, MT, true, false>), grid, block, smem, a);
    else if (rays)
        MC_LAUNCH(ctx, (fp_kernel<K, ONES, SUM, VT, MT, false, true>), grid, block, smem, a);
    else
        MC_LAUNCH(ctx, (fp_kernel<K, ONES, SUM, VT, MT, false, false>), grid, block, smem, a);
    return MCSART_OK;
}

}  // namespace mcsart
