// Checks fp_ref_kernel (mcsart_b200/csrc/projector.cuh) on the geometries read, in each
// storage type, at the volume pitch given (Geom::nzp): every asynchronous copy's
// addresses are aligned to its size, and every ray's sum has the bits of the
// reference's plain loops (fp_slab_general on every slab, a thread per ray).
// A geometry is a line nx ny nz nzp na nb SO SD da db ai bi angle.  Prints for each two
// counts, misaligned copies and rays that differ, and how often a warp took each of
// the forms: stages inside the volume, stages at its edge, slabs of narrow warps by at
// most two slices, by the general loops, slabs of other warps by at most three
// slices, by the general loops.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

__device__ unsigned long long g_misaligned;
#define MCSART_ON_COPY(dst, src, n)                                       \
    do {                                                                  \
        if ((((unsigned long long)(src)) | (dst)) & ((n) - 1))            \
            atomicAdd(&g_misaligned, 1ull);                               \
    } while (0)
__device__ unsigned long long g_forms[6];
#define MCSART_ON_FORM(form)                                              \
    do {                                                                  \
        if (threadIdx.x % 32 == 0) atomicAdd(&g_forms[form], 1ull);       \
    } while (0)
#include "projector.cuh"

using namespace mcsart;

template <int K, bool ONES, bool PAIR, typename VT>
__global__ void plain_kernel(const FPArgs<VT, K, VT> p, float *sums) {
    const Geom &g = p.g;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= (int64_t)g.na * g.nb) return;
    const int ia = (int)(i % g.na), ib = (int)(i / g.na);
    const RayGeom r = ray_geom(cosf(p.angle), sinf(p.angle), ia, ib, g);
    const VT *base[K];
    for (int k = 0; k < K; k++) base[k] = p.vol.zf[k];
    float acc[K], accw = 0.0f;
    for (int k = 0; k < K; k++) acc[k] = 0.0f;
    for (int d = 0; d < r.nd; d++)
        fp_slab_general<K, ONES, VT, PAIR>(r, g, d, base, (float)(g.nz / 2), acc, accw);
    for (int k = 0; k < K; k++) sums[i * 4 + k] = acc[k];
    sums[i * 4 + 3] = accw;
}

template <typename VT> __global__ void fill_kernel(VT *v, int64_t n, int nz, int nzp, unsigned seed) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        unsigned h = (unsigned)i * 2654435761u + seed;
        h ^= h >> 15; h *= 2246822519u; h ^= h >> 13;
        v[i] = cvt<VT>(i % nzp < nz ? (float)(h >> 8) * 0x1p-24f - 0.25f : 0.0f);
    }
}
// (first volume, pairs of the second and third; zero behind the depth)
template <typename VT> __global__ void fill_pairs(VT *v, int64_t n, int nz, int nzp, unsigned seed) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        unsigned h = (unsigned)i * 3266489917u + seed;
        h ^= h >> 16; h *= 668265263u; h ^= h >> 14;
        v[i] = cvt<VT>(i / 2 % nzp < nz ? (float)(h >> 8) * 0x1p-24f - 0.25f : 0.0f);
    }
}

static unsigned bits(float f) { unsigned u; memcpy(&u, &f, 4); return u; }

#define CHECK(x)                                                                     \
    do {                                                                             \
        cudaError_t e_ = (x);                                                        \
        if (e_ != cudaSuccess) {                                                     \
            fprintf(stderr, "%s: %s\n", #x, cudaGetErrorString(e_));                 \
            exit(1);                                                                 \
        }                                                                            \
    } while (0)

// (FP_IMAGE and FP_MOTION give the sums as residual and pair of a zero measurement:
//  one volume with the weights' sum, or three volumes)
template <int K, typename VT, bool WIDE = true> long long run(const Geom &g, float angle) {
    constexpr bool ONES = K == 1, PAIR = K == 3;
    const int64_t n = (int64_t)g.nx * g.ny * g.nzp, np = (int64_t)g.na * g.nb;
    VT *v0, *v1, *meas;
    float *sums, *resid;
    float2 *pair;
    double2 *part;
    const dim3 grid(div_up(g.na, FPC_COLS), div_up(g.nb, FPC_ROWS), 1);
    CHECK(cudaMalloc(&v0, n * sizeof(VT)));
    CHECK(cudaMalloc(&v1, 2 * n * sizeof(VT)));
    CHECK(cudaMalloc(&meas, np * sizeof(VT)));
    CHECK(cudaMalloc(&sums, np * 4 * sizeof(float)));
    CHECK(cudaMalloc(&resid, np * sizeof(float)));
    CHECK(cudaMalloc(&pair, np * sizeof(float2)));
    CHECK(cudaMalloc(&part, (size_t)grid.x * grid.y * sizeof(double2)));
    CHECK(cudaMemset(meas, 0, np * sizeof(VT)));
    fill_kernel<VT><<<512, 256>>>(v0, n, g.nz, g.nzp, 1u);
    fill_pairs<VT><<<512, 256>>>(v1, 2 * n, g.nz, g.nzp, 2u);
    FPArgs<VT, K, VT> a{};
    a.vol.zf[0] = v0;
    if (K == 3) a.vol.zf[K > 1 ? 1 : 0] = v1;
    a.g = g;
    a.angle = angle;
    a.mode = K == 1 ? FP_IMAGE : FP_MOTION;
    a.meas = meas;
    a.resid = resid;
    a.bp_in = pair;
    a.norm_part = part;
    plain_kernel<K, ONES, PAIR, VT><<<div_up(np, 128), 128>>>(a, sums);
    constexpr size_t smem = fp_ref_smem<VT, PAIR, fp_stage<K>(), 2>();
    fp_ref_kernel<K, ONES, VT, VT, false, fp_stage<K>(), 2, fp_min_blocks<K>(), PAIR, WIDE>
        <<<grid, FPC_THREADS, smem>>>(a);
    CHECK(cudaDeviceSynchronize());
    std::vector<float> s(np * 4), r(np);
    std::vector<float2> q(np);
    CHECK(cudaMemcpy(s.data(), sums, np * 16, cudaMemcpyDeviceToHost));
    CHECK(cudaMemcpy(r.data(), resid, np * 4, cudaMemcpyDeviceToHost));
    CHECK(cudaMemcpy(q.data(), pair, np * 8, cudaMemcpyDeviceToHost));
    long long bad = 0;
    for (int64_t i = 0; i < np; i++) {
        const float *t = &s[i * 4];
        // resid = -s0 (+ s1), the pair's second the weights' sum or s2
        const float res = K == 1 ? fmaf(t[0], -1.0f, 0.0f) : fmaf(t[1], 1.0f, fmaf(t[0], -1.0f, 0.0f));
        if (bits(r[i]) != bits(res) || bits(q[i].y) != bits(K == 1 ? t[3] : t[2])) bad++;
    }
    for (void *x : {(void *)v0, (void *)v1, (void *)meas, (void *)sums, (void *)resid, (void *)pair, (void *)part})
        CHECK(cudaFree(x));
    return bad;
}

int main() {
    Geom g;
    float angle;
    while (scanf("%d %d %d %d %d %d %f %f %f %f %f %f %f", &g.nx, &g.ny, &g.nz, &g.nzp, &g.na, &g.nb,
                 &g.SO, &g.SD, &g.da, &g.db, &g.ai, &g.bi, &angle) == 13) {
        unsigned long long mis = 0, f[6] = {};
        CHECK(cudaMemcpyToSymbol(g_misaligned, &mis, sizeof(mis)));
        CHECK(cudaMemcpyToSymbol(g_forms, f, sizeof(f)));
        const long long bad = run<1, float>(g, angle) + run<3, float>(g, angle) +
                              run<1, __half>(g, angle) + run<3, __nv_bfloat16>(g, angle) +
                              run<1, float, false>(g, angle);
        CHECK(cudaMemcpyFromSymbol(&mis, g_misaligned, sizeof(mis)));
        CHECK(cudaMemcpyFromSymbol(f, g_forms, sizeof(f)));
        printf("%llu %lld %llu %llu %llu %llu %llu %llu\n", mis, bad, f[0], f[1], f[2], f[3], f[4], f[5]);
    }
    return 0;
}
