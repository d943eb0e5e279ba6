// smcrt_render.cu -- the SDF voxel render (render_sub, src/sdfs/sdf_base.f90:302-346):
// the minimum over all regions of the scene's signed distance at every voxel of a
// samples(1) x samples(2) x samples(3) grid, stored FP32 in Fortran order (i fastest).
//
// Compiled without FMA contraction, so the FP64 evaluation follows the CPU
// restatement operation for operation.
//
// The render is bound by the arithmetic of its distances (a 256^3 image is 67
// MB, 10 us of HBM), so each CTA first finds which regions can be the minimum
// anywhere in its tile and its voxels evaluate those alone: one or two of the eight
// regions of layered_vessels.  Tiles of 16 x 8 x 16 voxels: small enough that few
// regions stay, large enough that the tile's own evaluations (one a region) are few
// beside its voxels', and 64 contiguous bytes a row.  A thread takes a column of
// voxels that share their x and y terms (column_min; FP64: four CTAs an SM by 64
// registers).  A 256^3 image of layered_vessels: FP64 500 us with every region at
// every voxel and 126 in tiles.  Images that tiles do not suit (use_tiles) take
// every region at every voxel.
#include <algorithm>
#include <cmath>

#include "smcrt_launch.h"

namespace smcrt {

namespace {

struct RenderGrid {
    long long n[3];
    double ns[3];  // nint(samples / 2), sdf_base.f90:320
    double w[3];   // extent / ns, sdf_base.f90:322
};

constexpr int kTx = 16, kTy = 8, kTz = 16;  // voxels of a tile
constexpr int kRenderBlock = 256;
constexpr int kPlanes = kRenderBlock / (kTx * kTy);  // planes of k a CTA covers at once
constexpr int kColumn = kTz / kPlanes;               // voxels of a thread, kPlanes apart in k

// One region's values at a thread's column of voxels, whose x and y are the same: a
// box's or sphere's x and y terms are formed once.  The sums are the general
// evaluation's, in its order (this unit has no contraction), so the bits are too.
template <class R>
__device__ __forceinline__ void column_min(const SceneT<R>& sc, int r, R x, R y, const R (&z)[kColumn],
                                           R (&d)[kColumn], bool first) {
    const DRegion<R>& g = sc.region[r];
    auto take = [&](int v, R e) { d[v] = first || e < d[v] ? e : d[v]; };
    if (g.shape == SHAPE_BOX) {
        const R dx = fabs(x + g.t[0]) - g.q[0], dy = fabs(y + g.t[1]) - g.q[1];
        const R mx = max_r(dx, (R)0), my = max_r(dy, (R)0);
        const R mxy = max_r(dx, dy), sxy = mx * mx + my * my;
#pragma unroll
        for (int v = 0; v < kColumn; ++v) {
            const R dz = fabs(z[v] + g.t[2]) - g.q[2];
            const R m = max_r(mxy, dz), mz = max_r(dz, (R)0);
            take(v, m <= (R)0 ? m : sqrt(sxy + mz * mz));
        }
    } else if (g.shape == SHAPE_SPHERE) {
        const R px = x + g.t[0], py = y + g.t[1], sxy = px * px + py * py;
#pragma unroll
        for (int v = 0; v < kColumn; ++v) {
            const R pz = z[v] + g.t[2];
            take(v, sqrt(sxy + pz * pz) - g.q[0]);
        }
    } else {
#pragma unroll 1
        for (int v = 0; v < kColumn; ++v) {
            R e = eval_region(sc, r, V3<R>{x, y, z[v]});
            // a NaN (a degenerate cone) is passed over, unless it is the first region's
            if (first && r > 0 && e != e) e = (R)INFINITY;
#pragma unroll
            for (int u = 0; u < kColumn; ++u)
                if (u == v) take(u, e);
        }
    }
}

// Voxel (i, j, k), 1-based, sits at ((i - ns1) w1, (j - ns2) w2, (k - ns3) w3),
// sdf_base.f90:326-331.  The coordinates are formed in FP64 as the reference's
// real(wp) arithmetic does; an FP32 render rounds the point, then evaluates.
//
// lip: the regions whose value changes by at most the distance moved (exact
// distances under rigid transforms, region_bound).  Such a region is nowhere in the
// tile the minimum when its value at the centre less the tile's half diagonal stays
// above another's value there plus the half diagonal (and the margin, which covers
// the rounding of all of these).
template <class R>
__global__ void __launch_bounds__(kRenderBlock, sizeof(R) == 8 ? 4 : 1) k_render(const __grid_constant__ SceneT<R> sc, const RenderGrid g,
                                                         unsigned lip, R margin, float* __restrict__ img) {
    __shared__ R s_d[kMaxRegions];
    const long long nx = (g.n[0] + kTx - 1) / kTx, ny = (g.n[1] + kTy - 1) / kTy, nz = (g.n[2] + kTz - 1) / kTz;
    const int t = threadIdx.x;
    const double half[3] = {0.5 * (kTx - 1) * g.w[0], 0.5 * (kTy - 1) * g.w[1], 0.5 * (kTz - 1) * g.w[2]};
    const R rho = (R)sqrt(half[0] * half[0] + half[1] * half[1] + half[2] * half[2]);
    const unsigned all = (1u << sc.nregions) - 1u;
    for (long long tile = blockIdx.x; tile < nx * ny * nz; tile += gridDim.x) {
        const long long i0 = tile % nx * kTx, j0 = tile / nx % ny * kTy, k0 = tile / (nx * ny) * kTz;
        if (t < sc.nregions) {
            const V3<R> c{(R)(((double)(i0 + 1) - g.ns[0]) * g.w[0] + half[0]),
                          (R)(((double)(j0 + 1) - g.ns[1]) * g.w[1] + half[1]),
                          (R)(((double)(k0 + 1) - g.ns[2]) * g.w[2] + half[2])};
            s_d[t] = lip >> t & 1u ? eval_region(sc, t, c) : (R)INFINITY;
        }
        __syncthreads();
        R least = (R)INFINITY;
        for (int r = 0; r < sc.nregions; ++r) least = fmin(least, s_d[r]);
        const R lim = least + (R)2 * rho + margin;
        unsigned keep = all & ~lip;
        for (int r = 0; r < sc.nregions; ++r)
            if (!(s_d[r] > lim)) keep |= 1u << r;
        __syncthreads();  // s_d is free for the next tile
        const int i = t % kTx, j = t / kTx % kTy;
        if (i0 + i < g.n[0] && j0 + j < g.n[1]) {
            const R x = (R)(((double)(i0 + i + 1) - g.ns[0]) * g.w[0]);
            const R y = (R)(((double)(j0 + j + 1) - g.ns[1]) * g.w[1]);
            const long long k1 = k0 + t / (kTx * kTy);
            R z[kColumn], d[kColumn];
#pragma unroll
            for (int v = 0; v < kColumn; ++v) z[v] = (R)(((double)(k1 + v * kPlanes + 1) - g.ns[2]) * g.w[2]);
            // minval(ds), sdf_base.f90:332-336
            for (unsigned m = keep; m; m &= m - 1u) column_min(sc, __ffs(m) - 1, x, y, z, d, m == keep);
#pragma unroll
            for (int v = 0; v < kColumn; ++v)
                if (k1 + v * kPlanes < g.n[2]) img[i0 + i + g.n[0] * (j0 + j + g.n[1] * (k1 + v * kPlanes))] = (float)d[v];
        }
    }
}

// Every region at every voxel: one thread per voxel, consecutive threads on
// consecutive i, so each warp writes 128 contiguous bytes of the image.
template <class R>
__global__ void __launch_bounds__(kRenderBlock) k_render_voxels(const __grid_constant__ SceneT<R> sc, const RenderGrid g,
                                                                float* __restrict__ img) {
    const long long total = g.n[0] * g.n[1] * g.n[2];
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < total; v += stride) {
        const long long i = v % g.n[0], jk = v / g.n[0], j = jk % g.n[1], k = jk / g.n[1];
        const V3<R> p{(R)(((double)(i + 1) - g.ns[0]) * g.w[0]), (R)(((double)(j + 1) - g.ns[1]) * g.w[1]),
                      (R)(((double)(k + 1) - g.ns[2]) * g.w[2])};
        // minval(ds), sdf_base.f90:332-336
        R d = eval_region(sc, 0, p);
        for (int r = 1; r < sc.nregions; ++r) {
            const R e = eval_region(sc, r, p);
            d = e < d ? e : d;
        }
        img[v] = (float)d;
    }
}

// Whether an image is rendered in tiles.  In us, every voxel against tiles:
// - enough tiles for the SMs (2.5 each): layered_vessels, FP64, 96^3 (432 tiles) 50
//   against 47, 80^3 (250) 43 against 56;
// - little padding: whole tiles are computed, so that a slice of 1024 x 1024 x 1 voxels
//   (1/16 full) takes 55 against 617; 1024 x 1024 x 24 (3/4 full) 734 against 702 for
//   layered_vessels but 225 against 259 for sphere_water;
// - regions that tiles can leave out.  Where all can (lip), a thread's columns share
//   their terms too.  The others (folds, modifiers) cost a column more than the same
//   voxels alone: eggs, FP64, 256^3, 399 against 481; a scene with two such regions of
//   seven 691 against 599 in FP64, 406 against 486 in FP32;
// - more than one tile along each axis: the only tile spans the scene and leaves little
//   out.  1024 x 1024 x 16: layered_vessels (8 regions) 501 against 558 and in FP32 312
//   against 421, but sphere_water (3 regions) 155 against 131 by its columns alone.
bool use_tiles(const smcrt_scene* scene, const RenderGrid& g, int nlip, bool fp64, long long tiles, int nsm) {
    const int n = scene->nregions;
    const long long total = g.n[0] * g.n[1] * g.n[2];
    if (2 * tiles < 5LL * nsm || 5 * total < 4 * tiles * (kTx * kTy * kTz)) return false;
    const bool thick = g.n[0] > kTx && g.n[1] > kTy && g.n[2] > kTz;
    if (nlip == n) return thick || n <= 4;
    return fp64 && thick && 2 * nlip > n;
}

template <class R>
cudaError_t render_t(const smcrt_scene* scene, const RenderGrid& g, float* d_img, int nsm, cudaStream_t s) {
    SceneT<R> sc;
    fill_scene(sc, scene);
    // the regions that may be left out, and a margin far above the rounding of values
    // and coordinates (and of a transform that is rigid to 1e-9)
    unsigned lip = 0;
    int nlip = 0;
    double scale = 1.0;
    for (int a = 0; a < 3; ++a) scale = std::fmax(scale, std::fabs(g.w[a]) * (double)(g.n[a] + 1));
    for (int r = 0; r < scene->nregions; ++r) {
        double c[3], rad;
        if (!region_bound(scene, r, c, &rad)) continue;
        lip |= 1u << r;
        ++nlip;
        scale = std::fmax(scale, std::fabs(c[0]) + std::fabs(c[1]) + std::fabs(c[2]) + rad);
    }
    const R margin = (R)((sizeof(R) == 4 ? 1e-4 : 1e-7) * scale);
    const long long tiles = ((g.n[0] + kTx - 1) / kTx) * ((g.n[1] + kTy - 1) / kTy) * ((g.n[2] + kTz - 1) / kTz);
    if (!use_tiles(scene, g, nlip, sizeof(R) == 8, tiles, nsm)) {
        const long long want = (g.n[0] * g.n[1] * g.n[2] + kRenderBlock - 1) / kRenderBlock;
        const int blocks = (int)std::min(want, 16LL * nsm);  // a few resident CTAs per SM, grid-stride beyond
        k_render_voxels<R><<<blocks, kRenderBlock, 0, s>>>(sc, g, d_img);
        return cudaGetLastError();
    }
    const int blocks = (int)std::min(tiles, 8LL * nsm);  // resident CTAs, grid-stride beyond
    k_render<R><<<blocks, kRenderBlock, 0, s>>>(sc, g, lip, margin, d_img);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_render(int precision, const smcrt_scene* scene, const int samples[3], const double extent[3],
                          float* d_img, int nsm, cudaStream_t s) {
    RenderGrid g;
    for (int a = 0; a < 3; ++a) {
        g.n[a] = samples[a];
        // nint rounds half away from zero: nint(n / 2) = (n + 1) / 2 for n >= 1
        g.ns[a] = (double)((samples[a] + 1) / 2);
        g.w[a] = extent[a] / g.ns[a];
    }
    if (g.n[0] * g.n[1] * g.n[2] == 0) return cudaSuccess;
    return precision == SMCRT_FP64 ? render_t<double>(scene, g, d_img, nsm, s)
                                   : render_t<float>(scene, g, d_img, nsm, s);
}

}  // namespace smcrt
