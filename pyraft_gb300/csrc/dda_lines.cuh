// dda_lines.cuh -- the rays of the DDA's line sums (dda_lines.cu) that are not
// summed as trapezoids: those of axis-aligned views, and those that meet or
// pass a non-finite pixel.
#pragma once

#include "dda.cuh"
#include "ss_tiles.cuh"

namespace rg {

// An axis-aligned view and, for each of its rays, the lines it meets: lines
// lo .. hi lie in pixel ja below line nc, in jb above it, and at nc by the
// parts wa and wb (ja, jb outside the line: nothing).
struct DLAxis {
    float sigma, sigma_lo;
    int view, fast_i;
};
struct __align__(16) DLRay {
    int lo, hi, nc, ja, jb;
    float wa, wb;
    int pad;
};
static_assert(sizeof(DLRay) == 32, "DLRay layout");

// What a Radon kernel needs for those rays.
struct DLArgs {
    DDAGeom g;
    const double *cs;                  // cos, sin of the views
    const float2 *prow, *pcol;         // the image's line pairs
    int nax;
    const DLAxis *axis;
    const DLRay *rays;
};

// The ray sum of ray k of view j by the walk.  A pair's difference carries a
// non-finite pixel to rays that only pass beside it, so every ray whose line
// sum is not finite is walked instead: it meets the pixels that the walk
// visits, no others.  The walk reads the line pairs too: the image may lie in
// memory that other CTAs store rays to by now.
inline __device__ __noinline__ float dl_walk_ray(const DLArgs &a, int k, int j)
{
    const DDAGeom &g = a.g;
    const double dts = __ddiv_rn(__dsub_rn(g.sbr_y, g.stl_y), (double)(g.R - 1));
    DDA it;
    dda_set_image(it, g.lines, g.columns, g.itl_x, g.itl_y, g.ibr_x, g.ibr_y);
    dda_set_theta(it, a.cs[2 * j], a.cs[2 * j + 1]);
    dda_set_t<kDdaSigma32>(it, __dadd_rn(g.stl_y, __dmul_rn((double)k, dts)));
    float acc = 0.f, comp = 0.f;
    dda_walk<kDdaSigma32>(it, 2 * (g.lines + g.columns) + 8, 0,
                          [&](int pi, int pj, float sg, int) {
        const float x = __ldg(&a.prow[(size_t)pi * pairs_pitch(g.columns) + 1 + pj].x) * sg;
        const float y = x - comp, t = acc + y;
        comp = (t - acc) - y;
        acc = t;
    });
    return acc - comp;
}

// The walks of rays k0 + 8 m (bit m of mask) of view j, stored over their line
// sums; a kernel's last act, so that it keeps no registers across the walks.
template <int EPI>
__device__ __noinline__ void dl_walk_rays(const DLArgs &a, unsigned mask, int k0, int j,
                                          float *__restrict__ out, long long ovs, long long ors,
                                          const float *__restrict__ y_am, int y_ld)
{
    for (int m = 0; m < 4; ++m)
        if (mask >> m & 1) {
            const int k = k0 + 8 * m;
            out[j * ovs + k * ors] =
                radon_epilogue(EPI, dl_walk_ray(a, k, j), y_am, (size_t)j * y_ld + k);
        }
}

// Axis-aligned ray e (of nax R) by one warp: its lines are runs of one column's
// or row's pairs.  Every lane returns the sum.
__device__ __forceinline__ float dl_axis_ray(const DLArgs &a, int e, const DLAxis &ax, int k)
{
    const int lane = threadIdx.x & 31;
    const DLRay r = a.rays[e];
    const int ne = ax.fast_i ? a.g.columns : a.g.lines;
    const size_t pitch = pairs_pitch(ax.fast_i ? a.g.lines : a.g.columns);
    const float2 *__restrict__ pairs = ax.fast_i ? a.pcol : a.prow;    // lines across the ray
    float sum = 0.f, c = 0.f;
    if ((unsigned)r.ja < (unsigned)ne) {
        const float2 *p = pairs + (size_t)r.ja * pitch + 1;
        const int end = min(r.hi + 1, r.nc);
#pragma unroll 8
        for (int i = r.lo + lane; i < end; i += 32) kahan_add(sum, c, p[i].x);
        if (lane == 0 && r.nc <= r.hi) kahan_add(sum, c, r.wa * p[r.nc].x);
    }
    if (r.nc <= r.hi && (unsigned)r.jb < (unsigned)ne) {
        const float2 *p = pairs + (size_t)r.jb * pitch + 1;
        for (int i = r.nc + 1 + lane; i <= r.hi; i += 32) kahan_add(sum, c, p[i].x);
        if (lane == 0) kahan_add(sum, c, r.wb * p[r.nc].x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        two_sum_add(sum, c, __shfl_xor_sync(0xffffffffu, sum, o), __shfl_xor_sync(0xffffffffu, c, o));
    const float val = fmaf(sum, ax.sigma, fmaf(sum, ax.sigma_lo, -c * ax.sigma));
    return isfinite(val) ? val : dl_walk_ray(a, k, ax.view);
}

// The axis-aligned rays of CTA `cta` (256 threads, 8 rays).
template <int EPI>
__device__ __forceinline__ void dl_axis_cta(const DLArgs &a, int cta, float *__restrict__ out,
                                            long long ovs, long long ors,
                                            const float *__restrict__ y_am, int y_ld)
{
    const int e = cta * 8 + (threadIdx.x >> 5);
    if (e >= a.nax * a.g.R) return;
    const int v = e / a.g.R, k = e - v * a.g.R;
    const DLAxis ax = a.axis[v];
    const float val = dl_axis_ray(a, e, ax, k);
    if ((threadIdx.x & 31) == 0)
        out[ax.view * ovs + k * ors] = radon_epilogue(EPI, val, y_am, (size_t)ax.view * y_ld + k);
}

}  // namespace rg
