// dda_lines.cu -- the DDA projector pair as interpolated line sums.
//
// The walk of raft_ddaiterator (raft/raft_ddaiterator.c:16-257) takes, on
// every line of its fast axis, the one or two pixels that the ray meets there
// and the lengths of its parts in them.  On square pixels those lengths are
// known without walking: on line i the ray's centre lies at x = x0 + k rk + i
// ri (pixels of the line; k the ray), it sweeps |ri| <= 1 pixels there, and
// the strip [u, u + |ri|) with u = x + 1/2 - |ri| / 2 = n + f puts
//     w = sat(1 - (1 - f) / |ri|)
// of the line's length sigma into pixel n + 1 and the rest into n.  So the
// ray sum is sigma * sum_i (p[n] + w (p[n+1] - p[n])), pixels outside the
// image being zero: the slant-stack Radon's line sum with a trapezoid in
// place of the linear weight, and its transpose a gather with
//     W(k) = sat((a + 1) / 2 - a |rk| |k - kappa|),   a = 1 / |ri|,
// kappa the ray position of the pixel's centre.  A walk is a serial chain of
// 64-bit integer steps (about 120 instructions a line, one L1 load or L2
// atomic a pixel); here all lines are independent, take one shared-memory
// load each, and the transpose needs no atomics.  2048^2 x 1800 on one
// GB300: Radon 25.0 -> 2.30 ms (issue-bound, as the slant-stack's), transpose
// 28.0 -> 2.05 ms (74 % of the shared-memory rate); 1024^2 x 720: 2.73 ->
// 0.26 and 3.2 -> 0.25 ms.  The normalised backprojection (A^T s / A^T 1, two
// FP64 atomics a pixel in the walk) keeps both sums in two FP32 numbers in the
// same gather: 68.8 -> 6.4 ms, 512^2 x 360 1.11 -> 0.14 ms.  Error against 64 bits
// (rel-L2): Radon 4.1e-8 -> 2.6e-8, transpose 4.4e-7 -> 8e-8, normalised 2.5e-8
// (the rounding of its result) as before.
//
// The walk decides in FP64, so it and these sums take the same pixels
// except where a decision falls within rounding of a tie; the ray sum is
// continuous there (the length in question goes to zero).  The exception is
// a ray that runs along a pixel boundary: views within 2^-30 of an axis
// (theta = 0, pi / 2, pi) are therefore taken from the walk itself, whose
// entry pixel and single possible crossing the plan holds per ray (DLRay).
// A ray through the corner where it enters the image may be lost by the walk's
// rounding (lost_ray): the Radon walks it, the transpose leaves its sample out,
// and the normalised backprojection of such a scan walks.
// Plans with views between 2^-30 and 2^-14 of an axis or with more than
// kDlAxisMax axis-aligned ones, pixels that are not square (where the walk
// departs from the geometry), images of more than 2097120 lines or columns (the
// grids' limit) or positions beyond 2^22 keep the walking kernels, and a ray
// whose line sum is not finite is walked (dl_walk_ray).
//
// Positions are Q24.40 (origins and steps within 2^-41 of a sample; at
// 4096 lines and rays within 2e-9), rounded to Q9.23 once per strip or pixel
// column.
#include <cuda.h>
#include <math.h>
#include <stdlib.h>

#include <algorithm>
#include <climits>
#include <vector>

#include "dda_lines.cuh"
#include "tma.cuh"

namespace rg {

namespace {

constexpr int kDlQ = 40;
constexpr int kDlBox = 256;                // widest TMA box (entries)
constexpr int kDlSlots = 16;               // views per staged chunk (most)

// Forms of the transpose (DLPlan::gather).
constexpr int kDlHalf = 1;      // half-turn pairs, two taps
constexpr int kDlTaps = 2;      // four taps
constexpr int kDlQuarter = 3;   // half-turn pairs of views and their reflections, two taps
// The partner windows of kDlQuarter lie this far behind the views' (bytes), an
// immediate of their loads.
constexpr int kDlPartner = 24576;

// Most axis-aligned views of a plan, which holds 32 bytes for each of their rays (a
// scan over 2 pi has five): a scan of nothing else would hold as much as the
// sinogram eight times over.
constexpr int kDlAxisMax = 16;

// Sums a thread keeps per row.
__host__ __device__ constexpr int dl_sums(int form)
{
    return form == kDlTaps ? 1 : form == kDlHalf ? 2 : 4;
}

bool to_q40(double v, long long &out)
{
    const double s = v * 1099511627776.0;
    if (!(fabs(s) < 4.0e18)) return false;
    out = llrint(s);
    return true;
}

// ----------------------------------------------------------------------------
// Plan

DLRay axis_ray(const DDA &it)
{
    DLRay r = {1, 0, INT_MAX, -1, -1, 0.f, 0.f, 0};
    if (dda_end(it)) return r;
    const int nl = it.fast_is_i ? it.lines : it.columns;
    const int line = it.fast_is_i ? it.i : it.j, s = it.fast_is_i ? it.j : it.i;
    const bool up = it.Delta_fast > 0;
    const int last = up ? nl - 1 : 0;
    int before = s, after = s, cross = INT_MAX;
    double wbefore = 1.0, wafter = 0.0;
    if (it.slow_move) {                               // the first line is split
        cross = line;
        wbefore = it.sigma / it.sigma_tilde;
        after = s + it.Delta_slow;
        wafter = 1.0 - wbefore;
    } else if (it.sigma != it.sigma_tilde) {          // enters through a side
        cross = line;
        before = -1;
        wbefore = 0.0;
        wafter = it.sigma / it.sigma_tilde;
    } else {
        // the walk's epsilon adds, as many at a time as round alike (the
        // sum moves by the same multiple of its ulp until it changes binade)
        double e = it.epsilon;
        const double u = it.epsilon_update, d = it.delta_slow;
        const int rem = up ? last - line : line - last;
        for (int done = 0, iter = 0; done < rem && iter < 256; ++iter) {
            const double n = rn_add(e, u);
            if (n > d) {
                cross = up ? line + done + 1 : line - done - 1;
                wbefore = (d - e) / u;                // as the walking sums take it
                after = s + it.Delta_slow;
                wafter = 1.0 - wbefore;
                break;
            }
            const double inc = n - e;
            if (!(inc > 0.0)) break;
            const double k = std::min(floor((d - n) / inc) - 1.0, (double)(rem - done - 1));
            const int jump = k > 0.0 ? (int)k : 0;
            e = n + jump * inc;
            done += 1 + jump;
        }
    }
    r.lo = up ? line : last;
    r.hi = up ? last : line;
    r.nc = cross;
    r.ja = up || cross == INT_MAX ? before : after;
    r.jb = up ? after : before;
    r.wa = (float)(up ? wbefore : wafter);
    r.wb = (float)(up ? wafter : wbefore);
    return r;
}

// The ray of the view set in `it` that the walk loses, or -1.  The walk takes a
// ray's entry side by comparing where it meets the two lines that bound the
// image's entry corner, then its entry pixel by rounding; for a ray through
// that corner the rounding may put the pixel outside, and the walk ends before
// it began, although the ray crosses the image (the diagonal of theta = 3 pi / 4
// on an even grid).  Every other ray enters through one side's inside, where
// a pixel more or less of rounding is a length of zero.
int lost_ray(const DDA &it, const DDAGeom &g, double dt)
{
    const double k = ((it.x0 * it.cos_theta + it.y0 * it.sin_theta) - g.stl_y) / dt;
    const double r = rint(k);
    if (!(r >= 0.0 && r <= g.R - 1) || fabs(k - r) > 1e-6) return -1;
    DDA ray = it;
    dda_set_t<kDdaExact>(ray, rn_add(g.stl_y, rn_mul(r, dt)));
    return dda_end(ray) ? (int)r : -1;
}

}  // namespace

void dl_plan_free(DLPlan &q)
{
    ss_plan_free(q.p);
    if (q.d_axis) cudaFree(q.d_axis);
    q.d_axis = nullptr;
    q.ok = false;
    q.gather = 0;
}

size_t dl_axis_bytes(const DLPlan &q)
{
    return (size_t)q.nax * (sizeof(DLAxis) + sizeof(DLRay) * (size_t)q.g.R +
                            sizeof(int2) * (size_t)q.ax_ne);
}

int dl_plan_build(DLPlan &q, const DDAGeom &g, const double *cs, const double *d_cs, int stride,
                  int first)
{
    q.ok = false;
    q.gather = 0;
    q.lost = false;
    q.g = g;
    q.first = first;
    q.stride = stride;
    const int L = g.lines, C = g.columns, R = g.R;
    const double dx = (g.ibr_x - g.itl_x) / (C - 1), dy = (g.ibr_y - g.itl_y) / (L - 1);
    const double dt = rn_div(rn_sub(g.sbr_y, g.stl_y), (double)(R - 1));
    if (!dl_sizes_ok(L, C, R) || !(fabs(dx) > 0.0) || !(fabs(dt) > 0.0) ||
        !(fabs(fabs(dx) - fabs(dy)) <= 1e-12 * fabs(dx)))
        return RG_OK;
    std::vector<View> hv;
    std::vector<DLAxis> ax;
    std::vector<DLRay> rays;
    DDA it;
    dda_set_image(it, L, C, g.itl_x, g.itl_y, g.ibr_x, g.ibr_y);
    double hmax = 0.0, wr[2] = {0.0, 0.0};
    for (int j = first; j < g.A; j += stride) {
        const double c = cs[2 * j], s = cs[2 * j + 1];
        dda_set_theta(it, c, s);
        const double u = it.epsilon_update / it.delta_slow;
        if (u < 9.3132257461547852e-10) {             // 2^-30
            if ((int)ax.size() == kDlAxisMax) return RG_OK;
            const float sg = (float)it.sigma_tilde;
            ax.push_back(DLAxis{sg, (float)(it.sigma_tilde - (double)sg), j, it.fast_is_i});
            for (int k = 0; k < R; ++k) {
                DDA ray = it;
                dda_set_t<kDdaSigma64>(ray, rn_add(g.stl_y, rn_mul((double)k, dt)));
                rays.push_back(axis_ray(ray));
            }
            continue;
        }
        if (!(u >= 6.103515625e-05)) return RG_OK;    // 2^-14
        View v = {};
        double rk, ri, r0;
        if (it.fast_is_i) {
            rk = dt / (c * dx);
            ri = -dy * s / (c * dx);
            r0 = ((g.stl_y - g.itl_y * s) / c - g.itl_x) / dx;
            v.flags = kLinesAreRows;
        } else {
            rk = dt / (s * dy);
            ri = -dx * c / (s * dy);
            r0 = ((g.stl_y - g.itl_x * c) / s - g.itl_y) / dy;
        }
        const double h = 0.5 * fabs(ri), a = std::max(1.0, 1.0 / fabs(ri));
        const double kl = -ri / rk, ks = 1.0 / rk, k0 = -r0 / rk;   // along lines, samples
        const double krow = it.fast_is_i ? kl : ks, kcol = it.fast_is_i ? ks : kl;
        r0 += 0.5 - h;
        const int nl = it.fast_is_i ? L : C;
        const double lim = 4194304.0;                 // 2^22
        if (!(fabs(r0) + (R - 1) * fabs(rk) + (nl - 1) * fabs(ri) < lim) ||
            !to_q40(rk, v.rk) || !to_q40(ri, v.ri) || !to_q40(r0, v.r0))
            return RG_OK;
        if (fabs(k0) + (L - 1) * fabs(krow) + (C - 1) * fabs(kcol) < lim &&
            to_q40(krow, v.krow) && to_q40(kcol, v.kcol) && to_q40(k0, v.k0)) {
            hmax = std::max(hmax, (0.5 + h) / fabs(rk));
            for (int t = 0; t < 2; ++t)
                wr[t] = std::max(wr[t], (t ? 63.0 : 31.0) * fabs(krow) + 31.0 * fabs(kcol));
        } else {
            hmax = 1e9;
        }
        v.delta = (float)it.sigma_tilde;
        v.delta_lo = (float)(it.sigma_tilde - (double)v.delta);
        v.P = (float)(a * fabs(rk));
        // where the trapezoid is at half its height, rays from its centre (Q2.30)
        if (fabs(rk) > 0.2) v.b0 = llrint(0.5 / fabs(rk) * 1073741824.0);
        v.wa = (float)a;
        v.brow = lost_ray(it, g, dt);
        q.lost = q.lost || v.brow >= 0;
        v.view = j;
        hv.push_back(v);
    }
    SSPlan &p = q.p;
    p.dda = true;
    p.nl[0] = p.ne[1] = L;
    p.nl[1] = p.ne[0] = C;
    p.nv = (int)hv.size();
    p.g.R = R;
    p.g.A = g.A;
    p.dense = fabs(dx) > 1.02 * fabs(dt);
    int rc;
    if ((rc = ensure_device_error_word())) return rc;
    q.d_cs = d_cs;
    if (p.nv > 0) {
        RG_CK(cudaMalloc(&p.d_views, sizeof(View) * hv.size()));
        RG_CK(cudaMemcpy(p.d_views, hv.data(), sizeof(View) * hv.size(), cudaMemcpyHostToDevice));
        if ((rc = st_blocks_build(p, hv.data()))) return rc;
    }
    q.nax = (int)ax.size();
    if (q.nax > 0) {
        // the rays of each (axis view, pixel of a line): a range of k, which
        // is monotone in the pixel
        const int ne = std::max(L, C);
        q.ax_ne = ne;
        std::vector<int2> range((size_t)q.nax * ne, make_int2(INT_MAX, 0));
        for (int v = 0; v < q.nax; ++v) {
            const int n = ax[v].fast_i ? C : L;
            for (int k = 0; k < R; ++k) {
                const DLRay &r = rays[(size_t)v * R + k];
                if (r.lo > r.hi) continue;
                for (int m : {r.ja, r.nc == INT_MAX ? -1 : r.jb})
                    if (m >= 0 && m < n) {
                        int2 &e = range[(size_t)v * ne + m];
                        e.x = std::min(e.x, k);
                        e.y = std::max(e.y, k + 1);
                    }
            }
        }
        const size_t b0 = sizeof(DLRay) * rays.size(), b1 = sizeof(DLAxis) * ax.size(),
                     b2 = sizeof(int2) * range.size();
        RG_CK(cudaMalloc(&q.d_axis, b0 + b1 + b2));
        char *b = (char *)q.d_axis;
        RG_CK(cudaMemcpy(b, rays.data(), b0, cudaMemcpyHostToDevice));
        RG_CK(cudaMemcpy(b + b0, ax.data(), b1, cudaMemcpyHostToDevice));
        RG_CK(cudaMemcpy(b + b0 + b1, range.data(), b2, cudaMemcpyHostToDevice));
        q.rays = (const DLRay *)b;
        q.axis = (const DLAxis *)(b + b0);
        q.range = (const int2 *)(b + b0 + b1);
    }
    for (int t = 0; t < 2; ++t)
        q.wg[t] = wr[t] < 4096.0 ? ((int)ceil(wr[t] + 1e-6) + 4 + 7) & ~7 : 1 << 20;
    // Two taps (and the half-turn pairs) where a pixel is met by at most two
    // rays of a view, on an image and a detector centred on 0; four taps
    // while it is met by at most four.  1e-6: the trapezoid's ends.
    const bool centred = g.itl_x == -g.ibr_x && g.itl_y == -g.ibr_y && g.stl_y == -g.sbr_y;
    // Reflected views: view nv - 1 - e at column C - 1 - c where view e is at c
    // (to 2^-25 rays).
    bool refl = p.nv > 0 && p.nv % 2 == 0;
    auto near = [](long long a, long long b) { return llabs(a - b) < (1LL << 15); };
    for (int e = 0; e < p.nv / 2 && refl; ++e) {
        const View &v = hv[e], &w = hv[p.nv - 1 - e];
        refl = near(w.krow * (L - 1), v.krow * (L - 1)) &&
               near(w.kcol * (C - 1), -v.kcol * (C - 1)) && near(w.k0 + w.kcol * (C - 1), v.k0) &&
               fabsf(w.P - v.P) <= 1e-6f * v.P && fabsf(w.wa - v.wa) <= 1e-6f * v.wa;
    }
    const int form = centred && hmax <= 1.0 - 1e-6 ? (refl ? kDlQuarter : kDlHalf)
                     : hmax <= 2.0 - 1e-6          ? kDlTaps
                                                   : 0;
    if (form && p.nv <= 65535 && q.wg[0] <= kDlBox) q.gather = form;
    q.ok = true;
    return RG_OK;
}

namespace {

// ----------------------------------------------------------------------------
// Radon

// One CTA packs the 32 x 32 image tile (blockIdx.x, .y) into both arrays of
// line pairs: entry 1 + n of a line holds (p[n], p[n+1] - p[n]), n = -1 ..
// ne - 1, pixels outside the line zero; the entries above are zero.
__global__ __launch_bounds__(256) void k_dl_pairs(const float *__restrict__ img, long long cs,
                                                  long long ls, int L, int C,
                                                  float2 *__restrict__ prow,
                                                  float2 *__restrict__ pcol)
{
    pdl_gate();
    __shared__ float t[33][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    const size_t pr = pairs_pitch(C), pc = pairs_pitch(L);
    for (int e = threadIdx.x; e < 33 * 33; e += 256) {
        const int y = e / 33, x = e - 33 * y, r = r0 + y, c = c0 + x;
        t[y][x] = (r < L && c < C) ? img[(long long)r * cs + (long long)c * ls] : 0.f;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c = c0 + lane, r = r0 + lane;
    if (c < C)
        for (int y = w; y < 32 && r0 + y < L; y += 8) {
            float2 *line = prow + (size_t)(r0 + y) * pr;
            line[1 + c] = make_float2(t[y][lane], t[y][lane + 1] - t[y][lane]);
            if (c == 0) line[0] = make_float2(0.f, t[y][0]);
            if (c == C - 1)
                for (int e = C + 1; e < (int)pr; ++e) line[e] = make_float2(0.f, 0.f);
        }
    if (r < L)
        for (int x = w; x < 32 && c0 + x < C; x += 8) {
            float2 *line = pcol + (size_t)(c0 + x) * pc;
            line[1 + r] = make_float2(t[lane][x], t[lane + 1][x] - t[lane][x]);
            if (r == 0) line[0] = make_float2(0.f, t[0][x]);
            if (r == L - 1)
                for (int e = L + 1; e < (int)pc; ++e) line[e] = make_float2(0.f, 0.f);
        }
}

// Direct form, for plans whose views do not come in runs (interleaved
// subsets) or are few: a warp is 32 rays of a view, lines from L1/L2; split
// > 1: a cluster of CTAs along x shares the lines, summed in rank order.
// (12 CTAs per SM, as without the walk's registers.)
template <int EPI>
__global__ __launch_bounds__(128, 12) void k_dl_radon(const float2 *__restrict__ prow,
                                                  const float2 *__restrict__ pcol, int L, int C,
                                                  const View *__restrict__ views, int nv, int R,
                                                  float *__restrict__ out, long long ovs,
                                                  long long ors, const float *__restrict__ y_am,
                                                  int split, const __grid_constant__ DLArgs dl)
{
    pdl_gate();
    __shared__ float red[2][128];
    const int rank = blockIdx.x % split;
    const int k = (int)(blockIdx.x / split) * 32 + (threadIdx.x & 31);
    const int e = blockIdx.y * 4 + (threadIdx.x >> 5);
    const bool active = e < nv && k < R;
    const View v = views[active ? e : 0];
    const bool rows = (v.flags & kLinesAreRows) != 0;
    const int nl = rows ? L : C, ne = rows ? C : L;
    const size_t pitch = pairs_pitch(ne);
    const long long u0 = v.r0 + (long long)k * v.rk;
    int lo, hi;
    radon_line_range<true>(u0, v.ri, nl, ne, lo, hi);
    lo = max(lo, (int)((long long)nl * rank / split));
    hi = min(hi, (int)((long long)nl * (rank + 1) / split) - 1);
    if (!active) { lo = 1; hi = 0; }
    const float wa = v.wa, wc = fmaf(-2.f, wa, 1.f);
    float acc = 0.f, comp = 0.f;
    long long u = u0 + (long long)lo * v.ri;
    const float2 *__restrict__ line = (rows ? prow : pcol) + (long long)lo * (long long)pitch + 1;
    for (int i = lo; i <= hi;) {
        // sums of at most four lines between compensations, as precise as the
        // staged kernel's
        const int iend = min(hi, i + 7);
        float part = 0.f, odd = 0.f;
#pragma unroll 8
        for (; i <= iend; ++i) {
            const float2 pr = __ldg(line + (int)(u >> kDlQ));
            odd += fmaf(fma_sat(wa, frac_plus_one((unsigned)(u >> (kDlQ - 23))), wc), pr.y, pr.x);
            const float other = part;
            part = odd;
            odd = other;
            u += v.ri;
            line += pitch;
        }
        kahan_add(acc, comp, part);
        kahan_add(acc, comp, odd);
    }
    if (split > 1) {
        namespace cg = cooperative_groups;
        cg::cluster_group cl = cg::this_cluster();
        red[0][threadIdx.x] = acc;
        red[1][threadIdx.x] = comp;
        cl.sync();
        if (rank == 0)
            for (int src = 1; src < split; ++src) {
                const float *peer = cl.map_shared_rank(&red[0][0], src);
                two_sum_add(acc, comp, peer[threadIdx.x], peer[128 + threadIdx.x]);
            }
        cl.sync();    // no CTA leaves while rank 0 still reads its partials
        if (rank != 0) return;
    }
    if (!active) return;
    const float val = fmaf(acc, v.delta, fmaf(acc, v.delta_lo, -comp * v.delta));
    out[v.view * ovs + k * ors] = radon_epilogue(EPI, val, y_am, (size_t)v.view * R + k);
    if (!isfinite(val) || k == v.brow)
        dl_walk_rays<EPI>(dl, 1u, k, v.view, out, ovs, ors, y_am, R);
}

// The axis-aligned views alone, beside the direct form.
template <int EPI>
__global__ __launch_bounds__(256) void k_dl_axis(const __grid_constant__ DLArgs dl,
                                                 float *__restrict__ out, long long ovs,
                                                 long long ors, const float *__restrict__ y_am)
{
    pdl_gate();
    dl_axis_cta<EPI>(dl, blockIdx.x, out, ovs, ors, y_am, dl.g.R);
}

template <int EPI>
int radon_epi(const DLPlan &q, const DLArgs &dl, const float *img, long long ics, long long ils,
              float2 *prow, float2 *pcol, float *out, long long ovs, long long ors,
              const float *y_am, cudaStream_t st)
{
    const SSPlan &p = q.p;
    const int L = q.g.lines, C = q.g.columns, R = q.g.R;
    RG_CK(launch_pdl(k_dl_pairs, dim3((C + 31) / 32, (L + 31) / 32), 256, 0, st, 1, img, ics, ils, L,
                     C, prow, pcol));
    RG_CK_LAUNCH("k_dl_pairs");
    if (p.nv > 0 && radon_tma_usable(p))
        return launch_radon_tma(p, prow, pcol, out, ovs, ors, y_am, R, st, 1, 0, 0, EPI, &dl);
    if (p.nv > 0) {
        const dim3 grid((R + 31) / 32, (p.nv + 3) / 4);
        int split = 1;                      // up to two waves of 16 CTAs per SM
        while (split < 4 && (long long)grid.x * grid.y * split * 2 <= 2LL * 16 * 152) split *= 2;
        RG_CK(launch_pdl(k_dl_radon<EPI>, dim3(grid.x * split, grid.y), 128, 0, st, split, prow,
                         pcol, L, C, p.d_views, p.nv, R, out, ovs, ors, y_am, split, dl));
        RG_CK_LAUNCH("k_dl_radon");
    }
    if (q.nax > 0) {
        const unsigned ctas = (unsigned)(((long long)q.nax * R + 7) / 8);
        RG_CK(launch_pdl(k_dl_axis<EPI>, dim3(ctas), 256, 0, st, 1, dl, out, ovs, ors, y_am));
        RG_CK_LAUNCH("k_dl_axis");
    }
    return RG_OK;
}

}  // namespace

// (65535 rows of CTAs take 32 lines each)
bool dl_sizes_ok(int L, int C, int R)
{
    return L >= 2 && L <= 65535 * 32 && C >= 2 && C <= 65535 * 32 && R >= 2 && R <= (1 << 20) &&
           (long long)L * C <= (1LL << 28);
}

size_t dl_radon_bytes(int L, int C)
{
    return ws_sum({(size_t)L * pairs_pitch(C) * sizeof(float2),
                   (size_t)C * pairs_pitch(L) * sizeof(float2)});
}

int launch_dl_radon(const DLPlan &q, const float *img, long long ics, long long ils, void *scratch,
                    float *out, long long ovs, long long ors, const float *y_am, cudaStream_t st)
{
    const int L = q.g.lines, C = q.g.columns;
    Scratch s;
    s.base = (char *)scratch;
    float2 *prow = (float2 *)s.take((size_t)L * pairs_pitch(C) * sizeof(float2));
    float2 *pcol = (float2 *)s.take((size_t)C * pairs_pitch(L) * sizeof(float2));
    const DLArgs dl = {q.g, q.d_cs, prow, pcol, q.nax, q.axis, q.rays};
    return y_am ? radon_epi<kEpiRatio>(q, dl, img, ics, ils, prow, pcol, out, ovs, ors, y_am, st)
                : radon_epi<kEpiSum>(q, dl, img, ics, ils, prow, pcol, out, ovs, ors, nullptr, st);
}

namespace {

// ----------------------------------------------------------------------------
// Transpose

// Entries per view of the quad array.  Half-turn form (M): entry 1 + k holds
// samples k, k + 1 and R - 2 - k, R - 1 - k, k = -1 .. R - 1; four-tap form:
// entry 2 + k holds samples k - 1 .. k + 2, k = -2 .. R; samples outside the
// row are zero.  All times sigma.
template <bool M> __host__ __device__ constexpr int dl_entries(int R) { return M ? R + 1 : R + 3; }

// s (d + dl), dl the step's part below FP32 (of either sign, or zero: an infinite
// sample takes d alone, which keeps its sign).
__device__ __forceinline__ float scaled(float s, float d, float dl)
{
    return isfinite(s) ? fmaf(s, d, s * dl) : s * d;
}

// One CTA writes the quads of one view.  bad[view]: it holds a non-finite
// sample.
template <bool M, bool RAW>
__global__ __launch_bounds__(256) void k_dl_quads(const float *__restrict__ s_am, int R,
                                                  const View *__restrict__ views,
                                                  float4 *__restrict__ quads,
                                                  unsigned char *__restrict__ bad)
{
    pdl_gate();
    const View &v = views[blockIdx.x];
    const float *__restrict__ row = s_am + (size_t)v.view * R;
    const float d = v.delta, dl = v.delta_lo;
    const int lost = (int)v.brow;
    float4 *__restrict__ out = quads + (size_t)blockIdx.x * dl_entries<M>(R);
    int nonfinite = 0;
    auto at = [&](int n) {
        const float s = (n >= 0 && n < R && n != lost) ? __ldg(row + n) : 0.f;
        nonfinite |= (__float_as_uint(s) & 0x7F800000u) == 0x7F800000u;
        return RAW ? s : scaled(s, d, dl);
    };
    for (int e = threadIdx.x; e < dl_entries<M>(R); e += 256)
        out[e] = M ? make_float4(at(e - 1), at(e), at(R - 1 - e), at(R - e))
                   : make_float4(at(e - 3), at(e - 2), at(e - 1), at(e));
    nonfinite = __syncthreads_or(nonfinite);
    if (threadIdx.x == 0) bad[blockIdx.x] = nonfinite ? 1 : 0;
}

// A staged view: position of the tile's first pixel (Q24.40, from the
// window's first entry), its steps, the Q9.23 step of four rows, and the
// weights' constants.
struct __align__(16) DLSlot {
    long long base, row, col;
    unsigned step;
    float P, c0;
    int state;          // -1: skip, 0, else CAREFUL (non-finite samples, detector's end)
    float sigma, sigma_lo;   // NORM: (base is not rounded, P is times 2^-30)
    int nlo;            // NORM: first entry's ray
    int half;           // NORM: where the trapezoid is at half its height (Q2.30)
};

template <int OFF>
__device__ __forceinline__ float4 lds_quad(unsigned addr)
{
    float4 q;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4+%5];"
                 : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w) : "r"(addr), "n"(OFF));
    return q;
}

// sum - c += a (w + wl), the product and the sum with their rounding errors (of
// the first terms, larger than the sum, to within an ulp of theirs): two FP32
// numbers that do what the walks' FP64 sums do.
__device__ __forceinline__ void dot_add(float &sum, float &c, float a, float w, float wl)
{
    const float p = a * w, e = fmaf(a, wl, fmaf(a, w, -p)), t = sum + p;
    c -= (p - (t - sum)) + e;
    sum = t;
}

// Sums of a thread.  NORM (the normalised backprojection): every sum comes with
// its rounding errors, and den sums the weights.  The reflected view at the
// reflected pixel and the half-turn mirror have the pixel's weights, so one
// sum of weights serves them all.
template <int F, int ROWS, bool NORM>
struct DLSums {
    float s[dl_sums(F)][ROWS];
    float c[NORM ? dl_sums(F) : 1][NORM ? ROWS : 1];
    float den[NORM ? ROWS : 1], dc[NORM ? ROWS : 1];
};

// The ROWS positions of a thread for one staged view (and its reflection),
// from pos (Q24.40 from the window's first entry).  CAREFUL: samples of weight
// zero are left out (a non-finite one would spread to pixels beside its ray),
// and rays off the detector weigh nothing.
//
// The weights come from the Q9.23 position by one saturated FMA each.  NORM
// steps the Q24.40 position and takes them from its distance to the
// trapezoid's half height in Q2.30 (an integer subtraction and a conversion
// more each): its quotients are rounded once, and the position's rounding
// would show beside that (512^2 x 360: 2.6e-8 against 2.45e-8 for the rounding
// alone, 300^2 x 200 2.9e-8 against 2.5e-8).  So would one rounding of every
// product, of the samples times sigma or of sigma (2.518e-8 and 2.532e-8 against
// 2.501e-8 for the rounding alone, which the walk's FP64 sums reach): the
// samples stay as they are, sigma goes with the weights in two parts, and the
// products keep their rounding errors: 2.502e-8 and 2.503e-8, 512^2 x 360 100 ->
// 143 us (the walk 1115).
template <int F, int ROWS, bool CAREFUL, bool NORM>
__device__ __forceinline__ void dl_slot(long long pos, const DLSlot &si, unsigned pw,
                                        unsigned quad_bytes, int R, DLSums<F, ROWS, NORM> &t)
{
    // W at distances w1 - 1, 2 - w1 (rays k, k + 1) and w1, 3 - w1 (k - 1, k + 2)
    const float P = si.P, c0 = si.c0;
    const float ca = c0 + P, cb = fmaf(-2.f, P, c0), cd = fmaf(-3.f, P, c0);
    constexpr int kOne = 1 << 30;
    auto weight = [&](int d) { return fma_sat(-P, (float)d, 0.5f); };
    unsigned vpos = (unsigned)(pos >> (kDlQ - 23));
    auto term = [](float sum, float v, float w) {
        if (CAREFUL) return w > 0.f ? fmaf(v, w, sum) : sum;
        return fmaf(v, w, sum);
    };
    // sum i of row r: + a wa + b wb (NORM: wa, wb with their lower parts la, lb)
    auto add2 = [&](int i, int r, float a, float wa, float b, float wb, float la, float lb) {
        if constexpr (NORM) {
            float &s = t.s[i][r], &c = t.c[i][r];
            if (!CAREFUL || wa > 0.f) dot_add(s, c, a, wa, la);
            if (!CAREFUL || wb > 0.f) dot_add(s, c, b, wb, lb);
            if (CAREFUL && !isfinite(c)) c = 0.f;     // an infinite sum stays infinite
        } else {
            t.s[i][r] = term(term(t.s[i][r], a, wa), b, wb);
        }
    };
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const unsigned e = NORM ? (unsigned)(pos >> kDlQ) : vpos >> 23;
        const unsigned addr = e * quad_bytes + pw;
        const float4 q = lds_quad<0>(addr);
        float wa, wb, wz = 0.f, wd = 0.f;
        if constexpr (NORM) {
            const int f = (int)((unsigned)(pos >> (kDlQ - 30)) & (kOne - 1));
            wa = weight(f - si.half);
            wb = weight(kOne - si.half - f);
            if constexpr (F == kDlTaps) {
                wz = weight(f - si.half + kOne);          // may wrap only where both are 0
                wd = weight(kOne - si.half - f + kOne);
            }
        } else {
            const float w1 = frac_plus_one(vpos);
            wa = fma_sat(-P, w1, ca);
            wb = fma_sat(P, w1, cb);
            if constexpr (F == kDlTaps) {
                wz = fma_sat(-P, w1, c0);
                wd = fma_sat(P, w1, cd);
            }
        }
        if constexpr (CAREFUL && NORM) {
            const int k = si.nlo + (int)e;
            if ((unsigned)k >= (unsigned)R) wa = 0.f;
            if ((unsigned)(k + 1) >= (unsigned)R) wb = 0.f;
            if ((unsigned)(k - 1) >= (unsigned)R) wz = 0.f;
            if ((unsigned)(k + 2) >= (unsigned)R) wd = 0.f;
        }
        float la = 0.f, lb = 0.f, lz = 0.f, ld = 0.f;
        if constexpr (NORM) {                         // the step goes with the weights
            auto step = [&](float &w, float &l) {
                const float v = w * si.sigma;
                l = fmaf(w, si.sigma_lo, fmaf(w, si.sigma, -v));
                w = v;
                const float n = t.den[r] + v;
                t.dc[r] -= (v - (n - t.den[r])) + l;
                t.den[r] = n;
            };
            step(wa, la);
            step(wb, lb);
            if constexpr (F == kDlTaps) {
                step(wz, lz);
                step(wd, ld);
            }
        }
        if constexpr (F == kDlTaps) {
            if constexpr (NORM) {
                add2(0, r, q.x, wz, q.y, wa, lz, la);
                add2(0, r, q.z, wb, q.w, wd, lb, ld);
            } else {
                t.s[0][r] = term(term(term(term(t.s[0][r], q.x, wz), q.y, wa), q.z, wb), q.w, wd);
            }
        } else {
            add2(0, r, q.x, wa, q.y, wb, la, lb);
            add2(1, r, q.w, wa, q.z, wb, la, lb);
        }
        if constexpr (F == kDlQuarter) {
            const float4 p = lds_quad<kDlPartner>(addr);
            add2(2, r, p.x, wa, p.y, wb, la, lb);
            add2(3, r, p.w, wa, p.z, wb, la, lb);
        }
        if constexpr (NORM) pos += 4 * si.row;
        else vpos += si.step;
    }
}

// What the axis-aligned views' rays add to pixel (row, col), and their
// weights.
__device__ __noinline__ float2 dl_axis_sum(int row, int col, int nax, const DLAxis *axis,
                                           const DLRay *rays, const int2 *range, int ax_ne,
                                           const float *s_am, int R)
{
    float sum = 0.f, den = 0.f;
    for (int v = 0; v < nax; ++v) {
        const DLAxis ax = axis[v];
        const int line = ax.fast_i ? row : col, m = ax.fast_i ? col : row;
        const int2 ks = range[(size_t)v * ax_ne + m];
        for (int k = ks.x; k < ks.y; ++k) {
            const DLRay r = rays[(size_t)v * R + k];
            if (line < r.lo || line > r.hi) continue;
            const float w = line < r.nc ? (r.ja == m ? 1.f : 0.f)
                          : line > r.nc ? (r.jb == m ? 1.f : 0.f)
                                        : (r.ja == m ? r.wa : r.jb == m ? r.wb : 0.f);
            if (w != 0.f) {           // (the walk's entry pixels may split as 6 and -5)
                const float s = s_am[(size_t)ax.view * R + k];
                sum = fmaf(w, scaled(s, ax.sigma, ax.sigma_lo), sum);
                den = fmaf(w, ax.sigma, den);
            }
        }
    }
    return make_float2(sum, den);
}

struct DLOut {
    float *out;                // strides cs, ls (not kDlUpdate)
    long long cs, ls;
    float *x;                  // kDlUpdate: x <- x * sum * inv, contiguous
    const float *inv;
};
enum { kDlStore = 0, kDlUpdate = 1, kDlInvert = 2, kDlNorm = 3 };

// (n + nl) / (d + dl), rounded once (to within 2^-40); 0 where the divisor is.
__device__ __forceinline__ float quotient(float n, float nl, float d, float dl)
{
    if (d == 0.f && dl == 0.f) return 0.f;
    const float q = n / d;
    if (!isfinite(q)) return q;
    return q + (fmaf(-q, d, n) + fmaf(-q, dl, nl)) / d;
}

template <int EP>
__device__ __forceinline__ void dl_store(const DLOut &o, int row, int col, int C, float sum,
                                         float lo, float den, float den_lo)
{
    if (EP == kDlNorm) {
        o.out[(long long)row * o.cs + (long long)col * o.ls] = quotient(sum, lo, den, den_lo);
    } else if (EP == kDlUpdate) {
        const size_t e = (size_t)row * C + col;
        o.x[e] = o.x[e] * sum * o.inv[e];
    } else {
        o.out[(long long)row * o.cs + (long long)col * o.ls] =
            EP == kDlStore ? sum : (sum > 0.f ? 1.f / sum : 0.f);
    }
}

// The transpose over a tile of 32 columns x 8 ROWS rows per CTA.
//
// kDlHalf: also the tile's mirror under a half turn -- on a centred geometry
// pixel (L - 1 - r, C - 1 - c) meets a view at ray position R - 1 - kappa, so
// its two weights are the pixel's, swapped, on the samples R - 2 - k and R - 1
// - k: one position, one pair of weights and one 128-bit load serve two
// updates.  The tiles then cover the upper half of the rows only (on an odd
// count the middle row is its own mirror, and only its primaries are stored).
//
// kDlQuarter: also the view's reflection pi - theta, which pixel (r, C - 1 -
// c) meets where pixel (r, c) meets theta: a position serves four updates.
// CTAs come in pairs (side 0, 1 of a cluster): side 0 walks columns col0 + c
// of the left half, side 1 the columns C - 1 - col0 - c, each summing the
// view at its own pixels and the reflection at the other side's, which they
// exchange in distributed shared memory.
//
// As in k_gather_rot_tma each view's window of quads is one TMA box, double
// buffered; warp 0 loads chunk c + 1 while all warps sum chunk c.  split > 1:
// `split` CTAs of a cluster along x share the views; the partials meet in
// distributed shared memory, each rank finishing its share of the rows, ranks
// added in order.
template <int F, int ROWS, int EP, bool DENSE>
__global__ __launch_bounds__(256) void k_dl_gather(
    const __grid_constant__ CUtensorMap tm, const View *__restrict__ views, int nv, int L, int C,
    DLOut o, int wb, int nslots, unsigned quad_bytes, int split,
    const unsigned char *__restrict__ bad, int nax, const DLAxis *__restrict__ axis,
    const DLRay *__restrict__ rays, const int2 *__restrict__ range, int ax_ne,
    const float *__restrict__ s_am, int R, int *__restrict__ err, int expire_first)
{
    pdl_gate();
    extern __shared__ __align__(128) float4 qbuf[];   // [2][nslots][wb]
    __shared__ __align__(8) unsigned long long full[2];
    __shared__ DLSlot slot[2][kDlSlots];
    constexpr bool kRefl = F == kDlQuarter;
    constexpr int TH = kWarps * ROWS, NS = dl_sums(F);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cl_rank = blockIdx.x % (kRefl ? 2 * split : split);
    const int side = kRefl ? cl_rank & 1 : 0, rank = kRefl ? cl_rank >> 1 : cl_rank;
    const int row0 = blockIdx.y * TH;
    const int col0 = (int)(blockIdx.x / (kRefl ? 2 * split : split)) * kTile;
    // warp w covers 8 columns x rows 4 ROWS (w >> 2) + 4 r .. + 4
    const int cofs = 8 * (warp & 3) + (gather_lane(lane, DENSE) & 7);
    const int rofs = 4 * ROWS * (warp >> 2) + (gather_lane(lane, DENSE) >> 3);

    constexpr bool kNorm = EP == kDlNorm;
    DLSums<F, ROWS, kNorm> t;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            t.s[i][r] = 0.f;
            if constexpr (kNorm) t.c[i][r] = 0.f;
        }
        if constexpr (kNorm) t.den[r] = t.dc[r] = 0.f;
    }

    const int nu = kRefl ? nv / 2 : nv;               // views, or pairs of them
    const int vbeg = (int)((long long)nu * rank / split);
    const int vend = (int)((long long)nu * (rank + 1) / split);
    const int nchunks = (vend - vbeg + nslots - 1) / nslots;
    const unsigned qbase = smem_addr(qbuf);
    const unsigned slot_bytes = (unsigned)wb * 16u;
    if (threadIdx.x == 0) {
        mbar_init(smem_addr(&full[0]), 1);
        mbar_init(smem_addr(&full[1]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // a compensated sum that turns infinite needs CAREFUL from there on
    int any_bad = 0;
    if constexpr (kNorm)
        for (int e = threadIdx.x; e < nv; e += 256) any_bad |= bad[e];
    any_bad = __syncthreads_or(any_bad);

    auto issue = [&](int c) {
        const int chunk = vbeg + c * nslots;
        const int n = min(nslots, vend - chunk), b = c & 1;
        DLSlot si = {0, 0, 0, 0u, 0.f, 0.f, -1, 0.f, 0.f, 0, 0};
        int nlo = 0;
        if (lane < n) {
            const View &v = views[chunk + lane];
            const long long kr = v.krow, kc = side ? -v.kcol : v.kcol;
            const long long origin = v.k0 + (long long)row0 * kr +
                                     (long long)(side ? C - 1 - col0 : col0) * v.kcol;
            const long long dr = (long long)(TH - 1) * kr, dc = (long long)(kTile - 1) * kc;
            const long long mn = origin + min(0LL, dr) + min(0LL, dc);
            const long long mx = origin + max(0LL, dr) + max(0LL, dc);
            nlo = (int)(mn >> kDlQ) - 1;
            if ((int)(mx >> kDlQ) + 1 - nlo + 1 <= wb) {
                // the rounding of the four-row step spread about the middle row
                const long long st = (4 * kr + (1LL << (kDlQ - 24))) >> (kDlQ - 23);
                si.base = origin - ((long long)nlo << kDlQ) + (1LL << (kDlQ - 24)) +
                          ((4 * kr - (st << (kDlQ - 23))) * (ROWS - 1) >> 1);
                si.row = kr;
                si.col = kc;
                si.step = (unsigned)st;
                si.P = v.P;
                si.c0 = 0.5f * (v.wa + 1.f);
                si.state = bad[chunk + lane];
                if (kRefl) si.state |= bad[nv - 1 - (chunk + lane)];
                if constexpr (kNorm) {
                    si.base = origin - ((long long)nlo << kDlQ);
                    si.P = v.P * 9.31322574615478515625e-10f;
                    si.sigma = v.delta;
                    si.sigma_lo = v.delta_lo;
                    si.nlo = nlo;
                    si.half = (int)v.b0;
                    if (any_bad || nlo < 1 || (int)(mx >> kDlQ) + 3 >= R) si.state |= 2;
                }
            } else if (err) {
                atomicOr(err, 1);
            }
        }
        if (lane < nslots) slot[b][lane] = si;
        const bool ok = si.state >= 0;
        const unsigned valid = __ballot_sync(0xffffffffu, ok);
        const unsigned bar = smem_addr(&full[b]);
        if (lane == 0) {
            fence_proxy_async_smem();
            mbar_expect_tx(bar, (unsigned)__popc(valid) * slot_bytes * (kRefl ? 2u : 1u));
        }
        __syncwarp();
        if (ok) {
            const unsigned dst = qbase + (unsigned)(b * nslots + lane) * slot_bytes;
            const int y = nlo + (F == kDlTaps ? 2 : 1);
            tma_load_3d(dst, &tm, 0, y, chunk + lane, bar);
            if (kRefl) tma_load_3d(dst + kDlPartner, &tm, 0, y, nv - 1 - (chunk + lane), bar);
        }
    };

    if (warp == 0 && nchunks > 0) issue(0);
    __syncthreads();
    int c = 0;
    bool failed = false;
    for (; c < nchunks; ++c) {
        const int b = c & 1;
        // buffer b ^ 1 was last read in chunk c - 1, which every thread
        // finished before the barrier that closed it
        if (warp == 0 && c + 1 < nchunks) issue(c + 1);
        const bool ok = (expire_first && c == 0) ? false
                                                 : mbar_wait(smem_addr(&full[b]), (c >> 1) & 1);
        const int n = min(nslots, vend - (vbeg + c * nslots));
        for (int s = 0; s < n; ++s) {
            const DLSlot si = slot[b][s];
            if (si.state < 0) continue;
            const unsigned pw = qbase + (unsigned)(b * nslots + s) * slot_bytes;
            const long long pos = si.base + cofs * si.col + rofs * si.row;
            if (si.state == 0)
                dl_slot<F, ROWS, false, kNorm>(pos, si, pw, quad_bytes, R, t);
            else
                dl_slot<F, ROWS, true, kNorm>(pos, si, pw, quad_bytes, R, t);
        }
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
    }
    if (failed) {
        if (threadIdx.x == 0) {
            if (err) atomicOr(err, 2);
            // copies still in flight: chunk c and, if issued, chunk c + 1
            for (int w = c; w < min(c + 2, nchunks); ++w)
                mbar_wait(smem_addr(&full[w & 1]), (w >> 1) & 1);
        }
        __syncthreads();
    }

    // Pixel of row r of the tile (or its mirror) gets sum + lo (over den +
    // den_lo).
    auto finish = [&](int r, bool mirror, float sum, float lo, float den, float den_lo) {
        int row = row0 + rofs + 4 * r, col = col0 + cofs;
        if (row >= (F == kDlTaps ? L : (L + 1) / 2) || col >= (kRefl ? (C + 1) / 2 : C)) return;
        if (kRefl && side) {
            if (col == C - 1 - col) return;           // the middle column is side 0's
            col = C - 1 - col;
        }
        if (mirror) {
            if (row == L - 1 - row) return;           // the middle row: primaries
            row = L - 1 - row;
            col = C - 1 - col;
        }
        if (nax > 0) {
            const float2 a = dl_axis_sum(row, col, nax, axis, rays, range, ax_ne, s_am, R);
            if constexpr (kNorm) {                    // kept apart from the rounded sums
                float c = -lo, dc = -den_lo;
                two_sum_add(sum, c, a.x, 0.f);
                two_sum_add(den, dc, a.y, 0.f);
                if (!isfinite(c)) c = 0.f;
                lo = -c;
                den_lo = -dc;
            } else {
                sum += a.x;
            }
        }
        dl_store<EP>(o, row, col, C, sum, lo, den, den_lo);
    };
    if (kRefl || split > 1) {
        namespace cg = cooperative_groups;
        cg::cluster_group cl = cg::this_cluster();
        // [NS][ROWS][256], NORM: then den, and all of it again for the
        // compensations
        constexpr int kDen = NS * ROWS * 256, kComp = kDen + ROWS * 256;
        float *red = reinterpret_cast<float *>(qbuf);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
#pragma unroll
            for (int i = 0; i < NS; ++i) {
                red[(i * ROWS + r) * 256 + threadIdx.x] = t.s[i][r];
                if constexpr (kNorm) red[kComp + (i * ROWS + r) * 256 + threadIdx.x] = t.c[i][r];
            }
            if constexpr (kNorm) {
                red[kDen + r * 256 + threadIdx.x] = t.den[r];
                red[kComp + kDen + r * 256 + threadIdx.x] = t.dc[r];
            }
        }
        cl.sync();
        const int per = (F == kDlTaps ? 1 : 2) * ROWS / split;
        for (int u = rank * per; u < (rank + 1) * per; ++u) {
            const int r = u < ROWS ? u : u - ROWS;
            float sum = 0.f, c = 0.f, den = 0.f, dc = 0.f;
            auto gather = [&](int src, int e, float &sv, float &cv) {
                const float *peer = cl.map_shared_rank(red, src) + threadIdx.x;
                if constexpr (kNorm) {
                    two_sum_add(sv, cv, peer[e], peer[kComp + e]);
                    if (!isfinite(cv)) cv = 0.f;
                } else {
                    sv += peer[e];
                }
            };
            for (int src = 0; src < split; ++src) {
                if (kRefl) {
                    gather(2 * src + side, u * 256, sum, c);
                    gather(2 * src + 1 - side, (2 * ROWS + u) * 256, sum, c);
                    if (kNorm) {
                        gather(2 * src + side, kDen + r * 256, den, dc);
                        gather(2 * src + 1 - side, kDen + r * 256, den, dc);
                    }
                } else {
                    gather(src, u * 256, sum, c);
                    if (kNorm) gather(src, kDen + r * 256, den, dc);
                }
            }
            finish(r, u >= ROWS, sum, -c, den, -dc);
        }
        cl.sync();    // no CTA leaves while a peer still reads its partials
        return;
    }
    if constexpr (!kRefl) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const int i = kNorm ? r : 0;
            finish(r, false, t.s[0][r], -t.c[0][i], t.den[i], -t.dc[i]);
            if (F == kDlHalf)
                finish(r, true, t.s[NS - 1][r], -t.c[kNorm ? NS - 1 : 0][i], t.den[i], -t.dc[i]);
        }
    }
}

template <int F, int ROWS, int EP>
int gather_rows(const DLPlan &q, const float *s_am, const DLOut &o, float4 *quads,
                unsigned char *bad, int split, cudaStream_t st)
{
    constexpr bool kRefl = F == kDlQuarter, kMirror = F != kDlTaps;
    const SSPlan &p = q.p;
    const int L = q.g.lines, C = q.g.columns, R = q.g.R;
    const int wb = q.wg[ROWS == 8 ? 1 : 0];
    // as many views per chunk (16 at most) as two buffers of them leave room
    // for four CTAs per SM
    const int ns = std::min(kDlSlots, (kRefl ? kDlPartner : 48 * 1024) / (2 * wb * 16));
    const size_t smem = std::max(kRefl ? (size_t)2 * kDlPartner : (size_t)2 * ns * wb * 16,
                                 (EP == kDlNorm ? 2 * (dl_sums(F) + 1) : dl_sums(F)) *
                                     (size_t)ROWS * 256 * sizeof(float));
    CUtensorMap tm = {};
    if (p.nv > 0) {
        EncodeTiledFn fn = tensor_map_encoder();
        if (!fn) return set_error(RG_ECUDA, "cuTensorMapEncodeTiled is not available");
        const cuuint64_t Rq = (cuuint64_t)dl_entries<kMirror>(R);
        cuuint64_t dims[3] = {4, Rq, (cuuint64_t)p.nv};
        cuuint64_t strides[2] = {16, Rq * 16};
        cuuint32_t box[3] = {4, (cuuint32_t)wb, 1};
        cuuint32_t estr[3] = {1, 1, 1};
        CUresult r = fn(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)quads, dims, strides, box,
                        estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            return set_error(RG_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
        RG_CK(launch_pdl(k_dl_quads<kMirror, EP == kDlNorm>, dim3(p.nv), 256, 0, st, 1, s_am, R, p.d_views, quads,
                         bad));
        RG_CK_LAUNCH("k_dl_quads");
    }
    auto k = p.dense ? k_dl_gather<F, ROWS, EP, true> : k_dl_gather<F, ROWS, EP, false>;
    RG_CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int rows = kMirror ? (L + 1) / 2 : L, cols = kRefl ? (C + 1) / 2 : C;
    const int cluster = kRefl ? 2 * split : split;
    const dim3 grid(((cols + kTile - 1) / kTile) * cluster,
                    (rows + kWarps * ROWS - 1) / (kWarps * ROWS));
    const int expire = test_switch("RG_TEST_EXPIRE_WAIT") ? 1 : 0;
    RG_CK(launch_pdl(k, grid, 256, smem, st, cluster, tm, p.d_views, p.nv, L, C, o, wb, ns,
                     (unsigned)sizeof(float4), split, bad, q.nax, q.axis, q.rays, q.range, q.ax_ne,
                     s_am, R, device_error_word(), expire));
    RG_CK_LAUNCH("k_dl_gather");
    return RG_OK;
}

// Launch shape: rows per thread and view split (CTAs per cluster and side).
// Tiles of 32 rows (4 per thread) keep the registers of four sums per row at
// 64, four CTAs per SM; a split of 4 pays while the unsplit grid is under two
// waves (of 4 CTAs x 152 SMs), with 16 views left per CTA.  Measured (us,
// view-major sinogram, rows,split): kDlQuarter 2048^2 x 1800 4,1 2048 / 4,4
// 2091 / 8,2 2064 / 8,4 2140; 1024^2 x 720 256 / 252 / 342 / 276; 999^2 x 901
// 322 / 306 / 428 / 341; 512^2 x 360 92 / 46 / 92 / 54.  kDlHalf 1024^2 x 720
// 4,4 288 / 8,4 281, 2048^2 x 1800 4,2 2499 / 8,2 2172: 8 rows from one wave.
// kDlTaps 1024^2 x (1484, 720) 4,1 673 / 4,2 661 / 8,2 602 / 8,4 740, 256^2 x
// (367, 180) 4,4 32 / 8,4 47: 8 rows and a split of 2 from one wave.
template <int F, int EP>
int gather_shape(const DLPlan &q, const float *s_am, const DLOut &o, float4 *quads,
                 unsigned char *bad, cudaStream_t st)
{
    constexpr bool kRefl = F == kDlQuarter, kMirror = F != kDlTaps;
    const int rows = kMirror ? (q.g.lines + 1) / 2 : q.g.lines;
    const int cols = kRefl ? (q.g.columns + 1) / 2 : q.g.columns;
    const int nu = kRefl ? q.p.nv / 2 : q.p.nv;
    const long long ctas4 = (long long)((cols + kTile - 1) / kTile) * (kRefl ? 2 : 1) *
                            ((rows + kWarps * 4 - 1) / (kWarps * 4));
    const long long wave = 152 * 4;
    // (the compensated sums of the normalised form leave no room for 8 rows)
    const bool tall = !kRefl && EP != kDlNorm && ctas4 >= wave && q.wg[1] <= kDlBox;
    int split = ctas4 / (tall ? 2 : 1) < 2 * wave ? 4 : 1;
    if (F == kDlTaps && tall) split = std::min(split, 2);
    while (split > 1 && nu < 16 * split) split /= 2;
    if constexpr (!kRefl && EP != kDlNorm)
        if (tall) return gather_rows<F, 8, EP>(q, s_am, o, quads, bad, split, st);
    return gather_rows<F, 4, EP>(q, s_am, o, quads, bad, split, st);
}

template <int EP>
int gather_form(const DLPlan &q, const float *s_am, const DLOut &o, void *scratch, cudaStream_t st)
{
    unsigned char *bad = (unsigned char *)scratch;
    float4 *quads = (float4 *)((char *)scratch + Scratch::align((size_t)std::max(q.p.nv, 1)));
    if (q.gather == kDlQuarter) return gather_shape<kDlQuarter, EP>(q, s_am, o, quads, bad, st);
    if (q.gather == kDlHalf) return gather_shape<kDlHalf, EP>(q, s_am, o, quads, bad, st);
    return gather_shape<kDlTaps, EP>(q, s_am, o, quads, bad, st);
}

}  // namespace

size_t dl_gather_bytes(int R, int nv)
{
    return ws_sum({(size_t)nv, (size_t)nv * dl_entries<false>(R) * sizeof(float4)});
}

int launch_dl_gather(const DLPlan &q, const float *s_am, float *out, long long cs, long long ls,
                     void *scratch, cudaStream_t st, bool invert)
{
    DLOut o = {out, cs, ls, nullptr, nullptr};
    return invert ? gather_form<kDlInvert>(q, s_am, o, scratch, st)
                  : gather_form<kDlStore>(q, s_am, o, scratch, st);
}

int launch_dl_normalised(const DLPlan &q, const float *s_am, float *out, long long cs, long long ls,
                         void *scratch, cudaStream_t st)
{
    DLOut o = {out, cs, ls, nullptr, nullptr};
    return gather_form<kDlNorm>(q, s_am, o, scratch, st);
}

int launch_dl_update(const DLPlan &q, const float *s_am, float *x, const float *inv, void *scratch,
                     cudaStream_t st)
{
    DLOut o = {nullptr, 0, 0, x, inv};
    return gather_form<kDlUpdate>(q, s_am, o, scratch, st);
}

}  // namespace rg
