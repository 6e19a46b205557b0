// radon_tma.cu -- slant-stack Radon with TMA-staged line windows.
//
// Same operator as radon_tile (raft/raft_radon_slantstack.c:122-214; see
// slantstack.cu): ray k of view j sums, over the lines i of the image, the
// linear interpolation at u = r0 + k rk + i ri (Q32.32), read as one pair
// (s - d, d) of the padded line-pair arrays.
//
// GB300 design.  A CTA owns 64 consecutive rays of a block of up to 16
// adjacent views of one orientation (lines = image rows, or columns).  On
// every image line those 64 x 16 sample positions fall inside one window of
// at most BW consecutive entries: the rays of a view are ~1 entry apart and
// adjacent views move the positions by a few entries.  The CTA walks the
// lines in strips of 16; for each strip one elected thread issues a single
// 3-D TMA load (cp.async.bulk.tensor) of the BW x 16 window box into shared
// memory, double-buffered on two mbarriers, so the next strip streams in
// while the current one is summed.  Entries outside the line-pair array
// (left of entry 0, right of the pitch, past line N-1) are zero-filled by the
// TMA unit, so the box needs no clamping.  Every (ray, view) then reads its
// samples with LDS.64 at a Q9.23 local position (index = bits 23..31, weight
// 1 + w from the low 23 bits); a thread carries one ray of four views.
//
// The host partitions the plan's views into blocks whose window provably
// fits: positions are affine in (ray, line), so the window width over all
// ray tiles and strips is largest at the corner tiles and strips, which are
// checked exactly in integer arithmetic.  The kernel re-derives each strip's
// window start from the same corner positions and checks the width again;
// a strip that would not fit is skipped with an error flag, never read out
// of bounds.  The window holds the positions of all the CTA's rays on all 16
// lines, on the image or off it, and holds zeros off it: so a warp walks a
// strip whole or not at all (lanes that start or end inside a strip each took a
// loop of their own: 512^2 x 360 53 -> 47.6 us, DDA 61 -> 54 us).  A slant-stack
// ray's run of strips is known from the start (ray_strips): the vote on a strip
// is two comparisons, where those of its two end positions took a twelfth of
// the kernel (2048^2 x 1800 2.05 -> 1.90 ms).  The plan also fixes the order in
// which the (ray tile, view block) CTAs are dispatched, most strips first
// (st_cta_order), so that the launch's last wave holds its lightest CTAs, and
// each CTA's range of strips, so that the first load starts before anything
// else.  One barrier closes a strip.  Every mbarrier wait is bounded; a CTA
// whose wait runs out sets the error flag, waits (bounded) for its own copies
// and leaves.
// expire_first (a test switch, 0 in normal use) makes each CTA's first strip
// wait give up at once, so that tests can see that path run and report.
#include <cuda.h>
#include <string.h>

#include <algorithm>
#include <climits>
#include <mutex>
#include <type_traits>
#include <vector>

#include "dda_lines.cuh"
#include "tma.cuh"

namespace rg {

constexpr int kTmRays = 64;     // rays per CTA (two warps of 32)
constexpr int kTmViews = 16;    // views per block (max)
constexpr int kTmVpt = 4;       // views per thread
constexpr int kTmLines = 16;    // lines per strip
// One full strip of a (ray, view): 16 lines, line r of the strip buffer at
// byte offset r * BW * 8 (an immediate of the load).  pb (== 8, the bytes
// of a pair) arrives as a kernel argument, so the sample's address is one
// integer multiply-add on the FMA pipe instead of a shift and an add on the
// integer pipe, which the position and weight bits keep busy (1024^2 x 720 230
// us; with the factor known to the compiler 254, with indexed shared memory
// 251).
//
// DDA: the pair is (s[n], s[n + 1] - s[n]) and the weight of s[n + 1] the
// part of the ray's strip that lies in pixel n + 1, a trapezoid: sat(wa f +
// 1 - wa) for position n + f, one saturated FMA of 1 + f (wc = 1 - 2 wa).
template <bool DDA>
__device__ __forceinline__ float line_sample(unsigned L, float2 pr, float wa, float wc)
{
    if constexpr (DDA) return fmaf(fma_sat(wa, frac_plus_one_opaque(L), wc), pr.y, pr.x);
    return fmaf(frac_plus_one_opaque(L), pr.y, pr.x);
}

// DDA: even and odd lines are summed apart (part, odd), each then added with
// compensation: the FP32 additions within a strip are most of the ray sum's
// error (256^2 x (367, 180): 3.8e-8 in one sum, 3.0e-8 in two, of which the
// final rounding is 2.5e-8).
template <int BW, int R0, bool DDA>
__device__ __forceinline__ void strip16(unsigned sb, unsigned &L, unsigned dq, unsigned pb,
                                        float wa, float wc, float &part, float &odd)
{
    if constexpr (R0 < kTmLines) {
        const float2 pr = lds_pair_at<R0 * BW * 8>((L >> 23) * pb + sb);
        if constexpr (DDA && R0 % 2 == 1) odd += line_sample<DDA>(L, pr, wa, wc);
        else part += line_sample<DDA>(L, pr, wa, wc);
        L += dq;
        strip16<BW, R0 + 1, DDA>(sb, L, dq, pb, wa, wc, part, odd);
    }
}

// Slant stack: the run of strips that a ray walks, from that of its first line on
// the image (bits 8 and up of `first`) to that of its last, by radon_line_range
// (whose check of the ends cannot fail here, where a strip's positions fit a
// window).
//
// A sample counts while its floor index is in [0, N - 2], and its value does not
// vanish at the ends, so it is one position that decides, to the last bit: on
// every strip the Q9.23 one that starts truncated at the ray's first line there
// and steps on.  That is the strip's first line but on the strip where the ray
// comes in; the low byte of `first` is the difference there, plus 128, between
// the position that starts at the ray's first line, brought back to the
// strip's, and the one that starts at the strip's (lines before the ray's first
// read zeros).  Positions centred on a strip give and take single samples.
__device__ __forceinline__ void ray_strips(long long u0, long long q, int N, unsigned &first,
                                           unsigned &last)
{
    const float uf = (float)u0 * 2.3283064365386963e-10f, qf = (float)q * 2.3283064365386963e-10f;
    int lo = 0, hi = N - 1;
    if (fabsf(qf) < 1e-20f) {
        if (!(uf >= -0.5f && uf <= (float)N - 0.5f)) hi = -1;
    } else {
        const float t1 = (-0.5f - uf) / qf, t2 = ((float)N - 0.5f - uf) / qf;
        lo = (int)ceilf(fmaxf(fminf(t1, t2), 0.f));
        hi = (int)floorf(fminf(fmaxf(t1, t2), (float)(N - 1)));
    }
    first = 0x7FFFFF00u;                              // no strip
    last = 0;
    if (lo > hi) return;
    const int m = lo & (kTmLines - 1);
    const long long ua = u0 + (long long)(lo - m) * q;
    const int c = (int)((ua + m * q) >> 9) - (int)(ua >> 9) - m * (int)((q + 256) >> 9);
    first = ((unsigned)lo / kTmLines << 8) | (unsigned)(c + 128);
    last = (unsigned)hi / kTmLines;
}

// Lane layout: each shared load of a warp covers RPL consecutive rays of
// 32 / RPL adjacent views.  Rays are >= 1 entry apart on a line while
// adjacent views sit a few entries apart, so fewer rays per load (more
// views) packs the 32 lanes' 8-byte reads into fewer shared-memory
// wavefronts.  A thread carries 4 (ray, view) pairs m: the warp's 32 rays x
// 4 views are covered as ray group m % (32 / RPL) and view group
// m / (32 / RPL).
//
// DDA: the line sums of dda_lines.cu.  Lines that are image rows are N lines
// of M samples, columns M lines of N; positions are Q24.40.  The grid's last
// rows of CTAs (from nblk) take the axis-aligned views, 8 rays each, beside the
// others instead of in a launch of their own (256^2 x (367, 180): 26 -> 21 us).
//
// Ray k of view j is stored at out[j ovs + k ors]: 16 consecutive views of 64
// rays per CTA, 16 bytes or more together in either layout, so that no pass
// follows to turn the sinogram over.
template <int EPI, int BW, int RPL, bool DDA>
__global__ __launch_bounds__(256, 3) void k_radon_tma(const __grid_constant__ CUtensorMap tm_rows,
                                                   const __grid_constant__ CUtensorMap tm_cols,
                                                   int N, int M, const View *__restrict__ views,
                                                   const StBlock *__restrict__ blocks,
                                                   const unsigned *__restrict__ order, int R,
                                                   float *__restrict__ out, long long ovs,
                                                   long long ors, const float *__restrict__ y_am,
                                                   int y_ld, long long zo, int *__restrict__ err,
                                                   unsigned pb, int expire_first, int split,
                                                   int nblk, const __grid_constant__
                                                   typename std::conditional<DDA, DLArgs, int>::type
                                                   dl)
{
    pdl_gate();
    if constexpr (DDA)
        if ((int)blockIdx.y >= nblk) {                // whole clusters
            dl_axis_cta<EPI>(dl, ((int)blockIdx.y - nblk) * gridDim.x + blockIdx.x, out, ovs, ors,
                             y_am, y_ld);
            return;
        }
    extern __shared__ __align__(128) float2 sbuf[];   // [2][kTmLines][BW]
    __shared__ __align__(8) unsigned long long full[2];
    __shared__ int xs[2];                             // window start entry per buffer
    __shared__ int bad[2];                            // window did not fit
    __shared__ long long cr0[kTmViews], crk[kTmViews], cri[kTmViews];
    // cluster partials (split > 1); DDA: sums, then their Kahan compensations
    __shared__ float red[(DDA ? 2 : 1) * kTmVpt][256];

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // split > 1: this CTA is rank `rank` of a cluster of `split` CTAs along x
    // that share the ray tile and view block; it walks its share of the
    // strips, and rank 0 sums the partials (distributed shared memory, rank
    // order) and writes the epilogue.  The cluster's (ray tile, view block)
    // comes from the plan's dispatch order (most lines first).
    const int rank = blockIdx.x % split;
    const unsigned slot = blockIdx.x / split + (gridDim.x / split) * blockIdx.y;
    const unsigned ord = order[slot];
    const unsigned range = order[gridDim.x / split * nblk + slot];
    const StBlock blk = blocks[ord & 0xffffu];
    const int k0 = (int)(ord >> 16) * kTmRays;
    constexpr int Q = DDA ? 40 : 32;                  // fraction bits of a position
    const int ne = !DDA || !(blk.flags & kLinesAreRows) ? N : M;
    constexpr int kRG = 32 / RPL;
    static_assert(RPL == 32 || RPL == 16 || RPL == 8, "rays per load");
    // pair m: ray k0 + 32 (warp & 1) + RPL (m % kRG) + lane % RPL,
    //         view (warp >> 1) * 4 + lane / RPL + (32 / RPL) (m / kRG)
    int kk_[kTmVpt], vv_[kTmVpt];
#pragma unroll
    for (int m = 0; m < kTmVpt; ++m) {
        kk_[m] = k0 + (warp & 1) * 32 + RPL * (m % kRG) + lane % RPL;
        vv_[m] = (warp >> 1) * kTmVpt + lane / RPL + (32 / RPL) * (m / kRG);
    }
    const int z = blockIdx.z;
    const CUtensorMap *tm = (blk.flags & kLinesAreRows) ? &tm_rows : &tm_cols;
    out += (long long)z * zo;

    // The strips that any ray of the CTA meets, first | last << 16 (the plan's;
    // first > last: none), and this rank's share of them.
    const int nall = (int)(range >> 16) - (int)(range & 0xffffu) + 1;
    const int s0 = (int)((long long)nall * rank / split);
    const int sfirst = (int)(range & 0xffffu) + s0;
    const int nstrips = (int)((long long)nall * (rank + 1) / split) - s0;
    const unsigned sbase = smem_addr(sbuf);
    constexpr unsigned kBufBytes = kTmLines * BW * 8;

    // Warp 0: window of strip n from the block's corner positions, then
    // lane 0 arms the buffer's barrier and issues the TMA load.
    auto issue = [&](int n) {
        const int i0 = (sfirst + n) * kTmLines;
        const int c = lane >> 1;
        int emin = INT_MAX, emax = INT_MIN;
        if (c < blk.count) {
            const int kk = (lane & 1) ? min(k0 + kTmRays - 1, R - 1) : k0;
            const long long ua = cr0[c] + (long long)kk * crk[c] + (long long)i0 * cri[c];
            const long long ub = ua + (kTmLines - 1) * cri[c];
            const int ea = (int)(ua >> Q) + 1, eb = (int)(ub >> Q) + 1;
            emin = min(ea, eb);
            emax = max(ea, eb);
        }
        emin = __reduce_min_sync(0xffffffffu, emin);
        emax = __reduce_max_sync(0xffffffffu, emax);
        // one entry of slack on both sides for the Q9.23 stepping
        const int x0 = (emin - 1) & ~1;
        if (lane == 0) {
            const int b = n & 1;
            xs[b] = x0;
            bad[b] = (emax + 1 - x0 >= BW) ? 1 : 0;
            fence_proxy_async_smem();
            mbar_expect_tx(smem_addr(&full[b]), kBufBytes);
            tma_load_3d(sbase + b * kBufBytes, tm, x0, i0, z, smem_addr(&full[b]));
        }
    };

    // Warp 0 starts the first strip's load before anything else is set up.
    if (warp == 0) {
        if (lane < blk.count) {
            const View &V = views[blk.first + lane];
            cr0[lane] = V.r0;
            crk[lane] = V.rk;
            cri[lane] = V.ri;
        }
        if (lane == 0) {
            mbar_init(smem_addr(&full[0]), 1);
            mbar_init(smem_addr(&full[1]), 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        if (nstrips > 0) issue(0);
    }

    // Threads past the block's views or the last ray walk the last ones again
    // (their windows hold no others) and store nothing.
    long long u0[kTmVpt], q[kTmVpt];
    unsigned first[kTmVpt], last[kTmVpt];             // slant stack: ray_strips
    // all four pairs of a thread are of one view at 8 rays per load
    static_assert(!DDA || RPL == 8, "the DDA form keeps one trapezoid per thread");
    float wa = 0.f, wc = 0.f;
#pragma unroll
    for (int v = 0; v < kTmVpt; ++v) {
        const View &V = views[blk.first + min(vv_[v], blk.count - 1)];
        u0[v] = V.r0 + (long long)min(kk_[v], R - 1) * V.rk;
        q[v] = V.ri;
        if constexpr (DDA) {
            wa = V.wa;
            wc = fmaf(-2.f, wa, 1.f);                 // exact
        } else {
            ray_strips(u0[v], q[v], N, first[v], last[v]);
        }
    }
    float acc[kTmVpt], comp[kTmVpt];
#pragma unroll
    for (int v = 0; v < kTmVpt; ++v) acc[v] = comp[v] = 0.f;
    __syncthreads();       // the barriers and strip 0's window are set up

    int n = 0;
    bool failed = false;
    for (; n < nstrips; ++n) {
        const int b = n & 1;
        // buffer b ^ 1 was last read in strip n - 1, which every thread
        // finished before the barrier that closed it
        if (warp == 0 && n + 1 < nstrips) issue(n + 1);
        // A wait that runs out is acted on at the strip's closing barrier:
        // until then the thread sums whatever the buffer holds (its reads
        // stay inside it), and the call reports the error.
        const bool ok = (expire_first && n == 0) ? false
                                                 : mbar_wait(smem_addr(&full[b]), (n >> 1) & 1);
        const int i0 = (sfirst + n) * kTmLines;
        if (!bad[b]) {
            const int x0 = xs[b];
            const unsigned sb = sbase + b * kBufBytes;
#pragma unroll
            for (int v = 0; v < kTmVpt; ++v) {
                // All 16 lines, for the whole warp, where any of its rays meets the
                // strip: samples off the line or past the last line read zeros
                // (the window covers every position of the CTA's rays).
                const long long ua = u0[v] + (long long)i0 * q[v];
                unsigned shift = 0;                   // under 256: the ray comes in here
                bool meets;
                if constexpr (DDA) {
                    const long long ub = ua + (kTmLines - 1) * q[v];
                    meets = max(ua, ub) >= -(1LL << Q) && min(ua, ub) < (long long)ne << Q;
                } else {
                    shift = first[v] - ((unsigned)i0 / kTmLines << 8);
                    meets = (int)shift < 256 && (unsigned)i0 / kTmLines <= last[v];
                }
                if (!__any_sync(0xffffffffu, meets)) continue;
                const long long dq64 = (q[v] + (1LL << (Q - 24))) >> (Q - 23);
                const unsigned dq = (unsigned)dq64;
                unsigned L;
                if constexpr (DDA) {
                    // The rounding of the Q9.23 step is spread evenly about the
                    // strip's middle line instead of growing along it.
                    L = (unsigned)((ua - ((long long)(x0 - 1) << Q) + (1LL << (Q - 24)) +
                                    ((q[v] - (dq64 << (Q - 23))) * (kTmLines - 1) >> 1)) >>
                                   (Q - 23));
                } else {
                    L = (unsigned)((ua - ((long long)(x0 - 1) << Q)) >> (Q - 23));
                    if (shift < 256u) L += shift - 128u;
                }
                float part = 0.f, odd = 0.f;
                strip16<BW, 0, DDA>(sb, L, dq, pb, wa, wc, part, odd);
                kahan_add(acc[v], comp[v], part);
                if constexpr (DDA) kahan_add(acc[v], comp[v], odd);
            }
        } else if (threadIdx.x == 0 && err) {
            atomicOr(err, 1);
        }
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
    }
    if (failed && threadIdx.x == 0) {
        if (err) atomicOr(err, 2);
        // copies still in flight: strip n (buffer n & 1) and, if issued,
        // strip n + 1; wait for them (bounded) before leaving
        mbar_wait(smem_addr(&full[n & 1]), (n >> 1) & 1);
        if (n + 1 < nstrips) mbar_wait(smem_addr(&full[(n + 1) & 1]), ((n + 1) >> 1) & 1);
    }

    float tot[kTmVpt];
#pragma unroll
    for (int v = 0; v < kTmVpt; ++v) tot[v] = acc[v] - comp[v];
    if (split > 1) {
        namespace cg = cooperative_groups;
        cg::cluster_group cl = cg::this_cluster();
#pragma unroll
        for (int v = 0; v < kTmVpt; ++v) {
            red[v][threadIdx.x] = DDA ? acc[v] : tot[v];
            if constexpr (DDA) red[kTmVpt + v][threadIdx.x] = comp[v];
        }
        cl.sync();
        if (rank == 0) {
            if constexpr (DDA) {                      // acc, comp: this rank's own
                for (int src = 1; src < split; ++src) {
                    const float *peer = cl.map_shared_rank(&red[0][0], src);
#pragma unroll
                    for (int v = 0; v < kTmVpt; ++v) {
                        two_sum_add(acc[v], comp[v], peer[v * 256 + threadIdx.x],
                                    peer[(kTmVpt + v) * 256 + threadIdx.x]);
                    }
                }
            } else {
#pragma unroll
                for (int v = 0; v < kTmVpt; ++v) tot[v] = 0.f;
                for (int src = 0; src < split; ++src) {
                    const float *peer = cl.map_shared_rank(&red[0][0], src);
#pragma unroll
                    for (int v = 0; v < kTmVpt; ++v) tot[v] += peer[v * 256 + threadIdx.x];
                }
            }
        }
        cl.sync();    // no CTA leaves while rank 0 still reads its partials
        if (rank != 0) return;
    }
    unsigned bad_rays = 0;
    int j = 0;
#pragma unroll
    for (int v = 0; v < kTmVpt; ++v) {
        if (vv_[v] >= blk.count || kk_[v] >= R) continue;
        const View &V = views[blk.first + vv_[v]];
        // DDA: (acc - comp) times Delta, rounded once
        const float val = DDA ? fmaf(acc[v], V.delta, fmaf(acc[v], V.delta_lo, -comp[v] * V.delta))
                              : tot[v] * V.delta;
        out[V.view * ovs + kk_[v] * ors] =
            radon_epilogue(EPI, val, y_am, (size_t)V.view * y_ld + kk_[v]);
        if constexpr (DDA) {
            j = V.view;
            if (!isfinite(val) || kk_[v] == V.brow) bad_rays |= 1u << v;
        }
    }
    if constexpr (DDA)
        if (bad_rays) dl_walk_rays<EPI>(dl, bad_rays, kk_[0], j, out, ovs, ors, y_am, y_ld);
}

// ----------------------------------------------------------------------------
// Host side.

// Window width (entries, with the kernel's slack) of a growing block of
// views, over the corner ray tiles and strips (positions are affine in
// (ray, line), so the width over every tile and strip is largest there).
struct BlockSpan {
    long long emin[4], emax[4];
    int k0[2], i0[2], Q;
    BlockSpan(int nl, int R, int Q) : Q(Q)
    {
        k0[0] = 0;
        k0[1] = ((R - 1) / kTmRays) * kTmRays;
        i0[0] = 0;
        i0[1] = ((nl - 1) / kTmLines) * kTmLines;
        for (int c = 0; c < 4; ++c) { emin[c] = LLONG_MAX; emax[c] = LLONG_MIN; }
    }
    void add(const View &v, long long *mn, long long *mx) const
    {
        for (int c = 0; c < 4; ++c) {
            mn[c] = emin[c];
            mx[c] = emax[c];
            const int ka = k0[c & 1], ia = i0[c >> 1];
            for (int kk : {ka, ka + kTmRays - 1})
                for (int ii : {ia, ia + kTmLines - 1}) {
                    const long long u = v.r0 + (long long)kk * v.rk + (long long)ii * v.ri;
                    const long long en = (u >> Q) + 1;
                    mn[c] = std::min(mn[c], en);
                    mx[c] = std::max(mx[c], en);
                }
        }
    }
    static long long width(const long long *mn, const long long *mx)
    {
        long long w = 0;
        for (int c = 0; c < 4; ++c) w = std::max(w, mx[c] + 2 - ((mn[c] - 1) & ~1LL));
        return w;
    }
};

static bool radon_kernel_direct()
{
    const char *e = getenv("RG_RADON_KERNEL");
    return e && !strcmp(e, "direct");
}

// Dispatch order of the TMA Radon's CTAs, as (ray tile << 16 | block): the
// CTA of ray tile t and view block b walks the strips of lines that any of
// its rays meets, so the central ray tiles of oblique views carry several
// times the lines of the edge tiles.  Launched in grid order, the last wave
// mixes heavy and light CTAs and the SMs that drew heavy ones finish late;
// issued longest first (CTAs are dispatched in linear order), the last wave
// holds the lightest CTAs.  A line is met by one of the tile's rays where the
// positions from its first ray's to its last's meet the line's samples, an
// interval of lines per view, taken with a line's margin.  The second half of
// the table is each CTA's range of strips (first | last << 16, first > last:
// none).
static std::vector<unsigned> st_cta_order(const std::vector<StBlock> &bl, const View *hv,
                                          const SSPlan &p)
{
    const int R = p.g.R;
    const int T = (R + kTmRays - 1) / kTmRays, nb = (int)bl.size();
    const double q1 = p.dda ? 0x1p-40 : 0x1p-32;
    std::vector<int> strips((size_t)T * nb, 0);
    std::vector<unsigned> range((size_t)T * nb, 1u);       // none
    for (int b = 0; b < nb; ++b) {
        const int o = (bl[b].flags & kLinesAreRows) ? 0 : 1, nl = p.nl[o], ne = p.ne[o];
        for (int t = 0; t < T; ++t) {
            int Lo = INT_MAX, Hi = INT_MIN;
            const int ka = t * kTmRays, kb = std::min(ka + kTmRays - 1, R - 1);
            for (int c = 0; c < bl[b].count; ++c) {
                const View &v = hv[bl[b].first + c];
                const double u = (double)v.r0 * q1 + ka * ((double)v.rk * q1);
                const double w = (kb - ka) * ((double)v.rk * q1), q = (double)v.ri * q1;
                // u + i q + [0, w] meets [-1, ne]
                const double lo = -1.0 - std::max(w, 0.0) - u, hi = ne - std::min(w, 0.0) - u;
                double i0 = 0.0, i1 = nl - 1.0;
                if (fabs(q) > 1e-12) {
                    i0 = std::max(i0, floor(std::min(lo / q, hi / q)) - 1.0);
                    i1 = std::min(i1, ceil(std::max(lo / q, hi / q)) + 1.0);
                } else if (lo > 1e-6 || hi < -1e-6) {
                    continue;
                }
                if (i0 > i1) continue;
                Lo = std::min(Lo, (int)i0);
                Hi = std::max(Hi, (int)i1);
            }
            if (Lo > Hi) continue;
            strips[(size_t)b * T + t] = Hi / kTmLines - Lo / kTmLines + 1;
            range[(size_t)b * T + t] =
                (unsigned)(Lo / kTmLines) | (unsigned)(Hi / kTmLines) << 16;
        }
    }
    std::vector<unsigned> order((size_t)T * nb);
    for (size_t i = 0; i < order.size(); ++i) order[i] = (unsigned)i;
    std::stable_sort(order.begin(), order.end(),
                     [&](unsigned a, unsigned b) { return strips[a] > strips[b]; });
    std::vector<unsigned> out(2 * order.size());
    for (size_t i = 0; i < order.size(); ++i) {
        const unsigned o = order[i];
        out[i] = ((o % (unsigned)T) << 16) | (o / (unsigned)T);
        out[order.size() + i] = range[o];
    }
    return out;
}

int st_blocks_build(SSPlan &p, const View *hv)
{
    p.nblocks = 0;
    p.st_bw = 0;
    const int R = p.g.R, nv = p.nv;
    // the dispatch order packs the ray tile, the strips and the block into 16 bits
    if (nv < 1 || (R + kTmRays - 1) / kTmRays > 65535 ||
        std::max(p.nl[0], p.nl[1]) / kTmLines > 65535)
        return RG_OK;
    for (int bw : {128, 256}) {
        std::vector<StBlock> bl;
        bool fits = true;
        for (int e = 0; e < nv && fits;) {
            BlockSpan sp(p.nl[(hv[e].flags & kLinesAreRows) ? 0 : 1], R, p.dda ? 40 : 32);
            long long mn[4], mx[4];
            sp.add(hv[e], mn, mx);
            if (BlockSpan::width(mn, mx) > bw) { fits = false; break; }
            memcpy(sp.emin, mn, sizeof mn);
            memcpy(sp.emax, mx, sizeof mx);
            int c = 1;
            while (c < kTmViews && e + c < nv &&
                   (hv[e + c].flags & kLinesAreRows) == (hv[e].flags & kLinesAreRows)) {
                sp.add(hv[e + c], mn, mx);
                if (BlockSpan::width(mn, mx) > bw) break;
                memcpy(sp.emin, mn, sizeof mn);
                memcpy(sp.emax, mx, sizeof mx);
                ++c;
            }
            bl.push_back(StBlock{e, c, hv[e].flags & kLinesAreRows, 0});
            e += c;
        }
        // worth it only when blocks share their windows among several views
        if (!fits || (int)bl.size() > 65535 || nv < 6 * (int)bl.size()) continue;
        if (bw == 128 && nv < 12 * (int)bl.size()) continue;   // 256 packs more views
        const std::vector<unsigned> order = st_cta_order(bl, hv, p);
        const size_t bb = sizeof(StBlock) * bl.size();
        RG_CK(cudaMalloc(&p.d_blocks, bb + sizeof(unsigned) * order.size()));
        RG_CK(cudaMemcpy(p.d_blocks, bl.data(), bb, cudaMemcpyHostToDevice));
        p.d_border = (const unsigned *)((char *)p.d_blocks + bb);
        RG_CK(cudaMemcpy((void *)p.d_border, order.data(), sizeof(unsigned) * order.size(),
                         cudaMemcpyHostToDevice));
        p.nblocks = (int)bl.size();
        p.st_bw = bw;
        return RG_OK;
    }
    return RG_OK;
}

EncodeTiledFn tensor_map_encoder()
{
    static std::once_flag once;
    static EncodeTiledFn fn = nullptr;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000,
                                             cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)f;
        else
            cudaGetLastError();
    });
    return fn;
}

// 3-D map over nz stacked line-pair arrays of nl lines of ne samples:
// (entry, line, image), 8-byte elements, box bw x kTmLines x 1, zero fill
// outside.
static int encode_pairs_map(CUtensorMap *tm, const float2 *pairs, int nl, int ne, int nz,
                            long long zp, int bw)
{
    EncodeTiledFn fn = tensor_map_encoder();
    if (!fn) return set_error(RG_ECUDA, "cuTensorMapEncodeTiled is not available");
    const int pitch = pairs_pitch(ne);
    cuuint64_t dims[3] = {(cuuint64_t)pitch, (cuuint64_t)nl, (cuuint64_t)nz};
    cuuint64_t strides[2] = {(cuuint64_t)pitch * 8,
                             (cuuint64_t)(nz > 1 ? zp : (long long)nl * pitch) * 8};
    cuuint32_t box[3] = {(cuuint32_t)bw, (cuuint32_t)kTmLines, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, (void *)pairs, dims, strides, box,
                    estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return set_error(RG_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return RG_OK;
}

bool radon_tma_usable(const SSPlan &p)
{
    const char *e = getenv("RG_RADON_KERNEL");
    const bool tiles = e && !strcmp(e, "tiles") && p.tt_ok && p.d_ovid;   // forced
    return p.nblocks > 0 && p.d_blocks && !tiles && !radon_kernel_direct();
}

// Rays per shared load (lane layout); RG_RADON_RPL=32|16|8 overrides.
static int radon_rpl()
{
    const char *e = getenv("RG_RADON_RPL");
    const int v = e ? atoi(e) : 0;
    return (v == 32 || v == 16 || v == 8) ? v : 8;
}

// Cluster size of the strip split for a grid of `ctas` CTAs at `slots`
// resident CTAs.  Measured on GB300 (slant-stack Radon, GUPS, split 1 / 2 / 4;
// waves of the unsplit grid): 2048^2 x 1800 (8.1) 3997 / 3960 / 3725; 1024^2 x
// 720 (1.6) 3410 / 3458 / 3212; 975^2, 886 rays x 621 (1.2) 3082 / 3255 / 3071;
// 512^2 x 360 (0.4) 1211 / 1992 / 2052.  Each rank repeats the CTA's set-up and
// the ranks' partials meet in distributed shared memory, so a split pays only
// where the unsplit grid leaves SMs idle: 1 from 2.5 waves up, 2 from one wave,
// else 4, with at least 4 strips of kTmLines lines per rank.
// RG_RADON_SPLIT_TMA=1|2|4 forces it.
static int tma_pick_split(long long ctas, int slots, int N)
{
    const char *e = getenv("RG_RADON_SPLIT_TMA");
    const int forced = e ? atoi(e) : 0;
    if (forced == 1 || forced == 2 || forced == 4) return forced;
    int s = ctas >= 5LL * slots / 2 ? 1 : ctas >= slots ? 2 : 4;
    while (s > 1 && (N / kTmLines) / s < 4) s /= 2;
    return s;
}

struct TmaOut {
    float *out;
    long long ovs, ors;
    const float *y_am;
    int y_ld, nz;
    long long zo;
};

template <int EPI, int BW, int RPL, bool DDA = false>
static int launch_tma_rpl(const SSPlan &p, const CUtensorMap &tr, const CUtensorMap &tc,
                          const TmaOut &o, const DLArgs *dl, cudaStream_t st)
{
    const size_t smem = (size_t)2 * kTmLines * BW * 8;
    auto k = k_radon_tma<EPI, BW, RPL, DDA>;
    RG_CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid((p.g.R + kTmRays - 1) / kTmRays, p.nblocks, o.nz);
    // resident CTAs of this instantiation (cached: no queries in a capture)
    static int slots = 0;
    if (!slots) {
        int dev = 0, sms = 0, per = 0;
        RG_CK(cudaGetDevice(&dev));
        RG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        RG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, 256, smem));
        slots = std::max(1, per) * sms;
    }
    const int split = tma_pick_split((long long)grid.x * grid.y * grid.z, slots,
                                     std::min(p.nl[0], p.nl[1]));
    const int expire = test_switch("RG_TEST_EXPIRE_WAIT") ? 1 : 0;
    int axis_rows = 0;
    typename std::conditional<DDA, DLArgs, int>::type args{};
    if constexpr (DDA) {
        args = *dl;
        const int ctas = (int)(((long long)dl->nax * p.g.R + 7) / 8), gx = (int)grid.x * split;
        axis_rows = (ctas + gx - 1) / gx;
    }
    RG_CK(launch_pdl(k, dim3(grid.x * split, grid.y + axis_rows, grid.z), 256, smem, st, split,
                     tr, tc, p.nl[0], p.ne[0], (const View *)p.d_views,
                     (const StBlock *)p.d_blocks, p.d_border, p.g.R, o.out, o.ovs, o.ors, o.y_am,
                     o.y_ld, o.zo, device_error_word(), (unsigned)sizeof(float2), expire, split,
                     p.nblocks, args));
    RG_CK_LAUNCH("k_radon_tma");
    return RG_OK;
}

template <int EPI, int BW>
static int launch_tma_bw(const SSPlan &p, const CUtensorMap &tr, const CUtensorMap &tc,
                         const TmaOut &o, const DLArgs *dl, cudaStream_t st)
{
    if (p.dda) return launch_tma_rpl<EPI, BW, 8, true>(p, tr, tc, o, dl, st);
    switch (radon_rpl()) {
    case 32: return launch_tma_rpl<EPI, BW, 32>(p, tr, tc, o, dl, st);
    case 16: return launch_tma_rpl<EPI, BW, 16>(p, tr, tc, o, dl, st);
    default: return launch_tma_rpl<EPI, BW, 8>(p, tr, tc, o, dl, st);
    }
}

template <int EPI>
static int launch_tma_epi(const SSPlan &p, const CUtensorMap &tr, const CUtensorMap &tc,
                          const TmaOut &o, const DLArgs *dl, cudaStream_t st)
{
    if (p.st_bw == 128) return launch_tma_bw<EPI, 128>(p, tr, tc, o, dl, st);
    return launch_tma_bw<EPI, 256>(p, tr, tc, o, dl, st);
}

int launch_radon_tma(const SSPlan &p, const float2 *prow, const float2 *pcol, float *out,
                     long long ovs, long long ors, const float *y_am, int y_ld, cudaStream_t st,
                     int nz, long long zp, long long zo, int epi, const DLArgs *dl)
{
    if (p.dda != (dl != nullptr))
        return set_error(RG_EINVAL, "TMA Radon: DDA plans come with their rays");
    CUtensorMap tr, tc;
    int rc = encode_pairs_map(&tr, prow, p.nl[0], p.ne[0], nz, zp, p.st_bw);
    if (!rc) rc = encode_pairs_map(&tc, pcol, p.nl[1], p.ne[1], nz, zp, p.st_bw);
    if (rc) return rc;
    const TmaOut o = {out, ovs, ors, y_am, y_ld, nz, zo};
    if (epi == kEpiRatio) return launch_tma_epi<kEpiRatio>(p, tr, tc, o, dl, st);
    if (epi == kEpiTransmission) return launch_tma_epi<kEpiTransmission>(p, tr, tc, o, dl, st);
    return launch_tma_epi<kEpiSum>(p, tr, tc, o, dl, st);
}


// ============================================================================
// Tile-driven Radon for plans of scattered views (OSEM subsets).
//
// The view-block windows above need adjacent views; a subset's views are S
// apart, so their positions on a line spread too far for one window.  Here
// the loop order is turned around: a CTA owns an image tile -- kTtLines lines
// x kTtWin line-pair entries [p0, p0 + kTtWin) of one orientation -- staged
// once, straight from the image (tt_stage), and every view of the plan with that orientation sends through it the rays
// that cross it.  Each staged entry then serves every view (tens to
// hundreds), not the few views of a block.
//
// Ownership: a sample (ray, line) belongs to the tile whose line block holds
// the line and whose window holds the sample's entry.  Each smem row carries
// kTtPad zero entries on both sides of the window, wide enough for any
// crossing ray's positions on the tile's lines (checked per plan on the host
// and per ray in the kernel), so a ray adds exactly its owned samples with
// the plain 7-instruction walk of the other kernels, and samples outside
// the window read zeros.  Each (ray, view, tile) partial, times Delta, is
// added to the sinogram with one atomic add (the zeroing pass before and
// the epilogue pass after are separate launches; the EM loops let one
// subset's epilogue clear the next one's rows); the order of those adds
// varies between runs, at the level of FP32 rounding.
//
// The walk waits on its shared loads (3.2 wavefronts a load where rays are as
// dense as pixels: L1 is 68 % busy at 24 warps an SM), so it wants warps: 3
// CTAs of 512 threads fit an SM.  1024^2, 72 views (one of 10 subsets): 53 us
// with CTAs of 256 threads, line pairs packed and rows zeroed by passes of
// their own; 49 us with 256 threads and 41 with 512 from the image; 39 with a
// view's last rays in one warp with the next view's first (tt_views).
constexpr int kTtThreads = 512;

__global__ __launch_bounds__(kTtThreads) void k_radon_tiles(const float *__restrict__ img,
                                                            long long ics, long long ils,
                                                            long long zi, int N,
                                                            const TtView *__restrict__ ttv,
                                                            int n_rows, int n_cols, int R,
                                                            float *__restrict__ out_am,
                                                            int out_ld, long long zo,
                                                            int *__restrict__ err, unsigned pb)
{
    pdl_gate();
    extern __shared__ __align__(128) float2 tile[];   // [kTtLines][kTtRow]
    const int o = blockIdx.z & 1, z = blockIdx.z >> 1;
    const int nvo = o ? n_cols : n_rows;
    if (nvo == 0) return;                              // CTA-uniform, before any barrier
    const int p0 = blockIdx.x * kTtWin, i0 = blockIdx.y * kTtLines;
    // zero pads on both sides of the window
    constexpr int pads = kTtRow - kTtWin;
    for (int e = threadIdx.x; e < kTtLines * pads; e += kTtThreads) {
        const int r = e / pads, c = e - r * pads;
        tile[r * kTtRow + (c < kTtPad ? c : kTtWin + c)] = make_float2(0.f, 0.f);
    }
    tt_stage<kTtLines, kTtWin, kTtPad, kTtRow, kTtThreads, 5, 10>(tile, img + z * zi, ics, ils, N,
                                                                  p0, i0, o);
    __syncthreads();
    tt_views<kTtRow, kTtLines, kTtPad, kTtThreads>(smem_addr(tile), p0, i0,
                                                   ttv + (o ? n_rows : 0), nvo, R,
                                                   out_am + (long long)z * zo, out_ld, err, pb);
}

// out[view][k] = 0 for the plan's views (EPI < 0), or the epilogue of the
// summed rays; the rows of CTAs past the plan's views (nz of `znext`) clear
// the rows of those views, which a later launch sums into.
template <int EPI>
__global__ __launch_bounds__(256) void k_views_rows(const View *__restrict__ views, int nv, int R,
                                                    float *__restrict__ out_am, int out_ld,
                                                    const float *__restrict__ y_am, int y_ld,
                                                    long long zo,
                                                    const View *__restrict__ znext)
{
    pdl_gate();
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (k >= R) return;
    const bool zero = EPI < 0 || j >= nv;
    const int view = zero && EPI >= 0 ? znext[j - nv].view : views[j].view;
    float *o = out_am + (long long)blockIdx.z * zo + (size_t)view * out_ld + k;
    if (zero) *o = 0.f;
    else *o = radon_epilogue(EPI, *o, y_am, (size_t)view * y_ld + k);
}

bool tt_pads_fit(const SSPlan &p, int lines, int pad)
{
    return (lines - 1) * p.tt_ri_max + 3.0 * p.tt_rk_max + 3.0 <= pad;
}

int tt_build(SSPlan &p, const View *hv)
{
    p.tt_ok = false;
    p.n_ovid[0] = p.n_ovid[1] = 0;
    const int nv = p.nv;
    if (nv < 1) return RG_OK;
    std::vector<int> ids;
    for (int o = 0; o < 2; ++o)
        for (int e = 0; e < nv; ++e)
            if (((hv[e].flags & kLinesAreRows) ? 0 : 1) == o) {
                ids.push_back(e);
                ++p.n_ovid[o];
            }
    // pads must hold any crossing ray's positions on the tile's lines: the
    // walk across the tile's lines plus the margin rays (two each side)
    for (int e = 0; e < nv; ++e) {
        p.tt_ri_max = std::max(p.tt_ri_max, fabs((double)hv[e].ri) * 2.3283064365386963e-10);
        p.tt_rk_max = std::max(p.tt_rk_max, fabs((double)hv[e].rk) * 2.3283064365386963e-10);
    }
    if (!tt_pads_fit(p, kTtLines, kTtPad)) return RG_OK;
    std::vector<TtView> tv(ids.size());
    for (size_t q = 0; q < ids.size(); ++q) {
        const View &v = hv[ids[q]];
        tv[q].r0 = v.r0;
        tv[q].rk = v.rk;
        tv[q].ri = v.ri;
        tv[q].delta = v.delta;
        tv[q].view = v.view;
    }
    RG_CK(cudaMalloc(&p.d_ovid, sizeof(TtView) * tv.size()));
    RG_CK(cudaMemcpy(p.d_ovid, tv.data(), sizeof(TtView) * tv.size(), cudaMemcpyHostToDevice));
    p.tt_ok = true;
    return RG_OK;
}

bool radon_tiles_usable(const SSPlan &p)
{
    const char *e = getenv("RG_RADON_KERNEL");
    if (e && !strcmp(e, "direct")) return false;
    if (!p.tt_ok || !p.d_ovid) return false;
    if (e && !strcmp(e, "tiles")) return true;
    return !radon_tma_usable(p) && p.nv >= 16;
}

int launch_radon_tiles(const SSPlan &p, const float *img, long long ics, long long ils,
                       long long zi, float *out_am, int out_ld, const float *y_am, int y_ld,
                       cudaStream_t st, int nz, long long zo, int epi, bool zeroed,
                       const SSPlan *next)
{
    const int N = p.g.N, R = p.g.R;
    const dim3 gv((R + 255) / 256, p.nv, nz);
    if (!zeroed) {
        RG_CK(launch_pdl(k_views_rows<-1>, gv, 256, 0, st, 1, p.d_views, p.nv, R, out_am, out_ld,
                         nullptr, 0, zo, nullptr));
        RG_CK_LAUNCH("k_views_rows (zero)");
    }
    const size_t smem = (size_t)kTtLines * kTtRow * 8;
    RG_CK(cudaFuncSetAttribute(k_radon_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem));
    const dim3 grid((pairs_pitch(N) + kTtWin - 1) / kTtWin, (N + kTtLines - 1) / kTtLines,
                    2 * nz);
    RG_CK(launch_pdl(k_radon_tiles, grid, kTtThreads, smem, st, 1, img, ics, ils, zi, N,
                     (const TtView *)p.d_ovid, p.n_ovid[0], p.n_ovid[1], R, out_am, out_ld, zo,
                     device_error_word(), (unsigned)sizeof(float2)));
    RG_CK_LAUNCH("k_radon_tiles");
    const dim3 ge(gv.x, p.nv + (next ? next->nv : 0), nz);
    const View *zv = next ? next->d_views : nullptr;
    if (epi == kEpiRatio)
        RG_CK(launch_pdl(k_views_rows<kEpiRatio>, ge, 256, 0, st, 1, p.d_views, p.nv, R, out_am,
                         out_ld, y_am, y_ld, zo, zv));
    else if (epi == kEpiTransmission)
        RG_CK(launch_pdl(k_views_rows<kEpiTransmission>, ge, 256, 0, st, 1, p.d_views, p.nv, R,
                         out_am, out_ld, y_am, y_ld, zo, zv));
    RG_CK_LAUNCH("k_views_rows (epilogue)");
    return RG_OK;
}

}  // namespace rg
