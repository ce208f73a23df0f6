// vorticity.cu -- induced vorticity of Gaussian blobs by direct summation.
//
//   w_k = 1/(pi ksigmasqr) sum_m g_m exp(-r2/ksigmasqr),
//   r2 = dx^2 + dy^2 + 1e-12,  (dx, dy) = target_k - blob_m
//
// Replaces ww2parGauss_C_cpu (src/cpp/blobs/c/ww2parGauss_C/
// ww2parGauss_C_cpu.c:89-150) and its GPU twin, reached from
// _vorticity_direct_{cpu,gpu}_gauss (src/python/blobs/base/induced/
// _induced.py:702-963).  Same structure as the velocity direct sum
// (direct.cu): a CTA owns 512 targets (two per lane, packed f32x2), sources
// stream through shared memory as hi/lo float pairs, FP32 partial sums over 32
// sources (one chunk) fold into TwoSum-compensated (hi, lo) accumulators, and the
// sources are cut into segments whose partial sums are added in segment order.
//
// Sets of many pairs (k_vort_gauss).  Beyond r2 = V_FAR ksigmasqr / log2(e) the exponential underflows to +0 in
// FP32 (ex2.approx.ftz: below 2^-126), so such a pair adds exactly nothing.
// Blobs of a remeshed set come in lattice order, so most sources lie that far
// from all 64 (consecutive) targets of a warp: each tile of sources is tested
// against the CTA's targets as it is loaded, each chunk that has a source in reach
// against the warp's, and only the sources in reach are evaluated, in their order:
// bitwise the sum over all sources of those tiles.  A segment takes every
// splits-th tile there, so that the tiles in reach are spread over the segments;
// targets without spatial order take every pair of contiguous segments, so the
// last bits of a target's value depend on which of the two its CTA takes.  (A
// source that is not finite is never skipped, nor any source for a target that is
// not.)  Bound: issue of the pairs in reach (15 instructions each), then the tests.
// 40,401 blobs of a 201 x 201 lattice at themselves: 617 -> 106 us.
//
// The CUTOFF variant is the cutoff kernel's induced vorticity of
// ww2par_C_cpu (src/cpp/blobs/c/ww2par_C/ww2par_C_cpu.c:132-145) and its GPU
// twin (src/cpp/blobs/cuda/ww2par_gpu/ww2par_device.cu:59-70), as
// those compute it: w_k = 1/(2 pi) sum_m g_m / sqrt(r2 + sigma^2).
#include "direct_api.cuh"
#include "gauss_pair.cuh"

#include <algorithm>
#include <climits>

namespace {

constexpr int VT_THREADS = 256;
constexpr int VT_CHUNK = 32;
constexpr int64_t VT_CTAS = 5;  // CTAs resident per SM (registers)
constexpr int64_t VT_TILE = VT_THREADS * 2;
constexpr double INV_PI = 0.3183098861837907;  // 1/pi
constexpr double INV_2PI = 0.15915494309189535;  // 1/(2 pi)

// Two targets (packed) against one source: acc += g * 2^(r2 * c_t).
__device__ __forceinline__ void wpair2(const ulonglong2 &hi, const ulonglong2 &lo, pfd::f32x2 g2,
                                       pfd::f32x2 txh, pfd::f32x2 tyh, pfd::f32x2 txl,
                                       pfd::f32x2 tyl, const pfd::GaussParams2 &gp,
                                       pfd::f32x2 &acc) {
    const pfd::f32x2 dx = pfd::add2(pfd::sub2(txh, hi.x), pfd::sub2(txl, lo.x));
    const pfd::f32x2 dy = pfd::add2(pfd::sub2(tyh, hi.y), pfd::sub2(tyl, lo.y));
    const pfd::f32x2 r2 = pfd::fma2(dx, dx, pfd::fma2(dy, dy, gp.eps));
    float ta, tb;
    pfd::unpack2(pfd::mul2(r2, gp.c_t), ta, tb);
    acc = pfd::fma2(g2, pfd::pack2(pfd::ex2_approx(ta), pfd::ex2_approx(tb)), acc);
}

// Cutoff kernel: acc += g / sqrt(r2 + sigma^2), s2 = {sigma^2, sigma^2}.
__device__ __forceinline__ void wpair2_cutoff(const ulonglong2 &hi, const ulonglong2 &lo,
                                              pfd::f32x2 g2, pfd::f32x2 txh, pfd::f32x2 tyh,
                                              pfd::f32x2 txl, pfd::f32x2 tyl, pfd::f32x2 s2,
                                              pfd::f32x2 &acc) {
    const pfd::f32x2 dx = pfd::add2(pfd::sub2(txh, hi.x), pfd::sub2(txl, lo.x));
    const pfd::f32x2 dy = pfd::add2(pfd::sub2(tyh, hi.y), pfd::sub2(tyl, lo.y));
    const pfd::f32x2 r2 = pfd::fma2(dx, dx, pfd::fma2(dy, dy, s2));
    float ra, rb;
    pfd::unpack2(r2, ra, rb);
    acc = pfd::fma2(g2, pfd::pack2(pfd::rsqrt_approx(ra), pfd::rsqrt_approx(rb)), acc);
}

// Pairs from which the Gaussian's sources are tested.  Below, a CTA has one or two
// tiles, so that a lattice's CTAs with a tile in reach take as long as with every
// pair, and the tests come on top: lattices of 3,000 / 5,000 / 7,100 / 9,200 blobs
// 19.9 / 24.9 / 33.3 / 47.6 us with every pair, 23.0 / 29.2 / 37.4 / 53.8 tested; of
// 9,409 and 10,000 47.7 and 51.9, tested 39.5 and 39.4 (between 7,500 and 9,200
// either may be 8% faster, by how the lattice's columns fall on the tiles).
constexpr double V_TEST_PAIRS = 8.5e7;
constexpr double V_FAR = 127.5;  // ex2(-V_FAR) is below 2^-126 whatever its rounding
constexpr int VT_DENSE = 20;     // sources in reach from which a whole chunk is run unrolled

// Every pair, segment y the seg sources from y seg on: the cutoff kernel, and the
// Gaussian where there are too few pairs for the tests (V_TEST_PAIRS).  (A least
// number of CTAs, so 48 registers, makes the cutoff kernel 2% faster: 40,401 blobs
// 586 -> 573 us; the Gaussian is fastest with the 41 the compiler takes by itself.)
// w = (c1 * sum) / scale: Gauss c1 = 1/pi, scale = ksigmasqr; cutoff c1 =
// 1/(2 pi), scale = 1.
template <bool CUTOFF>
__global__ void __launch_bounds__(VT_THREADS, CUTOFF ? VT_CTAS : 0)
k_vort_pairs(const double *__restrict__ xs, const double *__restrict__ ys,
             const double *__restrict__ gs, int64_t ns, int64_t seg,
             const double *__restrict__ xt, const double *__restrict__ yt, int64_t nt,
             pfd::GaussParams gp, double c1, double scale, float s2, double *__restrict__ w,
             float2 *__restrict__ part) {
    __shared__ ulonglong2 s_hi[VT_THREADS];  // {x_hi, x_hi}, {y_hi, y_hi}
    __shared__ ulonglong2 s_lo[VT_THREADS];  // {x_lo, x_lo}, {y_lo, y_lo}
    __shared__ unsigned long long s_g2[VT_THREADS];
    const int64_t s_begin = (int64_t)blockIdx.y * seg;
    const int64_t s_end = min(ns, s_begin + seg);
    const int64_t base = (int64_t)blockIdx.x * VT_TILE + threadIdx.x;
    float th[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int64_t i = base + (int64_t)j * VT_THREADS;
        double x = 0.0, y = 0.0;
        if (i < nt) {
            x = xt[i];
            y = yt[i];
        }
        pfd::split_hilo(x, th[j][0], th[j][2]);
        pfd::split_hilo(y, th[j][1], th[j][3]);
    }
    const pfd::f32x2 txh = pfd::pack2(th[0][0], th[1][0]), tyh = pfd::pack2(th[0][1], th[1][1]);
    const pfd::f32x2 txl = pfd::pack2(th[0][2], th[1][2]), tyl = pfd::pack2(th[0][3], th[1][3]);
    const pfd::GaussParams2 gp2 = pfd::make_params2(gp);
    const pfd::f32x2 s22 = pfd::pack2(s2, s2);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};  // (hi, lo) of targets a and b
    for (int64_t t0 = s_begin; t0 < s_end; t0 += VT_THREADS) {
        const int64_t s = t0 + threadIdx.x;
        double x = 0.0, y = 0.0, g = 0.0;  // padding blobs carry g = 0
        if (s < s_end) {
            x = xs[s];
            y = ys[s];
            g = gs[s];
        }
        float xh, xl, yh, yl;
        pfd::split_hilo(x, xh, xl);
        pfd::split_hilo(y, yh, yl);
        const float gf = (float)g;
        __syncthreads();
        s_hi[threadIdx.x] = make_ulonglong2(pfd::pack2(xh, xh), pfd::pack2(yh, yh));
        s_lo[threadIdx.x] = make_ulonglong2(pfd::pack2(xl, xl), pfd::pack2(yl, yl));
        s_g2[threadIdx.x] = pfd::pack2(gf, gf);
        __syncthreads();
        const int nvalid = (int)min((int64_t)VT_THREADS, s_end - t0);
        for (int c0 = 0; c0 < nvalid; c0 += VT_CHUNK) {
            pfd::f32x2 p = 0ull;
#pragma unroll 4
            for (int k = 0; k < VT_CHUNK; ++k) {
                if (CUTOFF)
                    wpair2_cutoff(s_hi[c0 + k], s_lo[c0 + k], s_g2[c0 + k], txh, tyh, txl, tyl,
                                  s22, p);
                else
                    wpair2(s_hi[c0 + k], s_lo[c0 + k], s_g2[c0 + k], txh, tyh, txl, tyl, gp2, p);
            }
            float pa, pb;
            pfd::unpack2(p, pa, pb);
            pfd::comp_add(acc[0], acc[1], pa);
            pfd::comp_add(acc[2], acc[3], pb);
        }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int64_t i = base + (int64_t)j * VT_THREADS;
        if (i >= nt) continue;
        if (part)
            part[(int64_t)blockIdx.y * nt + i] = make_float2(acc[2 * j], acc[2 * j + 1]);
        else
            w[i] = (c1 * ((double)acc[2 * j] + (double)acc[2 * j + 1])) / scale;
    }
}

// w = (c1 * sum) / scale, c1 = 1/pi, scale = ksigmasqr.  grid (target tiles,
// segments); segment y takes the source tiles y, y + gridDim.y, ..., or, where
// every pair is run, the seg sources from y seg on.
__global__ void __launch_bounds__(VT_THREADS, VT_CTAS)
k_vort_gauss(const double *__restrict__ xs, const double *__restrict__ ys,
             const double *__restrict__ gs, int64_t ns, int64_t seg,
             const double *__restrict__ xt, const double *__restrict__ yt, int64_t nt,
             pfd::GaussParams gp, float r2_zero, double c1, double scale, double *__restrict__ w,
             float2 *__restrict__ part) {
    constexpr int NW = VT_THREADS / 32;
    static_assert(NW * VT_CHUNK == VT_THREADS, "warp v loads chunk v of a tile");
    __shared__ ulonglong2 s_hi[VT_THREADS + 1];  // {x_hi, x_hi}, {y_hi, y_hi}; then a blob of g = 0
    __shared__ ulonglong2 s_lo[VT_THREADS + 1];  // {x_lo, x_lo}, {y_lo, y_lo}
    __shared__ unsigned long long s_g2[VT_THREADS + 1];
    __shared__ pfd::TargetBox s_box[NW];
    __shared__ unsigned s_any[NW];  // sources of each chunk within the CTA's reach
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * VT_TILE + wid * 64 + lane;
    float th[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int64_t i = base + 32 * j;
        double x = 0.0, y = 0.0;
        if (i < nt) {
            x = xt[i];
            y = yt[i];
        }
        pfd::split_hilo(x, th[j][0], th[j][2]);
        pfd::split_hilo(y, th[j][1], th[j][3]);
    }
    const pfd::f32x2 txh = pfd::pack2(th[0][0], th[1][0]), tyh = pfd::pack2(th[0][1], th[1][1]);
    const pfd::f32x2 txl = pfd::pack2(th[0][2], th[1][2]), tyl = pfd::pack2(th[0][3], th[1][3]);
    const pfd::GaussParams2 gp2 = pfd::make_params2(gp);
    // the warp's two boxes (32 consecutive targets each: a run of a lattice
    // column that wraps leaves the other box small) and the CTA's one
    pfd::TargetBox bx[2], cta;
#pragma unroll
    for (int j = 0; j < 2; ++j)
        bx[j] = pfd::warp_target_box(base + 32 * j < nt, th[j][0], th[j][1], r2_zero);
    if (lane == 0) {
        cta.x0 = fminf(bx[0].x0, bx[1].x0);
        cta.x1 = fmaxf(bx[0].x1, bx[1].x1);
        cta.y0 = fminf(bx[0].y0, bx[1].y0);
        cta.y1 = fmaxf(bx[0].y1, bx[1].y1);
        cta.reach2 = fmaxf(bx[0].reach2, bx[1].reach2);
        s_box[wid] = cta;
    }
    if (threadIdx.x == 0) {
        s_hi[VT_THREADS] = s_lo[VT_THREADS] = make_ulonglong2(0ull, 0ull);
        s_g2[VT_THREADS] = 0ull;
    }
    __syncthreads();
    cta = s_box[0];
#pragma unroll
    for (int v = 1; v < NW; ++v) {
        cta.x0 = fminf(cta.x0, s_box[v].x0);
        cta.x1 = fmaxf(cta.x1, s_box[v].x1);
        cta.y0 = fminf(cta.y0, s_box[v].y0);
        cta.y1 = fmaxf(cta.y1, s_box[v].y1);
        cta.reach2 = fmaxf(cta.reach2, s_box[v].reach2);
    }
    // targets without spatial order: each warp's box is the CTA's, and the
    // tests would find nothing (their cost: 4% of the pairs')
    const float r = sqrtf(cta.reach2);
    float area = 0.f, some = 0.f;  // over the warps that have targets
    for (int v = 0; v < NW; ++v)
        if (s_box[v].x0 <= s_box[v].x1) {
            area += (s_box[v].x1 - s_box[v].x0 + r) * (s_box[v].y1 - s_box[v].y0 + r);
            some += 1.f;
        }
    const bool tests =
        some == 1.f || area < 0.75f * some * (cta.x1 - cta.x0 + r) * (cta.y1 - cta.y0 + r);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};  // (hi, lo) of targets a and b
    auto fold = [&](pfd::f32x2 p) {
        float pa, pb;
        pfd::unpack2(p, pa, pb);
        pfd::comp_add(acc[0], acc[1], pa);
        pfd::comp_add(acc[2], acc[3], pb);
    };
    auto pair = [&](int k, pfd::f32x2 &p) {
        wpair2(s_hi[k], s_lo[k], s_g2[k], txh, tyh, txl, tyl, gp2, p);
    };
    const int64_t step = (int64_t)gridDim.y * VT_THREADS;
    double x = 0.0, y = 0.0, g = 0.0;  // padding blobs carry g = 0
    auto fetch = [&](int64_t t0) {
        const int64_t s = t0 + threadIdx.x;
        x = y = g = 0.0;
        if (s < ns) {
            x = xs[s];
            y = ys[s];
            g = gs[s];
        }
    };
    int64_t t0 = (int64_t)blockIdx.y * VT_THREADS;
    if (!tests) {  // every pair of one contiguous segment
        const int64_t s_end = min(ns, (int64_t)(blockIdx.y + 1) * seg);
        for (t0 = (int64_t)blockIdx.y * seg; t0 < s_end; t0 += VT_THREADS) {
            fetch(t0);
            if (t0 + threadIdx.x >= s_end) x = y = g = 0.0;
            float xh, xl, yh, yl;
            pfd::split_hilo(x, xh, xl);
            pfd::split_hilo(y, yh, yl);
            const float gf = (float)g;
            __syncthreads();
            s_hi[threadIdx.x] = make_ulonglong2(pfd::pack2(xh, xh), pfd::pack2(yh, yh));
            s_lo[threadIdx.x] = make_ulonglong2(pfd::pack2(xl, xl), pfd::pack2(yl, yl));
            s_g2[threadIdx.x] = pfd::pack2(gf, gf);
            __syncthreads();
            const int nvalid = (int)min((int64_t)VT_THREADS, s_end - t0);
            for (int c0 = 0; c0 < nvalid; c0 += VT_CHUNK) {
                pfd::f32x2 p = 0ull;
#pragma unroll 4
                for (int k = 0; k < VT_CHUNK; ++k) pair(c0 + k, p);
                fold(p);
            }
        }
    } else {
        fetch(t0);
        for (; t0 < ns; t0 += step) {
            float xh, xl, yh, yl;
            pfd::split_hilo(x, xh, xl);
            pfd::split_hilo(y, yh, yl);
            const float gf = (float)g;
            // chunk wid: its sources the CTA needs
            const unsigned any = __ballot_sync(
                0xffffffffu, t0 + threadIdx.x < ns && !pfd::beyond_reach(cta, xh, yh, gf));
            fetch(t0 + step);  // the next tile's loads overlap this one's pairs
            // (also: every warp is done with the previous tile)
            if (!__syncthreads_or(any != 0u)) continue;
            s_hi[threadIdx.x] = make_ulonglong2(pfd::pack2(xh, xh), pfd::pack2(yh, yh));
            s_lo[threadIdx.x] = make_ulonglong2(pfd::pack2(xl, xl), pfd::pack2(yl, yl));
            s_g2[threadIdx.x] = pfd::pack2(gf, gf);
            if (lane == 0) s_any[wid] = any;
            __syncthreads();
            const int nvalid = (int)min((int64_t)VT_THREADS, ns - t0);
            for (int c0 = 0; c0 < nvalid; c0 += VT_CHUNK) {
                unsigned need = s_any[c0 / VT_CHUNK];
                if (need == 0u) continue;
                float sx, sy, sg, dummy;
                pfd::unpack2(s_hi[c0 + lane].x, sx, dummy);
                pfd::unpack2(s_hi[c0 + lane].y, sy, dummy);
                pfd::unpack2(s_g2[c0 + lane], sg, dummy);
                need &= __ballot_sync(0xffffffffu, !(pfd::beyond_reach(bx[0], sx, sy, sg) &&
                                                     pfd::beyond_reach(bx[1], sx, sy, sg)));
                if (need == 0u) continue;
                pfd::f32x2 p = 0ull;
                if (__popc(need) >= VT_DENSE) {
#pragma unroll 4
                    for (int k = 0; k < VT_CHUNK; ++k) pair(c0 + k, p);
                } else {  // four at a time (the blob of g = 0 fills up), in order
                    while (need) {
                        int k[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            k[q] = need ? c0 + __ffs(need) - 1 : VT_THREADS;
                            need &= need - 1;  // 0 stays 0
                        }
#pragma unroll
                        for (int q = 0; q < 4; ++q) pair(k[q], p);
                    }
                }
                fold(p);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int64_t i = base + 32 * j;
        if (i >= nt) continue;
        if (part)
            part[(int64_t)blockIdx.y * nt + i] = make_float2(acc[2 * j], acc[2 * j + 1]);
        else
            w[i] = (c1 * ((double)acc[2 * j] + (double)acc[2 * j + 1])) / scale;
    }
}

// w = (c1 * sum over segments of (hi + lo)) / scale, segments in order.
__global__ void __launch_bounds__(VT_THREADS)
k_vort_reduce(const float2 *__restrict__ part, int64_t nt, int splits, double c1, double scale,
              double *__restrict__ w) {
    const int64_t i = (int64_t)blockIdx.x * VT_THREADS + threadIdx.x;
    if (i >= nt) return;
    double s = 0.0;
    for (int k = 0; k < splits; ++k) {
        const float2 p = part[(int64_t)k * nt + i];
        s += (double)p.x + (double)p.y;
    }
    w[i] = (c1 * s) / scale;
}

}  // namespace

static pf_status vorticity_direct(pf_ctx *ctx, const char *name, int64_t n_src, const double *x,
                                  const double *y, const double *g, int64_t n_tgt,
                                  const double *xt, const double *yt, double param, double *w,
                                  void *stream, bool cutoff) {
    PF_CHECK_ARG(ctx != nullptr, "%s: NULL context", name);
    PF_CHECK_ARG(n_src >= 0 && n_tgt >= 0, "%s: negative size", name);
    PF_CHECK_ARG(param > 0.0 && param < (cutoff ? 1e30 : 1e300),
                 "%s: %s must be positive and finite (got %g)", name,
                 cutoff ? "sigmasqr" : "ksigmasqr", param);
    PF_CHECK_ARG(n_src == 0 || (x && y && g), "%s: NULL blob array", name);
    PF_CHECK_ARG(n_tgt == 0 || (xt && yt && w), "%s: NULL target/output array", name);
    pf::DeviceGuard dg(ctx->device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n_tgt == 0) return PF_OK;
    if (n_src == 0) {
        PF_CUDA_TRY(cudaMemsetAsync(w, 0, sizeof(double) * n_tgt, st));
        return PF_OK;
    }
    const int64_t grid = pf::ceil_div(n_tgt, VT_TILE);
    PF_CHECK_ARG(grid <= INT32_MAX, "%s: too many targets (%lld)", name, (long long)n_tgt);
    const pfd::GaussParams gp = pfd::make_gauss_params(cutoff ? 1.0 : param);
    const double c1 = cutoff ? INV_2PI : INV_PI, scale = cutoff ? 1.0 : param;
    const float s2 = cutoff ? (float)param : 0.f;
    // Source segments: direct_split's (whole waves of resident CTAs).  Tested sets
    // beyond one wave or a few tiles per segment take at least 1.5 waves, as their
    // CTAs' shares of pairs in reach differ (40,401 lattice blobs: 740 CTAs 117 us,
    // 1184 107, 2368 100; more than that costs unordered sets more than it gives).
    // Below, the second wave costs more: 14,000 lattice blobs 57.0 us with, 46.2
    // without, unordered 96.8 and 90.7.
    const bool tested = !cutoff && (double)n_src * (double)n_tgt >= V_TEST_PAIRS;
    const pf::DirectSplit ds = pf::direct_split(n_src, n_tgt);
    int splits = ds.splits;
    int64_t seg = ds.seg;
    const int64_t resident = VT_CTAS * (int64_t)ctx->num_sms;
    if (tested && (grid * splits > resident || seg > 5 * VT_THREADS)) {
        const int64_t tiles = pf::ceil_div(n_src, (int64_t)VT_THREADS);
        const int64_t smax = std::min<int64_t>(tiles, pf::DT_SPLIT_MAX);
        int64_t best = INT64_MAX;
        for (int64_t k = std::min<int64_t>(smax, pf::ceil_div(3 * resident / 2, grid)); k <= smax;
             ++k) {
            const int64_t len =
                pf::ceil_div(pf::ceil_div(n_src, k), (int64_t)VT_CHUNK) * VT_CHUNK;
            const int64_t cost = pf::ceil_div(grid * k, resident) * len;
            if (cost < best) {
                best = cost;
                splits = (int)k;
                seg = len;
            }
        }
    }
    float2 *part = nullptr;
    if (splits > 1) {
        const size_t bytes = sizeof(float2) * (size_t)splits * (size_t)n_tgt;
        PF_TRY(pf::arena_reserve(ctx, bytes + 256));
        part = static_cast<float2 *>(pf::arena_take(ctx, bytes));
        if (!part) {
            pf::set_error("%s: scratch too small", name);
            return PF_ERR_OOM;
        }
    }
    const dim3 grd((unsigned)grid, (unsigned)splits);
    const float r2z = (float)(V_FAR / 1.4426950408889634 * param);
    if (tested)
        k_vort_gauss<<<grd, VT_THREADS, 0, st>>>(x, y, g, n_src, seg, xt, yt, n_tgt, gp, r2z, c1,
                                                 scale, w, part);
    else if (cutoff)
        k_vort_pairs<true><<<grd, VT_THREADS, 0, st>>>(x, y, g, n_src, seg, xt, yt, n_tgt, gp, c1,
                                                       scale, s2, w, part);
    else
        k_vort_pairs<false><<<grd, VT_THREADS, 0, st>>>(x, y, g, n_src, seg, xt, yt, n_tgt, gp, c1,
                                                        scale, s2, w, part);
    PF_TRY(pf::launch_status("k_vort_gauss"));
    if (!part) return PF_OK;
    k_vort_reduce<<<(unsigned)pf::ceil_div(n_tgt, VT_THREADS), VT_THREADS, 0, st>>>(
        part, n_tgt, splits, c1, scale, w);
    return pf::launch_status("k_vort_reduce");
}

extern "C" pf_status pf_vorticity_direct(pf_ctx *ctx, int64_t n_src, const double *x,
                                         const double *y, const double *g, int64_t n_tgt,
                                         const double *xt, const double *yt, double ksigmasqr,
                                         double *w, void *stream) {
    PF_RANGE("pf_vorticity_direct");
    pf::clear_error();
    return vorticity_direct(ctx, "pf_vorticity_direct", n_src, x, y, g, n_tgt, xt, yt, ksigmasqr,
                            w, stream, false);
}

extern "C" pf_status pf_vorticity_direct_cutoff(pf_ctx *ctx, int64_t n_src, const double *x,
                                                const double *y, const double *g, int64_t n_tgt,
                                                const double *xt, const double *yt,
                                                double sigmasqr, double *w, void *stream) {
    PF_RANGE("pf_vorticity_direct_cutoff");
    pf::clear_error();
    return vorticity_direct(ctx, "pf_vorticity_direct_cutoff", n_src, x, y, g, n_tgt, xt, yt,
                            sigmasqr, w, stream, true);
}
