// fmm.cu -- 2D fast multipole method for Gaussian vortex blobs on B200.
//
// Tree: uniform quadtree over the bounding square of sources and targets,
// every level a dense 2^l x 2^l grid addressed by Morton index (box (l, m) at
// global slot off[l] + m, off[l] = (4^l - 1)/3).  Particles are counting-
// sorted by leaf Morton key (ties in input order, so every sum has a fixed
// order) -- this replaces the reference's median-split partition
// (src/cpp/blobs/c++/fmm2d_py_cpu_gpu/fmmsort.cpp:441-790).
//
// Expansions (FP64, complex, scaled by the box width w so that all
// coefficients are O(sum |g|)):
//   multipole  M(z) = sum_j g_j / (z - z_j) = sum_k a_k w^k / (z - c)^(k+1),
//              a_k = sum_j g_j ((z_j - c)/w)^k                       (P2M)
//   local      L(z) = (1/w) sum_n lam_n ((z - c)/w)^n
//   M2M  a'_k  = sum_{m<=k} C(k,m) tau^(k-m) 2^-m a_m,  tau = (c_child - c_par)/w_par
//   M2L  lam_n += sum_k (-1)^(k+1) C(n+k,k) rho^(n+k+1) a_k,  rho = 1/(i + i j)
//              for a far box at integer offset (i, j): the operator depends
//              only on the offset, so rho^m is tabulated per offset
//   L2L  lam'_n = (1/2) sum_{m>=n} C(m,n) tau^(m-n) 2^-n lam_m
//   L2P  W = L(z);  u = Im W / 2pi,  v = Re W / 2pi
// (reference counterparts: mpexp_init fmm.cpp:1452-1509, shift_m2m
// fmmshift.cpp:80-236, shift_m2ps fmmshift.cpp:237-621, shift_p2p
// fmmshift.cpp:622-767, mpexp_eval fmm.cpp:1875-1931).
// M2M, M2L and L2L run on the FP64 tensor cores (mma.sync m8n8k4 .f64):
// their operators are fixed matrices (per child position, or the binomial
// matrix between the scalings by rho), applied to four boxes per warp task.
//
// Near field: the Gaussian kernel itself, FP32 with hi/lo coordinates and
// compensated accumulation (gauss_pair.cuh), for every target of a P2P block
// (2^kb x 2^kb leaves) against the block's source leaves; those leaves are
// sorted by Morton index and merged into runs of consecutive leaves, which
// are contiguous in the sorted particle arrays, and streamed through shared
// memory in full tiles.  The interaction lists come from fmm_plan.cu.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "fmm_api.cuh"
#include "fmm_plan.cuh"
#include "gauss_pair.cuh"
#include "p2p.cuh"
#include "scan.cuh"
#include "segsort.cuh"

#include "direct_api.cuh"

namespace {

constexpr double THETA = 0.5;
constexpr double INV_2PI = 0.15915494309189535;
constexpr int MAX_LEVEL = pf::fmmx::MAX_LEVEL;
constexpr int P2P_SETUP_THREADS = 128;
constexpr int P2P_QMAX = 1024;   // source leaves per P2P block
constexpr unsigned INVALID_KEY = 0xFFFFFFFFu;
// leaves of more particles than this are put in index order by the segment
// sort; smaller ones by k_gather_sorted itself, c comparisons per particle.  A
// layer around a body fills its leaves to 40-110 particles (the leaf level
// comes from the blob count, the box is mostly empty); 1.8e6 blobs in an
// annulus, gather + segment sort: 286 us at 64, 40 us at 256.
constexpr int LEAF_SMALL = 256;

// ---------------------------------------------------------------------------
// Morton helpers (x in even bits, y in odd bits)
__host__ __device__ __forceinline__ uint32_t part1by1(uint32_t v) {
    v &= 0x0000ffffu;
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}
__host__ __device__ __forceinline__ uint32_t compact1by1(uint32_t v) {
    v &= 0x55555555u;
    v = (v | (v >> 1)) & 0x33333333u;
    v = (v | (v >> 2)) & 0x0f0f0f0fu;
    v = (v | (v >> 4)) & 0x00ff00ffu;
    v = (v | (v >> 8)) & 0x0000ffffu;
    return v;
}
__host__ __device__ __forceinline__ uint32_t morton2(uint32_t x, uint32_t y) {
    return part1by1(x) | (part1by1(y) << 1);
}

// Morton code of (x + dx, y + dy) from the code m of (x, y) and the dilated
// offset d = morton2(dx mod 2^16, dy mod 2^16): each coordinate's bits are
// added with the other coordinate's bit positions filled with ones, so the
// carries run through them ("dilated integer" addition).  Exact whenever the
// shifted coordinates lie in [0, 2^16).
__device__ __forceinline__ uint32_t morton_add(uint32_t m, uint32_t d) {
    const uint32_t xm = 0x55555555u, ym = 0xaaaaaaaau;
    return (((m | ym) + (d & xm)) & xm) | (((m | xm) + (d & ym)) & ym);
}

// leaf coordinate of a position: floor((x - x0) / w) clamped to [0, 2^L)
__device__ __forceinline__ uint32_t leaf_coord(double x, double x0, double w, int L) {
    const double q = floor(__ddiv_rn(__dsub_rn(x, x0), w));
    const double hi = (double)((1u << L) - 1u);
    return (uint32_t)fmin(fmax(q, 0.0), hi);
}

// ---------------------------------------------------------------------------
// bounding box with order-preserving integer images of doubles
__device__ __forceinline__ unsigned long long ord_d(double v) {
    unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__host__ inline double unord_d(unsigned long long u) {
    u = (u >> 63) ? (u & 0x7fffffffffffffffull) : ~u;
    double d;
    memcpy(&d, &u, 8);
    return d;
}

struct BBox {
    unsigned long long mnx, mxx, mny, mxy;
    unsigned long long bad;
};

__device__ __forceinline__ void bbox_merge(BBox &a, const BBox &b) {
    a.mnx = min(a.mnx, b.mnx);
    a.mxx = max(a.mxx, b.mxx);
    a.mny = min(a.mny, b.mny);
    a.mxy = max(a.mxy, b.mxy);
    a.bad |= b.bad;
}

// the block's box, valid in thread 0
__device__ __forceinline__ void bbox_block(BBox &v, BBox *s_v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        BBox w;
        w.mnx = __shfl_xor_sync(0xffffffffu, v.mnx, o);
        w.mxx = __shfl_xor_sync(0xffffffffu, v.mxx, o);
        w.mny = __shfl_xor_sync(0xffffffffu, v.mny, o);
        w.mxy = __shfl_xor_sync(0xffffffffu, v.mxy, o);
        w.bad = 0;
        bbox_merge(v, w);
    }
    v.bad = __reduce_or_sync(0xffffffffu, (unsigned)v.bad);
    if ((threadIdx.x & 31) == 0) s_v[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < 8; ++w) bbox_merge(v, s_v[w]);
}

// Bounding box of n sources and nt targets in one launch: each CTA leaves its
// box in part[], the last one to finish (ticket, which wraps back to zero)
// merges them and writes the result to the host's pinned memory, where the
// caller reads it after the stream's synchronisation.  Latency-bound: a
// preparing launch, a second launch for separate targets and the copy cost
// 2-5 us each; with the other launches merged, see k_place, 1,000 blobs
// 83 -> 65 us, 30,000 146 -> 125 a call.
__global__ void __launch_bounds__(256)
k_bbox(const double *__restrict__ x, const double *__restrict__ y, int64_t n,
       const double *__restrict__ xt, const double *__restrict__ yt, int64_t nt, BBox *part,
       unsigned *ticket, BBox *out) {
    __shared__ BBox s_v[8];
    __shared__ bool s_last;
    BBox v{~0ull, 0, ~0ull, 0, 0};
    // four independent loads of x and y per thread in flight
    const int64_t stride = (int64_t)gridDim.x * 256, m = n + nt;
    for (int64_t i0 = (int64_t)blockIdx.x * 256 + threadIdx.x; i0 < m; i0 += 4 * stride) {
        double a[4], c[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t i = i0 + u * stride;
            a[u] = i < n ? x[i] : i < m ? xt[i - n] : 0.0;
            c[u] = i < n ? y[i] : i < m ? yt[i - n] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (i0 + u * stride >= m) continue;
            if (!isfinite(a[u]) || !isfinite(c[u])) {
                v.bad = 1;
                continue;
            }
            const unsigned long long oa = ord_d(a[u]), oc = ord_d(c[u]);
            bbox_merge(v, BBox{oa, oa, oc, oc, 0});
        }
    }
    bbox_block(v, s_v);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = v;
        __threadfence();
        s_last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    v = BBox{~0ull, 0, ~0ull, 0, 0};
    for (unsigned k = threadIdx.x; k < gridDim.x; k += 256) {
        const unsigned long long *p = reinterpret_cast<const unsigned long long *>(part + k);
        bbox_merge(v, BBox{__ldcg(p), __ldcg(p + 1), __ldcg(p + 2), __ldcg(p + 3), __ldcg(p + 4)});
    }
    bbox_block(v, s_v);
    if (threadIdx.x == 0) {
        *out = v;
        __threadfence_system();
    }
}

// ---------------------------------------------------------------------------
// counting sort by leaf key
__global__ void __launch_bounds__(256)
k_leaf_keys(const double *__restrict__ x, const double *__restrict__ y, int64_t n, double x0,
            double y0, double wl, int L, uint32_t *__restrict__ key, int32_t *__restrict__ rank,
            int32_t *__restrict__ cnt, int32_t *__restrict__ big_n,
            unsigned long long *__restrict__ ctr) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    // the first launch of a call clears its counters: memsets were launches
    if (i == 0 && big_n) *big_n = 0;
    if (i == 0 && ctr)
        for (int k = 0; k < pf::fmmx::FMM_COUNTERS; ++k) ctr[k] = 0;
    if (i >= n) return;
    const uint32_t k = morton2(leaf_coord(x[i], x0, wl, L), leaf_coord(y[i], y0, wl, L));
    key[i] = k;
    if (rank) rank[i] = atomicAdd(&cnt[k], 1);
}

__host__ __device__ __forceinline__ int64_t level_off(int l) {
    return ((((int64_t)1) << (2 * l)) - 1) / 3;
}

// Sorted copies of the points in leaf order, each leaf's particles by input
// index (the counting sort's atomic ranks are not reproducible; this fixes
// every later sum's order).  Thread j takes the particle i = perm[j] that the
// counting sort placed in its leaf's range [s0, s0 + c); its final position
// is s0 + (number of the leaf's particles with a smaller index), found by
// reading the leaf's c entries of perm (leaves above LEAF_SMALL particles are
// already in index order: seg_sort_listed).  Writes the final permutation to
// perm_out and, at that position, FP64 x, y (g), the hi/lo float4 and float g
// of the near field and the leaf key.
__global__ void __launch_bounds__(256)
k_gather_sorted(int64_t n, const int32_t *__restrict__ perm, const uint32_t *__restrict__ key,
                const int32_t *__restrict__ start, const int32_t *__restrict__ cnt,
                const double *__restrict__ x, const double *__restrict__ y,
                const double *__restrict__ g, int32_t *__restrict__ perm_out,
                double *__restrict__ sx, double *__restrict__ sy, double *__restrict__ sg,
                float4 *__restrict__ hl, float *__restrict__ g32, uint32_t *__restrict__ skey) {
    const int64_t j = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (j >= n) return;
    const int32_t i = perm[j];
    if (!PF_IDX_OK(i, n, 202)) return;
    const uint32_t m = key[i];
    const double a = x[i], b = y[i];
    const double gi = g ? g[i] : 0.0;
    const int s0 = start[m], c = cnt[m];
    int64_t d = j;
    if (c <= LEAF_SMALL && PF_IDX_OK((int64_t)s0 + c - 1, n, 206)) {
        int r = 0;
        for (int q = 0; q < c; ++q) r += perm[s0 + q] < i;
        d = (int64_t)s0 + r;
    }
    perm_out[d] = i;
    if (skey) skey[d] = m;  // leaf key in sorted order (targets)
    sx[d] = a;
    sy[d] = b;
    float4 h;
    pfd::split_hilo(a, h.x, h.z);
    pfd::split_hilo(b, h.y, h.w);
    hl[d] = h;
    if (g) {
        sg[d] = gi;
        g32[d] = (float)gi;
    }
}

// Box counts of nlev (<= 6) coarser levels from level lc: CTA b owns the
// 4^nlev level-lc boxes below box b of level lc - nlev (one contiguous Morton
// range) and sums them up level by level in shared memory (integer sums:
// exact, any order).
constexpr int COUNT_LEVELS = 6;
__device__ __forceinline__ void count_up_block(int lc, int nlev, int64_t b,
                                               int32_t *__restrict__ cnt_all) {
    __shared__ int32_t s_c[2][1024];
    const int nch = 1 << (2 * nlev);
    const int32_t *src = cnt_all + level_off(lc) + b * nch;
    for (int j = 1; j <= nlev; ++j) {
        const int np = nch >> (2 * j);
        int32_t *dst = s_c[j & 1];
        int32_t *all = cnt_all + level_off(lc - j) + b * np;
        for (int p = threadIdx.x; p < np; p += 256) {
            const int32_t v = src[4 * p] + src[4 * p + 1] + src[4 * p + 2] + src[4 * p + 3];
            dst[p] = v;
            all[p] = v;
        }
        __syncthreads();
        src = dst;
    }
}

__global__ void __launch_bounds__(256) k_count_up(int lc, int nlev, int32_t *__restrict__ cnt_all) {
    count_up_block(lc, nlev, blockIdx.x, cnt_all);
}

// ---------------------------------------------------------------------------
// complex helpers
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {  // a*b + c
    return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}

// P2M: one thread per leaf
template <int NP>
__global__ void __launch_bounds__(128)
k_p2m(int L, double x0, double y0, double wl, const int32_t *__restrict__ start,
      const int32_t *__restrict__ cnt, const double *__restrict__ sx,
      const double *__restrict__ sy, const double *__restrict__ sg, double2 *__restrict__ M) {
    // four consecutive lanes per leaf, lane q taking the leaf's particles
    // q, q + 4, ...; the four partial expansions are added in a fixed tree order
    const int64_t nleaf = (int64_t)1 << (2 * L);
    const int64_t t = (int64_t)blockIdx.x * 128 + threadIdx.x;
    const int64_t m = t >> 2;
    const int q = (int)(t & 3);
    const bool live = m < nleaf;
    const int c = live ? cnt[m] : 0;
    const uint32_t ix = compact1by1((uint32_t)m), iy = compact1by1((uint32_t)m >> 1);
    const double cx = x0 + ((double)ix + 0.5) * wl, cy = y0 + ((double)iy + 0.5) * wl;
    const double iw = 1.0 / wl;
    double2 a[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) a[k] = make_double2(0.0, 0.0);
    const int s0 = live ? start[m] : 0;
    for (int j = q; j < c; j += 4) {
        const double2 z = make_double2((sx[s0 + j] - cx) * iw, (sy[s0 + j] - cy) * iw);
        double2 zk = make_double2(sg[s0 + j], 0.0);
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            a[k].x += zk.x;
            a[k].y += zk.y;
            zk = cmul(zk, z);
        }
    }
#pragma unroll
    for (int k = 0; k < NP; ++k) {
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            a[k].x += __shfl_xor_sync(0xffffffffu, a[k].x, o);
            a[k].y += __shfl_xor_sync(0xffffffffu, a[k].y, o);
        }
    }
    if (!live || c == 0) return;
    const int64_t base = ((((int64_t)1 << (2 * L)) - 1) / 3 + m) * NP;
#pragma unroll
    for (int k = 0; k < NP; ++k)
        if ((k & 3) == q) M[base + k] = a[k];
}


// One FP64 tensor-core product d = a b + d of an 8 x 4 by 4 x 8 tile
// (mma.sync m8n8k4 .f64; tcgen05 has no FP64 kind).  Fragments: a = A[lane/4]
// [lane%4], b = B[lane%4][lane/4], (d0, d1) = D[lane/4][2 (lane%4) + 0, 1].
__device__ __forceinline__ void mma_f64(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// M2M and L2L on the FP64 tensor cores.  The translation of a box's
// expansion to (M2M) or from (L2L) child position c is a fixed complex NP x NP
// matrix T_c (lower triangular for M2M, upper for L2L).  A warp task applies
// it to four boxes at once: the B operand holds their coefficients (column
// 2j real, 2j + 1 imaginary parts of box j), the A operand the real and the
// imaginary part of T_c, from fragment tables built with the plan
// (frag[c][part][mt][ks][lane] = part of T_c[8 mt + lane/4][4 ks + lane%4]);
// tiles of zeros are skipped.  With U = Re T B and V = Im T B, lane (box
// lane%4, row n = lane/4 + 8 mt) holds Re = U_re - V_im and Im = U_im + V_re.
template <int NP>
struct TcShape {
    static constexpr int MT = (NP + 7) / 8, KS = (NP + 3) / 4;
};

// TRI = 1: T[row][col] = 0 for col > row (M2M); TRI = -1: for col < row (L2L)
template <int TRI>
__device__ __forceinline__ constexpr bool tc_tile_live(int mt, int ks) {
    return TRI > 0 ? 4 * ks <= 8 * mt + 7 : 4 * ks + 3 >= 8 * mt;
}

// d[mt] = T_c b for the lane's (box lane%4, rows lane/4 + 8 mt); b[s] = the
// lane's B element of k block s (row 4 s + lane%4, column lane/4).
template <int NP, int TRI>
__device__ __forceinline__ void tc_apply(const double *__restrict__ fr,
                                         const double (&b)[TcShape<NP>::KS],
                                         double2 (&d)[TcShape<NP>::MT]) {
    constexpr int MT = TcShape<NP>::MT, KS = TcShape<NP>::KS;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        double u0 = 0.0, u1 = 0.0, v0 = 0.0, v1 = 0.0;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            if (!tc_tile_live<TRI>(mt, ks)) continue;
            mma_f64(u0, u1, __ldg(fr + ((0 * MT + mt) * KS + ks) * 32 + lane), b[ks]);
            mma_f64(v0, v1, __ldg(fr + ((1 * MT + mt) * KS + ks) * 32 + lane), b[ks]);
        }
        d[mt] = make_double2(u0 - v1, u1 + v0);
    }
}

// The lane's B elements of four boxes' coefficients: coef(j, m) is
// coefficient m of box j (zero for an empty box).
template <int NP, class Coef>
__device__ __forceinline__ void tc_load_b(Coef coef, double (&b)[TcShape<NP>::KS]) {
    const int lane = threadIdx.x & 31;
    const int j = lane >> 3, part = (lane >> 2) & 1, kq = lane & 3;
#pragma unroll
    for (int ks = 0; ks < TcShape<NP>::KS; ++ks) {
        const int m = 4 * ks + kq;
        const double2 v = m < NP ? coef(j, m) : make_double2(0.0, 0.0);
        b[ks] = part ? v.y : v.x;
    }
}

constexpr int TC_THREADS = 128;  // four warp tasks per CTA

// M2M into parent level l for four consecutive parents per warp task:
// out_j[k] = sum_c T_c (children 4 P_j + c, empty ones as zeros), written for
// the non-empty parents.  With two_level, the same warp then forms the
// grandparent (level l - 1, box task) from those four parents.
template <int NP>
__global__ void __launch_bounds__(TC_THREADS)
k_m2m_tc(int l, bool two_level, const int32_t *__restrict__ scnt, double2 *__restrict__ M,
         const double *__restrict__ frag /* [4][2][MT][KS][32] */) {
    constexpr int MT = TcShape<NP>::MT;
    constexpr int FR = 2 * MT * TcShape<NP>::KS * 32;  // doubles per child position
    __shared__ double2 s_par[TC_THREADS / 32][4][NP];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t task = (int64_t)blockIdx.x * (TC_THREADS / 32) + wid;
    if (task >= ((int64_t)1 << (2 * l)) / 4) return;  // the whole warp
    const int64_t p0 = level_off(l) + 4 * task;        // parents p0 .. p0 + 3
    const int64_t c0 = level_off(l + 1) + 16 * task;   // their children
    double2 out[MT];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) out[mt] = make_double2(0.0, 0.0);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        double b[TcShape<NP>::KS];
        tc_load_b<NP>(
            [&](int j, int m) {
                const int64_t ch = c0 + 4 * j + c;
                const double2 v = M[ch * NP + m];  // loaded with the count
                return scnt[ch] != 0 ? v : make_double2(0.0, 0.0);
            },
            b);
        double2 d[MT];
        tc_apply<NP, 1>(frag + c * FR, b, d);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
            out[mt] = make_double2(out[mt].x + d[mt].x, out[mt].y + d[mt].y);
    }
    const int jd = lane & 3, nr = lane >> 2;
    const bool live = scnt[p0 + jd] != 0;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        const int n = 8 * mt + nr;
        if (n >= NP) continue;
        if (live) M[(p0 + jd) * NP + n] = out[mt];
        s_par[wid][jd][n] = live ? out[mt] : make_double2(0.0, 0.0);
    }
    if (!two_level) return;
    __syncwarp();
    // grandparent (task) of level l - 1 from the four parents: column 0 only
    double2 g[MT];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) g[mt] = make_double2(0.0, 0.0);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        double b[TcShape<NP>::KS];
        tc_load_b<NP>([&](int j, int m) { return j == 0 ? s_par[wid][c][m] : make_double2(0.0, 0.0); },
                      b);
        double2 d[MT];
        tc_apply<NP, 1>(frag + c * FR, b, d);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) g[mt] = make_double2(g[mt].x + d[mt].x, g[mt].y + d[mt].y);
    }
    const int64_t gp = level_off(l - 1) + task;
    if (jd == 0 && scnt[gp] != 0)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            const int n = 8 * mt + nr;
            if (n < NP) M[gp * NP + n] = g[mt];
        }
}

// L2L from parent level l - 1 into child level l for four consecutive parents
// per warp task: child 4 P_j + c += T_c L_{P_j}, for the non-empty children.
// With two_level the same warp first forms the four parents themselves from
// their parent (level l - 2, box task), then their children.
template <int NP>
__global__ void __launch_bounds__(TC_THREADS)
k_l2l_tc(int l, bool two_level, const int32_t *__restrict__ tcnt, double2 *__restrict__ Lc,
         const double *__restrict__ frag /* [4][2][MT][KS][32] */) {
    constexpr int MT = TcShape<NP>::MT;
    constexpr int FR = 2 * MT * TcShape<NP>::KS * 32;
    __shared__ double2 s_par[TC_THREADS / 32][4][NP];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int jd = lane & 3, nr = lane >> 2;
    const int64_t task = (int64_t)blockIdx.x * (TC_THREADS / 32) + wid;
    if (task >= ((int64_t)1 << (2 * l)) / 16) return;  // the whole warp
    const int64_t p0 = level_off(l - 1) + 4 * task;     // parents p0 .. p0 + 3
    const int64_t c0 = level_off(l) + 16 * task;        // their children
    if (two_level) {
        // the parents (children of box `task` of level l - 2): column 0 only
        const int64_t gp = level_off(l - 2) + task;
        const bool glive = tcnt[gp] != 0;
        double b[TcShape<NP>::KS];
        tc_load_b<NP>([&](int j, int m) {
            return (j == 0 && glive) ? Lc[gp * NP + m] : make_double2(0.0, 0.0);
        }, b);
        // lanes of column 0 (jd == 0) take parent c's rows: its own local
        // expansion is loaded before the products
        double2 old[4][MT];
        bool plive[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            plive[c] = tcnt[p0 + c] != 0;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                const int n = 8 * mt + nr;
                old[c][mt] = (jd == 0 && n < NP) ? Lc[(p0 + c) * NP + n] : make_double2(0.0, 0.0);
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            double2 d[MT];
            tc_apply<NP, -1>(frag + c * FR, b, d);
            if (jd == 0)
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    const int n = 8 * mt + nr;
                    if (n >= NP) continue;
                    double2 v = make_double2(0.0, 0.0);
                    if (plive[c]) {
                        v = make_double2(old[c][mt].x + d[mt].x, old[c][mt].y + d[mt].y);
                        Lc[(p0 + c) * NP + n] = v;
                    }
                    s_par[wid][c][n] = v;  // broadcast to the warp by shared memory
                }
        }
        __syncwarp();
    } else {
        for (int t = lane; t < 4 * NP; t += 32) {
            const int j = t / NP, n = t - j * NP;
            s_par[wid][j][n] = tcnt[p0 + j] != 0 ? Lc[(p0 + j) * NP + n] : make_double2(0.0, 0.0);
        }
        __syncwarp();
    }
    // the children's own local expansions, loaded before the products
    double2 old[4][MT];
    bool clive[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int64_t ch = c0 + 4 * jd + c;
        clive[c] = tcnt[ch] != 0;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            const int n = 8 * mt + nr;
            old[c][mt] = n < NP ? Lc[ch * NP + n] : make_double2(0.0, 0.0);
        }
    }
    double b[TcShape<NP>::KS];
    tc_load_b<NP>([&](int j, int m) { return s_par[wid][j][m]; }, b);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        double2 d[MT];
        tc_apply<NP, -1>(frag + c * FR, b, d);
        if (!clive[c]) continue;
        const int64_t ch = c0 + 4 * jd + c;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            const int n = 8 * mt + nr;
            if (n < NP)
                Lc[ch * NP + n] = make_double2(old[c][mt].x + d[mt].x, old[c][mt].y + d[mt].y);
        }
    }
}

constexpr int M2L_THREADS = 128;  // 4 warps, four target boxes each
constexpr int64_t M2L_AHEAD_QUADS = 1365;  // box quads up to which k_m2l loads ahead (6 levels)

// M2L for all levels 2..L on the FP64 tensor cores.  One translation adds
//   L_n += r^(n+1) sum_k C(n+k, k) c_k,   c_k = (-1)^(k+1) M_k r^k
// (r: the operator's powers), so the binomial matrix is the same for every
// translation.  A warp holds it as the A operand (rows n, columns k, in 8 x 4
// fragments) and takes four target boxes of one level with the same far list
// (same position class: Morton indices r0 + q stride) as the 8 columns of B,
// the real and imaginary parts of their c.  Per far-list entry: B from the
// four sources' multipoles, KS mma per 8 rows, then lane (n = lane/4 + 8 mt,
// box lane%4) scales its (re, im) pair by r^(n+1) into its coefficient.
//
// AHEAD (trees whose quads leave the device half empty): the next entry's
// counts, multipoles and powers are loaded before the current entry's products,
// so that a warp's chain is products, not load latency; the sums are the same.
// One warp per CTA there.  M2L time without / with it: 3,001 blobs (85 quads) 34 /
// 23 us, 60,007 (1365) 41 / 29, 150,000 (5461 quads) 58 / 66, 2^20 (21845) 135 /
// 160: up to M2L_AHEAD_QUADS, and where no other sets run beside this one.
template <int NP, bool AHEAD>
__global__ void __launch_bounds__(M2L_THREADS)
k_m2l(int L, int Bp, int64_t nquad, const int32_t *__restrict__ scnt,
      const int32_t *__restrict__ tcnt, const double2 *__restrict__ M, double2 *__restrict__ Lc,
      const int4 *__restrict__ far, const int32_t *__restrict__ far_ptr, int maxpos,
      const double2 *__restrict__ pw /* [nop][NP+1] */, const double *__restrict__ binom,
      unsigned long long *__restrict__ ntrans) {
    constexpr int MT = (NP + 7) / 8, KS = (NP + 3) / 4;
    const int lane = threadIdx.x & 31;
    constexpr int NWARP = AHEAD ? 1 : M2L_THREADS / 32;
    const int64_t u = (int64_t)blockIdx.x * NWARP + (threadIdx.x >> 5);
    if (u >= nquad) return;  // the whole warp
    int l = 2;
    int64_t j = u;
    while (l < L && j >= ((int64_t)1 << (2 * l)) / 4) {
        j -= ((int64_t)1 << (2 * l)) / 4;
        ++l;
    }
    const int64_t stride = (l == L) ? (int64_t)Bp * Bp : 4;
    const int64_t r0 = (j / stride) * 4 * stride + (j % stride);
    // B column lane/4: box tb, part (0 real, 1 imaginary); B row k = 4 s + kq
    const int tb = lane >> 3, part = (lane >> 2) & 1, kq = lane & 3;
    // D: box td, rows n = nr + 8 mt
    const int td = lane & 3, nr = lane >> 2;
    const uint32_t mb = (uint32_t)(r0 + tb * stride);
    const int64_t lo = level_off(l);
    const bool liveb = tcnt[lo + mb] != 0;
    if (!__any_sync(0xffffffffu, liveb)) return;
    const bool lived = __shfl_sync(0xffffffffu, liveb, 8 * td);
    double af[MT][KS];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int s = 0; s < KS; ++s) {
            const int n = 8 * mt + nr, k = 4 * s + kq;
            af[mt][s] = (n < NP && k < NP) ? binom[k * NP + n] : 0.0;
        }
    const int ixb = (int)compact1by1(mb), iyb = (int)compact1by1(mb >> 1);
    // the same for the four boxes
    const int pos = (l == L) ? ((ixb % Bp) + Bp * (iyb % Bp)) : ((ixb & 1) | ((iyb & 1) << 1));
    const int side = 1 << l;
    const int e0 = far_ptr[l * maxpos + pos];
    const int len = far_ptr[l * maxpos + pos + 1] - e0;
    const double sgn = (kq & 1) ? 1.0 : -1.0;  // (-1)^(k+1)
    double2 acc[MT];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) acc[mt] = make_double2(0.0, 0.0);
    unsigned nt = 0;
    // one far-list entry as the lane needs it
    struct Entry {
        double2 mv[KS], rv[KS], rs[MT];  // multipoles, powers, the scaling's powers
        bool use;
    };
    auto fetch = [&](const int4 &f, Entry &t) {
        const int sx = ixb + f.x, sy = iyb + f.y;
        const bool inr = liveb && sx >= 0 && sy >= 0 && sx < side && sy < side;
        const int64_t sg = inr ? lo + morton_add(mb, (uint32_t)f.w) : 0;
        // the source's count and multipole are loaded together (the box is
        // in range either way); an empty source is then skipped
        const int cs = inr ? scnt[sg] : 0;
        const double2 *rp = pw + (int64_t)f.z * (NP + 1);
#pragma unroll
        for (int s = 0; s < KS; ++s) {
            const int k = 4 * s + kq;
            t.mv[s] = (inr && k < NP) ? M[sg * NP + k] : make_double2(0.0, 0.0);
            t.rv[s] = (k < NP) ? rp[k] : make_double2(0.0, 0.0);
        }
        if (AHEAD)
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                const int n = 8 * mt + nr;
                t.rs[mt] = n < NP ? rp[n + 1] : make_double2(0.0, 0.0);
            }
        t.use = inr && cs != 0;
    };
    auto add = [&](const int4 &f, const Entry &t) {
        if (!__any_sync(0xffffffffu, t.use)) return;
        const bool used = __shfl_sync(0xffffffffu, t.use, 8 * td);
        nt += ((lane & 7) == 0 && t.use) ? 1u : 0u;
        const double2 *rp = pw + (int64_t)f.z * (NP + 1);
        double b[KS];
#pragma unroll
        for (int s = 0; s < KS; ++s) {
            const double2 m = t.mv[s], r = t.rv[s];
            const double v = part ? fma(m.x, r.y, m.y * r.x) : fma(m.x, r.x, -(m.y * r.y));
            b[s] = t.use ? sgn * v : 0.0;
        }
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            double d0 = 0.0, d1 = 0.0;
#pragma unroll
            for (int s = 0; s < KS; ++s) mma_f64(d0, d1, af[mt][s], b[s]);
            const int n = 8 * mt + nr;
            if (used && n < NP)
                acc[mt] = cfma(AHEAD ? t.rs[mt] : rp[n + 1], make_double2(d0, d1), acc[mt]);
        }
    };
    if constexpr (AHEAD) {
        if (len > 0) {
            int4 f0 = far[e0], f1 = far[e0 + min(1, len - 1)];
            Entry t0;
            fetch(f0, t0);
#pragma unroll 2
            for (int e = 0; e < len; ++e) {
                const int4 f2 = far[e0 + min(e + 2, len - 1)];
                Entry t1;
                fetch(f1, t1);  // past the end: the last entry again, not added
                add(f0, t0);
                t0 = t1;
                f0 = f1;
                f1 = f2;
            }
        }
    } else {
        for (int e = 0; e < len; ++e) {
            const int4 f = far[e0 + e];
            Entry t;
            fetch(f, t);
            add(f, t);
        }
    }
    if (lived) {
        const int64_t bgd = lo + r0 + td * stride;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            const int n = 8 * mt + nr;
            if (n < NP) Lc[bgd * NP + n] = acc[mt];
        }
    }
    nt = __reduce_add_sync(0xffffffffu, nt);
    if (lane == 0 && nt) atomicAdd(ntrans, (unsigned long long)nt);
}

// ---------------------------------------------------------------------------
// P2P run lists (once per plan; geometry only).  For P2P block b, the source
// leaves b's origin + q are sorted by Morton index and merged into runs of
// consecutive indices; consecutive leaves are contiguous in the sorted
// particle arrays, so a run is one particle range.  Pass 1 (runs == nullptr)
// writes the run count of each block, pass 2 the runs (first, last leaf).
__global__ void __launch_bounds__(P2P_SETUP_THREADS)
k_p2p_runs(int L, int kb, const int2 *__restrict__ q, int nq, int nqp,
           int32_t *__restrict__ nruns_or_off, int2 *__restrict__ runs) {
    __shared__ uint32_t s_key[P2P_QMAX];
    __shared__ int s_n;
    const uint32_t b = blockIdx.x;
    const int ox = (int)(compact1by1(b) << kb), oy = (int)(compact1by1(b >> 1) << kb);
    const int side = 1 << L;
    for (int t = threadIdx.x; t < nqp; t += P2P_SETUP_THREADS) {
        uint32_t k = INVALID_KEY;
        if (t < nq) {
            const int lx = ox + q[t].x, ly = oy + q[t].y;
            if (lx >= 0 && ly >= 0 && lx < side && ly < side) k = morton2(lx, ly);
        }
        s_key[t] = k;
    }
    __syncthreads();
    for (int kk = 2; kk <= nqp; kk <<= 1) {
        for (int j = kk >> 1; j > 0; j >>= 1) {
            for (int t = threadIdx.x; t < nqp; t += P2P_SETUP_THREADS) {
                const int p = t ^ j;
                if (p > t) {
                    const uint32_t a = s_key[t], c = s_key[p];
                    const bool up = ((t & kk) == 0);
                    if ((a > c) == up) {
                        s_key[t] = c;
                        s_key[p] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int nr = 0;
        const int base_out = runs ? nruns_or_off[b] : 0;
        for (int base = 0; base < nqp; base += 32) {
            const int t = base + lane;
            const uint32_t k = (t < nqp) ? s_key[t] : INVALID_KEY;
            const bool valid = k != INVALID_KEY;
            const bool head = valid && (t == 0 || s_key[t - 1] + 1u != k);
            const uint32_t kn = (t + 1 < nqp) ? s_key[t + 1] : INVALID_KEY;
            const bool tail = valid && (kn == INVALID_KEY || kn != k + 1u);
            const unsigned hm = __ballot_sync(0xffffffffu, head);
            if (runs) {
                if (head) runs[base_out + nr + __popc(hm & ((1u << lane) - 1u))].x = (int)k;
                // the run index of a tail is the number of heads at or before it, minus one
                if (tail) runs[base_out + nr + __popc(hm & ((2u << lane) - 1u)) - 1].y = (int)k;
            }
            nr += __popc(hm);
        }
        if (lane == 0) s_n = nr;
    }
    __syncthreads();
    if (!runs && threadIdx.x == 0) nruns_or_off[b] = s_n;
}

// Lists the target groups that are not tasks by themselves, as (block, group), of
// 256 blocks of the launch order per CTA: those beyond a block's first, whose
// CTAs run beside the first groups' instead of after them in one CTA (1.8e6 blobs
// in an annulus, three groups in each occupied block: P2P 2.34 -> 2.02 ms), or
// all, see P2P_DIRECT_MAX.  Each group is computed by one CTA, so results do not
// depend on the list's order; a block's groups are next to each other in it.
__device__ __forceinline__ void list_groups(const P2PDesc &d, int64_t i) {
    __shared__ int s_sum[8];
    __shared__ unsigned s_at;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int g0 = d.direct ? 1 : 0;
    int b = 0, ngrp = 0;
    if (i < d.nblk) {
        b = d.order[i];
        int t0;
        ngrp = p2p_groups(p2p_targets(d, b, t0));
    }
    const int n = max(ngrp - g0, 0);
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_sum[wid] = inc;
    __syncthreads();
    int pre = 0, all = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < wid) pre += s_sum[w];
        all += s_sum[w];
    }
    if (threadIdx.x == 0 && all) s_at = atomicAdd(d.nmore, (unsigned)all);
    __syncthreads();
    const int64_t at = (int64_t)s_at + pre + inc - n;
    for (int k = 0; k < n; ++k)
        if (PF_IDX_OK(at + k, d.more_cap, 207)) d.more[at + k] = make_int2(b, g0 + k);
}

// Second half of the counting sort, and what else needs only the leaf counts
// and starts, in CTAs after the sort's gn: nc CTAs sum the counts up `nlev`
// levels from the leaves (L), the rest list P2P groups (d.nblk = 0: none).  As launches of their own the two cost 2-4 us each
// with their gaps.
__global__ void __launch_bounds__(256)
k_place(int64_t n, const uint32_t *__restrict__ key, const int32_t *__restrict__ rank,
        const int32_t *__restrict__ start, int32_t *__restrict__ perm, int32_t *__restrict__ big,
        int32_t *__restrict__ big_n, unsigned gn, int L, int nlev, unsigned nc, int32_t *cnt_all,
        const P2PDesc d) {
    if (blockIdx.x >= gn + nc) {
        list_groups(d, (int64_t)(blockIdx.x - gn - nc) * 256 + threadIdx.x);
        return;
    }
    if (blockIdx.x >= gn) {
        count_up_block(L, nlev, blockIdx.x - gn, cnt_all);
        return;
    }
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const int64_t p = (int64_t)start[key[i]] + rank[i];
    if (PF_IDX_OK(p, n, 201)) perm[p] = (int32_t)i;
    // a leaf of more than LEAF_SMALL particles (exactly one has this rank) is
    // listed for the segment sort
    if (rank[i] == LEAF_SMALL) big[atomicAdd(big_n, 1)] = (int32_t)key[i];
}

// One CTA (one warp) per target group: CTA i < direct the first group of block i
// of the launch order (heaviest first), the CTAs after those the listed groups
// (several each where clusters make more of them than CTAs).
__global__ void __launch_bounds__(32, P2P_MIN_CTAS) k_p2p(const P2PDesc d) {
    __shared__ P2PSmem sm;
    const unsigned direct = (unsigned)d.direct;
#pragma unroll 1
    for (unsigned t = blockIdx.x;; t += gridDim.x - direct) {
        int b, gi;
        if (!p2p_task(d, t, b, gi)) return;
        int t0;
        const int tn = p2p_targets(d, b, t0);
        if (tn == 0) return;
        p2p_group(d, b, t0, tn, gi, sm);
        if (t < direct) return;
    }
}

// L2P + near + scatter to input order: one thread per sorted target
template <int NP>
__global__ void __launch_bounds__(256)
k_l2p(int64_t nt, int L, double x0, double y0, double wl, const double *__restrict__ tx,
      const double *__restrict__ ty, const uint32_t *__restrict__ tkey_sorted,
      const double2 *__restrict__ Lc, const double2 *__restrict__ nearv,
      const int32_t *__restrict__ perm, double *__restrict__ vx, double *__restrict__ vy) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= nt) return;
    const uint32_t m = tkey_sorted[i];
    const uint32_t ix = compact1by1(m), iy = compact1by1(m >> 1);
    const double iw = 1.0 / wl;
    const double2 z = make_double2((tx[i] - (x0 + ((double)ix + 0.5) * wl)) * iw,
                                   (ty[i] - (y0 + ((double)iy + 0.5) * wl)) * iw);
    const double2 *lam = Lc + (level_off(L) + m) * NP;
    double2 w = lam[NP - 1];
#pragma unroll
    for (int n = NP - 2; n >= 0; --n) w = cfma(w, z, lam[n]);
    const double2 nv = nearv[i];
    const int32_t o = perm[i];
    if (!PF_IDX_OK(o, nt, 205)) return;
    vx[o] = nv.x + INV_2PI * iw * w.y;
    vy[o] = nv.y + INV_2PI * iw * w.x;
}


// ---------------------------------------------------------------------------
// Host: plan cache (tables + operators on the device)
struct FmmCache {
    int L = -1, kb = -1, np = -1;
    double ratio = -1.0;       // cutoff / root width the tables were built with
    std::vector<int64_t> sep;  // separation key of those tables (fmm_plan.cuh)
    int maxpos = 0, nq = 0, nqp = 0;
    int4 *d_far = nullptr;
    int32_t *d_far_ptr = nullptr;
    int2 *d_q = nullptr;
    int32_t *d_run_off = nullptr;  // [nblk + 1]
    int2 *d_runs = nullptr;        // (first, last) leaf of each run
    int32_t *d_blk_order = nullptr;  // P2P block launch order (heaviest first)
    int64_t nruns = 0;
    size_t dev_bytes = 0;          // device memory held by this plan
    size_t bytes() const { return dev_bytes; }
    double2 *d_pw = nullptr;
    double *d_m2m = nullptr, *d_l2l = nullptr;  // tensor-core fragment tables
    double *d_bin = nullptr;
    void release() {
        cudaFree(d_far);
        cudaFree(d_far_ptr);
        cudaFree(d_q);
        cudaFree(d_pw);
        cudaFree(d_m2m);
        cudaFree(d_l2l);
        cudaFree(d_bin);
        cudaFree(d_run_off);
        cudaFree(d_runs);
        cudaFree(d_blk_order);
        d_blk_order = nullptr;
        d_run_off = nullptr;
        d_runs = nullptr;
        d_far = nullptr;
        d_far_ptr = nullptr;
        d_q = nullptr;
        d_pw = nullptr;
        d_m2m = d_l2l = nullptr;
        d_bin = nullptr;
        L = -1;
    }
};

struct cplx {
    double re, im;
};
static cplx cm(cplx a, cplx b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }

static double binom_d(int n, int k) {
    if (k < 0 || k > n) return 0.0;
    double r = 1.0;  // exact while the value stays below 2^53
    for (int i = 1; i <= k; ++i) r = r * (double)(n - k + i) / (double)i;
    return r;
}

template <typename T>
static pf_status upload(T **dst, const std::vector<T> &v, size_t &tally) {
    if (v.empty()) {
        *dst = nullptr;
        return PF_OK;
    }
    tally += sizeof(T) * v.size();
    PF_CUDA_TRY(cudaMalloc(reinterpret_cast<void **>(dst), sizeof(T) * v.size()));
    PF_CUDA_TRY(cudaMemcpy(*dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice));
    return PF_OK;
}

static std::atomic<uint64_t> g_plan_builds{0};  // plans built in this process

static pf_status build_cache(FmmCache &c, int L, int kb, int np, double w0, double cutoff) {
    c.release();
    size_t tally = 0;
    pf::fmm::Tables t;
    pf::fmm::build_tables(L, kb, w0, cutoff, THETA, t);
    const int B = 1 << kb, Bp = B > 2 ? B : 2;
    c.maxpos = std::max(4, Bp * Bp);
    // far lists with offset ids
    std::vector<int4> far;
    std::vector<int32_t> ptr((L + 1) * c.maxpos + 1, 0);
    std::vector<pf::fmm::Off> ops;
    auto op_id = [&](const pf::fmm::Off &o) {
        for (size_t k = 0; k < ops.size(); ++k)
            if (ops[k] == o) return (int)k;
        ops.push_back(o);
        return (int)ops.size() - 1;
    };
    for (int l = 0; l <= L; ++l) {
        for (int p = 0; p < c.maxpos; ++p) {
            ptr[l * c.maxpos + p] = (int32_t)far.size();
            if (l >= 2 && p < (int)t.far[l].size())
                for (const auto &o : t.far[l][p]) {
                    // .w: the offset in Morton-dilated form (two's complement per
                    // coordinate, 16 bits each), for morton_add in k_m2l
                    const uint32_t d = morton2((uint32_t)o.i & 0xffffu, (uint32_t)o.j & 0xffffu);
                    far.push_back(make_int4(o.i, o.j, op_id(o), (int)d));
                }
        }
    }
    ptr[(L + 1) * c.maxpos] = (int32_t)far.size();  // [l*maxpos + pos] .. next slot
    // powers rho^m, m = 0..np, rho = 1/(i + i j)
    std::vector<double2> pw(ops.size() * (np + 1));
    for (size_t k = 0; k < ops.size(); ++k) {
        const double i = ops[k].i, j = ops[k].j, d = i * i + j * j;
        const cplx rho = {i / d, -j / d};
        cplx pm = {1.0, 0.0};
        for (int m = 0; m <= np; ++m) {
            pw[k * (np + 1) + m] = make_double2(pm.re, pm.im);
            pm = cm(pm, rho);
        }
    }
    // M2M / L2L operators, stored transposed for coalesced lane access
    std::vector<double2> m2m(4 * np * np), l2l(4 * np * np);
    for (int cc = 0; cc < 4; ++cc) {
        const cplx tau = {(cc & 1) ? 0.25 : -0.25, (cc & 2) ? 0.25 : -0.25};
        std::vector<cplx> tp(np);
        tp[0] = {1.0, 0.0};
        for (int k = 1; k < np; ++k) tp[k] = cm(tp[k - 1], tau);
        for (int k = 0; k < np; ++k)
            for (int m = 0; m < np; ++m) {
                // M2M: out k, in m (m <= k): C(k,m) tau^(k-m) 2^-m   -> opT[c][m][k]
                cplx a = {0.0, 0.0};
                if (m <= k) {
                    const double s = binom_d(k, m) * std::ldexp(1.0, -m);
                    a = {tp[k - m].re * s, tp[k - m].im * s};
                }
                m2m[(size_t)cc * np * np + (size_t)m * np + k] = make_double2(a.re, a.im);
                // L2L: out n = k, in m (m >= n): 1/2 C(m,n) tau^(m-n) 2^-n -> opT[c][m][n]
                cplx b = {0.0, 0.0};
                if (m >= k) {
                    const double s = 0.5 * binom_d(m, k) * std::ldexp(1.0, -k);
                    b = {tp[m - k].re * s, tp[m - k].im * s};
                }
                l2l[(size_t)cc * np * np + (size_t)m * np + k] = make_double2(b.re, b.im);
            }
    }
    // the same operators as A-operand fragment tables of the tensor-core
    // kernels: [c][part][mt][ks][lane] = part of T_c[8 mt + lane/4][4 ks + lane%4]
    // with T_c[k][m] = m2m[c][m][k] (M2M) and T_c[n][m] = l2l[c][m][n] (L2L)
    const int MTh = (np + 7) / 8, KSh = (np + 3) / 4;
    std::vector<double> m2mf(4 * 2 * MTh * KSh * 32), l2lf(m2mf.size());
    for (int cc = 0; cc < 4; ++cc)
        for (int part = 0; part < 2; ++part)
            for (int mt = 0; mt < MTh; ++mt)
                for (int ks = 0; ks < KSh; ++ks)
                    for (int ln = 0; ln < 32; ++ln) {
                        const int row = 8 * mt + ln / 4, col = 4 * ks + ln % 4;
                        const size_t o = ((((size_t)cc * 2 + part) * MTh + mt) * KSh + ks) * 32 + ln;
                        double vm = 0.0, vl = 0.0;
                        if (row < np && col < np) {
                            const double2 a = m2m[(size_t)cc * np * np + (size_t)col * np + row];
                            const double2 b = l2l[(size_t)cc * np * np + (size_t)col * np + row];
                            vm = part ? a.y : a.x;
                            vl = part ? b.y : b.x;
                        }
                        m2mf[o] = vm;
                        l2lf[o] = vl;
                    }
    std::vector<double> bin(np * np);
    for (int k = 0; k < np; ++k)
        for (int n = 0; n < np; ++n) bin[k * np + n] = binom_d(n + k, k);
    std::vector<int2> q;
    for (const auto &o : t.p2p) q.push_back(make_int2(o.i, o.j));
    c.nq = (int)q.size();
    c.nqp = 1;
    while (c.nqp < c.nq) c.nqp <<= 1;
    PF_TRY(upload(&c.d_far, far, tally));
    PF_TRY(upload(&c.d_far_ptr, ptr, tally));
    PF_TRY(upload(&c.d_q, q, tally));
    PF_TRY(upload(&c.d_pw, pw, tally));
    PF_TRY(upload(&c.d_m2m, m2mf, tally));
    PF_TRY(upload(&c.d_l2l, l2lf, tally));
    PF_TRY(upload(&c.d_bin, bin, tally));
    if (c.nqp <= P2P_QMAX) {
        // P2P run lists of every block (geometry only, reused by every call)
        const int64_t nblk = (int64_t)1 << (2 * (L - kb));
        PF_CUDA_TRY(cudaMalloc(&c.d_run_off, sizeof(int32_t) * (nblk + 1)));
        k_p2p_runs<<<(unsigned)nblk, P2P_SETUP_THREADS>>>(L, kb, c.d_q, c.nq, c.nqp, c.d_run_off,
                                                          nullptr);
        PF_TRY(pf::launch_status("k_p2p_runs"));
        std::vector<int32_t> cnt(nblk + 1, 0);
        PF_CUDA_TRY(cudaMemcpy(cnt.data(), c.d_run_off, sizeof(int32_t) * nblk,
                               cudaMemcpyDeviceToHost));
        int64_t acc = 0;
        for (int64_t b = 0; b < nblk; ++b) {
            const int32_t v = cnt[b];
            cnt[b] = (int32_t)acc;
            acc += v;
        }
        cnt[nblk] = (int32_t)acc;
        c.nruns = acc;
        PF_CUDA_TRY(cudaMemcpy(c.d_run_off, cnt.data(), sizeof(int32_t) * (nblk + 1),
                               cudaMemcpyHostToDevice));
        PF_CUDA_TRY(cudaMalloc(&c.d_runs, sizeof(int2) * (acc > 0 ? acc : 1)));
        k_p2p_runs<<<(unsigned)nblk, P2P_SETUP_THREADS>>>(L, kb, c.d_q, c.nq, c.nqp, c.d_run_off,
                                                          c.d_runs);
        PF_TRY(pf::launch_status("k_p2p_runs"));
        PF_CUDA_TRY(cudaDeviceSynchronize());
        tally += sizeof(int32_t) * (nblk + 1) + sizeof(int2) * (acc > 0 ? acc : 1);
        // launch order of the blocks: most near-set leaves first, so that the
        // lighter blocks (near the domain edges) fill the end of the launch
        std::vector<int2> runs(acc > 0 ? acc : 1);
        if (acc > 0)
            PF_CUDA_TRY(cudaMemcpy(runs.data(), c.d_runs, sizeof(int2) * acc,
                                   cudaMemcpyDeviceToHost));
        std::vector<int64_t> wgt(nblk, 0);
        for (int64_t b = 0; b < nblk; ++b)
            for (int32_t r = cnt[b]; r < cnt[b + 1]; ++r) wgt[b] += runs[r].y - runs[r].x + 1;
        std::vector<int32_t> order(nblk);
        for (int64_t b = 0; b < nblk; ++b) order[b] = (int32_t)b;
        std::stable_sort(order.begin(), order.end(),
                         [&](int32_t a, int32_t b) { return wgt[a] > wgt[b]; });
        PF_TRY(upload(&c.d_blk_order, order, tally));
    }
    c.dev_bytes = tally;
    c.L = L;
    c.kb = kb;
    c.np = np;
    c.ratio = cutoff / w0;
    pf::fmm::separation_key(L, 1.0, c.ratio, THETA, c.sep);
    g_plan_builds.fetch_add(1, std::memory_order_relaxed);
    return PF_OK;
}

struct Sorted {
    uint32_t *key = nullptr;
    int32_t *rank = nullptr, *perm = nullptr, *cnt = nullptr, *start = nullptr;
    double *x = nullptr, *y = nullptr, *g = nullptr;
    float4 *hl = nullptr;
    float *g32 = nullptr;
};

// Sort by leaf; also the box counts of all levels (cnt_all, s.cnt its leaf
// level) up to COUNT_LEVELS above the leaves, see count_up, and with pd.nblk > 0
// the list of P2P groups.  ctr: the call's counters to clear, or nullptr.  n > 0.
static pf_status sort_points(int64_t n, const double *x, const double *y,
                             const double *g, double x0, double y0, double wl, int L, Sorted &s,
                             int32_t *scan_tmp, uint32_t *skey, int32_t *big, int32_t *big_n,
                             int32_t *cnt_all, unsigned long long *ctr, const P2PDesc &pd,
                             cudaStream_t st) {
    const int64_t nleaf = (int64_t)1 << (2 * L);
    PF_CUDA_TRY(cudaMemsetAsync(s.cnt, 0, sizeof(int32_t) * nleaf, st));
    const unsigned gn = (unsigned)pf::ceil_div(n, 256);
    k_leaf_keys<<<gn, 256, 0, st>>>(x, y, n, x0, y0, wl, L, s.key, s.rank, s.cnt, big_n, ctr);
    PF_TRY(pf::launch_status("k_leaf_keys"));
    PF_TRY(pf::exclusive_scan_i32(s.cnt, s.start, nleaf, scan_tmp, nullptr, st));
    const int nlev = std::min(L, COUNT_LEVELS);
    const unsigned nc = 1u << (2 * (L - nlev));
    const unsigned nm = (unsigned)pf::ceil_div(pd.nblk, 256);
    k_place<<<gn + nc + nm, 256, 0, st>>>(n, s.key, s.rank, s.start, s.perm, big, big_n, gn, L,
                                          nlev, nc, cnt_all, pd);
    PF_TRY(pf::launch_status("k_place"));
    // leaves above LEAF_SMALL particles (dense clusters); the ranks are free now
    PF_TRY(pf::seg_sort_listed(big, big_n, s.start, s.cnt, s.perm, s.rank,
                               n / (LEAF_SMALL + 1) + 1, st));
    // the ranks are free again: they receive the final permutation
    k_gather_sorted<<<gn, 256, 0, st>>>(n, s.perm, s.key, s.start, s.cnt, x, y, g, s.rank, s.x,
                                        s.y, s.g, s.hl, s.g32, skey);
    std::swap(s.perm, s.rank);
    return pf::launch_status("k_gather_sorted");
}

// the box counts of the levels above those that sort_points sums up
static pf_status count_up(int L, int32_t *cnt_all, cudaStream_t st) {
    static_assert(pf::fmmx::MAX_LEVEL <= 2 * COUNT_LEVELS, "two passes reach the root");
    if (L <= COUNT_LEVELS) return PF_OK;
    k_count_up<<<1, 256, 0, st>>>(L - COUNT_LEVELS, L - COUNT_LEVELS, cnt_all);
    return pf::launch_status("k_count_up");
}

struct FmmArgs {
    int64_t ns, nt;
    const double *x, *y, *g, *xt, *yt;
    double ksigmasqr, cutoff, tol;
    int ndirect;
    double *vx, *vy;
    int num_sms;
    int64_t groups_beside = 0;  // P2P groups of other sets whose calls run beside this one
};

// P2P target groups to expect: one per block and one more per 96 targets, but no
// more than the blocks of a partly filled tree can hold, 40 targets each or, in
// a tree of finer leaves, half as many again as a block has on average.
static int64_t p2p_groups_expected(int64_t nblk, int64_t nt) {
    const int64_t each = std::min<int64_t>(40, std::max<int64_t>(8, 3 * nt / (2 * nblk)));
    return std::min<int64_t>(nblk + nt / P2P_GROUP, nt / each);
}

// Warps per target group (the result is the same), from the number of groups to
// expect, this set's and (two thirds of) those of the sets beside it in a batch:
// the device holds 20 one-warp CTAs per SM (2960), and one group alone is a serial
// chain of 40-100 chunks; several warps cost barriers and exchanges, 40-75% where
// the device is full.  P2P time with 1 / 4 / 8 warps, uniform sets: 3,001 blobs 73 /
// 42 / 30 us; 30,000 163 / 89 / 79; 38,000 87 / 81 / 93; 100,000 185 / 163 / 187;
// 140,000 230 / 234 / 273; 150,000 198 / 280 / 325.  A call in a tree of finer
// leaves, 62,384 blobs at level 7: 280 / 333 / 408, 15,129 at level 6: 125 / 132 / 152.
static int p2p_warps(int64_t nblk, int64_t nt, int64_t groups_beside, int num_sms) {
    const int64_t groups = p2p_groups_expected(nblk, nt) + 2 * groups_beside / 3;
    const int64_t resident = (int64_t)num_sms * P2P_MIN_CTAS;
    return groups <= resident / 5 ? 8 : groups <= resident * 3 / 4 ? 4 : 1;
}

// Blocks up to which each block's first group is a CTA by itself, the heaviest
// blocks first; beyond, all groups are listed.  Uniform sets of 150,000 and 2^20
// blobs lose 4 and 2% of P2P when listed, by the order of the last CTAs.  From
// 65,536 blocks on that is 0.8% (2^22 blobs), and the empty blocks' CTAs and the
// second groups being far from the first cost more: 2^22 blobs in an annulus, P2P
// 3.10 ms, listed 2.77 (one CTA per block for all its groups 2.97).
constexpr int64_t P2P_DIRECT_MAX = 32768;

static int64_t p2p_direct(int64_t nblk) { return nblk <= P2P_DIRECT_MAX ? nblk : 0; }

// Most groups that can be listed.
static int64_t p2p_more_cap(int64_t nblk, int64_t nt) {
    return nt / P2P_GROUP + 1 + nblk - p2p_direct(nblk);
}

// CTAs for the listed groups: those of a layer around a body, or what the device
// holds (mostly idle CTAs for every group there could be cost 13 us at 2^20
// uniform blobs).
static int64_t p2p_more_ctas(int64_t nblk, int64_t nt, int num_sms) {
    const int64_t direct = p2p_direct(nblk), resident = (int64_t)num_sms * P2P_MIN_CTAS;
    return std::min<int64_t>(p2p_more_cap(nblk, nt),
                             std::max<int64_t>({resident, nblk - direct, nt / 60 - direct}));
}

static size_t fmm_scratch_bytes(const FmmCache &c, int64_t ns, int64_t nt, bool same) {
    const int L = c.L, NP = c.np;
    const int64_t nleaf = (int64_t)1 << (2 * L);
    const int64_t nbox = level_off(L + 1);
    size_t need = 0;
    auto add = [&](size_t b) { need += pf::align256(b); };
    add(4 * ns); add(4 * ns); add(4 * ns);          // key rank perm
    add(8 * ns); add(8 * ns); add(8 * ns);          // x y g
    add(16 * ns); add(4 * ns);                      // hl g32
    if (!same) {
        add(4 * nt); add(4 * nt); add(4 * nt);
        add(8 * nt); add(8 * nt); add(16 * nt);
    }
    add(4 * nt);                                    // sorted target keys
    add(4 * nbox); add(4 * nbox);                   // counts (all levels) src, tgt
    add(4 * nleaf); add(4 * nleaf);                 // starts src, tgt
    add(16 * (size_t)nbox * NP); add(16 * (size_t)nbox * NP);  // M, L
    add(16 * nt);                                   // near velocities
    add(4 * (std::max(ns, nt) / (LEAF_SMALL + 1) + 3));  // leaves for the segment sort
    add(8 * (size_t)p2p_more_cap((int64_t)1 << (2 * (L - c.kb)), nt));  // P2P groups listed
    add(4 * pf::scan_tmp_ints(nleaf));
    return need + 4096;
}

// Run the FMM for one blob set on `st` with a built plan and a scratch region
// of fmm_scratch_bytes(); enqueues kernels only (no host synchronisation).
// ctr: FMM_COUNTERS device counters (P2P pairs, M2L translations, P2P pairs
// evaluated without the exponential), zeroed here.
// ev: 7 events recorded around the phases, or nullptr.
// side: a second stream for the far field, or nullptr (everything on st).
template <int NP>
static pf_status exec_fmm(pf::Bump &sc, const FmmArgs &a, const FmmCache &c, double x0,
                          double y0, double w0, unsigned long long *ctr, cudaEvent_t *ev,
                          const pf::SideStream *side, cudaStream_t st) {
    const int L = c.L, kb = c.kb;
    const bool same = (a.xt == a.x && a.yt == a.y && a.nt == a.ns);
    const double wl = std::ldexp(w0, -L);
    const int64_t nleaf = (int64_t)1 << (2 * L);
    const int64_t nbox = level_off(L + 1);
    const int64_t ns = a.ns, nt = a.nt;
    auto take = [&](size_t b) { return sc.take(b); };
    Sorted S, T;
    S.key = (uint32_t *)take(4 * ns);
    S.rank = (int32_t *)take(4 * ns);
    S.perm = (int32_t *)take(4 * ns);
    S.x = (double *)take(8 * ns);
    S.y = (double *)take(8 * ns);
    S.g = (double *)take(8 * ns);
    S.hl = (float4 *)take(16 * ns);
    S.g32 = (float *)take(4 * ns);
    if (!same) {
        T.key = (uint32_t *)take(4 * nt);
        T.rank = (int32_t *)take(4 * nt);
        T.perm = (int32_t *)take(4 * nt);
        T.x = (double *)take(8 * nt);
        T.y = (double *)take(8 * nt);
        T.hl = (float4 *)take(16 * nt);
    }
    uint32_t *tkey_sorted = (uint32_t *)take(4 * nt);
    int32_t *scnt_all = (int32_t *)take(4 * nbox);
    int32_t *tcnt_all = (int32_t *)take(4 * nbox);
    S.cnt = scnt_all + level_off(L);
    S.start = (int32_t *)take(4 * nleaf);
    int32_t *tstart = (int32_t *)take(4 * nleaf);
    double2 *M = (double2 *)take(16 * (size_t)nbox * NP);
    double2 *Lc = (double2 *)take(16 * (size_t)nbox * NP);
    double2 *nearv = (double2 *)take(16 * nt);
    // leaves listed for the segment sort: [0] count, [1 ..] leaf ids
    int32_t *big = (int32_t *)take(4 * (std::max(ns, nt) / (LEAF_SMALL + 1) + 3));
    // P2P groups that are listed
    const int64_t nblk = (int64_t)1 << (2 * (L - kb));
    const int64_t more_cap = p2p_more_cap(nblk, nt);
    int2 *more = (int2 *)take(8 * (size_t)more_cap);
    int32_t *tmp = (int32_t *)take(4 * pf::scan_tmp_ints(nleaf));
    if (!tmp) {
        pf::set_error("pf_velocity_fmm: scratch layout error");
        return PF_ERR_OOM;
    }
    if (same) {  // targets are the sources: one tree, the target arrays alias the source ones
        T = S;
        tcnt_all = scnt_all;
        tstart = S.start;
    } else {
        T.cnt = tcnt_all + level_off(L);
        T.start = tstart;
    }

    // the near field's description
    P2PDesc pd;
    pd.nblk = nblk;
    pd.direct = p2p_direct(nblk);
    pd.kb = kb;
    pd.tstart = tstart;
    pd.tcnt = T.cnt;
    pd.sstart = S.start;
    pd.scnt = S.cnt;
    pd.shl = S.hl;
    pd.sg32 = S.g32;
    pd.thl = T.hl;
    pd.run_off = c.d_run_off;
    pd.runs = c.d_runs;
    pd.order = c.d_blk_order;
    pd.gp = pfd::make_gauss_params(a.ksigmasqr);
    pd.nearv = nearv;
    pd.pairs = ctr;
    pd.nmore = reinterpret_cast<unsigned *>(ctr + pf::fmmx::FMM_COUNTERS - 1);
    pd.more = more;
    pd.more_cap = more_cap;
    pd.ns = ns;
    pd.nt = nt;

    auto mark = [&](int k) -> pf_status {
        if (ev) PF_CUDA_TRY(cudaEventRecord(ev[k], st));
        return PF_OK;
    };
    PF_TRY(mark(0));
    // sort sources (and targets)
    // sorted target keys come out of the sorted copies of the targets
    P2PDesc none = pd;
    none.nblk = 0;
    PF_TRY(sort_points(ns, a.x, a.y, a.g, x0, y0, wl, L, S, tmp, same ? tkey_sorted : nullptr,
                       big + 1, big, scnt_all, ctr, same ? pd : none, st));
    if (!same)
        PF_TRY(sort_points(nt, a.xt, a.yt, nullptr, x0, y0, wl, L, T, tmp, tkey_sorted, big + 1,
                           big, tcnt_all, nullptr, pd, st));
    if (same) T = S;  // sort_points replaced S.perm by the final permutation

    PF_TRY(mark(1));
    const int warps = p2p_warps(nblk, nt, a.groups_beside, a.num_sms);
    auto near = [&]() -> pf_status {
        if (warps > 1) {
            PF_TRY(pf::fmmx::launch_p2p_multi(pd, warps, (unsigned)(pd.direct + more_cap), st));
        } else {
            k_p2p<<<(unsigned)(pd.direct + p2p_more_ctas(nblk, nt, a.num_sms)), 32, 0, st>>>(pd);
            PF_TRY(pf::launch_status("k_p2p"));
        }
        return PF_OK;
    };
    auto far = [&](cudaStream_t fs) -> pf_status {
        // upward pass
        k_p2m<NP><<<(unsigned)pf::ceil_div(4 * nleaf, 128), 128, 0, fs>>>(L, x0, y0, wl, S.start, S.cnt,
                                                                     S.x, S.y, S.g, M);
        PF_TRY(pf::launch_status("k_p2m"));
        PF_TRY(count_up(L, scnt_all, fs));
        if (!same) PF_TRY(count_up(L, tcnt_all, fs));
        // parents at levels L-1 .. 2: two levels per launch, one more when odd
        int lp = L - 1;
        for (; lp - 1 >= 2; lp -= 2) {
            const int64_t tasks = ((int64_t)1 << (2 * lp)) / 4;
            k_m2m_tc<NP><<<(unsigned)pf::ceil_div(tasks, TC_THREADS / 32), TC_THREADS, 0, fs>>>(
                lp, true, scnt_all, M, c.d_m2m);
            PF_TRY(pf::launch_status("k_m2m_tc"));
        }
        if (lp >= 2) {
            const int64_t tasks = ((int64_t)1 << (2 * lp)) / 4;
            k_m2m_tc<NP><<<(unsigned)pf::ceil_div(tasks, TC_THREADS / 32), TC_THREADS, 0, fs>>>(
                lp, false, scnt_all, M, c.d_m2m);
            PF_TRY(pf::launch_status("k_m2m_tc"));
        }
        PF_TRY(mark(2));
        // M2L, all levels >= 2
        const int B = 1 << kb, Bp = B > 2 ? B : 2;
        {
            const int64_t nquad = (nbox - level_off(2)) / 4;  // box quads of levels 2..L
            if (nquad <= M2L_AHEAD_QUADS && a.groups_beside == 0)
                k_m2l<NP, true><<<(unsigned)nquad, 32, 0, fs>>>(
                    L, Bp, nquad, scnt_all, tcnt_all, M, Lc, c.d_far, c.d_far_ptr, c.maxpos, c.d_pw,
                    c.d_bin, ctr + 1);
            else
                k_m2l<NP, false><<<(unsigned)pf::ceil_div(nquad, M2L_THREADS / 32), M2L_THREADS, 0,
                                   fs>>>(L, Bp, nquad, scnt_all, tcnt_all, M, Lc, c.d_far,
                                         c.d_far_ptr, c.maxpos, c.d_pw, c.d_bin, ctr + 1);
            PF_TRY(pf::launch_status("k_m2l"));
        }
        PF_TRY(mark(3));
        // child levels 3 .. L: two levels per launch, one more when odd
        int lch = 3;
        for (; lch + 1 <= L; lch += 2) {
            const int64_t tasks = ((int64_t)1 << (2 * (lch + 1))) / 16;
            k_l2l_tc<NP><<<(unsigned)pf::ceil_div(tasks, TC_THREADS / 32), TC_THREADS, 0, fs>>>(
                lch + 1, true, tcnt_all, Lc, c.d_l2l);
            PF_TRY(pf::launch_status("k_l2l_tc"));
        }
        if (lch <= L) {
            const int64_t tasks = ((int64_t)1 << (2 * lch)) / 16;
            k_l2l_tc<NP><<<(unsigned)pf::ceil_div(tasks, TC_THREADS / 32), TC_THREADS, 0, fs>>>(
                lch, false, tcnt_all, Lc, c.d_l2l);
            PF_TRY(pf::launch_status("k_l2l_tc"));
        }
        return PF_OK;
    };
    // The near field and the far field (upward pass, M2L, downward pass) share
    // no data: where the caller gives a second stream (and asks for no phase
    // events) they run side by side.  Few blobs leave the SMs idle under either
    // chain; many blobs keep the FP32/exp pipes busy in the one and the FP64
    // tensor pipe in the other.  Serial -> side by side, uniform blobs: 30,000
    // 197 -> 157 us, 60,000 222 -> 183, 200,000 426 -> 354, 500,000 806 -> 714,
    // 2^20 1315 -> 1224; 1.8 million beside a wall 2431 -> 2272.  Several warps per
    // group, so few groups: the near field is the longer chain and is enqueued
    // first (12,000 blobs 102 us, far first 106; 30,000 130 / 136).  One warp per
    // group: its CTAs take all registers of the SMs, and what is enqueued after
    // them waits for a CTA to end, so the far field goes first (the other way
    // round with the far field on a stream of high priority, 120,000 326 / 270).
    // The two streams have the same priority: high priority for the far field
    // gained 4-5% at 30,000-60,000 blobs, but while a process has streams of two
    // priorities its batch graphs run 3% slower (12 sets 1337 -> 1372).  Both
    // statuses are looked at after the join, so that the caller's stream always
    // waits for the far field.
    if (side && !ev) {
        PF_CUDA_TRY(cudaEventRecord(side->fork, st));
        PF_CUDA_TRY(cudaStreamWaitEvent(side->stream, side->fork, 0));
        const bool near_first = warps > 1;
        pf_status sn = PF_OK;
        if (near_first) sn = near();
        const pf_status sf = far(side->stream);
        if (!near_first) sn = near();
        PF_CUDA_TRY(cudaEventRecord(side->join, side->stream));
        PF_CUDA_TRY(cudaStreamWaitEvent(st, side->join, 0));
        PF_TRY(sn);
        PF_TRY(sf);
    } else {
        PF_TRY(far(st));
        PF_TRY(mark(4));
        PF_TRY(near());
        PF_TRY(mark(5));
    }
    k_l2p<NP><<<(unsigned)pf::ceil_div(nt, 256), 256, 0, st>>>(nt, L, x0, y0, wl, T.x, T.y,
                                                               tkey_sorted, Lc, nearv, T.perm,
                                                               a.vx, a.vy);
    PF_TRY(pf::launch_status("k_l2p"));
    return mark(6);
}

}  // namespace

// ---------------------------------------------------------------------------
namespace pf {

struct FmmTuning {
    int leaf_level = 0;  // 0 = automatic
    int np = 0;          // 0 = from tol
    int kb = 1;
};
static thread_local FmmTuning g_tune;

int fmmx::np_for_tol(double tol) {
    // Truncation after p+1 terms is bounded by ~theta^(p+1) per translation
    // (theta = 1/2), but the measured end-to-end error is far below that bound:
    // with 16 terms the point-vortex limit (theta-bound at every level) and the
    // Gaussian configurations all stay near 1e-7 at tol = 1e-6, where the FP32
    // near field sets the floor.  So p+1 = log2(1/tol) - 4, rounded up to an
    // instantiated size.
    const int want = (int)std::ceil(std::log2(1.0 / tol)) - 4;
    const int opts[] = {16, 20, 24, 28, 32};
    for (int o : opts)
        if (o >= want) return o;
    return 32;
}

pf_status fmm_exec(const FmmCache &c, double x0, double y0, double w0, Bump &sc,
                   const FmmArgs &a, unsigned long long *ctr, cudaEvent_t *ev,
                   const SideStream *side, cudaStream_t st) {
    switch (c.np) {
        case 16: return exec_fmm<16>(sc, a, c, x0, y0, w0, ctr, ev, side, st);
        case 20: return exec_fmm<20>(sc, a, c, x0, y0, w0, ctr, ev, side, st);
        case 24: return exec_fmm<24>(sc, a, c, x0, y0, w0, ctr, ev, side, st);
        case 28: return exec_fmm<28>(sc, a, c, x0, y0, w0, ctr, ev, side, st);
        case 32: return exec_fmm<32>(sc, a, c, x0, y0, w0, ctr, ev, side, st);
        default:
            // the plan's coefficient arrays are sized for c.np: never run another size on them
            set_error("FMM: %d expansion terms is not an instantiated size (16, 20, 24, 28, 32)",
                      c.np);
            return PF_ERR_INVALID_ARG;
    }
}

// Process-wide cache of read-only plans, shared by every context and thread.
// Tables depend on the geometry only through cutoff / root width, and on that
// ratio only through its separation key (fmm_plan.cuh), so plans are built
// normalised (root width 1) and keyed by (device, L, kb, np, key): a moving
// blob set whose box width drifts keeps its plan until a list changes.
// Least recently used plans are dropped past PF_PLAN_CACHE_BYTES (env,
// default 4 GiB); their device memory is freed when the last user lets go.
struct PlanKey {
    int dev, L, kb, np;
    std::vector<int64_t> sep;
    bool operator<(const PlanKey &o) const {
        if (dev != o.dev) return dev < o.dev;
        if (L != o.L) return L < o.L;
        if (kb != o.kb) return kb < o.kb;
        if (np != o.np) return np < o.np;
        return sep < o.sep;
    }
};
struct PlanCacheStore {
    std::mutex mu;
    std::map<PlanKey, std::pair<std::shared_ptr<FmmCache>, uint64_t>> map;  // plan, last use
    uint64_t tick = 0;
    size_t bytes = 0;
};
static PlanCacheStore &plan_store() {
    static PlanCacheStore *s = new PlanCacheStore();  // never destroyed: outlives the contexts
    return *s;
}
static size_t plan_budget() {
    const char *e = getenv("PF_PLAN_CACHE_BYTES");
    return e ? (size_t)strtoull(e, nullptr, 10) : ((size_t)4 << 30);
}

pf_status shared_plan(int dev, int L, int kb, int np, double ratio,
                      std::shared_ptr<FmmCache> *out) {
    PlanCacheStore &ps = plan_store();
    PlanKey key{dev, L, kb, np, {}};
    pf::fmm::separation_key(L, 1.0, ratio, THETA, key.sep);
    std::lock_guard<std::mutex> lock(ps.mu);
    auto it = ps.map.find(key);
    if (it != ps.map.end()) {
        it->second.second = ++ps.tick;
        *out = it->second.first;
        return PF_OK;
    }
    auto c = std::shared_ptr<FmmCache>(new FmmCache(), [](FmmCache *p) {
        p->release();
        delete p;
    });
    PF_TRY(build_cache(*c, L, kb, np, 1.0, ratio));
    const size_t b = c->bytes();
    while (!ps.map.empty() && ps.bytes + b > plan_budget()) {
        auto old = ps.map.begin();
        for (auto j = ps.map.begin(); j != ps.map.end(); ++j)
            if (j->second.second < old->second.second) old = j;
        ps.bytes -= old->second.first->bytes();
        ps.map.erase(old);
    }
    ps.map[key] = {c, ++ps.tick};
    ps.bytes += b;
    *out = c;
    return PF_OK;
}

}  // namespace pf

extern "C" uint64_t pf_fmm_plan_builds(void) {
    return g_plan_builds.load(std::memory_order_relaxed);
}

extern "C" pf_status pf_fmm_set_tuning(int leaf_level, int expansion_terms, int block_level_drop) {
    pf::clear_error();
    PF_CHECK_ARG(leaf_level == 0 || (leaf_level >= 2 && leaf_level <= MAX_LEVEL),
                 "pf_fmm_set_tuning: leaf level must be 0 (auto) or in [2, %d]", MAX_LEVEL);
    PF_CHECK_ARG(expansion_terms == 0 || expansion_terms == 16 || expansion_terms == 20 ||
                     expansion_terms == 24 || expansion_terms == 28 || expansion_terms == 32,
                 "pf_fmm_set_tuning: expansion terms must be 0 (auto) or one of 16,20,24,28,32");
    PF_CHECK_ARG(block_level_drop >= 0 && block_level_drop <= 2,
                 "pf_fmm_set_tuning: block level drop must be in [0, 2]");
    pf::g_tune.leaf_level = leaf_level;
    pf::g_tune.np = expansion_terms;
    pf::g_tune.kb = block_level_drop;
    return PF_OK;
}

extern "C" pf_status pf_fmm_tree_keys(pf_ctx *ctx, int64_t n, const double *x, const double *y,
                                      double x0, double y0, double leaf_width, int leaf_level,
                                      uint32_t *keys, void *stream) {
    PF_RANGE("pf_fmm_tree_keys");
    pf::clear_error();
    PF_CHECK_ARG(ctx != nullptr, "pf_fmm_tree_keys: NULL context");
    PF_CHECK_ARG(leaf_level >= 1 && leaf_level <= 15, "pf_fmm_tree_keys: leaf level outside [1, 15]");
    PF_CHECK_ARG(leaf_width > 0.0, "pf_fmm_tree_keys: leaf width must be positive");
    PF_CHECK_ARG(n >= 0 && (n == 0 || (x && y && keys)), "pf_fmm_tree_keys: bad arrays");
    pf::DeviceGuard dg(ctx->device);
    if (n == 0) return PF_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    k_leaf_keys<<<(unsigned)pf::ceil_div(n, 256), 256, 0, st>>>(x, y, n, x0, y0, leaf_width,
                                                               leaf_level, keys, nullptr, nullptr,
                                                               nullptr, nullptr);
    return pf::launch_status("k_leaf_keys");
}

namespace {

// pf_velocity_fmm (box == nullptr: bounding box of sources and targets read
// back from the device, one synchronisation) and pf_velocity_fmm_box (box
// given by the caller, no synchronisation).
pf_status velocity_fmm(pf_ctx *ctx, int64_t n_src, const double *x, const double *y,
                       const double *g, int64_t n_tgt, const double *xt, const double *yt,
                       double ksigmasqr, double cutoff, double tol, int ndirect, double *vx,
                       double *vy, const double *box, void *stream) {
    PF_CHECK_ARG(ctx != nullptr, "pf_velocity_fmm: NULL context");
    PF_CHECK_ARG(n_src >= 0 && n_tgt >= 0 && n_src < ((int64_t)1 << 31) &&
                     n_tgt < ((int64_t)1 << 31),
                 "pf_velocity_fmm: sizes outside [0, 2^31)");
    PF_CHECK_ARG(ksigmasqr > 0.0 && std::isfinite(ksigmasqr), "pf_velocity_fmm: bad ksigmasqr");
    PF_CHECK_ARG(std::isfinite(cutoff) && cutoff >= 0.0, "pf_velocity_fmm: bad cutoff");
    PF_CHECK_ARG(tol >= 0.0 && tol < 1.0, "pf_velocity_fmm: tol must be in [0, 1)");
    PF_CHECK_ARG(n_src == 0 || (x && y && g), "pf_velocity_fmm: NULL blob array");
    PF_CHECK_ARG(n_tgt == 0 || (xt && yt && vx && vy), "pf_velocity_fmm: NULL target array");
    PF_CHECK_ARG(!box || (std::isfinite(box[0]) && std::isfinite(box[1]) && std::isfinite(box[2]) &&
                          std::isfinite(box[3]) && box[0] <= box[1] && box[2] <= box[3]),
                 "pf_velocity_fmm_box: box must be finite with min <= max");
    pf::DeviceGuard dg(ctx->device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ctx->last_stream = st;
    pf_fmm_stats &stt = ctx->last_stats;
    memset(&stt, 0, sizeof(stt));
    stt.n_src = n_src;
    stt.n_tgt = n_tgt;
    stt.used_direct = 1;
    if (n_tgt == 0) return PF_OK;
    if (n_src == 0) {
        PF_CUDA_TRY(cudaMemsetAsync(vx, 0, sizeof(double) * n_tgt, st));
        PF_CUDA_TRY(cudaMemsetAsync(vy, 0, sizeof(double) * n_tgt, st));
        return PF_OK;
    }
    if (ndirect < 1) ndirect = 1;
    // leaf level: as the reference's level count, ceil(log4(N / Ndirect))
    int L = pf::g_tune.leaf_level;
    if (L == 0) L = pf::fmmx::auto_level(n_src, ndirect);
    if (tol == 0.0 || L < 3)
        return pf::launch_direct(ctx, n_src, x, y, g, n_tgt, xt, yt, ksigmasqr, vx, vy, st);
    const int np = pf::g_tune.np ? pf::g_tune.np : pf::fmmx::np_for_tol(tol);
    int kb = pf::g_tune.kb;

    // bounding square of sources and targets
    double xmin, xmax, ymin, ymax;
    if (box) {
        xmin = box[0];
        xmax = box[1];
        ymin = box[2];
        ymax = box[3];
    } else {
        const int cap = ctx->num_sms * 4;  // each CTA ends in an atomic on the ticket
        PF_TRY(pf::arena_reserve(ctx, pf::align256(cap * sizeof(BBox))));
        BBox *part = static_cast<BBox *>(pf::arena_take(ctx, cap * sizeof(BBox)));
        // targets that are the sources, or the first of them, are in their box (sources
        // that are the first of the targets, the same pointers, don't cover them)
        const int64_t nt_box = (xt == x && yt == y && n_tgt <= n_src) ? 0 : n_tgt;
        const int64_t nb = std::min<int64_t>(pf::ceil_div(n_src + nt_box, 256), cap);
        k_bbox<<<(unsigned)nb, 256, 0, st>>>(
            x, y, n_src, xt, yt, nt_box, part,
            reinterpret_cast<unsigned *>(ctx->dev_small + pf::fmmx::FMM_COUNTERS),
            reinterpret_cast<BBox *>(ctx->host_small));
        PF_TRY(pf::launch_status("k_bbox"));
        BBox hb;
        PF_CUDA_TRY(cudaStreamSynchronize(st));
        memcpy(&hb, ctx->host_small, sizeof(BBox));
        if (hb.bad) {
            pf::set_error("pf_velocity_fmm: NaN or Inf coordinate");
            return PF_ERR_NAN_INPUT;
        }
        xmin = unord_d(hb.mnx);
        xmax = unord_d(hb.mxx);
        ymin = unord_d(hb.mny);
        ymax = unord_d(hb.mxy);
    }
    double w0 = std::max(xmax - xmin, ymax - ymin);
    if (!(w0 > 0.0)) w0 = 1.0;
    w0 *= 1.0 + 1e-9;
    // the cutoff sets a floor on the leaf width: P2P blocks must stay bounded
    std::shared_ptr<FmmCache> cache;
    for (;;) {
        PF_TRY(pf::shared_plan(ctx->device, L, kb, np, cutoff / w0, &cache));
        if (cache->nqp <= P2P_QMAX) break;
        if (L <= 3) return pf::launch_direct(ctx, n_src, x, y, g, n_tgt, xt, yt, ksigmasqr, vx, vy, st);
        --L;  // cutoff too large for this leaf width: coarser leaves
    }
    ctx->fmm_plan_hold = cache;  // keep the plan alive while this call's kernels run
    FmmArgs a{n_src, n_tgt, x, y, g, xt, yt, ksigmasqr, cutoff, tol, ndirect, vx, vy, ctx->num_sms};
    stt.used_direct = 0;
    stt.leaf_level = L;
    stt.expansion_terms = np;
    stt.block_level_drop = kb;
    const bool same = (xt == x && yt == y && n_tgt == n_src);
    PF_TRY(pf::arena_reserve(ctx, fmm_scratch_bytes(*cache, n_src, n_tgt, same)));
    pf::Bump sc{ctx->arena.base, ctx->arena.cap, 0};
    return pf::fmm_exec(*cache, xmin, ymin, w0, sc, a,
                        reinterpret_cast<unsigned long long *>(ctx->dev_small),
                        ctx->fmm_profile ? ctx->ev : nullptr,
                        pf::side_stream(ctx, st), st);
}

}  // namespace

extern "C" pf_status pf_velocity_fmm(pf_ctx *ctx, int64_t n_src, const double *x, const double *y,
                                     const double *g, int64_t n_tgt, const double *xt,
                                     const double *yt, double ksigmasqr, double xopt,
                                     double cutoff, double tol, int ndirect, double *vx,
                                     double *vy, void *stream) {
    PF_RANGE("pf_velocity_fmm");
    pf::clear_error();
    (void)xopt;
    return velocity_fmm(ctx, n_src, x, y, g, n_tgt, xt, yt, ksigmasqr, cutoff, tol, ndirect, vx,
                        vy, nullptr, stream);
}

extern "C" pf_status pf_velocity_fmm_box(pf_ctx *ctx, int64_t n_src, const double *x,
                                         const double *y, const double *g, int64_t n_tgt,
                                         const double *xt, const double *yt, double ksigmasqr,
                                         double xopt, double cutoff, double tol, int ndirect,
                                         const double *box, double *vx, double *vy,
                                         void *stream) {
    PF_RANGE("pf_velocity_fmm_box");
    pf::clear_error();
    (void)xopt;
    PF_CHECK_ARG(box != nullptr, "pf_velocity_fmm_box: NULL box");
    return velocity_fmm(ctx, n_src, x, y, g, n_tgt, xt, yt, ksigmasqr, cutoff, tol, ndirect, vx,
                        vy, box, stream);
}

extern "C" pf_status pf_fmm_profile(pf_ctx *ctx, int enable) {
    pf::clear_error();
    PF_CHECK_ARG(ctx != nullptr, "pf_fmm_profile: NULL context");
    ctx->fmm_profile = enable != 0;
    return PF_OK;
}

extern "C" pf_status pf_fmm_last_stats(pf_ctx *ctx, pf_fmm_stats *out) {
    pf::clear_error();
    PF_CHECK_ARG(ctx != nullptr && out != nullptr, "pf_fmm_last_stats: NULL argument");
    pf::DeviceGuard dg(ctx->device);
    pf_fmm_stats s = ctx->last_stats;
    s.ms_sort = s.ms_upward = s.ms_m2l = s.ms_downward = s.ms_p2p = s.ms_l2p = s.ms_total = -1.f;
    if (!s.used_direct) {
        PF_CUDA_TRY(cudaStreamSynchronize(ctx->last_stream));
        unsigned long long c[pf::fmmx::FMM_COUNTERS];
        PF_CUDA_TRY(cudaMemcpy(c, ctx->dev_small, sizeof(c), cudaMemcpyDeviceToHost));
        s.p2p_pairs = (int64_t)c[0];
        s.m2l_translations = (int64_t)c[1];
        s.p2p_pairs_far = (int64_t)c[2];
        if (ctx->fmm_profile) {
            float t[6];
            for (int k = 0; k < 6; ++k) PF_CUDA_TRY(cudaEventElapsedTime(&t[k], ctx->ev[k], ctx->ev[k + 1]));
            s.ms_sort = t[0];
            s.ms_upward = t[1];
            s.ms_m2l = t[2];
            s.ms_downward = t[3];
            s.ms_p2p = t[4];
            s.ms_l2p = t[5];
            PF_CUDA_TRY(cudaEventElapsedTime(&s.ms_total, ctx->ev[0], ctx->ev[6]));
        }
    }
    *out = s;
    return PF_OK;
}

// ---------------------------------------------------------------------------
// internal interface (fmm_api.cuh)
namespace pf {
namespace fmmx {

struct Plan {
    FmmCache c;
    double x0 = 0.0, y0 = 0.0, w0 = 1.0;
};

Plan *plan_new() { return new Plan(); }

void plan_free(Plan *p) {
    if (!p) return;
    p->c.release();
    delete p;
}

pf_status plan_build(Plan *p, int L, int kb, int np, double x0, double y0, double w0,
                     double cutoff, bool *p2p_ok) {
    const double ratio = cutoff / w0;
    std::vector<int64_t> sep;
    pf::fmm::separation_key(L, 1.0, ratio, THETA, sep);
    if (p->c.L != L || p->c.kb != kb || p->c.np != np || p->c.sep != sep)
        PF_TRY(build_cache(p->c, L, kb, np, 1.0, ratio));
    p->x0 = x0;
    p->y0 = y0;
    p->w0 = w0;
    *p2p_ok = p->c.nqp <= P2P_QMAX;
    return PF_OK;
}

int plan_level(const Plan *p) { return p->c.L; }

size_t plan_scratch(const Plan *p, int64_t ns, int64_t nt, bool same) {
    return fmm_scratch_bytes(p->c, ns, nt, same);
}

int64_t plan_groups(const Plan *p, int64_t nt) {
    return p2p_groups_expected((int64_t)1 << (2 * (p->c.L - p->c.kb)), nt);
}

pf_status plan_exec(const Plan *p, Bump &sc, int64_t ns, const double *x, const double *y,
                    const double *g, int64_t nt, const double *xt, const double *yt,
                    double ksigmasqr, double *vx, double *vy, int num_sms, int64_t groups_beside,
                    unsigned long long *ctr, cudaEvent_t *ev, cudaStream_t st) {
    FmmArgs a{ns, nt, x, y, g, xt, yt, ksigmasqr, 0.0, 0.0, 0, vx, vy, num_sms, groups_beside};
    return fmm_exec(p->c, p->x0, p->y0, p->w0, sc, a, ctr, ev, nullptr, st);
}

void tuning_get(int *leaf_level, int *np, int *kb) {
    *leaf_level = g_tune.leaf_level;
    *np = g_tune.np;
    *kb = g_tune.kb;
}

void tuning_set(int leaf_level, int np, int kb) {
    g_tune.leaf_level = leaf_level;
    g_tune.np = np;
    g_tune.kb = kb;
}

int auto_level(int64_t ns, int ndirect) {
    if (ndirect < 1) ndirect = 1;
    int L = (int)std::ceil(0.5 * std::log2((double)ns / (double)ndirect));
    return std::min(std::max(L, 0), MAX_LEVEL);
}

}  // namespace fmmx
}  // namespace pf
