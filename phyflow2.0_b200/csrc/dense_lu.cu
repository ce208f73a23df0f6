// dense_lu.cu -- LU factorisation with partial pivoting and the matching
// solve, FP64, for the panel system A gamma = RHS.
//
// The reference factorises the panel influence matrix once per geometry with
// scipy.linalg.lu_factor and solves every step with lu_solve
// (src/python/panels/__panelsClass.py:782, :960-962).  Here the matrix stays
// on the device: blocked right-looking LU, two launches per panel of columns:
//   k_lu_panel_reg : one CTA factorises the panel with row pivoting (ties to
//                    the smallest row), its rows in registers;
//   k_lu_stripe    : one CTA per stripe of the other columns: the panel's row
//                    exchanges, U12 by forward substitution, and
//                    A22 -= L21 U12 on the FP64 tensor cores (mma.sync m8n8k4).
// Row-major storage; ipiv[k] is the row exchanged with row k at step k.  No
// device-side waits between CTAs and no scratch: the stripes find the row
// moves from ipiv.
//
// What bounds it: the serial chain of m pivot steps (one CTA, 0.75-0.97 us each
// at 256-512 rows) and two launches per panel, not flops or bytes.
// Measured (B200, m = 512): the panels 2758 -> 441 us, the other columns 653 ->
// 105 us (before: panel in global memory, one thread per column for U12, FP64
// tiles on the CUDA cores).
#include "pf_common.cuh"

#include <algorithm>
#include <atomic>

namespace {

constexpr int LU_THREADS = 256;   // k_lu_panel (panels too tall for registers)
constexpr int LU_NB_MAX = 32;     // widest panel
constexpr int LS_THREADS = 512;   // stripe CTA
constexpr int LV_ROW_WARPS = 16;  // solve CTA: warps for the rows ..
constexpr int LV_THREADS = 32 * (LV_ROW_WARPS + 1);  // .. and one for the triangles
constexpr int LV_PRE = 6;         // row passes (64 rows each) loaded before they are needed
constexpr int64_t LV_SMEM_MAX = 8192;  // right-hand sides kept in shared memory

// Factorise columns [j0, j0+nb) of the row-major m x m matrix, rows j0 .. m-1,
// at most R T of them: thread t holds the unfinished columns of rows t, t + T,
// .. of the panel in registers, staged through shared memory so that the
// global accesses are whole rows.  Per column: each warp finds its largest |a|
// (high words by __reduce_max_sync, low words if two lanes share that); every
// thread picks the winner among the warps; its owner and that of row k put
// their rows in shared memory; the two change places and every later row is
// scaled and updated.  Two barriers per column (with every warp's candidate
// row written before one barrier, those writes alone took 300-600 cycles).
// The pivot column is always register 0: the update writes column c to
// register c - 1, and finished entries (L, the rows of U) go to shared memory.
// So the column loop is a loop, of PW columns for each number W of registers
// still in use.  Unrolled over all columns, each column ran once through
// fresh instructions, 1.1-1.4 us a column; a panel in global memory took 5.4.
constexpr int PW = 8;

__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int NB, int R, int T, int W>
__device__ __forceinline__ void panel_columns(double (&a)[R][NB], int k0, int nb, int rows, int j0,
                                              double *__restrict__ s_a,
                                              double (*s_row)[2][NB], double *s_rd, int (*s_hi)[T / 32],
                                              unsigned (*s_lo)[T / 32], int (*s_best)[T / 32],
                                              int32_t *__restrict__ ipiv,
                                              int32_t *__restrict__ info) {
    constexpr int NW = T / 32, LD = NB + 1;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int k1 = min(k0 + PW, nb);
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
        const int buf = k & 1;
        // this thread's largest |a| (its first on ties); NaN is never chosen
        int hi = -1, row = 0x7fffffff;
        unsigned lo = 0;
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int r = threadIdx.x + q * T;
            const long long b = __double_as_longlong(fabs(a[q][0]));
            const int h = (int)(b >> 32);
            const unsigned l = (unsigned)b;
            if (r >= k && r < rows && a[q][0] == a[q][0] && (h > hi || (h == hi && l > lo))) {
                hi = h;
                lo = l;
                row = r;
            }
        }
        // the warp's, the smallest row on ties (rarely needed: one lane has the
        // largest high word)
        const int wh = __reduce_max_sync(0xffffffffu, hi);
        unsigned best = __ballot_sync(0xffffffffu, hi == wh);
        int wr;
        unsigned wl;
        if (__popc(best) == 1) {
            wr = __shfl_sync(0xffffffffu, row, __ffs(best) - 1);
            wl = __shfl_sync(0xffffffffu, lo, __ffs(best) - 1);
        } else {
            wl = __reduce_max_sync(0xffffffffu, hi == wh ? lo : 0u);
            wr = __reduce_min_sync(0xffffffffu, hi == wh && lo == wl ? row : 0x7fffffff);
        }
        if (lane == 0) {
            s_hi[buf][wid] = wh;
            s_lo[buf][wid] = wl;
            s_best[buf][wid] = wr;
        }
        __syncthreads();
        // the winner among the warps, found by every warp alike
        const int gh = lane < NW ? s_hi[buf][lane] : -1;
        const int gr = lane < NW ? s_best[buf][lane] : 0x7fffffff;
        const int mh = __reduce_max_sync(0xffffffffu, gh);
        best = __ballot_sync(0xffffffffu, gh == mh);
        int p;
        if (__popc(best) == 1) {
            p = __shfl_sync(0xffffffffu, gr, __ffs(best) - 1);
        } else {
            const unsigned gl = lane < NW ? s_lo[buf][lane] : 0u;
            const unsigned ml = __reduce_max_sync(0xffffffffu, gh == mh ? gl : 0u);
            p = __reduce_min_sync(0xffffffffu, gh == mh && gl == ml ? gr : 0x7fffffff);
        }
        if (mh < 0) p = k;  // every candidate is NaN: row k stays
        // its owner puts the row in shared memory, with the reciprocal of the
        // pivot; so does the owner of row k
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int r = threadIdx.x + q * T;
            if (r == p || r == k) {
                if (r == p) s_rd[buf] = 1.0 / a[q][0];
                double2 *dst = reinterpret_cast<double2 *>(s_row[buf][r == p ? 0 : 1]);
#pragma unroll
                for (int c = 0; c < W / 2; ++c) dst[c] = make_double2(a[q][2 * c], a[q][2 * c + 1]);
            }
        }
        __syncthreads();
        const double *pr = s_row[buf][0];
        const double d = pr[0], rd = s_rd[buf];
        if (threadIdx.x == 0) {
            ipiv[j0 + k] = j0 + p;
            if (d == 0.0 && *info == 0) *info = j0 + k + 1;
        }
        if (wid == NW - 1) {  // finished entries: row k of U, and the rows' L parts change places
            if (lane < W && k + lane < NB) s_a[k * LD + k + lane] = pr[lane];
            if (p != k && lane < k) {
                const double t = s_a[k * LD + lane];
                s_a[k * LD + lane] = s_a[p * LD + lane];
                s_a[p * LD + lane] = t;
            }
        }
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int r = threadIdx.x + q * T;
            if (p != k && r == p)  // takes over row k
#pragma unroll
                for (int c = 0; c < W; ++c) a[q][c] = s_row[buf][1][c];
        }
        __syncwarp();
        // l = a / d: from the reciprocal with one correction (|a| <= |d|, so q is
        // at most 1 and the residual is exact), or divided where d is near the
        // ends of the range, zero or not finite
        const bool mid = fabs(d) > 1e-200 && fabs(d) < 1e200;
        double l[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int r = threadIdx.x + q * T;
            if (mid) {
                const double t = a[q][0] * rd;
                l[q] = fma(fma(-t, d, a[q][0]), rd, t);
            } else {
                l[q] = d != 0.0 ? a[q][0] / d : a[q][0];
            }
            if (r > k && r < rows) s_a[r * LD + k] = l[q];
        }
        const double2 *pr2 = reinterpret_cast<const double2 *>(pr);
#pragma unroll
        for (int c = 0; c < W / 2; ++c) {
            const double2 u = pr2[c];
#pragma unroll
            for (int q = 0; q < R; ++q) {
                if (c > 0) a[q][2 * c - 1] = fma(-l[q], u.x, a[q][2 * c]);
                a[q][2 * c] = fma(-l[q], u.y, a[q][2 * c + 1]);
            }
        }
    }
}

template <int NB, int R, int T>
__global__ void __launch_bounds__(T)
k_lu_panel_reg(int64_t m, int j0, int nb, double *__restrict__ A, int32_t *__restrict__ ipiv,
               int32_t *__restrict__ info) {
    constexpr int NW = T / 32, LD = NB + 1;
    extern __shared__ __align__(16) double s_a[];  // [R T][LD]
    __shared__ __align__(16) double s_row[2][2][NB];  // the pivot row, row k
    __shared__ double s_rd[2];
    __shared__ int s_hi[2][NW], s_best[2][NW];
    __shared__ unsigned s_lo[2][NW];
    static_assert(NB % PW == 0 && NB <= 4 * PW && NW <= 32, "register counts of panel_columns");
    const int rows = (int)(m - j0);
    // whole rows, asynchronous 8-byte copies: every load is in flight at once
#pragma unroll 4
    for (int q = 0; q < R * NB; ++q) {
        const int e = threadIdx.x + q * T;
        const int r = e / NB, c = e % NB;
        if (r < rows && c < nb)
            cp_async8(&s_a[r * LD + c], &A[(int64_t)(j0 + r) * m + j0 + c]);
        else
            s_a[r * LD + c] = 0.0;
    }
    cp_async_wait_all();
    __syncthreads();
    double a[R][NB];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int r = threadIdx.x + q * T;
#pragma unroll
        for (int c = 0; c < NB; ++c) a[q][c] = r < rows ? s_a[r * LD + c] : 0.0;
    }
    __syncthreads();
#define PF_LU_COLUMNS(W)                                                                     \
    if constexpr (NB >= (W))                                                                 \
        panel_columns<NB, R, T, (W)>(a, NB - (W), nb, rows, j0, s_a, s_row, s_rd, s_hi, s_lo, \
                                     s_best, ipiv, info);
    PF_LU_COLUMNS(32)
    PF_LU_COLUMNS(24)
    PF_LU_COLUMNS(16)
    PF_LU_COLUMNS(8)
#undef PF_LU_COLUMNS
    __syncthreads();
#pragma unroll 8
    for (int q = 0; q < R * NB; ++q) {
        const int e = threadIdx.x + q * T;
        const int r = e / NB, c = e % NB;
        if (r < rows && c < nb) A[(int64_t)(j0 + r) * m + j0 + c] = s_a[r * LD + c];
    }
}

// The same panel in global memory, for panels of more than 2048 rows.
__global__ void __launch_bounds__(LU_THREADS)
k_lu_panel(int64_t m, int j0, int nb, double *__restrict__ A, int32_t *__restrict__ ipiv,
           int32_t *__restrict__ info) {
    __shared__ double s_v[LU_THREADS];
    __shared__ int s_i[LU_THREADS];
    for (int k = j0; k < j0 + nb; ++k) {
        // pivot: max |A[r][k]| over r >= k, smallest r on ties
        double best = -1.0;
        int bi = k;
        for (int64_t r = k + threadIdx.x; r < m; r += LU_THREADS) {
            const double v = fabs(A[r * m + k]);
            if (v > best) {
                best = v;
                bi = (int)r;
            }
        }
        s_v[threadIdx.x] = best;
        s_i[threadIdx.x] = bi;
        __syncthreads();
        for (int s = LU_THREADS / 2; s > 0; s >>= 1) {
            if (threadIdx.x < s) {
                const double a = s_v[threadIdx.x], b = s_v[threadIdx.x + s];
                const int ia = s_i[threadIdx.x], ib = s_i[threadIdx.x + s];
                if (b > a || (b == a && ib < ia)) {
                    s_v[threadIdx.x] = b;
                    s_i[threadIdx.x] = ib;
                }
            }
            __syncthreads();
        }
        const int p = s_i[0];
        if (threadIdx.x == 0) {
            ipiv[k] = p;
            if (A[(int64_t)p * m + k] == 0.0 && *info == 0) *info = k + 1;
        }
        if (p != k && threadIdx.x < nb) {  // the panel's columns; the stripes swap the others
            const int64_t c = j0 + threadIdx.x;
            const double t = A[(int64_t)k * m + c];
            A[(int64_t)k * m + c] = A[(int64_t)p * m + c];
            A[(int64_t)p * m + c] = t;
        }
        __syncthreads();
        const double d = A[(int64_t)k * m + k];
        if (d != 0.0)
            for (int64_t r = k + 1 + threadIdx.x; r < m; r += LU_THREADS) A[r * m + k] /= d;
        __syncthreads();
        // rank-1 update of the remaining panel columns
        const int nc = j0 + nb - (k + 1);
        if (nc > 0)
            for (int64_t e = threadIdx.x; e < (m - k - 1) * nc; e += LU_THREADS) {
                const int64_t r = k + 1 + e / nc;
                const int c = k + 1 + (int)(e % nc);
                A[r * m + c] -= A[r * m + k] * A[(int64_t)k * m + c];
            }
        __syncthreads();
    }
}

// d = a b + d of an 8 x 4 by 4 x 8 FP64 tile: a = A[lane/4][lane%4], b =
// B[lane%4][lane/4], (d0, d1) = D[lane/4][2 (lane%4) + 0, 1].
__device__ __forceinline__ void mma_f64(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// The row moves of the panel's exchanges j0 + k <-> ipiv[j0 + k], k < nb, as
// (destination, source) pairs, found by one warp: lane i follows the row at
// position j0 + i and, when step i is the first to name a row below the panel
// rows, the row at that position.  At most 2 nb pairs; returns their number.
__device__ __forceinline__ int lu_moves(int j0, int nb, const int32_t *__restrict__ ipiv,
                                        int *s_dst, int *s_src) {
    const int lane = threadIdx.x & 31;
    const int p = lane < nb ? ipiv[j0 + lane] : j0 + lane;
    if (!__any_sync(0xffffffffu, p != j0 + lane)) return 0;
    int cur = j0 + lane;          // row now at position j0 + lane
    int out = -1, outcur = -1;    // a position below the panel rows, and the row now there
    for (int k = 0; k < nb; ++k) {
        const int pk = __shfl_sync(0xffffffffu, p, k);
        if (pk == j0 + k) continue;
        const int ck = __shfl_sync(0xffffffffu, cur, k);
        if (pk < j0 + nb) {
            const int cp = __shfl_sync(0xffffffffu, cur, pk - j0);
            if (lane == k) cur = cp;
            if (lane == pk - j0) cur = ck;
        } else {
            const unsigned has = __ballot_sync(0xffffffffu, out == pk);
            const int e = has ? __ffs(has) - 1 : k;
            if (!has && lane == k) {
                out = pk;
                outcur = pk;
            }
            const int cp = __shfl_sync(0xffffffffu, outcur, e);
            if (lane == k) cur = cp;
            if (lane == e) outcur = ck;
        }
    }
    const unsigned lt = (1u << lane) - 1u;
    const unsigned m1 = __ballot_sync(0xffffffffu, lane < nb && cur != j0 + lane);
    if (m1 >> lane & 1u) {
        s_dst[__popc(m1 & lt)] = j0 + lane;
        s_src[__popc(m1 & lt)] = cur;
    }
    const unsigned m2 = __ballot_sync(0xffffffffu, out >= 0 && outcur != out);
    if (m2 >> lane & 1u) {
        s_dst[__popc(m1) + __popc(m2 & lt)] = out;
        s_src[__popc(m1) + __popc(m2 & lt)] = outcur;
    }
    return __popc(m1) + __popc(m2);
}

// One stripe of 8 NT columns outside the panel [j0, j0+nb): the panel's row
// exchanges; right of the panel also U12 (one warp per column: lane i holds
// row i, forward substitution with the unit lower block) and A22 -= L21 U12.
// The update keeps U12 as B fragments in registers and reads L21 as A
// fragments straight from global memory (8 rows x 32 bytes a load, every
// sector used whole), 8 rows x 8 NT columns per warp and iteration, two
// iterations' loads in flight.  A stripe owns its columns, so the row
// exchanges need no other launch; narrow stripes (NT = 1) give a 512-column
// matrix 60 CTAs, wide ones (NT = 4) reread L21 less often where the columns
// alone fill the device.
template <int NB, int NT>
__global__ void __launch_bounds__(LS_THREADS)
k_lu_stripe(int64_t m, int j0, int nb, double *__restrict__ A, const int32_t *__restrict__ ipiv) {
    constexpr int CW = 8 * NT, KS = NB / 4, NWARP = LS_THREADS / 32;
    constexpr int MV = (2 * LU_NB_MAX * CW + LS_THREADS - 1) / LS_THREADS;
    __shared__ int s_dst[2 * LU_NB_MAX], s_src[2 * LU_NB_MAX];
    __shared__ int s_n;
    __shared__ double s_l[NB][NB + 1];
    __shared__ double s_u[NB][CW + 1];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t c0 = (int64_t)blockIdx.x * CW;
    const int64_t j1 = (int64_t)j0 + nb;
    if (wid == 0) {
        const int n = lu_moves(j0, nb, ipiv, s_dst, s_src);
        if (lane == 0) s_n = n;
    }
    const bool right = c0 + CW > j1;  // some column right of the panel
    if (right)
        for (int e = threadIdx.x; e < NB * NB; e += LS_THREADS) {
            const int r = e / NB, c = e % NB;
            s_l[r][c] = (r < nb && c < nb) ? A[(int64_t)(j0 + r) * m + j0 + c] : 0.0;
        }
    __syncthreads();
    const int nmv = s_n;
    if (nmv > 0) {
        double v[MV];
#pragma unroll
        for (int q = 0; q < MV; ++q) {
            const int e = threadIdx.x + q * LS_THREADS;
            const int64_t c = c0 + e % CW;
            if (e < nmv * CW && c < m && (c < j0 || c >= j1)) v[q] = A[(int64_t)s_src[e / CW] * m + c];
        }
        __syncthreads();  // every source is read before a destination is written
#pragma unroll
        for (int q = 0; q < MV; ++q) {
            const int e = threadIdx.x + q * LS_THREADS;
            const int64_t c = c0 + e % CW;
            if (e < nmv * CW && c < m && (c < j0 || c >= j1)) A[(int64_t)s_dst[e / CW] * m + c] = v[q];
        }
        __syncthreads();
    }
    if (!right) return;  // the whole CTA
    for (int e = threadIdx.x; e < NB * CW; e += LS_THREADS) {
        const int r = e / CW;
        const int64_t c = c0 + e % CW;
        s_u[r][e % CW] = (r < nb && c < m && c >= j1) ? A[(int64_t)(j0 + r) * m + c] : 0.0;
    }
    __syncthreads();
    for (int c = wid; c < CW; c += NWARP) {
        double b = lane < NB ? s_u[lane][c] : 0.0;
#pragma unroll 4
        for (int k = 0; k < NB - 1; ++k) {
            const double bk = __shfl_sync(0xffffffffu, b, k);
            if (lane > k && lane < NB) b = fma(-s_l[lane][k], bk, b);
        }
        if (lane < nb) {
            s_u[lane][c] = b;
            if (c0 + c >= j1 && c0 + c < m) A[(int64_t)(j0 + lane) * m + c0 + c] = b;
        }
    }
    __syncthreads();
    double bf[NT][KS];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int s = 0; s < KS; ++s) bf[t][s] = s_u[4 * s + (lane & 3)][8 * t + (lane >> 2)];
    const int rq = lane >> 2, kq = lane & 3;
    for (int64_t r0 = j1 + 8 * wid; r0 < m; r0 += 2 * 8 * NWARP) {
        double af[2][KS];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t r = r0 + h * 8 * NWARP + rq;
#pragma unroll
            for (int s = 0; s < KS; ++s)
                af[h][s] = (r < m && 4 * s + kq < nb) ? A[r * m + j0 + 4 * s + kq] : 0.0;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t r = r0 + h * 8 * NWARP + rq;
            double2 old[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const int64_t c = c0 + 8 * t + 2 * kq;
                old[t].x = (r < m && c < m && c >= j1) ? A[r * m + c] : 0.0;
                old[t].y = (r < m && c + 1 < m && c + 1 >= j1) ? A[r * m + c + 1] : 0.0;
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                double d0 = 0.0, d1 = 0.0;
#pragma unroll
                for (int s = 0; s < KS; ++s) mma_f64(d0, d1, af[h][s], bf[t][s]);
                const int64_t c = c0 + 8 * t + 2 * kq;
                if (r < m && c < m && c >= j1) A[r * m + c] = old[t].x - d0;
                if (r < m && c + 1 < m && c + 1 >= j1) A[r * m + c + 1] = old[t].y - d1;
            }
        }
    }
}

// Back substitution of one block with a division per unknown, for blocks whose
// rows can't be divided by their diagonals first.  v, d: right-hand side and
// diagonal of the lane's row; t: the block's entries of U, negated.  (Out of line
// and with the entries in shared memory: inlined, or reading U again, the rarely
// taken path costs the usual one 6% by register allocation.)
__device__ __noinline__ double back_unscaled(double v, double d, const double (*t)[33]) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int k = 31; k >= 0; --k) {
        if (lane == k) v = v / d;
        const double xk = __shfl_sync(0xffffffffu, v, k);
        if (lane < k) v = fma(t[lane][k], xk, v);
    }
    return v;
}

// One substitution (BACK: with U from the last block up, else with the unit
// lower L from the first down) of k_lu_solve, by blocks of 32 unknowns.
//   s_t[buf]: the block's triangle, negated, zero elsewhere (BACK: each row
//     divided by its diagonal, which keeps the division out of the chain);
//   s_u[buf]: BACK: the triangle as it is.  The scaled one holds while every
//     quotient of the block is a normal number.  A block with another one or with
//     a diagonal that is zero or not finite (s_raw), and one whose scaled solution
//     is not finite (its right-hand side may overflow when it is divided before
//     the others' shares are taken off), is solved from s_u, unknown by unknown;
//   thread (wid, rq, cq) of the CTA works on columns cq + 8 q of rows
//     64 i + 4 wid + rq: the first LV_PRE row passes' factors are loaded
//     while another warp solves the triangle, and their products with the
//     solved unknowns are summed per thread until the row's own block comes.
template <bool BACK>
__device__ __forceinline__ void lu_substitute(int64_t m, const double *__restrict__ LU,
                                              double *b, double (*s_t)[32][33],
                                              double (*s_u)[32][33], double (*s_d)[32], int *s_raw, double *s_x) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    static_assert(LV_ROW_WARPS == 16, "two rows of a triangle per warp, 64 rows per pass");
    const bool solver = wid == LV_ROW_WARPS;  // the triangles' warp
    const int64_t nblk = (m + 31) / 32;
    const int rq = lane >> 3, cq = lane & 7, row0 = 4 * wid + rq;
    // rows wid and wid + 16 of block jb's triangle
    auto load_tri = [&](int64_t jb, double (&e)[2], double (&dg)[2]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t r = jb * 32 + wid + 16 * h, c = jb * 32 + lane;
            const bool in = jb >= 0 && jb < nblk && r < m;
            e[h] = in && c < m && (BACK ? c > r : c < r) ? -LU[r * m + c] : 0.0;
            dg[h] = BACK && in ? LU[r * m + r] : 1.0;
        }
    };
    auto store_tri = [&](int buf, const double (&e)[2], const double (&dg)[2]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int w = wid + 16 * h;
            double v = e[h];
            if (BACK) {
                // (zeros divide d by itself: a zero would take the division's slow path)
                const double sc = (v != 0.0 ? v : dg[h]) / dg[h];
                const unsigned ex = __double2hiint(sc) >> 20 & 0x7ff;
                const bool ok = ex - 1u < 0x7feu;  // a normal number
                if (!__all_sync(0xffffffffu, ok) && lane == 0) s_raw[buf] = 1;  // any writer: the same
                s_u[buf][w][lane] = v;
                v = v != 0.0 ? sc : 0.0;
                __syncwarp();
                if (lane == 0) s_d[buf][w] = dg[h];
            }
            s_t[buf][w][lane] = v;
        }
    };
    double acc[LV_PRE];
#pragma unroll
    for (int i = 0; i < LV_PRE; ++i) acc[i] = 0.0;
    const int64_t first = BACK ? nblk - 1 : 0;
    double e[2], dg[2];
    if (threadIdx.x < 2) s_raw[threadIdx.x] = 0;
    __syncthreads();
    if (!solver) {
        load_tri(first, e, dg);
        store_tri(0, e, dg);
    }
    for (int64_t st = 0; st < nblk; ++st) {
        const int64_t jb = BACK ? nblk - 1 - st : st;
        const int64_t j0 = jb * 32;
        const int buf = (int)(st & 1);
        // rows still to come: r >= lo (forward), r < hi (back)
        const int64_t lo = BACK ? 0 : j0 + 32, hi = BACK ? j0 : m;
        // this block's rows: their sums so far (picked by masks: indexing
        // would put the sums in local memory)
        if (!solver) {
            long long tb = 0;
#pragma unroll
            for (int i = 0; i < LV_PRE; ++i)
                tb |= __double_as_longlong(acc[i]) & -(long long)(i == (int)(j0 / 64));
            double t = __longlong_as_double(tb);
            const int64_t r = (j0 / 64) * 64 + row0;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (j0 / 64 < LV_PRE && cq == 0 && r >= j0 && r < j0 + 32 && r < m) b[r] -= t;
        } else if (lane == 0) {
            s_raw[buf ^ 1] = 0;
        }
        __syncthreads();
        double lu[LV_PRE][4];
        if (solver) {
            const bool in = j0 + lane < m;
            double v = in ? b[j0 + lane] : 0.0;
            if (BACK) {
                bool raw = s_raw[buf] != 0;
                if (!raw) {
                    v = v / s_d[buf][lane];
#pragma unroll
                    for (int k = 31; k > 0; --k)
                        v = fma(s_t[buf][lane][k], __shfl_sync(0xffffffffu, v, k), v);
                    raw = __any_sync(0xffffffffu, (__double2hiint(v) >> 20 & 0x7ff) == 0x7ff);
                }
                if (raw) v = back_unscaled(in ? b[j0 + lane] : 0.0, s_d[buf][lane], s_u[buf]);
            } else {
#pragma unroll
                for (int k = 0; k < 31; ++k)
                    v = fma(s_t[buf][lane][k], __shfl_sync(0xffffffffu, v, k), v);
            }
            if (in) b[j0 + lane] = v;
            s_x[lane] = in ? v : 0.0;
        } else {  // meanwhile the rows' factors and the next triangle
            load_tri(BACK ? jb - 1 : jb + 1, e, dg);
            const double *lp = LU + (int64_t)row0 * m + j0 + cq;
#pragma unroll
            for (int i = 0; i < LV_PRE; ++i) {
                const int64_t r = row0 + 64 * i;
                const bool in = r >= lo && r < hi;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    lu[i][q] = (in && j0 + cq + 8 * q < m) ? lp[(int64_t)(64 * i) * m + 8 * q] : 0.0;
            }
            store_tri(buf ^ 1, e, dg);
        }
        __syncthreads();
        if (solver) continue;
        double xv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) xv[q] = s_x[cq + 8 * q];
#pragma unroll
        for (int i = 0; i < LV_PRE; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i] = fma(lu[i][q], xv[q], acc[i]);
        // rows beyond the passes above
        for (int64_t r0 = 64 * LV_PRE; r0 < hi; r0 += 64) {
            const int64_t r = r0 + row0;
            const bool in = r >= lo && r < hi;
            double t = 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (in && j0 + cq + 8 * q < m) t = fma(LU[r * m + j0 + cq + 8 * q], xv[q], t);
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (cq == 0 && in) b[r] -= t;
        }
    }
    __syncthreads();
}

// x = A^-1 b from the factors, one CTA: the row exchanges, then forward and
// back substitution by blocks of 32 unknowns.  A block's triangle is solved by
// one warp (lane i holds unknown i; one shuffle and one FMA per unknown), then
// every other warp adds the block's products to its rows' sums, eight lanes per row
// reading 64-byte pieces.  b is worked on in shared memory (SM) or, above
// LV_SMEM_MAX unknowns, in place.
// What bounds it: the chain of 2 m/32 triangles, 31 x 36 cycles each; the
// factors are read once.  Column-wise updates with one thread per row, a
// strided 8-byte read each, took 482 us at 512 unknowns and 122 at 200; this
// takes 82 and 29.
template <bool SM>
__global__ void __launch_bounds__(LV_THREADS)
k_lu_solve(int64_t m, const double *__restrict__ LU, const int32_t *__restrict__ ipiv,
           double *bg) {
    extern __shared__ __align__(16) double s_b[];
    __shared__ double s_t[2][32][33], s_u[2][32][33];
    __shared__ double s_d[2][32], s_x[32];
    __shared__ int s_raw[2];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double *const b = SM ? s_b : bg;
    if (SM)
        for (int64_t i = threadIdx.x; i < m; i += LV_THREADS) s_b[i] = bg[i];
    // row exchanges: the warps look for any, one warp makes them in order
    bool moves = false;
    for (int64_t k = threadIdx.x; k < m; k += LV_THREADS) moves |= ipiv[k] != k;
    if (__syncthreads_or(moves)) {
        if (wid == 0) {
            for (int64_t k0 = 0; k0 < m; k0 += 32) {
                const int64_t k = k0 + lane;
                const int64_t p = k < m ? ipiv[k] : 0;
                unsigned todo = __ballot_sync(0xffffffffu, k < m && p != k && p >= 0 && p < m);
                while (todo) {
                    const int j = __ffs(todo) - 1;
                    todo &= todo - 1;
                    if (lane == j) {
                        const double t = b[k];
                        b[k] = b[p];
                        b[p] = t;
                    }
                    __syncwarp();
                }
            }
        }
        __syncthreads();
    }
    lu_substitute<false>(m, LU, b, s_t, s_u, s_d, s_raw, s_x);
    lu_substitute<true>(m, LU, b, s_t, s_u, s_d, s_raw, s_x);
    if (SM)
        for (int64_t i = threadIdx.x; i < m; i += LV_THREADS) bg[i] = s_b[i];
}

// Dynamic shared memory above the 48 KB default, set once per device and kernel.
template <class K>
cudaError_t lu_smem(K kernel, std::atomic<unsigned long long> &done, size_t bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && bit) done.fetch_or(bit, std::memory_order_acq_rel);
    return e;
}

template <int NB, int R, int T>
pf_status launch_panel_reg(int64_t m, int64_t j0, int nb, double *a, int32_t *ipiv, int32_t *info,
                           cudaStream_t st) {
    static std::atomic<unsigned long long> done{0};
    constexpr size_t bytes = sizeof(double) * R * T * (NB + 1);
    PF_CUDA_TRY(lu_smem(k_lu_panel_reg<NB, R, T>, done, bytes));
    k_lu_panel_reg<NB, R, T><<<1, T, bytes, st>>>(m, (int)j0, nb, a, ipiv, info);
    return pf::launch_status("k_lu_panel_reg");
}

template <int NB>
pf_status launch_stripes(int64_t m, int64_t j0, int nb, double *a, const int32_t *ipiv,
                         cudaStream_t st) {
    // 32-column stripes once they alone fill the device
    if (m > 4096)
        k_lu_stripe<NB, 4><<<(unsigned)pf::ceil_div(m, 32), LS_THREADS, 0, st>>>(m, (int)j0, nb, a,
                                                                                 ipiv);
    else
        k_lu_stripe<NB, 1><<<(unsigned)pf::ceil_div(m, 8), LS_THREADS, 0, st>>>(m, (int)j0, nb, a,
                                                                                ipiv);
    return pf::launch_status("k_lu_stripe");
}

}  // namespace

extern "C" pf_status pf_dense_lu_factor(pf_ctx *ctx, int64_t m, double *a, int32_t *ipiv,
                                        int32_t *info_dev, void *stream) {
    PF_RANGE("pf_dense_lu_factor");
    pf::clear_error();
    PF_CHECK_ARG(ctx != nullptr, "pf_dense_lu_factor: NULL context");
    PF_CHECK_ARG(m >= 0 && m <= 32768, "pf_dense_lu_factor: m = %lld outside [0, 32768]",
                 (long long)m);
    PF_CHECK_ARG(m == 0 || (a && ipiv && info_dev), "pf_dense_lu_factor: NULL array");
    pf::DeviceGuard dg(ctx->device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (m == 0) return PF_OK;
    PF_CUDA_TRY(cudaMemsetAsync(info_dev, 0, sizeof(int32_t), st));
    // panel width and rows per thread by the rows left: as many columns per
    // panel (fewer launches) as the register file holds rows for
    for (int64_t j0 = 0; j0 < m;) {
        const int64_t rows = m - j0;
        const int nb = (int)std::min<int64_t>(rows > 1024 && rows <= 2048 ? 8
                                              : rows > 512 && rows <= 1024 ? 16
                                                                           : 32,
                                              rows);
        if (rows <= 256) {
            PF_TRY((launch_panel_reg<32, 1, 256>(m, j0, nb, a, ipiv, info_dev, st)));
        } else if (rows <= 512) {
            PF_TRY((launch_panel_reg<32, 2, 256>(m, j0, nb, a, ipiv, info_dev, st)));
        } else if (rows <= 1024) {
            PF_TRY((launch_panel_reg<16, 1, 1024>(m, j0, nb, a, ipiv, info_dev, st)));
        } else if (rows <= 2048) {
            PF_TRY((launch_panel_reg<8, 2, 1024>(m, j0, nb, a, ipiv, info_dev, st)));
        } else {
            k_lu_panel<<<1, LU_THREADS, 0, st>>>(m, (int)j0, nb, a, ipiv, info_dev);
            PF_TRY(pf::launch_status("k_lu_panel"));
        }
        if (m > nb) {
            if (nb > 16)
                PF_TRY(launch_stripes<32>(m, j0, nb, a, ipiv, st));
            else if (nb > 8)
                PF_TRY(launch_stripes<16>(m, j0, nb, a, ipiv, st));
            else
                PF_TRY(launch_stripes<8>(m, j0, nb, a, ipiv, st));
        }
        j0 += nb;
    }
    return PF_OK;
}

extern "C" pf_status pf_dense_lu_solve(pf_ctx *ctx, int64_t m, const double *lu,
                                       const int32_t *ipiv, double *b, void *stream) {
    PF_RANGE("pf_dense_lu_solve");
    pf::clear_error();
    PF_CHECK_ARG(ctx != nullptr, "pf_dense_lu_solve: NULL context");
    PF_CHECK_ARG(m >= 0 && m <= 32768, "pf_dense_lu_solve: m = %lld outside [0, 32768]",
                 (long long)m);
    PF_CHECK_ARG(m == 0 || (lu && ipiv && b), "pf_dense_lu_solve: NULL array");
    pf::DeviceGuard dg(ctx->device);
    if (m == 0) return PF_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (m <= LV_SMEM_MAX) {
        static std::atomic<unsigned long long> done{0};
        PF_CUDA_TRY(lu_smem(k_lu_solve<true>, done, sizeof(double) * LV_SMEM_MAX));
        k_lu_solve<true><<<1, LV_THREADS, sizeof(double) * (size_t)m, st>>>(m, lu, ipiv, b);
    } else {
        k_lu_solve<false><<<1, LV_THREADS, 0, st>>>(m, lu, ipiv, b);
    }
    return pf::launch_status("k_lu_solve");
}
