// p2p.cuh -- device code of the FMM near field (P2P), shared by the one-warp
// kernel (fmm.cu) and the kernel of several warps per target group
// (p2p_multi.cu).  The two kernels are separate translation units: the chunk
// functions below are calls, and with both kernels in one unit the compiler
// built them for both at once, which cost the one-warp kernel 7%.
#pragma once
#include "fmm_api.cuh"
#include "gauss_pair.cuh"

namespace {

using pf::fmmx::P2PDesc;

constexpr double P2P_INV_2PI = 0.15915494309189535;
constexpr int P2P_RUNS_SM = 64;  // runs staged in shared memory at a time
constexpr int P2P_BUF = 64;      // sources per warp buffer (three buffers)
// unroll of the pair loop over a full chunk: the kernel holds nine copies of
// it (targets per lane x mode), which must stay within the instruction cache
constexpr int P2P_UNROLL = 8;
constexpr int P2P_MIN_CTAS = 20; // one-warp CTAs resident per SM: 96 registers each
constexpr int P2P_GROUP = 96;    // most targets per group

// P2P near field: the targets of a P2P block in balanced groups of at most 96,
// one warp (one CTA) per group.  Targets a and b of a lane run packed (f32x2); in a
// group of 65..96 the remaining targets are spread over the warp, each lane
// taking a share of the sources (p2p_split_sums).  Pair code modes, chosen
// per source from its box distance to the group's target box (with a
// rounding margin):
//   P2P_FAR:    sources beyond sqrt(r2_far): no ex2 (1 - exp(-x) rounds to
//               1.0f for every pair), one-float coordinates relative to the
//               group centre;
//   P2P_FULL:   the other sources beyond the series radius sqrt(r2_series):
//               no small-x check (every pair has r2 above r2_series);
//   P2P_SERIES: the sources within it: the pair code with the check.
// Full and series pairs give bitwise the value of the checked code.  The group's
// sources stream through three warp buffers, one per mode (each in stream
// order), and each buffer runs 32 sources at a time as it fills (the rest
// when the group's stream ends).
constexpr int P2P_FAR = 0, P2P_FULL = 1, P2P_SERIES = 2;

template <int MODE>
__device__ __forceinline__ void scalar_pair(const ulonglong2 &h, const ulonglong2 &l,
                                            unsigned long long g2, const float4 &t,
                                            const pfd::GaussParams &gp, float &px, float &py) {
    float sxh, syh, sxl, syl, g, dummy;
    pfd::unpack2(h.x, sxh, dummy);
    pfd::unpack2(h.y, syh, dummy);
    pfd::unpack2(l.x, sxl, dummy);
    pfd::unpack2(l.y, syl, dummy);
    pfd::unpack2(g2, g, dummy);
    const float dx = (t.x - sxh) + (t.z - sxl);
    const float dy = (t.y - syh) + (t.w - syl);
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, 1e-12f));
    const float sc = MODE == P2P_FAR ? g * pfd::rcp_approx(r2)
                                     : pfd::gauss_s<MODE == P2P_SERIES>(r2, g, gp);
    px = fmaf(-dy, sc, px);
    py = fmaf(dx, sc, py);
}

// One pair of the given mode for the lane's targets (NT per lane).
template <int NT, int MODE>
__device__ __forceinline__ void p2p_pair(const ulonglong2 &h, const ulonglong2 &l,
                                         unsigned long long g2, pfd::f32x2 txh, pfd::f32x2 tyh,
                                         pfd::f32x2 txl, pfd::f32x2 tyl, const float4 &ta,
                                         const float4 &tc, const pfd::GaussParams &gp,
                                         const pfd::GaussParams2 &gp2, pfd::f32x2 &nx,
                                         pfd::f32x2 &ny, float &pxa, float &pya, float &pxc,
                                         float &pyc) {
    if (NT >= 2) {
        if (MODE == P2P_FAR)
            pfd::pair2_far(h, l, g2, txh, tyh, txl, tyl, gp2, nx, ny);
        else
            pfd::pair2<MODE == P2P_SERIES>(h, l, g2, txh, tyh, txl, tyl, gp2, nx, ny);
    } else {
        scalar_pair<MODE>(h, l, g2, ta, gp, pxa, pya);
    }
    if (NT == 3) scalar_pair<MODE>(h, l, g2, tc, gp, pxc, pyc);
}

// Shared-memory loads by 32-bit shared address (the chunk functions below
// are separate calls, which see only generic pointers otherwise).
__device__ __forceinline__ ulonglong2 lds_u64x2(uint32_t a) {
    ulonglong2 v;
    asm("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ unsigned long long lds_u64(uint32_t a) {
    unsigned long long v;
    asm("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
}

struct P2PSums {
    float s[6];  // NT >= 2: -nx_a, ny_a, -nx_b, ny_b; NT = 1: px_a, py_a; NT = 3: px_c, py_c
};

// Sources [0, cnt) of a buffer (cnt <= 32) against the lane's targets; the
// partial sums are returned for one compensated fold by the caller.  Each
// (NT, MODE) is its own function, not inlined: nine inlined copies of the
// unrolled loop in one kernel measured about 20% more instructions (register
// copies between the copies' allocations) and instruction-cache stalls.
// (A per-source choice of the checked code inside a chunk, by a warp-uniform
// branch, measured slower too: the branch breaks the overlap of consecutive
// pairs.)
//
// P2P_FAR chunks hold coordinates relative to the group centre (cx, cy), one
// float each: {x - cx, x - cx, y - cy, y - cy} in the hi slot (pair2_far_local).
__device__ __forceinline__ void far_local_scalar(const ulonglong2 &loc, unsigned long long g2,
                                                 float tx, float ty, float &px, float &py) {
    float lx, ly, g, dummy;
    pfd::unpack2(loc.x, lx, dummy);
    pfd::unpack2(loc.y, ly, dummy);
    pfd::unpack2(g2, g, dummy);
    const float dx = tx - lx, dy = ty - ly;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, 1e-12f));
    const float sc = g * pfd::rcp_approx(r2);
    px = fmaf(-dy, sc, px);
    py = fmaf(dx, sc, py);
}

template <int NT, int MODE>
__device__ __noinline__ P2PSums p2p_chunk_sums(uint32_t a_hi, uint32_t a_lo, uint32_t a_g, int cnt,
                                               float4 ta, float4 tb, float4 tc, float cx,
                                               float cy, pfd::GaussParams gp) {
    const pfd::GaussParams2 gp2 = pfd::make_params2(gp);
    pfd::f32x2 nx = 0ull, ny = 0ull;  // +0.0f in both halves
    float pxa = 0.f, pya = 0.f, pxc = 0.f, pyc = 0.f;
    if constexpr (MODE == P2P_FAR) {
        const float axc = (ta.x - cx) + ta.z, ayc = (ta.y - cy) + ta.w;
        const pfd::f32x2 txc = pfd::pack2(axc, (tb.x - cx) + tb.z);
        const pfd::f32x2 tyc = pfd::pack2(ayc, (tb.y - cy) + tb.w);
        auto one = [&](int k) {
            const ulonglong2 loc = lds_u64x2(a_hi + 16 * k);
            const unsigned long long g2 = lds_u64(a_g + 8 * k);
            if (NT >= 2)
                pfd::pair2_far_local(loc, g2, txc, tyc, gp2, nx, ny);
            else
                far_local_scalar(loc, g2, axc, ayc, pxa, pya);
        };
        if (cnt == 32) {
#pragma unroll(P2P_UNROLL)
            for (int k = 0; k < 32; ++k) one(k);
        } else {
#pragma unroll 1
            for (int k = 0; k < cnt; ++k) one(k);
        }
    } else {
        const pfd::f32x2 txh = pfd::pack2(ta.x, tb.x), tyh = pfd::pack2(ta.y, tb.y);
        const pfd::f32x2 txl = pfd::pack2(ta.z, tb.z), tyl = pfd::pack2(ta.w, tb.w);
        if (cnt == 32) {  // full chunk (the common case)
#pragma unroll(P2P_UNROLL)
            for (int k = 0; k < 32; ++k)
                p2p_pair<NT, MODE>(lds_u64x2(a_hi + 16 * k), lds_u64x2(a_lo + 16 * k),
                                   lds_u64(a_g + 8 * k), txh, tyh, txl, tyl, ta, tc, gp, gp2, nx,
                                   ny, pxa, pya, pxc, pyc);
        } else {  // the rest of a buffer at the end of a group: kept small in code
#pragma unroll 1
            for (int k = 0; k < cnt; ++k)
                p2p_pair<NT, MODE>(lds_u64x2(a_hi + 16 * k), lds_u64x2(a_lo + 16 * k),
                                   lds_u64(a_g + 8 * k), txh, tyh, txl, tyl, ta, tc, gp, gp2, nx,
                                   ny, pxa, pya, pxc, pyc);
        }
    }
    P2PSums r;
    if (NT >= 2) {
        float nxa, nxb, nya, nyb;
        pfd::unpack2(nx, nxa, nxb);
        pfd::unpack2(ny, nya, nyb);
        r.s[0] = -nxa;
        r.s[1] = nya;
        r.s[2] = -nxb;
        r.s[3] = nyb;
    } else {
        r.s[0] = pxa;
        r.s[1] = pya;
        r.s[2] = r.s[3] = 0.f;
    }
    r.s[4] = pxc;
    r.s[5] = pyc;
    return r;
}

template <int NT, int MODE>
__device__ __forceinline__ void p2p_chunk(const ulonglong2 *shi, const ulonglong2 *slo,
                                          const unsigned long long *sg2, int cnt,
                                          const float4 &ta, const float4 &tb, const float4 &tc,
                                          float cx, float cy, const pfd::GaussParams &gp,
                                          float (&acc)[16]) {
    const P2PSums r = p2p_chunk_sums<NT, MODE>(
        (uint32_t)__cvta_generic_to_shared(shi), (uint32_t)__cvta_generic_to_shared(slo),
        (uint32_t)__cvta_generic_to_shared(sg2), cnt, ta, tb, tc, cx, cy, gp);
    pfd::comp_add(acc[0], acc[1], r.s[0]);
    pfd::comp_add(acc[2], acc[3], r.s[1]);
    if (NT >= 2) {
        pfd::comp_add(acc[4], acc[5], r.s[2]);
        pfd::comp_add(acc[6], acc[7], r.s[3]);
    }
    if (NT == 3) {
        pfd::comp_add(acc[8], acc[9], r.s[4]);
        pfd::comp_add(acc[10], acc[11], r.s[5]);
    }
}

// The third target slot of a group of 65..96 targets: the rem = size - 64
// remainder targets are paired (c, d) into rp = ceil(rem / 2) packed pairs
// spread over the warp, m = 32 / rp lanes per pair, lane (j + rp q) taking
// sources q, q + m, q + 2m, ... of the chunk for pair j with the packed pair
// code of the main slots; the m partial sums are combined at the end of the
// group.  Lanes with no share get q >= 32.  Returns -nx_c, ny_c, -nx_d, ny_d.
template <int MODE>
__device__ __noinline__ float4 p2p_split_sums(uint32_t a_hi, uint32_t a_lo, uint32_t a_g, int cnt,
                                              int q, int m, float4 tc, float4 td, float cx,
                                              float cy, pfd::GaussParams gp) {
    const pfd::GaussParams2 gp2 = pfd::make_params2(gp);
    pfd::f32x2 nx = 0ull, ny = 0ull;
    if constexpr (MODE == P2P_FAR) {
        const pfd::f32x2 txc = pfd::pack2((tc.x - cx) + tc.z, (td.x - cx) + td.z);
        const pfd::f32x2 tyc = pfd::pack2((tc.y - cy) + tc.w, (td.y - cy) + td.w);
#pragma unroll 2
        for (int k = q; k < cnt; k += m)
            pfd::pair2_far_local(lds_u64x2(a_hi + 16 * k), lds_u64(a_g + 8 * k), txc, tyc, gp2, nx,
                                 ny);
    } else {
        const pfd::f32x2 txh = pfd::pack2(tc.x, td.x), tyh = pfd::pack2(tc.y, td.y);
        const pfd::f32x2 txl = pfd::pack2(tc.z, td.z), tyl = pfd::pack2(tc.w, td.w);
#pragma unroll 2
        for (int k = q; k < cnt; k += m)
            pfd::pair2<MODE == P2P_SERIES>(lds_u64x2(a_hi + 16 * k), lds_u64x2(a_lo + 16 * k),
                                            lds_u64(a_g + 8 * k), txh, tyh, txl, tyl, gp2, nx, ny);
    }
    float nxc, nxd, nyc, nyd;
    pfd::unpack2(nx, nxc, nxd);
    pfd::unpack2(ny, nyc, nyd);
    return make_float4(-nxc, nyc, -nxd, nyd);
}

// p2p_chunk for the group's targets-per-lane count nt (warp-uniform).
// nt = 3: targets a, b packed plus the lane's share (qs of msp) of a
// remainder target pair (c, d).
template <int MODE>
__device__ __forceinline__ void p2p_run_chunk(int nt, const ulonglong2 *shi, const ulonglong2 *slo,
                                              const unsigned long long *sg2, int cnt,
                                              const float4 &ta, const float4 &tb,
                                              const float4 &tc, const float4 &td, int qs,
                                              int msp, float cx, float cy,
                                              const pfd::GaussParams &gp, float (&acc)[16]) {
    if (nt == 1) {
        p2p_chunk<1, MODE>(shi, slo, sg2, cnt, ta, tb, tc, cx, cy, gp, acc);
        return;
    }
    p2p_chunk<2, MODE>(shi, slo, sg2, cnt, ta, tb, tc, cx, cy, gp, acc);
    if (nt == 3) {
        const float4 r = p2p_split_sums<MODE>(
            (uint32_t)__cvta_generic_to_shared(shi), (uint32_t)__cvta_generic_to_shared(slo),
            (uint32_t)__cvta_generic_to_shared(sg2), cnt, qs, msp, tc, td, cx, cy, gp);
        pfd::comp_add(acc[8], acc[9], r.x);
        pfd::comp_add(acc[10], acc[11], r.y);
        pfd::comp_add(acc[12], acc[13], r.z);
        pfd::comp_add(acc[14], acc[15], r.w);
    }
}

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// A target group as one warp holds it: group gi of block b (groups of at most
// 96 targets, balanced: sizes differ by at most one; every group streams all
// the block's sources, so a small last group would cost nearly as much as a
// full one).
struct P2PGroup {
    float4 ta, tb, tc, td;  // the lane's targets a, b and remainder pair c, d
    int tg, gsz, nt;        // first target, targets; targets per lane: 1, 2, or 3 = two and a
    int rp, msp, qs;        // remainder share: remainder pairs, lanes per pair, this lane's share
    float bx0, bx1, by0, by1;  // box of the targets' hi parts
    float reach2, reachf2;     // box distances of the series and far classes, squared
    float cx, cy;              // centre for the far sources' relative coordinates
};

__device__ __forceinline__ bool p2p_group_setup(int t0, int tn, int ngrp, int gi,
                                                const float4 *__restrict__ thl,
                                                const pfd::GaussParams &gp, int64_t nt_all,
                                                P2PGroup &q) {
    const int lane = threadIdx.x & 31;
    const int tg = (int)((int64_t)gi * tn / ngrp);
    const int gsz = (int)((int64_t)(gi + 1) * tn / ngrp) - tg;
    const int nt = (gsz <= 32) ? 1 : (gsz <= 64) ? 2 : 3;  // warp-uniform
    // nt = 3: remainder targets tg + 64 + j, j < rem, in rp packed pairs
    // (tg + 64 + 2 p, + 1), each pair on msp lanes
    const int rem = nt == 3 ? gsz - 64 : 32;
    const int rp = (rem + 1) / 2;
    const int msp = 32 / rp;
    const bool cval = nt == 3 && lane < rp * msp;
    const int ic = tg + 64 + 2 * (lane % rp), id = ic + 1;
    const bool dval = cval && id < tg + gsz;
    q.tg = tg;
    q.gsz = gsz;
    q.nt = nt;
    q.rp = rp;
    q.msp = msp;
    q.qs = cval ? lane / rp : 32;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!PF_IDX_OK((int64_t)t0 + tg + gsz - 1, nt_all, 204)) return false;  // the group's last target
    q.ta = (lane < gsz) ? thl[t0 + tg + lane] : z4;
    q.tb = (lane + 32 < gsz) ? thl[t0 + tg + 32 + lane] : z4;
    q.tc = cval ? thl[t0 + ic] : z4;
    q.td = dval ? thl[t0 + id] : q.tc;  // an odd remainder's last pair repeats c
    // box of the group's targets (hi parts), for the series-free test
    float bx0 = INFINITY, bx1 = -INFINITY, by0 = INFINITY, by1 = -INFINITY;
    if (lane < q.gsz) { bx0 = bx1 = q.ta.x; by0 = by1 = q.ta.y; }
    if (lane + 32 < q.gsz) { bx0 = fminf(bx0, q.tb.x); bx1 = fmaxf(bx1, q.tb.x); by0 = fminf(by0, q.tb.y); by1 = fmaxf(by1, q.tb.y); }
    if (cval) { bx0 = fminf(bx0, fminf(q.tc.x, q.td.x)); bx1 = fmaxf(bx1, fmaxf(q.tc.x, q.td.x)); by0 = fminf(by0, fminf(q.tc.y, q.td.y)); by1 = fmaxf(by1, fmaxf(q.tc.y, q.td.y)); }
    q.bx0 = warp_min(bx0);
    q.bx1 = warp_max(bx1);
    q.by0 = warp_min(by0);
    q.by1 = warp_max(by1);
    // a source at box distance d has r2 >= (d - e)^2 for every target, e
    // covering the hi-part rounding of both points (2^-23 relative each)
    const float mag = fmaxf(fmaxf(fabsf(q.bx0), fabsf(q.bx1)), fmaxf(fabsf(q.by0), fabsf(q.by1)));
    const float rser = sqrtf(gp.r2_series);
    const float reach = rser * 1.001f + (mag + rser) * 4.8e-7f + 1e-30f;
    q.reach2 = reach * reach;
    const float rfar = sqrtf(gp.r2_far);
    const float reachf = rfar * 1.001f + (mag + rfar) * 4.8e-7f + 1e-30f;
    q.reachf2 = reachf * reachf;
    // centre for the far sources' relative coordinates (any float near the group)
    q.cx = 0.5f * (q.bx0 + q.bx1);
    q.cy = 0.5f * (q.by0 + q.by1);
    return true;
}

// Mode of a source of the group's stream.
__device__ __forceinline__ int p2p_class(const P2PGroup &q, const float4 &s) {
    const float ex = fmaxf(fmaxf(q.bx0 - s.x, s.x - q.bx1), 0.f);
    const float ey = fmaxf(fmaxf(q.by0 - s.y, s.y - q.by1), 0.f);
    const float d2 = ex * ex + ey * ey;
    return d2 > q.reachf2 ? P2P_FAR : d2 > q.reach2 ? P2P_FULL : P2P_SERIES;
}

// Puts a source of mode cls at entry k of that mode's buffer.
__device__ __forceinline__ void p2p_store(const P2PGroup &q, int cls, const float4 &s, float g,
                                          ulonglong2 *hi, ulonglong2 *lo, unsigned long long *g2) {
    if (cls == P2P_FAR) {  // coordinates relative to the group centre
        const float lx = (s.x - q.cx) + s.z, ly = (s.y - q.cy) + s.w;
        *hi = make_ulonglong2(pfd::pack2(lx, lx), pfd::pack2(ly, ly));
    } else {
        *hi = make_ulonglong2(pfd::pack2(s.x, s.x), pfd::pack2(s.y, s.y));
        *lo = make_ulonglong2(pfd::pack2(s.z, s.z), pfd::pack2(s.w, s.w));
    }
    *g2 = pfd::pack2(g, g);
}

// The group's near-field velocities from one warp's (hi, lo) sums.
__device__ __forceinline__ void p2p_group_write(const P2PGroup &q, int t0, const float (&acc)[16],
                                                double2 *__restrict__ nearv) {
    const int lane = threadIdx.x & 31;
    const int ia = q.tg + lane, ic = q.tg + 64 + 2 * (lane % q.rp);
    if (lane < q.gsz)
        nearv[t0 + ia] = make_double2(P2P_INV_2PI * ((double)acc[0] + (double)acc[1]),
                                        P2P_INV_2PI * ((double)acc[2] + (double)acc[3]));
    if (lane + 32 < q.gsz)
        nearv[t0 + ia + 32] = make_double2(P2P_INV_2PI * ((double)acc[4] + (double)acc[5]),
                                        P2P_INV_2PI * ((double)acc[6] + (double)acc[7]));
    if (q.nt == 3) {  // combine the msp shares of each remainder pair, in lane order
        float h[4] = {acc[8], acc[10], acc[12], acc[14]};
        float l[4] = {acc[9], acc[11], acc[13], acc[15]};
        for (int j = 1; j < q.msp; ++j) {
            const int sl = lane % q.rp + q.rp * j;  // < rp * msp <= 32
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const float a = __shfl_sync(0xffffffffu, acc[8 + 2 * v], sl);
                const float b = __shfl_sync(0xffffffffu, acc[9 + 2 * v], sl);
                pfd::comp_add(h[v], l[v], a);
                l[v] += b;
            }
        }
        if (lane < q.rp) {
            nearv[t0 + ic] = make_double2(P2P_INV_2PI * ((double)h[0] + (double)l[0]),
                                            P2P_INV_2PI * ((double)h[1] + (double)l[1]));
            if (ic + 1 < q.tg + q.gsz)
                nearv[t0 + ic + 1] = make_double2(P2P_INV_2PI * ((double)h[2] + (double)l[2]),
                                                P2P_INV_2PI * ((double)h[3] + (double)l[3]));
        }
    }
}

// Particle start and stream prefix of runs rc .. rc + nrc - 1 (one warp; nrc
// <= P2P_RUNS_SM); returns the stream's length.
__device__ __forceinline__ int p2p_load_runs(int rc, int nrc, const int32_t *__restrict__ sstart,
                                             const int32_t *__restrict__ scnt,
                                             const int2 *__restrict__ runs, int *s_rs, int *s_rp) {
    const int lane = threadIdx.x & 31;
    int pre = 0;
    for (int k0 = 0; k0 < nrc; k0 += 32) {
        const int k = k0 + lane;
        int st = 0, len = 0;
        if (k < nrc) {
            const int2 rr = runs[rc + k];
            st = sstart[rr.x];
            len = sstart[rr.y] + scnt[rr.y] - st;
        }
        int inc = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (k < nrc) {
            s_rs[k] = st;
            s_rp[k] = pre + inc - len;
        }
        pre += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) s_rp[nrc] = pre;
    __syncwarp();
    return pre;
}

template <int MODE>
__device__ __forceinline__ void p2p_chunk_of(const P2PGroup &q, const ulonglong2 *hi,
                                             const ulonglong2 *lo, const unsigned long long *g2,
                                             int cnt, const pfd::GaussParams &gp,
                                             float (&acc)[16]) {
    p2p_run_chunk<MODE>(q.nt, hi, lo, g2, cnt, q.ta, q.tb, q.tc, q.td, q.qs, q.msp, q.cx, q.cy, gp,
                        acc);
}

// Adds a group's pairs (all, and of mode P2P_FAR) to the call's counters.
__device__ __forceinline__ void p2p_count(unsigned long long *pairs, int nsrc, int nfar, int gsz) {
    if (threadIdx.x == 0 && nsrc) {
        atomicAdd(pairs, (unsigned long long)nsrc * (unsigned long long)gsz);
        atomicAdd(pairs + 2, (unsigned long long)nfar * (unsigned long long)gsz);
    }
}

// Target group gi of block b against the block's whole source stream, by one
// warp; writes the group's near-field velocities.
__device__ __forceinline__ void p2p_group_body(
    int64_t b, int t0, int tn, int ngrp, int gi, const int32_t *__restrict__ sstart,
    const int32_t *__restrict__ scnt, const float4 *__restrict__ shl,
    const float *__restrict__ sg32, const float4 *__restrict__ thl,
    const int32_t *__restrict__ run_off, const int2 *__restrict__ runs, pfd::GaussParams gp,
    double2 *__restrict__ nearv, ulonglong2 (*s_hi)[P2P_BUF], ulonglong2 (*s_lo)[P2P_BUF],
    unsigned long long (*s_g2)[P2P_BUF], int *s_rs, int *s_rp, unsigned long long *pairs,
    int64_t ns_all, int64_t nt_all) {
    const int lane = threadIdx.x;
    const unsigned lt = (1u << lane) - 1u;
    const int r0 = run_off[b], r1 = run_off[b + 1];
    P2PGroup q;
    if (!p2p_group_setup(t0, tn, ngrp, gi, thl, gp, nt_all, q)) return;
    int nsrc = 0, nfar = 0;  // sources of the stream, those of mode P2P_FAR
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    float acc[16] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f,
                     0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // the three buffers are rings of P2P_BUF = 64 entries: entries waiting
    // c0, c1, c2 from heads h0, h1, h2; a chunk is always the 32 entries at
    // the head (0 or 32), so it never wraps, and taking it flips the head
    int c0 = 0, c1 = 0, c2 = 0;
    int h0 = 0, h1 = 0, h2 = 0;
    for (int rc = r0; rc < r1; rc += P2P_RUNS_SM) {
        const int nrc = min(P2P_RUNS_SM, r1 - rc);
        const int S = p2p_load_runs(rc, nrc, sstart, scnt, runs, s_rs, s_rp);
        nsrc += S;
        // each lane's stream position only moves forward (by 32 per
        // round), so the run holding it is found by advancing an index:
        // the largest r with prefix[r] <= p (empty runs are stepped over).
        // The loads of round s0 + 32 are issued before round s0's chunks
        // run, so their latency overlaps the pair work.
        int rr = 0;
        float4 spv = z4;
        float gg = 0.f;
        auto fetch = [&](int p, float4 &v, float &w) {
            if (p < S) {
                while (rr + 1 < nrc && s_rp[rr + 1] <= p) ++rr;
                const int src = s_rs[rr] + (p - s_rp[rr]);
                if (PF_IDX_OK(src, ns_all, 203)) {
                    v = shl[src];
                    w = sg32[src];
                }
            }
        };
        fetch(lane, spv, gg);
        for (int s0 = 0; s0 < S; s0 += 32) {
            const int p = s0 + lane;
            int cls = -1;  // 0 far, 1 full, 2 series; -1 past the stream
            if (p < S) cls = p2p_class(q, spv);
            // append each source to the buffer of its mode, in stream order
            const unsigned m0 = __ballot_sync(0xffffffffu, cls == 0);
            const unsigned m1 = __ballot_sync(0xffffffffu, cls == 1);
            const unsigned m2 = __ballot_sync(0xffffffffu, cls == 2);
            if (cls >= 0) {
                const unsigned mm = cls == 0 ? m0 : cls == 1 ? m1 : m2;
                const int k =
                    ((cls == 0 ? h0 + c0 : cls == 1 ? h1 + c1 : h2 + c2) + __popc(mm & lt)) &
                    (P2P_BUF - 1);
                p2p_store(q, cls, spv, gg, &s_hi[cls][k], &s_lo[cls][k], &s_g2[cls][k]);
            }
            c0 += __popc(m0);
            c1 += __popc(m1);
            c2 += __popc(m2);
            spv = z4;
            gg = 0.f;
            fetch(p + 32, spv, gg);
            __syncwarp();
            bool ran = false;  // warp-uniform
            if (c0 >= 32) {
                p2p_chunk_of<P2P_FAR>(q, s_hi[0] + h0, s_lo[0] + h0, s_g2[0] + h0, 32, gp, acc);
                nfar += 32;
                c0 -= 32;
                h0 ^= 32;
                ran = true;
            }
            if (c1 >= 32) {
                p2p_chunk_of<P2P_FULL>(q, s_hi[1] + h1, s_lo[1] + h1, s_g2[1] + h1, 32, gp, acc);
                c1 -= 32;
                h1 ^= 32;
                ran = true;
            }
            if (c2 >= 32) {
                p2p_chunk_of<P2P_SERIES>(q, s_hi[2] + h2, s_lo[2] + h2, s_g2[2] + h2, 32, gp, acc);
                c2 -= 32;
                h2 ^= 32;
                ran = true;
            }
            if (ran) __syncwarp();  // the chunks are read before the next round refills them
        }
    }
    // what is left in the buffers (fewer than 32 each)
    // (fewer than 32 from a head of 0 or 32: no wrap)
    if (c0)
        p2p_chunk_of<P2P_FAR>(q, s_hi[0] + h0, s_lo[0] + h0, s_g2[0] + h0, c0, gp, acc);
    nfar += c0;
    if (c1)
        p2p_chunk_of<P2P_FULL>(q, s_hi[1] + h1, s_lo[1] + h1, s_g2[1] + h1, c1, gp, acc);
    if (c2)
        p2p_chunk_of<P2P_SERIES>(q, s_hi[2] + h2, s_lo[2] + h2, s_g2[2] + h2, c2, gp, acc);
    __syncwarp();
    p2p_group_write(q, t0, acc, nearv);
    p2p_count(pairs, nsrc, nfar, q.gsz);
}

// Shared memory of one P2P CTA (one warp).
struct P2PSmem {
    // source buffers, one per mode: [P2P_FAR], [P2P_FULL], [P2P_SERIES]
    ulonglong2 hi[3][P2P_BUF];  // {x_hi, x_hi}, {y_hi, y_hi}
    ulonglong2 lo[3][P2P_BUF];  // {x_lo, x_lo}, {y_lo, y_lo}
    unsigned long long g2[3][P2P_BUF];  // {g, g}
    int rs[P2P_RUNS_SM];      // particle start of run
    int rp[P2P_RUNS_SM + 1];  // stream prefix of run
};

// Targets of P2P block b: first sorted target t0, count returned.
__device__ __forceinline__ int p2p_targets(const P2PDesc &d, int64_t b, int &t0) {
    const uint32_t leaf0 = (uint32_t)b << (2 * d.kb), nl = 1u << (2 * d.kb);
    t0 = d.tstart[leaf0];
    return d.tstart[leaf0 + nl - 1] + d.tcnt[leaf0 + nl - 1] - t0;
}

// Target groups of a block of tn targets.
__device__ __forceinline__ int p2p_groups(int tn) { return (tn + P2P_GROUP - 1) / P2P_GROUP; }

// Block and group of task t: t < direct the first group of block t of the launch
// order, then the listed groups; false past those.
__device__ __forceinline__ bool p2p_task(const P2PDesc &d, unsigned t, int &b, int &gi) {
    const unsigned direct = (unsigned)d.direct;
    if (t < direct) {
        b = d.order[t];
        gi = 0;
        return true;
    }
    if (t - direct >= *d.nmore) return false;
    const int2 e = d.more[t - direct];
    b = e.x;
    gi = e.y;
    return true;
}

__device__ __forceinline__ void p2p_group(const P2PDesc &d, int64_t b, int t0, int tn, int gi,
                                          P2PSmem &sm) {
    p2p_group_body(b, t0, tn, p2p_groups(tn), gi, d.sstart, d.scnt, d.shl,
                   d.sg32, d.thl, d.run_off, d.runs, d.gp, d.nearv, sm.hi, sm.lo, sm.g2, sm.rs,
                   sm.rp, d.pairs, d.ns, d.nt);
}

}  // namespace
