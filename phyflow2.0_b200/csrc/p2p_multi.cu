// p2p_multi.cu -- the FMM near field with several warps per target group, for
// trees with too few groups to fill the device with one warp each.
#include "p2p.cuh"

namespace {

// Sums of a chunk for the lane's targets, not folded: r[0..1] (x, y) of target
// a, r[2..3] of b (nt >= 2), r[4..7] of the remainder pair's share (nt = 3).
template <int MODE>
__device__ __forceinline__ void p2p_chunk_raw(const P2PGroup &q, const ulonglong2 *hi,
                                              const ulonglong2 *lo, const unsigned long long *g2,
                                              int cnt, const pfd::GaussParams &gp, float (&r)[8]) {
    const uint32_t ah = (uint32_t)__cvta_generic_to_shared(hi),
                   al = (uint32_t)__cvta_generic_to_shared(lo),
                   ag = (uint32_t)__cvta_generic_to_shared(g2);
    if (q.nt == 1) {
        const P2PSums s = p2p_chunk_sums<1, MODE>(ah, al, ag, cnt, q.ta, q.tb, q.tc, q.cx, q.cy, gp);
        r[0] = s.s[0];
        r[1] = s.s[1];
        return;
    }
    const P2PSums s = p2p_chunk_sums<2, MODE>(ah, al, ag, cnt, q.ta, q.tb, q.tc, q.cx, q.cy, gp);
#pragma unroll
    for (int v = 0; v < 4; ++v) r[v] = s.s[v];
    if (q.nt == 3) {
        const float4 t =
            p2p_split_sums<MODE>(ah, al, ag, cnt, q.qs, q.msp, q.tc, q.td, q.cx, q.cy, gp);
        r[4] = t.x;
        r[5] = t.y;
        r[6] = t.z;
        r[7] = t.w;
    }
}

// One target group per CTA of W warps.  The warps share the group's three
// buffers.  A round: each warp stages and classifies 32 of 32 W sources; a scan
// of the warps' counts gives every source its place (stream order, as in the
// one-warp kernel); the chunks of 32 that are then complete are dealt out to
// the warps in turn, and their sums go to shared memory.  In the next round
// each warp folds some of the group's eight sums (x, y of targets a, b, c, d)
// over those chunks.  The order is the one-warp kernel's, in which the chunks
// complete 32 sources at a time, far before full before series: bit 4 v + c of
// the round's mask says that warp v's sources complete a chunk of class c.  So
// the result is bitwise that of the one-warp kernel.
template <int W>
struct P2PSmemW {
    static constexpr int RB = 32 * (W + 1);  // ring entries: 31 waiting + a round
    static constexpr int CH = W + 2;         // most chunks of a round
    ulonglong2 hi[3][RB];
    ulonglong2 lo[3][RB];
    unsigned long long g2[3][RB];
    float sum[CH][8][32];
    int rs[P2P_RUNS_SM];
    int rp[P2P_RUNS_SM + 1];
    int cnt[W];        // a round's sources per warp: far | full << 10 | series << 20
    unsigned mask[2];  // a round's chunks, in order (rounds alternate)
};

template <int W>
__global__ void __launch_bounds__(32 * W, P2P_MIN_CTAS / W) k_p2p_multi(const P2PDesc d) {
    using Smem = P2PSmemW<W>;
    constexpr int RB = Smem::RB;
    constexpr int NV = 8 / W;  // sums each warp folds: v = wid + W i
    __shared__ Smem sm;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    int b, gi, t0;
    if (!p2p_task(d, blockIdx.x, b, gi)) return;
    const int tn = p2p_targets(d, b, t0);
    if (tn == 0) return;
    const int ngrp = p2p_groups(tn);
    P2PGroup q;
    if (!p2p_group_setup(t0, tn, ngrp, gi, d.thl, d.gp, d.nt, q)) return;
    const int nv = q.nt == 1 ? 2 : q.nt == 2 ? 4 : 8;  // sums in use
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    float acc[NV][2];
#pragma unroll
    for (int i = 0; i < NV; ++i) acc[i][0] = acc[i][1] = 0.f;
    int c0 = 0, c1 = 0, c2 = 0, h0 = 0, h1 = 0, h2 = 0;  // waiting entries and heads
    int turn = wid;   // chunks until this warp's next one, modulo W
    int waiting = 0;  // chunks whose sums wait to be folded
    int nsrc = 0, nfar = 0;
    unsigned parity = 0;
    if (threadIdx.x < 2) sm.mask[threadIdx.x] = 0u;
    auto wrap = [](int k) { return k >= RB ? k - RB : k; };
    auto run_chunk = [&](int cls, int head, int n, int slot) {
        float r[8];
        if (cls == P2P_FAR)
            p2p_chunk_raw<P2P_FAR>(q, sm.hi[0] + head, sm.lo[0] + head, sm.g2[0] + head, n, d.gp, r);
        else if (cls == P2P_FULL)
            p2p_chunk_raw<P2P_FULL>(q, sm.hi[1] + head, sm.lo[1] + head, sm.g2[1] + head, n, d.gp, r);
        else
            p2p_chunk_raw<P2P_SERIES>(q, sm.hi[2] + head, sm.lo[2] + head, sm.g2[2] + head, n, d.gp,
                                      r);
#pragma unroll
        for (int v = 0; v < 8; ++v)
            if (v < nv) sm.sum[slot][v][lane] = r[v];
    };
    auto fold = [&]() {
        for (int t = 0; t < waiting; ++t)
#pragma unroll
            for (int i = 0; i < NV; ++i)
                if (wid + W * i < nv)
                    pfd::comp_add(acc[i][0], acc[i][1], sm.sum[t][wid + W * i][lane]);
    };
    const int r0 = d.run_off[b], r1 = d.run_off[b + 1];
    for (int rc = r0; rc < r1; rc += P2P_RUNS_SM) {
        const int nrc = min(P2P_RUNS_SM, r1 - rc);
        __syncthreads();  // every warp is done with the previous runs (and the masks are zero)
        // every warp writes the same values
        const int S = p2p_load_runs(rc, nrc, d.sstart, d.scnt, d.runs, sm.rs, sm.rp);
        nsrc += S;
        int rr = 0;
        float4 spv = z4;
        float gg = 0.f;
        auto fetch = [&](int p) {
            spv = z4;
            gg = 0.f;
            if (p < S) {
                while (rr + 1 < nrc && sm.rp[rr + 1] <= p) ++rr;
                const int src = sm.rs[rr] + (p - sm.rp[rr]);
                if (PF_IDX_OK(src, d.ns, 203)) {
                    spv = d.shl[src];
                    gg = d.sg32[src];
                }
            }
        };
        fetch(32 * wid + lane);
        for (int s0 = 0; s0 < S; s0 += 32 * W) {
            const int p = s0 + 32 * wid + lane;
            int cls = -1;
            if (p < S) cls = p2p_class(q, spv);
            const unsigned m0 = __ballot_sync(0xffffffffu, cls == 0);
            const unsigned m1 = __ballot_sync(0xffffffffu, cls == 1);
            const unsigned m2 = __ballot_sync(0xffffffffu, cls == 2);
            const int mine = __popc(m0) | __popc(m1) << 10 | __popc(m2) << 20;
            if (lane == 0) sm.cnt[wid] = mine;
            __syncthreads();  // the counts; and the previous round's chunks are done
            int pre = c0 | c1 << 10 | c2 << 20, tot = pre;
#pragma unroll
            for (int v = 0; v < W; ++v) {
                const int n = sm.cnt[v];
                if (v < wid) pre += n;
                tot += n;
            }
            if (cls >= 0) {
                const unsigned mm = cls == 0 ? m0 : cls == 1 ? m1 : m2;
                const int head = cls == 0 ? h0 : cls == 1 ? h1 : h2;
                const int k = wrap(head + (pre >> (10 * cls) & 1023) + __popc(mm & lt));
                p2p_store(q, cls, spv, gg, &sm.hi[cls][k], &sm.lo[cls][k], &sm.g2[cls][k]);
            }
            // the chunks this warp's sources complete: a count crosses a multiple of 32
            if (lane == 0) {
                const int e = pre + mine;
                const unsigned f = (unsigned)((e & 1023) >> 5 != (pre & 1023) >> 5) |
                                   (unsigned)((e >> 10 & 1023) >> 5 != (pre >> 10 & 1023) >> 5) << 1 |
                                   (unsigned)(e >> 25 != pre >> 25) << 2;
                if (f) atomicOr(&sm.mask[parity], f << (4 * wid));
                if (wid == 0) sm.mask[parity ^ 1] = 0u;  // last read before the barrier above
            }
            fold();
            fetch(p + 32 * W);
            __syncthreads();
            c0 = tot & 1023;
            c1 = tot >> 10 & 1023;
            c2 = tot >> 20;
            const unsigned mask = sm.mask[parity];
            const int n = __popc(mask);
            int t = turn;
            for (; t < n; t += W) {
                unsigned rest = mask;  // the round's chunk t: bit 4 v + class
                for (int k = 0; k < t; ++k) rest &= rest - 1;
                const int bit = __ffs(rest) - 1, cl = bit & 3;
                const int m = __popc(mask & (0x11111111u << cl) & ((1u << bit) - 1u));
                run_chunk(cl, wrap((cl == 0 ? h0 : cl == 1 ? h1 : h2) + 32 * m), 32, t);
            }
            turn = t - n;
            waiting = n;
            parity ^= 1u;
            nfar += c0 & ~31;
            h0 = wrap(h0 + (c0 & ~31));
            h1 = wrap(h1 + (c1 & ~31));
            h2 = wrap(h2 + (c2 & ~31));
            c0 &= 31;
            c1 &= 31;
            c2 &= 31;
        }
        __syncthreads();
        fold();
        waiting = 0;
    }
    // what is left in the buffers (fewer than 32 each; heads are multiples of
    // 32, so they do not wrap)
    nfar += c0;
    __syncthreads();
    int n = 0;
    if (c0 && n++ % W == wid) run_chunk(P2P_FAR, h0, c0, n - 1);
    if (c1 && n++ % W == wid) run_chunk(P2P_FULL, h1, c1, n - 1);
    if (c2 && n++ % W == wid) run_chunk(P2P_SERIES, h2, c2, n - 1);
    waiting = n;
    __syncthreads();
    fold();
    __syncthreads();
    // the sums to warp 0
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        sm.sum[0][wid + W * i][lane] = acc[i][0];
        sm.sum[1][wid + W * i][lane] = acc[i][1];
    }
    __syncthreads();
    if (wid > 0) return;
    float all[16];
#pragma unroll
    for (int v = 0; v < 8; ++v) {
        all[2 * v] = sm.sum[0][v][lane];
        all[2 * v + 1] = sm.sum[1][v][lane];
    }
    p2p_group_write(q, t0, all, d.nearv);
    p2p_count(d.pairs, nsrc, nfar, q.gsz);
}

}  // namespace

namespace pf {
namespace fmmx {

pf_status launch_p2p_multi(const P2PDesc &d, int warps, unsigned grid, cudaStream_t st) {
    if (warps >= 8)
        k_p2p_multi<8><<<grid, 256, 0, st>>>(d);
    else
        k_p2p_multi<4><<<grid, 128, 0, st>>>(d);
    return launch_status("k_p2p_multi");
}

}  // namespace fmmx
}  // namespace pf
