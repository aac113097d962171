// Tiled sm_100a kernels for 2-D windows with 16 real channels per unit
// (16 Float32 or 8 ComplexF32 channels per head) and softmax.
//
// Work decomposition.  A CTA owns TH consecutive rows (the fast axis h) of NQ
// consecutive columns w0..w0+NQ-1 of one unit (NQ = 4 in the forward and dq
// kernels, 3 in the dk/dv kernel).  A thread owns one row and the NQ pixels of
// that row ("centre" pixels: queries in the forward and dq kernels, keys in
// the dk/dv kernel) and keeps their 16-channel vectors in registers.  The other
// side of the window is streamed through shared memory one image column at a
// time: column stage s holds column w0 - p + s (wrapped circularly, or taken
// from the neighbour halo in band mode) for rows h0-p' .. h0+TH+p'-1.  Centre
// pixel r pairs with stage s iff r <= s <= r + 2p, so every loaded vector is
// used by up to NQ centre pixels straight from registers.
//
// Feeding the stages.  The reference layout is channel-planar, which no bulk
// copy can turn into pixel vectors, so a pack kernel first rewrites the two
// streamed tensors as ONE array [unit][column][row'][36] = (16 channels of the
// first | 16 of the second | 4 floats of padding) with the circular halo along
// h already unrolled (row' = h + p', p' = p rounded up to even; rows -p'..-1
// and H..H+p'-1 are copies of the wrapped rows).  A column stage is then a
// single contiguous box fetched by cp.async.bulk.tensor (TMA) and tracked by an
// mbarrier; three stages are in flight.  The wrap along w is just the column
// coordinate of the box.
//
// Shared-memory layout: a pixel row is 144 bytes (36 words).  The rows that the
// eight lanes of a 128-bit load phase touch are consecutive, 36 words apart,
// i.e. nine 4-bank groups apart: eight distinct groups, so the loads are
// conflict free without any address swizzle and every chunk of every row of a
// window column is the thread's row base plus a compile-time constant.
//
// Arithmetic: FP32 on the FMA pipe, channel pairs as two scalar FMAs.  Softmax in
// the log2 domain with ex2.approx.  The running maximum (forward) or the saved row
// statistic (backward) is folded into the initial value of the dot-product
// chain, and the forward only touches the maximum when the sign bits of a chunk
// of relative scores say that one of them is positive.
//
// Small grids.  When the grid would not fill the GPU, the column stages of a
// tile are split between two groups of warps of the same CTA (each with its own
// copy pipeline) whose partial results are merged through shared memory.
#include "tile_common.cuh"

namespace ca {
namespace {

// =====================================================================
// Forward
// =====================================================================
// Scores are kept relative to a running reference ref = (largest score seen when
// the reference was last set) + kHeadroom: the dot-product chain starts at -ref,
// so sc = s - ref and p = 2^sc needs no subtraction.  The reference moves only
// when some relative score of the chunk is non-negative (a score jumped more than
// kHeadroom log2 units above every earlier one), which the AND of the sign bits
// of the chunk reveals; with O(1) scores that happens almost never after the
// first key.  2^-kHeadroom only rescales p, l and acc together; it cancels in y.
constexpr float kHeadroom = 12.f;
// NS lanes share a pixel (units of 16*NS real channels): every lane holds one 16-channel slab of q and
// of the accumulator, scores are the lane sums of the per-slab partial dot products, and the terms that
// enter a score once (the running reference, in nm2) sit on slab 0 only.
template <int DC, bool DIST, int MASK, int NQ, int NS = 1>
__device__ __forceinline__ void fwd_stage(uint32_t rowbase, int ws, int rm, float sl2, const u64 (&q)[NQ][8],
                                          u64 (&acc)[NQ][8], u64 (&nm2)[NQ], float (&l)[NQ], const float (&bq)[NQ],
                                          int slab = 0) {
    constexpr int RB = kRowBytes * NS;
    for (int c0 = 0; c0 < ws; c0 += DC) {
        const uint32_t cb = rowbase + c0 * RB;
        float sc[NQ][DC];
        // one vector ahead: the next key (or the first v) is requested before this key's FMAs
        u64 nxt[8];
        lds_slab16<NS>(cb, 0, slab, nxt);
#pragma unroll
        for (int t = 0; t < DC; ++t) {
            {
                u64 k2[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) k2[i] = nxt[i];
                if (t + 1 < DC) lds_slab16<NS>(cb + (t + 1) * RB, 0, slab, nxt);
                else lds_slab16<NS>(cb, 1, slab, nxt);
                float bk = 0.f;
                if (DIST) {
                    u64 n = zero2();
#pragma unroll
                    for (int i = 0; i < 8; ++i) n = fma2(k2[i], k2[i], n);
                    bk = -0.5f * sl2 * hsum2(n);
                }
                if (MASK != 0) {
                    // all four chains advance together (4 independent FMAs in flight)
                    u64 sa[NQ];
#pragma unroll
                    for (int r = 0; r < NQ; ++r) {
                        sa[r] = nm2[r];                           // (-ref, 0)
                        if (DIST) sa[r] = add2(sa[r], pack2(bq[r] + bk, 0.f));
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int r = 0; r < NQ; ++r) sa[r] = fma2(q[r][i], k2[i], sa[r]);
#pragma unroll
                    for (int r = 0; r < NQ; ++r) sc[r][t] = lane_sum<NS>(hsum2(sa[r]));
                } else {
#pragma unroll
                    for (int r = 0; r < NQ; ++r)
                        if (CA_ON(r)) {
                            u64 sa = nm2[r];
                            if (DIST) sa = add2(sa, pack2(bq[r] + bk, 0.f));
#pragma unroll
                            for (int i = 0; i < 8; ++i) sa = fma2(q[r][i], k2[i], sa);
                            sc[r][t] = lane_sum<NS>(hsum2(sa));       // rm is warp-uniform: all lanes shuffle
                        } else {
                            sc[r][t] = -INFINITY;
                        }
                }
            }
        }
        // any relative score >= 0 ?  (sign bit clear)
        uint32_t allneg = 0x80000000u;
#pragma unroll
        for (int r = 0; r < NQ; ++r)
#pragma unroll
            for (int t = 0; t < DC; ++t) allneg &= __float_as_uint(sc[r][t]);
        if (__any_sync(0xffffffffu, allneg == 0u)) {
#pragma unroll
            for (int r = 0; r < NQ; ++r) {
                float cm = sc[r][0];
#pragma unroll
                for (int t = 1; t < DC; ++t) cm = fmaxf(cm, sc[r][t]);
                if (cm >= 0.f) {                // move the reference of this row up by cm + headroom
                    cm += kHeadroom;
                    const float corr = fast_exp2(-cm);
                    float nm, zero;
                    unpack2(nm2[r], nm, zero);
                    nm2[r] = pack2(nm - (NS == 1 || slab == 0 ? cm : 0.f), 0.f);
                    l[r] *= corr;
                    const u64 c2 = pack2(corr, corr);
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[r][i] = mul2(acc[r][i], c2);
#pragma unroll
                    for (int t = 0; t < DC; ++t) sc[r][t] -= cm;
                }
            }
        }
#pragma unroll
        for (int t = 0; t < DC; ++t) {
            {
                u64 v2[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) v2[i] = nxt[i];
                if (t + 1 < DC) lds_slab16<NS>(cb + (t + 1) * RB, 1, slab, nxt);
#pragma unroll
                for (int r = 0; r < NQ; ++r)
                    if (CA_ON(r)) {
                        const float pt = fast_exp2(sc[r][t]);
                        l[r] += pt;
                        const u64 p2 = pack2(pt, pt);
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[r][i] = fma2(p2, v2[i], acc[r][i]);
                    }
            }
        }
    }
}

// The ws keys of one window column.  EXACT: ws is a multiple of DC.  Otherwise (DC == 4): chunks of four keys, then
// the remaining one to three keys as one chunk of exactly that length, so that no chunk carries bounds checks
// (a checked chunk keeps its prefetched vector alive across branches, which costs a register copy per loaded
// word and made windows such as 13 slower than 15).
template <int DC, bool DIST, bool EXACT, int NQ, int NS>
__device__ __forceinline__ void fwd_window(uint32_t rowbase, int ws, int rm, float sl2, const u64 (&q)[NQ][8],
                                           u64 (&acc)[NQ][8], u64 (&nm2)[NQ], float (&l)[NQ], const float (&bq)[NQ],
                                           int slab) {
    constexpr int FULLM = (1 << NQ) - 1;
    if (EXACT) {
        fwd_stage<DC, DIST, FULLM, NQ, NS>(rowbase, ws, rm, sl2, q, acc, nm2, l, bq, slab);
        return;
    }
    static_assert(EXACT || DC == 4, "windows without a dividing chunk length run chunks of four plus a tail");
    const int main = ws & ~3;
    fwd_stage<4, DIST, FULLM, NQ, NS>(rowbase, main, rm, sl2, q, acc, nm2, l, bq, slab);
    const uint32_t tail = rowbase + main * (kRowBytes * NS);
    switch (ws - main) {                                     // warp-uniform
        case 1: fwd_stage<1, DIST, FULLM, NQ, NS>(tail, 1, rm, sl2, q, acc, nm2, l, bq, slab); break;
        case 2: fwd_stage<2, DIST, FULLM, NQ, NS>(tail, 2, rm, sl2, q, acc, nm2, l, bq, slab); break;
        case 3: fwd_stage<3, DIST, FULLM, NQ, NS>(tail, 3, rm, sl2, q, acc, nm2, l, bq, slab); break;
        default: break;
    }
}

// First score of each centre pixel that starts in this stage: the reference
// point of its running maximum.
template <bool DIST, int NQ, int NS = 1>
__device__ __forceinline__ void fwd_init_max(uint32_t rowbase, int init, float sl2, const u64 (&q)[NQ][8],
                                             u64 (&nm2)[NQ], const float (&bq)[NQ], int slab = 0) {
    u64 k2[8];
    lds_slab16<NS>(rowbase, 0, slab, k2);
    float bk = 0.f;
    if (DIST) {
        u64 n = zero2();
#pragma unroll
        for (int i = 0; i < 8; ++i) n = fma2(k2[i], k2[i], n);
        bk = -0.5f * sl2 * hsum2(n);
    }
#pragma unroll
    for (int r = 0; r < NQ; ++r)
        if ((init >> r) & 1) {
            u64 sa = zero2();
#pragma unroll
            for (int i = 0; i < 8; ++i) sa = fma2(q[r][i], k2[i], sa);
            const float s0 = lane_sum<NS>(hsum2(sa) + (DIST ? bq[r] + bk : 0.f));     // init is warp-uniform
            nm2[r] = pack2((NS == 1 || slab == 0) ? -s0 - kHeadroom : 0.f, 0.f);
        }
}

#define CA_MASK_SWITCH(FULL, mask, CALL)                            \
    if ((mask) == (FULL)) { constexpr int MK = (FULL); CALL; }      \
    else { constexpr int MK = 0; CALL; }

// NCRT = real channels per unit the kernel is compiled for: 16 (narrower units are zero-extended),
// 32 or 64 (NS = 2 or 4 lanes per pixel, one 16-channel slab each; launched without a stage split).
template <int DC, bool DIST, int CPE, bool EXACT, int NQ, int NCRT = 16>
__global__ void __launch_bounds__(128, (NQ <= 2 ? 3 : 2)) fwd_tiled_kernel(TileArgs a, const __grid_constant__ CUtensorMap mv,
                                                           const __grid_constant__ CUtensorMap msc) {
    constexpr int NS = NCRT <= 16 ? 1 : NCRT / 16;
    constexpr int RB = kRowBytes * NS;
    const Geo& g = a.g;
    const int ROWS = a.TH + 2 * (g.p + a.roff);
    const int NSTAGES = g.wsw + NQ - 1;
    const int w0 = blockIdx.x * NQ, h0 = blockIdx.y * a.TH, u = blockIdx.z;
    const float sl2 = a.scale * kLog2e;
    CA_PIPE_PROLOGUE(false)
    const int slab = NS == 1 ? 0 : (lt % NS);
    const int lr = NS == 1 ? lt : (lt >> 5) * (32 / NS) + (lt & 31) / NS, h = h0 + lr;
    const bool active = h < g.H;

    u64 q[NQ][8], acc[NQ][8];
    load_centre<CPE, NQ, NCRT>(a.c0, g, u, h, w0, active, sl2, q, 16 * slab);
    u64 nm2[NQ];
    float l[NQ], bq[NQ];
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        nm2[r] = pack2(INFINITY, 0.f);           // (-m, 0); running maximum -inf: no key seen yet
        l[r] = 0.f;
        bq[r] = 0.f;
        if (DIST) {
            u64 n = zero2();
#pragma unroll
            for (int i = 0; i < 8; ++i) n = fma2(q[r][i], q[r][i], n);
            bq[r] = -0.5f * hsum2(n) / sl2;      // q is pre-scaled by sl2
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[r][i] = zero2();
    }

    CA_PIPE_LOOP({
        const int mask = stage_mask<NQ>(s, radius_w(g));
        const uint32_t rowbase = smem_u32(pipe.vec(buf)) + (lr + a.roff) * RB;
        // pixels whose first stage (of this part) is s
        const int init = (s == s_begin) ? mask : (mask & ~stage_mask<NQ>(s - 1, radius_w(g)));
        if (init) fwd_init_max<DIST, NQ, NS>(rowbase, init, sl2, q, nm2, bq, slab);
        if (mask != (1 << NQ) - 1) {
            // a stage that pairs with only some of the columns: the all-slots code (interleaved chains) with the
            // unpaired slots' scores forced to -inf, so that they contribute exact zeros; measured 6-7 % faster
            // over a forward than computing the paired slots one after the other
            u64 nmE[NQ];
#pragma unroll
            for (int r = 0; r < NQ; ++r) nmE[r] = ((mask >> r) & 1) ? nm2[r] : pack2(-INFINITY, 0.f);
            fwd_window<DC, DIST, EXACT, NQ, NS>(rowbase, g.ws, mask, sl2, q, acc, nmE, l, bq, slab);
#pragma unroll
            for (int r = 0; r < NQ; ++r)
                if ((mask >> r) & 1) nm2[r] = nmE[r];
        } else {
            fwd_window<DC, DIST, EXACT, NQ, NS>(rowbase, g.ws, mask, sl2, q, acc, nm2, l, bq, slab);
        }
    })

    float nm[NQ];
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        float zero;
        unpack2(nm2[r], nm[r], zero);
    }
    if (a.nsplit == 2) {
        // merge the two partial softmaxes: part 1 publishes (m, l, acc), part 0 combines
        float* xch = reinterpret_cast<float*>(smem_al);
        if (part == 1) {
#pragma unroll
            for (int r = 0; r < NQ; ++r) {
                xch[(r * 18 + 0) * PT + lt] = nm[r];
                xch[(r * 18 + 1) * PT + lt] = l[r];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float x, y;
                    unpack2(acc[r][i], x, y);
                    xch[(r * 18 + 2 + 2 * i) * PT + lt] = x;
                    xch[(r * 18 + 3 + 2 * i) * PT + lt] = y;
                }
            }
        }
        __syncthreads();
        if (part == 1) return;
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            const float nm1 = xch[(r * 18 + 0) * PT + lt], l1 = xch[(r * 18 + 1) * PT + lt];
            const float nmn = fminf(nm[r], nm1);           // -max(m0, m1)
            const float c0 = (nm[r] == INFINITY) ? 0.f : fast_exp2(nmn - nm[r]);
            const float c1 = (nm1 == INFINITY) ? 0.f : fast_exp2(nmn - nm1);
            l[r] = l[r] * c0 + l1 * c1;
            nm[r] = nmn;
            const u64 c02 = pack2(c0, c0), c12 = pack2(c1, c1);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const u64 o = pack2(xch[(r * 18 + 2 + 2 * i) * PT + lt], xch[(r * 18 + 3 + 2 * i) * PT + lt]);
                acc[r][i] = fma2(o, c12, mul2(acc[r][i], c02));
            }
        }
    }
    CA_OUT_DISPATCH(
        _Pragma("unroll")
        for (int r = 0; r < NQ; ++r) {
            const float inv = 1.f / l[r] + ca_poison;
            _Pragma("unroll")
            for (int i = 0; i < 8; ++i) {
                float x, y;
                unpack2(acc[r][i], x, y);
                store_centre<CPE, NCRV, BF>(a.o0, g, u, h, w0, active, r, i, x * inv, y * inv, 16 * slab);
            }
        })
#pragma unroll
    for (int r = 0; r < NQ; ++r)
        if (a.ostats && active && slab == 0 && has_pixel(g, h, w0 + r))
            a.ostats[(int64_t)u * g.Np + h + g.H * (w0 + r)] = (log2f(l[r]) - nm[r]) * kLn2 + ca_poison;
}

// =====================================================================
// Backward, query-owned: dq.  The s chain starts at -L (log2 domain) and the
// dP chain at -D, so P = 2^chain and dS = P * chain'.
// =====================================================================
// MODE 0: softmax, P = 2^chain.  MODE 1: 1.5-entmax, g = max(chain, 0) with the chain = s/2 - tau, dS = g*(dP - D).
// MODE 2: the entmax pre-pass: only num += g*dP and den += g (in aux and sumds), D = num/den.
// The same query-owned sweep serves the entmax forward, which has no dy: MODE 3 the row maximum of s/2 (in aux);
// MODE 4 one step of the threshold search: with t = chain = s/2 - tau, the sum of max(t, 0) (sumds), of its
// square (aux), the size of the support {t > 0}, its smallest member and the largest t outside (ex[0..2]);
// MODE 5 the apply: dq (here y) += max(chain, 0)^2 * v.
template <bool DIST, int MASK, int NQ, int MODE, int NS = 1>
__device__ __forceinline__ void dq_stage(uint32_t rowbase, int ws, int rm, float sl2, const u64 (&q)[NQ][8],
                                         const u64 (&dy)[NQ][8], u64 (&dq)[NQ][8], const u64 (&nL2)[NQ],
                                         const u64 (&nD2)[NQ], const float (&bq)[NQ], float (&sumds)[NQ],
                                         float (&aux)[NQ], float (&ex)[NQ][3], int slab = 0) {
#pragma unroll 2      // two keys in flight: the second key's loads overlap the first key's FMAs
    for (int di = 0; di < ws; ++di) {
        const uint32_t a0 = rowbase + di * (kRowBytes * NS);
        float dp[NQ];
        if (MODE <= 2) {
            u64 v2[8];
            lds_slab16<NS>(a0, 1, slab, v2);
#pragma unroll
            for (int r = 0; r < NQ; ++r)
                if (CA_ON(r)) {
                    u64 t = nD2[r];                               // (-D, 0)
#pragma unroll
                    for (int i = 0; i < 8; ++i) t = fma2(dy[r][i], v2[i], t);
                    dp[r] = lane_sum<NS>(hsum2(t));              // -D sits on slab 0 only; rm is warp-uniform
                }
        }
        u64 k2[8];
        lds_slab16<NS>(a0, 0, slab, k2);
        float bk = 0.f;
        if (DIST) {
            u64 n = zero2();
#pragma unroll
            for (int i = 0; i < 8; ++i) n = fma2(k2[i], k2[i], n);
            bk = -0.5f * sl2 * hsum2(n);
        }
#pragma unroll
        for (int r = 0; r < NQ; ++r)
            if (CA_ON(r)) {
                u64 t = nL2[r];                                   // (-L, 0), log2 domain
                if (DIST) t = add2(t, pack2(bq[r] + bk, 0.f));
#pragma unroll
                for (int i = 0; i < 8; ++i) t = fma2(q[r][i], k2[i], t);
                const float chain = lane_sum<NS>(hsum2(t));
                if (MODE == 3) {
                    aux[r] = fmaxf(aux[r], chain);
                } else if (MODE == 4) {
                    const bool in = chain > 0.f;
                    const float tp = fmaxf(chain, 0.f);
                    sumds[r] += tp;
                    aux[r] = fmaf(tp, tp, aux[r]);
                    ex[r][0] += in ? 1.f : 0.f;
                    ex[r][1] = fminf(ex[r][1], in ? chain : INFINITY);
                    ex[r][2] = fmaxf(ex[r][2], in ? -INFINITY : chain);
                } else if (MODE == 5) {
                    u64 v2[8];
                    lds_slab16<NS>(a0, 1, slab, v2);
                    const float tp = fmaxf(chain, 0.f);
                    const float w = tp * tp;
                    const u64 w2 = pack2(w, w);
#pragma unroll
                    for (int i = 0; i < 8; ++i) dq[r][i] = fma2(w2, v2[i], dq[r][i]);
                } else if (MODE == 2) {
                    const float gg = fmaxf(chain, 0.f);
                    aux[r] = fmaf(gg, dp[r], aux[r]);
                    sumds[r] += gg;
                } else {
                    const float ds = (MODE == 0 ? fast_exp2(chain) : fmaxf(chain, 0.f)) * dp[r];
                    if (DIST) sumds[r] += ds;
                    const u64 d2 = pack2(ds, ds);
#pragma unroll
                    for (int i = 0; i < 8; ++i) dq[r][i] = fma2(d2, k2[i], dq[r][i]);
                }
            }
    }
}

template <bool DIST, int CPE, int NQ, int MODE, int NCRT = 16>
__global__ void __launch_bounds__(128, (NQ <= 2 ? 3 : 2)) dq_tiled_kernel(TileArgs a, const __grid_constant__ CUtensorMap mv,
                                                          const __grid_constant__ CUtensorMap msc) {
    constexpr int NS = NCRT <= 16 ? 1 : NCRT / 16;
    const Geo& g = a.g;
    const int ROWS = a.TH + 2 * (g.p + a.roff);
    const int NSTAGES = g.wsw + NQ - 1;
    const int w0 = blockIdx.x * NQ, h0 = blockIdx.y * a.TH, u = blockIdx.z;
    const float sl2 = MODE ? 0.5f * a.scale : a.scale * kLog2e;     // entmax: the chain is s/2 - tau
    bool settled[NQ];                                               // MODE 4: rows whose threshold is final
    if (MODE == 4) {
        // a block whose rows all have their final threshold leaves before any barrier or copy exists
        // (launched without a stage split and for one-slab units: thread = row)
        const int hh = h0 + (int)threadIdx.x;
        bool mine = true;
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            settled[r] = true;
            if (hh < g.H && has_pixel(g, hh, w0 + r)) settled[r] = __ldg(a.cs1 + (int64_t)u * g.Np + hh + g.H * (w0 + r)) != 0.f;
            mine = mine && settled[r];
        }
        if (__syncthreads_and(mine)) return;
    }
    CA_PIPE_PROLOGUE(false)
    const int slab = NS == 1 ? 0 : (lt % NS);
    const int lr = NS == 1 ? lt : (lt >> 5) * (32 / NS) + (lt & 31) / NS, h = h0 + lr;
    const bool active = h < g.H;

    u64 q[NQ][8], dy[NQ][8], dq[NQ][8];
    load_centre<CPE, NQ, NCRT>(a.c0, g, u, h, w0, active, sl2, q, 16 * slab);
    if (MODE <= 2) {
        load_centre<CPE, NQ, NCRT>(a.c1, g, u, h, w0, active, 1.f, dy, 16 * slab);
    } else {
#pragma unroll
        for (int r = 0; r < NQ; ++r)
#pragma unroll
            for (int i = 0; i < 8; ++i) dy[r][i] = zero2();
    }
    u64 nL2[NQ], nD2[NQ];
    float bq[NQ], sumds[NQ], aux[NQ], ex[NQ][3];
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        const bool ok = active && (has_pixel(g, h, w0 + r)) && slab == 0;       // row scalars enter the lane sums once
        const int64_t o = (int64_t)u * g.Np + h + g.H * (w0 + r);
        nL2[r] = pack2((ok && MODE != 3) ? -__ldg(a.cs0 + o) * (MODE ? 1.f : kLog2e) : 0.f, 0.f);
        nD2[r] = pack2((ok && MODE <= 1) ? -__ldg(a.cs1 + o) : 0.f, 0.f);
        sumds[r] = 0.f;
        aux[r] = MODE == 3 ? -INFINITY : 0.f;
        ex[r][0] = 0.f;
        ex[r][1] = INFINITY;
        ex[r][2] = -INFINITY;
        bq[r] = 0.f;
        if (DIST) {
            u64 n = zero2();
#pragma unroll
            for (int i = 0; i < 8; ++i) n = fma2(q[r][i], q[r][i], n);
            bq[r] = -0.5f * hsum2(n) / sl2;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) dq[r][i] = zero2();
    }

    CA_PIPE_LOOP({
        const int mask = stage_mask<NQ>(s, radius_w(g));
        CA_MASK_SWITCH(((1 << NQ) - 1), mask, (dq_stage<DIST, MK, NQ, MODE, NS>(smem_u32(pipe.vec(buf)) + (lr + a.roff) * (kRowBytes * NS), g.ws, mask,
                                                     sl2, q, dy, dq, nL2, nD2, bq, sumds, aux, ex, slab)));
    })

    if (MODE == 3) {
        // first threshold of the search: tau >= max - 1 always
#pragma unroll
        for (int r = 0; r < NQ; ++r)
            if (active && slab == 0 && has_pixel(g, h, w0 + r))
                a.ostats[(int64_t)u * g.Np + h + g.H * (w0 + r)] = aux[r] - 1.f + ca_poison;
        return;
    }
    if (MODE == 4) {
        // the quadratic sum_S (t - d)^2 = 1 solved on the support S of the current tau; final when tau + d has
        // the same support and the step was short against the distances it was computed from
#pragma unroll
        for (int r = 0; r < NQ; ++r)
            if (active && slab == 0 && has_pixel(g, h, w0 + r) && !settled[r]) {
                const int64_t o = (int64_t)u * g.Np + h + g.H * (w0 + r);
                const float n = ex[r][0], sa = sumds[r], sb = aux[r];
                float d = 0.f;
                bool same = true;
                if (n > 0.f) {
                    const float disc = fmaxf(fmaf(sa, sa, -n * (sb - 1.f)), 0.f);
                    d = (sa - sqrtf(disc)) / n;
                    same = (d >= 0.f ? d < ex[r][1] : d >= ex[r][2]) && d * n <= 0.5f * sa;
                    if (!same && a.iter >= 10) d = 0.5f * (sb - 1.f) / sa;     // late steps: Newton on the convex sum
                }
                float ntau, zero;
                unpack2(nL2[r], ntau, zero);
                a.ostats[o] = d - ntau + ca_poison;
                a.o1[o] = same ? 1.f : 0.f;
            }
        return;
    }
    if (MODE == 2) {
        // pre-pass of the entmax pullback: D = sum g*dP / sum g per query row (launched without a stage split)
#pragma unroll
        for (int r = 0; r < NQ; ++r)
            if (active && slab == 0 && has_pixel(g, h, w0 + r))
                a.ostats[(int64_t)u * g.Np + h + g.H * (w0 + r)] = (sumds[r] > 0.f ? aux[r] / sumds[r] : 0.f) + ca_poison;
        return;
    }
    if (a.nsplit == 2) {
        float* xch = reinterpret_cast<float*>(smem_al);
        if (part == 1) {
#pragma unroll
            for (int r = 0; r < NQ; ++r) {
                xch[(r * 17 + 16) * PT + lt] = sumds[r];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float x, y;
                    unpack2(dq[r][i], x, y);
                    xch[(r * 17 + 2 * i) * PT + lt] = x;
                    xch[(r * 17 + 2 * i + 1) * PT + lt] = y;
                }
            }
        }
        __syncthreads();
        if (part == 1) return;
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            sumds[r] += xch[(r * 17 + 16) * PT + lt];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                dq[r][i] = add2(dq[r][i], pack2(xch[(r * 17 + 2 * i) * PT + lt], xch[(r * 17 + 2 * i + 1) * PT + lt]));
        }
    }
    // dq = scale * (sum ds*k - [distance] sum(ds) * q);  q registers hold q*scale*log2(e) (entmax: q*scale/2)
    const float qfac = MODE ? 2.f : kLn2;
    CA_OUT_DISPATCH(
        _Pragma("unroll")
        for (int r = 0; r < NQ; ++r) {
            _Pragma("unroll")
            for (int i = 0; i < 8; ++i) {
                float x, y, qx, qy;
                unpack2(dq[r][i], x, y);
                unpack2(q[r][i], qx, qy);
                if (MODE == 5) {
                    x += ca_poison;
                    y += ca_poison;
                } else {
                    x = a.scale * x - (DIST ? sumds[r] * qx * qfac : 0.f) + ca_poison;
                    y = a.scale * y - (DIST ? sumds[r] * qy * qfac : 0.f) + ca_poison;
                }
                store_centre<CPE, NCRV, BF>(a.o0, g, u, h, w0, active, r, i, x, y, 16 * slab);
            }
        })
}

// =====================================================================
// Backward, key-owned: dk and dv of three key pixels per thread.  The stage
// rows carry (q | dy) of the query pixels plus their L and D.
// =====================================================================
template <bool DIST, int MASK, int NQ, bool ENT, int NS = 1>
__device__ __forceinline__ void dkdv_stage(uint32_t base, const float* Lb, const float* Db, int row0, int ws, int rm,
                                           float sl2, const u64 (&k)[NQ][8], const u64 (&v)[NQ][8], u64 (&dk)[NQ][8],
                                           u64 (&dv)[NQ][8], const float (&bk)[NQ], float (&sumds)[NQ], int slab = 0) {
#pragma unroll 1
    for (int di = 0; di < ws; ++di) {
        const int row = row0 + di;
        const uint32_t a0 = base + row * (kRowBytes * NS);
        // the row scalars enter the lane sums once: on slab 0
        const float nLj = (NS == 1 || slab == 0) ? -Lb[row] : 0.f, nDj = (NS == 1 || slab == 0) ? -Db[row] : 0.f;
        u64 y2[8];
        lds_slab16<NS>(a0, 1, slab, y2);
        float dp[NQ];
#pragma unroll
        for (int r = 0; r < NQ; ++r)
            if (CA_ON(r)) {
                u64 t = pack2(nDj, 0.f);
#pragma unroll
                for (int i = 0; i < 8; ++i) t = fma2(v[r][i], y2[i], t);
                dp[r] = lane_sum<NS>(hsum2(t));
            }
        u64 q2[8];
        lds_slab16<NS>(a0, 0, slab, q2);
        float bqj = 0.f;
        if (DIST) {
            u64 n = zero2();
#pragma unroll
            for (int i = 0; i < 8; ++i) n = fma2(q2[i], q2[i], n);
            bqj = -0.5f * sl2 * hsum2(n);
        }
#pragma unroll
        for (int r = 0; r < NQ; ++r)
            if (CA_ON(r)) {
                u64 t = pack2(DIST ? nLj + bk[r] + bqj : nLj, 0.f);
#pragma unroll
                for (int i = 0; i < 8; ++i) t = fma2(k[r][i], q2[i], t);
                const float chain = lane_sum<NS>(hsum2(t));
                float P, ds;
                if (!ENT) {
                    P = fast_exp2(chain);
                    ds = P * dp[r];
                } else {                                     // g = max(s/2 - tau, 0): P = g^2, dS = g*(dP - D)
                    const float gg = fmaxf(chain, 0.f);
                    P = gg * gg;
                    ds = gg * dp[r];
                }
                if (DIST) sumds[r] += ds;
                const u64 d2 = pack2(ds, ds), p2 = pack2(P, P);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    dk[r][i] = fma2(d2, q2[i], dk[r][i]);
                    dv[r][i] = fma2(p2, y2[i], dv[r][i]);
                }
            }
    }
}

template <bool DIST, int CPE, int NQ, bool ENT, int NCRT = 16>
__global__ void __launch_bounds__(128, (NQ <= 2 ? 3 : 2)) dkdv_tiled_kernel(TileArgs a, const __grid_constant__ CUtensorMap mv,
                                                            const __grid_constant__ CUtensorMap msc) {
    constexpr int NS = NCRT <= 16 ? 1 : NCRT / 16;
    const Geo& g = a.g;
    const int ROWS = a.TH + 2 * (g.p + a.roff);
    const int NSTAGES = g.wsw + NQ - 1;
    const int w0 = blockIdx.x * NQ, h0 = blockIdx.y * a.TH, u = blockIdx.z;
    const float sl2 = ENT ? 0.5f * a.scale : a.scale * kLog2e;      // entmax: the chain is s/2 - tau
    CA_PIPE_PROLOGUE(true)
    const int slab = NS == 1 ? 0 : (lt % NS);
    const int lr = NS == 1 ? lt : (lt >> 5) * (32 / NS) + (lt & 31) / NS, h = h0 + lr;
    const bool active = h < g.H;

    u64 k[NQ][8], v[NQ][8], dk[NQ][8], dv[NQ][8];
    load_centre<CPE, NQ, NCRT>(a.c0, g, u, h, w0, active, sl2, k, 16 * slab);
    load_centre<CPE, NQ, NCRT>(a.c1, g, u, h, w0, active, 1.f, v, 16 * slab);
    float bk[NQ], sumds[NQ];
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        sumds[r] = 0.f;
        bk[r] = 0.f;
        if (DIST) {
            u64 n = zero2();
#pragma unroll
            for (int i = 0; i < 8; ++i) n = fma2(k[r][i], k[r][i], n);
            bk[r] = -0.5f * hsum2(n) / sl2;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            dk[r][i] = zero2();
            dv[r][i] = zero2();
        }
    }

    CA_PIPE_LOOP({
        const int mask = stage_mask<NQ>(s, radius_w(g));
        CA_MASK_SWITCH(((1 << NQ) - 1), mask, (dkdv_stage<DIST, MK, NQ, ENT, NS>(smem_u32(pipe.vec(buf)), pipe.sc0(buf), pipe.sc1(buf),
                                                      lr + a.roff, g.ws, mask, sl2, k, v, dk, dv, bk, sumds, slab)));
    })

    if (a.nsplit == 2) {
        float* xch = reinterpret_cast<float*>(smem_al);
        if (part == 1) {
#pragma unroll
            for (int r = 0; r < NQ; ++r) {
                xch[(r * 33 + 32) * PT + lt] = sumds[r];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float x, y;
                    unpack2(dk[r][i], x, y);
                    xch[(r * 33 + 2 * i) * PT + lt] = x;
                    xch[(r * 33 + 2 * i + 1) * PT + lt] = y;
                    unpack2(dv[r][i], x, y);
                    xch[(r * 33 + 16 + 2 * i) * PT + lt] = x;
                    xch[(r * 33 + 17 + 2 * i) * PT + lt] = y;
                }
            }
        }
        __syncthreads();
        if (part == 1) return;
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            sumds[r] += xch[(r * 33 + 32) * PT + lt];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                dk[r][i] = add2(dk[r][i], pack2(xch[(r * 33 + 2 * i) * PT + lt], xch[(r * 33 + 2 * i + 1) * PT + lt]));
                dv[r][i] = add2(dv[r][i], pack2(xch[(r * 33 + 16 + 2 * i) * PT + lt], xch[(r * 33 + 17 + 2 * i) * PT + lt]));
            }
        }
    }
    // dk = scale * (sum ds*q - [distance] sum(ds) * k);  k registers hold k*scale*log2(e)
    CA_OUT_DISPATCH(
        _Pragma("unroll")
        for (int r = 0; r < NQ; ++r) {
            _Pragma("unroll")
            for (int i = 0; i < 8; ++i) {
                float x, y, kx, ky, vx, vy;
                unpack2(dk[r][i], x, y);
                unpack2(k[r][i], kx, ky);
                unpack2(dv[r][i], vx, vy);
                x = a.scale * x - (DIST ? sumds[r] * kx * (ENT ? 2.f : kLn2) : 0.f) + ca_poison;
                y = a.scale * y - (DIST ? sumds[r] * ky * (ENT ? 2.f : kLn2) : 0.f) + ca_poison;
                store_centre<CPE, NCRV, BF>(a.o0, g, u, h, w0, active, r, i, x, y, 16 * slab);
                store_centre<CPE, NCRV, BF>(a.o1, g, u, h, w0, active, r, i, vx + ca_poison, vy + ca_poison, 16 * slab);
            }
        })
}

// mode 0: softmax; 1: entmax; 2: entmax pre-pass (writes D, needs no D and no dq).  The entmax
// variants exist for four centre pixels per thread and run without a stage split.
int run_dq(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* dy, const float* stats,
           const float* D, const float* kv, float* dq, cudaStream_t st, int mode = 0, float* Dout = nullptr) {
    Launch L{};
    const int ns = slabs_of(g);
    if (ns > 1 && mode) return CA_ERR_UNSUPPORTED;             // the entmax variants exist for one-slab units
    if (mode >= 3) return CA_ERR_UNSUPPORTED;                  // the forward's sweeps go through run_entmax_fwd_sweep
    // two query columns per thread measured faster than four at every size for the softmax dq sweep of one-slab
    // units (160 registers, three blocks per SM, against 255 and two)
    const int nq = mode ? 4 : (ns > 1 ? (g.ws <= 9 ? 2 : 4) : tune_int("CIRCATT_DQ_NQ", 2));
    int rc = prepare(g, P, nq, 17 * nq, "CIRCATT_DQ_WARPS", kv, nullptr, &L, mode == 0 && ns == 1 ? 2 : 1, 4, ns);
    if (rc) return rc;
    L.a.scale = scale; L.a.c0 = q; L.a.c1 = dy; L.a.cs0 = stats; L.a.cs1 = D; L.a.o0 = dq; L.a.ostats = Dout;
    if (ns == 2 && nq == 2) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 2, 0, 32, L, st);
    else if (ns == 2) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 4, 0, 32, L, st);
    else if (ns == 4 && nq == 2) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 2, 0, 64, L, st);
    else if (ns == 4) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 4, 0, 64, L, st);
    else if (mode == 2) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 4, 2, 16, L, st);
    else if (mode == 1) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 4, 1, 16, L, st);
    else if (nq == 2) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 2, 0, 16, L, st);
    else CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 4, 0, 16, L, st);
    CA_CHECK_LAUNCH("tiled dq kernel");
    return CA_OK;
}

// One sweep of the entmax forward over the packed (k|v): mode 3 row maximum -> first threshold (tau),
// 4 one step of the threshold search (tau and `settled` updated in place), 5 y = sum max(s/2 - tau, 0)^2 v.
int run_entmax_fwd_sweep(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* kv,
                         float* tau, float* settled, float* y, int mode, int iter, cudaStream_t st) {
    Launch L{};
    if (slabs_of(g) > 1) return CA_ERR_UNSUPPORTED;
    int rc = prepare(g, P, 4, 17 * 4, "CIRCATT_DQ_WARPS", kv, nullptr, &L, 1, 4, 1);
    if (rc) return rc;
    L.a.scale = scale; L.a.c0 = q; L.a.cs0 = tau; L.a.cs1 = settled; L.a.o0 = y; L.a.o1 = settled; L.a.ostats = tau;
    L.a.iter = iter;
    if (mode == 3) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 4, 3, 16, L, st);
    else if (mode == 4) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 4, 4, 16, L, st);
    else CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 4, 5, 16, L, st);
    CA_CHECK_LAUNCH("tiled entmax forward sweep");
    return CA_OK;
}

int run_dkdv(const Geo& g, const Padded& P, float scale, int dist, const float* k, const float* v, const float* qdy,
             const float* planes, float* dk, float* dv, cudaStream_t st, bool entmax = false) {
    Launch L{};
    const int ns = slabs_of(g);
    if (ns > 1 && entmax) return CA_ERR_UNSUPPORTED;
    const int nq = 3;
    int rc = prepare(g, P, nq, 33 * nq, "CIRCATT_DKDV_WARPS", qdy, planes, &L, ns == 1 ? 2 : 1, 4, ns);
    if (rc) return rc;
    L.a.scale = scale; L.a.c0 = k; L.a.c1 = v; L.a.o0 = dk; L.a.o1 = dv;
    if (ns == 2) CA_DIST_CPE_NQ(dkdv_tiled_kernel, dist, g.cpe, 3, false, 32, L, st);
    else if (ns == 4) CA_DIST_CPE_NQ(dkdv_tiled_kernel, dist, g.cpe, 3, false, 64, L, st);
    else if (entmax) CA_DIST_CPE_NQ(dkdv_tiled_kernel, dist, g.cpe, 3, true, 16, L, st);
    else CA_DIST_CPE_NQ(dkdv_tiled_kernel, dist, g.cpe, 3, false, 16, L, st);
    CA_CHECK_LAUNCH("tiled dk/dv kernel");
    return CA_OK;
}

}  // namespace

// ---------------------------------------------------------------- entry points of this file
size_t tiled_fwd_workspace(const Geo& gin) {
    Geo g;
    if (!fold_geo(gin, &g)) return 0;
    if (!tiled_shape_ok(g)) return 0;
    return (padded_of(g).pair_floats + (size_t)g.Np * g.units) * sizeof(float);
}

size_t tiled_bwd_stage_workspace(const Geo& gin) {
    Geo g;
    if (!fold_geo(gin, &g)) return 0;
    if (!tiled_shape_ok(g)) return 0;
    const Padded P = padded_of(g);
    return (P.pair_floats + P.plane_floats) * sizeof(float);
}

size_t tiled_bwd_workspace(const Geo& gin) {
    Geo g;
    if (!fold_geo(gin, &g)) return 0;
    if (!tiled_shape_ok(g)) return 0;
    const Padded P = padded_of(g);
    return (2 * P.pair_floats + P.plane_floats) * sizeof(float);
}

int tiled_attention_fwd(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                        float* y, float* nz, float* stats, void* workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g) || (nz && g.Wk != g.W)) return CA_ERR_UNSUPPORTED;
    if (!workspace) { set_error("workspace of ca_attention_fwd_workspace() bytes is NULL"); return CA_ERR_NULL; }
    const Padded P = padded_of(g);
    float* kv = static_cast<float*>(workspace);
    if (nz && !stats) stats = kv + P.pair_floats;         // scratch statistics behind the packed pair
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1;
    pa.src[0] = k; pa.src[1] = v; pa.dst[0] = kv;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    Launch L{};
    const int ns = slabs_of(g);
    // four columns per thread, or two when the grid is small or the window is short (with ws <= 9 most
    // stages of a four-column tile pair with only some of its columns: measured 18 % faster at ws 7)
    const int nq = g.ws <= 9 ? tune_int("CIRCATT_FWD_NQ", 2) : (ns > 1 ? 4 : pick_nq(g, 4, 2, "CIRCATT_FWD_NQ"));
    if ((rc = prepare(g, P, nq, 18 * nq, "CIRCATT_FWD_WARPS", kv, nullptr, &L, ns == 1 ? 2 : 1, 4, ns))) return rc;
    L.a.scale = scale; L.a.c0 = q; L.a.o0 = y; L.a.ostats = stats;
#define CA_FWD2(DCV, EX, NQV, NCRV_)                                                            \
    do {                                                                                 \
        if (g.cpe == 1) {                                                                \
            if (dist) CA_LAUNCH_TILED((fwd_tiled_kernel<DCV, true, 1, EX, NQV, NCRV_>), L, st); \
            else CA_LAUNCH_TILED((fwd_tiled_kernel<DCV, false, 1, EX, NQV, NCRV_>), L, st);     \
        } else {                                                                         \
            if (dist) CA_LAUNCH_TILED((fwd_tiled_kernel<DCV, true, 2, EX, NQV, NCRV_>), L, st); \
            else CA_LAUNCH_TILED((fwd_tiled_kernel<DCV, false, 2, EX, NQV, NCRV_>), L, st);     \
        }                                                                                \
    } while (0)
#define CA_FWD(DCV)                                                                      \
    do {                                                                                 \
        if (nq == 2) CA_FWD2(DCV, true, 2, 16);                                          \
        else CA_FWD2(DCV, true, 4, 16);                                                  \
    } while (0)
    // wide units: chunks of 7 or 5 keys where they divide the window, else chunks of four plus a tail
    if (ns == 2 && nq == 2 && g.ws % 7 == 0) CA_FWD2(7, true, 2, 32);
    else if (ns == 4 && nq == 2 && g.ws % 7 == 0) CA_FWD2(7, true, 2, 64);
    else if (ns == 2 && nq == 4 && g.ws % 7 == 0) CA_FWD2(7, true, 4, 32);       // windows 21, 35, 49, 63
    else if (ns == 4 && nq == 4 && g.ws % 7 == 0) CA_FWD2(7, true, 4, 64);
    else if (ns == 2 && nq == 4 && g.ws % 5 == 0) CA_FWD2(5, true, 4, 32);       // windows 15, 25, 45, 55
    else if (ns == 4 && nq == 4 && g.ws % 5 == 0) CA_FWD2(5, true, 4, 64);
    else if (ns == 2 && nq == 2) CA_FWD2(4, false, 2, 32);
    else if (ns == 2) CA_FWD2(4, false, 4, 32);
    else if (ns == 4 && nq == 2) CA_FWD2(4, false, 2, 64);
    else if (ns == 4) CA_FWD2(4, false, 4, 64);
    else if (g.ws % 7 == 0) CA_FWD(7);
    else if (g.ws % 5 == 0) CA_FWD(5);
    else if (g.ws % 3 == 0) CA_FWD(3);
    else if (nq == 2) CA_FWD2(4, false, 2, 16);
    else CA_FWD2(4, false, 4, 16);
#undef CA_FWD2
#undef CA_FWD
    CA_CHECK_LAUNCH("tiled forward kernel");
    if (nz) return tiled_emit_a(g, scale, dist, q, stats, nz, workspace, st);
    return CA_OK;
}

int tiled_attention_bwd_dq(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                           const float* dy, const float* stats, const float* D, float* dq, void* workspace,
                           cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g)) return CA_ERR_UNSUPPORTED;
    if (!workspace) { set_error("workspace of ca_attention_bwd_stage_workspace() bytes is NULL"); return CA_ERR_NULL; }
    const Padded P = padded_of(g);
    float* kv = static_cast<float*>(workspace);
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1;
    pa.src[0] = k; pa.src[1] = v; pa.dst[0] = kv;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    return run_dq(g, P, scale, dist, q, dy, stats, D, kv, dq, st);
}

int tiled_attention_bwd_dkdv(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                             const float* dy, const float* stats, const float* D, float* dk, float* dv,
                             void* workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g)) return CA_ERR_UNSUPPORTED;
    if (!workspace) { set_error("workspace of ca_attention_bwd_stage_workspace() bytes is NULL"); return CA_ERR_NULL; }
    const Padded P = padded_of(g);
    float* qdy = static_cast<float*>(workspace);
    float* planes = qdy + P.pair_floats;
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1;
    pa.src[0] = q; pa.src[1] = dy; pa.dst[0] = qdy;
    pa.planes = planes; pa.stats = stats; pa.stat_mul = kLog2e; pa.Din = D;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    return run_dkdv(g, P, scale, dist, k, v, qdy, planes, dk, dv, st);
}

// Helper stream (one per host thread and device) on which the dk/dv sweep of a small problem runs
// next to the dq sweep: neither fills the GPU alone.  It is forked from and joined
// back to the caller's stream with events, so the caller sees ordinary stream order.  The
// stream and its two events belong to the calling host thread, so callers on different threads
// (and streams) neither share them nor wait for each other.
struct ForkJoin {
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};
static thread_local ForkJoin g_fork[64];

static ForkJoin* fork_join_for_current_device() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    ForkJoin& f = g_fork[dev];
    if (!f.side) {
        if (cudaStreamCreateWithFlags(&f.side, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&f.fork, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&f.join, cudaEventDisableTiming) != cudaSuccess) {
            f.side = nullptr;
            cudaGetLastError();
            return nullptr;
        }
    }
    return &f;
}

// Whole backward in three launches: pack (both pairs, D, planes), dq, dk/dv.
int tiled_attention_bwd(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                        const float* y, const float* dy, const float* stats, float* D, float* dq, float* dk,
                        float* dv, void* workspace, const void* fwd_workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g) || g.Wk != g.W) return CA_ERR_UNSUPPORTED;
    if (!workspace) { set_error("workspace is NULL"); return CA_ERR_NULL; }
    const Padded P = padded_of(g);
    float* kv = static_cast<float*>(workspace);
    float* qdy = kv + P.pair_floats;
    float* planes = qdy + P.pair_floats;
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp;
    if (fwd_workspace) {
        // the forward of the same problem left its packed (k|v) at the start of its workspace: only
        // (q|dy) and the planes are packed here
        kv = const_cast<float*>(static_cast<const float*>(fwd_workspace));
        pa.npairs = 1;
        pa.src[0] = q; pa.src[1] = dy;
        pa.dst[0] = qdy;
    } else {
        pa.npairs = 2;
        pa.src[0] = k; pa.src[1] = v; pa.src[2] = q; pa.src[3] = dy;
        pa.dst[0] = kv; pa.dst[1] = qdy;
    }
    pa.planes = planes; pa.stats = stats; pa.stat_mul = kLog2e; pa.y = y; pa.dy = dy; pa.Dout = D;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    const bool small = (long)g.Np * g.units < 2048L * sm_count();      // fewer than ~4 CTAs per SM per sweep
    if (small && tune_int("CIRCATT_CONCURRENT", 1)) {
        ForkJoin* f = fork_join_for_current_device();
        if (f && cudaEventRecord(f->fork, st) == cudaSuccess && cudaStreamWaitEvent(f->side, f->fork, 0) == cudaSuccess) {
            rc = run_dkdv(g, P, scale, dist, k, v, qdy, planes, dk, dv, f->side);
            int rc2 = run_dq(g, P, scale, dist, q, dy, stats, D, kv, dq, st);
            cudaError_t e = cudaEventRecord(f->join, f->side);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(st, f->join, 0);
            if (e != cudaSuccess) return cuda_fail(e, "joining the helper stream");
            return rc ? rc : rc2;
        }
        cudaGetLastError();
    }
    if ((rc = run_dq(g, P, scale, dist, q, dy, stats, D, kv, dq, st))) return rc;
    return run_dkdv(g, P, scale, dist, k, v, qdy, planes, dk, dv, st);
}

// Entmax-1.5 backward on the fused kernels.  Unlike the softmax, D = sum g*dP / sum g is not dy.y, so
// a pre-pass over the packed (k|v) computes it first: pack (k|v) -> pre-pass -> pack (q|dy) + planes
// (tau, D) -> dq and dk/dv.  `stats` holds tau.
int tiled_attention_bwd_entmax(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                               const float* dy, const float* stats, float* D, float* dq, float* dk, float* dv,
                               void* workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g) || g.Wk != g.W || g.bf16) return CA_ERR_UNSUPPORTED;
    if (!workspace) { set_error("workspace is NULL"); return CA_ERR_NULL; }
    const Padded P = padded_of(g);
    float* kv = static_cast<float*>(workspace);
    float* qdy = kv + P.pair_floats;
    float* planes = qdy + P.pair_floats;
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1;
    pa.src[0] = k; pa.src[1] = v; pa.dst[0] = kv;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    if ((rc = run_dq(g, P, scale, dist, q, dy, stats, nullptr, kv, nullptr, st, 2, D))) return rc;
    PackArgs pb{};
    pb.g = g; pb.pp = P.pp; pb.Hp = P.Hp; pb.npairs = 1;
    pb.src[0] = q; pb.src[1] = dy; pb.dst[0] = qdy;
    pb.planes = planes; pb.stats = stats; pb.stat_mul = 1.f; pb.Din = D;
    if ((rc = launch_pack(pb, st))) return rc;
    if ((rc = run_dq(g, P, scale, dist, q, dy, stats, D, kv, dq, st, 1))) return rc;
    return run_dkdv(g, P, scale, dist, k, v, qdy, planes, dk, dv, st, true);
}

// The 1.5-entmax forward in flash mode without A-sized memory: the packed (k|v) is swept once for the row
// maxima, a fixed number of times for the thresholds (blocks whose rows are all final leave at once) and once
// for y.  `stats` (nullable) receives tau and doubles as the search's state; the `settled` plane and a tau plane
// for callers without `stats` live behind the pair in the workspace (tiled_fwd_entmax_workspace bytes).
size_t tiled_fwd_entmax_workspace(const Geo& gin) {
    Geo g;
    if (!fold_geo(gin, &g)) return 0;
    if (!tiled_shape_ok(g) || g.bf16 || slabs_of(g) > 1) return 0;
    return padded_of(g).pair_floats * sizeof(float) + 2 * (size_t)g.Np * g.units * sizeof(float);
}

int tiled_attention_fwd_entmax(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                               float* y, float* stats, void* workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g) || g.Wk != g.W || g.bf16 || slabs_of(g) > 1) return CA_ERR_UNSUPPORTED;
    if (!workspace) return CA_ERR_UNSUPPORTED;
    const Padded P = padded_of(g);
    float* kv = static_cast<float*>(workspace);
    float* settled = kv + P.pair_floats;
    if (!stats) stats = settled + (size_t)g.Np * g.units;       // a caller that does not want tau
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1;
    pa.src[0] = k; pa.src[1] = v; pa.dst[0] = kv;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    cudaError_t e = cudaMemsetAsync(settled, 0, (size_t)g.Np * g.units * sizeof(float), st);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync");
    if ((rc = run_entmax_fwd_sweep(g, P, scale, dist, q, kv, stats, settled, nullptr, 3, 0, st))) return rc;
    // the support iteration ends after 3-5 steps on ordinary rows; the steps past the tenth are Newton steps,
    // which converge for every row
    for (int it = 0; it < kEntmaxFwdSteps; ++it)
        if ((rc = run_entmax_fwd_sweep(g, P, scale, dist, q, kv, stats, settled, nullptr, 4, it, st))) return rc;
    return run_entmax_fwd_sweep(g, P, scale, dist, q, kv, stats, settled, y, 5, 0, st);
}

}  // namespace ca
