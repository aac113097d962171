// Backward sweeps of the tiled kernels and the sweeps of the entmax forward (compiled by bwd_exact.cu and bwd_any.cu; the
// scheme is described in tiled.cu).
#include "tile_common.cuh"

namespace ca {
namespace {

#define CA_MASK_SWITCH(FULL, mask, CALL)                            \
    if ((mask) == (FULL)) { constexpr int MK = (FULL); CALL; }      \
    else { constexpr int MK = 0; CALL; }

// =====================================================================
// Backward, query-owned: dq.  The s chain starts at -L (log2 domain) and the
// dP chain at -D, so P = 2^chain and dS = P * chain'.
// =====================================================================
// MODE 0: softmax, P = 2^chain.  MODE 1: 1.5-entmax, g = max(chain, 0) with the chain = s/2 - tau, dS = g*(dP - D).
// MODE 2: the entmax pre-pass: only num += g*dP and den += g (in aux and sumds), D = num/den.
// The same query-owned sweep serves the entmax forward, which has no dy: MODE 3 the largest s/2 of a stage (in aux);
// MODE 4 one step of the threshold search: with t = chain = s/2 - tau, the sum of max(t, 0) (sumds), of its
// square (aux), the size of the support {t > 0}, its smallest member and the largest t outside (ex[0..2]);
// MODE 5 the apply: dq (here y) += max(chain, 0)^2 * v.
// STORE: the weights P and dS also go to memory, for dkdv_stored_kernel: `w[r]` is where this lane's entry of the stage's
// first key goes (lanes of slab 0 write P, of slab 1 dS), `step` the words to the next key's.
template <bool DIST, int MASK, int NQ, int MODE, int NS, bool STORE>
__device__ __forceinline__ void dq_stage(uint32_t rowbase, int ws, int rm, float sl2, const u64 (&q)[NQ][8],
                                         const u64 (&dy)[NQ][8], u64 (&dq)[NQ][8], const u64 (&nL2)[NQ],
                                         const u64 (&nD2)[NQ], const float (&bq)[NQ], float (&sumds)[NQ],
                                         float (&aux)[NQ], float (&ex)[NQ][3], int slab, float* (&w)[NQ], int step, int keep) {
#pragma unroll (NQ == 1 ? 4 : 2)      // keys in flight: the next key's loads overlap this key's FMAs
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
        if (DIST) bk = -0.5f * sl2 * lds_norm(a0, 128 * NS, slab);
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
#pragma unroll
                    for (int i = 0; i < 8; ++i) dq[r][i] = outer2(w, v2[i], dq[r][i]);
                } else if (MODE == 2) {
                    const float gg = fmaxf(chain, 0.f);
                    aux[r] = fmaf(gg, dp[r], aux[r]);
                    sumds[r] += gg;
                } else {
                    const float P = MODE == 0 ? fast_exp2(chain) : fmaxf(chain, 0.f);
                    const float ds = P * dp[r];
                    if (STORE) {
                        if ((keep >> r) & 1) *w[r] = slab ? ds : P;
                        w[r] += step;
                    }
                    if (DIST) sumds[r] += ds;
#pragma unroll
                    for (int i = 0; i < 8; ++i) dq[r][i] = outer2(ds, k2[i], dq[r][i]);
                }
            }
    }
}

template <bool DIST, int CPE, int NQ, int MODE, int NCRT = 16, bool STORE = false>
__global__ void __launch_bounds__(128, (NQ == 1 ? 5 : NQ == 2 ? 3 : 2)) dq_tiled_kernel(TileArgs a, const __grid_constant__ CUtensorMap mv,
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
    CA_PIPE_PROLOGUE(false, (NS == 1 ? kParts : 1))
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

    // MODE 3: the largest scores of eight classes of keys, window columns dealt out in turn (the stage's maxima always
    // enter the same register: the others move up)
    constexpr int kClasses = 8;
    float top[NQ][kClasses];
    if (MODE == 3) {
#pragma unroll
        for (int r = 0; r < NQ; ++r)
#pragma unroll
            for (int i = 0; i < kClasses; ++i) top[r][i] = -INFINITY;
    }
    int keep = 0;                                // STORE: columns whose weights this lane writes
    if (STORE) {
#pragma unroll
        for (int r = 0; r < NQ; ++r)
            if (active && slab < 2 && has_pixel(g, h, w0 + r)) keep |= 1 << r;
    }
    CA_PIPE_LOOP({
        const int mask = stage_mask<NQ>(s, radius_w(g));
        float* kept[NQ];
        if (STORE) {
            _Pragma("unroll")
            for (int r = 0; r < NQ; ++r)
                kept[r] = a.o1 + ((int64_t)(2 * u + (slab & 1)) * g.K + (s - r) * g.ws) * g.Np + h + g.H * (w0 + r);
        }
        CA_MASK_SWITCH(((1 << NQ) - 1), mask, (dq_stage<DIST, MK, NQ, MODE, NS, STORE>(pipe.vec(buf, a) + (lr + a.roff) * (kRowBytes * NS), g.ws, mask,
                                                     sl2, q, dy, dq, nL2, nD2, bq, sumds, aux, ex, slab, kept, g.Np, keep)));
        if (MODE == 3) {
            _Pragma("unroll")
            for (int r = 0; r < NQ; ++r) {
                const float first = fmaxf(top[r][0], aux[r]);
                _Pragma("unroll")
                for (int i = 0; i + 1 < kClasses; ++i) top[r][i] = top[r][i + 1];
                top[r][kClasses - 1] = first;
                aux[r] = -INFINITY;
            }
        }
    })

    if (MODE == 3) {
        // first threshold of the search
#pragma unroll
        for (int r = 0; r < NQ; ++r)
            if (active && slab == 0 && has_pixel(g, h, w0 + r))
                a.ostats[(int64_t)u * g.Np + h + g.H * (w0 + r)] = entmax_start(top[r]) + ca_poison;
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
    if (NS == 1 && a.nsplit > 1) {                                    // parts 1.. publish their partial sums, part 0 adds them up
        float* xch = reinterpret_cast<float*>(smem_al) + (size_t)max(part - 1, 0) * (17 * NQ) * PT;
        if (part > 0) {
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
        if (part > 0) return;
#pragma unroll 1
        for (int o = 1; o < a.nsplit; ++o, xch += (17 * NQ) * PT)
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
__device__ __forceinline__ void dkdv_stage(uint32_t a0, uint32_t sa, uint32_t plane, int ws, int rm,
                                           float sl2, const u64 (&k)[NQ][8], const u64 (&v)[NQ][8], u64 (&dk)[NQ][8],
                                           u64 (&dv)[NQ][8], const float (&bk)[NQ], float (&sumds)[NQ], int slab = 0) {
    // row statistics as C++ loads: the compiler places them, the vector loads are pinned (2 % at ws 21)
    const float* Lr = reinterpret_cast<const float*>(__cvta_shared_to_generic(sa));
    const float* Dr = reinterpret_cast<const float*>(__cvta_shared_to_generic(sa + plane));
#pragma unroll (NQ == 1 ? 2 : 1)
    for (int di = 0; di < ws; ++di) {
        // the row scalars enter the lane sums once: on slab 0
        const float nLj = (NS == 1 || slab == 0) ? -*Lr : 0.f, nDj = (NS == 1 || slab == 0) ? -*Dr : 0.f;
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
        if (DIST) bqj = -0.5f * sl2 * lds_norm(a0, 128 * NS, slab);
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
                // dv first: its vector was loaded first and is free again sooner (1024 x 1024, 2 units, ws 21: 3009 -> 2966 us)
#pragma unroll
                for (int i = 0; i < 8; ++i) dv[r][i] = outer2(P, y2[i], dv[r][i]);
#pragma unroll
                for (int i = 0; i < 8; ++i) dk[r][i] = outer2(ds, q2[i], dk[r][i]);
            }
        a0 += kRowBytes * NS;
        ++Lr;
        ++Dr;
    }
}

template <bool DIST, int CPE, int NQ, bool ENT, int NCRT = 16>
__global__ void __launch_bounds__(128, (NQ == 1 ? 4 : NQ == 2 ? 3 : 2)) dkdv_tiled_kernel(TileArgs a, const __grid_constant__ CUtensorMap mv,
                                                            const __grid_constant__ CUtensorMap msc) {
    constexpr int NS = NCRT <= 16 ? 1 : NCRT / 16;
    const Geo& g = a.g;
    const int ROWS = a.TH + 2 * (g.p + a.roff);
    const int NSTAGES = g.wsw + NQ - 1;
    const int w0 = blockIdx.x * NQ, h0 = blockIdx.y * a.TH, u = blockIdx.z;
    const float sl2 = ENT ? 0.5f * a.scale : a.scale * kLog2e;      // entmax: the chain is s/2 - tau
    CA_PIPE_PROLOGUE(true, (NS == 1 ? kParts : 1))
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
        CA_MASK_SWITCH(((1 << NQ) - 1), mask, (dkdv_stage<DIST, MK, NQ, ENT, NS>(pipe.vec(buf, a) + (lr + a.roff) * (kRowBytes * NS),
                                                      pipe.sc0(buf, a, ROWS) + (lr + a.roff) * 4, pipe.plane_bytes(ROWS), g.ws, mask, sl2, k, v, dk, dv, bk, sumds, slab)));
    })

    if (NS == 1 && a.nsplit > 1) {
        float* xch = reinterpret_cast<float*>(smem_al) + (size_t)max(part - 1, 0) * (33 * NQ) * PT;
        if (part > 0) {
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
        if (part > 0) return;
#pragma unroll 1
        for (int o = 1; o < a.nsplit; ++o, xch += (33 * NQ) * PT)
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

// =====================================================================
// dk and dv of wide units from the stored weights of the dq sweep: dv = sum P dy, dk = scale * sum dS q over the queries
// whose window holds the key.  Recomputing P and dS takes two of the four contractions, two shuffles for each of their
// scores and an exp2 in each of the NS lanes; stored they are 8 bytes per pair, written and read once, for
// 64 * NS FMAs saved.  [unit][P | dS][window entry][query pixel]: lanes on consecutive rows write and read consecutive words.
// The entry that key i needs of query j is the one at offset i - j (window symmetry).  The weights of the next stage are on
// their way to shared memory while one is used; pairs that do not exist weigh zero.  (Loaded into registers two keys
// ahead they were waited for in the move to the next key's: 1031 us, 320 x 320, 8 units of 64 channels, ws 7.)
// Bound: shared-memory reads, 32 cycles of vectors for NQ columns, next to 32 packed FMAs (8 cycles) per column.
// =====================================================================
// Copies four bytes to shared memory, or zero.
__device__ __forceinline__ void cp_async4_or_zero(uint32_t dst, const float* src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(on ? 4 : 0) : "memory");
}

template <bool DIST, int CPE, int NQ, int NCRT>
__global__ void __launch_bounds__(128, (NQ == 1 ? 5 : 3)) dkdv_stored_kernel(TileArgs a, const __grid_constant__ CUtensorMap mv,
                                                            const __grid_constant__ CUtensorMap msc) {
    constexpr int NS = NCRT / 16;
    constexpr int RW = 32 / NS;
    const Geo& g = a.g;
    const int ROWS = a.TH + 2 * (g.p + a.roff);
    const int NSTAGES = g.wsw + NQ - 1;
    const int w0 = blockIdx.x * NQ, h0 = blockIdx.y * a.TH, u = blockIdx.z, p = g.p;
    CA_PIPE_PROLOGUE(false, 1)
    const int slab = lt % NS, lr = (lt >> 5) * RW + (lt & 31) / NS, h = h0 + lr;
    const bool active = h < g.H;

    const float* unit = a.cs0 + (int64_t)(2 * u) * g.K * g.Np;
    const int64_t second = (int64_t)g.K * g.Np;                  // from P to dS
    const int64_t column = (int64_t)g.ws * g.Np;                 // from one window column's entries to the next's
    const int half = g.ws * (2 * NQ * RW * 4);                   // bytes of a stage's weights: [key row][P | dS][column][row]
    const uint32_t mine = smem_u32(smem_al) + a.extra_off + (lt >> 5) * (2 * half) + ((lt & 31) / NS) * 4;
    // starts the copies of the weights of stage s with the centre columns; the lanes of a pixel share them out
    auto fetch = [&](int s, int tb) {
        int wq = w0 - p + s;
        for (; wq < 0; wq += g.W) {}
        for (; wq >= g.W; wq -= g.W) {}
        const float* stage = unit + (int64_t)((2 * p - s) * g.ws + 2 * p) * g.Np + (int64_t)g.H * wq;
#pragma unroll
        for (int c0 = 0; c0 < 2 * NQ; c0 += NS) {
            const int c = c0 + slab, r = c % NQ;
            if (c >= 2 * NQ) break;
            const bool on = active && w0 + r < g.W && s >= r && s <= r + 2 * p;
            const float* at = on ? stage + r * column + (c >= NQ ? second : 0) : unit;
            uint32_t to = mine + tb * half + c * (RW * 4);
            int hq = h - p;
            for (int di = 0; di < g.ws; ++di) {
                cp_async4_or_zero(to, at + (on ? wrap_axis(hq, g.H) : 0), on);
                at -= on ? g.Np : 0;
                to += 2 * NQ * RW * 4;
                ++hq;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    u64 dk[NQ][8], dv[NQ][8];
    float sumds[NQ];
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        sumds[r] = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            dk[r][i] = zero2();
            dv[r][i] = zero2();
        }
    }
    fetch(0, 0);

    CA_PIPE_LOOP({
        uint32_t a0 = pipe.vec(buf, a) + (lr + a.roff) * (kRowBytes * NS);
        uint32_t at = mine + (s & 1) * half;
        if (s + 1 < s_end) {
            fetch(s + 1, (s + 1) & 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
        const int mask = stage_mask<NQ>(s, p);
        auto sweep = [&](auto full_tag) {
            constexpr bool FULL = decltype(full_tag)::value;
            _Pragma("unroll 2")
            for (int di = 0; di < g.ws; ++di) {
                u64 q2[8];
                u64 y2[8];
                lds_slab16<NS>(a0, 0, slab, q2);
                lds_slab16<NS>(a0, 1, slab, y2);
                _Pragma("unroll")
                for (int r = 0; r < NQ; ++r) {
                    if (!FULL && !((mask >> r) & 1)) continue;
                    const float P = lds32(at + r * (RW * 4));
                    const float S = lds32(at + (NQ + r) * (RW * 4));
                    if (DIST) sumds[r] += S;
                    _Pragma("unroll")
                    for (int i = 0; i < 8; ++i) dk[r][i] = outer2(S, q2[i], dk[r][i]);
                    _Pragma("unroll")
                    for (int i = 0; i < 8; ++i) dv[r][i] = outer2(P, y2[i], dv[r][i]);
                }
                a0 += kRowBytes * NS;
                at += 2 * NQ * RW * 4;
            }
        };
        if (mask == (1 << NQ) - 1) sweep(std::true_type{});
        else sweep(std::false_type{});
        __syncwarp();                                            // the next stage but one writes what was read here
    })

    u64 k[NQ][8];
    if (DIST) load_centre<CPE, NQ, NCRT>(a.c0, g, u, h, w0, active, 1.f, k, 16 * slab);
    CA_OUT_DISPATCH(
        _Pragma("unroll")
        for (int r = 0; r < NQ; ++r) {
            _Pragma("unroll")
            for (int i = 0; i < 8; ++i) {
                const float x = dk[r][i].x - (DIST ? sumds[r] * k[r][i].x : 0.f);
                const float y = dk[r][i].y - (DIST ? sumds[r] * k[r][i].y : 0.f);
                store_centre<CPE, NCRV, BF>(a.o0, g, u, h, w0, active, r, i, a.scale * x + ca_poison, a.scale * y + ca_poison, 16 * slab);
                store_centre<CPE, NCRV, BF>(a.o1, g, u, h, w0, active, r, i, dv[r][i].x + ca_poison, dv[r][i].y + ca_poison, 16 * slab);
            }
        })
}

}  // namespace

// Columns per thread: 1 (for short windows and small grids, and folded signals, whose streamed column pairs with one centre
// column only), 2 (160 registers, three blocks per SM) or 3 (255, two blocks).
static const SweepCost kDqCost[3][3] = {{{1, 20, 0, 123, 501, 4921}, {2, 12, 9, 135, 936, 7404}, {3, 8, 22, 183, 1437, 10612}},
                                        {{1, 20, 59, 112, 0, 6247}, {2, 12, 15, 158, 146, 9951}, {3, 8, 53, 207, 0, 15865}},
                                        {{1, 20, 79, 124, 645, 0}, {2, 12, 55, 167, 964, 0}, {3, 8, 122, 192, 1635, 0}}};

template <>
int run_dq<kAnyC>(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* dy, const float* stats,
           const float* D, const float* kv, float* dq, cudaStream_t st, int mode, float* Dout, float* weights) {
    Launch L{};
    const int ns = slabs_of(g);
    if (ns > 1 && mode) return CA_ERR_UNSUPPORTED;             // the entmax variants exist for one-slab units
    if (mode >= 3) return CA_ERR_UNSUPPORTED;                  // the forward's sweeps go through run_entmax_fwd_sweep
    // the entmax variants have two columns per thread (128 x 96, 8 units, ws 15, against four: dq 105 -> 67 us, its
    // pre-pass 84 -> 63 us); the pre-pass does not share stages
    const bool fold = g.wsw == 1 && mode == 0;
    const SweepCost* cost = kDqCost[ns == 1 ? 0 : ns / 2] + (mode ? 1 : 0);
    const TileShape t = choose_tile(g, P, ns, cost, fold || mode ? 1 : (weights ? 2 : 3), mode < 2 && ns == 1 ? kParts : 1);
    int rc = prepare(g, P, t, 17 * t.nq, kv, nullptr, &L, ns);
    if (rc) return rc;
    L.a.scale = scale; L.a.c0 = q; L.a.c1 = dy; L.a.cs0 = stats; L.a.cs1 = D; L.a.o0 = dq; L.a.o1 = weights; L.a.ostats = Dout;
    if (weights) {
        if (ns != 4 || mode) return CA_ERR_UNSUPPORTED;
#define CA_DQ_STORE(NQV, NCRV_)                                                                       \
    do {                                                                                              \
        if (g.cpe == 1) {                                                                             \
            if (dist) CA_LAUNCH_TILED((dq_tiled_kernel<true, 1, NQV, 0, NCRV_, true>), L, st);        \
            else CA_LAUNCH_TILED((dq_tiled_kernel<false, 1, NQV, 0, NCRV_, true>), L, st);            \
        } else {                                                                                      \
            if (dist) CA_LAUNCH_TILED((dq_tiled_kernel<true, 2, NQV, 0, NCRV_, true>), L, st);        \
            else CA_LAUNCH_TILED((dq_tiled_kernel<false, 2, NQV, 0, NCRV_, true>), L, st);            \
        }                                                                                             \
    } while (0)
        if (t.nq == 1) CA_DQ_STORE(1, 64);
        else CA_DQ_STORE(2, 64);
#undef CA_DQ_STORE
        CA_CHECK_LAUNCH("tiled dq kernel");
        return CA_OK;
    }
#define CA_DQ(NCRV_)                                                                          \
    do {                                                                                      \
        if (t.nq == 1) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 1, 0, NCRV_, L, st);      \
        else if (t.nq == 2) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 2, 0, NCRV_, L, st); \
        else CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 3, 0, NCRV_, L, st);                \
    } while (0)
    if (mode == 2) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 2, 2, 16, L, st);
    else if (mode == 1) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 2, 1, 16, L, st);
    else if (ns == 1) CA_DQ(16);
    else if (ns == 2) CA_DQ(32);
    else CA_DQ(64);
#undef CA_DQ
    CA_CHECK_LAUNCH("tiled dq kernel");
    return CA_OK;
}

// Four columns per thread and no stage split: these sweeps serve large problems (smaller ones normalise stored scores),
// where two measured slower (300 x 280, 8 units, ws 11: first threshold 149 and 173 us, apply 252 and 266 us).
template <>
int run_entmax_fwd_sweep<kAnyC>(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* kv,
                         float* tau, float* settled, float* y, int mode, int iter, cudaStream_t st) {
    Launch L{};
    if (slabs_of(g) > 1) return CA_ERR_UNSUPPORTED;
    int rc = prepare(g, P, TileShape{4, std::min(4, (g.H + 31) / 32), 1}, 17 * 4, kv, nullptr, &L, 1);
    if (rc) return rc;
    L.a.scale = scale; L.a.c0 = q; L.a.cs0 = tau; L.a.cs1 = settled; L.a.o0 = y; L.a.o1 = settled; L.a.ostats = tau;
    L.a.iter = iter;
    if (mode == 3) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 4, 3, 16, L, st);
    else if (mode == 4) CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 4, 4, 16, L, st);
    else CA_DIST_CPE_NQ(dq_tiled_kernel, dist, g.cpe, 4, 5, 16, L, st);
    CA_CHECK_LAUNCH("tiled entmax forward sweep");
    return CA_OK;
}

// Columns per thread: 1 (three or four blocks per SM) or 3 (255 registers, two).  Two measured slower than one of them at
// every shape.
static const SweepCost kDkdvCost[3][2] = {{{1, 16, 13, 135, 190, 7335}, {3, 8, 201, 188, 1070, 14075}},
                                          {{1, 16, 82, 118, 0, 6933}, {3, 8, 138, 239, 0, 15999}},
                                          {{1, 16, 70, 146, 804, 0}, {3, 8, 234, 225, 1472, 0}}};

template <>
int run_dkdv<kAnyC>(const Geo& g, const Padded& P, float scale, int dist, const float* k, const float* v, const float* qdy,
             const float* planes, float* dk, float* dv, cudaStream_t st, bool entmax) {
    Launch L{};
    const int ns = slabs_of(g);
    if (ns > 1 && entmax) return CA_ERR_UNSUPPORTED;
    const bool fold = g.wsw == 1 && !entmax;
    const SweepCost* cost = kDkdvCost[ns == 1 ? 0 : ns / 2] + (entmax ? 1 : 0);
    const TileShape t = choose_tile(g, P, ns, cost, fold || entmax ? 1 : 2, ns == 1 ? kParts : 1, true);
    int rc = prepare(g, P, t, 33 * t.nq, qdy, planes, &L, ns);
    if (rc) return rc;
    L.a.scale = scale; L.a.c0 = k; L.a.c1 = v; L.a.o0 = dk; L.a.o1 = dv;
#define CA_DKDV(NCRV_)                                                                                \
    do {                                                                                              \
        if (t.nq == 1) CA_DIST_CPE_NQ(dkdv_tiled_kernel, dist, g.cpe, 1, false, NCRV_, L, st);        \
        else CA_DIST_CPE_NQ(dkdv_tiled_kernel, dist, g.cpe, 3, false, NCRV_, L, st);                  \
    } while (0)
    if (entmax) CA_DIST_CPE_NQ(dkdv_tiled_kernel, dist, g.cpe, 3, true, 16, L, st);
    else if (ns == 1) CA_DKDV(16);
    else if (ns == 2) CA_DKDV(32);
    else CA_DKDV(64);
#undef CA_DKDV
    CA_CHECK_LAUNCH("tiled dk/dv kernel");
    return CA_OK;
}

// One column per thread (five blocks per SM) or three (three blocks).
static const SweepCost kStoredCost[2] = {{1, 20, 60, 90, 0, 5000}, {3, 12, 100, 120, 0, 9000}};

template <>
int run_dkdv_stored<kAnyC>(const Geo& g, const Padded& P, float scale, int dist, const float* k, const float* qdy, const float* weights,
                           float* dk, float* dv, cudaStream_t st) {
    Launch L{};
    const int ns = slabs_of(g);
    if (ns != 4) return CA_ERR_UNSUPPORTED;
    const int col_bytes = 2 * g.ws * 2 * (32 / ns) * (int)sizeof(float);       // weights of two stages
    const TileShape t = choose_tile(g, P, ns, kStoredCost, 2, 1, false, false, col_bytes, 2);
    int rc = prepare(g, P, t, 0, qdy, nullptr, &L, ns, false, 2, (size_t)t.warps * t.nq * col_bytes);
    if (rc) return rc;
    L.a.scale = scale; L.a.c0 = k; L.a.cs0 = weights; L.a.o0 = dk; L.a.o1 = dv;
#define CA_STORED(NQV, NCRV_)                                                                      \
    do {                                                                                           \
        if (g.cpe == 1) {                                                                          \
            if (dist) CA_LAUNCH_TILED((dkdv_stored_kernel<true, 1, NQV, NCRV_>), L, st);           \
            else CA_LAUNCH_TILED((dkdv_stored_kernel<false, 1, NQV, NCRV_>), L, st);               \
        } else {                                                                                   \
            if (dist) CA_LAUNCH_TILED((dkdv_stored_kernel<true, 2, NQV, NCRV_>), L, st);           \
            else CA_LAUNCH_TILED((dkdv_stored_kernel<false, 2, NQV, NCRV_>), L, st);               \
        }                                                                                          \
    } while (0)
    if (t.nq == 1) CA_STORED(1, 64);
    else CA_STORED(3, 64);
#undef CA_STORED
    CA_CHECK_LAUNCH("tiled dk/dv kernel");
    return CA_OK;
}

}  // namespace ca
