// Forward sweep of the tiled kernels (compiled by fwd_exact.cu and fwd_any.cu; the scheme is described in tiled.cu).
// fwd_values_exact.cu and fwd_values_any.cu compile the form that also writes A's values.
#include "tile_common.cuh"
#ifndef CA_FWD_VALUES
#define CA_FWD_VALUES 0
#endif
#if CA_FWD_VALUES
#define CA_VALUES_PARAM float* nz,
#else
#define CA_VALUES_PARAM
#endif

namespace ca {
namespace {
constexpr bool kValues = CA_FWD_VALUES != 0;

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
//
// VALUES: the scores of the window also go to shared memory (struct Values), from where A's values leave at the end.
template <int NQ>
struct Values {
    uint32_t run[NQ];        // where the runs of this lane's row start: window column fixed, window rows varying
    int pos, wrap;           // byte position of the next window row inside a run, which turns to 0 at `wrap`
    bool on;                 // this lane stores
};
template <int DC, bool DIST, int MASK, int NQ, int NS, bool VALUES>
__device__ __forceinline__ void fwd_stage(uint32_t rowbase, int ws, int rm, float sl2, const u64 (&q)[NQ][8],
                                          u64 (&acc)[NQ][8], u64 (&nm2)[NQ], float (&l)[NQ], const float (&bq)[NQ],
                                          int slab, Values<NQ>& vals) {
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
                if (DIST && NS == 4) {                     // shared memory is the tighter bound of four slabs: 164 against 171 us
                    u64 n = zero2();                       // (128 x 96, 4 units of 64 channels, ws 15, with A's values)
#pragma unroll
                    for (int i = 0; i < 8; ++i) n = fma2(k2[i], k2[i], n);
                    bk = -0.5f * sl2 * hsum2(n);
                } else if (DIST) {
                    bk = -0.5f * sl2 * lds_norm(cb + t * RB, 128 * NS, slab);
                }
                if (MASK != 0) {
                    // the chains of all columns advance together
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
        if constexpr (VALUES) {
#pragma unroll
            for (int t = 0; t < DC; ++t) {
#pragma unroll
                for (int r = 0; r < NQ; ++r)
                    if (vals.on && ((rm >> r) & 1)) sts32(vals.run[r] + vals.pos, sc[r][t] - nm2[r].x);
                vals.pos = vals.pos + 4 == vals.wrap ? 0 : vals.pos + 4;
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
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[r][i] = outer2(pt, v2[i], acc[r][i]);
                    }
            }
        }
    }
}

// The ws keys of one window column.  EXACT: ws is a multiple of DC.  Otherwise (DC == 4): chunks of four keys, then
// the remaining one to three keys as one chunk of exactly that length, so that no chunk carries bounds checks
// (a checked chunk keeps its prefetched vector alive across branches, which costs a register copy per loaded
// word and made windows such as 13 slower than 15).
template <int DC, bool DIST, bool EXACT, int NQ, int NS, bool VALUES>
__device__ __forceinline__ void fwd_window(uint32_t rowbase, int ws, int rm, float sl2, const u64 (&q)[NQ][8],
                                           u64 (&acc)[NQ][8], u64 (&nm2)[NQ], float (&l)[NQ], const float (&bq)[NQ],
                                           int slab, Values<NQ>& vals) {
    constexpr int FULLM = (1 << NQ) - 1;
    if (EXACT) {
        fwd_stage<DC, DIST, FULLM, NQ, NS, VALUES>(rowbase, ws, rm, sl2, q, acc, nm2, l, bq, slab, vals);
        return;
    }
    static_assert(EXACT || DC == 4, "windows without a dividing chunk length run chunks of four plus a tail");
    const int main = ws & ~3;
    fwd_stage<4, DIST, FULLM, NQ, NS, VALUES>(rowbase, main, rm, sl2, q, acc, nm2, l, bq, slab, vals);
    const uint32_t tail = rowbase + main * (kRowBytes * NS);
    switch (ws - main) {                                     // warp-uniform
        case 1: fwd_stage<1, DIST, FULLM, NQ, NS, VALUES>(tail, 1, rm, sl2, q, acc, nm2, l, bq, slab, vals); break;
        case 2: fwd_stage<2, DIST, FULLM, NQ, NS, VALUES>(tail, 2, rm, sl2, q, acc, nm2, l, bq, slab, vals); break;
        case 3: fwd_stage<3, DIST, FULLM, NQ, NS, VALUES>(tail, 3, rm, sl2, q, acc, nm2, l, bq, slab, vals); break;
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
    if (DIST) bk = -0.5f * sl2 * lds_norm(rowbase, 128 * NS, slab);
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

// NCRT = real channels per unit the kernel is compiled for: 16 (narrower units are zero-extended),
// 32 or 64 (NS = 2 or 4 lanes per pixel, one 16-channel slab each; launched without a stage split).
// VALUES: also writes A's values, for windows whose rows fit the shared memory: the raw scores of the warp's pixels stay
// there at their final positions, and once a row's log-sum-exp is known 2^(score - it) leaves as one contiguous piece per
// centre column.  That costs a store per score and two more instructions on the way out, where a second sweep over the keys
// forms every score again.
template <int DC, bool DIST, int CPE, bool EXACT, int NQ, int NCRT, bool VALUES>
__global__ void __launch_bounds__(128, (NQ == 1 ? 5 : NQ <= 3 ? 3 : 2)) fwd_tiled_kernel(TileArgs a, const __grid_constant__ CUtensorMap mv,
                                                           const __grid_constant__ CUtensorMap msc) {
    constexpr int NS = NCRT <= 16 ? 1 : NCRT / 16;
    constexpr int RB = kRowBytes * NS;
    const Geo& g = a.g;
    const int ROWS = a.TH + 2 * (g.p + a.roff);
    const int NSTAGES = g.wsw + NQ - 1;
    const int w0 = blockIdx.x * NQ, h0 = blockIdx.y * a.TH, u = blockIdx.z;
    const float sl2 = a.scale * kLog2e;
    CA_PIPE_PROLOGUE(false, (NS == 1 ? kParts : 1))
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

    constexpr int RW = 32 / NS;
    float* tile = nullptr;                       // VALUES: [NQ][RW][K] scores of the warp's rows, then [NQ][RW] log-sum-exps
    const int hw0 = h0 + (lt >> 5) * RW;
    Values<NQ> vals{};
    int rot = 0;
    if constexpr (VALUES) {
        tile = reinterpret_cast<float*>(smem_al + a.extra_off) + (lt >> 5) * (NQ * RW * (g.K + 1));
        rot = active && has_pixel(g, h, w0) ? run_rot(axis_coord(g, h, w0), axis_len(g), g.p, g.ws) : 0;    // 2-D: for all columns
        vals.wrap = 4 * g.ws;
        vals.on = slab == 0;
    }

    CA_PIPE_LOOP({
        const int mask = stage_mask<NQ>(s, radius_w(g));
        const uint32_t rowbase = pipe.vec(buf, a) + (lr + a.roff) * RB;
        if constexpr (VALUES) {
            vals.pos = 4 * rot;
            for (int r = 0; r < NQ; ++r) {
                const bool here = ((mask >> r) & 1) && w0 + r < g.W;
                vals.run[r] = smem_u32(tile + (r * RW + (lr & (RW - 1))) * g.K + (here ? axis_pos(s - radius_w(g) - r, w0 + r, g.W, radius_w(g), g.wsw) * g.ws : 0));
            }
        }
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
            fwd_window<DC, DIST, EXACT, NQ, NS, VALUES>(rowbase, g.ws, mask, sl2, q, acc, nmE, l, bq, slab, vals);
#pragma unroll
            for (int r = 0; r < NQ; ++r)
                if ((mask >> r) & 1) nm2[r] = nmE[r];
        } else {
            fwd_window<DC, DIST, EXACT, NQ, NS, VALUES>(rowbase, g.ws, mask, sl2, q, acc, nm2, l, bq, slab, vals);
        }
    })

    float nm[NQ];
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        float zero;
        unpack2(nm2[r], nm[r], zero);
    }
    if (NS == 1 && a.nsplit > 1) {
        // merge the partial softmaxes: parts 1.. publish (m, l, acc), part 0 combines
        float* xch = reinterpret_cast<float*>(smem_al) + (size_t)max(part - 1, 0) * (18 * NQ) * PT;
        if (part > 0) {
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
        if (part > 0) return;
#pragma unroll 1
        for (int o = 1; o < a.nsplit; ++o, xch += (18 * NQ) * PT)
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
    if constexpr (VALUES) {
        float* lse = tile + NQ * RW * g.K;
#pragma unroll
        for (int r = 0; r < NQ; ++r)
            if (slab == 0) lse[r * RW + (lr & (RW - 1))] = log2f(l[r]) - nm[r];
        __syncwarp();
        const int lane = threadIdx.x & 31;
#pragma unroll 1
        for (int r = 0; r < NQ && w0 + r < g.W; ++r) {
            // rows of this column (the last column of a folded signal may be shorter)
            const int n = min(RW, (kAnyC ? min(g.H, g.Np - g.H * (w0 + r)) : g.H) - hw0) * g.K;
            float* dst = a.o1 + ((int64_t)u * g.Np + hw0 + (int64_t)g.H * (w0 + r)) * g.K;
            const float* src = tile + r * RW * g.K;
            int row = 0, e = lane;
            for (; e >= g.K; e -= g.K) ++row;
#pragma unroll 4
            for (int i = lane; i < n; i += 32) {
                dst[i] = fast_exp2(src[i] - lse[r * RW + row]) + ca_poison;
                e += 32;
                while (e >= g.K) { e -= g.K; ++row; }
            }
        }
    }
}

}  // namespace

// Columns per thread: 1 (five blocks per SM; short windows, small grids, folded signals), 2 or 3 (168 registers, three
// blocks per SM; with packed outer products three beat four, 255 registers and two blocks, 5.68 against 6.07 ms at
// 1024 x 1024, 8 units, ws 21).
static const SweepCost kFwdCost[3][3] = {{{1, 20, 0, 129, 216, 3265}, {2, 12, 0, 121, 532, 5634}, {3, 12, 16, 138, 684, 8536}},
                                         {{1, 20, 36, 105, 145, 4276}, {2, 12, 0, 131, 130, 8597}, {3, 12, 53, 125, 0, 14976}},
                                         {{1, 20, 3, 141, 421, 0}, {2, 12, 0, 154, 726, 0}, {3, 12, 6, 166, 1454, 0}}};

#if CA_FWD_VALUES
#define RUN_FWD run_fwd_values
#else
#define RUN_FWD run_fwd
#endif
template <>
int RUN_FWD<kAnyC>(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* kv, float* y, float* stats,
                   CA_VALUES_PARAM cudaStream_t st) {
    Launch L{};
    const int ns = slabs_of(g);
#if CA_FWD_VALUES
    const int col_bytes = 32 / ns * (g.K + 1) * (int)sizeof(float);
    if (!values_fit(g, ns)) return CA_ERR_UNSUPPORTED;
    const TileShape t = choose_tile(g, P, ns, kFwdCost[ns == 1 ? 0 : ns / 2], g.wsw == 1 ? 1 : 2, ns == 1 ? kParts : 1, false, false, col_bytes, 2);
    int rc = prepare(g, P, t, 18 * t.nq, kv, nullptr, &L, ns, false, 2, t.warps * t.nq * col_bytes);
    L.a.o1 = nz;
#else
    const TileShape t = choose_tile(g, P, ns, kFwdCost[ns == 1 ? 0 : ns / 2], g.wsw == 1 ? 1 : 3, ns == 1 ? kParts : 1);
    int rc = prepare(g, P, t, 18 * t.nq, kv, nullptr, &L, ns);
#endif
    if (rc) return rc;
    L.a.scale = scale; L.a.c0 = q; L.a.o0 = y; L.a.ostats = stats;
#define CA_FWD2(DCV, EX, NQV, NCRV_)                                                            \
    do {                                                                                 \
        if (g.cpe == 1) {                                                                \
            if (dist) CA_LAUNCH_TILED((fwd_tiled_kernel<DCV, true, 1, EX, NQV, NCRV_, kValues>), L, st); \
            else CA_LAUNCH_TILED((fwd_tiled_kernel<DCV, false, 1, EX, NQV, NCRV_, kValues>), L, st);     \
        } else {                                                                         \
            if (dist) CA_LAUNCH_TILED((fwd_tiled_kernel<DCV, true, 2, EX, NQV, NCRV_, kValues>), L, st); \
            else CA_LAUNCH_TILED((fwd_tiled_kernel<DCV, false, 2, EX, NQV, NCRV_, kValues>), L, st);     \
        }                                                                                \
    } while (0)
    // chunks of 7, 5 or 3 keys where they divide the window, else chunks of four plus a tail
#define CA_FWD(NQV, NCRV_)                                                               \
    do {                                                                                 \
        if (g.ws % 7 == 0) CA_FWD2(7, true, NQV, NCRV_);                                 \
        else if (g.ws % 5 == 0) CA_FWD2(5, true, NQV, NCRV_);                            \
        else if (NQV > 1 && NCRV_ == 16 && g.ws % 3 == 0) CA_FWD2((NQV > 1 && NCRV_ == 16 ? 3 : 5), true, NQV, NCRV_); \
        else CA_FWD2(4, false, NQV, NCRV_);                                              \
    } while (0)
#define CA_FWD_NQ(NCRV_)                                                                 \
    do {                                                                                 \
        if (t.nq == 1) CA_FWD(1, NCRV_);                                                 \
        else if (kValues || t.nq == 2) CA_FWD(2, NCRV_);                                 \
        else CA_FWD((kValues ? 2 : 3), NCRV_);                                           \
    } while (0)
    if (ns == 1) CA_FWD_NQ(16);
    else if (ns == 2) CA_FWD_NQ(32);
    else CA_FWD_NQ(64);
#undef CA_FWD_NQ
#undef CA_FWD
#undef CA_FWD2
    CA_CHECK_LAUNCH("tiled forward kernel");
    return CA_OK;
}

}  // namespace ca
