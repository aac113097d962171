// Backward of the tensor-core sweeps (split.cuh): dq from the streamed (k|v), dk and dv from the streamed (q|dy).
//   P = 2^(s - L),  dS = P (dP - D),  dq = scale sum dS k,  dk = scale sum dS q,  dv = sum P dy
// (Distance: sum dS (k - q), sum dS (q - k)).  Weights enter the products as halves, so they are scaled by powers of two: P by
// 2^14, and dP - D by 2^14 over a bound that follows from the operands' norms, per row and step (dq) or per warp and
// step (dk); a step's sums are scaled back when they are added to the running ones.  P's factor is not part of its exponent:
// 14 + s - L has up to four times the last place of s - L (64 x 50, 8 units of 8 channels, ws 9: errors of dq, dk, dv against 64 bits 4.7e-7,
// 4.5e-7, 4.6e-7 with it, 3.9e-7, 3.8e-7, 3.8e-7 without; the backward is 1 % slower).
#include "split.cuh"

namespace ca {
namespace {

constexpr float kWeight = 0x1p14f;

// Biased exponent of the reciprocal of a bound of |dP| + |D|: `norm` above the centre vector's norm, `e` the exponent of the streamed
// group's scale, whose vectors have norms up to sqrt(16) 2^15, `d` above |D|.
__device__ __forceinline__ int bound_inverse(int norm, int e, int d) {
    const int x = max(norm + e - 127 + 17, d) + 1;
    return min(max(254 - x, 1), 236);
}

__device__ __noinline__ void exact_dq(const SplitArgs& a, int u, int row0, int w0, float* buf) {
    const Geo& g = a.g;
    const float sl2 = a.scale * kLog2e;
    const ExactLane L(g, row0, w0);
    float q[16], dy[16], acc[16];
    load_pixel(a.c0, g, u, g.Np, L.pix, q);
    load_pixel(a.c1, g, u, g.Np, L.pix, dy);
    const float stat = a.stats[(int64_t)u * g.Np + L.pix] * kLog2e, D = a.D[(int64_t)u * g.Np + L.pix];
#pragma unroll
    for (int c = 0; c < 16; ++c) acc[c] = 0.f;
#pragma unroll 1
    for (int s = 0; s <= g.ws; ++s) {
        __syncwarp();
        if (L.lane < 8 + 2 * g.p) exact_copy(a, u, L.streamed(g, row0, w0, s), buf + L.lane * kExactPitch);
        __syncwarp();
        if (!L.meets(g, s)) continue;
#pragma unroll 1
        for (int dh = L.half; dh < g.ws; dh += 2) {
            const float* row = buf + (L.dh0 + dh) * kExactPitch;
            float k[16], v[16];
            read16(row, k);
            read16(row + 16, v);
            const float ds = fast_exp2(score(a, q, k) * sl2 - stat) * (dot16(dy, v) - D);
            if (a.dist) {
#pragma unroll
                for (int c = 0; c < 16; ++c) k[c] -= q[c];
            }
            add_scaled(acc, ds, k);
        }
    }
    exact_store(a.o0, g, u, L, acc, a.scale);
}

__device__ __noinline__ void exact_dkdv(const SplitArgs& a, int u, int row0, int w0, float* buf) {
    const Geo& g = a.g;
    const float sl2 = a.scale * kLog2e;
    const ExactLane L(g, row0, w0);
    float k[16], v[16], dk[16], dv[16];
    load_pixel(a.c0, g, u, g.Np, L.pix, k);
    load_pixel(a.c1, g, u, g.Np, L.pix, v);
#pragma unroll
    for (int c = 0; c < 16; ++c) dk[c] = dv[c] = 0.f;
#pragma unroll 1
    for (int s = 0; s <= g.ws; ++s) {
        __syncwarp();
        if (L.lane < 8 + 2 * g.p) {
            const int pix = L.streamed(g, row0, w0, s);
            float* row = buf + L.lane * kExactPitch;
            exact_copy(a, u, pix, row);
            row[32] = a.xstats[(int64_t)u * g.Npk + pix] * kLog2e;
            row[33] = a.xD[(int64_t)u * g.Npk + pix];
        }
        __syncwarp();
        if (!L.meets(g, s)) continue;
#pragma unroll 1
        for (int dh = L.half; dh < g.ws; dh += 2) {
            const float* row = buf + (L.dh0 + dh) * kExactPitch;
            float q[16], dy[16];
            read16(row, q);
            read16(row + 16, dy);
            const float p = fast_exp2(score(a, q, k) * sl2 - row[32]), ds = p * (dot16(dy, v) - row[33]);
            if (a.dist) {
#pragma unroll
                for (int c = 0; c < 16; ++c) q[c] -= k[c];
            }
            add_scaled(dk, ds, q);
            add_scaled(dv, p, dy);
        }
    }
    exact_store(a.o0, g, u, L, dk, a.scale);
    exact_store(a.o1, g, u, L, dv, 1.f);
}

// What the two sweeps share: the tiles of a column against two centre operands.
template <int NT, bool LO>
struct BwdSweep {
    static constexpr int RB = split_row_bytes(LO), SB = split_stage_bytes(NT, LO);
    const SplitArgs& a;
    int lane, tq, h, u;
    uint32_t dot_off, outer_off, tail_off, word_off;
    float sl2;
    Centre<LO> c0, c1;
    uint32_t cur, word;                                      // the scales of the step's groups when they are all alike; this lane's
    bool bad, mixed;                                         // bad: a centre operand cannot be split

    __device__ __forceinline__ BwdSweep(const SplitArgs& a_) : a(a_) {
        const int row0 = blockIdx.y * 8 * kSplitWarps + 8 * (threadIdx.x >> 5);
        lane = threadIdx.x & 31;
        tq = lane & 3;
        h = row0 + (lane >> 2);
        u = blockIdx.z;
        sl2 = a.scale * kLog2e;
        dot_off = dot_offset(lane, LO);
        outer_off = outer_offset(lane, LO, 8 * RB);
        tail_off = outer_offset(lane, LO, SB);
        word_off = word_offset<NT, LO>(a.g, lane, row0);
    }
    __device__ __forceinline__ void load(int w0) {
        Raw r0, r1;
        r0.load(a.c0, a.g, u, h, w0, tq);
        r1.load(a.c1, a.g, u, h, w0, tq);
        c0.form(r0, a.g, h, w0, tq, kLeastExp);
        c1.form(r1, a.g, h, w0, tq, 0);
        bad = c0.bad || c1.bad;
        cur = 0;
#pragma unroll
        for (int r = 0; r < 2; ++r) c0.scale[r] = fmaxf(c0.scale[r] * sl2, 0x1p-70f);
    }
    // Centre column 0 does not meet the last column of the windows, centre column 1 not the first.
    template <int HALF>
    __device__ __forceinline__ void drop(bool first, bool last, float (&x)[NT][4]) {
        if (HALF == 0 && first) {
#pragma unroll
            for (int t = 0; t < NT; ++t) x[t][2] = x[t][3] = -INFINITY;
        }
        if (HALF == 1 && last) {
#pragma unroll
            for (int t = 0; t < NT; ++t) x[t][0] = x[t][1] = -INFINITY;
        }
    }
};

template <int NT, bool DIST, bool LO>
struct DqSweep : BwdSweep<NT, LO> {
    using B = BwdSweep<NT, LO>;
    using B::a; using B::lane; using B::tq; using B::h; using B::u; using B::c0; using B::c1; using B::cur; using B::word; using B::bad; using B::mixed;
    using B::RB; using B::SB;
    pair_t acc[2][2], sum[2], nref[NT][2], c[2], e[2], nd[2], S[2], Sd[2];     // Sd: Distance, the sums of dS
    float D[2];
    Tail tail;

    __device__ __forceinline__ DqSweep(const SplitArgs& a_) : B(a_) {}

    __device__ __forceinline__ void begin(int w0, uint32_t) {
        const Geo& g = a.g;
        float Ls[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int64_t o = (int64_t)u * g.Np + min(h, g.H - 1) + g.H * min(w0 + r, g.W - 1);
            Ls[r] = __ldg(a.stats + o);
            D[r] = __ldg(a.D + o);
        }
        B::load(w0);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const bool ok = h < g.H && w0 + r < g.W;
            const float L = ok ? Ls[r] * kLog2e : 0.f;
            D[r] = ok ? D[r] : 0.f;
            bad |= !(fabsf(L) < INFINITY) || !(fabsf(D[r]) < INFINITY);
            const float b = -L - (DIST ? 0.5f * B::sl2 * c0.norm2[r] : 0.f);
#pragma unroll
            for (int t = 0; t < NT; ++t) nref[t][r] = pair(b + window_mask(lane, g.p, t, 0), b + window_mask(lane, g.p, t, 1));
            sum[r] = c[r] = e[r] = nd[r] = S[r] = Sd[r] = 0;
        }
        Seen::clear(bad);
#pragma unroll
        for (int n = 0; n < 2; ++n) acc[n][0] = acc[n][1] = 0;
    }

    template <int HALF>
    __device__ __forceinline__ void column(uint32_t rb, bool first, bool last) {
        float x[NT][4], y[NT][4];
        dot_column<NT, LO>(c0, c1, rb + HALF * SB + B::dot_off, x, y);
        if (mixed) {
            scale_tiles<NT>(x, word, cur, 0, 1, HALF);
            scale_tiles<NT>(y, word, cur, 8, 0, HALF);
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const pair_t b = DIST ? lds_pair(rb + HALF * SB + (8 * t + 2 * tq) * RB + split_scalars(LO) + 8) : 0;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float2 z = unpair(fma_pair(pair(x[t][2 * r], x[t][2 * r + 1]), c[r], DIST ? add_pair(nref[t][r], b) : nref[t][r]));
                x[t][2 * r] = z.x;
                x[t][2 * r + 1] = z.y;
            }
        }
        B::template drop<HALF>(first, last, x);
        uint32_t hi[NT][2], lo[NT][2];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
#pragma unroll
            for (int i = 0; i < 4; ++i) x[t][i] = fast_exp2(x[t][i]);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const pair_t ds = mul_pair(pair(x[t][2 * r], x[t][2 * r + 1]), fma_pair(pair(y[t][2 * r], y[t][2 * r + 1]), e[r], nd[r]));
                if (DIST) sum[r] = fma_pair(ds, Sd[r], sum[r]);
                const float2 z = unpair(ds);
                x[t][2 * r] = z.x;
                x[t][2 * r + 1] = z.y;
            }
        }
        if (mixed) scale_tiles<NT>(x, word, cur, 0, 0, HALF);
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int r = 0; r < 2; ++r) split2(x[t][2 * r], x[t][2 * r + 1], hi[t][r], lo[t][r]);
        outer_column<NT, LO, HALF>(hi, lo, tail, rb + HALF * SB + B::outer_off, rb + B::tail_off, S, acc);
    }

    __device__ __forceinline__ void step(uint32_t rb, bool first, bool last) {
        word = ldsu32(rb + B::word_off) & 0xffffu;
        mixed = false;
        if (__any_sync(0xffffffffu, word != cur)) {
            // weights are mostly 2^-7 to 2^2 of 2^-24 steps: a scale further than 2^4 below the step's largest would show
            uint32_t ek, ev;
            Seen::tops(word, ek, ev);
            Seen::add(word, ek, ev, 4, 4, !(fmaxf(c0.scale[0], c0.scale[1]) * exp_scale(ek) < kMostFactor));
            cur = ek | ev << 8;
            mixed = __any_sync(0xffffffffu, word != cur);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int nb = bound_inverse(c1.top[r], ev, above(D[r]));
                const float nrm = exp_scale(nb) * kWeight, bd = exp_scale(254 - nb) / kWeight, back = exp_scale(ek) * bd;
                c[r] = pair(c0.scale[r] * exp_scale(ek), c0.scale[r] * exp_scale(ek));
                e[r] = pair(c1.scale[r] * nrm * exp_scale(ev), c1.scale[r] * nrm * exp_scale(ev));
                nd[r] = pair(-D[r] * nrm, -D[r] * nrm);
                S[r] = pair(back, back);
                Sd[r] = pair(bd, bd);
            }
        }
        column<0>(rb, first, last);
        column<1>(rb, first, last);
    }

    __device__ __forceinline__ void end(int w0, float poison) {
        const Geo& g = a.g;
        if (Seen::bad() && poison == 0.f) {
            exact_dq(a, u, h - (lane >> 2), w0, exact_rows<NT, LO>());
            return;
        }
        Raw raw = {};
        if (DIST) raw.load(a.c0, g, u, h, w0, tq);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const bool ok = h < g.H && w0 + r < g.W;
            const int pix = ok ? h + g.H * (w0 + r) : 0;
            float ds = 0.f;
            if (DIST) {
                const float2 z = unpair(sum[r]);
                ds = quad_sum(z.x + z.y);
            }
            if (!ok) continue;
            const float (&qv)[4] = raw.x[r];
            const float2 y0 = unpair(acc[0][r]), y1 = unpair(acc[1][r]);
            store_pixel(a.o0, g, u, pix, tq, a.scale * (y0.x - ds * qv[0]) + poison, a.scale * (y0.y - ds * qv[1]) + poison,
                        a.scale * (y1.x - ds * qv[2]) + poison, a.scale * (y1.y - ds * qv[3]) + poison);
        }
    }
};

template <int NT, bool DIST, bool LO>
struct DkdvSweep : BwdSweep<NT, LO> {
    using B = BwdSweep<NT, LO>;
    using B::a; using B::lane; using B::tq; using B::h; using B::u; using B::c0; using B::c1; using B::cur; using B::word; using B::bad; using B::mixed;
    using B::RB; using B::SB;
    pair_t dk[2][2], dv[2][2], sum[2], mk[NT], bk[2], c[2], e[2], nrm, Sk[2], Sv[2], Sd;      // Sd: Distance, the sums of dS
    int norm;
    int bound;                                               // exponent above the |dP| and the |D| of the step
    Tail tp, td;

    __device__ __forceinline__ DkdvSweep(const SplitArgs& a_) : B(a_) {}

    __device__ __forceinline__ void begin(int w0, uint32_t) {
        const Geo& g = a.g;
        B::load(w0);
        bound = 0;
        nrm = Sd = 0;
        // The largest norm bounds the weights of all 16 pixels.  Those four rows from a pixel meet queries that it does not.
        const int top = max(c1.top[0], c1.top[1]);
        const int upper = __reduce_max_sync(0xffffffffu, lane < 16 ? top : 0), lower = __reduce_max_sync(0xffffffffu, lane < 16 ? 0 : top);
        norm = max(upper, lower);
        Seen::clear(bad || (min(upper, lower) && abs(upper - lower) > 2));
#pragma unroll
        for (int t = 0; t < NT; ++t) mk[t] = pair(window_mask(lane, g.p, t, 0), window_mask(lane, g.p, t, 1));
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float b = -0.5f * B::sl2 * c0.norm2[r];
            bk[r] = pair(b, b);
            sum[r] = c[r] = e[r] = Sk[r] = Sv[r] = 0;
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) dk[n][0] = dk[n][1] = dv[n][0] = dv[n][1] = 0;
    }

    template <int HALF>
    __device__ __forceinline__ void column(uint32_t rb, bool first, bool last) {
        float x[NT][4], y[NT][4];
        dot_column<NT, LO>(c0, c1, rb + HALF * SB + B::dot_off, x, y);
        if (mixed) {
            scale_tiles<NT>(x, word, cur, 0, 1, HALF);
            scale_tiles<NT>(y, word, cur, 8, 0, HALF);
        }
        const uint32_t sc = rb + HALF * SB + 2 * tq * RB + split_scalars(LO) + 8;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const pair_t A = add_pair(mk[t], lds_pair(sc + 8 * t * RB)), Dn = mul_pair(lds_pair(sc + (8 * t + 1) * RB), nrm);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float2 z = unpair(fma_pair(pair(x[t][2 * r], x[t][2 * r + 1]), c[r], DIST ? add_pair(A, bk[r]) : A));
                const float2 w = unpair(fma_pair(pair(y[t][2 * r], y[t][2 * r + 1]), e[r], Dn));
                x[t][2 * r] = z.x;
                x[t][2 * r + 1] = z.y;
                y[t][2 * r] = w.x;
                y[t][2 * r + 1] = w.y;
            }
        }
        B::template drop<HALF>(first, last, x);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
#pragma unroll
            for (int i = 0; i < 4; ++i) x[t][i] = fast_exp2(x[t][i]);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const pair_t ds = mul_pair(pair(x[t][2 * r], x[t][2 * r + 1]), pair(y[t][2 * r], y[t][2 * r + 1]));
                if (DIST) sum[r] = fma_pair(ds, Sd, sum[r]);
                const float2 z = unpair(ds), p = unpair(mul_pair(pair(x[t][2 * r], x[t][2 * r + 1]), pair(kWeight, kWeight)));
                x[t][2 * r] = p.x;
                x[t][2 * r + 1] = p.y;
                y[t][2 * r] = z.x;
                y[t][2 * r + 1] = z.y;
            }
        }
        if (mixed) {
            scale_tiles<NT>(y, word, cur, 0, 0, HALF);
            scale_tiles<NT>(x, word, cur, 8, 0, HALF);
        }
        uint32_t hi[NT][2], lo[NT][2];
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int r = 0; r < 2; ++r) split2(x[t][2 * r], x[t][2 * r + 1], hi[t][r], lo[t][r]);
        outer_column<NT, LO, HALF>(hi, lo, tp, rb + HALF * SB + B::outer_off + split_second(LO), rb + B::tail_off + split_second(LO), Sv, dv);
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int r = 0; r < 2; ++r) split2(y[t][2 * r], y[t][2 * r + 1], hi[t][r], lo[t][r]);
        outer_column<NT, LO, HALF>(hi, lo, td, rb + HALF * SB + B::outer_off, rb + B::tail_off, Sk, dk);
    }

    __device__ __forceinline__ void step(uint32_t rb, bool first, bool last) {
        word = ldsu32(rb + B::word_off);
        const uint32_t top = word >> 16;
        word &= 0xffffu;
        mixed = false;
        if (__any_sync(0xffffffffu, word != cur || (int)top > bound)) {
            uint32_t eq, ed;
            Seen::tops(word, eq, ed);
            // Where a |D| rules the weights, groups with smaller ones lose bits to it; such a step's bound is not kept for the next.
            const int dp = norm + (int)ed - 127 + 17, most = __reduce_max_sync(0xffffffffu, top);
            bound = min(max(dp, most), 254);
            Seen::add(word, eq, ed, 4, 4,
                      most == 255 || (top && most > dp && most > (int)top + 6) || !(fmaxf(c0.scale[0], c0.scale[1]) * exp_scale(eq) < kMostFactor));
            cur = eq | ed << 8;
            mixed = __any_sync(0xffffffffu, word != cur);
            if (most > dp) cur |= 1u << 16;
            const int nb = bound_inverse(norm, ed, most);
            const float n = exp_scale(nb) * kWeight, bv = exp_scale(ed) / kWeight, bd = exp_scale(254 - nb) / kWeight, back = exp_scale(eq) * bd;
            nrm = pair(n, n);
            Sd = pair(bd, bd);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                c[r] = pair(c0.scale[r] * exp_scale(eq), c0.scale[r] * exp_scale(eq));
                e[r] = pair(c1.scale[r] * n * exp_scale(ed), c1.scale[r] * n * exp_scale(ed));
                Sv[r] = pair(bv, bv);
                Sk[r] = pair(back, back);
            }
        }
        column<0>(rb, first, last);
        column<1>(rb, first, last);
    }

    __device__ __forceinline__ void end(int w0, float poison) {
        const Geo& g = a.g;
        if (Seen::bad() && poison == 0.f) {
            exact_dkdv(a, u, h - (lane >> 2), w0, exact_rows<NT, LO>());
            return;
        }
        Raw raw = {};
        if (DIST) raw.load(a.c0, g, u, h, w0, tq);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const bool ok = h < g.H && w0 + r < g.W;
            const int pix = ok ? h + g.H * (w0 + r) : 0;
            float ds = 0.f;
            if (DIST) {
                const float2 z = unpair(sum[r]);
                ds = quad_sum(z.x + z.y);
            }
            if (!ok) continue;
            const float (&kv)[4] = raw.x[r];
            const float2 k0 = unpair(dk[0][r]), k1 = unpair(dk[1][r]), v0 = unpair(dv[0][r]), v1 = unpair(dv[1][r]);
            store_pixel(a.o0, g, u, pix, tq, a.scale * (k0.x - ds * kv[0]) + poison, a.scale * (k0.y - ds * kv[1]) + poison,
                        a.scale * (k1.x - ds * kv[2]) + poison, a.scale * (k1.y - ds * kv[3]) + poison);
            store_pixel(a.o1, g, u, pix, tq, v0.x + poison, v0.y + poison, v1.x + poison, v1.y + poison);
        }
    }
};

// Without lower halves one more block per SM pays for 4 to 128 bytes of spills (forward and backward, 1024 x 1024, 8 units, ws 21, with the same in
// the forward and dk/dv and rows of 80 bytes: 14812 -> 13340 us, Distance 15857 -> 14770).
template <int NT, bool DIST, bool LO>
__global__ void __launch_bounds__(32 * kSplitWarps, LO ? 4 : 5) split_dq_kernel(const __grid_constant__ SplitArgs a,
                                                                                           const __grid_constant__ CUtensorMap map) {
    DqSweep<NT, DIST, LO> sweep(a);
    split_run<NT, LO>(a, &map, sweep);
}
template <int NT, bool DIST, bool LO>
__global__ void __launch_bounds__(32 * kSplitWarps, NT == 2 || !LO ? 4 : 3) split_dkdv_kernel(const __grid_constant__ SplitArgs a,
                                                                                             const __grid_constant__ CUtensorMap map) {
    DkdvSweep<NT, DIST, LO> sweep(a);
    split_run<NT, LO>(a, &map, sweep);
}

}  // namespace

#define CA_SPLIT_BWD(KERNEL, NTV)                                                               \
    do {                                                                                             \
        if (g.bf16) {                                                                                \
            if (dist) CA_LAUNCH_SPLIT((KERNEL<NTV, true, false>), a, L, st);                    \
            else CA_LAUNCH_SPLIT((KERNEL<NTV, false, false>), a, L, st);                        \
        } else {                                                                                     \
            if (dist) CA_LAUNCH_SPLIT((KERNEL<NTV, true, true>), a, L, st);                     \
            else CA_LAUNCH_SPLIT((KERNEL<NTV, false, true>), a, L, st);                         \
        }                                                                                            \
    } while (0)
#define CA_SPLIT_BWD_NT(KERNEL)                                                                 \
    do {                                                                                             \
        if (nt == 2) CA_SPLIT_BWD(KERNEL, 2);                                                   \
        else if (nt == 3) CA_SPLIT_BWD(KERNEL, 3);                                              \
        else if (nt == 4) CA_SPLIT_BWD(KERNEL, 4);                                              \
        else return CA_ERR_UNSUPPORTED;                                                              \
    } while (0)

int run_split_dq(const Geo& g, float scale, int dist, const float* q, const float* k, const float* v, const float* dy, const float* stats,
                 const float* D, const float* kv, float* dq, cudaStream_t st) {
    Launch L{};
    SplitArgs a{};
    const int nt = split_tiles(g);
    const int rc = split_prepare(g, scale, dist, kv, &L, &a);
    if (rc) return rc;
    a.c0 = q; a.c1 = dy; a.stats = stats; a.D = D; a.o0 = dq; a.x0 = k; a.x1 = v;
    CA_SPLIT_BWD_NT(split_dq_kernel);
    CA_CHECK_LAUNCH("split dq kernel");
    return CA_OK;
}

int run_split_dkdv(const Geo& g, float scale, int dist, const float* q, const float* k, const float* v, const float* dy, const float* stats,
                   const float* D, const float* qdy, float* dk, float* dv, cudaStream_t st) {
    Launch L{};
    SplitArgs a{};
    const int nt = split_tiles(g);
    const int rc = split_prepare(g, scale, dist, qdy, &L, &a);
    if (rc) return rc;
    a.c0 = k; a.c1 = v; a.o0 = dk; a.o1 = dv; a.x0 = q; a.x1 = dy; a.xstats = stats; a.xD = D;
    CA_SPLIT_BWD_NT(split_dkdv_kernel);
    CA_CHECK_LAUNCH("split dk/dv kernel");
    return CA_OK;
}

}  // namespace ca
