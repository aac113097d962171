// Forward of the tensor-core sweeps (split.cuh): y and the row log-sum-exp.
#include "split.cuh"

namespace ca {
namespace {

// Weights are 2^(s - reference) <= 2^15, the most that a half holds with room to round.  The reference of a row is set from the
// largest score of its first window column, which gets weight 2^kStart, and moves when a score passes the bound.
constexpr float kTop = 15.f, kStart = 7.f;

__device__ __noinline__ void exact_fwd(const SplitArgs& a, int u, int row0, int w0, float* buf) {
    const Geo& g = a.g;
    const float sl2 = a.scale * kLog2e;
    const ExactLane L(g, row0, w0);
    float q[16], acc[16], m = -FLT_MAX, l = 0.f;
    load_pixel(a.c0, g, u, g.Np, L.pix, q);
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
            const float z = score(a, q, k) * sl2, mn = fmaxf(m, z), p = fast_exp2(z - mn);
            read16(row + 16, v);
            if (mn != m) {
                const float corr = fast_exp2(m - mn);
                l *= corr;
#pragma unroll
                for (int c = 0; c < 16; ++c) acc[c] *= corr;
                m = mn;
            }
            l += p;
            add_scaled(acc, p, v);
        }
    }
    const float top = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16)), f = fast_exp2(m - top);
    l *= f;
    const float sum = l + __shfl_xor_sync(0xffffffffu, l, 16);
#pragma unroll
    for (int c = 0; c < 16; ++c) acc[c] *= f;
    exact_store(a.o0, g, u, L, acc, 1.f / sum);
    if (a.ostats && L.ok && !L.half) a.ostats[(int64_t)u * g.Np + L.pix] = (top + log2f(sum)) * kLn2;
}

// The values of the warp's rows of A: here a lane owns a row of the windows, whose values are neighbours, and the centre vectors lie
// behind the column.
__device__ __noinline__ void exact_values(const SplitArgs& a, int u, int row0, int w0, float* buf) {
    const Geo& g = a.g;
    const float sl2 = a.scale * kLog2e;
    const ExactLane L(g, row0, w0);
    constexpr int kPitch = kExactValuesPitch;
    float* centre = buf + (8 + 2 * g.p) * kPitch;
    float x[16];
    __syncwarp();
    if (!L.half) {
        load_pixel(a.c0, g, u, g.Np, L.pix, x);
        write16(centre + L.lane * kPitch, x);
        centre[L.lane * kPitch + 16] = a.stats[(int64_t)u * g.Np + L.pix] * kLog2e;
    }
#pragma unroll 1
    for (int s = 0; s <= g.ws; ++s) {
        __syncwarp();
        if (L.lane < 8 + 2 * g.p) {
            load_pixel(a.x0, g, u, g.Npk, L.streamed(g, row0, w0, s), x);
            write16(buf + L.lane * kPitch, x);
        }
        __syncwarp();
        if (L.lane >= g.ws) continue;
#pragma unroll 1
        for (int i = 0; i < 16; ++i) {
            const int h = row0 + (i >> 1), r = i & 1, w = w0 + r;
            if (s == (r ? 0 : g.ws) || h >= g.H || w >= g.W) continue;
            float q[16];
            read16(centre + i * kPitch, q);
            read16(buf + ((i >> 1) + L.lane) * kPitch, x);
            a.o0[((int64_t)u * g.Np + h + g.H * w) * g.K + axis_pos(s - g.p - r, w, g.W, g.p, g.ws) * g.ws +
                 axis_pos(L.lane - g.p, h, g.H, g.p, g.ws)] = fast_exp2(score(a, q, x) * sl2 - centre[i * kPitch + 16]);
        }
    }
}

// A warp's eight rows of two columns; a step scores them against two columns of the window.
template <int NT, bool DIST, bool LO>
struct FwdSweep {
    static constexpr int RB = split_row_bytes(LO), SB = split_stage_bytes(NT, LO), T = 2 * NT;
    const SplitArgs& a;
    int lane, tq, h, u;
    uint32_t dot_off, outer_off, tail_off, word_off;
    float sl2;
    Centre<LO> q;
    pair_t acc[2][2], l[2], nref[NT][2], c[2], S[2];
    float shift[2];                                          // what the references have moved by
    uint32_t cur;                                            // the scales of the step's groups when they are all alike, as they mostly are

    __device__ __forceinline__ FwdSweep(const SplitArgs& a_) : a(a_) {
        const int warp = threadIdx.x >> 5, row0 = blockIdx.y * 8 * kSplitWarps + 8 * (warp % kSplitWarps);
        lane = threadIdx.x & 31;
        tq = lane & 3;
        h = row0 + (lane >> 2);
        u = blockIdx.z;
        sl2 = a.scale * kLog2e;
        dot_off = dot_offset(lane, LO);
        outer_off = outer_offset(lane, LO, 8 * RB) + split_second(LO);
        tail_off = outer_offset(lane, LO, SB) + split_second(LO);
        word_off = word_offset<NT, LO>(a.g, lane, row0);
    }

    __device__ __forceinline__ void begin(int w0, uint32_t) {
        const Geo& g = a.g;
        Raw raw;
        raw.load(a.c0, g, u, h, w0, tq);
        q.form(raw, g, h, w0, tq, kLeastExp);
        Seen::clear(q.bad);
        cur = 0;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            l[r] = c[r] = S[r] = 0;
            shift[r] = 0.f;
            const float bq = DIST ? -0.5f * sl2 * q.norm2[r] : 0.f;
#pragma unroll
            for (int t = 0; t < NT; ++t) nref[t][r] = pair(bq + window_mask(lane, g.p, t, 0), bq + window_mask(lane, g.p, t, 1));
            q.scale[r] = fmaxf(q.scale[r] * sl2, 0x1p-70f);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) acc[n][0] = acc[n][1] = 0;
    }

    __device__ __forceinline__ void step(uint32_t rb, bool first, bool last) {
        const uint32_t word = ldsu32(rb + word_off);
        bool mixed = false;
        if (__any_sync(0xffffffffu, word != cur)) {
            // Weights start at 2^7 for a row's largest and end at 2^-24: scales of v that are 2^8 apart leave them 23 bits.  A score
            // loses to other rows of its group what lies below 2^-36 of their largest.
            uint32_t ek, ev;
            Seen::tops(word, ek, ev);
            const float most = fmaxf(q.scale[0], q.scale[1]) * exp_scale(ek);
            Seen::add(word, ek, ev, __any_sync(0xffffffffu, most > kFineFactor) ? 8 : 255, 8, !(most < kMostFactor));
            cur = ek | ev << 8;
            mixed = __any_sync(0xffffffffu, word != cur);
            S[0] = S[1] = pair(exp_scale(ev), exp_scale(ev));
#pragma unroll
            for (int r = 0; r < 2; ++r) c[r] = pair(q.scale[r] * exp_scale(ek), q.scale[r] * exp_scale(ek));
        }
        float x[T][4];
        dot_tiles<NT, LO>(q, rb + dot_off, x);
        if (mixed) scale_tiles<NT>(x, word, cur, 0, 1);
        float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const pair_t b = DIST ? lds_pair(rb + tile_offset<NT, LO>(t) + 2 * tq * RB + split_scalars(LO) + 8) : 0;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float2 y = unpair(fma_pair(pair(x[t][2 * r], x[t][2 * r + 1]), c[r], DIST ? add_pair(nref[t % NT][r], b) : nref[t % NT][r]));
                x[t][2 * r] = y.x;
                x[t][2 * r + 1] = y.y;
                top[2 * (t / NT) + r] = max3(top[2 * (t / NT) + r], y.x, y.y);
            }
        }
        // centre column 0 does not meet the last column of the windows, centre column 1 not the first
        if (last) {
#pragma unroll
            for (int t = NT; t < T; ++t) x[t][0] = x[t][1] = -INFINITY;
            top[2] = -INFINITY;
        }
        // the first step sets the references; later they move when a score lies far above the earlier ones
        if (__any_sync(0xffffffffu, first || max3(fmaxf(top[0], top[1]), top[2], top[3]) > kTop)) {
            if (first) {
#pragma unroll
                for (int t = 0; t < NT; ++t) x[t][2] = x[t][3] = -INFINITY;
                top[1] = -INFINITY;
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                float d = quad_max(fmaxf(top[r], top[2 + r]));
                if ((first || d > kTop) && d > -INFINITY) {
                    d = kStart - d;
                    const float corr = first ? 1.f : fast_exp2(d);
                    const pair_t dd = pair(d, d), cc = pair(corr, corr);
                    shift[r] += d;
                    l[r] = mul_pair(l[r], cc);
#pragma unroll
                    for (int n = 0; n < 2; ++n) acc[n][r] = mul_pair(acc[n][r], cc);
#pragma unroll
                    for (int t = 0; t < T; ++t) {
                        x[t][2 * r] += d;
                        x[t][2 * r + 1] += d;
                        if (t < NT) nref[t][r] = add_pair(nref[t][r], dd);
                    }
                }
            }
        }
#pragma unroll
        for (int t = 0; t < T; ++t) {
#pragma unroll
            for (int i = 0; i < 4; ++i) x[t][i] = fast_exp2(x[t][i]);
#pragma unroll
            for (int r = 0; r < 2; ++r) l[r] = add_pair(l[r], pair(x[t][2 * r], x[t][2 * r + 1]));
        }
        if (mixed) scale_tiles<NT>(x, word, cur, 8, 0);
        uint32_t hi[T][2], lo[T][2];
#pragma unroll
        for (int t = 0; t < T; ++t) {
            split2(x[t][0], x[t][1], hi[t][0], lo[t][0]);
            split2(x[t][2], x[t][3], hi[t][1], lo[t][1]);
        }
        outer_tiles<NT, LO>(hi, lo, rb + outer_off, rb + tail_off, S, acc);
    }
    __device__ __forceinline__ void end(int w0, float poison) {
        const Geo& g = a.g;
        if (Seen::bad() && poison == 0.f) {
            exact_fwd(a, u, h - (lane >> 2), w0, exact_rows<NT, LO>());
            return;
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float2 ll = unpair(l[r]);
            const float sum = quad_sum(ll.x + ll.y);
            if (h >= g.H || w0 + r >= g.W) continue;
            const float inv = 1.f / sum + poison;
            const int pix = h + g.H * (w0 + r);
            const float2 y0 = unpair(acc[0][r]), y1 = unpair(acc[1][r]);
            store_pixel(a.o0, g, u, pix, tq, y0.x * inv, y0.y * inv, y1.x * inv, y1.y * inv);
            if (a.ostats && tq == 0) a.ostats[(int64_t)u * g.Np + pix] = (log2f(sum) - shift[r]) * kLn2 + poison;
        }
    }
};

// Five blocks per SM where the registers suffice: two tiles a column, or no lower halves (8 to 40 bytes spilled at three and four tiles).
template <int NT, bool DIST, bool LO>
__global__ void __launch_bounds__(32 * kSplitWarps, NT == 2 || !LO ? 5 : 4) split_fwd_kernel(const __grid_constant__ SplitArgs a, const __grid_constant__ CUtensorMap map) {
    FwdSweep<NT, DIST, LO> sweep(a);
    split_run<NT, LO>(a, &map, sweep);
}

// A's values: the scores once more, weighed with the row's log-sum-exp.  The runs of a step's two window columns are put in order in
// shared memory and leave row by row, 8 ws bytes that are contiguous but for the wrap: stored from the accumulators they
// were 4-byte pieces 8 bytes apart (128 x 96, 8 units, ws 15: 75 us).
template <int NT, bool DIST, bool LO>
struct EmitSweep {
    static constexpr int RB = split_row_bytes(LO), SB = split_stage_bytes(NT, LO), T = 2 * NT;
    const SplitArgs& a;
    int lane, tq, h, u, w, s, rows;                          // s: the next column of the window; rows of the warp in the image
    uint32_t dot_off, word_off, buf;
    float sl2;
    Centre<LO> q;
    pair_t nref[2], c[2];
    int at[NT][2];                                           // shared address of a tile's element for the first row and window column, -1: outside
    uint32_t cur;

    __device__ __forceinline__ EmitSweep(const SplitArgs& a_) : a(a_) {
        const int row0 = blockIdx.y * 8 * kSplitWarps + 8 * (threadIdx.x >> 5);
        lane = threadIdx.x & 31;
        tq = lane & 3;
        h = row0 + (lane >> 2);
        u = blockIdx.z;
        sl2 = a.scale * kLog2e;
        dot_off = dot_offset(lane, LO);
        word_off = word_offset<NT, LO>(a.g, lane, row0);
    }

    __device__ __forceinline__ void begin(int w0, uint32_t own) {
        const Geo& g = a.g;
        w = w0;
        s = 0;
        buf = own + (threadIdx.x >> 5) * (16 * 2 * g.ws * 4);
        rows = min(8, g.H - (h - (lane >> 2)));
        cur = 0;
        Raw raw;
        float L[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) L[r] = __ldg(a.stats + (int64_t)u * g.Np + min(h, g.H - 1) + g.H * min(w0 + r, g.W - 1));
        raw.load(a.c0, g, u, h, w0, tq);
        q.form(raw, g, h, w0, tq, kLeastExp);
        Seen::clear(q.bad);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float b = (DIST ? -0.5f * sl2 * q.norm2[r] : 0.f) - L[r] * kLog2e;
            nref[r] = pair(b, b);
            q.scale[r] *= sl2;
            c[r] = 0;
        }
        const int rot = run_rot(h, g.H, g.p, g.ws);
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int d = 8 * t + 2 * tq + i - (lane >> 2);
                at[t][i] = h >= g.H || d < 0 || d >= g.ws ? -1 : (int)buf + 4 * ((lane >> 2) * 2 * g.ws + (d + rot >= g.ws ? d + rot - g.ws : d + rot));
            }
    }

    __device__ __forceinline__ void step(uint32_t rb, bool first, bool last) {
        const Geo& g = a.g;
        const uint32_t word = ldsu32(rb + word_off) & 255u;
        bool mixed = false;
        if (__any_sync(0xffffffffu, word != cur)) {
            uint32_t none;
            Seen::tops(word, cur, none);
            const float most = fmaxf(q.scale[0], q.scale[1]) * exp_scale(cur);
            Seen::add(word, cur, none, __any_sync(0xffffffffu, most > kFineFactor) ? 8 : 255, 8, !(most < kMostFactor));
            mixed = __any_sync(0xffffffffu, word != cur);
#pragma unroll
            for (int r = 0; r < 2; ++r) c[r] = pair(q.scale[r] * exp_scale(cur), q.scale[r] * exp_scale(cur));
        }
        float x[T][4];
        dot_tiles<NT, LO>(q, rb + dot_off, x);
        if (mixed) scale_tiles<NT>(x, word, cur, 0, 1);
        __syncwarp();
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const pair_t b = DIST ? lds_pair(rb + half * SB + (8 * t + 2 * tq) * RB + split_scalars(LO) + 8) : 0;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float2 y = unpair(fma_pair(pair(x[half * NT + t][2 * r], x[half * NT + t][2 * r + 1]), c[r],
                                                     DIST ? add_pair(nref[r], b) : nref[r]));
                    if (at[t][0] >= 0) sts32(at[t][0] + (16 * r + half) * 4 * g.ws, fast_exp2(y.x));
                    if (at[t][1] >= 0) sts32(at[t][1] + (16 * r + half) * 4 * g.ws, fast_exp2(y.y));
                }
            }
        __syncwarp();
        // a lane takes one element of both columns' rows and goes through the eight rows
        for (int f = lane; f < 4 * g.ws; f += 32) {
            const int r = f >= 2 * g.ws, e = f - 2 * r * g.ws, half = e >= g.ws;
            // centre column 0 does not meet the last column of the windows, centre column 1 not the first
            if (w + r >= g.W || (half == 0 ? r == 1 && first : r == 0 && last)) continue;
            float* to = a.o0 + ((int64_t)u * g.Np + h - (lane >> 2) + (int64_t)g.H * (w + r)) * g.K +
                        axis_pos(s + half - g.p - r, w + r, g.W, g.p, g.ws) * g.ws + e - half * g.ws;
            const uint32_t src = buf + 4 * (16 * r * g.ws + e);
            float z[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) z[i] = lds32(src + 8 * i * g.ws);
#pragma unroll
            for (int i = 0; i < 8; ++i, to += g.K)
                if (i < rows) *to = z[i];
        }
        s += 2;
    }

    __device__ __forceinline__ void end(int w0, float poison) {
        const Geo& g = a.g;
        if (poison == 0.f) {
            if (Seen::bad()) exact_values(a, u, h - (lane >> 2), w0, exact_rows<NT, LO>());
        } else if (tq < 2 && h < g.H && w0 + tq < g.W) {
            for (int i = 0; i < g.K; ++i) a.o0[((int64_t)u * g.Np + h + g.H * (w0 + tq)) * g.K + i] = poison;
        }
    }
};

template <int NT, bool DIST, bool LO>
__global__ void __launch_bounds__(32 * kSplitWarps, 4) split_emit_kernel(const __grid_constant__ SplitArgs a, const __grid_constant__ CUtensorMap map) {
    EmitSweep<NT, DIST, LO> sweep(a);
    split_run<NT, LO>(a, &map, sweep);
}

}  // namespace

int run_split_fwd(const Geo& g, float scale, int dist, const float* q, const float* k, const float* v, const float* kv, float* y, float* stats,
                  cudaStream_t st) {
    Launch L{};
    SplitArgs a{};
    const int nt = split_tiles(g);
    const int rc = split_prepare(g, scale, dist, kv, &L, &a);
    if (rc) return rc;
    a.c0 = q; a.o0 = y; a.ostats = stats; a.x0 = k; a.x1 = v;
#define CA_SPLIT_FWD(KERNEL, NTV)                                                               \
    do {                                                                                             \
        if (g.bf16) {                                                                                \
            if (dist) CA_LAUNCH_SPLIT((KERNEL<NTV, true, false>), a, L, st);                    \
            else CA_LAUNCH_SPLIT((KERNEL<NTV, false, false>), a, L, st);                        \
        } else {                                                                                     \
            if (dist) CA_LAUNCH_SPLIT((KERNEL<NTV, true, true>), a, L, st);                     \
            else CA_LAUNCH_SPLIT((KERNEL<NTV, false, true>), a, L, st);                         \
        }                                                                                            \
    } while (0)
#define CA_SPLIT_FWD_NT(KERNEL)                                                                 \
    do {                                                                                             \
        if (nt == 2) CA_SPLIT_FWD(KERNEL, 2);                                                   \
        else if (nt == 3) CA_SPLIT_FWD(KERNEL, 3);                                              \
        else if (nt == 4) CA_SPLIT_FWD(KERNEL, 4);                                              \
        else return CA_ERR_UNSUPPORTED;                                                              \
    } while (0)
    CA_SPLIT_FWD_NT(split_fwd_kernel);
    CA_CHECK_LAUNCH("split forward kernel");
    return CA_OK;
}

int run_split_emit(const Geo& g, float scale, int dist, const float* q, const float* k, const float* stats, const float* kv, float* nz,
                   cudaStream_t st) {
    Launch L{};
    SplitArgs a{};
    const int nt = split_tiles(g);
    const int rc = split_prepare(g, scale, dist, kv, &L, &a, kSplitWarps * 16 * 2 * g.ws * sizeof(float));
    if (rc) return rc;
    a.c0 = q; a.stats = stats; a.o0 = nz; a.x0 = k;
    CA_SPLIT_FWD_NT(split_emit_kernel);
    CA_CHECK_LAUNCH("split values kernel");
    return CA_OK;
}

}  // namespace ca
