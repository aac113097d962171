// A's values in CSR order on the tiled kernels (compiled by emit_exact.cu and emit_any.cu).
//
// Second sweep over the same packed (k|v) stages: with the saved log-sum-exp the normalised entry is
// P = 2^(q.k - L) directly; without row statistics (cs0 == NULL) the kernels write the scaled scores themselves, which is
// the stand-alone similarity operator.  A thread produces, per stage, the ws entries of one (row, window column) run of
// each of its centre columns; they go through shared memory so that A is written with consecutive lanes on
// consecutive addresses.
//
// Bound: issue slots and shared memory.  Per key and column a warp needs 16 FMAs (4 cycles of an SM), 16 / NQ cycles
// of vector reads and one store; so the scores leave the registers untransformed (scale or exp2 is applied on the way out,
// where every lane has one), and the lanes that share a pixel split the sums among them instead of all forming every sum.
#include "tile_common.cuh"

namespace ca {
namespace {

// Sums over the NS lanes of a pixel of V values each; lane `slab` ends with the total of value scatter_index(slab) (the
// lanes that scatter_owner() names: a total may lie in several).  V values cost V / 2 + V / 4 .. shuffles where a sum in
// every lane costs V log2(NS).
template <int NS, int V>
struct Scatter {
    static __device__ __forceinline__ float sum(const float (&v)[V], int slab) {
        if constexpr (V == 1) return lane_sum<NS>(v[0]);
        if constexpr (V == 2) {
            const bool odd = slab & 1;
            float x = odd ? v[1] : v[0];
            x += __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[1], 1);
            if constexpr (NS == 4) x += __shfl_xor_sync(0xffffffffu, x, 2);
            return x;
        }
        if constexpr (V == 4) {                        // NS == 4: values 2t + r; bit 1 of the lane takes t, bit 0 takes r
            const bool hi = slab & 2;
            float w[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) w[r] = (hi ? v[2 + r] : v[r]) + __shfl_xor_sync(0xffffffffu, hi ? v[r] : v[2 + r], 2);
            const bool odd = slab & 1;
            return (odd ? w[1] : w[0]) + __shfl_xor_sync(0xffffffffu, odd ? w[0] : w[1], 1);
        }
    }
};

// Partial scores (this lane's slab) of the key at a0 with all centre columns, chains interleaved.
template <bool DIST, int NQ, int NS>
__device__ __forceinline__ void emit_scores(uint32_t a0, int RB, int slab, float sl2, const u64 (&q)[NQ][8], const u64 (&nL2)[NQ],
                                            const float (&bq)[NQ], float (&sc)[NQ]) {
    u64 k2[8], t[NQ];
    lds_slab16<NS>(a0, 0, slab, k2);
    float bk = 0.f;
    if (DIST) bk = -0.5f * sl2 * lds_norm(a0, RB - 16 * NS, slab);
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        t[r] = nL2[r];
        if (DIST) t[r] = add2(t[r], pack2(bq[r] + bk, 0.f));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int r = 0; r < NQ; ++r) t[r] = fma2(q[r][i], k2[i], t[r]);
#pragma unroll
    for (int r = 0; r < NQ; ++r) sc[r] = hsum2(t[r]);
}

// `len` keys from a0 on: the score of key e and column r goes to run[r] + pos, where pos starts at `pos`, moves on by a word
// per key and returns to 0 at `wrap` bytes.  Columns outside `mask` are computed and dropped (cheaper than serial chains).
template <bool DIST, int NQ, int NS>
__device__ __forceinline__ void emit_keys(uint32_t a0, int RB, int len, int slab, float sl2, const u64 (&q)[NQ][8],
                                          const u64 (&nL2)[NQ], const float (&bq)[NQ], const uint32_t (&run)[NQ], int pos, int wrap,
                                          int mask) {
    // the column whose totals this lane stores, and whether it stores any
    const int r_own = NQ == 2 && NS > 1 ? slab & 1 : 0;
    const uint32_t own = r_own ? run[NQ - 1] : run[0];
    const bool on = (mask >> r_own) & 1;
#pragma unroll 2
    for (; len >= 2; len -= 2, a0 += 2 * RB) {
        float s0[NQ], s1[NQ];
        emit_scores<DIST, NQ, NS>(a0, RB, slab, sl2, q, nL2, bq, s0);
        emit_scores<DIST, NQ, NS>(a0 + RB, RB, slab, sl2, q, nL2, bq, s1);
        const int pos1 = pos + 4 == wrap ? 0 : pos + 4;
        if constexpr (NS == 1) {
#pragma unroll
            for (int r = 0; r < NQ; ++r)
                if ((mask >> r) & 1) { sts32(run[r] + pos, s0[r]); sts32(run[r] + pos1, s1[r]); }
        } else if constexpr (NQ == 1) {
            const float v[2] = {s0[0], s1[0]};
            const float x = Scatter<NS, 2>::sum(v, slab);
            if (slab < 2) sts32(own + (slab ? pos1 : pos), x);
        } else if constexpr (NS == 2) {
            const float x0 = Scatter<2, 2>::sum(s0, slab), x1 = Scatter<2, 2>::sum(s1, slab);
            if (on) { sts32(own + pos, x0); sts32(own + pos1, x1); }
        } else {
            const float v[4] = {s0[0], s0[1], s1[0], s1[1]};
            const float x = Scatter<4, 4>::sum(v, slab);
            if (on) sts32(own + (slab & 2 ? pos1 : pos), x);
        }
        pos = pos1 + 4 == wrap ? 0 : pos1 + 4;
    }
    if (len) {
        float s0[NQ];
        emit_scores<DIST, NQ, NS>(a0, RB, slab, sl2, q, nL2, bq, s0);
        if constexpr (NS == 1) {
#pragma unroll
            for (int r = 0; r < NQ; ++r)
                if ((mask >> r) & 1) sts32(run[r] + pos, s0[r]);
        } else {
            const float x = Scatter<NS, NQ>::sum(s0, slab);
            if (slab < NQ && on) sts32(own + pos, x);
        }
    }
}

// What leaves the kernels for a score in the log2 domain.
__device__ __forceinline__ float emit_value(float x, bool raw) { return raw ? x * kLn2 : fast_exp2(x); }

// Centre pixels and row statistics of a thread.
template <bool DIST, int CPE, int NQ, int NCRT>
__device__ __forceinline__ void emit_centre(const TileArgs& a, int u, int h, int w0, bool active, int slab, float sl2, bool raw, u64 (&q)[NQ][8],
                                            u64 (&nL2)[NQ], float (&bq)[NQ]) {
    const Geo& g = a.g;
    load_centre<CPE, NQ, NCRT>(a.c0, g, u, h, w0, active, sl2, q, 16 * slab);
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        const bool ok = active && has_pixel(g, h, w0 + r) && slab == 0;   // the row statistic enters the lane sum once
        nL2[r] = pack2((ok && !raw) ? -__ldg(a.cs0 + (int64_t)u * g.Np + h + g.H * (w0 + r)) * kLog2e : 0.f, 0.f);
        bq[r] = 0.f;
        if (DIST) {
            u64 n = zero2();
#pragma unroll
            for (int i = 0; i < 8; ++i) n = fma2(q[r][i], q[r][i], n);
            bq[r] = -0.5f * hsum2(n) / sl2;
        }
    }
}

// =====================================================================
// Long rows: a warp stages its rows x ws run of a stage and writes it out before the next.
// =====================================================================
// NCRT = real channels per unit, zero-extended to 16, 32 or 64.  NQ = centre columns per thread (1: folded signals).
template <bool DIST, int CPE, int NQ, int NCRT>
__global__ void __launch_bounds__(128, (NQ == 1 ? 6 : 4)) emit_a_tiled_kernel(TileArgs a, const __grid_constant__ CUtensorMap mv,
                                                              const __grid_constant__ CUtensorMap msc) {
    constexpr int NS = NCRT <= 16 ? 1 : NCRT / 16;             // 16-channel slabs = lanes per pixel
    constexpr int RW = 32 / NS;                                // pixel rows per warp
    const Geo& g = a.g;
    const int RB = a.row_bytes;                                // packed row: pair (144*NS) or single tensor (80*NS)
    const int ROWS = a.TH + 2 * (g.p + a.roff);
    const int pw = radius_w(g);
    const int w0 = blockIdx.x * NQ, h0 = blockIdx.y * a.TH, u = blockIdx.z;
    const int NSTAGES = g.wsw + min(NQ - 1, g.W - 1 - w0);          // no stages for centre columns past the image
    const float sl2 = a.scale * kLog2e;
    CA_PIPE_PROLOGUE(false, kParts)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slab = lane % NS, lrow = lane / NS;              // this lane's channel slab and row inside the warp
    const int lr = (lt >> 5) * RW + lrow, h = h0 + lr;         // row inside the tile, image row
    const bool active = h < g.H;
    // per-warp staging tile [NQ][RW][CH] after the stage buffers: the entries of CH = min(ws, 32)
    // consecutive window rows at a time, then the run rotations of the warp's rows [NQ][RW]
    const int CH = min(g.ws, kRunChunk);
    const int CHS = CH | 1;                                    // odd row stride: conflict-free column access
    constexpr int nslots = NQ;                                 // one staging slot per centre column
    float* tile = reinterpret_cast<float*>(smem_al + a.extra_off) +
                  (size_t)warp * (nslots * RW * CHS + NQ * RW + RW * CH);     // tile, rotations, offset table
    int* rots = reinterpret_cast<int*>(tile + nslots * RW * CHS);
    // 2-D windows that fit one piece: the destination offset of every tile element is the same
    // for all stages and centre columns (row*K + sorted position) and comes from a table
    const bool tabled = g.ws <= kRunChunk && g.wsw != 1;
    int* etab = rots + NQ * RW;
    const int hw0 = h0 + (lt >> 5) * RW;                       // first image row of this warp
    for (int i = lane; i < NQ * RW; i += 32)
        rots[i] = run_rot(axis_coord(g, hw0 + i % RW, w0 + i / RW), axis_len(g), g.p, g.ws);
    if (tabled)
        for (int idx = lane; idx < RW * g.ws; idx += 32) {
            const int row = idx / g.ws, e = idx - row * g.ws;
            int posh = e + run_rot(hw0 + row, g.H, g.p, g.ws);
            posh -= (posh >= g.ws) ? g.ws : 0;
            etab[idx] = row * g.K + posh;
        }
    __syncwarp();

    const bool raw = a.cs0 == nullptr;
    u64 q[NQ][8], nL2[NQ];
    float bq[NQ];
    emit_centre<DIST, CPE, NQ, NCRT>(a, u, h, w0, active, slab, sl2, raw, q, nL2, bq);
    uint32_t run[NQ];
#pragma unroll
    for (int r = 0; r < NQ; ++r) run[r] = smem_u32(tile + (r * RW + lrow) * CHS);
    const int64_t warp_row0 = (int64_t)u * g.Np + hw0;

    CA_PIPE_LOOP({
        const int mask = stage_mask<NQ>(s, pw);
        const uint32_t rowbase = pipe.vec(buf, a) + (lr + a.roff) * RB;
        for (int d0 = 0; d0 < g.ws; d0 += CH) {
            const int len = min(CH, g.ws - d0);                // window rows d0 .. d0 + len - 1
            emit_keys<DIST, NQ, NS>(rowbase + d0 * RB, RB, len, slab, sl2, q, nL2, bq, run, 0, 1 << 20, mask);
            __syncwarp();
            // write this piece of the runs of the stage: row j, positions posw*ws + (d + rot_j) mod ws
            _Pragma("unroll 1")
            for (int r = 0; r < NQ; ++r) {
                if (!((mask >> r) & 1) || w0 + r >= g.W) continue;
                const int posw = axis_pos(s - pw - r, w0 + r, g.W, pw, g.wsw);
                float* dst = a.o0 + ((warp_row0 + (int64_t)g.H * (w0 + r)) * g.K + posw * g.ws);
                const float* src = tile + r * RW * CHS;
                // rows of this column (the last column of a folded signal may be shorter)
                const int n = min(RW, (kAnyC ? min(g.H, g.Np - g.H * (w0 + r)) : g.H) - hw0) * len;
                if (tabled) {                                      // CHS == len == ws: tile index == idx
                    _Pragma("unroll 4")
                    for (int idx = lane; idx < n; idx += 32) dst[etab[idx]] = emit_value(src[idx], raw);
                    continue;
                }
                int row = lane / len, e = lane - row * len;        // element idx = row*len + e
                const int drow = 32 / len, de = 32 - drow * len;
                for (int idx = lane; idx < n; idx += 32) {
                    int posh = d0 + e + rots[r * RW + row];
                    posh -= (posh >= g.ws) ? g.ws : 0;
                    dst[(int64_t)row * g.K + posh] = emit_value(src[row * CHS + e], raw);
                    row += drow;
                    e += de;
                    if (e >= len) { e -= len; ++row; }
                }
            }
            __syncwarp();
        }
    })
    if (ca_poison != 0.f) {                                    // a wait ran out: nothing of this tile passes for a result
        for (int r = 0; r < NQ && w0 + r < g.W; ++r) {
            const int64_t n = (int64_t)min(RW, (kAnyC ? min(g.H, g.Np - g.H * (w0 + r)) : g.H) - hw0) * g.K;
            for (int64_t i = lane; i < n; i += 32) a.o0[(warp_row0 + (int64_t)g.H * (w0 + r)) * g.K + i] = ca_poison;
        }
    }
}

// =====================================================================
// The same values where the rows of A are short: a warp keeps the whole rows of its pixels in shared memory, every
// score goes to its final position, and after the last stage the rows of a centre column, which are one contiguous
// piece of A, are stored with consecutive lanes on consecutive addresses.  (Written per stage, a row of a 7-wide
// window is seven runs of 28 bytes, each with its staging, its two warp barriers and its offset arithmetic.)  K is odd,
// so the lanes' rows lie in distinct banks.  Bound: the shared-memory reads of the keys, 16 bytes per four FMAs and column.
// The groups of warps that share the stages of a tile share its rows.
// =====================================================================
template <bool DIST, int CPE, int NQ, int NCRT>
__global__ void __launch_bounds__(128, (NQ == 1 ? 6 : 4)) emit_rows_kernel(TileArgs a, const __grid_constant__ CUtensorMap mv,
                                                              const __grid_constant__ CUtensorMap msc) {
    constexpr int NS = NCRT <= 16 ? 1 : NCRT / 16;
    constexpr int RW = 32 / NS;
    const Geo& g = a.g;
    const int RB = a.row_bytes;
    const int ROWS = a.TH + 2 * (g.p + a.roff);
    const int pw = radius_w(g);
    const int w0 = blockIdx.x * NQ, h0 = blockIdx.y * a.TH, u = blockIdx.z;
    const int NSTAGES = g.wsw + min(NQ - 1, g.W - 1 - w0);
    const float sl2 = a.scale * kLog2e;
    CA_PIPE_PROLOGUE(false, kParts)
    const int lane = threadIdx.x & 31, slab = lane % NS, lrow = lane / NS;
    const int lr = (lt >> 5) * RW + lrow, h = h0 + lr, hw0 = h0 + (lt >> 5) * RW;
    const bool active = h < g.H;
    float* tile = reinterpret_cast<float*>(smem_al + a.extra_off) + (lt >> 5) * (NQ * RW * g.K);
    const uint32_t mine = smem_u32(tile + lrow * g.K);
    // rotation of this lane's runs (2-D: the same in every column); rows without a pixel write plain rows that nobody stores
    const int rot = active && has_pixel(g, h, w0) ? run_rot(axis_coord(g, h, w0), axis_len(g), g.p, g.ws) : 0;

    const bool raw = a.cs0 == nullptr;
    u64 q[NQ][8], nL2[NQ];
    float bq[NQ];
    emit_centre<DIST, CPE, NQ, NCRT>(a, u, h, w0, active, slab, sl2, raw, q, nL2, bq);

    CA_PIPE_LOOP({
        const int mask = stage_mask<NQ>(s, pw);
        uint32_t run[NQ];                                  // where the runs of this lane's row start
        _Pragma("unroll")
        for (int r = 0; r < NQ; ++r)
            run[r] = mine + (r * RW * g.K + (((mask >> r) & 1) && w0 + r < g.W ? axis_pos(s - pw - r, w0 + r, g.W, pw, g.wsw) * g.ws : 0)) * 4;
        emit_keys<DIST, NQ, NS>(pipe.vec(buf, a) + (lr + a.roff) * RB, RB, g.ws, slab, sl2, q, nL2, bq, run, rot * 4, g.ws * 4, mask);
    })

#pragma unroll 1
    for (int r = 0; r < NQ; ++r) {
        if (w0 + r >= g.W) break;
        // rows of this column (the last column of a folded signal may be shorter)
        const int n = min(RW, (kAnyC ? min(g.H, g.Np - g.H * (w0 + r)) : g.H) - hw0) * g.K;
        float* dst = a.o0 + ((int64_t)u * g.Np + hw0 + (int64_t)g.H * (w0 + r)) * g.K;
        const float* src = tile + r * RW * g.K;
#pragma unroll 4
        for (int idx = part * 32 + lane; idx < n; idx += 32 * a.nsplit) dst[idx] = emit_value(src[idx], raw) + ca_poison;
    }
}

}  // namespace

// Whole rows of A in shared memory (emit_rows_kernel), one or two columns per thread, and runs (emit_a_tiled_kernel), two
// (folded signals: one).  The line lies at 7 KB of rows per warp and column: 320 x 320, 8 units of 64 channels, ws 7 (1.6 KB):
// rows 417, runs 457 us; 200 x 200, 2 of 64, ws 9 (2.6 KB): 75 and 87; 320 x 240, 4 of 16, ws 5 (3.2 KB): 35 and 40; 400 x 380,
// 2 of 16, ws 7 (6.3 KB): 63 and 69; 128 x 96, 4 of 64, ws 15 (7.2 KB): 113 and 108; 150 x 140, 4 of 32, ws 11 (7.7 KB): 63
// and 62; 256 x 256, 4 of 16, ws 9 (10.4 KB): 85 and 76.
static const SweepCost kRowsCost[3][2] = {{{1, 24, 56, 53, 994, 1479}, {2, 16, 85, 82, 1142, 2556}},
                                          {{1, 24, 42, 55, 880, 1543}, {2, 16, 49, 82, 1045, 2402}},
                                          {{1, 24, 74, 69, 225, 2049}, {2, 16, 49, 104, 523, 2277}}};
static const SweepCost kRunsCost[3] = {{2, 16, 0, 105, 1603, 3771}, {2, 16, 0, 92, 2025, 2969}, {2, 16, 50, 99, 1694, 1474}};

template <>
int run_emit<kAnyC>(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* stats, float* nz,
                    const float* packed, cudaStream_t st, bool single) {
    if (!tiled_operator_ok(g)) return CA_ERR_UNSUPPORTED;
    const int ns = slabs_of(g), rw = 32 / ns, slot = ns == 1 ? 0 : ns / 2;
    const int row_bytes = rw * g.K * (int)sizeof(float);
    const bool fold = g.wsw == 1, whole = row_bytes <= 7 * 1024;
    Launch L{};
    int rc = CA_OK, nq;
    if (whole) {
        const TileShape t = choose_tile(g, P, ns, kRowsCost[slot], fold ? 1 : 2, kParts, false, single, row_bytes, 2);
        nq = t.nq;
        if ((rc = prepare(g, P, t, 0, packed, nullptr, &L, ns, single, 2, (size_t)t.warps * nq * row_bytes))) return rc;
    } else {
        nq = fold ? 1 : 2;
        // of every warp: staging tile, run rotations, offset table
        const int ch = std::min(g.ws, kRunChunk), own = rw * (nq * (ch + 1) + nq + ch) * (int)sizeof(float);
        const TileShape t = fold ? TileShape{1, std::min(4, (g.H + rw - 1) / rw), 1}
                                 : choose_tile(g, P, ns, &kRunsCost[slot], 1, kParts, false, single, 0, 2, own);
        // three copy stages, or two when that lets one more CTA reside on an SM
        auto setup = [&](int stages) {
            L = Launch{};
            return rc = prepare(g, P, t, 0, packed, nullptr, &L, ns, single, stages, (size_t)t.warps * t.nsplit * own);
        };
        if (setup(kStages) && setup(2)) return rc;
        const size_t per_sm = 227 * 1024, with3 = L.smem + 1024;          // + the driver's per-CTA reservation
        const size_t with2 = with3 - (size_t)L.a.nsplit * L.a.stage_bytes;
        const size_t most = (nq == 1 ? 24 : 16) * 32 / L.threads;         // CTAs per SM that the registers allow
        if (L.a.nstages == kStages && std::min(most, per_sm / with2) > std::min(most, per_sm / with3) && setup(2)) return rc;
    }
    L.a.scale = scale; L.a.c0 = q; L.a.cs0 = stats; L.a.o0 = nz;
#define CA_EMIT(KERNEL, NQV, NSV)                                                            \
    do {                                                                                     \
        if (g.cpe == 1) {                                                                    \
            if (dist) CA_LAUNCH_TILED((KERNEL<true, 1, NQV, NSV>), L, st);                   \
            else CA_LAUNCH_TILED((KERNEL<false, 1, NQV, NSV>), L, st);                       \
        } else {                                                                             \
            if (dist) CA_LAUNCH_TILED((KERNEL<true, 2, NQV, NSV>), L, st);                   \
            else CA_LAUNCH_TILED((KERNEL<false, 2, NQV, NSV>), L, st);                       \
        }                                                                                    \
    } while (0)
#define CA_EMIT_NQ(NSV)                                                                      \
    do {                                                                                     \
        if (whole && nq == 1) CA_EMIT(emit_rows_kernel, 1, NSV);                             \
        else if (whole) CA_EMIT(emit_rows_kernel, 2, NSV);                                   \
        else if (nq == 1) CA_EMIT(emit_a_tiled_kernel, 1, NSV);                              \
        else CA_EMIT(emit_a_tiled_kernel, 2, NSV);                                           \
    } while (0)
    if (ns == 1) CA_EMIT_NQ(16);
    else if (ns == 2) CA_EMIT_NQ(32);
    else CA_EMIT_NQ(64);
#undef CA_EMIT_NQ
#undef CA_EMIT
    CA_CHECK_LAUNCH("tiled A kernel");
    return CA_OK;
}

}  // namespace ca
