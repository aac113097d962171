// A's values in CSR order on the tiled kernels (compiled by emit_exact.cu and emit_any.cu).
#include "tile_common.cuh"

namespace ca {
namespace {

// =====================================================================
// A in CSR order.  Second sweep over the same packed (k|v) stages: with the
// saved log-sum-exp the normalised entry is P = 2^(q.k - L) directly; without
// row statistics (cs0 == NULL) the kernel writes the scaled scores themselves,
// which is the stand-alone similarity operator.  A thread
// produces, per stage, the ws entries of one (row, window column) run, which
// are contiguous in the row's CSR segment; a warp stages its 32 rows x ws run
// in shared memory and writes it out with consecutive lanes on consecutive
// addresses, so the 4*K*heads bytes per pixel leave the SM in full sectors.
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
    float* tile = reinterpret_cast<float*>(smem_al + (size_t)a.nsplit * a.nstages * a.stage_bytes) +
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
    u64 q[NQ][8];
    load_centre<CPE, NQ, NCRT>(a.c0, g, u, h, w0, active, sl2, q, 16 * slab);
    u64 nL2[NQ];
    float bq[NQ];
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
    const int64_t warp_row0 = (int64_t)u * g.Np + hw0;

    CA_PIPE_LOOP({
        const int mask = stage_mask<NQ>(s, pw);
        const uint32_t rowbase = pipe.vec(buf, a) + (lr + a.roff) * RB;
        for (int d0 = 0; d0 < g.ws; d0 += CH) {
            const int len = min(CH, g.ws - d0);                // window rows d0 .. d0 + len - 1
            // the dot products of all centre columns run interleaved (the columns that do not pair with this stage are
            // computed too and dropped: cheaper than serial chains)
            {
                u64 kn[8];                                 // the next window row's vector, fetched one row ahead
                lds_slab16<NS>(rowbase + d0 * RB, 0, slab, kn);
#pragma unroll (NQ == 1 ? 4 : 2)
                for (int e = 0; e < len; ++e) {
                    u64 k2[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) k2[i] = kn[i];
                    if (e + 1 < len) lds_slab16<NS>(rowbase + (d0 + e + 1) * RB, 0, slab, kn);
                    float bk = 0.f;
                    if (DIST) {
                        u64 n = zero2();
#pragma unroll
                        for (int i = 0; i < 8; ++i) n = fma2(k2[i], k2[i], n);
                        bk = -0.5f * sl2 * hsum2(n);
                    }
                    u64 t[NQ];
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
                    for (int r = 0; r < NQ; ++r) {
                        if (!((mask >> r) & 1)) continue;
                        float sc = hsum2(t[r]);
#pragma unroll
                        for (int m = 1; m < NS; m <<= 1) sc += __shfl_xor_sync(0xffffffffu, sc, m);
                        if (slab == 0) tile[(r * RW + lrow) * CHS + e] = raw ? sc * kLn2 : fast_exp2(sc);
                    }
                }
            }
            __syncwarp();
            // write this piece of the runs of the stage: row j, positions posw*ws + (d + rot_j) mod ws
#pragma unroll 1
            for (int r = 0; r < NQ; ++r) {
                if (!((mask >> r) & 1) || w0 + r >= g.W) continue;
                const int posw = axis_pos(s - pw - r, w0 + r, g.W, pw, g.wsw);
                float* dst = a.o0 + ((warp_row0 + (int64_t)g.H * (w0 + r)) * g.K + posw * g.ws);
                const float* src = tile + r * RW * CHS;
                // rows of this column (the last column of a folded signal may be shorter)
                const int n = min(RW, (kAnyC ? min(g.H, g.Np - g.H * (w0 + r)) : g.H) - hw0) * len;
                if (tabled) {                                      // CHS == len == ws: tile index == idx
#pragma unroll 4
                    for (int idx = lane; idx < n; idx += 32) dst[etab[idx]] = src[idx];
                    continue;
                }
                int row = lane / len, e = lane - row * len;        // element idx = row*len + e
                const int drow = 32 / len, de = 32 - drow * len;
                for (int idx = lane; idx < n; idx += 32) {
                    int posh = d0 + e + rots[r * RW + row];
                    posh -= (posh >= g.ws) ? g.ws : 0;
                    dst[(int64_t)row * g.K + posh] = src[row * CHS + e];
                    row += drow;
                    e += de;
                    if (e >= len) { e -= len; ++row; }
                }
            }
            __syncwarp();
        }
    })
}

}  // namespace

// Two columns per thread, four CTAs per SM: the kernel waits on latencies, and four columns (156 registers, two to three
// CTAs) took 135 us where two take 77 us at 128 x 96 x 64 x 2, ws 15, 4 heads, Distance (88 MB of values: 14 us at the HBM
// peak); 320 x 320 x 32 complex, 8 units, ws 7: 638 -> 586 us.  Folded 1-D signals have one: 8192 x 64 x 4, ws 63, 4 heads
// 84 -> 55 us.
template <>
int run_emit<kAnyC>(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* stats, float* nz,
                    const float* packed, cudaStream_t st, bool single) {
    if (!tiled_operator_ok(g)) return CA_ERR_UNSUPPORTED;
    const int ns = slabs_of(g);
    Launch L{};
    // three copy stages, or two when that lets one more CTA reside on an SM
    const int ch = std::min(g.ws, kRunChunk), nq = g.wsw == 1 ? 1 : 2;
    int rc = CA_OK;
    auto setup = [&](int stages) {
        L = Launch{};
        rc = prepare(g, P, operator_tile(g, ns, nq, nq == 1 ? 1 : 2, 4), 0, packed, nullptr, &L, ns, single, stages);
        // per warp: staging tile, run rotations, offset table
        if (!rc) L.smem += (size_t)L.threads / 32 * (32 / ns) * (nq * (ch + 1) + nq + ch) * sizeof(float);
        return rc;
    };
    if (setup(kStages)) return rc;
    {
        const size_t per_sm = 227 * 1024, with3 = L.smem + 1024;          // + the driver's per-CTA reservation
        const size_t with2 = with3 - (size_t)L.a.nsplit * L.a.stage_bytes;
        const size_t most = nq == 1 ? 6 : 4;                 // CTAs per SM that the registers allow
        if (std::min(most, per_sm / with2) > std::min(most, per_sm / with3))
            if (setup(2)) return rc;
    }
    if (L.smem > 200 * 1024) return CA_ERR_UNSUPPORTED;
#define CA_EMIT(NQV, NSV)                                                                  \
    do {                                                                              \
        if (g.cpe == 1) {                                                             \
            if (dist) CA_LAUNCH_TILED((emit_a_tiled_kernel<true, 1, NQV, NSV>), L, st);  \
            else CA_LAUNCH_TILED((emit_a_tiled_kernel<false, 1, NQV, NSV>), L, st);   \
        } else {                                                                      \
            if (dist) CA_LAUNCH_TILED((emit_a_tiled_kernel<true, 2, NQV, NSV>), L, st);  \
            else CA_LAUNCH_TILED((emit_a_tiled_kernel<false, 2, NQV, NSV>), L, st);   \
        }                                                                             \
    } while (0)
    L.a.scale = scale; L.a.c0 = q; L.a.cs0 = stats; L.a.o0 = nz;
#define CA_EMIT_NQ(NSV)                                                               \
    do {                                                                              \
        if (nq == 1) CA_EMIT(1, NSV);                                                 \
        else CA_EMIT(2, NSV);                                                         \
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
