// A (x) V and A^T (x) V on the tiled kernels (compiled by apply_exact.cu and apply_any.cu).
#include "tile_common.cuh"

namespace ca {
namespace {

// =====================================================================
// A (x) V and A^T (x) V from stored values.  The dense operand is streamed as
// packed column stages exactly like the keys of the forward; the values of A
// that pair with a stage are, for every centre column r, one run of ws
// consecutive entries per CSR row (window column fixed, window rows varying),
// which a warp copies into shared memory before the FMAs that use them:
//   plain     : the runs of the warp's own rows; lane wr uses entry (e + rotation) of its row at step e;
//   transposed: the runs of the streamed column's rows hw0 - p .. hw0 + RW - 1 + p; lane wr uses the entry of the
//               opposite offset of row wr + e (window symmetry: A[j, i] sits in row j at offset i - j).
// out = alpha * (sum_e a_e v_e - (sum_e a_e) * centre) with centre optional: the
// second term is the Distance similarity pullback.
//
// Staging.  Runs are copied as aligned 16-byte pieces, eight lanes per row.  The misalignment of a run grows by K
// (odd) modulo four words per row, so a row pitch of 4*C + K % 4 words (C pieces per run) puts the run of row t at
// word t * pitch + a exactly, a = misalignment of row 0: source and destination of a lane's pieces advance by
// constants (4 rows each), and the odd pitch makes the lanes' reads conflict free.  (Four-byte copies of
// single entries took 36 instructions per copy with their address arithmetic: 95 us at 128 x 96 x 64 x 2, ws 15,
// 4 heads, 41 % of the issue slots busy.)
//
// Bound: reading A (4 bytes per entry) and, next to it, 16 FMAs per entry and slab.  One thread per pixel row of
// four columns is only 768 warps at that size, five per SM, so up to four warps of a CTA share the stages of a tile.
// FMAs are packed (an outer product: 61 against 50 TFLOP/s in registers).  Measured times stand at run_apply().
// =====================================================================
__device__ __forceinline__ void cp_async16(uint32_t dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// acc += (a, a) * v on a channel pair as one packed FMA (outer products run at the packed rate: the coefficient pair
// is reused by consecutive instructions).
__device__ __forceinline__ void fma_outer(uint64_t& acc, uint64_t a2, uint64_t v) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a2), "l"(v));
}
__device__ __forceinline__ uint64_t dup2(float a) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ u64 split2(uint64_t v) {
    u64 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void lds128p(uint32_t addr, uint64_t& lo, uint64_t& hi) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "r"(addr));
}

// 16-byte pieces that cover a run of ws words at any misalignment, and the row pitch in words.  Rows that wrap around
// an axis whose length is no multiple of four change their misalignment, which takes one more piece of room.
__host__ __device__ inline int run_pieces(int ws) { return (ws + 6) / 4; }
__host__ __device__ inline int run_pitch(const Geo& g, bool loose) { return 4 * run_pieces(g.ws) + (loose ? 4 : 0) + (g.K & 3); }
// Words of one warp's run area: nslots centre columns of `rows` rows.
__host__ __device__ inline int run_area(const Geo& g, int rows, int nslots, bool loose) { return nslots * ((rows * run_pitch(g, loose) + 8) & ~3); }

// Position of the entry that lane pixel n (coordinate on the window axis of length X) needs from the row of the streamed
// pixel n - p + e, inside that row's run: the sorted columns of a border row start at the front of the axis, where
// column n is the n-th entry, and end at its back, where it is the (X - n)-th from the end.
__device__ __forceinline__ int transposed_pos(int n, int e, int X, int p, int ws) { return max(min(2 * p - e, n), n - X + ws); }

// Merges the parts of a tile and stores alpha * (sum - [centre] asum * centre).
template <int CPE, int NQ, int NCRT>
__device__ __forceinline__ void apply_finish(const TileArgs& a, unsigned char* smem_al, int part, int lt, int PT, int u, int h, int w0, bool active,
                                             int slab, float ca_poison, const uint64_t (&acc)[NQ][8], float (&asum)[NQ]) {
    const Geo& g = a.g;
    // parts 1.. publish their partial sums, part 0 adds them up
    if (a.nsplit > 1) {
        float* xch = reinterpret_cast<float*>(smem_al);
        if (part > 0) {
            float* x = xch + (size_t)(part - 1) * (17 * NQ) * PT + lt;
#pragma unroll
            for (int r = 0; r < NQ; ++r) {
                x[(16 * NQ + r) * PT] = asum[r];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const u64 t = split2(acc[r][i]);
                    x[(r * 16 + 2 * i) * PT] = t.x;
                    x[(r * 16 + 2 * i + 1) * PT] = t.y;
                }
            }
        }
        __syncthreads();
        if (part > 0) return;
    }
    u64 res[NQ][8];
#pragma unroll
    for (int r = 0; r < NQ; ++r)
#pragma unroll
        for (int i = 0; i < 8; ++i) res[r][i] = split2(acc[r][i]);
    for (int q = 1; q < a.nsplit; ++q) {
        const float* x = reinterpret_cast<float*>(smem_al) + (size_t)(q - 1) * (17 * NQ) * PT + lt;
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            asum[r] += x[(16 * NQ + r) * PT];
#pragma unroll
            for (int i = 0; i < 8; ++i) res[r][i] = add2(res[r][i], pack2(x[(r * 16 + 2 * i) * PT], x[(r * 16 + 2 * i + 1) * PT]));
        }
    }
    if (a.c0) {
        u64 ctr[NQ][8];
        load_centre<CPE, NQ, NCRT>(a.c0, g, u, h, w0, active, 1.f, ctr, 16 * slab);
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            const u64 ns = pack2(-asum[r], -asum[r]);
#pragma unroll
            for (int i = 0; i < 8; ++i) res[r][i] = fma2(ns, ctr[r][i], res[r][i]);
        }
    }
    CA_OUT_DISPATCH(
        _Pragma("unroll")
        for (int r = 0; r < NQ; ++r)
            _Pragma("unroll")
            for (int i = 0; i < 8; ++i)
                store_centre<CPE, NCRV, BF>(a.o0, g, u, h, w0, active, r, i, a.scale * res[r][i].x + ca_poison,
                                            a.scale * res[r][i].y + ca_poison, 16 * slab);)
}

// NQ = centre columns per thread (1: folded signals).
template <int CPE, bool TRANS, int NQ, int NCRT>
__global__ void __launch_bounds__(128, (NQ == 1 ? 6 : 4)) apply_tiled_kernel(TileArgs a, const __grid_constant__ CUtensorMap mv,
                                                             const __grid_constant__ CUtensorMap msc) {
    constexpr int NS = NCRT <= 16 ? 1 : NCRT / 16;             // 16-channel slabs = lanes per pixel
    constexpr int RW = 32 / NS;                                // pixel rows per warp
    constexpr int RB = kSingleFloats * 4 * NS;                 // bytes of a packed row of a single tensor
    const Geo& g = a.g;
    const int ROWS = a.TH + 2 * (g.p + a.roff);
    const int pw = radius_w(g), p2 = TRANS ? g.p : 0;
    const bool fold = NQ == 1;                                 // folded 1-D signal: rows continue into neighbour columns
    const int w0 = blockIdx.x * NQ, h0 = blockIdx.y * a.TH, u = blockIdx.z;
    const int NSTAGES = g.wsw + min(NQ - 1, g.W - 1 - w0);          // no stages for centre columns past the image
    CA_PIPE_PROLOGUE(false, kParts)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slab = lane % NS, lrow = lane / NS;              // this lane's channel slab and row inside the warp
    const int lr = (lt >> 5) * RW + lrow, h = h0 + lr;         // row inside the tile, image row
    const bool active = h < g.H;
    const int X = axis_len(g);
    const bool loose = TRANS && (X & 3);
    const int SR = run_pitch(g, loose), C = run_pieces(g.ws);
    const int NR = RW + (TRANS ? g.ws - 1 : 0);                // staged rows per centre column
    const int slot_words = run_area(g, NR, 1, loose), buf_words = NQ * slot_words;
    const uint32_t wbase = smem_u32(smem_al) + (uint32_t)a.nsplit * a.nstages * a.stage_bytes + (uint32_t)warp * a.nbuf * buf_words * 4;
    const int hw0 = h0 + (lt >> 5) * RW;                       // first image row of this warp
    const int xs = hw0 - p2;                                   // first staged row (plain: the warp's own)
    const bool wraps = TRANS && (fold || xs < 0 || xs + NR > g.H);   // a staged row may lie past an end of the axis
    const float* nzw = a.cs0 + ((int64_t)u * g.Np + xs) * g.K;
    const int64_t colstep = (int64_t)g.H * g.K;                // words between the same rows of neighbouring columns
    const float* own = nzw + colstep * w0;                     // plain: centre column 0

    // starts the copies of the runs of stage s into buffer tb; returns the misalignments of staged row 0, two bits per
    // centre column
    const int wr0 = lane >> 3, j0 = lane & 7;
    const int64_t step = 4 * (int64_t)g.K;
    auto fetch_runs = [&](int s, int tb) {
        const int mask = stage_mask<NQ>(s, pw), wc = stage_column(g, w0, s);
        // staged rows that some pixel of the image needs: the rest of a ragged tile is not copied
        const int hc = kAnyC && fold ? min(g.H, g.Np - g.H * (w0 + s)) : g.H;
        const int nrows = hw0 >= hc ? 0 : min(NR, hc - hw0 + 2 * p2);
        const float* col = TRANS ? nzw + colstep * wc : own;
        int mis4 = 0;
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            const int posw = TRANS ? axis_pos(r + pw - s, wc, g.W, pw, g.wsw) : axis_pos(s - pw - r, w0 + r, g.W, pw, g.wsw);
            const float* row0 = col + posw * g.ws;             // run of staged row 0
            if (!TRANS) col += colstep;
            if (!((mask >> r) & 1) || w0 + r >= g.W) continue;
            const int ar = (int)((uintptr_t)row0 >> 2) & 3;
            mis4 |= ar << (2 * r);
            const uint32_t slot = wbase + (uint32_t)(tb * buf_words + r * slot_words) * 4;
            for (int j = j0; j < C; j += 8) {
                const int mis = (ar + wr0 * g.K) & 3;          // the same for every fourth row
                const float* src = row0 + (wr0 * g.K - mis + 4 * j);
                uint32_t dst = slot + (((wr0 * SR + ar) & ~3) + 4 * j) * 4;
                const uint32_t dstep = 16 * SR;
                if (loose && wraps) {
                    // rows past an end of an axis whose length is no multiple of four: another misalignment
                    for (int t = wr0; t < nrows; t += 4) {
                        const int x = xs + t + (fold ? g.H * wc : 0), dx = wrap_axis(x, X) - x;
                        const int q = t * SR + ((ar + dx * g.K) & 3), m = (ar + (t + dx) * g.K) & 3;
                        if (4 * j < g.ws + m)                  // else the piece starts past the run
                            cp_async16(slot + ((q & ~3) + 4 * j) * 4, row0 + (int64_t)(t + dx) * g.K - m + 4 * j);
                    }
                    continue;
                }
                if (4 * j >= g.ws + mis) continue;
                if (wraps) {
                    const int64_t turn = (int64_t)X * g.K;
                    int x = xs + wr0 + (fold ? g.H * wc : 0);
                    for (int t = wr0; t < nrows; t += 4) {
                        cp_async16(dst, src + (x < 0 ? turn : (x >= X ? -turn : 0)));
                        src += step;
                        dst += dstep;
                        x += 4;
                    }
                } else {
#pragma unroll 4
                    for (int t = wr0; t < nrows; t += 4) {
                        cp_async16(dst, src);
                        src += step;
                        dst += dstep;
                    }
                }
            }
        }
        cp_async_commit();
        return mis4;
    };

    uint64_t acc[NQ][8];
    float asum[NQ];
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        asum[r] = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[r][i] = 0;
    }
    int mis4 = 0, mis4_next = 0;
    if (a.nbuf == 2 && s_begin < s_end) mis4_next = fetch_runs(s_begin, 0);

    CA_PIPE_LOOP({
        const int mask = stage_mask<NQ>(s, pw);
        const uint32_t rowbase = pipe.vec(buf, a) + (lr + a.roff) * RB + slab * 16;
        const int tb = a.nbuf == 2 ? (s - s_begin) & 1 : 0;
        if (a.nbuf == 2) {
            mis4 = mis4_next;
            if (s + 1 < s_end) { mis4_next = fetch_runs(s + 1, tb ^ 1); cp_async_wait<1>(); }
            else cp_async_wait<0>();
        } else {
            mis4 = fetch_runs(s, 0);
            cp_async_wait<0>();
        }
        __syncwarp();
        // shared-space address of this lane's row 0 (transposed: row lrow), per centre column
        uint32_t pr[NQ];
#pragma unroll
        for (int r = 0; r < NQ; ++r)
            pr[r] = wbase + (uint32_t)(tb * buf_words + r * slot_words + lrow * SR + (loose ? 0 : (mis4 >> (2 * r)) & 3)) * 4;
        // coordinate of this lane's pixel on the window axis (folded: column w0 + s is the one that is on); pixels past
        // the image take one whose entries all exist
        const bool here = active && (!kAnyC || !fold || has_pixel(g, h, w0 + s));
        const int n = !here ? 2 * g.p : (fold ? h + g.H * (w0 + s) : h);
        const int rot = TRANS || !here ? 0 : run_rot(n, X, g.p, g.ws);
        auto sweep = [&](auto full_tag, auto loose_tag) {
            constexpr bool FULL = decltype(full_tag)::value, LOOSE = decltype(loose_tag)::value;
#pragma unroll (NQ == 1 ? 4 : 3)
            for (int e = 0; e < g.ws; ++e) {
                uint64_t v[8];
                const uint32_t vb = rowbase + e * RB;
                lds128p(vb, v[0], v[1]);
                lds128p(vb + 16 * NS, v[2], v[3]);
                lds128p(vb + 32 * NS, v[4], v[5]);
                lds128p(vb + 48 * NS, v[6], v[7]);
                // word of the entry after row lrow's start: the same for all centre columns, except for the
                // misalignment of wrapped rows (LOOSE)
                int off = 0, sh = 0;
                if (!TRANS) {
                    off = e + rot;
                    off -= off >= g.ws ? g.ws : 0;
                } else {
                    off = e * SR + transposed_pos(n, e, X, g.p, g.ws);
                    if (LOOSE) {
                        const int x = xs + lrow + e + (fold ? g.H * (w0 + s) : 0);
                        sh = (wrap_axis(x, X) - x) * g.K;
                    }
                }
#pragma unroll
                for (int r = 0; r < NQ; ++r) {
                    if (!FULL && !((mask >> r) & 1)) continue;
                    const float av = lds32(pr[r] + (uint32_t)(off + (LOOSE ? ((mis4 >> (2 * r)) + sh) & 3 : 0)) * 4);
                    asum[r] += av;
                    const uint64_t a2 = dup2(av);
#pragma unroll
                    for (int i = 0; i < 8; ++i) fma_outer(acc[r][i], a2, v[i]);
                }
            }
        };
        if (TRANS && loose) {
            if (mask == (1 << NQ) - 1) sweep(std::true_type{}, std::true_type{});
            else sweep(std::false_type{}, std::true_type{});
        } else {
            if (mask == (1 << NQ) - 1) sweep(std::true_type{}, std::false_type{});
            else sweep(std::false_type{}, std::false_type{});
        }
        __syncwarp();
    })

    apply_finish<CPE, NQ, NCRT>(a, smem_al, part, lt, PT, u, h, w0, active, slab, ca_poison, acc, asum);
}

// =====================================================================
// A (x) V where the rows of A are short: a warp fetches the whole rows of its pixels, which are one contiguous piece of A
// per centre column, into shared memory before the first stage, and the stages only stream V.  (Staged per window
// column, a run of a 7-wide window is 28 bytes: three 16-byte copies on eight lanes, with their address arithmetic and
// two warp barriers for seven window rows.)  K is odd, so the lanes' rows lie in distinct banks.
// Bound: the shared-memory reads, 16 cycles of vectors for NQ columns and one for each value, against 4 cycles of FMAs per column.
// =====================================================================
template <int CPE, int NQ, int NCRT>
__global__ void __launch_bounds__(128, (NQ == 1 ? 6 : 4)) apply_rows_kernel(TileArgs a, const __grid_constant__ CUtensorMap mv,
                                                              const __grid_constant__ CUtensorMap msc) {
    constexpr int NS = NCRT <= 16 ? 1 : NCRT / 16;
    constexpr int RW = 32 / NS;
    constexpr int RB = kSingleFloats * 4 * NS;
    const Geo& g = a.g;
    const int ROWS = a.TH + 2 * (g.p + a.roff);
    const int pw = radius_w(g);
    const int w0 = blockIdx.x * NQ, h0 = blockIdx.y * a.TH, u = blockIdx.z;
    const int NSTAGES = g.wsw + min(NQ - 1, g.W - 1 - w0);          // no stages for centre columns past the image
    CA_PIPE_PROLOGUE(false, kParts)
    const int lane = threadIdx.x & 31, slab = lane % NS, lrow = lane / NS;
    const int lr = (lt >> 5) * RW + lrow, h = h0 + lr, hw0 = h0 + (lt >> 5) * RW;
    const bool active = h < g.H;
    const int slot_words = (RW * g.K + 7) & ~3;                     // up to three words before the first row
    const uint32_t slots = smem_u32(smem_al) + a.extra_off + (lt >> 5) * (NQ * slot_words * 4);
    uint32_t mine[NQ];                                              // this lane's row
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        // rows of this column that hold pixels; the 16-byte pieces at both ends hold at least one word of them
        const int n = w0 + r < g.W ? min(RW, (kAnyC ? min(g.H, g.Np - g.H * (w0 + r)) : g.H) - hw0) * g.K : 0;
        const float* first = a.cs0 + ((int64_t)u * g.Np + hw0 + (int64_t)g.H * (w0 + r)) * g.K;
        const int mis = (int)((uintptr_t)first >> 2) & 3;
        const uint32_t slot = slots + r * slot_words * 4;
        mine[r] = slot + (mis + lrow * g.K) * 4;
        for (int i = 4 * (part * 32 + lane); i < n + mis; i += 128 * a.nsplit) cp_async16(slot + i * 4, first - mis + i);
    }
    cp_async_commit();
    const bool here = active && has_pixel(g, h, w0);
    const int rot = here ? run_rot(axis_coord(g, h, w0), axis_len(g), g.p, g.ws) : 0;     // 2-D: the same in every column

    uint64_t acc[NQ][8];
    float asum[NQ];
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        asum[r] = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[r][i] = 0;
    }
    cp_async_wait<0>();
    if (a.nsplit > 1) __syncthreads();                              // the parts fetched each other's pieces
    else __syncwarp();

    CA_PIPE_LOOP({
        const int mask = stage_mask<NQ>(s, pw);
        const uint32_t rowbase = pipe.vec(buf, a) + (lr + a.roff) * RB + slab * 16;
        uint32_t run[NQ];
        _Pragma("unroll")
        for (int r = 0; r < NQ; ++r)
            run[r] = mine[r] + (((mask >> r) & 1) && w0 + r < g.W ? axis_pos(s - pw - r, w0 + r, g.W, pw, g.wsw) * g.ws * 4 : 0);
        auto sweep = [&](auto full_tag) {
            constexpr bool FULL = decltype(full_tag)::value;
            int pos = rot * 4;
            uint32_t vb = rowbase;
            _Pragma("unroll 2")
            for (int e = 0; e < g.ws; ++e, vb += RB) {
                uint64_t v[8];
                lds128p(vb, v[0], v[1]);
                lds128p(vb + 16 * NS, v[2], v[3]);
                lds128p(vb + 32 * NS, v[4], v[5]);
                lds128p(vb + 48 * NS, v[6], v[7]);
                _Pragma("unroll")
                for (int r = 0; r < NQ; ++r) {
                    if (!FULL && !((mask >> r) & 1)) continue;
                    const float av = lds32(run[r] + pos);
                    asum[r] += av;
                    const uint64_t a2 = dup2(av);
                    _Pragma("unroll")
                    for (int i = 0; i < 8; ++i) fma_outer(acc[r][i], a2, v[i]);
                }
                pos = pos + 4 == g.ws * 4 ? 0 : pos + 4;
            }
        };
        if (mask == (1 << NQ) - 1) sweep(std::true_type{});
        else sweep(std::false_type{});
    })
    apply_finish<CPE, NQ, NCRT>(a, smem_al, part, lt, PT, u, h, w0, active, slab, ca_poison, acc, asum);
}
}  // namespace

// Whole rows (apply_rows_kernel) with one or two columns per thread, and runs (apply_tiled_kernel) plain and transposed with two
// (folded signals: one).  Four columns measured no faster with either.  Rows against runs, plain: 320 x 320, 8 units of 64
// channels, ws 7: 296 and 339 us; 400 x 380, 2 of 16, ws 7: 44 and 50; 320 x 240, 4 of 32, ws 5: 46 and 55; 256 x 256, 4 of 16,
// ws 9 (10.4 KB of rows per warp and column): 53 and 55; 100 x 64, 6 of 64, ws 11: 40 and 43; 75 x 53, 8 of 16, ws 11 (15.5
// KB): 18.1 and 17.5; 128 x 96, 4 of 64, ws 15 (7.2 KB): 77 and 73.
// Runs, before and after (one thread per pixel row, 4-byte copies with offset tables -> this kernel -> cut by predicted time), per
// launch, 128 x 96 x 64 x 2, ws 15, 4 heads: plain 124 -> 58 -> 48 us, transposed 142 -> 72 -> 65 us (88 MB of values: 14 us at
// the HBM peak).
static const SweepCost kApplyRowsCost[3][2] = {{{1, 24, 27, 58, 624, 1271}, {2, 16, 44, 68, 868, 2928}},
                                               {{1, 24, 2, 59, 680, 2064}, {2, 16, 35, 65, 759, 3886}},
                                               {{1, 24, 19, 62, 226, 1903}, {2, 16, 41, 68, 422, 3551}}};
static const SweepCost kApplyRunsCost[2][3] = {{{2, 16, 14, 71, 1454, 3579}, {2, 16, 0, 57, 1458, 4291}, {2, 16, 0, 57, 1254, 4071}},
                                               {{2, 16, 27, 80, 2811, 2390}, {2, 16, 0, 96, 2223, 2869}, {2, 16, 7, 57, 2668, 3735}}};

template <>
int run_apply<kAnyC>(const Geo& g, const Padded& P, const float* nz, const float* packed, const float* centre, float* out,
                     float alpha, int transposed, cudaStream_t st) {
    Launch L{};
    const int ns = slabs_of(g), slot = ns == 1 ? 0 : ns / 2;
    int rc = CA_OK;
    const bool fold = g.wsw == 1;
    const int row_bytes = ((32 / ns * g.K + 7) & ~3) * (int)sizeof(float);
    if (!transposed && g.K <= 121 && row_bytes <= 10600) {
        const TileShape t = choose_tile(g, P, ns, kApplyRowsCost[slot], fold ? 1 : 2, kParts, false, true, row_bytes, 2);
        if ((rc = prepare(g, P, t, 17 * t.nq, packed, nullptr, &L, ns, true, 2, (size_t)t.warps * t.nq * row_bytes))) return rc;
        L.a.scale = alpha; L.a.c0 = centre; L.a.cs0 = nz; L.a.o0 = out;
#define CA_APPLY_ROWS(NSV)                                                                       \
    do {                                                                                         \
        if (g.cpe == 1) {                                                                        \
            if (t.nq == 1) CA_LAUNCH_TILED((apply_rows_kernel<1, 1, NSV>), L, st);               \
            else CA_LAUNCH_TILED((apply_rows_kernel<1, 2, NSV>), L, st);                         \
        } else {                                                                                 \
            if (t.nq == 1) CA_LAUNCH_TILED((apply_rows_kernel<2, 1, NSV>), L, st);               \
            else CA_LAUNCH_TILED((apply_rows_kernel<2, 2, NSV>), L, st);                         \
        }                                                                                        \
    } while (0)
        if (ns == 1) CA_APPLY_ROWS(16);
        else if (ns == 2) CA_APPLY_ROWS(32);
        else CA_APPLY_ROWS(64);
#undef CA_APPLY_ROWS
        CA_CHECK_LAUNCH("tiled apply kernel");
        return CA_OK;
    }
    const bool loose = transposed && ((fold ? g.Np : g.H) & 3);
    const int rows = 32 / ns + (transposed ? g.ws - 1 : 0);
    const int nq = fold ? 1 : 2;
    const int area = run_area(g, rows, nq, loose) * (int)sizeof(float);
    // run buffers of a warp: two when as many CTAs still fit on an SM as the registers allow, else one
    auto setup = [&](int nbuf, TileShape t) {
        L = Launch{};
        rc = prepare(g, P, t, 17 * nq, packed, nullptr, &L, ns, true, 2);
        L.a.nbuf = nbuf;
        const size_t need = (size_t)t.nsplit * 2 * L.a.stage_bytes + (size_t)t.warps * t.nsplit * nbuf * area + 1024;
        if (!rc && need > L.smem) L.smem = need;
        return rc;
    };
    const int one = tile_stage_bytes(32 / ns + 2 * P.pp, kSingleFloats * 4 * ns, false, true);      // a stage of one warp
    const bool two = 16 * (2 * one + 2 * area + 2048) <= 227 * 1024;
    const TileShape t = fold ? operator_tile(g, ns, 1, 1, 4)
                             : choose_tile(g, P, ns, &kApplyRunsCost[transposed ? 1 : 0][slot], 1, kParts, false, true, 0, 2, (two ? 2 : 1) * area,
                                          transposed ? 1.f : 0.9f);     // 128 x 96, 8 of 16, ws 15: 52 us, four warps 61
    const size_t most = (fold ? 24 : 16) / (t.warps * t.nsplit);                              // CTAs per SM that the registers allow
    if (setup(2, t)) return rc;
    if (most * (L.smem + 1024) > 227 * 1024 && setup(1, t)) return rc;
    // wide windows, whose runs fill the shared memory, run fewer warps per CTA
    for (int split = 2; L.smem > 200 * 1024 && split >= 1; --split)
        if (setup(1, operator_tile(g, ns, nq, fold ? 1 : split, 1))) return rc;
    if (L.smem > 200 * 1024) {
        set_error("tiled apply: window %d with %d channels per unit needs %zu bytes of shared memory", g.ws, g.cr, L.smem);
        return CA_ERR_UNSUPPORTED;
    }
    L.a.scale = alpha; L.a.c0 = centre; L.a.cs0 = nz; L.a.o0 = out;
#define CA_APPLY(NQV, NSV)                                                                     \
    do {                                                                                  \
        if (g.cpe == 1) {                                                                 \
            if (transposed) CA_LAUNCH_TILED((apply_tiled_kernel<1, true, NQV, NSV>), L, st);   \
            else CA_LAUNCH_TILED((apply_tiled_kernel<1, false, NQV, NSV>), L, st);             \
        } else {                                                                          \
            if (transposed) CA_LAUNCH_TILED((apply_tiled_kernel<2, true, NQV, NSV>), L, st);   \
            else CA_LAUNCH_TILED((apply_tiled_kernel<2, false, NQV, NSV>), L, st);             \
        }                                                                                 \
    } while (0)
#define CA_APPLY_NQ(NSV)                                                                  \
    do {                                                                                  \
        if (nq == 1) CA_APPLY(1, NSV);                                                    \
        else CA_APPLY(2, NSV);                                                            \
    } while (0)
    if (ns == 1) CA_APPLY_NQ(16);
    else if (ns == 2) CA_APPLY_NQ(32);
    else CA_APPLY_NQ(64);
#undef CA_APPLY_NQ
#undef CA_APPLY
    CA_CHECK_LAUNCH("tiled apply kernel");
    return CA_OK;
}

}  // namespace ca
