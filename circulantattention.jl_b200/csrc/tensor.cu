// 2-D softmax attention on the tensor cores (tcgen05), Float32-exact, for units of at most 16 real channels.
//
// Why.  The FMA-pipe kernels of tiled.cu are at their wall: a scalar FMA with three distinct register operands runs at
// 50-60 TFLOP/s, every shared-memory word has to feed four FMAs, and the sweeps sit at 35-41 TFLOP/s.  Here the two
// contractions of a window run as bf16 MMAs on an exact split of every Float32 operand,
//     x = hi + mid + lo   (8 + 8 + 8 significand bits),
// with the six products hi*hi, hi*mid, mid*hi, hi*lo, mid*mid, lo*hi accumulated in FP32; the three that are left out
// are below 2^-24 of the result, which is less than the rounding of one FP32 FMA.  bfloat16 storage needs one piece.
//
// Tile.  A CTA owns 8 rows x 16 columns of centre pixels (128 = the M of an MMA); warp w owns columns 4w..4w+3, lane
// (h, w) = (lane & 7, lane >> 3), and the lane is the tensor-memory lane of its pixel.  The other side of the window is
// streamed in chunks of N keys: 2 or 4 image columns of RP rows (RP = 8 + 2p rounded up to 8).  Per chunk:
//     S  = A0 x B0^T                         six MMAs, K = 16 channels
//     dP = A1 x B1^T                         (the sweeps that need it)
//     W  = P or dS, in registers             window mask, 2^x, products; split in three, written back over S
//     O  = W x (B1 or B0)                    three MMAs per 16 keys: W_hi x [hi|mid|lo], W_mid x [hi|mid], W_lo x hi,
//                                            the pieces side by side along N
// and O is added to FP32 registers after every chunk, so that the tensor core's truncating accumulation only ever spans
// one chunk.  Four sweeps share this kernel: forward, dv (both apply B1), dq, dk (both need dP and apply B0).
//
// Bound: the tensor pipe; an MMA with its A operand (128 x 16) in tensor memory takes at least 32 cycles, so the
// O products run at N = 48, 32 and 16 for the price of 64.  Two CTAs per SM overlap one's MMAs with the other's
// arithmetic.  Dead ends: A in shared memory (an MMA then takes 77 cycles at N = 80); mma.sync (933 MAC per cycle and SM,
// a quarter of tcgen05).  Measured times stand at tc_route().
#include "tile_common.cuh"
#include "tc05.cuh"

namespace ca {
namespace {

constexpr int kTileH = 8, kTileW = 16;
constexpr int kTmemCols = 256;                 // per CTA; two CTAs per SM
constexpr int kColA0 = 0, kColA1 = 24, kColS = 48, kColO = 208;
constexpr int kChunkStages = 3;
constexpr float kScoreHeadroom = 12.f;         // see kHeadroom in tiled.cu

enum { SWEEP_FWD = 0, SWEEP_DV = 1, SWEEP_DQ = 2, SWEEP_DK = 3 };

struct TcArgs {
    Geo g;
    float scale;
    int Hp;                     // packed rows per column
    const uint4* packed;        // [unit][column][plane][Hp] pieces of 8 bf16: plane = ((tensor * splits) + split) * 2 + half
    const float* scal;          // [unit][column][2][Hp]: terms of the streamed pixel (see ScalarPlanes), nullable
    const float* a0;            // centre tensors, reference layout
    const float* a1;
    const float* row0;          // centre scalars: statistics, D (dq sweep)
    const float* row1;
    float* out;
    float* ostats;
    int* status;
    int* timeouts;
    uint32_t wait_tries;
};

// Rows of a streamed column that a tile needs, rounded to the 8 of a core matrix; columns per chunk; keys per chunk.
constexpr int kMaxRadius = 16;
__host__ __device__ constexpr int rows_of(int p) { return (kTileH + 2 * p + 7) & ~7; }
__host__ __device__ constexpr int chunk_cols(int RP) { return RP == 16 ? 4 : 2; }

// Orders the uses of registers that a tcgen05.ld fills after the wait for it: the compiler sees no other dependency.
template <int n>
__device__ __forceinline__ void settle(uint32_t* v) {
#pragma unroll
    for (int i = 0; i < n; ++i) asm volatile("" : "+r"(v[i]));
}

// 16 channels of the centre pixel `pix` (zero past the unit's), times `mul`.
template <int CPE, bool BF>
__device__ __forceinline__ void load_pixel(const float* src, const Geo& g, int u, int pix, bool ok, float mul, float (&v)[16]) {
    int64_t o = goff<CPE>(u, g.cr, 0, g.Np, ok ? pix : 0);
#pragma unroll
    for (int e = 0; e < 16; e += CPE) {
        if (CPE == 1) {
            v[e] = ld_real<BF>(src, o);
        } else {
            const float2 z = __ldg(reinterpret_cast<const float2*>(src + o));
            v[e] = z.x;
            v[e + CPE - 1] = z.y;
        }
        o += e + CPE < g.cr ? (int64_t)CPE * g.Np : 0;
    }
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = ok && e < g.cr ? v[e] * mul : 0.f;
}

// Writes a pixel vector as the A operand: 8 columns per split.
template <int NSPL>
__device__ __forceinline__ void store_operand(uint32_t t, const float (&v)[16]) {
    uint32_t piece[3][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (NSPL == 1) piece[0][i] = to_bf16x2(v[2 * i], v[2 * i + 1]);
        else split3(pair(v[2 * i], v[2 * i + 1]), piece[0][i], piece[1][i], piece[2][i]);
    }
#pragma unroll
    for (int s = 0; s < NSPL; ++s) tmem_st8(t + 8 * s, piece[s]);
}

template <int SWEEP, int RP, int CPE, bool DIST, bool BF>
__global__ void __launch_bounds__(128, 2) tc_sweep_kernel(const __grid_constant__ TcArgs a) {
    constexpr int NC = chunk_cols(RP), N = NC * RP, NO = RP / 8;      // image columns, keys per chunk, octets per column
    constexpr int NSPL = BF ? 1 : 3, NPL = 4 * NSPL;                  // bf16 pieces per value, planes per streamed column
    constexpr bool TWO = SWEEP == SWEEP_DQ || SWEEP == SWEEP_DK;      // needs dP
    constexpr bool OWN_STAT = SWEEP == SWEEP_DQ;                      // the row statistic belongs to the centre pixel
    constexpr bool SC0 = DIST || SWEEP == SWEEP_DV || SWEEP == SWEEP_DK, SC1 = SWEEP == SWEEP_DK;   // streamed terms
    constexpr int kPlane = N * 16, kStage = NPL * kPlane + (SC0 ? N * 4 : 0) + (SC1 ? N * 4 : 0);
    constexpr int kStageStride = (kStage + 127) & ~127;
    constexpr int kColX = kColS + N;                                  // dP; W_lo of the sweeps without dP
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[kChunkStages], bar_s, bar_o;
    __shared__ uint32_t s_tmem;
    const Geo& g = a.g;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int w0 = blockIdx.x * kTileW, h0 = blockIdx.y * kTileH, u = blockIdx.z;
    const int CW = kTileW + 2 * g.p, NCH = (CW + NC - 1) / NC;        // streamed columns, chunks
    const uint32_t stages = smem_u32(smem_raw) + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    const unsigned char* stages_g = smem_raw + (stages - smem_u32(smem_raw));

    if (warp == 0) tmem_alloc<kTmemCols>(&s_tmem);
    if (tid == 0) {
        for (int i = 0; i < kChunkStages; ++i) mbar_init(&full[i], 1);
        mbar_init(&bar_s, 1);
        mbar_init(&bar_o, 1);
        mbar_fence_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = s_tmem, tml = tm + ((uint32_t)warp << 21);    // this warp's 32 lanes

    // copies of chunk ch: one bulk copy per (plane, column) and per (scalar plane, column), a lane each
    auto issue = [&](int ch) {
        const int st = ch % kChunkStages;
        if (lane == 0) mbar_arrive_expect_tx(&full[st], (uint32_t)kStage);
        __syncwarp();
        constexpr int kCopies = NPL * NC, kScal = (SC0 ? NC : 0) + (SC1 ? NC : 0);
        for (int i = lane; i < kCopies + kScal; i += 32) {
            const bool sc = i >= kCopies;
            const int k = sc ? i - kCopies : i;
            const int pl = k / NC, c = k - pl * NC;
            const int kc0 = (w0 - g.p + ch * NC + c + g.wk_off) % g.Wk, kc = kc0 < 0 ? kc0 + g.Wk : kc0;
            const int64_t col = (int64_t)u * g.Wk + kc;
            const uint32_t base = stages + st * kStageStride;
            if (!sc) bulk_load(base + pl * kPlane + c * (RP * 16), a.packed + (col * NPL + pl) * a.Hp + h0, RP * 16, &full[st]);
            else bulk_load(base + NPL * kPlane + pl * (N * 4) + c * (RP * 4), a.scal + (col * 2 + pl) * a.Hp + h0, RP * 4, &full[st]);
        }
    };
    if (warp == 0)
        for (int ch = 0; ch < kChunkStages && ch < NCH; ++ch) issue(ch);

    // centre pixel of this thread
    const int lh = lane & 7, lw = lane >> 3;
    const int h = h0 + lh, w = w0 + 4 * warp + lw;
    const bool ok = h < g.H && w < g.W;
    const int pix = h + g.H * w;
    const float sl2 = a.scale * kLog2e;
    float cst = 0.f;                                                  // Distance: -1/2 |centre|^2, log2 domain
    {
        float v[16];
        // Float32: the scale goes into the operand; bfloat16 operands stay exact and the scores are scaled
        load_pixel<CPE, BF>(a.a0, g, u, pix, ok, 1.f, v);
        if (DIST) {
            float n = 0.f;
#pragma unroll
            for (int e = 0; e < 16; ++e) n = fmaf(v[e], v[e], n);
            cst = -0.5f * sl2 * n;
        }
        if (!BF) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] *= sl2;
        }
        store_operand<NSPL>(tml + kColA0, v);
        if (TWO) {
            load_pixel<CPE, BF>(a.a1, g, u, pix, ok, 1.f, v);
            store_operand<NSPL>(tml + kColA1, v);
        }
    }
    tmem_wait_st();

    // window mask of this lane's rows: row j of the first octet is in the window from j = lh on, row j of octet o up to
    // 8 o + j = lh + 2p, which cuts the last two octets only
    uint64_t m_lo[4], m_up[2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m_lo[i] = pair(2 * i >= lh ? 0.f : -INFINITY, 2 * i + 1 >= lh ? 0.f : -INFINITY);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int t = 8 * (NO - 2 + q) + 2 * i - lh;
            m_up[q][i] = pair(t <= 2 * g.p ? 0.f : -INFINITY, t + 1 <= 2 * g.p ? 0.f : -INFINITY);
        }
    }
    const uint64_t smul = pair(BF ? sl2 : 1.f, BF ? sl2 : 1.f);
    float nref = 0.f, l = 0.f;                                        // forward: -reference, sum of the weights
    uint64_t nD = 0;
    bool fresh = true;                                                // forward: no key seen yet
    if (OWN_STAT) {
        const int64_t so = (int64_t)u * g.Np + (ok ? pix : 0);
        nref = -__ldg(a.row0 + so) * kLog2e;
        const float d = -__ldg(a.row1 + so);
        nD = pair(d, d);
    }
    uint64_t acc[8], sumw = 0;                                        // O; Distance: sum of dS
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0;

    bool err = false, failed = false;                                 // this thread's waits; the CTA's
    int ch = 0;
    for (; ch < NCH; ++ch) {
        const int st = ch % kChunkStages;
        const uint32_t sb = stages + st * kStageStride;
        if (warp == 0) {
            err |= !mbar_wait(&full[st], (uint32_t)((ch / kChunkStages) & 1), a.wait_tries);
            tc_fence_after();
            if (elect_one()) {
                // smallest products first: the truncation of the accumulation then acts on small numbers
                constexpr uint32_t shape = mma_shape(N, false);
#pragma unroll
                for (int t = 0; t < (TWO ? 2 : 1); ++t) {
                    bool accumulate = false;
#pragma unroll
                    for (int order = 2 * NSPL - 2; order >= 0; --order)
#pragma unroll
                        for (int i = 0; i < NSPL; ++i) {
                            const int j = order - i;
                            if (order > NSPL - 1 || j < 0 || j >= NSPL) continue;
                            mma_ts(tm + (t ? kColX : kColS), tm + (t ? kColA1 : kColA0) + 8 * i,
                                   smem_operand(sb + (t * NSPL + j) * 2 * kPlane, kPlane, 128), shape, accumulate);
                            accumulate = true;
                        }
                }
                tc_commit(&bar_s);
            }
        }
        if (SC0) err |= !mbar_wait(&full[st], (uint32_t)((ch / kChunkStages) & 1), a.wait_tries);
        err |= !mbar_wait(&bar_s, (uint32_t)(ch & 1), a.wait_tries);
        tc_fence_after();

        const float* sc0 = reinterpret_cast<const float*>(stages_g + st * kStageStride + NPL * kPlane);
        const float* sc1 = sc0 + N;
        // relative scores of one octet: s * smul + base (+ streamed term) (+ window mask)
        auto rel = [&](const uint32_t* s, int o, int c, uint64_t base, uint64_t (&x)[4]) {
            uint64_t t0[4];
            if (SC0) {
                const ulonglong2 z0 = *reinterpret_cast<const ulonglong2*>(sc0 + c * RP + 8 * o);
                const ulonglong2 z1 = *reinterpret_cast<const ulonglong2*>(sc0 + c * RP + 8 * o + 4);
                t0[0] = z0.x; t0[1] = z0.y; t0[2] = z1.x; t0[3] = z1.y;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint64_t v = pair(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1]));
                x[i] = BF ? fma_pair(v, smul, base) : add_pair(v, base);
                if (SC0) x[i] = add_pair(x[i], t0[i]);
                if (o == 0) x[i] = add_pair(x[i], m_lo[i]);
                if (o >= NO - 2) x[i] = add_pair(x[i], m_up[o - (NO - 2)][i]);
            }
        };
        // streamed columns of this chunk: needed by this warp (uniform), inside this lane's window
        bool need[NC];
        float cadd[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int d = ch * NC + c - 4 * warp;
            need[c] = d >= 0 && d <= 2 * g.p + 3;
            cadd[c] = d - lw >= 0 && d - lw <= 2 * g.p ? 0.f : -INFINITY;
        }
        bool any = false;
#pragma unroll
        for (int c = 0; c < NC; ++c) any = any || need[c];

        auto put = [&](int gidx, const uint32_t (&hi)[8], const uint32_t (&mid)[8], const uint32_t (&lo)[8]) {
            tmem_st8(tml + kColS + 16 * gidx, hi);
            tmem_st8(tml + kColS + 16 * gidx + 8, mid);
            tmem_st8(tml + kColX + (TWO ? 16 : 8) * gidx, lo);
        };
        if (!any) {
            const uint32_t z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
            for (int gi = 0; gi < N / 16; ++gi) put(gi, z, z, z);
        } else if (!TWO) {
            uint32_t s[N];
#pragma unroll
            for (int k = 0; k < N / 8; ++k)
                if (need[k / NO]) tmem_ld8(tml + kColS + 8 * k, s + 8 * k);
            tmem_wait_ld();
            settle<N>(s);
            uint64_t x[N / 8][4];
            uint32_t neg = 0x80000000u;
#pragma unroll
            for (int k = 0; k < N / 8; ++k) {
                const int c = k / NO, o = k % NO;
                const float b = (SWEEP == SWEEP_FWD ? nref : 0.f) + cst + cadd[c];
                if (need[c]) {
                    rel(s + 8 * k, o, c, pair(b, b), x[k]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) x[k][i] = pair(-INFINITY, -INFINITY);
                }
                if (SWEEP == SWEEP_FWD) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = unpair(x[k][i]);
                        neg &= __float_as_uint(f.x) & __float_as_uint(f.y);
                    }
                }
            }
            if (SWEEP == SWEEP_FWD) {
                // the reference moves up to the largest relative score + headroom when one is not negative (and for the
                // first keys of a pixel), as in the FMA-pipe forward
                if (__any_sync(0xffffffffu, neg == 0u || fresh)) {
                    float cm = -INFINITY;
#pragma unroll
                    for (int k = 0; k < N / 8; ++k)
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float2 f = unpair(x[k][i]);
                            cm = fmaxf(cm, fmaxf(f.x, f.y));
                        }
                    if (cm >= 0.f || (fresh && cm > -INFINITY)) {
                        cm += kScoreHeadroom;
                        const float corr = fresh ? 0.f : fast_exp2(-cm);
                        fresh = false;
                        nref -= cm;
                        l *= corr;
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[i] = mul_pair(acc[i], pair(corr, corr));
#pragma unroll
                        for (int k = 0; k < N / 8; ++k)
#pragma unroll
                            for (int i = 0; i < 4; ++i) x[k][i] = add_pair(x[k][i], pair(-cm, -cm));
                    }
                }
            }
            uint64_t lsum = 0;
#pragma unroll
            for (int gi = 0; gi < N / 16; ++gi) {
                uint32_t hi[8], mid[8], lo[8];
#pragma unroll
                for (int q = 0; q < 2; ++q)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = unpair(x[2 * gi + q][i]);
                        const uint64_t P = pair(fast_exp2(f.x), fast_exp2(f.y));
                        if (SWEEP == SWEEP_FWD) lsum = add_pair(lsum, P);
                        split3(P, hi[4 * q + i], mid[4 * q + i], lo[4 * q + i]);
                    }
                put(gi, hi, mid, lo);
            }
            if (SWEEP == SWEEP_FWD) {
                const float2 f = unpair(lsum);
                l += f.x + f.y;
            }
        } else {
            // 16 keys at a time: the next group's scores are on their way while this one is computed
            uint32_t s[2][16], d[2][16];
            auto fetch = [&](int gi, int b) {
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    if (need[(2 * gi + q) / NO]) {
                        tmem_ld8(tml + kColS + 16 * gi + 8 * q, s[b] + 8 * q);
                        tmem_ld8(tml + kColX + 16 * gi + 8 * q, d[b] + 8 * q);
                    }
            };
            fetch(0, 0);
#pragma unroll
            for (int gi = 0; gi < N / 16; ++gi) {
                tmem_wait_ld();
                settle<16>(s[gi & 1]);
                settle<16>(d[gi & 1]);
                if (gi + 1 < N / 16) fetch(gi + 1, (gi + 1) & 1);
                uint32_t hi[8], mid[8], lo[8];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int k = 2 * gi + q, c = k / NO, o = k % NO;
                    if (!need[c]) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) hi[4 * q + i] = mid[4 * q + i] = lo[4 * q + i] = 0;
                        continue;
                    }
                    uint64_t x[4], t1[4];
                    const float b = (OWN_STAT ? nref : 0.f) + cst + cadd[c];
                    rel(s[gi & 1] + 8 * q, o, c, pair(b, b), x);
                    if (SC1) {
                        const ulonglong2 z0 = *reinterpret_cast<const ulonglong2*>(sc1 + c * RP + 8 * o);
                        const ulonglong2 z1 = *reinterpret_cast<const ulonglong2*>(sc1 + c * RP + 8 * o + 4);
                        t1[0] = z0.x; t1[1] = z0.y; t1[2] = z1.x; t1[3] = z1.y;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = unpair(x[i]);
                        const uint64_t P = pair(fast_exp2(f.x), fast_exp2(f.y));
                        const uint64_t dp = pair(__uint_as_float(d[gi & 1][8 * q + 2 * i]), __uint_as_float(d[gi & 1][8 * q + 2 * i + 1]));
                        const uint64_t dS = mul_pair(P, add_pair(dp, SC1 ? t1[i] : nD));
                        if (DIST) sumw = add_pair(sumw, dS);
                        split3(dS, hi[4 * q + i], mid[4 * q + i], lo[4 * q + i]);
                    }
                }
                put(gi, hi, mid, lo);
            }
        }
        tmem_wait_st();
        tc_fence_before();
        failed = __syncthreads_or(err);
        if (failed) break;
        if (warp == 0) {
            tc_fence_after();
            if (elect_one()) {
                const uint32_t vb = sb + (TWO ? 0 : NSPL * 2 * kPlane);          // the operand that is summed: B0 or B1
#pragma unroll
                for (int gi = 0; gi < N / 16; ++gi) {
                    const uint64_t b = smem_operand(vb + gi * 256, 128, kPlane);  // 16 keys x channels, MN-major
                    mma_ts(tm + kColO, tm + kColS + 16 * gi, b, mma_shape(16 * NSPL, true), gi > 0);
                    mma_ts(tm + kColO, tm + kColS + 16 * gi + 8, b, mma_shape(NSPL > 1 ? 32 : 16, true), true);
                    mma_ts(tm + kColO, tm + kColX + (TWO ? 16 : 8) * gi, b, mma_shape(16, true), true);
                }
                tc_commit(&bar_o);
            }
        }
        err |= !mbar_wait(&bar_o, (uint32_t)(ch & 1), a.wait_tries);
        tc_fence_after();
        if (warp == 0 && ch + kChunkStages < NCH) issue(ch + kChunkStages);     // the MMAs have read this stage
        {
            uint32_t o[16 * NSPL];
#pragma unroll
            for (int i = 0; i < 2 * NSPL; ++i) tmem_ld8(tml + kColO + 8 * i, o + 8 * i);
            tmem_wait_ld();
            settle<16 * NSPL>(o);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                uint64_t t = pair(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1]));
                if (NSPL > 1)
                    t = add_pair(t, add_pair(pair(__uint_as_float(o[16 + 2 * i]), __uint_as_float(o[17 + 2 * i])),
                                             pair(__uint_as_float(o[32 + 2 * i]), __uint_as_float(o[33 + 2 * i]))));
                acc[i] = add_pair(acc[i], t);
            }
        }
    }
    tc_fence_before();
    failed |= (bool)__syncthreads_or(err);
    tc_fence_after();
    float poison = 0.f;
    if (failed) {
        // a wait ran out: give what is in flight a bounded chance to end, report, and store NaN
        if (tid == 0) {
            for (int i = 0; i < kChunkStages; ++i) {
                mbar_wait(&full[i], 0, 1u << 12);
                mbar_wait(&full[i], 1, 1u << 12);
            }
            mbar_wait(&bar_s, (uint32_t)(ch & 1), 1u << 12);
            mbar_wait(&bar_o, (uint32_t)(ch & 1), 1u << 12);
            atomicAdd(a.timeouts, 1);
            if (a.status) atomicOr(a.status, 1);
        }
        poison = __int_as_float(0x7fc00000);
        __syncthreads();
    }
    if (warp == 0) tmem_free<kTmemCols>(tm);
    if (!ok) return;

    const float mul = SWEEP == SWEEP_FWD ? 1.f / l : (TWO ? a.scale : 1.f);
    float r[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float2 f = unpair(acc[i]);
        r[2 * i] = f.x * mul + poison;
        r[2 * i + 1] = f.y * mul + poison;
    }
    if (TWO && DIST) {
        // d centre = scale * (sum dS other - sum dS * centre)
        float v[16];
        load_pixel<CPE, BF>(a.a0, g, u, pix, true, 1.f, v);
        const float2 f = unpair(sumw);
        const float ss = (f.x + f.y) * a.scale;
#pragma unroll
        for (int e = 0; e < 16; ++e) r[e] = fmaf(-ss, v[e], r[e]);
    }
    int64_t o = goff<CPE>(u, g.cr, 0, g.Np, pix);
#pragma unroll
    for (int e = 0; e < 16; e += CPE) {
        if (e >= g.cr) break;
        if (CPE == 1) st_real<BF>(a.out, o, r[e]);
        else *reinterpret_cast<float2*>(a.out + o) = make_float2(r[e], r[e + CPE - 1]);
        o += (int64_t)CPE * g.Np;
    }
    if (SWEEP == SWEEP_FWD && a.ostats) a.ostats[(int64_t)u * g.Np + pix] = (log2f(l) - (nref)) * kLn2 + poison;
}

// =====================================================================
// Pack: two tensors in the reference layout -> pieces of 8 bf16 per (unit, column, plane, row'), the circular halo along
// h unrolled (row' = h + p; rows past H + 2p are zero), and the terms of the streamed pixels.  A thread owns a row:
// coalesced planar loads, consecutive lanes write consecutive 16-byte pieces.  Bound: HBM (reads 4, writes 6 bytes per
// Float32 value; the FMA-pipe pack writes 4.5).
// =====================================================================
struct TcPackArgs {
    Geo g;
    int Hp, mode;               // mode: 0 pieces only; 1: T0 = -1/2 |src0|^2 (Distance keys); 2: T0 = -L (Distance:
                                // -1/2 |src0|^2 more), T1 = -D; L and |.|^2 in the log2 domain
    int dist;
    float sl2;
    const float* src[2];
    uint4* packed;
    float* scal;
    const float* stats;
    const float* y;             // D = src1 . y
    float* Dout;
};

template <int CPE, bool BF>
__global__ void __launch_bounds__(128) tc_pack_kernel(TcPackArgs a) {
    constexpr int NSPL = BF ? 1 : 3, NPL = 4 * NSPL;
    const Geo& g = a.g;
    const int rr = blockIdx.x * 128 + threadIdx.x, w = blockIdx.y;
    const int slots = 2 + (a.mode ? 1 : 0);
    const int u = blockIdx.z / slots, slot = blockIdx.z % slots;
    if (rr >= a.Hp) return;
    const bool real_row = rr < g.H + 2 * g.p;
    const int pix = real_row ? wrap_axis(rr - g.p, g.H) + g.H * w : 0;
    const int64_t col = (int64_t)u * g.Wk + w;
    if (slot < 2) {
        float v[16];
        load_pixel<CPE, BF>(a.src[slot], g, u, pix, real_row, 1.f, v);
        uint32_t piece[3][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (NSPL == 1) piece[0][i] = to_bf16x2(v[2 * i], v[2 * i + 1]);
            else split3(pair(v[2 * i], v[2 * i + 1]), piece[0][i], piece[1][i], piece[2][i]);
        }
#pragma unroll
        for (int s = 0; s < NSPL; ++s)
#pragma unroll
            for (int half = 0; half < 2; ++half)
                a.packed[(col * NPL + (slot * NSPL + s) * 2 + half) * a.Hp + rr] =
                    make_uint4(piece[s][4 * half], piece[s][4 * half + 1], piece[s][4 * half + 2], piece[s][4 * half + 3]);
        return;
    }
    float t0 = 0.f, t1 = 0.f;
    if (real_row) {
        float v[16], z[16];
        if (a.dist) {
            load_pixel<CPE, BF>(a.src[0], g, u, pix, true, 1.f, v);
            float n = 0.f;
#pragma unroll
            for (int e = 0; e < 16; ++e) n = fmaf(v[e], v[e], n);
            t0 = -0.5f * a.sl2 * n;
        }
        if (a.mode == 2) {
            const int64_t so = (int64_t)u * g.Npk + pix;
            t0 -= __ldg(a.stats + so) * kLog2e;
            load_pixel<CPE, BF>(a.src[1], g, u, pix, true, 1.f, v);
            load_pixel<CPE, BF>(a.y, g, u, pix, true, 1.f, z);
            float d = 0.f;
#pragma unroll
            for (int e = 0; e < 16; ++e) d = fmaf(v[e], z[e], d);
            t1 = -d;
            if (rr >= g.p && rr < g.p + g.H) a.Dout[so] = d;
        }
    }
    a.scal[(col * 2) * a.Hp + rr] = t0;
    a.scal[(col * 2 + 1) * a.Hp + rr] = t1;
}

// ---------------------------------------------------------------- host side
struct TcSizes {
    int RP, Hp;
    size_t packed, scal;        // bytes of one packed pair of tensors and of its scalar planes
};
TcSizes sizes_of(const Geo& g) {
    TcSizes z;
    z.RP = rows_of(g.p);
    const int tiles = (g.H + kTileH - 1) / kTileH;
    z.Hp = std::max((tiles - 1) * kTileH + z.RP, g.H + 2 * g.p);
    z.Hp = (z.Hp + 7) & ~7;
    const size_t cols = (size_t)g.units * g.Wk;
    z.packed = cols * (g.bf16 ? 4 : 12) * z.Hp * 16;
    z.scal = (cols * 2 * z.Hp * 4 + 255) & ~(size_t)255;
    z.packed = (z.packed + 255) & ~(size_t)255;
    return z;
}

int pack(const TcPackArgs& a, cudaStream_t st) {
    dim3 grid((a.Hp + 127) / 128, a.g.Wk, a.g.units * (2 + (a.mode ? 1 : 0)));
    if (grid.y > 65535u || grid.z > 65535u) return CA_ERR_UNSUPPORTED;
    if (a.g.cpe == 2) tc_pack_kernel<2, false><<<grid, 128, 0, st>>>(a);
    else if (a.g.bf16) tc_pack_kernel<1, true><<<grid, 128, 0, st>>>(a);
    else tc_pack_kernel<1, false><<<grid, 128, 0, st>>>(a);
    CA_CHECK_LAUNCH("tensor-core pack kernel");
    return CA_OK;
}

template <int SWEEP, int RP, int CPE, bool DIST, bool BF>
int launch_one(const TcArgs& a, cudaStream_t st) {
    constexpr int N = chunk_cols(RP) * RP, NPL = BF ? 4 : 12;
    const size_t stage = ((NPL * N * 16 + 2 * N * 4) + 127) & ~127;
    // at most two CTAs per SM, for their tensor-memory columns
    const size_t smem = std::max<size_t>(kChunkStages * stage + 128, 80 * 1024);
    auto kernel = tc_sweep_kernel<SWEEP, RP, CPE, DIST, BF>;
    if (int rc = set_smem(kernel, smem)) return rc;
    dim3 grid((a.g.W + kTileW - 1) / kTileW, (a.g.H + kTileH - 1) / kTileH, a.g.units);
    kernel<<<grid, 128, smem, st>>>(a);
    count_tiled_launch();
    CA_CHECK_LAUNCH("tensor-core sweep");
    return CA_OK;
}

template <int SWEEP, int CPE, bool DIST, bool BF>
int launch_rows(const TcArgs& a, int RP, cudaStream_t st) {
    switch (RP) {
        case 16: return launch_one<SWEEP, 16, CPE, DIST, BF>(a, st);
        case 24: return launch_one<SWEEP, 24, CPE, DIST, BF>(a, st);
        case 32: return launch_one<SWEEP, 32, CPE, DIST, BF>(a, st);
        default: return launch_one<SWEEP, 40, CPE, DIST, BF>(a, st);
    }
}

template <int SWEEP>
int sweep(TcArgs a, const TcSizes& z, int dist, cudaStream_t st) {
    a.Hp = z.Hp;
    a.status = status_word();
    if (!(a.timeouts = stage_timeout_counter())) return cuda_fail(cudaGetLastError(), "cudaGetSymbolAddress(stage timeouts)");
    a.wait_tries = 1u << 14;
    if (a.g.cpe == 2) return dist ? launch_rows<SWEEP, 2, true, false>(a, z.RP, st) : launch_rows<SWEEP, 2, false, false>(a, z.RP, st);
    if (a.g.bf16) return dist ? launch_rows<SWEEP, 1, true, true>(a, z.RP, st) : launch_rows<SWEEP, 1, false, true>(a, z.RP, st);
    return dist ? launch_rows<SWEEP, 1, true, false>(a, z.RP, st) : launch_rows<SWEEP, 1, false, false>(a, z.RP, st);
}

}  // namespace

// Whether the tensor-core sweeps take this problem.
bool tc_route(const Geo& g) {
    if (g.wsw != g.ws || g.ws < 3 || g.p > kMaxRadius || g.Wk != g.W || g.H < 16) return false;
    if (g.bf16 ? g.cr != 8 && g.cr != 16 : g.cr > 16) return false;
    const int64_t tiles = (int64_t)((g.W + kTileW - 1) / kTileW) * ((g.H + kTileH - 1) / kTileH) * g.units;
    return tiles >= sm_count();
}

size_t tc_fwd_workspace(const Geo& g, bool want_nz) {
    const TcSizes z = sizes_of(g);
    // the packed (k|v) and its terms, which the backward reads again; with A, statistics and the packed keys of its kernel
    return z.packed + z.scal + (want_nz ? (((size_t)g.Np * g.units * 4 + 255) & ~(size_t)255) + tiled_operator_workspace(g) : 0);
}

size_t tc_bwd_workspace(const Geo& g) {
    const TcSizes z = sizes_of(g);
    return 2 * (z.packed + z.scal);
}

int tc_attention_fwd(const Geo& g, float scale, int dist, const float* q, const float* k, const float* v, float* y,
                     float* nz, float* stats, void* workspace, cudaStream_t st) {
    const TcSizes z = sizes_of(g);
    char* ws = static_cast<char*>(workspace);
    char* more = ws + z.packed + z.scal;
    if (nz && !stats) stats = reinterpret_cast<float*>(more);
    TcPackArgs pa{};
    pa.g = g; pa.Hp = z.Hp; pa.mode = dist ? 1 : 0; pa.dist = dist; pa.sl2 = scale * kLog2e;
    pa.src[0] = k; pa.src[1] = v;
    pa.packed = reinterpret_cast<uint4*>(ws);
    pa.scal = reinterpret_cast<float*>(ws + z.packed);
    int rc = pack(pa, st);
    if (rc) return rc;
    TcArgs a{};
    a.g = g; a.scale = scale; a.packed = pa.packed; a.scal = pa.scal; a.a0 = q; a.out = y; a.ostats = stats;
    if ((rc = sweep<SWEEP_FWD>(a, z, dist, st))) return rc;
    if (nz) return tiled_weights(g, scale, dist, q, k, stats, nz, more + (((size_t)g.Np * g.units * 4 + 255) & ~(size_t)255), st);
    return CA_OK;
}

int tc_attention_bwd(const Geo& g, float scale, int dist, const float* q, const float* k, const float* v, const float* y,
                     const float* dy, const float* stats, float* D, float* dq, float* dk, float* dv, void* workspace,
                     const void* fwd_workspace, cudaStream_t st) {
    const TcSizes z = sizes_of(g);
    char* ws = static_cast<char*>(workspace);
    const char* kv = static_cast<const char*>(fwd_workspace);
    int rc;
    TcPackArgs pa{};
    pa.g = g; pa.Hp = z.Hp; pa.dist = dist; pa.sl2 = scale * kLog2e;
    if (!kv) {
        pa.mode = dist ? 1 : 0;
        pa.src[0] = k; pa.src[1] = v;
        pa.packed = reinterpret_cast<uint4*>(ws + z.packed + z.scal);
        pa.scal = reinterpret_cast<float*>(ws + 2 * z.packed + z.scal);
        if ((rc = pack(pa, st))) return rc;
        kv = ws + z.packed + z.scal;
    }
    pa.mode = 2;
    pa.src[0] = q; pa.src[1] = dy;
    pa.packed = reinterpret_cast<uint4*>(ws);
    pa.scal = reinterpret_cast<float*>(ws + z.packed);
    pa.stats = stats; pa.y = y; pa.Dout = D;
    if ((rc = pack(pa, st))) return rc;
    TcArgs a{};
    a.g = g; a.scale = scale;
    a.packed = pa.packed; a.scal = pa.scal; a.a0 = k;
    a.out = dv;
    if ((rc = sweep<SWEEP_DV>(a, z, dist, st))) return rc;
    a.a1 = v; a.out = dk;
    if ((rc = sweep<SWEEP_DK>(a, z, dist, st))) return rc;
    a.packed = reinterpret_cast<const uint4*>(kv); a.scal = reinterpret_cast<const float*>(kv + z.packed);
    a.a0 = q; a.a1 = dy; a.row0 = stats; a.row1 = D; a.out = dq;
    return sweep<SWEEP_DQ>(a, z, dist, st);
}

}  // namespace ca
