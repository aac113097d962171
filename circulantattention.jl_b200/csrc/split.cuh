// Shared parts of the tensor-core sweeps (split_*.cu): softmax attention on 2-D windows with every Float32 operand as a pair
// of half-precision numbers.
//
// Arithmetic.  A Float32 number x is the sum of hi = half(x / s) and lo = half(x / s - hi), times a power of two s: 22 to 24
// of its bits.  A product of two such numbers is hi*hi + hi*lo + lo*hi on the tensor cores (mma.sync m16n8k16, Float32
// accumulators); lo*lo is below the last bit.  That is three tensor products where three-way bfloat16 splits take six and
// tf32 pairs three of twice the time: the warp-level unit runs 1024 half-precision FMAs per SM and cycle, 512 of tf32.
// tcgen05 is not used: its scores would leave and enter through tensor memory for the mask, the exponential and the
// split, which costs more than its rate gains at 16 to 64 channels (forward 70.6 us against 62.5 on the FMA pipe).
//
// Error against 64 bits (2-norm, standard normal, 57 x 54; y, dq, dk, dv in 1e-7, FMA pipe with 3 units and here with 4): ws 9, 8 channels
// 4.2, 4.6, 4.0, 3.7 and 2.2, 3.9, 3.7, 3.8, Distance 4.8, 6.6, 4.3, 3.9 and 2.2, 4.3, 3.9, 3.8; ws 11, 16 channels 5.6, 5.1, 4.7, 4.4 and
// 2.3, 3.8, 3.7, 3.7, Distance 6.1, 8.2, 5.1, 4.7 and 2.5, 4.5, 4.1, 4.0; ws 21, 16 channels 6.0, 6.3, 6.1, 6.1 and 2.7, 3.9, 3.8, 3.6,
// Distance 6.5, 8.7, 6.6, 6.2 and 2.7, 5.4, 4.6, 4.2.
//
// Tiles.  Rows of a product are 16 centre pixels: 8 rows (h) of two neighbouring columns (w), whose windows share all but two
// columns.  Columns are 8 pixels of the streamed column, so a window column takes NT = ceil((8 + 2p) / 8) tiles and 62 %
// (window 21) to 38 % (window 7) of the scores are inside the window; 16 rows of one column would leave 52 and 29 %.
// The mask costs nothing: it rides in the addend of the FMA that scales a score (-inf outside).
//
// Streamed rows.  [unit][column][row'][144 bytes] = hi then lo of the first tensor, hi then lo of the second, 16 bytes of
// scalars; row' = h + p with the circular halo unrolled.  bfloat16 tensors have no lower halves, and their rows no place for
// them: 80 bytes.  Either pitch is an odd number of 16-byte words, so ldmatrix reads eight rows without bank conflicts.  The power of
// two is common to a group of eight rows starting at a multiple of eight (a warp's window starts at one), so it is uniform over a
// tile.  It puts the group's largest magnitude into [2^11, 2^15): an element 2^13 below it keeps all bits, the least step is 2^-36 of
// the largest.
//
// Range.  Half pairs end at a fixed step, so large values would cost pixels whose window does not hold them: their operands when
// they share a group, their weights when they share a step.  A warp therefore recomputes its pixels from the tensors in Float32
// (exact_*) when one of its groups is marked (a NaN or an infinity, which a product of a tile would carry to pixels outside their
// window; a row or a channel too far below the group's largest; magnitudes below 2^-51 in a score's operand; split_pack.cu has the
// limits) or when the scales of its groups lie further apart than the sweep's weights have bits for (Seen).  Tensors whose
// magnitudes are alike within a window, or zero, meet neither.  One pixel of k times 1e2, 1e4, 1e6 (57 x 54, 4 units, ws 11), error of
// dq of the pixels whose windows do not hold it: 8.4e-7, 1.2e-5, 3.1e-3 without this and 4.0e-7, 3.7e-7, 3.7e-7 with it, FMA pipe
// 5.5e-7.  Where every warp recomputes (512 x 512, 8 units, ws 21, 2 % of v's pixels NaN) the forward takes 5.9 ms for 1.1, dq 7.1 for
// 1.4, dk/dv 8.9 for 1.9 (310, 379, 707 with a lane per pixel and loads from the tensors); one pixel in 10^4 times 1e6: 1.7, 2.1, 4.1.
//
// What bounds the sweeps (512 x 512, 8 units, ws 21): the tensor pipe is busy in 47 % (forward) to 54 % (dq, dk/dv) of the cycles, an
// instruction issues in 48 and 45 % (bfloat16: 29 to 37 %, 58 %); an mma also takes five issue slots from FMAs and waits behind them, and 12 to 16 warps of
// 128 to 168 registers do not cover the latencies of the chain score - exponential - split - sum.  Times are beside the rules of
// the dispatch (split_pack.cu).
#pragma once
#include "tile_common.cuh"
#include <cuda_fp16.h>
#include <float.h>

namespace ca {

struct SplitArgs {
    Geo g;
    float scale;
    int dist;
    const float* c0;        // centre tensors
    const float* c1;
    const float* stats;     // statistics of the centre pixels (dq)
    const float* D;
    float* o0;              // outputs
    float* o1;
    float* ostats;
    const float* x0;        // streamed tensors and their pixels' statistics in the reference layout, for the pixels that are recomputed
    const float* x1;
    const float* xstats;
    const float* xD;
    int* status;            // nullable device word of the caller: bit 0 is set when a stage wait ran out
    int* timeouts;          // device counter of the blocks that gave up waiting for a copy
    uint32_t wait_tries;    // polls before a wait gives up
};

struct SplitPackArgs {
    Geo g;
    int Hp;                 // padded rows per column: roundup4(H + 2p)
    const float* x0;
    const float* x1;
    float norm_mul;         // Distance: the scalar of a row is norm_mul |x0|^2 ...
    const float* stats;     // ... - stats log2(e), and -D goes with it (nullable: neither)
    const float* y;         // D = y . x1 ...
    const float* Din;       // ... or given
    float* Dout;            // nullable
    float* dst;
};

// Whether the forward, A's values and dq run here, and whether dk/dv does (wherever they do, and at more shapes).
bool split_shape_ok(const Geo& g, float scale);
bool split_dkdv_ok(const Geo& g, float scale);
// Packs (x0|x1); with `stats` also the scalars of the backward, D = y . x1 (written to Dout) or given.
int launch_split_pack(const Geo& g, float scale, int dist, const float* x0, const float* x1, const float* stats, const float* y, const float* Din,
                      float* Dout, float* dst, cudaStream_t st);
int run_split_fwd(const Geo& g, float scale, int dist, const float* q, const float* k, const float* v, const float* kv, float* y, float* stats,
                  cudaStream_t st);
// A's values in CSR order from the row statistics.
int run_split_emit(const Geo& g, float scale, int dist, const float* q, const float* k, const float* stats, const float* kv, float* nz,
                   cudaStream_t st);
int run_split_dq(const Geo& g, float scale, int dist, const float* q, const float* k, const float* v, const float* dy, const float* stats,
                 const float* D, const float* kv, float* dq, cudaStream_t st);
int run_split_dkdv(const Geo& g, float scale, int dist, const float* q, const float* k, const float* v, const float* dy, const float* stats,
                   const float* D, const float* qdy, float* dk, float* dv, cudaStream_t st);

namespace {

// Where the second tensor of a row begins, where its scalars, and the row's pitch; `lo`: with lower halves.
__host__ __device__ constexpr int split_second(bool lo) { return lo ? 64 : 32; }
__host__ __device__ constexpr int split_scalars(bool lo) { return 2 * split_second(lo); }
__host__ __device__ constexpr int split_row_bytes(bool lo) { return split_scalars(lo) + 16; }
constexpr int kSplitSteps = 3, kSplitWarps = 4;
__host__ __device__ constexpr int split_rows(int nt) { return 8 * (kSplitWarps - 1) + 8 * nt; }
__host__ __device__ constexpr int split_stage_bytes(int nt, bool lo) { return (split_rows(nt) * split_row_bytes(lo) + 127) & ~127; }
__host__ __device__ inline int split_hp(const Geo& g) { return (g.H + 2 * g.p + 3) & ~3; }
inline int split_tiles(const Geo& g) { return (8 + 2 * g.p + 7) / 8; }

// ---------------------------------------------------------------- device
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm2(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// d = a b + c, 16 x 16 by 16 x 8.
__device__ __forceinline__ void mma16(float (&d)[4], const uint32_t* a, uint32_t b0, uint32_t b1, const float (&c)[4]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ void mma16(float (&d)[4], const uint32_t* a, uint32_t b0, uint32_t b1) {                // d = a b
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// hi and lo of two numbers below 2^15.  The remainder as a mixed-precision FMA: 1.34 SM cycles a warp and pair; with a conversion
// back to Float32 and a subtraction 1.59, with the low bits masked off 1.82.
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x, y);
    float rx, ry;
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(rx) : "h"(__half_as_ushort(__low2half(h))), "h"((unsigned short)0xbc00), "f"(x));
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(ry) : "h"(__half_as_ushort(__high2half(h))), "h"((unsigned short)0xbc00), "f"(y));
    const __half2 l = __floats2half2_rn(rx, ry);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
// Pairs of Float32 numbers for the two-lane instructions, kept as one register pair: a coefficient that stands twice in a pair is
// then formed once and not for every use.
typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t pair(float x, float y) {
    pair_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpair(pair_t p) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
    return r;
}
__device__ __forceinline__ pair_t fma_pair(pair_t a, pair_t b, pair_t c) {
    pair_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ pair_t add_pair(pair_t a, pair_t b) {
    pair_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair_t mul_pair(pair_t a, pair_t b) {
    pair_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// Biased exponent of the power of two that brings magnitudes up to `bits` below 2^15: a multiple of `step`, 255 for a NaN or an
// infinity.  `least` is the smallest that is given, also to zeros.
__device__ __forceinline__ int scale_exp(uint32_t bits, int step, int least) {
    const int e = (int)(bits >> 23);
    if (bits == 0) return least;
    if (e == 255) return 255;
    return max((e - 14 + step - 1) / step * step, max(least, 4));
}
// Least exponent of a score's operands, 2^-55: the product of two scales is no denormal, so a start of -inf stays -inf.
constexpr int kLeastExp = 72;
// The least magnitude of a scaled number of which its halves hold all bits: 22 above the pair's last place of 2^-24, or the 8
// of a bfloat16 number above the 2^-24 of the upper half.  Groups reach 2^11 at least, so this is 2^-13 of their largest or less.
__host__ __device__ constexpr float least_value(bool lo) { return lo ? 0x1p-2f : 0x1p-16f; }
constexpr uint32_t kLeastNormal = 0x00800000u;
// A factor of scores above this may overflow them (a scaled product is at most 2^34), and a mask of -inf with them.
constexpr float kMostFactor = 0x1p93f;
// A factor of scores up to this: the last place of an operand, 2^-25, is no more than 2^-23 in a score.
constexpr float kFineFactor = 0x1p-14f;
__device__ __forceinline__ float exp_scale(int e) { return __uint_as_float((uint32_t)e << 23); }
__device__ __forceinline__ float exp_inverse(int e) { return e ? __uint_as_float((uint32_t)(254 - e) << 23) : 0.f; }

// One real channel of a dense tensor, whatever its storage.
__device__ __forceinline__ void st_channel(float* dst, const Geo& g, int u, int cc, int npix, int pix, float x) {
    if (g.cpe == 2) dst[goff<2>(u, g.cr, cc, npix, pix)] = x;
    else if (g.bf16) st_real<true>(dst, goff<1>(u, g.cr, cc, npix, pix), x);
    else st_real<false>(dst, goff<1>(u, g.cr, cc, npix, pix), x);
}

// The channels 2t, 2t+1, 2t+8, 2t+9 (t = lane % 4) of the two pixels of a lane's row: what a lane holds of a row of an A
// operand and of a result.  Pixels outside the image and channels past the unit's read some other element of the tensor and
// are zeroed in Centre::form: without conditions all loads of a warp are in flight together.
struct Raw {
    float x[2][4];
    __device__ __forceinline__ void load(const float* src, const Geo& g, int u, int h, int w, int tq) {
        const int hc = min(h, g.H - 1);
        const int pix[2] = {hc + g.H * w, hc + g.H * min(w + 1, g.W - 1)};
        if (g.cpe == 2) {
            const float2* s2 = reinterpret_cast<const float2*>(src) + (int64_t)u * g.c * g.Np;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float2 z = __ldg(s2 + (int64_t)min(tq + 4 * i, g.c - 1) * g.Np + pix[r]);
                    x[r][2 * i] = z.x;
                    x[r][2 * i + 1] = z.y;
                }
            return;
        }
        const int64_t o = (int64_t)u * g.cr * g.Np;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t c = o + (int64_t)min(2 * tq + (i & 1) + 8 * (i >> 1), g.cr - 1) * g.Np;
#pragma unroll
            for (int r = 0; r < 2; ++r) x[r][i] = g.bf16 ? ld_real<true>(src, c + pix[r]) : ld_real<false>(src, c + pix[r]);
        }
    }
};
// The channel of a lane's element i.
__device__ __forceinline__ int lane_channel(int i, int tq) { return 2 * tq + (i & 1) + 8 * (i >> 1); }

// All channels of one pixel, zeros behind the unit's last.
__device__ __forceinline__ void load_pixel(const float* src, const Geo& g, int u, int npix, int pix, float (&x)[16]) {
    if (g.cpe == 2) {
        const float2* s = reinterpret_cast<const float2*>(src) + (int64_t)u * g.c * npix + pix;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 z = i < g.c ? __ldg(s + (int64_t)i * npix) : make_float2(0.f, 0.f);
            x[2 * i] = z.x;
            x[2 * i + 1] = z.y;
        }
        return;
    }
    const int64_t o = (int64_t)u * g.cr * npix + pix;
    if (g.bf16) {
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = i < g.cr ? ld_real<true>(src, o + (int64_t)i * npix) : 0.f;
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = i < g.cr ? __ldg(src + o + (int64_t)i * npix) : 0.f;
    }
}
// Dot products in four short chains, which round less than one of 16.
__device__ __forceinline__ float dot16(const float (&x)[16], const float (&y)[16]) {
    pair_t s[2];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const pair_t a = pair(x[2 * i], x[2 * i + 1]), b = pair(y[2 * i], y[2 * i + 1]);
        s[i & 1] = i < 2 ? mul_pair(a, b) : fma_pair(a, b, s[i & 1]);
    }
    const float2 z = unpair(add_pair(s[0], s[1]));
    return z.x + z.y;
}
__device__ __forceinline__ float score(const SplitArgs& a, const float (&x)[16], const float (&y)[16]) {
    if (!a.dist) return dot16(x, y);
    float d[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) d[i] = x[i] - y[i];
    return -0.5f * dot16(d, d);
}
// acc += f x
__device__ __forceinline__ void add_scaled(float (&acc)[16], float f, const float (&x)[16]) {
    const pair_t ff = pair(f, f);
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        const float2 z = unpair(fma_pair(pair(x[i], x[i + 1]), ff, pair(acc[i], acc[i + 1])));
        acc[i] = z.x;
        acc[i + 1] = z.y;
    }
}

// The recomputing paths (see "Range").  A warp puts a column of the two streamed tensors into its share of the step buffers, whose sweep is
// over, as Float32 rows of kExactPitch numbers: 16 channels of the first, 16 of the second, two scalars.  Lanes l and l + 16 own
// pixel (row l / 2, column l % 2) of the warp's 16 and take every other row of its window; their sums are added at the end.
constexpr int kExactPitch = 36, kExactValuesPitch = 20;       // (A's values: the first tensor and the 16 pixels themselves)
template <int NT, bool LO>
__device__ __forceinline__ float* exact_rows() {
    extern __shared__ unsigned char smem_raw[];
    constexpr int share = 2 * kSplitSteps * split_stage_bytes(NT, LO) / kSplitWarps / 16 * 16;
    static_assert(share >= 8 * NT * kExactPitch * 4 && share >= (8 * NT + 16) * kExactValuesPitch * 4, "a column of each warp");
    const uint32_t begin = smem_u32(smem_raw);
    return reinterpret_cast<float*>(smem_raw + (((begin + 127u) & ~127u) - begin) + (threadIdx.x >> 5) * share);
}
struct ExactLane {
    int lane, half, dh0, r, h, w, pix;                       // dh0: the pixel's first row in the buffer; pix: clamped to the image
    bool ok;
    __device__ __forceinline__ ExactLane(const Geo& g, int row0, int w0) {
        lane = threadIdx.x & 31;
        half = lane >> 4;
        dh0 = (lane & 15) >> 1;
        r = lane & 1;
        h = row0 + dh0;
        w = w0 + r;
        ok = h < g.H && w < g.W;
        pix = min(h, g.H - 1) + g.H * min(w, g.W - 1);
    }
    // Whether the pixel's window holds the s-th column of the warp's.
    __device__ __forceinline__ bool meets(const Geo& g, int s) const { return s != (r ? 0 : g.ws); }
    // The pixel of the streamed tensors that this lane copies for the s-th column.
    __device__ __forceinline__ int streamed(const Geo& g, int row0, int w0, int s) const {
        return wrap_axis(row0 - g.p + lane, g.H) + g.H * wrap_axis(w0 - g.p + s + g.wk_off, g.Wk);
    }
};
__device__ __forceinline__ void write16(float* to, const float (&x)[16]) {
#pragma unroll
    for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(to + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
}
__device__ __forceinline__ void read16(const float* from, float (&x)[16]) {
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
        const float4 z = *reinterpret_cast<const float4*>(from + i);
        x[i] = z.x;
        x[i + 1] = z.y;
        x[i + 2] = z.z;
        x[i + 3] = z.w;
    }
}
__device__ __forceinline__ void exact_copy(const SplitArgs& a, int u, int pix, float* row) {
    float x[16];
    load_pixel(a.x0, a.g, u, a.g.Npk, pix, x);
    write16(row, x);
    load_pixel(a.x1, a.g, u, a.g.Npk, pix, x);
    write16(row + 16, x);
}
// The sums of a pixel's two lanes, times f, into the dense tensor.
__device__ __forceinline__ void exact_store(float* dst, const Geo& g, int u, const ExactLane& L, const float (&x)[16], float f) {
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        const float z = (x[c] + __shfl_xor_sync(0xffffffffu, x[c], 16)) * f;
        if (L.ok && !L.half && c < g.cr) st_channel(dst, g, u, c, g.Np, L.pix, z);
    }
}

// A lane's four channels of a pixel: x[0..1] in the result's first eight channels, x[2..3] in its second.
__device__ __forceinline__ void store_pixel(float* dst, const Geo& g, int u, int pix, int tq, float x0, float x1, float x2, float x3) {
    if (g.cpe == 2) {
        float2* d2 = reinterpret_cast<float2*>(dst);
        if (tq < g.c) d2[((int64_t)u * g.c + tq) * g.Np + pix] = make_float2(x0, x1);
        if (tq + 4 < g.c) d2[((int64_t)u * g.c + tq + 4) * g.Np + pix] = make_float2(x2, x3);
        return;
    }
    const float x[4] = {x0, x1, x2, x3};
    const int64_t o = (int64_t)u * g.cr * g.Np + pix;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int c = lane_channel(i, tq);
        if (c >= g.cr) continue;
        if (g.bf16) st_real<true>(dst, o + (int64_t)c * g.Np, x[i]);
        else st_real<false>(dst, o + (int64_t)c * g.Np, x[i]);
    }
}
__device__ __forceinline__ uint32_t abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t quad_max(uint32_t x) {
    x = max(x, __shfl_xor_sync(0xffffffffu, x, 1));
    return max(x, __shfl_xor_sync(0xffffffffu, x, 2));
}
__device__ __forceinline__ float quad_max(float x) {
    x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
    return fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
}
__device__ __forceinline__ float quad_sum(float x) {
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    return x + __shfl_xor_sync(0xffffffffu, x, 2);
}

// Biased exponent of a power of two above |x| (255 for what is no number).
__device__ __forceinline__ int above(float x) {
    const uint32_t b = abs_bits(x);
    return b ? min((int)(b >> 23) + 1, 255) : 0;
}

// An A operand: the split vectors of the two pixels of each row of a tile, with each pixel's scale, squared norm and `top`, the
// biased exponent of a power of two above its norm (0: the vector is zero).  `top` comes from the scaled vector, whose squares
// neither vanish nor overflow: those of cotangents of 1e-19 and below do.
// LO: the operands have lower halves.  bfloat16 tensors do not: their 8 bits fit the upper one, which leaves one product of a score
// and two of a weighted sum (1024 x 1024, 8 units, ws 21: forward 4277 -> 3590 us, dq 5517 -> 4173, dk/dv 7448 -> 6267), rows of 80
// bytes for 144, one ldmatrix for both tensors' scores in the backward, and registers for one more block per SM (pack and
// forward together 3930 -> 3815 us, forward and backward 14812 -> 13340; 512 x 512, 8 units: ws 9 1540 -> 1451, ws 13 2328 -> 2111;
// 200 x 180, 4 units, ws 25: 352 -> 317).
template <bool LO>
struct Centre {
    uint32_t hi[4], lo[4];
    float scale[2], norm2[2];
    int top[2];
    bool bad;
    __device__ __forceinline__ void form(const Raw& raw, const Geo& g, int h, int w, int tq, int least) {
        bad = false;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const bool ok = h < g.H && w + r < g.W;
            float x[4];
            uint32_t m = 0;
            float n = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                x[i] = ok && lane_channel(i, tq) < g.cr ? raw.x[r][i] : 0.f;
                m = max(m, abs_bits(x[i]));
                n = fmaf(x[i], x[i], n);
            }
            m = quad_max(m);
            const int e = scale_exp(m, 1, least);
            norm2[r] = quad_sum(n);
            bad |= e == 255;
            scale[r] = exp_scale(e);
            const float inv = exp_inverse(e == 255 ? 0 : e);
            if (least) bad |= m >= kLeastNormal && __uint_as_float(m) * inv < least_value(LO);
            float ns = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) ns = fmaf(x[i] * inv, x[i] * inv, ns);
            ns = quad_sum(ns);
            top[r] = ns > 0.f ? above(sqrtf(ns)) + e - 127 : 0;
            split2(x[0] * inv, x[1] * inv, hi[r], lo[r]);
            split2(x[2] * inv, x[3] * inv, hi[2 + r], lo[2 + r]);
        }
    }
};

// Tiles of a step: NT of its first column, then NT of its second; offset of tile f from the step's first row.
template <int NT, bool LO>
__device__ __forceinline__ constexpr int tile_offset(int f) {
    return (f / NT) * split_stage_bytes(NT, LO) + 8 * (f % NT) * split_row_bytes(LO);
}

// x[f] = centre . streamed over the channels for the tiles of a step: `b` is this lane's ldmatrix address inside the first tensor or
// the second.  The chains of the tiles advance together (a warp issues in order and a dependent product waits 20 cycles);
// small products first, since the unit cuts its sums.
template <int NT, bool LO>
__device__ __forceinline__ void dot_tiles(const Centre<LO>& a, uint32_t b, float (&x)[2 * NT][4]) {
    uint32_t f[2 * NT][4];
#pragma unroll
    for (int t = 0; t < 2 * NT; ++t) {
        if (LO) ldsm4(b + tile_offset<NT, LO>(t), f[t]);       // hi of 8 + 8 channels, lo of 8 + 8
        else ldsm2(b + tile_offset<NT, LO>(t), f[t]);
    }
    if (LO) {
#pragma unroll
        for (int t = 0; t < 2 * NT; ++t) mma16(x[t], a.lo, f[t][0], f[t][1]);
#pragma unroll
        for (int t = 0; t < 2 * NT; ++t) mma16(x[t], a.hi, f[t][2], f[t][3], x[t]);
    }
#pragma unroll
    for (int t = 0; t < 2 * NT; ++t) {
        if (LO) mma16(x[t], a.hi, f[t][0], f[t][1], x[t]);
        else mma16(x[t], a.hi, f[t][0], f[t][1]);
    }
}

// acc += S * (weights . streamed) over the pixels of a step.  The weights of its tiles are split pairs as A operands: two tiles of a
// column make one of 16 pixels, the odd last ones of the two columns another.  `b`: this lane's transposing ldmatrix address
// for 16 rows of a column, `bt` the one for 8 rows of each column.  The unit cuts its sums instead of rounding them, 0.7
// units of the last place of a partial sum on average; the sums of a step therefore start at zero, the products of the
// upper halves apart from the small ones, and are added to the running ones in Float32.
template <int NT, bool LO>
__device__ __forceinline__ void outer_tiles(const uint32_t (&hi)[2 * NT][2], const uint32_t (&lo)[2 * NT][2], uint32_t b, uint32_t bt, const pair_t (&S)[2],
                                            pair_t (&acc)[2][2]) {
    float c[2][4], d[2][4];
#pragma unroll
    for (int k = 0; k < NT; ++k) {
        const bool tail = (NT & 1) && k == NT - 1;
        const int t = tail ? NT - 1 : (k < NT / 2 ? 2 * k : NT + 2 * (k - NT / 2)), t1 = tail ? 2 * NT - 1 : t + 1;
        const uint32_t at = (tail ? bt : b) + tile_offset<NT, LO>(t);
        uint32_t x[4], y[4];
        ldsm4t(at, x);                                         // hi: channels 0-7 of 8 + 8 rows, channels 8-15
        if (LO) ldsm4t(at + 32, y);                            // lo
        const uint32_t ah[4] = {hi[t][0], hi[t][1], hi[t1][0], hi[t1][1]};
        const uint32_t al[4] = {lo[t][0], lo[t][1], lo[t1][0], lo[t1][1]};
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            if (k == 0) mma16(c[n], ah, x[2 * n], x[2 * n + 1]);
            else mma16(c[n], ah, x[2 * n], x[2 * n + 1], c[n]);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            if (k == 0) mma16(d[n], al, x[2 * n], x[2 * n + 1]);
            else mma16(d[n], al, x[2 * n], x[2 * n + 1], d[n]);
        }
        if (LO) {
#pragma unroll
            for (int n = 0; n < 2; ++n) mma16(d[n], ah, y[2 * n], y[2 * n + 1], d[n]);
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; i += 2)
            acc[n][i / 2] = fma_pair(add_pair(pair(c[n][i], c[n][i + 1]), pair(d[n][i], d[n][i + 1])), S[i / 2], acc[n][i / 2]);
}

// The same two products a column at a time, for the backward, whose four products need no other independent work.  Scores of one
// column against two centre operands: x from the first tensor (`b`), y from the second.
template <int NT, bool LO>
__device__ __forceinline__ void dot_column(const Centre<LO>& a0, const Centre<LO>& a1, uint32_t b, float (&x)[NT][4], float (&y)[NT][4]) {
    constexpr int RB = split_row_bytes(LO);
    uint32_t f[NT][4], e[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        ldsm4(b + 8 * t * RB, f[t]);
        if (LO) {
            ldsm4(b + 8 * t * RB + split_second(LO), e[t]);
        } else {                                               // the second tensor's upper halves stand where the first's lower ones would
            e[t][0] = f[t][2];
            e[t][1] = f[t][3];
        }
    }
    if (LO) {
#pragma unroll
        for (int t = 0; t < NT; ++t) mma16(x[t], a0.lo, f[t][0], f[t][1]);
#pragma unroll
        for (int t = 0; t < NT; ++t) mma16(y[t], a1.lo, e[t][0], e[t][1]);
#pragma unroll
        for (int t = 0; t < NT; ++t) mma16(x[t], a0.hi, f[t][2], f[t][3], x[t]);
#pragma unroll
        for (int t = 0; t < NT; ++t) mma16(y[t], a1.hi, e[t][2], e[t][3], y[t]);
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        if (LO) mma16(x[t], a0.hi, f[t][0], f[t][1], x[t]);
        else mma16(x[t], a0.hi, f[t][0], f[t][1]);
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        if (LO) mma16(y[t], a1.hi, e[t][0], e[t][1], y[t]);
        else mma16(y[t], a1.hi, e[t][0], e[t][1]);
    }
}
// acc += S * (weights . streamed) over one column.  An odd last tile of the first column (TAIL 0) waits in `tail` for that of the
// second (TAIL 1), with which it makes one operand.
struct Tail {
    uint32_t hi[2], lo[2];
};
template <int NT, bool LO, int TAIL>
__device__ __forceinline__ void outer_column(const uint32_t (&hi)[NT][2], const uint32_t (&lo)[NT][2], Tail& tail, uint32_t b, uint32_t bt,
                                             const pair_t (&S)[2], pair_t (&acc)[2][2]) {
    constexpr int RB = split_row_bytes(LO), K = NT / 2 + ((NT & 1) && TAIL ? 1 : 0);
    float c[2][4], d[2][4];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const bool last = k == NT / 2;                         // the tails of both columns
        const uint32_t at = (last ? bt : b) + (last ? 8 * (NT - 1) : 16 * k) * RB;
        const int t = last ? NT - 1 : 2 * k, t1 = last ? NT - 1 : 2 * k + 1;
        uint32_t x[4], y[4];
        ldsm4t(at, x);
        if (LO) ldsm4t(at + 32, y);
        const uint32_t ah[4] = {last ? tail.hi[0] : hi[t][0], last ? tail.hi[1] : hi[t][1], hi[t1][0], hi[t1][1]};
        const uint32_t al[4] = {last ? tail.lo[0] : lo[t][0], last ? tail.lo[1] : lo[t][1], lo[t1][0], lo[t1][1]};
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            if (k == 0) mma16(c[n], ah, x[2 * n], x[2 * n + 1]);
            else mma16(c[n], ah, x[2 * n], x[2 * n + 1], c[n]);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            if (k == 0) mma16(d[n], al, x[2 * n], x[2 * n + 1]);
            else mma16(d[n], al, x[2 * n], x[2 * n + 1], d[n]);
        }
        if (LO) {
#pragma unroll
            for (int n = 0; n < 2; ++n) mma16(d[n], ah, y[2 * n], y[2 * n + 1], d[n]);
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; i += 2)
            acc[n][i / 2] = fma_pair(add_pair(pair(c[n][i], c[n][i + 1]), pair(d[n][i], d[n][i + 1])), S[i / 2], acc[n][i / 2]);
    if ((NT & 1) && !TAIL) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            tail.hi[r] = hi[NT - 1][r];
            tail.lo[r] = lo[NT - 1][r];
        }
    }
}

// What a warp has met: the largest scale of both tensors, then the smallest but for zeros, in a byte each; 0 once its pixels have to be
// recomputed.  The word waits in shared memory, since it changes rarely and the sweeps have no register to spare; all lanes hold
// and write the same one.
struct Seen {
    static __device__ __forceinline__ volatile uint32_t* slot() {
        __shared__ uint32_t slots[kSplitWarps];
        return &slots[threadIdx.x >> 5];
    }
    static __device__ __forceinline__ void clear(bool bad) { *slot() = __any_sync(0xffffffffu, bad) ? 0u : 0xffff0000u; }
    static __device__ __forceinline__ bool bad() { return *slot() == 0; }
    // The largest scales of a step.
    static __device__ __forceinline__ void tops(uint32_t word, uint32_t& e0, uint32_t& e1) {
        e0 = __reduce_max_sync(0xffffffffu, word & 255u);
        e1 = __reduce_max_sync(0xffffffffu, word >> 8 & 255u);
    }
    // Takes them in; the pixels are recomputed from a mark on, when the extremes lie further apart than the limits (binary orders), or
    // when a lane says so.
    static __device__ __forceinline__ void add(uint32_t word, uint32_t e0, uint32_t e1, int limit0, int limit1, bool bad) {
        const uint32_t bytes = *slot(), b0 = word & 255u, b1 = word >> 8 & 255u;
        const uint32_t hi0 = max(bytes & 255u, e0), lo0 = min(bytes >> 16 & 255u, __reduce_min_sync(0xffffffffu, b0 ? b0 : 255u));
        const uint32_t hi1 = max(bytes >> 8 & 255u, e1), lo1 = min(bytes >> 24, __reduce_min_sync(0xffffffffu, b1 ? b1 : 255u));
        bad |= bytes == 0 || hi0 == 255u || hi1 == 255u || (int)hi0 > (int)lo0 + limit0 || (int)hi1 > (int)lo1 + limit1;
        *slot() = __any_sync(0xffffffffu, bad) ? 0u : hi0 | hi1 << 8 | lo0 << 16 | lo1 << 24;
    }
};

// 0 for a score inside the window of the lane's row, -inf outside (tile t, element i of the lane's four).
__device__ __forceinline__ float window_mask(int lane, int p, int t, int i) {
    const int d = 8 * t + 2 * (lane & 3) + (i & 1) - (lane >> 2);
    return d >= 0 && d <= 2 * p ? 0.f : -INFINITY;
}

__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    return done;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Runs a sweep: a block of four warps owns 32 rows of two columns, each warp eight of them.  The columns meet the ws + 1 columns of
// their windows two at a time ("steps"); thread 0 copies them, and every warp with rows in the image reads at its own
// pace.  A step's buffer is refilled one step after it was read, when the other warps have mostly left it as well.  Every
// wait is bounded.
// Sweep: begin(w0, own) with the shared address behind the buffers, step(rb, first, last) with the shared address of the warp's first row in the first of the step's columns (the
// second follows one stage on), end(w0, poison).  A wait that ran out ends the warp's sweep: the block reports it (device
// counter, caller's status word), and what it stores is poisoned with NaN.
// Measured against this cut at 512 x 512, 8 units, ws 21 (forward 1090 us): two pairs of columns per block on the same buffers with
// half the copies 1100, several pairs of columns one after the other 1100, two buffers instead of three 1170.
template <int NT, bool LO, class Sweep>
__device__ __forceinline__ void split_run(const SplitArgs& a, const CUtensorMap* map, Sweep& sweep) {
    constexpr int SB = split_stage_bytes(NT, LO);
    constexpr uint32_t kBytes = 2 * split_rows(NT) * split_row_bytes(LO);
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kSplitSteps];
    const Geo& g = a.g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int steps = (g.ws + 1) / 2, w0 = 2 * blockIdx.x, h0 = blockIdx.y * 8 * kSplitWarps, u = blockIdx.z;
    const uint32_t full = smem_u32(bars), stages = (smem_u32(smem_raw) + 127u) & ~127u;
    const bool live = h0 + 8 * warp < g.H;                    // the warp's rows reach into the image
    int kc = stage_column(g, w0, 0);
    auto copy = [&](uint32_t bar, uint32_t dst) {
        mbar_arrive_expect_tx(bar, kBytes);
        tma_load_4d(dst, map, 0, h0, kc, u, bar);
        kc = kc + 1 == g.Wk ? 0 : kc + 1;
        tma_load_4d(dst + SB, map, 0, h0, kc, u, bar);
        kc = kc + 1 == g.Wk ? 0 : kc + 1;
    };
    if (threadIdx.x == 0) {
        for (int i = 0; i < kSplitSteps; ++i) {
            mbar_init(&bars[i], 1);
            mbar_init(&bars[kSplitSteps + i], min(kSplitWarps, (g.H - h0 + 7) >> 3));
        }
        mbar_fence_init();
        for (int i = 0; i < kSplitSteps && i < steps; ++i) copy(full + 8 * i, stages + 2 * SB * i);
    }
    __syncthreads();
    bool lost = false;
    if (live) {
        sweep.begin(w0, stages + 2 * SB * kSplitSteps);
        uint32_t bar = full, ring = stages + 8 * warp * split_row_bytes(LO), phase = 0;
#pragma unroll 1
        for (int step = 0; step < steps; ++step) {
            if (!__all_sync(0xffffffffu, mbar_try(bar, phase))) {
                lost = !__all_sync(0xffffffffu, mbar_wait(bar, phase, a.wait_tries));
                if (lost) break;
            }
            sweep.step(ring, step == 0, step == steps - 1);
            __syncwarp();
            if (lane == 0) mbar_arrive(bar + 8 * kSplitSteps);
            if (warp == 0 && step > 0 && step - 1 + kSplitSteps < steps) {
                const bool first = bar == full;
                const uint32_t b = first ? bar + 8 * (kSplitSteps - 1) : bar - 8;
                const uint32_t d = (first ? ring + 2 * SB * (kSplitSteps - 1) : ring - 2 * SB);
                lost = !__all_sync(0xffffffffu, mbar_wait(b + 8 * kSplitSteps, first ? phase ^ 1 : phase, a.wait_tries));
                if (lost) break;
                if (lane == 0) copy(b, d);
            }
            bar += 8;
            ring += 2 * SB;
            if (bar == full + 8 * kSplitSteps) { bar = full; ring -= 2 * SB * kSplitSteps; phase ^= 1; }
        }
    }
    float poison = 0.f;
    if (__syncthreads_or(lost)) {
        if (threadIdx.x == 0) {
            // copies still in flight get a bounded chance to land before the block exits
            for (int i = 0; i < kSplitSteps; ++i) mbar_wait(full + 8 * i, 0, 1u << 12);
            atomicAdd(a.timeouts, 1);
            if (a.status) atomicOr(a.status, 1);
        }
        poison = __int_as_float(0x7fc00000);
    }
    if (live) sweep.end(w0, poison);
}

// This lane's ldmatrix offsets inside a stage, relative to the warp's first row.
__device__ __forceinline__ uint32_t dot_offset(int lane, bool lo) {      // [hi 0-7, hi 8-15, lo 0-7, lo 8-15] of 8 rows
    return (lane & 7) * split_row_bytes(lo) + ((lane >> 3) & 1) * 16 + (lane >> 4) * 32;
}
__device__ __forceinline__ uint32_t outer_offset(int lane, bool lo, int next) {   // [rows 0-7, those `next` bytes on] x [channels 0-7, 8-15]
    return (lane & 7) * split_row_bytes(lo) + ((lane >> 3) & 1) * next + (lane >> 4) * 16;
}
// Where the word of scales lies that this lane watches: lanes 0-3 the groups of the step's first column, lanes 4-7 those of its
// second, and so on; groups past the padded rows do not exist.
template <int NT, bool LO>
__device__ __forceinline__ uint32_t word_offset(const Geo& g, int lane, int row0) {
    const int t = min(min(lane & 3, NT - 1), (split_hp(g) - row0 - 1) >> 3);
    return ((lane >> 2) & 1) * split_stage_bytes(NT, LO) + 8 * t * split_row_bytes(LO) + split_scalars(LO);
}
// Tiles whose group has another scale than the step's largest (byte `shift` of the words), times the ratio; `least`: the smallest
// exponent of the ratio (0: it may vanish; groups without a scale hold zeros only).
// `column`: the first of the tiles.
template <int NT, int N>
__device__ __forceinline__ void scale_tiles(float (&x)[N][4], uint32_t word, uint32_t cur, int shift, int least, int column = 0) {
#pragma unroll
    for (int t = 0; t < N; ++t) {
        const int e = __shfl_sync(0xffffffffu, word, t < NT ? 4 * column + t : 4 + t - NT) >> shift & 255u;
        const float f = e ? exp_scale(max(127 + e - (int)(cur >> shift & 255u), least)) : 1.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) x[t][i] *= f;
    }
}
// Two neighbouring rows' scalars (see the layout above) at the shared address of the even or of the odd row's.
__device__ __forceinline__ pair_t lds_pair(uint32_t addr) {
    pair_t x;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(x) : "r"(addr));
    return x;
}
__device__ __forceinline__ uint32_t ldsu32(uint32_t addr) {
    uint32_t x;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(addr));
    return x;
}

// ---------------------------------------------------------------- host
// Launch geometry, shared memory (`extra` bytes of the sweep's own) and the tensor map of a sweep.
inline int split_prepare(const Geo& g, float scale, int dist, const float* packed, Launch* L, SplitArgs* a, size_t extra = 0) {
    const bool lo = !g.bf16;
    const int nt = split_tiles(g), rb = split_row_bytes(lo), rf = rb / 4, hp = split_hp(g);
    a->g = g;
    a->scale = scale;
    a->dist = dist;
    a->status = status_word();
    if (!(a->timeouts = stage_timeout_counter())) return cuda_fail(cudaGetLastError(), "cudaGetSymbolAddress(stage timeouts)");
    a->wait_tries = kWaitTries;
    L->grid = dim3((unsigned)((g.W + 1) / 2), (unsigned)((g.H + 8 * kSplitWarps - 1) / (8 * kSplitWarps)), (unsigned)g.units);
    L->threads = 32 * kSplitWarps;
    L->smem = (size_t)2 * kSplitSteps * split_stage_bytes(nt, lo) + 128 + extra;
    if (L->smem > kMaxDynamicSmem || L->grid.y > 65535u) return CA_ERR_UNSUPPORTED;
    const uint64_t dims[4] = {(uint64_t)rf, (uint64_t)hp, (uint64_t)g.Wk, (uint64_t)g.units};
    const uint64_t strides[3] = {(uint64_t)rb, (uint64_t)hp * rb, (uint64_t)hp * rb * g.Wk};
    const uint32_t box[4] = {(uint32_t)rf, (uint32_t)split_rows(nt), 1, 1};
    return encode_tensor_map(&L->mv, packed, 4, dims, strides, box);
}

#define CA_LAUNCH_SPLIT(KERNEL, a, L, st)                                             \
    do {                                                                              \
        static std::atomic<int> have__{0};                                            \
        int rc__ = set_smem(KERNEL, (L).smem, have__);                                \
        if (rc__) return rc__;                                                        \
        KERNEL<<<(L).grid, (L).threads, (L).smem, st>>>(a, (L).mv);                   \
        count_tiled_launch();                                                         \
        count_tensor_launch();                                                        \
    } while (0)

}  // namespace
}  // namespace ca
