// Shared parts of the tiled kernels (*_sweep.cuh, tiled.cu, operators.cu, pack.cu): the stage pipeline, the packed layout, the
// centre loads and stores, and the host side that shapes a launch.
#pragma once
#include "tiled.cuh"
#include "tma.cuh"
#include <cuda_bf16.h>
#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>

namespace ca {

struct PackArgs {
    Geo g;
    int pp;                 // p' (even)
    int Hp;                 // padded rows per column: roundup4(H + 2p')
    int npairs;             // 1 or 2 tensor pairs
    int single;             // 1: rows hold one tensor (src[0]) in 20 words per slab instead of a pair in 36
    const float* src[4];    // pair j = (src[2j], src[2j+1])
    float* dst[2];
    float* planes;          // nullable
    const float* stats;     // with planes
    float stat_mul;         // plane 0 = stats * stat_mul: log2(e) for the softmax log-sum-exp, 1 for the entmax tau
    const float* Din;       // with planes: D given ...
    const float* y;         // ... or computed as dy . y
    const float* dy;
    float* Dout;            // nullable: D in the reference layout (interior rows)
};

// Launches the pack kernel (pack.cu); CA_ERR_UNSUPPORTED beyond its grid limits.
int launch_pack(const PackArgs& a, cudaStream_t st);
// Device counter of the CTAs that gave up a stage wait, on the current device (NULL with the CUDA error set).
int* stage_timeout_counter();
struct Padded {
    int pp, Hp;
    size_t pair_floats;     // one packed tensor pair
    size_t single_floats;   // one packed single tensor
    size_t plane_floats;    // both scalar planes
};

// Launches of the sweeps, compiled for exact (false) and for other channel counts and shapes (true).
template <bool ANYC>
int run_fwd(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* kv, float* y, float* stats,
            cudaStream_t st);
// The same and A's values in CSR order; CA_ERR_UNSUPPORTED where the rows of A do not fit the shared memory (values_fit).
template <bool ANYC>
int run_fwd_values(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* kv, float* y, float* stats,
                   float* nz, cudaStream_t st);
// mode 0: softmax; 1: entmax; 2: entmax pre-pass (writes D, needs no D and no dq).
template <bool ANYC>
int run_dq(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* dy, const float* stats,
           const float* D, const float* kv, float* dq, cudaStream_t st, int mode, float* Dout, float* weights = nullptr);
// One sweep of the entmax forward over the packed (k|v): mode 3 class maxima -> first threshold (tau),
// 4 one step of the threshold search (tau and `settled` updated in place), 5 y = sum max(s/2 - tau, 0)^2 v.
template <bool ANYC>
int run_entmax_fwd_sweep(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* kv,
                         float* tau, float* settled, float* y, int mode, int iter, cudaStream_t st);
template <bool ANYC>
int run_dkdv(const Geo& g, const Padded& P, float scale, int dist, const float* k, const float* v, const float* qdy,
             const float* planes, float* dk, float* dv, cudaStream_t st, bool entmax);
// dk and dv from the weights that run_dq stored (`weights` of weight_floats()).
template <bool ANYC>
int run_dkdv_stored(const Geo& g, const Padded& P, float scale, int dist, const float* k, const float* qdy, const float* weights, float* dk,
                    float* dv, cudaStream_t st);
// A's values in CSR order: from q, a packed operand and the row statistics, or the raw scores without them.
template <bool ANYC>
int run_emit(const Geo& g, const Padded& P, float scale, int dist, const float* q, const float* stats, float* nz,
             const float* packed, cudaStream_t st, bool single);
// out = alpha * (A (x) v) or its transposed form from A's values and the packed v; `centre`: the Distance pullback's tensor.
template <bool ANYC>
int run_apply(const Geo& g, const Padded& P, const float* nz, const float* packed, const float* centre, float* out,
              float alpha, int transposed, cudaStream_t st);

namespace {

// Two-channel arithmetic: a channel pair lives in two ordinary registers.  A step of a dot product is two scalar FMAs: its
// two multiplicands are fresh in every instruction, and packed they measured slower in every sweep (600 x 500, 8
// units, ws 21: forward 1774 -> 1871 us, dq 2567 -> 2685, dk/dv 3822 -> 3879).  Outer products are packed, below.
struct u64 { float x, y; };
__device__ __forceinline__ u64 pack2(float a, float b) { return u64{a, b}; }
__device__ __forceinline__ void unpack2(u64 v, float& a, float& b) { a = v.x; b = v.y; }
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) { return u64{fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)}; }
// acc + w * v with one coefficient for the pair, packed: consecutive outer-product instructions reuse the coefficient, so
// they run at the packed rate (61 against 50 TFLOP/s in registers, which dot products do not).
__device__ __forceinline__ u64 outer2(float w, u64 v, u64 acc) {
    u64 r;
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %2};\n\tmov.b64 b, {%3, %4};\n\tmov.b64 c, {%5, %6};\n\t"
        "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(w), "f"(v.x), "f"(v.y), "f"(acc.x), "f"(acc.y));
    return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) { return u64{a.x * b.x, a.y * b.y}; }
__device__ __forceinline__ u64 add2(u64 a, u64 b) { return u64{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ u64 zero2() { return u64{0.f, 0.f}; }
__device__ __forceinline__ void lds128(uint32_t addr, u64& lo, u64& hi) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(lo.x), "=f"(lo.y), "=f"(hi.x), "=f"(hi.y) : "r"(addr));
}
__device__ __forceinline__ float lds32(uint32_t addr) {
    float x;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(addr));
    return x;
}
__device__ __forceinline__ void sts32(uint32_t addr, float x) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(x) : "memory"); }
__device__ __forceinline__ float hsum2(u64 v) {
    float a, b;
    unpack2(v, a, b);
    return a + b;
}

// Sum of a per-lane partial over the NS lanes that share a pixel (NS = 1: nothing to do).
template <int NS>
__device__ __forceinline__ float lane_sum(float x) {
#pragma unroll
    for (int m = 1; m < NS; m <<= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
    return x;
}

struct TileArgs {
    Geo g;
    float scale;
    int TH;                 // rows per CTA
    int roff;               // p' - p: first window row inside a stage buffer
    int stage_bytes;        // bytes of one stage buffer (multiple of 128)
    int nsplit;             // 1 to kParts groups of warps sharing the stages of a tile
    int iter;               // entmax threshold search: number of the step (late steps fall back to Newton)
    int row_bytes;          // bytes of one packed pixel row: 144 per 16-channel slab
    int nstages;            // copy stages in flight per part: 2 or 3 (kStages)
    int extra_off;          // shared memory of the kernel's own behind the stages and the merge buffers, bytes
    int nbuf;               // apply: buffers for the staged values of A per warp (1 or 2)
    const float* c0;        // centre tensors (reference layout)
    const float* c1;
    const float* cs0;       // centre scalars (dq kernel: stats, D)
    const float* cs1;
    float* o0;              // outputs
    float* o1;
    float* ostats;
    int* status;            // nullable device word of the caller: bit 0 is set when a stage wait ran out
    int* timeouts;          // device counter of the CTAs that gave up waiting for a stage copy
    uint32_t wait_tries;    // polls before a stage wait gives up
};

constexpr int kStages = 3;
constexpr int kMaxDynamicSmem = 220 * 1024;
constexpr int kParts = 4;                      // groups of warps that can share the stages of a tile
constexpr uint32_t kWaitTries = 1u << 20;
constexpr int kEntmaxFwdSteps = 16;            // launches of the entmax threshold step (settled blocks leave at once)

constexpr int kRowFloats = 36;                 // 16 + 16 + 4 padding
constexpr int kRowBytes = kRowFloats * 4;      // 144
constexpr int kRunChunk = 32;                  // window rows whose entries of A are staged at a time
constexpr int kSingleFloats = 20;              // single-tensor rows: 16 + 4 padding (80 bytes, also conflict free)

// Units with 16*NS real channels ("slabs" of 16) pack a pixel row as 36*NS words: the first
// tensor's channels, then the second's, then 4*NS words of padding.  Inside a tensor's part the
// order is [4-channel chunk][slab][4]: chunk c of slab s sits 16*(c*NS + s) bytes in, so the NS
// lanes that share a pixel read consecutive 16-byte pieces, and the row stride (144*NS bytes:
// 16, 32 or 64 bytes past a multiple of 128) spreads the 8/NS pixels of a 128-bit load phase over
// distinct bank groups.  NS = 1 is the plain channel order.
// 16-channel slab `slab` of tensor `which` of the pixel row at shared-space byte address `a0`.
template <int NS>
__device__ __forceinline__ void lds_slab16(uint32_t a0, int which, int slab, u64 (&v)[8]) {
    const uint32_t b = a0 + which * (64 * NS) + slab * 16;
    lds128(b, v[0], v[1]);
    lds128(b + 16 * NS, v[2], v[3]);
    lds128(b + 32 * NS, v[4], v[5]);
    lds128(b + 48 * NS, v[6], v[7]);
}

// The squared norm of slab `slab` of the first tensor of the pixel row at `a0`: the pack leaves it in the slab's padding words
// (`pad` bytes into the row), so that the Distance sweeps do not form it for every key they meet, 16 FMAs each in every
// thread (600 x 500, 8 units, ws 21: forward 2123 -> 1918 us, dq 3029 -> 2668, dk/dv 4070 -> 3768; 128 x 96, 8 units, ws 15: 61 -> 55,
// 81 -> 72, 120 -> 111).
__device__ __forceinline__ float lds_norm(uint32_t a0, int pad, int slab) { return lds32(a0 + pad + 16 * slab); }

// Global offset of real channel cc of unit u at pixel pix (npix pixels per plane, cr real channels per unit).
template <int CPE>
__device__ __forceinline__ int64_t goff(int u, int cr, int cc, int npix, int pix) {
    if (CPE == 1) return ((int64_t)u * cr + cc) * npix + pix;
    return (((int64_t)u * (cr / 2) + (cc >> 1)) * npix + pix) * 2 + (cc & 1);
}
// The same for units whose channel count the kernel knows: the plane offsets become multiples of one product.
template <int CPE, int NCR>
__device__ __forceinline__ int64_t goff_exact(int u, int cc, int npix, int pix) { return goff<CPE>(u, NCR, cc, npix, pix); }

// Window radius along w: p for 2-D windows, 0 for a folded 1-D signal (wsw == 1), whose window
// runs along h only and continues into the neighbouring columns through the packed halo rows.
__device__ __forceinline__ int radius_w(const Geo& g) { return (g.wsw - 1) >> 1; }

__device__ __forceinline__ int stage_column(const Geo& g, int w0, int s) {
    int kc = (w0 - radius_w(g) + s + g.wk_off) % g.Wk;
    return kc < 0 ? kc + g.Wk : kc;
}

// Rotation of the sorted run of a CSR row: the entry of window offset d sits at (d + p + rot) mod ws,
// where the row's pixel has coordinate x on the window axis of length X (src/circulant.jl:11-15).
__device__ __forceinline__ int run_rot(int x, int X, int p, int ws) {
    return x < p ? x - p + ws : (x >= X - p ? x - p - X + ws : 0);
}
// Coordinate and length of the window axis for pixel (h, w): the image row in 2-D, the linear
// index in a folded 1-D signal.
__device__ __forceinline__ int axis_coord(const Geo& g, int h, int w) { return g.wsw == 1 ? h + g.H * w : h; }
__device__ __forceinline__ int axis_len(const Geo& g) { return g.wsw == 1 ? g.Np : g.H; }

template <int NQ>
__device__ __forceinline__ int stage_mask(int s, int p) {
    int mask = 0;
#pragma unroll
    for (int r = 0; r < NQ; ++r)
        if (s >= r && s <= r + 2 * p) mask |= 1 << r;
    return mask;
}

// Barrier of one group of warps (ids 1..PARTS; id 0 stays the CTA-wide barrier) that also tells whether any thread of it
// passes a true `flag`.  A group of one warp needs no barrier.  Immediate ids: one in a register reserves all sixteen.
__device__ __forceinline__ bool part_any(int part, int nthreads, bool flag) {
    int any;
#define CA_BAR_OR(ID)                                                                                                 \
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %2, 0;\n\tbar.red.or.pred q, " #ID ", %1, p;\n\t"          \
                 "selp.s32 %0, 1, 0, q;\n\t}" : "=r"(any) : "r"(nthreads), "r"((int)flag) : "memory")
    if (nthreads == 32) return __any_sync(0xffffffffu, flag);
    if (part == 0) CA_BAR_OR(1);
    else CA_BAR_OR(2);                                   // groups of more than one warp come in pairs at most
#undef CA_BAR_OR
    return any != 0;
}

// ---------------------------------------------------------------------------
// Stage pipeline of one group of warps ("part").  Thread 0 of the part is the
// producer: it arms the stage's mbarrier with the byte count and issues the
// TMA boxes; every consumer wait is bounded.
// ---------------------------------------------------------------------------
template <bool NSC>
struct StagePipe {
    uint32_t full;           // kStages barriers of this part (shared-space address)
    uint32_t base;           // stage buffers of this part
    int kc;                  // next column to copy

    __device__ __forceinline__ uint32_t bar(int buf) const { return full + 8 * buf; }
    __device__ __forceinline__ uint32_t vec(int buf, const TileArgs& a) const { return base + buf * a.stage_bytes; }
    // the two scalar planes of a stage, behind its rows
    static __device__ __forceinline__ uint32_t plane_bytes(int rows) { return (rows * 4 + 127) & ~127; }
    __device__ __forceinline__ uint32_t sc0(int buf, const TileArgs& a, int rows) const { return vec(buf, a) + ((rows * a.row_bytes + 127) & ~127); }

    __device__ __forceinline__ void issue(int buf, const TileArgs& a, const CUtensorMap* mv, const CUtensorMap* msc, int rows, int u, int h0) {
        mbar_arrive_expect_tx(bar(buf), (uint32_t)(rows * a.row_bytes + (NSC ? rows * 8 : 0)));
        tma_load_4d(vec(buf, a), mv, 0, h0, kc, u, bar(buf));
        if (NSC) {
            const uint32_t s0 = sc0(buf, a, rows);
            tma_load_3d(s0, msc, h0, kc, 2 * u, bar(buf));
            tma_load_3d(s0 + plane_bytes(rows), msc, h0, kc, 2 * u + 1, bar(buf));
        }
        kc = kc + 1 == a.g.Wk ? 0 : kc + 1;
    }
};

// Declares the pipeline of this thread's part and starts the first copies.
// Needs in scope: a (TileArgs), g, ROWS, u, h0, w0, NSTAGES (stages of the tile), mv, msc.
// PARTS: most groups of warps that the kernel is launched with.
#define CA_PIPE_PROLOGUE(NSCV, PARTS)                                                                \
    extern __shared__ unsigned char smem_raw[];                                                      \
    __shared__ __align__(8) uint64_t full_bar[PARTS * kStages];                                         \
    const int PT = PARTS == 1 ? blockDim.x : blockDim.x / a.nsplit;          /* threads per part */  \
    const int part = PARTS == 1 ? 0 : threadIdx.x / PT;                                              \
    const int lt = threadIdx.x - part * PT;                                                          \
    const int s_begin = PARTS == 1 ? 0 : part * NSTAGES / a.nsplit;                                  \
    const int s_end = PARTS == 1 ? NSTAGES : (part + 1) * NSTAGES / a.nsplit;                        \
    unsigned char* smem_al = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);            \
    StagePipe<NSCV> pipe;                                                                            \
    pipe.full = smem_u32(full_bar) + part * kStages * 8;                                             \
    pipe.base = smem_u32(smem_al) + part * a.nstages * a.stage_bytes;                                \
    pipe.kc = stage_column(g, w0, s_begin);                                                          \
    if (threadIdx.x == 0) {                                                                          \
        for (int i = 0; i < PARTS * kStages; ++i) mbar_init(&full_bar[i], 1);                        \
        mbar_fence_init();                                                                           \
    }                                                                                                \
    __syncthreads();                                                                                 \
    if (lt == 0)                                                                                     \
        for (int i = 0; i < a.nstages && s_begin + i < s_end; ++i) pipe.issue(i, a, &mv, &msc, ROWS, u, h0);

// Consumer loop over the stages of this part: bounded wait, BODY (sees s and buf), recycle the buffer.  What a stage costs
// besides its window rows counts where windows are short: running counters instead of divisions, one barrier that
// also collects the error flag, 32-bit shared addresses (320 x 320, 4 units of 64 channels, ws 7: dq 464 -> 313 us, dk/dv
// 588 -> 435, forward 281 -> 249, apply 196 -> 178; a fifth to a third of each).
#define CA_PIPE_LOOP(...)                                                                            \
    bool s_err = false;                                                                              \
    int buf = 0;                                                                                     \
    uint32_t full_phase = 0;                                                                         \
    for (int s = s_begin; s < s_end; ++s) {                                                          \
        const bool lost = !mbar_wait(pipe.bar(buf), full_phase, a.wait_tries);                       \
        __VA_ARGS__                                                                                  \
        s_err = part_any(part, PT, lost);                                                            \
        if (s_err) break;                                                                            \
        if (lt == 0 && s + a.nstages < s_end) pipe.issue(buf, a, &mv, &msc, ROWS, u, h0);                \
        if (++buf == a.nstages) { buf = 0; full_phase ^= 1; }                                        \
    }                                                                                                \
    s_err = __syncthreads_or(s_err);                                                                 \
    /* A wait that ran out: the CTA stops computing, reports (device counter, caller's status word)  \
       and poisons what it still stores with NaN, so that the failure cannot pass for a result. */   \
    float ca_poison = 0.f;                                                                           \
    if (s_err) {                                                                                     \
        /* give copies still in flight a bounded chance to land before the CTA exits */              \
        if (lt == 0)                                                                                 \
            for (int i = 0; i < a.nstages; ++i) mbar_wait(pipe.bar(i), 0, 1u << 12);               \
        if (threadIdx.x == 0) {                                                                      \
            atomicAdd(a.timeouts, 1);                                                         \
            if (a.status) atomicOr(a.status, 1);                                                     \
        }                                                                                            \
        ca_poison = __int_as_float(0x7fc00000);                                                      \
    }

// One real element of a dense tensor stored as Float32 or bfloat16 (element offset `off`).
// BF is a compile-time flag so that a batch of loads stays a batch of independent loads; callers
// branch once on Geo::bf16 around the whole batch.
template <bool BF>
__device__ __forceinline__ float ld_real(const float* base, int64_t off) {
    if (BF) {
        const unsigned short h = __ldg(reinterpret_cast<const unsigned short*>(base) + off);
        return __uint_as_float((unsigned)h << 16);
    }
    return __ldg(base + off);
}
template <bool BF>
__device__ __forceinline__ void st_real(float* base, int64_t off, float v) {
    if (BF) reinterpret_cast<__nv_bfloat16*>(base)[off] = __float2bfloat16_rn(v);
    else base[off] = v;
}

// The sweeps are compiled twice (the *_exact.cu and *_any.cu files): for units whose real channels are exactly the 8, 16,
// 32 or 64 of a kernel, where the plane offsets are multiples of one product, and for every other count, which is read
// from the geometry and zero-extended.  One kernel for both made the 64-channel dk/dv sweep, whose tiles are short at small
// windows, a fifth slower (1.11 against 1.35 ms at 320 x 320, 8 units, window 7).
#ifndef CA_ANY_CHANNELS
#define CA_ANY_CHANNELS 1
#endif
constexpr bool kAnyC = CA_ANY_CHANNELS != 0;

// Runs the statements once with `constexpr bool BF` (bfloat16 storage) and `constexpr int NCRV` (the unit's channel
// count, 0: read it from the geometry): one uniform branch around a whole epilogue instead of one per element.
// Needs CPE, NCRT and g in scope.
#define CA_OUT_DISPATCH(...)                                       \
    if constexpr (kAnyC) {                                         \
        constexpr bool BF = false;                                 \
        constexpr int NCRV = 0;                                    \
        __VA_ARGS__                                                \
    } else if constexpr (NCRT > 16) {                              \
        constexpr bool BF = false;                                 \
        constexpr int NCRV = NCRT;                                 \
        __VA_ARGS__                                                \
    } else {                                                       \
        if (g.cr == 8) {                                           \
            constexpr int NCRV = 8;                                \
            if (CPE == 1 && g.bf16) {                              \
                constexpr bool BF = true;                          \
                __VA_ARGS__                                        \
            } else {                                               \
                constexpr bool BF = false;                         \
                __VA_ARGS__                                        \
            }                                                      \
        } else {                                                   \
            constexpr int NCRV = 16;                               \
            if (CPE == 1 && g.bf16) {                              \
                constexpr bool BF = true;                          \
                __VA_ARGS__                                        \
            } else {                                               \
                constexpr bool BF = false;                         \
                __VA_ARGS__                                        \
            }                                                      \
        }                                                          \
    }

// Whether centre column w0 + r of row h holds a pixel (the last column of a folded 1-D signal may be shorter; such
// signals take the kernels compiled for any channel count: the test costs the 64-channel dk/dv sweep 7 %).
__device__ __forceinline__ bool has_pixel(const Geo& g, int h, int w) {
    return w < g.W && (!kAnyC || g.wsw != 1 || h + g.H * w < g.Np);
}

// Loads the 16-channel vectors of the NQ centre pixels of this thread, times `mul`; channels past the unit's are zero.
// Every load is issued, from a clamped address where there is nothing to load, and the value dropped afterwards.
template <int CPE, int NQ>
__device__ __forceinline__ void load_centre_any(const float* src, const Geo& g, int u, int h, int w0, bool active,
                                                 float mul, u64 (&dst)[NQ][8], int ch0) {
    float2 raw[NQ][8];
    uint32_t po[NQ];                                     // element offset of the pixel inside a plane
#pragma unroll
    for (int r = 0; r < NQ; ++r) po[r] = CPE * (active && has_pixel(g, h, w0 + r) ? (uint32_t)(h + g.H * (w0 + r)) : 0u);
    const int64_t plane = (int64_t)CPE * g.Np;           // elements from one channel (complex: pair) to the next
    int64_t o = goff<CPE>(u, g.cr, min(ch0, g.cr - CPE), g.Np, 0);
#pragma unroll
    for (int e = 0; e < 16; e += CPE) {
#pragma unroll
        for (int r = 0; r < NQ; ++r) {
            if (CPE == 2) raw[r][e / 2] = __ldg(reinterpret_cast<const float2*>(src + o + po[r]));
            else if (e & 1) raw[r][e / 2].y = ld_real<false>(src, o + po[r]);
            else raw[r][e / 2].x = ld_real<false>(src, o + po[r]);
        }
        o += ch0 + e + CPE < g.cr ? plane : 0;
    }
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        const bool ok = active && has_pixel(g, h, w0 + r);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int cc = ch0 + 2 * i;
            dst[r][i] = pack2(ok && cc < g.cr ? raw[r][i].x * mul : 0.f, ok && cc + 1 < g.cr ? raw[r][i].y * mul : 0.f);
        }
    }
}

// The unit has exactly NCR channels: constant plane offsets.
template <int CPE, int NQ, int NCR, bool BF>
__device__ __forceinline__ void load_centre_exact(const float* src, const Geo& g, int u, int h, int w0, bool active,
                                                  float mul, u64 (&dst)[NQ][8], int ch0) {
#pragma unroll
    for (int r = 0; r < NQ; ++r) {
        const bool ok = active && has_pixel(g, h, w0 + r);
        const int pix = h + g.H * (w0 + r);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float x = 0.f, y = 0.f;
            if (ok && (NCR >= 16 || 2 * i < NCR)) {
                if (CPE == 1) {
                    x = ld_real<BF>(src, goff_exact<1, NCR>(u, ch0 + 2 * i, g.Np, pix));
                    y = ld_real<BF>(src, goff_exact<1, NCR>(u, ch0 + 2 * i + 1, g.Np, pix));
                } else {
                    const float2 t = __ldg(reinterpret_cast<const float2*>(src + goff_exact<2, NCR>(u, ch0 + 2 * i, g.Np, pix)));
                    x = t.x;
                    y = t.y;
                }
            }
            dst[r][i] = pack2(x * mul, y * mul);
        }
    }
}

template <int CPE, int NQ, int NCRT>
__device__ __forceinline__ void load_centre(const float* src, const Geo& g, int u, int h, int w0, bool active,
                                            float mul, u64 (&dst)[NQ][8], int ch0 = 0) {
    if constexpr (kAnyC) {
        load_centre_any<CPE, NQ>(src, g, u, h, w0, active, mul, dst, ch0);
    } else if constexpr (NCRT > 16) {
        load_centre_exact<CPE, NQ, NCRT, false>(src, g, u, h, w0, active, mul, dst, ch0);
    } else {
        if (g.cr == 8) {
            if (CPE == 1 && g.bf16) load_centre_exact<CPE, NQ, 8, true>(src, g, u, h, w0, active, mul, dst, ch0);
            else load_centre_exact<CPE, NQ, 8, false>(src, g, u, h, w0, active, mul, dst, ch0);
        } else {
            if (CPE == 1 && g.bf16) load_centre_exact<CPE, NQ, 16, true>(src, g, u, h, w0, active, mul, dst, ch0);
            else load_centre_exact<CPE, NQ, 16, false>(src, g, u, h, w0, active, mul, dst, ch0);
        }
    }
}

// NCR: the unit's channel count, or 0: take it from the geometry.
template <int CPE, int NCR, bool BF = false>
__device__ __forceinline__ void store_centre(float* dst, const Geo& g, int u, int h, int w0, bool active, int r,
                                             int i, float x, float y, int ch0 = 0) {
    const int cc = ch0 + 2 * i;
    if (!(active && has_pixel(g, h, w0 + r))) return;
    if (NCR == 0 ? cc >= g.cr : (NCR < 16 && 2 * i >= NCR)) return;
    const int pix = h + g.H * (w0 + r);
    const int64_t o = NCR ? goff_exact<CPE, NCR ? NCR : 16>(u, cc, g.Np, pix)
                          : goff<CPE>(u, g.cr, ch0, g.Np, pix) + (int64_t)(2 * i) * g.Np;
    if (CPE == 1) {
        st_real<BF>(dst, o, x);
        if (NCR) st_real<BF>(dst, goff_exact<1, NCR ? NCR : 16>(u, cc + 1, g.Np, pix), y);
        else if (cc + 1 < g.cr) st_real<BF>(dst, o + g.Np, y);
    } else {
        *reinterpret_cast<float2*>(dst + o) = make_float2(x, y);
    }
}

// MASK != 0: all centre pixels pair with this stage (compile time);
// MASK == 0: the set is the run-time `rm` (warp-uniform branches).
#define CA_ON(r) ((MASK != 0) || ((rm >> (r)) & 1))


// 16-channel slabs of a packed pixel row: 1, 2 or 4 (the channels past the unit's are zero).
inline int slabs_of(const Geo& g) { return g.cr <= 16 ? 1 : (g.cr <= 32 ? 2 : 4); }

// Whether the forward keeps the rows of A in shared memory and writes them itself: up to 11.6 KB per warp and column, past which
// too few warps are left on an SM.  Forward and values in one kernel against two: 320 x 320, 8 units of 64 channels,
// ws 7 (1.6 KB): 565 and 867 us; 150 x 140, 4 of 32, ws 11 (7.7 KB): 104 and 130; 100 x 100, 2 of 64, ws 19 (11.6 KB): 156
// and 197; 128 x 96, 8 of 16, ws 9 (10.4 KB): 55 and 67; 128 x 96, 4 of 32, ws 15 (14.4 KB): 115 and 109; 128 x 96, 8 of
// 16, ws 11 (15.5 KB): 85 and 72; folded signals 8192 x 64 x 4, ws 63 (2 KB): 60 and 95.
inline bool values_fit(const Geo& g, int ns) { return 32 / ns * g.K * 4 <= 11600; }

// Words of the weights (P and dS) that the backward of wide units keeps between its dq and dk/dv sweeps; 0: dk/dv recomputes them.
// 33 to 64 real channels: at 32 the weights cost as much to move as the contractions they save (150 x 140, 4 units, ws 11: 206
// and 211 us for both sweeps, 320 x 240, 4 units, ws 5: 210 and 195).  Windows whose weights take no more memory than the
// two packed pairs, and enough pixels to fill the chip: recomputing sweeps run side by side, which a few pixels need
// (40 x 40, 2 units, ws 7: 21 us side by side, 27 one after the other; 100 x 64, 6 units, ws 11: 246 and 211).
inline size_t weight_floats(const Geo& g) {
    if (slabs_of(g) != 4 || g.wsw != g.ws || g.Wk != g.W || g.K > 288 || (int64_t)g.Np * g.units < 20000) return 0;
    const size_t words = (size_t)2 * g.units * g.K * g.Np;
    return words <= ((size_t)1 << 28) ? words : 0;          // at most 1 GiB
}

inline bool exact_shape(const Geo& g) {
    return (g.cr == 8 || g.cr == 16 || g.cr == 32 || g.cr == 64) && (int64_t)g.H * g.W == g.Np;
}
#define CA_CHANNELS(g, FN, ...) (exact_shape(g) ? FN<false>(__VA_ARGS__) : FN<true>(__VA_ARGS__))

inline Padded padded_of(const Geo& g) {
    Padded P;
    P.pp = (g.p + 1) & ~1;
    P.Hp = (g.H + 2 * P.pp + 3) & ~3;
    P.pair_floats = (size_t)g.units * g.Wk * P.Hp * kRowFloats * slabs_of(g);
    P.single_floats = (size_t)g.units * g.Wk * P.Hp * kSingleFloats * slabs_of(g);
    P.plane_floats = (size_t)2 * g.units * g.Wk * P.Hp;
    return P;
}

inline bool tiled_window_ok(const Geo& g) {
    return (g.wsw == g.ws || g.wsw == 1) && g.ws >= 3 && g.H >= 16 && g.ws <= (g.wsw == 1 ? 127 : 63);
}

inline bool tiled_shape_ok(const Geo& g) {
    // up to 64 real channels per unit, zero-extended to 16, 32 or 64 (1, 2 or 4 lanes per pixel): at 12 channels the
    // FMAs spent on zeros are a quarter, the one-thread-per-pixel kernels take six times as long.  bfloat16 storage:
    // 8 or 16 channels.
    return (g.bf16 ? g.cr == 8 || g.cr == 16 : g.cr <= 64) && tiled_window_ok(g);
}

inline bool tiled_operator_ok(const Geo& g) { return g.cr <= 64 && tiled_window_ok(g) && g.Wk == g.W; }

// The geometry the tiled kernels run on.  2-D problems are taken as they are.  A 1-D signal of
// length N (H = N, W = 1) is folded column-major into columns of Hf pixels: pixel n = h + Hf*w keeps
// its address, its window is the rows h-p..h+p of its own column, and the halo rows of the packed
// columns continue into the neighbouring columns (the pack kernel fills them by linear index), so
// the 2-D kernels run unchanged with a window that is one column wide.  The last column may be shorter
// (Hf * W > Np): centre pixels past the signal are neither loaded nor stored.
inline bool fold_geo(const Geo& in, Geo* out) {
    *out = in;
    if (in.wsw == in.ws) return true;                      // 2-D
    if (in.wsw != 1 || in.Wk != in.W) return false;
    if (in.W != 1) return true;                            // already folded
    if (in.H < 16) return false;
    int hf = in.bf16 ? 0 : std::min(in.H, 128);            // bfloat16 storage exists in the kernels for exact shapes only
    for (int h : {128, 96, 64, 48, 32, 16}) {
        if (hf && h < 64) break;
        if (in.H % h == 0) { hf = h; break; }
    }
    if (!hf) return false;
    out->H = hf;
    out->W = out->Wk = (in.H + hf - 1) / hf;
    return true;
}

struct Launch {
    TileArgs a;
    CUtensorMap mv, msc;
    dim3 grid;
    int threads;
    size_t smem;
};

// How a sweep is cut into blocks: `nq` centre columns per thread, `warps` warps of pixel rows per block and `nsplit` groups
// of such warps that share the stages of a tile (warps * nsplit <= 4).
struct TileShape {
    int nq, warps, nsplit;
};

// What a sweep with `nq` columns per thread costs, in cycles: a window row takes a warp `lat` + `issue` for each warp on its
// scheduler, a stage `stage` more, a block `block`; an SM holds `sm_warps` warps of it.  Fitted to the measured times of
// 25 shapes (32 x 32 to 512 x 512, 1 to 16 units of 16, 32 and 64 channels, windows 5 to 21) in every cut; rms error of a
// predicted time 5 to 11 %.
struct SweepCost {
    int nq, sm_warps;
    float lat, issue, stage, block;
};

inline int tile_stage_bytes(int rows, int row_bytes, bool planes, bool single) {
    const int vbytes = (rows * row_bytes + 127) & ~127;
    return single ? vbytes : (vbytes + (planes ? 2 * ((rows * 4 + 127) & ~127) : 0) + 1023) & ~1023;
}

// The cut with the least predicted time.  What decides: rows of a tile past the image (75 rows are three warps, not two
// tiles of 64), whole waves of blocks, window rows left to a warp when the stages are shared, and few wide tiles
// against many narrow ones where a window is short or a grid small (a tile of nq columns streams ws + nq - 1).  Over the
// 25 shapes the choice is within 10 % of the best cut but for two.  Against four warps of rows and fixed columns:
// 75 x 53, 9 units, ws 11: forward 27 -> 21 us, dq 40 -> 24, dk/dv 66 -> 35; 128 x 96, 4 units of 64 channels, ws 15: dq
// 211 -> 160, dk/dv 262 -> 202; 32 x 32, 1 unit, ws 7: forward 8.0 -> 5.1, dq 10 -> 6, dk/dv 20 -> 6.8.
// `planes`: the stages carry the scalar planes; `single`: packed rows of one tensor; `col_bytes`: shared memory of a warp of
// rows for each centre column besides the stages, `warp_bytes` of every warp; `stages` copies in flight; `lone` weighs blocks of
// one warp within one wave.
inline TileShape search_tile(const Geo& g, const Padded& P, int ns, const SweepCost* cost, int n, int max_split, bool planes, bool single,
                             int col_bytes, int stages, int warp_bytes, float lone, int sm) {
    TileShape best{cost[0].nq, 1, 1};
    float least = INFINITY;
    const int rw = 32 / ns;                             // pixel rows per warp (ns lanes share a pixel)
    const float sms = (float)sm;
    for (const SweepCost* c = cost; c < cost + n; ++c) {
        const int nst = g.wsw + c->nq - 1;
        const float cols = (float)((g.W + c->nq - 1) / c->nq) * g.units;
        for (int w = 4; w >= 1; --w) {
            if (w > 1 && rw * (w - 1) >= g.H) continue;
            const int stage = tile_stage_bytes(rw * w + 2 * P.pp, (single ? kSingleFloats : kRowFloats) * 4 * ns, planes, single);
            const int rows_bytes = w * c->nq * col_bytes;
            const float blocks = cols * ((g.H + rw * w - 1) / (rw * w));
            for (int s = 1; w * s <= 4 && s <= max_split && s <= nst; ++s) {
                const int own = rows_bytes + w * s * warp_bytes;
                if (s * 2 * stage + own > 216 * 1024) break;        // not even two copies in flight
                const int resident = std::max(1, std::min(c->sm_warps / (w * s), 227 * 1024 / (s * stages * stage + own + 2048)));
                const float waves = blocks / (resident * sms);
                // warps per scheduler, and how many times a block's time passes: whole waves while there are few (the
                // blocks of a wave end together), later half a wave is lost at the end
                const float k = waves <= 1.f ? std::ceil(std::ceil(blocks / sms) * (w * s) / 4) : std::max(1.f, resident * (w * s) / 4.f);
                const float turns = waves <= 2.f ? std::ceil(waves) : std::min(std::ceil(waves), waves + 0.5f);
                float t = turns * (((nst + s - 1) / s) * (g.ws * (c->lat + c->issue * k) + c->stage) + c->block);
                // tiles of one or two warps copy more halo rows; it shows once blocks follow one another (the forward
                // at 500 x 400, 3 units, ws 11: 209 us with one warp, 172 with two, 167 with four)
                if (waves > 1.f) t *= w == 1 ? 1.08f : (w == 2 ? 1.02f : 1.f);
                else if (w * s == 1) t *= lone;
                if (t < least) { least = t; best = TileShape{c->nq, w, s}; }
            }
        }
    }
    return best;
}

// The search takes about a microsecond of a launch's three: a thread keeps the cuts of its last launches.
inline TileShape choose_tile(const Geo& g, const Padded& P, int ns, const SweepCost* cost, int n, int max_split, bool planes = false,
                             bool single = false, int col_bytes = 0, int stages = kStages, int warp_bytes = 0, float lone = 1.f) {
    struct Key {
        const SweepCost* cost;
        int v[14];
        bool operator==(const Key& o) const { return cost == o.cost && std::equal(v, v + 14, o.v); }
    };
    struct Entry { Key key; TileShape shape; };
    static thread_local Entry kept[16] = {};
    const int sm = sm_count();
    const Key key{cost, {g.H, g.W, g.units, g.ws, g.wsw, P.pp, ns, n, max_split, planes * 2 + single, col_bytes, stages, warp_bytes * 4 + (lone < 1.f), sm}};
    unsigned h = (unsigned)(reinterpret_cast<uintptr_t>(cost) >> 4);
    for (int x : key.v) h = h * 31u + (unsigned)x;
    Entry& e = kept[h % 16];
    if (!(e.key == key)) e = Entry{key, search_tile(g, P, ns, cost, n, max_split, planes, single, col_bytes, stages, warp_bytes, lone, sm)};
    return e.shape;
}

// The apply runs of folded signals, and of windows whose runs fill the shared memory: `max_warps` warps of rows; fewer than 6
// warps per SM share the stages of a tile (in four where the kernel can, in two up to 12 warps per SM).
inline TileShape operator_tile(const Geo& g, int ns, int nq, int max_split, int max_warps) {
    const int rw = 32 / ns;
    const int warps = std::min(max_warps, (g.H + rw - 1) / rw);
    const long tasks = (long)((g.W + nq - 1) / nq) * ((g.H + rw * warps - 1) / (rw * warps)) * g.units * warps;
    int nsplit = max_split == 4 ? (tasks < 6L * sm_count() ? 4 : (tasks < 12L * sm_count() ? 2 : 1)) : (tasks < 6L * sm_count() ? 2 : 1);
    nsplit = std::min(nsplit, max_split);
    return TileShape{nq, warps * nsplit > 4 ? 4 / nsplit : warps, nsplit};
}

// Fills the launch geometry and the tensor maps of the packed pair (and of the scalar planes when given).
// `xch_floats` per thread for the merge of a split tile; `extra` bytes of the kernel's own.
inline int prepare(const Geo& g, const Padded& P, TileShape t, int xch_floats, const float* pair, const float* planes, Launch* L,
                   int ns, bool single = false, int stages = kStages, size_t extra = 0) {
    const int rw = 32 / ns, warps = t.warps, nsplit = t.nsplit;
    const int rf = (single ? kSingleFloats : kRowFloats) * ns, rb = rf * 4;
    TileArgs& a = L->a;
    a.g = g;
    a.status = status_word();
    if (!(a.timeouts = stage_timeout_counter())) return cuda_fail(cudaGetLastError(), "cudaGetSymbolAddress(stage timeouts)");
    a.wait_tries = kWaitTries;
    a.TH = rw * warps;
    a.roff = P.pp - g.p;
    a.nsplit = nsplit;
    a.row_bytes = rb;
    const int ROWS = a.TH + 2 * P.pp;
    if (ROWS > 256) { set_error("tile of %d rows exceeds the TMA box limit", ROWS); return CA_ERR_UNSUPPORTED; }
    a.stage_bytes = tile_stage_bytes(ROWS, rb, planes != nullptr, single);
    L->grid = dim3((unsigned)((g.W + t.nq - 1) / t.nq), (g.H + a.TH - 1) / a.TH, g.units);
    L->threads = 32 * warps * nsplit;
    // long windows of wide units: two copies in flight where three do not fit
    if (stages > 2 && (size_t)nsplit * stages * a.stage_bytes > 216 * 1024) stages = 2;
    a.nstages = stages;
    size_t smem = (size_t)nsplit * stages * a.stage_bytes;
    const size_t xch = (size_t)(nsplit - 1) * xch_floats * 32 * warps * sizeof(float);
    if (xch > smem) smem = xch;
    a.extra_off = (int)smem;
    smem += extra;
    L->smem = smem + 1024;
    if (L->smem > kMaxDynamicSmem) return CA_ERR_UNSUPPORTED;     // window too large for the stage ring: generic kernels
    const uint64_t dims[4] = {(uint64_t)rf, (uint64_t)P.Hp, (uint64_t)g.Wk, (uint64_t)g.units};
    const uint64_t strides[3] = {(uint64_t)rb, (uint64_t)P.Hp * rb, (uint64_t)P.Hp * rb * g.Wk};
    const uint32_t box[4] = {(uint32_t)rf, (uint32_t)ROWS, 1, 1};
    int rc;
    if ((rc = encode_tensor_map(&L->mv, pair, 4, dims, strides, box))) return rc;
    if (planes) {
        const uint64_t sdims[3] = {(uint64_t)P.Hp, (uint64_t)g.Wk, (uint64_t)2 * g.units};
        const uint64_t sstr[2] = {(uint64_t)P.Hp * 4, (uint64_t)P.Hp * 4 * g.Wk};
        const uint32_t sbox[3] = {(uint32_t)ROWS, 1, 1};
        if ((rc = encode_tensor_map(&L->msc, planes, 3, sdims, sstr, sbox))) return rc;
    } else {
        L->msc = L->mv;
    }
    return CA_OK;
}

// Raises a kernel's limit of dynamic shared memory to the most that any launch asks for (prepare()), once per kernel and
// device: `have` remembers the device of the last call.  Always the same value, so threads cannot lower each other's.
template <typename K>
int set_smem(K kernel, size_t bytes, std::atomic<int>& have) {
    if (bytes <= 47 * 1024) return CA_OK;   // the default limit of 48 KB counts the kernel's static shared memory too
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && have.load(std::memory_order_relaxed) == dev + 1) return CA_OK;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(shared memory)");
    have.store(dev + 1, std::memory_order_relaxed);
    return CA_OK;
}

#define CA_LAUNCH_TILED(KERNEL, L, st)                                                \
    do {                                                                              \
        static std::atomic<int> have__{0};                                            \
        int rc__ = set_smem(KERNEL, (L).smem, have__);                                \
        if (rc__) return rc__;                                                        \
        KERNEL<<<(L).grid, (L).threads, (L).smem, st>>>((L).a, (L).mv, (L).msc);      \
        count_tiled_launch();                                                         \
    } while (0)

#define CA_DIST_CPE_NQ(KERNEL_T, dist, cpe, NQV, XV, NCRV_, L, st)                    \
    do {                                                                              \
        if ((cpe) == 1) {                                                             \
            if (dist) CA_LAUNCH_TILED((KERNEL_T<true, 1, NQV, XV, NCRV_>), L, st);    \
            else CA_LAUNCH_TILED((KERNEL_T<false, 1, NQV, XV, NCRV_>), L, st);        \
        } else {                                                                      \
            if (dist) CA_LAUNCH_TILED((KERNEL_T<true, 2, NQV, XV, NCRV_>), L, st);    \
            else CA_LAUNCH_TILED((KERNEL_T<false, 2, NQV, XV, NCRV_>), L, st);        \
        }                                                                             \
    } while (0)

}  // namespace
}  // namespace ca
