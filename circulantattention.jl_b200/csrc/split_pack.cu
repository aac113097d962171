// Pack kernel of the tensor-core sweeps (split.cuh has the layout): two tensors in the reference layout -> rows of split halves
// with the circular halo unrolled, the scales of each group of eight rows and the rows' scalars.
#include "split.cuh"

namespace ca {
namespace {

// Whether the halves would lose bits of a whole row of the lane's group of eight (`small`) or of a whole channel of it (`channels`: of few
// rows that are not zero, as at the end of a column, a channel may be any small numbers).
__device__ __forceinline__ bool marked(const float (&x)[16], bool small, bool channels, float inv, float least) {
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        uint32_t c = abs_bits(x[e]);
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) c = max(c, __shfl_xor_sync(0xffffffffu, c, d));
        small |= channels && c >= kLeastNormal && __uint_as_float(c) * inv < least;
    }
    return __ballot_sync(0xffffffffu, small) >> (threadIdx.x & 24) & 255u;
}

// How far the rows of a group may be apart, in the bits of a float: 2^6, since the bound of the gradients' weights is the group's and
// windows of 9 rows fit between lines that leave no group without a large row (57 x 54, 4 units, ws 9, every 12th row of dy and v times 3000:
// dq between them 3.1e-5 off without this, 3.4e-7 with it, FMA pipe 4.9e-7).  Rows of two and three channels may be any small numbers
// more often, and give only what the halves need; those of one channel nothing.
__device__ __forceinline__ uint32_t row_span(int channels) { return channels >= 4 ? 6u << 23 : channels > 1 ? 13u << 23 : 0x7f000000u; }

// A block gathers 128 packed rows of one column of one unit: a thread reads the 16 channels of its row of both tensors
// (consecutive lanes on consecutive rows: coalesced planar loads, all in flight together), the largest magnitude of each
// group of eight rows comes from shuffles, and the block writes its rows as one contiguous run of 16-byte stores.  Bound: HBM.
template <int CPE, bool BF>
__global__ void __launch_bounds__(128, 6) split_pack_kernel(SplitPackArgs a) {
    constexpr bool LO = !BF;
    constexpr int RB = 128, RF = split_row_bytes(LO) / 4;
    __shared__ __align__(16) uint32_t tile[RB * RF];
    const Geo& g = a.g;
    const int rl = threadIdx.x, rr0 = blockIdx.x * RB, rr = rr0 + rl, w = blockIdx.y, u = blockIdx.z;
    const bool real_row = rr < g.H + 2 * g.p;
    const int pix = real_row ? (rr - g.p + g.H) % g.H + g.H * w : 0;
    float x[2][16];
    float dot = 0.f;
    {
        // all loads first, from clamped addresses
        const float* src[2] = {a.x0, a.x1};
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < 16; e += CPE) {
                const int64_t o = goff<CPE>(u, g.cr, min(e, g.cr - CPE), g.Npk, pix);
                if (CPE == 2) {
                    const float2 z = __ldg(reinterpret_cast<const float2*>(src[t] + o));
                    x[t][e] = z.x;
                    x[t][e + CPE - 1] = z.y;
                } else {
                    x[t][e] = ld_real<BF>(src[t], o);
                }
            }
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < 16; ++e)
                if (!real_row || e >= g.cr) x[t][e] = 0.f;
        if (a.y) {
            float yv[16];
#pragma unroll
            for (int e = 0; e < 16; e += CPE) {
                const int64_t o = goff<CPE>(u, g.cr, min(e, g.cr - CPE), g.Npk, pix);
                if (CPE == 2) {
                    const float2 z = __ldg(reinterpret_cast<const float2*>(a.y + o));
                    yv[e] = z.x;
                    yv[e + CPE - 1] = z.y;
                } else {
                    yv[e] = ld_real<BF>(a.y, o);
                }
            }
#pragma unroll
            for (int e = 0; e < 16; ++e)
                if (e < g.cr) dot = fmaf(x[1][e], yv[e], dot);
            if (!real_row) dot = 0.f;
        }
    }
    float2 n2 = make_float2(0.f, 0.f);
#pragma unroll
    for (int e = 0; e < 16; e += 2) {
        n2.x = fmaf(x[0][e], x[0][e], n2.x);
        n2.y = fmaf(x[0][e + 1], x[0][e + 1], n2.y);
    }
    const float norm = n2.x + n2.y;
    uint32_t exps = 0;
    uint32_t* row = tile + rl * RF;
    int ex[2];
    float inv[2];
    bool small[2], channels[2], look = false;
    const uint32_t span = row_span(g.cr);
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        uint32_t m = 0;
        float low = INFINITY;
#pragma unroll
        for (int e = 0; e < 16; ++e) m = max(m, abs_bits(x[t][e]));
#pragma unroll
        for (int e = 0; e < 16; e += 2)
            if (e < g.cr) low = min3(low, fabsf(x[t][e]), e + 1 < g.cr ? fabsf(x[t][e + 1]) : INFINITY);
        const uint32_t mine = m;
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
        ex[t] = m ? scale_exp(m, 4, t == 0 ? kLeastExp : 0) : 0;
        inv[t] = exp_inverse(ex[t] == 255 ? 0 : ex[t]);
        // a row far below the group's largest, or a group below the least scale
        small[t] = mine >= kLeastNormal && (mine + span < m || __uint_as_float(m) * inv[t] < 64.f * least_value(LO));
        // a channel of small numbers has one in all eight rows, which is rare
        const uint32_t rows = __ballot_sync(0xffffffffu, low * inv[t] < least_value(LO)) >> (rl & 24) & 255u;
        const uint32_t filled = __ballot_sync(0xffffffffu, mine) >> (rl & 24) & 255u;
        channels[t] = rows == 255u && __popc(filled) >= 4;
        look |= small[t] || channels[t];
    }
    if (__any_sync(0xffffffffu, look)) {
#pragma unroll
        for (int t = 0; t < 2; ++t)
            if (marked(x[t], small[t], channels[t], inv[t], least_value(LO))) ex[t] = 255;
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        exps |= (uint32_t)ex[t] << (8 * t);
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) split2(x[t][2 * i] * inv[t], x[t][2 * i + 1] * inv[t], hi[i], lo[i]);
        uint4* d = reinterpret_cast<uint4*>(row + t * (split_second(LO) / 4));
        d[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        d[1] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
        if (LO) {
            d[2] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            d[3] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
        }
    }
    float A = a.norm_mul * norm;
    if (a.stats) {
        const int64_t so = (int64_t)u * g.Npk + pix;
        if (real_row) {
            A = fmaf(__ldg(a.stats + so), -kLog2e, A);
            if (a.Din) dot = __ldg(a.Din + so);
            else if (a.Dout && rr >= g.p && rr < g.p + g.H) a.Dout[so] = dot;
        }
        uint32_t m = abs_bits(dot);
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
        // a power of two above every |D| of the group; a statistic that is no number marks it, too
        uint32_t bad = abs_bits(A) >= 0x7f800000u;
        bad = __ballot_sync(0xffffffffu, bad) >> (rl & 24) & 255u;
        const uint32_t e = bad || m >= 0x7e800000u ? 255u : (m >> 23) + (m ? 1u : 0u);
        exps |= e << 16;
    }
    const float A1 = __shfl_xor_sync(0xffffffffu, A, 1), dot1 = __shfl_xor_sync(0xffffffffu, dot, 1);
    const uint4 odd = make_uint4(exps, 0u, __float_as_uint(-dot1), __float_as_uint(-dot));
    *reinterpret_cast<uint4*>(row + split_scalars(LO) / 4) = rl & 1 ? odd : make_uint4(exps, 0u, __float_as_uint(A), __float_as_uint(A1));
    __syncthreads();
    const int nrows = min(RB, a.Hp - rr0);
    uint4* out = reinterpret_cast<uint4*>(a.dst + (((int64_t)u * g.Wk + w) * a.Hp + rr0) * RF);
    const uint4* tin = reinterpret_cast<const uint4*>(tile);
    for (int i = threadIdx.x; i < nrows * (RF / 4); i += 128) out[i] = tin[i];
}

}  // namespace

// Whether the tiles of 32 rows of the FMA kernels leave a sixteenth of their lanes idle on this image.
static bool idle_rows(const Geo& g) { return 16 * ((32 - g.H % 32) % 32) >= g.H; }

// Units of one slab (more channels would need their results in registers for 32 or 64 channels), windows up to 25 (four tiles a
// column), and enough pixels to fill the chip: 12000 is on the safe side (forward and backward on the FMA pipe and here, us: 64 x 64, 2
// units, ws 9: 33 and 31, ws 21: 65 and 52).
// dk/dv from window 9 on, in bfloat16 from 7; in Float32 at 7 where the FMA kernels have idle rows and up to 2^18 pixels.  What a warp
// spends outside its steps, and the scores outside the window, weigh more the shorter it is.  Backward with the FMA pipe's dk/dv and
// with this one (dq on the FMA pipe), us: ws 7: 200 x 180, 4 units 104 and 99, 97 x 400, 4 units 119 and 114, 256 x 256, 4 units 152 and 158,
// 500 x 400, 8 units 814 and 837; bfloat16: 256 x 256, 4 units 158 and 143, 512 x 512, 8 units 1092 and 1011; ws 9: 256 x 256, 4 units 200
// and 186, 512 x 512, 8 units 1379 and 1307; ws 11: 260 and 248, 1808 and 1803; ws 13: 346 and 297, 2317 and 2127.
bool split_dkdv_ok(const Geo& g, float scale) {
    const int64_t pixels = (int64_t)g.Np * g.units;
    return tiled_shape_ok(g) && g.wsw == g.ws && slabs_of(g) == 1 && split_tiles(g) <= 4 && scale > 0.f && g.Wk <= 65535 && pixels > 12000 &&
           (g.ws >= 9 || (g.ws == 7 && (g.bf16 || (idle_rows(g) && pixels <= (1 << 18)))));
}

// Forward, A's values and dq, which share the packed (k|v): from window 13 on, in bfloat16 from 9; in Float32 at 9 and 11 where the FMA
// kernels have idle rows.  Forward on the FMA pipe and here, us: ws 9: 256 x 256, 4 units (no idle rows) 73 and 76, 500 x 400, 8 units
// (2 %) 361 and 378, 1001 x 300, 4 units (2 %) 277 and 288, 240 x 240, 4 units (7 %) 73 and 68, 257 x 255, 4 units (12 %) 84 and 81,
// 200 x 180, 4 units (12 %) 55 and 46; ws 11: 93 and 97, 467 and 509, 357 and 387, -, 109 and 104, 72 and 62; ws 13: 113 and 107, 578 and
// 561, 441 and 427, -, 134 and 113, 87 and 67; bfloat16, ws 9: 71 and 63, 363 and 326, 280 and 249, -, 82 and 67, 54 and 40.
bool split_shape_ok(const Geo& g, float scale) {
    return split_dkdv_ok(g, scale) && (g.ws >= 13 || (g.ws >= 9 && (g.bf16 || idle_rows(g))));
}

int launch_split_pack(const Geo& g, float scale, int dist, const float* x0, const float* x1, const float* stats, const float* y, const float* Din,
                      float* Dout, float* dst, cudaStream_t st) {
    SplitPackArgs a{};
    a.g = g; a.Hp = split_hp(g); a.x0 = x0; a.x1 = x1; a.stats = stats; a.y = y; a.Din = Din; a.Dout = Dout; a.dst = dst;
    a.norm_mul = dist ? -0.5f * scale * kLog2e : 0.f;
    const dim3 grid((a.Hp + 127) / 128, g.Wk, g.units);
    if (g.bf16) split_pack_kernel<1, true><<<grid, 128, 0, st>>>(a);
    else if (g.cpe == 1) split_pack_kernel<1, false><<<grid, 128, 0, st>>>(a);
    else split_pack_kernel<2, false><<<grid, 128, 0, st>>>(a);
    CA_CHECK_LAUNCH("split pack kernel");
    return CA_OK;
}

}  // namespace ca
