// Pack kernels of the tiled family, the tensor-map encoder and the bounded-wait bookkeeping.
#include "tile_common.cuh"

namespace ca {
namespace {

// Number of CTAs that gave up waiting for a stage copy (stays 0 in a healthy run).
__device__ int g_stage_timeouts = 0;

// =====================================================================
// Pack kernel: NT = 2 tensors (a pair) or 1 in the reference layout -> packed rows
// [unit][column][row'][36 or 20 words per slab] with the circular halo along h unrolled, plus (optionally, pairs) the
// two scalar planes [2*unit + {0: stats*stat_mul, 1: D}][column][row'].
//
// A block gathers RB = 128 / NS packed rows of one (column, unit, pair): thread (row, slab) reads the 16 channels of its
// slab of every tensor (consecutive lanes on consecutive rows: coalesced planar loads, all in flight together) into a
// shared tile in the packed order [tensor][4-channel chunk][slab][4], and the block writes the tile out as one
// contiguous run of 16-byte stores.  Bound: HBM.  Writing 16*NS-byte pieces from the threads instead reaches half
// the bandwidth (single tensor of 64 channels, 320 x 320, 8 units, 210 MB: 158 us).
// Channels past the unit's are zero.  z slots: one per pair and unit, plus one for the planes.
// =====================================================================
// NCR: the unit's channel count, or 0: read it from the geometry.
template <int CPE, int NS, int NT, int NCR, bool BF>
__device__ __forceinline__ void pack_rows_body(const PackArgs& a, float* tile) {
    constexpr int RB = 128 / NS, RF = (NT == 2 ? kRowFloats : kSingleFloats) * NS;
    const Geo& g = a.g;
    const int rl = threadIdx.x % RB, slab = threadIdx.x / RB;
    const int rr0 = blockIdx.x * RB, rr = rr0 + rl;
    const int w = blockIdx.y;
    const int slots = a.npairs + (a.planes ? 1 : 0);
    const int u = blockIdx.z / slots, slot = blockIdx.z % slots;
    const bool in_rows = rr < a.Hp;
    const bool real_row = in_rows && rr < g.H + 2 * a.pp;
    // source pixel of packed row rr: the halo rows wrap inside the column (2-D) or continue into the neighbouring
    // columns of a folded 1-D signal
    int pix = 0;
    if (real_row) {
        if (g.wsw == 1) {
            pix = (g.H * w + rr - a.pp) % g.Npk;
            if (pix < 0) pix += g.Npk;
        } else {
            pix = (rr - a.pp + g.H) % g.H + g.H * w;
        }
    }
    if (slot < a.npairs) {
        float4* trow = reinterpret_cast<float4*>(tile + rl * RF);
        float vals[NT][16];
        const int cr = NCR ? NCR : g.cr;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const float* src = a.src[NT * slot + t];
            if (BF) {
                // all loads first, from clamped addresses: under conditions each 16-bit load is waited for (455 against
                // 312 us at 1024 x 1024, 8 units)
                int64_t o = goff<CPE>(u, cr, 0, g.Npk, pix);
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    vals[t][e] = ld_real<BF>(src, o);
                    o += e + 1 < cr ? (int64_t)g.Npk : 0;
                }
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (!real_row || e >= cr) vals[t][e] = 0.f;
            } else {
#pragma unroll
                for (int e = 0; e < 16; e += CPE) {
                    const int cc = 16 * slab + e;
                    const bool ok = real_row && (NCR >= 16 || cc < cr);
                    vals[t][e] = vals[t][e + CPE - 1] = 0.f;
                    if (CPE == 1) {
                        if (ok) vals[t][e] = __ldg(src + goff<1>(u, cr, cc, g.Npk, pix));
                    } else if (ok) {
                        const float2 z = __ldg(reinterpret_cast<const float2*>(src + goff<2>(u, cr, cc, g.Npk, pix)));
                        vals[t][e] = z.x;
                        vals[t][e + CPE - 1] = z.y;
                    }
                }
            }
        }
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int c = 0; c < 4; ++c) trow[t * (4 * NS) + c * NS + slab] = make_float4(vals[t][4 * c], vals[t][4 * c + 1], vals[t][4 * c + 2], vals[t][4 * c + 3]);
        float2 norm = make_float2(0.f, 0.f);               // squared, of the first tensor, for the Distance sweeps
#pragma unroll
        for (int e = 0; e < 16; e += 2) {
            norm.x = fmaf(vals[0][e], vals[0][e], norm.x);
            norm.y = fmaf(vals[0][e + 1], vals[0][e + 1], norm.y);
        }
        trow[4 * NT * NS + slab] = make_float4(norm.x + norm.y, 0.f, 0.f, 0.f);         // padding words
        __syncthreads();
        const int nrows = min(RB, a.Hp - rr0);
        float4* out = reinterpret_cast<float4*>(a.dst[slot] + (((int64_t)u * g.Wk + w) * a.Hp + rr0) * RF);
        const float4* tin = reinterpret_cast<const float4*>(tile);
        for (int i = threadIdx.x; i < nrows * (RF / 4); i += 128) out[i] = tin[i];
        return;
    }
    // scalar planes: L and D = dy . y (or the given D); every thread sums its slab's 16 channels
    float part = 0.f;
    if (real_row && !a.Din) {
        const int cr = NCR ? NCR : g.cr;
        float dyv[16], yv[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const int64_t o = goff<CPE>(u, cr, NCR >= 16 ? 16 * slab + e : min(16 * slab + e, cr - 1), g.Npk, pix);
            dyv[e] = ld_real<BF>(a.dy, o);
            yv[e] = ld_real<BF>(a.y, o);
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) part = fmaf(16 * slab + e < cr ? dyv[e] : 0.f, yv[e], part);
    }
    if (NS > 1) {
        tile[rl * NS + slab] = part;
        __syncthreads();
        if (slab != 0) return;
#pragma unroll
        for (int sl = 1; sl < NS; ++sl) part += tile[rl * NS + sl];
    }
    if (!in_rows) return;
    float L = 0.f, D = 0.f;
    if (real_row) {
        const int64_t so = (int64_t)u * g.Npk + pix;
        L = __ldg(a.stats + so) * a.stat_mul;
        if (a.Din) {
            D = __ldg(a.Din + so);
        } else {
            D = part;
            if (a.Dout && rr >= a.pp && rr < a.pp + g.H) a.Dout[so] = D;
        }
    }
    const int64_t plane = (int64_t)g.Wk * a.Hp;
    a.planes[(2 * (int64_t)u) * plane + (int64_t)w * a.Hp + rr] = L;
    a.planes[(2 * (int64_t)u + 1) * plane + (int64_t)w * a.Hp + rr] = D;
}

template <int CPE, int NS, int NT, int NCR, bool BF>
__global__ void __launch_bounds__(128) pack_rows_kernel(PackArgs a) {
    __shared__ __align__(16) float tile[128 * (NT == 2 ? kRowFloats : kSingleFloats)];
    pack_rows_body<CPE, NS, NT, NCR, BF>(a, tile);
}

template <int CPE, int NT>
void launch_pack_rows(const PackArgs& a, dim3 grid, int ns, cudaStream_t st) {
    const int cr = a.g.cr;
    if (CPE == 1 && NT == 2 && a.g.bf16) pack_rows_kernel<1, 1, 2, 0, true><<<grid, 128, 0, st>>>(a);
    else if (cr == 16) pack_rows_kernel<CPE, 1, NT, 16, false><<<grid, 128, 0, st>>>(a);
    else if (cr == 32) pack_rows_kernel<CPE, 2, NT, 32, false><<<grid, 128, 0, st>>>(a);
    else if (cr == 64) pack_rows_kernel<CPE, 4, NT, 64, false><<<grid, 128, 0, st>>>(a);
    else if (ns == 1) pack_rows_kernel<CPE, 1, NT, 0, false><<<grid, 128, 0, st>>>(a);
    else if (ns == 2) pack_rows_kernel<CPE, 2, NT, 0, false><<<grid, 128, 0, st>>>(a);
    else pack_rows_kernel<CPE, 4, NT, 0, false><<<grid, 128, 0, st>>>(a);
}

}  // namespace

int launch_pack(const PackArgs& a, cudaStream_t st) {
    const int ns = slabs_of(a.g), rb = 128 / ns;
    dim3 grid((a.Hp + rb - 1) / rb, a.g.Wk, a.g.units * (a.npairs + (a.planes ? 1 : 0)));
    // beyond the grid limits (very long folded 1-D signals, very many units) the generic kernels run
    if (grid.y > 65535u || grid.z > 65535u) return CA_ERR_UNSUPPORTED;
    if (a.g.cpe == 1) {
        if (a.single) launch_pack_rows<1, 1>(a, grid, ns, st);
        else launch_pack_rows<1, 2>(a, grid, ns, st);
    } else {
        if (a.single) launch_pack_rows<2, 1>(a, grid, ns, st);
        else launch_pack_rows<2, 2>(a, grid, ns, st);
    }
    CA_CHECK_LAUNCH("pack kernel");
    return CA_OK;
}

// ---------------------------------------------------------------- tensor maps
int encode_tensor_map(CUtensorMap* map, const float* base, int rank, const uint64_t* dims,
                      const uint64_t* strides_bytes, const uint32_t* box) {
    typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q);
        if (e != cudaSuccess || !sym) {
            set_error("cuTensorMapEncodeTiled is not available from the driver");
            return CA_ERR_CUDA;
        }
        fn = reinterpret_cast<EncodeFn>(sym);
    }
    cuuint64_t gdims[5], gstr[4];
    cuuint32_t gbox[5], estr[5];
    for (int i = 0; i < rank; ++i) { gdims[i] = dims[i]; gbox[i] = box[i]; estr[i] = 1; }
    for (int i = 0; i + 1 < rank; ++i) gstr[i] = strides_bytes[i];
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank, const_cast<float*>(base), gdims, gstr,
                    gbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
        return CA_ERR_CUDA;
    }
    return CA_OK;
}

int* stage_timeout_counter() {
    static std::atomic<int*> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    int* p = cache[dev].load(std::memory_order_relaxed);
    if (!p) {
        if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_stage_timeouts) != cudaSuccess) return nullptr;
        cache[dev].store(p, std::memory_order_relaxed);
    }
    return p;
}

int tiled_stage_timeouts(int* count) {
    cudaError_t e = cudaMemcpyFromSymbol(count, g_stage_timeouts, sizeof(int));
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyFromSymbol(stage timeouts)");
    return CA_OK;
}

// ---------------------------------------------------------------- bounded-wait self test
// One CTA arms a stage barrier with more bytes than the single bulk copy it issues delivers, so the
// barrier never completes; the wait must run out after `tries` polls, the CTA must report through the
// same counter and status word as the tiled kernels and return.  Nothing faults and nothing spins
// without a limit; the copy itself lands (the thread polls its destination, again with a limit).
__device__ __align__(16) float g_probe_src[8] = {1.f, 2.f, 3.f, 4.f, 5.f, 6.f, 7.f, 8.f};

__global__ void __launch_bounds__(32) stage_timeout_probe_kernel(uint32_t tries, int* status, int* out) {
    __shared__ __align__(16) float dst[8];
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        dst[7] = 0.f;
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) {
        mbar_arrive_expect_tx(smem_u32(&bar), 64);                      // 64 bytes expected ...
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 32, [%2];"
                     ::"r"(smem_u32(dst)), "l"(g_probe_src), "r"(smem_u32(&bar)) : "memory");   // ... 32 delivered
        ok = mbar_wait(smem_u32(&bar), 0, tries);
        // the copy in flight gets a bounded chance to land before the CTA (and its shared memory) goes away
        for (uint32_t i = 0; i < (1u << 16) && *reinterpret_cast<volatile float*>(&dst[7]) != 8.f; ++i) {}
        if (!ok) {
            atomicAdd(&g_stage_timeouts, 1);
            if (status) atomicOr(status, 1);
        }
        if (out) *out = ok ? 0 : 1;
    }
}

int tiled_probe_stage_timeout(uint32_t tries, int* out, cudaStream_t st) {
    stage_timeout_probe_kernel<<<1, 32, 0, st>>>(tries, status_word(), out);
    CA_CHECK_LAUNCH("stage timeout probe kernel");
    return CA_OK;
}

}  // namespace ca
