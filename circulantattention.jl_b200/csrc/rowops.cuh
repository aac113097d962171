// Row-wise and elementwise kernels on the stored values of a Circulant:
// structure generation, row normalisers and their pullbacks, sums, algebra.
#pragma once
#include "common.cuh"

namespace ca {

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------- structure
// One thread per stored entry of one batch slice; the slice is written to all
// nbatch replicas.  Entry n of row j: position pos -> window offset -> column.
__global__ void structure_kernel(int H, int W, int ws, int wsw, int64_t nbatch,
                                 int32_t* __restrict__ rowptr, int32_t* __restrict__ colval) {
    const int p = (ws - 1) / 2;
    const int K = ws * wsw;
    const int64_t Np = (int64_t)H * W;
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n <= Np) {
        const int32_t r = (int32_t)(1 + (int64_t)K * n);
        for (int64_t b = 0; b < nbatch; ++b) rowptr[n + (Np + 1) * b] = r;
    }
    if (n >= Np * K) return;
    const int j = (int)(n / K);
    const int k = (int)(n - (int64_t)j * K);
    const int h = j % H, w = j / H;
    const int posh = k % ws, posw = k / ws;
    // invert axis_pos: the run of row coordinate x starts at the smallest column
    // of the window, so the column at position `pos` is the pos-th smallest of
    // {(x+d) mod X}.
    auto col_at = [&](int pos, int x, int X) {
        if (x < p) {
            const int nfront = x + p + 1;          // coordinates 0..x+p, then the wrapped tail
            return pos < nfront ? pos : X - (ws - nfront) + (pos - nfront);
        }
        if (x >= X - p) {
            const int nfront = x + p - X + 1;      // wrapped coordinates 0..x+p-X come first
            return pos < nfront ? pos : (x - p) + (pos - nfront);
        }
        return x - p + pos;
    };
    const int ch = col_at(posh, h, H);
    const int cw = (wsw == 1) ? 0 : col_at(posw, w, W);
    const int32_t col = (int32_t)(ch + H * cw + 1);
    for (int64_t b = 0; b < nbatch; ++b) colval[n + Np * K * b] = col;
}

// ---------------------------------------------------------------- row normalisers
// The K entries of a row are contiguous.  A row is held in the registers of G lanes, R entries each (G*R >= K), so
// that it is read and written once with all its loads in flight, and short rows share a warp: one warp per row with a
// loop over it had two loads in flight and a quarter of its lanes idle at K = 49 (row sums of 160 MB: 118 us,
// 1.4 TB/s).  Bound: HBM.
template <int G>
__device__ __forceinline__ float group_max(float v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
template <int G>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Runs the statements with `constexpr int G, R` for rows of K entries; rows of more than 512 take the loop kernels.
#define CA_ROW_SHAPE(K, CALL, LOOP)                                                     \
    do {                                                                                \
        if ((K) <= 16) { constexpr int G = 8, R = 2; CALL; }                            \
        else if ((K) <= 32) { constexpr int G = 8, R = 4; CALL; }                       \
        else if ((K) <= 64) { constexpr int G = 16, R = 4; CALL; }                      \
        else if ((K) <= 128) { constexpr int G = 32, R = 4; CALL; }                     \
        else if ((K) <= 256) { constexpr int G = 32, R = 8; CALL; }                     \
        else if ((K) <= 512) { constexpr int G = 32, R = 16; CALL; }                    \
        else { LOOP; }                                                                  \
    } while (0)

template <int G, int R>
__global__ void __launch_bounds__(256) row_softmax_reg_kernel(int64_t rows, int K, const float* s, float* p,
                                                              float* __restrict__ stats) {
    const int64_t row = ((int64_t)blockIdx.x * 256 + threadIdx.x) / G;
    const int lane = threadIdx.x % G;
    const bool ok = row < rows;
    const float* sr = s + row * K;
    float z[R];
    float m = -INFINITY;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int k = lane + G * i;
        z[i] = ok && k < K ? sr[k] : -INFINITY;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) m = fmaxf(m, z[i]);
    m = group_max<G>(m);
    float l = 0.f;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        z[i] = __expf(z[i] - m);
        l += z[i];
    }
    l = group_sum<G>(l);
    const float inv = 1.f / l;
    if (!ok) return;
    float* pr = p + row * K;
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (lane + G * i < K) pr[lane + G * i] = z[i] * inv;
    if (stats && lane == 0) stats[row] = m + logf(l);
}

// Rows of more than 512 entries: one warp per row.
__global__ void __launch_bounds__(256) row_softmax_kernel(int64_t rows, int K,
                                                          const float* s,
                                                          float* p,
                                                          float* __restrict__ stats) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float* sr = s + row * K;
    float* pr = p + row * K;
    float m = -INFINITY;
    for (int k = lane; k < K; k += 32) m = fmaxf(m, sr[k]);
    m = warp_max(m);
    float l = 0.f;
    for (int k = lane; k < K; k += 32) l += __expf(sr[k] - m);
    l = warp_sum(l);
    const float inv = 1.f / l;
    for (int k = lane; k < K; k += 32) pr[k] = __expf(sr[k] - m) * inv;
    if (stats && lane == 0) stats[row] = m + logf(l);
}

// 1.5-entmax: p = max(s/2 - tau, 0)^2 with sum p = 1.  tau is bracketed by
// bisection (which fixes the support), then solved in closed form on that
// support: tau = mean - sqrt((1 - sum (z-mean)^2) / n).
__global__ void __launch_bounds__(256) row_entmax15_kernel(int64_t rows, int K,
                                                           const float* s,
                                                           float* p,
                                                           float* __restrict__ stats) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float* sr = s + row * K;
    float* pr = p + row * K;
    float m = -INFINITY;
    for (int k = lane; k < K; k += 32) m = fmaxf(m, 0.5f * sr[k]);
    m = warp_max(m);
    // work with z - m for accuracy; tau' in [-1, 0)
    float lo = -1.f, hi = 0.f;
    for (int it = 0; it < 26; ++it) {
        const float mid = 0.5f * (lo + hi);
        float f = 0.f;
        for (int k = lane; k < K; k += 32) {
            const float t = fmaxf(0.5f * sr[k] - m - mid, 0.f);
            f = fmaf(t, t, f);
        }
        f = warp_sum(f);
        if (f > 1.f) lo = mid; else hi = mid;
    }
    const float tb = 0.5f * (lo + hi);
    float n = 0.f, sum = 0.f;
    for (int k = lane; k < K; k += 32) {
        const float z = 0.5f * sr[k] - m;
        if (z > tb) { n += 1.f; sum += z; }
    }
    n = warp_sum(n);
    sum = warp_sum(sum);
    const float mean = sum / n;
    float ss = 0.f;
    for (int k = lane; k < K; k += 32) {
        const float z = 0.5f * sr[k] - m;
        if (z > tb) ss = fmaf(z - mean, z - mean, ss);
    }
    ss = warp_sum(ss);
    const float tau = mean - sqrtf(fmaxf((1.f - ss) / n, 0.f));
    for (int k = lane; k < K; k += 32) {
        const float t = fmaxf(0.5f * sr[k] - m - tau, 0.f);
        pr[k] = t * t;
    }
    if (stats && lane == 0) stats[row] = tau + m;
}

// The same for rows of at most G*R entries, held in the registers of G lanes (one global read, one write).  A step
// solves the quadratic on the entries above the current threshold; when the root has as many entries above it, the
// support is known (supports are nested), and the closed form gives tau.  The bracket of the thresholds seen so far
// guards the search, which halves it where a root leaves it.  Two to four steps on ordinary rows.  Bound by the chain of
// group sums and by issue, not by memory, hence few lanes per row and several rows per warp: 98304 rows of 225 entries
// in 49 us (one warp per row 63, with bisection 89; their 177 MB take 27), 280000 rows of 49 in 43
// (96, 110; 17).
#define CA_ENTMAX_SHAPE(K, CALL, LOOP)                                                  \
    do {                                                                                \
        if ((K) <= 16) { constexpr int G = 8, R = 2; CALL; }                            \
        else if ((K) <= 32) { constexpr int G = 8, R = 4; CALL; }                       \
        else if ((K) <= 64) { constexpr int G = 8, R = 8; CALL; }                       \
        else if ((K) <= 128) { constexpr int G = 8, R = 16; CALL; }                     \
        else if ((K) <= 256) { constexpr int G = 16, R = 16; CALL; }                    \
        else if ((K) <= 512) { constexpr int G = 32, R = 16; CALL; }                    \
        else { LOOP; }                                                                  \
    } while (0)

template <int G, int R>
__global__ void __launch_bounds__(256) row_entmax15_reg_kernel(int64_t rows, int K,
                                                               const float* s,
                                                               float* p,
                                                               float* __restrict__ stats) {
    const int64_t row = ((int64_t)blockIdx.x * 256 + threadIdx.x) / G;
    const int lane = threadIdx.x % G;
    const bool ok = row < rows;
    const float* sr = s + row * K;
    float z[R];
    float m = -INFINITY;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int k = lane + G * i;
        z[i] = ok && k < K ? sr[k] : -INFINITY;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        z[i] *= 0.5f;
        m = fmaxf(m, z[i]);
    }
    const float lane_max = m;
    m = group_max<G>(m);
#pragma unroll
    for (int i = 0; i < R; ++i) z[i] -= m;                 // z - m in (-inf, 0]; tau' in [-1, 0)
    // first threshold: two Newton steps on the lanes' largest entries (compare entmax_start)
    float tau = -0.894427191f;
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const float t = fmaxf(lane_max - m - tau, 0.f);
        const float sa = group_sum<G>(t), sb = group_sum<G>(t * t);
        tau += sa > 0.f ? 0.5f * (sb - 0.8f) / sa : 0.f;
    }
    float lo = -1.001f, hi = 0.f;                          // a row with one entry in the support has its root at -1
    float n_lo = -1.f, n_hi = 0.f, n_solved = -1.f;        // entries above lo / above hi / in the support last solved for
    bool open = ok;
    for (int it = 0; it < 34 && __any_sync(0xffffffffu, open); ++it) {
        float n = 0.f, sa = 0.f, sb = 0.f;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float t = fmaxf(z[i] - tau, 0.f);
            sa += t;
            sb = fmaf(t, t, sb);
            n += z[i] > tau ? 1.f : 0.f;
        }
        sa = group_sum<G>(sa);
        sb = group_sum<G>(sb);
        n = group_sum<G>(n);
        if (!open) continue;
        if (sb > 1.f) { lo = tau; n_lo = n; } else { hi = tau; n_hi = n; }
        if (n == n_solved || n_lo == n_hi) { open = false; continue; }
        // the root for the current support; past the eighth step, or where it leaves the bracket, the middle
        const float root = tau + (sa - sqrtf(fmaxf(fmaf(sa, sa, -n * (sb - 1.f)), 0.f))) / n;
        const bool solve = it < 8 && root >= lo && root <= hi;
        n_solved = solve ? n : -1.f;
        tau = solve ? root : 0.5f * (lo + hi);
    }
    // support = entries above the last threshold
    float n = 0.f, sum = 0.f;
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (z[i] > tau) { n += 1.f; sum += z[i]; }
    n = group_sum<G>(n);
    sum = group_sum<G>(sum);
    const float mean = sum / n;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (z[i] > tau) ss = fmaf(z[i] - mean, z[i] - mean, ss);
    ss = group_sum<G>(ss);
    tau = mean - sqrtf(fmaxf((1.f - ss) / n, 0.f));
    if (!ok) return;
    float* pr = p + row * K;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const float t = fmaxf(z[i] - tau, 0.f);
        if (lane + G * i < K) pr[lane + G * i] = t * t;
    }
    if (stats && lane == 0) stats[row] = tau + m;
}

template <int G, int R>
__global__ void __launch_bounds__(256) row_normalize_bwd_reg_kernel(int64_t rows, int K, int entmax, const float* __restrict__ p,
                                                                    const float* dp, float* ds) {
    const int64_t row = ((int64_t)blockIdx.x * 256 + threadIdx.x) / G;
    const int lane = threadIdx.x % G;
    const bool ok = row < rows;
    const float* pr = p + row * K;
    const float* dr = dp + row * K;
    float g[R], d[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int k = lane + G * i;
        g[i] = ok && k < K ? pr[k] : 0.f;
        d[i] = ok && k < K ? dr[k] : 0.f;
    }
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (entmax) g[i] = sqrtf(g[i]);
        a = fmaf(g[i], d[i], a);
        b += g[i];
    }
    a = group_sum<G>(a);
    b = group_sum<G>(b);
    const float D = entmax ? a / b : a;
    if (!ok) return;
    float* out = ds + row * K;
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (lane + G * i < K) out[lane + G * i] = g[i] * (d[i] - D);
}

__global__ void __launch_bounds__(256) row_normalize_bwd_kernel(int64_t rows, int K, int entmax,
                                                                const float* __restrict__ p,
                                                                const float* dp,
                                                                float* ds) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float* pr = p + row * K;
    const float* dr = dp + row * K;
    float* out = ds + row * K;
    float a = 0.f, b = 0.f;
    for (int k = lane; k < K; k += 32) {
        const float g = entmax ? sqrtf(pr[k]) : pr[k];
        a = fmaf(g, dr[k], a);
        b += g;
    }
    a = warp_sum(a);
    b = warp_sum(b);
    const float D = entmax ? a / b : a;
    for (int k = lane; k < K; k += 32) {
        const float g = entmax ? sqrtf(pr[k]) : pr[k];
        out[k] = g * (dr[k] - D);
    }
}

// ---------------------------------------------------------------- sums
template <int G, int R>
__global__ void __launch_bounds__(256) sum_rows_reg_kernel(int64_t rows, int K, const float* __restrict__ nz, float* __restrict__ out) {
    // two rows per group of lanes
    const int64_t row = ((int64_t)blockIdx.x * 256 + threadIdx.x) / G * 2;
    const int lane = threadIdx.x % G;
    float z[2][R];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int k = lane + G * i;
            z[r][i] = row + r < rows && k < K ? __ldg(nz + (row + r) * K + k) : 0.f;
        }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        float a = 0.f;
#pragma unroll
        for (int i = 0; i < R; ++i) a += z[r][i];
        a = group_sum<G>(a);
        if (lane == 0 && row + r < rows) out[row + r] = a;
    }
}

__global__ void __launch_bounds__(256) sum_rows_kernel(int64_t rows, int K,
                                                       const float* __restrict__ nz,
                                                       float* __restrict__ out) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    float a = 0.f;
    for (int k = lane; k < K; k += 32) a += nz[row * K + k];
    a = warp_sum(a);
    if (lane == 0) out[row] = a;
}

// Column sums by window symmetry: column i collects A[j, i] from the rows
// j = i + e, stored in row j at the position of offset -e.  Deterministic gather.
__global__ void __launch_bounds__(128) sum_cols_kernel(Geo g, const float* __restrict__ nz,
                                                       float* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int u = blockIdx.y;
    if (i >= g.Np) return;
    const int h = i % g.H, w = i / g.H;
    const float* nzu = nz + (int64_t)u * g.Np * g.K;
    float a = 0.f;
    for (int iw = 0; iw < g.wsw; ++iw) {
        const int ew = (g.wsw == 1) ? 0 : iw - g.p;
        const int jw = wrap_axis(w + ew, g.W);
        for (int ih = 0; ih < g.ws; ++ih) {
            const int eh = ih - g.p;
            const int jh = wrap_axis(h + eh, g.H);
            const int pos = ((g.wsw == 1) ? 0 : axis_pos(-ew, jw, g.W, g.p, g.ws) * g.ws) +
                            axis_pos(-eh, jh, g.H, g.p, g.ws);
            a += __ldg(nzu + (int64_t)(jh + g.H * jw) * g.K + pos);
        }
    }
    out[(int64_t)u * g.Np + i] = a;
}

// ---------------------------------------------------------------- algebra
__global__ void __launch_bounds__(256) axpby_kernel(int64_t n, float alpha, const float* __restrict__ x,
                                                    float beta, const float* __restrict__ y,
                                                    float* __restrict__ out) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t n4 = n >> 2;
    const bool vec = ((((uintptr_t)x | (uintptr_t)out | (uintptr_t)(y ? y : x)) & 15) == 0);
    if (vec) {
        const float4* x4 = reinterpret_cast<const float4*>(x);
        const float4* y4 = reinterpret_cast<const float4*>(y);
        float4* o4 = reinterpret_cast<float4*>(out);
        for (int64_t t = i; t < n4; t += stride) {
            float4 a = x4[t], r;
            if (y) {
                float4 b = y4[t];
                r = make_float4(alpha * a.x + beta * b.x, alpha * a.y + beta * b.y,
                                alpha * a.z + beta * b.z, alpha * a.w + beta * b.w);
            } else {
                r = make_float4(alpha * a.x, alpha * a.y, alpha * a.z, alpha * a.w);
            }
            o4[t] = r;
        }
        for (int64_t t = (n4 << 2) + i; t < n; t += stride)
            out[t] = alpha * x[t] + (y ? beta * y[t] : 0.f);
    } else {
        for (int64_t t = i; t < n; t += stride) out[t] = alpha * x[t] + (y ? beta * y[t] : 0.f);
    }
}

// A block scales runs of 2048 entries of one slice, eight loads in flight per thread (one entry per thread: 43 us for 16
// slices of 2 MB; slices start at any word, so the accesses stay four bytes wide).
constexpr int kScaleRun = 8;
__global__ void __launch_bounds__(256) scale_batch_kernel(int64_t inner, int o1, int o2,
                                                          const float* __restrict__ a, int a1, int a2,
                                                          const float* __restrict__ c, int c1, int c2,
                                                          float* __restrict__ out) {
    const int i1 = blockIdx.y, i2 = blockIdx.z;
    const float* src = a + ((int64_t)(a1 > 1 ? i1 : 0) + (int64_t)a1 * (a2 > 1 ? i2 : 0)) * inner;
    const float cv = c[(c1 > 1 ? i1 : 0) + c1 * (c2 > 1 ? i2 : 0)];
    float* dst = out + ((int64_t)i1 + (int64_t)o1 * i2) * inner;
    for (int64_t t0 = (int64_t)blockIdx.x * (256 * kScaleRun) + threadIdx.x; t0 < inner; t0 += (int64_t)gridDim.x * (256 * kScaleRun)) {
        float v[kScaleRun];
#pragma unroll
        for (int i = 0; i < kScaleRun; ++i)
            if (t0 + 256 * i < inner) v[i] = src[t0 + 256 * i];
#pragma unroll
        for (int i = 0; i < kScaleRun; ++i)
            if (t0 + 256 * i < inner) dst[t0 + 256 * i] = cv * v[i];
    }
}

// One block per batch slice, fixed summation order: deterministic, no scratch.
__global__ void __launch_bounds__(1024) dot_batch_kernel(int64_t inner, int o1,
                                                         const float* __restrict__ x, int x1, int x2,
                                                         const float* __restrict__ y, int y1, int y2,
                                                         float* __restrict__ out) {
    const int i1 = blockIdx.x, i2 = blockIdx.y;
    const int64_t xo = ((int64_t)(x1 > 1 ? i1 : 0) + (int64_t)x1 * (x2 > 1 ? i2 : 0)) * inner;
    const int64_t yo = y ? ((int64_t)(y1 > 1 ? i1 : 0) + (int64_t)y1 * (y2 > 1 ? i2 : 0)) * inner : 0;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    int64_t t = threadIdx.x;
    for (; t + 3 * 1024 < inner; t += 4 * 1024) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int64_t e = t + r * 1024;
            acc[r] = y ? fmaf(x[xo + e], y[yo + e], acc[r]) : acc[r] + x[xo + e];
        }
    }
    for (; t < inner; t += 1024) acc[0] = y ? fmaf(x[xo + t], y[yo + t], acc[0]) : acc[0] + x[xo + t];
    float a = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    __shared__ float sm[32];
    a = warp_sum(a);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x < 32) {
        float v = sm[threadIdx.x];
        v = warp_sum(v);
        if (threadIdx.x == 0) out[i1 + o1 * i2] = v;
    }
}

__global__ void __launch_bounds__(256) sum_batch_kernel(int64_t inner, int b1, int b2, int sum1, int sum2,
                                                        const float* __restrict__ in,
                                                        float* __restrict__ out) {
    const int o1 = sum1 ? 1 : b1, o2 = sum2 ? 1 : b2;
    const int64_t total = inner * o1 * o2;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += stride) {
        const int64_t n = t % inner;
        const int64_t r = t / inner;
        const int i1 = (int)(r % o1), i2 = (int)(r / o1);
        float acc = 0.f;
        for (int j2 = sum2 ? 0 : i2; j2 < (sum2 ? b2 : i2 + 1); ++j2)
            for (int j1 = sum1 ? 0 : i1; j1 < (sum1 ? b1 : i1 + 1); ++j1)
                acc += in[((int64_t)j1 + (int64_t)b1 * j2) * inner + n];
        out[t] = acc;
    }
}

}  // namespace ca
