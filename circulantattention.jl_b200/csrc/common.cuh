// Shared host/device helpers of the circulant-attention kernels (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdarg.h>
#include <atomic>
#include "../../include/circatt_b200.h"
#include "../../include/circatt_b200_probe.h"

namespace ca {

// ---------------------------------------------------------------- errors
void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);

// Device word registered by the calling host thread with ca_status_word (NULL: none).
int* status_word();

void count_launch();
void count_tiled_launch();     // launches of the TMA-tiled kernels only (tests use it to see which path ran)
void count_tensor_launch();    // of those, the sweeps on the tensor cores

#define CA_CHECK_LAUNCH(what)                                        \
    do {                                                             \
        ca::count_launch();                                          \
        cudaError_t e__ = cudaGetLastError();                        \
        if (e__ != cudaSuccess) return ca::cuda_fail(e__, what);     \
    } while (0)

// ---------------------------------------------------------------- geometry
// Window geometry in pixel units.  The query side has H x W pixels; the key
// side has H x Wk pixels.  With Wk == W the window wraps circularly along both
// axes; in band mode (Wk = W + 2p, wk_off = p) the key-side tensors already
// hold the neighbouring columns, so only the fast axis wraps.
struct Geo {
    int H, W, Wk, wk_off;
    int ws, p;
    int wsw;      // window extent along w: ws in 2-D, 1 in 1-D
    int K;        // entries per row: ws * wsw
    int Np, Npk;  // pixels on the query side / key side
    int units;
    int c;        // channels per unit in elements
    int cpe;      // floats per element: 1 (f32) or 2 (c64)
    int cr;       // real channels per unit: c * cpe
    int bf16;     // dense tensors are stored as bfloat16 (cpe == 1); arithmetic stays Float32
};

__host__ __device__ inline int wrap_axis(int x, int X) {
    x += (x < 0) ? X : 0;
    x -= (x >= X) ? X : 0;
    return x;
}

// Position of window offset d (in [-p, p]) inside the ascending-column run of a
// row whose own coordinate on that axis is x (axis length X).  Border rows are
// rotated so that wrapped columns keep the run sorted, which is what the
// circshift_index calls of the reference (src/circulant.jl:11-15, 30-39) do.
__host__ __device__ inline int axis_pos(int d, int x, int X, int p, int ws) {
    if (x < p) {
        int t = d + x;
        return t < 0 ? t + ws : t;
    }
    if (x >= X - p) {
        int t = d + x - X;
        return t < 0 ? t + ws : t;
    }
    return d + p;
}

int make_geo(const ca_desc* d, Geo* g, bool allow_band);

static inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// ---------------------------------------------------------------- host
// SM count of the current device (cached per device ordinal).
inline int sm_count() {
    static std::atomic<int> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    int n = cache[dev].load(std::memory_order_relaxed);
    if (!n) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cache[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// ---------------------------------------------------------------- device math
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// First threshold of the entmax search from the largest scores of N classes of a row's keys (any partition; an empty
// class holds -inf): the root of sum_i max(top_i - tau, 0)^2 = 1 / 1.25, by three Newton steps from the left (the
// sum is convex and falls with tau, so they never pass the root).  The root of a subset is a lower bound of the row's
// threshold; the factor stands for the members of the support behind their class's largest.  With eight classes two
// threshold sweeps leave at most 3 rows in 128 open (15 to 127 keys, 4 to 16 channels, standard normal), where a start
// at max - 1 took three to four.  The start lies below the row's maximum by at least sqrt(1 / (1.25 N)), so no support
// is empty.
template <int N>
__device__ __forceinline__ float entmax_start(const float (&top)[N]) {
    float m = top[0];
#pragma unroll
    for (int i = 1; i < N; ++i) m = fmaxf(m, top[i]);
    float t = -0.894427191f;                      // relative to m: one member alone
#pragma unroll
    for (int it = 0; it < 3; ++it) {
        float sa = 0.f, sb = 0.f;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float p = fmaxf((top[i] - m) - t, 0.f);
            sa += p;
            sb = fmaf(p, p, sb);
        }
        t += sa > 0.f ? 0.5f * (sb - 0.8f) / sa : 0.f;
    }
    return m + t;
}
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

}  // namespace ca
