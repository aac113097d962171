// Tiled sm_100a kernels for 2-D windows and folded 1-D signals of up to 64 real channels per unit (Float32 or ComplexF32;
// bfloat16 storage at 8 and 16), softmax, and for one slab of channels the 1.5-entmax.
//
// Work decomposition.  A CTA owns TH consecutive rows (the fast axis h) of NQ consecutive columns w0..w0+NQ-1 of one unit.
// A thread owns one row and the NQ pixels of that row ("centre" pixels: queries in the forward and dq kernels, keys in
// the dk/dv kernels) and keeps their 16-channel vectors in registers; units of more channels give a pixel two or four
// lanes.  NQ, the rows and how many groups of warps share the stages of a tile follow from a prediction of the time
// (choose_tile).  The other
// side of the window is streamed through shared memory one image column at a
// time: column stage s holds column w0 - p + s (wrapped circularly, or taken
// from the neighbour halo in band mode) for rows h0-p' .. h0+TH+p'-1.  Centre
// pixel r pairs with stage s iff r <= s <= r + 2p, so every loaded vector is
// used by up to NQ centre pixels straight from registers.
//
// Feeding the stages.  The reference layout is channel-planar, which no bulk
// copy can turn into pixel vectors, so a pack kernel first rewrites the two
// streamed tensors as ONE array [unit][column][row'][36] = (16 channels of the
// first | 16 of the second | 4 floats of padding) with the circular halo along
// h already unrolled (row' = h + p', p' = p rounded up to even; rows -p'..-1
// and H..H+p'-1 are copies of the wrapped rows).  A column stage is then a
// single contiguous box fetched by cp.async.bulk.tensor (TMA) and tracked by an
// mbarrier; three stages are in flight.  The wrap along w is just the column
// coordinate of the box.
//
// Shared-memory layout: a pixel row is 144 bytes (36 words).  The rows that the
// eight lanes of a 128-bit load phase touch are consecutive, 36 words apart,
// i.e. nine 4-bank groups apart: eight distinct groups, so the loads are
// conflict free without any address swizzle and every chunk of every row of a
// window column is the thread's row base plus a compile-time constant.
//
// Arithmetic: FP32 on the FMA pipe, dot products scalar, outer products as packed FMAs.  Softmax in
// the log2 domain with ex2.approx.  The running maximum (forward) or the saved row
// statistic (backward) is folded into the initial value of the dot-product
// chain, and the forward only touches the maximum when the sign bits of a chunk
// of relative scores say that one of them is positive.
//
// Softmax at up to 16 real channels per unit on more than 12000 pixels x units runs on the tensor cores instead (split.cuh) where they are
// faster: windows 13 to 25, 9 and 11 in bfloat16 or where tiles of 32 rows would leave lanes idle, dk/dv also at all of 9 to 25 and at some
// of 7 (split_shape_ok and split_dkdv_ok have the rules and what they rest on).
//
// Small grids.  Where it pays, the column stages of a tile are split between up to four groups of warps of the same CTA
// (each with its own copy pipeline) whose partial results are merged through shared memory.
#include "split.cuh"

namespace ca {

// ---------------------------------------------------------------- entry points of this file
size_t tiled_fwd_workspace(const Geo& gin) {
    Geo g;
    if (!fold_geo(gin, &g)) return 0;
    if (!tiled_shape_ok(g)) return 0;
    return (padded_of(g).pair_floats + (size_t)g.Np * g.units) * sizeof(float);
}

size_t tiled_bwd_stage_workspace(const Geo& gin) {
    Geo g;
    if (!fold_geo(gin, &g)) return 0;
    if (!tiled_shape_ok(g)) return 0;
    const Padded P = padded_of(g);
    return (P.pair_floats + P.plane_floats) * sizeof(float);
}

size_t tiled_bwd_workspace(const Geo& gin) {
    Geo g;
    if (!fold_geo(gin, &g)) return 0;
    if (!tiled_shape_ok(g)) return 0;
    const Padded P = padded_of(g);
    return (2 * P.pair_floats + P.plane_floats + weight_floats(g)) * sizeof(float);
}

int tiled_attention_fwd(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                        float* y, float* nz, float* stats, void* workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g) || (nz && g.Wk != g.W)) return CA_ERR_UNSUPPORTED;
    if (!workspace) { set_error("workspace of ca_attention_fwd_workspace() bytes is NULL"); return CA_ERR_NULL; }
    const Padded P = padded_of(g);
    float* kv = static_cast<float*>(workspace);
    if (split_shape_ok(g, scale)) {
        if (nz && !stats) stats = kv + P.pair_floats;
        int rc = launch_split_pack(g, scale, dist, k, v, nullptr, nullptr, nullptr, nullptr, kv, st);
        if (rc) return rc;
        if ((rc = run_split_fwd(g, scale, dist, q, k, v, kv, y, stats, st)) || !nz) return rc;
        return run_split_emit(g, scale, dist, q, k, stats, kv, nz, st);
    }
    if (nz && !stats) stats = kv + P.pair_floats;         // scratch statistics behind the packed pair
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1;
    pa.src[0] = k; pa.src[1] = v; pa.dst[0] = kv;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    if (nz && values_fit(g, slabs_of(g))) {
        rc = CA_CHANNELS(g, run_fwd_values, g, P, scale, dist, q, kv, y, stats, nz, st);
        if (rc != CA_ERR_UNSUPPORTED) return rc;
    }
    if ((rc = CA_CHANNELS(g, run_fwd, g, P, scale, dist, q, kv, y, stats, st))) return rc;
    if (nz) return CA_CHANNELS(g, run_emit, g, P, scale, dist, q, stats, nz, kv, st, false);
    return CA_OK;
}

int tiled_attention_bwd_dq(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                           const float* dy, const float* stats, const float* D, float* dq, void* workspace,
                           cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g)) return CA_ERR_UNSUPPORTED;
    if (!workspace) { set_error("workspace of ca_attention_bwd_stage_workspace() bytes is NULL"); return CA_ERR_NULL; }
    const Padded P = padded_of(g);
    float* kv = static_cast<float*>(workspace);
    if (split_shape_ok(g, scale)) {
        int rc = launch_split_pack(g, scale, dist, k, v, nullptr, nullptr, nullptr, nullptr, kv, st);
        if (rc) return rc;
        return run_split_dq(g, scale, dist, q, k, v, dy, stats, D, kv, dq, st);
    }
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1;
    pa.src[0] = k; pa.src[1] = v; pa.dst[0] = kv;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    return CA_CHANNELS(g, run_dq, g, P, scale, dist, q, dy, stats, D, kv, dq, st, 0, nullptr);
}

int tiled_attention_bwd_dkdv(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                             const float* dy, const float* stats, const float* D, float* dk, float* dv,
                             void* workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g)) return CA_ERR_UNSUPPORTED;
    if (!workspace) { set_error("workspace of ca_attention_bwd_stage_workspace() bytes is NULL"); return CA_ERR_NULL; }
    const Padded P = padded_of(g);
    float* qdy = static_cast<float*>(workspace);
    if (split_dkdv_ok(g, scale)) {
        int rc = launch_split_pack(g, scale, dist, q, dy, stats, nullptr, D, nullptr, qdy, st);
        if (rc) return rc;
        return run_split_dkdv(g, scale, dist, q, k, v, dy, stats, D, qdy, dk, dv, st);
    }
    float* planes = qdy + P.pair_floats;
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1;
    pa.src[0] = q; pa.src[1] = dy; pa.dst[0] = qdy;
    pa.planes = planes; pa.stats = stats; pa.stat_mul = kLog2e; pa.Din = D;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    return CA_CHANNELS(g, run_dkdv, g, P, scale, dist, k, v, qdy, planes, dk, dv, st, false);
}

// Helper stream (one per host thread and device) on which the dk/dv sweep of a small problem runs
// next to the dq sweep: neither fills the GPU alone.  It is forked from and joined
// back to the caller's stream with events, so the caller sees ordinary stream order.  The
// stream and its two events belong to the calling host thread, so callers on different threads
// (and streams) neither share them nor wait for each other.
struct ForkJoin {
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};
static thread_local ForkJoin g_fork[64];

static ForkJoin* fork_join_for_current_device() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    ForkJoin& f = g_fork[dev];
    if (!f.side) {
        if (cudaStreamCreateWithFlags(&f.side, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&f.fork, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&f.join, cudaEventDisableTiming) != cudaSuccess) {
            f.side = nullptr;
            cudaGetLastError();
            return nullptr;
        }
    }
    return &f;
}

// Whole backward in three launches: pack (both pairs, D, planes), dq, dk/dv.  The two sweeps run side by side on small
// problems; where dq stores the weights for dk/dv (weight_floats) they run one after the other.
int tiled_attention_bwd(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                        const float* y, const float* dy, const float* stats, float* D, float* dq, float* dk,
                        float* dv, void* workspace, const void* fwd_workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g) || g.Wk != g.W) return CA_ERR_UNSUPPORTED;
    if (!workspace) { set_error("workspace is NULL"); return CA_ERR_NULL; }
    const Padded P = padded_of(g);
    float* kv = static_cast<float*>(workspace);
    float* qdy = kv + P.pair_floats;
    float* planes = qdy + P.pair_floats;
    // both sweeps: side by side where neither fills the GPU (fewer than ~4 CTAs per SM per sweep)
    auto run_both = [&](auto sweep_q, auto sweep_k) -> int {
        if ((long)g.Np * g.units < 2048L * sm_count()) {
            ForkJoin* f = fork_join_for_current_device();
            if (f && cudaEventRecord(f->fork, st) == cudaSuccess && cudaStreamWaitEvent(f->side, f->fork, 0) == cudaSuccess) {
                const int rc = sweep_k(f->side), rc2 = sweep_q(st);
                cudaError_t e = cudaEventRecord(f->join, f->side);
                if (e == cudaSuccess) e = cudaStreamWaitEvent(st, f->join, 0);
                if (e != cudaSuccess) return cuda_fail(e, "joining the helper stream");
                return rc ? rc : rc2;
            }
            cudaGetLastError();
        }
        const int rc = sweep_q(st);
        return rc ? rc : sweep_k(st);
    };
    // the forward of the same problem left its packed (k|v), split or not by the same rule, at the start of its workspace
    if (fwd_workspace) kv = const_cast<float*>(static_cast<const float*>(fwd_workspace));
    if (split_dkdv_ok(g, scale)) {
        const bool split = split_shape_ok(g, scale);
        int rc = CA_OK;
        if (!fwd_workspace && split) {
            rc = launch_split_pack(g, scale, dist, k, v, nullptr, nullptr, nullptr, nullptr, kv, st);
        } else if (!fwd_workspace) {
            PackArgs pa{};
            pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1;
            pa.src[0] = k; pa.src[1] = v; pa.dst[0] = kv;
            rc = launch_pack(pa, st);
        }
        if (rc || (rc = launch_split_pack(g, scale, dist, q, dy, stats, y, nullptr, D, qdy, st))) return rc;
        return run_both(
            [&](cudaStream_t s) {
                return split ? run_split_dq(g, scale, dist, q, k, v, dy, stats, D, kv, dq, s)
                             : CA_CHANNELS(g, run_dq, g, P, scale, dist, q, dy, stats, D, kv, dq, s, 0, nullptr);
            },
            [&](cudaStream_t s) { return run_split_dkdv(g, scale, dist, q, k, v, dy, stats, D, qdy, dk, dv, s); });
    }
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp;
    if (fwd_workspace) {
        // only (q|dy) and the planes are packed here
        pa.npairs = 1;
        pa.src[0] = q; pa.src[1] = dy;
        pa.dst[0] = qdy;
    } else {
        pa.npairs = 2;
        pa.src[0] = k; pa.src[1] = v; pa.src[2] = q; pa.src[3] = dy;
        pa.dst[0] = kv; pa.dst[1] = qdy;
    }
    pa.planes = planes; pa.stats = stats; pa.stat_mul = kLog2e; pa.y = y; pa.dy = dy; pa.Dout = D;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    if (weight_floats(g)) {
        float* weights = planes + P.plane_floats;
        if ((rc = CA_CHANNELS(g, run_dq, g, P, scale, dist, q, dy, stats, D, kv, dq, st, 0, nullptr, weights))) return rc;
        return CA_CHANNELS(g, run_dkdv_stored, g, P, scale, dist, k, qdy, weights, dk, dv, st);
    }
    return run_both([&](cudaStream_t s) { return CA_CHANNELS(g, run_dq, g, P, scale, dist, q, dy, stats, D, kv, dq, s, 0, nullptr); },
                    [&](cudaStream_t s) { return CA_CHANNELS(g, run_dkdv, g, P, scale, dist, k, v, qdy, planes, dk, dv, s, false); });
}

// Entmax-1.5 backward on the fused kernels.  Unlike the softmax, D = sum g*dP / sum g is not dy.y, so
// a pre-pass over the packed (k|v) computes it first: pack (k|v) -> pre-pass -> pack (q|dy) + planes
// (tau, D) -> dq and dk/dv.  `stats` holds tau.
int tiled_attention_bwd_entmax(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                               const float* dy, const float* stats, float* D, float* dq, float* dk, float* dv,
                               void* workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g) || g.Wk != g.W || g.bf16 || slabs_of(g) > 1) return CA_ERR_UNSUPPORTED;
    if (!workspace) { set_error("workspace is NULL"); return CA_ERR_NULL; }
    const Padded P = padded_of(g);
    float* kv = static_cast<float*>(workspace);
    float* qdy = kv + P.pair_floats;
    float* planes = qdy + P.pair_floats;
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1;
    pa.src[0] = k; pa.src[1] = v; pa.dst[0] = kv;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    if ((rc = CA_CHANNELS(g, run_dq, g, P, scale, dist, q, dy, stats, nullptr, kv, nullptr, st, 2, D))) return rc;
    PackArgs pb{};
    pb.g = g; pb.pp = P.pp; pb.Hp = P.Hp; pb.npairs = 1;
    pb.src[0] = q; pb.src[1] = dy; pb.dst[0] = qdy;
    pb.planes = planes; pb.stats = stats; pb.stat_mul = 1.f; pb.Din = D;
    if ((rc = launch_pack(pb, st))) return rc;
    if ((rc = CA_CHANNELS(g, run_dq, g, P, scale, dist, q, dy, stats, D, kv, dq, st, 1, nullptr))) return rc;
    return CA_CHANNELS(g, run_dkdv, g, P, scale, dist, k, v, qdy, planes, dk, dv, st, true);
}

// The 1.5-entmax forward in flash mode without A-sized memory: the packed (k|v) is swept once for the first
// thresholds, a fixed number of times for the thresholds (blocks whose rows are all final leave at once) and once
// for y.  `stats` (nullable) receives tau and doubles as the search's state; the `settled` plane and a tau plane
// for callers without `stats` live behind the pair in the workspace (tiled_fwd_entmax_workspace bytes).
size_t tiled_fwd_entmax_workspace(const Geo& gin) {
    Geo g;
    if (!fold_geo(gin, &g)) return 0;
    if (!tiled_shape_ok(g) || g.bf16 || slabs_of(g) > 1) return 0;
    return padded_of(g).pair_floats * sizeof(float) + 2 * (size_t)g.Np * g.units * sizeof(float);
}

int tiled_attention_fwd_entmax(const Geo& gin, float scale, int dist, const float* q, const float* k, const float* v,
                               float* y, float* stats, void* workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!tiled_shape_ok(g) || g.Wk != g.W || g.bf16 || slabs_of(g) > 1) return CA_ERR_UNSUPPORTED;
    if (!workspace) return CA_ERR_UNSUPPORTED;
    const Padded P = padded_of(g);
    float* kv = static_cast<float*>(workspace);
    float* settled = kv + P.pair_floats;
    if (!stats) stats = settled + (size_t)g.Np * g.units;       // a caller that does not want tau
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1;
    pa.src[0] = k; pa.src[1] = v; pa.dst[0] = kv;
    int rc = launch_pack(pa, st);
    if (rc) return rc;
    cudaError_t e = cudaMemsetAsync(settled, 0, (size_t)g.Np * g.units * sizeof(float), st);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync");
    if ((rc = CA_CHANNELS(g, run_entmax_fwd_sweep, g, P, scale, dist, q, kv, stats, settled, nullptr, 3, 0, st))) return rc;
    // the support iteration ends after 3-5 steps on ordinary rows; the steps past the tenth are Newton steps,
    // which converge for every row
    for (int it = 0; it < kEntmaxFwdSteps; ++it)
        if ((rc = CA_CHANNELS(g, run_entmax_fwd_sweep, g, P, scale, dist, q, kv, stats, settled, nullptr, 4, it, st))) return rc;
    return CA_CHANNELS(g, run_entmax_fwd_sweep, g, P, scale, dist, q, kv, stats, settled, y, 5, 0, st);
}

}  // namespace ca
