// The stand-alone operators on the tiled kernels: the similarity, A (x) V and A^T (x) V, the similarity pullback.  They share the packed layout and the stage pipeline of the fused kernels.
#include "tile_common.cuh"

namespace ca {

// ---------------------------------------------------------------- stand-alone operators
size_t tiled_operator_workspace(const Geo& gin) {
    Geo g;
    if (!fold_geo(gin, &g)) return 0;
    if (!tiled_operator_ok(g)) return 0;
    return padded_of(g).single_floats * sizeof(float);
}

// Packs one tensor as single-tensor rows.
static int pack_single(const Geo& g, const Padded& P, const float* src, float* dst, cudaStream_t st) {
    PackArgs pa{};
    pa.g = g; pa.pp = P.pp; pa.Hp = P.Hp; pa.npairs = 1; pa.single = 1;
    pa.src[0] = src; pa.dst[0] = dst;
    return launch_pack(pa, st);
}

// Scaled similarity scores in CSR order: x indexes the row pixel, y the column pixel.
int tiled_similarity(const Geo& gin, float scale, int dist, const float* x, const float* y, float* nz,
                     void* workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!workspace || !tiled_operator_workspace(g)) return CA_ERR_UNSUPPORTED;
    const Padded P = padded_of(g);
    int rc = pack_single(g, P, y, static_cast<float*>(workspace), st);
    if (rc) return rc;
    return CA_CHANNELS(g, run_emit, g, P, scale, dist, x, nullptr, nz, static_cast<const float*>(workspace), st, true);
}

// out = alpha * (A (x) v) or alpha * (A^T (x) v) from the values of A in CSR order.
int tiled_apply(const Geo& gin, const float* nz, const float* v, float* out, float alpha, int transposed,
                void* workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!workspace || !tiled_operator_workspace(g)) return CA_ERR_UNSUPPORTED;
    const Padded P = padded_of(g);
    float* packed = static_cast<float*>(workspace);
    int rc = pack_single(g, P, v, packed, st);
    if (rc) return rc;
    return CA_CHANNELS(g, run_apply, g, P, nz, packed, nullptr, out, alpha, transposed, st);
}

// Pullback of the similarity: dx[j] = scale * sum_i dS[j,i] y[i], dy[i] = scale * sum_j dS[j,i] x[j]
// (Distance: minus the sum of the dS involved times the pixel's own vector).
int tiled_similarity_bwd(const Geo& gin, float scale, int dist, const float* x, const float* y, const float* dS,
                         float* dx, float* dy, void* workspace, cudaStream_t st) {
    Geo g;
    if (!fold_geo(gin, &g)) return CA_ERR_UNSUPPORTED;
    if (!workspace || !tiled_operator_workspace(g)) return CA_ERR_UNSUPPORTED;
    const Padded P = padded_of(g);
    float* packed = static_cast<float*>(workspace);
    int rc;
    if (dx) {
        if ((rc = pack_single(g, P, y, packed, st))) return rc;
        if ((rc = CA_CHANNELS(g, run_apply, g, P, dS, packed, dist ? x : nullptr, dx, scale, 0, st))) return rc;
    }
    if (dy) {
        if ((rc = pack_single(g, P, x, packed, st))) return rc;
        if ((rc = CA_CHANNELS(g, run_apply, g, P, dS, packed, dist ? y : nullptr, dy, scale, 1, st))) return rc;
    }
    return CA_OK;
}

}  // namespace ca
