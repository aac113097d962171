"""How the tiled sweeps are cut into blocks: one to three columns per thread, one to four warps of rows, stages shared by one
to four groups of warps.  The shapes reach those cuts on a B200 (148 SMs)."""
import numpy as np
import pytest

from oracle import circatt_oracle as orc
from tests.helpers import KIND, assert_close, randn, up

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("shape,ws,nheads,cplx", [
    ((32, 32, 16, 1), 7, 1, False),       # one column, one warp, stages in four
    ((48, 48, 32, 1), 5, 2, False),       # stages in two and three; fewer stages than a thread's share would round to
    ((16, 17, 8, 1), 3, 1, False),        # three stages among four groups at most
    ((60, 50, 16, 2), 21, 1, False),      # three columns, stages in four
    ((75, 53, 36, 3), 11, 3, False),      # one and two columns, three warps of rows, 12 channels
    ((64, 64, 32, 4), 9, 2, False),       # two columns, two warps, stages in two
    ((70, 31, 32, 2), 9, 1, False),       # two slabs: rows of 16 per warp, no shared stages
    ((40, 40, 32, 2), 7, 1, True),        # four slabs, one column
])
def test_cuts(ca, shape, ws, nheads, cplx, simname):
    rng = np.random.default_rng(61)
    qn, kn, vn, rn = (randn(rng, shape, cplx) for _ in range(4))
    q, k, v = (ca.jl.from_numpy(t).requires_grad_(True) for t in (qn, kn, vn))
    sim = ca.DotSimilarity() if simname == "dot" else ca.DistanceSimilarity()
    n0 = ca.lib.ca_probe_tiled_launch_count()
    y, _ = ca.circulant_mh_attention(sim, q, k, v, ws, nheads, return_A=False)
    r = ca.jl.from_numpy(rn)
    ((y * r.conj()).real.sum() if cplx else (y * r).sum()).backward()
    assert ca.lib.ca_probe_tiled_launch_count() - n0 == 3
    yo, _ = orc.mh_attention(KIND[simname], up(qn), up(kn), up(vn), ws, nheads)
    dqo, dko, dvo = orc.mh_attention_pullback(KIND[simname], up(qn), up(kn), up(vn), ws, nheads, up(rn))
    for name, got, want in (("y", y, yo), ("dq", q.grad, dqo), ("dk", k.grad, dko), ("dv", v.grad, dvo)):
        assert_close(ca.jl.to_numpy(got), want, name)


@pytest.mark.parametrize("shape,ws,nheads", [((32, 32, 16, 1), 7, 1), ((75, 53, 36, 3), 11, 3)])
def test_cuts_entmax(ca, shape, ws, nheads):
    rng = np.random.default_rng(62)
    qn, kn, vn, rn = (randn(rng, shape) for _ in range(4))
    q, k, v = (ca.jl.from_numpy(t).requires_grad_(True) for t in (qn, kn, vn))
    y, _ = ca.circulant_mh_attention(ca.DotSimilarity(), q, k, v, ws, nheads, normalizer=ca.ENTMAX15, return_A=False)
    (y * ca.jl.from_numpy(rn)).sum().backward()
    yo, _ = orc.mh_attention(orc.DOT, up(qn), up(kn), up(vn), ws, nheads, orc.ENTMAX15)
    dqo, dko, dvo = orc.mh_attention_pullback(orc.DOT, up(qn), up(kn), up(vn), ws, nheads, up(rn), norm=orc.ENTMAX15)
    for name, got, want in (("y", y, yo), ("dq", q.grad, dqo), ("dk", k.grad, dko), ("dv", v.grad, dvo)):
        assert_close(ca.jl.to_numpy(got), want, name)


@pytest.mark.parametrize("shape,ws,nheads,cplx", [
    ((32, 32, 16, 1), 7, 1, False),       # rows of A kept by the forward: one column, stages in four
    ((37, 23, 24, 2), 9, 2, False),       # short channel count, rows past the image, wrapped rows
    ((41, 30, 32, 1), 9, 1, False),       # two slabs, at the limit of what the forward keeps
    ((33, 19, 32, 2), 7, 1, True),        # four slabs, an odd last column
    ((26, 25, 64, 1), 19, 1, False),      # four slabs, the largest window the forward keeps
    ((35, 26, 32, 1), 15, 1, False),      # past it: runs staged per window column
    ((36, 37, 16, 2), 35, 1, False),      # runs in two pieces
    ((131, 40, 1), 9, 1, False),          # folded signal, short last column
    ((300, 24, 2), 127, 1, False),        # folded signal, rows of 127
])
@pytest.mark.parametrize("simname", ["dot", "distance"])
def test_values(ca, shape, ws, nheads, cplx, simname):
    """A's values: written by the forward where a warp's rows fit, else by a second sweep; and the raw scores of the similarity."""
    rng = np.random.default_rng(63)
    qn, kn, vn = (randn(rng, shape, cplx) for _ in range(3))
    sim = ca.DotSimilarity() if simname == "dot" else ca.DistanceSimilarity()
    q, k, v = (ca.jl.from_numpy(t) for t in (qn, kn, vn))
    y, A = ca.circulant_mh_attention(sim, q, k, v, ws, nheads)
    yo, nzo = orc.mh_attention(KIND[simname], up(qn), up(kn), up(vn), ws, nheads)
    assert_close(ca.jl.to_numpy(y), yo, "y")
    assert_close(ca.jl.to_numpy(A.nzVal), nzo, "A")
    if nheads == 1:
        S = ca.circulant_similarity(sim, q, k, ws)
        assert_close(ca.jl.to_numpy(S.nzVal), orc.similarity(KIND[simname], up(qn), up(kn), ws), "scores")


@pytest.mark.parametrize("c", [24, 48])
def test_wide_entmax_backward_launches(ca, c):
    """Units past one slab take the operator chain at once: no pack is made for the fused sweeps they do not have."""
    rng = np.random.default_rng(64)
    q, k, v = (ca.jl.from_numpy(randn(rng, (20, 18, c, 1))).requires_grad_(True) for _ in range(3))
    y, _ = ca.circulant_attention(ca.DotSimilarity(), q, k, v, 5, normalizer=ca.ENTMAX15, return_A=False)
    n0 = ca.lib.ca_probe_launch_count()
    y.sum().backward()
    assert ca.lib.ca_probe_launch_count() - n0 == 12      # scores, weights, dv, dP, dS, dq, dk, and five packs


@pytest.mark.parametrize("spatial,ws,c,units,cplx", [
    ((32, 32), 7, 16, 1, False),      # whole rows: one column, stages in four
    ((75, 53), 9, 12, 3, False),      # whole rows at their limit for one slab, rows past the image
    ((38, 31), 11, 32, 2, False),     # two slabs, at the limit of the window
    ((41, 30), 7, 32, 2, True),       # four slabs, an odd last column, every alignment of a row
    ((131,), 21, 40, 2, False),       # folded signal, short last column
    ((75, 53), 11, 16, 3, False),     # runs, stages in three
    ((60, 40), 21, 16, 2, False),     # runs, stages in four
    ((39, 45), 13, 32, 2, False),     # loose runs of the transposed form (39 rows), two slabs
])
def test_apply_cuts(ca, spatial, ws, c, units, cplx):
    """A (x) v, its transpose and, for Distance, the pullback that subtracts the row sums times the centre."""
    rng = np.random.default_rng(65)
    K = ws ** len(spatial)
    nzn = rng.standard_normal((int(np.prod(spatial)) * K, units)).astype(np.float32)
    xn, yn = randn(rng, spatial + (c, units), cplx), randn(rng, spatial + (c, units), cplx)
    nz, x = ca.jl.from_numpy(np.asfortranarray(nzn)), ca.jl.from_numpy(xn)
    dS = up(nzn).reshape((K, -1, units), order="F")
    for transpose in (False, True):
        assert_close(ca.jl.to_numpy(ca.ops.apply(nz, x, ws, transpose)), orc.apply(dS, up(xn), ws, transpose), f"transpose {transpose}")
    xt, yt = ca.jl.from_numpy(xn).requires_grad_(True), ca.jl.from_numpy(yn).requires_grad_(True)
    S = ca.circulant_similarity(ca.DistanceSimilarity(), xt, yt, ws)
    S.nzVal.backward(nz.reshape(S.nzVal.shape) if S.nzVal.shape != nz.shape else nz)
    dxo, dyo = orc.similarity_pullback(orc.DISTANCE, up(xn), up(yn), ws, dS)
    # a sum of K differences of O(1) vectors: the centre enters with the sum of K weights
    assert_close(ca.jl.to_numpy(xt.grad), dxo, "dx")
    assert_close(ca.jl.to_numpy(yt.grad), dyo, "dy")


@pytest.mark.parametrize("shape,ws", [
    ((513, 8, 300), 97),      # 600 blocks of four pixels per thread, a block of one pixel at the end of each signal
    ((515, 6, 80), 33),       # 160: entmax with four, softmax with two
    ((513, 16, 100), 33),     # 16 channels, 200 blocks: forward with four
    ((514, 12, 4), 99),       # two everywhere
])
@pytest.mark.parametrize("norm", ["softmax", "entmax"])
def test_line_pixels(ca, shape, ws, norm):
    """1-D kernels with two and with four pixels per thread."""
    rng = np.random.default_rng(66)
    qn, kn, vn, rn = (randn(rng, shape) for _ in range(4))
    q, k, v = (ca.jl.from_numpy(t).requires_grad_(True) for t in (qn, kn, vn))
    y, _ = ca.circulant_attention(ca.DistanceSimilarity(), q, k, v, ws, normalizer=ca.ENTMAX15 if norm == "entmax" else ca.SOFTMAX, return_A=False)
    (y * ca.jl.from_numpy(rn)).sum().backward()
    which = orc.ENTMAX15 if norm == "entmax" else orc.SOFTMAX
    for u in (0, shape[-1] // 2, shape[-1] - 1):
        one = slice(u, u + 1)
        qo, ko, vo, ro = (up(t[..., one]) for t in (qn, kn, vn, rn))
        yo, _ = orc.attention(orc.DISTANCE, qo, ko, vo, ws, which)
        dqo, dko, dvo = orc.attention_pullback(orc.DISTANCE, qo, ko, vo, ws, ro, None, which)
        for name, got, want in (("y", y, yo), ("dq", q.grad, dqo), ("dk", k.grad, dko), ("dv", v.grad, dvo)):
            assert_close(ca.jl.to_numpy(got)[..., one], want, f"{name} of unit {u}")


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("shape,ws,cplx", [
    ((100, 53, 64, 4), 5, False),      # the weights of the dq sweep stored: an odd last column, rows past the image
    ((75, 70, 40, 4), 7, False),       # 40 channels in four slabs
    ((71, 71, 32, 4), 9, True),        # complex, three columns do not divide the width
    ((41, 37, 64, 14), 17, False),     # the largest window whose weights are stored
    ((41, 37, 64, 14), 19, False),     # past it: recomputed
])
def test_wide_backward(ca, shape, ws, cplx, simname):
    rng = np.random.default_rng(67)
    qn, kn, vn, rn = (randn(rng, shape, cplx) for _ in range(4))
    q, k, v = (ca.jl.from_numpy(t).requires_grad_(True) for t in (qn, kn, vn))
    sim = ca.DotSimilarity() if simname == "dot" else ca.DistanceSimilarity()
    y, _ = ca.circulant_attention(sim, q, k, v, ws, return_A=False)
    r = ca.jl.from_numpy(rn)
    ((y * r.conj()).real.sum() if cplx else (y * r).sum()).backward()
    for u in (0, shape[-1] - 1):
        one = slice(u, u + 1)
        dqo, dko, dvo = orc.attention_pullback(KIND[simname], *(up(t[..., one]) for t in (qn, kn, vn)), ws, up(rn[..., one]))
        for name, got, want in (("dq", q.grad, dqo), ("dk", k.grad, dko), ("dv", v.grad, dvo)):
            assert_close(ca.jl.to_numpy(got)[..., one], want, f"{name} of unit {u}")
