"""The tensor-core sweeps (tcgen05 on exact bf16 splits) against the float64 oracle: every streamed-row count, ragged
tiles, windows as wide as the image, complex units, narrow units, bfloat16 storage, large scores, and that their error is
that of Float32 arithmetic."""
import numpy as np
import pytest
import torch

from oracle import circatt_oracle as orc
from tests.helpers import KIND, assert_close, randn, rel_err, up

pytestmark = pytest.mark.gpu


def sim_of(ca, name):
    return ca.DotSimilarity() if name == "dot" else ca.DistanceSimilarity()


def step(ca, simname, arrays, ws, nheads, return_A=False, dtype=None):
    q, k, v, r = (ca.jl.from_numpy(t) if dtype is None else ca.jl.from_numpy(t).to(dtype) for t in arrays)
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    y, A = ca.circulant_mh_attention(sim_of(ca, simname), q, k, v, ws, nheads, return_A=return_A)
    grads = torch.autograd.grad(y, (q, k, v), r)
    ca.ops.check_status()
    return y, A, grads


# at least one tile of 8 x 16 pixels per SM: 32 or more units at these extents
@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("shape,ws,nheads,cplx", [
    ((16, 17, 32, 20), 3, 2, False),        # 16 streamed rows; one column in the second tile
    ((21, 16, 64, 13), 9, 4, False),        # 16 rows, full; ragged tile rows
    ((17, 33, 24, 10), 11, 2, False),       # 24 rows, 12 channels per head
    ((24, 20, 10, 26), 17, 2, False),       # 24 rows, full; 5 channels
    ((19, 19, 32, 13), 19, 2, False),       # 32 rows, window as wide as the image
    ((26, 30, 16, 20), 25, 1, False),       # 32 rows, full
    ((28, 27, 32, 10), 27, 2, False),       # 40 rows
    ((33, 34, 8, 11), 33, 1, False),        # 40 rows, full: the widest window
    ((18, 20, 16, 13), 7, 2, True),         # 8 complex channels per head
    ((16, 40, 6, 26), 13, 1, True),         # 6 complex channels
])
def test_tensor_core_sweeps_match_oracle(ca, shape, ws, nheads, cplx, simname):
    rng = np.random.default_rng(51)
    arrays = [randn(rng, shape, cplx) for _ in range(4)]
    n0 = ca.lib.ca_probe_tiled_launch_count()
    y, A, grads = step(ca, simname, arrays, ws, nheads, return_A=True)
    assert ca.lib.ca_probe_tiled_launch_count() - n0 == 5               # forward, A; dv, dk, dq
    a64 = [up(t) for t in arrays]
    yo, nzo = orc.mh_attention(KIND[simname], *a64[:3], ws, nheads)
    want = orc.mh_attention_pullback(KIND[simname], *a64[:3], ws, nheads, a64[3])
    assert_close(ca.jl.to_numpy(y), yo, "y")
    assert_close(ca.jl.to_numpy(A.nzVal), nzo, "A")
    for name, got, w in zip(("dq", "dk", "dv"), grads, want):
        assert_close(ca.jl.to_numpy(got), w, name)


def test_error_is_that_of_float32(ca):
    """Root-mean-square error against float64 of a few 2^-24: the split operands carry all 24 bits."""
    rng = np.random.default_rng(52)
    arrays = [randn(rng, (24, 32, 64, 8)) for _ in range(4)]
    y, _, grads = step(ca, "dot", arrays, 15, 4)
    a64 = [up(t) for t in arrays]
    yo, _ = orc.mh_attention(orc.DOT, *a64[:3], 15, 4)
    want = orc.mh_attention_pullback(orc.DOT, *a64[:3], 15, 4, a64[3])
    for name, got, w in zip(("y", "dq", "dk", "dv"), (y,) + grads, (yo,) + want):
        e = ca.jl.to_numpy(got) - w
        assert np.sqrt((e ** 2).mean() / (w ** 2).mean()) < 6e-7, name


def test_large_scores_and_retained_graph(ca):
    """Scores in the hundreds (the reference of the exponentials moves often), and a second pullback of one graph."""
    rng = np.random.default_rng(53)
    shape, ws = (16, 32, 64, 13), 9
    qn, kn, vn, rn = (randn(rng, shape, scale=s) for s in (8.0, 8.0, 1.0, 1.0))
    q, k, v = (ca.jl.from_numpy(t).requires_grad_(True) for t in (qn, kn, vn))
    y, _ = ca.circulant_mh_attention(ca.DotSimilarity(), q, k, v, ws, 4, return_A=False)
    r = ca.jl.from_numpy(rn)
    first = torch.autograd.grad(y, (q, k, v), r, retain_graph=True)
    second = torch.autograd.grad(y, (q, k, v), r)
    assert all(torch.equal(a, b) for a, b in zip(first, second))
    yo, _ = orc.mh_attention(orc.DOT, up(qn), up(kn), up(vn), ws, 4)
    want = orc.mh_attention_pullback(orc.DOT, up(qn), up(kn), up(vn), ws, 4, up(rn))
    assert rel_err(ca.jl.to_numpy(y), yo) < 1e-4                          # one float32 ulp of a score is 1e-5 in exp()
    for got, w in zip(first, want):
        assert rel_err(ca.jl.to_numpy(got), w) < 1e-4


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("shape,ws,nheads", [((17, 20, 32, 20), 7, 2), ((24, 18, 32, 20), 15, 4), ((22, 21, 16, 20), 21, 1)])
def test_bfloat16_on_the_tensor_cores(ca, shape, ws, nheads, simname):
    rng = np.random.default_rng(54)
    arrays = [randn(rng, shape) for _ in range(4)]
    y, _, grads = step(ca, simname, arrays, ws, nheads, dtype=torch.bfloat16)
    a64 = [up(ca.jl.to_numpy(ca.jl.from_numpy(t).to(torch.bfloat16).float())) for t in arrays]
    yo, _ = orc.mh_attention(KIND[simname], *a64[:3], ws, nheads)
    want = orc.mh_attention_pullback(KIND[simname], *a64[:3], ws, nheads, a64[3])
    for got, w in zip((y,) + grads, (yo,) + want):
        assert got.dtype == torch.bfloat16 and rel_err(ca.jl.to_numpy(got.float()), w) < 1e-2
