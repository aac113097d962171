"""The tensor-core sweeps (split halves): tile edges of rows, columns and windows, storage kinds, groups of eight rows whose
magnitudes differ, references that move, and values that are no numbers.

Bars: the usual ones.  A split operand keeps 22 to 24 bits of an element down to 2^-13 of the largest of its group of eight rows and 16
channels, and steps of 2^-36 of that largest below; the products and sums are Float32's.  The magnitudes below vary by less
than 2^13 within a group, except for zeros."""
import numpy as np
import pytest
import torch

from oracle import circatt_oracle as orc
from tests.helpers import KIND, assert_close, randn, up

pytestmark = pytest.mark.gpu


def sim_of(ca, name):
    return ca.DotSimilarity() if name == "dot" else ca.DistanceSimilarity()


def run(ca, simname, qn, kn, vn, rn, ws, heads, want_a=False):
    q, k, v = (ca.jl.from_numpy(t).requires_grad_(True) for t in (qn, kn, vn))
    y, A = ca.circulant_mh_attention(sim_of(ca, simname), q, k, v, ws, heads, return_A=want_a)
    grads = torch.autograd.grad(y, (q, k, v), ca.jl.from_numpy(rn))
    out = dict(zip(("y", "dq", "dk", "dv"), (y,) + grads))
    if want_a:
        out["A"] = A.nzVal
    return {name: ca.jl.to_numpy(t.detach()) for name, t in out.items()}


def oracle(simname, qn, kn, vn, rn, ws, heads):
    y, nz = orc.mh_attention(KIND[simname], up(qn), up(kn), up(vn), ws, heads)
    dq, dk, dv = orc.mh_attention_pullback(KIND[simname], up(qn), up(kn), up(vn), ws, heads, up(rn))
    return {"y": y, "A": nz, "dq": dq, "dk": dk, "dv": dv}


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("shape,ws,heads,cplx", [
    ((41, 40, 128, 1), 7, 8, False),     # dk/dv only; two tiles a column; one row past a warp's eight, rows past a block's 32
    ((64, 33, 96, 1), 9, 6, False),      # 16 keys exactly, an odd number of columns
    ((39, 47, 84, 1), 11, 7, False),     # three tiles, 12 channels
    ((17, 91, 72, 1), 17, 9, False),     # rows equal to the window: every row wraps; the longest of three tiles; 8 channels
    ((33, 47, 56, 1), 19, 8, False),     # four tiles, 7 channels
    ((65, 32, 32, 3), 25, 2, False),     # the longest window; batch of three
    ((40, 76, 32, 1), 13, 4, True),      # 8 complex channels
    ((47, 65, 20, 1), 9, 4, True),       # 5 complex channels
])
def test_edges(ca, shape, ws, heads, cplx, simname):
    rng = np.random.default_rng(61)
    t = [randn(rng, shape, cplx) for _ in range(4)]
    got = run(ca, simname, *t, ws, heads, want_a=True)
    want = oracle(simname, *t, ws, heads)
    for name in got:
        assert_close(got[name], want[name], name)


@pytest.mark.parametrize("what", ["pixels", "zeros", "small", "large", "scores"])
def test_magnitudes(ca, what):
    rng = np.random.default_rng(62)
    shape, ws, heads = (57, 54, 64, 1), 11, 4
    q, k, v, r = (randn(rng, shape) for _ in range(4))
    if what == "pixels":                     # every pixel another power of two: the groups of a step rarely share their scale
        for t, span in ((q, 1), (k, 1), (v, 5), (r, 5)):
            t *= (2.0 ** rng.integers(-span, span + 1, shape[:2] + (1, 1))).astype(np.float32)
    elif what == "zeros":                    # padding
        for t in (q, k, v, r):
            t[:, :9] = 0
            t[20:37] = 0
    elif what == "small":
        v *= 1e-12
        r *= 1e-9
    elif what == "large":
        v *= 1e9
        r *= 1e7
    else:                                    # scores of a thousand: the references move, rows are one-hot
        q *= 30
        k[:, ::3] *= 8
    got = run(ca, "dot", q, k, v, r, ws, heads, want_a=True)
    want = oracle("dot", q, k, v, r, ws, heads)
    # an ulp of a score of a thousand is already 1e-4 in the exponential
    bars = dict(tol=2e-3, elem_tol=2e-2) if what == "scores" else {}
    for name in got:
        assert_close(got[name], want[name], name, **bars)


def test_gradients_of_few_channels_and_a_short_window(ca):
    """Few terms leave the rounding of the weights itself: of s - L (up to 8: 2.4e-7 at most, ln 2 of that in the weight), of L
    twice, of the exponential and of the split, 1e-7 rms each, and the cut sums.  A binade more in the exponent shows."""
    rng = np.random.default_rng(67)
    shape, ws, heads = (50, 64, 64, 1), 9, 8
    t = [randn(rng, shape) for _ in range(4)]
    got, want = run(ca, "dot", *t, ws, heads), oracle("dot", *t, ws, heads)
    for name in ("dq", "dk", "dv"):
        err = np.linalg.norm(got[name] - want[name]) / np.linalg.norm(want[name])
        assert err < 4.2e-7, f"{name}: {err:.3g}"


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("which,mul", [("r", 1e-20), ("r", 1e-30), ("r", 1e20), ("v", 1e-20), ("v", 1e20)])
def test_norms_whose_squares_are_no_floats(ca, which, mul, simname):
    """The weights of the gradients are scaled by a bound that follows from the norms of dy and v, whose squares leave the range
    of Float32 long before the tensors do."""
    rng = np.random.default_rng(65)
    shape, ws, heads = (57, 54, 64, 1), 11, 4
    t = dict(zip("qkvr", (randn(rng, shape) for _ in range(4))))
    t[which] *= np.float32(mul)
    got = run(ca, simname, *t.values(), ws, heads)
    want = oracle(simname, *t.values(), ws, heads)
    for name in got:
        assert_close(got[name], want[name], name)


def test_pixels_with_small_cotangents(ca):
    """dq of a pixel is as accurate as its own dy, however small."""
    rng = np.random.default_rng(66)
    shape, ws, heads = (57, 54, 64, 1), 11, 4
    q, k, v, r = (randn(rng, shape) for _ in range(4))
    small = rng.random(shape[:2]) < 0.1
    r[small] *= np.float32(1e-20)
    dq, want = run(ca, "dot", q, k, v, r, ws, heads)["dq"], oracle("dot", q, k, v, r, ws, heads)["dq"]
    assert_close(dq[small], want[small], "dq of the small")
    assert_close(dq[~small], want[~small], "dq of the others")


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_what_is_no_number_stays_in_its_windows(ca, bad):
    rng = np.random.default_rng(63)
    shape, ws, heads = (56, 74, 48, 1), 9, 3
    q, k, v, r = (randn(rng, shape) for _ in range(4))
    clean = run(ca, "dot", q, k, v, r, ws, heads, want_a=True)
    v[30, 20, 5, 0] = bad                    # head 0
    got = run(ca, "dot", q, k, v, r, ws, heads, want_a=True)
    near = np.zeros(shape[:2], bool)         # pixels whose window holds the element
    near[26:35, 16:25] = True
    assert not np.isfinite(got["y"][26:35, 16:25, 5, 0]).any()
    assert_close(got["A"], clean["A"], "A")
    assert_close(got["y"][~near], clean["y"][~near], "y")
    far = np.ones(shape[:2], bool)           # gradients reach two windows
    far[22:39, 12:29] = False
    for name in ("dq", "dk", "dv"):
        assert_close(got[name][far], clean[name][far], name)
    for name in ("y", "dq", "dk", "dv"):     # and no other head
        assert_close(got[name][:, :, 16:], clean[name][:, :, 16:], name)


def test_bfloat16_storage(ca):
    rng = np.random.default_rng(64)
    shape, ws, heads = (50, 62, 64, 1), 15, 4
    t = [torch.from_numpy(randn(rng, shape)).to(torch.bfloat16).float().numpy() for _ in range(4)]
    q, k, v, r = (ca.jl.from_numpy(np.asfortranarray(x)).to(torch.bfloat16) for x in t)
    q, k, v = (x.requires_grad_(True) for x in (q, k, v))
    y, _ = ca.circulant_mh_attention(ca.DotSimilarity(), q, k, v, ws, heads, return_A=False)
    grads = torch.autograd.grad(y, (q, k, v), r)
    want = oracle("dot", *t, ws, heads)
    for name, got in zip(("y", "dq", "dk", "dv"), (y,) + grads):
        # results are rounded to 8 bits, dy . y is formed from the rounded y
        assert_close(ca.jl.to_numpy(got.detach().float()), want[name], name, tol=1e-2, elem_tol=2e-2)
