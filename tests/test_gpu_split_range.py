"""The tensor-core sweeps on tensors whose magnitudes differ: values that are large, small or too large for their scores cost the
other pixels nothing.  The bars are the usual ones, over pixels that do not see the value."""
import numpy as np
import pytest

from oracle import circatt_oracle as orc
from tests.helpers import assert_close, randn
from tests.test_gpu_split import oracle, run

pytestmark = pytest.mark.gpu

SHAPE, WS, HEADS = (57, 54, 64, 1), 11, 4
PIX = (30, 25)


def tensors(seed, shape=SHAPE):
    rng = np.random.default_rng(seed)
    return dict(zip("qkvr", (randn(rng, shape) for _ in range(4))))


def ring(least, most):
    """Pixels whose distance from PIX is above `least` and up to `most`."""
    d = np.maximum(np.abs(np.arange(SHAPE[0]) - PIX[0])[:, None], np.abs(np.arange(SHAPE[1]) - PIX[1])[None])
    return (d > least) & (d <= most)


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("which,mul", [("q", 1e4), ("q", 1e12), ("k", 1e4), ("k", 1e12), ("v", 1e3), ("v", 1e4), ("v", 1e6), ("v", 1e12),
                                       ("r", 1e3), ("r", 1e4), ("r", 1e6), ("r", 1e12)])
def test_a_large_pixel(ca, which, mul, simname):
    t = tensors(71)
    t[which][PIX][:16] *= np.float32(mul)              # head 0
    got, want = run(ca, simname, *t.values(), WS, HEADS, want_a=True), oracle(simname, *t.values(), WS, HEADS)
    p = WS // 2
    for name in ("y", "dq", "dk", "dv"):
        # k and v reach the gradients of keys through every window that holds the pixel
        far = 2 * p if name in ("dk", "dv") and which in "kv" else p
        near = ring(far, far + 9)
        assert_close(got[name][near][:, :16], want[name][near][:, :16], name)
        assert_close(got[name][:, :, 16:], want[name][:, :, 16:], name + " of the other heads")


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("which", ["q", "k", "v", "r"])
def test_a_small_channel(ca, which, simname):
    """Gradients and y of a channel are as accurate as the channel itself.  (Not dq of a small channel of k under the Distance: it is
    sum dS k - q sum dS, where the second sum is zero but for rounding and q is not small; 64 bits are needed for either kernel.)"""
    t = tensors(72)
    t[which][:, :, 3::16] *= np.float32(1e-6)
    got, want = run(ca, simname, *t.values(), WS, HEADS), oracle(simname, *t.values(), WS, HEADS)
    for name in got:
        if (which, simname, name) == ("k", "distance", "dq"):
            continue
        assert_close(got[name][:, :, 3::16], want[name][:, :, 3::16], name)


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("mul", [20, 3000])
@pytest.mark.parametrize("each", [10, 13])
def test_between_large_lines(ca, each, mul, simname):
    """Every group of eight rows that a warp meets may hold a large row, and the windows between the lines none.  A Float32 sum of 81
    terms of mixed signs, of weights with some 2^-22 of error each, is within 1e-6 of its norm."""
    t, ws = tensors(77), 9
    for name in "vr":
        t[name][::each] *= np.float32(mul)
    got, want = run(ca, simname, *t.values(), ws, HEADS), oracle(simname, *t.values(), ws, HEADS)
    lines = np.zeros(SHAPE[0], bool)
    lines[::each] = True
    between = ~np.any([np.roll(lines, d) for d in range(-(ws // 2), ws // 2 + 1)], axis=0)
    assert between.any()
    for name in got:
        err = np.linalg.norm(got[name][between] - want[name][between]) / np.linalg.norm(want[name][between])
        assert err < 1e-6, f"{name}: {err:.3g}"


@pytest.mark.parametrize("which", ["k", "v", "r"])
def test_a_large_half(ca, which):
    t = tensors(73)
    t[which][:, :SHAPE[1] // 2] *= np.float32(300 if which == "k" else 1e5)
    got, want = run(ca, "dot", *t.values(), WS, HEADS), oracle("dot", *t.values(), WS, HEADS)
    p = WS // 2
    for name in got:
        far = 2 * p if name in ("dk", "dv") and which in "kv" else 0 if which == "r" and name in ("y", "dq") else p
        cols = slice(SHAPE[1] // 2 + far, SHAPE[1] - far)
        assert_close(got[name][:, cols], want[name][:, cols], name)


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("mul", [1e-20, 1e-28])
def test_small_scores_operands(ca, mul, simname):
    """q below the least scale; k makes up for it in the Dot's scores."""
    t = tensors(74)
    t["q"] *= np.float32(mul)
    t["k"] *= np.float32(1 / mul if simname == "dot" else 1)
    got, want = run(ca, simname, *t.values(), WS, HEADS, want_a=True), oracle(simname, *t.values(), WS, HEADS)
    for name in got:
        assert_close(got[name], want[name], name)


def test_scores_that_overflow_stay_in_their_windows(ca):
    t = tensors(75)
    clean = oracle("dot", *t.values(), WS, HEADS)
    for name in "qk":
        t[name][PIX][:16] *= np.float32(1e20)
    got = run(ca, "dot", *t.values(), WS, HEADS, want_a=True)
    p = WS // 2
    for name in ("y", "dq", "dk", "dv"):
        far = ring(2 * p if name in ("dk", "dv") else p, 99)
        assert_close(got[name][far], clean[name][far], name)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("which", ["q", "k", "r"])
def test_what_is_no_number_stays_in_its_windows(ca, which, simname, bad):
    t = tensors(76)
    clean = oracle(simname, *t.values(), WS, HEADS)
    t[which][PIX][5] = bad
    got = run(ca, simname, *t.values(), WS, HEADS, want_a=True)
    p = WS // 2
    for name in ("y", "dq", "dk", "dv"):
        far = ring(2 * p if name in ("dk", "dv") and which == "k" else p, 99)
        assert_close(got[name][far], clean[name][far], name)
        assert_close(got[name][:, :, 16:], clean[name][:, :, 16:], name + " of the other heads")
    if which == "r":
        assert not np.isfinite(got["dq"][PIX][:16]).any()
        assert_close(got["A"], clean["A"], "A")
    if which == "q":
        assert not np.isfinite(got["y"][PIX][:16]).any()
