"""Shapes at the edges of the tiled and 1-D kernels' dispatch: channel counts that are zero-extended to 16, 32 or 64, 1-D
signals whose folded last column is short, stored values applied at every alignment, rows at the limits of the row
kernels' register shapes, columns per thread of the forward, and the classes of the first entmax threshold."""
import numpy as np
import pytest

from oracle import circatt_oracle as orc
from tests.helpers import KIND, TOL, assert_close, randn, rel_err, up

pytestmark = pytest.mark.gpu


def sim_of(ca, name):
    return ca.DotSimilarity() if name == "dot" else ca.DistanceSimilarity()


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("shape,ws,nheads,cplx,tiled", [
    ((19, 18, 24, 2), 5, 2, False, 3),       # 12 channels per head in one slab
    ((33, 21, 5, 1), 7, 1, False, 3),        # odd channel count
    ((20, 17, 48, 1), 9, 2, False, 3),       # 24 in two slabs
    ((17, 19, 48, 1), 7, 1, False, 3),       # 48 in four slabs
    ((18, 16, 9, 2), 5, 1, True, 3),         # 9 complex = 18 real channels
    ((290, 40, 1), 53, 1, False, 3),         # folded signal with a short last column, 40 channels
    ((131, 20, 2), 7, 1, False, 3),          # three pixels in the last column
    ((100, 33, 1), 99, 1, False, 3),         # one ragged column, the window almost the signal
])
def test_zero_extended_units_and_short_columns(ca, shape, ws, nheads, cplx, tiled, simname):
    rng = np.random.default_rng(41)
    qn, kn, vn, rn = (randn(rng, shape, cplx) for _ in range(4))
    q, k, v = (ca.jl.from_numpy(t).requires_grad_(True) for t in (qn, kn, vn))
    n0 = ca.lib.ca_probe_tiled_launch_count()
    y, A = ca.circulant_mh_attention(sim_of(ca, simname), q, k, v, ws, nheads)
    r = ca.jl.from_numpy(rn)
    ((y * r.conj()).real.sum() if cplx else (y * r).sum()).backward()
    assert ca.lib.ca_probe_tiled_launch_count() - n0 >= tiled           # forward, A and the two backward sweeps
    yo, nzo = orc.mh_attention(KIND[simname], up(qn), up(kn), up(vn), ws, nheads)
    dqo, dko, dvo = orc.mh_attention_pullback(KIND[simname], up(qn), up(kn), up(vn), ws, nheads, up(rn))
    for name, got, want in (("y", y, yo), ("A", A.nzVal, nzo), ("dq", q.grad, dqo), ("dk", k.grad, dko), ("dv", v.grad, dvo)):
        assert_close(ca.jl.to_numpy(got), want, name)


@pytest.mark.parametrize("spatial,ws,c,units", [
    ((16, 16), 15, 16, 2),      # extent == window + 1, the whole image in one tile: rows wrap on both sides
    ((39, 17), 5, 8, 3),        # height no multiple of four: wrapped rows change their alignment
    ((66, 21), 13, 16, 1),      # tile rows past the image
    ((34, 31), 29, 16, 1),      # eight pieces per run
    ((40, 33), 31, 16, 1),      # nine
    ((48, 9), 9, 40, 2),        # four slabs
    ((291,), 21, 16, 2),        # folded, short last column
    ((130,), 127, 20, 1),       # folded, two pixels in the last column, long window
])
def test_stored_values_applied(ca, spatial, ws, c, units):
    rng = np.random.default_rng(42)
    K = ws ** len(spatial)
    nzn = rng.standard_normal((int(np.prod(spatial)) * K, units)).astype(np.float32)
    xn = randn(rng, spatial + (c, units))
    nz, x = ca.jl.from_numpy(np.asfortranarray(nzn)), ca.jl.from_numpy(xn)
    for transpose in (False, True):
        n0 = ca.lib.ca_probe_tiled_launch_count()
        got = ca.ops.apply(nz, x, ws, transpose)
        assert ca.lib.ca_probe_tiled_launch_count() == n0 + 1
        want = orc.apply(up(nzn).reshape((K, -1, units), order="F"), up(xn), ws, transpose)
        assert rel_err(ca.jl.to_numpy(got), want) < TOL, transpose


@pytest.mark.parametrize("spatial,ws", [((9,), 9), ((16,), 15), ((40,), 31), ((34,), 33), ((70,), 65), ((131,), 129), ((300,), 257),
                                        ((21, 22), 21), ((600,), 513)])
def test_rows_at_the_limits_of_the_row_kernels(ca, spatial, ws):
    """Rows of 9 to 513 entries: every register shape, and the loop kernels past 512."""
    rng = np.random.default_rng(43)
    K = ws ** len(spatial)
    rows = int(np.prod(spatial))
    sn = np.asfortranarray(rng.standard_normal((rows * K, 3)).astype(np.float32))
    dn = np.asfortranarray(rng.standard_normal((rows * K, 3)).astype(np.float32))
    s, d = ca.jl.from_numpy(sn), ca.jl.from_numpy(dn)
    z = up(sn).reshape((K, rows, 3), order="F")
    e = np.exp(z - z.max(axis=0))
    p = e / e.sum(axis=0)
    got, stats = ca.ops.row_normalize(s, spatial, ws, 0, want_stats=True)
    assert rel_err(ca.jl.to_numpy(got), p.reshape((rows * K, 3), order="F")) < TOL
    assert rel_err(ca.jl.to_numpy(stats), z.max(axis=0) + np.log(e.sum(axis=0))) < TOL
    pe = orc.row_entmax15(z.copy())
    got_e = ca.ops.row_normalize(s, spatial, ws, 1)
    assert rel_err(ca.jl.to_numpy(got_e), pe.reshape((rows * K, 3), order="F")) < TOL
    dp = up(dn).reshape((K, rows, 3), order="F")
    ds = p * (dp - (p * dp).sum(axis=0))
    back = ca.ops.row_normalize_bwd(got, d, spatial, ws, 0)
    assert rel_err(ca.jl.to_numpy(back), ds.reshape((rows * K, 3), order="F")) < TOL
    assert rel_err(ca.jl.to_numpy(ca.ops.sum_rows(s, spatial, ws)), z.sum(axis=0)[:, None, :]) < TOL


@pytest.mark.parametrize("shape,ws", [
    ((30, 25, 16, 17), 11),     # 153 warps of three-column tiles: one column in the last tile
    ((30, 26, 16, 17), 13),     # two
    ((30, 27, 8, 17), 21),      # full tiles, chunks of seven
    ((30, 26, 16, 10), 15),     # fewer warps than SMs: two columns per thread
    ((32, 33, 32, 66), 11),     # two slabs, 1188 warps of four-column tiles, one column in the last
    ((17, 19, 64, 2), 11),      # four slabs, three columns per thread
])
def test_forward_column_tiles(ca, shape, ws):
    rng = np.random.default_rng(44)
    qn, kn, vn = (randn(rng, shape) for _ in range(3))
    y, _ = ca.circulant_attention(ca.DotSimilarity(), *(ca.jl.from_numpy(t) for t in (qn, kn, vn)), ws, return_A=False)
    units = range(0, shape[-1], max(1, shape[-1] // 4))
    for u in units:
        one = slice(u, u + 1)
        yo, _ = orc.attention(orc.DOT, up(qn[..., one]), up(kn[..., one]), up(vn[..., one]), ws)
        assert_close(ca.jl.to_numpy(y)[..., one], yo, f"y of unit {u}")


@pytest.mark.parametrize("c", [8, 16])
@pytest.mark.parametrize("ws", [5, 7, 9, 11, 13, 15, 17, 19, 33])
def test_entmax_first_threshold(ca, ws, c):
    """1-D windows of every remainder modulo the classes the first threshold is taken from; units of ordinary rows, of
    equal scores (everything in the support) and of one score far above the others (nothing else in it)."""
    rng = np.random.default_rng(45)
    qn, kn, vn = (randn(rng, (141, c, 3)) for _ in range(3))
    kn[..., 1] = kn[:1, :, 1]
    qn[..., 2] = 1.0
    kn[::ws + 1, :, 2] += 6.0
    y, _ = ca.circulant_attention(ca.DotSimilarity(), *(ca.jl.from_numpy(t) for t in (qn, kn, vn)), ws,
                                  normalizer=ca.ENTMAX15, return_A=False)
    for u in range(3):
        one = slice(u, u + 1)
        yo, _ = orc.attention(orc.DOT, up(qn[..., one]), up(kn[..., one]), up(vn[..., one]), ws, orc.ENTMAX15)
        assert_close(ca.jl.to_numpy(y)[..., one], yo, f"y of unit {u}")
