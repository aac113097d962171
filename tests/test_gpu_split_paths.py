"""Every way into the tensor-core sweeps: each count of tiles a column and each storage, the separately callable stages of the band
mode, buffers with guards around them, repeated runs; each test asserts that the sweeps ran."""
import contextlib

import numpy as np
import pytest
import torch

from oracle import circatt_oracle as orc
from tests.helpers import KIND, assert_close, elem_err, randn, up
from tests.test_gpu_band import ext_cols
from tests.test_gpu_interop import _guarded, _intact
from tests.test_gpu_split import oracle, run, sim_of

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def sweeps(ca, n):
    """The block launches n sweeps on the tensor cores."""
    before = ca.lib.ca_probe_tensor_launch_count()
    yield
    assert ca.lib.ca_probe_tensor_launch_count() - before == n


def test_small_problems_stay_on_the_fma_kernels(ca):
    rng = np.random.default_rng(80)
    with sweeps(ca, 0):
        run(ca, "dot", *(randn(rng, (40, 33, 32, 2)) for _ in range(4)), 9, 2)


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("ws", [9, 13, 25])                  # two, three and four tiles a column
@pytest.mark.parametrize("per_head", [8, 16])
def test_bfloat16_storage(ca, per_head, ws, simname):
    """Against the oracle on the same (rounded) tensors, next to the FMA kernels, which take two heads at a time.  Rounding y to 8 bits
    and dy . y with it leaves the gradients errors of 2e-3 (norm) to 2e-2 (an element) on either pipe; the Float32 arithmetic in
    between is 1e-6, so the two must agree in their errors to some percent."""
    rng = np.random.default_rng(81)
    shape, heads = (43, 58, 8 * per_head, 1), 8
    t = [torch.from_numpy(randn(rng, shape)).to(torch.bfloat16).float().numpy() for _ in range(4)]

    def run_heads(first, n):
        q, k, v, r = (ca.jl.from_numpy(np.asfortranarray(x[:, :, first * per_head:(first + n) * per_head])).to(torch.bfloat16) for x in t)
        q, k, v = (x.requires_grad_(True) for x in (q, k, v))
        y, _ = ca.circulant_mh_attention(sim_of(ca, simname), q, k, v, ws, n, return_A=False)
        return [ca.jl.to_numpy(x.detach().float()) for x in (y,) + torch.autograd.grad(y, (q, k, v), r)]

    with sweeps(ca, 3):
        got = run_heads(0, heads)
    with sweeps(ca, 0):
        fma = [np.concatenate(x, axis=2) for x in zip(*(run_heads(h, 2) for h in range(0, heads, 2)))]
    want = oracle(simname, *t, ws, heads)
    for name, a, b in zip(("y", "dq", "dk", "dv"), got, fma):
        w = want[name]
        norm = lambda x: np.linalg.norm(x - w) / np.linalg.norm(w)
        assert norm(a) < 3e-3 and norm(a) < 1.02 * norm(b), (name, norm(a), norm(b))
        assert elem_err(a, w) < 1.1 * elem_err(b, w), (name, elem_err(a, w), elem_err(b, w))


@pytest.mark.parametrize("which", ["k", "v", "r"])
def test_bfloat16_beside_a_large_pixel(ca, which):
    rng = np.random.default_rng(82)
    shape, ws, heads, pix = (57, 54, 64, 1), 13, 4, (30, 25)
    t = dict(zip("qkvr", (torch.from_numpy(randn(rng, shape)).to(torch.bfloat16).float().numpy() for _ in range(4))))
    t[which][pix][:16] *= np.float32(2.0 ** 30)
    q, k, v, r = (ca.jl.from_numpy(np.asfortranarray(x)).to(torch.bfloat16) for x in t.values())
    q, k, v = (x.requires_grad_(True) for x in (q, k, v))
    with sweeps(ca, 3):
        y, _ = ca.circulant_mh_attention(ca.DotSimilarity(), q, k, v, ws, heads, return_A=False)
        grads = torch.autograd.grad(y, (q, k, v), r)
    want = oracle("dot", *t.values(), ws, heads)
    d = np.maximum(np.abs(np.arange(57) - pix[0])[:, None], np.abs(np.arange(54) - pix[1])[None])
    for name, got in zip(("y", "dq", "dk", "dv"), (y,) + grads):
        far = 12 if name in ("dk", "dv") and which in "kv" else 6
        near = (d > far) & (d <= far + 9)
        assert_close(ca.jl.to_numpy(got.detach().float())[near][:, :16], want[name][near][:, :16], name, tol=1e-2, elem_tol=2e-2)


@pytest.mark.parametrize("simname", ["dot", "distance"])
@pytest.mark.parametrize("shape,ws,nheads,world,wild", [((70, 95, 80, 1), 9, 5, 1, False),       # one odd band: two halos of the same image
                                                        ((61, 101, 96, 1), 13, 6, 2, False),     # bands of 51 and 50 columns
                                                        ((64, 78, 128, 1), 21, 8, 2, False),
                                                        ((61, 101, 96, 1), 13, 6, 2, True)])     # and the recomputing paths
def test_bands(ca, shape, ws, nheads, world, wild, simname):
    """The stages that a band of the image calls, key side with halo columns (Wk = W + 2p), against the whole image."""
    rng = np.random.default_rng(83)
    p, kind = ws // 2, KIND[simname]
    qn, kn, vn, rn = (randn(rng, shape) for _ in range(4))
    if wild:
        vn *= (10.0 ** rng.integers(-3, 4, (shape[0] // 8 + 1, shape[1], 1, 1)).repeat(8, axis=0)[:shape[0]]).astype(np.float32)
    yo, _ = orc.mh_attention(kind, up(qn), up(kn), up(vn), ws, nheads)
    want = dict(zip(("dq", "dk", "dv"), orc.mh_attention_pullback(kind, up(qn), up(kn), up(vn), ws, nheads, up(rn))), y=yo)
    qs, ks, vs, rs = (orc.splitheads(t, nheads) for t in (qn, kn, vn, rn))
    plan = ca.parallel.BandPlan(shape[1], world, ws)
    ops, jl = ca.ops, ca.jl
    outs = {n: [] for n in ("y", "dq", "dk", "dv", "stats", "D")}

    def cut(rank):
        start, width = plan.band(rank)
        band = lambda t: jl.from_numpy(np.asfortranarray(t[:, start:start + width]))
        ext = lambda t: jl.from_numpy(ext_cols(t, start, width, p))
        return start, width, band, ext

    for rank in range(world):
        start, width, band, ext = cut(rank)
        q, k, v, dy = band(qs), band(ks), band(vs), band(rs)
        k_ext, v_ext = ext(ks), ext(vs)
        with sweeps(ca, 2):
            y, _, stats = ops.attention_fwd(kind, 0, q, k_ext, v_ext, ws, False, band=(width + 2 * p, p))
            D = ops.attention_bwd_pre(kind, 0, q, k, v, y, dy, stats, ws)
            dq = ops.attention_bwd_dq(kind, 0, q, k_ext, v_ext, dy, stats, D, ws, band=(width + 2 * p, p))
        outs["y"].append(jl.to_numpy(y)); outs["dq"].append(jl.to_numpy(dq))
        outs["stats"].append(jl.to_numpy(stats).reshape((shape[0], width, -1), order="F"))
        outs["D"].append(jl.to_numpy(D).reshape((shape[0], width, -1), order="F"))
    stats_full, D_full = (np.concatenate(outs[n], axis=1) for n in ("stats", "D"))
    for rank in range(world):
        start, width, band, ext = cut(rank)
        flat = lambda t: jl.from_numpy(np.asfortranarray(ext_cols(t, start, width, p).reshape((-1, t.shape[-1]), order="F")))
        with sweeps(ca, 1):
            dk, dv = ops.attention_bwd_dkdv(kind, 0, ext(qs), band(ks), band(vs), ext(rs), flat(stats_full), flat(D_full), ws,
                                            band=(width + 2 * p, p))
        outs["dk"].append(jl.to_numpy(dk)); outs["dv"].append(jl.to_numpy(dv))
    for name in ("y", "dq", "dk", "dv"):
        got = np.concatenate(outs[name], axis=1).reshape(shape, order="F")
        assert_close(got, want[name], name, **(dict(elem_tol=1e-3) if wild else {}))       # rms over six orders says little of an element


@pytest.mark.parametrize("wild", [False, True])
@pytest.mark.parametrize("shape,ws,nheads,with_a", [((33, 61, 112, 1), 9, 7, True), ((70, 45, 40, 1), 25, 5, False), ((70, 91, 32, 2), 13, 2, True)])
def test_outputs_and_workspaces_stay_inside_their_buffers(ca, shape, ws, nheads, with_a, wild):
    lib, ops, jl = ca.lib, ca.ops, ca.jl
    rng = np.random.default_rng(84)
    q, k, v, dy = (randn(rng, shape) for _ in range(4))
    if wild:
        v[::16] *= np.float32(1e6)                    # every warp recomputes
    q, k, v, dy = (ca.splitheads(jl.from_numpy(t), nheads) for t in (q, k, v, dy))
    m = ops.meta_of(q, ws)
    d = m.desc(scale=1.0 / np.sqrt(m.channels))
    st = torch.cuda.current_stream().cuda_stream
    P = ops.ptr
    gy, y, py, ny = _guarded(ca, tuple(q.shape))
    gs, stats, ps, nst = _guarded(ca, (m.Np, m.units))
    ga, A, pa, na = _guarded(ca, (m.K * m.Np, m.units)) if with_a else (None, None, 0, 0)
    nfw, nbw = lib.ca_attention_fwd_workspace(d, int(with_a)), lib.ca_attention_bwd_workspace(d, 0)
    gw, wsf, pw, nw = _guarded(ca, (nfw,), torch.uint8, fill=77)
    gb, wsb, pb, nb = _guarded(ca, (nbw,), torch.uint8, fill=77)
    grads = [_guarded(ca, tuple(q.shape)) for _ in range(3)]
    with sweeps(ca, 3 + with_a):
        ca._lib.check(lib.ca_attention_fwd(d, P(q), P(k), P(v), P(y), P(A) if with_a else None, P(stats), P(wsf), st))
        ca._lib.check(lib.ca_attention_bwd(d, P(q), P(k), P(v), P(y), P(dy), P(stats), None, None,
                                           P(grads[0][1]), P(grads[1][1]), P(grads[2][1]), P(wsb), P(wsf), st))
    torch.cuda.synchronize()
    assert _intact(gy, py, ny) and _intact(gs, ps, nst)
    assert bool((gw[:pw] == 77).all()) and bool((gw[pw + nw:] == 77).all())
    assert bool((gb[:pb] == 77).all()) and bool((gb[pb + nb:] == 77).all())
    for buf, view, pad, n in grads + [(gy, y, py, ny)] + ([(ga, A, pa, na)] if with_a else []):
        assert _intact(buf, pad, n)
        assert bool(torch.isfinite(view).all()) and not bool((view == buf[0]).any())


@pytest.mark.parametrize("wild", [False, True])
def test_repeated_runs_are_equal(ca, wild):
    rng = np.random.default_rng(85)
    t = [randn(rng, (57, 54, 64, 1)) for _ in range(4)]
    if wild:
        t[2][::16] *= np.float32(1e6)
    with sweeps(ca, 8):
        a, b = (run(ca, "dot", *t, 13, 4, want_a=True) for _ in range(2))
    for name in a:
        assert np.array_equal(a[name], b[name]), name
