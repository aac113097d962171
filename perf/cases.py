"""Performance cases of the framework: what its users have it do, through the public API.

A case is a dict of plain values:

    kind   "train"      y = attention(q, k, v) and the gradients of q, k, v for a given cotangent of y
           "infer"      y = attention(q, k, v) without gradients
           "mix"        z = (a*A + (1-a)*B) applied to v, A and B two adjacencies, and the gradients of every input
           "apply"      a stored adjacency applied to x, plain and transposed
           "algebra"    C = A + m .* A2 on stored adjacencies, C applied to u, and the row sums of C
    dtype  "f32", "c64" (ComplexF32) or "bf16" (storage of the fused attention)
    H, W   spatial extents; W = 0: a 1-D signal of length H
    C, B   channels of all heads, batch
    ws, heads
    sim    "dot" or "distance"
    norm   "softmax" or "entmax"
    A      whether the adjacency is returned (written to memory) besides y

`prepare` makes what a program holds before the call, `run` makes one pass, `work` gives the bytes and operations
that a pass cannot do without, `tolerance` how far two correct implementations may differ."""
import math

import torch

from __graft_entry__ import load_package

ca = load_package()

DTYPES = {"f32": torch.float32, "c64": torch.complex64, "bf16": torch.bfloat16}


def _case(kind, dtype, H, W, C, B, ws, heads, sim="dot", norm="softmax", A=False, name=None):
    case = dict(kind=kind, dtype=dtype, H=H, W=W, C=C, B=B, ws=ws, heads=heads, sim=sim, norm=norm, A=A)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # The smallest problem of the benchmark's configurations, with the adjacency returned: a first model, a
        # unit test, a shallow layer on a thumbnail.  Latency and launches count.
        _case("train", "f32", 32, 32, 16, 1, 7, 1, A=True, name="thumbnail train"),
        # The quickstart layer: the training step that the headline metric is quoted on.
        _case("train", "f32", 128, 96, 64, 2, 15, 4, name="quickstart train"),
        # The same layer in evaluation, Distance similarity, adjacency returned for reuse in later layers.
        _case("infer", "f32", 128, 96, 64, 2, 15, 4, sim="distance", A=True, name="quickstart infer with A"),
        # An image whose extents, batch and channels per head (12) are no multiples of anything.
        _case("train", "f32", 75, 53, 36, 3, 11, 3, name="ragged image train"),
        # A batch of short records of odd length in evaluation (1-D, softmax).
        _case("infer", "f32", 5001, 0, 32, 3, 63, 4, name="records infer"),
        # Long 1-D signals, long window, sparse normaliser (which draw() gives images too).
        _case("train", "f32", 16384, 0, 64, 16, 127, 8, sim="distance", norm="entmax", name="signals entmax train"),
        # MRI-style complex feature maps, one head, adjacency returned.
        _case("train", "c64", 320, 320, 32, 8, 7, 1, A=True, name="complex maps train"),
        # What such a model does with its adjacencies between layers.
        _case("algebra", "c64", 320, 320, 32, 8, 7, 1, name="complex maps algebra"),
        # The quickstart layer's adjacency, computed once and applied in the layers that follow.
        _case("apply", "f32", 128, 96, 64, 2, 15, 4, name="stored adjacency apply"),
        # Two adjacencies mixed and applied, with every gradient (the pattern of group-sparse denoisers).
        _case("mix", "f32", 96, 80, 32, 2, 9, 2, name="mixed adjacency train"),
        # A large image, evaluation from bfloat16 tensors and training in Float32.
        _case("infer", "bf16", 1024, 1024, 128, 1, 21, 8, name="large image infer bf16"),
        _case("train", "f32", 1024, 1024, 128, 1, 21, 8, name="large image train"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choice(("train", "train", "train", "train", "infer", "infer", "infer", "mix", "apply", "algebra"))
    one_d = rng.random() < 0.3
    # channels per head: the usual powers of two, and now and then a width that is none
    per_head = rng.choice((4, 8, 8, 12, 16, 16, 16, 24, 32, 48, 64))
    heads = rng.choice((1, 1, 2, 3, 4, 8))
    dtype = "f32"
    if kind in ("train", "infer", "algebra") and rng.random() < 0.25:
        dtype = "c64"
        per_head = max(2, per_head // 2)
    elif kind in ("train", "infer") and not one_d and rng.random() < 0.25:
        dtype = "bf16"                       # storage of softmax attention on images at 8 or 16 channels per head
        per_head = rng.choice((8, 16))
    sim = rng.choice(("dot", "dot", "distance"))
    norm = "entmax" if kind in ("train", "infer") and dtype != "bf16" and rng.random() < 0.25 else "softmax"
    want_a = kind in ("train", "infer") and dtype != "bf16" and rng.random() < 0.3
    B = _log_int(rng, 1, 8)
    stored = want_a or kind in ("mix", "apply", "algebra")
    if one_d:
        H, W = _log_int(rng, 256, 8192 if stored else 32768), 0
        ws = 2 * _log_int(rng, 4, 63) + 1
    else:
        H, W = _log_int(rng, 24, 256 if stored else 512), _log_int(rng, 24, 256 if stored else 512)
        ws = 2 * _log_int(rng, 2, 10) + 1
    # no more than the largest listed case in arithmetic, and adjacencies of at most half a gigabyte
    K = ws if one_d else ws * ws
    while True:
        pixels = H * (W or 1) * B
        if pixels * K * per_head * heads <= 2e10 and not (stored and pixels * K * heads > 1.25e8):
            break
        if B > 1:
            B = (B + 1) // 2
        elif heads > 1:
            heads = (heads + 1) // 2
        else:
            H = max(24, H // 2)
    return _case(kind, dtype, H, W, per_head * heads, B, ws, heads, sim, norm, want_a)


# ------------------------------------------------------------------------------------------------ one pass
class _State:
    pass


def _spatial(case):
    return (case["H"], case["W"]) if case["W"] else (case["H"],)


def prepare(case, seed):
    """Standard normal tensors, as the benchmark and the tests use; the stored adjacencies of "apply" and "algebra"
    are adjacencies of such tensors."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFF)
    dtype = DTYPES[case["dtype"]]
    shape = _spatial(case) + (case["C"], case["B"])

    def randn(grad=False):
        t = ca.jl.randn(*shape, dtype=torch.float32 if dtype is torch.bfloat16 else dtype, generator=gen)
        return t.to(dtype).requires_grad_(grad)

    s = _State()
    s.kind, s.ws, s.heads, s.want_a = case["kind"], case["ws"], case["heads"], case["A"]
    s.sim = ca.DotSimilarity() if case["sim"] == "dot" else ca.DistanceSimilarity()
    s.norm = ca.ENTMAX15 if case["norm"] == "entmax" else ca.SOFTMAX
    if s.kind == "train":
        s.q, s.k, s.v = randn(True), randn(True), randn(True)
        s.dy = randn()
    elif s.kind == "infer":
        s.q, s.k, s.v = randn(), randn(), randn()
    elif s.kind == "mix":
        s.x, s.y, s.v = randn(True), randn(True), randn(True)
        s.dz = randn()
    else:
        with torch.no_grad():
            s.adj = [ca.circulant_mh_adjacency(s.sim, randn(), randn(), s.ws, s.heads)
                     for _ in range(1 if s.kind == "apply" else 2)]
        s.x = randn()
        if s.kind == "algebra":
            s.m = ca.jl.randn(1, 1, 1, case["B"], generator=gen)
    return s


def run(s):
    if s.kind == "train":
        y, A = ca.circulant_mh_attention(s.sim, s.q, s.k, s.v, s.ws, s.heads, normalizer=s.norm, return_A=s.want_a)
        out = {"y": y, "grads": torch.autograd.grad(y, (s.q, s.k, s.v), s.dy)}
        if s.want_a:
            out["A"] = A.nzVal
        return out
    if s.kind == "infer":
        with torch.no_grad():
            y, A = ca.circulant_mh_attention(s.sim, s.q, s.k, s.v, s.ws, s.heads, normalizer=s.norm,
                                             return_A=s.want_a)
        return {"y": y, "A": A.nzVal} if s.want_a else {"y": y}
    if s.kind == "mix":
        A = ca.circulant_mh_adjacency(ca.DotSimilarity(), s.x, s.y, s.ws, s.heads)
        B = ca.circulant_mh_adjacency(ca.DistanceSimilarity(), s.y, s.y, s.ws, s.heads)
        z = ca.Otimes(0.8 * A + 0.2 * B, s.v)
        return {"z": z, "grads": torch.autograd.grad(z, (s.x, s.y, s.v), s.dz)}
    with torch.no_grad():
        if s.kind == "apply":
            return {"z": ca.Otimes(s.adj[0], s.x), "zt": ca.circulant_mh_transposed_attention(s.adj[0], s.x)}
        C = s.adj[0] + ca.scale(s.m, s.adj[1])
        return {"C": C.nzVal, "z": ca.Otimes(C, s.x), "rows": ca.sum(C, dims=2)}


# ------------------------------------------------------------------------------------------------ bounds
def work(case):
    """Window terms: 2 operations per term and real channel for each contraction (scores, applications, and their
    pullbacks), 1 more for the Distance; every input read once, every output written once."""
    pixels = case["H"] * (case["W"] or 1) * case["B"]
    K = case["ws"] ** (2 if case["W"] else 1)
    C = case["C"] * (2 if case["dtype"] == "c64" else 1)
    dense = pixels * case["C"] * {"f32": 4, "c64": 8, "bf16": 2}[case["dtype"]]
    adjacency = pixels * K * case["heads"] * 4
    terms = pixels * K * C
    extra = 1 if case["sim"] == "distance" else 0
    kind = case["kind"]
    if kind == "train":
        return {"bytes": 8 * dense + adjacency * case["A"], "flops": (14 + 2 * extra) * terms}
    if kind == "infer":
        return {"bytes": 4 * dense + adjacency * case["A"], "flops": (4 + extra) * terms}
    if kind == "mix":
        # two scores and one application forward, two pullbacks of each backward; x, y, v, dz in, z and gradients out
        return {"bytes": 8 * dense, "flops": 19 * terms}
    if kind == "apply":
        return {"bytes": adjacency + 3 * dense, "flops": 4 * terms}
    return {"bytes": 3 * adjacency + 2 * dense, "flops": 2 * terms + 3 * pixels * K * case["heads"]}


def tolerance(case):
    """Sums of Float32 products in another order; results rounded to bfloat16 where that is the storage."""
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 1e-5, "max": 1e-3}
