"""Timed cases of the solver: what a user's program has it do, through the public classes.

A case is a dict of plain values. `kind` names the entry point:

  solve      Solver.solve: charges on the GPU -> q_i phi_i, one particle set, tree kept
  gradient   fmm_phi forward and backward: phi, dL/dq, dL/dx (`save`: fields or recompute)
  adaptive   AdaptiveSolver.solve: clustered particles, heavy leaves refined
  batch      Batch.solve: many independent sets of uneven sizes in one call
  direct     the FP64 direct sum on sampled targets, the check of a solve

`n` is the Chebyshev order (4 or 8), `mode` the precision (d FP64, s FP32, mixed), `depth` the
leaf level, `layout` the positions (uniform in the cube, or Gaussian clusters clipped to it).
"""
import math

import torch

from bbfmm_b200 import AdaptiveSolver, Batch, Solver, batch_depth
from bbfmm_b200.autograd import fmm_phi
from bbfmm_b200.fmm import direct

DEVICE = "cuda:0"


def _case(name, kind, N, n=8, mode="mixed", depth=0, layout="uniform", **more):
    return dict(name=name, kind=kind, N=N, n=n, mode=mode, depth=depth, layout=layout, **more)


def listed():
    return [
        # a small molecule-sized set solved again and again: launches and latency count
        _case("solve-d4-4k", "solve", 4096, n=4, mode="d", depth=3),
        # the plain configuration: FP64, n = 4, about 8 particles a leaf
        _case("solve-d4-32k", "solve", 32768, n=4, mode="d", depth=4),
        # low order in FP32 over many particles (quick potentials of a large set)
        _case("solve-s4-1m", "solve", 1048576, n=4, mode="s", depth=6),
        # FP64 at high order, the accuracy run
        _case("solve-d8-262k", "solve", 262144, n=8, mode="d", depth=5),
        # FP32 at high order, an odd count of clustered particles
        _case("solve-s8-100k", "solve", 100003, n=8, mode="s", depth=4, layout="clusters"),
        # the mixed precision solve of a middling set
        _case("solve-mixed8-262k", "solve", 262144, depth=5),
        # the headline: four million particles, n = 8, depth 7
        _case("solve-mixed8-4m", "solve", 4194304, depth=7),
        # a training or fitting step: potentials, then gradients in charges and positions
        _case("gradient-mixed8-1m", "gradient", 1048576, depth=6, layout="clusters", save="fields"),
        # the same in FP32 at low order with nothing kept between the passes
        _case("gradient-s4-60k", "gradient", 60013, n=4, mode="s", depth=4, layout="clusters", save="recompute"),
        # strongly clustered particles on a two-level adaptive tree
        _case("adaptive-mixed8-500k", "adaptive", 500009, depth=4, fine=6, layout="clusters"),
        # many uneven sets, half uniform and half clustered, n = 4 and 8 mixed
        _case("batch-mixed-24", "batch", 24, depth=0, layout="uneven", largest=65536),
        # another kernel of the same solver (x / r^3) in FP64
        _case("solve-force-d8-30k", "solve", 30011, n=8, mode="d", depth=4, kernel="laplacianforce"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve"] * 5 + ["gradient", "adaptive", "batch", "direct"])
    if kind == "direct":
        return dict(kind="direct", N=_log(rng, 20000, 500000), targets=_log(rng, 100, 4096), n=0, mode="d", depth=0,
                    layout=rng.choice(["uniform", "clusters"]))
    if kind == "batch":
        return dict(kind="batch", N=rng.randint(5, 30), n=0, mode=rng.choice(["mixed", "mixed", "d", "s"]), depth=0,
                    layout="uneven", largest=_log(rng, 8192, 65536))
    if kind == "adaptive":
        depth = rng.choice([3, 4])
        return dict(kind="adaptive", N=_log(rng, 100000, 800000), n=8, mode="mixed", depth=depth, fine=depth + 2,
                    layout="clusters")
    n = rng.choice([4, 8])
    mode = rng.choice(["d", "s", "mixed", "mixed"]) if n == 8 else rng.choice(["d", "s"])
    layout = rng.choice(["uniform", "uniform", "clusters"])
    # about 2 to 60 particles a leaf; the high-order FP64 and FP32 sets stay below depth 6
    top = 3000000 if mode == "mixed" and layout == "uniform" else (300000 if n == 8 and mode != "mixed" else 1000000)
    if kind == "gradient":
        top = min(top, 500000)
    N = _log(rng, 3000, top)
    most = 7 if mode == "mixed" else (5 if n == 8 else 6)
    depth = min(most, batch_depth(N, rng.choice([4.0, 8.0, 32.0, 32.0])))
    c = dict(kind=kind, N=N, n=n, mode=mode, depth=depth, layout=layout)
    if kind == "gradient":
        c["save"] = rng.choice(["fields", "recompute"])
    elif rng.random() < 0.2:
        c["kernel"] = rng.choice(["laplacianforce", "oneoverr4"])
    return c


def _positions(g, N, layout):
    """(N, 3) FP64 positions in [-1/2, 1/2)^3 on the GPU."""
    x = torch.rand(N, 3, generator=g, device=DEVICE, dtype=torch.float64)
    if layout == "clusters":
        c = 0.15 + 0.7 * torch.rand(8, 3, generator=g, device=DEVICE, dtype=torch.float64)
        which = torch.randint(0, 8, (N,), generator=g, device=DEVICE)
        x = c[which] + 0.05 * torch.randn(N, 3, generator=g, device=DEVICE, dtype=torch.float64)
        x = x.clamp_(0.0, math.nextafter(1.0, 0.0))
    return x - 0.5


def _charges(g, N):
    return 2.0 * torch.rand(N, generator=g, device=DEVICE, dtype=torch.float64) - 1.0


def _dtype(case):
    return torch.float32 if case["mode"] == "s" else torch.float64


def _sizes(case):
    """(particles, order, depth) of the batch's sets: sizes evenly spread over the logarithm
    from 1,000 to `largest`, n = 4 and 8 in turn by pairs."""
    out = []
    for k in range(case["N"]):
        f = (k * 0.6180339887498949) % 1.0
        N = int(round(1000 * (case["largest"] / 1000) ** f))
        out.append((N, 4 if k // 2 % 2 else 8, batch_depth(N)))
    return out


def _sets(case, g):
    """The batch's sets, every other one clustered."""
    return [(_positions(g, N, "clusters" if k % 2 else "uniform").to(_dtype(case)), n, depth)
            for k, (N, n, depth) in enumerate(_sizes(case))]


def _inputs(case, seed):
    """Positions and charges (and the loss weights of a gradient case), rounded to the case's
    precision: the solve and the exact sum take the same numbers."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    d = {}
    if case["kind"] == "batch":
        d["sets"] = _sets(case, g)
        N = sum(x.shape[0] for x, _, _ in d["sets"])
    else:
        N = case["N"]
        d["x"] = _positions(g, N, case["layout"]).to(_dtype(case))
    d["q"] = _charges(g, N).to(_dtype(case))
    if case["kind"] == "gradient":
        d["w"] = torch.randn(N, generator=g, device=DEVICE, dtype=torch.float64).to(_dtype(case))
    if case["kind"] == "direct":
        d["targets"] = torch.randperm(N, generator=g, device=DEVICE)[: case["targets"]].to(torch.int32)
    return d


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    if kind == "batch":
        s["solver"] = Batch(s["sets"], mode=case["mode"])
        s["out"] = torch.empty_like(s["q"])
    elif kind == "adaptive":
        s["solver"] = AdaptiveSolver(case["n"], case["depth"], case["fine"], mode=case["mode"])
        s["solver"].set_particles(s["x"])
    elif kind != "direct":
        s["solver"] = Solver(case["n"], case["depth"], mode=case["mode"], kernel=case.get("kernel", "laplacian"))
        s["solver"].set_particles(s["x"])
    if kind == "gradient":
        s["q"].requires_grad_()
        s["x"].requires_grad_()
    return s


def run(state):
    kind = state["case"]["kind"]
    if kind == "direct":
        return direct(state["x"], state["q"], state["targets"])
    if kind == "batch":
        return state["solver"].solve(state["q"], out=state["out"])
    if kind == "gradient":
        q, x = state["q"], state["x"]
        phi = fmm_phi(state["solver"], q, x, save=state["case"]["save"])
        dq, dx = torch.autograd.grad(phi, (q, x), state["w"])
        return phi.detach(), dq, dx
    return state["solver"].solve(state["q"])


def _far_flops(n, depth):
    """Expansion work of one solve: per cell of levels 2 .. depth the two projections (2 n^3 r
    each) and the M2L. A cell has up to 189 translations of 2 r^2; those of mirrored offsets are
    equal up to the signs of the components' parities and fold to 39.5 of them."""
    r, n3 = n ** 3 // 2, n ** 3
    cells = sum(8 ** l for l in range(2, depth + 1))
    return cells * (39.5 * 2 * r * r + 2 * 2 * n3 * r)


def work(case):
    """Each input read once, each output written once (positions, charges, results and the
    operators); operations of the expansions and about 10 a near-field pair."""
    kind, N = case["kind"], case["N"]
    size = 4 if case["mode"] == "s" else 8
    if kind == "direct":
        return {"bytes": 32.0 * N + 12.0 * case["targets"], "flops": 10.0 * N * case["targets"]}
    if kind == "batch":
        sets = _sizes(case)
        ops = 56 * size * (32 ** 2 + 256 ** 2)
        return {"bytes": float(sum(N for N, _, _ in sets) * 5 * size + ops),
                "flops": sum(_far_flops(n, depth) + 270.0 * N * N / 8 ** depth for N, n, depth in sets)}
    r = case["n"] ** 3 // 2
    # particles a leaf and its 26 neighbours see: at least the uniform density's
    pairs = 27.0 * N * N / 8 ** case.get("fine", case["depth"])
    values = 4 + 1 + (5 if kind == "gradient" else 0)
    passes = 2 if kind == "gradient" else 1
    return {"bytes": float(values * size * N + 56 * size * r * r),
            "flops": passes * (_far_flops(case["n"], case["depth"]) + 10.0 * pairs)}


def tolerance(case):
    """Two correct solves of the same operators differ by the rounding of their sums: FP64 sums,
    FP32 sums (cancelling charges), and in the mixed mode the split products."""
    if case["kind"] == "direct":
        return {"rel": 1e-12}
    if case["kind"] == "gradient":  # the field loses digits to cancellation of near pairs
        return {"rel": {"d": 1e-11, "s": 2e-4, "mixed": 5e-6}[case["mode"]]}
    return {"rel": {"d": 1e-12, "s": 1.5e-5, "mixed": 3e-7}[case["mode"]]}


# The most pairs that exact() sums (about ten seconds).
MOST_PAIRS = 3.2e11


def _sum(x, charges, targets, kernel="laplacian", field=False):
    """For each charge vector: sum_{j != i} c_j K(x_j - x_i) at the targets, and the gradient of
    the potential there (1/r)."""
    pots = [torch.empty(targets.numel(), dtype=torch.float64, device=DEVICE) for _ in charges]
    flds = [torch.empty(targets.numel(), 3, dtype=torch.float64, device=DEVICE) for _ in charges]
    N = x.shape[0]
    step = max(1, 60000000 // N)
    for a in range(0, targets.numel(), step):
        t = targets[a:a + step].long()
        d = [x[None, :, k] - x[t, k][:, None] for k in range(3)]
        rr = d[0] * d[0]
        rr.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
        rinv = rr.rsqrt_().masked_fill_(rr.isinf(), 0.0)
        if kernel == "laplacianforce":
            k = d[0] * rinv ** 3
        elif kernel == "oneoverr4":
            k = rinv ** 4
        else:
            k = rinv
        for c, p, f in zip(charges, pots, flds):
            p[a:a + step] = k @ c
            if field:
                r3 = rinv ** 3
                for e in range(3):
                    f[a:a + step, e] = (r3 * d[e]) @ c
    return pots, flds


def exact(case, seed):
    """The direct sums in 64 bits; a solve is off them by the truncation of its order too."""
    d = _inputs(case, seed)
    kind = case["kind"]
    q = d["q"].double()
    if kind == "batch":
        out, at = [], 0
        for x, _, _ in d["sets"]:
            c = q[at:at + x.shape[0]]
            at += x.shape[0]
            out.append(c * _sum(x.double(), [c], torch.arange(x.shape[0], device=DEVICE))[0][0])
        return torch.cat(out)
    x, N = d["x"].double(), case["N"]
    if kind == "direct":
        t = d["targets"].long()
        return q[t] * _sum(x, [q], t)[0][0]
    if float(N) * N * (4 if kind == "gradient" else 1) > MOST_PAIRS:
        return None
    every = torch.arange(N, device=DEVICE)
    if kind == "gradient":
        w = d["w"].double()
        (p, p2), (f, f2) = _sum(x, [q, w * q], every, field=True)
        return q * p, w * p + p2, q[:, None] * (w[:, None] * f + f2)
    return q * _sum(x, [q], every, case.get("kernel", "laplacian"))[0][0]
