"""Performance cases of the FMM force backend.

Each case is one pass of a program that uses the library through its Python package
(``GpuContext``): a force evaluation from host arrays, a run of leapfrog steps, a tree
build, a gradient, a rollout with its reverse sweep, or the exact sampled sum of a
validation.  Sizes, presets, orders and leaf sizes are those of the benchmark's
configurations and of the tests, and the ranges between them.

Case fields: ``op`` (what a pass does), ``preset`` and ``n`` (the bodies), ``p`` and
``n_max`` (expansion order, bodies per leaf), ``form`` ("ref": the reference's lists in
FP64, the library's default; "fp64" and "mixed": the opening-angle lists), ``split``
(near-list split 0.4 and body-level P2L 0.3, as the benchmark runs them), ``pinned``
(page-locked host arrays), ``steps``, ``dt``, ``rebuild`` (leapfrog), ``samples``.

The mixed form computes forces in FP32, so a program keeps what is made of them alone
(accelerations, velocities, gradients) as float32; positions and everything of the other
forms stay float64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import galax_gb300 as G
from galax_gb300 import presets

THETA, THETA_W, THETA_B = 0.5, 0.4, 0.3


def listed():
    return [
        # the smallest call: the drop-in default (REF, FP64) on the reference's demo size
        dict(name="forces_ref_1k", op="forces", preset="uniform", n=1000, p=4, n_max=32, form="ref", split=False,
             pinned=False),
        # the uniform configuration: ten leapfrog steps on a static tree, drop-in form and mixed form
        dict(name="kdk_ref_10k", op="kdk", preset="uniform", n=10_000, p=4, n_max=32, form="ref", split=False,
             steps=10, dt=0.01, rebuild=0),
        dict(name="kdk_mixed_10k", op="kdk", preset="uniform", n=10_000, p=4, n_max=32, form="mixed", split=True,
             steps=10, dt=0.01, rebuild=0),
        # the headline evaluation, mixed and FP64, host arrays in and out
        dict(name="forces_mixed_1m", op="forces", preset="plummer", n=1_000_000, p=4, n_max=32, form="mixed",
             split=True, pinned=True),
        dict(name="forces_fp64_1m", op="forces", preset="plummer", n=1_000_000, p=4, n_max=32, form="fp64",
             split=True, pinned=True),
        # the drop-in form on the galaxy configuration (odd size, one dominant mass), pageable arrays
        dict(name="forces_ref_200k", op="forces", preset="galaxy", n=200_001, p=4, n_max=32, form="ref", split=False,
             pinned=False),
        # the accuracy/throughput sweep's size at a high order with wide leaves
        dict(name="forces_disk_4m_p6", op="forces", preset="disk", n=4_000_000, p=6, n_max=64, form="mixed",
             split=True, pinned=True),
        # a run whose tree follows the bodies: rebuild and plan before every step's evaluation
        dict(name="kdk_rebuild_1m", op="kdk", preset="plummer", n=1_000_000, p=4, n_max=32, form="mixed", split=True,
             steps=10, dt=1e-3, rebuild=1),
        # tree build alone: upload, sort, tree; the permutation and the sorted bodies back on the host
        dict(name="build_200k", op="build", preset="disk", n=200_003, p=4, n_max=16, form="mixed", split=False),
        # the backward of one evaluation, FP64
        dict(name="vjp_fp64_20k", op="vjp", preset="galaxy", n=20_001, p=4, n_max=32, form="fp64", split=False),
        # trajectory gradient of the galaxy configuration: rollout and its reverse sweep, tree rebuilt every step
        dict(name="rollout_mixed_200k", op="rollout", preset="galaxy", n=200_001, p=4, n_max=32, form="mixed",
             split=False, steps=10, dt=2e-3, rebuild=1, every=4),
        # validation: the exact sum on 1000 sampled bodies
        dict(name="validate_1m", op="validate", preset="plummer", n=1_000_000, p=4, n_max=32, form="mixed",
             split=False, samples=1000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges; sizes spread over their logarithm, odd ones among them."""
    op = rng.choice(["forces"] * 6 + ["kdk"] * 2 + ["build", "vjp", "rollout", "validate"])
    preset = rng.choice(["uniform", "plummer", "disk", "galaxy"])
    form = rng.choice(["ref", "fp64", "mixed", "mixed"])
    c = dict(op=op, preset=preset, p=rng.choice([2, 4, 4, 6, 8]), n_max=rng.choice([16, 32, 32, 64]), form=form,
             split=form != "ref" and rng.random() < 0.6)
    if op == "forces":
        c.update(n=_log_int(rng, 500, 2_000_000 if form == "mixed" else 150_000), pinned=rng.random() < 0.5)
    elif op == "kdk":
        c.update(n=_log_int(rng, 500, 500_000 if form == "mixed" else 30_000), steps=rng.randint(2, 8), dt=1e-3,
                 rebuild=rng.randint(0, 1), p=min(c["p"], 4))
    elif op == "build":
        c.update(n=_log_int(rng, 500, 1_000_000), form="mixed", split=False)
    elif op == "vjp":
        c.update(n=_log_int(rng, 500, 300_000 if form == "mixed" else 20_000), split=False,
                 form="mixed" if form == "mixed" else "fp64", p=min(c["p"], 6))
    elif op == "rollout":
        c.update(n=_log_int(rng, 500, 100_000), steps=rng.randint(3, 9), dt=1e-3, rebuild=rng.randint(0, 1),
                 every=rng.randint(1, 4), form="mixed", split=False, p=min(c["p"], 4))
    else:
        c.update(n=_log_int(rng, 2_000, 1_000_000), samples=rng.randint(100, 1000), form="mixed", split=False)
    if form == "ref" and op in ("forces", "kdk"):
        c["p"] = min(c["p"], 6)
    return c


def _bodies(case, seed):
    return presets.make(case["preset"], case["n"], seed=seed)


def prepare(case, seed):
    b = _bodies(case, seed)
    bounds = presets.BOUNDS[case["preset"]]
    n = case["n"]
    ctx = G.GpuContext(G.GpuConfig(max_n=n, max_nodes=0, p=case["p"]))
    if case["form"] == "ref":
        ctx.set_mode(G.MODE_REF, G.PREC_FP64)
    else:
        ctx.set_mode(G.MODE_ACCURATE, G.PREC_MIXED if case["form"] == "mixed" else G.PREC_FP64, THETA)
    if case["split"]:
        ctx.set_near_split(THETA_W)
        ctx.set_body_split(THETA_B)
    s = dict(case=case, ctx=ctx, bounds=bounds)
    if case["op"] == "build":
        s.update(bodies=b, out=G.Bodies.new(n))
        return s
    ctx.build_tree(b, case["n_max"], bounds)  # sorts b into tree order
    ctx.set_params(case["p"], presets.cli_softening(b.x, b.y))
    s["bodies"] = b
    if case["op"] == "forces":
        arrs = [torch.zeros(n, dtype=torch.float64, pin_memory=case["pinned"]).numpy() for _ in range(5)]
        for a, v in zip(arrs, (b.x, b.y, b.mass)):
            a[:] = v
        s["arrays"] = arrs
    elif case["op"] in ("kdk", "rollout"):
        s["out"] = G.Bodies.new(n)
    elif case["op"] == "validate":
        s["idx"] = np.sort(np.random.default_rng(seed + 1).permutation(n)[:case["samples"]])
    if case["op"] in ("vjp", "rollout"):
        rng = np.random.default_rng(seed + 2)
        s["lam"] = [rng.standard_normal(n) for _ in range(2 if case["op"] == "vjp" else 4)]
    return s


def _kept(case, *arrays):
    """The arrays as the program keeps them: float32 where the mixed form computed them."""
    if case["form"] != "mixed":
        return list(arrays)
    return [torch.from_numpy(a).to(torch.float32) for a in arrays]


def run(s):
    case, ctx, op = s["case"], s["ctx"], s["case"]["op"]
    if op == "forces":
        ctx.compute_forces(*s["arrays"])
        return _kept(case, s["arrays"][3], s["arrays"][4])
    if op == "kdk":
        ctx.upload_bodies(s["bodies"])
        if case["rebuild"]:
            ctx.rebuild_resident(case["n_max"], s["bounds"])
        ctx.kdk_run(case["steps"], case["dt"], rebuild_every=case["rebuild"])
        o = s["out"]
        ctx.download_bodies(o)
        state = [o.x, o.y, o.vx, o.vy]
        if case["rebuild"]:  # back to the order of the upload
            ids = torch.from_numpy(ctx.body_ids())
            back = [torch.empty(len(ids), dtype=torch.float64) for _ in state]
            for t, a in zip(back, state):
                t[ids] = torch.from_numpy(a)
            state = [t.numpy() for t in back]
        return state[:2] + _kept(case, *state[2:])
    if op == "build":
        ctx.upload_bodies(s["bodies"])
        perm = ctx.rebuild_resident(case["n_max"], s["bounds"], want_perm=True)
        o = s["out"]
        ctx.download_bodies(o)
        return dict(perm=perm, counts=list(ctx.tree_info()), x=o.x, y=o.y, mass=o.mass)
    if op == "vjp":
        return _kept(case, *ctx.force_vjp(*s["lam"]))
    if op == "rollout":
        ctx.upload_bodies(s["bodies"])
        ctx.rebuild_resident(case["n_max"], s["bounds"])
        ctx.rollout_forward(case["steps"], case["dt"], case["every"], case["rebuild"])
        ctx.download_bodies(s["out"])
        grads = ctx.rollout_backward(*s["lam"])[:5]
        return _kept(case, s["out"].x, s["out"].y, *grads)
    return list(ctx.n2_sampled(s["idx"]))


def work(case):
    """Bytes of the arrays that go in and come out, and the operations of the pass: about
    2000 near interactions of 14 operations and 30 far pairs of 2 C(p)^2 a body and
    evaluation at theta = 0.5 (three times that for a gradient)."""
    n, nc = case["n"], (case["p"] + 1) * (case["p"] + 2) // 2
    per = n * (2000 * 14 + 30 * 2 * nc * nc)
    op = case["op"]
    if op == "forces":
        return {"bytes": 40 * n, "flops": per}
    if op == "kdk":
        return {"bytes": 72 * n, "flops": per * case["steps"]}
    if op == "build":
        return {"bytes": (24 + 24 + 8) * n, "flops": 0}
    if op == "vjp":
        return {"bytes": 64 * n, "flops": 4 * per}
    if op == "rollout":
        return {"bytes": 128 * n, "flops": 5 * per * case["steps"]}
    return {"bytes": 24 * n + 24 * case["samples"], "flops": 14 * n * case["samples"]}


# ---------------------------------------------------------------- the same in 64 bits, without the library

EXACT_PAIRS = 4.5e10  # direct sums up to this many pairs take under 20 seconds


def _sorted(case, seed):
    """The bodies of prepare() in Morton order: 21 bits a coordinate, x in the even bits, ties in input order."""
    b = _bodies(case, seed)
    x0, x1, y0, y1 = presets.BOUNDS[case["preset"]]

    def spread(v, lo, hi):
        v = (np.clip((v - lo) / (hi - lo), 0.0, 1.0 - 1e-15) * 2097152.0).astype(np.uint64)
        for sh, m in ((16, 0x0000FFFF0000FFFF), (8, 0x00FF00FF00FF00FF), (4, 0x0F0F0F0F0F0F0F0F),
                      (2, 0x3333333333333333), (1, 0x5555555555555555)):
            v = (v | (v << np.uint64(sh))) & np.uint64(m)
        return v

    o = np.argsort(spread(b.x, x0, x1) | (spread(b.y, y0, y1) << np.uint64(1)), kind="stable")
    return [v[o] for v in (b.x, b.y, b.mass, b.vx, b.vy)]


def _rows(n):
    return max(1, min(n, 100_000_000 // n))


def _direct(x, y, m, eps, targets=None):
    """sum_j m_j (x_j - x_i) / (r^2 + eps^2)^(3/2) over all bodies but i itself, whose term is zero
    (with eps = 0 it is taken out)."""
    tx, ty = (x, y) if targets is None else (x[targets], y[targets])
    ax, ay = torch.empty_like(tx), torch.empty_like(tx)
    step = _rows(len(x))
    for i in range(0, len(tx), step):
        dx, dy = x[None] - tx[i:i + step, None], y[None] - ty[i:i + step, None]
        r2 = dx * dx + dy * dy + eps * eps
        w = torch.where(r2 > 0, m[None] * r2 ** -1.5, torch.zeros_like(r2))
        ax[i:i + step], ay[i:i + step] = (w * dx).sum(1), (w * dy).sum(1)
    return ax, ay


def _direct_vjp(x, y, m, lx, ly, eps):
    """lam . d(a)/d(x, y, m) of _direct."""
    gx, gy, gm = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    step = max(1, _rows(len(x)) // 2)
    for i in range(0, len(x), step):
        k = slice(i, i + step)
        dx, dy = x[None] - x[k, None], y[None] - y[k, None]
        ir2 = 1.0 / (dx * dx + dy * dy + eps * eps)
        ir3 = ir2 * torch.sqrt(ir2)
        wx, wy = m[k, None] * lx[None] - m[None] * lx[k, None], m[k, None] * ly[None] - m[None] * ly[k, None]
        dw = 3.0 * ir2 * ir3 * (dx * wx + dy * wy)
        gx[k], gy[k] = (ir3 * wx - dw * dx).sum(1), (ir3 * wy - dw * dy).sum(1)
        gm[k] = -((lx[None] * dx + ly[None] * dy) * ir3).sum(1)
    return gx, gy, gm


def exact(case, seed):
    op, n = case["op"], case["n"]
    pairs = {"forces": n * n, "kdk": n * n * (1 + case.get("steps", 0)), "vjp": 4 * n * n,
             "validate": n * case.get("samples", 0)}.get(op, math.inf)
    if pairs > EXACT_PAIRS or (case["form"] == "ref" and op != "validate"):
        return None  # too long, or the reference's capped lists, which no direct sum gives
    if op == "kdk" and case["rebuild"] and case["preset"] == "galaxy":
        return None
    x, y, m, vx, vy = _sorted(case, seed)
    eps = presets.cli_softening(x, y)
    d = "cuda" if torch.cuda.is_available() else "cpu"
    x, y, m, vx, vy = (torch.from_numpy(np.ascontiguousarray(v)).to(d) for v in (x, y, m, vx, vy))
    if op == "forces":
        out = _direct(x, y, m, eps)
    elif op == "kdk":
        ax, ay = torch.zeros_like(x), torch.zeros_like(x)  # the uploaded accelerations
        h = 0.5 * case["dt"]
        for _ in range(case["steps"]):
            vx, vy = vx + h * ax, vy + h * ay
            x, y = x + case["dt"] * vx, y + case["dt"] * vy
            ax, ay = _direct(x, y, m, eps)
            vx, vy = vx + h * ax, vy + h * ay
        out = x, y, vx, vy
    elif op == "vjp":
        rng = np.random.default_rng(seed + 2)
        lx, ly = (torch.from_numpy(rng.standard_normal(n)).to(d) for _ in range(2))
        out = _direct_vjp(x, y, m, lx, ly, eps)
    else:
        idx = np.sort(np.random.default_rng(seed + 1).permutation(n)[:case["samples"]])
        out = _direct(x, y, m, eps, torch.from_numpy(idx).to(d))
    return [v.cpu() for v in out]
