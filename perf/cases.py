"""Performance cases: the work a user of this engine has it do, through its
public entry points, from the smallest call to the largest.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what a program has in hand before the call (inputs, and the
tree or solver it keeps), ``run`` is one pass, ``work`` the bytes and
operations the pass cannot do without and ``exact`` the same outputs from
plain torch in 64 bits.

Kinds of case:

* ``oneshot``   ``accelerations(positions, masses)``: tree build and solve in
  one call, nothing kept between calls.
* ``step``      a simulation step: ``Tree.rebuild`` or ``Tree.refit`` with new
  positions, then the self accelerations.
* ``targets``   accelerations of a built ``Tree`` at external points.
* ``probes``    ``Tree.rebuild`` with new positions, then a few external
  points (massless tracers in a live potential): the build dominates.
* ``batch``     ``BatchedSolver``: new positions of many independent systems
  loaded and solved in one pass.
* ``direct``    ``direct_accelerations``, the FP64 direct sum.
"""
import math

import numpy as np
import torch

import bhut_gb300 as bh
from bhut_gb300.api import direct_accelerations
from bhut_gb300.batch import BatchedSolver

G = 1.0
MORTON_CELLS = 2.0 ** 21      # per axis
_FIELDS = dict(kind="oneshot", dist="plummer", masses="equal", dim=3, host=False, form="fast",
               criterion="bh", multipole="mono", theta=0.5, eps=0.01, leaf=32, update="rebuild",
               targets=0, nsys=1, nmin=0)


def _case(**kw):
    return {**_FIELDS, **kw}


def listed():
    return [
        # a script that solves one small system held in NumPy arrays: latency
        _case(name="oneshot_numpy_1k", n=1_000, dist="gaussian", host=True),
        # the reference's CPU-runnable workload, device-resident
        _case(name="oneshot_10k", n=10_000, dist="gaussian"),
        # every option at the reference's defaults (no softening), uneven
        # masses, a size that fills no tile
        _case(name="oneshot_unsoftened_100k", n=100_003, dist="cube", masses="uneven", eps=0.0),
        # the headline workload: rebuild and solve of a 1M Plummer sphere
        _case(name="step_rebuild_1m", kind="step", n=1_000_000),
        # a planar system stepped with refits, small leaves, uneven masses
        _case(name="step_refit_2d_60k", kind="step", n=60_001, dist="gaussian", dim=2,
              masses="uneven", leaf=16, update="refit"),
        # field evaluation of the 1M system at 250k points
        _case(name="targets_250k", kind="targets", n=1_000_000, targets=250_000),
        # tracers in a live 1M galaxy: build-bound
        _case(name="probes_rebuild_1m", kind="probes", n=1_000_000, dist="galaxy", targets=2_000,
              eps=0.005),
        # bit-compatible FP64 arithmetic
        _case(name="step_exact_100k", kind="step", n=100_000, form="exact"),
        # the precision form on the galaxy model
        _case(name="step_fp32_galaxy_2m", kind="step", n=2_000_000, dist="galaxy", form="fp32",
              theta=0.7, eps=0.005, leaf=16),
        # many uneven systems in one solve
        _case(name="batch_256", kind="batch", n=65_536, nmin=256, nsys=256, form="fp32", leaf=16),
        # a server tick: offset criterion and quadrupoles
        _case(name="batch_quad_24", kind="batch", n=100_000, nmin=1_000, nsys=24, form="fp32",
              criterion="bh_offset", multipole="quad", theta=0.7, leaf=16),
        # the accuracy check that users run on a sample of their system
        _case(name="direct_20k", kind="direct", n=20_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One case of the listed ranges."""
    kind = rng.choice(["oneshot", "oneshot", "step", "step", "targets", "probes", "batch", "direct"])
    c = dict(kind=kind, dist=rng.choice(["gaussian", "plummer", "cube", "galaxy"]),
             masses=rng.choice(["equal", "uneven"]), theta=rng.choice([0.4, 0.5, 0.7]),
             leaf=rng.choice([16, 32, 32]), eps=rng.choice([0.005, 0.01, 0.02]))
    if kind == "oneshot":
        c.update(n=_log_int(rng, 1_000, 200_000), host=rng.random() < 0.4,
                 form=rng.choice(["fast", "fast", "fp32"]))
        if rng.random() < 0.3:
            c.update(eps=0.0, form="fast")
    elif kind == "step":
        form = rng.choice(["fast", "fast", "fp32", "exact"])
        c.update(form=form, update=rng.choice(["rebuild", "refit"]),
                 n=_log_int(rng, 2_000, {"fast": 500_000, "fp32": 2_000_000, "exact": 60_000}[form]))
    elif kind in ("targets", "probes"):
        c.update(n=_log_int(rng, 50_000, 1_000_000),
                 targets=_log_int(rng, 500, 4_000 if kind == "probes" else 150_000))
    elif kind == "batch":
        c.update(nsys=rng.randrange(8, 200), nmin=256, n=_log_int(rng, 2_000, 40_000), leaf=16,
                 dist=rng.choice(["plummer", "cube"]), form=rng.choice(["fp32", "fp32", "fast"]))
        if c["form"] == "fp32" and rng.random() < 0.4:
            c.update(criterion="bh_offset", multipole="quad", theta=0.7)
    else:
        c.update(n=_log_int(rng, 2_000, 20_000))
    if kind in ("oneshot", "step") and c["dist"] in ("gaussian", "cube") and rng.random() < 0.25:
        c["dim"] = 2
    return _case(**c)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _directions(n, g):
    v = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True)


def _uniform(n, g):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _positions(dist, n, dim, g):
    if dist == "gaussian":
        return torch.randn((n, dim), generator=g, device="cuda", dtype=torch.float64)
    if dist == "cube":
        return 10.0 * torch.rand((n, dim), generator=g, device="cuda", dtype=torch.float64) - 5.0
    if dist == "plummer":       # a = 1, radii truncated at 20
        v = (_uniform(n, g) * (400.0 / 401.0) ** 1.5) ** (1.0 / 3.0)
        return _directions(n, g) * (v / (1.0 - v * v).sqrt())[:, None]
    # galaxy: 70 % exponential disc (rd 3, z0 0.3), 30 % Hernquist bulge (a 0.5, r <= 20 a)
    nd = round(0.7 * n)
    R = -3.0 * torch.log((1.0 - _uniform(nd, g)) * (1.0 - _uniform(nd, g)))
    phi = 2.0 * math.pi * _uniform(nd, g)
    z = 0.3 * torch.atanh((2.0 * _uniform(nd, g) - 1.0).clamp(-1.0 + 1e-15, 1.0 - 1e-15))
    s = _uniform(n - nd, g).sqrt() * (20.0 / 21.0)
    bulge = _directions(n - nd, g) * (0.5 * s / (1.0 - s))[:, None]
    return torch.cat([torch.stack([R * phi.cos(), R * phi.sin(), z], dim=1), bulge])


def _inputs(case, seed):
    """(initial positions, new positions, masses, targets, offsets)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    offsets = np.zeros(case["nsys"] + 1, dtype=np.int64)
    if case["kind"] == "batch":     # sizes evenly spread over the logarithm of the range
        sizes = np.geomspace(case["nmin"], case["n"], case["nsys"]).astype(np.int64)
        offsets[1:] = np.cumsum(np.random.RandomState(case["nsys"]).permutation(sizes))
        scale = 0.5 + 1.5 * _uniform(case["nsys"], g)
        x = torch.cat([_positions(case["dist"], int(k), 3, g) * a
                       for k, a in zip(np.diff(offsets), scale)])
        m = torch.cat([torch.full((int(k),), 1.0 / int(k), device="cuda", dtype=torch.float64)
                       for k in np.diff(offsets)])
    else:
        n = offsets[1] = case["n"]
        x = _positions(case["dist"], int(n), case["dim"], g)
        m = torch.full((int(n),), 1.0 / int(n), device="cuda", dtype=torch.float64)
    if case["masses"] == "uneven":
        m = m * (0.5 + _uniform(len(m), g))
    x1 = x + 0.002 * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)
    t = 10.0 * torch.rand((case["targets"], case["dim"]), generator=g, device="cuda",
                          dtype=torch.float64) - 5.0
    return x, x1, m, t, offsets


def prepare(case, seed):
    x, x1, m, t, offsets = _inputs(case, seed)
    s = dict(case=case, x=x1, m=m, t=t, offsets=offsets)
    if case["kind"] in ("oneshot", "direct"):
        if case["host"]:
            s.update(x=x1.cpu().numpy(), m=m.cpu().numpy())
    elif case["kind"] == "batch":
        s["solver"] = BatchedSolver(dim=3, leaf_size=case["leaf"], form=case["form"],
                                    criterion=case["criterion"], multipole=case["multipole"])
        s["solver"].load(x, m, offsets)
        s["out"] = torch.empty_like(x1)
    else:
        s["tree"] = bh.Tree(x1 if case["kind"] == "targets" else x, m, leaf_size=case["leaf"],
                            dim=case["dim"], form=case["form"]).build()
    return s


def run(s):
    c = s["case"]
    kw = dict(theta=c["theta"], softening=c["eps"], G=G)
    if c["kind"] == "oneshot":
        return bh.accelerations(s["x"], s["m"], dim=c["dim"], leaf_size=c["leaf"], form=c["form"],
                                **kw)
    if c["kind"] == "direct":
        return direct_accelerations(s["x"], s["m"], softening=c["eps"], G=G)
    if c["kind"] == "batch":
        s["solver"].load(s["x"], s["m"], s["offsets"])
        return s["solver"].solve(out=s["out"], **kw)
    tree = s["tree"]
    if c["kind"] == "targets":
        return tree.accelerations(s["t"], **kw)
    if c["kind"] == "probes":
        return tree.rebuild(s["x"]).accelerations(s["t"], **kw)
    return getattr(tree, c["update"])(s["x"]).accelerations(**kw)


def work(case):
    """Bytes: each position, mass and target read once, each acceleration
    written once.  Operations: 20 per interaction; a target of a
    Barnes-Hut solve meets about (4 pi / 3) (2 / theta)^3 cells' worth of
    neighbours per halving of the particle count beyond that, each pair of a
    direct sum once."""
    c = case
    if c["kind"] == "batch":
        sizes = np.geomspace(c["nmin"], c["n"], c["nsys"]).astype(np.int64)
    else:
        sizes = np.array([c["n"]])
    n = int(sizes.sum())
    nt = c["targets"] if c["kind"] in ("targets", "probes") else n
    d = c["dim"]
    sources = 0 if c["kind"] == "targets" else 8 * (d + 1) * n
    given = 8 * d * nt if c["kind"] in ("targets", "probes") else 0
    inter = 0.0
    for k in sizes.tolist():
        full = min(1.0, nt / n) * k * k
        if c["kind"] == "direct":
            inter += full
        else:
            near = math.pi * (2 if d == 2 else 4 / 3) * (2.0 / c["theta"]) ** d
            levels = max(0.0, math.log2(k / (near * c["leaf"]))) if k > near * c["leaf"] else 0.0
            inter += min(full, nt * k / n * near * c["leaf"] * (0.5 + 0.5 * levels))
    return {"bytes": sources + given + 8 * d * nt, "flops": 20.0 * inter}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _spread(q, dim):
    """Morton bit spreading of 21-bit integers, bit by bit."""
    out = torch.zeros_like(q)
    for b in range(21):
        out |= ((q >> b) & 1) << (dim * b)
    return out


def _morton_order(x):
    lo, hi = x.min(0).values, x.max(0).values
    ext = hi - lo
    flat = ext <= 0
    p = (x - lo) / torch.where(flat, torch.ones_like(ext), ext) + 0.5 * flat.to(x.dtype)
    q = (p.clamp(max=1.0 - 1e-12) * MORTON_CELLS).to(torch.int64).clamp(max=int(MORTON_CELLS) - 1)
    key = sum(_spread(q[:, d], x.shape[1]) << d for d in range(x.shape[1]))
    return torch.sort(key, stable=True).indices


class _Levels:
    """The count-split tree of Morton-ordered particles, level by level."""

    def __init__(self, xs, ms, leaf, geometry, quad):
        dev, dim = xs.device, xs.shape[1]
        self.levels = []
        start = torch.zeros(1, dtype=torch.int64, device=dev)
        count = torch.full((1,), len(xs), dtype=torch.int64, device=dev)
        while len(start):
            k = len(start)
            seg = torch.repeat_interleave(torch.arange(k, device=dev), count)
            at = torch.arange(len(seg), device=dev) - torch.repeat_interleave(
                torch.cumsum(count, 0) - count, count) + torch.repeat_interleave(start, count)
            x, m = xs[at], ms[at]
            M = torch.zeros(k, dtype=x.dtype, device=dev).index_add_(0, seg, m)
            com = torch.zeros((k, dim), dtype=x.dtype, device=dev).index_add_(0, seg, m[:, None] * x)
            com /= M[:, None]
            xo = (geometry if geometry is not None else xs)[at]
            seg2 = seg[:, None].expand(-1, dim)
            lo = torch.full((k, dim), math.inf, dtype=x.dtype, device=dev).scatter_reduce(
                0, seg2, xo, "amin")
            hi = torch.full((k, dim), -math.inf, dtype=x.dtype, device=dev).scatter_reduce(
                0, seg2, xo, "amax")
            Q = None
            if quad:
                d = x - com[seg]
                q = m[:, None, None] * (3.0 * d[:, :, None] * d[:, None, :]
                                        - (d * d).sum(1)[:, None, None]
                                        * torch.eye(dim, dtype=x.dtype, device=dev))
                Q = torch.zeros((k, dim, dim), dtype=x.dtype, device=dev).index_add_(0, seg, q)
            inner = count > leaf
            self.levels.append(dict(start=start, count=count, M=M, com=com, Q=Q, inner=inner,
                                    size=(hi - lo).max(1).values,
                                    off=(com - 0.5 * (lo + hi)).norm(dim=1),
                                    child=2 * (torch.cumsum(inner.to(torch.int64), 0) - 1)))
            s, c = start[inner], count[inner]
            half = c // 2
            start = torch.stack([s, s + half], 1).reshape(-1)
            count = torch.stack([half, c - half], 1).reshape(-1)


def _tree_forces(x, m, targets, c, geometry=None, rows=1 << 20):
    """Barnes-Hut accelerations of `targets`; `geometry`: the positions that
    fixed the order and the boxes (a refit keeps them)."""
    perm = _morton_order(x if geometry is None else geometry)
    xs, ms, leaf, eps2 = x[perm], m[perm], c["leaf"], c["eps"] ** 2
    lv = _Levels(xs, ms, leaf, None if geometry is None else geometry[perm],
                 c["multipole"] == "quad").levels
    out = torch.empty_like(targets)
    lane = torch.arange(leaf, device=x.device)
    block = max(256, int(4e8 / 4_000 / max(1, len(lv))))
    tperm = _morton_order(targets) if len(targets) > 1 else torch.zeros(1, dtype=torch.int64,
                                                                        device=x.device)
    for b in range(0, len(targets), block):
        ti = tperm[b:b + block]
        xt = targets[ti]
        acc = torch.zeros_like(xt)
        t = torch.arange(len(xt), device=x.device)
        node = torch.zeros_like(t)
        for L in lv:
            inner = L["inner"][node]
            lt, ln = t[~inner], node[~inner]
            for r in range(0, len(lt), rows):       # leaves: every particle
                a, k = lt[r:r + rows], ln[r:r + rows]
                at = L["start"][k][:, None] + lane
                live = lane < L["count"][k][:, None]
                at = at.clamp(max=len(xs) - 1)
                d = [xs[:, j][at] - xt[a, j][:, None] for j in range(x.shape[1])]
                r2 = eps2 + sum(v * v for v in d)
                w = torch.where(live & (r2 > 0), ms[at] / (r2 * r2.sqrt()), 0.0)
                acc.index_add_(0, a, torch.stack([(w * v).sum(1) for v in d], 1))
            t, node = t[inner], node[inner]
            if not len(t):
                break
            d = L["com"][node] - xt[t]
            d2 = (d * d).sum(1)
            dist = d2.sqrt()
            if c["criterion"] == "bh_offset":
                dist = dist - L["off"][node]
            op = (L["size"][node] >= c["theta"] * dist) | (d2 == 0)
            d, d2, k, a = d[~op], d2[~op] + eps2, node[~op], t[~op]
            f = L["M"][k][:, None] * d / (d2 * d2.sqrt())[:, None]
            if L["Q"] is not None:
                qd = torch.einsum("kij,kj->ki", L["Q"][k], d)
                f += (-qd + 2.5 * ((qd * d).sum(1) / d2)[:, None] * d) / (d2 ** 2.5)[:, None]
            acc.index_add_(0, a, f)
            t = t[op].repeat_interleave(2)
            node = L["child"][node[op]].repeat_interleave(2)
            node[1::2] += 1
        out[ti] = acc * G
    return out


def exact(case, seed):
    c = case
    x, x1, m, t, offsets = _inputs(c, seed)
    if c["kind"] == "direct":
        out = torch.empty_like(x1)
        for b in range(0, len(x1), 1024):
            d = x1[None, :, :] - x1[b:b + 1024, None, :]
            r2 = (d * d).sum(2) + c["eps"] ** 2
            w = torch.where(r2 > 0, m[None, :] / (r2 * r2.sqrt()), 0.0)
            out[b:b + 1024] = G * (w[:, :, None] * d).sum(1)
        return out
    if c["kind"] in ("targets", "probes"):
        return _tree_forces(x1, m, t, c)
    if c["kind"] == "batch":
        return torch.cat([_tree_forces(x1[i:j], m[i:j], x1[i:j], c)
                          for i, j in zip(offsets[:-1].tolist(), offsets[1:].tolist())])
    geometry = x if c["kind"] == "step" and c["update"] == "refit" else None
    out = _tree_forces(x1, m, x1, c, geometry)
    return out.cpu().numpy() if c["host"] else out
