"""The work that users of this framework have it do, as cases to be timed: one
pass each through the public entry points, over the range of sizes, geometries,
directions and precisions that programs use.

Families (the case's "kind"):

* ``neighbors``  a neighbour build of a moved or newly loaded particle set;
* ``update``     one operator update of a moving set, as a Lagrangian solver
                 does every step: Verlet list, re-assembly in the reference's
                 order, one application;
* ``assemble``   the fast assembly of batched FP32 (or FP64) weights over a list
                 that is there, as after small displacements;
* ``operator``   an operator applied in the reference's FP64 order (the default
                 of the operator objects);
* ``interp``     particle-to-particle interpolation between two sets;
* ``apply``      every output of a plan in one batched pass, per precision;
* ``autograd``   forward and backward with gradients of field and positions;
* ``gray_scott`` RK4 time steps from a captured graph and their adjoint.

Geometries: ``lattice`` (jittered, unit square or cube), ``periodic`` (the same
in a periodic box), ``graded`` (a 2D cloud whose density grows 4x along x, with
per-particle radii).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import operators as OPS
from openfpm_numerics_gb300.autograd import dcpse_apply
from openfpm_numerics_gb300.odeint import GrayScottRK4
from openfpm_numerics_gb300.plan import DcpsePlan

H_OVER_EPS = 0.9
# Gray-Scott parameters and the steps of one pass
DU, DV, FEED, KILL = 2e-5, 1e-5, 0.04, 0.06
GS_STEPS = 10


def listed():
    return [
        # a small 2D solver that moves its particles: latency of the whole update
        dict(name="update_2d_small", kind="update", geom="lattice", dim=2, side=64, ops="lap"),
        # the batched five operators of an uneven 2D cloud, updated each step
        dict(name="update_graded", kind="update", geom="graded", dim=2, side=447, ops="five"),
        # Gradient + Laplacian weights of a 3D set, FP32 for the batched applies
        dict(name="assemble_3d", kind="assemble", geom="lattice", dim=3, side=80, ops="grad_lap", precision="f32"),
        # the neighbour build of a production-size 3D set
        dict(name="neighbors_3d", kind="neighbors", geom="lattice", dim=3, side=128),
        # the default FP64 application of a Laplacian to a 3D field
        dict(name="operator_3d", kind="operator", geom="lattice", dim=3, side=96, ops="lap"),
        # remeshing: a field carried from moved particles to a regular set
        dict(name="interp_3d", kind="interp", geom="periodic", dim=3, side=64, precision="f64"),
        # the smallest apply: a call's latency
        dict(name="apply_2d_small", kind="apply", geom="lattice", dim=2, side=64, ops="lap", precision="f32"),
        # the benchmark's apply: four outputs on 2.1 million particles
        dict(name="apply_3d", kind="apply", geom="lattice", dim=3, side=128, ops="grad_lap", precision="f32"),
        # FP64-class results on the uneven cloud, particles in no spatial order
        dict(name="apply_graded_pair", kind="apply", geom="graded", dim=2, side=1000, ops="five",
             precision="f32-pair"),
        # gradients of a Laplacian loss with respect to field and positions, 2D
        dict(name="autograd_2d", kind="autograd", geom="lattice", dim=2, side=256, ops="lap"),
        # the same through Gradient + Laplacian in a periodic 3D box
        dict(name="autograd_3d", kind="autograd", geom="periodic", dim=3, side=40, ops="grad_lap"),
        # reaction-diffusion: ten steps forward and their checkpointed adjoint
        dict(name="gray_scott", kind="gray_scott", geom="periodic", dim=3, side=96),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["neighbors", "update", "assemble", "operator", "interp", "apply", "autograd", "gray_scott"])
    if kind == "gray_scott":
        return dict(kind=kind, geom="periodic", dim=3, side=_log_int(rng, 16, 96))
    geom = rng.choice(["lattice", "periodic"] if kind in ("interp", "autograd")
                      else ["lattice", "lattice", "periodic", "graded"])
    dim = 2 if geom == "graded" else rng.choice([2, 3])
    if kind == "autograd" and dim == 3:
        geom = "periodic"
    top = {"neighbors": (1000, 120), "update": (400, 40), "assemble": (500, 80), "operator": (1000, 96),
           "interp": (400, 64), "apply": (1000, 120), "autograd": (256, 40)}[kind][dim - 2]
    c = dict(kind=kind, geom=geom, dim=dim, side=_log_int(rng, 24 if dim == 2 else 10, top))
    if kind in ("update", "operator", "apply", "assemble", "autograd"):
        c["ops"] = rng.choice(["lap", "grad_lap", "five"] if dim == 2 else ["lap", "grad_lap"])
    if kind == "apply":
        c["precision"] = rng.choice(["f32", "f32-pair", "f64"])
    if kind == "assemble":
        c["precision"] = rng.choice(["f32", "f64"])
    if kind == "interp":
        c["precision"] = rng.choice(["f64", "f32"])
    return c


# ------------------------------------------------------------------ inputs --
def _signatures(dim, ops):
    """Outputs of a plan, each a list of the signatures summed into it."""
    e = lambda d, k: tuple(k if i == d else 0 for i in range(dim))  # noqa: E731
    grad, lap = [[e(d, 1)] for d in range(dim)], [[e(d, 2) for d in range(dim)]]
    if ops == "interp":
        return [[(0,) * dim]]
    if ops == "five":
        return [[(1, 0)], [(0, 1)], [(2, 0)], [(0, 2)], [(1, 1)]]
    return lap if ops == "lap" else grad + lap


def _lattice(side, dim, h, jitter, rng):
    """side^dim points, x fastest, every coordinate moved by U(-jitter h, jitter h)."""
    ax = np.arange(side, dtype=np.float64) * h
    grids = np.meshgrid(*([ax] * dim), indexing="ij")
    pos = np.stack([grids[dim - 1 - d].reshape(-1) for d in range(dim)], axis=1)
    if jitter:
        pos += rng.uniform(-jitter * h, jitter * h, size=pos.shape)
    return pos


def _inputs(case, seed):
    """Positions, spacing, cutoff(s), box and a smooth field, from the seed alone."""
    rng = np.random.default_rng([int(seed), 17])
    dim, side = case["dim"], case["side"]
    # where an output's length is the number of list entries, the set is one
    # cloud, mirrored and numbered by the seed: as many entries for every seed
    seeded, listing = rng, case["kind"] in ("neighbors", "assemble")
    if listing:
        rng = np.random.default_rng([side, dim, 17])
    box, rpp, mirror = None, None, range(dim)
    if case["geom"] == "graded":
        n = side * side
        x = (-1.0 + np.sqrt(1.0 + 15.0 * rng.random(n))) / 3.0
        pos = np.stack([x, rng.random(n)], axis=1)
        rpp = 3.1 / np.sqrt(n * (1.0 + 3.0 * x) / 2.5)
        h, rcut, mirror = 1.0 / side, 0.0, (1,)
    elif case["geom"] == "periodic":
        h = 1.0 / side
        pos = np.mod(_lattice(side, dim, h, 0.1, rng), 1.0)
        box = ((0.0,) * dim, (1.0,) * dim, (1,) * dim)
        rcut = (3.1 if dim == 2 else 2.8) * h
    else:
        h = 1.0 / (side - 1)
        pos = _lattice(side, dim, h, 0.1 if dim == 2 else 0.15, rng)
        rcut = (3.1 if dim == 2 else 2.8) * h
    if listing:
        rng = seeded
        for d in mirror:
            if rng.random() < 0.5:
                pos[:, d] = 1.0 - pos[:, d]
        first = int(rng.integers(pos.shape[0]))
        pos, rpp = np.roll(pos, first, 0), None if rpp is None else np.roll(rpp, first)
    if box is not None:
        pos[pos >= 1.0] = 0.0
    k = 2 * np.pi
    ph = rng.uniform(0, k, size=dim)
    f = np.ones(pos.shape[0])
    for d in range(dim):
        f *= np.sin(k * pos[:, d] + ph[d])
    f += 0.5 * np.cos(k * pos[:, 0] + ph[-1])
    dev = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    return dict(pos=dev(pos), h=h, rcut=rcut, rpp=dev(rpp), box=box, f=dev(f), rng=rng)


def _domain(case, seed, support):
    """The regular set that an interpolation writes to, inside the support set."""
    side, dim, h = case["side"], case["dim"], support["h"]
    rng = np.random.default_rng([int(seed), 23])
    if case["geom"] == "periodic":
        return torch.from_numpy(np.mod(_lattice(side, dim, h, 0.0, rng) + 0.3 * h, 1.0)).cuda()
    return torch.from_numpy(_lattice(side - 2, dim, h, 0.0, rng) + 0.7 * h).cuda()


def _gs_initial(pos, rng):
    """u = 1, v = 0 but for 20 random spheres of radius 0.05 (periodic)."""
    u, v = torch.ones(pos.shape[0], device="cuda"), torch.zeros(pos.shape[0], device="cuda")
    for c in rng.random((20, 3)):
        d = pos - torch.from_numpy(c).cuda()
        inside = ((d - d.round()) ** 2).sum(1) < 0.05 ** 2
        u[inside], v[inside] = 0.5, 0.25
    return u, v


_PREC = {"f32": C.F32, "f32-pair": C.F32_PAIR, "f64": C.F64}
_STORE = {"f32": C.ASSEMBLE_FAST | C.STORE_OUT_F32,
          "f32-pair": C.ASSEMBLE_FAST | C.STORE_OUT_F32 | C.STORE_OUT_F32_CORR,
          "f64": C.ASSEMBLE_FAST | C.STORE_OUT_F64}


def _plan(case, x, outputs, stream=None):
    plan = DcpsePlan(case["dim"], outputs, order=2, box=x["box"], stream=stream)
    plan.build_neighbors(x["pos"], x["rcut"], x["rpp"])
    return plan


def _parts(x):
    b = x["box"]
    return OPS.ParticleSet(x["pos"], box=b and b[:2], periodic=b and b[2])


def _verlet(parts, x):
    return OPS.VerletList(parts, x["rcut"], rcut_pp=x["rpp"])


def _operator(case, parts, vl, x):
    args = (parts, vl, 2, x["rcut"])
    # boundary particles of a random cloud may have too few neighbours
    kw = dict(allow_failed_particles=True)
    if case["ops"] == "lap":
        return OPS.Laplacian(*args, **kw)
    return OPS.OperatorSet(*args, ["x", "y", "xx", "yy", "xy"] if case["ops"] == "five" else ["gradient", "laplacian"],
                           **kw)


def prepare(case, seed):
    x = _inputs(case, seed)
    s = {"case": case, "x": x, "kind": case["kind"]}
    kind = case["kind"]
    if kind == "neighbors":
        s["plan"] = DcpsePlan(case["dim"], _signatures(case["dim"], "lap"), order=2, box=x["box"])
    elif kind in ("update", "operator"):
        s["parts"] = _parts(x)
        s["op"] = _operator(case, s["parts"], _verlet(s["parts"], x), x)
    elif kind == "interp":
        sup, dom = _parts(x), _parts(dict(x, pos=_domain(case, seed, x)))
        s["op"] = OPS.PPInterpolation(sup, dom, OPS.createVerletTwoPhase(dom, sup, x["rcut"]), 2, x["rcut"],
                                      allow_failed_particles=True)
        s["hold"] = (sup, dom)
    elif kind in ("assemble", "apply"):
        s["plan"] = _plan(case, x, _signatures(case["dim"], case["ops"]))
        if kind == "apply":
            s["plan"].assemble(x["pos"], _STORE[case["precision"]])
    elif kind == "autograd":
        outs = _signatures(case["dim"], case["ops"])
        s["plan"] = _plan(case, x, outs)
        s["f"] = x["f"].clone().requires_grad_()
        s["pos"] = x["pos"].clone().requires_grad_()
        s["g"] = torch.from_numpy(x["rng"].standard_normal((len(outs), x["pos"].shape[0]))).cuda()
    else:
        stream = torch.cuda.Stream()
        s["stream"] = stream
        u, v = _gs_initial(x["pos"], x["rng"])
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            s["plan"] = _plan(case, x, _signatures(3, "lap"), stream)
            s["plan"].assemble(x["pos"], C.ASSEMBLE_FAST | C.STORE_OUT_F32)
        gs = GrayScottRK4(s["plan"], u, v, DU, DV, FEED, KILL, 0.2 * x["h"] ** 2 / DU)
        gs.capture(GS_STEPS, stream)
        s.update(gs=gs, start=(u, v), ybar=(torch.zeros_like(u), torch.ones_like(v)))
    return s


def run(s):
    kind, x = s["kind"], s["x"]
    if kind == "neighbors":
        s["plan"].build_neighbors(x["pos"], x["rcut"], x["rpp"])
        return s["plan"].neighbors()
    if kind == "update":
        s["parts"].setPos(x["pos"])
        s["op"].update(s["parts"], _verlet(s["parts"], x))
        return s["op"](x["f"])
    if kind == "assemble":
        plan, p64 = s["plan"], s["case"]["precision"] == "f64"
        plan.assemble(x["pos"], _STORE[s["case"]["precision"]])
        return [plan.output_weights(o)[0 if p64 else 1] for o in range(plan.n_outputs)]
    if kind == "operator":
        return s["op"](x["f"])
    if kind == "interp":
        return s["op"](x["f"], s["case"]["precision"])
    if kind == "apply":
        return s["plan"].apply(x["f"], _PREC[s["case"]["precision"]])
    if kind == "autograd":
        y = dcpse_apply(s["f"], s["pos"], s["plan"])
        return (y.detach(),) + torch.autograd.grad(y, (s["f"], s["pos"]), s["g"])
    gs = s["gs"]
    with torch.cuda.stream(s["stream"]):
        gs.u.copy_(s["start"][0])
        gs.v.copy_(s["start"][1])
        gs.run(GS_STEPS)
        ub, vb = gs.backward([s["start"]], GS_STEPS, s["ybar"], stream=s["stream"])
        return gs.u, gs.v, ub, vb


# -------------------------------------------------------------------- work --
# mean neighbours of an interior particle
def _sizes(case):
    dim, side = case["dim"], case["side"]
    n = side ** dim
    if case["kind"] == "interp" and case["geom"] == "lattice":
        n = (side - 2) ** dim
    k = 30.2 if dim == 2 else 91.9
    if case["geom"] == "lattice":
        k *= (1.0 - (0.85 if dim == 2 else 0.7) * (3.1 if dim == 2 else 2.8) / side) ** dim
    return n, n * k


def _basis(dim, m, order=2):
    """Exponents of the DC-PSE basis of a signature of order m."""
    lim, lo = m + order, 1 if m and m % 2 == 0 else 0
    g = [t[::-1] for t in np.ndindex(*([lim] * dim))]
    return [t for t in g if lo <= sum(t) < lim]


def _assembly_flops(case, outs, n, nnz):
    """Moment matrices, solves and weights of every distinct basis, and the
    powers and exponentials of every entry."""
    f = nnz * 60.0
    for m in sorted({sum(s) for o in outs for s in o}):
        b = len(_basis(case["dim"], m))
        r = sum(any(sum(s) == m for s in o) for o in outs)
        f += nnz * b * (b + 1) + n * ((2 / 3) * b ** 3 + 2 * b * b * r) + 2 * nnz * b * r
    return f


def work(case):
    n, nnz = _sizes(case)
    dim, kind = case["dim"], case["kind"]
    outs = _signatures(dim, "interp" if kind == "interp" else case.get("ops", "lap"))
    no, nt = len(outs), sum(len(o) for o in outs)
    pos, lst = 8.0 * dim * n, 8.0 * n + 4.0 * nnz
    if kind == "neighbors":
        return {"bytes": pos + lst, "flops": 3.0 * dim * nnz}
    if kind == "assemble":
        return {"bytes": pos + lst + no * nnz * (8 if case["precision"] == "f64" else 4),
                "flops": _assembly_flops(case, outs, n, nnz)}
    if kind == "update":  # list, per-term kernels, the FP64 and FP32 sums, the application
        return {"bytes": pos + lst + nnz * (8.0 * nt + 16.0 * no) + 8.0 * n * (1 + no),
                "flops": _assembly_flops(case, outs, n, nnz) + 3.0 * nnz * nt}
    if kind == "operator":
        return {"bytes": lst + 8.0 * nnz * nt + 8.0 * n * (1 + no), "flops": 3.0 * nnz * nt}
    if kind == "interp":
        return {"bytes": lst + (8.0 if case["precision"] == "f64" else 4.0) * nnz + 16.0 * n, "flops": 2.0 * nnz}
    if kind == "apply":
        w = {"f32": 4.0, "f32-pair": 8.0, "f64": 8.0}[case["precision"]]
        return {"bytes": lst + w * nnz * no + 8.0 * n * (1 + no), "flops": (1.0 + 2.0 * no) * nnz}
    if kind == "autograd":
        # the assembly, the apply, its transpose, and the assembly's adjoint
        a = _assembly_flops(case, outs, n, nnz)
        return {"bytes": 2 * (pos + lst) + 8.0 * nnz * no + 16.0 * n * no + pos, "flops": 3 * a + 4.0 * nnz * no}
    # four stages forward, four again for the record, four adjoint: the weights once each
    return {"bytes": GS_STEPS * 12 * (8.0 * nnz + 48.0 * n), "flops": GS_STEPS * 12 * (6.0 * nnz + 30.0 * n)}


# ------------------------------------------------------------------- exact --
def _offsets(a, b, box):
    o = a - b
    if box is not None:
        o = o - torch.round(o)  # unit box
    return o


def _neighbors(x, dom=None):
    """Padded lists [n, K] (column, mask), ascending, by a cell search."""
    pos, box = x["pos"], x["box"]
    two = dom is not None
    dom = pos if dom is None else dom
    n, dim = dom.shape
    rc = x["rpp"] if x["rpp"] is not None else torch.full((n,), x["rcut"], dtype=torch.float64, device="cuda")
    rmax = float(rc.max())
    if box is not None:
        lo, nc = torch.zeros(dim, device="cuda", dtype=torch.float64), [max(int(1.0 / rmax), 1)] * dim
        side = 1.0 / nc[0]
    else:
        lo, side = torch.minimum(pos.min(0).values, dom.min(0).values), rmax
        nc = ((torch.maximum(pos.max(0).values, dom.max(0).values) - lo) / side).floor().to(torch.int64).add(1).tolist()
    cell = lambda p: torch.stack([((p[:, d] - lo[d]) / side).floor().to(torch.int64).clamp(0, nc[d] - 1)  # noqa: E731
                                  for d in range(dim)], 1)
    mul = [1]
    for d in range(dim - 1):
        mul.append(mul[-1] * nc[d])
    lin = sum(cell(pos)[:, d] * mul[d] for d in range(dim))
    order = torch.argsort(lin, stable=True)
    start = torch.searchsorted(lin[order], torch.arange(mul[-1] * nc[-1] + 1, device="cuda"))
    maxc = int((start[1:] - start[:-1]).max())
    cdom, cols = cell(dom), []
    lane = torch.arange(maxc, device="cuda")
    step = max(1, int(4e8 / (8 * 3 ** dim * maxc * 4)))
    for b in range(0, n, step):
        p = torch.arange(b, min(n, b + step), device="cuda")
        cand = []
        seen = []
        for off in np.ndindex(*([3] * dim)):
            c = [cdom[p, d] + (off[d] - 1) for d in range(dim)]
            ok = torch.ones_like(p, dtype=torch.bool)
            for d in range(dim):
                if box is not None:
                    c[d] = c[d] % nc[d]
                else:
                    ok &= (c[d] >= 0) & (c[d] < nc[d])
            l = sum(torch.where(ok, c[d], 0) * mul[d] for d in range(dim))
            for s in seen if box is not None and nc[0] < 3 else []:
                ok &= s != l
            seen.append(torch.where(ok, l, -1))
            i = start[l][:, None] + lane
            q = torch.where(ok[:, None] & (i < start[l + 1][:, None]), order[i.clamp(max=order.numel() - 1)], -1)
            cand.append(q)
        q = torch.cat(cand, 1)
        o = _offsets(dom[p][:, None, :], pos[q.clamp(min=0)], box)
        d2 = o[..., 0] * o[..., 0]
        for d in range(1, dim):
            d2 = d2 + o[..., d] * o[..., d]
        keep = (q >= 0) & (d2 < (rc[p] * rc[p])[:, None])
        if not two:
            keep &= q != p[:, None]
        q = torch.where(keep, q, pos.shape[0]).sort(1).values
        cols.append(q[:, : max(int(keep.sum(1).max()), 1)])
    K = max(c.shape[1] for c in cols)
    q = torch.cat([torch.nn.functional.pad(c, (0, K - c.shape[1]), value=pos.shape[0]) for c in cols])
    return q, q < pos.shape[0]


def _weights(x_dom, x_sup, q, m, outs, box):
    """Summed weights of every output, [n, no, K], of rows whose neighbours are
    q (masked by m): K_q = exp(-|u|^2) a.v(u), A a = b, times eps^-|alpha|."""
    dim, k = x_dom.shape[1], m.sum(1)
    off = _offsets(x_dom[:, None, :], x_sup[torch.where(m, q, 0)], box)
    off = torch.where(m[..., None], off, torch.ones_like(off))
    eps = (off.abs().sum(2) * m).sum(1) / k.clamp(min=1) / H_OVER_EPS
    u = off / torch.where(k > 0, eps, torch.ones_like(eps))[:, None, None]
    om = torch.exp(-(u * u).sum(2)) * m
    W = [torch.zeros_like(om) for _ in outs]
    for order in sorted({sum(s) for o in outs for s in o}):
        B = _basis(dim, order)
        pw = [[torch.ones_like(om)] for _ in range(dim)]
        for d in range(dim):
            for _ in range(order + 1):
                pw[d].append(pw[d][-1] * u[..., d])
        V = torch.stack([math.prod((pw[d][e[d]] for d in range(1, dim)), start=pw[0][e[0]]) for e in B], 2)
        A = torch.einsum("nk,nki,nkj->nij", om, V, V) if V.shape[1] < 2 else (V * om[..., None]).transpose(1, 2) @ V
        use = [[s for s in o if sum(s) == order] for o in outs]
        rhs = torch.zeros(len(B), len(outs), dtype=torch.float64, device="cuda")
        for j, sigs in enumerate(use):
            for s in sigs:
                rhs[B.index(s), j] += (-1.0) ** order * math.prod(math.factorial(t) for t in s)
        ok = k >= len(B)
        A = torch.where(ok[:, None, None], A, torch.eye(len(B), dtype=torch.float64, device="cuda"))
        a = torch.linalg.solve(A, rhs.expand(A.shape[0], -1, -1))
        w = (V @ a) * (om * ok[:, None] * eps[:, None] ** -order)[..., None]
        for j, sigs in enumerate(use):
            if sigs:
                W[j] = W[j] + w[..., j]
    return torch.stack(W, 1)


def _chunks(n, K, nb):
    step = max(1, int(1.5e9 / (8 * K * nb)))
    return [slice(b, min(n, b + step)) for b in range(0, n, step)]


def exact(case, seed):
    kind, dim = case["kind"], case["dim"]
    x = _inputs(case, seed)
    n = x["pos"].shape[0]
    if n > 2_200_000:
        return None
    dom = _domain(case, seed, x) if kind == "interp" else None
    q, m = _neighbors(x, dom)
    if kind == "neighbors":
        rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        rp[1:] = m.sum(1).cumsum(0)
        return rp, q[m].to(torch.int32)
    outs = _signatures(dim, "interp" if kind == "interp" else case.get("ops", "lap"))
    dom = x["pos"] if dom is None else dom
    ch = _chunks(dom.shape[0], q.shape[1], 20 if dim == 3 else 10)
    if kind == "autograd":
        f, pos = x["f"].requires_grad_(), x["pos"].requires_grad_()
        g = torch.from_numpy(x["rng"].standard_normal((len(outs), n))).cuda()
        ys, gf, gp = [], torch.zeros_like(f), torch.zeros_like(pos)
        for c in [slice(b, min(n, b + 8000)) for b in range(0, n, 8000)]:
            W = _weights(pos[c], pos, q[c], m[c], outs, x["box"])
            y = (W * (f[torch.where(m[c], q[c], 0)] - f[c][:, None])[:, None, :]).sum(2).T
            a, b = torch.autograd.grad(y, (f, pos), g[:, c])
            gf, gp = gf + a, gp + b
            ys.append(y.detach())
        return torch.cat(ys, 1), gf, gp
    W = [_weights(dom[c], x["pos"], q[c], m[c], outs, x["box"]) for c in ch]
    if kind == "assemble":
        return [torch.cat([w[:, o][m[c]] for w, c in zip(W, ch)]) for o in range(len(outs))]
    fq = lambda c, f: f[torch.where(m[c], q[c], 0)]  # noqa: E731
    if kind == "interp":
        return torch.cat([(w[:, 0] * fq(c, x["f"])).sum(1) for w, c in zip(W, ch)])
    if kind == "gray_scott":
        L = torch.cat([w[:, 0] for w in W])
        qq = torch.where(m, q, 0)
        lap = lambda y: (L * (y[qq] - y[:, None])).sum(1)  # noqa: E731
        dt = 0.2 * x["h"] ** 2 / DU

        def rhs(u, v):
            r = u * v * v
            return DU * lap(u) - r + FEED * (1 - u), DV * lap(v) + r - (FEED + KILL) * v

        def step(u, v):
            k1 = rhs(u, v)
            k2 = rhs(u + dt / 2 * k1[0], v + dt / 2 * k1[1])
            k3 = rhs(u + dt / 2 * k2[0], v + dt / 2 * k2[1])
            k4 = rhs(u + dt * k3[0], v + dt * k3[1])
            return tuple(y + dt / 6 * (a + 2 * b + 2 * c + d) for y, a, b, c, d in zip((u, v), k1, k2, k3, k4))

        states = [tuple(y.double() for y in _gs_initial(x["pos"], x["rng"]))]
        for _ in range(GS_STEPS):
            states.append(step(*states[-1]))
        bar = (torch.zeros(n, dtype=torch.float64, device="cuda"), torch.ones(n, dtype=torch.float64, device="cuda"))
        for y in states[-2::-1]:
            y = tuple(t.clone().requires_grad_() for t in y)
            bar = torch.autograd.grad(step(*y), y, bar)
        return tuple(states[-1]) + tuple(bar)
    y = torch.cat([(w * (fq(c, x["f"]) - x["f"][c][:, None])[:, None, :]).sum(2) for w, c in zip(W, ch)]).T
    if kind in ("update", "operator") and case["ops"] == "lap":
        return y[0]
    return y
