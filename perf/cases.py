"""Timed workloads of the FMM evaluate path, each through the package's public entry points.

A case names a call ("call"), a kernel, a precision, an order p, a leaf size ncrit, a point set and its
size(s):

  evaluate       new charges into a kept tree, then one evaluate; CUDA tensors in and out
  evaluate_host  the same with numpy arrays on both sides, as a caller of the pybind11 module has them
  adjoint        a differentiable evaluate on a kept tree and its backward pass (dL/dq and dL/dx)
  moved          new positions: tree, lists and schedules are built for them, then one evaluate; the Fmm
                 object (its operators) is kept from step to step
  batch          many independent systems in one captured graph
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "exafmm-t_b200"))

import exafmm.helmholtz as helmholtz  # noqa: E402
import exafmm.laplace as laplace  # noqa: E402
import exafmm.modified_helmholtz as yukawa  # noqa: E402
from exafmm.autograd import fmm_apply  # noqa: E402
from exafmm.batch import BatchedFmm, plummer  # noqa: E402

_MODULES = {"laplace": laplace, "modified_helmholtz": yukawa, "helmholtz": helmholtz}


def _case(name, call, kernel, precision, p, ncrit, points, n, ntrg=0, wavek=0.0, depth=-1):
    """ntrg 0: sources and targets coincide; depth -1: adaptive tree."""
    return {"name": name, "call": call, "kernel": kernel, "precision": precision, "p": p, "ncrit": ncrit,
            "points": points, "n": n, "ntrg": ntrg, "wavek": wavek, "depth": depth}


def listed():
    return [
        # one small system solved by itself (the smallest of the batched configuration): launches and latency
        _case("laplace_2k_mixed", "evaluate", "laplace", "mixed", 6, 64, "cube", 2003),
        # the constructors' defaults (FP64, p = 4, ncrit = 64) on a clustered set
        _case("laplace_20k_fp64", "evaluate", "laplace", "fp64", 4, 64, "plummer", 20011),
        # the reference's own calling convention: FP64, numpy arrays, the non-adaptive 100,000-body tree
        _case("laplace_100k_fp64_host", "evaluate_host", "laplace", "fp64", 8, 64, "cube", 100000, depth=4),
        # a time step of a moving set: tree, lists and evaluate at new positions
        _case("laplace_100k_moved", "moved", "laplace", "mixed", 6, 64, "cube", 100003),
        # sources and targets that differ (a field sampled on other points), adaptive tree
        _case("laplace_300k_probes", "evaluate", "laplace", "mixed", 8, 128, "plummer", 300007, ntrg=150001),
        # the full-precision path at scale
        _case("laplace_1m_fp64", "evaluate", "laplace", "fp64", 8, 128, "cube", 1000000),
        # the high-order configuration in mixed precision
        _case("laplace_1m_p10_mixed", "evaluate", "laplace", "mixed", 10, 128, "cube", 1000000),
        # the headline workload, the largest
        _case("laplace_4m_mixed", "evaluate", "laplace", "mixed", 8, 128, "cube", 4000000),
        # screened interactions on a surface, forward and backward: adaptive tree, operators per level
        _case("yukawa_300k_adjoint", "adjoint", "modified_helmholtz", "mixed", 10, 64, "sphere", 300000, wavek=10.0),
        # low-frequency scattering: complex charges and operators, mixed precision, high order
        _case("helmholtz_200k_mixed", "evaluate", "helmholtz", "mixed", 12, 64, "cube", 200000, wavek=20.0),
        # the complex kernel in full precision, a moderate size
        _case("helmholtz_50k_fp64", "evaluate", "helmholtz", "fp64", 8, 100, "cube", 50021, wavek=10.0),
        # many independent systems of uneven size (2,000 to 200,000 bodies, cubes and Plummer spheres) in one
        # graph, full precision
        _case("batch_24_fp64", "batch", "laplace", "fp64", 6, 64, "mixture", 24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case over the ranges that the listed ones stand for."""
    kind = rng.choice(["laplace", "laplace", "laplace", "laplace_fp64", "laplace_fp64", "host", "moved", "yukawa",
                       "helmholtz", "batch"])
    cloud = rng.choice(["cube", "plummer", "sphere"])
    ncrit = rng.choice([50, 64, 100, 128])
    if kind == "laplace":
        n = _log(rng, 2000, 3000000)
        ntrg = _log(rng, 1000, n) if rng.random() < 0.3 else 0
        return _case("", "evaluate", "laplace", "mixed", rng.choice([4, 6, 8, 10]), ncrit, cloud, n, ntrg)
    if kind == "laplace_fp64":
        n = _log(rng, 2000, 1000000)
        return _case("", "evaluate", "laplace", "fp64", rng.choice([4, 6, 8, 10]), ncrit, cloud, n)
    if kind == "host":
        return _case("", "evaluate_host", "laplace", rng.choice(["fp64", "mixed"]), rng.choice([4, 6, 8]), ncrit, "cube",
                     _log(rng, 10000, 300000), depth=rng.choice([-1, 3, 4]))
    if kind == "moved":
        return _case("", "moved", "laplace", rng.choice(["fp64", "mixed"]), rng.choice([4, 6, 8]), ncrit, cloud,
                     _log(rng, 5000, 500000))
    if kind == "yukawa":
        return _case("", rng.choice(["evaluate", "adjoint"]), "modified_helmholtz", rng.choice(["fp64", "mixed"]),
                     rng.choice([6, 8, 10]), ncrit, cloud, _log(rng, 3000, 300000), wavek=rng.choice([1.0, 5.0, 10.0]))
    if kind == "helmholtz":
        precision = rng.choice(["fp64", "mixed"])
        return _case("", "evaluate", "helmholtz", precision, rng.choice([6, 8, 10, 12]), ncrit, "cube",
                     _log(rng, 3000, 200000 if precision == "mixed" else 60000), wavek=rng.choice([5.0, 10.0, 20.0]))
    return _case("", "batch", "laplace", "fp64", rng.choice([4, 6]), 64, "mixture", rng.randint(6, 30))


# ---------------------------------------------------------------- inputs
def _cloud(points, n, gen):
    """n points: the unit cube, the surface of the unit sphere, or a Plummer sphere truncated at r = 10."""
    if points == "cube":
        return torch.rand(n, 3, dtype=torch.float64, device="cuda", generator=gen)
    g = torch.randn(n, 3, dtype=torch.float64, device="cuda", generator=gen)
    g /= g.norm(dim=1, keepdim=True)
    if points == "sphere":
        return g
    u = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    u = u * (1.0 + 0.01) ** -1.5  # mass inside r = 10
    r = 1.0 / torch.sqrt(torch.clamp(u, min=1e-300) ** (-2.0 / 3.0) - 1.0)
    return g * r[:, None]


def _charges(kernel, n, gen):
    q = torch.rand(n, 2 if kernel == "helmholtz" else 1, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    return torch.view_as_complex(q) if kernel == "helmholtz" else q[:, 0].contiguous()


def _inputs(case, seed):
    """(sources, charges, targets, cotangent) on the device, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = _cloud(case["points"], case["n"], gen)
    q = _charges(case["kernel"], case["n"], gen)
    y = _cloud(case["points"], case["ntrg"], gen) if case["ntrg"] else x
    w = torch.randn(y.shape[0], dtype=torch.float64, device="cuda", generator=gen) if case["call"] == "adjoint" else None
    return x, q, y, w


def _sizes(case):
    """Bodies of each system of a batch: log-uniform in [2,000, 200,000], fixed by the number of systems."""
    rng = np.random.default_rng(case["n"])
    return np.exp(rng.uniform(math.log(2000), math.log(200000), case["n"])).astype(np.int64).tolist()


def _systems(case, seed):
    """Cubes and Plummer spheres by turns, as the batched configuration has them: (coordinates, charges)."""
    rng = np.random.default_rng(seed)
    return [(rng.random((n, 3)) if i % 2 == 0 else plummer(n, rng), rng.uniform(-1.0, 1.0, n))
            for i, n in enumerate(_sizes(case))]


def _fmm(case):
    m, p, ncrit, prec = _MODULES[case["kernel"]], case["p"], case["ncrit"], case["precision"]
    if case["kernel"] == "laplace":
        return m, m.LaplaceFmm(p, ncrit, precision=prec)
    if case["kernel"] == "modified_helmholtz":
        return m, m.ModifiedHelmholtzFmm(p, ncrit, case["wavek"], precision=prec)
    return m, m.HelmholtzFmm(p, ncrit, complex(case["wavek"]), precision=prec)


def _depth(case):
    return None if case["depth"] < 0 else case["depth"]


# ---------------------------------------------------------------- one pass
def prepare(case, seed):
    if case["call"] == "batch":
        b = BatchedFmm(_systems(case, seed), lambda: _fmm(case)[1])
        b.capture(nstreams=8)
        return {"call": "batch", "batch": b}
    m, fmm = _fmm(case)
    x, q, y, w = _inputs(case, seed)
    s = {"call": case["call"], "m": m, "fmm": fmm, "x": x, "q": q, "y": y, "w": w, "depth": _depth(case)}
    if case["call"] == "moved":
        # the step before: operators and CUDA context are in place, the tree is that step's own
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        old = _cloud(case["points"], case["n"], gen)
        m.evaluate(_setup(m, fmm, old, q, old, None), fmm, out=_out(case, old.shape[0]))
        s["out"] = _out(case, y.shape[0])
        return s
    if case["call"] == "evaluate_host":
        s["x"], s["q"] = x.cpu().numpy(), q.cpu().numpy()
        s["y"] = s["x"] if y is x else y.cpu().numpy()
        s["tree"] = _setup(m, fmm, s["x"], s["q"], s["y"], s["depth"])
        return s
    s["tree"] = _setup(m, fmm, x, q, y, s["depth"])
    if case["call"] == "adjoint":
        s["q"].requires_grad_(True)
        s["x"].requires_grad_(True)
    else:
        s["out"] = _out(case, y.shape[0])
    return s


def _setup(m, fmm, x, q, y, depth):
    return m.setup(m.init_sources(x, q), m.init_targets(y), fmm, nonadaptive_depth=depth)


def _out(case, n):
    return torch.empty(n, 4, dtype=torch.complex128 if case["kernel"] == "helmholtz" else torch.float64, device="cuda")


def run(state):
    call = state["call"]
    if call == "batch":
        return list(state["batch"].replay())
    m, fmm = state["m"], state["fmm"]
    if call == "evaluate":
        m.update_charges(state["tree"], state["q"])
        return m.evaluate(state["tree"], fmm, out=state["out"])
    if call == "evaluate_host":
        m.update_charges(state["tree"], state["q"])
        return m.evaluate(state["tree"], fmm)
    if call == "moved":
        tree = _setup(m, fmm, state["x"], state["q"], state["y"], state["depth"])
        return m.evaluate(tree, fmm, out=state["out"])
    out = fmm_apply(state["q"], state["x"], state["x"], fmm, tree=state["tree"])
    dq, dx = torch.autograd.grad((out[:, 0] * state["w"]).sum(), (state["q"], state["x"]))
    return [out.detach(), dq, dx]


# ---------------------------------------------------------------- what a pass cannot do without
def _mean_spacing_pairs(case, n, nt):
    """Direct pairs of an FMM with leaves of about ncrit / 2 bodies: 27 neighbour leaves in a volume, 9 on a
    surface."""
    return nt * min(n, (9 if case["points"] == "sphere" else 27) * case["ncrit"] / 2.0)


def _work(case, n, nt):
    p, cplx = case["p"], case["kernel"] == "helmholtz"
    nsurf = 6 * (p - 1) ** 2 + 2
    pair = {"laplace": 20, "modified_helmholtz": 30, "helmholtz": 45}[case["kernel"]]
    cm = 4 if cplx else 1
    leaves = max(n, nt) / (case["ncrit"] / 2.0)
    flops = _mean_spacing_pairs(case, n, nt) * pair + (n + nt) * nsurf * pair  # P2P; P2M and L2P surfaces
    flops += leaves * cm * (4 * 2 * nsurf ** 2 + 2 * 2 * nsurf ** 2)           # pseudo-inverses, M2M and L2L
    nfreq = (2 * p) ** 3 if cplx else (2 * p) ** 2 * (p + 1)
    flops += leaves * (189 / 8.0) * nfreq * 8                                  # M2L products
    v = 2 if cplx else 1
    nbytes = 8 * (n * (3 + v) + (nt * 3 if case["ntrg"] else 0) + nt * 4 * v)
    return {"bytes": float(nbytes), "flops": float(flops)}


def work(case):
    if case["call"] == "batch":
        each = [_work(case, n, n) for n in _sizes(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    w = _work(case, case["n"], case["ntrg"] or case["n"])
    if case["call"] == "adjoint":
        w = {"bytes": w["bytes"] * 2, "flops": w["flops"] * 2}
    return w


# ---------------------------------------------------------------- direct sums in 64 bits
def _direct(kernel, wavek, x, q, y):
    """Potential and gradient at y of the charges q at x, (ntrg, 4), by direct summation."""
    cdtype = torch.complex128 if kernel == "helmholtz" else torch.float64
    out = torch.empty(y.shape[0], 4, dtype=cdtype, device=y.device)
    c = x.mean(dim=0)
    xc, yc = x - c, y - c
    rhs = torch.cat([q[:, None], q[:, None] * xc], dim=1)  # q, q x: the gradient's moments
    xt = xc.t().contiguous()
    rows = max(1, (1 << 23) // x.shape[0])
    buf = torch.empty(3, rows, x.shape[0], dtype=torch.float64, device=y.device)
    k = complex(wavek)
    for i in range(0, y.shape[0], rows):
        t = yc[i:i + rows]
        d, r2, inv = buf[0, :len(t)], buf[1, :len(t)], buf[2, :len(t)]
        torch.sub(t[:, :1], xt[:1], out=d)
        torch.mul(d, d, out=r2)
        for a in (1, 2):
            torch.sub(t[:, a:a + 1], xt[a:a + 1], out=d)
            r2.addcmul_(d, d)
        r2.masked_fill_(r2 == 0, math.inf)  # a coincident pair contributes nothing
        torch.rsqrt(r2, out=inv)
        if kernel == "laplace":
            g = inv
            c3 = torch.div(inv, r2, out=d)
        else:
            inv2 = inv * inv
            kr = r2.mul_(inv).nan_to_num_(posinf=0.0, nan=0.0).mul_(k.real)
            if kernel == "modified_helmholtz":
                g = torch.exp(-kr).mul_(inv)
                c3 = kr.add_(1.0).mul_(g).mul_(inv2)
            else:
                g = torch.polar(inv, kr)
                c3 = g * torch.complex(inv2, inv * -k.real)
        out[i:i + rows, 0] = g @ q
        m = c3 @ rhs
        out[i:i + rows, 1:] = m[:, 1:] - m[:, :1] * t
    return out * (1.0 / (4.0 * math.pi))


def exact(case, seed):
    if case["call"] == "batch":
        res = []
        for x, q in _systems(case, seed):
            x, q = torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda")
            res.append(_direct("laplace", 0.0, x, q, x))
        return res
    n, nt = case["n"], case["ntrg"] or case["n"]
    if float(n) * nt > 1.1e11:
        return None
    x, q, y, w = _inputs(case, seed)
    out = _direct(case["kernel"], case["wavek"], x, q, y)
    if case["call"] == "adjoint":
        psi = _direct(case["kernel"], case["wavek"], y, w, x)
        return [out, psi[:, 0].contiguous(), q[:, None] * psi[:, 1:] + w[:, None] * out[:, 1:]]
    return out.cpu().numpy() if case["call"] == "evaluate_host" else out
