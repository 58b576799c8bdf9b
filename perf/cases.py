"""The work that stands for this framework in use, as cases that can be timed and compared.

Each case is a plain dict; `prepare` makes its inputs on the GPU together with the object a program keeps (a solver
object, a context, a plan), `run` is one call through the public entry points, `work` the bytes and operations the
call cannot do without and `exact` the direct sum in 64 bits that the call approximates (or computes).

Kinds:
  exact    pyfmma's default solver, the direct sum
  fmm      one solve through Context.solve or (where inputs are float32 or the reference's own benchmark) pyfmma
  tree     the reference's O(N log N) solver
  adjoint  pyfmma.torch.fmm, forward and backward with respect to targets, sources and weights
  forest   many independent problems with several right-hand sides in one call
  plan     one geometry, new weights on every call
"""
import math

import numpy as np
import torch

import fmma_b200
import pyfmma
import pyfmma.torch as pyfmma_torch

# the radial kernels of the configurations and tests, with the parameters those use
P0 = {"inv_r": 0.0, "inv_r_safe": 0.0, "inv_diff": 0.0, "log_r": 0.0, "gaussian": 0.01, "multiquadric": 1e-4}


def _depth(n, dim, cap, dist):
    """Depth at which the fullest leaf holds about `cap` points (the 16 narrow clusters fill ~8^4 times fewer boxes
    than uniform points do)."""
    depth = int(math.ceil(math.log(max(n / cap, 1.0), 2 ** dim))) + 1
    return max(3, depth + (4 if dist == "clustered" else 0))


def _case(name, kind, dim, n, m=0, *, kernel="inv_r_safe", poly_ord=5, depth=-1, precision="fp64", nrhs=1,
          dist="uniform", weights="uniform", f32=False, problems=0, lo=0, hi=0, cap=64):
    c = dict(kind=kind, dim=dim, n=n, m=m or n, kernel=kernel, poly_ord=poly_ord, depth=depth, precision=precision,
             nrhs=nrhs, dist=dist, weights=weights, f32=f32, problems=problems, lo=lo, hi=hi, cap=cap)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call of the reference's published benchmark: the default solver, unweighted
        _case("exact-2d-2048", "exact", 2, 2048, kernel="inv_r", poly_ord=1, weights="none"),
        # the largest size of that benchmark, where the direct sum is what every other solver is checked against
        _case("exact-2d-131072", "exact", 2, 131072, kernel="inv_r", poly_ord=1, weights="none"),
        # a small fmm call, where latency and launches count: 1-D 1/(x-y), 8 nodes
        _case("fmm-1d-4096", "fmm", 1, 4096, kernel="inv_diff", poly_ord=7, depth=8),
        # the reference benchmark's 2-D fmm at its finest order and largest size, default Depth
        _case("fmm-2d-131072", "fmm", 2, 131072, kernel="inv_r", poly_ord=3, depth=-1, weights="none"),
        # a planar potential problem in mixed precision: 1M points, log r, 6 nodes
        _case("fmm-2d-1m-tf32x3", "fmm", 2, 1_000_000, kernel="log_r", poly_ord=5, depth=9, precision="tf32x3",
              weights="normal"),
        # plain double precision on clustered 3-D points, the default precision of every entry point
        _case("fmm-3d-clustered-fp64", "fmm", 3, 262_144, poly_ord=5, depth=9, dist="clustered"),
        # the headline configuration: 4M clustered points, split-precision tensor cores
        _case("fmm-3d-clustered-4m-bf16x3", "fmm", 3, 4_194_304, poly_ord=5, depth=10, precision="bf16x3",
              dist="clustered"),
        # float32 arrays through the float class, an odd size, more sources than targets
        _case("fmm-3d-float-bf16x3", "fmm", 3, 250_001, 333_333, poly_ord=4, depth=5, precision="bf16x3", f32=True),
        # training step through autograd: 3-D Gaussian, 5 nodes, every gradient
        _case("adjoint-3d-1m", "adjoint", 3, 1 << 20, kernel="gaussian", poly_ord=4, depth=6, weights="normal"),
        # a batch of 512 uneven 2-D problems with 16 right-hand sides
        _case("forest-2d-512x16", "forest", 2, 0, kernel="multiquadric", poly_ord=4, precision="bf16x3", nrhs=16,
              weights="normal", problems=512, lo=1000, hi=200_000, cap=64),
        # an iterative solver's matvec: one geometry, new weights on every call
        _case("plan-3d-200k", "plan", 3, 200_000, poly_ord=4, depth=5, nrhs=2),
        # the reference's tree solver
        _case("tree-3d-200k", "tree", 3, 200_000, poly_ord=5, depth=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["exact", "fmm", "fmm", "fmm", "fmm", "adjoint", "forest", "plan", "tree"])
    dim = rng.choice([1, 2, 2, 3, 3, 3])
    radial = ["inv_r_safe", "log_r", "gaussian", "multiquadric"]
    weights = rng.choice(["uniform", "normal"])
    if kind == "exact":
        n = _log(rng, 500, 131072)
        m = min(_log(rng, 500, 400_000), 131072 * 131072 // n)
        return _case("", kind, dim, n, m, kernel=rng.choice(radial), poly_ord=1, weights=rng.choice(["none", weights]),
                     f32=rng.random() < 0.25)
    if kind == "fmm":
        if dim == 1:
            n = _log(rng, 1000, 200_000)
            return _case("", kind, 1, n, kernel=rng.choice(["inv_diff", "log_r"]), poly_ord=rng.randint(3, 7),
                         depth=_depth(n, 1, 32, "uniform"), weights=weights)
        precision = rng.choice(["fp64", "fp64", "bf16x3", "tf32x3"])
        dist = rng.choice(["uniform", "clustered"])
        f32 = rng.random() < 0.25
        n = _log(rng, 2000, 1_000_000 if dim == 2 else 262_144 if precision == "fp64" else 1_000_000)
        m = int(n * rng.uniform(0.7, 1.3))
        return _case("", kind, dim, n, m, kernel=rng.choice(["inv_r_safe", "log_r"]),
                     poly_ord=rng.randint(3, 7 if dim == 2 else 5), depth=_depth(max(n, m), dim, 64 if dim == 2 else 128, dist),
                     precision=precision, nrhs=1 if n > 100_000 else rng.choice([1, 1, 3]), dist=dist, weights=weights,
                     f32=f32)
    if kind == "adjoint":
        dim = rng.choice([2, 3])
        n = _log(rng, 5000, 300_000)
        m = int(n * rng.uniform(0.7, 1.3))
        return _case("", kind, dim, n, m, kernel=rng.choice(["gaussian", "multiquadric", "inv_r_safe"]),
                     poly_ord=rng.randint(3, 5), depth=_depth(max(n, m), dim, 40, "uniform"), weights=weights,
                     precision=rng.choice(["fp64", "fp64", "bf16x3"]))
    if kind == "forest":
        return _case("", kind, 2, 0, kernel=rng.choice(["multiquadric", "log_r"]), poly_ord=rng.randint(3, 5),
                     precision=rng.choice(["bf16x3", "tf32x3", "fp64"]), nrhs=rng.choice([1, 4, 16]), weights=weights,
                     problems=rng.randint(5, 60), lo=1000, hi=_log(rng, 5000, 40_000))
    if kind == "plan":
        n = _log(rng, 5000, 300_000)
        dim = rng.choice([2, 3])
        return _case("", kind, dim, n, int(n * rng.uniform(0.7, 1.3)), kernel=rng.choice(["inv_r_safe", "multiquadric"]),
                     poly_ord=rng.randint(3, 5), depth=_depth(n, dim, 64, "uniform"), nrhs=rng.choice([1, 2, 4]))
    n = _log(rng, 3000, 200_000)
    return _case("", "tree", dim if dim > 1 else 2, n, kernel=rng.choice(["inv_r_safe", "log_r"]),
                 poly_ord=rng.randint(3, 5), depth=_depth(n, dim if dim > 1 else 2, 64, "uniform"), weights=weights)


def _points(case, gen, n):
    d = case["dim"]
    if case["dist"] == "uniform":
        return torch.rand((n, d), generator=gen, device="cuda", dtype=torch.float64)
    centres = torch.as_tensor(np.random.default_rng(7).uniform(0.1, 0.9, (16, d)), device="cuda")
    which = torch.randint(0, 16, (n,), generator=gen, device="cuda")
    noise = torch.randn((n, d), generator=gen, device="cuda", dtype=torch.float64)
    return (centres[which] + 0.02 * noise).clamp_(0.0, 1.0)


def _weights(case, gen, m):
    if case["weights"] == "none":
        return None
    shape = (m,) if case["nrhs"] == 1 else (case["nrhs"], m)
    if case["weights"] == "uniform":
        return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) * 2 - 1
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)


def _sizes(case):
    """Points of each problem of a forest: log-uniform, the same for every seed (the sizes are part of the case)."""
    r = np.random.default_rng(11)
    return np.exp(r.uniform(np.log(case["lo"]), np.log(case["hi"]), case["problems"])).astype(np.int64)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["kind"] == "forest":
        sizes = _sizes(case)
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        total, d = int(off[-1]), case["dim"]
        pid = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), torch.as_tensor(sizes, device="cuda"))
        side = torch.rand((len(sizes), 1), generator=gen, device="cuda", dtype=torch.float64) * 1.5 + 0.5
        corner = torch.rand((len(sizes), d), generator=gen, device="cuda", dtype=torch.float64) * 20 - 10
        t, s = (corner[pid] + side[pid] * torch.rand((total, d), generator=gen, device="cuda", dtype=torch.float64)
                for _ in range(2))
        return t, s, _weights(case, gen, total), off
    t, s = _points(case, gen, case["n"]), _points(case, gen, case["m"])
    w = _weights(case, gen, case["m"])
    if case["f32"]:
        t, s, w = t.float(), s.float(), None if w is None else w.float()
    return t, s, w, None


_HANDLES = {"inv_r": pyfmma.kernels.inv_r, "inv_r_safe": pyfmma.kernels.laplace, "inv_diff": pyfmma.kernels.inv_diff,
            "log_r": pyfmma.kernels.log_r, "gaussian": pyfmma.kernels.gaussian(P0["gaussian"]),
            "multiquadric": pyfmma.kernels.multiquadric(P0["multiquadric"])}


def prepare(case, seed):
    t, s, w, off = _inputs(case, seed)
    state = {"case": case, "t": t, "s": s, "w": w, "off": off, "ctx": fmma_b200.default_context(0)}
    kind, ctx = case["kind"], state["ctx"]
    if kind in ("exact", "tree") or (kind == "fmm" and (case["f32"] or case["weights"] == "none" or case["dim"] == 1)):
        f = getattr(pyfmma, "fmma%s%d" % ("f" if case["f32"] else "d", case["dim"]))()
        f.set_solver_type(kind)
        f.set_fn2(_HANDLES[case["kernel"]])
        f.set_poly_ord(case["poly_ord"])
        f.set_Depth(case["depth"])
        f.set_trans_sym_flag(1)
        f.set_precision(case["precision"])
        state["solver"] = f
        shape = (case["n"],) if case["nrhs"] == 1 else (case["nrhs"], case["n"])
        state["ans"] = torch.zeros(shape, dtype=t.dtype, device="cuda")
    elif kind == "adjoint":
        gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1_000_003)
        state["g"] = torch.randn(case["n"], generator=gen, device="cuda", dtype=torch.float64)
        for v in (t, s, w):
            v.requires_grad_(True)
    elif kind == "forest":
        ctx.set_kernel(case["kernel"], P0[case["kernel"]])
        state["depths"] = ctx.forest_depths(t, off, s, off, case["cap"])
    elif kind == "plan":
        ctx.set_kernel(case["kernel"], P0[case["kernel"]])
        state["plan"] = ctx.plan(t, [0, case["n"]], s, [0, case["m"]], case["nrhs"], [case["depth"]],
                                 poly_ord=case["poly_ord"], precision=case["precision"])
    return state


def run(state):
    case, t, s, w = state["case"], state["t"], state["s"], state["w"]
    if "solver" in state:
        args = (t, s) if w is None else (t, w, s)
        state["solver"].solve(*args, state["ans"])
        return state["ans"]
    if "plan" in state:
        return state["plan"].execute(w)
    if case["kind"] == "adjoint":
        for v in (t, s, w):
            v.grad = None
        c = pyfmma_torch.fmm(t, s, w, kernel=_HANDLES[case["kernel"]], poly_ord=case["poly_ord"], depth=case["depth"],
                             precision=case["precision"])
        c.backward(state["g"])
        return c.detach(), t.grad, s.grad, w.grad
    ctx = state["ctx"]
    with ctx.lock:
        ctx.set_kernel(case["kernel"], P0[case["kernel"]])
        if case["kind"] == "forest":
            return ctx.forest_solve(t, state["off"], s, state["off"], w, state["depths"], poly_ord=case["poly_ord"],
                                    precision=case["precision"])
        return ctx.solve(t, s, w, poly_ord=case["poly_ord"], depth=case["depth"], precision=case["precision"])[0]


def _pairs(case):
    """Point pairs of the direct sum."""
    if case["kind"] == "forest":
        return float(sum(float(x) ** 2 for x in _sizes(case)))
    return float(case["n"]) * case["m"]


def work(case):
    d, R, size = case["dim"], case["nrhs"], 4 if case["f32"] else 8
    n, m = (case["n"], case["m"]) if case["kind"] != "forest" else (int(_sizes(case).sum()),) * 2
    values = n * (d + R) + m * (d + (0 if case["weights"] == "none" else R))
    if case["kind"] == "plan":  # the geometry was read when the plan was made
        values = (n + m) * R
    pair = 3 * d + 2 + 2 * R  # difference, square and sum per dimension, the kernel, one multiply-add per weight set
    if case["kind"] == "exact":
        return {"bytes": values * size, "flops": _pairs(case) * pair}
    # each point through one leaf expansion and, with its neighbours in 3^d leaves, the near field
    P, near = (case["poly_ord"] + 1) ** d, 3 ** d * (16 if case["dist"] == "clustered" else 24)
    flops = 2.0 * (n + m) * P * R + float(n) * near * pair
    if case["kind"] == "adjoint":
        # g is read, one gradient per input written; the transposed field and the gradients in d directions
        return {"bytes": (values + n + n * d + m * d + m) * size, "flops": flops * (2 + d)}
    return {"bytes": values * size, "flops": flops}


def _kernel(case, r2, diff):
    """f and, for the gradient, its factor c in grad_x f = c (x - y), from |x - y|^2 (and x - y in one dimension)."""
    k, p0 = case["kernel"], P0[case["kernel"]]
    if k == "inv_diff":
        return torch.where(diff != 0, 1 / diff, 0.0), None
    if k == "log_r":
        return torch.where(r2 > 0, 0.5 * torch.log(r2), 0.0), None
    if k == "gaussian":
        f = torch.exp(-r2 / p0)
        return f, -2 / p0 * f
    if k == "multiquadric":
        f = torch.sqrt(r2 + p0)
        return f, 1 / f
    f = torch.rsqrt(r2)
    if k == "inv_r_safe":
        f = torch.where(r2 > 0, f, 0.0)
    return f, -f * f * f


def _direct(case, t, s, w, grad=False):
    """sum_j w[r, j] f(t_i, s_j) and, with `grad`, sum_j w[j] grad_x f(t_i, s_j), a block of targets at a time."""
    n, d = t.shape
    out = torch.empty((w.shape[0], n), dtype=torch.float64, device=t.device)
    g = torch.empty((n, d), dtype=torch.float64, device=t.device) if grad else None
    step = max(1, (1 << 26) // max(1, s.shape[0]))
    for i in range(0, n, step):
        x = t[i:i + step]
        diff = x[:, None, 0] - s[None, :, 0]
        r2 = diff * diff
        for q in range(1, d):
            r2 += (x[:, None, q] - s[None, :, q]) ** 2
        f, c = _kernel(case, r2, diff)
        out[:, i:i + step] = w @ f.T
        if grad:
            for q in range(d):
                g[i:i + step, q] = ((x[:, None, q] - s[None, :, q]) * c) @ w[0]
    return out, g


def exact(case, seed):
    if _pairs(case) * (4 if case["kind"] == "adjoint" else 1) > 1.5e11:
        return None  # over about 20 seconds
    t, s, w, off = _inputs(case, seed)
    one = w is None or w.dim() == 1
    t, s = t.double(), s.double()
    w = torch.ones((1, s.shape[0]), dtype=torch.float64, device=s.device) if w is None else w.double()
    w = w[None] if w.dim() == 1 else w
    if case["kind"] == "forest":
        out = torch.cat([_direct(case, t[a:b], s[a:b], w[:, a:b])[0] for a, b in zip(off[:-1], off[1:])], dim=1)
        return out[0] if one else out
    if case["kind"] != "adjoint":
        out, _ = _direct(case, t, s, w)
        return out[0] if one else out
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1_000_003)
    g = torch.randn(case["n"], generator=gen, device="cuda", dtype=torch.float64)
    c, dx = _direct(case, t, s, w, grad=True)
    dw, dy = _direct(case, s, t, g[None], grad=True)  # these kernels are symmetric: f(x, y) = f(y, x)
    return c[0], g[:, None] * dx, w[0][:, None] * dy, dw[0]
