"""Performance cases of the solver path.

A case is one call that a user's program repeats: the solver object (the plan)
is built once, and ``run`` puts fresh right-hand sides through it.  Sizes are
those of ``fixedeffects.jl_b200/synth.py`` (the benchmark configurations and
the reference's own benchmark problems) and generic ones around them.

The right-hand sides of mixed-precision cases are float32, those of FP64 cases
float64, solved to the default tol = 1e-8 except where a case says otherwise.
Returned are the residuals (or the fitted coefficients of every observation)
and the convergence flags; the iteration counts are a diagnostic that the
rounding of a sum can shift by one.
"""
import math

import numpy as np
import torch

import __graft_entry__ as entry

MAXITER = 10_000


def listed():
    return [
        # a small sample or one cell of a loop over subsamples: launches and latency
        _case("tiny_2k_1col", 2_000, "200,20"),
        # an ordinary regression, y and four regressors, three weighted effects, odd sizes
        _case("regressors_150k_5col", 150_001, "12007,701,23", cols=5, weighted=True),
        # the two-effect configuration in double precision
        _case("two_fe_1m_fp64", 1_000_000, "100000,100", precision="fp64"),
        # the reference's "simple" benchmark problem in double precision
        _case("simple_10m_fp64", 10_000_000, "100000,100", precision="fp64"),
        # three effects, the last one interacted with a covariate, weighted
        _case("three_fe_interacted_10m", 10_000_000, "1000000,100,1000", weighted=True,
              interacted=True),
        # the headline configuration: worker, firm and year effects, 32 columns at once
        _case("worker_firm_year_10m_32col", 10_000_000, "2000000,200000,20", zipf=1.1, cols=32),
        # many subsamples of uneven size solved together
        _case("uneven_256_problems", 1_000_000, "10,50", call="batch", problems=256,
              weighted=True),
        # the largest configuration: 100M weighted rows, a heavily skewed second effect
        _case("large_zipf_100m_8col", 100_000_000, "10000000,10000", zipf=1.3, cols=8,
              weighted=True),
        # the reference's "hard" worker-firm benchmark problem: thousands of iterations; at
        # 1e-8 its residuals are off by 1e-4, so it is solved until they are right in float32
        _case("hard_800k", 800_000, "400000,50000", local=True, tol=1e-11),
        # the fixed effects themselves: coefficients from host data, normalised, per row
        _case("coefficients_1m_fp64", 1_000_000, "50000,1000,20", precision="fp64",
              call="coefficients"),
        # iteratively reweighted least squares: new weights, then a solve, each pass
        _case("reweighted_2m_3col", 2_000_000, "150000,5000", cols=3, weighted=True,
              call="reweighted"),
        # a one-off call on host data: the plan is built, used once and freed
        _case("one_shot_300k_2col", 300_000, "20000,500,12", cols=2, call="one_shot"),
    ]


def _case(name, n, levels, *, cols=1, precision="mixed", weighted=False, interacted=False,
          zipf=0.0, local=False, call="device", problems=1, tol=1e-8):
    c = {"n": n, "levels": levels, "cols": cols, "precision": precision, "weighted": weighted,
         "interacted": interacted, "zipf": zipf, "local": local, "call": call,
         "problems": problems, "tol": tol}
    return dict({"name": name}, **c) if name else c


def draw(rng):
    """Rows from 2 thousand to 20 million, 1 to 32 columns, two or three
    effects, every call of the listed cases and the host-matrix and
    collection calls."""
    call = rng.choice(["device"] * 6 + ["host", "columns", "batch", "coefficients", "reweighted",
                                        "one_shot"])
    on_host = call in ("host", "columns", "coefficients", "one_shot")
    n = int(math.exp(rng.uniform(math.log(2e3), math.log(3e6 if on_host else 2e7)))) | 1
    precision = "fp64" if call == "coefficients" or rng.random() < 0.25 else "mixed"
    if call == "batch":
        n = min(n, 500_001)
        return _case("", n, "%d,%d" % (rng.randint(6, 20), rng.randint(8, 60)), call="batch",
                     problems=rng.randint(8, 150), precision=precision,
                     weighted=rng.random() < 0.5)
    first = max(4, int(n / math.exp(rng.uniform(math.log(4), math.log(60)))))
    second = max(3, int(math.exp(rng.uniform(math.log(3), math.log(max(4, first // 4))))))
    levels = [first, second]
    if rng.random() < 0.5:
        levels.append(rng.randint(3, 40) if rng.random() < 0.7 else min(1000, max(3, n // 50)))
    cols = 1 if call == "coefficients" else rng.choice([1, 1, 1, 2, 3, 5, 8, 13, 16, 24, 32])
    while cols > 1 and cols * n > 60_000_000:
        cols = (cols + 1) // 2
    return _case("", n, ",".join(map(str, levels)), cols=cols, precision=precision,
                 weighted=call == "reweighted" or rng.random() < 0.4,
                 interacted=len(levels) > 2 and call != "coefficients" and rng.random() < 0.3,
                 zipf=rng.choice([0.0, 0.0, 1.1, 1.3]), call=call)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _sizes(case):
    """Rows of each problem of a batch: log-uniform from 1000 to case["n"]."""
    p, hi = case["problems"], max(1001, case["n"])
    return [int(round(math.exp(math.log(1e3) + (i + 0.5) / p * math.log(hi / 1e3))))
            for i in range(p)]


def _levels(case):
    return [int(x) for x in case["levels"].split(",")]


def _float(case):
    return torch.float64 if case["precision"] == "fp64" else torch.float32


def _zipf(u, s, m):
    p = torch.arange(1, m + 1, dtype=torch.float64, device=u.device) ** -s
    cdf = torch.cumsum(p, 0)
    return torch.searchsorted(cdf / cdf[-1], u).clamp_(max=m - 1)


def _inputs(case, seed):
    """(refs, level counts, interactions, weights, y): 0-based int64 refs,
    y of shape (cols, n), all on the GPU; level ids of a batch are local to
    its problems and returned with their per-problem offsets added."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def uniform(n):
        return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)

    def normal(*shape, dtype=torch.float64):
        return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)

    if case["call"] == "batch":
        sizes = torch.tensor(_sizes(case), device="cuda")
        ratio, second = _levels(case)
        n = int(sizes.sum())
        prob = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), sizes)
        n1 = (sizes // ratio).clamp_(min=2)
        base = torch.cumsum(n1, 0) - n1
        refs = [base[prob] + (uniform(n) * n1[prob]).long(),
                second * prob + (uniform(n) * second).long()]
        nlev = [int(n1.sum()), second * len(sizes)]
        inter = [None, None]
    else:
        n, nlev = case["n"], _levels(case)
        if case["local"]:  # each worker's firms lie around worker / 8, as in the benchmark
            refs = [(uniform(n) * nlev[0]).long()]
            lo = (refs[0] // 8 - 10).clamp_(min=0)
            hi = torch.maximum((refs[0] // 8 + 10).clamp_(max=nlev[1] - 1), lo)
            refs.append(lo + (uniform(n) * (hi - lo + 1)).long())
        else:
            refs = [_zipf(uniform(n), case["zipf"], m) if k == 1 and case["zipf"] else
                    (uniform(n) * m).long() for k, m in enumerate(nlev)]
        inter = [None] * len(nlev)
        if case["interacted"]:
            inter[-1] = uniform(n)
    w = uniform(n) + 0.5 if case["weighted"] else None
    y = torch.empty(case["cols"], n, device="cuda", dtype=_float(case))
    for j in range(case["cols"]):
        if case["local"]:  # a uniform column, as the benchmark draws it
            y[j] = uniform(n)
            continue
        col = normal(n, dtype=y.dtype)
        for r, m, x in zip(refs, nlev, inter):
            e = normal(m, dtype=y.dtype)[r] * (0.2 + 0.05 * j)
            col += e if x is None else e * x.to(y.dtype)
        y[j] = col
    return refs, nlev, inter, w, y


def prepare(case, seed):
    fe = entry.load_package()
    refs, nlev, inter, w, y = _inputs(case, seed)
    T = np.float64 if case["precision"] == "fp64" else np.float32
    st = {"fe": fe, "call": case["call"], "y": y, "T": T, "tol": case["tol"]}
    host_w = None if w is None else w.cpu().numpy()
    host_x = [None if x is None else x.cpu().numpy() for x in inter]
    host = [r.add_(1).cpu().numpy() for r in refs]
    del refs, inter, w
    if case["call"] == "batch":
        sizes = _sizes(case)
        ratio, second = _levels(case)
        at, low = np.concatenate([[0], np.cumsum(sizes)]), 0
        problems = []
        for p, n in enumerate(sizes):
            s, n1 = slice(at[p], at[p + 1]), max(2, n // ratio)
            problems.append([fe.FixedEffect.from_refs(host[0][s] - low, n1),
                             fe.FixedEffect.from_refs(host[1][s] - p * second, second)])
            low += n1
        st["solver"] = fe.BatchSolver(
            problems, None if host_w is None else [host_w[at[p]:at[p + 1]]
                                                   for p in range(len(sizes))], T=T)
        st["work"] = torch.empty_like(y[0])
        st["y"] = y[0]
        return st
    fes = [fe.FixedEffect.from_refs(r, m, x) for r, m, x in zip(host, nlev, host_x)]
    if case["call"] == "one_shot":
        st["fes"], st["w"] = fes, host_w
    else:
        st["solver"] = fe.AbstractFixedEffectSolver(fes, host_w, "CUDA", T)
    if case["call"] in ("device", "reweighted"):
        st["work"] = torch.empty_like(y)
        st["w"] = host_w
    else:
        st["y"] = y.cpu().numpy()
    return st


def run(state):
    """One call.  A solve overwrites its right-hand sides, so the columns that
    the caller keeps are copied first."""
    call, y, tol = state["call"], state["y"], state["tol"]
    if call == "batch":
        state["work"].copy_(y)
        r, _, cv = state["solver"].solve_residuals_device(state["work"], tol=tol, maxiter=MAXITER)
    elif call in ("device", "reweighted"):
        if call == "reweighted":
            state["solver"].update_weights(state["w"])
        state["work"].copy_(y)
        r, _, cv = state["solver"].solve_residuals(state["work"].t(), tol=tol, maxiter=MAXITER)
    elif call == "coefficients":
        r, _, cv = state["solver"].solve_coefficients(y[0], tol=tol, maxiter=MAXITER)
    elif call == "columns":
        r, _, cv = state["solver"].solve_residuals([c.copy() for c in y], tol=tol,
                                                   maxiter=MAXITER)
    elif call == "host":
        r, _, cv = state["solver"].solve_residuals(y.copy().T, tol=tol, maxiter=MAXITER)
    else:
        r, _, cv = state["fe"].solve_residuals(y.copy().T, state["fes"], state["w"],
                                               double_precision=state["T"] == np.float64,
                                               tol=tol, maxiter=MAXITER)
    return {"result": r, "converged": cv}


def work(case):
    """Every right-hand side and level id read once, every result written once."""
    n = sum(_sizes(case)) if case["call"] == "batch" else case["n"]
    k = 2 if case["call"] == "batch" else len(_levels(case))
    s = 8 if case["precision"] == "fp64" else 4
    out = k * s * n if case["call"] == "coefficients" else n * case["cols"] * s
    ids = 4 * n * k + (8 * n if case["weighted"] else 0) + (8 * n if case["interacted"] else 0)
    if case["call"] == "one_shot":  # the level ids arrive as 64-bit host data
        ids += 4 * n * k
    # two operator applications at least: a multiply and an add per entry and column
    return {"bytes": n * case["cols"] * s + ids + out, "flops": 4 * n * k * case["cols"]}


# ---------------------------------------------------------------------------
# the same results in 64 bits, by conjugate gradients in plain torch
# ---------------------------------------------------------------------------
class _Design:
    """Columns of one effect: cw[i] at (i, ref[i])."""

    def __init__(self, ref, n, cw):
        self.ref, self.n, self.cw = ref, n, cw
        # hot levels are summed in several parts
        self.parts = max(1, min(64, 4_000_000 // max(1, n)))
        self.slot = ref * self.parts + torch.arange(ref.numel(), device="cuda") % self.parts

    def mul(self, x):
        return x[self.ref] if self.cw is None else x[self.ref] * self.cw[:, None]

    def tmul(self, u):
        s = torch.zeros(self.n * self.parts, u.shape[1], device="cuda", dtype=torch.float64)
        s.index_add_(0, self.slot, u if self.cw is None else u * self.cw[:, None])
        return s.view(self.n, self.parts, -1).sum(1)


def _least_squares(refs, nlev, inter, w, y):
    """(unweighted residuals (n, cols), coefficients per effect) of the
    weighted least-squares fit of y on the effects: the first effect is
    projected out, conjugate gradients on the normal equations of the rest."""
    sw = None if w is None else w.sqrt()
    cws = [sw if x is None else x if sw is None else x * sw for x in inter]
    first, *rest = [_Design(r, m, cw) for r, m, cw in zip(refs, nlev, cws)]
    one = torch.ones(refs[0].numel(), 1, device="cuda", dtype=torch.float64)

    def inverse(t):
        return torch.where(t > 0, 1 / torch.where(t > 0, t, torch.ones_like(t)),
                           torch.zeros_like(t))

    def norms(d):
        return d.tmul(one if d.cw is None else d.cw[:, None])

    d1 = inverse(norms(first))
    scale = [inverse(norms(d).sqrt()) for d in rest]
    b = y.t().double()
    if sw is not None:
        b = b * sw[:, None]

    def project(u):
        return u - first.mul(d1 * first.tmul(u))

    def forward(x):
        return sum(d.mul(s * v) for d, s, v in zip(rest, scale, x))

    def gradient(u):
        return [s * d.tmul(u) for d, s in zip(rest, scale)]

    def dot(p, q):
        return sum((a * c).sum(0) for a, c in zip(p, q))

    x = [torch.zeros(d.n, b.shape[1], device="cuda", dtype=torch.float64) for d in rest]
    g = gradient(project(b))
    p, gg = g, dot(g, g)
    goal = gg * 1e-27
    for it in range(20_000):
        if it % 16 == 0 and bool((gg <= goal).all()):
            break
        live = gg > goal
        q = gradient(project(forward(p)))
        step = torch.where(live, gg / dot(p, q).clamp_(min=1e-300), 0)
        x = [a + step * c for a, c in zip(x, p)]
        g = [a - step * c for a, c in zip(g, q)]
        new = torch.where(live, dot(g, g), gg)
        beta = torch.where(live, new / gg.clamp(min=1e-300), 0)
        p = [a + beta * c for a, c in zip(g, p)]
        gg = new
    rest_fit = forward(x)
    r = project(b - rest_fit)
    coefs = [d1 * first.tmul(b - rest_fit)] + [s * v for s, v in zip(scale, x)]
    return (r if sw is None else r / sw[:, None]), coefs


def exact(case, seed):
    refs, nlev, inter, w, y = _inputs(case, seed)
    cols = 8 if y.shape[0] * y.shape[1] > 50_000_000 else y.shape[0]  # columns at a time
    parts = [_least_squares(refs, nlev, inter, w, y[j:j + cols])
             for j in range(0, y.shape[0], cols)]
    if case["call"] == "coefficients":
        coefs = [c[:, 0] for c in parts[0][1]]
        for k in range(len(coefs) - 1, 0, -1):
            seen = torch.zeros(nlev[k], dtype=torch.bool, device="cuda")
            seen[refs[k]] = True
            mean = coefs[k][seen].mean()
            coefs[k] = coefs[k] - mean
            coefs[0] = coefs[0] + mean
        return {"result": [c[r].cpu() for c, r in zip(coefs, refs)], "converged": None}
    r = torch.cat([p[0] for p in parts], 1)
    if case["call"] == "batch":
        return {"result": r[:, 0], "converged": None}
    return {"result": list(r.t()) if case["call"] == "columns" else r, "converged": None}
