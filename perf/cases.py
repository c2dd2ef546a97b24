"""What is timed: fits of high-dimensional fixed-effects regressions as a user's
program runs them, over the shapes that the benchmark, the tests and the
documentation of this repository work on.

A case is one call of a public entry point ("call") on one kind of panel
("data") with the options a configuration can set. Panels are made on the GPU
from the seed alone; a case that hands host arrays over keeps them on the host,
and its upload counts.

Kinds of panel:
  wages    unbalanced person x year panel with an occupation (nlswork-like)
  matched  worker x period panel over firms of Pareto(1.5) sizes
  levels   rows drawn uniformly over one large and two small dimensions
  iv       2SLS panel with categorical regressors, given by a formula
  batch    many independent specifications of uneven size
"""
import math

import numpy as np
import torch

from fe_gpu_gb300 import fe_gpu_estimate, fe_gpu_estimate_device, fe_gpu_within_transform_device, fe_runtime_config
from fe_gpu_gb300.bin_io import fe_dataset_header, fe_host_arrays
from fe_gpu_gb300.estimator import fe_batch_spec, fe_gpu_estimate_batch
from fe_gpu_gb300.formula import RawDevice, expand_formula, fit_formula

IV_FORMULA = ("y ~ x_end i.2.cat_end x1 x2 x3 x4 x5 x6 x1&x2 i.cat_a&&i.cat_b (x_end i.2.cat_end ~ z1 i.zc), "
              "fe(f1 f2 f3) cluster(f1 f2)")
#: Columns that IV_FORMULA expands to: regressors and instruments.
IV_K, IV_L = 90, 20


def listed():
    return [
        # the smallest call: a short panel with the defaults, from host arrays
        dict(name="short_panel_host", call="host", data="wages", ids=100, k=2, fes=2, precision="fp64", cg=False,
             tol=1e-6, clusters=0),
        # a survey panel of about 28,000 rows as a script fits it: the defaults, SEs clustered by person
        dict(name="wages_host", call="host", data="wages", ids=3500, k=5, fes=3, precision="fp64", cg=False, tol=1e-6,
             clusters=1),
        # the same kind of panel with many regressors, resident on the device, the fast options, 3-way clusters
        dict(name="wages_many_columns", call="device", data="wages", ids=4700, k=29, fes=3, precision="mixed", cg=True,
             tol=1e-9, clusters=3),
        # a matched employer-employee panel with gaps, plain FP64, from host arrays, 3-way clusters
        dict(name="matched_900k_host", call="host", data="matched", workers=50_000, firms=5_000, periods=20, move=0.1,
             keep=0.9, shuffle=False, k=8, precision="fp64", cg=False, tol=1e-8, clusters=3),
        # register data: 5M rows, 940k persons and two small dimensions, plain FP64, homoskedastic
        dict(name="levels_5M", call="device", data="levels", n=5_000_000, g0=940_423, g1=13, g2=12, k=3,
             precision="fp64", cg=False, tol=1e-8, clusters=0),
        # few levels and many rows, plain FP64, 3-way clusters
        dict(name="levels_few_13M", call="device", data="levels", n=13_000_003, g0=4_142, g1=13, g2=12, k=3,
             precision="fp64", cg=False, tol=1e-8, clusters=3),
        # mixed precision without conjugate gradients on rows in no order, singletons dropped, 2-way clusters
        dict(name="matched_shuffled_mixed", call="device", data="matched", workers=120_000, firms=15_000, periods=12,
             move=0.15, keep=0.8, shuffle=True, k=4, precision="mixed", cg=False, tol=1e-8, clusters=2,
             singletons=True),
        # the benchmark's 20M-row panel: mixed precision, conjugate gradients, 3-way clusters
        dict(name="matched_20M", call="device", data="matched", workers=1_000_000, firms=100_000, periods=20, move=0.1,
             keep=1.0, shuffle=False, k=8, precision="mixed", cg=True, tol=1e-8, clusters=3),
        # the benchmark's largest panel
        dict(name="matched_150M", call="device", data="matched", workers=5_000_000, firms=1_000_000, periods=30,
             move=0.05, keep=1.0, shuffle=False, k=8, precision="mixed", cg=True, tol=1e-8, clusters=3),
        # 2SLS given by a formula: expansion to 111 columns and the fit
        dict(name="iv_formula_1M", call="formula", data="iv", n=1_000_001, g0=50_000, g1=5_000, g2=30,
             precision="mixed", cg=True, tol=1e-8),
        # a specification table: many regressions of uneven size in one call
        dict(name="batch_60", call="batch", data="batch", specs=60, lo=5_000, hi=200_000, precision="mixed", cg=True,
             tol=1e-8),
        # the within-transform alone, in place, for columns that go on to another estimator
        dict(name="within_2M", call="within", data="matched", workers=100_000, firms=12_000, periods=20, move=0.1,
             keep=0.97, shuffle=False, k=11, precision="fp64", cg=False, tol=1e-6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    data = rng.choice(["wages", "wages", "matched", "matched", "matched", "levels", "levels", "iv", "batch"])
    precision, cg = rng.choice([("fp64", False), ("fp64", False), ("mixed", True), ("mixed", True), ("mixed", False)])
    tol = rng.choice([1e-6, 1e-8]) if precision == "fp64" else 1e-8 if data == "matched" else 1e-9
    case = dict(data=data, precision=precision, cg=cg, tol=tol)
    if data == "wages":
        fes = rng.choice([2, 3, 3])
        case.update(call=rng.choice(["host", "device"]), ids=_log_int(rng, 60, 20_000), k=rng.randint(1, 29), fes=fes,
                    clusters=rng.randint(0, fes))
    elif data == "matched":
        workers = _log_int(rng, 2_000, 1_500_000 if cg else 80_000)
        periods = rng.randint(6, 30)
        case.update(call=rng.choice(["device", "within"]) if precision == "fp64" else "device", workers=workers,
                    firms=max(20, workers // rng.randint(6, 25)), periods=periods, move=rng.choice([0.08, 0.1, 0.2]),
                    keep=rng.choice([1.0, round(rng.uniform(0.75, 1.0), 3)]), shuffle=rng.random() < 0.3,
                    k=rng.randint(1, 12))
        if case["call"] == "device":
            case.update(clusters=rng.randint(0, 3), singletons=rng.random() < 0.25)
    elif data == "levels":
        n = _log_int(rng, 20_000, 13_000_000)
        case.update(call="device", n=n, g0=_log_int(rng, 200, max(400, n // 5)), g1=rng.randint(2, 90),
                    g2=rng.randint(2, 60), k=rng.randint(1, 6), clusters=rng.randint(0, 3))
    elif data == "iv":
        n = _log_int(rng, 30_000, 1_000_000)
        case.update(call="formula", n=n, g0=max(50, n // 20), g1=max(20, n // 200), g2=rng.randint(4, 40),
                    precision="mixed", cg=True, tol=1e-8)
    else:
        lo = _log_int(rng, 2_000, 20_000)
        case.update(call="batch", specs=rng.randint(5, 60), lo=lo, hi=lo * rng.randint(2, 10), precision="mixed",
                    cg=True, tol=1e-8)
    return case


# ------------------------------------------------------------------- panels


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1009 + salt)
    return g


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _wages(case, g):
    """Persons with 1-15 consecutive years of 15, Zipf(1.1) occupations; the
    first five regressors are hours, experience, union, tenure and weeks
    unemployed, the others N(0, 1)."""
    n_ids, n_years, n_occ, k = case["ids"], 15, 13, case["k"]
    length = torch.randint(1, n_years + 1, (n_ids,), generator=g, device="cuda")
    start = (_uniform(g, n_ids) * (n_years - length + 1)).long()
    person = torch.repeat_interleave(torch.arange(n_ids, device="cuda"), length)
    first = torch.cumsum(length, 0) - length
    year = start[person] + torch.arange(person.numel(), device="cuda") - first[person]
    n = person.numel()
    share = torch.arange(1, n_occ + 1, device="cuda", dtype=torch.float64) ** -1.1
    occ = torch.searchsorted(torch.cumsum(share / share.sum(), 0), _uniform(g, n)).clamp(max=n_occ - 1)
    W = _normal(g, k, n)
    known = [(37.0 + 10.0 * W[0]).clamp(1.0, 80.0)]
    known.append(-3.0 * torch.log(_uniform(g, n) * _uniform(g, n) + 1e-300))
    known.append((_uniform(g, n) < 0.25).double())
    known.append(-5.0 * torch.log(_uniform(g, n) + 1e-300))
    known.append(torch.poisson(torch.full((n,), 2.0, device="cuda", dtype=torch.float64), generator=g))
    for j, col in enumerate(known[:k]):
        W[j] = col
    ids = [person, occ, year][:case["fes"]]
    sizes = [n_ids, n_occ, n_years][:case["fes"]]
    y = 0.3 * _normal(g, n) + torch.linspace(-0.05, 0.05, k, device="cuda", dtype=torch.float64) @ W
    for i, size in zip(ids, sizes):
        y += 0.3 * _normal(g, size)[i]
    return y, W, [(i + 1).int() for i in ids]


def _matched(case, g):
    """Workers observed over all periods (a share `keep` of the rows), moving
    to a firm drawn by size with probability `move` each period; regressors
    correlated 0.3 with the worker effect."""
    nw, nf, np_, k = case["workers"], case["firms"], case["periods"], case["k"]
    weight = torch.cumsum((1.0 - _uniform(g, nf)) ** (-1.0 / 1.5), 0)

    def firms(m):
        at = torch.searchsorted(weight, _uniform(g, m) * weight[-1], right=True)
        return at.clamp(max=nf - 1).int()

    firm = torch.empty(nw, np_, device="cuda", dtype=torch.int32)
    firm[:, 0] = firms(nw)
    for t in range(1, np_):
        moves = _uniform(g, nw) < case["move"]
        firm[:, t] = torch.where(moves, firms(nw), firm[:, t - 1])
    n = nw * np_
    worker = torch.arange(nw, device="cuda", dtype=torch.int32).repeat_interleave(np_)
    period = torch.arange(np_, device="cuda", dtype=torch.int32).repeat(nw)
    firm = firm.reshape(-1)
    rows = None
    if case["keep"] < 1.0:
        rows = torch.randperm(n, generator=g, device="cuda")[:int(n * case["keep"])].sort().values
    if case["shuffle"]:
        order = torch.randperm(n if rows is None else rows.numel(), generator=g, device="cuda")
        rows = order if rows is None else rows[order]
    if rows is not None:
        worker, firm, period = worker[rows], firm[rows], period[rows]
        n = rows.numel()
    effect = _normal(g, nw)[worker]
    y = 0.5 * effect + (0.3 * _normal(g, nf))[firm] + (0.1 * _normal(g, np_))[period]
    W = torch.empty(k, n, device="cuda", dtype=torch.float64)
    beta = torch.linspace(-0.5, 0.5, k).tolist()
    for j in range(k):
        W[j] = 0.3 * effect + math.sqrt(1.0 - 0.09) * _normal(g, n)
        y += beta[j] * W[j]
    y += 0.5 * _normal(g, n)
    return y, W, [worker + 1, firm + 1, period + 1]


def _levels(case, g):
    n, k = case["n"], case["k"]
    sizes = [case["g0"], case["g1"], case["g2"]]
    ids = [torch.randint(0, s, (n,), generator=g, device="cuda", dtype=torch.int32) for s in sizes]
    W = _normal(g, k, n)
    y = _normal(g, n) + torch.linspace(-0.5, 0.5, k, device="cuda", dtype=torch.float64) @ W
    for i, s in zip(ids, sizes):
        effect = 0.3 * _normal(g, s)
        y += effect[i]
        W[0] += effect[i]
    return y, W, [i + 1 for i in ids]


PANELS = {"wages": _wages, "matched": _matched, "levels": _levels}


def _iv(case, g):
    """The raw columns of IV_FORMULA: structural and first-stage errors are
    correlated 0.4, the continuous instrument 0.5 with its regressor."""
    n = case["n"]
    sizes = [case["g0"], case["g1"], case["g2"]]
    fe = [torch.randint(0, s, (n,), generator=g, device="cuda", dtype=torch.int32) for s in sizes]
    effect = [0.3 * _normal(g, s) for s in sizes]
    x = _normal(g, n, 6)

    def cat(levels):
        return torch.randint(1, levels + 1, (n,), generator=g, device="cuda")

    zc, cat_a, cat_b, z1, u = cat(20), cat(20), cat(4), _normal(g, n), _normal(g, n)
    v1, v2 = (0.4 * u + math.sqrt(1 - 0.16) * _normal(g, n) for _ in range(2))
    zc_effect = 0.5 * _normal(g, 21)
    x_end = 0.5 * z1 + 0.3 * zc_effect[zc] + 0.3 * x[:, 0] + effect[0][fe[0]] + v1
    latent = 0.8 * z1 - 0.4 * zc_effect[zc] + v2
    cat_end = 1 + (latent > -0.8).long() + (latent > 0.0).long() + (latent > 0.8).long()
    value = torch.tensor([0.0, 0.25, -0.1, 0.4, 0.6], device="cuda", dtype=torch.float64)
    y = (0.7 * x_end + value[cat_end] + x @ torch.linspace(-0.3, 0.3, 6, device="cuda", dtype=torch.float64)
         + 0.15 * x[:, 0] * x[:, 1] + 0.0025 * cat_a + 0.1 * (cat_b == 3) + u)
    for e, i in zip(effect, fe):
        y += e[i]
    raw = dict(y=y, x_end=x_end, cat_end=cat_end.double(), cat_a=cat_a.double(), cat_b=cat_b.double(), z1=z1,
               zc=zc.double(), **{f"x{j + 1}": x[:, j] for j in range(6)})
    return raw, [i + 1 for i in fe]


IV_X = ["x_end", "cat_end", "x1", "x2", "x3", "x4", "x5", "x6", "cat_a", "cat_b"]
IV_Z = ["z1", "zc"]


def _batch(case, seed):
    """Specifications of log-uniform size: 1-3 dimensions of about rows^0.7
    levels, 2-24 regressors, a quarter of them 2SLS, 1-3-way clusters. The
    shapes go by the case, the values by the seed."""
    r = np.random.RandomState(case["specs"] * 7919 + case["lo"])
    specs = []
    for s in range(case["specs"]):
        n = int(math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]))))
        sizes = [max(2, int(c * n ** 0.7)) for c in r.uniform(0.2, 1.0, r.randint(1, 4))]
        k = int(r.randint(2, 25))
        iv = r.rand() < 0.25
        endog = min(int(r.randint(1, 3)), k - 1) if iv else 0
        l = endog + int(r.randint(0, 3)) if iv else 0
        clusters = sorted(int(d) + 1 for d in r.permutation(len(sizes))[:r.randint(1, len(sizes) + 1)])
        g = _gen(seed, s + 1)
        ids = [torch.randint(0, m, (n,), generator=g, device="cuda", dtype=torch.int32) for m in sizes]
        W, Z, u = _normal(g, k, n), _normal(g, l, n), _normal(g, n)
        for j in range(endog):
            W[j] += 0.4 * u + torch.linspace(0.4, 0.8, l, device="cuda", dtype=torch.float64) @ Z
        y = u + torch.linspace(-1.0, 1.0, k, device="cuda", dtype=torch.float64) @ W
        for i, m in zip(ids, sizes):
            y += (0.3 * _normal(g, m))[i]
        specs.append(dict(y=y, W=W, Z=Z, ids=[i + 1 for i in ids], clusters=clusters, endog=list(range(1, endog + 1))))
    return specs


# -------------------------------------------------------------------- calls


def _config(case, n_fe):
    return fe_runtime_config(fe_tolerance=case["tol"], fe_max_iterations=20_000, precision=case["precision"],
                             demean_cg=case["cg"], cluster_fe_dims=list(range(1, 1 + case.get("clusters", 0))),
                             drop_singletons=bool(case.get("singletons", False)))


def _host(y, W, ids, Z=None):
    return fe_host_arrays(y=y.cpu().numpy(), W=W.cpu().numpy().T,
                          Z=Z.cpu().numpy().T if Z is not None else np.zeros((y.numel(), 0), order="F"),
                          fe_ids=np.asfortranarray(torch.stack(ids, 1).cpu().numpy().T))


def prepare(case, seed):
    call = case["call"]
    if call == "batch":
        specs = _batch(case, seed)
        rows = [fe_batch_spec(n=s["y"].numel(), k=s["W"].shape[0], l=s["Z"].shape[0], d_y=s["y"].data_ptr(),
                              d_W=s["W"].data_ptr(), d_Z=s["Z"].data_ptr() if s["Z"].shape[0] else None,
                              d_fe_ids=[i.data_ptr() for i in s["ids"]], cluster_fe_dims=s["clusters"],
                              iv_regressors=s["endog"]) for s in specs]
        return dict(call=call, cfg=_config(case, 0), specs=rows, keep=specs)
    if call == "formula":
        raw, ids = _iv(case, _gen(seed))
        host = _host(raw["y"], torch.stack([raw[c] for c in IV_X]), ids, torch.stack([raw[c] for c in IV_Z]))
        header = fe_dataset_header(n_obs=case["n"], n_regressors=len(IV_X), n_instruments=len(IV_Z), n_fe=3,
                                   depvar_name="y", regressor_names=IV_X, instrument_names=IV_Z,
                                   fe_names=["f1", "f2", "f3"])
        return dict(call=call, cfg=_config(case, 3), header=header, raw=RawDevice(header, host))
    y, W, ids = PANELS[case["data"]](case, _gen(seed))
    state = dict(call=call, cfg=_config(case, len(ids)), n=y.numel(), k=W.shape[0])
    if call == "host":
        return dict(state, host=_host(y, W, ids))
    state.update(y=y, W=W, ids=ids)
    if call == "within":
        state.update(out_y=torch.empty_like(y), out_W=torch.empty_like(W))
    return state


def _outputs(res):
    return dict(beta=res.beta, se=res.se, rss=res.rss, tss_within=res.tss_within, r2=res.r2, r2_within=res.r2_within,
                dof_resid=int(res.dof_resid), rank=int(res.rank), n_obs=int(res.n_obs_used),
                converged=bool(res.converged))


def run(state):
    call, cfg = state["call"], state["cfg"]
    if call == "host":
        return _outputs(fe_gpu_estimate(cfg, None, state["host"]))
    if call == "formula":
        fit, bound = expand_formula(IV_FORMULA, state["raw"], cfg)
        return _outputs(fit_formula(fit, bound, state["header"]))
    if call == "batch":
        res = fe_gpu_estimate_batch(cfg, state["specs"])
        return dict(beta=np.concatenate([r.beta for r in res]), se=np.concatenate([r.se for r in res]),
                    rss=np.array([r.rss for r in res]), dof_resid=np.array([r.dof_resid for r in res]),
                    converged=np.array([bool(r.converged) for r in res]))
    n, k, ids = state["n"], state["k"], [i.data_ptr() for i in state["ids"]]
    if call == "within":
        # the caller keeps its raw columns and has a copy demeaned in place
        state["out_y"].copy_(state["y"])
        state["out_W"].copy_(state["W"])
        torch.cuda.current_stream().synchronize()
        converged, _, _ = fe_gpu_within_transform_device(cfg, n, k, 0, state["out_y"].data_ptr(),
                                                         state["out_W"].data_ptr(), None, ids)
        return dict(y=state["out_y"], W=state["out_W"], converged=converged)
    return _outputs(fe_gpu_estimate_device(cfg, n, k, 0, state["y"].data_ptr(), state["W"].data_ptr(), None, ids))


def _rows(case):
    if case["data"] == "wages":
        return 8 * case["ids"]
    if case["data"] == "matched":
        return int(case["workers"] * case["periods"] * case["keep"])
    return case["n"]


def work(case):
    """Bytes: the inputs once (columns of 8 bytes, ids of 4) and the outputs
    once. Operations: the Gram matrix of the columns."""
    if case["call"] == "batch":
        rows = case["specs"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return {"bytes": rows * (8 * 15 + 8), "flops": rows * 15 * 16}
    n = _rows(case)
    if case["call"] == "formula":
        c = 1 + IV_K + IV_L
        return {"bytes": n * (8.0 * (1 + len(IV_X) + len(IV_Z)) + 12), "flops": float(n) * c * (c + 1)}
    c, n_fe = 1 + case["k"], case.get("fes", 3)
    if case["call"] == "within":
        return {"bytes": n * (16.0 * c + 4 * n_fe), "flops": 2.0 * n * c * n_fe}
    return {"bytes": n * (8.0 * c + 4 * n_fe), "flops": float(n) * c * (c + 1)}


# ------------------------------------------------------------ in 64 bits


def _group_sums(X, i, size):
    return torch.zeros(size, X.shape[1], device=X.device, dtype=X.dtype).index_add_(0, i, X)


def _demean(X, ids, sizes):
    """X (n x C) less its projection on the dimensions' dummies: conjugate
    gradients on the normal equations, restarted from the true residual."""
    counts = [torch.bincount(i, minlength=s).clamp(min=1).double()[:, None] for i, s in zip(ids, sizes)]
    floor = 1e-14 * X.abs().amax(0)  # what FP64 group means of such rows resolve

    def spread(tables):
        out = tables[0][ids[0]]
        for t, i in zip(tables[1:], ids[1:]):
            out += t[i]
        return out

    def largest(tables):
        return torch.stack([t.abs().amax(0) for t in tables]).amax(0)

    for _ in range(2):
        r = [_group_sums(X, i, s) for i, s in zip(ids, sizes)]
        x = [torch.zeros_like(v) for v in r]
        z = [v / c for v, c in zip(r, counts)]
        p = [v.clone() for v in z]
        rz = sum((a * b).sum(0) for a, b in zip(r, z))
        worst = largest(z)
        goal, best = torch.maximum(1e-9 * worst, floor), worst
        for _ in range(3000):
            open_ = (worst > goal) & (worst < 1e3 * best)  # a column that is done stays as it is
            if not bool(open_.any()):
                break
            row = spread(p)
            q = [_group_sums(row, i, s) for i, s in zip(ids, sizes)]
            pq = sum((a * b).sum(0) for a, b in zip(p, q))
            a = torch.where(open_ & (pq > 0), rz / pq, torch.zeros_like(pq))
            for d in range(len(ids)):
                x[d] += a * p[d]
                r[d] -= a * q[d]
                z[d] = r[d] / counts[d]
            worst = largest(z)
            best = torch.minimum(best, worst)
            new = sum((u * v).sum(0) for u, v in zip(r, z))
            b = torch.where(open_ & (rz > 0), new / rz, torch.zeros_like(rz))
            rz = new
            p = [v + b * w for v, w in zip(z, p)]
        X = X - spread(x)
    return X


def _kept(ids):
    """Rows left after the iterated removal of groups of one row."""
    keep = torch.ones(ids[0].numel(), dtype=torch.bool, device="cuda")
    while True:
        bad = torch.zeros_like(keep)
        for i in ids:
            count = torch.bincount(i[keep], minlength=int(i.max()) + 1)
            bad |= keep & (count[i] == 1)
        if not bool(bad.any()):
            return keep
        keep &= ~bad


def _fit(y, W, Z, ids, clusters, endog=(), singletons=False):
    """OLS or 2SLS with FEs in 64 bits, with the conventions of the GPU
    estimator. y (n), W (k x n), Z (l x n), ids 1-based."""
    ids = [i.long() - 1 for i in ids]
    sizes = [int(i.max()) + 1 for i in ids]
    if singletons:
        keep = _kept(ids)
        y, W, Z, ids = y[keep], W[:, keep], Z[:, keep] if Z is not None else None, [i[keep] for i in ids]
    n, k = y.numel(), W.shape[0]
    cols = [y[None], W] + ([Z] if Z is not None and Z.shape[0] else [])
    tss = float((y - y.mean()).square().sum())
    X = _demean(torch.cat(cols).T.contiguous(), ids, sizes)
    yt, Wt, Zt = X[:, 0], X[:, 1:1 + k], X[:, 1 + k:]
    if len(endog):
        exog = [j for j in range(k) if j + 1 not in endog]
        A = torch.cat([Wt[:, exog], Zt], 1)
        Pi = torch.linalg.solve(A.T @ A, A.T @ Wt)
        Q, b = Pi.T @ (A.T @ A) @ Pi, Pi.T @ (A.T @ yt)
    else:
        A, Pi = Wt, None
        Q, b = Wt.T @ Wt, Wt.T @ yt
    Qi = torch.linalg.inv(Q)
    beta = Qi @ b
    e = yt - Wt @ beta
    rss = float(e.square().sum())
    dof = max(1, n - (k + sum(s - 1 for s in sizes) + 1))
    if clusters:
        S = A * e[:, None]
        cov = torch.zeros_like(Q)
        for mask in range(1, 1 << len(clusters)):
            dims = [clusters[j] - 1 for j in range(len(clusters)) if mask >> j & 1]
            key = torch.zeros_like(ids[0])
            for d in dims:
                key = key * sizes[d] + ids[d]
            level, where = torch.unique(key, return_inverse=True)
            s = _group_sums(S, where, level.numel())
            meat = s.T @ s
            if Pi is not None:
                meat = Pi.T @ meat @ Pi
            cov += (1.0 if len(dims) % 2 else -1.0) * (Qi @ meat @ Qi)
        least = min(sizes[d - 1] for d in clusters)
        nested = 1 if any(sizes[d - 1] > 1 for d in clusters) else 0
        cov *= (n - 1) / max(1, n - k - nested) * (least / (least - 1) if least > 1 else 1.0)
        value, vector = torch.linalg.eigh(0.5 * (cov + cov.T))
        se = ((vector * vector) @ value.clamp(min=0.0)).sqrt()
        dof = max(1, least - 1)
    else:
        se = (rss / dof * Qi.diagonal()).clamp(min=0.0).sqrt()
    within = float(yt.square().sum())
    return dict(beta=beta.cpu().numpy(), se=se.cpu().numpy(), rss=rss, tss_within=within, r2=1 - rss / tss,
                r2_within=1 - rss / within, dof_resid=dof, rank=k, n_obs=n, converged=True)


def _dummies(code, levels):
    return [(code == v).double() for v in levels]


def exact(case, seed):
    if case["call"] == "batch":
        fits = [_fit(s["y"], s["W"], s["Z"], s["ids"], s["clusters"], s["endog"]) for s in _batch(case, seed)]
        return dict(beta=np.concatenate([f["beta"] for f in fits]), se=np.concatenate([f["se"] for f in fits]),
                    rss=np.array([f["rss"] for f in fits]), dof_resid=np.array([f["dof_resid"] for f in fits]),
                    converged=np.array([True] * len(fits)))
    if case["call"] == "formula":
        raw, ids = _iv(case, _gen(seed))
        a, b = _dummies(raw["cat_a"], range(2, 21)), _dummies(raw["cat_b"], range(2, 5))
        W = [raw["x_end"]] + _dummies(raw["cat_end"], [1, 3, 4]) + [raw[f"x{j}"] for j in range(1, 7)] + a + b
        W += [raw["x1"] * raw["x2"]] + [u * v for u in a for v in b]
        Z = [raw["z1"]] + _dummies(raw["zc"], range(2, 21))
        return _fit(raw["y"], torch.stack(W), torch.stack(Z), ids, [1, 2], endog=[1, 2, 3, 4])
    if _rows(case) > 40_000_000:
        return None  # minutes in 64 bits
    y, W, ids = PANELS[case["data"]](case, _gen(seed))
    if case["call"] == "within":
        i = [v.long() - 1 for v in ids]
        X = _demean(torch.cat([y[None], W]).T.contiguous(), i, [int(v.max()) + 1 for v in i])
        return dict(y=X[:, 0].contiguous(), W=X[:, 1:].T.contiguous(), converged=True)
    return _fit(y, W, None, ids, list(range(1, 1 + case["clusters"])), singletons=case.get("singletons", False))
