"""The calls that the performance of this framework is measured on.

One pass is one call of a public entry point of `fereg_b200` on data that the caller holds: an OLS,
IV, logit, Poisson or wild-bootstrap call on a prepared session, a residualization through the
Absorber, a whole request through the serving engine, and the preparation of a raw sample. The
panels are the ones of bench.py (individuals x years with cyclic or random firms, the connected
ring of firms, the gravity panel, the requests of the serving stream) at their own and at smaller
sizes; draw() spreads over the same ranges.

`ols_device` and its like residualize the caller's device block in place, so a pass starts with
the copy of the raw block that such a program makes, on the handle's own stream.
"""

import math

import numpy as np
import torch

import fereg_b200 as fb

TOL = 1e-8


# ------------------------------------------------------------------------------------------------
# the cases


def listed():
    return [
        # A small two-way panel (1e4 individuals x 10 years, one regressor): the interactive call,
        # where launches, host round trips and latencies are the cost.
        dict(name="ols_small", kind="ols", n_ind=10_000, years=10, firms=0, graph="none", occ=0, k=1, vce="unadjusted",
             weights="none", shuffled=False, ragged=False),
        # The headline: 1e7 rows, three FE, ten regressors, one row per cell, iid SEs.
        dict(name="ols_panel", kind="ols", n_ind=1_000_000, years=10, firms=100_000, graph="cyclic", occ=0, k=10,
             vce="unadjusted", weights="none", shuffled=False, ragged=False),
        # The same size on one connected ring of firms (the difficult graph), robust SEs: the PCG
        # iterations are the cost.
        dict(name="ols_ring", kind="ols", n_ind=1_000_000, years=10, firms=43_478, graph="cyclic", occ=0, k=10,
             vce="robust", weights="none", shuffled=False, ragged=False),
        # A weighted, unbalanced panel in no particular order with SEs clustered by firm.
        dict(name="ols_weighted", kind="ols", n_ind=140_001, years=9, firms=23_017, graph="random", occ=0, k=6,
             vce="cluster", weights="aweight", shuffled=True, ragged=True),
        # 2SLS with four FE and robust SEs (one endogenous regressor, two instruments).
        dict(name="iv_robust", kind="iv", n_ind=81_000, years=10, firms=16_200, graph="random", occ=100, k=5,
             vce="robust", weights="none", shuffled=False, ragged=False),
        # Logit on firms, years and occupations with clustered SEs, at an ordinary size.
        dict(name="logit_cluster", kind="logit", n_ind=20_011, years=10, firms=4_003, graph="random", occ=100, k=4,
             vce="cluster", weights="none", shuffled=False, ragged=False),
        # Poisson PML on the gravity panel (200 countries, 50 years, 5 rows per pair and year).
        dict(name="poisson_gravity", kind="poisson", countries=200, years=50, sectors=5, vce="robust"),
        # WCR11 wild cluster bootstrap of one coefficient, 999 draws, clusters = firms.
        dict(name="wildboot", kind="wildboot", n_ind=100_000, years=10, firms=20_000, graph="random", occ=0, k=1,
             reps=999, tile=512, vce="cluster", weights="none", shuffled=False, ragged=False),
        # Firm-specific slopes: absorb(ind firm##c.x) through the Absorber, device block.
        dict(name="demean_slopes", kind="slopes", n_ind=20_000, years=10, firms=2_000, graph="random", occ=0, k=2,
             vce="none", weights="none", shuffled=False, ragged=False),
        # The drop-in Absorber on a host block with the FE coefficients handed back.
        dict(name="demean_host", kind="demean", n_ind=50_003, years=8, firms=9_001, graph="random", occ=0, k=2,
             vce="none", weights="pweight", shuffled=False, ragged=True),
        # A whole request from the caller's host columns through the serving engine: the cell
        # structure, the copies and the estimate.
        dict(name="serve_request", kind="serve", n_ind=60_000, years=10, firms=12_000, graph="random", occ=0, k=6,
             vce="cluster", weights="none", shuffled=False, ragged=False),
        # The sample preparation: ids to codes (sparse ids, dense ids, an interaction), singletons.
        dict(name="prepare_sample", kind="prepare", n_ind=100_000, years=10, firms=10_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ols", "ols", "ols", "iv", "logit", "poisson", "wildboot", "slopes", "demean", "serve", "prepare"])
    if kind == "poisson":
        return dict(kind=kind, countries=_log(rng, 20, 150), years=rng.randint(5, 40), sectors=rng.randint(1, 5),
                    vce="robust")
    years = rng.randint(5, 12)
    top = {"ols": 700_000, "iv": 300_000, "logit": 100_000, "wildboot": 60_000, "slopes": 20_000, "demean": 100_000,
           "serve": 150_000, "prepare": 150_000}[kind]
    n_ind = _log(rng, 1_000, top)
    firms = max(20, n_ind * years // rng.randint(40, 60))
    if kind == "prepare":
        firms = max(10, n_ind * years // 100)
        return dict(kind=kind, n_ind=n_ind, years=years, firms=firms)
    graph = rng.choice(["none", "cyclic", "random", "random"]) if kind in ("ols", "serve") else "random"
    vce = {"ols": rng.choice(["unadjusted", "robust", "cluster"]), "iv": rng.choice(["unadjusted", "robust", "cluster"]),
           "logit": rng.choice(["oim", "robust", "cluster"]), "serve": rng.choice(["unadjusted", "robust", "cluster"]),
           "wildboot": "cluster"}.get(kind, "none")
    if graph == "cyclic":
        # firm = row mod firms; whole runs of `years` firms keep each component small, as in the 1e7 panel
        firms = max(2, firms // years) * years
    case = dict(kind=kind, n_ind=n_ind, years=years, firms=0 if graph == "none" else firms, graph=graph,
                occ=rng.choice([0, 0, 100]) if kind in ("ols", "iv", "serve") and graph == "random" else
                (100 if kind == "logit" else 0),
                k=rng.randint(1, 4) if kind in ("slopes", "demean", "wildboot") else rng.randint(2, 12), vce=vce,
                weights=rng.choice(["none", "aweight", "pweight"]) if kind in ("ols", "demean") and vce != "unadjusted"
                else "none",
                shuffled=kind in ("ols", "iv", "serve") and graph == "random" and rng.random() < 0.5,
                ragged=kind in ("ols", "demean", "iv") and graph == "random" and rng.random() < 0.5)
    if kind == "wildboot":
        case["reps"], case["tile"] = rng.choice([99, 199, 399, 999]), rng.choice([128, 256, 512])
    return case


# ------------------------------------------------------------------------------------------------
# the data (everything on the GPU, from the seed alone)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFF)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _dense(c):
    """Codes renumbered over the levels present, and the level count."""
    u, inv = torch.unique(c, return_inverse=True)
    return inv, int(u.numel())


def _panel(case, seed):
    """Kept-order panel: term codes (int64 tensors) with their levels, cluster index among the
    terms, weights, and the columns [y, x1..xk] (for IV then endogenous and instruments)."""
    g = _gen(seed)
    n_ind, years, kind, k = case["n_ind"], case["years"], case["kind"], case["k"]
    n = n_ind * years
    i = torch.arange(n, device="cuda")
    ind, year = i // years, i % years
    firm = None
    if case["graph"] == "cyclic":
        firm = i % case["firms"]
    elif case["graph"] == "random":
        firm = torch.randint(0, case["firms"], (n,), generator=g, device="cuda")
    occ = torch.randint(0, case["occ"], (n,), generator=g, device="cuda") if case["occ"] else None
    sel = None
    if case["ragged"]:  # every individual's first year and 83% of the other rows
        rest = torch.nonzero(year > 0).flatten()
        pick = torch.randperm(rest.numel(), generator=g, device="cuda")[:int(rest.numel() * 0.83)]
        sel = torch.cat([torch.nonzero(year == 0).flatten(), rest[pick]]).sort().values
    if case["shuffled"]:
        p = torch.randperm(n if sel is None else sel.numel(), generator=g, device="cuda")
        sel = p if sel is None else sel[p]
    if sel is not None:
        ind, year = ind[sel], year[sel]
        firm = None if firm is None else firm[sel]
        occ = None if occ is None else occ[sel]
        n = int(sel.numel())
    terms = [] if kind == "logit" else [_dense(ind)]
    if firm is not None:
        terms.append(_dense(firm))
    if kind not in ("slopes",):
        terms.append(_dense(year))
    if occ is not None:
        terms.append(_dense(occ))
    psi = _randn(g, terms[0 if kind == "logit" else 1][1]) if firm is not None else None
    fc = None if firm is None else terms[0 if kind == "logit" else 1][0]
    y = _randn(g, n) + 0.7 * _randn(g, years)[year]
    if kind != "logit":
        y += _randn(g, terms[0][1])[terms[0][0]]
    if psi is not None:
        y += (0.5 if kind == "logit" else 1.0) * psi[fc]
    extra = 3 if kind == "iv" else 0
    rows = torch.empty(n, 1 + k + extra, dtype=torch.float64, device="cuda")
    for j in range(k):
        x = _randn(g, n)
        if psi is not None:
            x = 0.3 * psi[fc] + math.sqrt(0.91) * x
        rows[:, 1 + j] = x
        y += x * (0.0 if kind == "wildboot" and j == 0 else (0.5 if kind == "logit" else 1.0) / (j + 1))
    if kind == "iv":
        z1, z2, u = _randn(g, n), _randn(g, n), _randn(g, n)
        endog = 0.8 * z1 - 0.5 * z2 + u
        y += 0.5 * endog + 0.7 * u
        rows[:, 1 + k], rows[:, 2 + k], rows[:, 3 + k] = endog, z1, z2
    if kind == "logit":
        y = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) < torch.sigmoid(0.5 * y)).double()
    rows[:, 0] = y
    w = None
    if case["weights"] != "none":
        w = 0.5 + 1.5 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    xs = _randn(g, n) if kind == "slopes" else None
    cl = 0 if firm is None or kind == "logit" else 1
    return dict(n=n, terms=terms, cl=cl, w=w, rows=rows, xs=xs)


def _gravity(case, seed):
    g = _gen(seed)
    C, T, S = case["countries"], case["years"], case["sectors"]
    a = torch.arange(C * C, device="cuda")
    a = a[(a // C) != (a % C)]
    P = int(a.numel())
    idx = torch.arange(P * T * S, device="cuda")
    pair, year = idx // (T * S), (idx // S) % T
    ey, iy = (a // C)[pair] * T + year, (a % C)[pair] * T + year
    n = int(idx.numel())
    ld = math.log(100.0) + (math.log(2e4) - math.log(100.0)) * torch.rand(P, generator=g, device="cuda", dtype=torch.float64)
    x1, x2 = _randn(g, n), _randn(g, n)
    lin = 0.5 * x1 - 0.2 * x2 - 0.2 * ld[pair] + 0.5 * (_randn(g, C * T)[ey] + _randn(g, C * T)[iy] + _randn(g, P)[pair])
    y = torch.poisson(torch.exp(lin - lin.mean()), generator=g)
    # every FE group needs a positive outcome (the `fe` separation rule)
    for codes, m in ((ey, C * T), (iy, C * T), (pair, P)):
        tot = torch.zeros(m, dtype=torch.float64, device="cuda").index_add_(0, codes, y)
        first = torch.full((m,), n, device="cuda").scatter_reduce_(0, codes, idx, "amin")
        y[first[tot == 0]] = 1.0
    rows = torch.stack([y, x1, x2], dim=1).contiguous()
    return dict(n=n, terms=[(ey, C * T), (iy, C * T), (pair, P)], cl=2, w=None, rows=rows, xs=None)


def _raw_ids(case, seed):
    """Raw factor columns: sparse ids (ten digits, in no order), dense firm ids, decades; one
    individual in twelve has a single row."""
    g = _gen(seed)
    n_ind, years = case["n_ind"], case["years"]
    ids = 10**9 + 9000 * torch.randperm(n_ind, generator=g, device="cuda")
    ids += torch.randint(0, 9000, (n_ind,), generator=g, device="cuda")
    n = n_ind * years
    i = torch.arange(n, device="cuda")
    firm = 1000 + torch.randint(0, case["firms"], (n,), generator=g, device="cuda")
    half = 1 + (2 * (i % years)) // years
    once = torch.zeros(n_ind, dtype=torch.bool, device="cuda")
    once[torch.randperm(n_ind, generator=g, device="cuda")[:n_ind // 12]] = True
    keep = ~once[i // years] | (i % years == 0)
    return [c[keep].double().cpu().numpy() for c in (ids[i // years], firm, half)]


def _u32(terms):
    return [c.to(torch.int32).cpu().numpy().view(np.uint32) for c, _ in terms], [m for _, m in terms]


def _data(case, seed):
    return _gravity(case, seed) if case["kind"] == "poisson" else _panel(case, seed)


# ------------------------------------------------------------------------------------------------
# what a program has in hand, and one pass


def prepare(case, seed):
    kind = case["kind"]
    if kind == "prepare":
        return dict(case=case, factors=_raw_ids(case, seed))
    d = _data(case, seed)
    codes, g = _u32(d["terms"])
    w = None if d["w"] is None else d["w"].cpu().numpy()
    st = dict(case=case)
    if kind == "serve":
        clustered = case["vce"] == "cluster"
        st.update(srv=fb.Server(workers=2), codes=codes, g=g, cols=[c.contiguous().cpu().numpy() for c in d["rows"].T],
                  clusters=[codes[d["cl"]]] if clustered else [], cl_g=[g[d["cl"]]] if clustered else [])
        return st
    if kind in ("slopes", "demean"):
        if kind == "slopes":
            h = fb.Absorber(codes, g, w, intercept=[True] * len(codes),
                            slopes=[[]] + [[d["xs"].cpu().numpy()]] + [[]] * (len(codes) - 2))
        else:
            h = fb.Absorber(codes, g, w)
    else:
        clustered = case["vce"] == "cluster"
        h = fb.Session(codes, g, [codes[d["cl"]]] if clustered else [], [g[d["cl"]]] if clustered else [], w=w,
                       weight_kind=None if w is None else case["weights"])
    order = torch.from_numpy(h.row_order().view(np.int32)).cuda().long()
    rows = d["rows"][order].contiguous()
    if kind == "demean":
        st.update(h=h, rows=rows.cpu().pin_memory())
    else:
        st.update(h=h, rows=rows, stream=torch.cuda.ExternalStream(h.stream()))
    if kind not in ("logit", "poisson"):  # these leave the caller's block as it is
        st["work"] = torch.empty_like(st["rows"])
        if kind == "demean":
            st["work"] = st["work"].pin_memory()
    return st


def _fresh(st):
    """The raw block again in the buffer that the call residualizes in place."""
    with torch.cuda.stream(st["stream"]):
        st["work"].copy_(st["rows"], non_blocking=True)
    return st["work"]


def _scalars(r, names):
    return {s: float(r["scalars"][s]) for s in names}


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "ols":
        z = _fresh(st)
        r = st["h"].ols_device(z.data_ptr(), case["k"], vce=case["vce"], tol=TOL)
        return dict(b=r["b"], V=r["V"], status=r["status"], rows=z, dof=r["dof_table"],
                    scalars=_scalars(r, ("N", "df_r", "df_a", "rss", "tss", "tss_within", "r2", "F")))
    if kind == "iv":
        z = _fresh(st)
        r = st["h"].iv(z.data_ptr(), case["k"], 1, 2, vce=case["vce"], tol=TOL, on_device=True)
        return dict(b=r["b"], V=r["V"], status=r["status"], rows=z, scalars=_scalars(r, ("N", "df_r", "df_a", "rss", "F")))
    if kind in ("logit", "poisson"):
        nx = st["rows"].shape[1] - 1
        r = st["h"].glm(st["rows"].data_ptr(), kind, vce=case["vce"], tol=TOL, on_device=True, nx=nx)
        return dict(b=r["b"], V=r["V"], status=r["status"], deviance=r["deviance"], ll=r["ll"], chi2=r["chi2"])
    if kind == "wildboot":
        z = _fresh(st)
        r = st["h"].wildboot(z.data_ptr(), coef=0, reps=case["reps"], seed=1, tile=case["tile"], tol=TOL,
                             on_device=True, nx=case["k"])
        return dict(stat=r["stat"], se=r["se"], point=r["point"], pvalue=r["pvalue"], t_boot=r["t_boot"], rows=z)
    if kind == "slopes":
        z = _fresh(st)
        st["h"].residualize_device(z.data_ptr(), z.shape[1], tol=TOL)
        return dict(rows=z)
    if kind == "demean":
        st["work"].copy_(st["rows"])
        r = st["h"].residualize(st["work"].numpy(), tol=TOL, want_coefs=True)
        return dict(rows=st["work"], coefs=r["coefs"])
    if kind == "serve":
        t = st["srv"].submit("ols", st["codes"], st["g"], st["cols"], case["k"], clusters=st["clusters"],
                             cl_g=st["cl_g"], vce=case["vce"], tol=TOL)
        r = st["srv"].wait(t)
        if r["rc"]:
            raise RuntimeError(r["msg"])
        return dict(b=r["b"], V=r["V"], N=float(r["N"]))
    r = fb.prepare(st["factors"], [[0], [1], [1, 2]])
    return dict(alive=r["alive"], dropped=r["num_singletons"], codes=[c.view(np.int32) for c, _ in r["terms"]],
                levels=[m for _, m in r["terms"]])


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without, and its results in plain 64-bit torch


def work(case):
    """Bytes: the columns, codes and weights read once, the outputs written once (the residualized
    block, where the call leaves one). Operations: the products of the columns with one another
    (once per IRLS step for a GLM, eight steps), the draws' sums for a bootstrap."""
    kind = case["kind"]
    if kind == "poisson":
        n = case["countries"] * (case["countries"] - 1) * case["years"] * case["sectors"]
        return dict(bytes=n * (3 * 8 + 3 * 4), flops=8 * n * 2 * 9)
    n = case["n_ind"] * case["years"]
    if kind == "prepare":
        n -= case["n_ind"] // 12 * (case["years"] - 1)
        return dict(bytes=n * (3 * 8 + 3 * 4 + 1), flops=0)
    if case["ragged"]:
        n = int(n * 0.85)  # about
    R = 1 + case["k"] + (3 if kind == "iv" else 0)
    nt = (0 if kind == "logit" else 1) + (case["graph"] != "none") + (kind != "slopes") + (case["occ"] > 0)
    extra = (case["weights"] != "none") * 8 + (kind == "slopes") * 8
    b = n * (R * 8 + nt * 4 + extra)
    if kind in ("ols", "iv", "wildboot", "slopes", "demean"):
        b += n * R * 8
    f = n * 2 * R * R
    if kind == "logit":
        f *= 8
    if kind == "wildboot":
        f += case["reps"] * n * 2 * (nt + 1)
    return dict(bytes=b, flops=f)


def _absorb(z, terms, w=None, limit=400):
    """Residuals of the columns of z on the terms' dummies (times the term's variable, where it has
    one), W-weighted: Jacobi-preconditioned CG on the normal equations, twice (the second time on
    the residuals of the first). None when it does not converge in `limit` iterations."""
    dt, R = z.dtype, z.shape[1]
    wt = None if w is None else w[:, None]
    off, m = [], 0
    for c, g, _ in terms:
        off.append(m)
        m += g

    def tr(v):  # D'W v
        v = v if wt is None else v * wt
        out = torch.zeros(m, v.shape[1], dtype=dt, device=z.device)
        for (c, g, x), o in zip(terms, off):
            out[o:o + g].index_add_(0, c, v if x is None else v * x[:, None])
        return out

    def fwd(t):  # D t
        v = None
        for (c, g, x), o in zip(terms, off):
            u = t[o:o + g][c]
            u = u if x is None else u * x[:, None]
            v = u if v is None else v.add_(u)
        return v

    diag = torch.zeros(m, dtype=dt, device=z.device)
    one = torch.ones(z.shape[0], dtype=dt, device=z.device) if w is None else w
    for (c, g, x), o in zip(terms, off):
        diag[o:o + g].index_add_(0, c, one if x is None else one * x * x)
    inv = torch.where(diag > 0, 1 / diag, torch.zeros_like(diag))[:, None]
    z = z.clone()
    for _ in range(2):
        r = tr(z)
        t = torch.zeros_like(r)
        s = inv * r
        p = s.clone()
        rho = (r * s).sum(0)
        ref = (z * z if wt is None else z * z * wt).sum(0)
        for it in range(limit):
            q = tr(fwd(p))
            a = rho / (p * q).sum(0).clamp_min(1e-300)
            t += a * p
            r -= a * q
            s = inv * r
            new = (r * s).sum(0)
            if bool((new <= 1e-28 * ref).all()):
                break
            p = s + (new / rho.clamp_min(1e-300)) * p
            rho = new
        else:
            return None
        z -= fwd(t)
    return z


def _terms(d):
    return [(c, g, None) for c, g in d["terms"]]


def _order(d):
    """Row order of the cell structure: by the eliminated term (on these panels the one with the
    most levels), then by the small terms (fewest levels first into a total of 4096) and the large
    ones, each in term order, then by observation."""
    t = d["terms"]
    e = max(range(len(t)), key=lambda q: t[q][1])
    others = [q for q in range(len(t)) if q != e]
    small, total = set(), 0
    for q in sorted(others, key=lambda q: t[q][1]):
        if total + t[q][1] > 4096:
            break
        total += t[q][1]
        small.add(q)
    keys = [e] + [q for q in others if q in small] + [q for q in others if q not in small]
    order = torch.arange(d["n"], device="cuda")
    for q in reversed(keys):
        order = order[torch.sort(t[q][0][order], stable=True).indices]
    return order


def exact(case, seed):
    kind = case["kind"]
    if kind in ("prepare", "wildboot"):
        return None
    if case.get("graph") == "cyclic" and math.gcd(case["firms"], case["years"]) < case["years"]:
        return None  # the connected ring: plain CG needs thousands of iterations
    d = _data(case, seed)
    z, w, n = d["rows"], d["w"], d["n"]
    if kind in ("logit", "poisson"):
        return _exact_glm(kind, z, _terms(d))
    terms = _terms(d)
    if kind == "slopes":
        terms.append((d["terms"][1][0], d["terms"][1][1], d["xs"]))
    wn = None if w is None else w * (n / w.sum())
    res = _absorb(z, terms, w, 4000 if kind == "slopes" else 400)
    if res is None:
        return None
    if kind == "slopes":
        return dict(rows=res)  # rows in the order of the individuals, as they are given
    if kind == "demean":
        return dict(rows=res[_order(d)], coefs=None)
    k = case["k"]
    y = res[:, 0]
    wr = res if wn is None else res * wn[:, None]
    wm = torch.ones(n, dtype=torch.float64, device="cuda") / n if w is None else w / w.sum()
    if kind == "iv":
        X = torch.cat([res[:, 1 + k:2 + k], res[:, 1:1 + k]], 1)
        Z = torch.cat([res[:, 2 + k:], res[:, 1:1 + k]], 1)
        P = torch.linalg.solve(Z.T @ Z, Z.T @ X)
        b = torch.linalg.solve(P.T @ (Z.T @ X), P.T @ (Z.T @ y))
        e = y - X @ b
        return dict(b=b, V=None, status=None, rows=res[_order(d)],
                    scalars=dict(N=None, df_r=None, df_a=None, rss=float((e * e).sum()), F=None))
    X, WX = res[:, 1:], wr[:, 1:]
    b = torch.linalg.solve(WX.T @ X, WX.T @ y)
    mean = wm @ z
    full = torch.cat([b, (mean[0] - mean[1:] @ b)[None]])
    if kind == "serve":
        return dict(b=full, V=None, N=None)
    e = y - X @ b
    ww = 1.0 if wn is None else wn
    rss, tw = float((ww * e * e).sum()), float((ww * y * y).sum())
    tss = float((ww * (z[:, 0] - mean[0]) ** 2).sum())
    return dict(b=full, V=None, status=None, rows=res[_order(d)], dof=None,
                scalars=dict(N=None, df_r=None, df_a=None, rss=rss, tss=tss, tss_within=tw, r2=1 - rss / tss, F=None))


def _exact_glm(kind, rows, terms):
    y, X = rows[:, 0], rows[:, 1:]
    pois = kind == "poisson"
    mu = 0.5 * (y + (y.mean() if pois else 0.5))
    eta = torch.log(mu) if pois else torch.log(mu / (1 - mu))
    old = None
    for _ in range(40):
        w = mu if pois else mu * (1 - mu)
        zv = eta + (y - mu) / w
        res = _absorb(torch.cat([zv[:, None], X], 1), terms, w)
        if res is None:
            return None
        WX = res[:, 1:] * w[:, None]
        b = torch.linalg.solve(WX.T @ res[:, 1:], WX.T @ res[:, 0])
        eta = zv - (res[:, 0] - res[:, 1:] @ b)
        mu = torch.exp(eta) if pois else torch.sigmoid(eta)
        if old is not None and float((b - old).abs().max()) < 1e-13:
            break
        old = b
    if pois:
        dev = 2 * ((mu - y) + torch.xlogy(y, y) - y * eta).sum()
        ll = (y * eta - mu - torch.lgamma(y + 1)).sum()
    else:
        dev = 2 * (torch.nn.functional.softplus(eta) - y * eta).sum()
        ll = -dev / 2
    return dict(b=b, V=None, status=None, deviance=float(dev), ll=float(ll), chi2=None)
