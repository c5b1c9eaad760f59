"""Timed cases of the maximum-likelihood path, through the package's Python entry points.

``listed()`` names the cases, ``draw`` gives more of the same ranges, ``prepare`` builds what a
program holds before the call (locations, observations, the device-resident problem), ``run`` is
one pass, ``work`` the operations a pass cannot do without and ``exact`` the same results from
plain torch in 64 bits.  The ranges are those of the tests and of ``bench.py``: N from a few
hundred to 102,400, tiles 64 to 1024, Matern smoothness 0.3 to 2 (half-integer and general).
"""
import math

import numpy as np
import torch

import exageostatcpp_b200 as egs

TILES = (64, 100, 128, 192, 256, 320, 512, 560, 768, 960, 1024)


def listed():
    return [
        # One likelihood of a small region: an optimiser calls it hundreds of times, launches and latency count.
        {"name": "eval_n400", "kind": "eval", "n": 400, "dts": 128, "s2": 1.0, "beta": 0.1, "nu": 0.5},
        # The reference's N = 1,600 fit configuration (40 x 40 grid, tile 320), one objective evaluation.
        {"name": "eval_n1600", "kind": "eval", "n": 1600, "dts": 320, "s2": 1.0, "beta": 0.1, "nu": 0.5},
        # A mid-size evaluation with a ragged last tile and a general (Bessel) smoothness.
        {"name": "eval_n10000", "kind": "eval", "n": 10000, "dts": 960, "s2": 1.0, "beta": 0.05, "nu": 0.8},
        # The plain FP64 configuration at N = 40,000, tile 960.
        {"name": "eval_n40000", "kind": "eval", "n": 40000, "dts": 960, "s2": 1.0, "beta": 0.05, "nu": 0.8},
        # A mixed-precision evaluation of a size the serving loop sees, odd N.
        {"name": "mixed_n20011", "kind": "mixed", "n": 20011, "dts": 1024, "band": 2, "s2": 1.0, "beta": 0.05,
         "nu": 0.8},
        # The mixed-precision configuration at N = 102,400, tile 1024, band of 2 tiles.
        {"name": "mixed_n102400", "kind": "mixed", "n": 102400, "dts": 1024, "band": 2, "s2": 1.0, "beta": 0.1,
         "nu": 0.5},
        # One optimiser step over many regional problems of uneven N, in three size classes.
        {"name": "batch_512", "kind": "batch", "problems": 512, "nmin": 256, "nmax": 4096, "classes": 3, "dts": 320},
        # The diagonal super-tile approximation (--computation=diag_approx --band=4).
        {"name": "band_n10000", "kind": "band", "n": 10000, "dts": 320, "band": 4, "s2": 1.0, "beta": 0.01,
         "nu": 0.5},
        # Synthetic observations Z = L e, the first call of a simulation study.
        {"name": "sample_n5000", "kind": "sample", "n": 5000, "dts": 512, "s2": 1.0, "beta": 0.04, "nu": 1.5},
        # Kriging of 1,000 held-out points with the MSPE, the one-shot call of the prediction module.
        {"name": "predict_n10000", "kind": "predict", "n": 10000, "miss": 1000, "dts": 960, "s2": 1.0,
         "beta": 0.05, "nu": 0.8},
        # MLOE / MMOM of an estimated theta over 100 targets.
        {"name": "mloe_n1600", "kind": "mloe", "n": 1600, "miss": 100, "dts": 320, "s2": 1.0, "beta": 0.1, "nu": 0.5},
        # Inverse Fisher information at the fitted theta.
        {"name": "fisher_n1600", "kind": "fisher", "n": 1600, "dts": 320, "s2": 1.0, "beta": 0.1, "nu": 0.8},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_theta(rng, n, most):
    """A theta whose covariance on n jittered grid points stays numerically positive definite: the
    estimate (1 + (pi beta / h)^2)^(nu + 1) of its condition number, h = 1 / sqrt(n), is at most `most`."""
    nu = rng.choice((0.5, 0.5, 1.5, 0.8, rng.uniform(0.3, 2.0)))
    limit = math.sqrt(most ** (1.0 / (nu + 1.0)) - 1.0) / (math.pi * math.sqrt(n))
    return {"s2": round(rng.uniform(0.5, 2.0), 4), "beta": round(min(rng.uniform(0.02, 0.12), limit), 5),
            "nu": round(nu, 4)}


def _draw_tile(rng, n, least=64):
    """A tile of the usual list that gives at most 64 tile rows."""
    return rng.choice([t for t in TILES if t >= least and -(-n // t) <= 64])


def draw(rng):
    kind = rng.choice(("eval", "eval", "eval", "mixed", "batch", "band", "sample", "predict", "mloe", "fisher"))
    if kind == "batch":
        nmin = _log_uniform(rng, 100, 1000)
        return {"kind": kind, "problems": _log_uniform(rng, 8, 512), "nmin": nmin,
                "nmax": _log_uniform(rng, nmin + 50, 4096), "classes": rng.choice((1, 2, 3)),
                "dts": rng.choice((128, 192, 256, 320))}
    lo, hi, most = {"eval": (100, 30000, 1e7), "mixed": (2000, 60000, 1e6), "band": (500, 12000, 1e4),
                    "sample": (200, 12000, 1e7), "predict": (200, 12000, 1e6), "mloe": (200, 2500, 1e5),
                    "fisher": (100, 2000, 1e5)}[kind]
    n = _log_uniform(rng, lo, hi)
    c = {"kind": kind, "n": n, "dts": _draw_tile(rng, n, 512 if kind == "mixed" else 64)}
    if kind == "band":
        c["dts"] = rng.choice([t for t in TILES if t % 64 == 0 and -(-n // t) <= 64])
        c["band"] = rng.choice((1, 2, 3, 4, 6))
    if kind == "mixed":
        c["band"] = rng.choice((1, 2, 3))
    if kind in ("predict", "mloe"):
        c["miss"] = _log_uniform(rng, 10, 1000 if kind == "predict" else 100)
    c.update(_draw_theta(rng, n, most))
    if kind == "band":  # the approximation is indefinite for smooth or long-range fields
        c.update(beta=round(min(0.02, 1.0 / math.sqrt(n)), 5), nu=rng.choice((0.5, round(rng.uniform(0.3, 0.7), 4))))
    return c


def _theta(case):
    return (case["s2"], case["beta"], case["nu"])


def _estimate(case):
    """The misspecified theta of an MLOE / MMOM case."""
    return (0.8 * case["s2"], 1.2 * case["beta"], 1.2 * case["nu"])


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _field(x, y, theta, seed):
    """A random field with the Matern covariance of theta at (x, y): 2,048 plane waves whose frequencies
    follow the covariance's spectral density (a bivariate t with 2 nu degrees of freedom)."""
    rng = np.random.default_rng(seed)
    waves = 2048
    s2, beta, nu = theta
    w = rng.standard_normal((2, waves)) / (beta * np.sqrt(rng.chisquare(2.0 * nu, waves)))
    phase = rng.uniform(0.0, 2.0 * math.pi, waves)
    dev = _device()
    w, phase = torch.from_numpy(w).to(dev), torch.from_numpy(phase).to(dev)
    px, py = torch.from_numpy(x).to(dev), torch.from_numpy(y).to(dev)
    out = torch.empty(len(x), dtype=torch.float64, device=dev)
    for a in range(0, len(x), 16384):
        b = slice(a, a + 16384)
        out[b] = torch.cos(px[b, None] * w[0] + py[b, None] * w[1] + phase).sum(1)
    return (out * math.sqrt(2.0 * s2 / waves)).cpu().numpy()


def _split(case, seed):
    """Observed and held-out points of a kriging case, in the generator's order."""
    n, m = case["n"], case["miss"]
    x, y = egs.generate_locations(n + m, seed % 4096)
    miss = np.zeros(n + m, dtype=bool)
    miss[np.random.default_rng(seed + 1).choice(n + m, m, replace=False)] = True
    return x, y, miss


def _batch_inputs(case, seed):
    """Sizes log-uniform over the range and theta of each problem (the draws of the batched
    configuration, held where every covariance is positive definite)."""
    rng = np.random.default_rng(99 + case["problems"])  # sizes and tiles are the schedule: the same for every seed
    sizes = np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["problems"])).astype(int)
    rng = np.random.default_rng(seed)
    s2 = rng.uniform(0.5, 2.0, len(sizes))
    nu = rng.uniform(0.3, 2.0, len(sizes))
    limit = np.sqrt(1e6 ** (1.0 / (nu + 1.0)) - 1.0) / (math.pi * np.sqrt(sizes))
    beta = np.minimum(rng.uniform(0.02, 0.3, len(sizes)), limit)
    xs, ys = zip(*(egs.generate_locations(int(n), (seed + i) % 4096) for i, n in enumerate(sizes)))
    theta = np.stack([s2, beta, nu], 1)
    z = np.concatenate([rng.standard_normal(n) * math.sqrt(s) for n, s in zip(sizes, s2)])
    return sizes, np.concatenate(xs), np.concatenate(ys), z, theta


def _batch_classes(sizes, case):
    """Class bounds at equal shares of the n^3 cost, tiles around the case's tile."""
    s = np.sort(sizes)
    share = np.cumsum(s.astype(np.float64) ** 3)
    upper = sorted({int(s[np.searchsorted(share, share[-1] * (c + 1) / case["classes"] * (1 - 1e-12))])
                    for c in range(case["classes"])} | {int(s[-1])})
    tiles = [max(64, case["dts"] - 64 * (len(upper) - 1 - c)) for c in range(len(upper))]
    return upper, tiles


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sizes, x, y, z, theta = _batch_inputs(case, seed)
        upper, tiles = _batch_classes(sizes, case)
        return {"kind": kind, "set": egs.BatchSet(sizes, x, y, z, upper, tiles), "theta": theta}
    theta = _theta(case)
    state = {"kind": kind, "theta": theta, "dts": case["dts"]}
    if kind in ("predict", "mloe"):
        x, y, miss = _split(case, seed)
        state.update(xo=x[~miss], yo=y[~miss], xm=x[miss], ym=y[miss])
        if kind == "predict":
            z = _field(x, y, theta, seed)
            state.update(zo=z[~miss], za=z[miss])
        else:
            state["estimate"] = _estimate(case)
        return state
    x, y = egs.generate_locations(case["n"], seed % 4096)
    state.update(x=x, y=y)
    if kind == "fisher":
        return state
    p = egs.Problem(case["n"], case["dts"])
    state["problem"] = p
    if kind == "mixed":
        p.set_precision(egs.EGS_PRECISION_MIXED, case["band"])
    if kind == "band":
        p.set_band(case["band"])
    p.set_locations(x, y)
    if kind == "sample":
        state["seed"] = seed % 4096
    else:
        p.set_observations(_field(x, y, theta, seed))
    return state


def run(state):
    kind = state["kind"]
    if kind in ("eval", "mixed", "band"):
        return state["problem"].mle_eval(state["theta"])
    if kind == "batch":
        return state["set"].eval(state["theta"])
    if kind == "sample":
        return state["problem"].generate_observations(state["theta"], state["seed"])
    if kind == "predict":
        return egs.predict_host(state["xo"], state["yo"], state["zo"], state["xm"], state["ym"], state["theta"],
                                state["dts"], state["za"])
    if kind == "mloe":
        return egs.mloe_mmom_host(state["xo"], state["yo"], state["xm"], state["ym"], state["theta"],
                                  state["estimate"], state["dts"])
    return egs.fisher_host(state["x"], state["y"], state["theta"], state["dts"])


def work(case):
    """Flops of the factorisations and solves; bytes of the inputs and outputs (the covariance is not an input)."""
    kind = case["kind"]
    if kind == "batch":
        sizes = np.exp(np.random.default_rng(99 + case["problems"]).uniform(
            math.log(case["nmin"]), math.log(case["nmax"]), case["problems"])).astype(int).astype(np.float64)
        return {"bytes": float((24.0 * sizes + 32.0).sum()), "flops": float((sizes ** 3 / 3 + 1.5 * sizes ** 2).sum())}
    n = float(case["n"])
    potrf = n ** 3 / 3 + n ** 2 / 2
    if kind == "band":  # band rows of tiles: width w = band * dts below the diagonal
        w = min(n, float(case["band"] * case["dts"]))
        return {"bytes": 24 * n, "flops": n * w * w + n * n}
    if kind == "sample":
        return {"bytes": 24 * n, "flops": potrf + n * n}
    if kind == "predict":
        m = float(case["miss"])
        return {"bytes": 24 * n + 32 * m, "flops": potrf + 2 * n * n + 2 * n * m}
    if kind == "mloe":  # two factors, three forward solves, one product L^T w and one backward solve per target
        m = float(case["miss"])
        return {"bytes": 16 * (n + m), "flops": 2 * potrf + 5 * m * n * n}
    if kind == "fisher":  # one factor, L^-1 C_j L^-T for three derivatives
        return {"bytes": 16 * n, "flops": potrf + 6 * n ** 3}
    return {"bytes": 24 * n, "flops": potrf + n * n}


# ---------------------------------------------------------------------------------------------
# The same results in plain torch, 64 bits.
# ---------------------------------------------------------------------------------------------

def _bessel_sums(x, nu, derivative=False):
    """K_nu(x) (and dK_nu/dnu) for a tensor x > 0: the trapezoid rule on the integral of
    exp(-x cosh t) cosh(nu t), which converges like exp(-pi^2 / h)."""
    h = 0.125
    end = math.acosh(110.0 / min(100.0, float(x.min()))) + 0.5
    k = torch.full_like(x, 0.5).mul_(torch.exp(-x))
    d = torch.zeros_like(x) if derivative else None
    for i in range(1, int(end / h) + 2):
        t = i * h
        e = torch.exp(x * -math.cosh(t))
        k.add_(e, alpha=math.cosh(nu * t))
        if derivative:
            d.add_(e, alpha=t * math.sinh(nu * t))
    k.mul_(h)
    return (k, d.mul_(h)) if derivative else k


def _scaled_distance(x1, y1, x2, y2, beta):
    return torch.sqrt((x1[:, None] - x2[None, :]) ** 2 + (y1[:, None] - y2[None, :]) ** 2) / beta


def _matern(x1, y1, x2, y2, theta):
    s2, beta, nu = theta
    out = torch.empty(len(x1), len(x2), dtype=torch.float64, device=x1.device)
    rows = max(1, (1 << 26) // max(1, len(x2)))
    for a in range(0, len(x1), rows):
        r = _scaled_distance(x1[a:a + rows], y1[a:a + rows], x2, y2, beta)
        zero = r == 0
        r[zero] = 1.0
        if nu == 0.5:
            c = s2 * torch.exp(-r)
        elif nu == 1.5:
            c = s2 * (1.0 + r) * torch.exp(-r)
        else:
            c = r ** nu * _bessel_sums(r, nu) * (s2 / (2.0 ** (nu - 1.0) * math.gamma(nu)))
        c[zero] = s2
        out[a:a + rows] = c
    return out


def _on_device(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).to(_device()) for a in arrays]


def _likelihood(L, z):
    w = torch.linalg.solve_triangular(L, z[:, None], upper=False)[:, 0]
    logdet, dot = float(2.0 * torch.log(torch.diagonal(L)).sum()), float(w @ w)
    return -0.5 * dot - 0.5 * logdet - 0.5 * len(z) * math.log(2.0 * math.pi), logdet, dot


def _band_factor(C, ts, band):
    """The reference's diagonal super-tile factorisation of the lower triangle of C."""
    A = torch.tril(C)
    n = len(A)
    nt = -(-n // ts)
    b = [slice(i * ts, min(n, (i + 1) * ts)) for i in range(nt)]
    for k in range(nt):
        d = A[b[k], b[k]]
        A[b[k], b[k]] = torch.linalg.cholesky(torch.tril(d) + torch.tril(d, -1).T)
        end = min(nt, k + band)
        for m in range(k + 1, end):
            A[b[m], b[k]] = torch.linalg.solve_triangular(A[b[k], b[k]], A[b[m], b[k]].T, upper=False).T
        for c in range(k + 1, end):
            for m in range(c, min(nt, c + band)):
                A[b[m], b[c]] -= A[b[m], b[k]] @ A[b[c], b[k]].T
    return torch.tril(A)


def _normal_sequence(seed, n):
    """LAPACK's DLARNV(3, (seed, seed, seed, 1)): a 48-bit multiplicative generator, 64 pairs at a time."""
    mask, mult = (1 << 48) - 1, (494 << 36) | (322 << 24) | (2508 << 12) | 2549
    s = (seed << 36) | (seed << 24) | (seed << 12) | 1
    u = np.empty(2 * n)
    for i in range(2 * n):
        s = (s * mult) & mask
        u[i] = s / float(1 << 48)
    return np.sqrt(-2.0 * np.log(u[0::2])) * np.cos(2.0 * math.pi * u[1::2])


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sizes, x, y, z, theta = _batch_inputs(case, seed)
        at = np.concatenate([[0], np.cumsum(sizes)])
        out = np.empty(len(sizes))
        for i in range(len(sizes)):
            a, b = at[i], at[i + 1]
            dx, dy, dz = _on_device(x[a:b], y[a:b], z[a:b])
            out[i] = _likelihood(torch.linalg.cholesky(_matern(dx, dy, dx, dy, tuple(theta[i]))), dz)[0]
        return out, None
    if case["n"] > 41000:
        return None
    theta = _theta(case)
    if kind in ("predict", "mloe"):
        x, y, miss = _split(case, seed)
        xo, yo, xm, ym = _on_device(x[~miss], y[~miss], x[miss], y[miss])
        L = torch.linalg.cholesky(_matern(xo, yo, xo, yo, theta))
        k = _matern(xo, yo, xm, ym, theta)
        if kind == "predict":
            z, = _on_device(_field(x, y, theta, seed))
            hold = torch.from_numpy(miss).to(z.device)
            zm = k.T @ torch.cholesky_solve(z[~hold][:, None], L)[:, 0]
            return zm.cpu().numpy(), float(((z[hold] - zm) ** 2).mean())
        est = _estimate(case)
        La = torch.linalg.cholesky(_matern(xo, yo, xo, yo, est))
        ka = _matern(xo, yo, xm, ym, est)
        wa = torch.cholesky_solve(ka, La)
        e2 = theta[0] - 2.0 * (k * wa).sum(0) + ((L.T @ wa) ** 2).sum(0)
        e3 = theta[0] - (torch.linalg.solve_triangular(L, k, upper=False) ** 2).sum(0)
        e4 = est[0] - (ka * wa).sum(0)
        return float((e2 / e3 - 1.0).mean()), float((e4 / e2 - 1.0).mean())
    x, y = _on_device(*egs.generate_locations(case["n"], seed % 4096))
    if kind == "fisher":
        s2, beta, nu = theta
        r = _scaled_distance(x, y, x, y, beta)
        zero = r == 0
        r[zero] = 1.0
        k, dk = _bessel_sums(r, nu, derivative=True)
        knext = _bessel_sums(r, nu + 1.0)
        con, rn = 1.0 / (2.0 ** (nu - 1.0) * math.gamma(nu)), r ** nu
        psi = float(torch.special.digamma(torch.tensor(nu, dtype=torch.float64)))
        ds = con * rn * k
        db = s2 * con / beta * rn * (r * knext - 2.0 * nu * k)
        dn = s2 * con * rn * (-(math.log(2.0) + psi) * k + torch.log(r) * k + dk)
        ds[zero], db[zero], dn[zero] = 1.0, 0.0, 0.0
        c = s2 * ds
        c[zero] = s2
        L = torch.linalg.cholesky(c)
        m = [torch.cholesky_solve(d, L) for d in (ds, db, dn)]
        a = torch.stack([torch.stack([0.5 * (p * q.T).sum() for q in m]) for p in m])
        return torch.linalg.inv(a).cpu().numpy()
    C = _matern(x, y, x, y, theta)
    if kind == "sample":
        e, = _on_device(_normal_sequence(seed % 4096, case["n"]))
        return (torch.linalg.cholesky(C) @ e).cpu().numpy()
    z, = _on_device(_field(x.cpu().numpy(), y.cpu().numpy(), theta, seed))
    if kind == "band":
        return _likelihood(_band_factor(C, case["dts"], case["band"]), z)
    L, info = torch.linalg.cholesky_ex(C)
    del C
    return _likelihood(L, z)
