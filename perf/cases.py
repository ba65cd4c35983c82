"""The timed workloads of the package: what a user has it do, through `pmcmc`.

`listed()` names one workload a use, from the README's quick start to the largest
benchmark block; `draw(rng)` gives more of the same kinds over the whole range of
sizes.  `prepare` makes the model, sampler and inputs from a seed, `run` is one
call of the public API, and `exact` is the same result from a sequential FP64
chain (or recurrence) in plain NumPy / PyTorch, with the counter-based tape
(Philox4x32-10 and Box-Muller in FP32) restated.

A DEER solve returns the trajectory of the sequential MALA chain on the same
tape, so every chain workload has an exact value.  Step sizes follow the
stiffness of the target, as an adapted sampler's do: all of these solves converge.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "parallelmcmc.jl_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import pmcmc  # noqa: E402

_NP = {"f32": np.float32, "f64": np.float64}
_TT = {"f32": torch.float32, "f64": torch.float64}


# --------------------------------------------------------------------------- cases
def listed():
    return [
        # the README's quick start: 500 draws of a 2-D standard normal, host arrays, FP64;
        # eight blocks of 64 columns, all latency
        {"name": "quickstart", "kind": "diag", "D": 2, "T": 64, "N": 500, "dtype": "f64",
         "jac": "stoch_diag", "mem": "host", "span": 0.0, "el": 0.1},
        # a long run on an anisotropic diagonal Gaussian kept on the device: the benchmark's
        # moving variant (D = 100, blocks of 16384, exact diagonal, FP32 state)
        {"name": "diag_long", "kind": "diag", "D": 100, "T": 16384, "N": 65536, "dtype": "f32",
         "jac": "diag", "mem": "device", "span": 2.0, "el": 0.5},
        # a correlated Gaussian with a mass matrix, FP64, host arrays, ragged last block
        {"name": "dense_mass", "kind": "dense", "D": 50, "T": 1024, "N": 4000, "dtype": "f64",
         "jac": "stoch_diag", "mem": "host", "mass": True, "el": 0.3},
        # the dense-Jacobian mode on the benchmark's correlated Gaussian
        {"name": "full", "kind": "dense", "D": 64, "T": 8192, "N": 8192, "dtype": "f32",
         "jac": "full", "mem": "device", "mass": False, "el": 0.5},
        # a small logistic regression, one block to host arrays (the size of the smoke test):
        # what a notebook does, and what step-size adaptation does block after block
        {"name": "logit_small", "kind": "logit", "rows": 400, "D": 24, "T": 256,
         "mem": "host", "rule": "default"},
        # an ordinary logistic regression with odd sizes
        {"name": "logit_mid", "kind": "logit", "rows": 3001, "D": 101, "T": 4099,
         "mem": "device", "rule": "default"},
        # more than 256 coefficients
        {"name": "logit_wide", "kind": "logit", "rows": 5000, "D": 400, "T": 8192,
         "mem": "device", "rule": "default"},
        # the headline benchmark block, with the benchmark's stopping rule
        {"name": "logit_large", "kind": "logit", "rows": 10000, "D": 256, "T": 65536,
         "mem": "device", "rule": "tight"},
        # independent uneven logistic chains solved together (MCMCThreads): eight of the
        # benchmark fleet's distribution at a quarter of its rows and lengths
        {"name": "fleet", "kind": "fleet", "chains": 8, "first": 0, "scale": 0.25},
        # the backward direction: d ESJD / d epsilon of a logistic block
        {"name": "logit_adjoint", "kind": "adjoint", "rows": 2000, "D": 64, "T": 2048},
        # sequential chains side by side (warm-up states for many chains)
        {"name": "chains", "kind": "chains", "n": 256, "D": 20, "T": 500, "dtype": "f64",
         "el": 0.3},
        # the affine scan on its own, device tensors
        {"name": "scan", "kind": "scan", "D": 100, "T": 65536, "dtype": "f32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["diag", "diag", "dense", "full", "logit", "logit", "logit", "fleet",
                       "adjoint", "chains", "scan"])
    if kind == "diag":
        T = _log(rng, 64, 16384)
        return {"kind": "diag", "D": _log(rng, 2, 200), "T": T,
                "N": min(65536, _log(rng, T, 6 * T)), "dtype": rng.choice(["f32", "f64"]),
                "jac": rng.choice(["diag", "stoch_diag"]), "mem": rng.choice(["host", "device"]),
                "span": 1.0, "el": 0.3}
    if kind == "dense":
        T = _log(rng, 64, 4096)
        return {"kind": "dense", "D": _log(rng, 3, 80), "T": T, "N": _log(rng, T, 4 * T),
                "dtype": rng.choice(["f32", "f64"]), "jac": "stoch_diag",
                "mem": rng.choice(["host", "device"]), "mass": True, "el": 0.3}
    if kind == "full":
        T = _log(rng, 256, 8192)
        return {"kind": "dense", "D": _log(rng, 8, 100), "T": T, "N": T, "dtype": "f32",
                "jac": "full", "mem": "device", "mass": False, "el": 0.4}
    if kind == "logit":
        return {"kind": "logit", "rows": _log(rng, 300, 10000), "D": _log(rng, 12, 512),
                "T": _log(rng, 128, 16384), "mem": rng.choice(["host", "device"]),
                "rule": "default"}
    if kind == "fleet":
        return {"kind": "fleet", "chains": rng.randint(3, 10), "first": rng.randint(1, 999),
                "scale": round(rng.uniform(0.05, 0.25), 3)}
    if kind == "adjoint":
        return {"kind": "adjoint", "rows": _log(rng, 300, 4000), "D": _log(rng, 12, 128),
                "T": _log(rng, 128, 4096)}
    if kind == "chains":
        return {"kind": "chains", "n": _log(rng, 8, 512), "D": _log(rng, 2, 100),
                "T": _log(rng, 64, 600), "dtype": rng.choice(["f32", "f64"]), "el": 0.3}
    return {"kind": "scan", "D": _log(rng, 2, 300), "T": _log(rng, 256, 65536),
            "dtype": rng.choice(["f32", "f64"])}


# --------------------------------------------------------------------------- inputs
def _gauss(c, rng):
    """(precision: vector or matrix, mass factor or None, epsilon) of a Gaussian case."""
    D = c["D"]
    if c["kind"] in ("diag", "chains"):
        span = c.get("span", 0.5)
        lam = 10.0 ** rng.uniform(-span, span, D)
        lmax = 10.0 ** span
        return lam, None, c["el"] / lmax * min(1.0, 100.0 / D) ** (1 / 3)
    s = 10.0 ** rng.uniform(-1.0, 1.0, D)
    Q, R = np.linalg.qr(rng.standard_normal((D, D)))
    Q = Q * np.sign(np.diag(R))
    P = (Q / s) @ Q.T
    P = 0.5 * (P + P.T)
    if not c["mass"]:
        return P, None, c["el"] / 10.0 * min(1.0, 64.0 / D) ** (1 / 3)
    # a mass matrix as a warm-up estimates it: the covariance, scaled coordinate by coordinate
    w = np.sqrt(rng.uniform(0.7, 1.4, D))
    M = w[:, None] * ((Q * s) @ Q.T) * w[None, :]
    return P, np.linalg.cholesky(0.5 * (M + M.T)), c["el"] * min(1.0, 50.0 / D) ** (1 / 3)


def _logit_data(rng, rows, D):
    X = (rng.standard_normal((rows, D)) / math.sqrt(D)).astype(np.float32).astype(np.float64)
    th = rng.standard_normal(D)
    y = (rng.random(rows) < 1.0 / (1.0 + np.exp(-(X @ th)))).astype(np.float64)
    # step size from the curvature of the posterior: the benchmark's 0.01 at 10000 x 256
    curv = 1.0 + 0.2 * rows / D * (1.0 + math.sqrt(D / rows)) ** 2
    return X, y, 0.1 / curv * min(1.0, 256.0 / D) ** (1 / 3)


def _fleet_data(c, seed):
    out = []
    for k in range(c["chains"]):
        rng = np.random.default_rng([c["first"], k])  # the sizes are the case's
        D = int(16 * rng.integers(1, 33))
        rows = int(rng.integers(1000, 20001) * c["scale"])
        T = int(rng.integers(1024, 32769) * c["scale"])
        rng = np.random.default_rng([int(seed), k])
        out.append((*_logit_data(rng, rows, D), T))
    return out


def _scan_data(c, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    T, D, dt = c["T"], c["D"], _TT[c["dtype"]]
    # a (D, T) trajectory lies column by column, as the package itself returns it
    A = (torch.rand((T, D), generator=g, device="cuda", dtype=dt) * 0.3 + 0.69).T
    B = torch.randn((T, D), generator=g, device="cuda", dtype=dt).T
    return A, B, torch.randn((1, D), generator=g, device="cuda", dtype=dt).reshape(D)


def _logit_sampler(eps, T, rule="default"):
    tol = {"tol_abs": 1e-7, "tol_rel": 1e-6} if rule == "tight" else {}
    return pmcmc.ParallelMALASampler(eps, T=T, jacobian="stoch_diag", dtype=np.float32, **tol)


def prepare(case, seed):
    c, rng = case, np.random.default_rng(seed)
    h = pmcmc.default_handle(0)
    st = {"case": c, "seed": int(seed), "h": h}
    if c["kind"] == "scan":
        st["A"], st["B"], st["s0"] = _scan_data(c, seed)
        return st
    if c["kind"] == "fleet":
        st["chains"] = []
        for k, (X, y, eps, T) in enumerate(_fleet_data(c, seed)):
            m = pmcmc.DensityModel.logistic(X, y)
            m.device_target(h)
            st["chains"].append((m, _logit_sampler(eps, T), np.zeros(X.shape[1], np.float32),
                                 int(seed) + k, 0))
        return st
    if c["kind"] in ("logit", "adjoint"):
        X, y, eps = _logit_data(rng, c["rows"], c["D"])
        st["model"] = pmcmc.DensityModel.logistic(X, y)
        st["sampler"] = _logit_sampler(eps, c["T"], c.get("rule", "default"))
        x0 = np.zeros(c["D"], np.float32)
    else:
        P, mass, eps = _gauss(c, rng)
        st["model"] = (pmcmc.DensityModel.diag_gaussian(P) if P.ndim == 1
                       else pmcmc.DensityModel.dense_gaussian(P))
        st["sampler"] = pmcmc.ParallelMALASampler(
            eps, T=c["T"], jacobian=c.get("jac", "diag"), dtype=_NP[c["dtype"]],
            cholM=None if mass is None else pmcmc.Cholesky(L=mass))
        x0 = rng.standard_normal(c["D"]).astype(_NP[c["dtype"]])
    st["sampler"].target(st["model"], h)
    if c["kind"] == "chains":
        st["x0"] = rng.standard_normal((c["n"], c["D"])).astype(_NP[c["dtype"]])
        st["seeds"] = np.arange(c["n"], dtype=np.uint64) + np.uint64(seed)
        return st
    dev = c.get("mem") == "device" or c["kind"] == "adjoint"
    st["x0"] = torch.from_numpy(x0).cuda() if dev else x0
    if c["kind"] == "adjoint":  # the solved trajectory that its gradient is taken at
        st["S"], _ = pmcmc.solve(st["model"], st["sampler"], st["x0"], seed=st["seed"], handle=h)
    return st


def run(st):
    c, h, seed = st["case"], st["h"], st["seed"]
    if c["kind"] == "scan":
        return pmcmc.solve_affine_scan_diag(st["A"], st["B"], st["s0"], handle=h)
    if c["kind"] == "fleet":
        return [(S, lp, acc) for S, _, lp, acc in pmcmc.fleet_solve(st["chains"], handle=h)]
    if c["kind"] == "chains":
        return pmcmc.mala_chains(st["model"], st["sampler"], st["x0"], st["seeds"], handle=h)
    if c["kind"] == "adjoint":
        return pmcmc.adjoint(st["model"], st["sampler"], st["x0"], st["S"], objective="esjd",
                             seed=seed, handle=h)["d_epsilon"]
    if c["kind"] == "logit":
        S, _, lp, acc = pmcmc.solve(st["model"], st["sampler"], st["x0"], seed=seed, handle=h,
                                    return_logp=True)
        return S, lp, acc
    r = pmcmc.sample(st["model"], st["sampler"], c["N"], seed=seed, initial_params=st["x0"],
                     handle=h)
    return r.values, r.logp, r.accepted


# --------------------------------------------------------------------------- work
def work(case):
    """Inputs read and outputs written once; the operations of evaluating every step of
    the chain once (its forward step and, in a solve, the Jacobian estimate's product)."""
    c = case
    if c["kind"] == "fleet":  # the mean chain of the distribution
        n, s = c["chains"], c["scale"]
        return _logit_work(10500 * s, 264, 16896 * s, n)
    if c["kind"] in ("logit", "adjoint"):
        return _logit_work(c["rows"], c["D"], c["T"], 1)
    es = 4 if c["dtype"] == "f32" else 8
    D = c["D"]
    if c["kind"] == "scan":
        return {"bytes": es * (3 * c["T"] + 1) * D, "flops": 2 * c["T"] * D}
    n = c["n"] * c["T"] if c["kind"] == "chains" else c["N"]
    step = 30 * D if c["kind"] != "dense" else 8 * D * D
    return {"bytes": n * (D * es + es + 1) + es * D * (D if c["kind"] == "dense" else 1),
            "flops": n * step}


def _logit_work(rows, D, T, n):
    return {"bytes": int(n * (4 * rows * D + 4 * rows + T * (4 * D + 5))),
            "flops": int(n * 16 * rows * D * T)}


# --------------------------------------------------------------------------- exact values
def _philox(c0, c1, c2, c3, key):
    """Philox4x32-10 on uint64 arrays holding 32-bit words."""
    m = np.uint64(0xFFFFFFFF)
    k0, k1 = key & 0xFFFFFFFF, (key >> 32) & 0xFFFFFFFF
    sh = np.uint64(32)
    for r in range(10):
        p0 = np.uint64(0xD2511F53) * c0
        p1 = np.uint64(0xCD9E8D57) * c2
        c0, c2 = (p1 >> sh) ^ c1 ^ np.uint64(k0), (p0 >> sh) ^ c3 ^ np.uint64(k1)
        c1, c3 = p1 & m, p0 & m
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def _f(h):
    return np.float32(float.fromhex(h))


def _fma(a, b, c):
    return (a.astype(np.float64) * np.float64(b) + np.asarray(c, np.float64)).astype(np.float32)


def _u01(bits):
    k = (bits >> np.uint64(9)).astype(np.float64)
    return ((2.0 * k + 1.0) * 2.0 ** -24).astype(np.float32)


def _log32(x):
    m, e = np.frexp(x)  # x = m 2^e, m in [0.5, 1)
    m, e = (m * np.float32(2)).astype(np.float32), e - 1
    big = m > _f("0x1.6a09e6p+0")
    m = np.where(big, m * np.float32(0.5), m)
    e = e + big
    s = (m - np.float32(1)) / (m + np.float32(1))
    s2 = s * s
    p = np.full_like(s, _f("0x1.745d18p-4"))
    for k in ("0x1.c71c72p-4", "0x1.24924ap-3", "0x1.99999ap-3", "0x1.555556p-2"):
        p = _fma(p, s2, _f(k))
    t = np.float32(2) * s
    return _fma(e.astype(np.float32), _f("0x1.62e430p-1"), _fma(t * s2, p, t))


def _sincos(u):
    q4 = u * np.float32(4)
    k = np.rint(q4)
    phi = (q4 - k) * _f("0x1.921fb6p+0")
    p2 = phi * phi
    sp = np.full_like(phi, _f("0x1.71de3ap-19"))
    for c in ("-0x1.a01a02p-13", "0x1.111112p-7", "-0x1.555556p-3"):
        sp = _fma(sp, p2, _f(c))
    sn = _fma(phi * p2, sp, phi)
    cp = np.full_like(phi, _f("-0x1.27e4fcp-22"))
    for c in ("0x1.a01a02p-16", "-0x1.6c16c2p-10", "0x1.555556p-5", "-0x1p-1"):
        cp = _fma(cp, p2, _f(c))
    cs = _fma(p2, cp, np.float32(1))
    k = k.astype(np.int64) & 3
    return (np.choose(k, [sn, cs, -sn, -cs]), np.choose(k, [cs, -sn, -cs, sn]))


def _tape(seed, block, D, T, t0=0):
    """xi (T, D) and log u (T,) in FP64 of the tape of (seed, block), columns t0 .. t0 + T - 1."""
    nq = (D + 3) // 4
    t = np.arange(t0, t0 + T, dtype=np.uint64)
    z = np.zeros(T, np.uint64)
    blk = np.uint64(block)
    j, tt = np.tile(np.arange(nq, dtype=np.uint64), T), np.repeat(t, nq)
    w = _philox(j, tt, np.full_like(j, blk), np.full_like(j, 1), int(seed))
    xi = np.empty((T * nq, 4), np.float32)
    for i in (0, 2):
        r = np.sqrt(np.float32(-2) * _log32(_u01(w[i])))
        s, c = _sincos(_u01(w[i + 1]))
        xi[:, i], xi[:, i + 1] = r * c, r * s
    u = _u01(_philox(z, t, z + blk, z + np.uint64(2), int(seed))[0])
    return xi.reshape(T, 4 * nq)[:, :D].astype(np.float64), np.log(u.astype(np.float64))


def _gauss_chain(P, L, eps, x, xi, logu):
    """The sequential FP64 MALA chain (mass matrix L L^T), Gaussian with precision P."""
    T, D = xi.shape
    P = np.asarray(P, np.float64)
    c = math.sqrt(2 * eps)
    if P.ndim == 1:
        prec = lambda v: P * v  # noqa: E731
    else:
        prec = lambda v: P @ v  # noqa: E731
    drift = (lambda g: g) if L is None else (lambda g: L @ (L.T @ g))
    noise = xi if L is None else xi @ L.T
    S, lp, acc = np.empty((T, D)), np.empty(T), np.empty(T, bool)
    px = prec(x)
    ex, dx = 0.5 * (x @ px), drift(-px)
    for t in range(T):
        y = x + eps * dx + c * noise[t]
        py = prec(y)
        ey, dy = 0.5 * (y @ py), drift(-py)
        # the backward proposal's residual in the mass matrix's norm
        r = x - y - eps * dy
        rr = r @ r if L is None else np.sum(np.linalg.solve(L, r) ** 2)
        a = logu[t] < ex - ey - rr / (4 * eps) + 0.5 * (xi[t] @ xi[t])
        if a:
            x, ex, dx = y, ey, dy
        S[t], lp[t], acc[t] = x, -ex, a
    return S, lp, acc


def _logit_chain(X, y, eps, xi, logu):
    """The sequential FP64 chain of a logistic posterior (prior N(0, I)), on the GPU."""
    T, D = xi.shape
    c = math.sqrt(2 * eps)
    Xg, yg = torch.from_numpy(X).cuda(), torch.from_numpy(y).cuda()
    XT = Xg.T.contiguous()
    half = torch.from_numpy(0.5 * np.sum(xi * xi, axis=1) - logu).cuda()
    noise = torch.from_numpy(c * xi).cuda()
    S = torch.empty((T, D), dtype=torch.float64, device="cuda")
    lps = torch.empty(T, dtype=torch.float64, device="cuda")
    acc = torch.empty(T, dtype=torch.bool, device="cuda")

    def model(b):
        l = Xg @ b  # noqa: E741
        lp = torch.dot(yg, l) - torch.nn.functional.softplus(l, threshold=1e4).sum()
        return lp - 0.5 * torch.dot(b, b), XT @ (yg - torch.sigmoid(l)) - b

    x = torch.zeros(D, dtype=torch.float64, device="cuda")
    lx, gx = model(x)
    for t in range(T):
        v = x + eps * gx + noise[t]
        lv, gv = model(v)
        r = x - v - eps * gv
        a = lv - lx - torch.dot(r, r) / (4 * eps) + half[t] > 0
        x, lx, gx = torch.where(a, v, x), torch.where(a, lv, lx), torch.where(a, gv, gx)
        S[t], lps[t], acc[t] = x, lx, a
    return S, lps, acc


def _adjoint_chain(X, y, eps, xi, logu):
    """d/d eps of (1/T) sum_t min(1, alpha_t) |y_t - x_{t-1}|^2 along the sequential FP64
    chain with its accept decisions held fixed, by automatic differentiation."""
    T, D = xi.shape
    Xg, yg = torch.from_numpy(X).cuda(), torch.from_numpy(y).cuda()
    XT = Xg.T.contiguous()
    xig, lu = torch.from_numpy(xi).cuda(), logu
    half = 0.5 * np.sum(xi * xi, axis=1)
    e = torch.tensor(eps, dtype=torch.float64, device="cuda", requires_grad=True)

    def model(b):
        l = Xg @ b  # noqa: E741
        lp = torch.dot(yg, l) - torch.nn.functional.softplus(l, threshold=1e4).sum()
        return lp - 0.5 * torch.dot(b, b), XT @ (yg - torch.sigmoid(l)) - b

    x = torch.zeros(D, dtype=torch.float64, device="cuda")
    lx, gx = model(x)
    total = 0.0
    for t in range(T):
        v = x + e * gx + torch.sqrt(2 * e) * xig[t]
        lv, gv = model(v)
        r = x - v - e * gv
        la = lv - lx - torch.dot(r, r) / (4 * e) + half[t]
        d = v - x
        total = total + torch.exp(torch.clamp(la, max=0.0)) * torch.dot(d, d)
        if float(la.detach()) > lu[t]:
            x, lx, gx = v, lv, gv
    (total / T).backward()
    return float(e.grad)


def exact(case, seed):
    c, rng = case, np.random.default_rng(seed)
    if c["kind"] == "scan":
        A, B, s = (v.T.double().cpu().numpy() for v in _scan_data(c, seed))
        S = np.empty_like(A)
        for t in range(A.shape[0]):
            s = A[t] * s + B[t]
            S[t] = s
        return S.T
    if c["kind"] == "fleet":
        out = []
        for k, (X, y, eps, T) in enumerate(_fleet_data(c, seed)):
            S, lp, acc = _logit_chain(X, y, eps, *_tape(int(seed) + k, 0, X.shape[1], T))
            out.append((S.T, lp, acc))
        return out
    if c["kind"] == "logit":
        X, y, eps = _logit_data(rng, c["rows"], c["D"])
        S, lp, acc = _logit_chain(X, y, eps, *_tape(seed, 0, c["D"], c["T"]))
        return S.T, lp, acc
    if c["kind"] == "adjoint":
        X, y, eps = _logit_data(rng, c["rows"], c["D"])
        return _adjoint_chain(X, y, eps, *_tape(seed, 0, c["D"], c["T"]))
    P, L, eps = _gauss(c, rng)
    dt = _NP[c["dtype"]]
    x0 = rng.standard_normal(c["D"]).astype(dt).astype(np.float64)
    if c["kind"] == "chains":
        xs = rng.standard_normal((c["n"], c["D"])).astype(dt).astype(np.float64)
        r = [_gauss_chain(P, L, eps, xs[k], *_tape(int(seed) + k, 0, c["D"], c["T"]))
             for k in range(c["n"])]
        return tuple(np.stack([v[i] for v in r]) for i in range(3))
    parts, left, b = [], c["N"], 0
    while left > 0:
        n = min(left, c["T"])
        parts.append(_gauss_chain(P, L, eps, x0, *_tape(seed, b, c["D"], n)))
        x0, left, b = parts[-1][0][-1], left - n, b + 1
    return tuple(np.concatenate([p[i] for p in parts]) for i in range(3))
