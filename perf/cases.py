"""The workloads of this library that are timed and compared between versions.

Each case is one call (or the few calls that belong together) of the public
Python front end (highreg.py) as a user's program makes it, over the range in
which the library is used: the stateless boundary sums on host arrays, the
two-surface plan's right-hand side, operator and GMRES solve on device
vectors, the extend-to-grid sums, the Poisson transform, and the warm-start
network's training.

A case is a dict of plain values; ``what`` says which path it takes:

  sum      a stateless sum Context.{sl,dl}_{on,off}surf, host arrays in and out
  interp   Context.interpolate_dl_density, host arrays in and out
  matvec   Plan2S.matvec_dev, one operator application on device vectors
  rhs      Plan2S.rhs_dev
  solve    Plan2S.rhs_dev + Plan2S.solve_dev (GMRES to 1e-10)
  band     Context.e2g_sl_7ord + e2g_p_7ord at the grid points near the surface
  face     Context.e2g_sl_away + e2g_p_away at the box-face points
  dst      Context.dst_poisson3d, a grid of n^3 points
  train    ten MLP.train_step calls, then the weights (MLP.params)

N is 1/h (3/h for the extend-to-grid scene). Geometry is the library's own;
densities are smooth fields of the position drawn from the seed.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "high-order-regularization_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import highreg  # noqa: E402

PREC = {"fp64": highreg.HR_FP64, "mixed": highreg.HR_MIXED, "fp32": highreg.HR_FP32}
MODE = {"direct": highreg.HR_DIRECT, "tree": highreg.HR_TREE}
DEV = "cuda:0"
_ctx = None


def context():
    """A program has one context (one stream)."""
    global _ctx
    if _ctx is None:
        _ctx = highreg.Context(0)
    return _ctx


def listed():
    return [
        # the smallest call: a coarse surface's own Stokeslet sum, all pairs, host arrays: latency
        dict(name="sl_on_direct_h16", what="sum", kind="sl_on", mode="direct", N=16, P=4, N0=300, prec="fp64"),
        # a drop-in stresslet sum at the other surface's points through the treecode, host arrays
        dict(name="dl_off_tree_h32", what="sum", kind="dl_off", mode="tree", N=32, P=6, N0=1000, prec="fp64"),
        # the coarse two-surface solve, right-hand side to solution: the whole call of a parameter study
        dict(name="solve_h32", what="solve", N=32, P=6, N0=1000, prec="fp64"),
        # one operator application of the headline problem (n = 171,054), FP64
        dict(name="matvec_h64", what="matvec", N=64, P=6, N0=2000, prec="fp64"),
        # the same in the reduced precision of the refinement solver's inner cycles
        dict(name="matvec_h64_mixed", what="matvec", N=64, P=6, N0=2000, prec="mixed"),
        # the headline problem's right-hand side (Stokeslet sums)
        dict(name="rhs_h64", what="rhs", N=64, P=6, N0=2000, prec="fp64"),
        # an odd grid between the documented ones, another degree and leaf size
        dict(name="matvec_h101", what="matvec", N=101, P=7, N0=1500, prec="fp64"),
        # the largest documented problem (n = 2,740,992)
        dict(name="matvec_h256", what="matvec", N=256, P=10, N0=8000, prec="fp64"),
        # extend-to-grid at N = 96: velocity and pressure near the surface, and on the box faces
        dict(name="band_n96", what="band", N=96),
        dict(name="face_n96", what="face", N=96),
        # the Poisson transform of the same grid
        dict(name="dst_n95", what="dst", n=95),
        # warm-start training at its documented batch size
        dict(name="train_b16384", what="train", batch=16384, n=65536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["sum", "sum", "sum", "matvec", "matvec", "rhs", "solve", "band", "face", "dst", "train", "interp"])
    if what == "sum":
        return dict(what=what, kind=rng.choice(["sl_on", "sl_off", "dl_on", "dl_off"]),
                    mode=rng.choice(["direct", "tree"]), N=_log(rng, 12, 56), P=rng.randint(2, 9),
                    N0=_log(rng, 100, 3000), prec=rng.choice(["fp64", "fp64", "mixed", "fp32"]))
    if what == "interp":
        return dict(what=what, N=_log(rng, 14, 64))
    if what in ("matvec", "rhs"):
        return dict(what=what, N=_log(rng, 20, 150), P=rng.randint(3, 10), N0=_log(rng, 500, 6000),
                    prec="fp64" if what == "rhs" else rng.choice(["fp64", "fp64", "mixed", "fp32"]))
    if what == "solve":
        return dict(what=what, N=_log(rng, 16, 64), P=rng.randint(4, 8), N0=_log(rng, 500, 3000), prec="fp64")
    if what in ("band", "face"):
        return dict(what=what, N=2 * _log(rng, 20, 80))
    if what == "dst":
        return dict(what=what, n=2 * _log(rng, 15, 80) - 1)
    return dict(what=what, batch=_log(rng, 300, 60000), n=_log(rng, 20000, 200000))


# ------------------------------------------------------------------ inputs
def _field(seed):
    """A smooth vector field of the position, other for every seed."""
    r = np.random.default_rng(seed)
    a, b, c = r.standard_normal(3), 0.5 * r.standard_normal((3, 3)), r.standard_normal(3)
    w, ph = 2.0 * r.standard_normal((3, 3)), r.uniform(0, 2 * np.pi, 3)

    def f(xyz):
        x = np.asarray(xyz).reshape(-1, 3)
        return (a + x @ b + c * np.sin(x @ w + ph)).reshape(-1)

    return f


def _e2g_scene(N):
    e = highreg.E2G(context(), N)
    sc, info = e.scene(), dict(e.info)
    e.close()
    return sc, info


def _host(case, seed):
    """The host arrays of the sum, interp, band and face cases."""
    f = _field(seed)
    if case["what"] in ("band", "face"):
        sc, info = _e2g_scene(case["N"])
        d = dict(xq=sc["xq"], nrm=sc["nrm"], area=sc["area"], f=f(sc["xq"]), DEL=info["delta"])
        if case["what"] == "band":  # the tagged grid points outside or on the surface
            sel = sc["b"] >= -1e-12
            b, x0, n0 = sc["b"][sel], sc["x0"].reshape(-1, 3)[sel], sc["n0"].reshape(-1, 3)[sel]
            d.update(xt=(x0 + b[:, None] * n0).reshape(-1), b=b, n0=n0.reshape(-1).copy(), f0=f(x0))
        else:  # the grid points on the box's six faces
            N, h = case["N"], info["h"]
            g = np.arange(N + 1)
            i, j, k = (v.reshape(-1) for v in np.meshgrid(g, g, g, indexing="ij"))
            on = (i % N == 0) | (j % N == 0) | (k % N == 0)
            d.update(xt=(h * np.stack([i[on], j[on], k[on]], 1)).reshape(-1).astype(np.float64))
        return d
    geo = highreg.Geometry2S(case["N"]).scene
    on = case.get("kind", "dl_off").endswith("on")
    s, t = (0, 0) if on else (1, 0)  # off-surface: surface 1's sum at the points of surface 0
    d = dict(DEL=geo["DEL"], h=geo["h"], ctr=geo["ctr%d" % s], xq=geo["xq%d" % s], nrm=geo["nrm%d" % s],
             area=geo["area%d" % s], plane=geo["plane%d" % s], q=f(geo["xq%d" % s]))
    if not on:
        # points without a nearest-point subtraction (nrst 0) carry no nearest density, as in the plan
        q0 = f(geo["x0%d" % t]) * np.repeat(geo["nrst%d" % t] != 0, 3)
        d.update(xt=geo["xq%d" % t], b=geo["b%d" % t], x0=geo["x0%d" % t], n0=geo["n0%d" % t],
                 nrst=geo["nrst%d" % t], i123=geo["i123%d" % t], q0=q0)
    return d


def _train_data(case, seed):
    r = np.random.default_rng(seed)
    X = r.standard_normal((case["n"], highreg.NFEAT)).astype(np.float32)
    W = r.standard_normal((highreg.NFEAT, 3)) / math.sqrt(highreg.NFEAT)
    T = (np.tanh(X @ W) + 0.1 * r.standard_normal((case["n"], 3))).astype(np.float32)
    return X, T, r.normal(0, 0.1, highreg.NFEAT).astype(np.float32), r.uniform(0.8, 1.2, highreg.NFEAT).astype(np.float32)


LR, SCALE, STEPS = 1e-3, 0.7, 10


def prepare(case, seed):
    ctx, what = context(), case["what"]
    st = dict(case=dict(case))
    if what in ("sum", "interp", "band", "face"):
        st["d"] = _host(case, seed)
    elif what in ("matvec", "rhs", "solve"):
        geo = highreg.Geometry2S(case["N"]).scene
        st["plan"] = plan = highreg.Plan2S(ctx, geo, mode=highreg.HR_TREE, P=case["P"], N0=case["N0"], theta=0.6)
        f = _field(seed)
        if what == "matvec":
            r = np.random.default_rng(seed + 1)
            x = np.concatenate([f(geo["xq0"]), f(geo["xq1"])])
            st["x"] = torch.from_numpy(x + 0.01 * r.standard_normal(len(x))).to(DEV)
        else:
            # the scene's interfacial forces, modulated by the seed's field
            for s in (0, 1):
                st["f%d" % s] = torch.from_numpy(geo["f%d" % s] * (1.0 + 0.1 * np.sin(f(geo["xq%d" % s])))).to(DEV)
            st["x"] = torch.empty(plan.n, dtype=torch.float64, device=DEV)
        st["y"] = torch.empty(plan.n, dtype=torch.float64, device=DEV)
    elif what == "dst":
        st["f"] = np.random.default_rng(seed).standard_normal(case["n"] ** 3)
    else:
        X, T, mean, std = _train_data(case, seed)
        st["X"], st["T"] = torch.from_numpy(X).to(DEV), torch.from_numpy(T).to(DEV)
        st["mlp"] = highreg.MLP(ctx, seed=seed)
        st["mlp"].set_normalization(mean, std, SCALE)
        st["seed"] = seed
    torch.cuda.synchronize()  # the library works on its own stream
    return st


def run(st):
    ctx, case = context(), st["case"]
    what = case["what"]
    if what == "sum":
        d, kind = st["d"], case["kind"]
        opt = dict(mode=MODE[case["mode"]], P=case["P"], N0=case["N0"], theta=0.6, precision=PREC[case["prec"]])
        a = (d["DEL"], d["xq"], d["nrm"], d["area"], d["q"])
        if kind == "sl_on":
            return ctx.sl_onsurf(*a, ctr=d["ctr"], **opt)
        if kind == "dl_on":
            return ctx.dl_onsurf(*a, ctr=d["ctr"], **opt)
        if kind == "sl_off":
            return ctx.sl_offsurf(*a, d["xt"], d["b"], d["n0"], d["q0"], ctr=d["ctr"], **opt)
        return ctx.dl_offsurf(*a, d["xt"], d["b"], d["x0"], d["n0"], d["q0"], ctr=d["ctr"], **opt)
    if what == "interp":
        d = st["d"]
        return ctx.interpolate_dl_density(d["h"], d["xq"], d["q"], d["ctr"], d["plane"], d["x0"], d["nrst"], d["i123"])
    if what == "matvec":
        st["plan"].matvec_dev(st["x"], st["y"], PREC[case["prec"]])
        return st["y"]
    if what == "rhs":
        st["plan"].rhs_dev(st["f0"], st["f1"], st["y"])
        return st["y"]
    if what == "solve":
        st["plan"].rhs_dev(st["f0"], st["f1"], st["y"])
        rep = st["plan"].solve_dev(st["y"], st["x"], restart=50, tol=1e-10, precision=PREC[case["prec"]])
        return {"b": st["y"], "x": st["x"], "iterations": rep["iterations"]}
    if what == "band":
        d = st["d"]
        a = (d["DEL"], d["xq"], d["nrm"], d["area"], d["f"], d["xt"], d["b"], d["f0"], d["n0"])
        return {"u": ctx.e2g_sl_7ord(*a), "p": ctx.e2g_p_7ord(*a)}
    if what == "face":
        d = st["d"]
        a = (d["xq"], d["area"], d["f"], d["xt"])
        return {"u": ctx.e2g_sl_away(*a), "p": ctx.e2g_p_away(*a)}
    if what == "dst":
        return ctx.dst_poisson3d(case["n"], st["f"])
    for _ in range(STEPS):
        st["mlp"].train_step(st["X"], st["T"], case["batch"], LR, seed=st["seed"])
    return st["mlp"].params()


# -------------------------------------------------------------------- work
def _surface_points(N):
    return 6.83 * N * N  # points of one of the two surfaces (27,934 at N = 64)


def work(case):
    """Bytes: inputs once, outputs once. FLOPs: pair evaluations x the fixed
    per-pair counts of the sums (57 / 59 Stokeslet, 50 / 129 stresslet, 31 / 18
    plain Stokeslet / pressure); the treecode's pair count by a fit to its own
    statistics at the documented sizes."""
    what = case["what"]
    if what == "sum":
        n = _surface_points(case["N"])
        on, dl = case["kind"].endswith("on"), case["kind"].startswith("dl")
        per = (50 if on else 60) if dl else (57 if on else 45)
        pairs = n * n
        if case["mode"] == "tree":
            pairs = n * (min(n, 2.6 * case["N0"]) + (16 * (case["P"] + 1) ** 3 if n > 3 * case["N0"] else 0))
        return {"bytes": 8.0 * n * (13 if on else 26), "flops": pairs * per}
    if what == "interp":
        n = _surface_points(case["N"])
        return {"bytes": 8.0 * n * 13, "flops": 0.5 * n * 250}
    if what in ("matvec", "rhs", "solve"):
        n = _surface_points(case["N"])
        pairs = 4 * n * (min(n, 2.6 * case["N0"]) + (16 * (case["P"] + 1) ** 3 if n > 3 * case["N0"] else 0))
        times = {"matvec": 1, "rhs": 1, "solve": 14}[what]
        return {"bytes": 8.0 * 2 * n * (26 + 6) * times, "flops": pairs * (45 if what == "rhs" else 51) * times}
    if what in ("band", "face"):
        nq = 0.755 * case["N"] ** 2
        nt = 2.9 * case["N"] ** 2 if what == "band" else 6.0 * case["N"] ** 2
        return {"bytes": 8.0 * (10 * nq + 14 * nt), "flops": nq * nt * (123 if what == "band" else 49)}
    if what == "dst":
        n = case["n"]
        return {"bytes": 16.0 * n ** 3, "flops": 6 * 2.5 * n ** 3 * math.log2(n + 1)}
    params = 9347
    return {"bytes": STEPS * (4.0 * case["batch"] * 15 + 32 * params), "flops": STEPS * 6.0 * case["batch"] * params}


# ------------------------------------------------------------------- exact
_RP = math.sqrt(math.pi)


def _coeff(lam):
    """The target's coefficients c1, c2, c3 of the 7th-order regularized kernels."""
    l2, al = lam * lam, lam.abs()
    e, t = torch.exp(-l2) / _RP, al * torch.special.erfc(al)
    i0, i2 = e - t, 2 / 3 * ((0.5 - l2) * e + l2 * t)
    i4 = 8 / 15 * ((0.75 - 0.5 * l2 + l2 * l2) * e - l2 * l2 * t)
    e2 = torch.exp(l2)
    c3 = e2 * (2 * i0 - 4 * i2 + i4) / 8
    c2 = e2 * (i0 - i2) + (4 * l2 + 7) * c3
    c1 = 2 * e2 * i0 + 2 * (l2 + 1) * c2 - (4 * l2 * l2 + 6 * l2 + 6) * c3
    return c1[:, None], c2[:, None], c3[:, None]


def _factors(r2, DEL, c):
    """s1 ~ 1/r, s2 ~ 1/r^3, s3 ~ 1/r^5 with the target's coefficients."""
    r = r2.sqrt()
    rd = r / DEL
    s = rd * rd
    erf, x = torch.erf(rd), rd * torch.exp(-s)
    c1, c2, c3 = c
    p1 = c1 - 2 * (c2 + c3) * s + 4 * c3 * s ** 2
    p2 = -2 / _RP + 2 * (c1 + 2 * (c2 + c3)) * s - 4 * (c2 + 5 * c3) * s ** 2 + 8 * c3 * s ** 3
    p3 = -2 / _RP * (1 + 2 / 3 * s) + 4 / 3 * ((c1 + 4 * c2 + 12 * c3) * s ** 2 - 2 * (c2 + 9 * c3) * s ** 3 + 4 * c3 * s ** 4)
    far, zero = rd > 8, r < 1e-14
    s1 = torch.where(far, 1 / r, (erf + p1 * x) / r)
    s2 = torch.where(far, 1 / r ** 3, (erf + p2 * x) / r ** 3)
    s3 = torch.where(far, 1 / r ** 5, (erf + p3 * x) / r ** 5)
    one = torch.ones_like(r)
    return (torch.where(zero, 32 / 5 / _RP / DEL * one, s1), torch.where(zero, 256 / 15 / _RP / DEL ** 3 * one, s2),
            torch.where(zero, 0 * one, s3))


def _factors_on(r2, DEL):
    """The same for a target on the surface (b = 0, the stresslet's own polynomial)."""
    r = r2.sqrt()
    rd = r / DEL
    s = rd * rd
    erf, x = torch.erf(rd), 2 / _RP * rd * torch.exp(-s)
    far, zero, one = rd > 8, r < 1e-14, torch.ones_like(r)
    s1 = torch.where(far, 1 / r, (erf + (11 / 5 - 26 / 15 * s + 4 / 15 * s ** 2) * x) / r)
    s2 = torch.where(far, 1 / r ** 3, (erf + (-1 + (118 * s - 68 * s ** 2 + 8 * s ** 3) / 15) * x) / r ** 3)
    s3 = torch.where(far, 1 / r ** 5, (erf + (-1 - 2 / 3 * s + 52 / 45 * s ** 2 - 8 / 45 * s ** 3) * x) / r ** 5)
    return (torch.where(zero, 32 / 5 / _RP / DEL * one, s1), torch.where(zero, 256 / 15 / _RP / DEL ** 3 * one, s2),
            torch.where(zero, 128 / 45 / _RP / DEL ** 5 * one, s3))


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _sum_block(kind, DEL, src, q, tg):
    """One block of targets against all sources: the boundary sum's three components."""
    x, n, a = src  # 3 x (1, nq), 3 x (1, nq), (1, nq)
    d = [tg["x"][k] - x[k] for k in range(3)]
    r2 = _dot(d, d)
    if kind in ("sl_on", "sl_off", "sl7"):
        if kind == "sl_on":
            s1, s2, _ = _factors_on(r2, DEL)
            near = torch.ones_like(tg["b"], dtype=torch.bool)
        else:
            s1, s2, _ = _factors(r2, DEL, _coeff((tg["b"] / DEL).clamp(-8, 8)[:, 0]))
            near = (tg["b"].abs() / DEL <= 8) if kind == "sl_off" else torch.ones_like(tg["b"], dtype=torch.bool)
            r = r2.sqrt()
            s1, s2 = torch.where(near, s1, 1 / r), torch.where(near, s2, 1 / r ** 3)
        fn = torch.where(near, _dot(tg["q0"], tg["n0"]), torch.zeros_like(tg["b"]))
        f = [q[k] - fn * n[k] for k in range(3)]
        fd = _dot(f, d) * s2
        return [((f[k] * s1 + d[k] * fd) * a).sum(1) / (8 * math.pi) for k in range(3)]
    if kind == "p7":
        _, s2, _ = _factors(r2, DEL, _coeff((tg["b"] / DEL)[:, 0]))
        f0, n0 = tg["q0"], tg["n0"]
        cross = lambda u, v: [u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0]]  # noqa: E731
        nf, nf0, nd = cross(n, q), cross(n0, f0), cross(n, d)
        k = -(_dot(q, n) - _dot(f0, n0)) * _dot(n, d) - _dot([nf[i] - nf0[i] for i in range(3)], nd)
        return [-(k * s2 * a).sum(1) / (4 * math.pi) - torch.where(tg["b"] < -1e-12, _dot(f0, n0), 0 * tg["b"])[:, 0]]
    if kind == "dl_on":
        _, _, s3 = _factors_on(r2, DEL)
        g = [q[k] - tg["q0"][k] for k in range(3)]
        w = _dot(n, d) * _dot(g, d) * s3 * a
        return [-6 / (8 * math.pi) * (d[k] * w).sum(1) + 0.5 * tg["q0"][k][:, 0] for k in range(3)]
    near = tg["b"].abs() / DEL <= 8
    _, s2, s3 = _factors(r2, DEL, _coeff((tg["b"] / DEL).clamp(-8, 8)[:, 0]))
    b, n0, g0 = tg["b"], tg["n0"], tg["q0"]
    xh = [x[k] - tg["x0"][k] for k in range(3)]
    g = [q[k] - g0[k] for k in range(3)]
    sig = _dot(xh, xh) - 2 * b * _dot(xh, n0)
    gn0, gxh, nn, xn = _dot(g, n0), _dot(g, xh), _dot(n0, n), _dot(xh, n)
    c1a, c1b = gn0 * nn, gxh * nn + gn0 * xn
    c2a, c2b = gxh * xn, b * c1b
    plain = _dot(q, d) * _dot(n, d) / r2 ** 2.5
    out = []
    for k in range(3):
        m1 = d[k] * c1a - n0[k] * c1b
        m2 = -sig * m1 + d[k] * c2a + xh[k] * c2b
        v = torch.where(near, m1 * s2 + m2 * s3, d[k] * plain)
        out.append(-6 / (8 * math.pi) * (v * a).sum(1))
    return out


def _boundary_sum(kind, DEL, d, q, jump=None):
    """The all-pairs sum of one kind over every target, in float64, (3 or 1) x nt interleaved."""
    g = lambda v, w=3: torch.from_numpy(np.ascontiguousarray(v)).to(DEV).reshape(-1, w)  # noqa: E731
    cols = lambda t: [t[:, k][None, :] for k in range(3)]  # noqa: E731
    src, qs = (cols(g(d["xq"])), cols(g(d["nrm"])), g(d["area"], 1).T), cols(g(q))
    on = kind.endswith("on")
    xt = g(d["xq"] if on else d["xt"])
    nt = len(xt)
    z = np.zeros(nt)
    b = g(z if on else d["b"], 1)
    n0, q0 = g(d["nrm"] if on else d["n0"]), g(q if on else d["q0" if "q0" in d else "f0"])
    x0 = g(d["x0"]) if "x0" in d and not on else xt
    step = max(16, int(6e6 // src[2].numel()))
    outs = []
    for t0 in range(0, nt, step):
        sl = slice(t0, min(nt, t0 + step))
        tc = lambda t: [t[sl, k][:, None] for k in range(3)]  # noqa: E731
        o = _sum_block(kind, DEL, src, qs, dict(x=tc(xt), b=b[sl], n0=tc(n0), q0=tc(q0), x0=tc(x0)))
        outs.append(torch.stack(o, 1))
    out = torch.cat(outs)
    if kind == "dl_off":
        bb = b[:, 0]
        if jump == "tree":
            xi = torch.where(bb.abs() < 1e-12, 0.5, torch.where(bb < 0, 1.0, 0.0))
        else:
            xi = torch.where((bb.abs() / DEL <= 8) & ((bb < 0) | (bb.abs() < 1e-14)), 1.0, 0.0)
        out = out + xi[:, None].double() * q0
    return out.reshape(-1)


def _away_sums(d):
    g = lambda v, w=3: torch.from_numpy(np.ascontiguousarray(v)).to(DEV).reshape(-1, w)  # noqa: E731
    x, f, a, xt = g(d["xq"]), g(d["f"]), g(d["area"], 1).T, g(d["xt"])
    step, us, ps = max(16, int(8e6 // len(x))), [], []
    for t0 in range(0, len(xt), step):
        dx = [xt[t0:t0 + step, k][:, None] - x[:, k][None, :] for k in range(3)]
        r = _dot(dx, dx).sqrt()
        fc = [f[:, k][None, :] for k in range(3)]
        fd = _dot(fc, dx) / r ** 3 * a
        us.append(torch.stack([(fc[k] / r * a + dx[k] * fd).sum(1) for k in range(3)], 1))
        ps.append(fd.sum(1))
    return {"u": torch.cat(us).reshape(-1) / (8 * math.pi), "p": torch.cat(ps) / (4 * math.pi)}


def _mix64(x):
    x = x + np.uint64(0x9E3779B97F4A7C15)
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def _initial_weights(seed):
    shapes, p, off = [(12, 64), (64, 64), (64, 64), (64, 3)], [], 0
    with np.errstate(over="ignore"):
        for i, o in shapes:
            k = np.arange(off + 1, off + i * o + 1, dtype=np.uint64)
            h = np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * k
            h = (h ^ (h >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            h = (h ^ (h >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
            h ^= h >> np.uint64(31)
            u = (h >> np.uint64(11)).astype(np.float64) / 9007199254740992.0
            p += [((2 * u - 1) * math.sqrt(6.0 / (i + o))).astype(np.float32).reshape(i, o), np.zeros(o, np.float32)]
            off += i * o + o
    return [torch.from_numpy(v).double().to(DEV).requires_grad_() for v in p]


def _train(case, seed):
    """Ten Adam steps (0.9, 0.999, 1e-8) on the mean squared error of the 12-64-64-64-3 SiLU network."""
    X, T, mean, std = _train_data(case, seed)
    X = (torch.from_numpy(X).double() - torch.from_numpy(mean).double()) / torch.from_numpy(std).double()
    X, T, p = X.to(DEV), torch.from_numpy(T).double().to(DEV) / SCALE, _initial_weights(seed)
    m, v = [torch.zeros_like(w) for w in p], [torch.zeros_like(w) for w in p]
    for step in range(1, STEPS + 1):
        with np.errstate(over="ignore"):
            s = np.arange(case["batch"], dtype=np.uint64)
            at = _mix64(np.uint64(seed) ^ _mix64((np.uint64(step) << np.uint64(32)) ^ s)) % np.uint64(case["n"])
        at = torch.from_numpy(at.astype(np.int64)).to(DEV)
        a = X[at]
        for l in range(3):
            a = torch.nn.functional.silu(a @ p[2 * l] + p[2 * l + 1])
        loss = ((a @ p[6] + p[7] - T[at]) ** 2).mean()
        grads = torch.autograd.grad(loss, p)
        with torch.no_grad():
            for w, g, mi, vi in zip(p, grads, m, v):
                mi.mul_(0.9).add_(g, alpha=0.1)
                vi.mul_(0.999).addcmul_(g, g, value=0.001)
                w -= LR * (mi / (1 - 0.9 ** step)) / ((vi / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return torch.cat([w.detach().reshape(-1) for w in p])


def _dst_poisson(n, f):
    """DST-I on all axes, division by the eigenvalues of the 4th-order compact Laplacian, DST-I, scale."""
    N = n + 1
    k = torch.arange(1, N, dtype=torch.int64, device=DEV)
    S = 2 * torch.sin(math.pi / N * ((k[:, None] * k[None, :]) % (2 * N)).double())

    def dst(t):  # each product moves the transformed axis to the end: three restore the order
        for _ in range(3):
            t = torch.tensordot(t, S, dims=([0], [0]))
        return t

    k = k.double()
    c, s = torch.cos(math.pi / N * k), -2 * torch.sin(0.5 * math.pi / N * k) ** 2
    axes = lambda v: (v[:, None, None], v[None, :, None], v[None, None, :])  # noqa: E731
    (c0, c1, c2), (s0, s1, s2) = axes(c), axes(s)
    factor = 2 / 3 * (2 * (s0 + s1 + s2) + c0 * c1 * c2 - 1)
    return dst(dst(torch.from_numpy(f).to(DEV).reshape(n, n, n)) / factor).reshape(-1) / (2.0 * N) ** 3


def exact(case, seed):
    what = case["what"]
    if what == "sum":  # a treecode's sum is compared with the all-pairs sum that it approximates
        d = _host(case, seed)
        return _boundary_sum(case["kind"], d["DEL"], d, d["q"], jump=case["mode"])
    if what == "band":
        d = _host(case, seed)
        return {"u": _boundary_sum("sl7", d["DEL"], d, d["f"]), "p": _boundary_sum("p7", d["DEL"], d, d["f"])}
    if what == "face":
        return _away_sums(_host(case, seed))
    if what == "rhs" and case["N"] <= 64:
        geo = highreg.Geometry2S(case["N"]).scene
        f = _field(seed)
        q = [geo["f%d" % s] * (1.0 + 0.1 * np.sin(f(geo["xq%d" % s]))) for s in (0, 1)]
        b = []
        for t in (0, 1):
            g = lambda s: dict(xq=geo["xq%d" % s], nrm=geo["nrm%d" % s], area=geo["area%d" % s])  # noqa: E731
            off = dict(g(1 - t), xt=geo["xq%d" % t], b=geo["b%d" % t], x0=geo["x0%d" % t], n0=geo["n0%d" % t], q0=geo["f0%d" % t])
            b.append(_boundary_sum("sl_on", geo["DEL"], g(t), q[t]) + _boundary_sum("sl_off", geo["DEL"], off, q[1 - t]))
        return -2 / 3 * torch.cat(b)
    if what == "dst":
        return _dst_poisson(case["n"], np.random.default_rng(seed).standard_normal(case["n"] ** 3))
    if what == "train":
        return _train(case, seed)
    return None  # the operator with its density interpolation, and the solve
