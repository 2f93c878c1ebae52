"""The work that a user of this framework has it do, as cases to time.

A case is one pass through the public entry points of ``mcnla_b200.isvd``: a whole solve (FP64 or the
precision form), one stage of a solve (sketch, orthogonalizer, integrator, former), or a batch of
requests through the server.  Sizes are those of the repository's own configurations, tests and
benchmark: 100000 x 20000 with 64 sketches of 64 columns down to a few hundred rows, the uneven batch
(m in [512, 16384], n in [256, 4096], k in {8, 16, 32, 64}, 8 sketches) and the 1000 x 2000 problems.
"""
import math

import numpy as np
import torch

from mcnla_b200 import isvd

# Work of the largest drawn case against the largest listed one (FP64 operations of a solve).
MAX_FLOPS = 1.0e13
WY_STEPS = 12


# ----------------------------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------------------------
def _solve(name, m, n, k, p, N, integrator, former, tol, spectrum, layout="row", omega=True, mixed=0):
    return {"name": name, "kind": "solve", "m": m, "n": n, "k": k, "p": p, "N": N, "integrator": integrator,
            "former": former, "tol": tol, "spectrum": spectrum, "layout": layout, "omega": omega, "mixed": mixed}


def _stage(name, kind, m, n, k, p, N, stage="", tol=0.0, spectrum="power", layout="row", exponent=0):
    return {"name": name, "kind": kind, "m": m, "n": n, "k": k, "p": p, "N": N, "stage": stage, "tol": tol,
            "spectrum": spectrum, "layout": layout, "exponent": exponent}


def listed():
    return [
        # the smallest request of the uneven batch, solved alone: launches and waits are all there is
        _solve("solve_smallest", 512, 257, 8, 4, 8, "rb_gramian_kn", "rb_gramian", 1e-5, "power"),
        # the plain configuration: 1000 x 2000, 16 sketches of 20 columns, the default stages
        _solve("solve_plain", 1000, 2000, 10, 10, 16, "kn", "svd", 1e-4, "power"),
        # many wide sketches of a small matrix with a steep spectrum: the integrator's l x l work rules
        _solve("solve_steep", 1000, 2000, 64, 16, 32, "rb_gramian_kn", "svd", 1e-4, "steep"),
        # the headline configuration, FP64, Omega drawn on the device
        _solve("solve_large", 100000, 20000, 50, 14, 64, "rb_gramian_kn", "rb_gramian", 1e-6, "noise", omega=False),
        # the same shape at half the rows in the precision form, BF16 parts resident
        _solve("solve_large_mixed", 50000, 20000, 50, 14, 64, "rb_gramian_kn", "rb_gramian", 1e-6, "noise",
               omega=False, mixed=2),
        # the column-block driver: column-major A, Omega given
        _solve("solve_colblock", 16384, 8192, 50, 14, 32, "rb_kn", "cb_gramian", 1e-4, "noise", layout="col"),
        # one sketch stage at the top of the uneven batch, odd sizes
        _stage("sketch_ragged", "sketch", 16383, 4095, 64, 32, 8),
        # the orthogonalizer of a large request's sketches (l = 160: the widest the library takes)
        _stage("orthogonalize_wide", "orthogonalize", 20000, 2000, 128, 32, 16),
        # the Gramian integrator with the headline's sketches on fewer rows
        _stage("integrate_kn", "integrate", 20000, 2000, 50, 14, 64, stage="rb_gramian_kn", tol=1e-6,
               spectrum="noise"),
        # the drivers' default integrator (Wen-Yin) on a mid-size problem's sketches.  Its line search carries
        # rounding into its step sizes, more with every step, so it is timed on given bases for a given number of
        # steps (WY_STEPS, the drivers' maximum-iteration argument) and not in whole solves
        _stage("integrate_wy", "integrate", 16384, 2000, 50, 14, 16, stage="rb_wy", tol=1e-3, spectrum="noise"),
        # the SVD former of a wide request
        _stage("form_svd", "form", 16384, 4096, 64, 32, 8, stage="svd"),
        # served requests of uneven sizes, FP64 and precision form side by side
        {"name": "serve_mix", "kind": "serve", "count": 16, "workers": 8, "top": 16384, "shapes": 11},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_lp(rng):
    k = rng.choice([8, 10, 16, 24, 32, 50, 64, rng.randint(5, 64)])
    return k, rng.choice([k // 2, max(2, k // 4), 10, 14])


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "mixed", "sketch", "orthogonalize", "integrate", "form", "serve"])
    if kind == "serve":
        return {"kind": "serve", "count": rng.randint(6, 16), "workers": rng.choice([4, 8]),
                "top": _log_int(rng, 2048, 16384), "shapes": rng.randint(1, 10 ** 6)}
    while True:
        k, p = _draw_lp(rng)
        m = _log_int(rng, 512, 100000 if kind == "solve" else 40000)
        n = _log_int(rng, 256, 20000 if kind in ("solve", "mixed", "sketch", "form") else 3000)
        N = rng.choice([4, 8, 16, 32, 64])
        l = k + p
        L = l * N
        if min(m, n) < 4 * l or m * (n + L) > 1.5e9:
            continue
        if 2.0 * m * n * L + 2.0 * m * L * L + 60 * 4.0 * m * L * l > MAX_FLOPS:
            continue
        break
    spectrum = rng.choice(["power", "noise", "steep"])
    layout = rng.choice(["row", "row", "col"])
    if kind in ("solve", "mixed"):
        integrator = rng.choice(["kn", "rb_kn", "rb_gramian_kn", "rb_gramian_kn"])
        if kind == "mixed":
            integrator, layout = rng.choice(["kn", "rb_gramian_kn"]), "row"
        return _pure(_solve("", m, n, k, p, N, integrator, rng.choice(["svd", "gramian", "rb_gramian", "cb_gramian"]),
                            rng.choice([1e-4, 1e-5]), spectrum, layout, rng.random() < 0.5,
                            rng.choice([2, 3]) if kind == "mixed" else 0))
    stage, tol = "", 0.0
    if kind == "integrate":
        stage = rng.choice(["kn", "rb_kn", "rb_gramian_kn", "rb_gramian_kn", "rb_wy", "rb_gramian_wy"])
        spectrum = "noise" if stage.endswith("wy") else spectrum
        tol = 1e-3 if stage.endswith("wy") else rng.choice([1e-4, 1e-5])
    elif kind == "form":
        stage = rng.choice(["svd", "gramian", "rb_gramian", "cb_gramian"])
    exponent = 1 if kind == "sketch" and rng.random() < 0.25 and 6.0 * m * n * L < MAX_FLOPS else 0
    return _pure(_stage("", kind, m, n, k, p, N, stage, tol, spectrum, layout, exponent))


def _pure(case):
    return {key: v for key, v in case.items() if key != "name"}


# ----------------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------------
def _randn(g, *shape, dtype=torch.float64):
    return torch.randn(*shape, generator=g, dtype=dtype, device="cuda")


def _orthonormal(g, rows, cols):
    return torch.linalg.qr(_randn(g, rows, cols))[0]


def _matrix(g, m, n, spectrum, layout="row", dtype=torch.float64, alpha=1.0, rank=256):
    """U diag(sigma) V' with orthonormal U, V from Gaussians: sigma_j = j^-alpha, a steep 10^(-6 j / 200)
    over a 1e-8 noise floor, or exp(-j / 30) with 1e-4 noise."""
    r = min(m, n, rank)
    j = torch.arange(r, dtype=torch.float64, device="cuda")
    if spectrum == "power":
        sigma, noise = (j + 1) ** -alpha, 1e-5
    elif spectrum == "steep":
        sigma, noise = 10.0 ** (-6.0 * j / 199), 1e-8
    else:
        sigma, noise = torch.exp(-(j + 1) / 30.0), 1e-4
    us = _orthonormal(g, m, r) * sigma
    v = _orthonormal(g, n, r)
    if layout == "col":
        us, v, m, n = v, us, n, m
    a = torch.empty(m, n, dtype=dtype, device="cuda")
    for r0 in range(0, m, 8192):
        r1 = min(m, r0 + 8192)
        a[r0:r1] = us[r0:r1] @ v.T
        a[r0:r1] += noise * _randn(g, r1 - r0, n, dtype=dtype)
    return a.t() if layout == "col" else a


def _params(case):
    return (isvd.Parameters(device="cuda:0").setSize(case["m"], case["n"]).setRank(case["k"])
            .setOverRank(case["p"]).setNumSketch(case["N"]).sync())


def _bases(y, l, N):
    """The orthonormal bases of the N sketches, side by side."""
    m = y.shape[0]
    q = torch.linalg.qr(y.view(m, N, l).permute(1, 0, 2).contiguous())[0]
    return q.permute(1, 0, 2).reshape(m, N * l).contiguous()


def _prepare_serve(case, seed, g):
    """Requests of the uneven batch's ranges; a third each of FP64, two-part and three-part precision form with
    the parts of A resident, as a service that keeps its matrices holds them."""
    shapes = np.random.default_rng(case["shapes"])      # the sizes belong to the case, the values to the seed
    reqs = []
    for i in range(case["count"]):
        m = int(shapes.integers(512, case["top"] + 1))
        n = int(shapes.integers(256, max(512, case["top"] // 4) + 1))
        k = int(shapes.choice([8, 16, 32, 64]))
        alpha = float(shapes.uniform(0.5, 1.25))
        a = _matrix(g, m, n, "power", dtype=torch.float32, alpha=alpha)
        mixed = (0, 2, 3)[i % 3]
        split = former_split = None
        if mixed:
            split, former_split = isvd.resident_parts(a, mixed)
        reqs.append(isvd.Request(a, k, k // 2, 8, seed=int(seed) + i, integrator="rb_gramian_kn", former="svd",
                                 tol=1e-5, mixed=mixed, split=split, former_split=former_split))
    return {"kind": "serve", "requests": reqs, "server": isvd.Server(workers=case["workers"], budget_bytes=40 << 30)}


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    kind = case["kind"]
    if kind == "serve":
        return _prepare_serve(case, seed, g)
    m, n, k, p, N = (case[key] for key in ("m", "n", "k", "p", "N"))
    l = k + p
    L = l * N
    state = {"kind": kind, "case": case, "seed": int(seed)}
    if kind == "solve":
        a = _matrix(g, m, n, case["spectrum"], case["layout"])
        state["a"] = a
        if case["mixed"]:
            state["split"], state["former_split"] = isvd.resident_parts(a, case["mixed"])
        elif case["omega"]:
            state["omega"] = _randn(g, n, L)
        return state
    prm = state["params"] = _params(case)
    if kind == "sketch":
        state["a"] = _matrix(g, m, n, case["spectrum"], case["layout"])
        state["omega"] = _randn(g, n, L)
        state["stage"] = isvd.GaussianProjectionSketcher(prm, seed, case["exponent"]).setOmega(state["omega"])
        state["q"] = prm.createCollectionQ()
    elif kind == "orthogonalize":
        a = _matrix(g, m, n, case["spectrum"])
        state["y"] = a @ _randn(g, n, L)
        state["stage"] = isvd.RowBlockGramianOrthogonalizer(prm)
    elif kind == "integrate":
        a = _matrix(g, m, n, case["spectrum"])
        state["q"] = _bases(a @ _randn(g, n, L), l, N)
        stage = {"kn": isvd.KolmogorovNagumoIntegrator, "rb_kn": isvd.RowBlockKolmogorovNagumoIntegrator,
                 "rb_gramian_kn": isvd.RowBlockGramianKolmogorovNagumoIntegrator,
                 "rb_wy": isvd.RowBlockWenYinIntegrator, "rb_gramian_wy": isvd.RowBlockGramianWenYinIntegrator}
        state["stage"] = stage[case["stage"]](prm, WY_STEPS if case["stage"].endswith("wy") else 256, case["tol"])
        state["qbar"] = prm.createMatrixQbar()
    else:
        state["a"] = _matrix(g, m, n, case["spectrum"], case["layout"])
        state["qbar"] = torch.linalg.qr(state["a"] @ _randn(g, n, l))[0].contiguous()
        stage = {"svd": isvd.SvdFormer, "gramian": isvd.GramianFormer, "rb_gramian": isvd.RowBlockGramianFormer,
                 "cb_gramian": isvd.ColBlockGramianFormer}
        state["stage"] = stage[case["stage"]](prm)
    state["stage"].initialize()
    return state


# ----------------------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------------------
def _signed(u, *others):
    """Columns with the sign that makes the first row of u positive: singular vectors and bases are defined up to
    it, and a program that compares or stores them picks one."""
    sign = torch.copysign(torch.ones_like(u[0]), u[0])
    return [x * sign for x in (u, *others)]


def run(state):
    kind = state["kind"]
    if kind == "serve":
        srv = state["server"]
        for r in state["requests"]:
            srv.submit(r)
        for r in state["requests"]:
            srv.wait(r)
        # at most 64 outputs: all sigmas and iteration counts side by side, every U and V whole
        return {"s": torch.cat([r.s for r in state["requests"]]),
                "iterations": torch.tensor([int(r.result.iteration) for r in state["requests"]]),
                "uv": [_signed(r.u, r.v) for r in state["requests"]]}
    c = state["case"]
    if kind == "solve":
        if c["mixed"]:
            s, u, v, it = isvd.solve_mixed(state["a"], c["k"], c["p"], c["N"], seed=state["seed"],
                                           integrator=c["integrator"], former=c["former"], tol=c["tol"],
                                           split=state["split"], former_split=state["former_split"])
        else:
            s, u, v, it = isvd.solve(state["a"], c["k"], c["p"], c["N"], omega=state.get("omega"), seed=state["seed"],
                                     integrator=c["integrator"], former=c["former"], tol=c["tol"])
        u, v = _signed(u, v)
        return {"s": s, "u": u, "v": v, "iterations": it}
    stage = state["stage"]
    if kind == "sketch":
        stage(state["a"], state["q"])
        return {"q": state["q"]}
    if kind == "orthogonalize":
        q = state["y"].clone()          # the stage works in place, and the sketch is wanted again
        stage(q)
        return {"q": _signed(q)[0]}
    if kind == "integrate":
        stage(state["q"], state["qbar"])
        return {"qbar": state["qbar"], "iterations": stage.iteration()}
    stage(state["a"], state["qbar"])
    u, v = _signed(stage.matrixU(), stage.matrixV())
    return {"s": stage.vectorS(), "u": u, "v": v}


# ----------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------
def _solve_work(m, n, k, p, N, a_bytes=8):
    """The sketch of all N l columns, the orthogonalizer's Gram matrices and rescale, one step of the integrator
    (its step count depends on the values) and the former's products; A read once, results written once."""
    l = k + p
    L = l * N
    flops = 2.0 * m * n * L + 4.0 * m * L * l + 4.0 * m * L * l + 2.0 * m * n * l + 2.0 * (m + n) * l * k
    return {"bytes": float(a_bytes) * m * n + 8.0 * ((m + n) * k + k), "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "serve":
        shapes = np.random.default_rng(case["shapes"])
        total = {"bytes": 0.0, "flops": 0.0}
        for i in range(case["count"]):
            m = int(shapes.integers(512, case["top"] + 1))
            n = int(shapes.integers(256, max(512, case["top"] // 4) + 1))
            k = int(shapes.choice([8, 16, 32, 64]))
            shapes.uniform(0.5, 1.25)
            w = _solve_work(m, n, k, k // 2, 8, 4)
            total = {key: total[key] + w[key] for key in total}
        return total
    m, n, k, p, N = (case[key] for key in ("m", "n", "k", "p", "N"))
    l = k + p
    L = l * N
    if kind == "solve":
        w = _solve_work(m, n, k, p, N, 2 * case["mixed"] if case["mixed"] else 8)
        if case["omega"] and not case["mixed"]:
            w["bytes"] += 8.0 * n * L
        return w
    if kind == "sketch":
        e = case["exponent"]
        return {"bytes": 8.0 * (m * n + n * L * (1 + (e > 0)) + m * L), "flops": 2.0 * m * n * L * (1 + 2 * e)}
    if kind == "orthogonalize":
        return {"bytes": 16.0 * m * L, "flops": 4.0 * m * L * l}
    if kind == "integrate":
        return {"bytes": 8.0 * (m * L + m * l), "flops": 4.0 * m * L * l}
    return {"bytes": 8.0 * (m * n + m * l + (m + n) * k + k), "flops": 2.0 * m * n * l + 2.0 * (m + n) * l * k}


# ----------------------------------------------------------------------------------------------
# the same in plain 64-bit torch
# ----------------------------------------------------------------------------------------------
def _kn(q, l, N, tol, maxit=256):
    """The Kolmogorov-Nagumo average of the N bases in q (m x N l), starting from the first."""
    qc = q[:, :l].clone()
    eye = torch.eye(l, dtype=q.dtype, device=q.device)
    for _ in range(maxit):
        b = q.T @ qc
        x = (q @ b - qc @ (b.T @ b)) / N
        lam, vec = torch.linalg.eigh(x.T @ x)
        e = torch.sqrt(0.5 + torch.sqrt(0.25 - lam))
        c = (vec * e) @ vec.T
        ci = (vec / e) @ vec.T
        qc = qc @ c + x @ ci
        if not float(torch.linalg.norm(c - eye)) >= tol:
            break
    return qc


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return None
    m, n, k, p, N = (case[key] for key in ("m", "n", "k", "p", "N"))
    l = k + p
    if kind == "solve" and (case["mixed"] or not case["omega"]):
        return None                     # Omega is drawn by the library
    if kind == "solve" and 2.0 * m * n * l * N + 256 * 4.0 * m * l * l * N > 4e13:
        return None                     # too long
    if kind == "integrate" and case["stage"].endswith("wy"):
        return None
    if kind == "orthogonalize":
        return None                     # the order and the mixing of equal eigenvalues are free
    state = prepare(case, seed)
    if kind == "sketch":
        a, om = state["a"], state["omega"]
        q = a @ om
        for _ in range(case["exponent"]):
            q = a @ (a.T @ q)
        return {"q": q}
    if kind == "integrate":
        return {"qbar": _kn(state["q"], l, N, case["tol"]), "iterations": None}
    a = state["a"]
    qbar = state["qbar"] if kind == "form" else _kn(_bases(a @ state["omega"], l, N), l, N, case["tol"])
    s = torch.linalg.svdvals((qbar.T @ a).contiguous())[:k]
    out = {"s": s, "u": None, "v": None}
    return out if kind == "form" else {**out, "iterations": None}
