"""Performance cases: the work a program has this library do, through its public API.

Kinds of case:

* ``refactor``: a program keeps one handle per grid and options, and for every new
  coefficient field enters the operator, factors it and solves (PCG to ``tol``).
  Coefficients and right-hand sides are on the GPU. This is the whole path.
* ``apply``: F u or F^-1 u with a factor that is kept, on vectors on the GPU.
* ``solve``: PCG with a factor that is kept, on vectors on the GPU.
* ``node``: the reference's own operator (node coefficients, not symmetric) from host
  arrays: ``SetupStencil``, ``Factor``, restarted GMRES, result on the host.
* ``serve``: a burst of solve requests of several sizes against resident operators.
* ``schur``: the elimination of one dense block, host arrays in and out.

Sizes, fields and options are those of the benchmark (``bench.py``) and the tests: n
cells per direction up to 128, P = 4, eps 1e-6 (1e-3 and 1e-8 at the ends), Gaussian
random fields, independent lognormal faces and 10^6 contrast blocks; FP64 and mixed
precision; the reference partition where n is 4 * 2^l and the clipped one elsewhere.
"""
import math
import weakref

import numpy as np
import torch

import hifde3d_b200 as hb

DEV = "cuda"


def listed():
    return [
        # the benchmark's step (new coefficients, factor, one solve) in both precisions:
        # the largest grids, where the dense products carry the time
        {"name": "refactor_n128_mixed", "kind": "refactor", "n": 128, "precision": "mixed",
         "field": "grf", "eps": 1e-6, "nrhs": 1, "tol": 1e-10},
        {"name": "refactor_n128_fp64", "kind": "refactor", "n": 128, "precision": "fp64",
         "field": "grf", "eps": 1e-6, "nrhs": 1, "tol": 1e-10},
        # high contrast, tight eps, many right-hand sides in one solve; a grid that is
        # not a power of two (clipped partition)
        {"name": "contrast_n96_64rhs_fp64", "kind": "refactor", "n": 96, "precision": "fp64",
         "field": "contrast", "eps": 1e-8, "nrhs": 64, "tol": 1e-10},
        # the ordinary step: a medium grid inside a nonlinear or time loop
        {"name": "refactor_n64_mixed", "kind": "refactor", "n": 64, "precision": "mixed",
         "field": "grf", "eps": 1e-6, "nrhs": 1, "tol": 1e-10},
        # 13 cells per direction: every level's last cells are cut at the boundary
        {"name": "refactor_n52_fp64", "kind": "refactor", "n": 52, "precision": "fp64",
         "field": "lognormal", "eps": 1e-6, "nrhs": 3, "tol": 1e-10},
        # the smallest: launches and host work count
        {"name": "refactor_n16_fp64", "kind": "refactor", "n": 16, "precision": "fp64",
         "field": "grf", "eps": 1e-6, "nrhs": 1, "tol": 1e-10},
        # the reference's drivers: node coefficients, host arrays, a solve on the host
        {"name": "node_n32_host", "kind": "node", "n": 32, "sigma": 0.5, "eps": 1e-6,
         "tol": 1e-10},
        # one preconditioner application inside somebody's own Krylov loop
        {"name": "inverse_n96_fp64", "kind": "apply", "n": 96, "precision": "fp64",
         "field": "grf", "eps": 1e-6, "nrhs": 1, "inverse": True},
        # F u of a block of vectors (sampling, block methods)
        {"name": "forward_n48_24rhs_fp64", "kind": "apply", "n": 48, "precision": "fp64",
         "field": "lognormal", "eps": 1e-6, "nrhs": 24, "inverse": False},
        # further right-hand sides for an operator that is already factored
        {"name": "solve_n64_mixed", "kind": "solve", "n": 64, "precision": "mixed",
         "field": "grf", "eps": 1e-6, "nrhs": 1, "tol": 1e-10},
        # the serving loop: requests of 1 to 32 right-hand sides, three operators
        {"name": "serve_12_requests", "kind": "serve", "sizes": "32,48,64", "requests": 12,
         "max_nrhs": 32, "precision": "mixed", "tol": 1e-10},
        # the reference's free function on one block
        {"name": "schur_block_731_512", "kind": "schur", "red": 731, "skel": 512},
    ]


def _spread(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _operator(rng, lo, hi):
    """A grid, field, eps and precision of the declared ranges."""
    field = rng.choice(["grf", "grf", "lognormal", "contrast"])
    hi = min(hi, 88) if field == "contrast" else hi  # its decompositions cost more
    return {"n": 4 * max(lo // 4, min(hi // 4, round(_spread(rng, lo, hi) / 4))),
            "precision": rng.choice(["fp64", "mixed"]), "field": field,
            "eps": 1e-8 if field == "contrast" else rng.choice([1e-6, 1e-6, 1e-6, 1e-3])}


def draw(rng):
    kind = rng.choice(["refactor"] * 5 + ["apply"] * 2 + ["solve"] * 2 + ["node", "serve", "schur"])
    if kind == "refactor":
        op = _operator(rng, 12, 112)
        return {"kind": kind, **op, "nrhs": rng.choice([1, 1, 1, 2, 5, 17]), "tol": 1e-10}
    if kind == "apply":
        op = _operator(rng, 12, 88)
        op["precision"] = "fp64"
        return {"kind": kind, **op, "nrhs": round(_spread(rng, 1, 64)),
                "inverse": rng.random() < 0.6}
    if kind == "solve":
        op = _operator(rng, 12, 80)
        return {"kind": kind, **op, "nrhs": round(_spread(rng, 1, 40)), "tol": 1e-10}
    if kind == "node":
        return {"kind": kind, "n": rng.choice([8, 12, 16, 20, 24, 28, 32, 40]),
                "sigma": round(rng.uniform(0.1, 0.5), 3), "eps": 1e-6, "tol": 1e-10}
    if kind == "serve":
        sizes = sorted(rng.sample([24, 32, 40, 48, 52, 64], rng.choice([2, 3])))
        return {"kind": kind, "sizes": ",".join(map(str, sizes)), "requests": rng.randrange(4, 17),
                "max_nrhs": rng.choice([4, 16, 32]), "precision": rng.choice(["fp64", "mixed"]),
                "tol": 1e-10}
    return {"kind": kind, "red": round(_spread(rng, 20, 1500)), "skel": round(_spread(rng, 20, 1000))}


# ---- inputs ------------------------------------------------------------------------
def _generator(seed, device=DEV):
    return torch.Generator(device=device).manual_seed(seed)


def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, dtype=torch.float64, device=gen.device)


def _fields(n, field, seed):
    """Face coefficients ax, ay, az and V as (n+1)^3 tensors indexed [k, j, i] (i fastest)."""
    gen = _generator(seed)
    t = n + 1
    if field == "lognormal":  # independent faces
        ax, ay, az = torch.exp(_normal(gen, 3, t, t, t)).unbind(0)
    elif field == "contrast":  # 8^3 sub-cubes of 10^U(-3, 3), harmonic means at the faces
        v = torch.rand(8, 8, 8, generator=gen, dtype=torch.float64, device=DEV)
        at = torch.clamp(torch.arange(n + 2, device=DEV) * 8 // (n + 1), max=7)
        a = (10.0 ** (6.0 * v - 3.0))[at][:, at][:, :, at]
        c = a[:-1, :-1, :-1]
        ax, ay, az = (2 * c * b / (c + b) for b in (a[:-1, :-1, 1:], a[:-1, 1:, :-1],
                                                     a[1:, :-1, :-1]))
    else:  # Gaussian random field, correlation length 1/16 of the cube, sigma 1
        m = 2 * n
        x = torch.fft.fftfreq(m, d=1.0 / m, device=DEV, dtype=torch.float64) / n
        g = torch.exp(-x * x / (2 * 0.125 ** 2))
        cov = g[:, None, None] * g[None, :, None] * g[None, None, :]
        spec = torch.sqrt(torch.clamp(torch.fft.fftn(cov).real, min=0.0))
        f = torch.fft.ifftn(torch.fft.fftn(_normal(gen, m, m, m)) * spec).real
        f = torch.exp(f / f.std())
        ev = (2 * torch.arange(t, device=DEV)) % m
        od = (ev + 1) % m
        ax, ay, az = f[ev][:, ev][:, :, od], f[ev][:, od][:, :, ev], f[od][:, ev][:, :, ev]
    V = torch.full((t, t, t), 1e-2 if field == "contrast" else 0.0, dtype=torch.float64, device=DEV)
    return [c.contiguous() for c in (ax, ay, az, V)]


def _vectors(n, nrhs, seed, device=DEV):
    """(nrhs, n, n, n) vectors indexed [c, k, j, i], N(0, 1) on the DOFs, zero on the
    index-0 planes: each is one column of the library's column-major layout."""
    u = _normal(_generator(seed + 1, device), nrhs, n, n, n)
    u[:, 0], u[:, :, 0], u[:, :, :, 0] = 0, 0, 0
    return u


def _partition(n):
    return hb.PARTITION_REFERENCE if n >= 4 and n & (n - 1) == 0 else hb.PARTITION_CLIPPED


def _precision(case):
    return hb.PRECISION_MIXED if case["precision"] == "mixed" else hb.PRECISION_FP64


def _new_factor(case, stream):
    f = hb.HIFFactor(case["n"] - 1, 4, case["eps"], _partition(case["n"]))
    f.set_option(hb.OPT_PRECISION, _precision(case))
    hb.set_stream(f, stream.cuda_stream)
    return f


def _enter_operator(f, n, coef):
    hb.SetupStencilFacesDevice(f, n - 1, 1.0 / n, *[c.data_ptr() for c in coef])


# a program's handle for one grid and set of options, shared by its successive
# coefficient fields while any of them is in use
_handles = weakref.WeakValueDictionary()


class _Handle:
    def __init__(self, case):
        self.stream = torch.cuda.Stream()
        self.f = _new_factor(case, self.stream)


def _kept_handle(case):
    key = (case["n"], case["precision"], case["eps"])
    h = _handles.get(key)
    if h is None:
        h = _handles[key] = _Handle(case)
    return h


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "refactor":
        n = case["n"]
        s["handle"] = _kept_handle(case)
        s["coef"] = _fields(n, case["field"], seed)
        s["b"] = _vectors(n, case["nrhs"], seed)
        s["x"] = torch.zeros_like(s["b"])
    elif kind in ("apply", "solve"):
        n = case["n"]
        h = s["handle"] = _Handle(case)
        coef = _fields(n, case["field"], seed)
        s["b"] = _vectors(n, case["nrhs"], seed)
        s["x"] = torch.zeros_like(s["b"])
        torch.cuda.synchronize()
        _enter_operator(h.f, n, coef)
        h.f.Factor()
        h.f.trim()
    elif kind == "node":
        n = case["n"]
        gen = _generator(seed, "cpu")
        a = torch.exp(case["sigma"] * _normal(gen, n + 1, n + 1, n + 1))
        v = 0.1 * torch.rand(n + 1, n + 1, n + 1, generator=gen, dtype=torch.float64)
        # (N+2)^3 tensors indexed [i, j, k], i fastest in memory
        s["A"], s["V"] = a.numpy().T, v.numpy().T
        s["b"] = _vectors(n, 1, seed, "cpu").reshape(-1).numpy()
        s["f"] = hb.HIFFactor(n - 1, 4, case["eps"], _partition(n))
    elif kind == "serve":
        sizes = [int(t) for t in case["sizes"].split(",")]
        srv = s["server"] = hb.Server(budget_bytes=40 << 30, max_active_solves=64, factor_workers=2)
        ids = []
        for q, n in enumerate(sizes):
            # indexed [i, j, k] on the host
            coef = [c.cpu().numpy().T for c in _fields(n, "lognormal", seed + 17 * q)]
            ids.append(srv.submit_factor(q, n - 1, *coef, eps=1e-6, precision=_precision(case),
                                         partition=hb.PARTITION_CLIPPED))
        for i in ids:
            r = srv.wait(i)
            if r["status"] != hb.HIF_OK:
                raise RuntimeError("serving operator: %s" % r)
        s["requests"] = []
        for q in range(case["requests"]):
            op = q % len(sizes)
            nrhs = 1 + (q * 7919) % case["max_nrhs"]
            b = _vectors(sizes[op], nrhs, seed + 1000 + q)
            s["requests"].append((op, b.reshape(nrhs, -1).cpu().numpy().T))
    else:  # a diagonally dominant M-matrix, as the blocks of the factorization are
        m = case["red"] + case["skel"]
        gen = _generator(seed, "cpu")
        i = torch.arange(m, dtype=torch.float64)
        w = torch.exp(-(i[:, None] - i[None, :]).abs() / 16.0)
        w = w * torch.rand(m, m, generator=gen, dtype=torch.float64)
        w = torch.triu(w, 1)
        w = w + w.T
        M = torch.diag(w.sum(1) * 1.01) - w
        p = torch.randperm(m, generator=gen)
        s["M"] = np.asfortranarray(M.numpy())
        s["red"], s["skel"] = p[:case["red"]].numpy(), p[case["red"]:].numpy()
    torch.cuda.synchronize()
    return s


# ---- one pass ----------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "refactor":
        f, n, nrhs = s["handle"].f, case["n"], case["nrhs"]
        _enter_operator(f, n, s["coef"])
        f.Factor()
        f.solve_pcg_device(s["b"].data_ptr(), s["x"].data_ptr(), nrhs, n ** 3, case["tol"], 200)
        return s["x"]
    if kind == "apply":
        h = s["handle"]
        with torch.cuda.stream(h.stream):
            s["x"].copy_(s["b"])
        h.f.apply_device(s["x"].data_ptr(), case["nrhs"], case["n"] ** 3, case["inverse"])
        return s["x"]
    if kind == "solve":
        s["handle"].f.solve_pcg_device(s["b"].data_ptr(), s["x"].data_ptr(), case["nrhs"],
                                       case["n"] ** 3, case["tol"], 200)
        return s["x"]
    if kind == "node":
        f, n = s["f"], case["n"]
        hb.SetupStencil(f, n - 1, 1.0 / n, s["A"], s["V"])
        f.Initialize()
        f.Factor()
        return f.solve_gmres(s["b"], tol=case["tol"], maxit=200)[0]
    if kind == "serve":
        srv = s["server"]
        ids = [srv.submit_solve(op, b, tol=case["tol"]) for op, b in s["requests"]]
        done = [srv.wait(i) for i in ids]
        for r in done:
            if r["status"] != hb.HIF_OK:
                raise RuntimeError("serving request: %s" % r["error"])
        return [r["x"] for r in done]
    return list(hb.Schur(s["M"], s["red"], s["skel"]))


# ---- what a pass cannot do without ---------------------------------------------------
def _factor_work(n, eps):
    """(entries of the factor, flops of the eliminations) of an n^3 grid: cells of width
    w = 4, 8, ...; a face of width w keeps about min((w - 1)^2, c w) of its unknowns."""
    c = {1e-3: 5.0, 1e-6: 9.0, 1e-8: 11.0}.get(eps, 9.0)
    entries = flops = 0.0
    kept, w = 0.0, 4
    while True:
        top = w >= n
        if w == 4:
            r, face = 27.0, 9.0
        else:
            h = w // 2 - 1
            r, face = 12 * kept + 6 * h + 1, 4 * kept + 4 * h + 1
        cells = max(1.0, (n / w) ** 3)
        skel = 0.0 if top else 6 * face
        r = r if not top else 12 * kept + 6 * (w // 2 - 1) + 1
        entries += cells * (r * r + r * skel)
        flops += cells * (2 * r ** 3 / 3 + r * r * skel + r * skel * skel)
        if top:
            return entries, flops
        kept = min(face, c * w)
        gone = face - kept
        faces = 3 * cells
        entries += faces * (gone * gone + 2 * gone * kept)
        # the interpolative decomposition of a face's columns against its interactions
        flops += faces * (2 * 10 * face ** 2 * kept + 2 * gone ** 3 / 3 + 2 * gone * gone * kept
                          + gone * kept * kept)
        w *= 2


def work(case):
    kind = case["kind"]
    if kind == "schur":
        r, k = case["red"], case["skel"]
        return {"bytes": 8.0 * ((r + k) ** 2 + 2 * r * r + r * k + k * k),
                "flops": 2.0 * r ** 3 + 2.0 * r * r * k + 2.0 * r * k * k}
    if kind == "serve":
        by = fl = 0.0
        sizes = [int(t) for t in case["sizes"].split(",")]
        for q in range(case["requests"]):
            n, nrhs = sizes[q % len(sizes)], 1 + (q * 7919) % case["max_nrhs"]
            e, _ = _factor_work(n, 1e-6)
            by += 2 * 8.0 * n ** 3 * nrhs
            fl += 4 * 2 * e * nrhs
        return {"bytes": by + 8.0 * sum(4 * _factor_work(n, 1e-6)[0] for n in sizes), "flops": fl}
    n = case["n"]
    entries, flops = _factor_work(n, case["eps"])
    if kind == "node":
        return {"bytes": 8.0 * (2 * (n + 1) ** 3 + 2 * n ** 3 + 11 * entries), "flops": flops}
    vec = 2 * 8.0 * n ** 3 * case["nrhs"]
    if kind == "apply":
        return {"bytes": vec + 8.0 * entries, "flops": 2 * entries * case["nrhs"]}
    # PCG: about four applications of the preconditioner
    by, fl = vec + 4 * 8.0 * entries, 4 * 2 * entries * case["nrhs"]
    if kind == "refactor":
        by, fl = by + 8.0 * (4 * (n + 1) ** 3 + entries), fl + flops
    return {"bytes": by, "flops": fl}


# ---- the same in 64 bits without the library ---------------------------------------
def _shift(x, dim, step):
    """x moved by one along a grid axis, zero where there is no neighbour."""
    y = torch.zeros_like(x)
    n = x.shape[dim]
    if step > 0:
        y.narrow(dim, 0, n - 1).copy_(x.narrow(dim, 1, n - 1))
    else:
        y.narrow(dim, 1, n - 1).copy_(x.narrow(dim, 0, n - 1))
    return y


def _cg(diag, off, b, steps):
    """Conjugate gradients with the diagonal as preconditioner for
    (A x) = diag x - sum over axes of the two neighbours' terms; off[d] couples a node
    with the next one along dimension d of b's grid. Ends when the residual no longer falls."""
    def A(x):
        y = diag * x
        for d in range(3):
            y -= off[d] * _shift(x, d - 3, 1)
            y -= _shift(off[d] * x, d - 3, -1)
        return y

    def dot(u, v):
        return (u * v).sum(dim=(-3, -2, -1), keepdim=True)

    x = torch.zeros_like(b)
    for _ in range(2):  # the second run corrects what rounding left of the first
        r = b - A(x)
        z = r / diag
        p, rz = z.clone(), dot(r, z)
        stop = 1e-32 * dot(b, b / diag)
        for it in range(steps):
            q = A(p)
            a = rz / torch.clamp(dot(p, q), min=1e-300)
            x = x + a * p
            r = r - a * q
            z = r / diag
            new = dot(r, z)
            if it % 25 == 24 and bool((new <= stop).all()):
                break
            p = z + (new / torch.clamp(rz, min=1e-300)) * p
            rz = new
    return x


def _face_system(n, field, seed):
    ax, ay, az, V = _fields(n, field, seed)
    hh = (1.0 / n) ** 2
    c = slice(1, n)  # DOFs 1 .. n - 1
    m = slice(0, n - 1)
    xp, yp, zp = ax[c, c, c], ay[c, c, c], az[c, c, c]
    diag = (ax[c, c, m] + xp + ay[c, m, c] + yp + az[m, c, c] + zp) / hh + V[c, c, c]
    off = []
    for d, a in ((0, zp), (1, yp), (2, xp)):  # b's dimensions are [k, j, i]
        a = (a / hh).clone()
        a.narrow(d, n - 2, 1).zero_()  # the last plane has no next DOF
        off.append(a)
    return diag, off


def _solve_faces(n, field, seed, b):
    diag, off = _face_system(n, field, seed)
    out = torch.zeros_like(b)
    out[:, 1:, 1:, 1:] = _cg(diag, off, b[:, 1:, 1:, 1:], 6000)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("refactor", "solve"):
        if case["field"] == "contrast":
            return None  # thousands of plain CG steps at a contrast of 10^6
        return _solve_faces(case["n"], case["field"], seed, _vectors(case["n"], case["nrhs"], seed))
    if kind == "serve":
        sizes = [int(t) for t in case["sizes"].split(",")]
        out = []
        for q in range(case["requests"]):
            op = q % len(sizes)
            n, nrhs = sizes[op], 1 + (q * 7919) % case["max_nrhs"]
            x = _solve_faces(n, "lognormal", seed + 17 * op, _vectors(n, nrhs, seed + 1000 + q))
            out.append(x.reshape(nrhs, -1).cpu().numpy().T)
        return out
    if kind == "node":
        # A(p, q) = -a(q) / h^2: with y = sqrt(a) x the system is symmetric
        s = prepare(case, seed)
        n = case["n"]
        a = torch.from_numpy(np.ascontiguousarray(s["A"].T))
        V = torch.from_numpy(np.ascontiguousarray(s["V"].T))
        hh = (1.0 / n) ** 2
        c, m, p = slice(1, n), slice(0, n - 1), slice(2, n + 1)
        diag = V[c, c, c] + (a[c, c, m] + a[c, c, p] + a[c, m, c] + a[c, p, c] + a[m, c, c]
                             + a[p, c, c]) / hh
        root = torch.sqrt(a[c, c, c])
        off = []
        for d in range(3):
            o = root * _shift(root, d, 1) / hh
            o.narrow(d, n - 2, 1).zero_()
            off.append(o)
        b = torch.from_numpy(s["b"]).reshape(1, n, n, n)[:, 1:, 1:, 1:]
        x = torch.zeros(1, n, n, n, dtype=torch.float64)
        x[:, 1:, 1:, 1:] = _cg(diag, off, root * b, 3000) / root
        return x.reshape(-1).numpy()
    if kind == "schur":
        s = prepare(case, seed)
        M, r, k = torch.from_numpy(s["M"]), s["red"], s["skel"]
        a22 = M[r][:, r]
        inv = torch.linalg.inv(a22)
        X = torch.linalg.solve(a22, M[r][:, k])
        return [a22.numpy(), inv.numpy(), X.numpy(), (-M[k][:, r] @ X).numpy()]
    return None  # F u and F^-1 u of the library's own approximate factor
