"""The work that users of oocdag_gb300 have it do, as cases that can be timed and checked.

Matrices are column-major: row j of a torch tensor holds column j, so a matrix's lower
triangle is the tensor's upper one.  Only that triangle is given the system's values; the
other one is left as the random fill made it, as the library neither reads nor writes it.
One handle (and one server) per process, as a user's program keeps them.
"""
import math

import numpy as np
import torch

import oocdag_gb300 as ooc
from oocdag_gb300 import offload
from oocdag_gb300.server import Server

DEV = "cuda:0"
F64, F32 = torch.float64, torch.float32


def listed():
    return [
        # One step of a tiled factorization through the tile-offload calls (potrf, trsm, syrk,
        # gemm on one tile each), the way a host-side task runtime drives them: the smallest
        # calls, each of which waits for its own work.
        {"name": "tile_256", "kind": "tile", "nb": 256},
        # FP64 in core on a matrix that is already on the device: a small odd order ...
        {"name": "dpotrf_700", "kind": "dpotrf", "n": 700, "nb": 128, "pad": 0, "host": False, "share": 1.0},
        # ... and the in-core configuration of the benchmark (n = 4096, nb = 256).
        {"name": "dpotrf_4096", "kind": "dpotrf", "n": 4096, "nb": 256, "pad": 0, "host": False, "share": 1.0},
        # FP64 out of core: a page-locked host matrix of ragged order through a device budget
        # of about half of it, several left-looking panels.
        {"name": "dpotrf_host_8200", "kind": "dpotrf", "n": 8200, "nb": 512, "pad": 0, "host": True, "share": 0.55},
        # FP32 Cholesky in place, an odd order with a padded leading dimension.
        {"name": "spotrf_6001", "kind": "spotrf", "n": 6001, "nb": 256, "pad": 3},
        # The benchmark's mixed-precision solve: split-BF16 factor and FP64 refinement of a
        # device matrix at n = 65536, one right-hand side (the largest).
        {"name": "solve_65536", "kind": "solve", "n": 65536, "nb": 512, "prec": "bf16x3", "nrhs": 1, "delta": 0.1, "host": False},
        # The same from page-locked host memory and back to it, sixteen right-hand sides.
        {"name": "solve_host_16384", "kind": "solve", "n": 16384, "nb": 512, "prec": "bf16x3", "nrhs": 16, "delta": 0.01, "host": True},
        # Repeat solves with a factor that stays on the device: a fresh right-hand side.
        {"name": "resident_20000", "kind": "resident", "n": 20000, "nb": 512, "prec": "bf16x3", "nrhs": 1, "delta": 0.1},
        # Thousands of small uneven systems in one call, in both types.
        {"name": "batched_f32", "kind": "batched", "prec": "fp32", "count": 4000, "lo": 16, "hi": 512},
        {"name": "batched_f64", "kind": "batched", "prec": "fp64", "count": 1200, "lo": 16, "hi": 512},
        # The check solve after a factorization: dpotrs with the factor dpotrf left on the device.
        {"name": "dpotrs_8192", "kind": "dpotrs", "n": 8192, "nb": 512, "nrhs": 4, "host": False},
        # A burst of mixed requests to the serving loop, small ones batched, larger ones on
        # the pipelines; answers are collected as they complete.
        {"name": "serve_32", "kind": "serve", "count": 32, "lo": 64, "hi": 4096, "nb": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tile", "dpotrf", "dpotrf_host", "spotrf", "solve", "solve_host", "resident", "batched", "dpotrs", "serve"])
    nb = rng.choice([128, 256, 512])
    if kind == "tile":
        return {"kind": "tile", "nb": _log(rng, 60, 1024)}
    if kind == "dpotrf":
        return {"kind": "dpotrf", "n": _log(rng, 300, 6000), "nb": nb, "pad": rng.choice([0, 0, 1, 6]), "host": False, "share": 1.0}
    if kind == "dpotrf_host":
        return {"kind": "dpotrf", "n": _log(rng, 2500, 9000), "nb": nb, "pad": 0, "host": True, "share": round(rng.uniform(0.4, 1.3), 2)}
    if kind == "spotrf":
        return {"kind": "spotrf", "n": _log(rng, 600, 16000), "nb": nb, "pad": rng.choice([0, 0, 1, 4])}
    if kind == "solve":
        n = _log(rng, 1000, 40000)  # (at small orders the smallest margin would not be definite for every seed)
        return {"kind": "solve", "n": n, "nb": rng.choice([256, 512]), "prec": rng.choice(["bf16x3", "bf16x3", "fp32"]),
                "nrhs": rng.choice([1, 1, 4, 16]), "delta": rng.choice([1.0, 0.1, 0.01 if n >= 8000 else 0.3]), "host": False}
    if kind == "solve_host":
        return {"kind": "solve", "n": _log(rng, 2000, 16384), "nb": 512, "prec": "bf16x3", "nrhs": rng.choice([1, 16]), "delta": 0.1, "host": True}
    if kind == "resident":
        prec = rng.choice(["bf16x3", "bf16x3", "fp32", "fp64"])
        return {"kind": "resident", "n": _log(rng, 1000, 6000 if prec == "fp64" else 30000), "nb": rng.choice([256, 512]), "prec": prec,
                "nrhs": rng.choice([1, 1, 2, 5, 16]), "delta": 0.1}
    if kind == "batched":
        lo, hi = rng.choice([(16, 512), (16, 64), (64, 200), (200, 512)])
        return {"kind": "batched", "prec": rng.choice(["fp32", "fp64"]), "count": _log(rng, 150, 4000), "lo": lo, "hi": hi}
    if kind == "dpotrs":
        return {"kind": "dpotrs", "n": _log(rng, 800, 9000), "nb": nb, "nrhs": rng.choice([1, 1, 3, 8, 16]), "host": rng.random() < 0.4}
    return {"kind": "serve", "count": rng.randint(6, 40), "lo": 64, "hi": _log(rng, 600, 8192), "nb": 512}


# ---- what a user's program has in hand ------------------------------------------------
_kept = {}


def _handle(keep_a=False):
    if ("handle", keep_a) not in _kept:
        h = ooc.Handle(0)
        if keep_a:
            h.set_option(ooc.OPT_KEEP_A, 1)
        _kept["handle", keep_a] = h
    return _kept["handle", keep_a]


def _server(nb):
    if ("server", nb) not in _kept:
        _kept["server", nb] = Server(workers=4, nb=nb, prec="bf16x3", batch_window_ms=0.5, hbm_budget=24 << 30)
    return _kept["server", nb]


def _rng(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _uniform(n, ld, g, diag, dtype=F64):
    """A symmetric matrix with entries uniform in [-1/2, 1/2) and `diag` added to its diagonal."""
    A = torch.empty(n, ld, dtype=dtype, device=DEV).uniform_(-0.5, 0.5, generator=g)
    A[:, :n].diagonal().add_(diag)
    return A


def _alpha(case):
    return 0.5774 * math.sqrt(case["n"]) * (1.0 + case["delta"])


def _pinned(T):
    H = torch.empty(T.shape, dtype=T.dtype, pin_memory=True)
    H.copy_(T)
    return H


def _budget(case):
    bb = -(-case["n"] // case["nb"])
    tiles = max(5 * bb, int(case["share"] * bb * (bb + 1) / 2) + 2 * bb)
    return tiles * case["nb"] ** 2 * 8


def _orders(case):
    """The systems' orders (the case's own; the seed makes their values) and their offsets."""
    r = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    ns = r.integers(case["lo"], case["hi"] + 1, case["count"])
    return ns, np.concatenate([[0], np.cumsum(ns * ns)[:-1]]), np.concatenate([[0], np.cumsum(ns)[:-1]])


def _requests(case, seed):
    """Orders log-uniform in [lo, hi], with the matrix and right-hand-side seed of each."""
    r = np.random.default_rng([case["count"], case["hi"]])
    ns = np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"])).astype(int)
    return [(int(n), 100000 * seed + 2 * i + 1, 100000 * seed + 2 * i + 2) for i, n in enumerate(ns)]


def _inputs(case, seed):
    """The inputs alone, from the seed (all on the device)."""
    g, kind = _rng(seed), case["kind"]
    if kind == "tile":
        nb = case["nb"]
        return {"A": _uniform(nb, nb, g, nb), "rest": [_uniform(nb, nb, g, 0) for _ in range(4)]}
    if kind in ("dpotrf", "spotrf"):
        n = case["n"]
        return {"A": _uniform(n, n + case["pad"], g, n if kind == "dpotrf" else math.sqrt(n), F64 if kind == "dpotrf" else F32)}
    if kind in ("solve", "resident"):
        A = _uniform(case["n"], case["n"], g, _alpha(case))
        return {"A": A, "B": torch.randn(case["nrhs"], case["n"], dtype=F64, device=DEV, generator=g)}
    if kind == "dpotrs":  # a factor: unit-size off-diagonal part below a dominant diagonal
        n = case["n"]
        return {"L": _uniform(n, n, g, math.sqrt(n)), "B": torch.randn(case["nrhs"], n, dtype=F64, device=DEV, generator=g)}
    if kind == "batched":
        ns, ao, bo = _orders(case)
        dt = F32 if case["prec"] == "fp32" else F64
        A = torch.empty(int(np.sum(ns * ns)), dtype=dt, device=DEV)
        for n, o in zip(ns.tolist(), ao.tolist()):
            M = torch.randn(n, n, dtype=dt, device=DEV, generator=g)
            V = A[o : o + n * n].view(n, n)
            torch.mm(M, M.T, out=V)
            V.div_(n).diagonal().add_(1.0)
        return {"A": A, "B": torch.randn(int(ns.sum()), dtype=dt, device=DEV, generator=g)}
    raise ValueError(kind)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "serve":
        return {**s, "server": _server(case["nb"]), "requests": _requests(case, seed), "seed": seed}
    s.update(_inputs(case, seed))
    if kind == "tile":
        offload.init(0)
        s["work"] = [torch.empty_like(s["A"]) for _ in range(4)]
    elif kind in ("dpotrf", "spotrf"):
        s["handle"] = _handle()
        if case.get("host"):
            s["A"], s["work"] = _pinned(s["A"]), torch.empty(s["A"].shape, dtype=F64, pin_memory=True)
        else:
            s["work"] = torch.empty_like(s["A"])
    elif kind == "solve":
        s["handle"] = _handle(case["host"])
        s["X"] = torch.empty_like(s["B"])
        if case["host"]:
            s["A"], s["Bh"], s["Xh"] = _pinned(s["A"]), _pinned(s["B"]), torch.empty(s["B"].shape, dtype=F64, pin_memory=True)
    elif kind == "resident":
        s["handle"] = _handle()
        s["F"] = s["handle"].factor(s["A"], case["n"], case["n"], case["nb"], case["prec"])
        s["X"] = torch.empty_like(s["B"])
    elif kind == "dpotrs":
        s["handle"], s["X"] = _handle(), torch.empty_like(s["B"])
        if case["host"]:
            s["L"] = _pinned(s["L"])
    elif kind == "batched":
        s["handle"], s["orders"] = _handle(), [v.tolist() for v in _orders(case)]
        s["WA"], s["WB"] = torch.empty_like(s["A"]), torch.empty_like(s["B"])
    return s


# ---- one pass -------------------------------------------------------------------------
def run(s):
    return _RUN[s["case"]["kind"]](s, s["case"])


def _run_tile(s, c):
    nb = c["nb"]
    L, B, C, D = s["work"]
    for src, dst in zip([s["A"], *s["rest"][:3]], s["work"]):
        offload.dcopy(nb * nb, src, 1, dst, 1)
    info = offload.dpotrf("L", nb, L, nb)
    offload.dtrsm("R", "L", "T", "N", nb, nb, 1.0, L, nb, B, nb)
    offload.dsyrk("L", "N", nb, nb, -1.0, B, nb, 1.0, C, nb)
    offload.dgemm("N", "T", nb, nb, nb, -1.0, s["rest"][3], nb, B, nb, 1.0, D, nb)
    return {"info": info, "L": L, "B": B, "C": C, "D": D}


def _run_dpotrf(s, c):
    s["work"].copy_(s["A"])  # the factorization is in place
    r = s["handle"].dpotrf_L(s["work"], c["n"], c["n"] + c["pad"], c["nb"], _budget(c))
    return {"info": r.info, "L": s["work"]}


def _run_spotrf(s, c):
    s["work"].copy_(s["A"])
    r = s["handle"].spotrf_L(s["work"], c["n"], c["n"] + c["pad"], c["nb"])
    return {"info": r.info, "L": s["work"]}


def _run_solve(s, c):
    n = c["n"]
    with s["handle"].factor(s["A"], n, n, c["nb"], c["prec"]) as F:
        if c["host"]:
            s["B"].copy_(s["Bh"], non_blocking=True)
        F.refine(s["A"], n, s["B"], n, s["X"], n, c["nrhs"], 1e-14)
        if c["host"]:
            s["Xh"].copy_(s["X"])
    return {"info": F.info, "X": s["Xh"] if c["host"] else s["X"]}


def _run_resident(s, c):
    n = c["n"]
    if c["prec"] == "fp64":
        s["X"].copy_(s["B"])
        s["F"].solve(s["X"], n, c["nrhs"])
    else:
        s["F"].refine(s["A"], n, s["B"], n, s["X"], n, c["nrhs"], 1e-14)
    return {"X": s["X"]}


def _run_dpotrs(s, c):
    n = c["n"]
    s["X"].copy_(s["B"])
    s["handle"].dpotrs_L(s["L"], n, n, c["nb"], s["X"], n, c["nrhs"])
    return {"X": s["X"]}


def _run_batched(s, c):
    s["WA"].copy_(s["A"])
    s["WB"].copy_(s["B"])
    info, _ = s["handle"].batched_posv(c["prec"], *s["orders"], s["WA"], s["WB"])
    return {"info": np.array(info), "L": s["WA"], "X": s["WB"]}


def _run_serve(s, c):
    S = s["server"]
    ids = [S.submit(n, a, b, key=100000 * s["seed"] + i, keep_solution=True) for i, (n, a, b) in enumerate(s["requests"])]
    done = {}
    while len(done) < len(ids):
        for d in S.poll(wait_ms=1000):
            done[d["id"]] = d
    xs = [S.solution(i, n) for i, (n, _, _) in zip(ids, s["requests"])]
    return {"status": np.array([[done[i]["status"], done[i]["info"]] for i in ids]), "X": np.concatenate(xs)}


_RUN = {"tile": _run_tile, "dpotrf": _run_dpotrf, "spotrf": _run_spotrf, "solve": _run_solve, "resident": _run_resident,
        "dpotrs": _run_dpotrs, "batched": _run_batched, "serve": _run_serve}


# ---- what a pass cannot do without ----------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "tile":
        nb = case["nb"]
        return {"bytes": 8 * nb * nb * 8.0, "flops": nb**3 / 3 + nb**3 + nb**3 + 2.0 * nb**3}
    if kind in ("dpotrf", "spotrf"):  # the lower triangle in and out, and the copy that restores it
        n, w = case["n"], 8 if kind == "dpotrf" else 4
        return {"bytes": (n * (n + 1.0) + 2.0 * n * n) * w, "flops": n**3 / 3.0}
    if kind in ("solve", "resident"):
        n, r = case["n"], case["nrhs"]
        tri = n * (n + 1) / 2.0
        if kind == "solve":
            return {"bytes": 8 * tri + 4 * tri + 16.0 * n * r, "flops": n**3 / 3.0 + 4.0 * n * n * r}
        return {"bytes": (8 if case["prec"] == "fp64" else 8 + 4) * tri + 16.0 * n * r, "flops": (2.0 if case["prec"] == "fp64" else 4.0) * n * n * r}
    if kind == "dpotrs":
        n, r = case["n"], case["nrhs"]
        return {"bytes": 8 * n * (n + 1) / 2.0 + 16.0 * n * r, "flops": 2.0 * n * n * r}
    if kind == "batched":  # expected over the orders' distribution
        ns, w = np.arange(case["lo"], case["hi"] + 1, dtype=float), 4 if case["prec"] == "fp32" else 8
        return {"bytes": case["count"] * float(np.mean(ns * (ns + 1) + 2 * ns * ns + 4 * ns)) * w, "flops": case["count"] * float(np.mean(ns**3 / 3 + 2 * ns * ns))}
    u = np.exp(np.linspace(math.log(case["lo"]), math.log(case["hi"]), 513))
    return {"bytes": case["count"] * float(np.mean(4 * u * u)), "flops": case["count"] * float(np.mean(u**3 / 3 + 4 * u * u))}


# ---- the same in 64 bits, by plain torch ------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return {"status": None, "X": np.concatenate([_serve_exact(*q) for q in _requests(case, seed)])}
    v = _inputs(case, seed)
    if kind == "tile":
        L = _factor(v["A"], case["nb"])
        B = torch.linalg.solve_triangular(L.triu().mT, v["rest"][0], upper=False, left=True)
        C = v["rest"][1].tril(-1) + (v["rest"][1] - B.mT @ B).triu()
        return {"info": None, "L": L, "B": B, "C": C, "D": v["rest"][2] - B.mT @ v["rest"][3]}
    if kind in ("dpotrf", "spotrf"):
        return {"info": None, "L": _factor(v["A"].double(), case["n"])}
    if kind in ("solve", "resident"):
        return {"info": None, "X": _refined(v["A"], v["B"])}
    if kind == "dpotrs":
        U = v["L"].triu()
        return {"X": torch.linalg.solve_triangular(U, torch.linalg.solve_triangular(U.mT, v["B"].mT, upper=False), upper=True).mT}
    out, xs = torch.empty_like(v["A"], dtype=F64), []
    for n, a, b in zip(*[x.tolist() for x in _orders(case)]):
        V = v["A"][a : a + n * n].view(n, n).double()
        L = _factor(V, n)
        out[a : a + n * n].view(n, n).copy_(L)
        xs.append(torch.cholesky_solve(v["B"][b : b + n].double()[:, None], L.triu(), upper=True)[:, 0])
    return {"info": None, "L": out, "X": torch.cat(xs)}


def _factor(A, n):
    """A with its lower triangle (the tensor's upper one) replaced by the Cholesky factor."""
    out = A.clone()
    out[:, :n] = torch.linalg.cholesky(A[:, :n], upper=True).triu() + A[:, :n].tril(-1)
    return out


def _refined(A, B):
    """A^{-1} B in 64 bits: a 32-bit factor and refinement with 64-bit residuals."""
    n = A.shape[0]
    U = torch.linalg.cholesky(A.float(), upper=True).triu_()
    X = torch.zeros_like(B)
    for _ in range(8):
        R = B.clone()
        for j in range(0, n, 4096):
            T = A[j : j + 4096, j:].triu()
            R[:, j : j + 4096] -= X[:, j:] @ T.mT
            T.diagonal().zero_()
            R[:, j:] -= X[:, j : j + 4096] @ T
        Y = torch.linalg.solve_triangular(U.mT, R.float().mT, upper=False)
        X += torch.linalg.solve_triangular(U, Y, upper=True).mT.double()
    return X


_G = 0x9E3779B97F4A7C15


def _mix(z):
    """SplitMix64's output function on int64 (wrapping products, logical shifts)."""
    for shift, factor in ((30, 0xBF58476D1CE4E5B9), (27, 0x94D049BB133111EB), (31, 1)):
        z = (z ^ ((z >> shift) & ((1 << (64 - shift)) - 1))) * (factor - (1 << 64) if factor >> 63 else factor)
    return z


def _stream(key, index):
    """53-bit integers: output number `index` of the stream of `key`."""
    return (_mix(key + (index + 1) * (_G - (1 << 64))) >> 11) & ((1 << 53) - 1)


def _key(seed):
    z = (seed + _G) % (1 << 64)
    return _mix(torch.tensor(z - (1 << 64) if z >> 63 else z, dtype=torch.int64, device=DEV))


def _serve_exact(n, matrix_seed, rhs_seed):
    """x of A x = b for the served system: A = (R + R^T)/2 + n I, b normal by Box and Muller."""
    i = torch.arange(n, dtype=torch.int64, device=DEV)
    R = _stream(_key(matrix_seed), i[:, None] + i[None, :] * n).double() * 2.0**-53 - 0.5
    A = (R + R.mT) / 2
    A.diagonal().add_(n)
    k = _key(rhs_seed)
    u1, u2 = (_stream(k, 2 * i).double() + 0.5) * 2.0**-53, _stream(k, 2 * i + 1).double() * 2.0**-53
    b = torch.sqrt(-2 * torch.log(u1)) * torch.cos(2 * math.pi * u2)
    return torch.cholesky_solve(b[:, None], torch.linalg.cholesky(A))[:, 0].cpu().numpy()
