"""What a user of the eigensolver has it do, as a list of measurable cases.

``listed()`` gives the fixed cases, ``draw(rng)`` more of the same ranges,
``prepare`` what a program holds before the call (matrices, workspaces, result
buffers), ``run`` one pass through the public entry points, ``work`` the bytes
and operations the path cannot do without and ``exact`` the result of plain
FP64 torch on the same inputs.

Kinds:

* ``solve``   all eigenpairs, plain FP64 (``syevd``): orders 64 (the smallest
  of a batch) to 8192 (the largest served), any residue modulo the block size;
* ``mixed``   all eigenpairs with the contractions on the integer tensor cores
  (``syevd_mixed``), the form the server uses from order 2048 on;
* ``fp32``    all eigenpairs of an FP32 matrix (``syevd_s``);
* ``values``  eigenvalues only (``syevd_values``);
* ``batch``   many matrices of uneven orders in one call (``evd_syevd_batched``);
* ``refine``  Ogita-Aishima iterations on approximate eigenpairs;
* ``back``    the stage-2 back transformation of a block of eigenvectors
  (``bc_back_apply``): a program that wants some of the eigenvectors applies
  it to those columns only;
* ``syr2k``   the FP16-product rank-2k update of the FP32 API (``tc_syr2k``).

Eigenvectors are returned with a fixed sign (the entry of largest magnitude of
each column is positive), the usual step of programs that store or compare
them, because the solver leaves the sign free.
"""
import math

import torch

import evd4sc2025_b200 as evd
from evd4sc2025_b200 import lowprec, serve

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # the smallest requests of a batch: launches and latency only
        {"name": "solve_100", "kind": "solve", "n": 100, "nb": 0},
        # an ordinary small matrix, order not a multiple of the block
        {"name": "solve_1000", "kind": "solve", "n": 1000, "nb": 0},
        # the documented small run `myEVD 4096 32 1024`
        {"name": "solve_4096", "kind": "solve", "n": 4096, "nb": 1024},
        # the largest order that the server admits, plain FP64
        {"name": "solve_8192", "kind": "solve", "n": 8192, "nb": 1024},
        # a served request above the plain/mixed switch, odd order
        {"name": "mixed_3001", "kind": "mixed", "n": 3001, "nb": 0},
        # the headline: n = 16384, b = 32, nb = 1024
        {"name": "mixed_16384", "kind": "mixed", "n": 16384, "nb": 1024},
        # FP32 matrix in, FP32 eigenpairs out
        {"name": "fp32_2500", "kind": "fp32", "n": 2500, "nb": 0},
        # a spectrum without vectors
        {"name": "values_2048", "kind": "values", "n": 2048, "nb": 0},
        # uneven orders, log-uniform over [64, 1024], one call
        {"name": "batch_24", "kind": "batch", "count": 24, "lo": 64, "hi": 1024, "sizes": 7},
        # one refinement iteration of FP32-accurate eigenvectors
        {"name": "refine_3072", "kind": "refine", "n": 3072, "iters": 1},
        # a quarter of the eigenvectors through the stage-2 reflectors
        {"name": "back_6000", "kind": "back", "n": 6000, "ncols": 1500},
        # the FP32 API's trailing update on FP16 products
        {"name": "syr2k_8192", "kind": "syr2k", "n": 8192, "k": 1024},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "mixed", "mixed", "fp32", "values", "batch",
                       "refine", "back", "syr2k"])
    if kind == "solve":
        return {"kind": kind, "n": _logint(rng, 64, 8192), "nb": 0}
    if kind == "mixed":
        return {"kind": kind, "n": _logint(rng, 2048, 12288), "nb": 0}
    if kind == "fp32":
        return {"kind": kind, "n": _logint(rng, 256, 6000), "nb": 0}
    if kind == "values":
        return {"kind": kind, "n": _logint(rng, 64, 8192), "nb": 0}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(6, 30), "lo": 64, "hi": 1024,
                "sizes": rng.randrange(1 << 20)}
    if kind == "refine":
        return {"kind": kind, "n": _logint(rng, 512, 4096), "iters": rng.randint(1, 2)}
    if kind == "back":
        n = _logint(rng, 256, 8192)
        return {"kind": kind, "n": n, "ncols": _logint(rng, max(1, n // 16), n)}
    return {"kind": kind, "n": _logint(rng, 256, 12288), "k": 8 * _logint(rng, 8, 256)}


# ------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _gauss(n, g, dtype=F64):
    """(G + G^T) / 2 with standard normal G, column-major."""
    A = evd.empty_cm(n, n, device=DEV, dtype=dtype)
    G = torch.randn(n, n, generator=g, dtype=F64, device=DEV)
    A.copy_(0.5 * (G + G.t()))
    return A


def _sizes(case):
    g = torch.Generator().manual_seed(case["sizes"])
    u = torch.rand(case["count"], generator=g, dtype=F64).tolist()
    r = math.log(case["hi"] / case["lo"])
    return [int(round(case["lo"] * math.exp(r * x))) for x in u]


def _nb(case):
    """The block size: the case's own, or the library's choice for the order."""
    return case["nb"] or serve.solve_shape(case["n"])[1]


def _reflectors(n, g):
    """Stage-2 reflectors in the chase's layout: column s holds, from row s + 1
    on, 32-row segments of vectors with ||u||^2 = 2."""
    b = 32
    sweep = torch.arange(n, device=DEV)[:, None]
    length = -(-n // b) * b
    P = torch.randn(n, length, generator=g, dtype=F64, device=DEV)  # row s: sweep s from row s + 1
    # (a segment of one row would start at row n - 1: the chase stores none there)
    last = torch.where((n - 2 - sweep) % b == 0, n - sweep - 2, n - sweep - 1)
    P *= (torch.arange(length, device=DEV)[None, :] < last) & (sweep < n - 2)
    P = P.view(n, length // b, b)
    P *= torch.sqrt(2.0 / (P * P).sum(dim=2, keepdim=True).clamp_min(1e-300))
    at = torch.arange(n, device=DEV)[None, :] - sweep - 1
    U = evd.empty_cm(n, n, device=DEV)
    U.copy_((P.view(n, length).gather(1, at.clamp_min(0)) * (at >= 0)).t())
    return U


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "batch":
        return {"case": case, "A": [_gauss(n, g) for n in _sizes(case)]}
    n = case["n"]
    s = {"case": case}
    if kind in ("solve", "mixed", "values"):
        s["nb"] = _nb(case)
        s["A"] = _gauss(n, g)
        s["w"] = torch.empty(n, dtype=F64, device=DEV)
        if kind == "mixed":
            s["ws"] = evd.MixedWorkspace(n, 32, s["nb"], device=DEV)
        else:
            s["ws"] = evd.Workspace(n, 32, s["nb"], device=DEV)
        if kind != "values":
            s["X"] = evd.empty_cm(n, n, device=DEV)
    elif kind == "fp32":
        s["nb"] = _nb(case)
        s["A"] = _gauss(n, g, torch.float32)
        s["w"] = torch.empty(n, dtype=torch.float32, device=DEV)
        s["X"] = evd.empty_cm(n, n, device=DEV, dtype=torch.float32)
        s["work"] = torch.empty(int(evd.lib().evd_syevd_s_work_size(n, 32, s["nb"])),
                                dtype=torch.uint8, device=DEV)
    elif kind == "refine":
        # A = Q diag(lam) Q^T with lam in [-1, 1], and eigenvectors as an FP32
        # solver would give them
        Q = torch.linalg.qr(torch.randn(n, n, generator=g, dtype=F64, device=DEV)).Q
        step = 2.0 / n
        lam = -1.0 + step * (torch.arange(n, dtype=F64, device=DEV)
                             + 0.5 * torch.rand(n, generator=g, dtype=F64, device=DEV))
        M = (Q * lam) @ Q.t()
        s["A"] = evd.to_cm(0.5 * (M + M.t()), device=DEV)
        E = torch.randn(n, n, generator=g, dtype=F64, device=DEV)
        s["X0"] = evd.to_cm((Q + 1e-8 * E).float(), device=DEV)
        s["X"] = evd.empty_cm(n, n, device=DEV)
        s["w"] = torch.empty(n, dtype=F64, device=DEV)
        s["work"] = evd.refine_ozaki_work(n, device=DEV)
    elif kind == "back":
        s["U"] = _reflectors(n, g)
        s["Z"] = evd.to_cm(torch.randn(n, case["ncols"], generator=g, dtype=F64, device=DEV),
                           device=DEV)
        s["X"] = evd.empty_cm(n, case["ncols"], device=DEV)
        s["work"] = torch.empty(max(1, evd.lib().evd_bc_back_work_size(n)), dtype=F64, device=DEV)
    else:
        k = case["k"]
        for name, (r, c) in (("A", (n, k)), ("B", (n, k)), ("C", (n, n))):
            t = torch.randn(r, c, generator=g, dtype=torch.float32, device=DEV)
            s[name] = lowprec.to_cm(t, torch.float32, device=DEV)
        s["hwork"] = torch.empty(2 * n * k, dtype=torch.float16, device=DEV)
    return s


# ---------------------------------------------------------------------- run
def _fixed_sign(X):
    """Each column times +-1 so that its entry of largest magnitude is positive."""
    lo, hi = torch.aminmax(X, dim=0)
    return X.mul_(torch.where(hi >= -lo, 1.0, -1.0).to(X.dtype))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        w, X = evd.syevd(state["A"], 32, state["nb"], ws=state["ws"], w=state["w"], X=state["X"])
        return w, _fixed_sign(X)
    if kind == "mixed":
        w, X = evd.syevd_mixed(state["A"], 32, state["nb"], ws=state["ws"], w=state["w"],
                               X=state["X"])
        return w, _fixed_sign(X)
    if kind == "fp32":
        w, X = evd.syevd_s(state["A"], 32, state["nb"], work=state["work"], w=state["w"],
                           X=state["X"])
        return w, _fixed_sign(X)
    if kind == "values":
        return evd.syevd_values(state["A"], 32, state["nb"], ws=state["ws"], w=state["w"])
    if kind == "batch":
        pairs, _ = serve.syevd_batched_native(state["A"])
        return [(w, _fixed_sign(X)) for w, X in pairs]
    if kind == "refine":
        state["X"].copy_(state["X0"])
        return evd.refine_syev_ozaki(state["A"], state["X"], iters=case["iters"], w=state["w"],
                                     work=state["work"])
    if kind == "back":
        state["X"].copy_(state["Z"])
        return evd.bc_back_apply(state["X"], state["U"], work=state["work"])
    return lowprec.tc_syr2k(-1.0, state["A"], state["B"], 1.0, state["C"], hwork=state["hwork"])


# --------------------------------------------------------------------- work
def work(case):
    """All eigenpairs: A read, w and X written, 16/3 n^3 operations (4/3 n^3
    the reduction, 2 n^3 each back transformation); eigenvalues only: 4/3 n^3;
    a refinement iteration: 8 n^3; stage-2 reflectors: 2 n^2 per column;
    rank-2k update of a triangle: 2 n^2 k."""
    kind = case["kind"]
    if kind == "batch":
        ns = _sizes(case)
        return {"bytes": sum(16 * n * n + 8 * n for n in ns),
                "flops": sum(16 / 3 * n ** 3 for n in ns)}
    n = case["n"]
    if kind in ("solve", "mixed"):
        return {"bytes": 16 * n * n + 8 * n, "flops": 16 / 3 * n ** 3}
    if kind == "fp32":
        return {"bytes": 8 * n * n + 4 * n, "flops": 16 / 3 * n ** 3}
    if kind == "values":
        return {"bytes": 8 * n * n + 8 * n, "flops": 4 / 3 * n ** 3}
    if kind == "refine":
        return {"bytes": 24 * n * n + 8 * n, "flops": 8 * n ** 3 * case["iters"]}
    if kind == "back":
        return {"bytes": 4 * n * n + 16 * n * case["ncols"], "flops": 2 * n * n * case["ncols"]}
    k = case["k"]
    return {"bytes": 8 * n * k + 4 * n * n, "flops": 2 * n * n * k}


# -------------------------------------------------------------------- exact
def _eigh(A):
    w, X = torch.linalg.eigh(A.to(F64))
    return w, _fixed_sign(X)


def exact(case, seed):
    """The same outputs from torch in FP64; None for orders where that takes
    longer than about 20 seconds."""
    kind = case["kind"]
    if kind in ("solve", "mixed", "fp32", "values", "refine") and case["n"] > 8192:
        return None
    s = prepare(case, seed)
    if kind == "batch":
        return [_eigh(A) for A in s["A"]]
    if kind in ("solve", "mixed", "fp32"):
        return _eigh(s["A"])
    if kind == "values":
        return torch.linalg.eigvalsh(s["A"])
    if kind == "refine":
        # ascending here as in X0; each eigenvector on the side of its start
        w, X = torch.linalg.eigh(s["A"])
        return w, X * torch.where((X * s["X0"]).sum(dim=0) >= 0, 1.0, -1.0)
    if kind == "back":
        return _apply_reflectors(s["U"], s["Z"]) if case["n"] <= 1024 else None
    n = case["n"]
    a, b = s["A"].half().to(F64), s["B"].half().to(F64)
    c = s["C"].to(F64)
    full = c - (a @ b.t() + b @ a.t())
    low = torch.ones(n, n, dtype=torch.bool, device=DEV).tril_()
    return torch.where(low, full, c)


def _apply_reflectors(U, Z):
    """X = Q2 Z, sweep by sweep from the last (the segments of one sweep are
    disjoint, so they apply together)."""
    n, b = U.shape[0], 32
    X = Z.clone()
    for s in range(n - 3, -1, -1):
        m = n - s - 1
        pad = -m % b
        u = torch.nn.functional.pad(U[s + 1:, s], (0, pad)).view(-1, b, 1)
        x = torch.nn.functional.pad(X[s + 1:], (0, 0, 0, pad)).view(-1, b, X.shape[1])
        x = x - u * (u * x).sum(dim=1, keepdim=True)
        X[s + 1:] = x.reshape(-1, X.shape[1])[:m]
    return X
