"""Workloads the speed of this library is judged on, through its public Python entry points.

Every case is something a user of the library calls: a tridiagonal eigensolve (qr_algorithm_,
src/bulge_chasing.jl:146-288) in the reference's own sweep sequence or with multishift batches,
a bulk application of a rotation grid (bulk_wave_order_2x2_rmul_, src/wave.jl:36-162), a batch of
small solves, the pullback of a solve, and the reduction of a dense matrix that precedes one.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__

DTYPES = {"f64": torch.float64, "f32": torch.float32}


def _pkg():
    return __graft_entry__.load_package()


def _device():
    return torch.device("cuda", 0)


def _generator(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


# ---- the cases ------------------------------------------------------------------------------

def listed():
    return [
        # The smallest call: a numpy caller solves one small tridiagonal (a Lanczos or
        # quadrature matrix) with the defaults.  Latency, launches and copies.
        {"name": "solve_host_n64", "kind": "solve", "n": 64, "spectrum": "uniform", "q": "f64",
         "mode": 0, "where": "host"},
        # The default call at an ordinary size: the reference's sweep sequence, FP64 vectors.
        {"name": "solve_default_n750", "kind": "solve", "n": 750, "spectrum": "ramp", "q": "f64",
         "mode": 0, "where": "device"},
        # The reference's README example (n = 2000, d = 1:n) with the multishift chase.
        {"name": "solve_multishift_n2000", "kind": "solve", "n": 2000, "spectrum": "ramp",
         "q": "f64", "mode": 3, "where": "device"},
        # A random diagonal at an odd order with FP32 vectors: the FP32-Q variant.
        {"name": "solve_multishift_q32_n3001", "kind": "solve", "n": 3001, "spectrum": "normal",
         "q": "f32", "mode": 3, "where": "device"},
        # A small bulk apply, one of many a caller's own iteration makes.
        {"name": "apply_f64_small", "kind": "apply", "m": 200, "n": 201, "k": 32, "dtype": "f64",
         "side": "right", "where": "device"},
        # An ordinary bulk apply: a whole buffer of the default 128 layers.
        {"name": "apply_f64_mid", "kind": "apply", "m": 2500, "n": 2501, "k": 128, "dtype": "f64",
         "side": "right", "where": "device"},
        # The reference's benchmark shape (benchmark.jl): 64 layers on 16384 x 16384.
        {"name": "apply_f64_16384", "kind": "apply", "m": 16384, "n": 16384, "k": 64,
         "dtype": "f64", "side": "right", "where": "device"},
        # FP32 at a ragged size, layers not a multiple of a pass.
        {"name": "apply_f32_large", "kind": "apply", "m": 11000, "n": 10999, "k": 100,
         "dtype": "f32", "side": "right", "where": "device"},
        # The same operation on pinned host memory, copies included (the C ABI's host entry).
        {"name": "apply_host_6144", "kind": "apply", "m": 6144, "n": 6144, "k": 64, "dtype": "f64",
         "side": "right", "where": "host"},
        # Many small eigenproblems of uneven orders in one call.
        {"name": "batched_f64_256", "kind": "batched", "count": 256, "lo": 32, "hi": 320,
         "q": "f64"},
        # The backward pass of a differentiable eigensolve.
        {"name": "adjoint_n2047", "kind": "adjoint", "n": 2047, "batch": 1, "vectors": True},
        # A dense symmetric matrix to tridiagonal form and its orthogonal factor.
        {"name": "dense_n1300", "kind": "dense", "n": 1300},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "apply", "apply", "apply", "batched", "adjoint", "dense"])
    if kind == "solve":
        mode = rng.choice([0, 3])
        return {"kind": kind, "n": _log_int(rng, 16, 750 if mode == 0 else 2000),
                "spectrum": rng.choice(["ramp", "uniform", "normal"] if mode == 3 else ["ramp", "uniform"]),
                "q": rng.choice(["f64", "f64", "f32", "none"]), "mode": mode,
                "where": rng.choice(["device", "device", "host"])}
    if kind == "apply":
        where = rng.choice(["device", "device", "device", "host"])
        top = 16384 if where == "device" else 6144
        m, n = _log_int(rng, 32, top), _log_int(rng, 32, top)
        k = _log_int(rng, 4, 64 if where == "host" else 128) if rng.random() < 0.7 else 64
        return {"kind": kind, "m": m, "n": n, "k": min(k, 64 * 16384 ** 2 // (m * n)),
                "dtype": rng.choice(["f64", "f64", "f32"]), "side": rng.choice(["right", "right", "right", "left"]),
                "where": where}
    if kind == "batched":
        lo = _log_int(rng, 8, 64)
        return {"kind": kind, "count": _log_int(rng, 16, 256), "lo": lo,
                "hi": lo + _log_int(rng, 8, 256), "q": rng.choice(["f64", "f32", "none"])}
    if kind == "adjoint":
        n = _log_int(rng, 48, 2047)
        return {"kind": kind, "n": n, "batch": max(1, min(64, (1500 // n) ** 2)),
                "vectors": rng.random() < 0.7}
    return {"kind": kind, "n": _log_int(rng, 48, 1300)}


# ---- inputs ---------------------------------------------------------------------------------

def _tridiagonal(n, spectrum, gen, device):
    """d, e of the three families the reference's tests and benchmark use."""
    u = lambda k: torch.rand(k, generator=gen, dtype=torch.float64, device=device)  # noqa: E731
    z = lambda k: torch.randn(k, generator=gen, dtype=torch.float64, device=device)  # noqa: E731
    if spectrum == "ramp":       # d = 1:n, e ~ U[0, 1)
        return torch.arange(1, n + 1, dtype=torch.float64, device=device), u(n - 1)
    if spectrum == "uniform":    # d, e ~ U[0, 1)
        return u(n), u(n - 1)
    return z(n), 0.5 * z(n - 1)  # normal


def _apply_inputs(case, seed):
    gen, dt = _generator(seed), DTYPES[case["dtype"]]
    m, n, k = case["m"], case["n"], case["k"]
    A = torch.randn(n, m, generator=gen, dtype=dt, device=_device())      # memory of a column-major m x n
    rows = (n if case["side"] == "right" else m) - 1
    th = torch.rand(k, rows, generator=gen, dtype=torch.float64, device=_device()) * (2 * math.pi)
    g = torch.stack([th.cos(), th.sin()], dim=-1).to(dt)                  # memory of a Julia (rows, k) grid
    return A, g


def _batch_inputs(case, seed):
    # the orders belong to the case (a caller's fixed set of problems), the entries to the seed
    sizes = np.random.default_rng(case["count"]).integers(case["lo"], case["hi"] + 1, size=case["count"])
    gen = _generator(seed)
    d = torch.randn(int(sizes.sum()), generator=gen, dtype=torch.float64, device=_device())
    e = 0.1 + 0.9 * torch.rand(int((sizes - 1).sum()), generator=gen, dtype=torch.float64, device=_device())
    return sizes, d, e


def _adjoint_inputs(case, seed):
    """Eigenpairs of a Toeplitz tridiagonal (a, b) per matrix, columns in a random order with
    random signs, as a solver leaves them, and gradients of a loss with respect to them."""
    gen, dev = _generator(seed), _device()
    B, n = case["batch"], case["n"]
    f64 = dict(dtype=torch.float64, device=dev)
    j = torch.arange(1, n + 1, **f64)
    a, b = torch.randn(B, 1, generator=gen, **f64), 0.5 + torch.rand(B, 1, generator=gen, **f64)
    perm = torch.argsort(torch.rand(B, n, generator=gen, **f64), dim=1)
    jj = j[perm]                                                          # (B, n)
    lam = a + 2 * b * torch.cos(jj * (math.pi / (n + 1)))
    sign = torch.where(torch.rand(B, n, generator=gen, **f64) < 0.5, -1.0, 1.0) * math.sqrt(2.0 / (n + 1))
    # Qt[b, c, i]: row c of the memory is eigenvector c
    Qt = torch.sin(jj[:, :, None] * j[None, None, :] * (math.pi / (n + 1))) * sign[:, :, None]
    glam = torch.randn(B, n, generator=gen, **f64)
    gQt = torch.randn(B, n, n, generator=gen, **f64) if case["vectors"] else None
    Q = Qt.transpose(1, 2)
    gQ = gQt.transpose(1, 2) if gQt is not None else None
    if B == 1:
        return lam[0], Q[0], glam[0], None if gQ is None else gQ[0]
    return lam, Q, glam, gQ


def prepare(case, seed):
    pkg, kind = _pkg(), case["kind"]
    state = {"case": case, "pkg": pkg}
    if kind == "solve":
        d, e = _tridiagonal(case["n"], case["spectrum"], _generator(seed), _device())
        if case["where"] == "host":
            d, e = d.cpu().numpy(), e.cpu().numpy()
        state["H"] = pkg.SymTridiagonal(d, e)
    elif kind == "apply":
        A, g = _apply_inputs(case, seed)
        if case["where"] == "host":
            hA, hg = torch.empty(A.shape, dtype=A.dtype, pin_memory=True), torch.empty(g.shape, dtype=g.dtype, pin_memory=True)
            hA.copy_(A)
            hg.copy_(g)
            A, g = hA.numpy(), hg.numpy()
            state["keep"] = (hA, hg)
            state["A"], state["g"] = A.T, g.transpose(1, 0, 2)
        else:
            state["A"], state["g"] = A.T, g.permute(1, 0, 2)
    elif kind == "batched":
        sizes, d, e = _batch_inputs(case, seed)
        state.update(sizes=sizes, d=d, e=e)
        # where each matrix's diagonal of its Q lies, to lay out the identities in one call
        q0 = np.concatenate([[0], np.cumsum(sizes * sizes)])
        at = np.concatenate([q0[i] + np.arange(n) * (n + 1) for i, n in enumerate(sizes)])
        state["diag"], state["nq"] = torch.from_numpy(at).to(_device()), int(q0[-1])
        state["segment"] = torch.from_numpy(np.repeat(np.arange(len(sizes)), sizes)).to(_device())
    elif kind == "adjoint":
        state["in"] = _adjoint_inputs(case, seed)
    else:
        X = torch.randn(case["n"], case["n"], generator=_generator(seed), dtype=torch.float64, device=_device())
        state["A"] = ((X + X.T) * 0.5).T
    return state


# ---- one pass -------------------------------------------------------------------------------

def run(state):
    case, pkg = state["case"], state["pkg"]
    kind = case["kind"]
    if kind == "solve":
        # the spectrum in ascending order with its vectors
        n, H = case["n"], state["H"].copy()
        if case["where"] == "host":
            Q = None if case["q"] == "none" else np.asfortranarray(np.eye(n, dtype=np.float64 if case["q"] == "f64" else np.float32))
            _, conv, iters = pkg.qr_algorithm_(H, Q, chase_mode=case["mode"])
            order = np.argsort(H.dv, kind="stable")
            out = {"lam": H.dv[order], "converged": conv, "sweeps": iters}
        else:
            Q = None if case["q"] == "none" else torch.eye(n, dtype=DTYPES[case["q"]], device=H.dv.device).T
            _, conv, iters = pkg.qr_algorithm_(H, Q, chase_mode=case["mode"])
            lam, order = torch.sort(H.dv, stable=True)
            out = {"lam": lam, "converged": conv, "sweeps": iters}
        if Q is not None:
            out["V"] = Q[:, order]
        return out
    if kind == "apply":
        f = pkg.bulk_wave_order_2x2_rmul_ if case["side"] == "right" else pkg.bulk_wave_order_2x2_lmul_
        f(state["A"], state["g"])
        return {"A": state["A"]}
    if kind == "batched":
        d, e = state["d"].clone(), state["e"].clone()
        Q = None
        if case["q"] != "none":
            Q = torch.zeros(state["nq"], dtype=DTYPES[case["q"]], device=d.device)
            Q[state["diag"]] = 1.0
        conv, iters = pkg.qr_algorithm_batched_(d, e, state["sizes"], Q)
        # every matrix's spectrum in ascending order; the vectors stay as the solver left them
        lam, order = torch.sort(d, stable=True)
        lam = lam[torch.argsort(state["segment"][order], stable=True)]
        out = {"lam": lam, "converged": conv, "sweeps": iters}
        if Q is not None:
            out["Q"] = Q
        return out
    if kind == "adjoint":
        lam, Q, glam, gQ = state["in"]
        gd, ge = pkg.eig_adjoint(lam, Q, glam, gQ)
        return {"gd": gd, "ge": ge}
    A = state["A"].clone()          # sytrd_ overwrites its input
    d, e, tau = pkg.sytrd_(A)
    return {"d": d, "e": e, "tau": tau, "Q": pkg.orgtr(A, tau)}


# ---- what a pass cannot do without ----------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "solve":
        # about n^2 / 2 rotations (each about 30 flops of chase), applied to n rows at 6 flops
        n, q = case["n"], {"f64": 8, "f32": 4, "none": 0}[case["q"]]
        rot = n * n / 2
        return {"bytes": 2 * q * n * n + 2 * 16 * n, "flops": rot * (30 + (6 * n if q else 0))}
    if kind == "apply":
        size = 8 if case["dtype"] == "f64" else 4
        m, n, k = case["m"], case["n"], case["k"]
        cols, rows = (n, m) if case["side"] == "right" else (m, n)
        return {"bytes": size * (2 * m * n + 2 * (cols - 1) * k), "flops": 6.0 * rows * (cols - 1) * k}
    if kind == "batched":
        q = {"f64": 8, "f32": 4, "none": 0}[case["q"]]
        lo, hi, c = case["lo"], case["hi"], case["count"]
        n2 = (lo * lo + lo * hi + hi * hi) / 3                    # E[n^2], E[n^3] of n ~ U[lo, hi]
        n3 = (lo + hi) * (lo * lo + hi * hi) / 4
        return {"bytes": c * (2 * q * n2 + 16 * (lo + hi)), "flops": c * (15 * n2 + (3 * n3 if q else 0))}
    if kind == "adjoint":
        n, B = case["n"], case["batch"]
        if not case["vectors"]:
            return {"bytes": 8.0 * B * (n * n + 4 * n), "flops": 4.0 * B * n * n}
        # Q^T gQ, and of Q M Q^T only Q M and the band
        return {"bytes": 8.0 * B * (2 * n * n + 4 * n), "flops": B * (4.0 * n ** 3 + 6.0 * n * n)}
    n = case["n"]
    return {"bytes": 8.0 * 3 * n * n, "flops": 8.0 / 3 * n ** 3}


# ---- the same in 64 bits by plain torch -----------------------------------------------------

def _exact_apply(A, g):
    """X (columns as rows: n x m) through the grid g (k, n-1, 2), independent rotations together."""
    n, k = A.shape[0], g.shape[0]
    layers = torch.arange(k, device=A.device)
    for s in range(n - 1 + 2 * (k - 1)):
        # rotations (r, L) with r + 2 L = s
        lo, hi = max(0, -(-(s - (n - 2)) // 2)), min(k - 1, s // 2)
        if lo > hi:
            continue
        L = layers[lo:hi + 1].flip(0)
        c, t = g[L, s - 2 * L].unbind(-1)
        r0 = s - 2 * hi
        X = A[r0:r0 + 2 * (hi - lo + 1)].view(hi - lo + 1, 2, -1)
        x, y = X[:, 0], X[:, 1]
        nx = c[:, None] * x + t[:, None] * y
        ny = c[:, None] * y - t[:, None] * x
        X[:, 0], X[:, 1] = nx, ny
    return A


def _exact_sytrd(A):
    """Householder tridiagonalisation (lower, unblocked) and its orthogonal factor."""
    n = A.shape[0]
    A = A.clone()
    Q = torch.eye(n, dtype=A.dtype, device=A.device)
    e, tau, vs = [], [], []
    for j in range(n - 1):
        x = A[j + 1:, j].clone()
        alpha = x[0].clone()
        tail = torch.linalg.vector_norm(x[1:])
        beta = torch.where(tail > 0, -torch.sign(torch.where(alpha == 0, 1.0, alpha)) * torch.hypot(alpha, tail), alpha)
        t = torch.where(tail > 0, (beta - alpha) / beta, torch.zeros_like(beta))
        v = torch.where(tail > 0, x / (alpha - beta), torch.zeros_like(x))
        v[0] = 1.0
        S = A[j + 1:, j + 1:]
        p = t * (S @ v)
        w = p - (0.5 * t * (p @ v)) * v
        S -= torch.outer(v, w) + torch.outer(w, v)
        e.append(beta)
        tau.append(t)
        vs.append(v)
    for j in range(n - 2, -1, -1):
        v, R = vs[j], Q[j + 1:, j + 1:]
        R -= torch.outer(tau[j] * v, v @ R)
    return A.diagonal().clone(), torch.stack(e), torch.stack(tau), Q


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        d, e = _tridiagonal(case["n"], case["spectrum"], _generator(seed), _device())
        T = torch.diag(d) + torch.diag(e, 1) + torch.diag(e, -1)
        # the vectors' signs are the algorithm's own
        out = {"lam": torch.linalg.eigvalsh(T), "converged": None, "sweeps": None}
        if case["q"] != "none":
            out["V"] = None
        return out
    if kind == "apply":
        A, g = _apply_inputs(case, seed)
        A, g = A.double(), g.double()
        if case["side"] == "right":
            return {"A": _exact_apply(A, g).T}
        return {"A": _exact_apply(A.T.contiguous(), g)}
    if kind == "batched":
        sizes, d, e = _batch_inputs(case, seed)
        lam, i, j = [], 0, 0
        for n in sizes.tolist():
            T = torch.diag(d[i:i + n]) + torch.diag(e[j:j + n - 1], 1) + torch.diag(e[j:j + n - 1], -1)
            lam.append(torch.linalg.eigvalsh(T.cpu()))
            i, j = i + n, j + n - 1
        out = {"lam": torch.cat(lam), "converged": None, "sweeps": None}
        if case["q"] != "none":
            out["Q"] = None
        return out
    if kind == "adjoint":
        lam, Q, glam, gQ = _adjoint_inputs(case, seed)
        if lam.ndim == 1:
            lam, Q, glam, gQ = lam[None], Q[None], glam[None], None if gQ is None else gQ[None]
        M = torch.diag_embed(glam)
        if gQ is not None:
            gap = lam[:, None, :] - lam[:, :, None]
            F = torch.where(gap != 0, 1.0 / gap, torch.zeros_like(gap))
            M = M + F * (Q.transpose(1, 2) @ gQ)
        Ab = Q @ M @ Q.transpose(1, 2)
        gd = Ab.diagonal(dim1=1, dim2=2)
        ge = Ab.diagonal(offset=1, dim1=1, dim2=2) + Ab.diagonal(offset=-1, dim1=1, dim2=2)
        return {"gd": gd, "ge": ge} if case["batch"] > 1 else {"gd": gd[0], "ge": ge[0]}
    X = torch.randn(case["n"], case["n"], generator=_generator(seed), dtype=torch.float64, device=_device())
    d, e, tau, Q = _exact_sytrd((X + X.T) * 0.5)
    return {"d": d, "e": e, "tau": tau, "Q": Q}
