"""Performance cases: the work that programs have this library do, through
its public entry points, over the range of sizes they use it at.

A case is a plain dict; its "do" names one of these kinds of work:

  solve     one model through MadSDPSolver, to the default tolerance or for
            a bounded number of iterations
  iterate   initialize and a bounded number of iterations of one large model
            on the whole GPU (InstanceSolver with max_iter)
  batch     initialize and a bounded number of iterations of many models in
            one launch, as the waves of a serving loop run them (Batch)
  scaling   what a host driver asks of the GPU for one block of an iterate:
            set_iterate, prepare, the scaling matrices and the smallest
            eigenvalue behind a step length (InstanceSolver components)
  assembly  set_iterate, prepare and the Schur complement matrix of dense
            constraints (InstanceSolver components)
  schur     a host-assembled Schur system factored and solved
            (SchurWorkspace)
  product   a float64 product on the tensor cores (msdp_tc_gemm)

Inputs are seeded synthetic models of the package's own generators and
iterates near a central path.
"""

import ctypes
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "madsdp.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import madsdp_gpu as M  # noqa: E402
from madsdp_gpu import _lib, generators  # noqa: E402

# a host-driven loop's slice: the iterations a wave of the server advances
# its requests by, and enough for the iterate to have left the identity
SLICE = 3


def listed():
    return [
        # the smallest call: a slice of one max-cut relaxation of a dozen
        # nodes, where launches and the host side of a call count most
        {"name": "slice_tiny", "do": "solve", "n": 12, "p": 0.4, "max_iter": SLICE},
        # the benchmark's max-cut instance (n = 100, edge probability 0.1),
        # solved to the tolerance
        {"name": "solve_maxcut_100", "do": "solve", "n": 100, "p": 0.1, "max_iter": 100},
        # the benchmark's max-cut instance at scale (n = 2000, weights +-1)
        {"name": "iterate_maxcut_2000", "do": "iterate", "model": "maxcut", "n": 2000, "p": 0.005, "m": 0, "ns": 0,
         "blocks": 1, "direction": "NT", "precision": "fp64"},
        # dense constraints on mixed cones: four blocks, scalars, m = 1000
        {"name": "iterate_dense_cones", "do": "iterate", "model": "dense", "n": 120, "p": 0.0, "m": 1000, "ns": 200,
         "blocks": 4, "direction": "NT", "precision": "fp64"},
        # batched univariate SOS bounds, Gram blocks of side 6 to 64, FP64
        {"name": "batch_sos_fp64", "do": "batch", "model": "sos", "count": 512, "lo": 5, "hi": 63,
         "direction": "NT", "precision": "fp64"},
        # the whole batched workload of the benchmark in mixed precision
        {"name": "batch_sos_mixed", "do": "batch", "model": "sos", "count": 4096, "lo": 5, "hi": 63,
         "direction": "NT", "precision": "mixed"},
        # a wave of served max-cut requests beyond the SOS sizes
        {"name": "batch_maxcut_fp64", "do": "batch", "model": "maxcut", "count": 64, "lo": 50, "hi": 128,
         "direction": "NT", "precision": "fp64"},
        # a host driver's scaling and step length at an odd size
        {"name": "scaling_517", "do": "scaling", "n": 517},
        # the Schur complement of dense constraints, HKM direction
        {"name": "assembly_hkm", "do": "assembly", "n": 90, "m": 600, "ns": 50, "direction": "HKM"},
        # the Schur system of a model with two thousand constraints
        {"name": "schur_2000", "do": "schur", "m": 2000, "precision": "fp64"},
        # an odd-sized Schur system in mixed precision with refinement
        {"name": "schur_717_mixed", "do": "schur", "m": 717, "precision": "mixed"},
        # the assembly's contraction as a plain product, ragged, lower half
        {"name": "product_lower", "do": "product", "M": 1999, "N": 1999, "K": 5051, "ta": 0, "tb": 1, "lower": True,
         "precision": "fp64"},
    ]


def _log(rng, lo, hi):
    return int(round(float(lo) * (float(hi) / float(lo)) ** rng.random()))


def draw(rng):
    do = rng.choice(["solve", "iterate", "batch", "batch", "scaling", "assembly", "schur", "product"])
    if do == "solve":
        # a slice in one thread block, or a solve on the whole GPU
        n = _log(rng, 3, 64) if rng.random() < 0.5 else _log(rng, 65, 110)
        return {"do": do, "n": n, "p": min(0.5, max(10.0, 0.4 * n) / n * rng.uniform(0.5, 1.0)),
                "max_iter": SLICE if n <= 64 else 100}
    if do == "iterate":
        if rng.random() < 0.5:
            n = _log(rng, 130, 1900)
            return {"do": do, "model": "maxcut", "n": n, "p": 4.0 / n + 0.01 * rng.random(), "m": 0, "ns": 0,
                    "blocks": 1, "direction": rng.choice(["NT", "NT", "HKM"]), "precision": "fp64"}
        n = _log(rng, 40, 140)
        return {"do": do, "model": "dense", "n": n, "p": 0.0, "m": min(_log(rng, 60, 900), n * n // 5),
                "ns": rng.choice([0, 7, 40, 200]), "blocks": rng.randint(1, 4),
                "direction": rng.choice(["NT", "NT", "HKM"]), "precision": "fp64"}
    if do == "batch":
        if rng.random() < 0.6:
            lo = rng.randint(5, 20)
            return {"do": do, "model": "sos", "count": _log(rng, 16, 1500), "lo": lo, "hi": rng.randint(lo + 5, 63),
                    "direction": "NT", "precision": rng.choice(["fp64", "mixed"])}
        lo = _log(rng, 10, 60)
        return {"do": do, "model": "maxcut", "count": _log(rng, 4, 64), "lo": lo, "hi": rng.randint(lo + 4, 128),
                "direction": rng.choice(["NT", "HKM"]), "precision": "fp64"}
    if do == "scaling":
        return {"do": do, "n": _log(rng, 24, 1100)}
    if do == "assembly":
        n = _log(rng, 30, 130)
        return {"do": do, "n": n, "m": min(_log(rng, 60, 700), n * n // 4), "ns": rng.choice([0, 13, 100]),
                "direction": rng.choice(["NT", "HKM"])}
    if do == "schur":
        return {"do": do, "m": _log(rng, 40, 2000), "precision": rng.choice(["fp64", "mixed"])}
    lower = rng.random() < 0.4
    m = _log(rng, 60, 2500)
    return {"do": do, "M": m, "N": m if lower else _log(rng, 60, 2500), "K": _log(rng, 30, 6000),
            "ta": rng.randint(0, 1), "tb": rng.randint(0, 1), "lower": lower,
            "precision": rng.choice(["fp64", "fp64", "mixed"])}


# ---------------------------------------------------------------- inputs
def _direction(case):
    return M.HKM() if case.get("direction") == "HKM" else M.NT()


def _sides(case):
    return [max(4, case["n"] >> min(i, 2)) for i in range(case["blocks"])]


def _iterate_model(case, seed):
    if case["model"] == "maxcut":
        return generators.maxcut(case["n"], case["p"], weights="pm1", seed=seed)
    return generators.dense_random(_sides(case), case["ns"], case["m"], seed=seed)


def _batch_models(case, seed):
    # the sizes belong to the case, the data to the seed
    sizes = np.random.default_rng(case["count"]).integers(case["lo"], case["hi"] + 1, size=case["count"])
    if case["model"] == "sos":
        return [generators.sos_hankel(int(d), seed=seed * 100003 + i) for i, d in enumerate(sizes)]
    return [generators.maxcut(int(n), min(0.5, 4.0 / n + 0.1), seed=seed * 100003 + i) for i, n in enumerate(sizes)]


def _interior_point(n, rng):
    """X and S near a central path: X has eigenvalues spread over three
    decades and X S is similar to mu times a matrix of moderate spectrum."""
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    d = np.exp(rng.uniform(-2.0, 2.0, n))
    Y, Yi = Q * d, Q / d
    E = rng.standard_normal((n, n)) / np.sqrt(n)
    E = 0.5 * np.eye(n) + E @ E.T
    X, S = Y @ Y.T, 0.01 * (Yi @ E @ Yi.T)
    return (X + X.T) / 2, (S + S.T) / 2


def _scaling_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    X, S = _interior_point(n, rng)
    D = rng.standard_normal((n, n))
    return X, S, rng.standard_normal(n), np.linalg.cholesky(S), (D + D.T) * (0.3 / np.sqrt(n))


def _assembly_inputs(case, seed):
    rng = np.random.default_rng(seed)
    X, S = _interior_point(case["n"], rng)
    x, z = np.exp(rng.uniform(-2, 2, case["ns"])), np.exp(rng.uniform(-2, 2, case["ns"]))
    return generators.dense_random([case["n"]], case["ns"], case["m"], seed=seed), X, S, rng.standard_normal(case["m"]), x, z


def _schur_inputs(case, seed):
    rng = np.random.default_rng(seed)
    m = case["m"]
    B = rng.standard_normal((m, m + m // 4 + 8)) * np.exp(rng.uniform(-1.5, 1.5, m))[:, None]
    return B @ B.T, rng.standard_normal(m)


def _product_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))

    def operand(rows, cols, scale_rows):
        # column-major rows x cols, held as its (cols, rows) transpose
        a = torch.randn((cols, rows), generator=gen, device="cuda", dtype=torch.float64)
        s = torch.rand(rows if scale_rows else cols, generator=gen, device="cuda", dtype=torch.float64) * 8 - 4
        return a * torch.exp(s if scale_rows else s[:, None])

    Mr, N, K = case["M"], case["N"], case["K"]
    A = operand(K, Mr, False) if case["ta"] else operand(Mr, K, True)
    if case["lower"]:
        return A, (A if bool(case["ta"]) != bool(case["tb"]) else A.t().contiguous())
    return A, (operand(N, K, True) if case["tb"] else operand(K, N, False))


def prepare(case, seed):
    do = case["do"]
    state = {"case": case}
    if do == "solve":
        state["solver"] = M.MadSDPSolver(generators.maxcut(case["n"], case["p"], seed=seed), max_iter=case["max_iter"])
    elif do == "iterate":
        state["solver"] = M.InstanceSolver(_iterate_model(case, seed), direction=_direction(case),
                                           precision=case["precision"], max_iter=SLICE)
    elif do == "batch":
        state["batch"] = M.Batch(_batch_models(case, seed), direction=_direction(case), precision=case["precision"])
    elif do == "scaling":
        X, S, y, L, D = _scaling_inputs(case, seed)
        state.update(X=X, S=S, y=y, L=L, D=D,
                     solver=M.InstanceSolver(generators.maxcut(case["n"], 4.0 / case["n"], seed=seed)))
    elif do == "assembly":
        model, X, S, y, x, z = _assembly_inputs(case, seed)
        state.update(X=X, S=S, y=y, x=x, z=z, solver=M.InstanceSolver(model, direction=_direction(case)))
    elif do == "schur":
        H, rhs = _schur_inputs(case, seed)
        state.update(H=H, rhs=rhs, ws=M.SchurWorkspace(case["m"], precision=case["precision"]))
    else:
        A, B = _product_inputs(case, seed)
        state.update(A=A, B=B, lib=_lib.load(),
                     C=torch.zeros((case["N"], case["M"]), device="cuda", dtype=torch.float64))
    return state


def _packed(solutions):
    """X, y, x and z of many problems, each laid out one after the other."""
    return {"X": np.concatenate([X.ravel(order="K") for s in solutions for X in s[0]]),
            "y": np.concatenate([s[1] for s in solutions]),
            "x": np.concatenate([s[2] for s in solutions]),
            "z": np.concatenate([s[3] for s in solutions])}


def run(state):
    case = state["case"]
    do = case["do"]
    if do == "solve":
        s = state["solver"].solve()
        out = _packed([s.solution()])
        return {**out, "pobj": s.primal_objective(), "dobj": s.dual_objective(), "iter": int(s.iter),
                "status": int(s.status)}
    if do == "iterate":
        s = state["solver"].solve()
        st = s.stats()
        return {**_packed([s.solution()]), "pobj": st["pobj"], "dobj": st["dobj"], "iter": int(st["iter"])}
    if do == "batch":
        b = state["batch"]
        b.initialize()
        b.iterate(SLICE)
        stats = b.all_stats()
        return {**_packed(b.all_solutions()), "pobj": np.array([t["pobj"] for t in stats]),
                "dobj": np.array([t["dobj"] for t in stats]), "iter": np.array([t["iter"] for t in stats])}
    if do == "scaling":
        s = state["solver"]
        s.set_iterate([state["X"]], [state["S"]], state["y"])
        ok = s.prepare()
        return {"ok": ok, "W": s.block_matrix(0, "W"), "Sinv": s.block_matrix(0, "Sinv"),
                "lam": s.step_eig(0, state["L"], state["D"])}
    if do == "assembly":
        s = state["solver"]
        s.set_iterate([state["X"]], [state["S"]], state["y"], state["x"], state["z"])
        ok = s.prepare()
        return {"ok": ok, "H": s.schur_assemble()}
    if do == "schur":
        ok = state["ws"].factorize(state["H"])
        return {"ok": ok, "x": state["ws"].solve(state["rhs"])}
    A, B, C = state["A"], state["B"], state["C"]
    rc = state["lib"].msdp_tc_gemm(1 if case["precision"] == "mixed" else 0, case["ta"], case["tb"], case["M"],
                                   case["N"], case["K"], 1.0, ctypes.c_void_p(A.data_ptr()), A.shape[1],
                                   ctypes.c_void_p(B.data_ptr()), B.shape[1], 0.0, ctypes.c_void_p(C.data_ptr()),
                                   case["M"], int(case["lower"]),
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc != 0:
        raise RuntimeError("msdp_tc_gemm returned %d" % rc)
    return C


# ---------------------------------------------------------------- bytes and operations
def _iteration_work(sides, m, ns, dense_nnz, pair_nnz):
    """One interior-point iteration: 28 n^3 of block algebra, the Schur
    complement (A_j G' G products and the contraction, or entry pairs), its
    factorization and two solves, and the constraint data read once for each
    of A(X), A*(y) and the assembly."""
    n3 = sum(float(n) ** 3 for n in sides)
    n2 = sum(float(n) ** 2 for n in sides)
    flops = 28 * n3 + m ** 3 / 3.0 + 4.0 * m * m + m * m * ns + pair_nnz ** 2
    if dense_nnz:
        flops += sum(4.0 * n ** 3 * m + float(m) * m * n * (n + 1) / 2 for n in sides)
    return flops, 8.0 * (4 * n2 + m * m / 2 + m * ns) + 16.0 * (dense_nnz + pair_nnz)


def work(case):
    do = case["do"]
    if do == "solve":
        n = case["n"]
        f, b = _iteration_work([n], n, 0, 0, n)
        return {"bytes": 8.0 * (n * n + 2 * n) + b, "flops": min(case["max_iter"], 10) * f}  # about ten iterations to the tolerance
    if do == "iterate":
        sides = [case["n"]] if case["model"] == "maxcut" else _sides(case)
        m = case["n"] if case["model"] == "maxcut" else case["m"]
        dense = 0 if case["model"] == "maxcut" else sum(n * n for n in sides) * m
        f, b = _iteration_work(sides, m, case["ns"], dense, m if case["model"] == "maxcut" else 0)
        return {"bytes": SLICE * b, "flops": SLICE * f}
    if do == "batch":
        f = b = 0.0
        for t in range(8):  # mean over the range of sizes
            n = case["lo"] + (case["hi"] - case["lo"]) * (t + 0.5) / 8 + (1 if case["model"] == "sos" else 0)
            ft, bt = _iteration_work([n], 2 * n - 1 if case["model"] == "sos" else n, 0, 0,
                                     n * n if case["model"] == "sos" else n)
            f, b = f + ft / 8, b + bt / 8
        return {"bytes": SLICE * case["count"] * b, "flops": SLICE * case["count"] * f}
    if do == "scaling":
        n = float(case["n"])
        return {"bytes": 8 * 6 * n * n, "flops": 20 * n ** 3}
    if do == "assembly":
        n, m = float(case["n"]), float(case["m"])
        return {"bytes": 8 * (m * n * n + m * m + 2 * n * n), "flops": 4 * n ** 3 * m + m * m * n * n + 10 * n ** 3}
    if do == "schur":
        m = float(case["m"])
        return {"bytes": 8 * (m * m + 2 * m), "flops": m ** 3 / 3 + 4 * m * m}
    half = 0.5 if case["lower"] else 1.0
    operands = case["M"] * case["K"] * (1 if case["lower"] else 2) if case["M"] == case["N"] else \
        (case["M"] + case["N"]) * case["K"]
    return {"bytes": 8.0 * (operands + half * case["M"] * case["N"]),
            "flops": 2.0 * half * case["M"] * case["N"] * case["K"]}


# ---------------------------------------------------------------- values in 64 bits
def _scaling_exact(X, S):
    """W = S^-1/2 (S^1/2 X S^1/2)^1/2 S^-1/2 and S^-1."""
    L = np.linalg.cholesky(S)
    lam, V = np.linalg.eigh(L.T @ X @ L)
    Li = np.linalg.inv(L)
    R = Li.T @ V
    return (R * np.sqrt(lam)) @ R.T, Li.T @ Li


def exact(case, seed):
    do = case["do"]
    if do == "scaling":
        X, S, _, L, D = _scaling_inputs(case, seed)
        W, Si = _scaling_exact(X, S)
        Li = np.linalg.inv(L)
        Z = Li @ D @ Li.T
        return {"ok": None, "W": W, "Sinv": Si, "lam": float(np.linalg.eigvalsh((Z + Z.T) / 2)[0])}
    if do == "assembly":
        model, X, S, _, x, z = _assembly_inputs(case, seed)
        n, m = case["n"], case["m"]
        block = model.A[0]
        A = np.zeros((m, n, n))
        A[block.con, block.row, block.col] = block.val
        W, Si = _scaling_exact(X, S)
        T = np.matmul(np.matmul(Si, A), X) if case["direction"] == "HKM" else np.matmul(np.matmul(W, A), W)
        H = A.reshape(m, -1) @ T.reshape(m, -1).T + (model.C_lin * (x / z)) @ model.C_lin.T
        return {"ok": None, "H": np.tril(H)}
    if do == "schur":
        H, rhs = _schur_inputs(case, seed)
        return {"ok": None, "x": np.linalg.solve(H, rhs)}
    if do == "product":
        A, B = _product_inputs(case, seed)
        opA = A if case["ta"] else A.t()
        opB = B if case["tb"] else B.t()
        C = opA @ opB
        return (torch.tril(C) if case["lower"] else C).t().contiguous()
    return None
