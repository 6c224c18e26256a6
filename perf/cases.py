"""Performance cases of the HODLR solver: the calls its users make, over the sizes they make them at.

A case is one call (or the short sequence of calls) of the public interface:

  fp64     FastSolver.bfs_solve: the plain FP64 factor + solve of the loaded
           system, either node form, on a side stream (CUDA graphs) or on the
           default stream (eager launches)
  refined  FastSolver.solve_refined, mixed precision, to relres <= 1e-12
  resolve  FastSolver.solve with kept FP64 factors and a new right-hand side
  batch    SystemBatch.solve_refined of uneven systems
  host     FastSolver.solve_refined_host: pinned host memory in and out
  matvec   HodlrMatrix.matvec
  leaf     the leaf task body (leaf_solve) on one leaf block
  node     one internal node by its task bodies: a reduce per child, the node
           solve, a broadcast per child

Systems have leaf blocks G / sqrt(n) + 2 I, iid Gaussian U and V scaled so
that every off-diagonal block has spectral norm about 0.5 at most, and a
standard normal right-hand side.  Sizes are those of the benchmark's
workloads (N = 4096, 65536, 262144, 1048576; leaves of 256..1024 rows, ranks
16..100, 1..32 right-hand sides) and odd ones between them.
"""
from __future__ import annotations

import math
import random

import torch

import fastsolver_b200 as fs

TOL = 1e-12


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _system(kind, N, nrhs, rank, leaf, **more):
    return dict(kind=kind, N=N, nrhs=nrhs, rank=rank, leaf=leaf, **more)


def listed():
    return [
        # the small system of the reference's own CPU runs, default stream
        dict(name="fp64_n4096_default_stream", **_system("fp64", 4096, 1, 30, 256, schur2=False, side=False)),
        # an ordinary system whose size, rank and leaf match no tile
        dict(name="fp64_n60001_r37", **_system("fp64", 60001, 5, 37, 500, schur2=False, side=True)),
        # the plain FP64 solve of the headline system
        dict(name="fp64_n262144", **_system("fp64", 262144, 16, 64, 512, schur2=False, side=True)),
        # small refined solve: launches, barriers and host waits
        dict(name="refined_n4096", **_system("refined", 4096, 1, 30, 256, side=True)),
        # ordinary refined solve
        dict(name="refined_n65536", **_system("refined", 65536, 8, 50, 512, side=True)),
        # the headline: mixed factor + refinement
        dict(name="refined_n262144", **_system("refined", 262144, 16, 64, 512, side=True)),
        # the largest system, ranks and right-hand sides at their upper end
        dict(name="refined_n1048576", **_system("refined", 1048576, 32, 100, 512, side=True)),
        # factor once, solve many: one more right-hand side block
        dict(name="resolve_n131072", **_system("resolve", 131072, 16, 64, 512, side=True)),
        # many uneven systems at once
        dict(name="batch16", kind="batch", count=16, shapes=7, n_lo=8192, n_hi=131072),
        # the leaf task of the headline system's deepest columns [b | U]
        dict(name="leaf_n512_c592", kind="leaf", n=512, cols=592),
        # the tasks of one internal node at mid depth of the headline system
        dict(name="node_k16384_r64_c272", kind="node", k=16384, rank=64, cols=272),
        # host to host: the copies count
        dict(name="host_n65536", **_system("host", 65536, 8, 50, 512, side=True)),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["fp64", "refined", "resolve", "batch", "host", "matvec", "leaf", "node"],
                       [5, 6, 2, 2, 1, 1, 3, 3])[0]
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 16), shapes=rng.randrange(1 << 20),
                    n_lo=8192, n_hi=rng.choice([20000, 65536, 100000]))
    if kind == "leaf":
        n = _log(rng, 16, 1024)
        return dict(kind=kind, n=n, cols=_log(rng, 1, 1132))
    if kind == "node":
        return dict(kind=kind, k=_log(rng, 200, 131072), rank=rng.randint(8, 100),
                    cols=_log(rng, 1, 700))
    leaf = rng.choice([200, 256, 300, 512, 512, 700, 1024])
    rank = rng.randint(8, min(96, leaf // 2 - 1))
    hi = 65536 if kind == "host" else 262144
    case = _system(kind, _log(rng, 1500, hi), rng.randint(1, 32), rank, leaf,
                   side=rng.random() < 0.75)
    if kind == "fp64":
        case["schur2"] = 2 * rank <= 144 and rng.random() < 0.2
    return case


# ---------------------------------------------------------------------------
# trees and seeded inputs
# ---------------------------------------------------------------------------

def _tree(N, threshold):
    """Nodes (row, rows, depth, left, right) of the halving tree, parents first."""
    nodes = [[0, N, 0, -1, -1]]
    for q in nodes:
        if q[1] > threshold:
            q[3], q[4] = len(nodes), len(nodes) + 1
            h = q[1] // 2
            nodes.append([q[0], h, q[2] + 1, -1, -1])
            nodes.append([q[0] + h, q[1] - h, q[2] + 1, -1, -1])
    return nodes


def _shape(case):
    nodes = _tree(case["N"], case["leaf"])
    return nodes, max(q[2] for q in nodes), max(q[1] for q in nodes if q[3] < 0)


def _colmajor(rows, cols, gen):
    return torch.randn(cols, rows, generator=gen, device="cuda", dtype=torch.float64).T


def _inputs(case, seed):
    """(D, U, V, B), column-major on the GPU, in the library's global layout: D's
    leaf blocks stacked, column block r (d - 1) of U and V for the nodes of depth d."""
    nodes, depth, nmax = _shape(case)
    N, r = case["N"], case["rank"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    D = _colmajor(N, nmax, gen)
    U = _colmajor(N, r * depth, gen)
    V = _colmajor(N, r * depth, gen)
    B = _colmajor(N, case["nrhs"], gen)
    # per row: its leaf's size and first row; per depth: the scale of U and V
    scale = torch.zeros(max(depth, 1), N, dtype=torch.float64)
    leaf = torch.zeros(2, N, dtype=torch.int64)
    for row, n, d, left, _ in nodes:
        if d > 0:
            scale[d - 1, row:row + n] = math.sqrt(0.5) / (math.sqrt(n) + math.sqrt(r))
        if left < 0:
            leaf[0, row:row + n] = n
            leaf[1, row:row + n] = row
    scale, leaf = scale.cuda(), leaf.cuda()
    for d in range(depth):
        U[:, r * d:r * (d + 1)] *= scale[d].unsqueeze(1)
        V[:, r * d:r * (d + 1)] *= scale[d].unsqueeze(1)
    at = torch.arange(N, device="cuda")
    D *= leaf[0].double().rsqrt().unsqueeze(1)
    if int(leaf[0].min()) < nmax:
        D *= torch.arange(nmax, device="cuda") < leaf[0].unsqueeze(1)
    D[at, at - leaf[1]] += 2.0
    return D, U, V, B


def _load(case, seed):
    D, U, V, B = _inputs(case, seed)
    h = fs.HodlrMatrix(case["nrhs"], case["N"], case["rank"], case["leaf"]).create_tree()
    some = U.shape[1] > 0
    torch.cuda.synchronize()
    h.set_matrix(D, U if some else None, V if some else None)
    h.set_rhs(B)
    torch.cuda.synchronize()
    return h


def _batch_shapes(case):
    rng = random.Random(case["shapes"])
    return [_system("refined", _log(rng, case["n_lo"], case["n_hi"]), rng.randint(1, 32),
                    rng.randint(16, 96), rng.choice([256, 512, 1024]))
            for _ in range(case["count"])]


def _leaf_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]
    D = _colmajor(n, n, gen) / math.sqrt(n)
    D += 2.0 * torch.eye(n, device="cuda", dtype=torch.float64)
    return D, _colmajor(n, case["cols"], gen)


def _node_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k, r, c = case["k"], case["rank"], case["cols"]
    out = []
    for rows in (k, k + 1):
        V = _colmajor(rows, r, gen) * (0.7 / (math.sqrt(rows) + math.sqrt(r)))
        X = _colmajor(rows, c + r, gen)
        X[:, c:] *= 0.7 / (math.sqrt(rows) + math.sqrt(r))
        out += [V, X]
    return out


def _empty(rows, cols):
    return torch.empty(cols, rows, device="cuda", dtype=torch.float64).T


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "leaf":
        D, X = _leaf_inputs(case, seed)
        n, c = case["n"], case["cols"]
        st.update(D0=D, X0=X, D=_empty(n, n), X=_empty(n, c),
                  ipiv=torch.zeros(n, dtype=torch.int32, device="cuda"))
        return st
    if kind == "node":
        V0, X0, V1, X1 = _node_inputs(case, seed)
        r, c = case["rank"], case["cols"]
        st.update(V0=V0, V1=V1, X0=X0, X1=X1, d0=X0[:, :c].T.clone().T, d1=X1[:, :c].T.clone().T,
                  W0=_empty(r, c + r), W1=_empty(r, c + r))
        return st
    st["stream"] = torch.cuda.Stream() if case.get("side", True) else None
    if kind == "batch":
        shapes = _batch_shapes(case)
        st["systems"] = [_load(s, seed + 1000 * i) for i, s in enumerate(shapes)]
        st["batch"] = fs.SystemBatch(st["systems"])
        st["out"] = [_empty(s["N"], s["nrhs"]) for s in shapes]
        torch.cuda.empty_cache()
        return st
    N, m = case["N"], case["nrhs"]
    st["solver"] = fs.FastSolver()
    if kind == "host":
        host = []
        for x in _inputs(case, seed):
            p = torch.empty(x.shape[1], x.shape[0], dtype=torch.float64, pin_memory=True)
            p.copy_(x.T)
            host.append(p.T)
        st["h"] = fs.HodlrMatrix(m, N, case["rank"], case["leaf"]).create_tree()
        st["host"] = host
        st["out"] = torch.empty(m, N, dtype=torch.float64, pin_memory=True).T
        torch.cuda.empty_cache()
        return st
    st["h"] = _load(case, seed)
    st["out"] = _empty(N, m)
    gen = torch.Generator(device="cuda").manual_seed(seed + 77)
    if kind == "resolve":
        st["solver"].factor(st["h"], fs.PREC_FP64, stream=st["stream"])
        st["B"] = _colmajor(N, m, gen)
    elif kind == "matvec":
        st["x"] = _colmajor(N, m, gen)
    torch.cuda.empty_cache()
    return st


def run(st):
    kind = st["kind"]
    if kind == "leaf":
        st["D"].copy_(st["D0"])
        st["X"].copy_(st["X0"])
        fs.leaf_solve(st["D"], st["X"], st["ipiv"])
        return [st["D"], st["X"], st["ipiv"]]
    if kind == "node":
        c, r = st["case"]["cols"], st["case"]["rank"]
        for i in "01":
            X, W = st["X" + i], st["W" + i]
            X[:, :c].copy_(st["d" + i])
            W.zero_()
            fs.gemm_reduce(1.0, st["V" + i], X, 0, c + r, W)
        W0, W1 = st["W0"], st["W1"]
        fs.node_lu_solve(W0[:, c:], W1[:, c:], W0[:, :c], W1[:, :c])
        fs.gemm_broadcast(-1.0, 1.0, st["X0"], c, r, W1[:, :c], 0)
        fs.gemm_broadcast(-1.0, 1.0, st["X1"], c, r, W0[:, :c], 0)
        return [st["X0"], st["X1"], W0, W1]
    s = st["stream"]
    if kind == "batch":
        st["batch"].solve_refined(tol=TOL, maxiter=10, stream=s)
        for h, out in zip(st["systems"], st["out"]):
            h.solution_to(out, stream=s)
        return st["out"]
    h, out, solver = st["h"], st["out"], st["solver"]
    if kind == "fp64":
        solver.bfs_solve(h, schur2=st["case"]["schur2"], stream=s)
    elif kind == "refined":
        solver.solve_refined(h, fs.PREC_MIXED, tol=TOL, maxiter=10, stream=s)
    elif kind == "resolve":
        h.set_rhs(st["B"], stream=s)
        solver.solve(h, stream=s)
    elif kind == "matvec":
        h.matvec(st["x"], out, stream=s)
        return out
    elif kind == "host":
        solver.solve_refined_host(h, *st["host"], out=out, tol=TOL, maxiter=10, stream=s)
        return out
    h.solution_to(out, stream=s)
    return out


# ---------------------------------------------------------------------------
# work: each input read once, each output written once; the operations of the
# factorization and of the solve (one pass of them, whatever the precision)
# ---------------------------------------------------------------------------

def _system_work(case):
    nodes, depth, nmax = _shape(case)
    N, m, r, kind = case["N"], case["nrhs"], case["rank"], case["kind"]
    factor = kind in ("fp64", "refined", "host")
    flops = words = 0.0
    for _, n, d, left, right in nodes:
        if left < 0:
            c = m + r * d if factor else m
            flops += (2.0 / 3.0 * n ** 3 if factor else 0.0) + 2.0 * n * n * c
            words += float(n) * n
            continue
        c = m + r * d if factor else m      # columns in front of the children's own
        cr = c + r if factor else c
        flops += 2.0 * n * r * (cr + c) + (2.0 * r ** 3 * 4 if factor else 0.0) + 8.0 * r * r * c
    words += 2.0 * N * r * depth + 2.0 * N * m
    return 8.0 * words, flops


def work(case):
    kind = case["kind"]
    if kind == "leaf":
        n, c = case["n"], case["cols"]
        return {"bytes": 16.0 * (n * n + n * c), "flops": 2.0 / 3.0 * n ** 3 + 2.0 * n * n * c}
    if kind == "node":
        k, r, c = case["k"], case["rank"], case["cols"]
        return {"bytes": 8.0 * 2 * k * (2 * r + 2 * c),
                "flops": 2 * (2.0 * k * r * (c + r) + 2.0 * k * r * c) + 8.0 * r ** 3 + 8.0 * r * r * c}
    parts = [_system_work(s) for s in (_batch_shapes(case) if kind == "batch" else [case])]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


# ---------------------------------------------------------------------------
# exact: the same results by torch in 64 bits
# ---------------------------------------------------------------------------

def _exact_solve(case, D, U, V, B):
    """The HODLR solve, node by node (Woodbury at every internal node)."""
    nodes, depth, _ = _shape(case)
    m, r = case["nrhs"], case["rank"]
    X = torch.cat([B.T, U.T]).T.contiguous()          # rows x [b | U]
    eye = torch.eye(r, device="cuda", dtype=torch.float64)
    for row, n, d, left, right in reversed(nodes):
        if left < 0:
            c = m + r * d
            X[row:row + n, :c] = torch.linalg.solve(D[row:row + n, :n], X[row:row + n, :c])
            continue
        c = m + r * d
        halves = []
        for q in (left, right):
            a, k = nodes[q][0], nodes[q][1]
            x = X[a:a + k, :c + r]
            halves.append((x, V[a:a + k, r * d:r * (d + 1)].T @ x))
        (x0, w0), (x1, w1) = halves
        s = eye - w1[:, c:] @ w0[:, c:]
        eta0 = torch.linalg.solve(s, w1[:, :c] - w1[:, c:] @ w0[:, :c])
        eta1 = w0[:, :c] - w0[:, c:] @ eta0
        x0[:, :c] -= x0[:, c:] @ eta0
        x1[:, :c] -= x1[:, c:] @ eta1
    return X[:, :m]


def exact(case, seed):
    kind = case["kind"]
    if kind == "leaf":
        D, X = _leaf_inputs(case, seed)
        lu, _ = torch.linalg.lu_factor(D.cpu())
        return [lu, torch.linalg.solve(D, X), None]
    if kind == "node":
        V0, X0, V1, X1 = _node_inputs(case, seed)
        c, r = case["cols"], case["rank"]
        w0, w1 = V0.T @ X0, V1.T @ X1
        s = torch.eye(r, device="cuda", dtype=torch.float64) - w1[:, c:] @ w0[:, c:]
        eta0 = torch.linalg.solve(s, w1[:, :c] - w1[:, c:] @ w0[:, :c])
        eta1 = w0[:, :c] - w0[:, c:] @ eta0
        X0[:, :c] -= X0[:, c:] @ eta0
        X1[:, :c] -= X1[:, c:] @ eta1
        return [X0, X1, torch.cat([eta1, w0[:, c:]], 1), torch.cat([eta0, w1[:, c:]], 1)]
    if kind == "batch":
        return [_exact_solve(s, *_inputs(s, seed + 1000 * i))
                for i, s in enumerate(_batch_shapes(case))]
    if case["N"] > 400000:
        return None
    D, U, V, B = _inputs(case, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed + 77)
    if kind == "resolve":
        return _exact_solve(case, D, U, V, _colmajor(case["N"], case["nrhs"], gen))
    if kind != "matvec":
        x = _exact_solve(case, D, U, V, B)
        return x.cpu() if kind == "host" else x
    x = _colmajor(case["N"], case["nrhs"], gen)
    y = torch.empty_like(x)
    nodes, r = _tree(case["N"], case["leaf"]), case["rank"]
    for row, n, _, left, _ in nodes:
        if left < 0:
            y[row:row + n] = D[row:row + n, :n] @ x[row:row + n]
    for _, _, d, left, right in nodes:
        if left < 0:
            continue
        for p, q in ((left, right), (right, left)):
            (a, k), (b, l) = nodes[p][:2], nodes[q][:2]
            col = slice(r * d, r * (d + 1))
            y[a:a + k] += U[a:a + k, col] @ (V[b:b + l, col].T @ x[b:b + l])
    return y
