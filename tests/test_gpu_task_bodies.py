"""Parity of the four task bodies (C ABI) with the CPU oracle.

Each case runs the same seeded inputs through the GPU entry point and through
the oracle's restatement of the reference body; FP64 results must agree to
1e-12 relative (Frobenius), pivots exactly.
"""
import numpy as np
import pytest

from gpu_util import dev, host, ivec, relerr

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("n,c,ld", [(1, 1, 1), (7, 3, 9), (32, 16, 32), (33, 17, 40),
                                    (100, 1, 100), (256, 64, 300), (512, 592, 512),
                                    (1000, 40, 1003), (1024, 5, 1024)])
def test_leaf_solve(fs, oracle, cuda, n, c, ld):
    rng = np.random.default_rng(n * 1000 + c)
    D = rng.standard_normal((n, n)) / np.sqrt(n) + 2 * np.eye(n)
    X = rng.standard_normal((n, c))
    Dg, Xg, piv = dev(D, ld), dev(X, ld), ivec(n)
    assert fs.leaf_solve(Dg, Xg, piv) == 0
    Dr, Xr = np.asfortranarray(D.copy()), np.asfortranarray(X.copy())
    pr = np.zeros(n, dtype=np.int32)
    assert oracle.lib().ref_leaf_solve(n, c, oracle._p(Dr), n, oracle._p(Xr), n,
                                       pr.ctypes.data_as(oracle._ip)) == 0
    assert relerr(host(Xg), Xr) < TOL
    assert relerr(host(Dg), Dr) < TOL
    np.testing.assert_array_equal(piv.cpu().numpy()[:n], pr)


@pytest.mark.parametrize("n", [16, 100, 512])
def test_leaf_solve_needs_pivoting(fs, oracle, cuda, n):
    rng = np.random.default_rng(n)
    D = rng.standard_normal((n, n))  # no diagonal dominance: real interchanges
    X = rng.standard_normal((n, 9))
    Dg, Xg, piv = dev(D), dev(X), ivec(n)
    assert fs.leaf_solve(Dg, Xg, piv) == 0
    Dr, Xr = np.asfortranarray(D.copy()), np.asfortranarray(X.copy())
    pr = np.zeros(n, dtype=np.int32)
    oracle.lib().ref_leaf_solve(n, 9, oracle._p(Dr), n, oracle._p(Xr), n,
                                pr.ctypes.data_as(oracle._ip))
    np.testing.assert_array_equal(piv.cpu().numpy()[:n], pr)
    assert relerr(host(Dg), Dr) < 1e-11
    assert relerr(host(Xg), Xr) < 1e-10  # cond(D) ~ n for a Gaussian block


def test_leaf_solve_singular_reports_info(fs, oracle, cuda):
    n = 40
    D = np.eye(n)
    D[13, 13] = 0.0
    piv = ivec(n)
    info = fs.leaf_solve(dev(D), dev(np.ones((n, 2))), piv)
    Dr = np.asfortranarray(D.copy())
    Xr = np.asfortranarray(np.ones((n, 2)))
    assert info == oracle.lib().ref_leaf_solve(n, 2, oracle._p(Dr), n, oracle._p(Xr), n, None)
    assert info == 14


@pytest.mark.parametrize("k,r,ncol,col_beg", [(1, 1, 1, 0), (513, 30, 92, 2), (10000, 64, 80, 16),
                                               (131072, 64, 16, 0)])
def test_gemm_reduce(fs, oracle, cuda, k, r, ncol, col_beg):
    rng = np.random.default_rng(k + r)
    V = rng.standard_normal((k, r))
    U = rng.standard_normal((k, col_beg + ncol))
    W0 = rng.standard_normal((r, ncol))
    Vg, Ug, Wg = dev(V, k + 3), dev(U, k + 5), dev(W0, r + 1)
    fs.gemm_reduce(0.75, Vg, Ug, col_beg, ncol, Wg)
    Wr = np.asfortranarray(W0.copy())
    Vf, Uf = np.asfortranarray(V), np.asfortranarray(U)
    oracle.lib().ref_gemm_reduce(0.75, k, r, ncol, oracle._p(Vf), k, oracle._p(Uf), k, col_beg,
                                 oracle._p(Wr), r)
    assert relerr(host(Wg), Wr) < TOL


@pytest.mark.parametrize("k,r,c,u_col,d_col", [(1, 1, 1, 1, 0), (60, 30, 2, 62, 0),
                                                (512, 64, 528, 528, 0), (3000, 50, 358, 8, 58)])
def test_gemm_broadcast(fs, oracle, cuda, k, r, c, u_col, d_col):
    rng = np.random.default_rng(k * 7 + c)
    ncols = max(u_col + r, d_col + c)
    X = rng.standard_normal((k, ncols))
    eta = rng.standard_normal((r, c))
    Xg = dev(X, k + 2)
    fs.gemm_broadcast(-1.0, 1.0, Xg, u_col, r, dev(eta), d_col)
    Xr = np.asfortranarray(X.copy())
    etf = np.asfortranarray(eta)
    oracle.lib().ref_gemm_broadcast(-1.0, 1.0, k, r, c, oracle._p(Xr), k, u_col,
                                    oracle._p(etf), r, d_col)
    assert relerr(host(Xg), Xr) < TOL


@pytest.mark.parametrize("r,c", [(1, 1), (7, 3), (30, 92), (64, 592), (100, 40)])
@pytest.mark.parametrize("form", ["lu", "schur2"])
def test_node_solve(fs, oracle, cuda, r, c, form):
    if form == "schur2" and 2 * r > 144:
        pytest.skip("2r x 2r form is limited to 2r <= 144")
    rng = np.random.default_rng(r * 13 + c)
    V0Tu0 = 0.3 * rng.standard_normal((r, r)) / np.sqrt(r)
    V1Tu1 = 0.3 * rng.standard_normal((r, r)) / np.sqrt(r)
    V0Td0 = rng.standard_normal((r, c))
    V1Td1 = rng.standard_normal((r, c))
    g = [dev(V0Tu0, r + 1), dev(V1Tu1), dev(V0Td0, r + 2), dev(V1Td1)]
    fn = fs.node_lu_solve if form == "lu" else fs.node_schur2_solve
    assert fn(*g) == 0
    a = [np.asfortranarray(x.copy()) for x in (V0Tu0, V1Tu1, V0Td0, V1Td1)]
    ref = oracle.lib().ref_lu_node_solve if form == "lu" else oracle.lib().ref_schur2_solve
    assert ref(r, r, c, oracle._p(a[0]), r, oracle._p(a[1]), r, oracle._p(a[2]), r,
               oracle._p(a[3]), r) == 0
    assert relerr(host(g[2]), a[2]) < TOL
    assert relerr(host(g[3]), a[3]) < TOL


def test_node_solve_singular(fs, cuda):
    r = 5
    # S = I - V1Tu1 V0Tu0 = 0  when V1Tu1 = V0Tu0 = I
    g = [dev(np.eye(r)), dev(np.eye(r)), dev(np.ones((r, 2))), dev(np.ones((r, 2)))]
    assert fs.node_lu_solve(*g) > 0


def _gemm_bound(K, AB, C):
    """Elementwise rounding bound of C + A B over K terms, any order of sums: (K + 3) u each."""
    return (K + 3) * np.finfo(np.float64).eps * (AB + C)


@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("k,r,c", [(1, 1, 33), (31, 5, 63), (32, 16, 64), (33, 17, 65),
                                   (63, 15, 100), (64, 32, 128), (65, 33, 129), (127, 48, 40),
                                   (128, 100, 190), (129, 31, 64), (1000, 64, 257),
                                   (20011, 37, 129),
                                   # at most 32 columns: blocks of 128 rows, and of 512
                                   (1, 1, 1), (127, 15, 8), (128, 16, 9), (129, 17, 16),
                                   (513, 64, 17), (5000, 33, 32), (75777, 20, 8),
                                   (80001, 33, 16), (76000, 7, 31)])
def test_dmma_tiles_elementwise(fs, cuda, k, r, c, odd):
    """The FP64 tile GEMM at the edges of its tiles and K stages, with operands
    on and off 16-byte boundaries, C added in front (beta = 1) and behind."""
    rng = np.random.default_rng(k + 7 * r + c)
    X = rng.standard_normal((k, c + r + 1))
    eta = rng.standard_normal((r, c))
    U, d = X[:, c + 1:c + 1 + r], X[:, :c]
    for alpha, beta in ((-1.0, 1.0), (1.0, 1.0), (0.5, -2.0)):
        Xg = dev(X, k + 1 + (k + odd) % 2)   # even and odd leading dimensions
        fs.gemm_broadcast(alpha, beta, Xg, c + 1, r, dev(eta, r + odd), 0)
        got = host(Xg)
        err = np.abs(got[:, :c] - (beta * d + alpha * (U @ eta)))
        lim = _gemm_bound(r, abs(alpha) * (np.abs(U) @ np.abs(eta)), abs(beta) * np.abs(d))
        assert (err <= lim).all()
        assert (got[:, c:] == X[:, c:]).all()
    V = rng.standard_normal((k, r))
    W0 = rng.standard_normal((r, c))
    Wg = dev(W0, r + odd)
    fs.gemm_reduce(0.75, dev(V, k + odd), dev(X, k + 2 * odd), 0, c, Wg)
    err = np.abs(host(Wg) - (W0 + 0.75 * (V.T @ d)))
    assert (err <= _gemm_bound(k, 0.75 * (np.abs(V).T @ np.abs(d)), np.abs(W0))).all()


@pytest.mark.parametrize("count,n,c", [(1, 512, 40), (5, 33, 40), (70, 130, 1), (300, 250, 3)])
def test_leaf_solve_batched_groups(fs, cuda, count, n, c):
    """Batched leaves of uneven sizes and leading dimensions, one-level and
    blocked, and more than one group of them."""
    import ctypes
    import torch
    from fastsolver_b200 import _lib

    class Desc(ctypes.Structure):
        _fields_ = [("D", ctypes.c_void_p), ("X", ctypes.c_void_p), ("ipiv", ctypes.c_void_p),
                    ("perm", ctypes.c_void_p), ("ldd", ctypes.c_longlong),
                    ("ldx", ctypes.c_longlong), ("n", ctypes.c_int), ("nrhs", ctypes.c_int)]

    rng = np.random.default_rng(count + n)
    arr = (Desc * count)()
    keep = []
    for q in range(count):
        nq = n - q % 7 if n > 7 else n
        A, B = rng.standard_normal((nq, nq)) + 4 * np.eye(nq), rng.standard_normal((nq, c))
        D, X, piv, perm = dev(A, n + q % 2), dev(B, n + 1), ivec(nq), ivec(nq)
        keep.append((A, B, D, X, perm))
        arr[q] = Desc(D.data_ptr(), X.data_ptr(), piv.data_ptr(), perm.data_ptr() if q % 3 else None,
                      n + q % 2, n + 1, nq, c)
        keep[-1] += (piv,)
    raw = torch.frombuffer(bytearray(bytes(arr)), dtype=torch.uint8).cuda()
    info = torch.full((count,), -1, dtype=torch.int32, device="cuda")
    assert _lib.lib.hodlr_leaf_solve_batched(count, raw.data_ptr(), n, c, info.data_ptr(), None) == 0
    assert (info == 0).all()
    for q, (A, B, D, X, perm, piv) in enumerate(keep):
        nq = A.shape[0]
        x = np.linalg.solve(A, B)
        # two backward-stable solves: a few n u of the condition number each
        assert relerr(host(X), x) <= 20 * nq * np.linalg.cond(A) * 2.0 ** -53
        if q % 3:
            LU, p = host(D), perm.cpu().numpy()[:nq]
            L = np.tril(LU, -1) + np.eye(nq)
            assert np.abs(L @ np.triu(LU) - A[p]).max() <= 4 * nq * 2.0 ** -53 * (
                np.abs(L) @ np.abs(np.triu(LU))).max()


def test_leaf_solve_captured(fs, cuda):
    """With a device INFO pointer the call enqueues only: a captured one replays
    on what the buffers then hold."""
    import torch
    rng = np.random.default_rng(8)
    n, c = 300, 20
    D, X, piv, info = dev(np.eye(n)), dev(np.ones((n, c))), ivec(n), ivec(1)
    st = torch.cuda.Stream()
    fs.leaf_solve(D, X, piv, info=info, stream=st)
    st.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        fs.leaf_solve(D, X, piv, info=info, stream=torch.cuda.current_stream())
    for _ in range(2):
        A, B = rng.standard_normal((n, n)) + 4 * np.eye(n), rng.standard_normal((n, c))
        D.copy_(dev(A))
        X.copy_(dev(B))
        g.replay()
        torch.cuda.synchronize()
        assert int(info[0]) == 0
        assert relerr(host(X), np.linalg.solve(A, B)) <= 20 * n * np.linalg.cond(A) * 2.0 ** -53


@pytest.mark.parametrize("r0,r1", [(1, 1), (8, 8), (9, 9), (16, 17), (40, 25), (56, 56), (57, 57),
                                   (72, 72), (73, 73), (104, 104), (105, 105), (144, 144),
                                   (10, 300), (144, 9)])
def test_node_elimination_edges(fs, cuda, r0, r1):
    """The blocked elimination at the edges of its panels, tiles and shared-memory
    layouts, unequal ranks included, with pivots off the diagonal."""
    rng = np.random.default_rng(r0 * 1000 + r1)
    V0Tu0 = rng.standard_normal((r1, r0)) / np.sqrt(r1)
    V1Tu1 = 2 * rng.standard_normal((r0, r1)) / np.sqrt(r0)
    V0Td0, V1Td1 = rng.standard_normal((r1, 5)), rng.standard_normal((r0, 5))
    S = np.eye(r0) - V1Tu1 @ V0Tu0
    eta0 = np.linalg.solve(S, V1Td1 - V1Tu1 @ V0Td0)
    eta1 = V0Td0 - V0Tu0 @ eta0
    g = [dev(V0Tu0, r1 + 1), dev(V1Tu1), dev(V0Td0, r1 + 2), dev(V1Td1)]
    assert fs.node_lu_solve(*g) == 0
    # the solve and the products around it: a few s u of S's condition number
    # and of the blocks' norms each
    lim = 50 * max(r0, r1) * np.linalg.cond(S) * 2.0 ** -53 * (
        1 + np.linalg.norm(V0Tu0, 2)) ** 2 * (1 + np.linalg.norm(V1Tu1, 2)) ** 2
    assert np.linalg.norm(host(g[3]) - eta0) <= lim * np.linalg.norm(eta0)
    assert np.linalg.norm(host(g[2]) - eta1) <= lim * np.linalg.norm(eta1)


@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (63, 7, 9), (64, 8, 128), (65, 9, 129), (100, 32, 100),
                                   (127, 16, 8), (128, 17, 64), (129, 31, 7), (255, 8, 127),
                                   (256, 16, 144), (257, 32, 16), (1000, 5, 300), (4000, 32, 100)])
def test_fp32_skinny_elementwise(fs, cuda, m, n, k, odd):
    """The FP32 products of at most 32 columns at the edges of their row, column
    and K blocks, on and off 16-byte boundaries, both orientations."""
    import torch
    from fastsolver_b200 import _lib
    rng = np.random.default_rng(m + 3 * n + 7 * k)

    def put(a, ld):
        t = torch.zeros((a.shape[1], ld), dtype=torch.float32, device="cuda")
        t[:, :a.shape[0]] = torch.from_numpy(np.ascontiguousarray(a.T))
        return t

    for trans in (0, 1):
        A = rng.standard_normal((k, m) if trans else (m, k)).astype(np.float32)
        B = rng.standard_normal((k, n)).astype(np.float32)
        C = rng.standard_normal((m, n)).astype(np.float32)
        lda, ldb, ldc = ((x + 3) // 4 * 4 + odd for x in (A.shape[0], k, m))
        for alpha, beta in ((1.0, 0.0), (-1.0, 1.0), (0.5, -2.0)):
            Ag, Bg, Cg = put(A, lda), put(B, ldb), put(C, ldc)
            assert _lib.lib.hodlr_gemm_f32(trans, m, n, k, alpha, Ag.data_ptr(), lda, Bg.data_ptr(),
                                           ldb, beta, Cg.data_ptr(), ldc, 0, None) == 0
            op = (A.T if trans else A).astype(np.float64)
            Bd, Cd = B.astype(np.float64), C.astype(np.float64)
            err = np.abs(Cg.cpu().numpy().T[:m].astype(np.float64) - (alpha * (op @ Bd) + beta * Cd))
            lim = (k + 4) * 2.0 ** -24 * (abs(alpha) * (np.abs(op) @ np.abs(Bd)) + abs(beta * Cd))
            assert (err <= lim).all()


def _batch_descs(D, X, piv, n, c):
    """Descriptors of the leaves D[i] (n x n), X[i] (n x c), contiguous and column-major."""
    import ctypes
    import torch

    class Desc(ctypes.Structure):
        _fields_ = [("D", ctypes.c_void_p), ("X", ctypes.c_void_p), ("ipiv", ctypes.c_void_p),
                    ("perm", ctypes.c_void_p), ("ldd", ctypes.c_longlong),
                    ("ldx", ctypes.c_longlong), ("n", ctypes.c_int), ("nrhs", ctypes.c_int)]

    arr = (Desc * D.shape[0])(*[Desc(D[i].data_ptr(), X[i].data_ptr(),
                                     piv[i].data_ptr() if piv is not None else None, None, n, n, n, c)
                                for i in range(D.shape[0])])
    return torch.frombuffer(bytearray(bytes(arr)), dtype=torch.uint8).cuda()


@pytest.mark.parametrize("count,n", [(300, 250), (400, 512), (170, 1000)])
def test_leaf_solve_batched_scratch(fs, cuda, count, n):
    """The call's scratch stays within 64 MB, and equal leaves get equal results
    whichever group they fall into."""
    import threading
    import torch
    from fastsolver_b200 import _lib
    gen = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, n, generator=gen, device="cuda", dtype=torch.float64)
    B = torch.randn(3, n, generator=gen, device="cuda", dtype=torch.float64)
    D, X = A.repeat(count, 1, 1), B.repeat(count, 1, 1)
    piv = torch.zeros(count, n, dtype=torch.int32, device="cuda")
    raw = _batch_descs(D, X, piv, n, 3)
    info = torch.zeros(count, dtype=torch.int32, device="cuda")
    small = torch.zeros(1, n, n, dtype=torch.float64, device="cuda")
    small[0].fill_diagonal_(1.0)
    one = _batch_descs(small, X[:1].clone(), piv, n, 3)
    assert _lib.lib.hodlr_leaf_solve_batched(1, one.data_ptr(), n, 3, info.data_ptr(), None) == 0
    torch.cuda.synchronize()
    low, done = [torch.cuda.mem_get_info()[0]], threading.Event()
    before = low[0]

    def watch():
        while not done.is_set():
            low[0] = min(low[0], torch.cuda.mem_get_info()[0])

    th = threading.Thread(target=watch)
    th.start()
    try:
        for _ in range(5):
            D.copy_(A.expand_as(D))
            X.copy_(B.expand_as(X))
            torch.cuda.synchronize()
            assert _lib.lib.hodlr_leaf_solve_batched(count, raw.data_ptr(), n, 3, info.data_ptr(),
                                                     None) == 0
    finally:
        done.set()
        th.join()
    assert (info == 0).all()
    assert before - low[0] <= (64 << 20) + (34 << 20)  # the pool grows by 32 MB
    assert (X == X[0]).all() and (D == D[0]).all() and (piv == piv[0]).all()
    x = torch.linalg.solve(A.T, B.T)
    assert float((X[0].T - x).norm() / x.norm()) <= 20 * n * float(torch.linalg.cond(A)) * 2.0 ** -53


@pytest.mark.parametrize("n", [1, 33, 300, 700])
def test_leaf_solve_batched_without_pivots(fs, cuda, n):
    """Descriptors without ipiv (and perm) are solved like those with them."""
    import torch
    from fastsolver_b200 import _lib
    gen = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(3, n, n, generator=gen, device="cuda", dtype=torch.float64)
    B = torch.randn(3, 2, n, generator=gen, device="cuda", dtype=torch.float64)
    out = []
    for piv in (torch.zeros(3, n, dtype=torch.int32, device="cuda"), None):
        D, X = A.clone(), B.clone()
        info = torch.full((3,), -1, dtype=torch.int32, device="cuda")
        raw = _batch_descs(D, X, piv, n, 2)
        assert _lib.lib.hodlr_leaf_solve_batched(3, raw.data_ptr(), n, 2, info.data_ptr(), None) == 0
        assert (info == 0).all()
        out.append((D, X))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    x = torch.linalg.solve(A.transpose(1, 2), B.transpose(1, 2)).transpose(1, 2)
    cond = float(torch.linalg.cond(A).max())
    assert float((out[1][1] - x).norm() / x.norm()) <= 20 * n * cond * 2.0 ** -53


def test_leaf_solve_batched_empty_leaves(fs, cuda):
    """A batch of leaves without rows, and one with some among others."""
    import torch
    from fastsolver_b200 import _lib
    none = torch.zeros(3, 0, 0, dtype=torch.float64, device="cuda")
    raw = _batch_descs(none, none, None, 0, 0)
    for max_n in (0, 7):
        info = torch.full((3,), -1, dtype=torch.int32, device="cuda")
        assert _lib.lib.hodlr_leaf_solve_batched(3, raw.data_ptr(), max_n, 0, info.data_ptr(),
                                                 None) == 0
        assert (info == 0).all()
    D = 2 * torch.eye(7, dtype=torch.float64, device="cuda").repeat(2, 1, 1)
    X = torch.ones(2, 1, 7, dtype=torch.float64, device="cuda")
    raw = torch.cat([_batch_descs(none[:1], none[:1], None, 0, 0), _batch_descs(D, X, None, 7, 1)])
    assert _lib.lib.hodlr_leaf_solve_batched(3, raw.data_ptr(), 7, 1, info.data_ptr(), None) == 0
    assert (info == 0).all() and (X == 0.5).all()


@pytest.mark.parametrize("s,width", [(9, 1.0), (16, 1.0), (17, 0.5), (37, 1.0), (64, 1.0), (100, 1.0),
                                     (144, 1.0)])
def test_node_elimination_ill_conditioned(fs, cuda, s, width):
    """An ill-conditioned S = I - V1Tu1 V0Tu0 (V1Tu1 = I): the residual of the
    column-by-column Gauss-Jordan elimination with partial pivoting."""
    x = np.linspace(0, 1, s)
    K = np.exp(-((x[:, None] - x) / width) ** 2) + 1e-12 * np.eye(s)
    V0Tu0 = np.eye(s) - K
    S = np.eye(s) - V0Tu0                      # as the kernel forms it
    d1 = np.random.default_rng(s).standard_normal((s, 3))
    g = [dev(V0Tu0), dev(np.eye(s)), dev(np.zeros((s, 3))), dev(d1)]
    assert fs.node_lu_solve(*g) == 0
    eta0 = host(g[3])
    A, p = S.copy(), np.arange(s)
    for k in range(s):
        j = k + int(np.argmax(np.abs(A[k:, k])))
        A[[k, j]], p[[k, j]] = A[[j, k]], p[[j, k]]
        A[k + 1:, k] /= A[k, k]
        A[k + 1:, k + 1:] -= np.outer(A[k + 1:, k], A[k, k + 1:])
    L, U = np.abs(np.tril(A, -1) + np.eye(s)), np.triu(A)
    Ui = np.linalg.inv(U)
    X = np.abs(Ui @ np.linalg.inv(np.tril(A, -1) + np.eye(s)))   # |S^{-1}| of the permuted rows
    aU = np.abs(U)
    # columns x_j of the inverse: |e_j - S x_j| <= 8 s u |L| |U| |U^{-1}| |U| |x_j|, and
    # s u |S| |X| |d| for the product with the right-hand sides
    w = X @ np.abs(d1[p])
    lim = s * 2.0 ** -53 * (8 * (L @ (aU @ (np.abs(Ui) @ (aU @ w)))) + np.abs(S[p]) @ w)
    r = np.abs((S.astype(np.longdouble) @ eta0 - d1).astype(np.float64))[p]
    assert (r <= lim).all(), (r / lim).max()
